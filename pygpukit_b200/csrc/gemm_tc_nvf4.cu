// gemm_tc_nvf4.cu -- NVF4 (W4A16) products of a few dozen rows on the 5th-gen tensor cores (tcgen05 + TMEM + TMA).
//
//   C[M,N] = alpha * A[M,K] . dequant(Bd[K/2,N], Bs[K/32,N])     Bd: two E2M1 nibbles per byte (low = even k),
//                                                                 Bs: UE4M3 scale per (32 k, column), 1 <= M <= 64
//
// replaces the batched use of gemv_nvf4_bf16_kernel (native/ops/matmul/gemv/w4a16_bf16/sm120/nvf4_kernels.cu:79-233: one
// launch per row, weights re-read M times) and the role of the CUTLASS NVF4 GEMM the reference cannot build here
// (native/ops/matmul/gemm/w4a16_bf16/sm120/nvf4_cutlass.cu).  Forms: plain; a gate/up matrix interleaved by eight columns with silu(gate) * up;
// the experts of a mixture -- gate and up matrices with silu(gate) * up over gathered rows, and the down product of the sorted rows.
//
// What bounds it: the conversion of the nibbles -- three instructions a weight, 590 issue slots of an SM per block of 128 columns x 128 k, where
// the block's way from HBM is 360 cycles; 890 are seen.  What follows from that, as in gemm_tc.cu:
//   * transposed, D^T[n, m]: a TMEM lane per weight column, the batch is the MMA's N (16 / 32 / 64); the weights are the MMA's A operand in
//     TENSOR MEMORY, whose 32-bit element (lane, column) is a pair of neighbouring k -- exactly one byte of Bd.  A thread reads the bytes of
//     its column one by one (a warp's 32 bytes lie side by side), puts their bits where BF16 has them and multiplies by the scale: an E2M1
//     value has two significant bits, a UE4M3 scale four, the product is exact;
//   * the nibble's exponent goes into BF16's own as it is, which makes it 2^-126 of its value -- its subnormal 0.5 a subnormal of BF16 --, and the
//     scale's exponent brings it back up to a factor 2^8 (480 x 2^126 would not fit BF16), which the sums are multiplied by at the end;
//   * TMA brings codes, scales and activations (128-byte swizzle) into a ring; eight warps convert, one copies, one issues the MMAs; two blocks
//     per SM hide each other's start and end; K is cut over a cluster that pushes its partial rows to their owners' shared memory: no work memory;
//   * experts: a block per (slice of k, column tile, expert that has rows); the rows of an expert are at most the tokens of the call.  Gate
//     and up fetch their rows by token (gathering copies of four rows), down finds them in the experts' order.
// Measured on B200 (us, a pass of a feed-forward or mixture; conversion into shared memory and a launch for the activation, experts row by row ->
// here): 19 rows 2176 / 17280 72 -> 37, 28 rows 5376 / 3200 56 -> 27, 9 rows 6656 / 4864 74 -> 36; 45 tokens through 128 experts of 1792 /
// 896, eight each, 498 -> 176, 13 through eight of 3200 / 1920, two each, 154 -> 53.  37888 x 8192 alone: 60 (16 rows), 66 (64 rows), 2.7 TB/s.
#include "common.cuh"
#include "gemv_common.cuh"
#include "tc_common.cuh"
#include "tma.cuh"
#include "../../include/pgk_b200.h"

#include <cmath>
#include <initializer_list>

namespace pgk {

namespace {

constexpr int Q_BK = 128;                         // k per block: 64 rows of codes, 4 of scales
constexpr int Q_WARPS = 8;                        // conversion and output; one more for the copies, one for the MMAs
constexpr int Q_THREADS = (Q_WARPS + 2) * 32;
constexpr uint32_t Q_CODES = 64 * 128, Q_SCALES = 4 * 128;
constexpr int Q_MAX_TILES = 8192;
enum { Q_PLAIN, Q_SWIGLU, Q_GATEUP, Q_DOWN };     // the two last: experts
// 16 rows leave room for a third block per SM, with one converted block in tensor memory instead of three (us, 896 x 75776: 22.3 -> 20.8, 8192 x
// 18944 42.0 -> 40.5; 32 rows the same or slower)
__host__ __device__ constexpr int q_stages(int nb) { return nb <= 16 ? 5 : (nb <= 32 ? 6 : 4); }
__host__ __device__ constexpr int q_bufs(int nb) { return nb <= 16 ? 1 : 3; }                        // converted blocks in tensor memory
__host__ __device__ constexpr int q_blocks(int nb) { return nb <= 16 ? 3 : 2; }                      // blocks per SM
__host__ __device__ constexpr uint32_t q_stage_bytes(int nb) { return (uint32_t)nb * 256 + Q_CODES + 1024; }
__host__ __device__ constexpr size_t q_smem(int nb) { return (size_t)q_stages(nb) * q_stage_bytes(nb) + 1024; }

struct N4Params {
    uint16_t* C; const uint16_t* bias; const uint16_t* residual;
    int M, K, N, splits, kper;                    // N: columns of one matrix
    float alpha;
    const int* active; const int* first; const int* token;        // experts that have rows (their number first), first row of each, token of each row
    int offset;                                   // the expert whose matrix comes first
    int ahead;                                    // the first codes are read before the kernel before has finished
    int* err;                                     // raised when a bounded wait runs out
};

__device__ __forceinline__ uint32_t lds_u8(uint32_t at) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}
// a byte's two E2M1 values as BF16 times 2^-126: low nibble in the lower half
__device__ __forceinline__ uint32_t e2m1x2_to_bf16x2(uint32_t b) {
    return ((b * 0x00040040u) & 0x01c001c0u) | ((b * 0x01001000u) & 0x80008000u);
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// UE4M3 (bit 7 ignored, exponent 0 is normal) times 2^118, twice
__device__ __forceinline__ uint32_t ue4m3_to_bf16x2(uint32_t s) { return (((s & 0x7fu) << 4) + 0x7700u) * 0x00010001u; }

template <int NB, int FORM>
__global__ void __launch_bounds__(Q_THREADS, q_blocks(NB))
gemm_nvf4_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap smap, const __grid_constant__ CUtensorMap umap,
                    const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap amap, const __grid_constant__ N4Params p) {
    constexpr bool EXPERTS = FORM == Q_GATEUP || FORM == Q_DOWN, TWO = FORM == Q_GATEUP;
    constexpr int STAGES = q_stages(NB), COLS = NB / 2, TILE = TWO ? 64 : 128;       // TILE: columns of one matrix
    constexpr uint32_t STAGE = q_stage_bytes(NB), ACTS = NB * 256, TMEM_COLS = NB <= 16 ? 128 : 256;
    constexpr int Q_BUFS = q_bufs(NB);
    static_assert(NB + 64 * Q_BUFS <= (int)TMEM_COLS && q_blocks(NB) * (int)TMEM_COLS <= 512, "blocks per SM");
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], ready_bar[Q_BUFS], free_bar[Q_BUFS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int token_s[TWO ? NB : 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t ring = (smem_u32(smem) + 1023u) & ~1023u, full = smem_u32(full_bar), empty = smem_u32(empty_bar);
    const uint32_t ready = smem_u32(ready_bar), freed = smem_u32(free_bar);
    int* const err = p.err;
    const int rank = blockIdx.x, n0 = blockIdx.y * TILE, nkb_total = p.K / Q_BK;
    const int kb0 = rank * p.kper, nkb = max(0, min(nkb_total, kb0 + p.kper) - kb0);

    int z = 0, row0 = 0, rows = min(NB, p.M);
    if (EXPERTS || !p.ahead) griddep_wait();
    if constexpr (EXPERTS) {
        if ((int)blockIdx.z >= p.active[0]) return;       // the same in the whole cluster
        z = p.active[1 + blockIdx.z];
        row0 = p.first[z];
        rows = min(NB, p.first[z + 1] - row0);
        z -= p.offset;
        if (TWO && tid < NB) token_s[tid] = p.token[row0 + min(tid, rows - 1)];
    }
    if (warp == Q_WARPS + 1) tmem_alloc(&tmem_base_s, TMEM_COLS);
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < Q_BUFS; ++b) { mbar_init(&ready_bar[b], Q_WARPS); mbar_init(&free_bar[b], 1); }
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" :: "l"(&wmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&amap) : "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s, tmem_w = tmem + NB;       // the sums, then blocks of weights (64 columns each)

    if (warp == Q_WARPS) {
        // ---------------- copies; the first weights leave before the dependency wait
        if (elect_one()) {
            const uint64_t once = l2_evict_first();
            const int quads = TWO ? (rows + 3) / 4 : 0;
            const uint32_t bytes = Q_CODES + Q_SCALES + (TWO ? (uint32_t)quads * 1024u : ACTS);
            auto weights = [&](int it, uint32_t s) {
                const uint32_t at = ring + s * STAGE + ACTS, bar = full + 8u * s;
                mbar_expect_tx(bar, bytes);
                tma_load_3d_hint(at, &wmap, n0, (kb0 + it) * 64, z, bar, once);
                tma_load_3d_hint(at + Q_CODES, &smap, n0, (kb0 + it) * 4, z, bar, once);
                if constexpr (TWO) {
                    tma_load_3d_hint(at + Q_CODES / 2, &umap, n0, (kb0 + it) * 64, z, bar, once);
                    tma_load_3d_hint(at + Q_CODES + Q_SCALES / 2, &tmap, n0, (kb0 + it) * 4, z, bar, once);
                }
            };
            auto acts = [&](int it, uint32_t s) {
                const uint32_t at = ring + s * STAGE, bar = full + 8u * s;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    if constexpr (TWO) {
                        for (int q = 0; q < quads; ++q)
                            tma_gather4(at + (uint32_t)c * (NB * 128u) + (uint32_t)q * 512u, &amap, (kb0 + it) * Q_BK + c * 64, token_s[4 * q], token_s[4 * q + 1], token_s[4 * q + 2], token_s[4 * q + 3], bar);
                    } else
                        tma_load_2d(at + (uint32_t)c * (NB * 128u), &amap, (kb0 + it) * Q_BK + c * 64, row0, bar);
                }
            };
            const int first = min(nkb, STAGES);
            for (int it = 0; it < first; ++it) weights(it, (uint32_t)it);
            griddep_wait();
            griddep_launch();
            for (int it = 0; it < first; ++it) acts(it, (uint32_t)it);
            RingPos r;
            r.round = 1;
            int it = first;
            for (; it < nkb; ++it, r.next(STAGES)) {
                if (!bar_wait(err, empty + 8u * r.s, r.round ^ 1u)) break;
                weights(it, r.s);
                acts(it, r.s);
            }
            for (int j = max(0, it - STAGES); j < it; ++j)    // whoever gave up: do not leave with copies in flight
                bar_wait(err, full + 8u * (uint32_t)(j % STAGES), (uint32_t)((j / STAGES) & 1));
        } else {
            griddep_wait();
            griddep_launch();
        }
        __syncwarp();
    } else if (warp == Q_WARPS + 1) {
        // ---------------- MMAs
        griddep_wait();
        griddep_launch();
        if (elect_one()) {
            constexpr uint32_t idesc = umma_idesc_bf16(NB);
            RingPos r, w;
            for (int it = 0; it < nkb; ++it, r.next(STAGES), w.next(Q_BUFS)) {
                if (!bar_wait(err, full + 8u * r.s, r.round) || !bar_wait(err, ready + 8u * w.s, w.round)) break;
                tc_fence_after();
                const uint32_t a_s = ring + r.s * STAGE;
#pragma unroll
                for (int ks = 0; ks < Q_BK / 16; ++ks)
                    umma_bf16_ta(tmem, tmem_w + w.s * 64u + (uint32_t)ks * 8u, desc_sw128(a_s + (uint32_t)(ks >> 2) * (NB * 128u)) + (uint64_t)((ks & 3) * 2), idesc,
                                 (it > 0 || ks > 0) ? 1u : 0u);
                umma_commit(&free_bar[w.s]);
                umma_commit(&empty_bar[r.s]);
            }
        }
        __syncwarp();
    } else {
        // ---------------- codes -> TMEM
        griddep_wait();
        griddep_launch();
        const int quad = warp & 3, half = warp >> 2, col = quad * 32 + lane;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        // where the thread's column starts in a stage: rows of TILE bytes, the second matrix behind the first
        const uint32_t code_at = ACTS + (TWO ? (uint32_t)(quad >> 1) * (Q_CODES / 2) : 0u) + (uint32_t)(col & (TILE - 1)) + (uint32_t)half * (32 * TILE);
        const uint32_t scale_at = ACTS + Q_CODES + (TWO ? (uint32_t)(quad >> 1) * (Q_SCALES / 2) : 0u) + (uint32_t)(col & (TILE - 1)) + (uint32_t)half * (2 * TILE);
        bool ok = true;
        RingPos r, w;
        for (int it = 0; it < nkb; ++it, r.next(STAGES), w.next(Q_BUFS)) {
            const uint32_t st = ring + r.s * STAGE;
            ok = ok && bar_wait(err, full + 8u * r.s, r.round);
            __syncwarp();
            uint32_t b[32], s[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) s[h] = lds_u8(st + scale_at + (uint32_t)(h * TILE));
#pragma unroll
            for (int i = 0; i < 32; ++i) b[i] = lds_u8(st + code_at + (uint32_t)(i * TILE));
            if (it >= Q_BUFS) {                               // the products that read this buffer are done
                ok = ok && bar_wait(err, freed + 8u * w.s, w.round ^ 1u);
                __syncwarp();
                tc_fence_after();
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {                     // 32 k: 16 columns and a scale
                uint32_t o[16];
                const uint32_t sc = ue4m3_to_bf16x2(s[h]);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = mul_bf16x2(e2m1x2_to_bf16x2(b[16 * h + i]), sc);
                tmem_st16u(tmem_w + lanes + w.s * 64u + (uint32_t)(half * 32 + h * 16), o);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready_bar[w.s]);
        }
        if (nkb > 0) {                                        // products complete in order: the last one's end is everyone's
            const int last = nkb - 1;
            ok = ok && bar_wait(err, freed + 8u * (uint32_t)(last % Q_BUFS), (uint32_t)((last / Q_BUFS) & 1));
            __syncwarp();
            tc_fence_after();
        }
    }

    // ---------------- outputs: row m of the partial sums goes to block m % splits of the cluster, which adds them in the order of the ranks
    const int slots = (rows + p.splits - 1) / p.splits;
    __syncthreads();
    if (p.splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");     // every ring is free
    const int quad = warp & 3, half = warp >> 2;
    if (warp < Q_WARPS) {
        int owner = half * COLS % p.splits, slot = half * COLS / p.splits;
#pragma unroll 1
        for (int c0 = 0; c0 < COLS; c0 += 8) {
            float v[8];
            if (nkb > 0) tmem_ld8(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * COLS + c0), v);
            else {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (half * COLS + c0 + j < rows) {
                    const uint32_t to = ring + (uint32_t)((rank * slots + slot) * kTcRows + quad * 32 + lane) * 4u;
                    uint32_t remote;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(to), "r"(owner));
                    asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(remote), "f"(v[j]) : "memory");
                }
                if (++owner == p.splits) { owner = 0; ++slot; }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == Q_WARPS + 1) tmem_dealloc(tmem, TMEM_COLS);
    if (p.splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp >= Q_WARPS) return;
    const int parts = nkb_total > 0 ? (nkb_total + p.kper - 1) / p.kper : 0;              // blocks that had any k
    const float* part = (const float*)(smem + (ring - smem_u32(smem)));
    const float alpha = p.alpha * 256.f;
    // a thread's column of the output; PAIRED: the gate's column in the partial rows, the up value `other` columns on
    constexpr bool PAIRED = FORM == Q_SWIGLU || FORM == Q_GATEUP;
    constexpr int OUT = PAIRED ? 64 : 128, OTHER = FORM == Q_SWIGLU ? 8 : 64;
    const int oc = tid & (OUT - 1), c = FORM == Q_SWIGLU ? (oc >> 3) * 16 + (oc & 7) : oc;
    const int n = FORM == Q_SWIGLU ? n0 / 2 + oc : n0 + oc, ldc = FORM == Q_SWIGLU ? p.N / 2 : p.N;
    for (int slot = tid / OUT; slot * p.splits + rank < rows; slot += Q_WARPS * 32 / OUT) {
        const int m = slot * p.splits + rank;
        float x = 0.f, u = 0.f;
        for (int s = 0; s < parts; ++s) {
            x += part[(s * slots + slot) * kTcRows + c];
            if (PAIRED) u += part[(s * slots + slot) * kTcRows + c + OTHER];
        }
        x *= alpha;
        const size_t o = (size_t)(row0 + m) * ldc + n;
        if constexpr (PAIRED) p.C[o] = f32_to_bf16_bits(round_bf16(silu_ref(round_bf16(x))) * round_bf16(u * alpha));
        else {
            if (p.bias) x = round_bf16(x) + bf16_bits_to_f32(p.bias[n]);
            p.C[o] = p.residual ? hadd_bf16_bits(x, p.residual[o]) : f32_to_bf16_bits(x);
        }
    }
}

template <int NB, int FORM>
cudaError_t n4_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int splits) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_nvf4_tc_kernel<NB, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)q_smem(NB));
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cfg->blockDim = dim3(Q_THREADS);
    cfg->dynamicSmemBytes = q_smem(NB);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
    return cudaSuccess;
}

// Blocks that the device holds at one time in clusters of s, counted as in gemm_tc.cu
int n4_held(int s) {
    static int held[9] = {};
    if (held[s] == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        int n = 0;
        cfg.gridDim = dim3(s, 64);
        if (n4_config<64, Q_PLAIN>(&cfg, at, s) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, gemm_nvf4_tc_kernel<64, Q_PLAIN>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        held[s] = n > 0 ? n * s : -1;
    }
    return held[s];
}

// Blocks per tile: a k block takes 450 cycles of the SM that converts it and 600 at least from one to the next in a block; start and
// end cost 6000 cycles, half of it hidden where two blocks share an SM, an exchange 2000 more.
int n4_splits(long long tiles, int nkb) {
    const int sms = sm_count();
    int best = 1;
    double best_cost = 1e30;
    for (int s = 1; s <= 8; ++s) {
        if (s > 1 && (nkb < 2 * s || n4_held(s) <= 0)) continue;
        const double blocks = (double)tiles * s;
        const int held = s == 1 ? 2 * sms : n4_held(s);
        const double rounds = (double)(long long)((blocks + held - 1) / held), per_sm = blocks <= sms ? 1.0 : fmin(2.0, blocks / sms);
        const double cost = rounds * ((nkb + s - 1) / s) * fmax(per_sm * 450.0, 600.0) + 6000.0 + (rounds - 1.0) * 3000.0 + (s > 1 ? 2000.0 : 0.0);
        if (cost < best_cost * 0.999) { best_cost = cost; best = s; }
    }
    return best;
}

struct N4Operands { const void* A; int a_rows; const void* Bd; const void* Bs; const void* Ud; const void* Us; int matrices; int slots; long long tiles; };

template <int NB, int FORM>
int launch_n4(N4Params p, const N4Operands& b, cudaStream_t st) {
    constexpr bool TWO = FORM == Q_GATEUP;
    const int tiles = p.N / (TWO ? 64 : kTcRows), nkb = p.K / Q_BK;
    p.splits = n4_splits(b.tiles, nkb);
    p.kper = (nkb + p.splits - 1) / p.splits;
    p.ahead = pdl_enabled();
    p.err = wait_word(kWaitNvf4);
    PGK_REQUIRE(p.err, "gemm_nvf4_tc failed: no pinned host memory");
    PGK_REQUIRE(tma_encode_fn() != nullptr, "gemm_nvf4_tc failed: the driver does not export cuTensorMapEncodeTiled");
    CUtensorMap wmap, smap, umap, tmap, amap;
    const uint32_t cols = TWO ? 64 : kTcRows;
    const uint64_t E = (uint64_t)b.matrices, N = (uint64_t)p.N, K = (uint64_t)p.K;
    PGK_REQUIRE(tma_map_bytes_3d(&wmap, b.Bd, {N, K / 2, E}, {cols, 64, 1}) && tma_map_bytes_3d(&smap, b.Bs, {N, K / 32, E}, {cols, 4, 1}) &&
                tma_map_bytes_3d(&umap, TWO ? b.Ud : b.Bd, {N, K / 2, E}, {cols, 64, 1}) && tma_map_bytes_3d(&tmap, TWO ? b.Us : b.Bs, {N, K / 32, E}, {cols, 4, 1}) &&
                tma_map_bf16_2d(&amap, b.A, K, (uint64_t)b.a_rows, K * 2, 64, TWO ? 1 : NB), "gemm_nvf4_tc failed: cuTensorMapEncodeTiled refused the operands");
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    PGK_CUDA((n4_config<NB, FORM>(&cfg, at, p.splits)));
    cfg.gridDim = dim3(p.splits, tiles, b.slots);
    cfg.stream = st;
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_waiting
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    count_launch();
    PGK_CUDA(cudaLaunchKernelEx(&cfg, gemm_nvf4_tc_kernel<NB, FORM>, wmap, smap, umap, tmap, amap, p));
    return 0;
}

template <int FORM> int launch_n4_rows(const N4Params& p, const N4Operands& b, cudaStream_t st) {
    if (p.M <= 16) return launch_n4<16, FORM>(p, b, st);
    if (p.M <= 32) return launch_n4<32, FORM>(p, b, st);
    return launch_n4<64, FORM>(p, b, st);
}

}  // namespace

bool gemm_nvf4_tc_shape_ok(int M, int K, int N, const void* A, const void* Bd, const void* Bs) {
    return M >= 1 && M <= 64 && K % Q_BK == 0 && K >= Q_BK && N % kTcRows == 0 && N / kTcRows <= Q_MAX_TILES &&
           ((uintptr_t)A % 16 == 0) && ((uintptr_t)Bd % 16 == 0) && ((uintptr_t)Bs % 16 == 0);
}

// swiglu: the columns are eight of a gate matrix and eight of an up matrix by turns, C = silu(gate) * up [M, N / 2]
int gemm_nvf4_tc(const void* A, const void* Bd, const void* Bs, void* C, int M, int K, int N, float alpha, const void* bias,
                 const void* residual, bool swiglu, cudaStream_t st) {
    PGK_REQUIRE(gemm_nvf4_tc_shape_ok(M, K, N, A, Bd, Bs),
                "gemm_nvf4_tc failed: needs 1 <= M <= 64, K %% 128 == 0, N %% 128 == 0 and 16-byte aligned pointers (M=%d K=%d N=%d)",
                M, K, N);
    N4Params p = {};
    p.C = (uint16_t*)C; p.bias = (const uint16_t*)bias; p.residual = (const uint16_t*)residual;
    p.M = M; p.K = K; p.N = N; p.alpha = alpha;
    const N4Operands b{A, M, Bd, Bs, nullptr, nullptr, 1, 1, N / kTcRows};
    return swiglu ? launch_n4_rows<Q_SWIGLU>(p, b, st) : launch_n4_rows<Q_PLAIN>(p, b, st);
}

}  // namespace pgk

using namespace pgk;

extern "C" int pgk_gemm_nvf4_bf16_tc(const void* A, const void* B_data, const void* B_scale, void* C, int M, int K, int N,
                                     float alpha, const void* bias, const void* residual, void* stream) {
    return gemm_nvf4_tc(A, B_data, B_scale, C, M, K, N, alpha, bias, residual, false, (cudaStream_t)stream);
}

extern "C" int pgk_gemm_nvf4_wait_error(int* out) {
    PGK_CUDA(cudaDeviceSynchronize());
    *out = wait_raised(kWaitNvf4);
    return 0;
}

/* The experts of `tokens` rows (pgk_moe_route_rows says who gets which): gate and up over the tokens' rows, act[r] = silu(gate) * up in the experts'
 * order, and the down product of those rows.  K, N and the matrices as in pgk_moe_grouped_gemv_nvf4.  k is cut by how many experts there are, not by
 * how many are held, so that a row's bits do not depend on the ranks. */
static int experts_ok(const char* what, int tokens, int k, int K, int N, int held, std::initializer_list<const void*> ptrs) {
    uintptr_t all = 0;
    for (const void* q : ptrs) all |= (uintptr_t)q;
    PGK_REQUIRE(tokens >= 1 && tokens <= 64 && k >= 1 && held >= 1 && K % Q_BK == 0 && K >= Q_BK && N % kTcRows == 0 && N / 64 <= 65535 && all % 16 == 0,
                "%s failed: needs 1 <= tokens <= 64, K and N in multiples of 128 and 16-byte aligned pointers (tokens=%d K=%d N=%d)", what, tokens, K, N);
    return 0;
}
// experts that have rows, as many as there may be and as there are in the mean: what the launch holds room for, what its k is cut by
static int expert_slots(int tokens, int k, int experts) { return experts < tokens * k ? experts : tokens * k; }
static long long expert_tiles(int tokens, int k, int experts, int tiles) {
    const double used = experts * (1.0 - pow(1.0 - fmin(1.0, (double)k / experts), tokens));
    return (long long)(used * tiles + 0.5);
}

extern "C" int pgk_moe_experts_gateup_nvf4(const void* x, const void* Bg_data, const void* Bg_scale, const void* Bu_data, const void* Bu_scale, void* act,
                                           const int32_t* active, const int32_t* first, const int32_t* row_token, int tokens, int k, int K, int N, int experts,
                                           int expert_offset, int num_local_experts, void* stream) {
    if (int rc = experts_ok("moe_experts_gateup_nvf4", tokens, k, K, N, num_local_experts, {x, Bg_data, Bg_scale, Bu_data, Bu_scale})) return rc;
    N4Params p = {};
    p.C = (uint16_t*)act; p.M = tokens; p.K = K; p.N = N; p.alpha = 1.f;
    p.active = active; p.first = first; p.token = row_token; p.offset = expert_offset;
    const N4Operands b{x, tokens, Bg_data, Bg_scale, Bu_data, Bu_scale, num_local_experts, expert_slots(tokens, k, num_local_experts), expert_tiles(tokens, k, experts, N / 64)};
    return launch_n4_rows<Q_GATEUP>(p, b, (cudaStream_t)stream);
}
extern "C" int pgk_moe_experts_down_nvf4(const void* act, const void* B_data, const void* B_scale, void* C, const int32_t* active, const int32_t* first,
                                         int tokens, int k, int K, int N, int experts, int expert_offset, int num_local_experts, void* stream) {
    if (int rc = experts_ok("moe_experts_down_nvf4", tokens, k, K, N, num_local_experts, {act, B_data, B_scale})) return rc;
    N4Params p = {};
    p.C = (uint16_t*)C; p.M = tokens; p.K = K; p.N = N; p.alpha = 1.f;
    p.active = active; p.first = first; p.offset = expert_offset;
    const N4Operands b{act, tokens * k, B_data, B_scale, nullptr, nullptr, num_local_experts, expert_slots(tokens, k, num_local_experts), expert_tiles(tokens, k, experts, N / kTcRows)};
    return launch_n4_rows<Q_DOWN>(p, b, (cudaStream_t)stream);
}
