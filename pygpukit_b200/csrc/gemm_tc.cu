// gemm_tc.cu -- W8A16 GEMM for a few dozen rows on the 5th-gen tensor cores (tcgen05 + TMEM + TMA).
//
//   C[M,N] = A[M,K] . dequant(B[N,K])^T     B = FP8-E4M3 codes [N,K], S = bf16 [N/128, K/128]
//
// replaces gemv_fp8_warp_reduce_vec4_batched_kernel (fp8_opt.cuh:220-295, re-reads the weights M times) and
// the M >= 16 tensor-core path of pygpukit_w8a16_gemm_sm120 (w8a16_gemm.cu:104-339: dequantise to BF16 in
// shared memory, mma.sync m16n8k16, unpipelined).
//
// What bounds it: the weights' way from HBM, and close behind it what an SM does per 128 x 128 block of them: the conversion of
// 16384 codes and the traffic through its shared memory.  What follows from that:
//   * the GEMM is computed transposed, D^T[n, m] = W[n, :] . A[m, :]: a block owns 128 weight rows (MMA M, a TMEM lane per row), the
//     batch is the MMA's N (16 / 32 / 64 columns), so that every weight is read once, marked first to leave L2;
//   * TMA brings codes and activations as they are (128-byte swizzle) into a ring; eight warps turn the codes into BF16 exactly and
//     store them to TENSOR MEMORY, from where the MMA takes its A operand: through shared memory the BF16 form would be written
//     and read once more, 128 KB per block of weights instead of 64, which alone is 1000 cycles against 680 for the HBM stream;
//   * the block scale multiplies the partial sums of its 128 products in float32 (two accumulators by turns): products are exact and
//     the activations need no second term that holds their product with the scale (128 unscaled products must stay within float32:
//     activations up to 5e33);
//   * the same eight warps add the partial sums of the block before while the tensor cores multiply; MMAs and copies have a warp each;
//   * a stage holds a block's codes and rows together (rings of their own left too few slots for the rows: 65 -> 72 us);
//   * two blocks per SM (256 TMEM columns, 100 KB each) hide each other's start and end; K is cut over a cluster that pushes
//     its partial rows to their owners' shared memory and adds them in the order of the ranks: no work memory.
// Measured on B200 (us, cp.async and conversion through shared memory -> here), M = 5 / 64: 14336 x 4096 35 / 43 -> 20.7 / 24.5,
// 4096 x 4096 16.5 / 26.8 -> 10.5 / 13.9, 1024 x 4096 10.9 / 21.3 -> 8.3 / 10.4, 14336 x 14336 103 / 134 -> 55 / 65 (3.7 / 3.2 TB/s).
// Gate, up and their activation in one launch (PAIR; 64 rows, 14336 x 4096 and back): two products, silu, product and the down projection 85.2 us,
// with the pair in one launch 57.5, the same bits.
#include "common.cuh"
#include "gemv_common.cuh"
#include "tc_common.cuh"
#include "tma.cuh"
#include "../../include/pgk_b200.h"

namespace pgk {

constexpr int kTcBK = 128;        // k block = FP8 scale block
constexpr int kTcMaxKb = 256;     // k blocks (K <= 32768)
constexpr int kTcMaxTiles = 8192;

namespace {

constexpr int F_WARPS = 8;                        // conversion, partial sums, output; one more for the copies, one for the MMAs
constexpr int F_THREADS = (F_WARPS + 2) * 32;
constexpr uint32_t F_W_BYTES = kTcRows * kTcBK;   // codes of a stage
__host__ __device__ constexpr int f_stages(int nb) { return nb <= 16 ? 5 : (nb <= 32 ? 4 : 3); }
__host__ __device__ constexpr uint32_t f_stage_bytes(int nb) { return F_W_BYTES + (uint32_t)nb * kTcBK * 2; }
__host__ __device__ constexpr size_t f_smem(int nb) { return (size_t)f_stages(nb) * f_stage_bytes(nb) + 1024; }

struct F8TcParams {
    const uint16_t* S; const uint16_t* S1; uint16_t* C;          // scales (of gate and up), output
    const uint16_t* bias; const uint16_t* residual;
    int M, K, N, splits, kper;
    int ahead;                                    // scales and the first codes are read before the kernel before has finished
    int* err;                                     // raised when a bounded wait runs out
};

// PAIR: a tile is 64 rows of a gate and 64 of an up matrix, by turns of 16, so that a lane's partner is 16 lanes on; C = silu(gate) * up
template <int NB, bool PAIR>
__global__ void __launch_bounds__(F_THREADS, 2)
gemm_fp8_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap umap, const __grid_constant__ CUtensorMap amap,
                   const __grid_constant__ F8TcParams p) {
    constexpr int STAGES = f_stages(NB), COLS = NB / 2;          // columns of a warp
    constexpr uint32_t STAGE = f_stage_bytes(NB), TMEM_COLS = 2 * NB + 128 <= 256 ? 256 : 512;
    static_assert(TMEM_COLS == 256, "two blocks per SM");
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], w_bar[2], d_bar[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ float sc_s[(PAIR ? 2 : 1) * kTcMaxKb];
    constexpr int OUT = PAIR ? kTcRows / 2 : kTcRows;            // columns of C per tile
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t ring = (smem_u32(smem) + 1023u) & ~1023u, full = smem_u32(full_bar), empty = smem_u32(empty_bar);
    const uint32_t wb = smem_u32(w_bar), db = smem_u32(d_bar);
    int* const err = p.err;
    const int rank = blockIdx.x, n0 = blockIdx.y * OUT, nkb_total = p.K / kTcBK;
    const int kb0 = rank * p.kper, nkb = max(0, min(nkb_total, kb0 + p.kper) - kb0);

    if (!p.ahead) griddep_wait();
    // the block's scales are weights: staged before the dependency wait
    const size_t scales = (size_t)(blockIdx.y >> (PAIR ? 1 : 0)) * nkb_total + kb0;
    for (int i = tid; i < nkb; i += F_THREADS) {
        sc_s[i] = bf16_bits_to_f32(p.S[scales + i]);
        if (PAIR) sc_s[kTcMaxKb + i] = bf16_bits_to_f32(p.S1[scales + i]);
    }
    if (warp == F_WARPS + 1) tmem_alloc(&tmem_base_s, TMEM_COLS);
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&w_bar[b], F_WARPS); mbar_init(&d_bar[b], 1); }
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" :: "l"(&wmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&amap) : "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s, tmem_w = tmem + 2 * NB;   // accumulators, then two k blocks of weights (64 columns each)
    float acc[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = 0.f;

    if (warp == F_WARPS) {
        // ---------------- copies; the first weights leave before the dependency wait
        if (elect_one()) {
            const uint64_t once = l2_evict_first();
            auto weights = [&](int it, uint32_t s) {
                mbar_expect_tx(full + 8u * s, STAGE);
                if constexpr (PAIR) {
#pragma unroll 1
                    for (int q = 0; q < 4; ++q) {
                        tma_load_2d_hint(ring + s * STAGE + (uint32_t)q * 4096u, &wmap, (kb0 + it) * kTcBK, n0 + q * 16, full + 8u * s, once);
                        tma_load_2d_hint(ring + s * STAGE + (uint32_t)q * 4096u + 2048u, &umap, (kb0 + it) * kTcBK, n0 + q * 16, full + 8u * s, once);
                    }
                } else
                    tma_load_2d_hint(ring + s * STAGE, &wmap, (kb0 + it) * kTcBK, n0, full + 8u * s, once);
            };
            auto rows = [&](int it, uint32_t s) {
                const uint32_t at = ring + s * STAGE + F_W_BYTES;
                tma_load_2d(at, &amap, (kb0 + it) * kTcBK, 0, full + 8u * s);
                tma_load_2d(at + NB * 128u, &amap, (kb0 + it) * kTcBK + 64, 0, full + 8u * s);
            };
            const int first = min(nkb, STAGES);
            for (int it = 0; it < first; ++it) weights(it, (uint32_t)it);
            griddep_wait();
            griddep_launch();
            for (int it = 0; it < first; ++it) rows(it, (uint32_t)it);
            RingPos r;
            r.round = 1;
            int it = first;
            for (; it < nkb; ++it, r.next(STAGES)) {
                if (!bar_wait(err, empty + 8u * r.s, r.round ^ 1u)) break;
                weights(it, r.s);
                rows(it, r.s);
            }
            for (int j = max(0, it - STAGES); j < it; ++j)    // whoever gave up: do not leave with copies in flight
                bar_wait(err, full + 8u * (uint32_t)(j % STAGES), (uint32_t)((j / STAGES) & 1));
        } else {
            griddep_wait();
            griddep_launch();
        }
        __syncwarp();
    } else if (warp == F_WARPS + 1) {
        // ---------------- MMAs
        griddep_wait();
        griddep_launch();
        if (elect_one()) {
            constexpr uint32_t idesc = umma_idesc_bf16(NB);
            RingPos r;
            for (int it = 0; it < nkb; ++it, r.next(STAGES)) {
                const uint32_t b = (uint32_t)it & 1u;
                if (!bar_wait(err, full + 8u * r.s, r.round) || !bar_wait(err, wb + 8u * b, (uint32_t)(it >> 1) & 1u)) break;
                tc_fence_after();
                const uint32_t a_s = ring + r.s * STAGE + F_W_BYTES;
#pragma unroll
                for (int ks = 0; ks < kTcBK / 16; ++ks)
                    umma_bf16_ta(tmem + b * NB, tmem_w + b * 64u + (uint32_t)ks * 8u, desc_sw128(a_s + (uint32_t)(ks >> 2) * (NB * 128u)) + (uint64_t)((ks & 3) * 2),
                                 idesc, ks > 0 ? 1u : 0u);
                umma_commit(&d_bar[b]);
                umma_commit(&empty_bar[r.s]);
            }
        }
        __syncwarp();
    } else {
        // ---------------- codes -> TMEM, and the partial sums of the block before
        griddep_wait();
        griddep_launch();
        const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        bool ok = true;
        auto add = [&](int it) {                              // acc += scale x the products of block it
            const uint32_t b = (uint32_t)it & 1u;
            ok = ok && bar_wait(err, db + 8u * b, (uint32_t)(it >> 1) & 1u);
            __syncwarp();
            tc_fence_after();
            const float sc = sc_s[(PAIR && (lane & 16) ? kTcMaxKb : 0) + it];
            const uint32_t at = tmem + lanes + b * NB + (uint32_t)half * COLS;
            if constexpr (COLS == 8) {
                float v[8];
                tmem_ld8(at, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = fmaf(sc, v[j], acc[j]);
            } else {
#pragma unroll
                for (int c = 0; c < COLS; c += 16) {
                    float v[16];
                    tmem_ld16(at + c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(sc, v[j], acc[c + j]);
                }
            }
            tc_fence_before();
        };
        RingPos r;
        for (int it = 0; it < nkb; ++it, r.next(STAGES)) {
            const uint32_t b = (uint32_t)it & 1u, src = ring + r.s * STAGE + (uint32_t)row * 128u;
            ok = ok && bar_wait(err, full + 8u * r.s, r.round);
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) {                     // 32 codes: 16 columns
                uint32_t o[16];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint4 w;
                    const uint32_t at = src + (uint32_t)(((half * 4 + h * 2 + i) ^ (row & 7)) << 4);
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(at) : "memory");
                    e4m3x4_to_bf16x4(w.x, o[8 * i], o[8 * i + 1]);
                    e4m3x4_to_bf16x4(w.y, o[8 * i + 2], o[8 * i + 3]);
                    e4m3x4_to_bf16x4(w.z, o[8 * i + 4], o[8 * i + 5]);
                    e4m3x4_to_bf16x4(w.w, o[8 * i + 6], o[8 * i + 7]);
                }
                tmem_st16u(tmem_w + lanes + b * 64u + (uint32_t)(half * 32 + h * 16), o);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_bar[b]);
            if (it > 0) add(it - 1);                          // ... before block it + 1 takes its place
        }
        if (nkb > 0) add(nkb - 1);
    }

    // ---------------- outputs
    const int rows_here = min(NB, p.M);
    auto store_pair = [&](float g, float u, int m, int n) {
        p.C[(size_t)m * p.N + n] = f32_to_bf16_bits(round_bf16(silu_ref(round_bf16(g))) * round_bf16(u));
    };
    const bool up = PAIR && (lane & 16);
    auto store = [&](float x, int m, int n) {
        const size_t o = (size_t)m * p.N + n;
        if (p.bias) x = round_bf16(x) + bf16_bits_to_f32(p.bias[n]);
        p.C[o] = p.residual ? hadd_bf16_bits(x, p.residual[o]) : f32_to_bf16_bits(x);
    };
    const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
    if (p.splits == 1) {
        if (warp < F_WARPS) {
            if constexpr (PAIR) {
#pragma unroll
                for (int j = 0; j < COLS; j += 2) {           // a lane takes its partner's value of every second row for its own of the others
                    const float got = __shfl_xor_sync(0xffffffffu, up ? acc[j] : acc[j + 1], 16);
                    const int m = half * COLS + j + (up ? 1 : 0);
                    if (m < rows_here) store_pair(up ? got : acc[j], up ? acc[j + 1] : got, m, n0 + quad * 16 + (lane & 15));
                }
            } else {
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    if (half * COLS + j < rows_here) store(acc[j], half * COLS + j, n0 + row);
            }
        }
    } else {                                                  // column m belongs to block m % splits
        const int slots = (rows_here + p.splits - 1) / p.splits;
        __syncthreads();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");     // every ring is free
        if (warp < F_WARPS) {
            int owner = half * COLS % p.splits, slot = half * COLS / p.splits;
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                if (half * COLS + j < rows_here) {
                    const uint32_t to = ring + (uint32_t)((rank * slots + slot) * kTcRows + row) * 4u;
                    uint32_t remote;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(to), "r"(owner));
                    asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(remote), "f"(acc[j]) : "memory");
                }
                if (++owner == p.splits) { owner = 0; ++slot; }
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (warp < F_WARPS) {
            const int parts = (nkb_total + p.kper - 1) / p.kper;              // blocks that had any k
            const float* part = (const float*)(smem + (ring - smem_u32(smem)));
            for (int slot = half; slot * p.splits + rank < rows_here; slot += 2) {
                float x = 0.f;
                for (int s = 0; s < parts; ++s) x += part[(s * slots + slot) * kTcRows + row];
                if constexpr (PAIR) {
                    const float u = __shfl_xor_sync(0xffffffffu, x, 16);
                    if (!up) store_pair(x, u, slot * p.splits + rank, n0 + quad * 16 + lane);
                } else
                    store(x, slot * p.splits + rank, n0 + row);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == F_WARPS + 1) tmem_dealloc(tmem, TMEM_COLS);
}

template <int NB, bool PAIR>
cudaError_t f8tc_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int splits) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_fp8_tc_kernel<NB, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f_smem(NB));
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cfg->blockDim = dim3(F_THREADS);
    cfg->dynamicSmemBytes = f_smem(NB);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
    return cudaSuccess;
}

// Blocks that the device holds at one time in clusters of s, one per SM, as cudaOccupancyMaxActiveClusters counts them (for kernels that allocate
// tensor memory; two per SM run together all the same).
int f8tc_held(int s) {
    static int held[9] = {};
    if (held[s] == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        int n = 0;
        cfg.gridDim = dim3(s, 64);
        if (f8tc_config<64, false>(&cfg, at, s) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, gemm_fp8_tc_kernel<64, false>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        held[s] = n > 0 ? n * s : -1;
    }
    return held[s];
}

// Blocks per tile, by what a launch takes (us, a fit of 22 matrices of 1 ... 200 MB, 6 ... 64 rows, 1 ... 8 blocks per tile, within 10 % but for 2 %
// of them): 5 ... 6.5 for its start and end, 1.5 ... 2.4 for an exchange and 2.5 ... 5 for every further wave; per k block 0.41 ... 0.47 (16 ... 64 rows) while an SM has one block, 0.64 ... 0.78
// once some have two, a tenth more when all do.  The device holds two blocks per SM, in clusters some less for each of its processing
// clusters; what is left over follows in a wave of its own.  64 rows, the k blocks of HBM traffic alone as the line before -> this one: 14336 x 14336
// 62 -> 52, 10752 x 11776 47 -> 32, 11776 x 4352 23 -> 19, 14336 x 4096 21.5 -> 19, 5120 x 10240 25 -> 20, 4096 x 6144 16 -> 14.
double f8tc_time(int nb, int tiles, int nkb, int s) {
    const int sms = sm_count(), c = nb <= 16 ? 0 : (nb <= 32 ? 1 : 2);
    const double one[3] = {0.41, 0.425, 0.465}, some[3] = {0.64, 0.68, 0.775}, all[3] = {0.72, 0.74, 0.84}, ends[3] = {4.9, 5.4, 6.3}, again[3] = {2.5, 3.5, 5.0};
    const int per = (nkb + s - 1) / s, blocks = tiles * s, held = s == 1 ? 2 * sms : 2 * sms - 5 * s, alone = f8tc_held(s);
    auto wave = [&](int n) { return per * (n <= alone ? one[c] : some[c] + (all[c] - some[c]) * fmax(0, n - sms) / sms); };
    const int waves = blocks / held, rest = blocks - waves * held;
    const double full = waves * wave(held) + (rest > 0 ? wave(rest) : 0.0);
    return ends[c] + (s > 1 ? 1.2 + 0.15 * s : 0.0) + full + again[c] * (waves - (rest > 0 ? 0 : 1));
}
int f8tc_splits(int nb, int tiles, int nkb) {
    int best = 1;
    for (int s = 2; s <= 8; ++s)
        if (nkb >= 2 * s && f8tc_held(s) > 0 && f8tc_time(nb, tiles, nkb, s) < f8tc_time(nb, tiles, nkb, best) * 0.999) best = s;
    return best;
}

template <int NB, bool PAIR>
int launch_f8tc(F8TcParams p, const void* A, const void* B, const void* B1, cudaStream_t st) {
    const int tiles = p.N / (PAIR ? kTcRows / 2 : kTcRows), nkb = p.K / kTcBK;
    p.splits = f8tc_splits(NB, tiles, nkb);
    p.kper = (nkb + p.splits - 1) / p.splits;
    p.ahead = pdl_enabled();
    p.err = wait_word(kWaitFp8);
    PGK_REQUIRE(p.err, "gemm_fp8_tc failed: no pinned host memory");
    PGK_REQUIRE(tma_encode_fn() != nullptr, "gemm_fp8_tc failed: the driver does not export cuTensorMapEncodeTiled");
    CUtensorMap wmap, umap, amap;
    const uint32_t box = PAIR ? 16 : kTcRows;
    PGK_REQUIRE(tma_map_bytes_2d(&wmap, B, (uint64_t)p.K, (uint64_t)p.N, kTcBK, box) && tma_map_bytes_2d(&umap, B1, (uint64_t)p.K, (uint64_t)p.N, kTcBK, box) &&
                tma_map_bf16_2d(&amap, A, (uint64_t)p.K, (uint64_t)p.M, (uint64_t)p.K * 2, 64, NB), "gemm_fp8_tc failed: cuTensorMapEncodeTiled refused the operands");
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    PGK_CUDA((f8tc_config<NB, PAIR>(&cfg, at, p.splits)));
    cfg.gridDim = dim3(p.splits, tiles);
    cfg.stream = st;
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_waiting
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    count_launch();
    PGK_CUDA(cudaLaunchKernelEx(&cfg, gemm_fp8_tc_kernel<NB, PAIR>, wmap, umap, amap, p));
    return 0;
}

}  // namespace

bool gemm_fp8_tc_shape_ok(int M, int K, int N, const void* A, const void* B);

// Smallest batch sent to the tensor cores.  The copies zero-fill rows M..NB-1, so any M >= 1 works.  Up to four rows share one pass of the
// CUDA-core GEMV and get the bits of one row alone, which batches of that size are promised; from three rows on this kernel would be
// faster (us, GEMV / here: 4096 x 4096 M = 2 10.5 / 10.5, M = 3 14.1 / 10.5, M = 4 16.3 / 10.5; 14336 x 4096 20.8 / 20.7, 24.9 / 20.7, 30.4 /
// 20.7), and from five on the GEMV takes a second pass.  PGK_TC_MIN_M overrides (A/B timing).
int gemm_fp8_tc_min_m() {
    static const int v = [] { const char* e = getenv("PGK_TC_MIN_M"); int m = e ? atoi(e) : 5; return m < 1 ? 1 : m; }();
    return v;
}

// the dispatcher's test (batch >= crossover); the kernel itself takes any 1 <= M <= 64
bool gemm_fp8_tc_eligible(int M, int K, int N, const void* A, const void* B) {
    return M >= gemm_fp8_tc_min_m() && gemm_fp8_tc_shape_ok(M, K, N, A, B);
}

bool gemm_fp8_tc_shape_ok(int M, int K, int N, const void* A, const void* B) {
    return M >= 1 && M <= 64 && K / kTcBK <= kTcMaxKb && K % kTcBK == 0 && N % kTcRows == 0 && N / kTcRows <= kTcMaxTiles &&
           ((uintptr_t)A % 16 == 0) && ((uintptr_t)B % 16 == 0);
}

int gemm_fp8_tc(const void* A, const void* B_nk, const void* S, void* C, int M, int K, int N, const void* bias,
                const void* residual, cudaStream_t st) {
    PGK_REQUIRE(gemm_fp8_tc_shape_ok(M, K, N, A, B_nk),
                "gemm_fp8_tc failed: needs 1 <= M <= 64, K %% 128 == 0, N %% 128 == 0 and 16-byte aligned pointers "
                "(M=%d K=%d N=%d)", M, K, N);
    F8TcParams p = {};
    p.S = (const uint16_t*)S; p.C = (uint16_t*)C;
    p.bias = (const uint16_t*)bias; p.residual = (const uint16_t*)residual;
    p.M = M; p.K = K; p.N = N;
    if (M <= 16) return launch_f8tc<16, false>(p, A, B_nk, B_nk, st);
    if (M <= 32) return launch_f8tc<32, false>(p, A, B_nk, B_nk, st);
    return launch_f8tc<64, false>(p, A, B_nk, B_nk, st);
}

// silu(A . Wg^T) * (A . Wu^T) with the roundings of the two products, silu and the product (for shapes that gemm_fp8_tc takes)
int gemm_fp8_tc_pair(const void* A, const void* Wg, const void* Sg, const void* Wu, const void* Su, void* C, int M, int K, int N, cudaStream_t st) {
    F8TcParams p = {};
    p.S = (const uint16_t*)Sg; p.S1 = (const uint16_t*)Su; p.C = (uint16_t*)C;
    p.M = M; p.K = K; p.N = N;
    if (M <= 16) return launch_f8tc<16, true>(p, A, Wg, Wu, st);
    if (M <= 32) return launch_f8tc<32, true>(p, A, Wg, Wu, st);
    return launch_f8tc<64, true>(p, A, Wg, Wu, st);
}

}  // namespace pgk

extern "C" int pgk_gemm_fp8_bf16_tc(const void* A, const void* B_nk, const void* S, void* C, int M, int K, int N,
                                    const void* bias, const void* residual, void* stream) {
    bool clean = true;
    if (int rc = pgk::fp8_codes_clean(B_nk, (size_t)N * K, (cudaStream_t)stream, &clean)) return rc;
    PGK_REQUIRE(clean, "gemm_fp8_bf16_tc failed: the weights hold E4M3 codes 0x7F/0xFF (+-480 in the reference's tables, "
                "NaN for the tensor-core conversion); use pgk_gemv_fp8_bf16, which serves them exactly");
    return pgk::gemm_fp8_tc(A, B_nk, S, C, M, K, N, bias, residual, (cudaStream_t)stream);
}

extern "C" int pgk_gemm_fp8_wait_error(int* out) {
    PGK_CUDA(cudaDeviceSynchronize());
    *out = pgk::wait_raised(pgk::kWaitFp8);
    if (*out == 0) *out = pgk::wait_raised(pgk::kWaitFp8Rows);
    return 0;
}
