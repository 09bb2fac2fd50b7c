// gemm_tc_rows.cu -- W8A16 GEMM over many rows (prompts) on the 5th-gen tensor cores (tcgen05 + TMEM + TMA).
//
//   C[M,N] = A[M,K] . dequant(B[N,K])^T                    B = FP8-E4M3 codes [N,K], S = bf16 [N/128, K/128], M > 64
//   C[M,N] = bf16(bf16(silu(bf16(A.Wg^T))) * bf16(A.Wu^T))  the same for a gate and an up matrix (PAIR)
//
// The mathematics, the operands' way and the partial sums are those of gemm_tc.cu: codes are turned into BF16 exactly and stored to
// tensor memory, D^T[n, m] = W[n, :] . A[m, :], and the block scale multiplies the float32 sums of its 128 products.
//
// What bounds it: the MMAs.  A product of 128 x 128 x 128 is eight of them, 77 cycles each when nothing else runs and 112 beside the traffic
// of the other warps through tensor memory and shared memory, so 1800 cycles per block of 128 weight rows, 128 k and 256 activation rows;
// and what a thread does between them.  What follows from that:
//   * a tile is 128 weight rows by up to 256 activation rows, so that each block of codes is converted once per 256 rows; its sums stay
//     in registers (128 a thread);
//   * products of 128 columns go round three accumulators (3 x 128 TMEM columns beside two blocks of weights, 2 x 64: all 512), so that
//     the MMAs never wait for the addition of what they have just finished;
//   * conversion (500 cycles a block), sums (2 x 400) and MMAs have warps of their own, in step by one barrier per product; one pair of
//     warpgroups that converted and added by turns took 2400 cycles a block;
//   * codes and activations have a ring and a warp each: codes come four blocks ahead (HBM), activations two and a half (L2);
//   * a block per SM runs through its tiles; the next tile's first block is converted and multiplied before the last one's outputs are
//     written.  Tiles of the same weights follow one another, so that they meet in L2;
//   * few tiles: K is cut over a cluster that pushes its partial rows to their owners' shared memory, added in the order of the ranks;
//   * PAIR: gate and up rows alternate by 16 in a tile, a lane's partner is 16 lanes on.
// Measured on B200 (us; slabs of 64 rows through gemm_tc.cu -> here): 512 rows of 6144 x 4096 99 -> 39, 4096 x 4096 90 -> 29, 4096 x 14336
// 191 -> 61 (0.99 PFLOP/s), gate and up of 14336 x 4096 with their activation 470 -> 144; 128 rows 25 -> 21, 23 -> 17, 48 -> 29, 118 -> 57.
#include "common.cuh"
#include "gemv_common.cuh"
#include "tc_common.cuh"
#include "tma.cuh"
#include "../../include/pgk_b200.h"

namespace pgk {

namespace {

constexpr int P_BK = 128;                          // k block = FP8 scale block
// Warpgroups: two for sums and outputs, two for the conversion, one for copies of codes, copies of activations and the MMAs of two
// products.  Registers: 256 x 184 + 256 x 40 + 128 x 32 = 640 x 96, the block's at launch (f8rows_config asks for it: with fewer, the
// warps that want more would wait without end).
constexpr int P_SUMS = 8, P_CONV = 8;
constexpr int P_THREADS = (P_SUMS + P_CONV + 4) * 32;
constexpr int P_SUMS_REGS = 184, P_CONV_REGS = 40, P_REST_REGS = 32, P_REGS = P_SUMS * 32 * P_SUMS_REGS + P_CONV * 32 * P_CONV_REGS + 4 * 32 * P_REST_REGS;
constexpr int P_CODES_WARP = P_SUMS + P_CONV, P_ROWS_WARP = P_CODES_WARP + 1, P_MMA_WARP = P_CODES_WARP + 2;
constexpr int P_HALF = 128;                        // activation rows of one product
constexpr int P_CODES = 4, P_ROWS = 5, P_ACCS = 3;
constexpr uint32_t P_CODE_BYTES = kTcRows * P_BK, P_ROW_BYTES = P_HALF * P_BK * 2;
constexpr size_t P_SMEM = P_CODES * P_CODE_BYTES + P_ROWS * P_ROW_BYTES + 1024;
constexpr uint32_t P_TMEM_W = P_ACCS * P_HALF;     // first TMEM column of the weights

struct F8RowsParams {
    const uint16_t* S0; const uint16_t* S1; uint16_t* C;
    const uint16_t* bias; const uint16_t* residual;
    int M, K, N;                                   // N: columns of C
    int item0, items, m_tiles, mrows;              // tiles [item0, items), and of how many rows
    int splits, kper;
    int ahead;                                     // the first codes are read before the kernel before has finished
    int* err;
};

// two float32 products and sums, each rounded once, by one instruction
__device__ __forceinline__ void fma2(float& a0, float& a1, float s, float v0, float v1) {
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %2};\n\tmov.b64 c, {%3, %4};\n\tfma.rn.f32x2 a, b, c, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+f"(a0), "+f"(a1) : "f"(s), "f"(v0), "f"(v1));
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// eight neighbours of a thread's sums, the b-th of 16
__device__ __forceinline__ void take8(const float (&acc)[2][64], int b, float (&x)[8]) {
    switch (b) {
#define PGK_TAKE(k) case k: for (int e = 0; e < 8; ++e) x[e] = acc[k >> 3][(k & 7) * 8 + e]; break;
        PGK_TAKE(0) PGK_TAKE(1) PGK_TAKE(2) PGK_TAKE(3) PGK_TAKE(4) PGK_TAKE(5) PGK_TAKE(6) PGK_TAKE(7)
        PGK_TAKE(8) PGK_TAKE(9) PGK_TAKE(10) PGK_TAKE(11) PGK_TAKE(12) PGK_TAKE(13) PGK_TAKE(14)
#undef PGK_TAKE
        default: for (int e = 0; e < 8; ++e) x[e] = acc[1][56 + e];
    }
}
// A wait of a whole warp, each lane for a barrier of its own choice.  (For one elected lane a wait for a barrier that is long complete
// costs 270 cycles here, for the warp 130 ... 230: the loop of the MMAs went from 1500 to 1300 cycles.)
__device__ __forceinline__ bool bars_wait(int* err, uint32_t bar, uint32_t parity) {
    const bool ok = bar_wait(err, bar, parity);
    return __all_sync(0xffffffffu, ok);
}
template <int N> __device__ __forceinline__ void registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(N)); }
template <int N> __device__ __forceinline__ void registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(N)); }

template <bool PAIR>
__global__ void __launch_bounds__(P_THREADS, 1)
gemm_fp8_rows_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap umap, const __grid_constant__ CUtensorMap amap,
                     const __grid_constant__ F8RowsParams p) {
    constexpr int OUT = PAIR ? kTcRows / 2 : kTcRows;            // columns of C per tile
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t cfull_bar[P_CODES], cempty_bar[P_CODES], ready_bar[P_ROWS], aempty_bar[P_ROWS], wempty_bar[2], dfull_bar[P_ACCS];
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t codes = (smem_u32(smem) + 1023u) & ~1023u, acts = codes + P_CODES * P_CODE_BYTES;
    int* const err = p.err;
    const int rank = blockIdx.x, nkb_total = p.K / P_BK;
    const int kb0 = rank * p.kper, nkb = max(0, min(nkb_total, kb0 + p.kper) - kb0);
    const int first = p.item0 + blockIdx.y, step = gridDim.y;

    if (warp == P_MMA_WARP) tmem_alloc(&tmem_base_s, 512);
    if (tid == 0) {
        for (int s = 0; s < P_CODES; ++s) { mbar_init(&cfull_bar[s], 1); mbar_init(&cempty_bar[s], P_CONV); }
        for (int s = 0; s < P_ROWS; ++s) { mbar_init(&ready_bar[s], 1 + P_CONV + P_SUMS); mbar_init(&aempty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) mbar_init(&wempty_bar[b], 2);
        for (int b = 0; b < P_ACCS; ++b) mbar_init(&dfull_bar[b], 1);
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" :: "l"(&wmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&amap) : "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s, tmem_w = tmem + P_TMEM_W;
    // Product g (counted over blocks and tiles) uses activation slot g % 5 and accumulator g % 3; ready_bar of its slot counts the copy, the
    // warps that converted its weights and those that have read product g - 3.  That makes one wait of it, and bounds who can be
    // ahead: whoever has passed ready(g - 2) knows that g - 5, the slot's last user, is read, so no wait takes an older phase for its own.
    auto rows_of = [&](int item) { return min(p.mrows, p.M - (item % p.m_tiles) * p.mrows); };
    if (warp >= P_CODES_WARP) {
    registers_down<P_REST_REGS>();
    if (warp == P_CODES_WARP) {
        // ---------------- codes; weights, so the first ones leave before the dependency wait
        if (elect_one()) {
            const uint64_t once = l2_evict_first();
            RingPos c;
            int blk = 0;
            bool ok = true, waited = !p.ahead;
            if (waited) { griddep_wait(); griddep_launch(); }
            for (int item = first; ok && item < p.items; item += step) {
                const int n0 = item / p.m_tiles * OUT;
                for (int it = 0; it < nkb; ++it, ++blk, c.next(P_CODES)) {
                    if (blk == P_CODES && !waited) { griddep_wait(); griddep_launch(); waited = true; }
                    const uint32_t bar = smem_u32(cfull_bar) + 8u * c.s, at = codes + c.s * P_CODE_BYTES;
                    ok = bar_wait(err, smem_u32(cempty_bar) + 8u * c.s, c.round ^ 1u);
                    if (!ok) break;
                    mbar_expect_tx(bar, P_CODE_BYTES);
                    const int k = (kb0 + it) * P_BK;
                    if (PAIR) {
#pragma unroll 1
                        for (int q = 0; q < 4; ++q) {
                            tma_load_2d_hint(at + (uint32_t)q * 4096u, &wmap, k, n0 + q * 16, bar, once);
                            tma_load_2d_hint(at + (uint32_t)q * 4096u + 2048u, &umap, k, n0 + q * 16, bar, once);
                        }
                    } else
                        tma_load_2d_hint(at, &wmap, k, n0, bar, once);
                }
            }
            if (!waited) { griddep_wait(); griddep_launch(); }
            for (int j = max(0, blk - P_CODES); j < blk; ++j)     // whoever gave up: do not leave with copies in flight
                bar_wait(err, smem_u32(cfull_bar) + 8u * (uint32_t)(j % P_CODES), (uint32_t)((j / P_CODES) & 1));
        } else {
            griddep_wait();
            griddep_launch();
        }
        __syncwarp();
    } else if (warp == P_ROWS_WARP) {
        // ---------------- activations
        griddep_wait();
        griddep_launch();
        if (elect_one()) {
            RingPos a;
            int n = 0;
            bool ok = true;
            for (int item = first; ok && item < p.items; item += step) {
                const int m0 = item % p.m_tiles * p.mrows, halves = rows_of(item) > P_HALF ? 2 : 1;
                for (int it = 0; ok && it < nkb; ++it)
                    for (int h = 0; h < halves; ++h, ++n, a.next(P_ROWS)) {
                        const uint32_t bar = smem_u32(ready_bar) + 8u * a.s, at = acts + a.s * P_ROW_BYTES;
                        ok = bar_wait(err, smem_u32(aempty_bar) + 8u * a.s, a.round ^ 1u);
                        if (!ok) break;
                        mbar_expect_tx(bar, P_ROW_BYTES);
                        tma_load_2d(at, &amap, (kb0 + it) * P_BK, m0 + h * P_HALF, bar);
                        tma_load_2d(at + P_ROW_BYTES / 2, &amap, (kb0 + it) * P_BK + 64, m0 + h * P_HALF, bar);
                    }
            }
            for (int j = max(0, n - P_ROWS); j < n; ++j)
                bar_wait(err, smem_u32(ready_bar) + 8u * (uint32_t)(j % P_ROWS), (uint32_t)((j / P_ROWS) & 1));
        }
        __syncwarp();
    } else {
        // ---------------- MMAs, a warp for each product of a block: what one takes beside its MMAs -- wait, commits, the loop -- is 700 cycles
        griddep_wait();
        griddep_launch();
        const int h = warp - P_MMA_WARP;
        uint32_t group = 0, blk = 0;
        bool ok = true;
        for (int item = first; ok && item < p.items; item += step) {
            const int rows = rows_of(item), halves = rows > P_HALF ? 2 : 1;
            const uint32_t idesc = umma_idesc_bf16((min(P_HALF, rows - h * P_HALF) + 15) & ~15);              // the rows that are there
            for (int it = 0; it < nkb; ++it, ++blk, group += halves) {
                const bool idle = h >= halves;            // keeps step with the first warp
                const uint32_t b = blk & 1u, g = idle ? group : group + h, sl = g % P_ROWS, d = g % P_ACCS;
                ok = bars_wait(err, smem_u32(ready_bar) + 8u * sl, (g / P_ROWS) & 1u);
                if (!ok) break;
                if (idle) {
                    if (lane == 0) mbar_arrive(&wempty_bar[b]);
                    __syncwarp();
                    continue;
                }
                if (elect_one()) {
                    tc_fence_after();
                    const uint32_t at = acts + sl * P_ROW_BYTES;
#pragma unroll
                    for (int ks = 0; ks < P_BK / 16; ++ks)
                        umma_bf16_ta(tmem + d * P_HALF, tmem_w + b * 64u + (uint32_t)ks * 8u,
                                     desc_sw128(at + (uint32_t)(ks >> 2) * (P_ROW_BYTES / 2)) + (uint64_t)((ks & 3) * 2), idesc, ks > 0 ? 1u : 0u);
                    umma_commit(&dfull_bar[d]);
                    umma_commit(&aempty_bar[sl]);
                    umma_commit(&wempty_bar[b]);
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
    } else if (warp >= P_SUMS) {
        // ---------------- codes -> TMEM
        registers_down<P_CONV_REGS>();
        griddep_wait();
        griddep_launch();
        const int row = (warp & 3) * 32 + lane, kh = (warp - P_SUMS) >> 2;
        const uint32_t to = tmem_w + ((uint32_t)((warp & 3) * 32) << 16);
        bool ok = true;
        RingPos c;
        uint32_t blk = 0, group = 0;
        for (int item = first; item < p.items; item += step) {
            const int halves = rows_of(item) > P_HALF ? 2 : 1;
            for (int it = 0; it < nkb; ++it, ++blk, group += halves, c.next(P_CODES)) {
                const uint32_t b = blk & 1u, src = codes + c.s * P_CODE_BYTES + (uint32_t)row * 128u;
                ok = ok && bars_wait(err, lane & 1 ? smem_u32(cfull_bar) + 8u * c.s : smem_u32(wempty_bar) + 8u * b, lane & 1 ? c.round : ((blk >> 1) & 1u) ^ 1u);
                tc_fence_after();
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {                     // 32 codes: 16 columns; a short loop, five kinds of warps share the instruction caches
                    uint32_t o[16];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        uint4 w;
                        const uint32_t at = src + (uint32_t)(((kh * 4 + h * 2 + i) ^ (row & 7)) << 4);
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(at) : "memory");
                        e4m3x4_to_bf16x4(w.x, o[8 * i], o[8 * i + 1]);
                        e4m3x4_to_bf16x4(w.y, o[8 * i + 2], o[8 * i + 3]);
                        e4m3x4_to_bf16x4(w.z, o[8 * i + 4], o[8 * i + 5]);
                        e4m3x4_to_bf16x4(w.w, o[8 * i + 6], o[8 * i + 7]);
                    }
                    tmem_st16u(to + b * 64u + (uint32_t)(kh * 32 + h * 16), o);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                // lane 0: the codes are read; 1, 2: the block's products have their weights
                if (lane <= halves) mbar_arrive(lane == 0 ? &cempty_bar[c.s] : &ready_bar[(group + lane - 1) % P_ROWS]);
            }
        }
    } else {
        // ---------------- sums and outputs
        registers_up<P_SUMS_REGS>();
        griddep_wait();
        griddep_launch();
        const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        const bool up = PAIR && (lane & 16);
        float acc[2][64];                                         // a row of weights by 64 rows of each product
        bool ok = true;
        uint32_t group = 0;
        if (lane < P_ACCS) mbar_arrive(&ready_bar[lane]);
        for (int item = first; item < p.items; item += step) {
            const int rows = rows_of(item), halves = rows > P_HALF ? 2 : 1, n_tile = item / p.m_tiles, m0 = (item - n_tile * p.m_tiles) * p.mrows;
            const size_t scales = (size_t)(n_tile >> (PAIR ? 1 : 0)) * nkb_total + kb0;
            uint32_t s0 = 0, s1 = 0;                              // the scales of 32 blocks, one a lane
#pragma unroll
            for (int j = 0; j < 64; ++j) acc[0][j] = acc[1][j] = 0.f;
#pragma unroll 1
            for (int it = 0; it < nkb; ++it) {
                if ((it & 31) == 0) {
                    s0 = p.S0[scales + min(it + lane, nkb - 1)];
                    if (PAIR) s1 = p.S1[scales + min(it + lane, nkb - 1)];
                }
                uint32_t bits = __shfl_sync(0xffffffffu, s0, it & 31);
                if (PAIR) {
                    const uint32_t other = __shfl_sync(0xffffffffu, s1, it & 31);
                    bits = up ? other : bits;
                }
                const float sc = bf16_bits_to_f32(bits);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (h >= halves) break;
                    const uint32_t d = group % P_ACCS, at = tmem + lanes + d * P_HALF + (uint32_t)half * 64u;
                    ok = ok && bars_wait(err, smem_u32(dfull_bar) + 8u * d, (group / P_ACCS) & 1u);
                    tc_fence_after();
                    float v[2][16];
                    tmem_ld16_async(at, v[0]);
#pragma unroll
                    for (int j = 0; j < 64; j += 16) {            // the next columns are on their way while these are added
                        float (&x)[16] = v[(j >> 4) & 1];
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        tmem_pass(x);
                        if (j + 16 < 64) tmem_ld16_async(at + (uint32_t)j + 16u, v[((j >> 4) & 1) ^ 1]);
#pragma unroll
                        for (int e = 0; e < 16; e += 2) fma2(acc[h][j + e], acc[h][j + e + 1], sc, x[e], x[e + 1]);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ready_bar[(group + P_ACCS) % P_ROWS]);
                    ++group;
                }
            }
            const int turns = ((rows + 15) / 16 + p.splits - 1) / p.splits;
            // records of 16 rows in their owner's shared memory: [from][turn][4 rows][weight row][4]
            auto place = [&](int from, int turn) { return codes + (uint32_t)(((from * turns + turn) * 4 * kTcRows + row) * 16); };
            if (p.splits > 1) {                                   // one tile per cluster: 16 rows at a time go to block (rows / 16) % splits
                cluster_sync();                                   // every ring is free
                const uint32_t inv_splits = (65536u + p.splits - 1) / p.splits;       // exact for batch < 16
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const int j = (b & 3) * 16, batch = (b >> 2) * 8 + half * 4 + (b & 3), turn = (int)((uint32_t)batch * inv_splits >> 16), owner = batch - turn * p.splits;
                    if (batch * 16 >= rows || owner == rank) continue;
                    uint32_t to;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(place(rank, turn)), "r"(owner));
#pragma unroll
                    for (int e = 0; e < 16; e += 4)
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(to + (uint32_t)(e * kTcRows * 4)), "f"(acc[b >> 2][j + e]),
                                     "f"(acc[b >> 2][j + e + 1]), "f"(acc[b >> 2][j + e + 2]), "f"(acc[b >> 2][j + e + 3]) : "memory");
                }
                __syncwarp();
                cluster_sync();
            }
            // ---- outputs, 8 rows at a time.  A loop: as straight-line code, run once a tile, this took 30000 cycles, nearly all for its fetch.
            const int parts = (nkb_total + p.kper - 1) / p.kper;  // blocks that had any k
            const int n = n_tile * OUT + (PAIR ? quad * 16 + (lane & 15) : row);
            const float bias = p.bias ? bf16_bits_to_f32(p.bias[n]) : 0.f;
            uint16_t* const c = p.C + (size_t)m0 * p.N + n;
            uint16_t next[8] = {};
            auto fetch = [&](int m) {                             // C may be the residual: loaded a turn ahead of its store
                if (PAIR || !p.residual) return;
                const uint16_t* r = p.residual + (size_t)(m0 + m) * p.N + n;
#pragma unroll
                for (int e = 0; e < 8; ++e) next[e] = m + e < rows ? r[(size_t)e * p.N] : (uint16_t)0;
            };
            // 16 rows are two turns: batch = rank + turn x splits, of which this warp has every second four
            int turn = 0, batch = rank, sub = 0;
            auto skip = [&]() {
                while (batch * 16 < rows && ((batch >> 2) & 1) != half) { batch += p.splits; ++turn; }
            };
            skip();
            fetch(batch * 16);
#pragma unroll 1
            while (batch * 16 < rows) {
                const int m = batch * 16 + sub * 8, at_turn = turn, at_sub = sub, b = (batch >> 3) * 8 + (batch & 3) * 2 + sub;
                uint16_t res[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) res[e] = next[e];
                if (++sub == 2) { sub = 0; batch += p.splits; ++turn; skip(); }
                fetch(batch * 16 + sub * 8);
                float x[8];
                take8(acc, b, x);
                if (p.splits > 1) {
                    float t[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                    for (int s = 0; s < parts; ++s) {
                        float v[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] = x[e];
                        if (s != rank) {
#pragma unroll
                            for (int e = 0; e < 8; e += 4)
                                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[e]), "=f"(v[e + 1]), "=f"(v[e + 2]), "=f"(v[e + 3])
                                             : "r"(place(s, at_turn) + (uint32_t)((at_sub * 8 + e) * kTcRows * 4)) : "memory");
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) t[e] += v[e];
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = t[e];
                }
                uint16_t* const to = c + (size_t)m * p.N;
                if (PAIR) {
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {              // a lane takes its partner's value of every second row for its own of the others
                        const float got = __shfl_xor_sync(0xffffffffu, up ? x[e] : x[e + 1], 16);
                        const float g = round_bf16(up ? got : x[e]), u = round_bf16(up ? x[e + 1] : got);
                        const int r = e + (up ? 1 : 0);
                        if (m + r < rows) to[(size_t)r * p.N] = f32_to_bf16_bits(round_bf16(silu_ref(g)) * u);
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float v = p.bias ? round_bf16(x[e]) + bias : x[e];
                        const uint16_t bits = p.residual ? hadd_bf16_bits(v, res[e]) : f32_to_bf16_bits(v);
                        if (m + e < rows) to[(size_t)e * p.N] = bits;
                    }
                }
            }
            if (p.splits > 1) break;
        }
    }
    if (p.splits > 1 && warp >= P_SUMS) {
        __syncwarp();
        cluster_sync();
        cluster_sync();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == P_MMA_WARP) tmem_dealloc(tmem, 512);
}

template <bool PAIR>
cudaError_t f8rows_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int splits) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_fp8_rows_kernel<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P_SMEM);
        if (e != cudaSuccess) return e;
        cudaFuncAttributes fa;
        const cudaError_t f = cudaFuncGetAttributes(&fa, gemm_fp8_rows_kernel<PAIR>);
        if (f != cudaSuccess) return f;
        if (fa.numRegs * P_THREADS < P_REGS) return cudaErrorInvalidConfiguration;
        configured = true;
    }
    cfg->blockDim = dim3(P_THREADS);
    cfg->dynamicSmemBytes = P_SMEM;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
    return cudaSuccess;
}

// blocks that run together in clusters of s (clusters do not cross the device's processing clusters)
int f8rows_held(int s) {
    static int held[9] = {};
    if (held[s] == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        int n = 0;
        cfg.gridDim = dim3(s, 64);
        if (f8rows_config<false>(&cfg, at, s) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, gemm_fp8_rows_kernel<false>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        held[s] = n > 0 ? n * s : -1;
    }
    return held[s];
}

struct F8RowsPlan { int mrows, splits, tail, tail_splits; };

// What a launch costs in cycles: a block of 128 k takes 1000 with up to 128 rows, 1750 with 256; a block's start 5000, of which a run
// of tiles pays it once and 7000 for each tile's outputs; an exchange and the outputs that are left then 5000.
double f8rows_cost(int tiles, int nkb, int mrows, int s) {
    const int held = s == 1 ? sm_count() : f8rows_held(s);
    const double rounds = (double)((tiles * s + held - 1) / held), kb = (nkb + s - 1) / s, block = mrows > 128 ? 1750.0 : 1000.0;
    return s == 1 ? rounds * (kb * block + 7000.0) + 5000.0 : rounds * (kb * block + 5000.0 + 5000.0);
}
int f8rows_splits(int tiles, int nkb, int mrows, double* cost) {
    int best = 1;
    *cost = f8rows_cost(tiles, nkb, mrows, 1);
    for (int s = 2; s <= 8 && nkb >= 2 * s; ++s) {
        if (f8rows_held(s) <= 0) continue;
        const double c = f8rows_cost(tiles, nkb, mrows, s);
        if (c < *cost * 0.999) { *cost = c; best = s; }
    }
    return best;
}
// Rows of a tile, blocks that share its k, and whether the tiles beyond whole rounds get a launch of their own in which they share it (512
// rows of a gate and an up matrix of 14336 x 4096: 448 tiles on 148 SMs, 158 us in four rounds, 144 with the last four by themselves).
F8RowsPlan f8rows_plan(int n_tiles, int M, int nkb) {
    F8RowsPlan best = {256, 1, 0, 1};
    double best_cost = 1e30;
    for (int mrows = 128; mrows <= 256; mrows += 128) {
        if (mrows == 256 && M <= 128) break;
        const int tiles = n_tiles * ((M + mrows - 1) / mrows), sms = sm_count(), over = tiles > sms ? tiles % sms : 0;
        double cost;
        const int s = f8rows_splits(tiles, nkb, mrows, &cost);
        if (cost < best_cost * 0.999) { best_cost = cost; best = {mrows, s, 0, 1}; }
        if (over > 0) {
            double tail;
            const int ts = f8rows_splits(over, nkb, mrows, &tail);
            cost = f8rows_cost(tiles - over, nkb, mrows, 1) + tail + 6000.0;
            if (cost < best_cost * 0.999) { best_cost = cost; best = {mrows, 1, over, ts}; }
        }
    }
    return best;
}

template <bool PAIR>
int launch_f8rows(F8RowsParams p, const void* A, const void* B0, const void* B1, cudaStream_t st) {
    const int nkb = p.K / P_BK, n_tiles = p.N / (PAIR ? kTcRows / 2 : kTcRows);
    const F8RowsPlan plan = f8rows_plan(n_tiles, p.M, nkb);
    p.mrows = plan.mrows;
    p.m_tiles = (p.M + p.mrows - 1) / p.mrows;
    p.ahead = pdl_enabled();
    p.err = wait_word(kWaitFp8Rows);
    PGK_REQUIRE(p.err, "gemm_fp8 failed: no pinned host memory");
    PGK_REQUIRE(tma_encode_fn() != nullptr, "gemm_fp8 failed: the driver does not export cuTensorMapEncodeTiled");
    CUtensorMap wmap, umap, amap;
    const uint32_t box = PAIR ? 16 : kTcRows;
    PGK_REQUIRE(tma_map_bytes_2d(&wmap, B0, (uint64_t)p.K, (uint64_t)p.N, P_BK, box) && tma_map_bytes_2d(&umap, B1, (uint64_t)p.K, (uint64_t)p.N, P_BK, box) &&
                tma_map_bf16_2d(&amap, A, (uint64_t)p.K, (uint64_t)p.M, (uint64_t)p.K * 2, 64, P_HALF), "gemm_fp8 failed: cuTensorMapEncodeTiled refused the operands");
    auto run = [&](int item0, int items, int splits) {
        F8RowsParams q = p;
        q.item0 = item0;
        q.items = items;
        q.splits = splits;
        q.kper = (nkb + splits - 1) / splits;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        PGK_CUDA(f8rows_config<PAIR>(&cfg, at, splits));
        cfg.gridDim = dim3(splits, splits > 1 ? items - item0 : min(items - item0, sm_count()));
        cfg.stream = st;
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_waiting
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
        count_launch();
        PGK_CUDA(cudaLaunchKernelEx(&cfg, gemm_fp8_rows_kernel<PAIR>, wmap, umap, amap, q));
        return 0;
    };
    const int items = n_tiles * p.m_tiles;
    if (int rc = run(0, items - plan.tail, plan.splits)) return rc;
    return plan.tail ? run(items - plan.tail, items, plan.tail_splits) : 0;
}

}  // namespace

bool gemm_fp8_rows_ok(int M, int K, int N, const void* A, const void* B0, const void* B1) {
    return M > 64 && M <= 65536 && K % P_BK == 0 && N % kTcRows == 0 && (long long)(N / 64) * ((M + 127) / 128) <= 65535 && (uintptr_t)A % 16 == 0 &&
           (uintptr_t)B0 % 16 == 0 && (uintptr_t)B1 % 16 == 0 && tma_encode_fn() != nullptr;
}

int gemm_fp8_rows(const void* A, const void* B0, const void* S0, const void* B1, const void* S1, void* C, int M, int K, int N, const void* bias,
                  const void* residual, cudaStream_t st) {
    F8RowsParams p = {};
    p.S0 = (const uint16_t*)S0; p.S1 = (const uint16_t*)S1; p.C = (uint16_t*)C;
    p.bias = (const uint16_t*)bias; p.residual = (const uint16_t*)residual;
    p.M = M; p.K = K; p.N = N;
    return B1 ? launch_f8rows<true>(p, A, B0, B1, st) : launch_f8rows<false>(p, A, B0, B0, st);
}

}  // namespace pgk
