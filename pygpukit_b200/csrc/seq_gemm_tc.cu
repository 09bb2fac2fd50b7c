// seq_gemm_tc.cu -- the many-row products of the token-major models on tcgen05: C[m, n] = sum_k bf16(A[row(m), k]) W[g][n, k]
// with float32 activations, bfloat16 weights, float32 accumulators in TMEM and every epilogue of seq_gemm.cu.
//
// What bounds it: at prompt sizes the tensor pipe and, just behind it, the operand stream from L2; at a few dozen rows the
// weights' way from HBM.  What follows from that:
//   * the activations are rounded to bfloat16 ONCE (rows_to_bf16_kernel, 6 bytes per element, L2-resident for the product)
//     instead of in every tile: the float32 tile would be twice the operand bytes of the bfloat16 one, per tile that reads it;
//   * the tile is computed transposed, 128 weight rows (TMEM lanes) x up to 256 activation rows (accumulator columns), so
//     that a warp's lanes hold neighbouring output columns of one row -- stores are whole 128-byte lines without a pass
//     through shared memory -- and so that the tile's height follows the rows there are (16 ... 256): experts with 13 rows and
//     prompts with 2000 run the same code;
//   * TMA brings both operands (128-byte swizzle) into a ring of stages, one thread issues the MMAs, two accumulators in TMEM
//     let eight epilogue warps drain a tile while the next one is multiplied, and one block per SM walks the tiles;
//   * few tiles: a cluster of 2 ... 8 blocks shares a tile, each with a part of k, and the partial sums meet in shared memory
//     (distributed loads, added in the order of the ranks), so that all SMs pull on the weights.  How k is cut follows from the number
//     of rows, too: the bits of a row are those of the tiles only where it is not cut, and may differ between a whole prompt and its parts;
//   * up to 32 rows (decoding), and blocks of them while a product is small: a kernel of its own (gemm_few_tc_kernel), one launch without work memory.
// Measured on B200, 2000 x 9216 x 2048: 573 us on the 64 x 64 tiles of seq_gemm.cu (132 TFLOP/s), 6 + 59 us here (1.27 PFLOP/s in
// the product); 8000 gathered rows over 16 experts, 4096 x 2048 and 2048 x 2048: 1510 -> 262 us for both.
#include "seq_gemm.cuh"
#include "tc_common.cuh"
#include "tma.cuh"
#include "../../include/pgk_b200.h"

namespace pgk {

namespace {

constexpr int TBK = 64;                    // k per stage: one 128-byte swizzle row of bfloat16
constexpr int TC_THREADS = 320;            // TMA warp, MMA warp, eight epilogue warps
constexpr int TC_ROWS_MAX = 256;           // activation rows per tile = accumulator columns
constexpr int TC_MAX_GROUPS = 512;
constexpr uint32_t TC_W_BYTES = kTcRows * TBK * 2;
constexpr uint32_t TC_RING_BYTES = 200 * 1024;
constexpr int TC_MAX_STAGES = 10;
constexpr int TC_DIRECT_ROWS = 32;         // rows whose activations the kernel rounds itself, in blocks of 16 or 32
__host__ __device__ constexpr int few_stages(int r) { return r == 16 ? 5 : 4; }
__host__ __device__ constexpr uint32_t few_stage_bytes(int r) { return TC_W_BYTES + (uint32_t)r * TBK * 2; }
__host__ __device__ constexpr uint32_t few_smem(int r) { return few_stages(r) * few_stage_bytes(r) + 1024; }      // with the partial rows: two blocks per SM

struct TcArgs {
    GemmArgs g;
    int epi;
    int bn;              // rows of a tile at most (multiple of 16)
    int abox;            // rows per activation copy
    int mt, nt, nkb;     // row tiles (no groups), column tiles, k blocks
    int batch;           // products, or row groups
    int stages;
    uint32_t stage_bytes;
    int splits;          // blocks per tile (cluster size)
    int* err;            // raised when a bounded wait runs out (never, unless a copy or a product is lost)
};

// ---------------------------------------------------------------- activations -> bfloat16 rows [r][batch][K] (rows that are bfloat16 already stay where they are)
// Memory: reads 4 and writes 2 bytes per element; 16-byte accesses both ways.  2000 x 2048: 4.0 us warm, 6.0 us from HBM.
__global__ void __launch_bounds__(256) rows_to_bf16_kernel(GemmArgs a, uint16_t* out, int batch, int kpr, bool vec) {
    griddep_wait();
    griddep_launch();
    const int r = blockIdx.x;
    if (a.group_off && r >= a.group_off[batch]) return;
    const size_t src = (size_t)(a.a_rows ? a.a_rows[r] : r) * a.lda;
    const int nb = a.group_off ? 1 : batch, chunks = nb * kpr;                 // chunks of eight elements
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < chunks; c += gridDim.y * blockDim.x) {
        const int b = nb == 1 ? 0 : c / kpr, k = (c - b * kpr) * 8;
        const size_t p = src + (size_t)b * a.a_z + k;
        float v[8];
        if (vec && k + 8 <= a.ka) {
            *(float4*)&v[0] = a_at4(a, p);
            *(float4*)&v[4] = a_at4(a, p + 4);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = k + j < a.ka ? a_at(a, p + j) : 0.f;
        }
        uint4 o = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        *(uint4*)(out + ((size_t)r * nb + b) * a.K + k) = o;
    }
}

// ---------------------------------------------------------------- matrices whose rows start anywhere -> rows of a multiple of 16 bytes, zeros behind them
// Memory: reads and writes 2 bytes per element.  A row starts on a word or half a word behind one: four or five words per eight elements, single elements
// at the matrices' two ends and behind a row's.  5664 x 3574 (40 MB): 15 us.
__global__ void __launch_bounds__(256) pad_weights_kernel(const uint16_t* W, uint16_t* out, int K, int N, int kpr, long long stride, long long total) {
    griddep_wait();
    griddep_launch();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const long long row = i / kpr;
    const int k = (int)(i - row * kpr) * 8, m = (int)(row / N), n = (int)(row - (long long)m * N);
    const uint16_t* p = W + m * stride + (long long)n * K + k;
    const bool half = ((uintptr_t)p & 2) != 0, ends = (n == 0 && k == 0) || (n == N - 1 && k + 9 > K);
    uint32_t o[4];
    if (k + 8 <= K && !ends) {
        const uint32_t* q = (const uint32_t*)(p - (half ? 1 : 0));
        uint32_t w[5];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = q[j];
        w[4] = half ? q[4] : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = half ? __funnelshift_r(w[j], w[j + 1], 16) : w[j];
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t lo = k + 2 * j < K ? p[2 * j] : 0u, hi = k + 2 * j + 1 < K ? p[2 * j + 1] : 0u;
            o[j] = lo | hi << 16;
        }
    }
    *(uint4*)(out + i * 8) = make_uint4(o[0], o[1], o[2], o[3]);
}

// ---------------------------------------------------------------- small pieces
__device__ __forceinline__ void cluster_arrive_wait() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t local_addr, uint32_t rank) {
    uint32_t ra;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(local_addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ra) : "memory");
    return v;
}

struct Tile { int z, n0, m0, rows; };

// tile t of the launch: row tiles fastest, so that the blocks running at one time read few weight tiles
__device__ __forceinline__ Tile tile_at(const TcArgs& p, const int* pre, int t) {
    Tile w;
    if (!p.g.group_off) {
        const int mi = t % p.mt, r = t / p.mt;
        w.z = r / p.nt;
        w.n0 = (r - w.z * p.nt) * kTcRows;
        w.m0 = mi * p.bn;
        w.rows = min(p.bn, p.g.M - w.m0);
        return w;
    }
    int lo = 0, hi = p.batch;                    // pre[lo] <= t < pre[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[mid] <= t) lo = mid; else hi = mid;
    }
    const int begin = p.g.group_off[lo], R = p.g.group_off[lo + 1] - begin;
    const int mte = (R + p.bn - 1) / p.bn, h = ((R + mte - 1) / mte + 15) & ~15, loc = t - pre[lo], mi = loc % mte;
    w.z = lo;
    w.n0 = loc / mte * kTcRows;
    w.m0 = begin + mi * h;
    w.rows = min(h, R - mi * h);
    return w;
}

// ---------------------------------------------------------------- epilogue: R rows of one output column per lane
template <int R, typename F>
__device__ __forceinline__ void store_rows(const GemmArgs& a, const float (&v)[R], int row, int left, int col, F f) {
    if (col >= a.N) return;
    const size_t at = (size_t)row * a.ldc + col;
#pragma unroll
    for (int j = 0; j < R; ++j)
        if (j < left) put(a, at + (size_t)j * a.ldc, f(v[j], j));
}
// pairs (2j, 2j + 1) of columns sit in neighbouring lanes: the even lane finishes the even rows, the odd lane the odd ones
template <int R, typename F>
__device__ __forceinline__ void store_pairs(const GemmArgs& a, const float (&v)[R], int row, int left, int col, int lane, F f) {
    const bool odd = lane & 1;
    if constexpr (R == 1) {
        const float second = __shfl_xor_sync(0xffffffffu, v[0], 1);
        if (!odd && col + 1 < a.N && left > 0) put(a, (size_t)row * a.ldc + (col >> 1), f(v[0], second));
        return;
    } else {
#pragma unroll
        for (int j = 0; j < R; j += 2) {
            const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
            const float first = odd ? got : v[j], second = odd ? v[j + 1] : got;
            const int jj = odd ? j + 1 : j;
            if ((col | 1) < a.N && jj < left) put(a, (size_t)(row + jj) * a.ldc + (col >> 1), f(first, second));
        }
    }
}

template <int R>
__device__ __forceinline__ void epilogue_rows(const GemmArgs& a, int epi, const float (&v)[R], int row, int left, int col, int lane) {
    switch (epi) {
        case 1: store_pairs<R>(a, v, row, left, col, lane, [](float g, float u) { return silu_f(g) * u; }); return;
        case 7: store_pairs<R>(a, v, row, left, col, lane, [](float g, float u) { return gelu_tanh_f(g) * u; }); return;
        case 3:          // scale = alpha, cap = limit
            store_pairs<R>(a, v, row, left, col, lane, [&](float c0, float c1) {
                const float g = fminf(c0, a.cap), u = fminf(fmaxf(c1, -a.cap), a.cap);
                return g / (1.f + expf(-a.scale * g)) * (u + 1.f);
            });
            return;
        case 2:
            store_rows<R>(a, v, row, left, col, [&](float c, int) {
                c *= a.scale;
                return a.cap > 0.f ? a.cap * tanhf(c / a.cap) : c;
            });
            return;
        case 4: {
            if (col >= a.N) return;
            const float s = a.colv[col];
            float old[R];
            const float* p = a.C + (size_t)row * a.ldc + col;
#pragma unroll
            for (int j = 0; j < R; ++j) old[j] = j < left ? p[(size_t)j * a.ldc] : 0.f;
            store_rows<R>(a, v, row, left, col, [&](float c, int j) { return fmaf(s, c, old[j]); });
            return;
        }
        case 5:
            store_rows<R>(a, v, row, left, col, [&](float c, int j) { return gelu_tanh_f(c) * aux_at(a, row + j, col); });
            return;
        case 6:
            store_rows<R>(a, v, row, left, col, [](float c, int) { c = fmaxf(c, 0.f); return c * c; });
            return;
        case 8: store_rows<R>(a, v, row, left, col, [](float c, int) { return gelu_erf_f(c); }); return;
        case 9: store_rows<R>(a, v, row, left, col, [](float c, int) { return gelu_tanh_f(c); }); return;
        case 10:         // the gate's columns are as far apart as the output's: `aux` moves with C from batch to batch
            store_rows<R>(a, v, row, left, col, [&](float c, int j) {
                return c * (1.f / (1.f + expf(-((const float*)a.aux)[(size_t)(row + j) * a.aux_ld + a.aux_off + col])));
            });
            return;
        default: store_rows<R>(a, v, row, left, col, [](float c, int) { return c; });
    }
}

// ---------------------------------------------------------------- the product
template <bool R16>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_rows_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap amap, const __grid_constant__ TcArgs p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full_bar[TC_MAX_STAGES], empty_bar[TC_MAX_STAGES], done_bar[2], drained_bar[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int pre[TC_MAX_GROUPS + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ring = (smem_u32(smem) + 1023u) & ~1023u, full = smem_u32(full_bar), empty = smem_u32(empty_bar);

    if (warp == 1) tmem_alloc(&tmem_base_s, 512);
    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&done_bar[b], 1); mbar_init(&drained_bar[b], 8); }
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" :: "l"(&wmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&amap) : "memory");
    }
    griddep_wait();
    if (p.g.group_off && warp == 2) {            // tiles before every group
        int run = 0;
        for (int e0 = 0; e0 < p.batch; e0 += 32) {
            const int e = e0 + lane;
            int n = 0;
            if (e < p.batch) n = (p.g.group_off[e + 1] - p.g.group_off[e] + p.bn - 1) / p.bn * p.nt;
            int inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += up;
            }
            if (e < p.batch) pre[e] = run + inc - n;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) pre[p.batch] = run;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_launch();                            // tensor memory is held
    const uint32_t tmem = tmem_base_s;
    const int total = p.g.group_off ? pre[p.batch] : p.batch * p.mt * p.nt;
    const int rank = p.splits > 1 ? (int)cluster_rank() : 0;
    const int first = (int)blockIdx.x / p.splits, step = (int)gridDim.x / p.splits;
    const int per = (p.nkb + p.splits - 1) / p.splits, kb0 = rank * per, kb1 = min(p.nkb, kb0 + per);

    if (warp == 0) {
        if (elect_one()) {
            RingPos r;
            int i = 0;                            // stages filled so far
            bool ok = true;
            for (int t = first; ok && t < total; t += step) {
                const Tile w = tile_at(p, pre, t);
                const int boxes = (w.rows + p.abox - 1) / p.abox, az = p.g.group_off ? 0 : w.z;
                const uint32_t bytes = TC_W_BYTES + (uint32_t)(boxes * p.abox) * (TBK * 2);
                for (int kb = kb0; kb < kb1; ++kb, ++i, r.next(p.stages)) {
                    const uint32_t fb = full + 8u * r.s, dst = ring + r.s * p.stage_bytes;
                    if (!bar_wait(p.err, empty + 8u * r.s, r.round ^ 1u)) { ok = false; break; }
                    mbar_expect_tx(fb, bytes);
                    tma_load_3d(dst, &wmap, kb * TBK, w.n0, w.z, fb);
                    for (int b = 0; b < boxes; ++b)
                        tma_load_3d(dst + TC_W_BYTES + (uint32_t)(b * p.abox) * (TBK * 2), &amap, kb * TBK, az, w.m0 + b * p.abox, fb);
                }
            }
            for (int j = max(0, i - p.stages); j < i; ++j)        // whoever gave up: do not leave with copies in flight
                bar_wait(p.err, smem_u32(&full_bar[j % p.stages]), (uint32_t)((j / p.stages) & 1));
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            RingPos r;
            int u = 0;
            bool ok = true;
            for (int t = first; ok && t < total; t += step, ++u) {
                const Tile w = tile_at(p, pre, t);
                const uint32_t idesc = umma_idesc_bf16((w.rows + 15) & ~15), acc = tmem + (uint32_t)(u & 1) * TC_ROWS_MAX;
                if (!bar_wait(p.err, smem_u32(&drained_bar[u & 1]), (uint32_t)(((u >> 1) & 1) ^ 1))) break;
                tc_fence_after();
                for (int kb = kb0; kb < kb1; ++kb, r.next(p.stages)) {
                    if (!bar_wait(p.err, full + 8u * r.s, r.round)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t addr = ring + r.s * p.stage_bytes;
                    const uint64_t dw = desc_sw128(addr), da = desc_sw128(addr + TC_W_BYTES);
#pragma unroll
                    for (int ks = 0; ks < TBK / 16; ++ks)         // 32 bytes of k per MMA: +2 in the descriptor's 16-byte units
                        umma_bf16(acc, dw + (uint64_t)(ks * 2), da + (uint64_t)(ks * 2), idesc, (kb > kb0 || ks > 0) ? 1u : 0u);
                    umma_commit(&empty_bar[r.s]);
                }
                if (ok) umma_commit(&done_bar[u & 1]);
            }
        }
        __syncwarp();
    } else {
        const int ew = warp - 2, quad = warp & 3, half = ew >> 2;
        int u = 0;
        for (int t = first; t < total; t += step, ++u) {
            const Tile w = tile_at(p, pre, t);
            if (!__all_sync(0xffffffffu, bar_wait(p.err, smem_u32(&done_bar[u & 1]), (uint32_t)((u >> 1) & 1)))) break;
            tc_fence_after();
            const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(u & 1) * TC_ROWS_MAX;
            const int col = w.n0 + quad * 32 + lane;
            if (p.splits == 1) {
                GemmArgs a = p.g;
                if (!R16) a.c16 = 0;
                if (!a.group_off) {
                    move_c(a, w.z * a.c_z);
                    if (p.epi == 10) a.aux = (const float*)a.aux + (size_t)w.z * a.c_z;
                }
                for (int c = half * 16; c < w.rows; c += 32) {
                    float v[16];
                    tmem_ld16(acc + c, v);
                    epilogue_rows<16>(a, p.epi, v, w.m0 + c, w.rows - c, col, lane);
                    __syncwarp();
                }
            } else {                              // this block's share of k: row c of the partial tile, 128 columns
                for (int c = half * 16; c < w.rows; c += 32) {
                    float v[16];
                    tmem_ld16(acc + c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        asm volatile("st.shared.f32 [%0], %1;" :: "r"(ring + (uint32_t)((c + j) * kTcRows + quad * 32 + lane) * 4u), "f"(v[j]) : "memory");
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&drained_bar[u & 1]);
        }
    }
    if (p.splits > 1) {
        __syncthreads();
        cluster_arrive_wait();
        if (warp >= 2 && first < total) {         // one tile per cluster: block `rank` finishes every splits-th group of 16 rows
            const Tile w = tile_at(p, pre, first);
            const int ew = warp - 2, quad = warp & 3, half = ew >> 2, col = w.n0 + quad * 32 + lane;
            GemmArgs a = p.g;
            if (!R16) a.c16 = 0;
            if (!a.group_off) {
                move_c(a, w.z * a.c_z);
                if (p.epi == 10) a.aux = (const float*)a.aux + (size_t)w.z * a.c_z;
            }
            const int parts = (p.nkb + per - 1) / per;            // blocks that had any k
            for (int c = (rank * 2 + half) * 16; c < w.rows; c += p.splits * 32) {
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.f;
                for (int s = 0; s < parts; ++s)
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] += ld_cluster(ring + (uint32_t)((c + j) * kTcRows + quad * 32 + lane) * 4u, (uint32_t)s);
                epilogue_rows<16>(a, p.epi, v, w.m0 + c, w.rows - c, col, lane);
            }
        }
        __syncwarp();                             // lanes beyond N left the epilogue early; the barrier's arrival takes whole warps
        cluster_arrive_wait();                    // the others may still read this block's partial sums
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------- up to 32 rows, and blocks of 32
// One tile of `th` weight rows (or a share of its k) per block, two blocks per SM: the next block's start -- barriers, TMEM,
// the first copies' way from HBM, 5000 cycles -- hides behind the other's stream.  No work memory: the epilogue warps, idle until
// the tile is done, round the float32 rows into the stages, eight k blocks per fence (a fence also waits for loads in flight).
// A cluster that shares a tile along k pushes its partial rows to their owners' shared memory, one barrier, and every block
// finishes its rows.  Measured at 8 rows, against a warp per column pair (gemm_few_rows_kernel): see few_tc_pays.  R: rows of the accumulator, 16 or 32;
// more rows than that are blocks of 32 side by side (see few_rows_pay).
// The weights are marked first to leave L2: at the default they push out what the small kernels in between keep reading (norm
// weights, page tables, rows), which then cost 4 us more each: a decode step of 0.5 GB of weights 598 -> 536 us.  Rows that name the same
// matrix read it at nearly the same time and lose nothing (64 rows of 4096 x 2048, all of one matrix 72.1 us, 73.6 without the mark).
struct FewArgs {
    GemmArgs g;
    int epi, th, nkb, kper, splits, rpb, avec;
    int blocks;          // blocks of R rows that share a matrix, one behind the other in grid.z
    int* err;
};

// ODD: bfloat16 rows, or rows that end within the matrix's (K is a multiple of eight, ka any number)
template <bool ODD>
__device__ __forceinline__ float4 direct_load(const GemmArgs& a, const float* row, int k, bool vec) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!ODD) {
        if (row && k < a.K) {
            if (vec) v = *(const float4*)(row + k);
            else { v.x = row[k]; v.y = row[k + 1]; v.z = row[k + 2]; v.w = row[k + 3]; }
        }
        return v;
    }
    if (!row || k >= a.ka) return v;
    const uint16_t* h = (const uint16_t*)row + k;
    if (vec && k + 4 <= a.ka) {
        if (!a.a16) return *(const float4*)(row + k);
        const uint2 u = *(const uint2*)h;
        return make_float4(bf16lo(u.x), bf16hi(u.x), bf16lo(u.y), bf16hi(u.y));
    }
    float e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = k + j < a.ka ? (a.a16 ? bf16_bits_to_f32(h[j]) : row[k + j]) : 0.f;
    return make_float4(e[0], e[1], e[2], e[3]);
}

template <int R, bool ODD>
__global__ void __launch_bounds__(TC_THREADS, 2)
gemm_few_tc_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ FewArgs p) {
    constexpr int FEW_STAGES = few_stages(R);
    constexpr uint32_t FEW_STAGE_BYTES = few_stage_bytes(R);
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full_bar[FEW_STAGES], empty_bar[FEW_STAGES], done_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ float part[(R + 7) * kTcRows];                          // partial rows: [rank][row slot][128]
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t ring = (smem_u32(smem) + 1023u) & ~1023u, full = smem_u32(full_bar), empty = smem_u32(empty_bar);
    const int rank = blockIdx.x, n0 = blockIdx.y * p.th, kb0 = rank * p.kper, kb1 = min(p.nkb, kb0 + p.kper);

    if (warp == 1) tmem_alloc(&tmem_base_s, 32);
    if (tid == 0) {
        for (int s = 0; s < FEW_STAGES; ++s) { mbar_init(&full_bar[s], 9); mbar_init(&empty_bar[s], 1); }
        mbar_init(&done_bar, 1);
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" :: "l"(&wmap) : "memory");
    }
    griddep_wait();
    int m0 = p.rpb ? (int)blockIdx.z * p.rpb : 0, z = p.rpb ? p.g.row_group[m0] : (int)blockIdx.z;
    if (p.blocks > 1) { m0 = z % p.blocks * R; z /= p.blocks; }
    const int rows = z < 0 ? 0 : min(p.rpb ? p.rpb : R, p.g.M - m0);      // no matrix: nothing to do, the same in the cluster
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_launch();                            // tensor memory is held
    const uint32_t tmem = tmem_base_s;
    if (p.splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");       // this block runs
    float v[16];

    if (rows > 0 && warp == 0) {
        if (elect_one()) {
            RingPos r;
            const uint32_t bytes = (uint32_t)p.th * (TBK * 2);
            const uint64_t once = l2_evict_first();
            int i = 0;                            // stages filled so far
            for (int kb = kb0; kb < kb1; ++kb, ++i, r.next(FEW_STAGES)) {
                if (!bar_wait(p.err, empty + 8u * r.s, r.round ^ 1u)) break;
                mbar_expect_tx(full + 8u * r.s, bytes);
                tma_load_3d_hint(ring + r.s * FEW_STAGE_BYTES, &wmap, kb * TBK, n0, z, full + 8u * r.s, once);
            }
            for (int j = max(0, i - FEW_STAGES); j < i; ++j)      // whoever gave up: do not leave with copies in flight
                bar_wait(p.err, full + 8u * (uint32_t)(j % FEW_STAGES), (uint32_t)((j / FEW_STAGES) & 1));
        }
        __syncwarp();
    } else if (rows > 0 && warp == 1) {
        if (elect_one()) {
            RingPos r;
            constexpr uint32_t idesc = umma_idesc_bf16(R);
            for (int kb = kb0; kb < kb1; ++kb, r.next(FEW_STAGES)) {
                if (!bar_wait(p.err, full + 8u * r.s, r.round)) break;
                tc_fence_after();
                const uint32_t addr = ring + r.s * FEW_STAGE_BYTES;
                const uint64_t dw = desc_sw128(addr), da = desc_sw128(addr + TC_W_BYTES);
#pragma unroll
                for (int ks = 0; ks < TBK / 16; ++ks)
                    umma_bf16(tmem, dw + (uint64_t)(ks * 2), da + (uint64_t)(ks * 2), idesc, (kb > kb0 || ks > 0) ? 1u : 0u);
                umma_commit(&empty_bar[r.s]);
            }
            umma_commit(&done_bar);
        }
        __syncwarp();
    } else if (rows > 0) {
        // this thread's row and C groups of four columns of every k block
        constexpr int C = R / 16, DEPTH = 8 / C, GROUP = 4 / C;
        const int et = tid - 64, r = et / (16 / C), c4 = et % (16 / C) * C;
        const float* row = nullptr;
        if (r < rows) {
            const size_t off = (size_t)(p.rpb ? 0 : z) * p.g.a_z + (size_t)(p.g.a_rows ? p.g.a_rows[m0 + r] : m0 + r) * p.g.lda;
            row = ODD && p.g.a16 ? (const float*)((const uint16_t*)p.g.A + off) : p.g.A + off;
        }
        const uint32_t at = ring + TC_W_BYTES + (uint32_t)r * 128u + (uint32_t)(((c4 >> 1) ^ (r & 7)) << 4) + (uint32_t)(c4 & 1) * 8u;
        RingPos f;
        bool ok = true;
        for (int kb = kb0; kb < kb1; kb += DEPTH) {
            const int nb = min(DEPTH, kb1 - kb);
            float4 v[DEPTH][C];
#pragma unroll
            for (int d = 0; d < DEPTH; ++d)
#pragma unroll
                for (int c = 0; c < C; ++c) v[d][c] = direct_load<ODD>(p.g, d < nb ? row : nullptr, (kb + d) * TBK + (c4 + c) * 4, p.avec);
            // hand over in groups that the ring can hold: a group's stages are free before any of them is written
#pragma unroll
            for (int d0 = 0; d0 < DEPTH; d0 += GROUP) {
                if (d0 >= nb) break;
                RingPos h = f;
#pragma unroll
                for (int d = d0; d < d0 + GROUP; ++d) {
                    if (d >= nb) break;
                    ok = ok && bar_wait(p.err, empty + 8u * f.s, f.round ^ 1u);
                    if constexpr (C == 1)
                        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" :: "r"(at + f.s * FEW_STAGE_BYTES), "r"(pack_bf16x2(v[d][0].x, v[d][0].y)),
                                     "r"(pack_bf16x2(v[d][0].z, v[d][0].w)) : "memory");
                    else
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(at + f.s * FEW_STAGE_BYTES), "r"(pack_bf16x2(v[d][0].x, v[d][0].y)),
                                     "r"(pack_bf16x2(v[d][0].z, v[d][0].w)), "r"(pack_bf16x2(v[d][C - 1].x, v[d][C - 1].y)), "r"(pack_bf16x2(v[d][C - 1].z, v[d][C - 1].w)) : "memory");
                    f.next(FEW_STAGES);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0)
                    for (int d = d0; d < min(d0 + GROUP, nb); ++d, h.next(FEW_STAGES)) mbar_arrive(&full_bar[h.s]);
            }
        }
        const int quad = warp & 3, col = n0 + quad * 32 + lane, first = R > 16 ? (warp - 2) / 4 * 16 : 0;
        if (warp < 2 + R / 4) {                                // four warps drain 16 rows: lane = output column, v = the rows
            bar_wait(p.err, smem_u32(&done_bar), 0);
            __syncwarp();
            tc_fence_after();
            tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)first, v);
            if (p.splits == 1 && first < rows) {
                GemmArgs a = p.g;
                if (!ODD) a.c16 = 0;
                a.N = min(a.N, n0 + p.th);
                if (!p.rpb) {
                    move_c(a, z * a.c_z);
                    if (p.epi == 10) a.aux = (const float*)a.aux + (size_t)z * a.c_z;
                }
                epilogue_rows<16>(a, p.epi, v, m0 + first, rows - first, col, lane);
            }
        }
    }
    if (p.splits > 1) {
        const int quad = warp & 3, col = n0 + quad * 32 + lane, slots = (rows + p.splits - 1) / p.splits, first = R > 16 ? (warp - 2) / 4 * 16 : 0;
        const bool drains = warp >= 2 && warp < 2 + R / 4;
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");                       // so do the others
        if (rows > 0 && drains) {                         // row j belongs to block j % splits
            int owner = first % p.splits, slot = first / p.splits;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (first + j < rows) {
                    const uint32_t to = smem_u32(part) + (uint32_t)((rank * slots + slot) * kTcRows + quad * 32 + lane) * 4u;
                    uint32_t remote;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(to), "r"(owner));
                    asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(remote), "f"(v[j]) : "memory");
                }
                if (++owner == p.splits) { owner = 0; ++slot; }
            }
        }
        __syncwarp();
        cluster_arrive_wait();
        if (rows > 0 && drains) {
            const int parts = (p.nkb + p.kper - 1) / p.kper;          // blocks that had any k
            GemmArgs a = p.g;
            if (!ODD) a.c16 = 0;
            a.N = min(a.N, n0 + p.th);
            if (!p.rpb) {
                move_c(a, z * a.c_z);
                if (p.epi == 10) a.aux = (const float*)a.aux + (size_t)z * a.c_z;
            }
            for (int slot = first / 16, j = rank + slot * p.splits; j < rows; j += R / 16 * p.splits, slot += R / 16) {
                float sum[1] = {0.f};
                for (int s = 0; s < parts; ++s) sum[0] += part[(s * slots + slot) * kTcRows + quad * 32 + lane];
                epilogue_rows<1>(a, p.epi, sum, m0 + j, 1, col, lane);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 32);
}

// ---------------------------------------------------------------- how a product is cut
// Costs in cycles per SM, of one k block of a tile: the MMAs take 2 per row, the operands 16 KB + 128 bytes per row at the rate
// an SM draws from L2.  Among the tile heights and cluster sizes the cheapest wins: whole waves of 148 blocks against tiles
// so low that the weights are read too often, and k cut over a cluster only where the tiles alone would leave SMs idle.
constexpr double TC_L2_BYTES_PER_CLK = 48.0;

struct Plan { int bn, mt, splits; };

Plan tc_plan(int M, long long ntz, int nkb) {
    Plan best{16, 1, 1};
    double best_cost = 1e30;
    const int sms = sm_count();
    for (int want = 16; want <= TC_ROWS_MAX; want += 16) {
        const int mt = (M + want - 1) / want, bn = ((M + mt - 1) / mt + 15) & ~15;
        const double block = fmax(2.0 * bn, (TC_W_BYTES + 128.0 * bn) / TC_L2_BYTES_PER_CLK);
        for (int s = 1; s <= 8; s *= 2) {
            if (s > 1 && (nkb < 4 * s || (long long)mt * ntz * s > 2LL * sms)) break;
            const long long blocks = (long long)mt * ntz * s;
            const double waves = (double)((blocks + sms - 1) / sms), k = (double)((nkb + s - 1) / s);
            const double cost = s == 1 ? waves * fmax(k * block, 12.0 * bn) + 12.0 * bn + 3000.0
                                       : waves * (k * block + 3000.0 + 20.0 * bn + 3000.0);
            if (cost < best_cost) { best_cost = cost; best = {bn, mt, s}; }
        }
    }
    return best;
}
// clusters of s blocks of the few-row kernel that the device holds at one time, as the runtime counts them: clusters do not cross its
// processing clusters, whose SMs are no multiple of s; one block per SM is counted for a kernel that allocates tensor memory
int clusters_held(int s) {
    static int held[9] = {};
    if (held[s] == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(s, 64); cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = few_smem(16);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = s; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(gemm_few_tc_kernel<16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few_smem(16)) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, gemm_few_tc_kernel<16, false>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        held[s] = n > 0 ? n : -1;
    }
    return held[s];
}
struct FewPlan { int th, splits; };
// Tile height and blocks per tile.  An SM draws 24 bytes of weights per cycle when all do (HBM), a copy takes 300 cycles at
// least; a block's start and end cost 6000 cycles, half hidden where two blocks share an SM, a shared tile 1500 more.
FewPlan few_plan(int N, int zs, int nkb) {
    FewPlan best{kTcRows, 1};
    double best_cost = 1e30;
    const int sms = sm_count();
    for (int s = 1; s <= 8; ++s) {
        if (s > 1 && (nkb < 2 * s || s > 1 && clusters_held(s) <= 0)) continue;
        for (int th = 16; th <= kTcRows; th += 8) {
            const long long tiles = (long long)((N + th - 1) / th) * zs, blocks = tiles * s;
            const int held = s == 1 ? 2 * sms : clusters_held(s) * s;
            const double rounds = (double)((blocks + held - 1) / held), per_sm = blocks <= sms ? 1.0 : fmin(2.0, (double)blocks / sms);
            const double block = (double)((nkb + s - 1) / s) * fmax(per_sm * th * (TBK * 2) / 24.0, 300.0);
            const double cost = rounds * block + 6000.0 + (rounds - 1.0) * 3000.0 + (s > 1 ? 1500.0 : 0.0);
            if (cost < best_cost * 0.999) { best_cost = cost; best = {th, s}; }
        }
    }
    return best;
}

cudaError_t launch_clustered(const void* kernel, dim3 grid, size_t smem, int cluster, cudaStream_t st, void** args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = cluster; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
    ++n;
    // both kernels wait before they touch anything (see launch_waiting)
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
    cfg.attrs = at; cfg.numAttrs = n;
    count_launch();
    return cudaLaunchKernelExC(&cfg, kernel, args);
}

bool weight_map(CUtensorMap* m, const GemmArgs& a, uint64_t matrices, bool many, int height) {
    const uint64_t wd[3] = {(uint64_t)a.K, (uint64_t)a.N, matrices};
    const uint64_t ws[2] = {(uint64_t)a.K * 2, (uint64_t)(many ? a.w_stride : (long long)a.N * a.K) * 2};
    const uint32_t wb[3] = {TBK, (uint32_t)height, 1};
    return tma_map_bf16_3d(m, a.W, wd, ws, wb);
}

}  // namespace

int pad_weights(const GemmArgs& a, int matrices, cudaStream_t st, GemmArgs* b, bool* done) {
    *done = false;
    const int kpr = (a.K + 7) / 8;
    const long long total = (long long)matrices * a.N * kpr;
    void* buf = nullptr;
    if (total > (1LL << 38) || scratch_alloc(&buf, (size_t)total * 16, st)) {
        set_error("");
        return 0;
    }
    *b = a;
    b->W = buf; b->K = kpr * 8; b->ka = a.K; b->w_stride = (long long)a.N * kpr * 8;
    const cudaError_t e = launch_waiting(pad_weights_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, st, (const uint16_t*)a.W, (uint16_t*)buf, a.K, a.N, kpr,
                                         a.w_stride, total);
    if (e != cudaSuccess) {
        scratch_free(buf, st);
        return cuda_fail(e, "pad_weights", __FILE__, __LINE__);
    }
    *done = true;
    return 0;
}

int gemm_few_tc(const GemmArgs& a, int epilogue, int batch, int rows_per_block, cudaStream_t st, bool* served) {
    *served = false;
    const bool own = a.row_group != nullptr, many = own || batch > 1;
    if (a.K % 8 || a.K < TBK || (uintptr_t)a.W % 16 || (many && (a.w_stride % 8 || a.w_stride <= 0)) || !tma_encode_fn()) return 0;
    if (a.group_off || (own && (rows_per_block > TC_DIRECT_ROWS || batch > 1)) || a.M <= 0) return 0;
    const int R = (own ? rows_per_block : a.M) <= 16 ? 16 : TC_DIRECT_ROWS, blocks = own ? 1 : (a.M + R - 1) / R;
    const int zs = own ? (a.M + rows_per_block - 1) / rows_per_block : batch * blocks;
    if (zs > 65535) return 0;
    FewArgs p{};
    p.g = a;
    if (!a.ka) p.g.ka = a.K;
    p.epi = epilogue;
    p.nkb = (a.K + TBK - 1) / TBK;
    const FewPlan plan = few_plan(a.N, zs, p.nkb);
    if ((a.N + plan.th - 1) / plan.th > 65535) return 0;
    p.th = plan.th;
    p.splits = plan.splits;
    p.kper = (p.nkb + p.splits - 1) / p.splits;
    p.rpb = own ? rows_per_block : 0;
    p.blocks = blocks;
    p.avec = a.lda % 4 == 0 && a.a_z % 4 == 0 && (uintptr_t)a.A % (a.a16 ? 8 : 16) == 0;
    p.err = wait_word(kWaitRows);
    PGK_REQUIRE(p.err, "gemm_rows failed: no pinned host memory");
    CUtensorMap wmap;
    if (!weight_map(&wmap, a, own ? 1u << 20 : (uint64_t)batch, many, p.th)) return 0;      // row groups name matrices that exist
    static bool configured = false;
    const void* const kernels[2][2] = {{(const void*)gemm_few_tc_kernel<16, false>, (const void*)gemm_few_tc_kernel<16, true>},
                                       {(const void*)gemm_few_tc_kernel<32, false>, (const void*)gemm_few_tc_kernel<32, true>}};
    if (!configured) {
        for (int r = 0; r < 4; ++r)
            PGK_CUDA(cudaFuncSetAttribute(kernels[r >> 1][r & 1], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few_smem(r >> 1 ? 32 : 16)));
        configured = true;
    }
    void* args[] = {&wmap, &p};
    const cudaError_t e = launch_clustered(kernels[R / 16 - 1][a.a16 || a.c16 || p.g.ka != a.K], dim3(p.splits, (a.N + p.th - 1) / p.th, zs), few_smem(R), p.splits, st, args);
    if (e != cudaSuccess) return cuda_fail(e, "gemm_few_tc", __FILE__, __LINE__);
    *served = true;
    return 0;
}

int gemm_rows_tc(const GemmArgs& a, int epilogue, int batch, int rows, int max_rows, cudaStream_t st, bool* served) {
    *served = false;
    // what the copies can fetch: k rows of a multiple of 16 bytes, matrices on 16-byte boundaries
    if (a.K % 8 || a.K < TBK || (uintptr_t)a.W % 16 || (batch > 1 && (a.w_stride % 8 || a.w_stride <= 0)) || !tma_encode_fn()) return 0;
    if (a.group_off && batch > TC_MAX_GROUPS) return 0;
    if (rows <= 0) return 0;
    const bool grouped = a.group_off != nullptr;
    if (!grouped && few_rows_pay(a.M, a.N, a.K, batch)) return gemm_few_tc(a, epilogue, batch, a.M, st, served);
    const bool direct = a.a16 && (!a.ka || a.ka == a.K) && a.lda % 8 == 0 && a.a_z % 8 == 0 && (uintptr_t)a.A % 16 == 0 && !a.a_rows;
    TcArgs p{};
    p.g = a;
    if (!a.ka) p.g.ka = a.K;
    p.epi = epilogue;
    p.batch = batch;
    p.err = wait_word(kWaitRows);
    PGK_REQUIRE(p.err, "gemm_rows failed: no pinned host memory");
    p.nt = (a.N + kTcRows - 1) / kTcRows;
    p.nkb = (a.K + TBK - 1) / TBK;
    if (grouped) {
        // rows per group are known on the device only; aim at the mean
        const int mean = (rows + batch - 1) / batch, most = max_rows < rows ? max_rows : rows;
        const int cap = 2 * mean < most ? 2 * mean : most;
        p.bn = cap >= 192 ? 256 : (cap >= 96 ? 128 : (cap >= 48 ? 64 : 32));
        p.abox = p.bn >= 64 ? 64 : 32;
        p.mt = 0;
        p.splits = 1;
    } else {
        const Plan plan = tc_plan(a.M, (long long)p.nt * batch, p.nkb);
        p.bn = plan.bn; p.mt = plan.mt; p.splits = plan.splits;
        p.abox = p.bn;
    }
    const int held = (p.bn + p.abox - 1) / p.abox * p.abox;
    p.stage_bytes = (TC_W_BYTES + (uint32_t)held * (TBK * 2) + 1023u) & ~1023u;
    p.stages = (int)(TC_RING_BYTES / p.stage_bytes);
    if (p.stages > TC_MAX_STAGES) p.stages = TC_MAX_STAGES;

    const int nb = grouped ? 1 : batch;
    void* abuf = nullptr;
    CUtensorMap wmap, amap;
    bool described = weight_map(&wmap, a, (uint64_t)batch, batch > 1, kTcRows);
    const uint64_t ad[3] = {(uint64_t)a.K, (uint64_t)nb, (uint64_t)rows};
    const uint32_t ab[3] = {TBK, 1, (uint32_t)p.abox};
    cudaError_t e = cudaSuccess;
    if (direct) {                                 // rows as the product before left them: fetched where they are
        const uint64_t as[2] = {(uint64_t)(nb > 1 ? a.a_z : a.lda) * 2, (uint64_t)a.lda * 2};
        described = described && tma_map_bf16_3d(&amap, a.A, ad, as, ab);
    } else {
        const size_t bytes = (size_t)rows * nb * a.K * 2;
        if (scratch_alloc(&abuf, bytes, st)) {    // no room for the copy: the tiles of seq_gemm.cu need none
            set_error("");
            return 0;
        }
        const uint64_t as[2] = {(uint64_t)a.K * 2, (uint64_t)nb * a.K * 2};
        described = described && tma_map_bf16_3d(&amap, abuf, ad, as, ab);
    }
    if (!described) {
        if (abuf) scratch_free(abuf, st);
        set_error("gemm_rows failed: the copies of a %d x %d x %d product cannot be described", rows, a.N, a.K);
        return 1;
    }
    if (!direct) {
        const int kpr = a.K / 8, chunks = nb * kpr;
        const bool vec = a.lda % 4 == 0 && a.a_z % 4 == 0 && (uintptr_t)a.A % (a.a16 ? 8 : 16) == 0;
        int gy = (chunks + 255) / 256;
        if (gy > 8) gy = 8;
        e = launch_waiting(rows_to_bf16_kernel, dim3(rows, gy), dim3(chunks >= 256 ? 256 : (chunks + 31) / 32 * 32), 0, st, p.g, (uint16_t*)abuf, batch, kpr, vec);
    }
    if (e == cudaSuccess) {
        const int sms = sm_count();
        const long long tiles = (long long)batch * p.mt * p.nt;
        const int grid = grouped ? sms : (p.splits > 1 ? (int)(tiles * p.splits) : (int)(tiles < sms ? tiles : sms));
        static bool configured = false;
        if (!configured) {
            e = cudaFuncSetAttribute(gemm_rows_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_RING_BYTES + 1024);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_rows_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_RING_BYTES + 1024);
            configured = e == cudaSuccess;
        }
        void* args[] = {&wmap, &amap, &p};
        if (e == cudaSuccess) e = launch_clustered(a.c16 ? (const void*)gemm_rows_tc_kernel<true> : (const void*)gemm_rows_tc_kernel<false>, dim3(grid), TC_RING_BYTES + 1024, p.splits, st, args);
    }
    const int rc = abuf ? scratch_free(abuf, st) : 0;
    if (e != cudaSuccess) return cuda_fail(e, "gemm_rows_tc", __FILE__, __LINE__);
    *served = rc == 0;
    return rc;
}

}  // namespace pgk

extern "C" int pgk_gemm_rows_wait_error(int* out) {
    PGK_CUDA(cudaDeviceSynchronize());
    *out = pgk::wait_raised(pgk::kWaitRows);
    return 0;
}
