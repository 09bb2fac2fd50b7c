// seq_gemm.cu -- C[m, n] = sum_k A[row(m), k] * W[g][n, k] for the token-major ("ragged batch") models: float32
// activations, weights [N, K] K-contiguous in bfloat16 or float32, float32 accumulation and output.
//
//   * many rows (prompts): bfloat16 weights run in seq_gemm_tc.cu (tcgen05) wherever its copies can fetch the operands; the
//     64 x 64 x 32 tiles here (four warps, mma.sync m16n8k16, the activation tile rounded to bfloat16 while it is staged) serve
//     the rest, and float32 weights on FMAs with no reduced-precision mode anywhere;
//   * few rows (decoding): a warp per output column streams its weight row once with 128-bit loads and serves up to
//     eight rows of A held in shared memory;
//   * groups: `group_off` [E + 1] cuts the rows into E consecutive runs, run e uses weight matrix e (mixture of experts:
//     the rows are (token, slot) pairs sorted by expert); `a_rows` gathers the rows of A, so the tokens are never copied;
//   * epilogues: plain; gate/up pairs (W holds gate_j in row 2j and up_j in row 2j + 1, the output is silu(gate) * up,
//     [M, N / 2]); scale then tanh cap (the logit head); clamped gate/up pairs g = min(gate, limit), u = clamp(up, +-limit),
//     output g sigmoid(alpha g) (u + 1); C += column vector * product (layer scale and residual add in one pass);
//     gelu_tanh(product) * gathered table entry (per-layer token inputs); squared ReLU; gate/up pairs with gelu_tanh(gate) * up;
//     gelu_erf(product); gelu_tanh(product); product * sigmoid(gate row's element);
//   * batches: grid.z can also walk `batch` independent products whose A columns, matrices and C columns are a fixed number
//     of elements apart (one product per attention head on slices of the same rows).
#include "common.cuh"
#include "seq_gemm.cuh"
#include "../../include/pgk_b200.h"

using namespace pgk;

namespace {

// What a caller asks of the rows beside the weights' type: bfloat16 A (16) and C (32), for bfloat16 weights, many rows and a C that is only written.
struct Rows16 {
    int wdt, a16, c16;
    explicit Rows16(int dt) : wdt(dt & 15), a16(dt >> 4 & 1), c16(dt >> 5 & 1) {}
};

template <int EPI>
__device__ __forceinline__ void store_pair(const GemmArgs& a, int row, int col, float c0, float c1) {
    // (row, col) and (row, col + 1), col even
    if (EPI == 1) {
        if (col + 1 < a.N) put(a, (size_t)row * a.ldc + (col >> 1), silu_f(c0) * c1);
        return;
    }
    if (EPI == 7) {
        if (col + 1 < a.N) put(a, (size_t)row * a.ldc + (col >> 1), gelu_tanh_f(c0) * c1);
        return;
    }
    if (EPI == 3) {          // scale = alpha, cap = limit
        if (col + 1 < a.N) {
            const float g = fminf(c0, a.cap), u = fminf(fmaxf(c1, -a.cap), a.cap);
            put(a, (size_t)row * a.ldc + (col >> 1), g / (1.f + expf(-a.scale * g)) * (u + 1.f));
        }
        return;
    }
    if (EPI == 2) {
        c0 *= a.scale; c1 *= a.scale;
        if (a.cap > 0.f) { c0 = a.cap * tanhf(c0 / a.cap); c1 = a.cap * tanhf(c1 / a.cap); }
    }
    if (EPI == 6) {          // squared ReLU
        c0 = fmaxf(c0, 0.f); c1 = fmaxf(c1, 0.f);
        c0 *= c0; c1 *= c1;
    }
    if (EPI == 8) { c0 = gelu_erf_f(c0); c1 = gelu_erf_f(c1); }
    if (EPI == 9) { c0 = gelu_tanh_f(c0); c1 = gelu_tanh_f(c1); }
    if (EPI == 10) {         // the gate's columns are as far apart as the output's: `aux` moves with C from batch to batch
        const float* g = (const float*)a.aux + (size_t)row * a.aux_ld + a.aux_off + col;
        if (col < a.N) c0 *= 1.f / (1.f + expf(-g[0]));
        if (col + 1 < a.N) c1 *= 1.f / (1.f + expf(-g[1]));
    }
    const size_t at = (size_t)row * a.ldc + col;
    if (EPI == 4) {
        float* p = a.C + at;
        if (col < a.N) p[0] = fmaf(a.colv[col], c0, p[0]);
        if (col + 1 < a.N) p[1] = fmaf(a.colv[col + 1], c1, p[1]);
        return;
    }
    if (EPI == 5) {
        if (col < a.N) put(a, at, gelu_tanh_f(c0) * aux_at(a, row, col));
        if (col + 1 < a.N) put(a, at + 1, gelu_tanh_f(c1) * aux_at(a, row, col + 1));
        return;
    }
    if (col < a.N) put(a, at, c0);
    if (col + 1 < a.N) put(a, at + 1, c1);
}

constexpr int BM = 64, BN = 64, BK = 32;

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem_row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(smem_row)));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// ---------------------------------------------------------------- many rows, bfloat16 weights: tensor cores
template <int EPI, bool R16>
__global__ void __launch_bounds__(128) gemm_rows_bf16_kernel(GemmArgs a) {
    if (!R16) a.a16 = a.c16 = 0;
    const int e = blockIdx.z;
    move_a(a, e * a.a_z);
    move_c(a, e * a.c_z);
    if (EPI == 10) a.aux = (const float*)a.aux + (size_t)e * a.c_z;
    const int m_begin = a.group_off ? a.group_off[e] : 0;
    const int m_end = a.group_off ? a.group_off[e + 1] : a.M;
    const int m0 = m_begin + blockIdx.y * BM;
    if (m0 >= m_end) return;
    const int n0 = blockIdx.x * BN;
    const uint16_t* W = (const uint16_t*)a.W + (size_t)e * a.w_stride;

    __shared__ __align__(16) uint16_t As[2][BM][BK + 8];
    __shared__ __align__(16) uint16_t Ws[2][BN][BK + 8];
    __shared__ int rows[BM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < BM) {
        const int r = m0 + tid;
        rows[tid] = r < m_end ? (a.a_rows ? a.a_rows[r] : r) : -1;
    }
    __syncthreads();
    const bool avec = (a.K % 4 == 0) && (a.lda % 4 == 0) && (((uintptr_t)a.A & (a.a16 ? 7 : 15)) == 0);
    const bool wvec = (a.K % 8 == 0) && (((uintptr_t)W & 15) == 0);

    float4 ra[4];
    uint4 rw[2];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = tid + i * 128, r = idx >> 3, c = (idx & 7) * 4, gr = rows[r], k = k0 + c;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (gr >= 0) {
                const size_t p = (size_t)gr * a.lda + k;
                if (avec && k + 3 < a.K) v = a_at4(a, p);
                else {
                    if (k < a.K) v.x = a_at(a, p);
                    if (k + 1 < a.K) v.y = a_at(a, p + 1);
                    if (k + 2 < a.K) v.z = a_at(a, p + 2);
                    if (k + 3 < a.K) v.w = a_at(a, p + 3);
                }
            }
            ra[i] = v;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int idx = tid + i * 128, r = idx >> 2, c = (idx & 3) * 8, n = n0 + r, k = k0 + c;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (n < a.N) {
                const uint16_t* p = W + (size_t)n * a.K + k;
                if (wvec && k + 7 < a.K) v = *(const uint4*)p;
                else {
                    uint16_t t[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) t[j] = (k + j < a.K) ? p[j] : (uint16_t)0;
                    v.x = t[0] | ((uint32_t)t[1] << 16); v.y = t[2] | ((uint32_t)t[3] << 16);
                    v.z = t[4] | ((uint32_t)t[5] << 16); v.w = t[6] | ((uint32_t)t[7] << 16);
                }
            }
            rw[i] = v;
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = tid + i * 128, r = idx >> 3, c = (idx & 7) * 4;
            uint2 v = make_uint2(pack_bf16x2(ra[i].x, ra[i].y), pack_bf16x2(ra[i].z, ra[i].w));
            *(uint2*)&As[buf][r][c] = v;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int idx = tid + i * 128, r = idx >> 2, c = (idx & 3) * 8;
            *(uint4*)&Ws[buf][r][c] = rw[i];
        }
    };

    float acc[2][4][4] = {};
    const int wm = warp >> 1, wn = warp & 1, g = lane >> 2, tg = lane & 3;
    const int nk = (a.K + BK - 1) / BK;
    fetch(0);
    stash(0);
    __syncthreads();
    for (int kt = 0; kt < nk; ++kt) {
        const int buf = kt & 1;
        if (kt + 1 < nk) fetch((kt + 1) * BK);
#pragma unroll
        for (int kk = 0; kk < BK; kk += 16) {
            // fragments by ldmatrix (rows are 80 bytes apart: 16-byte aligned and conflict-free)
            uint32_t af[2][4], bf[4][2];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)      // 16 x 16 of A: lanes 0-15 name rows 0-15 at k, lanes 16-31 the same rows at k + 8
                ldmatrix_x4(af[mi], &As[buf][wm * 32 + mi * 16 + (lane & 15)][kk + ((lane >> 4) << 3)]);
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {    // 16 columns x 16 k of W: (n 0-7, k 0-7), (n 0-7, k 8-15), (n 8-15, k 0-7), (n 8-15, k 8-15)
                uint32_t r[4];
                ldmatrix_x4(r, &Ws[buf][wn * 32 + nj * 16 + (lane & 7) + ((lane >> 4) << 3)][kk + (((lane >> 3) & 1) << 3)]);
                bf[2 * nj][0] = r[0]; bf[2 * nj][1] = r[1]; bf[2 * nj + 1][0] = r[2]; bf[2 * nj + 1][1] = r[3];
            }
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) mma_bf16(acc[mi][ni], af[mi], bf[ni]);
        }
        if (kt + 1 < nk) stash(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
            const int r = m0 + wm * 32 + mi * 16 + g, c = n0 + wn * 32 + ni * 8 + 2 * tg;
            if (r < m_end) store_pair<EPI>(a, r, c, acc[mi][ni][0], acc[mi][ni][1]);
            if (r + 8 < m_end) store_pair<EPI>(a, r + 8, c, acc[mi][ni][2], acc[mi][ni][3]);
        }
}

// ---------------------------------------------------------------- many rows, float32 weights: FMAs, summed in k order
// Tiles of 8 TM x 64; a thread has TM rows and four columns and reads four k of each at once.  What bounds small products is a tile's walk over k, one
// slab after the other: slabs are on their way in registers while one is multiplied -- two with the lower tiles, whose slabs take less than
// a load's way; with TM = 8 one, the registers of a second cost more --, and lower tiles put products of few tiles on all SMs (us, one slab of 16 at
// a time and 64 rows -> here: 983 x 256 x 1650 230 -> 56, 101 x 802 x 212 33 -> 10.4, 700 x 700 x 700 99 -> 35, 1000 x 3000 x 2048 658 -> 372; copies by
// cp.async, which an SM takes 16 bytes a cycle of, 60, 8.5, 38 and 418).  Every sum goes over k in order, whatever the tile.
template <int EPI, int TM>
__global__ void __launch_bounds__(128) gemm_rows_f32_kernel(GemmArgs a) {
    constexpr int TR = 8 * TM, FK = 32, AHEAD = TM == 8 ? 1 : 2, LD = FK + 4, L4 = FK / 4, LR = 128 / L4, LA = TR / LR, LW = BN / LR;
    const int e = blockIdx.z;
    a.a16 = a.c16 = 0;
    a.A += (size_t)e * a.a_z;
    a.C += (size_t)e * a.c_z;
    if (EPI == 10) a.aux = (const float*)a.aux + (size_t)e * a.c_z;
    const int m_begin = a.group_off ? a.group_off[e] : 0;
    const int m_end = a.group_off ? a.group_off[e + 1] : a.M;
    const int m0 = m_begin + blockIdx.y * TR;
    if (m0 >= m_end) return;
    const int n0 = blockIdx.x * BN;
    const float* W = (const float*)a.W + (size_t)e * a.w_stride;
    __shared__ __align__(16) float As[2][TR][LD];
    __shared__ __align__(16) float Ws[2][BN][LD];
    const int tid = threadIdx.x, lk = tid % L4 * 4, lr = tid / L4;        // loads: four k of the slab, every LR-th row
    const bool avec = a.lda % 4 == 0 && ((uintptr_t)a.A & 15) == 0, wvec = a.K % 4 == 0 && ((uintptr_t)W & 15) == 0;
    const float *pa[LA], *pw[LW];                                         // rows beyond the edge: none
#pragma unroll
    for (int i = 0; i < LA; ++i) {
        const int r = m0 + lr + LR * i;
        pa[i] = r < m_end ? a.A + (size_t)(a.a_rows ? a.a_rows[r] : r) * a.lda + lk : nullptr;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) pw[i] = n0 + lr + LR * i < a.N ? W + (size_t)(n0 + lr + LR * i) * a.K + lk : nullptr;
    float4 ra[AHEAD][LA], rw[AHEAD][LW];
    auto four = [&](const float* p, int k, bool vec) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!p) return v;
        if (vec && k + lk + 4 <= a.K) return *(const float4*)(p + k);
        if (k + lk < a.K) v.x = p[k];
        if (k + lk + 1 < a.K) v.y = p[k + 1];
        if (k + lk + 2 < a.K) v.z = p[k + 2];
        if (k + lk + 3 < a.K) v.w = p[k + 3];
        return v;
    };
    auto fetch = [&](float4 (&ra)[LA], float4 (&rw)[LW], int k0) {
#pragma unroll
        for (int i = 0; i < LA; ++i) ra[i] = four(pa[i], k0, avec);
#pragma unroll
        for (int i = 0; i < LW; ++i) rw[i] = four(pw[i], k0, wvec);
    };
    auto stash = [&](const float4 (&ra)[LA], const float4 (&rw)[LW], int b) {
#pragma unroll
        for (int i = 0; i < LA; ++i) *(float4*)&As[b][lr + LR * i][lk] = ra[i];
#pragma unroll
        for (int i = 0; i < LW; ++i) *(float4*)&Ws[b][lr + LR * i][lk] = rw[i];
    };
    const int ty = tid >> 4, tx = tid & 15;          // rows ty + 8 i, columns tx + 16 j: no two lanes of a quarter warp share a bank
    float acc[TM][4] = {};
    auto multiply = [&](int b) {
#pragma unroll 2
        for (int k = 0; k < FK; k += 4) {
            float4 av[TM], wv[4];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *(const float4*)&As[b][ty + 8 * i][k];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = *(const float4*)&Ws[b][tx + 16 * j][k];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(av[i].x, wv[j].x, acc[i][j]);
                    acc[i][j] = fmaf(av[i].y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(av[i].z, wv[j].z, acc[i][j]);
                    acc[i][j] = fmaf(av[i].w, wv[j].w, acc[i][j]);
                }
        }
    };
    fetch(ra[0], rw[0], 0);
    if (AHEAD == 2 && FK < a.K) fetch(ra[AHEAD - 1], rw[AHEAD - 1], FK);
    stash(ra[0], rw[0], 0);
    __syncthreads();
    for (int k0 = 0; k0 < a.K; k0 += 2 * FK) {       // slabs k0 and k0 + FK
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int k = k0 + q * FK, from = AHEAD == 2 ? q ^ 1 : 0;
            if (k >= a.K) break;
            if (k + AHEAD * FK < a.K) fetch(ra[AHEAD == 2 ? q : 0], rw[AHEAD == 2 ? q : 0], k + AHEAD * FK);
            multiply(q);
            if (k + FK < a.K) stash(ra[from], rw[from], q ^ 1);
            __syncthreads();
        }
    }
    // neighbouring columns, as the epilogue wants them, meet in shared memory
    float* const out = &Ws[0][0][0];                 // [TR][BN + 2]
    static_assert(TR * (BN + 2) <= 2 * BN * LD);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) out[(ty + 8 * i) * (BN + 2) + tx + 16 * j] = acc[i][j];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = m0 + ty + 8 * i;
        if (r >= m_end) continue;
        const float* v = out + (ty + 8 * i) * (BN + 2) + 2 * tx;
        store_pair<EPI>(a, r, n0 + 2 * tx, v[0], v[1]);
        store_pair<EPI>(a, r, n0 + 32 + 2 * tx, v[32], v[33]);
    }
}

// ---------------------------------------------------------------- few rows: one warp per output column (pair)
// Block = 4 .. 16 warps; the block's rows of A (<= RMAX, all using the same weight matrix) sit in shared memory as float32;
// a warp owns two consecutive output columns (a gate/up pair under EPI 1), reads their weight rows once with 128-bit
// loads and forms the dot products of every row.  grid = (column pairs / 8, row blocks).
constexpr int RMAX = 8;

template <typename TW> struct WLoad;
template <> struct WLoad<uint16_t> {
    static constexpr int VEC = 8;
    static __device__ __forceinline__ void unpack(const uint4& v, float (&w)[8]) {
        w[0] = bf16lo(v.x); w[1] = bf16hi(v.x); w[2] = bf16lo(v.y); w[3] = bf16hi(v.y);
        w[4] = bf16lo(v.z); w[5] = bf16hi(v.z); w[6] = bf16lo(v.w); w[7] = bf16hi(v.w);
    }
    static __device__ __forceinline__ float one(const uint16_t* p) { return bf16_bits_to_f32(*p); }
};
template <> struct WLoad<float> {
    static constexpr int VEC = 4;
    static __device__ __forceinline__ void unpack(const uint4& v, float (&w)[8]) {
        w[0] = __uint_as_float(v.x); w[1] = __uint_as_float(v.y); w[2] = __uint_as_float(v.z); w[3] = __uint_as_float(v.w);
        w[4] = w[5] = w[6] = w[7] = 0.f;
    }
    static __device__ __forceinline__ float one(const float* p) { return *p; }
};

constexpr int FEW_MAX_WARPS = 16;  // warps (= column pairs) per block: 4 .. 16, more when the staged rows take much shared memory
constexpr int FEW_UN = 4;         // 128-bit loads per weight row in flight per lane

template <typename TW, int EPI, bool ROUND>
__global__ void __launch_bounds__(FEW_MAX_WARPS * 32) gemm_few_rows_kernel(GemmArgs a, int rows_per_block) {
    extern __shared__ __align__(16) float xs[];                 // [rows][K]
    const int r0 = blockIdx.y * rows_per_block;
    const int nr = min(rows_per_block, a.M - r0);
    a.a16 = a.c16 = 0;
    const int grp = a.row_group ? a.row_group[r0] : (int)blockIdx.z;
    if (grp < 0) return;                                        // a row without a matrix (its output is formed elsewhere)
    a.A += (size_t)blockIdx.z * a.a_z;
    a.C += (size_t)blockIdx.z * a.c_z;
    if (EPI == 10) a.aux = (const float*)a.aux + (size_t)blockIdx.z * a.c_z;
    const TW* W = (const TW*)a.W + (size_t)grp * a.w_stride;
    constexpr int VEC = WLoad<TW>::VEC;
    const bool vec = (a.K % VEC == 0) && (((uintptr_t)W & 15) == 0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = (blockIdx.x * (blockDim.x >> 5) + warp) * 2;
    const bool live = c0 < a.N;
    const bool two = c0 + 1 < a.N;
    const TW* w0 = W + (size_t)(live ? c0 : 0) * a.K;
    const TW* w1 = W + (size_t)(two ? c0 + 1 : (live ? c0 : 0)) * a.K;
    // the first weight loads do not depend on the activations: issue them before staging x
    uint4 ru[FEW_UN], rv[FEW_UN];
    const int kstep = 32 * VEC;
    if (vec) {
#pragma unroll
        for (int j = 0; j < FEW_UN; ++j) {
            const int k = lane * VEC + j * kstep;
            ru[j] = rv[j] = make_uint4(0u, 0u, 0u, 0u);
            if (live && k < a.K) { ru[j] = ldg_stream(w0 + k); rv[j] = ldg_stream(w1 + k); }
        }
    }
    const bool xvec = (a.K % 4 == 0) && (a.lda % 4 == 0) && (((uintptr_t)a.A & 15) == 0);
    if (xvec) {
        const int k4 = a.K >> 2;
        for (int i = threadIdx.x; i < nr * k4; i += blockDim.x) {
            const int r = i / k4, k = (i - r * k4) * 4;
            const int gr = a.a_rows ? a.a_rows[r0 + r] : r0 + r;
            float4 v = *(const float4*)(a.A + (size_t)gr * a.lda + k);
            if (ROUND) { v.x = round_bf16(v.x); v.y = round_bf16(v.y); v.z = round_bf16(v.z); v.w = round_bf16(v.w); }
            *(float4*)(xs + r * a.K + k) = v;
        }
    } else {
        for (int i = threadIdx.x; i < nr * a.K; i += blockDim.x) {
            const int r = i / a.K, k = i - r * a.K;
            const int gr = a.a_rows ? a.a_rows[r0 + r] : r0 + r;
            const float v = a.A[(size_t)gr * a.lda + k];
            xs[i] = ROUND ? round_bf16(v) : v;
        }
    }
    __syncthreads();
    if (!live) return;
    float acc0[RMAX] = {}, acc1[RMAX] = {};
    if (vec) {
        for (int kb = 0; kb < a.K; kb += FEW_UN * kstep) {
            uint4 cu[FEW_UN], cv[FEW_UN];
#pragma unroll
            for (int j = 0; j < FEW_UN; ++j) { cu[j] = ru[j]; cv[j] = rv[j]; }
            const int kn = kb + FEW_UN * kstep;
            if (kn < a.K) {
#pragma unroll
                for (int j = 0; j < FEW_UN; ++j) {
                    const int k = kn + lane * VEC + j * kstep;
                    if (k < a.K) { ru[j] = ldg_stream(w0 + k); rv[j] = ldg_stream(w1 + k); }
                }
            }
#pragma unroll
            for (int j = 0; j < FEW_UN; ++j) {
                const int k = kb + lane * VEC + j * kstep;
                if (k >= a.K) continue;
                float u[8], v[8];
                WLoad<TW>::unpack(cu[j], u);
                WLoad<TW>::unpack(cv[j], v);
#pragma unroll
                for (int r = 0; r < RMAX; ++r) {
                    if (r < nr) {
                        float x[8];
                        *(float4*)&x[0] = *(const float4*)(xs + r * a.K + k);
                        if (VEC == 8) *(float4*)&x[4] = *(const float4*)(xs + r * a.K + k + 4);
#pragma unroll
                        for (int q = 0; q < VEC; ++q) {
                            acc0[r] = fmaf(x[q], u[q], acc0[r]);
                            acc1[r] = fmaf(x[q], v[q], acc1[r]);
                        }
                    }
                }
            }
        }
    } else {
        for (int k = lane; k < a.K; k += 32) {
            const float u = WLoad<TW>::one(w0 + k), v = WLoad<TW>::one(w1 + k);
#pragma unroll
            for (int r = 0; r < RMAX; ++r)
                if (r < nr) {
                    acc0[r] = fmaf(xs[r * a.K + k], u, acc0[r]);
                    acc1[r] = fmaf(xs[r * a.K + k], v, acc1[r]);
                }
        }
    }
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
        if (r < nr) {
            const float s0 = warp_sum(acc0[r]), s1 = warp_sum(acc1[r]);
            if (lane == 0) store_pair<EPI>(a, r0 + r, c0, s0, s1);
        }
    }
}

// The tcgen05 form (seq_gemm_tc.cu) takes 10 us from the rounding of the rows to its last store, little more for more work; the tiles
// below 4 us and 18 ns per k in a wave, again for every further wave.  Beyond the kernel of few rows (few_rows_pay), which needs no rounding pass, the line lies
// where the two meet, by the tiles there are (us, tiles -> tcgen05): K = 64 5.2 -> 10.3 for one tile or 128, 12.4 -> 15.1 for 1024,
// 42 -> 35 for 4608; K = 256 9.3 -> 10.4 for 128, 11.4 -> 10.5 for 256; K = 320 10.4 -> 10.4 for 32; K = 512 14.4 -> 12.4 for 4.  Groups: by
// the tiles that have rows, groups of the mean length taken, and a little for the grid's empty ones: 32 tiles K = 384 10.4 -> 12.5, K =
// 512 12.5 -> 12.5; 512 tiles K = 192 14.7 -> 16.5, K = 256 18.6 -> 16.5.
inline bool many_tc_pays(const GemmArgs& a, int groups, int max_rows, int rows) {
    const double nt = (a.N + BN - 1) / BN;
    if (!a.group_off) return few_rows_pay(a.M, a.N, a.K, groups) || a.K * ((double)groups * ((a.M + BM - 1) / BM) * nt + 512.0) >= 180000.0;
    const int mean = (rows + groups - 1) / groups;
    const double live = (double)groups * ((mean + BM - 1) / BM) * nt, grid = (double)groups * ((max_rows + BM - 1) / BM) * nt;
    return a.K * (2.0 * live + 0.25 * grid + 1000.0) >= 500000.0;
}

inline bool off_boundaries(const GemmArgs& a, int matrices) {
    return a.K % 8 != 0 || (uintptr_t)a.W % 16 != 0 || (matrices > 1 && a.w_stride % 8 != 0);
}
// Bringing the matrices to boundaries first (pad_weights) takes 2 us and 0.9 us per million elements, the tcgen05 form then what it takes; the kernels
// for any K cost (us, before -> with it): tiles 36 ns per k and more, from 160 on always slower (9 rows 600 x 300 14.5 -> 8.3, 768 x 1004 39 -> 8.6, 5664 x 3574 236 ->
// 29; 3500 rows 1536 x 2668 399 -> 47, 5664 x 3574 2137 -> 197); a warp per column pair 4 ns per k, 2 more for every further row (a third of that where K is
// a multiple of four), or 2.5 us per million elements (one row 768 x 1004 6.4 -> 8.9, 1536 x 2668 20.5 -> 10.6, 5664 x 3574 56 -> 27; eight rows 600 x 300 7.1 -> 8.4, 1024 x 746
// 16.6 -> 8.7).
inline bool pad_pays(const GemmArgs& a, int matrices) {
    if (a.M > RMAX) return a.K >= 160;
    const double m = (double)matrices * a.N * a.K * 1e-6, chain = a.K * (0.004 + 0.0019 * (a.M - 1) * (a.K % 4 ? 1.0 : 0.3));
    return a.K >= 64 && 4.5 + (chain > 2.45 * m ? chain : 2.45 * m) > 1.05 * (8.5 + 0.92 * m);
}

// bfloat16 weights go to the tcgen05 form wherever it is faster and its copies can fetch the operands; `rows` bounds the rows of
// A (-1: the groups' total is not known here).  The tiles below serve what is left: short k, K no multiple of 8, matrices off
// 16-byte boundaries, groups without a bound.
template <int EPI>
int launch_many(const GemmArgs& a, int wdt, int groups, int max_rows, cudaStream_t st, int rows = -1) {
    if (wdt == 2 && !a.group_off && off_boundaries(a, groups) && pad_pays(a, groups)) {
        GemmArgs b;
        bool done = false;
        if (const int rc = pad_weights(a, groups, st, &b, &done)) return rc;
        if (done) {
            bool served = false;
            const int rc = gemm_rows_tc(b, EPI, groups, rows, max_rows, st, &served), rf = scratch_free((void*)b.W, st);
            if (rc || rf || served) return rc ? rc : rf;
        }
    }
    if (wdt == 2 && rows >= 0 && many_tc_pays(a, groups, max_rows, rows)) {
        bool served = false;
        if (const int rc = gemm_rows_tc(a, EPI, groups, rows, max_rows, st, &served)) return rc;
        if (served) return 0;
    }
    dim3 grid((a.N + BN - 1) / BN, (max_rows + BM - 1) / BM, groups);
    if (a.a16 || a.c16) PGK_CUDA(launch(gemm_rows_bf16_kernel<EPI, true>, grid, dim3(128), 0, st, a));
    else if (wdt == 2) PGK_CUDA(launch(gemm_rows_bf16_kernel<EPI, false>, grid, dim3(128), 0, st, a));
    else {
        // the highest tiles when lower ones would not fit the SMs at one time (1000 x 3000 x 2048 493 -> 372, 700 x 1500 x 800 101 -> 58; 151 x 1830 x 2003, 145
        // tiles of 32 rows, 66 against 95 and 84 with 64 and 16), the lowest when not half of them have one (64 x 512 x 400 16.6 -> 14.5)
        const long long low = (long long)grid.x * ((max_rows + 31) / 32) * groups;
        const int tm = low > sm_count() ? 8 : (2 * low >= sm_count() ? 4 : 2);
        grid.y = (max_rows + 8 * tm - 1) / (8 * tm);
        if (tm == 8) PGK_CUDA(launch(gemm_rows_f32_kernel<EPI, 8>, grid, dim3(128), 0, st, a));
        else if (tm == 4) PGK_CUDA(launch(gemm_rows_f32_kernel<EPI, 4>, grid, dim3(128), 0, st, a));
        else PGK_CUDA(launch(gemm_rows_f32_kernel<EPI, 2>, grid, dim3(128), 0, st, a));
    }
    return 0;
}

template <typename TW, int EPI, bool ROUND>
int launch_few_t(const GemmArgs& a, int rows_per_block, cudaStream_t st, int batch) {
    const size_t smem = (size_t)rows_per_block * a.K * sizeof(float);
    static size_t configured = 0;
    if (smem > 48 * 1024 && smem > configured) {
        PGK_CUDA(cudaFuncSetAttribute(gemm_few_rows_kernel<TW, EPI, ROUND>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured = 200 * 1024;
    }
    // a block's shared memory decides how many blocks fit an SM: keep about 16 warps per SM streaming
    const int warps = smem <= 48 * 1024 ? 4 : (smem <= 100 * 1024 ? 8 : FEW_MAX_WARPS);
    dim3 grid(((a.N + 1) / 2 + warps - 1) / warps, (a.M + rows_per_block - 1) / rows_per_block, batch);
    PGK_CUDA(launch(gemm_few_rows_kernel<TW, EPI, ROUND>, grid, dim3(warps * 32), smem, st, a, rows_per_block));
    return 0;
}

// Few rows, bfloat16 weights: the tcgen05 form (gemm_few_tc) reads the weights at the rate of HBM whatever the rows, but takes 7 us
// from its first barrier to its last store; a warp per column pair starts faster and then costs time per row.  The line lies where
// the two meet, rows^2 N K (matrices) = 2^24 (us, warp per pair -> tcgen05): one row of 2048 x 2048 7.4 -> 8.3, of 8192 x 2048
// 11 -> 11, of 32768 x 2048 35 -> 25; eight rows of 512 x 2048 14.4 -> 8.0, 2048 x 8192 37 -> 14.5, 24576 x 4096 158 -> 37; eight
// rows with matrices of their own, 4096 x 2048, 37 -> 14.5.  Up to 4096 columns the warps are one wave, whose time is its longest
// warp's: four rows of 4096 x 512 6.3 -> 8.3, two of 4096 x 1024 6.3 -> 8.2, eight of 2048 x 128 5.2 -> 5.7, but eight of 4096 x 256 7.2 -> 6.0,
// four of 2048 x 1024 8.3 -> 6.5, two of 4096 x 2048 10.4 -> 9.1: there rows^2 K must reach 2^14 as well, or K 2048 for two rows.
inline bool few_tc_pays(const GemmArgs& a, int rows_per_block, int batch) {
    const double rows = a.row_group ? rows_per_block : a.M;
    const double matrices = a.row_group ? (a.M + rows_per_block - 1) / rows_per_block : batch;
    if (matrices * a.N <= 4096.0 && rows * rows * a.K < 16384.0 && (rows < 2.0 || a.K < 2048)) return false;
    return rows * rows * matrices * (double)a.N * (double)a.K >= 16777216.0;
}

template <int EPI>
int launch_few(const GemmArgs& a, int wdt, int rows_per_block, cudaStream_t st, int batch = 1) {
    if (wdt == 2 && !a.row_group && a.M <= rows_per_block && off_boundaries(a, batch) && pad_pays(a, batch)) {
        GemmArgs b;
        bool done = false;
        if (const int rc = pad_weights(a, batch, st, &b, &done)) return rc;
        if (done) {
            bool served = false;
            const int rc = gemm_few_tc(b, EPI, batch, a.M, st, &served), rf = scratch_free((void*)b.W, st);
            if (rc || rf || served) return rc ? rc : rf;
        }
    }
    if (wdt == 2 && few_tc_pays(a, rows_per_block, batch)) {
        bool served = false;
        if (const int rc = gemm_few_tc(a, EPI, batch, rows_per_block, st, &served)) return rc;
        if (served) return 0;
    }
    if (wdt == 2) return launch_few_t<uint16_t, EPI, true>(a, rows_per_block, st, batch);
    return launch_few_t<float, EPI, false>(a, rows_per_block, st, batch);
}

// ---------------------------------------------------------------- many rows, few columns, float32 weights (router logits)
// A 64 x 64 tile would leave all but one tile column empty and the grid a handful of blocks.  Here a warp owns SKM rows and SKN
// columns and walks K with a lane per element; the partial sums meet in a warp reduction.  Plain epilogue only.  Latency bounds it: a
// warp per column group instead of one for all columns, addresses that need no test (us, one warp per row group -> here: 2000 rows of
// 2048, 4 / 16 / 64 columns 14.5 / 25.2 / 84 -> 12.8 / 14.5 / 28.8; two rows per warp 16.4 / 22.7 / 45.2).  Where rows keep 16-byte
// boundaries a lane takes four k at once (18 columns 16.6 -> 10.3, 40 rows of 64 columns 8.0 -> 5.7): chains of the same length over other k.
constexpr int SKM = 4, SK_WARPS = 4;

// (One block per SM as the stated least: without it the compiler keeps to 96 registers and half the loads in flight, 14.4 -> 18.5 us at 18 columns.)
template <int SKN, bool VEC>
__global__ void __launch_bounds__(SK_WARPS * 32, 1) gemm_skinny_f32_kernel(GemmArgs a) {
    griddep_wait();
    griddep_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = (blockIdx.x * SK_WARPS + warp) * SKM, n0 = blockIdx.y * SKN;
    if (m0 >= a.M) return;
    const float* x[SKM];
    const float* w[SKN];                                  // rows and columns beyond the edge repeat the last one
#pragma unroll
    for (int i = 0; i < SKM; ++i) x[i] = a.A + (size_t)min(m0 + i, a.M - 1) * a.lda;
#pragma unroll
    for (int j = 0; j < SKN; ++j) w[j] = (const float*)a.W + (size_t)min(n0 + j, a.N - 1) * a.K;
    float acc[SKM][SKN];
#pragma unroll
    for (int i = 0; i < SKM; ++i)
#pragma unroll
        for (int j = 0; j < SKN; ++j) acc[i][j] = 0.f;
    if (VEC) {                                            // a lane takes four k at a time
#pragma unroll 2
        for (int k = lane * 4; k < a.K; k += 128) {
            float4 xv[SKM], wv[SKN];
#pragma unroll
            for (int i = 0; i < SKM; ++i) xv[i] = *(const float4*)(x[i] + k);
#pragma unroll
            for (int j = 0; j < SKN; ++j) wv[j] = *(const float4*)(w[j] + k);
#pragma unroll
            for (int i = 0; i < SKM; ++i)
#pragma unroll
                for (int j = 0; j < SKN; ++j) {
                    acc[i][j] = fmaf(xv[i].x, wv[j].x, acc[i][j]);
                    acc[i][j] = fmaf(xv[i].y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(xv[i].z, wv[j].z, acc[i][j]);
                    acc[i][j] = fmaf(xv[i].w, wv[j].w, acc[i][j]);
                }
        }
    } else {
#pragma unroll 4
    for (int k = lane; k < a.K; k += 32) {
        float xv[SKM], wv[SKN];
#pragma unroll
        for (int i = 0; i < SKM; ++i) xv[i] = x[i][k];
#pragma unroll
        for (int j = 0; j < SKN; ++j) wv[j] = w[j][k];
#pragma unroll
        for (int i = 0; i < SKM; ++i)
#pragma unroll
            for (int j = 0; j < SKN; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
    }
    }
#pragma unroll
    for (int i = 0; i < SKM; ++i)
#pragma unroll
        for (int j = 0; j < SKN; ++j) {
            const float v = warp_sum(acc[i][j]);
            if (lane == 0 && m0 + i < a.M && n0 + j < a.N) a.C[(size_t)(m0 + i) * a.ldc + n0 + j] = v;
        }
}

}  // namespace

extern "C" {

int pgk_gemm_rows_f32(const float* A, int lda, const int32_t* a_rows, const void* W, int wdt, long long w_group_stride,
                      float* C, int ldc, int M, int N, int K, const int32_t* group_off, int groups, int max_rows,
                      int epilogue, float scale, float cap, void* stream) {
    return pgk_gemm_groups_f32(A, lda, a_rows, W, wdt, w_group_stride, C, ldc, M, N, K, group_off, groups, max_rows, -1, epilogue, scale,
                               cap, stream);
}

int pgk_gemm_groups_f32(const float* A, int lda, const int32_t* a_rows, const void* W, int wdt, long long w_group_stride,
                        float* C, int ldc, int M, int N, int K, const int32_t* group_off, int groups, int max_rows, int total_rows,
                        int epilogue, float scale, float cap, void* stream) {
    const Rows16 dt(wdt);
    PGK_REQUIRE(wdt == 0 || (wdt & ~48) == 2, "gemm_rows_f32 failed: weights must be float32 (0) or bfloat16 (2), got %d", wdt);
    wdt = dt.wdt;
    PGK_REQUIRE(N > 0 && K > 0 && M >= 0, "gemm_rows_f32 failed: invalid shape M=%d N=%d K=%d", M, N, K);
    PGK_REQUIRE((epilogue >= 0 && epilogue <= 2) || (epilogue >= 6 && epilogue <= 9), "gemm_rows_f32 failed: unknown epilogue %d", epilogue);
    PGK_REQUIRE((epilogue != 1 && epilogue != 7) || N % 2 == 0, "gemm_rows_f32 failed: the gate/up epilogue needs an even N");
    const int G = group_off ? groups : 1;
    const int rows = group_off ? max_rows : M;
    if (rows <= 0 || G <= 0) return 0;
    GemmArgs a{A, a_rows, W, C, group_off, nullptr, w_group_stride, lda, ldc, M, N, K, scale, cap, nullptr, nullptr, nullptr, 0, 0, 0, 0, 0, dt.a16, dt.c16};
    cudaStream_t st = (cudaStream_t)stream;
    if (wdt == 0 && epilogue == 0 && !group_off && !a_rows && N <= 64) {        // router logits: few columns, float32 weights
        const int gx = (M + SK_WARPS * SKM - 1) / (SK_WARPS * SKM);
        const bool vec = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
        const auto kernel = N <= 4 ? (vec ? gemm_skinny_f32_kernel<4, true> : gemm_skinny_f32_kernel<4, false>)
                                   : (vec ? gemm_skinny_f32_kernel<8, true> : gemm_skinny_f32_kernel<8, false>);
        PGK_CUDA(launch_waiting(kernel, dim3(gx, N <= 4 ? 1 : (N + 7) / 8), dim3(SK_WARPS * 32), 0, st, a));
        return 0;
    }
    const int bound = group_off ? total_rows : M;
    if (epilogue == 0) return launch_many<0>(a, wdt, G, rows, st, bound);
    if (epilogue == 1) return launch_many<1>(a, wdt, G, rows, st, bound);
    if (epilogue == 6) return launch_many<6>(a, wdt, G, rows, st, bound);
    if (epilogue == 7) return launch_many<7>(a, wdt, G, rows, st, bound);
    if (epilogue == 8) return launch_many<8>(a, wdt, G, rows, st, bound);
    if (epilogue == 9) return launch_many<9>(a, wdt, G, rows, st, bound);
    return launch_many<2>(a, wdt, G, rows, st, bound);
}

/* Few rows (decoding): every block of `rows_per_block` (<= 8) consecutive rows shares one weight matrix; row_group
 * (NULL: matrix 0) names it per row and must be constant inside a block. */
int pgk_gemm_few_rows_f32(const float* A, int lda, const int32_t* a_rows, const void* W, int wdt, long long w_group_stride,
                          float* C, int ldc, int M, int N, int K, const int32_t* row_group, int rows_per_block,
                          int epilogue, float scale, float cap, void* stream) {
    PGK_REQUIRE(wdt == 0 || wdt == 2, "gemm_few_rows_f32 failed: weights must be float32 (0) or bfloat16 (2), got %d", wdt);
    PGK_REQUIRE(N > 0 && K > 0 && M >= 0, "gemm_few_rows_f32 failed: invalid shape M=%d N=%d K=%d", M, N, K);
    PGK_REQUIRE(rows_per_block >= 1 && rows_per_block <= RMAX, "gemm_few_rows_f32 failed: 1..%d rows per block", RMAX);
    PGK_REQUIRE((size_t)rows_per_block * K * 4 <= 200 * 1024, "gemm_few_rows_f32 failed: %d rows of K=%d do not fit shared memory", rows_per_block, K);
    PGK_REQUIRE((epilogue >= 0 && epilogue <= 2) || (epilogue >= 6 && epilogue <= 9), "gemm_few_rows_f32 failed: unknown epilogue %d", epilogue);
    PGK_REQUIRE((epilogue != 1 && epilogue != 7) || N % 2 == 0, "gemm_few_rows_f32 failed: the gate/up epilogue needs an even N");
    if (M == 0) return 0;
    GemmArgs a{A, a_rows, W, C, nullptr, row_group, w_group_stride, lda, ldc, M, N, K, scale, cap, nullptr, nullptr, nullptr, 0, 0, 0, 0, 0};
    cudaStream_t st = (cudaStream_t)stream;
    if (epilogue == 0) return launch_few<0>(a, wdt, rows_per_block, st);
    if (epilogue == 1) return launch_few<1>(a, wdt, rows_per_block, st);
    if (epilogue == 6) return launch_few<6>(a, wdt, rows_per_block, st);
    if (epilogue == 7) return launch_few<7>(a, wdt, rows_per_block, st);
    if (epilogue == 8) return launch_few<8>(a, wdt, rows_per_block, st);
    if (epilogue == 9) return launch_few<9>(a, wdt, rows_per_block, st);
    return launch_few<2>(a, wdt, rows_per_block, st);
}

/* The general form: `batch` independent products (A columns a_batch apart, matrices w_batch apart, C columns c_batch apart)
 * over the same M rows, every epilogue.  rows_per_block > 0 selects the few-row kernel (M <= 8 rows share one pass over the
 * weights), 0 the tiled kernel. */
int pgk_gemm_seq_f32(const float* A, int lda, long long a_batch, const void* W, int wdt, long long w_batch, float* C, int ldc,
                     long long c_batch, int M, int N, int K, int batch, int epilogue, float p0, float p1, const float* col_scale,
                     const void* aux, int aux_dtype, const int32_t* aux_rows, int aux_ld, int aux_off, int rows_per_block,
                     void* stream) {
    const Rows16 dt(wdt);
    PGK_REQUIRE(wdt == 0 || (wdt & ~48) == 2, "gemm_seq_f32 failed: weights must be float32 (0) or bfloat16 (2), got %d", wdt);
    PGK_REQUIRE(wdt < 16 || rows_per_block == 0, "gemm_seq_f32 failed: bfloat16 rows need the form of many rows");
    PGK_REQUIRE(!dt.c16 || epilogue != 4, "gemm_seq_f32 failed: the scaled-accumulate epilogue adds to float32 rows");
    wdt = dt.wdt;
    PGK_REQUIRE(N > 0 && K > 0 && M >= 0 && batch >= 1, "gemm_seq_f32 failed: invalid shape M=%d N=%d K=%d batch=%d", M, N, K, batch);
    PGK_REQUIRE(epilogue >= 0 && epilogue <= 10, "gemm_seq_f32 failed: unknown epilogue %d", epilogue);
    PGK_REQUIRE((epilogue != 1 && epilogue != 3 && epilogue != 7) || N % 2 == 0, "gemm_seq_f32 failed: a gate/up epilogue needs an even N");
    PGK_REQUIRE(epilogue != 4 || col_scale, "gemm_seq_f32 failed: the scaled-accumulate epilogue needs its column factors");
    PGK_REQUIRE(epilogue != 5 || (aux && aux_rows && (aux_dtype == 0 || aux_dtype == 2)), "gemm_seq_f32 failed: the gather epilogue needs its table and rows");
    PGK_REQUIRE(epilogue != 10 || (aux && aux_dtype == 0), "gemm_seq_f32 failed: the gate epilogue needs its float32 rows");
    PGK_REQUIRE(rows_per_block >= 0 && rows_per_block <= RMAX, "gemm_seq_f32 failed: 0..%d rows per block", RMAX);
    PGK_REQUIRE(rows_per_block == 0 || (size_t)rows_per_block * K * 4 <= 200 * 1024, "gemm_seq_f32 failed: %d rows of K=%d do not fit shared memory", rows_per_block, K);
    if (M == 0) return 0;
    GemmArgs a{A, nullptr, W, C, nullptr, nullptr, w_batch, lda, ldc, M, N, K, p0, p1, col_scale, aux, aux_rows, aux_ld, aux_off, aux_dtype, a_batch, c_batch, dt.a16, dt.c16};
    cudaStream_t st = (cudaStream_t)stream;
    if (rows_per_block > 0) {
        switch (epilogue) {
            case 0: return launch_few<0>(a, wdt, rows_per_block, st, batch);
            case 1: return launch_few<1>(a, wdt, rows_per_block, st, batch);
            case 2: return launch_few<2>(a, wdt, rows_per_block, st, batch);
            case 3: return launch_few<3>(a, wdt, rows_per_block, st, batch);
            case 4: return launch_few<4>(a, wdt, rows_per_block, st, batch);
            case 5: return launch_few<5>(a, wdt, rows_per_block, st, batch);
            case 6: return launch_few<6>(a, wdt, rows_per_block, st, batch);
            case 7: return launch_few<7>(a, wdt, rows_per_block, st, batch);
            case 8: return launch_few<8>(a, wdt, rows_per_block, st, batch);
            case 9: return launch_few<9>(a, wdt, rows_per_block, st, batch);
            default: return launch_few<10>(a, wdt, rows_per_block, st, batch);
        }
    }
    switch (epilogue) {
        case 0: return launch_many<0>(a, wdt, batch, M, st, M);
        case 1: return launch_many<1>(a, wdt, batch, M, st, M);
        case 2: return launch_many<2>(a, wdt, batch, M, st, M);
        case 3: return launch_many<3>(a, wdt, batch, M, st, M);
        case 4: return launch_many<4>(a, wdt, batch, M, st, M);
        case 5: return launch_many<5>(a, wdt, batch, M, st, M);
        case 6: return launch_many<6>(a, wdt, batch, M, st, M);
        case 7: return launch_many<7>(a, wdt, batch, M, st, M);
        case 8: return launch_many<8>(a, wdt, batch, M, st, M);
        case 9: return launch_many<9>(a, wdt, batch, M, st, M);
        default: return launch_many<10>(a, wdt, batch, M, st, M);
    }
}

}  // extern "C"
