// seq_linear_tc.cu -- linear attention over long prompts on tcgen05: the three passes of seq_recurrent.cu (what a chunk adds to the state, the
// states before every chunk, the chunks' outputs) over chunks of 128 tokens, one head of up to 128 x 128 each.
//
//   U_c = sum_s a^(n_c - 1 - s) k_s v_s^T        S_(c+1) = a^(n_c) S_c + U_c        o_t = a^(t + 1) S_c^T q_t + sum_{s <= t} (q_t . k_s a^(t - s)) v_s
//
// Everything is float32: an operand enters as three BF16 terms that together hold its 24 bits (rounded, so that what is left changes sign),
// a product as the six term products above 2^-27 of it, smallest first into one float32 accumulator (Q S and A V have one each: what is small would be cut off).
//
// What bounds it: the tensor cores' 48 MMAs per product of 128 x 128 x 128 (77 cycles each, 110 where both operands are in shared memory),
// the split of 128 x 128 operands by 256 threads (1500 cycles each), and rounds: 16 heads of 2000 tokens are 256 blocks on 148 SMs.  What
// follows from that:
//   * 128 tokens a chunk: a quarter of the states that chunks of 32 write and read back (17 MB for 16 heads of 2000 tokens: they stay in L2);
//   * queries and the masked, decayed scores are A operands in tensor memory; keys, values and states lie in shared memory as the copies
//     leave them, rows of 64 elements: the same image serves products along the elements (scores) and along the rows (the others);
//   * a block does one step after the other; two blocks do not fit an SM (3 x 64 KB of operands), so each step uses all eight warps.
// A chunk that holds an infinite or NaN operand (its terms would make NaN of what is infinite) is computed by plain float32 loops instead.
// Measured on B200 (us, chunks of 32 on the ordinary cores -> here): 16 heads of 128 x 128, 2000 tokens 264 -> 89, 800 99 -> 47, 200 64 -> 45; 64 x 64,
// 2000 tokens 79 -> 55.  Errors against float64: outputs 3.0e-7 -> 2.1e-7, states 2.5e-7 -> 1.2e-7 (with Q S and A V in one accumulator 8.8e-7).
#include "common.cuh"
#include "tc_common.cuh"
#include "../../include/pgk_b200.h"

namespace pgk {

namespace {

constexpr int LT = 128;                            // tokens per chunk
constexpr uint32_t L_CHUNK = LT * 128;             // 128 rows x 64 elements
constexpr uint32_t L_TERM = 2 * L_CHUNK, L_OPERAND = 3 * L_TERM;
constexpr size_t L_SMEM = 2 * L_OPERAND + 1024;
constexpr uint32_t L_Q = 0, L_A = 192, L_O = 384;  // TMEM columns: query terms, scores and then their terms, outputs

struct LinTcArgs {
    const float* proj; int ld, q_off, k_off, v_off;
    float* out; int ldo;
    float* state; const float* decay; const int4* seqs;
    int H, D, Dv, begin, end, chunks;              // tokens [begin, end) of every sequence, in at most `chunks` chunks
    float* ws;                                     // [sequences][chunks][H][D][Dv]
    int* err;
};

// x = hi + mid + lo of two neighbours; beyond 2^127 (and for infinities and NaN) `bad` is raised
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16x2(x0, x1);
    const float a = x0 - bf16lo(hi), b = x1 - bf16hi(hi);
    mid = pack_bf16x2(a, b);
    lo = pack_bf16x2(a - bf16lo(mid), b - bf16hi(mid));
}
__device__ __forceinline__ bool unfit(float x) { return !(fabsf(x) < 1.7e38f); }

// rows [0, rows) x columns [0, cols) of a float32 matrix, row r scaled by pw[p0 - r] where pw is given, as three terms at `dst`; the rest of
// 128 x width is zero.  Returns whether a value does not fit the terms.
__device__ __forceinline__ bool operand(uint32_t dst, const float* src, size_t ld, int rows, int cols, int width, const float* pw, int p0) {
    const int per = width >> 3;
    bool bad = false;
#pragma unroll 2
    for (int i = threadIdx.x; i < LT * per; i += 256) {
        const int r = i / per, c = (i - r * per) * 8;
        float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (r < rows && c < cols) {
            const float4 u = __ldcg((const float4*)(src + (size_t)r * ld + c)), w = __ldcg((const float4*)(src + (size_t)r * ld + c + 4));
            const float s = pw ? pw[p0 - r] : 1.f;
            x[0] = u.x * s; x[1] = u.y * s; x[2] = u.z * s; x[3] = u.w * s;
            x[4] = w.x * s; x[5] = w.y * s; x[6] = w.z * s; x[7] = w.w * s;
#pragma unroll
            for (int e = 0; e < 8; ++e) bad |= unfit(x[e]);
        }
        uint32_t t[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split2(x[2 * e], x[2 * e + 1], t[0][e], t[1][e], t[2][e]);
        const uint32_t at = dst + (uint32_t)(c >> 6) * L_CHUNK + (uint32_t)r * 128u + (uint32_t)((((c & 63) >> 3) ^ (r & 7)) << 4);
#pragma unroll
        for (int k = 0; k < 3; ++k)
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(at + (uint32_t)k * L_TERM), "r"(t[k][0]), "r"(t[k][1]), "r"(t[k][2]), "r"(t[k][3]) : "memory");
    }
    return bad;
}
// which terms meet, smallest product first
__device__ __forceinline__ int term_a(int i) { return (0x001012 >> (4 * i)) & 15; }      // lo mid hi mid hi hi
__device__ __forceinline__ int term_b(int i) { return (0x010210 >> (4 * i)) & 15; }      // hi mid lo hi mid hi

struct LinBlock { int c, h, nc, r0; int4 sq; float dec; };

__device__ __forceinline__ bool lin_block(const LinTcArgs& a, LinBlock& b) {
    b.sq = a.seqs[blockIdx.y];
    b.c = blockIdx.x;
    b.h = blockIdx.z;
    const int t0 = a.begin + b.c * LT, last = min(a.end, b.sq.y);
    if (t0 >= last) return false;
    b.nc = min(LT, last - t0);
    b.r0 = b.sq.x + t0;
    b.dec = a.decay[b.h];
    return true;
}

__global__ void __launch_bounds__(256, 1) linear_tc_update_kernel(const __grid_constant__ LinTcArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t done;
    __shared__ uint32_t tmem_base_s;
    __shared__ float pw[LT + 1];
    LinBlock b;
    griddep_wait();
    if (!lin_block(a, b)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t ks = (smem_u32(smem) + 1023u) & ~1023u, vs = ks + L_OPERAND;
    if (warp == 0) tmem_alloc(&tmem_base_s, 128);
    if (tid == 0) { mbar_init(&done, 1); mbar_fence_init(); }
    if (tid <= LT) pw[tid] = powf(b.dec, (float)tid);
    __syncthreads();
    griddep_launch();                              // tensor memory is held
    const float* kp = a.proj + (size_t)b.r0 * a.ld + a.k_off + (size_t)b.h * a.D;
    const float* vp = a.proj + (size_t)b.r0 * a.ld + a.v_off + (size_t)b.h * a.Dv;
    const int vw = (a.Dv + 63) & ~63, N = (a.Dv + 15) & ~15;
    bool bad = operand(ks, kp, a.ld, b.nc, a.D, 128, pw, b.nc - 1);
    bad |= operand(vs, vp, a.ld, b.nc, a.Dv, vw, nullptr, 0);
    fence_proxy_async();
    tc_fence_before();
    bad = __syncthreads_or(bad);
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    float* U = a.ws + (((size_t)blockIdx.y * a.chunks + b.c) * a.H + b.h) * a.D * a.Dv;
    if (!bad) {
        if (warp == 0 && elect_one()) {
            const uint32_t id = umma_idesc_bf16_mn(N);
            const int nk = (b.nc + 15) >> 4;
            uint32_t acc = 0;
#pragma unroll 1
            for (int i = 0; i < 6; ++i)
#pragma unroll 1
                for (int k = 0; k < nk; ++k, acc = 1)
                    umma_bf16(tmem, desc_mn_sw128(ks + (uint32_t)term_a(i) * L_TERM, L_CHUNK) + (uint64_t)(k * 128),
                              desc_mn_sw128(vs + (uint32_t)term_b(i) * L_TERM, L_CHUNK) + (uint64_t)(k * 128), id, acc);
            umma_commit(&done);
        }
        __syncwarp();
        bar_wait(a.err, smem_u32(&done), 0);
        __syncwarp();
        tc_fence_after();
        const int quad = warp & 3, half = warp >> 2, d = quad * 32 + lane;
#pragma unroll 1
        for (int c = half * 64; c < min(N, half * 64 + 64); c += 16) {
            float o[16];
            __syncwarp();
            tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c, o);
            if (d < a.D) {
#pragma unroll
                for (int e = 0; e < 16; e += 4)
                    if (c + e < a.Dv) __stcg((float4*)(U + (size_t)d * a.Dv + c + e), make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]));
            }
        }
        __syncwarp();
    } else {
        for (int i = tid; i < a.D * a.Dv; i += 256) {
            const int d = i / a.Dv, v = i - d * a.Dv;
            float u = 0.f;
            for (int s = 0; s < b.nc; ++s) u = fmaf(kp[(size_t)s * a.ld + d] * pw[b.nc - 1 - s], vp[(size_t)s * a.ld + v], u);
            __stcg(U + i, u);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 128);
}

// a thread per (sequence, head, four state elements): ws[c] <- the state before chunk c; the state after the last one to the slot's array
__global__ void __launch_bounds__(128) linear_tc_scan_kernel(const __grid_constant__ LinTcArgs a) {
    griddep_wait();
    griddep_launch();
    const size_t per = (size_t)a.D * a.Dv, e = ((size_t)blockIdx.x * 128 + threadIdx.x) * 4;
    const int h = blockIdx.y;
    const int4 sq = a.seqs[blockIdx.z];
    const int last = min(a.end, sq.y), n = (last - a.begin + LT - 1) / LT;
    if (e >= per || n <= 0) return;
    const float dec = a.decay[h], full = powf(dec, (float)LT), rest = powf(dec, (float)(last - a.begin - (n - 1) * LT));
    float* slot = a.state + ((size_t)sq.z * a.H + h) * per + e;
    float4 S = sq.w > 0 || a.begin > 0 ? *(const float4*)slot : make_float4(0.f, 0.f, 0.f, 0.f);
    float* u = a.ws + ((size_t)blockIdx.z * a.chunks * a.H + h) * per + e;
    const size_t step = (size_t)a.H * per;
    constexpr int B = 8;                           // loads in flight
    for (int c = 0; c < n; c += B) {
        float4 add[B];
#pragma unroll
        for (int i = 0; i < B; ++i) add[i] = c + i < n ? __ldcg((const float4*)(u + (size_t)(c + i) * step)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < B; ++i)
            if (c + i < n) {
                __stcg((float4*)(u + (size_t)(c + i) * step), S);
                const float f = c + i == n - 1 ? rest : full;
                S.x = fmaf(S.x, f, add[i].x); S.y = fmaf(S.y, f, add[i].y); S.z = fmaf(S.z, f, add[i].z); S.w = fmaf(S.w, f, add[i].w);
            }
    }
    *(float4*)slot = S;
}

__global__ void __launch_bounds__(256, 1) linear_tc_output_kernel(const __grid_constant__ LinTcArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t done[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ float pw[LT + 1];
    LinBlock b;
    griddep_wait();
    if (!lin_block(a, b)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t r1 = (smem_u32(smem) + 1023u) & ~1023u, r2 = r1 + L_OPERAND;
    if (warp == 0) tmem_alloc(&tmem_base_s, 512);
    if (tid == 0) { mbar_init(&done[0], 1); mbar_init(&done[1], 1); mbar_fence_init(); }
    if (tid <= LT) pw[tid] = powf(b.dec, (float)tid);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    griddep_launch();
    const float* qp = a.proj + (size_t)b.r0 * a.ld + a.q_off + (size_t)b.h * a.D;
    const float* kp = a.proj + (size_t)b.r0 * a.ld + a.k_off + (size_t)b.h * a.D;
    const float* vp = a.proj + (size_t)b.r0 * a.ld + a.v_off + (size_t)b.h * a.Dv;
    const float* Sc = a.ws + (((size_t)blockIdx.y * a.chunks + b.c) * a.H + b.h) * a.D * a.Dv;
    const int dw = (a.D + 63) & ~63, vw = (a.Dv + 63) & ~63, N = (a.Dv + 15) & ~15, nkd = (a.D + 15) >> 4, nks = (b.nc + 15) >> 4;
    const int quad = warp & 3, half = warp >> 2, t = quad * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);

    // ---- queries: row t, this warp's half of the elements
    bool bad = false;
#pragma unroll 1
    for (int c = half * 64; c < min(dw, half * 64 + 64); c += 32) {
        float x[32];
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
            const float4 w = t < b.nc && c + e < a.D ? __ldcg((const float4*)(qp + (size_t)t * a.ld + c + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
            x[e] = w.x; x[e + 1] = w.y; x[e + 2] = w.z; x[e + 3] = w.w;
        }
        uint32_t hi[16], mid[16], lo[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            bad |= unfit(x[2 * e]) || unfit(x[2 * e + 1]);
            split2(x[2 * e], x[2 * e + 1], hi[e], mid[e], lo[e]);
        }
        __syncwarp();
        tmem_st16u(lanes + L_Q + (uint32_t)(c / 2), hi);
        tmem_st16u(lanes + L_Q + 64u + (uint32_t)(c / 2), mid);
        tmem_st16u(lanes + L_Q + 128u + (uint32_t)(c / 2), lo);
    }
    tmem_st_wait();
    bad |= operand(r1, kp, a.ld, b.nc, a.D, dw, nullptr, 0);
    bad |= operand(r2, Sc, a.Dv, a.D, a.Dv, vw, nullptr, 0);
    fence_proxy_async();
    tc_fence_before();
    bad = __syncthreads_or(bad);
    tc_fence_after();
    if (!bad) {
        // ---- scores Q K^T and what the state before the chunk gives, Q S
        if (warp == 0 && elect_one()) {
            const uint32_t id_a = umma_idesc_bf16(LT), id_o = umma_idesc_bf16(N) | (1u << 16);
            uint32_t acc = 0;
#pragma unroll 1
            for (int i = 0; i < 6; ++i)
#pragma unroll 1
                for (int k = 0; k < nkd; ++k, acc = 1)
                    umma_bf16_ta(tmem + L_A, tmem + L_Q + (uint32_t)(term_a(i) * 64 + k * 8),
                                 desc_sw128(r1 + (uint32_t)term_b(i) * L_TERM + (uint32_t)(k >> 2) * L_CHUNK) + (uint64_t)((k & 3) * 2), id_a, acc);
            umma_commit(&done[0]);
            acc = 0;
#pragma unroll 1
            for (int i = 0; i < 6; ++i)
#pragma unroll 1
                for (int k = 0; k < nkd; ++k, acc = 1)
                    umma_bf16_ta(tmem + L_O, tmem + L_Q + (uint32_t)(term_a(i) * 64 + k * 8),
                                 desc_mn_sw128(r2 + (uint32_t)term_b(i) * L_TERM, L_CHUNK) + (uint64_t)(k * 128), id_o, acc);
            umma_commit(&done[1]);
        }
        __syncwarp();
        bar_wait(a.err, smem_u32(&done[0]), 0);
        __syncwarp();
        tc_fence_after();
        // ---- the scores masked and decayed, as A operand; the values meanwhile where the keys were
        float x[64];
#pragma unroll
        for (int c = 0; c < 64; c += 16) tmem_ld16_async(lanes + L_A + (uint32_t)(half * 64 + c), *(float (*)[16])(x + c));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int c = 0; c < 64; c += 16) tmem_pass(*(float (*)[16])(x + c));
        asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");              // the row's other half has read its scores, too
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
            uint32_t hi[16], mid[16], lo[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                float y[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int s = half * 64 + c + 2 * e + u;
                    y[u] = s <= t ? x[c + 2 * e + u] * pw[max(t - s, 0)] : 0.f;
                    bad |= unfit(y[u]);
                }
                split2(y[0], y[1], hi[e], mid[e], lo[e]);
            }
            const uint32_t col = (uint32_t)(half * 32 + c / 2);
            __syncwarp();
            tmem_st16u(lanes + L_A + col, hi);
            tmem_st16u(lanes + L_A + 64u + col, mid);
            tmem_st16u(lanes + L_A + 128u + col, lo);
        }
        tmem_st_wait();
        bad |= operand(r1, vp, a.ld, b.nc, a.Dv, vw, nullptr, 0);
        bar_wait(a.err, smem_u32(&done[1]), 0);
        __syncwarp();
        tc_fence_after();
        fence_proxy_async();
        tc_fence_before();
        bad = __syncthreads_or(bad);
        tc_fence_after();
    }
    if (!bad) {
        if (warp == 0 && elect_one()) {
            const uint32_t id_o = umma_idesc_bf16(N) | (1u << 16);
#pragma unroll 1
            for (int i = 0; i < 6; ++i)
#pragma unroll 1
                for (int k = 0; k < nks; ++k)                     // where the queries were: added to Q S, small terms would be cut off
                    umma_bf16_ta(tmem + L_Q, tmem + L_A + (uint32_t)(term_a(i) * 64 + k * 8),
                                 desc_mn_sw128(r1 + (uint32_t)term_b(i) * L_TERM, L_CHUNK) + (uint64_t)(k * 128), id_o, (i | k) ? 1u : 0u);
            umma_commit(&done[0]);
        }
        __syncwarp();
        bar_wait(a.err, smem_u32(&done[0]), 1);
        __syncwarp();
        tc_fence_after();
        float* out = a.out + (size_t)(b.r0 + t) * a.ldo + (size_t)b.h * a.Dv;
#pragma unroll 1
        for (int c = half * 64; c < min(N, half * 64 + 64); c += 16) {
            float o[16], x[16];
            __syncwarp();
            tmem_ld16(lanes + L_O + (uint32_t)c, x);
            tmem_ld16(lanes + L_Q + (uint32_t)c, o);
            if (t < b.nc) {
#pragma unroll
                for (int e = 0; e < 16; ++e) o[e] = fmaf(x[e], pw[t + 1], o[e]);
#pragma unroll
                for (int e = 0; e < 16; e += 4)
                    if (c + e < a.Dv) *(float4*)(out + c + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
            }
        }
        __syncwarp();
    } else {
        float* A = (float*)(smem + (r1 - smem_u32(smem)));        // [128][128]
        __syncthreads();
        for (int i = tid; i < LT * LT; i += 256) {
            const int r = i >> 7, s = i & 127;
            float z = 0.f;
            if (r < b.nc && s <= r) {
                for (int d = 0; d < a.D; ++d) z = fmaf(qp[(size_t)r * a.ld + d], kp[(size_t)s * a.ld + d], z);
                z *= pw[r - s];
            }
            A[i] = z;
        }
        __syncthreads();
        for (int i = tid; i < b.nc * a.Dv; i += 256) {
            const int r = i / a.Dv, v = i - r * a.Dv;
            float z = 0.f;
            for (int d = 0; d < a.D; ++d) z = fmaf(qp[(size_t)r * a.ld + d], __ldcg(Sc + (size_t)d * a.Dv + v), z);
            z *= pw[r + 1];
            for (int s = 0; s <= r; ++s) z = fmaf(A[r * LT + s], vp[(size_t)s * a.ld + v], z);
            a.out[(size_t)(b.r0 + r) * a.ldo + (size_t)b.h * a.Dv + v] = z;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace

// Heads of up to 128 x 128 in multiples of eight whose rows keep 16-byte boundaries.
bool linear_tc_ok(const float* proj, int ld, int q_off, int k_off, int v_off, const float* out, int ldo, const float* state, int D, int Dv, const float* ws) {
    return D <= 128 && Dv <= 128 && D % 8 == 0 && Dv % 8 == 0 && (ld | q_off | k_off | v_off | ldo) % 4 == 0 &&
           (((uintptr_t)proj | (uintptr_t)out | (uintptr_t)state | (uintptr_t)ws) & 15) == 0;
}

// tokens [begin, end) of every sequence; ws holds a state per 128 of them
int linear_tc(const float* proj, int ld, int q_off, int k_off, int v_off, float* out, int ldo, float* state, const float* decay, const int32_t* seqs, int n_seqs,
              int H, int D, int Dv, int begin, int end, float* ws, cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        PGK_CUDA(cudaFuncSetAttribute(linear_tc_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L_SMEM));
        PGK_CUDA(cudaFuncSetAttribute(linear_tc_output_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L_SMEM));
        configured = true;
    }
    int* err = wait_word(kWaitLinear);
    PGK_REQUIRE(err, "seq_linear_attention_chunks failed: no pinned host memory");
    LinTcArgs a{proj, ld, q_off, k_off, v_off, out, ldo, state, decay, (const int4*)seqs, H, D, Dv, begin, end, (end - begin + LT - 1) / LT, ws, err};
    const dim3 grid(a.chunks, n_seqs, H);
    PGK_CUDA(launch_waiting(linear_tc_update_kernel, grid, dim3(256), L_SMEM, st, a));
    PGK_CUDA(launch_waiting(linear_tc_scan_kernel, dim3((unsigned)((D * Dv + 511) / 512), H, n_seqs), dim3(128), 0, st, a));
    PGK_CUDA(launch_waiting(linear_tc_output_kernel, grid, dim3(256), L_SMEM, st, a));
    return 0;
}

}  // namespace pgk
