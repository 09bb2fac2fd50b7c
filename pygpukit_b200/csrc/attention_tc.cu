// attention_tc.cu -- attention of many query rows over the fixed BF16 cache (prompts) on tcgen05; the same mathematics as
// sdpa_decode_kernel (attention.cu): exact products of BF16 queries and keys summed in float32, float32 softmax, float32 weights.
//
//   out[h, t, :] = softmax_j( Q[h,t,:] . K[kv(h), j, :] * scale ) V[kv(h), j, :],   j < context_len - q_len + t + 1,   128 elements a head
//
// What bounds it: a block of 128 rows (query, head) and a tile of 128 keys cost the tensor cores 616 cycles for the scores and 3 x 616 for
// the values, the ordinary units 128 x 14 instructions a row.  What follows from that:
//   * A operands sit in tensor memory, where an MMA of 128 columns takes 77 cycles (110 with A in shared memory): the queries all along,
//     the weights written there by the warps that form them, which also saves their way through shared memory;
//   * a weight is float32: three BF16 terms, cut off and not rounded, that together hold its 24 bits, enter the product one after the
//     other.  The second and third are never zero (2^-126 stands in), so that an infinite value gives infinity, as in float32;
//   * a masked key's weight is zero, and zero times an infinite or NaN value is NaN: rows that came out NaN in a range with keys behind
//     their own last one are summed again over their own keys, in float32 on the ordinary units;
//   * the scores of tile i + 1 are multiplied while tile i's weights are formed; the first two terms lie where its scores were;
//   * eight warps, a lane a row, two warps a row (64 keys each); a row's reference moves only when its maximum has grown by LAZY (log2
//     units): the outputs in tensor memory are rescaled then;
//   * rows are QB queries by HB heads of one KV head, so that keys and values are read once per group; blocks with the longest rows first;
//     few blocks share a row's keys and leave records that a second kernel folds;
//   * the tensor maps end at the context, so that rows behind it arrive as zeros.
// Measured on B200 (us, sdpa_decode_kernel -> here), 32 / 8 heads: 512 queries over 512 keys 328 -> 16.5, over 8192 4477 -> 125; 64 over 512
// 52 -> 15.6, over 8192 658 -> 39; 16 over 512 29 -> 14.5.  Errors against float64 are the same (BF16 outputs).
#include "common.cuh"
#include "tc_common.cuh"
#include "tma.cuh"
#include "../../include/pgk_b200.h"

namespace pgk {

namespace {

constexpr int M_ROWS = 128, M_KEYS = 128, M_D = 128;
constexpr int M_SOFT = 8;                          // warps; then one for the copies, one for the MMAs
constexpr int M_THREADS = (M_SOFT + 2) * 32;
constexpr int M_STAGES = 2;                        // tiles of K, tiles of V
constexpr uint32_t M_TILE = M_KEYS * M_D * 2;      // 32 KB, two chunks of 64 elements
constexpr size_t M_SMEM = 2 * M_STAGES * M_TILE + 1024;
constexpr uint32_t M_O = 0, M_Q = 128, M_S = 192, M_LO = 448;      // TMEM columns: outputs, queries, two tiles of scores, third terms
constexpr float M_LAZY = 8.f;

struct PromptAttnParams {
    const uint16_t* Q; const uint16_t* K; const uint16_t* V; uint16_t* out;
    int max_seq;
    long q_sh, q_st, o_sh, o_st;
    int hq, n_kv, q_len, context_len;
    int HB, QB, hsplit, splits;
    int t0, t1;                                    // the launch's queries
    float scale_log2;
    float* ws;                                     // splits > 1: records (m, l, -, -, o[128]) [query - t0][head][split]
    int* err;
};

__device__ __forceinline__ bool all_wait(int* err, uint32_t bar, uint32_t parity) {
    const bool ok = bar_wait(err, bar, parity);
    return __all_sync(0xffffffffu, ok);
}
// the upper halves of two words: two float32 values cut off to BF16
__device__ __forceinline__ uint32_t cut2(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }

// 16 elements of one row's sum over keys [from, to), by a warp: q, k and v are the row's query and the first rows of its keys and values
__device__ __forceinline__ void sum_again(const uint16_t* q, const uint16_t* k, const uint16_t* v, int from, int to, float scale_log2, float neg, float (&o)[16]) {
#pragma unroll
    for (int e = 0; e < 16; ++e) o[e] = 0.f;
#pragma unroll 1
    for (int j = from + (int)(threadIdx.x & 31); j < to; j += 32) {
        float s = 0.f;
#pragma unroll 1
        for (int i = 0; i < M_D; i += 8) {
            const uint4 a = ld_act16(q + i), b = ld_act16(k + (size_t)j * M_D + i);
            s = fmaf(bf16lo(a.x), bf16lo(b.x), s); s = fmaf(bf16hi(a.x), bf16hi(b.x), s);
            s = fmaf(bf16lo(a.y), bf16lo(b.y), s); s = fmaf(bf16hi(a.y), bf16hi(b.y), s);
            s = fmaf(bf16lo(a.z), bf16lo(b.z), s); s = fmaf(bf16hi(a.z), bf16hi(b.z), s);
            s = fmaf(bf16lo(a.w), bf16lo(b.w), s); s = fmaf(bf16hi(a.w), bf16hi(b.w), s);
        }
        const float w = ex2(fmaf(s, scale_log2, neg));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 x = ld_act16(v + (size_t)j * M_D + 8 * i);
            o[8 * i] = fmaf(w, bf16lo(x.x), o[8 * i]); o[8 * i + 1] = fmaf(w, bf16hi(x.x), o[8 * i + 1]);
            o[8 * i + 2] = fmaf(w, bf16lo(x.y), o[8 * i + 2]); o[8 * i + 3] = fmaf(w, bf16hi(x.y), o[8 * i + 3]);
            o[8 * i + 4] = fmaf(w, bf16lo(x.z), o[8 * i + 4]); o[8 * i + 5] = fmaf(w, bf16hi(x.z), o[8 * i + 5]);
            o[8 * i + 6] = fmaf(w, bf16lo(x.w), o[8 * i + 6]); o[8 * i + 7] = fmaf(w, bf16hi(x.w), o[8 * i + 7]);
        }
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) o[e] = warp_sum(o[e]);
}

__global__ void __launch_bounds__(M_THREADS, 1)
sdpa_prompt_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, const __grid_constant__ PromptAttnParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t kfull[M_STAGES], kempty[M_STAGES], vfull[M_STAGES], vempty[M_STAGES], sfull[2], pready, pvdone;
    __shared__ uint32_t tmem_base_s;
    __shared__ float wmax[2][2][M_ROWS];                 // by turns: a warp may be a tile ahead of its partner's look
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t ks = (smem_u32(smem) + 1023u) & ~1023u, vs = ks + M_STAGES * M_TILE;
    int* const err = p.err;

    if (warp == M_SOFT + 1) tmem_alloc(&tmem_base_s, 512);
    if (tid == 0) {
        for (int s = 0; s < M_STAGES; ++s) { mbar_init(&kfull[s], 1); mbar_init(&kempty[s], 1); mbar_init(&vfull[s], 1); mbar_init(&vempty[s], 1); }
        mbar_init(&sfull[0], 1); mbar_init(&sfull[1], 1);
        mbar_init(&pready, M_SOFT); mbar_init(&pvdone, 1);
        mbar_fence_init();
        asm volatile("prefetch.tensormap [%0];" :: "l"(&kmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&vmap) : "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    griddep_wait();
    griddep_launch();

    const int rep = p.hq / p.n_kv, g = blockIdx.y / p.hsplit, part = blockIdx.y - g * p.hsplit, h0 = part * p.HB, nh = min(p.HB, rep - h0);
    const int q0 = p.t0 + (int)(gridDim.x - 1 - blockIdx.x) * p.QB, nq = min(p.QB, p.t1 - q0), pos0 = p.context_len - p.q_len + q0;
    const int ntile = (pos0 + nq - 1) / M_KEYS + 1, per = (ntile + p.splits - 1) / p.splits;
    const int tbeg = (int)blockIdx.z * per, n = max(0, min(ntile, tbeg + per) - tbeg);
    // row r: head r / QB, query r % QB
    const int quad = warp & 3, half = (warp >> 2) & 1, row = quad * 32 + lane, rh = row / p.QB, rq = row - rh * p.QB;
    const bool live = rh < nh && rq < nq;

    if (warp < 4) {                                // queries to tensor memory
        const uint16_t* src = p.Q + (size_t)(g * rep + h0 + rh) * p.q_sh + (size_t)(q0 + rq) * p.q_st;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            uint32_t v[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 w = live ? ld_act16(src + c * 32 + i * 8) : make_uint4(0, 0, 0, 0);
                v[4 * i] = w.x; v[4 * i + 1] = w.y; v[4 * i + 2] = w.z; v[4 * i + 3] = w.w;
            }
            __syncwarp();
            tmem_st16u(tmem + ((uint32_t)(quad * 32) << 16) + M_Q + (uint32_t)c * 16u, v);
        }
        tmem_st_wait();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp == M_SOFT) {
        // ---------------- copies
        if (elect_one()) {
            bool ok = true;
            auto load = [&](const CUtensorMap* map, uint32_t base, uint64_t* full, uint64_t* empty, int i) {
                const uint32_t s = (uint32_t)i % M_STAGES, bar = smem_u32(full) + 8u * s, at = base + s * M_TILE;
                ok = ok && bar_wait(err, smem_u32(empty) + 8u * s, (((uint32_t)i / M_STAGES) & 1u) ^ 1u);
                if (!ok) return;
                mbar_expect_tx(bar, M_TILE);
                tma_load_3d(at, map, 0, (tbeg + i) * M_KEYS, g, bar);
                tma_load_3d(at + M_TILE / 2, map, 64, (tbeg + i) * M_KEYS, g, bar);
            };
            int nk = 0, nv = 0;
            for (int i = 0; ok && i < n; ++i) {
                load(&kmap, ks, kfull, kempty, i);
                nk += ok;
                load(&vmap, vs, vfull, vempty, i);
                nv += ok;
            }
            for (int j = max(0, nk - M_STAGES); j < nk; ++j)      // whoever gave up: do not leave with copies in flight
                bar_wait(err, smem_u32(kfull) + 8u * (uint32_t)(j % M_STAGES), (uint32_t)((j / M_STAGES) & 1));
            for (int j = max(0, nv - M_STAGES); j < nv; ++j)
                bar_wait(err, smem_u32(vfull) + 8u * (uint32_t)(j % M_STAGES), (uint32_t)((j / M_STAGES) & 1));
        }
        __syncwarp();
    } else if (warp == M_SOFT + 1) {
        // ---------------- MMAs
        constexpr uint32_t id_s = umma_idesc_bf16(M_KEYS), id_o = umma_idesc_bf16(M_D) | (1u << 16);      // values: the elements are contiguous
        bool ok = true;
        auto scores = [&](int i) {                 // S = Q . K^T of tile i, where the weights of tile i - 2 were
            const uint32_t s = (uint32_t)i % M_STAGES;
            ok = ok && all_wait(err, smem_u32(kfull) + 8u * s, ((uint32_t)i / M_STAGES) & 1u);
            if (!ok) return;
            if (elect_one()) {
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < M_D / 16; ++k)
                    umma_bf16_ta(tmem + M_S + (uint32_t)(i & 1) * 128u, tmem + M_Q + (uint32_t)k * 8u,
                                 desc_sw128(ks + s * M_TILE + (uint32_t)(k >> 2) * (M_TILE / 2)) + (uint64_t)((k & 3) * 2), id_s, k ? 1u : 0u);
                umma_commit(&sfull[i & 1]);
                umma_commit(&kempty[s]);
            }
            __syncwarp();
        };
        if (n > 0) scores(0);
        for (int i = 0; ok && i < n; ++i) {
            const uint32_t s = (uint32_t)i % M_STAGES;
            if (i > 0) ok = all_wait(err, smem_u32(&pvdone), (uint32_t)((i - 1) & 1));
            if (ok && i + 1 < n) scores(i + 1);
            ok = ok && all_wait(err, lane & 1 ? smem_u32(vfull) + 8u * s : smem_u32(&pready), lane & 1 ? ((uint32_t)i / M_STAGES) & 1u : (uint32_t)(i & 1));
            if (!ok) break;
            if (elect_one()) {
                tc_fence_after();
                const uint32_t at = tmem + M_S + (uint32_t)(i & 1) * 128u;
#pragma unroll 1
                for (int k = 0; k < M_KEYS / 16; ++k) {           // 16 keys: 2048 bytes of V; the smallest terms first
                    const uint64_t dv = desc_mn_sw128(vs + s * M_TILE, M_TILE / 2) + (uint64_t)(k * 128);
                    umma_bf16_ta(tmem + M_O, tmem + M_LO + (uint32_t)k * 8u, dv, id_o, (i | k) ? 1u : 0u);
                    umma_bf16_ta(tmem + M_O, at + 64u + (uint32_t)k * 8u, dv, id_o, 1u);
                    umma_bf16_ta(tmem + M_O, at + (uint32_t)k * 8u, dv, id_o, 1u);
                }
                umma_commit(&pvdone);
                umma_commit(&vempty[s]);
            }
            __syncwarp();
        }
    } else {
        // ---------------- weights
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const int limit = live ? pos0 + rq : -1;                  // the last key that the row sees
        float m = -INFINITY, neg = 0.f, l = 0.f;
        bool ok = true;
        for (int i = 0; i < n; ++i) {
            const uint32_t at = lanes + M_S + (uint32_t)(i & 1) * 128u;
            const int j0 = (tbeg + i) * M_KEYS + half * 64;
            ok = ok && all_wait(err, smem_u32(sfull) + 8u * (uint32_t)(i & 1), (uint32_t)((i >> 1) & 1));
            __syncwarp();
            tc_fence_after();
            float s[64];
#pragma unroll
            for (int c = 0; c < 64; c += 16) tmem_ld16_async(at + (uint32_t)(half * 64 + c), *(float (*)[16])(s + c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 64; c += 16) tmem_pass(*(float (*)[16])(s + c));
            float top = -INFINITY;
            if (j0 + 63 <= pos0) {                                // every row sees every key (rows that nobody has: anything)
#pragma unroll
                for (int c = 0; c < 64; ++c) { s[c] *= p.scale_log2; top = fmaxf(top, s[c]); }
            } else {
#pragma unroll
                for (int c = 0; c < 64; ++c) {
                    s[c] = j0 + c <= limit ? s[c] * p.scale_log2 : -INFINITY;
                    top = fmaxf(top, s[c]);
                }
            }
            wmax[i & 1][half][row] = top;
            __syncwarp();
            asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");          // the row's two warps; both have read their scores
            top = fmaxf(top, wmax[i & 1][half ^ 1][row]);
            bool waited = i == 0;
            const bool up = top > m + M_LAZY;                     // (also the first finite maximum)
            if (__any_sync(0xffffffffu, up)) {                    // the same in both warps: each has half of the outputs
                const float f = !up ? 1.f : (m == -INFINITY ? 0.f : exp2f(m - top));
                if (up) { m = top; neg = -top; }
                l *= f;
                if (i > 0) {
                    ok = ok && all_wait(err, smem_u32(&pvdone), (uint32_t)((i - 1) & 1));
                    __syncwarp();
                    waited = true;
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 64; c += 16) {
                        float o[16];
                        const uint32_t to = lanes + M_O + (uint32_t)(half * 64 + c);
                        tmem_ld16(to, o);
#pragma unroll
                        for (int e = 0; e < 16; ++e) o[e] *= f;
                        tmem_st16(to, o);
                    }
                }
            }
            const float tiny = 1.17549435e-38f;
#pragma unroll
            for (int c = 0; c < 64; c += 32) {                    // 32 keys: 16 columns of each term
                uint32_t hi[16], mid[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    float a = ex2(s[c + 2 * e] + neg), b = ex2(s[c + 2 * e + 1] + neg);
                    l += a + b;
                    hi[e] = cut2(a, b);
                    a = fmaxf(a - bf16lo(hi[e]), tiny);
                    b = fmaxf(b - bf16hi(hi[e]), tiny);
                    mid[e] = cut2(a, b);
                    lo[e] = cut2(fmaxf(a - bf16lo(mid[e]), tiny), fmaxf(b - bf16hi(mid[e]), tiny));
                }
                const uint32_t col = (uint32_t)(half * 32 + c / 2);
                __syncwarp();
                tmem_st16u(at + col, hi);
                tmem_st16u(at + 64u + col, mid);
                if (!waited) {                                    // the last tile's product has read the third terms
                    ok = ok && all_wait(err, smem_u32(&pvdone), (uint32_t)((i - 1) & 1));
                    __syncwarp();
                    tc_fence_after();
                    waited = true;
                }
                tmem_st16u(lanes + M_LO + col, lo);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&pready);
        }
        // ---------------- outputs
        if (n > 0) all_wait(err, smem_u32(&pvdone), (uint32_t)((n - 1) & 1));
        __syncwarp();
        tc_fence_after();
        asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");              // the last tile's maxima are read
        wmax[0][half][row] = l;
        __syncwarp();
        asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");
        l = wmax[0][0][row] + wmax[0][1][row];
        const int h = g * rep + h0 + rh, t = q0 + rq;
        const float inv = p.splits > 1 ? 1.f : (l > 0.f || l != l ? 1.f / l : 0.f);
        float* rec = p.splits > 1 ? p.ws + (((size_t)(t - p.t0) * p.hq + h) * p.splits + blockIdx.z) * (M_D + 4) : nullptr;
        if (rec && live && half == 0) { rec[0] = m; rec[1] = l; }
        const int from = tbeg * M_KEYS, end = min(p.context_len, (tbeg + n) * M_KEYS);
        const size_t kv = (size_t)g * p.max_seq * M_D;
#pragma unroll 1
        for (int c = 0; c < 64; c += 16) {
            float o[16];
            __syncwarp();
            if (n > 0) tmem_ld16(lanes + M_O + (uint32_t)(half * 64 + c), o);
            else {
#pragma unroll
                for (int e = 0; e < 16; ++e) o[e] = 0.f;
            }
            bool nan = false;
#pragma unroll
            for (int e = 0; e < 16; ++e) nan |= o[e] != o[e];
            uint32_t rows = __ballot_sync(0xffffffffu, live && nan && limit + 1 < end);
#pragma unroll 1
            while (rows) {
                const int s = __ffs(rows) - 1, r = quad * 32 + s, sh = r / p.QB, sq = r - sh * p.QB;
                rows &= rows - 1;
                float x[16];
                sum_again(p.Q + (size_t)(g * rep + h0 + sh) * p.q_sh + (size_t)(q0 + sq) * p.q_st, p.K + kv, p.V + kv + half * 64 + c, from, pos0 + sq + 1,
                          p.scale_log2, __shfl_sync(0xffffffffu, neg, s), x);
#pragma unroll
                for (int e = 0; e < 16; ++e) o[e] = lane == s ? x[e] : o[e];
            }
            if (live && rec) {
#pragma unroll
                for (int e = 0; e < 16; e += 4) *(float4*)(rec + 4 + half * 64 + c + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
            } else if (live) {
                uint32_t y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = pack_bf16x2(o[2 * e] * inv, o[2 * e + 1] * inv);
                uint16_t* dst = p.out + (size_t)h * p.o_sh + (size_t)t * p.o_st + half * 64 + c;
                *(uint4*)dst = make_uint4(y[0], y[1], y[2], y[3]);
                *(uint4*)(dst + 8) = make_uint4(y[4], y[5], y[6], y[7]);
            }
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == M_SOFT + 1) tmem_dealloc(tmem, 512);
}

// a warp per (query, head): the records of its key ranges in their order.  A range in which the row sees no key has m = -inf and l = 0; one
// whose scores are all NaN has m = -inf and l = NaN, and the row becomes NaN as it does in one range.
__global__ void __launch_bounds__(256) sdpa_prompt_fold_kernel(const __grid_constant__ PromptAttnParams p) {
    griddep_wait();
    griddep_launch();
    const int lane = threadIdx.x & 31, i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= (p.t1 - p.t0) * p.hq) return;
    const int t = p.t0 + i / p.hq, h = i % p.hq;
    const float* rec = p.ws + (size_t)i * p.splits * (M_D + 4);
    float M = -INFINITY, L = 0.f;
    for (int s = 0; s < p.splits; ++s) M = fmaxf(M, __ldcg(rec + s * (M_D + 4)));
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < p.splits; ++s) {
        const float* r = rec + s * (M_D + 4);
        const float m = __ldcg(r), l = __ldcg(r + 1), w = m == -INFINITY ? l - l : exp2f(m - M);
        const float4 v = __ldcg((const float4*)(r + 4 + lane * 4));
        L = fmaf(w, l, L);
        o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w);
    }
    const float inv = L > 0.f || L != L ? 1.f / L : 0.f;
    *(uint2*)(p.out + (size_t)h * p.o_sh + (size_t)t * p.o_st + lane * 4) = make_uint2(pack_bf16x2(o.x * inv, o.y * inv), pack_bf16x2(o.z * inv, o.w * inv));
}

}  // namespace

// What the kernel takes: BF16 heads of 128 whose rows, copied 16 bytes at a time, keep that alignment, and a context that the host knows.
bool sdpa_prompt_ok(const void* Q, const void* K, const void* V, const void* out, int hq, int n_kv, int q_len, int max_seq, int context_len, long q_sh, long q_st,
                    long o_sh, long o_st) {
    const long strides = q_sh | q_st | o_sh | o_st;
    const uintptr_t ptrs = (uintptr_t)Q | (uintptr_t)K | (uintptr_t)V | (uintptr_t)out;
    return strides % 8 == 0 && ptrs % 16 == 0 && context_len >= q_len && context_len <= max_seq && (long long)q_len * hq < (1ll << 30) && n_kv <= 4096 &&
           hq / n_kv <= 128 && tma_encode_fn() != nullptr;
}

struct PromptPlan { int HB, QB, hsplit, splits, ranges, rows; };       // ranges: the fewest splits that the sums allow

// Key ranges until the blocks fill the SMs, four tiles (a record costs what half a tile does) at least in each and 64 at most: a range's
// sums stay in the tensor cores' accumulators, which cut off (over 32768 keys in one range the error against float64 was 1.665e-3, in
// ranges of 8192 it is that of the float32 kernel, 1.661e-3: BF16 outputs).  Records take up to kRecordBytes (512 queries of 64 heads over
// 131072 keys would have 277 MB); more queries go one launch after the other, each with blocks for all SMs.
constexpr size_t kRecordBytes = 64ull << 20;
static PromptPlan prompt_plan(int hq, int n_kv, int q_len, int context_len, int sms) {
    PromptPlan p;
    const int rep = hq / n_kv;
    p.HB = rep < 16 ? rep : 16;
    p.QB = M_ROWS / p.HB;
    p.hsplit = (rep + p.HB - 1) / p.HB;
    const long long blocks = (long long)((q_len + p.QB - 1) / p.QB) * n_kv * p.hsplit;
    const int ntile = (context_len + M_KEYS - 1) / M_KEYS;
    p.splits = (int)(sms / blocks);
    if (p.splits > ntile / 4) p.splits = ntile / 4;
    p.ranges = (ntile + 63) / 64;
    if (p.splits < p.ranges) p.splits = p.ranges;
    p.rows = q_len;
    if (p.splits > 1) {
        const size_t fit = kRecordBytes / ((size_t)hq * p.splits * (M_D + 4) * sizeof(float)) / p.QB * p.QB;
        if (fit < (size_t)q_len) p.rows = fit > (size_t)p.QB ? (int)fit : (p.QB < q_len ? p.QB : q_len);
    }
    return p;
}

// `no_room`: nothing was done, the records of the ranges that the sums need do not fit the device
int sdpa_prompt(const void* Q, const void* K, const void* V, void* out, int hq, int n_kv, int q_len, int max_seq, int context_len, float scale_log2, long q_sh,
                long q_st, long o_sh, long o_st, cudaStream_t st, bool* no_room) {
    static bool configured = false;
    if (!configured) {
        PGK_CUDA(cudaFuncSetAttribute(sdpa_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M_SMEM));
        configured = true;
    }
    PromptAttnParams p = {};
    p.Q = (const uint16_t*)Q; p.K = (const uint16_t*)K; p.V = (const uint16_t*)V; p.out = (uint16_t*)out;
    p.max_seq = max_seq;
    p.q_sh = q_sh; p.q_st = q_st; p.o_sh = o_sh; p.o_st = o_st;
    p.hq = hq; p.n_kv = n_kv; p.q_len = q_len; p.context_len = context_len;
    p.scale_log2 = scale_log2;
    const PromptPlan plan = prompt_plan(hq, n_kv, q_len, context_len, sm_count());
    p.HB = plan.HB; p.QB = plan.QB; p.hsplit = plan.hsplit; p.splits = plan.splits;
    p.err = wait_word(kWaitPrompt);
    PGK_REQUIRE(p.err, "sdpa_causal_fixed_cache failed: no pinned host memory");
    CUtensorMap kmap, vmap;
    const uint64_t dims[3] = {M_D, (uint64_t)context_len, (uint64_t)n_kv}, strides[2] = {M_D * 2, (uint64_t)max_seq * M_D * 2};
    const uint32_t box[3] = {64, M_KEYS, 1};
    PGK_REQUIRE(tma_map_bf16_3d(&kmap, K, dims, strides, box) && tma_map_bf16_3d(&vmap, V, dims, strides, box),
                "sdpa_causal_fixed_cache failed: cuTensorMapEncodeTiled refused the operands");
    int rows = plan.rows;
    if (p.splits > 1) {
        void* ws = nullptr;
        const int rc = scratch_alloc(&ws, (size_t)rows * hq * p.splits * (M_D + 4) * sizeof(float), st);
        if (rc == (int)cudaErrorMemoryAllocation) {
            set_error("");
            if (plan.ranges > 1) { *no_room = true; return 0; }
            p.splits = 1;                                 // the ranges were to fill the SMs only
            rows = q_len;
        } else if (rc)
            return rc;
        p.ws = (float*)ws;
    }
    cudaError_t e = cudaSuccess;
    for (int t = 0; e == cudaSuccess && t < q_len; t += rows) {
        p.t0 = t;
        p.t1 = t + rows < q_len ? t + rows : q_len;
        e = launch_waiting(sdpa_prompt_kernel, dim3((p.t1 - t + p.QB - 1) / p.QB, n_kv * p.hsplit, p.splits), dim3(M_THREADS), M_SMEM, st, kmap, vmap, p);
        if (e == cudaSuccess && p.splits > 1)
            e = launch_waiting(sdpa_prompt_fold_kernel, dim3(((p.t1 - t) * hq + 7) / 8), dim3(256), 0, st, p);
    }
    if (int rc = scratch_free(p.ws, st)) return rc;
    PGK_CUDA(e);
    return 0;
}

}  // namespace pgk

extern "C" int pgk_sdpa_prompt_plan(int n_heads_q, int n_kv, int q_len, int context_len, int sms, int32_t* plan) {
    PGK_REQUIRE(n_kv > 0 && n_heads_q % n_kv == 0 && n_heads_q / n_kv > 0 && n_heads_q / n_kv <= 128 && q_len > 0 && context_len >= q_len && sms > 0,
                "sdpa_prompt_plan failed: %d / %d heads, %d queries over %d keys", n_heads_q, n_kv, q_len, context_len);
    const pgk::PromptPlan p = pgk::prompt_plan(n_heads_q, n_kv, q_len, context_len, sms);
    plan[0] = p.QB; plan[1] = p.splits; plan[2] = p.rows;
    return 0;
}
