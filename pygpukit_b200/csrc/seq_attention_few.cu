// seq_attention_few.cu -- decoding over the paged bfloat16 cache: one query per request, up to 16 heads of a key/value head per block.  Same
// mathematics as seq_attention_decode_kernel (seq_attention.cu): float32 queries and key weights -- three bfloat16 terms each, which
// together hold all 24 bits --, exact products, float32 sums and softmax.
//
// What bounds it: the way from the first load to the last store; the keys of a step are read in two or three microseconds.  The kernel of
// prompts (seq_attention_tc.cu), which served decoding too, spends its time on chunks of a row passing a ring of four one after the other, on
// 32 rows where a group has 16, and on records in memory that the block which comes last folds alone.  Here:
//   * a tile is 128 keys with all their elements, on its way by TMA as a whole; the scores' MMAs start with the first 64 elements that arrive, a
//     chunk that its last product has read is fetched for the next tile at once.  Values that are a prefix of the keys (latent rows) are read once;
//   * 16 (head) rows as 3 x 16 = 48 MMA columns: scores S^T[128 keys = TMEM lanes, 48], outputs O^T[128 value elements = lanes, 48], one accumulator
//     per term.  A tile's outputs start from zero and are added to registers in float32;
//   * a request's keys are cut over a cluster of up to 16 blocks; they fold their partial outputs through each other's shared memory, a
//     share of the elements each: no records in memory, no block that comes last.
// A score that comes out NaN is formed again in float32, and so is an output (the smaller terms of an infinite operand are zeros).  (The same
// with mma.sync m16n8k16, 16 heads as its M, needs neither tensor memory nor its lanes: a tile of 64 keys of 576 / 512 took 5 us of its MMAs.)
// Measured on B200 (us with caches flushed, 16 heads over latent rows of 576 / 512, seq_attention_tc.cu in the best number of slices -> here): eight
// requests over 2000 keys 43.0 -> 28.6, over 200 33.6 -> 21.2, 24 over 1000 40.9 -> 30.7, one over 2000 40.9 -> 22.5.
#include "seq_attention.cuh"
#include "tc_common.cuh"
#include "tma.cuh"
#include "../../include/pgk_b200.h"

namespace pgk {

namespace {

constexpr int W_KEYS = 128, W_ROWS = 16, W_N = 3 * W_ROWS, W_CLUSTER = 16;
constexpr int W_WARPS = 8, W_THREADS = (W_WARPS + 2) * 32;                   // softmax and outputs; one for the copies, one for the MMAs
constexpr int W_CHUNKS = 12, W_GROUPS = 4;         // 64-element chunks of a tile, 128-element groups of a value row
constexpr uint32_t W_CHUNK = W_KEYS * 128, W_QCHUNK = W_N * 128, W_PGROUP = W_KEYS * 64, W_WEIGHTS = 2 * W_PGROUP;
constexpr float W_LOG2E = 1.4426950408889634f;

struct FewAttnArgs {
    AttnArgs a;
    int nd, ndv;             // 64-element chunks of a key row and of a value row
    int hb, bp, cluster;     // heads per block, positions per copy, blocks per request
    int qvec;                // queries by pairs
    int* err;
};

// a value's three terms; what is not finite has a first term only
__device__ __forceinline__ void split3(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        t[i] = pack_bf16x2(x, y);
        x = fabsf(x) < INFINITY ? x - bf16lo(t[i]) : 0.f;
        y = fabsf(y) < INFINITY ? y - bf16hi(t[i]) : 0.f;
    }
}
__device__ __forceinline__ uint32_t remote(uint32_t at, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_remote(uint32_t at) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ float2 ld_remote2(uint32_t at) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void all_blocks(int cluster) {
    if (cluster > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
}
// eight columns of three accumulators, loaded together
__device__ __forceinline__ void tmem_ld8x3(uint32_t t0, uint32_t t1, uint32_t t2, float (&a)[8], float (&b)[8], float (&c)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%25];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%26];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]), "=f"(a[7]),
                   "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]), "=f"(b[4]), "=f"(b[5]), "=f"(b[6]), "=f"(b[7]),
                   "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]), "=f"(c[4]), "=f"(c[5]), "=f"(c[6]), "=f"(c[7])
                 : "r"(t0), "r"(t1), "r"(t2) : "memory");
}
// the lanes' 8 values reduced over the warp: lane l ends with value l & 7
template <typename F> __device__ __forceinline__ float reduce8(float (&v)[8], int lane, F f) {
#pragma unroll
    for (int w = 4; w > 0; w >>= 1) {
        const bool up = lane & w;
#pragma unroll
        for (int j = 0; j < w; ++j) {
            const float got = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + w], w);
            v[j] = f(up ? v[j + w] : v[j], got);
        }
    }
    const float x = f(v[0], __shfl_xor_sync(0xffffffffu, v[0], 8));
    return f(x, __shfl_xor_sync(0xffffffffu, x, 16));
}
__device__ __forceinline__ bool warp_waits(int* err, uint32_t bar, uint32_t parity) {
    const bool ok = bar_wait(err, bar, parity);
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ const uint16_t* cache_row(const AttnArgs& a, const void* base, int ld, int slot, int g, int j) {
    const int pg = j / a.PS;
    return (const uint16_t*)base + (size_t)((a.table[(size_t)slot * a.max_pages + pg] * a.G + g) * a.PS + j - pg * a.PS) * ld;
}

__global__ void __launch_bounds__(W_THREADS, 1)
seq_attention_few_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, const __grid_constant__ FewAttnArgs p) {
    constexpr uint32_t TMEM_COLS = 256;
    static_assert(W_N * (1 + W_GROUPS) <= (int)TMEM_COLS, "scores and outputs");
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full_bar[W_CHUNKS], s_done, s_read, p_ready, o_done[W_GROUPS], o_read;
    __shared__ uint32_t tmem_base_s;
    __shared__ __align__(16) float wmax[W_ROWS][4];
    __shared__ float fold[W_ROWS][W_CLUSTER], m_sh[W_ROWS], l_sh[W_ROWS];
    const AttnArgs& a = p.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const bool alias = a.valias;
    const int chunks = p.nd + (alias ? 0 : p.ndv), v0 = alias ? 0 : p.nd;     // first chunk of the values
    const uint32_t base = (smem_u32(smem) + 1023u) & ~1023u, q_s = base + (uint32_t)chunks * W_CHUNK, p_s = q_s + (uint32_t)p.nd * W_QCHUNK;
    int* const err = p.err;

    if (warp == W_WARPS + 1) tmem_alloc(&tmem_base_s, TMEM_COLS);
    if (tid == 0) {
        for (int c = 0; c < chunks; ++c) mbar_init(&full_bar[c], 1);
        mbar_init(&s_done, 1);
        mbar_init(&s_read, W_WARPS);
        mbar_init(&p_ready, W_WARPS);
        mbar_init(&o_read, W_WARPS);
        for (int j = 0; j < W_GROUPS; ++j) mbar_init(&o_done[j], 1);
        mbar_fence_init();
    }
    griddep_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    griddep_launch();
    const uint32_t tmem = tmem_base_s, tmem_o = tmem + W_N;
    const int4 tile = a.tiles[blockIdx.y];
    const int t0 = tile.x, slot = tile.z, pos = tile.w, D = a.D, Dv = a.Dv;
    const int rep = a.H / a.G, hsplit = (rep + p.hb - 1) / p.hb, g = blockIdx.z / hsplit, hpart = blockIdx.z - g * hsplit;
    const int h0 = g * rep + hpart * p.hb, nh = min(p.hb, rep - hpart * p.hb);
    const int jlo = first_key(a, pos), jal = jlo & ~(p.bp - 1), ntile = (pos - jal) / W_KEYS + 1, per = (ntile + p.cluster - 1) / p.cluster;
    const int rank = blockIdx.x, tb = rank * per, n = max(0, min(ntile, tb + per) - tb);
    const float* const q = a.proj + (size_t)t0 * a.ld + a.q_off + (size_t)h0 * D;

    // ---------------- queries, beside the first copies: row 16 t + r of chunk c holds term t of head r's elements 64 c ... 64 c + 63
    if (warp < W_WARPS) {
        for (int i = tid; i < W_ROWS * p.nd * 8; i += W_WARPS * 32) {
            const int r = i / (p.nd * 8), k8 = i - r * p.nd * 8;
            float x[8];
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const float* const at = q + (size_t)r * D + k8 * 8 + e;
                float2 v = make_float2(0.f, 0.f);
                if (r < nh && k8 * 8 < D) v = p.qvec ? *(const float2*)at : make_float2(at[0], at[1]);
                x[e] = v.x; x[e + 1] = v.y;
            }
            uint32_t t[4][3];
#pragma unroll
            for (int e = 0; e < 4; ++e) split3(x[2 * e], x[2 * e + 1], t[e]);
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const int row = W_ROWS * s + r;
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(q_s + (uint32_t)(k8 >> 3) * W_QCHUNK + (uint32_t)row * 128u + (uint32_t)(((k8 & 7) ^ (row & 7)) << 4)),
                             "r"(t[0][s]), "r"(t[1][s]), "r"(t[2][s]), "r"(t[3][s]) : "memory");
            }
        }
        fence_proxy_async();
    }
    __syncwarp();
    if (warp != W_WARPS) asm volatile("bar.sync 3, %0;" :: "n"((W_WARPS + 1) * 32) : "memory");        // the MMAs' warp finds them

    if (warp == W_WARPS) {
        // ---------------- copies
        const int pieces = W_KEYS / p.bp;
        bool ok = true;
        int i = 0;
        for (; ok && i < n; ++i) {
            const int j0 = jal + (tb + i) * W_KEYS, have = min(pieces, (pos - j0) / p.bp + 1), j = j0 + lane * p.bp;
            int row = 0;
            if (lane < have) {
                const int pg = j / a.PS;
                row = (a.table[(size_t)slot * a.max_pages + pg] * a.G + g) * a.PS + j - pg * a.PS;
            }
            for (int c = 0; c < chunks; ++c) {
                // the tile before: its scores are formed, and a chunk of values has been multiplied
                const int vg = (c - v0) >> 1;
                if (i > 0) ok = ok && warp_waits(err, c >= v0 && vg < W_GROUPS ? smem_u32(&o_done[vg]) : smem_u32(&s_done), (uint32_t)((i - 1) & 1));
                if (!ok) break;
                const uint32_t bar = smem_u32(&full_bar[c]), dst = base + (uint32_t)c * W_CHUNK + (uint32_t)(lane * p.bp) * 128u;
                if (lane == 0) mbar_expect_tx(bar, (uint32_t)(have * p.bp) * 128u);
                __syncwarp();
                if (lane < have) {
                    if (c < p.nd) tma_load_2d(dst, &kmap, c * 64, row, bar);
                    else tma_load_2d(dst, &vmap, (c - p.nd) * 64, row, bar);
                }
            }
        }
        if (i > 0)                                         // whoever gives up: do not leave with copies in flight
            for (int c = 0; c < chunks; ++c) bar_wait(err, smem_u32(&full_bar[c]), (uint32_t)((i - 1) & 1));
    } else if (warp == W_WARPS + 1) {
        // ---------------- MMAs
        constexpr uint32_t id_s = umma_idesc_bf16(W_N), id_o = umma_idesc_bf16_mn(W_N);
        bool ok = true;
        for (int i = 0; ok && i < n; ++i) {
            const uint32_t par = (uint32_t)(i & 1);
            if (i > 0) ok = warp_waits(err, smem_u32(&s_read), par ^ 1u);
            for (int c = 0; ok && c < p.nd; ++c) {
                ok = warp_waits(err, smem_u32(&full_bar[c]), par);
                if (!ok) break;
                if (elect_one()) {
                    tc_fence_after();
                    const uint64_t dk = desc_sw128(base + (uint32_t)c * W_CHUNK), dq = desc_sw128(q_s + (uint32_t)c * W_QCHUNK);
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) umma_bf16(tmem, dk + (uint64_t)(ks * 2), dq + (uint64_t)(ks * 2), id_s, (c | ks) ? 1u : 0u);
                    if (c == p.nd - 1) umma_commit(&s_done);
                }
                __syncwarp();
            }
            if (!alias)
                for (int c = v0; ok && c < chunks; ++c) ok = warp_waits(err, smem_u32(&full_bar[c]), par);
            ok = ok && warp_waits(err, smem_u32(&p_ready), par);              // the outputs of the tile before are read, too
            if (!ok) break;
            if (elect_one()) {
                tc_fence_after();
#pragma unroll 1
                for (int j = 0; j < W_GROUPS; ++j) {
                    if (j * 128 < Dv) {
                        const uint64_t dv = desc_mn_sw128(base + (uint32_t)(v0 + 2 * j) * W_CHUNK, W_CHUNK), dp = desc_mn_sw64(p_s, W_PGROUP);
#pragma unroll
                        for (int ks = 0; ks < W_KEYS / 16; ++ks)              // 16 keys: 2048 bytes of V, 1024 of the weights
                            umma_bf16(tmem_o + (uint32_t)j * W_N, dv + (uint64_t)(ks * 128), dp + (uint64_t)(ks * 64), id_o, ks ? 1u : 0u);
                    }
                    umma_commit(&o_done[j]);
                }
            }
            __syncwarp();
        }
    }
    float o[W_GROUPS][8];                                    // rows r0 ... r0 + 7 of this lane's value elements
#pragma unroll
    for (int j = 0; j < W_GROUPS; ++j)
#pragma unroll
        for (int r = 0; r < 8; ++r) o[j][r] = 0.f;
    const int quad = warp & 3, half = (warp >> 2) & 1, r0 = half * 8;
    if (warp < W_WARPS) {
        // ---------------- scores, weights, outputs; lane = key, then value element
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        const int mine = r0 + (lane & 7), key = quad * 32 + lane;             // the row whose reference the lane keeps; its key
        const bool has_sink = a.sinks && rank == 0 && mine < nh;
        float m_r = has_sink ? a.sinks[h0 + mine] * W_LOG2E : -INFINITY;
        const float slope_r = a.slopes && mine < nh ? a.slopes[h0 + mine] : 0.f, slope2_r = a.slopes2 && mine < nh ? a.slopes2[h0 + mine] : 0.f;
        const float inv_cap = a.cap > 0.f ? 1.f / a.cap : 0.f;
        float l[8];                                        // this lane's share of the sums; a sink is counted once
#pragma unroll
        for (int r = 0; r < 8; ++r) l[r] = a.sinks && rank == 0 && quad == 0 && lane == 0 ? 1.f : 0.f;
        bool ok = true;
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
            const uint32_t par = (uint32_t)(i & 1);
            const int j0 = jal + (tb + i) * W_KEYS, jk = j0 + key;
            const bool seen = jk >= jlo && jk <= pos;
            ok = ok && warp_waits(err, smem_u32(&s_done), par);
            tc_fence_after();
            float s[8];
            {
                float x[8], y[8];
                tmem_ld8x3(tmem + lanes + (uint32_t)r0, tmem + lanes + W_ROWS + (uint32_t)r0, tmem + lanes + 2 * W_ROWS + (uint32_t)r0, s, x, y);
#pragma unroll
                for (int r = 0; r < 8; ++r) s[r] += x[r] + y[r];
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                if (s[r] != s[r] && seen && r0 + r < nh) {                    // an infinite operand?
                    const uint16_t* k = cache_row(a, a.kc, a.kld, slot, g, jk);
                    float z = 0.f;
#pragma unroll 1
                    for (int d = 0; d < D; ++d) z = fmaf(q[(size_t)(r0 + r) * D + d], bf16_bits_to_f32(k[d]), z);
                    s[r] = z;
                }
                s[r] *= a.scale;
                if (a.cap > 0.f) s[r] = a.cap * tanhf(s[r] * inv_cap);
                if (a.slopes) s[r] -= distance_term(__shfl_sync(0xffffffffu, slope_r, r), __shfl_sync(0xffffffffu, slope2_r, r), a.slopes2 != nullptr, pos - jk);
                if (!seen) s[r] = -INFINITY;
            }
            float v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) v[r] = s[r];
            const float top = reduce8(v, lane, [](float x, float y) { return fmaxf(x, y); });
            if (lane < 8) wmax[r0 + lane][quad] = top;
            __syncwarp();
            asm volatile("bar.sync %0, 128;" :: "r"(1 + half) : "memory");
            const float4 w = *(const float4*)wmax[mine];
            const float up = fmaxf(m_r, fmaxf(fmaxf(w.x, w.y), fmaxf(w.z, w.w)) * W_LOG2E);
            const float f_r = m_r == -INFINITY ? 0.f : exp2f(m_r - up);
            m_r = up;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_read);           // the maxima are read, too
            float f[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float m = __shfl_sync(0xffffffffu, m_r, r);
                f[r] = __shfl_sync(0xffffffffu, f_r, r);
                s[r] = ex2(fmaf(s[r], W_LOG2E, m == -INFINITY ? 0.f : -m));
                l[r] = fmaf(l[r], f[r], s[r]);
            }
            const int below = jlo - j0, above = pos - j0 + 1;
            if (below > 0 || above < W_KEYS) {             // values of keys outside the run become zeros
                for (int c = 0; c < p.ndv; ++c) ok = ok && warp_waits(err, smem_u32(&full_bar[v0 + c]), par);
                for (int u = tid; u < p.ndv * W_KEYS * 8; u += W_WARPS * 32) {
                    const int r = (u >> 3) & (W_KEYS - 1);
                    if (r >= below && r < above) continue;
                    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" :: "r"(base + (uint32_t)(v0 + (u >> 10)) * W_CHUNK + (uint32_t)r * 128u + (uint32_t)(u & 7) * 16u), "r"(0u) : "memory");
                }
            }
            if (i > 0) ok = ok && warp_waits(err, smem_u32(&o_read), par ^ 1u);          // who forms an output again reads the weights
            uint32_t t[4][3];
#pragma unroll
            for (int e = 0; e < 4; ++e) split3(s[2 * e], s[2 * e + 1], t[e]);
#pragma unroll
            for (int x = 0; x < 3; ++x) {                  // a key's row: 32 bytes of the first and of the second terms, then of the third
                const uint32_t unit = (uint32_t)((x == 1 ? 2 : 0) + half);
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(p_s + (x == 2 ? W_PGROUP : 0u) + (uint32_t)key * 64u + ((unit ^ (uint32_t)((key >> 1) & 3)) << 4)),
                             "r"(t[0][x]), "r"(t[1][x]), "r"(t[2][x]), "r"(t[3][x]) : "memory");
            }
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready);
#pragma unroll
            for (int j = 0; j < W_GROUPS; ++j) {
                ok = ok && warp_waits(err, smem_u32(&o_done[j]), par);
                if (j * 128 >= Dv) continue;
                tc_fence_after();
                float x[8], y[8], z[8];
                const uint32_t at = tmem_o + lanes + (uint32_t)(j * W_N + r0);
                tmem_ld8x3(at, at + W_ROWS, at + 2 * W_ROWS, x, y, z);
                const int dv = j * 128 + key;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    x[r] += y[r] + z[r];
                    if (x[r] != x[r] && dv < Dv && r0 + r < nh) {             // an infinite value, a weight that is not finite: as float32 has it
                        const int row = r0 + r;
                        float sum = 0.f;
#pragma unroll 1
                        for (int k = max(0, below); k < min(W_KEYS, above); ++k) {
                            float pw = 0.f;
                            for (int e = 2; e >= 0; --e) {
                                const uint32_t unit = (uint32_t)((e == 1 ? 2 : 0) + (row >> 3));
                                uint16_t bits;
                                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(bits)
                                             : "r"(p_s + (e == 2 ? W_PGROUP : 0u) + (uint32_t)k * 64u + ((unit ^ (uint32_t)((k >> 1) & 3)) << 4) + (uint32_t)(row & 7) * 2u));
                                pw += bf16_bits_to_f32(bits);
                            }
                            sum = fmaf(pw, bf16_bits_to_f32(cache_row(a, a.vc, a.vld, slot, g, j0 + k)[dv]), sum);
                        }
                        x[r] = sum;
                    }
                    o[j][r] = fmaf(o[j][r], f[r], x[r]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_read);
        }
        const float sum = reduce8(l, lane, [](float x, float y) { return x + y; });
        asm volatile("bar.sync %0, 128;" :: "r"(1 + half) : "memory");       // the last tile's maxima are read
        if (lane < 8) wmax[r0 + lane][quad] = sum;
        __syncwarp();
        asm volatile("bar.sync %0, 128;" :: "r"(1 + half) : "memory");
        if (quad == 0 && lane < 8) {
            const float4 w = *(const float4*)wmax[mine];
            m_sh[mine] = m_r;
            l_sh[mine] = (w.x + w.y) + (w.z + w.w);
        }
    }
    tc_fence_before();
    __syncthreads();                                       // the tiles are read, the products done
    if (warp == W_WARPS + 1) tmem_dealloc(tmem, TMEM_COLS);
    // ---------------- fold over the cluster: partial outputs [row][pitch] where the tiles were
    const int pitch = Dv + 4;
    float* const os = (float*)(smem + (base - smem_u32(smem)));
    if (warp < W_WARPS) {
#pragma unroll
        for (int j = 0; j < W_GROUPS; ++j) {
            const int dv = j * 128 + quad * 32 + lane;
            if (dv >= Dv) break;
#pragma unroll
            for (int r = 0; r < 8; ++r) os[(r0 + r) * pitch + dv] = o[j][r];
        }
    }
    __syncwarp();
    all_blocks(p.cluster);
    if (warp < W_WARPS) {                                  // thread: a row and a block of the cluster
        const int s = tid & 15, row = tid >> 4;
        float ms = -INFINITY, ls = 0.f;
        if (s < p.cluster) {
            ms = ld_remote(remote(smem_u32(m_sh + row), s));
            ls = ld_remote(remote(smem_u32(l_sh + row), s));
        }
        float M = ms;
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, w));
        const float e = ms == -INFINITY ? (ls != ls ? ls : 0.f) : exp2f(ms - M);         // scores of NaN: no reference, sums of NaN
        float L = ls * e;
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) L += __shfl_xor_sync(0xffffffffu, L, w);
        fold[row][s] = e * (L > 0.f || L != L ? 1.f / L : 0.f) * a.out_mult;
    }
    __syncthreads();
    const int half_dv = Dv / 2, total = nh * half_dv;
#pragma unroll 1
    for (int u = rank * W_THREADS + tid; u < total; u += p.cluster * W_THREADS) {
        const int row = u / half_dv, dv = 2 * (u - row * half_dv), h = h0 + row;
        const uint32_t at = base + (uint32_t)(row * pitch + dv) * 4u;
        float g0 = 0.f, g1 = 0.f;
        if (a.gate) {
            g0 = gate_logit(a, (size_t)t0, h, dv);
            g1 = gate_logit(a, (size_t)t0, h, dv + 1);
        }
        float2 r = make_float2(0.f, 0.f);
        for (int s0 = 0; s0 < p.cluster; s0 += 8) {
            float2 v[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) v[s] = s0 + s < p.cluster ? ld_remote2(remote(at, s0 + s)) : make_float2(0.f, 0.f);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (s0 + s >= p.cluster) break;
                const float w = fold[row][s0 + s];
                r.x = fmaf(w, v[s].x, r.x);
                r.y = fmaf(w, v[s].y, r.y);
            }
        }
        if (a.gate) {
            r.x *= 1.f / (1.f + expf(-g0));
            r.y *= 1.f / (1.f + expf(-g1));
        }
        float* const dst = a.out + (size_t)t0 * a.ldo + (size_t)h * Dv + dv;
        dst[0] = r.x;
        dst[1] = r.y;
    }
    __syncwarp();
    all_blocks(p.cluster);                                 // the others may still read this block's outputs
}

size_t few_smem(int D, int Dv, bool alias) {
    const int nd = (D + 63) / 64, chunks = nd + (alias ? 0 : (Dv + 63) / 64);
    return (size_t)chunks * W_CHUNK + (size_t)nd * W_QCHUNK + W_WEIGHTS + 1024;
}
// Value rows of 136 to 512 elements (shorter ones are no faster than on seq_attention_tc.cu, whose two blocks per SM hide each other: 16 / 4 heads of 128, eight
// requests over 1024 keys 20.4 / 20.5), key and value rows that shared memory holds (a second chunk of values that is not there reads what
// comes behind), copies of at least eight positions
bool few_fits(int D, int Dv, int kld, int vld, bool alias, int cache_dtype, int PS) {
    return cache_dtype == 2 && D % 8 == 0 && Dv % 8 == 0 && Dv > 128 && Dv <= 128 * W_GROUPS && kld % 8 == 0 && vld % 8 == 0 && PS % 8 == 0 &&
           few_smem(D, Dv, alias) <= 222 * 1024 && (D + 63) / 64 + (alias ? 0 : (Dv + 63) / 64) <= W_CHUNKS && tma_encode_fn() != nullptr;
}
cudaError_t few_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int D, int Dv, bool alias, int cluster) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(seq_attention_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(seq_attention_few_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cfg->blockDim = dim3(W_THREADS);
    cfg->dynamicSmemBytes = few_smem(D, Dv, alias);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
    return cudaSuccess;
}
// clusters that run together, as the runtime counts them: a block per SM
int few_held(int cluster) {
    static int held[W_CLUSTER + 1] = {};
    int& h = held[cluster];
    if (h == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        int n = 0;
        cfg.gridDim = dim3(cluster, 64);
        if (few_config(&cfg, at, 576, 512, true, cluster) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, seq_attention_few_kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        h = n > 0 ? n : -1;
    }
    return h;
}

}  // namespace

// Blocks per request: the fewest rounds of tiles one after the other, a block's start and end counted as two and a cluster's fold as half a tile (5.6 us of
// 576 / 512; us, blocks 1 / 2 / 4 / 8 / 16 a request: eight over 200 28.7 / 22.5 / 21.4 / 21.2 / 37.9, over 2000 102 / 59 / 38 / 28.6 / 41 -- seven
// clusters of 16 run together --, 24 over 1000 61 / 39 / 30.7 / 41 / 72, one over 2000 104 / 59 / 37 / 26.6 / 22.5).  0: not served.
int seq_attention_few_plan(int D, int Dv, int kld, int vld, bool alias, int H, int G, int cache_dtype, int PS, int requests, int keys) {
    if (!few_fits(D, Dv, kld, vld, alias, cache_dtype, PS) || keys > 1 << 24) return 0;
    const int rep = H / G, hb = rep < W_ROWS ? rep : W_ROWS;
    const long long n = (long long)requests * G * ((rep + hb - 1) / hb);
    if (n > 65535 || G * ((rep + hb - 1) / hb) > 65535) return 0;
    const int tiles = (keys + W_KEYS - 1) / W_KEYS + 1;                       // a window starts anywhere
    int best = 0;
    double best_cost = 1e30;
    for (int c = 1; c <= W_CLUSTER; c *= 2) {
        const int held = few_held(c);
        if (held <= 0 || (c > 1 && c > tiles)) continue;
        const double rounds = (double)((n + held - 1) / held), cost = rounds * ((tiles + c - 1) / c + 2.0) + (c > 1 ? 0.5 : 0.0);
        if (cost < best_cost * 0.999) { best_cost = cost; best = c; }
    }
    return best;
}

int seq_attention_few(const AttnArgs& a, int tiles, int cluster, cudaStream_t st, bool* served) {
    *served = false;
    const bool alias = a.valias;
    if (!few_fits(a.D, a.Dv, a.kld, a.vld, alias, 2, a.PS) || cluster < 1 || cluster > W_CLUSTER || few_held(cluster) <= 0) return 0;
    if (a.prob || a.pool || a.o_inv_freq || a.keep || (uintptr_t)a.kc % 16 || (uintptr_t)a.vc % 16) return 0;
    FewAttnArgs p{};
    p.a = a;
    p.qvec = (uintptr_t)a.proj % 8 == 0 && a.ld % 2 == 0 && a.q_off % 2 == 0;
    p.nd = (a.D + 63) / 64;
    p.ndv = (a.Dv + 63) / 64;
    const int rep = a.H / a.G;
    p.hb = rep < W_ROWS ? rep : W_ROWS;
    p.bp = a.PS & -a.PS;
    if (p.bp > W_KEYS) p.bp = W_KEYS;
    p.cluster = cluster;
    p.err = wait_word(kWaitFew);
    PGK_REQUIRE(p.err, "seq_attention failed: no pinned host memory");
    const int heads = a.G * ((rep + p.hb - 1) / p.hb);
    if (tiles > 65535 || heads > 65535) return 0;
    CUtensorMap kmap, vmap;
    const uint64_t rows = 1ull << 31;                     // cache rows: the table names only pages that exist
    if (!tma_map_bf16_2d(&kmap, a.kc, (uint64_t)a.D, rows, (uint64_t)a.kld * 2, 64, (uint32_t)p.bp) ||
        !tma_map_bf16_2d(&vmap, a.vc, (uint64_t)a.Dv, rows, (uint64_t)a.vld * 2, 64, (uint32_t)p.bp)) return 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    PGK_CUDA(few_config(&cfg, at, a.D, a.Dv, alias, cluster));
    cfg.gridDim = dim3(cluster, tiles, heads);
    cfg.stream = st;
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_waiting
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    count_launch();
    void* args[] = {&kmap, &vmap, &p};
    PGK_CUDA(cudaLaunchKernelExC(&cfg, (const void*)seq_attention_few_kernel, args));
    *served = true;
    return 0;
}

}  // namespace pgk

extern "C" int pgk_seq_attention_few_plan(int dim, int vdim, int k_ld, int v_ld, int same_rows, int heads, int kv_heads, int cache_dtype, int page_size,
                                          int requests, int keys) {
    return heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && vdim > 0 && page_size > 0 && requests > 0
               ? pgk::seq_attention_few_plan(dim, vdim, k_ld, v_ld, same_rows != 0, heads, kv_heads, cache_dtype, page_size, requests, keys) : 0;
}
