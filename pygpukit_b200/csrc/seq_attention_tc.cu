// seq_attention_tc.cu -- prompt attention of the token-major models on tcgen05, for a bfloat16 cache.  Same mathematics, tiles and
// fold as seq_attention_kernel (seq_attention.cu), float32 throughout: the queries (float32) enter the score product as THREE
// bfloat16 terms that together hold all 24 bits, the key weights (float32) the value product likewise, and each term keeps
// accumulators of its own, so that what the tensor cores sum are exact products in float32.
//
// What bounds it: the multiprocessors' ordinary arithmetic (a score costs an exponential, a mask, a cap, the split of its weight:
// 30 ... 60 instructions), then the key stream from L2.  What follows from that:
//   * a block keeps the tile of 32 (query, head) rows that the float32 kernel has, as 3 x 32 = 96 MMA columns: scores are formed
//     TRANSPOSED, S^T[128 keys = TMEM lanes, 96], and so are the outputs, O^T[128 value elements = lanes, 96] per 128 value
//     elements.  An accumulator of 512 value elements (latent rows) then fits TMEM beside the scores, and 96 columns amortise the
//     operand reads of the MMA where 32 would not;
//   * eight warps take a tile's scores, a lane a key, 16 rows each; row maxima meet by 16 shuffles per warp and one exchange among
//     the four warps of a half; sums stay with the lane until the end;
//   * the running reference of a row moves only when a tile's maximum exceeds it by LAZY (log2 units): outputs in TMEM are then
//     rescaled.  Tiles run from the nearest keys to the farthest, so that under a distance term the first tile settles it;
//   * the scores of tile i + 1 are multiplied while tile i's weights are formed; K and V chunks (128 keys x 64 elements) come
//     through one ring, by TMA from pages of a multiple of eight positions (cp.async, which an SM takes at 16 bytes per cycle
//     only, serves the others); value rows of keys outside the run are zeroed, their scores masked;
//   * heads of 128: 113 KB of shared memory and 256 TMEM columns, two blocks per SM hide each other's chains; ten warps leave
//     96 registers a thread; the forms of the score are template parameters, since a tile's straight-line code is long enough
//     for instruction fetch to show.
//   * the copies start beside the queries' conversion, an edge tile's zeros are written while the next pair of chunks arrives, the
//     outputs leave four rows at a time in a short loop (code that runs once per block costs its fetch), and rows that no query
//     has are left out: what decoding, one tile per block, spends its time on.
// Measured on B200, 2000 tokens: 32 / 4 heads of 128 in chunks of 1024 with cap and slopes 1336 -> 186 us; 16 heads over latent rows
// of 576 / 512 5097 -> 445 us.  Decoding, 8 requests: latent rows over 2000 keys 129 -> 50 us, 16 / 4 heads of 128 over 1024 65 -> 24
// us.  (Weights reach 2^LAZY before their reference moves: sums of values above 2^120 may overflow.)  Against float64 the errors are the float32 kernel's or smaller (rms 4.7e-8 -> 3.3e-8 at heads of
// 128).
#include "seq_attention.cuh"
#include "tc_common.cuh"
#include "tma.cuh"
#include "../../include/pgk_b200.h"

namespace pgk {

namespace {

constexpr int AR = 32;                     // (query, head) rows per block
constexpr int AN = 3 * AR;                 // MMA columns: the three terms of every row
constexpr int AK = 128;                    // keys per tile
constexpr int A_SOFT = 8;                  // warps: softmax; one for the copies, one that issues the MMAs
constexpr int A_THREADS = (A_SOFT + 2) * 32;
constexpr int A_RING = 4;
constexpr uint32_t A_CHUNK = AK * 128;     // 128 keys x 64 elements
constexpr uint32_t A_QCHUNK = AN * 128;
constexpr uint32_t A_PTERM = AK * AR * 2;
constexpr uint32_t A_PBYTES = 3 * A_PTERM;
constexpr uint32_t A_TAIL = 128 + 512 + 256 + 128;   // barriers and TMEM address, row maxima, what a row knows, its output
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LAZY = 8.f;

struct TcAttnArgs {
    AttnArgs a;
    int nd, nd2, ndv;        // 64-element chunks of a key row (and rounded up to even), 128-element chunks of a value row
    uint32_t tmem_cols;
    int qvec;                // query rows keep 16-byte boundaries
    int bp;                  // positions per TMA copy (a power of two that divides the page), 0: cp.async
    int* err;                // raised when a bounded wait runs out
};

__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void half_sync(int half) {
    __syncwarp();                                         // bar.sync takes whole warps, and a few lanes' stores come before it
    asm volatile("bar.sync %0, 128;" :: "r"(1 + half) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// the lanes' 16 values reduced over the warp: lane l (and l + 16) ends with value l & 15
template <typename F> __device__ __forceinline__ float reduce16(float (&v)[16], int lane, F f) {
#pragma unroll
    for (int w = 8; w > 0; w >>= 1) {
        const bool up = lane & w;
#pragma unroll
        for (int j = 0; j < w; ++j) {
            const float got = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + w], w);
            v[j] = f(up ? v[j + w] : v[j], got);
        }
    }
    return f(v[0], __shfl_xor_sync(0xffffffffu, v[0], 16));
}
__device__ __forceinline__ float max_nan(float a, float b) {       // NaN if either is
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// A product whose leading term is infinite or NaN: with an infinite operand that is what float32 gives, while the smaller terms --
// zeros, of either sign, or infinity minus itself -- make NaN of it.
__device__ __forceinline__ float leading_or(float lead, float sum) { return fabsf(lead) < INFINITY ? sum : lead; }
// a + b + c of three accumulators' 16 columns, smallest first
__device__ __forceinline__ void tmem_sum3(uint32_t t0, uint32_t t1, uint32_t t2, float (&v)[16], bool infinities) {
    float x[16], y[16];
    tmem_ld16_async(t2, v);
    tmem_ld16_async(t1, x);
    tmem_ld16_async(t0, y);
    tmem_ld_wait(v, x, y);
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = (v[r] + x[r]) + y[r];
    if (infinities) {
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = leading_or(y[r], v[r]);
    }
}

// CAP: tanh cap; SLOPE: 0 none, 1 per-head slopes, 2 the logarithmic form; PROB: sigmoid weights
template <bool CAP, int SLOPE, bool PROB>
__global__ void __launch_bounds__(A_THREADS, 2)
seq_attention_tc_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, const __grid_constant__ TcAttnArgs p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const AttnArgs& a = p.a;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t q_s = smem_u32(smem), p_s = q_s + (uint32_t)p.nd * A_QCHUNK, ring = p_s + A_PBYTES, tail = ring + A_RING * A_CHUNK;
    const uint32_t full_bar = tail, empty_bar = tail + 32, s_full = tail + 64, s_read = tail + 72, p_ready = tail + 80, pv_done = tail + 88,
                   land_bar = tail + 96;                  // and at + 112: pairs of an edge tile by turns
    unsigned char* tail_p = smem + (tail - q_s);
    uint32_t* tmem_slot = (uint32_t*)(tail_p + 104);
    float* wmax = (float*)(tail_p + 128);                // [32 rows][4]
    float2* rowi = (float2*)(tail_p + 640);              // [32 rows] position, slope
    int* rowo = (int*)(tail_p + 896);                    // [32 rows] query << 16 | head of the row, -1: nobody's
    if (q_s & 1023u) {                                   // the layout relies on it (uniform over the grid)
        if (tid == 0) *(volatile int*)p.err = 2;
        return;
    }

    if (warp == A_SOFT + 1) tmem_alloc(tmem_slot, p.tmem_cols);
    if (tid == 0) {
        uint64_t* b = (uint64_t*)tail_p;
        for (int s = 0; s < A_RING; ++s) { mbar_init(b + s, 1); mbar_init(b + A_RING + s, 1); }
        mbar_init(b + 8, 1); mbar_init(b + 9, A_SOFT); mbar_init(b + 10, A_SOFT); mbar_init(b + 11, 1); mbar_init(b + 12, 2); mbar_init(b + 14, 2);
        mbar_fence_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    griddep_wait();
    griddep_launch();
    // blocks start in the order of their numbers: the last request's last queries first, each request's from its last, which see the most keys, to its first,
    // so that with one request none of the long ones starts when the others end (16 heads over latent rows, 2000 tokens, 1000 blocks of 1 to 16 tiles 466 -> 445 us;
    // 32 / 4 heads of 128 in chunks of 1024, 2000 blocks 195 -> 186).  Which of several requests is the longest moves a prompt of 2 to 7 unequal ones by 1 % at most
    const int nth = (int)(blockIdx.y * gridDim.x + blockIdx.x), block = nth / (int)gridDim.y, part = nth - block * (int)gridDim.y;
    const int4 tile = a.tiles[(int)gridDim.x - 1 - block];
    const int t0 = tile.x, nq = tile.y, slot = tile.z, pos0 = tile.w, D = a.D, Dv = a.Dv, HB = a.HB;
    const int rep = a.H / a.G, hsplit = (rep + HB - 1) / HB;
    const int g = part / hsplit, hpart = part - g * hsplit;
    const int hb0 = g * rep + hpart * HB, nh = min(HB, rep - hpart * HB);
    const int live = min(AR, nq * HB);                   // rows that a query has

    // the block's key tiles: the kept first positions below the window, then [jlo, jhi] from a copy's boundary on
    const int jlo = first_key(a, pos0), jhi = pos0 + nq - 1, jal = p.bp ? jlo & ~(p.bp - 1) : jlo;
    const int kept = a.window > 0 ? min(a.keep, jlo) : 0, nkept = (kept + AK - 1) / AK;
    const int ntile = nkept + (jhi - jal) / AK + 1, per = (ntile + a.splits - 1) / a.splits;
    const int tbeg = (int)blockIdx.z * per, tend = min(ntile, tbeg + per), n = max(0, tend - tbeg);
    const int nv2 = 2 * p.ndv;
    int* const err = p.err;

    if (warp != A_SOFT) {
        // ---------------- queries, beside the first copies: rows 32 t + r of chunk c hold term t of row r's elements 64 c ... 64 c + 63
        if (tid < AR) {
            const int qi = tid / HB, hh = tid - qi * HB;
            const bool has = qi < nq && hh < nh;
            rowi[tid] = make_float2((float)(pos0 + qi), SLOPE && has ? a.slopes[hb0 + hh] : 0.f);
            rowo[tid] = has ? qi << 16 | hh : -1;
        }
        if (warp < A_SOFT) {
            const int items = AR * p.nd * 8;
            auto fetch = [&](int i, float (&x)[8]) {
                const int r = i / (p.nd * 8), d = (i - r * p.nd * 8) * 8, qi = r / HB, hh = r - qi * HB;
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = 0.f;
                if (i < items && qi < nq && hh < nh && d < D) {
                    const float* src = a.proj + (size_t)(t0 + qi) * a.ld + a.q_off + (size_t)(hb0 + hh) * D + d;
                    if (p.qvec) {
                        *(float4*)&x[0] = *(const float4*)src;
                        *(float4*)&x[4] = *(const float4*)(src + 4);
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) x[e] = src[e];
                    }
                }
            };
            float next[8];
            fetch(tid, next);
#pragma unroll 1
            for (int i = tid; i < items; i += A_SOFT * 32) {
                float x[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = next[e];
                fetch(i + A_SOFT * 32, next);
                const int r = i / (p.nd * 8), k8 = i - r * p.nd * 8;
#pragma unroll
                for (int t = 0; t < 3; ++t) {            // three terms that together hold all 24 bits
                    uint32_t v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        v[e] = pack_bf16x2(x[2 * e], x[2 * e + 1]);
                        x[2 * e] -= bf16lo(v[e]);
                        x[2 * e + 1] -= bf16hi(v[e]);
                    }
                    const int row = AR * t + r;
                    sts128(q_s + (uint32_t)(k8 >> 3) * A_QCHUNK + (uint32_t)row * 128u + (uint32_t)(((k8 & 7) ^ (row & 7)) << 4), v);
                }
            }
            fence_proxy_async();
        }
        __syncwarp();
        asm volatile("bar.sync 3, %0;" :: "n"((A_SOFT + 1) * 32) : "memory");
    }
    if (warp == A_SOFT) {
        // ---------------- copies
        int k = 0;                                        // slots issued
        bool ok = true;
        if (p.bp) {                                       // TMA: piece l is positions l bp ... of a tile
            const int pieces = AK / p.bp;
            uint32_t phase = 0;
            // lane l: the cache row of tile ti's piece l, and how many pieces there are (tiles i and i + 1 by turns)
            int row0 = 0, row1 = 0, have0 = 0, have1 = 0;
            auto where = [&](int ti, int u) {
                const bool early = ti < nkept;
                const int j0 = early ? ti * AK : jal + (ti - nkept) * AK, j = j0 + lane * p.bp, jmax = early ? kept - 1 : jhi;
                int row = 0;
                if (lane < pieces && j <= jmax) {
                    const int pg = j / a.PS;
                    row = (a.table[(size_t)slot * a.max_pages + pg] * a.G + g) * a.PS + j - pg * a.PS;
                }
                const int have = __popc(__ballot_sync(0xffffffffu, lane < pieces && j <= jmax));
                if (u) { row1 = row; have1 = have; } else { row0 = row; have0 = have; }
            };
            // the pair of slots from `at` on has arrived: rows outside the run become zeros, then the MMAs may have it
            auto clear = [&](int at, int below, int above) {
                __syncwarp();
                bar_wait(err, land_bar + 8u * (uint32_t)(at & 2), (phase >> (at & 2)) & 1u);
                phase ^= 1u << (at & 2);
                const uint32_t pair = ring + (uint32_t)(at & (A_RING - 1)) * A_CHUNK;
                for (int r = lane >> 3; r < AK; r += 4) {
                    if (r >= below && r < above) continue;
                    const uint32_t z[4] = {0u, 0u, 0u, 0u};
                    sts128(pair + (uint32_t)r * 128u + (uint32_t)(lane & 7) * 16u, z);
                    sts128(pair + A_CHUNK + (uint32_t)r * 128u + (uint32_t)(lane & 7) * 16u, z);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive((uint64_t*)(tail_p + 8 * (at & (A_RING - 1))));
                    mbar_arrive((uint64_t*)(tail_p + 8 * ((at + 1) & (A_RING - 1))));
                }
            };
            // every lane waits for the slot and fetches its piece at once: the ring is short, its round trip is what counts
            auto issue = [&](const CUtensorMap* map, int c, int u, bool pad, bool edge) {
                const uint32_t sl = (uint32_t)(k & (A_RING - 1)), dst = ring + sl * A_CHUNK + (uint32_t)(lane * p.bp) * 128u;
                const uint32_t bar = edge ? land_bar + 8u * (sl & 2u) : full_bar + 8u * sl;
                const int have = pad ? 0 : (u ? have1 : have0), row = u ? row1 : row0;
                ok = ok && bar_wait(err, empty_bar + 8u * sl, (uint32_t)(((k / A_RING) & 1) ^ 1));
                if (ok && lane < have) tma_load_2d(dst, map, c * 64, row, bar);
                if (ok && lane == 0) mbar_expect_tx(bar, (uint32_t)(have * p.bp) * 128u);
                ++k;
            };
            if (n > 0) {
                where(tend - 1, 0);
                for (int c = 0; c < p.nd2; ++c) issue(&kmap, c, 0, c >= p.nd, false);
            }
            for (int i = 0; i < n; ++i) {
                const int ti = tend - 1 - i, u = i & 1;
                if (i + 1 < n) {
                    where(ti - 1, u ^ 1);
                    for (int c = 0; c < p.nd2; ++c) issue(&kmap, c, u ^ 1, c >= p.nd, false);
                }
                const bool early = ti < nkept;
                const int j0 = early ? ti * AK : jal + (ti - nkept) * AK;
                const int below = early ? 0 : max(0, jlo - j0), above = min(AK, (early ? kept - 1 : jhi) - j0 + 1);
                const bool edge = below > 0 || above < AK;          // some rows lie outside the run: their values become zeros
                for (int c = 0; c < nv2; c += 2) {
                    issue(&vmap, c, u, false, edge);
                    issue(&vmap, c + 1, u, (c + 1) * 64 >= Dv, edge);
                    if (!edge) continue;
                    if (c) clear(k - 4, below, above);    // a pair is cleared while the next one arrives
                    if (c + 2 >= nv2) clear(k - 2, below, above);
                }
            }
            for (int j = max(0, k - A_RING); j < k; ++j)  // whoever gave up: do not leave with copies in flight
                bar_wait(err, full_bar + 8u * (uint32_t)(j & (A_RING - 1)), (uint32_t)((j / A_RING) & 1));
        } else {                                          // cp.async: eight lanes fetch one key's 128 bytes, zeros outside the run
            const int sub = lane >> 3, col16 = lane & 7;
            int cur[4], nxt[4] = {-1, -1, -1, -1};
            auto rows_of = [&](int ti, int (&mine)[4]) {  // lane: cache rows of keys lane + 32 u
                const bool early = ti < nkept;
                const int j0 = early ? ti * AK : jal + (ti - nkept) * AK, jmax = early ? kept - 1 : jhi;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = j0 + lane + 32 * u;
                    mine[u] = j <= jmax ? (a.table[(size_t)slot * a.max_pages + j / a.PS] * a.G + g) * a.PS + j % a.PS : -1;
                }
            };
            auto land = [&](int s) {                      // slot s has arrived: hand it to the MMAs
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive((uint64_t*)(tail_p + 8 * (s & (A_RING - 1))));
            };
            auto chunk = [&](const uint16_t* base, int ld, int c0, int width, const int (&mine)[4]) {
                ok = ok && __all_sync(0xffffffffu, bar_wait(err, empty_bar + 8u * (uint32_t)(k & (A_RING - 1)), (uint32_t)(((k / A_RING) & 1) ^ 1)));
                const int c = c0 + col16 * 8;
                const uint32_t dst = ring + (uint32_t)(k & (A_RING - 1)) * A_CHUNK;
                if (ok && c0 < width) {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll 1
                        for (int r = 0; r < 8; ++r) {
                            const int row = __shfl_sync(0xffffffffu, mine[u], r * 4 + sub), key = u * 32 + r * 4 + sub;
                            const bool in = row >= 0 && c < width;
                            cp_async16_zfill(dst + (uint32_t)key * 128u + (uint32_t)((col16 ^ (key & 7)) << 4),
                                             in ? base + (long long)row * ld + c : base, in ? 16u : 0u);
                        }
                }
                cp_async_commit();
                ++k;
                if (k > 2) { cp_async_wait<2>(); land(k - 3); }
            };
            const uint16_t* kc = (const uint16_t*)a.kc;
            const uint16_t* vc = (const uint16_t*)a.vc;
            if (n > 0) {
                rows_of(tend - 1, cur);
                for (int c = 0; c < p.nd2; ++c) chunk(kc, a.kld, c * 64, D, cur);
                for (int i = 0; i < n; ++i) {
                    if (i + 1 < n) {
                        rows_of(tend - 2 - i, nxt);
                        for (int c = 0; c < p.nd2; ++c) chunk(kc, a.kld, c * 64, D, nxt);
                    }
                    for (int c = 0; c < nv2; ++c) chunk(vc, a.vld, c * 64, Dv, cur);
#pragma unroll
                    for (int u = 0; u < 4; ++u) cur[u] = nxt[u];
                }
                cp_async_wait<1>();
                land(k - 2);
                cp_async_wait<0>();
                land(k - 1);
            }
        }
    } else if (warp == A_SOFT + 1) {
        // ---------------- MMAs
        if (elect_one()) {
            constexpr uint32_t id_s = umma_idesc_bf16(AN), id_o = umma_idesc_bf16_mn(AN);
            int k = 0;
            bool ok = true;
            auto scores = [&]() {
                for (int c = 0; ok && c < p.nd2; ++c, ++k) {
                    const uint32_t s = (uint32_t)(k & (A_RING - 1));
                    ok = bar_wait(err, full_bar + 8u * s, (uint32_t)((k / A_RING) & 1));
                    if (!ok) return;
                    tc_fence_after();
                    if (c < p.nd) {
                        const uint64_t dk = desc_sw128(ring + s * A_CHUNK), dq = desc_sw128(q_s + (uint32_t)c * A_QCHUNK);
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) umma_bf16(tmem, dk + (uint64_t)(ks * 2), dq + (uint64_t)(ks * 2), id_s, (c | ks) ? 1u : 0u);
                    }
                    umma_commit((uint64_t*)(tail_p + 32 + 8 * s));
                }
                umma_commit((uint64_t*)(tail_p + 64));
            };
            if (n > 0) scores();
            for (int i = 0; ok && i < n; ++i) {
                if (i + 1 < n) {
                    ok = bar_wait(err, s_read, (uint32_t)(i & 1));
                    if (!ok) break;
                    tc_fence_after();
                    scores();
                    if (!ok) break;
                }
                ok = bar_wait(err, p_ready, (uint32_t)(i & 1));
                if (!ok) break;
                tc_fence_after();
                for (int c = 0; ok && c < p.ndv; ++c, k += 2) {
                    const uint32_t s = (uint32_t)(k & (A_RING - 1));
                    ok = bar_wait(err, full_bar + 8u * s, (uint32_t)((k / A_RING) & 1)) && bar_wait(err, full_bar + 8u * (s + 1), (uint32_t)((k / A_RING) & 1));
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t dv = desc_mn_sw128(ring + s * A_CHUNK, A_CHUNK), dp = desc_mn_sw64(p_s, A_PTERM);
#pragma unroll
                    for (int ks = 0; ks < AK / 16; ++ks)              // 16 keys: 2048 bytes of V, 1024 of the weights
                        umma_bf16(tmem + AN + (uint32_t)c * AN, dv + (uint64_t)(ks * 128), dp + (uint64_t)(ks * 64), id_o, (i | ks) ? 1u : 0u);
                    umma_commit((uint64_t*)(tail_p + 32 + 8 * s));
                    umma_commit((uint64_t*)(tail_p + 32 + 8 * (s + 1)));
                }
                umma_commit((uint64_t*)(tail_p + 88));
            }
        }
        __syncwarp();
    } else {
        // ---------------- weights
        const int quad = warp & 3, half = warp >> 2, r0 = half * 16;
        const bool has_sink = a.sinks && blockIdx.z == 0;         // the sink counts once: slice 0
        const float inv_cap = CAP ? 1.f / a.cap : 0.f, keep_f = (float)a.keep;
        const int lo_max = first_key(a, jhi);
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        // lane r (and r + 16) knows row r0 + r: where its window starts, its reference (log2 units), ...
        float lo_r, extra_r = 0.f, pb_r = 0.f, m_r = PROB ? 0.f : -INFINITY;
        {
            const int row = r0 + (lane & 15), qi = row / HB, hh = row - qi * HB;
            lo_r = (float)first_key(a, pos0 + qi);
            if (qi < nq && hh < nh) {
                if (SLOPE == 2) extra_r = a.slopes2[hb0 + hh];
                if (PROB && a.pbias) pb_r = a.pbias[hb0 + hh];
                if (has_sink) m_r = a.sinks[hb0 + hh] * LOG2E;
            }
        }
        float nm[16], l[16];                              // minus the rows' references (0 while there is none), this lane's share of the sums
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float m = __shfl_sync(0xffffffffu, m_r, r);
            nm[r] = m == -INFINITY ? 0.f : -m;
            l[r] = ((PROB && blockIdx.z == 0) || has_sink) && quad == 0 && lane == 0 ? 1.f : 0.f;
        }
        bool ok = true;
        if (r0 >= live) {                                 // nobody's rows (decoding): keep the barriers' count
            for (int i = 0; i < n; ++i) {
                ok = ok && bar_wait(err, s_full, (uint32_t)(i & 1));
                __syncwarp();
                if (lane == 0) mbar_arrive((uint64_t*)(tail_p + 72));
                if (i > 0) ok = ok && bar_wait(err, pv_done, (uint32_t)((i - 1) & 1));
                __syncwarp();
                if (lane == 0) mbar_arrive((uint64_t*)(tail_p + 80));
            }
        } else
        for (int i = 0; i < n; ++i) {
            const int ti = tend - 1 - i;
            const bool early = ti < nkept;
            const int j0 = early ? ti * AK : jal + (ti - nkept) * AK, jmin = early ? 0 : jlo, jmax = early ? kept - 1 : jhi;
            const int j = j0 + quad * 32 + lane;
            const float jf = (float)j;
            const bool whole = !early && j0 >= lo_max && j0 + AK - 1 <= pos0;        // every row sees every key
            ok = ok && bar_wait(err, s_full, (uint32_t)(i & 1));       // (when a wait runs out the rest runs through without waiting)
            __syncwarp();
            tc_fence_after();
            float s[16], top;
#pragma unroll 1
            for (bool again = false;; again = true) {     // a second time only where a score is NaN: an infinite operand?
                tmem_sum3(lanes + r0, lanes + AR + r0, lanes + 2 * AR + r0, s, again);
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    s[r] *= a.scale;
                    if (CAP) s[r] = a.cap * tanhf(s[r] * inv_cap);
                    if (SLOPE) {
                        const float2 w = rowi[r0 + r];
                        const float d = fmaxf(w.x - jf, 0.f);
                        if (SLOPE == 2) s[r] -= w.y * log1pf(__shfl_sync(0xffffffffu, extra_r, r) * d);
                        else s[r] = fmaf(-w.y, d, s[r]);
                    }
                }
                if (!whole) {
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const float pi = rowi[r0 + r].x, lo = __shfl_sync(0xffffffffu, lo_r, r);
                        if (!(j >= jmin && j <= jmax && jf <= pi && (jf >= lo || jf < keep_f))) s[r] = -INFINITY;
                    }
                }
                if (PROB) {
                    top = 0.f;
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const float z = s[r] + __shfl_sync(0xffffffffu, pb_r, r);
                        s[r] = s[r] == -INFINITY ? 0.f : 1.f / (1.f + expf(-z));
                        top = max_nan(top, s[r]);
                    }
                } else {
                    float v[16];
#pragma unroll
                    for (int r = 0; r < 16; ++r) v[r] = s[r];
                    top = reduce16(v, lane, [](float x, float y) { return max_nan(x, y); });
                }
                if (again || !__any_sync(0xffffffffu, top != top)) break;
            }
            bool waited = false;
            if (PROB) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive((uint64_t*)(tail_p + 72));
            } else {
                if (lane < 16) wmax[(r0 + lane) * 4 + quad] = top;
                half_sync(half);
                const float4 w = *(const float4*)(wmax + (r0 + (lane & 15)) * 4);
                const float mt = fmaxf(fmaxf(w.x, w.y), fmaxf(w.z, w.w)) * LOG2E;
                const bool up = mt > m_r + LAZY;          // (also the first finite maximum: m = -inf)
                if (__any_sync(0xffffffffu, up)) {        // the same in the half's four warps: its columns of O^T move along
                    const float f_r = !up ? 1.f : (m_r == -INFINITY ? 0.f : exp2f(m_r - mt));
                    if (up) m_r = mt;
                    float f[16];
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const float m = __shfl_sync(0xffffffffu, m_r, r);
                        f[r] = __shfl_sync(0xffffffffu, f_r, r);
                        nm[r] = m == -INFINITY ? 0.f : -m;
                        l[r] *= f[r];
                    }
                    if (i > 0) {
                        ok = ok && bar_wait(err, pv_done, (uint32_t)((i - 1) & 1));
                        __syncwarp();
                        waited = true;
                        tc_fence_after();
                        for (int c = 0; c < 3 * p.ndv; ++c) {
                            float o[16];
                            const uint32_t at = lanes + AN + (uint32_t)c * AR + (uint32_t)r0;
                            tmem_ld16(at, o);
#pragma unroll
                            for (int r = 0; r < 16; ++r) o[r] *= f[r];
                            tmem_st16(at, o);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive((uint64_t*)(tail_p + 72));              // the maxima are read, too
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    s[r] = ex2(fmaf(s[r], LOG2E, nm[r]));
                    l[r] += s[r];
                }
            }
            if (i > 0 && !waited) {                       // the last tile's product has read the weights
                ok = ok && bar_wait(err, pv_done, (uint32_t)((i - 1) & 1));
                __syncwarp();
            }
            const int key = quad * 32 + lane;
            const uint32_t at_p = p_s + (uint32_t)key * 64u;
#pragma unroll
            for (int t = 0; t < 3; ++t) {                 // three terms that together hold all 24 bits
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    w[e] = pack_bf16x2(s[2 * e], s[2 * e + 1]);
                    s[2 * e] -= bf16lo(w[e]);
                    s[2 * e + 1] -= bf16hi(w[e]);
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const uint32_t v[4] = {w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]};
                    sts128(at_p + (uint32_t)t * A_PTERM + (uint32_t)(((2 * half + q) ^ ((key >> 1) & 3)) << 4), v);
                }
            }
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive((uint64_t*)(tail_p + 80));
        }
        // ---------------- outputs: lane = value element
        if (ok && n > 0) bar_wait(err, pv_done, (uint32_t)((n - 1) & 1));
        __syncwarp();
        tc_fence_after();
        {
            const float sum = reduce16(l, lane, [](float x, float y) { return x + y; });
            half_sync(half);                              // the maxima of the last tile are read
            if (lane < 16) wmax[(r0 + lane) * 4 + quad] = sum;
            half_sync(half);
            const float4 w = *(const float4*)(wmax + (r0 + (lane & 15)) * 4);
            const float l_r = (w.x + w.y) + (w.z + w.w);
            if (a.splits > 1 && quad == 0 && lane < 16) {
                const int r = r0 + lane, qi = r / HB, hh = r - qi * HB;
                if (qi < nq && hh < nh) {
                    float* rec = a.ws + (((size_t)(t0 + qi) * a.H + hb0 + hh) * a.splits + blockIdx.z) * (Dv + 2);
                    rec[0] = m_r; rec[1] = l_r;
                }
            }
            const float inv_r = a.splits > 1 ? 1.f : (l_r > 0.f ? 1.f / l_r : 0.f) * a.out_mult;
            // four rows at a time and only a query's: what runs once costs its fetch, 16 rows in a row 7000 cycles per 128 elements
            const int steps = 4 * p.ndv;
            const bool gated = a.gate && a.splits == 1;
            float gz[4], go[4] = {0.f, 0.f, 0.f, 0.f};
            auto gates = [&](int u) {
                const int dv = (u >> 2) * 128 + quad * 32 + lane, rr = r0 + (u & 3) * 4;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int ro = rowo[rr + e];
                    go[e] = u < steps && dv < Dv && ro >= 0 ? gate_logit(a, (size_t)(t0 + (ro >> 16)), hb0 + (ro & 0xffff), dv) : 0.f;
                }
            };
            if (gated) gates(0);
#pragma unroll 1
            for (int u = 0; u < steps; ++u) {
                const int rr = r0 + (u & 3) * 4, dv = (u >> 2) * 128 + quad * 32 + lane;
                float o[4] = {0.f, 0.f, 0.f, 0.f}, x[4], y[4];
                if (gated) {                              // the next step's loads go out before this one's use
#pragma unroll
                    for (int e = 0; e < 4; ++e) gz[e] = go[e];
                    gates(u + 1);
                }
                if (rr >= live) continue;
                __syncwarp();                             // lanes beyond the row's end skipped the last stores; the load takes whole warps
                if (n > 0) {
                    const uint32_t at = lanes + AN + (uint32_t)(u >> 2) * AN + (uint32_t)rr;
                    tmem_ld4x3(at, at + AR, at + 2 * AR, o, x, y);
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[e] = leading_or(o[e], o[e] + (x[e] + y[e]));
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float v = o[e] * __shfl_sync(0xffffffffu, inv_r, rr - r0 + e);
                    const int ro = rowo[rr + e];
                    if (dv >= Dv || ro < 0) continue;
                    const size_t t = t0 + (ro >> 16);
                    const int h = hb0 + (ro & 0xffff);
                    if (a.splits > 1) a.ws[((t * a.H + h) * a.splits + blockIdx.z) * (Dv + 2) + 2 + dv] = v;
                    else {
                        if (gated) v *= 1.f / (1.f + expf(-gz[e]));
                        const size_t to = t * a.ldo + (size_t)h * Dv + dv;
                        if (a.out16) ((uint16_t*)a.out)[to] = f32_to_bf16_bits(v);
                        else a.out[to] = v;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == A_SOFT + 1) tmem_dealloc(tmem, p.tmem_cols);
    if (a.splits == 1) return;
    // ---------------- key slices: the block that arrives last folds the records (references in log2 units)
    unsigned* last = (unsigned*)wmax;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned* tk = a.tickets + (size_t)blockIdx.x * gridDim.y + blockIdx.y;
        const unsigned got = atomicAdd(tk, 1u);
        *last = got == (unsigned)a.splits - 1u;
        if (*last) *tk = 0u;
    }
    __syncthreads();
    if (!*last) return;
    __threadfence();
    float* wsl = (float*)(smem + (ring - q_s));          // [32][64]: the ring is done
    for (int r = warp; r < AR; r += A_THREADS / 32) {
        const int qi = r / HB, hh = r - qi * HB;
        if (qi >= nq || hh >= nh) continue;
        const float* rec = a.ws + ((size_t)(t0 + qi) * a.H + hb0 + hh) * a.splits * (Dv + 2);
        float ms[2], ls[2], M = -INFINITY;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int sp = lane + 32 * u;
            ms[u] = sp < a.splits ? __ldcg(rec + (size_t)sp * (Dv + 2)) : -INFINITY;
            ls[u] = sp < a.splits ? __ldcg(rec + (size_t)sp * (Dv + 2) + 1) : 0.f;
            M = fmaxf(M, ms[u]);
        }
        M = warp_max(M);
        float e[2], L = 0.f;
#pragma unroll
        for (int u = 0; u < 2; ++u) { e[u] = ms[u] == -INFINITY ? 0.f : exp2f(ms[u] - M); L += ls[u] * e[u]; }
        L = warp_sum(L);
        const float inv = L > 0.f ? 1.f / L : 0.f;
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (lane + 32 * u < a.splits) wsl[r * 64 + lane + 32 * u] = e[u] * inv;
    }
    __syncthreads();
    // pairs of elements (records start on 8 bytes), four per thread and round: one at a time, the loads' latency is all it does
    const int half_dv = Dv / 2, total = live * half_dv;
    for (int i0 = tid; i0 < total; i0 += 4 * A_THREADS) {
        const float2* src[4];
        float2 o[4];
        int row[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = i0 + q * A_THREADS, r = i / half_dv, ro = i < total ? rowo[r] : -1;
            row[q] = ro >= 0 ? r : -1;
            o[q] = make_float2(0.f, 0.f);
            src[q] = (const float2*)(a.ws + ((size_t)(t0 + (max(ro, 0) >> 16)) * a.H + hb0 + (max(ro, 0) & 0xffff)) * a.splits * (Dv + 2) + 2) +
                     (ro >= 0 ? i - r * half_dv : 0);
        }
#pragma unroll 4
        for (int sp = 0; sp < a.splits; ++sp)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float w = wsl[max(row[q], 0) * 64 + sp];
                const float2 v = __ldcg(src[q] + (size_t)sp * (half_dv + 1));
                o[q].x = fmaf(w, v.x, o[q].x);
                o[q].y = fmaf(w, v.y, o[q].y);
            }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (row[q] < 0) continue;
            const int ro = rowo[row[q]], dv = 2 * (i0 + q * A_THREADS - row[q] * half_dv), h = hb0 + (ro & 0xffff);
            const size_t t = t0 + (ro >> 16);
            const size_t to = t * a.ldo + (size_t)h * Dv + dv;
            if (a.gate) {
                o[q].x *= 1.f / (1.f + expf(-gate_logit(a, t, h, dv)));
                o[q].y *= 1.f / (1.f + expf(-gate_logit(a, t, h, dv + 1)));
            }
            o[q].x *= a.out_mult;
            o[q].y *= a.out_mult;
            if (a.out16) {
                ((uint16_t*)a.out)[to] = f32_to_bf16_bits(o[q].x);
                ((uint16_t*)a.out)[to + 1] = f32_to_bf16_bits(o[q].y);
            } else {
                a.out[to] = o[q].x;
                a.out[to + 1] = o[q].y;
            }
        }
    }
}

template <bool CAP, int SLOPE, bool PROB>
int launch_form(const TcAttnArgs& p, const CUtensorMap& kmap, const CUtensorMap& vmap, int tiles, size_t smem, cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        PGK_CUDA(cudaFuncSetAttribute(seq_attention_tc_kernel<CAP, SLOPE, PROB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        configured = true;
    }
    const int rep = p.a.H / p.a.G, hsplit = (rep + p.a.HB - 1) / p.a.HB;
    PGK_CUDA(launch_waiting(seq_attention_tc_kernel<CAP, SLOPE, PROB>, dim3(tiles, p.a.G * hsplit, p.a.splits), dim3(A_THREADS), smem, st, kmap, vmap, p));
    return 0;
}

size_t smem_bytes(int D) { return (size_t)((D + 63) / 64) * A_QCHUNK + A_PBYTES + A_RING * A_CHUNK + A_TAIL; }

// Copies of 16 bytes from rows of the cache; at most 512 value elements (TMEM) and 704 key elements (shared memory); positions are
// compared as float32, which holds whole numbers to 2^24.
bool sizes_fit(int D, int Dv, int kld, int vld, int HB, long long positions) {
    return D % 8 == 0 && Dv % 8 == 0 && kld % 8 == 0 && vld % 8 == 0 && Dv <= 512 && HB <= AR && smem_bytes(D) <= 227 * 1024 && positions <= 1 << 24;
}

}  // namespace

int seq_attention_tc(const AttnArgs& a, int tiles, cudaStream_t st, bool* served) {
    *served = false;
    if (!sizes_fit(a.D, a.Dv, a.kld, a.vld, a.HB, (long long)a.max_pages * a.PS) || (uintptr_t)a.kc % 16 || (uintptr_t)a.vc % 16) return 0;
    if (a.splits > 1 && (uintptr_t)a.ws % 8) return 0;    // the fold reads pairs
    TcAttnArgs p{};
    p.a = a;
    p.nd = (a.D + 63) / 64;
    p.nd2 = (p.nd + 1) & ~1;
    p.ndv = (a.Dv + 127) / 128;
    p.tmem_cols = AN + AN * p.ndv <= 256 ? 256 : 512;
    p.qvec = a.ld % 4 == 0 && a.q_off % 4 == 0 && (uintptr_t)a.proj % 16 == 0;
    const size_t smem = smem_bytes(a.D);
    // copies of bp positions: the largest power of two that divides a page
    CUtensorMap kmap{}, vmap{};
    int bp = a.PS & -a.PS;
    if (bp > AK) bp = AK;
    if (bp >= 8 && tma_encode_fn()) {
        const uint64_t rows = 1ull << 31;                 // cache rows: the table names only pages that exist
        if (tma_map_bf16_2d(&kmap, a.kc, (uint64_t)a.D, rows, (uint64_t)a.kld * 2, 64, (uint32_t)bp) &&
            tma_map_bf16_2d(&vmap, a.vc, (uint64_t)a.Dv, rows, (uint64_t)a.vld * 2, 64, (uint32_t)bp)) p.bp = bp;
    }
    p.err = wait_word(kWaitAttention);
    PGK_REQUIRE(p.err, "seq_attention failed: no pinned host memory");
    *served = true;
    switch ((a.cap > 0.f ? 1 : 0) + (a.slopes2 ? 4 : (a.slopes ? 2 : 0)) + (a.prob ? 6 : 0)) {
        case 0: return launch_form<false, 0, false>(p, kmap, vmap, tiles, smem, st);
        case 1: return launch_form<true, 0, false>(p, kmap, vmap, tiles, smem, st);
        case 2: return launch_form<false, 1, false>(p, kmap, vmap, tiles, smem, st);
        case 3: return launch_form<true, 1, false>(p, kmap, vmap, tiles, smem, st);
        case 4: return launch_form<false, 2, false>(p, kmap, vmap, tiles, smem, st);
        case 5: return launch_form<true, 2, false>(p, kmap, vmap, tiles, smem, st);
        case 6: return launch_form<false, 0, true>(p, kmap, vmap, tiles, smem, st);
        case 7: return launch_form<true, 0, true>(p, kmap, vmap, tiles, smem, st);
        case 8: return launch_form<false, 1, true>(p, kmap, vmap, tiles, smem, st);
        case 9: return launch_form<true, 1, true>(p, kmap, vmap, tiles, smem, st);
        case 10: return launch_form<false, 2, true>(p, kmap, vmap, tiles, smem, st);
        default: return launch_form<true, 2, true>(p, kmap, vmap, tiles, smem, st);
    }
}

}  // namespace pgk

extern "C" int pgk_seq_attention_tensor(int dim, int vdim, int k_ld, int v_ld, int heads, int kv_heads, int cache_dtype, long long positions) {
    return cache_dtype == 2 && dim > 0 && vdim > 0 && pgk::sizes_fit(dim, vdim, k_ld, v_ld, pgk_seq_heads_per_block(heads, kv_heads), positions) ? 1 : 0;
}
extern "C" int pgk_seq_attention_wait_error(int* out) {
    PGK_CUDA(cudaDeviceSynchronize());
    *out = 0;
    for (pgk::WaitKind k : {pgk::kWaitAttention, pgk::kWaitFew, pgk::kWaitPrompt, pgk::kWaitLinear})
        if (*out == 0) *out = pgk::wait_raised(k);
    return 0;
}
