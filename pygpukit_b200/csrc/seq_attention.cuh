// seq_attention.cuh -- the argument block and the small rules that the attention kernels of the token-major models share.
#pragma once
#include "common.cuh"

namespace pgk {

struct AttnArgs {
    const float* proj; int ld, q_off, g_off;
    float* out; int ldo;
    const void* kc; const void* vc; const int* table; int max_pages, PS;
    const float* gsrc; int ldg;         // rows the gate is read from (gate 1: g_off + h * Dv + dv, gate 2: g_off + h)
    const float* sinks;                 // [H] or NULL: a score per head that joins the denominator and has no value
    int window;                         // > 0: key j is visible from i only when i - j < window
    int kld, vld;                       // elements between consecutive positions' rows in the K / V arrays
    int valias;                         // the value rows are the first Dv elements of the key rows (one staging)
    const int4* tiles;                  // (first token row, queries, slot, first position)
    const float* slopes;                // [H] or NULL
    const float* slopes2;               // [H] or NULL: the distance term is slopes[h] * ln(1 + slopes2[h] * (i - j)) instead
    int keep;                           // with a window: the first `keep` positions stay visible beyond it
    int prob;                           // 0: softmax over the visible keys; 1: weight sigmoid(score + pbias[h]), not normalised
    const float* pbias;                 // [H] or NULL
    float out_mult;                     // constant factor on the output
    int H, G, D, Dv, chunk, HB, gate;
    float scale, cap;
    int splits; float* ws;              // splits > 1: partial (m, l, acc[Dv]) records [row][H][splits][Dv + 2]
    unsigned* tickets;                  // one arrival counter per (tile, head block), zero between launches
    int pool, pool_rows;                // pool > 0 (with a window): means of blocks of `pool` positions, rows per page of pk / pv
    const void* pk; const void* pv;     // [pages][G][pool_rows][D] / [Dv], dense rows
    const double* o_inv_freq;           // [Dv / 2] or NULL: pair m of an output (elements m and m + Dv / 2, or 2m and 2m + 1
    int o_pairs;                        // with o_pairs) turns by -position * o_inv_freq[m]
    int out16;                          // bfloat16 outputs (tensor cores): rows that only a product reads, which rounds them so
};

__device__ __forceinline__ float gate_logit(const AttnArgs& a, size_t t, int h, int dv) {
    return a.gsrc[t * a.ldg + a.g_off + (a.gate == 2 ? (size_t)h : (size_t)h * a.Dv + dv)];
}
__device__ __forceinline__ int first_key(const AttnArgs& a, int pos) {
    int lo = a.chunk > 0 ? (pos / a.chunk) * a.chunk : 0;
    if (a.window > 0) lo = max(lo, pos - a.window + 1);
    return lo;
}
__device__ __forceinline__ float distance_term(float slope, float slope2, bool log_form, int dist) {
    const float d = (float)max(dist, 0);
    return log_form ? slope * log1pf(slope2 * d) : slope * d;
}

// The tensor-core form for prompts and portions (seq_attention_tc.cu): bfloat16 cache, softmax or sigmoid weights, windows, kept
// positions, chunks, distance terms, sinks, gates, key slices.  *served is false, and nothing is launched, when the operands do
// not fit its copies or the on-chip memory.
int seq_attention_tc(const AttnArgs& a, int tiles, cudaStream_t st, bool* served);

// Decoding (seq_attention_few.cu): bfloat16 cache, softmax weights, windows, chunks, distance terms, sinks, gates; `cluster` blocks share a
// request's keys.
int seq_attention_few(const AttnArgs& a, int tiles, int cluster, cudaStream_t st, bool* served);

}  // namespace pgk
