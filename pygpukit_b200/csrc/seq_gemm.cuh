// seq_gemm.cuh -- what the products of the token-major models share: their argument block, the activations of the epilogues,
// and the entry of the tcgen05 form (seq_gemm_tc.cu).
#pragma once
#include "common.cuh"

namespace pgk {

struct GemmArgs {
    const float* A;
    const int* a_rows;
    const void* W;
    float* C;
    const int* group_off;
    const int* row_group;     // few-row form: weight matrix of every row (NULL: matrix 0)
    long long w_stride;       // elements between the weight matrices of consecutive groups
    int lda, ldc, M, N, K;
    float scale, cap;
    const float* colv;        // epilogue 4: [N] factors of the accumulated product
    const void* aux;          // epilogue 5: table [*, aux_ld] (float32 or bfloat16), entry (aux_rows[m], aux_off + n);
                              // epilogue 10: float32 gate rows, element (m, aux_off + C column)
    const int* aux_rows;
    int aux_ld, aux_off, aux_dt;
    long long a_z, c_z;       // batches: elements between the A columns / C columns of consecutive products
    int a16, c16;             // A / C are bfloat16 rows: what one product leaves and only the next one reads
    int ka;                   // elements of a row of A where the matrices were brought to a multiple of eight by zeros, K more (0: K)
};

__device__ __forceinline__ void move_a(GemmArgs& a, long long n) { a.A = a.a16 ? (const float*)((const uint16_t*)a.A + n) : a.A + n; }
__device__ __forceinline__ void move_c(GemmArgs& a, long long n) { a.C = a.c16 ? (float*)((uint16_t*)a.C + n) : a.C + n; }
__device__ __forceinline__ void put(const GemmArgs& a, size_t at, float v) {
    if (a.c16) ((uint16_t*)a.C)[at] = f32_to_bf16_bits(v);
    else a.C[at] = v;
}
__device__ __forceinline__ float a_at(const GemmArgs& a, size_t at) { return a.a16 ? bf16_bits_to_f32(((const uint16_t*)a.A)[at]) : a.A[at]; }
// four elements from an even multiple of four on (16-byte float32, 8-byte bfloat16 loads)
__device__ __forceinline__ float4 a_at4(const GemmArgs& a, size_t at) {
    if (!a.a16) return *(const float4*)(a.A + at);
    const uint2 v = *(const uint2*)((const uint16_t*)a.A + at);
    return make_float4(bf16lo(v.x), bf16hi(v.x), bf16lo(v.y), bf16hi(v.y));
}

__device__ __forceinline__ float gelu_tanh_f(float z) {
    return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float gelu_erf_f(float z) { return 0.5f * z * (1.f + erff(z * 0.7071067811865476f)); }
__device__ __forceinline__ float aux_at(const GemmArgs& a, int row, int col) {
    const size_t i = (size_t)a.aux_rows[row] * a.aux_ld + a.aux_off + col;
    return a.aux_dt == 2 ? bf16_bits_to_f32(((const uint16_t*)a.aux)[i]) : ((const float*)a.aux)[i];
}

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }

// The tcgen05 form of the many-row product (bfloat16 weights).  `batch`: independent products a.a_z / a.w_stride / a.c_z apart
// (a.group_off NULL), or the number of row groups; `rows`: rows of A (groups: an upper bound of group_off[groups]), `max_rows`:
// bound of the longest group.  *served is false, and nothing is launched, when the operands do not fit its copies.
int gemm_rows_tc(const GemmArgs& a, int epilogue, int batch, int rows, int max_rows, cudaStream_t st, bool* served);

// Where the kernel of few rows is faster than the rounding pass and the product of many rows: up to 32 rows, for which the weights are read once, and blocks of
// 32 that read them again out of L2 while the device has room for all of them at one time (us, many rows -> few, 24 rows: 512 x 512 8.9 -> 6.1, 2048 x
// 2048 19.1 -> 7.2, 8192 x 2048 26.9 -> 13.9, 2048 x 32768 27.2 -> 21.5; 2048 x 2048, 64 / 128 / 192 rows 20.1 -> 10.7, 23.2 -> 14.6, 13.3 -> 16.5; 8192 x 2048, 64
// / 128 rows 27.4 -> 23.4, 30.2 -> 47.0; 192 rows 1024 x 1024 10.5 -> 9.7, 512 x 4096 8.8 -> 7.6, 2048 x 8192 15.2 -> 30.6).
inline bool few_rows_pay(int M, int N, int K, int batch) {
    return M <= 32 || (M <= 256 && (double)batch * N * K * ((M + 31) / 32) <= 16777216.0);
}

// Matrices whose rows the copies cannot fetch, brought to 16-byte boundaries in work memory: *b is the product on them.  *done is false, and nothing is
// launched, without room for them.  (Inside a capture the room is had when the graph is made or launched, and that call fails without it.)
int pad_weights(const GemmArgs& a, int matrices, cudaStream_t st, GemmArgs* b, bool* done);

// The same for few rows, in one launch without work memory: `batch` products over the same rows, or blocks of rows_per_block (at most 32)
// rows that share the matrix a.row_group names.
int gemm_few_tc(const GemmArgs& a, int epilogue, int batch, int rows_per_block, cudaStream_t st, bool* served);

}  // namespace pgk
