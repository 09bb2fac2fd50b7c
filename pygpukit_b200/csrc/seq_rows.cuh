// seq_rows.cuh -- rows in registers: loads, stores and sums that the row kernels of the token-major models share.
//
// A thread keeps its share of the row in registers: all loads of a row go out together -- weights and the rows that the result joins among
// them -- and one or two barriers later it is stored; what bounds a step's few rows is that chain, a prompt's the memory.  Two groups of
// four elements per thread, four in long rows (VEC: 16-byte accesses; else four strided elements); the number of threads follows from the
// width alone, so that a row's sum has the same order whatever rows share the launch.  Against loops of single elements through shared
// memory (B200, us, rows of 2048, cold caches): LayerNorm joined to 2000 rows 28.4 -> 11.8, of one 11.6 -> 4.3; RMS norm of 2000 rows
// 15.8 -> 9.2, of 8 8.7 -> 3.4; two norms of a seam over 8 rows 13.0 -> 3.7; embedding and norm of 2000 rows 15.5 -> 7.4.
#pragma once
#include <initializer_list>

#include "common.cuh"

namespace pgk {

constexpr int ROW_THREADS = 512;
constexpr int ROW_G = 2, ROW_G2 = 4;             // groups per thread: rows of up to 4096 elements, of up to 8192

template <bool VEC, int G> __device__ __forceinline__ int row_at(int g, int e) {
    return VEC ? ((int)threadIdx.x + g * (int)blockDim.x) * 4 + e : (int)threadIdx.x + (g * 4 + e) * (int)blockDim.x;
}
template <bool VEC, int G> __device__ __forceinline__ void row_load(float (&v)[4 * G], const float* p, int W) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (VEC) {
            const int i = row_at<VEC, G>(g, 0);
            *(float4*)&v[4 * g] = i < W ? *(const float4*)(p + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) { const int i = row_at<VEC, G>(g, e); v[4 * g + e] = i < W ? p[i] : 0.f; }
        }
    }
}
template <bool VEC, int G> __device__ __forceinline__ void row_load(float (&v)[4 * G], const uint16_t* p, int W) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (VEC) {
            const int i = row_at<VEC, G>(g, 0);
            const uint2 u = i < W ? *(const uint2*)(p + i) : make_uint2(0u, 0u);
            v[4 * g] = bf16lo(u.x); v[4 * g + 1] = bf16hi(u.x); v[4 * g + 2] = bf16lo(u.y); v[4 * g + 3] = bf16hi(u.y);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) { const int i = row_at<VEC, G>(g, e); v[4 * g + e] = i < W ? bf16_bits_to_f32(p[i]) : 0.f; }
        }
    }
}
template <bool VEC, int G> __device__ __forceinline__ void row_store(float* p, const float (&v)[4 * G], int W) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (VEC) {
            const int i = row_at<VEC, G>(g, 0);
            if (i < W) *(float4*)(p + i) = *(const float4*)&v[4 * g];
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) { const int i = row_at<VEC, G>(g, e); if (i < W) p[i] = v[4 * g + e]; }
        }
    }
}
__device__ __forceinline__ float row_total(const float* red) {
    const int lane = threadIdx.x & 31;
    return warp_sum(lane < ((int)blockDim.x >> 5) ? red[lane] : 0.f);
}
// the sum over the block; red: 32 floats that nothing else uses until the next barrier but one
__device__ __forceinline__ float row_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    return row_total(red);
}
// the same for two sums behind one barrier
__device__ __forceinline__ void row_sums(float v, float u, float (*red)[32]) {
    v = warp_sum(v);
    u = warp_sum(u);
    if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = v; red[1][threadIdx.x >> 5] = u; }
    __syncthreads();
}
template <int N> __device__ __forceinline__ float square_sum(const float (&v)[N]) {
    float q = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) q = fmaf(v[j], v[j], q);
    return q;
}

// four cached elements
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) { *(float4*)p = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(uint16_t* p, const float (&v)[4]) { *(uint2*)p = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3])); }
__device__ __forceinline__ void store1(float* p, float v) { *p = v; }
__device__ __forceinline__ void store1(uint16_t* p, float v) { *p = f32_to_bf16_bits(v); }

// threads of a block whose row has `width` elements, G groups of four in each
inline int row_threads(int width, int G) {
    const int nt = ((width + 4 * G - 1) / (4 * G) + 31) / 32 * 32;
    return nt < 64 ? 64 : (nt > ROW_THREADS ? ROW_THREADS : nt);
}
inline bool row_vec(int width, std::initializer_list<const void*> ptrs) {
    uintptr_t all = 0;
    for (const void* p : ptrs) all |= (uintptr_t)p;
    return width % 4 == 0 && all % 16 == 0;
}

}  // namespace pgk
