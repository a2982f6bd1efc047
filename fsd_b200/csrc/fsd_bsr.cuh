// Block-sparse row products for the learned preconditioner (6x6 fp32 blocks):
// 16 or 32 lanes per row, on a matrix laid out by components.
//
// Row i with n blocks is 36 n contiguous floats; component r of the row's
// result is the dot product of 6 n consecutive floats (r 6n + 6 e + c for block
// e, column c) with the gathered operand (x_col(e), c).  A lane takes pairs of
// consecutive elements: it gathers one operand pair and multiplies it with the
// same place of the six components' runs, so each of its six loads is part of
// 128 contiguous bytes of the row's lanes.
//
// Latency- and L2-bound: products with G and A take 5.4 and 3.2 us at N = 8000,
// phi = 0.45.  Eight lanes per row on tiles streamed into shared memory by bulk
// copies took 7.2 and 4.2 us (each block's lines were looked up three times), a
// whole warp per row on this layout 5.7 and 4.2 (half its lanes idle).  Where
// the matrices no longer stay in L2 the whole warp is the faster form (the
// inner GMRES, N = 32768: 21.3 against 26.5 us with G).  Rows padded to whole
// chunks of 16 pairs cost 32 us there.
#pragma once

#include <cuda_runtime.h>

namespace fsd {

constexpr int kBsrRows = 2;  // rows per warp
__device__ __forceinline__ int bsr_sub() { return (threadIdx.x >> 4) & 1; }
// Component that a row's lane returns (six of its W lanes; else -1).
template <int W = 16>
__device__ __forceinline__ int bsr_component() {
    const int l = threadIdx.x & (W - 1), q = l / (W / 8);
    return l % (W / 8) == 0 && (q & 3) != 3 ? 3 * (q >> 2) + (q & 3) : -1;
}

// sum over the row's n blocks (0 for lanes without a row) of block * x_col in
// the component lanes; row = its 36 n floats, ld(j, k) loads operand pair k
// (components 2k, 2k + 1) of particle j.  All lanes of the warp take part.
template <int W = 16, class LD>
__device__ __forceinline__ float bsr_row(const float* row, const int* cols, int n, LD ld) {
    const int l = threadIdx.x & (W - 1);
    const int np = 3 * n;  // pairs per component
    unsigned long long acc[6] = {0, 0, 0, 0, 0, 0};
    const unsigned long long* m = reinterpret_cast<const unsigned long long*>(row) + l;
    for (int p = l; p < np; p += W, m += W) {
        unsigned long long g[6];
#pragma unroll
        for (int r = 0; r < 6; ++r) g[r] = m[r * np];
        const int e = p / 3;
        const float2 x = ld(cols[e], p - 3 * e);
        unsigned long long x2;
        asm("mov.b64 %0, {%1, %2};" : "=l"(x2) : "f"(x.x), "f"(x.y));
#pragma unroll
        for (int r = 0; r < 6; ++r) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r]) : "l"(g[r]), "l"(x2));
    }
    __syncwarp();
    float v[6];
#pragma unroll
    for (int r = 0; r < 6; ++r) {
        float2 t;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(t.x), "=f"(t.y) : "l"(acc[r]));
        v[r] = t.x + t.y;
    }
    // halving exchanges: components 0-2 and 3-5, then {0, 1} and {2}, then 0 and 1
    const bool h8 = l & (W / 2), h4 = l & (W / 4), h2 = l & (W / 8);
    float a[3], b[2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float keep = h8 ? v[3 + k] : v[k], send = h8 ? v[k] : v[3 + k];
        a[k] = keep + __shfl_xor_sync(0xffffffffu, send, W / 2);
    }
    {
        const float keep = h4 ? a[2] : a[0], send = h4 ? a[0] : a[2];
        b[0] = keep + __shfl_xor_sync(0xffffffffu, send, W / 4);
        b[1] = a[1] + __shfl_xor_sync(0xffffffffu, a[1], W / 4);  // wanted by the lower half
    }
    const float keep = (h2 && !h4) ? b[1] : b[0], send = (h2 || h4) ? b[0] : b[1];
    float s = keep + __shfl_xor_sync(0xffffffffu, send, W / 8);
#pragma unroll
    for (int o = W / 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Operand pairs of a plain 6N vector (8-byte aligned), and of the saddle
// input's difference t = b[0:6N] - b[11N:17N] (4-byte aligned).
struct BsrPlain {
    const float* x;
    __device__ __forceinline__ float2 operator()(int j, int k) const {
        return reinterpret_cast<const float2*>(x)[3 * j + k];
    }
};
struct BsrSaddle {
    const float* b;
    size_t off;  // 11 N
    __device__ __forceinline__ float2 operator()(int j, int k) const {
        const float* p = b + 6 * (size_t)j + 2 * k;
        return make_float2(p[0] - p[off], p[1] - p[off + 1]);
    }
};

}  // namespace fsd
