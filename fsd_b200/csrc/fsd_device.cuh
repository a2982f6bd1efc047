// Device helpers shared by the kernels: periodic box arithmetic, table
// interpolation and warp/group reductions.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fsd_internal.h"

namespace fsd {

// Minimum image with an xy tilt, rint based (HOOMD BoxDim::minImage, device path).
__device__ __forceinline__ float3 min_image(float3 w, const Box& b) {
    float img = rintf(w.z * (1.0f / b.Lz));
    w.z -= b.Lz * img;
    img = rintf(w.y * (1.0f / b.Ly));
    w.x -= b.Ly * b.xy * img;
    w.y -= b.Ly * img;
    w.x -= b.Lx * rintf(w.x * (1.0f / b.Lx));
    return w;
}

// Pair separation j - i (or i - j) and its squared length evaluated without
// fused multiply-adds, so that separations and gaps are the correctly rounded
// single-precision values of the reference's arithmetic (minImage, dot,
// sqrtf).  Near contact the lubrication functions are steep in the gap, so
// this rounding is part of the result.
__device__ __forceinline__ float3 min_image_rn(float3 w, const Box& b) {
    float img = rintf(__fmul_rn(w.z, 1.0f / b.Lz));
    w.z = __fsub_rn(w.z, __fmul_rn(b.Lz, img));
    img = rintf(__fmul_rn(w.y, 1.0f / b.Ly));
    w.x = __fsub_rn(w.x, __fmul_rn(__fmul_rn(b.Ly, b.xy), img));
    w.y = __fsub_rn(w.y, __fmul_rn(b.Ly, img));
    w.x = __fsub_rn(w.x, __fmul_rn(b.Lx, rintf(__fmul_rn(w.x, 1.0f / b.Lx))));
    return w;
}

__device__ __forceinline__ float dist2_rn(float3 r) {
    return __fadd_rn(__fadd_rn(__fmul_rn(r.x, r.x), __fmul_rn(r.y, r.y)), __fmul_rn(r.z, r.z));
}

// Fractional coordinates in [0,1) of the sheared box (HOOMD BoxDim::makeFraction).
__device__ __forceinline__ float3 make_fraction(float3 v, const Box& b) {
    float3 d = make_float3(v.x + b.Lx / 2, v.y + b.Ly / 2, v.z + b.Lz / 2);
    d.x -= b.xy * v.y;
    return make_float3(d.x / b.Lx, d.y / b.Ly, d.z / b.Lz);
}

// Wrap a position back into the box, updating its image (HOOMD BoxDim::wrap).
__device__ __forceinline__ void wrap_position(float3& w, int3& img, const Box& b) {
    const float tilt_x = b.xy * w.y;
    if (w.x >= b.Lx / 2 + tilt_x) { w.x -= b.Lx; img.x++; }
    else if (w.x < -b.Lx / 2 + tilt_x) { w.x += b.Lx; img.x--; }
    if (w.y >= b.Ly / 2) { w.y -= b.Ly; w.x -= b.Ly * b.xy; img.y++; }
    else if (w.y < -b.Ly / 2) { w.y += b.Ly; w.x += b.Ly * b.xy; img.y--; }
    if (w.z >= b.Lz / 2) { w.z -= b.Lz; img.z++; }
    else if (w.z < -b.Lz / 2) { w.z += b.Lz; img.z--; }
}

// 32 bytes in one load (32-byte aligned).  A gather costs the L1 one tag lookup
// per lane and instruction, so records of 32 bytes take half the lookups of two
// float4.  Volatile, so it stays behind pdl_wait(); the kernel must not write
// what it reads.  load8_const: tables that no overlapped kernel writes.
__device__ __forceinline__ void load8(const float* p, float* v) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ void load8_const(const float* p, float* v) {
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

// Interpolated near-field resistance scalars [first, first+count) of the table
// row bracketing distance r.  Pairs at r <= 2.001 use the regularised row 232
// (Lubrication.cu:172-186).  Beyond the last tabulated gap the index reaches
// row 999 whose values are zero; those pairs contribute nothing, which is what
// the reference's read past the last row yields as well.
template <int COUNT>
__device__ __forceinline__ void res_interp(const ResTable& t, float r, int first, float* out) {
    if ((double)r <= 2.001) {
        const float* v = t.vals + 232 * kResFuncs + first;
#pragma unroll
        for (int c = 0; c < COUNT; ++c) out[c] = __ldg(v + c);
        return;
    }
    const float s = (float)(((double)r - 2.0) / (double)kResMin);
    const int ind = (int)(log10f(s) / kResDr);
    if (ind >= kResRows - 1) {
#pragma unroll
        for (int c = 0; c < COUNT; ++c) out[c] = 0.0f;
        return;
    }
    const float dl = __ldg(t.dist + ind), du = __ldg(t.dist + ind + 1);
    const float fac = (r - dl) / (du - dl);
    const float* lo = t.vals + ind * kResFuncs + first;
    const float* hi = lo + kResFuncs;
#pragma unroll
    for (int c = 0; c < COUNT; ++c) {
        const float a = __ldg(lo + c), b = __ldg(hi + c);
        out[c] = a + (b - a) * fac;
    }
}

// Sum over aligned groups of G lanes (G a power of two <= 32).
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int G>
__device__ __forceinline__ double group_sum_d(double v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Last-block reduction: the threads that wrote this block's partials have
// fenced them; the block that takes the last ticket sees every block's
// partials, and the caller resets the ticket there.
__device__ __forceinline__ bool last_block(unsigned* ticket) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Sum of part[0:n] in a fixed order by one warp (same result every run).
__device__ __forceinline__ double warp_sum_parts(const double* part, int n) {
    double s = 0.0;
    for (int b = threadIdx.x & 31; b < n; b += 256) {  // eight loads in flight, added in the same order
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = b + 32 * k < n ? __ldcg(part + b + 32 * k) : 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) s += v[k];
    }
    return group_sum_d<32>(s);
}

// Block sum of v written (and fenced) to part[blockIdx.x].
__device__ __forceinline__ void block_partial(double v, double* part) {
    __shared__ double sh[32];
    v = group_sum_d<32>(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0;
        t = group_sum_d<32>(t);
        if (threadIdx.x == 0) {
            part[blockIdx.x] = t;
            __threadfence();
        }
    }
}

// Launches that begin while their predecessor in the stream drains.  Kernels
// launched this way call pdl_wait() first: it returns once the previous kernel
// has completed and its writes are visible (at once in an ordinary launch), and
// lets the next kernel's blocks come up meanwhile.  Dispatch and block start-up,
// about a microsecond per launch, then overlap the previous kernel.  Every
// thread waits before anything else, so a kernel's completion implies that of
// all before it.
//
// Such a kernel's lifetime begins while its predecessor still writes, so data
// from the stream is read by ordinary loads: no __ldg and no ld.global.nc, which
// presume data that does not change meanwhile, and no __restrict__ pointer, whose
// accesses a compiler may move across the wait.  What is written once, or by
// launches that are not overlapped (tables, the matrix A of the inner GMRES), may
// go the read-only way.
//
// Grids of more than two blocks per SM are launched the ordinary way: blocks
// that come up early crowd the SMs that have room, and the overlap is short
// beside the kernel.  A step at N = 500 went from 11993 to 9860 us and a
// mobility call at N = 1000 from 66 to 52; with every launch overlapped, the
// polynomial solve at N = 8000 took 13.8 ms instead of 12.7 and a step at
// N = 32768 127 instead of 121.
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
constexpr unsigned kPdlBlocks = 2 * 148;
template <class... P, class... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = grid.x * grid.y * grid.z <= kPdlBlocks;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &attr;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, P(args)...);  // errors are read by the caller's cudaGetLastError
}

// Exclusive scan of count[0:n] into start[0:n] (start[n] = total) by one block
// of up to 1024 threads; count is padded to a multiple of 16 and read past the
// L1 (other blocks' atomics).
__device__ __forceinline__ void block_scan_counts(const unsigned* count, unsigned* start, int n) {
    __shared__ unsigned sh[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned carry = 0;
    for (int base = 0; base < n; base += 16 * blockDim.x) {
        const int c0 = base + 16 * threadIdx.x;
        unsigned v[16], sum = 0;
#pragma unroll
        for (int k = 0; k < 16; k += 4) {
            const uint4 q = c0 + k < n ? __ldcg(reinterpret_cast<const uint4*>(count + c0 + k))
                                       : make_uint4(0u, 0u, 0u, 0u);
            v[k] = q.x;
            v[k + 1] = q.y;
            v[k + 2] = q.z;
            v[k + 3] = q.w;
            sum += q.x + q.y + q.z + q.w;
        }
        unsigned x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) sh[wid] = x;
        __syncthreads();
        unsigned before = 0, all = 0;
        for (int k = 0; k < nw; ++k) {
            if (k < wid) before += sh[k];
            all += sh[k];
        }
        unsigned off = carry + before + x - sum;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            if (c0 + k < n) start[c0 + k] = off;
            off += v[k];
        }
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) start[n] = carry;
}

}  // namespace fsd
