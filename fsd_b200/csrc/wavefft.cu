// Transforms and Green's function of the wave-space mobility for grids whose
// lines factor as N1 * N2 with register-sized radices (fsd_dft.cuh).
//
// The 11 real grids travel as 6 packed complex grids.  The y and z passes of
// one (grid, x) plane run in one kernel with the plane in shared memory; it
// then splits each packed plane into the half spectra (z <= Nz / 2) of its two
// real grids, A(k) = (C(k) + conj C(-k)) / 2 and B(k) = -i (C(k) - conj C(-k)) / 2
// over the in-plane mirror k = (y, z).  So the x pass needs no mirror lines:
// each of its points applies the Green's function to its own 11 spectra, and
// its z runs start on 32-byte sectors.
//
// What bounds it: at 72^3 a pass moves 18 MB in and 18 MB out, all in L2 (4 us
// at its bandwidth); the rest is shared-memory passes and arithmetic.  The
// radices are factored (a line of 72 takes about 1500 operations, 3900 as full
// radix-8 and radix-9 matrix sums), the first and last stages of an axis go
// between global memory and registers, and the x pass reads the Green factors
// from a table instead of evaluating sin, cos and FP64 products per point.
// Measured per call, before (plane kernel for 72, 36 and 27, generic Stockham
// lines elsewhere) and after: 72^3 y+z 21.6 -> 13.9 us forward, 12.8 us
// inverse, x pass 51.4 -> 20.4 us; 120^3 y+z 249 -> 70 and 67 us, x pass
// 318 -> 76 us; 27^3 y+z 5.6 -> 4.6 and 4.2 us, x pass 10.2 -> 4.6 us.
// The generic lines are kept for lengths without two register-sized factors
// (125, 162), for boxes with Ny != Nz and for lengths above 150: a plane of 160
// (16 x 10, 220 KB) would be the last to fit in shared memory, and has no kernel.
#include "fsd_device.cuh"
#include "fsd_dft.cuh"
#include "fsd_green.cuh"
#include "fsd_kernels.cuh"
#include "fsd_profile.h"
#include "fsd_wavefft.h"

namespace fsd {

namespace {

// A line of N = N1 * N2 in shared memory: element n1 + N1 q sits at
// n1 + GP q.  The N2-point DFTs run over q for fixed n1 (with the roots
// w_N^(n1 k2) after them), the N1-point DFTs over n1 for fixed k2, each in
// place, so coefficient k2 + N2 k1 ends at GP k2 + k1.  GP is N1 made odd:
// walking the coefficients in order then strides by an odd number of float2.
template <int N1_, int N2_>
struct Line {
    static constexpr int N1 = N1_, N2 = N2_, N = N1 * N2, GP = N1 | 1;
    static constexpr int LEN = N2 * GP;
    static constexpr int RS = LEN | 1;  // line stride, odd
    __device__ static __forceinline__ int slot(int k) { return (k % N2) * GP + k / N2; }
    __device__ static __forceinline__ int natural(int n) { return (n / N1) * GP + n % N1; }
};

// Threads for `tasks` register DFTs per stage: as few rounds of at most
// `cap` threads as they need, evenly filled.
constexpr int stage_threads(int tasks, int cap) {
    const int rounds = (tasks + cap - 1) / cap;
    return ((tasks + rounds - 1) / rounds + 31) / 32 * 32;
}

template <class L>
struct Plane {
    static constexpr int tasks = L::N * (L::N1 > L::N2 ? L::N1 : L::N2);
    static constexpr int threads = stage_threads(tasks, L::N >= 90 ? 640 : 384);
    static constexpr size_t smem = sizeof(float2) * (L::N + (size_t)L::N * L::RS);
};

// The N2-point stage along one axis of the plane for lines l = 0..N-1 (the
// other axis' coordinate is lane-fastest), in shared memory.
template <class L, bool INV, bool ROWS>
__device__ __forceinline__ void stage_n2(float2* pl, const float2* tw) {
    constexpr int es = ROWS ? 1 : L::RS, ls = ROWS ? L::RS : 1;
    for (int t = threadIdx.x; t < L::N * L::N1; t += blockDim.x) {
        const int l = t % L::N, n1 = t / L::N;
        float2* p = pl + l * ls + n1 * es;
        float2 y[L::N2];
#pragma unroll
        for (int q = 0; q < L::N2; ++q) y[q] = p[q * (ROWS ? L::GP : L::N1) * es];
        dft<L::N2, INV>(y);
        p[0] = y[0];
#pragma unroll
        for (int q = 1; q < L::N2; ++q) p[q * (ROWS ? L::GP : L::N1) * es] = c_twiddle<INV>(y[q], tw[n1 * q]);
    }
    __syncthreads();
}

template <class L, bool INV, bool ROWS>
__device__ __forceinline__ void stage_n1(float2* pl) {
    constexpr int es = ROWS ? 1 : L::RS, ls = ROWS ? L::RS : 1;
    for (int t = threadIdx.x; t < L::N * L::N2; t += blockDim.x) {
        const int l = t % L::N, k2 = t / L::N;
        float2* p = pl + l * ls + k2 * (ROWS ? L::GP : L::N1) * es;
        float2 y[L::N1];
#pragma unroll
        for (int q = 0; q < L::N1; ++q) y[q] = p[q * es];
        dft<L::N1, INV>(y);
#pragma unroll
        for (int q = 0; q < L::N1; ++q) p[q * es] = y[q];
    }
    __syncthreads();
}

// Plane layout: row y (stride RS), element z along the row.  Rows are not
// padded within the y axis: coefficient y = k2 + N2 k1 ends in row k2 N1 + k1.
template <class L>
__device__ __forceinline__ int row_slot(int k) {
    return (k % L::N2) * L::N1 + k / L::N2;
}

// Within a row the z coordinate is stored at natural(z) before the z stages.
// Lines of the y stages are the columns, whose lane-fastest index is the
// stored position; positions that are padding (natural() skips them) are
// never used.
template <class L>
__global__ void __launch_bounds__(Plane<L>::threads) k_yz_fwd(const float2* grid, float2* spec,
                                                              int Nx, int zp, const float2* __restrict__ tw_global) {
    pdl_wait();
    constexpr int N = L::N;
    extern __shared__ float2 smem[];
    float2* tw = smem;
    float2* pl = smem + N;
    for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = tw_global[i];
    const int p = blockIdx.x / Nx, x = blockIdx.x - p * Nx;
    const float2* in = grid + (size_t)blockIdx.x * N * N;
    __syncthreads();
    // y axis, N2-point stage straight from global memory
    for (int t = threadIdx.x; t < N * L::N1; t += blockDim.x) {
        const int z = t % N, n1 = t / N;
        float2 y[L::N2];
#pragma unroll
        for (int q = 0; q < L::N2; ++q) y[q] = in[(n1 + L::N1 * q) * N + z];
        dft<L::N2, false>(y);
        float2* o = pl + n1 * L::RS + L::natural(z);
        o[0] = y[0];
#pragma unroll
        for (int q = 1; q < L::N2; ++q) o[q * L::N1 * L::RS] = c_twiddle<false>(y[q], tw[n1 * q]);
    }
    __syncthreads();
    // y axis, N1-point stage (columns at their stored positions)
    for (int t = threadIdx.x; t < N * L::N2; t += blockDim.x) {
        const int z = t % N, k2 = t / N;
        float2* q0 = pl + k2 * L::N1 * L::RS + L::natural(z);
        float2 y[L::N1];
#pragma unroll
        for (int q = 0; q < L::N1; ++q) y[q] = q0[q * L::RS];
        dft<L::N1, false>(y);
#pragma unroll
        for (int q = 0; q < L::N1; ++q) q0[q * L::RS] = y[q];
    }
    __syncthreads();
    stage_n2<L, false, true>(pl, tw);
    stage_n1<L, false, true>(pl);
    // split into the half spectra of the two real grids
    const int nz = N / 2 + 1;
    const size_t fs = (size_t)Nx * N * zp;
    float2* oa = spec + (size_t)packA(p) * fs + (size_t)x * N * zp;
    float2* ob = packB(p) >= 0 ? spec + (size_t)packB(p) * fs + (size_t)x * N * zp : nullptr;
    for (int e = threadIdx.x; e < N * nz; e += blockDim.x) {
        const int y = e / nz, z = e - y * nz;
        const int ym = y ? N - y : 0, zm = z ? N - z : 0;
        const float2 c = pl[row_slot<L>(y) * L::RS + L::slot(z)];
        const float2 m = pl[row_slot<L>(ym) * L::RS + L::slot(zm)];
        oa[y * zp + z] = make_float2(0.5f * (c.x + m.x), 0.5f * (c.y - m.y));
        if (ob) ob[y * zp + z] = make_float2(0.5f * (c.y + m.y), -0.5f * (c.x - m.x));
    }
}

template <class L>
__global__ void __launch_bounds__(Plane<L>::threads) k_yz_inv(const float2* spec, float2* grid,
                                                              int Nx, int zp, const float2* __restrict__ tw_global) {
    pdl_wait();
    constexpr int N = L::N;
    extern __shared__ float2 smem[];
    float2* tw = smem;
    float2* pl = smem + N;
    for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = tw_global[i];
    const int p = blockIdx.x / Nx, x = blockIdx.x - p * Nx;
    const int nz = N / 2 + 1;
    const size_t fs = (size_t)Nx * N * zp;
    const float2* ia = spec + (size_t)packA(p) * fs + (size_t)x * N * zp;
    const float2* ib = packB(p) >= 0 ? spec + (size_t)packB(p) * fs + (size_t)x * N * zp : nullptr;
    // C(k) = A + i B and C(-k) = conj A + i conj B
    for (int e = threadIdx.x; e < N * nz; e += blockDim.x) {
        const int y = e / nz, z = e - y * nz;
        const float2 a = ia[y * zp + z];
        const float2 b = ib ? ib[y * zp + z] : make_float2(0.f, 0.f);
        pl[y * L::RS + L::natural(z)] = make_float2(a.x - b.y, a.y + b.x);
        if (z > 0 && 2 * z < N)
            pl[(y ? N - y : 0) * L::RS + L::natural(N - z)] = make_float2(a.x + b.y, b.x - a.y);
    }
    __syncthreads();
    stage_n2<L, true, true>(pl, tw);
    stage_n1<L, true, true>(pl);
    // y axis over the columns at their stored positions
    for (int t = threadIdx.x; t < N * L::N1; t += blockDim.x) {
        const int z = t % N, n1 = t / N;
        float2* q0 = pl + n1 * L::RS + L::natural(z);
        float2 y[L::N2];
#pragma unroll
        for (int q = 0; q < L::N2; ++q) y[q] = q0[q * L::N1 * L::RS];
        dft<L::N2, true>(y);
        q0[0] = y[0];
#pragma unroll
        for (int q = 1; q < L::N2; ++q) q0[q * L::N1 * L::RS] = c_twiddle<true>(y[q], tw[n1 * q]);
    }
    __syncthreads();
    // last stage straight to global memory: column z (stored at slot(z)), coefficient y = k2 + N2 q
    float2* out = grid + (size_t)blockIdx.x * N * N;
    for (int t = threadIdx.x; t < N * L::N2; t += blockDim.x) {
        const int z = t % N, k2 = t / N;
        const float2* q0 = pl + k2 * L::N1 * L::RS + L::slot(z);
        float2 y[L::N1];
#pragma unroll
        for (int q = 0; q < L::N1; ++q) y[q] = q0[q * L::RS];
        dft<L::N1, true>(y);
#pragma unroll
        for (int q = 0; q < L::N1; ++q) out[(k2 + L::N2 * q) * N + z] = y[q];
    }
}

// x pass.  A block holds the x lines of kXz consecutive z at one y, for all
// 11 fields: line l = f * kXz + zz.
constexpr int kXz = 4;  // one 32-byte sector of float2
constexpr int kXLines = 11 * kXz;

template <class L>
struct XPass {
    static constexpr int tasks = kXLines * (L::N1 > L::N2 ? L::N1 : L::N2);
    static constexpr int threads = stage_threads(tasks, 256);
    static constexpr int blocks = 65536 / (threads * 72);  // 72 registers: three blocks of 256, four of 224
    static constexpr size_t smem = sizeof(float2) * (L::N + (size_t)kXLines * L::RS);
};

template <class L, bool GREEN>
__global__ void __launch_bounds__(XPass<L>::threads, XPass<L>::blocks) k_x_pass(float2* spec, const float4* __restrict__ table,
                                                              const float4* __restrict__ gridk, int Ny, int Nz, int zp,
                                                              const float2* __restrict__ tw_global) {
    pdl_wait();
    constexpr int N = L::N;
    extern __shared__ float2 smem[];
    float2* tw = smem;
    float2* a = smem + N;
    for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = tw_global[i];
    const int nzc = zp / kXz;
    const int y = blockIdx.x / nzc, z0 = (blockIdx.x - y * nzc) * kXz;
    const int nzh = Nz / 2 + 1;
    const size_t xs = (size_t)Ny * zp, fs = (size_t)N * xs;
    float2* base = spec + (size_t)y * zp + z0;
    __syncthreads();
    if (GREEN) {
        // forward N2-point stage straight from global memory
        for (int t = threadIdx.x; t < kXLines * L::N1; t += blockDim.x) {
            const int l = t % kXLines, n1 = t / kXLines;
            const int f = l / kXz, zz = l - f * kXz;
            if (z0 + zz >= nzh) continue;  // padding
            const float2* g = base + (size_t)f * fs + zz + (size_t)n1 * xs;
            float2 v[L::N2];
#pragma unroll
            for (int q = 0; q < L::N2; ++q) v[q] = g[(size_t)q * L::N1 * xs];
            dft<L::N2, false>(v);
            float2* o = a + l * L::RS + n1;
            o[0] = v[0];
#pragma unroll
            for (int q = 1; q < L::N2; ++q) o[q * L::GP] = c_twiddle<false>(v[q], tw[n1 * q]);
        }
        __syncthreads();
        for (int t = threadIdx.x; t < kXLines * L::N2; t += blockDim.x) {
            const int l = t % kXLines, k2 = t / kXLines;
            if (z0 + l % kXz >= nzh) continue;
            float2* o = a + l * L::RS + k2 * L::GP;
            float2 v[L::N1];
#pragma unroll
            for (int q = 0; q < L::N1; ++q) v[q] = o[q];
            dft<L::N1, false>(v);
#pragma unroll
            for (int q = 0; q < L::N1; ++q) o[q] = v[q];
        }
        __syncthreads();
        // Green's function; on Nyquist planes averaged with the mirror point's
        // operator (whose wave vector is not -k there), which reproduces the real
        // part the reference keeps after its complex inverse transform
        for (int t = threadIdx.x; t < kXz * N; t += blockDim.x) {
            const int zz = t % kXz, s = t / kXz;
            const int z = z0 + zz;
            if (z >= nzh) continue;
            const int k2 = s / L::N1, k1 = s - k2 * L::N1;
            const int x = k2 + L::N2 * k1;
            const size_t pt = ((size_t)x * Ny + y) * zp + z;
            const float4 kv = table[2 * pt], gf = table[2 * pt + 1];
            float2* c = a + zz * L::RS + k2 * L::GP + k1;
            float2 f[11], o[11];
#pragma unroll
            for (int q = 0; q < 11; ++q) f[q] = c[q * kXz * L::RS];
            GreenFactors g;
            g.uf = gf.x;
            g.df = gf.y;
            g.dc = gf.z;
            g.ik2 = kv.w;
            const bool nyq = 2 * x == N || 2 * y == Ny || 2 * z == Nz;
            green_apply(kv.x, kv.y, kv.z, g, f, o, 1.0f);
            const float half = nyq ? 0.5f : 1.0f;
#pragma unroll
            for (int q = 0; q < 11; ++q) c[q * kXz * L::RS] = make_float2(half * o[q].x, half * o[q].y);
            if (nyq) {
                const int xm = x ? N - x : 0, ym = y ? Ny - y : 0, zm = z ? Nz - z : 0;
                green_apply(gridk[((size_t)xm * Ny + ym) * Nz + zm], f, o, -1.0f);
#pragma unroll
                for (int q = 0; q < 11; ++q) {
                    const float2 v = c[q * kXz * L::RS];
                    c[q * kXz * L::RS] = make_float2(fmaf(0.5f, o[q].x, v.x), fmaf(0.5f, o[q].y, v.y));
                }
            }
        }
    } else {
        for (int t = threadIdx.x; t < kXLines * N; t += blockDim.x) {
            const int l = t % kXLines, x = t / kXLines;
            const int f = l / kXz, zz = l - f * kXz;
            if (z0 + zz < nzh) a[l * L::RS + L::slot(x)] = base[(size_t)f * fs + zz + (size_t)x * xs];
        }
    }
    __syncthreads();
    // inverse: the adjoint stages in reverse order, from coefficient order back to natural order
    for (int t = threadIdx.x; t < kXLines * L::N2; t += blockDim.x) {
        const int l = t % kXLines, k2 = t / kXLines;
        if (z0 + l % kXz >= nzh) continue;
        float2* o = a + l * L::RS + k2 * L::GP;
        float2 v[L::N1];
#pragma unroll
        for (int q = 0; q < L::N1; ++q) v[q] = o[q];
        dft<L::N1, true>(v);
        o[0] = v[0];
#pragma unroll
        for (int q = 1; q < L::N1; ++q) o[q] = c_twiddle<true>(v[q], tw[q * k2]);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kXLines * L::N1; t += blockDim.x) {
        const int l = t % kXLines, n1 = t / kXLines;
        const int f = l / kXz, zz = l - f * kXz;
        if (z0 + zz >= nzh) continue;
        const float2* o = a + l * L::RS + n1;
        float2 v[L::N2];
#pragma unroll
        for (int q = 0; q < L::N2; ++q) v[q] = o[q * L::GP];
        dft<L::N2, true>(v);
        float2* g = base + (size_t)f * fs + zz + (size_t)n1 * xs;
#pragma unroll
        for (int q = 0; q < L::N2; ++q) g[(size_t)q * L::N1 * xs] = v[q];
    }
}

// Wave vector with 1 / k^2 and the Green factors of each half-spectrum point
// (zero at k = 0, so that mode is dropped).
__global__ void k_green_table(const float4* __restrict__ gridk, int Nx, int Ny, int Nz, int zp, float4* table) {
    const int z = blockIdx.x * blockDim.x + threadIdx.x;
    const int xy = blockIdx.y;
    if (z > Nz / 2) return;
    const float4 tk = gridk[(size_t)xy * Nz + z];
    float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), gf = kv;
    if (xy != 0 || z != 0) {
        const GreenFactors g = green_factors(tk);
        kv = make_float4(tk.x, tk.y, tk.z, g.ik2);
        gf = make_float4(g.uf, g.df, g.dc, 0.f);
    }
    const size_t pt = (size_t)xy * zp + z;
    table[2 * pt] = kv;
    table[2 * pt + 1] = gf;
}

// Calls f(Line<N1, N2>{}) for a supported line length; false otherwise.
template <class F>
bool with_line(int n, F&& f) {
    switch (n) {
        case 12: f(Line<3, 4>{}); return true;
        case 15: f(Line<3, 5>{}); return true;
        case 16: f(Line<4, 4>{}); return true;
        case 18: f(Line<3, 6>{}); return true;
        case 20: f(Line<5, 4>{}); return true;
        case 24: f(Line<4, 6>{}); return true;
        case 25: f(Line<5, 5>{}); return true;
        case 27: f(Line<3, 9>{}); return true;
        case 30: f(Line<5, 6>{}); return true;
        case 32: f(Line<4, 8>{}); return true;
        case 36: f(Line<6, 6>{}); return true;
        case 40: f(Line<5, 8>{}); return true;
        case 45: f(Line<5, 9>{}); return true;
        case 48: f(Line<6, 8>{}); return true;
        case 50: f(Line<5, 10>{}); return true;
        case 54: f(Line<9, 6>{}); return true;
        case 60: f(Line<6, 10>{}); return true;
        case 64: f(Line<8, 8>{}); return true;
        case 72: f(Line<9, 8>{}); return true;
        case 75: f(Line<5, 15>{}); return true;
        case 80: f(Line<8, 10>{}); return true;
        case 81: f(Line<9, 9>{}); return true;
        case 90: f(Line<9, 10>{}); return true;
        case 96: f(Line<8, 12>{}); return true;
        case 100: f(Line<10, 10>{}); return true;
        case 108: f(Line<9, 12>{}); return true;
        case 120: f(Line<15, 8>{}); return true;
        case 128: f(Line<8, 16>{}); return true;
        case 135: f(Line<9, 15>{}); return true;
        case 144: f(Line<12, 12>{}); return true;
        case 150: f(Line<15, 10>{}); return true;
        default: return false;
    }
}

}  // namespace

bool wave_fft_ok(const GridParams& g) {
    return g.Ny == g.Nz && with_line(g.Nx, [](auto) {}) && with_line(g.Ny, [](auto) {});
}

size_t wave_spec_elems(const GridParams& g) { return 11 * (size_t)g.Nx * g.Ny * wave_zp(g.Nz); }
size_t wave_table_elems(const GridParams& g) { return 2 * (size_t)g.Nx * g.Ny * wave_zp(g.Nz); }

void wave_set_table(fsd_handle* h) {
    const GridParams& g = h->g;
    count_launch();
    k_green_table<<<dim3((g.Nz / 2 + 32) / 32, g.Nx * g.Ny), 32, 0, h->stream>>>(h->w.gridk, g.Nx, g.Ny, g.Nz,
                                                                                wave_zp(g.Nz), h->w.green_table);
}

static void yz(fsd_handle* h, bool inv) {
    const GridParams& g = h->g;
    const float2* tw = h->w.twiddle + g.Nx;
    with_line(g.Ny, [&](auto line) {
        using L = decltype(line);
        const void* fn = inv ? (const void*)k_yz_inv<L> : (const void*)k_yz_fwd<L>;
        if (!smem_limit_ok(fn, Plane<L>::smem, "plane transform shared memory")) return;
        count_launch();
        if (inv)
            launch_pdl(k_yz_inv<L>, 6 * g.Nx, Plane<L>::threads, Plane<L>::smem, h->stream, h->w.spec, h->w.grid, g.Nx,
                                                                                   wave_zp(g.Nz), tw);
        else
            launch_pdl(k_yz_fwd<L>, 6 * g.Nx, Plane<L>::threads, Plane<L>::smem, h->stream, h->w.grid, h->w.spec, g.Nx,
                                                                                   wave_zp(g.Nz), tw);
    });
}

static void x_pass(fsd_handle* h, bool green) {
    const GridParams& g = h->g;
    const int zp = wave_zp(g.Nz);
    with_line(g.Nx, [&](auto line) {
        using L = decltype(line);
        const void* fn = green ? (const void*)k_x_pass<L, true> : (const void*)k_x_pass<L, false>;
        if (!smem_limit_ok(fn, XPass<L>::smem, "x pass shared memory")) return;
        count_launch();
        const int nb = g.Ny * (zp / kXz);
        if (green)
            launch_pdl(k_x_pass<L, true>, nb, XPass<L>::threads, XPass<L>::smem, h->stream, 
                h->w.spec, h->w.green_table, h->w.gridk, g.Ny, g.Nz, zp, h->w.twiddle);
        else
            launch_pdl(k_x_pass<L, false>, nb, XPass<L>::threads, XPass<L>::smem, h->stream, 
                h->w.spec, h->w.green_table, h->w.gridk, g.Ny, g.Nz, zp, h->w.twiddle);
    });
}

void wave_forward_yz(fsd_handle* h) { yz(h, false); }
void wave_inverse_yz(fsd_handle* h) { yz(h, true); }
void wave_x_green(fsd_handle* h) { x_pass(h, true); }
void wave_inverse_x(fsd_handle* h) { x_pass(h, false); }

}  // namespace fsd
