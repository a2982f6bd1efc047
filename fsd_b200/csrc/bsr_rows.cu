// Products of the learned preconditioner's inner polynomial (and of the
// approximate inverse applied once), each fused with the step around it, and
// the by-component layout of blocks that all row products read (fsd_bsr.cuh).
#include "fsd_bsr.cuh"
#include "fsd_device.cuh"
#include "fsd_kernels.cuh"
#include "fsd_learned.h"
#include "fsd_solver.h"

namespace fsd {

// Rows of blocks (block CSR, or padded rows of kPrunedCap blocks) by components
// at dst + 36 rowptr[i].
__global__ void __launch_bounds__(256) k_bsr_layout(const int* __restrict__ rowptr, bool padded, int N,
                                                    const float* __restrict__ src, float* __restrict__ dst) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= N) return;
    const int n = rowptr[i + 1] - rowptr[i];
    src += 36 * (padded ? (size_t)i * kPrunedCap : (size_t)rowptr[i]);
    dst += 36 * (size_t)rowptr[i];
    for (int t = threadIdx.x & 31; t < 36 * n; t += 32) {
        const int r = t / (6 * n), k = t - r * 6 * n, e = k / 6, c = k - 6 * e;
        dst[t] = src[36 * e + 6 * r + c];
    }
}

// Blocks in block CSR (rowptr in place) into G.
int bsr_import(fsd_handle* h, const float* blocks) {
    LearnedState* s = learned(h);
    count_launch();
    k_bsr_layout<<<(h->p.N + 7) / 8, 256, 0, h->stream>>>(s->g_rowptr, false, h->p.N, blocks, s->g_val);
    FSD_CHECK_CUDA(cudaGetLastError());
    return FSD_OK;
}

// Brings the polynomial's copy of A up to date: only the blocks that the
// pruned list holds (25 MB of its 151 MB of padded rows at N = 32768, phi = 0.4).
int bsr_sync_a(fsd_handle* h) {
    LearnedState* s = learned(h);
    const int N = h->p.N;
    cudaStream_t st = h->stream;
    if (!s->a_dirty || !s->a_blocks) return FSD_OK;
    if (!s->a_rowptr) {
        FSD_CHECK_CUDA(cudaMalloc(&s->a_rowptr, sizeof(int) * (N + 1)));
        FSD_CHECK_CUDA(cudaMalloc(&s->a_scan, sizeof(unsigned) * scan_scratch_elems(N)));
    }
    exclusive_scan(s->a_pn, (unsigned*)s->a_rowptr, N, s->a_scan, st);
    int nnzb = 0;
    FSD_CHECK_CUDA(cudaMemcpyAsync(&nnzb, s->a_rowptr + N, sizeof(int), cudaMemcpyDeviceToHost, st));
    FSD_CHECK_CUDA(cudaStreamSynchronize(st));
    if (nnzb > s->a_cap) {
        if (s->a_comp) cudaFree(s->a_comp);
        s->a_comp = nullptr;
        s->a_cap = 0;
        const int cap = nnzb + nnzb / 8 + 1024;
        FSD_CHECK_CUDA(cudaMalloc(&s->a_comp, sizeof(float) * 36 * (size_t)cap));
        s->a_cap = cap;
    }
    count_launch();
    k_bsr_layout<<<(N + 7) / 8, 256, 0, st>>>(s->a_rowptr, true, N, s->a_blocks, s->a_comp);
    FSD_CHECK_CUDA(cudaGetLastError());
    s->a_dirty = false;
    return FSD_OK;
}

// Modes: kBsrFirst = first product of the Clenshaw recurrence (operand
// t = b[0:6N] - b[11N:17N], writes T = t, B = c_{k-1} t, out = c_{k-1} G t);
// kBsrPlain = plain product out = M x; kBsrLast = last product y = G v with
// the saddle post step into xs; kBsrStep = Clenshaw step
// out = c_m T + f ((2/lambda) A u - B1) - B2; kBsrOnce = y = G t with the
// saddle pre and post steps (xs must not overlap b).
template <int MODE>
__global__ void __launch_bounds__(256) k_bsr_rows(BsrArgs a) {
    pdl_wait();
    const int N = a.N;
    const int q = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kBsrRows + bsr_sub();
    const bool have = q < N;
    const int i = have ? q : 0;
    const size_t offU = 11 * (size_t)N;
    const int r = have ? bsr_component() : -1;
    const size_t i6 = 6 * (size_t)i + (r < 0 ? 0 : r);
    // the row's epilogue operands, loaded before the product
    float e_a = 0.f, e_b = 0.f, e_c = 0.f;
    if (r >= 0) {
        if (MODE == kBsrFirst) {
            e_a = a.x[i6];
            e_b = a.x[offU + i6];
        } else if (MODE == kBsrLast || MODE == kBsrOnce) {
            e_a = a.b[i6];
        } else if (MODE == kBsrStep) {
            e_a = a.T[i6];
            e_b = a.B1[i6];
            e_c = a.B2 ? a.B2[i6] : 0.f;
        }
    }
    const int q0 = a.rowptr[i], n = have ? a.rowptr[i + 1] - q0 : 0;
    const float* row = a.val + 36 * (size_t)q0;
    const int* cols = a.col + (MODE == kBsrStep ? (size_t)i * kPrunedCap : (size_t)q0);  // A: the padded pruned list
    float acc;
    if constexpr (MODE == kBsrFirst || MODE == kBsrOnce)
        acc = bsr_row(row, cols, n, BsrSaddle{MODE == kBsrFirst ? a.x : a.b, offU});
    else
        acc = bsr_row(row, cols, n, BsrPlain{a.x});
    if (MODE == kBsrLast || MODE == kBsrOnce) {
        if (r >= 0 && r < 5) {
            const size_t q5 = 6 * (size_t)N + 5 * (size_t)i + r;
            a.xs[q5] = a.b[q5];
        }
    }
    if (r < 0) return;
    if (MODE == kBsrFirst) {
        const float c = a.pc[a.k - 1];
        const float tv = e_a - e_b;
        a.T[i6] = tv;
        a.B[i6] = c * tv;
        a.out[i6] = c * acc;
    } else if (MODE == kBsrPlain) {
        a.out[i6] = acc;
    } else if (MODE == kBsrLast || MODE == kBsrOnce) {
        a.xs[i6] = e_a - acc;
        a.xs[offU + i6] = acc;
    } else {
        const float s2 = 2.0f / a.pc[kMaxPoly];
        const float f = a.m >= 1 ? 2.0f : 1.0f;
        float v = fmaf(a.pc[a.m], e_a, f * fmaf(s2, acc, -e_b));
        if (a.B2) v -= e_c;
        a.out[i6] = v;
    }
}

// Kernel entry of a mode (for launches and graph-node updates).
const void* bsr_kernel(int mode) {
    switch (mode) {
        case kBsrFirst: return (const void*)k_bsr_rows<kBsrFirst>;
        case kBsrPlain: return (const void*)k_bsr_rows<kBsrPlain>;
        case kBsrLast: return (const void*)k_bsr_rows<kBsrLast>;
        case kBsrStep: return (const void*)k_bsr_rows<kBsrStep>;
        default: return (const void*)k_bsr_rows<kBsrOnce>;
    }
}

int bsr_blocks(int N) { return (N + 8 * kBsrRows - 1) / (8 * kBsrRows); }

void bsr_launch(int mode, const BsrArgs& a, cudaStream_t st) {
    const int grid = bsr_blocks(a.N);
    switch (mode) {
        case kBsrFirst: launch_pdl(k_bsr_rows<kBsrFirst>, grid, 256, 0, st, a); break;
        case kBsrPlain: launch_pdl(k_bsr_rows<kBsrPlain>, grid, 256, 0, st, a); break;
        case kBsrLast: launch_pdl(k_bsr_rows<kBsrLast>, grid, 256, 0, st, a); break;
        case kBsrStep: launch_pdl(k_bsr_rows<kBsrStep>, grid, 256, 0, st, a); break;
        default: launch_pdl(k_bsr_rows<kBsrOnce>, grid, 256, 0, st, a); break;
    }
}

}  // namespace fsd
