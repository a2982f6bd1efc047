// Learned Chebyshev polynomial inner solve of FSD_PRECOND_LEARNED.
//
// The saddle preconditioner (Saddle.cu:171-264) needs y ~ A^-1 t for the
// lubrication block A = R_FU^pruned + D.  Here
//   y = G q(AG) t,   q(x) = sum_{m<k} c_m T_m(2x/lambda - 1),
// with G the two-hop sparse approximate inverse of A (spai.cu), T_m the
// Chebyshev polynomials, lambda an upper bound of the spectrum of AG (power
// iteration when the preconditioner is built, times 1.1), and coefficients c
// that the message-passing network predicts for each configuration (mpnn.cu,
// the mean over particles of its node head) or that the caller sets.
// q(AG) t is evaluated by Clenshaw's recurrence with S = (2/lambda) AG - I:
//   b_{k-1} = c_{k-1} t,
//   b_m = c_m t + 2 S b_{m+1} - b_{m+2}        m = k-2 .. 1,
//   v = c_0 t + S b_1 - b_2,
// so one application costs k products with G, k-1 with A and no reductions.
// The map t -> y is linear and fixed within a solve, so the outer GMRES keeps
// no flexible basis.  The 2k-1 kernels are replayed from a CUDA graph whose
// first and last nodes (the only ones that touch b and x) are re-pointed at
// each application's vectors.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "fsd_brownian.h"
#include "fsd_bsr.cuh"
#include "fsd_device.cuh"
#include "fsd_kernels.cuh"
#include "fsd_learned.h"
#include "fsd_profile.h"
#include "fsd_solver.h"

namespace fsd {

namespace {

constexpr int kPowerIters = 12;      // power iterations for the spectral bound
constexpr float kLambdaMargin = 1.1f;
constexpr int kPowerBlocks = 6 * 148;

// ---------------------------------------------------------- spectral bound
__global__ void k_set_double(double* p, double v) { *p = v; }

// W = A U, |W| into nrm[0] and kLambdaMargin |W| into pc[kMaxPoly] by the last block.
__global__ void __launch_bounds__(256) k_power_a(const int* __restrict__ rowptr, const int* __restrict__ plist,
                                                 const float* __restrict__ A, const float* __restrict__ U, int N,
                                                 float* __restrict__ W, double* part, unsigned* ticket, double* nrm,
                                                 float* pc) {
    const int rc = bsr_component();
    double s = 0.0;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int t0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t0 * kBsrRows < N; t0 += nw) {
        const int q = t0 * kBsrRows + bsr_sub();
        const bool have = q < N;
        const int i = have ? q : 0;
        const int q0 = rowptr[i];
        const float acc = bsr_row(A + 36 * (size_t)q0, plist + (size_t)i * kPrunedCap, have ? rowptr[i + 1] - q0 : 0,
                                  BsrPlain{U});
        if (have && rc >= 0) {
            W[6 * (size_t)i + rc] = acc;
            s += (double)acc * acc;
        }
    }
    block_partial(s, part);
    if (!last_block(ticket)) return;
    if (threadIdx.x < 32) {
        const double t = sqrt(warp_sum_parts(part, gridDim.x));
        if (threadIdx.x == 0) {
            nrm[0] = t;
            pc[kMaxPoly] = (float)(kLambdaMargin * t);
            *ticket = 0;
        }
    }
}

// U = G (W / nrm[0]).
__global__ void __launch_bounds__(256) k_power_g(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                 const float* __restrict__ G, const float* __restrict__ W,
                                                 const double* __restrict__ nrm, int N, float* __restrict__ U) {
    const int q = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kBsrRows + bsr_sub();
    const bool have = q < N;
    const int i = have ? q : 0, r = have ? bsr_component() : -1;
    const int q0 = rowptr[i];
    const float acc = bsr_row(G + 36 * (size_t)q0, col + q0, have ? rowptr[i + 1] - q0 : 0, BsrPlain{W});
    const double nv = *nrm;
    const float f = nv > 0.0 ? (float)(1.0 / nv) : 0.f;
    if (r >= 0) U[6 * (size_t)i + r] = f * acc;
}

}  // namespace

int poly_alloc(fsd_handle* h) {
    LearnedState* s = learned(h);
    if (s->pc) return FSD_OK;
    const size_t n6 = 6 * (size_t)h->p.N;
    FSD_CHECK_CUDA(cudaMalloc(&s->pc, sizeof(float) * (kMaxPoly + 1)));
    FSD_CHECK_CUDA(cudaMemsetAsync(s->pc, 0, sizeof(float) * (kMaxPoly + 1), h->stream));
    FSD_CHECK_CUDA(cudaMalloc(&s->pbuf, sizeof(float) * n6 * 5));
    FSD_CHECK_CUDA(cudaMalloc(&s->ppart, sizeof(double) * kPowerBlocks));
    FSD_CHECK_CUDA(cudaMalloc(&s->pnrm, sizeof(double) * 2));
    FSD_CHECK_CUDA(cudaMalloc(&s->pticket, sizeof(unsigned)));
    FSD_CHECK_CUDA(cudaMemsetAsync(s->pticket, 0, sizeof(unsigned), h->stream));
    return FSD_OK;
}

bool poly_active(const fsd_handle* h) {
    return h->p.precond == FSD_PRECOND_LEARNED && h->p.learned_poly >= 2;
}

// Upper bound of the spectrum of AG into pc[kMaxPoly]: kPowerIters power
// iterations from a fixed counter-based start vector, times 1.1.
int poly_lambda(fsd_handle* h) {
    LearnedState* s = learned(h);
    const int N = h->p.N;
    const size_t n6 = 6 * (size_t)N;
    cudaStream_t st = h->stream;
    float* W = s->pbuf;
    float* U = s->pbuf + n6;
    const int e = bsr_sync_a(h);
    if (e != FSD_OK) return e;
    const int rows = bsr_blocks(N), arows = std::min(rows, kPowerBlocks);
    gaussian(h, W, n6, 1, kStreamGain, 1.0f);
    count_launch();
    k_set_double<<<1, 1, 0, st>>>(s->pnrm, std::sqrt((double)n6));
    for (int it = 0; it < kPowerIters; ++it) {
        count_launch();
        k_power_g<<<rows, 256, 0, st>>>(s->g_rowptr, s->g_col, s->g_val, W, s->pnrm, N, U);
        count_launch();
        k_power_a<<<arows, 256, 0, st>>>(s->a_rowptr, (const int*)s->a_plist, s->a_comp, U, N, W, s->ppart, s->pticket,
                                         s->pnrm, s->pc);
    }
    FSD_CHECK_CUDA(cudaGetLastError());
    return FSD_OK;
}

// Clenshaw slots: b_{k-1} in slot 0; each b_m goes to the slot that holds
// neither b_{m+1} nor b_{m+2}.
static int poly_next_slot(int cur, int prev) { return (cur + 1) % 3 == prev ? (cur + 2) % 3 : (cur + 1) % 3; }

// Slot that holds v = b_0 after the recurrence for k coefficients.
static int poly_v_slot(int k) {
    int cur = 0, prev = -1;
    for (int m = k - 2; m >= 0; --m) {
        const int nxt = poly_next_slot(cur, prev);
        prev = cur;
        cur = nxt;
    }
    return cur;
}

static BsrArgs g_args(const LearnedState* s, int N) {
    BsrArgs a{};
    a.rowptr = s->g_rowptr;
    a.col = s->g_col;
    a.val = s->g_val;
    a.N = N;
    a.pc = s->pc;
    return a;
}

static BsrArgs a_args(const LearnedState* s, int N) {
    BsrArgs a{};
    a.rowptr = s->a_rowptr;
    a.col = (const int*)s->a_plist;
    a.val = s->a_comp;
    a.N = N;
    a.pc = s->pc;
    return a;
}

// Arguments of the first (kBsrFirst) and last (kBsrLast) products for b and x.
static BsrArgs first_args(const LearnedState* s, int N, int k, const float* b) {
    const size_t n6 = 6 * (size_t)N;
    BsrArgs a = g_args(s, N);
    a.x = b;
    a.T = s->pbuf;
    a.out = s->pbuf + n6;
    a.B = s->pbuf + 2 * n6;
    a.k = k;
    return a;
}

static BsrArgs last_args(const LearnedState* s, int N, int k, const float* b, float* x) {
    const size_t n6 = 6 * (size_t)N;
    BsrArgs a = g_args(s, N);
    a.x = s->pbuf + (2 + poly_v_slot(k)) * n6;
    a.b = b;
    a.xs = x;
    return a;
}

// Kernels of one application on b into x, enqueued on st (for capture):
// k products with G and k - 1 with A.
static int poly_enqueue(fsd_handle* h, const float* b, float* x, cudaStream_t st) {
    LearnedState* s = learned(h);
    const int N = h->p.N;
    const int k = h->p.learned_poly;
    const size_t n6 = 6 * (size_t)N;
    float* T = s->pbuf;
    float* U = s->pbuf + n6;
    float* Bs[3] = {s->pbuf + 2 * n6, s->pbuf + 3 * n6, s->pbuf + 4 * n6};
    bsr_launch(kBsrFirst, first_args(s, N, k, b), st);  // U = c_{k-1} G t, b_{k-1} -> slot 0
    int cur = 0, prev = -1;
    for (int m = k - 2; m >= 0; --m) {
        if (m < k - 2) {
            BsrArgs ga = g_args(s, N);
            ga.x = Bs[cur];
            ga.out = U;
            bsr_launch(kBsrPlain, ga, st);
        }
        const int nxt = poly_next_slot(cur, prev);
        BsrArgs aa = a_args(s, N);
        aa.x = U;
        aa.T = T;
        aa.B1 = Bs[cur];
        aa.B2 = prev >= 0 ? Bs[prev] : nullptr;
        aa.m = m;
        aa.out = Bs[nxt];
        bsr_launch(kBsrStep, aa, st);
        prev = cur;
        cur = nxt;
    }
    bsr_launch(kBsrLast, last_args(s, N, k, b, x), st);
    FSD_CHECK_CUDA(cudaGetLastError());
    return FSD_OK;
}

static int poly_kernels(int k) { return 2 * k - 1; }

static int poly_graph(fsd_handle* h, const float* b, float* x) {
    LearnedState* s = learned(h);
    const void* key[10] = {s->g_rowptr, s->g_col, s->g_val, s->a_rowptr, s->a_plist,
                           s->a_comp,   s->pbuf,  s->pc,    nullptr,     nullptr};
    bool same = s->pexec && s->pkey_k == h->p.learned_poly;
    for (int i = 0; i < 10 && same; ++i) same = key[i] == s->pkey[i];
    if (same) return FSD_OK;
    if (s->pexec) cudaGraphExecDestroy(s->pexec);
    if (s->pgraph) cudaGraphDestroy(s->pgraph);
    s->pexec = nullptr;
    s->pgraph = nullptr;
    if (!s->cap_stream) FSD_CHECK_CUDA(cudaStreamCreateWithFlags(&s->cap_stream, cudaStreamNonBlocking));
    cudaGraph_t g = nullptr;
    FSD_CHECK_CUDA(cudaStreamBeginCapture(s->cap_stream, cudaStreamCaptureModeThreadLocal));
    const int e = poly_enqueue(h, b, x, s->cap_stream);
    const cudaError_t ce = cudaStreamEndCapture(s->cap_stream, &g);
    if (e != FSD_OK) {
        if (g) cudaGraphDestroy(g);
        return e;
    }
    FSD_CHECK_CUDA(ce);
    size_t nn = 0;
    FSD_CHECK_CUDA(cudaGraphGetNodes(g, nullptr, &nn));
    std::vector<cudaGraphNode_t> nodes(nn);
    FSD_CHECK_CUDA(cudaGraphGetNodes(g, nodes.data(), &nn));
    s->pnode_first = s->pnode_last = nullptr;
    for (cudaGraphNode_t nd : nodes) {
        cudaGraphNodeType t;
        FSD_CHECK_CUDA(cudaGraphNodeGetType(nd, &t));
        if (t != cudaGraphNodeTypeKernel) continue;
        cudaKernelNodeParams kp;
        FSD_CHECK_CUDA(cudaGraphKernelNodeGetParams(nd, &kp));
        if (kp.func == bsr_kernel(kBsrFirst)) s->pnode_first = nd;
        if (kp.func == bsr_kernel(kBsrLast)) s->pnode_last = nd;
    }
    if (!s->pnode_first || !s->pnode_last) {
        cudaGraphDestroy(g);
        return FSD_ERR_CUDA;
    }
    const cudaError_t ie = cudaGraphInstantiate(&s->pexec, g, 0);
    if (ie != cudaSuccess) {
        cudaGraphDestroy(g);
        FSD_CHECK_CUDA(ie);
    }
    s->pgraph = g;
    for (int i = 0; i < 10; ++i) s->pkey[i] = key[i];
    s->pkey_k = h->p.learned_poly;
    return FSD_OK;
}

// Point the first node at b and the last at (b, x).
static int poly_bind(fsd_handle* h, const float* b, float* x) {
    LearnedState* s = learned(h);
    const int N = h->p.N, k = h->p.learned_poly;
    BsrArgs fa = first_args(s, N, k, b), la = last_args(s, N, k, b, x);
    void* fargs[] = {&fa};
    void* largs[] = {&la};
    cudaKernelNodeParams kp = {};
    kp.gridDim = dim3(bsr_blocks(N));
    kp.blockDim = dim3(256);
    kp.func = (void*)bsr_kernel(kBsrFirst);
    kp.kernelParams = fargs;
    FSD_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(s->pexec, s->pnode_first, &kp));
    kp.func = (void*)bsr_kernel(kBsrLast);
    kp.kernelParams = largs;
    FSD_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(s->pexec, s->pnode_last, &kp));
    return FSD_OK;
}

int poly_apply(fsd_handle* h, const float* b, float* x) {
    LearnedState* s = learned(h);
    int e = bsr_sync_a(h);
    if (e != FSD_OK) return e;
    e = poly_graph(h, b, x);
    if (e != FSD_OK) return e;
    e = poly_bind(h, b, x);
    if (e != FSD_OK) return e;
    FSD_CHECK_CUDA(cudaGraphLaunch(s->pexec, h->stream));
    for (int i = 0; i < poly_kernels(h->p.learned_poly); ++i) count_launch();
    return FSD_OK;
}

// Coefficients of q for the Chebyshev interval [rho lambda, lambda]: the
// residual polynomial 1 - x q(x) = T_k((1 + rho - 2u)/(1 - rho)) /
// T_k((1 + rho)/(1 - rho)), u = x / lambda, is the classical Chebyshev
// acceleration on that interval (bounded by one on all of [0, lambda], so no
// eigenvalue of AG is amplified, and smallest on [rho lambda, lambda]).  q has
// degree k - 1 and is expanded exactly in T_m(2u - 1), m < k, by Chebyshev
// interpolation at k nodes (FP64).
static double cheb_T(int n, double z) {
    if (std::fabs(z) <= 1.0) return std::cos(n * std::acos(z));
    const double v = std::cosh(n * std::acosh(std::fabs(z)));
    return (z < 0 && (n & 1)) ? -v : v;
}

void poly_interval_coefficients(double rho, double lambda, int k, float* c) {
    const double zs = (1.0 + rho) / (1.0 - rho);
    const double Tz = cheb_T(k, zs);
    std::vector<double> gu(k), uu(k);
    for (int j = 0; j < k; ++j) {
        const double th = M_PI * (j + 0.5) / k;
        const double u = 0.5 * (std::cos(th) + 1.0);
        const double r = cheb_T(k, (1.0 + rho - 2.0 * u) / (1.0 - rho)) / Tz;
        uu[j] = u;
        gu[j] = (1.0 - r) / (lambda * u);
    }
    for (int m = 0; m < k; ++m) {
        double acc = 0.0;
        for (int j = 0; j < k; ++j) acc += gu[j] * std::cos(m * M_PI * (j + 0.5) / k);
        c[m] = (float)((m == 0 ? 1.0 : 2.0) * acc / k);
    }
}

// Coefficients for the interval ratio rho (in (0, 1)) with the spectral
// bound of the last power iteration; caller's stream, synchronised.
int poly_set_interval(fsd_handle* h, double rho) {
    LearnedState* s = learned(h);
    const int k = h->p.learned_poly;
    float pc[kMaxPoly + 1];
    FSD_CHECK_CUDA(cudaMemcpyAsync(pc, s->pc, sizeof(float) * (kMaxPoly + 1), cudaMemcpyDeviceToHost, h->stream));
    FSD_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    const double lambda = pc[kMaxPoly];
    if (!(lambda > 0.0) || !(rho > 0.0 && rho < 1.0)) return FSD_ERR_BREAKDOWN;
    float c[kMaxPoly] = {};
    poly_interval_coefficients(rho, lambda, k, c);
    FSD_CHECK_CUDA(cudaMemcpyAsync(s->pc, c, sizeof(float) * kMaxPoly, cudaMemcpyHostToDevice, h->stream));
    FSD_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    s->poly_ratio = (float)rho;
    return FSD_OK;
}

int poly_set_coefficients(fsd_handle* h, const float* host_c, int k) {
    if (k < 2 || k > kMaxPoly || !host_c) return FSD_ERR_BAD_PARAMS;
    const int e = poly_alloc(h);
    if (e != FSD_OK) return e;
    LearnedState* s = learned(h);
    float c[kMaxPoly] = {};
    for (int m = 0; m < k; ++m) c[m] = host_c[m];
    FSD_CHECK_CUDA(cudaMemcpyAsync(s->pc, c, sizeof(float) * kMaxPoly, cudaMemcpyHostToDevice, h->stream));
    FSD_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    s->poly_user = true;
    s->user_ratio = -1.f;
    return FSD_OK;
}

int poly_get_coefficients(fsd_handle* h, float* host_c, int n) {
    LearnedState* s = learned(h);
    if (!host_c || n < kMaxPoly + 1 || !s->pc) return FSD_ERR_BAD_PARAMS;
    FSD_CHECK_CUDA(cudaMemcpyAsync(host_c, s->pc, sizeof(float) * (kMaxPoly + 1), cudaMemcpyDeviceToHost, h->stream));
    FSD_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    return FSD_OK;
}

void poly_free(LearnedState* s) {
    void* ptrs[] = {s->pc, s->pbuf, s->ppart, s->pnrm, s->pticket};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (s->pexec) cudaGraphExecDestroy(s->pexec);
    if (s->pgraph) cudaGraphDestroy(s->pgraph);
}

}  // namespace fsd
