// Block-sparse preconditioner slot G for FSD_PRECOND_LEARNED.
//
// G ~ (R_FU^pruned + relaxer D)^-1 is an explicit block-sparse matrix (6x6
// fp32 blocks in block-CSR over particles, original particle order): the
// two-hop sparse approximate inverse of the pruned matrix (spai.cu), plus the
// loaded network's correction (mpnn.cu), or blocks set directly through
// fsd_precond_set_blocks.  Applied once (learned_inner = 0, fused with the
// saddle pre/post steps of Saddle.cu:171-264) or as the right preconditioner
// of a few inner GMRES steps on the pruned matrix itself, replayed from a
// CUDA graph.
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fsd_bsr.cuh"
#include "fsd_device.cuh"
#include "fsd_kernels.cuh"
#include "fsd_learned.h"
#include "fsd_profile.h"
#include "fsd_solver.h"

namespace fsd {

LearnedState* learned(fsd_handle* h) {
    if (!h->learned) h->learned = new LearnedState();
    return (LearnedState*)h->learned;
}

void learned_free(fsd_handle* h) {
    LearnedState* s = (LearnedState*)h->learned;
    if (!s) return;
    mpnn_free(h);
    void* ptrs[] = {s->a_rowptr, s->a_scan, s->a_comp, s->g_rowptr, s->g_col,   s->g_val,     s->Vi,        s->Zi,        s->part,   s->H,
                    s->nrm,      s->ticket,  s->sp_sets,   s->sp_size,   s->sp_rowptr, s->sp_scan, s->sp_bucket,
                    s->sp_cnt};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (s->sp_host) cudaFreeHost(s->sp_host);
    poly_free(s);
    if (s->gexec) cudaGraphExecDestroy(s->gexec);
    if (s->graph) cudaGraphDestroy(s->graph);
    if (s->cap_stream) cudaStreamDestroy(s->cap_stream);
    delete s;
    h->learned = nullptr;
}

// Grow the block-CSR storage of G to hold nnzb blocks.
int learned_reserve(fsd_handle* h, int nnzb) {
    LearnedState* s = learned(h);
    const int N = h->p.N;
    if (!s->g_rowptr) FSD_CHECK_CUDA(cudaMalloc(&s->g_rowptr, sizeof(int) * (N + 1)));
    if (nnzb + 8 > s->g_cap) {
        if (s->g_col) cudaFree(s->g_col);
        if (s->g_val) cudaFree(s->g_val);
        s->g_col = nullptr;
        s->g_val = nullptr;
        s->g_cap = 0;
        // headroom, so that pattern growth from step to step rarely reallocates
        const int cap = nnzb + nnzb / 8 + 1024;
        FSD_CHECK_CUDA(cudaMalloc(&s->g_col, sizeof(int) * (size_t)cap));
        FSD_CHECK_CUDA(cudaMalloc(&s->g_val, sizeof(float) * 36 * (size_t)cap));
        s->g_cap = cap;
    }
    return FSD_OK;
}

// A checked block-CSR G from the caller's arrays, which may lie on another
// device; `staged` receives its blocks as they came.
static int learned_take_blocks(fsd_handle* h, int nnzb, const int* d_rowptr, const int* d_col, const float* d_val,
                               float* staged) {
    const int N = h->p.N;
    const size_t nb = (size_t)nnzb;
    const int e = learned_reserve(h, nnzb);
    if (e != FSD_OK) return e;
    LearnedState* s = learned(h);
    FSD_CHECK_CUDA(cudaMemcpyAsync(s->g_rowptr, d_rowptr, sizeof(int) * (N + 1), cudaMemcpyDeviceToDevice, h->stream));
    if (nnzb) {
        FSD_CHECK_CUDA(cudaMemcpyAsync(s->g_col, d_col, sizeof(int) * nb, cudaMemcpyDeviceToDevice, h->stream));
        FSD_CHECK_CUDA(cudaMemcpyAsync(staged, d_val, sizeof(float) * 36 * nb, cudaMemcpyDeviceToDevice, h->stream));
    }
    s->g_nnzb = nnzb;
    s->g_user = true;
    return nnzb ? bsr_import(h, staged) : FSD_OK;
}

// Copy a caller's block-CSR G after checking its structure on the host, so
// that no kernel ever indexes outside the vectors it reads.
int learned_set_blocks(fsd_handle* h, int nnzb, const int* d_rowptr, const int* d_col, const float* d_val) {
    const int N = h->p.N;
    if (nnzb < 0) return FSD_ERR_BAD_PARAMS;
    std::vector<int> rp(N + 1), cl((size_t)nnzb);
    FSD_CHECK_CUDA(cudaMemcpyAsync(rp.data(), d_rowptr, sizeof(int) * (N + 1), cudaMemcpyDeviceToHost, h->stream));
    if (nnzb)
        FSD_CHECK_CUDA(
            cudaMemcpyAsync(cl.data(), d_col, sizeof(int) * (size_t)nnzb, cudaMemcpyDeviceToHost, h->stream));
    FSD_CHECK_CUDA(cudaStreamSynchronize(h->stream));
    if (rp[0] != 0 || rp[N] != nnzb) return FSD_ERR_BAD_PARAMS;
    for (int i = 0; i < N; ++i)
        if (rp[i + 1] < rp[i]) return FSD_ERR_BAD_PARAMS;
    for (int c : cl)
        if (c < 0 || c >= N) return FSD_ERR_BAD_PARAMS;
    // the blocks as they came, until they are laid out by components; taken
    // before anything of the present G changes
    float* staged = nullptr;
    if (nnzb) FSD_CHECK_CUDA(cudaMalloc(&staged, sizeof(float) * 36 * (size_t)nnzb));
    const int e = learned_take_blocks(h, nnzb, d_rowptr, d_col, d_val, staged);
    if (staged) cudaFree(staged);  // waits for the layout
    return e;
}

// ----------------------------------------------------------- inner solve
// The blocks stay fp32: the lubrication blocks are ill-conditioned (gaps down
// to 1e-3), and fp16 copies, even scaled per block, raised the outer
// iteration counts by a quarter.

// k steps of GMRES on A, right-preconditioned by G.  The basis U_j is kept
// unnormalised with |U_j| in nrm[j], and Z_j = G U_j:
//   k_inner_g (step j): Z_j, and |U_j| by the last block; the first step forms
//       U_0 from the right-hand side in its gathers;
//   k_inner_a: w = A Z_j / |U_j| and its dots with U_0..U_j;
//   k_inner_orth: U_{j+1} = w less its parts along U_0..U_j, or at the last
//   step k_inner_last: only the norm of that, and the least-squares solution.
// Launch- and latency-bound below some thousand particles; G and A (78 MB
// between them) do not both stay in L2 at N = 32768.  Taking the norm beside
// the product instead of at the end of the orthogonalisation leaves that a map
// without a reduction, 7.0 -> 2.9 us at N = 32768, and the first right-hand
// side needs no kernel.  Eight lanes per row suit the plain rows of A (15.9 us;
// 18.3 with a warp per row by components).
//
// Slower or less accurate: the orthogonalisation inside the product (by
// linearity, Z_j = G w - sum c_q Z_q; the application's error against 64 bits
// grew by a quarter); every second product over the rows in descending order,
// so as to meet what L2 still holds (25 -> 38 us).

// Row r of a 6x6 fp32 block times x, summed over a group of eight lanes
// (lane c < 6 holds x_c in xj).
__device__ __forceinline__ float block_row(const float* blk, int rr, float xj, unsigned gmask) {
    const float2* g = reinterpret_cast<const float2*>(blk + rr * 6);
    const float2 g01 = g[0], g23 = g[1], g45 = g[2];
    float sum = g01.x * __shfl_sync(gmask, xj, 0, 8);
    sum = fmaf(g01.y, __shfl_sync(gmask, xj, 1, 8), sum);
    sum = fmaf(g23.x, __shfl_sync(gmask, xj, 2, 8), sum);
    sum = fmaf(g23.y, __shfl_sync(gmask, xj, 3, 8), sum);
    sum = fmaf(g45.x, __shfl_sync(gmask, xj, 4, 8), sum);
    sum = fmaf(g45.y, __shfl_sync(gmask, xj, 5, 8), sum);
    return sum;
}

constexpr int kInnerBlocks = 296;
constexpr int kInnerRowBlocks = 4 * 148;  // at most: every block resident, its rows strided over the warps
constexpr int kInnerThreads = 256;
constexpr int kBetaSlot = (kMaxInner + 1) * kMaxInner;  // in H: beta, then the k coefficients

// Z_j = G U_j, a warp per row on G by components, and |U_j|; FIRST:
// U_0 = b[0:6N] - b[11N:17N], taken from b in the gathers too.
template <bool FIRST>
__global__ void __launch_bounds__(kInnerThreads, 4) k_inner_g(const int* rowptr, const int* col,
                                                              const float* G, const float* b,
                                                              float* U, float* __restrict__ z, int N, double* beta,
                                                              double* nrm, double* part, unsigned* ticket) {
    pdl_wait();
    const int r = bsr_component<32>();
    const size_t offU = 11 * (size_t)N;
    double s = 0.0;
    for (int i = (blockIdx.x * kInnerThreads + threadIdx.x) >> 5; i < N; i += (gridDim.x * kInnerThreads) >> 5) {
        const int q0 = rowptr[i], n = rowptr[i + 1] - q0;
        const size_t i6 = 6 * (size_t)i + (r < 0 ? 0 : r);
        float u = 0.f, acc;
        if (r >= 0) u = FIRST ? b[i6] - b[offU + i6] : U[i6];
        if constexpr (FIRST)
            acc = bsr_row<32>(G + 36 * (size_t)q0, col + q0, n, BsrSaddle{b, offU});
        else
            acc = bsr_row<32>(G + 36 * (size_t)q0, col + q0, n, BsrPlain{U});
        if (r >= 0) {
            if (FIRST) U[i6] = u;
            z[i6] = acc;
            s += (double)u * u;
        }
    }
    block_partial(s, part);
    if (!last_block(ticket)) return;
    if (threadIdx.x < 32) {
        const double t = sqrt(warp_sum_parts(part, gridDim.x));
        if (threadIdx.x == 0) {
            *nrm = t;
            *beta = t;  // H's beta slot, or the subdiagonal of the previous column
            *ticket = 0;
        }
    }
}

// w = A z / |U_j| over the pruned list (self included), written to the basis
// slot U_nv, fused with the dots H[j][q] = (U_q . w) / |U_q| for q < nv = j + 1.
__global__ void __launch_bounds__(256) k_inner_a(const unsigned* __restrict__ pn, const unsigned* __restrict__ plist,
                                                 const float* __restrict__ A, const float* z, float* U, size_t ld, int nv,
                                                 const double* nrm, double* part, unsigned* ticket, double* H, int j,
                                                 int N) {
    pdl_wait();
    __shared__ double sh[kMaxInner + 1][8];
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = gid >> 3;  // rows in storage order: the kernel streams A
    const bool row_ok = i < N;
    const int r = threadIdx.x & 7;
    const bool act = row_ok && r < 6;
    float acc = 0.f;
    if (row_ok) {  // whole groups of eight; every thread reaches the reductions below
        const unsigned gmask = 0xffu << (threadIdx.x & 24);
        const int rr = r < 6 ? r : 0;
        const unsigned n = pn[i];
        const size_t e0 = (size_t)i * kPrunedCap;
        unsigned q = 0;
        for (; q + 3 < n; q += 4) {  // four blocks in flight per lane
            const unsigned j0 = plist[e0 + q], j1 = plist[e0 + q + 1], j2 = plist[e0 + q + 2], j3 = plist[e0 + q + 3];
            const float x0 = (r < 6) ? z[6 * j0 + r] : 0.f, x1 = (r < 6) ? z[6 * j1 + r] : 0.f;
            const float x2 = (r < 6) ? z[6 * j2 + r] : 0.f, x3 = (r < 6) ? z[6 * j3 + r] : 0.f;
            const float* Ae = A + (e0 + q) * 36;
            acc += block_row(Ae, rr, x0, gmask);
            acc += block_row(Ae + 36, rr, x1, gmask);
            acc += block_row(Ae + 72, rr, x2, gmask);
            acc += block_row(Ae + 108, rr, x3, gmask);
        }
        for (; q < n; ++q) {
            const size_t e = e0 + q;
            const unsigned jj = plist[e];
            const float xj = (r < 6) ? z[6 * jj + r] : 0.f;
            acc += block_row(A + e * 36, rr, xj, gmask);
        }
        const double nj = nrm[j];
        acc *= nj > 0.0 ? (float)(1.0 / nj) : 0.f;
        if (act) U[(size_t)nv * ld + 6 * i + r] = acc;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int q = 0; q < nv; ++q) {
        double d = act ? (double)U[(size_t)q * ld + 6 * i + r] * (double)acc : 0.0;
        d = group_sum_d<32>(d);
        if (lane == 0) sh[q][wid] = d;
    }
    __syncthreads();
    if (threadIdx.x < nv) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += sh[threadIdx.x][w];
        part[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = v;
        __threadfence();
    }
    if (!last_block(ticket)) return;
    for (int q = wid; q < nv; q += blockDim.x >> 5) {
        const double t = warp_sum_parts(part + (size_t)q * gridDim.x, gridDim.x);
        if (lane == 0) H[(size_t)j * (kMaxInner + 1) + q] = nrm[q] > 0.0 ? t / nrm[q] : 0.0;
    }
    if (threadIdx.x == 0) *ticket = 0;
}

// The factors of U_q in w's orthogonalisation against nv vectors.
__device__ __forceinline__ void inner_factors(float* cs, const double* hj, const double* nrm, int nv) {
    if ((int)threadIdx.x < nv)
        cs[threadIdx.x] = nrm[threadIdx.x] > 0.0 ? (float)(hj[threadIdx.x] / nrm[threadIdx.x]) : 0.f;
    __syncthreads();
}
__device__ __forceinline__ float2 inner_pair(const float* U, size_t ld, int nv, const float* cs, size_t k) {
    float2 u = *reinterpret_cast<const float2*>(U + nv * ld + k);
#pragma unroll 6
    for (int q = 0; q < nv; ++q) {
        const float2 v = *reinterpret_cast<const float2*>(U + q * ld + k);
        u.x = fmaf(-cs[q], v.x, u.x);
        u.y = fmaf(-cs[q], v.y, u.y);
    }
    return u;
}

// U_nv -= sum_{q<nv} (H[j][q] / |U_q|) U_q, by pairs (ld = 6N is even).
__global__ void __launch_bounds__(kInnerThreads) k_inner_orth(float* U, size_t ld, int nv, const double* hj,
                                                              const double* nrm) {
    pdl_wait();
    __shared__ float cs[kMaxInner];
    inner_factors(cs, hj, nrm, nv);
    const size_t k = 2 * (blockIdx.x * (size_t)kInnerThreads + threadIdx.x);
    if (k < ld) *reinterpret_cast<float2*>(U + nv * ld + k) = inner_pair(U, ld, nv, cs, k);
}

// Least squares min || beta e1 - H y || by Givens rotations in FP64, one warp:
// lane q holds column q, every lane the rotated right-hand side.  Columns after
// a breakdown (zero subdiagonal or zero pivot) are dropped.  The coefficients of
// Z_q = G U_q, y_q / |U_q|, are written after H's beta slot.  (One thread on
// arrays in local memory took 10 us.)
template <int K>
__device__ __forceinline__ void inner_lsq(double* H, const double* nrm) {
    const int lane = threadIdx.x & 31;
    double R[K + 1], g[K + 1];
#pragma unroll
    for (int r = 0; r <= K; ++r) {
        R[r] = lane < K && r <= lane + 1 ? H[(size_t)lane * (kMaxInner + 1) + r] : 0.0;
        g[r] = 0.0;
    }
    const double beta = H[kBetaSlot];
    g[0] = beta;
    int used = K;
#pragma unroll
    for (int c = 0; c < K; ++c) {
        if (used < K) continue;
        const double a = __shfl_sync(0xffffffffu, R[c], c), b = __shfl_sync(0xffffffffu, R[c + 1], c);
        const double rr = sqrt(a * a + b * b);
        if (!(rr > 1e-300 * (beta > 0 ? beta : 1.0))) {
            used = c;
            continue;
        }
        const double cs = a / rr, sn = b / rr;
        const double x0 = R[c], x1 = R[c + 1];
        R[c] = cs * x0 + sn * x1;
        R[c + 1] = -sn * x0 + cs * x1;
        const double g0 = g[c], g1 = g[c + 1];
        g[c] = cs * g0 + sn * g1;
        g[c + 1] = -sn * g0 + cs * g1;
    }
    double y = 0.0;  // lane q: y_q
#pragma unroll
    for (int c = K - 1; c >= 0; --c) {
        if (c >= used) continue;
        const double yc = g[c] / __shfl_sync(0xffffffffu, R[c], c);
        if (lane == c) y = yc;
#pragma unroll
        for (int r = 0; r < c; ++r) g[r] -= __shfl_sync(0xffffffffu, R[r], c) * yc;
    }
    if (lane < kMaxInner) {
        const double nq = lane < K ? nrm[lane] : 0.0;
        H[kBetaSlot + 1 + lane] = nq > 0.0 ? y / nq : 0.0;
    }
}

// The norm of U_K orthogonalised as above (not stored: nothing reads it), and
// the K-step least squares solution by the last block.
template <int K>
__global__ void __launch_bounds__(kInnerThreads) k_inner_last(const float* U, size_t ld, double* H, const double* nrm,
                                                              double* part, unsigned* ticket) {
    pdl_wait();
    __shared__ float cs[kMaxInner];
    double* hj = H + (size_t)(K - 1) * (kMaxInner + 1);
    inner_factors(cs, hj, nrm, K);
    double s = 0.0;
    for (size_t k = 2 * (blockIdx.x * (size_t)kInnerThreads + threadIdx.x); k < ld;
         k += 2 * (size_t)gridDim.x * kInnerThreads) {
        const float2 u = inner_pair(U, ld, K, cs, k);
        s += (double)u.x * u.x;
        s += (double)u.y * u.y;
    }
    block_partial(s, part);
    if (!last_block(ticket)) return;
    if (threadIdx.x < 32) {
        const double t = sqrt(warp_sum_parts(part, gridDim.x));
        if (threadIdx.x == 0) {
            hj[K] = t;
            *ticket = 0;
        }
        __syncwarp();
        inner_lsq<K>(H, nrm);
    }
}

// x = post(b, sum_i c_i Z_i): x[0:6N] = b - y, x[6N:11N] = b, x[11N:] = y.
__global__ void k_inner_post(const float* Z, size_t ld, int k, const double* c,
                             const float* b, float* x, int N) {
    pdl_wait();
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    if (kk < 6 * N) {
        float acc = 0.f;
        for (int i = 0; i < k; ++i) acc += (float)c[i] * Z[(size_t)i * ld + kk];
        const float bk = b[kk];
        x[kk] = bk - acc;
        x[11 * (size_t)N + kk] = acc;
    } else if (kk < 11 * N) {
        x[kk] = b[kk];
    }
}

static int inner_alloc(fsd_handle* h) {
    LearnedState* s = learned(h);
    if (s->inner_cap >= 0) return FSD_OK;
    const size_t N = h->p.N;
    const size_t n6 = 6 * N;
    FSD_CHECK_CUDA(cudaMalloc(&s->Vi, sizeof(float) * n6 * (kMaxInner + 1)));
    FSD_CHECK_CUDA(cudaMalloc(&s->Zi, sizeof(float) * n6 * kMaxInner));
    const size_t nb = std::max<size_t>(kInnerRowBlocks, (8 * N + 255) / 256);
    FSD_CHECK_CUDA(cudaMalloc(&s->part, sizeof(double) * (kMaxInner + 1) * nb));
    FSD_CHECK_CUDA(cudaMalloc(&s->H, sizeof(double) * ((kMaxInner + 1) * kMaxInner + 1 + kMaxInner)));
    FSD_CHECK_CUDA(cudaMalloc(&s->nrm, sizeof(double) * (kMaxInner + 1)));
    FSD_CHECK_CUDA(cudaMalloc(&s->ticket, sizeof(unsigned)));
    FSD_CHECK_CUDA(cudaMemsetAsync(s->ticket, 0, sizeof(unsigned), h->stream));
    s->inner_cap = kMaxInner;
    return FSD_OK;
}

bool precond_is_flexible(const fsd_handle* h) {
    return h->p.precond == FSD_PRECOND_LEARNED && h->p.learned_inner > 0 && !poly_active(h);
}

// Blocks of a kernel with eight lanes per row.
static int inner_rows(int N) { return (8 * N + kInnerThreads - 1) / kInnerThreads; }

// Blocks of a kernel with a warp per row: every warp takes about the same number of rows.
static int inner_warps(int N) {
    const int need = (N + 7) / 8, rounds = (need + kInnerRowBlocks - 1) / kInnerRowBlocks;
    return (need + rounds - 1) / rounds;
}

// k_inner_last of k steps.
template <int K = 1, class... Args>
static void launch_inner_last(int k, cudaStream_t st, Args... args) {
    if constexpr (K <= kMaxInner) {
        if (k == K) launch_pdl(k_inner_last<K>, kInnerBlocks, kInnerThreads, 0, st, args...);
        else launch_inner_last<K + 1>(k, st, args...);
    }
}

// Kernels of one inner solve on the right-hand side b into x, enqueued on st
// (for graph capture).
static int inner_enqueue(fsd_handle* h, const float* b, float* x, cudaStream_t st) {
    LearnedState* s = learned(h);
    const int N = h->p.N;
    const int k = h->p.learned_inner;
    const size_t n6 = 6 * (size_t)N;
    const int rows = inner_rows(N), warps = inner_warps(N);
    const int pairs = (int)((n6 / 2 + kInnerThreads - 1) / kInnerThreads);
    launch_pdl(k_inner_g<true>, warps, kInnerThreads, 0, st, s->g_rowptr, s->g_col, s->g_val, b, s->Vi, s->Zi, N,
                                                    s->H + kBetaSlot, s->nrm, s->part, s->ticket);
    for (int j = 0; j < k; ++j) {
        double* hj = s->H + (size_t)j * (kMaxInner + 1);
        float* zj = s->Zi + (size_t)j * n6;
        launch_pdl(k_inner_a, rows, kInnerThreads, 0, st, s->a_pn, s->a_plist, s->a_blocks, zj, s->Vi, n6, j + 1, s->nrm,
                                                  s->part, s->ticket, s->H, j, N);
        if (j == k - 1) break;
        launch_pdl(k_inner_orth, pairs, kInnerThreads, 0, st, s->Vi, n6, j + 1, hj, s->nrm);
        launch_pdl(k_inner_g<false>, warps, kInnerThreads, 0, st, s->g_rowptr, s->g_col, s->g_val, b, s->Vi + (j + 1) * n6,
                                                         zj + n6, N, hj + j + 1, s->nrm + j + 1, s->part, s->ticket);
    }
    launch_inner_last(k, st, s->Vi, n6, s->H, s->nrm, s->part, s->ticket);
    launch_pdl(k_inner_post, (11 * N + 255) / 256, 256, 0, st, s->Zi, n6, k, s->H + kBetaSlot + 1, b, x, N);
    FSD_CHECK_CUDA(cudaGetLastError());
    return FSD_OK;
}

static int inner_kernels(int k) { return 3 * k + 1; }

// (Re)capture the inner solve when the arrays it reads were reallocated or k
// changed.  The first and last kernel nodes (the only ones that touch b and
// x) are kept so that each application can point them at its own vectors.
static int inner_graph(fsd_handle* h, const float* b, float* x) {
    LearnedState* s = learned(h);
    const void* key[8] = {s->g_rowptr, s->g_col, s->g_val, s->a_pn, s->a_plist, s->a_blocks, s->Vi, s->Zi};
    bool same = s->gexec && s->gkey_k == h->p.learned_inner;
    for (int i = 0; i < 8 && same; ++i) same = key[i] == s->gkey[i];
    if (same) return FSD_OK;
    if (s->gexec) cudaGraphExecDestroy(s->gexec);
    if (s->graph) cudaGraphDestroy(s->graph);
    s->gexec = nullptr;
    s->graph = nullptr;
    if (!s->cap_stream) FSD_CHECK_CUDA(cudaStreamCreateWithFlags(&s->cap_stream, cudaStreamNonBlocking));
    cudaGraph_t g = nullptr;
    FSD_CHECK_CUDA(cudaStreamBeginCapture(s->cap_stream, cudaStreamCaptureModeThreadLocal));
    const int e = inner_enqueue(h, b, x, s->cap_stream);
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
    s->node_rhs = s->node_post = nullptr;
    for (cudaGraphNode_t nd : nodes) {
        cudaGraphNodeType t;
        FSD_CHECK_CUDA(cudaGraphNodeGetType(nd, &t));
        if (t != cudaGraphNodeTypeKernel) continue;
        cudaKernelNodeParams kp;
        FSD_CHECK_CUDA(cudaGraphKernelNodeGetParams(nd, &kp));
        if (kp.func == (void*)k_inner_g<true>) s->node_rhs = nd;
        if (kp.func == (void*)k_inner_post) s->node_post = nd;
    }
    if (!s->node_rhs || !s->node_post) {
        cudaGraphDestroy(g);
        return FSD_ERR_CUDA;
    }
    const cudaError_t ie = cudaGraphInstantiate(&s->gexec, g, 0);
    if (ie != cudaSuccess) {
        cudaGraphDestroy(g);
        FSD_CHECK_CUDA(ie);
    }
    s->graph = g;
    for (int i = 0; i < 8; ++i) s->gkey[i] = key[i];
    s->gkey_k = h->p.learned_inner;
    s->captures += 1;
    if (getenv("FSD_DEBUG_GRAPH")) fprintf(stderr, "inner graph captured (%d)\n", s->captures);
    return FSD_OK;
}

// Point the graph's first and last kernels at b and x.
static int inner_bind(fsd_handle* h, const float* b, float* x) {
    LearnedState* s = learned(h);
    int N = h->p.N;
    size_t ld = 6 * (size_t)N;
    double* beta = s->H + kBetaSlot;
    void* rhs_args[] = {&s->g_rowptr, &s->g_col, &s->g_val, &b,       &s->Vi,    &s->Zi,
                        &N,           &beta,     &s->nrm,   &s->part, &s->ticket};
    cudaKernelNodeParams kr = {};
    kr.func = (void*)k_inner_g<true>;
    kr.gridDim = dim3(inner_warps(N));
    kr.blockDim = dim3(kInnerThreads);
    kr.kernelParams = rhs_args;
    FSD_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(s->gexec, s->node_rhs, &kr));
    const float* Z = s->Zi;
    int k = h->p.learned_inner;
    const double* c = s->H + kBetaSlot + 1;
    void* post_args[] = {&Z, &ld, &k, &c, &b, &x, &N};
    cudaKernelNodeParams kp = {};
    kp.func = (void*)k_inner_post;
    kp.gridDim = dim3((11 * N + 255) / 256);
    kp.blockDim = dim3(256);
    kp.kernelParams = post_args;
    FSD_CHECK_CUDA(cudaGraphExecKernelNodeSetParams(s->gexec, s->node_post, &kp));
    return FSD_OK;
}

// x = P^-1 b.  Without inner steps G is applied once (fused with the saddle
// pre/post steps).  With k inner steps, y ~ (R_FU^pruned + D)^-1 t comes from
// k steps of GMRES on that matrix from a zero guess, right-preconditioned by
// G; the map b -> x then depends on b nonlinearly, which the flexible outer
// GMRES allows.  The inner solve is one CUDA graph launch reading b and
// writing x directly; no host synchronisation.  With inner steps or the
// polynomial b and x may be the same vector; G applied once gathers from b
// while it writes x, so they must not overlap.
int precond_apply_learned(fsd_handle* h, const float* b, float* x) {
    LearnedState* s = learned(h);
    const int N = h->p.N;
    cudaStream_t st = h->stream;
    if (poly_active(h)) return poly_apply(h, b, x);
    const int k = h->p.learned_inner;
    if (k == 0) {
        BsrArgs a{};
        a.rowptr = s->g_rowptr;
        a.col = s->g_col;
        a.val = s->g_val;
        a.N = N;
        a.b = b;
        a.xs = x;
        count_launch();
        bsr_launch(kBsrOnce, a, st);
        FSD_CHECK_CUDA(cudaGetLastError());
        return FSD_OK;
    }
    int e = inner_graph(h, b, x);
    if (e != FSD_OK) return e;
    e = inner_bind(h, b, x);
    if (e != FSD_OK) return e;
    FSD_CHECK_CUDA(cudaGraphLaunch(s->gexec, st));
    for (int i = 0; i < inner_kernels(k); ++i) count_launch();
    return FSD_OK;
}

// Blocks set through fsd_precond_set_blocks are used as given.  Otherwise G
// is the two-hop sparse approximate inverse of the pruned matrix, plus the
// loaded network's correction on the same pattern.
int precond_build_learned(fsd_handle* h, const float4* pos) {
    LearnedState* s = learned(h);
    ProfRegion pr(h, R_PRECOND_BUILD);
    int e = FSD_OK;
    const bool poly = h->p.learned_poly >= 2;
    if (poly) e = poly_alloc(h);
    else if (h->p.learned_inner > 0) e = inner_alloc(h);
    if (e != FSD_OK) return e;
    e = precond_assemble_pruned(h, pos, 1.0f, &s->a_pn, &s->a_plist, &s->a_blocks);
    if (e != FSD_OK) return e;
    if (!s->g_user) {
        e = spai_build(h);
        if (e != FSD_OK) return e;
        // The network either predicts the inner polynomial (learned_poly) or
        // corrects G on its own pattern.
        if (mpnn_loaded(h) && !poly) {
            e = mpnn_infer(h, pos, s->a_pn, s->a_plist, s->a_blocks);
            if (e != FSD_OK) return e;
        }
    }
    if (poly) {
        e = poly_lambda(h);
        if (e != FSD_OK) return e;
        // Coefficients: the caller's; else the Chebyshev interval whose lower
        // end the network predicts for this configuration; else a fixed
        // interval ratio (poly_interval > 0); else a least-squares fit on
        // probe vectors.
        s->poly_ratio = -1.f;
        if (s->poly_user) {
            s->poly_source = 3;
        } else if (s->user_ratio > 0.f) {
            e = poly_set_interval(h, s->user_ratio);
            if (e != FSD_OK) return e;
            s->poly_source = 4;
        } else if (mpnn_loaded(h)) {
            double rho = 0.0;
            float log_rho = 0.f;
            e = mpnn_poly_ratio(h, pos, &rho, &log_rho);
            if (e != FSD_OK) return e;
            const bool finite = std::isfinite(log_rho);  // else the fixed interval (or 0.05)
            e = poly_set_interval(h, finite ? rho : (h->p.poly_interval > 0.f ? h->p.poly_interval : 0.05));
            if (e != FSD_OK) return e;
            s->poly_source = finite ? 1 : 4;
        } else if (h->p.poly_interval > 0.f) {
            e = poly_set_interval(h, h->p.poly_interval);
            if (e != FSD_OK) return e;
            s->poly_source = 4;
        } else {
            e = mpnn_poly_calibrate(h, h->p.learned_poly, ++s->poly_builds);
            if (e != FSD_OK) return e;
        }
    }
    h->pc_valid = true;
    return FSD_OK;
}

int learned_set_weights(fsd_handle* h, const float* host_w, int n) {
    const int e = mpnn_set_weights(h, host_w, n);
    if (e == FSD_OK) {
        learned(h)->g_user = false;
        learned(h)->poly_user = false;  // the network's coefficients from now on
        learned(h)->user_ratio = -1.f;
    }
    return e;
}

}  // namespace fsd
