// Sparse approximate inverse of A = R_FU^pruned + D on the two-hop pattern of
// the pruned contact graph (the base of FSD_PRECOND_LEARNED).
//
// For each particle c, S_c = {c} + pruned neighbours + their pruned
// neighbours (first kSpaiCap, in that order).  The columns of A restricted to
// S_c give the least-squares problem
//     min || A[:, S_c] X_c - E_c ||_F,     E_c = the 6 columns of particle c,
// whose normal equations (A^2)[S_c, S_c] X_c = A[S_c, c] are assembled and
// solved by block Cholesky in FP64, one CTA per particle with the lower
// triangle in shared memory as 6x6 blocks.  X_c is column c of a right
// approximate inverse, A G ~ I (Grote and Huckle's SPAI with a fixed pattern),
// which suits the right-preconditioned inner GMRES.
// Launches are bucketed by |S_c| so that small systems share an SM.
//
// Latency-bound FP64 work on small matrices (2.7 GFMA in all at N = 32768,
// phi = 0.4).  One thread per pair for the assembly, one thread for each
// pivot block and one thread per entry of the trailing update took 10.7 ms
// there, this 5.0 ms: a pivot block is factored by six lanes and one step ahead of the
// trailing update (which the other warps run meanwhile), six lanes update a
// block with its rows in registers, and the right-hand side rides along as one
// more block row.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fsd_device.cuh"
#include "fsd_kernels.cuh"
#include "fsd_learned.h"
#include "fsd_profile.h"
#include "fsd_solver.h"

namespace fsd {

namespace {
// Buckets of set sizes (particles per two-hop set): each launch sizes its
// shared memory for its largest set, and its warps so that the CTAs that fit an
// SM hold 16 to 24 of them.
constexpr int kBuckets = 6;
constexpr int kBucketMax[kBuckets] = {8, 12, 16, 20, 24, kSpaiCap};
__host__ __device__ constexpr int bucket_of(int n) { return n <= 8 ? 0 : n <= 12 ? 1 : n <= 16 ? 2 : n <= 20 ? 3 : n <= 24 ? 4 : 5; }

// FP64 blocks of the lower triangle and of the right-hand side's row.
__host__ __device__ constexpr int spai_blocks(int m) { return m * (m + 1) / 2 + m; }
inline size_t spai_smem(int m) { return sizeof(double) * 36 * spai_blocks(m) + sizeof(int) * m * (kPrunedCap + 2); }
}  // namespace

// Two-hop sets (c first, then the 1-hop list, then new 2-hop members in list
// order), truncated at kSpaiCap; bucket lists for the solve launches.
__global__ void k_spai_sets(const unsigned* __restrict__ pn, const unsigned* __restrict__ plist, int N, int* sets,
                            unsigned* ns, unsigned* bucket_cnt, int* bucket_list, int* truncated) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    int* S = sets + (size_t)c * kSpaiCap;
    int n = 0;
    bool over = false;
    S[n++] = c;
    const unsigned* row = plist + (size_t)c * kPrunedCap;
    for (unsigned q = 0; q < pn[c]; ++q)
        if ((int)row[q] != c) {
            if (n < kSpaiCap) S[n++] = (int)row[q];
            else over = true;
        }
    const int n1 = n;
    for (int a = 1; a < n1; ++a) {
        const int k = S[a];
        const unsigned* rk = plist + (size_t)k * kPrunedCap;
        for (unsigned q = 0; q < pn[k]; ++q) {
            const int s = (int)rk[q];
            bool seen = false;
            for (int b = 0; b < n; ++b)
                if (S[b] == s) {
                    seen = true;
                    break;
                }
            if (seen) continue;
            if (n < kSpaiCap) S[n++] = s;
            else over = true;
        }
    }
    ns[c] = (unsigned)n;
    if (over) atomicAdd(truncated, 1);
    const int b = bucket_of(n);
    const unsigned slot = atomicAdd(bucket_cnt + b, 1u);
    bucket_list[(size_t)b * N + slot] = c;
}

__device__ __forceinline__ int tri_block(int a, int b) { return (a * (a + 1) / 2 + b) * 36; }  // a >= b

// (a, b), b <= a, of entry t of a lower triangle stored by rows.
__device__ __forceinline__ void tri_decode(int t, int& a, int& b) {
    a = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while ((a + 1) * (a + 2) / 2 <= t) ++a;
    while (a * (a + 1) / 2 > t) --a;
    b = t - a * (a + 1) / 2;
}

// Block (s, k) of A from the pruned list of s (k must be on it), or null.
__device__ __forceinline__ const float* a_block(const unsigned* pn, const unsigned* plist, const float* A, int s,
                                                int k) {
    const unsigned* row = plist + (size_t)s * kPrunedCap;
    const unsigned n = pn[s];
    for (unsigned q = 0; q < n; ++q)
        if ((int)row[q] == k) return A + ((size_t)s * kPrunedCap + q) * 36;
    return nullptr;
}

__device__ __forceinline__ void load_row6(const double* p, double* v) {  // 16-byte aligned
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 x = q[0], y = q[1], z = q[2];
    v[0] = x.x;
    v[1] = x.y;
    v[2] = y.x;
    v[3] = y.y;
    v[4] = z.x;
    v[5] = z.y;
}
__device__ __forceinline__ void store_row6(double* p, const double* v) {
    double2* q = reinterpret_cast<double2*>(p);
    q[0] = make_double2(v[0], v[1]);
    q[1] = make_double2(v[2], v[3]);
    q[2] = make_double2(v[4], v[5]);
}

// Cholesky factor of the 6x6 block at d by one warp (lane r < 6 holds row r);
// the diagonal keeps 1 / L_jj.  Returns false on a non-positive pivot.
__device__ __forceinline__ bool factor6(double* d) {
    const int lane = threadIdx.x & 31;
    const int r = lane < 6 ? lane : 0;
    double a[6];
    load_row6(d + 6 * r, a);
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        double pv = __shfl_sync(0xffffffffu, a[j], j);
        if (!(pv > 0.0)) {
            ok = false;
            pv = 1.0;
        }
        const double inv = rsqrt(pv);
        const double l = a[j] * inv;
        a[j] = r == j ? inv : l;
#pragma unroll
        for (int c = j + 1; c < 6; ++c) a[c] -= l * __shfl_sync(0xffffffffu, l, c);
    }
    if (lane < 6) store_row6(d + 6 * r, a);
    return ok;
}

// Row r of C (a, b) -= P_a P_b^T, P_a = (a, jb), P_b = (b, jb).
__device__ __forceinline__ void update_row(double* c, const double* pa, const double* pb, int r) {
    double v[6], x[6];
    load_row6(pa + 6 * r, x);
    load_row6(c + 6 * r, v);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        double y[6];
        load_row6(pb + 6 * k, y);
        v[k] -= x[0] * y[0] + x[1] * y[1] + x[2] * y[2] + x[3] * y[3] + x[4] * y[4] + x[5] * y[5];
    }
    store_row6(c + 6 * r, v);
}

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_spai_solve(const unsigned* __restrict__ pn,
                                                           const unsigned* __restrict__ plist,
                                                           const float* __restrict__ A, const int* __restrict__ sets,
                                                           const unsigned* __restrict__ ns,
                                                           const unsigned* __restrict__ bucket_cnt,
                                                           const int* __restrict__ bucket_list, int bucket, int N,
                                                           const int* __restrict__ rowptr, float* g_val, int* fail) {
    if (blockIdx.x >= bucket_cnt[bucket]) return;
    const int c = bucket_list[(size_t)bucket * N + blockIdx.x];
    extern __shared__ __align__(16) double H[];  // 6x6 blocks (a, b), b <= a < m, then the right-hand side's (m, b)
    const int m = (int)ns[c];
    int* S = (int*)(H + 36 * spai_blocks(m));
    int* nS = S + m;
    int* list = nS + m;  // m x kPrunedCap: the members' pruned lists
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int a = threadIdx.x; a < m; a += 32 * WARPS) {
        const int s = sets[(size_t)c * kSpaiCap + a];
        S[a] = s;
        nS[a] = (int)pn[s];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < m * kPrunedCap; e += 32 * WARPS) {
        const int a = e / kPrunedCap, q = e - a * kPrunedCap;
        if (q < nS[a]) list[e] = (int)plist[(size_t)S[a] * kPrunedCap + q];
    }
    __syncthreads();
    // Normal matrix: H[a][b] = sum_k A_{s_a k} A_{s_b k}^T over k in both pruned
    // lists (ascending), two lanes per block, three of its rows each.
    const int npairs = m * (m + 1) / 2;
    for (int t = threadIdx.x; t < 2 * npairs; t += 32 * WARPS) {
        int a, b;
        tri_decode(t >> 1, a, b);
        const int r0 = 3 * (t & 1);
        const int na = nS[a], nb = nS[b];
        const int* la = list + a * kPrunedCap;
        const int* lb = list + b * kPrunedCap;
        const float* Aa = A + (size_t)S[a] * kPrunedCap * 36 + 6 * r0;
        const float* Ab = A + (size_t)S[b] * kPrunedCap * 36;
        double acc[3][6];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int q = 0; q < 6; ++q) acc[r][q] = 0.0;
        int ia = 0, ib = 0;
        while (ia < na && ib < nb) {
            const int ka = la[ia], kb = lb[ib];
            if (ka == kb) {
                const float2* Pa = reinterpret_cast<const float2*>(Aa + 36 * ia);
                const float2* Pb = reinterpret_cast<const float2*>(Ab + 36 * ib);
                float2 xa[9];
#pragma unroll
                for (int u = 0; u < 9; ++u) xa[u] = __ldg(Pa + u);
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const float2 y0 = __ldg(Pb + 3 * q), y1 = __ldg(Pb + 3 * q + 1), y2 = __ldg(Pb + 3 * q + 2);
#pragma unroll
                    for (int r = 0; r < 3; ++r)
                        acc[r][q] += (double)xa[3 * r].x * y0.x + (double)xa[3 * r].y * y0.y +
                                     (double)xa[3 * r + 1].x * y1.x + (double)xa[3 * r + 1].y * y1.y +
                                     (double)xa[3 * r + 2].x * y2.x + (double)xa[3 * r + 2].y * y2.y;
                }
            }
            ia += ka <= kb;
            ib += kb <= ka;
        }
        double* o = H + tri_block(a, b) + 6 * r0;
#pragma unroll
        for (int r = 0; r < 3; ++r) store_row6(o + 6 * r, acc[r]);
    }
    // Right-hand side, transposed: row q of block (m, a) is column q of A_{s_a c}.
    for (int t = threadIdx.x; t < 6 * m; t += 32 * WARPS) {
        const int a = t / 6, q = t - 6 * a;
        const int* la = list + a * kPrunedCap;
        int p = -1;
        for (int k = 0; k < nS[a]; ++k)
            if (la[k] == c) p = k;
        const float* blk = A + ((size_t)S[a] * kPrunedCap + (p < 0 ? 0 : p)) * 36;
        double v[6];
#pragma unroll
        for (int r = 0; r < 6; ++r) v[r] = p < 0 ? 0.0 : (double)blk[6 * r + q];
        store_row6(H + tri_block(m, a) + 6 * q, v);
    }
    __shared__ int bad;
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    // Right-looking block Cholesky; the row of the right-hand side (a = m) takes
    // part in the panels and updates, which is the forward substitution.
    if (wid == 0 && !factor6(H) && lane == 0) bad = 1;
    __syncthreads();
    for (int jb = 0; jb < m; ++jb) {
        const double* D = H + tri_block(jb, jb);
        // panel: rows below times L_jj^-T, one row per lane
        for (int t = threadIdx.x; t < 6 * (m - jb); t += 32 * WARPS) {
            const int a = jb + 1 + t / 6, r = t % 6;
            double* row = H + tri_block(a, jb) + 6 * r;
            double x[6];
            load_row6(row, x);
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                double v = x[q];
#pragma unroll
                for (int p = 0; p < q; ++p) v -= x[p] * D[6 * q + p];
                x[q] = v * D[7 * q];
            }
            store_row6(row, x);
        }
        __syncthreads();
        const int T = m - 1 - jb;  // block rows left
        if (T == 0) break;
        // warp 0: the next pivot block, one step ahead
        if (wid == 0) {
            double* d = H + tri_block(jb + 1, jb + 1);
            const double* P = H + tri_block(jb + 1, jb);
            if (lane < 6) update_row(d, P, P, lane);
            __syncwarp();
            if (!factor6(d) && lane == 0) bad = 1;
        }
        // trailing update: five blocks per warp, six lanes each; entry 0 of the
        // triangle is the block above, entries from T (T + 1) / 2 on are the
        // right-hand side's.  Warp 0 comes last in each round.
        const int ntri = T * (T + 1) / 2, items = ntri + T;
        const int g = lane / 6, r = lane - 6 * g;
        for (int t0 = 1 + 5 * ((wid + WARPS - 1) % WARPS); t0 < items; t0 += 5 * WARPS) {
            const int t = t0 + g;
            if (g < 5 && t < items) {
                int a, b;
                if (t < ntri) {
                    tri_decode(t, a, b);
                    a += jb + 1;
                    b += jb + 1;
                } else {
                    a = m;
                    b = jb + 1 + t - ntri;
                }
                update_row(H + tri_block(a, b), H + tri_block(a, jb), H + tri_block(b, jb), r);
            }
        }
        __syncthreads();
    }
    // Backward substitution on the transposed right-hand side: X_jb^T solves
    // x L_jj = y (six lanes, one row each), then leaves the blocks above.
    for (int jb = m - 1; jb >= 0; --jb) {
        double* Y = H + tri_block(m, jb);
        if (wid == 0 && lane < 6) {
            const double* D = H + tri_block(jb, jb);
            double x[6];
            load_row6(Y + 6 * lane, x);
#pragma unroll
            for (int q = 5; q >= 0; --q) {
                double v = x[q];
#pragma unroll
                for (int p = q + 1; p < 6; ++p) v -= x[p] * D[6 * p + q];
                x[q] = v * D[7 * q];
            }
            store_row6(Y + 6 * lane, x);
        }
        __syncthreads();
        for (int t = threadIdx.x; t < 6 * jb; t += 32 * WARPS) {
            const int b = t / 6, r = t - 6 * b;
            const double* L = H + tri_block(jb, b);
            double* y = H + tri_block(m, b) + 6 * r;
            double v[6], x[6];
            load_row6(Y + 6 * r, x);
            load_row6(y, v);
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                double l[6];
                load_row6(L + 6 * q, l);
#pragma unroll
                for (int k = 0; k < 6; ++k) v[k] -= x[q] * l[k];
            }
            store_row6(y, v);
        }
        __syncthreads();
    }
    // Column c of G: block (s_a, c) = X block a, stored (by components) in row s_a
    // at the position of c in that row's set (the sets are mutual unless one was
    // truncated; a block without a slot is dropped).  A failed factorisation
    // (never expected: the normal matrix of a full-rank A[:, S] is SPD) leaves
    // the block-Jacobi inverse in column c.
    if (!bad) {
        for (int a = wid; a < m; a += WARPS) {
            const int sa = S[a];
            const int* Ss = sets + (size_t)sa * kSpaiCap;
            const unsigned hit = __ballot_sync(0xffffffffu, lane < (int)ns[sa] && Ss[lane] == c);
            if (!hit) continue;
            float* out = g_val + (size_t)rowptr[sa] * 36 + 6 * (__ffs(hit) - 1);
            const int ld = 6 * (int)ns[sa];
            const double* X = H + tri_block(m, a);
            for (int k = lane; k < 36; k += 32) out[(k / 6) * ld + k % 6] = (float)X[6 * (k % 6) + k / 6];
        }
    } else if (threadIdx.x == 0) {
        atomicAdd(fail, 1);
        const float* d = a_block(pn, plist, A, c, c);
        double M[6][12];
        for (int r = 0; r < 6; ++r)
            for (int q = 0; q < 12; ++q) M[r][q] = q < 6 ? (double)d[r * 6 + q] : (q - 6 == r ? 1.0 : 0.0);
        for (int k = 0; k < 6; ++k) {
            const double pv = M[k][k] != 0.0 ? 1.0 / M[k][k] : 0.0;
            for (int q = 0; q < 12; ++q) M[k][q] *= pv;
            for (int r = 0; r < 6; ++r)
                if (r != k) {
                    const double f = M[r][k];
                    for (int q = 0; q < 12; ++q) M[r][q] -= f * M[k][q];
                }
        }
        for (int r = 0; r < 6; ++r)
            for (int q = 0; q < 6; ++q) g_val[(size_t)rowptr[c] * 36 + r * 6 * m + q] = (float)M[r][6 + q];
    }
}

// Column indices of G's rows: row s holds its own set.
__global__ void k_spai_cols(const int* __restrict__ sets, const unsigned* __restrict__ ns,
                            const int* __restrict__ rowptr, int N, int* g_col) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= N) return;
    for (unsigned q = 0; q < ns[s]; ++q) g_col[rowptr[s] + q] = sets[(size_t)s * kSpaiCap + q];
}

int spai_build(fsd_handle* h) {
    LearnedState* s = learned(h);
    const int N = h->p.N;
    cudaStream_t st = h->stream;
    if (!s->sp_sets) {
        FSD_CHECK_CUDA(cudaMalloc(&s->sp_sets, sizeof(int) * (size_t)N * kSpaiCap));
        FSD_CHECK_CUDA(cudaMalloc(&s->sp_size, sizeof(unsigned) * N));
        FSD_CHECK_CUDA(cudaMalloc(&s->sp_rowptr, sizeof(unsigned) * (N + 1)));
        FSD_CHECK_CUDA(cudaMalloc(&s->sp_scan, sizeof(unsigned) * scan_scratch_elems(N)));
        FSD_CHECK_CUDA(cudaMalloc(&s->sp_bucket, sizeof(int) * (size_t)kBuckets * N));
        FSD_CHECK_CUDA(cudaMalloc(&s->sp_cnt, sizeof(unsigned) * (kBuckets + 2)));
        FSD_CHECK_CUDA(cudaMallocHost(&s->sp_host, sizeof(unsigned) * (kBuckets + 2)));
    }
    // counters: buckets [0, kBuckets), then truncated sets, then failed rows
    FSD_CHECK_CUDA(cudaMemsetAsync(s->sp_cnt, 0, sizeof(unsigned) * (kBuckets + 2), st));
    int* truncated = (int*)(s->sp_cnt + kBuckets);
    int* fail = (int*)(s->sp_cnt + kBuckets + 1);
    count_launch();
    k_spai_sets<<<(N + 127) / 128, 128, 0, st>>>(s->a_pn, s->a_plist, N, s->sp_sets, s->sp_size, s->sp_cnt,
                                                 s->sp_bucket, truncated);
    exclusive_scan(s->sp_size, s->sp_rowptr, N, s->sp_scan, st);
    // block count, truncated sets and the bucket sizes (the launches below are sized by them)
    FSD_CHECK_CUDA(cudaMemcpyAsync(s->sp_host, s->sp_rowptr + N, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    FSD_CHECK_CUDA(cudaMemcpyAsync(s->sp_host + 1, s->sp_cnt, sizeof(unsigned) * (kBuckets + 1),
                                   cudaMemcpyDeviceToHost, st));
    FSD_CHECK_CUDA(cudaStreamSynchronize(st));
    const int nnzb = (int)s->sp_host[0];
    s->sp_truncated = (int)s->sp_host[1 + kBuckets];
    int e = learned_reserve(h, nnzb);
    if (e != FSD_OK) return e;
    FSD_CHECK_CUDA(cudaMemcpyAsync(s->g_rowptr, s->sp_rowptr, sizeof(int) * (N + 1), cudaMemcpyDeviceToDevice, st));
    FSD_CHECK_CUDA(cudaMemsetAsync(s->g_val, 0, sizeof(float) * 36 * (size_t)nnzb, st));
    count_launch();
    k_spai_cols<<<(N + 127) / 128, 128, 0, st>>>(s->sp_sets, s->sp_size, s->g_rowptr, N, s->g_col);
    auto solve = [&](auto kern, int b, int warps) -> int {
        const unsigned cnt = s->sp_host[1 + b];
        if (cnt == 0) return FSD_OK;
        const size_t smem = spai_smem(kBucketMax[b]);
        FSD_CHECK_CUDA(ensure_smem_limit((const void*)kern, smem));
        count_launch();
        kern<<<cnt, 32 * warps, smem, st>>>(s->a_pn, s->a_plist, s->a_blocks, s->sp_sets, s->sp_size, s->sp_cnt,
                                            s->sp_bucket, b, N, s->g_rowptr, s->g_val, fail);
        return FSD_OK;
    };
    int es = solve(k_spai_solve<16>, 5, 16);  // the longest first
    if (es == FSD_OK) es = solve(k_spai_solve<8>, 4, 8);
    if (es == FSD_OK) es = solve(k_spai_solve<6>, 3, 6);
    if (es == FSD_OK) es = solve(k_spai_solve<4>, 2, 4);
    if (es == FSD_OK) es = solve(k_spai_solve<2>, 1, 2);
    if (es == FSD_OK) es = solve(k_spai_solve<1>, 0, 1);
    if (es != FSD_OK) return es;
    FSD_CHECK_CUDA(cudaGetLastError());
    s->g_nnzb = nnzb;
    return FSD_OK;
}

}  // namespace fsd
