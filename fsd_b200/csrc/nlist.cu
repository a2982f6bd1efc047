// Neighbour list: every pair within r_list = ewald_cut + buffer, both
// directions, no self.  Replaces HOOMD's NeighborListGPUBinned as configured by
// PSEv3 (integrate.py:80-85: cell list, r_buff 0.4, rebuilt every step).
//
// Particles are binned into cells no narrower than r_list (measured between
// opposite faces of the sheared box), each cell's members are sorted by index,
// and each particle scans its 27 neighbouring cells in a fixed order, so row
// contents and order are deterministic.  Boxes with fewer than three cells
// along an axis fall back to an all-pairs scan.
//
// One warp per particle: three cells that follow one another along z are one
// range of the cell order, lanes test its members (positions stored in that
// order, so the reads are contiguous) and a ballot places the hits, in order,
// in the row and in the lubrication sub-list.  A thread per particle, with a
// pass of its own for the sub-list and one thread sorting each cell, took
// 319 + 35 + 39 us at N = 32768, phi = 0.4; the search with the sub-list is
// 71 us.
#include <mutex>

#include "fsd.h"
#include "fsd_device.cuh"
#include "fsd_kernels.cuh"
#include "fsd_profile.h"

namespace fsd {

// ---------------------------------------------------------------- scan utility
// Exclusive scan of n unsigned values, out may alias in.  out[n] receives the
// total.  Uses block-level scans plus one pass over the block sums.
namespace {
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned* sh, unsigned* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        unsigned s = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        sh[lane] = s;
    }
    __syncthreads();
    const unsigned warp_off = wid ? sh[wid - 1] : 0u;
    if (total) *total = sh[(blockDim.x >> 5) - 1];
    return warp_off + x - v;
}

__global__ void scan_tiles(const unsigned* in, unsigned* out, unsigned* sums, int n) {
    __shared__ unsigned sh[32];
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    unsigned v[kScanItems], s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = (base + i < n) ? in[base + i] : 0u;
        s += v[i];
    }
    unsigned total;
    unsigned off = block_exclusive_scan(s, sh, &total);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        if (base + i < n) out[base + i] = off;
        off += v[i];
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void scan_sums(unsigned* sums, int nb, unsigned* out_total) {
    __shared__ unsigned sh[32];
    unsigned carry = 0;
    for (int base = 0; base < nb; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const unsigned v = (i < nb) ? sums[i] : 0u;
        unsigned total;
        const unsigned ex = block_exclusive_scan(v, sh, &total);
        if (i < nb) sums[i] = ex + carry;
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *out_total = carry;
}

__global__ void scan_add(unsigned* out, const unsigned* sums, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += sums[i / kScanTile];
}
}  // namespace

size_t scan_scratch_elems(int n) { return (size_t)(n + kScanTile - 1) / kScanTile + 1; }

void exclusive_scan(const unsigned* in, unsigned* out, int n, unsigned* scratch, cudaStream_t st) {
    const int nb = (n + kScanTile - 1) / kScanTile;
    count_launch();
    scan_tiles<<<nb, kScanThreads, 0, st>>>(in, out, scratch, n);
    count_launch();
    scan_sums<<<1, kScanThreads, 0, st>>>(scratch, nb, out + n);
    count_launch();
    scan_add<<<(n + 255) / 256, 256, 0, st>>>(out, scratch, n);
}

// ------------------------------------------------------------------ cell list
__device__ __forceinline__ int3 cell_of(float4 p, const Box& b, int3 nc) {
    const float3 f = make_fraction(make_float3(p.x, p.y, p.z), b);
    int cx = (int)floorf(f.x * nc.x), cy = (int)floorf(f.y * nc.y), cz = (int)floorf(f.z * nc.z);
    cx = ((cx % nc.x) + nc.x) % nc.x;
    cy = ((cy % nc.y) + nc.y) % nc.y;
    cz = ((cz % nc.z) + nc.z) % nc.z;
    return make_int3(cx, cy, cz);
}

// Cell and slot within it (in the order the atomics gave) of each particle;
// the last block scans the counts.
__global__ void __launch_bounds__(1024) k_cell_count(const float4* pos, int n, Box b, int3 nc,
                                                     unsigned* key, unsigned* slot,
                                                     unsigned* count, unsigned* start,
                                                     unsigned* ticket) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const int3 c = cell_of(pos[i], b, nc);
        const unsigned k = (unsigned)((c.x * nc.y + c.y) * nc.z + c.z);
        key[i] = k;
        slot[i] = atomicAdd(&count[k], 1u);
    }
    __threadfence();
    if (!last_block(ticket)) return;
    block_scan_counts(count, start, nc.x * nc.y * nc.z);
}

__global__ void k_cell_fill(const unsigned* key, const unsigned* slot, int n,
                            const unsigned* start, unsigned* items) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) items[start[key[i]] + slot[i]] = (unsigned)i;
}

// One warp per cell: a member's place is the number of smaller indices.
// sorted_pos (optional) receives the positions in that order, index in w;
// order (optional) a copy of parts.
__global__ void __launch_bounds__(256) k_cell_sort(const float4* pos, const unsigned* start,
                                                   int ncells, const unsigned* items,
                                                   unsigned* parts, unsigned* order,
                                                   float4* sorted_pos) {
    pdl_wait();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (c >= ncells) return;
    const unsigned s0 = start[c], n = start[c + 1] - s0;
    for (unsigned e = lane; e < n; e += 32) {
        const unsigned me = items[s0 + e];
        unsigned rank = 0;
        for (unsigned k = 0; k < n; ++k) rank += items[s0 + k] < me ? 1u : 0u;
        parts[s0 + rank] = me;
        if (order) order[s0 + rank] = me;
        if (sorted_pos) {
            const float4 p = pos[me];
            sorted_pos[s0 + rank] = make_float4(p.x, p.y, p.z, __uint_as_float(me));
        }
    }
}

// Rows of the neighbour list, and of the sub-list within sub2 (optional), one
// warp per particle in cell order.
__global__ void __launch_bounds__(128) k_nlist_cells(const float4* pos, int n, Box b, int3 nc,
                                                     const unsigned* cstart,
                                                     const unsigned* cparts,
                                                     const float4* sorted_pos, float rlist2,
                                                     unsigned* nneigh, unsigned* nlist,
                                                     int stride, int* max_count, float sub2,
                                                     unsigned* sub_n, unsigned* sub) {
    pdl_wait();
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= n) return;
    const unsigned i = cparts[w];
    const float4 pi = pos[i];
    const int3 c = cell_of(pi, b, nc);
    // Runs 2 q and 2 q + 1 of (dx, dy) pair q: cells cz - 1, cz, cz + 1 in that
    // order, as one range of the cell order, or two where they wrap.
    unsigned rs = 0, re = 0;
    if (lane < 18) {
        const int q = lane >> 1;
        const int x = (c.x + q / 3 - 1 + nc.x) % nc.x, y = (c.y + q % 3 - 1 + nc.y) % nc.y;
        const unsigned* cs = cstart + (x * nc.y + y) * nc.z;
        const bool lo = c.z == 0, hi = c.z == nc.z - 1;
        int z0, z1;  // cells [z0, z1)
        if (!(lane & 1)) {
            z0 = lo ? nc.z - 1 : c.z - 1;
            z1 = lo ? nc.z : hi ? nc.z : c.z + 2;
        } else {
            z0 = 0;
            z1 = lo ? 2 : hi ? 1 : 0;
        }
        if (z1 > z0) {
            rs = cs[z0];
            re = cs[z1];
        }
    }
    unsigned* row = nlist + (size_t)i * stride;
    unsigned* srow = sub ? sub + (size_t)i * stride : nullptr;
    unsigned cnt = 0, scnt = 0;
    const unsigned below = (1u << lane) - 1u;
    for (int r = 0; r < 18; ++r) {
        const unsigned s = __shfl_sync(0xffffffffu, rs, r), e = __shfl_sync(0xffffffffu, re, r);
        for (unsigned base = s; base < e; base += 32) {
            const unsigned k = base + lane;
            unsigned j = i;
            float d2 = 0.f;
            if (k < e) {
                float4 pj;
                if (sorted_pos) {
                    pj = sorted_pos[k];
                    j = __float_as_uint(pj.w);
                } else {
                    j = cparts[k];
                    pj = pos[j];
                }
                d2 = dist2_rn(min_image_rn(make_float3(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z), b));
            }
            const bool hit = j != i && d2 < rlist2;
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            const unsigned at = cnt + __popc(m & below);
            if (hit && at < (unsigned)stride) row[at] = j;
            cnt += __popc(m);
            if (srow) {
                const bool near = hit && d2 < sub2;
                const unsigned ms = __ballot_sync(0xffffffffu, near);
                const unsigned as = scnt + __popc(ms & below);
                if (near && as < (unsigned)stride) srow[as] = j;
                scnt += __popc(ms);
            }
        }
    }
    if (lane == 0) {
        nneigh[i] = min(cnt, (unsigned)stride);
        if (srow) sub_n[i] = min(scnt, (unsigned)stride);
        atomicMax(max_count, (int)cnt);
    }
}

__global__ void k_nlist_allpairs(const float4* __restrict__ pos, int n, Box b, float rlist2, unsigned* nneigh,
                                 unsigned* nlist, int stride, int* max_count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 pi = pos[i];
    unsigned cnt = 0;
    unsigned* row = nlist + (size_t)i * stride;
    for (int j = 0; j < n; ++j) {
        if (j == i) continue;
        const float4 pj = pos[j];
        const float3 r = min_image_rn(make_float3(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z), b);
        if (dist2_rn(r) < rlist2) {
            if (cnt < (unsigned)stride) row[cnt] = j;
            ++cnt;
        }
    }
    nneigh[i] = cnt < (unsigned)stride ? cnt : (unsigned)stride;
    atomicMax(max_count, (int)cnt);
}

// Cells per axis so that a cell is at least r_list wide between faces.
int3 cell_dims(const Box& b, float rlist) {
    const float wx = b.Lx / sqrtf(1.0f + b.xy * b.xy);
    int3 nc;
    nc.x = (int)floorf(wx / rlist);
    nc.y = (int)floorf(b.Ly / rlist);
    nc.z = (int)floorf(b.Lz / rlist);
    return nc;
}

// Entries of each particle's neighbour list closer than sqrt(r2), in list
// order (so pair sums over them add in the same order as over the full list):
// the lubrication kernels' list for the all-pairs case.
__global__ void k_sublist(const float4* __restrict__ pos, int n, Box b, const unsigned* __restrict__ nneigh,
                          const unsigned* __restrict__ nlist, int stride, float r2, unsigned* __restrict__ sub_n,
                          unsigned* __restrict__ sub) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 pi = pos[i];
    const unsigned* row = nlist + (size_t)i * stride;
    unsigned* out = sub + (size_t)i * stride;
    const unsigned nn = nneigh[i];
    unsigned k = 0;
    for (unsigned q = 0; q < nn; ++q) {
        const unsigned j = row[q];
        const float4 pj = pos[j];
        const float3 r = min_image(make_float3(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z), b);
        if (r.x * r.x + r.y * r.y + r.z * r.z < r2) out[k++] = j;
    }
    sub_n[i] = k;
}

// Builds the list and the lubrication kernels' sub-list (pairs within rlub
// plus the list buffer, so that it stays complete for as long as the full list
// does); returns the largest neighbour count in *max_count_host.
int build_neighbor_list(fsd_handle* h, const float4* pos, int* max_count_host) {
    Workspace& w = h->w;
    const int n = h->p.N;
    const float rlist = h->ewald_cut + h->p.nlist_buffer;
    const float rlist2 = rlist * rlist;
    const int3 nc = cell_dims(h->box, rlist);
    cudaStream_t st = h->stream;
    ProfRegion pr(h, R_NLIST);
    FSD_CHECK_CUDA(cudaMemsetAsync(w.nl_overflow, 0, sizeof(int), st));
    if (nc.x >= 3 && nc.y >= 3 && nc.z >= 3 && (size_t)nc.x * nc.y * nc.z <= w.ncell_cap) {
        const int ncells = nc.x * nc.y * nc.z;
        FSD_CHECK_CUDA(cudaMemsetAsync(w.cell_count, 0, sizeof(unsigned) * w.ncell_pad, st));
        count_launch();
        launch_pdl(k_cell_count, (n + 1023) / 1024, 1024, 0, st, pos, n, h->box, nc, w.part_cell, w.part_slot, w.cell_count,
                                                         w.cell_start, w.cell_count + w.ncell_pad - 1);
        count_launch();
        launch_pdl(k_cell_fill, (n + 255) / 256, 256, 0, st, w.part_cell, w.part_slot, n, w.cell_start, w.cell_items);
        count_launch();
        launch_pdl(k_cell_sort, (ncells + 7) / 8, 256, 0, st, pos, w.cell_start, ncells, w.cell_items, w.cell_parts, w.order,
                                                      w.cell_pos);
        count_launch();
        const float rsub = h->p.rlub + h->p.nlist_buffer;
        launch_pdl(k_nlist_cells, (n + 3) / 4, 128, 0, st, pos, n, h->box, nc, w.cell_start, w.cell_parts, w.cell_pos, rlist2,
                                                   w.nneigh, w.nlist, w.nl_stride, w.nl_overflow, rsub * rsub,
                                                   w.lub_n, w.lub_list);
    } else {
        count_launch();
        k_nlist_allpairs<<<(n + 127) / 128, 128, 0, st>>>(pos, n, h->box, rlist2, w.nneigh, w.nlist, w.nl_stride,
                                                          w.nl_overflow);
        const float rsub = h->p.rlub + h->p.nlist_buffer;
        count_launch();
        k_sublist<<<(n + 127) / 128, 128, 0, st>>>(pos, n, h->box, w.nneigh, w.nlist, w.nl_stride, rsub * rsub,
                                                   w.lub_n, w.lub_list);
    }
    FSD_CHECK_CUDA(cudaGetLastError());
    FSD_CHECK_CUDA(cudaMemcpyAsync(w.host_flag, w.nl_overflow, sizeof(int), cudaMemcpyDeviceToHost, st));
    FSD_CHECK_CUDA(cudaStreamSynchronize(st));
    *max_count_host = *w.host_flag;
    return FSD_OK;
}

__global__ void k_iota(unsigned* v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (unsigned)i;
}

int init_particle_order(fsd_handle* h) {
    count_launch();
    k_iota<<<(h->p.N + 255) / 256, 256, 0, h->stream>>>(h->w.order, h->p.N);
    FSD_CHECK_CUDA(cudaGetLastError());
    return FSD_OK;
}

// ------------------------------------------- allocation-free neighbour list
// Scratch of fsd_neighbor_list_noalloc: the cell key and cell members of every
// particle and the binning arrays of every cell, in one file-scope
// device array (about 1.25 MiB, held on each device that loads the library
// until the process exits).  All calls on a device share it.
namespace {
constexpr int kNoAllocMaxN = FSD_NOALLOC_MAX_N;
constexpr int kNoAllocMaxCells = FSD_NOALLOC_MAX_CELLS;
static_assert(kNoAllocMaxCells >= kNoAllocMaxN, "the cell counts' space is reused for the particles");
constexpr size_t kOffKey = 0;
constexpr size_t kOffParts = kOffKey + kNoAllocMaxN;
constexpr size_t kOffCount = kOffParts + kNoAllocMaxN;
constexpr size_t kOffSlot = kOffCount + kNoAllocMaxCells;
constexpr size_t kOffStart = kOffSlot + kNoAllocMaxN;
constexpr size_t kOffTicket = kOffStart + kNoAllocMaxCells + 1;
constexpr size_t kNoAllocElems = kOffTicket + 1;

static __device__ __align__(256) unsigned g_nlist_scratch[kNoAllocElems];

// Device address of g_nlist_scratch on the current device, looked up once per
// device.  In host code the array's name is only a host-side stand-in, so the
// kernels are always given this address instead.
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
unsigned* g_scratch_addr[kMaxDevices] = {};

int noalloc_scratch(unsigned** out) {
    int dev = -1;
    FSD_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return FSD_ERR_BAD_PARAMS;
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        FSD_CHECK_CUDA(cudaGetSymbolAddress(&p, g_nlist_scratch));
        g_scratch_addr[dev] = (unsigned*)p;
    }
    *out = g_scratch_addr[dev];
    return FSD_OK;
}
}  // namespace

int neighbor_list_noalloc(const float4* pos, int n, Box b, float rlist, unsigned* nneigh, unsigned* nlist,
                          int stride, int* max_count, cudaStream_t st) {
    unsigned* scratch = nullptr;
    const int e = noalloc_scratch(&scratch);
    if (e != FSD_OK) return e;
    const float rlist2 = rlist * rlist;
    // Cells per axis, clamped to the scratch's cell capacity before the
    // conversion to int (a large box over a small r_list would overflow it).
    const float wx = b.Lx / sqrtf(1.0f + b.xy * b.xy);
    auto axis_cells = [](float len, float r) {
        return (int)fminf(floorf(len / r), (float)kNoAllocMaxCells);
    };
    int3 nc = make_int3(axis_cells(wx, rlist), axis_cells(b.Ly, rlist), axis_cells(b.Lz, rlist));
    // Wider cells than r_list stay correct, so a box with more cells than the
    // scratch holds uses fewer, wider cells along its longest cell axis.
    while ((size_t)nc.x * nc.y * nc.z > (size_t)kNoAllocMaxCells) {
        if (nc.x >= nc.y && nc.x >= nc.z) --nc.x;
        else if (nc.y >= nc.z) --nc.y;
        else --nc.z;
    }
    FSD_CHECK_CUDA(cudaMemsetAsync(max_count, 0, sizeof(int), st));
    if (nc.x >= 3 && nc.y >= 3 && nc.z >= 3) {
        const int ncells = nc.x * nc.y * nc.z;
        unsigned* key = scratch + kOffKey;
        unsigned* parts = scratch + kOffParts;
        unsigned* count = scratch + kOffCount;
        unsigned* start = scratch + kOffStart;
        unsigned* slot = scratch + kOffSlot;
        unsigned* ticket = scratch + kOffTicket;
        FSD_CHECK_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned) * ((ncells + 15) & ~15), st));
        FSD_CHECK_CUDA(cudaMemsetAsync(ticket, 0, sizeof(unsigned), st));
        count_launch();
        launch_pdl(k_cell_count, (n + 1023) / 1024, 1024, 0, st, pos, n, b, nc, key, slot, count, start, ticket);
        unsigned* items = count;  // the counts are not needed past the scan
        count_launch();
        launch_pdl(k_cell_fill, (n + 255) / 256, 256, 0, st, key, slot, n, start, items);
        count_launch();
        launch_pdl(k_cell_sort, (ncells + 7) / 8, 256, 0, st, pos, start, ncells, items, parts, nullptr, nullptr);
        count_launch();
        launch_pdl(k_nlist_cells, (n + 3) / 4, 128, 0, st, pos, n, b, nc, start, parts, nullptr, rlist2, nneigh, nlist, stride,
                                                   max_count, 0.f, nullptr, nullptr);
    } else {
        count_launch();
        k_nlist_allpairs<<<(n + 127) / 128, 128, 0, st>>>(pos, n, b, rlist2, nneigh, nlist, stride, max_count);
    }
    FSD_CHECK_CUDA(cudaGetLastError());
    return FSD_OK;
}

}  // namespace fsd

extern "C" int fsd_neighbor_list_noalloc(const float* d_pos, int N, float Lx, float Ly, float Lz, float xy,
                                         float rlist, unsigned int* d_nneigh, unsigned int* d_nlist, int stride,
                                         int* d_max_count, void* cuda_stream) {
    if (!d_pos || !d_nneigh || !d_nlist || !d_max_count) return FSD_ERR_BAD_PARAMS;
    if (N < 1 || N > FSD_NOALLOC_MAX_N || stride < 1) return FSD_ERR_BAD_PARAMS;
    if (!(rlist > 0.f) || !(Lx > 0.f) || !(Ly > 0.f) || !(Lz > 0.f) || !std::isfinite(rlist) ||
        !std::isfinite(Lx) || !std::isfinite(Ly) || !std::isfinite(Lz) || !std::isfinite(xy))
        return FSD_ERR_BAD_PARAMS;
    return fsd::neighbor_list_noalloc((const float4*)d_pos, N, fsd::Box{Lx, Ly, Lz, xy}, rlist, d_nneigh, d_nlist,
                                      stride, d_max_count, (cudaStream_t)cuda_stream);
}
