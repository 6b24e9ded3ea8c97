// n-nearest-neighbour stencils on the device: the stencil generation of
// Grid::generateStencilsKDTree (src/grids/grid_interface.cpp:688-725) with the
// k-d tree of external/kdtree/KDTree.h:407-433, bit-identical to the host
// search rbffd_stencils_knn (host_inputs.cpp).
//
// A stencil is the n smallest (squared distance, index) pairs, closest first,
// with the squared distance summed as ((0 + dx^2) + dy^2) + dz^2 in FP64
// without contraction (the k-d tree's distance_squared, KDTree.h:45-51); a
// duplicate point at distance 0 sorted ahead of the centre swaps with it.
// That definition fixes the result whatever order candidates are visited in,
// so the device search only has to see every point that can be among them.
//
// Layout: the points are binned into a uniform cell grid (the host search's) on
// the device -- box, counts per cell, a scan, points scattered into cell order
// as (x, y, z, index); their order within a cell does not matter.  One warp per
// query point (queries taken in cell order, so neighbouring warps read
// neighbouring cells): shell by shell of cells at Chebyshev distance R from the
// query's, it appends the points to a shared-memory buffer of KNN_CAP (distance,
// index) pairs; when the buffer fills it is sorted (bitonic, by distance then
// index) and cut to the best n + 1.  A shell's cells are consecutive along the
// third axis, so a lane looks up one (first, second) pair of coordinates: one
// run of points on the shell's faces, two single cells inside, and the warp
// takes the points of all its lanes' runs 32 at a time.  After a shell, n
// candidates below the searched reach prove that no unvisited point can enter;
// only those candidates are sorted.  The reach is R times the smallest cell edge
// of the axes along which there are cells left to visit: on a flat or straight
// point set the thin axes, whose cells are all visited at once, do not hold the
// search open (40000 points in a plane, n = 31: 136 ms a call while they did, 1.8
// now).  The runs' places are passed between lanes in registers: in shared memory
// they cost the ninth block of an SM (1.37, 1.32 ms at 163842 nodes, n = 50; 32.5,
// 29.9 ms at 40962, 31, half of the points in a thousandth of the box's width).
//
// Bound by the sort and the shells' look-ups.  163842 nodes, n = 50: 1.4 ms of
// kernels, 5.3 ms with one cell looked up at a time by the whole warp and every
// shell sorted; binning on the host took another 7 ms.
//
// The same search serves the reference's default brute-force generator
// (Grid::generateStencilsBruteForce, grid_interface.cpp:637-686): there equal
// distances fall in decreasing index (DESC), with no centre swap; both cut a
// list at the first node not closer than max_st_radius.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "internal.h"

namespace {

constexpr int KNN_CAP = 512;        // candidate buffer per warp (power of two)
constexpr int KNN_WARPS = 4;        // queries per block
constexpr int KNN_MAX_N = KNN_CAP / 2 - 1;

struct CellGrid {
    double lo[3], hc[3];
    int dims[3];
};

__device__ __forceinline__ int cell_coord(const CellGrid& G, double p, int a)
{
    int c = (int)floor((p - G.lo[a]) / G.hc[a]);
    return max(0, min(G.dims[a] - 1, c));
}

template <bool DESC>
__device__ __forceinline__ bool pair_less(double da, int ia, double db, int ib)
{
    return da < db || (da == db && (DESC ? ia > ib : ia < ib));
}

// Sort the first cnt (<= KNN_CAP) entries of (d, id) ascending by distance,
// then index (descending with DESC): a bitonic network over the next power of
// two, the slots beyond cnt padded with +inf distances.  One warp.
template <bool DESC>
__device__ void warp_bitonic_sort(double* d, int* id, int cnt, int lane)
{
    int S = 32;
    while (S < cnt) S <<= 1;
    for (int t = cnt + lane; t < S; t += 32) {
        d[t] = __longlong_as_double(0x7ff0000000000000ll);
        id[t] = 0x7fffffff;
    }
    __syncwarp();
    for (int k = 2; k <= S; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int t = lane; t < S; t += 32) {
                const int p = t ^ j;
                if (p > t) {
                    const bool up = (t & k) == 0;
                    const bool sw = up ? pair_less<DESC>(d[p], id[p], d[t], id[t])
                                       : pair_less<DESC>(d[t], id[t], d[p], id[p]);
                    if (sw) {
                        const double td = d[t];
                        d[t] = d[p];
                        d[p] = td;
                        const int ti = id[t];
                        id[t] = id[p];
                        id[p] = ti;
                    }
                }
            }
            __syncwarp();
        }
}

// ---- binning ---------------------------------------------------------------

constexpr int BOX_BLOCKS = 256, SCAN_THREADS = 512, SCAN_PER = 8, SCAN_TILE = SCAN_THREADS * SCAN_PER;

// part[block] = {min x, y, z, max x, y, z} of the block's points
__global__ void __launch_bounds__(256) k_box(const double* __restrict__ xyz, int N, double* __restrict__ part)
{
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int i = blockIdx.x * 256 + threadIdx.x; i < N; i += gridDim.x * 256)
        for (int a = 0; a < 3; a++) {
            const double v = xyz[3 * (size_t)i + a];
            lo[a] = fmin(lo[a], v);
            hi[a] = fmax(hi[a], v);
        }
    __shared__ double sh[8][6];
    for (int a = 0; a < 3; a++)
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fmin(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmax(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    if ((threadIdx.x & 31) == 0)
        for (int a = 0; a < 3; a++) {
            sh[threadIdx.x >> 5][a] = lo[a];
            sh[threadIdx.x >> 5][3 + a] = hi[a];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = sh[0][threadIdx.x];
        for (int w = 1; w < 8; w++) v = threadIdx.x < 3 ? fmin(v, sh[w][threadIdx.x]) : fmax(v, sh[w][threadIdx.x]);
        part[blockIdx.x * 6 + threadIdx.x] = v;
    }
}

// cell_of[i] and counts, two places on: cnt[cell + 2]
__global__ void k_bin_count(const double* __restrict__ xyz, int N, CellGrid G, int* __restrict__ cell_of, int* cnt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double* p = xyz + 3 * (size_t)i;
    const int c = (cell_coord(G, p[0], 0) * G.dims[1] + cell_coord(G, p[1], 1)) * G.dims[2] + cell_coord(G, p[2], 2);
    cell_of[i] = c;
    atomicAdd(cnt + c + 2, 1);
}

// Inclusive sums of the tile's elements in place; sums[tile] = its total.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(int* __restrict__ x, size_t n, int* __restrict__ sums)
{
    __shared__ int part[SCAN_THREADS];
    const size_t base = (size_t)blockIdx.x * SCAN_TILE + (size_t)threadIdx.x * SCAN_PER;
    int v[SCAN_PER], sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) {
        v[k] = base + k < n ? x[base + k] : 0;
        sum += v[k];
        v[k] = sum;
    }
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 1; o < SCAN_THREADS; o <<= 1) {
        const int t = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
        __syncthreads();
        part[threadIdx.x] += t;
        __syncthreads();
    }
    const int before = part[threadIdx.x] - sum;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++)
        if (base + k < n) x[base + k] = before + v[k];
    if (threadIdx.x == SCAN_THREADS - 1) sums[blockIdx.x] = part[threadIdx.x];
}

// Exclusive sums of the tiles' totals, in place, one block.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_sums(int* sums, int tiles)
{
    __shared__ int part[SCAN_THREADS];
    int carry = 0;
    for (int t0 = 0; t0 < tiles; t0 += SCAN_THREADS) {
        const int t = t0 + threadIdx.x, own = t < tiles ? sums[t] : 0;
        part[threadIdx.x] = own;
        __syncthreads();
        for (int o = 1; o < SCAN_THREADS; o <<= 1) {
            const int v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
            __syncthreads();
            part[threadIdx.x] += v;
            __syncthreads();
        }
        if (t < tiles) sums[t] = carry + part[threadIdx.x] - own;
        carry += part[SCAN_THREADS - 1];
        __syncthreads();
    }
}

__global__ void k_scan_add(int* __restrict__ x, size_t n, const int* __restrict__ sums)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) x[e] += sums[e / SCAN_TILE];
}

// start[cell + 1], the cell's first place, advances to the next cell's: start becomes the usual offsets.
__global__ void k_bin_fill(const double* __restrict__ xyz, const int* __restrict__ cell_of, int N, int* start,
                           double4* __restrict__ pts)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double* p = xyz + 3 * (size_t)i;
    pts[atomicAdd(start + cell_of[i] + 1, 1)] = make_double4(p[0], p[1], p[2], (double)i);
}

// ---- search ------------------------------------------------------------------

template <bool DESC>
__global__ void __launch_bounds__(32 * KNN_WARPS)
k_knn(const double4* __restrict__ pts, const int* __restrict__ start, CellGrid G, int N, int n, double max_radius,
      int* __restrict__ st, int* __restrict__ st_len, int* __restrict__ ties)
{
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ double sd[KNN_WARPS][KNN_CAP];
    __shared__ int si[KNN_WARPS][KNN_CAP];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qs = blockIdx.x * KNN_WARPS + w;  // query slot in cell order
    if (qs >= N) return;
    double* d = sd[w];
    int* id = si[w];
    const double4 q = pts[qs];
    const int qi = (int)q.w;
    const int cc[3] = {cell_coord(G, q.x, 0), cell_coord(G, q.y, 1), cell_coord(G, q.z, 2)};
    const int maxr = max(G.dims[0], max(G.dims[1], G.dims[2]));
    int cnt = 0;
    for (int R = 0; R <= maxr; R++) {
        const int side = 2 * R + 1, pairs = side * side;
        for (int p0 = 0; p0 < pairs; p0 += 32) {
            // this lane's pair of coordinates: a run of points (first, len), then another
            int first = 0, len = 0, second = 0, len2 = 0;
            const int pr = p0 + lane;
            if (pr < pairs) {
                const int da = pr / side - R, db = pr % side - R;
                const int a = cc[0] + da, b = cc[1] + db;
                if (a >= 0 && a < G.dims[0] && b >= 0 && b < G.dims[1]) {
                    const int* const row = start + ((size_t)a * G.dims[1] + b) * G.dims[2];
                    const int c0 = cc[2] - R, c1 = cc[2] + R;
                    if (max(abs(da), abs(db)) == R) {
                        first = row[max(c0, 0)];
                        len = row[min(c1, G.dims[2] - 1) + 1] - first;
                    } else {
                        if (c0 >= 0) {
                            first = row[c0];
                            len = row[c0 + 1] - first;
                        }
                        if (c1 < G.dims[2]) {
                            second = row[c1];
                            len2 = row[c1 + 1] - second;
                        }
                    }
                }
            }
            int upto = len + len2;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, upto, o);
                if (lane >= o) upto += v;
            }
            const int total = __shfl_sync(FULL, upto, 31);
            const int off = upto - len - len2;
            for (int t = 0; t < total; t += 32) {
                if (cnt + 32 > KNN_CAP) {  // full: keep the best n + 1
                    warp_bitonic_sort<DESC>(d, id, cnt, lane);
                    cnt = n + 1;
                }
                const int e = t + lane;
                int o = 0;  // the last lane whose runs begin at or before e
#pragma unroll
                for (int h = 16; h > 0; h >>= 1)
                    if (__shfl_sync(FULL, off, o + h) <= e) o += h;
                const int k = e - __shfl_sync(FULL, off, o), l1 = __shfl_sync(FULL, len, o);
                const int f1 = __shfl_sync(FULL, first, o), f2 = __shfl_sync(FULL, second, o);
                if (e < total) {
                    const double4 p = pts[k < l1 ? f1 + k : f2 + k - l1];
                    const double dx = __dsub_rn(q.x, p.x), dy = __dsub_rn(q.y, p.y), dz = __dsub_rn(q.z, p.z);
                    double v = __dmul_rn(dx, dx);
                    v = __dadd_rn(v, __dmul_rn(dy, dy));
                    v = __dadd_rn(v, __dmul_rn(dz, dz));
                    d[cnt + lane] = v;
                    id[cnt + lane] = (int)p.w;
                }
                __syncwarp();
                cnt += min(32, total - t);
            }
        }
        if (cnt >= n) {
            // every unvisited point is at least reach away, along an axis with cells left
            double reach = INFINITY;
            for (int a = 0; a < 3; a++)
                if (cc[a] - R > 0 || cc[a] + R < G.dims[a] - 1) reach = fmin(reach, R * G.hc[a]);
            const bool all = isinf(reach);
            const double r2 = reach * reach;
            int below = 0;
            for (int t = 0; t < cnt; t += 32)
                below += __popc(__ballot_sync(FULL, t + lane < cnt && d[t + lane] < r2));
            if (below < n && !all && R < maxr) continue;
            if (below >= n) {  // the list is among these
                int kept = 0;
                for (int t = 0; t < cnt; t += 32) {
                    const bool have = t + lane < cnt;
                    const double v = have ? d[t + lane] : 0.0;
                    const int j = have ? id[t + lane] : 0;
                    const bool keep = have && v < r2;
                    const unsigned m = __ballot_sync(FULL, keep);
                    __syncwarp();
                    if (keep) {
                        const int o = kept + __popc(m & ((1u << lane) - 1));
                        d[o] = v;
                        id[o] = j;
                    }
                    __syncwarp();
                    kept += __popc(m);
                }
                cnt = kept;
            }
            warp_bitonic_sort<DESC>(d, id, cnt, lane);
            cnt = min(cnt, n + 1);
            break;
        }
    }
    // d/id hold the sorted best min(cnt, n + 1) candidates; the list stops at
    // the first one not closer than max_radius (the rest: the centre)
    int len = n, centre = n, tie = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        const unsigned out = __ballot_sync(FULL, k < n && !(sqrt(d[k]) < max_radius));
        if (out && len == n) len = k0 + __ffs(out) - 1;
        const unsigned at = __ballot_sync(FULL, k < n && id[k] == qi);
        if (at && centre == n) centre = k0 + __ffs(at) - 1;
        tie |= __any_sync(FULL, k < n && k + 1 < cnt && d[k] == d[k + 1]);
    }
    // k-d tree lists: a duplicate at distance 0 sorted ahead of the centre swaps with it
    const bool swap = !DESC && centre > 0 && centre < len;
    int* out = st + (size_t)qi * n;
    for (int k = lane; k < n; k += 32) {
        int j = k < len ? id[k] : qi;
        if (swap && k == 0) j = qi;
        if (swap && k == centre) j = id[0];
        out[k] = j;
    }
    if (lane == 0) {
        if (st_len) st_len[qi] = len;
        if (tie) atomicAdd(ties, 1);
    }
}

}  // namespace

static int stencils_gpu(rbffd_ctx* ctx, const double* xyz, int N, int n, int method, double max_radius, int* st,
                        int* st_len, int* ties)
{
    if (!ctx || !xyz || !st || N <= 0 || n <= 0 || n > N) return RBFFD_ERR_INVALID;
    if (method != RBFFD_ST_KDTREE && method != RBFFD_ST_BRUTE_FORCE) return RBFFD_ERR_INVALID;
    if (!(max_radius > 0.0)) return RBFFD_ERR_INVALID;
    if (n > KNN_MAX_N) return set_error(ctx, RBFFD_ERR_UNSUPPORTED, "stencil size %d above %d", n, KNN_MAX_N);
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    // points, then stencils, lengths and the tie count, in one allocation; the cells in another once their
    // number is known
    const size_t b_st = (size_t)N * n * sizeof(int), b_len = (size_t)N * sizeof(int);
    const size_t o_xyz = (size_t)N * sizeof(double4), o_cell = o_xyz + (size_t)N * 3 * sizeof(double),
                 o_box = (o_cell + b_len + 15) / 16 * 16, o_tie = o_box + BOX_BLOCKS * 6 * sizeof(double),
                 o_len = o_tie + 16, o_st = (o_len + b_len + 15) / 16 * 16, b_all = o_st + b_st;
    char* all = nullptr;
    int* d_start = nullptr;
    size_t b_start = 0;
    int rc = dev_alloc(ctx, (void**)&all, b_all);
    if (rc) return rc;
    double4* d_pts = (double4*)all;
    double *d_xyz = (double*)(all + o_xyz), *d_box = (double*)(all + o_box);
    int *d_cell = (int*)(all + o_cell), *d_tie = (int*)(all + o_tie), *d_len = (int*)(all + o_len), *d_st = (int*)(all + o_st);
    cudaError_t e = cudaMemcpyAsync(d_xyz, xyz, (size_t)N * 3 * sizeof(double), cudaMemcpyHostToDevice, s);
    const int boxes = std::min(BOX_BLOCKS, (N + 255) / 256);
    std::vector<double> box((size_t)boxes * 6);
    if (e == cudaSuccess) {
        k_box<<<boxes, 256, 0, s>>>(d_xyz, N, d_box);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(box.data(), d_box, box.size() * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) {
        // the host search's cell grid (host_inputs.cpp)
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int b = 0; b < boxes; b++)
            for (int a = 0; a < 3; a++) {
                lo[a] = std::min(lo[a], box[6 * b + a]);
                hi[a] = std::max(hi[a], box[6 * b + 3 + a]);
            }
        const double rk = std::sqrt(4.0 * n / (double)N);
        const double h = std::max(rk * 0.5, 1e-12);
        CellGrid G;
        for (int a = 0; a < 3; a++) {
            G.lo[a] = lo[a];
            G.dims[a] = std::max(1, std::min(400, (int)std::ceil((hi[a] - lo[a]) / h) + 1));
            G.hc[a] = std::max((hi[a] - lo[a]) / G.dims[a], 1e-300) * (1.0 + 1e-12);
        }
        const size_t ncell = (size_t)G.dims[0] * G.dims[1] * G.dims[2], nstart = ncell + 2;
        const int tiles = (int)((nstart + SCAN_TILE - 1) / SCAN_TILE);
        b_start = (nstart + tiles) * sizeof(int);
        if ((rc = dev_alloc(ctx, (void**)&d_start, b_start))) {
            dev_free(ctx, all, b_all);
            return rc;
        }
        int* d_sums = d_start + nstart;
        e = cudaMemsetAsync(d_start, 0, nstart * sizeof(int), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(d_tie, 0, sizeof(int), s);
        if (e == cudaSuccess) {
            k_bin_count<<<(N + 255) / 256, 256, 0, s>>>(d_xyz, N, G, d_cell, d_start);
            k_scan_tiles<<<tiles, SCAN_THREADS, 0, s>>>(d_start, nstart, d_sums);
            k_scan_sums<<<1, SCAN_THREADS, 0, s>>>(d_sums, tiles);
            k_scan_add<<<(unsigned)((nstart + 255) / 256), 256, 0, s>>>(d_start, nstart, d_sums);
            k_bin_fill<<<(N + 255) / 256, 256, 0, s>>>(d_xyz, d_cell, N, d_start, d_pts);
            const unsigned nb = (unsigned)((N + KNN_WARPS - 1) / KNN_WARPS);
            int* len = st_len ? d_len : nullptr;
            if (method == RBFFD_ST_BRUTE_FORCE)
                k_knn<true><<<nb, 32 * KNN_WARPS, 0, s>>>(d_pts, d_start, G, N, n, max_radius, d_st, len, d_tie);
            else
                k_knn<false><<<nb, 32 * KNN_WARPS, 0, s>>>(d_pts, d_start, G, N, n, max_radius, d_st, len, d_tie);
            e = cudaGetLastError();
        }
    }
    int tie = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(st, d_st, b_st, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&tie, d_tie, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && st_len) e = cudaMemcpyAsync(st_len, d_len, b_len, cudaMemcpyDeviceToHost, s);
    const cudaError_t f = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = f;
    dev_free(ctx, all, b_all);
    dev_free(ctx, d_start, b_start);
    if (e != cudaSuccess) return cuda_error(ctx, e, "stencils on the device");
    if (ties) *ties = tie;
    return RBFFD_OK;
}

extern "C" int rbffd_stencils_knn_gpu(rbffd_ctx* ctx, const double* xyz, int N, int n, int* st, int* ties)
{
    return stencils_gpu(ctx, xyz, N, n, RBFFD_ST_KDTREE, DBL_MAX, st, nullptr, ties);
}

extern "C" int rbffd_stencils_generate_gpu(rbffd_ctx* ctx, const double* xyz, int N, int n, int method,
                                           double max_radius, int* st, int* st_len, int* ties)
{
    return stencils_gpu(ctx, xyz, N, n, method, max_radius, st, st_len, ties);
}
