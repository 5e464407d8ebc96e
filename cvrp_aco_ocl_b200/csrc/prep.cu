// prep.cu -- instance preprocessing on the device: the distance matrix
// (compute_distances, vrpHelper.cpp:160-184, with the per-type formulas of
// vrpHelper.cpp:35-158) and the nearest-neighbour lists (compute_nn_lists,
// vrpHelper.cpp:188-236, sorted by utilities.cpp:246-266), bit-identical to
// the host versions in host.cpp.
//
// Distances: EUC_2D, CEIL_2D and ATT use only correctly rounded operations
// (fp32 products and sums, fp32 or fp64 square root and division), so the
// device reproduces the host bits.  GEO goes through cos/acos, whose last bits
// differ between math libraries; it stays on the host.
//
// Lists: one warp per row stages it; when the list's nodes and the next one have
// distinct distances the warp collects and sorts them (row_list), otherwise
// it runs the reference's quicksort (middle pivot swapped to the
// left end, Lomuto partition with strict <, both halves recursed) on its row in
// shared memory.  Only positions below the list depth
// are needed, so ranges starting at or beyond it are skipped; the ranges are
// disjoint, so the order they are processed in does not matter and the
// smaller one goes first (explicit stack of at most log2(n) + 1 entries).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/cvrp_aco.h"
#include "aco_device.cuh"
#include "kernels.h"

namespace aco {
namespace {

__device__ __forceinline__ float dist_of(const float *x, const float *y, int type, int i, int j)
{
    const float dx = __fsub_rn(x[i], x[j]), dy = __fsub_rn(y[i], y[j]);
    const float s = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
    if (type == ACO_DIST_CEIL_2D) return (float)(int)ceilf(__fsqrt_rn(s));
    if (type == ACO_DIST_ATT) {
        const float r = (float)__dsqrt_rn(__ddiv_rn((double)s, 10.0));
        const float t = (float)(int)r;
        return (float)(t < r ? (int)t + 1 : (int)t);
    }
    return __fsqrt_rn(s);
}

__global__ void dist_kernel(int n, const float *x, const float *y, int type, float *dist, int ld)
{
    const size_t total = (size_t)n * n;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / n), j = (int)(e - (size_t)i * n);
        dist[(size_t)i * ld + j] = dist_of(x, y, type, i, j);
    }
}

constexpr int kStack = 40;

// The reference's quicksort (utilities.cpp:246-266) on one row, stopping below `depth`.
__device__ void sort_row(float *v, int *idx, int n, int depth, int *status)
{
    int sl[kStack], sr[kStack], top = 0;
    sl[0] = 0;
    sr[0] = n - 1;
    top = 1;
    while (top > 0) {
        top--;
        const int l = sl[top], r = sr[top];
        if (l >= r || l >= depth) continue;
        const int m = (l + r) / 2;
        float tv = v[l]; v[l] = v[m]; v[m] = tv;
        int ti = idx[l]; idx[l] = idx[m]; idx[m] = ti;
        int last = l;
        const float pv = v[l];
        for (int k = l + 1; k <= r; k++)
            if (v[k] < pv) {
                ++last;
                tv = v[last]; v[last] = v[k]; v[k] = tv;
                ti = idx[last]; idx[last] = idx[k]; idx[k] = ti;
            }
        tv = v[l]; v[l] = v[last]; v[last] = tv;
        ti = idx[l]; idx[l] = idx[last]; idx[last] = ti;
        // ranges [l, last] and [last+1, r]: push the larger first
        const bool left_small = (last - l) <= (r - last - 1);
        if (top + 2 > kStack) { // cannot happen (depth <= log2(n) + 1); report rather than overflow
            if (status) atomicCAS(status, 0, ACO_ERR_CAPACITY);
            return;
        }
        if (left_small) {
            sl[top] = last + 1; sr[top] = r; top++;
            sl[top] = l; sr[top] = last; top++;
        } else {
            sl[top] = l; sr[top] = last; top++;
            sl[top] = last + 1; sr[top] = r; top++;
        }
    }
}

// The same sort of a whole row by the warp.  While the range [0, r] is long and the
// part right of the pivot starts at or beyond `depth`, only the left part is ever
// looked at again, and the partition leaves it in a simple order: the smaller
// elements in their order, the last of them first, the pivot at the end.  The warp
// makes that by compaction; lane 0 sorts what is left as written.
__device__ void sort_row_warp(float *v, int *idx, int n, int depth, int lane, int *status)
{
    const unsigned FULLM = 0xffffffffu;
    auto swap = [&](int a, int b) {
        if (lane == 0) {
            const float tv = v[a]; v[a] = v[b]; v[b] = tv;
            const int ti = idx[a]; idx[a] = idx[b]; idx[b] = ti;
        }
        __syncwarp();
    };
    int r = n - 1;
    while (r >= 64) {
        swap(0, r / 2);
        const float pv = v[0];
        int last = 0;
        for (int k = 1 + lane; k <= r; k += 32) last += v[k] < pv;
        last = (int)__reduce_add_sync(FULLM, (unsigned)last);
        if (last + 1 < depth) { // the right part is needed too
            swap(0, r / 2);
            break;
        }
        int cnt = 0;
        for (int k0 = 1; k0 <= r; k0 += 32) {
            const int k = k0 + lane;
            const float x = k <= r ? v[k] : 0.f;
            const int ix = k <= r ? idx[k] : 0;
            const bool small = k <= r && x < pv;
            const unsigned m = __ballot_sync(FULLM, small);
            if (small) { // at or before its own place: nothing unread is overwritten
                const int to = 1 + cnt + __popc(m & ((1u << lane) - 1u));
                v[to] = x;
                idx[to] = ix;
            }
            cnt += __popc(m);
            __syncwarp();
        }
        swap(0, last);
        r = last;
    }
    if (lane == 0) sort_row(v, idx, r + 1, depth, status);
    __syncwarp();
}

constexpr int kPick = 64;      // candidates the list's extraction sorts
constexpr int kListWarps = 8;  // warps (rows) of a CTA of the list kernels

// The first `depth` entries of a staged row's list, warp-wide.  When the
// depth + 1 smallest values are all distinct, every correct sort puts the same
// nodes in the first depth positions, so the warp bisects for a value that at
// least depth + 1 and at most kPick of the row are no larger than, collects those
// and sorts them by (value bits, index) -- for values from +0 to +inf the bits
// order as the floats.  Otherwise (a tie decides which node comes first, as with
// integer coordinates, or a row holds a negative value, -0 or NaN) the reference's
// quicksort runs (sort_row_warp), whose partition order settles ties exactly as
// the host's.  On return idx[0, depth) holds the list.  buf: kPick keys of the warp.
// 25.8 k rows of 101-701 nodes, depth 25: 453 -> 148 us against extracting
// the minima one by one (a pass over the row for each) and one lane sorting ties.
__device__ void row_list(float *v, int *idx, unsigned long long *buf, int n, int depth, int lane, int *status)
{
    const unsigned FULLM = 0xffffffffu;
    if (depth < 32) {
        const uint32_t *bits = reinterpret_cast<const uint32_t *>(v);
        uint32_t lo = 0x7f800000u, hi = 0u; // smallest, largest finite value
        bool odd = false;                   // a negative value, -0 or NaN
        for (int i = lane; i < n; i += 32) {
            const uint32_t b = bits[i];
            odd = odd || b > 0x7f800000u;
            lo = min(lo, b);
            hi = b < 0x7f800000u ? max(hi, b) : hi;
        }
        lo = __reduce_min_sync(FULLM, lo);
        hi = __reduce_max_sync(FULLM, hi);
        bool sorted = !__any_sync(FULLM, odd);
        uint32_t t = 0x7f800000u; // every value is a candidate of a short row
        if (sorted && n > kPick) {
            sorted = false;
            uint32_t below = lo; // the bisection's lower end: too few values up to below - 1
            for (int it = 0; it < 32 && below <= hi; it++) {
                t = below + ((hi - below) >> 1);
                int c = 0;
                for (int i = lane; i < n; i += 32) c += bits[i] <= t;
                c = (int)__reduce_add_sync(FULLM, (unsigned)c);
                if (c > depth && c <= kPick) {
                    sorted = true;
                    break;
                }
                if (c <= depth) below = t + 1u;
                else if (t == 0u) break;
                else hi = t - 1u;
            }
        }
        if (sorted) {
            int cnt = 0;
            for (int i0 = 0; i0 < n; i0 += 32) {
                const int i = i0 + lane;
                const bool in = i < n && bits[i] <= t;
                const unsigned m = __ballot_sync(FULLM, in);
                if (in) buf[cnt + __popc(m & ((1u << lane) - 1u))] = ((unsigned long long)bits[i] << 32) | (unsigned)i;
                cnt += __popc(m);
            }
            __syncwarp();
            unsigned long long x = lane < cnt ? buf[lane] : ~0ull, y = lane + 32 < cnt ? buf[lane + 32] : ~0ull;
            // bitonic sort of 64: positions lane and lane + 32
            for (int size = 2; size <= 64; size *= 2) {
                if (size == 64) { // positions lane and lane + 32
                    const unsigned long long l = x < y ? x : y;
                    y = x < y ? y : x;
                    x = l;
                }
                for (int stride = size > 32 ? 16 : size >> 1; stride > 0; stride >>= 1) {
                    const unsigned long long ox = __shfl_xor_sync(FULLM, x, stride), oy = __shfl_xor_sync(FULLM, y, stride);
                    const bool low = (lane & stride) == 0;
                    const bool upx = size >= 64 || (lane & size) == 0, upy = size >= 64 || ((lane + 32) & size) == 0;
                    x = (low == upx) == (x < ox) ? x : ox;
                    y = (low == upy) == (y < oy) ? y : oy;
                }
            }
            // lanes 0..depth hold the depth + 1 smallest in order: a tie among them ends the fast path
            const unsigned nxt = __shfl_down_sync(FULLM, (unsigned)(x >> 32), 1);
            const bool tie = lane < depth && (unsigned)(x >> 32) == nxt;
            if (!__any_sync(FULLM, tie)) {
                if (lane < depth) idx[lane] = (int)(x & 0xffffffffu);
                __syncwarp();
                return;
            }
        }
    }
    sort_row_warp(v, idx, n, depth, lane, status);
}

// One warp per row: the lanes stage the row and pick its list (row_list), the
// lanes write the list.
__global__ void nn_kernel(int n, const float *dist, int ld, int depth, int rows_per_cta, int *nn, int *status)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ unsigned long long buf[kListWarps][kPick];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * rows_per_cta + w;
    if (w >= rows_per_cta || row >= n) return;
    float *v = reinterpret_cast<float *>(sm) + (size_t)w * 2 * n;
    int *idx = reinterpret_cast<int *>(v + n);
    for (int i = lane; i < n; i += 32) {
        v[i] = dist[(size_t)row * ld + i];
        idx[i] = i;
    }
    __syncwarp();
    if (lane == 0) {
        v[row] = __int_as_float(0x7f800000); // the node itself and the depot never make the list
        v[0] = __int_as_float(0x7f800000);
    }
    __syncwarp();
    row_list(v, idx, buf[w], n, depth, lane, status);
    for (int i = lane; i < depth; i += 32) nn[(size_t)row * depth + i] = idx[i];
}


// Distances of every instance's rows, a warp per row (same bits as dist_kernel),
// and the node's rank by (demand, node) for the construct's tables: the number
// of customers before it, the depot first.
__global__ void dist_rows_kernel(const PrepArgs *pa, const int *row_base, const int *row_inst, int total_rows)
{
    const int lane = threadIdx.x & 31;
    const int w0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int g = w0; g < total_rows; g += nw) {
        const int b = row_inst[g];
        const PrepArgs &a = pa[b];
        const int i = g - row_base[b];
        if (a.K > 0) {
            const int d = a.demand[i];
            int before = 0;
            if (i != 0)
                for (int j = 1 + lane; j < a.n; j += 32) {
                    const int e = a.demand[j];
                    before += e < d || (e == d && j < i);
                }
            const int r = i != 0 ? 1 + (int)__reduce_add_sync(0xffffffffu, (unsigned)before) : 0;
            if (lane == 0) {
                a.rank[i] = (uint16_t)r;
                a.perm[r] = (uint16_t)i;
                a.demr[r] = i != 0 ? d : (int)0x80000000;
            }
        }
        if (!a.device_prep) continue;
        float *row = a.dist + (size_t)i * a.ld;
        for (int j = lane; j < a.n; j += 32) row[j] = dist_of(a.x, a.y, a.dist_type, i, j);
    }
}

// Lists and tables of every instance's rows: a warp per row stages it and picks
// its list (row_list, as nn_kernel), and the lanes write the candidate list
// (first K, padded with node 0 to Kp) and the 2-opt list (first nn_ls) straight
// from the list; then, with host-made lists too, the construct's tables by rank.
__global__ void lists_rows_kernel(const PrepArgs *pa, const int *row_base, const int *row_inst, int total_rows,
                                  int rows_per_cta, int n_max, int *status)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ unsigned long long buf[kListWarps][kPick];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *v = reinterpret_cast<float *>(sm) + (size_t)w * 2 * n_max;
    int *idx = reinterpret_cast<int *>(v + n_max);
    for (int g = blockIdx.x * rows_per_cta + w; g < total_rows; g += gridDim.x * rows_per_cta) {
        const int b = row_inst[g];
        const PrepArgs &a = pa[b];
        const int n = a.n, i = g - row_base[b];
        const size_t crow = (size_t)i * a.Kp;
        if (a.device_prep && a.depth > 0) {
            for (int k = lane; k < n; k += 32) {
                v[k] = a.dist[(size_t)i * a.ld + k];
                idx[k] = k;
            }
            __syncwarp();
            if (lane == 0) {
                v[i] = __int_as_float(0x7f800000); // the node itself and the depot never make the list
                v[0] = __int_as_float(0x7f800000);
            }
            __syncwarp();
            row_list(v, idx, buf[w], n, a.depth, lane, status);
            if (a.K > 0)
                for (int j = lane; j < a.Kp; j += 32) a.nn16[crow + j] = (uint16_t)(j < a.K ? idx[j] : 0);
            for (int j = lane; j < a.nn_ls; j += 32) a.nnls[(size_t)i * a.nn_ls + j] = idx[j];
            if (a.nn_ls > 0) { // the list's last distance, and whether unlisted nodes are as far
                const float *row = a.dist + (size_t)i * a.ld;
                const float last = row[idx[a.nn_ls - 1]];
                int more = 0; // nodes at that distance, less the listed ones
                for (int k = lane; k < n; k += 32) more += k != 0 && k != i && row[k] == last;
                for (int j = lane; j < a.nn_ls; j += 32) more -= row[idx[j]] == last;
                more = __reduce_add_sync(0xffffffffu, more);
                if (lane == 0) a.nnr[i] = make_float2(last, more != 0 ? 1.f : 0.f);
            }
        }
        if (a.K > 0) {
            const size_t rrow = (size_t)a.rank[i] * a.Kp;
            for (int j = lane; j < a.Kp; j += 32) { // a lane reads back the entries it wrote
                const int c = a.nn16[crow + j], r = a.rank[c];
                a.nnr16[rrow + j] = (uint16_t)r;
                a.cand32[rrow + j] = (uint32_t)r | ((uint32_t)(a.demand[c] & 0xFFFF) << 16);
                if (a.cdist) a.cdist[rrow + j] = a.dist[(size_t)i * a.ld + c];
            }
        }
        __syncwarp(); // the row's buffers are reused by the warp's next row
    }
}

} // namespace

bool device_dist_supported(int dist_type) { return dist_type != ACO_DIST_GEO; }

size_t nn_rows_per_cta(int n)
{
    const size_t per_row = (size_t)8 * n;
    size_t rows = (size_t)(200 * 1024) / per_row;
    return std::min<size_t>(rows, 32);
}

cudaError_t launch_dist(int n, const float *x, const float *y, int dist_type, float *dist, int ld, int sm_count,
                        cudaStream_t st)
{
    const size_t total = (size_t)n * n;
    const int blocks = (int)std::min<size_t>((total + 255) / 256, (size_t)sm_count * 16);
    dist_kernel<<<std::max(blocks, 1), 256, 0, st>>>(n, x, y, dist_type, dist, ld);
    return cudaGetLastError();
}

cudaError_t launch_nn(int n, const float *dist, int ld, int depth, int *nn, int *status, cudaStream_t st)
{
    int rows = (int)nn_rows_per_cta(n);
    if (rows < 1) return cudaErrorInvalidValue;
    if (rows > kListWarps) rows = kListWarps;
    const size_t smem = (size_t)rows * 8 * n;
    cudaError_t e = cudaFuncSetAttribute(nn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    nn_kernel<<<(n + rows - 1) / rows, 32 * rows, smem, st>>>(n, dist, ld, depth, rows, nn, status);
    return cudaGetLastError();
}

// The ants' lane seeds (g_aco.cpp:714-722): seed i = (int)(T0 + m (m + r_i) A)
// with m = i mod A and r_i the (i+1)-th ran01 draw from rnd_seed, in fp32 as
// written and converted as x86 cvttss2si does (NaN and out-of-range values give
// INT_MIN).  Draw i+1 is x0 * 16807^(i+1) mod (2^31 - 1), so every seed is
// computed independently.  Instance b of a batch draws from rnd_seed + b (int
// arithmetic, as the host adds it).
constexpr int kSeedRun = 16; // consecutive seeds of one ant a thread makes (nloc a multiple of it)

__global__ void seeds_kernel(const PrepArgs *pa, const int *ant_base, const int *ant_inst, long long runs, int nloc,
                             int seed_time, int rnd_seed)
{
    const float t0 = (float)seed_time;
    const int per_ant = nloc / kSeedRun;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < runs;
         e += (long long)gridDim.x * blockDim.x) {
        const int g = (int)(e / per_ant), c = (int)(e - (long long)g * per_ant);
        const int b = ant_inst[g];
        const PrepArgs &a = pa[b];
        const long long i0 = (long long)(g - ant_base[b]) * nloc + (long long)c * kSeedRun;
        long long r = (long long)(int)((unsigned)rnd_seed + (unsigned)b) % 2147483647ll;
        if (r < 0) r += 2147483647ll;
        uint32_t x = pm_mul((uint32_t)r, pm_pow16807(i0 + 1)); // draw i0 + 1; the next ones one step apart
        const float av = (float)a.n_ants;
        for (int k = 0; k < kSeedRun; k++) {
            const long long i = i0 + k;
            const float m = (float)(int)(i % a.n_ants);
            const float v = __fadd_rn(t0, __fmul_rn(__fmul_rn(m, __fadd_rn(m, pm_uniform(x))), av));
            a.seeds[i] = (v >= -2147483648.0f && v < 2147483648.0f) ? __float2int_rz(v) : (int)0x80000000;
            x = pm_mul(x, 16807u);
        }
    }
}

// Scatter of staged uploads: piece k copies bytes [src_off, src_off + bytes)
// of the blob to dst, a CTA a piece (the host cuts large ones, kScatterPiece).  With
// the whole grid on one piece after another, 192 pieces take 105 us, so 5.
__global__ void scatter_kernel(const ScatterPiece *pieces, int count, const unsigned char *blob)
{
    for (int k = blockIdx.x; k < count; k += gridDim.x) {
        const ScatterPiece pc = pieces[k];
        unsigned char *dst = reinterpret_cast<unsigned char *>(pc.dst);
        const unsigned char *src = blob + pc.src_off;
        const unsigned b = (unsigned)pc.bytes, t0 = threadIdx.x, stride = blockDim.x;
        if (((pc.dst | pc.src_off | b) & 15ull) == 0) {
            for (unsigned i = t0; i < b / 16; i += stride)
                reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
        } else if (((pc.dst | pc.src_off | b) & 3ull) == 0) {
            for (unsigned i = t0; i < b / 4; i += stride)
                reinterpret_cast<uint32_t *>(dst)[i] = reinterpret_cast<const uint32_t *>(src)[i];
        } else {
            for (unsigned i = t0; i < b; i += stride) dst[i] = src[i];
        }
    }
}

cudaError_t launch_scatter(const ScatterPiece *d_pieces, int count, const unsigned char *d_blob, int sm_count,
                           cudaStream_t st)
{
    if (count <= 0) return cudaSuccess;
    scatter_kernel<<<std::min(count, sm_count * 8), 256, 0, st>>>(d_pieces, count, d_blob);
    return cudaGetLastError();
}

cudaError_t launch_prep_batch(const PrepArgs *d_args, const int *d_row_base, const int *d_row_inst, int total_rows,
                              int n_max, const int *d_ant_base, const int *d_ant_inst, int total_ants, int nloc,
                              int seed_time, int rnd_seed, int *status, int sm_count, cudaStream_t st)
{
    if (total_rows > 0) {
        const int blocks = std::min((total_rows + 7) / 8, sm_count * 8); // a warp per row, 8 a CTA
        dist_rows_kernel<<<std::max(blocks, 1), 256, 0, st>>>(d_args, d_row_base, d_row_inst, total_rows);
        int rows = (int)nn_rows_per_cta(n_max);
        if (rows < 1) return cudaErrorInvalidValue;
        if (rows > kListWarps) rows = kListWarps;
        const size_t smem = (size_t)rows * 8 * n_max;
        cudaError_t e = cudaFuncSetAttribute(lists_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        const int lblocks = std::min((total_rows + rows - 1) / rows, sm_count * 16);
        lists_rows_kernel<<<std::max(lblocks, 1), 32 * rows, smem, st>>>(d_args, d_row_base, d_row_inst, total_rows,
                                                                         rows, n_max, status);
    }
    if (nloc % kSeedRun != 0) return cudaErrorInvalidValue;
    const long long runs = (long long)total_ants * (nloc / kSeedRun);
    if (runs > 0) {
        long long blocks = (runs + 255) / 256;
        if (blocks > sm_count * 8) blocks = sm_count * 8;
        seeds_kernel<<<(unsigned)blocks, 256, 0, st>>>(d_args, d_ant_base, d_ant_inst, runs, nloc, seed_time, rnd_seed);
    }
    return cudaGetLastError();
}

} // namespace aco

using namespace aco;

extern "C" {

int aco_compute_distances_device(int n, const float *x, const float *y, int dist_type, float *dist, int ld,
                                 void *stream)
{
    if (n < 1 || !x || !y || !dist || ld < n || !device_dist_supported(dist_type)) return ACO_ERR_INVALID;
    int dev = 0, sm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev);
    return launch_dist(n, x, y, dist_type, dist, ld, sm, static_cast<cudaStream_t>(stream)) == cudaSuccess
               ? ACO_OK
               : ACO_ERR_CUDA;
}

int aco_compute_nn_lists_device(int n, const float *dist, int ld, int nn_ls, int nn_ants, int *nn, int *depth,
                                void *stream)
{
    if (n < 2 || !dist || !depth || ld < n || nn_rows_per_cta(n) < 1) return ACO_ERR_INVALID;
    int d = nn_ls >= nn_ants ? nn_ls : nn_ants;
    if (d >= n) d = n - 1;
    if (d < 0) d = 0;
    *depth = d;
    if (d == 0) return ACO_OK;
    if (!nn) return ACO_ERR_INVALID;
    return launch_nn(n, dist, ld, d, nn, nullptr, static_cast<cudaStream_t>(stream)) == cudaSuccess ? ACO_OK
                                                                                                     : ACO_ERR_CUDA;
}

} // extern "C"
