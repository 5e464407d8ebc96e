// swap.cu -- the inter-route swap stage after 2-opt: LocalSearch::swap
// (localSearch.cpp:301-410) on every ant's tour, then the tour length as
// compute_tour_length sums it (vrpHelper.cpp:244-253).
//
// The reference scans positions i < j in order and applies the first exchange
// of two customers whose gain is below -EPSILON and that keeps both routes
// within capacity and max_distance, then resumes the scan at the same i.  Depot
// positions never move (only customers are exchanged), so each position's route
// index is fixed for the whole stage.  Every float expression keeps the
// reference's evaluation order.
//
// One CTA per ant.  Its warps examine consecutive positions i at once, each
// scanning j in order, 64 candidates a round; the lowest i that found an
// exchange is the one the sequential scan would reach first (the positions
// before it have none), it is applied, and the scan resumes there.  Distances
// of tour edges are kept per position, so a candidate costs four independent
// reads of the matrix, three rows of it when it is symmetric.  What bounds it is
// the latency of those reads times the rounds: 302 nodes, 128 ants, 0.28 ms (1.01
// with a warp an ant and eight ants a CTA).
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/cvrp_aco.h"
#include "aco_device.cuh"
#include "kernels.h"

namespace aco {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kMaxWarps = 8;

// Shared arrays of the ant: edge length at every position, route loads and
// lengths, tour, route index of every position.
struct SwapLayout {
    size_t edge, load, dist, tour, rpos, bytes;
};

__host__ __device__ inline SwapLayout swap_layout(int n)
{
    SwapLayout L;
    size_t o = 0;
    L.edge = o; o += (size_t)2 * n * 4;
    L.load = o; o += (size_t)n * 4;
    L.dist = o; o += (size_t)n * 4;
    L.tour = o; o += (size_t)2 * n * 2;
    L.rpos = o; o += (size_t)2 * n * 2;
    L.bytes = (o + 15) & ~(size_t)15;
    return L;
}

// One candidate exchange of positions i and j: the four new edges and both
// routes' loads and lengths after it.
struct Swap {
    bool ok;
    float a, b, c, d; // D(p1, n2), D(n2, s1), D(p2, n1), D(n1, s2)
    int load1, load2;
    float dist1, dist2;
};

__global__ void __launch_bounds__(kMaxWarps * 32) swap_kernel(const ConstructArgs *args, const int *ant_inst,
                                                              const int *ant_base, int max_swaps_per_node)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int s_found[kMaxWarps];
    const int inst = __ldg(ant_inst + blockIdx.x), ant = blockIdx.x - __ldg(ant_base + inst);
    const ConstructArgs &a = args[inst];
    const int n = a.n, ld = a.ld, T = a.T, capacity = a.capacity;
    const float max_dist = a.max_dist, serv = a.serv_time;
    const float *D = a.dist;
    const int *demand = a.demand;
    const bool symmetric = a.sym != 0;
    const SwapLayout L = swap_layout(n);
    float *edge = reinterpret_cast<float *>(sm + L.edge), *rdist = reinterpret_cast<float *>(sm + L.dist);
    int *rload = reinterpret_cast<int *>(sm + L.load);
    uint16_t *tour = reinterpret_cast<uint16_t *>(sm + L.tour), *rpos = reinterpret_cast<uint16_t *>(sm + L.rpos);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    int *gt = a.solutions + (size_t)ant * T;
    const int size = gt[T - 1];
    if (size < 2) return; // a failed construction: nothing to do (its status is already set)
    for (int p = threadIdx.x; p < size; p += blockDim.x) tour[p] = (uint16_t)gt[p];
    __syncthreads();
    for (int p = threadIdx.x; p < size - 1; p += blockDim.x) edge[p] = __ldg(D + (size_t)tour[p] * ld + tour[p + 1]);
    if (warp == 0) { // route index of every position (depots at or before it, counted from position 1)
        int base = 0;
        for (int p0 = 0; p0 < size; p0 += 32) {
            const int p = p0 + lane;
            const unsigned m = __ballot_sync(FULL, p >= 1 && p < size && tour[p] == 0);
            if (p < size) rpos[p] = (uint16_t)(base + __popc(m & ((1u << lane) - 1u)));
            base += __popc(m);
        }
    }
    __syncthreads();
    // route loads and lengths (localSearch.cpp:322-341): one thread per route
    // walks it; the route of a depot position p >= 1 ends there
    for (int p = 1 + threadIdx.x; p < size; p += blockDim.x) {
        if (tour[p] != 0) continue;
        int beg = p - 1;
        while (beg > 0 && tour[beg] != 0) beg--;
        int load = 0;
        float dd = 0.f;
        for (int q = beg + 1; q <= p; q++) {
            load += __ldg(demand + tour[q]);
            dd = __fadd_rn(dd, edge[q - 1]);
        }
        const int k = rpos[p];
        rload[k] = load;
        rdist[k] = __fadd_rn(dd, __fmul_rn(serv, (float)(p - beg - 1)));
    }
    __syncthreads();

    const int max_swaps = max_swaps_per_node * n;
    int swaps = 0;
    bool over = false;
    for (int i0 = 1; i0 < size && !over;) {
        const int i = i0 + warp, n1 = i < size ? tour[i] : 0;
        int hit_j = 0, hit_n2 = 0, hit_lane = 0;
        Swap hit;
        if (n1 != 0) {
            const int p1 = tour[i - 1], s1 = tour[i + 1], r1 = rpos[i], dem1 = __ldg(demand + n1), load_1 = rload[r1];
            const float d_p1_n1 = edge[i - 1], d_n1_s1 = edge[i], dist_1 = rdist[r1];
            const float *row_p1 = D + (size_t)p1 * ld, *row_n1 = D + (size_t)n1 * ld, *row_s1 = D + (size_t)s1 * ld;
            auto eval = [&](int j, int &n2) {
                Swap s;
                n2 = j < size ? tour[j] : 0;
                s.ok = n2 != 0;
                const int jc = s.ok ? j : i + 1; // an in-range position for the reads
                const int x = tour[jc], p2 = tour[jc - 1], s2 = jc + 1 < size ? tour[jc + 1] : 0, r2 = rpos[jc];
                s.a = __ldg(row_p1 + x);
                s.d = __ldg(row_n1 + s2);
                s.b = symmetric ? __ldg(row_s1 + x) : __ldg(D + (size_t)x * ld + s1);
                s.c = symmetric ? __ldg(row_n1 + p2) : __ldg(D + (size_t)p2 * ld + n1);
                const int dem2 = __ldg(demand + x);
                const float d_p2_n2 = edge[jc - 1], d_n2_s2 = jc < size - 1 ? edge[jc] : 0.f;
                float gain;
                if (j == i + 1) {
                    gain = __fadd_rn(-__fadd_rn(d_p1_n1, d_n2_s2), __fadd_rn(s.a, s.d));
                } else {
                    const float rem = __fadd_rn(__fadd_rn(__fadd_rn(d_p1_n1, d_n1_s1), d_p2_n2), d_n2_s2);
                    const float add = __fadd_rn(__fadd_rn(__fadd_rn(s.a, s.b), s.c), s.d);
                    gain = __fadd_rn(-rem, add);
                }
                if (r1 != r2) {
                    s.load1 = load_1 - dem1 + dem2;
                    s.load2 = rload[r2] - dem2 + dem1;
                    s.dist1 = __fadd_rn(__fsub_rn(dist_1, __fadd_rn(d_p1_n1, d_n1_s1)), __fadd_rn(s.a, s.b));
                    s.dist2 = __fadd_rn(__fsub_rn(rdist[r2], __fadd_rn(d_p2_n2, d_n2_s2)), __fadd_rn(s.c, s.d));
                    s.ok = s.ok && gain < -kEps &&
                           !((s.load1 > capacity || s.load2 > capacity) || (s.dist1 > max_dist || s.dist2 > max_dist));
                } else {
                    s.load1 = s.load2 = load_1;
                    s.dist1 = s.dist2 = __fadd_rn(dist_1, gain);
                    s.ok = s.ok && gain < -kEps;
                }
                return s;
            };
            for (int j0 = i + 1; j0 < size; j0 += 64) { // two groups of 32 with their reads in flight together
                int x0, x1;
                const Swap c0 = eval(j0 + lane, x0), c1 = eval(j0 + 32 + lane, x1);
                const unsigned m0 = __ballot_sync(FULL, c0.ok), m1 = __ballot_sync(FULL, c1.ok);
                if (m0 | m1) {
                    hit = m0 ? c0 : c1;
                    hit_lane = __ffs(m0 ? m0 : m1) - 1;
                    hit_j = j0 + (m0 ? 0 : 32) + hit_lane;
                    hit_n2 = m0 ? x0 : x1; // this lane's; the hit lane's is the one applied
                    break;
                }
            }
        }
        if (lane == 0) s_found[warp] = hit_j;
        __syncthreads();
        const unsigned any = __ballot_sync(FULL, lane < W && s_found[lane & (kMaxWarps - 1)] != 0);
        if (any) {
            const int w = __ffs(any) - 1;
            if (warp == w && lane == hit_lane) {
                const int r1 = rpos[i], r2 = rpos[hit_j];
                tour[i] = (uint16_t)hit_n2;
                tour[hit_j] = (uint16_t)n1;
                rload[r1] = hit.load1;
                rload[r2] = hit.load2;
                rdist[r1] = hit.dist1;
                rdist[r2] = hit.dist2;
                edge[i - 1] = hit.a;
                edge[hit_j] = hit.d;
                if (hit_j == i + 1) {
                    edge[i] = __ldg(D + (size_t)hit_n2 * ld + n1);
                } else {
                    edge[i] = hit.b;
                    edge[hit_j - 1] = hit.c;
                }
            }
            i0 += w; // an accepted swap re-examines its position (the reference's i--)
            over = ++swaps > max_swaps;
        } else {
            i0 += W;
        }
        __syncthreads();
    }
    if (over && threadIdx.x == 0) set_status(a.status, ACO_ERR_LS_LIMIT);
    for (int p = threadIdx.x; p < size; p += blockDim.x) gt[p] = tour[p];
    if (warp != 0) return;
    // compute_tour_length: fp32 sum of the edges in position order
    float len = 0.f;
    for (int b0 = 0; b0 < size - 1; b0 += 32) {
        const float e = b0 + lane < size - 1 ? edge[b0 + lane] : 0.f;
        const int m = size - 1 - b0 < 32 ? size - 1 - b0 : 32;
#pragma unroll
        for (int k = 0; k < 32; k++) {
            const float y = __shfl_sync(FULL, e, k);
            if (k < m) len = __fadd_rn(len, y);
        }
    }
    if (lane == 0) a.lens[ant] = len;
}

} // namespace

size_t swap_smem(int n) { return swap_layout(n).bytes; }

cudaError_t launch_swap(const ConstructArgs *d_args, const int *d_ant_inst, const int *d_ant_base, int total_ants,
                        int warps, size_t smem, int max_swaps_per_node, cudaStream_t st)
{
    const cudaError_t e = cudaFuncSetAttribute(swap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    swap_kernel<<<total_ants, warps * 32, smem, st>>>(d_args, d_ant_inst, d_ant_base, max_swaps_per_node);
    return cudaGetLastError();
}

} // namespace aco
