// noalloc.cu -- aco_pheromone_update_noalloc: the pheromone update
// (evaporation, rank-based deposit, total_info) for callers that must not have
// this library allocate device memory.
//
// Who needs it: hosts whose own memory manager owns every byte of device memory
// and forbids libraries from calling cudaMalloc (fixed memory budgets, pooled
// allocators), and loops that cannot afford the device-wide synchronisation that
// cudaMalloc / cudaFree imply.  Such a caller passes its own device buffers; the
// update touches no other device memory, so calls on different streams and
// threads do not meet.
//
// Limits: n <= kMaxNodes (4096) nodes and ras_ranks <= kMaxRanks (8); larger
// problems are rejected with ACO_ERR_CAPACITY.
//
// One launch.  A CTA owns a block of matrix rows and finds for itself what its
// rows receive: it selects the elites from the lengths, walks the elite tours (a
// few times 2n ints, from L2) and keeps the edges that leave its rows in shared
// memory, then streams the rows.  What bounds it: the instructions of one CTA's phases
// (37 k a CTA at half the issue slots) and the chain of dependent reads between
// them (lengths, tour sizes, tours; the rows' first part is loaded ahead); 16 MB at
// the copy bandwidth would take 2.5 us.  n = 1001, 256 ants: 12.3 us a call, 28.7 with
// deposit lists written by one CTA for a second launch.
//
// The elite tours come from the caller's buffers, so they are checked before
// they are used as indices: an elite whose tour size lies outside [2, 2n-1] or
// that holds a node id outside [0, n) deposits nothing, and its elites_out entry
// reads ACO_ERR_INVALID instead of the ant id.
#include <cuda_runtime.h>

#include <atomic>

#include "../../include/cvrp_aco.h"
#include "aco_device.cuh"

namespace aco {
namespace {

constexpr int kMaxNodes = 4096;
constexpr int kMaxRanks = 8;
constexpr int kThreads = 1024;
constexpr int kLens = 2048;  // lengths kept in shared memory (more are read again in every round)
constexpr int kRowsMax = 32; // rows of a CTA
constexpr int kU = 4;        // columns of a lane in a chunk of 32 kU

__device__ __forceinline__ unsigned long long block_min_key(unsigned long long v, unsigned long long *red)
{
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w < v ? w : v;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[threadIdx.x & 31];
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w < v ? w : v;
    }
    return v;
}

// Rows [blockIdx.x * rows, + rows).  eta^beta is recomputed from the distance
// (kernel.cl:782-789).
template <bool PLAIN>
__global__ void __launch_bounds__(kThreads) noalloc_update_kernel(int n, int ld, int n_ants, int R, int rows, float evap,
                                                                  float alpha, int alpha_int, float beta, int beta_int,
                                                                  float *tau, float *total, const float *dist,
                                                                  const int *solutions, const float *lens,
                                                                  int *elites_out)
{
    static_assert(kThreads == 1024, "block_min_key reads 32 warps' minima");
    __shared__ unsigned long long red[32];
    __shared__ float s_len[kLens], s_amt[kMaxRanks];
    __shared__ int s_elite[kMaxRanks], s_size[kMaxRanks], s_bad[kMaxRanks];
    __shared__ int s_succ[kMaxRanks][kRowsMax]; // successor of the CTA's customers in elite r's tour, -1 if none
    __shared__ uint32_t s_dep[kMaxNodes];       // row 0's CTA: bit r, elite r's tour goes depot -> column
    const int A = n_ants, T = 2 * n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = blockIdx.x * rows, i1 = min(n, i0 + rows);
    // chunks of 32 kU columns over the CTA's rows; the warp's first is loaded ahead
    const int per_row = (n + 32 * kU - 1) / (32 * kU), chunks = (i1 - i0) * per_row;
    float t[kU], d[kU];
    auto load = [&](int c) {
        const int i = i0 + c / per_row, j0 = (c % per_row) * 32 * kU + lane;
#pragma unroll
        for (int u = 0; u < kU; u++) {
            const int j = j0 + 32 * u;
            t[u] = j < n ? tau[(size_t)i * ld + j] : 0.f;
            d[u] = j < n ? dist[(size_t)i * ld + j] : 0.f;
        }
    };
    if (warp < chunks) load(warp);

    // elites (kernel.cl:717-741): the best-so-far slot, then rounds of "first
    // minimum, knocked out to +inf"
    const float inf = __int_as_float(0x7f800000);
    for (int k = tid; k < A && k < kLens; k += kThreads) s_len[k] = lens[k];
    for (int e = tid; e < kMaxRanks * kRowsMax; e += kThreads) s_succ[0][e] = -1;
    if (i0 == 0)
        for (int j = tid; j < n; j += kThreads) s_dep[j] = 0u;
    if (tid < kMaxRanks) s_bad[tid] = 0;
    if (tid == 0) s_elite[0] = A;
    __syncthreads();
    if (A <= kLens) { // one warp runs the rounds, without block barriers
        if (warp == 0) {
            for (int r = 1; r < R; r++) {
                // a lane without ants has no index; one whose lengths all have the largest bits
                // (a buffer cleared to 0xff) has its first
                uint32_t lo = 0xffffffffu, at = lane < A ? (uint32_t)lane : 0xffffffffu;
                for (int k = lane; k < A; k += 32) {
                    const uint32_t b = __float_as_uint(s_len[k]);
                    at = b < lo ? (uint32_t)k : at;
                    lo = b < lo ? b : lo;
                }
                const uint32_t least = __reduce_min_sync(0xffffffffu, lo);
                const int target = (int)__reduce_min_sync(0xffffffffu, lo == least ? at : 0xffffffffu);
                if (lane == 0) {
                    s_elite[r] = target;
                    s_len[target] = inf;
                }
                __syncwarp();
            }
        }
        __syncthreads();
    } else {
        for (int r = 1; r < R; r++) {
            unsigned long long m = ~0ull;
            for (int k = tid; k < A; k += kThreads) {
                float v = k < kLens ? s_len[k] : lens[k];
                if (k >= kLens)
                    for (int q = 1; q < r; q++) v = s_elite[q] == k ? inf : v;
                const unsigned long long key = ((unsigned long long)__float_as_uint(v) << 32) | (unsigned)k;
                m = key < m ? key : m;
            }
            m = block_min_key(m, red);
            if (tid == 0) {
                const int target = (int)(m & 0xffffffffu);
                s_elite[r] = target;
                if (target < kLens) s_len[target] = inf;
            }
            __syncthreads();
        }
    }
    if (tid < R) {
        const int e = s_elite[tid], size = solutions[(size_t)T * e + T - 1];
        const bool bad = size < 2 || size > T - 1;
        s_size[tid] = bad ? 0 : size;
        s_bad[tid] = bad ? 1 : 0;
        s_amt[tid] = __fdiv_rn((float)(R - tid), lens[e]);
    }
    __syncthreads();
    // every node of the elite tours checked, the edges that leave this CTA's rows
    // kept: the warps are dealt out over the elites, four nodes a lane in flight
    {
        const int per = kThreads / 32 / R, r = warp / per; // warps of an elite (at least 4)
        const int size = r < R ? s_size[r] : 0, step = per * 32;
        const int *tour = solutions + (size_t)T * (r < R ? s_elite[r] : A);
        for (int k0 = (warp - r * per) * 32 + lane; k0 < size; k0 += 4 * step) {
            int uu[4], vv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int k = k0 + q * step;
                uu[q] = k < size ? __ldg(tour + k) : 0;
                vv[q] = k + 1 < size ? __ldg(tour + k + 1) : -1;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if ((unsigned)uu[q] >= (unsigned)n) s_bad[r] = 1;
                if (uu[q] < i0 || uu[q] >= i1 || (unsigned)vv[q] >= (unsigned)n) continue;
                if (uu[q] == 0) atomicOr(&s_dep[vv[q]], 1u << r);
                else s_succ[r][uu[q] - i0] = vv[q];
            }
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && tid < R && elites_out) elites_out[tid] = s_bad[tid] ? ACO_ERR_INVALID : s_elite[tid];
    uint32_t good = 0u;
    for (int r = 0; r < R; r++) good |= (s_bad[r] ? 0u : 1u) << r;

    // evaporation + deposit (elite order) + total_info
    for (int c = warp; c < chunks; c += kThreads / 32) {
        if (c != warp) load(c);
        const int i = i0 + c / per_row, j0 = (c % per_row) * 32 * kU + lane;
        const size_t off = (size_t)i * ld;
        float v[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) v[u] = __fmul_rn(evap, t[u]);
        if (i != 0) {
            for (int r = 0; r < R; r++) {
                const unsigned at = (unsigned)(s_succ[r][i - i0] - (j0 - lane)); // place in the chunk
                if (at >= 32u * kU || !((good >> r) & 1u)) continue;             // warp-uniform
                if ((at & 31u) == (unsigned)lane) {
                    const float amt = s_amt[r];
#pragma unroll
                    for (int u = 0; u < kU; u++) v[u] = (at >> 5) == (unsigned)u ? __fadd_rn(v[u], amt) : v[u];
                }
            }
        } else {
#pragma unroll
            for (int u = 0; u < kU; u++)
                for (uint32_t m = j0 + 32 * u < n ? s_dep[j0 + 32 * u] & good : 0u; m; m &= m - 1u)
                    v[u] = __fadd_rn(v[u], s_amt[__ffs(m) - 1]);
        }
#pragma unroll
        for (int u = 0; u < kU; u++) {
            const int j = j0 + 32 * u;
            if (j >= n) continue;
            const float eta = __fdiv_rn(1.0f, __fadd_rn(d[u], 0.1f));
            tau[off + j] = v[u];
            // the defaults alpha 1, beta 2 without pow_rule's loops (the same products)
            total[off + j] = PLAIN ? __fmul_rn(v[u], __fmul_rn(eta, eta))
                                   : __fmul_rn(pow_rule(v[u], alpha, alpha_int), pow_rule(eta, beta, beta_int));
        }
    }
}

int exp_int(float e)
{
    if (e >= 0.0f && e <= 8.0f && e == (float)(int)e) return (int)e;
    return -1;
}

// Multiprocessors of the current device, asked once per device.
int multiprocessors()
{
    static std::atomic<int> known[64];
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    v = known[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        known[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

} // namespace
} // namespace aco

extern "C" int aco_pheromone_update_noalloc(int n, int ld, int n_ants, int ras_ranks, float rho, float alpha,
                                            float beta, float *tau, float *total_info, const float *dist,
                                            const int *solutions, const float *lens, int *elites_out, void *stream)
{
    using namespace aco;
    if (n < 2 || ld < n || n_ants < 1 || ras_ranks < 1 || !tau || !total_info || !dist || !solutions || !lens)
        return ACO_ERR_INVALID;
    if (!(rho > 0.0f && rho <= 1.0f)) return ACO_ERR_INVALID;
    if (n > kMaxNodes || ras_ranks > kMaxRanks) return ACO_ERR_CAPACITY; // beyond a CTA's shared memory
    const int sm = multiprocessors();
    if (sm < 1) return ACO_ERR_CUDA;
    int rows = (n + sm - 1) / sm; // one CTA an SM
    if (rows > kRowsMax) rows = kRowsMax;
    const int ai = exp_int(alpha), bi = exp_int(beta);
    auto kern = ai == 1 && bi == 2 ? noalloc_update_kernel<true> : noalloc_update_kernel<false>;
    kern<<<(n + rows - 1) / rows, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        n, ld, n_ants, ras_ranks, rows, 1.0f - rho, alpha, ai, beta, bi, tau, total_info, dist, solutions, lens,
        elites_out);
    if (cudaGetLastError() != cudaSuccess) return ACO_ERR_CUDA;
    return ACO_OK;
}
