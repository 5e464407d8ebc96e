// two_opt.cuh -- the register path of the route 2-opt (first improvement in
// sequence order with don't-look bits, kernel.cl:126-277) for routes of at most
// 32 nodes, shared by the 2-opt kernels and the construct kernel that improves
// routes while later ones are still being built.
//
// Lane p holds everything about route position p: the local node there (tq), its
// neighbours on the tour, the length of the edge leaving it (dq, dist_tour_wrk)
// and the mask of the route nodes on its neighbour list.  An examination takes
// the examined position's words by shuffle, and every lane evaluates its own
// node as the move partner from its own registers and three entries of `tile`,
// the route's 32x32 distance sub-matrix.
//
// The lists are sorted by distance, so the reference's scan (stop at the first
// entry past the radius or improving) finds a move exactly when some listed
// route node inside the radius improves, and takes the nearest of them; equal
// distances are settled by the list itself.  No list is read otherwise: a node
// is listed exactly when it is no farther than the list's last entry, whose
// distance is kept per node (nnr), except where the list ends inside a group of
// equal distances (flagged there, looked up).  Instances with distances that
// are not finite do not come here.
//
// Warp instructions: about 45 an examination and 45 a move (90 and 75 with the
// lists filtered into shared memory and the partner's words fetched by shuffle),
// 10 a row to build the tile (60 with the list filtering); routes of at most 16
// nodes take two examinations and two rows at a time.  The issue slots bound it.
// 512 instances, 2.9 M routes of 14 nodes: 9.81 ms with the lists in shared memory,
// 6.58 by position, 5.78 with the pairs; 201 ants with full lists: 74 -> 27 us.
#pragma once

#include <cstdint>

#include "aco_device.cuh"

namespace aco {
namespace {

constexpr int kRL = kRegRoute; // largest route (nodes, depot included) of the register path

constexpr unsigned kFullMask = 0xffffffffu;

// The distance tile of a route and, as the return value of lane k, the mask of
// the route's customers on the neighbour list of route node k (its own bit and
// the depot's are never set).  Lane q < R holds route node q's global id (v); a
// round's loads are in flight together.  PAIR (R <= 16, lanes 16-31 repeat lanes
// 0-15): each half of the warp takes a row, the tile's rows are 16 entries.
template <int ROWS, bool PAIR>
__device__ __forceinline__ uint32_t route_tile(int lane, int R, int v, const float *dist, int ld, const float2 *nnr,
                                               const int *nn, int nn_ls, float *tile)
{
    constexpr int W = PAIR ? 16 : kRL, PER = PAIR ? 2 : 1; // row length, rows a load takes
    const int l = PAIR ? lane & 15 : lane, h = PAIR ? lane >> 4 : 0;
    const uint32_t cust = (R >= 32 ? kFullMask : (1u << R) - 1u) & ~1u;
    float2 last = make_float2(-__int_as_float(0x7f800000), 0.f); // the list's last distance; 1: others share it
    if (lane < R && nn_ls > 0) last = __ldg(nnr + v);
    uint32_t nm = 0u;
    for (int k0 = 0; k0 < R; k0 += PER * ROWS) {
        float d[ROWS];
#pragma unroll
        for (int u = 0; u < ROWS; u++) {
            const int k = k0 + PER * u + h;
            const int node1 = __shfl_sync(kFullMask, v, k & (W - 1));
            d[u] = (k < R && l < R) ? __ldg(dist + (size_t)node1 * ld + v) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < ROWS; u++) {
            const int k1 = k0 + PER * u;
            if (k1 >= R) break; // warp-uniform
            tile[k1 * W + lane] = d[u];
            const uint32_t m =
                __ballot_sync(kFullMask, d[u] <= __shfl_sync(kFullMask, last.x, (k1 + h) & (W - 1)));
            if (l / PER == k1 / PER) nm = (PAIR && (l & 1) ? m >> 16 : m) & cust & ~(1u << l);
        }
    }
    // lists that end inside a group of equal distances: look those route nodes up
    for (uint32_t amb = __ballot_sync(kFullMask, lane < R && last.y != 0.f); amb; amb &= amb - 1u) {
        const int k1 = __ffs(amb) - 1;
        const float thr = __shfl_sync(kFullMask, last.x, k1);
        const int *list = nn + (size_t)__shfl_sync(kFullMask, v, k1) * nn_ls;
        for (uint32_t at = __ballot_sync(kFullMask, tile[k1 * W + l] == thr) & cust & ~(1u << k1); at; at &= at - 1u) {
            const int b = __ffs(at) - 1, node = __shfl_sync(kFullMask, v, b);
            bool hit = false;
            for (int h1 = lane; h1 < nn_ls; h1 += 32) hit = hit || __ldg(list + h1) == node;
            if (!__any_sync(kFullMask, hit) && l == k1) nm &= ~(1u << b);
        }
    }
    __syncwarp();
    return nm;
}

// The lane of `mv` (improving partners) the scan reaches first: the smallest
// distance, equal ones in list order.  gnode: the lane's global node.
__device__ __forceinline__ int first_listed(uint32_t mv, int lane, float d12, int gnode, const int *list, int nn_ls)
{
    const uint32_t b = __float_as_uint(__fadd_rn(d12, 0.f)); // -0 as +0
    const uint32_t ord = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    const bool in = (mv >> lane) & 1u;
    const uint32_t lo = __reduce_min_sync(kFullMask, in ? ord : 0xffffffffu);
    const uint32_t tied = __ballot_sync(kFullMask, in && ord == lo);
    if (tied & (tied - 1u))
        for (int h = 0; h < nn_ls; h++) {
            const uint32_t m = __ballot_sync(kFullMask, ((tied >> lane) & 1u) && __ldg(list + h) == gnode);
            if (m) return __ffs(m) - 1;
        }
    return __ffs(tied) - 1;
}

// ---------------------------------------------------------------------------
// Register path: routes of at most 32 nodes.  tq, dq: on entry lane p's local
// node p and edge length, on return the improved route's; nm: lane k's mask
// (route_tile); v: lane k's global node.  SYM: the distances are symmetric, so
// an edge's length is its dist_tour_wrk entry (otherwise the tile's).
// PAIR (R <= 16, lanes 16-31 hold copies of lanes 0-15): lanes 16-31 examine the
// position after the one that lanes 0-15 examine.  An examination that finds no
// move changes nothing but its own don't-look bit, so the second one stands when
// the first finds none, and is dropped otherwise.
// ---------------------------------------------------------------------------
template <bool SYM, bool PAIR>
__device__ int two_opt_route_regs(int lane, int R, bool first_route, const float *tile, uint32_t nm, int v,
                                  const int *nn, int nn_ls, int &tq, float &dq, int pass_limit)
{
    constexpr int W = PAIR ? 16 : kRL;
    constexpr uint32_t ROW = PAIR ? 0xffffu : kFullMask; // a half's lanes in a ballot
    const int l = PAIR ? lane & 15 : lane;
    // `open`: bit p set while the don't-look bit of position p's node is clear; a
    // move carries it along with the positions it reverses
    uint32_t open = (R >= 32 ? kFullMask : (1u << R) - 1u) & ~(first_route ? 0u : 1u);
    if (!open) return ACO_OK;
    const int pn = l + 1 < R ? l + 1 : 0, pp = l > 0 ? l - 1 : R - 1; // next and previous position
    int ts, tp;   // the local nodes there
    float dqp;    // dist_tour_wrk of the previous position
    uint32_t word; // tq | ts << 8 | tp << 16
    auto neighbours = [&]() {
        ts = __shfl_sync(kFullMask, tq, pn);
        tp = __shfl_sync(kFullMask, tq, pp);
        dqp = __shfl_sync(kFullMask, dq, pp);
        word = (uint32_t)tq | ((uint32_t)ts << 8) | ((uint32_t)tp << 16);
    };
    neighbours();
    int passes = 1;
    bool imp = false;
    int q1 = __ffs(open) - 1;
    for (;;) {
        uint32_t next = open & (0xfffffffeu << q1); // open positions left in this pass
        const int q2 = PAIR && next ? __ffs(next) - 1 : q1;
        const int q = PAIR && lane >= 16 ? q2 : q1;
        const uint32_t w1 = __shfl_sync(kFullMask, word, q), m1 = __shfl_sync(kFullMask, nm, q);
        const int k1 = w1 & 0xff, ks1 = (w1 >> 8) & 0xff, kp1 = w1 >> 16;
        const float d12 = tile[k1 * W + tq], xs = tile[ks1 * W + ts], xp = tile[kp1 * W + tp];
        // radii: the examined node's two tour edges
        const float rs = SYM ? __shfl_sync(kFullMask, dq, q) : tile[k1 * W + ks1];
        const float rp = SYM ? __shfl_sync(kFullMask, dqp, q) : tile[kp1 * W + k1];
        const bool act = (m1 >> tq) & 1u;
        // successor and predecessor searches (kernel.cl:180-198, 202-230); -r + d is -(r - d)
        const float us = __fsub_rn(rs, d12), up = __fsub_rn(rp, d12);
        const float gs = __fsub_rn(__fsub_rn(xs, us), dq), gp = __fsub_rn(__fsub_rn(xp, up), dqp);
        const uint32_t smove = __ballot_sync(kFullMask, act & (us > kEps) & (gs < -kEps));
        const uint32_t pmove =
            __ballot_sync(kFullMask, act & (up > kEps) & (tp != k1) & (tq != kp1) & (gp < -kEps));
        if ((smove | pmove) == 0u) {
            open &= ~((1u << q1) | (1u << q2)); // kernel.cl:232
            if (PAIR) next &= next - 1u;        // q2 is done as well
        } else { // the predecessor's result counts only when the successor search finds no move
            imp = true;
            int at = 0; // the first lane of the examination that moves
            if (PAIR && ((smove | pmove) & ROW) == 0u) {
                at = 16;
                open &= ~(1u << q1);
                q1 = q2;
            }
            const uint32_t sm = (smove >> at) & ROW;
            const uint32_t mv = sm ? sm : (pmove >> at) & ROW;
            int f = __ffs(mv) - 1;
            if (mv & (mv - 1u))
                f = first_listed(mv << at, lane, d12, __shfl_sync(kFullMask, v, tq),
                                 nn + (size_t)__shfl_sync(kFullMask, v, __shfl_sync(kFullMask, k1, at)) * nn_ls,
                                 nn_ls) & (W - 1);
            // exchange (kernel.cl:235-270): the edges leaving positions i < j make way for
            // (i, j) and (i + 1, j + 1); positions i + 1 .. j are reversed
            const int pa = sm ? q1 : (q1 > 0 ? q1 - 1 : R - 1), pb = sm ? f : f - 1;
            const int i = min(pa, pb), j = max(pa, pb), jn = j + 1 < R ? j + 1 : 0;
            const uint32_t wi = __shfl_sync(kFullMask, word, i), wj = __shfl_sync(kFullMask, word, j);
            const float d13 = tile[(wi & 0xff) * W + (wj & 0xff)];
            const float d24 = tile[((wi >> 8) & 0xff) * W + ((wj >> 8) & 0xff)];
            const bool in = l > i && l <= j;
            const int src = in ? i + 1 + j - l : l;
            tq = __shfl_sync(kFullMask, tq, src);
            nm = __shfl_sync(kFullMask, nm, src);
            const float dr = __shfl_sync(kFullMask, dq, in && l < j ? i + j - l : l);
            dq = l == j ? d24 : l == i ? d13 : dr;
            open = (__ballot_sync(kFullMask, (open >> src) & 1u) & ROW) | (1u << i) | (2u << i) | (1u << j) | (1u << jn);
            neighbours();
            next = open & (0xfffffffeu << q1);
        }
        if (next == 0u) { // end of the pass
            if (!imp || open == 0u) break;
            if (pass_limit > 0 && passes >= pass_limit) return ACO_ERR_LS_LIMIT;
            passes++;
            imp = false;
            next = open;
        }
        q1 = __ffs(next) - 1;
    }
    return ACO_OK;
}

// ---------------------------------------------------------------------------
// Best improvement (a non-parity option: the reference improves first in scan
// order): every 2-opt move of the route -- reverse positions i+1..j, 0 <= i <
// j <= R-1, the position after R-1 being the depot at 0 -- is evaluated at once
// from the route's distance tile, lane j taking the pairs (i, j) of one i at a
// time; a warp argmin picks the most negative change of the tour length (ties:
// the lowest (i, j)), which is applied while it is below -EPSILON.  tpos: 32
// bytes of the warp's shared memory for the local node at every position.  At
// most move_limit moves (then ACO_ERR_LS_LIMIT).
// ---------------------------------------------------------------------------
__device__ int two_opt_route_best(int lane, int R, const float *tile, uint8_t *tpos, int &tq, float &dq, int move_limit)
{
    const unsigned FULLM = 0xffffffffu;
    for (int moves = 0;; moves++) {
        if (lane < R) tpos[lane] = (uint8_t)tq;
        __syncwarp();
        unsigned long long best = ~0ull;
        const int j = lane, tj = lane < R ? tpos[lane] : 0, tj1 = lane + 1 < R ? tpos[lane + 1] : tpos[0];
        for (int i = 0; i + 1 < R; i++) {
            if (j > i && j < R) {
                const int ti = tpos[i], ti1 = tpos[i + 1];
                const float add = __fadd_rn(tile[ti * kRL + tj], tile[ti1 * kRL + tj1]);
                const float rem = __fadd_rn(tile[ti * kRL + ti1], tile[tj * kRL + tj1]);
                const uint32_t b = __float_as_uint(__fsub_rn(add, rem));
                const uint32_t ord = (b & 0x80000000u) ? ~b : (b | 0x80000000u); // ascending as the floats
                const unsigned long long key = ((unsigned long long)ord << 32) | (unsigned)(i << 8 | j);
                best = key < best ? key : best;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long w = __shfl_xor_sync(FULLM, best, o);
            best = w < best ? w : best;
        }
        __syncwarp();
        if (best == ~0ull) break;
        const uint32_t ord = (uint32_t)(best >> 32);
        const uint32_t b = (ord & 0x80000000u) ? (ord & 0x7fffffffu) : ~ord;
        if (!(__uint_as_float(b) < -kEps)) break;
        if (move_limit > 0 && moves >= move_limit) return ACO_ERR_LS_LIMIT;
        const int i = (int)((best >> 8) & 0xffu), jj = (int)(best & 0xffu);
        // the exchange of the first-improvement path with h1..h4 = the nodes at i, i+1, jj, jj+1
        const int h1 = tpos[i], h2 = tpos[i + 1], h3 = tpos[jj], h4 = jj + 1 < R ? tpos[jj + 1] : tpos[0];
        const int a = i + 1;
        const float d13 = tile[h1 * kRL + h3], d24 = tile[h2 * kRL + h4];
        const float dsrc = __shfl_sync(FULLM, dq, (lane > i && lane < jj) ? i + jj - lane : lane);
        if (lane == jj) dq = d24;
        else if (lane == i) dq = d13;
        else if (lane > i && lane < jj) dq = dsrc;
        const int tsrc = __shfl_sync(FULLM, tq, (lane >= a && lane <= jj) ? a + jj - lane : lane);
        if (lane >= a && lane <= jj) tq = tsrc;
    }
    return ACO_OK;
}

// ---------------------------------------------------------------------------
// Routes of 33 to 64 nodes: as two_opt_route_regs with two positions a lane
// (p and p + 32).  Their tile would not fit the warp's share of shared memory,
// so the three distances of a partner come from the matrix, loaded together: one
// trip to the cache an examination, where the list-scanning path waits for its
// list entry, its distance and its neighbour's distance in turn.  1001 nodes, 256
// ants, 2% of the routes of 33-48 nodes: 2-opt 160 -> 113 us with these taken first.
// nodes: the route's nodes in sequence, on return the improved ones; dist_tour:
// on return its edge lengths.
// ---------------------------------------------------------------------------
constexpr int kRW = 64; // largest route of this path

__device__ __forceinline__ int two_opt_route_wide(int lane, int R, bool first_route, bool sym, uint16_t *nodes,
                                               float *dist_tour, const float *dist, int ld, const float2 *nnr,
                                               const int *nn, int nn_ls, int pass_limit)
{
    auto D = [&](int a, int b) { return __ldg(dist + (size_t)a * ld + b); };
    // position q of an array held two a lane: q per lane, and q the same in all lanes
    auto any = [&](auto x0, auto x1, int q) {
        const auto y0 = __shfl_sync(kFullMask, x0, q & 31), y1 = __shfl_sync(kFullMask, x1, q & 31);
        return q & 32 ? y1 : y0;
    };
    auto one = [&](auto x0, auto x1, int q) { return __shfl_sync(kFullMask, q & 32 ? x1 : x0, q & 31); };

    int id[2], g[2], gs[2], gp[2], pn[2], pp[2]; // local id (entry position), node, its neighbours; their positions
    float dq[2], dqp[2];
    uint32_t lo[2] = {0u, 0u}, hi[2] = {0u, 0u}; // the route's customers on the node's list, by local id
    float2 last[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int p = lane + 32 * u;
        id[u] = p < R ? p : 0;
        g[u] = p < R ? (int)nodes[p] : 0;
        pn[u] = p + 1 < R ? p + 1 : 0;
        pp[u] = p == 0 ? R - 1 : p - 1;
        last[u] = make_float2(-__int_as_float(0x7f800000), 0.f);
        if (p < R && nn_ls > 0) last[u] = __ldg(nnr + g[u]);
    }
    const bool has1 = lane + 32 < R; // position lane < R always
#pragma unroll
    for (int u = 0; u < 2; u++)
        for (int k0 = 32 * u; k0 < min(R, 32 * u + 32); k0 += 4) {
            float d0[4], d1[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int node1 = __shfl_sync(kFullMask, g[u], (k0 + c) & 31);
                d0[c] = k0 + c < R ? D(node1, g[0]) : 0.f;
                d1[c] = k0 + c < R && has1 ? D(node1, g[1]) : 0.f;
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float thr = __shfl_sync(kFullMask, last[u].x, (k0 + c) & 31);
                const uint32_t b0 = __ballot_sync(kFullMask, d0[c] <= thr);
                const uint32_t b1 = __ballot_sync(kFullMask, has1 && d1[c] <= thr);
                if (lane == ((k0 + c) & 31)) {
                    lo[u] = b0 & ~1u & ~(u == 0 ? 1u << lane : 0u);
                    hi[u] = b1 & ~(u == 1 ? 1u << lane : 0u);
                }
            }
        }
    // lists that end inside a group of equal distances (see route_tile)
#pragma unroll
    for (int u = 0; u < 2; u++)
        for (uint32_t amb = __ballot_sync(kFullMask, lane + 32 * u < R && last[u].y != 0.f); amb; amb &= amb - 1u) {
            const int k1 = __ffs(amb) - 1, node1 = __shfl_sync(kFullMask, g[u], k1);
            const float thr = __shfl_sync(kFullMask, last[u].x, k1);
            const int *list = nn + (size_t)node1 * nn_ls;
#pragma unroll
            for (int w = 0; w < 2; w++) {
                const bool in = w == 0 ? lane > 0 : has1;
                for (uint32_t at = __ballot_sync(kFullMask, in && D(node1, g[w]) == thr) & ~(u == w ? 1u << k1 : 0u); at;
                     at &= at - 1u) {
                    const int b = __ffs(at) - 1, node = __shfl_sync(kFullMask, g[w], b);
                    bool hit = false;
                    for (int h = lane; h < nn_ls; h += 32) hit = hit || __ldg(list + h) == node;
                    if (!__any_sync(kFullMask, hit) && lane == k1) (w == 0 ? lo[u] : hi[u]) &= ~(1u << b);
                }
            }
        }
    auto neighbours = [&]() {
#pragma unroll
        for (int u = 0; u < 2; u++) {
            gs[u] = any(g[0], g[1], pn[u]);
            gp[u] = any(g[0], g[1], pp[u]);
            dqp[u] = any(dq[0], dq[1], pp[u]);
        }
    };
    dq[0] = dq[1] = 0.f;
    neighbours();
    dq[0] = D(g[0], gs[0]);
    dq[1] = has1 ? D(g[1], gs[1]) : 0.f;
    neighbours();

    unsigned long long open = (R >= 64 ? ~0ull : (1ull << R) - 1ull) & ~(first_route ? 0ull : 1ull);
    int passes = 1, q1 = __ffsll((long long)open) - 1, status = ACO_OK;
    bool imp = false;
    for (;;) {
        const int g1 = one(g[0], g[1], q1), gs1 = one(gs[0], gs[1], q1), gp1 = one(gp[0], gp[1], q1);
        const uint32_t mlo = one(lo[0], lo[1], q1), mhi = one(hi[0], hi[1], q1);
        const float rs = sym ? one(dq[0], dq[1], q1) : D(g1, gs1), rp = sym ? one(dqp[0], dqp[1], q1) : D(gp1, g1);
        float d12[2], xs[2], xp[2];
        bool act[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            act[u] = ((id[u] & 32 ? mhi : mlo) >> (id[u] & 31)) & 1u;
            d12[u] = act[u] ? D(g1, g[u]) : 0.f;
            xs[u] = act[u] ? D(gs1, gs[u]) : 0.f;
            xp[u] = act[u] ? D(gp1, gp[u]) : 0.f;
        }
        uint32_t sm[2], pm[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const float us = __fsub_rn(rs, d12[u]), up = __fsub_rn(rp, d12[u]);
            const float gsu = __fsub_rn(__fsub_rn(xs[u], us), dq[u]), gpu = __fsub_rn(__fsub_rn(xp[u], up), dqp[u]);
            sm[u] = __ballot_sync(kFullMask, act[u] & (us > kEps) & (gsu < -kEps));
            pm[u] = __ballot_sync(kFullMask, act[u] & (up > kEps) & (gp[u] != g1) & (g[u] != gp1) & (gpu < -kEps));
        }
        if ((sm[0] | sm[1] | pm[0] | pm[1]) == 0u) {
            open &= ~(1ull << q1);
        } else {
            imp = true;
            const bool succ = (sm[0] | sm[1]) != 0u;
            const uint32_t m0 = succ ? sm[0] : pm[0], m1 = succ ? sm[1] : pm[1];
            int f = m0 ? __ffs(m0) - 1 : __ffs(m1) + 31;
            if (__popc(m0) + __popc(m1) > 1) { // the nearest, equal ones in list order
                uint32_t ord[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const uint32_t b = __float_as_uint(__fadd_rn(d12[u], 0.f)); // -0 as +0
                    ord[u] = ((u == 0 ? m0 : m1) >> lane) & 1u ? ((b & 0x80000000u) ? ~b : (b | 0x80000000u)) : 0xffffffffu;
                }
                const uint32_t near = __reduce_min_sync(kFullMask, min(ord[0], ord[1]));
                const uint32_t t0 = __ballot_sync(kFullMask, ((m0 >> lane) & 1u) && ord[0] == near);
                const uint32_t t1 = __ballot_sync(kFullMask, ((m1 >> lane) & 1u) && ord[1] == near);
                f = t0 ? __ffs(t0) - 1 : __ffs(t1) + 31;
                if (__popc(t0) + __popc(t1) > 1) {
                    const int *list = nn + (size_t)g1 * nn_ls;
                    for (int h = 0; h < nn_ls; h++) {
                        const int node = __ldg(list + h);
                        const uint32_t e0 = __ballot_sync(kFullMask, ((t0 >> lane) & 1u) && g[0] == node);
                        const uint32_t e1 = __ballot_sync(kFullMask, ((t1 >> lane) & 1u) && g[1] == node);
                        if (e0 | e1) {
                            f = e0 ? __ffs(e0) - 1 : __ffs(e1) + 31;
                            break;
                        }
                    }
                }
            }
            const int pa = succ ? q1 : (q1 > 0 ? q1 - 1 : R - 1), pb = succ ? f : f - 1;
            const int i = min(pa, pb), j = max(pa, pb), jn = j + 1 < R ? j + 1 : 0;
            const float d13 = D(one(g[0], g[1], i), one(g[0], g[1], j));
            const float d24 = D(one(gs[0], gs[1], i), one(gs[0], gs[1], j));
            int nid[2], ng[2];
            uint32_t nlo[2], nhi[2], nop[2];
            float nd[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int p = lane + 32 * u;
                const bool in = p > i && p <= j;
                const int src = in ? i + 1 + j - p : p, dsrc = in && p < j ? i + j - p : p;
                nid[u] = any(id[0], id[1], src);
                ng[u] = any(g[0], g[1], src);
                nlo[u] = any(lo[0], lo[1], src);
                nhi[u] = any(hi[0], hi[1], src);
                nd[u] = any(dq[0], dq[1], dsrc);
                nd[u] = p == j ? d24 : p == i ? d13 : nd[u];
                nop[u] = __ballot_sync(kFullMask, (open >> src) & 1ull);
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                id[u] = nid[u];
                g[u] = ng[u];
                lo[u] = nlo[u];
                hi[u] = nhi[u];
                dq[u] = nd[u];
            }
            open = nop[0] | (unsigned long long)nop[1] << 32 | 1ull << i | 2ull << i | 1ull << j | 1ull << jn;
            neighbours();
        }
        unsigned long long next = open & (~1ull << q1); // open positions left in this pass
        if (next == 0ull) {
            if (!imp) break;
            if (pass_limit > 0 && passes >= pass_limit) {
                status = ACO_ERR_LS_LIMIT;
                break;
            }
            passes++;
            imp = false;
            if (open == 0ull) break;
            next = open;
        }
        q1 = __ffsll((long long)next) - 1;
    }
    nodes[lane] = (uint16_t)g[0];
    dist_tour[lane] = dq[0];
    if (has1) {
        nodes[lane + 32] = (uint16_t)g[1];
        dist_tour[lane + 32] = dq[1];
    }
    __syncwarp();
    return status;
}

// A route of at most 32 nodes: lane q < R brings route node q's global id (v) and
// takes back the local node at position q and the edge length there.
template <int ROWS>
__device__ __forceinline__ int two_opt_route(int lane, int R, bool first_route, bool best, bool sym, int v,
                                             const float *dist, int ld, const float2 *nnr, const int *nn, int nn_ls,
                                             float *tile, uint8_t *tpos, int &tq, float &dq, int pass_limit)
{
    const int l = R <= 16 && !best ? lane & 15 : lane;
    tq = l < R ? l : 0;
    // edge lengths: position q -> q+1, the last one back to the next depot (node 0 = local 0)
    const int to = l + 1 < R ? l + 1 : 0;
    if (R <= 16 && !best) {
        v = __shfl_sync(kFullMask, v, l);
        const uint32_t nm = route_tile<ROWS, true>(lane, R, v, dist, ld, nnr, nn, nn_ls, tile);
        dq = l < R ? tile[l * 16 + to] : 0.f;
        return sym ? two_opt_route_regs<true, true>(lane, R, first_route, tile, nm, v, nn, nn_ls, tq, dq, pass_limit)
                   : two_opt_route_regs<false, true>(lane, R, first_route, tile, nm, v, nn, nn_ls, tq, dq, pass_limit);
    }
    const uint32_t nm = route_tile<ROWS, false>(lane, R, v, dist, ld, nnr, nn, nn_ls, tile);
    dq = l < R ? tile[l * kRL + to] : 0.f;
    if (best) return two_opt_route_best(lane, R, tile, tpos, tq, dq, pass_limit);
    return sym ? two_opt_route_regs<true, false>(lane, R, first_route, tile, nm, v, nn, nn_ls, tq, dq, pass_limit)
               : two_opt_route_regs<false, false>(lane, R, first_route, tile, nm, v, nn, nn_ls, tq, dq, pass_limit);
}

} // namespace
} // namespace aco
