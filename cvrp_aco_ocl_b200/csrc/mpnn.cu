// mpnn.cu -- the edge-scoring message-passing network of the learned prior:
// forward, backward and the Adam step, with every dense product on the
// tcgen05 tensor cores (BF16 operands, FP32 accumulation in tensor memory).
//
// Graph: node i has k out-edges, rows i*k .. i*k+k-1 of every edge array, to
// its k nearest customers (nbr).  Hidden width 64.  Per layer (the oracle in
// oracle/mpnn_oracle.py states the same equations in FP64):
//   P  = h W^T + b              node GEMM, N = 256 (U | V | B | C)
//   q  = e A^T + a + B_i + C_j  edge GEMM + gathers
//   e' = e + relu(q);  g = sigmoid(e')
//   u  = U + (1/k) sum_j g V_j;  h' = h + relu(u)
// Head: z = relu(e W_h^T + b_h), logit s = z . w_o + b_o; weighted BCE loss.
//
// Common shape of the kernels: 256 threads work on a tile of up to 128 rows of
// 64 channels.  Half-warp w (16 lanes, four channels a lane) owns rows 8w..8w+7,
// so every global access is a whole 256-byte row.  BF16 operand tiles use the
// 128-byte swizzle of umma.cuh, in which one staged copy serves as the
// K-major operand of one product and the transposed (MN-major) operand of
// another: no operand is staged twice.  The accumulator goes through a shared
// FP32 tile (row stride 68) that takes the place of the operand tiles once the
// product is done, which keeps a CTA at 44 KB and three CTAs on an SM.
// Edge tiles hold whole nodes, so the per-node sums need no atomics: a node's dB
// is the sum of its k rows in edge order.  Sums over a node's in-edges (dV, dC)
// are 16-byte vector reductions; weight gradients accumulate in tensor memory
// over the tiles of a persistent CTA, bias gradients row by row in registers,
// and are added to the gradient buffer once per CTA.  Layer 0 makes its edge
// embedding from the edge feature on the fly (it is never stored).  The backward
// keeps the sign of q as one nibble a lane (16 bytes a row) in place of q itself.
//
// Order of the sums.  The biases and embeddings enter the network in FP32, and a
// last-bit change of one moves the BF16 operands of the next step by whole BF16
// units.  Their gradients are therefore summed in orders that do not depend on
// timing, but for what has no order of its own: dV and dC, and the last sum of
// a bias over the CTAs.
//
// Measured on 32 graphs (9.2 k nodes, 185 k edges, k = 20), us, with one thread a
// row and an atomic a channel, and now: edge forward 162 -> 51, head 1362 -> 35,
// edge backward 970 -> 113 (last layer 66), node backward 82 -> 17, node GEMM
// 30 -> 6, embedding backward 419 -> 25; the whole step 5.50 -> 0.62 ms.  The sums in
// order cost 76 us of it: 128-row tiles across nodes take five rounds of the 296
// CTAs where whole nodes take six, and the embedding's strands are a pass of
// their own.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "../../include/cvrp_aco.h"
#include "aco_device.cuh"
#include "umma.cuh"

namespace aco {
namespace {

constexpr int H = 64;
constexpr int FN = ACO_MPNN_NODE_FEATURES;
constexpr int TPB = 256;
constexpr int RT = 128; // rows of an edge tile
constexpr int RPH = RT / (TPB / 16); // rows of a half-warp
constexpr int MS = 68;  // row stride of the FP32 tile: 16-byte accesses by row and by TMEM lane are conflict-free

// ---- packed parameter layout (same order as the oracle) --------------------
struct ParamOffsets {
    int W_n, b_n, W_e, b_e;
    int W[8], b[8], A[8], a[8];
    int W_h, b_h, w_o, b_o, count;
};

__host__ __device__ inline ParamOffsets param_offsets(int L)
{
    ParamOffsets o{};
    int p = 0;
    o.W_n = p; p += H * FN;
    o.b_n = p; p += H;
    o.W_e = p; p += H;
    o.b_e = p; p += H;
    for (int l = 0; l < L; l++) {
        o.W[l] = p; p += 4 * H * H;
        o.b[l] = p; p += 4 * H;
        o.A[l] = p; p += H * H;
        o.a[l] = p; p += H;
    }
    o.W_h = p; p += H * H;
    o.b_h = p; p += H;
    o.w_o = p; p += H;
    o.b_o = p; p += 1;
    o.count = p;
    return o;
}

// ---- workspace layout ------------------------------------------------------
struct Workspace {
    int *status; // [0] the call's status, [4] embed_bwd_kernel's counter
    float *loss;
    float *h, *e, *P, *u; // saved activations (e: layers 1..L, e0 is made from the edge feature)
    uint8_t *qm;          // sign of q: bit i of byte 16 r + l is q > 0 at row r, channel 4 l + i
    float *s;             // edge logits
    float *dh, *de, *dP;  // backward
    float *emb;           // embed_bwd_kernel's partial sums
    size_t bytes;
};

inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

Workspace carve(void *base, int N, int k, int L)
{
    const size_t E = (size_t)N * k;
    Workspace w{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = al256(off + bytes);
        return o;
    };
    const size_t o_status = take(64), o_loss = take(64);
    const size_t o_h = take(sizeof(float) * (L + 1) * N * H), o_e = take(sizeof(float) * L * E * H);
    const size_t o_P = take(sizeof(float) * L * N * 4 * H), o_q = take(L * E * (H / 4));
    const size_t o_u = take(sizeof(float) * L * N * H), o_s = take(sizeof(float) * E);
    const size_t o_dh = take(sizeof(float) * N * H), o_de = take(sizeof(float) * E * H);
    const size_t o_dP = take(sizeof(float) * N * 4 * H), o_emb = take(sizeof(float) * 16 * (FN + 3) * H);
    w.bytes = off;
    if (base) {
        char *b = static_cast<char *>(base);
        w.status = (int *)(b + o_status);
        w.loss = (float *)(b + o_loss);
        w.h = (float *)(b + o_h);
        w.e = (float *)(b + o_e);
        w.P = (float *)(b + o_P);
        w.qm = (uint8_t *)(b + o_q);
        w.u = (float *)(b + o_u);
        w.s = (float *)(b + o_s);
        w.dh = (float *)(b + o_dh);
        w.de = (float *)(b + o_de);
        w.dP = (float *)(b + o_dP);
        w.emb = (float *)(b + o_emb);
    }
    return w;
}

// ---- device helpers ----------------------------------------------------------
__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

__device__ __forceinline__ float4 ldg4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// The components of v whose bit of m is set.
__device__ __forceinline__ float4 masked4(float4 v, unsigned m)
{
    return make_float4(m & 1u ? v.x : 0.f, m & 2u ? v.y : 0.f, m & 4u ? v.z : 0.f, m & 8u ? v.w : 0.f);
}

__device__ __forceinline__ void acc4(float4 &a, float4 b)
{
    a.x += b.x;
    a.y += b.y;
    a.z += b.z;
    a.w += b.w;
}

// Asynchronous copies into shared memory, in groups of a thread's own.
template <int BYTES>
__device__ __forceinline__ void async_copy(void *dst, const void *src)
{
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// All but the thread's last N groups are there.
template <int N>
__device__ __forceinline__ void async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// 16-byte vector reduction into global memory.
__device__ __forceinline__ void red4(float *p, float4 v)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// The same into a caller's gradient, which need not be 16-byte aligned.
__device__ __forceinline__ void add4(float *p, float4 v)
{
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        red4(p, v);
    } else {
        atomicAdd(p, v.x);
        atomicAdd(p + 1, v.y);
        atomicAdd(p + 2, v.z);
        atomicAdd(p + 3, v.w);
    }
}

// Channels 4l..4l+3 of row r into a 64-channel BF16 tile.
__device__ __forceinline__ void put4(uint8_t *tile, int r, int l, float4 v)
{
    const uint32_t lo = (uint32_t)umma::bf16_bits(v.x) | ((uint32_t)umma::bf16_bits(v.y) << 16);
    const uint32_t hi = (uint32_t)umma::bf16_bits(v.z) | ((uint32_t)umma::bf16_bits(v.w) << 16);
    *reinterpret_cast<uint2 *>(tile + umma::sw_offset(r, l >> 1) + ((l & 1) << 3)) = make_uint2(lo, hi);
}

// R rows of 64 channels (row stride ld) into a BF16 tile; rows >= valid are zero.
__device__ __forceinline__ void stage_tile(uint8_t *tile, const float *src, size_t ld, int R, int valid)
{
    const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15;
#pragma unroll 4
    for (int r = hw; r < R; r += TPB / 16) put4(tile, r, hl, r < valid ? ldg4(src + (size_t)r * ld + 4 * hl) : zero4());
}

// The 1024-byte aligned start of the dynamic shared memory (the swizzle's period).
__device__ __forceinline__ uint8_t *tiles_base(uint8_t *sm) { return sm + ((1024u - (smem_u32(sm) & 1023u)) & 1023u); }

// Products issued by thread 0 on 64-channel tiles (umma.cuh), K a multiple of 16:
// D(128 x N) (+)= A B^T, each operand a tile read by rows (K = its 64 channels)
// or transposed (K = K rows of it, M or N = its channels; a_lbo: byte
// distance of the next 64 channels of a transposed A, 0: the same again).
__device__ __forceinline__ void gemm_rows_cols(uint32_t d, const uint8_t *a, const uint8_t *b, bool b_transposed, int N)
{
    if (threadIdx.x == 0) {
        const uint32_t id = umma::idesc_bf16(128, N, false, b_transposed);
        const uint32_t aa = smem_u32(a), bb = smem_u32(b);
        for (int s = 0; s < H / 16; s++)
            umma::mma_bf16(d, umma::desc_k(aa, s), b_transposed ? umma::desc_mn(bb, s, 0) : umma::desc_k(bb, s), id, s > 0);
    }
}

__device__ __forceinline__ void gemm_outer(uint32_t d, const uint8_t *a, uint32_t a_lbo, const uint8_t *b, int K,
                                           bool accumulate)
{
    if (threadIdx.x == 0) {
        const uint32_t id = umma::idesc_bf16(128, H, true, true);
        const uint32_t aa = smem_u32(a), bb = smem_u32(b);
        for (int s = 0; s < (K >> 4); s++)
            umma::mma_bf16(d, umma::desc_mn(aa, s, a_lbo), umma::desc_mn(bb, s, 0), id, accumulate || s > 0);
    }
}

// Make staged operands visible to the tensor core and the CTA.
__device__ __forceinline__ void operands_ready()
{
    umma::fence_async_smem();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
}

// Commit the issued MMAs and wait for them (bounded).  Returns false (uniformly)
// on timeout after recording ACO_ERR_TIMEOUT.
__device__ bool gemm_wait(uint64_t *bar, uint32_t &phase, int *status)
{
    if (threadIdx.x == 0) umma::commit(bar);
    bool ok = mbar_wait(bar, phase);
    if (!ok) {
        set_status(status, ACO_ERR_TIMEOUT);
        mbar_wait(bar, phase); // let the MMAs in flight finish before the CTA lets go of its memory
    }
    phase ^= 1u;
    ok = !__syncthreads_or(!ok);
    umma::fence_after();
    return ok;
}

// Tensor-memory set-up shared by the kernels: mbarrier + allocation by warp 0.
__device__ void tmem_setup(uint64_t *bar, uint32_t *slot, uint32_t ncols)
{
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    if (threadIdx.x < 32) umma::tmem_alloc(slot, ncols);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
}

__device__ void tmem_teardown(uint32_t base, uint32_t ncols)
{
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (threadIdx.x < 32) umma::tmem_dealloc(base, ncols);
}

// The 64 accumulator columns from col0 into the FP32 tile: warp w takes TMEM
// lanes 32 (w mod 4) .. + 31 (tile rows) and columns 32 (w / 4) .. + 31.
__device__ __forceinline__ void acc_to_tile(uint32_t base, int col0, float *ms)
{
    const int w = threadIdx.x >> 5, lane0 = (w & 3) << 5, c0 = (w >> 2) << 5;
    float v[32];
    umma::tmem_ld32(umma::taddr(base, lane0, col0 + c0), v);
    float *row = ms + (size_t)(lane0 + (threadIdx.x & 31)) * MS + c0;
#pragma unroll
    for (int i = 0; i < 32; i += 4) st4(row + i, make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
}

// Rows [0, 64) of the FP32 tile added into a 64 x 64 gradient.
__device__ __forceinline__ void add_tile_rows(const float *ms, float *dst)
{
    const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15;
    for (int r = hw; r < H; r += TPB / 16) add4(dst + r * H + 4 * hl, ld4(ms + (size_t)r * MS + 4 * hl));
}

// ---- forward -----------------------------------------------------------------
__global__ void embed_nodes_kernel(int N, const float *prm, ParamOffsets o, const float *nf, float *h0)
{
    const size_t NH = (size_t)N * H;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < NH; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t i = idx / H;
        const int c = (int)(idx % H);
        float acc = 0.f;
        for (int f = 0; f < FN; f++) acc = __fmaf_rn(prm[o.W_n + c * FN + f], nf[i * FN + f], acc);
        h0[idx] = acc + prm[o.b_n + c];
    }
}

// The embedding of an edge feature on channels with weights w and biases b.
__device__ __forceinline__ float4 embed4(float f, float4 w, float4 b)
{
    return make_float4(__fmaf_rn(w.x, f, b.x), __fmaf_rn(w.y, f, b.y), __fmaf_rn(w.z, f, b.z), __fmaf_rn(w.w, f, b.w));
}

// Shared memory of the edge kernels and the node GEMM: weights, then two
// operand tiles whose place the FP32 tile takes after the product.
struct TileSmem {
    static constexpr size_t W = 0, A = W + H * H * 2, A2 = A + RT * H * 2, M = A, END = M + (size_t)RT * MS * 4,
                            BYTES = END + 1024;
    static_assert(A2 + RT * H * 2 <= END, "the FP32 tile covers both operand tiles");
};

// P = h W^T + b: a CTA takes 128 nodes x one 64-channel section of the 256
// outputs (blockIdx.y), four times the CTAs of whole rows: 9.2 k nodes give 288.
__global__ void __launch_bounds__(TPB) node_gemm_kernel(int N, const float *h, const float *W, const float *bias,
                                                        float *P, int *status)
{
    extern __shared__ uint8_t sm_raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    uint8_t *sm = tiles_base(sm_raw);
    uint8_t *Ws = sm + TileSmem::W, *As = sm + TileSmem::A;
    float *ms = reinterpret_cast<float *>(sm + TileSmem::M);
    tmem_setup(&bar, &slot, 64);
    const uint32_t tm = slot;
    uint32_t phase = 0;
    const int sec = blockIdx.y * H, hw = threadIdx.x >> 4, hl = threadIdx.x & 15;
    stage_tile(Ws, W + (size_t)sec * H, H, H, H);
    const float4 b4 = ldg4(bias + sec + 4 * hl);
    const int tiles = (N + RT - 1) / RT;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int r0 = t * RT, valid = min(RT, N - r0);
        stage_tile(As, h + (size_t)r0 * H, H, RT, valid);
        operands_ready();
        gemm_rows_cols(tm, As, Ws, false, H);
        if (!gemm_wait(&bar, phase, status)) break;
        acc_to_tile(tm, 0, ms);
        __syncthreads();
#pragma unroll
        for (int s = 0; s < RPH; s++) {
            const int r = hw * RPH + s;
            if (r < valid) {
                float4 v = ld4(ms + (size_t)r * MS + 4 * hl);
                acc4(v, b4);
                st4(P + (size_t)(r0 + r) * 4 * H + sec + 4 * hl, v);
            }
        }
        umma::fence_before();
        __syncthreads();
    }
    tmem_teardown(tm, 64);
}

// Edge layer forward on tiles of npt = 128/k nodes.  EMBED: layer 0, e_in is the
// edge feature.  TRAIN: keep the sign of q and u for the backward.  What bounds
// it: HBM (a row of e read, one written) once enough gathers are in flight;
// the P rows come from L2.
template <bool EMBED, bool TRAIN>
__global__ void __launch_bounds__(TPB, 3) edge_fwd_kernel(int N, int k, const float *Wt, const float *a_bias,
                                                          const float *e_in, const float *w_e, const float *b_e,
                                                          const float *P, const float *h_in, const int *nbr,
                                                          uint8_t *qm, float *e_out, float *u_out, float *h_out,
                                                          int *status)
{
    extern __shared__ uint8_t sm_raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    uint8_t *sm = tiles_base(sm_raw);
    uint8_t *Ws = sm + TileSmem::W, *As = sm + TileSmem::A;
    float *ms = reinterpret_cast<float *>(sm + TileSmem::M);
    tmem_setup(&bar, &slot, 64);
    const uint32_t tm = slot;
    uint32_t phase = 0;
    stage_tile(Ws, Wt, H, H, H); // A_l[o][i]: rows o, K = i
    const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15, c = 4 * hl;
    const float4 ab = ldg4(a_bias + c);
    float4 we = zero4(), be = zero4();
    if (EMBED) {
        we = ldg4(w_e + c);
        be = ldg4(b_e + c);
    }
    const int npt = RT / k, tiles = (N + npt - 1) / npt, q0 = hw * RPH / k, rem0 = hw * RPH - q0 * k;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int n0 = t * npt, nodes = min(npt, N - n0), rows = nodes * k;
        const size_t e0 = (size_t)n0 * k;
        float4 ein[RPH];
        int jn[RPH];
#pragma unroll
        for (int s = 0; s < RPH; s++) {
            const int r = hw * RPH + s;
            ein[s] = zero4();
            if (r < rows) ein[s] = EMBED ? embed4(__ldg(e_in + e0 + r), we, be) : ldg4(e_in + (e0 + r) * H + c);
        }
#pragma unroll
        for (int s = 0; s < RPH; s++) {
            const int r = hw * RPH + s;
            put4(As, r, hl, ein[s]);
            jn[s] = r < rows ? __ldg(nbr + e0 + r) : 0;
        }
        operands_ready();
        gemm_rows_cols(tm, As, Ws, false, H);
        if (!gemm_wait(&bar, phase, status)) break;
        acc_to_tile(tm, 0, ms);
        __syncthreads();
        int src = n0 + q0, rem = rem0;
#pragma unroll
        for (int s = 0; s < RPH; s++) {
            const int r = hw * RPH + s;
            if (r < rows) {
                const size_t ei = e0 + r;
                int j = jn[s];
                if ((unsigned)j >= (unsigned)N) { // a neighbour id outside the batch: report, read node 0
                    if (hl == 0) set_status(status, ACO_ERR_INVALID);
                    j = 0;
                }
                const float *Pj = P + (size_t)j * 4 * H + c;
                const float4 pi = ldg4(P + (size_t)src * 4 * H + 2 * H + c), pj = ldg4(Pj + 3 * H), vj = ldg4(Pj + H);
                float *mr = ms + (size_t)r * MS + c;
                const float4 d = ld4(mr);
                const float x0 = d.x + ab.x + pi.x + pj.x, x1 = d.y + ab.y + pi.y + pj.y;
                const float x2 = d.z + ab.z + pi.z + pj.z, x3 = d.w + ab.w + pi.w + pj.w;
                const float4 en = make_float4(ein[s].x + fmaxf(x0, 0.f), ein[s].y + fmaxf(x1, 0.f),
                                              ein[s].z + fmaxf(x2, 0.f), ein[s].w + fmaxf(x3, 0.f));
                st4(e_out + ei * H + c, en);
                if (TRAIN)
                    qm[ei * 16 + hl] = (uint8_t)((x0 > 0.f ? 1 : 0) | (x1 > 0.f ? 2 : 0) | (x2 > 0.f ? 4 : 0) |
                                                 (x3 > 0.f ? 8 : 0));
                // the gated message replaces the accumulator
                st4(mr, make_float4(sigmoidf_(en.x) * vj.x, sigmoidf_(en.y) * vj.y, sigmoidf_(en.z) * vj.z,
                                    sigmoidf_(en.w) * vj.w));
            }
            if (++rem == k) {
                rem = 0;
                src++;
            }
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < nodes * H; idx += TPB) {
            const int qn = idx / H, cc = idx - qn * H, i = n0 + qn;
            float acc = 0.f;
            for (int j = 0; j < k; j++) acc += ms[(size_t)(qn * k + j) * MS + cc];
            const float uv = P[(size_t)i * 4 * H + cc] + acc / (float)k;
            if (TRAIN) u_out[(size_t)i * H + cc] = uv;
            h_out[(size_t)i * H + cc] = h_in[(size_t)i * H + cc] + fmaxf(uv, 0.f);
        }
        umma::fence_before();
        __syncthreads();
    }
    tmem_teardown(tm, 64);
}

// Sum of each of a thread's 32 values over the warp's lanes: lane l ends with
// the total of value l (31 shuffles, against 160 for 32 separate reductions).
__device__ __forceinline__ float transpose_sum32(float (&v)[32])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0];
}

// Head (tiles of 128 edges).  Inference: logits only.  TRAIN: also the
// weighted BCE loss, dL/ds, dz, de = dz W_h and the head's weight gradients.
// Two threads a row (warps w and w + 4 take channels 0-31 and 32-63), column
// sums of dz and ds z by a transposing warp reduction.
template <bool TRAIN>
__global__ void __launch_bounds__(TPB, 3) head_kernel(size_t E, const float *prm, ParamOffsets o, const float *eL,
                                                      float *s_out, const float *labels, float pos_weight, float inv_E,
                                                      float *de, float *grad, float *loss, int *status)
{
    extern __shared__ uint8_t sm_raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    __shared__ float part[RT], s_bh[H], s_wo[H];
    uint8_t *sm = tiles_base(sm_raw);
    uint8_t *Ws = sm + TileSmem::W, *Es = sm + TileSmem::A, *DZs = sm + TileSmem::A2;
    float *ms = reinterpret_cast<float *>(sm + TileSmem::M);
    constexpr uint32_t kCols = TRAIN ? 128 : 64; // cols 0-63 z, then de; 64-127 dW_h
    if (threadIdx.x < H) {
        s_bh[threadIdx.x] = prm[o.b_h + threadIdx.x];
        s_wo[threadIdx.x] = prm[o.w_o + threadIdx.x];
    }
    tmem_setup(&bar, &slot, kCols);
    const uint32_t tm = slot;
    uint32_t phase = 0;
    const float bo = prm[o.b_o];
    stage_tile(Ws, prm + o.W_h, H, H, H); // W_h[o][i]
    const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, half = w >> 2, r = ((w & 3) << 5) + lane, c0 = half << 5;
    float sum_bh = 0.f, sum_wo = 0.f, sum_bo = 0.f, sum_loss = 0.f; // channel c0 + lane; rows of this thread
    bool wg_started = false;
    const size_t tiles = (E + RT - 1) / RT;
    for (size_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const size_t e0 = t * RT;
        const int rows = (int)min((size_t)RT, E - e0);
        stage_tile(Es, eL + e0 * H, H, RT, rows);
        operands_ready();
        gemm_rows_cols(tm, Es, Ws, false, H);
        if (!gemm_wait(&bar, phase, status)) break;
        float zp[32];
        umma::tmem_ld32(umma::taddr(tm, (w & 3) << 5, c0), zp);
#pragma unroll
        for (int i = 0; i < 32; i++) zp[i] += s_bh[c0 + i];
        // the logit is summed channel by channel: the lower half's threads start it, the upper half's end it
        float sv = bo;
        if (half == 0) {
#pragma unroll
            for (int i = 0; i < 32; i++) sv += fmaxf(zp[i], 0.f) * s_wo[i];
            part[r] = sv;
        }
        __syncthreads();
        if (half == 1) {
            sv = part[r];
#pragma unroll
            for (int i = 0; i < 32; i++) sv += fmaxf(zp[i], 0.f) * s_wo[32 + i];
            if (r < rows) s_out[e0 + r] = sv;
        }
        if (!TRAIN) {
            umma::fence_before();
            __syncthreads();
            continue;
        }
        float ds = 0.f;
        if (half == 1) {
            if (r < rows) {
                const float y = labels[e0 + r];
                const float sg = sigmoidf_(sv);
                // -(w y log sig(s) + (1-y) log(1-sig(s))), with log sig(s) = -softplus(-s)
                const float sp_neg = fmaxf(-sv, 0.f) + log1pf(expf(-fabsf(sv)));
                const float sp_pos = fmaxf(sv, 0.f) + log1pf(expf(-fabsf(sv)));
                sum_loss += (pos_weight * y * sp_neg + (1.f - y) * sp_pos) * inv_E;
                ds = (pos_weight * y * (sg - 1.f) + (1.f - y) * sg) * inv_E;
                sum_bo += ds;
            }
            part[r] = ds;
        }
        __syncthreads();
        ds = part[r];
        float tmp[32];
#pragma unroll
        for (int i = 0; i < 32; i++) {
            const float z = fmaxf(zp[i], 0.f);
            tmp[i] = ds * z;
            zp[i] = zp[i] > 0.f ? ds * s_wo[c0 + i] : 0.f; // dz (rows past the end: ds = 0)
        }
        if (r >= rows) // keep whatever the padding rows hold out of the sums and products
#pragma unroll
            for (int i = 0; i < 32; i++) zp[i] = tmp[i] = 0.f;
        sum_wo += transpose_sum32(tmp);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t u[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
                u[i] = (uint32_t)umma::bf16_bits(zp[8 * j + 2 * i]) | ((uint32_t)umma::bf16_bits(zp[8 * j + 2 * i + 1]) << 16);
            *reinterpret_cast<uint4 *>(DZs + umma::sw_offset(r, (c0 >> 3) + j)) = make_uint4(u[0], u[1], u[2], u[3]);
        }
        operands_ready();
        gemm_rows_cols(tm, DZs, Ws, true, H);           // de = dz W_h
        gemm_outer(tm + 64, DZs, 0, Es, RT, wg_started); // dW_h += dz^T eL
        wg_started = true;
        sum_bh += transpose_sum32(zp);
        if (!gemm_wait(&bar, phase, status)) break;
        acc_to_tile(tm, 0, ms);
        __syncthreads();
#pragma unroll
        for (int s = 0; s < RPH; s++) {
            const int rr = hw * RPH + s;
            if (rr < rows) st4(de + (e0 + rr) * H + 4 * hl, ld4(ms + (size_t)rr * MS + 4 * hl));
        }
        umma::fence_before();
        __syncthreads();
    }
    if (TRAIN) {
        __syncthreads();
        umma::fence_after();
        if (wg_started) { // rows o < 64 of the accumulated dW_h (TMEM lanes 0-63)
            acc_to_tile(tm, 64, ms);
            __syncthreads();
            add_tile_rows(ms, grad + o.W_h);
        }
        atomicAdd(&grad[o.b_h + c0 + lane], sum_bh);
        atomicAdd(&grad[o.w_o + c0 + lane], sum_wo);
        if (half == 1) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                sum_bo += __shfl_xor_sync(0xffffffffu, sum_bo, off);
                sum_loss += __shfl_xor_sync(0xffffffffu, sum_loss, off);
            }
            if (lane == 0) {
                atomicAdd(&grad[o.b_o], sum_bo);
                atomicAdd(loss, sum_loss);
            }
        }
    }
    tmem_teardown(tm, kCols);
}

// ---- backward ------------------------------------------------------------------
// Edge layer backward on tiles of npt = 128/k nodes.  dh = dL/dh', de = dL/de'
// (overwritten by dL/de); dP receives du and dB (owned) and dV and dC (vector
// reductions into a zeroed buffer).  LAST: the last layer, where dh = 0 and so
// du and dV are zero.  EMBED: layer 0, whose e_in is made from the edge feature.
template <bool LAST, bool EMBED>
__global__ void __launch_bounds__(TPB, 2) edge_bwd_kernel(int N, int k, const float *A_w, const float *P,
                                                          const float *u, const uint8_t *qm, const float *e_in,
                                                          const float *w_e, const float *b_e, const float *e_out,
                                                          const int *nbr, const float *dh, float *de, float *dP,
                                                          float *gA, float *ga, int *status)
{
    extern __shared__ uint8_t sm_raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    uint8_t *sm = tiles_base(sm_raw);
    uint8_t *Ws = sm + TileSmem::W, *DQs = sm + TileSmem::A, *Es = sm + TileSmem::A2;
    float *ms = reinterpret_cast<float *>(sm + TileSmem::M);
    tmem_setup(&bar, &slot, 128);
    const uint32_t tm = slot; // cols 0-63 dq A, 64-127 dA
    uint32_t phase = 0;
    stage_tile(Ws, A_w, H, H, H); // A[o][i]
    const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15, c = 4 * hl;
    constexpr int kNodeThreads = TPB - H; // the last H threads sum the columns, the others the nodes
    float4 we = zero4(), be = zero4();
    if (EMBED) {
        we = ldg4(w_e + c);
        be = ldg4(b_e + c);
    }
    const float kf = (float)k;
    float sum_a = 0.f;
    bool wg_started = false;
    const int npt = RT / k, tiles = (N + npt - 1) / npt, q0 = hw * RPH / k, rem0 = hw * RPH - q0 * k;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int n0 = t * npt, nodes = min(npt, N - n0), rows = nodes * k;
        const size_t e0 = (size_t)n0 * k;
        int src = n0 + q0, rem = rem0;
        float4 dt[RPH];
        int jn[RPH];
        uint32_t mask = 0u; // the rows' signs of q, a nibble each
#pragma unroll
        for (int s = 0; s < RPH; s++) {
            const int r = hw * RPH + s;
            float4 dq = zero4(), ei4 = zero4();
            dt[s] = zero4();
            if (r < rows) {
                const size_t ei = e0 + r;
                int j = __ldg(nbr + ei);
                if (EMBED) ei4 = embed4(__ldg(e_in + ei), we, be);
                else ei4 = ldg4(e_in + ei * H + c);
                const unsigned m = qm[ei * 16 + hl];
                mask |= m << (4 * s);
                float4 d = ld4(de + ei * H + c);
                if ((unsigned)j >= (unsigned)N) {
                    if (hl == 0) set_status(status, ACO_ERR_INVALID);
                    j = 0;
                }
                jn[s] = j;
                if (!LAST) {
                    const float4 eo = ldg4(e_out + ei * H + c), vj = ldg4(P + (size_t)j * 4 * H + H + c);
                    const float4 uu = ldg4(u + (size_t)src * H + c), hh = ldg4(dh + (size_t)src * H + c);
                    const float4 du = make_float4(uu.x > 0.f ? hh.x : 0.f, uu.y > 0.f ? hh.y : 0.f,
                                                  uu.z > 0.f ? hh.z : 0.f, uu.w > 0.f ? hh.w : 0.f);
                    if (rem == 0) st4(dP + (size_t)src * 4 * H + c, du);
                    const float4 du_e = make_float4(du.x / kf, du.y / kf, du.z / kf, du.w / kf);
                    const float g0 = sigmoidf_(eo.x), g1 = sigmoidf_(eo.y), g2 = sigmoidf_(eo.z), g3 = sigmoidf_(eo.w);
                    red4(dP + (size_t)j * 4 * H + H + c, make_float4(du_e.x * g0, du_e.y * g1, du_e.z * g2, du_e.w * g3));
                    d.x += du_e.x * vj.x * g0 * (1.f - g0);
                    d.y += du_e.y * vj.y * g1 * (1.f - g1);
                    d.z += du_e.z * vj.z * g2 * (1.f - g2);
                    d.w += du_e.w * vj.w * g3 * (1.f - g3);
                }
                dt[s] = d; // the residual part; the product is added below
                dq = masked4(d, m);
                if (!LAST) red4(dP + (size_t)j * 4 * H + 3 * H + c, dq);
            }
            put4(DQs, r, hl, dq);
            put4(Es, r, hl, ei4);
            if (++rem == k) {
                rem = 0;
                src++;
            }
        }
        operands_ready();
        gemm_rows_cols(tm, DQs, Ws, true, H);           // dq A
        gemm_outer(tm + 64, DQs, 0, Es, RT, wg_started); // dA += dq^T e_in
        wg_started = true;
        if (!gemm_wait(&bar, phase, status)) break;
        acc_to_tile(tm, 0, ms);
        __syncthreads();
#pragma unroll
        for (int s = 0; s < RPH; s++) {
            const int r = hw * RPH + s;
            if (r < rows) {
                float *mr = ms + (size_t)r * MS + c;
                const float4 d = ld4(mr);
                st4(de + (e0 + r) * H + c,
                    make_float4(dt[s].x + d.x, dt[s].y + d.y, dt[s].z + d.z, dt[s].w + d.w));
                const float4 dq = masked4(dt[s], mask >> (4 * s));
                if (LAST) red4(dP + (size_t)jn[s] * 4 * H + 3 * H + c, dq); // out of the way of the rows' reads
                st4(mr, dq); // replaces the product
            }
        }
        __syncthreads();
        if (threadIdx.x < kNodeThreads) {
            for (int idx = threadIdx.x; idx < nodes * H; idx += kNodeThreads) {
                const int qn = idx / H, cc = idx - qn * H;
                float acc = 0.f;
                for (int j = 0; j < k; j++) acc += ms[(size_t)(qn * k + j) * MS + cc];
                dP[(size_t)(n0 + qn) * 4 * H + 2 * H + cc] = acc;
            }
        } else {
            const float *col = ms + (threadIdx.x - kNodeThreads);
            float acc = 0.f;
#pragma unroll 8
            for (int r = 0; r < rows; r++) acc += col[(size_t)r * MS];
            sum_a += acc;
        }
        umma::fence_before();
        __syncthreads();
    }
    __syncthreads();
    umma::fence_after();
    if (wg_started) {
        acc_to_tile(tm, 64, ms);
        __syncthreads();
        add_tile_rows(ms, gA);
    }
    if (threadIdx.x >= kNodeThreads) atomicAdd(ga + (threadIdx.x - kNodeThreads), sum_a);
    tmem_teardown(tm, 128);
}

// dh += dP W (K = 256), dW += dP^T h (two halves of 128 outputs) on tiles of 64
// nodes (twice the CTAs of 128: 9.2 k nodes give 144), db += sum dP.  The
// accumulator of dP W has 128 rows; its upper 64 come from whatever follows
// the operand's 64 rows in shared memory and are not read.  LAST: dh = 0 on
// entry.  db: the first bias_groups CTAs sum an output a thread over every
// bias_groups-th 128 nodes in order, beside the others (two CTAs fit an SM).
struct NodeBwdSmem {
    static constexpr int NT = 64;
    static constexpr size_t A = 0, W = A + 4 * NT * H * 2, HT = W + 4 * H * H * 2, M = HT + NT * H * 2,
                            END = M + (size_t)RT * MS * 4, BYTES = END + 1024;
};

template <bool LAST>
__global__ void __launch_bounds__(TPB, 2) node_bwd_kernel(int N, const float *W, const float *h_in, const float *dP,
                                                       float *dh, float *gW, float *gb, int bias_groups, int *status)
{
    extern __shared__ uint8_t sm_raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    constexpr int NT = NodeBwdSmem::NT, RH = NT / (TPB / 16);
    constexpr uint32_t kAtom = NT * H * 2; // bytes of 64 channels of the dP tile
    if ((int)blockIdx.x < bias_groups) {
        float sum = 0.f;
        for (int i0 = (int)blockIdx.x * RT; i0 < N; i0 += bias_groups * RT) {
            const float *col = dP + (size_t)i0 * 4 * H + threadIdx.x;
            const int rows = min(RT, N - i0);
            float acc = 0.f;
#pragma unroll 64
            for (int i = 0; i < rows; i++) acc += __ldg(col + (size_t)i * 4 * H);
            sum += acc;
        }
        atomicAdd(gb + threadIdx.x, sum);
        return;
    }
    uint8_t *sm = tiles_base(sm_raw);
    uint8_t *As = sm + NodeBwdSmem::A, *Ws = sm + NodeBwdSmem::W, *Hs = sm + NodeBwdSmem::HT;
    float *ms = reinterpret_cast<float *>(sm + NodeBwdSmem::M);
    tmem_setup(&bar, &slot, 256);
    const uint32_t tm = slot; // 0-63 dgrad, 64-127 dW rows 0-127, 128-191 dW rows 128-255
    uint32_t phase = 0;
    stage_tile(Ws, W, H, 4 * H, 4 * H); // W[o][c], 256 rows
    const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15, c = 4 * hl;
    const int sec = (threadIdx.x >> 4) & 3, rq = threadIdx.x >> 6; // staging: section and row group of the thread
    bool wg_started = false;
    const int tiles = (N + NT - 1) / NT;
    for (int t = (int)blockIdx.x - bias_groups; t < tiles; t += (int)gridDim.x - bias_groups) {
        const int r0 = t * NT, valid = min(NT, N - r0);
#pragma unroll 8
        for (int r = rq; r < NT; r += 4) {
            const float4 v = r < valid ? ldg4(dP + (size_t)(r0 + r) * 4 * H + sec * H + c) : zero4();
            put4(As + sec * kAtom, r, hl, v);
        }
        stage_tile(Hs, h_in + (size_t)r0 * H, H, NT, valid);
        operands_ready();
        if (threadIdx.x == 0) { // dP W: K = 256 outputs, A by rows (four 64-channel sections), W transposed
            const uint32_t id = umma::idesc_bf16(128, H, false, true);
            const uint32_t aa = smem_u32(As), bb = smem_u32(Ws);
            for (int s = 0; s < 4 * H / 16; s++)
                umma::mma_bf16(tm, umma::desc_k(aa + (s >> 2) * kAtom, s & 3), umma::desc_mn(bb, s, 0), id, s > 0);
        }
        gemm_outer(tm + 64, As, kAtom, Hs, NT, wg_started);
        gemm_outer(tm + 128, As + 2 * kAtom, kAtom, Hs, NT, wg_started);
        wg_started = true;
        if (!gemm_wait(&bar, phase, status)) break;
        acc_to_tile(tm, 0, ms);
        __syncthreads();
#pragma unroll
        for (int s = 0; s < RH; s++) {
            const int r = hw * RH + s;
            if (r < valid) {
                float4 d = ld4(ms + (size_t)r * MS + c);
                float *row = dh + (size_t)(r0 + r) * H + c;
                if (!LAST) {
                    const float4 o = ld4(row);
                    d = make_float4(o.x + d.x, o.y + d.y, o.z + d.z, o.w + d.w);
                }
                st4(row, d);
            }
        }
        umma::fence_before();
        __syncthreads();
    }
    __syncthreads();
    umma::fence_after();
    if (wg_started) {
        for (int half = 0; half < 2; half++) {
            acc_to_tile(tm, 64 + 64 * half, ms);
            __syncthreads();
            for (int r = hw; r < RT; r += TPB / 16) add4(gW + (size_t)(half * RT + r) * H + c, ld4(ms + (size_t)r * MS + c));
            __syncthreads();
        }
    }
    tmem_teardown(tm, 256);
}

// Gradients of the input embeddings (K = 5 and 1).  Strand t of 256 sums the nodes
// and the edges t, t + 256, ... in order; each 32 strands then add up in a
// butterfly (lanes 16 apart, 8, 4, 2, 1), and the eight results in turn.  A CTA
// takes all channels of two strands 16 apart, a cluster the even or the odd
// lanes of a butterfly, and the last CTA to finish adds the 16 clusters' sums
// (half, a counter in done).  The edge rows come through a ring of asynchronous
// copies made by half of the CTA's warps, 32 KB of them in flight a CTA: the 16 k
// chains of sums are too few to hide the reads by themselves.
constexpr int kStrands = 256, kEmbedSums = (FN + 3) * H, kEmbedCtas = kStrands / 2;

__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(4 * H)
    embed_bwd_kernel(int N, int E, const float *nf, const float *ef, const float *dh, const float *de, float *half,
                     int *done, float *gwn, float *gbn, float *gwe, float *gbe)
{
    static_assert(FN + 3 == 8, "a CTA of the cluster adds one of the sums");
    constexpr int R = 16, D = 5; // rows of a strand a stage, stages of the ring
    __shared__ __align__(16) float rows[D][2][R][H];
    __shared__ float feat[D][2][R], part[2][FN + 3][H], pair[FN + 3][H];
    __shared__ int last;
    const auto cluster = cooperative_groups::this_cluster();
    const int c = threadIdx.x % H, s = (threadIdx.x / H) & 1, r = (int)cluster.block_rank(), q = (int)(blockIdx.x >> 3);
    const int t0 = 32 * (q >> 1) + 2 * r + (q & 1), t = t0 + 16 * s; // its first strand, the thread's
    auto strand = [](int n, int t) { return n > t ? (n - t + kStrands - 1) / kStrands : 0; };
    const int n_nodes = strand(N, t), n_edges = strand(E, t), stages = (strand(E, t0) + R - 1) / R;
    // threads from 2 H on: 16 bytes of row p (and p + 8 of the stage, in both strands)
    const bool copies = threadIdx.x >= 2 * H;
    const int p = (threadIdx.x >> 4) & 7, c4 = 4 * (threadIdx.x & 15);
    auto fetch = [&](int i) { // stage i, if there is one, into its place of the ring
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = p + 8 * (j & 1), ss = j >> 1;
            const size_t e = ((size_t)i * R + k) * kStrands + t0 + 16 * ss;
            if (e >= (size_t)E) continue;
            async_copy<16>(&rows[i % D][ss][k][c4], de + e * H + c4);
            if (c4 == 0) async_copy<4>(&feat[i % D][ss][k], ef + e);
        }
        async_commit();
    };
    if (copies)
        for (int i = 0; i < D - 1; i++) fetch(i);
    float acc[FN + 3];
#pragma unroll
    for (int f = 0; f < FN + 3; f++) acc[f] = 0.f;
    constexpr int UN = 12; // nodes in flight
    for (int i0 = 0; i0 < n_nodes && !copies; i0 += UN) {
        const size_t at = (size_t)i0 * kStrands + t;
        const float *pd = dh + at * H + c, *pf = nf + at * FN;
        float d[UN], x[UN][FN];
#pragma unroll
        for (int i = 0; i < UN; i++) {
            const bool in = i0 + i < n_nodes;
            d[i] = in ? __ldg(pd + i * kStrands * H) : 0.f;
#pragma unroll
            for (int f = 0; f < FN; f++) x[i][f] = in ? __ldg(pf + i * kStrands * FN + f) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < UN; i++) {
            if (i0 + i >= n_nodes) break;
#pragma unroll
            for (int f = 0; f < FN; f++) acc[f] += d[i] * x[i][f];
            acc[FN] += d[i];
        }
    }
    for (int i = 0; i < stages; i++) {
        if (copies) async_wait<D - 2>();
        __syncthreads(); // stage i is there, and the place of stage i - 1 is free
        if (copies) {
            fetch(i + D - 1);
            continue;
        }
        float d[R], x[R];
#pragma unroll
        for (int k = 0; k < R; k++) {
            d[k] = rows[i % D][s][k][c];
            x[k] = feat[i % D][s][k];
        }
#pragma unroll
        for (int k = 0; k < R; k++)
            if (i * R + k < n_edges) {
                acc[FN + 1] += d[k] * x[k];
                acc[FN + 2] += d[k];
            }
    }
    if (!copies)
#pragma unroll
        for (int f = 0; f < FN + 3; f++) part[s][f][c] = acc[f];
    __syncthreads();
    for (int i = threadIdx.x; i < kEmbedSums; i += 4 * H) pair[0][i] = part[0][0][i] + part[1][0][i];
    cluster.sync();
    if (threadIdx.x < H) { // sum r of the cluster's 16 strands
        float v[8];
        for (int i = 0; i < 8; i++) v[i] = *cluster.map_shared_rank(&pair[r][c], i);
        __stcg(half + (size_t)q * kEmbedSums + r * H + c,
               ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7])));
        __threadfence();
    }
    cluster.sync(); // the pairs have been read, the sums written
    if (threadIdx.x == 0) last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < kEmbedSums; i += 4 * H) {
        const int f = i / H, ch = i % H;
        float v = 0.f;
        for (int w = 0; w < 8; w++)
            v += __ldcg(half + (size_t)(2 * w) * kEmbedSums + i) + __ldcg(half + (size_t)(2 * w + 1) * kEmbedSums + i);
        if (f < FN) gwn[ch * FN + f] = v;
        else if (f == FN) gbn[ch] = v;
        else if (f == FN + 1) gwe[ch] = v;
        else gbe[ch] = v;
    }
}

__global__ void adam_kernel(int n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2,
                            float eps, float c1, float c2)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

int g_sm_count = 0;

int sm_count()
{
    if (g_sm_count == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (g_sm_count <= 0) g_sm_count = 148;
    }
    return g_sm_count;
}

template <typename K>
cudaError_t set_smem(K kern, size_t bytes)
{
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

bool args_ok(int N, int k, int L)
{
    return N >= 1 && k >= 1 && k <= 32 && L >= 1 && L <= 8 && (size_t)N * k < ((size_t)1 << 31);
}

// A persistent grid: at most as many CTAs as are resident at once (ctas per SM).
unsigned grid_of(size_t tiles, int ctas) { return (unsigned)std::min(tiles, (size_t)sm_count() * ctas); }

template <bool EMBED, bool TRAIN>
cudaError_t launch_edge_fwd(int N, int k, const float *prm, const ParamOffsets &o, int l, const float *e_in,
                            const float *h, const int *nbr, const float *P, const Workspace &w, cudaStream_t st)
{
    const size_t E = (size_t)N * k;
    const cudaError_t e = set_smem(edge_fwd_kernel<EMBED, TRAIN>, TileSmem::BYTES);
    if (e != cudaSuccess) return e;
    const int npt = RT / k;
    edge_fwd_kernel<EMBED, TRAIN><<<grid_of((N + npt - 1) / npt, 3), TPB, TileSmem::BYTES, st>>>(
        N, k, prm + o.A[l], prm + o.a[l], e_in, prm + o.W_e, prm + o.b_e, P, h, nbr, w.qm + (size_t)l * E * 16,
        w.e + (size_t)l * E * H, w.u + (size_t)l * N * H, w.h + (size_t)(l + 1) * N * H, w.status);
    return cudaGetLastError();
}

template <bool TRAIN>
int run_forward(int N, int k, int L, const float *prm, const float *nf, const float *ef, const int *nbr,
                const Workspace &w, cudaStream_t st)
{
    const ParamOffsets o = param_offsets(L);
    const size_t E = (size_t)N * k;
    embed_nodes_kernel<<<grid_of(((size_t)N * H + 255) / 256, 8), 256, 0, st>>>(N, prm, o, nf, w.h);
    if (set_smem(node_gemm_kernel, TileSmem::BYTES) != cudaSuccess) return ACO_ERR_CUDA;
    const size_t ntiles = (N + RT - 1) / RT;
    for (int l = 0; l < L; l++) {
        const float *h = w.h + (size_t)l * N * H;
        float *P = w.P + (size_t)l * N * 4 * H;
        node_gemm_kernel<<<dim3(grid_of(ntiles, 1), 4), TPB, TileSmem::BYTES, st>>>(N, h, prm + o.W[l], prm + o.b[l], P,
                                                                                   w.status);
        const cudaError_t e = l == 0 ? launch_edge_fwd<true, TRAIN>(N, k, prm, o, l, ef, h, nbr, P, w, st)
                                     : launch_edge_fwd<false, TRAIN>(N, k, prm, o, l, w.e + (size_t)(l - 1) * E * H, h,
                                                                     nbr, P, w, st);
        if (e != cudaSuccess) return ACO_ERR_CUDA;
    }
    return cudaGetLastError() == cudaSuccess ? ACO_OK : ACO_ERR_CUDA;
}

template <bool TRAIN>
cudaError_t launch_head(size_t E, const float *prm, const ParamOffsets &o, const float *eL, float *scores,
                        const float *labels, float pos_weight, float *de, float *grad, float *loss, int *status,
                        cudaStream_t st)
{
    const cudaError_t e = set_smem(head_kernel<TRAIN>, TileSmem::BYTES);
    if (e != cudaSuccess) return e;
    head_kernel<TRAIN><<<grid_of((E + RT - 1) / RT, 3), TPB, TileSmem::BYTES, st>>>(
        E, prm, o, eL, scores, labels, pos_weight, 1.0f / (float)E, de, grad, loss, status);
    return cudaGetLastError();
}

template <bool LAST, bool EMBED>
cudaError_t launch_layer_bwd(int N, int k, const float *prm, const ParamOffsets &o, int l, const float *ef,
                             const int *nbr, const Workspace &w, float *grad, cudaStream_t st)
{
    const size_t E = (size_t)N * k;
    cudaError_t e = cudaMemsetAsync(w.dP, 0, sizeof(float) * N * 4 * H, st);
    if (e == cudaSuccess) e = set_smem(edge_bwd_kernel<LAST, EMBED>, TileSmem::BYTES);
    if (e == cudaSuccess) e = set_smem(node_bwd_kernel<LAST>, NodeBwdSmem::BYTES);
    if (e != cudaSuccess) return e;
    const int npt = RT / k;
    edge_bwd_kernel<LAST, EMBED><<<grid_of((N + npt - 1) / npt, 2), TPB, TileSmem::BYTES, st>>>(
        N, k, prm + o.A[l], w.P + (size_t)l * N * 4 * H, w.u + (size_t)l * N * H, w.qm + (size_t)l * E * 16,
        EMBED ? ef : w.e + (size_t)(l - 1) * E * H, prm + o.W_e, prm + o.b_e, w.e + (size_t)l * E * H, nbr, w.dh, w.de,
        w.dP, grad + o.A[l], grad + o.a[l], w.status);
    const unsigned bias_groups = grid_of((N + RT - 1) / RT, 2);
    node_bwd_kernel<LAST><<<bias_groups + grid_of((N + NodeBwdSmem::NT - 1) / NodeBwdSmem::NT, 1), TPB,
                            NodeBwdSmem::BYTES, st>>>(N, prm + o.W[l], w.h + (size_t)l * N * H, w.dP, w.dh,
                                                      grad + o.W[l], grad + o.b[l], (int)bias_groups, w.status);
    return cudaGetLastError();
}

} // namespace
} // namespace aco

using namespace aco;

extern "C" {

int aco_mpnn_param_count(int layers)
{
    if (layers < 1 || layers > 8) return ACO_ERR_INVALID;
    return param_offsets(layers).count;
}

int aco_mpnn_workspace_bytes(int n_nodes, int k, int layers, size_t *bytes)
{
    if (!bytes || !args_ok(n_nodes, k, layers)) return ACO_ERR_INVALID;
    *bytes = carve(nullptr, n_nodes, k, layers).bytes;
    return ACO_OK;
}

int aco_mpnn_forward(int n_nodes, int k, int layers, const float *params, const float *node_feat,
                     const float *edge_feat, const int *nbr, void *workspace, size_t ws_bytes, float *scores,
                     void *stream)
{
    if (!args_ok(n_nodes, k, layers) || !params || !node_feat || !edge_feat || !nbr || !workspace || !scores)
        return ACO_ERR_INVALID;
    const Workspace w = carve(workspace, n_nodes, k, layers);
    if (ws_bytes < w.bytes) return ACO_ERR_CAPACITY;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(w.status, 0, 64, st) != cudaSuccess) return ACO_ERR_CUDA;
    int rc = run_forward<false>(n_nodes, k, layers, params, node_feat, edge_feat, nbr, w, st);
    if (rc != ACO_OK) return rc;
    const size_t E = (size_t)n_nodes * k;
    return launch_head<false>(E, params, param_offsets(layers), w.e + (size_t)(layers - 1) * E * H, scores, nullptr, 0.f,
                              nullptr, nullptr, nullptr, w.status, st) == cudaSuccess
               ? ACO_OK
               : ACO_ERR_CUDA;
}

int aco_mpnn_grad(int n_nodes, int k, int layers, const float *params, const float *node_feat, const float *edge_feat,
                  const int *nbr, const float *labels, float pos_weight, void *workspace, size_t ws_bytes, float *grad,
                  float *loss, float *scores, void *stream)
{
    if (!args_ok(n_nodes, k, layers) || !params || !node_feat || !edge_feat || !nbr || !labels || !workspace ||
        !grad || !loss)
        return ACO_ERR_INVALID;
    const Workspace w = carve(workspace, n_nodes, k, layers);
    if (ws_bytes < w.bytes) return ACO_ERR_CAPACITY;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const ParamOffsets o = param_offsets(layers);
    const size_t E = (size_t)n_nodes * k;
    const int N = n_nodes, L = layers;
    if (cudaMemsetAsync(w.status, 0, 64, st) != cudaSuccess) return ACO_ERR_CUDA;
    if (cudaMemsetAsync(grad, 0, sizeof(float) * o.count, st) != cudaSuccess) return ACO_ERR_CUDA;
    if (cudaMemsetAsync(loss, 0, sizeof(float), st) != cudaSuccess) return ACO_ERR_CUDA;
    int rc = run_forward<true>(N, k, L, params, node_feat, edge_feat, nbr, w, st);
    if (rc != ACO_OK) return rc;
    if (launch_head<true>(E, params, o, w.e + (size_t)(L - 1) * E * H, scores ? scores : w.s, labels, pos_weight, w.de,
                          grad, loss, w.status, st) != cudaSuccess)
        return ACO_ERR_CUDA;
    for (int l = L - 1; l >= 0; l--) {
        const bool last = l == L - 1, embed = l == 0;
        const cudaError_t e =
            last ? (embed ? launch_layer_bwd<true, true>(N, k, params, o, l, edge_feat, nbr, w, grad, st)
                          : launch_layer_bwd<true, false>(N, k, params, o, l, edge_feat, nbr, w, grad, st))
                 : (embed ? launch_layer_bwd<false, true>(N, k, params, o, l, edge_feat, nbr, w, grad, st)
                          : launch_layer_bwd<false, false>(N, k, params, o, l, edge_feat, nbr, w, grad, st));
        if (e != cudaSuccess) return ACO_ERR_CUDA;
    }
    embed_bwd_kernel<<<kEmbedCtas, 4 * H, 0, st>>>(
        N, (int)E, node_feat, edge_feat, w.dh, w.de, w.emb, w.status + 4, grad + o.W_n, grad + o.b_n, grad + o.W_e, grad + o.b_e);
    return cudaGetLastError() == cudaSuccess ? ACO_OK : ACO_ERR_CUDA;
}

int aco_mpnn_adam(int count, float *params, const float *grad, float *m, float *v, float lr, float beta1, float beta2,
                  float eps, int step, void *stream)
{
    if (count <= 0 || !params || !grad || !m || !v || step < 1) return ACO_ERR_INVALID;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<std::min((count + 255) / 256, 1024), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        count, params, grad, m, v, lr, beta1, beta2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? ACO_OK : ACO_ERR_CUDA;
}

int aco_mpnn_status(void *workspace, void *stream)
{
    if (!workspace) return ACO_ERR_INVALID;
    int h = 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(&h, workspace, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return ACO_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return ACO_ERR_CUDA;
    return h;
}

} // extern "C"
