// Learned warm start for swing-network steady states: a message-passing network on one
// fixed graph maps per-instance power injections P and line weights K to steady-state
// phases, trained and evaluated by the kernels below (FP32).  It has no counterpart in
// the reference, whose find_fixpoint (src/initialization.jl:44-144) starts Newton from a
// caller-given guess; its prediction only replaces that guess.
//
// Architecture (hidden width H = 64, L layers), per instance b and vertex i:
//   s_i  = Σ_j K_ij / κ                        (κ = kWeightScale; j over the neighbours)
//   x_i  = [P_i, log(1 + s_i)]
//   h0_i = tanh(W_in x_i + b_in)
//   m    = M^k h,  (M h)_i = (1 / s_i) Σ_j (K_ij / κ) h_j    (k = hops weighted-mean steps)
//   a_i  = tanh(W_s h_i + W_m m_i + b),  h'_i = h_i + a_i          (L residual layers)
//   y_i  = w_out · h_i + b_out,  θ̂_i = y_i - mean_i(y)          (phases up to a shift)
// The steady-state frequency is ω* = 0 at every fixpoint of the swing equations, so only
// θ is predicted.  Loss = mean over instances and vertices of (θ̂ - (θ* - mean θ*))².
//
// Parameters are one flat FP32 vector: W_in[H][2], b_in[H], per layer W_s[H][H],
// W_m[H][H], b[H] (row = output unit), then w_out[H], b_out.  Rows of every activation
// array are r = b * nv + i with H contiguous floats.  Weight gradients are reduced as
// fixed per-block partials followed by an ordered sum, so a training run is
// deterministic.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include "nd_internal.h"

namespace nd {
namespace mpnn {

constexpr int kH = 64;
constexpr float kWeightScale = 10.0f;
constexpr int kBlock = 256;
constexpr int kGradBlocks = 304;             // blocks of the weight-gradient reductions (2 per SM)
static_assert(kGradBlocks % 8 == 0, "shares of reduce_partials_kernel");
constexpr int kPartialStride = 2 * kH * kH + kH;

__host__ __device__ inline int64_t off_win() { return 0; }
__host__ __device__ inline int64_t off_bin() { return 2 * kH; }
__host__ __device__ inline int64_t off_layer(int l) { return 3 * kH + (int64_t)l * (2 * kH * kH + kH); }
__host__ __device__ inline int64_t off_wout(int L) { return off_layer(L); }
__host__ __device__ inline int64_t off_bout(int L) { return off_layer(L) + kH; }
inline int64_t num_params(int L) { return off_bout(L) + 1; }

__host__ __device__ inline int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

inline unsigned grid_for(int64_t n, int block = kBlock) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + block - 1) / block, 152 * 16));
}

// ---- forward --------------------------------------------------------------------------------

// wt[b][k] = K / κ of incidence k of the CSR, a thread per (instance, incidence): every message
// pass reads these in order instead of dividing a gathered K per lane
__global__ void weights_kernel(int64_t n, int64_t ninc, int64_t ne, const int32_t* __restrict__ eid,
                               const float* __restrict__ K, float* __restrict__ wt) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = t / ninc;
        wt[t] = __ldg(K + b * ne + __ldg(eid + (t - b * ninc))) / kWeightScale;
    }
}

// x = [P, log1p(s)], inv_s = 1 / s (0 for isolated vertices) and h0 = tanh(W_in x + b_in), a
// half-warp per row, four units per lane
__global__ void __launch_bounds__(kBlock) encode_kernel(int64_t R, int64_t nv, int64_t ninc,
                                                        const uint32_t* __restrict__ row_ptr,
                                                        const float* __restrict__ wt, const float* __restrict__ P,
                                                        const float* __restrict__ prm, float* __restrict__ x,
                                                        float* __restrict__ inv_s, float* __restrict__ h0) {
    const int sub = threadIdx.x & 15;
    const unsigned half = 0xffffu << (threadIdx.x & 16);
    const float4 Wa = reinterpret_cast<const float4*>(prm + off_win())[2 * sub];  // units 4 sub, 4 sub + 1
    const float4 Wb = reinterpret_cast<const float4*>(prm + off_win())[2 * sub + 1];
    const float4 bb = reinterpret_cast<const float4*>(prm + off_bin())[sub];
    const int64_t groups = (int64_t)gridDim.x * (blockDim.x >> 4);
    for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 4) + (threadIdx.x >> 4); r < R; r += groups) {
        const int64_t b = r / nv, i = r - b * nv;
        float s = 0.f;
        const uint32_t k1 = __ldg(row_ptr + i + 1);
        for (uint32_t k = __ldg(row_ptr + i) + sub; k < k1; k += 16) s += __ldg(wt + b * ninc + k);
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(half, s, off, 16);
        const float x0 = __ldg(P + r), x1 = log1pf(s);
        if (sub == 0) {
            reinterpret_cast<float2*>(x)[r] = make_float2(x0, x1);
            inv_s[r] = s > 0.f ? 1.f / s : 0.f;
        }
        reinterpret_cast<float4*>(h0 + r * kH)[sub] =
            make_float4(tanhf(fmaf(Wa.x, x0, fmaf(Wa.y, x1, bb.x))), tanhf(fmaf(Wa.z, x0, fmaf(Wa.w, x1, bb.y))),
                        tanhf(fmaf(Wb.x, x0, fmaf(Wb.y, x1, bb.z))), tanhf(fmaf(Wb.z, x0, fmaf(Wb.w, x1, bb.w))));
    }
}

// out_r (=, or += with accumulate) post_r · Σ_k wt_k · pre_n · in_n over the neighbours n of row
// r (pre / post may be NULL = 1).  A half-warp per row, four units per lane: its 16 lanes load 16
// neighbours and weights at once, and the rows of four neighbours are in flight before the
// first is added (one neighbour at a time is a chain of two memory round trips each).  The
// vertices come in order of degree, every instance's copy of one after the other, so that the
// hubs start first: in row order the last instance's hubs left 40 % of the SMs idle at the end.
// At 128,000 rows of 4 neighbours on average: 72 µs -> 31 µs (131 MB of neighbour rows from L2).
__global__ void __launch_bounds__(kBlock) aggregate_kernel(int64_t R, int64_t nv, int64_t batch, int64_t ninc,
                                                           const int32_t* __restrict__ order,
                                                           const uint32_t* __restrict__ row_ptr,
                                                           const int32_t* __restrict__ nbr, const float* __restrict__ wt,
                                                           const float* __restrict__ pre, const float* __restrict__ post,
                                                           const float* __restrict__ in, float* __restrict__ out,
                                                           int accumulate) {
    const int sub = threadIdx.x & 15;
    const unsigned half = 0xffffu << (threadIdx.x & 16);
    const int64_t t = (int64_t)blockIdx.x * (kBlock / 16) + (threadIdx.x >> 4);
    if (t >= R) return;  // uniform in the half-warp
    const int64_t vi = t / batch, b = t - vi * batch;
    const int64_t i = __ldg(order + vi), r = b * nv + i;
    const uint32_t k1 = __ldg(row_ptr + i + 1);
    const float4* rows = reinterpret_cast<const float4*>(in + b * nv * kH) + sub;
    const float* wb = wt + b * ninc;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t k0 = __ldg(row_ptr + i); k0 < k1; k0 += 16) {
        int n = 0;
        float w = 0.f;
        if (k0 + sub < k1) {
            n = __ldg(nbr + k0 + sub);
            w = __ldg(wb + k0 + sub);
            if (pre) w *= __ldg(pre + b * nv + n);
        }
        const int m = (int)min(16u, k1 - k0);
        for (int j = 0; j < m; j += 4) {
            float4 v[4];
            float wj[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                wj[q] = __shfl_sync(half, w, j + q, 16);  // 0 past the row's end
                const int nj = __shfl_sync(half, n, j + q, 16);
                v[q] = j + q < m ? __ldg(rows + (int64_t)nj * (kH / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                acc.x = fmaf(wj[q], v[q].x, acc.x);
                acc.y = fmaf(wj[q], v[q].y, acc.y);
                acc.z = fmaf(wj[q], v[q].z, acc.z);
                acc.w = fmaf(wj[q], v[q].w, acc.w);
            }
        }
    }
    if (post) {
        const float sc = __ldg(post + r);
        acc.x *= sc;
        acc.y *= sc;
        acc.z *= sc;
        acc.w *= sc;
    }
    float4* o = reinterpret_cast<float4*>(out + r * kH) + sub;
    if (accumulate) {
        const float4 prev = *o;
        acc.x += prev.x;
        acc.y += prev.y;
        acc.z += prev.z;
        acc.w += prev.w;
    }
    *o = acc;
}

// ---- dense layers ------------------------------------------------------------------------------
// Register-tiled FP32 products on packed pairs (fma.rn.f32x2, two IEEE multiply-adds an
// instruction, so that the loads from shared memory have issue slots left).  A warp computes
// 32 x 32 outputs, a thread 8 rows x 4 columns spread so that its lanes' 16-byte reads fall into
// different banks: rows ty + 4 i, columns tx + 8 j with ty = lane / 8, tx = lane % 8 and row
// strides of 4 mod 32 floats.  Where both operands have the contraction index contiguous, a pair
// is two consecutive contraction indices (even and odd partial sums, joined at the end).
using F2 = unsigned long long;
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ F2 pack2(float lo, float hi) {
    F2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpack2(F2 v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}
struct __align__(16) F2x2 {
    F2 a, b;
};

// acc[i][j] += Σ_k A[ty + 4 i][k] B[tx + 8 j][k], k < KN
template <int KN, int LDA, int LDB, int NI>
__device__ __forceinline__ void tile_product(const float* __restrict__ A, const float* __restrict__ B, F2 (&acc)[NI][4]) {
#pragma unroll 4
    for (int k = 0; k < KN; k += 4) {
        F2x2 bv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) bv[j] = *reinterpret_cast<const F2x2*>(B + 8 * j * LDB + k);
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const F2x2 av = *reinterpret_cast<const F2x2*>(A + 4 * i * LDA + k);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fma2(av.b, bv[j].b, fma2(av.a, bv[j].a, acc[i][j]));
        }
    }
}

// 16 bytes from global to shared memory without registers; zeros where !in.
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

constexpr int kLdHm = 2 * kH + 4;  // padded row strides (4 mod 32 floats): [h | m] and W rows
constexpr int kLdDz = kH + 4;      // dh, a and dz rows, the transposed weights
constexpr int kTileRowsD = 64;     // forward
constexpr int kTileRowsB = 32;     // backward
constexpr int kFwdSmem = (kH + 2 * kTileRowsD) * kLdHm * (int)sizeof(float);
constexpr int kBwdSmem = (2 * kH * kLdDz + kTileRowsB * (2 * (2 * kLdDz + kLdHm) + kLdDz)) * (int)sizeof(float);
constexpr int kDenseBlocks = 304;  // two blocks per SM, by shared memory; each takes every 304th tile

// Rows r0 .. r0 + ROWS - 1 of h and m side by side into shared memory (zeros past the end).
template <int ROWS>
__device__ __forceinline__ void stage_hm(int64_t r0, int64_t R, const float* __restrict__ h, const float* __restrict__ m,
                                         float* __restrict__ As) {
#pragma unroll
    for (int f = threadIdx.x; f < ROWS * 32; f += kBlock) {
        const int row = f >> 5, qd = f & 31;
        const int64_t r = r0 + row < R ? r0 + row : R - 1;
        copy_async(As + row * kLdHm + 4 * qd, (qd < 16 ? h : m) + r * kH + 4 * (qd & 15), r0 + row < R);
    }
}

// One residual layer forward for tiles of rows: a = tanh([h | m] · Wᵀ + b), h' = h + a.  The
// weights stay as stored: [unit][input], W_s and W_m side by side.  The next tile is copied in
// while the current one is multiplied, and the results leave through the tile's own buffer as
// whole rows.  At 128,000 rows (BA(2000, 2), 64 instances): 96 µs -> 69 µs; bound by the reads
// from shared memory (70 % of its wavefronts, 42 % of the FP32 pipe).
__global__ void __launch_bounds__(kBlock, 2) layer_forward_kernel(int64_t R, const float* __restrict__ h,
                                                                  const float* __restrict__ m,
                                                                  const float* __restrict__ Wl, float* __restrict__ a,
                                                                  float* __restrict__ hn) {
    extern __shared__ __align__(16) float smem[];
    float* Ws = smem;  // [H][kLdHm], then two tiles [kTileRowsD][kLdHm]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = (warp >> 1) * 16 + (lane >> 3), col0 = (warp & 1) * 32 + (lane & 7);
    const int64_t step = (int64_t)gridDim.x * kTileRowsD;
    int64_t r0 = (int64_t)blockIdx.x * kTileRowsD;
    for (int f = tid; f < kH * 32; f += kBlock) {
        const int n = f >> 5, qd = f & 31;
        copy_async(Ws + n * kLdHm + 4 * qd, Wl + (qd < 16 ? 0 : kH * kH) + n * kH + 4 * (qd & 15), true);
    }
    if (r0 < R) stage_hm<kTileRowsD>(r0, R, h, m, Ws + kH * kLdHm);
    copy_commit();
    float bias[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) bias[j] = __ldg(Wl + 2 * kH * kH + col0 + 8 * j);
    for (int t = 0; r0 < R; r0 += step, ++t) {
        float* As = Ws + (kH + (t & 1) * kTileRowsD) * kLdHm;
        copy_wait();
        __syncthreads();
        if (r0 + step < R) stage_hm<kTileRowsD>(r0 + step, R, h, m, Ws + (kH + ((t + 1) & 1) * kTileRowsD) * kLdHm);
        copy_commit();
        F2 acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = pack2(bias[j], 0.f);
        tile_product<2 * kH, kLdHm, kLdHm>(As + row0 * kLdHm, Ws + col0 * kLdHm, acc);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float* row = As + (row0 + 4 * i) * kLdHm + col0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 z = unpack2(acc[i][j]);
                const float av = tanhf(z.x + z.y);
                row[8 * j] += av;
                row[kH + 8 * j] = av;
            }
        }
        __syncthreads();
#pragma unroll
        for (int f = tid; f < kTileRowsD * 32; f += kBlock) {
            const int rw = f >> 5, qd = f & 31;
            if (r0 + rw < R)
                reinterpret_cast<float4*>((qd < 16 ? hn : a) + (r0 + rw) * kH)[qd & 15] =
                    *reinterpret_cast<const float4*>(As + rw * kLdHm + 4 * qd);
        }
    }
}

// y_r = w_out · h_r + b_out, a warp per row
__global__ void decode_kernel(int64_t R, const float* __restrict__ h, const float* __restrict__ prm, int L,
                              float* __restrict__ y) {
    const int lane = threadIdx.x & 31;
    const float* w = prm + off_wout(L);
    const float b = prm[off_bout(L)];
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < R; r += warps) {
        const float2 hv = reinterpret_cast<const float2*>(h + r * kH)[lane];
        float s = fmaf(w[2 * lane], hv.x, w[2 * lane + 1] * hv.y);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) y[r] = s + b;
    }
}

// Fixed-order block sum (256 threads).
__device__ float block_sum(float v, float* red) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int off = kBlock / 2; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    const float r = red[0];
    __syncthreads();
    return r;
}

// A block per instance: θ̂ = y - mean(y) into theta (if not NULL); with a target also the
// instance's loss term (into loss_part[b]) and dy = 2 (e - mean e) / count, e = θ̂ - (t - mean t).
__global__ void __launch_bounds__(kBlock) center_loss_kernel(int64_t nv, int64_t count, const float* __restrict__ y,
                                                             const float* __restrict__ target,
                                                             float* __restrict__ theta, float* __restrict__ dy,
                                                             float* __restrict__ loss_part) {
    __shared__ float red[kBlock];
    const int64_t b = blockIdx.x;
    const float* yb = y + b * nv;
    float s = 0.f;
    for (int64_t i = threadIdx.x; i < nv; i += kBlock) s += yb[i];
    const float ym = block_sum(s, red) / (float)nv;
    if (theta)
        for (int64_t i = threadIdx.x; i < nv; i += kBlock) theta[b * nv + i] = yb[i] - ym;
    if (!target) return;
    const float* tb = target + b * nv;
    s = 0.f;
    for (int64_t i = threadIdx.x; i < nv; i += kBlock) s += tb[i];
    const float tm = block_sum(s, red) / (float)nv;
    float l = 0.f, es = 0.f;
    for (int64_t i = threadIdx.x; i < nv; i += kBlock) {
        const float e = (yb[i] - ym) - (tb[i] - tm);
        l = fmaf(e, e, l);
        es += e;
    }
    const float lsum = block_sum(l, red);
    const float em = block_sum(es, red) / (float)nv;
    for (int64_t i = threadIdx.x; i < nv; i += kBlock) {
        const float e = (yb[i] - ym) - (tb[i] - tm);
        dy[b * nv + i] = 2.f * (e - em) / (float)count;
    }
    if (threadIdx.x == 0) loss_part[b] = lsum / (float)count;
}

// ---- backward -------------------------------------------------------------------------------

// One layer backward for tiles of rows, in one pass over its activations:
//   dz = dh ⊙ (1 - a²);
//   dh += dz · W_s (the residual path already holds dh'), dmsc = (dz · W_m) ⊙ inv_s (the scaled
//   message gradient, aggregated into dh afterwards);
//   this block's partial weight gradients: [o][i] Σ dz_o h_i, [o][i] Σ dz_o m_i, then [o] Σ dz_o.
// For the last layer dh is not read but is dy_r · w_out (dy not NULL).  dz, h and m are staged
// once for both products; the weights sit transposed in shared memory; the next tile is copied
// in meanwhile, and dh and dmsc leave through the tile's buffers as whole rows.  At 128,000 rows
// the three kernels that did this (tanh, weight gradients, input gradients) took 168 µs, this
// one takes 117; bound by the reads from shared memory (70 % of its wavefronts).
__global__ void __launch_bounds__(kBlock, 2) layer_backward_kernel(
    int64_t R, const float* __restrict__ a, const float* __restrict__ h, const float* __restrict__ m,
    const float* __restrict__ Wl, const float* __restrict__ inv_s, const float* __restrict__ dy,
    const float* __restrict__ w_out, float* __restrict__ dh, float* __restrict__ dmsc, float* __restrict__ partial) {
    extern __shared__ __align__(16) float smem[];
    constexpr int kBuf = kTileRowsB * (2 * kLdDz + kLdHm);  // one tile: dh, a, [h | m]
    float* Wt = smem;                  // [2H][kLdDz]: Wt[i][o] = W_s[o][i], W_m[o][i - H]
    float* Dz = Wt + 2 * kH * kLdDz;   // [kTileRowsB][kLdDz]
    float* bufs = Dz + kTileRowsB * kLdDz;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t step = (int64_t)gridDim.x * kTileRowsB;
    int64_t r0 = (int64_t)blockIdx.x * kTileRowsB;
    auto stage = [&](int64_t rt, float* buf) {
        stage_hm<kTileRowsB>(rt, R, h, m, buf + 2 * kTileRowsB * kLdDz);
#pragma unroll
        for (int f = tid; f < kTileRowsB * 32; f += kBlock) {
            const int row = f >> 5, qd = f & 31;
            if (qd < 16 && dy) continue;
            const int64_t r = rt + row < R ? rt + row : R - 1;
            copy_async(buf + ((qd >> 4) * kTileRowsB + row) * kLdDz + 4 * (qd & 15),
                       (qd < 16 ? dh : a) + r * kH + 4 * (qd & 15), rt + row < R);
        }
    };
    if (r0 < R) stage(r0, bufs);
    copy_commit();
    for (int t = tid; t < 2 * kH * kH; t += kBlock) {
        const int o = (t / kH) & (kH - 1), i = (t & (kH - 1)) + (t >= kH * kH ? kH : 0);
        Wt[i * kLdDz + o] = __ldg(Wl + t);
    }
    // input gradients: 16 x 32 pieces of rows x inputs per warp (2 x 4 warps); weight gradients:
    // 32 x 32 pieces of units x inputs, units unit0 .. unit0 + 7 in pairs, inputs col0 + 8 j
    const int row0 = (warp >> 2) * 16 + (lane >> 3), col0 = (warp & 3) * 32 + (lane & 7);
    const int unit0 = (warp >> 2) * 32 + 8 * (lane >> 3);
    F2 gw[4][4];
    float gb = 0.f;  // unit tid & 63, rows tid >> 6, + 4, ...
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) gw[i][j] = 0;
    for (int t = 0; r0 < R; r0 += step, ++t) {
        float* Dh = bufs + (t & 1) * kBuf;
        float* Aa = Dh + kTileRowsB * kLdDz;
        float* As = Aa + kTileRowsB * kLdDz;
        copy_wait();
        __syncthreads();
        if (r0 + step < R) stage(r0 + step, bufs + ((t + 1) & 1) * kBuf);
        copy_commit();
#pragma unroll
        for (int f = tid; f < kTileRowsB * 16; f += kBlock) {
            const int row = f >> 4, qd = f & 15;
            float4 d;
            if (dy) {
                const float s = r0 + row < R ? __ldg(dy + r0 + row) : 0.f;
                const float* w = w_out + 4 * qd;
                d = make_float4(s * __ldg(w), s * __ldg(w + 1), s * __ldg(w + 2), s * __ldg(w + 3));
                *reinterpret_cast<float4*>(Dh + row * kLdDz + 4 * qd) = d;
            } else {
                d = *reinterpret_cast<const float4*>(Dh + row * kLdDz + 4 * qd);
            }
            const float4 av = *reinterpret_cast<const float4*>(Aa + row * kLdDz + 4 * qd);
            d.x *= 1.f - av.x * av.x;
            d.y *= 1.f - av.y * av.y;
            d.z *= 1.f - av.z * av.z;
            d.w *= 1.f - av.w * av.w;
            *reinterpret_cast<float4*>(Dz + row * kLdDz + 4 * qd) = d;
        }
        __syncthreads();
        // weight gradients
        const float* dzu = Dz + unit0;
        const float* hmi = As + col0;
#pragma unroll 8
        for (int row = 0; row < kTileRowsB; ++row) {
            const F2x2 d01 = *reinterpret_cast<const F2x2*>(dzu + row * kLdDz);
            const F2x2 d23 = *reinterpret_cast<const F2x2*>(dzu + row * kLdDz + 4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float v = hmi[row * kLdHm + 8 * j];
                const F2 vv = pack2(v, v);
                gw[0][j] = fma2(d01.a, vv, gw[0][j]);
                gw[1][j] = fma2(d01.b, vv, gw[1][j]);
                gw[2][j] = fma2(d23.a, vv, gw[2][j]);
                gw[3][j] = fma2(d23.b, vv, gw[3][j]);
            }
        }
#pragma unroll
        for (int row = tid >> 6; row < kTileRowsB; row += 4) gb += Dz[row * kLdDz + (tid & 63)];
        // input gradients: into dh's tile, and over the message tile
        F2 acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0;
        tile_product<kH, kLdDz, kLdDz>(Dz + row0 * kLdDz, Wt + col0 * kLdDz, acc);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = row0 + 4 * i;
            if (col0 < kH) {  // warp-uniform: inputs of h or of m
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 z = unpack2(acc[i][j]);
                    Dh[row * kLdDz + col0 + 8 * j] += z.x + z.y;
                }
            } else {
                const float sc = r0 + row < R ? __ldg(inv_s + r0 + row) : 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 z = unpack2(acc[i][j]);
                    As[row * kLdHm + col0 + 8 * j] = (z.x + z.y) * sc;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int f = tid; f < kTileRowsB * 32; f += kBlock) {
            const int row = f >> 5, qd = f & 31;
            if (r0 + row >= R) continue;
            const float* from = qd < 16 ? Dh + row * kLdDz + 4 * qd : As + row * kLdHm + 4 * qd;
            reinterpret_cast<float4*>((qd < 16 ? dh : dmsc) + (r0 + row) * kH)[qd & 15] =
                *reinterpret_cast<const float4*>(from);
        }
    }
    float* out = partial + (int64_t)blockIdx.x * kPartialStride;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 g = unpack2(gw[i][j]);
            const int c = col0 + 8 * j, o = unit0 + 2 * i;
            float* to = out + (c < kH ? c : kH * kH + c - kH);
            to[o * kH] = g.x;
            to[(o + 1) * kH] = g.y;
        }
    __syncthreads();
    Dz[tid] = gb;
    __syncthreads();
    if (tid < kH) out[2 * kH * kH + tid] = ((Dz[tid] + Dz[tid + 64]) + Dz[tid + 128]) + Dz[tid + 192];
}

// Per-block partials of the encoder's or the decoder's gradients, in one coalesced pass over the
// block's rows: thread (q, i) of a 16 x 16 block takes units 4 i .. 4 i + 3 of every 16th row.
//   encoder  dz = dh ⊙ (1 - h0²):  [o][k] Σ dz_o x_k (k < 2), then [o] Σ dz_o
//   decoder  [i] Σ dy h_i, then Σ dy
// At 128,000 rows 98 + 14 (tanh) µs -> 16 µs and 185 µs -> 12 µs: a thread per output walked the
// rows one load at a time.
template <bool kEncoder>
__global__ void __launch_bounds__(kBlock) edge_wgrad_kernel(int64_t R, const float* __restrict__ d,
                                                            const float* __restrict__ h, const float* __restrict__ x,
                                                            float* __restrict__ partial) {
    constexpr int kSums = kEncoder ? 3 : 2;
    __shared__ float4 red[kSums][16][16];
    const int64_t per = (R + gridDim.x - 1) / gridDim.x;
    const int64_t r0 = (int64_t)blockIdx.x * per, r1 = imin64(R, r0 + per);
    const int i = threadIdx.x & 15, q = threadIdx.x >> 4;
    float4 s[3] = {};
    auto add = [](float4& a, float4 v, float w) {
        a.x = fmaf(v.x, w, a.x);
        a.y = fmaf(v.y, w, a.y);
        a.z = fmaf(v.z, w, a.z);
        a.w = fmaf(v.w, w, a.w);
    };
#pragma unroll 4
    for (int64_t r = r0 + q; r < r1; r += 16) {
        const float4 hv = __ldg(reinterpret_cast<const float4*>(h + r * kH) + i);
        if constexpr (kEncoder) {
            float4 dz = __ldg(reinterpret_cast<const float4*>(d + r * kH) + i);
            dz.x *= 1.f - hv.x * hv.x;
            dz.y *= 1.f - hv.y * hv.y;
            dz.z *= 1.f - hv.z * hv.z;
            dz.w *= 1.f - hv.w * hv.w;
            const float2 xv = __ldg(reinterpret_cast<const float2*>(x) + r);
            add(s[0], dz, xv.x);
            add(s[1], dz, xv.y);
            add(s[2], dz, 1.f);
        } else {
            const float dy = __ldg(d + r);
            add(s[0], hv, dy);
            s[1].x += dy;
        }
    }
#pragma unroll
    for (int k = 0; k < kSums; ++k) red[k][q][i] = s[k];
    __syncthreads();
    if (threadIdx.x >= kH) return;
    const int o = threadIdx.x;
    float* out = partial + (int64_t)blockIdx.x * kPartialStride;
    float t[kSums] = {};
#pragma unroll
    for (int k = 0; k < kSums; ++k)
#pragma unroll
        for (int j = 0; j < 16; ++j) t[k] += reinterpret_cast<const float*>(&red[k][j][0])[o];
    if constexpr (kEncoder) {
        out[2 * o] = t[0];
        out[2 * o + 1] = t[1];
        out[2 * kH + o] = t[2];
    } else {
        out[o] = t[0];
        if (o == 0) out[kH] = t[1];
    }
}

// All gradients from their partials: g[j] = Σ_blk partial[...][blk][...].  Group 0 is the encoder,
// 1 .. L the layers, L + 1 the decoder, each with kGradBlocks partials of its own; a block takes
// 32 entries, 8 threads each with a contiguous share of the partials, joined in order (9 µs for 4
// layers; a launch per group with one thread per entry took 22 µs each).
__global__ void __launch_bounds__(kBlock) reduce_partials_kernel(int L, int64_t n, const float* __restrict__ partial,
                                                                 float* __restrict__ g) {
    __shared__ float red[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t j = (int64_t)blockIdx.x * 32 + tx;
    float s = 0.f;
    if (j < n) {
        const int64_t l = j < off_layer(0) ? 0 : imin64(1 + (j - off_layer(0)) / kPartialStride, L + 1);
        const int64_t first = l == 0 ? 0 : off_layer((int)l - 1);
        const float* p = partial + l * kGradBlocks * kPartialStride + (j - first);
        constexpr int kShare = kGradBlocks / 8;
#pragma unroll 8
        for (int b = 0; b < kShare; ++b) s += __ldg(p + (int64_t)(ty * kShare + b) * kPartialStride);
    }
    red[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && j < n) {
        s = red[0][tx];
#pragma unroll
        for (int k = 1; k < 8; ++k) s += red[k][tx];
        g[j] = s;
    }
}

// loss = Σ_b loss_part[b] in order
__global__ void sum_loss_kernel(int64_t n, const float* __restrict__ part, float* __restrict__ loss) {
    __shared__ float red[kBlock];
    float s = 0.f;
    const int64_t per = (n + kBlock - 1) / kBlock;
    for (int64_t i = threadIdx.x * per; i < imin64(n, (threadIdx.x + 1) * per); ++i) s += part[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) *loss = s;
}

// Adam (Kingma & Ba 2015, Algorithm 1) with bias corrections c1 = 1 - β1^t, c2 = 1 - β2^t.
__global__ void adam_kernel(int64_t n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

}  // namespace mpnn
}  // namespace nd

using namespace nd::mpnn;

struct nd_mpnn {
    int64_t nv = 0, ne = 0;
    int layers = 0;
    int hops = 1;  // weighted-mean steps per message (receptive field = layers * hops)
    int64_t nparams = 0;
    int device = 0;
    uint32_t* row_ptr = nullptr;  // [nv + 1] CSR over both endpoints of every edge
    int32_t* nbr = nullptr;       // [2 ne]
    int32_t* eid = nullptr;       // [2 ne]
    int32_t* order = nullptr;     // [nv] vertices by degree, descending
    float* params = nullptr;
    float* grads = nullptr;
    float* adam_m = nullptr;
    float* adam_v = nullptr;
    int64_t adam_t = 0;
    int64_t cap = 0;  // instances the activation buffers hold
    float* x = nullptr;      // [R][2]
    float* inv_s = nullptr;  // [R]
    float* h = nullptr;      // [L + 1][R][H]
    float* a = nullptr;      // [L][R][H]
    float* m = nullptr;      // [L][R][H]
    float* y = nullptr;      // [R]
    float* dy = nullptr;     // [R]
    float* dh = nullptr;     // [R][H]
    float* hop = nullptr;    // [R][H] message buffer of networks with several hops
    float* wt = nullptr;     // [cap][2 ne] K / κ by CSR incidence
    float* dmsc = nullptr;   // [R][H]
    float* partial = nullptr;    // [L + 2][kGradBlocks][kPartialStride]
    float* loss_part = nullptr;  // [cap]
};

namespace {

void free_batch(nd_mpnn* m) {
    float** bufs[] = {&m->x, &m->inv_s, &m->h, &m->a, &m->m, &m->y, &m->dy, &m->dh, &m->hop, &m->wt, &m->dmsc, &m->loss_part};
    for (float** b : bufs) {
        cudaFree(*b);
        *b = nullptr;
    }
    m->cap = 0;
}

cudaError_t ensure_batch(nd_mpnn* m, int64_t batch) {
    if (batch <= m->cap) return cudaSuccess;
    free_batch(m);
    const int64_t R = batch * m->nv;
    const int64_t L = m->layers;
    struct Want {
        float** p;
        int64_t n;
    } want[] = {{&m->x, 2 * R},          {&m->inv_s, R},         {&m->h, (L + 1) * R * kH}, {&m->a, L * R * kH},
                {&m->m, L * R * kH},     {&m->y, R},             {&m->dy, R},               {&m->dh, R * kH},
                {&m->hop, R * kH},       {&m->wt, batch * 2 * m->ne}, {&m->dmsc, R * kH},    {&m->loss_part, batch}};
    for (const Want& w : want) {
        cudaError_t err = cudaMalloc(w.p, sizeof(float) * std::max<int64_t>(w.n, 1));
        if (err != cudaSuccess) {
            free_batch(m);
            return err;
        }
    }
    m->cap = batch;
    return cudaSuccess;
}

cudaError_t set_dense_smem() {
    static std::once_flag once;
    static cudaError_t status = cudaSuccess;
    std::call_once(once, [] {
        status = cudaFuncSetAttribute(layer_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
        if (status == cudaSuccess)
            status =
                cudaFuncSetAttribute(layer_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem);
    });
    return status;
}

// One message pass over every row (see aggregate_kernel).
void aggregate(const nd_mpnn* m, int64_t R, const float* pre, const float* post, const float* in, float* out,
               int accumulate, cudaStream_t s) {
    aggregate_kernel<<<(unsigned)((R * 16 + kBlock - 1) / kBlock), kBlock, 0, s>>>(
        R, m->nv, R / m->nv, 2 * m->ne, m->order, m->row_ptr, m->nbr, m->wt, pre, post, in, out, accumulate);
}

// Forward pass over `batch` instances; with a target also the loss terms and dy.
cudaError_t forward(nd_mpnn* m, int64_t batch, const float* P, const float* K, const float* target, float* theta,
                    cudaStream_t s) {
    const int64_t R = batch * m->nv, ninc = 2 * m->ne;
    const int L = m->layers;
    cudaError_t err = set_dense_smem();
    if (err != cudaSuccess) return err;
    if (ninc > 0)
        weights_kernel<<<grid_for(batch * ninc), kBlock, 0, s>>>(batch * ninc, ninc, m->ne, m->eid, K, m->wt);
    encode_kernel<<<grid_for(R * 16), kBlock, 0, s>>>(R, m->nv, ninc, m->row_ptr, m->wt, P, m->params, m->x, m->inv_s,
                                                      m->h);
    for (int l = 0; l < L; ++l) {
        const float* hl = m->h + (int64_t)l * R * kH;
        float* ml = m->m + (int64_t)l * R * kH;
        // m = M^hops h, ping-ponging through hop and (idle in the forward pass) dmsc
        const float* src = hl;
        for (int k = 0; k < m->hops; ++k) {
            float* dst = k == m->hops - 1 ? ml : ((k & 1) ? m->dmsc : m->hop);
            aggregate(m, R, nullptr, m->inv_s, src, dst, 0, s);
            src = dst;
        }
        layer_forward_kernel<<<(unsigned)std::min<int64_t>((R + kTileRowsD - 1) / kTileRowsD, kDenseBlocks), kBlock, kFwdSmem,
                               s>>>(
            R, hl, ml, m->params + off_layer(l), m->a + (int64_t)l * R * kH, m->h + (int64_t)(l + 1) * R * kH);
    }
    decode_kernel<<<grid_for(R * 32), kBlock, 0, s>>>(R, m->h + (int64_t)L * R * kH, m->params, L, m->y);
    center_loss_kernel<<<(unsigned)batch, kBlock, 0, s>>>(m->nv, R, m->y, target, theta, m->dy, m->loss_part);
    return cudaGetLastError();
}

// Backward pass after forward() with a target: gradients into m->grads.
cudaError_t backward(nd_mpnn* m, int64_t batch, cudaStream_t s) {
    const int64_t R = batch * m->nv;
    const int L = m->layers;
    auto partial = [&](int group) { return m->partial + (int64_t)group * kGradBlocks * kPartialStride; };
    edge_wgrad_kernel<false><<<kGradBlocks, kBlock, 0, s>>>(R, m->dy, m->h + (int64_t)L * R * kH, nullptr,
                                                            partial(L + 1));
    for (int l = L - 1; l >= 0; --l) {
        layer_backward_kernel<<<kGradBlocks, kBlock, kBwdSmem, s>>>(
            R, m->a + (int64_t)l * R * kH, m->h + (int64_t)l * R * kH, m->m + (int64_t)l * R * kH,
            m->params + off_layer(l), m->inv_s, l == L - 1 ? m->dy : nullptr, m->params + off_wout(L), m->dh, m->dmsc,
            partial(l + 1));
        // dh += (Mᵀ)^hops dm with Mᵀ x = A (x / s) (the weights are symmetric); dmsc already
        // holds dm / s
        const float* src = m->dmsc;
        for (int k = 0; k < m->hops; ++k) {
            const bool last = k == m->hops - 1;
            float* dst = last ? m->dh : ((k & 1) ? m->dmsc : m->hop);
            aggregate(m, R, k == 0 ? nullptr : m->inv_s, nullptr, src, dst, last ? 1 : 0, s);
            src = dst;
        }
    }
    edge_wgrad_kernel<true><<<kGradBlocks, kBlock, 0, s>>>(R, m->dh, m->h, m->x, partial(0));
    reduce_partials_kernel<<<(unsigned)((m->nparams + 31) / 32), kBlock, 0, s>>>(L, m->nparams, m->partial, m->grads);
    return cudaGetLastError();
}

uint64_t splitmix64(uint64_t& state) {
    uint64_t z = (state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Glorot-uniform weights (scaled by 1/2 on the residual layers), zero biases.
std::vector<float> init_params(int L, uint64_t seed) {
    std::vector<float> p((size_t)num_params(L), 0.f);
    uint64_t st = seed;
    auto fill = [&](int64_t off, int64_t n, int fan_in, int fan_out, float gain) {
        const double a = gain * std::sqrt(6.0 / (fan_in + fan_out));
        for (int64_t k = 0; k < n; ++k) {
            const double u01 = (double)(splitmix64(st) >> 11) * (1.0 / 9007199254740992.0);
            p[(size_t)(off + k)] = (float)((2.0 * u01 - 1.0) * a);
        }
    };
    fill(off_win(), 2 * kH, 2, kH, 1.f);
    for (int l = 0; l < L; ++l) {
        fill(off_layer(l), kH * kH, kH, kH, 0.5f);
        fill(off_layer(l) + kH * kH, kH * kH, kH, kH, 0.5f);
    }
    fill(off_wout(L), kH, kH, 1, 1.f);
    return p;
}

void destroy(nd_mpnn* m) {
    if (!m) return;
    free_batch(m);
    cudaFree(m->row_ptr);
    cudaFree(m->nbr);
    cudaFree(m->eid);
    cudaFree(m->order);
    cudaFree(m->params);
    cudaFree(m->grads);
    cudaFree(m->adam_m);
    cudaFree(m->adam_v);
    cudaFree(m->partial);
    delete m;
}

}  // namespace

extern "C" {

int nd_mpnn_create(int64_t nv, int64_t ne, const int64_t* src, const int64_t* dst, int layers, int hidden,
                   uint64_t seed, nd_mpnn** out) {
    nd::clear_error();
    if (!out) return nd::fail(ND_ERR_ARG, "nd_mpnn_create: out is NULL");
    *out = nullptr;
    if (nv <= 0 || ne < 0 || (ne > 0 && (!src || !dst)))
        return nd::fail(ND_ERR_ARG, "nd_mpnn_create: need nv > 0 and src / dst for ne > 0");
    if (hidden != kH) return nd::fail(ND_ERR_UNSUPPORTED, "nd_mpnn_create: the hidden width must be 64");
    if (layers < 1 || layers > 16) return nd::fail(ND_ERR_ARG, "nd_mpnn_create: layers must be in 1..16");
    if (nv > INT32_MAX || 2 * ne > UINT32_MAX) return nd::fail(ND_ERR_ARG, "nd_mpnn_create: graph too large");
    std::vector<uint32_t> rp((size_t)nv + 1, 0);
    for (int64_t e = 0; e < ne; ++e) {
        if (src[e] < 0 || src[e] >= nv || dst[e] < 0 || dst[e] >= nv)
            return nd::fail(ND_ERR_ARG, "nd_mpnn_create: edge endpoint out of range");
        ++rp[(size_t)src[e] + 1];
        ++rp[(size_t)dst[e] + 1];
    }
    for (int64_t v = 0; v < nv; ++v) rp[(size_t)v + 1] += rp[(size_t)v];
    std::vector<int32_t> nbr((size_t)(2 * ne)), eid((size_t)(2 * ne));
    std::vector<uint32_t> fillp(rp.begin(), rp.end() - 1);
    for (int64_t e = 0; e < ne; ++e) {
        const uint32_t a = fillp[(size_t)dst[e]]++;
        nbr[a] = (int32_t)src[e];
        eid[a] = (int32_t)e;
        const uint32_t b = fillp[(size_t)src[e]]++;
        nbr[b] = (int32_t)dst[e];
        eid[b] = (int32_t)e;
    }
    std::vector<int32_t> order((size_t)nv);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
        return rp[(size_t)x + 1] - rp[(size_t)x] > rp[(size_t)y + 1] - rp[(size_t)y];
    });
    nd_mpnn* m = new nd_mpnn();
    m->nv = nv;
    m->ne = ne;
    m->layers = layers;
    m->nparams = num_params(layers);
    cudaGetDevice(&m->device);
    const std::vector<float> p0 = init_params(layers, seed);
    cudaError_t err;
    const size_t pb = sizeof(float) * (size_t)m->nparams;
    if ((err = cudaMalloc(&m->row_ptr, sizeof(uint32_t) * rp.size())) != cudaSuccess ||
        (err = cudaMalloc(&m->nbr, sizeof(int32_t) * std::max<size_t>(nbr.size(), 1))) != cudaSuccess ||
        (err = cudaMalloc(&m->eid, sizeof(int32_t) * std::max<size_t>(eid.size(), 1))) != cudaSuccess ||
        (err = cudaMalloc(&m->order, sizeof(int32_t) * order.size())) != cudaSuccess ||
        (err = cudaMemcpy(m->order, order.data(), sizeof(int32_t) * order.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (err = cudaMalloc(&m->params, pb)) != cudaSuccess || (err = cudaMalloc(&m->grads, pb)) != cudaSuccess ||
        (err = cudaMalloc(&m->adam_m, pb)) != cudaSuccess || (err = cudaMalloc(&m->adam_v, pb)) != cudaSuccess ||
        (err = cudaMalloc(&m->partial, sizeof(float) * (size_t)(layers + 2) * kGradBlocks * kPartialStride)) != cudaSuccess ||
        (err = cudaMemcpy(m->row_ptr, rp.data(), sizeof(uint32_t) * rp.size(), cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (err = cudaMemcpy(m->nbr, nbr.data(), sizeof(int32_t) * nbr.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (err = cudaMemcpy(m->eid, eid.data(), sizeof(int32_t) * eid.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (err = cudaMemcpy(m->params, p0.data(), pb, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (err = cudaMemset(m->grads, 0, pb)) != cudaSuccess || (err = cudaMemset(m->adam_m, 0, pb)) != cudaSuccess ||
        (err = cudaMemset(m->adam_v, 0, pb)) != cudaSuccess) {
        destroy(m);
        return nd::cuda_fail(err, "nd_mpnn_create");
    }
    *out = m;
    return ND_OK;
}

int nd_mpnn_destroy(nd_mpnn* m) {
    nd::clear_error();
    destroy(m);
    return ND_OK;
}

int nd_mpnn_num_params(const nd_mpnn* m, int64_t* n) {
    nd::clear_error();
    if (!m || !n) return nd::fail(ND_ERR_ARG, "nd_mpnn_num_params: NULL argument");
    *n = m->nparams;
    return ND_OK;
}

int nd_mpnn_get_params(const nd_mpnn* m, float* dst, void* stream) {
    nd::clear_error();
    if (!m || !dst) return nd::fail(ND_ERR_ARG, "nd_mpnn_get_params: NULL argument");
    cudaError_t err = cudaMemcpyAsync(dst, m->params, sizeof(float) * (size_t)m->nparams, cudaMemcpyDefault,
                                      (cudaStream_t)stream);
    return err == cudaSuccess ? ND_OK : nd::cuda_fail(err, "nd_mpnn_get_params");
}

int nd_mpnn_set_params(nd_mpnn* m, const float* src, void* stream) {
    nd::clear_error();
    if (!m || !src) return nd::fail(ND_ERR_ARG, "nd_mpnn_set_params: NULL argument");
    cudaError_t err = cudaMemcpyAsync(m->params, src, sizeof(float) * (size_t)m->nparams, cudaMemcpyDefault,
                                      (cudaStream_t)stream);
    return err == cudaSuccess ? ND_OK : nd::cuda_fail(err, "nd_mpnn_set_params");
}

int nd_mpnn_get_grads(const nd_mpnn* m, float* dst, void* stream) {
    nd::clear_error();
    if (!m || !dst) return nd::fail(ND_ERR_ARG, "nd_mpnn_get_grads: NULL argument");
    cudaError_t err = cudaMemcpyAsync(dst, m->grads, sizeof(float) * (size_t)m->nparams, cudaMemcpyDefault,
                                      (cudaStream_t)stream);
    return err == cudaSuccess ? ND_OK : nd::cuda_fail(err, "nd_mpnn_get_grads");
}

int nd_mpnn_forward(nd_mpnn* m, int64_t batch, const float* P, const float* K, float* theta, void* stream) {
    ND_NVTX("nd_mpnn_forward");
    nd::clear_error();
    if (!m || batch <= 0 || !P || (m->ne > 0 && !K) || !theta)
        return nd::fail(ND_ERR_ARG, "nd_mpnn_forward: bad arguments");
    cudaError_t err = ensure_batch(m, batch);
    if (err != cudaSuccess) return nd::fail(ND_ERR_NOMEM, "nd_mpnn_forward: activation buffers");
    err = forward(m, batch, P, K, nullptr, theta, (cudaStream_t)stream);
    return err == cudaSuccess ? ND_OK : nd::cuda_fail(err, "nd_mpnn_forward");
}

int nd_mpnn_loss_grad(nd_mpnn* m, int64_t batch, const float* P, const float* K, const float* theta_star, float* loss,
                      void* stream) {
    ND_NVTX("nd_mpnn_loss_grad");
    nd::clear_error();
    if (!m || batch <= 0 || !P || (m->ne > 0 && !K) || !theta_star || !loss)
        return nd::fail(ND_ERR_ARG, "nd_mpnn_loss_grad: bad arguments");
    cudaError_t err = ensure_batch(m, batch);
    if (err != cudaSuccess) return nd::fail(ND_ERR_NOMEM, "nd_mpnn_loss_grad: activation buffers");
    cudaStream_t s = (cudaStream_t)stream;
    if ((err = forward(m, batch, P, K, theta_star, nullptr, s)) != cudaSuccess ||
        (err = backward(m, batch, s)) != cudaSuccess)
        return nd::cuda_fail(err, "nd_mpnn_loss_grad");
    sum_loss_kernel<<<1, kBlock, 0, s>>>(batch, m->loss_part, loss);
    err = cudaGetLastError();
    return err == cudaSuccess ? ND_OK : nd::cuda_fail(err, "nd_mpnn_loss_grad");
}

int nd_mpnn_adam(nd_mpnn* m, double lr, double beta1, double beta2, double eps, void* stream) {
    ND_NVTX("nd_mpnn_adam");
    nd::clear_error();
    if (!m || !(lr > 0) || !(beta1 >= 0 && beta1 < 1) || !(beta2 >= 0 && beta2 < 1) || !(eps > 0))
        return nd::fail(ND_ERR_ARG, "nd_mpnn_adam: bad arguments");
    ++m->adam_t;
    const double c1 = 1.0 - std::pow(beta1, (double)m->adam_t), c2 = 1.0 - std::pow(beta2, (double)m->adam_t);
    adam_kernel<<<grid_for(m->nparams), kBlock, 0, (cudaStream_t)stream>>>(
        m->nparams, m->params, m->grads, m->adam_m, m->adam_v, (float)lr, (float)beta1, (float)beta2, (float)eps,
        (float)c1, (float)c2);
    cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? ND_OK : nd::cuda_fail(err, "nd_mpnn_adam");
}

int nd_mpnn_set_hops(nd_mpnn* m, int hops) {
    nd::clear_error();
    if (!m || hops < 1 || hops > 64) return nd::fail(ND_ERR_ARG, "nd_mpnn_set_hops: hops must be in 1..64");
    m->hops = hops;
    return ND_OK;
}

int nd_mpnn_reset_optimizer(nd_mpnn* m, void* stream) {
    nd::clear_error();
    if (!m) return nd::fail(ND_ERR_ARG, "nd_mpnn_reset_optimizer: NULL handle");
    m->adam_t = 0;
    const size_t pb = sizeof(float) * (size_t)m->nparams;
    cudaError_t err = cudaMemsetAsync(m->adam_m, 0, pb, (cudaStream_t)stream);
    if (err == cudaSuccess) err = cudaMemsetAsync(m->adam_v, 0, pb, (cudaStream_t)stream);
    return err == cudaSuccess ? ND_OK : nd::cuda_fail(err, "nd_mpnn_reset_optimizer");
}

}  // extern "C"
