// Analytic Jacobian-vector product of the network RHS, jv = (∂f/∂u)(u, p) · v.
//
// The reference differentiates the core loop with ForwardDiff (Dual numbers through
// src/coreloop.jl, cache promotion at :10-21; tested against finite differences in
// test/AD_test.jl:54-60).  For the library components the derivative is written out:
//   diffusion edge    d[w (u_s - u_d)]      = w (v_s - v_d)
//   unit diffusion    d[u_s - u_d]          = v_s - v_d
//   kuramoto / line   d[K sin(θ_s - θ_d)]   = K cos(θ_s - θ_d) (v_s - v_d)
// and AntiSymmetric hands -d(y_dst) to the source, so at row v with neighbour n every
// incidence contributes c (v_n - v_v) with c = w, 1 or K cos(θ_n - θ_v).  Vertices:
//   diffusion / kuramoto   jv = Σ                  swing   jv_θ = v_ω,  jv_ω = (Σ - D v_ω) / M
// One launch over the slot-ordered CSR (rows by degree, the longest first): a block per row of
// kJvpBlockMin terms and more, a warp per row above 32, a thread per row for the rest, which
// sums in edge order.  A row is bound by the latency of its gathers (the neighbour, then its
// state, direction and line weight), so each thread asks for four terms at a time, and the
// longest rows start first and are split widest: as two launches with a warp for the longest
// row, BA(5e5, 2) swing took 126 + 50 µs, now 41; a block from 256 terms on (two round
// trips for a warp, one for the block).
#include "nd_components.cuh"
#include "nd_internal.h"

namespace nd {

int jacobian_times(nd_handle* h, void* jv, const void* u, const void* p, const void* v, cudaStream_t s);

namespace {

template <typename T, int VK>
__device__ __forceinline__ void jvp_vertex(int64_t v, T acc, const T* __restrict__ pv, const T* __restrict__ vv,
                                           T* __restrict__ jv) {
    using A = Arith<T>;
    if constexpr (VK == ND_V_SWING) {
        const T M = pv[3 * v], D = pv[3 * v + 1];
        jv[2 * v] = vv[2 * v + 1];
        jv[2 * v + 1] = A::div(A::sub(acc, A::mul(D, vv[2 * v + 1])), M);
    } else {
        jv[v] = acc;
    }
}

// Blocks of 128, eight to an SM (64 registers): a block's slots are free again sooner where its rows
// differ in length.  BA(n, k) swing, FP64, against blocks of 256 at the 72 registers the kernel
// takes uncapped, µs: (5e5, 2) 41.0 / 47.4, (2e5, 4) 37.1 / 43.0, (5e3, 2) 20.7 / 22.6; 256 by 4
// 45.2, 128 by 10 44.6, 64 by 16 41.3 on the first.
constexpr int kJvpBlock = 128;

// Σ over the terms k, k + step, ... < end of a row, four in flight.
template <typename T, int VK, int EK>
__device__ __forceinline__ T jvp_sum(uint32_t k, uint32_t end, uint32_t step, const int2* __restrict__ incid, T uv, T dv,
                                     const T* __restrict__ u, const T* __restrict__ pe, const T* __restrict__ vv) {
    using A = Arith<T>;
    constexpr int DV = VertexDims<VK>::dim;
    constexpr int kB = 4;
    T acc = T(0);
    for (; k < end; k += kB * step) {
        int2 inc[kB];
        T un[kB], dn[kB], w[kB];
#pragma unroll
        for (int j = 0; j < kB; ++j) inc[j] = k + j * step < end ? __ldg(incid + k + j * step) : int2{-1, 0};
#pragma unroll
        for (int j = 0; j < kB; ++j) {
            un[j] = dn[j] = w[j] = T(0);
            if (inc[j].x < 0) continue;
            const int64_t n = (int64_t)inc[j].x * DV;
            un[j] = EK == ND_E_KURAMOTO ? __ldg(u + n) : T(0);
            dn[j] = __ldg(vv + n);
            w[j] = EK == ND_E_DIFFUSION_UNIT ? T(1) : __ldg(pe + (inc[j].y & 0x7fffffff));
        }
#pragma unroll
        for (int j = 0; j < kB; ++j) {
            if (inc[j].x < 0) continue;
            const T c = EK == ND_E_KURAMOTO ? A::times_cos(w[j], A::sub(un[j], uv)) : w[j];
            acc = A::add(acc, EK == ND_E_DIFFUSION_UNIT ? A::sub(dn[j], dv) : A::mul(c, A::sub(dn[j], dv)));
        }
    }
    return acc;
}

template <typename T, int VK, int EK>
__global__ void __launch_bounds__(kJvpBlock, 8) jvp_kernel(int64_t n_block, int64_t n_long, int64_t nv,
                                                           const uint32_t* __restrict__ slot_ptr,
                                                           const int32_t* __restrict__ slot_vertex,
                                                           const int2* __restrict__ incid, const T* __restrict__ u,
                                                           const T* __restrict__ p, const T* __restrict__ vv,
                                                           T* __restrict__ jv) {
    using A = Arith<T>;
    constexpr int DV = VertexDims<VK>::dim;
    constexpr int kWarps = kJvpBlock / 32;
    const T* pe = p + nv * VertexDims<VK>::pdim;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t b = blockIdx.x, warp_blocks = (n_long - n_block + kWarps - 1) / kWarps;
    // how many lanes share a row: the block, a warp, or one
    const int share = b < n_block ? kJvpBlock : (b < n_block + warp_blocks ? 32 : 1);
    const int64_t s = share == kJvpBlock ? b
                      : share == 32      ? n_block + (b - n_block) * kWarps + warp
                                         : n_long + (b - n_block - warp_blocks) * kJvpBlock + tid;
    if (s >= (share == 32 ? n_long : nv)) return;  // never for a block's row: warp-uniform where a warp shares
    const int64_t v = __ldg(slot_vertex + s);
    const T uv = __ldg(u + v * DV), dv = __ldg(vv + v * DV);
    const int first = share == kJvpBlock ? tid : (share == 32 ? lane : 0);
    T acc = jvp_sum<T, VK, EK>(__ldg(slot_ptr + s) + first, __ldg(slot_ptr + s + 1), share, incid, uv, dv, u, pe, vv);
    if (share > 1) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc = A::add(acc, __shfl_xor_sync(0xffffffffu, acc, off));
        if (share == kJvpBlock) {
            __shared__ T red[kWarps];
            if (lane == 0) red[warp] = acc;
            __syncthreads();
            acc = red[0];
#pragma unroll
            for (int w = 1; w < kWarps; ++w) acc = A::add(acc, red[w]);
        }
    }
    if (first == 0) jvp_vertex<T, VK>(v, acc, p, vv, jv);
}

template <typename T>
cudaError_t launch_jvp(const nd_handle* h, const void* u, const void* p, const void* v, void* jv, cudaStream_t s) {
    const Topology& t = h->topo;
    const int64_t n_long = (int64_t)t.n_heavy + t.n_medium;  // the first slots: degree > 32
    const int64_t n_block = t.n_jvp_block, warps = kJvpBlock / 32;
    const unsigned grid = (unsigned)(n_block + (n_long - n_block + warps - 1) / warps +
                                     (t.nv - n_long + kJvpBlock - 1) / kJvpBlock);
    const int2* inc = reinterpret_cast<const int2*>(t.incid);
#define ND_CASE(VK, EK)                                                                                          \
    if (h->vertex_kind == VK && h->edge_kind == EK) {                                                             \
        jvp_kernel<T, VK, EK><<<grid, kJvpBlock, 0, s>>>(n_block, n_long, t.nv, t.slot_ptr, t.slot_vertex, inc,   \
                                                         static_cast<const T*>(u), static_cast<const T*>(p),      \
                                                         static_cast<const T*>(v), static_cast<T*>(jv));          \
        return cudaGetLastError();                                                                                \
    }
    ND_CASE(ND_V_DIFFUSION, ND_E_DIFFUSION)
    ND_CASE(ND_V_DIFFUSION, ND_E_DIFFUSION_UNIT)
    ND_CASE(ND_V_DIFFUSION, ND_E_KURAMOTO)
    ND_CASE(ND_V_KURAMOTO, ND_E_DIFFUSION)
    ND_CASE(ND_V_KURAMOTO, ND_E_DIFFUSION_UNIT)
    ND_CASE(ND_V_KURAMOTO, ND_E_KURAMOTO)
    ND_CASE(ND_V_SWING, ND_E_DIFFUSION)
    ND_CASE(ND_V_SWING, ND_E_DIFFUSION_UNIT)
    ND_CASE(ND_V_SWING, ND_E_KURAMOTO)
#undef ND_CASE
    return cudaErrorInvalidValue;
}

}  // namespace

}  // namespace nd

using namespace nd;

extern "C" int nd_jvp(nd_handle* h, int dtype, void* jv, const void* u, const void* p, const void* v, double t,
                      void* stream) {
    ND_NVTX("nd_jvp");
    (void)t;
    clear_error();
    if (!h || !jv || !u || !v) return fail(ND_ERR_ARG, "nd_jvp: NULL argument");
    if (dtype != h->dtype) return fail(ND_ERR_DTYPE, "nd_jvp: element type differs from the handle's");
    if (h->pdim > 0 && !p) return fail(ND_ERR_ARG, "nd_jvp: p is NULL");
    if (h->batched.enabled) return jacobian_times(h, jv, u, p, v, (cudaStream_t)stream);
    cudaError_t err = h->dtype == ND_F64 ? launch_jvp<double>(h, u, p, v, jv, (cudaStream_t)stream)
                                         : launch_jvp<float>(h, u, p, v, jv, (cudaStream_t)stream);
    return err == cudaSuccess ? ND_OK : cuda_fail(err, "nd_jvp");
}
