// Fused network right-hand side over the destination-sorted CSR.
//
// One RHS replaces the reference's phased core loop (src/coreloop.jl:22-101): vertex g,
// edge g/f, the gather of vertex outputs into edge inputs (src/gbufs.jl:7-25), the
// aggregation (src/aggregators.jl:133-151) and vertex f.  Vertex outputs are the first
// state (StateMask(1)), so edges read u directly; edge values live in registers or shared
// memory; each row is summed in ascending edge id, the SequentialAggregator order; du is
// written once.  There are no output, gather or aggregation buffers.
//
// One launch, two roles chosen per block (degree buckets and slot order: nd_internal.h):
//   heavy   (FP32) a block per row, which sums thread-strided slices with Kahan compensation and
//           joins them in a fixed tree;
//   window  a block per window of rows: phase A evaluates the window's edge terms, one
//           incidence per thread (coalesced incidence loads, independent gathers and FP64
//           operations in flight) into shared memory; phase B sums one row per thread.
// Heavy blocks come first so the long rows start early.  FP64 heavy rows, and the longest FP32
// ones, have a kernel of their own (heavy_solo_kernel) beside this one.
//
// Cache policy: u is gathered at random and is re-read by every incidence, so its loads
// ask L2 to keep the lines (evict_last); the incidence stream and the edge parameters are
// read once per side and ask to be evicted first.
//
// FP64 on GB300 retires ~2 lanes/clock/SM and a DADD holds its sub-partition's FP64 pipe
// for a full warp even with one lane active.  Window rows (at most kMediumMaxDeg long)
// add with hardware DADDs, all lanes busy on rows of similar length.  A hub's sum would
// be a chain of thousands of DADDs on one sub-partition, so it runs on the integer pipes, by the
// block-wide exact scan (nd_scan.cuh), whose result equals the sequential sum bit for bit.

#include "nd_components.cuh"
#include "nd_exact.cuh"
#include "nd_internal.h"
#include "nd_scan.cuh"

namespace nd {

namespace {

using namespace dev;

// Shared memory of one block: a window's (a row's block needs a few words of it).
template <typename T>
struct Smem {
    static constexpr int kBytes = (kWindowIncidences + kWindow) * (int)sizeof(T) + kWindowIncidences;
};

// ---- heavy: a block per row (FP32, and FP64 in the tree mode) ------------------------------
template <typename T, int VK, int EK>
__device__ __forceinline__ void block_row(const RhsArgs& a, int slot, unsigned char* smem) {
    using A = Arith<T>;
    constexpr int DV = VertexDims<VK>::dim;
    const T* __restrict__ u = static_cast<const T*>(a.u);
    const T* __restrict__ p = static_cast<const T*>(a.p);
    const T* __restrict__ pe = p + a.nv * VertexDims<VK>::pdim;
    const int2* __restrict__ incid = reinterpret_cast<const int2*>(a.incid);
    const uint64_t keep = policy_evict_last(), stream = policy_evict_first();
    const int64_t v = __ldg(a.slot_vertex + slot);
    const uint32_t beg = __ldg(a.slot_ptr + slot), end = __ldg(a.slot_ptr + slot + 1);
    const T uv = __ldg(u + v * DV);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    T* red = reinterpret_cast<T*>(smem);
    T acc = T(0), comp = T(0);
#pragma unroll 4
    for (uint32_t k = beg + tid; k < end; k += kBlock) {
        const int2 inc = ld_hint(incid + k, stream);
        const T un = ld_hint(u + (int64_t)inc.x * DV, keep);
        const T w = edge_param<T, EK>(pe, inc.y & 0x7fffffff, stream);
        const T term = incidence_term_w<T, EK>(uv, un, w, inc.y < 0);
        if constexpr (sizeof(T) == 4) {
            const T y = A::sub(term, comp);
            const T s = A::add(acc, y);
            comp = A::sub(A::sub(s, acc), y);
            acc = s;
        } else {
            acc = A::add(acc, term);
        }
    }
    if constexpr (sizeof(T) == 4) acc = A::sub(acc, comp);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc = A::add(acc, __shfl_xor_sync(kFull, acc, off));
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (tid == 0) {
        T s = red[0];
#pragma unroll
        for (int w = 1; w < kWarpsPerBlock; ++w) s = A::add(s, red[w]);
        vertex_f<T, VK>(static_cast<T*>(a.du), u, p, v, s);
    }
}

// ---- windows: a block per window of rows ----------------------------------------------------
// Up to this many rows above kLightMaxDeg terms in 32 rows are marked by the warp, one after the
// other; more by a thread each.  FP32, BA(1e5, 2) diffusion / swing, µs: always by the warp 12.6 / 14.6,
// up to 12 10.4 / 11.6, up to 4 8.5 / 10.4 (never 8.4 / 10.4); a complete graph of 300, FP64, 17.5
// by the warp and 18.6 by a thread.
constexpr int kMarkTogether = 4;

template <typename T, int VK, int EK>
__device__ __forceinline__ void window_block(const RhsArgs& a, int win, unsigned char* smem) {
    using A = Arith<T>;
    constexpr int DV = VertexDims<VK>::dim;
    const T* __restrict__ u = static_cast<const T*>(a.u);
    const T* __restrict__ p = static_cast<const T*>(a.p);
    const T* __restrict__ pe = p + a.nv * VertexDims<VK>::pdim;
    const int2* __restrict__ incid = reinterpret_cast<const int2*>(a.incid);
    T* s_term = reinterpret_cast<T*>(smem);                        // [kWindowIncidences]
    T* s_uv = s_term + kWindowIncidences;                          // [kWindow]
    uint8_t* s_owner = reinterpret_cast<uint8_t*>(s_uv + kWindow);  // [kWindowIncidences]
    const uint64_t keep = policy_evict_last(), stream = policy_evict_first();
    const int first = a.n_heavy;
    const int slot0 = first + __ldg(a.win_ptr + win), slot1 = first + __ldg(a.win_ptr + win + 1);
    const uint32_t i0 = __ldg(a.slot_ptr + slot0), i1 = __ldg(a.slot_ptr + slot1);
    const int n = (int)(i1 - i0);  // <= kWindowIncidences
    const int tid = threadIdx.x;
    // phase 0: each row's vertex value and the owner (row) of each incidence
    const int s = slot0 + tid;
    const bool has_row = s < slot1;
    int64_t v = 0;
    int beg = 0, end = 0;
    if (has_row) {
        v = __ldg(a.slot_vertex + s);
        beg = (int)(__ldg(a.slot_ptr + s) - i0);
        end = (int)(__ldg(a.slot_ptr + s + 1) - i0);
        s_uv[tid] = ld_hint(u + v * DV, keep);
    }
    // where a warp has few long rows it marks their incidences together; many, each its own
    unsigned shared_rows = __ballot_sync(kFull, end - beg > kLightMaxDeg);
    if (__popc(shared_rows) > kMarkTogether) shared_rows = 0;
    if (!((shared_rows >> (tid & 31)) & 1u))
        for (int j = beg; j < end; ++j) s_owner[j] = (uint8_t)tid;
    for (unsigned m = shared_rows; m; m &= m - 1) {
        const int l = __ffs(m) - 1, e = __shfl_sync(kFull, end, l);
        for (int j = __shfl_sync(kFull, beg, l) + (tid & 31); j < e; j += 32) s_owner[j] = (uint8_t)((tid & ~31) + l);
    }
    __syncthreads();
    // phase A: the edge terms, one incidence per thread: coalesced incidence loads, many
    // independent gathers and FP64 operations in flight
#pragma unroll 4
    for (int k = tid; k < n; k += kBlock) {
        const int2 inc = ld_hint(incid + i0 + k, stream);
        const T un = ld_hint(u + (int64_t)inc.x * DV, keep);
        const T w = edge_param<T, EK>(pe, inc.y & 0x7fffffff, stream);
        s_term[k] = incidence_term_w<T, EK>(s_uv[s_owner[k]], un, w, inc.y < 0);
    }
    __syncthreads();
    // phase B: one row per thread, in edge order.  FP64: hardware adds (a row is at most
    // kMediumMaxDeg long; one DADD per term is cheaper than the ~100 integer operations
    // of an emulated add).  FP32: compensated sums on the rows above kLightMaxDeg.
    if (!has_row) return;
    T acc = T(0);
    if constexpr (sizeof(T) == 8) {
        for (int j = beg; j < end; ++j) acc = __dadd_rn(acc, s_term[j]);
    } else {
        if (end - beg > kLightMaxDeg) {
            T comp = T(0);
            for (int j = beg; j < end; ++j) {
                const T y = A::sub(s_term[j], comp);
                const T t = A::add(acc, y);
                comp = A::sub(A::sub(t, acc), y);
                acc = t;
            }
            acc = A::sub(acc, comp);
        } else {
            for (int j = beg; j < end; ++j) acc = A::add(acc, s_term[j]);
        }
    }
    vertex_f<T, VK>(static_cast<T*>(a.du), u, p, v, acc);
}

template <typename T, int VK, int EK>
__global__ void __launch_bounds__(kBlock, 8) rhs_kernel(RhsArgs a) {
    __shared__ __align__(16) unsigned char smem[Smem<T>::kBytes];
    const int b = blockIdx.x;
    if constexpr (sizeof(T) == 4) {
        const int nh = a.n_heavy - a.n_apart;
        if (b < nh) block_row<T, VK, EK>(a, a.n_apart + b, smem);
        else window_block<T, VK, EK>(a, b - nh, smem);
    } else {  // FP64 heavy rows are all launched apart
        window_block<T, VK, EK>(a, b, smem);
    }
}

// Heavy rows alone, a block per row.  The FP32 and tree rows ask for most of an SM's shared
// memory, which keeps all but four other blocks off the SM: the row's summation chain is
// serial, and on a crowded SM each of its steps waits for other blocks' instructions.
constexpr int kHeavySoloSmem = 160 * 1024;

// S + the n terms of `tile` (tile_at layout) by hardware adds, in order: a chain of dependent adds
// (63 clocks each on an SM without other FP64 work), so the next sixteen terms are read from shared
// memory while sixteen are added.
__device__ __forceinline__ double chain_sum(double S, const double* __restrict__ tile, int n) {
    constexpr int kB = 16;
    double cur[kB], nxt[kB];
    const int full = n / kB * kB;
    if (full > 0) {
#pragma unroll
        for (int k = 0; k < kB; ++k) cur[k] = tile[tile_at(k)];
    }
    for (int i = 0; i < full; i += kB) {
        const int j = min(i + kB, full - kB);
#pragma unroll
        for (int k = 0; k < kB; ++k) nxt[k] = tile[tile_at(j + k)];
#pragma unroll
        for (int k = 0; k < kB; ++k) S = __dadd_rn(S, cur[k]);
#pragma unroll
        for (int k = 0; k < kB; ++k) cur[k] = nxt[k];
    }
    for (int i = full; i < n; ++i) S = __dadd_rn(S, tile[tile_at(i)]);
    return S;
}

// FP64 sequential sum of a heavy row by one block: tiles of kScanTile terms, each added by the
// block-wide exact scan (or the hardware DADD chain in the native mode).  A thread's incidence
// data of the next tile are in flight while the current tile is added.
template <int VK, int EK, int MODE>
__device__ __forceinline__ void solo_row_fp64(const RhsArgs& a, int slot, double* tile, BlockScanShared& sh) {
    constexpr int DV = VertexDims<VK>::dim;
    const double* __restrict__ u = static_cast<const double*>(a.u);
    const double* __restrict__ p = static_cast<const double*>(a.p);
    const double* __restrict__ pe = p + a.nv * VertexDims<VK>::pdim;
    const int2* __restrict__ incid = reinterpret_cast<const int2*>(a.incid);
    const uint64_t keep = policy_evict_last(), stream = policy_evict_first();
    const int64_t v = __ldg(a.slot_vertex + slot);
    const uint32_t beg = __ldg(a.slot_ptr + slot), end = __ldg(a.slot_ptr + slot + 1);
    const double uv = __ldg(u + v * DV);
    const int tid = threadIdx.x;
    double un[kBlockPer], w[kBlockPer];
    unsigned src_side = 0;
    auto load = [&](uint32_t base) {  // positions tid, tid + kScanThreads, ...: coalesced
        src_side = 0;
#pragma unroll
        for (int k = 0; k < kBlockPer; ++k) {
            const uint32_t i = base + (uint32_t)(tid + k * kScanThreads);
            un[k] = w[k] = 0.0;
            if (i < end) {
                const int2 inc = ld_hint(incid + i, stream);
                un[k] = ld_hint(u + (int64_t)inc.x * DV, keep);
                w[k] = edge_param<double, EK>(pe, inc.y & 0x7fffffff, stream);
                src_side |= (unsigned)(inc.y < 0) << k;
            }
        }
    };
    load(beg);
    double S = 0.0;
    for (uint32_t base = beg; base < end; base += kScanTile) {
        const int n = (int)min((uint32_t)kScanTile, end - base);
#pragma unroll
        for (int k = 0; k < kBlockPer; ++k)
            if (tid + k * kScanThreads < n)
                tile[tile_at(tid + k * kScanThreads)] = incidence_term_w<double, EK>(uv, un[k], w[k], (src_side >> k) & 1u);
        __syncthreads();
        load(base + kScanTile);
        if constexpr (MODE == kModeNative) {
            if (tid < 32) S = chain_sum(S, tile, n);
        } else {
            S = exact_scan_block(S, tile, n, sh);
        }
        __syncthreads();
    }
    if (tid == 0) vertex_f<double, VK>(static_cast<double*>(a.du), u, p, v, S);
}

template <typename T, int VK, int EK, int MODE>
__global__ void __launch_bounds__(kBlock, 1) heavy_solo_kernel(RhsArgs a) {
    if constexpr (sizeof(T) == 8 && MODE != kModeTree) {
        __shared__ double tile[kScanTilePadded];
        __shared__ BlockScanShared sh;
        solo_row_fp64<VK, EK, MODE>(a, blockIdx.x, tile, sh);
    } else {
        extern __shared__ __align__(16) unsigned char smem_dyn[];
        block_row<T, VK, EK>(a, blockIdx.x, smem_dyn);
    }
}

// The FP64 sequential rows ask for 15 KB of shared memory and 128 threads, so that a block also
// fits on an SM that holds several edge-phase blocks; they run on the handle's high-priority side stream.
// The FP32 and tree rows ask for most of an SM (kHeavySoloSmem).
template <typename T, int VK, int EK, int MODE>
cudaError_t launch_heavy_solo(const RhsArgs& a, cudaStream_t s) {
    constexpr bool scan = sizeof(T) == 8 && MODE != kModeTree;
    constexpr int smem = scan ? 0 : kHeavySoloSmem;
    if constexpr (smem > 0) {
        static int attr_set = 0;  // per instantiation; the attribute is per function
        if (attr_set < smem) {
            cudaError_t err = cudaFuncSetAttribute(heavy_solo_kernel<T, VK, EK, MODE>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (err != cudaSuccess) return err;
            attr_set = smem;
        }
    }
    heavy_solo_kernel<T, VK, EK, MODE><<<a.n_apart, scan ? kScanThreads : kBlock, smem, s>>>(a);
    return cudaGetLastError();
}

template <typename T, int VK, int EK>
cudaError_t launch_heavy_typed(const RhsArgs& a, cudaStream_t s) {
    if (a.n_apart == 0) return cudaSuccess;
    if constexpr (sizeof(T) == 4) {
        return launch_heavy_solo<T, VK, EK, kModeTree>(a, s);
    } else {
        switch (a.mode) {
            case kModeNative: return launch_heavy_solo<T, VK, EK, kModeNative>(a, s);
            case kModeTree: return launch_heavy_solo<T, VK, EK, kModeTree>(a, s);
            default: return launch_heavy_solo<T, VK, EK, kModeExact>(a, s);
        }
    }
}

template <typename T, int VK, int EK>
cudaError_t launch_typed(const RhsArgs& a, cudaStream_t s) {
    if (a.heavy_only) return launch_heavy_typed<T, VK, EK>(a, s);
    const int grid = a.n_heavy - a.n_apart + a.n_windows;
    if (grid == 0) return cudaSuccess;
    rhs_kernel<T, VK, EK><<<grid, kBlock, 0, s>>>(a);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_dtype(const RhsArgs& a, cudaStream_t s) {
#define ND_CASE(VK, EK) \
    if (a.vertex_kind == VK && a.edge_kind == EK) return launch_typed<T, VK, EK>(a, s);
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

// Self-test of the integer-exact adder.
__global__ void exact_add_selftest_kernel(const double* a, const double* b, double* out, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = exact::add_rn(a[i], b[i]);
}

// Self-test of the integer division.
__global__ void exact_div_selftest_kernel(const double* a, const double* b, double* out, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = exact::div_rn(a[i], b[i]);
}

// Self-test of the fixed-point sine and cosine.
__global__ void trig_selftest_kernel(const double* x, double* s, double* c, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        s[i] = trig::sin(x[i]);
        c[i] = trig::cos(x[i]);
    }
}

// Self-test of the exact scans: one block per segment; odd segments use the 32-term warp
// scan on registers, even segments shared-memory tiles with the 32-term scan (w % 4 == 2),
// the sliding 256-term scan (w % 8 == 0) or the block-wide scan of the heavy rows (w % 8 == 4).
__global__ void exact_scan_selftest_kernel(const double* terms, const int64_t* seg, const double* s0, double* out,
                                           int64_t nseg) {
    __shared__ double tile[kTile];  // kScanTilePadded entries or more
    __shared__ BlockScanShared sh;
    const int64_t w = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double S = s0[w];
    if (w & 1) {
        if (warp == 0) {
            for (int64_t c = seg[w]; c < seg[w + 1]; c += 32) {
                const int64_t k = c + lane;
                const double t = k < seg[w + 1] ? terms[k] : 0.0;
                const int n = (int)min((int64_t)32, seg[w + 1] - c);
                S = exact_scan_add(S, t, n, lane);
            }
        }
    } else if ((w & 7) == 4) {
        for (int64_t base = seg[w]; base < seg[w + 1]; base += kScanTile) {
            const int n = (int)min((int64_t)kScanTile, seg[w + 1] - base);
            for (int i = threadIdx.x; i < n; i += blockDim.x) tile[tile_at(i)] = terms[base + i];
            __syncthreads();
            S = exact_scan_block(S, tile, n, sh);
            __syncthreads();
        }
    } else {
        for (int64_t base = seg[w]; base < seg[w + 1]; base += kTile) {
            const int n = (int)min((int64_t)kTile, seg[w + 1] - base);
            for (int i = threadIdx.x; i < n; i += blockDim.x) tile[i] = terms[base + i];
            __syncthreads();
            if (warp == 0) S = (w & 2) ? exact_scan_smem(S, tile, n, lane) : exact_scan_wide(S, tile, n, lane);
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) out[w] = S;
}

}  // namespace

cudaError_t launch_rhs(int dtype, const RhsArgs& a, cudaStream_t s) {
    return dtype == ND_F64 ? launch_dtype<double>(a, s) : launch_dtype<float>(a, s);
}

cudaError_t launch_exact_selftest(const double* a, const double* b, double* out, int64_t n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    exact_add_selftest_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, b, out, n);
    return cudaGetLastError();
}

cudaError_t launch_div_selftest(const double* a, const double* b, double* out, int64_t n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    exact_div_selftest_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, b, out, n);
    return cudaGetLastError();
}

cudaError_t launch_trig_selftest(const double* x, double* s, double* c, int64_t n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    trig_selftest_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, s, c, n);
    return cudaGetLastError();
}

cudaError_t launch_scan_selftest(const double* terms, const int64_t* seg, const double* s0, double* out, int64_t nseg,
                                 cudaStream_t s) {
    if (nseg <= 0) return cudaSuccess;
    exact_scan_selftest_kernel<<<(unsigned)nseg, kScanThreads, 0, s>>>(terms, seg, s0, out, nseg);
    return cudaGetLastError();
}

}  // namespace nd
