// Device building blocks shared by the RHS kernels: cache-policy loads and the exact
// (bitwise sequential) summation of FP64 terms on the integer pipes.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "nd_components.cuh"
#include "nd_exact.cuh"
#include "nd_internal.h"

namespace nd {
namespace dev {

constexpr int kBlock = 256;
constexpr int kWarpsPerBlock = kBlock / 32;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kTile = 2048;  // heavy rows: terms per shared-memory tile

// ---- L2 eviction policies -----------------------------------------------------------------
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// ---- a kernel that starts before the one ahead of it in the stream has ended ---------------
// Row kernels of the two-launch right-hand sides are launched as programmatic dependents of
// their edge kernel (launch_secondary), where that is the faster way: once every edge block has started, row blocks take the
// slots that edge blocks free, load what does not depend on the edges, and wait in
// wait_for_primary until the edge grid has ended and its writes are visible.  What the edges
// wrote is read by the volatile, coherent loads below (ld_edge), which stay behind the wait;
// the read-only path may not be used for memory that is written while the kernel runs.  Whole RHS,
// launched after the edge kernel's end against beside its last blocks, µs: diffusion BA(1e6, 4)
// FP32 54.4 / 51.2, BA(2e6, 4) FP64 128 / 122; power grids of 1e3, 1e4 and 1e5 buses, FP64,
// with the loads before the wait 20.5 / 12.3, 22.5 / 14.3, 43 / 35.
__device__ __forceinline__ void dependents_may_start() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_primary() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// (zero where `on` is false, nothing read)
__device__ __forceinline__ double ld_edge(const double* ptr, uint64_t pol, bool on) {
    double r{};
    asm volatile("{.reg .pred q; setp.ne.s32 q, %3, 0; @q ld.global.L2::cache_hint.f64 %0, [%1], %2;}"
                 : "+d"(r)
                 : "l"(ptr), "l"(pol), "r"((int)on));
    return r;
}
__device__ __forceinline__ float ld_edge(const float* ptr, uint64_t pol, bool on) {
    float r{};
    asm volatile("{.reg .pred q; setp.ne.s32 q, %3, 0; @q ld.global.L2::cache_hint.f32 %0, [%1], %2;}"
                 : "+f"(r)
                 : "l"(ptr), "l"(pol), "r"((int)on));
    return r;
}
__device__ __forceinline__ double2 ld_edge(const double2* ptr, uint64_t pol, bool on) {
    double2 r{};
    asm volatile("{.reg .pred q; setp.ne.s32 q, %4, 0; @q ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;}"
                 : "+d"(r.x), "+d"(r.y)
                 : "l"(ptr), "l"(pol), "r"((int)on));
    return r;
}
__device__ __forceinline__ float2 ld_edge(const float2* ptr, uint64_t pol, bool on) {
    float2 r{};
    asm volatile("{.reg .pred q; setp.ne.s32 q, %4, 0; @q ld.global.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;}"
                 : "+f"(r.x), "+f"(r.y)
                 : "l"(ptr), "l"(pol), "r"((int)on));
    return r;
}

// ---- loads with an L2 eviction policy -------------------------------------------------
__device__ __forceinline__ int2 ld_hint(const int2* ptr, uint64_t pol) {
    int2 r;
    asm("ld.global.nc.L2::cache_hint.v2.s32 {%0, %1}, [%2], %3;" : "=r"(r.x), "=r"(r.y) : "l"(ptr), "l"(pol));
    return r;
}
__device__ __forceinline__ double ld_hint(const double* ptr, uint64_t pol) {
    double r;
    asm("ld.global.nc.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(r) : "l"(ptr), "l"(pol));
    return r;
}
__device__ __forceinline__ int32_t ld_hint(const int32_t* ptr, uint64_t pol) {
    int32_t r;
    asm("ld.global.nc.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(r) : "l"(ptr), "l"(pol));
    return r;
}
__device__ __forceinline__ uint32_t ld_hint(const uint32_t* ptr, uint64_t pol) {
    uint32_t r;
    asm("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(r) : "l"(ptr), "l"(pol));
    return r;
}
__device__ __forceinline__ int4 ld_hint(const int4* ptr, uint64_t pol) {
    int4 r;
    asm("ld.global.nc.L2::cache_hint.v4.s32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
        : "l"(ptr), "l"(pol));
    return r;
}
__device__ __forceinline__ double2 ld_hint(const double2* ptr, uint64_t pol) {
    double2 r;
    asm("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(r.x), "=d"(r.y) : "l"(ptr), "l"(pol));
    return r;
}
__device__ __forceinline__ float2 ld_hint(const float2* ptr, uint64_t pol) {
    float2 r;
    asm("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(r.x), "=f"(r.y) : "l"(ptr), "l"(pol));
    return r;
}
__device__ __forceinline__ float ld_hint(const float* ptr, uint64_t pol) {
    float r;
    asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(r) : "l"(ptr), "l"(pol));
    return r;
}
// Stores with an L2 eviction-priority hint (streamed outputs: evict_first).
__device__ __forceinline__ void st_hint(double* ptr, double v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(ptr), "d"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_hint(float* ptr, float v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(ptr), "f"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_hint(double2* ptr, double2 v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.v2.f64 [%0], {%1, %2}, %3;" ::"l"(ptr), "d"(v.x), "d"(v.y), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void st_hint(float2* ptr, float2 v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(ptr), "f"(v.x), "f"(v.y), "l"(pol)
                 : "memory");
}

// Edge parameter of edge e (0 for the parameter-free unit diffusion edge).
template <typename T, int EK>
__device__ __forceinline__ T edge_param(const T* __restrict__ pe, int32_t e, uint64_t pol) {
    if constexpr (EK == ND_E_DIFFUSION_UNIT) {
        return T(0);
    } else {
        return ld_hint(pe + e, pol);
    }
}

// ---- exact sequential sums on the integer pipes ----------------------------------------

// Scaled term R = RN(t / 2^(eS-1075)) for a running sum whose exponent field is eS.
// ok = false when the step cannot be taken by the scan (too large, inf/nan).  For a
// tie (t / ulp exactly halfway between two integers) the truncated magnitude is returned
// with tie = true; the scan then rounds it to even against the running sum's parity.
__device__ __forceinline__ int64_t scaled_term(double t, int eS, bool& ok, bool& tie) {
    const uint64_t tb = exact::to_bits(t);
    uint64_t ft = tb & exact::kFrac;
    int et = (int)((tb >> 52) & 0x7ff);
    if ((tb & ~exact::kSign) == 0) return 0;
    if (et == 0x7ff) {
        ok = false;
        return 0;
    }
    if (et) ft |= exact::kHidden;
    else et = 1;
    const int sh = eS - et;  // t / ulp(S) = ft · 2^-sh
    uint64_t mag;
    if (sh <= 0) {
        if (sh < -9) {
            ok = false;
            return 0;
        }
        mag = ft << (-sh);
    } else if (sh >= 64) {
        mag = 0;  // |t| < 2^-11 ulp: rounds to zero, never a tie
    } else {
        mag = ft >> sh;
        const uint64_t rem = ft & ((1ull << sh) - 1);
        const uint64_t half = 1ull << (sh - 1);
        if (rem > half) mag += 1;
        else if (rem == half) tie = true;
    }
    if (mag >= (1ull << 52)) ok = false;
    return (tb & exact::kSign) ? -(int64_t)mag : (int64_t)mag;
}

// Add the terms held by lanes [0, n) of the warp to S, in lane order, exactly as the
// sequential loop S = S + t_0; S = S + t_1; ... would.  S is warp-uniform.
__device__ __forceinline__ double exact_scan_add(double S, double t, int n, int lane) {
    int j0 = 0;
    while (j0 < n) {
        const uint64_t sb = exact::to_bits(S);
        const int eS = (int)((sb >> 52) & 0x7ff);
        if (eS == 0 || eS == 0x7ff) {  // zero / subnormal / non-finite sum: one exact step
            S = exact::add_rn(S, __shfl_sync(kFull, t, j0));
            ++j0;
            continue;
        }
        const bool active = lane >= j0 && lane < n;
        bool ok = true, tie = false;
        int64_t x = active ? scaled_term(t, eS, ok, tie) : 0;
        // Ties round to even against the running sum.  Its parity evolves as p -> p ^ (R & 1)
        // for ordinary steps and p -> 0 after a tie step; the composition of such maps
        // (p -> (p & ka) ^ kb) is scanned to give each lane the parity before its step.
        unsigned ka = tie ? 0u : 1u, kb = tie ? 0u : (unsigned)(x & 1);
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned pa = __shfl_up_sync(kFull, ka, off), pb = __shfl_up_sync(kFull, kb, off);
            if (lane >= off) {
                kb = (pb & ka) ^ kb;
                ka = pa & ka;
            }
        }
        if (__any_sync(kFull, tie)) {
            unsigned xa = __shfl_up_sync(kFull, ka, 1), xb = __shfl_up_sync(kFull, kb, 1);
            if (lane == 0) {
                xa = 1u;
                xb = 0u;
            }
            const unsigned p_prev = ((unsigned)(sb & 1) & xa) ^ xb;
            if (tie) {
                const uint64_t mag = (uint64_t)(x < 0 ? -x : x);
                const uint64_t c = (p_prev ^ (unsigned)(mag & 1)) & 1u;  // 1: round away from zero
                x = (exact::to_bits(t) & exact::kSign) ? -(int64_t)(mag + c) : (int64_t)(mag + c);
            }
        }
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int64_t y = __shfl_up_sync(kFull, x, off);
            if (lane >= off) x += y;
        }
        const int64_t mS = (int64_t)((sb & exact::kFrac) | exact::kHidden);
        const int64_t m = (sb & exact::kSign) ? x - mS : x + mS;
        const uint64_t am = (uint64_t)(m < 0 ? -m : m);
        const bool valid = ok && am >= (1ull << 52) + 1 && am <= (1ull << 53) - 2;
        const unsigned bad = __ballot_sync(kFull, active && !valid);
        const int L = bad ? __ffs(bad) - 1 : n;
        if (L > j0) {
            const int64_t mL = __shfl_sync(kFull, m, L - 1);
            const uint64_t aL = (uint64_t)(mL < 0 ? -mL : mL);
            S = exact::from_bits((mL < 0 ? exact::kSign : 0) | ((uint64_t)eS << 52) | (aL & exact::kFrac));
        }
        if (L < n) S = exact::add_rn(S, __shfl_sync(kFull, t, L));
        j0 = L + 1;
    }
    return S;
}

// Sequential exact sum of n terms in shared memory by one warp, 32 at a time.
__device__ __forceinline__ double exact_scan_smem(double S, const double* __restrict__ tile, int n, int lane) {
    for (int c = 0; c < n; c += 32) {
        const int k = c + lane;
        const double t = k < n ? tile[k] : 0.0;
        S = exact_scan_add(S, t, min(32, n - c), lane);
    }
    return S;
}

// The same sum with a sliding window of 8 terms per lane (256 per step): each lane scales
// its 8 terms (resolving ties against the running sum's parity) and prefix-sums them
// locally, one warp scan adds the lanes before it, and every position checks that its
// running sum stays strictly inside S's binade.  The window then slides to just past the
// first position that failed (a binade change), which is added with the hardware adder.
// Long hub rows change binade every ~100 terms, so a step advances far at the cost of a
// single warp scan.
constexpr int kScanPer = 8;
constexpr int kScanFallback = 16;
constexpr int kScanFallbackMax = 1024;
static __device__ __forceinline__ double exact_scan_wide(double S, const double* __restrict__ tile, int n, int lane) {
    int pos = 0;
    int fallback = kScanFallback;  // length of the next run of hardware adds after a stall
    while (pos < n) {
        const uint64_t sb = exact::to_bits(S);
        const int eS = (int)((sb >> 52) & 0x7ff);
        if (eS == 0 || eS == 0x7ff) {  // zero / subnormal / non-finite sum: one exact step
            S = exact::add_rn(S, tile[pos]);
            ++pos;
            continue;
        }
        const int end = min(n, pos + 32 * kScanPer);
        const int base = pos + lane * kScanPer;
        int64_t pre[kScanPer];
        unsigned okmask = 0, tiemask = 0;
#pragma unroll
        for (int i = 0; i < kScanPer; ++i) {
            bool ok = true, tie = false;
            const int q = base + i;
            pre[i] = q < end ? scaled_term(tile[q], eS, ok, tie) : 0;
            okmask |= (unsigned)ok << i;
            tiemask |= (unsigned)tie << i;
        }
        if (__any_sync(kFull, tiemask != 0)) {
            // Ties round to even against the running sum, whose parity evolves as
            // p -> p ^ (R & 1) for an ordinary step and p -> 0 after a tie.  Each lane
            // composes its steps into p -> (p & ka) ^ kb, a warp scan composes the lanes,
            // and each lane replays its steps from the parity before its first one.
            unsigned ka = 1u, kb = 0u;
#pragma unroll
            for (int i = 0; i < kScanPer; ++i) {
                if ((tiemask >> i) & 1u) ka = kb = 0u;
                else kb ^= (unsigned)(pre[i] & 1);
            }
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned pa = __shfl_up_sync(kFull, ka, off), pb = __shfl_up_sync(kFull, kb, off);
                if (lane >= off) {
                    kb = (pb & ka) ^ kb;
                    ka = pa & ka;
                }
            }
            unsigned xa = __shfl_up_sync(kFull, ka, 1), xb = __shfl_up_sync(kFull, kb, 1);
            if (lane == 0) {
                xa = 1u;
                xb = 0u;
            }
            unsigned par = ((unsigned)(sb & 1) & xa) ^ xb;
#pragma unroll
            for (int i = 0; i < kScanPer; ++i) {
                if ((tiemask >> i) & 1u) {
                    const uint64_t mag = (uint64_t)(pre[i] < 0 ? -pre[i] : pre[i]);
                    const uint64_t c = (par ^ (unsigned)(mag & 1)) & 1u;  // 1: away from zero
                    pre[i] = (exact::to_bits(tile[base + i]) & exact::kSign) ? -(int64_t)(mag + c)
                                                                              : (int64_t)(mag + c);
                    par = 0u;
                } else {
                    par ^= (unsigned)(pre[i] & 1);
                }
            }
        }
        int64_t run = 0;
#pragma unroll
        for (int i = 0; i < kScanPer; ++i) {
            run += pre[i];
            pre[i] = run;
        }
        int64_t x = run;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int64_t y = __shfl_up_sync(kFull, x, off);
            if (lane >= off) x += y;
        }
        const int64_t mS0 = (int64_t)((sb & exact::kFrac) | exact::kHidden);
        const int64_t mS = (sb & exact::kSign) ? -mS0 : mS0;
        const int64_t before = mS + x - run;  // running sum before this lane's first term
        int firstbad = 0x7fffffff;
#pragma unroll
        for (int i = kScanPer - 1; i >= 0; --i) {
            const int64_t m = before + pre[i];
            const uint64_t am = (uint64_t)(m < 0 ? -m : m);
            const bool valid = ((okmask >> i) & 1u) && am >= (1ull << 52) + 1 && am <= (1ull << 53) - 2;
            if (base + i < end && !valid) firstbad = base + i;
        }
        const int P = (int)__reduce_min_sync(kFull, (unsigned)firstbad);
        const int acc_end = P < end ? P : end;  // positions [pos, acc_end) are exact
        if (acc_end > pos) {
            const int q = acc_end - 1 - pos, owner = q / kScanPer, idx = q % kScanPer;
            int64_t mine = 0;
#pragma unroll
            for (int i = 0; i < kScanPer; ++i)
                if (i == idx) mine = before + pre[i];
            const int64_t mL = __shfl_sync(kFull, mine, owner);
            const uint64_t aL = (uint64_t)(mL < 0 ? -mL : mL);
            S = exact::from_bits((mL < 0 ? exact::kSign : 0) | ((uint64_t)eS << 52) | (aL & exact::kFrac));
        }
        if (P < end) {
            S = __dadd_rn(S, tile[P]);
            const int advanced = P + 1 - pos;
            pos = P + 1;
            // A sum hovering at a binade boundary changes binade every few terms and the
            // scan stalls; then a run of hardware adds on lane 0 is cheaper per term.  The
            // run doubles while the stalls persist (up to kScanFallbackMax terms) and drops
            // back once a step advances far, so a row never costs much more than a plain
            // chain of adds.
            if (advanced < kScanPer && pos < n) {
                const int stop = min(n, pos + fallback);
                if (lane == 0)
                    for (int i = pos; i < stop; ++i) S = __dadd_rn(S, tile[i]);
                S = __shfl_sync(kFull, S, 0);
                pos = stop;
                fallback = min(2 * fallback, kScanFallbackMax);
            } else if (advanced >= 64) {
                fallback = kScanFallback;
            }
        } else {
            pos = end;
            fallback = kScanFallback;
        }
    }
    return S;
}


// ---- the same sum by a whole block ------------------------------------------------------------
// A long row is one chain of dependent roundings: 63 clocks a term with hardware adds on an
// idle SM (several times that beside other FP64 work, which shares the SM's one FP64 unit), and
// a restart of the scan above at every binade change, which a sum of mixed signs has every few
// terms.  Here a block takes kScanTile terms a step on the integer pipes, across binade changes:
//   1. the terms as integers in units of 2^-9 ulps of the frame's top binade (rounded down, a set
//      last bit standing for the bits below) and one scan of them predict the binade of every
//      running sum;
//   2. with g_i the ulp of S_i's predicted binade in that unit,
//          S_i = g_i · RNE((S_{i-1} + t_i) / g_i).
//      Where g_i <= g_{i-1} and t_i is not halfway between multiples of g_i, that is S_{i-1} plus
//      t_i rounded to g_i, whatever S_{i-1} is: a second scan adds these.  The others, "events"
//      (ties, and steps into a higher binade, which round S_{i-1}'s own last bits), are few;
//   3. one warp goes through the events in order (an integer add, a rounding and a subtraction
//      each, about 50 clocks) and hands every position the correction of the last event before it;
//   4. every position checks that its sum lies inside its predicted binade, not next to its ends:
//      up to the first that does not, all are the sequential sum's bits, by induction.
// The frame spans 8 binades (the starting sum's, four above, three below).  A step ends at the
// first position outside it (mostly a sum close to zero).
// The heavy kernel alone, 36 rows of 129 to 935 terms of BA(1e5, 2) swing / 264 rows of 400 to 6327
// terms of BA(2e6, 4) diffusion: 38 / 48 µs; with 256 threads of four terms, 64-bit binade tests
// and a scan of their own for the predictions 71 / 52 µs.  A thread of the row phase takes 56 to
// 75 µs for the 935-term row, and the 256-term warp scan took 164 µs for the 6327-term one.
constexpr int kScanThreads = 128;
constexpr int kScanWarps = kScanThreads / 32;
constexpr int kBlockPer = 4;
constexpr int kScanTile = kScanThreads * kBlockPer;
// Position i of a tile in shared memory: one pad entry per thread's terms keeps the threads'
// reads of their own terms free of bank conflicts.
__device__ __forceinline__ int tile_at(int i) { return i + i / kBlockPer; }
constexpr int kScanTilePadded = kScanTile + kScanTile / kBlockPer;
constexpr int kFrameUp = 4, kFrameTop = 9, kFrameLow = 2;  // log2 of g: kFrameTop in the top binade
// A step costs about as much as 48 hardware adds.  A step that advanced less is followed by a run
// of them, doubled while that persists; a longer one by the two that bring a sum close to zero
// back to the terms' size.
constexpr int kScanShort = 48, kRunMin = 2, kRunShort = 32, kRunMax = 512;

struct BlockScanShared {
    int64_t term[kScanWarps], total[kScanWarps];
    int count[kScanWarps];
    unsigned outside[kScanWarps], first_bad[kScanWarps];
    int n_events;
    double sum;
    // events: the prefix before it (then the correction behind it), its term, log2 g
    int64_t ev_prefix[kScanTile], ev_term[kScanTile];
    int8_t ev_shift[kScanTile];
};

// The upper word of |m|, one too small for negative m whose lower word is zero.  So an exact negative
// power of two counts to the binade below its own: a sum that is one is refused (its bits there are
// all ones), and a start that is one only makes the first step an event.
__device__ __forceinline__ uint32_t abs_hi(int64_t m) {
    const int32_t h = (int32_t)(m >> 32);
    return (uint32_t)(h ^ (h >> 31));
}

// S + the n terms of `tile` (tile_at layout), in order; S is the same in every thread, and so
// is the result.  All kScanThreads threads call it; `tile` is visible to all of them before.
static __device__ __forceinline__ double exact_scan_block(double S, const double* __restrict__ tile, int n,
                                                          BlockScanShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = tid * kBlockPer;
    // this thread's terms: signed significands and exponent fields (subnormals: 1)
    int64_t sig[kBlockPer];
    int et[kBlockPer];
#pragma unroll
    for (int i = 0; i < kBlockPer; ++i) {
        const uint64_t b = base + i < n ? exact::to_bits(tile[tile_at(base + i)]) : 0;
        const int e = (int)((b >> 52) & 0x7ff);
        const int64_t m = (int64_t)((b & exact::kFrac) | (e ? exact::kHidden : 0));
        sig[i] = (b & exact::kSign) ? -m : m;
        et[i] = e ? e : 1;
    }
    int pos = 0, run_len = 0;
    int fallback = (exact::to_bits(S) << 1) == 0 ? 8 : 0;  // > 0: the next run is this many hardware adds
    while (pos < n) {
        const uint64_t sb = exact::to_bits(S);
        const int eS = (int)((sb >> 52) & 0x7ff);
        if (fallback == 0 && (eS < 16 || eS > 0x7ff - 32)) fallback = kRunShort;  // zero, subnormal, not finite
        if (fallback > 0) {  // one warp, so that the SM's FP64 unit serves this chain alone
            const int stop = min(n, pos + fallback);
            if (warp == 0) {
                for (int i = pos; i < stop; ++i) S = __dadd_rn(S, tile[tile_at(i)]);
                if (lane == 0) sh.sum = S;
            }
            __syncthreads();
            S = sh.sum;
            __syncthreads();
            pos = stop;
            fallback = 0;
            continue;
        }
        // 1. the terms in frame units, and their scan
        const int64_t mS = (int64_t)(((sb & exact::kFrac) | exact::kHidden) << (kFrameTop - kFrameUp));
        const int64_t m0 = (sb & exact::kSign) ? -mS : mS;
        int64_t term[kBlockPer];
        int64_t run = 0;
        unsigned outside = 0xffffffffu;
#pragma unroll
        for (int i = kBlockPer - 1; i >= 0; --i) {
            const int L = et[i] - eS + (kFrameTop - kFrameUp);  // significand · 2^L
            int64_t t;
            if (L >= 0) {
                t = sig[i] << min(L, 10);
            } else {
                const int r = min(-L, 63);
                t = sig[i] >> r;
                t |= (int64_t)((t << r) != sig[i]);
            }
            const bool active = base + i >= pos;  // 0 behind the end of the tile
            if (active && L > 10 && sig[i] != 0) outside = (unsigned)(base + i);
            term[i] = active ? t : 0;
            run += term[i];
        }
        int64_t x = run;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int64_t y = __shfl_up_sync(kFull, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) sh.term[warp] = x;
        __syncthreads();
        int64_t before = m0 + (x - run);
#pragma unroll
        for (int w = 0; w < kScanWarps - 1; ++w)
            if (w < warp) before += sh.term[w];
        // 2. predicted log2 g (kFrameTop in the binade with |S| in [2^61, 2^62)), rounded terms, events
        auto log_g = [](int64_t A) { return kFrameTop + 2 - exact::clz32(abs_hi(A)); };
        int64_t pre[kBlockPer];
        int lg[kBlockPer];
        unsigned events = 0;
        int prev = log_g(before);
        run = 0;
#pragma unroll
        for (int i = 0; i < kBlockPer; ++i) {
            before += term[i];
            const int s = log_g(before);
            if (base + i >= pos && base + i < n && (unsigned)(s - kFrameLow) > (unsigned)(kFrameTop - kFrameLow))
                outside = min(outside, (unsigned)(base + i));
            lg[i] = max(kFrameLow, min(kFrameTop, s));
            const uint32_t g = 1u << lg[i], half = g >> 1;
            const bool event = s > prev || ((uint32_t)term[i] & (g - 1)) == half;
            events |= (unsigned)event << i;
            if (!event) run += (term[i] + (int64_t)half) & ~(int64_t)(g - 1);
            pre[i] = run;
            prev = s;
        }
        x = run;
        int cnt = __popc(events);
        const int mine = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int64_t y = __shfl_up_sync(kFull, x, off);
            const int c = __shfl_up_sync(kFull, cnt, off);
            if (lane >= off) {
                x += y;
                cnt += c;
            }
        }
        outside = __reduce_min_sync(kFull, outside);
        if (lane == 31) {
            sh.total[warp] = x;
            sh.count[warp] = cnt;
            sh.outside[warp] = outside;
        }
        __syncthreads();
        before = x - run;
        cnt -= mine;
        int P = n;
#pragma unroll
        for (int w = 0; w < kScanWarps; ++w) {
            if (w < warp) {
                before += sh.total[w];
                cnt += sh.count[w];
            }
            P = (int)min((unsigned)P, sh.outside[w]);
        }
        // the events before the first position outside the frame, in order
        int idx = cnt;
#pragma unroll
        for (int i = 0; i < kBlockPer; ++i) {
            if (((events >> i) & 1u) && base + i < P) {
                sh.ev_prefix[idx] = before + pre[i];
                sh.ev_term[idx] = term[i];
                sh.ev_shift[idx] = (int8_t)lg[i];
                ++idx;
            }
        }
        if (P > base && P <= base + kBlockPer) sh.n_events = idx;
        if (P == 0 && tid == 0) sh.n_events = 0;
        __syncthreads();
        // 3. the events, in order
        if (warp == 0) {
            const int ne = sh.n_events;
            int64_t c = m0;
            int64_t b = sh.ev_prefix[0], t = sh.ev_term[0];
            int s = sh.ev_shift[0];
            for (int k = 0; k < ne; ++k) {
                const int kn = min(k + 1, kScanTile - 1);
                const int64_t bn = sh.ev_prefix[kn], tn = sh.ev_term[kn];
                const int sn = sh.ev_shift[kn];
                const int64_t v = c + (b + t);
                const uint32_t g = 1u << s, lsb = ((uint32_t)v >> s) & 1u;
                c = ((v + (int64_t)(g / 2 - 1 + lsb)) & ~(int64_t)(g - 1)) - b;
                __syncwarp();
                if (lane == 0) sh.ev_prefix[k] = c;
                b = bn;
                t = tn;
                s = sn;
            }
        }
        __syncthreads();
        // 4. the sums, and the first position whose sum is not inside its binade: the upper word
        // of |S_i| has 22 or more bits of it, which must be those of the binade and neither all
        // zero nor all one below the first
        int64_t val[kBlockPer];
        unsigned firstbad = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < kBlockPer; ++i) {
            cnt += (int)((events >> i) & 1u);
            const bool in = base + i >= pos && base + i < P;
            val[i] = before + pre[i] + (cnt > 0 && in ? sh.ev_prefix[cnt - 1] : m0);
            const uint32_t h = abs_hi(val[i]);
            const int lz = exact::clz32(h);
            const uint32_t low = (h << lz) & 0x7ffffe00u;
            if (in && (kFrameTop + 2 - lz != lg[i] || low == 0 || low == 0x7ffffe00u))
                firstbad = min(firstbad, (unsigned)(base + i));
        }
        firstbad = __reduce_min_sync(kFull, firstbad);
        if (lane == 0) sh.first_bad[warp] = firstbad;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kScanWarps; ++w) P = (int)min((unsigned)P, sh.first_bad[w]);
        // positions [pos, P) are exact: the owner of P - 1 publishes the sum behind it
        if (P > pos) {
#pragma unroll
            for (int i = 0; i < kBlockPer; ++i)
                if (base + i == P - 1) {
                    const uint64_t am = (uint64_t)(val[i] < 0 ? -val[i] : val[i]) >> lg[i];
                    sh.sum = exact::from_bits((val[i] < 0 ? exact::kSign : 0) |
                                              ((uint64_t)(eS + lg[i] - (kFrameTop - kFrameUp)) << 52) |
                                              (am & exact::kFrac));
                }
            __syncthreads();
            S = sh.sum;
        }
        run_len = P - pos >= kScanShort ? 0 : min(kRunMax, max(kRunShort, 2 * run_len));
        pos = P;
        if (pos < n) fallback = max(kRunMin, run_len);
        __syncthreads();  // sh is written again
    }
    return S;
}


// Host side: launch `k` as a programmatic dependent of the kernel before it in stream `s`.  That
// kernel is one of the same call, launched normally: what `k` reads before wait_for_primary was
// complete before that kernel began.  Behind a kernel that is not ours nothing would promise that.
template <typename... P>
inline cudaError_t launch_secondary(void (*k)(P...), unsigned grid, int block, cudaStream_t s, P... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace dev
}  // namespace nd
