// B200 box-least-squares search kernels (sm_100a).
//
// One persistent launch processes work items of (curve, segment, tile of up to
// kMaxTile consecutive trial periods).  Per item a CTA
//   1. folds every point of the curve into one shared-memory histogram per
//      period of the tile.  The phase bin is the reference's
//      w = x - P*floor(x/P); ind = int(w/bin) + 1   (cuPeriod
//      src/cuperiod/methods/_bls_core.py:369-376 / 536-538), computed by a fast
//      FP64 path (FoldConst) whose result is used only when it is provably the
//      reference's; otherwise the reference's own IEEE chain runs.  Bin sums are
//      exact integers built with native 32-bit shared reductions only (64-bit and
//      floating-point shared atomics are emulated on sm_100), except for curves of
//      more than 2^17 points or of extreme scale, whose sums stay FP64.  A lane holds
//      8 time-consecutive points (the lanes of a warp 8 points apart, so their bins
//      rarely collide);
//   2. per period: applies the reference's wrap pad (_bls_core.py:377-381), turns the
//      bins into prefix sums in place and writes an FP32 screen copy;
//   3. sweeps every (duration, start) box.  Each lane keeps the largest FP32 upper bound
//      of the box objective it meets and where; the boxes that provably cannot be the
//      period's best drop out against the largest lower bound, and the few left are
//      evaluated with the reference's FP64 formulas (_bls_core.py:410-426) on the exact
//      sums, the winner the first in (duration index, start) order among equals, as in
//      the reference;
//   4. writes the reference's seven per-period fields (_bls_core.py:443-460).
// A period takes two CTA barriers: one between the scan's two passes (which also ends
// the previous period's sweep), one before its sweep.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>
#include <cfloat>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "bls_device.h"
#include "bls_fold.cuh"
#include "bls_launch.h"

namespace blsb200 {
namespace {

constexpr int kThreads = kChunkThreads;
constexpr int kWarps = kThreads / 32;
constexpr int kPts = kChunkPts;
constexpr unsigned kFull = 0xffffffffu;
constexpr float kRel = 1.0f / 262144.0f;    // 2^-18: relative slack of FP32 key bounds
constexpr int kCasLimit = 1 << 16;          // retries of one FP64 shared add
constexpr int kList = 512;                  // candidates of one tile
constexpr int kRegBins = 9;                 // bins a lane holds in registers while scanning
constexpr int kOpenBits = 28;               // open point: period << kOpenBits | point
constexpr uint32_t kNoPoint = 0xffffffffu;  // (of a 17th period)
constexpr int kBoxBits = 20;                // box key: duration index << kBoxBits | start
// Per-point weights: the FP32 screen holds them scaled by 2^-shift, their sum (below
// 2^54, 2^60 and 2^54) at most 2^41, so that the likelihood's iv_in * iv_out^2 stays
// below 2^126
template <int MODE>
__device__ __host__ constexpr int screen_shift() {
    return MODE == MODE_WIDE ? 13 : (MODE == MODE_EXACT || MODE == MODE_GENERAL) ? 20 : 0;
}

// One work item's inputs, copied to shared memory while the item before it is searched.
struct Tile {
    CurveDesc curve;
    SegmentDesc seg;
    double per[kMaxTile];
    double freq[kMaxTile];
    uint32_t scale[kMaxTile];
    int32_t nb[kMaxTile];
    alignas(16) int32_t dur[kMaxDur + 4];   // box widths, the last one repeated to a multiple
                                            // of four (a repeated box only ties itself)
    int32_t p_begin, p_count;
    int32_t d_min, d_max;                   // smallest and largest width
    int32_t item;                           // work item, >= n_items: none left
};

struct TileShared {
    Tile tile[2];
    uint32_t thr_bits[kMaxTile];    // per period: a lower bound of its best key (bits of a
                                    // float >= 0)
    int32_t win[kMaxTile];          // per period: the best box's key, -1 when there is none
    long long tot[2][2][kWarps];    // scan: per-warp totals (by block parity, value)
    double tot_d[2][kWarps];
    float red_t[kWarps];
    double red_v[kWarps];
    int red_box[kWarps];
    int red_ne[kWarps];             // GENERAL scan: last non-empty bin per warp
    // candidates: period << 25 | box, standing for the four widths of the box's group at
    // its start
    uint32_t list[kList];
    int list_n;
    // shared address of the next entry of the fold's list of open points, period << kOpenBits |
    // point: in the dynamic shared memory past the histograms, which is free until the scans
    uint32_t open_at;
    uint32_t rescan;                // bit q: period q needs every box in FP64
};

// Shared-memory accesses by 32-bit shared-space address (the hot loops compute
// addresses in 32-bit arithmetic instead of converting generic pointers).
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void red_add_u32(uint32_t a, uint32_t v) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void st_u32(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ double ld_f64(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void st_f64(uint32_t a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ float2 ld_f2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ void st_f2(uint32_t a, float2 v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
// {b.x - a.x, b.y - a.y} in one packed add, given {-a.x, -a.y}.
__device__ __forceinline__ float2 add_f2(float2 b, float2 na) {
    float2 r;
    asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
        " add.rn.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(b.x), "f"(b.y), "f"(na.x), "f"(na.y));
    return r;
}

// 1 / x to an ulp (0 for x above 2^126).
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// FP64 add to a shared-memory word by a bounded compare-and-swap loop in the
// shared state space.  The loop is lock-free (a failed swap means another thread
// succeeded); the bound only guards against the impossible and sets `flag`.
__device__ __forceinline__ void shared_add_f64(uint32_t addr, double v, int32_t* flag) {
    if (v == 0.0) return;
    unsigned long long old;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(old) : "r"(addr) : "memory");
    for (int it = 0; it < kCasLimit; ++it) {
        const unsigned long long want = __double_as_longlong(__longlong_as_double(old) + v);
        unsigned long long seen;
        asm volatile("atom.shared.cas.b64 %0, [%1], %2, %3;"
                     : "=l"(seen) : "r"(addr), "l"(old), "l"(want) : "memory");
        if (seen == old) return;
        old = seen;
    }
    atomicExch(flag, 2);
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}

// Sums of one box inside and outside, in the reference's units: the reference
// forms the outside as sum_y - y_in and sum_ivar - iv_in; WIDE and EXACT curves take
// them from the exact quantised totals instead (CurveDesc::rq_total).
struct BoxSums {
    double y_in, iv_in, y_out, iv_out;
};

// The reference's objective of one box (_bls_core.py:410-426); -inf when the box
// is not admissible.
__device__ __forceinline__ double box_objective(const BoxSums& s, const CurveDesc& c, int obj) {
    const double iv_out = s.iv_out;
    if (!(s.iv_in >= c.ivar_floor) || !(iv_out >= c.ivar_floor)) return -CUDART_INF;
    const double yin = s.y_in / s.iv_in;
    const double yout = s.y_out / iv_out;
    if (yout < yin) return -CUDART_INF;
    const double depth = yout - yin;
    if (obj == 0) return depth / sqrt(1.0 / s.iv_in + 1.0 / iv_out);
    return 0.5 * s.iv_in * depth * depth;
}

// ---- histogram layout ---------------------------------------------------------
// Integer modes keep kW planes of 32-bit words per period, one word per bin in each
// (a bin is one word of a bank in every plane, so 32 random bins fall on 32 banks;
// records of 8 or 16 bytes would use half or a quarter of them).  A point adds one
// word to each plane, a native 32-bit reduction without a return value:
//  PAIR:    {v, (v >> 20) << 12 | 1}: the quantised centred flux*weight v (28 bits
//           and sign) modulo 2^32, and its top part above a count.  The second plane
//           gives the count (a bin holds at most kPairMax points, host bound) and
//           H = sum of v >> 20; the sum of v is 2^20 H plus what the first plane
//           holds above 2^20 H modulo 2^32 -- at most kPairMax * 2^20 < 2^32, so no
//           carry is lost;
//  UNIFORM: {low 13 bits of v, v >> 13, 1}: as PAIR for any number of points in a bin;
//  WIDE:    {r, r >> 19, i, i >> 19} of the 38-bit flux*weight and weight, at most
//           kWideMax points in a bin;
//  EXACT:   {r, r >> 15, r >> 30, i, i >> 15, i >> 30} of 61-bit values, any number
//           of points (the same argument twice: 2^17 points x 2^15 <= 2^32).
// GENERAL keeps 16-byte records of two FP64 sums.  The scan leaves exact prefix sums
// in place: 64-bit integers in the words' first planes (PAIR / UNIFORM one, packed
// as sum << kCountShift | count; WIDE / EXACT two), or the FP64 record.  One bin past
// the last takes what the reference never reads.
template <int MODE>
__device__ __host__ constexpr int point_words() {
    return MODE == MODE_PAIR ? 2 : MODE == MODE_UNIFORM ? 3 : MODE == MODE_WIDE ? 4
           : MODE == MODE_EXACT ? 6 : 0;
}
template <int MODE>
__device__ __host__ constexpr bool one_weight() {
    return MODE == MODE_PAIR || MODE == MODE_UNIFORM;
}
template <int MODE>
__device__ __host__ __forceinline__ uint32_t plane_bytes(int hl) {
    return 4u * (uint32_t)((hl + 1 + 3) & ~3);
}
template <int MODE>
__device__ __host__ __forceinline__ uint32_t hist_period_bytes(int hl) {
    return MODE == MODE_GENERAL ? 16u * (uint32_t)(hl + 1)
                                : (uint32_t)point_words<MODE>() * plane_bytes<MODE>(hl);
}
// planes of the weight's words start here (WIDE / EXACT)
template <int MODE>
__device__ __host__ constexpr int weight_plane() {
    return MODE == MODE_EXACT ? 3 : 2;
}

// One period's histogram: its address and the distance between planes.
struct Hist {
    uint32_t base, plane;
};

__device__ __forceinline__ long long ld_planes(uint32_t a, uint32_t plane) {
    return (long long)(((unsigned long long)ld_u32(a + plane) << 32) | ld_u32(a));
}
__device__ __forceinline__ void st_planes(uint32_t a, uint32_t plane, long long v) {
    st_u32(a, (uint32_t)v);
    st_u32(a + plane, (uint32_t)((unsigned long long)v >> 32));
}

// A sum kept as its value modulo 2^32 (`low`) and the sum of its points' values
// shifted right by S (`high`): exact while the points' remainders add up below 2^32.
template <int S>
__device__ __forceinline__ long long join_sum(long long high, uint32_t low) {
    return high * (1ll << S) + (long long)(uint32_t)(low - ((uint32_t)high << S));
}

// The sums of bin i: flux*weight and weight (packed with its count when there is one
// weight).
template <int MODE>
__device__ __forceinline__ void bin_sums(const Hist& h, int i, long long& r, long long& w) {
    const uint32_t a = h.base + 4u * (uint32_t)i;
    w = 0;
    if (MODE == MODE_PAIR) {
        // 2^20 H as a 64-bit value: the second plane's top 20 bits, 8 up; the first plane
        // is its low word plus the remainder modulo 2^32, so a low word above it carries
        const uint32_t lo = ld_u32(a), b = ld_u32(a + h.plane);
        const uint32_t base = (b << (32 - 2 * kPairBits)) & ~((1u << (32 - kPairBits)) - 1u);
        const uint32_t hi = (uint32_t)((int32_t)b >> (2 * kPairBits)) + (lo < base ? 1u : 0u);
        r = (long long)(((unsigned long long)__funnelshift_l(lo, hi, kCountShift) << 32) |
                        ((lo << kCountShift) | (b & ((1u << kPairBits) - 1u))));
    } else if (MODE == MODE_UNIFORM) {
        const long long sum = (long long)(int32_t)ld_u32(a + h.plane) * (1ll << kHalfBits) +
                              (long long)ld_u32(a);
        r = (sum << kCountShift) + (long long)ld_u32(a + 2 * h.plane);
    } else if (MODE == MODE_WIDE) {
        r = join_sum<kWideBits>((int32_t)ld_u32(a + h.plane), ld_u32(a));
        w = join_sum<kWideBits>((int32_t)ld_u32(a + 3 * h.plane), ld_u32(a + 2 * h.plane));
    } else {
        // the middle sum modulo 2^32 is completed by the high one, then completes the low
        r = join_sum<kExactBits>(join_sum<kExactBits>((int32_t)ld_u32(a + 2 * h.plane),
                                                      ld_u32(a + h.plane)),
                                 ld_u32(a));
        w = join_sum<kExactBits>(join_sum<kExactBits>((int32_t)ld_u32(a + 5 * h.plane),
                                                      ld_u32(a + 4 * h.plane)),
                                 ld_u32(a + 3 * h.plane));
    }
}

// Prefix sums at bin i, as the scan left them.
__device__ __forceinline__ long long prefix_r(const Hist& h, int i) {
    return ld_planes(h.base + 4u * (uint32_t)i, h.plane);
}
template <int MODE>
__device__ __forceinline__ long long prefix_w(const Hist& h, int i) {
    return ld_planes(h.base + 4u * (uint32_t)i + weight_plane<MODE>() * h.plane, h.plane);
}

// Exact sums of box (n, d) in the reference's units from one period's prefixes.
template <int MODE>
__device__ __forceinline__ BoxSums box_sums(const Hist& h, const CurveDesc& cv, int n, int d) {
    BoxSums b;
    if (one_weight<MODE>()) {
        const long long v = prefix_r(h, n + d) - prefix_r(h, n);
        const double cnt = (double)(v & ((1ll << kCountShift) - 1));
        b.iv_in = cnt * cv.w_uniform;
        b.y_in = ldexp((double)(v >> kCountShift), -cv.e_r) + cv.center * cnt;
    } else if (MODE != MODE_GENERAL) {
        const long long qi = prefix_w<MODE>(h, n + d) - prefix_w<MODE>(h, n);
        const long long qr = prefix_r(h, n + d) - prefix_r(h, n);
        b.iv_in = ldexp((double)qi, -cv.e_i);
        b.y_in = ldexp((double)qr, -cv.e_r) + cv.ybar * b.iv_in;
        b.iv_out = ldexp((double)(cv.iq_total - qi), -cv.e_i);
        b.y_out = ldexp((double)(cv.rq_total - qr), -cv.e_r) + cv.ybar * b.iv_out;
        return b;
    } else {
        const uint32_t r1 = h.base + (uint32_t)(n + d) * 16u, r0 = h.base + (uint32_t)n * 16u;
        b.iv_in = ldexp(ld_f64(r1 + 8) - ld_f64(r0 + 8), -cv.e_i);
        b.y_in = ldexp(ld_f64(r1) - ld_f64(r0), -cv.e_r) + cv.ybar * b.iv_in;
    }
    b.iv_out = cv.sum_ivar - b.iv_in;
    b.y_out = cv.sum_y - b.y_in;
    return b;
}

// The reference's objective of box (n, d), out of line: reached rarely.
template <int MODE, int OBJ>
__device__ __noinline__ double exact_objective(uint32_t base, uint32_t plane, const CurveDesc* cv,
                                               int n, int d) {
    return box_objective(box_sums<MODE>(Hist{base, plane}, *cv, n, d), *cv, OBJ);
}

// The better of two boxes by exact objective: larger, then the earlier (duration
// index, start) -- the reference's first-wins order.  key < 0: no box.
__device__ __forceinline__ void keep_better(double& v, int& key, double ov, int okey) {
    if (okey >= 0 && ov > -CUDART_INF && (key < 0 || ov > v || (ov == v && okey < key))) {
        v = ov;
        key = okey;
    }
}

// ---- fold -----------------------------------------------------------------------

// NR time-consecutive points of one lane: the time offset and, ready to add, the
// words (or FP64 sums) of the point's contribution.
template <int MODE, int NR>
struct PointRegs {
    static constexpr int kW = point_words<MODE>();
    double x[NR];
    uint32_t w[kW > 0 ? NR : 1][kW > 0 ? kW : 1];
    double rv[kW > 0 ? 1 : NR], iv[kW > 0 ? 1 : NR];
};

// The words of the point in slot `i`, nothing when !ok.
template <int MODE, int NR>
__device__ __forceinline__ void load_words(const BatchArgs& a, int64_t i, bool ok,
                                           PointRegs<MODE, NR>& p, int r) {
    if constexpr (one_weight<MODE>()) {
        const int32_t v = ok ? __ldg(a.pay_r + i) : 0;
        if constexpr (MODE == MODE_PAIR) {
            p.w[r][0] = (uint32_t)v;
            p.w[r][1] = ((uint32_t)(v >> (32 - kPairBits)) << kPairBits) | (ok ? 1u : 0u);
        } else {
            p.w[r][0] = (uint32_t)v & ((1u << kHalfBits) - 1u);
            p.w[r][1] = (uint32_t)(v >> kHalfBits);
            p.w[r][2] = ok ? 1u : 0u;
        }
    } else if constexpr (MODE != MODE_GENERAL) {
        const long long rq = ok ? __ldg(reinterpret_cast<const long long*>(a.r64) + i) : 0ll;
        const long long iq = ok ? __ldg(reinterpret_cast<const long long*>(a.iv64) + i) : 0ll;
        constexpr int kStep = MODE == MODE_WIDE ? kWideBits : kExactBits;
        constexpr int kHalf = point_words<MODE>() / 2;
#pragma unroll
        for (int w = 0; w < kHalf; ++w) {
            p.w[r][w] = (uint32_t)(rq >> (w * kStep));
            p.w[r][kHalf + w] = (uint32_t)(iq >> (w * kStep));
        }
    } else {
        p.rv[r] = ok ? __ldg(a.r64 + i) : 0.0;
        p.iv[r] = ok ? __ldg(a.iv64 + i) : 0.0;
    }
}

// This lane's r-th point of the block of kThreads * NR points at `base` (may lie past the
// last point): slot base + r * kThreads + tid of a full chunk (stored lane-interleaved),
// time index base + tid * NR + r of the tail.
template <int NR, bool TAIL>
__device__ __forceinline__ int point_index(int base, int r) {
    return TAIL ? base + (int)threadIdx.x * NR + r : base + r * kThreads + (int)threadIdx.x;
}

// The lane's points; a tail slot past the last point repeats that point's time with
// nothing to add.
template <int MODE, int NR, bool TAIL>
__device__ __forceinline__ void load_points(const BatchArgs& a, const CurveDesc& c, int base,
                                            PointRegs<MODE, NR>& p) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int j = point_index<NR, TAIL>(base, r);
        const int64_t i = c.point_off + (TAIL ? min(j, c.n_points - 1) : j);
        p.x[r] = __ldg(a.tau + i);
        load_words<MODE, NR>(a, i, !TAIL || j < c.n_points, p, r);
    }
}

template <int N>
__device__ __forceinline__ void add_words(uint32_t rec, uint32_t plane, const uint32_t (&w)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) red_add_u32(rec + k * plane, w[k]);
}

// One point's contribution to the record at shared address `rec`.
template <int MODE, int NR>
__device__ __forceinline__ void add_point(uint32_t rec, uint32_t plane,
                                          const PointRegs<MODE, NR>& p, int r, int32_t* flag) {
    if constexpr (MODE == MODE_GENERAL) {
        shared_add_f64(rec, p.rv[r], flag);
        shared_add_f64(rec + 8, p.iv[r], flag);
    } else {
        add_words(rec, plane, p.w[r]);
    }
}

template <int MODE>
__device__ __host__ constexpr uint32_t bin_stride() {
    return MODE == MODE_GENERAL ? 16u : 4u;
}

// Where the fold's list of open points begins: past the histograms (at the end of the memory,
// which is no list, for more points than an entry can name).
template <int MODE>
__device__ __forceinline__ uint32_t open_list(const Tile& tl, uint32_t smem_s,
                                              uint32_t smem_bytes) {
    return smem_s + (tl.curve.n_points < (1 << kOpenBits) - kChunk
                         ? (uint32_t)tl.p_count * hist_period_bytes<MODE>(tl.seg.hist_len)
                         : smem_bytes);
}

// One point at period q that the fast fold leaves open, by the reference's IEEE chain: moved
// from the bin the fast fold gave it to the reference's (the sums are integers modulo 2^32, so
// taking its words out again leaves no trace), or added there (GENERAL, where the fold leaves
// it out).  What the reference never reads, bins past n_bins, is dropped.
template <int MODE>
__device__ __forceinline__ void settle_point(const Tile& tl, int fast_bin, double x,
                                             const PointRegs<MODE, 1>& p, int q, uint32_t hist_s,
                                             int32_t* flag) {
    const uint32_t hq = hist_s + (uint32_t)q * hist_period_bytes<MODE>(tl.seg.hist_len);
    const uint32_t plane = plane_bytes<MODE>(tl.seg.hist_len);
    constexpr uint32_t kB = bin_stride<MODE>();
    const int e = fold_exact(x, tl.per[q], tl.seg.bin_duration, tl.seg.width);
    if constexpr (MODE != MODE_GENERAL) {
        if (e == fast_bin) return;
        constexpr int kW = point_words<MODE>();
        uint32_t out[kW];
#pragma unroll
        for (int k = 0; k < kW; ++k) out[k] = 0u - p.w[0][k];
        add_words<kW>(hq + kB * (uint32_t)fast_bin, plane, out);
    }
    if (e <= tl.nb[q]) add_point<MODE, 1>(hq + kB * (uint32_t)e, plane, p, 0, flag);
}

// The points j, j + step, ... of the curve, `count` of them, at those of the periods q_mask at
// which they are open.
template <int MODE>
__device__ __noinline__ void settle_open(const BatchArgs* a, const Tile* tl, int j, int count,
                                         int step, uint32_t q_mask, uint32_t hist_s) {
    const SegmentDesc& g = tl->seg;
    const FoldConst fc(g.frac_bits, g.margin_u, g.margin_phi, true);
    for (; count > 0; --count, j += step) {
        if (j >= tl->curve.n_points) return;        // (a tail's slots past the last point)
        const int64_t i = tl->curve.point_off + j;
        const double x = __ldg(a->tau + i);
        PointRegs<MODE, 1> p;
        load_words<MODE, 1>(*a, i, true, p, 0);
        for (uint32_t m = q_mask; m != 0u; m &= m - 1u) {
            const int q = __ffs(m) - 1;
            const uint32_t v = fc.position(x, tl->freq[q], tl->scale[q]);
            if (fc.edge(v) >= fc.limit)
                settle_point<MODE>(*tl, (int)(v >> fc.fb) + 1, x, p, q, hist_s, a->error_flag);
        }
    }
}

// Fold this lane's NR points into the histograms of the tile's pt periods.
// Bound by the shared-memory pipe (the reductions and their bank conflicts: 3.8
// wavefronts each on a survey cadence), then by issue.
// MERGE: a lane's points are consecutive in time, so where a bin is wider than the
// sampling each run of equal bins adds its sums once; elsewhere the comparisons only
// cost (one-weight batch of 16 curves, 50,000 periods: 27.7 ms without, 29.8 with).
//
// Open points (not decided by the fast fold: 2 in 10^4 of a survey cadence, those on bin
// edges; many where a cadence meets the edges, as round times and durations do) are added to
// the fast fold's bin like the others (GENERAL: left out) and put on a list, which the CTA
// settles at the end, a point a thread; a lane that finds the list full settles its own after
// the block.  Folding them here, in whatever form, took a call inside the loop, whose calling
// convention halves the registers that stay live (4 four-year curves 53.7 ms so, 48.7 ms with
// the list; 16 curves of the batched workload 18.3 -> 16.7 ms).  The list takes what shared
// memory the histograms leave: with 512 entries and the lanes past them left to themselves,
// 4 curves of 60,000 points at a tenth of a bin, 4,000 periods, took 1.63 ms, 1.38 ms so;
// 16 curves of 4,000 points, all on edges, 900 periods, 1.24 ms, 0.64 ms so.
template <int MODE, int NR, bool TAIL, bool MERGE>
__device__ __forceinline__ uint32_t fold_points(const BatchArgs& a, TileShared& sh, const Tile& s,
                                                uint32_t hist_s, const PointRegs<MODE, NR>& p,
                                                int base, int pt, int hl) {
    const SegmentDesc& g = s.seg;
    const FoldConst fc(g.frac_bits, g.margin_u, g.margin_phi, true);
    const uint32_t plane = plane_bytes<MODE>(hl);
    const uint32_t pbytes = hist_period_bytes<MODE>(hl);
    constexpr uint32_t kB = bin_stride<MODE>();
    uint32_t hq = hist_s;
    uint32_t lost = 0u;             // periods whose open points found the list full
    for (int q = 0; q < pt; ++q, hq += pbytes) {
        const double f = s.freq[q];
        const uint32_t S = s.scale[q];
        uint32_t rec[NR], worst = 0u, skip = 0u;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint32_t v = fc.position(p.x[r], f, S);
            worst = max(worst, fc.edge(v));
            rec[r] = hq + kB + (v >> fc.fb) * kB;
            // (formed here once where runs are merged: left to the compiler they are formed
            // behind the branch, from positions that take the registers meanwhile; 4 four-year
            // curves 47.7 -> 46.8 ms.  Without runs, or with six words, it costs up to 1%)
            if (MERGE && MODE != MODE_EXACT) asm("" : "+r"(rec[r]));
        }
        if (__builtin_expect(worst >= fc.limit, 0)) {
            uint32_t open = 0u;
#pragma unroll
            for (int r = NR - 1; r >= 0; --r)
                open = open + open + (fc.edge(fc.position(p.x[r], f, S)) >= fc.limit ? 1u : 0u);
            if (MODE == MODE_GENERAL) skip = open;
            // (a full list is not counted further: open_at stays below the list's end plus the
            // CTA's points in flight, however many points are open)
            const uint32_t end = hist_s + a.smem_bytes, bytes = 4u * (uint32_t)__popc(open);
            uint32_t at = end;
            if (*static_cast<volatile uint32_t*>(&sh.open_at) < end)
                at = atomicAdd(&sh.open_at, bytes);
            if (at + bytes <= end) {
                for (; open != 0u; at += 4u, open &= open - 1u)
                    st_u32(at, ((uint32_t)q << kOpenBits) |
                                   (uint32_t)point_index<NR, TAIL>(base, __ffs(open) - 1));
            } else {
                lost |= 1u << q;
                for (; at < end; at += 4u) st_u32(at, kNoPoint);
            }
        }
        if constexpr (MODE == MODE_GENERAL) {
#pragma unroll
            for (int r = 0; r < NR; ++r)
                if (!(skip >> r & 1u)) add_point<MODE, NR>(rec[r], plane, p, r, a.error_flag);
        } else if constexpr (!MERGE) {
#pragma unroll
            for (int r = 0; r < NR; ++r) add_words(rec[r], plane, p.w[r]);
        } else {
            constexpr int kW = point_words<MODE>();
            uint32_t run[kW];
#pragma unroll
            for (int k = 0; k < kW; ++k) run[k] = p.w[0][k];
#pragma unroll
            for (int r = 1; r < NR; ++r) {
                if (rec[r] != rec[r - 1]) {
                    add_words<kW>(rec[r - 1], plane, run);
#pragma unroll
                    for (int k = 0; k < kW; ++k) run[k] = 0u;
                }
#pragma unroll
                for (int k = 0; k < kW; ++k) run[k] += p.w[r][k];
            }
            add_words<kW>(rec[NR - 1], plane, run);
        }
    }
    return lost;
}

// Fold the block of kThreads * NR points at `base`; lanes past the tail's last
// point sit it out.
template <int MODE, int NR, bool TAIL, bool MERGE>
__device__ __forceinline__ void fold_block(const BatchArgs& a, TileShared& sh, const Tile& s,
                                           uint32_t hist_s, int base, int pt, int hl) {
    if (TAIL && base + (int)threadIdx.x * NR >= s.curve.n_points) return;
    uint32_t lost;
    {
        PointRegs<MODE, NR> p;
        load_points<MODE, NR, TAIL>(a, s.curve, base, p);
        lost = fold_points<MODE, NR, TAIL, MERGE>(a, sh, s, hist_s, p, base, pt, hl);
    }
    // the list was full: this lane's open points of those periods now
    if (lost != 0u)
        settle_open<MODE>(&a, &s, point_index<NR, TAIL>(base, 0), NR, TAIL ? 1 : kThreads, lost,
                          hist_s);
}

// Fold the curve into the histograms of a tile whose segment has no provable fast fold (more
// cycles than it covers): the reference's IEEE chain for every point and period.  Bound by
// its two divisions, of which four points keep as many chains going in a lane.
template <int MODE>
__device__ __noinline__ void fold_curve_exactly(const BatchArgs* a, const Tile* tl,
                                                uint32_t hist_s) {
    constexpr int NR = 4;
    const int pt = tl->p_count, n = tl->curve.n_points, width = tl->seg.width;
    const uint32_t plane = plane_bytes<MODE>(tl->seg.hist_len);
    const uint32_t pbytes = hist_period_bytes<MODE>(tl->seg.hist_len);
    const double bin = tl->seg.bin_duration;
    for (int j0 = (int)threadIdx.x; j0 < n; j0 += kThreads * NR) {
        PointRegs<MODE, NR> p;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int j = j0 + r * kThreads;
            const int64_t i = tl->curve.point_off + min(j, n - 1);
            p.x[r] = __ldg(a->tau + i);
            load_words<MODE, NR>(*a, i, j < n, p, r);
        }
        uint32_t hq = hist_s;
        for (int q = 0; q < pt; ++q, hq += pbytes) {
            const double P = tl->per[q];
            const int nb = tl->nb[q];
            int e[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) e[r] = fold_exact(p.x[r], P, bin, width);
#pragma unroll
            for (int r = 0; r < NR; ++r)        // (the reference never reads a bin past n_bins)
                if (j0 + r * kThreads < n && e[r] <= nb)
                    add_point<MODE, NR>(hq + bin_stride<MODE>() * (uint32_t)e[r], plane, p, r,
                                        a->error_flag);
        }
    }
}

// Fold the curve into the histograms of the tile.
template <int MODE>
__device__ __forceinline__ void fold_curve(const BatchArgs& a, TileShared& s, const Tile& tl,
                                           uint32_t smem_s) {
    if (!tl.seg.fast_fold) {
        fold_curve_exactly<MODE>(&a, &tl, smem_s);
        return;
    }
    const int pt = tl.p_count, hl = tl.seg.hist_len, n = tl.curve.n_points;
    int base = 0;
    if (MODE != MODE_GENERAL && tl.seg.bin_duration > 1.5f * tl.curve.gap)
        for (; base + kChunk <= n; base += kChunk)
            fold_block<MODE, kPts, false, true>(a, s, tl, smem_s, base, pt, hl);
    else
        for (; base + kChunk <= n; base += kChunk)
            fold_block<MODE, kPts, false, false>(a, s, tl, smem_s, base, pt, hl);
    // the tail: fewer points a lane when few are left, so that more warps share them
    const int left = n - base;
    if (left > 4 * kThreads)
        fold_block<MODE, kPts, true, false>(a, s, tl, smem_s, base, pt, hl);
    else if (left > 2 * kThreads)
        fold_block<MODE, 4, true, false>(a, s, tl, smem_s, base, pt, hl);
    else if (left > 0)
        fold_block<MODE, 2, true, false>(a, s, tl, smem_s, base, pt, hl);
    __syncthreads();
    const uint32_t end = min(s.open_at, smem_s + a.smem_bytes);
    for (uint32_t at = open_list<MODE>(tl, smem_s, a.smem_bytes) + 4u * threadIdx.x; at < end;
         at += 4u * kThreads) {
        const uint32_t p = ld_u32(at);
        if (p != kNoPoint)
            settle_open<MODE>(&a, &tl, (int)(p & ((1u << kOpenBits) - 1u)), 1, 1,
                              1u << (p >> kOpenBits), smem_s);
    }
}

// ---- prefix sums -----------------------------------------------------------------

// The FP32 screen copy of one prefix: {t, weight}, and the magnitude that bounds t's
// rounding error.
template <int MODE>
__device__ __forceinline__ float2 screen_record(long long r, long long w, float cfrac, float& tm) {
    if (one_weight<MODE>()) {
        // the screen's t is centred by ybar itself: the stored prefix minus
        // center_frac per point, in FP32.  It is within 2^-23 (|pf| + 2 |cf|) of the
        // exact value (pf and t round once each, cf twice), |pf| <= |t| + |cf|, and
        // |cf| <= |cfrac| n over a whole scan (2 n with the pad): the caller adds that
        const float cnt = (float)(uint32_t)(r & ((1ll << kCountShift) - 1));
        const float t = fmaf(-cfrac, cnt, (float)(r >> kCountShift));
        tm = fabsf(t);
        return make_float2(t, cnt);
    }
    const float t = (float)r;
    tm = fabsf(t);
    // exact scaling by a power of two
    return make_float2(t, (float)w * (MODE == MODE_EXACT ? 0x1p-20f : 0x1p-13f));
}

// Integer modes: the wrap pad (bins 1..o repeated in nb-o..nb-1, _bls_core.py:377-381)
// and prefix sums of one period, in place, with the FP32 screen copy.  Returns after
// the period's second barrier; `first` runs after its first one (what the previous
// period left to do once every warp has finished its sweep).  A lane owns K
// consecutive bins, K odd so that the lanes' words sit in distinct banks, and holds
// their running sums in registers between the two barriers, so each bin is read once
// and written once; more than kThreads * kRegBins bins go in several such blocks.
template <int MODE, typename F>
__device__ __forceinline__ void scan_period(TileShared& s, const Tile& tl, const Hist& h, uint32_t scr_s, int L,
                                            int o, F&& first) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = L - 1;
    constexpr int kW = point_words<MODE>();
    constexpr bool kTwo = !one_weight<MODE>();
    const bool single = L <= kThreads * kRegBins;
    // several blocks, or a pad that overlaps its source: copied before the scan (the
    // overlapping one by one thread in the reference's order); else the lane that owns
    // a pad bin reads the bin it repeats (no word changes before the first barrier)
    const bool overlap = nb - o <= o;
    const bool copied = overlap || !single;
    if (copied) {
        auto copy_bin = [&](int dst, int src) {
            if (dst < 0 || dst >= tl.seg.width || dst > tl.seg.hist_len || src > tl.seg.hist_len) return;
            const uint32_t rd = h.base + 4u * (uint32_t)dst, rs = h.base + 4u * (uint32_t)src;
#pragma unroll
            for (int k = 0; k < kW; ++k) st_u32(rd + k * h.plane, ld_u32(rs + k * h.plane));
        };
        if (overlap) {
            if (tid == 0)
                for (int k = 0; k < o; ++k) copy_bin(nb - o + k, 1 + k);
        } else {
            for (int k = tid; k < o; k += kThreads) copy_bin(nb - o + k, 1 + k);
        }
        __syncthreads();
    }
    const int K = single ? (((L + kThreads - 1) / kThreads) | 1) : kRegBins;
    const float cfrac = (float)tl.curve.center_frac;
    long long carry_r = 0, carry_w = 0;
    float tmax = 0.0f;
    int par = 0;
    for (int b0 = 0; b0 < L; b0 += kThreads * K, par ^= 1) {
        const int l0 = b0 + tid * K;
        long long ar[kRegBins], aw[kTwo ? kRegBins : 1];
        long long run_r = 0, run_w = 0;
#pragma unroll
        for (int r = 0; r < kRegBins; ++r) {
            if (r < K) {
                const int i = l0 + r;
                if (i < L) {
                    const int src = !copied && i >= nb - o && i < nb ? i - (nb - o) + 1 : i;
                    long long br, bw;
                    bin_sums<MODE>(h, src, br, bw);
                    run_r += br;
                    run_w += bw;
                }
                ar[r] = run_r;
                if (kTwo) aw[kTwo ? r : 0] = run_w;
            }
        }
        long long in_r = run_r, in_w = run_w;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const long long x = __shfl_up_sync(kFull, in_r, k);
            if (lane >= k) in_r += x;
            if (kTwo) {
                const long long y = __shfl_up_sync(kFull, in_w, k);
                if (lane >= k) in_w += y;
            }
        }
        if (lane == 31) {
            s.tot[par][0][warp] = in_r;
            if (kTwo) s.tot[par][1][warp] = in_w;
        }
        __syncthreads();
        if (b0 == 0) first();
        // the warps before this one: lane w takes warp w's total
        long long off_r = lane < kWarps ? s.tot[par][0][lane] : 0ll, off_w = 0ll;
        if (kTwo) off_w = lane < kWarps ? s.tot[par][1][lane] : 0ll;
        if (!single) {          // the block's total, for the next one
            long long all_r = off_r, all_w = off_w;
            all_r = warp_sum(all_r);
            if (kTwo) all_w = warp_sum(all_w);
            if (lane >= warp) off_r = off_w = 0ll;
            off_r = warp_sum(off_r) + carry_r;
            if (kTwo) off_w = warp_sum(off_w) + carry_w;
            carry_r += all_r;
            carry_w += all_w;
        } else {
            if (lane >= warp) off_r = off_w = 0ll;
#pragma unroll
            for (int k = kWarps / 2; k > 0; k >>= 1) {
                off_r += __shfl_xor_sync(kFull, off_r, k);
                if (kTwo) off_w += __shfl_xor_sync(kFull, off_w, k);
            }
            off_r = __shfl_sync(kFull, off_r, 0);
            if (kTwo) off_w = __shfl_sync(kFull, off_w, 0);
        }
        off_r += in_r - run_r;
        off_w += in_w - run_w;
#pragma unroll
        for (int r = 0; r < kRegBins; ++r) {
            const int i = l0 + r;
            if (r < K && i < L) {
                const uint32_t a = h.base + 4u * (uint32_t)i;
                const long long vr = off_r + ar[r], vw = kTwo ? off_w + aw[kTwo ? r : 0] : 0;
                st_planes(a, h.plane, vr);
                if (kTwo) st_planes(a + weight_plane<MODE>() * h.plane, h.plane, vw);
                float tm;
                st_f2(scr_s + 8u * (uint32_t)i, screen_record<MODE>(vr, vw, cfrac, tm));
                tmax = fmaxf(tmax, tm);
            }
        }
    }
    tmax = warp_max(tmax);
    if (lane == 0) s.red_t[warp] = tmax;
    // sentinel records past the last bin: t = NaN fails every screen
    if (tid < kScreenPad) st_f2(scr_s + 8u * (uint32_t)(L + tid), make_float2(CUDART_NAN_F, 0.0f));
    __syncthreads();
}

// GENERAL: the same on FP64 sums.  The lanes' partial sums associate differently from
// one running sum, so at a lane boundary an empty bin could move the FP64 prefix by a
// rounding; the reference's running sum keeps it exactly constant, which makes boxes
// that differ only by empty end bins tie exactly (first wins), so the lanes copy the
// prefix of the last non-empty bin into their leading empty bins (a third barrier).
template <typename F>
__device__ __forceinline__ void scan_period_f64(TileShared& s, const Tile& tl, const Hist& h, uint32_t scr_s, int L,
                                                int o, F&& first) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = L - 1;
    auto copy_bin = [&](int dst, int src) {
        if (dst < 0 || dst >= tl.seg.width || dst > tl.seg.hist_len || src > tl.seg.hist_len) return;
        const uint32_t rd = h.base + 16u * (uint32_t)dst, rs = h.base + 16u * (uint32_t)src;
        st_f64(rd, ld_f64(rs));
        st_f64(rd + 8, ld_f64(rs + 8));
    };
    if (nb - o <= o) {
        if (tid == 0)
            for (int k = 0; k < o; ++k) copy_bin(nb - o + k, 1 + k);
    } else {
        for (int k = tid; k < o; k += kThreads) copy_bin(nb - o + k, 1 + k);
    }
    __syncthreads();
    const int K = ((L + kThreads - 1) / kThreads) | 1;
    const int l0 = min(L, tid * K), l1 = min(L, l0 + K);
    double ur = 0.0, uw = 0.0;
    int lead = 0, last_ne = -1;     // leading empty bins, last non-empty bin of the lane
    for (int i = l0; i < l1; ++i) {
        const uint32_t rec = h.base + 16u * (uint32_t)i;
        const double br = ld_f64(rec), bw = ld_f64(rec + 8);
        ur += br;
        uw += bw;
        if (br != 0.0 || bw != 0.0) last_ne = i;
        else if (last_ne < 0) ++lead;
    }
    double ir = ur, iw = uw;
    int im = last_ne;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const double xr = __shfl_up_sync(kFull, ir, k);
        const double xw = __shfl_up_sync(kFull, iw, k);
        const int xm = __shfl_up_sync(kFull, im, k);
        if (lane >= k) {
            ir += xr;
            iw += xw;
            im = max(im, xm);
        }
    }
    double rr = __shfl_up_sync(kFull, ir, 1), rw = __shfl_up_sync(kFull, iw, 1);
    last_ne = __shfl_up_sync(kFull, im, 1);
    if (lane == 0) {
        rr = rw = 0.0;
        last_ne = -1;
    }
    if (lane == 31) {
        s.tot_d[0][warp] = ir;
        s.tot_d[1][warp] = iw;
        s.red_ne[warp] = im;
    }
    __syncthreads();
    first();
    for (int w = 0; w < warp; ++w) {
        rr += s.tot_d[0][w];
        rw += s.tot_d[1][w];
        last_ne = max(last_ne, s.red_ne[w]);
    }
    float tmax = 0.0f;
    for (int i = l0; i < l1; ++i) {
        const uint32_t rec = h.base + 16u * (uint32_t)i;
        rr += ld_f64(rec);
        rw += ld_f64(rec + 8);
        st_f64(rec, rr);
        st_f64(rec + 8, rw);
        st_f2(scr_s + 8u * (uint32_t)i, make_float2((float)rr, (float)(rw * 0x1p-20)));
        tmax = fmaxf(tmax, fabsf((float)rr));
    }
    tmax = warp_max(tmax);
    if (lane == 0) s.red_t[warp] = tmax;
    if (tid < kScreenPad) st_f2(scr_s + 8u * (uint32_t)(L + tid), make_float2(CUDART_NAN_F, 0.0f));
    __syncthreads();
    if (lead > 0 && last_ne >= 0) {
        const uint32_t rs = h.base + 16u * (uint32_t)last_ne;
        const double pr = ld_f64(rs), pw = ld_f64(rs + 8);
        for (int i = l0; i < l0 + lead; ++i) {
            const uint32_t rec = h.base + 16u * (uint32_t)i;
            st_f64(rec, pr);
            st_f64(rec + 8, pw);
            st_f2(scr_s + 8u * (uint32_t)i, make_float2((float)pr, (float)(pw * 0x1p-20)));
        }
    }
    __syncthreads();
}

// ---- the search --------------------------------------------------------------------

// The last i in [0, n) with a[i * stride] <= v (a[0] <= v), by one warp, 32 at a time.
__device__ __forceinline__ int last_at_most(const int32_t* a, int stride, int n, int v) {
    const int lane = threadIdx.x & 31;
    int lo = 0;
    while (n > 1) {
        const int step = (n + 31) / 32;
        const int i = lane * step;
        const bool le = i < n && __ldg(a + (int64_t)(lo + i) * stride) <= v;
        const int k = __popc(__ballot_sync(kFull, le)) - 1;
        lo += k * step;
        n = min(step, n - k * step);
    }
    return lo;
}

template <typename T>
__device__ __forceinline__ void copy_words(T* to, const T* from, int lane) {
    static_assert(sizeof(T) % 4 == 0, "whole words");
    for (int i = lane; i < (int)(sizeof(T) / 4); i += 32)
        reinterpret_cast<uint32_t*>(to)[i] = __ldg(reinterpret_cast<const uint32_t*>(from) + i);
}

// Persistent search; see the head of this file.  One weight runs three CTAs an SM (80
// registers), per-point weights two.  Bound by latency between its barriers with 24 (16)
// resident warps: neither issue nor the shared-memory pipe is above two thirds busy.
// 96 curves of the batched workload (mean 9,900 points, 50,000 periods): 152.8 ms with
// three words a point, five barriers a period and a screened sweep; 99.4 ms as built.
// 16 curves with per-point errors 52.7 -> 30.3 ms (38-bit weights), 8 with outlying
// errors 56.2 -> 21.3 ms (FP64 sums by compare-and-swap before).
template <int MODE, int OBJ>
__global__ void __launch_bounds__(kThreads, one_weight<MODE>() ? 3 : 2)
    bls_search_kernel(const __grid_constant__ BatchArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ TileShared s;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;

    // Claims the next work item and copies its inputs to tile slot `to`: one warp, while
    // the others search (the chain of dependent loads takes a few microseconds).
    auto fetch = [&](int to) {
        Tile& t = s.tile[to];
        const int it = __shfl_sync(kFull, lane == 0 ? atomicAdd(a.work_counter, 1) : 0, 0);
        if (it >= a.n_items) {
            if (lane == 0) t.item = it;
            return;
        }
        // one grid: the group is a launch parameter; several: a search
        WorkGroup gr = a.group0;
        if (a.n_groups > 1)
            gr = a.groups[last_at_most(&a.groups[0].item_begin, sizeof(WorkGroup) / 4, a.n_groups,
                                       it)];
        const int local = it - gr.item_begin;
        const int r = local / gr.tiles_per_curve;
        const int j = local - r * gr.tiles_per_curve;
        const int32_t* tiles = a.seg_tiles + gr.tiles_begin;
        const int lo = last_at_most(tiles, 1, gr.n_segments, j);
        const int sg = gr.seg_begin + lo;
        const int cap = __ldg(a.seg_cap + sg);
        const int curve = __ldg(a.order + gr.order_begin + r);
        const int p_begin = (j - __ldg(tiles + lo)) * cap;
        copy_words(&t.seg, a.segments + sg, lane);
        copy_words(&t.curve, a.curves + curve, lane);
        __syncwarp();
        const int p_count = min(cap, t.seg.n_periods - p_begin);
        const int64_t g0 = t.seg.period_off + p_begin;
        if (lane < p_count && lane < kMaxTile) {
            t.per[lane] = __ldg(a.period + g0 + lane);
            t.freq[lane] = __ldg(a.freq + g0 + lane);
            t.scale[lane] = __ldg(a.scale + g0 + lane);
            t.nb[lane] = __ldg(a.nbins + g0 + lane);
        }
        const int n_dur = t.seg.n_dur;
        int d = 0;
        if (n_dur > 0 && n_dur <= kMaxDur) d = __ldg(a.dur_bins + t.seg.dur_off + min(lane, n_dur - 1));
        t.dur[lane] = d;
        if (lane < 4) t.dur[kMaxDur + lane] = 0;
        const int d_min = __reduce_min_sync(kFull, d), d_max = __reduce_max_sync(kFull, d);
        if (lane == 0) {
            t.p_begin = p_begin;
            t.p_count = p_count;
            t.d_min = d_min;
            t.d_max = d_max;
            t.item = it;
        }
    };
    constexpr int kFetcher = kWarps - 1;    // its share of a sweep is the smallest
    if (warp == kFetcher) fetch(0);

    for (int slot = 0;; slot ^= 1) {
        __syncthreads();
        const Tile& tl = s.tile[slot];
        if (tl.item >= a.n_items) break;
        if (tid == 0) {
            s.list_n = 0;
            s.rescan = 0u;
        }
        // (what the fold needs is read here and again below, so that little stays in
        // registers over it)
        bool search;
        {
            const int pt = tl.p_count, hl = tl.seg.hist_len, n_dur = tl.seg.n_dur;
            const bool bad = pt < 1 || pt > kMaxTile || n_dur < 0 || n_dur > kMaxDur || hl < 2 ||
                             hl >= (1 << kBoxBits);
            if (bad && tid == 0) atomicExch(a.error_flag, 1);
            search = !bad && !tl.curve.skip && n_dur > 0;
            if (!search) {
                if (!bad && tid < pt) {         // nothing admissible anywhere
                    double* out = a.out + tl.curve.out_off + tl.seg.period_off + tl.p_begin + tid;
                    out[0] = -CUDART_INF;
                    for (int f = 1; f < kFields; ++f) out[f * a.out_stride] = 0.0;
                }
                if (warp == kFetcher) fetch(slot ^ 1);
                continue;
            }
            if (tid < pt) s.thr_bits[tid] = 0u;
        }

        // ---- 1. fold ---------------------------------------------------------
        const uint32_t smem_s = smem_addr(smem);
        if (tid == 0) s.open_at = open_list<MODE>(tl, smem_s, a.smem_bytes);
        {
            const int n16 = (int)(tl.p_count * hist_period_bytes<MODE>(tl.seg.hist_len) / 16u);
            uint4* z = reinterpret_cast<uint4*>(smem);
            for (int i = tid; i < n16; i += kThreads) z[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
        fold_curve<MODE>(a, s, tl, smem_s);
        __syncthreads();

        // ---- 2-3. per period: pad, prefix, sweep --------------------------------
        const int pt = tl.p_count, hl = tl.seg.hist_len, n_dur = tl.seg.n_dur;
        const uint32_t pbytes = hist_period_bytes<MODE>(hl);
        const uint32_t plane = plane_bytes<MODE>(hl);
        const uint32_t scr_s = smem_s + (uint32_t)pt * pbytes;       // FP32 screen copy
        const CurveDesc& cv = tl.curve;
        const int o = tl.seg.oversample;
        auto hist = [&](int q) { return Hist{smem_s + (uint32_t)q * pbytes, plane}; };

        // what a lane keeps of its sweep of one period: its best and second-best group
        // (four widths at one start) by screened key, and the best group's place
        float best = -1.0f, second = -1.0f;
        int place = 0;
        // Once every sweep of period q is done its threshold is final: lanes whose best
        // group reaches it are candidates.  A second group that reaches it too (ties
        // across groups of one lane) or a full list leaves the period to the CTA.
        auto submit = [&](int q) {
            const float Lc = __uint_as_float(s.thr_bits[q]);
            if (best >= Lc) {
                const int pos = second >= Lc ? kList : atomicAdd(&s.list_n, 1);
                if (pos < kList) s.list[pos] = ((uint32_t)q << 25) | (uint32_t)place;
                else atomicOr(&s.rescan, 1u << q);
            }
            best = second = -1.0f;
        };

        for (int q = 0; q < pt; ++q) {
            const int nb = tl.nb[q];
            const int L = nb + 1;
            const Hist h = hist(q);
            auto previous = [&] { if (q > 0) submit(q - 1); };
            if constexpr (MODE == MODE_GENERAL) scan_period_f64(s, tl, h, scr_s, L, o, previous);
            else scan_period<MODE>(s, tl, h, scr_s, L, o, previous);
            float tmax = 0.0f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) tmax = fmaxf(tmax, s.red_t[w]);

            if (a.debug_prefix != nullptr && q == 0) {   // test hook: this period's prefixes
                for (int i = tid; i < L; i += kThreads) {
                    double r_i, w_i;
                    if constexpr (one_weight<MODE>()) {
                        const long long v = prefix_r(h, i);
                        const double cnt = (double)(v & ((1ll << kCountShift) - 1));
                        r_i = ldexp((double)(v >> kCountShift), -cv.e_r) + cv.center * cnt;
                        w_i = cnt * cv.w_uniform;
                    } else if constexpr (MODE == MODE_GENERAL) {
                        w_i = ldexp(ld_f64(h.base + 16u * (uint32_t)i + 8u), -cv.e_i);
                        r_i = ldexp(ld_f64(h.base + 16u * (uint32_t)i), -cv.e_r) + cv.ybar * w_i;
                    } else {
                        w_i = ldexp((double)prefix_w<MODE>(h, i), -cv.e_i);
                        r_i = ldexp((double)prefix_r(h, i), -cv.e_r) + cv.ybar * w_i;
                    }
                    a.debug_prefix[i] = r_i;
                    a.debug_prefix[hl + i] = w_i;
                }
            }

            // Bound on the FP32 error of a box's t: 2^-21 of the largest prefix
            // (one rounding per prefix, one per difference: 2^-22, 2x slack; one
            // weight: 1.5 * 2^-22 of the largest tm, 1.33x slack), and never 0, so
            // that a box of exactly the mean counts as the dip it is.  Ei: the same of
            // the weight inside or outside a box, in units of 2^-24 of the total Wt: a
            // prefix is up to 2 Wt (the pad counts bins 1..o again) and rounds by 2, two of
            // them by 4; their difference by 1, Wt by 1 and Wt less the difference by 1,
            // 7 in all where 8 are taken.
            if (one_weight<MODE>())
                tmax += 4.0f * fabsf((float)cv.center_frac) * (float)cv.n_points;
            const float Et =
                cv.exact_all ? CUDART_INF_F : tmax * (1.0f / 2097152.0f) + 0.0625f;
            constexpr int kShift = screen_shift<MODE>();
            const float Wt = one_weight<MODE>() ? (float)cv.n_points
                                                : (float)ldexp(cv.i_total, -kShift);
            const float Ei = one_weight<MODE>() ? 0.0f : Wt * (1.0f / 2097152.0f);
            const float small = cv.w_small;

            // Sweep: starts outer, 32 per warp and step; widths inner in groups of four
            // (one broadcast load).  Maximising snr (likelihood) is maximising the key
            // t^2 / (iv_in iv_out) (t^2 / (iv_in iv_out^2)) over dips, t = y_in - ybar
            // iv_in.  th = Et - t bounds |t_exact| for every dip and den is at most the
            // box's exact denominator, so th |th| / den bounds its key from above: a
            // lane keeps the largest per group, and its place.  One weight: counts are
            // exact in FP32, and th = c Et - t is 0 for an empty box (key NaN, which
            // the maximum drops).  Per-point weights: each side is lowered by the
            // weights' FP32 error; a box that this leaves without a bound, and that is
            // not certainly empty, is evaluated in FP64 at once.  In a step that some
            // width does not fit, it reads the sentinel record and its key is NaN.
            // Screened in order with a shared threshold instead (what passes bounded and
            // listed), the passing boxes alone took as long as the sweep itself.
            double ex_v = -CUDART_INF;
            int ex_box = -1;
            {
                const int nmax_all = nb - tl.d_min;
                const int n_all = nb - tl.d_max;    // every width fits a step below this
                const uint32_t sent = scr_s + 8u * (uint32_t)L;    // first sentinel record
                // the largest key of four widths at this lane's start
                auto group = [&](auto fits_all, int n0, int g, uint32_t sa, float2 na,
                                 float& den_min) -> float {
                    const int4 dg = *reinterpret_cast<const int4*>(&tl.dur[g]);
                    const int dk[4] = {dg.x, dg.y, dg.z, dg.w};
                    float m = -1.0f;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        uint32_t sb = sa + 8u * (uint32_t)dk[k];
                        if (!decltype(fits_all)::value)
                            sb = (dk[k] < nb) & (n0 <= nb - dk[k]) ? sb : sent;
                        const float2 diff = add_f2(ld_f2(sb), na);
                        const float t = diff.x, c = diff.y;
                        float th, den;
                        if constexpr (one_weight<MODE>()) {
                            th = fmaf(c, Et, -t);
                            const float oc = Wt - c;
                            den = OBJ ? c * oc * oc : c * oc;
                        } else {
                            th = Et - t;
                            const float il = c - Ei, ol = fmaxf(Wt - c - Ei, 0.0f);
                            den = OBJ ? il * ol * ol : il * ol;
                            if (c > small) den_min = fminf(den_min, den);
                        }
                        m = fmaxf(m, th * fabsf(th) * rcp_approx(den));
                    }
                    return m;
                };
                for (int n0 = warp * 32; n0 <= nmax_all; n0 += kThreads) {
                    const uint32_t sa = scr_s + 8u * (uint32_t)(n0 + lane);
                    const float2 x = ld_f2(sa);
                    const float2 na = make_float2(-x.x, -x.y);
                    for (int g = 0; g < n_dur; g += 4) {
                        float den_min = 1.0f;
                        const float m = n0 < n_all
                                            ? group(std::true_type{}, n0, g, sa, na, den_min)
                                            : group(std::false_type{}, n0, g, sa, na, den_min);
                        second = fmaxf(second, fminf(m, best));
                        if (m > best) {
                            best = m;
                            place = (g << kBoxBits) | (n0 + lane);
                        }
                        if constexpr (!one_weight<MODE>()) {
                            if (!(den_min > 0.0f)) {
                                const int n = n0 + lane;
#pragma unroll 1
                                for (int k = 0; k < 4; ++k) {
                                    const int d = tl.dur[g + k];
                                    if (d >= nb || n > nb - d) continue;
                                    const float2 diff = add_f2(ld_f2(sa + 8u * (uint32_t)d), na);
                                    const float il = diff.y - Ei;
                                    if (il * (Wt - diff.y - Ei) > 0.0f && il > 0.0f) continue;
                                    // an empty box is exactly 0 in the prefix
                                    bool holds;
                                    if constexpr (MODE == MODE_GENERAL)
                                        holds = ld_f64(h.base + 16u * (uint32_t)(n + d) + 8u) !=
                                                ld_f64(h.base + 16u * (uint32_t)n + 8u);
                                    else holds = prefix_w<MODE>(h, n + d) != prefix_w<MODE>(h, n);
                                    if (holds)
                                        keep_better(ex_v, ex_box,
                                                    exact_objective<MODE, OBJ>(h.base, h.plane, &cv,
                                                                               n, d),
                                                    ((g + k) << kBoxBits) | n);
                                }
                            }
                        }
                    }
                }
            }

            // A warp whose best group may be the period's publishes the largest key lower
            // bound of its boxes that are certainly admissible dips.
            {
                const uint32_t top =
                    __reduce_max_sync(kFull, __float_as_uint(fmaxf(best, 0.0f)));
                if (top > *reinterpret_cast<volatile uint32_t*>(&s.thr_bits[q])) {
                    const unsigned at = __ballot_sync(kFull, __float_as_uint(best) == top);
                    const int pl = __shfl_sync(kFull, place, __ffs(at) - 1);
                    const int n = pl & ((1 << kBoxBits) - 1);
                    const int d = tl.dur[(pl >> kBoxBits) + (lane & 3)];
                    float lo = 0.0f;
                    if (d < nb && n <= nb - d) {
                        const uint32_t sa = scr_s + 8u * (uint32_t)n;
                        const float2 x = ld_f2(sa), y = ld_f2(sa + 8u * (uint32_t)d);
                        const float t = y.x - x.x, c = y.y - x.y, ov = Wt - c;
                        const float ih = c + Ei, oh = ov + Ei;
                        const float den = OBJ ? ih * oh * oh : ih * oh;
                        bool valid = (c > 0.0f) & (ov > 0.0f);
                        if constexpr (!one_weight<MODE>()) {
                            const float floor_q =
                                (float)ldexp(cv.ivar_floor, cv.e_i - kShift) * (1.0f + 1e-3f);
                            valid = (c - Ei >= floor_q) & (ov - Ei >= floor_q) & (c > Ei) & (ov > Ei);
                        }
                        const float tl_ = fmaxf(-t - Et, 0.0f);
                        const float key = tl_ * tl_ * rcp_approx(den) * (1.0f - 2.0f * kRel);
                        if (valid & (key < CUDART_INF_F)) lo = key;
                    }
                    const uint32_t lo_top = __reduce_max_sync(kFull, __float_as_uint(lo));
                    if (lane == 0 && lo_top > 0u) atomicMax(&s.thr_bits[q], lo_top);
                }
            }
            if (q == 0 && warp == kFetcher) fetch(slot ^ 1);
            if constexpr (!one_weight<MODE>()) {
                // the warp's best box without a bound is a candidate as it stands
                if (__any_sync(kFull, ex_box >= 0)) {
#pragma unroll
                    for (int k = 16; k > 0; k >>= 1) {
                        const double ov = __shfl_xor_sync(kFull, ex_v, k);
                        const int ob = __shfl_xor_sync(kFull, ex_box, k);
                        keep_better(ex_v, ex_box, ov, ob);
                    }
                    if (lane == 0 && ex_box >= 0) {
                        const int pos = atomicAdd(&s.list_n, 1);
                        if (pos < kList)
                            s.list[pos] = ((uint32_t)q << 25) | (uint32_t)(ex_box & ~(3 << kBoxBits));
                        else atomicOr(&s.rescan, 1u << q);
                    }
                }
            }
        }
        __syncthreads();
        submit(pt - 1);
        __syncthreads();

        // Each period's winner: the boxes of its candidate groups (one or two, more in
        // near ties) with the reference's formulas on the exact sums, a box a lane, in
        // its first-wins order.
        const int n_list = min(s.list_n, kList);
        for (int q = warp; q < pt; q += kWarps) {
            double v = -CUDART_INF;
            int key = -1;
            const Hist h = hist(q);
            const int nb = tl.nb[q];
            for (int e = lane >> 2; e < n_list; e += 8) {
                const uint32_t c = s.list[e];
                if ((int)(c >> 25) != q) continue;
                const int box = (int)(c & ((1u << 25) - 1u)) + ((lane & 3) << kBoxBits);
                const int d = tl.dur[box >> kBoxBits], n = box & ((1 << kBoxBits) - 1);
                if (d < nb && n <= nb - d)
                    keep_better(v, key, exact_objective<MODE, OBJ>(h.base, h.plane, &cv, n, d), box);
            }
            __syncwarp();
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) {
                const double ov = __shfl_xor_sync(kFull, v, k);
                const int ok = __shfl_xor_sync(kFull, key, k);
                keep_better(v, key, ov, ok);
            }
            if (lane == 0) s.win[q] = key;
        }
        __syncthreads();

        // periods of more candidates than that (a constant flux, sums outside FP32's
        // range): every box in FP64, by the whole CTA
        if (s.rescan != 0u) {
            for (int q = 0; q < pt; ++q) {
                if (!(s.rescan >> q & 1u)) continue;
                const Hist h = hist(q);
                const int nb = tl.nb[q];
                double v = -CUDART_INF;
                int key = -1;
                for (int k = 0; k < n_dur; ++k) {
                    const int d = tl.dur[k];
                    for (int n = tid; d < nb && n <= nb - d; n += kThreads)
                        keep_better(v, key, exact_objective<MODE, OBJ>(h.base, h.plane, &cv, n, d),
                                    (k << kBoxBits) | n);
                }
                __syncwarp();
#pragma unroll
                for (int k = 16; k > 0; k >>= 1) {
                    const double ov = __shfl_xor_sync(kFull, v, k);
                    const int ok = __shfl_xor_sync(kFull, key, k);
                    keep_better(v, key, ov, ok);
                }
                if (lane == 0) {
                    s.red_v[warp] = v;
                    s.red_box[warp] = key;
                }
                __syncthreads();
                if (tid == 0) {
                    for (int w = 1; w < kWarps; ++w) keep_better(v, key, s.red_v[w], s.red_box[w]);
                    s.win[q] = key;
                }
                __syncthreads();
            }
        }

        // ---- 4. the tile's seven output fields, one thread per period ----------
        if (tid < pt) {
            const int q = tid;
            double* op = a.out + tl.curve.out_off + tl.seg.period_off + tl.p_begin + q;
            const int64_t ostride = a.out_stride;
            const int box = s.win[q];
            if (box < 0) {
                op[0] = -CUDART_INF;
                for (int f = 1; f < kFields; ++f) op[f * ostride] = 0.0;
            } else {
                const int vn = box & ((1 << kBoxBits) - 1);
                const int d = tl.dur[box >> kBoxBits];
                const BoxSums b = box_sums<MODE>(hist(q), cv, vn, d);
                const double iv_out = b.iv_out;
                const double yin = b.y_in / b.iv_in;
                const double yout = b.y_out / iv_out;
                const double depth = yout - yin;
                const double derr = sqrt(1.0 / b.iv_in + 1.0 / iv_out);
                const double dsnr = depth / derr;
                const double ll = 0.5 * b.iv_in * depth * depth;
                const double bin = tl.seg.bin_duration;
                const double dur = (double)d * bin;
                op[0] = OBJ == 0 ? dsnr : ll;
                op[1 * ostride] = depth;
                op[2 * ostride] = derr;
                op[3 * ostride] = dsnr;
                op[4 * ostride] = dur;
                op[5 * ostride] = fmod((double)vn * bin + 0.5 * dur, tl.per[q]) + cv.t_min;
                op[6 * ostride] = ll;
            }
        }
    }
}

// ---- per-curve result rows: SDE normalisation and alias-diverse peaks -------
// The reference's row (src/cuperiod/batch/io.py:507-571) ranks the peaks of the
// assembled spectrum (methods/bls.py:274-301): power with non-finite values as
// 0, SDE = (power - mean) / std, candidates = interior local maxima in ascending
// frequency (strictly above the lower-frequency neighbour, >= the higher) plus
// the boundary points (core/result.py:369-406), then greedy highest-score
// candidates skipping any alias-related to one already chosen
// (core/peaks.py:128-231).  Greedy selection equals taking, n times, the best
// remaining candidate and dropping every candidate related to it, which is what
// one CTA per curve does here: over a list of the highest-scoring candidates (whole
// score bins, so that every candidate outside it scores less), refilled with the next
// bins' when it is used up, and over a bitmap of the others where one bin alone
// exceeds the list.  The grid is in ascending period, so frequency
// order is reversed grid order.
//
// Bound by three passes over the spectrum by one CTA.  Testing every candidate of the
// bitmap against every peak, as the rounds past the list do, took 4.7 ms for 200,000
// periods and 1.6 ms for 96 curves of 50,000; with the list 0.84 and 1.4 ms.

__device__ __forceinline__ double nan_to_zero(double v) { return isfinite(v) ? v : 0.0; }

// is_alias_related(f_new, f_chosen) with the reference's FP64 operations in its
// order (no contraction): duplicate within `sep`, harmonics and subharmonics up
// to `hmax`, sidereal/solar day offsets (x1, x2) and the yearly offset.
__device__ bool alias_related(double fn, double fc, double tol, int hmax, double sep,
                              const double* offs) {
    if (fabs(__dsub_rn(fn, fc)) < sep) return true;
    for (int m = 2; m <= hmax; ++m) {
        const double md = (double)m;
        if (fabs(__dsub_rn(fn, __dmul_rn(md, fc))) < __dmul_rn(md, tol)) return true;
        if (fabs(__dsub_rn(fn, __ddiv_rn(fc, md))) < tol) return true;
    }
    for (int k = 0; k < 5; ++k) {
        const double off = offs[k];
        if (fabs(__dsub_rn(fn, fabs(__dsub_rn(fc, off)))) < tol ||
            fabs(__dsub_rn(fn, __dadd_rn(fc, off))) < tol)
            return true;
    }
    return false;
}

// The alias test of candidates fn against one chosen peak fc, both directions,
// with fc's multiples, subharmonics and offsets computed once per round.  The
// only division per candidate, fn / m in the reverse subharmonic test, is taken
// as fn * (1/m) unless the comparison is within a few ulps of the tolerance,
// where the IEEE quotient decides as in the reference.
struct AliasRound {
    static constexpr int kMaxH = 32;
    double fc, tol, sep;
    int hmax;
    double mfc[kMaxH + 1], mtol[kMaxH + 1], fcm[kMaxH + 1];
    double lo[5], hi[5], off[5];

    __device__ void init(double f, double t, double s, int h, const double* offs) {
        fc = f; tol = t; sep = s; hmax = h;
        for (int m = 2; m <= h; ++m) {
            const double md = (double)m;
            mfc[m] = __dmul_rn(md, f);
            mtol[m] = __dmul_rn(md, t);
            fcm[m] = __ddiv_rn(f, md);
        }
        for (int k = 0; k < 5; ++k) {
            off[k] = offs[k];
            lo[k] = fabs(__dsub_rn(f, offs[k]));
            hi[k] = __dadd_rn(f, offs[k]);
        }
    }
    // is_alias_related(fn, fc) or is_alias_related(fc, fn)
    __device__ bool related(double fn) const {
        if (fabs(__dsub_rn(fn, fc)) < sep) return true;          // either way
        for (int m = 2; m <= hmax; ++m) {
            const double md = (double)m;
            if (fabs(__dsub_rn(fn, mfc[m])) < mtol[m]) return true;
            if (fabs(__dsub_rn(fn, fcm[m])) < tol) return true;
            if (fabs(__dsub_rn(fc, __dmul_rn(md, fn))) < mtol[m]) return true;
            double q = __dmul_rn(fn, __drcp_rn(md));
            const double gap = fabs(__dsub_rn(fc, q));
            if (fabs(gap - tol) <= 8.0 * DBL_EPSILON * fmax(fabs(fc), fmax(fabs(q), tol)))
                q = __ddiv_rn(fn, md);
            if (fabs(__dsub_rn(fc, q)) < tol) return true;
        }
        for (int k = 0; k < 5; ++k) {
            if (fabs(__dsub_rn(fn, lo[k])) < tol || fabs(__dsub_rn(fn, hi[k])) < tol) return true;
            if (fabs(__dsub_rn(fc, fabs(__dsub_rn(fn, off[k])))) < tol ||
                fabs(__dsub_rn(fc, __dadd_rn(fn, off[k]))) < tol)
                return true;
        }
        return false;
    }
};

// Position of grid index j among the reference's candidates: interior maxima in
// ascending frequency, then the lowest-frequency point, then the highest.  Among
// equal scores the later position ranks first (a stable ascending sort, reversed).
__device__ __forceinline__ long long cand_pos(long long j, long long P) {
    if (P == 1) return 0;
    if (j == P - 1) return P;
    if (j == 0) return P + 1;
    return P - 1 - j;
}

constexpr int kRowBins = 2048;          // score bins of the list's threshold
constexpr int kRowList = 2048;          // candidates the list holds

__global__ void __launch_bounds__(kThreads) rows_kernel(
    const double* __restrict__ out, int64_t out_stride, const int64_t* __restrict__ spec_off,
    const int64_t* __restrict__ grid_base, const double* __restrict__ freq_all,
    const double* __restrict__ sep_c,
    const double* __restrict__ tol_c, int n_best, int hmax, int list_cap, int32_t* n_peaks,
    int64_t* index, double* fields) {
    // list_cap scores, frequencies and positions and the bins, then ceil(P / 32) words of
    // candidates
    extern __shared__ __align__(8) unsigned char rows_dyn[];
    double* l_score = reinterpret_cast<double*>(rows_dyn);
    double* l_freq = l_score + list_cap;
    int32_t* l_j = reinterpret_cast<int32_t*>(l_freq + list_cap);       // -1: dropped
    int* s_bins = l_j + list_cap;                        // kRowBins of them with a list
    uint32_t* cand = reinterpret_cast<uint32_t*>(s_bins + (list_cap > 0 ? kRowBins : 0));
    __shared__ double red_d[kWarps];
    __shared__ double red_s[kWarps];
    __shared__ long long red_p[kWarps];
    __shared__ long long red_j[kWarps];
    __shared__ double s_mean, s_std;
    __shared__ long long s_win;
    __shared__ int s_total, s_bin0, s_listed;
    __shared__ AliasRound s_alias;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = blockIdx.x;
    const int64_t so = spec_off[c];
    const int64_t P = spec_off[c + 1] - so;              // curve c's trial periods
    const double* pw = out + so;                         // field 0 (power) of curve c
    const double* freq = freq_all + grid_base[c];        // its grid's RN(1/P)
    const int64_t nw = (P + 31) / 32;
    if (P < 1) {
        if (tid == 0) n_peaks[c] = 0;
        return;
    }
    const double sep = sep_c[c], tol = tol_c[c];
    double offs[5];
    offs[0] = 1.0027379;                                 // sidereal day, cycles/day
    offs[1] = __dmul_rn(2.0, 1.0027379);
    offs[2] = 1.0;                                       // solar day
    offs[3] = 2.0;
    offs[4] = __ddiv_rn(1.0, 365.25);                    // year

    // mean and population standard deviation of the power (two passes); the largest power
    double sum = 0.0, top = -CUDART_INF;
#pragma unroll 4
    for (int64_t j = tid; j < P; j += kThreads) {
        const double v = nan_to_zero(pw[j]);
        sum += v;
        top = fmax(top, v);
    }
    sum = warp_sum(sum);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(kFull, top, o));
    if (lane == 0) {
        red_d[warp] = sum;
        red_s[warp] = top;
    }
    for (int b = tid; b < kRowBins && list_cap > 0; b += kThreads) s_bins[b] = 0;
    if (tid == 0) s_total = s_listed = 0;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < kWarps; ++w) t += red_d[w];
        s_mean = t / (double)P;
    }
    for (int w = 0; w < kWarps; ++w) top = fmax(top, red_s[w]);
    __syncthreads();
    const double mean = s_mean;
    // a score's bin never falls with the score
    const double inv = top > mean && list_cap > 0 ? (kRowBins - 1) / (top - mean) : 0.0;
    auto score_bin = [&](double v) {
        const double b = (v - mean) * inv;
        return b > 0.0 ? min(kRowBins - 1, (int)b) : 0;  // (0 too when inv is not finite)
    };
    // the candidates: bit j % 32 of word j / 32
    double ss = 0.0;
#pragma unroll 2
    for (int64_t j0 = 0; j0 < P; j0 += kThreads) {
        const int64_t j = j0 + tid;
        bool is = false;
        if (j < P) {
            const double v = nan_to_zero(pw[j]);
            const double d = v - mean;
            ss += d * d;
            if (P == 1) {
                is = true;
            } else if (j == P - 1) {                     // lowest frequency
                is = v >= nan_to_zero(pw[j - 1]);
            } else if (j == 0) {                         // highest frequency
                is = v > nan_to_zero(pw[1]);
            } else {                                     // above the lower frequency, >= the higher
                is = (v > nan_to_zero(pw[j + 1])) & (v >= nan_to_zero(pw[j - 1]));
            }
            if (is && list_cap > 0) atomicAdd(&s_bins[score_bin(v)], 1);
        }
        const uint32_t bits = __ballot_sync(kFull, is);
        if (lane == 0 && j < P) {
            cand[j >> 5] = bits;
            if (bits) atomicAdd(&s_total, __popc(bits));
        }
    }
    ss = warp_sum(ss);
    if (lane == 0) red_d[warp] = ss;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < kWarps; ++w) t += red_d[w];
        s_std = sqrt(t / (double)P);
    }
    // The list is filled from the candidates of the highest bins that fit it, which leave the
    // bitmap and the bins' counts; false: not even the highest bin left fits, or none is left.
    int bin0 = kRowBins, rest = 0;
    auto fill = [&] {
        __syncthreads();
        if (tid == 0) s_listed = 0;
        if (warp == 1 && list_cap == 0) {
            if (lane == 0) s_bin0 = kRowBins;
        } else if (warp == 1) {
            constexpr int kPer = kRowBins / 32;
            int mine = 0;
            for (int b = 0; b < kPer; ++b) mine += s_bins[lane * kPer + b];
            int above = mine;                            // of this lane's bins and the higher
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_down_sync(kFull, above, o);
                if (lane + o < 32) above += t;
            }
            const unsigned fits = __ballot_sync(kFull, above <= list_cap);
            const int first = fits ? __ffs(fits) - 1 : 32;      // lanes first.. fit whole
            int n = above - mine, b = lane * kPer + kPer;
            if (lane == first - 1)
                while (n + s_bins[b - 1] <= list_cap) n += s_bins[--b];
            b = __shfl_sync(kFull, b, max(first - 1, 0));
            if (lane == 0) s_bin0 = first == 0 ? 0 : b;
        }
        __syncthreads();
        rest = s_total;
        const int hi = bin0;
        bin0 = s_bin0;
        for (int64_t w = warp; w < nw && bin0 < hi; w += kWarps) {
            const uint32_t bits = cand[w];
            if (!bits) continue;
            const int64_t j = w * 32 + lane;
            bool take = false;
            double v = 0.0;
            if ((bits >> lane) & 1u) {
                v = nan_to_zero(pw[j]);
                take = score_bin(v) >= bin0;
            }
            const uint32_t taken = __ballot_sync(kFull, take);
            if (!taken) continue;
            int at = 0;
            if (lane == 0) {
                at = atomicAdd(&s_listed, __popc(taken));
                cand[w] = bits & ~taken;
            }
            at = __shfl_sync(kFull, at, 0) + __popc(taken & ((1u << lane) - 1u));
            if (take) {
                l_score[at] = v;
                l_freq[at] = freq[j];
                l_j[at] = (int32_t)j;
            }
        }
        for (int b = bin0 + tid; b < hi; b += kThreads) s_bins[b] = 0;
        __syncthreads();
        if (tid == 0) s_total = rest - s_listed;
        return s_listed > 0;
    };

    // the best of the threads' candidates (bs, bp, bj) becomes row r
    auto choose = [&](int r, double bs, long long bp, long long bj) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double os = __shfl_xor_sync(kFull, bs, o);
            const long long op = __shfl_xor_sync(kFull, bp, o);
            const long long oj = __shfl_xor_sync(kFull, bj, o);
            if (oj >= 0 && (bj < 0 || os > bs || (os == bs && op > bp))) { bs = os; bp = op; bj = oj; }
        }
        if (lane == 0) { red_s[warp] = bs; red_p[warp] = bp; red_j[warp] = bj; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kWarps; ++w)
                if (red_j[w] >= 0 && (bj < 0 || red_s[w] > bs || (red_s[w] == bs && red_p[w] > bp))) {
                    bs = red_s[w]; bp = red_p[w]; bj = red_j[w];
                }
            s_win = bj;
            if (bj >= 0) {
                const double f = freq[bj];
                const double v = nan_to_zero(pw[bj]);
                double* fo = fields + ((int64_t)c * n_best + r) * 8;
                fo[0] = __ddiv_rn(1.0, f);                          // period = 1 / frequency
                fo[1] = f;
                fo[2] = v;                                          // power
                fo[3] = out[1 * out_stride + so + bj];              // depth
                fo[4] = out[3 * out_stride + so + bj];              // depth_snr
                fo[5] = out[4 * out_stride + so + bj];              // duration
                fo[6] = out[5 * out_stride + so + bj];              // t0
                fo[7] = s_std > 0.0 ? (v - s_mean) / s_std : 0.0;  // sde
                index[(int64_t)c * n_best + r] = bj;
            }
        }
        __syncthreads();
        return s_win;
    };
    const bool fast = hmax <= AliasRound::kMaxH;
    auto set_peak = [&](double fc) {                     // fc: RN(1/P), numpy's 1.0 / period
        if (fast && tid == 0) s_alias.init(fc, tol, sep, hmax, offs);
        __syncthreads();
    };
    auto related = [&](double fn, double fc) {           // either way
        return fast ? s_alias.related(fn)
                    : alias_related(fn, fc, tol, hmax, sep, offs) ||
                          alias_related(fc, fn, tol, hmax, sep, offs);
    };
    auto drop_rest = [&](long long win) {                // from the bitmap
        const double fc = freq[win];
        set_peak(fc);
        for (int64_t w = tid; w < nw; w += kThreads) {
            uint32_t bits = cand[w], keep = bits;
            while (bits) {
                const int b = __ffs(bits) - 1;
                bits &= bits - 1u;
                const long long j = w * 32 + b;
                if (j == win || related(freq[j], fc)) keep &= ~(1u << b);
            }
            cand[w] = keep;
        }
        __syncthreads();
    };

    auto drop_listed = [&](int listed, long long win) {
        const double fc = freq[win];
        set_peak(fc);
        for (int i = tid; i < listed; i += kThreads)
            if (l_j[i] >= 0 && (l_j[i] == win || related(l_freq[i], fc))) l_j[i] = -1;
        __syncthreads();
    };

    int count = 0;
    while (count < n_best && fill()) {
        const int listed = s_listed;
        // without what the peaks so far exclude
        for (int r = 0; r < count; ++r) drop_listed(listed, index[(int64_t)c * n_best + r]);
        while (count < n_best) {
            // the best remaining candidate: highest score, then later position
            double bs = -CUDART_INF;
            long long bp = -1, bj = -1;
            for (int i = tid; i < listed; i += kThreads) {
                const long long j = l_j[i];
                if (j < 0) continue;
                const double v = l_score[i];
                const long long pos = cand_pos(j, P);
                if (v > bs || (v == bs && pos > bp)) { bs = v; bp = pos; bj = j; }
            }
            const long long win = choose(count, bs, bp, bj);
            if (win < 0) break;
            ++count;
            // drop the winner and every candidate alias-related to it, either way
            drop_listed(listed, win);
        }
    }
    if (count < n_best && rest > 0) {
        // the others, without what the peaks so far exclude
        for (int r = 0; r < count; ++r) drop_rest(index[(int64_t)c * n_best + r]);
        while (count < n_best) {
            double bs = -CUDART_INF;
            long long bp = -1, bj = -1;
            for (int64_t w = tid; w < nw; w += kThreads) {
                uint32_t bits = cand[w];
                while (bits) {
                    const int b = __ffs(bits) - 1;
                    bits &= bits - 1u;
                    const long long j = w * 32 + b;
                    const double v = nan_to_zero(pw[j]);
                    const long long pos = cand_pos(j, P);
                    if (v > bs || (v == bs && pos > bp)) { bs = v; bp = pos; bj = j; }
                }
            }
            const long long win = choose(count, bs, bp, bj);
            if (win < 0) break;
            ++count;
            drop_rest(win);
        }
    }
    if (tid == 0) n_peaks[c] = count;
}

// Phase bins of every point at one period through the fast path with its
// fallback (the tests compare them with the reference's fold bit for bit).
__global__ void fold_bins_kernel(const double* tau, int n, double P, double f, uint32_t S,
                                 double bin, int width, int fb, uint32_t mu, uint32_t mphi,
                                 int fast, int32_t* out, int32_t* used_fast) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    int ind = fold_fast(tau[j], f, S, FoldConst(fb, mu, mphi, fast != 0));
    used_fast[j] = ind >= 0;
    if (ind < 0) ind = fold_exact(tau[j], P, bin, width);
    out[j] = ind;
}

// Per curve: the largest power (non-finite values count as 0, as the
// reference's assembly does before its SDE and peak search) with its first
// index, and the mean and population standard deviation of that power.
__global__ void best_kernel(const double* power, const int64_t* spec_off, int64_t* best_index,
                            double* best_power, double* mean_out, double* std_out) {
    __shared__ double red_s[kWarps];
    __shared__ double red_v[kWarps];
    __shared__ long long red_i[kWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double* p = power + spec_off[blockIdx.x];
    const int64_t n_periods = spec_off[blockIdx.x + 1] - spec_off[blockIdx.x];
    double sum = 0.0, bv = -CUDART_INF;
    long long bi = -1;
    for (int64_t i = tid; i < n_periods; i += kThreads) {
        const double v = p[i];
        const double z = isfinite(v) ? v : 0.0;
        sum += z;
        if (z > bv || (z == bv && i < bi)) { bv = z; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(kFull, sum, o);
        const double ov = __shfl_xor_sync(kFull, bv, o);
        const long long oi = __shfl_xor_sync(kFull, bi, o);
        if (ov > bv || (ov == bv && oi >= 0 && (bi < 0 || oi < bi))) { bv = ov; bi = oi; }
    }
    if (lane == 0) { red_s[warp] = sum; red_v[warp] = bv; red_i[warp] = bi; }
    __syncthreads();
    sum = 0.0;
    bv = -CUDART_INF;
    bi = -1;
    for (int w = 0; w < kWarps; ++w) {
        sum += red_s[w];
        if (red_v[w] > bv || (red_v[w] == bv && red_i[w] >= 0 && (bi < 0 || red_i[w] < bi))) {
            bv = red_v[w];
            bi = red_i[w];
        }
    }
    const double mean = n_periods > 0 ? sum / (double)n_periods : 0.0;
    __syncthreads();
    double ss = 0.0;
    for (int64_t i = tid; i < n_periods; i += kThreads) {
        const double v = p[i];
        const double z = (isfinite(v) ? v : 0.0) - mean;
        ss += z * z;
    }
    ss = warp_sum(ss);
    if (lane == 0) red_s[warp] = ss;
    __syncthreads();
    if (tid == 0) {
        ss = 0.0;
        for (int w = 0; w < kWarps; ++w) ss += red_s[w];
        best_index[blockIdx.x] = bi;
        best_power[blockIdx.x] = bv;
        mean_out[blockIdx.x] = mean;
        std_out[blockIdx.x] = n_periods > 0 ? sqrt(ss / (double)n_periods) : 0.0;
    }
}

}  // namespace

namespace {
using SearchKernel = void (*)(BatchArgs);
template <int OBJ>
SearchKernel search_fn(int mode) {
    switch (mode) {
        case MODE_UNIFORM: return bls_search_kernel<MODE_UNIFORM, OBJ>;
        case MODE_PAIR: return bls_search_kernel<MODE_PAIR, OBJ>;
        case MODE_WIDE: return bls_search_kernel<MODE_WIDE, OBJ>;
        case MODE_EXACT: return bls_search_kernel<MODE_EXACT, OBJ>;
        default: return bls_search_kernel<MODE_GENERAL, OBJ>;
    }
}
const void* search_ptr(int mode, int obj) {
    return (const void*)(obj ? search_fn<1>(mode) : search_fn<0>(mode));
}
}  // namespace

cudaError_t raise_smem_limit(const void* fn, size_t smem) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> limit;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t& have = limit[{dev, fn}];
    if (smem <= have) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) have = smem;
    return e;
}

cudaError_t configure_search(int mode, size_t smem) {
    for (int obj = 0; obj < 2; ++obj) {
        const cudaError_t e = raise_smem_limit(search_ptr(mode, obj), smem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_search(const BatchArgs& args, int mode, int n_ctas, size_t smem,
                          cudaStream_t stream) {
    const SearchKernel k = args.obj_flag != 0 ? search_fn<1>(mode) : search_fn<0>(mode);
    k<<<n_ctas, kThreads, smem, stream>>>(args);
    return cudaGetLastError();
}

cudaError_t launch_best(const double* power, int n_curves, const int64_t* spec_off,
                        int64_t* best_index, double* best_power, double* mean, double* sd,
                        cudaStream_t stream) {
    if (n_curves <= 0) return cudaSuccess;
    best_kernel<<<n_curves, kThreads, 0, stream>>>(power, spec_off, best_index, best_power, mean,
                                                   sd);
    return cudaGetLastError();
}

cudaError_t launch_rows(const double* out, int64_t out_stride, int n_curves,
                        const int64_t* spec_off, const int64_t* grid_base, int64_t max_periods,
                        const double* freq, const double* sep, const double* tol, int n_best,
                        int harmonic_max, int32_t* n_peaks, int64_t* index, double* fields,
                        cudaStream_t stream) {
    if (n_curves <= 0) return cudaSuccess;
    // the list while it fits beside the bitmap: up to 917,504 periods
    const size_t bits = sizeof(uint32_t) * (size_t)((max_periods + 31) / 32);
    const size_t list = kRowList * (2 * sizeof(double) + sizeof(int32_t)) + kRowBins * sizeof(int);
    const int list_cap = bits + list <= 160 * 1024 && max_periods <= INT32_MAX ? kRowList : 0;
    const size_t smem = bits + (list_cap > 0 ? list : 0);
    cudaError_t e = raise_smem_limit((const void*)rows_kernel, smem);
    if (e != cudaSuccess) return e;
    rows_kernel<<<n_curves, kThreads, smem, stream>>>(out, out_stride, spec_off, grid_base, freq,
                                                      sep, tol, n_best, harmonic_max, list_cap,
                                                      n_peaks, index, fields);
    return cudaGetLastError();
}

cudaError_t launch_fold_bins(const double* tau, int n, double P, double f, uint32_t S, double bin,
                             int width, int fb, uint32_t mu, uint32_t mphi, int fast,
                             int32_t* out, int32_t* used_fast, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    fold_bins_kernel<<<(n + 255) / 256, 256, 0, stream>>>(tau, n, P, f, S, bin, width, fb, mu,
                                                          mphi, fast, out, used_fast);
    return cudaGetLastError();
}

// 2 MiB + 256 B per device, in the library's module (no allocation at run time).
__device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

cudaError_t static_scratch_address(int device, void** ptr) {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static void* addr[kMaxDevices] = {};
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[device]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess) return e;
        addr[device] = p;
    }
    *ptr = addr[device];
    return cudaSuccess;
}

int search_threads() { return kThreads; }

size_t period_hist_bytes(int mode, int hl) {
    switch (mode) {
        case MODE_UNIFORM: return hist_period_bytes<MODE_UNIFORM>(hl);
        case MODE_PAIR: return hist_period_bytes<MODE_PAIR>(hl);
        case MODE_WIDE: return hist_period_bytes<MODE_WIDE>(hl);
        case MODE_EXACT: return hist_period_bytes<MODE_EXACT>(hl);
        default: return hist_period_bytes<MODE_GENERAL>(hl);
    }
}

int screen_shift(int mode) {
    return mode == MODE_WIDE ? screen_shift<MODE_WIDE>()
           : mode == MODE_EXACT ? screen_shift<MODE_EXACT>() : 0;
}

size_t search_static_smem(int mode) {
    size_t most = 0;
    for (int obj = 0; obj < 2; ++obj) {
        cudaFuncAttributes at{};
        if (cudaFuncGetAttributes(&at, search_ptr(mode, obj)) == cudaSuccess)
            most = std::max(most, at.sharedSizeBytes);
    }
    return most;
}

int max_resident_ctas(int mode, size_t smem) {
    // the smaller of the two objectives' occupancies
    int b0 = 0, b1 = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, search_ptr(mode, 0), kThreads, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, search_ptr(mode, 1), kThreads, smem);
    return b0 < b1 ? b0 : b1;
}

}  // namespace blsb200
