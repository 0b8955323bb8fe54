// Joint-ephemeris multi-band BLS search kernel (sm_100a): one box, one duration
// and one phase, shared by every band of a star (cuPeriod
// src/cuperiod/multiband/_bls_joint.py:412-507 for the sweep, 359-404 for the
// reported fields).
//
// A persistent grid of 1024-thread CTAs (one per SM: a six-band star's
// histograms take up to ~190 KB of shared memory) claims trial periods from a
// global counter.  Per period a CTA
//   1. folds every point of the star into its band's histogram (per bin the centred
//      flux*weight and the weight, exact 64-bit fixed point, added with native 32-bit
//      shared atomics and carries -- or in a per-CTA global slice when the bands do
//      not fit; the words' high halves lie in one plane, their low halves in another);
//      the bin is the reference's, from the fast fold where its margins prove it, else
//      from the reference's IEEE chain;
//   2. applies the reference's wrap pad per band and turns each histogram into
//      prefix sums in place;
//   3. sweeps every (duration, start) box in units of 32 starts and four durations: an
//      FP32 upper bound on each box's total, from the high words alone, of which a lane
//      keeps its largest and where.  Boxes below a total that some box certainly reaches
//      (an FP32 lower bound) drop out, and the few left are evaluated as the reference
//      does: per band the admissibility floor and dip test, and the
//      band-ordered FP64 sum of depth^2 / (1/iv_in + 1/iv_out) (or
//      0.5 iv_in depth^2); the box with the largest total that any band
//      supports wins, the first in (duration index, start) order among equals;
//   4. writes power (the sum of the bands' squared depth SNRs at that box), the
//      depth of the band with the largest SNR, depth_snr, duration, the
//      mid-transit time and that band's index, by one warp while the others begin the
//      next period.
// Box sums are exact differences of integer prefix sums, converted to FP64 with
// one rounding and scaled by a power of two; from there every operation is the
// reference's, each rounded on its own.
// One six-band star of 2,000 points over 17,815 periods of 1,000 to 2,000 bins: 1.50 ms,
// where 2.92 ms went before into 64-bit conversions in the screen (all boxes' both words)
// and into phases that waited for one warp.  Of a period's 25,000 cycles the sweep takes
// 11,600 (issue: about 20 instructions a box and band), the scan 5,400 and the candidates
// 3,500 (latency and shared memory; the histograms leave room for one CTA), and clearing,
// folding and the last period's report, at the same time, 4,800.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "bls_device.h"
#include "bls_fold.cuh"
#include "bls_launch.h"

namespace blsb200 {
namespace {

constexpr int kJThreads = 1024;
constexpr int kJWarps = kJThreads / 32;
constexpr int kQueue = 2048;            // candidate boxes of one period
constexpr unsigned kAll = 0xffffffffu;

enum : int { JERR_BIN = 1, JERR_DESC = 2 };

// One period to search: p (n_periods or more: none left) and what the fold needs of it.
struct JointWork {
    double period, freq;
    int64_t p;
    int32_t nb;
    uint32_t scale;
    JointSegment seg;
    alignas(16) int32_t dur[kMaxDur + 4];   // the last one repeated to a multiple of four
};

struct JointShared {
    JointBand band[kMaxJointBands];
    longlong2 utot[kMaxJointBands];     // scan: totals of each warp's unit
    double red_v[kJWarps];
    long long red_key[kJWarps];
    int red_hit[kJWarps];
    double ep_snr[kMaxJointBands];
    double ep_depth[kMaxJointBands];
    long long ep_y[kMaxJointBands], ep_i[kMaxJointBands];   // the winning box's sums
    uint32_t queue[kQueue];             // candidate boxes: duration index << 24 | start, which
                                        // with kGroup set stand for a group of four durations
    JointWork work[2];                  // this period's and the next one's
    int qn;
    int rescan;                         // every box must be evaluated
    uint32_t thr_bits;                  // a total some box of the period reaches, FP32 bits
};
constexpr uint32_t kGroup = 1u << 31;
constexpr int kStartBits = 24;

// One period's histograms: band k's bin j at [k * L + j], {y, weight}: the high words, the
// low words.  The fold's sums are split at bit 32 (`get`), the prefix sums at bit 31, the
// high word of y with 2^31 added (`sum`): magnitudes stay below 2^62, and the upper 23 bits
// of either high word serve as a float's mantissa (`level`).
struct Hist {
    int2* hi;
    uint2* lo;
};
__device__ __forceinline__ longlong2 get(const Hist& h, int i) {
    const int2 a = h.hi[i];
    const uint2 b = h.lo[i];
    return make_longlong2((long long)(((unsigned long long)(uint32_t)a.x << 32) | b.x),
                          (long long)(((unsigned long long)(uint32_t)a.y << 32) | b.y));
}
__device__ __forceinline__ void put(const Hist& h, int i, longlong2 v) {
    h.hi[i] = make_int2((int)(v.x >> 32), (int)(v.y >> 32));
    h.lo[i] = make_uint2((uint32_t)v.x, (uint32_t)v.y);
}
__device__ __forceinline__ longlong2 sum(const Hist& h, int i) {
    const int2 a = h.hi[i];
    const uint2 b = h.lo[i];
    return make_longlong2(((long long)(a.x ^ (int)0x80000000) << 31) | b.x,
                          ((long long)(uint32_t)a.y << 31) | b.y);
}
__device__ __forceinline__ void put_sum(const Hist& h, int i, longlong2 v) {
    h.hi[i] = make_int2((int)(v.x >> 31) ^ (int)0x80000000, (int)(v.y >> 31));
    h.lo[i] = make_uint2((uint32_t)v.x & 0x7fffffffu, (uint32_t)v.y & 0x7fffffffu);
}
// 2^23 plus the high word / 2^9, rounded down: the prefix sum in units of 2^40 quanta
__device__ __forceinline__ float level(int hi) {
    return __uint_as_float(__funnelshift_r((uint32_t)hi, 0x96u, 9));
}

// The box (its total and (duration index << 32 | start) key) that the reference's
// first-wins sweep keeps of two: the larger total, then the earlier box.
__device__ __forceinline__ void keep_better(double& v, long long& key, int& hit, double ov,
                                            long long okey, int ohit) {
    if (ohit && (!hit || ov > v || (ov == v && okey < key))) {
        v = ov;
        key = okey;
        hit = 1;
    }
}

__device__ __forceinline__ long long warp_inclusive(long long v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(kAll, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// In-place inclusive prefix sums of K histograms of L {Y, I} bins (band k at k*L), split as
// `sum` reads them.  Up to 32 bands: a band is cut into C runs, one warp each, whose totals
// meet in shared memory; else a warp takes whole bands.  A lane owns R bins of its warp's
// run (odd, so that the lanes' banks differ) and reads them twice.
__device__ void block_prefix(const Hist& h, int K, int L, JointShared& s, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    const int C = K <= kJWarps ? kJWarps / K : 1;
    const int CL = (L + C - 1) / C;
    const int R = ((CL + 31) / 32) | 1;
    const int units = K * C;
    for (int u = warp;; u += kJWarps) {
        const bool on = u < units;
        const int k = u / C, c0 = (u - k * C) * CL, c1 = on ? min(c0 + CL, L) : 0;
        const int r0 = min(c0 + lane * R, c1), r1 = min(r0 + R, c1);
        const int x = k * L;
        long long ry = 0, ri = 0;
        for (int j = r0; j < r1; ++j) {
            const longlong2 e = get(h, x + j);
            ry += e.x;
            ri += e.y;
        }
        long long runy = warp_inclusive(ry, lane), runi = warp_inclusive(ri, lane);
        if (C > 1) {
            if (on && lane == 31) s.utot[u] = make_longlong2(runy, runi);
            __syncthreads();            // (C > 1: one turn of this loop for every warp)
            for (int q = k * C; on && q < u; ++q) {
                runy += s.utot[q].x;
                runi += s.utot[q].y;
            }
        }
        runy -= ry;
        runi -= ri;
        for (int j = r0; j < r1; ++j) {
            const longlong2 e = get(h, x + j);
            runy += e.x;
            runi += e.y;
            put_sum(h, x + j, make_longlong2(runy, runi));
        }
        if (C > 1 || u + kJWarps >= units) break;
    }
    __syncthreads();
}

// The same of histograms in global memory: a warp takes its run 32 consecutive bins at a time,
// the next ones on their way while it scans.  With a run of bins a lane, as above, a warp's
// loads touched 32 lines each in both planes, more than L1 holds of a CTA's 30 warps: a
// six-band star of 1,800 points and up to 8,000 bins, 2,000 periods, 4.57 ms so, 0.96 ms here;
// 64 bands of 1,000 bins, 5,000 periods, 5.80 and 2.49 ms.
__device__ void block_prefix_global(const Hist& h, int K, int L, JointShared& s, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    const int C = K <= kJWarps ? kJWarps / K : 1;
    const int CL = (L + C - 1) / C;
    const int units = K * C;
    if (C > 1) {                        // (one run a warp)
        const int k = warp / C, c0 = (warp - k * C) * CL;
        long long ry = 0, ri = 0;
        for (int j = c0 + lane; warp < units && j < min(c0 + CL, L); j += 32) {
            const longlong2 e = get(h, k * L + j);
            ry += e.x;
            ri += e.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ry += __shfl_xor_sync(kAll, ry, o);
            ri += __shfl_xor_sync(kAll, ri, o);
        }
        if (lane == 0 && warp < units) s.utot[warp] = make_longlong2(ry, ri);
        __syncthreads();
    }
    for (int u = warp; u < units; u += kJWarps) {
        const int k = u / C, c0 = (u - k * C) * CL, c1 = min(c0 + CL, L);
        const int x = k * L;
        long long runy = 0, runi = 0;
        for (int q = k * C; q < u; ++q) {
            runy += s.utot[q].x;
            runi += s.utot[q].y;
        }
        const longlong2 none = make_longlong2(0, 0);
        longlong2 next = c0 + lane < c1 ? get(h, x + c0 + lane) : none;
        for (int j = c0 + lane; j - lane < c1; j += 32) {
            const longlong2 e = next;
            next = j + 32 < c1 ? get(h, x + j + 32) : none;
            const long long y = runy + warp_inclusive(e.x, lane);
            const long long i = runi + warp_inclusive(e.y, lane);
            if (j < c1) put_sum(h, x + j, make_longlong2(y, i));
            runy = __shfl_sync(kAll, y, 31);
            runi = __shfl_sync(kAll, i, 31);
        }
    }
    __syncthreads();
}

// Per-band constants of the screen, in units of 2^40 quanta (the sums' magnitudes add up to
// less than 2^21 of them).
struct Screen {
    float ybar, d, s;           // mean, t's error bound, total weight less its error
    float c;                    // the objective per unit of the one in these units
    float near;                 // a weight below this: the full words decide
    int pad[3];
};

// An FP32 upper bound on box (n, d)'s FP64 total (as exact_box computes it), from the prefix
// sums' full words; 0 when no band can dip in it, +inf when no bound can be formed.  a = iv_in,
// y = y_in, t = y - ybar a, whose sign is the dip's (depth = -S t / (a b), b = S - a), so a
// dipping band's objective is at most (|t| + dt)^2 S / (a b) (likelihood: 0.5 (|t| + dt)^2 S^2
// / (a b^2)) times c_n, dt covering the FP32 conversions and products and the FP64 rounding
// that could flip a dip decision.  A band of which the box holds no weight, or all of it when
// that fails the floor, adds nothing, as in FP64.
__device__ __noinline__ float full_bound(const Hist& h, const JointBand* band, int K, int L, int n,
                                         int d, int obj) {
    float U = 0.0f;
    for (int k = 0; k < K; ++k) {
        const longlong2 e0 = sum(h, k * L + n), e1 = sum(h, k * L + n + d);
        const JointBand& b = band[k];
        const long long qi = e1.y - e0.y;
        if (qi == 0 || (qi >= b.qi_total && b.full_skip)) continue;
        const float a = __ll2float_rn(qi) * 0x1p-61f;
        const float y = __ll2float_rn(e1.x - e0.x) * 0x1p-61f;
        const float t = fmaf(-b.ybar_n, a, y);
        const float dt =
            0x1p-20f * (fabsf(y) + fabsf(b.ybar_n) * (a + 0x1p-20f * b.s_n)) + 0x1p-100f;
        if (t > dt) continue;           // the box is certainly brighter: no dip
        const float a_lo = a * (1.0f - 0x1p-20f);
        const float b_lo = b.s_n - a - 0x1p-20f * b.s_n;
        const float den = obj == 0 ? a_lo * b_lo : a_lo * b_lo * b_lo;
        // __fdividef needs a normal denominator below 2^126
        if (!(a_lo > 0.0f) || !(b_lo > 0.0f) || !(den > 0x1p-100f)) return CUDART_INF_F;
        const float ta = fabsf(t) + dt;
        const float num = obj == 0 ? ta * ta * b.s_n : 0.5f * ta * ta * b.s_n * b.s_n;
        U += fmaxf(__fdividef(num, den) * b.c_n, 0x1p-100f);        // not 0: it may dip
    }
    return U;
}

// One band's part of the same bound from the high words alone, exact integers in FP32
// (levels): a level is within 1 below its sum, so with e0's weight level raised by 1 (w0) the
// difference a lies up to 2 below the weight, and with e0's y level raised by d (y0) th =
// ybar a + y0 - y1 is above -t: d = 1.5 + 3 |ybar| (1 for y, 2 |ybar| for a, the rest for the
// roundings of ybar and of the FMA).  th is positive for every box that may dip.  A box without
// weight has a = -1 and adds nothing.  A weight below `near` (bands of which a point may be
// that small) or a rest too small for its error makes the box one for full_bound.  About 17
// instructions a box and band, one of them (the reciprocal) on the unit that conversions would
// also need: converting the differences of 32-bit words instead took three such instructions.
template <int OBJ>
__device__ __forceinline__ float screen_part(int2 e1, float w0, float y0, const Screen& b,
                                             bool& full) {
    const float a = level(e1.y) - w0;
    const float out = b.s - a;
    full |= (a < b.near) | !(out >= 1.0f);
    const float th = fmaxf(fmaf(b.ybar, a, y0 - level(e1.x)), 0.0f);
    const float den = OBJ ? a * out * out : a * out;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(den));
    return fmaxf(th * th * r, 0.0f) * b.c;
}

// A lower bound on a box's FP64 total from band k (0 when the band is not certain to count):
// a band that certainly passes both floor tests (a and b above twice the floor) and certainly
// dips (t < -dt) adds at least (|t| - dt)^2 S / (a b) (likelihood: 0.5 (|t| - dt)^2 S^2 /
// (a b^2)), with a, b and S bounded on the unfavourable side; the other bands add >= 0.  The
// screen's threshold may be any such bound, since some box reaches it.
__device__ __forceinline__ float lower_part(longlong2 e0, longlong2 e1, const JointBand& b,
                                            int obj) {
    const float a = __ll2float_rn(e1.y - e0.y) * 0x1p-61f;
    const float y = __ll2float_rn(e1.x - e0.x) * 0x1p-61f;
    const float t = fmaf(-b.ybar_n, a, y);
    const float dt = 0x1p-20f * (fabsf(y) + fabsf(b.ybar_n) * (a + 0x1p-20f * b.s_n)) + 0x1p-100f;
    const float a_lo = a * (1.0f - 0x1p-20f);
    const float b_lo = b.s_n - a - 0x1p-20f * b.s_n;
    if (!(t < -dt && a_lo > 2.0f * b.floor_n && b_lo > 2.0f * b.floor_n)) return 0.0f;
    const float tl = fabsf(t) - dt;
    const float s_lo = b.s_n * (1.0f - 0x1p-20f);
    const float a_hi = a * (1.0f + 0x1p-20f);
    const float b_hi = b.s_n - a + 0x1p-19f * b.s_n;
    const float dl = obj == 0 ? a_hi * b_hi : a_hi * b_hi * b_hi;
    if (!(dl > 0x1p-100f && dl < 0x1p100f)) return 0.0f;
    const float nl = obj == 0 ? tl * tl * s_lo : 0.5f * tl * tl * s_lo * s_lo;
    return __fdividef(nl, dl) * b.c_n;
}

// One band's term of the reference's box total (_bls_joint.py:474-493) on the exact sums;
// false: the band does not count.
__device__ __forceinline__ bool exact_term(longlong2 e0, longlong2 e1, const JointBand& b, int obj,
                                           double& term) {
    const double y_in = __dmul_rn(__ll2double_rn(e1.x - e0.x), b.y_unit);
    const double iv_in = __dmul_rn(__ll2double_rn(e1.y - e0.y), b.i_unit);
    const double iv_out = __dsub_rn(b.sum_ivar, iv_in);
    if (iv_in < b.ivar_floor || iv_out < b.ivar_floor) return false;
    const double yin = __ddiv_rn(y_in, iv_in);
    const double yout = __ddiv_rn(__dsub_rn(b.sum_y, y_in), iv_out);
    if (!(yout >= yin)) return false;
    const double depth = __dsub_rn(yout, yin);
    term = obj == 0 ? __ddiv_rn(__dmul_rn(depth, depth),
                                __dadd_rn(__ddiv_rn(1.0, iv_in), __ddiv_rn(1.0, iv_out)))
                    : __dmul_rn(__dmul_rn(__dmul_rn(0.5, iv_in), depth), depth);
    return true;
}

// The reference's box total: the bands' terms, added in band order.
__device__ __noinline__ void exact_box(const Hist& h, const JointBand* band, int K, int L, int n,
                                       int d, int obj, double& total, int& hit) {
    total = 0.0;
    hit = 0;
    for (int k = 0; k < K; ++k) {
        double term;
        if (!exact_term(sum(h, k * L + n), sum(h, k * L + n + d), band[k], obj, term)) continue;
        hit = 1;
        total = __dadd_rn(total, term);
    }
}

// The sweep of one period: see the head of this file.
template <int OBJ>
__device__ __forceinline__ void sweep(JointShared& s, const JointWork& w, const Screen* screen,
                                      const Hist& h, int K, int L, int n_dur, float& best,
                                      float& second, uint32_t& place) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = L - 1;
    const int groups = (n_dur + 3) >> 2;
    int d_min = nb;
    for (int k = 0; k < n_dur; ++k) d_min = min(d_min, w.dur[k]);
    const int units = ((nb - d_min + 32) >> 5) * groups;
    best = second = -1.0f;
    place = 0u;
    for (int u = warp; u < units; u += kJWarps) {
        const int g = (u % groups) * 4, n = (u / groups) * 32 + lane;
        const int4 dg = *reinterpret_cast<const int4*>(&w.dur[g]);
        const int dk[4] = {dg.x, dg.y, dg.z, dg.w};
        int at[4];
        float U[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        bool full[4] = {false, false, false, false};
#pragma unroll
        for (int i = 0; i < 4; ++i) at[i] = min(n + dk[i], nb);
        const int n_at = min(n, nb);
        const int2* x = h.hi;
        for (int k = 0; k < K; ++k, x += L) {
            const int2 e0 = x[n_at];
            const Screen b = screen[k];
            const float w0 = level(e0.y) + 1.0f, y0 = __fadd_ru(level(e0.x), b.d);
#pragma unroll
            for (int i = 0; i < 4; ++i) U[i] += screen_part<OBJ>(x[at[i]], w0, y0, b, full[i]);
        }
        float m = -1.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!((dk[i] < nb) & (n <= nb - dk[i]))) continue;
            if (full[i]) {
                U[i] = g + i < n_dur ? full_bound(h, s.band, K, L, n, dk[i], OBJ) : 0.0f;
                if (U[i] == CUDART_INF_F) {         // no bound: a candidate by itself
                    const int pos = atomicAdd(&s.qn, 1);
                    if (pos < kQueue)
                        s.queue[pos] = ((uint32_t)(g + i) << kStartBits) | (uint32_t)n;
                    else
                        s.rescan = 1;
                    continue;
                }
            }
            if (!(U[i] <= 0.0f)) m = U[i] < CUDART_INF_F ? fmaxf(m, U[i] * (1.0f + 0x1p-16f))
                                                         : CUDART_INF_F;
        }
        if (!(m < CUDART_INF_F)) s.rescan = 1;
        second = fmaxf(second, fminf(m, best));
        if (m > best) {
            best = m;
            place = ((uint32_t)g << kStartBits) | (uint32_t)n;
        }
    }
    // a warp whose best group may be the period's publishes a lower bound of its boxes: box
    // lane / 8, the bands over the eight lanes
    __syncwarp();
    const uint32_t top = __reduce_max_sync(kAll, __float_as_uint(fmaxf(best, 0.0f)));
    if (__any_sync(kAll, top > *reinterpret_cast<volatile uint32_t*>(&s.thr_bits))) {
        const unsigned who = __ballot_sync(kAll, __float_as_uint(best) == top);
        const uint32_t pl = __shfl_sync(kAll, place, __ffs(who) - 1);
        const int n = (int)(pl & ((1u << kStartBits) - 1u));
        const int di = (int)(pl >> kStartBits) + (lane >> 3);
        const int d = w.dur[di];
        float lo = 0.0f;
        if (di < n_dur && d < nb && n <= nb - d)
            for (int k = lane & 7; k < K; k += 8)
                lo += lower_part(sum(h, k * L + n), sum(h, k * L + n + d), s.band[k], OBJ);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) lo += __shfl_xor_sync(kAll, lo, o);
        lo *= 1.0f - 0x1p-16f;
        if (lo > 0x1p-100f && lo < 0x1p126f) atomicMax(&s.thr_bits, __float_as_uint(lo));
    }
}

// The next period and its segment (the last one that begins at or before it), by one warp.
__device__ __forceinline__ void fetch(const JointArgs& a, JointWork& w, int lane) {
    int p = 0;
    if (lane == 0) p = atomicAdd(a.work_counter, 1);
    p = __shfl_sync(kAll, p, 0);
    if (lane == 0) w.p = p;
    if (p < a.n_periods) {
        int c = 0;
        for (int i = lane; i < a.n_segments; i += 32) c += a.segments[i].period_off <= p;
        c = __reduce_add_sync(kAll, c);
        constexpr int kWords = sizeof(JointSegment) / 4;
        static_assert(sizeof(JointSegment) % 4 == 0 && kWords <= 32, "one word a lane");
        const JointSegment* seg = a.segments + c - 1;
        if (lane < kWords)
            reinterpret_cast<int32_t*>(&w.seg)[lane] = reinterpret_cast<const int32_t*>(seg)[lane];
        const int n_dur = min(seg->n_dur, kMaxDur);
        for (int i = lane; i < kMaxDur + 4; i += 32)
            w.dur[i] = n_dur > 0 ? a.dur_bins[seg->dur_off + min(i, n_dur - 1)] : 0;
        if (lane == 0) {
            w.period = a.period[p];
            w.freq = a.freq[p];
            w.scale = a.scale[p];
            w.nb = a.nbins[p];
        }
    }
    __syncwarp();
}

template <bool SMEM>
__global__ void __launch_bounds__(kJThreads, 1)
    joint_kernel(const __grid_constant__ JointArgs a) {
    extern __shared__ __align__(16) unsigned char joint_dyn[];
    __shared__ JointShared s;
    __shared__ Screen screen[kMaxJointBands];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = a.n_bands;
    for (int k = tid; k < K; k += kJThreads) {
        const JointBand b = a.bands[k];
        s.band[k] = b;
        Screen c;
        c.ybar = b.ybar_n;
        c.d = 1.5f + 3.0f * fabsf(b.ybar_n);
        c.s = b.s_n * 0x1p21f - 3.5f;   // 2 for a, the rest for the roundings
        // for the roundings of the product; not so small that the bound of a box that may dip
        // (th >= 1/8) is flushed
        c.c = (a.obj_flag == 0 ? b.s_n * b.c_n : 0x1p20f * b.s_n * b.s_n * b.c_n) *
              (1.0f + 0x1p-18f);
        c.c = fmaxf(c.c, 0x1p-60f);
        // points of 4 units or more: any other weight is none
        c.near = b.qi_min >= (4ll << 40) ? -2.0f : 3.0f;
        c.pad[0] = c.pad[1] = c.pad[2] = 0;
        screen[k] = c;
    }
    const int64_t bins = (int64_t)K * a.hist_stride;
    unsigned char* hist = SMEM ? joint_dyn
                               : reinterpret_cast<unsigned char*>(a.scratch) +
                                     (size_t)blockIdx.x * 16 * bins;
    const Hist h{reinterpret_cast<int2*>(hist), reinterpret_cast<uint2*>(hist + 8 * bins)};
    constexpr int kFetcher = kJWarps - 1;   // the last warp has the fewest units to sweep
    if (warp == kFetcher) fetch(a, s.work[0], lane);
    __syncthreads();
    for (int slot = 0;; slot ^= 1) {
        const JointWork& w = s.work[slot];
        const int64_t p = w.p;
        if (p >= a.n_periods) break;
        const JointSegment& seg = w.seg;
        const double P = w.period;
        const int nb = w.nb;
        const int L = nb + 1;
        const int n_dur = seg.n_dur;
        const bool bad = nb < seg.oversample + 1 || L > seg.hist_len || L > a.hist_stride ||
                         n_dur > kMaxDur || nb > seg.width - 1;
        if (bad) {
            if (tid == 0) {
                atomicOr(a.error_flag, JERR_DESC);
                for (int f = 0; f < kJointFields; ++f) a.out[f * a.n_periods + p] = 0.0;
            }
            if (warp == kFetcher) fetch(a, s.work[slot ^ 1], lane);
            __syncthreads();
            continue;
        }

        // 0. the other warps clear the histograms and fold while warp 0 still reports the
        // last period
        if (warp != 0) {
            constexpr int kFolders = kJThreads - 32;
            const int me = tid - 32;
            if (me == 0) {
                s.thr_bits = 0u;
                s.qn = 0;
                s.rescan = a.screen == 0 || nb >= (1 << kStartBits);
            }
            // (a thread's next point is on its way while it clears, or folds the last one)
            int j = me, k1 = 0;
            double x1 = 0.0;
            long long qy1 = 0, qi1 = 0;
            auto load = [&]() {
                if (j < a.n_points) {
                    k1 = a.band_of[j];
                    x1 = a.tau[j];
                    qy1 = a.qy[j];
                    qi1 = a.qi[j];
                }
            };
            load();
            // (the stride is even, so both planes are whole 16-byte words)
            int4* zh = reinterpret_cast<int4*>(h.hi);
            int4* zl = reinterpret_cast<int4*>(h.lo);
            const int nz = (K * L + 1) >> 1;
            for (int i = me; i < nz; i += kFolders) {
                zh[i] = make_int4(0, 0, 0, 0);
                zl[i] = make_int4(0, 0, 0, 0);
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kFolders) : "memory");

            // 1. fold (_bls_joint.py:436-451): every point of the star into its band
            const double bin = seg.bin_duration, f = w.freq;
            const uint32_t S = w.scale;
            const FoldConst fc(seg.frac_bits, seg.margin_u, seg.margin_phi, seg.fast_fold != 0);
            const int width = seg.width;
            while (j < a.n_points) {
                const int k = k1;
                const double x = x1;
                const long long qy = qy1, qi = qi1;
                j += kFolders;
                load();
                int ind = fold_fast(x, f, S, fc);
                if (ind < 0) ind = fold_exact(x, P, bin, width);
                if (ind > nb) {
                    atomicOr(a.error_flag, JERR_BIN);
                    continue;
                }
                const int i = k * L + ind;
                add_i64_split(&h.lo[i].x, &h.hi[i].x, qy);
                add_i64_split(&h.lo[i].y, &h.hi[i].y, qi);
            }
        }
        __syncthreads();

        // 2. wrap pad (452-459), in the reference's order, then prefix sums (460-465)
        const int os = seg.oversample;
        if (nb - os > os) {
            // the repeated bins and their copies apart: in any order
            for (int i = tid; i < K * os; i += kJThreads) {
                const int k = i / os, o = i - k * os;
                put(h, k * L + min(nb - os + o, seg.width - 1), get(h, k * L + 1 + o));
            }
        } else if (tid < K) {
            for (int o = 0; o < os; ++o) {
                int dst = nb - os + o;
                dst = dst < 0 ? 0 : (dst > seg.width - 1 ? seg.width - 1 : dst);
                put(h, tid * L + dst, get(h, tid * L + 1 + o));
            }
        }
        __syncthreads();
        if (SMEM) block_prefix(h, K, L, s, tid);
        else block_prefix_global(h, K, L, s, tid);

        // 3. the sweep (466-496)
        float best = -1.0f, second = -1.0f;
        uint32_t place = 0u;
        if (warp == kFetcher) fetch(a, s.work[slot ^ 1], lane);
        if (a.screen != 0 && nb < (1 << kStartBits) && n_dur > 0) {
            if (a.obj_flag == 0) sweep<0>(s, w, screen, h, K, L, n_dur, best, second, place);
            else sweep<1>(s, w, screen, h, K, L, n_dur, best, second, place);
        }
        __syncthreads();
        // the threshold is final: groups whose bound reaches it are candidates
        const float thr = __uint_as_float(s.thr_bits);
        if (best >= thr && best > 0.0f) {
            const int pos = atomicAdd(&s.qn, 1);
            if (pos < kQueue) s.queue[pos] = kGroup | place;
            if (pos >= kQueue || second >= thr) s.rescan = 1;
        }
        __syncthreads();
        double top = -CUDART_INF;
        long long key = 0;
        int hit_any = 0;
        const bool all = s.rescan != 0;
        const int qn = min(s.qn, kQueue);
        auto take = [&](int di, int n) {
            const int d = w.dur[di];
            if (d >= nb || n > nb - d || d >= seg.width) return;
            double total;
            int hit;
            exact_box(h, s.band, K, L, n, d, a.obj_flag, total, hit);
            if (hit) keep_better(top, key, hit_any, total, ((long long)di << 32) | (long long)n, 1);
        };
        if (all) {
            for (int di = 0; di < n_dur; ++di)
                for (int n = tid; n <= nb; n += kJThreads) take(di, n);
        } else {
            // a warp per entry: box lane / 8 of it, the bands over the eight lanes
            for (int e = warp; e < qn; e += kJWarps) {
                const uint32_t q = s.queue[e];
                const int n = (int)(q & ((1u << kStartBits) - 1u));
                const int di = (int)((q & ~kGroup) >> kStartBits) + (lane >> 3);
                const int d = w.dur[di];
                const bool in = (lane < 8 || (q & kGroup)) && di < n_dur && d < nb && n <= nb - d;
                double total = 0.0;
                unsigned any = 0u;
                for (int k0 = 0; k0 < K; k0 += 8) {
                    const int k = k0 + (lane & 7);
                    double term = 0.0;
                    bool hit = false;
                    if (in && k < K)
                        hit = exact_term(sum(h, k * L + n), sum(h, k * L + n + d), s.band[k],
                                         a.obj_flag, term);
                    if (!hit) term = 0.0;       // (adding 0 leaves the total as it is)
                    any |= __ballot_sync(kAll, hit);
                    for (int o = 0; o < min(8, K - k0); ++o)
                        total = __dadd_rn(total, __shfl_sync(kAll, term, (lane & 24) + o));
                }
                if ((any >> (lane & 24)) & 0xffu)
                    keep_better(top, key, hit_any, total, ((long long)di << 32) | (long long)n, 1);
            }
        }
        __syncwarp();
        const bool one = !all && qn <= 1;       // warp 0 holds every candidate
        const int o_min = all ? 1 : 8;
        if (!one || warp == 0) {
            for (int o = 16; o >= o_min; o >>= 1) {
                const double ov = __shfl_xor_sync(kAll, top, o);
                const long long ok = __shfl_xor_sync(kAll, key, o);
                const int oh = __shfl_xor_sync(kAll, hit_any, o);
                keep_better(top, key, hit_any, ov, ok, oh);
            }
        }
        if (!one) {
            if (lane == 0) {
                s.red_v[warp] = top;
                s.red_key[warp] = key;
                s.red_hit[warp] = hit_any;
            }
            __syncthreads();
            if (warp == 0) {
                top = s.red_v[lane];
                key = s.red_key[lane];
                hit_any = s.red_hit[lane];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const double ov = __shfl_xor_sync(kAll, top, o);
                    const long long ok = __shfl_xor_sync(kAll, key, o);
                    const int oh = __shfl_xor_sync(kAll, hit_any, o);
                    keep_better(top, key, hit_any, ov, ok, oh);
                }
            }
        }

        // 4. the reported fields (_finish, 359-404), by warp 0: it reads the winning box's
        // sums, and while the others go on takes band k's depth and SNR there in lane k
        // (and k + 32), then the band-ordered sum in lane 0
        const int bn = (int)(key & 0xffffffffll);
        const int bd = warp == 0 && hit_any ? w.dur[(int)(key >> 32)] : 0;
        if (warp == 0)
            for (int k = lane; hit_any && k < K; k += 32) {
                const longlong2 e0 = sum(h, k * L + bn), e1 = sum(h, k * L + bn + bd);
                s.ep_y[k] = e1.x - e0.x;
                s.ep_i[k] = e1.y - e0.y;
            }
        const double bin = seg.bin_duration;
        __syncthreads();
        if (warp == 0) {
            for (int k = lane; hit_any && k < K; k += 32) {
                const JointBand& b = s.band[k];
                const double y_in = __dmul_rn(__ll2double_rn(s.ep_y[k]), b.y_unit);
                const double iv_in = __dmul_rn(__ll2double_rn(s.ep_i[k]), b.i_unit);
                const double iv_out = __dsub_rn(b.sum_ivar, iv_in);
                const bool ok = iv_in >= b.ivar_floor && iv_out >= b.ivar_floor;
                const double safe_in = ok ? iv_in : 1.0;
                const double safe_out = ok ? iv_out : 1.0;
                const double yin = __ddiv_rn(y_in, safe_in);
                const double yout = __ddiv_rn(__dsub_rn(b.sum_y, y_in), safe_out);
                const bool dip = ok && yout >= yin;
                const double dd = __dsub_rn(yout, yin);
                s.ep_depth[k] = dip ? dd : 0.0;
                s.ep_snr[k] =
                    dip ? __ddiv_rn(dd, __dsqrt_rn(__dadd_rn(__ddiv_rn(1.0, safe_in),
                                                             __ddiv_rn(1.0, safe_out))))
                        : 0.0;
            }
            __syncwarp();
            if (lane == 0) {
                double f_power = 0.0, f_depth = 0.0, f_snr = 0.0, f_dur = 0.0, f_t0 = 0.0,
                       f_band = 0.0;
                if (hit_any) {
                    double power = 0.0;
                    int top_k = 0;
                    for (int k = 0; k < K; ++k) {
                        const double snr = s.ep_snr[k];
                        power = __dadd_rn(power, __dmul_rn(snr, snr));
                        if (snr > s.ep_snr[top_k]) top_k = k;   // np.argmax: the first largest
                    }
                    const double duration = __dmul_rn((double)bd, bin);
                    const double mid =
                        __dadd_rn(__dmul_rn((double)bn, bin), __dmul_rn(0.5, duration));
                    f_power = power;
                    f_depth = s.ep_depth[top_k];
                    f_snr = __dsqrt_rn(power);
                    f_dur = duration;
                    f_t0 = __dadd_rn(mid < P ? mid : fmod(mid, P), a.t_min);
                    f_band = (double)top_k;
                }
                double* o = a.out + p;
                o[0] = f_power;
                o[a.n_periods] = f_depth;
                o[2 * a.n_periods] = f_snr;
                o[3 * a.n_periods] = f_dur;
                o[4 * a.n_periods] = f_t0;
                o[5 * a.n_periods] = f_band;
            }
            __syncwarp();
        }
    }
}

}  // namespace

size_t joint_static_smem() { return sizeof(JointShared) + sizeof(Screen) * kMaxJointBands; }

cudaError_t configure_joint(size_t smem) {
    return raise_smem_limit((const void*)joint_kernel<true>, smem);
}

int joint_resident_ctas(bool in_smem, size_t smem) {
    int n = 0;
    cudaError_t e = in_smem
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, joint_kernel<true>, kJThreads, smem)
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, joint_kernel<false>, kJThreads, 0);
    return e == cudaSuccess ? n : 0;
}

cudaError_t launch_joint(const JointArgs& args, bool in_smem, size_t smem, int n_ctas,
                         cudaStream_t stream) {
    if (in_smem)
        joint_kernel<true><<<n_ctas, kJThreads, smem, stream>>>(args);
    else
        joint_kernel<false><<<n_ctas, kJThreads, 0, stream>>>(args);
    return cudaGetLastError();
}

}  // namespace blsb200
