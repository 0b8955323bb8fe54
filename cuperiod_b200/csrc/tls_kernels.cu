// Transit least squares matched-filter kernel (sm_100a): the limb-darkened
// template search of cuPeriod src/cuperiod/methods/tls.py:516-593 (its CUDA
// tls_block, 323-414, searches one period per block).
//
// A persistent grid of 256-thread CTAs pulls work items (curve, tile of up to
// kTlsMaxTile consecutive trial periods).  Per item a CTA
//   1. folds every point of the curve into one phase histogram per period of
//      the tile: the reference's bin, q = tau/P, ph = q - floor(q),
//      bin = int(ph * n_bins) clipped -- from a fixed-point fast path where its
//      host-derived margins prove the result, else (listed, and put right after the
//      fold) from those IEEE operations.  A thread holds time-consecutive points (the
//      BLS engine's chunked layout).  yw and w are 64-bit fixed point (a power-of-two
//      scale per curve, magnitudes summing below 2^61); a sum is added to a bin's int64
//      as two native 32-bit shared atomics, the low word first and then the high word
//      plus the carry the low word's old value shows (64-bit shared atomics are emulated
//      on sm_100), so every bin holds the exact integer sum; the words lie in four planes
//      (low and high of yw, of w), so different bins use different banks.  Where a bin is
//      wider than the sampling, runs of equal bins are summed in registers first;
//   2. turns every bin into FP64 (one rounding of the exact sum) and pads the
//      histogram circularly by max_width - 1 bins (the reference's pad);
//   3. per period, one thread per start phase slides every template over the
//      bins, four widths at a time so that a bin is read once for them: num = sum g a,
//      cwg = sum g b, den = sum g^2 b, accumulated in k
//      order with the reference's FP64 operations; a start counts when
//      num < 0, den > w_eps and de = den - cwg^2 / w_total > den_rel * den, and
//      the largest sr = num^2 / de wins, the first in (width, start) order among
//      equals (the reference's strict '>' sweep);
//   4. writes sr, depth = -num/de, duration = width / n_bins * P and the
//      mid-transit phase time (centre - floor(centre)) * P.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <type_traits>

#include "bls_device.h"
#include "bls_launch.h"

namespace blsb200 {
namespace {

constexpr int kTThreads = kChunkThreads;
constexpr int kTWarps = kTThreads / 32;
constexpr int kTPts = kChunkPts;
constexpr int kTHalf = 4;               // points a lane holds where runs are not merged
constexpr unsigned kTAll = 0xffffffffu;

enum : int { TERR_DESC = 1 };

constexpr int kTList = 256;             // open points of one tile
// Points from which the sweep estimates a template's residue before it divides (tls_templates):
// with fewer, most templates hold the same point and tie, every lane passes, and the estimate
// only costs (3 curves, 200,000 periods, with and without it: 20 points 10.2 and 9.2 ms, 50
// points 9.8 and 9.4, 100 points 9.2 and 9.4 ms).
constexpr int kTlsEstimate = 80;

struct TlsShared {
    union {
        struct {                        // the fold: points the fast path leaves open, by
            uint32_t list_j[kTList];    // index and period
            uint8_t list_p[kTList];
        };
        struct {                        // the sweep: each warp's best of every period
            double red_sr[kTlsMaxTile][kTWarps];
            double red_depth[kTlsMaxTile][kTWarps];
            long long red_key[kTlsMaxTile][kTWarps];
        };
    };
    double per[kTlsMaxTile], freq[kTlsMaxTile];
    int list_n;
    int next;
};

// The reference's phase bin (tls.py:535-542).
__device__ __forceinline__ int tls_bin(double x, double P, int n_bins) {
    const double q = __ddiv_rn(x, P);
    const double ph = __dsub_rn(q, floor(q));
    int b = (int)__dmul_rn(ph, (double)n_bins);
    b = b > n_bins - 1 ? n_bins - 1 : b;
    return b < 0 ? 0 : b;
}

// Fast TLS bin: the phase frac(x * RN(1/P)) on a 2^-32 grid (one FMA, as the BLS fast
// fold), times n_bins as a 64-bit integer product whose high word is the bin (always in
// [0, n_bins)) and low word the position inside it.  The cycle-edge margin mphi is added
// to the phase inside the FMA's constant, which shifts the position by mphi * n_bins and
// turns a phase just below a cycle edge into one just above bin 0's lower edge; the host's
// margin mu covers that shift and the bin-edge error, so the bin is the reference's when
// edge < limit.
struct TlsFold {
    uint32_t nb, mu, limit;
    double magic;
    __device__ __forceinline__ TlsFold(int n_bins, uint32_t margin_u, uint32_t mphi)
        : nb((uint32_t)n_bins), mu(margin_u), limit(0u - 2u * margin_u),
          magic(1572864.0 + (double)mphi * (1.0 / 4294967296.0)) {}
    __device__ __forceinline__ uint32_t bin(double x, double f, uint32_t& edge) const {
        const unsigned long long prod =
            (unsigned long long)(uint32_t)__double2loint(__fma_rn(x, f, magic)) * nb;
        edge = (uint32_t)prod - mu;
        return (uint32_t)(prod >> 32);
    }
};

// Of two candidates (sr, key = width index << 32 | start, depth), the one the
// reference keeps: the larger sr, then the earlier (width, start); key < 0 is
// no candidate.
__device__ __forceinline__ void tls_keep(double& sr, long long& key, double& depth, double osr,
                                         long long okey, double odepth) {
    if (okey >= 0 && (key < 0 || osr > sr || (osr == sr && okey < key))) {
        sr = osr;
        key = okey;
        depth = odepth;
    }
}

__device__ __forceinline__ uint32_t atom_add(uint32_t a, uint32_t v) {
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ void red_add(uint32_t a, uint32_t v) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_word(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// Add y and w to the bin whose first word is at shared address `rec`; the bin's four words
// are `plane` bytes apart (low and high of yw, of w).
__device__ __forceinline__ void add_bin(uint32_t rec, uint32_t plane, long long y, long long w) {
    const uint32_t yl = (uint32_t)y, wl = (uint32_t)w;
    const uint32_t oy = atom_add(rec, yl);
    const uint32_t ow = atom_add(rec + 2 * plane, wl);
    red_add(rec + plane, (uint32_t)((unsigned long long)y >> 32) + (oy + yl < oy ? 1u : 0u));
    red_add(rec + 3 * plane, (uint32_t)((unsigned long long)w >> 32) + (ow + wl < ow ? 1u : 0u));
}

// The 64-bit value of a bin's two words.
__device__ __forceinline__ long long plane_value(uint32_t a, uint32_t plane) {
    return (long long)(((unsigned long long)ld_word(a + plane) << 32) | ld_word(a));
}

// This lane's r-th point of a block at `base`: slot base + (first + r) * kTThreads + tid of
// a full chunk (first: of the lane's 8), time index base + tid * NR + r of the tail.
template <int NR, bool TAIL>
__device__ __forceinline__ int tls_point(int base, int first, int r) {
    return TAIL ? base + (int)threadIdx.x * NR + r
                : base + (first + r) * kTThreads + (int)threadIdx.x;
}

// Point j at period p, which the fast fold left open: moved from the bin the fast path
// gave it to the reference's.
__device__ __noinline__ void tls_put_right(const TlsArgs* a, const TlsShared* s, int64_t slot,
                                           int p, uint32_t words, uint32_t plane) {
    const TlsFold fold(a->n_bins, a->margin_u, a->margin_phi);
    const double x = a->tau[slot];
    uint32_t edge;
    const int b0 = (int)fold.bin(x, s->freq[p], edge);
    const int b = tls_bin(x, s->per[p], a->n_bins);
    if (b == b0) return;
    const long long y = a->qy[slot], w = a->qw[slot];
    add_bin(words + 4u * (uint32_t)b0, plane, -y, -w);
    add_bin(words + 4u * (uint32_t)b, plane, y, w);
}

// Fold this lane's NR points of a block into the tile's np histograms (period p's words at
// words + p * region).  MERGE: runs of equal bins are summed in registers first, which pays
// where a bin is wider than the sampling.  Else the points' low words go first, all of
// them, so that the old values that the carries need come back together.
template <int NR, bool TAIL, bool MERGE>
__device__ __forceinline__ void tls_fold(const TlsArgs& a, TlsShared& s, const TlsCurveDesc& cv,
                                         int base, int first, int np, uint32_t words,
                                         uint32_t region, uint32_t plane) {
    if (TAIL && base + (int)threadIdx.x * NR >= cv.n_points) return;
    uint32_t lost = 0u;             // periods whose open points found the list full
    {
        double x[NR];
        long long y[NR], w[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int j = tls_point<NR, TAIL>(base, first, r);
            const int64_t slot = cv.point_off + (TAIL ? min(j, cv.n_points - 1) : j);
            const bool ok = !TAIL || j < cv.n_points;
            x[r] = __ldg(a.tau + slot);
            y[r] = ok ? __ldg(a.qy + slot) : 0ll;
            w[r] = ok ? __ldg(a.qw + slot) : 0ll;
        }
        const TlsFold fold(a.n_bins, a.margin_u, a.margin_phi);
        uint32_t h = words;
        for (int p = 0; p < np; ++p, h += region) {
            const double f = s.freq[p];
            uint32_t rec[NR], worst = 0u;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                uint32_t edge;
                rec[r] = h + 4u * fold.bin(x[r], f, edge);
                worst = max(worst, edge);
            }
            if (worst >= fold.limit) {
                uint32_t open = 0u;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    uint32_t edge;
                    fold.bin(x[r], f, edge);
                    const int j = tls_point<NR, TAIL>(base, first, r);
                    if (edge >= fold.limit && (!TAIL || j < cv.n_points)) open |= 1u << r;
                }
                // (a full list is not counted further: the counter stays below kTList plus
                // the CTA's points in flight)
                int pos = kTList;
                if (*static_cast<volatile int*>(&s.list_n) < kTList)
                    pos = atomicAdd(&s.list_n, __popc(open));
                if (pos + __popc(open) > kTList) {
                    lost |= 1u << p;
                    for (; pos < kTList && open != 0u; ++pos, open &= open - 1u)
                        s.list_p[pos] = 0xffu;
                }
                for (; open != 0u; ++pos, open &= open - 1u)
                    if (pos < kTList && !(lost >> p & 1u)) {
                        s.list_j[pos] =
                            (uint32_t)tls_point<NR, TAIL>(base, first, __ffs(open) - 1);
                        s.list_p[pos] = (uint8_t)p;
                    }
            }
            if (MERGE) {
                long long ay = y[0], aw = w[0];
#pragma unroll
                for (int r = 1; r < NR; ++r) {
                    if (rec[r] != rec[r - 1]) {
                        add_bin(rec[r - 1], plane, ay, aw);
                        ay = y[r];
                        aw = w[r];
                    } else {
                        ay += y[r];
                        aw += w[r];
                    }
                }
                add_bin(rec[NR - 1], plane, ay, aw);
            } else {
                uint32_t oy[NR], ow[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    oy[r] = atom_add(rec[r], (uint32_t)y[r]);
                    ow[r] = atom_add(rec[r] + 2 * plane, (uint32_t)w[r]);
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    red_add(rec[r] + plane, (uint32_t)((unsigned long long)y[r] >> 32) +
                                                (oy[r] + (uint32_t)y[r] < oy[r] ? 1u : 0u));
                    red_add(rec[r] + 3 * plane, (uint32_t)((unsigned long long)w[r] >> 32) +
                                                    (ow[r] + (uint32_t)w[r] < ow[r] ? 1u : 0u));
                }
            }
        }
    }
    // the list was full: this lane's open points of those periods now
    for (; lost != 0u; lost &= lost - 1u) {
        const int p = __ffs(lost) - 1;
        const TlsFold fold(a.n_bins, a.margin_u, a.margin_phi);
        for (int r = 0; r < NR; ++r) {
            const int j = tls_point<NR, TAIL>(base, first, r);
            if (TAIL && j >= cv.n_points) break;
            uint32_t edge;
            fold.bin(__ldg(a.tau + cv.point_off + j), s.freq[p], edge);
            if (edge >= fold.limit)
                tls_put_right(&a, &s, cv.point_off + j, p, words + p * region, plane);
        }
    }
}

// Every point of the curve into the tile's histograms.
__device__ __forceinline__ void tls_fold_curve(const TlsArgs& a, TlsShared& s,
                                               const TlsCurveDesc& cv, int np, uint32_t words,
                                               uint32_t region, uint32_t plane) {
    const int n = cv.n_points, nb = a.n_bins;
    if (!a.fast_fold) {
        // no provable fast fold: the reference's operations for every point
        for (int j = threadIdx.x; j < n; j += kTThreads) {
            const int64_t slot = cv.point_off + j;
            const double x = a.tau[slot];
            const long long y = a.qy[slot], w = a.qw[slot];
            for (int p = 0; p < np; ++p)
                add_bin(words + p * region + 4u * (uint32_t)tls_bin(x, s.per[p], nb), plane, y, w);
        }
        __syncthreads();
        return;
    }
    int base = 0;
    if (s.per[np - 1] > cv.merge_period) {
        for (; base + kChunk <= n; base += kChunk)
            tls_fold<kTPts, false, true>(a, s, cv, base, 0, np, words, region, plane);
        for (; base < n; base += kTThreads * kTPts)
            tls_fold<kTPts, true, true>(a, s, cv, base, 0, np, words, region, plane);
    } else {
        for (; base + kChunk <= n; base += kChunk)
#pragma unroll 1
            for (int first = 0; first < kTPts; first += kTHalf)
                tls_fold<kTHalf, false, false>(a, s, cv, base, first, np, words, region, plane);
        for (; base < n; base += kTThreads * kTHalf)
            tls_fold<kTHalf, true, false>(a, s, cv, base, 0, np, words, region, plane);
    }
    __syncthreads();
    const int open = min(s.list_n, kTList);
    for (int e = threadIdx.x; e < open; e += kTThreads) {
        const int p = s.list_p[e];
        if (p < np)
            tls_put_right(&a, &s, cv.point_off + s.list_j[e], p, words + p * region, plane);
    }
    __syncthreads();
}

// NG templates from di at this lane's start st (`in`: there is one) of the bins v, kept
// when one is the best so far.  With EST the reference's two divisions per template and start
// are taken only by the lanes that may hold the warp's best: an FP32 bound on sr decides (one
// out of FP32's range always passes).  The first samples are taken ahead of the loop: chosen
// inside it they cost six selections a template and sample, and the registers that the fold
// needs (60,000 points in wide bins 12.2 ms so, 8.2 ms; 1,000 points 9.56 and 8.92).
template <int NG, bool EST>
__device__ __forceinline__ void tls_templates(const TlsArgs& a, double w_total, float w_inv, float de_rel,
                                              const double2* v, const double* g, int di, int st,
                                              bool in, float& top, double& best, long long& key,
                                              double& depth) {
    int W[NG], off[NG], wmax = 0;
    double num[NG], cwg[NG], den[NG];
#pragma unroll
    for (int i = 0; i < NG; ++i) {
        W[i] = __ldg(a.dur_bins + di + i);
        off[i] = __ldg(a.tmpl_off + di + i);
        wmax = max(wmax, W[i]);
    }
    const double2 e0 = v[st];
#pragma unroll
    for (int i = 0; i < NG; ++i) {
        const double t = g[off[i]];
        num[i] = __dmul_rn(t, e0.x);
        cwg[i] = __dmul_rn(t, e0.y);
        den[i] = __dmul_rn(__dmul_rn(t, t), e0.y);
    }
    for (int k = 1; k < wmax; ++k) {
        const double2 e = v[st + k];
#pragma unroll
        for (int i = 0; i < NG; ++i)
            if (k < W[i]) {
                const double t = g[off[i] + k];
                num[i] = __dadd_rn(num[i], __dmul_rn(t, e.x));
                cwg[i] = __dadd_rn(cwg[i], __dmul_rn(t, e.y));
                den[i] = __dadd_rn(den[i], __dmul_rn(__dmul_rn(t, t), e.y));
            }
    }
    float est[NG], most = 0.0f;
    if (EST) {
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            const float n = (float)num[i], c = (float)cwg[i], d = (float)den[i];
            // cwg^2 / w_total <= den, so de is within 3e-7 den of the exact difference; with de
            // above 1e-4 den (and the template certainly admissible) the quotient bounds sr
            // from above and is within 2e-2 of it.  (c w_inv is at most about 1, and n over
            // the difference as large as sr / n: a square of c or n would leave FP32's normal
            // range for weights below 1e-19)
            const float cc = c * (c * w_inv), de = d - cc;
            float s = n * (n / (de - 1e-6f * d));
            if (!(s > 1e-30f && s < 1e37f) || !(d > 1e-30f) || !(de > de_rel * d)) s = CUDART_INF_F;
            est[i] = in && num[i] < 0.0 && den[i] > a.w_eps ? s : -1.0f;
            if (est[i] < CUDART_INF_F) most = fmaxf(most, est[i]);
        }
        top = fmaxf(top, __uint_as_float(__reduce_max_sync(kTAll, __float_as_uint(most))));
    }
#pragma unroll
    for (int i = 0; i < NG; ++i)
        if (EST ? est[i] >= top * (1.0f - 2e-2f) : in && num[i] < 0.0 && den[i] > a.w_eps) {
            const double de = __dsub_rn(den[i], __ddiv_rn(__dmul_rn(cwg[i], cwg[i]), w_total));
            if (de > __dmul_rn(a.den_rel, den[i])) {
                const double sr = __ddiv_rn(__dmul_rn(num[i], num[i]), de);
                if (sr > 0.0)
                    tls_keep(best, key, depth, sr, ((long long)(di + i) << 32) | (long long)st,
                             __ddiv_rn(-num[i], de));
            }
        }
}

// Bound by the shared-memory pipe: four word atomics a point and period, 3.2 wavefronts
// each.  3 curves of 20,000 points, 119,788 periods: 20.7 ms with runs merged everywhere
// and a returning atomic at a time, 15.9 ms as built.
__global__ void __launch_bounds__(kTThreads, 3) tls_kernel(const __grid_constant__ TlsArgs a) {
    extern __shared__ __align__(16) unsigned char tls_dyn[];
    __shared__ TlsShared s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = a.n_bins, ext = a.n_bins + a.max_width - 1;
    // dynamic shared memory: tile + 1 regions of ext FP64 bins {a, b} (the last of nb) --
    // period p's words lie in region p + 1 and turn into the bins of region p -- then the
    // templates
    double2* ab = reinterpret_cast<double2*>(tls_dyn);
    double* g = reinterpret_cast<double*>(ab + (size_t)a.tile * ext + nb);
    const uint32_t region = 16u * (uint32_t)ext, plane = 4u * (uint32_t)nb;
    const uint32_t words = (uint32_t)__cvta_generic_to_shared(ab) + region;
    for (int i = tid; i < a.n_tmpl; i += kTThreads) g[i] = a.tmpl[i];
    for (;;) {
        if (tid == 0) {
            s.next = atomicAdd(a.work_counter, 1);
            s.list_n = 0;
        }
        __syncthreads();
        const int item = s.next;
        if (item >= a.n_items) break;
        const int c = item / a.tiles_per_curve;
        const int64_t p0 = (int64_t)(item % a.tiles_per_curve) * a.tile;
        const int np = (int)min((int64_t)a.tile, a.n_periods - p0);
        const TlsCurveDesc& cv = a.curves[c];
        if (tid < np) {
            s.per[tid] = a.period[p0 + tid];
            s.freq[tid] = a.freq[p0 + tid];
        }
        for (int p = 0; p < np; ++p) {
            uint4* z = reinterpret_cast<uint4*>(ab + (size_t)(p + 1) * ext);
            for (int i = tid; i < nb; i += kTThreads) z[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();

        // 1. fold
        tls_fold_curve(a, s, cv, np, words, region, plane);

        // 2. FP64 bins (a = sum yw, b = sum w) with the circular pad (544-546)
        const double y_unit = cv.y_unit, w_unit = cv.w_unit;
        for (int p = 0; p < np; ++p) {
            const uint32_t h = words + (uint32_t)p * region;
            double2* v = ab + (size_t)p * ext;
            for (int i = tid; i < ext; i += kTThreads) {
                const uint32_t w = h + 4u * (uint32_t)(i < nb ? i : i - nb);
                v[i] = make_double2(__dmul_rn(__ll2double_rn(plane_value(w, plane)), y_unit),
                                    __dmul_rn(__ll2double_rn(plane_value(w + 2 * plane, plane)),
                                              w_unit));
            }
            __syncthreads();
        }

        // 3. the template sweep: each warp's best of every period
        const double w_total = cv.w_total;
        const float w_inv = (float)(1.0 / w_total);
        const float de_rel = 1e-4f + 1.001f * (float)a.den_rel;
        for (int p = 0; p < np; ++p) {
            const double2* v = ab + (size_t)p * ext;
            double best = 0.0, best_depth = 0.0;
            long long best_key = -1;
            float top = 0.0f;
            for (int s0 = warp * 32; s0 < nb; s0 += kTThreads) {
                const bool in = s0 + lane < nb;
                const int st = in ? s0 + lane : 0;
                auto templates = [&](auto est) {
                    constexpr bool kEst = decltype(est)::value;
                    int di = 0;
                    for (; di + 4 <= a.n_dur; di += 4)
                        tls_templates<4, kEst>(a, w_total, w_inv, de_rel, v, g, di, st, in, top,
                                               best, best_key, best_depth);
                    for (; di < a.n_dur; ++di)
                        tls_templates<1, kEst>(a, w_total, w_inv, de_rel, v, g, di, st, in, top,
                                               best, best_key, best_depth);
                };
                if (cv.n_points >= kTlsEstimate) templates(std::true_type{});
                else templates(std::false_type{});
            }
            __syncwarp();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double osr = __shfl_down_sync(kTAll, best, o);
                const long long okey = __shfl_down_sync(kTAll, best_key, o);
                const double odep = __shfl_down_sync(kTAll, best_depth, o);
                tls_keep(best, best_key, best_depth, osr, okey, odep);
            }
            if (lane == 0) {
                s.red_sr[p][warp] = best;
                s.red_key[p][warp] = best_key;
                s.red_depth[p][warp] = best_depth;
            }
        }
        __syncthreads();

        // 4. one thread per period
        if (tid < np) {
            const int p = tid;
            double best = 0.0, best_depth = 0.0;
            long long best_key = -1;
            for (int w = 0; w < kTWarps; ++w)
                tls_keep(best, best_key, best_depth, s.red_sr[p][w], s.red_key[p][w],
                         s.red_depth[p][w]);
            const double P = s.per[p];
            double o_sr = 0.0, o_depth = 0.0, o_dur = 0.0, o_t0 = 0.0;
            if (best_key >= 0) {
                const int di = (int)(best_key >> 32);
                const int st = (int)(best_key & 0xffffffffll);
                if (di < a.n_dur) {
                    const double W = (double)a.dur_bins[di];
                    o_sr = best;
                    o_depth = best_depth;
                    o_dur = __dmul_rn(__ddiv_rn(W, (double)nb), P);
                    const double centre =
                        __ddiv_rn(__dadd_rn((double)st, __ddiv_rn(W, 2.0)), (double)nb);
                    o_t0 = __dmul_rn(__dsub_rn(centre, floor(centre)), P);
                } else {
                    atomicOr(a.error_flag, TERR_DESC);
                }
            }
            double* o = a.out + (int64_t)c * a.n_periods + p0 + p;
            o[0] = o_sr;
            o[a.out_stride] = o_depth;
            o[2 * a.out_stride] = o_dur;
            o[3 * a.out_stride] = o_t0;
        }
        __syncthreads();
    }
}

}  // namespace

size_t tls_smem_bytes(int n_bins, int max_width, int tile, int n_tmpl) {
    return ((size_t)tile * (size_t)(n_bins + max_width - 1) + (size_t)n_bins) * sizeof(double2) +
           (size_t)n_tmpl * sizeof(double);
}

cudaError_t configure_tls(size_t smem) {
    return raise_smem_limit((const void*)tls_kernel, smem);
}

int tls_resident_ctas(size_t smem) {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tls_kernel, kTThreads, smem) ==
                   cudaSuccess
               ? n
               : 0;
}

cudaError_t launch_tls(const TlsArgs& args, int n_ctas, size_t smem, cudaStream_t stream) {
    tls_kernel<<<n_ctas, kTThreads, smem, stream>>>(args);
    return cudaGetLastError();
}

}  // namespace blsb200
