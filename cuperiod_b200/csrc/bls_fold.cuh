// The reference's phase bin of one point.  fold_exact runs its own IEEE
// operations:
//   w = x - P*floor(x/P); ind = int(w/bin) + 1, clipped to [0, width-1]
// (cuPeriod src/cuperiod/methods/_bls_core.py:369-376 / 536-538,
// src/cuperiod/multiband/_bls_joint.py:442-449).  Every operation is rounded on
// its own (no contraction), as the reference's compiled loop does.
#pragma once
#include <stdint.h>

namespace blsb200 {

__device__ __forceinline__ int fold_exact(double x, double P, double bin, int width) {
    const double q = __ddiv_rn(x, P);
    const double w = __dsub_rn(x, __dmul_rn(P, floor(q)));
    int ind = (int)__ddiv_rn(w, bin) + 1;
    ind = ind < 0 ? 0 : ind;
    ind = ind > width - 1 ? width - 1 : ind;
    return ind;
}

// Fast fold: q = x * RN(1/P) rounded onto a 2^-32 grid, then one 32-bit multiply-high
// by S = round(P/bin * 2^fb); the bin is the position's integer part plus 1 when the
// position is provably on the reference's side of every cycle and bin edge.
//
// The phase is taken with the cycle-edge margin mphi added to it inside the FMA's
// constant, which shifts the position by at most mphi and turns a phase just below a
// cycle edge into one just above bin 0's lower edge.  The host's margin mu covers that
// shift on top of the bin-edge error, and the 2 mphi that phases next to a cycle edge
// land in, so one comparison per point decides both: `edge` is the position inside the
// bin, top aligned and less mu, and is below `limit` when the bin is certain (a running
// maximum over several points tests them all).  Without a provable fold no position is
// below the limit.
struct FoldConst {
    int fb;                 // fraction bits of a position
    uint32_t up, sub, limit;
    double magic;
    __device__ __forceinline__ FoldConst(int frac_bits, uint32_t mu, uint32_t mphi, bool fast)
        : fb(frac_bits), up(1u << ((32 - frac_bits) & 31)), sub(0u - mu * up),
          limit(fast ? 0u - 2u * mu * up : 0u),
          magic(1572864.0 + (double)mphi * (1.0 / 4294967296.0)) {}
    // phase * P/bin * 2^fb: x*f + 1.5*2^20 in one rounding has an ulp of 2^-32, so its
    // low word is round(frac(x*f) * 2^32)
    __device__ __forceinline__ uint32_t position(double x, double f, uint32_t S) const {
        return __umulhi((uint32_t)__double2loint(__fma_rn(x, f, magic)), S);
    }
    __device__ __forceinline__ uint32_t edge(uint32_t v) const { return v * up + sub; }
};

// The reference's bin, or -1 when the fast fold does not decide it.
__device__ __forceinline__ int fold_fast(double x, double f, uint32_t S, const FoldConst& fc) {
    const uint32_t v = fc.position(x, f, S);
    return fc.edge(v) < fc.limit ? (int)(v >> fc.fb) + 1 : -1;
}

// Add v to an int64 kept as a low and a high 32-bit word with two native 32-bit atomics -- the low word,
// then the high word plus the carry out of the low word -- where a 64-bit
// shared atomic would be emulated (sm_100).
// Each add sees the old low word it added to, so every carry is counted once
// and the int64 is the exact sum at any number of adds.
__device__ __forceinline__ void add_i64_split(unsigned* lo_word, int* hi_word, long long v) {
    const unsigned lo = (unsigned)v;
    const unsigned old = atomicAdd(lo_word, lo);
    atomicAdd(hi_word, (int)(v >> 32) + (old + lo < old ? 1 : 0));
}

}  // namespace blsb200
