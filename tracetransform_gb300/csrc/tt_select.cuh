// tt_select.cuh -- weighted selection used by T6, T7 and P2.
//
// TFunctional6/7 (c++/src/functionals.cpp:226-276) sort a key sequence,
// accumulate sqrt-weights in sorted order and return the key at the first
// index where twice the cumulative weight reaches the total.  That key is
// the smallest key k with 2 * W(<= k) >= W, so no sort is needed:
//
//   1. weights become u32 fixed point (2^-30 of a power-of-two bound on the
//      total, so twice any sum fits 32 bits), summed exactly and
//      deterministically by integer atomics;
//   2. a 256-bin histogram linear in the key over [0, top] locates the bin
//      holding the crossing (bins are monotone in the key);
//   3. the entries of that bin are collected, and each lane adds up the
//      weights of the entries up to its own: the smallest that qualifies is
//      the answer.  A bin of more than kSelList entries is refined first:
//      step 2 repeats over its key range with bins linear in the keys' bit
//      patterns, which no range is too narrow for (a bin whose keys are
//      all equal is the answer).
//
// One warp per line.  What bounds it is the instruction count: a histogram
// pass and a collecting pass over half the line, each with as little per
// element as it needs -- bins by one multiply-add into the mantissa of 2^23,
// weights (a square root each) only in the histogram pass and for the few
// collected entries -- and the fixed work per line.  The collected list takes
// the histogram's place in shared memory.  The sinogram kernel at 1024^2 x 360
// angles, T0-T7, by this alone: 2.55 ms, from 3.21 with the bins recomputed by
// conversions and the weights in both passes, 64-bit scans and a 64-entry bitonic
// sort (2.07 with the roots and the sampling since).
#pragma once

#include <climits>

#include "tt_common.cuh"

namespace tt {

constexpr int kSelBins = 256;
constexpr int kSelList = 188; // collected entries (in the histogram's place)

struct SelPick {
    unsigned bin, below, total;
};
struct __align__(16) SelScratch {
    union {
        unsigned hist[kSelBins];
        uint2 list[kSelList]; // key bits, then the sample's bits or its weight
    };
    // several warps on one line: its pick, the weight at the largest sample,
    // the entries collected
    SelPick pick;
    unsigned wtop;
    int count;
};
static_assert(sizeof(SelScratch) == 1536, "the lines per CTA and line lengths it allows");

// The TW warps of a line: this warp's place among them and their barrier.
template <int TW> struct SelTeam {
    int role, bar;
    __device__ __forceinline__ void sync() const {
        if (TW == 1)
            __syncwarp();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(32 * TW) : "memory");
    }
};

// Fixed-point weight of a sample v: sqrt(v) (T6, T7) or v itself (P2).
struct SqrtWeight {
    float qs;
    bool odd; // the line holds samples sqrt_pos does not take (warp-uniform)
    __device__ __forceinline__ unsigned operator()(float v) const {
        return __float2uint_rn((odd ? sqrt_nn(v) : sqrt_pos(v)) * qs);
    }
};
struct LinearWeight {
    float qs;
    __device__ __forceinline__ unsigned operator()(float v) const {
        return __float2uint_rn(v * qs);
    }
};
// 2^(30 - E) for weights whose total stays below 2^E (total: their float sum).
__device__ __forceinline__ float sel_scale(float total) {
    const float qb = total * 1.001f;
    const int E = ((__float_as_int(qb) >> 23) & 0xff) - 126;
    return __int_as_float((127 + 30 - E) << 23);
}

// Bins per unit of a key in [0, top].  At most the largest float, which the
// quotient exceeds for top < 2^-120: the bins are then wider than top / 256 but
// still part the samples from the zeros.
__device__ __forceinline__ float sel_per_key(float top) {
    return fminf((float)kSelBins / top, 3.402823466e38f);
}
// Histogram bin of key k >= 0, bs = sel_per_key: the integer that k bs rounds
// to, in the mantissa of 2^23, at most 255 -- monotone in k.  A negative or NaN
// key gives a valid bin too (255), so no input can index outside the
// histogram; such keys carry no weight.
constexpr unsigned kSelOne = 0x4B000000u; // 2^23
__device__ __forceinline__ unsigned sel_bin(float k, float bs) {
    return min((unsigned)kSelBins - 1, __float_as_uint(fmaf(k, bs, 8388608.f)) - kSelOne);
}

__device__ __forceinline__ void sel_clear(SelScratch *sc, int lane) {
    uint4 *h = reinterpret_cast<uint4 *>(sc->hist);
    h[lane] = make_uint4(0u, 0u, 0u, 0u);
    h[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
}

// The crossing bin: the smallest bin with 2 (below + weight of the bins up to
// it) >= total.  On entry `below` is the weight of all keys under the
// histogram's range, on return that of all keys under the bin.  kTotal: the
// histogram holds every weight, its sum is the total.
template <bool kTotal>
__device__ __forceinline__ SelPick sel_pick(const SelScratch *sc, unsigned below, unsigned total,
                                            int lane) {
    const uint4 *h4 = reinterpret_cast<const uint4 *>(sc->hist) + 2 * lane;
    const uint4 a = h4[0], b = h4[1];
    const unsigned h[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    unsigned run = 0;
#pragma unroll
    for (int k = 0; k < 8; k++)
        run += h[k];
    unsigned inc = run;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned t = __shfl_up_sync(TT_FULL_MASK, inc, d);
        if (lane >= d)
            inc += t;
    }
    if (kTotal)
        total = __shfl_sync(TT_FULL_MASK, inc, 31);
    const unsigned ball = __ballot_sync(TT_FULL_MASK, 2u * (below + inc) >= total);
    const int ln = ball ? __ffs(ball) - 1 : 31;
    unsigned cum = below + inc - run, k = 0;
#pragma unroll
    for (int i = 0; i < 7; i++) { // prefix sums rise: count those that fall short
        const bool shorter = 2u * (cum + h[i]) < total && k == (unsigned)i;
        cum += shorter ? h[i] : 0u;
        k += shorter;
    }
    SelPick p;
    p.bin = __shfl_sync(TT_FULL_MASK, 8u * lane + k, ln);
    p.below = __shfl_sync(TT_FULL_MASK, cum, ln);
    p.total = total;
    return p;
}

// Is key k in bin `bin` of a histogram (bs as in sel_bin)?
struct SelTest {
    float bs;
    unsigned first, span;
    __device__ __forceinline__ SelTest(float bs_, unsigned bin)
        : bs(bs_), first(kSelOne + bin),
          span(bin == kSelBins - 1 ? 0xffffffffu - kSelOne - bin : 0u) {}
    __device__ __forceinline__ bool operator()(float k) const {
        return __float_as_uint(fmaf(k, bs, 8388608.f)) - first <= span;
    }
};

// Append (key, sample) of the lanes with `in` set to the list (counted past
// its end, never written there); kTeam: several warps append to it.
template <bool kTeam = false>
__device__ __forceinline__ void sel_append(SelScratch *sc, int &count, bool in, float k, float v,
                                           int lane) {
    const unsigned m = __ballot_sync(TT_FULL_MASK, in);
    if (kTeam) {
        if (!m)
            return;
        int at = 0;
        if (lane == 0)
            at = atomicAdd(&sc->count, __popc(m));
        count = __shfl_sync(TT_FULL_MASK, at, 0);
    }
    const int pos = count + __popc(m & ((1u << lane) - 1u));
    if (in && pos < kSelList)
        sc->list[pos] = make_uint2(__float_as_uint(k), __float_as_uint(v));
    count += __popc(m);
}

// The answer from a list of count <= kSelList (key, sample) entries: the
// smallest key with 2 (below + weight of the entries up to it) >= total.
// Keys are compared as bit patterns (the order of non-negative floats).
template <class WFn>
__device__ __forceinline__ float sel_answer(SelScratch *sc, int count, unsigned below,
                                            unsigned total, WFn wfn, int lane) {
    for (int i = lane; i < count; i += 32)
        sc->list[i].y = wfn(__uint_as_float(sc->list[i].y));
    __syncwarp();
    unsigned best = 0xffffffffu, last = 0u;
    for (int o = 0; o < count; o += 32) {
        const bool own = o + lane < count;
        const unsigned k = own ? sc->list[o + lane].x : 0u;
        unsigned w = below;
#pragma unroll 4
        for (int i = 0; i < count; i++) {
            const uint2 e = sc->list[i];
            w += e.x <= k ? e.y : 0u;
        }
        if (own && 2u * w >= total)
            best = min(best, k);
        last = max(last, k);
    }
    best = __reduce_min_sync(TT_FULL_MASK, best);
    last = __reduce_max_sync(TT_FULL_MASK, last); // never needed: the bin holds the crossing
    return __uint_as_float(best == 0xffffffffu ? last : best);
}

// Refinement of a crossing bin that held more than kSelList entries: `in` tells
// its members among the line's elements e in [0, cnt) (samples xb[e], keys
// keyfn(e, v)).  Each level histograms the bit patterns of the members' keys
// (as integers in the floats' order; -0, of no weight, is below the range) from
// the lowest to the highest, 256 bins: at most 31 bits to begin with and 8 fewer
// after each level.  Not unrolled: that spilled in the callers' hot loops
// (4096^2 x 720 angles, T0-T7: 66.3 ms, 65.3 rolled).
template <class KeyFn, class WFn>
__device__ __noinline__ float sel_refine(const float *xb, int cnt, KeyFn keyfn, WFn wfn,
                                         SelTest in, SelPick p, SelScratch *sc, int lane) {
    int lo = 0, hi = 0x7f800000; // the members' range
    for (int level = 0; level < 5; level++) {
        int mn = INT_MAX, mx = 0;
#pragma unroll 1
        for (int e = lane; e < cnt; e += 32) {
            const float k = keyfn(e, xb[e]);
            const int u = __float_as_int(k);
            if (u >= lo && u <= hi && (level > 0 || in(k))) {
                mn = min(mn, u);
                mx = max(mx, u);
            }
        }
        lo = __reduce_min_sync(TT_FULL_MASK, mn);
        hi = __reduce_max_sync(TT_FULL_MASK, mx);
        if (hi <= lo)
            break;
        const int shift = max(24 - __clz(hi - lo), 0);
        __syncwarp();
        sel_clear(sc, lane);
        __syncwarp();
#pragma unroll 1
        for (int e = lane; e < cnt; e += 32) {
            const float v = xb[e];
            const int u = __float_as_int(keyfn(e, v));
            if (u >= lo && u <= hi)
                atomicAdd(sc->hist + ((u - lo) >> shift), wfn(v));
        }
        __syncwarp();
        p = sel_pick<false>(sc, p.below, p.total, lane);
        lo += (int)p.bin << shift;
        hi = min(hi, lo + ((1 << shift) - 1));
        __syncwarp();
        int count = 0;
#pragma unroll 1
        for (int e0 = 0; e0 < cnt; e0 += 32) {
            const int e = e0 + lane;
            const float v = e < cnt ? xb[e] : 0.f, k = keyfn(e, v);
            const int u = __float_as_int(k);
            sel_append(sc, count, e < cnt && u >= lo && u <= hi, k, v, lane);
        }
        __syncwarp();
        if (count <= kSelList)
            return sel_answer(sc, count, p.below, p.total, wfn, lane);
    }
    return __int_as_float(min(lo, hi));
}

// Clears a line's two histograms; before the team's next sync, which comes
// before select_t67.
template <int TW>
__device__ __forceinline__ void sel_begin(SelScratch *s6, SelScratch *s7, SelTeam<TW> team,
                                          int lane) {
    if (TW == 1 || team.role == TW - 1)
        sel_clear(s7, lane);
    if (TW == 1 || team.role == TW - 2)
        sel_clear(s6, lane);
    if (TW > 1 && team.role == TW - 1 && lane == 0) {
        s7->wtop = 0u;
        s7->count = s6->count = 0;
    }
    if (TW == 1)
        __syncwarp();
}

// T6 and T7 of one line (c++/src/functionals.cpp:226-276).  T6: keys
// r1 * x[m2 + r1], r1 in [0, N - m2); T7: keys x[m1 ..]; both weighted by
// sqrt(x).  Elements are the line's stored rows at x[row - jlo]; every other
// row is a zero sample (key 0, weight 0), which cannot move the crossing
// unless all weights are zero, in which case the reference returns its
// smallest key, 0.  One histogram pass and one collecting pass serve both (a
// chunked sweep: far-apart elements in flight, so fewer atomic collisions).
// xmax and qtot (the line's largest sample and sum of square roots) bound
// every key and weight total, so no separate range pass is needed; odd: some
// sample is none sqrt_pos takes.  The line's TW warps share both passes; T7's
// answer is the first one's, T6's the second one's (TW = 1: both its own).
template <int TW>
__device__ __forceinline__ void select_t67(const float *x, int jlo, int jhi, int m1, int m2,
                                           bool want6, bool want7, float xmax, float qtot,
                                           bool odd, SelScratch *s6, SelScratch *s7,
                                           SelTeam<TW> team, int lane, float *r6, float *r7) {
    *r6 = 0.f;
    *r7 = 0.f;
    const int b7 = max(m1, jlo), b6 = max(m2, jlo);
    const int b = min(want7 ? b7 : jhi, want6 ? b6 : jhi);
    const int cnt = jhi - b;
    if (cnt <= 0 || !(xmax > 0.f) || !(qtot > 0.f))
        return;
    const int per = ((cnt + 32 * TW - 1) / (32 * TW)) | 1; // odd: conflict-free chunks
    const SqrtWeight wfn{sel_scale(qtot), odd};
    const float k6max = __fmul_rn((float)max(jhi - 1 - m2, 0), xmax);
    want6 = want6 && k6max > 0.f; // otherwise every T6 key is 0
    const float bs7 = sel_per_key(xmax), bs6 = want6 ? sel_per_key(k6max) : 0.f;
    // element e of [0, cnt) is row b + e; this lane's are e0 .. e0 + mine - 1,
    // of which T7 takes those from i = f7 on and T6 those from f6
    const float *xb = x + (b - jlo);
    const int e0 = (team.role * 32 + lane) * per, mine = min(max(cnt - e0, 0), per);
    const int f7 = want7 ? b7 - b - e0 : per, f6 = want6 ? b6 - b - e0 : per;
    const float r0 = (float)(b + e0 - m2); // T6's factor of the lane's first element

    unsigned l7max = 0;
    float rf = r0; // exact: integers below 2^24
    // a warp-uniform trip count (per), lanes past their chunk predicated off
    for (int i0 = 0; i0 < per; i0 += 4, rf += 4.f) {
        float vb[4]; // four loads in flight before the atomics
#pragma unroll
        for (int u = 0; u < 4; u++)
            vb[u] = i0 + u < mine ? xb[e0 + i0 + u] : 0.f;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + u;
            const float v = vb[u];
            const unsigned wq = wfn(v); // 0 past the chunk
            l7max += v == xmax && i >= f7 ? wq : 0u;
            if (wq && i >= f7)
                atomicAdd(s7->hist + sel_bin(v, bs7), wq);
            if (wq && i >= f6)
                atomicAdd(s6->hist + sel_bin(__fmul_rn(rf + (float)u, v), bs6), wq);
        }
    }
    unsigned wtop = __reduce_add_sync(TT_FULL_MASK, l7max);
    if (TW > 1 && lane == 0 && wtop)
        atomicAdd(&s7->wtop, wtop);
    team.sync();
    SelPick p7{0u, 0u, 0u}, p6{0u, 0u, 0u};
    const int own6 = TW > 1 ? 1 : 0; // the warp that finishes T6
    if (want7 && team.role == 0)
        p7 = sel_pick<true>(s7, 0u, 0u, lane);
    if (want6 && team.role == own6)
        p6 = sel_pick<true>(s6, 0u, 0u, lane);
    if (TW > 1) {
        if (lane == 0 && team.role == 0)
            s7->pick = p7;
        if (lane == 0 && team.role == own6)
            s6->pick = p6;
    }
    team.sync(); // both histograms are read: the lists take their place
    if (TW > 1) {
        p7 = s7->pick;
        p6 = s6->pick;
        wtop = s7->wtop;
    }
    // Saturated lines (samples clipped at the image's maximum) put the
    // crossing on the largest key: when the keys below the maximum weigh
    // less than half the total, 2 W(< xmax) < W, the answer is xmax.
    if (want7 && wtop > 0 && 2u * (p7.total - wtop) < p7.total) {
        *r7 = xmax;
        want7 = false;
    }
    if (!want6 && !want7)
        return;
    const SelTest in7(bs7, p7.bin), in6(bs6, p6.bin);
    int c6 = 0, c7 = 0;
    rf = r0;
    for (int i0 = 0; i0 < per; i0 += 4, rf += 4.f) {
        float vb[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            vb[u] = i0 + u < mine ? xb[e0 + i0 + u] : 0.f;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + u;
            const float v = vb[u], k6 = __fmul_rn(rf + (float)u, v);
            const bool a7 = want7 && i >= f7 && i < mine && in7(v);
            const bool a6 = want6 && i >= f6 && i < mine && in6(k6);
            if (__any_sync(TT_FULL_MASK, a7 || a6)) {
                sel_append<(TW > 1)>(s7, c7, a7, v, v, lane);
                sel_append<(TW > 1)>(s6, c6, a6, k6, v, lane);
            }
        }
    }
    team.sync();
    if (TW > 1) {
        c7 = s7->count;
        c6 = s6->count;
    }
    if (want7 && team.role == 0) {
        if (c7 <= kSelList) {
            *r7 = sel_answer(s7, c7, p7.below, p7.total, wfn, lane);
        } else {
            const int o7 = b7 - b;
            *r7 = sel_refine(xb + o7, cnt - o7, [](int, float v) { return v; }, wfn, in7, p7, s7,
                             lane);
        }
    }
    if (want6 && team.role == own6) {
        if (c6 <= kSelList) {
            *r6 = sel_answer(s6, c6, p6.below, p6.total, wfn, lane);
        } else {
            const int o6 = b6 - b;
            const float rb = (float)(b6 - m2);
            *r6 = sel_refine(xb + o6, cnt - o6,
                             [rb](int e, float v) { return __fmul_rn(rb + (float)e, v); }, wfn,
                             in6, p6, s6, lane);
        }
    }
}

// PFunctional2 of one non-negative column (c++/src/functionals.cpp:303-311):
// the column sorted, weighted by itself, its weighted median -- the smallest
// value v with 2 * sum(x <= v) >= sum(x), found without sorting.  x: the
// column in shared memory, n values, xmax their maximum, xsum their sum (a
// bound for the fixed-point scale).  One warp.
inline __device__ float select_p2(const float *x, int n, float xmax, float xsum, SelScratch *sc,
                                  int lane) {
    if (n <= 0)
        return 0.f;
    if (!(xmax > 0.f) || !(xsum > 0.f))
        return 0.f; // all zero: the first sorted value
    const int per = ((n + 31) >> 5) | 1;
    const int j0 = lane * per, mine = min(max(n - j0, 0), per);
    const LinearWeight wfn{sel_scale(xsum)};
    const float bs = sel_per_key(xmax);
    sel_clear(sc, lane);
    __syncwarp();
    for (int i0 = 0; i0 < per; i0 += 4) { // warp-uniform trip count
        float vb[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            vb[u] = i0 + u < mine ? x[j0 + i0 + u] : 0.f;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const unsigned wq = wfn(vb[u]);
            if (wq)
                atomicAdd(sc->hist + sel_bin(vb[u], bs), wq);
        }
    }
    __syncwarp();
    const SelPick p = sel_pick<true>(sc, 0u, 0u, lane);
    __syncwarp();
    const SelTest in(bs, p.bin);
    int c = 0;
    for (int i0 = 0; i0 < per; i0 += 4) {
        float vb[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            vb[u] = i0 + u < mine ? x[j0 + i0 + u] : 0.f;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const bool a = i0 + u < mine && in(vb[u]);
            if (__any_sync(TT_FULL_MASK, a))
                sel_append(sc, c, a, vb[u], vb[u], lane);
        }
    }
    __syncwarp();
    if (c <= kSelList)
        return sel_answer(sc, c, p.below, p.total, wfn, lane);
    return sel_refine(x, n, [](int, float v) { return v; }, wfn, in, p, sc, lane);
}

} // namespace tt
