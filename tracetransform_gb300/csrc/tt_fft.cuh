// tt_fft.cuh -- the chirp-z (Bluestein) DFT of a column pair in one CTA.
//
// A complex DFT of any length n is a circular convolution of M = 2^LOGM >=
// 2n - 1 points: F_k = w_k sum_j (z_j w_j) conj(w_{k-j}), w_j = exp(-i pi
// j^2 / n).  The sinogram columns are real, so two of them ride in one
// transform, z = x1 + i x2 (F1 and F2 are the Hermitian and anti-Hermitian
// parts of F): half the transforms per column.
//
// The M-point transform runs in shared memory in radix-16 passes: a thread
// holds 16 elements in registers, so the data crosses shared memory (LOGM -
// 1) / 4 times instead of LOGM times for radix 2.  LOGM is split as one
// leading radix 2, 4, 8 or 16 and then 16s.  The forward passes decimate in
// frequency (natural input, digit-reversed output), the inverse ones undo
// them in mirrored order, so nothing is ever bit-reversed: the filter table
// is stored in the digit-reversed order instead, and the last forward pass,
// the product with the filter and the first inverse pass share one trip
// through registers.  Element i sits at i + i / 16, which makes the stride-1
// groups of 16 of that pass free of bank conflicts; every other pass has
// lanes on consecutive elements.  Bound by shared-memory traffic and the
// barriers between passes (6 trips of 128 KB each way at M = 16384, one CTA
// per SM).
#pragma once

#include "tt_common.cuh"
#include "tt_internal.h"

namespace tt {

constexpr int kFftMinLog = 6, kFftMaxLog = 14; // transform lengths 64 .. 16384

__host__ __device__ constexpr int fft_pad(int i) { return i + (i >> 4); }
// log2 of the leading pass's radix
__host__ __device__ constexpr int fft_lead(int logm) { return ((logm - 1) & 3) + 1; }
__host__ __device__ constexpr int fft_threads(int logm) {
    return logm <= 9 ? 32 : logm >= 13 ? 512 : 1 << (logm - 4);
}
// float2 entries of shared memory one transform needs
__host__ __device__ constexpr int fft_smem_len(int logm) { return fft_pad(1 << logm); }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmul_conj(float2 a, float2 b) { // a conj(b)
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
    return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
    return make_float2(a.x - b.x, a.y - b.y);
}
// a times -i (forward) or +i (inverse)
template <bool kInv> __device__ __forceinline__ float2 crot(float2 a) {
    return kInv ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
// a times exp(-+ 2 pi i / 16 * q) for the roots a radix-8 / 16 butterfly uses, the
// roots as sums of two floats: unlike the table's twiddles, whose roundings
// average out, these few enter every butterfly of every pass, and rounded to
// floats they made P3 systematically small (by 1.8e-7 at 2049 rows, 0.5e-7 so).
// Where the passes wait for shared memory this costs nothing (P1-P3 of 5760 columns
// of 5793 rows 737 us either way); the adjoint of 69120 columns of 363 rows takes
// 441 us, from 430.
template <bool kInv, int q> __device__ __forceinline__ float2 croot16(float2 a) {
    constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173,
                     h = 0.70710678118654752440;
    if constexpr (q == 0)
        return a;
    else if constexpr (q == 4)
        return crot<kInv>(a);
    else {
        static_assert(q == 1 || q == 2 || q == 3 || q == 6 || q == 9, "roots of the 4 x 4 split");
        constexpr double re = q == 1 ? c1 : q == 2 ? h : q == 3 ? s1 : q == 6 ? -h : -c1;
        constexpr double up = q == 1 ? s1 : q == 2 ? h : q == 3 ? c1 : q == 6 ? h : -s1;
        constexpr double im = kInv ? up : -up;
        constexpr float c = (float)re, cl = (float)(re - (double)c);
        constexpr float s = (float)im, sl = (float)(im - (double)s);
        return make_float2(fmaf(a.x, c, fmaf(-a.y, s, fmaf(a.x, cl, -a.y * sl))),
                           fmaf(a.x, s, fmaf(a.y, c, fmaf(a.x, sl, a.y * cl))));
    }
}

template <bool kInv>
__device__ __forceinline__ void dft4(float2 &v0, float2 &v1, float2 &v2, float2 &v3) {
    const float2 a = cadd(v0, v2), b = csub(v0, v2), c = cadd(v1, v3),
                 d = crot<kInv>(csub(v1, v3));
    v0 = cadd(a, c);
    v1 = cadd(b, d);
    v2 = csub(a, c);
    v3 = csub(b, d);
}

// DFT of R values in registers, natural order in and out.
template <int R, bool kInv> __device__ __forceinline__ void dft_small(float2 (&v)[R]) {
    if constexpr (R == 2) {
        const float2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    } else if constexpr (R == 4) {
        dft4<kInv>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) { // j = 2 j1 + j2, k = k1 + 4 k2
        dft4<kInv>(v[0], v[2], v[4], v[6]);
        dft4<kInv>(v[1], v[3], v[5], v[7]);
        const float2 o[4] = {v[1], croot16<kInv, 2>(v[3]), croot16<kInv, 4>(v[5]),
                             croot16<kInv, 6>(v[7])};
        const float2 e[4] = {v[0], v[2], v[4], v[6]};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = cadd(e[k], o[k]);
            v[k + 4] = csub(e[k], o[k]);
        }
    } else { // 16: j = 4 j1 + j2, k = k1 + 4 k2
        static_assert(R == 16, "radices 2, 4, 8, 16");
#pragma unroll
        for (int j2 = 0; j2 < 4; j2++)
            dft4<kInv>(v[j2], v[4 + j2], v[8 + j2], v[12 + j2]);
        // now v[4 k1 + j2]; times W16^(j2 k1)
        v[5] = croot16<kInv, 1>(v[5]);
        v[6] = croot16<kInv, 2>(v[6]);
        v[7] = croot16<kInv, 3>(v[7]);
        v[9] = croot16<kInv, 2>(v[9]);
        v[10] = croot16<kInv, 4>(v[10]);
        v[11] = croot16<kInv, 6>(v[11]);
        v[13] = croot16<kInv, 3>(v[13]);
        v[14] = croot16<kInv, 6>(v[14]);
        v[15] = croot16<kInv, 9>(v[15]);
#pragma unroll
        for (int k1 = 0; k1 < 4; k1++)
            dft4<kInv>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
        // v[4 k1 + k2] is output k1 + 4 k2: transpose
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = a + 1; b < 4; b++) {
                const float2 t = v[4 * a + b];
                v[4 * a + b] = v[4 * b + a];
                v[4 * b + a] = t;
            }
    }
}

// The passes from sub-length 2^LOGL down to 16 and back up, in place.  tw:
// the twiddles of this pass ((R - 1) x stride, exp(-2 pi i j k / 2^LOGL) at
// (k - 1) stride + j), the following passes' behind them.  load(i) gives
// element i of the (leading) pass's input.
template <int LOGM, int LOGL, int LOGR, class Load>
__device__ __forceinline__ void fft_convolve_from(float2 *s, const float2 *__restrict__ tw,
                                                  const float2 *__restrict__ filt, Load load) {
    constexpr int T = fft_threads(LOGM), R = 1 << LOGR, N = 1 << (LOGM - LOGR);
    if constexpr (LOGL == 4) {
        // stride 1: forward, filter (digit-reversed order, [k][block]), inverse
        for (int b = threadIdx.x; b < N; b += T) {
            float2 *p = s + 17 * b;
            float2 v[16];
#pragma unroll
            for (int r = 0; r < 16; r++)
                v[r] = p[r];
            dft_small<16, false>(v);
#pragma unroll
            for (int k = 0; k < 16; k++)
                v[k] = cmul(v[k], __ldg(filt + k * N + b));
            dft_small<16, true>(v);
#pragma unroll
            for (int r = 0; r < 16; r++)
                p[r] = v[r];
        }
        __syncthreads();
    } else {
        constexpr int S = 1 << (LOGL - LOGR), SP = S + S / 16;
        static_assert(S >= 16, "padded strides");
        for (int i = threadIdx.x; i < N; i += T) {
            const int j = i & (S - 1), base = ((i >> (LOGL - LOGR)) << LOGL) + j;
            float2 v[R];
#pragma unroll
            for (int r = 0; r < R; r++)
                v[r] = load(base + r * S);
            dft_small<R, false>(v);
            float2 *p = s + fft_pad(base);
            p[0] = v[0];
#pragma unroll
            for (int k = 1; k < R; k++)
                p[k * SP] = cmul(v[k], __ldg(tw + (k - 1) * S + j));
        }
        __syncthreads();
        fft_convolve_from<LOGM, LOGL - LOGR, 4>(s, tw + (R - 1) * S, filt,
                                                [s](int i) { return s[fft_pad(i)]; });
        for (int i = threadIdx.x; i < N; i += T) {
            const int j = i & (S - 1), base = ((i >> (LOGL - LOGR)) << LOGL) + j;
            float2 *p = s + fft_pad(base);
            float2 v[R];
            v[0] = p[0];
#pragma unroll
            for (int k = 1; k < R; k++)
                v[k] = cmul_conj(p[k * SP], __ldg(tw + (k - 1) * S + j));
            dft_small<R, true>(v);
#pragma unroll
            for (int r = 0; r < R; r++)
                p[r * SP] = v[r];
        }
        __syncthreads();
    }
}

// Circular convolution of load(0 .. M-1) with the filter; the result is at
// s[fft_pad(i)], in natural order, for every thread on return.  s must not be
// in use by anyone on entry.
template <int LOGM, class Load>
__device__ __forceinline__ void fft_convolve(float2 *s, const float2 *__restrict__ tw,
                                             const float2 *__restrict__ filt, Load load) {
    static_assert(LOGM >= kFftMinLog && LOGM <= kFftMaxLog, "transform length");
    fft_convolve_from<LOGM, LOGM, fft_lead(LOGM)>(s, tw, filt, load);
}

// Whether two columns of squared norms q1 and q2 share a transform: both are
// normal floats.  A zero, subnormal or non-finite one has no scale below that
// brings its column to its neighbour's size; such columns take transforms of
// their own, as they are.
__device__ __forceinline__ bool pair_shares(float q1, float q2) {
    const float inf = __int_as_float(0x7f800000);
    return q1 >= 0x1p-126f && q2 >= 0x1p-126f && q1 < inf && q2 < inf;
}

// 2^-e and 2^e for a column of squared norm ss (a normal float, else of no
// use), e half of its exponent, so that both columns of a pair enter the
// transform with norms of about one (a small column must not drown in the
// rounding of a large neighbour).
struct PairScale {
    float down, up;
};
__device__ __forceinline__ PairScale pair_scale(float ss) {
    const int e = (((__float_as_int(ss) >> 23) & 0xff) - 127) >> 1; // -63 .. 63 if normal
    return PairScale{__int_as_float((127 - e) << 23), __int_as_float((127 + e) << 23)};
}

// F1_k and F2_k from Z = DFT(x1 + i x2): Zk = Z_k, Zm = Z_{n-k}.
__device__ __forceinline__ float2 pair_first(float2 Zk, float2 Zm) {
    return make_float2(0.5f * (Zk.x + Zm.x), 0.5f * (Zk.y - Zm.y));
}
__device__ __forceinline__ float2 pair_second(float2 Zk, float2 Zm) {
    return make_float2(0.5f * (Zk.y + Zm.y), 0.5f * (Zm.x - Zk.x));
}

} // namespace tt
