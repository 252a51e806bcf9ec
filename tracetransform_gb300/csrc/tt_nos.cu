// tt_nos.cu -- nearest orthonormal sinogram on the device.
//
// The reference's orthonormal mode (c++/src/circus.cpp:68-102) shifts every
// sinogram column by its weighted-median offset into an m x A matrix
// (m = N + padding) and replaces it by the polar factor U V^T of its SVD,
// computed by Eigen's float JacobiSVD with a column-pivoting Householder QR
// preconditioner.  Here, for n_sino sinograms at once, the same structure
// with the precision split that GB300's rates call for: no FP64 at all
// (its pipe is narrow enough that a few scalar FP64 operations per step
// dominate), double-float pairs on the FP32 pipes where float is too short:
//
//   nos_offsets   per column: weighted median row - center, with the
//                 reference's sequential float sums (one warp per column)
//   nos_align     the shifted columns into a zeroed m x A matrix of
//                 double-float pairs (hi + lo, ~48 significant bits)
//   QR            column-pivoting Householder QR, A P = Q R, in double-float
//                 (the only stage beyond float precision: it fixes the small
//                 singular directions that a float factorisation would lose;
//                 the O(m A) work per step runs on the FP32 pipes); one
//                 launch per column step, in which every CTA picks the pivot
//                 itself and applies the reflector to its own columns,
//                 LAPACK-style otherwise (tau, partial column norms downdated
//                 and recomputed when cancellation sets in)
//   Jacobi        one-sided Jacobi on X = R^T in float (R^T of a pivoted QR is
//                 graded, so float rotations keep relative accuracy), block-
//                 cyclic: round-robin rounds of 12-column block pairs, each
//                 pair rotated in one CTA's shared memory; V follows a
//                 sweep behind through the rounds' accumulated rotations;
//                 X V = U_X S, so polar(R) = V U_X^T
//   assemble      P = V U_X^T (float) with one Newton-Schulz step to clean
//                 its orthogonality, then polar(A P) = Q [P; 0] applied
//                 reflector by reflector to groups of columns held in
//                 registers (up to 4096 aligned rows) or by blocks of 32
//                 reflectors in compact-WY form (above), straight into the
//                 result columns, which undoes the column permutation
//
// Against the oracle's double one-sided Jacobi on the aligned matrix the
// result agrees to ~3e-5 absolute (entries up to ~0.7) for condition numbers
// up to ~1e6; Eigen's float SVD of the same matrices is far less accurate.
// Every launch is bounded; there is no grid-wide wait.
#include <climits>

#include "tt_common.cuh"
#include "tt_internal.h"

namespace tt {
namespace {

// Weighted-median row - center of every column, one warp per column: the column is
// copied to shared memory, lane 0 replaces it by its running sums in
// the reference's order (the sum is the last of them, and the second pass's
// integral is the first pass's running sum again), and the warp looks for the
// first that reaches half the total.  Bound by that lane's chain of additions,
// 4 cycles a row.  8 x 360 columns of 1449 rows: 24 us, from 197 (one thread per column
// reading it twice, 32 cache lines per load, before).
constexpr int kOffWarps = 4, kOffPad = 16;
__host__ __device__ constexpr int offsets_stride(int rows) {
    return (rows + kOffPad - 1) / kOffPad * kOffPad + kOffPad; // one block read ahead
}
__global__ void __launch_bounds__(32 * kOffWarps)
nos_offsets_kernel(const float *__restrict__ sino, int rows, int n_cols, int center,
                   int *__restrict__ offsets) {
    extern __shared__ __align__(16) float s_off[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long idx = blockIdx.x * (long long)kOffWarps + warp;
    if (idx >= n_cols)
        return; // whole warps, no CTA barrier
    const int stride = offsets_stride(rows);
    float *x = s_off + (size_t)warp * stride;
    const float *src = sino + (size_t)idx * rows;
    for (int i = lane; i < stride; i += 32)
        x[i] = i < rows ? src[i] : 0.f;
    __syncwarp();
    if (lane == 0) {
        constexpr int kV = kOffPad / 4;
        float4 *x4 = reinterpret_cast<float4 *>(x), v[kV], next[kV];
#pragma unroll
        for (int u = 0; u < kV; u++)
            v[u] = x4[u];
        float sum = 0.f;
        for (int i = 0; i < rows; i += kOffPad, x4 += kV) {
#pragma unroll
            for (int u = 0; u < kV; u++)
                next[u] = x4[kV + u];
#pragma unroll
            for (int u = 0; u < kV; u++) {
                v[u].x = sum = __fadd_rn(sum, v[u].x);
                v[u].y = sum = __fadd_rn(sum, v[u].y);
                v[u].z = sum = __fadd_rn(sum, v[u].z);
                v[u].w = sum = __fadd_rn(sum, v[u].w);
                x4[u] = v[u];
                v[u] = next[u];
            }
        }
    }
    __syncwarp();
    const float sum = x[rows - 1];
    int m = rows - 1;
    for (int i0 = 0; i0 < rows; i0 += 32) {
        const int i = i0 + lane;
        const unsigned b = __ballot_sync(TT_FULL_MASK, i < rows && 2.f * x[min(i, rows - 1)] >= sum);
        if (b) {
            m = i0 + __ffs(b) - 1;
            break;
        }
    }
    if (lane == 0)
        offsets[idx] = m - center;
}

// The same, one thread per column, for columns over nos_max_rows(): these only
// tell how many aligned rows the call asks for, which is then refused.
__global__ void nos_offsets_long_kernel(const float *sino, int rows, int n_cols, int center,
                                        int *offsets) {
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= n_cols)
        return;
    const float *x = sino + (size_t)idx * rows;
    float sum = 0.f;
    for (int i = 0; i < rows; i++)
        sum = __fadd_rn(sum, x[i]);
    float integral = 0.f;
    int m = rows - 1;
    for (int i = 0; i < rows; i++) {
        integral = __fadd_rn(integral, x[i]);
        if (2.f * integral >= sum) {
            m = i;
            break;
        }
    }
    offsets[idx] = m - center;
}

// ---- double-float arithmetic -------------------------------------------------
//
// The aligned matrices hold each element as an unevaluated sum hi + lo of two
// floats (~48 significant bits).  The QR's O(m n) work -- dot products and
// trailing updates -- runs on these pairs with error-free float transforms
// (Knuth's two-sum, the FMA two-product, Dekker's renormalisation; the
// products that feed a two-sum are __fmul_rn, which the compiler never
// contracts into a fused multiply-add), i.e. on
// the FP32 pipes, which GB300 runs far faster than FP64; so do the scalars
// (norms, reflector coefficients, with double-float division and square
// root): a handful of FP64 operations per column step, each waiting on the
// narrow FP64 pipe, cost more than the step's O(m n) double-float work.

__device__ __forceinline__ float2 df_quick(float a, float b) { // |a| >= |b|
    const float s = a + b;
    return make_float2(s, b - (s - a));
}
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
    const float s = a.x + b.x, bb = s - a.x;
    const float e = (a.x - (s - bb)) + (b.x - bb);
    return df_quick(s, e + a.y + b.y);
}
__device__ __forceinline__ float2 df_mul(float2 a, float2 b) {
    const float p = __fmul_rn(a.x, b.x); // never contracted into a later add
    float e = fmaf(a.x, b.x, -p);
    e = fmaf(a.x, b.y, e);
    e = fmaf(a.y, b.x, e);
    return df_quick(p, e);
}
// acc + a b with the product's rounding error carried into the low word
// instead of renormalising the product first
__device__ __forceinline__ float2 df_fma(float2 a, float2 b, float2 acc) {
    const float p = __fmul_rn(a.x, b.x); // never contracted into a later add
    float e = fmaf(a.x, b.x, -p);
    e = fmaf(a.x, b.y, e);
    e = fmaf(a.y, b.x, e);
    const float s = acc.x + p, bb = s - acc.x;
    const float err = (acc.x - (s - bb)) + (p - bb);
    return df_quick(s, err + e + acc.y);
}
// Compensated dot product of double-float vectors (Ogita, Rump and Oishi's
// Dot2, extended by the low-word cross terms): the high words' products go
// into s with Knuth's two-sum, whose errors, the products' FMA rounding
// errors and the cross terms collect in e; only s + p is on the dependent
// path per element.  df_dot_end renormalises.
struct DfDot {
    float s = 0.f, e = 0.f;
};
__device__ __forceinline__ void df_dot_add(DfDot &d, float2 a, float2 b) {
    const float p = __fmul_rn(a.x, b.x); // never contracted into a later add
    const float pe = fmaf(a.x, b.x, -p);
    const float t = d.s + p, bb = t - d.s;
    const float err = (d.s - (t - bb)) + (p - bb);
    d.e += (err + pe) + fmaf(a.x, b.y, a.y * b.x);
    d.s = t;
}
__device__ __forceinline__ float2 df_dot_end(DfDot d) { return df_quick(d.s, d.e); }
__device__ __forceinline__ float2 df_neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 df_sub(float2 a, float2 b) { return df_add(a, df_neg(b)); }
// a / b: float quotient, corrected once by the double-float remainder
__device__ __forceinline__ float2 df_div(float2 a, float2 b) {
    const float q1 = a.x / b.x;
    const float2 r = df_sub(a, df_mul(make_float2(q1, 0.f), b));
    return df_quick(q1, r.x / b.x);
}
// sqrt(a), a >= 0: float root, corrected once by the double-float residual
__device__ __forceinline__ float2 df_sqrt(float2 a) {
    if (!(a.x > 0.f))
        return make_float2(0.f, 0.f);
    const float r0 = sqrtf(a.x);
    const float2 res = df_sub(a, df_mul(make_float2(r0, 0.f), make_float2(r0, 0.f)));
    return df_quick(r0, res.x / (2.f * r0));
}
__device__ __forceinline__ float2 df_shfl_xor(float2 v, int o) {
    return make_float2(__shfl_xor_sync(TT_FULL_MASK, v.x, o),
                       __shfl_xor_sync(TT_FULL_MASK, v.y, o));
}

// grid (cols, n_sino); A_s must be zeroed before.
__global__ void nos_align_kernel(const float *__restrict__ sino, int rows, int cols,
                                 const NosDesc *__restrict__ desc,
                                 const int *__restrict__ offsets, float2 *__restrict__ A) {
    const int col = blockIdx.x, s = blockIdx.y;
    const NosDesc d = desc[s];
    const int shift = d.mx - offsets[(size_t)s * cols + col];
    const float *src = sino + ((size_t)s * cols + col) * rows;
    float2 *dst = A + d.a_off + (size_t)col * d.ld + shift;
    for (int r = threadIdx.x; r < rows; r += blockDim.x)
        dst[r] = make_float2(src[r], 0.f);
}

template <int kThreads> __device__ __forceinline__ float2 block_sum_df(float2 v, float2 *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = df_add(v, df_shfl_xor(v, o));
    if (lane == 0)
        red[warp] = v;
    __syncthreads();
    float2 t = red[0];
#pragma unroll
    for (int w = 1; w < kThreads / 32; w++)
        t = df_add(t, red[w]);
    __syncthreads();
    return t;
}

// ---- column-pivoting Householder QR (double-float) ---------------------------

constexpr int kQrThreads = 256;

// Squared column norms (partial, by position, in the step-0 half of the
// double buffer, double-float; and the reference copy, by stored column,
// float) and the identity position map.  grid (n, n_sino).
__global__ void __launch_bounds__(kQrThreads)
qr_init_kernel(const float2 *__restrict__ A, const NosDesc *__restrict__ desc, int n,
               NosWork w) {
    __shared__ float2 red[kQrThreads / 32];
    const int j = blockIdx.x, s = blockIdx.y;
    const NosDesc d = desc[s];
    const float2 *a = A + d.a_off + (size_t)j * d.ld;
    float2 v = make_float2(0.f, 0.f);
    for (int i = threadIdx.x; i < d.m; i += kQrThreads)
        v = df_fma(a[i], a[i], v);
    v = block_sum_df<kQrThreads>(v, red);
    if (threadIdx.x == 0) {
        w.norms[(size_t)s * n + j] = v;
        w.orig[(size_t)s * n + j] = v.x;
        w.cmap[(size_t)s * n + j] = j;
    }
}

// Warp-then-block double-float sum through red[T / 32]; one barrier.
// Consecutive calls must alternate between two red buffers.
template <int T> __device__ __forceinline__ float2 qr_block_sum(float2 v, float2 *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = df_add(v, df_shfl_xor(v, o));
    if (lane == 0)
        red[warp] = v;
    __syncthreads();
    v = red[0];
#pragma unroll
    for (int u = 1; u < T / 32; u++)
        v = df_add(v, red[u]);
    return v;
}

// GB double-float warp sums in the butterfly's order (the lower lane's operand
// first): lane g (32 / GB) ends with sum g.  Four sums share their first two
// levels: each lane keeps the half of them that its lane bit selects.
template <int GB> __device__ __forceinline__ float2 qr_warp_sums(float2 (&v)[GB], int lane) {
    static_assert(GB == 1 || GB == 2 || GB == 4, "halving exchanges");
    int o = 16;
#pragma unroll
    for (int h = GB / 2; h > 0; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const float2 mine = up ? v[i + h] : v[i], give = up ? v[i] : v[i + h];
            const float2 got = df_shfl_xor(give, o);
            v[i] = df_add(up ? got : mine, up ? mine : got);
        }
    }
#pragma unroll
    for (; o > 0; o >>= 1)
        v[0] = df_add(v[0], df_shfl_xor(v[0], o));
    return v[0];
}

// Column step k of the pivoted QR in one launch, grid (G, n_sino): CTA b
// handles positions k + b, k + b + G, ... in groups of GB (G is chosen so that
// the grid is one wave).
//
// Every CTA picks the pivot itself -- the remaining position of largest
// partial norm, lowest position on ties -- and reads the pivot column
// x = A[k:, c_p].  The CTA owning position p stores the reflector's scalars
// (beta = R[k, k], scale = 1 / (alpha - beta), tau); every other column gets
// H = I - tau v v^T, v = (1, x[k+1:] scale), in place, with
// v . a = a[k] + scale (x[k+1:] . a[k+1:]), and then its partial norm loses
// a[k]^2 (recomputed from the column when that leaves less than ~sqrt(eps)
// of the norm at the last recompute, as LAPACK does).
//
// Columns never move: cmap maps positions to stored columns and the pivot
// swap exchanges two of its entries.  The pivot column is left as it is (its
// rows above k are R[:k, k], those below k the reflector up to `scale`), so
// no CTA writes what another reads in the same step; the partial norms (by
// position) and cmap are double-buffered by step parity.  perm[k] receives
// the stored column that ends at position k.
//
// What bounds a step is the instructions issued per element, then the chain
// map, pivot, pivot column, sums, scalars, update.  Thread t holds rows
// k + 1 + t + T u, u < keff, of columns padded with zeros (nos_ld): every access is at a
// constant offset from one pointer per column, and no row is tested.  A
// group's columns come in by asynchronous copies issued before the pivot is
// known, into slots of shared memory that only their own thread reads (no
// barrier); a slot is refilled for the next group once its column is written.
// The sums of a whole group and |x|^2 share one barrier, lane g of every warp
// then forms column g's scalars, and the two divisions of the reflector run in
// two lanes.  Sums, updates and scalars are all double-float; their order
// hangs on T alone (polar factors of nearly dependent columns change visibly
// with their last bits).
// The whole orthonormal circus with an address and a row test per access, a
// reduction and a barrier per column, then by this alone, then with the other
// kernels of this file as they are now: 8 x 1449 x 360, 9.28, 8.4 and 7.90 ms;
// 4 x 450 x 360, 6.2, 5.6 and 4.89; 8 x 5793 x 720, 90.6, 87 and 85.6.  Two rows at a
// time in packed operations took 40 % fewer instructions and as long: a step then
// waits for its chain.
//
// K: rows per thread.  CTAs per SM: by registers (two floats per row of x, and
// more to have the column's loads in flight: bounds of 5 and 3 CTAs for K = 16 took
// 10.7 ms at 8 x 1700 x 360 and 12.7 at 8 x 3000 x 360, these 9.6 and 11.0) and by the
// slots' shared memory.  Groups of two: of four, fewer CTAs fit; of one, 8 x 5795
// x 720 takes a tenth longer.
constexpr int kQrGroup = 2;
__host__ __device__ constexpr size_t qr_smem(int K, int T) {
    return sizeof(float2) * (size_t)kQrGroup * K * T;
}
__host__ __device__ constexpr int qr_ctas(int K, int T) {
    return T == 128 ? (K == 4 ? 8 : K == 8 ? 6 : 3) : 1;
}
template <int K, int T>
__global__ void __launch_bounds__(T, qr_ctas(K, T))
qr_step_kernel(float2 *__restrict__ A, const NosDesc *__restrict__ desc, int n, int n_sino,
               int k, NosWork w) {
    constexpr int kW = T / 32, GB = kQrGroup, kStep = 32 / GB;
    extern __shared__ __align__(16) float2 s_slot[]; // [GB][K][T]
    __shared__ int s_bv[kW];
    __shared__ int s_bi[kW];
    __shared__ float2 s_xn[kW];
    __shared__ float2 s_dot[2][GB][kW];
    __shared__ float2 s_red[2][kW];
    const int s = blockIdx.y, G = gridDim.x, b = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const NosDesc d = desc[s];
    const size_t ld = d.ld;
    const int keff = (d.m - k - 1 + T - 1) / T; // slots that cover the rows below k
    float2 *As = A + d.a_off;
    const size_t cur = (size_t)(k & 1) * n_sino + s, nxt = (size_t)((k + 1) & 1) * n_sino + s;
    const float2 *nr = w.norms + cur * n;
    const int *cm = w.cmap + cur * n;
    float *og = w.orig + (size_t)s * n;
    const int j0 = k + b, cnt = (n - j0 + G - 1) / G;
    const int g_mine = lane % GB;   // the group's column whose scalars this lane forms
    float2 *slot = s_slot + threadIdx.x;
    auto below = [&](int c) { // this thread's rows of column c, T apart
        return As + c * ld + k + 1 + threadIdx.x;
    };
    auto issue = [&](int g, int c) { // column c into the slots of group member g
        const float2 *src = below(c);
        const unsigned dst = (unsigned)__cvta_generic_to_shared(slot + g * K * T);
#pragma unroll
        for (int u = 0; u < K; u++)
            if (u < keff)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                 dst + (unsigned)(u * T * sizeof(float2))),
                             "l"(src + u * T)
                             : "memory");
    };

    // first group, on its way while the pivot is chosen
    int c_mine = -1;     // stored column, -1 past the CTA's share
    float2 n_mine = make_float2(0.f, 0.f), k_mine = n_mine; // partial norm and a[k]
    float o_mine = 0.f;  // norm at the last recompute
    if (g_mine < cnt) {
        c_mine = cm[j0 + g_mine * G];
        n_mine = nr[j0 + g_mine * G];
    }
#pragma unroll
    for (int g = 0; g < GB; g++) {
        const int c = __shfl_sync(TT_FULL_MASK, c_mine, g);
        if (c >= 0)
            issue(g, c);
    }
    if (c_mine >= 0) {
        k_mine = As[c_mine * ld + k];
        o_mine = og[c_mine];
    }

    // pivot: argmax of the partial norms over positions k..n-1, compared as
    // the bit patterns of their (non-negative) high words on the integer
    // pipe; a NaN or negative norm counts as 0.  The stored column travels with
    // the position (n is far below 2^15).
    int best = -1, bidx = INT_MAX;
    for (int jj = k + threadIdx.x; jj < n; jj += T) {
        int v = __float_as_int(nr[jj].x);
        const int at = jj << 16 | cm[jj];
        if (v < 0 || v > 0x7F800000)
            v = 0;
        if (v > best) { // positions rise per thread: the first maximum stays
            best = v;
            bidx = at;
        }
    }
    {
        const int top = __reduce_max_sync(TT_FULL_MASK, best);
        bidx = __reduce_min_sync(TT_FULL_MASK, best == top ? bidx : INT_MAX);
        best = top;
    }
    if (lane == 0) {
        s_bv[warp] = best;
        s_bi[warp] = bidx;
    }
    __syncthreads();
    best = s_bv[0];
    bidx = s_bi[0];
#pragma unroll
    for (int u = 1; u < kW; u++)
        if (s_bv[u] > best || (s_bv[u] == best && s_bi[u] < bidx)) {
            best = s_bv[u];
            bidx = s_bi[u];
        }
    const int p = bidx >> 16, cp = bidx & 0xffff;
    const float2 *x = below(cp);
    float2 xv[K];
#pragma unroll
    for (int u = 0; u < K; u++)
        xv[u] = u < keff ? x[u * T] : make_float2(0.f, 0.f);
    const float2 xk = As[cp * ld + k];
    {
        DfDot dn[2];
#pragma unroll
        for (int u = 0; u < K; u++)
            if (u < keff)
                df_dot_add(dn[u & 1], xv[u], xv[u]);
        float2 xn = df_add(df_dot_end(dn[0]), df_dot_end(dn[1]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            xn = df_add(xn, df_shfl_xor(xn, o));
        if (lane == 0)
            s_xn[warp] = xn;
    }

    float2 scale_df = make_float2(0.f, 0.f), tau_df = scale_df;
    bool zero = false;
    int rb = 0, buf = 0;
    for (int t0 = 0; t0 < cnt; t0 += GB, buf ^= 1) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        const int live = min(GB, cnt - t0);
        float2 v[GB]; // x[k+1:] . a[k+1:] of the group's columns
#pragma unroll
        for (int g = 0; g < GB; g++) {
            DfDot dv[2];
            if (g < live) // uniform
#pragma unroll
                for (int u = 0; u < K; u++)
                    if (u < keff)
                        df_dot_add(dv[u & 1], xv[u], slot[(g * K + u) * T]);
            v[g] = df_add(df_dot_end(dv[0]), df_dot_end(dv[1]));
        }
        const float2 part = qr_warp_sums<GB>(v, lane);
        if (lane % kStep == 0)
            s_dot[buf][lane / kStep][warp] = part;
        __syncthreads();
        if (t0 == 0) {
            // reflector scalars (double-float, no FP64: GB300's FP64 pipe would
            // serialise them): even lanes divide for scale, odd ones for tau
            float2 xn = s_xn[0];
#pragma unroll
            for (int u = 1; u < kW; u++)
                xn = df_add(xn, s_xn[u]);
            zero = xn.x == 0.f; // uniform: H = I, x stays as it is
            float2 beta = xk;
            if (!zero) {
                const float2 root = df_sqrt(df_fma(xk, xk, xn));
                beta = xk.x >= 0.f ? df_neg(root) : root;
                const bool tau_lane = lane & 1;
                const float2 quot =
                    df_div(tau_lane ? df_sub(beta, xk) : make_float2(1.f, 0.f),
                           tau_lane ? beta : df_sub(xk, beta));
                scale_df = make_float2(__shfl_sync(TT_FULL_MASK, quot.x, 0),
                                       __shfl_sync(TT_FULL_MASK, quot.y, 0));
                tau_df = make_float2(__shfl_sync(TT_FULL_MASK, quot.x, 1),
                                     __shfl_sync(TT_FULL_MASK, quot.y, 1));
            }
            if (threadIdx.x == 0 && (p - k) % G == b) {
                const size_t o = (size_t)s * n + k;
                w.beta[o] = beta;
                w.scale[o] = scale_df;
                w.tau[o] = tau_df;
                w.perm[o] = cp;
            }
        }
        // column g_mine's scalars: a -= tau v (v . a), v . a = a[k] + scale
        // (x[k+1:] . a[k+1:]); its partial norm for step k + 1
        const int j = j0 + (t0 + g_mine) * G;
        const bool on = c_mine >= 0 && j != p;
        float2 ntws = make_float2(0.f, 0.f), n2;
        {
            float2 xa = s_dot[buf][g_mine][0];
#pragma unroll
            for (int u = 1; u < kW; u++)
                xa = df_add(xa, s_dot[buf][g_mine][u]);
            if (!zero) {
                const float2 vc = df_add(k_mine, df_mul(scale_df, xa));
                const float2 ntw = df_neg(df_mul(tau_df, vc));
                ntws = df_mul(ntw, scale_df);
                k_mine = df_add(k_mine, ntw);
            }
            n2 = df_sub(n_mine, df_mul(k_mine, k_mine));
        }
        const bool rec = on && n2.x <= 1.5e-8f * o_mine;
        const unsigned rec_mask = __ballot_sync(TT_FULL_MASK, rec);
        const unsigned on_mask = __ballot_sync(TT_FULL_MASK, on);
        const int c_now = c_mine;
        const float2 k_now = k_mine;
        if (t0 + GB < cnt) { // the next group's column of this lane
            const int tn = t0 + GB + g_mine;
            c_mine = tn < cnt ? cm[j0 + tn * G] : -1;
            if (c_mine >= 0) {
                n_mine = nr[j0 + tn * G];
                k_mine = As[c_mine * ld + k];
                o_mine = og[c_mine];
            }
        }
#pragma unroll
        for (int g = 0; g < GB; g++) {
            const int cj = __shfl_sync(TT_FULL_MASK, c_now, g);
            const float2 f = make_float2(__shfl_sync(TT_FULL_MASK, ntws.x, g),
                                         __shfl_sync(TT_FULL_MASK, ntws.y, g));
            if (on_mask >> g & 1) { // uniform
                const bool again = rec_mask >> g & 1;
                if (!zero) {
                    float2 *c = below(cj);
#pragma unroll
                    for (int u = 0; u < K; u++)
                        if (u < keff)
                            c[u * T] = df_fma(f, xv[u], slot[(g * K + u) * T]);
                }
                if (again) { // rare: the norm of the new column below row k
                    DfDot dr[2];
#pragma unroll
                    for (int u = 0; u < K; u++)
                        if (u < keff) { // as this thread wrote it
                            const float2 a = zero ? slot[(g * K + u) * T] : below(cj)[u * T];
                            df_dot_add(dr[u & 1], a, a);
                        }
                    const float2 r = qr_block_sum<T>(
                        df_add(df_dot_end(dr[0]), df_dot_end(dr[1])), s_red[rb]);
                    rb ^= 1;
                    if (g == g_mine)
                        n2 = r;
                    if (threadIdx.x == 0)
                        og[cj] = r.x;
                }
            }
            if (t0 + GB < cnt) {
                const int c = __shfl_sync(TT_FULL_MASK, c_mine, g);
                if (c >= 0)
                    issue(g, c);
            }
        }
        if (on && threadIdx.x < GB) {
            if (!zero)
                As[c_now * ld + k] = k_now;
            const int dest = j == k ? p : j;
            w.norms[nxt * n + dest] = n2;
            w.cmap[nxt * n + dest] = c_now;
        }
    }
}

// ---- one-sided Jacobi on X = R^T (float) ----------------------------------

// Directions of R whose norm is below kNullRel |R[0, 0]| (|R[0, 0]| is the
// largest column norm of the aligned matrix) are below the double precision
// of the input: they take no rotations and no part in U, as the oracle
// treats exactly-zero directions.
constexpr float kNullRel = 1e-15f;

// X[i + j n] = R[j, i] (upper triangle of the QR result), V = I, and the
// null-direction bound tiny[s] = (kNullRel R[0, 0])^2.
// grid (ceil(n * n / 256), n_sino).
__global__ void nos_rt_kernel(const float2 *__restrict__ A, const NosDesc *__restrict__ desc,
                              int n, NosWork w) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nn = (long long)n * n;
    if (e >= nn)
        return;
    const int s = blockIdx.y, i = (int)(e % n), j = (int)(e / n);
    const NosDesc d = desc[s];
    const float2 *beta = w.beta + (size_t)s * n;
    if (e == 0) {
        const float r = kNullRel * (beta[0].x + beta[0].y);
        w.tiny[s] = r * r;
    }
    // R[j, i]: the diagonal from beta, above it the stored column of position i
    float r = 0.f;
    if (j == i)
        r = beta[i].x + beta[i].y;
    else if (j < i) {
        const float2 a = A[d.a_off + j + (size_t)w.perm[(size_t)s * n + i] * d.ld];
        r = a.x + a.y;
    }
    w.X[s * nn + e] = r;
    w.V[s * nn + e] = i == j ? 1.f : 0.f;
}

// A pair is rotated when |x_p . x_q| > kJacTol |x_p| |x_q| -- a few times the
// rounding of a float dot product over n terms split across a warp -- and a
// sweep that rotates none (or whose largest rotated pair is below
// kJacDone) ends the iteration.  Near convergence the cyclic method is
// quadratic (measured at 1449 x 360: 7.6e-4, 2.1e-5, then 1.0e-6, the float
// floor), so a sweep whose largest rotated cosine is below 1e-4 leaves every
// pair at that floor and the next sweep would only confirm it.
constexpr float kJacTol = 1e-6f, kJacDone = 1e-4f;

// Two-level (block) Jacobi.  The n columns form blocks of kBJ, and a sweep
// visits every column pair once, in nbp - 1 launches (rounds of a
// round-robin tournament of the nbp blocks, a dummy block making nbp even):
// in each round a CTA copies its block pair -- 2 kBJ columns of X -- into
// shared memory and rotates the kBJ^2 pairs across the two blocks in kBJ
// inner rounds of kBJ disjoint pairs (one warp per pair, __syncthreads
// between inner rounds); the first round of a sweep first rotates the pairs
// inside each of its two blocks (kBJ - 1 more inner rounds).  A block-cyclic
// ordering of the cyclic Jacobi method.
//
// V does not take part in the rounds: a round's rotations are accumulated into
// one 2 kBJ x 2 kBJ orthogonal J per block pair (in shared memory), which
// goes to global memory, and a whole sweep of them is applied to V by another
// kernel (jacobi_v_kernel) beside the next sweep's rounds.  Columns sit in shared memory zero-padded to a
// multiple of 128 rows, so a lane moves 4 consecutive rows per 128-bit
// access and no row needs a bounds test.  Blocks of 12 (measured at 8
// sinograms of 1449 x 360 and 5795 x 720: 11 % and 29 % faster sweeps than
// blocks of 16, whose inner rounds are longer; blocks of 8 took one sweep
// more) give a round of 8 x 360-angle sinograms 120 CTAs.
constexpr int kBJ = 12, kBCols = 2 * kBJ, kBThreads = 32 * kBJ;
static_assert(kBJ % 2 == 0 && kBCols <= 32, "whole pairs per block; a J row per lane");

__device__ __forceinline__ void round_robin(int players, int round, int k, int &p, int &q) {
    const int P1 = players - 1;
    if (k == 0) {
        p = P1;
        q = round;
    } else {
        p = (round + k) % P1;
        q = (round - k + P1) % P1;
    }
    if (p > q) {
        const int t = p;
        p = q;
        q = t;
    }
}

// Dynamic shared memory of the round kernel with K4 slots of 128 rows
// (floats): the X block and J.
__host__ __device__ constexpr size_t block_round_smem_floats(int k4) {
    return (size_t)kBCols * 128 * k4 + kBCols * (kBCols + 1);
}

// Floats of a block pair's J, row-major; a sweep holds one per round and pair.
constexpr int kBJFloats = kBCols * kBCols;

__device__ __forceinline__ float4 f4_lin(float a, float4 x, float b, float4 y) {
    return make_float4(a * x.x + b * y.x, a * x.y + b * y.y, a * x.z + b * y.z, a * x.w + b * y.w);
}

// 4-byte asynchronous global -> shared copy; src_bytes 0 writes a zero
// without reading src.
__device__ __forceinline__ void cp_async4(float *dst, const float *src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src),
                 "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// 16-byte asynchronous copy of src_bytes (0 or 16) bytes, zero-filling the rest.
__device__ __forceinline__ void cp_async16(float *dst, const float *src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
                 "r"(src_bytes)
                 : "memory");
}

// Rows [r0, r0 + rows) of the 2 kBJ columns of the block (global column
// gcol(c), none past n) into a shared column-major block with leading
// dimension ld, zero-filled past n, as asynchronous copies: warp w takes
// local columns w and w + kBJ, its lanes consecutive rows -- 16 bytes at a
// time when n is a multiple of 4 (every column then starts 16-byte
// aligned, given a 16-byte aligned matrix), else 4.  rows and r0 are
// multiples of 4.
template <typename G>
__device__ __forceinline__ void stage_cols_async(float *dst, int ld, const float *src, int n,
                                                 int r0, int rows, G gcol) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool vec = (n & 3) == 0 && ((uintptr_t)src & 15) == 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = warp + kBJ * h, gc = gcol(c);
        float *d = dst + (size_t)c * ld;
        const float *g = src + (size_t)(gc < n ? gc : 0) * n;
        if (vec) {
            for (int q = lane; q < rows / 4; q += 32) {
                const int r = r0 + 4 * q;
                const bool ok = gc < n && r < n;
                cp_async16(d + 4 * q, ok ? g + r : src, ok ? 16 : 0);
            }
        } else {
            for (int q = lane; q < rows; q += 32) {
                const int r = r0 + q;
                const bool ok = gc < n && r < n;
                cp_async4(d + q, ok ? g + r : src, ok ? 4 : 0);
            }
        }
    }
}

// The inverse of stage_cols_async (plain stores, none past n).
template <typename G>
__device__ __forceinline__ void store_cols(float *dst, const float *sm, int ld, int n, int r0,
                                           int rows, G gcol) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool vec = (n & 3) == 0 && ((uintptr_t)dst & 15) == 0;
    const int lim = min(rows, n - r0); // rows of the block inside the matrix
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = warp + kBJ * h, gc = gcol(c);
        if (gc >= n)
            continue;
        const float *l = sm + (size_t)c * ld;
        float *g = dst + (size_t)gc * n + r0;
        if (vec) {
            for (int q = lane; 4 * q < lim; q += 32)
                *reinterpret_cast<float4 *>(g + 4 * q) = *reinterpret_cast<const float4 *>(l + 4 * q);
        } else {
            for (int q = lane; q < lim; q += 32)
                g[q] = l[q];
        }
    }
}

// One Jacobi rotation of the column pair (x, y) held by a warp (lane l
// holds rows 4 l + 128 u .. + 3): cos of the pair = |x . y| / (|x| |y|);
// rotated (x and y replaced) unless a column is null (norm^2 <= tn, or a zero
// column past n) or the pair is already orthogonal to kJacTol.  The
// rotation parameters come from the (2-ulp) hardware reciprocal square root:
// the rotation only has to be orthogonal (c^2 + s^2 = 1 to float precision),
// not exact.  Returns the pair's cos when rotated, else 0.
template <int K4>
__device__ __forceinline__ float jacobi_pair(float4 (&x)[K4], float4 (&y)[K4], float tn,
                                             float &c, float &sn) {
    float al = 0.f, be = 0.f, ga = 0.f;
#pragma unroll
    for (int u = 0; u < K4; u++) {
        al = fmaf(x[u].x, x[u].x, al);
        be = fmaf(y[u].x, y[u].x, be);
        ga = fmaf(x[u].x, y[u].x, ga);
        al = fmaf(x[u].y, x[u].y, al);
        be = fmaf(y[u].y, y[u].y, be);
        ga = fmaf(x[u].y, y[u].y, ga);
        al = fmaf(x[u].z, x[u].z, al);
        be = fmaf(y[u].z, y[u].z, be);
        ga = fmaf(x[u].z, y[u].z, ga);
        al = fmaf(x[u].w, x[u].w, al);
        be = fmaf(y[u].w, y[u].w, be);
        ga = fmaf(x[u].w, y[u].w, ga);
    }
    al = warp_sum(al);
    be = warp_sum(be);
    ga = warp_sum(ga);
    const float cosv = fabsf(ga) * (rsqrtf(al) * rsqrtf(be));
    if (!(al > tn && be > tn && ga != 0.f && cosv > kJacTol))
        return 0.f; // uniform across the warp
    const float zeta = __fdividef(be - al, 2.f * ga);
    const float az = fabsf(zeta);
    float t;
    if (az < 1e15f) {
        const float z2 = fmaf(zeta, zeta, 1.f);
        t = __fdividef(1.f, az + z2 * rsqrtf(z2));
    } else {
        t = __fdividef(0.5f, az);
    }
    t = zeta >= 0.f ? t : -t;
    c = rsqrtf(fmaf(t, t, 1.f));
    sn = c * t;
#pragma unroll
    for (int u = 0; u < K4; u++) {
        const float4 xo = x[u];
        x[u] = f4_lin(c, xo, -sn, y[u]);
        y[u] = f4_lin(sn, xo, c, y[u]);
    }
    return cosv;
}

// grid (nbp / 2, n_sino), kBThreads threads, dynamic shared memory
// block_round_smem_floats(K4) floats, 128 K4 >= n: lane l holds rows
// 4 l + 128 u .. + 3 (u < K4) of a column.
template <int K4>
__global__ void __launch_bounds__(kBThreads)
rt_block_round_kernel(float *__restrict__ X, float *__restrict__ J, int n, int nbp, int round,
                      unsigned *__restrict__ off_bits, const float *__restrict__ tiny,
                      const unsigned *__restrict__ state) {
    extern __shared__ __align__(16) float bsm[];
    constexpr int NP = 128 * K4; // padded rows
    float *Xl = bsm;             // kBCols x NP
    float(*Jt)[kBCols + 1] = reinterpret_cast<float(*)[kBCols + 1]>(Xl + (size_t)kBCols * NP);
    const int s = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = (n + kBJ - 1) / kBJ;
    int bp, bq;
    round_robin(nbp, round, blockIdx.x, bp, bq);
    const bool intra = round == 0; // the sweep's first round also rotates within blocks
    if (bq >= nb && !intra)
        return; // the bye (the dummy block's columns are zeros and never rotate)
    const size_t nn = (size_t)n * n;
    float *Xg = X + s * nn;
    // global column of local column c
    auto gcol = [&](int c) { return c < kBJ ? bp * kBJ + c : bq * kBJ + c - kBJ; };
    // X block (zero-padded to NP rows); J = I
    stage_cols_async(Xl, NP, Xg, n, 0, NP, gcol);
    cp_async_commit();
    for (int e = threadIdx.x; e < kBCols * kBCols; e += kBThreads)
        Jt[e / kBCols][e % kBCols] = e / kBCols == e % kBCols ? 1.f : 0.f;
    const unsigned parity = state[1] & 1; // of the sweep: which half of J
    cp_async_wait<0>();
    __syncthreads();
    const float tn = tiny[s];
    float wmax = 0.f;
    // J <- J G on columns p, q (row `lane` of each)
    auto j_rotate = [&](int p, int q, float c, float sn) {
        if (kBCols < 32 && lane >= kBCols)
            return;
        const float a = Jt[p][lane], b = Jt[q][lane];
        Jt[p][lane] = c * a - sn * b;
        Jt[q][lane] = sn * a + c * b;
    };
    float4 x[K4], y[K4];
    if (intra) {
        // pairs within each block: warps 0 .. kBJ / 2 - 1 block bp, the rest block bq
        const int half = warp / (kBJ / 2);
        for (int ir = 0; ir < kBJ - 1; ir++) {
            int p, q;
            round_robin(kBJ, ir, warp % (kBJ / 2), p, q);
            p += half * kBJ;
            q += half * kBJ;
            float4 *xp = reinterpret_cast<float4 *>(Xl + (size_t)p * NP);
            float4 *xq = reinterpret_cast<float4 *>(Xl + (size_t)q * NP);
#pragma unroll
            for (int u = 0; u < K4; u++) {
                x[u] = xp[lane + 32 * u];
                y[u] = xq[lane + 32 * u];
            }
            float c, sn;
            const float cosv = jacobi_pair<K4>(x, y, tn, c, sn);
            if (cosv > 0.f) {
                wmax = fmaxf(wmax, cosv);
#pragma unroll
                for (int u = 0; u < K4; u++) {
                    xp[lane + 32 * u] = x[u];
                    xq[lane + 32 * u] = y[u];
                }
                j_rotate(p, q, c, sn);
            }
            __syncthreads();
        }
    }
    // pairs across the blocks: in inner round r warp w pairs column w of bp
    // (kept in registers throughout) with column (w + r) % kBJ of bq
    float4 *xw = reinterpret_cast<float4 *>(Xl + (size_t)warp * NP);
#pragma unroll
    for (int u = 0; u < K4; u++)
        x[u] = xw[lane + 32 * u];
    for (int r = 0; r < kBJ; r++) {
        const int q = kBJ + (warp + r) % kBJ;
        float4 *xq = reinterpret_cast<float4 *>(Xl + (size_t)q * NP);
#pragma unroll
        for (int u = 0; u < K4; u++)
            y[u] = xq[lane + 32 * u];
        float c, sn;
        const float cosv = jacobi_pair<K4>(x, y, tn, c, sn);
        if (cosv > 0.f) {
            wmax = fmaxf(wmax, cosv);
#pragma unroll
            for (int u = 0; u < K4; u++)
                xq[lane + 32 * u] = y[u];
            j_rotate(warp, q, c, sn);
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < K4; u++)
        xw[lane + 32 * u] = x[u];
    __syncthreads();
    if (lane == 0 && wmax > 0.f)
        atomicMax(off_bits + s, __float_as_uint(wmax));
    // X block back
    store_cols(Xg, Xl, NP, n, 0, NP, gcol);
    const size_t pair =
        (((size_t)parity * gridDim.y + s) * (nbp - 1) + round) * (nbp / 2) + blockIdx.x;
    float *Jg = J + pair * kBJFloats;
    for (int e = threadIdx.x; e < kBJFloats; e += kBThreads)
        Jg[e] = Jt[e % kBCols][e / kBCols];
}

// V <- V J_0 J_1 ... : the last finished sweep's rotations, round by round, applied
// to the rows of V, which are independent: a warp keeps 4 rows (all columns, in
// shared memory) for the whole sweep.  Per round a lane takes tiles of 4 rows x
// 4 columns of a block pair, 24 steps of two 16-byte loads and 16
// multiply-adds; the CTA's warps share the J's, staged 16 pairs (3 tiles
// per lane) ahead.  Runs beside the next sweep's rounds, which are chains that leave
// most of the machine idle.  Against V rotated inside the rounds the orthonormal
// circus gained 0.6 ms of 5.6 at 4 x 450 x 360, 0.25 of 8.0 at 8 x 1449 x 360 and 0.6
// of 77 at 8 x 5795 x 720 (with a QR that summed in another order).  Keeping the
// rounds' CTAs off its SMs (one CTA with all the shared memory on each SM they
// leave) took 0.06 ms longer at 8 x 1449 x 360.
// grid (ceil(n / (4 warps)), n_sino).
constexpr int kVMaxWarps = 8, kVPairs = 16, kVPairLd = kBJFloats + 24; // pairs 24 banks apart
constexpr int kVTiles = kVPairs * (kBCols / 4) / 32;
static_assert(kVTiles * 32 == kVPairs * (kBCols / 4), "whole tiles per lane");
constexpr size_t jacobi_v_smem(int nbp, int warps) {
    return sizeof(float) * ((size_t)2 * kVPairs * kVPairLd + (size_t)warps * 4 * kBJ * nbp);
}
__global__ void __launch_bounds__(32 * kVMaxWarps)
jacobi_v_kernel(float *__restrict__ V, const float *__restrict__ J, int n, int nbp,
                const unsigned *__restrict__ state) {
    extern __shared__ __align__(16) float vsm[];
    const unsigned done = state[1];
    if (done == 0)
        return; // no sweep yet: V = I
    const int s = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rounds = nbp - 1, pairs = nbp / 2, chunks = (pairs + kVPairs - 1) / kVPairs;
    const int nb = (n + kBJ - 1) / kBJ, total = rounds * chunks;
    const float *Jg = J + ((size_t)((done - 1) & 1) * gridDim.y + s) * rounds * pairs * kBJFloats;
    // chunk c of the sweep: pairs p0 .. of one round, into buffer c & 1
    auto stage = [&](int c) {
        const int round = c / chunks, p0 = (c - round * chunks) * kVPairs;
        const int count = min(kVPairs, pairs - p0);
        const float *src = Jg + ((size_t)round * pairs + p0) * kBJFloats;
        float *dst = vsm + (c & 1) * kVPairs * kVPairLd;
        for (int e = threadIdx.x; e < count * (kBJFloats / 4); e += blockDim.x) {
            const int p = e / (kBJFloats / 4), q = e - p * (kBJFloats / 4);
            cp_async16(dst + p * kVPairLd + 4 * q, src + 4 * (size_t)e, 16);
        }
        cp_async_commit();
    };
    stage(0);
    float4 *vr = reinterpret_cast<float4 *>(vsm + 2 * kVPairs * kVPairLd) + (size_t)warp * kBJ * nbp;
    const int row = (blockIdx.x * (blockDim.x >> 5) + warp) * 4;
    float *Vg = V + (size_t)s * n * n;
    for (int c = lane; c < kBJ * nbp; c += 32) {
        const float *g = Vg + (size_t)c * n + row;
        vr[c] = make_float4(c < n && row < n ? g[0] : 0.f, c < n && row + 1 < n ? g[1] : 0.f,
                            c < n && row + 2 < n ? g[2] : 0.f, c < n && row + 3 < n ? g[3] : 0.f);
    }
    for (int c = 0; c < total; c++) {
        cp_async_wait<0>();
        __syncthreads(); // chunk c is in place, chunk c - 1 is read
        if (c + 1 < total)
            stage(c + 1);
        const int round = c / chunks, p0 = (c - round * chunks) * kVPairs;
        const float *Jc = vsm + (c & 1) * kVPairs * kVPairLd;
        float4 acc[kVTiles][4]; // by column
        int first[kVTiles];     // the tile's first column, -1: none
#pragma unroll
        for (int u = 0; u < kVTiles; u++) {
            const int tile = lane + 32 * u, p = tile / (kBCols / 4), cg = 4 * (tile % (kBCols / 4));
            int bp, bq;
            round_robin(nbp, round, min(p0 + p, pairs - 1), bp, bq);
            // the bye (a sweep's first round also rotates within its block)
            const bool on = p0 + p < pairs && (bq < nb || round == 0);
            first[u] = !on ? -1 : cg < kBJ ? bp * kBJ + cg : bq * kBJ + cg - kBJ;
            if (!on)
                continue;
            const float4 *vp = vr + bp * kBJ, *vq = vr + bq * kBJ - kBJ;
            const float *j = Jc + p * kVPairLd + cg;
#pragma unroll
            for (int v = 0; v < 4; v++)
                acc[u][v] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kBCols; i++) {
                const float4 x = i < kBJ ? vp[i] : vq[i];
                const float4 jr = *reinterpret_cast<const float4 *>(j + i * kBCols);
                const float jv[4] = {jr.x, jr.y, jr.z, jr.w};
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    acc[u][v].x = fmaf(x.x, jv[v], acc[u][v].x);
                    acc[u][v].y = fmaf(x.y, jv[v], acc[u][v].y);
                    acc[u][v].z = fmaf(x.z, jv[v], acc[u][v].z);
                    acc[u][v].w = fmaf(x.w, jv[v], acc[u][v].w);
                }
            }
        }
        __syncwarp(); // the rows are read
#pragma unroll
        for (int u = 0; u < kVTiles; u++)
            if (first[u] >= 0)
#pragma unroll
                for (int v = 0; v < 4; v++)
                    vr[first[u] + v] = acc[u][v];
        __syncwarp();
    }
    for (int c = lane; c < n; c += 32) {
        float *g = Vg + (size_t)c * n + row;
        const float4 x = vr[c];
        const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int v = 0; v < 4; v++)
            if (row + v < n)
                g[v] = xv[v];
    }
}

// ---- assembly ---------------------------------------------------------------

// 1 / |x_k| per column of the converged X (0 for a null direction).  grid
// (ceil(n / 4), n_sino), one warp per column.
__global__ void rt_invnorm_kernel(const float *__restrict__ X, int n, const float *__restrict__ tiny,
                                  float *__restrict__ inv) {
    const int k = blockIdx.x * 4 + (threadIdx.x >> 5), s = blockIdx.y, lane = threadIdx.x & 31;
    if (k >= n)
        return;
    const float *x = X + (size_t)s * n * n + (size_t)k * n;
    float v = 0.f;
    for (int i = lane; i < n; i += 32)
        v = fmaf(x[i], x[i], v);
    v = warp_sum(v);
    if (lane == 0)
        inv[(size_t)s * n + k] = v > tiny[s] ? rsqrtf(v) : 0.f;
}

// X[:, k] *= inv[k]: the columns of X become U_X.  grid (ceil(n n / 256), n_sino).
__global__ void rt_scale_kernel(float *__restrict__ X, const float *__restrict__ inv, int n) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nn = (long long)n * n;
    if (e < nn)
        X[blockIdx.y * nn + e] *= inv[(size_t)blockIdx.y * n + (int)(e / n)];
}

// C = alpha op(A) op(B) + beta D for n x n column-major float matrices per
// sinogram, op given by strides: op(A)(i, k) = A[i ai + k ak], op(B)(k, j) =
// B[k bk + j bj], one stride of each pair being 1 (the tile's loads run along
// it).  64 x 64 output tiles, 4 x 4 per thread from two 16-byte loads per k,
// k in steps of 16 with the next step's elements fetched meanwhile.  Three
// products at 8 x 360^3: 96 us, from 307 (32 x 32 tiles, 4 outputs and five
// loads per k and thread); sums in the same order.  grid (ceil(n / 64),
// ceil(n / 64), n_sino).
constexpr int kGemmTile = 64, kGemmStep = 16, kGemmLd = kGemmTile + 4;
__global__ void __launch_bounds__(256)
rt_gemm_kernel(const float *__restrict__ A, int ai, int ak, const float *__restrict__ B, int bk,
               int bj, const float *__restrict__ D, float alpha, float beta, int n,
               float *__restrict__ C) {
    __shared__ __align__(16) float as[kGemmStep][kGemmLd], bs[kGemmStep][kGemmLd];
    const int i0 = blockIdx.x * kGemmTile, j0 = blockIdx.y * kGemmTile;
    const int ti = 4 * (threadIdx.x & 15), tj = 4 * (threadIdx.x >> 4);
    const size_t off = (size_t)blockIdx.z * n * n;
    A += off;
    B += off;
    C += off;
    // this thread's four elements of a step: (row of the tile, k) of each operand
    constexpr int kPer = kGemmTile * kGemmStep / 256;
    auto place = [](bool along_k, int q, int &r, int &kk) {
        const int e = threadIdx.x + 256 * q;
        r = along_k ? e / kGemmStep : e % kGemmTile;
        kk = along_k ? e % kGemmStep : e / kGemmTile;
    };
    float an[kPer], bn[kPer];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            int r, kk;
            place(ak == 1, q, r, kk);
            an[q] = k0 + kk < n && i0 + r < n ? A[(size_t)(i0 + r) * ai + (size_t)(k0 + kk) * ak]
                                              : 0.f;
            place(bk == 1, q, r, kk);
            bn[q] = k0 + kk < n && j0 + r < n ? B[(size_t)(k0 + kk) * bk + (size_t)(j0 + r) * bj]
                                              : 0.f;
        }
    };
    float acc[4][4] = {};
    fetch(0);
    for (int k0 = 0; k0 < n; k0 += kGemmStep) {
        __syncthreads(); // the last step's tiles are read
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            int r, kk;
            place(ak == 1, q, r, kk);
            as[kk][r] = an[q];
            place(bk == 1, q, r, kk);
            bs[kk][r] = bn[q];
        }
        __syncthreads();
        if (k0 + kGemmStep < n)
            fetch(k0 + kGemmStep);
#pragma unroll
        for (int kk = 0; kk < kGemmStep; kk++) {
            const float4 a = *reinterpret_cast<const float4 *>(&as[kk][ti]);
            const float4 b = *reinterpret_cast<const float4 *>(&bs[kk][tj]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int v = 0; v < 4; v++)
                    acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
        }
    }
#pragma unroll
    for (int v = 0; v < 4; v++)
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + ti + u, j = j0 + tj + v;
            if (i < n && j < n) {
                const size_t e = i + (size_t)j * n;
                C[e] = beta != 0.f ? alpha * acc[u][v] + beta * D[off + e] : alpha * acc[u][v];
            }
        }
}

// Y = Q [P; 0] = H_0 H_1 ... H_{n-1} [P; 0], out[:, perm[j]] = Y[:, j]:
// one reflector at a time with Y in registers while the aligned columns fit
// (m <= 16 kQThreads), by blocks of reflectors above.
constexpr int kQThreads = 256, kQCols = 4; // columns of Y per CTA
constexpr int kNosMaxCols = 1024;              // angles the orthonormal circus takes

// The reflectors as floats, in their order: refl[s][k][i] = 1 at i = k, the scaled
// pivot column below it, 0 above and in the rows past m, reflector stride ldv (a
// multiple of kQThreads).  grid (n, n_sino).
__global__ void __launch_bounds__(kQThreads)
nos_refl_kernel(const float2 *__restrict__ A, const NosDesc *__restrict__ desc,
                const float2 *__restrict__ scale, const int *__restrict__ perm, int n, int ldv,
                float *__restrict__ refl) {
    const int k = blockIdx.x, s = blockIdx.y;
    const NosDesc d = desc[s];
    const float2 sc = scale[(size_t)s * n + k];
    const float vs = sc.x + sc.y;
    const float2 *x = A + d.a_off + (size_t)perm[(size_t)s * n + k] * d.ld;
    float *v = refl + ((size_t)s * n + k) * ldv;
    for (int i = threadIdx.x; i < ldv; i += kQThreads) {
        float vi = i == k ? 1.f : 0.f;
        if (i > k && i < d.m) {
            const float2 xi = x[i];
            vi = (xi.x + xi.y) * vs;
        }
        v[i] = vi;
    }
}

// The product with Y held in registers, for m <= K kQThreads: thread t
// owns rows t + kQThreads u (u < K) of the kQCols columns, so applying a
// reflector needs one block reduction (double-buffered: one barrier) and no
// other exchange; the next reflector is loaded while the current one is applied.
// Bound by its instructions: the reflectors are formed once, not by every
// CTA, and the four columns' warp sums share their first two levels.  8 x 1843 x
// 360: 463 us, from 723; the same sums.
template <int K>
__global__ void __launch_bounds__(kQThreads, K == 8 ? 3 : 1) // 3 CTAs per SM fit K = 8 unspilled
nos_apply_q_reg_kernel(const float *__restrict__ refl, int ldv,
                       const NosDesc *__restrict__ desc, const float2 *__restrict__ tau,
                       const int *__restrict__ perm, const float *__restrict__ P, int n,
                       float *__restrict__ out) {
    static_assert(kQCols == 4, "the halving exchanges below");
    __shared__ float s_t[kNosMaxCols];
    __shared__ __align__(16) float red[2][kQThreads / 32][kQCols];
    const int s = blockIdx.y, j0 = blockIdx.x * kQCols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const NosDesc d = desc[s];
    const int m = d.m, nc = min(kQCols, n - j0);
    const int nu = (m + kQThreads - 1) / kQThreads; // row slots in use
    const size_t nn = (size_t)n * n;
    for (int k = threadIdx.x; k < n; k += kQThreads) {
        const float2 t = tau[(size_t)s * n + k];
        s_t[k] = t.x + t.y;
    }
    float y[kQCols][K];
#pragma unroll
    for (int u = 0; u < K; u++) {
        const int i = threadIdx.x + kQThreads * u;
#pragma unroll
        for (int c = 0; c < kQCols; c++)
            y[c][u] = (c < nc && i < n) ? P[s * nn + i + (size_t)(j0 + c) * n] : 0.f;
    }
    __syncthreads(); // scalars in place
    const float *vp = refl + ((size_t)s * n + n - 1) * ldv + threadIdx.x;
    float v[K], vn[K];
#pragma unroll
    for (int u = 0; u < K; u++)
        v[u] = vn[u] = u < nu ? vp[kQThreads * u] : 0.f;
    int rb = 0;
    for (int k = n - 1; k >= 0; k--) {
        vp -= ldv;
        if (k > 0)
#pragma unroll
            for (int u = 0; u < K; u++)
                if (u < nu)
                    vn[u] = vp[kQThreads * u];
        const float t = s_t[k];
        if (t != 0.f) { // uniform
            float w[kQCols];
#pragma unroll
            for (int c = 0; c < kQCols; c++) {
                w[c] = 0.f;
#pragma unroll
                for (int u = 0; u < K; u++)
                    w[c] = fmaf(v[u], y[c][u], w[c]);
            }
            // lane 8 c ends with the warp's sum of column c
            {
                const bool up = lane & 16;
                const float g0 = up ? w[0] : w[2], g1 = up ? w[1] : w[3];
                float a0 = (up ? w[2] : w[0]) + __shfl_xor_sync(TT_FULL_MASK, g0, 16);
                const float a1 = (up ? w[3] : w[1]) + __shfl_xor_sync(TT_FULL_MASK, g1, 16);
                const bool odd = lane & 8;
                const float g = odd ? a0 : a1;
                a0 = (odd ? a1 : a0) + __shfl_xor_sync(TT_FULL_MASK, g, 8);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
                    a0 += __shfl_xor_sync(TT_FULL_MASK, a0, o);
                if ((lane & 7) == 0)
                    red[rb][warp][lane >> 3] = a0;
            }
            __syncthreads();
            float4 tot = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < kQThreads / 32; q++) {
                const float4 r = *reinterpret_cast<const float4 *>(red[rb][q]);
                tot.x += r.x;
                tot.y += r.y;
                tot.z += r.z;
                tot.w += r.w;
            }
            w[0] = t * tot.x;
            w[1] = t * tot.y;
            w[2] = t * tot.z;
            w[3] = t * tot.w;
            rb ^= 1;
#pragma unroll
            for (int u = 0; u < K; u++)
#pragma unroll
                for (int c = 0; c < kQCols; c++)
                    y[c][u] = fmaf(-w[c], v[u], y[c][u]);
        }
#pragma unroll
        for (int u = 0; u < K; u++)
            v[u] = vn[u];
    }
    for (int c = 0; c < nc; c++) {
        float *o = out + d.out_off + (size_t)perm[(size_t)s * n + j0 + c] * m;
#pragma unroll
        for (int u = 0; u < K; u++) {
            const int i = threadIdx.x + kQThreads * u;
            if (i < m)
                o[i] = y[c][u];
        }
    }
}

// Y = Q [P; 0] = H_0 H_1 ... H_{n-1} [P; 0] by blocks of kWyB reflectors in
// compact WY form (the LAPACK larft / larfb scheme): the product of reflectors
// k0 .. k0 + b - 1 is I - V T V^T with V = [v_k0 .. v_k0+b-1] (v_k: 1 at row
// k, the scaled stored pivot column below it, 0 above) and T upper
// triangular, T[i, i] = tau_i, T[0:i, i] = -tau_i T[0:i, 0:i] V[:, 0:i]^T v_i.
// The blocks apply last to first, each as Y <- Y - V (T (V^T Y)) over rows
// k0.. (V is zero above): V^T Y by row chunks into partial sums, T times
// their sum, then the rank-b update -- float GEMM tiles instead of one
// latency-bound pass over Y per reflector.  Y lives in the output: its
// column j is out[:, perm[j]].
constexpr int kWyB = 32;          // reflectors per block
constexpr int kWyThreads = 256;   // threads of every WY kernel
constexpr int kWyCols = 128;      // columns of Y per CTA of the GEMM passes
constexpr int kWyVLd = 36;        // V tile row stride (float4 rows, conflict-free fill)
constexpr int kWyYLd = 132;       // Y / W tile row stride
constexpr int kWyGramRows = 128;  // rows per pass of the T kernel

// out[:, perm[j]] = [P[:, j]; 0].  grid (n, n_sino).
__global__ void __launch_bounds__(kWyThreads)
wy_init_kernel(const float *__restrict__ P, const NosDesc *__restrict__ desc,
               const int *__restrict__ perm, int n, float *__restrict__ out) {
    const int j = blockIdx.x, s = blockIdx.y;
    const NosDesc d = desc[s];
    float *o = out + d.out_off + (size_t)perm[(size_t)s * n + j] * d.m;
    const float *p = P + (size_t)s * n * n + (size_t)j * n;
    for (int i = threadIdx.x; i < d.m; i += kWyThreads)
        o[i] = i < n ? p[i] : 0.f;
}

// Per-block reflector data in shared memory: stored column, float scale and
// tau (0 past n, which makes those columns of V and T zero).
struct WyRefl {
    int pm[kWyB];
    float vs[kWyB], t[kWyB];
};
__device__ __forceinline__ void wy_load_refl(WyRefl &R, const float2 *tau, const float2 *scale,
                                             const int *perm, int n, int s, int k0) {
    if (threadIdx.x < kWyB) {
        const int k = k0 + threadIdx.x;
        const bool ok = k < n;
        const size_t o = (size_t)s * n + k;
        R.pm[threadIdx.x] = ok ? perm[o] : 0;
        R.vs[threadIdx.x] = ok ? scale[o].x + scale[o].y : 0.f;
        R.t[threadIdx.x] = ok ? tau[o].x + tau[o].y : 0.f;
    }
}
// v_{k0 + r}[row] for a row inside the matrix (row < m).
__device__ __forceinline__ float wy_v(const float2 *As, int ld, const WyRefl &R, int n, int k0,
                                      int r, int row) {
    const int k = k0 + r;
    if (k >= n || row < k)
        return 0.f;
    if (row == k)
        return 1.f;
    const float2 x = As[(size_t)R.pm[r] * ld + row];
    return (x.x + x.y) * R.vs[r];
}

// T of every block: the Gram matrix G = V^T V over rows k0..m-1 (kWyGramRows
// rows of V staged per pass; thread t accumulates G[t / 32 + 8 q][t % 32]),
// then the recurrence on one warp.  grid (blocks, n_sino); T row-major,
// 32 x 32 per (sinogram, block).
__global__ void __launch_bounds__(kWyThreads)
wy_t_kernel(const float2 *__restrict__ A, const NosDesc *__restrict__ desc,
            const float2 *__restrict__ tau, const float2 *__restrict__ scale,
            const int *__restrict__ perm, int n, float *__restrict__ T) {
    __shared__ float Vs[kWyGramRows][kWyB + 1];
    __shared__ float Gs[kWyB][kWyB + 1];
    __shared__ float Ts[kWyB][kWyB + 1];
    __shared__ WyRefl R;
    const int jb = blockIdx.x, s = blockIdx.y, k0 = jb * kWyB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const NosDesc d = desc[s];
    const int m = d.m;
    const float2 *As = A + d.a_off;
    wy_load_refl(R, tau, scale, perm, n, s, k0);
    __syncthreads(); // R in place
    constexpr int kPer = kWyGramRows * kWyB / kWyThreads;
    float vr[kPer]; // the next pass, fetched while the current one is reduced
    auto fetch = [&](int row0) {
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            const int i = e % kWyGramRows, r = e / kWyGramRows, row = row0 + i;
            vr[q] = row < m ? wy_v(As, d.ld, R, n, k0, r, row) : 0.f;
        }
    };
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (k0 < m)
        fetch(k0);
    for (int row0 = k0; row0 < m; row0 += kWyGramRows) {
        __syncthreads(); // the previous pass is read
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            Vs[e % kWyGramRows][e / kWyGramRows] = vr[q];
        }
        __syncthreads();
        if (row0 + kWyGramRows < m)
            fetch(row0 + kWyGramRows);
#pragma unroll 4
        for (int i = 0; i < kWyGramRows; i++) {
            const float b = Vs[i][lane];
#pragma unroll
            for (int q = 0; q < 4; q++)
                acc[q] = fmaf(Vs[i][warp + 8 * q], b, acc[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
        Gs[warp + 8 * q][lane] = acc[q];
    __syncthreads();
    if (warp == 0) {
        for (int c = 0; c < kWyB; c++)
            Ts[lane][c] = 0.f;
        __syncwarp();
        for (int i = 0; i < kWyB; i++) {
            float v = 0.f;
            if (lane < i) {
                for (int c = lane; c < i; c++)
                    v = fmaf(Ts[lane][c], Gs[c][i], v);
                v *= -R.t[i];
            }
            __syncwarp();
            if (lane < i)
                Ts[lane][i] = v;
            else if (lane == i)
                Ts[i][i] = R.t[i];
            __syncwarp();
        }
        float *o = T + ((size_t)s * gridDim.x + jb) * kWyB * kWyB;
        for (int r = 0; r < kWyB; r++)
            o[r * kWyB + lane] = Ts[r][lane];
    }
}

// Column offsets of the CTA's kWyCols columns of Y in out (-1 past n).
__device__ __forceinline__ void wy_load_cols(long long *cols, const NosDesc &d, const int *perm,
                                             int n, int s, int j0) {
    if (threadIdx.x < kWyCols) {
        const int j = j0 + threadIdx.x;
        cols[threadIdx.x] = j < n ? d.out_off + (long long)perm[(size_t)s * n + j] * d.m : -1;
    }
}

// Partial W = V^T Y over rows [k0 + c R, k0 + (c + 1) R) of each sinogram
// (R = 32 ns rows; none past m): part[s][c][r][j], 32 x kWyCols per CTA,
// thread (warp, lane) owning reflectors 4 warp .. + 3 and columns 4 lane ..
// + 3.  Rows are staged 32 at a time; the fills map a warp to 8 rows x 4
// columns, which makes their shared-memory stores conflict-free.
// grid (ceil(n / kWyCols), nchunk, n_sino).
__global__ void __launch_bounds__(kWyThreads)
wy_vty_kernel(const float2 *__restrict__ A, const NosDesc *__restrict__ desc,
              const float2 *__restrict__ tau, const float2 *__restrict__ scale,
              const int *__restrict__ perm, int n, int k0, int ns,
              const float *__restrict__ out, float *__restrict__ part) {
    __shared__ __align__(16) float Vs[32 * kWyVLd];
    __shared__ __align__(16) float Ys[32 * kWyYLd];
    __shared__ long long cols[kWyCols];
    __shared__ WyRefl R;
    const int j0 = blockIdx.x * kWyCols, c = blockIdx.y, s = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const NosDesc d = desc[s];
    const int m = d.m;
    const float2 *As = A + d.a_off;
    const int rb = k0 + c * 32 * ns, re = min(rb + 32 * ns, m);
    wy_load_refl(R, tau, scale, perm, n, s, k0);
    wy_load_cols(cols, d, perm, n, s, j0);
    __syncthreads(); // R and cols in place
    constexpr int kPV = 32 * kWyB / kWyThreads, kPY = 32 * kWyCols / kWyThreads;
    float vr[kPV], yr[kPY]; // the next 32 rows, fetched during the current ones
    auto fetch = [&](int row0) {
#pragma unroll
        for (int q = 0; q < kPV; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            const int i = (e >> 8) * 8 + (e & 7), r = (e >> 3) & 31, row = row0 + i;
            vr[q] = row < re ? wy_v(As, d.ld, R, n, k0, r, row) : 0.f;
        }
#pragma unroll
        for (int q = 0; q < kPY; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            const int i = (e >> 10) * 8 + (e & 7), col = (e >> 3) & 127, row = row0 + i;
            const long long o = cols[col];
            yr[q] = o >= 0 && row < re ? out[o + row] : 0.f;
        }
    };
    float acc[4][4];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++)
            acc[u][v] = 0.f;
    if (rb < re)
        fetch(rb);
    for (int row0 = rb; row0 < re; row0 += 32) {
        __syncthreads(); // the previous tiles are read
#pragma unroll
        for (int q = 0; q < kPV; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            Vs[((e >> 8) * 8 + (e & 7)) * kWyVLd + ((e >> 3) & 31)] = vr[q];
        }
#pragma unroll
        for (int q = 0; q < kPY; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            Ys[((e >> 10) * 8 + (e & 7)) * kWyYLd + ((e >> 3) & 127)] = yr[q];
        }
        __syncthreads();
        if (row0 + 32 < re)
            fetch(row0 + 32);
#pragma unroll 8
        for (int i = 0; i < 32; i++) {
            const float4 a = *reinterpret_cast<const float4 *>(&Vs[i * kWyVLd + 4 * warp]);
            const float4 y = *reinterpret_cast<const float4 *>(&Ys[i * kWyYLd + 4 * lane]);
            const float av[4] = {a.x, a.y, a.z, a.w}, yv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int v = 0; v < 4; v++)
                    acc[u][v] = fmaf(av[u], yv[v], acc[u][v]);
        }
    }
    float *p = part + ((size_t)s * gridDim.y + c) * kWyB * n;
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const int j = j0 + 4 * lane + v;
            if (j < n)
                p[(size_t)(4 * warp + u) * n + j] = acc[u][v];
        }
}

// W2 = T (sum of the nchunk partials), 32 x n per sinogram.  grid
// (ceil(n / 32), n_sino).
__global__ void __launch_bounds__(kWyThreads)
wy_w2_kernel(const float *__restrict__ T, const float *__restrict__ part, int nchunk, int n,
             int jb, int nbk, float *__restrict__ W2) {
    __shared__ float Ws[kWyB][33];
    __shared__ float Tt[kWyB][kWyB + 1];
    const int j0 = blockIdx.x * 32, s = blockIdx.y;
    const float *Tb = T + ((size_t)s * nbk + jb) * kWyB * kWyB;
    for (int e = threadIdx.x; e < kWyB * 32; e += kWyThreads) {
        const int r = e >> 5, jj = e & 31, j = j0 + jj;
        // four independent sums, so that the chunks' loads overlap
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        if (j < n) {
            const float *q = part + ((size_t)s * nchunk * kWyB + r) * n + j;
            const size_t step = (size_t)kWyB * n;
            int c = 0;
#pragma unroll 2
            for (; c + 4 <= nchunk; c += 4)
#pragma unroll
                for (int h = 0; h < 4; h++)
                    s4[h] += q[(c + h) * step];
            for (; c < nchunk; c++)
                s4[0] += q[c * step];
        }
        Ws[r][jj] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
        Tt[r][jj] = Tb[r * kWyB + jj];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kWyB * 32; e += kWyThreads) {
        const int r = e >> 5, jj = e & 31, j = j0 + jj;
        float v = 0.f;
        for (int c = r; c < kWyB; c++)
            v = fmaf(Tt[r][c], Ws[c][jj], v);
        if (j < n)
            W2[((size_t)s * kWyB + r) * n + j] = v;
    }
}

// Y[rows, cols] -= V[rows, :] W2[:, cols] over rows [k0 + c R, .. + R)
// (none past m): W2's 32 x kWyCols tile staged once, V 32 rows at a time;
// lane = row, warp w = columns 16 w .. + 15, so each column's 32 rows are
// one coalesced read-modify-write.  grid (ceil(n / kWyCols), nchunk, n_sino).
__global__ void __launch_bounds__(kWyThreads)
wy_update_kernel(const float2 *__restrict__ A, const NosDesc *__restrict__ desc,
                 const float2 *__restrict__ tau, const float2 *__restrict__ scale,
                 const int *__restrict__ perm, int n, int k0, int ns,
                 const float *__restrict__ W2, float *__restrict__ out) {
    __shared__ __align__(16) float Ws[kWyB * kWyYLd];
    __shared__ float Vs[32 * 33];
    __shared__ long long cols[kWyCols];
    __shared__ WyRefl R;
    const int j0 = blockIdx.x * kWyCols, c = blockIdx.y, s = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const NosDesc d = desc[s];
    const int m = d.m;
    const int rb = k0 + c * 32 * ns, re = min(rb + 32 * ns, m);
    if (rb >= re)
        return; // uniform: no rows of this sinogram here
    const float2 *As = A + d.a_off;
    wy_load_refl(R, tau, scale, perm, n, s, k0);
    wy_load_cols(cols, d, perm, n, s, j0);
    for (int e = threadIdx.x; e < kWyB * kWyCols; e += kWyThreads) {
        const int r = e >> 7, q = e & 127, j = j0 + q;
        Ws[r * kWyYLd + q] = j < n ? W2[((size_t)s * kWyB + r) * n + j] : 0.f;
    }
    const int cw = 16 * warp;
    constexpr int kPV = 32 * kWyB / kWyThreads;
    float vr[kPV]; // the next 32 rows of V, fetched during the current ones
    auto fetch = [&](int row0) {
#pragma unroll
        for (int q = 0; q < kPV; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            const int i = e & 31, r = e >> 5, row = row0 + i;
            vr[q] = row < re ? wy_v(As, d.ld, R, n, k0, r, row) : 0.f;
        }
    };
    __syncthreads(); // R, cols and Ws in place
    fetch(rb);
    for (int row0 = rb; row0 < re; row0 += 32) {
        __syncthreads(); // the previous V tile is read
#pragma unroll
        for (int q = 0; q < kPV; q++) {
            const int e = threadIdx.x + kWyThreads * q;
            Vs[(e & 31) * 33 + (e >> 5)] = vr[q];
        }
        __syncthreads();
        if (row0 + 32 < re)
            fetch(row0 + 32);
        const int row = row0 + lane;
        float yo[16]; // the rows' current values, loaded ahead of the FMAs
#pragma unroll
        for (int v = 0; v < 16; v++) {
            const long long o = cols[cw + v];
            yo[v] = o >= 0 && row < re ? out[o + row] : 0.f;
        }
        float acc[16];
#pragma unroll
        for (int v = 0; v < 16; v++)
            acc[v] = 0.f;
#pragma unroll 4
        for (int r = 0; r < kWyB; r++) {
            const float a = Vs[lane * 33 + r];
            const float4 *w = reinterpret_cast<const float4 *>(&Ws[r * kWyYLd + cw]);
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float4 x = w[h];
                acc[4 * h] = fmaf(a, x.x, acc[4 * h]);
                acc[4 * h + 1] = fmaf(a, x.y, acc[4 * h + 1]);
                acc[4 * h + 2] = fmaf(a, x.z, acc[4 * h + 2]);
                acc[4 * h + 3] = fmaf(a, x.w, acc[4 * h + 3]);
            }
        }
        if (row < re)
#pragma unroll
            for (int v = 0; v < 16; v++) {
                const long long o = cols[cw + v];
                if (o >= 0)
                    out[o + row] = yo[v] - acc[v];
            }
    }
}

// The stop rule after a sweep: the largest rotated cosine over the
// sinograms below kJacDone, or below 1e-3 and no longer falling by 4x (the
// float rounding floor of the rotated columns, which grows with sqrt(n) --
// near convergence the cyclic method is quadratic, so a real decrease is by
// orders of magnitude), or max_sweeps done.  state = {previous sweep's
// largest cosine (float bits; 1 before the first), sweeps done}.
__global__ void nos_sweep_check_kernel(const unsigned *__restrict__ off_bits, int n_sino,
                                       unsigned *__restrict__ state, int max_sweeps,
                                       cudaGraphConditionalHandle loop) {
    float worst = 0.f;
    for (int i = threadIdx.x; i < n_sino; i += 32)
        worst = fmaxf(worst, __uint_as_float(off_bits[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        worst = fmaxf(worst, __shfl_xor_sync(TT_FULL_MASK, worst, o));
    if (threadIdx.x != 0)
        return;
    const unsigned done = state[1] + 1;
    const float prev = done == 1 ? 1.f : __uint_as_float(state[0]);
    state[0] = __float_as_uint(worst);
    state[1] = done;
    const bool stop = worst < kJacDone || (worst < 1e-3f && worst > 0.25f * prev) ||
                      (int)done >= max_sweeps;
    cudaGraphSetConditional(loop, stop ? 0u : 1u);
}

} // namespace

cudaError_t launch_nos_offsets(const float *sino, int rows, int cols, int n_sino, int center,
                               int *offsets, cudaStream_t st) {
    const long long n = (long long)cols * n_sino;
    if (n <= 0)
        return cudaSuccess;
    if (rows > nos_max_rows()) {
        nos_offsets_long_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(sino, rows, (int)n,
                                                                             center, offsets);
        return cudaGetLastError();
    }
    const size_t smem = sizeof(float) * (size_t)kOffWarps * offsets_stride(rows);
    if (smem > opt_in_smem((const void *)nos_offsets_kernel))
        return cudaErrorInvalidValue;
    nos_offsets_kernel<<<(unsigned)((n + kOffWarps - 1) / kOffWarps), 32 * kOffWarps, smem, st>>>(
        sino, rows, (int)n, center, offsets);
    return cudaGetLastError();
}

cudaError_t launch_nos_align(const float *sino, int rows, int cols, int n_sino,
                             const NosDesc *desc, const int *offsets, float2 *A, size_t a_elems,
                             cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(A, 0, sizeof(float2) * a_elems, st);
    if (e != cudaSuccess)
        return e;
    nos_align_kernel<<<dim3(cols, n_sino), 128, 0, st>>>(sino, rows, cols, desc, offsets, A);
    return cudaGetLastError();
}

template <int K, int T>
static cudaError_t qr_steps(float2 *A, const NosDesc *desc, int n, int n_sino, const NosWork &w,
                            cudaStream_t st) {
    // CTAs per sinogram: one wave over all sinograms
    constexpr size_t smem = qr_smem(K, T);
    if (smem > opt_in_smem((const void *)qr_step_kernel<K, T>))
        return cudaErrorInvalidValue;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, qr_step_kernel<K, T>, T, smem);
    const int wave = std::max(1, sms * std::max(per_sm, 1) / std::max(n_sino, 1));
    for (int k = 0; k < n; k++) {
        // CTAs of one column while that makes at most 6 per SM, of whole groups above:
        // the work a CTA does whatever its columns then counts for more than
        // the chain over them (1 x 1449 x 360, 0.31 ms less in all than with groups;
        // 4 x 450 x 360, 0.17 more)
        const long long left = n - k;
        const long long g =
            left * n_sino <= 6LL * sms ? left : (left + kQrGroup - 1) / kQrGroup;
        qr_step_kernel<K, T><<<dim3((unsigned)std::min<long long>(g, wave), n_sino), T, smem,
                               st>>>(A, desc, n, n_sino, k, w);
    }
    return cudaSuccess;
}

int nos_max_rows() { return 32 * kQrThreads; }

// Threads per CTA and rows per thread of the QR by longest column: 128 threads up to
// 2048 rows (more CTAs, and so more column chains, in flight per SM), 256
// above; short columns take fewer rows per thread, so fewer registers and more
// CTAs per SM with fewer columns each.
struct QrClass {
    int threads, rows;
};
constexpr QrClass kQrClasses[kNosQrClasses] = {{128, 4},  {128, 8},  {128, 12}, {128, 16},
                                               {256, 16}, {256, 24}, {256, 32}};

int nos_qr_class(int max_m) {
    int c = 0;
    while (c < kNosQrClasses - 1 && max_m > kQrClasses[c].threads * kQrClasses[c].rows)
        c++;
    return c;
}

int nos_class_rows(int max_m) {
    const QrClass c = kQrClasses[nos_qr_class(max_m)];
    return std::max(max_m, c.threads * c.rows);
}

// A column step reads and writes up to threads - 1 rows past the last.
int nos_ld(int m, int max_m) { return (m + kQrClasses[nos_qr_class(max_m)].threads + 3) & ~3; }

cudaError_t launch_nos_factor(float2 *A, const NosDesc *desc, int n, int n_sino, int max_m,
                              const NosWork &w, cudaStream_t st) {
    if (max_m > nos_max_rows())
        return cudaErrorInvalidValue;
    qr_init_kernel<<<dim3(n, n_sino), kQrThreads, 0, st>>>(A, desc, n, w);
    cudaError_t e = cudaSuccess;
    switch (nos_qr_class(max_m)) {
    case 0:
        e = qr_steps<kQrClasses[0].rows, kQrClasses[0].threads>(A, desc, n, n_sino, w, st);
        break;
    case 1:
        e = qr_steps<kQrClasses[1].rows, kQrClasses[1].threads>(A, desc, n, n_sino, w, st);
        break;
    case 2:
        e = qr_steps<kQrClasses[2].rows, kQrClasses[2].threads>(A, desc, n, n_sino, w, st);
        break;
    case 3:
        e = qr_steps<kQrClasses[3].rows, kQrClasses[3].threads>(A, desc, n, n_sino, w, st);
        break;
    case 4:
        e = qr_steps<kQrClasses[4].rows, kQrClasses[4].threads>(A, desc, n, n_sino, w, st);
        break;
    case 5:
        e = qr_steps<kQrClasses[5].rows, kQrClasses[5].threads>(A, desc, n, n_sino, w, st);
        break;
    default:
        e = qr_steps<kQrClasses[6].rows, kQrClasses[6].threads>(A, desc, n, n_sino, w, st);
    }
    if (e != cudaSuccess)
        return e;
    const long long nn = (long long)n * n;
    nos_rt_kernel<<<dim3((unsigned)((nn + 255) / 256), n_sino), 256, 0, st>>>(A, desc, n, w);
    return cudaGetLastError();
}

static int nos_blocks(int n) { // of kBJ columns, an even number
    const int nb = (n + kBJ - 1) / kBJ;
    return nb + (nb & 1);
}

template <int K4>
static cudaError_t block_rounds(int n, int n_sino, const NosWork &w, cudaStream_t st) {
    const int nbp = nos_blocks(n);
    const size_t smem = sizeof(float) * block_round_smem_floats(K4);
    if (128 * K4 < n)
        return cudaErrorInvalidValue;
    if (smem > opt_in_smem((const void *)rt_block_round_kernel<K4>))
        return cudaErrorInvalidValue;
    for (int r = 0; r < nbp - 1; r++)
        rt_block_round_kernel<K4><<<dim3(nbp / 2, n_sino), kBThreads, smem, st>>>(
            w.X, w.J, n, nbp, r, w.off_bits, w.tiny, w.sweep_state);
    return cudaGetLastError();
}

size_t nos_rotation_floats(int n, int n_sino) {
    const size_t nbp = nos_blocks(n);
    return 2 * n_sino * (nbp - 1) * (nbp / 2) * kBJFloats;
}

// Eight warps per CTA where the sweeps' rounds fill the machine (fewer copies of the
// J's: 1.8 ms less of the orthonormal circus at 8 x 5795 x 720 than with four), else
// four (0.12 ms less at 8 x 1449 x 360).
static cudaError_t rotate_v(int n, int n_sino, const NosWork &w, cudaStream_t st) {
    const int nbp = nos_blocks(n);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int warps = nbp / 2 * n_sino > sms ? kVMaxWarps : 4, rows = 4 * warps;
    const size_t smem = jacobi_v_smem(nbp, warps); // 209 KB at 1024 columns and 8 warps
    if (smem > opt_in_smem((const void *)jacobi_v_kernel))
        return cudaErrorInvalidValue;
    jacobi_v_kernel<<<dim3((n + rows - 1) / rows, n_sino), 32 * warps, smem, st>>>(
        w.V, w.J, n, nbp, w.sweep_state);
    return cudaGetLastError();
}

cudaError_t launch_nos_sweep(int n, int n_sino, const NosWork &w, int max_sweeps,
                             cudaGraphConditionalHandle loop, cudaStream_t st, cudaStream_t side,
                             cudaEvent_t fork, cudaEvent_t join) {
    cudaError_t e = cudaMemsetAsync(w.off_bits, 0, sizeof(unsigned) * n_sino, st);
    // the previous sweep's rotations of V beside this sweep's rounds
    if (e == cudaSuccess)
        e = cudaEventRecord(fork, st);
    if (e == cudaSuccess)
        e = cudaStreamWaitEvent(side, fork, 0);
    if (e == cudaSuccess)
        e = rotate_v(n, n_sino, w, side);
    if (e == cudaSuccess)
        e = cudaEventRecord(join, side);
    if (e != cudaSuccess)
        return e;
    if (n <= 128)
        e = block_rounds<1>(n, n_sino, w, st);
    else if (n <= 256)
        e = block_rounds<2>(n, n_sino, w, st);
    else if (n <= 384)
        e = block_rounds<3>(n, n_sino, w, st);
    else if (n <= 512)
        e = block_rounds<4>(n, n_sino, w, st);
    else if (n <= 768)
        e = block_rounds<6>(n, n_sino, w, st);
    else if (n <= 1024)
        e = block_rounds<8>(n, n_sino, w, st);
    else
        e = cudaErrorInvalidValue; // more than 1024 angles
    if (e != cudaSuccess)
        return e;
    e = cudaStreamWaitEvent(st, join, 0);
    if (e != cudaSuccess)
        return e;
    nos_sweep_check_kernel<<<1, 32, 0, st>>>(w.off_bits, n_sino, w.sweep_state, max_sweeps,
                                             loop);
    return cudaGetLastError();
}

// Shape of the blocked Q application: row chunks of 32 ns rows, ns halved
// from 8 until the GEMM passes have at least 3 CTAs per SM (or ns is 1).
struct WyShape {
    int nbk, tiles, ns, nchunk0;
    size_t t_floats, part_floats, w2_floats;
};
static WyShape wy_shape(int n, int n_sino, int max_m) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    WyShape w;
    w.nbk = (n + kWyB - 1) / kWyB;
    w.tiles = (n + kWyCols - 1) / kWyCols;
    w.ns = 8;
    auto chunks = [&](int ns) { return (max_m + 32 * ns - 1) / (32 * ns); };
    while (w.ns > 1 && (long long)w.tiles * chunks(w.ns) * n_sino < 3LL * std::max(sms, 1))
        w.ns /= 2;
    w.nchunk0 = chunks(w.ns);
    w.t_floats = (size_t)n_sino * w.nbk * kWyB * kWyB;
    w.part_floats = (size_t)n_sino * w.nchunk0 * kWyB * n;
    w.w2_floats = (size_t)n_sino * kWyB * n;
    return w;
}

// The blocked application takes over from the register kernel where the
// aligned columns no longer fit its registers (measured on 8 sinograms of
// 5795 x 720: the whole assembly 9.5 ms against 32.4 ms with a shared-memory
// form of the one-reflector-at-a-time kernel; on 1843 x 360 the register
// kernel is the faster: 1.04 against 1.33 ms, and 0.6 since).
static bool wy_path(int n, int max_m) { return n > kNosMaxCols || max_m > 16 * kQThreads; }

static int nos_refl_ld(int max_m) { return (max_m + kQThreads - 1) / kQThreads * kQThreads; }

size_t nos_assemble_floats(int n, int n_sino, int max_m) {
    if (!wy_path(n, max_m))
        return (size_t)n_sino * n * nos_refl_ld(max_m);
    const WyShape w = wy_shape(n, n_sino, max_m);
    return w.t_floats + w.part_floats + w.w2_floats;
}

cudaError_t launch_nos_assemble(const float2 *A, const NosDesc *desc, int n, int n_sino,
                                int max_m, const NosWork &w, float *out, cudaStream_t st) {
    const long long nn = (long long)n * n;
    const dim3 ge((unsigned)((nn + 255) / 256), n_sino), gt((n + kGemmTile - 1) / kGemmTile, (n + kGemmTile - 1) / kGemmTile, n_sino);
    const cudaError_t e = rotate_v(n, n_sino, w, st); // the last sweep's
    if (e != cudaSuccess)
        return e;
    rt_invnorm_kernel<<<dim3((n + 3) / 4, n_sino), 128, 0, st>>>(w.X, n, w.tiny, w.inv);
    rt_scale_kernel<<<ge, 256, 0, st>>>(w.X, w.inv, n);
    // P = V U^T, then one Newton-Schulz step P <- P (3 I - P^T P) / 2 (in the
    // V buffer), which removes the symmetric part of P's distance from
    // orthogonality left by the float sweeps' stopping bound; S = P^T P goes
    // to the X buffer
    rt_gemm_kernel<<<gt, 256, 0, st>>>(w.V, 1, n, w.X, n, 1, nullptr, 1.f, 0.f, n, w.P);
    rt_gemm_kernel<<<gt, 256, 0, st>>>(w.P, n, 1, w.P, 1, n, nullptr, 1.f, 0.f, n, w.X);
    rt_gemm_kernel<<<gt, 256, 0, st>>>(w.P, 1, n, w.X, 1, n, w.P, -0.5f, 1.5f, n, w.V);
    const dim3 gq((n + kQCols - 1) / kQCols, n_sino);
    if (!wy_path(n, max_m)) {
        const int ldv = nos_refl_ld(max_m);
        nos_refl_kernel<<<dim3(n, n_sino), kQThreads, 0, st>>>(A, desc, w.scale, w.perm, n, ldv,
                                                                w.wy);
        if (max_m <= 8 * kQThreads)
            nos_apply_q_reg_kernel<8><<<gq, kQThreads, 0, st>>>(w.wy, ldv, desc, w.tau, w.perm,
                                                                 w.V, n, out);
        else
            nos_apply_q_reg_kernel<16><<<gq, kQThreads, 0, st>>>(w.wy, ldv, desc, w.tau, w.perm,
                                                                  w.V, n, out);
        return cudaGetLastError();
    }
    // Y = Q [P; 0] in the output, block by block (last block first)
    const WyShape sh = wy_shape(n, n_sino, max_m);
    float *T = w.wy, *part = T + sh.t_floats, *W2 = part + sh.part_floats;
    wy_init_kernel<<<dim3(n, n_sino), kWyThreads, 0, st>>>(w.V, desc, w.perm, n, out);
    wy_t_kernel<<<dim3(sh.nbk, n_sino), kWyThreads, 0, st>>>(A, desc, w.tau, w.scale, w.perm,
                                                              n, T);
    for (int jb = sh.nbk - 1; jb >= 0; jb--) {
        const int k0 = jb * kWyB;
        const int nch = (max_m - k0 + 32 * sh.ns - 1) / (32 * sh.ns);
        const dim3 g(sh.tiles, nch, n_sino);
        wy_vty_kernel<<<g, kWyThreads, 0, st>>>(A, desc, w.tau, w.scale, w.perm, n, k0, sh.ns,
                                                 out, part);
        wy_w2_kernel<<<dim3((n + 31) / 32, n_sino), kWyThreads, 0, st>>>(T, part, nch, n, jb,
                                                                         sh.nbk, W2);
        wy_update_kernel<<<g, kWyThreads, 0, st>>>(A, desc, w.tau, w.scale, w.perm, n, k0,
                                                    sh.ns, W2, out);
    }
    return cudaGetLastError();
}

} // namespace tt
