// Line passes of the fused kernels: the 1D operators of the Daubechies-16 local
// Hamiltonian, each composed along its axis into ONE pass over a line in
// shared memory.
//
//  B   = magic filter . synthesis: wavelet line [s | w] of N + N points ->
//        real-space line, 31 taps per wavelet half and pair of outputs
//          r(j) = sum_i gs(j - 2i) s(i) + gw(j - 2i) w(i),  j - 2i in [-14, 16]
//          gs(m) = sum_l fil(l) ch(m + l),  gw(m) = sum_l fil(l) cg(m + l)
//        (convolut_simple_per.f90:59-103 followed by :200-243)
//  B^T = analysis . transposed magic filter (:246-291 followed by :11-57):
//          c(i) = sum_j gs(j - 2i) r(j),  d(i) = sum_j gw(j - 2i) r(j)
//  T   = analysis . kinetic . synthesis, the kinetic operator in the wavelet
//        basis (the a, b, c, e filters of convolut_ib_optim.f90:987-1035):
//          s'(i) = sum_l a(l) s(i+l) + c(-l) w(i+l)
//          w'(i) = sum_l c(l) s(i+l) + e(l) w(i+l),  l in [-14, 14],
//        times -1/(2 h^2), h the coarse spacing
// Periodic lines wrap; free lines are zero outside [0, N) and grow to the
// 2N + 29 points j in [-14, 2N + 14], stored at j + 14 (the j = 2N + 15 that
// completes the last pair is exactly zero).  The compositions need no
// intermediate bounds: the grown lines hold the whole support.
//
// Why composed: B costs 31 multiply-adds per output against 16 + 16 in two
// passes, T 46 (FP32) or 54 (FP64) against 16 + 29 + 16 in three, with one
// window load, one store and one barrier instead of two or three.  The passes
// they replace were bound by instruction issue, half of it addressing, window
// loads and stores.
//
// Taps left out of T: at |l| = 14 (FP64 keeps |l| <= 13) they are up to 1.2e-17,
// 3.0e-17 in all for an output, a seventh of half a rounding of the largest
// scaling tap, 3.55; at |l| >= 12 (FP32 keeps |l| <= 11) up to 1.05e-10, 2.5e-10
// in all, 1/470 of half a rounding.
//
// FP64 energies: a tap of B off by a rounding moves |B x|^2, and so E_pot and
// the density, the same way for every orbital.  wvl_composed.h holds the exact
// sums of products, rounded so that these moves cancel: |B x|^2 is right to 1e-17
// of itself per axis at every frequency (sums rounded at each step: 4e-16; the
// nearest doubles: 9e-17), the outputs to 2e-16.  E_kin of a smooth orbital is a
// small difference of large terms: T's taps are those of the same doubles as
// the separate passes (not the published a, c, e of the many-digit filters, off
// by 1e-15 at zero frequency), rounded so that the scaling part is right to 3e-19
// at zero frequency and 4e-18 below 0.5, the rest to 1e-15 of T's norm of 40.
//
// FP32 energies: a tap c rounded to FP32 is off by lo = c - fl(c), the same way
// for every output, and E_kin = <x | T x> by lo(l) sum_i x(i) x(i+l).  The FP32
// taps of T are kept times TNorm (the scale -1/(2 h^2) divides by it), a factor
// found by a scan so that the taps above 0.02 round to within 7.5e-9 (unscaled: up to
// 8.3e-7), and rounded in turn: the scaling part is right to 2.2e-11 at zero
// frequency and 1.9e-9 below 0.5 (nearest values: 1.5e-8), all of T to 3.9e-8,
// times 1 / (2 h^2) in Ha per axis on a normalised orbital (h = 0.45: 5e-11, 5e-9
// and 1e-7; the separate passes with their corrections: 4e-8, 4e-8 and 3e-7).
// B's FP32 taps are kept times 0.9752 and rounded as in FP64: |B x|^2 is
// right to 2.1e-9 of itself per axis at every frequency and to 6e-10 on smooth
// lines (nearest FP32 taps: 3.1e-8 and 2.4e-8, all smooth orbitals the same way),
// the outputs to 1.1e-8 (2.3e-8).  E_pot, the potential's term of H psi and the
// density each hold six B: BInv6 comes in where they are formed (once a thread,
// in K3's addition of Z2, on the orbital's factor), at no cost.
#pragma once
#include <cuda_runtime.h>

#include "wvl_composed.h"
#include "wvlh_common.cuh"

namespace wvlh {

// ---------------------------------------------------------------- taps
// taps of B (FP32: times 0.9752, gen_composed.py): gs (half 0, scaling function) and gw
// (half 1, wavelet) at m
template <class T> __device__ __forceinline__ constexpr T b_tap(int half, int m)
{
    if (m < -14 || m > 16) return T(0);
    if constexpr (sizeof(T) == 4) {
        constexpr T s[31] = WVL_B32_S_INIT, w[31] = WVL_B32_W_INIT;
        return half ? w[m + 14] : s[m + 14];
    } else {
        constexpr T s[31] = WVL_B64_S_INIT, w[31] = WVL_B64_W_INIT;
        return half ? w[m + 14] : s[m + 14];
    }
}
// what six passes of scaled taps (B on three axes, twice) are multiplied by
template <class T> struct BInv6 { static constexpr double v = sizeof(T) == 4 ? WVL_B32_INV6 : 1.0; };
// tap of output half `o` from input half `i` at offset l of TNorm T
template <class V> __device__ __forceinline__ constexpr V t_tap(int o, int i, int l)
{
    const int al = l < 0 ? -l : l;
    if (al > 14) return V(0);
    if constexpr (sizeof(V) == 4) {
        constexpr V a[15] = WVL_T32_A_INIT, c[29] = WVL_T32_C_INIT, e[15] = WVL_T32_E_INIT;
        return o == i ? (o ? e[al] : a[al]) : (o ? c[l + 14] : c[14 - l]);
    } else {
        constexpr V a[15] = WVL_T64_A_INIT, c[29] = WVL_T64_C_INIT, e[15] = WVL_T64_E_INIT;
        return o == i ? (o ? e[al] : a[al]) : (o ? c[l + 14] : c[14 - l]);
    }
}
template <class T> struct TReach { static constexpr int v = sizeof(T) == 4 ? 11 : 13; };
template <class T> struct TNorm { static constexpr double v = sizeof(T) == 4 ? WVL_T32_NORM : 1.0; };

// ---------------------------------------------------------------- units
// What one thread carries of a point: a column pass takes 8 bytes of a row of
// columns, two FP32 columns (every tap one packed fma.rn.f32x2, which halves
// the instructions per multiply-add) or one FP64 column; a row pass takes one
// value.
struct U1f {
    using T = float;
    using V = float;
    static __device__ __forceinline__ V fma(float c, V x, V a) { return ::fmaf(c, x, a); }
    static __device__ __forceinline__ V fmav(V c, V x, V a) { return ::fmaf(c, x, a); }
    static __device__ __forceinline__ V zero() { return 0.f; }
    static __device__ __forceinline__ float sum(V a) { return a; }
};
struct U2f {
    using T = float;
    using V = float2;
    static constexpr int n = 2;
    static __device__ __forceinline__ V fma(float c, V x, V a) { return __ffma2_rn(make_float2(c, c), x, a); }
    static __device__ __forceinline__ V fmav(V c, V x, V a) { return __ffma2_rn(c, x, a); }
    static __device__ __forceinline__ V mul(float c, V x) { return __fmul2_rn(make_float2(c, c), x); }
    static __device__ __forceinline__ V mulv(V c, V x) { return __fmul2_rn(c, x); }
    static __device__ __forceinline__ V zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ float sum(V a) { return a.x + a.y; }
    static __device__ __forceinline__ float first(V a) { return a.x; }
    // e += x . r in FP64
    static __device__ __forceinline__ void dot(double &e, V x, V r)
    {
        e = ::fma((double)x.x, (double)r.x, e);
        e = ::fma((double)x.y, (double)r.y, e);
    }
};
struct U1d {
    using T = double;
    using V = double;
    static constexpr int n = 1;
    static __device__ __forceinline__ V fma(double c, V x, V a) { return ::fma(c, x, a); }
    static __device__ __forceinline__ V fmav(V c, V x, V a) { return ::fma(c, x, a); }
    static __device__ __forceinline__ V mul(double c, V x) { return c * x; }
    static __device__ __forceinline__ V mulv(V c, V x) { return c * x; }
    static __device__ __forceinline__ void dot(double &e, V x, V r) { e = ::fma(x, r, e); }
    static __device__ __forceinline__ V zero() { return 0.0; }
    static __device__ __forceinline__ double sum(V a) { return a; }
    static __device__ __forceinline__ double first(V a) { return a; }
};
template <class T> struct ColUnit;
template <> struct ColUnit<float> { using U = U2f; };
template <> struct ColUnit<double> { using U = U1d; };
template <class T> struct RowUnit;
template <> struct RowUnit<float> { using U = U1f; };
template <> struct RowUnit<double> { using U = U1d; };

// ---------------------------------------------------------------- windows
// A window streams through its consumer: f(k, x) with x = point p0 + k of the
// line, k < W a constant after unrolling, so that only the accumulators (and
// not the window) live in registers.  Points outside a free line are zero; a
// periodic line is walked by a byte offset that returns to its start at the
// line's end, in one fused add-and-minimum (right for lines shorter than the
// window): min(u + step, u + step - length), both unsigned, is the first while
// u + step stays below the length and the second, wrapped, at the end.  Two
// integer instructions a load (three for rows); a compare and select per point
// took nine, and more of the kernels' issue slots than the multiply-adds.

// p0 moved into [0, L) along a periodic line
__device__ __forceinline__ int wrap_start(int p0, int L)
{
    while (p0 < 0) p0 += L;
    while (p0 >= L) p0 -= L;
    return p0;
}
__device__ __forceinline__ unsigned wrap_step(unsigned u, unsigned step, unsigned len)
{
    return __viaddmin_u32(u, step - len, u + step);
}
template <class V, class T> __device__ __forceinline__ V load_at(const T *in, unsigned byte)
{
    return *reinterpret_cast<const V *>(reinterpret_cast<const char *>(in) + byte);
}

// The unit at column `col` of a buffer whose points (rows) lie ps elements
// apart.  The column's own offset rides in the walker (it is smaller than a
// step, so the wrap still falls between the line's ends): the base is the same
// for every thread and a load needs no address add.
template <class U, int W, class F>
__device__ __forceinline__ void col_stream(const typename U::T *base, int col, int ps, int p0, int L, int per, F &&f)
{
    using T = typename U::T;
    using V = typename U::V;
    if (per) {
        const unsigned step = ps * (unsigned)sizeof(T), len = L * step;
        unsigned u = wrap_start(p0, L) * step + col * (unsigned)sizeof(T);
#pragma unroll
        for (int k = 0; k < W; ++k) {
            f(k, load_at<V>(base, u));
            u = wrap_step(u, step, len);
        }
    } else {
        const T *b = base + col + p0 * ps;
#pragma unroll
        for (int k = 0; k < W; ++k)
            f(k, (unsigned)(p0 + k) < (unsigned)L ? *reinterpret_cast<const V *>(b + k * ps) : U::zero());
    }
}

// Unit-stride rows that start on a point pair: x = row(q0 + SHIFT + k), q0
// even, read as point pairs.  Rows hold at least L + 1 points when L is odd;
// periodic rows of odd length walk point by point (a pair would straddle the
// wrap).
template <class T, int W, int SHIFT, class F>
__device__ __forceinline__ void row_stream(const T *in, int q0, int L, int per, F &&f)
{
    using V = typename Pair<T>::type;
    constexpr int R = SHIFT & 1, A0 = SHIFT - R, NV = (W + R + 1) / 2;
    const unsigned len = L * (unsigned)sizeof(T);
    if (per && (L & 1)) {
        unsigned u = wrap_start(q0 + SHIFT, L) * (unsigned)sizeof(T);
#pragma unroll
        for (int k = 0; k < W; ++k) {
            f(k, load_at<T>(in, u));
            u = wrap_step(u, sizeof(T), len);
        }
    } else if (per) {
        unsigned u = wrap_start(q0 + A0, L) * (unsigned)sizeof(T);
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            const V v = load_at<V>(in, u);
            u = wrap_step(u, 2 * sizeof(T), len);
            if (2 * c - R >= 0) f(2 * c - R, v.x);
            if (2 * c + 1 - R < W) f(2 * c + 1 - R, v.y);
        }
    } else {
        const int p = q0 + A0;
        const T *b = in + p;
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            V v;
            v.x = T(0);
            v.y = T(0);
            if ((unsigned)(p + 2 * c) < (unsigned)L) v = *reinterpret_cast<const V *>(b + 2 * c);
            if (p + 2 * c + 1 >= L) v.y = T(0);
            if (2 * c - R >= 0) f(2 * c - R, v.x);
            if (2 * c + 1 - R < W) f(2 * c + 1 - R, v.y);
        }
    }
}

// ---------------------------------------------------------------- tap sums
// acc[2t + o] (pair u0 + t of B's output, o = 0, 1) from window point k of one
// wavelet half, x = coarse point u0 - 8 + k
template <class U, int HS>
__device__ __forceinline__ void b_point(typename U::V (&acc)[2 * HS], int k, typename U::V x, int half)
{
#pragma unroll
    for (int t = 0; t < HS; ++t)
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const int m = 16 + o - 2 * (k - t);
            if (m >= -14 && m <= 16) acc[2 * t + o] = U::fma(b_tap<typename U::T>(half, m), x, acc[2 * t + o]);
        }
}
// c[t], d[t] (coarse point i0 + t of B^T) from x = r(2 i0 - 14 + k)
template <class U, int HS>
__device__ __forceinline__ void bt_point(typename U::V (&c)[HS], typename U::V (&d)[HS], int k, typename U::V x)
{
    using T = typename U::T;
#pragma unroll
    for (int t = 0; t < HS; ++t) {
        const int m = k - 14 - 2 * t;
        if (m < -14 || m > 16) continue;
        c[t] = U::fma(b_tap<T>(0, m), x, c[t]);
        d[t] = U::fma(b_tap<T>(1, m), x, d[t]);
    }
}
// s[t], w[t] (coarse point i0 + t of TNorm T) from x = point i0 - R + k of input half i
template <class U, int SEG, int R>
__device__ __forceinline__ void t_point(typename U::V (&s)[SEG], typename U::V (&w)[SEG], int k, typename U::V x, int i)
{
    using T = typename U::T;
#pragma unroll
    for (int t = 0; t < SEG; ++t) {
        const int l = k - R - t;
        if (l < -R || l > R) continue;
        s[t] = U::fma(t_tap<T>(0, i, l), x, s[t]);
        w[t] = U::fma(t_tap<T>(1, i, l), x, w[t]);
    }
}
template <class U, int n>
__device__ __forceinline__ void clear(typename U::V (&acc)[n])
{
#pragma unroll
    for (int t = 0; t < n; ++t) acc[t] = U::zero();
}

// ---------------------------------------------------------------- column passes
// One segment of the column unit at column `col` of buffer `in`; points lie ps
// elements apart, the wavelet half starts at point H.

// pairs u0 .. u0 + HS - 1 of B's output (free lines: pair u is the points
// j = 2u - 14, 2u - 13, stored at 2u, 2u + 1)
template <class U, int HS>
__device__ __forceinline__ void col_b(typename U::V (&acc)[2 * HS], const typename U::T *in, int col, int ps, int H, int N,
                                      int per, int u0)
{
    using V = typename U::V;
    const int p0 = u0 - (per ? 8 : 15);
    clear<U>(acc);
    col_stream<U, HS + 15>(in, col, ps, p0, N, per, [&](int k, V x) { b_point<U, HS>(acc, k, x, 0); });
    col_stream<U, HS + 15>(in + H * ps, col, ps, p0, N, per, [&](int k, V x) { b_point<U, HS>(acc, k, x, 1); });
}
// coarse outputs i0 .. i0 + HS - 1 of B^T; L points of the real-space line
template <class U, int HS>
__device__ __forceinline__ void col_bt(typename U::V (&c)[HS], typename U::V (&d)[HS], const typename U::T *in, int col, int ps,
                                       int L, int per, int i0)
{
    using V = typename U::V;
    clear<U>(c);
    clear<U>(d);
    col_stream<U, 2 * HS + 29>(in, col, ps, 2 * i0 - (per ? 14 : 0), L, per, [&](int k, V x) { bt_point<U, HS>(c, d, k, x); });
}
// coarse outputs i0 .. i0 + SEG - 1 of TNorm T
template <class U, int SEG>
__device__ __forceinline__ void col_t(typename U::V (&s)[SEG], typename U::V (&w)[SEG], const typename U::T *in, int col, int ps,
                                      int H, int N, int per, int i0)
{
    using V = typename U::V;
    constexpr int R = TReach<typename U::T>::v, W = SEG + 2 * R;
    clear<U>(s);
    clear<U>(w);
#pragma unroll
    for (int i = 0; i < 2; ++i)
        col_stream<U, W>(in + i * H * ps, col, ps, i0 - R, N, per, [&](int k, V x) { t_point<U, SEG, R>(s, w, k, x, i); });
}

// ---------------------------------------------------------------- row passes
// Rows of unit stride, one thread per (row, segment), lanes on consecutive
// rows: the pitch (vec_pitch) keeps their point pairs on distinct banks.  The
// wavelet half of a coarse row starts at the even point H.

__device__ __forceinline__ void store_pair(float *p, float a, float b) { *reinterpret_cast<float2 *>(p) = make_float2(a, b); }
__device__ __forceinline__ void store_pair(double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); }

// dst row = B of the src row: 2N points, or 2N + 30 with the zero that
// completes a free line's last pair (dst rows hold them)
template <class T, int HS>
__device__ __forceinline__ void row_b(const T *src, T *dst, int nrows, int pitch, int N, int H, int per)
{
    using U = typename RowUnit<T>::U;
    const int npair = per ? N : N + 15;
    for_items(nrows, (npair + HS - 1) / HS, [&](int row, int s) {
        const T *in = src + row * pitch;
        T *out = dst + row * pitch;
        const int u0 = s * HS;
        T acc[2 * HS];
        clear<U>(acc);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            auto f = [&](int k, T x) { b_point<U, HS>(acc, k, x, i); };
            if (per) row_stream<T, HS + 15, -8>(in + i * H, u0, N, 1, f);
            else row_stream<T, HS + 15, -15>(in + i * H, u0, N, 0, f);
        }
#pragma unroll
        for (int t = 0; t < HS; ++t)
            if (u0 + t < npair) store_pair(out + 2 * (u0 + t), acc[2 * t], acc[2 * t + 1]);
    });
}

// dst row [c | d at H] = B^T of the src row of L points
template <class T, int HS>
__device__ __forceinline__ void row_bt(const T *src, T *dst, int nrows, int pitch, int L, int N, int H, int per)
{
    using U = typename RowUnit<T>::U;
    for_items(nrows, (N + HS - 1) / HS, [&](int row, int s) {
        const T *in = src + row * pitch;
        T *out = dst + row * pitch;
        const int i0 = s * HS;
        T c[HS], d[HS];
        clear<U>(c);
        clear<U>(d);
        auto f = [&](int k, T x) { bt_point<U, HS>(c, d, k, x); };
        if (per) row_stream<T, 2 * HS + 29, -14>(in, 2 * i0, L, 1, f);
        else row_stream<T, 2 * HS + 29, 0>(in, 2 * i0, L, 0, f);
        // an odd line's last pair spills one value into the pad before the
        // wavelet half, or behind it
#pragma unroll
        for (int t = 0; t < HS; t += 2)
            if (i0 + t < N) {
                store_pair(out + i0 + t, c[t], c[t + 1]);
                store_pair(out + H + i0 + t, d[t], d[t + 1]);
            }
    });
}

// dst row += scale TNorm T src row (SHIFT: + cshift src row); EN: *energy +=
// <src | scale TNorm T src> (a segment's terms in T, the segments in FP64)
template <class T, int SEG, bool SHIFT, bool EN>
__device__ __forceinline__ void row_t(const T *src, T *dst, int nrows, int pitch, int N, int H, int per, double scale_d,
                                      T cshift, double *energy)
{
    using U = typename RowUnit<T>::U;
    using V2 = typename Pair<T>::type;
    constexpr int R = TReach<T>::v, W = SEG + 2 * R;
    const T scale = (T)scale_d;
    double e = 0.0;
    for_items(nrows, (N + SEG - 1) / SEG, [&](int row, int sg) {
        const T *in = src + row * pitch;
        T *out = dst + row * pitch;
        const int i0 = sg * SEG;
        T s[SEG], w[SEG];
        clear<U>(s);
        clear<U>(w);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            row_stream<T, W, -R>(in + i * H, i0, N, per, [&](int k, T x) { t_point<U, SEG, R>(s, w, k, x, i); });
        T es = T(0);
        auto put = [&](int off, const T(&v)[SEG]) {
#pragma unroll
            for (int t = 0; t < SEG; t += 2)
                if (i0 + t < N) {
                    const V2 p = *reinterpret_cast<const V2 *>(in + off + i0 + t);
                    V2 o = *reinterpret_cast<const V2 *>(out + off + i0 + t);
                    if (SHIFT) {
                        o.x = U::fma(cshift, p.x, o.x);
                        o.y = U::fma(cshift, p.y, o.y);
                    }
                    if (EN) {
                        es = U::fma(p.x, v[t], es);
                        if (i0 + t + 1 < N) es = U::fma(p.y, v[t + 1], es);
                    }
                    o.x = U::fma(scale, v[t], o.x);
                    o.y = U::fma(scale, v[t + 1], o.y);
                    *reinterpret_cast<V2 *>(out + off + i0 + t) = o;
                }
        };
        put(0, s);
        put(H, w);
        if (EN) e += (double)es * scale_d;
    });
    if (EN) *energy += e;
}

}  // namespace wvlh
