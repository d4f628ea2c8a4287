// Host build of the fused kernels' line passes (wvlh_lines.cuh) with one
// thread standing for a block, so that their index arithmetic and tap sums can
// be checked against dense matrices without a GPU.  Buffers have exactly the
// size that the kernels lay out, between guard words.
#include <cuda_runtime.h>

#undef __device__
#undef __host__
#undef __forceinline__
#undef __global__
#define __device__
#define __host__
#define __forceinline__ inline
#define __global__

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

using std::max;
using std::min;
static struct { int x; } threadIdx = {0}, blockDim = {1}, blockIdx = {0};
static void __syncthreads() {}
static double __shfl_xor_sync(unsigned, double, int) { return 0.0; }
static unsigned __viaddmin_u32(unsigned a, unsigned b, unsigned c) { return std::min(a + b, c); }
static float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)}; }
static float2 __fmul2_rn(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }

#include "wvlh_lines.cuh"

using namespace wvlh;

// A buffer of exactly n values, aligned for point pairs and pre-filled with a
// value that would show in the results, between guards: a stray read brings
// that value into a result, a stray write changes a guard.
static int g_broken = 0;
template <class T> struct Buf {
    static constexpr size_t kGuard = 64;
    T *base, *p;
    size_t n;
    explicit Buf(size_t n_) : n(n_)
    {
        const size_t all = n + 2 * kGuard;
        base = (T *)aligned_alloc(16, (all * sizeof(T) + 15) / 16 * 16);
        for (size_t i = 0; i < all; ++i) base[i] = T(1e30);
        p = base + kGuard;
    }
    ~Buf()
    {
        for (size_t i = 0; i < kGuard; ++i)
            if (base[i] != T(1e30) || p[n + i] != T(1e30)) g_broken = 1;
        free(base);
    }
};

template <class T, int SEG> static void rows(int op, int N, int per, int nrows, const double *in, double *out, double *energy)
{
    const int H = half_off(N), I = isf_len(N, per), F = fine_len(N, per);
    const int pitch = vec_pitch(max(2 * H, max(F, I)));
    Buf<T> a(nrows * pitch), b(nrows * pitch);
    const int nin = op == 1 ? I : 2 * N, nout = op == 0 ? I : 2 * N;
    auto wpos = [&](int c) { return c < N ? c : c - N + H; };
    for (int r = 0; r < nrows; ++r)
        for (int c = 0; c < nin; ++c) a.p[r * pitch + (op == 1 ? c : wpos(c))] = (T)in[r * nin + c];
    double e = 0.0;
    if (op == 0) row_b<T, SEG>(a.p, b.p, nrows, pitch, N, H, per);
    else if (op == 1) row_bt<T, SEG>(a.p, b.p, nrows, pitch, I, N, H, per);
    else for (int i = 0; i < nrows * pitch; ++i) b.p[i] = T(0);
    if (op == 2) row_t<T, SEG, true, true>(a.p, b.p, nrows, pitch, N, H, per, -0.5 / TNorm<T>::v, T(0.25), &e);
    for (int r = 0; r < nrows; ++r)
        for (int c = 0; c < nout; ++c) out[r * nout + c] = b.p[r * pitch + (op == 0 ? c : wpos(c))];
    *energy = e;
}

template <class T, int SEG> static void cols(int op, int N, int per, int ncol, const double *in, double *out, double *energy)
{
    using U = typename ColUnit<T>::U;
    using V = typename U::V;
    const int I = isf_len(N, per), nin = op == 1 ? I : 2 * N, nout = op == 0 ? I : 2 * N;
    const int ps = (ncol + 1) & ~1;
    Buf<T> a(nin * ps);
    if (ps > ncol)
        for (int p = 0; p < nin; ++p) a.p[p * ps + ncol] = T(0);   // the kernels zero an odd plane's pad column
    for (int c = 0; c < ncol; ++c)
        for (int p = 0; p < nin; ++p) a.p[p * ps + c] = (T)in[c * nin + p];
    auto put = [&](int u, int q, V v) {
        const T *e = (const T *)&v;
        for (int k = 0; k < U::n; ++k)
            if (u * U::n + k < ncol) out[(u * U::n + k) * nout + q] = (double)e[k] / (op == 2 ? TNorm<T>::v : 1.0);
    };
    double e = 0.0;
    for (int u = 0; u * U::n < ncol; ++u) {
        const int col = u * U::n;
        if (op == 0) {
            const int np = per ? N : N + 15;
            for (int u0 = 0; u0 < np; u0 += SEG) {
                V acc[2 * SEG];
                col_b<U, SEG>(acc, a.p, col, ps, N, N, per, u0);
                for (int t = 0; t < 2 * SEG; ++t)
                    if (2 * u0 + t < I) put(u, 2 * u0 + t, acc[t]);
            }
        } else {
            for (int i0 = 0; i0 < N; i0 += SEG) {
                V c[SEG], d[SEG];
                if (op == 1) col_bt<U, SEG>(c, d, a.p, col, ps, I, per, i0);
                else col_t<U, SEG>(c, d, a.p, col, ps, N, N, per, i0);
                V es = U::zero();
                for (int t = 0; t < SEG; ++t)
                    if (i0 + t < N) {
                        put(u, i0 + t, c[t]);
                        put(u, N + i0 + t, d[t]);
                        if (op == 2) {
                            es = U::fmav(c[t], *(const V *)(a.p + col + (i0 + t) * ps), es);
                            es = U::fmav(d[t], *(const V *)(a.p + col + (N + i0 + t) * ps), es);
                        }
                    }
                e += (double)U::sum(es) / TNorm<T>::v;
            }
        }
    }
    *energy = e;
}

extern "C" double b_inv6(int prec) { return prec == 32 ? BInv6<float>::v : BInv6<double>::v; }

// op 0: B, 1: B^T (FP32: scaled as the taps are), 2: T (rows: 0.25 x - 0.5 T x and <x | -0.5 T x>; columns:
// T x and <x | T x>); lines are dense rows of in / out; seg: wavelet points of
// a segment, 6 (FP32 plane kernels, density) or 8
template <int SEG>
static void run(int prec, int as_rows, int op, int N, int per, int nline, const double *in, double *out, double *energy)
{
    if (as_rows && prec == 32) rows<float, SEG>(op, N, per, nline, in, out, energy);
    else if (as_rows) rows<double, SEG>(op, N, per, nline, in, out, energy);
    else if (prec == 32) cols<float, SEG>(op, N, per, nline, in, out, energy);
    else cols<double, SEG>(op, N, per, nline, in, out, energy);
}
extern "C" int line_pass(int prec, int as_rows, int op, int seg, int N, int per, int nline, const double *in, double *out,
                         double *energy)
{
    g_broken = 0;
    seg == 6 ? run<6>(prec, as_rows, op, N, per, nline, in, out, energy)
             : run<8>(prec, as_rows, op, N, per, nline, in, out, energy);
    return g_broken;
}
