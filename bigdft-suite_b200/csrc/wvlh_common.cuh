// Common device code of the wvlh library: extents and layouts, and the 1D line
// passes of the plain path (one kernel per operator, wvlh_plain.cu).  The fused
// kernels compose these operators, wvlh_lines.cuh.
//
// A "line pass" applies one 1D operator of the Daubechies-16 local
// Hamiltonian (synthesis, analysis, magic filter, transposed magic filter,
// 29-tap kinetic) along lines of a shared-memory buffer.  Lines are addressed
// as base + line*ls + p*ps.  Each thread owns a segment of SEG consecutive
// outputs of one line, loads the input window for the whole segment into
// registers once, and issues SEG*taps FMAs from registers; the filter taps are
// compile-time immediates.
//
// Operator definitions (the math of the reference, Fortran indices):
//  syn  (orbitals/convolut_simple_per.f90:89-103, free: OpenCL syngrow1d):
//       y(2i+o) = sum_{l=-4..4} ch(2l+o) s(i-l) + cg(2l+o) w(i-l)
//  ana  (convolut_simple_per.f90:11-57, free: OpenCL anashrink1d):
//       c(i) = sum_{l=-7..8} ch(l) y(2i+l),  d(i) = sum cg(l) y(2i+l)
//  mf   (convrot_n_per :200-243):  r(i) = sum_{l=-8..7} fil(l) x(i+l)
//  mft  (convrot_t_per :246-291):  x(i) = sum_{l=-7..8} fil(-l) r(i+l)
//  kin  (convolut_kinetic_per_T :377-460):
//       y(i) += -1/(2h^2) sum_{l=-14..14} a(|l|) x(i+l)
// Periodic lines wrap; free lines are zero outside and grow/shrink:
// fine grid f in [-7, 2N+6] (stored at q=f+7), ISF grid in [-14, 2N+14]
// (stored at r+14), exactly the OpenCL grow/shrink kernels' extents.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "wvl_filters.h"

namespace wvlh {

template <class T> struct Filt {
    static __device__ __forceinline__ constexpr T ch(int i) { return (T)(WVL_CH_AT(i)); }
    static __device__ __forceinline__ constexpr T cg(int i) { return (T)(WVL_CG_AT(i)); }
    static __device__ __forceinline__ constexpr T mf(int i) { return (T)(WVL_MF_AT(i)); }
    static __device__ __forceinline__ constexpr T kin(int i) { return (T)(WVL_KIN_AT(i)); }
};

// Fine-grid and ISF-grid extents of one dimension with N coarse cells.
__host__ __device__ __forceinline__ int fine_len(int N, int per) { return per ? 2 * N : 2 * N + 14; }
__host__ __device__ __forceinline__ int isf_len(int N, int per) { return per ? 2 * N : 2 * N + 29; }

// Row pitch of a real-space plane in the fused kernels' scratch: the 2N points
// of a periodic row, or a free row's 2N + 29 rounded up to 16 bytes of FP32,
// so that rows start on a point pair and TMA can stride them.
__host__ __device__ __forceinline__ int isf_pitch(int N, int per) { return per ? 2 * N : (2 * N + 29 + 3) & ~3; }

// Scratch of one orbital in the fused kernels, in elements: D at 0, Z2 at z, Q
// (then Z1) at q.  The total is the room of three planes stacks on the fine
// and real-space grids (what callers budget, wvlh_region_scratch_bytes): the
// two wavelet stacks are smaller than fine ones in free directions, which
// covers Q's padded rows.
struct OrbScratch {
    long long z, q, total;
    // from one orbital of a batch to the next: on 16 bytes of FP32 (TMA strides),
    // and never more than callers budget; Q's last row ends well before
    __host__ __device__ long long stride() const { return total & ~3LL; }
};
__host__ __device__ inline OrbScratch orb_scratch(const int *N, const int *per)
{
    const long long G3 = 2LL * N[2], F1 = fine_len(N[0], per[0]), F2 = fine_len(N[1], per[1]);
    const long long w = G3 * 4 * N[0] * N[1];
    return OrbScratch{w, 2 * w, 2 * G3 * F1 * F2 + G3 * isf_len(N[0], per[0]) * isf_len(N[1], per[1])};
}

// Periodic index for -L <= p < 3L, without a division.
__device__ __forceinline__ int wrap_near(int p, int L)
{
    p += p < 0 ? L : 0;
    p -= p >= L ? L : 0;
    p -= p >= L ? L : 0;
    return p;
}

// Plane layout of the fused kernels' shared-memory buffers.  A coarse line is
// [s(0..N-1) | w(0..N-1)] with the wavelet half at the even offset
// half_off(N), so both halves start on a point pair.  Buffers whose lines run
// along rows use a row pitch with pitch % 4 == 2: every row starts on a point
// pair (8 bytes FP32, 16 bytes FP64), which lets the unit-stride passes load
// two points per instruction, and lanes that take consecutive rows still hit
// distinct banks (half-warp phases for 8-byte, quarter-warp for 16-byte).
__host__ __device__ constexpr int half_off(int N) { return (N + 1) & ~1; }
__host__ __device__ constexpr int coarse_width(int N) { return half_off(N) + N; }
__host__ __device__ constexpr int vec_pitch(int m) { return ((m + 1) & ~1) + ((((m + 1) & ~1) & 3) == 0 ? 2 : 0); }

// row pitch of the plane kernels' buffers for a box of N1 coarse cells in x
__host__ __device__ __forceinline__ int plane_pitch(int N1, int per1)
{
    const int w = 2 * half_off(N1), f = fine_len(N1, per1), r = isf_len(N1, per1);
    const int m = w > f ? w : f;
    return vec_pitch(m > r ? m : r);
}

// Cell table of one key set (LrDev::pos_c / pos_f): one warp per segment.
static __global__ void k_cell_places(int N1, int N2, int pitch, int nseg, const int32_t *__restrict__ keyg,
                                     const int32_t *__restrict__ keyv, uint16_t *__restrict__ pos)
{
    const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (s >= nseg) return;
    const int i = keyg[2 * s] - 1, len = keyg[2 * s + 1] - i, j = keyv[s] - 1;
    const int line = i / N1, x = i - line * N1, y = line % N2;
    for (int t = lane; t < len; t += 32) pos[j + t] = (uint16_t)(y * pitch + x + t);
}

template <class T> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };

// Load x[k] = line(p0 + k), k < W, with periodic wrap or zero padding; the
// common interior case takes a single base address and constant strides.
template <class T, int W>
__device__ __forceinline__ void load_window(T (&x)[W], const T *in, int ps, int p0, int L, int per)
{
    if (p0 >= 0 && p0 + W <= L) {
        const T *b = in + p0 * ps;
#pragma unroll
        for (int k = 0; k < W; ++k) x[k] = b[k * ps];
    } else if (per) {
#pragma unroll
        for (int k = 0; k < W; ++k) x[k] = in[wrap_near(p0 + k, L) * ps];
    } else {
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int p = p0 + k;
            x[k] = ((unsigned)p < (unsigned)L) ? in[p * ps] : T(0);
        }
    }
}

// Distribute (line, segment) work items over the block: consecutive threads
// take consecutive lines so that x-passes (lanes = rows, odd pitch) and
// y/z-passes (lanes = contiguous columns) are both bank-conflict free.
template <class F>
__device__ __forceinline__ void for_items(int nlines, int nseg, F &&f)
{
    // item it = s * nlines + line, stepped by blockDim with one division per pass
    const int items = nlines * nseg;
    const int bd = blockDim.x;
    int s = threadIdx.x / nlines, line = threadIdx.x - s * nlines;
    const int ds = bd / nlines, dl = bd - ds * nlines;
    for (int it = threadIdx.x; it < items; it += bd) {
        f(line, s);
        line += dl;
        s += ds;
        if (line >= nlines) {
            line -= nlines;
            ++s;
        }
    }
}

// (row, col) of element i = row * cols + col for i = threadIdx.x + k * blockDim.x,
// advanced without a division per element
struct RowCol {
    int r, c, dr, dc, cols;
    __device__ __forceinline__ explicit RowCol(int cols_) : cols(cols_)
    {
        r = threadIdx.x / cols;
        c = threadIdx.x - r * cols;
        dr = blockDim.x / cols;
        dc = blockDim.x - dr * cols;
    }
    __device__ __forceinline__ void next()
    {
        c += dc;
        r += dr;
        if (c >= cols) {
            c -= cols;
            ++r;
        }
    }
};

// for_items over a pass body instantiated twice: FULL = true for segments
// whose outputs all fall inside the line (no per-output bounds test), false
// for the clipped ones; full(line, s) tells which.
template <class Full, class Body>
__device__ __forceinline__ void for_items2(int nlines, int nseg, Full &&full, Body &&body)
{
    for_items(nlines, nseg, [&](int line, int s) {
        if (full(s)) body(line, s, std::true_type{});
        else body(line, s, std::false_type{});
    });
}

struct LineGeom {
    int nlines;
    int src_ls, src_ps;
    int dst_ls, dst_ps;
};

// ---------------------------------------------------------------- synthesis
// src line: [s(0..N-1) | w(0..N-1)], the wavelet half at offset H (N, or
// half_off(N) in the fused planes); dst line: F = fine_len(N,per) values.
template <class T, int SEG>
__device__ __forceinline__ void pass_syn(const T *src, T *dst, const LineGeom g, int N, int H, int per)
{
    static_assert(SEG % 2 == 0, "even segment");
    constexpr int W = SEG / 2 + 8;
    const int F = fine_len(N, per);
    const int off = per ? 0 : 7;      // storage index q = f + off
    const int fstart = per ? 0 : -8;  // even start in Fortran fine coordinates
    const int nseg = (F + off - fstart + SEG - 1) / SEG;
    auto full = [&](int s) {
        const int q0 = fstart + s * SEG + off;
        return q0 >= 0 && q0 + SEG <= F;
    };
    for_items2(g.nlines, nseg, full, [&](int line, int s, auto full_t) {
        constexpr bool FULL = decltype(full_t)::value;
        const T *in = src + line * g.src_ls;
        T *out = dst + line * g.dst_ls;
        const int f0 = fstart + s * SEG;
        const int c0 = f0 / 2;  // f0 is even, so f0/2 is exact (and even)
        T xs[W], xw[W];
        load_window<T, W>(xs, in, g.src_ps, c0 - 4, N, per);
        load_window<T, W>(xw, in + H * g.src_ps, g.src_ps, c0 - 4, N, per);
#pragma unroll
        for (int t = 0; t < SEG; ++t) {
            const int q = f0 + t + off;
            const int o = t & 1;
            const int ic = t / 2 + 4;  // window index of coarse position i0 + t/2
            T acc = T(0);
#pragma unroll
            for (int l = -4; l <= 4; ++l) {
                const int m = 2 * l + o;  // ch_syn(m) = ch(m) for m in [-7,8]
                if (m < -7 || m > 8) continue;
                acc = fma(Filt<T>::ch(m + 7), xs[ic - l], acc);
                acc = fma(Filt<T>::cg(m + 7), xw[ic - l], acc);
            }
            if (FULL || (unsigned)q < (unsigned)F) out[q * g.dst_ps] = acc;
        }
    });
}

// ---------------------------------------------------------------- analysis
// src line: F fine values; dst line: [c(0..N-1) | d(0..N-1)], d at offset H
template <class T, int SEG>
__device__ __forceinline__ void pass_ana(const T *src, T *dst, const LineGeom g, int N, int H, int per)
{
    static_assert(SEG % 2 == 0, "even segment");
    constexpr int HS = SEG / 2;
    constexpr int W = SEG + 14;
    const int F = fine_len(N, per);
    const int nseg = (N + HS - 1) / HS;
    auto full = [&](int s) { return s * HS + HS <= N; };
    for_items2(g.nlines, nseg, full, [&](int line, int s, auto full_t) {
        constexpr bool FULL = decltype(full_t)::value;
        const T *in = src + line * g.src_ls;
        T *out = dst + line * g.dst_ls;
        const int i0 = s * HS;
        T x[W];
        load_window<T, W>(x, in, g.src_ps, 2 * i0 - (per ? 7 : 0), F, per);
#pragma unroll
        for (int t = 0; t < HS; ++t) {
            T ci = T(0), di = T(0);
#pragma unroll
            for (int l = 0; l < 16; ++l) {
                ci = fma(Filt<T>::ch(l), x[2 * t + l], ci);
                di = fma(Filt<T>::cg(l), x[2 * t + l], di);
            }
            const int i = i0 + t;
            if (FULL || i < N) {
                out[i * g.dst_ps] = ci;
                out[(i + H) * g.dst_ps] = di;
            }
        }
    });
}

// ---------------------------------------------------------------- magic filter
// MODE 0: mf periodic, 1: mft periodic, 2: mf grow (F -> F+15), 3: mft shrink (F+15 -> F)
template <class T, int SEG, int MODE>
__device__ __forceinline__ void pass_mf(const T *src, T *dst, const LineGeom g, int Lin, int Lout)
{
    constexpr int W = SEG + 15;
    constexpr int shift = MODE == 0 ? -8 : MODE == 1 ? -7 : MODE == 2 ? -15 : 0;
    constexpr bool rev = (MODE == 1 || MODE == 3);
    constexpr int per = (MODE <= 1);
    const int nseg = (Lout + SEG - 1) / SEG;
    auto full = [&](int s) { return s * SEG + SEG <= Lout; };
    for_items2(g.nlines, nseg, full, [&](int line, int s, auto full_t) {
        constexpr bool FULL = decltype(full_t)::value;
        const T *in = src + line * g.src_ls;
        T *out = dst + line * g.dst_ls;
        const int q0 = s * SEG;
        T x[W];
        load_window<T, W>(x, in, g.src_ps, q0 + shift, Lin, per);
#pragma unroll
        for (int t = 0; t < SEG; ++t) {
            T acc = T(0);
#pragma unroll
            for (int k = 0; k < 16; ++k) acc = fma(Filt<T>::mf(rev ? 15 - k : k), x[t + k], acc);
            const int q = q0 + t;
            if (FULL || q < Lout) out[q * g.dst_ps] = acc;
        }
    });
}

// ---------------------------------------------------------------- kinetic
// dst(q) = cshift * src(q) + scale * sum_l a(|l|) src(q+l) with scale =
// -1/(2h^2) (cshift: the preconditioner's c of (T + c),
// OpenCL/Preconditioner.c:108); ekin += src(q) * scale * conv in FP64
template <class T, int SEG>
__device__ __forceinline__ void pass_kin(const T *src, T *dst, const LineGeom g, int L, int per, double scale_d, T cshift,
                         double *ekin)
{
    constexpr int W = SEG + 28;
    const T scale = (T)scale_d;
    const int nseg = (L + SEG - 1) / SEG;
    double e = 0.0;
    auto full = [&](int s) { return s * SEG + SEG <= L; };
    for_items2(g.nlines, nseg, full, [&](int line, int s, auto full_t) {
        constexpr bool FULL = decltype(full_t)::value;
        const T *in = src + line * g.src_ls;
        T *out = dst + line * g.dst_ls;
        const int q0 = s * SEG;
        T x[W];
        load_window<T, W>(x, in, g.src_ps, q0 - 14, L, per);
        T es = T(0);
#pragma unroll
        for (int t = 0; t < SEG; ++t) {
            T conv = Filt<T>::kin(0) * x[t + 14];
#pragma unroll
            for (int l = 1; l <= 14; ++l) {
                const T pr = x[t + 14 + l] + x[t + 14 - l];
                conv = fma(Filt<T>::kin(l), pr, conv);
            }
            const int q = q0 + t;
            if (FULL || q < L) {
                es = fma(x[t + 14], conv, es);
                out[q * g.dst_ps] = fma(scale, conv, cshift * x[t + 14]);
            }
        }
        e += (double)es * scale_d;
    });
    if (ekin) *ekin += e;
}

// ---------------------------------------------------------------- reductions
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// block-wide sum, result valid in thread 0; red must hold 32 doubles
__device__ __forceinline__ double block_sum(double v, double *red)
{
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (wid == 0) {
        r = (lane < (int)(blockDim.x >> 5)) ? red[lane] : 0.0;
        r = warp_sum(r);
    }
    return r;
}

}  // namespace wvlh
