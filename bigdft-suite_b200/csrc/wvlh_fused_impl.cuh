// Fused, batched local Hamiltonian (Hpsi, E_kin, E_pot), density and
// preconditioner operator for many orbitals and many localisation regions,
// FP32 or FP64.
//
// The reference applies locham to one orbital at a time as 13 full-array
// passes (uncompress, 3x syn, 3x MF, xV, 3x MF^T, 3x kinetic, 3x ana,
// compress: orbitals/daubisf.f90:214-331, locregs/locreg_operations.f90:2502-2937,
// OpenCL/Hamiltonian.c:105-172).  Every 1D operator acts on one axis, and
// synthesis is an isometry per axis with analysis its transpose, so the chain is
//     Hpsi = B^T_x B^T_y B^T_z V B_z B_y B_x psi + (T_x + T_y + T_z) psi
//     B = M S (synthesis, then magic filter), T = A K S (the kinetic operator
//     in the wavelet basis), each one composed pass (wvlh_lines.cuh):
//     D = psi's wavelet plane, Q = B_y B_x D                  (plane kernel K1)
//     Z1 = B^T_z (V . B_z Q) in place of Q, Z2 = T_z D          (z kernel K2)
//     Hpsi = B^T_x B^T_y Z1 + (T_x + T_y) D + Z2              (plane kernel K3)
// so that each kernel keeps a whole xy-plane or a whole z-pencil tile in
// shared memory.  E_pot = sum V r^2 comes from K2; E_kin = <psi | T psi>, its
// z part from K2, the x and y parts from K3.  Energies are reduced in FP64
// into per-CTA partial slots and summed in a fixed order.
//
// The same kernels in MODE_LOCDEN give the density rho += hfac (M^3 S^3 psi)^2
// (OpenCL/Density.c:37-55, sumrho.f90:472-577) through K1 (Q only) and a
// z-kernel that loops over the orbitals sharing a density grid, and in
// MODE_PRECOND the preconditioner operator D^-1/2 A (c + T) S D^-1/2 of
// OpenCL/Preconditioner.c:98-128, which is D^-1/2 (c + T_x + T_y + T_z) D^-1/2
// in the wavelet basis, through K1 (scaled gather, D only), T_z of K2 and K3
// (Z2 + c D + (T_x + T_y) D, scaled scatter).
//
// This file is the implementation shared by the translation units
// wvlh_{locham,locden,precond}_{f32,f64}.cu, each of which instantiates one
// launcher in one precision (they compile in parallel); the common out-of-line
// helpers are compiled in one of them (WVLH_FUSED_COMMON).
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <type_traits>

#include "wvlh_common.cuh"
#include "wvlh_internal.h"
#include "wvlh_lines.cuh"
#include "wvlh_tma.cuh"

namespace wvlh {

constexpr int TX = TX_;
constexpr int TY = TY_;
constexpr int TC = TX * TY;
// alignment of the z kernel's tile buffer (a TMA box destination), and the
// bytes its launches add to the two tile buffers: the block-sum slots and
// the TMA barrier
constexpr int kZAlign = 128;
constexpr int kZExtra = 32 * 8 + 16;

// A wavelet line holds N scaling and N wavelet coefficients.  In global memory
// a wavelet plane is dense, G2 = 2 N2 rows of G1 = 2 N1 points.  In shared
// memory the wavelet half of a row starts at the even offset H1 (rows move as
// point pairs), the rows stay dense: row y of the wavelet half at N2 + y.
struct Dims {
    int N1, N2, N3, p1, p2, p3;
    int H1;               // offset of the wavelet half of a row in shared memory
    int G1, G2, G3, I1, I2, I3;
    int IP1;              // row pitch of the real-space planes Q / Z1 in scratch
    // allper: the batch is known to be periodic in every direction, which lets
    // the compiler drop the free-boundary variants from the kernel
    __device__ __forceinline__ Dims(const LrDev &L, bool allper)
    {
        N1 = L.N[0]; N2 = L.N[1]; N3 = L.N[2];
        p1 = allper ? 1 : L.per[0];
        p2 = allper ? 1 : L.per[1];
        p3 = allper ? 1 : L.per[2];
        H1 = half_off(N1);
        G1 = 2 * N1; G2 = 2 * N2; G3 = 2 * N3;
        I1 = isf_len(N1, p1); I2 = isf_len(N2, p2); I3 = isf_len(N3, p3);
        IP1 = isf_pitch(N1, p1);
    }
    // row pitch of the plane buffers A and B; A holds a real-space plane (I2
    // rows) or a wavelet plane (G2 rows), B G2 rows
    __device__ __forceinline__ int pitch() const { return plane_pitch(N1, p1); }
    __device__ __forceinline__ int rows() const { return max(G2, I2); }
};

// fine component c=1..7 of psi_f -> (s1,s2,s3) bits (wavelib/un-compress.f90:930-936)
__device__ __forceinline__ int fs1(int c) { return c & 1; }
__device__ __forceinline__ int fs2(int c) { return (c >> 1) & 1; }
__device__ __forceinline__ int fs3(int c) { return (c >> 2) & 1; }

// Preconditioner diagonal D^-1/2 per component k = s1 + 2 s2 + 4 s3: GPUscal0..7
// of OpenCL/Uncompress.c:380-470 with h = hgrid/2 (the host passes 0.5*hgrid).
__device__ __forceinline__ double prec_scal(const LrDev &L, double c, int k)
{
    double s = c;
    for (int d = 0; d < 3; ++d) {
        const double h = 0.5 * L.hgrid[d];
        s += (((k >> d) & 1) ? WVL_B2 : WVL_A2) * (0.125 / (h * h));
    }
    return 1.0 / sqrt(s);
}

// The cells of a wavelet z-plane are consecutive in the compressed vector, and
// each has its place in the shared plane in the region's cell table, so
// gathering and scattering walk the plane's values with all lanes busy, no
// segment in sight.  (A warp per segment left a third of the lanes of 48-cell
// rows idle and cost the plane kernels 45 to 50 instructions a point.)  A fine
// cell holds the seven components c = s1 + 2 s2 + 4 s3; a plane takes those of
// its own s3: the three after the coarse coefficient (s3 = 0) or the last four
// (s3 = 1).  Where values are written, consecutive lanes take the components of
// one cell, then the next cell's, so that a warp's store covers 11 or 8
// neighbouring cells.  (One cell a lane put every store on 28 sectors, each
// moved for four bytes: 36 of the 172 us of the preconditioner's K3 on
// 24 x 48^3.)

// value c (its s1, s2 bits) of a cell sits this far from the cell's place
__device__ __forceinline__ int comp_ofs(int c, int H1, int wrow) { return fs1(c) * H1 + fs2(c) * wrow; }

// f(j, place of cell j) for j = j0, j0 + step, ... < end, the places of K cells
// read together: their latency would stand before every copy or store
template <int K, class F>
__device__ __forceinline__ void for_cells(int j0, int end, int step, const uint16_t *__restrict__ pos, F &&f)
{
    for (; j0 < end; j0 += K * step) {
        int at[K];
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (j0 + k * step < end) at[k] = __ldg(pos + j0 + k * step);
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (j0 + k * step < end) f(j0 + k * step, at[k]);
    }
}

// A thread's share of the fine values of a plane of s3 = S3: component c of the
// cells j0, j0 + step, ... (up to two threads of a block stay out when a cell
// gives three values)
template <int S3> struct FineShare {
    static constexpr int NC = S3 ? 4 : 3, C0 = S3 ? 4 : 1;
    int j0, c, step;
    bool in;
    __device__ __forceinline__ FineShare()
    {
        step = blockDim.x / NC;
        j0 = threadIdx.x / NC;
        c = C0 + threadIdx.x - j0 * NC;
        in = j0 < step;
    }
};

struct PlaneCells {
    int a_c, b_c, a_f, b_f;   // the plane's coarse cells (none when s3 = 1), fine cells
    int H1, wrow;             // offsets of the x and y wavelet halves in the shared plane
    __device__ __forceinline__ PlaneCells(const LrDev &L, int pitch, int i3, bool coarse)
    {
        a_c = coarse ? L.plane_c[i3] : 0;
        b_c = coarse ? L.plane_c[i3 + 1] : 0;
        a_f = L.plane_f[i3];
        b_f = L.plane_f[i3 + 1];
        H1 = half_off(L.N[0]);
        wrow = L.N[1] * pitch;
    }
};

// Write the wavelet plane kz into (or add it to) the compressed output at
// [psi_c|psi_f]; sc (8 factors) scales each component when non-null.  The z
// component s3 of a plane is uniform over the CTA: one copy of the component
// loop per s3, so no instruction is issued for the other half.
template <class T, class TO, int S3>
__device__ __forceinline__ void scatter_plane_s(const T *A, int pitch, const LrDev &L, int i3, TO *out, bool accumulate,
                                                const T *sc)
{
    const PlaneCells p(L, pitch, i3, !S3);
    const T s0 = sc ? sc[0] : T(1);
    auto put = [&](TO *dst, T v) { *dst = accumulate ? *dst + (TO)v : (TO)v; };
    for_cells<8>(p.a_c + threadIdx.x, p.b_c, blockDim.x, L.pos_c, [&](int j, int at) { put(out + j, A[at] * s0); });
    const FineShare<S3> w;
    TO *pf = out + L.nvctr_c - 1 + w.c;
    const T *a = A + comp_ofs(w.c, p.H1, p.wrow);
    const T sf = sc ? sc[w.c] : T(1);
    for_cells<8>(p.a_f + w.j0, w.in ? p.b_f : 0, w.step, L.pos_f, [&](int j, int at) { put(pf + 7 * (size_t)j, a[at] * sf); });
}

template <class T, class TO>
__device__ void scatter_plane(const T *A, int pitch, const LrDev &L, int kz, TO *out, bool accumulate, const T *sc)
{
    if (kz >= L.N[2]) scatter_plane_s<T, TO, 1>(A, pitch, L, kz - L.N[2], out, accumulate, sc);
    else scatter_plane_s<T, TO, 0>(A, pitch, L, kz, out, accumulate, sc);
}

// Rows of `cols` points walked as point pairs, every thread on pairs i =
// threadIdx.x + k * blockDim.x of the plane: f(shared offset r * spitch + c,
// global offset r * gpitch + c), c even, advanced without a multiplication.
template <class F>
__device__ __forceinline__ void for_row_pairs(int rows, int cols, int spitch, int gpitch, F &&f)
{
    const int np = cols >> 1, nt = blockDim.x;
    int r = threadIdx.x / np, c = threadIdx.x - r * np;
    const int dr = nt / np, dc = nt - dr * np;
    int so = r * spitch + 2 * c, go = r * gpitch + 2 * c;
    const int ds = dr * spitch + 2 * dc, dg = dr * gpitch + 2 * dc;
    const int ws = spitch - 2 * np, wg = gpitch - 2 * np;   // one row on, from a column past the end
    const int n = rows * np;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += nt) {
        f(so, go);
        c += dc;
        so += ds;
        go += dg;
        if (c >= np) {
            c -= np;
            so += ws;
            go += wg;
        }
    }
}

// a global plane with rows `pitch` points apart can move as point pairs when
// the pitch is even and the plane starts on a pair
template <class T>
__device__ __forceinline__ bool pair_rows(int pitch, const T *g)
{
    return !(pitch & 1) && !(reinterpret_cast<uintptr_t>(g) & (2 * sizeof(T) - 1));
}

template <class T>
__device__ __forceinline__ void zero_region(T *A, int rows, int pitch)
{
    // rows * pitch is even and A starts on a pair
    using V = typename Pair<T>::type;
    V *a = reinterpret_cast<V *>(A);
    V z;
    z.x = T(0);
    z.y = T(0);
    for (int i = threadIdx.x; i < (rows * pitch) >> 1; i += blockDim.x) a[i] = z;
}

// column of a dense wavelet row -> its place in a shared-memory row
__device__ __forceinline__ int wcol(const Dims &d, int c) { return c < d.N1 ? c : c - d.N1 + d.H1; }

// the dense global wavelet plane of shared buffer A (its rows start on pairs:
// G1 is even and so are the scratch offsets)
template <class T>
__device__ __forceinline__ void store_wavelet(const T *A, int pitch, const Dims &d, T *g)
{
    using V = typename Pair<T>::type;
    if (d.N1 & 1) {
        RowCol q(d.G1);
        for (int i = threadIdx.x; i < d.G2 * d.G1; i += blockDim.x, q.next()) g[i] = A[q.r * pitch + wcol(d, q.c)];
        return;
    }
    for_row_pairs(d.G2, d.G1, pitch, d.G1,
                  [&](int so, int go) { *reinterpret_cast<V *>(g + go) = *reinterpret_cast<const V *>(A + so); });
}

// A = scale A + the dense wavelet plane g
template <class T>
__device__ __forceinline__ void scale_add_wavelet(T *A, int pitch, const Dims &d, T scale, const T *__restrict__ g)
{
    if (d.N1 & 1) {
        RowCol q(d.G1);
        for (int i = threadIdx.x; i < d.G2 * d.G1; i += blockDim.x, q.next()) {
            T *a = A + q.r * pitch + wcol(d, q.c);
            *a = fma(scale, *a, g[i]);
        }
        return;
    }
    using V = typename Pair<T>::type;
    for_row_pairs(d.G2, d.G1, pitch, d.G1, [&](int so, int go) {
        const V v = *reinterpret_cast<const V *>(g + go);
        V *a = reinterpret_cast<V *>(A + so);
        V r = *a;
        r.x = fma(scale, r.x, v.x);
        r.y = fma(scale, r.y, v.y);
        *a = r;
    });
}

// Owner of work item `it` when the items are laid out in runs, one run per
// orbital (or density chunk): prefix[0..n] ascending, prefix[0] = 0,
// prefix[n] = total.  Returns the o with prefix[o] <= it < prefix[o+1] by a
// 32-way search, each lane probing one point per round (the table is small
// and read by every CTA, so the probes hit L1).  All 32 lanes of the warp
// must call it.
__device__ __forceinline__ int find_owner(const int *__restrict__ prefix, int n, int it)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) >> 5;
        const int idx = lo + lane * step;
        const bool le = idx < hi && __ldg(prefix + idx) <= it;
        const unsigned m = __ballot_sync(0xffffffffu, le);
        lo += (31 - __clz(m)) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// Asynchronous element copy global -> shared (cp.async, 4 or 8 bytes) with
// zero fill: every thread queues all its copies of a tile before waiting once,
// instead of one dependent load/store pair per element.  When !valid nothing
// is read and the element is set to zero (src is still a valid address).
template <class T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? (int)sizeof(T) : 0;
    if constexpr (sizeof(T) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}
template <class T>
__device__ __forceinline__ void cp_async_one(T *dst, const T *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// point-pair copy global -> shared (8 bytes FP32, 16 bytes FP64), both addresses on a pair
template <class T>
__device__ __forceinline__ void cp_async_pair(T *dst, const T *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// point-pair copy with zero fill: when !valid nothing is read (src must still be
// a valid address) and the pair is set to zero
template <class T>
__device__ __forceinline__ void cp_async_pair_z(T *dst, const T *src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? 2 * (int)sizeof(T) : 0;
    if constexpr (sizeof(T) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// real-space plane Z1 (I2 rows, IP1 apart) into A; the caller waits
template <class T>
__device__ __forceinline__ void load_real_async(T *A, int pitch, const Dims &d, const T *g)
{
    for_row_pairs(d.I2, (d.I1 + 1) & ~1, pitch, d.IP1, [&](int so, int go) { cp_async_pair(A + so, g + go); });
}

// dense wavelet plane into the shared layout, its pad column (odd N1) zero;
// the caller waits.  ASYNC: through cp.async (the buffer is shared memory)
template <class T, bool ASYNC>
__device__ __forceinline__ void load_wavelet(T *B, int pitch, const Dims &d, const T *g)
{
    if (!(d.N1 & 1)) {
        for_row_pairs(d.G2, d.G1, pitch, d.G1, [&](int so, int go) {
            using V = typename Pair<T>::type;
            if (ASYNC) cp_async_pair(B + so, g + go);
            else *reinterpret_cast<V *>(B + so) = *reinterpret_cast<const V *>(g + go);
        });
        return;
    }
    RowCol q(d.G1);
    for (int i = threadIdx.x; i < d.G2 * d.G1; i += blockDim.x, q.next()) {
        T *b = B + q.r * pitch + wcol(d, q.c);
        if (ASYNC) cp_async_elem(b, g + i, true);
        else *b = g[i];
    }
    for (int r = threadIdx.x; r < d.G2; r += blockDim.x) {
        B[r * pitch + d.N1] = T(0);
        B[r * pitch + d.H1 + d.N1] = T(0);
    }
}

// Scatter the compressed coefficients of a wavelet plane (psi at [psi_c|psi_f])
// into buffer A, which must be zero, through cp.async; the caller waits.  Each
// coefficient is one queued copy to its slot of the plane.
template <class T, int S3>
__device__ __forceinline__ void gather_plane_async_s(T *A, int pitch, const LrDev &L, int i3, const T *psi)
{
    const PlaneCells p(L, pitch, i3, !S3);
    for_cells<4>(p.a_c + threadIdx.x, p.b_c, blockDim.x, L.pos_c, [&](int j, int at) { cp_async_one(A + at, psi + j); });
    // a cell a lane here: the copies of a cell's values share its place and hit
    // L1 after the first (values across lanes: K1 0.51 -> 0.55 ms on 128 x 48^3,
    // 0.33 -> 0.36 on 40^3)
    const T *pf = psi + L.nvctr_c;
    for_cells<4>(p.a_f + threadIdx.x, p.b_f, blockDim.x, L.pos_f, [&](int j, int at) {
        const T *src = pf + 7 * (size_t)j;
#pragma unroll
        for (int c = 1; c <= 7; ++c)
            if (fs3(c) == S3) cp_async_one(A + at + comp_ofs(c, p.H1, p.wrow), src + c - 1);
    });
}

template <class T>
__device__ void gather_plane_async(T *A, int pitch, const LrDev &L, int kz, const T *psi)
{
    if (kz >= L.N[2]) gather_plane_async_s<T, 1>(A, pitch, L, kz - L.N[2], psi);
    else gather_plane_async_s<T, 0>(A, pitch, L, kz, psi);
}

template <class TI>
__device__ __forceinline__ const TI *in_ptr(const OrbDev &o, const TI *base)
{
    return o.in_ptr ? (const TI *)o.in_ptr : base + o.psi;
}
template <class TO>
__device__ __forceinline__ TO *out_ptr(const OrbDev &o, TO *base)
{
    return o.out_ptr ? (TO *)o.out_ptr : base + o.psi;
}

// Resident CTAs per SM the plane kernels are compiled for (plane_ctas_per_sm in
// wvlh_internal.h); the persistent variants take what their registers need.
__host__ __device__ constexpr int plane_min_blocks(bool fp32, bool persist, int nt)
{
    return persist ? 1 : plane_ctas_per_sm(fp32, nt);
}

// ---------------------------------------------------------------------------
// CG vectors the preconditioner's plane kernels fold in (MODE_PRECOND): K1
// forms the search direction while it gathers it (dir 1: d = r, the first
// iteration; dir 2: d = beta d + r with beta = rrn / rr, in T), and
// writes d back; K3 accumulates <d | A d> of its plane, into one partial per
// plane (as <D | W> of the scaled plane D = D^-1/2 d that it holds and
// W = (c + T) D).  dir 0 / d null: plain gather / scatter.
template <class T> struct CgIo {
    T *d;
    const T *r;
    const double *rr, *rrn;
    int dir;
};

// The CG direction of wavelet plane kz, formed while it is gathered: every
// coefficient gets v = r (first) or beta d + r, written back to d and into A
// scaled by D^-1/2.  A thread loads d and r of two cells (four coarse values)
// before it stores any: a store to d would hold back the next cell's loads.
template <class T, int S3>
__device__ __forceinline__ void cg_dir_plane_s(T *A, int pitch, const LrDev &L, int i3, T *d, const T *__restrict__ r,
                                               T beta, bool first, const T *sc)
{
    const PlaneCells p(L, pitch, i3, !S3);
    // NC values of each of K cells, a cell's at index idx(j) + c, place at + ofs[c]
    auto run = [&](auto kc, auto nc, int j0, int end, const uint16_t *__restrict__ pos, int stride, T *dv, const T *__restrict__ rv,
                   int c0) {
        constexpr int K = decltype(kc)::value, NC = decltype(nc)::value;
        const int step = blockDim.x;
        for (; j0 < end; j0 += K * step) {
            T v[K][NC];
            int at[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int j = j0 + k * step;
                if (j < end) {
                    at[k] = __ldg(pos + j);
                    const size_t i = (size_t)stride * j;
#pragma unroll
                    for (int c = 0; c < NC; ++c) v[k][c] = first ? rv[i + c] : fma(beta, dv[i + c], rv[i + c]);
                }
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int j = j0 + k * step;
                if (j < end) {
                    const size_t i = (size_t)stride * j;
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        dv[i + c] = v[k][c];
                        A[at[k] + comp_ofs(c0 + c, p.H1, p.wrow)] = v[k][c] * sc[c0 + c];
                    }
                }
            }
        }
    };
    using std::integral_constant;
    run(integral_constant<int, 4>(), integral_constant<int, 1>(), p.a_c + threadIdx.x, p.b_c, L.pos_c, 1, d, r, 0);
    constexpr int NC = S3 ? 4 : 3, C0 = S3 ? 4 : 1;
    run(integral_constant<int, 2>(), integral_constant<int, NC>(), p.a_f + threadIdx.x, p.b_f, L.pos_f, 7,
        d + L.nvctr_c + C0 - 1, r + L.nvctr_c + C0 - 1, C0);
}

// ---------------------------------------------------------------------------
// K1: compressed psi -> D, its wavelet plane (not in MODE_LOCDEN), and
// Q = B_y B_x D (not in MODE_PRECOND) for one wavelet z-plane.
//
// Plane kernels (K1, K3) hold two plane buffers A and B in shared memory.
// When two planes do not fit (FP64 boxes above about 60^3 periodic / 45^3
// free), B lives in gtmp, a global slice of gstride elements per CTA, and the
// grid is one CTA per SM looping over the work items (PERSIST; the slice is
// indexed by blockIdx, so no two running CTAs share it).  Otherwise every CTA
// runs one item.
//
// The x pass walks rows (one thread per row and segment, scalar multiply-adds),
// the y pass columns (two FP32 columns or one FP64 column a thread) and writes
// its outputs straight to global memory: lanes hold neighbouring columns.
template <class T, class TI, bool ALLPER, int MODE>
__device__ __forceinline__ void k1_item(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs,
                                        const int *__restrict__ pre, int norb, const TI *__restrict__ psi,
                                        T *__restrict__ scratch, const double *__restrict__ cprec, int it, T *sc,
                                        T *bslice, const CgIo<T> &cg)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using U = typename ColUnit<T>::U;
    constexpr int kSeg = plane_seg(sizeof(T) == 4);
    static_assert(std::is_same<T, TI>::value, "the gather copies elements as they are");
    {
        const int oi = find_owner(pre, norb, it);   // item = (orbital, wavelet plane kz)
        const int kz = it - pre[oi];
        const OrbDev o = orbs[oi];
        const LrDev L = lrs[o.lr];
        const Dims d(L, ALLPER);
        const int pitch = d.pitch();
        T *A = reinterpret_cast<T *>(smem_raw);
        T *B = bslice ? bslice : A + d.rows() * pitch;

        if (MODE == MODE_PRECOND && threadIdx.x < 8) sc[threadIdx.x] = (T)prec_scal(L, cprec[oi], threadIdx.x);
        zero_region(A, d.G2, pitch);
        __syncthreads();
        if (MODE == MODE_PRECOND && cg.dir) {
            // the CG direction, updated and scaled on the way in
            T *dv = cg.d + o.psi;
            const T *rv = cg.r + o.psi;
            const bool first = cg.dir == 1;
            const T beta = first ? T(0) : (T)(cg.rrn[oi] / cg.rr[oi]);
            if (kz >= d.N3) cg_dir_plane_s<T, 1>(A, pitch, L, kz - d.N3, dv, rv, beta, first, sc);
            else cg_dir_plane_s<T, 0>(A, pitch, L, kz, dv, rv, beta, first, sc);
        } else {
            gather_plane_async<T>(A, pitch, L, kz, in_ptr(o, psi));
            cp_async_wait_all();
            if constexpr (MODE == MODE_PRECOND) {
                // D^-1/2 per component k = s1 + 2 s2 + 4 s3 of each plane position
                __syncthreads();
                const int s3 = kz >= d.N3 ? 4 : 0;
                RowCol q(2 * d.H1);
                for (int i = threadIdx.x; i < d.G2 * 2 * d.H1; i += blockDim.x, q.next())
                    A[q.r * pitch + q.c] *= sc[(q.c >= d.H1 ? 1 : 0) + (q.r >= d.N2 ? 2 : 0) + s3];
            }
        }
        __syncthreads();
        if (MODE != MODE_LOCDEN) store_wavelet(A, pitch, d, scratch + o.sP + (size_t)kz * d.G2 * d.G1);
        if (MODE == MODE_PRECOND) return;
        row_b<T, kSeg>(A, B, d.G2, pitch, d.N1, d.H1, d.p1);   // B_x into B: G2 rows of I1 points
        __syncthreads();
        // B_y: columns of B, G2 -> I2 points, to the Q plane
        T *q = scratch + o.sQ + (size_t)kz * d.I2 * d.IP1;
        const int npair = d.p2 ? d.N2 : d.N2 + 15;
        for_items((d.I1 + U::n - 1) / U::n, (npair + kSeg - 1) / kSeg, [&](int u, int s) {
            const int u0 = s * kSeg;
            typename U::V acc[2 * kSeg];
            col_b<U, kSeg>(acc, B, u * U::n, pitch, d.N2, d.N2, d.p2, u0);
            T *o = q + (size_t)(2 * u0) * d.IP1 + u * U::n;
#pragma unroll
            for (int t = 0; t < 2 * kSeg; ++t)
                if (2 * u0 + t < d.I2) *reinterpret_cast<typename U::V *>(o + t * d.IP1) = acc[t];
        });
    }
}

template <class T, class TI, bool ALLPER, int MODE, bool PERSIST, int NT>
__global__ void __launch_bounds__(NT, plane_min_blocks(sizeof(T) == 4, PERSIST, NT)) k1_plane_forward(const LrDev *__restrict__ lrs,
                                                                  const OrbDev *__restrict__ orbs,
                                                                  const int *__restrict__ pre, int norb,
                                                                  const TI *__restrict__ psi, T *__restrict__ scratch,
                                                                  const double *__restrict__ cprec, T *gtmp,
                                                                  long long gstride, const CgIo<T> cg)
{
    __shared__ T sc[8];
    if (!PERSIST) {
        k1_item<T, TI, ALLPER, MODE>(lrs, orbs, pre, norb, psi, scratch, cprec, blockIdx.x, sc, nullptr, cg);
        return;
    }
    const int nwork = pre[norb];
    for (int it = blockIdx.x; it < nwork; it += gridDim.x) {
        __syncthreads();  // the previous item is done with A, B and sc
        k1_item<T, TI, ALLPER, MODE>(lrs, orbs, pre, norb, psi, scratch, cprec, it, sc,
                                     gtmp + (size_t)blockIdx.x * gstride, cg);
    }
}

// ---------------------------------------------------------------------------
// K2: z-pencil tiles, one kernel instance per chain.  CHAIN 0:
// Z1 = B^T_z (V . B_z Q) in place of Q, E_pot partial.  CHAIN 1: Z2 = T_z D,
// E_kin(z) partial.  CHAIN 2: chain 1 without the energy (the preconditioner's
// operator).
// A tile is TC columns of the plane times the whole z extent, columns side by
// side; a thread takes one column unit (two FP32 columns or one FP64 column)
// of one z segment.  Chain 0 keeps the tile and its real-space form in shared
// memory, chain 1 the tile alone; both write their outputs straight to global
// memory, lanes on neighbouring columns.
// At most NT threads per CTA (256, or for FP32 320 / 384), as many as share the
// tile's segments evenly over its rounds (z_block).  At the FP32 bounds of 256 and
// 384 the compiler gives 80 registers and spills in chain 0 (64 bytes a thread
// periodic, 112 free) and in free chain 1 (16 to 40); at 320 it gives 96 and
// spills up to 16.
__host__ __device__ constexpr int z_min_blocks(bool fp32, int nt) { return fp32 ? (nt > 256 ? 2 : 3) : 2; }

template <class T, class TV, bool ALLPER, int CHAIN>
__device__ __forceinline__ void k2_tile(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs,
                                        const int *__restrict__ pre, int norb, const TV *__restrict__ pot,
                                        T *__restrict__ scratch, double *__restrict__ part_pot,
                                        double *__restrict__ part_kin, int part_stride, const CUtensorMap &tm_in, int tma,
                                        int item)
{
    // dynamic shared memory only (the tile, chain 0's real-space tile, then the
    // reduction slots and the TMA barrier), so that the tile starts the
    // block's shared window
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using U = typename ColUnit<T>::U;
    using V = typename U::V;
    // item = (orbital, tile): chain 0 tiles the I1 x I2 plane of Q, chain 1
    // the G1 x G2 plane of D, row-major; pre is the chain's own prefix table
    constexpr int chain = CHAIN == 2 ? 1 : CHAIN;
    constexpr bool EN = CHAIN != 2;
    constexpr int NU = TC / U::n;       // column units
    const int DS = blockDim.x / NU;     // segments in flight (blockDim.x: whole ones)
    const int oi = find_owner(pre, norb, item);
    const int jj = item - pre[oi];   // tile index, also the energy slot
    const OrbDev o = orbs[oi];
    const LrDev L = lrs[o.lr];
    const Dims d(L, ALLPER);
    const int W = chain == 0 ? d.I1 : d.G1;   // plane width, height and row pitch of the data
    const int H = chain == 0 ? d.I2 : d.G2;
    const int WP = chain == 0 ? d.IP1 : d.G1;
    const int ntx = (W + TX - 1) / TX;
    const int ty = jj / ntx, tx = jj - ty * ntx;
    const int x0 = tx * TX, y0 = ty * TY;
    T *A = reinterpret_cast<T *>(smem_raw);
    T *B = A + d.G3 * TC;
    double *red = reinterpret_cast<double *>(B + (chain == 0 ? d.I3 * TC : 0));
    uint64_t *tma_bar = reinterpret_cast<uint64_t *>(red + 32);
    // TMA writes the tile only into a kZAlign-aligned buffer
    tma = tma && !(smem_addr(A) & (kZAlign - 1));
    const T *g = scratch + (chain == 0 ? o.sQ : o.sP);
    T *gz = scratch + (chain == 0 ? o.sQ : o.sZ);
    const size_t plane = (size_t)WP * H;

    // load the tile: TC columns x G3 z rows, zero outside the plane
    if (tma) {
        // one box {32, 2, G3} of the batch's (x, y, z, orbital) scratch tensor
        if (threadIdx.x == 0) mbar_init(tma_bar, 1);
        __syncthreads();
        if (threadIdx.x == 0) {
            mbar_expect_tx(tma_bar, (unsigned)(TC * d.G3 * sizeof(T)));
            tma_load_4d(A, &tm_in, x0, y0, 0, oi, tma_bar);
        }
        const bool ok = mbar_wait_bounded(tma_bar, 0);
        if (!__syncthreads_and(ok)) {
            // the copy did not complete in time: give it one more bounded wait,
            // then leave NaN in place of the tile's results (what the orbital's
            // Hpsi or CG vectors take) and in its energy slot
            if (threadIdx.x == 0) {
                mbar_wait_bounded(tma_bar, 0);
                if (EN && part_kin)
                    (chain == 0 ? part_pot : part_kin)[(size_t)oi * part_stride + jj] = __longlong_as_double(-1LL);
            }
            __syncthreads();
            for (int i = threadIdx.x; i < TC * d.G3; i += blockDim.x) {
                const int c = i % TC, x = x0 + c % TX, y = y0 + c / TX;
                if (x < W && y < H) gz[(i / TC) * plane + (size_t)y * WP + x] = (T)__longlong_as_double(-1LL);
            }
            return;
        }
    } else {
        // column pairs (x, x + 1) of one tile row: the rows have an even pitch
        // and start on a pair
        constexpr int TP = TC / 2;
        const int ZP = blockDim.x / TP;
        const int pc = 2 * (threadIdx.x % TP);
        const int xp = x0 + (pc % TX), yp = y0 + (pc / TX);
        const bool pin = xp < W && yp < H;
        const T *gp = pin ? g + (size_t)yp * WP + xp : g;
        for (int z = threadIdx.x / TP; z < d.G3; z += ZP)
            cp_async_pair_z(A + z * TC + pc, pin ? gp + (size_t)z * plane : g, pin);
        cp_async_wait_all();
        __syncthreads();
    }
    // this thread's column unit; a pair may hang over the edge of a plane of
    // odd width by the pad column (in1 false), never over the row's pitch
    const int uc = (threadIdx.x % NU) * U::n, sg = threadIdx.x / NU;
    const int xu = x0 + (uc % TX), yu = y0 + (uc / TX);
    const bool in0 = xu < W && yu < H;
    [[maybe_unused]] const bool in1 = in0 && xu + 1 < W;
    gz += in0 ? (size_t)yu * WP + xu : 0;
    double e = 0.0;
    if constexpr (chain == 0) {
        // psir <- V psir, epot += V psir^2 (orbitals/potential.f90:1011-1031);
        // per-thread partial sum in T, one FP64 conversion per thread
        const TV *pv = (o.pot_ptr ? (const TV *)o.pot_ptr : pot + o.pot);
        const bool vpair = pair_rows(W, pv);
        const size_t vplane = (size_t)W * H;
        pv += in0 ? (size_t)yu * W + xu : 0;
        T ep = T(0);
        const int npair = d.p3 ? d.N3 : d.N3 + 15;
        for (int s = sg; s * kSegZ < npair; s += DS) {
            const int z0 = 2 * s * kSegZ;
            // the potential's points are on their way while the filter runs
            V v[2 * kSegZ], acc[2 * kSegZ];
#pragma unroll
            for (int t = 0; t < 2 * kSegZ; ++t) {
                v[t] = U::zero();
                if (z0 + t < d.I3 && in0) {
                    const TV *a = pv + (size_t)(z0 + t) * vplane;
                    if constexpr (U::n == 2) {
                        if (vpair) {
                            v[t] = *reinterpret_cast<const V *>(a);
                        } else {
                            v[t].x = a[0];
                            if (in1) v[t].y = a[1];
                        }
                    } else {
                        v[t] = a[0];
                    }
                }
            }
            col_b<U, kSegZ>(acc, A, uc, TC, d.N3, d.N3, d.p3, s * kSegZ);
            V es = U::zero();
#pragma unroll
            for (int t = 0; t < 2 * kSegZ; ++t) {
                if (z0 + t < d.I3) {
                    const V w = U::mulv(v[t], acc[t]);
                    es = U::fmav(w, acc[t], es);
                    *reinterpret_cast<V *>(B + (z0 + t) * TC + uc) = w;
                }
            }
            // only the plane's own columns count: the pad column of a free row,
            // which the FP64 K1 leaves as the scratch was, may hold anything,
            // and 0 * NaN is NaN
            if (in0) ep += U::n == 1 || in1 ? U::sum(es) : U::first(es);
        }
        e = (double)ep * BInv6<T>::v;
        __syncthreads();
        for (int s = sg; s * kSegZ < d.N3; s += DS) {
            const int i0 = s * kSegZ;
            V c[kSegZ], w[kSegZ];
            col_bt<U, kSegZ>(c, w, B, uc, TC, d.I3, d.p3, i0);
            if (in0) {
#pragma unroll
                for (int t = 0; t < kSegZ; ++t)
                    if (i0 + t < d.N3) {
                        *reinterpret_cast<V *>(gz + (size_t)(i0 + t) * plane) = c[t];
                        *reinterpret_cast<V *>(gz + (size_t)(d.N3 + i0 + t) * plane) = w[t];
                    }
            }
        }
    } else {
        const double scale = -0.5 / (L.hgrid[2] * L.hgrid[2] * TNorm<T>::v);
        for (int s = sg; s * kSegZ < d.N3; s += DS) {
            const int i0 = s * kSegZ;
            V c[kSegZ], w[kSegZ], es = U::zero();
            col_t<U, kSegZ>(c, w, A, uc, TC, d.N3, d.N3, d.p3, i0);
            if (in0) {
#pragma unroll
                for (int t = 0; t < kSegZ; ++t)
                    if (i0 + t < d.N3) {
                        if (EN) {
                            es = U::fmav(c[t], *reinterpret_cast<const V *>(A + (i0 + t) * TC + uc), es);
                            es = U::fmav(w[t], *reinterpret_cast<const V *>(A + (d.N3 + i0 + t) * TC + uc), es);
                        }
                        *reinterpret_cast<V *>(gz + (size_t)(i0 + t) * plane) = U::mul((T)scale, c[t]);
                        *reinterpret_cast<V *>(gz + (size_t)(d.N3 + i0 + t) * plane) = U::mul((T)scale, w[t]);
                    }
                if (EN) e += (double)U::sum(es) * scale;
            }
        }
    }
    if constexpr (EN) {
        const double s = block_sum(e, red);
        if (threadIdx.x == 0 && part_kin)
            (chain == 0 ? part_pot : part_kin)[(size_t)oi * part_stride + jj] = s;
    }
}

template <class T, class TV, bool ALLPER, int CHAIN, int NT = kZThreads>
__global__ void __launch_bounds__(NT, z_min_blocks(sizeof(T) == 4, NT))
    k2_zpencil(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs, const int *__restrict__ pre, int norb,
               const TV *__restrict__ pot, T *__restrict__ scratch, double *__restrict__ part_pot,
               double *__restrict__ part_kin, int part_stride, const __grid_constant__ CUtensorMap tm_in, int tma)
{
    k2_tile<T, TV, ALLPER, CHAIN>(lrs, orbs, pre, norb, pot, scratch, part_pot, part_kin, part_stride, tm_in, tma,
                                  blockIdx.x);
}

// Both chains in one launch, chain 0's n0 tiles first: for calls whose tiles of
// both chains fit the chip at once, where the second launch's latency would
// stand alone (one 32^3 orbital: 64 + 64 tiles on 148 SMs).
template <class T, class TV, bool ALLPER>
__global__ void __launch_bounds__(kZThreads, 2)
    k2_both(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs, const int *__restrict__ pre0,
            const int *__restrict__ pre1, int n0, int norb, const TV *__restrict__ pot, T *__restrict__ scratch,
            double *__restrict__ part_pot, double *__restrict__ part_kin, int part_stride,
            const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_p, int okq, int okp)
{
    if ((int)blockIdx.x < n0)
        k2_tile<T, TV, ALLPER, 0>(lrs, orbs, pre0, norb, pot, scratch, part_pot, part_kin, part_stride, tm_q, okq,
                                  blockIdx.x);
    else
        k2_tile<T, TV, ALLPER, 1>(lrs, orbs, pre1, norb, pot, scratch, part_pot, part_kin, part_stride, tm_p, okp,
                                  blockIdx.x - n0);
}

// ---------------------------------------------------------------------------
// K3 (MODE_LOCHAM): Hpsi plane kz = BInv6 B^T_x B^T_y Z1 + (T_x + T_y) D + Z2
// (the FP32 taps of B are scaled)
// K3 (MODE_PRECOND): D^-1/2 [(c + T_x + T_y) D + Z2]
template <class T, class TO, bool ALLPER, int MODE>
__device__ __forceinline__ void k3_item(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs,
                                        const int *__restrict__ pre, int norb, const T *__restrict__ scratch,
                                        TO *__restrict__ hpsi, double *__restrict__ part_kin, int part_stride,
                                        int accumulate, const double *__restrict__ cprec, int it, T *sc,
                                        double *red, T *bslice, const TO *__restrict__ dotv)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using U = typename ColUnit<T>::U;
    using V = typename U::V;
    constexpr int kSeg = plane_seg(sizeof(T) == 4);
    {
        const int oi = find_owner(pre, norb, it);   // item = (orbital, wavelet plane kz)
        const int kz = it - pre[oi];
        const OrbDev o = orbs[oi];
        const LrDev L = lrs[o.lr];
        const Dims d(L, ALLPER);
        const int pitch = d.pitch();
        T *A = reinterpret_cast<T *>(smem_raw);
        T *B = bslice ? bslice : A + d.rows() * pitch;
        const size_t wofs = (size_t)kz * d.G2 * d.G1;

        T cshift = T(0);
        if (MODE == MODE_PRECOND) {
            cshift = (T)cprec[oi];
            if (threadIdx.x < 8) sc[threadIdx.x] = (T)prec_scal(L, cprec[oi], threadIdx.x);
        } else {
            load_real_async(A, pitch, d, scratch + o.sQ + (size_t)kz * d.I2 * d.IP1);
            cp_async_wait_all();
            __syncthreads();
            // B^T_y: columns of A, I2 -> G2 points, into B
            for_items((d.I1 + U::n - 1) / U::n, (d.N2 + kSeg - 1) / kSeg, [&](int u, int s) {
                const int i0 = s * kSeg;
                V c[kSeg], w[kSeg];
                col_bt<U, kSeg>(c, w, A, u * U::n, pitch, d.I2, d.p2, i0);
                T *b = B + i0 * pitch + u * U::n;
#pragma unroll
                for (int t = 0; t < kSeg; ++t)
                    if (i0 + t < d.N2) {
                        *reinterpret_cast<V *>(b + t * pitch) = c[t];
                        *reinterpret_cast<V *>(b + (d.N2 + t) * pitch) = w[t];
                    }
            });
            __syncthreads();
            row_bt<T, kSeg>(B, A, d.G2, pitch, d.I1, d.N1, d.H1, d.p1);   // B^T_x: I1 -> G1 points, into A
            __syncthreads();
        }
        if (bslice) load_wavelet<T, false>(B, pitch, d, scratch + o.sP + wofs);
        else load_wavelet<T, true>(B, pitch, d, scratch + o.sP + wofs);
        // Z2 into A while D is on its way (in the y pass's epilogue its loads
        // stood at the end of every thread's work: 70 of the kernel's 172 us on
        // 24 x 48^3, where that pass computes for 26)
        const T *z2 = scratch + o.sZ + wofs;
        if (MODE == MODE_PRECOND) load_wavelet<T, true>(A, pitch, d, z2);
        else scale_add_wavelet(A, pitch, d, (T)BInv6<T>::v, z2);
        cp_async_wait_all();
        __syncthreads();
        // e: the kinetic energy partial (MODE_LOCHAM) or <d | A d>
        // (MODE_PRECOND), which with D = D^-1/2 d is <D, W> for the plane
        // W = (c + T) D before its scaling
        constexpr bool EN = MODE != MODE_PRECOND;
        double e = 0.0;
        const double sx = -0.5 / (L.hgrid[0] * L.hgrid[0] * TNorm<T>::v);
        const double sy = -0.5 / (L.hgrid[1] * L.hgrid[1] * TNorm<T>::v);
        row_t<T, kSeg, !EN, EN>(B, A, d.G2, pitch, d.N1, d.H1, d.p1, sx, cshift, &e);   // += T_x D (+ c D)
        __syncthreads();
        // + T_y D, the plane's columns (the pad columns of odd rows are zero in D)
        for_items(2 * d.H1 / U::n, (d.N2 + kSeg - 1) / kSeg, [&](int u, int sg) {
            const int i0 = sg * kSeg, col = u * U::n;
            V s[kSeg], w[kSeg], es = U::zero();
            col_t<U, kSeg>(s, w, B, col, pitch, d.N2, d.N2, d.p2, i0);
            auto put = [&](int row, V conv) {
                V *a = reinterpret_cast<V *>(A + row * pitch + col);
                const V x = *reinterpret_cast<const V *>(B + row * pitch + col);
                const V r = U::fma((T)sy, conv, *a);
                *a = r;
                if (EN) es = U::fmav(x, conv, es);
                else if (dotv) U::dot(e, x, r);
            };
#pragma unroll
            for (int t = 0; t < kSeg; ++t)
                if (i0 + t < d.N2) {
                    put(i0 + t, s[t]);
                    put(d.N2 + i0 + t, w[t]);
                }
            if (EN) e += (double)U::sum(es) * sy;
        });
        __syncthreads();
        scatter_plane<T, TO>(A, pitch, L, kz, out_ptr(o, hpsi), accumulate != 0, MODE == MODE_PRECOND ? sc : nullptr);
        const double s = block_sum(e, red);
        // slots 0 .. ntx1*nty1-1 belong to the z kernel's chain-1 tiles
        const int slot = ((d.G1 + TX - 1) / TX) * ((d.G2 + TY - 1) / TY) + kz;
        if (threadIdx.x == 0 && part_kin) part_kin[(size_t)oi * part_stride + slot] = s;
    }
}

template <class T, class TO, bool ALLPER, int MODE, bool PERSIST, int NT>
__global__ void __launch_bounds__(NT, plane_min_blocks(sizeof(T) == 4, PERSIST, NT)) k3_plane_backward(const LrDev *__restrict__ lrs,
                                                                   const OrbDev *__restrict__ orbs,
                                                                   const int *__restrict__ pre, int norb,
                                                                   const T *__restrict__ scratch, TO *__restrict__ hpsi,
                                                                   double *__restrict__ part_kin, int part_stride,
                                                                   int accumulate, const double *__restrict__ cprec,
                                                                   T *gtmp, long long gstride,
                                                                   const TO *__restrict__ dotv)
{
    __shared__ double red[32];
    __shared__ T sc[8];
    if (!PERSIST) {
        k3_item<T, TO, ALLPER, MODE>(lrs, orbs, pre, norb, scratch, hpsi, part_kin, part_stride, accumulate, cprec,
                                     blockIdx.x, sc, red, nullptr, dotv);
        return;
    }
    const int nwork = pre[norb];
    for (int it = blockIdx.x; it < nwork; it += gridDim.x) {
        __syncthreads();  // the previous item is done with A, B, sc and red
        k3_item<T, TO, ALLPER, MODE>(lrs, orbs, pre, norb, scratch, hpsi, part_kin, part_stride, accumulate, cprec,
                                     it, sc, red, gtmp + (size_t)blockIdx.x * gstride, dotv);
    }
}

// energy slots of an orbital: one per chain-0 tile (potential); one per chain-1
// tile, then one per wavelet plane (kinetic)
__device__ __forceinline__ int pot_slots(const Dims &d) { return ((d.I1 + TX - 1) / TX) * ((d.I2 + TY - 1) / TY); }
__device__ __forceinline__ int plane_slot0(const Dims &d) { return ((d.G1 + TX - 1) / TX) * ((d.G2 + TY - 1) / TY); }

// fixed-order per-orbital sum of the energy partials, over the slots that the
// orbital's tiles and planes write (so nothing has to clear the others first:
// two memsets less in front of every call)
static __global__ void k_reduce_energies(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs,
                                  const double *__restrict__ part_pot, const double *__restrict__ part_kin,
                                  int part_stride, int norb, double *__restrict__ ekin, double *__restrict__ epot)
{
    __shared__ double red[32];
    const int orb = blockIdx.x;
    if (orb >= norb) return;
    const Dims d(lrs[orbs[orb].lr], false);
    const int npot = pot_slots(d), nkin = plane_slot0(d) + d.G3;
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < nkin; i += blockDim.x) a += part_kin[(size_t)orb * part_stride + i];
    for (int i = threadIdx.x; i < npot; i += blockDim.x) b += part_pot[(size_t)orb * part_stride + i];
    const double sa = block_sum(a, red);
    __syncthreads();
    const double sb = block_sum(b, red);
    if (threadIdx.x == 0) {
        if (ekin) ekin[orb] = sa;
        if (epot) epot[orb] = sb;
    }
}

// ---------------------------------------------------------------------------
// Density z-kernel: for a tile of ISF columns, loop over the orbitals of one
// chunk: R = M_z S_z Q, acc += hfac R^2 (FP64), then write the chunk partial.
// Segments of six points: 256 threads then share the 32 column units of a
// 48-cell line's eight segments in one round.
constexpr int kDenSeg = 6;
template <class T, bool ALLPER, int MAXP>
__global__ void __launch_bounds__(kZThreads, MAXP > 32 ? 1 : 2) kd_density(const LrDev *__restrict__ lrs,
                                                        const OrbDev *__restrict__ orbs,
                                                        const int *__restrict__ pre, int nchunk,
                                                        const int *__restrict__ chunk_orb_start,
                                                        const int *__restrict__ chunk_orbs,
                                                        const long long *__restrict__ chunk_part,
                                                        const T *__restrict__ scratch, const double *__restrict__ hfac,
                                                        double *__restrict__ part)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // MAXP accumulators per thread: I3 * TC <= MAXP * kZThreads
    // item = (chunk, tile of the I1 x I2 plane, row-major)
    const int chunk = find_owner(pre, nchunk, blockIdx.x);
    const int j = blockIdx.x - pre[chunk];
    const int ob = chunk_orb_start[chunk], oe = chunk_orb_start[chunk + 1];
    const OrbDev o0 = orbs[chunk_orbs[ob]];
    const LrDev L = lrs[o0.lr];
    const Dims d(L, ALLPER);
    const int ntx = (d.I1 + TX - 1) / TX;
    const int x0 = (j % ntx) * TX, y0 = (j / ntx) * TY;
    T *A = reinterpret_cast<T *>(smem_raw);
    T *B = A + d.G3 * TC;
    const int W = d.I1, H = d.I2;
    using U = typename ColUnit<T>::U;
    constexpr int NU = TC / U::n, DS = kZThreads / NU;
    const size_t plane = (size_t)d.IP1 * H;
    // column pairs as point pairs (even row pitch)
    constexpr int TP = TC / 2, ZP = kZThreads / TP;
    const int pc = 2 * (threadIdx.x % TP);
    const int xp = x0 + (pc % TX), yp = y0 + (pc / TX);
    const bool pin = xp < W && yp < H;
    const size_t pofs = pin ? (size_t)yp * d.IP1 + xp : 0;
    const int uc = (threadIdx.x % NU) * U::n;
    const int npair = d.p3 ? d.N3 : d.N3 + 15;
    double acc[MAXP];
#pragma unroll
    for (int k = 0; k < MAXP; ++k) acc[k] = 0.0;
    for (int oi = ob; oi < oe; ++oi) {
        const int orb = chunk_orbs[oi];
        const OrbDev o = orbs[orb];
        const T *g = scratch + o.sQ;
        __syncthreads();
        for (int z = threadIdx.x / TP; z < d.G3; z += ZP)
            cp_async_pair_z(A + z * TC + pc, g + (pin ? (size_t)z * plane + pofs : 0), pin);
        cp_async_wait_all();
        __syncthreads();
        for (int s = threadIdx.x / NU; s * kDenSeg < npair; s += DS) {
            typename U::V r[2 * kDenSeg];
            col_b<U, kDenSeg>(r, A, uc, TC, d.N3, d.N3, d.p3, s * kDenSeg);
#pragma unroll
            for (int t = 0; t < 2 * kDenSeg; ++t)
                if (2 * s * kDenSeg + t < d.I3) *reinterpret_cast<typename U::V *>(B + (2 * s * kDenSeg + t) * TC + uc) = r[t];
        }
        __syncthreads();
        const double hf = hfac[orb] * BInv6<T>::v;
#pragma unroll
        for (int k = 0; k < MAXP; ++k) {
            const int i = threadIdx.x + k * blockDim.x;
            if (i < d.I3 * TC) {
                const double r = (double)B[i];
                acc[k] = fma(hf * r, r, acc[k]);
            }
        }
    }
    double *out = part + chunk_part[chunk];
#pragma unroll
    for (int k = 0; k < MAXP; ++k) {
        const int i = threadIdx.x + k * blockDim.x;
        if (i < d.I3 * TC) {
            const int z = i / TC, c = i - z * TC;
            const int x = x0 + (c % TX), y = y0 + (c / TX);
            if (x < W && y < H) out[((size_t)z * H + y) * W + x] = acc[k];
        }
    }
}

// rho[group] += sum of the group's chunk partials, in chunk order
static __global__ void k_density_reduce(const int *__restrict__ group_chunk_start, const long long *__restrict__ group_rho,
                                 const int *__restrict__ group_n, const long long *__restrict__ chunk_part,
                                 const double *__restrict__ part, double *__restrict__ rho)
{
    const int g = blockIdx.y;
    const int n = group_n[g];
    const int cb = group_chunk_start[g], ce = group_chunk_start[g + 1];
    // packed batches: offsets into rho; orbital batches: addresses (rho null)
    double *r = rho ? rho + group_rho[g] : reinterpret_cast<double *>(group_rho[g]);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s = r[i];
        for (int c = cb; c < ce; ++c) s += part[chunk_part[c] + i];
        r[i] = s;
    }
}

// ---------------------------------------------------------------------------
// Batched CG vector kernels (OpenCL/Preconditioner.c:130-195 with per-orbital
// scalars kept on the device).  Vectors are [psi_c | psi_f] per orbital at
// off[o], len[o] values; grid.y = orbital, grid.x = chunks of the vector.
// With VEC the values move 16 bytes per access (a scalar head up to the first
// 16-byte boundary of the orbital's range, then groups of 16 bytes, then a
// scalar tail); the launcher takes VEC when every vector of the call starts on
// a 16-byte boundary, so that all of them split alike.  Each thread's terms
// and the block sums come in a fixed order: the reductions are deterministic.
constexpr int kCgChunks = 16;

template <class T> struct alignas(16) Lanes {
    static constexpr int n = 16 / (int)sizeof(T);
    T v[n];
};
template <class T> __device__ __forceinline__ Lanes<T> ldv(const T *p) { return *reinterpret_cast<const Lanes<T> *>(p); }
template <class T> __device__ __forceinline__ void stv(T *p, const Lanes<T> &a) { *reinterpret_cast<Lanes<T> *>(p) = a; }

// e(i) for single values, g(i) for the 16-byte group starting at value i
template <class T, bool VEC, class E1, class EG>
__device__ __forceinline__ void cg_range(const T *p, int n, E1 &&e, EG &&g)
{
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    if constexpr (!VEC) {
        for (int i = tid; i < n; i += nt) e(i);
    } else {
        constexpr int E = Lanes<T>::n;
        const int mis = (int)((reinterpret_cast<uintptr_t>(p) / sizeof(T)) % E);
        int head = mis ? E - mis : 0;
        head = head < n ? head : n;
        const int nv = (n - head) / E, t0 = head + nv * E;
        if (tid < head) e(tid);
        for (int j = tid; j < nv; j += nt) g(head + j * E);
        for (int i = t0 + tid; i < n; i += nt) e(i);
    }
}

// out[o] = sum of its chunk partials (fixed order); optionally copy into hist
static __global__ void k_cg_sum(int norb, const double *__restrict__ part, double *__restrict__ out,
                         double *__restrict__ hist)
{
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= norb) return;
    double s = 0.0;
    for (int c = 0; c < kCgChunks; ++c) s += part[o * kCgChunks + c];
    out[o] = s;
    if (hist) hist[o] = s;
}

// r = b - A x and the chunk partials of <r|r> (the first direction d = r is
// formed by the next K1)
template <class T, bool VEC>
__global__ void k_cg_init(const long long *__restrict__ off, const int *__restrict__ len, const T *__restrict__ b,
                          const T *__restrict__ ax, T *__restrict__ r, double *__restrict__ part)
{
    __shared__ double red[32];
    const int o = blockIdx.y;
    const long long base = off[o];
    const T *bo = b + base, *ao = ax + base;
    T *ro = r + base;
    double s = 0.0;
    cg_range<T, VEC>(
        bo, len[o],
        [&](int i) {
            const T v = bo[i] - ao[i];
            ro[i] = v;
            s += (double)v * (double)v;
        },
        [&](int i) {
            Lanes<T> v = ldv(bo + i);
            const Lanes<T> a = ldv(ao + i);
#pragma unroll
            for (int k = 0; k < Lanes<T>::n; ++k) {
                v.v[k] -= a.v[k];
                s += (double)v.v[k] * (double)v.v[k];
            }
            stv(ro + i, v);
        });
    const double t = block_sum(s, red);
    if (threadIdx.x == 0) part[o * kCgChunks + blockIdx.x] = t;
}

// alpha = rr / dAd; x += alpha d, r -= alpha A d, and the chunk partials of
// the new <r|r>
template <class T, bool VEC>
__global__ void k_cg_step(const long long *__restrict__ off, const int *__restrict__ len,
                          const double *__restrict__ rr, const double *__restrict__ dad, T *__restrict__ x,
                          const T *__restrict__ d, T *__restrict__ r, const T *__restrict__ ad,
                          double *__restrict__ part)
{
    __shared__ double red[32];
    const int o = blockIdx.y;
    const long long base = off[o];
    T *xo = x + base, *ro = r + base;
    const T *dn = d + base, *ao = ad + base;
    const T alpha = (T)(rr[o] / dad[o]);
    double s = 0.0;
    cg_range<T, VEC>(
        xo, len[o],
        [&](int i) {
            xo[i] = fma(alpha, dn[i], xo[i]);
            const T v = fma(-alpha, ao[i], ro[i]);
            ro[i] = v;
            s += (double)v * (double)v;
        },
        [&](int i) {
            Lanes<T> xv = ldv(xo + i), rv = ldv(ro + i);
            const Lanes<T> dv = ldv(dn + i), av = ldv(ao + i);
#pragma unroll
            for (int k = 0; k < Lanes<T>::n; ++k) {
                xv.v[k] = fma(alpha, dv.v[k], xv.v[k]);
                rv.v[k] = fma(-alpha, av.v[k], rv.v[k]);
                s += (double)rv.v[k] * (double)rv.v[k];
            }
            stv(xo + i, xv);
            stv(ro + i, rv);
        });
    const double t = block_sum(s, red);
    if (threadIdx.x == 0) part[o * kCgChunks + blockIdx.x] = t;
}

static __global__ void k_copy_scalars(int n, const double *__restrict__ a, double *__restrict__ b)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[i];
}

// x *= D^-1/2 per component (scale_psi_d, OpenCL/Uncompress.c:596): value i
// is coarse below nvctr_c, else fine component 1 + (i - nvctr_c) % 7
template <class T, bool VEC>
__global__ void k_cg_scale(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs,
                           const long long *__restrict__ off, const int *__restrict__ len,
                           const double *__restrict__ cprec, T *__restrict__ x)
{
    const int o = blockIdx.y;
    const OrbDev ob = orbs[o];
    const LrDev L = lrs[ob.lr];
    T sc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) sc[k] = (T)prec_scal(L, cprec[o], k);
    T *xo = x + off[o];
    const int nc = L.nvctr_c;
    auto comp = [&](int i) { return i < nc ? 0 : 1 + (i - nc) % 7; };
    cg_range<T, VEC>(
        xo, len[o], [&](int i) { xo[i] *= sc[comp(i)]; },
        [&](int i) {
            Lanes<T> v = ldv(xo + i);
            int k = comp(i);
#pragma unroll
            for (int j = 0; j < Lanes<T>::n; ++j) {
                v.v[j] *= sc[k];
                // the next value's component: coarse until nvctr_c, then 1..7 cyclically
                k = (i + j + 1 < nc) ? 0 : (k == 0 || k == 7 ? 1 : k + 1);
            }
            stv(xo + i, v);
        });
}

// ---------------------------------------------------------------------------
// host launchers

// Launch shape of the plane kernels: two shared-memory planes when they fit,
// else one shared plane + a global slice per CTA after the batch scratch.
static int sm_count()
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

struct PlaneCfg {
    size_t smem = 0;
    int grid = 0;
    int threads = kPlaneThreads;
    long long gstride = 0;
    bool global_b = false;
};

static PlaneCfg plane_cfg(const Plan &p, int fp, int nwork)
{
    int dev = 0, lim = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    PlaneCfg c;
    c.global_b = p.smem13[fp] > (size_t)lim - 1024;
    c.smem = c.global_b ? (size_t)p.plane_elems * (fp ? 8 : 4) : p.smem13[fp];
    c.grid = c.global_b ? (nwork < nsm ? nwork : nsm) : nwork;
    c.gstride = c.global_b ? p.planeB_elems : 0;
    c.threads = c.global_b ? kPlaneThreads : p.plane_threads[fp];
    return c;
}

// the variant compiled for the smallest size that takes pc.threads
template <class T, class TI, bool ALLPER, int MODE>
static auto k1_for(const PlaneCfg &pc) -> decltype(&k1_plane_forward<T, TI, ALLPER, MODE, true, kPlaneThreads>)
{
    if (pc.global_b) return k1_plane_forward<T, TI, ALLPER, MODE, true, kPlaneThreads>;
    if (pc.threads <= kPlaneSizes[4]) return k1_plane_forward<T, TI, ALLPER, MODE, false, kPlaneSizes[4]>;
    if (pc.threads <= kPlaneSizes[3]) return k1_plane_forward<T, TI, ALLPER, MODE, false, kPlaneSizes[3]>;
    if (pc.threads <= kPlaneSizes[2]) return k1_plane_forward<T, TI, ALLPER, MODE, false, kPlaneSizes[2]>;
    if (pc.threads <= kPlaneSizes[1]) return k1_plane_forward<T, TI, ALLPER, MODE, false, kPlaneSizes[1]>;
    return k1_plane_forward<T, TI, ALLPER, MODE, false, kPlaneSizes[0]>;
}

template <class T, class TO, bool ALLPER, int MODE>
static auto k3_for(const PlaneCfg &pc) -> decltype(&k3_plane_backward<T, TO, ALLPER, MODE, true, kPlaneThreads>)
{
    if (pc.global_b) return k3_plane_backward<T, TO, ALLPER, MODE, true, kPlaneThreads>;
    if (pc.threads <= kPlaneSizes[4]) return k3_plane_backward<T, TO, ALLPER, MODE, false, kPlaneSizes[4]>;
    if (pc.threads <= kPlaneSizes[3]) return k3_plane_backward<T, TO, ALLPER, MODE, false, kPlaneSizes[3]>;
    if (pc.threads <= kPlaneSizes[2]) return k3_plane_backward<T, TO, ALLPER, MODE, false, kPlaneSizes[2]>;
    if (pc.threads <= kPlaneSizes[1]) return k3_plane_backward<T, TO, ALLPER, MODE, false, kPlaneSizes[1]>;
    return k3_plane_backward<T, TO, ALLPER, MODE, false, kPlaneSizes[0]>;
}

// TMA maps of the z kernel's tiles: when every orbital of the batch lies in
// one region, the scratch planes of all orbitals form regular 4-D tensors
// (x, y, z, orbital) for Q (chain 0) and D (chain 1); otherwise (several
// regions, or rows whose byte length TMA cannot stride) the tiles move with
// cp.async.
struct ZMaps {
    CUtensorMap q, p;
    int okq = 0, okp = 0;
};
template <class T>
static void zmaps(const Plan &p, T *scratch, ZMaps &m)
{
    memset(&m, 0, sizeof(m));
    if (p.orb_scratch <= 0) return;
    const int es = (int)sizeof(T);
    const TileDims &t = p.tile;
    m.okq = encode_tile_map(&m.q, scratch + t.ofs_q, es, t.I1, t.IP1, t.I2, t.G3, p.norb, p.orb_scratch);
    m.okp = encode_tile_map(&m.p, scratch, es, t.G1, t.G1, t.G2, t.G3, p.norb, p.orb_scratch);
}

// K1 / K3 launch with the plane configuration of the batch
template <class T, class TI, bool ALLPER, int MODE>
static cudaError_t run_k1(const Plan &p, const PlaneCfg &pc, const TI *psi, T *scratch, const double *cprec, T *gtmp,
                          cudaStream_t st, CgIo<T> cg = CgIo<T>{nullptr, nullptr, nullptr, nullptr, 0})
{
    cudaError_t err;
    auto k = k1_for<T, TI, ALLPER, MODE>(pc);
    if ((err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pc.smem))) return err;
    k<<<pc.grid, pc.threads, pc.smem, st>>>(p.d_lr, p.d_orb, p.d_pre13, p.norb, psi, scratch, cprec, gtmp, pc.gstride,
                                            cg);
    return cudaSuccess;
}

template <class T, class TO, bool ALLPER, int MODE>
static cudaError_t run_k3(const Plan &p, const PlaneCfg &pc, const T *scratch, TO *out, double *part_kin,
                          int part_stride, int accumulate, const double *cprec, T *gtmp, cudaStream_t st,
                          const TO *dotv = nullptr)
{
    cudaError_t err;
    auto k = k3_for<T, TO, ALLPER, MODE>(pc);
    if ((err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pc.smem))) return err;
    k<<<pc.grid, pc.threads, pc.smem, st>>>(p.d_lr, p.d_orb, p.d_pre13, p.norb, scratch, out, part_kin, part_stride,
                                            accumulate, cprec, gtmp, pc.gstride, dotv);
    return cudaSuccess;
}

// threads of a z-kernel CTA compiled for nt: the tile's segments (its longest
// line's) in equal rounds
static int z_block(bool fp32, int segs, int nt)
{
    const int nu = TC / (fp32 ? 2 : 1), most = nt / nu, rounds = (segs + most - 1) / most;
    return rounds > 0 ? nu * ((segs + rounds - 1) / rounds) : nt;
}

// K2 launch with the kernel compiled for zt threads (FP32: 256, 320 or 384; FP64: 256)
template <class T, class TV, bool ALLPER, int CHAIN>
static cudaError_t run_k2(int zt, int nwork, size_t sm2, const Plan &p, const int *pre, const TV *pot, T *scratch,
                          double *part_pot, double *part_kin, int part_stride, const CUtensorMap &m_in, int tma,
                          cudaStream_t st)
{
    auto k = k2_zpencil<T, TV, ALLPER, CHAIN, kZThreads>;
    if constexpr (sizeof(T) == 4) {
        if (zt == 320) k = k2_zpencil<T, TV, ALLPER, CHAIN, 320>;
        else if (zt == 384) k = k2_zpencil<T, TV, ALLPER, CHAIN, 384>;
        else zt = kZThreads;
    } else {
        zt = kZThreads;
    }
    zt = z_block(sizeof(T) == 4, CHAIN == 0 ? p.z_segs0 : p.z_segs1, zt);
    cudaError_t err;
    if ((err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2))) return err;
    k<<<nwork, zt, sm2, st>>>(p.d_lr, p.d_orb, pre, p.norb, pot, scratch, part_pot, part_kin, part_stride, m_in,
                              tma);
    return cudaSuccess;
}

#ifdef WVLH_FUSED_COMMON
long long plane_tmp_elems(const Plan &p, int fp)
{
    int dev = 0, lim = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return p.smem13[fp] > (size_t)lim - 1024 ? (long long)nsm * p.planeB_elems : 0;
}
#endif
template <class T, class TIO, bool ALLPER>
static cudaError_t launch_locham_bc(const Plan &p, const TIO *psi, const TIO *pot, TIO *hpsi, T *scratch,
                                    double *part_pot, double *part_kin, double *ekin, double *epot, int accumulate,
                                    cudaStream_t st, cudaEvent_t *ev)
{
    const int fp = sizeof(T) == 8 ? 1 : 0;
    const PlaneCfg pc = plane_cfg(p, fp, p.n_work13);
    const size_t sm2 = p.smem_z0[fp] + kZExtra, sm2p = p.smem_z1[fp] + kZExtra;
    T *gtmp = pc.global_b ? scratch + p.scratch_elems : nullptr;
    cudaError_t err;
    ZMaps zm;
    zmaps(p, scratch, zm);
    // optional per-kernel timing: ev[0..4] bracket K1, K2, K3 and the reduction
    if (ev) cudaEventRecord(ev[0], st);
    if ((err = run_k1<T, TIO, ALLPER, MODE_LOCHAM>(p, pc, psi, scratch, nullptr, gtmp, st))) return err;
    if (ev) cudaEventRecord(ev[1], st);
    // both chains' tiles in one wave (two CTAs an SM, as k2_both is compiled and
    // FP64 tiles of 64 cells fit): one launch for the two
    if (p.n_work2 + p.n_work2p <= 2 * sm_count() && 2 * (sm2 + 1024) <= (size_t)227 * 1024) {
        auto k = k2_both<T, TIO, ALLPER>;
        if ((err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2))) return err;
        k<<<p.n_work2 + p.n_work2p, z_block(sizeof(T) == 4, p.z_segs0, kZThreads), sm2, st>>>(
            p.d_lr, p.d_orb, p.d_pre2, p.d_pre2p, p.n_work2, p.norb, pot, scratch, part_pot, part_kin, p.part_stride,
            zm.q, zm.p, zm.okq, zm.okp);
    } else if ((err = run_k2<T, TIO, ALLPER, 0>(p.z_threads[fp], p.n_work2, sm2, p, p.d_pre2, pot, scratch, part_pot,
                                                part_kin, p.part_stride, zm.q, zm.okq, st)) ||
               (err = run_k2<T, TIO, ALLPER, 1>(p.z_threads[fp], p.n_work2p, sm2p, p, p.d_pre2p, pot, scratch,
                                                part_pot, part_kin, p.part_stride, zm.p, zm.okp, st))) {
        return err;
    }
    if (ev) cudaEventRecord(ev[2], st);
    if ((err = run_k3<T, TIO, ALLPER, MODE_LOCHAM>(p, pc, scratch, hpsi, part_kin, p.part_stride, accumulate, nullptr,
                                                   gtmp, st)))
        return err;
    if (ev) cudaEventRecord(ev[3], st);
    k_reduce_energies<<<p.norb, 128, 0, st>>>(p.d_lr, p.d_orb, part_pot, part_kin, p.part_stride, p.norb, ekin, epot);
    if (ev) cudaEventRecord(ev[4], st);
    return cudaGetLastError();
}

template <class T, class TIO>
cudaError_t launch_locham(const Plan &p, const TIO *psi, const TIO *pot, TIO *hpsi, T *scratch, double *part_pot,
                          double *part_kin, double *ekin, double *epot, int accumulate, cudaStream_t st,
                          cudaEvent_t *ev)
{
    if (p.all_periodic)
        return launch_locham_bc<T, TIO, true>(p, psi, pot, hpsi, scratch, part_pot, part_kin, ekin, epot,
                                              accumulate, st, ev);
    return launch_locham_bc<T, TIO, false>(p, psi, pot, hpsi, scratch, part_pot, part_kin, ekin, epot, accumulate,
                                           st, ev);
}

#if defined(WVLH_FUSED_F32) && defined(WVLH_FUSED_LOCHAM)
template cudaError_t launch_locham<float, float>(const Plan &, const float *, const float *, float *, float *,
                                                 double *, double *, double *, double *, int, cudaStream_t,
                                                 cudaEvent_t *);
#endif
#if defined(WVLH_FUSED_F64) && defined(WVLH_FUSED_LOCHAM)
template cudaError_t launch_locham<double, double>(const Plan &, const double *, const double *, double *, double *,
                                                   double *, double *, double *, double *, int, cudaStream_t,
                                                   cudaEvent_t *);
#endif

template <class T, bool ALLPER>
static cudaError_t launch_locden_bc(const Plan &p, const T *psi, const double *hfac, double *rho, T *scratch,
                                    double *part, cudaStream_t st)
{
    const int fp = sizeof(T) == 8 ? 1 : 0;
    const PlaneCfg pc = plane_cfg(p, fp, p.n_work13);
    const size_t sm2 = p.smem_z0[fp] + kZExtra;
    T *gtmp = pc.global_b ? scratch + p.scratch_elems : nullptr;
    cudaError_t err;
    auto kd = p.den_acc > 32 ? kd_density<T, ALLPER, 48> : kd_density<T, ALLPER, 32>;
    if ((err = cudaFuncSetAttribute(kd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2))) return err;
    if ((err = run_k1<T, T, ALLPER, MODE_LOCDEN>(p, pc, psi, scratch, nullptr, gtmp, st))) return err;
    kd<<<p.n_workd, kZThreads, sm2, st>>>(p.d_lr, p.d_orb, p.d_pred, p.nchunk, p.d_chunk_orb_start, p.d_chunk_orbs,
                                          p.d_chunk_part, scratch, hfac, part);
    dim3 g((p.max_group_n + 255) / 256 < 4096 ? (p.max_group_n + 255) / 256 : 4096, p.ngroup);
    k_density_reduce<<<g, 256, 0, st>>>(p.d_group_chunk_start, p.d_group_rho, p.d_group_n, p.d_chunk_part, part,
                                        rho);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_locden(const Plan &p, const T *psi, const double *hfac, double *rho, T *scratch, double *part,
                          cudaStream_t st)
{
    if (p.all_periodic) return launch_locden_bc<T, true>(p, psi, hfac, rho, scratch, part, st);
    return launch_locden_bc<T, false>(p, psi, hfac, rho, scratch, part, st);
}
#if defined(WVLH_FUSED_F32) && defined(WVLH_FUSED_LOCDEN)
template cudaError_t launch_locden<float>(const Plan &, const float *, const double *, double *, float *, double *,
                                          cudaStream_t);
#endif
#if defined(WVLH_FUSED_F64) && defined(WVLH_FUSED_LOCDEN)
template cudaError_t launch_locden<double>(const Plan &, const double *, const double *, double *, double *,
                                           double *, cudaStream_t);
#endif

// preconditioner operator y = D^-1/2 A (c + T) S D^-1/2 x for every orbital;
// cg.dir: x is the CG direction, formed by K1 (see CgIo); dotpart: K3's
// partials of <x | y> per plane, or null
template <class T, bool ALLPER>
static cudaError_t launch_prec_apply_bc(const Plan &p, const T *x, T *y, const double *cprec, T *scratch,
                                        cudaStream_t st, const CgIo<T> &cg, double *dotpart)
{
    const int fp = sizeof(T) == 8 ? 1 : 0;
    PlaneCfg pc = plane_cfg(p, fp, p.n_work13);
    if (!pc.global_b) pc.threads = p.plane_threads_pre[fp];
    const size_t sm2 = p.smem_z1[fp] + kZExtra;
    T *gtmp = pc.global_b ? scratch + p.scratch_elems : nullptr;
    cudaError_t err;
    if ((err = run_k1<T, T, ALLPER, MODE_PRECOND>(p, pc, x, scratch, cprec, gtmp, st, cg))) return err;
    ZMaps zm;
    zmaps(p, scratch, zm);
    if ((err = run_k2<T, T, ALLPER, 2>(p.z_threads_pre[fp], p.n_work2p, sm2, p, p.d_pre2p, (const T *)nullptr, scratch,
                                       nullptr, nullptr, 0, zm.p, zm.okp, st)))
        return err;
    if ((err = run_k3<T, T, ALLPER, MODE_PRECOND>(p, pc, scratch, y, dotpart, dotpart ? p.part_stride : 0, 0, cprec,
                                                  gtmp, st, dotpart ? x : nullptr)))
        return err;
    return cudaGetLastError();
}

// out[o] = the sum of orbital o's plane partials (K3's slots): one warp per
// orbital, lane l summing planes l, l + 32, ... then a fixed shuffle tree
// (deterministic)
static __global__ void k_cg_sum_slots(const LrDev *__restrict__ lrs, const OrbDev *__restrict__ orbs, int norb,
                                      const double *__restrict__ part, int stride, double *__restrict__ out)
{
    const int o = blockIdx.x;
    if (o >= norb) return;
    const Dims d(lrs[orbs[o].lr], false);
    const int k0 = plane_slot0(d);
    double s = 0.0;
    for (int k = threadIdx.x; k < d.G3; k += 32) s += part[(size_t)o * stride + k0 + k];
    s = warp_sum(s);
    if (threadIdx.x == 0) out[o] = s;
}

static bool aligned16(const void *p) { return !(reinterpret_cast<uintptr_t>(p) & 15); }

// The recurrence of Preconditioner.c:130-195 with two of its vector passes
// folded into the operator's kernels: K1 forms the direction
// d = r / d = beta d + r while gathering it, K3 accumulates <d | A d> while
// scattering A d.  Per iteration: apply (K1, K2, K3), alpha = rr / dAd, the
// x and r updates with the new <r|r> (k_cg_step), then rr <- rr_new once
// the next K1 has read both.
template <class T, bool VEC, class Apply>
static cudaError_t cg_loop(const Plan &p, int ncong, const double *cprec, T *x, const T *b, T *r, T *dvec, T *ad,
                           double *rr, double *dad, double *rrn, double *part, double *dotpart, double *hist,
                           Apply &&apply, cudaStream_t st)
{
    const dim3 vg(kCgChunks, p.norb);
    const int sg = (p.norb + 127) / 128;
    cudaError_t err;
    if ((err = apply(x, ad, CgIo<T>{nullptr, nullptr, nullptr, nullptr, 0}, nullptr))) return err;
    k_cg_init<T, VEC><<<vg, 256, 0, st>>>(p.d_orb_off, p.d_orb_len, b, ad, r, part);
    k_cg_sum<<<sg, 128, 0, st>>>(p.norb, part, rr, hist);
    for (int it = 0; it < ncong; ++it) {
        if ((err = apply(dvec, ad, CgIo<T>{dvec, r, rr, rrn, it == 0 ? 1 : 2}, dotpart))) return err;
        if (it > 0) k_copy_scalars<<<sg, 128, 0, st>>>(p.norb, rrn, rr);
        k_cg_sum_slots<<<p.norb, 32, 0, st>>>(p.d_lr, p.d_orb, p.norb, dotpart, p.part_stride, dad);
        k_cg_step<T, VEC><<<vg, 256, 0, st>>>(p.d_orb_off, p.d_orb_len, rr, dad, x, dvec, r, ad, part);
        k_cg_sum<<<sg, 128, 0, st>>>(p.norb, part, rrn, hist ? hist + (size_t)(it + 1) * p.norb : nullptr);
    }
    k_cg_scale<T, VEC><<<vg, 256, 0, st>>>(p.d_lr, p.d_orb, p.d_orb_off, p.d_orb_len, cprec, x);
    return cudaGetLastError();
}

// Batched CG of ocl_preconditioner_generic: x (in: initial guess, out:
// preconditioned), b right-hand side; work: r, d, ad vectors; scal:
// (5 + kCgChunks + part_stride) * norb doubles (scalars, chunk partials of
// the vector kernels, K3's per-plane partials of <d|Ad>); hist (optional):
// (ncong+1)*norb squared residual norms, entry 0 the initial one.
template <class T>
cudaError_t launch_precond(const Plan &p, int ncong, const double *cprec, T *x, const T *b, T *r, T *dvec, T *ad,
                           T *scratch, double *scal, double *hist, cudaStream_t st)
{
    double *rr = scal, *dad = scal + p.norb, *rrn = scal + 2 * p.norb, *part = scal + 5 * p.norb;
    double *dotpart = part + (size_t)kCgChunks * p.norb;
    auto apply = [&](const T *in, T *out, const CgIo<T> &cg, double *dp) {
        return p.all_periodic ? launch_prec_apply_bc<T, true>(p, in, out, cprec, scratch, st, cg, dp)
                              : launch_prec_apply_bc<T, false>(p, in, out, cprec, scratch, st, cg, dp);
    };
    const bool vec = aligned16(x) && aligned16(b) && aligned16(r) && aligned16(dvec) && aligned16(ad);
    return vec ? cg_loop<T, true>(p, ncong, cprec, x, b, r, dvec, ad, rr, dad, rrn, part, dotpart, hist, apply, st)
               : cg_loop<T, false>(p, ncong, cprec, x, b, r, dvec, ad, rr, dad, rrn, part, dotpart, hist, apply, st);
}
#if defined(WVLH_FUSED_F32) && defined(WVLH_FUSED_PRECOND)
template cudaError_t launch_precond<float>(const Plan &, int, const double *, float *, const float *, float *, float *,
                                           float *, float *, double *, double *, cudaStream_t);
#endif
#if defined(WVLH_FUSED_F64) && defined(WVLH_FUSED_PRECOND)
template cudaError_t launch_precond<double>(const Plan &, int, const double *, double *, const double *, double *,
                                            double *, double *, double *, double *, double *, cudaStream_t);
#endif

#ifdef WVLH_FUSED_COMMON
// FP32/FP64 FMA throughput probe: independent FMA chains held in registers.
template <class T>
__global__ void __launch_bounds__(256) k_fma_probe(T *out, int iters, T a, T b)
{
    T x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = T(threadIdx.x + k) * T(1e-3);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = fma(x[k], a, b);
    }
    T s = T(0);
#pragma unroll
    for (int k = 0; k < 16; ++k) s += x[k];
    if (s == T(12345.678)) out[blockIdx.x] = s;  // keep the chains alive
}

cudaError_t fma_probe(int precision, int iters, float *ms, double *flops, cudaStream_t st)
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int blocks = nsm * 8;
    void *buf = nullptr;
    cudaError_t e = cudaMalloc(&buf, 8 * (size_t)blocks);
    if (e) return e;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    for (int rep = 0; rep < 2; ++rep) {  // first launch warms up
        cudaEventRecord(a, st);
        if (precision == 64) k_fma_probe<double><<<blocks, 256, 0, st>>>((double *)buf, iters, 0.999999, 1e-7);
        else k_fma_probe<float><<<blocks, 256, 0, st>>>((float *)buf, iters, 0.999999f, 1e-7f);
        cudaEventRecord(b, st);
    }
    cudaEventSynchronize(b);
    cudaEventElapsedTime(ms, a, b);
    *flops = 2.0 * 16.0 * (double)iters * 256.0 * blocks;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(buf);
    return cudaGetLastError();
}

#endif

}  // namespace wvlh
