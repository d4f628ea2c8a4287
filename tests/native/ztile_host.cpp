// Host build of the z kernel's tile (wvlh_fused_impl.cuh up to its host
// launchers, as ztile.cuh) with a TMA whose waits run out (the test's own
// wvlh_tma.cuh).  On that path the threads of a block do nothing together, so
// they run one after the other.
#include <cuda_runtime.h>

#undef __device__
#undef __host__
#undef __forceinline__
#undef __global__
#undef __shared__
#undef __launch_bounds__
#undef __grid_constant__
#define __device__
#define __host__
#define __forceinline__ inline
#define __global__
#define __shared__
#define __launch_bounds__(...)
#define __grid_constant__

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

using std::max;
using std::min;
static struct { int x, y; } threadIdx, blockDim, blockIdx, gridDim;
static void __syncthreads() {}
static int __syncthreads_and(int v) { return v; }
static unsigned __ballot_sync(unsigned, bool) { return 1; }
static int __clz(unsigned) { return 31; }
template <class T> static T __ldg(const T *p) { return *p; }
static size_t __cvta_generic_to_shared(const void *) { return 0; }
static double __longlong_as_double(long long v)
{
    double d;
    memcpy(&d, &v, sizeof d);
    return d;
}
template <class T> static T __shfl_xor_sync(unsigned, T v, int) { return v; }
static unsigned __viaddmin_u32(unsigned a, unsigned b, unsigned c) { return std::min(a + b, c); }
static float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)}; }
static float2 __fmul2_rn(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }

// inline PTX drops out: asm volatile(...) -> ;
#define asm
#define volatile(...)
#include "ztile.cuh"
#undef asm
#undef volatile

namespace wvlh {
unsigned char smem_raw[1 << 20];
}
using namespace wvlh;

// One tile of a free box's orbital whose copy does not arrive: 0 when the
// results of the tile's columns are NaN, all else is as it was, and the energy
// slot (chains 0 and 1) is NaN.
template <class T, int CHAIN> static int timed_out(const int *N, int tile)
{
    LrDev L{};
    for (int k = 0; k < 3; ++k) {
        L.N[k] = N[k];
        L.hgrid[k] = 0.4;
    }
    const Dims d(L, false);
    const OrbScratch sc = orb_scratch(L.N, L.per);
    OrbDev o{};
    o.sZ = sc.z;
    o.sQ = sc.q;
    std::vector<T> scratch(sc.total, T(1)), pot((size_t)d.I1 * d.I2 * d.I3, T(1));
    const int W = CHAIN ? d.G1 : d.I1, H = CHAIN ? d.G2 : d.I2, WP = CHAIN ? d.G1 : d.IP1;
    const int ntx = (W + TX - 1) / TX, ntile = ntx * ((H + TY - 1) / TY), pre[2] = {0, ntile};
    std::vector<double> ep(ntile, 1.0), ek(ntile, 1.0);
    const bool en = CHAIN != 2;
    blockDim.x = kZThreads;
    for (threadIdx.x = 0; threadIdx.x < kZThreads; ++threadIdx.x)
        k2_tile<T, T, false, CHAIN>(&L, &o, pre, 1, pot.data(), scratch.data(), en ? ep.data() : nullptr,
                                    en ? ek.data() : nullptr, ntile, CUtensorMap{}, 1, tile);
    const int x0 = tile % ntx * TX, y0 = tile / ntx * TY;
    const T *g = scratch.data() + (CHAIN ? o.sZ : o.sQ);
    size_t seen = 0;
    for (int z = 0; z < d.G3; ++z)
        for (int y = y0; y < min(y0 + TY, H); ++y)
            for (int x = x0; x < min(x0 + TX, W); ++x, ++seen)
                if (!std::isnan(g[((size_t)z * H + y) * WP + x])) return 1;
    size_t nan = 0;
    for (const T &v : scratch) nan += std::isnan(v);
    if (nan != seen) return 2;
    for (int i = 0; i < ntile; ++i)
        if (std::isnan(ep[i]) != (CHAIN == 0 && i == tile) || std::isnan(ek[i]) != (CHAIN == 1 && i == tile)) return 3;
    return 0;
}

extern "C" int ztile_timed_out(int prec, int chain, int n1, int n2, int n3, int tile)
{
    const int N[3] = {n1, n2, n3};
    if (prec == 32) return chain == 0 ? timed_out<float, 0>(N, tile) : chain == 1 ? timed_out<float, 1>(N, tile) : timed_out<float, 2>(N, tile);
    return chain == 0 ? timed_out<double, 0>(N, tile) : chain == 1 ? timed_out<double, 1>(N, tile) : timed_out<double, 2>(N, tile);
}
