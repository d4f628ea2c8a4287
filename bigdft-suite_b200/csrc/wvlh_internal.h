// Internal host/device structures of the wvlh library (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

namespace wvlh {

// z-kernel tile: TX_ consecutive x by TY_ rows of columns
constexpr int TX_ = 32;
constexpr int TY_ = 2;
// Wavelet points of a line segment one thread takes in the fused kernels'
// passes: eight, 16 accumulators in flight, as boxes are mostly multiples of
// eight; six in the FP32 plane kernels, whose passes then come in rounds that
// divide better over their threads on most boxes (K1 + K3 of 128 orbitals, six
// against eight points: 48^3 0.512 + 1.161 against 0.516 + 1.164 ms, 40^3 0.329 +
// 0.780 against 0.336 + 0.824; 32^3 0.165 + 0.396 against 0.147 + 0.359 the other
// way).  The FP64 plane kernels (32^3: K3 0.85 -> 0.68 ms) and the z kernel (40^3
// FP32 0.60 -> 0.49 ms) gain from eight: fewer window loads an output.
constexpr int kSegZ = 8;
__host__ __device__ constexpr int plane_seg(bool fp32) { return fp32 ? 6 : 8; }
// block size of the persistent plane kernels
constexpr int kPlaneThreads = 384;

// The plane kernels (K1, K3) run with any block size; they are compiled for
// these bounds, at what the compiler gives a thread under bound x CTAs per SM:
// FP32 56, 56, 72, 64, 64 registers; FP64 96, 168, 96, 96, 128 (576 threads are 18
// warps, five to a quarter of the SM's registers).  K1 fits (at most 8 bytes
// spilled), so does FP32 K3.  FP64 K3 spills 96 to 120 bytes a thread in periodic
// and 264 to 324 in free boxes at 96 registers, 68 to 108 at 128, none at the
// 384 bound; 576 threads still came out ahead of 384 (64 x 48^3: 2.46 against
// 2.53 ms a call).  Two planes of a 96 x 96 box leave room for three FP32 CTAs or
// one FP64 CTA.
constexpr int kPlaneSizes[5] = {576, 384, 288, 192, 128};
__host__ __device__ constexpr int plane_ctas_per_sm(bool fp32, int nt)
{
    return fp32 ? (nt > 384 ? 2 : nt > 192 ? 3 : nt > 128 ? 5 : 8) : (nt > 288 ? 1 : nt > 192 ? 2 : nt > 128 ? 3 : 4);
}

// Block size of the plane kernels, chosen per batch by a small occupancy model.
// A pass over rows has `rows` lines, one over columns `len` lines (two FP32
// columns or one FP64 column a thread), each cut into segments of plane_seg
// wavelet points (twice as many points of a line); with nt threads a pass of n
// items takes ceil(n / nt) rounds, so the busy fraction is the two passes'
// items over their rounds times nt (a column item of two FP32 columns weighs
// two); the SM holds as many CTAs as registers (the compiled count above),
// shared memory and threads allow.  The expected rate is busy x resident
// threads x ctas / (ctas + 1/2) -- the last factor because a CTA's barrier
// waits are covered only by the other resident CTAs; each orbital's planes
// weigh by their work, and the size with the least total cost wins.
struct PlaneShape {
    long long rows, len, smem_bytes, weight;
};
inline double plane_cost(const std::vector<PlaneShape> &shapes, bool fp32, int nt)
{
    const long long seg = 2 * plane_seg(fp32), cu = fp32 ? 2 : 1;
    double cost = 0.0;
    for (const PlaneShape &s : shapes) {
        const long long ri = s.rows * ((s.len + seg - 1) / seg);
        const long long ci = (s.len + cu - 1) / cu * ((s.rows + seg - 1) / seg);
        const long long rounds = (ri + nt - 1) / nt + cu * ((ci + nt - 1) / nt);
        const double busy = (double)(ri + cu * ci) / (double)(rounds * nt);
        const long long by_regs = plane_ctas_per_sm(fp32, nt);
        const long long by_smem = (227LL * 1024) / (s.smem_bytes + 1024);
        long long ctas = by_regs < by_smem ? by_regs : by_smem;
        if (ctas < 1) ctas = 1;
        cost += (double)s.weight / (busy * (double)ctas * nt * ((double)ctas / ((double)ctas + 0.5)));
    }
    return cost;
}
// the best block size of each compiled bound (those above the next smaller
// bound), and the best of all
inline int choose_plane_threads(const std::vector<PlaneShape> &shapes, bool fp32, int *cand = nullptr)
{
    double best = 0.0;
    int pick = 0;
    for (int k = 0; k < 5; ++k) {
        double bk = 0.0;
        int nk = 0;
        for (int nt = kPlaneSizes[k]; nt > (k < 4 ? kPlaneSizes[k + 1] : 32); nt -= 32) {
            const double c = plane_cost(shapes, fp32, nt);
            if (!nk || c < bk * 0.999) {
                bk = c;
                nk = nt;
            }
        }
        if (cand) cand[k] = nk;
        if (!pick || bk < best * 0.999) {
            best = bk;
            pick = nk;
        }
    }
    return pick;
}
constexpr int kZThreads = 256;

// One localisation region (box + compressed-key tables) as seen by kernels.
// The reference's 1-based keyg/keyv (wavelib/un-compress.f90:896-905) are
// expanded on upload to 16 bits per cell: pos_c / pos_f[j] is the place of the
// j-th coarse / fine cell of the compressed vector in a wavelet plane of the
// plane kernels' shared-memory layout (y * pitch + x; a plane that fits shared
// memory has fewer than 65536 places, larger boxes are refused at launch).  Keys are sorted, so the
// cells of one z-plane are consecutive: plane_c / plane_f[i3 .. i3+1] delimit
// those of coarse plane i3.
struct LrDev {
    int N[3];
    int per[3];
    int nseg_c, nseg_f;
    int nvctr_c, nvctr_f;
    const uint16_t *pos_c;
    const uint16_t *pos_f;
    const int *plane_c;  // N3+1 entries
    const int *plane_f;  // N3+1 entries
    double hgrid[3];     // coarse grid spacing
};

// One orbital job of a batch.
struct OrbDev {
    int lr;
    int pad;
    long long psi;   // element offset of [psi_c | psi_f] in the psi/hpsi arrays
    long long pot;   // element offset of this orbital's potential / density (ISF grid)
    // scratch element offsets of the orbital's planes, one per wavelet z-plane:
    long long sP;    //   D (2N2 x 2N1 dense)
    long long sQ;    //   Q / Z1 (I2 rows, isf_pitch apart)
    long long sZ;    //   Z2 (2N2 x 2N1 dense)
    double c;        // shift of (T + c), preconditioner only
    // optional absolute buffers (a batch that spans several owners' arrays);
    // when set they replace base + offset
    const void *in_ptr;
    void *out_ptr;
    const void *pot_ptr;
};

// plane shapes of a batch whose orbitals all lie in one region (TMA tiles)
struct TileDims {
    long long G1, G2, G3, I1, IP1, I2;
    long long ofs_q;   // Q's element offset in an orbital's scratch
};

enum FusedMode { MODE_LOCHAM = 0, MODE_LOCDEN = 1, MODE_PRECOND = 2 };

// Host view of an uploaded batch (plan) — owned by the context.
struct Plan {
    int nlr = 0, norb = 0;
    bool all_periodic = false;  // every region periodic in x, y and z
    std::vector<int> lr_N;  // 3*nlr
    std::vector<int> lr_per;
    std::vector<int> orb_lr;
    std::vector<long long> orb_psi;  // element offsets
    long long psi_total = 0;
    long long scratch_elems = 0;     // per "chunk" of all orbitals (full batch)
    // device tables
    LrDev *d_lr = nullptr;
    OrbDev *d_orb = nullptr;
    // work items in runs of one orbital: prefix sums over the orbitals (norb+1
    // entries) of the plane kernels' items (G3 wavelet planes each) and of the
    // z kernels' 32 x 2-column tiles: chain 0 over I1 x I2 (d_pre2), chain 1
    // over 2 N1 x 2 N2 (d_pre2p)
    int *d_pre13 = nullptr;
    int *d_pre2 = nullptr;
    int *d_pre2p = nullptr;
    int n_work13 = 0, n_work2 = 0, n_work2p = 0;
    // density: z-kernel tiles of the I1 x I2 plane, in runs of one chunk
    // (prefix over the chunks) of orbitals that share one density grid (same
    // region, same density key)
    int *d_pred = nullptr;
    int n_workd = 0;
    int nchunk = 0, ngroup = 0;
    int *d_chunk_orb_start = nullptr;    // nchunk + 1 offsets into d_chunk_orbs
    int *d_chunk_orbs = nullptr;
    long long *d_chunk_part = nullptr;   // element offset of each chunk's partial density
    long long part_den_elems = 0;
    int *d_group_chunk_start = nullptr;  // ngroup + 1 chunk ranges
    long long *d_group_rho = nullptr;    // density offset (or address) of each group
    int *d_group_n = nullptr;            // ISF points of each group
    int max_group_n = 0;
    int den_acc = 32;                    // FP64 accumulators per thread of kd_density (32 or 48)
    // per-orbital compressed vector offset / length (preconditioner vector ops)
    long long *d_orb_off = nullptr;
    int *d_orb_len = nullptr;
    int part_stride = 0;           // energy partial slots per orbital
    size_t smem13[2] = {0, 0};     // dynamic smem bytes (float, double) of the two plane buffers
    long long plane_elems = 0;     // elements of plane buffer A (rows x pitch)
    long long planeB_elems = 0;    // elements of buffer B (2 N2 rows)
    int plane_threads[2] = {kPlaneThreads, kPlaneThreads};   // plane-kernel CTA size (float, double)
    int plane_threads_pre[2] = {kPlaneThreads, kPlaneThreads};   // the same for the preconditioner operator
    int plane_cand[2][5] = {};                       // the sizes that the autotuner measures
    int z_segs0 = 1, z_segs1 = 1;                    // segments of the longest z line (chain 0, chain 1)
    int z_threads[2] = {kZThreads, kZThreads};       // z-kernel CTA bound (FP32: 256, 320 or 384)
    int z_threads_pre[2] = {kZThreads, kZThreads};   // the same for the preconditioner operator
    // two tile columns of the longest grid in z: more than the z kernels ask for
    // (smem_z0, smem_z1), it decides which boxes the entry points take
    size_t smem2[2] = {0, 0};
    size_t smem_z0[2] = {0, 0};    // dynamic smem bytes of the z kernel's chain 0 (and the density) ...
    size_t smem_z1[2] = {0, 0};    // ... and of chain 1
    // scratch elements per orbital when every orbital lies in one region (the
    // planes then form regular (x, y, z, orbital) tensors: TMA tiles), else 0
    long long orb_scratch = 0;
    TileDims tile = {};
    std::vector<void *> owned;     // device allocations to free
};

// Checks the reference's 1-based keys of one region (compression.f90:29-39):
// keyg = (first, last) linear index of each segment in the N[0] x N[1] x N[2]
// box, x fastest, strictly increasing, each segment on one x-line; keyv the
// running 1-based offset of each segment in the compressed vector.  Returns
// WVLH_OK or WVLH_ERR_KEYS; on success nvctr is the number of values.
inline int check_keys(const int *N, int nseg, const int32_t *keyg, const int32_t *keyv, long long *nvctr)
{
    const long long n12 = (long long)N[0] * N[1], ntot = n12 * N[2];
    long long prev_end = 0, cum = 0;
    for (int s = 0; s < nseg; ++s) {
        const long long j0 = keyg[2 * s], j1 = keyg[2 * s + 1];
        if (j0 < 1 || j1 < j0 || j1 > ntot || j0 <= prev_end) return 3;          // WVLH_ERR_KEYS
        if ((j0 - 1) / N[0] != (j1 - 1) / N[0]) return 3;                         // one x-line per segment
        if ((long long)keyv[s] != cum + 1) return 3;
        cum += j1 - j0 + 1;
        prev_end = j1;
    }
    if (nvctr) *nvctr = cum;
    return 0;
}

}  // namespace wvlh
