// resident.cuh -- the acoustic time loop with its wavefields kept on chip (resident.cu): which
// shots it takes, how a grid is cut into tiles, and the launch.
#pragma once

#include <algorithm>
#include <vector>

#include "w2d_common.cuh"

namespace w2d {

constexpr int RS_CT = 480;          // compute threads (15 warps)
constexpr int RS_T = RS_CT + 32;    // and one halo warp: 16 warps, 128 registers a thread
constexpr int RS_MAXR = 15;         // rows of one phase-I thread: its tensor-memory words
constexpr int RS_SMEM = 227 * 1024; // always the whole SM: no second CTA, which could wait
                                    // for tensor memory while its neighbours wait for it
// Shortest pass of an engine that runs here: loading and storing the tiles of a shorter one takes
// longer than the launches saved.  us on the device, a launch per step -> here: forward, 40 x 80,
// 1 step 15.7 -> 24, 4 steps 32 -> 29; 1000 x 4000, 1 step 30 -> 54, 6 steps 80 -> 80; migration,
// 150 x 400, 2 steps 47 -> 77, 6 steps 90 -> 88; 1000 x 4000, 6 steps 207 -> 213, 8 steps 257 -> 239.
constexpr int RS_MIN_STEPS = 6;
constexpr int RS_POLLS = 1 << 21;    // looks at a missing packet before giving up (about 1 s)
// Groups of 32 packets a warp has in flight: the halo warp, and a compute warp that is done.
// (More of them look at packets that have not come, and compete with those that come: 8 for
// the halo warp took 3.1 us a step in place of 1.7 at 301 x 1203.)
constexpr int RS_FLIGHT_H = 1, RS_FLIGHT_C = 2;

// One shot (or one pass of it) as the resident kernel runs it.  Phase step k is forward
// step k for k < nt, else backward step 2*nt-1-k.
struct RsShot {
    int nx, nz, ldx, gx, gz, maxc, maxr;
    float inv_dx2, inv_dz2;
    int fs, n_sponge;
    const float* lut;          // sponge by frame distance, non-increasing (null: none)
    int src_ix, src_iz, rec_iz, n_rec, rec_c0;
    const int* rec_ptr;        // at most one receiver per column
    const int* rec_list;
    int nt, interval, k0, k1;
    float* wave[6];            // forward triple, backward triple, roles by step as elsewhere
    const float* vel[2];       // v^2 dt^2 of the forward and the backward pass
    float* snaps;              // forward: written when not null; backward: read when imaging
    int slot0, n_snaps;        // first snapshot held; snapshots that exist (backward)
    // The velocity gradient.  With q = c a, c = v^2 dt^2, the adjoint of the step
    // (adjoint_kernels.cuh) is the step itself: q[n] = s (2 q[n+1] - q[n+2] + c (L q[n+1] +
    // r[n-1])), and dJ/dc = (1/c) sum_n q[n+1] L P[n].  So (lap) the forward pass keeps
    // L P[n], which it computes anyway, in place of P[n], and (adjoint) the backward pass
    // images with it, its receivers' injection times c s, its free surface the transpose
    // of the forward one: row 2 reads -q[2] and -q[3] for rows 1 and 0, which stay zero.
    int lap, adjoint;
    size_t plane;
    float* illum;              // forward: accumulated when not null
    float* image;              // backward: accumulated when not null
    const float* wavelet;
    const float* data;
    float* rec_out;            // forward: sampled when not null
    float dt2_inj, img_dt;
    float minus_zero = -0.0f;  // an operand the compiler must not know (see mul2)
    uint4* xbuf;               // packets: tile, slot, {left, right, top, bottom}
    unsigned tag0;             // the launch's tags are tag0 + 1 ..: none was used in xbuf before
    unsigned* err;
};

// ---- host: how a grid is cut -------------------------------------------------------
struct RsPlan {
    int gx = 0, gz = 0, maxc = 0, maxr = 0;
    double cost = 0;  // estimated us of a step
    bool ok() const { return gx > 0; }
    int ctas() const { return gx * gz; }
    size_t packets() const { return 2 * (size_t)(2 * maxr + 8 * maxc); }  // of one tile
    size_t xbuf_bytes() const { return packets() * ctas() * sizeof(uint4); }
};

constexpr int RS_TILE_FLOATS = 64, RS_SHOT_FLOATS = 96;  // the tile's and the shot's records

// floats of shared memory of a tile of nrows x ncol units
__host__ __device__ inline size_t rs_smem_floats(int nrows, int ncol)
{
    const size_t pitch = 4 * (size_t)ncol;
    return RS_TILE_FLOATS + RS_SHOT_FLOATS + 2 * (nrows + 4) * pitch + 8 * (size_t)nrows +
           4 * pitch + (nrows + 3) / 4 * 4 + 24;
}

// Phase I of a tile: columns 1..ncol-2 by rows 2..nrows-3 in segments of R rows.
__host__ __device__ inline void rs_interior(int nrows, int ncol, int* nci, int* nseg, int* R)
{
    *nci = ncol - 2;
    const int ni = nrows - 4;
    *nseg = *R = 0;
    if (*nci <= 0 || ni <= 0) return;
    const int s = min(RS_CT / *nci, ni);
    *R = (ni + s - 1) / s;
    *nseg = (ni + *R - 1) / *R;
}

// The cuts of an nx x nz grid: element n is the one into at most n tiles (n = 1 ..
// max_ctas) with the least estimated step time, none where the grid does not fit the
// shared memory of n SMs.  What a step costs is its slowest tile, so columns and rows are
// split evenly and the estimate (in us) is that of the largest tile: a fixed chain, the edge
// units (columns cost more: their snapshot accesses do not coalesce), the interior.
inline std::vector<RsPlan> rs_plans(int nx, int nz, int max_ctas)
{
    std::vector<RsPlan> best(std::max(max_ctas, 0) + 1);
    const int w4 = (nx + 3) / 4;
    for (int gx = 1; gx <= max_ctas && (gx == 1 || w4 / gx >= 2); ++gx)
        for (int gz = 1; gx * gz <= max_ctas && (gz == 1 || nz / gz >= 4); ++gz) {
            const int ncol = (w4 + gx - 1) / gx, nrows = (nz + gz - 1) / gz;
            const int ne = 2 * nrows + 4 * (ncol - 2);
            if (ncol < 2 || nrows < 5 - (gz > 1) || ne > RS_CT) continue;
            if (rs_smem_floats(nrows, ncol) * 4 > (size_t)RS_SMEM) continue;
            int nci, nseg, R;
            rs_interior(nrows, ncol, &nci, &nseg, &R);
            if (R > RS_MAXR) continue;
            // fitted to 86 cuts of 7 grids (migrations, every second step imaged): 6 % rms
            const double warps = (nci * nseg + 31) / 32;
            const double cost = 1.69 + 0.0087 * nrows + 0.0061 * ncol + 0.019 * R * warps;
            RsPlan& b = best[gx * gz];
            if (b.ok() && b.cost <= cost) continue;
            b.gx = gx;
            b.gz = gz;
            b.maxc = ncol;
            b.maxr = nrows;
            b.cost = cost;
        }
    for (int n = 1; n <= max_ctas; ++n)
        if (!best[n].ok() || (best[n - 1].ok() && best[n - 1].cost <= best[n].cost))
            best[n] = best[n - 1];
    return best;
}

// The sources and receivers the kernel takes: on interior rows (and columns, for the
// source), at most one receiver per column.  src_ix < 0: no source.
inline bool rs_shot_fits(int nx, int nz, int src_ix, int src_iz, int n_rec, int rec_iz,
                         bool unique_columns)
{
    if (src_ix >= 0 && (src_ix < 2 || src_ix >= nx - 2 || src_iz < 2 || src_iz >= nz - 2))
        return false;
    return n_rec == 0 || (unique_columns && rec_iz >= 2 && rec_iz < nz - 2);
}

// The sponge as a product of nothing but the larger frame distance's factor needs
// factors that do not increase with distance: lut[max(a, b)] = min(lut[a], lut[b]).
inline bool rs_lut_fits(const float* lut, int n)
{
    for (int d = 0; d <= n; ++d)
        if (!(lut[d] <= (d ? lut[d - 1] : 1.0f)) || (d == 0 && lut[d] != 1.0f)) return false;
    return true;
}

// Phase steps of one shot, or (many) of several, items[CTA] = {shot, tile}: one cooperative
// launch of `ctas` CTAs.  Packets of earlier launches must be gone from xbuf.
cudaError_t launch_acoustic_resident(const RsShot& one, const RsShot* many, const int2* items,
                                     int ctas, cudaStream_t st);

// CTAs that are resident at once on the current device (0 on error or where a
// cooperative launch is not available).
int rs_capacity();

}  // namespace w2d
