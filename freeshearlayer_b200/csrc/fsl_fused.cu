// fsl_fused.cu -- FP64 instantiations of the fused stage kernels (the plain
// method) and the choice between them.  Compiled with --fmad=false: every value is formed with the
// reference's expressions and rounds exactly like the reference's serial code.
#define FSL_CHK_UNIT FSL_CHK_FUSED
#include "fsl_stage.cuh"
#include "fsl_stage_dir.cuh"

FSL_CHK_EXPORT(fused)

namespace fsl {

static stage::BF<double> bf64(Ctx &c)
{
    stage::BF<double> b;
    b.x0 = c.bf.x0; b.xL = c.bf.xL; b.y0 = c.bf.y0; b.yH = c.bf.yH; b.z0 = c.bf.z0; b.zD = c.bf.zD;
    return b;
}

void launch_boundary(Ctx &c, double *cur, const Disturb &d)
{
    stage::launch_boundary_t<double>(c, cur, d, bf64(c));
}

// How a domain's tiles (tj x tk output cells) are cut along x when one block
// fits on an SM: the blocks run in waves and a segment of n planes costs n +
// `start` planes, so take the n whose waves cost least.  One search over all n a domain
// (2.6 ms at 2^20 planes), not one a launch.
static Cut cut_tiles(const Grid &g, int sms, int tj, int tk, double start)
{
    const long long tiles = (long long)((g.D + tk - 1) / tk) * ((g.H + tj - 1) / tj);
    Cut best{g.L, -1.};
    for (int n = 1; n <= g.L; n++) {
        const long long segs = (g.L + n - 1) / n;
        const double t = (double)((tiles * segs + sms - 1) / sms) * (n + start);
        if (best.cost < 0. || t < best.cost) best = {n, t};
    }
    return best;
}
void stage_cuts(Ctx &c)
{
    c.ring_cut = cut_tiles(c.g, c.sms, 14, 30, 1.2);
    c.ppm_cut = cut_tiles(c.g, c.sms, 10, 30, 1.2);
    c.dir_cut = cut_tiles(c.g, c.sms, dirs::WJ, dirs::WK, 2.0);
}

// The ring tile marches a plane of 14 x 30 cells in 10.8 us, the direction-split
// kernel one of 4 x 32 in 4.95 us and 3 us a launch, whatever the grid (measured
// from 24x16x16 to 256x128x128): per cell the ring is faster by half, but the
// smaller tiles leave fewer SMs idle on small grids and no columns empty where
// DEP is a multiple of 32, and on the temporal setup the direction split needs no
// boundary pass (6 us a stage and more on large grids).  Per step, ring with its
// passes against direction split: 64x32x32 163 / 107 us, 96x48x48 261 / 284,
// 512x64x32 1288 / 924, 100x80x35 (spatial) 361 / 515, 256x128x128 3076 / 3553.
bool stage_splits_directions(const Ctx &c)
{
    if (c.p.recon != FSL_RECON_CHARMINMOD || c.stage_tje != 0 || c.seg_set) return false;
    const double pass = c.p.setup == FSL_SETUP_TEMPORAL ? 6. : 0.;
    return 3. + 4.95 * c.dir_cut.cost < 10.8 * c.ring_cut.cost + pass;
}

template <bool SST>
static int stage64(Ctx &c, int stage, const double *cur, const double *un, double *out, bool courant)
{
    // PPM: halo 2, a ring of five planes, the one in flight included.  A 16-row FP64
    // tile would need more than the 227 KB of shared memory a block may have; 12 rows
    // measured fastest at 512x256x256 (35.5 ms per step against 46.4 for 8, and 34.5 with
    // the planes per block by the grid), so 16 runs as 12
    if (c.p.recon == FSL_RECON_PPM) {
        if (c.stage_tje == 8)
            return stage::launch_stage_t<double, 8, 1, true, SST>(c, stage, cur, un, out, c.mu, bf64(c), courant);
        return stage::launch_stage_t<double, 12, 1, true, SST>(c, stage, cur, un, out, c.mu, bf64(c), courant,
                                                               c.stage_tje || c.seg_set ? 0 : c.ppm_cut.seg);
    }
    switch (c.stage_tje) {
    case 0:
        if (stage_splits_directions(c))
            return dirs::launch_stage_dir<SST>(c, stage, cur, un, out, c.mu, bf64(c), courant, c.dir_cut.seg);
        return stage::launch_stage_t<double, 16, 1, false, SST>(c, stage, cur, un, out, c.mu, bf64(c), courant,
                                                                c.seg_set ? 0 : c.ring_cut.seg);
    case 8: return stage::launch_stage_t<double, 8, 1, false, SST>(c, stage, cur, un, out, c.mu, bf64(c), courant);
    case 12: return stage::launch_stage_t<double, 12, 1, false, SST>(c, stage, cur, un, out, c.mu, bf64(c), courant);
    default: return stage::launch_stage_t<double, 16, 1, false, SST>(c, stage, cur, un, out, c.mu, bf64(c), courant);
    }
}

int launch_stage(Ctx &c, int stage, const double *cur, const double *un, double *out, bool courant)
{
    // the static Smagorinsky model forms the face viscosity in the kernel
    if (c.p.sgs == FSL_SGS_STATIC) return stage64<true>(c, stage, cur, un, out, courant);
    return stage64<false>(c, stage, cur, un, out, courant);
}

} // namespace fsl
