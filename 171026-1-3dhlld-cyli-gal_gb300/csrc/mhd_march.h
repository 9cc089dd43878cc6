/*
 * mhd_march.h -- which faces a thread of the merged face launch marches over.
 *
 * A line's cells along k are taken in groups of 32, one warp each; the warps
 * of a run of faces are numbered group by group and line by line, and blocks
 * of four warps take them in that order, whatever the number of groups in a
 * line.  So every face has one thread, and every warp but a run's last few has
 * work.  (A block laid out as whole rows holds one row of three groups and
 * leaves a warp over: given the next line's first group, which the next block
 * takes as well, that warp's faces are stored by two blocks.)
 *
 * Plain C++: the host compiles it too, for the tests.
 */
#ifndef MHD_MARCH_H
#define MHD_MARCH_H

#ifdef __CUDACC__
#define MHD_MARCH_FN __host__ __device__ __forceinline__
#else
#define MHD_MARCH_FN static inline
#endif

namespace mhd {

/* nl lines of nk cells and nf faces, mr faces per run: groups of 32 cells in a
 * line, warps and blocks of a run, blocks in all */
struct MarchPlan {
    int nk, nf, mr, groups, warps, run_blocks, nblk;
};

static inline MarchPlan march_plan(int nk, int nl, int nf, int mr)
{
    MarchPlan p;
    p.nk = nk;
    p.nf = nf;
    p.mr = mr;
    p.groups = (nk + 31) / 32;
    p.warps = nl * p.groups;
    p.run_blocks = (p.warps + 3) / 4;
    p.nblk = p.run_blocks * ((nf + mr - 1) / mr);
    return p;
}

/* thread t (of 128) of block b: its line and cell, from 1, and its faces f0 ..
 * fe-1; false where it has none.  Divided as unsigned: the signs' handling took
 * registers that the plain form's faces do not have (20 words reloaded a face). */
MHD_MARCH_FN bool march_thread(const MarchPlan &p, int b, int t, int &line, int &k, int &f0, int &fe)
{
    const int run = (int)((unsigned)b / (unsigned)p.run_blocks), w = (b - run * p.run_blocks) * 4 + (int)((unsigned)t >> 5);
    const int l = (int)((unsigned)w / (unsigned)p.groups);
    line = 1 + l;
    k = 1 + (w - l * p.groups) * 32 + (t & 31);
    f0 = run * p.mr;
    fe = f0 + p.mr < p.nf ? f0 + p.mr : p.nf;
    return w < p.warps && k <= p.nk;
}

/* Whether the r, phi and z faces of ni x nj x nk interior cells go into one
 * launch, or into one per direction.  One launch fills the GPU where a
 * direction alone does not, and packs rows of 5, 6, 7, 9 .. groups of 32 cells
 * without idle warps, where a launch per direction takes rows in blocks of four
 * warps (`whole`: it leaves none idle either).  On large FP32 grids the launches
 * per direction win: their marches hold 62 to 64 registers instead of 72, and
 * superbee, which waits on memory most, gains most.  A step in FP32, one launch
 * / one per direction:
 *   minmod   256x256x128 2623 / 2663 us, 384x384x256 10960 / 10964, 512x384x256
 *            14567 / 14544, 512x512x256 19425 / 19360; rows of 7 groups:
 *            512x512x224 17146 / 17237
 *   van Leer 384x384x256 11244 / 11171, 512x512x256 19979 / 19721
 *   superbee 192x160x128 2150 / 2243, 224x224x128 3455 / 3441, 384x384x128 9865 /
 *            9387, 512x512x256 33643 / 31255; rows of 6 groups: 320x320x192
 *            10172 / 10281, 512x256x192 12926 / 12823
 * The pair-state form, the same faces, alike.  The plain form (128 registers
 * either way): 512x512x192 324 / 327 ms. */
static inline bool one_face_launch(bool fp32, bool superbee, int ni, int nj, int nk)
{
    const int groups = (nk + 31) / 32;
    const bool whole = groups <= 4 || groups % 4 == 0;
    const double cells = (double)ni * nj * nk;
    if (!fp32) return true;
    if (superbee) return cells < (whole ? 6e6 : 20e6);
    return !whole || cells < 40e6;
}

} /* namespace mhd */

#endif
