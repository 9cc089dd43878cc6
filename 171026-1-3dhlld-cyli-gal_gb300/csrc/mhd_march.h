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
 * fe-1; false where it has none */
MHD_MARCH_FN bool march_thread(const MarchPlan &p, int b, int t, int &line, int &k, int &f0, int &fe)
{
    const int run = b / p.run_blocks, w = (b - run * p.run_blocks) * 4 + (t >> 5);
    const int l = w / p.groups;
    line = 1 + l;
    k = 1 + (w - l * p.groups) * 32 + (t & 31);
    f0 = run * p.mr;
    fe = f0 + p.mr < p.nf ? f0 + p.mr : p.nf;
    return w < p.warps && k <= p.nk;
}

} /* namespace mhd */

#endif
