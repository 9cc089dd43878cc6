"""The merged face launch's marches (csrc/mhd_march.h): every face of every
line belongs to exactly one thread -- two threads on one face would store the
same words unordered -- and a warp's cells are one group of 32 of one line, at
row lengths on both sides of every multiple of 32 and of a block's 128."""
import os
import subprocess

from conftest import PKG

SRC = r"""
#include <cstdio>
#include <vector>
#include "mhd_march.h"
using namespace mhd;
int main()
{
    long bad = 0;
    for (int nk = 2; nk <= 300; nk++)
        for (int nl : {1, 2, 3, 7, 12})
            for (int nf : {3, 16, 33})
                for (int mr : {1, 4, 16}) {
                    const MarchPlan p = march_plan(nk, nl, nf, mr);
                    std::vector<int> seen((size_t)nk * nl * nf);
                    long twice = 0, outside = 0, split = 0;
                    for (int b = 0; b < p.nblk; b++)
                        for (int t = 0; t < 128; t++) {
                            int line, k, f0, fe;
                            if (!march_thread(p, b, t, line, k, f0, fe)) continue;
                            if (line < 1 || line > nl || k < 1 || k > nk || f0 < 0 || fe > nf) { outside++; continue; }
                            if ((k - 1) % 32 != t % 32) split++;
                            for (int f = f0; f < fe; f++) twice += seen[((size_t)(line - 1) * nk + k - 1) * nf + f]++ > 0;
                        }
                    long missed = 0;
                    for (int s : seen) missed += s == 0;
                    if ((twice || outside || missed || split) && bad++ < 5)
                        printf("nk %d nl %d nf %d mr %d: %ld twice, %ld outside, %ld missed, %ld off a group\n",
                               nk, nl, nf, mr, twice, outside, missed, split);
                }
    printf("bad %ld\n", bad);
    return bad != 0;
}
"""


def test_each_face_has_one_thread(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(PKG, "csrc"), str(tmp_path / "t.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


RULE = r"""
#include <cstdio>
#include "mhd_march.h"
int main()
{
    int fp32, superbee, ni, nj, nk;
    while (scanf("%d %d %d %d %d", &fp32, &superbee, &ni, &nj, &nk) == 5) printf("%d\n", mhd::one_face_launch(fp32, superbee, ni, nj, nk));
    return 0;
}
"""
# FP32: cells on both sides of each line, in rows that a launch per direction
# packs whole (1 to 4 groups of 32, or whole blocks of 4) and in rows that it
# does not; the plain form always in one launch
ONE = [(1, 0, 12, 4, 12), (1, 0, 384, 384, 256), (1, 0, 512, 512, 224), (1, 0, 640, 640, 160), (1, 1, 64, 64, 32),
       (1, 1, 192, 160, 128), (1, 1, 320, 320, 192), (0, 0, 512, 512, 256), (0, 1, 512, 512, 256)]
EACH = [(1, 0, 512, 384, 256), (1, 0, 512, 512, 250), (1, 0, 1024, 512, 128), (1, 1, 224, 224, 128), (1, 1, 384, 384, 64),
        (1, 1, 512, 512, 96), (1, 1, 512, 256, 192), (1, 1, 512, 512, 256)]


def test_which_grids_take_one_launch(tmp_path):
    (tmp_path / "r.cpp").write_text(RULE)
    exe = str(tmp_path / "r")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(PKG, "csrc"), str(tmp_path / "r.cpp"), "-o", exe])
    r = subprocess.run([exe], input="".join("%d %d %d %d %d\n" % c for c in ONE + EACH), capture_output=True, text=True)
    assert r.stdout.split() == ["1"] * len(ONE) + ["0"] * len(EACH)
