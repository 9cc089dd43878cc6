"""The FP32 forms' slots (csrc/mhd_layout.h): a row takes at most seven slots
more than it has cells -- device memory is what limits the largest grid or
batch -- cells and their variables do not overlap, a row's cells from k = 1 on
start a group, and the staged update's tiles, the one that runs past the last
interior cell among them, stay inside the array at the smallest grids."""
import os
import subprocess

from conftest import PKG

SRC = r"""
#include <cstdio>
#include <vector>
#include "mhd_layout.h"
using namespace mhd;
static long bad = 0;
#define CHECK(c) do { if (!(c) && bad++ < 8) printf("kzmax %d, %d rows: %s\n", kzmax, (int)rows, #c); } while (0)
int main()
{
    for (int kzmax = 14; kzmax <= 300; kzmax++)
        for (int ixjy = 0; ixjy < 8; ixjy++) {
            const int jymax = ixjy % 2 ? 8 : 6, ixmax = 14 + ixjy / 2;
            const long long rows = (long long)ixmax * jymax;
            const int kp = row_slots(kzmax);
            const long long n = array_slots(rows, kp);
            CHECK(kp >= kzmax && kp <= kzmax + 7);
            CHECK(kp % MHD_GROUP == 0 && n % MHD_GROUP == 0);
            std::vector<char> used(9 * n);
            for (long long r = 0; r < rows; r++) {
                CHECK(row_slot(r, kp, 1) % MHD_GROUP == 0);
                for (int k = 0; k < kzmax; k++) {
                    const long long q = row_slot(r, kp, k);
                    CHECK(q >= 0 && q < n);
                    for (int m = 0; m < 9; m++) {
                        const long long o = slot_offset(q) + m * MHD_GROUP;
                        CHECK(o >= 0 && o < 9 * n && !used[o]);
                        if (o >= 0 && o < 9 * n) used[o] = 1;
                    }
                }
            }
            const long long beg = row_slot(jymax, kp, 1), end = row_slot((long long)(ixmax - 1) * jymax, kp, 1);
            const long long last = beg + (end - beg + MHD_UPD_TILE - 1) / MHD_UPD_TILE * MHD_UPD_TILE;
            CHECK(last <= n);
            CHECK(beg - MHD_GROUP >= 0 && beg - (long long)jymax * kp >= 0);
            CHECK(slot_offset(beg) % 4 == 0 && slot_offset(kp) % 4 == 0);   /* bulk copies: 16 bytes */
        }
    printf("bad %ld\n", bad);
    return bad != 0;
}
"""


def test_rows_are_tight_and_in_range(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(PKG, "csrc"), str(tmp_path / "t.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
