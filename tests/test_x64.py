"""The plain form's division, square root, comparisons and slope on integers
(csrc/mhd_x64.h) against the host's IEEE arithmetic, bit for bit: mantissas at
both ends, quotients next to 1, exponents to both ends of the range, zeros,
subnormals, infinities, NaNs; and again with the approximate reciprocal and
root that the digits start from off by the two ulp the device's may be."""
import os
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include <cstdio>
#include <random>
#include "%s"
using namespace mhd;
static uint64_t B(double a) { uint64_t u; memcpy(&u, &a, 8); return u; }
static double D(uint64_t u) { double a; memcpy(&a, &u, 8); return a; }
static long bad = 0;
static void same(const char *what, double got, double want, double a, double b)
{
    if (B(got) != B(want) && !(got != got && want != want) && bad++ < 5) printf("%%s(%%a, %%a) = %%a, want %%a\n", what, a, b, got, want);
}
static double rmin(double a, double b) { return a > b ? b : a; }
static double rmax(double a, double b) { return a > b ? a : b; }
static void check(double a, double b, double c)
{
    same("div", x_div(a, b), a / b, a, b);
    same("sqrt", x_sqrt(a), sqrt(a), a, b);
    same("gt", x_gt(a, b), a > b, a, b);
    same("ge0", x_ge0(a), a >= 0.0, a, b);
    same("le0", x_le0(a), a <= 0.0, a, b);
    same("sign", x_sign(a), fabs(a) / a, a, b);
    const double one = B(b) >> 63 ? -1.0 : 1.0;
    same("mulsign", x_mulsign(a, one), a * one, a, one);
    same("mulsign", x_mulsign(a, b), a * b, a, b);
    same("doubled_half", x_doubled_half(a, one), (a + a * one) * 0.5, a, one);
    same("doubled_half", x_doubled_half(a, b), (a + a * b) * 0.5, a, b);
    same("half", x_half(a), a * 0.5, a, b);
    same("up", x_up(a, 1), a * 2.0, a, b);
    same("up", x_up(a, 2), a * 4.0, a, b);
    same("minmod", x_same_sign(a, b) ? x_nearer(a, b) : 0.0,
         a * b <= 0.0 ? 0.0 : a > 0.0 ? rmin(a, b) : rmax(a, b), a, b);
    c = 0.25 * (a + b);
    same("mc", x_same_sign(a, b) ? x_nearest(a, b, c) : 0.0,
         a * b <= 0.0 ? 0.0 : a > 0.0 ? rmin(a, rmin(b, c)) : rmax(a, rmax(b, c)), a, b);
}
int main()
{
    std::mt19937_64 g(11);
    const double edge[] = {0.0, -0.0, 1.0, -1.0, D(1), D(0xfffffffffffffull), D(0x10000000000000ull), D(0x7fefffffffffffffull),
                           1.0 / 0.0, -1.0 / 0.0, 0.0 / 0.0, D(0x3fefffffffffffffull), D(0x3ff0000000000001ull), 2.0, 3.0, 1e-200, 1e200, -1e-170};
    for (double a : edge) for (double b : edge) check(a, b, 0);
    for (long i = 0; i < 3000000; i++) {
        uint64_t x = g(), y = g();
        const uint64_t m = 0xfffffffffffffull;
        const int mode = i %% 8;
        if (mode < 6) {
            x = (x & (m | 1ull << 63)) | (uint64_t)(1023 - 40 + (x >> 52) %% 80) << 52;
            y = (y & (m | 1ull << 63)) | (uint64_t)(1023 - 40 + (y >> 52) %% 80) << 52;
        }
        if (mode == 1) y = (y & ~m) | g() %% 64;
        if (mode == 2) { y |= 0xfffffffff0000ull; x = (x & ~m) | g() %% 3; }
        if (mode == 3) x = (x & ~m) | ((y + g() %% 5 - 2) & m);
        if (mode == 4) { x &= ~0xffffffffull; y &= ~0xfffffffffull; }
        if (mode == 5) { x = (x & ~m) | (m - g() %% 4); y = (y & ~m) | (m - g() %% 4); }
        check(D(x), D(y), 0);
    }
    printf("bad %%ld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.parametrize("off", [0, 2])
def test_x64_equals_ieee(tmp_path, off):
    head = open(os.path.join(PKG, "csrc", "mhd_x64.h")).read()
    if off:
        a, b = "{ return 1.0f / f; }", "{ return 1.0f / sqrtf(f); }"
        assert a in head and b in head
        head = head.replace(a, "{ return x_float(x_bits(1.0f / f) + x_bits(f) % 5 - 2); }")
        head = head.replace(b, "{ return x_float(x_bits(1.0f / sqrtf(f)) + x_bits(f) % 5 - 2); }")
    (tmp_path / "x64.h").write_text(head)
    (tmp_path / "t.cpp").write_text(SRC % (tmp_path / "x64.h"))
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", str(tmp_path / "t.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
