"""The plain form's division and square root on integers (csrc/mhd_x64.h) as the
GPU computes them, from its approximate reciprocal and root, against the GPU's
own IEEE division and square root, bit for bit: random significands and those at
either end, quotients next to 1, every leading 24 bits of a divisor and of a
radicand of either parity, and exponents to both ends of the range."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cstdio>
#include "mhd_x64.h"
using namespace mhd;
typedef unsigned long long u64;
struct Bad { unsigned n; double a, b, got, want; };
__device__ u64 rnd(u64 &s)   /* splitmix64 */
{
    u64 z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ z >> 30) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ z >> 27) * 0x94d049bb133111ebull;
    return z ^ z >> 31;
}
__device__ double D(u64 u) { return __longlong_as_double((long long)u); }
__device__ u64 B(double a) { return (u64)__double_as_longlong(a); }
__device__ void same(Bad *bad, double got, double want, double a, double b)
{
    if (B(got) == B(want) || (got != got && want != want)) return;
    if (atomicAdd(&bad->n, 1u) == 0) { bad->a = a; bad->b = b; bad->got = got; bad->want = want; }
}
__global__ void check(Bad *bad, int lead)
{
    const u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x, m = 0xfffffffffffffull;
    u64 s = t * 0x1234567ull + 99;
    for (int i = 0; i < 16; i++) {
        u64 x = rnd(s), y = rnd(s);
        const int mode = lead ? 8 : i % 8;
        if (mode != 7) {
            x = (x & (m | 1ull << 63)) | (u64)(1023 - 40 + (x >> 52) % 80) << 52;
            y = (y & (m | 1ull << 63)) | (u64)(1023 - 40 + (y >> 52) % 80) << 52;
        }
        if (mode == 1) y = (y & ~m) | rnd(s) % 64;
        if (mode == 2) { y |= 0xfffffffff0000ull; x = (x & ~m) | rnd(s) % 3; }
        if (mode == 3) x = (x & ~m) | ((y + rnd(s) % 5 - 2) & m);
        if (mode == 4) { x &= ~0xffffffffull; y &= ~0xfffffffffull; }
        if (mode == 5) { x = (x & ~m) | (m - rnd(s) % 4); y = (y & ~m) | (m - rnd(s) % 4); }
        if (mode == 8) {   /* leading bits t (23 of them), the rest at an end or random */
            const u64 tail = i % 3 == 0 ? 0 : i % 3 == 1 ? 0x1fffffffull : rnd(s) & 0x1fffffffull;
            y = (y & ~m) | (t & 0x7fffffull) << 29 | tail;
        }
        const double a = D(x), b = D(y), r = fabs(b);
        same(bad, x_div(a, b), a / b, a, b);
        same(bad, x_sqrt(r), sqrt(r), r, 0.0);
        same(bad, x_sqrt(2.0 * r), sqrt(2.0 * r), 2.0 * r, 0.0);
    }
}
int main()
{
    Bad *bad, h;
    if (cudaMalloc(&bad, sizeof h) != cudaSuccess || cudaMemset(bad, 0, sizeof h) != cudaSuccess) return 2;
    for (int lead = 0; lead < 2; lead++) check<<<32768, 256>>>(bad, lead);   /* 2^23 threads */
    if (cudaMemcpy(&h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    printf("bad %u: %a, %a: %a, want %a\n", h.n, h.a, h.b, h.got, h.want);
    return h.n != 0;
}
"""


def test_division_and_root_on_the_gpu_are_ieee(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "t.cu").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--fmad=false",
                           "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-I", os.path.join(PKG, "csrc"),
                           str(tmp_path / "t.cu"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
