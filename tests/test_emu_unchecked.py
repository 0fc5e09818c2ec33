"""The unchecked integer-pipe operations that the FP64 kernels call behind their
range tests (products, quotients, thirds, square roots, 1 - x), compiled for the
host, must return the host's IEEE results over the ranges those tests admit, with
quotients and roots next to rounding midpoints among them; squares over every
number."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

SRC = r"""
#define main check_main
#include "%s"
#undef main
int main() {
    long long bad = 0;
    for (int64_t i = 0; i < 4000000; i++) {
        const uint64_t r = mix64(i), s = mix64(i ^ 0x55555), e = mix64(i + (1ll << 40));
        const uint64_t fm = i %% 3 ? kEmuFrac : 0x000FFFFFC0000000ull;
        const double a = normal(r, 523 + e %% 1001, fm), b = normal(s, 523 + (e >> 10) %% 1001, fm);
        bad += !same(emu_mul_n(a, b), a * b);
        double n = normal(r, 223 + (e >> 20) %% 1601, fm), d = normal(s, 823 + (e >> 31) %% 401, fm);
        if (i & 1) n = emu_double((emu_bits(d * normal(r, 1023)) + (e >> 60) %% 5 - 2));
        bad += !same(emu_div_n(n, emu_divisor(d)), n / d);
        double x = emu_double(((1 + (e >> 42) %% 2046) << 52) | (r & kEmuFrac));
        if (i & 2) { const double q = normal(r & kEmuFrac, 600 + e %% 800); x = emu_double(emu_bits(q * q) + s %% 5 - 2); }
        bad += !same(emu_sqrt_n(x), std::sqrt(x));
        double t = emu_double(((1022 - (e >> 53) %% 162) << 52) | (r & kEmuFrac));
        if (i & 4) t = 3.0 * emu_double(((1000 - (e >> 53) %% 140) << 52) | (s & kEmuFrac));
        bad += !same(emu_div3_n(t), t / 3.0);
        const double h = emu_double((1022ull << 52) | (i %% 5 ? r & kEmuFrac : kEmuFrac - (r %% 5000000)));
        bad += !same(emu_one_minus_n(h), 1.0 - h);
        const double any = emu_double(r);
        bad += !same(emu_sq(any), any * any);
    }
    const double ends[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 0x1p-500, 0x1p-501, 0x1p500, 0x1.fffffffffffffp499, 0x1p-1074};
    for (double x : ends) bad += !same(emu_sq(x), x * x);
    std::printf("differing %%lld\n", bad);
    return bad != 0;
}
"""


def test_unchecked_operations_match_the_host(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "unchecked.cpp", str(tmp_path / "unchecked")
    src.write_text(SRC % os.path.join(HERE, "emu_host_check.cpp"))
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I", HERE, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
