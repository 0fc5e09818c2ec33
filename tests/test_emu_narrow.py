"""emu_d2f (the binning's double-to-float conversion on the integer pipes) must
return the host's conversion bit for bit: ordinary values, exponents around
both ends of FP32's range, ties and halfway neighbours, infinities and NaN."""
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
    for (int64_t i = 0; i < 6000000; i++) {
        const uint64_t r = mix64(i), e = mix64(i ^ 0x55555), m = r & 0x800FFFFFFFFFFFFFull;
        double x;
        switch (i %% 5) {
        case 0: x = emu_double(r); break;
        case 1: x = emu_double(m | ((900 + e %% 250) << 52)); break;
        case 2: x = emu_double((r & 0x800FFFFFE0000000ull) | ((e %% 4) << 27) | ((880 + e %% 300) << 52)); break;
        case 3: x = emu_double((r & 0x800FFFFFE0000000ull) | (0x10000000u + (e %% 3) - 1) | ((1000 + e %% 40) << 52)); break;
        default: x = emu_double(m | ((1140 + e %% 20) << 52));
        }
        bad += !samef(emu_d2f(x), (float)x);
    }
    const double ends[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 0x1.fffffefffffffp127, 0x1.ffffffp127, 0x1p-126, 0x1.fffffffp-127};
    for (double x : ends) bad += !samef(emu_d2f(x), (float)x);
    std::printf("differing %%lld\n", bad);
    return bad != 0;
}
"""


def test_narrowing_matches_the_host(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "narrow.cpp", str(tmp_path / "narrow")
    src.write_text(SRC % os.path.join(HERE, "emu_host_check.cpp"))
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I", HERE, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
