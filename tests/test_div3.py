"""Three quotients by one denominator (dem_div.cuh) have the bits of three divisions: the header compiled
for the host, on random mantissas, hard cases next to a rounding boundary, zeros of both signs, and the
values outside its range (tiny, huge, infinite, NaN)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "cabanadem_b200", "csrc")

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
static int __double2hiint(double v) { uint64_t b; std::memcpy(&b, &v, 8); return (int)(b >> 32); }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
#include "dem_div.cuh"
static uint64_t bits(double v) { uint64_t b; std::memcpy(&b, &v, 8); return v != v ? 1 : b; }
int main() {
    std::mt19937_64 rng(7);
    long bad = 0;
    auto check = [&](double a0, double a1, double a2, double b) {
        volatile double x = a0 / b, y = a1 / b, z = a2 / b;
        double q0, q1, q2;
        b200dem::div3(a0, a1, a2, b, q0, q1, q2);
        if (bits(q0) != bits(x) || bits(q1) != bits(y) || bits(q2) != bits(z))
            if (bad++ < 5) std::printf("%a %a %a / %a: %a %a %a\n", a0, a1, a2, b, q0, q1, q2);
    };
    auto value = [&](int span) {
        const double m = 1.0 + (double)(rng() >> 12) * 0x1p-52;
        return std::ldexp(rng() & 1 ? m : -m, (int)(rng() % (2 * span + 1)) - span);
    };
    for (int k = 0; k < 3000000; ++k) check(value(40), value(40), value(40), value(40));
    for (int k = 0; k < 500000; ++k) check(value(540), value(540), value(3), value(540));
    for (int k = 0; k < 1000000; ++k) {   // numerators next to a product: quotients next to a double or a midpoint
        const double b = k % 2 ? value(3) : std::nextafter(std::ldexp(2.0, k % 5), 0.0) - (k % 97) * 0x1p-50, q = value(3);
        const double a = q * b, mid = (q + std::nextafter(q, 4.0)) * 0.5;
        check(std::nextafter(a, 1e9), std::nextafter(a, -1e9), std::fma(mid, b, q * b * 0x1p-54), b);
    }
    const double edge[] = {0.0, -0.0, 1.0, -1.0, 5e-324, -2.2250738585072014e-308, 1e-160, 1e-151, 1e150, 1e151, -1.7976931348623157e308,
                           std::ldexp(1.0, -500), std::ldexp(1.0, 499), std::ldexp(1.0, 500), INFINITY, -INFINITY, NAN, 3.0};
    for (double a : edge)
        for (double b : edge)
            for (double c : edge) check(a, c, 0.3, b);
    std::printf("bad %ld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="no host compiler")
def test_div3_has_the_bits_of_three_divisions(tmp_path):
    src = tmp_path / "div3.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "div3"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
