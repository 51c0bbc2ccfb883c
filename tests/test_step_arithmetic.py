"""The 5-D model's divisions (csrc/systems.cuh) against a / b, on the CPU (the header
is host code too): by a constant, for dividends of its range and quotients next to
rounding boundaries; of zeros; and the whole step against the literal one for states
of every kind, zeros, infinities, NaNs and subnormals among them.  Bit for bit.
"""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <cmath>
#include "systems.cuh"
static uint64_t s = 0x9E3779B97F4A7C15ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double bits(uint64_t b) { double v; memcpy(&v, &b, 8); return v; }
static uint64_t raw(double v) { uint64_t b; memcpy(&b, &v, 8); return b; }
static bool same(double a, double b) { return raw(a) == raw(b) || (a != a && b != b); }
static double near(int e) { return bits((rnd() & 0x800fffffffffffffull) | ((uint64_t)(1023 + e) << 52)); }
int main()
{
    using cbf::Memristive5;
    long long n = 0;
    auto usable = [](double a) { return cbf::operand_place(a) < cbf::kOperandSpan; };
    auto check = [&](double a, double b) {
        if (!usable(a) || !cbf::divisor_in_range(b)) return true;
        const double q = cbf::divide(a, cbf::ConstDivisor{b, 1.0 / b}), w = a / b;
        ++n;
        if (!same(q, w)) { std::printf("divide %a / %a = %a, not %a\n", a, b, q, w); return false; }
        return true;
    };
    const double odd[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 4.9e-324, -2.2e-308, 1.7e308, 0x1p-200,
                          -0x1.fffffffffffffp-201, 0x1.fffffffffffffp199, 0x1p200, -0x1p-149, 3.4e38};
    for (double a : odd)
        if (usable(a) != (a == 0 || (fabs(a) >= 0x1p-200 && fabs(a) < 0x1p200))) { std::printf("range of %a\n", a); return 1; }
    for (int i = 0; i < 4000000; ++i) {
        const double b = near((int)(rnd() % 9) - 4);
        if (!check(near((int)(rnd() % 40) - 20), b)) return 1;
        // a quotient one unit of 2^-54 away from halfway between two doubles
        const double q = near(0), mid = q + bits(raw(q) + 1);
        const double a = (mid * 0.5) * b;
        if (!check(a, b) || !check(bits(raw(a) + 1), b) || !check(bits(raw(a) - 1), b)) return 1;
        if (!check(near((int)(rnd() % 400) - 200), bits(rnd()))) return 1;
        // divisors as the model has them, 1 + h1 a
        if (!check(near((int)(rnd() % 60) - 50), 1.0 + 0.0025 * (double)(i % 4001) * 0.01)) return 1;
        const double all1 = bits(raw(near(0)) | 0xfffffffffffffull);
        if (!check(near(0), all1)) return 1;
    }
    for (double a : odd) {
        for (double b : odd) {
            ++n;
            if (!same(cbf::divide_maybe_zero(a, b), a / b)) { std::printf("%a / %a\n", a, b); return 1; }
        }
        if (!check(a, 1.0175) || !check(a, -0.3)) return 1;
    }
    // whole steps: model parameters, and parameters and states out of the ordinary
    for (int i = 0; i < 400000; ++i) {
        double a[8] = {8, 35, 15, 0.01, -1.6676, 0.0676, 0.3682, 0.5}, x[5], y[5];
        for (int k = 0; k < 8; ++k)
            if (rnd() % 16 == 0) a[k] = rnd() % 3 ? near((int)(rnd() % 80) - 40) : odd[rnd() % 16];
        for (int k = 0; k < 5; ++k) x[k] = y[k] = rnd() % 8 ? near((int)(rnd() % 8) - 4)
                                                : rnd() % 2 ? near((int)(rnd() % 300) - 150) : odd[rnd() % (i % 2 ? 2 : 16)];
        if (i % 50 == 0) for (int k = 0; k < 5; ++k) x[k] = y[k] = odd[rnd() % 2];
        const auto c = Memristive5::prep(a, i % 7 ? 0.005 : near((int)(rnd() % 40) - 30));
        for (int t = 0; t < 8; ++t) {
            Memristive5::step(x, c);
            Memristive5::evaluate<true>(y, c);
            for (int k = 0; k < 5; ++k)
                if (!same(x[k], y[k])) { std::printf("step %d: x[%d] %a, not %a\n", t, k, x[k], y[k]); return 1; }
            ++n;
        }
    }
    std::printf("%lld\n", n);
    return 0;
}
"""


def test_divisions_and_steps(tmp_path):
    nvcc = Path("/usr/local/cuda/bin/nvcc")
    if not nvcc.exists():
        pytest.skip("nvcc not found")
    src = tmp_path / "arith.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "arith"
    subprocess.run([str(nvcc), "-O2", "-std=c++17", "-fmad=false", "-Xcompiler", "-ffp-contract=off,-mfma", "-I",
                    str(ROOT / "cudabifurcation3.0_b200" / "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout) > 20_000_000
