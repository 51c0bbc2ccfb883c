"""The rises of a block of samples (RiseMask, csrc/peak_stream.cuh), built as the
kernels build them, on the CPU: the header is host code too.

Every sequence of up to 8 samples over five levels around zero -- both zeros, a
number below 2^-1042 and one on either side -- is fed in blocks of 1 to 4 samples and
sample by sample; peaks (to the bit: the sign of a zero counts), intervals and counts
must be the same.  A mask of the differences' signs alone takes -0 to +0 for a rise;
that the sequences show it is checked too.
"""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include "peak_stream.cuh"
using namespace cbf;
constexpr int K = 4;
// block 0: sample by sample; `plain`: the signs as they are
static int run(const std::vector<double>& d, int block, bool plain, double* pk, double* iv)
{
    PeakStream ps;
    NoPeakHook hook;
    ps.init();
    ps.push<true>(d[0], 0, pk, iv, 8, hook);
    int t = 0;
    const int n = (int)d.size();
    double ring[(K + 1) * 32];
    while (t + 1 < n) {
        if (block && t + block < n) {
            RiseMask<K> rises;
            rises.init();
            double p = ps.prev1;
            ring[0] = p;
            for (int i = 1; i <= block; ++i) {
                const double v = d[t + i];
                const int hi = rises.add(p, v);
                rises.seen(hi, hi);
                ring[32 * i] = p = v;
            }
            const unsigned up = plain ? rises.signs << (K - block) : rises.mask(block, ring);
            ps.push_block<K, true>(up, t, block, p, ring, pk, iv, 8, hook);
            t += block;
        } else {
            ++t;
            ps.push<true>(d[t], t, pk, iv, 8, hook);
        }
    }
    return ps.emitted();
}
int main()
{
    const double level[5] = {-0.0, 0.0, 1.0, -1.0, 0x1p-1060};
    long long sequences = 0, withPeaks = 0, signsFail = 0;
    for (int len = 1; len <= 8; ++len) {
        long long total = 1;
        for (int i = 0; i < len; ++i) total *= 5;
        for (long long code = 0; code < total; ++code) {
            std::vector<double> d(len);
            long long c = code;
            for (int i = 0; i < len; ++i) { d[i] = level[c % 5]; c /= 5; }
            double p0[8] = {}, i0[8] = {};
            const int a = run(d, 0, false, p0, i0);
            for (int block = 1; block <= K; ++block) {
                for (int plain = 0; plain < 2; ++plain) {
                    double p1[8] = {}, i1[8] = {};
                    const int b = run(d, block, plain, p1, i1);
                    const bool same = a == b && !memcmp(p0, p1, sizeof p0) && !memcmp(i0, i1, sizeof i0);
                    if (plain) signsFail += !same;
                    else if (!same) { std::printf("differs: len %d code %lld block %d: %d %d\n", len, code, block, a, b); return 1; }
                }
                ++sequences;
                withPeaks += a > 0;
            }
        }
    }
    std::printf("%lld %lld %lld\n", sequences, withPeaks, signsFail);
    return 0;
}
"""


def test_blocks_equal_samples_around_zero(tmp_path):
    nvcc = Path("/usr/local/cuda/bin/nvcc")
    if not nvcc.exists():
        pytest.skip("nvcc not found")
    src = tmp_path / "rises.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "rises"
    subprocess.run([str(nvcc), "-O2", "-std=c++17", "-I", str(ROOT / "cudabifurcation3.0_b200" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    sequences, with_peaks, signs_fail = map(int, out.stdout.split())
    assert sequences == 4 * sum(5 ** n for n in range(1, 9)) and with_peaks > 1000
    assert signs_fail > 0
