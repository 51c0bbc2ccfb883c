"""The peak finder's block form (PeakStream::push_block, csrc/peak_stream.cuh)
against its sample form (push), on the CPU: the header is host code too.

Every sequence over three levels -- so every pattern of rises, descents and
plateaus, at every position relative to the block edges -- of up to 11 samples
is fed in blocks of 4 (the rest sample by sample) and sample by sample; peaks,
intervals and counts must be the same.  The sample form itself is pinned to the
reference's peakFinder (cudaLibrary.cu:220-266) on the GPU.
"""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "peak_stream.cuh"
using namespace cbf;
constexpr int K = 4;
static int run(const std::vector<double>& d, bool blocks, double* pk, double* iv, int cap)
{
    PeakStream ps;
    NoPeakHook hook;
    ps.init();
    ps.push<true>(d[0], 0, pk, iv, cap, hook);
    int t = 0;
    const int n = (int)d.size();
    double ring[(K + 1) * 32];
    while (t + 1 < n) {
        if (blocks && t + K < n) {
            unsigned up = 0;
            for (int i = 0; i <= K; ++i) ring[32 * i] = d[t + i];
            for (int i = 0; i < K; ++i) up = (up << 1) | (d[t + i + 1] > d[t + i] ? 1u : 0u);
            ps.push_block<K, true>(up, t, K, d[t + K], ring, pk, iv, cap, hook);
            t += K;
        } else {
            ++t;
            ps.push<true>(d[t], t, pk, iv, cap, hook);
        }
    }
    return ps.emitted();
}
int main()
{
    long long sequences = 0, withPeaks = 0;
    for (int cap = 1; cap <= 8; cap += 7)
        for (int len = 1; len <= 11; ++len) {
            long long total = 1;
            for (int i = 0; i < len; ++i) total *= 3;
            for (long long code = 0; code < total; ++code) {
                std::vector<double> d(len);
                long long c = code;
                for (int i = 0; i < len; ++i) { d[i] = (double)(c % 3); c /= 3; }
                double p1[8] = {}, i1[8] = {}, p2[8] = {}, i2[8] = {};
                const int a = run(d, true, p1, i1, cap), b = run(d, false, p2, i2, cap);
                bool same = a == b;
                for (int k = 0; k < 8; ++k) same = same && p1[k] == p2[k] && i1[k] == i2[k];
                if (!same) { std::printf("differs: len %d code %lld: %d %d\n", len, code, a, b); return 1; }
                ++sequences;
                withPeaks += a > 0;
            }
        }
    std::printf("%lld %lld\n", sequences, withPeaks);
    return 0;
}
"""


def test_blocks_equal_samples_on_every_pattern(tmp_path):
    nvcc = Path("/usr/local/cuda/bin/nvcc")
    if not nvcc.exists():
        pytest.skip("nvcc not found")
    src = tmp_path / "peaks.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "peaks"
    subprocess.run([str(nvcc), "-O2", "-std=c++17", "-I", str(ROOT / "cudabifurcation3.0_b200" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    sequences, with_peaks = map(int, out.stdout.split())
    assert sequences == 2 * sum(3 ** n for n in range(1, 12)) and with_peaks > 10_000
