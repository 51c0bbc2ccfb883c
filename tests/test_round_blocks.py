"""The blocks per SM by which the surrogate map sizes its recompute rounds
(csrc/engine.cuh: blocks_by_shared_memory), on the CPU, against what
cudaOccupancyMaxActiveBlocksPerMultiprocessor says on a B200 (233 472 bytes an SM,
1024 reserved a block) on either side of a block more or less.  A round's points
follow from it, and with them which points a map recomputes.
"""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
OCCUPANCY = {37632: 6, 37872: 6, 37888: 6, 45568: 5, 45584: 4, 45600: 4, 45664: 4, 45696: 4, 57216: 4, 57344: 4}


def test_blocks_by_shared_memory(tmp_path):
    nvcc = Path("/usr/local/cuda/bin/nvcc")
    if not nvcc.exists():
        pytest.skip("nvcc not found")
    src = tmp_path / "blocks.cu"
    src.write_text('#include <cstdio>\n#include "engine.cuh"\nint main() {\n    for (long long b : {'
                   + ", ".join(f"{b}ll" for b in OCCUPANCY)
                   + '}) std::printf("%lld ", cbf::blocks_by_shared_memory(233472, b, 1024));\n}\n')
    exe = tmp_path / "blocks"
    subprocess.run([str(nvcc), "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    str(ROOT / "cudabifurcation3.0_b200" / "csrc"), "-I", str(ROOT / "include"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert list(map(int, out.split())) == list(OCCUPANCY.values())
