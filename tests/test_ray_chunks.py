"""The split of large ray queries into launches (verion_gb300/csrc/ray_chunks.h): the launches take every ray once,
and no launch's 32-bit work counter can wrap, up to the most rays that the entry points take. Compiled with
g++ from the header the library uses."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "verion_gb300" / "csrc"

HARNESS = r"""
#include "ray_chunks.h"
#include <cstdio>
using namespace vgx;
int main()
{
    const uint32_t C = RAY_CHUNK;
    const uint32_t counts[] = {0, 1, 31, 1000003, C - 1, C, C + 1, 2 * C, 3 * C + 7, 0x7fffffffu, 0xfffffff0u, 0xffffffffu};
    for (uint32_t n : counts) {
        uint64_t next = 0;
        for (uint32_t k = 0; k < ray_chunks(n); k++) {
            RayChunk q = ray_chunk(n, k);
            // What the counter can reach: every ray, and 32 more for each warp.
            if (q.at != next || q.n == 0 || (uint64_t)q.n + 32ull * RAY_QUERY_WARPS > 0xffffffffull)
                return 1;
            next += q.n;
        }
        if (next != n)
            return 2;
    }
    // A full GB300 (152 SMs, 16 blocks of 4 warps on each) is within the bound on warps.
    return 152 * 16 * 4 <= RAY_QUERY_WARPS ? 0 : 3;
}
"""


def test_launches_cover_the_rays_and_counters_cannot_wrap(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
