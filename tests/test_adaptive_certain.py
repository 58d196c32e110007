"""The adaptive test in single precision (verion_gb300/csrc/adaptive_test.h) never contradicts the test in double: pixels of
one radiance, of nearly one and of many, radiances from 1e-40 to 1e10, thresholds from zero to 10. Compiled with g++
from the header the kernels use."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "verion_gb300" / "csrc"

HARNESS = r"""
#include "adaptive_test.h"
#include <cmath>
#include <cstdio>
#include <random>
static int in_double(double n, double s1, double s2, float threshold)
{
    double mean = s1 / n, var = s2 / n - mean * mean;
    var = (var > 0.0 ? var : 0.0) * n / (n - 1.0);
    double m = mean > (double)0.05f ? mean : (double)0.05f;
    return std::sqrt(var / n) > (double)threshold * m;
}
int main()
{
    std::mt19937 rng(1);
    std::uniform_real_distribution<double> uni(0.0, 1.0);
    long sure = 0, trials = 1500000;
    for (long t = 0; t < trials; t++) {
        int n = 1 + (int)(rng() % 64), kind = (int)(rng() % 4);
        double scale = std::pow(10.0, -40.0 + 50.0 * uni(rng)), s1 = 0.0, s2 = 0.0;
        float base = (float)(scale * uni(rng));
        for (int i = 0; i < n; i++) {
            float l = kind == 0 ? base : kind == 1 ? (float)(base * (1.0 + 1e-3 * uni(rng))) : kind == 2 ? (float)(scale * uni(rng)) : 0.0f;
            s1 += (double)l;
            s2 += (double)l * (double)l;
        }
        float threshold = rng() % 4 == 0 ? 0.0f : (float)std::pow(10.0, -30.0 + 31.0 * uni(rng));
        if (rng() % 2)
            threshold = 0.02f;
        int a = vgd::adaptive_certain(n, s1, s2, threshold);
        if (a >= 0 && a != in_double(n, s1, s2, threshold)) {
            printf("n %d radiance %g threshold %g: %d\n", n, base, threshold, a);
            return 1;
        }
        sure += a >= 0;
    }
    return sure > trials / 2 ? 0 : 2;
}
"""


def test_single_precision_is_certain_or_says_so(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-O1", "-ffp-contract=off", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
