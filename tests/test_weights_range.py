"""Kernels of several steps of weights far from 1 in size: a step count is taken
only while its taps are normal numbers (cs_selfconv.h, on the CPU), and 1D runs
then agree with single steps (GPU; bar 1e-12 of the largest value, the FP64
paths' bar)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import convstencil_gb300 as cs

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "convstencil_gb300", "csrc")

CODE = r"""
#include "cs_selfconv.h"
#include <cstdio>

int main()
{
    const double one[3] = {0.3, 0.4, 0.3}, two[5] = {0.1, 0.2, 0.4, 0.25, 0.05};
    for (int r = 1; r <= 2; ++r)
        for (int e = -70; e <= 70; ++e)
            for (int t = 1; t * r <= 24; ++t) {
                double w[5], out[49], sum = 0.0, taps = 0.0;
                for (int i = 0; i <= 2 * r; ++i) sum += w[i] = std::ldexp(r == 1 ? one[i] : two[i], e);
                const bool ok = cs::selfconv(w, 1, r, t, 24, out);
                if (!ok && std::abs(e) < 64 && (std::abs(e) + 1) * t < 900) return printf("refused r %d e %d t %d\n", r, e, t), 1;
                if (!ok) continue;
                for (int i = 24 - t * r; i <= 24 + t * r; ++i) {
                    if (!std::isnormal(out[i])) return printf("tap %d: r %d e %d t %d\n", i, r, e, t), 1;
                    taps += out[i];
                }
                const double want = std::pow(sum, t);
                if (!(std::fabs(taps - want) <= 1e-13 * want)) return printf("sum: r %d e %d t %d\n", r, e, t), 1;
            }
    return 0;
}
"""


def test_taps_stay_normal_numbers(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "range.cpp", tmp_path / "range"
    src.write_text(CODE)
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("scale,data", [(46, -500), (60, -900), (-45, 500), (-47, 900)])
@pytest.mark.parametrize("n", [8192, 9001])
def test_1d_steps_of_large_and_small_weights(scale, data, n):
    torch = pytest.importorskip("torch")
    cs.build()
    w = np.array([0.3, 0.4, 0.3]) * 2.0 ** scale
    p = cs.Plan("1d1r", (n,), w)
    if n % 64 == 0:
        p.set_option(cs.Option.ALGO, cs.Algo.FP64_TC)
    x = np.random.default_rng(3).random(n) * 2.0 ** data
    a = torch.from_numpy(p.pack(x)).cuda()
    b = torch.zeros_like(a)
    in_b = p.run(a, b, 23)
    torch.cuda.synchronize()
    got = p.unpack((b if in_b else a).cpu().numpy())
    u = np.pad(x, 1)
    for _ in range(23):
        u[1:-1] = w[0] * u[:-2] + w[1] * u[1:-1] + w[2] * u[2:]
    assert np.abs(got - u[1:-1]).max() <= 1e-12 * np.abs(u).max() and np.abs(u).max() > 0
