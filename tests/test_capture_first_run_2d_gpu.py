"""A plan's first run inside a caller's stream capture, for the plans whose tile or
time block the first run measures: FP64 2D (the FP64 FMA kernel's tiles) and
split 2D radius 1 and 1D (steps per double-float launch). In a process of its
own, where nothing is tuned; the replayed graph's result is the plain run's with
that kernel, bitwise."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

CODE = """
import numpy as np, torch, convstencil_gb300 as cs
shape, ext, prec = {shape!r}, {ext!r}, cs.Precision[{prec!r}]
w = np.random.default_rng(3).random(cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]][1])
w /= w.sum()
x = np.random.default_rng(4).random(ext)
split = prec == cs.Precision.SPLIT
def grids(p):
    raw = torch.from_numpy(p.pack(x)).cuda()
    a, b = raw.clone(), torch.zeros_like(raw)
    if split:
        p.split_from_fp64(raw, a)
    return a, b
p = cs.Plan(shape, ext, w, precision=prec)
a, b = grids(p)
g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
torch.cuda.synchronize()
with torch.cuda.graph(g, stream=s):
    in_b = p.run(a, b, 3, torch.cuda.current_stream())
g.replay()
torch.cuda.synchronize()
q = cs.Plan(shape, ext, w, precision=prec)
q.set_option(cs.Option.ALGO, cs.Algo.SPLIT_FMA if split else cs.Algo.FP64_FMA)
q.set_option(cs.Option.TIME_BLOCK if split else cs.Option.TILE_ROWS, 1 if split else 16)
c, d = grids(q)
in_d = q.run(c, d, 3)
torch.cuda.synchronize()
assert in_b == in_d and torch.equal(b if in_b else a, d if in_d else c)
a, b = grids(p)
p.run(a, b, 3)  # outside a capture it is measured as ever
torch.cuda.synchronize()
print("captured")
"""


@pytest.mark.parametrize("shape,ext,prec", [("star2d1r", (300, 333), "FP64"), ("box2d3r", (1200, 1040), "FP64"),
                                            ("star2d1r", (300, 333), "SPLIT"), ("1d1r", (70_001,), "SPLIT")])
def test_first_run_inside_a_capture(shape, ext, prec):
    import convstencil_gb300 as cs
    cs.build()
    code = CODE.format(shape=shape, ext=ext, prec=prec)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
