"""A host-buffer run gives the same bits every time: the first call of a kind, whose
kernel is not known yet and which runs whole, and the later ones, which may
run in bands of one step per launch. In a process of its own, where nothing is
tuned; FP64 2D radius 1 is the kind that may take three steps per launch."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

CODE = """
import numpy as np, convstencil_gb300 as cs
shape, ext = {shape!r}, {ext!r}
w = np.random.default_rng(3).random(cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]][1])
w /= w.sum()
p = cs.Plan(shape, ext, w)
x = p.pack(np.random.default_rng(4).random(ext))
for steps in (5, 12):
    got = [p.run_host(x, steps).copy() for _ in range(3)]
    assert all(np.array_equal(got[0], g) for g in got[1:]), steps
print("equal", p.algo)
"""


@pytest.mark.parametrize("shape,ext", [("star2d1r", (4096, 2000)), ("box2d1r", (3000, 2801)), ("box3d1r", (200, 190, 130))])
def test_first_and_later_calls_agree(shape, ext):
    import convstencil_gb300 as cs
    cs.build()
    r = subprocess.run([sys.executable, "-c", CODE.format(shape=shape, ext=ext)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "equal" in r.stdout, r.stderr[-2000:]
