"""A plan's first run inside a caller's stream capture: no timing run is
possible there, so plans whose kernel is not known yet take FP64 FMA (1D arrays
and 3D radius-3 grids; in a process of its own, where nothing is tuned). The
replayed graph's result is the plain run's with that kernel, bitwise."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

CODE = """
import numpy as np, torch, convstencil_gb300 as cs
shape, ext, fused = {shape!r}, {ext!r}, {fused}
info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
w = np.random.default_rng(3).random(info[2] if fused else info[1])
w /= w.sum()
p = cs.Plan(shape, ext, w, semantics=cs.Semantics(fused))
x = p.pack(np.random.default_rng(4).random(ext))
a, b = torch.from_numpy(x).cuda(), torch.zeros(p.elements, dtype=torch.float64, device="cuda")
steps = 3 * ({per} if fused else 1)
g = torch.cuda.CUDAGraph()
s = torch.cuda.Stream()
torch.cuda.synchronize()
with torch.cuda.graph(g, stream=s):
    in_b = p.run(a, b, steps, torch.cuda.current_stream())
a.copy_(torch.from_numpy(x))
b.zero_()
g.replay()
torch.cuda.synchronize()
got = (b if in_b else a).cpu().numpy()
q = cs.Plan(shape, ext, w, semantics=cs.Semantics(fused))
q.set_option(cs.Option.ALGO, cs.Algo.FP64_FMA)
c, d = torch.from_numpy(x).cuda(), torch.zeros(p.elements, dtype=torch.float64, device="cuda")
in_d = q.run(c, d, steps)
torch.cuda.synchronize()
assert in_b == in_d and (got == (d if in_d else c).cpu().numpy()).all()
print("captured")
"""


@pytest.mark.parametrize("shape,ext,fused,per", [("1d1r", (70_001,), 0, 1), ("1d2r", (9_999,), 1, 2),
                                                 ("box3d1r", (20, 24, 33), 1, 3)])
def test_first_run_inside_a_capture(shape, ext, fused, per):
    import convstencil_gb300 as cs
    cs.build()
    code = CODE.format(shape=shape, ext=ext, fused=fused, per=per)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
