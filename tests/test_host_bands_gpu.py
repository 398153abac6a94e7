"""Host-buffer runs in skewed bands: a band's sweeps run one after the other on
slabs that move up a tile per sweep, from fewer sweeps than bands to more than
a band has tiles. Each kernel's result must be bitwise the device path's, as
every cut is a multiple of its tiles (2D widths odd and even, 3D, both
precisions, boundary values in the first grid's halo)."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()


CASES = [("box2d3r", (4100, 2050), cs.Precision.FP64, cs.Algo.FP64_TC),
         ("box2d3r", (4100, 2050), cs.Precision.SPLIT, cs.Algo.SPLIT_TC),
         ("box2d3r", (3001, 4096), cs.Precision.FP64, cs.Algo.FP64_FMA),
         ("star2d1r", (4096, 2000), cs.Precision.FP64, cs.Algo.FP64_TC),
         ("star3d1r", (300, 150, 130), cs.Precision.FP64, cs.Algo.FP64_FMA),
         ("box3d1r", (333, 190, 130), cs.Precision.FP64, cs.Algo.FP64_TC),
         ("box3d1r", (300, 190, 130), cs.Precision.SPLIT, cs.Algo.SPLIT_TC)]


@pytest.mark.parametrize("shape,ext,prec,algo", CASES)
@pytest.mark.parametrize("steps", [1, 2, 5, 12])
def test_skewed_bands_equal_device_run(shape, ext, prec, algo, steps):
    info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
    w = O.seeded_weights(info[1], 40 + steps)
    p = cs.Plan(shape, ext, w, precision=prec)
    p.set_option(cs.Option.ALGO, algo)
    buf = O.splitmix_uniform(p.elements, 41)  # halo included
    raw = torch.from_numpy(buf).cuda()
    a, b = raw.clone(), torch.zeros_like(raw)
    if prec == cs.Precision.SPLIT:
        p.split_from_fp64(raw, a)
    elif algo == cs.Algo.FP64_TC and shape == "star2d1r":
        q = cs.Plan(shape, ext, w, precision=prec)  # one step at a time, as bands do
        q.set_option(cs.Option.ALGO, algo)
        q.set_option(cs.Option.TIME_BLOCK, 1)
        in_b = q.run(a, b, steps)
    if not (algo == cs.Algo.FP64_TC and shape == "star2d1r"):
        in_b = p.run(a, b, steps)
    dev = b if in_b else a
    if prec == cs.Precision.SPLIT:
        p.split_to_fp64(dev, raw)
        dev = raw
    torch.cuda.synchronize()
    inner = p.interior_index().reshape(-1)
    for _ in range(2):
        host = p.run_host(buf, steps)
        np.testing.assert_array_equal(host[inner], dev.cpu().numpy()[inner])
    assert cs.device_wait_timeouts() == 0
