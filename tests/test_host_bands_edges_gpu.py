"""Host-buffer runs in bands whose height, rounded up to the kernels' tiles,
leaves a last copy of few slabs or of the halo alone: bitwise the device path,
call after call with another grid and another halo (the device grids are kept
between calls, so a read before its copy would see the call before)."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()


@pytest.mark.parametrize("shape,ext,prec,algo", [
    ("box2d3r", (800, 8192), cs.Precision.FP64, cs.Algo.FP64_TC),
    ("box2d3r", (800, 8192), cs.Precision.SPLIT, cs.Algo.SPLIT_TC),
    ("box2d3r", (641, 8192), cs.Precision.FP64, cs.Algo.FP64_FMA),
    ("box3d1r", (100, 512, 512), cs.Precision.FP64, cs.Algo.FP64_TC),
    ("box3d1r", (97, 512, 512), cs.Precision.SPLIT, cs.Algo.SPLIT_TC),
    ("star3d1r", (81, 512, 512), cs.Precision.FP64, cs.Algo.FP64_FMA)])
@pytest.mark.parametrize("steps", [1, 2])
def test_short_last_copies(shape, ext, prec, algo, steps):
    info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
    p = cs.Plan(shape, ext, O.seeded_weights(info[1], 3), precision=prec)
    p.set_option(cs.Option.ALGO, algo)
    for seed in (5, 6):
        raw = torch.rand(p.elements, dtype=torch.float64, device="cuda",  # halo included
                         generator=torch.Generator("cuda").manual_seed(seed))
        buf = raw.cpu().numpy()
        host = p.run_host(buf, steps)
        a, b = raw.clone(), torch.zeros_like(raw)
        if prec == cs.Precision.SPLIT:
            p.split_from_fp64(raw, a)
        in_b = p.run(a, b, steps)
        dev = b if in_b else a
        if prec == cs.Precision.SPLIT:
            p.split_to_fp64(dev, raw)
            dev = raw
        inner = torch.from_numpy(p.interior_index().reshape(-1))
        assert torch.equal(torch.from_numpy(host)[inner], dev.cpu()[inner])
        if steps % 2 == 0 and prec == cs.Precision.FP64:  # the halo of the first grid comes back too
            outside = torch.ones(p.elements, dtype=torch.bool)
            outside[inner] = False
            assert torch.equal(torch.from_numpy(host)[outside], torch.from_numpy(buf)[outside])
    assert cs.device_wait_timeouts() == 0
