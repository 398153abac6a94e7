"""Host-buffer runs in bands on odd layouts (odd pitch or first column): bitwise
the device path of one step per launch, with rows of very different size on
either side of the bands' cuts (a tile's scale is set by all of its window)."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape,r,taps", [("box2d1r", 1, 9), ("box2d3r", 3, 49)])
@pytest.mark.parametrize("left,right", [(4, 5), (5, 5)])
def test_odd_layouts_in_bands(shape, r, taps, left, right):
    cs.build()
    m, n = 2048, 2048
    ld = n + left + right
    lay = {"dims": 2, "halo": r, "extent": [m, n], "pitch": [ld, 1], "origin": 3 * ld + left, "elements": (m + 6) * ld}
    w = O.seeded_weights(taps, 5)
    p = cs.Plan(shape, (m, n), w, layout=lay)
    x = np.random.default_rng(6).random((m + 6, ld))
    x[3:-3] *= 2.0 ** (np.random.default_rng(7).integers(-9, 9, (m, 1)))
    buf = torch.from_numpy(x.reshape(-1)).cuda()
    warm = [buf.clone(), torch.zeros_like(buf)]
    p.run(*warm, 1)  # the kernel is known from here on
    assert p.algo == cs.Algo.FP64_TC, "the tensor cores are the faster here"
    for steps in (1, 2, 4):
        q = cs.Plan(shape, (m, n), w, layout=lay)
        q.set_option(cs.Option.TIME_BLOCK, 1)
        a, b = buf.clone(), torch.zeros_like(buf)
        in_b = q.run(a, b, steps)
        dev = (b if in_b else a).cpu().numpy()
        host = p.run_host(x.reshape(-1), steps)
        inner = p.interior_index().reshape(-1)
        np.testing.assert_array_equal(host[inner], dev[inner])
    assert cs.device_wait_timeouts() == 0
