"""FP64 2D grids of odd pitch or odd first column on the tcgen05 digit kernels
(windows copied point by point instead of by TMA): caller layouts with
boundary values in both halos and huge values past them, against numpy. Bar:
1e-12 of the largest value, the FP64 paths' bar (a launch rounds at 2^-52 of its
tile's largest value, and at most 20 launches run here)."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 1e-12


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()


def steps_of(a, b, w, steps):
    """Grids with halos of the radius, ping-pong as cs_run: returns the interior."""
    a, b = a.copy(), b.copy()
    r = w.shape[0] // 2
    m, n = a.shape[0] - 2 * r, a.shape[1] - 2 * r
    for _ in range(steps):
        b[r:-r, r:-r] = sum(w[i, j] * a[i:i + m, j:j + n] for i in range(2 * r + 1) for j in range(2 * r + 1))
        a, b = b, a
    return a[r:-r, r:-r]


@pytest.mark.parametrize("shape,r,taps", [("box2d1r", 1, 9), ("box2d3r", 3, 49)])
@pytest.mark.parametrize("m,n,left,right", [(1031, 1409, 4, 4), (1088, 1408, 5, 6), (1025, 1537, 3, 4), (700, 2111, 7, 3)])
@pytest.mark.parametrize("steps", [1, 3, 8, 20])
def test_odd_pitches_and_first_columns(shape, r, taps, m, n, left, right, steps):
    top = 3
    ld = n + left + right
    assert ld % 2 or left % 2
    lay = {"dims": 2, "halo": r, "extent": [m, n], "pitch": [ld, 1], "origin": top * ld + left,
           "elements": (m + 2 * top) * ld}
    w = O.seeded_weights(taps, 3)
    p = cs.Plan(shape, (m, n), w, layout=lay)
    with pytest.raises(Exception):
        p.set_option(cs.Option.ALGO, cs.Algo.FP64_TC)  # a pin wants the even layouts
    rows, cols = slice(top - r, top + m + r), slice(left - r, left + n + r)
    grids = []
    for seed in (11, 12):
        g = np.full((m + 2 * top, ld), 1e200)
        g[rows, cols] = O.splitmix_uniform((m + 2 * r) * (n + 2 * r), seed).reshape(m + 2 * r, n + 2 * r)
        grids.append(g)
    ref = steps_of(grids[0][rows, cols], grids[1][rows, cols], w.reshape(2 * r + 1, -1), steps)
    da, db = (torch.from_numpy(g.reshape(-1)).cuda() for g in grids)
    in_b = p.run(da, db, steps)
    torch.cuda.synchronize()
    assert cs.device_wait_timeouts() == 0
    got, inner = (db if in_b else da).cpu().numpy().reshape(-1, ld), (slice(top, top + m), slice(left, left + n))
    if r == 3 or steps >= 8:
        assert p.algo == cs.Algo.FP64_TC, "the tensor cores are the faster here"
    assert np.abs(got[inner] - ref).max() <= TOL * np.abs(ref).max()
    outside = np.ones(got.shape, bool)
    outside[inner] = False
    assert (got[outside] == grids[1 if in_b else 0][outside]).all(), "only the interior is written"
