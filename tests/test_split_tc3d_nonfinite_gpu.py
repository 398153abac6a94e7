"""Split 3D radius-1 sweeps on the tcgen05 kernel with an Inf or NaN in the
grid: the outputs that read it are not finite, and those whose tile does not see
it (16 rows x 64 columns, planes more than one away) are as without it, within the
split sweeps' bar of 1e-12."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def sweep(w, x):
    p = cs.Plan("box3d1r", x.shape, w, precision=cs.Precision.SPLIT)
    p.set_option(cs.Option.ALGO, cs.Algo.SPLIT_TC)
    raw = torch.from_numpy(p.pack(x)).cuda()
    a = torch.zeros(p.elements * 2, dtype=torch.float32, device="cuda")
    b = torch.zeros_like(a)
    p.split_from_fp64(raw, a)
    in_b = p.run(a, b, 1)
    p.split_to_fp64(b if in_b else a, raw)
    torch.cuda.synchronize()
    return p.unpack(raw.cpu().numpy())


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("at", [(4, 20, 100), (0, 0, 0), (8, 47, 149)])
def test_non_finite_points_stay_in_their_tiles(value, at):
    cs.build()
    x = O.splitmix_uniform(9 * 48 * 150, 8).reshape(9, 48, 150) - 0.5
    w = O.seeded_weights(27, 9)
    good = sweep(w, x)
    x[at] = value
    got = sweep(w, x)
    z, y, c = at
    near = tuple(slice(max(0, k - 1), k + 2) for k in at)
    assert not np.isfinite(got[near]).any()
    seen = np.zeros(x.shape, bool)  # the tiles whose windows (one point wider) hold the point
    for ty in range(0, 48, 16):
        for tx in range(0, 150, 64):
            if ty - 1 <= y <= ty + 16 and tx - 4 <= c <= tx + 67:
                seen[max(0, z - 1):z + 2, ty:ty + 16, tx:tx + 64] = True
    assert np.abs(got - good)[~seen].max() <= 1e-12 * np.abs(good).max()
