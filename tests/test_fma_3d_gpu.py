"""The FP64 FMA kernel of 3D radius-1 grids (an output a thread) against numpy,
at the edges of its 4 x 32 tiles and on grids of more planes, rows or tiles than
a grid axis holds. Bar: 27 products and their sum round by at most 27 * 2^-53 of
the sum of |weight x value| each sweep, which is the result here (all
positive); 3 sweeps stay below 1e-14."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape,taps", [("star3d1r", 7), ("box3d1r", 27)])
@pytest.mark.parametrize("ext", [(1, 1, 1), (2, 3, 31), (5, 4, 32), (3, 5, 33), (17, 70, 65), (70_000, 2, 3),
                                 (2, 270_000, 3), (2, 1, 70_000)])
def test_fma_3d_equals_numpy(shape, taps, ext):
    cs.build()
    w = O.seeded_weights(taps, 5)
    w = w / w.sum()
    dense = (O.star3d1r_to_dense(w) if shape == "star3d1r" else w).reshape(3, 3, 3)
    p = cs.Plan(shape, ext, w)
    p.set_option(cs.Option.ALGO, cs.Algo.FP64_FMA)
    x = O.splitmix_uniform(int(np.prod(ext)), 6).reshape(ext)
    a = torch.from_numpy(p.pack(x)).cuda()
    b = torch.zeros_like(a)
    in_b = p.run(a, b, 3)
    torch.cuda.synchronize()
    got = p.unpack((b if in_b else a).cpu().numpy())
    for _ in range(3):
        g = np.pad(x, 1)
        x = sum(dense[i, j, k] * g[i:i + ext[0], j:j + ext[1], k:k + ext[2]]
                for i in range(3) for j in range(3) for k in range(3))
    assert np.abs(got - x).max() <= 1e-14 * np.abs(x).max()
