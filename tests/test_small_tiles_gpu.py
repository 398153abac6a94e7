"""The FP64 FMA 2D kernel's small tiles (16 rows of 8 columns, grids of few
points) sum every point's taps in the order of the 64-column tiles: bitwise
equal, at the edges of a tile and beyond it."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape,fused", [("star2d1r", 0), ("box2d1r", 0), ("star2d3r", 0), ("box2d3r", 0),
                                         ("star2d1r", 1)])
@pytest.mark.parametrize("ext", [(1, 1), (15, 7), (16, 8), (17, 9), (96, 130), (33, 700), (500, 513)])
def test_small_tiles_equal_wide_tiles(shape, fused, ext):
    cs.build()
    info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
    if fused:  # three steps of a cross: a diamond of 25 taps
        base = np.zeros(9)
        base[[1, 3, 4, 5, 7]] = O.seeded_weights(5, 3)
        w = cs.selfconv(base, 2, 1, 3)
    else:
        w = O.seeded_weights(info[1], 3)
    outs = []
    for rows in (0, 16):  # 0: the small tiles at these sizes
        p = cs.Plan(shape, ext, w, semantics=cs.Semantics.FUSED if fused else cs.Semantics.STEP)
        p.set_option(cs.Option.ALGO, cs.Algo.FP64_FMA)
        p.set_option(cs.Option.TILE_ROWS, rows)
        a = torch.from_numpy(p.pack(O.splitmix_uniform(ext[0] * ext[1], 4).reshape(ext))).cuda()
        b = torch.zeros_like(a)
        in_b = p.run(a, b, 9)
        torch.cuda.synchronize()
        outs.append((b if in_b else a).cpu().numpy())
    np.testing.assert_array_equal(outs[0], outs[1])
