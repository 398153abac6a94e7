"""Values that fall by a factor 2^16 to 2^64 within a tile, in the tcgen05 forms
that AUTO takes in the place of FP64 FMA sweeps: one launch stays within the
format's error, relative to its tile's largest value M (weights of sum 1). Bar:
2^-50 M; inputs round at 2^-53 M, outputs at 2^-53 of themselves, and what the
dropped digits weigh is below 2^-53 M (49 taps, 2^-63 of digit products up to
2^16 each), together below 2^-51 M, and the reference's own rounding below that.
Where M is subnormal (the end of one 1D ramp) single steps round each of their
products to the smallest subnormal: 64 of those, at 11 steps of 5 taps."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()


@pytest.mark.parametrize("shape,ext,fused,steps,odd,tile,reach,fall", [
    ("box2d3r", (700, 1111), 0, 1, True, 64, 4, 4), ("star2d1r", (1024, 1030), 0, 3, False, 64, 4, 2),
    ("1d2r", (100_001,), 0, 11, False, 4096, 24, 64), ("1d1r", (100_001,), 0, 23, False, 4096, 24, 256),
    ("box3d1r", (24, 40, 500), 1, 3, False, 64, 4, 1)])
def test_error_is_relative_to_the_tile(shape, ext, fused, steps, odd, tile, reach, fall):
    info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
    w = O.seeded_weights(info[1 + fused], 71)
    w /= w.sum() * (1.9 if fused else 1)  # the box's planes count twice but one
    n = ext[-1]
    amp = 2.0 ** -(np.arange(n) / fall)
    x = (O.splitmix_uniform(int(np.prod(ext)), 72).reshape(ext) - 0.5) * amp
    kw = {}
    if odd:
        ld = n + 9
        kw["layout"] = {"dims": 2, "halo": 3, "extent": list(ext), "pitch": [ld, 1], "origin": 3 * ld + 5,
                        "elements": (ext[0] + 6) * ld}
    out = []
    for algo in (cs.Algo.AUTO, cs.Algo.FP64_FMA):
        p = cs.Plan(shape, ext, w, semantics=cs.Semantics(fused), **kw)
        p.set_option(cs.Option.ALGO, algo)
        a = torch.from_numpy(p.pack(x)).cuda()
        b = torch.zeros_like(a)
        in_b = p.run(a, b, steps)
        torch.cuda.synchronize()
        out.append((p.algo, p.unpack((b if in_b else a).cpu().numpy())))
    assert out[0][0] == cs.Algo.FP64_TC, "the tensor cores are the faster here"
    largest = amp[np.maximum(np.arange(n) // tile * tile - reach, 0)]
    assert (np.abs(out[0][1] - out[1][1]) <= 2.0 ** -50 * largest + 64 * 2.0 ** -1074).all()
