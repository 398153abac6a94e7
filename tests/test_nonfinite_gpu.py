"""An Inf or NaN in a grid whose sweeps go to the tcgen05 digit kernels in the
place of FP64 FMA or double-float ones (AUTO's odd 2D layouts, 1D arrays, fused
3D kernels and launches of several steps, and small served grids): it reaches the
outputs that read it and no other, as with those kernels. The same points are
NaN, Inf and -Inf; the others agree within 1e-12 of the largest, the paths' bar."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
P, S, A = cs.Precision, cs.Semantics, cs.Algo


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()


def odd_layout(ext, r):
    ld = ext[1] + 9
    return {"dims": 2, "halo": r, "extent": list(ext), "pitch": [ld, 1], "origin": 3 * ld + 5, "elements": (ext[0] + 6) * ld}


def solve(shape, x, w, steps, sem, prec, lay, algo):
    p = cs.Plan(shape, x.shape, w, semantics=sem, precision=prec, **({"layout": lay} if lay else {}))
    p.set_option(cs.Option.ALGO, algo)
    raw = torch.from_numpy(p.pack(x)).cuda()
    a, b = raw.clone(), torch.zeros_like(raw)
    if prec == P.SPLIT:
        p.split_from_fp64(raw, a)
    in_b = p.run(a, b, steps)
    out = b if in_b else a
    if prec == P.SPLIT:
        p.split_to_fp64(out, raw)
        out = raw
    torch.cuda.synchronize()
    return p.algo, p.unpack(out.cpu().numpy())


def same(got, ref, kinds=True):
    bad = ~np.isfinite(ref)
    assert (~np.isfinite(got) == bad).all()
    if kinds:
        assert np.array_equal(got[bad], ref[bad], equal_nan=True)
    assert np.abs(got[~bad] - ref[~bad]).max() <= 1e-12 * np.abs(ref[~bad]).max()


def grid(shape, ext, fused, at, value):
    info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
    w = O.seeded_weights(info[2] if fused else info[1], 41)
    x = O.splitmix_uniform(int(np.prod(ext)), 42).reshape(ext) - 0.25
    for p in at:
        x[p] = value
    return w / w.sum(), x


CASES = [("box2d3r", (700, 1111), S.STEP, P.FP64, True, 2), ("star2d3r", (1500, 2111), S.STEP, P.FP64, True, 1),
         ("star2d1r", (1024, 1030), S.STEP, P.FP64, False, 7), ("box2d1r", (1031, 1409), S.STEP, P.FP64, True, 8),
         ("1d1r", (100_001,), S.STEP, P.FP64, False, 25), ("1d2r", (100_001,), S.STEP, P.FP64, False, 12),
         ("box3d1r", (24, 40, 100), S.FUSED, P.FP64, False, 6), ("star3d1r", (80, 90, 100), S.FUSED, P.FP64, False, 3),
         ("star2d1r", (1024, 1030), S.STEP, P.SPLIT, False, 6), ("1d1r", (300_001,), S.STEP, P.SPLIT, False, 25)]


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("shape,ext,sem,prec,odd,steps", CASES)
def test_reaches_only_what_reads_it(shape, ext, sem, prec, odd, steps, value):
    corner = tuple(0 for _ in ext)
    end = tuple(n - 1 for n in ext)
    w, x = grid(shape, ext, sem == S.FUSED, [tuple(n // 2 for n in ext), corner, end], value)
    lay = odd_layout(ext, 3 if "3r" in shape else 1) if odd else None
    algo, got = solve(shape, x, w, steps, sem, prec, lay, A.AUTO)
    assert algo in (A.FP64_TC, A.SPLIT_TC), "the tensor cores are the faster here"
    _, ref = solve(shape, x, w, steps, sem, prec, lay, A.SPLIT_FMA if prec == P.SPLIT else A.FP64_FMA)
    same(got, ref, kinds=prec == P.FP64)
    assert cs.device_wait_timeouts() == 0


def test_more_tiles_than_are_kept():
    """An Inf in each of 11,000 tiles of 4,096 points, more per CTA than its list holds."""
    n = 45_000_001
    w = O.seeded_weights(3, 43)
    x = O.splitmix_uniform(n, 44)
    x[100::4096] = np.inf
    algo, got = solve("1d1r", x, w / w.sum(), 5, S.STEP, P.FP64, None, A.AUTO)
    assert algo == A.FP64_TC
    same(got, solve("1d1r", x, w / w.sum(), 5, S.STEP, P.FP64, None, A.FP64_FMA)[1])


@pytest.mark.parametrize("shape,ext,steps,sem", [("box2d3r", (256, 250), 3, S.STEP), ("star2d1r", (520, 600), 8, S.STEP),
                                                 ("box3d1r", (48, 50, 70), 4, S.STEP), ("1d2r", (300_007,), 13, S.STEP),
                                                 ("box3d1r", (40, 44, 70), 3, S.FUSED)])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_served(shape, ext, steps, sem, value):
    w, x = grid(shape, ext, sem == S.FUSED, [tuple(n // 2 for n in ext), tuple(0 for _ in ext)], value)
    server = cs.Server(hbm_fraction=0.05)
    got, _ = server.wait(server.submit(shape, x, w, steps, semantics=sem))
    same(got, solve(shape, x, w, steps, sem, P.FP64, None, A.FP64_FMA)[1])
