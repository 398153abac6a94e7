"""Layouts whose halo does not lie in whole rows and planes of the buffer: one that
ends with the last tap, and one whose left halo columns are the end of the row
before. Boundary values there are read like any others, by whichever kernel a
plan or a pin takes (tensor maps are made of whole rows and read zeros past
them). Bar: 1e-12 of the largest value, the FP64 and split paths' bar."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()


def layout(ext, r, kind, even):
    """Pitches even or odd; origin and elements by kind."""
    d = len(ext)
    pitch = [1] * d
    pitch[d - 2] = ext[-1] + 2 * r + 2 + (ext[-1] + even + 1) % 2
    if d == 3:
        pitch[0] = pitch[1] * (ext[1] + 2 * r)
    left = 0 if kind == "columns" else r + (r + even + 1) % 2
    # one row (plane) more before the grid where its columns run into it
    origin = left + sum((r + (kind == "columns" and k == 0)) * pitch[k] for k in range(d - 1))
    last = origin + sum((ext[k] - 1 + r) * pitch[k] for k in range(d))
    whole = -(-(last + 1) // pitch[0]) * pitch[0]
    return {"dims": d, "halo": r, "extent": list(ext), "pitch": pitch, "origin": origin,
            "elements": last + 1 if kind == "end" else whole}


def solve(shape, ext, w, sem, prec, lay, algo, raw, steps):
    p = cs.Plan(shape, ext, w, semantics=sem, precision=prec, layout=lay)
    p.set_option(cs.Option.ALGO, algo)
    a, b = raw.clone(), raw * 0.5
    if prec == cs.Precision.SPLIT:
        p.split_from_fp64(a.clone(), a)
        p.split_from_fp64(b.clone(), b)
    in_b = p.run(a, b, steps)
    out = b if in_b else a
    if prec == cs.Precision.SPLIT:
        p.split_to_fp64(out, a if in_b else b)
        out = a if in_b else b
    torch.cuda.synchronize()
    return p.unpack(out.cpu().numpy())


A, P, S = cs.Algo, cs.Precision, cs.Semantics
CASES = [("box3d1r", (40, 48, 64), S.FUSED, P.FP64, A.AUTO), ("star3d1r", (40, 48, 64), S.FUSED, P.FP64, A.AUTO),
         ("box3d1r", (64, 64, 64), S.STEP, P.FP64, A.FP64_TC), ("box3d1r", (64, 64, 64), S.STEP, P.SPLIT, A.SPLIT_TC),
         ("star2d1r", (600, 570), S.STEP, P.FP64, A.AUTO), ("box2d3r", (600, 570), S.STEP, P.FP64, A.AUTO),
         ("box2d3r", (256, 250), S.STEP, P.SPLIT, A.AUTO), ("star2d1r", (600, 570), S.STEP, P.SPLIT, A.AUTO)]


@pytest.mark.parametrize("kind", ["end", "columns"])
@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("shape,ext,sem,prec,algo", CASES)
def test_halo_outside_whole_rows(shape, ext, sem, prec, algo, even, kind):
    info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
    d, r = len(ext), 3 if sem == S.FUSED or "3r" in shape else 1
    lay = layout(ext, r, kind, even)
    w = O.seeded_weights(info[2] if sem == S.FUSED else info[1], 17)
    w /= w.sum()
    raw = torch.from_numpy(O.splitmix_uniform(lay["elements"], 19)).cuda()
    steps = info[3] if sem == S.FUSED else 3
    ref = solve(shape, ext, w, sem, prec, lay, A.SPLIT_FMA if prec == P.SPLIT else A.FP64_FMA, raw, steps)
    for _ in range(2):
        got = solve(shape, ext, w, sem, prec, lay, algo, raw, steps)
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    assert cs.device_wait_timeouts() == 0
