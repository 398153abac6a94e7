"""FP64 3D radius-3 sweeps on tcgen05 (the tuner's pick for fused 3D plans of
ordinary size), against the FP64 CPU oracle. Bar: 1e-12 pointwise relative
error (denominator floored at 1e-3 of the largest value), the FP64 paths' bar;
normwise for signed data. The sizes are odd and even pitches (TMA or cp.async
windows), first interior columns of both parities, remainders of the 16 x 64
tile and of the column of planes."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O
from tests.util import rel_err

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOL = 1e-12


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()
    O.build()


def params_of(shape, seed, signed=False):
    cells = np.abs(np.indices((7, 7, 7)) - 3).sum(0) <= 3 if shape == "star3d1r" else np.ones((7, 7, 7), bool)
    d = np.where(cells, np.random.default_rng(seed).random((7, 7, 7)) - (0.45 if signed else 0.0), 0.0)
    d = (d + d[::-1]) / np.abs(d + d[::-1]).sum()
    if shape == "box3d1r":
        return d[:4].reshape(-1), d
    return np.concatenate([d[p][cells[p]] for p in range(4)]), d


def steps_of(a, b, d, sweeps):
    """Padded grids (halo 3), ping-pong; the final interior."""
    a, b = a.copy(), b.copy()
    n = [s - 6 for s in a.shape]
    for _ in range(sweeps):
        acc = np.zeros(n)
        for t in np.ndindex(7, 7, 7):
            if d[t] != 0.0:
                acc += d[t] * a[t[0]:t[0] + n[0], t[1]:t[1] + n[1], t[2]:t[2] + n[2]]
        b[3:-3, 3:-3, 3:-3] = acc
        a, b = b, a
    return a[3:-3, 3:-3, 3:-3]


def layout_ref(e):
    p1 = e[2] + 6
    p0 = p1 * (e[1] + 6)
    return {"dims": 3, "halo": 3, "extent": list(e), "pitch": [p0, p1, 1], "origin": 3 * p0 + 3 * p1 + 3,
            "elements": (e[0] + 6) * p0}


def run(p, a, b, steps):
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    in_b = p.run(da, db, steps)
    torch.cuda.synchronize()
    assert cs.device_wait_timeouts() == 0
    return (db if in_b else da).cpu().numpy()


@pytest.mark.parametrize("shape", ["box3d1r", "star3d1r"])
@pytest.mark.parametrize("ext", [(40, 48, 128), (37, 33, 129), (70, 17, 250), (33, 49, 63)])
@pytest.mark.parametrize("ref_layout", [True, False])
def test_fused_3d_sweeps(shape, ext, ref_layout):
    params, d = params_of(shape, 3 + ext[2])
    p = cs.Plan(shape, ext, params, semantics=cs.Semantics.FUSED, layout=layout_ref(ext) if ref_layout else None)
    x = O.splitmix_uniform(int(np.prod(ext)), 9).reshape(ext)
    buf = p.pack(x)
    got = run(p, buf, np.zeros_like(buf), 6)
    if shape == "box3d1r":
        assert p.algo == cs.Algo.FP64_TC
    ref = steps_of(np.pad(x, 3), np.zeros([s + 6 for s in ext]), d, 2)
    assert rel_err(p.unpack(got), ref)[0] <= TOL
    halo = np.ones(p.elements, bool)
    halo[p.interior_index().reshape(-1)] = False
    assert not got[halo].any(), "halo must stay zero"


@pytest.mark.parametrize("ext", [(40, 48, 128), (37, 48, 129)])
def test_signed_data_and_planes_of_different_scale(ext):
    """Planes 2^0 .. 2^-40 in turn: the parts of an output have different
    exponents; errors are relative to the window's largest value (normwise)."""
    params, d = params_of("box3d1r", 5, signed=True)
    x = O.splitmix_uniform(int(np.prod(ext)), 10).reshape(ext) - 0.5
    x *= np.ldexp(1.0, -(np.arange(ext[0]) * 13) % 41)[:, None, None]
    p = cs.Plan("box3d1r", ext, params, semantics=cs.Semantics.FUSED, layout=layout_ref(ext))
    buf = p.pack(x)
    got = p.unpack(run(p, buf, np.zeros_like(buf), 6))
    assert p.algo == cs.Algo.FP64_TC
    ref = steps_of(np.pad(x, 3), np.zeros([s + 6 for s in ext]), d, 2)
    assert np.linalg.norm(got - ref) <= 1e-14 * np.linalg.norm(ref)


@pytest.mark.parametrize("odd", [0, 1])
def test_boundary_values_and_nothing_past_the_halo(odd):
    """Boundary values in the halos of both buffers; huge values past them."""
    e, pad = (40, 40, 100 + odd), 5
    shp = [s + 2 * pad for s in e]
    p0, p1 = shp[1] * shp[2], shp[2]
    lay = {"dims": 3, "halo": 3, "extent": list(e), "pitch": [p0, p1, 1], "origin": pad * (p0 + p1 + 1),
           "elements": shp[0] * p0}
    params, d = params_of("box3d1r", 6)
    p = cs.Plan("box3d1r", e, params, semantics=cs.Semantics.FUSED, layout=lay)
    w = tuple(slice(pad - 3, pad + s + 3) for s in e)
    grids = []
    for seed in (1, 2):
        g = np.full(shp, 1e200)
        g[w] = np.random.default_rng(seed).random([s + 6 for s in e])
        grids.append(g)
    ref = steps_of(grids[0][w], grids[1][w], d, 3)
    got = run(p, grids[0].reshape(-1), grids[1].reshape(-1), 9).reshape(shp)
    assert p.algo == cs.Algo.FP64_TC
    inner = tuple(slice(pad, pad + s) for s in e)
    assert rel_err(got[inner], ref)[0] <= TOL


@pytest.mark.parametrize("ext", [(33, 40, 97), (64, 40, 96)])
def test_reference_wrappers(ext):
    for shape, call in (("box3d1r", cs.gpu_box_3d1r), ("star3d1r", cs.gpu_star_3d1r)):
        params, d = params_of(shape, 8)
        g = np.zeros([s + 6 for s in ext])
        g[3:-3, 3:-3, 3:-3] = O.splitmix_uniform(int(np.prod(ext)), 12).reshape(ext)
        ref = steps_of(g, np.zeros_like(g), d, 3)
        for _ in range(2):  # the second call overlaps its copies where it can
            out = np.zeros(g.size)
            call(g.reshape(-1).copy(), out, params, 3, *ext)
            assert rel_err(out.reshape(g.shape)[3:-3, 3:-3, 3:-3], ref)[0] <= TOL
