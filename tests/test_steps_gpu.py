"""Several steps per launch of the FP64 tcgen05 digit kernel (2D radius-1
plans): three steps as one 7x7 sweep away from the boundary, the frame along it
step by step. Compared with single steps in numpy. Bar: 1e-12 of the largest
value, the FP64 paths' bar (a launch rounds at 2^-52 of its tile's largest
value, and at most 40 launches run here)."""
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


def dense_of(shape, w):
    return O.star2d1r_to_dense(w).reshape(3, 3) if shape == "star2d1r" else w.reshape(3, 3)


def steps_of(a, b, w, steps):
    """(m+2) x (n+2) grids with halos, ping-pong as cs_run: returns the interior."""
    a, b = a.copy(), b.copy()
    m, n = a.shape[0] - 2, a.shape[1] - 2
    for _ in range(steps):
        b[1:-1, 1:-1] = sum(w[i, j] * a[i:i + m, j:j + n] for i in range(3) for j in range(3))
        a, b = b, a
    return a[1:-1, 1:-1]


def run(plan, a, b, steps):
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    in_b = plan.run(da, db, steps)
    torch.cuda.synchronize()
    assert cs.device_wait_timeouts() == 0
    return (db if in_b else da).cpu().numpy()


@pytest.mark.parametrize("shape,taps", [("star2d1r", 5), ("box2d1r", 9)])
@pytest.mark.parametrize("ext", [(512, 512), (8, 4096), (4097, 9), (515, 577), (1023, 514)])
@pytest.mark.parametrize("steps", [1, 2, 3, 4, 8, 40])
def test_steps_equal_single_steps(shape, taps, ext, steps):
    w = O.seeded_weights(taps, 7 + taps) - 0.04
    p = cs.Plan(shape, ext, w)
    p.set_option(cs.Option.ALGO, cs.Algo.FP64_TC)
    x = O.splitmix_uniform(ext[0] * ext[1], 5 + ext[0]).reshape(ext) - 0.25
    buf = p.pack(x)
    got = run(p, buf, np.zeros_like(buf), steps)
    assert p.algo == cs.Algo.FP64_TC and p.time_block == 3
    ref = steps_of(np.pad(x, 1), np.zeros((ext[0] + 2, ext[1] + 2)), dense_of(shape, w), steps)
    assert np.abs(p.unpack(got) - ref).max() <= TOL * np.abs(ref).max()
    halo = np.ones(p.elements, bool)
    halo[p.interior_index().reshape(-1)] = False
    assert not got[halo].any(), "halo must stay zero"


@pytest.mark.parametrize("steps", [2, 3, 5])
def test_steps_read_each_buffers_halo_and_nothing_beyond(steps):
    """A caller's layout with boundary values in both halos (each step reads
    those of the buffer it reads) and huge values past the halo, which must
    not reach any output, not even through a tile's scale."""
    m, n, pad = 600, 520, 6
    ld = n + 2 * pad
    lay = {"dims": 2, "halo": 1, "extent": [m, n], "pitch": [ld, 1], "origin": pad * ld + pad,
           "elements": (m + 2 * pad) * ld}
    w = O.seeded_weights(9, 3)
    p = cs.Plan("box2d1r", (m, n), w, layout=lay)
    p.set_option(cs.Option.ALGO, cs.Algo.FP64_TC)
    grids = []
    for seed in (11, 12):
        g = np.full((m + 2 * pad, ld), 1e200)
        g[pad - 1:pad + m + 1, pad - 1:pad + n + 1] = O.splitmix_uniform((m + 2) * (n + 2), seed).reshape(m + 2, n + 2)
        grids.append(g)
    inner = [g[pad - 1:pad + m + 1, pad - 1:pad + n + 1] for g in grids]
    ref = steps_of(inner[0], inner[1], w.reshape(3, 3), steps)
    got = run(p, grids[0].reshape(-1), grids[1].reshape(-1), steps).reshape(m + 2 * pad, ld)
    assert p.time_block == 3
    assert np.abs(got[pad:pad + m, pad:pad + n] - ref).max() <= TOL * np.abs(ref).max()


def test_small_grids_and_odd_buffers_keep_single_steps():
    w = O.seeded_weights(9, 4)
    p = cs.Plan("box2d1r", (448, 512), w)  # 56 tiles
    p.set_option(cs.Option.ALGO, cs.Algo.FP64_TC)
    x = O.splitmix_uniform(448 * 512, 6).reshape(448, 512)
    run(p, p.pack(x), np.zeros(p.elements), 5)
    assert p.time_block == 1
    q = cs.Plan("box2d1r", (512, 512), w)
    y = O.splitmix_uniform(512 * 512, 8).reshape(512, 512)
    ref = steps_of(np.pad(y, 1), np.zeros((514, 514)), w.reshape(3, 3), 7)
    a = torch.zeros(q.elements + 1, dtype=torch.float64, device="cuda")
    b = torch.zeros_like(a)
    a[1:] = torch.from_numpy(q.pack(y)).cuda()  # 8-byte aligned grids: no TMA
    in_b = q.run(a[1:], b[1:], 7)
    torch.cuda.synchronize()
    assert q.time_block == 1
    got = q.unpack((b if in_b else a)[1:].cpu().numpy())
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


def test_weights_out_of_range_keep_single_steps():
    """Weights whose powers leave the FP64 range (here they would overflow)."""
    w = O.seeded_weights(9, 4) * 2.0 ** 70
    p = cs.Plan("box2d1r", (512, 512), w)
    p.set_option(cs.Option.ALGO, cs.Algo.FP64_TC)
    x = O.splitmix_uniform(512 * 512, 8).reshape(512, 512) * 2.0 ** -300
    got = p.unpack(run(p, p.pack(x), np.zeros(p.elements), 3))
    assert p.time_block == 1
    ref = steps_of(np.pad(x, 1), np.zeros((514, 514)), w.reshape(3, 3), 3)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


def steps_1d(a, b, w, steps):
    """1D grids with halos of the radius, ping-pong; returns the interior."""
    a, b = a.copy(), b.copy()
    r = len(w) // 2
    n = a.size - 2 * r
    for _ in range(steps):
        b[r:-r] = sum(w[t] * a[t:t + n] for t in range(2 * r + 1))
        a, b = b, a
    return a[r:-r]


@pytest.mark.parametrize("shape,taps,fused", [("1d1r", 3, 0), ("1d2r", 5, 0), ("1d1r", 7, 1)])
@pytest.mark.parametrize("n", [512, 4096, 4160, 8192, 64 * 1231])
@pytest.mark.parametrize("steps", [1, 2, 5, 8, 11, 16, 23, 50])
def test_1d_steps_equal_single_steps(shape, taps, fused, n, steps):
    w = O.seeded_weights(taps, 7 + taps) - 0.03
    p = cs.Plan(shape, (n,), w, semantics=cs.Semantics.FUSED if fused else cs.Semantics.STEP)
    p.set_option(cs.Option.ALGO, cs.Algo.FP64_TC)
    r = taps // 2
    x = O.splitmix_uniform(n, 5 + n) - 0.25
    buf = p.pack(x)
    got = run(p, buf, np.zeros_like(buf), steps * (3 if fused else 1))
    assert p.algo == cs.Algo.FP64_TC and p.time_block == {1: 23, 2: 11, 3: 7, 4: 5}[r]
    ref = steps_1d(np.pad(x, r), np.zeros(n + 2 * r), w, steps)
    assert np.abs(p.unpack(got) - ref).max() <= TOL * np.abs(ref).max()
    halo = np.ones(p.elements, bool)
    halo[p.interior_index().reshape(-1)] = False
    assert not got[halo].any(), "halo must stay zero"


@pytest.mark.parametrize("shape,taps,fused", [("1d1r", 3, 0), ("1d2r", 5, 0), ("1d1r", 7, 1), ("1d2r", 9, 1)])
@pytest.mark.parametrize("n,pad", [(300_001, 9), (300_032, 8), (262_143, 4)])
def test_1d_layouts_halos_and_nothing_beyond(shape, taps, fused, n, pad):
    """Caller layouts of odd and even origin, boundary values in both halos and
    huge values past them (AUTO: the tuner picks the tensor cores here)."""
    r = taps // 2
    w = O.seeded_weights(taps, 11)
    lay = {"dims": 1, "halo": r, "extent": [n], "pitch": [1], "origin": pad, "elements": n + 2 * pad}
    p = cs.Plan(shape, (n,), w, semantics=cs.Semantics.FUSED if fused else cs.Semantics.STEP, layout=lay)
    grids = []
    for seed in (21, 22):
        g = np.full(n + 2 * pad, 1e200)
        g[pad - r:pad + n + r] = O.splitmix_uniform(n + 2 * r, seed)
        grids.append(g)
    inner = [g[pad - r:pad + n + r] for g in grids]
    per = {"1d1r": 3, "1d2r": 2}[shape] if fused else 1
    sweeps = 43
    ref = steps_1d(inner[0], inner[1], w, sweeps)
    got = run(p, grids[0], grids[1], sweeps * per)
    assert p.algo == cs.Algo.FP64_TC and p.time_block == {1: 23, 2: 11, 3: 7, 4: 5}[r]
    assert np.abs(got[pad:pad + n] - ref).max() <= TOL * np.abs(ref).max()


def run_split(plan, buf, steps):
    raw = torch.from_numpy(buf).cuda()
    a = torch.zeros(plan.elements * 2, dtype=torch.float32, device="cuda")
    b = torch.zeros_like(a)
    plan.split_from_fp64(raw, a)
    in_b = plan.run(a, b, steps)
    plan.split_to_fp64(b if in_b else a, raw)
    torch.cuda.synchronize()
    assert cs.device_wait_timeouts() == 0
    return raw.cpu().numpy()


@pytest.mark.parametrize("shape,taps,ext", [("star2d1r", 5, (1023, 1026)), ("box2d1r", 9, (900, 1101)),
                                            ("star2d1r", 5, (4096, 4096)), ("1d1r", 3, (1_000_003,)),
                                            ("1d2r", 5, (1_048_576,))])
@pytest.mark.parametrize("steps", [3, 20, 107])
def test_split_steps(shape, taps, ext, steps):
    """Split plans under AUTO, re-anchor sweeps included, against FP64 single
    steps: 1e-12 of the largest value (at most 36 launches, each rounding to
    pairs of 48 bits, 3.6e-15), also where the tuner keeps the double-float
    kernel (2^-44 per step)."""
    w = O.seeded_weights(taps, 31)
    p = cs.Plan(shape, ext, w, precision=cs.Precision.SPLIT)
    x = O.splitmix_uniform(int(np.prod(ext)), 32).reshape(ext)
    got = p.unpack(run_split(p, p.pack(x), steps))
    if len(ext) == 2:
        ref = steps_of(np.pad(x, 1), np.zeros((ext[0] + 2, ext[1] + 2)), dense_of(shape, w), steps)
    else:
        r = taps // 2
        ref = steps_1d(np.pad(x, r), np.zeros(ext[0] + 2 * r), w, steps)
    if np.prod(ext) >= 1 << 24:
        assert p.algo == cs.Algo.SPLIT_TC and p.time_block == 3
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
