"""What a program does with this library, as cases that can be timed.

Three kinds of call:

* ``device``: a plan over device buffers. One pass is one solve: the initial
  grid is copied into the plan's buffer (split precision: converted to
  (hi, lo) pairs), advanced by ``steps`` time steps, and the final grid is the
  output (split precision: converted back to FP64).
* ``host``: one call of a reference-named wrapper on pinned host buffers, the
  reference's padded layouts, copies included.
* ``served``: a list of solves handed to a running server at once, then every
  result waited for.

The stencil's weights belong to the program, so they depend on the case only;
the grids (uniform in [0, 1)) come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import convstencil_gb300 as cs

# shape -> (dims, base radius, fused radius, steps per fused sweep)
SHAPES = {
    "1d1r": (1, 1, 3, 3), "1d2r": (1, 2, 4, 2),
    "star2d1r": (2, 1, 3, 3), "box2d1r": (2, 1, 3, 3),
    "star2d3r": (2, 3, 3, 1), "box2d3r": (2, 3, 3, 1),
    "star3d1r": (3, 1, 3, 3), "box3d1r": (3, 1, 3, 3),
}
WRAPPERS = {
    "1d1r": cs.gpu_1d1r, "1d2r": cs.gpu_star_1d2r_step2,
    "box2d1r": cs.gpu_box_2d1r, "box2d3r": cs.gpu_box_2d3r,
    "star3d1r": cs.gpu_star_3d1r, "box3d1r": cs.gpu_box_3d1r,
}
# The largest work of one pass: point updates, operations, bytes in and out.
MOST_UPDATES, MOST_FLOPS, MOST_BYTES = 2.7e9, 1.46e11, 2.15e9


def _device(name, shape, extent, steps, precision="fp64", fused=False):
    e = tuple(extent) + (1,) * (3 - len(extent))
    return {"name": name, "kind": "device", "shape": shape, "e0": e[0], "e1": e[1], "e2": e[2],
            "steps": steps, "precision": precision, "fused": fused}


def _host(name, shape, extent, sweeps):
    e = tuple(extent) + (1,) * (3 - len(extent))
    return {"name": name, "kind": "host", "shape": shape, "e0": e[0], "e1": e[1], "e2": e[2],
            "steps": sweeps * SHAPES[shape][3], "precision": "fp64", "fused": True}


def listed():
    return [
        # The smallest call: a short solve of a small ragged grid, latency and launches.
        _device("box2d3r_130x96", "box2d3r", (96, 130), 10),
        # A cache-resident 5-point heat step loop (the benchmark's first configuration).
        _device("star2d1r_1024", "star2d1r", (1024, 1024), 100),
        # An ordinary 9-point solve on a grid of odd sizes.
        _device("box2d1r_2047x1531", "box2d1r", (2047, 1531), 60),
        # The 5-point step loop in split precision.
        _device("star2d1r_4096_split", "star2d1r", (4096, 4096), 50, precision="split"),
        # The headline 49-point sweep in both precisions.
        _device("box2d3r_8192", "box2d3r", (8192, 8192), 20),
        _device("box2d3r_8192_split", "box2d3r", (8192, 8192), 20, precision="split"),
        # The benchmark's long 1D array.
        _device("1d2r_10240000", "1d2r", (10240000,), 100),
        # 3D solves at the benchmark's size: 7 points FP64, 27 points split.
        _device("star3d1r_512", "star3d1r", (512, 512, 512), 20),
        _device("box3d1r_512_split", "box3d1r", (512, 512, 512), 20, precision="split"),
        # The reference's entry points, host buffers in and out: the 3D box
        # (three steps per 7x7x7 sweep) and the 2D 3x3 box.
        _host("gpu_box_3d1r_200", "box3d1r", (200, 184, 192), 10),
        _host("gpu_box_2d1r_4096", "box2d1r", (4096, 4096), 20),
        # A server's burst of mixed requests.
        {"name": "served_24", "kind": "served", "requests": 24, "mix": 1, "most_2d": 2048, "most_3d": 160,
         "most_steps": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more solve: any shape, precision and kind of call, sizes over their
    whole range (odd ones among them), never more work than the largest above."""
    kind = rng.choices(("device", "host", "served"), (7, 3, 1))[0]
    if kind == "served":
        return {"kind": kind, "requests": rng.randint(4, 32), "mix": rng.randint(2, 1 << 30),
                "most_2d": _log_int(rng, 256, 2048), "most_3d": _log_int(rng, 64, 160),
                "most_steps": rng.randint(20, 100)}
    while True:
        shape = rng.choice(sorted(WRAPPERS if kind == "host" else SHAPES))
        dims, base_r, fused_r, fuse = SHAPES[shape]
        lo, hi = {1: (2000, 16777216), 2: (64, 8192), 3: (32, 512)}[dims]
        ext = [_log_int(rng, lo, hi) for _ in range(dims)] + [1] * (3 - dims)
        fused = kind == "host" or rng.random() < 0.15
        steps = _log_int(rng, 4, 120)
        if fused:
            steps = max(1, steps // fuse) * fuse
        c = {"kind": kind, "shape": shape, "e0": ext[0], "e1": ext[1], "e2": ext[2], "steps": steps,
             "precision": "split" if kind == "device" and rng.random() < 0.4 else "fp64", "fused": fused}
        w = work(c)
        if math.prod(ext) * _sweeps(c) <= MOST_UPDATES and w["flops"] <= MOST_FLOPS and w["bytes"] <= MOST_BYTES:
            return c


# ------------------------------------------------------------------ the case
def _extent(c):
    return [c["e0"], c["e1"], c["e2"]][: SHAPES[c["shape"]][0]]


def _sweeps(c):
    return c["steps"] // (SHAPES[c["shape"]][3] if c["fused"] else 1)


def _cells(shape, fused):
    """Boolean cell array of the kernel's taps and its radius."""
    dims, base_r, fused_r, _ = SHAPES[shape]
    r = fused_r if fused else base_r
    idx = np.abs(np.indices((2 * r + 1,) * dims) - r)
    if shape.startswith("star"):
        if not fused or shape == "star2d3r":
            return (idx > 0).sum(0) <= 1, r  # the axis cross
        return idx.sum(0) <= r, r           # a cross applied r times
    return np.ones((2 * r + 1,) * dims, bool), r


def _weights(c):
    """(the parameters the call takes, the dense kernel they stand for)."""
    cells, r = _cells(c["shape"], c["fused"])
    dims = cells.ndim
    g = np.random.Generator(np.random.PCG64(sum(map(ord, c["shape"])) + 7 * bool(c["fused"])))
    dense = np.where(cells, 0.05 + g.random(cells.shape), 0.0)
    if dims == 3 and c["fused"]:  # plane p of the parameters serves dz = +-(3 - p)
        dense = dense + dense[::-1]
        dense /= dense.sum()
        if c["shape"] == "box3d1r":
            return dense[:4].reshape(-1), dense
        # the octahedron's cells, plane by plane from |dz| = 3 to 0
        return np.concatenate([dense[p][cells[p]] for p in range(4)]), dense
    dense /= dense.sum()
    if dims == 2 and c["fused"]:
        return dense.reshape(-1), dense
    return dense[cells], dense


def _grid(extent, seed, salt=0):
    g = torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return torch.rand(tuple(extent), generator=g, dtype=torch.float64, device="cuda")


def _host_layout(c):
    """The reference's padded host arrays: (array shape, interior slices, elements in, first element out)."""
    e = _extent(c)
    if c["shape"] == "1d1r":
        return (e[0] + 7,), (slice(4, 4 + e[0]),), 1
    if c["shape"] == "1d2r":
        return (e[0] + 8,), (slice(4, 4 + e[0]),), 0
    if len(e) == 2:
        return (e[0] + 6, e[1] + 8), (slice(3, 3 + e[0]), slice(4, 4 + e[1])), 0
    return tuple(x + 6 for x in e), tuple(slice(3, 3 + x) for x in e), 0


def _requests(c):
    """The served solves: device-style cases drawn from the mix number."""
    import random
    rng, got = random.Random(c["mix"]), []
    for _ in range(c["requests"]):
        shape = rng.choice(("star2d1r", "box2d3r", "star3d1r", "box3d1r"))
        if SHAPES[shape][0] == 2:
            ext = (_log_int(rng, 64, c["most_2d"]), _log_int(rng, 64, c["most_2d"]))
        else:
            ext = tuple(_log_int(rng, 32, c["most_3d"]) for _ in range(3))
        got.append(_device("", shape, ext, rng.randint(10, c["most_steps"]),
                           precision=rng.choice(("fp64", "split"))))
    return got


def _precision(c):
    return cs.Precision.SPLIT if c["precision"] == "split" else cs.Precision.FP64


class _Served:
    """A running server and one burst of requests for it."""

    def __init__(self, c, seed):
        self.server = cs.Server(hbm_fraction=0.2)
        self.requests = [(r["shape"], _grid(_extent(r), seed, k).cpu().numpy(), _weights(r)[0], r["steps"],
                          _precision(r)) for k, r in enumerate(_requests(c))]


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "served":
        return {"c": c, "served": _Served(c, seed)}
    params, _ = _weights(c)
    x = _grid(_extent(c), seed)
    if c["kind"] == "host":
        shape, inner, first = _host_layout(c)
        a = torch.zeros(shape, dtype=torch.float64, device="cuda")
        a[inner] = x
        inp = torch.empty(a.numel(), dtype=torch.float64, pin_memory=True)
        inp.copy_(a.reshape(-1))
        out = torch.zeros(a.numel() - (len(shape) == 1), dtype=torch.float64, pin_memory=True)
        torch.cuda.synchronize()
        return {"c": c, "call": WRAPPERS[c["shape"]], "in": inp.numpy(), "out": out.numpy(), "params": params,
                "keep": (inp, out)}
    plan = cs.Plan(c["shape"], _extent(c), params,
                   semantics=cs.Semantics.FUSED if c["fused"] else cs.Semantics.STEP, precision=_precision(c))
    first = torch.zeros(plan.elements, dtype=torch.float64, device="cuda")
    _interior(plan, first).copy_(x)
    return {"c": c, "plan": plan, "first": first, "a": torch.zeros_like(first), "b": torch.zeros_like(first),
            "final": torch.zeros_like(first) if c["precision"] == "split" else None}


def _interior(plan, flat):
    L, d = plan.layout, plan.layout.dims
    return torch.as_strided(flat, [int(v) for v in L.extent[:d]], [int(v) for v in L.pitch[:d]], int(L.origin))


def run(state):
    c = state["c"]
    if c["kind"] == "served":
        srv = state["served"]
        return [srv.server.wait(i)[0] for i in srv.server.submit_many(srv.requests)]
    if c["kind"] == "host":
        sweeps = c["steps"] // SHAPES[c["shape"]][3]
        state["call"](state["in"], state["out"], state["params"], sweeps, *_extent(c))
        return state["out"]
    plan, a, b = state["plan"], state["a"], state["b"]
    stream = torch.cuda.current_stream()
    if c["precision"] == "split":
        plan.split_from_fp64(state["first"], a, stream)
        in_b = plan.run(a, b, c["steps"], stream)
        plan.split_to_fp64(b if in_b else a, state["final"], stream)
        return _interior(plan, state["final"])
    a.copy_(state["first"])
    in_b = plan.run(a, b, c["steps"], stream)
    return _interior(plan, b if in_b else a)


def work(case):
    """Grids read and written once; one multiply-add per tap and point update."""
    if case["kind"] == "served":
        parts = [work(r) for r in _requests(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    pts = math.prod(_extent(case))
    taps = int(_cells(case["shape"], case["fused"])[0].sum())
    return {"bytes": 16.0 * pts, "flops": 2.0 * taps * pts * _sweeps(case)}


def _solve(c, x):
    """The sweeps of `c` on the interior grid x, zero outside it, in 64 bits."""
    _, dense = _weights(c)
    r, dims = dense.shape[0] // 2, dense.ndim
    inner = tuple(slice(r, r + n) for n in x.shape)
    u = torch.zeros([n + 2 * r for n in x.shape], dtype=torch.float64, device=x.device)
    u[inner] = x
    v = torch.zeros_like(u)
    taps = [(t, float(dense[t])) for t in np.ndindex(*dense.shape) if dense[t] != 0.0]
    for _ in range(_sweeps(c)):
        acc = v[inner].zero_()
        for t, w in taps:
            acc.add_(u[tuple(slice(t[d], t[d] + x.shape[d]) for d in range(dims))], alpha=w)
        u, v = v, u
    return u[inner]


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "served":
        return [_solve(r, _grid(_extent(r), seed, k)).cpu().numpy() for k, r in enumerate(_requests(c))]
    y = _solve(c, _grid(_extent(c), seed))
    if c["kind"] == "host":
        shape, inner, first = _host_layout(c)
        a = torch.zeros(shape, dtype=torch.float64, device=y.device)
        a[inner] = y
        flat = a.reshape(-1)
        return (flat[first:] if first else flat[: flat.numel() - (len(shape) == 1)]).cpu().numpy()
    return y
