"""Error of the FP64 tcgen05 kernels that AUTO takes where FP64 FMA sweeps ran
before them, against sums in two doubles: on uniform and on smooth data no larger
in the norm than that of FP64 FMA sweeps (the bar is that error itself, measured
on the same data)."""
import itertools

import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    cs.build()


def halves(a):
    """Veltkamp's split: two doubles of 26 bits whose products are exact."""
    c = a * 134217729.0
    h = c - (c - a)
    return h, a - h


def two_doubles(x, dense, sweeps):
    """`sweeps` sweeps of x, zero outside it, every value as a sum of two doubles."""
    r = dense.shape[0] // 2
    inner = tuple(slice(r, r + n) for n in x.shape)
    hi = torch.zeros([n + 2 * r for n in x.shape], dtype=torch.float64, device="cuda")
    lo = torch.zeros_like(hi)
    hi[inner] = x
    taps = [(t, float(dense[t])) for t in itertools.product(*map(range, dense.shape)) if dense[t] != 0]
    for _ in range(sweeps):
        h, l = torch.zeros_like(x), torch.zeros_like(x)
        ah, al = halves(hi)
        for t, w in taps:
            at = tuple(slice(k, k + n) for k, n in zip(t, x.shape))
            wh, wl = halves(w)
            p = hi[at] * w
            e = ((ah[at] * wh - p) + ah[at] * wl + al[at] * wh) + al[at] * wl + lo[at] * w
            s = h + p
            b = s - h
            l += (h - (s - b)) + (p - b) + e
            h = s
        hi[inner] = h + l
        lo[inner] = l - (hi[inner] - h)
    return hi[inner], lo[inner]


def field(ext, kind):
    if kind == "uniform":
        return torch.rand(ext, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    axes = torch.meshgrid(*[torch.arange(n, dtype=torch.float64, device="cuda") for n in ext], indexing="ij")
    return 1.3 + sum(torch.sin(a / (17.0 + 5 * i)) for i, a in enumerate(axes)) / len(ext)


def errors(shape, ext, w, dense, sweeps, steps, kind, make):
    x = field(ext, kind)
    hi, lo = two_doubles(x, dense, sweeps)
    out = []
    for algo in (cs.Algo.AUTO, cs.Algo.FP64_FMA):
        p = make()
        p.set_option(cs.Option.ALGO, algo)
        L = p.layout
        inner = lambda g: torch.as_strided(g, list(ext), [int(v) for v in L.pitch[:L.dims]], int(L.origin))
        a = torch.zeros(p.elements, dtype=torch.float64, device="cuda")
        b = torch.zeros_like(a)
        inner(a).copy_(x)
        in_b = p.run(a, b, steps)
        out.append((p.algo, float(((inner(b if in_b else a) - hi) - lo).norm())))
    assert out[0][0] == cs.Algo.FP64_TC, "the tensor cores are the faster here"
    return out[0][1], out[1][1]


@pytest.mark.parametrize("kind", ["uniform", "smooth"])
@pytest.mark.parametrize("shape", ["box3d1r", "star3d1r"])
def test_fused_3d(shape, kind):
    ext = (64, 60, 66)
    w = O.seeded_weights(196 if shape == "box3d1r" else 44, 31)
    expand = O.box3d_planes_to_dense if shape == "box3d1r" else O.star3d_params_to_dense
    dense = expand(w).reshape(7, 7, 7)
    w, dense = w / dense.sum(), dense / dense.sum()
    tc, fma = errors(shape, ext, w, dense, 10, 30, kind, lambda: cs.Plan(shape, ext, w, semantics=cs.Semantics.FUSED))
    assert tc <= fma
