"""The longest 1D array a plan takes, 2^31 - 1 points (n + radius does not fit 32
bits): several steps per tcgen05 launch against FP64 FMA sweeps. Bar: 1e-12 of
the largest value, the FP64 paths' bar (at most four launches run here)."""
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape,taps", [("1d1r", 3), ("1d2r", 5)])
def test_longest_array(shape, taps):
    cs.build()
    n, steps = (1 << 31) - 1, 24
    if torch.cuda.mem_get_info()[0] < 90 << 30:
        pytest.skip("needs 90 GB on the device")
    w = O.seeded_weights(taps, 21)
    got = []
    for algo in (cs.Algo.AUTO, cs.Algo.FP64_FMA):
        p = cs.Plan(shape, (n,), w)
        p.set_option(cs.Option.ALGO, algo)
        a = torch.rand(p.elements, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(8))
        b = torch.zeros_like(a)
        in_b = p.run(a, b, steps)
        torch.cuda.synchronize()
        got.append((p.algo, (b if in_b else a)[p.layout.origin:p.layout.origin + n]))
        del a, b
    assert got[0][0] == cs.Algo.FP64_TC, "the tensor cores are the faster here"
    x, y = got[0][1], got[1][1]
    worst = max(float((x[i:i + (1 << 28)] - y[i:i + (1 << 28)]).abs().max()) for i in range(0, n, 1 << 28))
    assert worst <= 1e-12
    assert float(y[-64:].abs().max()) > 0.01
    assert cs.device_wait_timeouts() == 0
