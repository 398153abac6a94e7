"""Served FP64 requests whose kernels take several steps per launch, or came to
the tcgen05 kernels with them: the same bits whatever the chunk length and the
mix, small requests (issued whole) and large ones (a chunk a turn), step counts
that leave 0, 1 and 2 steps over, and FP64 FMA sweeps' values within 1e-12 of the
largest, the FP64 paths' bar."""
import numpy as np
import pytest

import convstencil_gb300 as cs
from oracle import cs_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

REQUESTS = [("star2d1r", (520, 600), 48, 0), ("star2d1r", (520, 600), 49, 0), ("box2d1r", (515, 577), 50, 0),
            ("star2d1r", (2048, 2048), 61, 0), ("1d1r", (300_007,), 70, 0), ("1d2r", (300_007,), 56, 0),
            ("1d2r", (300_032,), 62, 1), ("box3d1r", (40, 44, 50), 12, 1), ("star3d1r", (132, 128, 125), 9, 0),
            ("box3d1r", (60, 50, 44), 9, 0), ("box2d3r", (200, 333), 20, 0)]


def test_chunks_and_mix_leave_the_bits_alone():
    cs.build()
    reqs, refs = [], []
    for k, (shape, ext, steps, fused) in enumerate(REQUESTS):
        info = cs.SHAPE_INFO[cs.SHAPE_BY_NAME[shape]]
        w = O.seeded_weights(info[1 + fused], 50 + k)
        w /= w.sum()
        x = O.splitmix_uniform(int(np.prod(ext)), 60 + k).reshape(ext) - 0.25
        reqs.append((shape, x, w, steps, cs.Precision.FP64, cs.Semantics(fused)))
        p = cs.Plan(shape, ext, w, semantics=cs.Semantics(fused))
        p.set_option(cs.Option.ALGO, cs.Algo.FP64_FMA)
        a = torch.from_numpy(p.pack(x)).cuda()
        b = torch.zeros_like(a)
        in_b = p.run(a, b, steps)
        refs.append(p.unpack((b if in_b else a).cpu().numpy()))
    results = []
    for chunk in (6, 32, 1000):
        with cs.Server(streams=4, max_active=8, hbm_fraction=0.2, chunk_steps=chunk) as server:
            results.append([server.wait(i, timeout=120)[0] for i in server.submit_many(reqs)])
    with cs.Server(streams=1, max_active=1, hbm_fraction=0.2) as server:
        results.append([server.wait(server.submit(*r[:4], precision=r[4], semantics=r[5]), timeout=120)[0] for r in reqs])
    for k, ref in enumerate(refs):
        for got in results[1:]:
            np.testing.assert_array_equal(results[0][k], got[k])
        assert np.abs(results[0][k] - ref).max() <= 1e-12 * np.abs(ref).max(), REQUESTS[k]
    assert cs.device_wait_timeouts() == 0
