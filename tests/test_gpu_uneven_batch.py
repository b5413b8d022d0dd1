"""Batches of uneven and of large boxes: blocks of small boxes that end at once
go to the large one, and batches past the teams' shared memory leave them."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel
from oracle import oracle as O
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S
from test_gpu_onchip_bicg import system

pytestmark = pytest.mark.gpu

TOL, BAR = 1e-10, 1e-12


@pytest.mark.parametrize("precision", [sv.FP64, sv.MIXED], ids=["fp64", "mixed"])
def test_blocks_of_small_boxes_go_to_the_large_one(cuda, precision):
    boxes = [(80, 79, 81)] + [(7, 8, 6)] * 63
    ss = [S.build(S.params(n=b, jitter=0.2, log10k=(-1.0, 1.0), seed=i))
          for i, b in enumerate(boxes)]

    def batch(part):
        g = sv.GpuBatch([(s.neq, s.ia, s.ja) for s in part], sv.CSRD, True)
        g.set_values([s.al for s in part], [s.ad for s in part])
        b = [s.b[0] for s in part]
        xs, infos = g.solve(sv.PCG, b, tol=TOL, precision=precision)
        t = min(g.solve(sv.PCG, b, tol=TOL, precision=precision)[1][0].seconds for _ in range(5))
        g.close()
        return xs, infos, t

    xs, infos, t = batch(ss)
    _, _, alone = batch(ss[:1])
    for s, x, info in list(zip(ss, xs, infos))[:3]:
        one = system(s)
        want, ref = one.solve(sv.PCG, s.b[0], tol=TOL)
        one.close()
        assert info.status == sv.OK
        if precision == sv.FP64:
            assert abs(info.iters - ref.iters) <= 1
        assert rel(x, want) < (BAR if precision == sv.FP64 else 1e-7)
    assert all(np.isfinite(x).all() and i.status == sv.OK for x, i in zip(xs, infos))
    # a few rounds' launches and the small boxes' 0.3 ms more than the large
    # one alone; with 85 of 148 blocks to the end it is 1.6 times that
    assert t < 1.25 * alone


# mixed batches whose q and r fit the teams' shared memory (two 96^3 boxes), and
# past it (three of 112^3), where the persistent kernels take over
@pytest.mark.parametrize("n,count,teams", [(96, 2, True), (112, 3, False)])
def test_large_mixed_batches(cuda, n, count, teams):
    s = S.build(S.params(n=(n, n, n), jitter=0.2, log10k=(-1.0, 1.0), seed=4))
    g = sv.GpuBatch([(s.neq, s.ia, s.ja)] * count, sv.CSRD, True)
    g.set_values([s.al] * count, [s.ad] * count)
    b = [s.b[0] * (i + 1) for i in range(count)]
    xs, infos = g.solve(sv.PCG, b, tol=1e-8, precision=sv.MIXED)
    assert (g.stats()["grid"] <= cuda.cuda.get_device_properties(0).multi_processor_count) == teams
    for x, bi, info in zip(xs, b, infos):
        assert info.status == sv.OK and info.refinements >= 1
        r = bi - O.matvec(O.CSRD, True, s.ia, s.ja, s.al, s.ad, x)
        assert np.sqrt(r @ (r / s.ad)) < 1e-8 * np.sqrt(bi @ (bi / s.ad)) * (1 + 1e-6)
    g.close()
