"""BiCGSTAB on the graph engine's kernels (and its host loop, engine 3), whose
phase C adds the x that earlier phases left due: stops after the half step,
breakdowns after it and after the full step, caps, and right-hand sides that
end in different iterations of one call, against the oracle and the persistent
kernel.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel
from oracle import oracle as O
from sfr3d_b200 import solver as sv
from test_gpu_onchip_bicg import diagonals, flow, system

pytestmark = pytest.mark.gpu

BAR = 1e-12


def two_parts(n):
    """Rows without neighbours (their part of a right-hand side is solved by the
    first half step, exactly) beside a flow's rows."""
    f = flow((n, n, n - 1), nrhs=3, dt=1.0)
    m = 70
    ia = np.concatenate([np.zeros(m, np.int32), f.ia]).astype(np.int32)
    ja = (f.ja + m).astype(np.int32)
    ad = np.concatenate([np.full(m, 2.0), f.ad])
    b = np.zeros((3, m + f.neq))
    b[0, m:] = f.b[0]
    b[1, :m] = 2.0 ** np.arange(-3, 4).repeat(10)
    b[2, m:] = f.b[1]
    b[2, :m] = 1.0
    return m + f.neq, ia, ja, f.al, ad, b


def solve(g, b, engine, **kw):
    g.set_engine(engine)
    return g.solve_multi(sv.PBICGSTAB, b, raise_on_error=False, **kw)


@pytest.mark.parametrize("tol,maxit", [(1e-10, 100), (1e-10, 3), (1e-10, 1), (0.0, 4)],
                         ids=["converge", "cap", "one", "breakdown"])
@pytest.mark.parametrize("engine", [2, 3], ids=["graph", "loop"])
def test_right_hand_sides_that_end_apart(cuda, engine, tol, maxit):
    """Right-hand side 1 leaves no residual after its first half step: it stops
    there, or with tol = 0 breaks down there (0 / 0), with the half step in x;
    the others go on, in the same call, to their end or the cap."""
    n, ia, ja, al, ad, b = two_parts(12)
    g = sv.GpuSystem(n, ia, ja, sv.CSRD, True)
    g.set_values(al, ad)
    if tol:
        refs = [O.pbicgstab(O.CSRD, True, ia, ja, al, ad, b[i], tol=tol, maxit=maxit)
                for i in range(3)]
        xs = [r.x for r in refs]
    else:  # the reference does not look for 0 / 0
        xs, refs = solve(g, b, 1, tol=tol, maxit=maxit)
    assert refs[1].iters == 1 and refs[1].status == (sv.OK if tol else sv.BREAKDOWN)
    assert rel(xs[1][:70], b[1, :70] / 2.0) < 1e-15
    if maxit == 100:
        assert refs[0].iters > 3 and refs[2].iters > 3
    for k, order in ((3, [0, 1, 2]), (3, [1, 2, 0]), (2, [1, 0]), (1, [1]), (1, [0])):
        x, infos = solve(g, b[order], engine, tol=tol, maxit=maxit)
        for xi, info, r in zip(x, infos, order):
            ref = refs[r]
            assert info.status == ref.status
            assert abs(info.iters - ref.iters) <= (1 if info.status == sv.OK else 0)
            assert rel(xi, xs[r]) < BAR
    g.close()


@pytest.mark.parametrize("engine,precision", [
    (1, sv.FP64), (2, sv.FP64), (3, sv.FP64), (2, sv.MIXED), (3, sv.MIXED)],
    ids=["persistent", "graph", "loop", "graph-mixed", "loop-mixed"])
def test_breakdown_after_the_full_step(cuda, engine, precision):
    """Blocks [[1, 1], [-3, 1]] and b = (-1, 1) repeated, in whole numbers:
    alpha = 1/2, s = (-1, -1), t = (-2, 2), so omega = 0 and beta is 0 / 0.  x
    holds the half step."""
    m = 1000
    ia = np.arange(2 * m + 1, dtype=np.int32)
    ja = (np.arange(2 * m) ^ 1).astype(np.int32)
    al = np.tile([1.0, -3.0], m)
    ad = np.ones(2 * m)
    b = np.tile([-1.0, 1.0], m)
    g = sv.GpuSystem(2 * m, ia, ja, sv.CSRD, True)
    g.set_values(al, ad)
    x, infos = solve(g, np.stack([b, 2.0 * b]), engine, tol=1e-10, maxit=50, precision=precision)
    assert all(i.status == sv.BREAKDOWN and i.iters == 1 for i in infos)
    assert np.array_equal(x[0], 0.5 * b) and np.array_equal(x[1], b)
    g.close()


@pytest.mark.parametrize("box", [(1, 1, 1), (33, 1, 1), (17, 16, 16), (23, 29, 31)],
                         ids=lambda b: "x".join(map(str, b)))
@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_boxes_against_the_oracle(cuda, box, k):
    s = flow(box, nrhs=k)
    ad = diagonals(s, k)
    g = system(s)
    x, infos = solve(g, s.b, 2, ad_k=ad, tol=1e-10)
    for i in range(k):
        ref = O.pbicgstab(O.CSRD, True, s.ia, s.ja, s.al, ad[i], s.b[i], tol=1e-10)
        assert infos[i].status == sv.OK and abs(infos[i].iters - ref.iters) <= 1
        assert rel(x[i], ref.x) < BAR
    g.close()


@pytest.mark.parametrize("maxit", [1, 2, 5])
def test_mixed_caps_hold_every_step_taken(cuda, maxit):
    """Mixed, capped: the residual of x is that of the FP64 solve capped at the
    same iteration, to what FP32 vectors leave of it."""
    s = flow((14, 13, 12), dt=1.0)
    g = system(s)
    out = {p: solve(g, s.b, 2, tol=1e-10, maxit=maxit, precision=p)[0]
           for p in (sv.FP64, sv.MIXED)}
    for i in range(3):
        r = {p: np.linalg.norm(s.b[i] - O.matvec(O.CSRD, True, s.ia, s.ja, s.al, s.ad, x[i]))
             for p, x in out.items()}
        assert r[sv.MIXED] < 1.01 * r[sv.FP64] + 1e-5 * np.linalg.norm(s.b[i])
    g.close()
