"""Meshes without numbering: rows gather from far and scattered columns, for
which the on-chip engines choose other forms and limits."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import bits_equal, rel
from oracle import oracle as O
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S
from test_gpu_onchip_bicg import diagonals, system

pytestmark = pytest.mark.gpu

TOL, BAR = 1e-10, 1e-12


def pressure(n, rcm):
    return S.build(S.params(n=(n, n, n), jitter=0.2, log10k=(-1.0, 1.0), permute=True, rcm=rcm,
                            seed=3))


def best(f, reps=6):
    return min(f() for _ in range(reps))


# one block; 8 and 9 slices a block (the cluster's last size there, and the grid
# form's first); the numbered cluster's last size
@pytest.mark.parametrize("box", [(6, 6, 6), (16, 16, 16), (17, 16, 16), (24, 32, 32)])
def test_pcg_against_the_oracle(cuda, box):
    s = S.build(S.params(n=box, jitter=0.2, log10k=(-1.0, 1.0), permute=True, rcm=False, seed=7))
    ref = O.pcg(O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
    d_it, d_x = O.order_spread(O.PCG, O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
    g = system(s)
    x, info = g.solve(sv.PCG, s.b[0], tol=TOL)
    assert info.status == sv.OK and abs(info.iters - ref.iters) <= max(1, 2 * d_it)
    assert rel(x, ref.x) < max(BAR, 20 * d_x)
    g.close()


def test_pcg_iteration_is_not_a_multiple_of_the_numbered_one(cuda):
    """28^3: 1.4 times the numbered mesh's in the grid form, 4.1 in the cluster."""
    us = []
    for rcm in (True, False):
        s = pressure(28, rcm)
        g = system(s)
        us.append(best(lambda: g.solve(sv.PCG, s.b[0], tol=1e-30, maxit=200)[1].seconds))
        g.close()
    assert us[1] < 2.5 * us[0]


def flow(n, rcm, permute=True):
    return S.build(S.params(kind=S.SFR_SYS_CONVDIFF, n=(n, n, n), lengths=(np.pi,) * 3,
                            dirichlet=S.ALL_FACES, nrhs=3, rhs_normal=True, peclet=50.0, nu=1e-3,
                            dt=1e-2, permute=permute, rcm=rcm, seed=5))


# shared memory up to the 196 KB carve-out: the operator held, and part of the
# vectors for one to three systems
@pytest.mark.parametrize("n,k", [(44, 3), (52, 3), (56, 2), (64, 3), (72, 2), (84, 1)])
def test_bicgstab_beats_the_graph_kernels(cuda, n, k):
    """Device time 0.5 to 0.65 of the graph kernels', 1.0 where the vectors take
    the L1 the gathers need."""
    s = flow(n, rcm=False)
    ad = diagonals(s, k)
    g = system(s)

    def solve():
        return g.solve_multi(sv.PBICGSTAB, s.b[:k], ad_k=ad, tol=TOL)

    x, infos = solve()
    t = best(lambda: solve()[1][0].seconds)
    g.set_engine(sv.ENGINE_GRAPH)
    y, graph = solve()
    tg = best(lambda: solve()[1][0].seconds)
    for i in range(k):
        assert infos[i].status == sv.OK and abs(infos[i].iters - graph[i].iters) <= 1
        assert rel(x[i], y[i]) < BAR
    assert not bits_equal(x, y)
    assert t < 0.9 * tg
    g.close()


def banded(n, half):
    """Rows of 2 * half neighbours, diagonally dominant and not symmetric."""
    off = np.concatenate([np.arange(-half, 0), np.arange(1, half + 1)])
    col = np.arange(n)[:, None] + off
    ok = (col >= 0) & (col < n)
    ia = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    rng = np.random.default_rng(half)
    al = -rng.uniform(0.5, 1.0, ia[-1])
    ad = np.full(n, 2.0 * half)
    return ia, col[ok].astype(np.int32), al, ad, rng.standard_normal((3, n))


# (rows, neighbours either side or None: a box of that edge, systems, on chip)
@pytest.mark.parametrize("n,half,k,chip", [
    (100000, 50, 1, False), (100000, 50, 2, False), (100000, 50, 3, False),
    (250000, 20, 2, False), (200000, 20, 1, True), (200000, 20, 3, True), (80000, 50, 2, True),
    (84, None, 2, True), (88, None, 2, False), (78, None, 3, True), (88, None, 3, False)])
def test_bicgstab_limits_of_what_l2_holds(cuda, n, half, k, chip):
    """The automatic choice is on chip up to the measured line, the graph
    engine's kernels past it."""
    if half is None:
        s = flow(n, rcm=True, permute=False)
        g, b = system(s), s.b[:k]
    else:
        ia, ja, al, ad, b = banded(n, half)
        g, b = sv.GpuSystem(n, ia, ja, sv.CSRD, True), b[:k]
        g.set_values(al, ad)
    x, infos = g.solve_multi(sv.PBICGSTAB, b, tol=1e-8, maxit=8)
    g.set_engine(sv.ENGINE_GRAPH)
    y, graph = g.solve_multi(sv.PBICGSTAB, b, tol=1e-8, maxit=8)
    assert bits_equal(x, y) != chip
    assert [i.iters for i in infos] == [i.iters for i in graph]
    # a handful of iterations: the order of the sums alone
    assert rel(x, y) < BAR
    g.close()


@pytest.mark.parametrize("precision", [sv.FP64, sv.MIXED], ids=["fp64", "mixed"])
def test_batch_of_unnumbered_boxes(cuda, precision):
    """Three boxes, as accurate as alone, in well under the single solves' time:
    0.61 and 0.24 of it, as long as L1 is left for the gathers."""
    ss = [pressure(48, False)] * 3
    g = sv.GpuBatch([(s.neq, s.ia, s.ja) for s in ss], sv.CSRD, True)
    g.set_values([s.al for s in ss], [s.ad for s in ss])
    b = [s.b[0] * (i + 1) for i, s in enumerate(ss)]
    xs, infos = g.solve(sv.PCG, b, tol=TOL, precision=precision)
    t = best(lambda: g.solve(sv.PCG, b, tol=TOL, precision=precision)[1][0].seconds)
    one = system(ss[0])
    alone = best(lambda: one.solve(sv.PCG, b[0], tol=TOL, precision=precision)[1].seconds)
    for x, bi, info in zip(xs, b, infos):
        want, ref = one.solve(sv.PCG, bi, tol=TOL)
        assert info.status == sv.OK
        assert rel(x, want) < (BAR if precision == sv.FP64 else 1e-7)
    assert t < (0.8 if precision == sv.FP64 else 0.35) * 3 * alone
    g.close()
    one.close()
