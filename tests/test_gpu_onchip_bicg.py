"""On-chip FP64 BiCGSTAB (onchip_bicg.cu): the automatic choice for one to
three right-hand sides, with the operator held in shared memory, the vectors
of the SpMV phases there, or part of them.

Bar: the suite's FP64 bar, 1e-12 relative in x at equal iteration count (+-1),
against the oracle on small boxes and the graph engine's kernels above; where
the reference itself moves further when only its dot products' order changes
(nearly steady flow, whose residual history is irregular), that spread.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import bits_equal, layouts, rel
from oracle import oracle as O
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S

pytestmark = pytest.mark.gpu

TOL, BAR = 1e-10, 1e-12


def flow(box, nrhs=3, dt=1e-2, seed=5):
    return S.build(S.params(kind=S.SFR_SYS_CONVDIFF, n=box, lengths=(np.pi,) * 3,
                            dirichlet=S.ALL_FACES, nrhs=nrhs, rhs_normal=True, peclet=50.0,
                            nu=1e-3, dt=dt, permute=True, seed=seed))


def system(s, lname="csrd_full"):
    st, un, ia, ja, al, _ = layouts(s)[lname]
    g = sv.GpuSystem(s.neq, ia, ja, st, un)
    g.set_values(al, s.ad)
    return g


def diagonals(s, k):
    """k diagonals of a system, as u, v and w have them."""
    return np.stack([s.ad * (1.0 + 0.05 * i) for i in range(k)])


# one row, part of a slice, one block (16 slices), two, a ragged last slice
@pytest.mark.parametrize("box", [(1, 1, 1), (3, 1, 1), (33, 1, 1), (8, 8, 8), (19, 27, 1),
                                 (17, 16, 16), (23, 29, 31)], ids=lambda b: "x".join(map(str, b)))
@pytest.mark.parametrize("k", [1, 2, 3])
def test_boxes_against_the_oracle(cuda, box, k):
    s = flow(box)
    ad = diagonals(s, k)
    refs = [O.pbicgstab(O.CSRD, True, s.ia, s.ja, s.al, ad[i], s.b[i], tol=TOL) for i in range(k)]
    for lname in ("csrd_full", "csrc_unsym", "ellpack"):
        g = system(s, lname)
        x, infos = g.solve_multi(sv.PBICGSTAB, s.b[:k], ad_k=ad, tol=TOL)
        for i, ref in enumerate(refs):
            assert infos[i].status == sv.OK and abs(infos[i].iters - ref.iters) <= 1, lname
            assert rel(x[i], ref.x) < BAR, lname
            assert infos[i].relres < 2 * TOL
        x2, _ = g.solve_multi(sv.PBICGSTAB, s.b[:k], ad_k=ad, tol=TOL)
        assert bits_equal(x, x2)
        g.close()


# nearly steady: tens of iterations, breakdowns near, tests a phase later
@pytest.mark.parametrize("n,seed", [(10, 3), (16, 4), (24, 41)])
def test_nearly_steady_flow_within_the_order_spread(cuda, n, seed):
    s = flow((n, n, n), nrhs=1, dt=1e3, seed=seed)
    ref = O.pbicgstab(O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
    d_it, d_x = O.order_spread(O.PBICGSTAB, O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
    g = system(s)
    x, info = g.solve(sv.PBICGSTAB, s.b[0], tol=TOL)
    assert info.status == sv.OK and abs(info.iters - ref.iters) <= max(1, 2 * d_it)
    assert rel(x, ref.x) < max(BAR, 20 * d_x)


# the operator held; its vectors only; six, four and three vectors on chip;
# one and three right-hand sides past the L2 line (the graph engine's kernels)
@pytest.mark.parametrize("box,k", [((61, 47, 53), 3), ((64, 64, 66), 3), ((72, 71, 70), 3),
                                   ((96, 95, 94), 1), ((80, 81, 78), 2), ((101, 100, 104), 1),
                                   ((88, 88, 80), 3)])
def test_large_boxes_against_the_graph_kernels(cuda, box, k):
    s = flow(box)
    ad = diagonals(s, k)
    g = system(s)
    x, infos = g.solve_multi(sv.PBICGSTAB, s.b[:k], ad_k=ad, tol=TOL)
    g.set_engine(sv.ENGINE_GRAPH)
    g.set_fused(0)
    xg, graph = g.solve_multi(sv.PBICGSTAB, s.b[:k], ad_k=ad, tol=TOL)
    for i in range(k):
        assert infos[i].status == sv.OK and abs(infos[i].iters - graph[i].iters) <= 1
        assert rel(x[i], xg[i]) < BAR
        for name in ("xKx", "norm_x", "conv"):
            assert abs(getattr(infos[i], name) - getattr(graph[i], name)) <= \
                1e-11 * abs(getattr(graph[i], name))
    g.close()


@pytest.mark.parametrize("n,width,far", [(700, 3, 0), (700, 20, 0), (90000, 5, 80000)])
def test_rows_of_any_width_and_reach(cuda, n, width, far):
    """Slots beyond a chunk, none at all, and columns past the 16-bit offsets."""
    rng = np.random.default_rng(n + width)
    count = rng.integers(0, width + 1, n)
    count[5] = 0
    ia = np.concatenate([[0], np.cumsum(count)]).astype(np.int32)
    ja = np.empty(ia[-1], np.int32)
    for i in range(n):
        reach = far if i < n - far and i % 1000 == 0 else 300
        lo, hi = max(0, i - 300), min(n, i + max(reach, 300) + 1)
        pool = np.setdiff1d(np.arange(lo, hi) if reach == 300 else rng.integers(lo, hi, 64), [i])
        ja[ia[i]:ia[i + 1]] = np.sort(rng.choice(pool, count[i], replace=False))
    al = rng.uniform(-1.0, 1.0, ia[-1])
    ad = rng.uniform(1.5, 2.0, n) * (width + 1)
    b = rng.standard_normal(n)
    ref = O.pbicgstab(O.CSRD, True, ia, ja, al, ad, b, tol=TOL)
    g = sv.GpuSystem(n, ia, ja, sv.CSRD, True)
    g.set_values(al, ad)
    x, info = g.solve(sv.PBICGSTAB, b, tol=TOL)
    assert info.status == sv.OK and abs(info.iters - ref.iters) <= 1
    assert rel(x, ref.x) < BAR


@pytest.mark.parametrize("maxit", [0, 1, 2, 3])
def test_capped_and_warm_solves_follow_the_persistent_kernel(cuda, maxit):
    s = flow((13, 12, 11))
    ad, x0 = diagonals(s, 3), np.random.default_rng(1).standard_normal((3, s.neq))
    out = []
    for engine in (0, 1):
        g = system(s)
        g.set_engine(engine)
        out.append(g.solve_multi(sv.PBICGSTAB, s.b, ad_k=ad, x0=x0, newx=False, tol=TOL,
                                 maxit=maxit, raise_on_error=False))
    (x, infos), (xp, pers) = out
    for k in range(3):
        assert (infos[k].status, infos[k].iters) == (pers[k].status, pers[k].iters)
        assert rel(x[k], xp[k]) < BAR


@pytest.mark.parametrize("what", ["zero", "not a number", "one zero"])
def test_breakdowns_are_those_of_the_persistent_kernel(cuda, what):
    s = flow((9, 9, 9))
    b = s.b.copy()
    if what == "zero":
        b[:] = 0.0
    elif what == "not a number":
        b[1, 3] = np.nan
    else:
        b[2] = 0.0
    out = []
    for engine in (0, 1):
        g = system(s)
        g.set_engine(engine)
        out.append(g.solve_multi(sv.PBICGSTAB, b, tol=TOL, raise_on_error=False))
    (x, infos), (xp, pers) = out
    for k in range(3):
        assert (infos[k].status, infos[k].iters) == (pers[k].status, pers[k].iters)
        assert np.allclose(x[k], xp[k], rtol=0, atol=BAR * np.linalg.norm(xp[k]))


def test_x_may_lie_over_the_right_hand_sides_and_the_diagonals(cuda):
    import torch
    s = flow((21, 20, 19))
    ad = diagonals(s, 3)
    g = system(s)
    want, _ = g.solve_multi(sv.PBICGSTAB, s.b, ad_k=ad, tol=TOL)
    n = s.neq
    for shift in (0, n // 2):
        for over in ("b", "ad"):
            buf = torch.zeros(3 * n + shift, dtype=torch.float64, device="cuda")
            tb, tad = torch.from_numpy(s.b.copy()).cuda(), torch.from_numpy(ad.copy()).cuda()
            buf[shift:] = (tb if over == "b" else tad).reshape(-1)
            src = buf.data_ptr() + 8 * shift
            torch.cuda.synchronize()
            g.solve_multi_device(sv.PBICGSTAB, 3, src if over == "b" else tb.data_ptr(),
                                 buf.data_ptr(), d_ad_k=src if over == "ad" else tad.data_ptr(),
                                 tol=TOL)
            torch.cuda.synchronize()
            assert bits_equal(buf[:3 * n].cpu().numpy().reshape(3, n), want)
