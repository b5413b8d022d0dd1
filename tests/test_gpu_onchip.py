"""On-chip FP64 PCG (onchip.cu): the automatic choice for one right-hand
side, in its cluster form (the system in one thread-block cluster's shared
memory) and its grid form (one block per SM, four levels of what stays in
shared memory, slots held / kept in L2 / streamed).

Bar: the suite's FP64 bar, 1e-12 relative in x at equal iteration count
(+-1), against the oracle where its serial solve is quick and against the
fused one-launch iteration (mode 4, itself held to the oracle) above.  On a
chain of cells the reference itself moves further than that when only its dot
products' order changes (31 cells of contrast 1e4: 8e-12); the small boxes
are held to that spread where it is the larger, as the suite's other
order-sensitive solves are.
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


def system(s, lname="csrd_full"):
    st, un, ia, ja, al, _ = layouts(s)[lname]
    g = sv.GpuSystem(s.neq, ia, ja, st, un)
    g.set_values(al, s.ad)
    return g


# one row, a ragged slice, one block; the cluster's edges at 8 slices a block
# (1, 2, 4, 8, 16 blocks) and past them; its last size (48 slices a block:
# 24,576 rows) and the grid form's first
BOXES = [(1, 1, 1), (3, 1, 1), (31, 1, 1), (4, 8, 1), (11, 3, 1), (16, 16, 1), (257, 1, 1),
         (8, 8, 8), (19, 27, 1), (16, 16, 16), (17, 16, 16), (23, 29, 31), (32, 32, 24),
         (32, 32, 25), (37, 31, 29)]


@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_small_boxes_against_the_oracle(cuda, box):
    s = S.build(S.params(n=box, jitter=0.2, log10k=(-2.0, 2.0), permute=True, seed=7))
    ref = O.pcg(O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
    d_it, d_x = O.order_spread(O.PCG, O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
    slack, bar = max(1, 2 * d_it), max(BAR, 20 * d_x)
    for lname in ("csrd_full", "csrc_sym", "ellpack"):
        g = system(s, lname)
        x, info = g.solve(sv.PCG, s.b[0], tol=TOL)
        assert info.status == sv.OK, (lname, info)
        assert abs(info.iters - ref.iters) <= slack, (lname, info.iters, ref.iters)
        assert rel(x, ref.x) < bar, lname
        x2, info2 = g.solve(sv.PCG, s.b[0], tol=TOL)
        assert bits_equal(x, x2) and info2.iters == info.iters
        g.close()


# slots held in shared memory; kept in L2 at levels 3 and 2; streamed at
# levels 1 and 0
@pytest.mark.parametrize("box", [(64, 64, 64), (72, 71, 73), (101, 100, 99), (112, 113, 111),
                                 (128, 128, 127)], ids=lambda b: "x".join(map(str, b)))
def test_large_boxes_against_the_fused_iteration(cuda, box):
    s = S.build(S.params(n=box, jitter=0.2, log10k=(-1.0, 1.0), seed=8))
    g = system(s)
    x, info = g.solve(sv.PCG, s.b[0], tol=TOL)
    g.set_engine(sv.ENGINE_GRAPH)
    g.set_fused(4)
    xf, fused = g.solve(sv.PCG, s.b[0], tol=TOL)
    assert info.status == sv.OK and fused.status == sv.OK
    assert abs(info.iters - fused.iters) <= 1
    assert rel(x, xf) < BAR
    for name in ("xKx", "norm_x", "conv"):
        assert abs(getattr(info, name) - getattr(fused, name)) <= 1e-11 * abs(getattr(fused, name))
    g.close()


def dense_rows(n, width, seed):
    """A symmetric positive definite CSRD system whose rows couple to
    `width` random others (rows of uneven length, long range)."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for i in range(n):
        for j in rng.choice(n, rng.integers(0, width), replace=False):
            if i != j:
                A[i, j] = A[j, i] = -rng.uniform(0.1, 1.0)
    ad = -A.sum(1) + 0.05
    ia = np.concatenate([[0], np.cumsum((A != 0).sum(1))]).astype(np.int32)
    ja = np.concatenate([np.flatnonzero(r) for r in A]).astype(np.int32)
    al = np.concatenate([r[r != 0] for r in A])
    return n, ia, ja, al, ad, rng.standard_normal(n)


@pytest.mark.parametrize("n,width", [(100, 6), (700, 40), (3000, 90)])
def test_uneven_rows(cuda, n, width):
    n, ia, ja, al, ad, b = dense_rows(n, width, seed=n)
    g = sv.GpuSystem(n, ia, ja, sv.CSRD, True)
    g.set_values(al, ad)
    x, info = g.solve(sv.PCG, b, tol=TOL)
    ref = O.pcg(O.CSRD, True, ia, ja, al, ad, b, tol=TOL)
    assert info.status == sv.OK and abs(info.iters - ref.iters) <= 1
    assert rel(x, ref.x) < BAR
    g.close()


@pytest.mark.parametrize("rcm", [True, False], ids=["offsets", "indices"])
def test_column_forms_of_the_grid_form(cuda, rcm):
    """Without RCM the bandwidth passes 32,767 and columns are 32-bit."""
    s = S.build(S.params(n=(40, 40, 40), jitter=0.2, permute=True, rcm=rcm, seed=9))
    g = system(s)
    assert (g.stats()["bandwidth"] > 32767) != rcm
    x, info = g.solve(sv.PCG, s.b[0], tol=TOL)
    ref = O.pcg(O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
    assert info.status == sv.OK and abs(info.iters - ref.iters) <= 1
    assert rel(x, ref.x) < BAR
    g.close()


@pytest.mark.parametrize("n", [14, 36], ids=["cluster", "grid"])
def test_starts_caps_and_breakdowns(cuda, n):
    torch = cuda
    s = S.poisson_jittered(n, seed=10)
    g = system(s)
    args = (O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0])
    x0 = np.cos(np.arange(s.neq))
    x, info = g.solve(sv.PCG, s.b[0], x0=x0, newx=False, tol=1e-9)
    ref = O.pcg(*args, x0=x0, newx=False, tol=1e-9)
    assert abs(info.iters - ref.iters) <= 1 and rel(x, ref.x) < BAR
    # the iteration cap: the reference's count and its x so far
    x, info = g.solve(sv.PCG, s.b[0], tol=TOL, maxit=7)
    ref = O.pcg(*args, tol=TOL, maxit=7)
    assert info.status == sv.MAXIT and info.iters == 8
    assert rel(x, ref.x) < BAR
    # a zero and a NaN right-hand side are statuses
    _, info = g.solve(sv.PCG, np.zeros(s.neq), tol=TOL, maxit=50)
    assert info.status == sv.BREAKDOWN and info.iters == 1
    bad = s.b[0].copy()
    bad[n] = np.nan
    _, info = g.solve(sv.PCG, bad, tol=TOL, maxit=50)
    assert info.status == sv.BREAKDOWN
    # x may be the array b is in
    want, _ = g.solve(sv.PCG, s.b[0], tol=TOL)
    d = torch.tensor(s.b[0], device="cuda")
    torch.cuda.synchronize()
    info = g.solve_device(sv.PCG, d.data_ptr(), d.data_ptr(), tol=TOL)
    assert info.status == sv.OK and bits_equal(d.cpu().numpy(), want)
    # a diagonal of the call's own
    xs, infos = g.solve_multi(sv.PCG, s.b[:1], ad_k=1.25 * s.ad[None], tol=TOL)
    ref = O.pcg(O.CSRD, True, s.ia, s.ja, s.al, 1.25 * s.ad, s.b[0], tol=TOL)
    assert abs(infos[0].iters - ref.iters) <= 1 and rel(xs[0], ref.x) < BAR
    g.close()


def test_one_step_convergence(cuda):
    """A diagonal system: the first update leaves no residual at all, or one
    of rounding size, and the measured product decides the stop."""
    n = 5000
    ad = np.linspace(1.0, 3.0, n)
    b = np.sin(np.arange(n)) + 2.0
    g = sv.GpuSystem(n, np.zeros(n + 1, np.int32), np.zeros(0, np.int32), sv.CSRD, True)
    g.set_values(np.zeros(0), ad)
    x, info = g.solve(sv.PCG, b, tol=1e-12)
    assert info.status == sv.OK and info.iters <= 2
    assert rel(x, b / ad) < 1e-14
    g.close()


def batch_of(boxes, **kw):
    ss = [S.build(S.params(n=b, jitter=0.2, log10k=(-1.0, 1.0), seed=20 + i, **kw))
          for i, b in enumerate(boxes)]
    g = sv.GpuBatch([(s.neq, s.ia, s.ja) for s in ss], sv.CSRD, True)
    g.set_values([s.al for s in ss], [s.ad for s in ss])
    return ss, g


# teams of one block; of one and of many; nearly as many systems as blocks;
# rows that fill a block's shared memory in part (level 2) and past it (0)
@pytest.mark.parametrize("boxes", [
    [(1, 1, 1), (5, 1, 1), (33, 1, 1), (7, 6, 5)],
    [(2, 2, 2), (40, 36, 44), (9, 9, 9), (21, 20, 19)],
    [(4, 4, 4)] * 290,
    [(58, 60, 62)] * 3,
    [(97, 100, 101)] * 2], ids=["tiny", "uneven", "many", "level2", "level0"])
def test_team_launches(cuda, boxes):
    ss, g = batch_of(boxes)
    xs, infos = g.solve(sv.PCG, [s.b[0] for s in ss], tol=TOL)
    for i, (s, x, info) in enumerate(zip(ss, xs, infos)):
        if i >= 8:
            break
        one = system(s)
        want, ref = one.solve(sv.PCG, s.b[0], tol=TOL)
        one.close()
        assert info.status == sv.OK and abs(info.iters - ref.iters) <= 1, (i, info.iters)
        assert rel(x, want) < BAR, i
    assert all(i.status == sv.OK for i in infos)
    again, _ = g.solve(sv.PCG, [s.b[0] for s in ss], tol=TOL)
    assert all(bits_equal(a, b) for a, b in zip(xs, again))
    # a warm start under a cap: each team's own status, as the persistent
    # kernel gives it for that system alone (a one-row system's start is
    # exact, and 0 / 0 a breakdown)
    x0s = [0.999 * x for x in xs]
    x0s[0] = xs[0]
    xs2, infos2 = g.solve(sv.PCG, [s.b[0] for s in ss], x0s=x0s, newx=False, tol=1e-6, maxit=4,
                          raise_on_error=False)
    for i, (s, x, info) in enumerate(list(zip(ss, xs2, infos2))[:8]):
        one = system(s)
        one.set_engine(sv.ENGINE_PERSISTENT)
        want, ref = one.solve(sv.PCG, s.b[0], x0=x0s[i], newx=False, tol=1e-6, maxit=4,
                              raise_on_error=False)
        one.close()
        assert (info.status, info.iters) == (ref.status, ref.iters), i
        assert rel(x, want) < BAR, i
    g.close()


def test_team_launch_with_wide_columns(cuda):
    """A box without RCM in the batch: 32-bit columns for every system."""
    ss, g = batch_of([(40, 40, 40), (6, 7, 8)], permute=True, rcm=False)
    xs, infos = g.solve(sv.PCG, [s.b[0] for s in ss], tol=TOL)
    for s, x, info in zip(ss, xs, infos):
        ref = O.pcg(O.CSRD, True, s.ia, s.ja, s.al, s.ad, s.b[0], tol=TOL)
        assert info.status == sv.OK and abs(info.iters - ref.iters) <= 1
        assert rel(x, ref.x) < BAR
    g.close()


@pytest.mark.parametrize("precision", [sv.FP64, sv.MIXED], ids=["fp64", "mixed"])
def test_rounds_of_a_team_launch(cuda, precision):
    """Anisotropic boxes that take far more iterations than their size
    suggests, beside cubes that take fewer: several rounds, with the blocks
    shared out anew between them.  FP64 at the FP64 bar; mixed meets the
    reference's criterion on the FP64 residual."""
    boxes = [((8, 8, 40), (8.0, 80.0, 40.0)), ((24, 24, 24), (1.0,) * 3), ((3, 3, 3), (1.0,) * 3),
             ((40, 9, 9), (40.0, 9.0, 90.0)), ((16, 20, 18), (1.0,) * 3),
             ((48, 40, 36), (48.0, 40.0, 360.0))]
    ss = [S.build(S.params(n=n, lengths=ln, seed=30 + i, dirichlet=S.FACE_XMIN))
          for i, (n, ln) in enumerate(boxes)]
    g = sv.GpuBatch([(s.neq, s.ia, s.ja) for s in ss], sv.CSRD, True)
    g.set_values([s.al for s in ss], [s.ad for s in ss])
    xs, infos = g.solve(sv.PCG, [s.b[0] for s in ss], tol=TOL, precision=precision)
    for s, x, info in zip(ss, xs, infos):
        args = (O.CSRD, True, s.ia, s.ja, s.al, s.ad)
        assert info.status == sv.OK
        if precision == sv.FP64:
            ref = O.pcg(*args, s.b[0], tol=TOL)
            d_it, d_x = O.order_spread(O.PCG, *args, s.b[0], tol=TOL)
            assert abs(info.iters - ref.iters) <= max(1, 2 * d_it)
            assert rel(x, ref.x) < max(BAR, 20 * d_x)
        else:
            r = s.b[0] - O.matvec(*args, x)
            assert np.sqrt(abs(r @ (r / s.ad))) < TOL * np.sqrt(s.b[0] @ (s.b[0] / s.ad))
            assert info.refinements >= 1
    again, infos2 = g.solve(sv.PCG, [s.b[0] for s in ss], tol=TOL, precision=precision)
    assert all(bits_equal(a, b) for a, b in zip(xs, again))
    # the cap is each system's own, also past the first round
    cap = max(i.iters for i in infos) - 5
    _, capped = g.solve(sv.PCG, [s.b[0] for s in ss], tol=TOL, maxit=cap, precision=precision,
                        raise_on_error=False)
    assert [i.status for i in capped] == [sv.OK if i.iters <= cap else sv.MAXIT for i in infos]
    g.close()
