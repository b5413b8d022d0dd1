"""Mixed PCG below 100,000 rows on the resident engine (automatic choice): one
block and many, operators held on chip and read from L2, ragged last slices."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S

pytestmark = pytest.mark.gpu


def box(shape, log10k=(-2.0, 2.0)):
    return S.build(S.params(n=shape, jitter=0.2, log10k=log10k, permute=True, seed=19))


def criterion(s, b, x):
    """The reference's stopping norms: ||b - A x||_M and ||b||_M."""
    r = b - O.matvec(O.CSRD, True, s.ia, s.ja, s.al, s.ad, x)
    return np.sqrt(np.dot(r, r / s.ad)), np.sqrt(np.dot(b, b / s.ad))


# 7^3 = 343 rows stays in the persistent kernel; 8^3 = 512 is the first of the
# resident engine (one block); 33 slices need a third block; 59 x 41 x 40 =
# 96,760 rows hold their operator, and so does the smallest size past 100,000
@pytest.mark.parametrize("shape", [(7, 7, 7), (8, 8, 8), (9, 9, 13), (11, 12, 8), (31, 17, 23),
                                   (59, 41, 40), (46, 47, 47)])
@pytest.mark.parametrize("tol", [1e-6, 1e-12])
def test_mixed_pcg_meets_the_reference_criterion(cuda, shape, tol):
    s = box(shape)
    g = sv.GpuSystem(s.neq, s.ia, s.ja, sv.CSRD, True)
    g.set_values(s.al, s.ad)
    x, info = g.solve(sv.PCG, s.b[0], tol=tol, precision=sv.MIXED)
    assert info.status == sv.OK and info.refinements >= 1
    rm, bm = criterion(s, s.b[0], x)
    # the criterion is tested on b - A x in FP64; its rounding is 1e-3 of it
    assert rm < 1.001 * tol * bm
    # a second start from the solution ends at its first refresh
    x2, again = g.solve(sv.PCG, s.b[0], x0=x, newx=False, tol=2 * tol,
                        precision=sv.MIXED)
    assert again.iters == 0 and np.array_equal(x2, x)


@pytest.mark.parametrize("shape", [(8, 8, 8), (9, 9, 9), (20, 16, 18)])
def test_mixed_pcg_holds_its_residual_at_the_fp64_floor(cuda, shape):
    s = S.poisson_jittered(shape[0], seed=9) if len(set(shape)) == 1 else box(shape, (-1.0, 1.0))
    g = sv.GpuSystem(s.neq, s.ia, s.ja, sv.CSRD, True)
    g.set_values(s.al, s.ad)
    x, info = g.solve(sv.PCG, s.b[0], tol=1e-17, maxit=3000, precision=sv.MIXED,
                      raise_on_error=False)
    assert info.status == sv.MAXIT
    # between refreshes the residual moves by the refresh ratio (0.1) at most;
    # 1e-11 leaves four decades above the floor of about 1e-15
    rm, bm = criterion(s, s.b[0], x)
    assert rm < 1e-11 * bm


@pytest.mark.parametrize("what", ["no iterations", "not a number", "negative diagonal"])
def test_small_mixed_calls_end_as_in_the_persistent_kernel(cuda, what):
    s = box((9, 9, 9))
    ad, b, maxit = s.ad.copy(), s.b[0].copy(), 50
    if what == "no iterations":
        maxit = 0
    elif what == "not a number":
        b[3] = np.nan
    else:
        ad[5] = -ad[5]
    out = []
    for engine in (0, 1):
        g = sv.GpuSystem(s.neq, s.ia, s.ja, sv.CSRD, True)
        g.set_values(s.al, ad)
        g.set_engine(engine)
        out.append(g.solve(sv.PCG, b, tol=1e-12, maxit=maxit, precision=sv.MIXED,
                           raise_on_error=False))
    (x0, i0), (x1, i1) = out
    assert (i0.status, i0.iters) == (i1.status, i1.iters)
    assert np.array_equal(x0, x1)
