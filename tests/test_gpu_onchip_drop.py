"""On-chip FP64 PCG (onchip.cu) where one step takes the residual down by nine
orders and the solve must go on: beta is formed from the predicted norm of the
next residual, which then has few correct digits or none."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel
from oracle import oracle as O
from sfr3d_b200 import solver as sv

pytestmark = pytest.mark.gpu


def laplacian(n):
    """7-point Laplacian of n^3 nodes and its smoothest eigenvector."""
    i = np.arange(n ** 3).reshape(n, n, n)
    col = np.full((n, n, n, 6), -1)
    for k, ax in enumerate((2, 1, 0)):
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[ax], hi[ax] = slice(0, n - 1), slice(1, n)
        col[tuple(hi) + (2 - k,)] = i[tuple(lo)]
        col[tuple(lo) + (3 + k,)] = i[tuple(hi)]
    col = col.reshape(-1, 6)
    ok = col >= 0
    ia = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    v = np.sin(np.pi * np.arange(1, n + 1) / (n + 1))
    v = np.einsum("i,j,k->ijk", v, v, v).ravel()
    return ia, col[ok].astype(np.int32), np.full(ia[-1], -1.0), np.full(n ** 3, 6.0), v


# the cluster; the grid form with the operator held, and at level 2
@pytest.mark.parametrize("n", [12, 24, 36, 92])
@pytest.mark.parametrize("rest", [1e-6, 1e-9, 1e-11])
def test_goes_on_past_a_sharp_drop(cuda, n, rest):
    ia, ja, al, ad, v = laplacian(n)
    b = v / np.linalg.norm(v)
    r = np.random.default_rng(n).standard_normal(n ** 3)
    b = b + rest * r / np.linalg.norm(r)
    args = (O.CSRD, True, ia, ja, al, ad, b)
    tol = 1e-3 * rest
    ref = O.pcg(*args, tol=tol, maxit=2000)
    d_it, d_x = O.order_spread(O.PCG, *args, tol=tol, maxit=2000)
    assert ref.status == sv.OK and ref.iters > 5
    g = sv.GpuSystem(n ** 3, ia, ja, sv.CSRD, True)
    g.set_values(al, ad)
    x, info = g.solve(sv.PCG, b, tol=tol, maxit=2000)
    assert info.status == sv.OK
    assert abs(info.iters - ref.iters) <= max(1, 2 * d_it)
    assert rel(x, ref.x) < max(1e-12, 20 * d_x)
    g.close()
