"""Mixed BiCGSTAB under the automatic engine choice: FP64 on chip where the
system fits, the mixed engines where it does not, where an engine was chosen,
and where the on-chip residual falls short of the criterion.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import bits_equal, rel
from oracle import oracle as O
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S
from test_gpu_onchip_bicg import diagonals, flow, system

pytestmark = pytest.mark.gpu

TOL = 1e-10


def residuals(s, ad, x):
    return [np.linalg.norm(s.b[i] - O.matvec(O.CSRD, True, s.ia, s.ja, s.al, ad[i], x[i]))
            / np.linalg.norm(s.b[i]) for i in range(len(x))]


@pytest.mark.parametrize("box", [(3, 1, 1), (8, 8, 8), (23, 29, 31)],
                         ids=lambda b: "x".join(map(str, b)))
@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_automatic_choice(cuda, box, k):
    s = flow(box, nrhs=k)
    ad = diagonals(s, k)
    g = system(s)
    x, infos = g.solve_multi(sv.PBICGSTAB, s.b, ad_k=ad, tol=TOL, precision=sv.MIXED)
    assert all(i.status == sv.OK for i in infos)
    # the stopping test, on a residual formed in another order
    assert max(residuals(s, ad, x)) < TOL * (1 + 1e-4)
    if k <= 3:
        y, ref = g.solve_multi(sv.PBICGSTAB, s.b, ad_k=ad, tol=TOL)
        assert bits_equal(x, y) and all(i.refinements == 0 for i in infos)
    else:
        assert any(i.refinements > 0 for i in infos)
    # a chosen engine stays the mixed one
    for engine in (1, 2):
        g.set_engine(engine)
        z, infos = g.solve_multi(sv.PBICGSTAB, s.b, ad_k=ad, tol=TOL, precision=sv.MIXED)
        assert all(i.refinements > 0 for i in infos)
        assert rel(z, x) < 1e-7
    g.close()


def test_x_in_place_of_b(cuda):
    import torch
    s = flow((12, 11, 10), nrhs=1)
    g = system(s)
    d = torch.from_numpy(s.b[0].copy()).cuda()
    info = g.solve_device(sv.PBICGSTAB, d.data_ptr(), d.data_ptr(), tol=TOL, precision=sv.MIXED)
    assert info.status == sv.OK
    assert residuals(s, [s.ad], [d.cpu().numpy()])[0] < TOL * (1 + 1e-4)
    g.close()


@pytest.mark.parametrize("tol", [1e-13, 1e-15])
def test_tolerance_near_the_floor(cuda, tol):
    """Converged means the true residual's norm met the criterion."""
    s = flow((20, 19, 18), nrhs=2, dt=1.0)
    g = system(s)
    x, infos = g.solve_multi(sv.PBICGSTAB, s.b, tol=tol, maxit=200, precision=sv.MIXED,
                             raise_on_error=False)
    for i, info in enumerate(infos):
        assert info.status in (sv.OK, sv.MAXIT, sv.BREAKDOWN)
        if info.status == sv.OK:
            assert info.norm_r < info.conv
    assert max(residuals(s, [s.ad] * 2, x)) < 1e-12
    g.close()


def test_tuned_choice(cuda, tmp_path, monkeypatch):
    monkeypatch.setenv("SFR_TUNE_CACHE", str(tmp_path / "tune"))
    s = flow((14, 13, 15), nrhs=3)
    x, sources = [], []
    for _ in range(2):  # measured, then read back
        g = system(s)
        rep = g.autotune(sv.PBICGSTAB, s.b, tol=TOL, precision=sv.MIXED)
        assert rep["default_engine"] == 0
        sources.append(rep["source"])
        x.append(g.solve_multi(sv.PBICGSTAB, s.b, tol=TOL, precision=sv.MIXED)[0])
        g.close()
    assert sources == [0, 2] and bits_equal(x[0], x[1])
    assert max(residuals(s, [s.ad] * 3, x[0])) < TOL * (1 + 1e-4)
