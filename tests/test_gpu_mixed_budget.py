"""Mixed BiCGSTAB whose on-chip part ends short of the true-residual test: the
mixed engine goes on with what is left of the call's iterations, and the
report counts both parts."""
from __future__ import annotations

import pytest

from helpers import bits_equal
from sfr3d_b200 import solver as sv
from test_gpu_onchip_bicg import flow, system

pytestmark = pytest.mark.gpu

TOL = 1e-15  # below what FP64 sums of these systems resolve


def test_the_cap_is_the_calls(cuda):
    s = flow((20, 19, 18), nrhs=2, dt=1.0)
    g = system(s)
    x, chip = g.solve_multi(sv.PBICGSTAB, s.b, tol=TOL, maxit=200)
    # the residual of the recurrence met the tolerance, the true one did not
    assert all(i.status == sv.OK for i in chip)
    missed = [not i.norm_r < i.conv for i in chip]
    assert any(missed)
    most = max(i.iters for i in chip)
    for maxit in (most, most + 1, most + 3, 200):
        y, infos = g.solve_multi(sv.PBICGSTAB, s.b, tol=TOL, maxit=maxit, precision=sv.MIXED,
                                 raise_on_error=False)
        for i, (info, ref) in enumerate(zip(infos, chip)):
            assert info.iters <= maxit + 1 and info.inner_iters == info.iters
            assert info.iters >= ref.iters
            assert (info.status == sv.MAXIT) == (info.iters == maxit + 1)
            if info.status == sv.OK:
                assert info.norm_r < info.conv
            if not missed[i]:
                assert info.iters == ref.iters
        if maxit == most:
            assert bits_equal(y, x)
            assert [i.status == sv.MAXIT for i in infos] == missed
    g.close()


def test_the_time_is_both_parts(cuda):
    s = flow((20, 19, 18), nrhs=2, dt=1.0)
    g = system(s)
    for _ in range(2):
        _, chip = g.solve_multi(sv.PBICGSTAB, s.b, tol=TOL, maxit=200)
        _, both = g.solve_multi(sv.PBICGSTAB, s.b, tol=TOL, maxit=200, precision=sv.MIXED,
                                raise_on_error=False)
        g.set_engine(sv.ENGINE_PERSISTENT)
        _, rest = g.solve_multi(sv.PBICGSTAB, s.b, x0=g.solve_multi(
            sv.PBICGSTAB, s.b, tol=TOL, maxit=200)[0], newx=False, tol=TOL,
            maxit=200 - max(i.iters for i in chip), precision=sv.MIXED, raise_on_error=False)
        g.set_engine(0)
    assert both[0].seconds > 0.5 * (chip[0].seconds + rest[0].seconds)
    g.close()
