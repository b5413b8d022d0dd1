"""What a caller's choice of engine and options selects: engine 2 the graph
engine's kernels, set_fused the PCG iteration alone, and the transposed
system's solves run as the system's own."""
from __future__ import annotations

import pytest

from helpers import bits_equal, rel
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S
from test_gpu_onchip_bicg import flow, system

pytestmark = pytest.mark.gpu

TOL, BAR = 1e-10, 1e-12


def pressure(n):
    return S.build(S.params(n=(n, n - 1, n + 1), jitter=0.2, log10k=(-1.0, 1.0), seed=8))


@pytest.mark.parametrize("n", [12, 36])
def test_engine_2_runs_the_graph_kernels(cuda, n):
    """FP64 PCG in fused mode 4, its default there, and BiCGSTAB in the graph's
    kernels, not on chip: the same bits whether or not set_fused was called,
    and others than the automatic choice's."""
    s, f = pressure(n), flow((n, n, n))
    g, h = system(s), system(f)
    auto = g.solve(sv.PCG, s.b[0], tol=TOL)[0], h.solve_multi(sv.PBICGSTAB, f.b, tol=TOL)[0]
    for sys_ in (g, h):
        sys_.set_engine(sv.ENGINE_GRAPH)
    got = g.solve(sv.PCG, s.b[0], tol=TOL)[0], h.solve_multi(sv.PBICGSTAB, f.b, tol=TOL)[0]
    for sys_ in (g, h):
        sys_.set_fused(4)
    want = g.solve(sv.PCG, s.b[0], tol=TOL)[0], h.solve_multi(sv.PBICGSTAB, f.b, tol=TOL)[0]
    for a, x, y in zip(auto, got, want):
        assert bits_equal(x, y) and not bits_equal(x, a)
        assert rel(x, a) < BAR * 20
    for sys_ in (g, h):  # back under the automatic choice
        sys_.set_engine(0)
        sys_.close()


def test_engine_2_takes_its_launch_shape(cuda):
    """Fewer slices a warp are more blocks, whose dot products add up in
    another order: the shape a caller sets reaches the solve."""
    f = flow((24, 23, 25))
    h = system(f)
    xs = []
    for spw in (1, 8):
        h.set_engine(sv.ENGINE_GRAPH, 128, spw)
        xs.append(h.solve_multi(sv.PBICGSTAB, f.b, tol=TOL)[0])
    assert not bits_equal(*xs) and rel(*xs) < BAR
    h.close()


def test_tuned_choice_still_reaches_the_on_chip_engine(cuda, tmp_path, monkeypatch):
    """The tuner times the on-chip engine for FP64 solves, keeps and stores it
    as engine 2 in mode 5, and later automatic solves take it."""
    monkeypatch.setenv("SFR_TUNE_CACHE", str(tmp_path / "tune"))
    s, f = pressure(40), flow((40, 40, 40))
    for sys_, solver, b in ((s, sv.PCG, s.b[:1]), (f, sv.PBICGSTAB, f.b)):
        g = system(sys_)
        auto, _ = g.solve_multi(solver, b, tol=TOL)
        for source in (0, 2):
            rep = g.autotune(solver, b, tol=TOL)
            assert (rep["source"], rep["engine"], rep["fused"]) == (source, 2, 5)
            assert (rep["default_engine"], rep["default_fused"]) == (2, 5)
            assert bits_equal(g.solve_multi(solver, b, tol=TOL)[0], auto)
            g.close()
            g = system(sys_)
        g.set_engine(sv.ENGINE_GRAPH)  # a chosen engine does not change what 0 stands for
        rep = g.autotune(solver, b, tol=TOL)
        assert (rep["source"], rep["default_engine"]) == (2, 2)
        assert not bits_equal(g.solve_multi(solver, b, tol=TOL)[0], auto)
        g.set_engine(0)
        assert bits_equal(g.solve_multi(solver, b, tol=TOL)[0], auto)
        g.close()


@pytest.mark.parametrize("precision", [sv.FP64, sv.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("mode", [0, 4])
def test_set_fused_concerns_pcg_alone(cuda, precision, mode, tmp_path, monkeypatch):
    monkeypatch.setenv("SFR_TUNE_CACHE", str(tmp_path / "tune"))
    s, f = pressure(20), flow((20, 21, 19))
    g, h = system(s), system(f)
    x = g.solve(sv.PCG, s.b[0], tol=TOL)[0]
    y = h.solve_multi(sv.PBICGSTAB, f.b, tol=TOL, precision=precision)[0]
    g.set_fused(mode)
    h.set_fused(mode)
    assert not bits_equal(g.solve(sv.PCG, s.b[0], tol=TOL)[0], x)
    assert bits_equal(h.solve_multi(sv.PBICGSTAB, f.b, tol=TOL, precision=precision)[0], y)
    rep = h.autotune(sv.PBICGSTAB, f.b, tol=TOL, precision=precision)
    assert rep["default_fused"] == 5
    if rep["fused"] == 5:  # the automatic choice won, and is what runs
        assert bits_equal(h.solve_multi(sv.PBICGSTAB, f.b, tol=TOL, precision=precision)[0], y)
    g.close()
    h.close()


@pytest.mark.parametrize("engine", [0, 2])
@pytest.mark.parametrize("fused", [None, 0, 3, 4])
def test_transposed_solves_run_as_the_system_does(cuda, engine, fused):
    """A symmetric system is its own transpose, entry for entry, so the same
    engine in the same mode gives the same bits."""
    s = pressure(18)
    g = system(s)
    g.set_engine(engine)
    if fused is not None:
        g.set_fused(fused)
    x, info = g.solve(sv.PCG, s.b[0], tol=TOL)
    xt, it = g.solve_transpose(sv.PCG, s.b[0], tol=TOL)
    assert bits_equal(x, xt) and info.iters == it.iters
    g.close()
