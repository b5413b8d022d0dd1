"""linear_solve on tensors that live on the GPU: the results of the host path,
for each layout, on the caller's stream, and what falls back to it.

Both paths run the same solves on the same values, so the solution agrees to
the last bits of its sums; a gradient is one product of two such values.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import layouts
from sfr3d_b200 import adjoint as A
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _gpu(s, lname):
    st, un, ia, ja, al, _ = layouts(s)[lname]
    al, au = np.split(al, 2) if lname == "csrc_unsym" else (al, None)
    return sv.GpuSystem(s.neq, ia, ja, st, un), al, au


def grads(g, values, w, solver, device, dtype=torch.float64, stream=None):
    ctx = torch.cuda.stream(stream) if stream else torch.cuda.stream(torch.cuda.current_stream())
    with ctx:
        leaves = [None if v is None else
                  torch.tensor(v, dtype=dtype, device=device).requires_grad_() for v in values]
        al, ad, au, b = leaves
        x = A.linear_solve(g, al, ad, b, au=au, solver=solver, tol=1e-12)
        kept = x.detach().clone()
        x_in_place = x * 1.0
        (torch.tensor(w, device=device) * x_in_place).sum().backward()
        out = [kept] + [t.grad for t in leaves if t is not None]
    if stream:
        stream.synchronize()
    return [t.cpu().double().numpy() for t in out]


def close(a, b, tol=1e-12):
    return all(p.shape == q.shape and np.linalg.norm(p - q) <= tol * np.linalg.norm(q)
               for p, q in zip(a, b, strict=True))


# x is solved to 1e-12 on diagonally dominant systems by the same kernel; the
# two runs differ by nothing but the order in which two gradient terms are
# added onto zero, which is exact
@pytest.mark.parametrize("n", [1, 3, 12, 33])
@pytest.mark.parametrize("lname", ["csrd_full", "csrc_unsym", "ellpack"])
def test_device_tensors_give_the_host_path_results(cuda, lname, n):
    s = S.momentum(n, peclet=20.0, seed=71, nrhs=1)
    g, al, au = _gpu(s, lname)
    w = np.random.default_rng(71).standard_normal(s.neq)
    values = (al, s.ad, au, s.b[0])
    host = grads(g, values, w, sv.PBICGSTAB, "cpu")
    assert close(grads(g, values, w, sv.PBICGSTAB, "cuda"), host)
    assert close(grads(g, values, w, sv.PBICGSTAB, "cuda", stream=torch.cuda.Stream()), host)
    g.close()


@pytest.mark.parametrize("lname", ["csrd_sym", "csrc_sym"])
def test_mirrored_values(cuda, lname):
    s = S.poisson_jittered(9, seed=72)
    g, al, au = _gpu(s, lname)
    w = np.random.default_rng(72).standard_normal(s.neq)
    values = (al, s.ad, None, s.b[0])
    assert close(grads(g, values, w, sv.PCG, "cuda"), grads(g, values, w, sv.PCG, "cpu"))
    g.close()


def test_backward_uses_the_forward_values(cuda):
    """Values and x as they were at the call, though the tensors and the
    system changed before backward; zero and strided gradients of x."""
    s = S.momentum(10, peclet=20.0, seed=73, nrhs=1)
    g, al, au = _gpu(s, "csrd_full")
    w = np.random.default_rng(73).standard_normal(s.neq)
    host = grads(g, (al, s.ad, None, s.b[0]), w, sv.PBICGSTAB, "cpu")
    leaves = [torch.tensor(v, device="cuda").requires_grad_() for v in (al, s.ad, s.b[0])]
    x = A.linear_solve(g, *leaves)
    with torch.no_grad():
        for t in leaves:
            t.mul_(1.7)
    x.detach().zero_()
    g.set_values(2.0 * al, 2.0 * s.ad)
    wd = torch.tensor(np.repeat(w, 2), device="cuda")[::2]
    got = torch.autograd.grad(x, leaves, grad_outputs=wd, retain_graph=True)
    assert close([t.cpu().numpy() for t in got], host[1:])
    zero = torch.autograd.grad(x, leaves, grad_outputs=torch.zeros_like(wd))
    assert all(not t.any() for t in zero)
    g.close()


def test_single_precision_leaves(cuda):
    s = S.momentum(8, peclet=20.0, seed=74, nrhs=1)
    g, al, au = _gpu(s, "csrd_full")
    w = np.random.default_rng(74).standard_normal(s.neq)
    values = (al, s.ad, None, s.b[0])
    dev = grads(g, values, w, sv.PBICGSTAB, "cuda", torch.float32)
    host = grads(g, values, w, sv.PBICGSTAB, "cpu", torch.float32)
    assert close(dev, host, 1e-6)  # gradients come back in single precision
    g.close()


def test_counts_are_checked_before_device_memory_is_read(cuda):
    s = S.momentum(6, peclet=20.0, seed=75, nrhs=1)
    g, al, au = _gpu(s, "csrd_full")
    t = torch.tensor(al, device="cuda")
    d = torch.tensor(s.ad, device="cuda")
    with pytest.raises(sv.SolverError) as e:
        g.set_values_device(len(al) - 1, t.data_ptr(), d.data_ptr())
    assert e.value.status == sv.BAD_INPUT
    assert A._on_device(g, t[:-1], d, None, d) is None
    assert A._on_device(g, t, d[:-1], None, d) is None
    assert A._on_device(g, t, d, None, d.cpu()) is None
    g.close()
