"""On-chip FP64 PCG (onchip.cu) with x over the right-hand side or over the
call's own diagonal: the same bits as with arrays apart."""
from __future__ import annotations

import pytest

from helpers import bits_equal
from sfr3d_b200 import solver as sv
from sfr3d_b200 import systems as S

pytestmark = pytest.mark.gpu


# the cluster; slots held; levels 3, 2, 1 and 0
@pytest.mark.parametrize("box", [(12, 11, 10), (60, 61, 59), (80, 79, 81), (96, 95, 97),
                                 (112, 113, 111), (128, 128, 127)],
                         ids=lambda b: "x".join(map(str, b)))
def test_x_over_b_or_the_diagonal(cuda, box):
    torch = cuda
    s = S.build(S.params(n=box, jitter=0.2, log10k=(-1.0, 1.0), seed=8))
    n = s.neq
    g = sv.GpuSystem(n, s.ia, s.ja, sv.CSRD, True)
    g.set_values(s.al, s.ad)
    b, ad = (torch.from_numpy(v).cuda() for v in (s.b[0].copy(), 1.1 * s.ad))

    def solve(tb, tad, px):
        torch.cuda.synchronize()
        info = g.solve_multi_device(sv.PCG, 1, tb, px, d_ad_k=tad, tol=1e-8, maxit=60)[0]
        return info.iters, info.xKx, info.norm_x, info.norm_r, info.norm_r_m, info.conv

    want = torch.zeros_like(b)
    ref = solve(b.data_ptr(), ad.data_ptr(), want.data_ptr())
    for shift in (0, n // 2):
        for over in ("b", "ad"):
            buf = torch.zeros(n + shift, dtype=torch.float64, device="cuda")
            buf[shift:] = b if over == "b" else ad
            src = buf.data_ptr() + 8 * shift
            got = solve(src if over == "b" else b.data_ptr(),
                        src if over == "ad" else ad.data_ptr(), buf.data_ptr())
            assert bits_equal(buf[:n].cpu().numpy(), want.cpu().numpy()), (over, shift)
            assert got == ref, (over, shift)
    g.close()
