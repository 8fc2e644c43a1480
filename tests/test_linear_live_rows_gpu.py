"""Linears of a bucket whose step brings fewer rows: the step's rows as without the bound, the others untouched."""
import ctypes as C

import pytest
import torch

from saber_engine_b200.models import stack_weights as SW
from saber_engine_b200.ops import functional as F
from saber_engine_b200.ops import layouts as L
from saber_engine_b200.ops import native as N


@pytest.mark.gpu
@pytest.mark.parametrize("M,n,K,splits,fp32", [(512, 1000, 192, 1, 0), (256, 40, 640, 5, 0), (1024, 12800, 64, 1, 0), (300, 520, 128, 1, 1), (300, 520, 128, 1, 0)])
@pytest.mark.parametrize("live", [0, 1, 128, 129, 200, 255, 256])
@pytest.mark.parametrize("fuse", [1, 0])
def test_rows_behind_the_step_are_left_alone(M, n, K, splits, fp32, live, fuse):
    g = torch.Generator(device="cuda").manual_seed(M + n)
    n_pad, m_pad, dt = L.round_up(n, 256), L.padded_rows(M), torch.float32 if fp32 else torch.bfloat16
    w = torch.zeros(n_pad, K, device="cuda")
    w[:n] = torch.randn(n, K, generator=g, device="cuda") / K ** 0.5
    lin = SW.pack_linear(w.to(dt), dt)
    a = torch.randn(m_pad * K, generator=g, device="cuda").to(dt)          # (as tiles or rows: the same operand for both launches)
    sc, ws = F.scratch("cuda"), torch.zeros(M * n_pad + (1 << 23), device="cuda")
    rows = torch.tensor([live], dtype=torch.int32, device="cuda")
    outs = []
    for bound in (None, rows.data_ptr()):
        out = torch.full((M, L.round_up(n, 8)), 7.0, device="cuda")
        p = N.LinParams()
        p.w, p.a, p.err, p.ws, p.counters = lin.w.data_ptr(), a.data_ptr(), sc.err.data_ptr(), ws.data_ptr(), sc.counters.data_ptr()
        p.M, p.M_pad, p.N_pad, p.K, p.nt, p.splits, p.fp32, p.fuse, p.live = M, m_pad, n_pad, K, L.token_tile(M), splits, fp32, fuse, bound
        p.mtiles = 2 if m_pad % 256 == 0 and splits == 1 else 1
        p.e.out, p.e.ldo, p.e.n_plain, p.e.act_tile0 = out.data_ptr(), out.stride(0), n, n_pad // 256
        N.check(N.lib().saber_linear_launch(C.byref(p), N.stream_handle()), "linear")
        torch.cuda.synchronize()
        sc.check()
        outs.append(out)
    upto = live if live else M                                             # (no rows: a bucket's walk ahead of its capture, all of them)
    assert torch.equal(outs[0][:upto], outs[1][:upto]) and bool((outs[1][upto:] == 7.0).all())
