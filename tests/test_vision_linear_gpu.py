"""The tower's rows and linears against float64 of the same operands."""
import ctypes as C

import pytest
import torch

from saber_engine_b200.ops import native as N


def _tiled(x, rows):
    """[n][K] -> [k-block][rows][64], 16-byte pieces XOR (row & 7)."""
    n, K = x.shape
    kb = (K + 63) // 64
    t = torch.zeros(rows, kb * 64, dtype=torch.bfloat16, device="cuda")
    t[:n, :K] = x
    t = t.view(rows, kb, 8, 8)
    at = torch.arange(8, device="cuda")[None, :] ^ (torch.arange(rows, device="cuda")[:, None] & 7)
    return torch.gather(t, 2, at[:, None, :, None].expand(-1, kb, -1, 8)).transpose(0, 1).contiguous()


# Every tile width and cut of the reduction (by the shapes that choose them), ragged rows, columns and reductions; several tiles of a CTA.
@pytest.mark.gpu
@pytest.mark.parametrize("M,N_,K", [(1, 8, 64), (127, 72, 576), (129, 1152, 4304), (308, 1152, 4304), (308, 4304, 1152), (640, 3456, 1152), (1024, 1160, 584), (4096, 3456, 192),
                                    (4100, 4304, 320), (33, 520, 4608)])
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
def test_linear_matches_float64(M, N_, K, epi):
    g = torch.Generator(device="cuda").manual_seed(M + N_ + epi)
    x, w = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((M, K), (N_, K)))
    w = (w.float() * K ** -0.5).bfloat16()
    b, res = torch.randn(N_, generator=g, device="cuda"), torch.randn(M, N_, generator=g, device="cuda").bfloat16()
    m_pad, n_pad, ldo = (M + 31) // 32 * 32, (N_ + 255) // 256 * 256, (N_ + 7) // 8 * 8
    a_t, w_t = _tiled(x, m_pad), torch.cat([_tiled(w[i:i + 256], 256)[None] for i in range(0, N_, 256)]).contiguous()
    out = torch.full((M, ldo), 7.0, dtype=torch.bfloat16, device="cuda")
    if epi == 3:
        out[:, :N_] = res
    ws, counters, err = torch.zeros(148 * 256 * 128, device="cuda"), torch.zeros(148, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    p = N.VisLinearParams()
    p.w, p.a, p.bias, p.res, p.out, p.ws, p.counters, p.err = (t.data_ptr() for t in (w_t, a_t, b, out, out, ws, counters, err))
    p.M, p.M_pad, p.N, p.N_pad, p.K, p.ldo, p.epi = M, m_pad, N_, n_pad, (K + 63) // 64 * 64, ldo, epi
    N.check(N.lib().saber_vis_linear_launch(C.byref(p), N.stream_handle()), "vis_linear")
    torch.cuda.synchronize()
    assert int(err[0]) == 0 and int(counters.abs().sum()) == 0
    y = x.double() @ w.double().T + b.double()
    size = x.double().abs() @ w.double().abs().T
    if epi in (1, 2):
        want = 0.5 * y * (1 + torch.tanh(0.7978845608028654 * (y + 0.044715 * y ** 3))) if epi == 1 else torch.nn.functional.gelu(y)
    else:
        want = y + res.double() if epi == 3 else y
    # Two roundings to bf16 (2^-8 each of the linear's value, whose slope through the gelu is at most 1.13, and of the result), fp32 sums of K products
    # (K 2^-24 of the sum of their sizes at most), and the fast tanh's 2^-10.5 of half the value.
    bound = 1.2 * 2.0 ** -8 * y.abs() + 2.0 ** -8 * want.abs() * (1 + 2.0 ** -8) + K * 2.0 ** -24 * size + (2.0 ** -11 * y.abs() if epi in (1, 2) else 0)
    assert bool(((out[:, :N_].double() - want).abs() <= bound + 1e-6).all())
    assert bool((out[:, N_:] == 7.0).all())


# A row per warp up to 1280 columns, per CTA beyond; ragged last warps; rows grouped by four; fp32 and bf16 rows.
@pytest.mark.gpu
@pytest.mark.parametrize("M,K,group", [(1, 72, 1), (5, 1152, 1), (130, 1280, 1), (33, 1288, 1), (9, 4608, 1), (6, 128, 4), (40, 1152, 4), (8, 1344, 4)])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_match_float64(M, K, group, norm, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = (torch.randn(M, K, generator=g, device="cuda") * 3 + 1).to(dtype)
    w, b = torch.randn(K, generator=g, device="cuda"), torch.randn(K, generator=g, device="cuda")
    k_pad, rows = (K + 63) // 64 * 64, (M + group - 1) // group
    m_pad = (rows + 31) // 32 * 32
    out = torch.full((k_pad * group // 64, m_pad, 8, 8), 7.0, dtype=torch.bfloat16, device="cuda")
    p = N.VisRowsParams()
    p.x, p.x_f32, p.ldx, p.tiled, p.eps = x.data_ptr(), int(dtype == torch.float32), K, out.data_ptr(), 1e-6
    p.ln_w, p.ln_b = (w.data_ptr(), b.data_ptr()) if norm else (None, None)
    p.M, p.K, p.K_pad, p.M_pad, p.group = M, K, k_pad, m_pad, group
    N.check(N.lib().saber_vis_rows_launch(C.byref(p), N.stream_handle()), "vis_rows")
    torch.cuda.synchronize()
    at = torch.arange(8, device="cuda")[None, :] ^ (torch.arange(m_pad, device="cuda")[:, None] & 7)
    got = torch.gather(out, 2, at[None, :, :, None].expand(out.shape[0], -1, -1, 8)).transpose(0, 1).reshape(m_pad, -1)[:rows].double()
    want = x.double()
    size = torch.zeros_like(want)
    if norm:
        d = want - want.mean(-1, keepdim=True)
        f = torch.rsqrt((d * d).mean(-1, keepdim=True) + 1e-6)
        want, size = d * f * w.double() + b.double(), (d * f * w.double()).abs() + b.double().abs()
    full = torch.zeros(rows * group, K if group > 1 else k_pad, dtype=torch.float64, device="cuda")
    room = torch.zeros_like(full)
    full[:M, :K], room[:M, :K] = want, 2.0 ** -8 * want.abs() + 2.0 ** -16 * size              # one rounding to bf16; fp32 sums of a row
    got, full, room = got[:, :full.shape[1] * group], full.view(rows, -1), room.view(rows, -1)
    live = torch.arange(rows * group, device="cuda").view(rows, group).repeat_interleave(full.shape[1] // group, 1) < M
    assert bool(((got - full).abs() <= room)[live].all())
