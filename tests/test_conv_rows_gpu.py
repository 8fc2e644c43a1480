"""The causal convolution of prompt portions (gdn.cu) against float64."""
import ctypes as C

import pytest
import torch

from saber_engine_b200.ops import native as N


# Rows that end ahead of, on and behind the eight of a round and the sixteen of a CTA; heads that do and do not fill the last CTA's four warps; x rows
# that are not whole 8-byte groups apart (the row-at-a-time form).
@pytest.mark.gpu
@pytest.mark.parametrize("lens", [(1,), (7, 8, 9), (16, 17), (300, 2, 33)])
@pytest.mark.parametrize("q,k,v,extra", [(1, 1, 2, 0), (2, 2, 3, 4), (0, 0, 1, 0), (2, 1, 2, 3)])
def test_committing_rows_match_float64(lens, q, k, v, extra):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + q + v)
    Cc, M, scale = (q + k + v) * 128, sum(lens), 128 ** -0.5
    ld = Cc + extra
    x, w = torch.randn(M, ld, generator=g, device="cuda").bfloat16(), torch.randn(Cc, 4, generator=g, device="cuda")
    hist = torch.randn(len(lens) + 1, 5, Cc, generator=g, device="cuda").bfloat16()
    old, out = hist.clone(), torch.full((M, Cc), float("nan"), device="cuda")
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32).cuda()                        # noqa: E731
    cu, slots, shift = i32([sum(lens[:j]) for j in range(len(lens) + 1)]), i32([j + 1 for j in range(len(lens))]), i32([j % 3 for j in range(len(lens))])
    p = N.GdnConvParams()
    p.x, p.conv_w, p.hist, p.cu_rows, p.slots, p.shift, p.out = (t.data_ptr() for t in (x, w, hist, cu, slots, shift, out))
    p.C, p.n_q, p.n_k, p.ldx, p.hist_rows, p.commit, p.q_scale, p.max_rows = Cc, q * 128, k * 128, ld, 5, 1, scale, max(lens)
    N.check(N.lib().saber_gdn_conv_launch(C.byref(p), len(lens), N.stream_handle()), "conv")
    torch.cuda.synchronize()
    for j, n in enumerate(lens):
        r0 = sum(lens[:j])
        rows = torch.cat([old[j + 1, j % 3:j % 3 + 3], x[r0:r0 + n, :Cc]]).double()
        y = sum(rows[i:i + n] * w[:, i].double() for i in range(4))
        y = (y * torch.sigmoid(y)).view(n, -1, 128)
        f = 1 / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)
        want = torch.cat([y[:, :q] * f[:, :q] * scale, y[:, q:q + k] * f[:, q:q + k], y[:, q + k:]], 1).view(n, Cc)
        got = out[r0:r0 + n].double()
        # four products (4 units of 2^-24 of the sum of their sizes), the fast exponential and quotient (a few units of 2^-22), a head's norm
        size = sum(rows[i:i + n].abs() * w[:, i].double().abs() for i in range(4)).view(n, -1, 128)
        size = torch.cat([size[:, :q] * f[:, :q] * scale, size[:, q:q + k] * f[:, q:q + k], size[:, q + k:]], 1).view(n, Cc)
        assert bool(((got - want).abs() <= 2.0 ** -19 * size + 2.0 ** -19 * want.abs()).all())
        assert torch.equal(hist[j + 1, :3], torch.cat([old[j + 1, j % 3:j % 3 + 3], x[r0:r0 + n, :Cc]])[-3:])
