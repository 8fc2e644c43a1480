"""Greedy tokens of logits rows: the first of the largest, NaN never."""
import pytest
import torch

from saber_engine_b200.ops import native as N


# Rows that leave CTAs of a row's cluster without a piece, end inside a 16-byte piece, or start off a 16-byte boundary.
@pytest.mark.gpu
@pytest.mark.parametrize("V", [1, 7, 8, 63, 4096, 4099, 65544])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1])
def test_first_of_the_largest(V, dtype, off):
    rows, ld = 5, (V + 7) // 8 * 8
    g = torch.Generator().manual_seed(V)
    x = torch.randn(rows, V, generator=g).to(dtype)
    x[0, V // 2:] = x[0].max()                       # ties
    x[1, ::2] = float("nan")
    x[2] = -float("inf")
    x[3, V - 1] = float("inf")
    buf = torch.full((rows * ld + 8,), 1e9, dtype=dtype, device="cuda")
    for r in range(rows):
        buf[off + r * ld:off + r * ld + V] = x[r].cuda()
    idx, val = torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.zeros(rows, device="cuda")
    N.check(N.lib().saber_argmax_launch(buf.data_ptr() + off * buf.element_size(), int(dtype == torch.float32), rows, ld, V, 100, idx.data_ptr(), val.data_ptr(), N.stream_handle()), "argmax")
    torch.cuda.synchronize()
    for r in range(rows):
        f = x[r].float()
        best, at = -float("inf"), V
        if (~f.isnan()).any():
            best = float(f[~f.isnan()].max())
            at = int((f == best).nonzero()[0])
        assert (int(idx[r]), float(val[r])) == (100 + at, best)
