"""Paged attention on tcgen05 (fp8 pages) against float64 over the same rounded operands."""
import ctypes as C

import pytest
import torch

from saber_engine_b200.ops import native as N

D, PAGE = 256, 16


def _pages(k, v, order, n_blocks, nkv):
    """Keys and values [tokens][nkv][256] as the pool's pages, in the order that the kernel multiplies."""
    n = len(order)
    pad = lambda t: torch.cat([t, torch.zeros(n * PAGE - t.shape[0], nkv, D, device="cuda")]).view(n, PAGE, nkv, D)    # noqa: E731
    pool = torch.zeros(n_blocks, nkv, 2, 4096, dtype=torch.float8_e4m3fn, device="cuda")
    kk = pad(k).view(n, 2, 8, nkv, 16, 16).permute(0, 3, 1, 4, 2, 5).reshape(n, nkv, 4096)      # [2 key groups][16 dim chunks][8 keys][16 dims]
    vv = pad(v).view(n, PAGE, nkv, 32, 8).permute(0, 2, 3, 4, 1).reshape(n, nkv, 4096)          # [32 dim groups][8 dims][16 keys]
    pool[order, :, 0], pool[order, :, 1] = kk.to(torch.float8_e4m3fn), vv.to(torch.float8_e4m3fn)
    return pool


# Tiles of 128 keys in groups of four looked up ahead, query tiles of 128 / group tokens; a row of zeros; windows that begin and end inside a tile.
@pytest.mark.gpu
@pytest.mark.parametrize("nq,nkv", [(24, 4), (8, 8), (16, 1)])
@pytest.mark.parametrize("rows,past,window", [(1, 0, 0), (21, 0, 0), (22, 107, 0), (130, 383, 0), (64, 1000, 0), (40, 520, 100), (200, 0, 33)])
def test_prompt_rows_match_float64(rows, past, window, nq, nkv):
    g = torch.Generator(device="cuda").manual_seed(rows + past + nq)
    kv, scale = rows + past, D ** -0.5
    q = (torch.randn(rows, nq, D, generator=g, device="cuda") * 2).bfloat16()
    q[rows // 2, 0] = 0
    f8 = lambda t: t.to(torch.float8_e4m3fn).float()                                            # noqa: E731
    k, v = (f8(torch.randn(kv, nkv, D, generator=g, device="cuda")) for _ in range(2))
    n = (kv + PAGE - 1) // PAGE
    order = torch.randperm(n, generator=torch.Generator().manual_seed(kv)) + 1
    pool = _pages(k, v, order.cuda(), n + 1, nkv)
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32).cuda()                                # noqa: E731
    out, err, table, cu, kl = torch.zeros(rows, nq, D, dtype=torch.bfloat16, device="cuda"), i32([0] * 4), order.int().cuda(), i32([0, rows]), i32([kv])
    p = N.AttnParams()
    p.q, p.kv_cache, p.block_table, p.cu_q, p.kv_len, p.out, p.err = (t.data_ptr() for t in (q, pool, table, cu, kl, out, err))
    p.nseq, p.nq, p.nkv, p.max_blocks, p.splits, p.q_tiles, p.n_blocks, p.impl, p.window = 1, nq, nkv, n, 1, (rows + 15) // 16, n + 1, 1, window
    p.sm_scale, p.k_scale, p.v_scale = scale, 1.0, 1.0
    N.check(N.lib().saber_attn_tc_launch(C.byref(p), N.stream_handle()), "attn")
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    amax = q.float().abs().amax(-1, keepdim=True)
    q8 = f8(q.float() * torch.where(amax > 0, 448.0 / amax, 0.0)).double() * (amax.double() / 448.0)
    s = torch.einsum("rhd,khd->hrk", q8, k.double().repeat_interleave(nq // nkv, 1)) * scale
    i, t = torch.arange(past, kv, device="cuda")[:, None], torch.arange(kv, device="cuda")[None]
    seen = (t <= i) & ((i - t < window) if window else True)
    w, vv = torch.softmax(s.masked_fill(~seen, float("-inf")), -1), v.double().repeat_interleave(nq // nkv, 1)
    want = torch.einsum("hrk,khv->rhv", w, vv)
    # Probabilities as e4m3, relative to a reference that is the row's maximum or up to 2^8 below: half a unit in the last place is 2^-4 of a value, or
    # 2^-10 of the largest one; 2^-7 for the result's bf16, the scale of a query row (one division in fp32, a few units of 2^-24) and fp32 sums.
    size, flat = torch.einsum("hrk,khv->rhv", w, vv.abs()), torch.einsum("hrk,khv->rhv", seen.double().expand_as(w) * w.amax(-1, keepdim=True), vv.abs())
    assert bool(((out.double() - want).abs() <= (2.0 ** -4 + 2.0 ** -7) * size + 2.0 ** -10 * flat).all())
