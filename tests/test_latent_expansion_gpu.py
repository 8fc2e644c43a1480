"""Keys and values of a prompt portion's pages from their latents (mla_expand_tc.cu) against float64."""
import ctypes as C

import pytest
import torch

from saber_engine_b200.ops import native as N

DEV = "cuda"


# Weight tiles of 128 rows that cut heads, end inside one or are few; latents in whole and part k-blocks; a sequence whose last pair of pages is one page.
# (20: heads that are no whole groups of eight values, the `mma.sync` form.)
@pytest.mark.gpu
@pytest.mark.parametrize("H,D,V,c", [(2, 128, 128, 512), (3, 8, 40, 16), (5, 72, 64, 80), (1, 40, 128, 272), (24, 128, 96, 512), (3, 20, 24, 64)])
@pytest.mark.parametrize("lens,rows", [((70, 200), (70, 33)), ((1, 64), (1, 1)), ((640, 129), (5, 129))])
def test_expanded_pages_match_float64(H, D, V, c, lens, rows):
    g = torch.Generator(device=DEV).manual_seed(H + D + lens[0])
    R, CP, DP = 16, (c + 15) // 16 * 16, (D + 15) // 16 * 16
    VP = next(n for n in (32, 64, 128) if n >= V)
    RP, KT, pages = 16, (DP + 16 + 63) // 64, [(n + 63) // 64 for n in lens]
    n_blocks, M = sum(pages) + 2, sum(rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).bfloat16()                       # noqa: E731
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32).to(DEV)                              # noqa: E731
    cache, uk, uv = rnd(n_blocks, 64, CP + RP), rnd(H * D, CP), rnd(H * V, CP)
    cache[:, :, c:CP], uk[:, c:], uv[:, c:] = 0, 0, 0
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(3)) + 1
    table = torch.zeros(2, max(pages), dtype=torch.int32)
    for j in range(2):
        table[j, :pages[j]] = order[sum(pages[:j]):sum(pages[:j]) + pages[j]].int()
    k_exp, v_exp = torch.zeros(n_blocks, H, KT, 64, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(n_blocks, H, VP, 64, dtype=torch.bfloat16, device=DEV)
    x, q, out = torch.randn(M, 1024 + H * V, generator=g, device=DEV), torch.randn(M, H * (D + R), generator=g, device=DEV), torch.zeros(M, H * V, device=DEV)
    q_eff, freq, err = torch.zeros(M * H * (max(CP, DP) + RP), dtype=torch.bfloat16, device=DEV), torch.rand(R // 2, generator=g, device=DEV), i32([0] * 4)
    slot = i32([int(table[j, t // 64]) * 64 + t % 64 for j in range(2) for t in range(lens[j] - rows[j], lens[j])])
    pos, cu, kl, tab = i32([t for j in range(2) for t in range(lens[j] - rows[j], lens[j])]), i32([0, rows[0], M]), i32(lens), table.to(DEV)
    p = N.MlaParams()
    p.x, p.ldx, p.q_off, p.dkv_off, p.g_off, p.q, p.ldq = x.data_ptr(), x.shape[1], 0, -1, 0, q.data_ptr(), q.shape[1]
    p.rot_amp, p.freq, p.w_uk, p.w_uv, p.cache, p.q_eff, p.k_exp, p.v_exp = 1.0, *(t.data_ptr() for t in (freq, uk, uv, cache, q_eff, k_exp, v_exp))
    p.slot_map, p.pos, p.cu_rows, p.kv_len, p.block_table, p.err = (t.data_ptr() for t in (slot, pos, cu, kl, tab, err))
    p.out, p.M, p.nseq, p.H, p.D, p.R, p.V, p.C, p.CP, p.RP, p.DP, p.VP = N.Operand(out.data_ptr(), M, H * V, 1), M, 2, H, D, R, V, c, CP, RP, DP, VP
    p.page, p.n_blocks, p.max_blocks, p.splits, p.expand, p.max_rows, p.scale, p.eps = 64, n_blocks, max(pages), 1, 2, max(rows), (D + R) ** -0.5, 1e-6
    assert N.lib().saber_mla_expand_ok(C.byref(p)) == 2
    N.check(N.lib().saber_mla_launch(C.byref(p), N.stream_handle()), "mla")
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    swz = torch.arange(8, device=DEV)[None] ^ (torch.arange(64, device=DEV)[:, None] & 7)
    keys = torch.gather(k_exp.view(n_blocks, H, KT, 64, 8, 8), 4, swz[None, None, None, :, :, None].expand(n_blocks, H, KT, -1, -1, 8))
    keys = keys.permute(0, 3, 1, 2, 4, 5).reshape(n_blocks, 64, H, KT * 64).double()
    vz = torch.arange(8, device=DEV)[None] ^ (torch.arange(VP, device=DEV)[:, None] & 7)
    vals = torch.gather(v_exp.view(n_blocks, H, VP, 8, 8), 3, vz[None, None, :, :, None].expand(n_blocks, H, -1, -1, 8)).reshape(n_blocks, H, VP, 64)[:, :, :V].double()
    lat = cache[:, :, :CP].double()
    seen = torch.unique(torch.cat([table[j, :pages[j]] for j in range(2)])).long().to(DEV)
    for got, w, n, how in ((keys[..., :D], uk, D, "btc,hdc->bthd"), (vals, uv, V, "btc,hdc->bhdt")):
        want, size = torch.einsum(how, lat, w.double().view(H, n, CP)), torch.einsum(how, lat.abs(), w.double().abs().view(H, n, CP))
        assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + CP * 2.0 ** -24 * size)[seen].all())         # one rounding to bf16, fp32 sums
    assert torch.equal(keys[seen][..., DP:DP + RP], cache[seen][:, :, None, CP:].double().expand(-1, -1, H, -1))
    assert not k_exp[0].any() and not v_exp[0].any()
