"""Attention of prompt portions and of images on the tensor cores against float64 of the same rounded inputs.

Bound, element by element: probabilities are rounded to bf16 (2^-8 of each at most), and 2^-13 is left for the exponential and the fp32 sums: no more
than 2^-8 + 2^-13 of sum(probability * |value|)."""
import ctypes as C

import pytest
import torch

from saber_engine_b200.ops import native as N
from saber_engine_b200.vision.tower import attn_blocks

BOUND = 2.0 ** -8 + 2.0 ** -13


def _attend(q, k, v, seen, scale):
    """[rows][H][D] x [keys][H][D]: result and sum(probability * |value|), in float64."""
    s = torch.einsum("rhd,khd->hrk", q.double(), k.double()) * scale
    w = torch.softmax(s.masked_fill(~seen, float("-inf")), -1)
    return torch.einsum("hrk,khv->rhv", w, v.double()), torch.einsum("hrk,khv->rhv", w, v.double().abs())


def _untile(t, rows, cols):
    kb = (cols + 63) // 64
    x = t.view(kb, -1, 8, 8)[:, :rows]
    at = torch.arange(8, device=t.device)[None, :] ^ (torch.arange(rows, device=t.device)[:, None] & 7)
    return torch.gather(x, 2, at[None, :, :, None].expand(kb, -1, -1, 8)).permute(1, 0, 2, 3).reshape(rows, kb * 64)[:, :cols].float()


# Two tiles of a CTA are heads of an even group or neighbouring rows: each with rows that fill, pass and leave tiles empty; a block of keys is two pages.
@pytest.mark.gpu
@pytest.mark.parametrize("lens", [(1,), (128, 129, 63), (257, 5), (640,)])
@pytest.mark.parametrize("H,G,D,V,window,chunk", [(4, 2, 128, 128, 0, 0), (3, 3, 64, 64, 0, 0), (2, 1, 192, 128, 0, 0), (5, 1, 80, 72, 0, 0), (4, 1, 64, 40, 100, 0),
                                                  (3, 1, 48, 96, 0, 64), (3, 1, 64, 192, 0, 0)])
def test_prompt_portions_match_float64(lens, H, G, D, V, window, chunk):
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + D)
    scale, pages_of = D ** -0.5, [(n + 63) // 64 for n in lens]
    KP, VP, most = (D + 63) // 64 * 64, (V + 31) // 32 * 32, max(pages_of)
    table = torch.zeros(len(lens), most, dtype=torch.int32)
    order = torch.randperm(sum(pages_of), generator=torch.Generator().manual_seed(1)).int()
    for j, n in enumerate(pages_of):
        table[j, :n] = order[sum(pages_of[:j]):sum(pages_of[:j]) + n]
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32).cuda()                      # noqa: E731
    cache = torch.zeros(sum(pages_of) * G * 64 * (KP + VP), dtype=torch.bfloat16, device="cuda")
    err, table_d = i32([0, 0, 0, 0]), table.cuda()
    x = [torch.randn(n, H * D + G * D + G * V, generator=g, device="cuda").bfloat16().float() for n in lens]
    done, out = [0] * len(lens), [[] for _ in lens]
    for part in (0.4, 1.0):                                                           # the second portion meets the first one's keys
        upto = [max(1, int(n * part)) for n in lens]
        rows = [u - d for u, d in zip(upto, done)]
        M = sum(rows)
        if M == 0:
            continue
        xs = torch.cat([x[j][done[j]:upto[j]] for j in range(len(lens))]).contiguous()
        pos = [t for j in range(len(lens)) for t in range(done[j], upto[j])]
        slot = [int(table[j, t // 64]) * 64 + t % 64 for j in range(len(lens)) for t in range(done[j], upto[j])]
        o, q = torch.zeros(M, H * V, device="cuda"), torch.zeros(M, H, D, dtype=torch.bfloat16, device="cuda")
        cu, kv, pos, slot = i32([sum(rows[:j]) for j in range(len(lens) + 1)]), i32(upto), i32(pos), i32(slot)
        p = N.GqaParams()
        p.x, p.ldx, p.q_off, p.k_off, p.v_off, p.g_off = xs.data_ptr(), xs.shape[1], 0, H * D, (H + G) * D, -1
        p.cache, p.q, p.slot_map, p.pos, p.cu_rows, p.kv_len, p.block_table = (t.data_ptr() for t in (cache, q, slot, pos, cu, kv, table_d))
        p.out = N.Operand(o.data_ptr(), M, H * V, 1)
        p.M, p.nseq, p.H, p.G, p.D, p.DK, p.KP, p.V, p.VP, p.page = M, len(lens), H, G, D, D, KP, V, VP, 64
        p.n_blocks, p.max_blocks, p.form, p.max_rows, p.chunk, p.window, p.scale, p.eps, p.out_scale = sum(pages_of), most, 2, max(rows), chunk, window, scale, 1e-6, 1.0
        p.err = err.data_ptr()
        assert N.lib().saber_gqa_form(C.byref(p)) == 2
        N.check(N.lib().saber_gqa_launch(C.byref(p), N.stream_handle()), "gqa")
        torch.cuda.synchronize()
        assert int(err[0]) == 0
        for j in range(len(lens)):
            out[j].append(o[sum(rows[:j]):sum(rows[:j]) + rows[j]].view(-1, H, V))
        done = upto
    for j, n in enumerate(lens):
        q, k, v = x[j][:, :H * D].view(n, H, D), x[j][:, H * D:(H + G) * D].view(n, G, D), x[j][:, (H + G) * D:].view(n, G, V)
        i, t = torch.arange(n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
        seen = (t <= i) & ((i - t < window) if window else True) & ((t // chunk == i // chunk) if chunk else True)
        want, size = _attend(q, k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), seen, scale)
        assert bool(((torch.cat(out[j]).double() - want).abs() <= BOUND * size).all())


@pytest.mark.gpu
@pytest.mark.parametrize("grids", [[(1, 2, 2)], [(1, 8, 8), (1, 2, 32), (1, 10, 13)], [(1, 16, 16), (1, 2, 2)], [(1, 18, 22)], [(2, 12, 12)] + [(1, 2, 2)] * 20])
def test_images_match_float64(grids):
    heads, hd, n = 3, 72, [t * h * w for t, h, w in grids]
    M, W = sum(n), heads * hd
    g = torch.Generator(device="cuda").manual_seed(M)
    qkv = torch.randn(M, 3 * W, generator=g, device="cuda").bfloat16()
    ang = torch.rand(M, hd // 2, generator=g, device="cuda") * 6
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32).cuda()                      # noqa: E731
    blocks, per = torch.from_numpy(attn_blocks(grids)).cuda(), [(x + 63) // 64 for x in n]
    pages = torch.zeros(len(n), max(per), dtype=torch.int32)
    for j, c in enumerate(per):
        pages[j, :c] = sum(per[:j]) + torch.arange(c)
    size = [C.c_size_t() for _ in range(3)]
    N.lib().saber_vis_attn_scratch(blocks.shape[0], M, heads, *(C.byref(s) for s in size))
    scratch = [torch.full((s.value,), 255, dtype=torch.uint8, device="cuda") for s in size]      # (NaN wherever nothing is written)
    m_pad = (M + 31) // 32 * 32
    out, err = torch.zeros((W + 63) // 64 * m_pad * 64, dtype=torch.bfloat16, device="cuda"), i32([0, 0, 0, 0])
    cos, sin, cu, kv, pages_d = ang.cos().contiguous(), ang.sin().contiguous(), i32([sum(n[:j]) for j in range(len(n) + 1)]), i32(n), pages.cuda()
    p = N.VisAttnParams()
    p.qkv, p.ldq, p.cos_t, p.sin_t, p.out_tiled, p.M_pad, p.blocks = qkv.data_ptr(), 3 * W, cos.data_ptr(), sin.data_ptr(), out.data_ptr(), m_pad, blocks.data_ptr()
    p.heads, p.width, p.scale = heads, W, hd ** -0.5
    p.q, p.k, p.v = (s.data_ptr() for s in scratch)
    p.cu_rows, p.kv_len, p.pages, p.images, p.max_pages, p.max_rows, p.err = cu.data_ptr(), kv.data_ptr(), pages_d.data_ptr(), len(n), max(per), max(n), err.data_ptr()
    N.check(N.lib().saber_vis_attn_launch(C.byref(p), blocks.shape[0], N.stream_handle()), "vis_attn")
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    got = _untile(out, M, W).view(M, heads, hd)
    half = hd // 2

    def turn(x):                     # in float32 and rounded once, as the kernel does: of the same products, whichever is fused
        a, b, c, s = x[..., :half].double(), x[..., half:].double(), cos.double()[:, None], sin.double()[:, None]
        return torch.cat([a * c - b * s, b * c + a * s], -1).bfloat16()
    q, k, v = (qkv[:, i * W:(i + 1) * W].view(M, heads, hd) for i in range(3))
    q, k = turn(q), turn(k)
    for j, c in enumerate(n):
        at = slice(sum(n[:j]), sum(n[:j]) + c)
        want, mag = _attend(q[at], k[at], v[at], torch.ones(c, c, dtype=torch.bool, device="cuda"), p.scale)
        # 2^-8 more for the result's own bf16.  (A rotated value next to a rounding edge may fall to its other side: one bf16 step of one of 72 products, far
        # below the roundings counted, as those are never all at their largest.)
        assert bool(((got[at].double() - want).abs() <= (BOUND + 2.0 ** -8) * mag).all())
