"""Delta rules over prompt portions in chunks of sixteen tokens, against float64."""
import ctypes as C
import math

import pytest
import torch

from saber_engine_b200.ops import native as N

DEV = "cuda"
# A chunk passes through some 32 fp32 roundings of 2^-24 and the rules contract, so that a few chunks' errors add up.
BOUND = 64 * 2.0 ** -24
# Ragged portions that end ahead of, on and behind a chunk's last token; a sequence without rows in a portion.
PIECES = [[[90, 33, 17, 1]], [[16, 15, 1, 0], [17, 1, 16, 1], [57, 17, 0, 0]], [[31, 33, 15, 1], [59, 0, 2, 0]]]


def _f32(*s):
    return torch.zeros(*s, device=DEV)


def _i32(a):
    return torch.as_tensor(a, dtype=torch.int32).to(DEV)


def _offsets(parts):
    off, n = {}, 0
    for k, c in parts:
        off[k] = n
        n = (n + c + 7) // 8 * 8
    return off, n


def _near(got, want):
    assert float((got.double() - want).norm()) <= BOUND * float(want.norm())


def _portions(pieces, launch):
    """Calls launch(rows per sequence, first token of each) for the pieces, and gives the lengths."""
    done = [0] * len(pieces[0])
    for piece in pieces:
        if sum(piece):
            launch(piece, list(done))
        done = [d + n for d, n in zip(done, piece)]
    return done


def _tables(piece, done):
    cu = [sum(piece[:j]) for j in range(len(piece) + 1)]
    return _i32(cu), _i32([j + 1 for j in range(len(piece))]), _i32([done[j] + i for j in range(len(piece)) for i in range(piece[j])]), cu


@pytest.mark.gpu
@pytest.mark.parametrize("pieces", PIECES)
@pytest.mark.parametrize("H,HK,D,V", [(4, 2, 128, 128), (3, 3, 64, 48), (6, 1, 40, 20), (2, 1, 192, 36), (2, 2, 256, 64)])
@pytest.mark.parametrize("gate", [0.1, 4.0])
def test_delta_rule(H, HK, D, V, gate, pieces):
    taps, lens = 4, [sum(p[j] for p in pieces) for j in range(4)]
    DP, VP, g = (D + 63) // 64 * 64, (V + 7) // 8 * 8, torch.Generator(device=DEV).manual_seed(H + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)                  # noqa: E731
    off, ld = _offsets((("q", HK * D), ("k", HK * D), ("v", H * V), ("b", H), ("a", H), ("g", H * V)))
    x = [rnd(n, ld) for n in lens]
    for t in x:
        t[:, off["a"]:off["a"] + H] *= gate
    Cc = 2 * HK * D + H * V
    cw, A_log, nw = rnd(Cc, taps) * 0.5, torch.log(torch.rand(H, generator=g, device=DEV) * 15 + 1), torch.ones(V, device=DEV)
    dt = torch.log(torch.expm1(torch.exp(torch.rand(H, generator=g, device=DEV) * math.log(100.0) + math.log(1e-3))))
    state, hist, err = _f32(5, H, VP, DP), _f32(5, taps, Cc), _i32([0] * 4)
    got = [[] for _ in lens]

    def launch(piece, done):
        cu, slots, pos, at = _tables(piece, done)
        M = at[-1]
        xs, o, out = torch.cat([x[j][done[j]:done[j] + n] for j, n in enumerate(piece)]).contiguous(), _f32(M, H, VP), _f32(M, H * V)
        p = N.DeltaParams()
        p.x, p.ldx = xs.data_ptr(), ld
        p.q_off, p.k_off, p.v_off, p.b_off, p.a_off, p.g_off = (off[z] for z in "qkvbag")
        p.conv_w, p.A_log, p.dt_bias, p.norm_w, p.hist, p.state, p.o = (t.data_ptr() for t in (cw, A_log, dt, nw, hist, state, o))
        p.cu_rows, p.slots, p.pos, p.out, p.err = cu.data_ptr(), slots.data_ptr(), pos.data_ptr(), N.Operand(out.data_ptr(), M, H * V, 1), err.data_ptr()
        p.M, p.nseq, p.H, p.HK, p.D, p.DP, p.V, p.VP, p.taps, p.n_slots = M, 4, H, HK, D, DP, V, VP, taps, 5
        p.eps, p.unit_eps, p.q_scale = 1e-6, 1e-6, D ** -0.5
        floats = N.lib().saber_delta_chunk_floats(C.byref(p))
        assert floats > 0
        scratch = torch.full((floats,), float("nan"), device=DEV)
        p.chunk = scratch.data_ptr()
        N.check(N.lib().saber_delta_launch(C.byref(p), 0, N.stream_handle()), "delta")
        torch.cuda.synchronize()
        assert int(err[0]) == 0
        for j in range(4):
            got[j].append(o[at[j]:at[j + 1], :, :V])
    _portions(pieces, launch)

    def unit(t):
        return t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    for j, n in enumerate(lens):
        X, W, y = x[j].double(), cw.double(), torch.zeros(n, Cc, dtype=torch.float64, device=DEV)
        raw = torch.cat([X[:, off["q"]:off["q"] + HK * D], X[:, off["k"]:off["k"] + HK * D], X[:, off["v"]:off["v"] + H * V]], 1)
        for i in range(min(taps, n)):
            y[i:] += raw[:n - i] * W[:, taps - 1 - i]
        y = y * torch.sigmoid(y)
        q, k = (unit(y[:, i * HK * D:(i + 1) * HK * D].view(n, HK, D)).repeat_interleave(H // HK, 1) for i in range(2))
        v, beta = y[:, 2 * HK * D:].view(n, H, V), torch.sigmoid(X[:, off["b"]:off["b"] + H])
        dec = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(X[:, off["a"]:off["a"] + H] + dt.double()))
        S, want = torch.zeros(H, D, V, dtype=torch.float64, device=DEV), []
        for t in range(n):
            S = S * dec[t][:, None, None]
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None]
            want.append(torch.einsum("hdv,hd->hv", S, q[t] * D ** -0.5))
        _near(torch.cat(got[j]), torch.stack(want))
        _near(state[j + 1, :, :V, :D].transpose(1, 2), S)
    assert not state[0].any()


@pytest.mark.gpu
@pytest.mark.parametrize("pieces", PIECES)
@pytest.mark.parametrize("H,D,rank", [(5, 128, 96), (4, 64, 16), (3, 72, 256), (9, 20, 33)])
def test_channel_delta_rule(H, D, rank, pieces):
    lens = [sum(p[j] for p in pieces) for j in range(4)]
    DP, VP, g = (D + 63) // 64 * 64, (D + 7) // 8 * 8, torch.Generator(device=DEV).manual_seed(H + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)                  # noqa: E731
    off, ld = _offsets((("r", H * D), ("k", H * D), ("v", H * D), ("a", H * D), ("l", rank), ("g", H * D)))
    x, w2 = [rnd(n, ld) for n in lens], (rnd(H * D, rank) * rank ** -0.5).bfloat16()
    w0, nw = torch.rand(H * D, generator=g, device=DEV) * 6 - 5, torch.ones(H * D, device=DEV)
    w2_p = torch.zeros(H * D, (rank + 15) // 16 * 16, dtype=torch.bfloat16, device=DEV)
    w2_p[:, :rank] = w2
    state, err, got = _f32(5, H, VP, DP), _i32([0] * 4), [[] for _ in lens]

    def launch(piece, done):
        cu, slots, pos, at = _tables(piece, done)
        M = at[-1]
        xs, o, out = torch.cat([x[j][done[j]:done[j] + n] for j, n in enumerate(piece)]).contiguous(), _f32(M, H, VP), _f32(M, H * D)
        p = N.CdeltaParams()
        p.x, p.ldx = xs.data_ptr(), ld
        p.r_off, p.k_off, p.v_off, p.a_off, p.l_off, p.g_off = (off[z] for z in "rkvalg")
        p.w2, p.w2_f32, p.rank, p.w0, p.norm_w, p.state, p.o = w2_p.data_ptr(), 0, rank, w0.data_ptr(), nw.data_ptr(), state.data_ptr(), o.data_ptr()
        p.cu_rows, p.slots, p.pos, p.out, p.out_scale, p.err = cu.data_ptr(), slots.data_ptr(), pos.data_ptr(), N.Operand(out.data_ptr(), M, H * D, 1), 1.0, err.data_ptr()
        p.M, p.nseq, p.H, p.D, p.DP, p.VP, p.n_slots, p.eps, p.unit_eps = M, 4, H, D, DP, VP, 5, 1e-6, 1e-6
        floats = N.lib().saber_cdelta_chunk_floats(C.byref(p))
        assert floats > 0
        scratch = torch.full((floats,), float("nan"), device=DEV)
        p.chunk = scratch.data_ptr()
        N.check(N.lib().saber_cdelta_launch(C.byref(p), 0, N.stream_handle()), "cdelta")
        torch.cuda.synchronize()
        assert int(err[0]) == 0
        for j in range(4):
            got[j].append(o[at[j]:at[j + 1], :, :D])
    _portions(pieces, launch)
    for j, n in enumerate(lens):
        X = x[j].double()
        r, k, v, a = (X[:, off[z]:off[z] + H * D].view(n, H, D) for z in "rkva")
        low = torch.tanh(X[:, off["l"]:off["l"] + rank]) @ w2.double().T + w0.double()
        dec, u = torch.exp(-math.exp(-0.5) * torch.sigmoid(low)).view(n, H, D), k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S, want = torch.zeros(H, D, D, dtype=torch.float64, device=DEV), []
        for t in range(n):
            held = torch.einsum("hd,hdv->hv", u[t], S)
            S = dec[t][..., None] * S - (torch.sigmoid(a[t]) * u[t])[..., None] * held[:, None] + k[t][..., None] * v[t][:, None]
            want.append(torch.einsum("hdv,hd->hv", S, r[t]))
        _near(torch.cat(got[j]), torch.stack(want))
        _near(state[j + 1, :, :D, :D].transpose(1, 2), S)
    assert not state[0].any()
