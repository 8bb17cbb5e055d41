"""The recurrences taken chunk by chunk against float64 and against their token-by-token kernels, at the edges of the chunks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = [(64,), (1, 130), (63, 65, 200), (700,), (129, 2, 64, 31)]


def _ops():
    from math_utils_b200.csrc import ops
    return ops


def _ints(x):
    return torch.as_tensor(np.asarray(x, dtype=np.int32)).cuda()


def _step(lens):
    first = np.concatenate([[0], np.cumsum(lens)])
    tiles = [(first[s] + o, min(64, n - o)) for s, n in enumerate(lens) for o in range(0, n, 64)]
    return _ints(tiles[::-1]), _ints(np.repeat(np.arange(len(lens)), lens)), _ints(first), first


def _rand(shape, seed, scale=1.0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


def _no_further_off(chunks, token_by_token, want, heads=1):
    """Operands at 22 bits, sums of some hundred float32 terms in runs of sixteen: a term is off by some 2^-22 of itself, a sum
    by a few 2^-24.  In norm held to four of those (2.5e-7; measured up to 2.1e-7, token by token up to 1.7e-7) or to
    one and a half times what the token-by-token kernel shows; every row of a head to 1e-6 of its own size and the rows'."""
    assert _rel(chunks, want) < max(2.5e-7, 1.5 * _rel(token_by_token, want))
    rows = lambda x: x.double().reshape(-1, x.shape[-1] // heads)
    size = rows(want).norm(dim=1)
    assert float(((rows(chunks) - rows(want)).norm(dim=1) / (size + size.square().mean().sqrt())).max()) < 1e-6


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,dk,dv,norm", [(2, 128, 128, True), (3, 16, 4, True), (1, 48, 100, False), (2, 96, 200, True)])
def test_linear_scan_in_chunks(lens, H, dk, dv, norm):
    ops = _ops()
    tiles, tok_seq, seq_first, first = _step(lens)
    T, slots = sum(lens), list(range(len(lens)))[::-1]
    u = _rand((T, H * (2 * dk + dv) + 4), 1)
    q, k, v = u[:, :H * dk], u[:, H * dk:2 * H * dk], u[:, 2 * H * dk:2 * H * dk + H * dv]
    decay = torch.rand((T, H), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    decay = 1.0 - 0.1 * decay ** 3                               # memories of ten tokens to thousands
    decay[T // 2] = 0.0                                          # all that was is forgotten
    gates = torch.zeros((T, H, 4), device="cuda")
    gates[..., 0], gates[..., 1] = decay, _rand((T, H), 3).abs()
    values = H * dk * (dv + (1 if norm else 0))
    start = _rand((len(lens), values + -values % 4), 4, 0.3)
    scale = dk ** -0.5
    got = {}
    for name in ("chunks", "tokens"):
        state, out = start.clone(), torch.zeros((T, H * dv), device="cuda")
        read = torch.zeros((T, H), device="cuda") if norm else None
        if name == "chunks":
            ops.linear_scan_chunks(q, k, v, gates, H, dk, dv, scale, tiles, tok_seq, seq_first, _ints(slots), state, 0, out, read)
        else:
            ops.linear_scan(q, k, v, gates, H, dk, dv, scale, seq_first, _ints(slots), state, 0, out, norm_out=read)
        got[name] = (out, state[:, :values], read)
    want_out = torch.zeros((T, H, dv + 1), dtype=torch.float64, device="cuda")
    want_state = start[:, :values].double().clone()
    for s, slot in enumerate(slots):
        held = start[slot, :values].double()
        S = held[:H * dk * dv].reshape(H, dv, dk)
        n = held[H * dk * dv:].reshape(H, 1, dk) if norm else torch.zeros((H, 1, dk), dtype=torch.float64, device="cuda")
        S = torch.cat([S, n], 1)
        for t in range(first[s], first[s + 1]):
            vt = torch.cat([v[t].double().reshape(H, dv), torch.ones((H, 1), dtype=torch.float64, device="cuda")], 1)
            S = S * gates[t, :, 0].double()[:, None, None] + (gates[t, :, 1].double()[:, None] * vt)[:, :, None] * k[t].double().reshape(H, 1, dk)
            want_out[t] = scale * torch.einsum("hvd,hd->hv", S, q[t].double().reshape(H, dk))
        want_state[slot] = torch.cat([S[:, :dv].reshape(-1)] + ([S[:, dv].reshape(-1)] if norm else []))
    _no_further_off(got["chunks"][0], got["tokens"][0], want_out[..., :dv].reshape(T, H * dv), H)
    _no_further_off(got["chunks"][1], got["tokens"][1], want_state)
    if norm:
        _no_further_off(got["chunks"][2], got["tokens"][2], want_out[..., dv])


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,P,N,G,dtype", [(4, 64, 128, 1, torch.bfloat16), (2, 4, 16, 2, torch.float32), (6, 100, 48, 2, torch.bfloat16)])
def test_state_space_scan_in_chunks(lens, H, P, N, G, dtype):
    ops = _ops()
    tiles, tok_seq, seq_first, first = _step(lens)
    T, slots, inner = sum(lens), list(range(len(lens)))[::-1], H * P
    xbc = _rand((T, inner + 2 * G * N), 1)
    dt_raw = _rand((T, H + 3), 2).to(dtype)[:, :H]
    dt_bias, skip = _rand((H,), 3) - 3.0, _rand((H,), 4)
    a_log = torch.log(1.0 + 7.0 * torch.rand((H,), generator=torch.Generator(device="cuda").manual_seed(5), device="cuda"))
    offset = 8
    start = _rand((len(lens), offset + H * N * P), 6, 0.3)
    got = {}
    for name in ("chunks", "tokens"):
        state, y = start.clone(), torch.zeros((T, inner), device="cuda")
        if name == "chunks":
            ops.ssd_scan_chunks(xbc, dt_raw, dt_bias, a_log, skip, H, P, N, G, tiles, tok_seq, seq_first, _ints(slots), state, offset, y)
        else:
            ops.ssd_scan(xbc, dt_raw, dt_bias, a_log, skip, H, P, N, G, seq_first, _ints(slots), state, offset, y)
        got[name] = (y, state)
    want_state, want = start.double().clone(), torch.zeros((T, inner), dtype=torch.float64, device="cuda")
    dt = torch.nn.functional.softplus(dt_raw.double() + dt_bias.double(), threshold=200.0)
    decay = torch.exp(-torch.exp(a_log.double()) * dt)
    x = xbc.double()
    for s, slot in enumerate(slots):
        S = start[slot, offset:].double().reshape(H, N, P)
        for t in range(first[s], first[s + 1]):
            B, C = (x[t, a:a + G * N].reshape(G, N).repeat_interleave(H // G, 0) for a in (inner, inner + G * N))
            xt = x[t, :inner].reshape(H, P)
            S = S * decay[t][:, None, None] + (dt[t][:, None] * B)[:, :, None] * xt[:, None, :]
            want[t] = (torch.einsum("hnp,hn->hp", S, C) + skip.double()[:, None] * xt).reshape(-1)
        want_state[slot, offset:] = S.reshape(-1)
    _no_further_off(got["chunks"][0], got["tokens"][0], want, H)
    _no_further_off(got["chunks"][1], got["tokens"][1], want_state)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("at", [0, 7, 40, 63, 64, 149])
@pytest.mark.parametrize("by_key", [False, True])
def test_chunks_keep_values_that_are_not_finite_from_tokens_before_them(by_key, at, bad):
    """One value entry of one token against the same step with a finite one: tokens before it, other entries and other heads
    differ by the order of their sums alone (float32 sums of some hundred terms, by 2^-24 each)."""
    ops = _ops()
    lens, H, dk, dv = (130, 150), 2, 32, 40
    tiles, tok_seq, seq_first, first = _step(lens)
    T, slots, at, col = sum(lens), [0, 1], int(first[1]) + at, 35
    u = _rand((T, H * (dv + 2 * dk)), 1)
    gates, outs = torch.rand((T, H, 4), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda"), []
    for _ in range(2):
        state, out = torch.zeros((2, H * dk * (dv + 1)), device="cuda"), torch.zeros((T, H * dv), device="cuda")
        if by_key:
            ops.ssd_scan_chunks(u, gates[..., 0].contiguous(), gates[0, :, 1].contiguous(), gates[0, :, 2].contiguous(),
                                gates[0, :, 3].contiguous(), H, dv, dk, H, tiles, tok_seq, seq_first, _ints(slots), state, 0, out)
        else:
            v, q, k = u[:, :H * dv], u[:, H * dv:H * (dv + dk)], u[:, H * (dv + dk):]
            ops.linear_scan_chunks(q, k, v, gates, H, dk, dv, 1.0, tiles, tok_seq, seq_first, _ints(slots), state, 0, out)
        outs.append(out)
        u[at, col] = bad
    hit = torch.zeros((T, H * dv), dtype=torch.bool, device="cuda")
    hit[at:, col] = True
    assert not outs[1][hit].isfinite().any() and torch.isfinite(outs[1][~hit]).all()
    assert float((outs[1] - outs[0])[~hit].abs().max() / outs[0].square().mean().sqrt()) < 1e-5


@pytest.mark.parametrize("lens", [(800,), (1025, 1), (1000, 255, 3), (40, 1281)])
@pytest.mark.parametrize("C,N,dtype", [(40, 16, torch.bfloat16), (17, 5, torch.float32), (24, 40, torch.float32), (16, 130, torch.bfloat16)])
def test_selective_scan_in_segments(lens, C, N, dtype):
    """Segments put together against the whole sequences' scan: the same sums but for the starting states of segments, which
    a product of 256 decays reaches in one exponential, off by 2^-22 of its argument's size."""
    ops = _ops()
    T, slots = sum(lens), list(range(len(lens)))[::-1]
    first = _ints(np.concatenate([[0], np.cumsum(lens)]))
    x, z = _rand((T, C), 1).to(dtype), _rand((T, C), 2).to(dtype)
    dt = torch.nn.functional.softplus(_rand((T, C), 3) - 3.0)
    n4 = -(-N // 4) * 4
    bc = _rand((T, 2 * n4), 4)
    bc[:, N:n4] = bc[:, n4 + N:] = 0        # as the product leaves the columns that only pad a row
    rates = -torch.exp(_rand((C, N), 5)).contiguous() * 1.4427
    skip = _rand((C,), 6)
    values = 6 + C * N
    start = _rand((len(lens), values + -values % 4), 7)
    got = []
    for most in (0, max(lens)):
        state, out = start.clone(), torch.zeros((T, C), dtype=dtype, device="cuda")
        ops.selective_scan(x, z, dt, bc, 0, n4, rates, skip, first, _ints(slots), state, 6, out, max_len=most)
        got.append((out, state))
    assert torch.equal(got[0][1][:, :6], start[:, :6]) and torch.equal(got[1][1][:, :6], start[:, :6])
    assert _rel(got[1][1], got[0][1].double()) < 2e-6
    assert _rel(got[1][0], got[0][0].double()) < (2e-6 if dtype == torch.float32 else 2e-3)
    worst = (got[1][0].double() - got[0][0].double()).abs() / (got[0][0].double().abs() + got[0][0].double().square().mean().sqrt())
    assert float(worst.max()) < (1e-5 if dtype == torch.float32 else 2.0 ** -7)


@pytest.mark.parametrize("lens", [(5,), (16, 7), (35, 2, 49), (150,)])
@pytest.mark.parametrize("H,G,dk,dv", [(2, 1, 128, 20), (2, 2, 20, 132), (4, 2, 64, 16), (1, 1, 256, 12),
                                       (8, 4, 128, 132)])        # one column a lane, two, and single tokens as the sequences grow
def test_delta_scan_in_blocks_of_four(lens, H, G, dk, dv):
    """Blocks of four tokens and what is left of a step against float64; the steps of one token show what float32 gives."""
    ops = _ops()
    T, slots = sum(lens), list(range(len(lens)))[::-1]
    first = np.concatenate([[0], np.cumsum(lens)])
    q, k = (torch.nn.functional.normalize(_rand((T, G, dk), s), dim=-1) for s in (1, 2))
    q = q * dk ** -0.5
    v = _rand((T, H * dv), 3)
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v], 1).contiguous()
    kq = (q.double() * k.double()).sum(-1).float().contiguous()
    beta, decay = torch.sigmoid(_rand((T, H), 4)), 1.0 - 0.2 * torch.sigmoid(_rand((T, H), 5)) ** 2
    decay[T // 2] = 0.0                                          # all that was is forgotten
    start = _rand((len(lens), 4 + H * dv * dk), 6, 0.3)
    block_out, block_state = torch.zeros((T, H * dv), device="cuda"), start.clone()
    ops.delta_scan(qkv, kq, beta, decay, H, G, dk, dv, _ints(first), _ints(slots), block_state, 4, block_out)
    token_out, token_state = torch.zeros((T, H * dv), device="cuda"), start.clone()
    want, want_state = torch.zeros((T, H * dv), dtype=torch.float64, device="cuda"), start.double()
    for s, slot in enumerate(slots):
        S = start[slot, 4:].double().reshape(H, dv, dk)
        for t in range(first[s], first[s + 1]):
            row = slice(t, t + 1)
            ops.delta_scan(qkv[row], kq[row], beta[row], decay[row], H, G, dk, dv, _ints([0, 1]), _ints([slot]), token_state, 4,
                           token_out[row])
            kt, qt = (x[t].double().repeat_interleave(H // G, 0) for x in (k, q))
            S = S * decay[t].double()[:, None, None]
            u = beta[t].double()[:, None] * (v[t].double().reshape(H, dv) - torch.einsum("hvd,hd->hv", S, kt))
            S = S + u[:, :, None] * kt[:, None, :]
            want[t] = torch.einsum("hvd,hd->hv", S, qt).reshape(-1)
        want_state[slot, 4:] = S.reshape(-1)
    _no_further_off(block_out, token_out, want, H)
    _no_further_off(block_state, token_state, want_state)
