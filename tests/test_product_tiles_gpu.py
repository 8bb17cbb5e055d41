"""The products over tiles whose height or list follows from the shape, at the edges of their tiles, against float64."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from math_utils_b200.csrc import ops
    return ops


def _rand(shape, seed, dtype=torch.float32, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(dtype)


# heights of 16 to 80 rows (several are taken between one tile and many waves of them), columns and k at and past the
# ends of a tile; a leading dimension that is longer than the row
@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (15, 64, 32), (17, 65, 36), (33, 130, 28), (49, 3000, 100), (81, 700, 260),
                                   (161, 2500, 64), (777, 768, 96), (1300, 1030, 40)])
def test_float32_tiles(m, n, k):
    """Four sums of k / 4 terms each, rounded term by term: within 1e-5 of the rms (a running sum of some 500 terms is)."""
    ops = _ops()
    a, w = _rand((m, k + 8), 1)[:, :k], _rand((n, k), 2, scale=k ** -0.5)
    bias, res = _rand((n,), 3), _rand((m, n), 4)
    want = torch.relu(a.double() @ w.double().T + bias.double()) ** 2 + res.double()
    x = res.clone()
    ops.linear(a, w, bias, act="relu2", residual=x, out=x)
    assert float((x.double() - want).abs().max() / want.square().mean().sqrt()) < 1e-5
    odd = torch.zeros((m, n + 3), device="cuda")                      # rows that are no whole 16-byte pieces
    ops.linear(a, w, None, out=odd[:, 1:n + 1])
    plain = a.double() @ w.double().T
    assert float((odd[:, 1:n + 1].double() - plain).abs().max() / plain.square().mean().sqrt().clamp_min(1e-30)) < 1e-5
    assert not odd[:, 0].any() and not odd[:, n + 1:].any()
    assert torch.equal(ops.linear(a[m // 2:m // 2 + 1], w, bias), ops.linear(a, w, bias)[m // 2:m // 2 + 1])


# a pair's tile of 256 rows: none, one and all of the second block's rows, one row more; columns at and past a tile's and a
# block's half; k of less than a stage, of a stage and more than the ring holds
@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (128, 130, 64), (129, 256, 72), (256, 97, 200), (257, 520, 1000), (700, 391, 520)])
@pytest.mark.parametrize("tile", [-128, -192, -256])
def test_products_by_pairs_of_sms(m, n, k, tile):
    """The one-SM product's bits: the same products in the same order.  Bulk stores, stores by row (rows that are no whole
    16-byte pieces), a residual in place and beside."""
    ops = _ops()
    dt = torch.bfloat16
    a, w, bias, res = _rand((m, k), 1, dt), _rand((n, k), 2, dt, k ** -0.5), _rand((n,), 3), _rand((m, n), 4)
    for kwargs in ({"act": "gelu_new"}, {"residual": res, "out_dtype": torch.float32, "act": "relu2"}):
        want, got = (ops.gemm_tc(a, w, bias, tile=t, splits=0, **kwargs) for t in (64, tile))
        assert torch.equal(got, want)
    plain = a.double() @ w.double().T + bias.double()
    x, odd = res.clone(), torch.zeros((m, n + 3), dtype=torch.float32, device="cuda")
    ops.gemm_tc(a, w, bias, residual=x, out=x, tile=tile)
    ops.gemm_tc(a, w, bias, out=odd[:, 1:n + 1], tile=tile)
    assert float((x.double() - plain - res.double()).abs().max()) < 1e-5 * max(1.0, float(plain.abs().max()))
    assert float((odd[:, 1:n + 1].double() - plain).abs().max()) < 1e-5 * max(1.0, float(plain.abs().max()))
    assert not odd[:, 0].any() and not odd[:, n + 1:].any()
    ops.check_status()


# one row, rows and columns at and past the ends of warps and tiles, k at the rule's line, past a step, at, past and far past a
# run of 768, more than eight runs' worth
@pytest.mark.parametrize("m,n,k", [(1, 1, 384), (33, 31, 388), (129, 161, 420), (300, 97, 768), (64, 65, 772), (200, 320, 2308), (40, 70, 6500)])
def test_float32_tensor_tiles(m, n, k):
    """Whole operands, sums in float32: within 1e-5 of the rms like the multiply-adds, and no further off in the 2-norm; the tile's
    width, the cut and the rows beside it change no bit."""
    ops = _ops()
    a, w = _rand((m, k + 4), 1)[:, :k], _rand((n, k), 2, scale=k ** -0.5)
    bias, res = _rand((n,), 3), _rand((m, n), 4)
    plain = a.double() @ w.double().T
    want = torch.relu(plain + bias.double()) ** 2 + res.double()
    x = res.clone()
    ops.linear(a, w, bias, act="relu2", residual=x, out=x)
    assert float((x.double() - want).abs().max() / want.square().mean().sqrt()) < 1e-5
    full = ops.linear(a, w)
    error, before = ((f.double() - plain).norm() for f in (full, ops.gemm_simt(a, w)))
    assert m * n < 100 or float(error) <= float(before)
    odd = torch.zeros((m, n + 3), device="cuda")
    ops.linear(a, w, out=odd[:, 1:n + 1])
    assert torch.equal(odd[:, 1:n + 1], full) and not odd[:, 0].any() and not odd[:, n + 1:].any()
    assert torch.equal(ops.linear(a[m // 2:m // 2 + 1], w), full[m // 2:m // 2 + 1])
    for tile in (32, 64, 96, 128, 160):
        for cut in (0, 1):
            assert torch.equal(ops.gemm_f32_tc(a, w, tile=tile, cut=cut), full), (tile, cut)
    ops.check_status()


def test_float32_tensor_products_that_are_exact():
    """What float32 holds comes out: products with an identity (of 24 bits, over magnitudes down to 1e-25), sums of whole numbers
    below 2^24, one product a row rounded once; whole and cut."""
    ops = _ops()
    eye, x = torch.eye(1600, device="cuda"), _rand((130, 1600), 1) * torch.exp(8 * _rand((130, 1600), 2))
    i = torch.randint(-100, 101, (70, 2048), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).float()
    j = torch.randint(-80, 81, (90, 2048), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)).float()
    for cut in (0, 1):
        assert torch.equal(ops.gemm_f32_tc(x, eye, cut=cut), x) and torch.equal(ops.gemm_f32_tc(eye, x, cut=cut), x.T)
        assert torch.equal(ops.gemm_f32_tc(i, j, cut=cut).double(), i.double() @ j.double().T)
    one = torch.zeros_like(x).scatter_(1, torch.arange(130, device="cuda")[:, None] * 12, x.gather(1, torch.arange(130, device="cuda")[:, None] * 12))
    w = _rand((64, 1600), 5)
    got, want = ops.gemm_f32_tc(one, w).double(), one.double() @ w.double().T
    # half a last bit, and the 2^-36 that is left out together with what the small products' sum is cut by (2^-24 of 2^-8)
    assert ((got - want).abs() <= want.abs() * (2.0 ** -24 + 2.0 ** -30)).all()
    ops.check_status()


# rows of few values, positive and of any sign, full rows, and full rows of wide magnitudes (0)
@pytest.mark.parametrize("k", [384, 768, 1024, 3072])
@pytest.mark.parametrize("values", [1, 4, 16, 64, 9999, 0])
def test_float32_tensor_products_against_multiply_adds(k, values):
    """No further from float64 than multiply-adds, output by output against the size of its terms (rms; half a percent for the
    luck of the draw, where both round once)."""
    ops = _ops()
    a, w = _rand((400, k), k), _rand((400, k), 2)
    if values:
        g = torch.Generator(device="cuda").manual_seed(k + values)
        a = a * (torch.rand((400, k), generator=g, device="cuda").argsort(1) < values)
    else:
        a, w = a * torch.exp(2 * _rand((400, k), 3)), w * torch.exp(2 * _rand((400, k), 4))
    for x, y in ((a, w), (a.abs(), w.abs()))[:2 if values else 1]:
        plain, size = x.double() @ y.double().T, x.abs().double() @ y.abs().double().T
        error, before = (float(((f(x, y).double() - plain) / size).square().mean()) ** 0.5 for f in (ops.gemm_f32_tc, ops.gemm_simt))
        assert error <= 1.005 * before, (error, before)


def test_float32_tensor_tiles_pass_on_what_is_not_finite():
    """An infinite, NaN or largest value gives what multiply-adds give, in whole and in cut products."""
    ops = _ops()
    a, w = _rand((150, 800), 1), _rand((70, 800), 2)
    a[3, 5], a[70, 100], a[149, 0], w[7, 3], w[9, 9] = float("inf"), float("nan"), 3.4e38, -float("inf"), 1e30
    a[90, 799], a[91, 798], a[91, 2] = float("nan"), -float("inf"), float("inf")           # (found at the end; two infinities)
    want = ops.gemm_simt(a, w)
    for cut in (0, 1):
        got = ops.gemm_f32_tc(a, w, cut=cut)
        known = torch.isfinite(want)
        assert torch.equal(torch.nan_to_num(got[~known], nan=7.0), torch.nan_to_num(want[~known], nan=7.0))
        assert torch.equal(torch.isfinite(got), known) and torch.allclose(got[known], want[known], rtol=1e-4, atol=1e-3)
    ops.check_status()


# tiles of 128 slots: an expert without rows, with one, with exactly a tile and one more; few and many experts; columns and
# k past a box; identity experts (no slots) and weights on the input
@pytest.mark.parametrize("form,experts,identity,top,tokens,D,F", [
    ("gated", 3, 0, 1, 1, 64, 64), ("gated", 5, 0, 2, 300, 200, 136), ("gated", 40, 0, 4, 70, 72, 264),
    ("relu2", 4, 0, 4, 128, 128, 128), ("relu2", 6, 3, 3, 129, 136, 72), ("relu2", 2, 0, 1, 700, 328, 520),
    ("relu2", 64, 8, 6, 8, 256, 704)])
def test_experts_over_tiles_of_128_slots(form, experts, identity, top, tokens, D, F):
    """bfloat16 operands, float32 sums: the float32 result within 1e-5 of its rms per term's root, the hidden rows within
    their rounding (2^-8 of a value, and as much of the rms for values near zero)."""
    ops = _ops()
    rng = np.random.default_rng(tokens)
    dt = torch.bfloat16
    h, gate, up = _rand((tokens, D), 1, dt), _rand((experts, F, D), 2, dt, D ** -0.5), _rand((experts, F, D), 3, dt, D ** -0.5)
    down = _rand((experts, D, F), 4, dt, F ** -0.5)
    chosen = np.stack([rng.permutation(experts + identity)[:top] for _ in range(tokens)]).astype(np.int32)
    if experts > 3:
        chosen[chosen == 1] = 0                                        # an expert that nobody chose
    P, rows = tokens * top, ops.MOE_TC_ROWS
    expert_of = torch.as_tensor(chosen.reshape(-1)).cuda()
    slot_of, pair_of = (torch.zeros(P, dtype=torch.int32, device="cuda") for _ in range(2))
    most = P // rows + experts
    info, n = torch.zeros(3 * most, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.moe_group(expert_of, experts + identity, slot_of, pair_of, info, n, rows, n_real=experts if identity else 0)
    xs = ops.moe_gather(h, slot_of, top, torch.zeros((P, D), dtype=dt, device="cuda"))
    hidden, y = torch.zeros((P, F), dtype=dt, device="cuda"), torch.zeros((P, D), device="cuda")
    weight = _rand((P,), 5).abs()
    if form == "gated":
        ops.moe_gemm(xs, pair_of, top, gate, up, info, n, most, hidden, tile_rows=rows, row_weight=weight)
    else:
        ops.moe_gemm(xs, pair_of, top, up, None, info, n, most, hidden, tile_rows=rows, act="relu2")
    ops.moe_gemm(hidden, None, top, down, None, info, n, most, y, tile_rows=rows)
    ops.check_status()
    slots = slot_of.cpu().numpy()
    assert sorted(s for s in slots if s >= 0) == list(range(int((chosen < experts).sum())))
    for p in range(P):
        e = int(chosen.reshape(-1)[p])
        if e >= experts:
            assert slots[p] == -1
    real = torch.as_tensor(np.nonzero(slots >= 0)[0]).cuda()
    at, e = slot_of[real].long(), expert_of[real].long()
    x = h[real // top].double()
    z = torch.einsum("pd,pfd->pf", x, up.double()[e])
    if form == "gated":
        z, g = z * weight[real].double()[:, None], torch.einsum("pd,pfd->pf", x, gate.double()[e]) * weight[real].double()[:, None]
        want = g * torch.sigmoid(g) * z
    else:
        want = torch.relu(z) ** 2
    got = hidden[at].double()
    rms = want.square().mean().sqrt()
    assert float(((got - want).abs() / (want.abs() + rms)).max()) < 2.0 ** -8
    want = torch.einsum("pf,pdf->pd", got, down.double()[e])
    assert float((y[at].double() - want).abs().max() / want.square().mean().sqrt()) < 1e-5 * max(1.0, math.sqrt(F / 512))


# more rows than the small kernel takes, a row past a tile, output columns past a tile, slices with gaps between them
@pytest.mark.parametrize("rows,heads,n,k,lead", [(65, 3, 128, 64, 32), (129, 2, 40, 128, 0), (300, 5, 264, 64, 8), (128, 1, 512, 192, 0)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_products_per_head_on_tcgen05(rows, heads, n, k, lead, out_dtype, monkeypatch):
    ops = _ops()
    monkeypatch.setattr(ops, "HEADS_TC_FLOP", 0.0)
    xs, os_ = k + lead, n + 8
    x, w = _rand((rows, heads * xs), 1, torch.bfloat16), _rand((heads, n, k), 2, torch.bfloat16, k ** -0.5)
    gate = _rand((rows, heads * os_), 3, torch.bfloat16)
    for g in (None, gate):
        out = torch.zeros((rows, heads * os_), device="cuda", dtype=out_dtype)
        ops.heads_gemm(x, w, out, xs, os_, gate=g)
        ops.check_status()
        want = torch.einsum("thk,hnk->thn", x.double().reshape(rows, heads, xs)[:, :, :k], w.double())
        if g is not None:
            want = want * torch.sigmoid(g.double().reshape(rows, heads, os_)[:, :, :n])
        got = out.reshape(rows, heads, os_)
        if g is None:
            assert not got[:, :, n:].any()                             # nothing written between the slices
        bound = 1e-5 if out_dtype == torch.float32 else 2.0 ** -8
        assert float(((got[:, :, :n].double() - want).abs() / (want.abs() + want.square().mean().sqrt())).max()) < bound


# one stage of 128 and half of the next (k past a whole number of 128), columns of one box and less
@pytest.mark.parametrize("n,k,lead", [(128, 64, 32), (40, 192, 0), (128, 320, 64), (264, 64, 8)])
def test_products_per_head_see_their_own_slice_alone(n, k, lead, monkeypatch):
    """Whatever lies between the slices or in another head's: the same bits as with zeros there."""
    ops = _ops()
    monkeypatch.setattr(ops, "HEADS_TC_FLOP", 0.0)
    rows, heads, xs = 130, 3, k + lead
    x, w = _rand((rows, heads * xs), 1, torch.bfloat16), _rand((heads, n, k), 2, torch.bfloat16, k ** -0.5)
    slices = x.reshape(rows, heads, xs)
    slices[:, :, k:] = 0.0
    outs = []
    for _ in range(2):
        out = torch.zeros((rows, heads * n), device="cuda")
        ops.heads_gemm(x, w, out, xs, n)
        ops.check_status()
        outs.append(out.reshape(rows, heads, n))
        slices[:, :, k:] = float("nan")
        slices[:, 1] = float("inf")
    assert torch.equal(outs[0][:, 0], outs[1][:, 0]) and torch.equal(outs[0][:, 2], outs[1][:, 2])


def test_products_per_head_of_rows_that_overlap(monkeypatch):
    """One row for all (a stride of zero), and rows that begin inside the row before: the kernel without tensor maps takes them."""
    ops = _ops()
    monkeypatch.setattr(ops, "HEADS_TC_FLOP", 0.0)
    heads, n, k = 2, 64, 64
    w, flat = _rand((heads, n, k), 2, torch.bfloat16, k ** -0.5), _rand((130 * 64 + heads * k,), 1, torch.bfloat16)
    for x in (flat[:heads * k].expand(130, heads * k), flat.as_strided((130, heads * k), (64, 1))):
        out = torch.zeros((130, heads * n), device="cuda")
        ops.heads_gemm(x, w, out, k, n)
        want = torch.einsum("thk,hnk->thn", x.double().reshape(130, heads, k), w.double()).reshape(130, -1)
        assert float((out.double() - want).abs().max() / want.square().mean().sqrt()) < 1e-4


# one block of 128 threads, of 1024, pairs beyond those it keeps in registers; identity experts; more experts than a warp
@pytest.mark.parametrize("P,experts,real", [(1, 4, 4), (48, 72, 64), (256, 33, 33), (257, 5, 4), (12288, 64, 64), (20001, 70, 64)])
@pytest.mark.parametrize("rows", [32, 128])
def test_grouping_of_pairs(P, experts, real, rows):
    """Every pair of a real expert has a slot of its own among its expert's, which lie together; the tiles cover them."""
    ops = _ops()
    rng = np.random.default_rng(P)
    expert = rng.integers(0, experts, P).astype(np.int32)
    expert[expert == 1] = 0
    slot, pair = (torch.full((P,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    most = P // rows + experts
    info, n = torch.full((3 * most,), -7, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.moe_group(torch.as_tensor(expert).cuda(), experts, slot, pair, info, n, rows, n_real=real)
    slot, pair, info, n = slot.cpu().numpy(), pair.cpu().numpy(), info.cpu().numpy().reshape(-1, 3), int(n)
    chosen = np.nonzero(expert < real)[0]
    assert (slot[expert >= real] == -1).all()
    assert sorted(slot[chosen]) == list(range(len(chosen))) and (pair[slot[chosen]] == chosen).all()
    by_slot = expert[pair[:len(chosen)]]
    assert (np.diff(by_slot) >= 0).all()
    want = [(e, a + i, min(rows, c - i)) for e in range(real) for a, c in [(int((expert[chosen] < e).sum()), int((expert == e).sum()))]
            for i in range(0, c, rows)]
    assert n == len(want) and [tuple(t) for t in info[:n]] == want


# seven, eight (1,100 are two rounds of seven), four and two tokens a block (what the staged rows leave room for), a block's tokens
# cut off, an odd number of rows
@pytest.mark.parametrize("tokens,hidden,experts,gate", [(601, 256, 64, True), (1100, 260, 65, True), (700, 2048, 17, False), (650, 4096, 16, True),
                                                        (593, 6200, 5, True), (600, 8200, 5, True), (595, 12776, 9, False)])
def test_router_of_several_tokens_a_block(tokens, hidden, experts, gate):
    """Each logit a float32 sum of `hidden` terms in 128 parts: scores within 1e-5; and the bits that a token alone gives."""
    ops = _ops()
    h = _rand((tokens, hidden), 1, torch.bfloat16)
    router, g = _rand((experts, hidden), 2, scale=hidden ** -0.5), _rand((hidden,), 3, scale=hidden ** -0.5) if gate else None
    top = 3

    def route(x):
        expert = torch.zeros(x.shape[0] * top, dtype=torch.int32, device="cuda")
        weight, out = torch.zeros(x.shape[0] * top, device="cuda"), torch.zeros(x.shape[0], device="cuda") if gate else None
        ops.moe_route(x, router, None, top, 1.0, expert, weight, gate_weight=g, gate_out=out)
        return expert.reshape(-1, top), weight.reshape(-1, top), out

    expert, weight, out = route(h)
    s = torch.sigmoid(h.double() @ router.double().T)
    assert float((weight.double() - torch.gather(s, 1, expert.long())).abs().max()) < 1e-5
    assert float((s.sort(dim=1, descending=True)[0][:, :top] - weight.double()).abs().max()) < 1e-5
    if gate:
        assert float((out.double() - torch.sigmoid(h.double() @ g.double())).abs().max()) < 1e-5
    for t in (0, 7, tokens - 1) if hidden < 12000 else ():               # (a token alone has less room)
        e1, w1, g1 = route(h[t:t + 1])
        assert torch.equal(e1[0], expert[t]) and torch.equal(w1[0], weight[t]) and (not gate or torch.equal(g1[0], out[t]))


# clusters of eight blocks, of four and single blocks a token at their lines (half the SMs, all of them); lanes with a piece more
@pytest.mark.parametrize("tokens", [1, 74, 75, 148, 149])
def test_router_of_few_tokens_by_clusters(tokens):
    """The bits of the form for many tokens."""
    ops = _ops()
    h, router = _rand((600, 520), 1, torch.bfloat16), _rand((70, 520), 2, scale=520 ** -0.5)

    def route(x):
        expert, weight = torch.zeros(x.shape[0] * 4, dtype=torch.int32, device="cuda"), torch.zeros(x.shape[0] * 4, device="cuda")
        ops.moe_route(x, router, None, 4, 1.0, expert, weight)
        return expert, weight

    assert all(torch.equal(few, many[:tokens * 4]) for few, many in zip(route(h[:tokens]), route(h)))


# the widest rows: one token's 12,288 values with the scores of its experts twice, two of many tokens 25,600; rows that end off a
# 16-byte boundary
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,experts,hidden", [(1, 7, 12274), (20, 24, 12240), (592, 7, 12786), (592, 24, 12752)])
def test_router_takes_the_widths_it_took(tokens, experts, hidden, dtype):
    ops = _ops()

    def route(width):
        h, router = _rand((tokens, width), 1, dtype), _rand((experts, width), 2, scale=width ** -0.5)
        expert, weight = torch.zeros(tokens * 2, dtype=torch.int32, device="cuda"), torch.zeros(tokens * 2, device="cuda")
        ops.moe_route(h, router, None, 2, 1.0, expert, weight)
        top = torch.topk(h.double() @ router.double().T, 2)
        # (float32 logits: a pair closer than their error may fall either way)
        sure = (top.values[:, 0] - top.values[:, 1]) > 1e-3
        assert torch.equal(expert.view(tokens, 2)[sure, 0].long(), top.indices[sure, 0])

    route(hidden)
    with pytest.raises(ops.KernelError):
        route(hidden + 2)
