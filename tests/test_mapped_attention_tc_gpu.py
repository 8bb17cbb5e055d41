"""Prompt attention with score maps on tcgen05 against float64: tiles of 128 queries whose last is short, steps that bring only
a sequence's last tokens, edges of windows, chunks and kept positions, every option of the kernel."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENS, NEW = [130, 1, 64, 129, 7, 500, 257], [130, 1, 64, 3, 7, 270, 257]


def _rand(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale).to(torch.bfloat16)


def _ints(x):
    return torch.as_tensor(np.asarray(x, dtype=np.int32)).cuda()


def _case(H, G, maps, dim, vdim, window=0, chunk=0, keep=0, shared=False, softcap=0.0, sink=False, slopes=False, gate=None,
          head_scale=False, head_sink=False, unit=False):
    return locals()


CASES = [
    _case(2, 1, 2, 64, 128, window=100, unit=True),
    _case(3, 3, 2, 16, 48, unit=True, window=300),
    _case(2, 2, 2, 128, 128),                                   # 256 key entries a head: two stages of pages
    _case(4, 2, 1, 128, 128, sink=True, gate="head", head_scale=True),
    _case(2, 2, 1, 192, 128, head_sink=True),
    _case(4, 1, 1, 16, 16, window=7),
    _case(2, 1, 1, 96, 96, chunk=64, gate="head"),
    _case(2, 1, 1, 80, 112, chunk=150, sink=True),
    _case(2, 2, 1, 64, 64, window=70, keep=5, slopes=True),
    _case(3, 1, 1, 32, 80, window=90, keep=130, slopes=True),
    _case(2, 1, 1, 48, 64, window=130, softcap=3.0, gate="entry"),
    _case(4, 2, 1, 64, 64, chunk=100, shared=True, sink=True),
    _case(1, 1, 1, 128, 128, shared=True),
]


@pytest.mark.parametrize("c", CASES, ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items() if v))
def test_mapped_attention_on_tcgen05(c):
    """The result is rounded to bfloat16 (2^-9 of a value); weights act with 16 bits, scores are float32 sums of bfloat16
    products, and the fast exponential is off by 2^-22 of its argument's size: 2^-8 of a value plus 2^-9 of the row's rms."""
    from math_utils_b200.csrc import ops
    H, G, maps, dim, vdim, shared = (c[k] for k in ("H", "G", "maps", "dim", "vdim", "shared"))
    scale, lam, out_scale, eps = 2.0 * dim ** -0.5, 0.45 if maps == 2 else 0.0, 0.8, 1e-3
    width = G * (maps * dim + (0 if shared else vdim))
    n_pages = [-(-n // 64) for n in LENS]
    order = np.random.default_rng(1).permutation(sum(n_pages) + 2)
    table, at = np.zeros((len(LENS), max(n_pages)), dtype=np.int32), 0
    for s, n in enumerate(n_pages):
        table[s, :n] = order[at:at + n]
        at += n
    rows = _rand((sum(n_pages) + 2, 64, width), 2)
    tok_seq = np.repeat(np.arange(len(LENS)), NEW)
    tok_pos = np.concatenate([np.arange(n - k, n) for n, k in zip(LENS, NEW)])
    T, tiles, at = len(tok_seq), [], 0
    for k in NEW:
        tiles += [(at + o, min(128, k - o)) for o in range(0, k, 128)]
        at += k
    padded = _rand((T, H * maps * dim + 8), 3)
    q = padded[:, :H * maps * dim]
    heads = torch.arange(H, device="cuda")
    slopes = 2.0 ** (-8.0 * (heads + 1).float() / H) if c["slopes"] else None
    head_scale = 0.5 + heads.float() / H if c["head_scale"] else None
    head_sink = heads.float() - 0.5 if c["head_sink"] else None
    gate = _rand((T, H * (vdim if c["gate"] == "entry" else 1)), 4) if c["gate"] else None
    out = torch.zeros((T, H * vdim), device="cuda", dtype=torch.bfloat16)
    assert ops.mapped_tc_ok(q, out, G, maps, dim, vdim, 64, shared)
    ops.mapped_attention(q, rows, _ints(table), 64, _ints(tok_pos), _ints(tok_seq), H, G, maps, dim, vdim, scale, c["window"], out,
                         lam=lam, out_scale=out_scale, eps=eps, unit_rms=c["unit"], chunk=c["chunk"], keep=c["keep"],
                         slopes=slopes, softcap=c["softcap"], sink=c["sink"], shared=shared, gate=gate, head_scale=head_scale,
                         head_sink=head_sink, tiles_wide=_ints(tiles))
    ops.check_status()
    want = torch.zeros((T, H, vdim), dtype=torch.float64, device="cuda")
    for s, (n, k) in enumerate(zip(LENS, NEW)):
        held = rows[torch.as_tensor(table[s, :n_pages[s]].astype(np.int64)).cuda()].double().reshape(-1, width)[:n]
        mine = torch.as_tensor(np.nonzero(tok_seq == s)[0]).cuda()
        keys = held[:, :G * maps * dim].reshape(n, G, maps, dim).repeat_interleave(H // G, 1)
        values = (keys[:, :, 0] if shared else held[:, G * maps * dim:].reshape(n, G, vdim).repeat_interleave(H // G, 1))
        p = torch.arange(n - k, n, device="cuda")[:, None]
        j = torch.arange(n, device="cuda")[None, :]
        lo = p - p % c["chunk"] if c["chunk"] else p - c["window"] + 1 if c["window"] else 0 * p
        seen = (j <= p) & ((j >= lo) | (j < c["keep"]))
        parts = []
        for m in range(maps):
            x = torch.einsum("ihd,jhd->hij", q[mine].double().reshape(k, H, maps, dim)[:, :, m], keys[:, :, m]) * scale
            if head_scale is not None:
                x = x * head_scale.double()[:, None, None]
            if c["softcap"]:
                x = c["softcap"] * torch.tanh(x / c["softcap"])
            if slopes is not None:
                x = x - slopes.double()[:, None, None] * (p - j)
            x = x.masked_fill(~seen, -math.inf)
            extra = torch.zeros(H, dtype=torch.float64, device="cuda") if c["sink"] else head_sink.double() if c["head_sink"] else None
            if extra is not None:
                x = torch.cat([x, extra[:, None, None].expand(H, k, 1)], -1)
            parts.append(torch.einsum("hij,jhd->ihd", torch.softmax(x, -1)[..., :n], values))
        o = parts[0] - (lam * parts[1] if maps == 2 else 0.0)
        if c["unit"]:
            o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)
        o = o * out_scale
        if gate is not None:
            o = o * torch.sigmoid(gate[mine].double()).reshape(k, H, -1)
        want[mine] = o
    err = (out.double().reshape(T, H, vdim) - want).abs()
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -9 * want.square().mean(-1, keepdim=True).sqrt() + 1e-6
    worst = (err / bound).amax((1, 2))
    bad = int(worst.argmax())
    assert float(worst[bad]) < 1.0, f"{float(worst[bad]):.2f} of the bound at token {bad} (sequence {tok_seq[bad]}, position {tok_pos[bad]})"


# (sequences, tokens each): as many wide tiles as SMs, one sequence more, and as many of more than 64 tokens
@pytest.mark.parametrize("seqs,n,wide", [(18, 17, True), (19, 17, False), (19, 65, True), (64, 64, False)])
def test_short_sequences_keep_tiles_of_64(seqs, n, wide, monkeypatch):
    """Which kernel a step of 8 heads takes on 148 SMs, by its launch; results as from the other, each rounded once."""
    from math_utils_b200.csrc import ops
    H, G, dim = 8, 2, 64
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    took, check = [], ops._check
    monkeypatch.setattr(ops, "_check", lambda code, what, *a, **k: (took.append(str(what)), check(code, what, *a, **k))[1])
    pages = -(-n // 64)
    rows, q = _rand((seqs * pages, 64, 2 * G * dim), 1), _rand((seqs * n, H * dim), 2)
    table = _ints(np.arange(seqs * pages).reshape(seqs, pages))
    tiles = {w: _ints([(s * n + o, min(w, n - o)) for s in range(seqs) for o in range(0, n, w)]) for w in (64, 128)}
    pos, seq, outs = _ints(np.tile(np.arange(n), seqs)), _ints(np.repeat(np.arange(seqs), n)), []
    for given in ({"tiles": tiles[64], "tiles_wide": tiles[128]}, {"tiles_wide" if not wide else "tiles": tiles[128 if not wide else 64]}):
        out = torch.zeros((seqs * n, H * dim), device="cuda", dtype=torch.bfloat16)
        ops.mapped_attention(q, rows, table, 64, pos, seq, H, G, 1, dim, dim, dim ** -0.5, 0, out, **given)
        outs.append(out.double())
    ops.check_status()
    assert ["attention_tc" in t for t in took] == [wide, not wide]
    bound = 2.0 ** -7 * outs[1].abs() + 2.0 ** -8 * outs[1].square().mean(1, keepdim=True).sqrt() + 1e-6
    assert float(((outs[0] - outs[1]).abs() / bound).max()) < 1.0


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("c", [CASES[i] for i in (0, 1, 3, 8, 9, 10, 11)], ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items() if v))
def test_values_that_are_not_finite_stay_with_the_queries_that_see_them(c, bad):
    """One position's values, and whatever the last page holds behind the sequence's end, against the same rows with finite
    values there: queries that do not see the position differ by no more than two results that are each rounded once."""
    from math_utils_b200.csrc import ops
    H, G, maps, dim, vdim, shared = (c[k] for k in ("H", "G", "maps", "dim", "vdim", "shared"))
    n, new, at = 410, 405, 171                                     # the tiles begin inside a page
    width, n_pages = G * (maps * dim + (0 if shared else vdim)), -(-n // 64)
    table, rows = _ints([list(range(n_pages))[::-1]]), _rand((n_pages, 64, width), 2)
    q = _rand((new, H * maps * dim), 3)
    gate = _rand((new, H * (vdim if c["gate"] == "entry" else 1)), 4) if c["gate"] else None
    slopes = 2.0 ** (-8.0 * (torch.arange(H, device="cuda") + 1).float() / H) if c["slopes"] else None
    tiles, outs = _ints([(o, min(128, new - o)) for o in range(0, new, 128)]), []
    for _ in range(2):
        out = torch.zeros((new, H * vdim), device="cuda", dtype=torch.bfloat16)
        ops.mapped_attention(q, rows, table, 64, _ints(range(n - new, n)), _ints([0] * new), H, G, maps, dim, vdim, dim ** -0.5,
                             c["window"], out, lam=0.45 if maps == 2 else 0.0, out_scale=0.8, eps=1e-3, unit_rms=c["unit"],
                             chunk=c["chunk"], keep=c["keep"], slopes=slopes, softcap=c["softcap"], sink=c["sink"], shared=shared,
                             gate=gate, tiles_wide=tiles)
        ops.check_status()
        outs.append(out.double())
        rows[n_pages - 1 - at // 64, at % 64, 0 if shared else G * maps * dim:] = bad
        rows[0, n % 64:] = bad
    p = torch.arange(n - new, n, device="cuda")
    lo = p - p % c["chunk"] if c["chunk"] else p - c["window"] + 1 if c["window"] else 0 * p
    sees = (at <= p) & ((at >= lo) | (at < c["keep"]))
    assert sees.any() and not outs[1][sees].isfinite().all(1).any()
    want, got = outs[0][~sees], outs[1][~sees]
    bound = 2.0 ** -7 * want.abs() + 2.0 ** -8 * want.reshape(len(want), H, vdim).square().mean(-1).sqrt().repeat_interleave(vdim, 1) + 1e-6
    assert torch.isfinite(got).all() and float(((got - want).abs() / bound).max()) < 1.0


def test_one_query_row_for_all_tokens():
    """Queries with a stride of zero have no tensor map: the other kernels take them, given wide tiles or not."""
    from math_utils_b200.csrc import ops
    n, H, dim = 130, 2, 64
    rows, q, outs = _rand((3, 64, 2 * H * dim), 1), _rand((1, H * dim), 2), []
    for x in (q.expand(n, H * dim), q.repeat(n, 1)):
        out = torch.zeros((n, H * dim), device="cuda", dtype=torch.bfloat16)
        ops.mapped_attention(x, rows, _ints([range(3)]), 64, _ints(range(n)), _ints([0] * n), H, H, 1, dim, dim, 0.1, 0, out,
                             tiles=_ints([(0, 64), (64, 64), (128, 2)]), tiles_wide=_ints([(0, 128), (128, 2)]))
        outs.append(out.double())
    bound = 2.0 ** -7 * outs[1].abs() + 2.0 ** -8 * outs[1].square().mean(1, keepdim=True).sqrt()
    assert float(((outs[0] - outs[1]).abs() / bound).max()) < 1.0


def test_expanded_values_that_are_not_finite_stay_with_the_queries_that_see_them():
    from math_utils_b200.csrc import ops
    H, dim, rot, vdim, n, at = 2, 64, 32, 48, 300, 130
    rows, q = _rand((5, 64, H * (dim + vdim) + rot), 1), _rand((n, H * (dim + rot)), 2)
    tiles, outs = _ints([(o, min(128, n - o)) for o in range(0, n, 128)]), []
    for _ in range(2):
        out = torch.zeros((n, H * vdim), device="cuda", dtype=torch.bfloat16)
        ops.latent_prompt(q, rows, _ints([range(5)]), _ints(range(n)), _ints([0] * n), tiles, H, dim, rot, vdim, 0.1, out)
        ops.check_status()
        outs.append(out.double())
        rows[at // 64, at % 64, H * dim: H * (dim + vdim)] = float("nan")
    assert outs[1][at:].isnan().all() and torch.isfinite(outs[1][:at]).all()
    want = outs[0][:at]
    assert float(((outs[1][:at] - want).abs() / (2.0 ** -7 * want.abs() + 2.0 ** -8 * want.square().mean(1, keepdim=True).sqrt())).max()) < 1.0


LATENTS = [(4, 64, 32, 64, 256, 96, "pairs", False, True), (2, 128, 64, 128, 64, 0, "half", True, False),
           (3, 64, 16, 48, 72, 0, "half", True, True)]


def _latent_part(H, dim, rot, vdim, rank, q_rank, layout, gate, sink):
    """A layer whose prompt steps expand their rows whatever their size."""
    from math_utils_b200.config.base import PartSpec
    from math_utils_b200.engine.runtime import Runtime
    from math_utils_b200.parts.base import build_part
    names = ["dkv", "dkv_norm", "uk", "uv", "out"] + (["dq", "dq_norm", "uq"] if q_rank else ["q"])
    names += ["gate"] * gate + ["sink"] * sink
    params = dict(hidden_size=192, n_heads=H, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=rank, q_rank=q_rank, gate=gate, sink=sink,
                  softmax_scale=(dim + rot) ** -0.5, eps=1e-5, rot_layout=layout, exact_weights=True, rot={"base": 10000.0, "dims": rot})
    part = build_part("mixer", PartSpec("latent_attention", params, {n: n for n in names}))
    tensors = {}
    for i, spec in enumerate(part.tensor_specs()):
        x = torch.randn(spec.shape, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda")
        tensors[spec.name] = (x * spec.shape[-1] ** -0.5).to(torch.bfloat16) if spec.role == "matrix" else 1.0 + 0.1 * x
    part.bind(tensors, Runtime.create("bfloat16", "cuda:0"))
    assert part.expand is not None
    part.EXPANDED_FLOP = 0.0
    return part


def _latent_steps(part, steps, monkeypatch, trace=None):
    """The results of one step after another of three sequences, and how often each step expanded its rows."""
    from math_utils_b200.cache import SequenceCache
    from math_utils_b200.csrc import ops
    from math_utils_b200.engine.batch import PinnedRing, StepEntry, build_context
    took, found, check = [], [], ops._check
    cache = SequenceCache([part.cache_spec()], 4096, 4096, torch.bfloat16, part.runtime.device, n_slots=3)
    slots, ring, work = [cache.acquire() for _ in range(3)], PinnedRing(), {}
    with monkeypatch.context() as m:
        m.setattr(ops, "_check", lambda code, what, *a, **k: (took.append(str(what)), check(code, what, *a, **k))[1])
        for k, lens in enumerate(steps):
            entries = [StepEntry(s, [0] * n, ()) for s, n in zip(slots, lens)]
            ctx = build_context(part.runtime, None, cache, entries, [cache.reserve(s, n) for s, n in zip(slots, lens)], ring, work, trace)
            y = torch.zeros((sum(lens), 192), device="cuda")
            part.forward(_rand((sum(lens), 192), 50 + k), y, ctx, cache.entry(0), True, accumulate=False)
            for s, n in zip(slots, lens):
                cache.commit(s, n)
            found.append(y)
            took.append("|")
    ops.check_status()
    return found, [(step.count("latent_rows"), step.count("latent_prompt(")) for step in " ".join(took).split("|")[:-1]]


@pytest.mark.parametrize("H,dim,rot,vdim,rank,q_rank,layout,gate,sink", LATENTS)
def test_latent_prompts_over_expanded_rows(H, dim, rot, vdim, rank, q_rank, layout, gate, sink, monkeypatch):
    """A layer's prompt steps with keys and values expanded against the same layer in latent space: whole prompts, then steps
    that go on from cached positions.  Both round a row's keys, values and sums to bfloat16 in different places: some three
    roundings of 2^-9 of a value each side, held to 1.2 % of the output's rms, rms over rms."""
    part = _latent_part(H, dim, rot, vdim, rank, q_rank, layout, gate, sink)
    steps = [[70, 1, 200], [100, 130, 64], [3, 2, 190]]
    expanded, runs = _latent_steps(part, steps, monkeypatch)
    part.expand = None
    latent, none = _latent_steps(part, steps, monkeypatch)
    assert runs == [(1, 1)] * 3 and none == [(0, 0)] * 3
    for a, b in zip(expanded, latent):
        assert torch.isfinite(a).all()
        off = (a - b).double().square().mean(1).sqrt() / b.double().square().mean().sqrt()
        assert float(off.max()) < 0.05 and float(off.square().mean().sqrt()) < 0.012


def test_latent_prompt_steps_with_sequences_that_bring_nothing(monkeypatch):
    """Pages are counted for the sequences that attend: the same bits with a sequence without tokens before or between."""
    part = _latent_part(*LATENTS[0])
    want, _ = _latent_steps(part, [[70, 200, 0], [40, 100, 0]], monkeypatch)
    for steps in ([[0, 70, 200], [0, 40, 100]], [[70, 0, 200], [40, 0, 100]]):
        found, runs = _latent_steps(part, steps, monkeypatch)
        assert runs == [(1, 1)] * 2 and all(torch.equal(a, b) for a, b in zip(found, want))


def test_latent_prompt_steps_tell_a_trace_what_both_forms_go_through(monkeypatch):
    part, steps, names = _latent_part(*LATENTS[1]), [[70, 1, 200]], []
    plain, runs = _latent_steps(part, steps, monkeypatch)
    traced, also = _latent_steps(part, steps, monkeypatch, lambda name, tensor: names.append(name))
    assert names == ["proj", "q_latent", "mixed", "q", "kv", "attn"] and torch.equal(plain[0], traced[0]) and runs == also == [(1, 1)]

    class Times:
        wants_values = False

        def __call__(self, name, tensor):
            names.append(name)

    names.clear()
    _latent_steps(part, steps, monkeypatch, Times())
    assert names == ["proj", "q", "kv", "attn"]


def test_latent_prompt_steps_without_room_stay_in_latent_space(monkeypatch):
    part = _latent_part(*LATENTS[0])
    monkeypatch.setattr(part.runtime.ops, "STEP_ROOM", 2 * (200 + 64 * 3) * (4 * 128 + 256 + 32) - 1)
    assert _latent_steps(part, [[70, 0, 129], [0, 0, 72]], monkeypatch)[1] == [(1, 1), (0, 0)]


def test_latent_layers_hold_their_value_projection_once():
    part = _latent_part(*LATENTS[2])
    H, dim = part.n_heads, part.dim
    assert part.v_up.data_ptr() == part.expand.weight[H * dim:].data_ptr() and part.v_up.is_contiguous()


def test_queries_rotate_more_pairs_than_a_block_keeps_angles_of():
    """Queries alone (no cache row is written) of any rotated size, as the angles in float32 turn them."""
    from math_utils_b200.csrc import ops
    T, H, rot = 5, 2, 1604
    q, qa = _rand((T, H * rot), 1).float(), torch.zeros((T, H * rot), device="cuda")
    freqs = 10000.0 ** (-torch.arange(rot // 2, device="cuda").float() * 2 / rot)
    rows = torch.zeros((1, 64, 8 + rot), device="cuda")
    ops.latent_append(None, None, 0.0, freqs, 1.0, rot, 8, rot, _ints(range(T)), _ints([0] * T), _ints([[0]]), 64, rows,
                      queries=(q, rot, qa, rot, H))
    angle = torch.arange(T, device="cuda")[:, None].float() * freqs
    cos, sin = (f(angle.double())[:, None] for f in (torch.cos, torch.sin))
    lo, hi = q.double().reshape(T, H, 2, rot // 2).unbind(2)
    want = torch.stack([lo * cos - hi * sin, hi * cos + lo * sin], 2).reshape(T, -1)
    assert float((qa.double() - want).abs().max()) < 1e-5


# pieces of eight entries: one a slice, lanes without a piece (24, 40, 96, 200), all of a warp's; no rotation, a part of the slice
# and all of it, by halves and by pairs (6: within a piece); with and without norms; more slices than a block takes at once
@pytest.mark.parametrize("heads,kv_heads,maps,dim,vdim,rot,pairs,normed", [
    (3, 1, 1, 8, 8, 0, False, True), (4, 2, 2, 24, 16, 16, False, True), (5, 1, 1, 40, 24, 6, True, False),
    (16, 4, 2, 64, 128, 32, False, True), (8, 8, 1, 96, 96, 96, False, True), (4, 2, 1, 128, 64, 128, True, True),
    (2, 1, 1, 200, 40, 16, False, False), (9, 3, 1, 256, 128, 32, True, True)])
def test_preparation_by_pieces_is_the_general_one(heads, kv_heads, maps, dim, vdim, rot, pairs, normed):
    """Against the form for any alignment (rows one entry off): float32 in between, so a result differs by the last bit of a
    bfloat16 (2^-7 of its size at most) where a sum of another order rounds the other way, and rarely."""
    from math_utils_b200.csrc import ops
    rng = np.random.default_rng(dim)
    T, qw, kw, vw = 70, heads * maps * dim, kv_heads * maps * dim, kv_heads * vdim
    width = qw + kw + vw
    x = torch.as_tensor(rng.normal(0, 2, (T, width)), dtype=torch.float32).cuda().bfloat16()
    weights = [torch.as_tensor(rng.normal(1, 0.2, dim), dtype=torch.float32).cuda() if normed else None for _ in range(2)]
    freqs = torch.as_tensor(300.0 ** -np.linspace(0, 1, max(rot // 2, 1)), dtype=torch.float32).cuda()
    ints = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.int32).cuda()
    pos, table = ints(np.arange(T) + 30), ints([[2, 0]])
    got = []
    for off in (0, 1):
        proj = torch.zeros((T, width + 8 if off == 0 else width + 9), dtype=torch.bfloat16, device="cuda")
        proj[:, off:off + width] = x
        rows = torch.zeros((3, 64, kw + vw), dtype=torch.bfloat16, device="cuda")
        q, k, v = proj[:, off:off + qw], proj[:, off + qw:off + qw + kw], proj[:, off + qw + kw:off + width]
        ops.qk_prepare(q, k, v, *weights, freqs, 1.25, rot, 1e-3, heads, kv_heads, maps, dim, vdim, pos, ints([0] * T), table, 64,
                       rows, pairs=pairs)
        assert not proj[:, :off].any() and not proj[:, off + width:].any()
        got.append((q.float().clone(), rows.float()))
    for a, b in zip(*got):
        assert ((a - b).abs() <= b.abs() * 2.0 ** -7).all() and float((a != b).float().mean()) < 0.01
    untouched = torch.ones(3, 64, dtype=torch.bool)
    untouched[2, 30:] = untouched[0, :36] = False
    assert not got[0][1][untouched.cuda()].any()


# a layer that reads another layer's rows prepares its queries alone: slices that leave lanes of a warp without one, and that fill it
@pytest.mark.parametrize("heads,maps,dim", [(6, 1, 64), (3, 1, 128), (3, 2, 64), (1, 1, 8), (5, 1, 96), (16, 2, 64)])
@pytest.mark.parametrize("rot,pairs", [(0, False), (16, False), (6, True)])
def test_queries_alone_by_pieces(heads, maps, dim, rot, pairs):
    """The general form's values (rows one entry off), as above, and the float64 ones."""
    from math_utils_b200.csrc import ops
    rng = np.random.default_rng(heads * dim)
    T, width = 37, heads * maps * dim
    rot = rot if dim >= 16 or pairs else 0
    x = torch.as_tensor(rng.normal(0, 2, (T, width)), dtype=torch.float32).cuda().bfloat16()
    weight = torch.as_tensor(rng.normal(1, 0.2, dim), dtype=torch.float32).cuda()
    freqs = torch.as_tensor(300.0 ** -np.linspace(0, 1, max(rot // 2, 1)), dtype=torch.float32).cuda()
    pos = torch.arange(T, dtype=torch.int32, device="cuda") + 30
    got = []
    for off in (0, 1):
        proj = torch.zeros((T, width + 8 if off == 0 else width + 9), dtype=torch.bfloat16, device="cuda")
        proj[:, off:off + width] = x
        ops.qk_prepare(proj[:, off:off + width], None, None, weight, None, freqs, 1.25, rot, 1e-3, heads, 1, maps, dim, dim, pos, None,
                       None, 64, None, pairs=pairs)
        assert not proj[:, :off].any() and not proj[:, off + width:].any()
        got.append(proj[:, off:off + width].float())
    a, b = got
    assert ((a - b).abs() <= b.abs() * 2.0 ** -7).all() and float((a != b).float().mean()) < 0.01
    y = x.double().reshape(T, heads * maps, dim)
    y = y / (y.square().mean(-1, keepdim=True) + 1e-3).sqrt() * weight.double()
    if rot:
        angle = (pos[:, None].float() * freqs).double()[:, None]
        cos, sin = angle.cos() * 1.25, angle.sin() * 1.25
        lo, hi = (y[..., 0:rot:2], y[..., 1:rot:2]) if pairs else (y[..., :rot // 2], y[..., rot // 2:rot])
        turned = torch.stack([lo * cos - hi * sin, hi * cos + lo * sin], -1 if pairs else -2).reshape(T, -1, rot)
        y = torch.cat([turned, y[..., rot:]], -1)
    # half a bfloat16's last bit, and float32 angles, norms and turns in front of it
    assert ((a.double() - y.reshape(T, -1)).abs() <= y.reshape(T, -1).abs() * 2.0 ** -8 + 1e-4).all()
