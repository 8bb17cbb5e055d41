"""Cases for timing the framework, with their inputs, their results in 64 bits and what the results may differ by.

Two cases are whole steps of a GPT-2-sized model as its programs make them: single tokens replayed by a
``DecodeSession`` and a prompt step.  The others are single layers of the other designs, each built from its
``PartSpec`` and run on a cache and a step context as the model's step runs it: prompt steps through the part's
``forward``, single-token steps replayed from a CUDA graph of that ``forward``, as every single-token step of the
framework is.  Sizes are those of the repository's own configurations (GPT-2 small; the sizes s and m of the
benchmark's families); ``draw`` spreads over sequence counts and lengths, contexts, widths and heads around them.
"""
import math

import numpy as np
import torch

from math_utils_b200.cache import SequenceCache
from math_utils_b200.config.base import PartSpec
from math_utils_b200.config.gpt2 import Gpt2Config
from math_utils_b200.engine.assemble import collect_tensor_specs
from math_utils_b200.engine.batch import PinnedRing, StepEntry, build_context
from math_utils_b200.engine.decode_session import DecodeSession
from math_utils_b200.engine.model import DecoderModel
from math_utils_b200.engine.runtime import Runtime
from math_utils_b200.parts.base import FreeSize, build_part
from math_utils_b200.sampling import SamplingParams

DEVICE = "cuda:0"
EPS = 1e-5


# ---------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one token for each of eight conversations half-way through GPT-2 small's context: the library's headline step
        {"name": "gpt2_single_b8", "kind": "gpt2", "phase": "single", "n_layer": 12, "width": 768, "heads": 12,
         "inner": 3072, "vocab": 50257, "batch": 8, "context": 520},
        # two whole prompts of GPT-2 small's context in one step
        {"name": "gpt2_prompt_2x1024", "kind": "gpt2", "phase": "prompt", "n_layer": 12, "width": 768, "heads": 12,
         "inner": 3072, "vocab": 50257, "lens": "1024,1024"},
        # windowed attention with two score maps over a prompt of two sequences (Lusalorn, size s)
        {"name": "differential_prompt", "kind": "differential", "phase": "prompt", "width": 1024, "heads": 8,
         "kv_heads": 2, "dim": 64, "vdim": 128, "window": 512, "lens": "1024,1024"},
        # one token for each of eight conversations through grouped-query attention with a sink and gates: the smallest
        # call of a layer (Seledra, size s)
        {"name": "sink_single_b8", "kind": "sink", "phase": "single", "width": 1024, "heads": 8, "kv_heads": 2,
         "dim": 128, "vdim": 128, "batch": 8, "context": 1500},
        # latent attention with a query latent over an unequal batch of prompts (Tibopel, size m)
        {"name": "latent_prompt", "kind": "latent", "phase": "prompt", "width": 2048, "heads": 16, "dim": 128,
         "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 768, "lens": "1001,700,347"},
        # routed experts over a full prompt step: the largest layer (Forisun, size m)
        {"name": "experts_prompt", "kind": "experts", "phase": "prompt", "form": "gated_silu", "width": 2048,
         "inner": 1408, "experts": 64, "top": 6, "identity": 0, "shared": 0, "lens": "1024,1024"},
        # routed experts with identity experts and a shared one, one token for each of eight conversations (Tibopel, m)
        {"name": "experts_single_b8", "kind": "experts", "phase": "single", "form": "relu2", "width": 2048,
         "inner": 1408, "experts": 64, "top": 6, "identity": 8, "shared": 2816, "batch": 8, "context": 0},
        # the gated delta rule over two prompts (Seledra, size s)
        {"name": "delta_prompt", "kind": "delta", "phase": "prompt", "width": 1024, "heads": 8, "kv_heads": 4,
         "dim": 128, "vdim": 128, "taps": 4, "lens": "1024,1024"},
        # the state-space mixer over two prompts (Lusalorn, size s)
        {"name": "state_space_prompt", "kind": "state_space", "phase": "prompt", "width": 1024, "heads": 16, "vdim": 64,
         "state": 128, "groups": 1, "taps": 4, "lens": "1024,1024"},
        # the matrix memory of xLSTM over two unequal prompts of odd lengths (Pelenex, size s)
        {"name": "matrix_lstm_prompt", "kind": "matrix_lstm", "phase": "prompt", "width": 1024, "heads": 8, "dim": 128,
         "vdim": 128, "lens": "1501,517"},
        # the selective scan over three prompts, one of them short (Tokolorn, size s)
        {"name": "selective_prompt", "kind": "selective", "phase": "prompt", "width": 1024, "inner": 2048, "state": 16,
         "dt_rank": 64, "taps": 4, "lens": "1000,83,900"},
        # the feed-forward of the true 32-bit path over an odd number of tokens (GPT-2 small, float32)
        {"name": "ffn_float32_prompt", "kind": "ffn", "phase": "prompt", "dtype": "float32", "width": 768,
         "inner": 3072, "lens": "500,277"},
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _lens(rng, most):
    """Between one and four sequences, 48 to ``most`` tokens together, cut at random places."""
    total = _spread(rng, 48, most)
    n = min(rng.randint(1, 4), total)
    cuts = sorted(rng.sample(range(1, total), n - 1))
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))


def draw(rng):
    kind = rng.choice(["gpt2", "differential", "sink", "latent", "experts", "delta", "state_space", "matrix_lstm",
                       "selective", "ffn"])
    c = {"kind": kind, "phase": "prompt"}
    if kind == "gpt2":
        heads = rng.choice([6, 8, 12])
        c.update(n_layer=rng.randint(2, 10), width=64 * heads, heads=heads, inner=rng.choice([3, 4]) * 64 * heads,
                 vocab=rng.choice([1031, 8192, 50257]))
        if rng.random() < 0.5:
            c.update(phase="single", batch=_spread(rng, 1, 64), context=_spread(rng, 16, 1000))
        else:
            c["lens"] = ",".join(str(min(1000, int(n))) for n in _lens(rng, 1900).split(","))
        return c
    c["width"] = rng.choice([512, 768, 1024])
    if kind in ("differential", "sink"):
        kv = rng.choice([1, 2, 4])
        c.update(heads=kv * rng.choice([2, 4]), kv_heads=kv, dim=rng.choice([64, 96, 128]))
        c["vdim"] = 128 if kind == "differential" else c["dim"]
        if kind == "differential":
            c.update(dim=64, heads=min(c["heads"], 8), window=rng.choice([128, 300, 512]))
        c["heads"] = min(c["heads"], 8)
        if rng.random() < 0.4:
            c.update(phase="single", batch=_spread(rng, 1, 24), context=_spread(rng, 16, 1800))
    elif kind == "latent":
        s = rng.random() < 0.6
        c.update(heads=rng.choice([4, 8, 16]), dim=64 if s else 128, rot_dim=32 if s else 64, vdim=64 if s else 128,
                 kv_rank=256 if s else 512, q_rank=rng.choice([256, 384, 768]))
        if rng.random() < 0.3:
            c.update(phase="single", batch=_spread(rng, 1, 24), context=_spread(rng, 16, 1800))
    elif kind == "experts":
        c.update(form=rng.choice(["gated_silu", "relu2"]), inner=rng.choice([512, 704, 1024]),
                 experts=rng.choice([8, 16, 48]), top=rng.randint(1, 6))
        relu2 = c["form"] == "relu2"
        c.update(identity=rng.choice([0, 4]) if relu2 else 0, shared=rng.choice([0, 1024]) if relu2 else 0)
        if rng.random() < 0.3:
            c.update(phase="single", batch=_spread(rng, 1, 48), context=0)
    elif kind == "delta":
        kv = rng.choice([2, 4])
        c.update(heads=kv * rng.choice([1, 2]), kv_heads=kv, dim=rng.choice([64, 96, 128]), vdim=rng.choice([64, 128]),
                 taps=rng.choice([3, 4]))
    elif kind == "state_space":
        c.update(heads=rng.choice([4, 8, 16]), vdim=64, state=rng.choice([64, 96, 128]), groups=rng.choice([1, 2]),
                 taps=rng.choice([3, 4]))
    elif kind == "matrix_lstm":
        c.update(heads=rng.choice([2, 4, 8]), dim=rng.choice([64, 96, 128]), vdim=rng.choice([64, 128]))
    elif kind == "selective":
        c.update(inner=rng.choice([512, 1000, 2048]), state=16, dt_rank=rng.choice([32, 48, 64]), taps=4)
    else:
        c.update(dtype=rng.choice(["float32", "float32", "bfloat16"]), inner=rng.choice([1024, 2000, 3072]))
    if c["phase"] == "prompt":
        c["lens"] = _lens(rng, 700 if c.get("dtype") == "float32" else 2000)
    return c


def _lengths(case):
    """(tokens before the step, tokens of the step) of every sequence."""
    if case["phase"] == "single":
        return [(int(case["context"]), 1)] * int(case["batch"])
    return [(0, int(n)) for n in case["lens"].split(",")]


# ------------------------------------------------------------------------------------------- weights and inputs
def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _generator(seed, which):
    return torch.Generator(device=DEVICE).manual_seed(seed * 1_000_003 + which)


def _spec(case):
    """(role, the part's specification) of a layer case."""
    kind, D = case["kind"], case["width"]
    sizes = {k: case[k] for k in ("dim", "vdim") if k in case}
    sizes.update(hidden_size=D, eps=EPS)
    if "heads" in case:
        sizes["n_heads"] = case["heads"]
    if kind == "differential":
        names = ["q", "k", "v", "q_norm", "k_norm", "out", "q_bias", "k_bias", "v_bias", "out_bias", "lq1", "lk1", "lq2", "lk2"]
        sizes.update(n_kv_heads=case["kv_heads"], maps=2, softmax_scale=case["dim"] ** -0.5, window=case["window"],
                     bias=True, diff=0.2, rot={"base": 500000.0, "dims": case["dim"] // 2})
        return "mixer", PartSpec("mapped_attention", sizes, {n: n for n in names})
    if kind == "sink":
        names = ["q", "k", "v", "q_norm", "k_norm", "out", "q_bias", "k_bias", "v_bias", "head_scale", "gate"]
        sizes.update(n_kv_heads=case["kv_heads"], softmax_scale=case["dim"] ** -0.5, bias=True, value_norm=True, sink=True,
                     head_scale=True, head_gate=True)
        return "mixer", PartSpec("sink_attention", sizes, {n: n for n in names})
    if kind == "latent":
        names = ["dq", "dq_norm", "uq", "dkv", "dkv_norm", "uk", "uv", "sink", "out"]
        sizes.update(rot_dim=case["rot_dim"], kv_rank=case["kv_rank"], q_rank=case["q_rank"], gate=False, sink=True,
                     softmax_scale=(case["dim"] + case["rot_dim"]) ** -0.5, rot_layout="pairs", exact_weights=True,
                     rot={"base": 10000.0, "dims": case["rot_dim"]})
        return "mixer", PartSpec("latent_attention", sizes, {n: n for n in names})
    if kind == "experts":
        sizes.update(inner_size=case["inner"], n_experts=case["experts"], top=case["top"], correction=True)
        names = {"router": "router", "correction": "correction", "up": "e{e}.up", "down": "e{e}.down"}
        if case["form"] == "gated_silu":
            sizes.update(score="sigmoid", router_scale=2.0)
            names["gate"] = "e{e}.gate"
        else:
            sizes.update(score="softmax", renormalize=True, renorm_eps=1e-20, expert_form="relu2", identity=case["identity"])
            if case["shared"]:
                sizes["shared"] = {"inner_size": case["shared"], "gate": True}
                names.update(shared_up="shared_up", shared_down="shared_down", shared_gate="shared_gate")
        return "feed_forward", PartSpec("routed_experts", sizes, names)
    if kind == "delta":
        names = ["q", "k", "v", "q_conv", "k_conv", "v_conv", "beta", "decay", "A_log", "dt_bias", "norm", "gate", "out"]
        sizes.update(n_kv_heads=case["kv_heads"], conv=case["taps"])
        return "mixer", PartSpec("gated_delta", sizes, {n: n for n in names})
    if kind == "state_space":
        names = ["in", "conv", "conv_bias", "dt_bias", "A_log", "D", "norm", "out"]
        sizes.update(head_dim=case["vdim"], state=case["state"], groups=case["groups"], conv=case["taps"], norm_groups=1)
        return "mixer", PartSpec("state_space", sizes, {n: n for n in names})
    if kind == "matrix_lstm":
        names = ["q", "k", "v", "gate", "i", "i_bias", "f", "f_bias", "norm", "out"]
        sizes["gate_cap"] = 15.0
        return "mixer", PartSpec("matrix_lstm", sizes, {n: n for n in names})
    if kind == "selective":
        names = ["in", "conv", "conv_bias", "x", "dt", "dt_bias", "A_log", "D", "out"]
        sizes.update(inner=case["inner"], state=case["state"], dt_rank=case["dt_rank"], conv=case["taps"])
        return "mixer", PartSpec("selective_scan", sizes, {n: n for n in names})
    names = ["up_weight", "up_bias", "down_weight", "down_bias"]
    sizes.update(inner_size=case["inner"], activation="gelu_new")
    return "feed_forward", PartSpec("dense_ffn", sizes, {n: n for n in names})


def _values(case, spec, gen):
    """One tensor's values, float32: matrices that keep a row's size, and the recurrences' rates where trained models
    have them (memories of ten to some thousand tokens)."""
    shape = tuple(s.default if isinstance(s, FreeSize) else int(s) for s in spec.shape)
    normal = torch.randn(shape, generator=gen, device=DEVICE)
    name = spec.name
    if spec.role in ("matrix", "matrix32"):
        return normal * shape[-1] ** -0.5
    if name.endswith("conv"):
        return normal * 0.5
    if name == "A_log" and case["kind"] == "selective":
        return torch.log(torch.arange(1, shape[1] + 1, device=DEVICE, dtype=torch.float32)).expand(shape) + 0.05 * normal
    if name == "A_log":
        return torch.log(1.0 + 7.0 * torch.rand(shape, generator=gen, device=DEVICE))
    if name == "dt_bias":
        return -5.0 + 3.0 * torch.rand(shape, generator=gen, device=DEVICE)
    if name == "f_bias":
        return 3.0 + 3.0 * torch.rand(shape, generator=gen, device=DEVICE)
    if spec.init in ("norm_weight", "head_scale"):
        return 1.0 + 0.1 * normal
    return 0.1 * normal


def _tensors(case, specs, seed):
    """Name -> (tensor as the part takes it, in the layout of ``[out, in]``)."""
    gen, dt, found = _generator(seed, 1), _dtype(case), {}
    for spec in specs:
        x = _values(case, spec, gen)
        found[spec.name] = x.to(dt if spec.role in ("matrix", "table") else torch.float32).contiguous()
    return found


def _rows(case, seed):
    """A layer's input, the normed stream of every token that the sequences hold after the step: [sequence][tokens, width]."""
    gen = _generator(seed, 2)
    return [torch.randn((before + n, case["width"]), generator=gen, device=DEVICE).to(_dtype(case))
            for before, n in _lengths(case)]


def _gpt2_config(case):
    return Gpt2Config(n_layer=case["n_layer"], n_embd=case["width"], n_head=case["heads"], vocab_size=case["vocab"],
                      n_positions=1024, n_inner=case["inner"])


def _gpt2_tensors(case, plan, seed):
    """The tensors as GPT-2's seeded initialisation draws them."""
    gen, found = _generator(seed, 1), {}
    for spec in collect_tensor_specs(plan):
        shape = tuple(reversed(spec.shape)) if spec.transpose else tuple(spec.shape)
        x = torch.randn(shape, generator=gen, device=DEVICE) * 0.02
        if spec.init == "residual_projection":
            x /= math.sqrt(2 * case["n_layer"])
        if spec.init == "norm_weight":
            x += 1.0
        found[spec.name] = x.to(torch.bfloat16 if spec.role in ("matrix", "table") else torch.float32)
    return found


def _tokens(case, seed):
    rng = np.random.RandomState(seed % (1 << 31))
    return [rng.randint(0, case["vocab"], before + n).tolist() for before, n in _lengths(case)]


# ------------------------------------------------------------------------------------------------------- prepare
def _pages(tokens):
    return -(-tokens // 64) * 64


def _prepare_gpt2(case, seed):
    plan = _gpt2_config(case).plan()
    model = DecoderModel(plan, _gpt2_tensors(case, plan, seed), Runtime.create("bfloat16", DEVICE))
    tokens = _tokens(case, seed)
    cache = model.new_cache(max_tokens=sum(_pages(len(t)) for t in tokens), n_slots=len(tokens))
    state = {"case": case, "model": model, "cache": cache, "tokens": tokens}
    if case["phase"] == "single":
        slots = [cache.acquire() for _ in tokens]
        model.step(cache, [StepEntry(s, t[:-1], ()) for s, t in zip(slots, tokens)])
        for s in slots:
            cache.reserve(s, 1)
        session = DecodeSession(model, cache, slots, SamplingParams(temperature=0.0), list(range(len(slots))))
        session.sync_block_tables()
        state.update(session=session, last=[t[-1] for t in tokens], at=[len(t) - 1 for t in tokens])
        session.feed(state["last"], state["at"])
        session.capture()
    return state


def prepare(case, seed):
    if case["kind"] == "gpt2":
        return _prepare_gpt2(case, seed)
    role, spec = _spec(case)
    part = build_part(role, spec)
    runtime = Runtime.create(_dtype(case), DEVICE)
    part.bind(_tensors(case, part.tensor_specs(), seed), runtime)
    rows, lengths = _rows(case, seed), _lengths(case)
    cache_spec = part.cache_spec() if role == "mixer" else None
    cache = SequenceCache([cache_spec], sum(_pages(b + n) for b, n in lengths), 4096, runtime.dtype, runtime.device,
                          n_slots=len(lengths))
    slots, ring, workspace = [cache.acquire() for _ in lengths], PinnedRing(), {}
    view = cache.entry(0)

    def context(counts):
        entries = [StepEntry(s, [0] * n, ()) for s, n in zip(slots, counts) if n]
        starts = [cache.reserve(e.slot, len(e.tokens)) for e in entries]
        return build_context(runtime, None, cache, entries, starts, ring, workspace)

    def forward(h, y, ctx):
        if role == "mixer":
            part.forward(h, y, ctx, view, True, accumulate=False)
        else:
            part.forward(h, y, ctx, accumulate=False)

    if role == "mixer" and any(b for b, _ in lengths):             # what the sequences hold before the step
        before = torch.cat([r[:b] for r, (b, _) in zip(rows, lengths)])
        ctx = context([b for b, _ in lengths])
        forward(before, torch.empty(before.shape, dtype=torch.float32, device=DEVICE), ctx)
        for s, (b, _) in zip(slots, lengths):
            cache.commit(s, b)
    h = torch.cat([r[b:] for r, (b, _) in zip(rows, lengths)]).contiguous()
    y = torch.zeros(h.shape, dtype=torch.float32, device=DEVICE)
    ctx = context([n for _, n in lengths])
    state = {"case": case, "forward": forward, "h": h, "y": y, "ctx": ctx, "view": view, "graph": None}
    if case["phase"] == "single":
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            forward(h, y, ctx)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            forward(h, y, ctx)
    return state


# ----------------------------------------------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    if case["kind"] == "gpt2":
        cache = state["cache"]
        if case["phase"] == "single":
            session = state["session"]
            session.feed(state["last"], state["at"])
            session.launch()
            return {"logits": session.logits, "pages": [cache.entry(i).pages for i in range(case["n_layer"])]}
        slots = [cache.acquire() for _ in state["tokens"]]
        logits = state["model"].step(cache, [StepEntry(s, t, [len(t) - 1]) for s, t in zip(slots, state["tokens"])])
        for s in slots:
            cache.release(s)
        return {"logits": logits, "pages": [cache.entry(i).pages for i in range(case["n_layer"])]}
    if state["graph"] is not None:
        state["graph"].replay()
    else:
        state["forward"](state["h"], state["y"], state["ctx"])
    view = state["view"]
    if view is None:
        return {"out": state["y"]}
    return {"out": state["y"], "kept": view.values if hasattr(view, "values") else view.pages}


# ----------------------------------------------------------------------------------------------- work, tolerance
def _pairs(before, n, window=0):
    """(query, key) pairs that are seen."""
    q = np.arange(before, before + n, dtype=np.float64) + 1.0
    return float(np.minimum(q, window).sum() if window else q.sum())


def work(case):
    kind, D, lengths = case["kind"], case["width"], _lengths(case)
    T = float(sum(n for _, n in lengths))
    size = 4.0 if case.get("dtype") == "float32" else 2.0
    if kind == "gpt2":
        L, inner, V = case["n_layer"], case["inner"], case["vocab"]
        matrices = L * (4.0 * D * D + 2.0 * D * inner)
        held = sum(b + n for b, n in lengths)
        seqs = len(lengths)
        pairs = sum(_pairs(b, n) for b, n in lengths)
        read = held if case["phase"] == "single" else T                     # a prompt's own rows are written once
        return {"bytes": 2.0 * (matrices + V * D) + 4.0 * L * D * read + 4.0 * seqs * V,
                "flops": 2.0 * T * matrices + 4.0 * D * L * pairs + 2.0 * seqs * V * D}
    io = T * D * (size + 4.0)                                                # the input rows and the float32 result
    if kind == "ffn":
        return {"bytes": io + 2.0 * D * case["inner"] * size, "flops": 4.0 * T * D * case["inner"]}
    if kind == "experts":
        per = (3 if case["form"] == "gated_silu" else 2) * D * case["inner"]
        real = case["top"] * case["experts"] / (case["experts"] + case["identity"])
        used = case["experts"] * (1.0 - (1.0 - case["top"] / (case["experts"] + case["identity"])) ** T)
        return {"bytes": io + 2.0 * (used * per + 2.0 * D * case["shared"]) + 4.0 * D * (case["experts"] + case["identity"]),
                "flops": 2.0 * T * (real * per + 2.0 * D * case["shared"] + D * (case["experts"] + case["identity"]))}
    if kind in ("differential", "sink"):
        H, G, maps = case["heads"], case["kv_heads"], 2 if kind == "differential" else 1
        window = case.get("window", 0)
        widths = H * maps * case["dim"] + G * (maps * case["dim"] + case["vdim"])
        matrices = float(D * (widths + H * case["vdim"] + (H if kind == "sink" else 0)))
        row = G * (maps * case["dim"] + case["vdim"])
        seen = sum(min(b + n, window) if window and case["phase"] == "single" else b + n for b, n in lengths)
        pairs = sum(_pairs(b, n, window) for b, n in lengths)
        return {"bytes": io + 2.0 * matrices + 2.0 * row * seen,
                "flops": 2.0 * T * matrices + 2.0 * pairs * H * maps * (case["dim"] + case["vdim"])}
    if kind == "latent":
        H, r, d, dr, dv = case["heads"], case["kv_rank"], case["dim"], case["rot_dim"], case["vdim"]
        matrices = float(D * (case["q_rank"] + r + dr) + case["q_rank"] * H * (d + dr) + H * (d + dv) * r + H * dv * D)
        held = sum(b + n for b, n in lengths)
        pairs = sum(_pairs(b, n) for b, n in lengths)
        per_pair = 2.0 * H * (d + dr + dv) if case["phase"] == "prompt" else 2.0 * H * (2 * r + dr)
        return {"bytes": io + 2.0 * matrices + 2.0 * (r + dr) * held, "flops": 2.0 * T * matrices + pairs * per_pair}
    seqs = float(len(lengths))
    if kind == "delta":
        H, G, d, dv = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
        matrices = float(D * (2 * G * d + 3 * H * dv + 2 * H))
        kept, scan = H * d * dv + (case["taps"] - 1) * (2 * G * d + H * dv), 6.0 * T * H * d * dv
    elif kind == "state_space":
        H, P, N, G = case["heads"], case["vdim"], case["state"], case["groups"]
        matrices = float(D * (3 * H * P + 2 * G * N + H))
        kept, scan = H * P * N + (case["taps"] - 1) * (H * P + 2 * G * N), 4.0 * T * H * P * N
    elif kind == "matrix_lstm":
        H, d, dv = case["heads"], case["dim"], case["vdim"]
        matrices = float(D * (2 * H * d + 3 * H * dv + 2 * H))
        kept, scan = H * d * (dv + 1) + H, 4.0 * T * H * d * (dv + 1)
    else:
        C, N, R = case["inner"], case["state"], case["dt_rank"]
        matrices = float(3 * D * C + C * (R + 2 * N) + R * C)
        kept, scan = C * N + (case["taps"] - 1) * C, 6.0 * T * C * N
    return {"bytes": io + 2.0 * matrices + 8.0 * seqs * kept, "flops": 2.0 * T * matrices + scan}


def tolerance(case):
    # measured against 64 bits: 0.0016 to 0.005 where weights and rows are bfloat16, 1e-6 in float32
    return {"rel": 1e-5 if case.get("dtype") == "float32" else 1e-2}


# --------------------------------------------------------------------------------------------- results in 64 bits
def _unit(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.logaddexp(torch.zeros_like(x), x)


def _turned(x, freqs, pairs):
    """The first 2 * len(freqs) entries of x [T, ..., n] rotated by position (counted from 0)."""
    half = len(freqs)
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * freqs
    angle = angle.reshape((x.shape[0],) + (1,) * (x.dim() - 2) + (half,))
    cos, sin, out = torch.cos(angle), torch.sin(angle), x.clone()
    first, second = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if pairs else (slice(0, half), slice(half, 2 * half))
    out[..., first] = x[..., first] * cos - x[..., second] * sin
    out[..., second] = x[..., second] * cos + x[..., first] * sin
    return out


def _frequencies(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) / dims)


def _attend(q, k, v, scale, first, window=0, sink=None):
    """q [n, H, d] of the tokens from position ``first`` on, k [T, H, d], v [T, H, dv] -> [n, H, dv]; ``sink``: a score
    per head without a value."""
    out = []
    at_k = torch.arange(k.shape[0], device=k.device)
    for a in range(0, q.shape[0], 256):
        s = torch.einsum("ihd,jhd->hij", q[a:a + 256], k) * scale
        at = first + a + torch.arange(s.shape[1], device=k.device)
        hidden = at_k[None, :] > at[:, None]
        if window:
            hidden |= at[:, None] - at_k[None, :] >= window
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.reshape(-1, 1, 1).expand(s.shape[0], s.shape[1], 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., :k.shape[0]]
        out.append(torch.einsum("hij,jhd->ihd", p, v))
    return torch.cat(out)


def _exact_differential(case, w, h, before):
    H, G, d, dv = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
    T, freqs = h.shape[0], _frequencies(case["dim"] // 2, 500000.0)
    q = _turned(_unit((h @ w["q"].T + w["q_bias"]).reshape(T, H, 2, d)) * w["q_norm"], freqs, False)[before:]
    k = _turned(_unit((h @ w["k"].T + w["k_bias"]).reshape(T, G, 2, d)) * w["k_norm"], freqs, False).repeat_interleave(H // G, 1)
    v = (h @ w["v"].T + w["v_bias"]).reshape(T, G, dv).repeat_interleave(H // G, 1)
    first, second = (_attend(q[:, :, m], k[:, :, m], v, d ** -0.5, before, case["window"]) for m in range(2))
    lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + 0.2
    o = _unit(first - lam * second) * 0.8
    return o.reshape(-1, H * dv) @ w["out"].T + w["out_bias"]


def _exact_sink(case, w, h, before):
    H, G, d, dv = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
    T = h.shape[0]
    q = (_unit(h @ w["q"].T + w["q_bias"]) * w["q_norm"]).reshape(T, H, d)[before:] * w["head_scale"][:, None]
    k = (_unit(h @ w["k"].T + w["k_bias"]) * w["k_norm"]).reshape(T, G, d).repeat_interleave(H // G, 1)
    v = _unit((h @ w["v"].T + w["v_bias"]).reshape(T, G, dv)).repeat_interleave(H // G, 1)
    o = _attend(q, k, v, d ** -0.5, before, sink=torch.zeros(H, dtype=torch.float64, device=DEVICE))
    o = o * torch.sigmoid(h[before:] @ w["gate"].T)[:, :, None]
    return o.reshape(-1, H * dv) @ w["out"].T


def _exact_latent(case, w, h, before):
    H, d, dr, dv, r = case["heads"], case["dim"], case["rot_dim"], case["vdim"], case["kv_rank"]
    T, freqs = h.shape[0], _frequencies(case["rot_dim"], 10000.0)
    q = ((_unit(h @ w["dq"].T) * w["dq_norm"]) @ w["uq"].T).reshape(T, H, d + dr)
    q = torch.cat([q[..., :d], _turned(q[..., d:], freqs, True)], -1)[before:]
    down = h @ w["dkv"].T
    c, shared = _unit(down[:, :r]) * w["dkv_norm"], _turned(down[:, r:], freqs, True)
    k = torch.cat([(c @ w["uk"].T).reshape(T, H, d), shared[:, None].expand(T, H, dr)], -1)
    v = (c @ w["uv"].T).reshape(T, H, dv)
    o = _attend(q, k, v, (d + dr) ** -0.5, before, sink=w["sink"])
    return o.reshape(-1, H * dv) @ w["out"].T


def _exact_experts(case, w, h):
    E, top = case["experts"], case["top"]
    z = h @ w["router"].double().T
    s = torch.sigmoid(z) if case["form"] == "gated_silu" else torch.softmax(z, -1)
    chosen = torch.sort(s + w["correction"].double(), dim=-1, descending=True, stable=True)[1][:, :top]
    weight = torch.gather(s, 1, chosen)
    weight = weight * 2.0 if case["form"] == "gated_silu" else weight / (weight.sum(-1, keepdim=True) + 1e-20)
    y = torch.zeros_like(h)
    for e in range(E + case["identity"]):
        token, place = torch.nonzero(chosen == e, as_tuple=True)
        x = h[token]
        if e < E:
            up = x @ w[f"e{e}.up"].double().T
            up = _silu(x @ w[f"e{e}.gate"].double().T) * up if case["form"] == "gated_silu" else torch.relu(up) ** 2
            x = up @ w[f"e{e}.down"].double().T
        y.index_add_(0, token, x * weight[token, place][:, None])
    if case["shared"]:
        x = torch.relu(h @ w["shared_up"].double().T) ** 2 @ w["shared_down"].double().T
        y += x * torch.sigmoid(h @ w["shared_gate"].double().T)
    return y


def _convolved(u, taps, bias=None):
    """A causal convolution per channel from zeros, then silu; and the inputs that it keeps, newest last."""
    n = taps.shape[1]
    padded = torch.cat([torch.zeros((n - 1, u.shape[1]), dtype=u.dtype, device=u.device), u])
    out = sum(padded[i:i + u.shape[0]] * taps[:, i] for i in range(n))
    return _silu(out if bias is None else out + bias), padded[u.shape[0]:]


def _exact_delta(case, w, h):
    H, G, d, dv = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
    T = h.shape[0]
    u = h @ torch.cat([w["q"], w["k"], w["v"]]).T
    u, tail = _convolved(u, torch.cat([w["q_conv"], w["k_conv"], w["v_conv"]]))
    q, k, v = u[:, :G * d].reshape(T, G, d), u[:, G * d:2 * G * d].reshape(T, G, d), u[:, 2 * G * d:].reshape(T, H, dv)
    q, k = ((x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for x in (q, k))
    q = q * d ** -0.5
    beta = torch.sigmoid(h @ w["beta"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * _softplus(h @ w["decay"].T + w["dt_bias"]))
    S, out = torch.zeros((H, d, dv), dtype=torch.float64, device=DEVICE), []
    for t in range(T):
        S = S * decay[t][:, None, None]
        wrote = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * wrote[:, None, :]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    o = _unit(torch.stack(out)) * w["norm"] * _silu((h @ w["gate"].T).reshape(T, H, dv))
    return o.reshape(T, H * dv) @ w["out"].T, torch.cat([tail.reshape(-1), S.transpose(1, 2).reshape(-1)])


def _exact_state_space(case, w, h):
    H, P, N, G = case["heads"], case["vdim"], case["state"], case["groups"]
    T, inner = h.shape[0], case["heads"] * case["vdim"]
    u = h @ w["in"].T
    z, dt = u[:, :inner], _softplus(u[:, -H:] + w["dt_bias"])
    xbc, tail = _convolved(u[:, inner:-H], w["conv"], w["conv_bias"])
    x = xbc[:, :inner].reshape(T, H, P)
    B, C = (xbc[:, a:a + G * N].reshape(T, G, N).repeat_interleave(H // G, 1) for a in (inner, inner + G * N))
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)
    S, out = torch.zeros((H, N, P), dtype=torch.float64, device=DEVICE), []
    for t in range(T):
        S = S * decay[t][:, None, None] + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
        out.append(torch.einsum("hnp,hn->hp", S, C[t]))
    y = (torch.stack(out) + w["D"][:, None] * x).reshape(T, inner) * _silu(z)
    return (_unit(y) * w["norm"]) @ w["out"].T, torch.cat([tail.reshape(-1), S.reshape(-1)])


def _exact_matrix_lstm(case, w, h):
    H, d, dv = case["heads"], case["dim"], case["vdim"]
    T = h.shape[0]
    q, k = (h @ w["q"].T).reshape(T, H, d) * d ** -0.5, (h @ w["k"].T).reshape(T, H, d)
    v = (h @ w["v"].T).reshape(T, H, dv)
    i = 15.0 * torch.tanh((h @ w["i"].T + w["i_bias"]) / 15.0)
    f = -_softplus(-15.0 * torch.tanh((h @ w["f"].T + w["f_bias"]) / 15.0))
    S = torch.zeros((H, d, dv + 1), dtype=torch.float64, device=DEVICE)
    m, out, v = torch.zeros(H, dtype=torch.float64, device=DEVICE), [], torch.cat([v, torch.ones_like(v[..., :1])], -1)
    for t in range(T):
        new = torch.maximum(f[t] + m, i[t])
        S = S * torch.exp(f[t] + m - new)[:, None, None] + (torch.exp(i[t] - new)[:, None] * k[t])[:, :, None] * v[t][:, None, :]
        m = new
        read = torch.einsum("hdv,hd->hv", S, q[t])
        out.append(read[:, :dv] / (torch.maximum(read[:, dv].abs(), torch.exp(-m)) + 1e-6)[:, None])
    o = _unit(torch.stack(out)).reshape(T, H * dv) * w["norm"] * torch.sigmoid(h @ w["gate"].T)
    return o @ w["out"].T, torch.cat([S[..., :dv].transpose(1, 2).reshape(-1), S[..., dv].reshape(-1), m])


def _exact_selective(case, w, h):
    C, N, R = case["inner"], case["state"], case["dt_rank"]
    u = h @ w["in"].T
    x, tail = _convolved(u[:, :C], w["conv"], w["conv_bias"])
    low = x @ w["x"].T
    dt = _softplus(low[:, :R] @ w["dt"].T + w["dt_bias"])
    A, S, out = -torch.exp(w["A_log"]), torch.zeros((C, N), dtype=torch.float64, device=DEVICE), []
    for t in range(h.shape[0]):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * x[t])[:, None] * low[t, R:R + N]
        out.append(S @ low[t, R + N:])
    y = (torch.stack(out) + w["D"] * x) * _silu(u[:, C:])
    return y @ w["out"].T, torch.cat([tail.reshape(-1), S.reshape(-1)])


def _gelu_new(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _exact_gpt2(case, seed):
    plan = _gpt2_config(case).plan()
    names = {(i, part): spec for i, layer in enumerate(plan.layers) for part, spec in
             (("n1", layer.norm1), ("mix", layer.mixer), ("n2", layer.norm2), ("ff", layer.feed_forward))}
    w = {n: t.double() for n, t in _gpt2_tensors(case, plan, seed).items()}
    D, H = case["width"], case["heads"]

    def norm(x, spec):
        centred = x - x.mean(-1, keepdim=True)
        return (centred / torch.sqrt((centred * centred).mean(-1, keepdim=True) + 1e-5) * w[spec.tensors["weight"]]
                + w[spec.tensors["bias"]])

    table, rows = w[plan.embedding.tensors["weight"]], []
    for tokens in _tokens(case, seed):
        T = len(tokens)
        x = table[torch.tensor(tokens, device=DEVICE)] + w[plan.position.tensors["weight"]][:T]
        for i in range(case["n_layer"]):
            n1, mix, n2, ff = (names[i, p] for p in ("n1", "mix", "n2", "ff"))
            qkv = norm(x, n1) @ w[mix.tensors["qkv_weight"]].T + w[mix.tensors["qkv_bias"]]
            q, k, v = (y.reshape(T, H, D // H) for y in qkv.split(D, -1))
            o = _attend(q, k, v, (D // H) ** -0.5, 0).reshape(T, D)
            x = x + o @ w[mix.tensors["out_weight"]].T + w[mix.tensors["out_bias"]]
            up = _gelu_new(norm(x, n2) @ w[ff.tensors["up_weight"]].T + w[ff.tensors["up_bias"]])
            x = x + up @ w[ff.tensors["down_weight"]].T + w[ff.tensors["down_bias"]]
        rows.append(norm(x[-1:], plan.final_norm))
    return {"logits": torch.cat(rows) @ table.T, "pages": [None] * case["n_layer"]}


def exact(case, seed):
    if case["kind"] == "gpt2":
        return _exact_gpt2(case, seed)
    role, spec = _spec(case)
    w = _tensors(case, build_part(role, spec).tensor_specs(), seed)
    rows, lengths = [r.double() for r in _rows(case, seed)], _lengths(case)
    kind = case["kind"]
    if kind == "experts":
        return {"out": _exact_experts(case, w, torch.cat(rows))}
    w = {n: t.double() for n, t in w.items()}
    if kind == "ffn":
        hidden = _gelu_new(torch.cat(rows) @ w["up_weight"].T + w["up_bias"])
        return {"out": hidden @ w["down_weight"].T + w["down_bias"]}
    if kind in ("differential", "sink", "latent"):
        layer = {"differential": _exact_differential, "sink": _exact_sink, "latent": _exact_latent}[kind]
        return {"out": torch.cat([layer(case, w, h, before) for h, (before, _) in zip(rows, lengths)]), "kept": None}
    layer = {"delta": _exact_delta, "state_space": _exact_state_space, "matrix_lstm": _exact_matrix_lstm,
             "selective": _exact_selective}[kind]
    found = [layer(case, w, h) for h in rows]
    kept = torch.stack([k for _, k in found])
    # slots in the order in which a new cache hands them out (0, 1, ...), each padded to whole 16-byte pieces
    kept = torch.nn.functional.pad(kept, (0, build_part(role, spec).cache_spec().n_values - kept.shape[1]))
    return {"out": torch.cat([y for y, _ in found]), "kept": kept}
