"""32-bit products at work on two streams at once: launches share nothing in device memory, so the results have the bits of
the same launches one after the other."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from math_utils_b200.csrc import ops
    return ops


def _rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda") * scale


def _both(ops, left, right, repeats):
    """(left, right) outputs of products on two streams at once, ``repeats`` times over."""
    main, side = torch.cuda.current_stream(), torch.cuda.Stream()
    side.wait_stream(main)
    outs = []
    for _ in range(repeats):
        with torch.cuda.stream(side):
            b = ops.gemm_f32_tc(*right, cut=1)
        outs.append((ops.gemm_f32_tc(*left, cut=1), b))
    main.wait_stream(side)
    return outs


# two to eight runs of k, tiles of few and of all rows
@pytest.mark.parametrize("m,left,right", [(8, (3072, 2048), (4384, 2048)), (1, (2048, 8192), (1000, 1100)), (150, (700, 4096), (768, 3072))])
def test_cut_products_on_two_streams(m, left, right):
    ops = _ops()
    left, right = ((_rand((m, k), 1 + i), _rand((n, k), 3 + i, k ** -0.5)) for i, (n, k) in enumerate((left, right)))
    want = tuple(ops.gemm_f32_tc(*p, cut=1) for p in (left, right))
    for p, w in zip((left, right), want):
        assert torch.equal(ops.gemm_f32_tc(*p, cut=0), w)
    for got in _both(ops, left, right, 50):
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = _both(ops, left, right, 4)
    for _ in range(10):
        graph.replay()
    for got in outs:
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    ops.check_status()


def _model():
    """One layer of width 2,048 whose two mixers run side by side, beside the feed-forward."""
    from math_utils_b200.config.pelenex import PelenexConfig
    from math_utils_b200.engine.assemble import collect_tensor_specs
    from math_utils_b200.engine.model import DecoderModel
    from math_utils_b200.engine.runtime import Runtime
    from math_utils_b200.parts.base import FreeSize
    both = {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 512, "keep_first": 4}},
            "right": {"heads": 16, "dim": 128, "vdim": 128, "tau": 8.0}}
    plan = PelenexConfig.from_json({"architecture": "Pelenex", "vocab": 509, "width": 2048, "norm": {"eps": 1e-5, "groups": 4},
                                    "logit_softcap": 30.0,
                                    "layers": [{"type": "parallel", "mixer": both, "mlp": {"kind": "dense", "ff": 4096}}]}).plan()
    tensors = {}
    for i, s in enumerate(collect_tensor_specs(plan)):
        shape = [n.default if isinstance(n, FreeSize) else int(n) for n in s.shape]
        shape = tuple(reversed(shape)) if s.transpose else tuple(shape)
        tensors[s.name] = _rand(shape, i, shape[-1] ** -0.5) + (1.0 if s.init == "norm_weight" else 0.0)
    return DecoderModel(plan, tensors, Runtime.create("float32", "cuda:0"))


def test_float32_steps_with_members_side_by_side(monkeypatch):
    """Eager steps of 1, 8 and 32 single tokens, and the replayed step, of a layer that runs its members on streams of their
    own: the bits of the members one after the other."""
    from math_utils_b200.engine.batch import StepEntry
    from math_utils_b200.engine.decode_session import DecodeSession
    from math_utils_b200.parts.block import ParallelPreNormBlock
    from math_utils_b200.parts.parallel import ParallelMixers
    from math_utils_b200.sampling import SamplingParams
    model, ops = _model(), _ops()
    rng = np.random.default_rng(5)
    for n in (1, 8, 32):
        prompts = [rng.integers(0, 509, 3).tolist() for _ in range(n)]

        def steps(tokens_side_by_side, replayed):
            monkeypatch.setattr(ParallelMixers, "SIDE_BY_SIDE_TOKENS", tokens_side_by_side)
            monkeypatch.setattr(ParallelPreNormBlock, "SIDE_BY_SIDE_TOKENS", tokens_side_by_side)
            cache = model.new_cache(max_tokens=64 * n, n_slots=n)
            slots = [cache.acquire() for _ in range(n)]
            model.step(cache, [StepEntry(s, p, ()) for s, p in zip(slots, prompts)])
            if not replayed:
                return [model.step(cache, [StepEntry(s, [(7 * i + s) % 509], [0]) for s in slots]).clone() for i in range(12)]
            for s in slots:
                cache.reserve(s, 1)
            session = DecodeSession(model, cache, slots, SamplingParams(temperature=0.0), list(range(n)))
            session.sync_block_tables()
            session.feed([s % 509 for s in slots], [3] * n)
            session.capture()
            out = []
            for _ in range(12):                       # the same step over and over
                session.feed([s % 509 for s in slots], [3] * n)
                session.launch()
                out.append(session.logits.clone())
            return out

        for replayed in (False, True):
            alone, beside = steps(0, replayed), steps(32, replayed)
            assert all(torch.equal(a, b) for a, b in zip(alone, beside)), (n, replayed)
    ops.check_status()


def test_first_product_of_a_process_inside_a_capture():
    """A float32 product is the same kernel whatever the process has run before: recorded as its first launch, then eager."""
    code = """
import torch
from math_utils_b200.csrc import ops
g = torch.Generator(device="cuda").manual_seed(1)
a, w = torch.randn((40, 768), generator=g, device="cuda"), torch.randn((300, 768), generator=g, device="cuda")
out = torch.zeros((40, 300), device="cuda")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    ops.linear(a, w, out=out)
for _ in range(3):
    out.zero_()
    graph.replay()
    eager = ops.linear(a, w)
    assert torch.equal(out, eager) and torch.equal(eager, ops.gemm_f32_tc(a, w))
x, y = a.bfloat16().repeat(4, 1), w.bfloat16()
assert torch.equal(ops.linear(x, y), ops.gemm_tc(x, y))
word = ops.status_word(a.device)
assert word.data_ptr() == ops.status_word("cuda:0").data_ptr() and int(word) == 0
word.fill_(2)
try:
    ops.check_status()
    raise SystemExit("no error for a wait that ran out")
except ops.KernelError as e:
    assert "tensor cores" in str(e)
ops.check_status()
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    proc = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout + proc.stderr
