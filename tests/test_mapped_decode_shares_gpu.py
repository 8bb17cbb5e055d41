"""Single tokens over cached rows, pages shared out over blocks, against the kernel that takes any step: positions at the edges
of pages and shares, empty shares, runs of pages before a window's, more heads than warps, rows of every alignment."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HELD = [1, 32, 33, 64, 65, 2047, 2048, 2049, 4200]


@pytest.mark.parametrize("pages", [70, 66])                    # wider than the longest sequence, and as wide as it
@pytest.mark.parametrize("H,G,maps,dim,vdim,dtype,options", [
    (8, 2, 1, 128, 128, torch.bfloat16, {"sink": True}),
    (4, 4, 2, 64, 128, torch.bfloat16, {"window": 300, "lam": 0.4}),
    (6, 1, 1, 96, 96, torch.float32, {}),
    (3, 3, 1, 17, 23, torch.float32, {"window": 130, "keep": 70}),
    (16, 1, 2, 32, 64, torch.bfloat16, {"chunk": 1000, "lam": 0.4}),
    (4, 2, 1, 64, 64, torch.bfloat16, {"shared": True, "window": 64, "keep": 1}),
])
def test_shares_of_single_tokens(H, G, maps, dim, vdim, dtype, options, pages):
    """Both kernels sum float32 products; a sum of n weights is off by some n 2^-24, its exponentials by 2^-22 of arguments up
    to 16: 1e-5 of the rows' rms in float32; in bfloat16 two sums on either side of a tie are a unit in the last place apart,
    twice the 2^-8 of a value that one rounding is off by."""
    from math_utils_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *shape: torch.randn(shape, generator=gen, device="cuda").to(dtype)
    ints = lambda x: torch.as_tensor(np.asarray(x, dtype=np.int32)).cuda()
    need = [-(-n // 64) for n in HELD]
    order, at = np.random.default_rng(2).permutation(sum(need)), 0
    table = np.zeros((len(HELD), pages), dtype=np.int32)
    for s, n in enumerate(need):
        table[s, :n] = order[at:at + n]
        at += n
    rows = rand(sum(need), 64, G * (maps * dim + (0 if options.get("shared") else vdim)))
    q, T = rand(len(HELD), H * maps * dim), len(HELD)
    rest = {k: v for k, v in options.items() if k != "window"}
    # the parts' room keeps what a call before left: nothing of an empty share may come back
    out = [torch.zeros((T, H * vdim), device="cuda", dtype=dtype) for _ in range(3)]
    for o, single, x in ((out[0], True, q * float("nan")), (out[1], True, q), (out[2], False, q)):
        ops.mapped_attention(x, rows, ints(table), 64, ints([n - 1 for n in HELD]), ints(range(T)), H, G, maps, dim, vdim,
                             dim ** -0.5, options.get("window", 0), o, single_tokens=single, tensor_cores=False, **rest)
    got, want = out[1].double(), out[2].double()
    off = (got - want).abs() / (want.abs() + want.square().mean(1, keepdim=True).sqrt())
    assert out[0].isnan().all() and float(off.max()) < (1e-5 if dtype == torch.float32 else 2.0 ** -7)
