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
