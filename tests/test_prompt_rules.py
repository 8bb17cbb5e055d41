"""Which form a prompt step takes, on the host: wide batches keep the forms whose time does not grow with all their tokens."""
import pytest

from math_utils_b200.config.base import PartSpec
from math_utils_b200.parts.base import build_part


# (heads, key and value entries, lengths, whether in chunks): the layer's time on the device, token by token and in chunks,
# is beside the rule; these are steps where one side is at least 4 % ahead, on either side of it
@pytest.mark.parametrize("heads,dim,lens,chunks", [
    (8, 128, [300], False), (8, 128, [512], True), (8, 128, [2000], True), (8, 128, [1000] * 4, True), (8, 128, [512] * 6, False),
    (8, 128, [512] * 16, False), (8, 128, [1000] * 8, False), (8, 128, [448] * 8, False), (8, 128, [1000] + [100] * 7, True),
    (4, 128, [512] * 16, False), (4, 128, [1000] * 8, True), (8, 64, [1000] * 8, True), (16, 64, [1000] * 16, False),
    (2, 64, [512] * 16, True), (8, 128, [1501, 517], True)])
def test_matrix_memory_in_chunks_by_load(heads, dim, lens, chunks):
    sizes = dict(hidden_size=512, n_heads=heads, dim=dim, vdim=dim, gate_cap=15.0, eps=1e-5)
    part = build_part("mixer", PartSpec("matrix_lstm", sizes, {}))
    assert part.in_chunks(max(lens), sum(lens)) == chunks


# (channels, longest, segments scanned twice, whether cut) at 16 state entries a channel
@pytest.mark.parametrize("inner,lens,cut", [
    (2048, [800], False), (2048, [1000], True), (2048, [700], False), (2048, [1000] * 3, False), (2048, [2000] * 3, True),
    (2048, [2000] * 4, False), (2048, [1000, 500, 250, 250], True), (2048, [1000, 83, 900], True), (256, [768] * 8, False),
    (256, [1000] * 8, True), (512, [700], True), (4096, [2000] * 2, False), (1000, [800] * 2, False), (512, [655], False)])
@pytest.mark.gpu
def test_selective_scan_cut_by_load(inner, lens, cut):
    from math_utils_b200.csrc import ops
    if ops.sm_count("cuda:0") != 148:
        pytest.skip("measured on 148 SMs")
    tokens, least = ops._selective_sizes()
    again = sum((n - 1) // tokens for n in lens)
    assert (ops.library().mu_selective_scan_segments(inner, 16, max(lens), again) > 1) == cut
