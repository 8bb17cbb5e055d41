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
