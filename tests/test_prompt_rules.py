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


@pytest.mark.parametrize("form,experts,width,inner,pairs,gathered", [
    ("gated_silu", 48, 768, 512, 1320, False), ("gated_silu", 48, 768, 512, 3000, False), ("gated_silu", 48, 768, 512, 6000, True),
    ("relu2", 48, 768, 512, 3000, True), ("gated_silu", 48, 1024, 704, 1800, True), ("gated_silu", 16, 512, 512, 3000, True),
    ("relu2", 64, 2048, 1408, 48, True), ("gated_silu", 16, 1024, 704, 300, False)])
def test_experts_rows_gathered_by_work(form, experts, width, inner, pairs, gathered):
    import torch
    names = {"router": "router", "up": "e{e}.up", "down": "e{e}.down", "gate": "e{e}.gate"}
    sizes = dict(hidden_size=width, inner_size=inner, n_experts=experts, top=1, score="sigmoid", expert_form=form)
    part = build_part("feed_forward", PartSpec("routed_experts", sizes, names))

    class Runtime:
        device, dtype = "cuda:0", torch.bfloat16

        class ops:
            moe_tile_rows, sm_count = staticmethod(lambda: 32), staticmethod(lambda device: 148)

    part.bind({t.name: torch.empty(t.shape, dtype=torch.bfloat16, device="meta") for t in part.tensor_specs()}, Runtime)
    assert (pairs >= part.gathered_pairs) == gathered


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
