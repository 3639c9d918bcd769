"""What the host decides about a launch, and what every kernel's source has to keep, without a GPU."""

import pytest
import torch

from libmir_b200 import kernels


class Recorder:
    """Stands in for a native library: every call is written down and succeeds."""

    def __init__(self, **answers):
        self.calls, self.answers = [], answers

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return self.answers.get(name, 0)
        return call

    def last(self, name):
        return [args for called, args in self.calls if called == name][-1]


@pytest.fixture
def recorder(monkeypatch):
    made = Recorder(mir_moe_tile_slots=8)
    monkeypatch.setattr(kernels, "library", lambda name: made)
    monkeypatch.setattr(kernels, "_cuda", lambda *tensors: None)
    made.stream = 7
    monkeypatch.setattr(kernels, "_stream", lambda: made.stream)
    return made


def test_a_down_product_looks_ahead_only_behind_its_own_gate_up(recorder):
    """The lists of an order may be read ahead of the wait when moe_gate_up of that order went over the same stream before: not
    without it, not for another order, not on another stream."""
    tokens, top, experts, width, inter = 3, 2, 4, 16, 8
    alloc = lambda shape, kind: torch.zeros(shape, dtype=kind)
    weights = torch.zeros(3 * experts, inter, width, dtype=torch.bfloat16)
    h, hidden = torch.zeros(tokens, width, dtype=torch.bfloat16), torch.zeros(tokens * top, inter, dtype=torch.bfloat16)
    pair_rows = torch.zeros(tokens * top, width)

    def order():
        found = kernels.ExpertOrder(alloc, tokens * top, experts, 16)
        found.rows = torch.zeros(tokens * top, width, dtype=torch.bfloat16)
        return found

    def looks_ahead(found):
        kernels.moe_down(hidden, found, weights[2 * experts:].view(experts, width, inter), pair_rows)
        return recorder.last("mir_gemm_tc_stream_grouped_bf16")[-2]

    def gate_up(found):
        kernels.moe_gate_up(h, found, top, weights[:experts], weights[experts:2 * experts], hidden, alloc)
        assert recorder.last("mir_gemm_tc_stream_grouped_bf16")[-2] == 0

    first, second = order(), order()
    assert looks_ahead(first) == 0
    gate_up(first)
    assert looks_ahead(first) == 1
    assert looks_ahead(second) == 0
    recorder.stream = 9
    assert looks_ahead(first) == 0
    gate_up(second)
    assert looks_ahead(second) == 1 and looks_ahead(first) == 0


@pytest.mark.parametrize("rows, allowed, together", [(128, 201, True), (129, 201, False), (32, 33, True), (33, 33, True), (34, 33, False)])
def test_products_side_by_side_keep_to_the_rows_the_weight_stream_takes(recorder, monkeypatch, rows, allowed, together):
    """few_rows_max may be raised beyond the 128 rows of the streaming kernel: more rows go one product behind the other."""
    recorder.answers["mir_get_option"] = allowed                 # (an odd number: also few_rows_modes with the store epilogue)
    alone = []
    monkeypatch.setattr(kernels, "linear", lambda x, w, out, alloc=None: alone.append(x.shape))
    x, w = torch.zeros(4, rows, 16, dtype=torch.bfloat16), torch.zeros(4, 24, 16, dtype=torch.bfloat16)
    kernels.linear_side_by_side(x, w, torch.zeros(4, rows, 24, dtype=torch.bfloat16))
    streamed = [args for name, args in recorder.calls if name == "mir_gemm_tc_stream_side_by_side_bf16"]
    assert (len(streamed), len(alone)) == ((1, 0) if together else (0, 4))
