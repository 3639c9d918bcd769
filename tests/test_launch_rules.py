"""What the host decides about a launch, and what every kernel's source has to keep, without a GPU."""

import re
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from libmir_b200 import KernelError, kernels


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


def kernels_of(source):
    """(name, body) of every kernel in a CUDA source, comments left out."""
    source = re.sub(r"//[^\n]*", "", source)
    for match in re.finditer(r"\b__global__\b", source):
        opened = source.index("{", match.end())
        if ";" in source[match.end():opened]:
            continue                                             # a declaration
        depth, at = 1, opened + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(source[at], 0)
            at += 1
        head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", source[match.end():opened])
        yield re.search(r"(\w+)\s*\(", head).group(1), source[opened + 1:at - 1]


def leaves_before_it_waits(body):
    """Whether some return of a kernel is not behind a wait that every thread coming there has been through: one in the same
    block or in a block around it, under no condition of its own."""
    blocks, waited = [False], [False]                            # of each open block: a function of its own; waited in it
    token = re.compile(r"\{|\}|grid_dependency_wait\(\)|\breturn\b")
    for match in token.finditer(body):
        statement = re.split(r"[;{}]", body[:match.start()])[-1]
        if match.group() == "{":
            blocks.append(blocks[-1] or re.search(r"\]\s*\([^()]*\)\s*(mutable\s*)?(->\s*\w+\s*)?$", statement) is not None)
            waited.append(waited[-1])
        elif match.group() == "}":
            blocks.pop()
            waited.pop()
        elif match.group() == "return":
            if not blocks[-1] and not waited[-1]:
                return True
        elif not re.search(r"\b(if|else|for|while)\b", statement):
            waited[-1] = True
    return False


def test_kernels_wait_for_the_one_in_front_on_every_way_out():
    """A kernel that is over before the one in front of it lets the next kernel run beside that one.  So every kernel that may be
    released early waits, also where it has nothing to do; only what is always launched plainly need not."""
    plain = {"cast_kernel", "random_normal_kernel", "paged_attention_mixed_kernel", "mixed_row_sums_kernel", "mixed_weights_kernel",
             "mixed_values_kernel", "mixed_row_sums_tc_kernel", "mixed_weights_tc_kernel", "mixed_values_tc_kernel"}
    folder = Path(kernels.__file__).parent.parent / "csrc"
    sources = {path.name: path.read_text() for path in sorted(folder.glob("*.cu*"))}
    found = [(file, name, body) for file, source in sources.items() for name, body in kernels_of(source)]
    assert len(found) > 60
    launched_plainly = {re.sub(r"<.*", "", name) for source in sources.values() for name in re.findall(r"(\w+(?:<[\w, ]*>)?)<<<", source)}
    assert launched_plainly - {"kernel"} <= plain                # ("kernel": the macro for what writes weights)
    for file, name, body in found:
        if name in plain:
            assert "grid_launch_dependents" not in body, (file, name)
            continue
        assert "grid_dependency_wait()" in body, (file, name)
        assert not leaves_before_it_waits(body), (file, name)


def test_the_check_of_waits_sees_a_way_out_without_one():
    wait = "mir::grid_dependency_wait();"
    fine = ("int a = 0; " + wait + " if (a) return;", "if (a) { " + wait + " return; }", "auto f = [&](int x) { return x; }; " + wait,
            "auto f = [&](int x) -> int { if (x) { return 1; } return x; }; " + wait, "if (!a) " + wait + " if (a) " + wait)
    wrong = ("if (a) return; " + wait, "if (a) { b(); return; } " + wait, "if (a) " + wait + " if (b) return; " + wait,
             "if (a) { " + wait + " } if (b) return;", "for (;;) { " + wait + " } return;")
    assert not any(leaves_before_it_waits(body) for body in fine)
    assert all(leaves_before_it_waits(body) for body in wrong)


def test_a_weight_streams_ring_is_the_one_asked_for():
    lib = kernels.library("bf16")
    try:
        for forced in (72, 108, 40, 0):
            assert lib.mir_gemm_tc_stream_set_splits(0, forced, 0) == 0
            assert [lib.mir_gemm_tc_stream_ring(ctas) for ctas in (1, 222, 223, 10000)] == \
                ([forced * 1024] * 4 if forced else [108 * 1024] * 2 + [72 * 1024] * 2)
        assert lib.mir_gemm_tc_stream_set_splits(0, 201, 0) != 0 and lib.mir_gemm_tc_stream_set_splits(0, 31, 0) != 0
    finally:
        lib.mir_gemm_tc_stream_set_splits(0, 0, 0)


@pytest.mark.parametrize("tiles, splits", [(1, 8), (48, 8), (49, 4), (50, 4), (55, 4), (100, 4), (104, 4), (105, 2), (192, 2), (193, 2), (222, 2),
                                           (223, 1), (1000, 1)])
@pytest.mark.parametrize("swiglu", [0, 1])
def test_weight_streams_are_cut_as_far_as_whole_clusters_fit_at_once(tiles, splits, swiglu):
    """384 blocks in clusters of eight, 416 in clusters of four, 444 in clusters of two; a block has four steps of 64 or more."""
    lib, width = kernels.library("bf16"), 64 if swiglu else 128
    for n in (tiles * width, tiles * width - width + 1):
        assert lib.mir_gemm_tc_stream_splits(n, 4096, swiglu, 1) == splits
        assert lib.mir_gemm_tc_stream_splits(n, 511, swiglu, 1) == min(splits, 2)
        assert lib.mir_gemm_tc_stream_splits(n, 448, swiglu, 1) == 1
    if tiles % 2 == 0:
        assert lib.mir_gemm_tc_stream_splits(tiles // 2 * width, 4096, swiglu, 2) == splits


@pytest.mark.parametrize("block, pinned, device, fits", [(8, 8, 8, True), (8, 8, 20, True), (8, 7, 20, False), (8, 20, 7, False)])
def test_an_upload_stays_within_its_buffers(recorder, block, pinned, device, fits):
    event = SimpleNamespace(cuda_event=0)
    buffers = torch.zeros(pinned, dtype=torch.int32), np.zeros(block, np.int32), torch.zeros(device, dtype=torch.int32)
    if fits:
        kernels.upload(event, *buffers)
        assert recorder.last("mir_upload")[3] == 4 * block
        return
    with pytest.raises(KernelError, match="upload"):
        kernels.upload(event, *buffers)
    assert not recorder.calls


@pytest.mark.parametrize("block", [np.zeros(4, np.int64), np.zeros(16, np.int32)[::2]])
def test_an_upload_takes_words_that_lie_side_by_side(recorder, block):
    with pytest.raises(KernelError, match="upload"):
        kernels.upload(SimpleNamespace(cuda_event=0), torch.zeros(64, dtype=torch.int32), block, torch.zeros(64, dtype=torch.int32))
    assert not recorder.calls
