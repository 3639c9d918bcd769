"""Steps whose kernels start beside the one in front (the default) against the same steps with every kernel launched behind the
end of the one in front, bit by bit; and repeated captured steps against steps that take the whole host path."""

from importlib import import_module

import numpy as np
import pytest
import torch

from helpers import make_folder

pytestmark = pytest.mark.gpu


def model_of(tmp_path, design, name, dtype, pages=96):
    from libmir_b200 import CacheConfig, CudaConfig, Library, RuntimeConfig, SchedulerConfig
    configs = import_module(f"{design}_configs")
    config = configs.ALL[name]
    folder = tmp_path / f"{design}{name}{dtype}"
    if not folder.exists():
        folder = make_folder(folder, config, 3, dtype, 4.0) if design == "tiny" else configs.make_folder(folder, config, 3, dtype)
    runtime = RuntimeConfig(kv_cache=CacheConfig(block_size=configs.PAGE_SIZES[name], block_count=pages),
                            scheduler=SchedulerConfig(max_batch_requests=4), cuda=CudaConfig(decode_graphs=True), dtype=dtype)
    return Library(runtime).load(folder), config.get("vocab") or config["vocab_size"]


def served(model, vocab, seed):
    """Logits of prompts packed into a step, captured steps, a portion beside decoded tokens, and captured steps of all."""
    from libmir_b200 import StepEntry
    from libmir_b200.sampling import RequestSampler
    rng = np.random.default_rng(seed)
    ids = lambda n: rng.integers(0, vocab, size=n).tolist()
    samplers = [RequestSampler() for _ in range(3)]
    logits = []

    def step(entries, drawn=True):
        logits.append(model.step(entries, samplers[:sum(len(e.want) for e in entries)] if drawn else None).logits.clone())
    for name in "abc":
        model.admit(name)
    step([StepEntry("a", ids(137), [0, 136]), StepEntry("b", ids(70), [69])], False)
    for _ in range(6):
        step([StepEntry(name, ids(1), [0]) for name in "ab"])
    for count in (50, 21):
        step([StepEntry("a", ids(1), [0]), StepEntry("c", ids(count), [count - 1]), StepEntry("b", ids(1), [0])], False)
    for _ in range(6):
        step([StepEntry(name, ids(1), [0]) for name in "cab"])
    for name in "abc":
        model.release(name)
    return torch.cat(logits)


@pytest.mark.parametrize("design, name, dtype", [
    ("tiny", "E", "bfloat16"), ("tiny", "F", "bfloat16"), ("tiny", "C", "float32"), ("doderax", "W", "bfloat16"),
    ("doderax", "X", "float32"), ("zufotar", "A", "bfloat16"), ("zufotar", "D", "bfloat16"), ("dalesun", "C", "bfloat16"),
    ("gumazen", "A", "bfloat16"), ("gumazen", "D", "bfloat16"), ("pedotar", "D", "bfloat16"), ("biravik", "A", "bfloat16"),
    ("biravik", "D", "bfloat16"), ("biravik", "C", "float32")])
def test_early_starts_change_no_bit(tmp_path, design, name, dtype):
    from libmir_b200 import kernels
    outputs = []
    try:
        for mode in (0, 2, 1):
            kernels.set_programmatic_launch(mode)
            model, vocab = model_of(tmp_path, design, name, dtype)   # (captured steps keep the mode they were captured in)
            outputs += [served(model, vocab, 9) for _ in range(3)]
            model.unload()
    finally:
        kernels.set_programmatic_launch(1)
    assert torch.isfinite(outputs[0]).all()
    for other in outputs[1:]:
        assert torch.equal(outputs[0], other)


@pytest.mark.parametrize("design, name", [("tiny", "E"), ("tiny", "C"), ("doderax", "W"), ("doderax", "Z"), ("gumazen", "C"),
                                          ("pedotar", "A"), ("dalesun", "D"), ("biravik", "C")])
def test_repeated_steps_take_the_short_path_while_no_page_comes_or_goes(tmp_path, design, name):
    """One model takes the short path where it may, another never: equal bits and equal tables at every step, and the short path
    is taken just where the other's tables stay as they were uploaded last (windows, kept first keys, several groups, pairs of
    tokens): no page is taken for the step and none is given back behind it or behind the step before."""
    from libmir_b200 import StepEntry
    from libmir_b200.sampling import RequestSampler
    (quick, vocab), (whole, _) = (model_of(tmp_path, design, name, "bfloat16") for _ in range(2))
    rng = np.random.default_rng(4)
    samplers = [RequestSampler(), RequestSampler()]
    tables = lambda model: [[list(table) for table in model.runner.manager.live[r].tables] for r in "ab"]
    for r, count in (("a", 61), ("b", 30)):
        ids = rng.integers(0, vocab, size=count).tolist()
        for model in (quick, whole):
            model.admit(r)
            model.step([StepEntry(r, ids, [])])
    given_back = lambda every: sum(page < 0 for request in every for table in request for page in table)
    taken, last = [], None
    for step in range(80):
        entries = [StepEntry(r, [int(rng.integers(vocab))], [0]) for r in "ab"]
        whole.runner._again = None
        before, count = tables(whole), quick.runner.steps_again
        results = [model.step(entries, samplers).logits.clone() for model in (quick, whole)]
        taken.append(quick.runner.steps_again > count)
        assert torch.equal(*results), step
        assert tables(quick) == tables(whole), step
        after = tables(whole)
        assert taken[-1] == (step > 0 and before == after and given_back(before) == last), step
        last = given_back(before)
    assert whole.runner.steps_again == 0 and True in taken[1:]
    assert False in taken[1:]
    for model in (quick, whole):
        model.cache.check()
        model.unload()
