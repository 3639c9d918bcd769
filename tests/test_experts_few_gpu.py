"""Routed experts of a step of few tokens: the one kernel that routes, orders and gathers against the three kernels it stands
for, bit by bit, and the streaming grouped products against 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def alloc(shape, kind):
    return torch.zeros(shape, dtype=kind, device="cuda")


# tokens around a warp row of the kernel and a tile of 16 pairs; experts ranked (up to 64) and searched for, with and
# without identity experts; every pair of one expert; widths that are no multiple of a 64-wide step, inner sizes that are no
# multiple of a tile of 64 or 128 columns
SIZES = [(1, 64, 64, 6, 8, 4, 2048, 1024), (3, 64, 56, 6, 8, 4, 512, 264), (16, 64, 64, 6, 8, 4, 1024, 512),
         (15, 6, 4, 2, 1, 1, 72, 40), (7, 200, 200, 5, 40, 7, 136, 72), (16, 2, 2, 1, 1, 1, 64, 8), (5, 600, 592, 4, 1, 1, 64, 136)]


@pytest.mark.parametrize("score, group_score", [("sigmoid", "top2"), ("softmax", "max")])
@pytest.mark.parametrize("tokens, experts, real, top, groups, keep, width, inter", SIZES)
def test_few_tokens_through_their_experts(tokens, experts, real, top, groups, keep, width, inter, score, group_score):
    from libmir_b200 import kernels
    generator = torch.Generator().manual_seed(tokens * 1000 + experts)
    bf16 = torch.bfloat16
    h = torch.randn(tokens, width + 8, generator=generator).to(bf16)[:, :width]
    logits = torch.randn(tokens, experts + 3, generator=generator)
    correction = torch.randn(experts, generator=generator) if score == "sigmoid" else None
    if experts == 2:
        logits[:, 0] += 50.0                                               # expert 1 gets no token
    both = (torch.randn(2 * real, inter, width, generator=generator) / width ** 0.5).to(bf16)
    w_down = (torch.randn(real, width, inter, generator=generator) / inter ** 0.5).to(bf16)
    h_d, logits_d = torch.zeros(tokens, width + 8, dtype=bf16, device="cuda")[:, :width].copy_(h), logits.cuda()
    correction_d = None if correction is None else correction.cuda()
    assert kernels.moe_plan_few_takes(bf16, tokens, width, inter, experts, real, top, groups)
    outputs = []
    for few in (False, True):
        ids, weights, gate = alloc((tokens, top), torch.int32), alloc((tokens, top), torch.float32), alloc((tokens,), torch.float32)
        if few:
            found = kernels.moe_plan_few(h_d, logits_d, correction_d, True, ids, weights, gate, experts, real, top, groups, keep,
                                         2.5, alloc, score=score, group_score=group_score)
        else:
            kernels.moe_route(logits_d, correction_d, True, ids, weights, gate, experts, top, groups, keep, 2.5, score=score,
                              group_score=group_score)
            found = kernels.moe_sort(ids, real, alloc, 8)
        outputs.append((ids, weights, gate, found.order, found.offsets))
    for one, other in zip(*outputs):
        assert torch.equal(one, other)
    ids, placed = outputs[0][0].cpu(), int(found.offsets[real])
    order, tiles = found.order.cpu()[:placed], found.tiles.cpu()[:2 * int(found.tile_count)].reshape(-1, 2)
    assert torch.equal(found.rows.cpu()[:placed], h[order.long() // top])
    counts = torch.bincount(ids.reshape(-1).long(), minlength=experts)[:real]
    assert tiles[:, 0].tolist() == counts.nonzero().reshape(-1).tolist()   # one tile for every expert that has a pair
    assert tiles[:, 1].tolist() == found.offsets.cpu()[:-1][counts > 0].tolist()

    both_d, w_down_d = both.cuda(), w_down.cuda()
    hidden, pair_rows = alloc((tokens * top, inter), bf16), alloc((tokens * top, width), torch.float32)
    kernels.moe_gate_up(h_d, found, top, both_d[:real], both_d[real:], hidden, alloc)
    kernels.moe_down(hidden, found, w_down_d, pair_rows)
    pair_rows, hidden = pair_rows.cpu().double(), hidden.cpu().double()
    for place, pair in enumerate(order.tolist()):
        e, x = int(ids.reshape(-1)[pair]), h[pair // top].double()
        g = both[e].double() @ x
        want = g * torch.sigmoid(g) * (both[real + e].double() @ x)
        # stored in 8 bits of mantissa (2^-9 of each value); the 32-bit sums and the exponential are far below that
        assert (hidden[place] - want).abs().max() <= 2 ** -8 * want.abs().max()
        want = w_down[e].double() @ hidden[place]
        # sums of `inter` products in 32 bits: each partial sum off by at most 2^-24 of the sum of the products' sizes
        bound = inter * 2 ** -24 * (w_down[e].double().abs() @ hidden[place].abs()) + 1e-30
        assert ((pair_rows[pair] - want).abs() <= bound).all()
    assert kernels.tensor_core_linear_error() == 0


def test_experts_behind_kernels_that_still_run():
    """The tokens' rows and the router's logits come from products that are still running when the next kernels of a captured
    step are released, and the down product asks for weights by lists that the plan left a kernel before: every replay with
    other tokens leaves what the same kernels leave when each starts behind the end of the one in front."""
    from libmir_b200 import kernels
    generator = torch.Generator(device="cuda").manual_seed(1)
    make = lambda *shape: (torch.randn(*shape, generator=generator, device="cuda") * 0.05).to(torch.bfloat16)
    tokens, width, deep, experts, top, inter = 3, 512, 65536, 64, 6, 256
    weight, router, x = make(width, deep), make(experts, width), make(tokens, deep)
    both, w_down = make(2 * experts, inter, width), make(experts, width, inter)

    def step(buffers):
        h, logits, ids, weights, hidden, pair_rows = buffers
        kernels.linear(x, weight, h)
        kernels.linear(h, router, logits)
        found = kernels.moe_plan_few(h, logits, None, False, ids, weights, None, experts, experts, top, 8, 4, 1.0, alloc)
        kernels.moe_gate_up(h, found, top, both[:experts], both[experts:], hidden, alloc)
        kernels.moe_down(hidden, found, w_down, pair_rows)
        return found

    buffers, others = ([alloc((tokens, width), torch.bfloat16), alloc((tokens, experts), torch.float32),
                        alloc((tokens, top), torch.int32), alloc((tokens, top), torch.float32),
                        alloc((tokens * top, inter), torch.bfloat16), alloc((tokens * top, width), torch.float32)] for _ in range(2))
    step(buffers)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        found = step(buffers)
    chosen = set()
    for _ in range(6):
        x.copy_(make(tokens, deep))
        graph.replay()
        torch.cuda.synchronize()
        kernels.set_programmatic_launch(0)
        try:
            plain = step(others)
        finally:
            kernels.set_programmatic_launch(1)
        for one, other in zip(buffers, others):
            assert torch.equal(one, other)
        assert torch.equal(found.order, plain.order) and torch.equal(found.rows, buffers[0][found.order.long() // top])
        chosen.add(tuple(buffers[2].flatten().tolist()))
    assert len(chosen) == 6                                                # another routing every time
    assert kernels.tensor_core_linear_error() == 0
