"""Kernels that have several forms, one of which is taken by the sizes of the call: both sides of every rule against plain torch
in 64 bits, exactly where the numbers are whole or only moved."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def ints(values):
    return torch.as_tensor(values, dtype=torch.int32).to("cuda")


def batch(counts, slots=None):
    """(row_of_token, query_starts, state_slots, positions) of portions that start their requests."""
    counts = list(counts)
    starts = np.concatenate([[0], np.cumsum(counts)])
    return (ints(np.repeat(np.arange(len(counts)), counts)), ints(starts), ints(range(len(counts)) if slots is None else slots),
            ints(np.concatenate([np.arange(n) for n in counts])))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,dim,rows", [(32, 64, 210), (16, 128, 230), (5, 20, 7)])
def test_what_the_delta_rule_needs_of_many_single_tokens(dtype, heads, dim, rows):
    """A step of many decoded tokens (one token a warp, however many there are) against the same tokens a few at a time and in a
    step that also brings a portion (eight tokens a warp): the same bits, and the same inputs kept."""
    from libmir_b200 import kernels
    torch.manual_seed(rows)
    width, decays = 3 * heads * dim, heads * dim
    make = lambda *shape: torch.randn(*shape, device="cuda")
    tokens = rows + 2500
    x, weight, beta_raw = make(tokens, width).to(dtype), make(width, 4).to(dtype), make(tokens, heads).to(dtype)
    decay_raw, bias, a_log = make(tokens, decays).to(dtype), make(decays), make(heads)
    tail0 = make(rows + 1, 3, width)

    def prepare(first, counts, slots, tail):
        n = sum(counts)
        row_of, starts, slots, positions = batch(counts, slots)
        made = [torch.full((n, w), float("nan"), device="cuda") for w in (width, heads, decays)]
        kernels.delta_rule_prepare(x[first:first + n], weight, tail, beta_raw[first:first + n], decay_raw[first:first + n], bias, a_log,
                                   row_of, starts, slots, positions, *made, heads, heads, dim, dim)
        return made
    tails = [tail0.clone() for _ in range(3)]
    whole = prepare(0, [1] * rows, range(rows), tails[0])
    pieces = [prepare(first, [1] * min(3, rows - first), range(first, min(first + 3, rows)), tails[1]) for first in range(0, rows, 3)]
    beside = prepare(0, [1] * rows + [2500], range(rows + 1), tails[2])
    for got, parts, other in zip(whole, zip(*pieces), beside):
        assert bool(torch.isfinite(got).all()) and torch.equal(got, torch.cat(parts)) and torch.equal(got, other[:rows])
    assert torch.equal(tails[0], tails[1]) and torch.equal(tails[0][:rows], tails[2][:rows])


ROUTERS = [(experts, top, groups, keep) for experts in (8, 32, 36, 64, 72, 96, 128, 200, 256, 288) for top in (1, 2, 4, 6, 8)
           for groups, keep in ((1, 1), (4, 2), (36, 5)) if experts % groups == 0 and top <= keep * (experts // groups) - experts // 16]


@pytest.mark.parametrize("experts,top,groups,keep", ROUTERS)
def test_experts_that_are_ranked_and_experts_that_are_searched(experts, top, groups, keep):
    """Scores with many equal ones (the lower expert comes first), masked experts among them; whole numbers are exact."""
    from libmir_b200 import kernels
    generator = torch.Generator().manual_seed(experts + top)
    tokens = 9
    logits = (torch.randint(-3, 4, (tokens, experts + 1), generator=generator) * 0.5).float()
    logits[:, :experts][torch.rand(tokens, experts, generator=generator) < 1 / 32] = -float("inf")
    ids, weights = torch.full((tokens, top), -1, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda")
    gate = torch.empty(tokens, device="cuda")
    kernels.moe_route(logits.cuda(), None, True, ids, weights, gate, experts, top, groups, keep, 1.5)
    score = torch.sigmoid(logits[:, :experts].double())
    for t in range(tokens):
        choice = score[t].clone()
        if keep < groups:
            per = choice.view(groups, -1)
            best = per.topk(min(2, per.shape[1]), dim=1).values.sum(1)
            kept = sorted(range(groups), key=lambda g: (-float(best[g].float()), g))[:keep]
            dropped = [g for g in range(groups) if g not in kept]
            choice.view(groups, -1)[dropped] = -1.0
        want = sorted(range(experts), key=lambda e: (-float(choice[e].float()), e))[:top]
        assert ids[t].tolist() == want, (t, ids[t].tolist(), want)
        chosen = score[t][want]
        assert torch.allclose(weights[t].double().cpu(), chosen / chosen.sum() * 1.5, rtol=1e-5)
    assert torch.allclose(gate.double().cpu(), torch.sigmoid(logits[:, experts].double()), rtol=1e-5)


@pytest.mark.parametrize("pairs,experts", [(416, 64), (417, 64), (1023, 200), (1024, 200), (1023, 300), (4095, 300), (4096, 300),
                                           (700, 1024), (20000, 1), (3001, 3), (900, 148), (900, 149), (17, 1024)])
def test_pairs_by_expert_on_both_sides_of_the_rules(pairs, experts):
    """One CTA (416 pairs at most), 256 and 1,024 threads an expert; every ninth pair is in no list; more than 1,024 tiles of one expert."""
    from libmir_b200 import kernels
    generator = torch.Generator().manual_seed(pairs)
    ids = torch.randint(0, experts, (pairs,), generator=generator)
    ids[8::9] = experts + 1
    alloc = lambda shape, kind: torch.full(shape, -7, dtype=kind, device="cuda")
    found = kernels.moe_sort(ids.view(pairs, 1).int().cuda(), experts, alloc, 8)
    held = ids < experts
    want = torch.argsort(torch.where(held, ids, experts), stable=True)[:int(held.sum())].tolist()
    counts = torch.bincount(ids[held], minlength=experts).tolist()
    offsets = np.concatenate([[0], np.cumsum(counts)]).tolist()
    tiles = [[e, offsets[e] + first] for e in range(experts) for first in range(0, counts[e], 8)]
    assert found.order.cpu().tolist()[:len(want)] == want and found.offsets.cpu().tolist() == offsets
    assert int(found.tile_count.cpu()) == len(tiles) and found.tiles.cpu().view(-1, 2).tolist()[:len(tiles)] == tiles


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("dim,value_dim", [(64, 128), (64, 129), (192, 192), (256, 250), (576, 640), (24, 320)])
def test_reference_attention_of_every_value_width(dtype, tol, dim, value_dim):
    """Value heads that a lane holds in four places or in twenty; keys that fill no run of them."""
    from libmir_b200 import kernels
    generator = torch.Generator().manual_seed(value_dim)
    lengths, heads, kv_heads, page = [1, 2, 17, 33, 71], 4, 2, 8
    pages = [-(-n // page) for n in lengths]
    order = torch.randperm(sum(pages) + 1, generator=generator).tolist()
    k_pool = torch.full(((sum(pages) + 1) * page, kv_heads, dim), 50.0, dtype=dtype)
    v_pool = torch.full(((sum(pages) + 1) * page, kv_heads, value_dim), float("nan"), dtype=dtype)
    table = torch.full((len(lengths), max(pages)), -1, dtype=torch.int32)
    q = (torch.randn(len(lengths), heads, dim, generator=generator)).to(dtype)
    want, cursor = [], 0
    for r, n in enumerate(lengths):
        k = (torch.randn(n, kv_heads, dim, generator=generator) * 0.3).to(dtype)
        v = torch.randn(n, kv_heads, value_dim, generator=generator).to(dtype)
        for block in range(pages[r]):
            at = order[cursor] * page
            cursor += 1
            piece = slice(block * page, min((block + 1) * page, n))
            k_pool[at:at + piece.stop - piece.start], v_pool[at:at + piece.stop - piece.start] = k[piece], v[piece]
            table[r, block] = at // page
        for h in range(heads):
            weights = torch.softmax(q[r, h].double() @ k[:, h // 2].double().T * 0.2, -1)
            want.append(weights @ v[:, h // 2].double())
    out = torch.full((len(lengths), heads * value_dim), float("nan"), dtype=dtype, device="cuda")
    kernels.paged_attention_generic(q.flatten(1).cuda(), out, k_pool.cuda(), v_pool.cuda(), table.cuda(), ints(range(len(lengths))),
                                    ints([n - 1 for n in lengths]), page, heads, kv_heads, dim, 0.2, None, value_dim=value_dim)
    want = torch.stack(want).view(len(lengths), -1)
    error = (out.double().cpu() - want).abs().max()
    assert float(error) <= tol * float(want.abs().max()), float(error)


def rounded(x):
    return x.astype(np.float32).astype(np.float64)


def sum_of_squares(row, threads):
    """A row's sum of squares as the norms form it: quads dealt out to `threads` threads, a thread's chain of multiply-adds, then
    neighbours' sums by halves of a warp and of the warps (each step rounded to 32 bits)."""
    quads = np.zeros((-(-len(row) // 4 // threads) * threads, 4))
    quads.reshape(-1)[:len(row)] = row
    total = np.zeros(threads)
    for quad in quads.reshape(-1, threads, 4):
        for i in (3, 2, 1, 0):
            total = rounded(quad[:, i] * quad[:, i] + total)
    sums = total.reshape(-1, 32)
    for _ in range(2):
        for step in (16, 8, 4, 2, 1):
            sums = rounded(sums + sums[:, np.arange(32) ^ step])
        sums = np.concatenate([sums[:, 0], np.zeros(32 - len(sums))])[None, :] if _ == 0 else sums
    return sums[0, 0]


@pytest.mark.parametrize("hidden", [100, 1020, 1024, 2560, 4096, 4100, 5120, 8192, 8196, 16384, 16388, 20480])
def test_rms_norm_sums_in_one_order_whatever_holds_the_row(hidden):
    """Rows in registers and rows read twice: bit for bit the sums of 256 threads (128 below 1,024 columns)."""
    from libmir_b200 import kernels
    torch.manual_seed(hidden)
    x, weight = torch.randn(5, hidden), torch.rand(hidden) + 0.5
    sums = torch.tensor([sum_of_squares(row.double().numpy(), 256 if hidden >= 1024 else 128) for row in x], dtype=torch.float32)
    mean = sums.numpy() / np.float32(hidden) + np.float32(1e-5)
    inverse = torch.rsqrt(torch.from_numpy(mean).cuda())
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.empty(5, hidden, dtype=dtype, device="cuda")
        kernels.rms_norm(x.cuda(), weight.cuda(), 1e-5, out)
        assert torch.equal(out, (x.cuda() * inverse[:, None] * weight.cuda()).to(dtype))
    rows = ints([4, 0])
    out = torch.empty(2, hidden, device="cuda")
    kernels.rms_norm(x.cuda(), weight.cuda(), 1e-5, out, rows)
    assert torch.equal(out, (x.cuda() * inverse[:, None] * weight.cuda())[rows.long()])


@pytest.mark.parametrize("hidden", [100, 2048, 2052, 4100, 8192, 16384, 16388])
def test_two_norms_of_the_same_rows(hidden):
    from libmir_b200 import kernels
    torch.manual_seed(hidden)
    x, a, b = torch.randn(3, hidden), torch.rand(hidden) + 0.5, torch.rand(hidden) + 0.5
    normed = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5)
    for dtype, tol in ((torch.float32, 2e-6), (torch.bfloat16, 2 ** -8)):
        out_a, out_b = (torch.empty(3, hidden, dtype=dtype, device="cuda") for _ in range(2))
        kernels.rms_norm_pair(x.cuda(), a.cuda(), b.cuda(), 1e-5, out_a, out_b)
        for out, weight in ((out_a, a), (out_b, b)):
            want = normed * weight.double()
            assert bool(((out.double().cpu() - want).abs() <= tol * want.abs() + 1e-7).all())


@pytest.mark.parametrize("hidden", [36, 512, 2048, 2052, 2560, 4096, 4100, 5124, 8192, 8196, 16384, 16388])
@pytest.mark.parametrize("count", [1, 2, 3, 4])
def test_normed_branches_of_every_count_and_width(count, hidden):
    """Rows in registers and rows read twice; the roundings are those of the sums, a product and the addition."""
    from libmir_b200 import kernels
    torch.manual_seed(hidden + count)
    branches = [torch.randn(3, hidden) * (b + 1) for b in range(count)]
    weights = [torch.rand(hidden) + 0.5 for _ in range(count)]
    residual = torch.randn(3, hidden)
    want = residual.double()
    for branch, weight in zip(branches, weights):
        want = want + 0.7 * branch.double() * torch.rsqrt((branch.double() ** 2).mean(-1, keepdim=True) + 1e-5) * weight.double()
    got, half = residual.cuda(), torch.empty(3, hidden, dtype=torch.bfloat16, device="cuda")
    kernels.add_normed_branches([b.cuda() for b in branches], [w.cuda() for w in weights], got, 1e-5, 0.7, half)
    bound = 2e-6 * (1 + sum(b.abs().max() for b in branches))
    assert float((got.double().cpu() - want).abs().max()) <= float(bound)
    assert torch.equal(half, got.bfloat16())


@pytest.mark.parametrize("tokens", [1, 147, 148, 149])
@pytest.mark.parametrize("width", [7, 2048, 4096, 4100])
def test_addition_of_a_layer_norm_with_weights_asked_for_early_and_late(tokens, width):
    from libmir_b200 import kernels
    torch.manual_seed(tokens + width)
    x, y, rows = torch.randn(tokens, width), torch.randn(tokens, width) * 2 + 1, torch.randn(tokens, width)
    w, b, next_w, next_b = (torch.randn(width) for _ in range(4))

    def norm(u, weight, bias):
        mean = u.mean(-1, keepdim=True)
        return (u - mean) / torch.sqrt(((u - mean) ** 2).mean(-1, keepdim=True) + 1e-5) * weight.double() + bias.double()
    want = x.double() + norm(y.double(), w, b) + rows.double()
    got, out = x.cuda(), torch.empty(tokens, width, device="cuda")
    kernels.add_layer_norm(got, y.cuda(), w.cuda(), b.cuda(), 1e-5, rows.cuda(), next_w.cuda(), next_b.cuda(), 1e-5, out)
    assert float((got.double().cpu() - want).abs().max()) <= 5e-6 * float(want.abs().max())
    assert float((out.double().cpu() - norm(want, next_w, next_b)).abs().max()) <= 2e-5 * float(want.abs().max())


@pytest.mark.parametrize("partitions", [2, 5, 40])
@pytest.mark.parametrize("rank,rotary", [(8, 8), (64, 32), (128, 0), (136, 8), (256, 64), (264, 8), (512, 64)])
def test_merge_of_partitions_of_every_value_width(rank, rotary, partitions):
    """One, two or four columns a thread; requests whose last partitions have no keys."""
    from libmir_b200 import kernels
    generator = torch.Generator().manual_seed(rank)
    width, heads, page, contexts = rank + rotary, 3, 16, [1, 64, 65, 500, 40 * 64]
    contexts = [min(c, partitions * 64) for c in contexts]
    pages = [-(-c // page) for c in contexts]
    table = torch.full((len(contexts), max(pages)), -1, dtype=torch.int32)
    pool = torch.randn(sum(pages) * page, 1, width, generator=generator).to(torch.bfloat16)
    q = (torch.randn(len(contexts), heads, width, generator=generator)).to(torch.bfloat16)
    want, first = [], 0
    for r, (context, count) in enumerate(zip(contexts, pages)):
        table[r, :count] = torch.arange(first, first + count)
        keys = pool[first * page:first * page + context, 0].double()
        want.append(torch.softmax(q[r].double() @ keys.T * 0.1, -1) @ keys[:, :rank])
        first += count
    out = torch.full((len(contexts), heads * rank), float("nan"), dtype=torch.bfloat16, device="cuda")
    alloc = lambda shape, kind: torch.full(shape, float("nan"), dtype=kind, device="cuda")
    kernels.latent_attention(q.flatten(1).cuda(), out, pool.cuda(), table.cuda(), ints(range(len(contexts) + 1)), ints(contexts), page,
                             heads, width, rank, 0.1, heads, 64, partitions, alloc)
    want = torch.stack(want).view(len(contexts), -1)
    # (weights rounded to 8 bits, then the result)
    assert float((out.double().cpu() - want).abs().max()) <= 1e-2 * float(want.abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden", [8, 100, 1000, 2048, 2056, 4096, 4104, 9000])
def test_embedding_rows_of_every_width(dtype, hidden):
    """Only moved and multiplied by a power of two: exact; ids outside the table give zeros."""
    from libmir_b200 import kernels
    torch.manual_seed(hidden)
    table, ids = torch.randn(50, hidden).to(dtype), [49, 0, -1, 7, 50]
    out = torch.full((5, hidden), float("nan"), device="cuda")
    kernels.embed(table.cuda(), ints(ids), out, 2.0)
    want = torch.stack([table[i].float() * 2.0 if 0 <= i < 50 else torch.zeros(hidden) for i in ids])
    assert torch.equal(out.cpu(), want)


@pytest.mark.parametrize("wkv", [True, False])
@pytest.mark.parametrize("limit", [1 << 14, 1 << 16, 1 << 19])
def test_a_recurrence_walked_in_runs_of_the_steps_tokens(monkeypatch, wkv, limit):
    """Scratch beyond its bound: from one to many runs, single tokens and several requests in a run; wkv gives the bits of one walk,
    the delta rule in groups of four the same sums from other group borders."""
    from libmir_b200 import kernels
    from libmir_b200.parts import base
    monkeypatch.setattr(base, "RECURRENCE_SCRATCH", limit)
    torch.manual_seed(limit)
    counts, heads, dim = [1, 1, 130, 3, 61, 200], 3, 64
    row_of, starts, slots, positions = batch(counts, [5, 0, 3, 1, 2, 4])
    tokens, width = sum(counts), heads * dim
    make = lambda *shape: torch.randn(*shape, device="cuda")
    state0 = make(6, heads, dim, dim)
    x, raw, bias, bonus = make(3, tokens, width).bfloat16(), make(tokens, width) - 3, make(width), make(width)
    qkv, beta, decay = make(tokens, 3 * width) * 0.1, torch.rand(tokens, heads, device="cuda"), torch.rand(tokens, width, device="cuda")
    qkv[:, width:2 * width] = torch.nn.functional.normalize(qkv[:, width:2 * width].view(tokens, heads, dim), dim=-1).view(tokens, width)

    def walk(runs):
        state, out = state0.clone(), torch.full((tokens, width), float("nan"), device="cuda")
        for run, held in runs:
            count = run.stop - run.start
            if wkv:
                kernels.wkv_scan(x[0, run], x[1, run], x[2, run], raw[run], bias, bonus, state, held, slots, positions[run], out[run],
                                 heads, dim)
            else:
                grouped = torch.empty(kernels.delta_rule_grouped_floats(count, len(counts), heads, dim), device="cuda")
                kernels.delta_rule_scan(qkv[run], beta[run], decay[run], state, held, slots, positions[run], out[run], heads, heads, dim,
                                        dim, grouped=grouped)
        return out, state
    floats = kernels.wkv_prepared_floats(tokens, heads, dim) if wkv else kernels.delta_rule_grouped_floats(tokens, len(counts), heads, dim)
    runs = base.scratch_runs(starts, tokens, 4 * floats)
    assert len(runs) > 1 and runs[-1][0].stop == tokens
    for got, want in zip(walk(runs), walk([(slice(0, tokens), starts)])):
        if wkv:
            assert torch.equal(got, want)
        else:
            assert float((got - want).norm() / want.norm()) <= 2e-6


def portions_alone(run, counts, *tokens):
    """What `run` gives for each request in a step of its own: run(slot, tensors of its tokens) -> (out, state)."""
    starts = np.concatenate([[0], np.cumsum(counts)])
    return [run(r, *(t[..., starts[r]:starts[r + 1], :] for t in tokens)) for r in range(len(counts))]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,dim", [(2, 64), (24, 64), (32, 64), (64, 64), (64, 20), (150, 6), (40, 33), (70, 96)])
def test_wkv_walks_with_one_two_and_four_columns_a_lane(dtype, heads, dim):
    """Three requests (portions of every remainder of a run and a chunk) against the recurrence in 64 bits, and bit for bit against each
    request alone, which takes fewer columns a lane."""
    from libmir_b200 import kernels
    torch.manual_seed(heads + dim)
    counts, width = [37, 2, 50], heads * dim
    tokens = sum(counts)
    x = (torch.randn(3, tokens, width, device="cuda") * 0.5).to(dtype)
    raw, bias, bonus = torch.randn(tokens, width, device="cuda") - 2, torch.randn(width, device="cuda"), torch.randn(width, device="cuda")
    state0 = torch.randn(4, heads, dim, dim, device="cuda")
    slots = [2, 0, 3]

    def run(rows, x, raw, lengths):
        _, starts, held, positions = batch(lengths, rows)
        state, out = state0.clone(), torch.full((sum(lengths), width), float("nan"), device="cuda")
        kernels.wkv_scan(x[0], x[1], x[2], raw, bias, bonus, state, starts, held, positions, out, heads, dim)
        return out, state
    out, state = run(slots, x, raw, counts)
    assert torch.equal(state[1], state0[1])
    begin = 0
    per_head = lambda t: t.double().view(heads, dim)
    for r, (alone, alone_state) in enumerate(portions_alone(lambda r, x, raw: run([slots[r]], x, raw.contiguous(), [raw.shape[0]]),
                                                            counts, x, raw)):
        assert torch.equal(alone, out[begin:begin + counts[r]]) and torch.equal(alone_state[slots[r]], state[slots[r]])
        s = state0[slots[r]].double()                             # [head, value, key]
        for t in range(begin, begin + counts[r]):
            q, k, v = (per_head(x[i, t]) for i in range(3))
            want = torch.einsum("hvk,hk->hv", s, q) + (q * per_head(bonus) * k).sum(-1, keepdim=True) * v
            w = torch.exp(-torch.exp(per_head(raw[t]) + per_head(bias)))
            s = s * w[:, None, :] + v[:, :, None] * k[:, None, :]
            assert float((per_head(out[t]) - want).norm() / want.norm()) <= 2e-6
        assert float((state[slots[r]].double() - s).norm() / s.norm()) <= 2e-6
        begin += counts[r]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,dim,value_dim", [(2, 64, 64), (24, 64, 65), (24, 30, 9), (24, 128, 130), (60, 32, 1), (24, 64, 128), (9, 200, 70)])
def test_retention_walks_with_two_and_four_columns_a_lane(dtype, heads, dim, value_dim):
    from libmir_b200 import kernels
    torch.manual_seed(heads + value_dim)
    counts = [37, 2, 50]
    tokens, qk, width = sum(counts), heads * dim, heads * value_dim
    packed = (torch.randn(tokens, 2 * qk + width, device="cuda") * 0.5).to(dtype)
    decays = torch.rand(heads, device="cuda") * 0.2 + 0.8
    state0 = torch.randn(4, heads, value_dim, dim, device="cuda")
    slots = [2, 0, 3]

    def run(rows, packed, lengths):
        _, starts, held, positions = batch(lengths, rows)
        state, out = state0.clone(), torch.full((sum(lengths), width), float("nan"), device="cuda")
        prepared = torch.full((kernels.retention_prepared_floats(sum(lengths), heads, dim),), float("nan"), device="cuda")
        kernels.retention_scan(packed[:, :qk], packed[:, qk:2 * qk], packed[:, 2 * qk:], None, decays, 0.25, state, starts, held, positions,
                               out, heads, dim, value_dim, prepared=prepared)
        return out, state
    out, state = run(slots, packed, counts)
    assert torch.equal(state[1], state0[1])
    begin = 0
    for r, (alone, alone_state) in enumerate(portions_alone(lambda r, packed: run([slots[r]], packed, [packed.shape[0]]), counts, packed)):
        assert torch.equal(alone, out[begin:begin + counts[r]]) and torch.equal(alone_state[slots[r]], state[slots[r]])
        s = state0[slots[r]].double()
        for t in range(begin, begin + counts[r]):
            q, k = (packed[t, i * qk:(i + 1) * qk].double().view(heads, dim) for i in range(2))
            v = packed[t, 2 * qk:].double().view(heads, value_dim)
            s = s * decays.double()[:, None, None] + 0.25 * v[:, :, None] * k[:, None, :]
            want = torch.einsum("hvk,hk->hv", s, q)
            assert float((out[t].double().view(heads, value_dim) - want).norm() / want.norm()) <= 2e-6
        assert float((state[slots[r]].double() - s).norm() / s.norm()) <= 2e-6
        begin += counts[r]


@pytest.mark.parametrize("dtype,gate_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("value_dim,heads", [(1, 3), (32, 5), (33, 3), (64, 7), (65, 2), (128, 5), (200, 3), (256, 2), (257, 3)])
@pytest.mark.parametrize("per_head", [False, True])
def test_gated_norms_of_heads_sum_in_one_order_whatever_holds_them(dtype, gate_dtype, value_dim, heads, per_head):
    """Eight, 16 and 32 lanes a head, and heads that are read twice: lane l of 32 sums the numbers l, l + 32, ... and
    the lanes' sums are added by halves; gates off the 16-byte boundary."""
    from libmir_b200 import kernels
    torch.manual_seed(value_dim)
    tokens = 5
    o, gate = torch.randn(tokens, heads * value_dim), torch.randn(tokens, heads * value_dim + 3).to(gate_dtype)
    weight = torch.rand(heads * value_dim if per_head else value_dim) + 0.5
    rows = np.zeros((tokens * heads, -(-value_dim // 32) * 32))
    rows[:, :value_dim] = o.double().numpy().reshape(tokens * heads, value_dim)
    total = np.zeros((tokens * heads, 32))
    for piece in np.split(rows, rows.shape[1] // 32, axis=1):
        total = rounded(piece * piece + total)
    for step in (16, 8, 4, 2, 1):
        total = rounded(total + total[:, np.arange(32) ^ step])
    mean = total[:, 0].astype(np.float32) / np.float32(value_dim) + np.float32(1e-5)
    inverse = torch.rsqrt(torch.from_numpy(mean).cuda()).view(tokens, heads, 1)
    out = torch.empty(tokens, heads * value_dim, dtype=dtype, device="cuda")
    kernels.gated_head_norm(o.cuda(), gate.cuda()[:, 3:], weight.cuda(), out, heads, value_dim, 1e-5, False)
    z = gate[:, 3:].double().view(tokens, heads, value_dim)
    scaled = o.cuda().view(tokens, heads, value_dim) * inverse * weight.cuda().view(-1, value_dim)
    want = scaled.double().cpu() * z * torch.sigmoid(z)
    # the gate's own function is good to a few units in the last place; with the sum in another order a row would be off as a whole
    error = (out.double().cpu().view_as(want) - want).abs()
    assert bool((error <= (2 ** -8 if dtype == torch.bfloat16 else 4e-7) * want.abs() + 1e-30).all())


@pytest.mark.parametrize("groups,rows,n,k", [(4, 1, 128, 64), (4, 3, 200, 136), (5, 16, 40, 72), (2, 17, 256, 512), (3, 32, 130, 64), (4, 33, 64, 64), (2, 5, 64, 60)])
def test_products_side_by_side(groups, rows, n, k):
    """Products of one shape in one launch (up to 32 rows; a row more and a k that is no multiple of eight go one by one): columns and steps that end inside a tile,
    neighbouring groups' rows inside a tile."""
    from libmir_b200 import kernels
    torch.manual_seed(rows)
    x, w = torch.randn(groups, rows, k).bfloat16(), torch.randn(groups, n, k).bfloat16()
    out = torch.full((groups, rows, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    kernels.linear_side_by_side(x.cuda(), w.cuda(), out, alloc=lambda shape, kind: torch.empty(shape, dtype=kind, device="cuda"))
    want = x.double() @ w.double().transpose(1, 2)
    # rounded to 8 bits of mantissa; the 32-bit sums are off by far less than one of its units unless they cancel
    bound = 2 ** -8 * want.abs() + k * 2 ** -24 * (x.double().abs() @ w.double().abs().transpose(1, 2))
    assert ((out.cpu().double() - want).abs() <= bound).all()


@pytest.mark.parametrize("n,k", [(14208, 520), (14209, 512), (24576, 512), (24577, 520), (28416, 256), (28417, 264),
                                 (28416, 512), (28417, 512), (6144, 2048), (6145, 2056), (13312, 1024), (13313, 1032)])
@pytest.mark.parametrize("rows", [1, 32])
def test_weight_streams_on_both_sides_of_the_rings_and_the_cuts(rows, n, k):
    """111 and 112 tiles of columns cut in two (222 and 224 blocks), 192, 193 and 222 cut in two, 222 and 223 that are not; 48
    cut in eight and 49 in four, 104 cut in four and 105 in two: the large ring and the small one, with steps that do not fill
    it."""
    from libmir_b200 import kernels
    torch.manual_seed(n + rows)
    x, w = torch.randn(rows, k).bfloat16(), torch.randn(n, k).bfloat16()
    out = torch.full((rows, n), float("nan"), device="cuda")
    kernels.linear(x.cuda(), w.cuda(), out)
    # sums of k products in 32 bits: each partial sum off by at most 2^-24 of the sum of the products' sizes
    bound = k * 2 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((out.cpu().double() - x.double() @ w.double().T).abs() <= bound).all()
    assert kernels.tensor_core_linear_error() == 0


@pytest.mark.parametrize("experts,width,full", [(640, 2560, 0), (1024, 2560, 0), (1024, 2568, 300)])
def test_grouped_products_of_more_tiles_than_are_looked_up_at_once(experts, width, full):
    """43, 69 and 76 tiles a block: one expert's tiles behind another's, with an expert of several tiles of rows among them."""
    from libmir_b200 import kernels
    torch.manual_seed(experts)
    inter, alloc = 8, lambda shape, kind: torch.zeros(shape, dtype=kind, device="cuda")
    ids = torch.cat([torch.arange(experts), torch.full((full,), experts // 2)]).int()[:, None].contiguous()
    found = kernels.moe_sort(ids.cuda(), experts, alloc, 128)
    hidden, w = torch.randn(len(ids), inter).bfloat16().cuda(), torch.randn(experts, width, inter).bfloat16().cuda()
    out = torch.full((len(ids), width), float("nan"), device="cuda")
    kernels.moe_down(hidden, found, w, out)
    order = found.order.long()
    for first in range(0, len(ids), 64):
        pairs = order[first:first + 64]
        x, rows = hidden[first:first + 64].double(), w[ids[:, 0].cuda().long()[pairs]].double()
        error = (out[pairs].double() - torch.einsum("pi,pwi->pw", x, rows)).abs()
        # eight products in 32 bits, each partial sum off by at most 2^-24 of the sum of their sizes
        assert (error <= inter * 2 ** -24 * torch.einsum("pi,pwi->pw", x.abs(), rows.abs())).all()
    assert kernels.tensor_core_linear_error() == 0


@pytest.mark.parametrize("position, keep_first, window", [(40, 0, None), (33, 0, None), (70, 0, 30), (52, 4, 25), (127, 20, 100)])
def test_decoded_tokens_read_no_page_beyond_their_table(position, keep_first, window):
    """A position beyond what the block table holds: the mma.sync kernel takes the keys there as released, as the tcgen05 kernel
    does.  What lies behind the table in memory are pages whose keys and values would show."""
    from libmir_b200 import kernels
    torch.manual_seed(position)
    rows, width, wide, page, heads, dim = 2, 2, 8, 16, 4, 128
    qkv = torch.randn(rows, 3 * heads * dim).bfloat16().cuda()
    pages = torch.randn(2, 32 * page, heads, dim).bfloat16().cuda()
    pages[:, 16 * page:] = float("nan")
    memory = torch.arange(16, 32, dtype=torch.int32, device="cuda")
    memory[:rows * width] = torch.arange(rows * width)
    narrow, same = memory[:rows * width].view(rows, width), torch.full((rows, wide), -1, dtype=torch.int32, device="cuda")
    same[:, :width] = narrow
    positions = torch.full((rows,), position, dtype=torch.int32, device="cuda")
    outputs = []
    for table in (narrow, same):
        outputs.append(torch.full((rows, heads * dim), float("nan"), dtype=torch.bfloat16, device="cuda"))
        numbering = torch.zeros(rows, dtype=torch.int32, device="cuda")
        kernels.decode_attention(qkv, outputs[-1], pages[0], pages[1], table, positions, page, heads, heads, dim, dim ** -0.5, window,
                                 128, 1, None, keep_first=keep_first, numbering=numbering, short=keep_first == 0)
    assert torch.isfinite(outputs[0]).all() and torch.equal(*outputs)
