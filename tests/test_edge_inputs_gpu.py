"""Inputs that real ones turn into when something upstream goes wrong, and steps of unusual make-up: rows that are no numbers,
infinities, experts named twice, and as many entries as do not fit the GPU at once."""

import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import dev, f64
from test_product_kernels_gpu import recurrence_case

pytestmark = pytest.mark.gpu


def expert_tables(rng, experts, inner, width):
    total = experts * inner
    gates, ups = (dev(rng.normal(size=(total, width)) / math.sqrt(width), torch.bfloat16) for _ in range(2))
    downs = dev(rng.normal(size=(width, total)) / math.sqrt(inner), torch.bfloat16)
    at = lambda matrix, step: torch.tensor([matrix.data_ptr() + 2 * step * e * inner for e in range(experts)], dtype=torch.int64, device="cuda")
    return (at(gates, width), at(ups, width), at(downs, 1), dev(np.full(experts, inner, np.int32))), (gates, ups, downs)


@pytest.mark.parametrize("tokens, experts, top, broken", [(31, 8, 2, 20), (31, 8, 8, 6), (6, 16, 8, 5)])
def test_tokens_that_are_no_numbers_beside_healthy_ones_in_expert_tiles(tokens, experts, top, broken):
    """The router names the first expert for every choice of such a token: more pairs of one expert than there are tokens."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(tokens + top)
    width, inner = 264, 296
    tables, _held = expert_tables(rng, experts, inner, width)
    values = rng.normal(size=(tokens, width))
    sick = np.sort(rng.permutation(tokens)[:broken])
    healthy = np.setdiff1d(np.arange(tokens), sick)
    values[sick] = np.nan
    x, router = dev(values, torch.bfloat16), dev(rng.normal(size=(experts, width)) / math.sqrt(width), torch.bfloat16)
    choice = torch.full((tokens * top,), -7, dtype=torch.int32, device="cuda")
    in_weight, out_weight = (torch.full((tokens * top,), math.nan, device="cuda") for _ in range(2))
    ops.route(x, router, None, top, choice, in_weight, out_weight)
    assert (choice.view(tokens, top)[torch.tensor(sick)] == 0).all()
    before, results = rng.normal(size=(tokens, width)).astype(np.float32), []
    for tiles in (True, False):
        hidden, act = dev(before), torch.full((tokens * top, inner), math.nan, dtype=torch.bfloat16, device="cuda")
        ops.experts(hidden, act, x, choice, in_weight, out_weight, *tables, inner, top, ld_down=experts * inner, tiles=tiles)
        results.append(f64(hidden))
    # activations are rounded to 8 bits once, here and there by different 32-bit sums: a neighbour's step is 2^-8 of the activation,
    # and few of a row's top x 296 products see one
    np.testing.assert_allclose(results[0][healthy], results[1][healthy], rtol=0, atol=4e-3)
    assert np.isfinite(results[0][healthy]).all()
    np.testing.assert_array_equal(np.isnan(results[0][sick]), np.isnan(results[1][sick]))


def test_an_expert_named_more_than_once_by_its_tokens():
    """More pairs of an expert than a list of its tiles holds, with weights of their own each; one that no table has counts as none."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(3)
    tokens, experts, top, width, inner = 19, 3, 6, 72, 136
    tables, (gates, ups, downs) = expert_tables(rng, experts, inner, width)
    x = dev(rng.normal(size=(tokens, width)), torch.bfloat16)
    chosen = rng.integers(0, 2, (tokens, top)).astype(np.int32)
    chosen[4, 2] = -1
    in_weight, out_weight = (rng.uniform(0.2, 1.0, (tokens, top)).astype(np.float32) for _ in range(2))
    expected = np.zeros((tokens, width))
    for t in range(tokens):
        for e, a, b in zip(chosen[t], in_weight[t], out_weight[t]):
            if e >= 0:
                part = slice(e * inner, (e + 1) * inner)
                into = f64(dev(a * f64(x)[t].astype(np.float32), torch.bfloat16))
                g, u = f64(gates)[part] @ into, f64(ups)[part] @ into
                expected[t] += b * (f64(downs)[:, part] @ (g / (1 + np.exp(-g)) * u))
    for tiles in (True, False):
        hidden, act = torch.zeros(tokens, width, device="cuda"), torch.full((tokens * top, inner), math.nan, dtype=torch.bfloat16, device="cuda")
        ops.experts(hidden, act, x, dev(chosen.reshape(-1)), dev(in_weight.reshape(-1)), dev(out_weight.reshape(-1)), *tables, inner, top,
                    ld_down=experts * inner, tiles=tiles)
        # an activation's rounding is 2^-9 of it, 6 x 136 of them go into a sum of size 6
        np.testing.assert_allclose(f64(hidden), expected, rtol=0, atol=2e-2, err_msg=f"tiles={tiles}")


def sigmoid_log(x):
    return -np.logaddexp(0.0, -x)


# six slices of the values and more blocks than the GPU holds at once; slices that take two launches; one slice
@pytest.mark.parametrize("entries, heads, dim, vdim", [(63, 4, 96, 192), (5, 2, 40, 300), (9, 3, 16, 20)])
@pytest.mark.parametrize("chunked", [False, True])
@pytest.mark.parametrize("writes", [True, False])
def test_gated_memories_of_more_entries_than_are_resident(entries, heads, dim, vdim, chunked, writes):
    """The vector and the maximum that a head's slices share are read by every slice and written by one."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(entries + vdim)
    cap, scale = 15.0, dim ** -0.5
    bias = rng.normal(size=2 * heads).astype(np.float32)
    state = dev(rng.normal(0, 0.5, (entries + 2, ops.memory_state_floats(heads, dim, vdim, True))), torch.float32)
    slots = rng.permutation(entries + 2)[:entries]
    held = f64(state)
    S = held[slots, :heads * dim * vdim].reshape(entries, heads, dim, vdim)
    n = held[slots, heads * dim * vdim:heads * dim * (vdim + 1)].reshape(entries, heads, dim)
    m = held[slots, heads * dim * (vdim + 1):heads * dim * (vdim + 1) + heads]
    for most in (1, 2, 3):
        counts = rng.integers(0, most + 1, entries)
        counts[:3] = (most, 0, 1)
        offsets, total = np.cumsum(counts) - counts, int(counts.sum())
        q, k, v = (dev(rng.normal(size=(total, heads * size)), torch.bfloat16) for size in (dim, dim, vdim))
        gates = dev(rng.normal(0, 3, (total, 2 * heads)), torch.float32)
        before, readers = state.clone(), torch.zeros(entries * heads + 1, dtype=torch.int32, device="cuda")
        expected = np.zeros((total, heads, vdim))
        S1, n1, m1 = S.copy(), n.copy(), m.copy()
        for t in range(most):
            e = np.flatnonzero(counts > t)
            at = offsets[e] + t
            qt, kt, vt = (f64(x)[at].reshape(len(e), heads, -1) for x in (q, k, v))
            raw = f64(gates)[at] + bias
            li, lf = cap * np.tanh(raw[:, :heads] / cap), sigmoid_log(cap * np.tanh(raw[:, heads:] / cap))
            new = np.maximum(lf + m1[e], li)
            a, b = np.exp(lf + m1[e] - new)[..., None], np.exp(li - new)[..., None]
            S1[e] = a[..., None] * S1[e] + b[..., None] * kt[..., None] * vt[:, :, None]
            n1[e], m1[e] = a * n1[e] + b * kt, new
            qt = qt * scale
            below = np.maximum(np.abs((n1[e] * qt).sum(-1)), np.exp(-new)) + 1e-6
            expected[at] = np.einsum("ehdv,ehd->ehv", S1[e], qt) / below[..., None]
        out = torch.full((total, heads * vdim), math.nan, device="cuda")
        ops.memory_scan(out, q, k, v, state, dev(slots.astype(np.int32)), dev(offsets.astype(np.int32)), dev(counts.astype(np.int32)), heads, dim,
                        vdim, q_scale=scale, gates=gates, gate_bias=dev(bias), gate_cap=cap, writes=writes, chunked=chunked,
                        readers=readers if most > 1 else None)
        assert int(readers.abs().sum()) == 0
        # a state's entries below 10 and sums of `dim` products of them in 32 bits; the quotient's divisor is 0.01 or more here
        np.testing.assert_allclose(f64(out), expected.reshape(total, -1), rtol=2e-5, atol=2e-5 * max(1.0, np.abs(expected).max()))
        if writes:
            S, n, m = S1, n1, m1
            both = np.concatenate([S.reshape(entries, -1), n.reshape(entries, -1), m], 1)
            np.testing.assert_allclose(f64(state)[slots], both, rtol=0, atol=5e-5)
        else:
            assert torch.equal(state, before)


@pytest.mark.parametrize("m, k", [(1, 102400), (1, 14344), (2, 51200), (8, 12800), (16, 6400), (3, 25600)])
def test_norms_inside_few_row_products_of_the_longest_rows_they_take(m, k):
    from mini_llm_b200.kernels import ops
    assert ops.skinny_linear_takes(m, k)
    rng = np.random.default_rng(k)
    n = 24
    x, w = dev(rng.normal(2.0, 3.0, (m + 2, k)), torch.float32), dev(rng.normal(size=(n, k)) / math.sqrt(k), torch.bfloat16)
    gain, shift = dev(rng.uniform(0.5, 1.5, k), torch.float32), dev(rng.normal(0, 0.1, k), torch.float32)
    rows, out = rng.permutation(m + 2)[:m], torch.full((m, n), math.nan, device="cuda")
    ops.skinny_linear(out, x, w, None, "store", norm=(gain, shift, 1e-5, dev(rows.astype(np.int32))))
    c = f64(x)[rows] - f64(x)[rows].mean(-1, keepdims=True)
    normed = c / np.sqrt((c * c).mean(-1, keepdims=True) + 1e-5) * f64(gain) + f64(shift)
    # an entry of the normed row is rounded by 2^-9 of itself at most; over k products of size 1 / sqrt(k) that walks to 2^-9, of
    # which no sum here is more than four times off
    np.testing.assert_allclose(f64(out), normed @ f64(w).T, rtol=0, atol=8e-3)


@pytest.mark.parametrize("m, n, k", [(2, 16384, 3072), (8, 24, 4096), (8, 768, 768), (16, 3072, 768)])
def test_few_row_products_of_one_sign(m, n, k):
    """Sums that only grow: what is cut off them instead of rounded would add up."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(n)
    x, w = dev(rng.uniform(size=(m, k)), torch.bfloat16), dev(rng.uniform(size=(n, k)), torch.bfloat16)
    out, heads = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
    ops.skinny_linear(out, x, w, None, "store")
    ops.skinny_heads(heads, x, w[None].contiguous(), 1, k, n)
    want = (x.double() @ w.double().T)
    # 16 entries' product is cut off by 2^-24 of itself at most, their additions and the last rounding are off by as much of what is
    # summed, up or down: some 2^-23 of a result together (as one chain in the tensor cores 1.1e-7 to 5e-6)
    for got in (out, heads):
        assert float((got.double() - want).norm() / want.norm()) < 1.0e-7


def test_expert_tiles_of_one_sign():
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(0)
    tokens, experts, inner, width = 16, 4, 768, 64
    total = experts * inner
    gates, ups, downs = (dev(rng.uniform(0.0, 0.1, s), torch.bfloat16) for s in ((total, width), (total, width), (width, total)))
    at = lambda matrix, step: torch.tensor([matrix.data_ptr() + 2 * step * e * inner for e in range(experts)], dtype=torch.int64, device="cuda")
    chosen = np.stack([rng.permutation(experts)[:2] for _ in range(tokens)]).astype(np.int32)
    x, ones = dev(rng.uniform(size=(tokens, width)), torch.bfloat16), torch.ones(tokens * 2, device="cuda")
    hidden, act = torch.zeros(tokens, width, device="cuda"), torch.empty(tokens * 2, inner, dtype=torch.bfloat16, device="cuda")
    ops.experts(hidden, act, x, dev(chosen.reshape(-1)), ones, ones, at(gates, width), at(ups, width), at(downs, 1), dev(np.full(experts, inner, np.int32)),
                inner, 2, ld_down=total, tiles=True)
    want = np.zeros((tokens, width))
    for t in range(tokens):
        for j, e in enumerate(chosen[t]):
            want[t] += f64(downs)[:, e * inner:(e + 1) * inner] @ f64(act)[2 * t + j]
    assert np.linalg.norm(f64(hidden) - want) / np.linalg.norm(want) < 1.0e-7          # (as above; 2.5e-7 as chains of 256)


# tokens that stand alone beside a portion (few tokens a block) and a prompt whose blocks fill the GPU (as many as fit)
@pytest.mark.parametrize("lengths, new, heads, kv_heads, window", [
    ([90 + 7 * i for i in range(20)] + [60], [1] * 20 + [60], 12, 4, 0), ([700], [700], 12, 4, 0), ([200] * 9 + [33, 2], [1] * 9 + [33, 2], 4, 4, 64)])
def test_capped_attention_of_tokens_that_stand_alone_beside_portions(lengths, new, heads, kv_heads, window):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(len(new))
    dim, page = 64, 16
    table, (k_pages, v_pages) = pages_of(rng, lengths, page, kv_heads, (dim, dim))
    positions = dev(np.concatenate([np.arange(l - m, l) for l, m in zip(lengths, new)]).astype(np.int32))
    items, n = dev(np.repeat(np.arange(len(new)), new).astype(np.int32)), sum(new)
    q = dev(rng.normal(size=(n, heads * dim)), torch.bfloat16)
    want, got = (torch.full((n, heads * dim), math.nan, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    for out, tiled in ((want, False), (got, True)):
        ops.capped_attention(out, q, k_pages, v_pages, table.cuda(), positions, items, heads, kv_heads, dim, dim, page, dim ** -0.5, cap=20.0,
                             window=window, tiled=tiled)
    # both keep scores, weights and sums in 32 bits, so they may differ by the last rounding to 8 bits: 2^-8 of values below 4
    np.testing.assert_allclose(f64(got), f64(want), rtol=2 ** -7, atol=2 ** -10)


def pages_of(rng, lengths, page, heads, size):
    blocks = [-(-n // page) for n in lengths]
    table = torch.zeros(len(lengths), max(blocks), dtype=torch.int32)
    order = rng.permutation(sum(blocks))
    for i, count in enumerate(blocks):
        table[i, :count] = torch.tensor(order[sum(blocks[:i]):sum(blocks[:i]) + count])
    return table, [dev(rng.normal(size=(sum(blocks), page, heads, s)), torch.bfloat16) for s in size]


# portions of some tokens beside tokens that stand alone: more than the kernel for one token an entry takes, fewer than the chunks'
@pytest.mark.parametrize("heads, qk_heads, dim, vdim, delta", [(2, 1, 64, 24, True), (4, 2, 128, 33, True), (3, 3, 40, 65, False)])
def test_recurrence_of_uneven_entries(heads, qk_heads, dim, vdim, delta):
    recurrence_case(heads, qk_heads, dim, vdim, delta, ([1, 1, 11, 1], [2, 2, 1, 3], [1, 3, 1, 1]))


def cell(pages, table, entry, position):
    return pages[int(table[entry, position // pages.shape[1]]), position % pages.shape[1]]


@pytest.mark.parametrize("dim", [64, 128])
def test_infinite_cached_values_in_tiled_attention(dim):
    """An infinite value makes its column infinite where its key is seen, and a key that is infinitely far away weighs nothing."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(dim)
    heads, kv_heads, page, lengths = 4, 2, 16, [100, 70]
    table, (k_pages, v_pages) = pages_of(rng, lengths, page, kv_heads, (dim, dim))
    cell(v_pages, table, 0, 3)[1, 5] = math.inf
    cell(v_pages, table, 0, 40)[0, 9] = -math.inf
    cell(v_pages, table, 1, 20)[1, 7] = math.inf
    cell(k_pages, table, 1, 2)[0, 1] = -math.inf                  # (queries are positive there: the score is -infinity)
    new = [50, 45]
    positions = dev(np.concatenate([np.arange(l - m, l) for l, m in zip(lengths, new)]).astype(np.int32))
    items, n = dev(np.repeat(np.arange(2), new).astype(np.int32)), sum(new)
    q = dev(rng.normal(size=(n, heads * dim)), torch.bfloat16)
    q.view(n, heads, dim)[:, :, 1].abs_()
    tiled, split = (torch.full((n, heads * dim), math.nan, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    common = (k_pages, v_pages, table.cuda(), positions, items, heads, kv_heads, dim)
    ops.capped_attention(tiled, q, *common, dim, page, dim ** -0.5, tiled=True)
    scratch = (torch.empty(n * heads * 4 * dim, device="cuda"), torch.empty(n * heads * 8, device="cuda"),
               torch.zeros(n * heads, dtype=torch.int32, device="cuda"))
    ops.split_attention(split, q, *common, page, dim ** -0.5, 0, 64, -(-table.shape[1] * page // 64), *scratch)
    want = np.zeros((n, heads, dim))
    for t, (entry, position) in enumerate(zip(f64(items).astype(int), f64(positions).astype(int))):
        k, v = (np.stack([f64(cell(pages, table, entry, j)) for j in range(position + 1)]) for pages in (k_pages, v_pages))
        for h in range(heads):
            scores = k[:, h // 2] @ f64(q)[t, h * dim:(h + 1) * dim] * dim ** -0.5
            weights = np.exp(scores - scores.max())
            want[t, h] = (weights[:, None] / weights.sum() * v[:, h // 2]).sum(0)
    assert (want[:50, 2:, 5] == math.inf).all() and (want[:50, :2, 9] == -math.inf).all() and (want[50:, 2:, 7] == math.inf).all()
    assert np.isinf(want).sum() == (50 + 50 + 45) * 2 and not np.isnan(want).any()
    for got in (tiled, split):                                    # (rounded to 8 bits once)
        np.testing.assert_allclose(f64(got).reshape(n, heads, dim), want, rtol=2 ** -8, atol=1e-5)


@pytest.mark.parametrize("new", [[8, 20, 40], [3, 5, 300], [1, 1, 1, 1, 1, 35]])
def test_cached_values_that_are_no_numbers_stay_with_their_request(new):
    """Requests that share a tile of queries: what is wrong in the second one's cache is not seen by the others."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(len(new))
    heads, dim, page, lengths = 16, 64, 16, [m + 30 for m in new]         # (16 heads: eight tokens a block and more)
    table, (k_pages, v_pages) = pages_of(rng, lengths, page, heads, (dim, dim))
    positions = dev(np.concatenate([np.arange(l - m, l) for l, m in zip(lengths, new)]).astype(np.int32))
    items, n = np.repeat(np.arange(len(new)), new), sum(new)
    q = dev(rng.normal(size=(n, heads * dim)), torch.bfloat16)
    healthy, beside = (torch.full((n, heads * dim), math.nan, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    for out in (healthy, beside):
        ops.capped_attention(out, q, k_pages, v_pages, table.cuda(), positions, dev(items.astype(np.int32)), heads, heads, dim, dim, page,
                             dim ** -0.5, tiled=True)
        for j in range(lengths[1]):                               # (for the second pass)
            cell(v_pages, table, 1, j)[:] = math.nan if j % 2 else math.inf
    assert np.isfinite(f64(healthy)).all() and np.isnan(f64(beside)[items == 1]).all()
    np.testing.assert_array_equal(f64(beside)[items != 1], f64(healthy)[items != 1])


@pytest.mark.parametrize("rank", [128, 256])
def test_infinite_cached_rows_in_tiled_latent_attention(rank):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(rank)
    heads, rot, page, lengths, new = 3, 32, 16, [90], [30]
    row = rank + rot
    table, (pages,) = pages_of(rng, lengths, page, 1, (row,))
    cell(pages, table, 0, 11)[0, rank + 2] = -math.inf            # (in the part that is no value)
    positions, items = dev(np.arange(60, 90).astype(np.int32)), torch.zeros(30, dtype=torch.int32, device="cuda")
    q = dev(rng.normal(size=(30, heads * row)), torch.float32)
    q.view(30, heads, row)[:, :, rank + 2] = 0.5                  # (one significant bit: its second and third terms are nothing)
    want, got = torch.full((30, heads * rank), math.nan, device="cuda"), torch.full((30, heads * rank), math.nan, device="cuda")
    ops.latent_attention_plain(want, q, pages, table.cuda(), positions, items, heads, rank, rot, page, 0.1)
    tiles, _, _ = ops.attention_tiles([0], new, [60])
    ops.latent_attention_tiled(got, q, pages, table.cuda(), positions, items, heads, rank, rot, page, 0.1,
                               tiles=dev(np.array(tiles, dtype=np.int32)), n_tiles=len(tiles))
    assert np.isfinite(f64(want)).all()
    np.testing.assert_allclose(f64(got), f64(want), rtol=2e-5, atol=3e-5)        # 32-bit sums on both sides


@pytest.mark.parametrize("delta", [True, False])
@pytest.mark.parametrize("where", ["value", "key", "state", "nan"])
def test_numbers_that_are_not_finite_in_recurrences_over_portions(delta, where):
    """They reach the tokens behind them, as token by token, and none before."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(5)
    heads, dim, vdim, counts, bad = 2, 64, 24, [70, 33], 37
    n = sum(counts)
    q, k = (dev(np.abs(rng.normal(size=(n, heads * dim))) + 0.1, torch.bfloat16) for _ in range(2))
    v = dev(rng.normal(size=(n, heads * vdim)), torch.bfloat16)
    gate_a, gate_b = dev(rng.normal(size=(n, heads)), torch.float32), dev(rng.normal(size=(n, heads)), torch.float32)
    state = dev(np.abs(rng.normal(0, 0.3, (2, heads * dim * vdim))), torch.float32)
    if where == "value":
        v[bad, vdim + 3] = math.inf
    elif where == "nan":
        v[bad, vdim + 3] = math.nan
    elif where == "key":
        k[bad, dim + 1] = math.nan
    else:
        state.view(2, heads, dim, vdim)[0, 1, 6, 3] = math.inf
    S, expected, t = f64(state).reshape(2, heads, dim, vdim), np.zeros((n, heads, vdim)), 0
    with np.errstate(all="ignore"):
        for entry, count in enumerate(counts):
            for t in range(t, t + count):
                for h in range(heads):
                    qt, kt, vt = f64(q)[t, h * dim:(h + 1) * dim], f64(k)[t, h * dim:(h + 1) * dim], f64(v)[t, h * vdim:(h + 1) * vdim]
                    step = np.log1p(np.exp(f64(gate_a)[t, h]))
                    a, b = np.exp(-step), step
                    if delta:
                        qt, kt, b = qt / np.sqrt(qt @ qt + 1e-6), kt / np.sqrt(kt @ kt + 1e-6), 1 / (1 + np.exp(-f64(gate_b)[t, h]))
                    old = a * S[entry, h]
                    S[entry, h] = old + kt[:, None] * (b * (vt - ((old * kt[:, None]).sum(0) if delta else 0)))[None]
                    expected[t, h] = (S[entry, h] * qt[:, None]).sum(0) + 0.0 * vt           # (no skip: a factor of zero)
            t += 1
    zeros, out = torch.zeros(heads, device="cuda"), torch.full((n, heads * vdim), math.nan, device="cuda")
    ints = lambda x: dev(np.array(x, np.int32))
    ops.linear_recurrence(out, q, k, v, gate_a, gate_b if delta else None, zeros, zeros, state, ints([0, 1]), ints([0, 70]), ints(counts), heads, heads,
                          dim, vdim, delta, unit_norm=delta)
    got = f64(out).reshape(n, heads, vdim)
    assert np.isfinite(got[:bad if where != "state" else 0]).all() and np.isfinite(got[70:]).all() and np.isfinite(got[:, 0]).all()
    assert not np.isfinite(got[bad:70, 1, 3]).any()
    sound = np.isfinite(expected)
    np.testing.assert_array_equal(np.isfinite(got), sound)
    if not delta and where in ("value", "state"):
        np.testing.assert_array_equal(got[~sound], expected[~sound])          # infinities, as all keys and queries are positive
    np.testing.assert_allclose(got[sound], expected[sound], rtol=0, atol=4e-6 * max(1.0, np.abs(expected[sound]).max()))


# groups of one and of many quads, widths that end inside a warp, the widest row a block takes
@pytest.mark.parametrize("width, groups", [(96, 3), (768, 4), (20, 5), (4096, 1), (1036, 7)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_and_four_taps_in_one_step(width, groups, dtype):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(width)
    tokens, slots = 5, np.array([6, 0, 3, 1, 5], np.int32)
    x, gain, w = (dev(v, torch.float32) for v in (rng.normal(0, 2, (tokens, width)), rng.uniform(0.5, 1.5, width), rng.normal(0, 0.5, (width, 4))))
    state = dev(rng.normal(size=(7, 3, width)), torch.float32)
    items, before = dev(np.array([4, 2, 0, 1, 3], np.int32)), f64(state)
    mine = slots[f64(items).astype(int)]
    kept, out = state.clone(), torch.full((tokens, width), math.nan, dtype=dtype, device="cuda")
    ops.norm_taps_step(out, x, gain, groups, 1e-5, w, kept, items, dev(slots), writes=False)
    assert torch.equal(kept, state)
    again = torch.empty_like(out)
    ops.norm_taps_step(again, x, gain, groups, 1e-5, w, state, items, dev(slots))
    assert torch.equal(again, out)
    moved = f64(state)
    pieces = f64(x).reshape(tokens, groups, -1)
    normed = (pieces / np.sqrt((pieces ** 2).mean(-1, keepdims=True) + 1e-5)).reshape(tokens, width) * f64(gain)
    rounding = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-6
    np.testing.assert_allclose(moved[mine, 2], normed, rtol=rounding, atol=1e-6)             # (rounded as an activation)
    np.testing.assert_array_equal(moved[mine, :2], before[mine, 1:])
    np.testing.assert_array_equal(moved[[2, 4]], before[[2, 4]])
    taps = f64(w)
    expected = moved[mine, 2] * (1 + taps[:, 3]) + sum(before[mine, j] * taps[:, j] for j in range(3))
    np.testing.assert_allclose(f64(out), expected, rtol=rounding, atol=4e-6)                 # five 32-bit products of values below 8


@pytest.mark.parametrize("width, identity, bias, silu", [(8, True, False, False), (24, False, True, True), (1288, False, False, True), (1536, True, True, False)])
@pytest.mark.parametrize("dtype, counts", [(torch.bfloat16, [1, 7, 4, 0, 13, 2, 3]), (torch.bfloat16, None), (torch.float32, None)])
def test_filters_of_four_taps(width, identity, bias, silu, dtype, counts):
    """Portions that begin and end inside a thread's run of four tokens, from a state and moving it on; and steps of single tokens."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(width)
    single = counts is None
    counts = [1] * 6 if single else counts
    n, entries = sum(counts), len(counts)
    slots, starts, offsets = rng.permutation(entries + 2)[:entries], rng.integers(0, 9, entries), np.cumsum(counts) - counts
    wide, into = dev(rng.normal(size=(n, width + 16)), dtype), torch.full((n, width + 8), math.nan, dtype=dtype, device="cuda")
    h, out = wide[:, 8:8 + width], into[:, 8:]
    w, state = dev(rng.normal(0, 0.5, (width, 4)), torch.float32), dev(rng.normal(size=(entries + 2, 3, width)), torch.float32)
    b = dev(rng.normal(size=width), torch.float32) if bias else None
    items = np.repeat(np.arange(entries), counts)
    positions = np.concatenate([np.arange(s, s + c) for s, c in zip(starts, counts)])
    ints = lambda values: dev(np.asarray(values).astype(np.int32))
    before, expected, after = f64(state), np.zeros((n, width)), f64(state)
    for entry, (slot, offset, count) in enumerate(zip(slots, offsets, counts)):
        rows = np.concatenate([before[slot], f64(h)[offset:offset + count]])
        for t in range(count):
            y = (rows[t:t + 4] * f64(w).T).sum(0) + (rows[t + 3] if identity else 0) + (f64(b) if bias else 0)
            expected[offset + t] = y / (1 + np.exp(-y)) if silu else y
        after[slot] = rows[-3:]
    kept = state.clone()
    for moving, writes in ((kept, False), (state, True)):
        if single and not writes:
            continue                                                         # (a step of single tokens that writes nothing is a portion's)
        ops.causal_taps(out, h, w, moving, ints(positions), ints(items), ints(slots), ints(starts), ints(offsets), ints(counts), writes, identity, b, silu,
                        single_tokens=single)
        # five 32-bit products of values below 4, rounded once
        np.testing.assert_allclose(f64(out), expected, rtol=2 ** -8 if dtype == torch.bfloat16 else 2e-6, atol=4e-6)
    if not single:
        np.testing.assert_array_equal(f64(kept), before)
    np.testing.assert_array_equal(f64(state), after)
    assert torch.isnan(into[:, :8]).all()


def test_one_product_by_its_sizes_alone():
    """A caller of the kernel library that knows of no batches leaves that field zero."""
    import ctypes
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(0)
    x, w, out = dev(rng.normal(size=(3, 64)), torch.bfloat16), dev(rng.normal(size=(40, 64)) / 8, torch.bfloat16), torch.empty(3, 40, device="cuda")
    params = ops._SkinnyParams()
    params.out, params.x, params.w, params.M, params.N, params.K = out.data_ptr(), x.data_ptr(), w.data_ptr(), 3, 40, 64
    params.ldx, params.ldo, params.epilogue, params.out_f32 = 64, 40, ops.EPILOGUES["store"], 1
    ops._skinny(ctypes.byref(params), ops._stream())
    np.testing.assert_allclose(f64(out), f64(x) @ f64(w).T, rtol=0, atol=2e-6)
