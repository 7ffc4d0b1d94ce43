"""Kernels that read ahead of the wait for the kernels ahead: what the kernel right before them on the stream still writes must be taken
behind the wait.  The producer and the kernel are launched as dependents behind products that keep some of the SMs busy, from a replayed
graph, over memory that holds NaN wherever the producer writes."""

import math

import numpy as np
import pytest
import torch

from engine_helpers import random_tokens, run_schedule, schedule_mixed, schedule_tail_one_by_one
from test_kernels_gpu import dev, f64, paged_case, split_scratch

pytestmark = pytest.mark.gpu


def replays(before, launches, after, times=40):
    """``before`` (torch operations), then what a step begins with and busy products, then ``launches`` (the producer, the kernel), from a
    graph; ``after`` looks at the result of every replay."""
    from mini_llm_b200.kernels import ops
    status, ids = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(8, dtype=torch.int32, device="cuda")
    x, w = (torch.ones(shape, dtype=torch.bfloat16, device="cuda") for shape in ((64, 2048), (8192, 2048)))
    busy = torch.empty(64, 8192, dtype=torch.bfloat16, device="cuda")

    def step():
        before()
        ops.resolve_tokens(ids, ids)                      # (launched behind the kernels ahead, as a step's first kernels are)
        for _ in range(2):
            ops.gemm_bf16(busy, x, w, None, "store", status)
        launches()

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), ops.launches_on_current_stream():
        step()
        torch.cuda.synchronize()
        after()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            step()
        for _ in range(times):
            graph.replay()
            stream.synchronize()
            after()


def seen_keys(p, window, keep):
    low = max(0, p - window + 1) if window else 0
    return list(range(min(keep, low))) + list(range(low, p + 1))


# entries of one new token and of several, one that begins at nothing, new ones at a tile's and a page's edges, tokens whose own keys lie in the
# first tiles and far behind them; windows that let the first keys stay, which are new ones where an entry is that short.  times: eight warps
# a block, four of three stages, four of two; heads of whole and of partial rows
@pytest.mark.parametrize("head, value", [(64, 64), (64, 48), (16, 16), (128, 128), (256, 240)])
@pytest.mark.parametrize("window, keep", [(0, 0), (24, 8)])
@pytest.mark.parametrize("times, chunk", [(1, 32), (1, 1024), (6, 1024), (8, 1024)])
def test_split_attention_takes_a_step_s_own_keys_behind_the_wait(head, value, window, keep, times, chunk):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(head + value + times)
    lengths, new, heads, page = [1, 5, 17, 64, 130, 300, 33, 260] * times, [1, 5, 1, 2, 1, 1, 3, 1] * times, 5, 16
    k_pages, v_pages, table, positions, items, dense = paged_case(rng, lengths, new, heads, heads, head, page, torch.bfloat16)
    v_pages = v_pages.reshape(-1, heads, head)[:, :, :value].reshape(-1, page, heads * value).contiguous()
    n, at, who = sum(new), f64(positions).astype(int), f64(items).astype(int)
    qkv = torch.zeros(n, heads * (2 * head + value), dtype=torch.bfloat16, device="cuda")
    qkv[:, :heads * head] = dev(rng.normal(size=(n, heads * head)), torch.bfloat16)
    k_holes, v_holes = k_pages.clone(), v_pages.clone()
    for t in range(n):
        row = int(table[who[t], at[t] // page]), at[t] % page
        qkv[t, heads * head:2 * heads * head], qkv[t, 2 * heads * head:] = k_pages[row], v_pages[row]
        k_holes[row], v_holes[row] = math.nan, math.nan
    max_chunks = -(-table.shape[1] * page // chunk)
    scratch, out = split_scratch(n, heads, max_chunks, head), torch.empty(n, heads * value, dtype=torch.bfloat16, device="cuda")
    first_new, no_turns = dev(np.array(lengths) - np.array(new), torch.int32), torch.zeros(1, dtype=torch.float64, device="cuda")
    expected = np.zeros((n, heads, value))
    for t in range(n):
        k, v = (f64(dev(side, torch.bfloat16)).reshape(-1, heads, head)[seen_keys(at[t], window, keep)] for side in dense[who[t]])
        s = np.einsum("jhd,hd->hj", k, f64(qkv)[t, :heads * head].reshape(heads, head)) * head ** -0.5
        weights = np.exp(s - s.max(axis=1, keepdims=True))
        expected[t] = np.einsum("hj,jhd->hd", weights / weights.sum(axis=1, keepdims=True), v[:, :, :value])

    def before():
        k_pages.copy_(k_holes)
        v_pages.copy_(v_holes)
        out.fill_(math.nan)

    def launches():
        ops.rotary_store(qkv, heads * head, 2 * heads * head, heads, heads, head, value, 0, no_turns, 1.0, positions, items, table, page, k_pages, v_pages)
        ops.split_attention(out, qkv[:, :heads * head], k_pages, v_pages, table, positions, items, heads, heads, head, page, head ** -0.5, window, chunk, max_chunks, *scratch,
                            value_size=value, keep=keep, first_new=first_new)

    # weights and sums are 32-bit; the result is rounded to 8 bits once
    replays(before, launches, lambda: np.testing.assert_allclose(f64(out).reshape(n, heads, value), expected, rtol=2 ** -8, atol=1e-5), times=10)


def same_as_one_after_the_other(before, launches, *outputs):
    """The outputs of ``launches(True)``, reading ahead, are those of ``launches(False)`` with a wait of the host between the kernels, bit for bit."""
    before()
    for launch in launches(False):
        torch.cuda.synchronize()
        launch()
    torch.cuda.synchronize()
    expected = [out.clone() for out in outputs]
    assert all(bool(torch.isfinite(out).all()) for out in expected)

    def after():
        for out, was in zip(outputs, expected):
            assert torch.equal(out, was)

    def both():
        for launch in launches(True):
            launch()

    replays(before, both, after)


@pytest.mark.parametrize("heads, rank, rot, window", [(12, 256, 32, 0), (16, 128, 64, 40)])
def test_latent_attention_takes_the_token_s_row_behind_the_wait(heads, rank, rot, window):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(rank)
    lengths, page, dim = [1, 2, 31, 32, 33, 64, 65, 400, 1030], 16, 8
    n, row = len(lengths), rank + rot
    blocks = [-(-length // page) for length in lengths]
    order, table = rng.permutation(sum(blocks)), np.full((n, max(blocks)), -1, dtype=np.int32)
    for i, count in enumerate(blocks):
        table[i, :count] = order[sum(blocks[:i]):sum(blocks[:i]) + count]
    pages = dev(rng.normal(size=(sum(blocks), page, 1, row)), torch.bfloat16)
    for i, length in enumerate(lengths):
        pages[table[i, (length - 1) // page], (length - 1) % page:] = math.nan
    holes, q_eff, out = pages.clone(), dev(rng.normal(size=(n, heads * row)), torch.float32), torch.empty(n, heads * rank, device="cuda")
    down, gain = dev(rng.normal(size=(n, row)), torch.float32), dev(rng.uniform(0.5, 1.5, rank), torch.float32)
    q, turns = dev(rng.normal(size=(n, heads * (dim + rot))), torch.bfloat16), dev(1.0 / 100.0 ** (np.arange(rot // 2) / (rot // 2)), torch.float64)
    q_holes = q_eff.reshape(n, heads, row).clone()
    q_holes[:, :, rank:] = math.nan
    places, who, table = dev(np.array(lengths) - 1, torch.int32), dev(np.arange(n), torch.int32), dev(table, torch.int32)
    assert ops.latent_step_takes(q_eff, pages, heads, rank, rot)

    def before():
        pages.copy_(holes)
        q_eff.copy_(q_holes.reshape(n, -1))
        out.fill_(math.nan)

    def launches(ahead):
        return [lambda: ops.latent_prepare(pages, q_eff, down, q, gain, turns, places, who, table, page, rank, rot, rot, heads, dim, 1e-5),
                lambda: ops.latent_attention_tiled(out, q_eff, pages, table, places, who, heads, rank, rot, page, 0.1, window=window, rows_ahead=ahead)]

    same_as_one_after_the_other(before, launches, out)


def recurrent_rows(rng, n, sizes):
    """A product that writes [q | k | v] side by side, its inputs, and the three views."""
    from mini_llm_b200.kernels import ops
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    x, w = dev(rng.normal(size=(n, 256)), torch.bfloat16), dev(rng.normal(size=(sum(sizes), 256)) / 16, torch.bfloat16)
    rows = torch.empty(n, sum(sizes), dtype=torch.bfloat16, device="cuda")
    views = torch.split(rows, list(sizes), dim=1)
    return rows, views, lambda: ops.gemm_bf16(rows, x, w, None, "store", status)


def places_of(n):
    return dev(np.arange(n)[::-1] + 1, torch.int32), dev(np.arange(n), torch.int32), dev(np.ones(n), torch.int32)


@pytest.mark.parametrize("heads, dim, vdim, gated", [(4, 96, 192, True), (2, 64, 320, True), (12, 64, 64, False)])
def test_matrix_memories_take_a_token_s_rows_behind_the_wait(heads, dim, vdim, gated):
    from mini_llm_b200.kernels import ops
    rng, n = np.random.default_rng(dim), 5
    rows, (q, k, v), product = recurrent_rows(rng, n, (heads * dim, heads * dim, heads * vdim))
    start = dev(rng.normal(size=(n + 2, ops.memory_state_floats(heads, dim, vdim, gated))), torch.float32)
    state, out, places = start.clone(), torch.empty(n, heads * vdim, device="cuda"), places_of(n)
    how = dict(gates=dev(rng.normal(size=(n, 2 * heads)), torch.float32), gate_bias=torch.zeros(2 * heads, device="cuda"), gate_cap=15.0, q_scale=0.1) if gated \
        else dict(decay=dev(rng.uniform(0.5, 1, heads), torch.float32), silu=True)

    def before():
        state.copy_(start)
        rows.fill_(math.nan)

    same_as_one_after_the_other(before, lambda ahead: [product, lambda: ops.memory_scan(out, q, k, v, state, *places, heads, dim, vdim, state_ahead=ahead, **how)],
                                out, state)


@pytest.mark.parametrize("heads, dim, vdim, delta, channel", [(6, 128, 128, True, False), (6, 128, 128, True, True), (24, 128, 64, False, False)])
def test_recurrences_take_a_token_s_rows_behind_the_wait(heads, dim, vdim, delta, channel):
    from mini_llm_b200.kernels import ops
    rng, n, qk_heads = np.random.default_rng(dim + vdim), 3, heads // 3
    rows, (q, k, v), product = recurrent_rows(rng, n, (qk_heads * dim, qk_heads * dim, heads * vdim))
    start = dev(rng.normal(size=(n + 2, heads * dim * vdim)), torch.float32)
    state, out, places = start.clone(), torch.empty(n, heads * vdim, device="cuda"), places_of(n)
    rates = heads * dim if channel else heads
    gate_a, gate_b = dev(rng.normal(size=(n, rates)), torch.float32), dev(rng.normal(size=(n, heads)), torch.float32)
    log_rate, bias = dev(rng.normal(-1, 1, heads), torch.float32), dev(rng.normal(size=rates), torch.float32)

    def before():
        state.copy_(start)
        rows.fill_(math.nan)

    def launches(ahead):
        return [product, lambda: ops.linear_recurrence(out, q, k, v, gate_a, gate_b if delta else None, log_rate, bias, state, *places, heads, qk_heads, dim, vdim,
                                                       delta, unit_norm=delta, channel_decay=channel, state_ahead=ahead)]

    same_as_one_after_the_other(before, launches, out, state)


# ---- whole steps ---------------------------------------------------------------------------------------------------

def stacks():
    """Layers whose single tokens take the kernels that read ahead: a latent of 128 in a cluster, matrix memories, recurrences of few
    tokens, rotations and norms that store keys, experts in tiles; two of them over another layer's rows."""
    import deluvik_helpers as dh
    import fuvolix_helpers as fh
    import kerepel_helpers as kh
    import lipulorn_helpers as lh
    import nufavik_helpers as nh
    import sumozen_helpers as sh
    latent = dict(heads=4, dim=16, rot_dim=16, vdim=16, kv_rank=112 + 16)
    return {
        "fuvolix": (fh, fh.config([fh.latent(**latent, ff=128), fh.mlstm(heads=2, dim=32, vdim=64), fh.lightning(heads=4, dim=16, vdim=16, ff=128)] * 2, width=128, groups=4)),
        "lipulorn": (lh, lh.config([lh.latent(**latent, q_rank=32, window=30), lh.attention(heads=4, dim=16, vdim=16, chunk=32), lh.delta(heads=4, dim=32, vdim=32, a_rank=16, g_rank=16),
                                    lh.latent(**latent, q_rank=32, window=40, kv_from=0)], width=128)),
        "sumozen": (sh, sh.config([sh.parallel(dim=32, vdim=32, r_dim=32, r_vdim=32, mlp=sh.moe(ff=64, shared=128)), sh.mamba(heads=4, vdim=32, state=32, norm_groups=2, mlp=sh.moe(ff=64, shared=128))] * 2, width=128)),
        "deluvik": (dh, dh.full_stack()), "kerepel": (kh, kh.full_stack(width=128, side=16)), "nufavik": (nh, nh.full_stack()),
    }


@pytest.mark.parametrize("name", ["fuvolix", "lipulorn", "sumozen", "deluvik", "kerepel", "nufavik"])
def test_architectures_launched_as_dependents_give_the_same_logits(tmp_path, name):
    """With dependent launches and without, bit for bit: portions beside decoding requests, requests that come and go in the same slots, and runs
    of single tokens, which are replayed from graphs."""
    from mini_llm_b200.engine import Engine
    from mini_llm_b200.kernels import ops
    helpers, raw = stacks()[name]
    folder = helpers.make_model(str(tmp_path / "m"), raw, seed=7)
    requests = {f"r{i}": random_tokens(60 + i, n, 211) for i, n in enumerate((90, 14, 45, 70))}
    results = {}
    try:
        for on in (True, False):
            ops.set_dependent_launch(on)
            engine = Engine(folder, dtype="bfloat16", page_size=16, cache_tokens=1024, max_requests=4)
            got = run_schedule(engine, requests, schedule_mixed(requests, {"r0": 60, "r1": 5, "r2": 31, "r3": 40}, max_live=3, portion_sizes=(33, 3, 17)))
            again = run_schedule(engine, requests, schedule_tail_one_by_one(requests, tail=12))
            engine.check_status()
            assert engine.step_kinds["replayed"] > 0
            results[on] = {(run, n): rows for run, side in (("mixed", got), ("tail", again)) for n, rows in side.items()}
            del engine
    finally:
        ops.set_dependent_launch(True)
    for key, rows in results[True].items():
        assert np.isfinite(rows).all() and np.array_equal(rows, results[False][key]), key


def test_an_embedding_that_does_not_say_how_it_begins_has_a_kernel_put_before_it(tmp_path):
    import fuvolix_helpers as fh
    from mini_llm_b200.engine import Engine, StepEntry
    folder = fh.make_model(str(tmp_path / "m"), fh.full_stack(), seed=3)
    tokens, rows = random_tokens(5, 30, 211), {}
    for says in (True, False):
        engine = Engine(folder, dtype="bfloat16", page_size=16, cache_tokens=256, max_requests=1)
        assert engine.model.begins_apart
        engine.model.begins_apart = says
        resolved, real = [], engine.kernels.resolve_tokens
        engine.kernels.resolve_tokens = lambda *a: resolved.append(1) or real(*a)
        slot = engine.open_request()
        rows[says] = [engine.step([StepEntry(slot, part, [len(part) - 1])]).cpu().numpy() for part in (tokens[:20], tokens[20:21], tokens[21:22], tokens[22:23])]
        assert bool(resolved) == (not says)
    for one, other in zip(rows[True], rows[False]):
        assert np.array_equal(one, other)
