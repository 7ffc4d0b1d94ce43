"""Products, norms and attention of few rows at the sizes where their tiles, shares of K and chunks end, against 64-bit sums."""

import math

import numpy as np
import pytest
import torch

import plain_gpt2 as plain
from test_kernels_gpu import attention_expected, dev, f64, paged_case, split_scratch, tol

pytestmark = pytest.mark.gpu


# rows: the few-row kernel's 1 to 8, then tiles of 64; features: a warp's, a block's and a tile's edges, four features a warp
# from 16,384 on; K: one 16-byte piece, less than a warp's share, shares that are no multiple of a load, K shared by 2, 4 and 8
@pytest.mark.parametrize("m", [1, 2, 3, 8, 9, 64, 65])
@pytest.mark.parametrize("n, k", [(1, 4), (63, 100), (65, 768), (768, 3076), (130, 516), (16385, 132)])
@pytest.mark.parametrize("epilogue", ["store", "add", "gelu_erf"])
def test_linear_in_32_bits(m, n, k, epilogue):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(m * 31 + n + k)
    a = dev(rng.normal(size=(m, k + 4)), torch.float32)[:, 4:]
    w, bias = dev(rng.normal(size=(n, k)) / math.sqrt(k), torch.float32), dev(rng.normal(size=n), torch.float32)
    out = dev(rng.normal(size=(m, n + 3)), torch.float32)
    before = f64(out)
    acc = f64(a) @ f64(w).T + f64(bias)
    expected = {"store": acc, "add": before[:, :n] + acc, "gelu_erf": plain.gelu_erf(acc)}[epilogue]
    ops.linear_plain(out[:, :n], a, w, bias, epilogue)
    # every product and every sum rounds by at most 2^-24 of values below 2^3; their roots-of-K walk stays under 2e-5
    np.testing.assert_allclose(f64(out)[:, :n], expected, rtol=0, atol=2e-5)
    np.testing.assert_array_equal(f64(out)[:, n:], before[:, n:])


def test_linear_in_32_bits_off_16_byte_boundaries_and_with_infinities():
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(8)
    base, w = dev(rng.normal(size=(5, 131)), torch.float32), dev(rng.normal(size=(70, 128)) / 11, torch.float32)
    out = torch.empty(5, 70, device="cuda")
    for a in (base[:, 1:129], base[:, 3:131]):            # rows that start on 4-byte boundaries only
        ops.linear_plain(out, a, w, None, "store")
        np.testing.assert_allclose(f64(out), f64(a) @ f64(w).T, rtol=0, atol=2e-5)
    a = dev(rng.normal(size=(3, 128)), torch.float32)
    a[1, 127] = math.inf                                  # stays in its row, and in no other share of K
    ops.linear_plain(out[:3], a, w, None, "store")
    np.testing.assert_array_equal(f64(out)[1], np.sign(f64(w)[:, 127]) * math.inf)
    assert np.isfinite(f64(out)[[0, 2]]).all()


@pytest.mark.parametrize("width", [4, 1020, 1024, 4096, 4100, 771])
def test_layernorm_in_32_bits(width):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(width)
    x = dev(rng.normal(3.0, 5.0, size=(5, width)), torch.float32)
    gain, shift = dev(rng.uniform(0.5, 1.5, width), torch.float32), dev(rng.normal(0, 0.1, width), torch.float32)
    out = torch.empty(3, width, device="cuda")
    ops.layernorm(out, x, gain, shift, 1e-5, dev([4, 0, 4], torch.int32))
    np.testing.assert_allclose(f64(out), plain.layer_norm(f64(x), f64(gain), f64(shift), 1e-5)[[4, 0, 4]], rtol=0, atol=tol(torch.float32, 4))


# every number of lanes a key, head sizes that leave lanes idle, one that no lane layout takes; 1 key up to several rounds
@pytest.mark.parametrize("head", [4, 12, 20, 32, 48, 64, 100, 128, 144, 10])
@pytest.mark.parametrize("window", [0, 33])
def test_attention_in_32_bits(head, window):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(head)
    k_pages, v_pages, table, positions, items, dense = paged_case(rng, [1, 37, 300, 64], [1, 5, 2, 1], 4, 2, head, 8, torch.float32)
    q = dev(rng.normal(size=(len(f64(positions)), 4 * head)), torch.float32)
    out = torch.full_like(q, float("nan"))
    expected = attention_expected(f64(q), dense, f64(positions).astype(int), f64(items).astype(int), 4, 2, head, head ** -0.5, window)
    ops.attention_plain(out, q, k_pages, v_pages, table, positions, items, 4, 2, head, 8, head ** -0.5, window)
    np.testing.assert_allclose(f64(out), expected, rtol=0, atol=tol(torch.float32))


@pytest.mark.parametrize("lengths, heads", [([9000, 3, 2200], 12), ([700] * 33, 16)])
def test_split_attention_with_more_keys_than_the_launch_has_chunks(lengths, heads):
    """A block table that reaches over a whole cache: a launch has far fewer chunks than the reach would take, and tokens that
    see more keys than those chunks hold at the asked length take longer ones."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(len(lengths))
    head, page, chunk = 64, 64, 64
    k_pages, v_pages, table, positions, items, dense = paged_case(rng, lengths, [1] * len(lengths), heads, heads, head, page, torch.bfloat16)
    dense = [(f64(dev(k, torch.bfloat16)), f64(dev(v, torch.bfloat16))) for k, v in dense]
    n, max_chunks = len(lengths), 1024
    table = torch.cat([table, torch.full((n, max_chunks - table.shape[1]), -1, dtype=torch.int32, device="cuda")], 1).contiguous()
    q = dev(rng.normal(size=(n, heads * head)), torch.bfloat16)
    out = torch.full_like(q, float("nan"))
    scratch = split_scratch(n, heads, max_chunks, head)
    expected = attention_expected(f64(q), dense, f64(positions).astype(int), f64(items).astype(int), heads, heads, head, head ** -0.5, 0)
    for _ in range(2):
        ops.split_attention(out, q, k_pages, v_pages, table, positions, items, heads, heads, head, page, head ** -0.5, 0, chunk,
                            max_chunks, *scratch)
        np.testing.assert_allclose(f64(out), expected, rtol=0, atol=tol(torch.bfloat16, 2))
        assert int(scratch[2].abs().sum()) == 0


def test_two_memory_shapes_share_scratch_without_moving_it():
    from mini_llm_b200.kernels.dispatch import Kernels
    kernels = Kernels(torch.bfloat16)
    first = kernels._memory_scratch("cuda", (100, 20, 30))
    second = kernels._memory_scratch("cuda", (50, 40, 10))
    moved = kernels.scratch_generation
    assert [t.numel() for t in second] == [100, 40, 30] and [t.numel() for t in first] == [100, 20, 30]
    for floats in ((100, 20, 30), (50, 40, 10)):
        assert kernels._memory_scratch("cuda", floats) is second
    assert kernels.scratch_generation == moved


# one expert and many, pairs that name none, inner sizes that end inside a tile of 16 features and a unit of 256, every form
@pytest.mark.parametrize("tokens, experts, top, inners, width, form", [
    (1, 8, 2, (24, 40), 64, "gated_silu"), (31, 3, 3, (264, 8), 768, "gated_silu"), (17, 40, 4, (512, 776), 72, "relu_squared"),
    (8, 5, 1, (16, 96), 1160, "clamped_glu"), (9, 1, 1, (256, 256), 8, "clamped_glu")])
def test_experts_in_tiles(tokens, experts, top, inners, width, form):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(tokens + experts)
    sizes = [inners[e % 2] for e in range(experts)]
    total, most = sum(sizes), max(sizes)
    x = dev(rng.normal(size=(tokens, width)), torch.bfloat16)
    gates, ups, downs = (dev(rng.normal(size=s) / math.sqrt(s[1]), torch.bfloat16) for s in ((total, width), (total, width), (width, total)))
    starts = np.cumsum([0] + sizes[:-1])
    chosen = np.stack([rng.permutation(experts)[:top] for _ in range(tokens)]).astype(np.int32)
    chosen[rng.random(chosen.shape) < 0.1] = -1
    in_weight, out_weight = rng.uniform(0.5, 1.0, (tokens, top)).astype(np.float32), rng.uniform(0.1, 1.0, (tokens, top)).astype(np.float32)
    before = rng.normal(size=(tokens, width)).astype(np.float32)
    constants = dict(limit=1.5, shared_limit=0.5, alpha=1.702, n_experts=experts - 1) if form == "clamped_glu" else {}
    expected = before.astype(np.float64)
    xs, gs, us, ds = f64(x), f64(gates), f64(ups), f64(downs)
    for t in range(tokens):
        for e, a, b in zip(chosen[t], in_weight[t], out_weight[t]):
            if e < 0:
                continue
            part = slice(starts[e], starts[e] + sizes[e])
            into = f64(dev(np.float32(a) * f64(x)[t].astype(np.float32), torch.bfloat16))
            g, u = gs[part] @ into, us[part] @ into
            if form == "gated_silu":
                act = g / (1 + np.exp(-g)) * u
            elif form == "relu_squared":
                act = np.maximum(u, 0) ** 2
            else:
                limit = 0.5 if e == experts - 1 else 1.5
                g = np.minimum(g, limit)
                act = g / (1 + np.exp(-1.702 * g)) * (np.clip(u, -limit, limit) + 1)
            expected[t] += b * (ds[:, part] @ act)
    at = lambda matrix, step: torch.tensor([matrix.data_ptr() + 2 * step * int(s) for s in starts], dtype=torch.int64, device="cuda")
    act = torch.full((tokens * top, most), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert ops.expert_tiles_take(x, act, experts, total)
    for tiles in (True, False):
        hidden = dev(before)
        ops.experts(hidden, act, x, dev(chosen.reshape(-1)), dev(in_weight.reshape(-1)), dev(out_weight.reshape(-1)),
                    at(gates, width) if form != "relu_squared" else None, at(ups, width), at(downs, 1), dev(np.array(sizes, np.int32)), most, top,
                    ld_down=total, form=form, tiles=tiles, **constants)
        # activations are rounded to 8 bits once: each of a sum's terms is off by 2^-9 of itself at most, and the largest sums here
        # hold 3 experts x 264 terms of squares' size 1 / 264
        np.testing.assert_allclose(f64(hidden), expected, rtol=0, atol=2e-2, err_msg=f"tiles={tiles}")


# what the launcher gives a whole tile row: groups of 1, 5, 64 and more heads; sizes that end inside a tile; each mask and option
@pytest.mark.parametrize("heads, kv_heads, dim, vdim, window, chunk, keep, cap, options", [
    (1, 1, 8, 8, 0, 0, 0, 0.0, ()), (5, 1, 64, 64, 0, 0, 0, 30.0, ("sink",)), (8, 4, 72, 56, 0, 32, 0, 0.0, ("gate",)),
    (64, 1, 24, 128, 65, 0, 7, 0.0, ("slopes", "gate_wide")), (70, 1, 128, 128, 1, 0, 130, 0.0, ("sink", "slopes")), (6, 6, 128, 40, 200, 0, 0, 5.0, ("gate",))])
def test_capped_attention_in_tensor_core_tiles(heads, kv_heads, dim, vdim, window, chunk, keep, cap, options):
    """Three requests' portions whose borders fall inside a block's rows, against one block per (token, head)."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(heads + dim)
    page, lengths, new = 16, [3, 210, 333], [3, 101, 64]
    blocks = [-(-n // page) for n in lengths]
    table = torch.zeros(3, max(blocks), dtype=torch.int32)
    order = rng.permutation(sum(blocks))
    for i, count in enumerate(blocks):
        table[i, :count] = torch.tensor(order[sum(blocks[:i]):sum(blocks[:i]) + count])
    k_pages, v_pages = (dev(rng.normal(size=(sum(blocks), page, kv_heads, d)), torch.bfloat16) for d in (dim, vdim))
    positions = dev(np.concatenate([np.arange(l - m, l) for l, m in zip(lengths, new)]).astype(np.int32))
    items = dev(np.repeat(np.arange(3), new).astype(np.int32))
    n = sum(new)
    q = dev(rng.normal(size=(n, heads * dim + 8)), torch.bfloat16)[:, 8:]
    how = dict(window=window, chunk=chunk, keep=keep, cap=cap)
    if "sink" in options:
        how["sink"] = dev(rng.normal(size=heads), torch.float32)
    if "slopes" in options:
        how["slopes"] = dev(rng.uniform(0, 0.5, heads), torch.float32)
    if "gate" in options or "gate_wide" in options:
        how.update(gate=dev(rng.normal(size=(n, heads * (vdim if "gate_wide" in options else 1))), torch.float32), gate_wide="gate_wide" in options)
    want, got = (torch.full((n, heads * vdim), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    for out, tiled in ((want, False), (got, True)):
        ops.capped_attention(out, q, k_pages, v_pages, table.cuda(), positions, items, heads, kv_heads, dim, vdim, page, dim ** -0.5, tiled=tiled, **how)
    # both keep scores, weights and sums in 32 bits, so they may differ by the last rounding to 8 bits: 2^-8 of values below 4
    np.testing.assert_allclose(f64(got), f64(want), rtol=2 ** -7, atol=2 ** -10)


@pytest.mark.parametrize("heads, rank, rot, window, gated", [(1, 128, 0, 0, False), (3, 128, 64, 50, True), (12, 256, 32, 0, False), (5, 256, 80, 1, True)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_latent_attention_in_tensor_core_tiles(heads, rank, rot, window, gated, out_dtype):
    """bfloat16 pages: portions that end inside a tile of 64 pairs and of 64 keys, against one block per (token, head)."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(heads + rank)
    page, lengths, new, row = 8, [331, 9, 64], [260, 9, 1], rank + rot
    blocks = [-(-n // page) for n in lengths]
    table = torch.zeros(3, max(blocks), dtype=torch.int32)
    order = rng.permutation(sum(blocks))
    for i, count in enumerate(blocks):
        table[i, :count] = torch.tensor(order[sum(blocks[:i]):sum(blocks[:i]) + count])
    pages = dev(rng.normal(size=(sum(blocks), page, 1, row)), torch.bfloat16)
    starts, offsets = [n - m for n, m in zip(lengths, new)], [0, 260, 269]
    positions = dev(np.concatenate([np.arange(s, l) for s, l in zip(starts, lengths)]).astype(np.int32))
    items, n = dev(np.repeat(np.arange(3), new).astype(np.int32)), sum(new)
    q = dev(rng.normal(size=(n, heads * row)) * 0.7, torch.float32)
    gate = dev(rng.normal(size=(n, heads)), torch.float32) if gated else None
    want, got = torch.empty(n, heads * rank, device="cuda"), torch.full((n, heads * rank), float("nan"), dtype=out_dtype, device="cuda")
    ops.latent_attention_plain(want, q, pages, table.cuda(), positions, items, heads, rank, rot, page, 0.1, window=window, gate=gate)
    tiles, _, _ = ops.attention_tiles(offsets, new, starts)
    ops.latent_attention_tiled(got, q, pages, table.cuda(), positions, items, heads, rank, rot, page, 0.1,
                               tiles=dev(np.array(tiles, dtype=np.int32)), n_tiles=len(tiles), window=window, gate=gate)
    # queries and weights keep all 24 bits and sums are 32-bit; a result of 16 bits is rounded once
    np.testing.assert_allclose(f64(got), f64(want), rtol=2 ** -8 if out_dtype == torch.bfloat16 else 2e-5, atol=3e-5)


# keys that fill a row and that end inside a 32-entry quarter, values that end inside a block's 16 columns; portions of one token, a chunk,
# a chunk and one, more than the rows' ring holds
@pytest.mark.parametrize("heads, qk_heads, dim, vdim, delta", [(2, 1, 40, 8, True), (3, 3, 64, 24, False), (4, 2, 128, 40, True), (2, 1, 96, 16, False)])
def test_recurrence_in_chunks_of_tokens(heads, qk_heads, dim, vdim, delta):
    recurrence_case(heads, qk_heads, dim, vdim, delta, ([17, 1, 32, 0], [129, 16, 1, 3]))


@pytest.mark.parametrize("heads, qk_heads, dim, vdim, delta", [(2, 1, 33, 33, True), (4, 2, 128, 32, False), (3, 3, 128, 65, True)])
def test_recurrence_of_few_tokens(heads, qk_heads, dim, vdim, delta):
    recurrence_case(heads, qk_heads, dim, vdim, delta, ([1, 0, 1, 1], [3, 1, 0, 2]))


def recurrence_case(heads, qk_heads, dim, vdim, delta, portions):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(dim + vdim)
    log_rate, bias, skip = (rng.normal(m, 1, heads).astype(np.float32).astype(np.float64) for m in (-1, 0, 0))
    state = dev(rng.normal(0, 0.3, (5, heads * dim * vdim)), torch.float32)
    slots, S = [3, 0, 4, 1], f64(state).reshape(5, heads, dim, vdim)
    for counts in portions:
        n = sum(counts)
        q, k, v = (dev(rng.normal(size=(n, size + 8)), torch.bfloat16)[:, :size] for size in (qk_heads * dim, qk_heads * dim, heads * vdim))
        gate_a, gate_b = dev(rng.normal(0, 2, (n, heads)), torch.float32), dev(rng.normal(0, 3, (n, heads)), torch.float32)
        expected, t = np.zeros((n, heads, vdim)), 0
        for slot, count in zip(slots, counts):
            for t in range(t, t + count):
                for head in range(heads):
                    g = head // (heads // qk_heads)
                    qt, kt, vt = f64(q)[t, g * dim:(g + 1) * dim], f64(k)[t, g * dim:(g + 1) * dim], f64(v)[t, head * vdim:(head + 1) * vdim]
                    step = np.log1p(np.exp(f64(gate_a)[t, head] + bias[head]))
                    a, b = np.exp(-np.exp(log_rate[head]) * step), step
                    if delta:
                        qt, kt, b = qt / np.sqrt(qt @ qt + 1e-6) * 0.5, kt / np.sqrt(kt @ kt + 1e-6), 1 / (1 + np.exp(-f64(gate_b)[t, head]))
                    S[slot, head] *= a
                    S[slot, head] += np.outer(kt, b * (vt - (S[slot, head].T @ kt if delta else 0)))
                    expected[t, head] = S[slot, head].T @ qt + (0 if delta else skip[head] * vt)
            t += count > 0
        out = torch.full((n, heads * vdim), float("nan"), device="cuda")
        offsets = np.cumsum([0] + counts[:-1])
        ops.linear_recurrence(out, q, k, v, gate_a, gate_b if delta else None, dev(log_rate, torch.float32), dev(bias, torch.float32), state,
                              dev(np.array(slots, np.int32)), dev(offsets.astype(np.int32)), dev(np.array(counts, np.int32)), heads, qk_heads, dim,
                              vdim, delta, unit_norm=delta, q_scale=0.5 if delta else 1.0, skip=None if delta else dev(skip, torch.float32))
        # sums of some hundred products of 32-bit numbers: their rounding follows the largest values that went into them
        np.testing.assert_allclose(f64(out), expected.reshape(n, -1), rtol=0, atol=4e-6 * max(1.0, np.abs(expected).max()))
        np.testing.assert_allclose(f64(state).reshape(S.shape), S, rtol=0, atol=4e-6 * max(1.0, np.abs(S).max()))


# keys that end at a tile's, a round's and a chunk's edges; few pairs (three stages) and more than a wave (two)
@pytest.mark.parametrize("head", [16, 64, 128, 256])
@pytest.mark.parametrize("times, chunk", [(1, 64), (1, 1024), (20, 1024)])
def test_split_attention_at_the_edges_of_its_tiles(head, times, chunk):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(head)
    lengths, heads, page = [1, 15, 16, 17, 63, 64, 65, 129] * times, 4, 16
    k_pages, v_pages, table, positions, items, dense = paged_case(rng, lengths, [1] * len(lengths), heads, heads, head, page, torch.bfloat16)
    dense = [(f64(dev(k, torch.bfloat16)), f64(dev(v, torch.bfloat16))) for k, v in dense]
    q = dev(rng.normal(size=(len(lengths), heads * head)), torch.bfloat16)
    max_chunks = -(-table.shape[1] * page // chunk)
    scratch, out = split_scratch(len(lengths), heads, max_chunks, head), torch.full_like(q, float("nan"))
    expected = attention_expected(f64(q), dense, f64(positions).astype(int), f64(items).astype(int), heads, heads, head, head ** -0.5, 0)
    ops.split_attention(out, q, k_pages, v_pages, table, positions, items, heads, heads, head, page, head ** -0.5, 0, chunk, max_chunks, *scratch)
    # weights and sums are 32-bit; the result is rounded to 8 bits once
    np.testing.assert_allclose(f64(out), expected, rtol=2 ** -8, atol=1e-5)
    assert int(scratch[2].abs().sum()) == 0


# rows of one and two tiles; features that end inside a tile, K shared by four, eight and sixteen warps and no multiple of a warp's share
@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n, k", [(5, 8), (24, 72), (1000, 2056), (3072, 768), (130, 4104)])
def test_few_row_products_at_the_edges_of_their_tiles(m, n, k):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(m + n + k)
    x, w = dev(rng.normal(size=(m, k)), torch.bfloat16), dev(rng.normal(size=(n, k)) / math.sqrt(k), torch.bfloat16)
    bias, out = dev(rng.normal(size=n), torch.float32), torch.full((m, n), float("nan"), device="cuda")
    ops.skinny_linear(out, x, w, bias, "store")
    np.testing.assert_allclose(f64(out), f64(x) @ f64(w).T + f64(bias), rtol=0, atol=2e-5)      # 32-bit sums of products of size 1 in all


@pytest.mark.parametrize("m, heads, n, k", [(1, 12, 64, 256), (16, 3, 256, 72), (9, 5, 20, 8)])
def test_few_row_products_per_head(m, heads, n, k):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(n + k)
    a, w = dev(rng.normal(size=(m, heads * k + 8)), torch.bfloat16)[:, 8:], dev(rng.normal(size=(heads, n, k)) / math.sqrt(k), torch.bfloat16)
    out = torch.full((m, heads * n), float("nan"), device="cuda")
    assert ops.skinny_heads_takes(a, w, k)
    ops.skinny_heads(out, a, w, heads, k, n)
    np.testing.assert_allclose(f64(out).reshape(m, heads, n), np.einsum("mhk,hnk->mhn", f64(a).reshape(m, heads, k), f64(w)), rtol=0, atol=2e-5)


@pytest.mark.parametrize("heads, kv_heads, window", [(4, 4, 0), (6, 2, 30)])
def test_split_attention_of_the_tokens_a_work_list_names(heads, kv_heads, window):
    """Lone tokens beside a portion, by their records at an odd place of the list, one of them twice; the portion's rows stay as they are."""
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(heads)
    lengths, new, head, page = [40, 1, 300, 77, 2], [1, 1, 90, 1, 1], 64, 16
    k_pages, v_pages, table, positions, items, dense = paged_case(rng, lengths, new, heads, kv_heads, head, page, torch.bfloat16)
    dense = [(f64(dev(k, torch.bfloat16)), f64(dev(v, torch.bfloat16))) for k, v in dense]
    q = dev(rng.normal(size=(sum(new), heads * head)), torch.bfloat16)
    offsets = np.cumsum([0] + new[:-1])
    alone = [3, 0, 4, 1, 3]
    records = [(9, 9, 9, 9, 9, 9, 9, 9)] + [(i, offsets[i], 1, lengths[i] - 1, 0, 1, 0, 1) for i in alone]
    expected = attention_expected(f64(q), dense, f64(positions).astype(int), f64(items).astype(int), heads, kv_heads, head, head ** -0.5, window)
    for chunk in (32, 1024):
        max_chunks = -(-table.shape[1] * page // chunk)
        out, scratch = torch.full_like(q, 7.0), split_scratch(len(alone), heads, max_chunks, head)
        ops.split_attention(out, q, k_pages, v_pages, table, positions, items, heads, kv_heads, head, page, head ** -0.5, window, chunk, max_chunks,
                            *scratch, records=dev(np.array(records, np.int32)).reshape(-1)[8:], n_records=len(alone))
        rows = sorted({int(offsets[i]) for i in alone})
        np.testing.assert_allclose(f64(out)[rows], expected[rows], rtol=2 ** -8, atol=1e-5)      # rounded to 8 bits once
        assert (np.delete(f64(out), rows, axis=0) == 7.0).all()


# tokens: an eighth's edges, every number of token tiles, shared by one and two blocks; features: less than a tile, its edges; K: one
# 16-byte piece, less than a block of 32 a warp, shares that end inside one, a cluster's shares of unequal length
@pytest.mark.parametrize("m", [1, 16, 17, 24, 25, 33, 48, 49, 64])
@pytest.mark.parametrize("n, k", [(16, 8), (50, 264), (768, 768), (100, 2056)])
@pytest.mark.parametrize("epilogue", ["add", "store", "gelu_tanh"])
def test_narrow_products(m, n, k, epilogue):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(m * 7 + n + k)
    a = dev(rng.normal(size=(m, k + 8)), torch.bfloat16)[:, 8:]
    w, bias = dev(rng.normal(size=(n, k)) / math.sqrt(k), torch.bfloat16), dev(rng.normal(size=n), torch.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    acc = f64(a) @ f64(w).T + f64(bias)
    for shares in (0, 100):
        for tiles in (10, 20, 30):
            for blocks in (1, 2, 4):
                out = torch.full((m + 1, n + 4), 0.5, dtype=torch.bfloat16 if epilogue == "gelu_tanh" else torch.float32, device="cuda")
                ops.gemm_bf16_tile(out[:m, :n], a, w, bias, epilogue, status, 8000 + shares + tiles + blocks)
                expected = {"add": 0.5 + acc, "store": acc, "gelu_tanh": plain.gelu_tanh(acc)}[epilogue]
                # sums: 2,056 terms whose sizes add up to 30, each cut off at 2^-23 of them, and with gelu a result rounded to
                # 8 bits and a tanh of 2^-11, of values up to 6
                np.testing.assert_allclose(f64(out)[:m, :n], expected, rtol=0, atol=2e-5 if epilogue != "gelu_tanh" else 0.03)
                assert bool((out[m] == 0.5).all()) and bool((out[:m, n:] == 0.5).all())
    assert int(status) == 0


# both sides of the line between narrow and swapped tiles: blocks that fit the SMs at once, a second round of them, a long K that blocks share or not
@pytest.mark.parametrize("m, n, k", [(17, 9472, 64), (17, 9480, 64), (33, 7104, 72), (64, 4096, 2048), (64, 7120, 64), (24, 1600, 6400), (24, 4096, 6400), (16, 16376, 64)])
def test_products_at_the_edge_of_the_narrow_tiles(m, n, k):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(m + n + k)
    a, w = dev(rng.normal(size=(m, k)), torch.bfloat16), dev(rng.normal(size=(n, k)) / math.sqrt(k), torch.bfloat16)
    status, out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((m + 1, n), 0.5, device="cuda")
    ops.gemm_bf16(out[:m], a, w, None, "add", status)
    # (as above: 6,400 terms whose sizes add up to 80)
    np.testing.assert_allclose(f64(out)[:m], 0.5 + f64(a) @ f64(w).T, rtol=0, atol=1e-4)
    assert bool((out[m] == 0.5).all()) and int(status) == 0


# widths: a ring that holds all of K, rows whose end is no block of 32 of K, rows of two rounds of the second kernel's blocks, which other kernels
# take; tokens: of which nearly every expert has one and hardly any, tiles of 8, 16 and 32 pairs
@pytest.mark.parametrize("tokens, experts, top, inner, width", [(1, 24, 1, 40, 768), (2, 8, 2, 136, 776), (16, 3, 2, 264, 1000), (31, 2, 2, 72, 1032),
                                                                (9, 4, 2, 80, 2056), (31, 5, 1, 48, 4096), (3, 40, 2, 64, 2048)])
@pytest.mark.parametrize("gated", [True, False])
def test_experts_in_tiles_of_other_widths(tokens, experts, top, inner, width, gated):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(tokens + width)
    total = experts * inner
    ups = dev(rng.normal(size=((2 if gated else 1) * total, width)) / math.sqrt(width), torch.bfloat16)
    downs = dev(rng.normal(size=(width, total)) / math.sqrt(inner), torch.bfloat16)
    x = dev(rng.normal(size=(tokens, width)), torch.bfloat16)
    chosen = np.stack([rng.permutation(experts)[:top] for _ in range(tokens)]).astype(np.int32)
    weights = rng.uniform(0.5, 1.5, size=(tokens, top)).astype(np.float32)
    table = lambda matrix, first, step: torch.tensor([matrix.data_ptr() + 2 * (first + e * step) for e in range(experts)], dtype=torch.int64, device="cuda")
    act = torch.full((tokens * top, inner), math.nan, dtype=torch.bfloat16, device="cuda")
    hidden = dev(rng.normal(size=(tokens, width)), torch.float32)
    expected = f64(hidden)
    up, down, rows = f64(ups)[-total:], f64(downs), f64(x)
    for t in range(tokens):
        for k, e in enumerate(chosen[t]):
            at = slice(e * inner, (e + 1) * inner)
            u = up[at] @ rows[t]
            if gated:
                g = f64(ups)[at] @ rows[t]
                u = g / (1.0 + np.exp(-g)) * u
            else:
                u = np.maximum(u, 0.0) ** 2
            expected[t] += weights[t, k] * (down[:, at] @ f64(dev(u, torch.bfloat16)))
    ops.experts(hidden, act, x, dev(chosen.reshape(-1)), dev(np.ones(tokens * top), torch.float32), dev(weights.reshape(-1), torch.float32),
                table(ups, 0, inner * width) if gated else None, table(ups, (total if gated else 0) * width, inner * width), table(downs, 0, inner),
                dev(np.full(experts, inner, np.int32)), inner, top, ld_down=total, tiles=True, n_experts=experts)
    # of the activations, of size 1, one in some thousands rounds the other way (2^-8 of it): far below 1e-3 of the sums
    assert np.linalg.norm(f64(hidden) - expected) <= 1e-3 * np.linalg.norm(expected)
    assert np.abs(f64(hidden) - expected).max() <= 0.03


# more units of all experts than there is room for, chosen by few tokens and by many; tables of nearly 64 experts, whose rows are all warps' or nearly so
@pytest.mark.parametrize("tokens, experts, top, inner, width", [(13, 24, 2, 768, 768), (31, 24, 2, 768, 768), (2, 60, 4, 256, 1024), (20, 64, 4, 264, 1184)])
def test_experts_of_more_units_than_there_is_room_for(tokens, experts, top, inner, width):
    test_experts_in_tiles_of_other_widths(tokens, experts, top, inner, width, True)


# tokens that name their experts again and again, on both sides of what shared memory holds beside the weights
@pytest.mark.parametrize("top, width", [(150, 1184), (160, 1184)])
def test_experts_named_by_a_token_many_times(top, width):
    from mini_llm_b200.kernels import ops
    tokens, experts, inner = 31, 40, 16
    rng = np.random.default_rng(top)
    ups, downs = (dev(rng.normal(size=shape) / math.sqrt(shape[1]), torch.bfloat16) for shape in ((experts * inner, width), (width, experts * inner)))
    x = dev(rng.normal(size=(tokens, width)), torch.bfloat16)
    chosen = rng.integers(0, experts, size=(tokens, top)).astype(np.int32)
    weights = rng.uniform(0.5, 1.5, size=(tokens, top)).astype(np.float32)
    table = lambda matrix, step: torch.tensor([matrix.data_ptr() + 2 * e * step for e in range(experts)], dtype=torch.int64, device="cuda")
    act, hidden = torch.full((tokens * top, inner), math.nan, dtype=torch.bfloat16, device="cuda"), dev(rng.normal(size=(tokens, width)), torch.float32)
    rows = f64(dev(np.maximum(f64(x) @ f64(ups).T, 0.0) ** 2, torch.bfloat16))
    of_pairs = np.zeros((tokens, experts))
    np.add.at(of_pairs, (np.arange(tokens)[:, None], chosen), weights)
    expected = f64(hidden) + (rows * np.repeat(of_pairs, inner, axis=1)) @ f64(downs).T
    ops.experts(hidden, act, x, dev(chosen.reshape(-1)), dev(np.ones(tokens * top), torch.float32), dev(weights.reshape(-1), torch.float32), None,
                table(ups, inner * width), table(downs, inner), dev(np.full(experts, inner, np.int32)), inner, top, ld_down=experts * inner, tiles=True, n_experts=experts)
    # (as above: activations rounded to 8 bits, some the other way)
    assert np.linalg.norm(f64(hidden) - expected) <= 1e-3 * np.linalg.norm(expected)


@pytest.mark.parametrize("ints", [4, 1020, 4096, 4100, 70000])       # a piece, a thread's, a block's and all blocks' edges
def test_control_block_from_the_ring(ints):
    from mini_llm_b200.kernels import ops
    parts, step = 3, ints + 8
    ring = torch.arange(parts * step, dtype=torch.int32).pin_memory()
    steps, block = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.empty(ints + 4, dtype=torch.int32, device="cuda")
    for taken in range(5):
        block.fill_(-1)
        ops.control(block, ops.device_address(ring), step, parts, steps, ints)
        start = taken % parts * step
        assert bool((block[:ints].cpu() == ring[start:start + ints]).all()) and bool((block[ints:] == -1).all())
        assert steps.tolist() == [(taken + 1) % parts, 0]


def test_an_emptied_slot_and_draws_on_the_host():
    from mini_llm_b200.kernels import ops
    states = [torch.ones(3, 5, 8, 16, device="cuda"), torch.ones(1, 5, 7, dtype=torch.bfloat16, device="cuda"), torch.ones(2, 5, 3, dtype=torch.int32, device="cuda")]
    table = torch.tensor([[s.data_ptr(), s.shape[0], s.stride(0) * s.element_size(), s.stride(1) * s.element_size()] for s in states],
                         dtype=torch.int64, device="cuda")
    for slot in (4, 0):
        ops.zero_slot(table, slot)
    for s in states:
        assert bool((s[:, [0, 4]] == 0).all()) and bool((s[:, 1:4] == 1).all())
    ids, words = torch.full((2, 200), -1, dtype=torch.int32).pin_memory(), torch.zeros(2, dtype=torch.int32).pin_memory()
    kept, status = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.tensor([7], dtype=torch.int32, device="cuda")
    slots, tokens = dev(np.arange(130) % 9 - 4, torch.int32), dev(np.arange(130) + 50, torch.int32)
    for turn in (0, 1):
        ops.keep_tokens(kept, slots, tokens + turn, (ops.device_address(ids), 200, ops.device_address(words), dev([turn], torch.int32), status))
    torch.cuda.synchronize()
    for turn in (0, 1):
        assert ids[turn].tolist() == [50 + turn + r for r in range(130)] + [-1] * 70
    assert words.tolist() == [7, 7]


# a cluster's share of the keys: none for most blocks, one tile's edges, two tiles and one more, a ring that is asked for again; windows that
# cut the first tile; the token's own row in the first, the second and a later tile of its block; all numbers of blocks a cluster has
@pytest.mark.parametrize("tokens, heads, rank, rot, window", [(1, 12, 256, 32, 0), (3, 16, 256, 64, 70), (5, 3, 128, 0, 0), (19, 5, 128, 48, 0), (40, 12, 256, 32, 33), (90, 2, 128, 16, 0),
                                                              (150, 1, 128, 32, 200)])
@pytest.mark.parametrize("ahead", [True, False])
def test_latent_attention_of_single_tokens(tokens, heads, rank, rot, window, ahead, most_blocks=0):
    from mini_llm_b200.kernels import ops
    rng = np.random.default_rng(tokens + rank)
    page, row = 16, rank + rot
    lengths = [(1, 32, 33, 64, 65, 512, 513, 1030, 1500)[i % 9] + i // 9 for i in range(tokens)]
    blocks = [-(-n // page) for n in lengths]
    order = rng.permutation(sum(blocks))
    table = np.full((tokens, max(blocks)), -1, dtype=np.int32)
    for i, count in enumerate(blocks):
        table[i, :count] = order[sum(blocks[:i]):sum(blocks[:i]) + count]
    pages = dev(rng.normal(size=(sum(blocks), page, 1, row)), torch.bfloat16)
    for i, n in enumerate(lengths):                       # what lies past a request's end must not matter
        pages[table[i, -(-n // page) - 1], (n - 1) % page + 1:] = math.nan
    q, gate = dev(rng.normal(size=(tokens, heads * row)) * 0.7, torch.float32), dev(rng.normal(size=(tokens, heads)), torch.float32)
    common = (q, pages, dev(table, torch.int32), dev(np.array(lengths) - 1, torch.int32), dev(np.arange(tokens), torch.int32), heads, rank, rot, page, 0.1)
    got = torch.full((tokens, heads * rank), math.nan, device="cuda")
    scratch = (torch.empty(tokens * heads * 2 * rank, device="cuda"), torch.empty(tokens * heads * 4, device="cuda"))
    ops.latent_attention_tiled(got, *common, parts=2, scratch=scratch, window=window, gate=gate, rows_ahead=ahead, most_blocks=most_blocks)
    for i, n in enumerate(lengths):
        rows = f64(pages[table[i, :blocks[i]]]).reshape(-1, row)[max(0, n - window) if window else 0:n]
        s = f64(q)[i].reshape(heads, row) @ rows.T * 0.1
        w = np.exp(s - s.max(axis=1, keepdims=True))
        want = w / w.sum(axis=1, keepdims=True) @ rows[:, :rank] / (1.0 + np.exp(-f64(gate)[i]))[:, None]
        # queries and weights keep all 24 bits and sums are 32-bit: scores of up to 8 off by some 2^-21, weights by as much
        np.testing.assert_allclose(f64(got)[i].reshape(heads, rank), want, rtol=2e-5, atol=1e-5)


# clusters smaller than the launcher would take (on a part of a device that refuses 16 blocks they are of 8); rows of more than 320 entries, of which one
# block fits an SM, and the widest ones
@pytest.mark.parametrize("tokens, heads, rank, rot, window, most_blocks", [(3, 12, 256, 32, 0, 8), (5, 7, 128, 16, 40, 4), (2, 16, 256, 32, 0, 2), (2, 3, 128, 0, 0, 1),
                                                                           (3, 12, 256, 80, 0, 0), (2, 16, 128, 384, 0, 0), (20, 16, 256, 256, 90, 0), (80, 4, 256, 112, 0, 0)])
def test_latent_attention_of_single_tokens_in_other_clusters(tokens, heads, rank, rot, window, most_blocks):
    test_latent_attention_of_single_tokens(tokens, heads, rank, rot, window, True, most_blocks)
