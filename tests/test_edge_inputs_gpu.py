"""Inputs that real ones turn into when something upstream goes wrong, and steps of unusual make-up: rows that are no numbers,
infinities, experts named twice, and as many entries as do not fit the GPU at once."""

import math

import numpy as np
import pytest
import torch

from test_kernels_gpu import dev, f64

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
