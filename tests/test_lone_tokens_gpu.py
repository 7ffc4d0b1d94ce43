"""Steps of many decoding requests beside prompt portions: their tokens leave the prompt tiles for the split-key attention."""

import numpy as np
import pytest

from engine_helpers import bf16_atol, make_model, plain_logits, random_tokens

pytestmark = pytest.mark.gpu

VOCAB, DECODING = 331, 41              # (41 tokens of 4 heads are a wave of 148 pairs; their records are filled up to 48)


@pytest.fixture(scope="module")
def folder(tmp_path_factory):
    config = {"architectures": ["GPT2LMHeadModel"], "n_layer": 2, "n_embd": 256, "n_head": 4, "n_inner": 512, "vocab_size": VOCAB,
              "n_positions": 512, "activation_function": "gelu_new", "layer_norm_epsilon": 1e-5}
    return make_model(str(tmp_path_factory.mktemp("lone")), config, "gpt2", 5, sharpen=2.0)


# tiles of 128 tokens; units of two tiles; a step that is round already and needs no filler; several portions, one of a single token
@pytest.mark.parametrize("portions", [[60], [290], [128 - DECODING], [30, 1, 44]])
@pytest.mark.parametrize("graphs", [True, False])
def test_lone_tokens_beside_portions(folder, portions, graphs):
    from mini_llm_b200.engine import Engine, StepEntry
    engine = Engine(folder, dtype="bfloat16", page_size=16, cache_tokens=DECODING * 96 + 2 * 512, max_requests=DECODING + 4)
    engine.cuda_graphs = graphs
    requests = [random_tokens(i, 9 + 2 * (i % 30), VOCAB) for i in range(DECODING)]
    slots, prompt = [engine.open_request() for _ in requests], [len(r) - 6 for r in requests]
    for first in range(0, DECODING, 16):
        engine.step([StepEntry(slots[i], requests[i][:prompt[i]], []) for i in range(first, min(first + 16, DECODING))])
    singles = []
    run = engine._run

    def watched(ctx, sample_views):
        singles.append(ctx.n_att_singles)
        return run(ctx, sample_views)
    engine._run = watched
    lone = DECODING + portions.count(1)
    for step in range(5):                                    # eager (twice: the first one allocates), captured, replayed
        others = [random_tokens(1000 + 10 * step + j, n, VOCAB) for j, n in enumerate(portions)]
        opened = [engine.open_request() for _ in others]
        entries = [StepEntry(slots[i], [requests[i][prompt[i] + step]], [0]) for i in range(DECODING)]
        entries[7:7] = [StepEntry(slot, tokens, [len(tokens) - 1]) for slot, tokens in zip(opened, others)]
        logits = engine.step(entries).cpu().numpy()
        engine.check_status()
        wanted = [(requests[i][:prompt[i] + step + 1]) for i in range(DECODING)]
        wanted[7:7] = others
        for row, tokens in zip(logits, wanted):
            expected = plain_logits(folder, tokens, bf16_weights=True)
            assert np.abs(row - expected[-1]).max() <= bf16_atol(expected), (step, len(tokens))
        for slot in opened:
            engine.close_request(slot)
    assert all(lone <= n <= lone + 7 for n in singles), singles
    if graphs:
        assert engine.step_kinds["captured"] >= 1 and engine.step_kinds["replayed"] >= 1
