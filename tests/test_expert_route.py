"""Which kernels a step's experts go to, by the rule's sizes (no GPU)."""

import pytest
import torch

from mini_llm_b200.kernels import ops
from mini_llm_b200.kernels.dispatch import Kernels


@pytest.mark.parametrize("tokens, features, tables, eights, tiles", [
    (1, 3072, 9, True, True), (2, 1536, 17, True, True), (3, 3072, 9, True, False), (6, 3072, 9, True, False), (7, 3072, 9, True, True),
    (12, 1536, 17, True, False), (13, 1536, 17, True, True), (31, 1536, 17, True, True), (32, 1536, 17, True, False), (16, 3072, 65, True, False),
    (16, 3072, 9, False, False)])
def test_experts_go_to_tiles_where_pairs_would_take_more_than_one_wave(monkeypatch, tokens, features, tables, eights, tiles):
    seen = {}
    monkeypatch.setattr(ops, "experts", lambda *args, **how: seen.update(how))
    x, act = torch.zeros(tokens, 64, dtype=torch.bfloat16), torch.zeros(tokens * 3, 64, dtype=torch.bfloat16)
    inner_of = torch.zeros(tables, dtype=torch.int32)
    Kernels(torch.bfloat16).experts(None, act, x, None, None, None, None, None, None, inner_of, 64, 3, ld_down=64, eights=eights, features=features)
    assert seen["tiles"] is tiles
