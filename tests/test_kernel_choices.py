"""Which kernel a launcher takes, where the launcher decides by sizes alone (host code of the kernel libraries, no device)."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

SMS = 148


@pytest.fixture(scope="module")
def narrow_plan():
    from mini_llm_b200.kernels import build
    return ctypes.CDLL(build.library_path("gemm")).mllm_gemm_narrow_plan


# measured (us, swapped tiles and narrow ones): the faster kernel is the one that runs
@pytest.mark.parametrize("m, n, k, swapped, narrow", [
    (24, 2304, 768, 5.0, 3.0), (64, 768, 768, 6.6, 3.4), (64, 3072, 768, 7.4, 5.4), (48, 6144, 1024, 9.8, 8.4), (24, 8192, 4096, 17.6, 15.4),
    (64, 2304, 4096, 15.8, 10.9), (12, 16000, 768, 9.6, 8.6), (16, 1600, 8192, 10.3, 10.1), (24, 8192, 6400, 23.7, 22.9),
    (32, 8192, 1024, 9.0, 9.7), (64, 4096, 2048, 10.1, 13.2), (64, 8192, 2048, 15.0, 24.4), (24, 12288, 1024, 10.6, 12.3),
    (64, 12288, 4096, 28.6, 41.5), (32, 16000, 768, 9.8, 14.9), (24, 1600, 6400, 9.2, 10.7), (24, 1600, 11008, 12.2, 16.0), (64, 50257, 768, 21.4, 58.9)])
def test_products_of_few_tokens_take_the_faster_tiles(narrow_plan, m, n, k, swapped, narrow):
    assert (narrow_plan(m, n, k, SMS) != 0) == (narrow < swapped)


# measured (us, in tiles and pair by pair): tokens, tables, pairs a token, features a token
@pytest.mark.parametrize("tokens, tables, pairs, features, tiles, by_pairs", [
    (1, 17, 3, 1536, 13.4, 14.1), (2, 17, 3, 1536, 14.2, 15.4), (8, 17, 3, 1536, 19.8, 18.5), (13, 17, 3, 1536, 20.8, 25.0), (1, 9, 3, 3072, 14.4, 20.9),
    (16, 9, 3, 3072, 19.8, 38.5), (4, 8, 2, 4096, 31.7, 27.6), (5, 8, 2, 4096, 33.6, 36.7), (1, 24, 2, 1536, 13.6, 9.6), (31, 24, 2, 1536, 35.8, 40.4),
    (1, 48, 2, 1024, 15.4, 9.1), (2, 48, 2, 1024, 16.6, 9.5), (24, 48, 2, 1024, 43.4, 32.1), (1, 60, 4, 1024, 18.5, 10.9), (20, 60, 4, 1024, 42.4, 34.5)])
def test_experts_take_the_faster_kernels(tokens, tables, pairs, features, tiles, by_pairs):
    from mini_llm_b200.kernels.dispatch import Kernels
    assert Kernels.experts_in_tiles(tokens, tables, pairs, features) == (tiles < by_pairs)


@pytest.mark.parametrize("steps_apart, decode_only, writes, ahead", [(True, True, True, True), (True, False, True, False), (True, True, False, False),
                                                                     (False, True, True, False)])
def test_states_are_read_ahead_of_the_wait_by_single_tokens_of_their_writer(monkeypatch, steps_apart, decode_only, writes, ahead):
    """512 is a key size that the kernels for chunks do not take: portions walk token by token, as single tokens do."""
    from mini_llm_b200.kernels import dispatch
    from mini_llm_b200.kernels.dispatch import Kernels
    seen = {}
    monkeypatch.setattr(dispatch.ops, "memory_scan", lambda *a, state_ahead=None, **k: seen.update(memory=state_ahead, chunked=k["chunked"]))
    monkeypatch.setattr(dispatch.ops, "linear_recurrence", lambda *a: seen.update(recurrence=a[-1]))
    rows, ints = torch.zeros(3, 512), torch.zeros(3, dtype=torch.int32)
    ctx = SimpleNamespace(steps_apart=steps_apart, decode_only=decode_only, n_items=3, item_slot=ints, item_offset=ints, item_count=ints, device=rows.device)
    kernels = Kernels(torch.float32)
    kernels.memory_scan(ctx, rows, rows, rows, rows, rows, 1, 512, 512, writes=writes, decay=rows[0, :1])
    kernels.linear_recurrence(ctx, rows, rows, rows, rows, rows, rows, rows, rows, rows, 1, 1, 512, 512, True, True, 1.0, None, writes, False)
    assert bool(seen["memory"]) == ahead and not seen["chunked"]
    assert bool(seen["recurrence"]) == (steps_apart and writes)       # (only its kernel for few tokens an entry reads ahead)


@pytest.mark.parametrize("heads, rank, dtype, step", [(12, 256, torch.bfloat16, True), (16, 128, torch.bfloat16, True), (17, 256, torch.bfloat16, False),
                                                      (4, 64, torch.bfloat16, False), (4, 128, torch.float32, False)])
def test_single_tokens_over_a_latent_are_one_launch_where_the_kernel_merges_itself(monkeypatch, heads, rank, dtype, step):
    from mini_llm_b200.kernels import dispatch
    from mini_llm_b200.kernels.dispatch import Kernels
    seen, rot, ints = {}, 32, torch.zeros(2, dtype=torch.int32)
    monkeypatch.setattr(dispatch.ops, "latent_attention_tiled", lambda *a, **k: seen.update(k))
    pages, q = torch.zeros(4, 16, 1, rank + rot, dtype=dtype), torch.zeros(2, heads * (rank + rot))
    ctx = SimpleNamespace(steps_apart=True, decode_only=True, att_tiles=None, positions=ints, token_item=ints, device=q.device)
    cache = SimpleNamespace(k_pages=pages, block_table=ints.view(1, 2), page_size=16)
    kernels = Kernels(torch.bfloat16)
    kernels.latent_attention(ctx, torch.zeros(2, heads * rank), q, cache, heads, rank, rot, 0.1)
    assert kernels.launches == (1 if step else 2) and kernels.scratch_generation == (0 if step else 1)
    assert ("scratch" in seen) != step and seen.get("rows_ahead", False) == step
    assert {kernel for kernel in kernels.choices.values()} == {"latent_step" if step else "latent_attention_tiled_parts"}


def test_an_embedding_with_a_forward_of_its_own_says_itself_how_it_begins():
    from mini_llm_b200.parts.base import Embedding
    from mini_llm_b200.parts.embedding import PairedTokenEmbedding, TokenEmbedding

    class Other(TokenEmbedding):
        def forward(self, ctx, position=None, cache=None):
            raise NotImplementedError

    class Same(TokenEmbedding):
        pass

    assert TokenEmbedding.forward_begins_apart() and PairedTokenEmbedding.forward_begins_apart() and Same.forward_begins_apart()
    assert not Other.forward_begins_apart() and not Embedding.forward_begins_apart()
