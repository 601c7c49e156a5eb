"""The order of the prompt attention's tiles: the ones with the most keys first, over all sequences of a step."""

import pytest

pytest.importorskip("torch")


@pytest.mark.parametrize("q_lens,contexts", [
    ([2048], [0]), ([300, 17, 512, 40], [0, 600, 100, 3000]), ([1, 40, 0, 100], [5, 0, 9, 0]), ([64, 64], [0, 0])])
@pytest.mark.parametrize("group", [1, 9, 12])
def test_most_keys_first(q_lens, contexts, group):
    from matricxon_b200.ops.kernels import attention_tile_lists

    narrow, wide = attention_tile_lists(q_lens, group, True, contexts)
    plain_narrow, plain = attention_tile_lists(q_lens, group, True)
    tiles = list(zip(wide[::2], wide[1::2]))
    assert narrow == plain_narrow and sorted(tiles) == sorted(zip(plain[::2], plain[1::2]))
    newest = [contexts[seq] + token for seq, token in tiles]
    assert newest == sorted(newest, reverse=True)


def test_lists_of_rows_keep_their_order():
    from matricxon_b200.ops.kernels import attention_tile_lists

    assert attention_tile_lists([40, 1, 90], 2, False, [0, 7, 500]) == attention_tile_lists([40, 1, 90], 2, False)


@pytest.mark.parametrize("group,float_blocks", [(1, 1), (4, 1), (5, 1), (6, 1), (7, 2), (8, 2), (9, 2), (12, 2), (13, 3), (16, 3), (24, 4)])
def test_key_shares_count_the_blocks_of_the_kernel_that_runs(group, float_blocks):
    """Float heads of 128 on pages of whole sixteens go four or six to a block, others up to sixteen."""
    from types import SimpleNamespace

    import torch
    from matricxon_b200.ops.kernels import attention_head_blocks
    from matricxon_b200.parts.attention import simt_splits

    def blocks(dtype, head_dim=128, page_size=16, stride=8192):
        memory = torch.zeros(1024, dtype=dtype)
        aligned = memory[-(memory.data_ptr() // memory.element_size()) % 32:]
        return attention_head_blocks(aligned, stride, aligned, page_size, head_dim, group)

    general = -(-group // 16)
    assert blocks(torch.float32) == float_blocks
    assert blocks(torch.float32, 64) == blocks(torch.float32, 128, 8) == blocks(torch.float32, stride=8190) == general
    assert blocks(torch.bfloat16) == general
    ctx = SimpleNamespace(n_tokens=4, max_kv_len=4096, sm_count=148, scratch=lambda nbytes: nbytes)
    shares, scratch = simt_splits(ctx, 2 * group, 2, 128, None, float_blocks)
    # four blocks an SM, at least two chunks of 32 keys a share, 64 shares at most
    assert shares == min(64, 592 // (8 * float_blocks)) and scratch >= 4 * 2 * group * shares * 130 * 4
