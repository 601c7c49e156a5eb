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
