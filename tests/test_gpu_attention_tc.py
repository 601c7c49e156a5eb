"""The tcgen05 prompt attention where a tile's last chunk of keys ends: the slots beyond the newest key hold NaN."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


# keys in the last chunk of 128: one, around a group of eight, around the half that a softmax warp owns, all but one, all
@pytest.mark.parametrize("last", [1, 8, 9, 63, 64, 65, 71, 127, 128])
@pytest.mark.parametrize("page_size", [16, 32])
@pytest.mark.parametrize("n_splits", [1, 2])
def test_every_end_of_the_last_chunk(last, page_size, n_splits):
    from test_gpu_kernels import kernels, paged_case, reference_attention, run_attention, tol

    seq_lens, q_lens = [384 + last, 256 + last], [40, 256 + last]
    q, cache, tables, tok_seq, positions, dense = paged_case(torch.bfloat16, 12, 2, 128, page_size, seq_lens, q_lens, seed=last)
    for window in (None, 100):
        ref = reference_attention(dense, q_lens, seq_lens, 128 ** -0.5, window)
        out, st = run_attention(kernels(), q, cache, tables, tok_seq, positions, 12, 2, 128, window, 128 ** -0.5,
                                n_splits, impl="tc")
        assert st == 0
        assert torch.allclose(out.double().cpu(), ref, **tol(torch.bfloat16)), (window, (out.double().cpu() - ref).abs().max())


@pytest.mark.parametrize("half", [0, 1])
def test_scores_of_one_half_far_above_the_others(half):
    """The two halves of a chunk's keys keep maxima of their own: whichever is larger has to win where they join."""
    from test_gpu_kernels import kernels, paged_case, reference_attention, run_attention, tol

    def larger(_s, qs, ks, vs):
        qs.abs_()
        for first in range(64 * half, ks.shape[1], 128):
            ks[:, first:first + 64] = ks[:, first:first + 64].abs() + 0.2 * (first // 128)

    q, cache, tables, tok_seq, positions, dense = paged_case(torch.bfloat16, 8, 2, 128, 16, [700], [300], seed=5, scale_up=larger)
    ref = reference_attention(dense, [300], [700], 128 ** -0.5, None)
    out, st = run_attention(kernels(), q, cache, tables, tok_seq, positions, 8, 2, 128, None, 128 ** -0.5, 1, impl="tc")
    assert st == 0 and torch.allclose(out.double().cpu(), ref, **tol(torch.bfloat16))
