"""Decoding requests and prompt portions of one step: their two attention kernels run at a time and give what they give one
after the other."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"


@pytest.mark.parametrize("heads,kv_heads,seq_lens,q_lens", [
    (24, 2, [300, 17, 700, 1], [1, 1, 200, 1]),
    (36, 4, [5, 90] * 40 + [600], [1, 1] * 40 + [129]),               # more tiles than SMs in the first kernel
    (8, 8, [40, 600], [16, 300])])
def test_the_same_rows(heads, kv_heads, seq_lens, q_lens):
    from matricxon_b200.ops import kernels as k
    from test_gpu_kernels import paged_case

    q, cache, tables, tok_seq, positions, _ = paged_case(torch.bfloat16, heads, kv_heads, 128, 16, seq_lens, q_lens, 7)
    n = q.shape[0]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu_q = [0]
    for length in q_lens:
        cu_q.append(cu_q[-1] + length)
    context = [a - b for a, b in zip(seq_lens, q_lens)]
    narrow, wide = k.attention_tile_lists(q_lens, heads // kv_heads, token_tiles=True, context_lens=context)
    assert narrow and wide
    narrow, wide, cu_q, context = ints(narrow), ints(wide), ints(cu_q), ints(context)
    source, results, status = q.clone(), [], torch.zeros(1, dtype=torch.int32, device=DEV)
    for beside in (False, True, True):
        out = torch.full((n, heads * 128), float("nan"), dtype=torch.bfloat16, device=DEV)
        q.zero_()
        k.set_chained_launch(True)
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                q.copy_(source)                                         # the queries are the kernel's before
                for call, tiles, more in ((k.paged_attention_mma, narrow, (True,)), (k.paged_attention_tc, wide, ())):
                    call(q, q.stride(0), cache, tables, cu_q, context, tiles, tiles.numel() // 2, *more, n, heads, kv_heads, 128,
                         None, 128 ** -0.5, out, status, beside=beside)
                after = out.clone()                                     # reads both kernels' rows
        finally:
            k.set_chained_launch(False)
        for _ in range(3):
            q.zero_()
            out.fill_(float("nan"))
            graph.replay()
        torch.cuda.synchronize()
        results.append(after.clone())
    assert status.item() == 0 and bool(results[0].isfinite().all())
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])


def test_only_the_launch_before_is_run_beside():
    """The second kernel does not wait for what the first one has waited for: it is refused after any other launch."""
    from matricxon_b200.ops import kernels as k
    from matricxon_b200.ops.library import KernelLibraryError
    from test_gpu_kernels import paged_case

    q, cache, tables, _, _, _ = paged_case(torch.bfloat16, 8, 2, 128, 16, [40, 200], [1, 150], 3)
    n = q.shape[0]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu_q, context = ints([0, 1, 151]), ints([39, 50])
    narrow, wide = (ints(t) for t in k.attention_tile_lists([1, 150], 4, token_tiles=True, context_lens=[39, 50]))
    out, status = torch.empty(n, 8 * 128, dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)

    def first(**options):
        k.paged_attention_mma(q, q.stride(0), cache, tables, cu_q, context, narrow, narrow.numel() // 2, True, n, 8, 2, 128,
                              None, 0.1, out, status, **options)

    def second(queries=q, **options):
        k.paged_attention_tc(queries, q.stride(0), cache, tables, cu_q, context, wide, wide.numel() // 2, n, 8, 2, 128, None,
                             0.1, out, status, **options)

    def refused(call, *args, **options):
        with pytest.raises(KernelLibraryError):
            call(*args, **options)

    refused(second, beside=True)
    first()
    refused(second, beside=True)                        # a launch that lets its successor start at once
    first(beside=True)
    refused(second, q.clone(), beside=True)             # other tensors
    first(beside=True)
    k.softcap(torch.ones(4, device=DEV), 1.0)
    refused(second, beside=True)                        # another kernel between them
    refused(first, n_splits=2, scratch=torch.empty(1 << 20, device=DEV), beside=True)
    first(beside=True)
    second(beside=True)
    refused(second, beside=True)                        # once
    first(beside=True)
    second()
    torch.cuda.synchronize()
    assert status.item() == 0
