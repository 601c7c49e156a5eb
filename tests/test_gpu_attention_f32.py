"""The float attention that gives a warp sixteen keys, beside the general kernel: head counts, ends of chunks, pages of 16
and 32 slots, shares of the keys, every mask and option, slots that hold NaN, pages that are missing."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"
DIM = 128


def paged(lengths, kv_heads, page_size, seed):
    """Keys and values of several sequences on shuffled pages; slots beyond a sequence's end hold NaN."""
    g = torch.Generator().manual_seed(seed)
    pages = [-(-n // page_size) for n in lengths]
    order = torch.randperm(sum(pages) + 2, generator=g).tolist()
    cache = torch.full((sum(pages) + 2, 2, kv_heads, page_size, DIM), float("nan"))
    tables = torch.full((len(lengths), max(pages) + 1), -1, dtype=torch.int32)
    for s, n in enumerate(lengths):
        for lp in range(pages[s]):
            tables[s, lp] = page = order.pop()
            here = min(page_size, n - lp * page_size)
            cache[page, 0, :, :here] = torch.randn(kv_heads, here, DIM, generator=g)
            cache[page, 1].view(kv_heads, DIM, page_size)[:, :, :here] = torch.randn(kv_heads, DIM, here, generator=g)
    return cache.to(DEV), tables.to(DEV)


def both(heads, kv_heads, lengths, q_lens, page_size, splits, window=None, **options):
    """(this kernel's result, the general kernel's, whose query rows do not start on 16-byte boundaries, status word)."""
    from matricxon_b200.ops import kernels as k

    cache, tables = paged(lengths, kv_heads, page_size, heads + sum(lengths))
    seqs = [s for s, n in enumerate(q_lens) for _ in range(n)] + [-1]                  # and a padding row
    at = [lengths[s] - n + i for s, n in enumerate(q_lens) for i in range(n)] + [0]
    seqs, at = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in (seqs, at))
    n = len(at)
    q = torch.randn(n, heads * DIM + 3, device=DEV, generator=torch.Generator(DEV).manual_seed(n))
    results = []
    for rows in (q[:, :heads * DIM].contiguous(), q[:, :heads * DIM]):                 # the second: an odd row stride
        out = torch.full((n, heads * DIM), float("nan"), device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        scratch = torch.full((k.attention_scratch_bytes(n, heads, DIM, splits) // 4,), float("nan"), device=DEV)
        k.paged_attention(rows, rows.stride(0), cache, tables, seqs, at, n, heads, kv_heads, DIM, window, DIM ** -0.5, out,
                          status, n_splits=splits, scratch=scratch, **options)
        results.append(out)
    assert bool((results[0][-1] == 0).all())
    return *results, status.item()


def close(one, two):
    # scores of some 128 products and weights that sum to one: 128 roundings of either sum, relative to values of up to 5
    return bool(((one - two).abs() <= 5 * 128 * 2.0 ** -24).all())


@pytest.mark.parametrize("splits", [1, 3, 9])
@pytest.mark.parametrize("heads,kv_heads,page_size", [(1, 1, 16), (8, 2, 32), (10, 2, 16), (24, 2, 16), (13, 1, 48), (48, 2, 16)])
def test_heads_ends_and_shares(heads, kv_heads, page_size, splits):
    lengths, q_lens = [1, 15, 16, 17, 64, 65, 333], [1, 3, 1, 2, 1, 5, 40]
    one, two, status = both(heads, kv_heads, lengths, q_lens, page_size, splits)
    assert close(one, two) and status == 0


@pytest.mark.parametrize("splits", [1, 4])
@pytest.mark.parametrize("options", [{"window": 20}, {"window": 33, "keep_first": 5}, {"window": 100, "keep_first": 40},
                                     {"window": -32}, {"softcap": 2.0}, {"sink": 0}, {"distance": 0},
                                     {"window": 17, "softcap": 3.0, "sink": 0, "distance": 0, "keep_first": 16}])
def test_masks_and_options(options, splits):
    options = dict(options)
    if "sink" in options:
        options["sink"] = torch.linspace(-2, 3, 24, device=DEV)
    if "distance" in options:
        options["distance"] = torch.rand(2, 24, device=DEV)
    one, two, status = both(24, 2, [40, 129, 300], [40, 30, 1], 16, splits, **options)
    assert close(one, two) and status == 0


def test_missing_pages_read_as_zeros_and_are_reported():
    from matricxon_b200.ops import kernels as k

    cache, tables = paged([50], 1, 16, 3)
    tables[0, 1] = -1
    seqs, at = torch.zeros(1, dtype=torch.int32, device=DEV), torch.full((1,), 49, dtype=torch.int32, device=DEV)
    wide = torch.randn(1, 4 * DIM + 1, device=DEV)
    results = []
    for q in (wide[:, 1:].clone(), wide[:, 1:]):                                        # the second: not 16-byte aligned
        out, status = torch.empty(1, 4 * DIM, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        k.paged_attention(q, q.stride(0), cache, tables, seqs, at, 1, 4, 1, DIM, None, 0.1, out, status)
        results.append(out)
        assert status.item() == 4
    assert close(*results)
