"""Products of a decode step's heads or blocks with at most 16 rows: the tensor-core kernel (K a multiple of 32) and the other one."""

import math

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"


# K: one block of 32, fewer blocks than warps, one each, one warp with a fifth, more than are held at a time, no multiple of 32
@pytest.mark.parametrize("k_dim", [32, 96, 128, 160, 544, 40])
@pytest.mark.parametrize("n", [1, 15, 16, 33, 128])
@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_interleaved_members(m, n, k_dim, dtype):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(k_dim + n)
    batch = 3
    a = torch.randn(m, batch, k_dim + 8, device=DEV).bfloat16()[:, :, :k_dim]
    w = (torch.randn(batch, n, k_dim, device=DEV) / math.sqrt(k_dim)).bfloat16()
    wide = torch.full((m, batch, n + 8), float("nan"), device=DEV, dtype=dtype)
    out = wide[:, :, :n]
    assert k.batched_skinny_supported(a, w, out)
    k.gemm_batched_skinny(a, w, out)
    exact = torch.einsum("mbk,bnk->mbn", a.double(), w.double())
    # float sums of exact products, then one rounding to the result's dtype
    bound = (k_dim * 2.0 ** -24) * torch.einsum("mbk,bnk->mbn", a.double().abs(), w.double().abs())
    if dtype == torch.bfloat16:
        bound = bound + 2.0 ** -8 * exact.abs()
    assert bool(((out.double() - exact).abs() <= bound + 1e-30).all())
    assert bool(wide[:, :, n:].isnan().all())
    alone = torch.empty(1, batch, n, device=DEV, dtype=dtype)
    k.gemm_batched_skinny(a[m - 1:m], w, alone)
    assert torch.equal(alone[0], out[m - 1])             # a row's result does not depend on the others


@pytest.mark.parametrize("k_dim", [128, 512])
def test_weights_that_the_kernel_before_wrote(k_dim):
    """Chained launches: the product may be on the GPU before the norm that writes its weights has ended."""
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(k_dim)
    batch, n, rounds = 16, 128, 12
    a = torch.randn(4, batch, k_dim, device=DEV).bfloat16()
    xs = [torch.randn(batch * n, k_dim, device=DEV) for _ in range(rounds)]
    scale = torch.ones(k_dim, device=DEV)
    w = torch.zeros(batch * n, k_dim, device=DEV, dtype=torch.bfloat16)
    outs = [torch.empty(4, batch, n, device=DEV) for _ in range(rounds)]
    kept = [torch.empty_like(w) for _ in range(rounds)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):                            # back to back, with nothing of the host's in between
        for x, out, copy in zip(xs, outs, kept):
            k.rmsnorm(x, scale, 0.0, 1e-6, w)
            k.gemm_batched_skinny(a, w.view(batch, n, k_dim), out)
            copy.copy_(w)
    graph.replay()
    torch.cuda.synchronize()
    for x, out, copy in zip(xs, outs, kept):
        members = copy.double().view(batch, n, k_dim)
        exact = torch.einsum("mbk,bnk->mbn", a.double(), members)
        bound = (k_dim * 2.0 ** -24) * torch.einsum("mbk,bnk->mbn", a.double().abs(), members.abs())
        assert bool(((out.double() - exact).abs() <= bound + 1e-30).all())
        assert bool((copy.float() - x / x.pow(2).mean(dim=1, keepdim=True).sqrt()).abs().max() < 0.05)


@pytest.mark.parametrize("k_dim", [32, 128, 512])
def test_float_results_are_as_good_as_multiply_adds(k_dim):
    """Against 64 bits no further off than one rounding a product and one an addition of the lanes' tree gave."""
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(k_dim)
    batch, n = 16, 128
    a = torch.randn(16, batch, k_dim, device=DEV).bfloat16()
    w = torch.randn(batch, n, k_dim, device=DEV).bfloat16()
    out = torch.empty(16, batch, n, device=DEV)
    k.gemm_batched_skinny(a, w, out)
    exact = torch.einsum("mbk,bnk->mbn", a.double(), w.double())
    # A rounding is 0.40 units of 2^-24 on average (uniform within half a last place, over all mantissas). Sums are added in
    # pairs, so each level's roundings together are one such error of the whole sum, and above products of 16 k there
    # are at most eight levels (512 long): sqrt(8) x 0.40 = 1.13. One chain of the tensor cores' own additions: 2.1.
    off = float((out.double() - exact).norm() / exact.norm())
    assert off <= 1.15 * 2.0 ** -24, off * 2.0 ** 24


def test_infinities_and_nan_stay_in_their_rows():
    from matricxon_b200.ops import kernels as k

    for dtype in (torch.float32, torch.bfloat16):
        a, w = torch.randn(5, 2, 64, device=DEV).bfloat16(), torch.randn(2, 20, 64, device=DEV).bfloat16()
        a[0, 0, 5], a[1, 0, 63], a[2, 1, 0] = math.inf, math.nan, -math.inf
        out = torch.empty(5, 2, 20, device=DEV, dtype=dtype)
        k.gemm_batched_skinny(a, w, out)
        assert torch.equal(out[0, 0].float(), w[0, :, 5].sign().float() * math.inf) and bool(out[1, 0].isnan().all())
        assert torch.equal(out[2, 1].float(), -w[1, :, 0].sign().float() * math.inf)
        kept = torch.ones(5, 2, dtype=torch.bool)
        kept[0, 0] = kept[1, 0] = kept[2, 1] = False
        assert bool(out[kept.to(DEV)].isfinite().all())
