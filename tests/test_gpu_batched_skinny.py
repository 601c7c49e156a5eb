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
