"""Products of few rows whose weights the kernel before wrote: chained launches may not read them early."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"


@pytest.mark.parametrize("m", [1, 9, 16, 100])
@pytest.mark.parametrize("kernel", ["gemm_skinny", "gemm_stream"])
def test_weights_that_the_kernel_before_wrote(m, kernel):
    from matricxon_b200.ops import kernels as k

    if kernel == "gemm_skinny" and m > 16:
        pytest.skip("more rows than the kernel takes")
    torch.manual_seed(m)
    n, k_dim, rounds = 5120, 512, 12
    a = torch.randn(m, k_dim, device=DEV).bfloat16()
    xs = [torch.randn(n, k_dim, device=DEV) for _ in range(rounds)]
    scale = torch.ones(k_dim, device=DEV)
    w = torch.zeros(n, k_dim, device=DEV, dtype=torch.bfloat16)
    outs = [torch.empty(m, n, device=DEV) for _ in range(rounds)]
    kept = [torch.empty_like(w) for _ in range(rounds)]
    k.default_status(w.device)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):                            # back to back, with nothing of the host's in between
        for x, out, copy in zip(xs, outs, kept):
            k.rmsnorm(x, scale, 0.0, 1e-6, w)
            getattr(k, kernel)(a, w, None, None, out, k.EPILOGUE_F32)
            copy.copy_(w)
    graph.replay()
    torch.cuda.synchronize()
    for x, out, copy in zip(xs, outs, kept):
        exact = a.double() @ copy.double().T
        # float sums of exact products, which the tensor cores cut off: a unit of 2^-23 an addition
        bound = k_dim * 2.0 ** -23 * (a.double().abs() @ copy.double().abs().T)
        assert bool(((out.double() - exact).abs() <= bound).all())
        assert bool((copy.float() - x / x.pow(2).mean(dim=1, keepdim=True).sqrt()).abs().max() < 0.05)
