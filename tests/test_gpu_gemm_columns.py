"""The product with the tokens as the columns of pairs of SMs: against float64 at the edges of tiles, token counts, stages and
parts of K, every epilogue, more items than pairs, and what is not finite."""

import math

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"


# tokens: one, a group of 16 and one more, a whole tile and one more, several; columns: less than a block's rows, ragged, more
# tiles than pairs of SMs; K: less than a slice, ragged, parts of unequal length, rings that come round
@pytest.mark.parametrize("m", [1, 17, 256, 257, 543, 1100])
@pytest.mark.parametrize("n,k_dim", [(3, 8), (130, 72), (300, 1096), (20011, 200), (384, 3072), (257, 9000)])
def test_all_epilogues(m, n, k_dim):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(m * 1000 + n)
    a = torch.randn(m, k_dim + 8, device=DEV).bfloat16()[:, :k_dim]         # rows of a wider buffer
    w = (torch.randn(n, k_dim, device=DEV) / math.sqrt(k_dim)).bfloat16()
    bias, residual = torch.randn(n, device=DEV), torch.randn(m, n, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    exact = a.double() @ w.double().T
    # a cut-off of the running sum at every 16 of K; sums stay below |a| . |w|
    bound = (k_dim / 16 + 16) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)
    out = torch.full((m, n), float("nan"), device=DEV)
    k.gemm_columns(a, w, None, None, out, k.EPILOGUE_F32, status)
    assert bool(((out.double() - exact).abs() <= bound).all())
    both = torch.full((m, n), float("nan"), device=DEV)
    k.gemm_columns(a, w, bias, residual, both, k.EPILOGUE_RESIDUAL, status)
    assert torch.equal(both, (out + bias) + residual)
    both = residual.clone()
    k.gemm_columns(a, w, bias, both, both, k.EPILOGUE_RESIDUAL, status)     # in place: K in parts, added in memory
    more = 10 * 2.0 ** -24 * (exact.abs() + bias.abs() + residual.abs())    # eight parts and the bias
    assert bool(((both.double() - (exact + bias + residual)).abs() <= 2 * bound + more).all())
    half = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.gemm_columns(a, w, bias, None, half, k.EPILOGUE_NONE, status)
    assert torch.equal(half, (out + bias).bfloat16())
    k.gemm_columns(a, w, bias, None, half, k.EPILOGUE_RELU2, status)
    assert torch.equal(half, ((out + bias).clamp(min=0) ** 2).bfloat16())
    k.gemm_columns(a, w, bias, None, half, k.EPILOGUE_GELU, status)
    ref = torch.nn.functional.gelu((out + bias).double(), approximate="tanh")
    # one rounding to bfloat16, and the hardware's tanh (2^-11 of one half of the argument)
    assert bool(((half.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -11 * (out + bias).abs().double()).all())
    assert status.item() == 0


def test_rule():
    from matricxon_b200.ops.linear import chosen_backend

    def at(m, n, k_dim):
        return chosen_backend(torch.empty(m, k_dim, dtype=torch.bfloat16, device=DEV), torch.empty(n, k_dim, dtype=torch.bfloat16, device=DEV))

    assert at(257, 8192, 64) == at(367, 1024, 8192) == at(1024, 128, 64) == at(2047, 128, 12288) == at(2048, 128, 8192) == "columns"
    assert at(2048, 128, 12288) == at(4096, 128, 8192) == at(8192, 128, 6144) == "tcgen05"
    assert at(256, 8192, 64) == at(1023, 4096, 4096) == "library"


def test_nan_stays_in_its_row():
    from matricxon_b200.ops import kernels as k

    a, w = torch.randn(400, 512, device=DEV).bfloat16(), torch.randn(300, 512, device=DEV).bfloat16()
    a[3, 100], a[5, 0] = math.nan, math.inf
    out = torch.empty(400, 300, device=DEV)
    k.gemm_columns(a, w, None, None, out, k.EPILOGUE_F32)
    bad = ~out.isfinite().all(dim=1)
    assert bad.nonzero().flatten().tolist() == [3, 5] and bool(out[3].isnan().all())
    assert torch.equal(out[5], w[:, 0].float().sign() * math.inf)
