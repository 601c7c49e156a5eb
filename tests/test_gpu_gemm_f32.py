"""The 32-bit path's products with 16-byte reads: the kernel for few rows and the one for many give the general
kernel's bits, at the edges of their tiles, pieces and row counts."""

import math

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"


# pieces of K (a quarter, rounded up to 32): one, one and a short one, three and a short one, four whole ones
@pytest.mark.parametrize("k_dim", [4, 36, 100, 640])
@pytest.mark.parametrize("n", [1, 33, 131])
def test_every_row_count_gives_the_general_kernels_bits(n, k_dim):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(n * 1000 + k_dim)
    a = torch.randn(130, k_dim + 4, device=DEV)[:, :k_dim]                 # rows of a wider buffer
    w = torch.randn(n, k_dim, device=DEV) / math.sqrt(k_dim)
    bias, residual = torch.randn(n, device=DEV), torch.randn(130, n, device=DEV)
    exact = a.double().cpu() @ w.double().cpu().T
    shifted = torch.empty(130 * k_dim + 1, device=DEV)[1:].view(130, k_dim).copy_(a)      # not 16-byte aligned
    general = torch.empty(130, n, device=DEV)
    k.gemm_simt(shifted, w, None, None, general, k.EPILOGUE_F32)
    # a chain of K / 4 roundings of sums that stay below |a| . |w|
    bound = (k_dim / 4 + 4) * 2.0 ** -24 * (a.double().abs().cpu() @ w.double().abs().cpu().T)
    assert bool(((general.double().cpu() - exact).abs() <= bound).all())
    for m in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 130):
        out = torch.full((m, n), float("nan"), device=DEV)
        k.gemm_simt(a[:m], w, None, None, out, k.EPILOGUE_F32)
        assert torch.equal(out, general[:m]), m
        k.gemm_simt(a[:m], w, bias, residual[:m], out, k.EPILOGUE_RESIDUAL)
        assert torch.equal(out, residual[:m] + (general[:m] + bias)), m
    k.gemm_simt(a[:40], w, bias, None, general[:40], k.EPILOGUE_GELU)
    few = torch.empty(7, n, device=DEV)
    k.gemm_simt(a[:7], w, bias, None, few, k.EPILOGUE_GELU)
    assert torch.equal(few, general[:7])


# Blocks of several weight rows, with a short last one: seven rows (1,000 columns over 148 SMs), and 17 in two rounds (4,737
# and 5,003 columns). Pieces of six chunks of 32 (a ring filled once and one chunk more), of thirteen with a short end, of
# twenty-four: rings that come round four times.
@pytest.mark.parametrize("k_dim", [644, 1572, 3072])
@pytest.mark.parametrize("n", [1000, 4737, 5003])
def test_blocks_of_several_rows_and_rings_that_come_round(n, k_dim):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(n + k_dim)
    a = torch.randn(130, k_dim, device=DEV)
    w = torch.randn(n, k_dim, device=DEV) / math.sqrt(k_dim)
    shifted = torch.empty(130 * k_dim + 1, device=DEV)[1:].view(130, k_dim).copy_(a)      # not 16-byte aligned
    general = torch.empty(130, n, device=DEV)
    k.gemm_simt(shifted, w, None, None, general, k.EPILOGUE_F32)
    exact = a.double() @ w.double().T
    bound = (k_dim / 4 + 4) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((general.double() - exact).abs() <= bound).all())
    for m in (1, 2, 4, 8, 16, 17, 32, 33, 130):
        out = torch.full((m, n), float("nan"), device=DEV)
        k.gemm_simt(a[:m], w, None, None, out, k.EPILOGUE_F32)
        assert torch.equal(out, general[:m]), m


def test_infinities_and_nan_stay_in_their_rows():
    from matricxon_b200.ops import kernels as k

    for m in (3, 70):
        a, w = torch.randn(m, 64, device=DEV), torch.randn(40, 64, device=DEV)
        a[0, 5], a[1, 63] = math.inf, math.nan
        out = torch.empty(m, 40, device=DEV)
        k.gemm_simt(a, w, None, None, out, k.EPILOGUE_F32)
        assert torch.equal(out[0], w[:, 5].sign() * math.inf) and bool(out[1].isnan().all())
        assert bool(out[2:].isfinite().all())


# pieces of K: one, one and a short one, three and a short one, four; members interleaved as heads in a row
@pytest.mark.parametrize("k_dim", [31, 33, 100, 512])
@pytest.mark.parametrize("m", [1, 64, 130])
def test_batched_members_give_a_plain_products_bits(m, k_dim):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(m * 1000 + k_dim)
    batch, n = 3, 70
    a, w = torch.randn(m, batch, k_dim, device=DEV), torch.randn(batch, n, k_dim, device=DEV)
    bias = torch.randn(batch, n, device=DEV)
    out = torch.full((m, batch, n + 2), float("nan"), device=DEV)
    k.gemm_batched_simt(a, w, bias, out[:, :, :n])
    alone = torch.empty(m, n, device=DEV)
    for b in range(batch):
        k.gemm_simt(a[:, b], w[b], bias[b], None, alone, k.EPILOGUE_F32)
        assert torch.equal(out[:, b, :n], alone), b
    assert bool(out[:, :, n:].isnan().all())
