"""The 16-row product around the numbers of blocks at which it changes how its loads are placed: a row's bits stay."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"


# 16 columns a block: two blocks an SM of 148 and one column more, a short last block between, three an SM and one more
@pytest.mark.parametrize("n", [4736, 4737, 5130, 7104, 7105])
@pytest.mark.parametrize("k_dim", [32, 160, 1088])
def test_rows_of_a_full_batch_equal_rows_of_half_a_batch(n, k_dim):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(n + k_dim)
    x = torch.randn(16, k_dim, device=DEV).bfloat16()
    w = (torch.randn(n, k_dim, device=DEV) / k_dim ** 0.5).bfloat16()
    bias, residual = torch.randn(n, device=DEV), torch.randn(16, n, device=DEV)
    halves = torch.empty(16, n, device=DEV)
    for first in (0, 8):
        rows = slice(first, first + 8)
        k.gemm_skinny(x[rows], w, bias, residual[rows], halves[rows], k.EPILOGUE_RESIDUAL)
    exact = residual.double() + bias.double() + x.double() @ w.double().T
    # a float chain over K and two additions, of numbers below |x| . |w| and the result's parts
    bound = (k_dim + 2) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + bias.double().abs() + residual.double().abs())
    assert bool(((halves.double() - exact).abs() <= bound).all())
    for m in (9, 16):
        out = torch.full((m, n), float("nan"), device=DEV)
        k.gemm_skinny(x[:m], w, bias, residual[:m], out, k.EPILOGUE_RESIDUAL)
        assert torch.equal(out, halves[:m]), m


@pytest.mark.parametrize("heads,kv_heads", [(36, 4), (33, 2), (48, 4)])          # 352, 296 and 448 blocks of 16 columns
def test_rotated_rows_of_a_full_batch_equal_rows_of_half_a_batch(heads, kv_heads):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(heads)
    k_dim, dim, n = 320, 128, (heads + 2 * kv_heads) * 128
    x = torch.randn(16, k_dim, device=DEV).bfloat16()
    w = (torch.randn(n, k_dim, device=DEV) / k_dim ** 0.5).bfloat16()
    bias = torch.randn(n, device=DEV)
    positions = torch.arange(100, 116, dtype=torch.int32, device=DEV)
    slots = torch.arange(3, 19, dtype=torch.int32, device=DEV)
    inv_freq = (1.0 / (10000.0 ** (torch.arange(0, dim, 2, dtype=torch.float32) / dim))).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    results = []
    for parts in ([slice(0, 16)], [slice(0, 8), slice(8, 16)]):
        qkv = torch.zeros(16, n, device=DEV, dtype=torch.bfloat16)
        cache = torch.zeros(2, 2, kv_heads, 16, dim, device=DEV, dtype=torch.bfloat16)
        for rows in parts:
            k.gemm_skinny_rope(x[rows], w, bias, qkv[rows], positions[rows], inv_freq, slots[rows], cache, heads,
                               kv_heads, dim, 16, status)
        results.append((qkv[:, :heads * dim], cache))
    assert status.item() == 0 and bool(results[0][1].any())
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
