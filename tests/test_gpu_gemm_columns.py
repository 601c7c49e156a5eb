"""The product with the tokens as the columns of pairs of SMs: against float64 at the edges of tiles, token counts, stages and
parts of K, every epilogue, more items than pairs, and what is not finite."""

import math
import os
import subprocess
import sys

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


@pytest.mark.parametrize("m,n,k_dim", [(257, 3072, 12288), (512, 3072, 12288), (600, 2048, 8192), (1024, 1024, 6144),
                                       (2048, 1024, 6144)])
def test_parts_of_k_are_added_in_their_order(m, n, k_dim):
    """A product whose K is cut into parts gives the same bits every time, whoever adds the parts up."""
    from matricxon_b200.ops import kernels as k
    from matricxon_b200.ops.linear import PendingSum, linear

    assert k.columns_gemm_parts(m, n, k_dim) > 1
    torch.manual_seed(m)
    a, w = torch.randn(m, k_dim, device=DEV).bfloat16(), (torch.randn(n, k_dim, device=DEV) / math.sqrt(k_dim)).bfloat16()
    bias, residual = torch.randn(n, device=DEV), 100 * torch.randn(m, n, device=DEV)
    weight, shift = torch.randn(n, device=DEV), torch.randn(n, device=DEV)

    def product(**options):
        x = residual.clone()
        return linear(a, w, bias, k.EPILOGUE_RESIDUAL, residual=x, out=x, backend="columns", **options)

    first = product()
    for _ in range(12):
        assert torch.equal(product(), first)
    exact = residual.double() + a.double() @ w.double().T + bias.double()
    # the cut-offs of the running sum, and eight roundings of sums of the stream's size
    bound = (k_dim / 16 + 16) * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T) + 8 * 2.0 ** -23 * (exact.abs() + residual.abs())
    assert bool(((first.double() - exact).abs() <= bound).all())
    pending = product(defer_sum=True)
    assert isinstance(pending, PendingSum) and torch.equal(pending.tensor(), first) and torch.equal(pending.tensor(), first)
    pending = product(defer_sum=True)
    normed, alone = (torch.empty(m, n, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    x = pending.added_by_kernel()
    k.layernorm_sum(x, pending.parts, pending.bias, weight, shift, 1e-5, normed)
    k.layernorm(first, weight, shift, 1e-5, alone)
    assert torch.equal(x, first) and torch.equal(normed, alone)
    pending = product(defer_sum=True)                                      # for norms that take one tensor
    assert bool(((pending.acc.double() - (exact - residual - bias)).abs() <= bound).all()) and pending.parts is None
    assert bool(((pending.tensor().double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("rows,columns,n_parts", [(1, 4, 2), (300, 3072, 3), (7, 8196, 8), (5, 30, 4), (3, 52000, 2)])
def test_norm_of_parts(rows, columns, n_parts):
    """Rows in registers, rows too long for them, rows that cannot be read 16 bytes at a time."""
    from matricxon_b200.ops import kernels as k

    parts, residual = torch.randn(n_parts, rows, columns, device=DEV), torch.randn(rows, columns, device=DEV)
    bias, weight = torch.randn(columns, device=DEV), torch.randn(columns, device=DEV)
    total = parts[0].clone()
    for p in parts[1:]:
        total += p
    want = (total + bias) + residual
    added = residual.clone()
    k.add_parts(parts, bias, added)
    assert torch.equal(added, want)
    if columns <= 51200:
        x, out, alone = residual.clone(), torch.empty_like(want), torch.empty_like(want)
        k.layernorm_sum(x, parts, bias, weight, None, 1e-5, out)
        k.layernorm(want, weight, None, 1e-5, alone)
        assert torch.equal(x, want) and torch.equal(out, alone)


FIRST_CALLS = """
import sys, threading
sys.path.insert(0, sys.argv[1])
import torch
from matricxon_b200.ops import kernels as k
a, w = torch.randn(300, 512, device="cuda").bfloat16(), torch.randn(1024, 512, device="cuda").bfloat16()
outs = [torch.empty(300, 1024, device="cuda") for _ in range(8)]
k.default_status(a.device)
torch.cuda.synchronize()
barrier, failed = threading.Barrier(len(outs)), []
def call(out):
    barrier.wait()
    try:
        k.gemm_columns(a, w, None, None, out, k.EPILOGUE_F32)
    except Exception as error:
        failed.append(error)
threads = [threading.Thread(target=call, args=(out,)) for out in outs]
for t in threads: t.start()
for t in threads: t.join()
torch.cuda.synchronize()
assert not failed, failed
assert all(torch.equal(out, outs[0]) for out in outs)
"""


def test_first_calls_from_several_threads():
    """What the first call of a process looks up (pairs of SMs, shared memory) is there for all that come meanwhile."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", FIRST_CALLS, root], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
