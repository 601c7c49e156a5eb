"""Float products on the tensor cores, three bfloat16 numbers a float: against 64 bits at the edges of tiles, stages and
shares of K, no further off than the FP32 cores, every epilogue, and what is not finite."""

import math

import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda:0"
# the parts left out are m l + l m + l l of a term, with |m| up to 2^-8 and |l| up to 2^-17 of a float
LEFT_OUT = 1.01 * 2.0 ** -24


# tokens: a tile of 16, one row more, the last that are split in passing and one more, a tile of 208 and one more, several
# tiles; columns: less than a tile, ragged, several tiles; K: less than a stage, ragged stages, shares of K of 5 and 6 stages
# (up to eight rows a kernel of its own, whose columns are the tokens: each count of them)
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16, 17, 64, 65, 130, 208, 209, 700])
@pytest.mark.parametrize("n,k_dim", [(1, 4), (131, 36), (260, 332), (1027, 1500), (384, 3072)])
def test_against_64_bits_and_the_fp32_cores(m, n, k_dim):
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(m * 1000 + n)
    a = torch.randn(m, k_dim + 4, device=DEV)[:, :k_dim]                   # rows of a wider buffer
    w = torch.randn(n, k_dim, device=DEV) / math.sqrt(k_dim)
    bias, residual = torch.randn(n, device=DEV), torch.randn(m, n, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    exact = a.double() @ w.double().T
    out, plain = torch.full((m, n), float("nan"), device=DEV), torch.empty(m, n, device=DEV)
    k.gemm_f32_split(a, w, None, None, out, k.EPILOGUE_F32, status)
    k.gemm_simt(a, w, None, None, plain, k.EPILOGUE_F32)
    # each 32 values of k: the parts left out, twelve cut-offs of a sum below |a| . |w|, one rounding
    size = a.double().abs() @ w.double().abs().T
    assert bool(((out.double() - exact).abs() <= (LEFT_OUT + 13 * 2.0 ** -23) * size).all())
    if m * n > 4000 and k_dim > 300:
        assert (out.double() - exact).norm() <= (plain.double() - exact).norm()
    # the epilogues add to the same sums
    biased = torch.empty_like(out)
    k.gemm_f32_split(a, w, bias, residual, biased, k.EPILOGUE_RESIDUAL, status)
    assert torch.equal(biased, residual + (out + bias))
    inplace = residual.clone()
    k.gemm_f32_split(a, w, bias, inplace, inplace, k.EPILOGUE_RESIDUAL, status)
    assert torch.equal(inplace, biased)
    k.gemm_f32_split(a, w, bias, None, biased, k.EPILOGUE_GELU, status)
    ref = torch.nn.functional.gelu((out + bias).double(), approximate="tanh")
    assert bool(((biased.double() - ref).abs() <= 2e-6 * (1 + ref.abs())).all())
    assert status.item() == 0


def test_sizes_of_numbers():
    """Rows of very large, very small and subnormal floats, and terms that cancel."""
    from matricxon_b200.ops import kernels as k

    a, w = torch.randn(40, 256, device=DEV), torch.randn(300, 256, device=DEV)
    scale = torch.tensor([2.0 ** e for e in (-120, -60, 0, 60, 100)], device=DEV).repeat(8)[:, None]
    out, plain = torch.empty(40, 300, device=DEV), torch.empty(40, 300, device=DEV)
    k.gemm_f32_split(a, w, None, None, out, k.EPILOGUE_F32)
    k.gemm_f32_split(a * scale, w, None, None, plain, k.EPILOGUE_F32)
    big = scale[:, 0] > 2.0 ** -100
    assert torch.equal(plain[big], (out * scale)[big])                     # powers of two move exponents only
    # third parts of 2^-120 are below the smallest subnormal (2^-133): up to that of each term is lost
    assert bool(((plain[~big].double() - (out * scale)[~big].double()).abs() <= 256 * 5 * 2.0 ** -133).all())
    twice = torch.cat([a, -a], dim=1).contiguous()
    k.gemm_f32_split(twice, torch.cat([w, w], dim=1).contiguous(), None, None, out, k.EPILOGUE_F32)
    size = 2 * (a.double().abs() @ w.double().abs().T)
    assert bool((out.double().abs() <= (LEFT_OUT + 13 * 2.0 ** -23) * size).all())


def test_infinities_and_nan_stay_in_their_rows():
    from matricxon_b200.ops import kernels as k

    for m in (3, 4, 8, 20, 300):
        a, w = torch.randn(m, 512, device=DEV), torch.randn(261, 512, device=DEV)
        a[0, 5], a[1, 511], a[2, 3] = math.inf, math.nan, 3.4e38           # the last rounds to infinity in bfloat16
        w[7, 3] = 0.5
        out, plain = torch.empty(m, 261, device=DEV), torch.empty(m, 261, device=DEV)
        k.gemm_f32_split(a, w, None, None, out, k.EPILOGUE_F32)
        k.gemm_simt(a, w, None, None, plain, k.EPILOGUE_F32)
        assert torch.equal(out[0], w[:, 5].sign() * math.inf) and bool(out[1].isnan().all())
        assert torch.equal(out[2], plain[2]) and bool(out[2, 7].isfinite())
        assert bool(out[3:].isfinite().all())


@pytest.mark.parametrize("m,k_dim", [(4, 1024), (4, 3072), (8, 512), (16, 2048), (32, 1024), (200, 512), (200, 3072)])
def test_errors_of_other_operands(m, k_dim):
    """Operands whose errors do not cancel as those of random signs do: sums of one sign, a term that dominates, few terms, one.
    The root mean square error against 64 bits, beside the FP32 cores', at the shortest K that the engine sends here and above.
    Sums of one sign and dominating terms are no further off (relu^2 times |normal| as far at K = 512 and 640: 0.92 to 1.03
    times over 3 to 200 rows, and few rows scatter); few terms (one in fifty) up to 1.3 times, a single term, which the FP32
    cores round once, 1.9 times as far."""
    from matricxon_b200.ops import kernels as k

    torch.manual_seed(m + k_dim)
    a, w = torch.randn(m, k_dim, device=DEV), torch.randn(1024, k_dim, device=DEV)
    one = torch.nn.functional.one_hot(torch.randint(0, k_dim, (m,), device=DEV), k_dim).float()
    for x, y, times in ((a.abs(), w.abs(), 1.0), (a.clamp(min=0) ** 2, w, 1.0), (a.clamp(min=0) ** 2, w.abs(), 1.2),
                        (a * 1e-3 + 10 * one, w, 1.0), (a * (torch.rand_like(a) < 0.02), w, 1.5), (a * one, w, 2.2)):
        out, plain = torch.empty(m, 1024, device=DEV), torch.empty(m, 1024, device=DEV)
        k.gemm_f32_split(x, y, None, None, out, k.EPILOGUE_F32)
        k.gemm_simt(x, y, None, None, plain, k.EPILOGUE_F32)
        exact = x.double() @ y.double().T
        assert (out.double() - exact).norm() <= times * (plain.double() - exact).norm()


def test_the_engine_takes_it_for_many_rows():
    from matricxon_b200.ops.linear import chosen_backend

    w = torch.empty(512, 512, device=DEV)
    assert chosen_backend(torch.empty(200, 512, device=DEV), w) == "split"
    assert chosen_backend(torch.empty(200, 512, device=DEV), w, "simt") == "simt"
    assert chosen_backend(torch.empty(200, 513, device=DEV)[:, 1:], w) == "simt"      # cannot be read 16 bytes at a time


@pytest.mark.parametrize("m", [3, 8, 20, 300])
def test_rows_that_are_not_finite_cost_the_others_little(m):
    """Their results are what the FP32 cores give, and a NaN is found by a look at its row: not a chain of K multiply-adds for
    every column, which made a step with one such row some ten times as long."""
    from matricxon_b200.ops import kernels as k

    n, k_dim = 2052, 4096
    w = torch.randn(n, k_dim, device=DEV)
    clean = torch.randn(m, k_dim, device=DEV)
    with_nan, every, mixed = clean.clone(), clean.clone(), clean.clone()
    with_nan[m - 1, k_dim - 1] = math.nan
    every[:, 77] = math.nan
    mixed[0, 9], mixed[1, 10], mixed[2, 100] = math.inf, -math.inf, 3.4e38
    mixed[2] *= 1e-3
    mixed[2, 100] = 3.4e38
    out, plain = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)

    def micros(a):
        best = math.inf
        for _ in range(6):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(4):
                k.gemm_f32_split(a, w, None, None, out, k.EPILOGUE_F32)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end) * 250)
        return best

    for a in (with_nan, every, mixed):
        k.gemm_f32_split(a, w, None, None, out, k.EPILOGUE_F32)
        k.gemm_simt(a, w, None, None, plain, k.EPILOGUE_F32)
        odd = ~plain.isfinite()
        assert bool((~out[odd].isfinite()).all()) and torch.equal(out[odd].isnan(), plain[odd].isnan())
        assert bool((out[odd][~plain[odd].isnan()] == plain[odd][~plain[odd].isnan()]).all())
        size = a.double().abs() @ w.double().abs().T
        good = plain.isfinite()
        assert bool(((out.double() - plain.double()).abs() <= (2.0 ** -24 + k_dim * 2.0 ** -24) * size)[good].all())
    usual = micros(clean)
    # a look at 16 KB of a row, and (every row) at 208 of them in eight warps; plain chains took 10 and 300 times as long
    assert micros(with_nan) <= 2 * usual + 20 and micros(every) <= 8 * usual + 20


@pytest.mark.parametrize("m,n,twice", [(3, 300, False), (64, 300, False), (65, 300, None), (96, 300, None), (130, 1000, None),
                                       (300, 300, None), (389, 12288, True)])
def test_launches_are_counted(m, n, twice):
    """Tiles of more than 64 tokens have them split by a kernel of its own, into scratch memory; others need neither (None:
    whichever the plan takes)."""
    from torch.profiler import ProfilerActivity, profile

    from matricxon_b200.ops import kernels as k
    from matricxon_b200.ops.library import library

    a, w, out = torch.randn(m, 512, device=DEV), torch.randn(n, 512, device=DEV), torch.empty(m, n, device=DEV)
    k.gemm_f32_split(a, w, None, None, out, k.EPILOGUE_F32)
    torch.cuda.synchronize()
    before = k.launch_count
    with profile(activities=[ProfilerActivity.CUDA]) as seen:
        k.gemm_f32_split(a, w, None, None, out, k.EPILOGUE_F32)
        torch.cuda.synchronize()
    kernels = sum(e.count for e in seen.key_averages() if "f32_split" in e.key or "f32_skinny" in e.key)
    assert k.launch_count - before == kernels == 1 + (library().mx_gemm_f32_split_scratch(m, n, 512) > 0)
    assert twice is None or kernels == 1 + twice
