"""Which kernel a bfloat16 product of 9 to 16 rows runs on: the streaming one where the 16-row kernel's blocks stop fitting
at a time and an SM's share of the weights fills the streaming kernel's ring, or is 64 rows."""

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,n,k_dim,expected", [
    (8, 49152, 64, "skinny"), (9, 4736, 3072, "skinny"), (9, 4752, 3072, "stream"), (16, 4737, 3072, "stream"),
    # less than a ring's worth an SM (5,120 x 2,048 takes the 16-row kernel 8.4 us and the streaming one 9.7)
    (9, 4752, 2048, "skinny"), (16, 4737, 2048, "skinny"), (9, 5120, 2048, "skinny"), (16, 6144, 1024, "skinny"),
    (16, 6511, 2048, "skinny"), (16, 6512, 2048, "stream"), (9, 9324, 512, "skinny"), (9, 9325, 512, "stream"),
    # K in two halves: twice the blocks, up to the width at which the kernel does that
    (16, 2368, 6144, "skinny"), (16, 2384, 6144, "stream"), (16, 3552, 6144, "stream"), (16, 3568, 6144, "skinny"),
    (16, 2384, 6112, "skinny"), (16, 3072, 6176, "skinny"), (17, 37889, 64, "stream"), (17, 4752, 64, "library")])
def test_rule(m, n, k_dim, expected, monkeypatch):
    from matricxon_b200.ops import kernels, linear

    monkeypatch.setattr(kernels, "sm_count", lambda device: 148)
    monkeypatch.setattr(kernels, "stream_gemm_supported", lambda a, w: True)
    x, w = torch.empty(m, k_dim, dtype=torch.bfloat16), torch.empty(n, k_dim, dtype=torch.bfloat16)
    assert linear.chosen_backend(x, w) == expected
