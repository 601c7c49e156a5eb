"""Which float products the kernels for few and for many rows take, and which are too short in K for them."""

import pytest


@pytest.mark.parametrize("m,n,least", [
    (1, 2048, 0), (8, 4096, 0), (8, 8192, 32), (9, 2048, 32), (16, 8192, 64), (17, 2048, 64), (32, 8192, 128),
    (33, 16, 100), (2048, 2048, 100)])
def test_shortest_k(m, n, least):
    from matricxon_b200.ops.library import library

    pays = library().mx_gemm_f32_pays
    assert pays(m, n, least) and (least == 0 or not pays(m, n, least - 4))
    # a low-rank factor of a prompt stays with the general kernel, and so does a K whose fourth piece would be empty
    assert not pays(389, 2048, 16) and not pays(389, 2048, 160) and pays(389, 2048, 192)


def test_rows_that_lie_in_one_another_stay_on_the_fp32_cores():
    import torch
    from matricxon_b200.ops.linear import chosen_backend

    def at(make, m=40):
        memory = torch.zeros(200 * 1028 + 8)
        memory = memory[-(memory.data_ptr() // 4) % 4:]
        return chosen_backend(make(memory, m), torch.zeros(512, 1024))

    assert at(lambda x, m: x[:m * 1024].view(m, 1024)) == "split"
    assert at(lambda x, m: x.as_strided((m, 1024), (1028, 1))) == "split"
    assert at(lambda x, m: x[:1024].expand(m, 1024)) == "simt"              # one row for all
    assert at(lambda x, m: x.as_strided((m, 1024), (4, 1))) == "simt"       # windows that slide by four numbers
    assert at(lambda x, m: x.as_strided((m, 1024), (1026, 1))) == "simt"


@pytest.mark.parametrize("m,n,least", [(3, 256, 1024), (4, 16384, 1024), (5, 49152, 512), (8, 256, 512), (9, 4096, 2048),
                                       (16, 4096, 2048), (17, 4096, 1024), (32, 4096, 1024), (33, 4096, 512), (2048, 256, 512)])
def test_shortest_k_on_the_tensor_cores(m, n, least):
    from matricxon_b200.ops.library import library

    pays = library().mx_gemm_f32_split_pays
    assert pays(m, n, least) and not pays(m, n, least - 4) and not pays(m, 255, least)
    # one and two rows never, and three or four of a wide result not
    assert not pays(2, n, 12288) and not pays(1, n, 12288) and not pays(4, 16385, 12288)
