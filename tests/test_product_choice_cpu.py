"""Which product runs, asked where there is no device to answer."""
import pytest
import torch


@pytest.mark.skipif(torch.cuda.is_available(), reason="the question has an answer here")
def test_an_answer_that_does_not_come_is_an_error_each_time():
    """How many clusters fit is asked of the device; without one the choice is not made, and nothing is remembered."""
    from dispec_b200.ops import library, tuning
    for _ in range(2):
        with pytest.raises(library.KernelError, match="how many clusters"):
            tuning._few_rows_faster(300, 1536, 8960, 148)


def pairs_plan(M, N, K, fits):
    import ctypes
    from dispec_b200.ops import library
    plan = (ctypes.c_int * 3)()
    rc = library.core().dsp_gemm_pairs_plan(M, N, K, (ctypes.c_int * 4)(*fits), plan)
    return None if rc else tuple(plan)


@pytest.mark.parametrize("M,N,K", [(300, 1536, 8960), (137, 512, 4096), (536, 1536, 1536)])
def test_pairs_of_a_device_that_holds_fewer_clusters(M, N, K):
    """A cluster size of which the device holds none is not planned with, and hides none of the others."""
    splits, _, clusters = pairs_plan(M, N, K, [74, 36, 22, 16])
    assert splits > 1
    for held in range(1, 4):
        fits = [74, 36, 22, 16][:held] + [0] * (4 - held)
        splits, chunks, clusters = pairs_plan(M, N, K, fits)
        assert 1 <= splits <= held and 0 < clusters <= fits[splits - 1] and chunks >= -(-M // 256)
    assert pairs_plan(M, N, K, [0, 0, 0, 0]) is None
    assert pairs_plan(M, N, K, [0, 36, 0, 0])[0] == 2


@pytest.mark.skipif(torch.cuda.is_available(), reason="the question has an answer here")
def test_a_cluster_query_that_fails_is_an_error():
    import ctypes
    from dispec_b200.ops import library
    with pytest.raises(library.KernelError, match="how many clusters"):
        library.check(library.core().dsp_gemm_pairs_faster(300, 1536, 8960, 148, 0))


@pytest.mark.parametrize("N,K,split", [(64, 512, False), (1536, 1024, False), (4096, 1532, False), (1, 1536, True), (1536, 1538, False),
                                       (3072, 2048, True)])
def test_which_products_of_floats_run_on_the_tensor_cores(N, K, split):
    from dispec_b200.ops import gemm
    w = torch.zeros((N, K))
    assert w.data_ptr() % 16 == 0 and gemm.split_supported(w) == split
    shifted = torch.zeros(N * K + 1)[1:].view(N, K)
    assert not gemm.split_supported(shifted)
