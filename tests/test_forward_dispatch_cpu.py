"""Which kernel a plain forward product goes to, by sizes alone (148 SMs)."""
import pytest
import torch

from llmc_b200.ops import kernels as KN

DEV = torch.device("cuda", 0)


@pytest.fixture(autouse=True)
def sms(monkeypatch):
    monkeypatch.setattr(KN, "sm_count", lambda device: 148)


# deep products that both the swapped and the split-K kernel can do: the swapped one has conditions on the output that the other does not have
@pytest.mark.parametrize("M,N,K", [(500, 2056, 14336), (385, 2056, 6144), (2048, 1000, 6144)])
def test_ragged_outputs_stay_with_the_split_k_kernel(M, N, K):
    assert KN.forward_kernel(M, N, K, DEV) == KN.FORWARD_SWAPPED
    assert KN.forward_kernel(M, N + 4, K, DEV) == KN.FORWARD_STREAM
    assert KN.forward_kernel(M, N - 7, K, DEV) == KN.FORWARD_STREAM
    assert KN.forward_kernel(M, N, K, DEV, aligned=False) == KN.FORWARD_STREAM


# either side of the line of the sliced forward products: rows, depth against the number of tiles, tiles whose four slices are resident at once
@pytest.mark.parametrize("M,N,K,kernel", [
    (129, 768, 768, KN.FORWARD_SLICED), (128, 768, 768, KN.FORWARD_STREAM), (256, 768, 760, KN.FORWARD_GEMM), (256, 768, 3072, KN.FORWARD_SLICED),
    (1024, 1024, 4096, KN.FORWARD_SLICED), (1025, 1024, 4096, KN.FORWARD_SWAPPED), (512, 1024, 1024, KN.FORWARD_SLICED), (513, 1024, 1024, KN.FORWARD_SWAPPED),
    (256, 2304, 768, KN.FORWARD_SWAPPED), (300, 2048, 7168, KN.FORWARD_SLICED), (300, 4096, 14336, KN.FORWARD_STREAM)])
def test_sliced_products(M, N, K, kernel):
    assert KN.forward_kernel(M, N, K, DEV) == kernel
    if kernel == KN.FORWARD_SLICED:
        assert KN.forward_kernel(M, N - 3, K, DEV, aligned=False) == kernel
