"""How the split-K kernel cuts an input gradient, and a forward product like one (csrc/stream_gemm.cu): rows of a tile and slices of K on a chip of 148 SMs."""
import ctypes

import pytest

from llmc_b200 import _lib


@pytest.fixture(scope="module")
def plan():
    lib = _lib.cuda()
    if lib.llmc_device_sm_count() not in (0, 148):
        pytest.skip("another number of SMs")

    def f(M, N, K, w_mn=1):
        rows, slices = ctypes.c_int(0), ctypes.c_int(0)
        lib.llmc_stream_gemm_plan(M, N, K, w_mn, ctypes.byref(rows), ctypes.byref(slices))
        return rows.value, slices.value
    return f


# small tiles while K is shallow, large ones with more slices where it is deep
@pytest.mark.parametrize("M,N,K,rows,slices", [
    (256, 768, 768, 64, 4), (256, 768, 3072, 64, 8), (1024, 768, 3072, 112, 4), (129, 768, 768, 48, 4), (1024, 1024, 2304, 128, 4), (256, 768, 50304, 64, 8),
    (384, 768, 50304, 192, 8), (512, 768, 50304, 256, 8), (384, 768, 14336, 192, 8), (200, 1600, 14336, 208, 8), (256, 2048, 14336, 64, 4),
    (512, 2048, 128256, 256, 4), (1024, 768, 50304, 256, 4), (129, 4096, 28672, 144, 4)])
def test_input_gradients(plan, M, N, K, rows, slices):
    assert plan(M, N, K) == (rows, slices)


def test_few_rows_and_forward_products_are_cut_as_before(plan):
    assert plan(4, 768, 50304) == (16, 8) and plan(100, 2048, 7168) == (112, 8)
    assert plan(300, 2048, 7168, 0) == (160, 4) and plan(128, 768, 3072, 0) == (128, 8)


# 15 clusters of eight large tiles fit the chip, 16 do not; deep forward products take small tiles only where the estimate is clearly for them
@pytest.mark.parametrize("M,N,K,gradient,forward", [
    (641, 576, 6784, (224, 8), (224, 8)), (768, 640, 6144, (256, 8), (256, 8)), (500, 1024, 8192, (64, 4), (64, 4)), (554, 704, 6400, (64, 4), (64, 4)),
    (269, 448, 14208, (64, 8), (144, 8)), (521, 1152, 7360, (80, 4), (176, 4)), (561, 1024, 6336, (80, 4), (80, 4)), (256, 768, 3072, (64, 8), (64, 8))])
def test_large_and_small_tiles(plan, M, N, K, gradient, forward):
    assert plan(M, N, K) == gradient and plan(M, N, K, 2) == forward
