"""How the split-K kernel cuts an input gradient (csrc/stream_gemm.cu): rows of a tile and slices of K on a chip of 148 SMs."""
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
