"""Width of the tiles of a product on single SMs (148 of them): narrow where that keeps more SMs busy, but not for a handful of rows of wide outputs."""
import pytest

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN


@pytest.mark.parametrize("M,N,K,mode,width", [
    (256, 2304, 768, KN.MODE_STORE, 64), (256, 3072, 768, KN.MODE_GELU, 64), (1024, 2304, 768, KN.MODE_STORE, 128), (896, 3072, 2048, KN.MODE_STORE, 256),
    (4, 3072, 768, KN.MODE_GELU, 64), (63, 768, 3072, KN.MODE_GELU, 64),
    (4, 6144, 4096, KN.MODE_GELU, 128), (16, 8192, 2048, KN.MODE_DGELU, 128), (1, 14336, 2048, KN.MODE_GELU, 256), (4, 6400, 1600, KN.MODE_STORE, 128),
    (48, 14336, 768, KN.MODE_STORE, 256), (64, 6144, 4096, KN.MODE_GELU, 64)])
def test_width(M, N, K, mode, width):
    lib = _lib.cuda()
    if lib.llmc_device_sm_count() not in (0, 148):
        pytest.skip("another number of SMs")
    assert lib.llmc_gemm_pick_width(M, N, K, mode) == width
