"""Which kernel a weight gradient goes to, by sizes and by whether it adds to what is there (148 SMs)."""
import pytest
import torch

from llmc_b200 import _lib
from llmc_b200.ops import kernels as KN


class Library:
    def __init__(self):
        self.called = []

    def __getattr__(self, name):
        return lambda *args: self.called.append(name) or 0


@pytest.mark.parametrize("rows,OC,C,accumulate,kernel", [
    (256, 2304, 768, False, "llmc_gemm"), (1024, 3072, 768, False, "llmc_gemm"),             # 27 and 36 tiles for 74 pairs
    (256, 2304, 768, True, "llmc_gemm2"), (64, 768, 768, True, "llmc_gemm2"),                # adding
    (256, 1600, 1600, False, "llmc_gemm2"), (1024, 3072, 1024, False, "llmc_gemm2"),         # 49 and 48 tiles
    (1032, 768, 768, False, "llmc_gemm2"), (256, 384, 384, True, "llmc_gemm"),               # many rows; four tiles
])
def test_kernel(monkeypatch, rows, OC, C, accumulate, kernel):
    lib = Library()
    monkeypatch.setattr(_lib, "cuda", lambda: lib)
    monkeypatch.setattr(KN, "sm_count", lambda device: 148)
    monkeypatch.setattr(KN, "_stream", lambda: None)
    z = lambda *s: torch.empty(*s, dtype=torch.bfloat16)
    KN.matmul_wgrad(z(OC, C), z(rows, OC), z(rows, C), accumulate=accumulate)
    assert [n for n in lib.called if n in ("llmc_gemm", "llmc_gemm2")] == [kernel]
