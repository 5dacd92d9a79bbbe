"""Which bias gradients take one launch without scratch: few rows, but neither very wide nor too large for L2."""
import pytest

from llmc_b200 import _lib


@pytest.mark.parametrize("rows,OC,one_launch", [(1, 8, True), (1024, 2304, True), (1025, 2304, False), (1024, 28672, True), (777, 50304, True), (1024, 50304, False),
                                                (1, 65536, True), (1, 65544, False), (384, 128256, False)])
def test_rule(rows, OC, one_launch):
    assert (_lib.cuda().llmc_bias_grad_scratch(rows, OC) == 0) == one_launch
