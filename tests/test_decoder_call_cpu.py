"""The argument of the natively issued decoder pass is declared twice, in C++ and for ctypes: same fields, same order, same size."""
import ctypes
import os
import re

import pytest

from llmc_b200 import _lib

CSRC = os.path.join(os.path.dirname(_lib.__file__), "csrc")


def test_fields():
    body = re.search(r"struct DecoderCall \{(.*?)\n\};", open(os.path.join(CSRC, "decoder.cu")).read(), re.S).group(1)
    want = []
    for decl in re.sub(r"//.*", "", body).split(";"):
        m = re.match(r"\s*(?:const )?(bf16|float|int)\b(.*)", decl, re.S)
        if m:
            for name in m.group(2).split(","):
                kind = ctypes.c_void_p if "*" in m.group(2) else {"int": ctypes.c_int, "float": ctypes.c_float}[m.group(1)]
                want.append((name.strip(" *\n"), kind))
    assert want == list(_lib.DecoderCall._fields_)


def test_a_library_with_another_size_is_refused(monkeypatch):
    class Shorter(ctypes.Structure):
        _fields_ = _lib.DecoderCall._fields_[:-2]

    monkeypatch.setattr(_lib, "_cuda", None)
    assert _lib.cuda().llmc_decoder_call_size() == ctypes.sizeof(_lib.DecoderCall)
    monkeypatch.setattr(_lib, "_cuda", None)
    monkeypatch.setattr(_lib, "DecoderCall", Shorter)
    with pytest.raises(_lib.KernelError):
        _lib.cuda()
