"""Sizes that the product's C entries refuse, found before anything is asked of a GPU."""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from oneccl_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent
_ENTRIES = {  # arguments behind the sizes and the epilogue
    "cclx_gemm_bf16": (C.c_int(0), None, None),
    "cclx_gemm_bf16_2sm": (C.c_int(0), None, None),
    "cclx_gemm_bf16_rows": (None, None, None),
}


@pytest.mark.skipif(torch.cuda.is_available(), reason="what happens without a device")
def test_without_a_device_the_question_for_the_faster_mlp_is_an_error():
    """An exception that left the C entry would end the process."""
    lib, answer = _lib.load(), C.c_int(-7)
    assert lib.cclx_mlp_preferred(8192, 4096, C.byref(answer)) != 0 and answer.value == 0
    assert b"CUDA" in lib.cclx_last_error()


def test_the_mlp_leaves_cta_pairs_where_they_are_turned_off():
    code = ("import ctypes as C; from oneccl_b200 import _lib; n = C.c_int(-7); "
            "assert _lib.load().cclx_mlp_preferred(8192, 4096, C.byref(n)) == 0 and n.value == 0")
    subprocess.run([sys.executable, "-c", code], env={**os.environ, "CCL_CUDA_GEMM_2SM": "0"}, cwd=ROOT, check=True, timeout=300)


@pytest.mark.parametrize("M,N,K", [(0, 64, 64), (64, 0, 64), (64, 64, 0), (0, 0, 0), (-1, 64, 64), (3, 12, 64), (3, 64, 12)])
@pytest.mark.parametrize("entry", sorted(_ENTRIES))
def test_empty_and_odd_products_are_refused(entry, M, N, K):
    lib = _lib.load()
    assert getattr(lib, entry)(None, None, None, M, N, K, 0, *_ENTRIES[entry]) != 0
    assert b"unsupported GEMM shape" in lib.cclx_last_error()
