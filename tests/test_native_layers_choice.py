"""When the layers of a step are issued natively: only while ``torch.mm``, which the native products stand in for, would do the same,
and only through the library that PyTorch itself has loaded."""
import os
from types import SimpleNamespace

import pytest
import torch

from inf_engine_b200.parts import prenorm_layers
from inf_engine_b200.parts.prenorm_layers import NativeLayers


@pytest.fixture
def taken(monkeypatch):
    monkeypatch.setattr(prenorm_layers, "_library_product", lambda: 1)
    layers = NativeLayers.__new__(NativeLayers)
    return lambda: layers.takes(SimpleNamespace(n_tokens=200, max_q_len=100, host={}))


def test_full_precision_partial_sums_are_torch_mms(taken):
    assert taken()
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    try:
        assert not taken()
    finally:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = True
    assert taken()


def test_another_library_or_tuned_kernels_are_torch_mms(taken, monkeypatch):
    before = torch.backends.cuda.preferred_blas_library()
    try:
        torch.backends.cuda.preferred_blas_library("cublaslt")
        assert not taken()
    finally:
        torch.backends.cuda.preferred_blas_library(before)
    assert taken()
    monkeypatch.setattr(torch.cuda.tunable, "is_enabled", lambda: True)
    assert not taken()


@pytest.fixture
def looked_up(monkeypatch):
    """``_library_product`` anew, with the library that it opens and how."""
    opened = []

    class Library:
        def __init__(self, name, mode=0):
            opened.append((name, mode))
            if name != "libcublas.so.12":
                raise OSError(name)
            self.cublasGemmEx = prenorm_layers.ctypes.c_void_p(4096)

    monkeypatch.setattr(prenorm_layers, "_gemm_ex", None)
    monkeypatch.setattr(prenorm_layers.ctypes, "CDLL", Library)
    return lambda: (prenorm_layers._library_product(), opened)


def test_the_product_comes_from_a_library_that_is_loaded(looked_up):
    address, opened = looked_up()
    assert address == 4096 and len(opened) == 1 and opened[0][1] & os.RTLD_NOLOAD


def test_a_pytorch_of_another_major_version_gets_no_product_of_this_one(looked_up, monkeypatch):
    monkeypatch.setattr(torch.version, "cuda", "13.0")
    address, opened = looked_up()
    assert address == 0 and not opened
