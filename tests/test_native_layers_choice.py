"""When the layers of a step are issued natively: only while ``torch.mm``, which the native products stand in for, would do the same."""
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
