"""Which biases the one-call linear layer hands to the GEMM: the entry is replaced by one that writes zeros and notes the
bias pointer it was given, so that no GPU is needed."""

from __future__ import annotations

import ctypes

import pytest
import torch
import torch.nn as nn
from torch.autograd import forward_ad

import fouroversix_b200 as fos
from fouroversix_b200 import _native


class _Entry:
    def __init__(self):
        self.bias = None

    def fos_linear_workspace_bytes(self, rows, k):
        return 256

    def fos_linear_forward_bias(self, *args):
        rows, out_features, self.bias, out = args[2], args[10], args[11], args[12]
        ctypes.memset(out, 0, rows * out_features * 2)
        return 0


@pytest.fixture
def layer(monkeypatch):
    entry = _Entry()
    monkeypatch.setattr(_native, "lib", lambda: entry)
    monkeypatch.setattr(_native, "stream_ptr", lambda device: 0)
    fl = fos.FourOverSixLinear(nn.Linear(64, 24, bias=True, dtype=torch.bfloat16), fos.ModuleQuantizationConfig())
    weight = fos.QuantizedTensor(torch.zeros(128, 32, dtype=torch.uint8), torch.zeros(512).to(torch.float8_e4m3fn), torch.ones(1),
                                 "nvfp4", (24, 64), "mse", "nearest", (128, 64))
    x = torch.zeros(3, 64, dtype=torch.bfloat16)

    def forward(bias):
        fl._parameters["bias"] = bias
        entry.bias = None
        return fl._forward_one_call(x, weight)

    return entry, forward


def test_a_bias_of_one_element_per_feature_goes_to_the_gemm(layer):
    entry, forward = layer
    bias = torch.randn(24).bfloat16()
    forward(bias)
    assert entry.bias == bias.data_ptr()


@pytest.mark.parametrize("shape", [(1,), (), (3, 24), (1, 24), (3, 1)])
def test_a_bias_of_another_shape_is_broadcast(layer, shape):
    entry, forward = layer
    bias = torch.randn(shape).bfloat16()
    assert torch.equal(forward(bias), bias.expand(3, 24)) and entry.bias == 0


@pytest.mark.parametrize("length", [0, 23, 25])
def test_a_bias_of_a_wrong_length_is_refused(layer, length):
    _, forward = layer
    with pytest.raises(RuntimeError):
        forward(torch.zeros(length, dtype=torch.bfloat16))


def test_a_tangent_of_the_bias_reaches_the_output(layer):
    entry, forward = layer
    bias, tangent = torch.randn(24).bfloat16(), torch.randn(24).bfloat16()
    with forward_ad.dual_level():
        y, dy = forward_ad.unpack_dual(forward(forward_ad.make_dual(bias, tangent)))
        assert torch.equal(y, bias.expand(3, 24)) and torch.equal(dy, tangent.expand(3, 24)) and entry.bias == 0


def test_a_batch_of_biases(layer):
    _, forward = layer
    biases = torch.randn(5, 24).bfloat16()
    assert torch.equal(torch.func.vmap(forward)(biases), biases[:, None].expand(5, 3, 24))


def test_a_bias_with_a_pending_negation_and_one_of_a_subclass(layer):
    entry, forward = layer

    class Own(torch.Tensor):
        pass

    bias = torch.randn(24).bfloat16()
    assert torch.equal(forward(torch._neg_view(bias)), -bias.expand(3, 24)) and entry.bias == 0
    assert type(forward(bias.as_subclass(Own))) is Own and entry.bias == 0
