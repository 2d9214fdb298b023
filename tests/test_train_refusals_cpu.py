"""What a training pass hands to its one-call form, and what it leaves to the calls one by one, which refuse with a reason."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

import fouroversix_b200 as fos
from fouroversix_b200.model.linear import _one_call_training_applies


def _operand(rows=64, cols=128, dtype=torch.bfloat16, ld=None):
    strides = (ld or cols, 1)
    return SimpleNamespace(shape=(rows, cols), dtype=dtype, device="cuda:0", is_cuda=True, stride=lambda i: strides[i], data_ptr=lambda: 1 << 20)


@pytest.mark.parametrize("output,taken", [("bfloat16", True), ("float16", True), ("float32", True), ("nvfp4", False), ("mxfp4", False)])
def test_an_output_type_that_is_none_is_left_to_be_refused(output, taken):
    """(Taken, it ended in a bare KeyError.)"""
    config = fos.ModuleQuantizationConfig(keep_master_weights=True, output_dtype=output)
    assert _one_call_training_applies(config, _operand(), _operand(32)) is taken


@pytest.mark.parametrize("output", ["bfloat16", "float32"])
def test_an_output_type_by_its_name_is_one(output):
    config = fos.ModuleQuantizationConfig(keep_master_weights=True)
    config.output_dtype = output
    assert _one_call_training_applies(config, _operand(), _operand(32))


@pytest.mark.parametrize("operand", [_operand(cols=100), _operand(ld=132), _operand(rows=0), _operand(dtype=torch.float32), _operand(dtype=torch.float16)])
def test_operands_it_does_not_take(operand):
    config = fos.ModuleQuantizationConfig(keep_master_weights=True)
    assert not _one_call_training_applies(config, _operand(), operand)
