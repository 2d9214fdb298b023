"""What a training pass hands to its one-call form, and what it leaves to the calls one by one, which refuse with a reason."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

import fouroversix_b200 as fos
from fouroversix_b200 import _native
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


def _packed(rows, cols):
    values = (rows + 127) // 128 * 128 * ((cols + 63) // 64 * 64)
    return (values // 2 + 255) // 256 * 256 + (values // 16 + 255) // 256 * 256


@pytest.mark.parametrize("tokens,k,n", [(16, 16, 16), (4096, 4096, 4096), (32768, 8192, 28672), (272, 520, 1032)])
def test_a_pass_asks_for_the_room_of_its_own_operands(tokens, k, n):
    """Forward needs x and W packed and nothing of what backward needs (32768 tokens, 8192 -> 28672: 283 MB of 679)."""
    lib = _native.lib()
    forward, backward = (getattr(lib, f"fos_linear_train_{name}_workspace_bytes")(tokens, k, n) for name in ("forward", "backward"))
    assert forward == 256 + _packed(tokens, k) + _packed(n, k)
    assert backward == 256 + max(_packed(tokens, n), _packed(n, tokens)) + max(_packed(k, n), _packed(k, tokens))
    assert lib.fos_linear_train_workspace_bytes(tokens, k, n) == max(forward, backward)
    for name in ("forward_", "backward_", ""):
        assert getattr(lib, f"fos_linear_train_{name}workspace_bytes")(tokens, 0, n) == -1
