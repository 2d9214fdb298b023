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


def test_the_passes_check_their_arguments_without_a_gpu():
    lib = _native.lib()
    p, invalid, unsupported, misaligned = 4096, -1, -2, -3           # (never read: every call below ends before a launch)
    big = 1 << 40

    def forward(x=p, w=p, dtype=0, rows=32, k=64, n=96, ld_x=64, ld_w=64, out=p, work=p, size=big):
        return lib.fos_linear_train_forward(x, w, dtype, rows, k, n, ld_x, ld_w, 3, 3, 1, out, 0, n, work, size, 0)

    def backward(dy=p, x=p, w=p, dtype=0, rows=32, k=64, n=96, ld_dy=96, ld_x=64, ld_w=64, rounding=1, dx=p, dw=p, work=p, size=big):
        return lib.fos_linear_train_backward(dy, x, w, dtype, rows, k, n, ld_dy, ld_x, ld_w, 3, rounding, 1, 2, 3, 3, 1, dx, dw, 0, k, k, work, size, 0)

    for null in ("x", "w", "out", "work"):
        assert forward(**{null: 0}) == invalid, null
    for null in ("dy", "x", "w", "dx", "dw", "work"):
        assert backward(**{null: 0}) == invalid, null
    for call, others in ((forward, []), (backward, [{"ld_dy": 88}, {"rounding": 3}, {"rounding": -1}])):
        for wrong in ({"rows": 0}, {"k": 0}, {"n": 0}, {"ld_x": 56}, {"ld_w": 56}, {"dtype": 2}, {"size": 1024}, *others):
            assert call(**wrong) == invalid, (call, wrong)
        for wrong in ({"x": p + 8}, {"w": p + 8}, {"ld_x": 68}, {"ld_w": 68}, {"k": 60, "ld_x": 64, "ld_w": 64}):
            assert call(**wrong) == unsupported, (call, wrong)
        assert call(work=p + 16) == misaligned
    assert backward(rows=24) == unsupported and backward(dy=p + 8) == unsupported
    # a workspace that is one byte short
    assert forward(size=lib.fos_linear_train_forward_workspace_bytes(32, 64, 96) - 1) == invalid
    assert backward(size=lib.fos_linear_train_backward_workspace_bytes(32, 64, 96) - 1) == invalid


def test_scaled_if4_products_check_their_arguments_without_a_gpu():
    lib = _native.lib()
    p = 4096

    def call(a=p, a_sf=p, amax_a=p, fa=1, rule_a=3, b=p, amax_b=p, fb=1, rule_b=3, out=p, k_p=64, ldd=128, work=p, size=1 << 40):
        return lib.fos_gemm_if4_scaled(a, a_sf, amax_a, fa, 0, rule_a, 0, b, p, amax_b, fb, 0, rule_b, 0, out, 0, 128, 128, k_p, 128, 128, ldd, work, size, 0, 0)

    for wrong in ({"a": 0}, {"a_sf": 0}, {"amax_a": 0}, {"amax_b": 0}, {"b": 0}, {"out": 0}, {"fa": 7}, {"fb": 7}, {"rule_a": 9}, {"rule_b": -1}, {"k_p": 60},
                  {"ldd": 64}, {"work": 0}, {"size": lib.fos_gemm_if4_workspace_bytes(128, 128, 64) - 1}):
        assert call(**wrong) == -1, wrong
    assert call(work=p + 64) == -3
