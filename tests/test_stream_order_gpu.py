"""Kernels that may be resident while the kernel before them in the stream still writes (programmatic dependents): each
result is compared with the same call after a synchronisation."""

from __future__ import annotations

import pytest
import torch

import fouroversix_b200 as fos
from fouroversix_b200 import _native
from fouroversix_b200.quantize.backend import B200QuantizeBackend

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _gather(x, rows, out):
    """`out` = x[rows] by fos_experts_gather_rows, which lets its dependents start before it writes."""
    _native.check(_native.lib().fos_experts_gather_rows(
        x.data_ptr(), _native.elem_code(x.dtype), x.stride(0), rows.data_ptr(), out.data_ptr(), out.stride(0), out.shape[0],
        out.shape[1], 0, 0, _native.stream_ptr(x.device)), "fos_experts_gather_rows")


def _same(got, want):
    return (torch.equal(got.amax, want.amax) and torch.equal(got.values, want.values)
            and torch.equal(got.scale_factors.view(torch.uint8), want.scale_factors.view(torch.uint8)))


@pytest.mark.parametrize("rule", ["mse", "static_6"])
@pytest.mark.parametrize("first_column,kernel", [(1, "auto"), (0, "no_tma"), (0, "auto")])
def test_quantize_with_a_given_amax_behind_the_writer_of_its_input(first_column, kernel, rule):
    """A view off the 16-byte grid, and an aligned one, take the kernel that loads x into registers."""
    g = torch.Generator(device=DEV).manual_seed(first_column)
    x = torch.randn(256, 4096, generator=g, device=DEV).bfloat16()
    rows = torch.randint(256, (4096,), generator=g, device=DEV, dtype=torch.int32)
    amax = x.abs().max().float()
    cfg = fos.QuantizationConfig(scale_rule=rule)
    want = None
    for _ in range(8):
        out = torch.full((4096, 4096), 3.0, dtype=torch.bfloat16, device=DEV)
        view = out[:, first_column:]
        _gather(x, rows, out)
        if want is None:
            torch.cuda.synchronize()
            want = B200QuantizeBackend.quantize(view, cfg, amax=amax, kernel=kernel)
        else:
            assert _same(B200QuantizeBackend.quantize(view, cfg, amax=amax, kernel=kernel), want)


def test_product_right_behind_the_kernel_that_packs_its_second_operand():
    """The amax word of a small second operand is written at the end of the kernel before the GEMM."""
    g = torch.Generator(device=DEV).manual_seed(5)
    qx = fos.quantize(torch.randn(256, 512, generator=g, device=DEV).bfloat16())
    ws = [(torch.randn(256, 512, generator=g, device=DEV) * 2.0 ** i).bfloat16() for i in range(-4, 4)]
    want = []
    for w in ws:
        qw = fos.quantize(w)
        torch.cuda.synchronize()
        want.append(fos.quantized_matmul(qx, qw))
    for w, y in zip(ws, want, strict=True):
        assert torch.equal(fos.quantized_matmul(qx, w), y)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("columns", [512, 509])
def test_small_tensor_right_behind_its_writer(columns, dtype):
    g = torch.Generator(device=DEV).manual_seed(columns)
    x = torch.randn(64, 512, generator=g, device=DEV).to(dtype)
    for i in range(8):
        rows = torch.randint(64, (128,), generator=g, device=DEV, dtype=torch.int32)
        out = torch.full((128, 512), 3.0, dtype=dtype, device=DEV)
        _gather(x, rows, out)
        got = fos.quantize(out[:, :columns])
        torch.cuda.synchronize()
        assert _same(got, fos.quantize(out[:, :columns])), i


def test_experts_layer_with_another_routing_each_time():
    from fouroversix_b200.model.experts import FourOverSixExperts

    g = torch.Generator(device=DEV).manual_seed(8)
    e, h, i, tokens = 8, 512, 256, 96
    weights = [torch.randn(*s, generator=g, device=DEV).mul(0.05).bfloat16() for s in ((e, 2 * i, h), (e, 2 * i), (e, h, i), (e, h))]
    layer = FourOverSixExperts(*weights)
    calls = []
    with torch.no_grad():
        for _ in range(6):
            x = torch.randn(tokens, h, generator=g, device=DEV).bfloat16()
            scores, indices = torch.randn(tokens, e, generator=g, device=DEV).topk(2)
            calls.append((x, indices, scores.softmax(-1).bfloat16()))
        want = []
        for c in calls:
            want.append(layer(*c))
            torch.cuda.synchronize()
        got = [layer(*c) for c in calls]
    for y, z in zip(got, want, strict=True):
        assert torch.equal(y, z)
