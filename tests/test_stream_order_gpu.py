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
