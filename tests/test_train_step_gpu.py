"""A training step's passes as one host call each: the bits of the quantizations and products one by one."""

from __future__ import annotations

import pytest
import torch
from torch import nn

import fouroversix_b200 as fos
from fouroversix_b200 import _native
from fouroversix_b200.model.linear import FourOverSixLinearFunction, _one_call_training_applies

pytestmark = pytest.mark.gpu


def _step(layer, x, dy):
    torch.manual_seed(17)                      # the seeds of the noise come from torch's CPU generator
    x.grad = layer.weight.grad = None
    y = layer(x)
    y.backward(dy)
    return y.detach(), x.grad, layer.weight.grad


@pytest.mark.parametrize("tokens,k,n", [(16, 16, 16), (16, 24, 40), (48, 1040, 264), (272, 520, 1032), (1024, 512, 768), (2048, 2048, 2048)])
@pytest.mark.parametrize("style", ["nearest", "stochastic", "stochastic_unbiased"])
@pytest.mark.parametrize("rule,two_d", [("mse", True), ("static_6", False), ("mae", False)])
def test_one_call_passes_equal_call_by_call(monkeypatch, tokens, k, n, style, rule, two_d):
    g = torch.Generator(device="cuda").manual_seed(tokens + k)
    dtype = torch.float16 if rule == "static_6" else torch.bfloat16
    lin = nn.Linear(k, n, bias=False, device="cuda", dtype=dtype)
    layer = fos.FourOverSixLinear(lin, fos.ModuleQuantizationConfig(
        keep_master_weights=True, weight_scale_2d=two_d, scale_rule=rule, gradient_round_style=style,
        output_dtype="float16" if dtype is torch.float16 else "bfloat16"))
    x = torch.randn(tokens, k, generator=g, device="cuda").to(dtype).requires_grad_()
    dy = (torch.randn(tokens, n, generator=g, device="cuda") * 1e-3).to(dtype)
    assert _one_call_training_applies(layer.config, dy, x.detach(), lin.weight.data)
    one = _step(layer, x, dy)
    monkeypatch.setattr("fouroversix_b200.model.linear._one_call_training_applies", lambda *a: False)
    each = _step(layer, x, dy)
    for name, a, b in zip(("y", "dx", "dw"), one, each):
        assert torch.equal(a, b), (name, int((a != b).sum()))


def test_views_and_other_types_keep_their_results(monkeypatch):
    """Operands the one call does not take as they are (a column-major activation, a base that is not 16-byte aligned) and a
    strided one that it does take; an expanded gradient and rows that are not a multiple of 16 stay refused."""
    g = torch.Generator(device="cuda").manual_seed(2)
    lin = nn.Linear(64, 96, bias=True, device="cuda", dtype=torch.bfloat16)
    layer = fos.FourOverSixLinear(lin, fos.ModuleQuantizationConfig(keep_master_weights=True, gradient_round_style="nearest"))
    base = torch.randn(64, 256, generator=g, device="cuda").bfloat16()
    taken = FourOverSixLinearFunction._backward_one_call
    calls = []
    monkeypatch.setattr(FourOverSixLinearFunction, "_backward_one_call", staticmethod(lambda *a: calls.append(1) or taken(*a)))
    dense = torch.randn(64, 96, generator=g, device="cuda").bfloat16()
    for x, dy, expected in ((base[:, :64], dense, 1), (base[:, 4:68], dense, 0), (base.T[:64, :64], dense, 0)):
        calls.clear()
        got = _step(layer, x.detach().requires_grad_(), dy)
        assert len(calls) == expected
        want = _step(layer, x.detach().contiguous().requires_grad_(), dy.contiguous())
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    for x, dy in ((base[:20, :64], dense[:20]), (base[:, :64], dense[:1].expand(64, 96))):
        with pytest.raises(ValueError):
            _step(layer, x.detach().requires_grad_(), dy)


@pytest.mark.parametrize("tokens,k,n", [(16, 24, 40), (272, 520, 1032), (1024, 512, 64)])
def test_a_pass_stays_within_its_workspace(tokens, k, n):
    """Each with exactly the bytes that it asks for, in front of bytes that must stay as they are."""
    lib, g = _native.lib(), torch.Generator(device="cuda").manual_seed(n)
    draw = lambda rows, cols: torch.randn(rows, cols, generator=g, device="cuda").bfloat16()
    x, w, dy = draw(tokens, k), draw(n, k), draw(tokens, n)
    y, dx, dw = torch.empty_like(dy), torch.empty_like(x), torch.empty_like(w)
    stream = _native.stream_ptr(x.device)
    for name in ("forward", "backward"):
        need = getattr(lib, f"fos_linear_train_{name}_workspace_bytes")(tokens, k, n)
        work = torch.full((need + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
        if name == "forward":
            status = lib.fos_linear_train_forward(x.data_ptr(), w.data_ptr(), _native.FOS_BF16, tokens, k, n, k, k, 3, 3, 1, y.data_ptr(), _native.FOS_BF16, n,
                                                  work.data_ptr(), need, stream)
        else:
            status = lib.fos_linear_train_backward(dy.data_ptr(), x.data_ptr(), w.data_ptr(), _native.FOS_BF16, tokens, k, n, n, k, k, 3, 1, 5, 6, 3, 3, 1,
                                                   dx.data_ptr(), dw.data_ptr(), _native.FOS_BF16, k, k, work.data_ptr(), need, stream)
        _native.check(status, name)
        assert (work[need:] == 0x5A).all(), name
