"""The experts layer as one call (rows gathered by the quantization, SwiGLU in the gate-up GEMM's epilogue where that runs on
CTA pairs) against its kernels called one by one, bit by bit."""

from __future__ import annotations

import pytest
import torch

from fouroversix_b200 import _native
from fouroversix_b200.model import FourOverSixExperts
from fouroversix_b200.model.config import ModuleQuantizationConfig

pytestmark = pytest.mark.gpu


def _layer(experts, hidden, inter, dtype, rule="mse"):
    g = torch.Generator(device="cuda").manual_seed(hidden + inter)
    cfg = ModuleQuantizationConfig(scale_rule=rule, output_dtype="bfloat16" if dtype is torch.bfloat16 else "float16")
    draw = lambda scale, *shape: (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)
    return FourOverSixExperts(draw(0.05, experts, 2 * inter, hidden), draw(0.1, experts, 2 * inter), draw(0.05, experts, hidden, inter),
                              draw(0.1, experts, hidden), cfg)


# tokens, experts per token, experts, hidden, inter; the last three: groups long enough for CTA pairs
SHAPES = [(1, 1, 2, 64, 64), (37, 3, 5, 128, 192), (256, 4, 32, 192, 128), (2050, 2, 4, 192, 320), (1777, 3, 6, 64, 448),
          (4096, 4, 16, 320, 512)]
# with the SwiGLU in the gate-up GEMM: 327 to 1152 buffer rows per group, products that end within a 256-column tile (640, 896, 1408,
# 5760) or on one (1024), K of whole and of broken stages. The last: tiles of 128 columns for few rows per expert
FUSED = [(2050, 2, 4, 1536, 320), (1777, 3, 6, 1600, 448), (800, 2, 4, 2048, 704), (1030, 3, 5, 2112, 512), (1600, 4, 32, 2880, 2880)]
SHAPES += FUSED + [(190, 2, 8, 128, 1024)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,top,experts,hidden,inter", SHAPES)
def test_one_call_equals_the_kernels_one_by_one(tokens, top, experts, hidden, inter, dtype):
    layer = _layer(experts, hidden, inter, dtype)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, hidden, generator=g, device="cuda").to(dtype)
    scores = torch.randn(tokens, experts, generator=g, device="cuda")
    scores[:, 0] += 1.0                                            # groups of different lengths
    if experts > top:
        scores[:, -1] = -1e9                                       # an expert nobody is routed to
    weights, indices = scores.softmax(-1).topk(top)
    weights = weights.to(dtype)
    if tokens > 100:
        x[tokens // 2] *= 300                                      # a token beyond the clamp's limit on both sides
        x[7, 5] = float("nan")
        indices[11, 0] = -1                                        # no expert for this slot
    got = layer(x, indices, weights)
    layer.single_call = False
    want = layer(x, indices, weights)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num(), want.nan_to_num()), int((got != want).sum())
    assert _native.wait_failure_site() == 0


@pytest.mark.parametrize("rule", ["mse", "static_6"])
@pytest.mark.parametrize("tokens,top,experts,hidden,inter", [SHAPES[1], SHAPES[3], FUSED[2], (300, 2, 4, 512, 64)])
def test_a_call_stays_within_its_workspace(monkeypatch, tokens, top, experts, hidden, inter, rule):
    """Two layers one after the other in the same scratch, with bytes behind it that must stay as they are."""
    layer = _layer(experts, hidden, inter, torch.bfloat16, rule)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    need = _native.lib().fos_experts_forward_workspace_bytes(tokens, top, experts, hidden, inter)
    work = torch.full((need + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
    empty = torch.empty
    cases = []
    for _ in range(2):
        x = torch.randn(tokens, hidden, generator=g, device="cuda").bfloat16()
        weights, indices = torch.randn(tokens, experts, generator=g, device="cuda").softmax(-1).topk(top)
        cases.append((x, indices, weights.bfloat16()))
    monkeypatch.setattr(torch, "empty", lambda *a, **k: work[:need] if a == (need,) else empty(*a, **k))
    got = [layer(*case) for case in cases]
    monkeypatch.undo()
    layer.single_call = False
    for case, out in zip(cases, got):
        assert torch.equal(out, layer(*case))
    assert (work[need:] == 0x5A).all()


@pytest.mark.parametrize("tokens,top,experts,hidden,inter", FUSED)
def test_the_fused_shapes_are(tokens, top, experts, hidden, inter):
    rows = (tokens * top + 127 * experts + 127) // 128 * 128
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _native.lib().fos_experts_glu_is_fused(rows, hidden, inter, experts, sms) == 1


@pytest.mark.parametrize("rule", ["static_6", "mae"])
def test_other_rules_gather_first(rule):
    layer = _layer(4, 192, 320, torch.bfloat16, rule)
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(2050, 192, generator=g, device="cuda").bfloat16()
    weights, indices = torch.randn(2050, 4, generator=g, device="cuda").softmax(-1).topk(2)
    got = layer(x, indices, weights.bfloat16())
    layer.single_call = False
    assert torch.equal(got, layer(x, indices, weights.bfloat16()))


@pytest.mark.parametrize("top", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("hidden", [8, 264, 2880])
def test_combine_keeps_the_order_of_the_experts(top, hidden):
    """(y + bias) * weight added in ascending order of the expert, every step rounded to the type."""
    g = torch.Generator(device="cuda").manual_seed(top)
    tokens, experts, rows = 53, 9, 53 * 8
    y = torch.randn(rows, hidden, generator=g, device="cuda").bfloat16()
    bias = torch.randn(experts, hidden, generator=g, device="cuda").bfloat16()
    weight = torch.rand(tokens, top, generator=g, device="cuda").bfloat16()
    expert = torch.stack([torch.randperm(experts, generator=g, device="cuda")[:top] for _ in range(tokens)]).int()
    row = torch.randperm(rows, generator=g, device="cuda")[: tokens * top].reshape(tokens, top).int()
    row[3, 0] = -1
    out = torch.empty(tokens, hidden, dtype=torch.bfloat16, device="cuda")
    _native.check(_native.lib().fos_experts_combine(
        y.data_ptr(), _native.FOS_BF16, y.stride(0), bias.data_ptr(), row.data_ptr(), expert.data_ptr(), weight.data_ptr(), top,
        out.data_ptr(), out.stride(0), tokens, hidden, _native.stream_ptr(y.device)), "fos_experts_combine")
    want = torch.zeros_like(out)
    order = expert.argsort(1)
    for k in range(top):
        at = order[:, k : k + 1].long()
        r, e, w = row.gather(1, at).squeeze(1), expert.gather(1, at).squeeze(1), weight.gather(1, at).squeeze(1)
        term = (y[r.clamp(min=0).long()] + bias[e.long()]) * w[:, None]
        want = torch.where((r >= 0)[:, None], want + term, want)
    assert torch.equal(out, want)
