"""The kernels for few tokens (K split over a cluster), for tiles on CTA pairs and for small tensors to quantize, at the
sizes where their tiles, splits and paddings end; the other kernels of the library and plain tensor operations are the
reference."""

from __future__ import annotations

import pytest
import torch
import torch.nn as nn

import fouroversix_b200 as fos
from fouroversix_b200.matmul import B200MatmulBackend
from fouroversix_b200.quantize.backend import B200QuantizeBackend

pytestmark = pytest.mark.gpu

DEV = "cuda"
# fp32 accumulation of K products in two different orders: each sum is off by about sqrt(K) u of a typical output, and the
# largest output is some 4 times that (sqrt(8192) * 2^-24 / 4 = 1.3e-6); the bar of the other GEMM tests
SUM_ORDER = 1e-5


def _operands(m, n, k, fmt, seed=1):
    g = torch.Generator(device=DEV).manual_seed(seed)
    cfg = fos.QuantizationConfig(dtype=fmt, scale_rule="static_6" if fmt == "mxfp4" else "mse")
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) * 0.05).bfloat16()
    return fos.quantize(x, cfg), fos.quantize(w, cfg)


def _exact(qx, qw):
    return fos.dequantize(qx, torch.float32).double() @ fos.dequantize(qw, torch.float32).double().T


def _run(qx, qw, out_dtype="float32", **kw):
    return B200MatmulBackend.quantized_matmul(qx, qw, out_dtype=fos.DataType(out_dtype), check_status=True, **kw)


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp4"])
@pytest.mark.parametrize("m,n,k", [(1, 8, 64), (16, 130, 1984), (17, 1000, 2048), (32, 264, 4096), (33, 128, 4160), (64, 384, 8192),
                                   (65, 1024, 4032), (128, 136, 16384)])
def test_few_tokens(m, n, k, fmt):
    qx, qw = _operands(m, n, k, fmt)
    want = _exact(qx, qw)
    canvas = torch.full((m + 1, n + 8), 7.0, device=DEV)
    out = _run(qx, qw, out=canvas[:m, :n])
    assert ((out - want).abs().max() / want.abs().max()).item() < SUM_ORDER
    assert (canvas[m:] == 7).all() and (canvas[:, n:] == 7).all()
    for t in ("bfloat16", "float16"):
        assert torch.equal(_run(qx, qw, t), out.to(getattr(torch, t)))
    assert torch.equal(_run(qx, qw), out)                                  # the partial sums are added in a fixed order


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp4"])
@pytest.mark.parametrize("m,n,k", [(129, 264, 64), (256, 256, 320), (384, 640, 1344), (300, 1000, 2880), (2304, 2176, 704)])
def test_cta_pairs_equal_single_ctas(m, n, k, fmt):
    """Odd row and column blocks, scale groups that end inside and across tiles, several tiles per pair: every MMA adds
    the same products in the same order as in the single-CTA kernel."""
    qx, qw = _operands(m, n, k, fmt)
    for t in ("float32", "bfloat16"):
        canvas = torch.full((m + 1, n + 16), 7.0, device=DEV, dtype=getattr(torch, t))
        out = _run(qx, qw, t, out=canvas[:m, :n], variant=2)
        assert torch.equal(out, _run(qx, qw, t, variant=256))
        assert (canvas[m:] == 7).all() and (canvas[:, n:] == 7).all()
    assert torch.equal(_run(qx, qw, variant=2, max_ctas=4), _run(qx, qw, variant=256))


@pytest.mark.parametrize("m,n,k", [(4736, 2048, 64), (2176, 4744, 192), (1920, 5000, 1088)])
def test_if4_on_cta_pairs(m, n, k):
    qx, qw = _operands(m, n, k, "if4")
    want = _exact(qx, qw)
    out = _run(qx, qw)
    # the fp16 operands round value * scale (2^-11 each, independent: far below the sum's own size)
    assert ((out - want).abs().max() / want.abs().max()).item() < 1e-3
    assert torch.equal(_run(qx, qw, "bfloat16"), out.bfloat16())


@pytest.mark.parametrize("rule", ["mse", "static_6", "mae"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 1000), (128, 64), (16, 8192), (17, 8192), (128, 2048), (129, 1008), (4097, 64)])
def test_small_tensors_equal_the_general_kernels(rows, cols, dtype, rule):
    """At most 8192 blocks (16384 without padding rows) in one cluster, and beyond; a strided input; the padding is zero in
    values and scales."""
    g = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.randn(rows, cols + 8, generator=g, device=DEV)
    x[:, ::97] *= 30
    x[rows // 2] = 0
    x = x.to(dtype)[:, :cols]
    cfg = fos.QuantizationConfig(scale_rule=rule)
    got = B200QuantizeBackend.quantize(x, cfg)
    for other in ("general", "no_tma"):
        want = B200QuantizeBackend.quantize(x, cfg, kernel=other)
        assert torch.equal(got.amax, want.amax) and torch.equal(got.values, want.values)
        assert torch.equal(got.scale_factors.view(torch.uint8), want.scale_factors.view(torch.uint8))


@pytest.mark.parametrize("tokens", [5, 100, 333])
@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
def test_bias_added_by_the_gemm(tokens, dtype):
    t = getattr(torch, dtype)
    torch.manual_seed(tokens)
    layer = nn.Linear(2880, 5000, bias=True, device=DEV, dtype=t)
    fl = fos.FourOverSixLinear(layer, fos.ModuleQuantizationConfig(output_dtype=dtype)).quantize_weight_()
    x = torch.randn(tokens, 2880, device=DEV, dtype=t)
    recorded = fl(x)                                       # the bias wants a gradient: added outside
    assert recorded.requires_grad
    with torch.no_grad():
        assert torch.equal(fl(x), recorded.detach())


@pytest.mark.parametrize("counts", [(1000, 0, 1281, 127, 1792, 1), (640, 900)])
@pytest.mark.parametrize("n,k", [(2904, 320), (1000, 1344)])
def test_grouped_problems_on_cta_pairs(counts, n, k):
    """Groups of odd and even numbers of row blocks, an empty one, one row: the buffer is long enough per group for
    256-row tiles, whose second half reaches into the next group; the 128-row kernel is the reference."""
    from fouroversix_b200.matmul.grouped import GroupLayout, StackedQuantizedTensor, grouped_quantize, grouped_quantized_matmul

    g = torch.Generator(device=DEV).manual_seed(n)
    layout = GroupLayout.from_counts(torch.tensor(counts, device=DEV), sum(counts))
    x = torch.randn(layout.capacity, k, generator=g, device=DEV).bfloat16()
    w = [fos.quantize((torch.randn(n, k, generator=g, device=DEV) * 0.05).bfloat16()) for _ in counts]
    gq, stacked = grouped_quantize(x, layout), StackedQuantizedTensor.stack(w)
    outs = {}
    for variant in (0, 256):
        canvas = torch.full((layout.capacity, n), 7.0, dtype=torch.bfloat16, device=DEV)
        outs[variant] = grouped_quantized_matmul(gq, stacked, out_dtype=fos.DataType.bfloat16, out=canvas, variant=variant)
    assert torch.equal(outs[0], outs[256])


@pytest.mark.parametrize("variant", [0, 2])
def test_a_limit_of_one_cta(variant):
    qx, qw = _operands(300, 600, 320, "nvfp4")
    assert torch.equal(_run(qx, qw, variant=variant, max_ctas=1), _run(qx, qw, variant=256))
