"""The kernels for few tokens (K split over a cluster), for tiles on CTA pairs and for small tensors to quantize, at the
sizes where their tiles, splits and paddings end; the other kernels of the library and plain tensor operations are the
reference."""

from __future__ import annotations

import ctypes

import pytest
import torch
import torch.nn as nn

import fouroversix_b200 as fos
from fouroversix_b200 import _native
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


FEW_ROWS, PAIRS, SINGLE_128 = 1, 2, 128


def _kernel(m, n, k):
    """(kernel, CTAs that share a tile's K) of a problem on this device."""
    split = ctypes.c_int(0)
    sms = torch.cuda.get_device_properties(DEV).multi_processor_count
    return _native.lib().fos_gemm_fp4_kernel(m, n, k, 0, None, sms, ctypes.byref(split)), split.value


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp4"])
@pytest.mark.parametrize("m,n,k,kernel", [
    # the kernel for few rows: 16 and 32 token columns, splits of 2, 4 and 8 and none (more tiles than SMs), features and K
    # that end inside a tile and a stage
    (1, 8, 4096, (FEW_ROWS, 2)), (1, 136, 4160, (FEW_ROWS, 2)), (16, 392, 4032, (FEW_ROWS, 2)), (16, 130, 8128, (FEW_ROWS, 4)),
    (16, 1000, 8192, (FEW_ROWS, 4)), (7, 264, 16384, (FEW_ROWS, 8)), (17, 520, 8256, (FEW_ROWS, 4)), (32, 1032, 14336, (FEW_ROWS, 4)),
    (31, 264, 16448, (FEW_ROWS, 8)), (16, 18952, 1088, (FEW_ROWS, 1)), (32, 19000, 1024, (FEW_ROWS, 1)), (3, 18945, 64, (FEW_ROWS, 1)),
    # the 128 x 128 tiles of the single-CTA kernel
    (1, 8, 64, (SINGLE_128, 1)), (16, 130, 1984, (SINGLE_128, 1)), (17, 1000, 2048, (SINGLE_128, 1)), (32, 264, 4096, (SINGLE_128, 1)),
    (33, 128, 4160, (SINGLE_128, 1)), (64, 384, 8192, (SINGLE_128, 1)), (65, 1024, 4032, (SINGLE_128, 1)),
    (128, 136, 16384, (SINGLE_128, 1))])
def test_few_tokens(m, n, k, kernel, fmt):
    assert _kernel(m, n, k) == kernel
    qx, qw = _operands(m, n, k, fmt)
    want = _exact(qx, qw)
    canvas = torch.full((m + 1, n + 8), 7.0, device=DEV)
    out = _run(qx, qw, out=canvas[:m, :n])
    assert ((out - want).abs().max() / want.abs().max()).item() < SUM_ORDER
    assert (canvas[m:] == 7).all() and (canvas[:, n:] == 7).all()
    for t in ("bfloat16", "float16"):
        assert torch.equal(_run(qx, qw, t), out.to(getattr(torch, t)))
    assert torch.equal(_run(qx, qw), out)                                  # the partial sums are added in a fixed order
    assert ((_run(qx, qw, variant=128) - out).abs().max() / want.abs().max()).item() < SUM_ORDER


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


@pytest.mark.parametrize("tokens,k,kernel", [(5, 8192, (FEW_ROWS, 4)), (32, 8192, (FEW_ROWS, 4)), (5, 2880, (SINGLE_128, 1)),
                                             (100, 2880, (SINGLE_128, 1)), (333, 2880, (SINGLE_128, 1)), (2100, 1024, (PAIRS, 1))])
@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
def test_bias_added_by_the_gemm(tokens, k, kernel, dtype):
    """5000 features: the last tile of every kernel ends inside a piece of its columns."""
    assert _kernel(tokens, 5000, k) == kernel
    t = getattr(torch, dtype)
    torch.manual_seed(tokens)
    layer = nn.Linear(k, 5000, bias=True, device=DEV, dtype=t)
    fl = fos.FourOverSixLinear(layer, fos.ModuleQuantizationConfig(output_dtype=dtype)).quantize_weight_()
    x = torch.randn(tokens, k, device=DEV, dtype=t)
    recorded = fl(x)                                       # the bias wants a gradient: added outside
    assert recorded.requires_grad
    with torch.no_grad():
        fused = fl(x)
        assert torch.equal(fused, recorded.detach())
        fl.bias, bias = None, fl.bias
        assert torch.equal(fused, fl(x) + bias)


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
