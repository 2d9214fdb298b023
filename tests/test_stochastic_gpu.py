"""Stochastic rounding and the rotation against restatements in plain torch: the noise is a hash of (seed, block, candidate,
value), so the bytes are defined, not only their distribution."""

from __future__ import annotations

import pytest
import torch

import fouroversix_b200 as fos
from fouroversix_b200.quantize import from_blocked
from fouroversix_b200.quantize.backend import B200QuantizeBackend

pytestmark = pytest.mark.gpu

M32 = 0xFFFFFFFF
SEED = 0x1234_5678_9ABC
GRID = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])


def _hash32(h: torch.Tensor) -> torch.Tensor:
    h = h ^ (h >> 16)
    h = (h * 0x7FEB352D) & M32
    h = h ^ (h >> 15)
    h = (h * 0x846CA68B) & M32
    return h ^ (h >> 16)


def _static_6_codes(x: torch.Tensor, amax: float) -> torch.Tensor:
    """Codes [rows, cols] of a tensor whose sides need no padding, NVFP4, static_6, every step in binary32."""
    rows, cols = x.shape
    v = x.float().reshape(rows, cols // 16, 16)
    encode = torch.tensor(2688.0) / torch.tensor(amax)
    decode = 1.0 / encode
    # (the maximum skips NaN, as the kernels' does)
    bmax = v.abs().nan_to_num(nan=0.0).amax(-1)
    scale = ((bmax / 6.0) * encode).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    r = torch.where(scale != 0, 1.0 / (decode * scale), torch.zeros(()))
    xs = v * r.unsqueeze(-1)
    block = torch.arange(rows * (cols // 16)).reshape(rows, cols // 16, 1)
    key = _hash32(_hash32(torch.tensor(SEED >> 32) ^ (block >> 27)) ^ (SEED & M32))
    i = torch.arange(16)
    h = _hash32(key ^ ((block * 32 + (i & ~1)) & M32))
    bits = torch.where(i % 2 == 0, h & 0xFFFF, h >> 16)
    noise = ((bits * 128 + 64).double() / 2 ** 23 - 0.5).float()          # (bits << 7 | 0x40) as a mantissa, minus 1.5
    a = xs.abs()
    step = torch.where(a < 2, 0.5, torch.where(a < 4, 1.0, 2.0))
    total = (a.double() / step + noise.double()).float()                   # one rounding, as a fused multiply-add
    mag = (total.round().clamp(min=0) * step).clamp(max=6.0)
    mag = torch.where(a.isnan(), torch.zeros(()), mag)
    code = torch.searchsorted(GRID, mag.contiguous())
    sign = torch.signbit(xs) & (xs != 0) & ~xs.isnan()
    code = torch.where(scale.unsqueeze(-1) != 0, code + 8 * sign, torch.zeros((), dtype=torch.long))
    return code.reshape(rows, cols)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["plain", "outlier", "nan", "small_amax", "zeros"])
@pytest.mark.parametrize("transpose", [False, True])
def test_stochastic_codes_are_the_hash(kind, dtype, transpose):
    g = torch.Generator().manual_seed(3)
    x = torch.randn(128, 448 if not transpose else 384, generator=g)
    if kind == "outlier":
        x[:, ::50] *= 20
    if kind == "nan":
        x[5, 7] = x[100, 300] = float("nan")
    if kind == "zeros":
        x[:, : x.shape[1] // 2] = 0.0
        x[3] = -x[3].abs() * 0.0
    x = x.to(dtype)
    # an amax below the maximum: scaled values beyond the grid, where the arranged form does not apply
    amax = float(x.float().abs().nan_to_num(nan=0.0).max()) * (0.05 if kind == "small_amax" else 1.0)
    cfg = fos.QuantizationConfig(scale_rule="static_6", round_style="stochastic", transpose=transpose)
    q = B200QuantizeBackend.quantize(x.cuda(), cfg, amax=torch.tensor([amax], device="cuda"), seed=SEED)
    want = _static_6_codes(x.T.contiguous() if transpose else x, amax)
    values = q.values.cpu().long()
    got = torch.stack((values & 15, values >> 4), -1).reshape(values.shape[0], -1)[: want.shape[0], : want.shape[1]]
    assert torch.equal(got, want), int((got != want).sum())


def _fma(a: torch.Tensor, b: torch.Tensor, c: torch.Tensor) -> torch.Tensor:
    """fl(a * b + c) of binary32 numbers (the product is exact in 64 bits)."""
    return (a.double() * b.double() + c.double()).float()


def _scaled(x: torch.Tensor, amax: float, largest_scale: float):
    """(blocks [rows, n, 16], block maximum / 6 times the encoding factor, the factor's inverse)."""
    rows, cols = x.shape
    v = x.float().reshape(rows, cols // 16, 16)
    encode = torch.tensor(6.0 * largest_scale) / torch.tensor(amax)
    return v, (v.abs().nan_to_num(nan=0.0).amax(-1) / 6.0) * encode, 1.0 / encode


def _draw(v: torch.Tensor, scale: torch.Tensor, decode: torch.Tensor, candidate: int, integers: bool = False):
    """(4-bit codes, sum of squared residuals in units of the scale) of one candidate, the sum in the order of the values."""
    rows, n, _ = v.shape
    r = torch.where(scale != 0, 1.0 / (decode * scale), torch.zeros(())).unsqueeze(-1)
    xs = v * r
    block = torch.arange(rows * n).reshape(rows, n, 1)
    key = _hash32(_hash32(torch.tensor(SEED >> 32) ^ (block >> 27)) ^ (SEED & M32))
    i = torch.arange(16)
    h = _hash32(key ^ ((block * 32 + candidate * 16 + (i & ~1)) & M32))
    bits = torch.where(i % 2 == 0, h & 0xFFFF, h >> 16)
    noise = ((bits * 128 + 64).double() / 2 ** 23 - 0.5).float()
    if integers:
        u = xs * torch.tensor(1.16666666)
        mag = (u.abs() + noise).round().clamp(min=0, max=7)
        q = torch.copysign(torch.where(u.isnan(), torch.zeros(()), mag), u)
        t = _fma(q, torch.tensor(0.8571428571), -xs)
        code = q.nan_to_num().long() & 15
    else:
        a = xs.abs()
        step = torch.where(a < 2, 0.5, torch.where(a < 4, 1.0, 2.0))
        mag = (_fma(a, 1.0 / step, noise).round().clamp(min=0) * step).clamp(max=6.0)
        mag = torch.where(a.isnan(), torch.zeros(()), mag)
        t = torch.copysign(mag, xs) - xs
        code = torch.searchsorted(GRID, mag.contiguous()) + 8 * (torch.signbit(xs) & (xs != 0) & ~xs.isnan())
    total = torch.zeros(rows, n)
    for k in range(16):
        total = _fma(t[..., k], t[..., k], total)
    zero = scale == 0
    return torch.where(zero.unsqueeze(-1), torch.zeros((), dtype=torch.long), code), torch.where(zero, torch.zeros(()), total)


def _byte(scale: torch.Tensor) -> torch.Tensor:
    return scale.to(torch.float8_e4m3fn).view(torch.uint8).long()


def _e4m3(x: torch.Tensor) -> torch.Tensor:
    return x.clamp(max=448.0).to(torch.float8_e4m3fn).float()


def _adaptive_codes(x: torch.Tensor, amax: float):
    """NVFP4 with a 4/6 rule: both candidates drawn with noise of their own, the smaller squared error of the draw wins."""
    v, hp, decode = _scaled(x, amax, 256.0)
    codes, errors, scales = [], [], []
    for candidate, scale in enumerate((_e4m3(hp), _e4m3(hp * 1.5))):
        c, e = _draw(v, scale, decode, candidate)
        g = (scale * torch.tensor(amax)) * torch.tensor(1.0 / 1536.0)
        codes.append(c)
        errors.append(torch.where(scale != 0, (e * g) * g, torch.zeros(())))
        scales.append(_byte(scale))
    take = errors[1] < errors[0]
    return torch.where(take.unsqueeze(-1), codes[1], codes[0]).reshape(x.shape), torch.where(take, scales[1], scales[0])


def _if4_codes(x: torch.Tensor, amax: float):
    """IF4: the E2M1 grid against the integer grid under one scale; the scale's sign bit says which."""
    v, hp, decode = _scaled(x, amax, 448.0)
    scale = _e4m3(hp)
    (c0, e0), (c1, e1) = _draw(v, scale, decode, 0), _draw(v, scale, decode, 1, integers=True)
    take = e1 < e0
    return torch.where(take.unsqueeze(-1), c1, c0).reshape(x.shape), _byte(scale) + 128 * take


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["plain", "outlier", "nan", "small_amax", "zeros"])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("form,rule", [("nvfp4", "mse"), ("nvfp4", "abs_max"), ("if4", "mse")])
def test_the_better_of_two_draws_is_taken(form, rule, kind, dtype, transpose):
    """The pick between two stochastically rounded candidates, codes and scale bytes, with the errors summed as stated."""
    g = torch.Generator().manual_seed(11)
    x = torch.randn(256, 448 if not transpose else 384, generator=g)
    if kind == "outlier":
        x[:, ::50] *= 20
    if kind == "nan":
        x[5, 7] = x[100, 300] = float("nan")
    if kind == "zeros":
        x[:, : x.shape[1] // 2] = 0.0
        x[3] = -x[3].abs() * 0.0
    x = x.to(dtype)
    amax = float(x.float().abs().nan_to_num(nan=0.0).max()) * (0.05 if kind == "small_amax" else 1.0)
    cfg = fos.QuantizationConfig(dtype=form, scale_rule=rule, round_style="stochastic", transpose=transpose)
    q = B200QuantizeBackend.quantize(x.cuda(), cfg, amax=torch.tensor([amax], device="cuda"), seed=SEED)
    y = x.T.contiguous() if transpose else x
    want, want_scales = (_if4_codes if form == "if4" else _adaptive_codes)(y, amax)
    values, scales = q.values.cpu().long(), q.scale_factors.view(torch.uint8).cpu().flatten()
    got = torch.stack((values & 15, values >> 4), -1).reshape(values.shape[0], -1)[: want.shape[0], : want.shape[1]]
    shape = (q.padded_shape[0], q.padded_shape[1] // 16)
    scales = (from_blocked(scales, shape) if q.scale_factors_are_in_blackwell_layout else scales.reshape(shape)).long()
    assert torch.equal(scales[: want_scales.shape[0], : want_scales.shape[1]], want_scales)
    assert torch.equal(got, want), int((got != want).sum())
    # both candidates win somewhere, or the comparison shows nothing
    if kind in ("plain", "outlier"):
        first = _draw(*(lambda v, hp, d: (v, _e4m3(hp), d))(*_scaled(y, amax, 448.0 if form == "if4" else 256.0)), 0)[0].reshape(y.shape)
        share = float((first != want).float().mean())
        assert 0.02 < share < 0.98, share

@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("shape", [(16, 16), (48, 80), (272, 1040)])
def test_rotated_amax(shape, transpose, dtype):
    """max |rotated tensor|: sums of sixteen 16-bit numbers that binary32 holds exactly (integers below 2^8), so the
    transform in 64 bits, rounded once to the type, is the value itself."""
    g = torch.Generator().manual_seed(shape[0] + transpose)
    x = torch.randint(-128, 129, shape, generator=g).to(dtype)
    signs = torch.tensor([1, 1, 1, -1, 1, -1, -1, -1, -1, -1, -1, 1, -1, 1, -1, -1], dtype=torch.float64)
    h = torch.ones(1, 1, dtype=torch.float64)
    for _ in range(4):
        h = torch.cat((torch.cat((h, h), 1), torch.cat((h, -h), 1)), 0)
    y = (x.T if transpose else x).double()
    rotated = ((y.reshape(y.shape[0], -1, 16) * signs) @ h * 0.25).to(dtype)
    q = fos.quantize(x.cuda(), fos.QuantizationConfig(rht=True, transpose=transpose))
    assert float(q.amax) == float(rotated.abs().max())
