"""Which kernel an FP4 GEMM takes: `fos_gemm_fp4_kernel`, the function that the entries decide with, needs no GPU."""

from __future__ import annotations

import ctypes

import pytest

from fouroversix_b200 import _native

SMS = 148
FEW_ROWS, PAIRS, NARROW, WIDE = 1, 2, 128, 256


def choice(m, n, k, groups=0, variant=0, max_ctas=0):
    split = ctypes.c_int(0)
    opts = _native.GemmOpts(variant, max_ctas)
    kernel = _native.lib().fos_gemm_fp4_kernel(m, n, k, groups, ctypes.byref(opts), SMS, ctypes.byref(split))
    return kernel, split.value


@pytest.mark.parametrize("m,n,k,groups", [(1, 8192, 8192, 0), (333, 5000, 2880, 0), (4096, 10240, 8192, 0), (32768, 28672, 8192, 0),
                                          (36864, 5760, 2880, 32)])
def test_a_limit_of_one_cta_is_kept(m, n, k, groups):
    """A pair is two CTAs."""
    for variant in (0, 2) if groups == 0 else (0,):
        assert choice(m, n, k, groups, variant, max_ctas=1)[0] in (NARROW, WIDE)
        assert choice(m, n, k, groups, variant, max_ctas=2)[0] in (NARROW, WIDE, PAIRS)
    if m > 1000:
        assert choice(m, n, k, groups)[0] == PAIRS and choice(m, n, k, groups, max_ctas=2)[0] == PAIRS


def test_a_named_variant_is_taken():
    for m, n, k in ((1, 8192, 8192), (4096, 10240, 8192), (100, 100, 64)):
        assert [choice(m, n, k, variant=v)[0] for v in (128, 256, 2)] == [NARROW, WIDE, PAIRS]
    assert choice(100, 100, 64, variant=3)[0] == -1 and choice(0, 100, 64)[0] == -1 and choice(512, 512, 64, 2, variant=2)[0] == -1
