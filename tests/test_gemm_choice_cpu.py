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


def test_where_the_kernel_for_few_rows_is_taken():
    """Up to 16 rows from 16 stages of K (256 values each), 17 to 32 from 32; any K where there are more tiles than SMs."""
    for m, n, k, kernel in ((16, 1000, 3841, FEW_ROWS), (16, 1000, 3840, NARROW), (17, 1000, 7937, FEW_ROWS), (17, 1000, 7936, NARROW),
                            (32, 1000, 7937, FEW_ROWS), (33, 1000, 16384, NARROW), (32, 128 * SMS, 64, FEW_ROWS),
                            (32, 128 * (SMS - 1), 64, NARROW)):
        assert choice(m, n, k)[0] == kernel, (m, n, k)
        assert choice(m, n, k, max_ctas=SMS)[0] != FEW_ROWS and choice(m, n, k, variant=128)[0] != FEW_ROWS
    # K is shared by as many CTAs as are resident at once (two per SM), each keeping eight stages, eight at most
    assert [choice(16, n, 16384)[1] for n in (8, 128 * 37, 128 * 38, 128 * 74, 128 * 75, 128 * SMS)] == [8, 8, 4, 4, 2, 2]
    assert [choice(16, 8, k)[1] for k in (4096, 8191, 8192, 16384, 1 << 20)] == [2, 4, 4, 8, 8]


def test_where_the_swiglu_is_fused():
    """From 640 buffer rows per group with K of 1536 and more, from 512 with K of 2048 and more, from 320 with K of 2880 and six sure
    rounds, never with a smaller K: there the epilogue, and below those rows the idle halves of the pairs, cost more than the
    kernel that they save."""
    fused = lambda rows, hidden, inter, experts: _native.lib().fos_experts_glu_is_fused(rows, hidden, inter, experts, SMS)
    for experts, inter in ((8, 1024), (32, 2880)):
        for rows, hidden, want in ((256, 2880, 0), (384, 2816, 0), (512, 1984, 0), (512, 2048, 1), (640, 1472, 0), (640, 1536, 1), (2048, 1024, 0)):
            assert fused(rows * experts, hidden, inter, experts) == want, (rows, hidden)
        assert fused(640 * experts - 128, 1536, inter, experts) == 0 and fused(512 * experts - 128, 2048, inter, experts) == 0
    # 32 groups of 320 buffer rows, 23 column tiles: 24 row tiles of their own at least, 552 tiles on 74 pairs
    assert fused(320 * 32, 2880, 2880, 32) == 1 and fused(320 * 32 - 128, 2880, 2880, 32) == 0
    assert fused(320 * 32, 2880, 1024, 32) == 0 and fused(384 * 8, 4096, 2048, 8) == 0                # 192 tiles; 128
    assert fused(640, 2048, 64, 1) == 0                      # one narrow tile per row block: not a problem for wide tiles
    assert fused(100, 2048, 64, 1) < 0 and fused(640, 2000, 64, 1) < 0 and fused(640, 2048, 64, 0) < 0


def test_where_few_rows_take_narrow_tiles():
    """Up to 64 rows of a group's own beside its 127 spare ones, where narrow tiles fill their last round better."""
    for rows, want in ((47 * 128, NARROW), (48 * 128, WIDE)):                  # 32 groups: 191 rows each are 6112
        assert choice(rows, 2880, 2880, 32)[0] == want
    assert choice(40 * 128, 2880, 2880, 32)[0] == NARROW                       # 3 x 256 columns against 5 x 128
    assert choice(40 * 128, 5760, 2880, 32)[0] == WIDE                         # 5 x 256 either way: the wide tiles stay
    assert choice(11 * 128, 2048, 1024, 8)[0] == NARROW and choice(12 * 128, 2048, 1024, 8)[0] == WIDE
