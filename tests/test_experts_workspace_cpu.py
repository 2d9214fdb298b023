"""The scratch of an experts layer: buffers whose lives do not meet share their place."""

from __future__ import annotations

import pytest

from fouroversix_b200 import _native


@pytest.mark.parametrize("tokens,top,experts,hidden,inter", [(1, 1, 1, 64, 64), (256, 4, 32, 2880, 2880), (8192, 4, 32, 2880, 2880), (8192, 2, 8, 4096, 1024)])
def test_gathered_rows_product_and_result_share_their_place(tokens, top, experts, hidden, inter):
    lib = _native.lib()
    capacity = (tokens * top + 127 * experts + 127) // 128 * 128
    need = lib.fos_experts_forward_workspace_bytes(tokens, top, experts, hidden, inter)
    packed = capacity * (hidden + inter) * 9 // 16
    shared = max(2 * hidden, 4 * inter) * capacity
    tables = 4 * (tokens * (2 * top + 1) + 2 * capacity + 140 * experts)
    assert shared + 2 * inter * capacity + packed <= need <= shared + 2 * inter * capacity + packed + tables + 16 * 256
    apart = lib.fos_experts_workspace_bytes(tokens, top, experts, hidden, inter)
    assert apart - need == (4 * hidden + 4 * inter) * capacity - shared
    assert lib.fos_experts_forward_workspace_bytes(0, top, experts, hidden, inter) == -1
