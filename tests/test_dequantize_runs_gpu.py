"""dequantize over the widths where a run of blocks begins to span rows, ends within one, or takes several, against the oracle."""

from __future__ import annotations

import pytest
import torch

import fouroversix_b200 as fos
from oracle import fos_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 512), (295, 1032), (296, 1040), (593, 520), (591, 1024), (67, 2048), (1185, 272), (1200, 528), (1183, 64),
                                       (9, 2056), (130, 4096), (3, 4104), (5, 8200)])
@pytest.mark.parametrize("dtype", ["nvfp4", "if4"])
def test_every_run_length(rows, cols, dtype):
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(rows + cols)).bfloat16()
    q = fos.quantize(x.cuda(), fos.QuantizationConfig(dtype=dtype))
    ref = fos_oracle.quantize(x, dtype=dtype)
    for out, view in ((torch.bfloat16, torch.int16), (torch.float16, torch.int16), (torch.float32, torch.int32)):
        assert torch.equal(fos.dequantize(q, out).cpu().view(view), fos_oracle.dequantize(ref, out).view(view))
