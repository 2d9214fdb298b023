"""A kernel launched as a programmatic dependent may be resident while the kernel before it still writes what it will read.
__ldg and ld.global.nc are for memory that nobody writes while a kernel runs, so behind griddepcontrol.wait they have no
place (whatever a run shows: it is the compiler's choice where such a load lands)."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fouroversix_b200" / "csrc"
READ_ONLY = re.compile(r"__ldg\s*\(|\bldg_nc_\w+\s*\(|ld\.global\.nc")
# the kernels that start when the one-word zero kernel before them has ended: whatever wrote x was complete before that
BEHIND_A_FINISHED_WRITER = {"amax_kernel", "amax_rht_kernel"}


def _code(name: str) -> str:
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _functions(text: str) -> dict[str, str]:
    """Top-level functions by name (a body ends at the first line that is a lone brace)."""
    found = {}
    for m in re.finditer(r"^(?:template[^\n]*\n)?(?:__global__|__device__)[^{;]*?\b(\w+)\(.*?^}", text, re.S | re.M):
        head = m.group(0).split("{", 1)[0]
        name = re.findall(r"\b(\w+)\s*\(", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", head))[0]
        found[name] = found.get(name, "") + m.group(0)
    return found


@pytest.mark.parametrize("name", ["fos_experts.cu", "fos_gemm_nvfp4.cu", "fos_gemm_skinny.cuh", "fos_pair.cuh"])
def test_files_whose_kernels_are_all_dependents(name):
    assert not READ_ONLY.findall(_code(name))


@pytest.mark.parametrize("name", ["fos_quantize.cu", "fos_gemm_if4.cu"])
def test_kernels_that_wait(name):
    functions = _functions(_code(name))
    waiting = {n for n, body in functions.items() if "griddepcontrol.wait" in body}
    assert len(waiting) >= (7 if name == "fos_quantize.cu" else 1), waiting
    for n in (waiting | {"group_tiles"} & set(functions)) - BEHIND_A_FINISHED_WRITER:
        assert not READ_ONLY.findall(functions[n]), n


def test_small_tensors_are_loaded_coherently():
    """quantize_small_kernel loads through a helper whose default is for memory that is already complete."""
    body = _functions(_code("fos_quantize.cu"))["quantize_small_kernel"]
    assert "load_block_words<T, true>(" in body and "load_block_words<T>(" not in body
