"""Rules of programmatic dependent launch (csrc/common/launch.cuh) that can be read off the kernel sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csrc"
SOURCES = [p for p in sorted(CSRC.rglob("*.cu")) if "launch_pdl" in p.read_text()]


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def _kernels(code):
    """(name, parameter list, body) of every `__global__` function."""
    for m in re.finditer(r"__global__[^;{(]*(?:\([^()]*(?:\([^()]*\))?[^()]*\)\s*)??\b(\w+)\s*\(", code):
        i = m.end()
        depth = 1
        while depth:
            depth += {"(": 1, ")": -1}.get(code[i], 0)
            i += 1
        params = code[m.end():i - 1]
        b = code.index("{", i)
        j, depth = b + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(code[j], 0)
            j += 1
        yield m.group(1), params, code[b:j]


def test_the_sources_are_found():
    assert {"norm.cu", "elementwise.cu", "gemm_sm100.cu", "flash_fwd_sm100.cu", "flash_bwd_sm100.cu", "block_fwd.cu"} <= {p.name for p in SOURCES}
    waiting = {n for p in SOURCES for n, _, body in _kernels(_code(p)) if "pdl_wait()" in body}
    assert {"layernorm_fwd_vec_kernel", "layernorm_bwd_vec_kernel", "binary_kernel", "gate_kernel", "colsum_vec_kernel", "dact_colsum_kernel"} <= waiting


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_kernels_launched_early_stay_off_the_read_only_path(path):
    """A kernel that may be resident before its predecessor has finished must not read what that one writes through L1's
    read-only path: neither explicitly nor by a `const T* __restrict__` parameter, which lets the compiler take it."""
    code = _code(path)
    assert "__ldg(" not in code
    for name, params, body in _kernels(code):
        if "pdl_wait()" in body:
            assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", params), name


@pytest.mark.parametrize("path", sorted(CSRC.rglob("*.cu")), ids=lambda p: p.name)
def test_shared_arrays_read_as_vectors_are_declared_aligned(path):
    """A `__shared__ float` array is aligned to 4 bytes; reading it as float4 needs the declaration to say 16."""
    code = _code(path)
    scalars = {"float", "int", "uint32_t", "unsigned", "__nv_bfloat16", "uint8_t", "char", "half"}
    for m in re.finditer(r"__shared__\s+((?:__align__\(\d+\)\s*)?)(\w+)\s+([^;]*);", code):
        align, typ, names = m.groups()
        if typ not in scalars or align:
            continue
        for name in re.findall(r"(\w+)\s*\[", names):
            assert not re.search(r"reinterpret_cast<(?:const )?(?:float|uint|int)[24]\s*\*>\(\s*&?\s*%s\b" % name, code), (path.name, name)


@pytest.mark.parametrize("path", [p for p in sorted(CSRC.rglob("*.cuh")) if "pdl_wait()" in p.read_text() and p.name != "launch.cuh"], ids=lambda p: p.name)
def test_kernel_headers_stay_off_the_read_only_path(path):
    code = _code(path)
    assert "__ldg(" not in code and not re.search(r"const\s+\w+\s*\*\s*__restrict__", code)
