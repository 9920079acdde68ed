"""Kernels that are launched while the one before them still runs read memory that it may still be writing.  Non-coherent loads (__ldg, and
what the compiler makes of const __restrict__) want memory that nobody writes while the kernel is resident: none in the sources of
those kernels.  Which load a kernel takes cannot be seen from its results, so this reads the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kvmix_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _kernels(code):
    """Name and text, from the template line or the __global__ to the closing brace at the start of a line."""
    return [(m.group(1), m.group(0)) for m in re.finditer(r"__global__[^{;]*?\b(\w+_kernel)\(.*?\n}\n", code, flags=re.S)]


def _reached(name, seen):
    if name not in seen:
        seen.add(name)
        for inc in re.findall(r'#include "([\w.]+)"', _code(name)):
            _reached(inc, seen)
    return seen


def _early():
    """(file, kernel) of what is launched early."""
    out = set()
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            code = _code(name)
            if "launch_early(" in code or "cudaLaunchAttributeProgrammaticStreamSerialization" in code:
                out |= {(name, k) for k, text in _kernels(code) if "grid_wait()" in text}
    return sorted(out)


def test_early_kernels_are_found():
    assert {k for _, k in _early()} == {"decode_attn_gqa_kernel", "decode_attn_mma_kernel", "gemv_mma_kernel", "prefill_kernel"}


@pytest.mark.parametrize("name,kernel", _early())
def test_no_load_wants_constant_memory(name, kernel):
    code = _code(name)
    for other, text in _kernels(code):                         # kernels of the same file that are launched in the ordinary way
        if other != kernel and "grid_wait()" not in text:
            code = code.replace(text, "")
    for where, text in [(name, code)] + [(f, _code(f)) for f in sorted(_reached(name, set()) - {name})]:
        assert not re.search(r"__ldg\b|ld\.global\.nc|const\s+[\w:]+\s*\*\s*__restrict__", text), where
