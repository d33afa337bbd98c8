"""CPU tests of rules that the kernel sources keep and no run can show broken reliably."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kiln_b200", "csrc")


def _code():
    """{file: source without comments}"""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
        out[os.path.basename(path)] = re.sub(r"//[^\n]*", "", text)
    return out


def test_no_non_coherent_loads():
    """A kernel launched with programmatic serialization lives while its predecessor still writes what it will read, and the
    non-coherent load path is outside the ordering of griddepcontrol.wait. `const T* __restrict__` parameters let the compiler choose
    that path by itself: only kernels that are launched plainly may have them."""
    code = _code()
    dependent = set(re.findall(r"launch_dependent\(\s*(?:split_k > 1 \? )?(\w+)", code["abi.cu"]))
    assert {"attn_fwd_kernel", "attn_bwd_kernel", "gemm16_kernel", "qk_prep_kernel"} <= dependent
    for name, text in code.items():
        assert not re.search(r"\b__ldg\b|ld\.global(\.\w+)*\.nc\b", text), f"{name}: non-coherent load"
        for kernel, params in re.findall(r"__global__[^;{]*?\b(\w+_kernel)\s*\(([^)]*)\)\s*\{", text):
            assert kernel not in dependent or "__restrict__" not in params, f"{name}: {kernel} has __restrict__ parameters"
