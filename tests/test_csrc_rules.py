"""Rules of the CUDA sources that no run can be relied on to show, checked on the text.

A kernel launched with the programmatic-stream-serialization attribute is resident while its predecessor still writes.  Its
inputs are therefore not read-only for its lifetime, which is what ld.global.nc asks for; __ldg is that load, and a pointer
to const that is __restrict__ lets the compiler choose it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "pariskv_b200", "csrc")


def _source(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _block(text, at, opening, closing):
    """The text from the first `opening` behind `at` to its match."""
    start = text.index(opening, at)
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == opening) - (text[i] == closing)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced")


def _kernels(text):
    """{name: (parameters, body)} of the __global__ functions."""
    out = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^{;]*?\)\s+)?(\w+)\s*\(", text):
        params = _block(text, m.end() - 1, "(", ")")
        out[m.group(1)] = (params, _block(text, m.end() + len(params) - 1, "{", "}"))
    return out


def _dependent(text):
    """Kernels that the file launches dependently."""
    return set(re.findall(r"(?:launch_chain\(|cudaLaunchKernelEx\(&cfg,)\s*(\w+)", text))


def test_dependently_launched_kernels_use_plain_loads_and_wait():
    seen = set()
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = _source(path)
        kernels, names = _kernels(text), _dependent(text)
        for name in names - {"kernel"}:
            params, body = kernels[name]
            seen.add(name)
            assert not re.search(r"\bconst\b[^,()]*__restrict__", params), f"{name}: a pointer to const is __restrict__"
            assert "pdl_wait()" in body and "pdl_trigger()" in body, f"{name}: no wait or no trigger"
            assert body.index("pdl_wait()") < body.index("pdl_trigger()"), f"{name}: triggers before it has waited"
    assert len(seen) >= 15, seen


def test_no_read_only_loads_in_device_code():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = _source(path)
        assert "__ldg(" not in text and "ld.global.nc" not in text, path
