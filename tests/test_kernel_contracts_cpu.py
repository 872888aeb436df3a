"""What kernels that begin beside the end of the one before them (csrc/cuda/launch.cuh) have to keep to, checked in the
sources: the faults it prevents come from rare timing, which no run on a GPU shows."""
import re
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parent.parent / "rannc_b200" / "csrc" / "cuda"


def _source(name):
    """The file without comments."""
    text = re.sub(r"/\*.*?\*/", " ", (CUDA / name).read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _closing(text, start, pair="{}"):
    """Position behind the bracket that closes the one at `start`."""
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def _kernels(name):
    """{kernel: (parameters, body)} of one file."""
    text, out = _source(name), {}
    for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^)]*(?:\([^)]*\))?[^)]*\)\s*)?(\w+)\(", text):
        end = _closing(text, m.end() - 1, "()")
        body = text.index("{", end)
        out[m.group(1)] = (text[m.end():end - 1], text[body:_closing(text, body)])
    return out


# kernels that are launched with launch_after
EARLY = [(f.name, k) for f in sorted(CUDA.glob("*.cu")) for k, (_, body) in _kernels(f.name).items() if "grid_wait()" in body]


def test_every_kernel_that_begins_early_waits():
    text = "".join(_source(f.name) for f in sorted(CUDA.glob("*.cu")))
    names = {k for _, k in EARLY}
    assert {"gemm_tcgen05_kernel", "attn_fwd_kernel", "attn_fwd_persist_kernel", "attn_bwd_kernel", "ln_fwd_kernel"} <= names
    # a launch names the kernel, or a variable that was set to it
    for m in re.finditer(r"launch_after\w*\(\s*(?:\w+,\s*)?(\w+)", text):
        arg = m.group(1)
        sets = set(re.findall(rf"auto {arg}\s*=\s*([^;]+);", text)) or {arg}
        assert all(set(re.findall(r"\w+_kernel", s)) <= names for s in sets), arg


@pytest.mark.parametrize("file,kernel", EARLY)
def test_what_a_kernel_that_begins_early_reads(file, kernel):
    params, body = _kernels(file)[kernel]
    assert not re.search(r"const\s+[\w:]+\s*\*\s*(?:const\s*)?__restrict__", params)
    for text in (body, _source(file), *(_source(h.name) for h in CUDA.glob("*.cuh"))):
        assert not re.search(r"ld\.global(\.\w+)*\.nc\b|\b__ldg\b", text)
