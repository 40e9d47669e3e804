"""Rules of the kernels that are launched before their predecessor's end, checked in
their source: no thread leaves before it has waited for the predecessor, and a load
that the compiler may take for constant must not read what an earlier kernel of the
chain writes."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cuda_pf_localization_b200" / "csrc"
# filled by copies from the host or before the chain, never by one of its kernels
HOST_WRITTEN = {"F", "T", "cyc", "obs", "lm", "draw_f"}
# the map's cells, and the weights of a kernel of its own launch
CONSTANT_LOADS = {"src[k]", "w4[q]"}


def _source(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced source")


def _kernels():
    """(name, parameters, body) of every kernel that waits for its predecessor."""
    for path in sorted(CSRC.glob("*.cu")):
        text = _source(path)
        for m in re.finditer(r"__global__", text):
            k = re.compile(r"\b(k_\w+)\s*\(").search(text, m.end())
            end = _closing(text, k.end() - 1, "()")
            start = text.index("{", end)
            body = text[start:_closing(text, start, "{}")]
            if "pdl_wait()" in body:
                yield k.group(1), text[k.end():end], body


def _launched():
    return {n for p in CSRC.glob("*.cu")
            for n in re.findall(r"launch_pdl\(\s*(k_\w+)", _source(p))}


KERNELS = list(_kernels())


def test_every_programmatic_kernel_waits():
    assert _launched() and _launched() == {n for n, _, _ in KERNELS}


@pytest.mark.parametrize("name,params", [(n, p) for n, p, _ in KERNELS],
                         ids=[n for n, _, _ in KERNELS])
def test_nothing_a_chain_writes_is_constant(name, params):
    held = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
    assert held <= HOST_WRITTEN


def test_constant_loads():
    for path in list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")):
        for arg in re.findall(r"__ldg\(\s*&((?:[^()]|\([^()]*\))*)\)", _source(path)):
            assert re.sub(r"\s+", "", arg) in CONSTANT_LOADS, (path.name, arg)


@pytest.mark.parametrize("name,body", [(n, b) for n, _, b in KERNELS],
                         ids=[n for n, _, _ in KERNELS])
def test_no_thread_leaves_before_the_wait(name, body):
    assert body.count("pdl_wait()") == 1
    assert not re.search(r"\breturn\b", body[:body.index("pdl_wait()")])
