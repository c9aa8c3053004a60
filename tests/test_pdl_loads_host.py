"""Kernels under programmatic launch and the non-coherent load path, by reading
the sources: such a kernel is resident while its predecessor still writes, so
only the operator's tables, which the handle's creation finished, may go through
__ldg or a const __restrict__ parameter."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "doublyexcited_b200", "csrc")
TABLES = ("a.t1a", "a.v12", "tq +", "vt +")  # tq, vt: pointers into the two tables


def _kernels(text):
    """(name, parameters, body) of every __global__ function."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params = text[m.end():i - 1]
        start = i = text.index("{", i) + 1
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), params, text[start:i]


def violations(text):
    out = []
    for name, params, body in _kernels(text):
        if "pdl_enter()" not in body and "grid_wait()" not in body:
            continue
        if re.search(r"const\s+[\w:]+\s*\*\s*__restrict__", params):
            out.append(f"{name}: const __restrict__ parameter")
        out += [f"{name}: __ldg({a}" for a in re.findall(r"__ldg\(\s*([^,;]{1,12})", body) if not a.startswith(TABLES)]
        out += [f"{name}: {f}" for f in re.findall(r"\b(col_elem|ld2|__ldcg)\(", body)]
    return out


@pytest.mark.parametrize("source", ["blockops.cu", "gram_tile.cu", "hammult_line.cu", "symops.cu"])
def test_kernels_under_programmatic_launch_load_coherently(source):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    assert sum("pdl_enter()" in b or "grid_wait()" in b for _, _, b in _kernels(text)) >= 2
    assert violations(text) == []
