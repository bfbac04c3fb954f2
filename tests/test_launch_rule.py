"""Kernels launched while the one before may still run: what holds their loads behind the wait, read from the source.

A kernel that begins with grid_wait() either takes its block index from it, so that every address depends on the
wait, and then does not use blockIdx; or it declares no pointer __restrict__, so that its loads are ordinary ones."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "appfis_gb300", "csrc")


def _kernels():
    """(file, name, parameters, body) of every kernel."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            at, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            params = text[m.end():at - 1]
            begin = text.index("{", at)
            end, depth = begin + 1, 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            out.append((os.path.basename(path), m.group(1), params, text[begin + 1:end - 1]))
    return out


KERNELS = _kernels()


def test_all_kernels_are_seen():
    sources = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
    assert len(KERNELS) == len(re.findall(r"^[^/\n]*__global__\s+void", sources, re.M)) > 30
    waiting = {k[1] for k in KERNELS if "grid_wait()" in k[3]}
    launched = set(re.findall(r"gb::launch\((?:first \? )?(\w+)", sources))
    named = launched & {k[1] for k in KERNELS}
    assert len(named) > 15 and named <= waiting


@pytest.mark.parametrize("kernel", [k for k in KERNELS if "grid_wait()" in k[3]], ids=lambda k: "%s:%s" % k[:2])
def test_loads_stay_behind_the_wait(kernel):
    _, _, params, body = kernel
    first = body.strip()
    if first.startswith("const gb::BlockId bid = gb::grid_wait();"):
        assert "blockIdx" not in body
    else:
        assert first.startswith("gb::grid_wait();")
        assert "__restrict__" not in params
