"""Kernels that write another CTA's shared memory wait for the whole cluster first.

The CTAs of a cluster are scheduled together, but one may still be starting while
another already stores into its shared memory; the store is defined only after a
cluster barrier that all have arrived at. Read from the sources: such a race shows
on no device reliably."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "bartels_gb300", "csrc")


def _source(f):
    """Without comments and launch bounds."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
    return re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)


def _functions(text):
    """{name: body} of the functions of a source."""
    out = {}
    for m in re.finditer(r"(\w+)\s*\([^;{}]*\)\s*(?:const\s*)?\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out.setdefault(m.group(1), text[m.end():i])
    return out


def _kernels():
    found = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = _source(f)
        if "shared::cluster" not in text:
            continue
        fns = _functions(text)
        writers = [n for n, b in fns.items() if "st.shared::cluster" in b]
        for k in re.findall(r"__global__\s+void\s+(\w+)\s*\([^;{}]*\)\s*\{", text):
            hits = [m.start() for w in writers for m in re.finditer(rf"\b{w}\s*(?:<|\()", fns[k])]
            hits += [m.start() for m in re.finditer(r"st\.shared::cluster", fns[k])]
            if hits:
                waits = [n for n, b in fns.items() if "barrier.cluster.wait" in b and n not in writers]
                found.append(pytest.param(fns[k], min(hits), waits, id=f"{f}:{k}"))
    return found


KERNELS = _kernels()


def test_there_is_one():
    assert KERNELS


@pytest.mark.parametrize("body,first,waits", KERNELS)
def test_a_cluster_wait_precedes_the_first_remote_store(body, first, waits):
    before = [m.start() for w in waits for m in re.finditer(rf"\b{w}\s*\(", body)]
    before += [m.start() for m in re.finditer(r"barrier\.cluster\.wait", body)]
    assert any(i < first for i in before)
