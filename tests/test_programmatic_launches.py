"""Kernels that may run beside the kernel before them on their stream.

A kernel launched programmatically (launch_pass, pass_wait) is resident while
its predecessor still writes.  The read-only data path (ld.global.nc: __ldg, or
a const __restrict__ pointer) is defined only for memory that nobody writes
during the kernel's life, so such a kernel may use it for nothing but what no
kernel of its chain writes.  This reads the sources, those of the device
functions that the kernels call included: no GPU is needed.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mantaflow_gb300", "csrc")
# built once per solve, before the chain: the stencil codes and the ghost-fluid
# diagonal, their vector views, and a tuple of the multigrid's stencil dictionary
UNWRITTEN = {"code", "A0f", "c2", "A4", "t"}


def _source(path):
    text = open(path).read()
    return re.sub(r"/\*.*?\*/|//[^\n]*", "", text, flags=re.S)


def _functions(text):
    """name -> (parameters, body) of the functions with a body at the top level"""
    out = {}
    for m in re.finditer(r"\b(\w+)\s*\(([^(){};]*)\)\s*(?:const\s*)?\{", text):
        if m.group(1) in ("if", "for", "while", "switch"):
            continue
        depth, at = 1, m.end()
        while depth and at < len(text):
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        out[m.group(1)] = (m.group(2), text[m.end():at])
    return out


def _read_only_uses(name, functions, seen):
    """(function, pointer) of every use of the read-only path in name and what it calls"""
    if name in seen or name not in functions:
        return []
    seen.add(name)
    params, body = functions[name]
    uses = [(name, p) for p in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params)]
    uses += [(name, p) for p in re.findall(r"__ldg\s*\(\s*&?\s*\(?\s*(\w+)", body)]
    for callee in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", body)):
        uses += _read_only_uses(callee, functions, seen)
    return uses


def _kernels(path):
    shared = "".join(_source(p) for p in sorted(glob.glob(os.path.join(CSRC, "*.cuh"))))
    text = _source(path)
    functions = _functions(shared)
    functions.update(_functions(text))
    return functions, [n for n, (_, body) in functions.items() if n.startswith("k_") and "pass_wait()" in body]


FILES = ["advect.cu", "pressure.cu", "miccluster.cu", "multigrid.cu"]


@pytest.mark.parametrize("name", FILES)
def test_overlapped_kernels_read_what_others_write_with_ordinary_loads(name):
    functions, kernels = _kernels(os.path.join(CSRC, name))
    for k in kernels:
        bad = sorted({u for u in _read_only_uses(k, functions, set()) if u[1] not in UNWRITTEN})
        assert not bad, "%s: read-only loads of %s" % (k, bad)
