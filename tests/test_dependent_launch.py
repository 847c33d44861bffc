"""Kernels launched before their predecessor ends (common.cuh, launch_dependent), read as text: each waits before
its work, and none promises the compiler that what it reads is unchanged for its whole lifetime."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "zolo-svd_b200", "csrc")


def _sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                out[f] = re.sub(r"//[^\n]*", "", fh.read())
    return out


def _match(text, i, a, b):
    depth = 0
    for k in range(i, len(text)):
        depth += (text[k] == a) - (text[k] == b)
        if depth == 0:
            return k + 1
    raise ValueError(f"unbalanced {a}")


def _dependent_kernels():
    src = _sources()
    found = []
    for f, text in src.items():
        names = set()
        for m in re.finditer(r"\blaunch_dependent\(", text):
            args = text[m.end():_match(text, m.end() - 1, "(", ")")]
            if args.lstrip().startswith("void"):
                continue  # its definition
            first = re.split(r",\s*(?:grid|dim3)", args)[0]
            names |= set(re.findall(r"\b\w+_kernel\b", first))
        for name in sorted(names):
            found.append((f, name, text))
    return found


KERNELS = _dependent_kernels()


def test_kernels_are_found():
    assert len(KERNELS) >= 25


@pytest.mark.parametrize("f,name,text", KERNELS, ids=[k[1] for k in KERNELS])
def test_dependent_kernel(f, name, text):
    m = re.search(r"__global__[^;{}]*?\b" + name + r"\(", text)
    assert m, f"{name} is not defined in {f}"
    end = _match(text, m.end() - 1, "(", ")")
    params = text[m.end():end]
    start = text.index("{", end)
    body = text[start:_match(text, start, "{", "}")]
    assert "__restrict__" not in params and "__ldg" not in body and "global.nc" not in body
    assert len(re.findall(r"\bdependency_wait\(\)", body)) == 1
