"""Kernels launched with programmatic serialization may start before their predecessor has finished: each of them has to wait for it
(csrc/common.cuh).  Read from the sources, since a kernel that does not wait gives right results most of the time."""
import glob
import os
import re

import pytest

import iian_b200

CSRC = os.path.join(os.path.dirname(iian_b200.__file__), "csrc")


def bodies(text):
    """name -> body of every ``__global__`` function of a source."""
    out = {}
    src = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\(", src):
        at = src.index("{", m.end())
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
            if depth == 0:
                break
        out[m.group(1)] = src[at:end]
    return out


def launched(text):
    """The kernels named in calls of ``iian_launch``; a variable is looked up where it was given its kernel."""
    names = set()
    for m in re.finditer(r"\biian_launch\(\s*(\w+)", text):
        name = m.group(1)
        if re.search(r"\bauto\s+%s\s*=" % name, text):
            names.update(n for v in re.findall(r"\bauto\s+%s\s*=([^;]*);" % name, text) for n in re.findall(r"\b(\w+_kernel)\b", v))
        else:
            names.add(name)
    return names


SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
FOUND = [(os.path.basename(path), name) for path in SOURCES if os.path.basename(path) != "common.cuh"
         for name in sorted(launched(open(path).read()))]


@pytest.mark.parametrize("source,name", FOUND)
def test_kernel_waits_for_its_predecessor(source, name):
    body = re.sub(r"//[^\n]*", "", bodies(open(os.path.join(CSRC, source)).read())[name])
    assert "pdl_wait()" in body, f"{name} ({source}) is launched with programmatic serialization and never waits"
