"""CPU check of the kernels that may be resident while the kernel before them still runs (launch_chained): each of them waits for it, and loads what it
wrote with ordinary loads, never with those for data that is constant while the grid runs (__ldg, pointers marked const __restrict__)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "onemodel-csharp_b200", "csrc")
SOURCES = {os.path.basename(f): re.sub(r"//.*", "", open(f).read()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def kernels(text):
    """(name, head and body) of every kernel."""
    for m in re.finditer(r"__global__ void(?P<head>[^;{]*?)\{", text, re.S):
        body = text[m.end():text.index("\n}\n", m.end())]
        names = re.findall(r"(\w+)\s*\(", re.sub(r"__\w+__\((?:[^()]|\([^()]*\))*\)", "", m["head"]))
        yield names[0], m["head"] + body


@pytest.mark.parametrize("name", [n for n in SOURCES if n.endswith(".cu")])
def test_chained_kernels_wait_and_load_plainly(name):
    text = SOURCES[name]
    found = dict(kernels(text))
    for k in set(re.findall(r"launch_chained\(ctx,\s*(\w+_kernel)\b", text)):
        assert re.search(r"\bpdl_(enter|wait)\(\)", found[k]), k
    for k, source in found.items():
        if re.search(r"\bpdl_(enter|wait)\(\)", source):
            assert "__ldg(" not in source, k
            assert not re.search(r"const \w+\s*\*\s*__restrict__", source), k


def test_helpers_of_chained_kernels_load_plainly():
    """Device functions that such kernels call: every source with a chained launch, but for the kernels in it that do not wait."""
    for name, text in SOURCES.items():
        if "launch_chained(" not in text and name != "om_tc.cuh" or name == "om_common.cuh":
            continue
        rest = text
        for k, source in kernels(text):
            rest = rest.replace(source[source.index("("):], "")
        for m in re.finditer(r"__device__ [^;{]*\{", rest, re.S):
            body = m[0] + rest[m.end():rest.find("\n}\n", m.end())]
            assert "__ldg(" not in body and not re.search(r"const \w+\s*\*\s*__restrict__", m[0]), (name, m[0])
