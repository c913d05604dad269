"""Kernels that may be set up while the kernel before them still runs
(launch_after, programmatic stream serialization) see what earlier kernels have
written only after their wait: nothing that a parameter points to may be
touched before it.  Read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fledge_gb300", "csrc")
SOURCES = {os.path.basename(p): open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu")))}
SCALARS = {"int", "int32_t", "int64_t", "uint32_t", "uint64_t", "float", "bool", "unsigned", "size_t"}


def _matching(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0 and text[i] == pair[1]:
            return i
    raise ValueError("unbalanced")


def _kernels():
    """name -> (parameter list, body) of every __global__ function."""
    out = {}
    for src in SOURCES.values():
        src = re.sub(r"//[^\n]*", "", src)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\([^)]*\)\s*)?(\w+)\s*\(", src):
            end = _matching(src, m.end() - 1, "()")
            at = src.index("{", end)
            if src[end + 1:at].strip():
                continue  # a declaration
            out[m.group(1)] = (src[m.end():end], src[at + 1:_matching(src, at, "{}")])
    return out


KERNELS = _kernels()
WAITING = sorted(k for k, (_, body) in KERNELS.items() if "after_wait()" in body)


def test_every_chained_kernel_waits():
    named = set()
    for src in SOURCES.values():
        for m in re.finditer(r"launch_after\(", src):
            named |= set(re.findall(r"\bk_\w+", src[m.end():_matching(src, m.end() - 1, "()")]))
        for m in re.finditer(r"\b(?:kern|shade|shadow)\s*=[^;]*;", src):  # kernels picked by a variable
            named |= set(re.findall(r"\bk_\w+", m.group(0)))
    assert len(named) > 15 and named <= set(KERNELS)
    assert named <= set(WAITING), named - set(WAITING)


@pytest.mark.parametrize("name", WAITING)
def test_nothing_in_memory_is_touched_before_the_wait(name):
    params, body = KERNELS[name]
    before = body[:body.index("after_wait()")]
    assert before.count("{") == before.count("}"), "the wait is conditional"
    for p in params.split(","):
        words = re.findall(r"\w+", p)
        if "*" not in p and SCALARS & set(words[:-1]):
            continue
        assert not re.search(r"\b%s\b" % words[-1], before), (words[-1], before)
    assert "launch_dependents" not in body
