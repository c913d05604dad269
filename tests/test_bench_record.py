"""The traversal's profile that the benchmark reads counts as current only while
the sources that decide the kernel's traffic are the ones it was taken on: the
kernel, every header it includes, and the collapse that lays out its nodes."""
import json
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = "fledge_gb300/csrc/"


def test_profile_covers_the_sources_of_the_traversal():
    import bench
    need = {CSRC + "trace.cu", CSRC + "collapse.cu"}
    todo = ["trace.cu"]
    while todo:
        for h in re.findall(r'#include "(\w+\.cuh?|internal\.h)"', open(os.path.join(ROOT, CSRC, todo.pop())).read()):
            if CSRC + h not in need:
                need.add(CSRC + h)
                todo.append(h)
    assert need <= set(bench.TRACE_SOURCES), need - set(bench.TRACE_SOURCES)
    rec = json.load(open(bench.TRACE_PROFILE))
    assert rec["source_files"] == bench.TRACE_SOURCES
    assert re.fullmatch("[0-9a-f]{16}", rec["source_sha16"])
