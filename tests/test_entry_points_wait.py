"""Every entry point of the C ABI that puts kernels or copies of the caller's data
on the handle's stream is done with them when it returns, so that its status is
that of its own work (no GPU: read from the source).  The control block, which
the library copies from memory of its own, may follow in stream order."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = os.path.join(ROOT, "anuga-cuda_gb300", "csrc", "swgpu_api.cu")

WORK = re.compile(r"\b(launch_\w+|issue_\w+|refresh_edges|cudaMemcpyAsync)\(")
WAIT = re.compile(r"\b(cudaStreamSynchronize|sync_ctrl|finish|finish_run|run_graphs|upload|"
                  r"download)\(")


def entry_points():
    text = open(SOURCE).read()
    text = text[text.index('extern "C" {'):]
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for m in re.finditer(r"^int (swgpu_\w+)\([^;{]*\) \{\n(.*?)^\}", text, re.M | re.S):
        out[m.group(1)] = m.group(2)
    return out


def test_work_is_waited_for():
    found = entry_points()
    working = [n for n, body in found.items() if WORK.search(body)]
    assert len(found) >= 30 and len(working) >= 15
    late = []
    for name in working:
        body = found[name]
        last_work = max(m.start() for m in WORK.finditer(body))
        if not any(m.start() > last_work for m in WAIT.finditer(body)):
            late.append(name)
    assert not late, late
