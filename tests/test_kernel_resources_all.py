"""Registers and spills of the step kernels that test_kernel_resources.py does not
name or reads from the wrong line, from ptxas's resource report (no GPU): those
of small and middle meshes (the `late` forms, the update with boundary tags, the
resident step), the FP64 kernels, and the distributes.

A kernel's own figures are on the first properties line after its entry; the
lines after those are of functions that it calls."""
import os
import re
import shutil
import subprocess

import pytest

from anuga_cuda import _build as B

ENTRY = re.compile(r"Compiling entry function '_ZN5swgpu(\d+)(\w+)'")
SPILL = re.compile(r"(\d+) bytes spill stores, (\d+) bytes spill loads")
USED = re.compile(r"Used (\d+) registers")

# (kernel, template arguments): registers, bytes of spill stores and loads per thread.
# The registers follow from the launch bounds; the spills are what the build
# had when the kernels were measured.
BUDGET = {
    "swgpu_mixed.cu": {
        ("flux_mixed", None): (40, 0, 0), ("flux_late", None): (40, 0, 0),
        ("update_mixed", None): (32, 0, 0), ("update_late", None): (32, 8, 8),
        ("update_with_tags", "Lb0ELb0"): (32, 4, 4), ("update_with_tags", "Lb1ELb0"): (32, 4, 4),
        ("update_with_tags", "Lb0ELb1"): (32, 24, 16),
        ("update_with_tags", "Lb1ELb1"): (32, 16, 8),
        ("distribute_mixed", None): (32, 48, 32), ("distribute_late", None): (32, 60, 44),
        ("steps_resident", "Li128"): (126, 0, 0), ("steps_resident", "Li256"): (126, 0, 0),
        ("steps_resident", "Li512"): (96, 60, 52), ("step_clock_mixed", None): (32, 0, 0),
    },
    "swgpu_fp64.cu": {
        ("flux_fp64", "Li1"): (104, 0, 0), ("flux_fp64", "Li3"): (80, 96, 48),
        ("update_fp64", None): (64, 0, 0),
        ("distribute_fp64", "Li2"): (128, 20, 20), ("distribute_fp64", "Li3"): (80, 232, 256),
        ("distribute_de_fp64", "Li2"): (128, 0, 0),
        ("distribute_de_fp64", "Li3"): (80, 68, 84),
        ("distribute_split_fp64", None): (96, 0, 0),
        ("distribute_de_split_fp64", None): (64, 0, 0),
    },
}


def _report(tmp_path, unit):
    if not (shutil.which("nvcc") or os.path.exists("/usr/local/cuda/bin/nvcc")):
        pytest.skip("nvcc not available")
    cmd = [B._nvcc()] + B.COMMON + B.UNITS[unit] + [
        "-Xptxas", "-v", "-c", os.path.join(B.CSRC, unit), "-o", str(tmp_path / "unit.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out, cur = {}, None
    for line in r.stderr.splitlines():
        m = ENTRY.search(line)
        if m:
            n = int(m.group(1))
            name, rest = m.group(2)[:n], m.group(2)[n:]
            args = rest[1:rest.index("EEEv")] if rest.startswith("I") else ""
            cur = out[(name, args)] = {}
            continue
        m = SPILL.search(line)
        if m and cur is not None and "spill" not in cur:
            cur["spill"] = (int(m.group(1)), int(m.group(2)))
        m = USED.search(line)
        if m and cur is not None and "regs" not in cur:
            cur["regs"] = int(m.group(1))
    return out


@pytest.mark.parametrize("unit", BUDGET)
def test_step_kernels_within_budget(unit, tmp_path):
    rep = _report(tmp_path, unit)
    for (kernel, ending), (regs, stores, loads) in BUDGET[unit].items():
        mine = {k: v for k, v in rep.items()
                if k[0] == kernel and (ending is None or k[1].endswith(ending))}
        assert mine, (kernel, ending)
        for k, v in mine.items():
            assert v["regs"] <= regs, (k, v)
            assert v["spill"][0] <= stores and v["spill"][1] <= loads, (k, v)
