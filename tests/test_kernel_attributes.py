"""Kernel attributes (the opt-in to more than 48 KB of shared memory) belong to a device, and a process may use
several: no result of cudaFuncSetAttribute is kept in a static, which would set it on the first caller's device
only. Read from the sources, since it takes a second GPU to see the refused launch."""

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "holovibes_gb300" / "csrc"


def test_attributes_are_set_at_every_launch():
    calls = 0
    for src in sorted(CSRC.glob("*.c*")) + sorted(CSRC.glob("*.h")):
        text = re.sub(r"//[^\n]*", "", src.read_text())
        calls += len(re.findall(r"\bcudaFuncSetAttribute\s*\(", text))
        for m in re.finditer(r"\b(?:static|thread_local)\b[^;{}]*=([^;]*);", text):
            assert "cudaFuncSetAttribute" not in m.group(1), (src.name, m.group(0))
    assert calls >= 10
