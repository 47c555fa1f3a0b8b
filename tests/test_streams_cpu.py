"""Every copy, fill and launch of the library is ordered on a stream of its
own: a context's stream is non-blocking, so work on the legacy default stream
is not ordered with it, stalls every other stream of the process and breaks a
capture of another thread."""
from __future__ import annotations

import re

from conftest import ROOT

SOURCES = sorted((ROOT / "quantum-harness-peps-naive_gb300" / "csrc").glob("*.c*"))


def test_no_work_on_the_default_stream():
    found = []
    for path in SOURCES:
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"\b(cudaMemcpy|cudaMemset|cudaMemcpyToSymbol|cudaMemcpyFromSymbol)\s*\(", text):
            found.append((path.name, m.group(1)))
        for m in re.finditer(r"<<<([^;]*?)>>>", text):
            if m.group(1).count(",") < 3:
                found.append((path.name, m.group(0)))
    assert SOURCES and not found
