"""Kernel times of a process's first call: a kernel's first launch takes the
host 10 ms and more, which is in no kernel's time."""
from __future__ import annotations

import json
import subprocess
import sys

import pytest

from conftest import PACKAGE, ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import importlib, json, sys
qp = importlib.import_module(sys.argv[1])
n, kind, opts = json.loads(sys.argv[2])
c = qp.Context(0)
c.set_tuning(scatter_kind=kind)
runs = [c.contract_rows(n, **opts) for _ in range(4)]
print(json.dumps([[r.device["scatter_kernel_ms"], r.device["merge_kernel_ms"], r.elapsed,
                   sum(l.elapsed for l in r.layers)] for r in runs]))
"""


@pytest.mark.parametrize("n,kind,opts", [(13, 1, {}), (14, 4, {}), (13, 1, {"key_bits": 128}), (11, 1, {"granularity": 1})])
def test_first_launches_are_in_no_kernel_time(qp, n, kind, opts):
    done = subprocess.run([sys.executable, "-c", SCRIPT, PACKAGE, json.dumps([n, kind, opts])], cwd=ROOT,
                          capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    first, *later = json.loads(done.stdout)
    for i in range(2):
        assert 0 < first[i] <= 3 * max(t[i] for t in later) + 0.5
    # The rows share the call's time.
    for _, _, elapsed, rows in (first, *later):
        assert 0 < rows <= elapsed * 1.001
