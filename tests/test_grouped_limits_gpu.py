"""Column-grouped rows beyond their limits: a weight that may pass its word, or
a unit with more segments than its list holds, hands the whole batch to the
partitioned rows, with nothing counted twice. No board of up to 18 columns
passes either limit, so the library is linked once more with the limits set
lower."""
from __future__ import annotations

import importlib
import json
import subprocess
import sys

import pytest

from conftest import PACKAGE, ROOT

pytestmark = pytest.mark.gpu

CALLS = [(15, [], {}), (15, [], {"symmetry": 0}), (16, [7], {}), (15, [], {"device_budget_bytes": 700 << 20})]

SCRIPT = """
import importlib, json, pathlib, sys
qp = importlib.import_module(sys.argv[1])
if sys.argv[2]:
    qp.LIBRARY_PATH = pathlib.Path(sys.argv[2])
out = []
for n, prefix, opts in json.loads(sys.argv[3]):
    c = qp.Context(0)
    c.set_tuning(slice_margin=1.0)
    count, r = c.count_with_stats(n, prefix, **opts) if prefix else (None, c.contract_rows(n, **opts))
    c.close()
    sliced = r.device["batches"] > 1
    rows = [(l.row, l.output_weight) + (() if sliced else (l.input_states, l.row_operator_matched, l.output_states))
            for l in r.layers]
    out.append([r.count, r.device["row_forms"], r.device["batches"], rows,
                None if sliced else [r.peak_states, r.device["candidates"], r.device["entries_in"]]])
print(json.dumps(out))
"""


def _run(library=""):
    done = subprocess.run([sys.executable, "-c", SCRIPT, PACKAGE, str(library), json.dumps(CALLS)], cwd=ROOT,
                          capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    return json.loads(done.stdout)


@pytest.fixture(scope="module")
def normal(qp):
    runs = _run()
    assert all(r[1] == qp.ROWS_GROUPED for r in runs) and runs[-1][2] > 1
    return runs


# Passed in the first rows, behind the largest ones (weights of 20 and more), and
# by long lists only.
@pytest.mark.parametrize("limit", ["WEIGHT_BITS=6", "WEIGHT_BITS=10", "MAX_SEG=24"])
def test_a_batch_beyond_a_limit_is_handed_back(qp, normal, tmp_path, limit):
    build = importlib.import_module(PACKAGE + ".buildlib")
    obj, lib = tmp_path / "group.o", tmp_path / "libqpeps.so"
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, f"-DQPEPS_GROUP_{limit}", "-c",
                    str(build.CSRC / "qpeps_group_kernels.cu"), "-o", str(obj)], check=True)
    others = [str(build.OBJ / (s[:-3] + ".o")) for s in build.LIB_SOURCES if s != "qpeps_group_kernels.cu"]
    subprocess.run([build.nvcc(), *build.ARCH, "-shared", "-o", str(lib), *others, str(obj)], check=True)
    for got, want in zip(_run(lib), normal):
        assert got[1] & qp.ROWS_GROUPED == 0 and got[1] != 0
        assert [got[0]] + got[2:] == [want[0]] + want[2:]
