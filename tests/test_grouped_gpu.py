"""Column-grouped rows (large boundaries, up to N = 18) against
the partitioned rows, which run with the direct scatter: every row's metrics,
the peak and the count are equal."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("row", "input_states", "row_operator_candidates", "row_operator_matched", "completed_row_terms",
          "output_states", "output_weight")


@pytest.fixture(scope="module")
def pair(qp):
    grouped, partitioned = qp.Context(0), qp.Context(0)
    partitioned.set_tuning(scatter_kind=qp.SCATTER_DIRECT)
    yield grouped, partitioned
    grouped.close()
    partitioned.close()


def _same(g, p):
    # Another route each: grouped rows report their plan kernels as the scatter.
    assert g.device["scatter_kernel_ms"] < 0.3 * g.device["merge_kernel_ms"]
    assert p.device["scatter_kernel_ms"] > 0.5 * p.device["merge_kernel_ms"]
    assert (g.count, g.peak_states, g.row_operator_candidates, g.row_operator_matched) == (
        p.count, p.peak_states, p.row_operator_candidates, p.row_operator_matched)
    assert [tuple(getattr(l, f) for f in FIELDS) for l in g.layers] == [
        tuple(getattr(l, f) for f in FIELDS) for l in p.layers]


# Orbits and none, one residue (12 free rows and fewer) and exact words, the
# bits that N = 18 leaves to the bucket, uneven prefixes.
@pytest.mark.parametrize("n,prefix,symmetry", [
    (15, [], 1), (15, [], 0), (16, [], 1), (16, [7], 1), (17, [8], 1), (17, [0], 1), (18, [8], 1), (18, [0], 1), (14, [], 0),
])
def test_grouped_rows_equal_partitioned_rows(pair, qp, n, prefix, symmetry):
    if prefix:
        (gc, g), (pc, p) = (c.count_with_stats(n, prefix) for c in pair)
        assert gc == pc
    else:
        g, p = (c.contract_rows(n, symmetry=symmetry) for c in pair)
        assert g.count == qp.known_count(n)
    _same(g, p)


# Slices whose average is far below the largest one: its rows outgrow their
# buffer and run again from there, in a larger one.
def test_a_row_beyond_its_buffer_runs_again(qp):
    results = []
    for kind in (qp.SCATTER_WINDOW, qp.SCATTER_DIRECT):
        c = qp.Context(0)
        c.set_tuning(scatter_kind=kind, slice_margin=1.0)
        results.append(c.contract_rows(17, device_budget_bytes=12 << 30))
        c.close()
    assert results[0].device["batches"] > 1 and results[0].count == qp.known_count(17)
    _same(*results)


# A budget that holds neither form's buffers of the whole board, and one that
# holds the grouped rows but not beside what the context already keeps.
@pytest.mark.parametrize("budget", [1 << 30, 3 << 30])
def test_grouped_rows_within_a_budget(pair, qp, budget):
    g = pair[0].contract_rows(16, device_budget_bytes=budget)
    assert g.count == qp.known_count(16)
    assert g.device["peak_device_bytes"] >= 0
    again = pair[0].contract_rows(14)
    assert again.count == qp.known_count(14)
