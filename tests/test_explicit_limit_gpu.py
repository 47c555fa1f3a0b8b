"""The explicit-C frontier's support limit stops the work itself: no chain of
site steps is queued far past the site over the limit, and no more memory is
taken than boundaries within the limit need."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("count", "complete", "peak_states", "peak_open_bonds", "contracted_sites")
CHAIN = 16  # site steps a chain that may stop has at most (two at a limit of one)


# Limits passed by the first sites, inside a later chain and at the default of
# the interface; one that the whole board stays below.
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("n,limit", [(20, 1), (20, 2), (14, 500), (14, 5000), (13, 100000), (11, 1 << 40), (11, 2**64 - 1)])
def test_work_and_memory_end_at_the_limit(qp, oracle, n, order, limit):
    c = qp.Context(0)
    try:
        g = c.explicit_frontier(n, order, limit)
    finally:
        c.close()
    o = oracle.explicit_frontier(n, order, limit)
    assert [g[f] for f in FIELDS] == [o[f] for f in FIELDS]
    assert g["gpu_launches"] <= 2 * (g["contracted_sites"] + (2 if limit == 1 else 1 + CHAIN)) + 1
    if not g["complete"]:
        # A boundary (three times its need), its partitions at two CTAs an SM
        # with 64 candidates each, cursors, scalars and the step list.
        assert g["peak_rss_bytes"] <= (24 << 20) + 512 * limit
