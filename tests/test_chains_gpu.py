"""Rows and sites queued as chains sized on the device, the one-CTA form of
small partly placed boards, and the serving batch's chains: exact equality with
the CPU oracle (or with the global-table merge, which runs row by row) where
each can go wrong."""
from __future__ import annotations

import random

import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("row", "input_states", "row_operator_candidates", "row_operator_matched", "completed_row_terms",
          "output_states", "output_weight")
SITE_FIELDS = ("row", "input_states", "completed_row_terms", "output_states", "output_weight")


@pytest.fixture()
def fresh(qp):
    c = qp.Context(0)
    yield c
    c.close()


def _layers(r, fields=FIELDS):
    return [tuple(getattr(l, f) for f in fields) for l in r.layers]


# One CTA: one row left, one and many residues, a full board of N = 9, the
# largest key of 64 bits; and boards beyond its 4096 entries or 6144 terms (5092
# entries; 20111 and 48829 terms), where it gives up and the rows run on the
# device's whole width.
@pytest.mark.parametrize("n,prefix,resident", [
    (5, [1, 3, 0, 2], True), (9, [4], True), (11, [6, 9], True), (14, [10, 6, 3, 0], True),
    (16, [4, 9, 5, 13, 15], False), (18, [9, 11, 6, 16, 1, 17], False),
    (21, [13, 15, 8, 14, 2, 17, 3, 0], False),
    (22, [9, 19, 4, 8, 11, 3, 17, 0, 14, 21, 2, 10], True),
])
def test_one_cta_boards(ctx, oracle, n, prefix, resident):
    count, r = ctx.count_with_stats(n, prefix)
    o = oracle.contract(n, symmetry=False, prefix=prefix)
    assert count == o["count"]
    assert (r.peak_states, r.row_operator_candidates, r.row_operator_matched) == (
        o["peak_states"], o["row_operator_candidates"], o["row_operator_matched"])
    assert (r.device["gpu_launches"] == 1) == resident


# A fill near a partition's capacity overflows some partition in the larger
# rows of a chain: the row fails on the device, the rows after it are skipped,
# and the host goes on from its input.
@pytest.mark.parametrize("key_bits", [64, 128])
@pytest.mark.parametrize("fill", [0.3, 0.95])
@pytest.mark.parametrize("n,symmetry", [(4, 0), (10, 0), (12, 1), (13, 0)])
def test_row_chains_and_their_resumption(fresh, oracle, n, symmetry, fill, key_bits):
    fresh.set_tuning(partition_fill=fill)
    o = oracle.contract(n, symmetry=bool(symmetry))
    want = (o["count"], o["peak_states"], [tuple(l[f] for f in FIELDS) for l in o["layers"]])
    for _ in range(2):
        g = fresh.contract_rows(n, symmetry=symmetry, key_bits=key_bits)
        assert (g.count, g.peak_states, _layers(g)) == want


# Rows beyond the terms a chain may have: at N = 15 the middle rows run by
# themselves and the last ones are a chain again.
@pytest.mark.parametrize("key_bits", [64, 128])
def test_chains_around_large_rows(fresh, qp, key_bits):
    g = fresh.contract_rows(15, key_bits=key_bits)
    t = fresh.contract_rows(15, key_bits=key_bits, merge=qp.MERGE_HASH)
    assert g.count == qp.known_count(15)
    assert _layers(g) == _layers(t)


# Rows of 4 to 64 M terms are a chain of their own; the last one is below that
# again. The prefix's estimate is above (N = 19) and below (N = 17) its boundary.
@pytest.mark.parametrize("n,prefix", [(19, [0, 2, 5]), (17, [8, 2])])
def test_chains_of_large_rows(fresh, qp, n, prefix):
    count, g = fresh.count_with_stats(n, prefix)
    want, t = fresh.count_with_stats(n, prefix, merge=qp.MERGE_HASH)
    assert count == want
    assert (g.peak_states, g.row_operator_candidates, g.row_operator_matched) == (
        t.peak_states, t.row_operator_candidates, t.row_operator_matched)
    assert g.device["gpu_launches"] < t.device["gpu_launches"]


@pytest.mark.parametrize("n", [2, 11, 13, 14])
def test_site_chains(fresh, qp, n):
    s = fresh.contract_rows(n, granularity=qp.GRAIN_SITE)
    r = fresh.contract_rows(n)
    assert s.count == qp.known_count(n)
    assert _layers(s, SITE_FIELDS) == _layers(r, SITE_FIELDS)


# The support limit inside the first chain, at its end and beyond it.
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("limit", [1, 4096, 60000, 1 << 40])
def test_explicit_chains_stop_at_the_limit(fresh, oracle, order, limit):
    g = fresh.explicit_frontier(10, order, limit)
    o = oracle.explicit_frontier(10, order, limit)
    # (A site beyond the limit is counted whole here, up to the limit there.)
    fields = ["count", "complete", "peak_states", "peak_open_bonds", "contracted_sites"]
    fields += ["tensor_entries_examined", "tensor_entries_accepted"] if o["complete"] else []
    assert [g[f] for f in fields] == [o[f] for f in fields]


def test_a_longer_chain_keeps_the_captured_graph(fresh, qp, oracle):
    eager = fresh.contract_rows(8, use_graph=1)
    replay = fresh.contract_rows(8, use_graph=1)
    prefix = [6, 9]
    assert fresh.count(14, prefix) == oracle.contract(14, symmetry=False, prefix=prefix)["count"]
    again = fresh.contract_rows(8, use_graph=1)
    assert replay.device["gpu_launches"] == again.device["gpu_launches"] < eager.device["gpu_launches"]
    assert _layers(eager) == _layers(again)


# Boards of one size end in the same step, others in others; boards with one
# row left and the empty prefix are among them.
def test_served_boards_that_end_together(qp, oracle):
    rng = random.Random(31)
    reqs = [(n, qp.random_prefix(rng, n, k)) for n in (4, 7, 12, 13) for k in (0, 1, n // 2, n - 1) for _ in range(5)]
    rng.shuffle(reqs)
    with qp.Server(0, use_cache=0) as sv:
        got = {}
        for tag, (n, prefix) in enumerate(reqs):
            sv.submit(n, prefix, tag)
        while len(got) < len(reqs):
            done = sv.poll(wait_ms=20000)
            assert done
            got.update((c["tag"], c) for c in done)
    for tag, (n, prefix) in enumerate(reqs):
        want = oracle.contract(n, symmetry=False, prefix=prefix)["count"] if prefix else oracle.known_count(n)
        assert (got[tag]["status"], got[tag]["count"]) == (0, want), (n, prefix)
