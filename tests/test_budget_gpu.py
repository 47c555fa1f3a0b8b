"""Calls with a device budget on a context that keeps larger buffers of an
earlier call: equal results, and no more memory held than the budget."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("row", "input_states", "row_operator_candidates", "row_operator_matched", "completed_row_terms",
          "output_states", "output_weight")


@pytest.fixture()
def fresh(qp):
    c = qp.Context(0)
    yield c
    c.close()


def _layers(r):
    return [tuple(getattr(l, f) for f in FIELDS) for l in r.layers]


def _held(r):
    return r.layers[-1].peak_rss_bytes


# A kept boundary buffer (540 MiB, of N = 15 row by row) that the budget holds
# but not beside a row's scratch: the live boundary moves into a smaller one
# through the host, which the bytes copied show. The call after it finds the
# context as any other.
@pytest.mark.parametrize("budget", [541, 544])
def test_a_kept_boundary_gives_way(fresh, qp, budget):
    c = qp.Context(0)
    try:
        c.set_tuning(scatter_kind=qp.SCATTER_DIRECT)
        c.contract_rows(15)
        for again in (False, True):
            g = c.contract_rows(14, symmetry=0, device_budget_bytes=budget << 20)
            assert _layers(g) == _layers(fresh.contract_rows(14, symmetry=0))
            assert _held(g) <= budget << 20
            if not again:
                assert min(g.device["h2d_bytes"], g.device["d2h_bytes"]) > 1 << 20
        assert _layers(c.contract_rows(13)) == _layers(fresh.contract_rows(13))
    finally:
        c.close()


# Budgets that hold neither form's buffers of the whole board, or the grouped
# rows but not beside what the context already keeps.
@pytest.mark.parametrize("budget", [1 << 30, 3 << 30])
def test_held_memory_stays_within_the_budget(fresh, qp, budget):
    fresh.contract_rows(16)
    g = fresh.contract_rows(16, device_budget_bytes=budget)
    assert g.count == qp.known_count(16)
    assert _held(g) <= budget


# Budgets that hold a chain's boundary and its scratch, at a quarter more than
# the scratch needs, but not the few KB of its scalars beside them (on 152 SMs).
@pytest.mark.parametrize("n,budget,opts", [
    (11, 40517584, {}), (13, 45581584, {}), (11, 75892560, {"key_bits": 128}),
    (12, 26845824, {"granularity": 1}), (12, 33565824, {"granularity": 1}),
])
def test_chain_scalars_fit_a_tight_budget(fresh, qp, n, budget, opts):
    g = fresh.contract_rows(n, device_budget_bytes=budget, **opts)
    assert g.count == qp.known_count(n)
    assert _held(g) <= budget


# What earlier calls left goes where it exceeds the budget, also before a call
# that needs no device memory of its own (a board in one CTA). Freed memory is
# seen by the device: 11 GB of column-grouped rows.
@pytest.mark.parametrize("call", [
    lambda c, b: c.count(14, [10, 6, 3, 0], device_budget_bytes=b),
    lambda c, b: c.contract_rows(8, device_budget_bytes=b),
    lambda c, b: (c.contract_rows(8), c.contract_rows(8, device_budget_bytes=b)),
    lambda c, b: c.contract_rows(8, granularity=1, device_budget_bytes=b),
])
def test_kept_buffers_beyond_the_budget_go(fresh, qp, call):
    torch = pytest.importorskip("torch")
    before = torch.cuda.mem_get_info()[0]
    fresh.contract_rows(17)
    kept = before - torch.cuda.mem_get_info()[0]
    call(fresh, 64 << 20)
    assert kept > 8 << 30
    assert before - torch.cuda.mem_get_info()[0] < 1 << 30


# What a context keeps of other calls (chain scalars, site steps, the slice
# tail's lists) takes nothing from a tight budget: calls that fit a fresh
# context fit after any of them.
@pytest.mark.parametrize("prep", [
    lambda c: c.contract_rows(12), lambda c: c.contract_rows(9, granularity=1), lambda c: c.explicit_frontier(10, 1),
    lambda c: c.contract_rows(12, tail_row=9), lambda c: c.contract_rows(15),
], ids=["chain", "sites", "explicit", "tail", "grouped"])
@pytest.mark.parametrize("n,opts,budgets", [
    (11, {"granularity": 1, "symmetry": 0}, range(409600, 1740800, 56789)),
    (10, {"granularity": 1}, range(204800, 921600, 40961)),
    (12, {}, range(307200, 2560000, 98765)), (11, {"merge": 1}, range(307200, 2560000, 98765)),
    (11, {"key_bits": 128}, range(307200, 2560000, 98765)),
])
def test_kept_buffers_take_nothing_from_a_budget(qp, prep, n, opts, budgets):
    for budget in budgets:
        c = qp.Context(0)
        try:
            prep(c)
            assert c.contract_rows(n, device_budget_bytes=budget, **opts).count == qp.known_count(n)
        finally:
            c.close()


# A boundary kept from a smaller board, which the budget does not hold beside a
# larger one: the chains of a board in slices find room or leave the rows'
# buffers alone (freed and reserved again for every row, they took twice the
# time).
@pytest.mark.parametrize("budget", [119383412, 130862880])
def test_chains_under_a_kept_boundary(fresh, qp, budget):
    fresh.count(13, [1], device_budget_bytes=budget)
    g = fresh.contract_rows(15, device_budget_bytes=budget)
    assert g.count == qp.known_count(15) and g.device["batches"] > 1
    assert g.device["row_forms"] & qp.ROWS_CHAIN
    assert _held(g) <= budget
