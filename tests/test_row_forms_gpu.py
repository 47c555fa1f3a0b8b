"""Which form the rows of a call ran in, as the result reports it."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def fresh(qp):
    c = qp.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n,opts,forms", [
    (1, {}, ""), (4, {}, "CHAIN"), (8, {"merge": 1}, "SINGLE"), (9, {"granularity": 1}, "CHAIN"),
    (14, {}, "CHAIN"), (14, {"symmetry": 0}, "GROUPED"), (14, {"granularity": 1}, "CHAIN SINGLE"),
    (15, {}, "GROUPED"), (15, {"key_bits": 128}, "CHAIN"), (16, {"use_graph": 1}, "CHAIN SINGLE"),
])
def test_boards(fresh, qp, n, opts, forms):
    r = fresh.contract_rows(n, **opts)
    assert r.count == qp.known_count(n)
    assert r.device["row_forms"] == sum(getattr(qp, f"ROWS_{f}") for f in forms.split())


@pytest.mark.parametrize("n,prefix,forms", [
    (14, [10, 6, 3, 0], "ONE_CTA"), (16, [4, 9, 5, 13, 15], "CHAIN"), (16, [7], "GROUPED"), (8, [0, 1], ""),
])
def test_partly_placed_boards(fresh, qp, n, prefix, forms):
    assert fresh.count_with_stats(n, prefix)[1].device["row_forms"] == sum(
        getattr(qp, f"ROWS_{f}") for f in forms.split())


def test_a_replay_is_reported(fresh, qp):
    seen = [fresh.contract_rows(11, use_graph=1).device["row_forms"] for _ in range(3)]
    assert seen == [qp.ROWS_CHAIN, qp.ROWS_REPLAY, qp.ROWS_REPLAY]


# A prefix whose boundary passes its estimate: a row of the chain does not fit,
# and another chain goes on from its input (two kernels more than the rows take).
def test_an_ended_chain_goes_on(fresh, qp):
    prefix = [8, 2]
    count, r = fresh.count_with_stats(17, prefix)
    assert count == fresh.count(17, prefix, merge=qp.MERGE_HASH)
    assert r.device["row_forms"] == qp.ROWS_CHAIN
    assert r.device["gpu_launches"] > 1 + 2 * (17 - len(prefix))


# Bytes are counted in the form's own entry size: key and weight in 32 bits
# each, or a 64-bit key and a weight's two words.
@pytest.mark.parametrize("kind,entry", [("WINDOW", 8), ("DIRECT", 16)])
def test_bytes_are_the_entries_read_and_written(fresh, qp, kind, entry):
    fresh.set_tuning(scatter_kind=getattr(qp, f"SCATTER_{kind}"))
    d = fresh.contract_rows(15).device
    assert d["merge_kernel_bytes"] == entry * (d["entries_in"] + d["entries_out"])


# What use_graph does not capture (column-grouped and one-CTA rows) is compared
# row by row with the recorded run; another call's record is not taken for it.
def test_uncaptured_runs_are_compared(fresh, qp):
    one, other = [10, 6, 3, 0], [10, 6, 3, 1]
    boards = [(17, None), (14, one), (14, other)]
    for n, prefix in boards:
        form = qp.ROWS_ONE_CTA if prefix else qp.ROWS_GROUPED
        runs = [fresh.count_with_stats(n, prefix, use_graph=1)[1] if prefix else fresh.contract_rows(n, use_graph=1)
                for _ in range(3)]
        assert [r.device["row_forms"] for r in runs] == [form] + 2 * [form | qp.ROWS_CHECKED]
        assert runs[0].count == runs[1].count == runs[2].count
    assert fresh.contract_rows(17).device["row_forms"] == qp.ROWS_GROUPED


# The autotuner's picks leave the forms that other calls run in: none of those
# that it may turn off is slower than what replaces it at these sizes.
@pytest.mark.parametrize("n", [11, 11, 11, 13, 14, 15])
def test_autotuned_calls_keep_their_form(fresh, qp, n):
    form = fresh.contract_rows(n).device["row_forms"]
    fresh.autotune(n, repeats=2)
    r = fresh.contract_rows(n)
    assert r.count == qp.known_count(n)
    assert r.device["row_forms"] == form
