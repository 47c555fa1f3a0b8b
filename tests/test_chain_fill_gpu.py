"""A partition fill near the capacity, meant for rows that run by themselves,
does not end the chains of queued steps: the launches are those of a low fill,
in the first call and in the next."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _launches(qp, fill, call):
    c = qp.Context(0)
    try:
        c.set_tuning(partition_fill=fill)
        return [call(c) for _ in range(2)]
    finally:
        c.close()


@pytest.mark.parametrize("fill", [0.9, 0.95])
@pytest.mark.parametrize("n,opts", [(13, {}), (13, {"symmetry": 0}), (14, {}), (13, {"key_bits": 128}),
                                    (13, {"key_bits": 128, "symmetry": 0})])
def test_high_fills_keep_row_chains(qp, n, opts, fill):
    def call(c):
        r = c.contract_rows(n, **opts)
        assert r.count == qp.known_count(n)
        return r.device["gpu_launches"]

    assert _launches(qp, fill, call) == _launches(qp, 0.5, call)


@pytest.mark.parametrize("order", [0, 1])
def test_high_fills_keep_site_chains(qp, order):
    def call(c):
        g = c.explicit_frontier(11, order)
        assert g["count"] == qp.known_count(11)
        return g["gpu_launches"]

    assert _launches(qp, 0.95, call) == _launches(qp, 0.5, call)
