"""Bounded waits of the device-driven rounds (2) and of staged rounds (3) that run
out: OG_E_TIMEOUT, nothing written by the step that gave up, a GPU that stays
usable, and queries that are right afterwards."""
import numpy as np
import pytest

import onegraph_gb300 as og
import oracle

from test_gpu_engine import budget_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [2, 3])
@pytest.mark.parametrize("limit", [1, 300, 5000])
def test_wait_gives_up(which, limit):
    assert og.lib().og_k_wait_check(which, limit) == 6, og.lib().og_last_error()  # OG_E_TIMEOUT
    assert b"gave up" in og.lib().og_last_error()
    g = og.Graph.rmat(9, 8)
    off, col = np.array(g.offsets), np.array(g.columns)
    for kw in ({}, dict(budget=budget_for(g, 3 * 2048), advisek=0.05)):
        e = og.Engine(g, **kw)
        np.testing.assert_array_equal(oracle.normalise_bfs(e.bfs(3), g.V), oracle.bfs(off, col, 3)[0])
        e.close()


def test_unknown_check_is_refused():
    assert og.lib().og_k_wait_check(4, 10) == 1 and og.lib().og_k_wait_check(-1, 10) == 1  # OG_E_ARG
