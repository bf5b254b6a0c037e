"""Finest level (mra_finest.cu) against the oracle where its work splits change:
finest regions around one 64-observation tile and beyond it (tile-by-tile
factorization, the last tile ragged), sibling groups around the limits of the
grouped path, odd and even knot counts around the conditioning kernel's tile
heights (16, 32, 64), and a tree whose root is the only ancestor.  Tolerances as
in test_gpu_parity: 1e-8 relative on the log-likelihood, 1e-6 on predictions."""
import numpy as np
import pytest

import mra_oracle as oracle
from nonstationary_mra_b200 import api

from test_gpu_parity import LL_RTOL, close_pred, random_case, run_loglik, to_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # seed, J, M, r, n, n_pred, clustered, nu_x2, nonstationary
    (21, 4, 3, 17, 1024, 20, False, 1, True),    # r = 15 (odd); regions of 64 +- 8
    (22, 4, 3, 35, 2070, 20, False, 3, True),    # r = 30; two tiles, the second of a few rows
    (23, 4, 3, 49, 3100, 20, True, 1, True),     # r = 49 (odd); clustered, several tiles beside small regions
    (24, 2, 5, 65, 1500, 20, True, 3, True),     # r = 63 (odd)
    (25, 4, 2, 64, 700, 20, False, 3, True),     # the root is the only ancestor; 175 per region
    (26, 4, 4, 16, 64 * 16, 20, False, 1, True),  # sibling groups of about 64: grouped and per-region items
    (27, 2, 4, 81, 900, 20, True, 1, True),      # r = 81: conditioning through the general products
    (28, 4, 4, 9, 40, 10, True, 1, False),       # fewer observations than regions; stationary
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"s{c[0]}J{c[1]}M{c[2]}r{c[3]}n{c[4]}")
def test_finest_level_vs_oracle(case):
    st, md = random_case(*case)
    ost, omd = to_oracle(st, md)
    _, ll_ref = oracle.loglik(ost, omd)
    m_ref, v_ref = oracle.predict(ost, omd)
    ctx, (d, ll) = run_loglik(st, md)
    assert abs(ll - ll_ref) <= LL_RTOL * abs(ll_ref), (ll, ll_ref)
    m, v = ctx.predict()
    assert close_pred(m, m_ref) and close_pred(v, v_ref)
    ctx.capture_graph()
    assert ctx.loglik()[0] == d       # the forked launches replay in order
    ctx.close()


def test_stats_survive_graph_capture():
    """The event times of an evaluation are read when the statistics are asked for,
    also after a capture (which lists the launches of another evaluation) in between."""
    st, md = random_case(*CASES[0])
    ctx, (d, _) = run_loglik(st, md)
    ctx.capture_graph()
    s = ctx.stats()
    assert s["d"] == d and s["ms_predict"] == 0 and s["ms_prior"] > 0
    assert [l["kernel"] for l in s["launches"]].count("prior_level") == st.M - 1
    ctx.predict()
    assert ctx.stats()["ms_predict"] > 0
    ctx.close()
