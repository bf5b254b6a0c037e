"""Posterior levels (mra_posterior.cu) against the oracle: dense regions in tiles
(knot counts at the tile sizes and their remainders, triangular solves beyond
128 knots), dense and factored regions side by side on several levels, every
region dense, and the dense scratch in several chunks.  Tolerances as in
test_gpu_parity: 1e-8 relative on the log-likelihood, 1e-6 on predictions."""
import pytest

import mra_oracle as oracle
from nonstationary_mra_b200 import api

from test_gpu_parity import LL_RTOL, close_pred, random_case, run_loglik, to_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # (seed, J, M, r, n, n_pred, clustered, nu_x2, nonstationary), environment
    ((31, 4, 4, 16, 2500, 20, True, 1, True), {}),                            # r = 16: one small tile
    ((32, 2, 6, 17, 900, 20, True, 3, True), {}),                             # r = 15, odd
    ((33, 4, 4, 36, 2500, 20, False, 3, True), {}),                           # r = 36: one tile of 64 partly filled
    ((34, 4, 4, 33, 1500, 20, True, 1, True), {"MRA_FACTORED_MAX": "0"}),     # r = 30, every region dense
    ((35, 4, 3, 81, 2000, 20, True, 3, True), {"MRA_FACTORED_MAX": "0"}),     # r = 81, odd, two tiles a side
    ((36, 2, 4, 132, 1500, 20, False, 1, True), {"MRA_FACTORED_MAX": "64"}),  # r = 132: triangular solves
    ((37, 4, 5, 64, 9000, 20, False, 1, True), {"MRA_COV_BUF_MB": "1"}),      # scratch of one region at a time
]


@pytest.mark.parametrize("case,env", CASES, ids=lambda c: f"s{c[0]}J{c[1]}M{c[2]}r{c[3]}" if isinstance(c, tuple) else None)
def test_posterior_vs_oracle(case, env, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    st, md = random_case(*case)
    ost, omd = to_oracle(st, md)
    _, ll_ref = oracle.loglik(ost, omd)
    m_ref, v_ref = oracle.predict(ost, omd)
    ctx, (d, ll) = run_loglik(st, md)
    assert abs(ll - ll_ref) <= LL_RTOL * abs(ll_ref), (ll, ll_ref)
    m, v = ctx.predict()
    assert close_pred(m, m_ref) and close_pred(v, v_ref)
    assert ctx.loglik()[0] == d
    ctx.close()
