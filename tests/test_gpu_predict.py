"""Prediction in chunks (mra_predict.cu) against the oracle at the edges of its split:
regions with up to 12 prediction points (vectors, 4 at a time) and with more (tiles, 64
at a time), regions without observations, factors around one block of 32 rows and
several, odd and even knot counts around the tile heights, a root as the only
ancestor, more points below one region than a chunk holds.  Tolerance as in
test_gpu_parity: 1e-6 on means and variances."""
import numpy as np
import pytest

import mra_oracle as oracle
from nonstationary_mra_b200 import api

from test_gpu_parity import close_pred, random_case, to_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # seed, J, M, r, n, n_pred, clustered, nu_x2, nonstationary
    (31, 4, 2, 16, 130, 20, False, 1, True),     # about 32 observations and 5 points per region
    (32, 4, 2, 35, 500, 36, False, 3, True),     # r = 30; about 9 points: vectors and tiles side by side
    (33, 4, 2, 64, 700, 300, False, 1, True),    # more than 64 points per region
    (34, 2, 5, 49, 600, 400, True, 3, True),     # r = 49 (odd); chunks across sibling groups; empty regions
    (35, 4, 4, 65, 900, 1, True, 1, True),       # r = 63 (odd); a single point
    (36, 4, 3, 9, 30, 200, True, 3, False),      # most regions without observations; stationary
    (37, 2, 7, 17, 3000, 150, True, 1, True),    # r = 15 (odd); factors of several blocks
    (38, 4, 5, 32, 2000, 700, False, 3, True),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"s{c[0]}J{c[1]}M{c[2]}r{c[3]}p{c[5]}")
def test_predict_vs_oracle(case):
    st, md = random_case(*case)
    ost, omd = to_oracle(st, md)
    m_ref, v_ref = oracle.predict(ost, omd)
    ctx = api.Context(st, md)
    ctx.set_theta(sill=md.sill, range_=md.range_, nugget=md.nugget)
    m, v = ctx.predict()
    assert close_pred(m, m_ref) and close_pred(v, v_ref)
    ctx.capture_graph()
    m2, v2 = ctx.predict()
    assert np.array_equal(m, m2) and np.array_equal(v, v2)
    ctx.close()
