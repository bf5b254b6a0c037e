"""Mixed path, finest regions of more than 64 observations (factored over the chip in
16-wide block columns) against the FP64 oracle.  Tolerance: FP32 storage rounds the
conditional covariances to 2^-24 of the marginal ones, which their conditioning (up to
about 1e3 at these sizes) amplifies: 6e-5, taken as 1e-4 relative."""
import numpy as np
import pytest

import mra_oracle as oracle

from test_gpu_parity import random_case, run_loglik, to_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # seed, J, M, r, n, n_pred, clustered, nu_x2, nonstationary
    (41, 4, 2, 16, 4 * 66, 5, False, 1, True),    # regions of 64 +- a few
    (42, 4, 2, 25, 4 * 130, 5, False, 1, True),   # around 128
    (43, 2, 2, 36, 2 * 257, 5, False, 1, True),   # around 256
    (44, 4, 4, 49, 2500, 5, True, 1, True),       # heavy regions beside small ones
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"s{c[0]}J{c[1]}M{c[2]}r{c[3]}n{c[4]}")
def test_mixed_heavy_regions(case):
    st, md = random_case(*case)
    assert np.diff(st.obs_offset).max() > 64
    ost, omd = to_oracle(st, md)
    _, ll_ref = oracle.loglik(ost, omd)
    ctx, (d, ll) = run_loglik(st, md, precision="mixed")
    assert abs(ll - ll_ref) <= 1e-4 * abs(ll_ref), (ll, ll_ref)
    ctx.capture_graph()
    assert ctx.loglik()[0] == d
    ctx.close()
