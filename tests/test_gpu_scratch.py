"""The posterior's scratch, shared by the dense and the factored regions of a level: the
mixed path with a short limit for factored regions and few regions per level, where a
dense region needs more than half of the buffer.  Tolerance as in test_gpu_mixed_heavy."""
import numpy as np
import pytest

import mra_oracle as oracle
from nonstationary_mra_b200 import partition, synth

from test_gpu_parity import random_case, run_loglik, to_oracle

pytestmark = pytest.mark.gpu


def quadrant_case(seed, J, M, r, per_quadrant):
    """per_quadrant points in each quarter of the unit square."""
    rng = np.random.default_rng(seed)
    xy = np.concatenate([0.5 * rng.random((2, n)) * 0.96 + 0.01 + np.array([[0.5 * (q & 1)], [0.5 * (q >> 1)]])
                         for q, n in enumerate(per_quadrant)], axis=1)
    n = xy.shape[1]
    st = partition.build_by_program(xy[0], xy[1], rng.standard_normal(n), J, M, r, np.exp(1) / 100, None, None,
                                    distance=2)
    theta = synth.true_theta(synth.Config("t", n, M, J, r, 1, 0, "uniform", 0.3), rng)
    return st, synth.model_from_theta(theta, 1)


@pytest.mark.parametrize("J,M,limit,per_quadrant", [
    (4, 3, 30, (70, 25, 20, 10)),     # one dense region beside three factored ones
    (4, 3, 15, (40, 12, 11, 10)),
    (2, 4, 80, (200, 60, 50, 40)),
    (2, 4, 16, (60, 14, 13, 12)),
])
def test_dense_region_needs_most_of_the_scratch(J, M, limit, per_quadrant, monkeypatch):
    r = 64
    st, md = quadrant_case(5, J, M, r, per_quadrant)
    assert st.r == r
    ost, omd = to_oracle(st, md)
    _, ll_ref = oracle.loglik(ost, omd)
    monkeypatch.setenv("MRA_FACTORED_MAX", str(limit))
    ctx, (d, ll) = run_loglik(st, md, precision="mixed")
    assert abs(ll - ll_ref) <= 1e-4 * abs(ll_ref), (ll, ll_ref)
    ctx.capture_graph()
    assert ctx.loglik()[0] == d
    ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_levels_in_chunks(precision, monkeypatch):
    """A covariance buffer of about a third of what the deepest level asks for (the least that a
    context takes is one region per resident CTA): its prior regions, and its dense and its
    factored posterior regions, which share the buffer, run in chunks.  A region's steps do not
    depend on the chunk, so the results are bitwise the same."""
    J, M, r = 4, 7, 16
    st, md = random_case(50, J, M, r, 33000, 2000, False, 1, True)   # about 2 r observations per level M-2 region
    parent = np.asarray(st.finest_parent)
    per_region = np.bincount(parent - parent.min(), weights=np.diff(st.obs_offset))
    assert (per_region > 2 * r).sum() > 200 and (per_region <= 2 * r).sum() > 200
    out = []
    for mb in (None, "1"):
        if mb:
            monkeypatch.setenv("MRA_COV_BUF_MB", mb)
        ctx, (d, _) = run_loglik(st, md, precision=precision)
        launches = [ctx.stats()["kernel_launches"]]
        mean, var = ctx.predict()
        launches.append(ctx.stats()["kernel_launches"])
        out.append((d, mean, var, launches))
        ctx.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
    # the prior's level in four chunks and the posterior's kinds of region in two at least
    assert all(b >= a + 6 + 4 for a, b in zip(out[0][3], out[1][3])), (out[0][3], out[1][3])
