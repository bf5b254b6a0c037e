"""Covariance blocks (the straight-line forms and the general one, tiles, parameters
passed by value or copied) against the oracle.

Tolerance: a block entry is a square root, a power, a division and an exponential of
an argument of at most 60 here, each of a few units in the last place; the argument's
relative error is multiplied by the argument: 60 * 8 * 1.1e-16 < 1e-13.  1e-12 is
what the library's other covariance tests ask for."""
import ctypes as C
import itertools

import numpy as np
import pytest

import mra_oracle as oracle
from nonstationary_mra_b200 import api, capi
from nonstationary_mra_b200.model import Field, Model

pytestmark = pytest.mark.gpu

RTOL = 1e-12
CHORDAL, GREAT_CIRCLE, PLANAR = 0, 1, 2


def model(rng, distance, nu_x2, pref, nb=5, nonstat=True):
    """nb basis functions per field around the points of `points`."""
    fields = [Field(0.2 * rng.standard_normal(), points(rng, distance, nb), 0.5 * rng.standard_normal(nb))
              for _ in range(3)]
    fields[1].intercept -= 1.0
    return Model(nonstationary=nonstat, distance=distance, nu_x2=nu_x2, prefactor_exp=pref, dist_scale=1.0,
                 basis_len=0.4, fields=fields, sill=1.3, range_=0.2, nugget=0.07)


def points(rng, distance, n):
    p = rng.random((3, n)) * 0.5
    if distance == GREAT_CIRCLE:   # degrees; no pair so close that the arc cosine loses digits
        p = p * [[720.0], [240.0], [0.0]] - [[180.0], [60.0], [0.0]]
    elif distance == PLANAR:
        p[2] = 0.0
    else:
        p[2] += 0.3
        p /= np.linalg.norm(p, axis=0)
    return p


def expected(md, p1, p2=None):
    omd = oracle.Model(nonstationary=md.nonstationary, distance=md.distance, nu_x2=md.nu_x2,
                       prefactor_exp=md.prefactor_exp, dist_scale=md.dist_scale, basis=md.basis, basis_len=md.basis_len,
                       fields=[oracle.Field(f.intercept, f.centers, f.weights) for f in md.fields],
                       sill=md.sill, range_=md.range_, nugget=md.nugget)
    f1 = oracle.field_values(omd, p1)
    return oracle.var_cov(omd, p1, f1) if p2 is None else oracle.cross_cov(omd, p1, f1, p2, oracle.field_values(omd, p2))


THETA = dict(sill_scale=1.0, range_scale=1.0, nugget_scale=1.0)


def static_block(md, p1, p2, sill_scale=1.0):
    import torch
    m, keep = api._model_struct(md)
    th = capi.mra_theta()
    th.sill, th.range, th.nugget = md.sill, md.range_, md.nugget
    th.range_scale = th.nugget_scale = 1.0
    th.sill_scale = sill_scale
    d1, d2 = (torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in (p1, p2))
    out = torch.full((p1.shape[1], p2.shape[1]), -1.0, dtype=torch.float64, device="cuda")
    capi.check(capi.load().mra_eval_covariance_static(
        C.byref(m), C.byref(th), C.c_void_p(d1.data_ptr()), p1.shape[1], C.c_void_p(d2.data_ptr()), p2.shape[1], 0,
        C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "mra_eval_covariance_static")
    torch.cuda.synchronize()
    del keep
    return out.cpu().numpy()


FORMS = [(d, nu, p, True) for d, nu, p in itertools.product((CHORDAL, PLANAR), (1, 3), (1.0, 1.5))]
FORMS += [(PLANAR, 1, 1.25, True), (CHORDAL, 3, 0.75, True), (GREAT_CIRCLE, 1, 1.5, True), (GREAT_CIRCLE, 3, 1.0, True),
          (PLANAR, 3, 1.5, False), (CHORDAL, 1, 1.5, False)]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f"d{f[0]}nu{f[1]}p{f[2]}{'' if f[3] else 's'}")
def test_every_form_with_coincident_points(form):
    rng = np.random.default_rng(5)
    distance, nu, pref, nonstat = form
    md = model(rng, distance, nu, pref, nonstat=nonstat)
    th = dict(THETA, sill=md.sill, range=md.range_, nugget=md.nugget)
    p1, p2 = points(rng, distance, 75), points(rng, distance, 131)
    if distance != GREAT_CIRCLE:   # (the arc cosine has no digits left there)
        p2[:, 64:70] = p1[:, 31:37]
        p1[:, 50] = p1[:, 49]
    np.testing.assert_allclose(api.eval_covariance(md, th, p1, p2), expected(md, p1, p2), rtol=RTOL)
    np.testing.assert_allclose(api.eval_covariance(md, th, p1), expected(md, p1), rtol=RTOL)
    np.testing.assert_allclose(static_block(md, p1, p2), expected(md, p1, p2), rtol=RTOL)


# set-2 points are the rows: tiles of 256 or 64 rows, runs of at most 64 columns
@pytest.mark.parametrize("n1,n2", [(1, 1), (1, 700), (700, 1), (8, 64), (9, 65), (63, 255), (64, 256), (65, 257),
                                   (1200, 1300)])
def test_block_sizes(n1, n2):
    rng = np.random.default_rng(n1 + n2)
    md = model(rng, PLANAR, 3, 1.5)
    p1, p2 = points(rng, PLANAR, n1), points(rng, PLANAR, n2)
    np.testing.assert_allclose(static_block(md, p1, p2), expected(md, p1, p2), rtol=RTOL)


@pytest.mark.parametrize("nb", [36, 37, 300])
def test_basis_tables_by_value_and_copied(nb):
    """3 fields x 4 doubles x 36 functions are the most that travel with the launch."""
    rng = np.random.default_rng(nb)
    md = model(rng, CHORDAL, 1, 1.5, nb=nb)
    p1, p2 = points(rng, CHORDAL, 90), points(rng, CHORDAL, 40)
    np.testing.assert_allclose(static_block(md, p1, p2), expected(md, p1, p2), rtol=RTOL)


def test_negative_sill_scale():
    """The entry holds sqrt(sigma_a^2 sigma_b^2): both of one sign, whichever it is."""
    rng = np.random.default_rng(8)
    md = model(rng, PLANAR, 1, 1.5)
    p1, p2 = points(rng, PLANAR, 30), points(rng, PLANAR, 20)
    np.testing.assert_allclose(static_block(md, p1, p2, -1.0), expected(md, p1, p2), rtol=RTOL)
