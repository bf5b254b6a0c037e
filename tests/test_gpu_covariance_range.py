"""Covariance blocks at the ends of their range, against the oracle: scaled distances
where the exponential becomes denormal and then zero, infinite and undefined coordinates.

Tolerance: an argument of at most 745 with a relative error of a few roundings gives an
entry with 745 * 8 * 1.1e-16 < 1e-12 relative error.  A denormal exponential may be off by
its last digit, 5e-324 (the device's e^-745 is 0), which sigma^2 (1 + s) multiplies:
1.3 * 747 * 5e-324 < 5e-321, and as much for the rounding of the product."""
import itertools

import numpy as np
import pytest

import mra_oracle as oracle
from nonstationary_mra_b200 import api
from nonstationary_mra_b200.model import Field, Model

from test_gpu_covariance import CHORDAL, PLANAR, RTOL, THETA, expected, model, points, static_block

pytestmark = pytest.mark.gpu

FORMS = list(itertools.product((CHORDAL, PLANAR), (1, 3), (1.0, 1.5)))


def plain_model(distance, nu_x2, pref, dist_scale=1.0):
    """Constant fields (no basis functions): sigma^2 = 1.3, beta = 0.5, tau^2 = 0.1."""
    fields = [Field(np.log(v), np.zeros((3, 0)), np.zeros(0)) for v in (1.3, 0.5, 0.1)]
    return Model(nonstationary=True, distance=distance, nu_x2=nu_x2, prefactor_exp=pref, dist_scale=dist_scale,
                 basis_len=0.4, fields=fields)


def line(x):
    return np.vstack([x, np.zeros((2, len(x)))])


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f"d{f[0]}nu{f[1]}p{f[2]}")
def test_block_tail_and_undefined(form):
    distance, nu, pref = form
    md = plain_model(*form)
    # exponents (sqrt(3) d / 0.5 or d / 0.5) of 0, 1, 60, ... infinity, and an undefined coordinate
    h = np.array([0.0, 1.0, 60.0, 699.0, 699.9, 700.0, 700.0004, 701.0, 708.0, 709.0, 720.0, 744.0, 746.0, 800.0, 1e4, 1e9,
                  1e160, np.inf, np.nan])
    p1, p2 = line(0.5 * h / (np.sqrt(3.0) if nu == 3 else 1.0)), line(np.array([0.0, 0.25]))
    th = dict(THETA, sill=1.0, range=1.0, nugget=0.0)
    with np.errstate(all="ignore"):
        ref = expected(md, p1, p2)
        ref_self = expected(md, p1)
    for out, want in ((api.eval_covariance(md, th, p1, p2), ref), (static_block(md, p1, p2), ref),
                      (api.eval_covariance(md, th, p1), ref_self)):
        assert np.array_equal(np.isnan(out), np.isnan(want))
        np.testing.assert_allclose(out, want, rtol=RTOL, atol=1e-320)


@pytest.mark.parametrize("form", list(itertools.product((1, 3), (1.0, 1.5, 1.25))), ids=lambda f: f"nu{f[0]}p{f[1]}")
def test_third_coordinate_of_planar_points(form):
    """The straight-line distances are one formula: planar points enter it with all three
    coordinates (zero in the third, as the readers write it), in every kernel."""
    rng = np.random.default_rng(12)
    md = model(rng, PLANAR, *form)
    p1, p2 = rng.random((3, 70)) * 0.5, rng.random((3, 90)) * 0.5
    md.fields[0].centers[2] = 0.1
    th = dict(THETA, sill=1.0, range=1.0, nugget=0.0)
    md.distance = CHORDAL
    ref, ref_self = expected(md, p1, p2), expected(md, p1)
    md.distance = PLANAR
    np.testing.assert_allclose(api.eval_covariance(md, th, p1, p2), ref, rtol=RTOL)
    np.testing.assert_allclose(static_block(md, p1, p2), ref, rtol=RTOL)
    np.testing.assert_allclose(api.eval_covariance(md, th, p1), ref_self, rtol=RTOL)


def test_third_coordinate_in_an_evaluation():
    """The same problem on planar points as on chordal ones: bitwise, through every kernel (small
    and heavy finest regions, prediction in vectors and in tiles)."""
    from test_gpu_parity import random_case, run_loglik
    st, md = random_case(44, 4, 4, 49, 2500, 300, True, 1, True)
    rng = np.random.default_rng(3)
    for a in (st.knots, st.obs, st.pred):
        a[2] = 0.05 * rng.random(a.shape[1])
    out = []
    for md.distance in (PLANAR, CHORDAL):
        ctx, (d, _) = run_loglik(st, md)
        mean, var = ctx.predict()
        out.append((d, mean, var))
        ctx.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f"d{f[0]}nu{f[1]}p{f[2]}")
def test_negative_distance_scale(form):
    """A block takes the scale with its sign; an evaluation's straight-line entries take its square."""
    from test_gpu_parity import random_case, run_loglik
    md = plain_model(*form, dist_scale=-1.5)
    rng = np.random.default_rng(2)
    p1, p2 = line(rng.random(70)), line(rng.random(90))
    th = dict(THETA, sill=1.0, range=1.0, nugget=0.0)
    ref = expected(md, p1, p2)
    np.testing.assert_allclose(api.eval_covariance(md, th, p1, p2), ref, rtol=RTOL)
    np.testing.assert_allclose(static_block(md, p1, p2), ref, rtol=RTOL)
    st, md = random_case(4, 4, 3, 16, 900, 40, True, form[1], True)
    md.distance, md.prefactor_exp = form[0], form[2]
    out = []
    for md.dist_scale in (1.0, -1.0):
        ctx, (d, _) = run_loglik(st, md)
        out.append((d, *ctx.predict()))
        ctx.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("nu", [1, 3])
@pytest.mark.parametrize("distance,pref,dist_scale", [(CHORDAL, 1.5, 6371.0), (PLANAR, 1.0, 1.0)])
def test_block_error_against_extended_precision(distance, pref, dist_scale, nu):
    """From the library's own fields, a block is no further from its value in extended precision
    than the literal expression evaluated in 64 bits (norm over 2 million entries; counting the
    roundings of both gives 0.88 to 0.96 of the literal form's error)."""
    L = np.longdouble
    rng = np.random.default_rng(20)
    if distance == CHORDAL:
        def draw(n):
            lon, lat = np.radians(-120 + 40 * rng.random(n)), np.radians(25 + 25 * rng.random(n))
            return np.stack([np.cos(lat) * np.cos(lon), np.cos(lat) * np.sin(lon), np.sin(lat)])
    else:
        def draw(n):
            return np.vstack([rng.random((2, n)), np.zeros((1, n))])
    centers = [draw(9) for _ in range(3)]
    fields = [Field(a, c, 0.3 * rng.standard_normal(9))
              for a, c in zip((0.1, np.log(300.0 if distance == CHORDAL else 0.1), -3.0), centers)]
    md = Model(nonstationary=True, distance=distance, nu_x2=nu, prefactor_exp=pref, dist_scale=dist_scale, basis_len=0.25,
               fields=fields)
    p1, p2 = draw(1500), draw(1300)
    th = dict(THETA, sill=1.0, range=1.0, nugget=0.0)
    f1, f2 = api.eval_fields(md, th, p1), api.eval_fields(md, th, p2)
    omd = oracle.Model(nonstationary=True, distance=distance, nu_x2=nu, prefactor_exp=pref, dist_scale=dist_scale,
                       basis=md.basis, basis_len=md.basis_len, fields=[])
    literal = oracle.cross_cov(omd, p1, f1, p2, f2)
    d2 = sum((p1[c].astype(L)[:, None] - p2[c].astype(L)[None, :]) ** 2 for c in range(3))
    (s1, b1, _), (s2, b2, _) = f1.astype(L), f2.astype(L)
    bms = (b1[:, None] ** 2 + b2[None, :] ** 2) / 2
    h = L(dist_scale) * np.sqrt(d2 / bms) * (np.sqrt(L(3)) if nu == 3 else 1)
    exact = np.sqrt(s1[:, None] * s2[None, :]) * (b1[:, None] * b2[None, :] / bms) ** L(pref) * np.exp(-h)
    if nu == 3:
        exact *= 1 + h
    norm = lambda out: float(np.sqrt(((out - exact) ** 2).sum() / (exact ** 2).sum()))
    for out in (static_block(md, p1, p2), api.eval_covariance(md, th, p1, p2)):
        assert norm(out) <= norm(literal), (norm(out), norm(literal))


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f"d{f[0]}nu{f[1]}p{f[2]}")
def test_negative_sill_scale_of_every_form(form):
    """sqrt(sigma_a^2 sigma_b^2) of two negative values: its square root once, or a root per point."""
    rng = np.random.default_rng(8)
    md = model(rng, *form)
    p1, p2 = points(rng, form[0], 75), points(rng, form[0], 20)
    ref = expected(md, p1, p2)
    np.testing.assert_allclose(static_block(md, p1, p2, -1.0), ref, rtol=RTOL)
    np.testing.assert_allclose(api.eval_covariance(md, dict(THETA, sill_scale=-1.0), p1, p2), ref, rtol=RTOL)


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f"d{f[0]}nu{f[1]}p{f[2]}")
def test_undefined_distance_scale(form):
    """An undefined scale makes the entries undefined: an error status, not a finite log-likelihood."""
    from nonstationary_mra_b200.capi import MRAError
    from test_gpu_parity import random_case, run_loglik
    st, md = random_case(4, 4, 3, 16, 900, 40, False, form[1], True)
    md.distance, md.prefactor_exp, md.dist_scale = form[0], form[2], float("nan")
    with pytest.raises(MRAError, match="NOT_SPD"):
        run_loglik(st, md)
