"""The radar frames' chi-square sums (m2 = sum fit^2/var, om = sum fit obs/var)
against exact sums of the same terms, formed from the fit image that the
evaluation left."""
import math

import numpy as np
import pytest

from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu

FORMS = [eng.FORM_PLAIN_FP64, eng.FORM_BATCHED_FP64, eng.FORM_BATCHED_FP32]


def _engine(m, p, ds, obs, oov):
    ds.obs[:], ds.oneovervar[:] = obs, oov
    return eng.make_engine(m, p, deldops=[ds])


# a wide image whose lit box (about half of it) has many bins for every thread,
# one of a few bins a thread
@pytest.mark.parametrize("side,pos", [(1024, 601), (200, 151)])
@pytest.mark.parametrize("form", FORMS)
def test_small_terms_behind_a_large_one(cuda_device, form, side, pos):
    """Every lit bin's term is about 1 but the first one's, 2^54, beside which a
    term of 1 is less than half an ulp: a plain running sum loses each one that
    follows it. A thread may add 16 bins in plain FP64 before it compensates
    (each of those additions is off by at most half an ulp of 2^54, 2): 32
    with the rounded total's own 2."""
    m = synth.harmonic_model()
    p = synth.eval_params()
    ds = synth.batched_dataset(1, (pos, pos), (side, side), (side, side), None, p, seed=3)
    n = side * side
    e = _engine(m, p, ds, np.zeros(n), np.ones(n))
    e.evaluate(form)
    fit = e.fit(0)
    e.close()
    lit = np.nonzero(fit)[0]
    oov = np.zeros(n)
    oov[lit] = 1.0 / fit[lit] ** 2
    oov[lit[0]] *= 2.0 ** 54
    e = _engine(m, p, ds, fit, oov)
    e.evaluate(form)
    f, r = e.fit(0), e.results()[0]
    e.close()
    m2, om = math.fsum(f * f * oov), math.fsum(f * fit * oov)
    assert m2 > 2.0 ** 53
    assert abs(r["m2"] - m2) <= 32 and abs(r["om"] - om) <= 32


@pytest.mark.parametrize("form", FORMS)
def test_bins_without_fit_add_nothing(cuda_device, form):
    """Bins that the model does not light, among them those between the lit ones
    of its box, leave m2 and om as they are even where 1/var is infinite or the
    observation is not a number (the sum of obs^2/var is then neither)."""
    m = synth.harmonic_model()
    p = synth.eval_params()
    ds = synth.batched_dataset(1, (151, 151), (200, 200), (200, 200), None, p, seed=3)
    n = 200 * 200
    obs = np.random.default_rng(17).standard_normal(n)
    e = _engine(m, p, ds, obs, np.ones(n))
    e.evaluate(form)
    fit, a = e.fit(0), e.results()[0]
    size = {"m2": a["m2"], "om": np.abs(fit * obs).sum()}
    e.close()
    dark = np.nonzero(fit == 0)[0]
    rows, cols = np.nonzero(fit.reshape(200, 200))
    box = (dark // 200 >= rows.min()) & (dark // 200 <= rows.max()) & (dark % 200 >= cols.min()) & \
        (dark % 200 <= cols.max())
    assert box.sum() > 100
    oov = np.ones(n)
    oov[dark[::2]] = np.inf
    obs[dark[1::2]] = np.nan
    e = _engine(m, p, ds, obs, oov)
    e.evaluate(form)
    b = e.results()[0]
    e.close()
    # two evaluations' images differ in the order of their additions: the
    # forms' own bars
    tol = 1e-6 if form == eng.FORM_BATCHED_FP32 else 1e-12
    assert not np.isfinite(b["o2"])
    for k in size:
        assert abs(b[k] - a[k]) <= tol * size[k], k


# images of one share of the data's sum, of eight and of 256
@pytest.mark.parametrize("side", [30, 200, 1024])
def test_observed_sum(cuda_device, side):
    """sum obs^2/var, formed once per dataset: a term of 2^54 before terms of 1,
    each addition compensated, so the total is off by its own rounding (2)."""
    m = synth.harmonic_model()
    p = synth.eval_params()
    ds = synth.batched_dataset(1, (151, 151), (side, side), (side, side), None, p, seed=3)
    oov = np.ones(side * side)
    oov[0] = 2.0 ** 54
    e = _engine(m, p, ds, np.ones(side * side), oov)
    e.evaluate(eng.FORM_BATCHED_FP64)
    assert abs(e.results()[0]["o2"] - math.fsum(oov)) <= 2
    e.close()
