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
