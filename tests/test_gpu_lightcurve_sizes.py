"""Lightcurves from one point to more points than the finalize kernel's shared
memory holds (its work arrays are then in device memory), tiles inside and at
the edge of the window, every optical law; and plane-of-sky frames of unequal
sizes, whose fit grids and sky pixels are sliced over the same number of
blocks. Uniform epochs with the observations at the middle of each gap, so the
spline passes on the brightnesses' rounding (2e-16) with a factor of order one:
y and fit to rtol 1e-12 against the oracle, chi-square to 1e-10 of the sums it
is a difference of."""
import numpy as np
import pytest

import cases
from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,side,law", [(1, 17, 11), (2, 33, 2), (3, 31, 3), (33, 49, 11), (2600, 17, 11)])
def test_lightcurve_sizes(cuda_device, npts, side, law):
    m = synth.ellipsoid_model()
    p = synth.eval_params()
    ds = synth.lightcurve_dataset(npts, (side, side), None, p, seed=4, law_type=law)
    ds.x = 2458000.0 + 0.5 * np.arange(npts) / max(1, npts - 1)
    ds.t = ds.x[:-1] + 0.5 * np.diff(ds.x) if npts > 1 else ds.x.copy()
    for i, pt in enumerate(ds.points):
        synth.cd.fill9(pt.ae, synth.body_matrix(synth.ecl_dir(30.0, 60.0), 4 * np.pi * (ds.x[i] - ds.x[0])))
    n = len(ds.t)
    ds.set.n, ds.set.dof = n, float(n)
    ds.obs = 1e-17 * (1.0 + 0.1 * np.random.default_rng(npts).standard_normal(n))
    ds.oneovervar = 1.0 / (0.01 * ds.obs) ** 2
    ds.bind()
    o = cases.orc().eval_lghtcrv(m, ds, p)
    e = eng.make_engine(m, p, lghtcrvs=[ds])
    scale = float((ds.obs ** 2 * ds.oneovervar).sum())
    for form in (eng.FORM_PLAIN_FP64, eng.FORM_BATCHED_FP64, eng.FORM_BATCHED_FP32):
        s = e.evaluate(form)
        g = e.lghtcrv(0, ds)
        np.testing.assert_allclose(g["y"], o["y"], rtol=1e-12)
        np.testing.assert_allclose(g["fit"], o["fit"], rtol=1e-12)
        # one point has no spline: its fit and chi-square are the oracle's NaN
        assert abs(s["chi2"] - o["chi2"]) <= 1e-10 * scale or (np.isnan(s["chi2"]) and np.isnan(o["chi2"])), form
    e.close()


def test_sky_frames_of_unequal_sizes(cuda_device):
    """Each frame of a set of three sizes equals the frame evaluated alone:
    fit and brightness images exactly, sums to their order (1e-13)."""
    m = synth.ellipsoid_model()
    p = synth.eval_params()
    sizes = [(20, 11, 9), (75, 50, 37), (41, 64, 64)]
    frames, obs = [], []
    for k, (n, nc, nr) in enumerate(sizes):
        one = synth.poset_dataset(1, None, p, pos_n=n, ncol=nc, nrow=nr, fit_scale=2.6 * (2 * n + 1) / (2.2 * max(nc, nr)),
                                  resample=4, seed=3 + k)
        frames.append(one.frames[0])
        obs.append(np.random.default_rng(k).uniform(0.0, 1.0, nc * nr))
    law, oov = one.law, [np.full(o.size, 2.0) for o in obs]
    both = synth.PosetDataset(frames, law, 4, False, np.concatenate(obs), np.concatenate(oov))
    for form in (eng.FORM_PLAIN_FP64, eng.FORM_BATCHED_FP64, eng.FORM_BATCHED_FP32):
        e = eng.make_engine(m, p, posets=[both])
        e.evaluate(form)
        for k in range(len(sizes)):
            a = eng.make_engine(m, p, posets=[synth.PosetDataset([frames[k]], law, 4, False, obs[k], oov[k])])
            a.evaluate(form)
            fit, sky, r = e.poset(0, k)
            fit1, sky1, r1 = a.poset(0, 0)
            assert np.array_equal(fit, fit1) and np.array_equal(sky, sky1), (form, k)
            assert fit.max() > 0.0
            assert r["badposet"] == r1["badposet"] and r["badposet_logfactor"] == r1["badposet_logfactor"]
            for key in ("o2", "m2", "om", "cal"):
                assert abs(r[key] - r1[key]) <= 1e-13 * abs(r1[key]), (form, k, key)
            assert abs(r["chi2"] - r1["chi2"]) <= 1e-12 * r1["o2"], (form, k)
            a.close()
        e.close()
