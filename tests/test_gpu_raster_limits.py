"""Tiles past the raster's lists, rastered in chunks of facets: chunks whose own
candidates overflow, scans of all facets that meet a tile whose bin is full,
limb pixels whose cosine is several winners back. And coarse bodies, whose tiles
hold few facets of many pixels. Maps equal the oracle's in
every form and kernel, cos(e) in the FP64 forms; lightcurve views' too."""
import numpy as np
import pytest

import cases
from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu


def _rough(levels, sigma, seed=5):
    dirs, fv = synth.octa_sphere(levels)
    r = 1.0 + sigma * np.random.default_rng(seed).uniform(-1.0, 1.0, dirs.shape[0])
    return synth.make_model(dirs, fv, r)


def _engines(m, p, cap, add):
    for form in (eng.FORM_PLAIN_FP64, eng.FORM_BATCHED_FP64, eng.FORM_BATCHED_FP32):
        for mode in ((0, 1) if form != eng.FORM_PLAIN_FP64 else (0,)):
            e = eng.Engine()
            e.set_model(m)
            e.set_params(p)
            add(e)
            if cap:
                e.set_bin_capacity(cap)
            e.finalize()
            e.set_raster_tuning(mode)
            e.keep_pos(True)
            e.evaluate(form)
            yield e, form, mode
            e.close()


# (octahedron levels, roughness, POS half width, smoothing, bin capacity or 0)
GRID = [
    (3, 0.95, 3, 1, 0),         # 512 facets on one tile of 49 pixels: every chunk's candidates overflow
    (5, 0.6, 15, 1, 16),        # full bins, many layers: the chunks come from a scan
    (6, 0.95, 7, 1, 64),        # one tile of 15^2 pixels scanned out of 32768 facets
    (4, 0.45, 15, 0, 32),       # facet normals
    (2, 0.3, 40, 1, 1),         # few facets, each over several tiles
    # coarse bodies: tiles of few entries, whose pixels test all of them
    (0, 0.0, 33, 1, 0),         # 8 facets, edges through pixel centres
    (1, 0.5, 60, 1, 0),
    (2, 0.6, 50, 1, 0),         # limb pixels among them
    (3, 0.5, 50, 1, 0),         # some tiles of more than FEW entries
    (3, 0.5, 50, 0, 0),
    (2, 0.6, 50, 1, 5),         # few entries, full bins
]


@pytest.mark.parametrize("levels,sigma,n,smooth,cap", GRID)
def test_radar(cuda_device, levels, sigma, n, smooth, cap):
    m = _rough(levels, sigma)
    p = synth.eval_params(pos_smooth=smooth)
    ds = synth.batched_dataset(2, (2 * n + 1, 2 * n + 1), (64, 64), (64, 64), None, p, seed=3, radius=1.5)
    ds.obs[:] = np.random.default_rng(17).standard_normal(ds.obs.size)
    o = cases.orc().eval_deldop(m, ds, p, keep_pos=True)
    for e, form, mode in _engines(m, p, cap, lambda e: e.add_deldop(ds)):
        for f in range(ds.nframes):
            g = e.pos(f)
            for k in ("f", "z") + (("cose",) if form != eng.FORM_BATCHED_FP32 else ()):
                assert np.array_equal(g[k], o["pos"][f][k]), (form, mode, f, k)


@pytest.mark.parametrize("levels,sigma,pos,cap", [(6, 0.95, 31, 0), (4, 0.45, 41, 16), (2, 0.5, 101, 0)])
def test_lightcurve(cuda_device, levels, sigma, pos, cap):
    m = _rough(levels, sigma)
    p = synth.eval_params(mask_tol=0.0)
    lc = synth.lightcurve_dataset(3, (pos, pos), cases.lc_synth(m), p)
    o = cases.orc().eval_lghtcrv(m, lc, p, keep_pos=True)
    for e, form, mode in _engines(m, p, cap, lambda e: e.add_lghtcrv(lc)):
        for i, pt in enumerate(lc.points):
            g = e.lghtcrv_pos(0, i, pt)
            for k in g:
                assert np.array_equal(g[k], o["pos"][i][k]), (form, mode, i, k)
