"""The tile raster where its shared-memory lists run out: rough bodies whose
tiles hold more facets than a CTA has threads, pixels under more layers of
facets than a pixel's candidate list, tiles past the overflow list, bins
past their capacity, and windows that cut the body. Facet and depth maps
equal the oracle's in every form and kernel, cos(e) in the FP64 forms (the
limb pixels of a rough body take it from an earlier winner)."""
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


# (octahedron levels, roughness, POS half width, window in body radii, smoothing, bin capacity or 0)
GRID = [
    (2, 0.3, 8, 1.5, 1, 0),         # 128 facets, two tiles a side: fewer facets than threads
    (4, 0.45, 15, 1.6, 1, 0),       # 2048 facets on 31^2 pixels: bins past 128 and 256 entries, 8 layers and more
    (5, 0.6, 15, 1.8, 1, 0),        # 8192 facets on 31^2 pixels: 14 layers, some entries in the overflow lists
    (6, 0.95, 15, 2.2, 1, 0),       # 32768 facets on 31^2 pixels: the overflow lists run out
    (4, 0.45, 15, 1.6, 0, 0),       # facet normals
    (4, 0.45, 15, 0.7, 1, 0),       # the window cuts the body
    (3, 0.4, 23, 1.6, 1, 16),       # bins of 16 entries: the facet-scan path
]


@pytest.mark.parametrize("levels,sigma,n,window,smooth,cap", GRID)
def test_layers(cuda_device, levels, sigma, n, window, smooth, cap):
    m = _rough(levels, sigma)
    p = synth.eval_params(pos_smooth=smooth)
    ds = synth.batched_dataset(2, (2 * n + 1, 2 * n + 1), (64, 64), (64, 64), None, p, seed=3, radius=1.5)
    for fr in ds.frames:
        fr.km_per_pixel = window / n
    ds.obs[:] = np.random.default_rng(17).standard_normal(ds.obs.size)
    o = cases.orc().eval_deldop(m, ds, p, keep_pos=True)
    for form in (eng.FORM_PLAIN_FP64, eng.FORM_BATCHED_FP64, eng.FORM_BATCHED_FP32):
        for mode in ((0, 1) if form != eng.FORM_PLAIN_FP64 else (0,)):
            e = eng.Engine()
            e.set_model(m)
            e.set_params(p)
            e.add_deldop(ds)
            if cap:
                e.set_bin_capacity(cap)
            e.finalize()
            e.set_raster_tuning(mode)
            e.keep_pos(True)
            e.evaluate(form)
            for f in range(ds.nframes):
                g = e.pos(f)
                assert np.array_equal(g["f"], o["pos"][f]["f"]), (form, mode, f)
                assert np.array_equal(g["z"], o["pos"][f]["z"]), (form, mode, f)
                if form != eng.FORM_BATCHED_FP32:
                    assert np.array_equal(g["cose"], o["pos"][f]["cose"]), (form, mode, f)
            e.keep_pos(False)
            a, b = e.evaluate(form)["chi2"], sum(r["chi2"] for r in o["results"])
            assert abs(a - b) <= (1e-6 if form == eng.FORM_BATCHED_FP32 else 1e-10) * abs(b), (form, mode)
            e.close()
