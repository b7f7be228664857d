"""Binning and vertex normals within a batched evaluation's first launch (few
facets and views) against the plain form, which bins and realizes in launches
of their own: mesh sizes around a block of vertices, poles with more facets
than a block has threads, views x facets at the limit and just past it, and
evaluations that follow one another with changed parameters, also after the
other forms. Maps, normals and marked facets are equal. Then many views, whose
vertices a thread of that launch writes for several at a time."""
import numpy as np
import pytest

from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu

# (mesh, frames, launches before the raster)
GRID = [
    (("octa", 0), 1, 1),            # 6 vertices, 8 facets
    (("octa", 2), 2, 1),            # 66 vertices: three blocks of vertices, the last of two
    (("ring", 5, 300), 2, 1),       # poles of 300 facets
    (("octa", 6), 4, 1),            # 4 x 32768 facets: the most that the first launch bins
    (("octa", 6), 5, 2),
]


def _model(mesh):
    dirs, fv = synth.octa_sphere(mesh[1]) if mesh[0] == "octa" else synth.ring_sphere(mesh[1], mesh[2])
    r = 1.0 + 0.1 * np.random.default_rng(3).uniform(-1.0, 1.0, dirs.shape[0])
    return synth.make_model(dirs, fv, r)


@pytest.mark.parametrize("mesh,frames,launches", GRID)
def test_front_bins(cuda_device, mesh, frames, launches):
    m = _model(mesh)
    p = synth.eval_params()
    ds = synth.batched_dataset(frames, (41, 75), (48, 48), (48, 48), None, p, seed=3, radius=1.5)
    ds.obs[:] = np.random.default_rng(17).standard_normal(ds.obs.size)
    a, b = (eng.make_engine(m, p, deldops=[ds]) for _ in range(2))
    assert a.kernels_per_eval(eng.FORM_BATCHED_FP64) == launches + 2      # raster, chi-square
    for e in (a, b):
        e.keep_pos(True)
    for step in range(4):
        for e in (a, b):
            if step == 1:
                e.set_scale(0, 1.04)
            if step == 2:                       # more changes than travel with the launch
                for i in range(min(m.nv, 20)):
                    e.set_vertex_r(i, 0.01 * i)
            if step == 3:
                e.set_vertex_r(1, 0.05)
        if step == 2:
            a.stage_times(eng.FORM_BATCHED_FP64)
            a.evaluate(eng.FORM_PLAIN_FP64)
        x = a.evaluate(eng.FORM_BATCHED_FP64)["chi2"]
        y = b.evaluate(eng.FORM_PLAIN_FP64)["chi2"]
        assert abs(x - y) <= 1e-10 * abs(y)
        for f in range(frames):
            u, v = a.pos(f), b.pos(f)
            for k in ("f", "z", "cose"):
                assert np.array_equal(u[k], v[k]), (step, f, k)
        u, v = a.realized(), b.realized()
        for k in u:
            assert np.array_equal(u[k], v[k]), (step, k)
        assert np.array_equal(a.seen(), b.seen())
    a.close()
    b.close()


# views x blocks of 256 vertices over 8 blocks per SM give the views of a
# thread: 17 blocks, 1 + 2 x 34 views: one each; 151: two, the last group of
# one; 211: three, the last of one; 601: eight, the last of one
@pytest.mark.parametrize("points", [34, 75, 105, 300])
def test_front_views(cuda_device, points):
    m = _model(("octa", 5))
    p = synth.eval_params()
    lc = synth.lightcurve_dataset(points, (33, 49), None, p)
    lc.obs[:] = 1.0
    ds = synth.batched_dataset(1, (41, 41), (48, 48), (48, 48), None, p, seed=3, radius=1.5)
    ds.obs[:] = np.random.default_rng(17).standard_normal(ds.obs.size)
    a, b = (eng.make_engine(m, p, deldops=[ds], lghtcrvs=[lc]) for _ in range(2))
    for scale in (1.0, 0.97):
        for e in (a, b):
            e.keep_pos(True)
            e.set_scale(2, scale)
        x, y = a.evaluate(eng.FORM_BATCHED_FP64)["chi2"], b.evaluate(eng.FORM_PLAIN_FP64)["chi2"]
        assert abs(x - y) <= 1e-10 * abs(y)
        u, v = a.pos(0), b.pos(0)
        assert all(np.array_equal(u[k], v[k]) for k in ("f", "z", "cose"))
        for k in (0, points // 2, points - 1):
            u, v = (e.lghtcrv_pos(1, k, lc.points[k]) for e in (a, b))
            assert all(np.array_equal(u[q], v[q]) for q in u), k
        # a tile's brightness is summed in the order of its CTA's threads, of
        # which the forms may have 256 or 128: the lightcurves' own bar
        assert np.allclose(a.lghtcrv(1, lc)["y"], b.lghtcrv(1, lc)["y"], rtol=1e-12, atol=0.0)
    a.close()
    b.close()
