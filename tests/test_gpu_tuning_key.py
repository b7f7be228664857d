"""Which engines share a raster choice, and which lines of a tuning file count:
the radar, sun and observer views' rasters are kernels of their own, and a line
that an older build wrote was timed on other kernels."""
import ctypes as C
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import cases
from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_radar_and_lightcurve_views_are_timed_apart(cuda_device):
    """Two points whose sun stands behind the observer and four radar frames of
    the same views: equal models, views, tiles and bins."""
    m = cases.c2_model()
    p = synth.eval_params()
    lc = synth.lightcurve_dataset(2, (101, 101), None, p)
    lc.obs[:] = 1.0
    for q in lc.points:
        q.se[:] = q.oe[:]
    ds = synth.batched_dataset(4, (101, 101), (64, 64), (64, 64), None, p, seed=3)
    ds.obs[:] = np.random.default_rng(17).standard_normal(ds.obs.size)
    for k, f in enumerate(ds.frames):
        q = lc.points[k // 2]
        f.ae[:], f.oe[:], f.km_per_pixel = q.ae[:], q.oe[:], q.km_per_pixel
    radar, curve = eng.make_engine(m, p, deldops=[ds]), eng.make_engine(m, p, lghtcrvs=[lc])
    info = []
    for e in (radar, curve):
        e.evaluate(eng.FORM_BATCHED_FP64)
        bins = (C.c_int * 5)()                  # capacity, fullest tile, tiles with facets, tiles, tile side
        assert e.L.shape_engine_get_tuning(e.h, bins, 5) == 5
        info.append((e.raster_tuning(eng.FORM_BATCHED_FP64), list(bins)))
    assert info[0][1] == info[1][1]
    assert info[0][0]["ms"] != info[1][0]["ms"]
    radar.close()
    curve.close()


_SNIPPET = r"""
import json, os, sys
sys.path.insert(0, os.environ["REPO"]); sys.path.insert(0, os.path.join(os.environ["REPO"], "tests"))
sys.path.insert(0, os.path.join(os.environ["REPO"], "shape-cuda-v1.2_b200", "python"))
import cases
from shape_b200 import engine as eng
m, p, ds = cases.c2(12)
e = eng.make_engine(m, p, deldops=[ds])
e.evaluate(eng.FORM_BATCHED_FP64)
print(json.dumps(e.raster_tuning(eng.FORM_BATCHED_FP64)))
e.close()
"""


def _run(path):
    env = dict(os.environ, REPO=REPO, SHAPE_B200_TUNING_CACHE=str(path))
    out = subprocess.run([sys.executable, "-c", _SNIPPET], env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    return json.loads(out.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("line", ["first format", "other kernels"])
def test_lines_of_other_builds_are_not_taken(cuda_device, tmp_path, line):
    path = tmp_path / "tuning.jsonl"
    _run(path)
    rec = json.loads(path.read_text())
    planted = [9.0, 8.0, 7.0, 6.0]
    if line == "first format":
        old = {k: rec[k] for k in ("gpu", "form")}
        old["exact"] = 0
        old.update({k: rec[k] for k in ("views", "facets")})
        old["nonempty"] = int(np.sum(rec["nonempty"]))
        old.update({k: rec[k] for k in ("maxcount16", "variant", "persistent")})
        old["ms"] = planted
    else:
        old = dict(rec, kernels=rec.get("kernels", 2) + 1, ms=planted)
    path.write_text(json.dumps(old) + "\n")
    assert _run(path)["ms"] != planted
    # a line of this build's is
    path.write_text(json.dumps(dict(rec, ms=planted)) + "\n")
    assert _run(path)["ms"] == planted


def test_fp32_exact_keeps_the_choice(cuda_device):
    """The switch changes no result, so it does not have the form timed again."""
    m, p, ds = cases.c2(12)
    e = eng.make_engine(m, p, deldops=[ds])
    e.evaluate(eng.FORM_BATCHED_FP32)
    a = e.raster_tuning(eng.FORM_BATCHED_FP32)
    for exact in (False, True):
        e.set_fp32_exact(exact)
        assert e.raster_tuning(eng.FORM_BATCHED_FP32) == a and a["tuned"]
        e.evaluate(eng.FORM_BATCHED_FP32)
        assert e.raster_tuning(eng.FORM_BATCHED_FP32) == a
    e.close()
