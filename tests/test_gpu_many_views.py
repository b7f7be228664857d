"""As many radar views as a launch grid takes in one dimension."""
import numpy as np
import pytest

from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views", [65534, 65535])
def test_grid_limit(cuda_device, views):
    dirs, fv = synth.octa_sphere(0)
    m = synth.make_model(dirs, fv, np.ones(dirs.shape[0]))
    p = synth.eval_params()
    ds = synth.batched_dataset(1, (9, 9), (8, 8), (8, 8), None, p, seed=3)
    ds.obs[:] = np.random.default_rng(17).standard_normal(ds.obs.size)
    e = eng.make_engine(m, p, deldops=[ds])
    one = e.evaluate(eng.FORM_BATCHED_FP64)["chi2"]
    e.close()
    n = ds.obs.size
    ds.frames, ds.obs, ds.oneovervar = ds.frames * views, np.tile(ds.obs, views), np.tile(ds.oneovervar, views)
    ds.offsets = np.arange(views + 1, dtype=np.int64) * n
    e = eng.make_engine(m, p, deldops=[ds])
    # 65535 rows of blocks bin the views; the vertex normals share a row beside
    # them or, where there is none left, have a launch of their own
    assert e.kernels_per_eval(eng.FORM_BATCHED_FP64) == (4 if views < 65535 else 5)
    for _ in range(2):
        assert e.evaluate(eng.FORM_BATCHED_FP64)["chi2"] == pytest.approx(views * one, rel=1e-10)
    e.close()
