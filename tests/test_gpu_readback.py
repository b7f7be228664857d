"""Images read back through a buffer that may be smaller than they are: just under
a buffer's bytes, exactly these and just over, several buffers, and past the size
that is copied straight. Each equals the oracle's image to the FP64 forms' bar."""
import numpy as np
import pytest

import cases
from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu

# delay x Doppler bins; the buffer holds 131072 doubles, and straight copies begin
# past 524288
SIZES = [(127, 129), (129, 1016), (256, 512), (331, 396), (301, 871), (512, 1024), (725, 724), (1025, 1024)]


@pytest.mark.parametrize("ndel,ndop", SIZES)
@pytest.mark.parametrize("form", [eng.FORM_BATCHED_FP64, eng.FORM_BATCHED_FP32])
def test_fit(cuda_device, form, ndel, ndop):
    m = synth.ellipsoid_model()
    p = synth.eval_params()
    ds = synth.batched_dataset(2, (101, 101), (ndel, ndel), (ndop, ndop), None, p, seed=3)
    o = cases.orc().eval_deldop(m, ds, p)["fits"]
    e = eng.make_engine(m, p, deldops=[ds])
    e.evaluate(form)
    tol = 1e-5 if form == eng.FORM_BATCHED_FP32 else 1e-12
    for _ in range(2):                          # the second read finds the buffer
        for f in range(2):
            a = e.fit(f)
            assert a.size == ndel * ndop
            assert np.abs(a - o[f]).max() <= tol * o[f].max()
            assert np.array_equal(a != 0, e.fit(f) != 0)
    e.close()
