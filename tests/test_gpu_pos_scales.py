"""shape_posvis in other length units: the model, its offsets and the pixel size
multiplied by a power of two give the oracle's images at that scale bit for bit,
also where a facet's area leaves FP32's range."""
import ctypes as C

import numpy as np
import pytest

import cases
from oracle.bindings import OrcPos
from shape_b200 import ctypes_defs as cd
from shape_b200 import engine as eng
from shape_b200 import synth
from test_gpu_pos_layers import PosImages, PosView

pytestmark = pytest.mark.gpu


# facets of a hundred pixels, and of a few
@pytest.mark.parametrize("levels,n", [(0, 120), (1, 120), (2, 60), (5, 60)])
@pytest.mark.parametrize("power", [-140, -64, 0, 60, 64, 66, 68, 72, 130, 400])
def test_units(cuda_device, levels, n, power):
    orc = cases.orc()
    lib = eng.load_library()
    unit = 2.0 ** power
    dirs, fv = synth.octa_sphere(levels)
    m = synth.make_model(dirs, fv, 1.0 + 0.2 * np.random.default_rng(3).uniform(-1.0, 1.0, dirs.shape[0]))
    real = orc.realize(m)
    real["x"] = real["x"] * unit
    R = orc._real(real)
    ae = synth.body_matrix(synth.ecl_dir(30.0, 60.0), 0.7)
    oe = synth.observer_matrix(synth.ecl_dir(0.0, 10.0))
    pos = OrcPos()
    orc.lib.orc_pos_alloc(C.byref(pos), n, 0)
    pos.kmpp = 1.3 / n * unit
    view = PosView(n, pos.kmpp, bistatic=0)
    for q in (pos, view):
        for k, a in (("ae", ae), ("oe", oe), ("se", oe)):
            getattr(q, k)[:] = np.asarray(a).ravel().tolist()
    orc.lib.orc_posclr(C.byref(pos))
    before = orc.pos_arrays(pos)
    img, own = PosImages(), {k: before[k].copy() for k in ("cose", "z", "f")}
    own["body"], own["comp"] = (np.full(own["f"].size, -1, dtype=np.int32) for _ in range(2))
    for k, a in own.items():
        setattr(img, k, cd.as_iptr(a) if a.dtype == np.int32 else cd.as_dptr(a))
    img.xlim[:], img.ylim[:] = pos.xlim[:], pos.ylim[:]
    orc.lib.orc_posvis.argtypes = [C.c_void_p, cd.dptr, C.c_void_p, C.c_int, C.c_int]
    lib.shape_posvis.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, cd.dptr, cd.dptr, C.c_int, cd.iptr,
                                 cd.dptr, cd.dptr, C.c_int, C.c_int, C.c_int, C.c_int]
    off = np.array([0.05, -0.03, 0.02]) * unit
    a = orc.lib.orc_posvis(C.byref(R), cd.as_dptr(off), C.byref(pos), 1, 0)
    b = lib.shape_posvis(0, C.byref(view), C.byref(img), R.nv, R.x, R.vn, R.nf, R.fv, R.fn, cd.as_dptr(off), 1, 0, 0, 0)
    assert a == b
    o = orc.pos_arrays(pos)
    assert (o["f"] >= 0).any()
    for k in ("f", "z", "cose"):
        assert np.array_equal(own[k], o[k]), k
    orc.lib.orc_pos_free(C.byref(pos))
