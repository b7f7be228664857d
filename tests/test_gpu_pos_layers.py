"""shape_posvis on images that already hold a body, where the raster's lists run
out: a second rough body added to a first one's images, each pixel keeping the
nearer. Images and limits equal the oracle's bit for bit."""
import ctypes as C

import numpy as np
import pytest

import cases
from oracle.bindings import OrcPos
from shape_b200 import ctypes_defs as cd
from shape_b200 import engine as eng
from shape_b200 import synth

pytestmark = pytest.mark.gpu


class PosView(C.Structure):
    _fields_ = [("n", C.c_int), ("km_per_pixel", C.c_double), ("ae", C.c_double * 9), ("oe", C.c_double * 9),
                ("se", C.c_double * 9), ("bistatic", C.c_int)]


class PosImages(C.Structure):
    _fields_ = [("b", cd.dptr), ("cose", cd.dptr), ("cosi", cd.dptr), ("z", cd.dptr), ("body", cd.iptr),
                ("comp", cd.iptr), ("f", cd.iptr), ("cosill", cd.dptr), ("zill", cd.dptr), ("bodyill", cd.iptr),
                ("compill", cd.iptr), ("fill", cd.iptr), ("xlim", C.c_int * 2), ("ylim", C.c_int * 2),
                ("xlim2", C.c_int * 2), ("ylim2", C.c_int * 2), ("posbnd_logfactor", C.c_double)]


def _rough(levels, sigma, seed):
    dirs, fv = synth.octa_sphere(levels)
    r = 1.0 + sigma * np.random.default_rng(seed).uniform(-1.0, 1.0, dirs.shape[0])
    return synth.make_model(dirs, fv, r)


# (octahedron levels, roughness, POS half width, smoothing)
GRID = [
    (2, 0.5, 45, 1),        # tiles of few facets
    (3, 0.4, 20, 1),
    (4, 0.45, 15, 0),
    (5, 0.6, 15, 1),        # pixels past their own candidate lists
    (6, 0.95, 15, 1),       # tiles past the overflow lists
    (3, 0.95, 3, 1),        # 49 pixels in one tile: chunks past the overflow list too
    (7, 0.9, 7, 1),         # one tile of more facets than a bin may hold: all facets are scanned
]


@pytest.mark.parametrize("levels,sigma,n,smooth", GRID)
@pytest.mark.parametrize("src", [0, 1])
def test_added_body(cuda_device, levels, sigma, n, smooth, src):
    orc = cases.orc()
    lib = eng.load_library()
    pole = synth.ecl_dir(30.0, 60.0)
    ae = synth.body_matrix(pole, 0.7)
    oe, se = synth.observer_matrix(synth.ecl_dir(0.0, 10.0)), synth.observer_matrix(synth.ecl_dir(55.0, -5.0))
    kmpp = 1.8 / n
    pos = OrcPos()
    orc.lib.orc_pos_alloc(C.byref(pos), n, 1)
    pos.kmpp, pos.bistatic = kmpp, 1
    view = PosView(n, kmpp, bistatic=1)
    for q in (pos, view):
        for k, m in (("ae", ae), ("oe", oe), ("se", se)):
            getattr(q, k)[:] = np.asarray(m).ravel().tolist()
    orc.lib.orc_posclr(C.byref(pos))
    before = orc.pos_arrays(pos)
    img, own = PosImages(), {}
    for k in ("cose", "cosi", "z", "f", "zill", "fill"):
        own[k] = before[k].copy()
        setattr(img, k, (cd.as_iptr if k in ("f", "fill") else cd.as_dptr)(own[k]))
    own["cosill"] = np.zeros(own["z"].size)
    img.cosill = cd.as_dptr(own["cosill"])
    for k in ("body", "comp", "bodyill", "compill"):
        own[k] = np.full(own["z"].size, -1, dtype=np.int32)
        setattr(img, k, cd.as_iptr(own[k]))
    for k in ("xlim", "ylim", "xlim2", "ylim2"):
        getattr(img, k)[:] = getattr(pos, k)[:]
    orc.lib.orc_posvis.argtypes = [C.c_void_p, cd.dptr, C.c_void_p, C.c_int, C.c_int]
    lib.shape_posvis.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, cd.dptr, cd.dptr, C.c_int, cd.iptr,
                                 cd.dptr, cd.dptr, C.c_int, C.c_int, C.c_int, C.c_int]
    for body, seed in enumerate((5, 6)):
        real = orc.realize(_rough(levels, sigma, seed))
        R = orc._real(real)
        off = np.array([0.3, -0.2, 0.1]) * body
        a = orc.lib.orc_posvis(C.byref(R), cd.as_dptr(off), C.byref(pos), smooth, src)
        b = lib.shape_posvis(0, C.byref(view), C.byref(img), R.nv, R.x, R.vn, R.nf, R.fv, R.fn, cd.as_dptr(off),
                             smooth, src, body, 0)
        assert a == b
        o = orc.pos_arrays(pos)
        o["cosill"] = np.ctypeslib.as_array(C.cast(pos.cosill, C.POINTER(C.c_double)), shape=o["z"].shape)
        for k in ("f", "z", "cose", "cosi", "fill", "zill", "cosill"):
            assert np.array_equal(own[k], o[k]), (body, k)
        for k in ("xlim", "ylim", "xlim2", "ylim2"):
            assert tuple(getattr(img, k)) == o[k], (body, k)
        who = own["bodyill" if src else "body"]
        assert (who[own["fill" if src else "f"] < 0] == -1).all() and (body == 0 or (who == 1).any())
    orc.lib.orc_pos_free(C.byref(pos))
