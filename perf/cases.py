"""The work this framework is used for, as measurable cases.

A SHAPE fit evaluates its objective thousands of times: a trial moves a few
model parameters, the engine renders every view of every dataset, synthesizes
the radar images, spectra, brightnesses and sky images, and returns the
chi-square. The cases go through the engine's public calls (`make_engine`,
`set_scale`, `set_vertex_r`, `evaluate`, `fit`, `lghtcrv`, `poset`, `Server.run`)
as a fitting program does, from one small radar frame (latency) to hundreds
of lightcurve views (throughput).

Observed data are made from the true model by the FP64 renderer at the end of
this file, which is plain torch and uses none of the engine; `exact` gives the
outputs of a case from the same renderer.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "shape-cuda-v1.2_b200", "python"))

from shape_b200 import ctypes_defs as cd  # noqa: E402
from shape_b200 import engine as eng  # noqa: E402
from shape_b200 import synth  # noqa: E402

SHORT, LONG_ORIG, LONG_MOD = 0, 1, 2
LAMBERT, LOMMEL, KAASALAINEN = 2, 3, 11
BILINEAR, CUBICCONV = 2, 4


# ------------------------------------------------------------------- the cases

def _case(name, kind, form, **kw):
    """Defaults: a unit body of 2300 facets, smoothed normals, LONG_ORIG code
    with one sample per baud, one sinc^2 point per pixel, the cosine law."""
    c = dict(name=name, kind=kind, form=form, rings=23, per=50, octa=0, smooth=True, layout=7, frames=1, views=1,
             side_lo=151, side_hi=151, ndel_lo=100, ndel_hi=100, ndop_lo=100, ndop_hi=100, code=LONG_ORIG, spb=1,
             stride=1, nsinc2=1, law=1, images=False, seen=False)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest trial: one delay-Doppler frame of a coarse ellipsoid, one objective value back
        _case("one_frame_fp32", "radar", "batched_fp32"),
        # the last evaluation of a fit on that frame: the fitted image and the frame's results are read back
        _case("one_frame_fp64_image", "radar", "batched_fp64", images=True),
        # an ordinary trial: a radar campaign of 64 frames of uneven sizes, an 8000-facet model
        _case("campaign64_fp32", "radar", "batched_fp32", rings=40, per=100, frames=64, side_lo=101, side_hi=301,
              ndel_lo=64, ndel_hi=256, ndop_lo=64, ndop_hi=512),
        # the same trial where the fit asks for the reference's own precision
        _case("campaign64_fp64", "radar", "batched_fp64", rings=40, per=100, frames=64, side_lo=101, side_hi=301,
              ndel_lo=64, ndel_hi=256, ndop_lo=64, ndop_hi=512, seen=True),
        # close approach: few frames, large sky windows, a fine model
        _case("close16_fp32", "radar", "batched_fp32", octa=6, frames=16, side_lo=511, side_hi=511, ndel_lo=256,
              ndel_hi=256, ndop_lo=256, ndop_hi=256),
        # frames smeared over three views, a code of two samples per baud, four sinc^2 points per pixel; images read
        _case("smeared4_fp64", "radar", "batched_fp64", frames=4, views=3, code=LONG_MOD, spb=2, nsinc2=2, images=True),
        # Doppler-only spectra of odd lengths
        _case("spectra9_fp32", "doppler", "batched_fp32", rings=40, per=100, frames=9, side_lo=101, side_hi=301,
              ndop_lo=63, ndop_hi=255),
        # one short lightcurve, its curve read back
        _case("light25_fp64", "light", "batched_fp64", frames=25, sets=1, side_lo=129, side_hi=257, rings=40, per=100),
        # four lightcurves of 200 points: the largest evaluation, curves read back
        _case("light800_fp32", "light", "batched_fp32", frames=200, sets=4, side_lo=129, side_hi=257, rings=40, per=100),
        # resolved sky images (adaptive optics): rendering, resampling, images read back
        _case("sky3_fp32", "sky", "batched_fp32", frames=3, side_lo=181, side_hi=181, ncol=57, nrow=46, fit_scale=2.6,
              resample=CUBICCONV),
        # a stretch of a fit: line-search trials of the scale factors and of five vertices, one after the other
        _case("trials24_fp64", "fit", "batched_fp64", frames=4, vertices=5),
        # a burst of requests to the evaluation server: workloads of one to eight frames
        _case("serve48_fp32", "serve", "batched_fp32", frames=8, workloads=4, requests=48),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: sizes over their logarithm, the options that change a path at random."""
    kind = rng.choice(["radar"] * 5 + ["doppler", "light", "light", "sky", "fit", "serve"])
    form = rng.choice(["batched_fp32", "batched_fp64"])
    c = _case("", kind, form, layout=rng.randrange(1, 10 ** 6), rings=_log_int(rng, 13, 60), per=_log_int(rng, 24, 150),
              smooth=rng.random() < 0.85, images=rng.random() < 0.3, law=rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7]))
    del c["name"]
    side = _log_int(rng, 61, 511) | 1
    c["side_lo"], c["side_hi"] = max(61, int(0.6 * side)), side
    c["ndel_hi"], c["ndop_hi"] = _log_int(rng, 48, 256), _log_int(rng, 48, 512)
    c["ndel_lo"], c["ndop_lo"] = max(48, c["ndel_hi"] // 2), max(48, c["ndop_hi"] // 2)
    most = max(1, int(4.0e6 / side ** 2))        # views of this size that stay below the largest listed case
    if kind in ("radar", "doppler"):
        c["frames"] = _log_int(rng, 1, min(64, most))
        c["nsinc2"] = rng.choice([1, 1, 1, 2, 3])
    if kind == "radar":
        c["code"], c["spb"], c["stride"] = rng.choice(
            [(LONG_ORIG, 1, 1)] * 4 + [(SHORT, 1, 1), (LONG_ORIG, 2, 1), (LONG_MOD, 2, 1), (LONG_MOD, 4, 2), (SHORT, 3, 1)])
        if c["frames"] * 3 <= most and rng.random() < 0.2:
            c["views"] = rng.choice([2, 3])
    elif kind == "light":
        c["side_hi"] = min(c["side_hi"], 257)
        c["side_lo"] = min(c["side_lo"], c["side_hi"])
        c["sets"] = rng.randint(1, 4)
        c["frames"] = _log_int(rng, 5, 160)
    elif kind == "sky":
        c["frames"] = rng.randint(1, 4)
        c["side_hi"] = min(c["side_hi"], 301)
        c.update(ncol=rng.randint(20, 90), nrow=rng.randint(20, 90), resample=rng.choice([BILINEAR, CUBICCONV]))
        c["fit_scale"] = 1.3 * c["side_hi"] / min(c["ncol"], c["nrow"])
    elif kind in ("fit", "serve"):
        c["side_hi"] = min(c["side_hi"], 201)
        c["frames"] = rng.randint(1, 6)
        c.update(dict(vertices=rng.randint(0, 4)) if kind == "fit" else
                 dict(workloads=rng.randint(1, 4), requests=rng.randint(8, 40)))
        c["images"] = False
    c["side_lo"] = min(c["side_lo"], c["side_hi"])
    if c["images"]:
        c["frames"] = min(c["frames"], 12)
    return c


# ------------------------------------------------------------------ the inputs

@functools.lru_cache(None)
def _mesh(octa, rings, per):
    return synth.octa_sphere(octa) if octa else synth.ring_sphere(rings, per)


def _model(case, seed):
    """A triaxial body with radial deviations of a few per cent, smooth on ring meshes and rough on octahedral ones."""
    dirs, fv = _mesh(case["octa"], case["rings"], case["per"])
    rng = np.random.default_rng([seed, 1])
    if case["octa"]:
        dev = 0.03 * rng.standard_normal(len(dirs))
    else:
        basis = synth._real_sph_harm_basis(dirs, 6)
        dev = basis @ rng.standard_normal(basis.shape[1])
        dev *= 0.04 / math.sqrt((dev * dev).mean())
    return synth.make_model(dirs, fv, 1.0 + np.clip(dev, -0.1, 0.1), name="body")


def _params(case):
    return synth.eval_params(pos_smooth=1 if case["smooth"] else 0, nsinc2=case["nsinc2"])


def _radar_law(kind):
    law = synth.radar_cosine()
    if kind != 1:
        law.type, law.diff_R, law.diff_C = kind, 0.08, 1.3
        law.qs_R, law.qs_C, law.qs_cos_cutoff = 0.05, 4.0, math.cos(math.radians(60.0))
    return law


def _turn(frames, seed):
    """Rotation phases from the seed (sizes come from the case alone)."""
    pole = synth.ecl_dir(30.0, 60.0)
    for fr, phase in zip(frames, np.random.default_rng([seed, 2]).uniform(0.0, 2 * math.pi, len(frames))):
        cd.fill9(fr.ae, synth.body_matrix(pole, float(phase)))


def _datasets(case, seed):
    """The case's datasets without observations: (delay-Doppler, Doppler, lightcurve, sky) sets."""
    sides, k = (case["side_lo"], case["side_hi"]), case["kind"]
    if k in ("radar", "fit", "serve"):
        ds = synth.batched_dataset(case["frames"], sides, (case["ndel_lo"], case["ndel_hi"]),
                                   (case["ndop_lo"], case["ndop_hi"]), seed=case["layout"], radius=1.15,
                                   codemethod=case["code"], spb=case["spb"], stride=case["stride"],
                                   law=_radar_law(case["law"]))
        _turn(ds.frames, seed)
        if case["views"] > 1:
            # views a few minutes apart; the epoch view is rendered last
            nv, omega, pole = case["views"], 2 * math.pi / 0.25, synth.ecl_dir(30.0, 60.0)
            ds.views = []
            phases = np.random.default_rng([seed, 2]).uniform(0.0, 2 * math.pi, len(ds.frames))
            for f, fr in enumerate(ds.frames):
                row = []
                for v in range(1, nv):
                    w = cd.DeldopFrame.from_buffer_copy(fr)
                    cd.fill9(w.ae, synth.body_matrix(pole, float(phases[f]) + omega * 0.004 * v))
                    row.append(w)
                ds.views.append(row + [fr])
        return [ds], [], [], []
    if k == "doppler":
        ds = synth.doppler_dataset(case["frames"], sides, (case["ndop_lo"], case["ndop_hi"]), seed=case["layout"],
                                   radius=1.25, law=_radar_law(case["law"]))
        _turn(ds.frames, seed)
        return [], [ds], [], []
    if k == "light":
        sets = [synth.lightcurve_dataset(case["frames"], sides, seed=case["layout"], set_index=s, radius=1.15,
                                         law_type=(KAASALAINEN, LOMMEL, LAMBERT, KAASALAINEN)[s])
                for s in range(case["sets"])]
        pole = synth.ecl_dir(30.0, 60.0)
        for s, ds in enumerate(sets):
            p0 = float(np.random.default_rng([seed, 2, s]).uniform(0.0, 2 * math.pi))
            for i, pt in enumerate(ds.points):
                cd.fill9(pt.ae, synth.body_matrix(pole, p0 + 2 * math.pi * (ds.x[i] - ds.x[0]) / 0.25))
        return [], [], sets, []
    ds = synth.poset_dataset(case["frames"], None, None, pos_n=case["side_hi"] // 2, ncol=case["ncol"],
                             nrow=case["nrow"], fit_scale=case["fit_scale"], resample=case["resample"], radius=1.3,
                             seed=case["layout"] % 1000, law_type=KAASALAINEN)
    pole = synth.ecl_dir(30.0, 60.0)
    for fr, ph in zip(ds.frames, np.random.default_rng([seed, 2]).uniform(0.0, 2 * math.pi, len(ds.frames))):
        fr["ae"] = synth.body_matrix(pole, float(ph))
    return [], [], [], [ds]


def _observe(case, seed, model, sets):
    """Fills the sets' observations: the true model's images scaled to a peak of 20 with unit noise (radar, sky),
    brightnesses with 1 % noise (lightcurves)."""
    rng = np.random.default_rng([seed, 3])
    dds, dops, lcs, skies = sets
    body = _Body(model, np.ones(3))
    for ds in dds + dops + skies:
        fits = _radar_fits(body, ds, _params(case)) if ds not in skies else _sky_fits(body, ds, _params(case))[0]
        for f, fit in enumerate(fits):
            fit = fit.cpu().numpy().ravel()
            ds.obs[ds.offsets[f]:ds.offsets[f + 1]] = 20.0 * fit / max(fit.max(), 1e-300) + rng.standard_normal(fit.size)
    for ds in lcs:
        y = _light_y(body, ds, _params(case))
        ds.obs = y * (1.0 + 0.01 * rng.standard_normal(len(y)))
        ds.oneovervar = 1.0 / (0.01 * ds.obs) ** 2
        ds.bind()


def _trials(case, seed):
    """Trial scale factors: one per evaluation, or one per request."""
    n = case["requests"] if case["kind"] == "serve" else 1
    return 1.0 + 0.02 * np.random.default_rng([seed, 4]).uniform(-1.0, 1.0, (n, 3))


def prepare(case, seed):
    model = _model(case, seed)
    sets = _datasets(case, seed)
    _observe(case, seed, model, sets)
    dds, dops, lcs, skies = sets
    st = {"case": case, "form": eng.FORMS[case["form"]], "trials": [[float(v) for v in t] for t in _trials(case, seed)],
          "sets": sets, "images": case["images"]}
    if case["kind"] == "serve":
        st["server"] = eng.Server(hbm_budget_bytes=8 << 30, max_slots=8)
        loads = [("", model, [synth.frame_prefix(dds[0], n)], []) for n in _loads(case)]
        eng.register_workloads(st["server"], loads, _params(case), st["form"])
        st["requests"] = [(i % len(loads), 0.0, tuple(t)) for i, t in enumerate(st["trials"])]
        return st
    st["engine"] = eng.make_engine(model, _params(case), dds, lcs, dopplers=dops, posets=skies)
    if case["kind"] == "fit":
        st["steps"] = _steps(case, seed, model)
        st["r0"] = {i: float(model.r[i]) for what, i, _ in st["steps"] if what == "r"}
    return st


def _steps(case, seed, model):
    """Line-search trials: three values of each parameter about its start, ("scale", j, value) or ("r", vertex, value);
    a parameter keeps its last trial value while the next ones move."""
    rng = np.random.default_rng([seed, 5])
    params = [("scale", j, 1.0, 0.02) for j in range(3)]
    params += [("r", int(i), float(model.r[i]), 0.02) for i in np.linspace(3, model.nv - 4, case["vertices"]).astype(int)]
    return [(k, i, float(v0 + step * x)) for k, i, v0, step in params for x in rng.uniform(-1.0, 1.0, 3)]


def _loads(case):
    """Frames of each of the server's workloads: 1 .. frames."""
    n = case["workloads"]
    return [max(1, round(case["frames"] * (w + 1) / n)) for w in range(n)]


# --------------------------------------------------------------------- a pass

def run(state):
    kind, form = state["case"]["kind"], state["form"]
    if kind == "serve":
        res, _ = state["server"].run(state["requests"])
        return {"chi2": np.array([r["chi2"] for r in res], dtype=_dtype(state["case"])),
                "objective": np.array([r["objective"] for r in res], dtype=_dtype(state["case"]))}
    e = state["engine"]
    for j in range(3):
        e.set_scale(j, state["trials"][0][j])
    if kind == "fit":
        objective = []
        for i, r in state["r0"].items():
            e.set_vertex_r(i, r)
        for what, i, value in state["steps"]:
            (e.set_scale if what == "scale" else e.set_vertex_r)(i, value)
            objective.append(e.evaluate(form)["objective"])
        return {"objective": np.array(objective, dtype=_dtype(state["case"])), "summary": e.evaluate(form)}
    out = {"summary": e.evaluate(form)}
    if state["case"]["seen"] or kind == "light":
        out["seen"] = e.seen()                     # the facets that the data constrain
    if kind == "light":
        for s, ds in enumerate(state["sets"][2]):
            c = e.lghtcrv(s, ds)
            out["y%d" % s], out["fit%d" % s], out["chi2_%d" % s] = c["y"], c["fit"], c["chi2"]
    elif kind == "sky":
        for f in range(state["case"]["frames"]):
            fit, sky, r = e.poset(0, f)
            out["fit%d" % f], out["sky%d" % f], out["chi2_%d" % f] = fit, sky, r["chi2"]
    elif state["images"]:
        # the FP32 form's images are single precision on the device
        for f in range(state["case"]["frames"]):
            out["fit%d" % f] = e.fit(f).astype(_dtype(state["case"]), copy=False)
        res = e.results()
        for k in ("o2", "m2", "om", "cal", "chi2"):
            out[k] = np.array([r[k] for r in res], dtype=_dtype(state["case"]))
        for k in ("idellim", "idoplim", "xlim", "ylim"):
            out[k] = np.array([r[k] for r in res])
    return out


def _dtype(case):
    return np.float32 if case["form"] == "batched_fp32" else np.float64


# ---------------------------------------------------- what a pass cannot do without

def work(case):
    """Bytes: the model and the trial read, each observed image and its 1/variance read, each fit value written, and
    for lightcurve and sky views the depth and facet maps of posmask's two renderings written and read once.
    Operations: 60 per visible facet and view (transform, culling, edge terms), 40 per covered pixel (coverage
    test and depth of its facet, normal) and 12 per delay-Doppler bin that it adds to."""
    model_nf = 8 * 4 ** case["octa"] if case["octa"] else 2 * case["rings"] * case["per"]
    nv = model_nf // 2 + 2
    s = 4 if case["form"] == "batched_fp32" else 8

    def one(k, prefix=None):
        dds, dops, lcs, skies = _datasets(dict(case, kind=k), 0)
        pix, views, img = 0, 0, 0
        for ds in dds + dops:
            for fr in ds.frames[:prefix]:
                n = case["views"] if k != "doppler" else 1
                pix += n * (2 * fr.pos_n + 1) ** 2
                views += n
                img += getattr(fr, "ndel", 1) * fr.ndop
        lpix = sum(2 * (2 * p.pos_n + 1) ** 2 for ds in lcs for p in ds.points)
        lpix += sum(2 * (2 * f["pos_n"] + 1) ** 2 for ds in skies for f in ds.frames)
        views += sum(2 * len(ds.points) for ds in lcs) + sum(2 * len(ds.frames) for ds in skies)
        img += sum(f["ncol"] * f["nrow"] for ds in skies for f in ds.frames)
        by = nv * 56 + model_nf * 12 + img * (16 + s) + lpix * 24
        fl = views * model_nf // 2 * 60 + 0.5 * (pix + lpix) * 40 + 0.5 * pix * 14 * 12
        return np.array([by, fl])

    k = case["kind"]
    if k == "serve":
        loads = _loads(case)
        w = sum(one("radar", loads[i % len(loads)]) for i in range(case["requests"]))
    elif k == "fit":
        w = (3 * (3 + case["vertices"]) + 1) * one("radar")
    else:
        w = one(k)
    return {"bytes": float(w[0]), "flops": float(w[1])}


# --------------------------------------------------------- FP64 values in plain torch

def exact(case, seed):
    model = _model(case, seed)
    sets = _datasets(case, seed)
    _observe(case, seed, model, sets)
    dds, dops, lcs, skies = sets
    par = _params(case)
    trials = _trials(case, seed)
    if case["kind"] == "serve":
        loads, chi, obj = _loads(case), [], []
        for i, sc in enumerate(trials):
            ds = synth.frame_prefix(dds[0], loads[i % len(loads)])
            c = float(sum(t["chi2"] for t in _radar_terms(_Body(model, sc), ds, par)))
            chi.append(c)
            obj.append(c / sum(fr.dof for fr in ds.frames))
        return {"chi2": np.array(chi), "objective": np.array(obj)}
    if case["kind"] == "fit":
        scale, chi = np.array(trials[0]), []
        for what, i, value in _steps(case, seed, model):
            if what == "scale":
                scale[i] = value
            else:
                model.r[i] = value
            chi.append(float(sum(t["chi2"] for t in _radar_terms(_Body(model, scale), dds[0], par))))
        dof = float(sum(fr.dof for fr in dds[0].frames))
        return {"objective": np.array(chi) / dof, "summary": {"chi2": chi[-1], "dof": dof}}
    body = _Body(model, trials[0])
    out, chi2, dof = {}, {"dd": 0.0, "lc": 0.0, "ps": 0.0}, 0.0
    for ds in dds + dops:
        terms = _radar_terms(body, ds, par)
        chi2["dd"] += sum(t["chi2"] for t in terms)
        dof += sum(fr.dof for fr in ds.frames)
        if case["images"]:
            for f, t in enumerate(terms):
                out["fit%d" % f] = t["fit"]
            for k in ("o2", "m2", "om", "cal", "chi2"):
                out[k] = np.array([t[k] for t in terms])
    for s, ds in enumerate(lcs):
        y = _light_y(body, ds, par)               # observed at the calculated epochs: the spline passes through y
        c = _chi2(y, ds.obs, ds.oneovervar)["chi2"]
        out["y%d" % s], out["fit%d" % s], out["chi2_%d" % s] = y, y.copy(), c
        chi2["lc"] += c
        dof += ds.set.dof
    for ds in skies:
        fits, sky = _sky_fits(body, ds, par)
        for f, fit in enumerate(fits):
            a, b = ds.offsets[f], ds.offsets[f + 1]
            fit = fit.cpu().numpy()
            c = _chi2(fit.ravel(), ds.obs[a:b], ds.oneovervar[a:b])["chi2"]
            out["fit%d" % f], out["sky%d" % f], out["chi2_%d" % f] = fit, sky[f].cpu().numpy(), c
            chi2["ps"] += c
            dof += ds.frames[f]["dof"]
    total = float(sum(chi2.values()))
    out["summary"] = {"chi2": total, "dof": float(dof), "chi2_deldop": float(chi2["dd"]),
                      "chi2_lghtcrv": float(chi2["lc"]), "chi2_poset": float(chi2["ps"])}
    return out


_DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
_SMALL, _HUGE, _AU, _KM2US, _KM2HZ = 1.0e-10, 1.0e20, 1.4959787061e8, 6.67128190396304, 7.72139109254982e-5


def _dev(x, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device=_DEV)


class _Body:
    """The realized model: vertices, facet normals, vertex normals (realize_mod)."""

    def __init__(self, m, scale):
        x = np.asarray(scale)[None, :] * (m.u * m.r[:, None] + m.a)
        p = x[m.fv]
        a, b = p[:, 1] - p[:, 0], p[:, 2] - p[:, 1]
        fn = _normalize(np.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                                  a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], axis=1))
        vn = np.zeros_like(x)
        np.add.at(vn, np.repeat(np.arange(m.nv), np.diff(m.af_ptr)), fn[m.af_idx])
        self.x, self.fn, self.vn, self.fv = _dev(x), _dev(fn), _dev(_normalize(vn)), _dev(m.fv, torch.int64)


def _normalize(c):
    n = np.sqrt(c[:, 0] * c[:, 0] + c[:, 1] * c[:, 1] + c[:, 2] * c[:, 2])[:, None]
    return np.where(n != 0.0, c / np.where(n != 0.0, n, 1.0), c)


def _mat(a):
    return np.array(a, dtype=np.float64).reshape(3, 3)


def _mul_bt(b, a):
    """b a^T with the sums in index order."""
    t = b[:, None, 0] * a[None, :, 0]
    for k in (1, 2):
        t = t + b[:, None, k] * a[None, :, k]
    return t


def _rot(oa, v):
    """Rows of oa (..., 3, 3) times v (..., 3), the sums in index order."""
    return torch.stack([oa[..., r, 0] * v[..., 0] + oa[..., r, 1] * v[..., 1] + oa[..., r, 2] * v[..., 2]
                        for r in range(3)], dim=-1)


def _render(body, views):
    """posvis for views (oa, half width n, km per pixel, smooth, sun direction or None): per view (facet, depth, cos e,
    cos i) images, side x side. Every operation is posvis's, in its order; no sums are fused."""
    out, start = [], 0
    while start < len(views):
        stop, load = start, 0
        while stop < len(views) and (stop == start or load < 1.2e7):
            load += 2 * (2 * views[stop][1] + 1) ** 2 + body.fv.shape[0]
            stop += 1
        out += _render_some(body, views[start:stop])
        start = stop
    return out


def _render_some(body, views):
    oa = _dev(np.stack([v[0] for v in views]))
    n = _dev([v[1] for v in views], torch.int64)
    km = _dev([v[2] for v in views])
    smooth = _dev([bool(v[3]) for v in views], torch.bool)
    bistatic = _dev([v[4] is not None for v in views], torch.bool)
    sun = _dev([v[4] if v[4] is not None else (0.0, 0.0, 1.0) for v in views])
    side = 2 * n + 1
    base = torch.cumsum(side * side, 0) - side * side
    total = int((side * side).sum())
    xt = _rot(oa[:, None], body.x[None])                              # [view, vertex, 3]
    nz = oa[:, None, 2, 0] * body.fn[None, :, 0] + oa[:, None, 2, 1] * body.fn[None, :, 1] \
        + oa[:, None, 2, 2] * body.fn[None, :, 2]
    vi, fi = torch.nonzero(nz > 0.0, as_tuple=True)                   # by view, then facet
    p = xt[vi[:, None], body.fv[fi]]                                  # [pair, corner, 3]
    kv, nn = km[vi], n[vi]

    def span(c):
        lo = torch.floor(p[..., c].amin(1) / kv - _SMALL + 0.5).long().clamp_min(-nn)
        hi = torch.floor(p[..., c].amax(1) / kv + _SMALL + 0.5).long().clamp_max(nn)
        return lo, hi
    i1, i2 = span(0)
    j1, j2 = span(1)
    area = (i2 - i1 + 1).clamp_min(0) * (j2 - j1 + 1).clamp_min(0)
    q = torch.repeat_interleave(torch.arange(len(area), device=_DEV), area)
    k = torch.arange(len(q), device=_DEV) - (torch.cumsum(area, 0) - area)[q]
    w = (j2 - j1 + 1)[q]
    pi, pj = i1[q] + torch.div(k, w, rounding_mode="floor"), j1[q] + k % w
    p0, p1, p2 = p[:, 0], p[:, 1], p[:, 2]
    A, B, C, D = p2[:, 1] - p1[:, 1], p2[:, 0] - p1[:, 0], p1[:, 0] - p0[:, 0], p1[:, 1] - p0[:, 1]
    E, F = p1[:, 2] - p0[:, 2], p2[:, 2] - p1[:, 2]
    den = 1.0 / (C * A - B * D)
    dx, dy = pi * km[vi[q]] - p0[q, 0], pj * km[vi[q]] - p0[q, 1]
    s = (dx * A[q] - B[q] * dy) * den[q]
    t = (C[q] * dy - dx * D[q]) * den[q]
    ok = (s >= -_SMALL) & (s <= 1.0 + _SMALL) & (t >= -_SMALL) & (t <= s + _SMALL)
    q, s, t, pi, pj = q[ok], s[ok], t[ok], pi[ok], pj[ok]
    z = p0[q, 2] + s * E[q] + t * F[q]
    v, f = vi[q], fi[q]
    pix = base[v] + (pi + n[v]) * side[v] + pj + n[v]
    zmax = torch.full((total,), -_HUGE, dtype=torch.float64, device=_DEV).scatter_reduce_(0, pix, z, "amax")
    top = z == zmax[pix]
    none = body.fv.shape[0]
    fac = torch.full((total,), none, dtype=torch.int64, device=_DEV).scatter_reduce_(0, pix[top], f[top], "amin")
    cose = torch.zeros(total, dtype=torch.float64, device=_DEV)
    cosi = torch.zeros_like(cose)

    def shade(i):
        """Sets cos e and cos i of the pixels of pairs i from those pairs; true where the normal faces the viewer."""
        c, sm = body.fv[f[i]], smooth[v[i]][:, None]
        q0, q1, q2 = body.vn[c[:, 0]], body.vn[c[:, 1]], body.vn[c[:, 2]]
        m = torch.where(sm, q0 + s[i, None] * (q1 - q0) + t[i, None] * (q2 - q1), body.fn[f[i]])
        r = _rot(oa[v[i]], m)
        faces = (r[:, 2] > 0.0) | ~sm[:, 0]
        norm = torch.sqrt(r[:, 0] * r[:, 0] + r[:, 1] * r[:, 1] + r[:, 2] * r[:, 2])[:, None]
        r = torch.where(sm & (norm != 0.0), r / norm, r)
        ci = r[:, 0] * sun[v[i], 0] + r[:, 1] * sun[v[i], 1] + r[:, 2] * sun[v[i], 2]
        ci = torch.where(bistatic[v[i]], ci, torch.zeros_like(ci))
        ce = torch.where(bistatic[v[i]] & (ci <= 0.0), torch.zeros_like(ci), r[:, 2])
        up = faces & (r[:, 2] > 0.0)
        cose[pix[i[up]]], cosi[pix[i[up]]] = ce[up], ci[up]
        return faces
    win = torch.nonzero(top & (f == fac[pix]))[:, 0]
    limb = pix[win[~shade(win)]]
    if len(limb):
        # the last winner's normal faces away: cos e stays that of the last earlier winner whose normal faces the
        # viewer, found by walking the pixel's facets in index order
        at = torch.zeros(total, dtype=torch.bool, device=_DEV)
        at[limb] = True
        i = torch.nonzero(at[pix])[:, 0]
        i = i[torch.argsort(pix[i], stable=True)]                    # by pixel, then facet
        first = torch.ones(len(i), dtype=torch.bool, device=_DEV)
        first[1:] = pix[i[1:]] != pix[i[:-1]]
        pos = torch.arange(len(i), device=_DEV)
        rank = pos - torch.cummax(torch.where(first, pos, torch.zeros_like(pos)), 0)[0]
        zz = torch.full((total,), -_HUGE, dtype=torch.float64, device=_DEV)
        for step in range(int(rank.max()) + 1):
            now = i[rank == step]
            now = now[z[now] > zz[pix[now]]]
            zz[pix[now]] = z[now]
            shade(now)
    fac[fac == none] = -1
    res = []
    for k in range(len(views)):
        a, sd = int(base[k]), int(side[k])
        res.append([x[a:a + sd * sd].view(sd, sd) for x in (fac, zmax, cose, cosi)])
    return res


def _radlaw(L, c):
    diff = L.diff_R * (L.diff_C + 1) * c ** (2 * L.diff_C - 1)
    inside = c >= L.qs_cos_cutoff
    s = torch.where(inside, c, torch.ones_like(c))
    gauss = L.qs_R * L.qs_C * torch.exp(-L.qs_C * (1 / (s * s) - 1)) / s ** 5
    hag = 0.5 * L.qs_R * L.qs_C * (s ** 4 + L.qs_C * (1 - s * s)) ** -1.5 / s
    cos = L.qs_R * (L.qs_C + 1) * s ** (2 * L.qs_C - 1)
    qs = {1: 0 * s, 2: gauss, 3: hag, 4: cos, 5: gauss, 6: hag, 7: cos}[L.type]
    return torch.where(inside, qs, torch.zeros_like(qs)) + (diff if L.type in (1, 5, 6, 7) else 0.0)


def _sinc2(x):
    a = math.pi * x.abs()
    return torch.where(a > 1.0e-4, (torch.sin(a) / a.clamp_min(1e-300)) ** 2, torch.ones_like(a))


def _tri(x):
    return (1.0 - x.abs()).clamp_min(0.0)


def _radar_fits(body, ds, par):
    """pos2deldop / pos2doppler: the fit image of each frame, [ndel, ndop]."""
    views = getattr(ds, "views", None) or [[fr] for fr in ds.frames]
    flat = [fr for row in views for fr in row]
    maps = _render(body, [(_mul_bt(_mat(fr.oe), _mat(fr.ae)), fr.pos_n, fr.km_per_pixel, par.pos_smooth, None)
                          for fr in flat])
    fits, k = [], 0
    for row in views:
        nd = getattr(row[-1], "ndel", 1)
        img = torch.zeros(nd * row[-1].ndop, dtype=torch.float64, device=_DEV)
        for fr in row:
            _synthesize(img, fr, ds.set, par, maps[k], len(row))
            k += 1
        fits.append(img.view(nd, row[-1].ndop))
    return fits


def _synthesize(img, fr, S, par, pos, nviews):
    doppler = not hasattr(fr, "ndel")
    code, spb, stride = (LONG_ORIG, 1, 1) if doppler else (S.codemethod, S.spb, S.stride)
    _, z, cose, _ = pos
    n, km, ns, width = fr.pos_n, fr.km_per_pixel, par.nsinc2, par.sinc2width
    oe, spin = _mat(fr.oe), np.array(list(fr.spin))
    w = oe[:, 0] * spin[0] + oe[:, 1] * spin[1] + oe[:, 2] * spin[2]
    per_bin = S.dop_per_bin if doppler else S.dop_per_pixel
    fact = S.dopscale * _KM2HZ * km * S.Ftx / per_bin
    ax, ay = -w[1] * fact, w[0] * fact
    sos = spb // stride
    c1, c2 = ((3 * spb - 1) / (2.0 * stride), (spb - 1) / (2.0 * stride)) if code != LONG_ORIG else (float(sos), 0.0)
    lit = torch.nonzero(cose > 0.0)
    c, zl = cose[lit[:, 0], lit[:, 1]], z[lit[:, 0], lit[:, 1]]
    x, y = (lit[:, 0] - n).double(), (lit[:, 1] - n).double()
    if doppler:
        delay = torch.ones_like(zl)
    else:
        delay = zl * (-_KM2US / S.del_per_pixel) + (fr.delcom_vig + fr.deloff)
    dop = ax * x + ay * y + (fr.dopcom_vig + fr.dopoff + 0.0)
    xi, yi = ax / ns, ay / ns
    far = (ns - 1) * (abs(xi) + abs(yi)) / 2
    e1, e2 = torch.floor(delay - c1).long() + 1, torch.ceil(delay + c1).long() - 1
    o1, o2 = torch.floor(dop - far + 1 - width / 2.0).long(), torch.floor(dop + far + width / 2.0).long()
    ndel = 1 if doppler else fr.ndel
    ok = (e1 >= 1) & (e2 <= ndel) & (o1 >= 1) & (o2 <= fr.ndop) & (e2 - e1 + 1 <= 100)
    delay, dop, e1, e2, o1, o2, c = (v[ok] for v in (delay, dop, e1, e2, o1, o2, c))
    amp = _radlaw(S.law, c) * km * km / nviews
    if code == SHORT:
        amp = amp * _sinc2((dop - fr.dopDC_vig) / S.dopfftlen)
    if not len(c):
        return

    def rows(e):
        d = delay - e
        if code == LONG_ORIG:
            return _tri(d / sos) ** 2
        if spb == 1:
            return _tri(d) ** 2
        arg, r = (delay - (e - c2)) / sos, torch.zeros_like(d)
        if spb == 2:
            return (_tri(arg) + _tri(arg - 0.5)) ** 2 / 4
        m1 = torch.floor((d - c2) * stride).clamp_min(0)
        m2 = torch.ceil((d + c1) * stride).clamp_max(spb) - 1
        for m in range(spb):
            r = r + torch.where((m >= m1) & (m <= m2), _tri(arg - m / spb), torch.zeros_like(r))
        return r * r / spb ** 2

    def cols(o):
        if ns == 1:
            return _sinc2(dop - o)
        left = dop - (ns - 1) * (xi + yi) / 2 - o
        return sum(_sinc2(left + i * yi + j * xi) for i in range(ns) for j in range(ns)) / ns ** 2
    dr = [(e1 + r, torch.where(e1 + r <= e2, rows(e1 + r), 0.0)) for r in range(int((e2 - e1).max()) + 1)]
    dc = [(o1 + k, torch.where(o1 + k <= o2, cols(o1 + k), 0.0)) for k in range(int((o2 - o1).max()) + 1)]
    amp = amp / (sum(v for _, v in dr) * sum(v for _, v in dc))
    for e, we in dr:
        for o, wo in dc:
            inside = (e <= e2) & (o <= o2)
            img.index_add_(0, ((e - 1) * fr.ndop + o - 1)[inside], (amp * we * wo)[inside])


def _chi2(fit, obs, oov):
    o2, m2, om = float((obs * obs * oov).sum()), float((fit * fit * oov).sum()), float((fit * obs * oov).sum())
    cal = om / m2 if om > 0.0 else 1.0e-40
    return {"o2": o2, "m2": m2, "om": om, "cal": cal, "chi2": o2 - 2 * cal * om + cal * cal * m2}


def _radar_terms(body, ds, par):
    out = []
    for f, fit in enumerate(_radar_fits(body, ds, par)):
        a, b = ds.offsets[f], ds.offsets[f + 1]
        fit = fit.cpu().numpy().ravel()
        out.append(dict(_chi2(fit, ds.obs[a:b], ds.oneovervar[a:b]), fit=fit))
    return out


def _brightness(body, points, law, par):
    """posvis from the observer and the sun, posmask, apply_photo: the brightness image of each point."""
    views = []
    for pt in points:
        oe, se, ae = _mat(pt["oe"]), _mat(pt["se"]), _mat(pt["ae"])
        us = se[2]
        us = oe[:, 0] * us[0] + oe[:, 1] * us[1] + oe[:, 2] * us[2]
        views.append((_mul_bt(oe, ae), pt["pos_n"], pt["km_per_pixel"], par.pos_smooth, us))
        views.append((_mul_bt(se, ae), pt["pos_n"], pt["km_per_pixel"], 0, None))
    imgs, maps = [], _render(body, views)
    for k, pt in enumerate(points):
        (fac, z, cose, cosi), (fill, zill, _, _) = maps[2 * k], maps[2 * k + 1]
        n, km = pt["pos_n"], pt["km_per_pixel"]
        side = 2 * n + 1
        so = _mul_bt(_mat(pt["se"]), _mat(pt["oe"]))
        i, j = torch.nonzero(cose != 0.0, as_tuple=True)
        xi, yi, zi = (i - n).double() * km, (j - n).double() * km, z[i, j]
        x = [so[r, 0] * xi + so[r, 1] * yi + so[r, 2] * zi for r in range(3)]
        i0, j0 = x[0] * (1 / km), x[1] * (1 / km)
        im, jm = (torch.trunc(torch.where(v < 0.0, v - 0.5, v + 0.5)).long() for v in (i0, j0))
        near = (i0.abs() < n) & (j0.abs() < n)

        def at(a, b):
            inside = (a.abs() <= n) & (b.abs() <= n)
            v = zill.reshape(-1)[((a + n).clamp(0, side - 1)) * side + (b + n).clamp(0, side - 1)]
            return torch.where(inside, v, torch.full_like(v, -_HUGE))
        big = -0.99 * _HUGE
        fi = torch.where(near, fill.reshape(-1)[((im + n).clamp(0, side - 1)) * side + (jm + n).clamp(0, side - 1)],
                         torch.full_like(im, -1))
        test = near & (at(im, jm) > big) & (fac[i, j] != fi)
        i1, j1 = torch.floor(i0).long(), torch.floor(j0).long()
        q = [at(i1, j1), at(i1 + 1, j1), at(i1 + 1, j1 + 1), at(i1, j1 + 1)]
        u, w = i0 - i1, j0 - j1
        four = (1 - u) * (1 - w) * q[0] + u * (1 - w) * q[1] + u * w * q[2] + (1 - u) * w * q[3]
        one = at(im, jm)
        for d0, m, step in ((i0, im, (1, 0)), (j0, jm, (0, 1))):
            sg = torch.where(d0 >= m, 1, -1)
            a, b = (at(im + e * sg * step[0], jm + e * sg * step[1]) for e in (1, -1))
            dist, mid = (d0 - m).abs(), at(im, jm)
            one = one + torch.where(a > big, dist * (a - mid), torch.where(b > big, -dist * (b - mid),
                                                                           torch.zeros_like(dist)))
        depth = torch.where((q[0] > big) & (q[1] > big) & (q[2] > big) & (q[3] > big), four, one)
        shadow = test & (depth - x[2] > par.mask_tol)
        ce, ci = cose[i, j], cosi[i, j]
        lit = ~shadow & (ce > 0.0) & (ci > 0.0)
        f0 = (km / _AU) ** 2.0
        if law.type == LAMBERT:
            b = f0 * (law.R / math.pi) * ci
        elif law.type == LOMMEL:
            b = f0 * (law.R / (4 * math.pi)) * ci / (ci + ce)
        else:
            ph = law.A0 * math.exp(-pt["solar_phase"] / law.D) + law.k * pt["solar_phase"] + 1
            b = f0 * ci * ((1 - law.wt) * ph * law.R / (4 * math.pi) / (ci + ce) + law.wt * ph * law.R / math.pi)
        img = torch.zeros(side, side, dtype=torch.float64, device=_DEV)
        img[i[lit], j[lit]] = b[lit]
        imgs.append(img)
    return imgs


def _light_y(body, ds, par):
    pts = [{k: getattr(p, k) for k in ("pos_n", "km_per_pixel", "ae", "oe", "se", "solar_phase")} for p in ds.points]
    return torch.stack([b.sum() for b in _brightness(body, pts, ds.set.law, par)]).cpu().numpy()


def _sky_fits(body, ds, par):
    """calc_poset: the brightness images resampled onto the fit grids. Returns (fit images, brightness images)."""
    skies = _brightness(body, ds.frames, ds.law, par)
    fits = []
    for fr, sky in zip(ds.frames, skies):
        n, nc, nr = fr["pos_n"], fr["ncol"], fr["nrow"]
        fact = fr["fit_km_per_pixel"] / fr["km_per_pixel"]
        x0 = -((fr["colcom_vig"] - (nc + 1) / 2.0) + fr["xoff"]) * fact
        y0 = -((fr["rowcom_vig"] - (nr + 1) / 2.0) + fr["yoff"]) * fact
        ca, sa = math.cos(-fr["northangle"]), math.sin(-fr["northangle"])
        i = (torch.arange(nc, device=_DEV, dtype=torch.float64) - (nc - 1) / 2.0)[:, None]
        j = (torch.arange(nr, device=_DEV, dtype=torch.float64) - (nr - 1) / 2.0)[None, :]
        x, y = x0 + fact * (i * ca + j * sa), y0 + fact * (-i * sa + j * ca)
        ix, iy = torch.floor(x).long(), torch.floor(y).long()
        u, w = x - ix, y - iy

        def at(a, b):
            return sky.reshape(-1)[(a + n).clamp(0, 2 * n) * (2 * n + 1) + (b + n).clamp(0, 2 * n)]
        if ds.resample == BILINEAR:
            v = (1 - u) * (1 - w) * at(ix, iy) + u * (1 - w) * at(ix + 1, iy) + u * w * at(ix + 1, iy + 1) \
                + (1 - u) * w * at(ix, iy + 1)
            v = torch.where((ix >= -n) & (ix < n) & (iy >= -n) & (iy < n), v, torch.zeros_like(v))
        else:
            def kern(d):
                d = d.abs()
                return torch.where(d < 1, d ** 3 - 2 * d ** 2 + 1, torch.where(d < 2, -(d ** 3 - 5 * d ** 2 + 8 * d - 4),
                                                                               torch.zeros_like(d)))
            v = sum(kern(b - w) * sum(kern(a - u) * at(ix + a, iy + b) for a in range(-1, 3)) for b in range(-1, 3))
            v = torch.where((ix > -n) & (ix < n - 1) & (iy > -n) & (iy < n - 1), v, torch.zeros_like(v)).clamp_min(0.0)
        fits.append(v)
    return fits, skies
