"""LM steps by a team of warps (a CTA per peak) and by one warp per peak.

Which of the two a sweep of FP32 Gaussians takes depends on how many peaks
are RUNNING and how densely they lie, so the results must not: a batch large
enough for the warp steps gives, bit for bit, what its frames give alone
(team steps).  A team has a thread per ROI pixel, so its remainders come with
the ROI's size: both engines are held to the FP64 oracle at the usual bar
over ROI sizes whose pixel counts lie on both sides of the multiples of 32
and beyond a team's 128 threads."""
import os
import sys

import numpy
import pytest

from gpu_helpers import concat, fit_workload_gpu

pytestmark = pytest.mark.gpu

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "storm-analysis_gb300"))

# configuration, fitter arguments
GAUSSIANS = [(0, {}), (1, dict(roi_size=10)), (2, dict(roi_size=10))]


def batch_fit(wl, frames):
    from sa_gb300 import engine
    kw = dict(wl["fitter"])
    model = kw.pop("model")
    fit = engine.BatchFitter(model, (wl["ny"], wl["nx"]), len(frames), rqe=wl["rqe"], scmos_cal=wl["scmos_cal"],
                             precision=32, **kw)
    fit.load(numpy.stack([wl["images"][k] for k in frames]), numpy.stack([wl["backgrounds"][k] for k in frames]),
             [wl["guesses"][k] for k in frames], "hdf5")
    fit.fit(60)
    values, ints = fit.results_fast()
    fit.close()
    return numpy.array(values), numpy.array(ints)


@pytest.mark.parametrize("cfg,kw", GAUSSIANS)
def test_large_batches_give_the_frames_own_results(cfg, kw):
    """120 frames of 400 peaks (48,000 RUNNING peaks of two footprints a
    pixel: warp steps at first, team steps as the peaks converge) against
    the two frames they repeat (team steps throughout)."""
    from sa_gb300 import synth
    wl = synth.make_workload(cfg, frames=2, nx=128, ny=128, seed=17, n_emitters=400)
    wl["fitter"].update(kw)
    one_v, one_i = batch_fit(wl, [0, 1])
    all_v, all_i = batch_fit(wl, [0, 1] * 60)
    assert all_v.shape[0] == 60 * one_v.shape[0]
    assert numpy.array_equal(all_v, numpy.tile(one_v, (60, 1)), equal_nan=True)
    assert numpy.array_equal(all_i, numpy.tile(one_i, (60,) + (1,) * (one_i.ndim - 1)))


@pytest.mark.parametrize("roi", [5, 6, 7, 9, 12, 13, 16, 19, 24])
@pytest.mark.parametrize("cfg", [0, 1])
def test_team_steps_over_roi_sizes(cfg, roi):
    from oracle.oracle import OracleFitter
    from sa_gb300 import parity, synth
    wl = synth.make_workload(cfg, frames=1, nx=96, ny=90, seed=100 + roi, n_emitters=24)
    wl["fitter"]["roi_size"] = roi
    kw = dict(wl["fitter"])
    f = OracleFitter(kw.pop("model"), (90, 96), **kw)
    f.newImage(wl["images"][0])
    f.newBackground(wl["backgrounds"][0])
    f.newPeaks(wl["guesses"][0], "hdf5")
    f.doFit(200)
    ref = {p: f.getPeakProperty(p) for p in ("x", "y", "z", "height", "background", "status", "iterations", "error")}
    f.cleanup(verbose=False)
    for precision in (64, 32):
        st = parity.compare(concat(fit_workload_gpu(wl, [0], precision)), ref)
        assert st["status_agree"] >= 0.999, (precision, st)
        assert parity.within_tolerance(st, min_fraction=0.999), (precision, st)


def wild_workload(cfg, seed, frames=2, n=60):
    """Starts up to 6 px off, some at the frame's edge, heights off by up to
    e^2: trials are rejected by the dozen, and by the check of the margin."""
    from sa_gb300 import synth
    wl = synth.make_workload(cfg, frames=frames, nx=96, ny=90, seed=seed, n_emitters=n)
    rng = numpy.random.default_rng(seed)
    for g in wl["guesses"]:
        m = g["x"].size
        g["x"] = numpy.clip(g["x"] + rng.uniform(-6.0, 6.0, m), 12.0, 84.0)
        g["y"] = numpy.clip(g["y"] + rng.uniform(-6.0, 6.0, m), 12.0, 78.0)
        g["height"] = g["height"] * numpy.exp(rng.uniform(-2.0, 2.0, m))
    return wl


def model_fitter(wl, precision, **extra):
    from sa_gb300 import cubic_fit_c, engine
    kw = dict(wl["fitter"])
    model = kw.pop("model")
    spl = kw.pop("spline", None)
    if spl is not None:
        kw["spline"] = cubic_fit_c.SplinePSF(coeff=spl["coeff"])
    kw.update(extra)
    return engine.BatchFitter(model, (wl["ny"], wl["nx"]), len(wl["images"]), rqe=wl["rqe"],
                              scmos_cal=wl["scmos_cal"], precision=precision, **kw)


def fit_rows(fit, wl, sweeps):
    """Result rows, integers and what each counter rose by."""
    before = fit.counters()
    fit.load(numpy.stack(wl["images"]), numpy.stack(wl["backgrounds"]), wl["guesses"], "hdf5")
    fit.fit(sweeps)
    values, ints = fit.results_fast()
    return numpy.array(values), numpy.array(ints), fit.counters() - before


@pytest.mark.parametrize("cfg,roi", [(3, None), (0, 10), (0, 20), (1, 20), (2, None)])
def test_rejected_trials_do_not_reach_their_successors(cfg, roi):
    """While a team's first warp decides a trial the others prepare its
    write-back; after a rejection it makes the next trial, which may lie
    anywhere.  ROIs of one and several pixels a thread, repeated: one result
    and one set of counters."""
    wl = wild_workload(cfg, 70 + cfg)
    fit = model_fitter(wl, 32, **({} if roi is None else dict(roi_size=roi)))
    assert fit.clib.saSetTailPeaks(fit.h, 0) == 0
    first = fit_rows(fit, wl, 100)
    n_dposv, n_iter, n_lost, n_margin, n_neg_fi, n_neg_height, _, n_non_decr, _ = first[2]
    assert n_margin > 0 and n_neg_height > 0 and n_non_decr > 0
    for _ in range(30):
        again = fit_rows(fit, wl, 100)
        for a, b in zip(first, again):
            assert numpy.array_equal(a, b, equal_nan=True)
    fit.close()


@pytest.mark.parametrize("cfg,precision,per_cta", [(1, 32, 4), (2, 32, 4), (0, 64, 4), (3, 32, 1)])
def test_a_capped_grid_steps_the_same_peaks_at_once(cfg, precision, per_cta):
    """saSetSweepCTAs counts CTAs of a peak per warp: teams of four warps take
    as many peaks at once, teams of eight a peak per CTA, none more than the
    full grid; the results are the uncapped ones."""
    wl = wild_workload(cfg, 60 + cfg)
    rows = []
    full = numpy.zeros(4, dtype=numpy.int32)
    for ctas in (0, 1, 3, 12, 100000):
        fit = model_fitter(wl, precision)
        shape = numpy.zeros(4, dtype=numpy.int32)
        assert fit.clib.saGetSweepShape(fit.h, shape) == -1   # no image yet
        assert fit.clib.saSetSweepCTAs(fit.h, ctas) == 0
        rows.append(fit_rows(fit, wl, 40))
        assert fit.clib.saGetSweepShape(fit.h, shape) == 0
        if ctas == 0:
            full[:] = shape
            assert full[0] == fit.clib.saGetSweepGrid(fit.h) and full[1] == 4
            assert full[3] == (128 if per_cta == 4 else 256)
        else:
            assert shape[0] == min(ctas, full[0]) and shape[1] == full[1]
            assert shape[2] == min(ctas * per_cta, full[2]) and shape[3] == full[3]
        fit.close()
    for r in rows[1:]:
        for a, b in zip(rows[0], r):
            assert numpy.array_equal(a, b, equal_nan=True)


def spline2d_workload(knots, nx, ny, n, seed):
    """Emitters of a measured 2D PSF (the Z model's at focus, knots - 1 px wide)."""
    from sa_gb300 import synth
    rng = numpy.random.default_rng(seed)
    a = numpy.arange(knots) - 0.5 * (knots - 1)
    coef = rng.normal(0.0, 1.0, 6)
    samples = synth._aberrated_psf(a[:, None], a[None, :], 0.0, coef)
    half = 0.5 * (knots - 1)
    x, y = rng.uniform(half + 2, nx - half - 3, n), rng.uniform(half + 2, ny - half - 3, n)
    h = rng.uniform(1000.0, 4000.0, n)
    img = numpy.full((ny, nx), 20.0)
    for i in range(n):
        img += h[i] * synth._aberrated_psf(numpy.arange(nx)[None, :] - x[i], numpy.arange(ny)[:, None] - y[i], 0.0, coef)
    return dict(nx=nx, ny=ny, images=[rng.poisson(img).astype(numpy.float64)], backgrounds=[numpy.full((ny, nx), 20.0)],
                guesses=[dict(x=x + rng.normal(0.0, 0.3, n), y=y + rng.normal(0.0, 0.3, n), z=numpy.zeros(n),
                              background=numpy.full(n, 20.0), height=h * rng.uniform(0.8, 1.2, n))],
                rqe=numpy.ones((ny, nx)), scmos_cal=numpy.zeros((ny, nx)),
                fitter=dict(model="spline2D", spline=dict(coeff=synth.bicubic_coefficients(samples))))


def any_workload(model):
    from sa_gb300 import psf_fft_c, pupil_fn, synth
    if model in ("fft", "pupil"):
        make = synth.fft_workload if model == "fft" else synth.pupil_workload
        wl = make(frames=2, nx=96, ny=90, n_emitters=25, seed=33, **({} if model == "fft" else dict(size=20)))
        fk = wl["fitter"]
        wl["fitter"] = dict(model=model, psf_fft=psf_fft_c.PSFFFT(fk["psf"])) if model == "fft" else dict(
            model=model, pupil_fn=pupil_fn.PupilFunction(pf_data=fk["pf_data"], zmin=-500.0, zmax=500.0))
        rng = numpy.random.default_rng(34)
        for g in wl["guesses"]:
            g["x"] = numpy.clip(g["x"] + rng.uniform(-3.0, 3.0, 25), 12.0, 84.0)
            g["y"] = numpy.clip(g["y"] + rng.uniform(-3.0, 3.0, 25), 12.0, 78.0)
        return wl
    if model == "spline2D":
        wl = spline2d_workload(20, 96, 90, 40, 35)
        wl["guesses"][0]["x"] = numpy.clip(wl["guesses"][0]["x"] + numpy.linspace(-5.0, 5.0, 40), 12.0, 84.0)
        return wl
    wl = wild_workload({"2dfixed": 0, "2d": 0, "3d": 1, "Z": 2, "spline3D": 3}[model], 80)
    wl["fitter"]["model"] = model
    return wl


@pytest.mark.parametrize("model,precision", [("2dfixed", 32), ("2d", 32), ("3d", 32), ("Z", 32), ("spline2D", 32),
                                             ("spline3D", 32), ("2dfixed", 64), ("2d", 64), ("3d", 64), ("Z", 64),
                                             ("spline2D", 64), ("spline3D", 64), ("fft", 64), ("pupil", 64)])
def test_team_and_warp_steps_give_the_same_bits(model, precision):
    """Every model and engine, from starts that reject trials, leave ROIs and
    lose peaks: sweeps and tails by teams against sweeps and tails by warps."""
    wl = any_workload(model)
    rows = []
    shape = numpy.zeros(4, dtype=numpy.int32)
    for on in (1, 0):
        for tail in (0, 8):
            fit = model_fitter(wl, precision)
            assert fit.clib.saSetTeamSteps(fit.h, on) == 0 and fit.clib.saSetTailPeaks(fit.h, tail) == 0
            rows.append(fit_rows(fit, wl, 150))
            assert fit.clib.saGetSweepShape(fit.h, shape) == 0 and (shape[2] > 0) == (on == 1)
            fit.close()
    assert rows[0][2][1] > 0
    for r in rows[1:]:
        for a, b in zip(rows[0], r):
            assert numpy.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("model,precision,roi", [("2d", 64, 60), ("3d", 64, 60), ("3d", 32, 64), ("spline2D", 32, 62),
                                                 ("spline2D", 64, 62), ("spline2D", 32, 19), ("spline2D", 64, 19)])
def test_rois_too_large_for_a_team(model, precision, roi):
    """ROIs whose team workspace does not fit an SM take a warp per peak; the
    2D spline at a usual size a team.  Both against the FP64 oracle."""
    from oracle.oracle import OracleFitter
    from sa_gb300 import parity, synth
    if model == "spline2D":
        wl = spline2d_workload(roi + 1, 150, 140, 12, 41)
    else:
        wl = synth.make_workload(0 if model == "2d" else 1, frames=1, nx=150, ny=140, seed=42, n_emitters=12)
        for k in ("x", "y"):   # inside the larger ROI's margin
            n = (150 if k == "x" else 140) - roi - 3
            wl["guesses"][0][k] = roi / 2 + 1 + (wl["guesses"][0][k] - 12.0) * n / ((150 if k == "x" else 140) - 24.0)
            wl["truth"][0][k] = roi / 2 + 1 + (wl["truth"][0][k] - 12.0) * n / ((150 if k == "x" else 140) - 24.0)
        t, g = wl["truth"][0], wl["guesses"][0]
        yy, xx = numpy.mgrid[0:140, 0:150]
        img = numpy.full((140, 150), g["background"][0])
        for i in range(12):
            img += t["height"][i] * numpy.exp(-(xx - t["x"][i]) ** 2 / (2 * g["xsigma"][i] ** 2)
                                              - (yy - t["y"][i]) ** 2 / (2 * g["ysigma"][i] ** 2))
        wl["images"][0] = numpy.random.default_rng(43).poisson(img).astype(numpy.float64)
        wl["fitter"]["roi_size"] = roi
    kw = dict(wl["fitter"])
    m = kw.pop("model")
    if m == "spline2D":
        kw["spline"] = kw["spline"]["coeff"]
    ref = OracleFitter(m, (140, 150), **kw)
    ref.newImage(wl["images"][0])
    ref.newBackground(wl["backgrounds"][0])
    ref.newPeaks(wl["guesses"][0], "hdf5")
    ref.doFit(100)
    props = ("x", "y", "z", "height", "background", "status", "iterations")
    want = {p: ref.getPeakProperty(p) for p in props}
    ref.cleanup()
    assert (want["status"] == 1).sum() >= 8
    fit = model_fitter(wl, precision)
    fit.load(numpy.stack(wl["images"]), numpy.stack(wl["backgrounds"]), wl["guesses"], "hdf5")
    shape = numpy.zeros(4, dtype=numpy.int32)
    assert fit.clib.saGetSweepShape(fit.h, shape) == 0 and (shape[2] > 0) == (roi == 19), shape
    fit.fit(100)
    st = parity.compare(fit.results(), want)
    fit.close()
    assert parity.within_tolerance(st, min_fraction=0.999), st
