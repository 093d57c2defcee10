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
