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
