"""The tail of a fit (saSetTailPeaks): once every frame still fitting has
at most a few RUNNING peaks, their remaining sweeps run in one launch, each
frame's steps one after another in index order.  The results -- every
peak's parameters, status and iteration count, the counters and the sweep
count -- are the ones the per-sweep ticks give, with fewer launches."""
import numpy
import pytest

pytestmark = pytest.mark.gpu

CASES = [(1, 32, {}), (1, 64, {}), (2, 32, {}), (3, 32, dict(n_emitters=60))]


def fit_once(wl, precision, tail_peaks, max_iterations=2000):
    from sa_gb300 import cubic_fit_c, engine
    kw = dict(wl["fitter"])
    model = kw.pop("model")
    spl = kw.pop("spline", None)
    if spl is not None:
        kw["spline"] = cubic_fit_c.SplinePSF(coeff=spl["coeff"])
    fit = engine.BatchFitter(model, (wl["ny"], wl["nx"]), len(wl["images"]), rqe=wl["rqe"],
                             scmos_cal=wl["scmos_cal"], precision=precision, **kw)
    assert fit.clib.saSetTailPeaks(fit.h, tail_peaks) == 0
    fit.load(numpy.stack(wl["images"]), numpy.stack(wl["backgrounds"]), wl["guesses"], "hdf5")
    l0 = fit.kernel_launches()
    sweeps = fit.fit(max_iterations)
    out = fit.results()
    out["counters"] = fit.counters()
    out["sweeps"] = sweeps
    out["launches"] = fit.kernel_launches() - l0
    fit.close()
    return out


@pytest.mark.parametrize("cfg,precision,kw", CASES)
def test_tail_launch_gives_the_ticks_results(cfg, precision, kw):
    from sa_gb300 import synth
    wl = synth.make_workload(cfg, frames=2, nx=128, ny=128, seed=41, **kw)
    ticks = fit_once(wl, precision, 0)
    tail = fit_once(wl, precision, 4)
    for k in ("x", "y", "z", "height", "background", "status", "iterations", "counters"):
        assert numpy.array_equal(tail[k], ticks[k]), k
    assert tail["sweeps"] == ticks["sweeps"]
    assert tail["launches"] <= ticks["launches"]


@pytest.mark.parametrize("cfg,precision,peaks", [(0, 32, 2), (1, 32, 8), (2, 32, 3), (1, 64, 4), (3, 32, 5)])
def test_tail_counts_every_step(cfg, precision, peaks):
    """Frames of so few peaks that all sweeps but the first are the tail's:
    200 fits give the counters that the ticks give, every time."""
    from sa_gb300 import cubic_fit_c, engine, synth
    wl = synth.make_workload(cfg, frames=5, nx=64, ny=60, seed=90 + peaks, n_emitters=peaks)
    kw = dict(wl["fitter"])
    model = kw.pop("model")
    spl = kw.pop("spline", None)
    if spl is not None:
        kw["spline"] = cubic_fit_c.SplinePSF(coeff=spl["coeff"])
    fit = engine.BatchFitter(model, (wl["ny"], wl["nx"]), len(wl["images"]), rqe=wl["rqe"],
                             scmos_cal=wl["scmos_cal"], precision=precision, **kw)
    images, backgrounds = numpy.stack(wl["images"]), numpy.stack(wl["backgrounds"])

    def counted(tail_peaks):
        assert fit.clib.saSetTailPeaks(fit.h, tail_peaks) == 0
        before = fit.counters()
        fit.load(images, backgrounds, wl["guesses"], "hdf5")
        fit.fit(100)
        return fit.counters() - before

    ticks = counted(0)
    assert ticks[1] > 0
    for _ in range(200):
        assert numpy.array_equal(counted(8), ticks)
    fit.close()
