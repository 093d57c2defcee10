"""
The work a user of this framework has it do, as measured cases.

A case is one call sequence of a localisation analysis through the public
Python entry points (dao_fit_c, engine, mp_fit_dao_c, fitting, find_peaks):
frames in, fitted or found peaks out.  Sizes, densities and parameters are
those of the benchmark configurations (sa_gb300/synth.py, bench.py) and of
the tests.

  kind "frame"    one frame through a MultiFitter object, the reference's
                  per-frame API: new image, background and peaks, doFit,
                  the properties an analysis reads, the fit image
  kind "batch"    many frames through engine.BatchFitter: host frames in,
                  results out
  kind "planes"   multi-plane frames through MPFitDao2D.fitBatch
  kind "finder"   two consecutive chunks of a movie, already on the GPU,
                  through BatchPeakFinder
  kind "find1"    two frames of a movie, host arrays, through
                  PeakFinderGaussian (the reference's per-frame finder)
  kind "loop"     whole find / fit analysis of frames with BatchFindFit
"""
import math
import os
import sys

import numpy
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "storm-analysis_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from sa_gb300 import cubic_fit_c, dao_fit_c, engine, find_peaks, fitting, mp_fit_dao_c  # noqa: E402
from sa_gb300 import psf_fft_c, pupil_fn, synth  # noqa: E402

MAX_SWEEPS = 200            # the benchmark configurations' sweep limit
PEAK_COLUMNS = 8            # x y z height background xsigma ysigma error

# Finder parameters of the benchmark's finder and find / fit workloads.
FIND = dict(background_sigma=8.0, foreground_sigma=1.0, find_max_radius=5, iterations=20, sigma=1.5,
            threshold=6.0, roi_size=18)

GAUSSIAN = {
    "2dfixed": dict(roi_size=10),
    "2d": dict(roi_size=10, sigma_range=[0.5, 3.0]),
    "3d": dict(roi_size=18, sigma_range=[0.5, 4.0]),
    "Z": dict(roi_size=12, wx_params=synth.WX_PARAMS, wy_params=synth.WY_PARAMS, min_z=-0.5, max_z=0.5),
}
FRAME_CLASS = {"2dfixed": dao_fit_c.MultiFitter2DFixed, "2d": dao_fit_c.MultiFitter2D,
               "3d": dao_fit_c.MultiFitter3D, "Z": dao_fit_c.MultiFitterZ}


def listed():
    return [
        # a user fitting one frame interactively or frame by frame, as the
        # reference does: the smallest call (benchmark configuration 0)
        dict(name="frame_2d", kind="frame", model="2d", precision=32, ny=256, nx=256, emitters=200),
        # one full camera frame at 0.5 emitters / um^2: the lone-frame latency
        # of a live analysis
        dict(name="frame_3d", kind="frame", model="3d", precision=32, ny=512, nx=512, emitters=3355),
        # a movie's chunk through the batched engine, the benchmark's headline
        # workload (configuration 1) and the largest case
        dict(name="batch_3d", kind="batch", model="3d", precision=32, frames=64, ny=512, nx=512, emitters=3355),
        # astigmatic z fitting of a sCMOS movie (configuration 2)
        dict(name="batch_z_scmos", kind="batch", model="Z", precision=32, frames=16, ny=256, nx=256,
             emitters=1000),
        # the same engine asked for FP64 throughout (a user checking results
        # against the reference), odd sizes
        dict(name="batch_2d_fp64", kind="batch", model="2d", precision=64, frames=8, ny=251, nx=317, emitters=400),
        # Spliner's measured-PSF fitting (configuration 3)
        dict(name="batch_spline3d", kind="batch", model="spline3D", precision=32, frames=8, ny=256, nx=256,
             emitters=800),
        # the FFT PSF and pupil-function fitters (the bench's model reports)
        dict(name="batch_fft", kind="batch", model="fft", precision=64, frames=8, ny=256, nx=256, emitters=300),
        dict(name="batch_pupil", kind="batch", model="pupil", precision=64, frames=8, ny=256, nx=256,
             emitters=300),
        # biplane imaging: two planes fitted jointly
        dict(name="planes", kind="planes", channels=2, frames=64, ny=256, nx=256, emitters=200),
        # peak finding over a movie's chunks on the GPU
        dict(name="finder", kind="finder", frames=32, ny=512, nx=512, emitters=3355),
        # peak finding frame by frame, host arrays in and out
        dict(name="find1", kind="find1", ny=256, nx=256, emitters=400),
        # the whole 3D-DAOSTORM analysis of a small movie
        dict(name="loop", kind="loop", model="3d", frames=4, ny=128, nx=128, emitters=120, passes=4),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "batch", "batch", "batch", "batch", "batch", "planes", "finder", "find1",
                       "loop"])
    if kind == "frame":
        model = rng.choice(["2dfixed", "2d", "3d", "Z", "spline3D"])
        ny, nx = _logint(rng, 64, 512), _logint(rng, 64, 512)
        return dict(kind=kind, model=model, precision=32, ny=ny, nx=nx, emitters=_emitters(rng, model, ny, nx))
    if kind == "batch":
        model = rng.choice(["2dfixed", "2d", "3d", "Z", "spline3D", "fft", "pupil"])
        slow = model in ("spline3D", "fft", "pupil")
        precision = 64 if model in ("fft", "pupil") or (model in ("2d", "3d") and rng.random() < 0.25) else 32
        hi = 256 if slow or precision == 64 else 512
        ny, nx = _logint(rng, 80, hi), _logint(rng, 80, hi)
        return dict(kind=kind, model=model, precision=precision, frames=_logint(rng, 1, 8 if hi == 256 else 64),
                    ny=ny, nx=nx, emitters=_emitters(rng, model, ny, nx))
    if kind == "planes":
        ny, nx = _logint(rng, 96, 256), _logint(rng, 96, 256)
        return dict(kind=kind, channels=rng.choice([2, 3]), frames=_logint(rng, 1, 64), ny=ny, nx=nx,
                    emitters=max(4, int(200 * ny * nx / 65536 * rng.uniform(0.3, 1.0))))
    if kind == "loop":
        return dict(kind=kind, model=rng.choice(["2d", "3d"]), frames=rng.randint(1, 4), ny=_logint(rng, 64, 128),
                    nx=_logint(rng, 64, 128), emitters=rng.randint(10, 100), passes=rng.randint(1, 4))
    ny, nx = _logint(rng, 100, 512), _logint(rng, 100, 512)
    n = max(1, int(3355 * ny * nx / 262144 * rng.uniform(0.1, 1.0)))
    if kind == "finder":
        return dict(kind=kind, frames=_logint(rng, 1, 32), ny=ny, nx=nx, emitters=n)
    return dict(kind=kind, ny=ny, nx=nx, emitters=n)


def _emitters(rng, model, ny, nx):
    """Emitters a frame holds at the densities of the benchmark configurations
    (0.1 to 0.6 per um^2 of 0.16 um pixels)."""
    top = 0.25 if model in ("fft", "pupil") else 0.6
    return max(2, int(ny * nx * 0.0256 * math.exp(rng.uniform(math.log(0.05), math.log(top)))))


# ---------------------------------------------------------------------------
# synthetic frames (drawn on the GPU: the seed alone decides them)
# ---------------------------------------------------------------------------

RADIUS = 10                 # pixels drawn around an emitter


def _render(frame, x, y, h, sx, sy, n_frames, ny, nx, background):
    """Expected photo-electrons (n_frames, ny, nx): a background per frame plus
    h exp(-(c - x)^2 / 2 sx^2 - (r - y)^2 / 2 sy^2).  The contributions are
    summed as integers (2^-20) so that the order of the additions does not
    matter."""
    dev = x.device
    acc = (background.view(-1, 1, 1) * 1048576.0).round().to(torch.int64).expand(n_frames, ny, nx).contiguous()
    d = torch.arange(-RADIUS, RADIUS + 1, device=dev)
    for a in range(0, x.numel(), 65536):
        s = slice(a, a + 65536)
        cx, cy = x[s].round().to(torch.int64)[:, None] + d, y[s].round().to(torch.int64)[:, None] + d
        gx = torch.exp(-(cx - x[s, None]) ** 2 / (2.0 * sx[s, None] ** 2))
        gy = torch.exp(-(cy - y[s, None]) ** 2 / (2.0 * sy[s, None] ** 2))
        v = ((h[s, None, None] * gy[:, :, None] * gx[:, None, :]) * 1048576.0).round().to(torch.int64)
        inside = ((cy >= 0) & (cy < ny))[:, :, None] & ((cx >= 0) & (cx < nx))[:, None, :]
        at = frame[s, None, None] * (ny * nx) + cy[:, :, None] * nx + cx[:, None, :]
        acc.view(-1).index_add_(0, at[inside], v[inside])
    return acc.double() / 1048576.0


def _gaussian_frames(model, n_frames, ny, nx, emitters, seed):
    """Frames, backgrounds, starting peaks and calibration of a Gaussian
    model, with the distributions of synth.make_workload: heights, widths, z
    and the camera of the model's benchmark configuration, guesses off the
    truth by 0.3 px and 20 %."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = n_frames * emitters
    f64 = dict(dtype=torch.float64, device="cuda")

    def uniform(lo, hi, size=n):
        return lo + (hi - lo) * torch.rand(size, generator=g, **f64)

    roi = GAUSSIAN[model]["roi_size"]
    m = roi // 2 + 2
    frame = torch.arange(n_frames, device="cuda").repeat_interleave(emitters)
    x, y = uniform(m, nx - m - 1), uniform(m, ny - m - 1)
    bg = torch.full((n_frames,), 20.0, **f64)
    z = torch.zeros(n, **f64)
    if model == "3d":
        sx, sy = uniform(1.0, 2.0), uniform(1.0, 2.0)
        h = torch.exp(uniform(math.log(200.0), math.log(5000.0)))
        bg = uniform(5.0, 50.0, n_frames)
    elif model == "Z":
        z = uniform(-0.4, 0.4)
        sx, sy = synth._widths_from_z(z.cpu(), synth.WX_PARAMS).cuda(), synth._widths_from_z(z.cpu(), synth.WY_PARAMS).cuda()
        h = uniform(1000.0, 4000.0)
    else:
        sx = torch.full((n,), 1.3, **f64)
        sy = sx.clone()
        h = uniform(500.0, 3000.0)
    expected = _render(frame, x, y, h, sx, sy, n_frames, ny, nx, bg)
    images = torch.poisson(expected, generator=g)
    rqe, scmos = numpy.ones((ny, nx)), numpy.zeros((ny, nx))
    if model == "Z":
        # a sCMOS camera: offset, read noise and gain of every pixel
        variance = -2.0 * (torch.log(uniform(1e-12, 1.0, (ny, nx))) + torch.log(uniform(1e-12, 1.0, (ny, nx))))
        gain = 2.0 + 0.05 * torch.randn((ny, nx), generator=g, **f64)
        images = images + torch.randn(images.shape, generator=g, **f64) * torch.sqrt(variance) / gain
        scmos = (variance / (gain * gain)).cpu().numpy()
    images = images.clamp_(min=1.0)
    noise = lambda s: s * torch.randn(n, generator=g, **f64)
    cols = dict(x=x + noise(0.3), y=y + noise(0.3), z=z + (noise(0.05) if model == "Z" else 0.0),
                background=bg[frame], height=h * uniform(0.8, 1.2), xsigma=sx * uniform(0.8, 1.2),
                ysigma=sy * uniform(0.8, 1.2))
    if model in ("2d", "2dfixed"):
        cols["ysigma"] = cols["xsigma"] if model == "2d" else sx
        cols["xsigma"] = cols["xsigma"] if model == "2d" else sx
    cols = {k: v.cpu().numpy() for k, v in cols.items()}
    peaks = [{k: v[f * emitters:(f + 1) * emitters] for k, v in cols.items()} for f in range(n_frames)]
    return images, bg.view(-1, 1, 1).expand(n_frames, ny, nx), peaks, rqe, scmos


def _frames(case, seed):
    """(images, backgrounds, peaks, rqe, scmos, fitter arguments): images and
    backgrounds as (frames, ny, nx) float64 numpy arrays."""
    model, n_frames = case["model"], case.get("frames", 1)
    ny, nx, n = case["ny"], case["nx"], case["emitters"]
    if model in GAUSSIAN:
        images, bgs, peaks, rqe, scmos = _gaussian_frames(model, n_frames, ny, nx, n, seed)
        return images.cpu().numpy(), bgs.cpu().numpy().copy(), peaks, rqe, scmos, dict(GAUSSIAN[model])
    if model == "spline3D":
        # one measured PSF (camera_seed) for every movie of it
        wl = synth.make_workload(3, frames=n_frames, nx=nx, ny=ny, seed=seed, n_emitters=n, camera_seed=3)
        kw = dict(spline=cubic_fit_c.SplinePSF(coeff=wl["spline"]["coeff"]))
    elif model == "fft":
        wl = synth.fft_workload(frames=n_frames, nx=nx, ny=ny, n_emitters=n, seed=seed)
        kw = dict(psf_fft=psf_fft_c.PSFFFT(wl["fitter"]["psf"]))
    else:
        wl = synth.pupil_workload(frames=n_frames, nx=nx, ny=ny, n_emitters=n, seed=seed)
        kw = dict(pupil_fn=pupil_fn.PupilFunction(pf_data=wl["fitter"]["pf_data"], zmin=-500.0, zmax=500.0))
    return numpy.stack(wl["images"]), numpy.stack(wl["backgrounds"]), wl["guesses"], wl["rqe"], wl["scmos_cal"], kw


def _movie(case, seed, n_frames):
    """Frames for the finder, mirror-padded by its margin, float64."""
    images = _gaussian_frames("3d", n_frames, case["ny"], case["nx"], case["emitters"], seed)[0].cpu().numpy()
    margin = int(FIND["roi_size"] / 2 + 2)
    return numpy.ascontiguousarray(numpy.stack([fitting.padArray(im, margin) for im in images]))


class _Held(object):
    """A device array of the library as torch sees it (no copy)."""

    def __init__(self, address, shape):
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f8", data=(address, False), version=2)


class _State(object):
    """What a program keeps between calls; its handles go with it."""

    def __init__(self, case):
        self.case = case
        self.close = None

    def __del__(self):
        try:
            if self.close is not None:
                self.close()
        except Exception:
            pass


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    if kind == "frame":
        images, bgs, peaks, rqe, scmos, kw = _frames(case, seed)
        s.image, s.background, s.peaks = images[0], bgs[0], peaks[0]
        kw["rqe"], kw["scmos_cal"] = rqe, scmos
        if case["model"] == "spline3D":
            s.fitter = cubic_fit_c.CSpline3DFit(spline_fn=kw.pop("spline"), precision=case["precision"], **kw)
        else:
            s.fitter = FRAME_CLASS[case["model"]](precision=case["precision"], **kw)
        s.fitter.initializeC(s.image)
        s.close = lambda f=s.fitter: f.cleanup(verbose=False)
    elif kind == "batch":
        images, bgs, s.peaks, rqe, scmos, kw = _frames(case, seed)
        # a movie chunk as a reader hands it over: float32 in pinned memory
        s.images = torch.from_numpy(images.astype(numpy.float32)).pin_memory().numpy()
        s.backgrounds = torch.from_numpy(bgs.astype(numpy.float32)).pin_memory().numpy()
        s.fitter = engine.BatchFitter(case["model"], (case["ny"], case["nx"]), case["frames"], rqe=rqe,
                                      scmos_cal=scmos, precision=case["precision"],
                                      peaks_capacity=case["emitters"], **kw)
        s.close = s.fitter.close
    elif kind == "planes":
        rng = numpy.random.default_rng(seed)
        shape = (case["ny"], case["nx"])
        wls = [synth.multiplane_workload(case["channels"], case["nx"], case["ny"], case["emitters"], seed=seed)]
        wls += [_plane_frame(wls[0]["maps"], case, rng) for _ in range(case["frames"] - 1)]
        s.images = [numpy.stack([w["images"][c] for w in wls]) for c in range(case["channels"])]
        s.backgrounds = [numpy.full((len(wls),) + shape, 20.0) for _ in range(case["channels"])]
        s.peaks = [w["peaks"] for w in wls]
        f = mp_fit_dao_c.MPFitDao2D(n_channels=case["channels"], roi_size=10, sigma_range=(1.0, 3.0))
        for c in range(case["channels"]):
            f.initializeChannel(numpy.ones(shape), numpy.zeros(shape), c)
        f.setMapping(*wls[0]["maps"])
        f.setWeights(verbose=False)
        s.fitter = f
        s.close = lambda f=f: f.cleanup(verbose=False)
    elif kind == "finder":
        movie = _movie(case, seed, 2 * case["frames"])
        s.chunks = [torch.from_numpy(movie[k * case["frames"]:(k + 1) * case["frames"]]).cuda() for k in range(2)]
        s.finder = fitting.BatchPeakFinder(FIND, movie.shape[1:], case["frames"])
        s.close = s.finder.cleanUp
    elif kind == "find1":
        s.images = list(_movie(case, seed, 2))
        s.finder = fitting.PeakFinderGaussian(FIND)
        s.close = s.finder.cleanUp
    else:
        s.images = _gaussian_frames(case["model"], case["frames"], case["ny"], case["nx"], case["emitters"],
                                    seed)[0].cpu().numpy()
        params = dict(FIND, model=case["model"], iterations=case["passes"])
        s.loop = find_peaks.BatchFindFit(params, (case["ny"], case["nx"]), case["frames"])
        s.close = s.loop.cleanUp
    return s


def _plane_frame(maps, case, rng):
    """One more multi-plane frame of the same optics (affine maps)."""
    ny, nx, n = case["ny"], case["nx"], case["emitters"]
    x, y = rng.uniform(14.0, nx - 14.0, n), rng.uniform(14.0, ny - 14.0, n)
    h = rng.uniform(400.0, 1500.0, n)
    images = []
    d = numpy.arange(-8, 9)
    for c in range(case["channels"]):
        cx = maps[0][3 * c] + maps[0][3 * c + 1] * x + maps[0][3 * c + 2] * y
        cy = maps[1][3 * c] + maps[1][3 * c + 1] * x + maps[1][3 * c + 2] * y
        sig = 1.3 + 0.35 * c
        px, py = cx.astype(int)[:, None] + d, cy.astype(int)[:, None] + d
        v = (h / (1.0 + 0.5 * c))[:, None, None] * numpy.exp(
            -((px - cx[:, None]) ** 2)[:, None, :] / (2 * sig * sig) - ((py - cy[:, None]) ** 2)[:, :, None] / (2 * sig * sig))
        img = numpy.full((ny + 32, nx + 32), 20.0)
        numpy.add.at(img, (py[:, :, None] + 16, px[:, None, :] + 16), v)
        images.append(rng.poisson(img[16:-16, 16:-16]).astype(numpy.float64))
    peaks = {"x": numpy.round(x) + rng.uniform(-0.4, 0.4, n), "y": numpy.round(y) + rng.uniform(-0.4, 0.4, n),
             "z": numpy.zeros(n), "sigma": numpy.full(n, 1.5)}
    return {"images": images, "peaks": peaks}


FRAME_PROPS = ("x", "y", "z", "height", "background", "error", "significance", "iterations", "status")


def run(state):
    kind = state.case["kind"]
    if kind == "frame":
        f = state.fitter
        f.newImage(state.image)
        f.newBackground(state.background)
        f.newPeaks(state.peaks, "hdf5")
        f.doFit(MAX_SWEEPS)
        out = {p: f.getPeakProperty(p) for p in FRAME_PROPS}
        if state.case["model"] != "spline3D":
            out["xsigma"], out["ysigma"] = f.getPeakProperty("xsigma"), f.getPeakProperty("ysigma")
        out["fit_image"] = f.getFitImage()
        return out
    if kind == "batch":
        f = state.fitter
        f.load(state.images, state.backgrounds, state.peaks, "hdf5")
        f.fit(MAX_SWEEPS)
        values, ints = f.results_fast()
        if state.case["model"] in ("spline3D", "fft", "pupil"):
            values = values[:, [0, 1, 2, 3, 4, 7]]   # these models have no widths
        return {"values": values, "ints": ints}
    if kind == "planes":
        out, _ = state.fitter.fitBatch(state.images, state.backgrounds, state.peaks, "finder", max_iterations=MAX_SWEEPS)
        return out
    if kind == "finder":
        f = state.finder
        out = []
        for chunk in state.chunks:
            f.newImages(chunk)
            f.estimateBackground()
            counts, _ = f.findPeaks()
            peaks = f.peaks()
            peaks = {k: numpy.concatenate([p[k] for p in peaks]) for k in ("x", "y", "z", "sigma")}
            bg = torch.as_tensor(_Held(f.device_pointers()[0], chunk.shape), device="cuda").clone()
            out.append({"background": bg, "counts": counts, "peaks": _table(state.case, peaks)})
        return out
    if kind == "find1":
        f = state.finder
        out = []
        for image in state.images:
            f.newImage(image)
            zero = numpy.zeros(image.shape)
            bg = f.estimateBackground(zero)
            peaks, _, _ = f.findPeaks(zero)
            out.append({"background": bg, "counts": peaks["x"].size, "peaks": _table(state.case, peaks)})
        return out
    per_frame = state.loop.analyze(state.images)
    out = _table(state.case, {k: numpy.concatenate([p[k] for p in per_frame]) for k in per_frame[0]})
    out["counts"] = numpy.array([p["x"].size for p in per_frame])
    return out


def _table(case, columns):
    """Columns of found peaks as arrays of one length for every movie of the
    case (zeros after the last peak)."""
    rows = case.get("frames", 1) * (2 * case["emitters"] + 64)
    out = {}
    for k, v in columns.items():
        out[k] = numpy.zeros(max(rows, v.size), dtype=v.dtype)
        out[k][:v.size] = v
    return out


# LM iterations a peak takes on these workloads (measured), for work().
ITERATIONS = {"2dfixed": 12, "2d": 14, "3d": 25, "Z": 18, "spline3D": 20, "fft": 15, "pupil": 15}


def work(case):
    """Every input read and every output written once; the arithmetic of the
    LM iterations (per ROI pixel the model, its Jacobian row, the normal
    equations and the error, bench.py's count) or of the filters' taps."""
    kind = case["kind"]
    px = case["ny"] * case["nx"]
    if kind in ("finder", "find1"):
        pad = 2 * int(FIND["roi_size"] / 2 + 2)
        frames = 2 * case.get("frames", 1)
        ppx = (case["ny"] + pad) * (case["nx"] + pad) * frames
        # separable passes: background 81 + 81, variance 11 + 11, foreground 11 + 11 taps
        return {"bytes": 16.0 * ppx, "flops": 2.0 * 206 * ppx}
    model = case.get("model", "2d")
    frames = case.get("frames", 1) * case.get("channels", 1)
    n = frames * case["emitters"]
    k = {"2dfixed": 4, "2d": 5, "3d": 6}.get(model, 5)
    roi = {"spline3D": 19, "fft": 20, "pupil": 30}.get(model) or GAUSSIAN[model]["roi_size"]
    nroi = math.pi * roi * roi / 4.0
    per_pixel = 2 * (k * (k + 1) // 2 + k) + 3 * k + 5 + 21 + (512 if model == "spline3D" else 0)
    item = 4 if kind == "batch" else 8
    passes = case.get("passes", 1)
    return {"bytes": 2.0 * item * px * frames + n * 8.0 * (7 + PEAK_COLUMNS + 1),
            "flops": n * ITERATIONS[model] * nroi * per_pixel * passes}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    if case["kind"] in ("finder", "find1"):
        return _exact_background(case, seed)
    if case["kind"] == "frame" and case["model"] == "2d" and case["emitters"] <= 400:
        return _exact_frame_2d(case, seed)
    return None   # the sequential fit of thousands of peaks takes minutes in numpy


def _exact_background(case, seed):
    """The background estimate: circular convolution of the frame with the
    normalised Gaussian, drawn out to 5 sigma as the finder draws it."""
    frames = case.get("frames", 1)
    movie = torch.from_numpy(_movie(case, seed, 2 * frames)).cuda()
    ny, nx = movie.shape[1:]
    kernel = [_unit_axis(n) for n in (ny, nx)]
    psf = kernel[0][:, None] * kernel[1][None, :]
    k = torch.fft.rfft2((psf / psf.sum()).cuda())
    out = []
    for c in range(2):
        bg = torch.fft.irfft2(torch.fft.rfft2(movie[c * frames:(c + 1) * frames]) * k, s=(ny, nx))
        out.append({"background": bg if case["kind"] == "finder" else bg[0].cpu().numpy(), "counts": None,
                    "peaks": None})
    return out


def _unit_axis(n):
    """The Gaussian along an axis of n pixels, about n / 2 and cut at 5 sigma,
    moved to the axis' origin as the finder moves it (by int(n / 2))."""
    sigma = FIND["background_sigma"]
    at = torch.arange(n, dtype=torch.float64)
    g = torch.exp(-(at - 0.5 * n) ** 2 / (2.0 * sigma * sigma))
    g[(at - n // 2).abs() > int(5.0 * sigma)] = 0.0
    return torch.roll(g, n // 2)


def _exact_frame_2d(case, seed):
    """The multi-emitter LM fit (MLE, 2D Gaussians with one width) of one
    frame, peak after peak in index order, in numpy doubles."""
    images, _, peaks, rqe, scmos, kw = _frames(case, seed)
    x_data, (ny, nx), roi = images[0], images[0].shape, kw["roi_size"]
    off = 0.5 * roi - 1.0
    c = 0.5 * roi
    ry, rx = numpy.nonzero((numpy.arange(roi)[:, None] - c + 0.5) ** 2 + (numpy.arange(roi)[None, :] - c + 0.5) ** 2 <= c * c)
    fit, bgs, cnt = numpy.zeros((ny, nx)), numpy.zeros((ny, nx)), numpy.zeros((ny, nx))
    wmin, wmax = (1.0 / (2.0 * s * s) for s in (kw["sigma_range"][1], kw["sigma_range"][0]))
    p = peaks[0]
    n = p["x"].size
    # parameters: height, x, y, x width, y width, background
    q = [numpy.array([p["height"][i], p["x"][i] - off, p["y"][i] - off, 0.5 / p["xsigma"][i] ** 2,
                      0.5 / p["ysigma"][i] ** 2, p["background"][i]]) for i in range(n)]
    anchor = [[int(math.floor(v[1])), int(math.floor(v[2]))] for v in q]
    status, lam, err, its = [0] * n, [1.0] * n, [0.0] * n, [0] * n

    def inside(a):
        return 0 <= a[0] < nx - roi and 0 <= a[1] < ny - roi

    def shape(v, a):
        tx, ty = rx - (v[1] - a[0]) - off, ry - (v[2] - a[1]) - off
        return tx, ty, numpy.exp(-tx * tx * v[3]) * numpy.exp(-ty * ty * v[4])

    def put(v, a, sign):
        at = (ry + a[1], rx + a[0])
        fit[at] += sign * v[0] * shape(v, a)[2]
        bgs[at] += sign * v[5]
        cnt[at] += sign

    def deviance(a):
        at = (ry + a[1], rx + a[0])
        fi, x = fit[at] + bgs[at] / cnt[at], x_data[at]
        if not (fi > 0.0).all():
            return fi, None
        return fi, float(numpy.sum(2.0 * ((fi - x) - x * numpy.log(fi / x))))

    for i in range(n):
        if not inside(anchor[i]) or q[i][0] < 0.0:
            status[i] = 2
            continue
        q[i][3] = min(max(q[i][3], wmin), wmax)
        put(q[i], anchor[i], 1)
    for sweep in range(1 + MAX_SWEEPS):
        if 0 not in status:
            break
        for i in range(n):
            if status[i] != 0:
                continue
            v0, a0 = q[i].copy(), list(anchor[i])
            fi, e0 = deviance(a0)
            x = x_data[ry + a0[1], rx + a0[0]]
            tx, ty, g = shape(v0, a0)
            jac = numpy.stack([g, 2.0 * v0[0] * v0[3] * tx * g, 2.0 * v0[0] * v0[3] * ty * g,
                               -v0[0] * (tx * tx + ty * ty) * g, numpy.ones_like(g)])
            grad = jac @ (2.0 * (1.0 - x / fi))
            hess = (jac * (2.0 * x / (fi * fi))) @ jac.T
            put(v0, a0, -1)
            e0 = err[i] if e0 is None else e0
            while True:
                if lam[i] > 1.0e20:
                    status[i] = 2
                    break
                its[i] += 1
                status[i] = 0
                try:
                    damped = hess + lam[i] * numpy.diag(numpy.diag(hess))
                    numpy.linalg.cholesky(damped)
                    d = numpy.linalg.solve(damped, grad)
                except numpy.linalg.LinAlgError:
                    status[i] = 2
                    lam[i] *= 4.0
                    continue
                v, a = v0.copy(), list(a0)
                v[:4] -= d[:4]
                v[4] = v[3]
                v[5] -= d[4]
                for k in (0, 1):
                    if not -0.5 <= v[1 + k] - a[k] <= 1.5:
                        a[k] = int(math.floor(v[1 + k]))
                if not inside(a) or v[0] < 0.0:
                    status[i] = 2
                    lam[i] *= 4.0
                    continue
                v[3] = min(max(v[3], wmin), wmax)
                put(v, a, 1)
                e = deviance(a)[1]
                if e is not None and (e <= e0 or (e - e0) / e0 < 1.0e-6):
                    if abs(e - e0) / e0 < 1.0e-6:
                        status[i] = 1
                    elif lam[i] > 1.0e-3:
                        lam[i] *= 0.75
                    q[i], anchor[i], err[i] = v, a, e
                    break
                put(v, a, -1)
                if e is None:
                    status[i] = 2
                lam[i] *= 4.0
        for i in range(n):
            d = [q[i][1 + k] - anchor[i][k] for k in (0, 1)]
            if status[i] == 0 and not all(-0.25 <= t <= 1.25 for t in d):
                put(q[i], anchor[i], -1)
                anchor[i] = [int(math.floor(q[i][1 + k])) for k in (0, 1)]
                if inside(anchor[i]) and q[i][0] >= 0.0:
                    put(q[i], anchor[i], 1)
                else:
                    status[i] = 2
    v = numpy.array(q)
    sig = numpy.zeros(n)
    for i in range(n):
        g = shape(q[i], anchor[i])[2]
        at = (ry + anchor[i][1], rx + anchor[i][0]) if inside(anchor[i]) else None
        bg = numpy.sum((x_data[at] - q[i][0] * g) * g * g) if at is not None else 0.0
        s1, s2 = numpy.sum(g), numpy.sum(g * g)
        sig[i] = (q[i][0] * s2 / s1 if at is not None else 1.0) / math.sqrt(bg / (s1 * s1) if bg > 0.0 else 1.0)
    return {"x": v[:, 1] + off, "y": v[:, 2] + off, "z": numpy.zeros(n), "height": v[:, 0], "background": v[:, 5],
            "error": numpy.array(err), "significance": sig, "iterations": None, "status": None,
            "xsigma": numpy.sqrt(0.5 / v[:, 3]), "ysigma": numpy.sqrt(0.5 / v[:, 4]), "fit_image": fit}
