// sa_team.cuh -- the LM step by a team of warps (one CTA per peak) for the
// FP64 engine and the FP32 spline models: the sums of lm_step
// (sa_kernels.cuh), in the same order, so that both give the same bits.
//
// The split is lm_step_g32's: one thread per ROI pixel leaves its terms in
// shared memory; the sums are shared out over the warps, each closed by one
// warp in the warp step's order; warp 0 solves, sums the trial's error and
// decides.  What depends on the peak's record alone -- shape tables, model
// values and derivatives of every pixel, the contribution to take out -- is
// computed while the step waits for its predecessors.  The fit image is
// written once, with the net change of an accepted step.
//
// What bounds it: in the FP64 engine the FP64 pipe, which takes one warp
// instruction per 64 cycles on each of the SM's four schedulers -- a step of
// one warp used a quarter of an SM's; for splines the chain of dependent
// float-float operations.  First sweeps, 8 frames of 256 x 256: spline 12.5 ms a sweep with a
// warp per peak, 2.1 with a team; FFT PSF 13.6 ms, 2.6; pupil function 25.4 ms,
// 4.9; 2D Gaussians in FP64 0.84 ms, 0.44.
#pragma once

#include "sa_g32.cuh"

namespace sa {

// A team step's view of the workspace: the warp step's arrays and tables (b)
// and what only the team keeps.
template <typename T>
struct TeamWS {
  WarpWS<T> b;
  int n;                       // stride of the per-pixel arrays
  T* psf0;                     // model value of the start record
  T* t1;                       // first-order weight (FP32: high word)
  T* t1l;                      // FP32: its low word
  T* t2;                       // Hessian weight
  T* jt;                       // Jacobian row but its last entry (rqe): [entry][n]
  T* c0;                       // per-pixel terms of the current sums
  T* c1;
  T* c2;
  T* c3;
  long long* q0f;              // FP32: fixed-point words of the start contribution and of
  long long* q0b;              // the trial's change of it
  long long* q1f;
  long long* q1b;
  double* rows;                // pupil model: row buffers of warps 1, 2, ...
  const unsigned short* inv;   // ROI pixel (ry * roi + rx) -> its index
};

__host__ __device__ inline size_t team_align(size_t b) { return (b + 15) & ~(size_t)15; }

// The part after the warp workspace.
template <typename T>
__host__ __device__ inline size_t team_ws_bytes(const ModelCfg& cfg, int threads) {
  const size_t n = (size_t)((cfg.nroi + 31) / 32) * 32;
  size_t b = warp_ws_bytes<T>(cfg, cfg.nroi);
  if (sizeof(T) == 4) b += n * (7 + cfg.jac - 1) * sizeof(T) + 4 * n * sizeof(long long);
  else b += n * (3 + cfg.jac - 1) * sizeof(T);
  if (is_pupil(cfg.model)) b += (size_t)(threads / 32 - 1) * 6 * cfg.sx * sizeof(double);
  return b + team_align((size_t)cfg.roi * cfg.roi * sizeof(unsigned short));
}

template <typename T>
__device__ inline TeamWS<T> team_ws(char* base, const ModelCfg& cfg, int threads) {
  TeamWS<T> ws{};
  ws.b = warp_ws<T>(base, cfg, cfg.nroi);
  const int n = ((cfg.nroi + 31) / 32) * 32;
  ws.n = n;
  char* p = base + warp_ws_bytes<T>(cfg, cfg.nroi);
  if (sizeof(T) == 4) {
    long long* q = reinterpret_cast<long long*>(p);
    ws.q0f = q;
    ws.q0b = q + n;
    ws.q1f = q + 2 * n;
    ws.q1b = q + 3 * n;
    p += 4 * n * sizeof(long long);
  }
  T* t = reinterpret_cast<T*>(p);
  ws.t1 = t;
  ws.t2 = t + n;
  if (sizeof(T) == 4) {
    ws.psf0 = ws.b.psf0;   // the warp layout has these for FP32
    ws.t1l = t + 2 * n;
    ws.c0 = t + 3 * n;
    ws.c1 = t + 4 * n;
    ws.c2 = t + 5 * n;
    ws.c3 = t + 6 * n;
    ws.jt = t + 7 * n;
    t += (7 + cfg.jac - 1) * n;
  } else {
    ws.psf0 = t + 2 * n;
    // the sums' terms share memory with arrays that are dead by then
    ws.c0 = ws.b.psf;   // start: f0, then its error terms (a trial's psf comes later)
    ws.c1 = ws.t1;      // trial: error terms
    ws.jt = t + 3 * n;
    t += (3 + cfg.jac - 1) * n;
  }
  ws.rows = reinterpret_cast<double*>(t);
  char* e = reinterpret_cast<char*>(t);
  if (is_pupil(cfg.model)) e += (size_t)(threads / 32 - 1) * 6 * cfg.sx * sizeof(double);
  ws.inv = reinterpret_cast<const unsigned short*>(e);
  return ws;
}

// Shape tables by `count` threads (barrier id).
template <typename T>
__device__ inline void team_tables(const ModelCfg& cfg, const PeakRec& w, TeamWS<T>& ws, int tid, int id, int count,
                                   bool deriv) {
  auto sync = [id, count]() { bar_sync(id, count); };
  if (is_fft(cfg.model)) {
    fft_tables(cfg, w, ws.b, tid, deriv, count, sync);
  } else if (is_pupil(cfg.model)) {
    pupil_tables(cfg, w, ws.b, tid, deriv, count, ws.rows, sync);
  } else if (is_spline(cfg.model)) {
    const SplinePos s = spline_pos(w.p, w.xi, w.yi, w.zi);
    if (deriv || sizeof(T) != 4) spline_tables(cfg, s, ws.b, tid, count);
    else spline_value_monomials(cfg, s, ws.b, tid, count);
  } else if constexpr (sizeof(T) == 8) {
    gauss_tables(cfg, w.p, w.xi, w.yi, ws.b, tid, count);
  }
  sync();
}

template <typename T>
__device__ __forceinline__ SplinePos team_pos(const ModelCfg& cfg, const PeakRec& w) {
  if (is_spline(cfg.model)) return spline_pos(w.p, w.xi, w.yi, w.zi);
  return SplinePos{};
}

// -- what differs between the pixel types ------------------------------------

// The static terms of pixel p (see the header).
__device__ __forceinline__ void team_pixel_static(const ModelCfg& cfg, const FrameSet<double>& fs, TeamWS<double>& ws,
                                                  const PeakRec& o, const SplinePos& s0, double gx, double gy, int p) {
  int rx, ry;
  roi_rc(ws.b.roi, p, rx, ry);
  const double rq = __ldg(fs.rqe + pix_index(cfg, o.xi, o.yi, rx, ry));
  const double psf = psf_at(cfg, fs.aij, ws.b, s0, rx, ry);
  double jt[MAX_JAC];
  jt_row(cfg, fs.aij, ws.b, s0, o, gx, gy, rx, ry, rq, psf, jt);
  ws.b.R[p] = rq;
  ws.psf0[p] = psf;
#pragma unroll
  for (int l = 0; l < MAX_JAC - 1; l++)
    if (l < cfg.jac - 1) ws.jt[l * ws.n + p] = jt[l];
}

__device__ __forceinline__ void team_pixel_static(const ModelCfg& cfg, const FrameSet<float>& fs, TeamWS<float>& ws,
                                                  const PeakRec& o, const SplinePos& s0, float gx, float gy, int p) {
  int rx, ry;
  roi_rc(ws.b.roi, p, rx, ry);
  const long long k = pix_index(cfg, o.xi, o.yi, rx, ry);
  const float rq = __ldg(fs.rqe + k);
  const ff psf = spline_value_ff(cfg, fs.aij, ws.b, s0, rx, ry);
  float jt[MAX_JAC];
  jt_row(cfg, fs.aij, ws.b, s0, o, gx, gy, rx, ry, rq, psf.h, jt);
  ws.b.R[p] = rq;
  ws.psf0[p] = psf.h;
#pragma unroll
  for (int l = 0; l < MAX_JAC - 1; l++)
    if (l < cfg.jac - 1) ws.jt[l * ws.n + p] = jt[l];
  Q2 cf, cb;
  spl32_contrib(psf, ff_from_double(o.p[PH]), ff_from_double(o.p[PBG]), rq, __ldg(fs.scmos + k), cf, cb);
  ws.q0f[p] = cf.h;
  ws.q0b[p] = cb.h;
}

// The start contribution of pixel p at image pixel k of the start ROI.
__device__ __forceinline__ void team_start_contrib(const FrameSet<double>& fs, const TeamWS<double>& ws,
                                                   const PeakRec& o, int p, double rq, double sc, Q2& cf, Q2& cb) {
  cf = quant_t<double>(contrib_f(o.p[PH], ws.psf0[p], rq));
  cb = quant_t<double>(contrib_bg(o.p[PBG], rq, sc));
}
__device__ __forceinline__ void team_start_contrib(const FrameSet<float>& fs, const TeamWS<float>& ws,
                                                   const PeakRec& o, int p, float rq, float sc, Q2& cf, Q2& cb) {
  cf.h = ws.q0f[p];
  cb.h = ws.q0b[p];
  cf.l = cb.l = 0;
}

// The start state of pixel p: model value, weights and the base state (the fit
// image without this peak).
__device__ __forceinline__ void team_pixel_start(const ModelCfg& cfg, const FrameSet<double>& fs, long long fbase,
                                                 TeamWS<double>& ws, const PeakRec& o, int p, bool& fail) {
  int rx, ry;
  roi_rc(ws.b.roi, p, rx, ry);
  const long long k = pix_index(cfg, o.xi, o.yi, rx, ry);
  const Q2 Fq = acc_load<2>(fs.f, fbase + k);
  const Q2 Bq = acc_load<2>(fs.bg, fbase + k);
  const int Cg = __ldcg(fs.cnt + fbase + k);
  const double xv = __ldg(fs.x + fbase + k);
  const double sc = __ldg(fs.scmos + k), rq = ws.b.R[p];
  const double fi0 = acc_value<2>(Fq) + acc_value<2>(Bq) / (double)Cg;
  if (!(fi0 > 0.0)) fail = true;
  // the reference's forms (dao_fit.c:454-460)
  ws.t1[p] = 2.0 * (1.0 - xv / fi0);
  ws.t2[p] = 2.0 * xv / (fi0 * fi0);
  ws.c0[p] = fi0;
  Q2 cf, cb;
  team_start_contrib(fs, ws, o, p, rq, sc, cf, cb);
  ws.b.Fb[p] = acc_value<2>(q_sub(Fq, cf));
  ws.b.Bs[p] = acc_value<2>(q_sub(Bq, cb)) + sc;
  ws.b.X[p] = xv;
  ws.b.IC[p] = (double)Cg;   // (Cg - 1) + 1 once the peak is re-added
}

__device__ __forceinline__ void team_pixel_start(const ModelCfg& cfg, const FrameSet<float>& fs, long long fbase,
                                                 TeamWS<float>& ws, const PeakRec& o, int p, bool& fail) {
  int rx, ry;
  roi_rc(ws.b.roi, p, rx, ry);
  const long long k = pix_index(cfg, o.xi, o.yi, rx, ry);
  const long long Fq = __ldcg(fs.f + fbase + k), Bq = __ldcg(fs.bg + fbase + k);
  const int Cg = __ldcg(fs.cnt + fbase + k);
  const long long Xq = __ldg(fs.xq + fbase + k);
  const float2 xd = __ldg(fs.xff + fbase + k);
  const float sc = __ldg(fs.scmos + k);
  // as lm_step's FP32 branch
  const ff rh = ff_add(ff_from_fixed(Fq - Xq), ff_div(ff_from_fixed(Bq), ff{(float)Cg, 0.0f}));
  const ff f0 = ff_add(rh, ff{xd.x, xd.y});
  const ff t1 = ff_div(ff{2.0f * rh.h, 2.0f * rh.l}, f0);
  ws.b.f0[p] = f0.h;
  ws.t1[p] = t1.h;
  ws.t1l[p] = t1.l;
  float c = 0.0f, r = 0.0f;
  if (!(f0.h > 0.0f)) {
    fail = true;
  } else {
    c = 2.0f * xd.x;
    r = r_minus_log1p(rh.h * rcp_approx(xd.x));
  }
  ws.c0[p] = c;
  ws.c1[p] = r;
  ws.t2[p] = ff_div(ff_sub(ff{2.0f, 0.0f}, t1), f0).h;
  ws.b.Fb[p] = fx_to_float(Fq - ws.q0f[p]);
  ws.b.Bs[p] = fx_to_float(Bq - ws.q0b[p]) + sc;
  ws.b.IC[p] = ic_store<float>(Cg);
}

// The base state at another anchor (load_base, with the start contribution
// taken out where the ROIs overlap).
template <typename T>
__device__ __forceinline__ void team_load_base(const ModelCfg& cfg, const FrameSet<T>& fs, long long fbase,
                                               TeamWS<T>& ws, const PeakRec& o, int ax, int ay, int tid, int count) {
  for (int p = tid; p < cfg.nroi; p += count) {
    int rx, ry;
    roi_rc(ws.b.roi, p, rx, ry);
    const long long k = pix_index(cfg, ax, ay, rx, ry);
    Q2 Fq = acc_load<AccW<T>::W>(fs.f, fbase + k);
    Q2 Bq = acc_load<AccW<T>::W>(fs.bg, fbase + k);
    int Cg = __ldcg(fs.cnt + fbase + k);
    const T sc = __ldg(fs.scmos + k), rq = __ldg(fs.rqe + k);
    const int ox = rx + ax - o.xi, oy = ry + ay - o.yi;   // the same image pixel in the start ROI
    if (in_roi(ox, oy, cfg.roi)) {
      Q2 cf, cb;
      team_start_contrib(fs, ws, o, ws.inv[oy * cfg.roi + ox], rq, sc, cf, cb);
      Fq = q_sub(Fq, cf);
      Bq = q_sub(Bq, cb);
      Cg -= 1;
    }
    if constexpr (sizeof(T) == 4) {
      ws.b.Fb[p] = fx_to_float(Fq.h);
      ws.b.Bs[p] = fx_to_float(Bq.h) + sc;
    } else {
      ws.b.Fb[p] = (T)acc_value<AccW<T>::W>(Fq);
      ws.b.Bs[p] = (T)(acc_value<AccW<T>::W>(Bq) + (double)sc);
    }
    ws.b.R[p] = rq;
    ws.b.X[p] = __ldg(fs.x + fbase + k);
    ws.b.IC[p] = ic_store<T>(Cg + 1);
  }
}

// -- the step's sums (one warp each) ------------------------------------------

// Jacobian entry l of pixel p (the last one is rqe).
template <typename T>
__device__ __forceinline__ T team_jt(const ModelCfg& cfg, const TeamWS<T>& ws, int l, int p) {
  return l < cfg.jac - 1 ? ws.jt[l * ws.n + p] : ws.b.R[p];
}

// Row and column of packed upper-triangle entry e of a k x k matrix.
__device__ __forceinline__ void hes_rc(int k, int e, int& r, int& c) {
  r = 0;
  while (e >= k - r) {
    e -= k - r;
    r++;
  }
  c = r + e;
}

// The normal equations: entries e, e + warps, ... on warp e.
__device__ inline void team_sums(const ModelCfg& cfg, TeamWS<double>& ws, int w, int warps, int lane) {
  const int k = cfg.jac, nh = k + k * (k + 1) / 2;
  for (int e = w; e < nh; e += warps) {
    double acc = 0.0;
    if (e < k) {
      for (int p = lane; p < cfg.nroi; p += 32) acc += ws.t1[p] * team_jt(cfg, ws, e, p);
    } else {
      int l, m;
      hes_rc(k, e - k, l, m);
      for (int p = lane; p < cfg.nroi; p += 32) acc += ws.t2[p] * team_jt(cfg, ws, l, p) * team_jt(cfg, ws, m, p);
    }
    acc = warp_sum(acc);
    if (lane == 0) ws.b.jh[e] = acc;
  }
}

// FP32: the lanes' partial sums to red (columns as lm_step has them; entry e's
// lane sums in column e, the gradient's lo words from column nh on).
__device__ inline void team_sums(const ModelCfg& cfg, TeamWS<float>& ws, int w, int warps, int lane) {
  const int k = cfg.jac, nh = k + k * (k + 1) / 2;
  float* red = ws.b.red;
  for (int e = w; e < nh; e += warps) {
    if (e < k) {
      ff g{0.0f, 0.0f};
      for (int p = lane; p < cfg.nroi; p += 32)
        ff_acc(g, ff_mul_raw(ff{ws.t1[p], ws.t1l[p]}, ff{team_jt(cfg, ws, e, p), 0.0f}));
      g = fast_two_sum(g.h, g.l);
      red[lane * 33 + e] = g.h;
      red[lane * 33 + nh + e] = g.l;
    } else {
      int l, m;
      hes_rc(k, e - k, l, m);
      float acc = 0.0f;
      for (int p = lane; p < cfg.nroi; p += 32) acc += ws.t2[p] * team_jt(cfg, ws, l, p) * team_jt(cfg, ws, m, p);
      red[lane * 33 + e] = acc;
    }
  }
}

// The close of the sums (warp 0; FP32: the columns of red in lane order).
__device__ __forceinline__ void team_close_sums(const ModelCfg&, TeamWS<double>&, int) {}
__device__ inline void team_close_sums(const ModelCfg& cfg, TeamWS<float>& ws, int lane) {
  const int k = cfg.jac, nh = k + k * (k + 1) / 2;
  const float* red = ws.b.red;
  if (lane < nh) {
    float hi = 0.0f, lo = 0.0f;
#pragma unroll 8
    for (int j = 0; j < 32; j++) ff_add(hi, lo, red[j * 33 + lane]);
    if (lane < k) {
#pragma unroll 8
      for (int j = 0; j < 32; j++) ff_add(hi, lo, red[j * 33 + nh + lane]);
    }
    ws.b.jh[lane] = (double)hi + (double)lo;
  }
  __syncwarp();
}

// The start error: the pixels' terms (FP64: still to be computed from f0), by
// warps 1 .. warps - 1 while warp 0 solves; the sum on warp 1's lanes.
__device__ inline double team_start_error(const ModelCfg& cfg, TeamWS<double>& ws, int tid, int threads) {
  for (int p = tid - 32; p < cfg.nroi; p += threads - 32) {
    const double fi = ws.c0[p];
    ws.c0[p] = fi > 0.0 ? deviance(fi, ws.b.X[p]) : 0.0;
  }
  bar_sync(2, threads - 32);
  double dev = 0.0;
  if (tid < 64) {
    for (int p = tid - 32; p < cfg.nroi; p += 32) dev += ws.c0[p];
    dev = warp_sum(dev);
  }
  return dev;
}
__device__ inline double team_start_error(const ModelCfg& cfg, TeamWS<float>& ws, int tid, int) {
  float dev = 0.0f;
  if (tid < 64) {
    for (int p = tid - 32; p < cfg.nroi; p += 32) dev = fmaf(ws.c0[p], ws.c1[p], dev);
    return warp_sum_ff(dev);
  }
  return 0.0;
}

// -- the trial ------------------------------------------------------------------

// Trial update of the models' delta orders (apply_update + check_for,
// dao_fit.c:1777-1880, cubic_fit.c:939-1005, fft_fit.c:481-524, pupil_fit.c:529-570)
// on the trial record t from the start record o, one parameter per lane of warp
// 0 with the same double operations.  Returns check_for's code on every lane.
__device__ inline int team_update(const ModelCfg& cfg, const PeakRec& o, PeakRec& t, double dl, int lane) {
  const int model = cfg.model, k = cfg.jac;
  const bool act = lane < k;
  const int j = act ? lane : 0;
  int pi;
  if (model == M_3D) pi = j == 0 ? PH : j == 1 ? PX : j == 2 ? PXW : j == 3 ? PY : j == 4 ? PYW : PBG;
  else if (model == M_2D) pi = j == 0 ? PH : j == 1 ? PX : j == 2 ? PY : j == 3 ? PXW : PBG;
  else if (k == 4) pi = j == 0 ? PH : j == 1 ? PX : j == 2 ? PY : PBG;
  else pi = j == 0 ? PH : j == 1 ? PX : j == 2 ? PY : j == 3 ? PZ : PBG;
  double nv = o.p[pi] - dl;
  double wt = 0.0, wv = 0.0;
  if (act && pi == PZ) {
    double lo = cfg.zmin, hi = cfg.zmax;
    if (model == M_FFT) {
      hi = ((double)cfg.sz) * 0.5 - 1.0e-12;
      lo = -hi;
    } else if (model == M_SPLINE3D) {
      lo = 1.0e-12;
      hi = ((double)cfg.sz) - 1.0e-12;
    }
    if (nv < lo) nv = lo;
    if (nv > hi) nv = hi;
  }
  if (model == M_Z) {
    // widths from the new z: wx on lane 0, wy on lane 1 (widths_from_z)
    const double z = __shfl_sync(0xffffffffu, nv, 3);
    const bool sy = (lane == 1);
    const double c0 = sy ? cfg.wy[0] : cfg.wx[0], c1 = sy ? cfg.wy[1] : cfg.wx[1];
    const double c2 = sy ? cfg.wy[2] : cfg.wx[2], c3 = sy ? cfg.wy[3] : cfg.wx[3];
    const double c4 = sy ? cfg.wy[4] : cfg.wx[4];
    const double z0 = (z - c1) / c2;
    const double z1 = z0 * z0, z2 = z1 * z0, z3 = z2 * z0;
    const double tt = 1.0 + z1 + c3 * z2 + c4 * z3;
    wt = tt * tt;
    wv = 2.0 / (c0 * tt);
  }
  // re-anchor on the PX and PY lanes
  const bool axis = act && (pi == PX || pi == PY);
  int ai = (pi == PY) ? o.yi : o.xi;
  const double d = nv - (double)ai;
  if (axis && (dbl_lt_neg(d, -0.5) || dbl_gt_pos(d, 1.5))) ai = (int)floor(nv);
  const int lim = (pi == PY) ? (cfg.ny - cfg.roi) : (cfg.nx - cfg.roi);
  const bool margin = __any_sync(0xffffffffu, axis && ((ai < 0) || (ai >= lim)));
  const bool negh = __any_sync(0xffffffffu, act && pi == PH && dbl_negative(nv));
  double cv = nv;
  if ((model == M_2D && pi == PXW) || (model == M_3D && (pi == PXW || pi == PYW))) {
    if (cv < cfg.wmin) cv = cfg.wmin;
    else if (cv > cfg.wmax) cv = cfg.wmax;
  }
  if (act) {
    t.p[pi] = cv;
    if (model == M_2D && pi == PXW) t.p[PYW] = nv;   // the unclamped x width
    if (pi == PX) t.xi = ai;
    if (pi == PY) t.yi = ai;
    if (model == M_SPLINE3D && pi == PZ) t.zi = (int)nv;
  }
  if (model == M_Z && lane < 2) {
    (lane ? t.wyt : t.wxt) = wt;
    t.p[lane ? PYW : PXW] = wv;
  }
  __syncwarp();
  return margin ? 1 : (negh ? 2 : 0);
}

// A trial's per-pixel error terms.  FP64: psf (kept for the write-back) and
// the deviance.
__device__ __forceinline__ void team_pixel_trial(const ModelCfg& cfg, const FrameSet<double>& fs, long long fbase,
                                                 TeamWS<double>& ws, const PeakRec& o, const PeakRec& t,
                                                 const SplinePos& s, bool, int p, bool& fail) {
  int rx, ry;
  roi_rc(ws.b.roi, p, rx, ry);
  const double psf = psf_at(cfg, fs.aij, ws.b, s, rx, ry);
  ws.b.psf[p] = psf;
  const double rq = ws.b.R[p];
  const double bgT = t.p[PBG];
  const double fi = ws.b.Fb[p] + contrib_f(t.p[PH], psf, rq) + bg_div(ws.b.Bs[p] + bgT * rq, ws.b.IC[p]);
  double d = 0.0;
  if (!(fi > 0.0)) fail = true;
  else d = deviance(fi, ws.b.X[p]);
  ws.c1[p] = d;
}

// FP32 splines, delta: the change of the error from the start of the step
// (ROI and spline cell unchanged); else the absolute error.
__device__ __forceinline__ void team_pixel_trial(const ModelCfg& cfg, const FrameSet<float>& fs, long long fbase,
                                                 TeamWS<float>& ws, const PeakRec& o, const PeakRec& t,
                                                 const SplinePos& s, bool delta, int p, bool& fail) {
  int rx, ry;
  roi_rc(ws.b.roi, p, rx, ry);
  const float rq = ws.b.R[p];
  if (delta) {
    const float h1 = (float)t.p[PH];
    const float dh = (float)(t.p[PH] - o.p[PH]);
    const float dbg = (float)(t.p[PBG] - o.p[PBG]);
    const float dpsf = spline_dot(cfg, fs.aij, spline_cell(cfg, s.zi, ry + s.ys, rx + s.xs), ws.b.xt);
    const float df = rq * fmaf(h1, dpsf, dh * ws.psf0[p]) + dbg * rq * ws.b.IC[p];
    const float f0 = ws.b.f0[p];
    ff m{0.0f, 0.0f};
    float c = 0.0f, r = 0.0f;
    if (!(f0 + df > 0.0f)) {
      fail = true;
    } else {
      const float t1h = ws.t1[p];
      m = ff_mul_raw(ff{df, 0.0f}, ff{t1h, ws.t1l[p]});
      const float xv = fmaf(-0.5f * t1h, f0, f0);
      c = 2.0f * xv;
      r = r_minus_log1p(__fdiv_rn(df, f0));
    }
    ws.c0[p] = c;
    ws.c1[p] = r;
    ws.c2[p] = m.h;
    ws.c3[p] = m.l;
  } else {
    const float psf = spline_value_ff(cfg, fs.aij, ws.b, s, rx, ry).h;
    const float bgT = (float)t.p[PBG];
    const float fi = ws.b.Fb[p] + contrib_f(t.p[PH], psf, rq) + bg_div(ws.b.Bs[p] + bgT * rq, ws.b.IC[p]);
    float c = 0.0f, r = 0.0f;
    if (!(fi > 0.0f)) {
      fail = true;
    } else {
      const float x = ws.b.X[p];
      c = 2.0f * x;
      r = r_minus_log1p((fi - x) * rcp_approx(x));
    }
    ws.c0[p] = c;
    ws.c1[p] = r;
  }
}

// Their sum (one warp; every lane gets it).
__device__ inline double team_trial_sum(const ModelCfg& cfg, const TeamWS<double>& ws, bool, int lane) {
  double dev = 0.0;
  for (int p = lane; p < cfg.nroi; p += 32) dev += ws.c1[p];
  return warp_sum(dev);
}
__device__ inline double team_trial_sum(const ModelCfg& cfg, const TeamWS<float>& ws, bool delta, int lane) {
  ff s1{0.0f, 0.0f};
  float s2 = 0.0f;
  for (int p = lane; p < cfg.nroi; p += 32) {
    if (delta) ff_acc(s1, ff{ws.c2[p], ws.c3[p]});
    s2 = fmaf(ws.c0[p], ws.c1[p], s2);
  }
  if (!delta) return warp_sum_ff(s2);
  s1 = fast_two_sum(s1.h, s1.l);
  return ff_to_double(warp_sum_ffv(s1)) + warp_sum_ff(s2);
}

// The trial's contribution (height h, background bg) at pixel p of its ROI
// (image pixel k).
__device__ __forceinline__ void team_trial_contrib(const ModelCfg& cfg, const FrameSet<double>& fs,
                                                   const TeamWS<double>& ws, double h, double bg, const SplinePos&,
                                                   int p, int, int, long long k, Q2& cf, Q2& cb) {
  const double rq = ws.b.R[p];
  cf = quant_t<double>(contrib_f(h, ws.b.psf[p], rq));
  cb = quant_t<double>(contrib_bg(bg, rq, __ldg(fs.scmos + k)));
}
__device__ __forceinline__ void team_trial_contrib(const ModelCfg& cfg, const FrameSet<float>& fs,
                                                   const TeamWS<float>& ws, double h, double bg, const SplinePos& s,
                                                   int p, int rx, int ry, long long k, Q2& cf, Q2& cb) {
  spl32_contrib(spline_value_ff(cfg, fs.aij, ws.b, s, rx, ry), ff_from_double(h), ff_from_double(bg),
                ws.b.R[p], __ldg(fs.scmos + k), cf, cb);
}

// What the step needs of its own record, by the first NT threads.
template <int NT, typename T>
__device__ inline void team_prologue(const ModelCfg& cfg, const FrameSet<T>& fs, const PeakRec* recp, TeamWS<T>& ws,
                                     int tid) {
  if (tid < 8) {
    const double2 v = __ldcg(reinterpret_cast<const double2*>(recp) + tid);
    reinterpret_cast<double2*>(ws.b.orig)[tid] = v;
    reinterpret_cast<double2*>(ws.b.w)[tid] = v;
    reinterpret_cast<double2*>(ws.b.t)[tid] = v;
  } else if (tid < 8 + NCOUNTERS) {
    reinterpret_cast<int*>(ws.b.scratch)[tid - 8] = 0;
  }
  bar_sync(1, NT);
  const PeakRec& o = *ws.b.orig;
  team_tables(cfg, o, ws, tid, 1, NT, true);
  double gx, gy;
  z_factors(cfg, cfg.model, o, gx, gy);
  const SplinePos s0 = team_pos<T>(cfg, o);
#pragma unroll 1
  for (int p = tid; p < cfg.nroi; p += NT) team_pixel_static(cfg, fs, ws, o, s0, (T)gx, (T)gy, p);
}

// The step, after team_prologue and a barrier (all threads; see lm_step_g32).
template <int NT, typename T>
__device__ bool team_step(const ModelCfg& cfg, const FrameSet<T>& fs, long long fbase, PeakRec* recp, bool unbounded,
                          int dil, TeamWS<T>& ws, TeamCtl& tc, int* ctr_out, int tid) {
  constexpr int W = AccW<T>::W;
  const int lane = tid & 31, wid = tid >> 5;
  const PeakRec& orig = *ws.b.orig;
  const int k = cfg.jac;

  // -- 1. starting error, Jacobian / Hessian (multi_fit.c:1107-1142); the
  // subtraction (:1141) is deferred to the write-back
  bool fail = false;
#pragma unroll 1
  for (int p = tid; p < cfg.nroi; p += NT) team_pixel_start(cfg, fs, fbase, ws, orig, p, fail);
  const bool fail0 = __syncthreads_or(fail);
  team_sums(cfg, ws, wid, NT / 32, lane);
  __syncthreads();
  if (wid == 0) {
    team_close_sums(cfg, ws, lane);
  } else {
    double se = team_start_error(cfg, ws, tid, NT);
    if (tid == 32) {
      // a start with f <= 0 keeps the record's error
      tc.se = fail0 ? orig.error : se;
      if (fail0) reinterpret_cast<int*>(ws.b.scratch)[C_STARTFAIL]++;
    }
  }

  // -- 2. LM loop (multi_fit.c:1145-1325); warp 0 holds the scalar state of the
  // working record (from_se: its error is the step's start error)
  int* ctr = reinterpret_cast<int*>(ws.b.scratch);
  double lambda = orig.lambda, error = 0.0;
  int its = orig.iterations, status = orig.status;
  bool from_se = true;
  int cax = orig.xi, cay = orig.yi;   // anchor of the base arrays
  bool reloaded = false;              // FP32: a trial took the absolute path
  const SplinePos s0 = team_pos<T>(cfg, orig);
  int act = ACT_CONTINUE;
  for (;;) {
    if (wid == 0) {
      while (act == ACT_CONTINUE) {
        // lambda bound and iteration count (multi_fit.c:1153-1171)
        if (dbl_gt_pos(lambda, LAMBDA_MAX)) {
          if (lane == 0) ctr[C_LOST]++;
          status = ERROR;
          act = ACT_BREAK;
          break;
        }
        its++;
        if (lane == 0) ctr[C_ITER]++;
        status = RUNNING;
        // damped solve (multi_fit.c:1174-1203)
        double b[MAX_JAC];
        const int info = __shfl_sync(0xffffffffu, solve_damped<T>(ws.b, k, lambda, b, lane), 0);
        if (info != 0) {
          if (lane == 0) ctr[C_DPOSV]++;
          status = ERROR;
          lambda = lambda * LAMBDA_UP;
          continue;
        }
        double dl = 0.0;
#pragma unroll
        for (int j = 0; j < MAX_JAC; j++) {
          if (j < k) {
            const double v = __shfl_sync(0xffffffffu, b[j], 0);
            if (lane == j) dl = v;
          }
        }
        const int c = team_update(cfg, orig, *ws.b.t, dl, lane);
        const PeakRec& t = *ws.b.t;
        if (c) {
          if (lane == 0) ctr[c == 1 ? C_MARGIN : C_NEGH]++;
          // mFitResetPeak multi_fit.c:1788-1798
          its = orig.iterations;
          error = orig.error;
          from_se = false;
          lambda = lambda * LAMBDA_UP;
          status = ERROR;
        } else if (!unbounded && (abs(t.xi - orig.xi) > dil || abs(t.yi - orig.yi) > dil)) {
          act = ACT_ESCAPE;
        } else {
          act = ACT_EVAL;
        }
      }
      if (lane == 0) tc.act = act;
    }
    __syncthreads();
    act = tc.act;
    if (act != ACT_EVAL) break;
    // -- trial evaluation: shape, add, error (multi_fit.c:1229-1256)
    const PeakRec& t = *ws.b.t;
    const SplinePos s = team_pos<T>(cfg, t);
    bool delta = false;
    if constexpr (sizeof(T) == 4) {
      delta = !reloaded && t.xi == orig.xi && t.yi == orig.yi && s.xs == s0.xs && s.ys == s0.ys && s.zi == s0.zi;
      if (delta) diff_tables(cfg, orig, t, s0, s, ws.b, tid, NT);
    }
    if (sizeof(T) == 4 ? (!delta && (!reloaded || t.xi != cax || t.yi != cay)) : (t.xi != cax || t.yi != cay)) {
      team_load_base(cfg, fs, fbase, ws, orig, t.xi, t.yi, tid, NT);
      cax = t.xi;
      cay = t.yi;
      reloaded = true;
    }
    team_tables(cfg, t, ws, tid, 0, NT, false);
    fail = false;
#pragma unroll 1
    for (int p = tid; p < cfg.nroi; p += NT) team_pixel_trial(cfg, fs, fbase, ws, orig, t, s, delta, p, fail);
    // Past this barrier warp 0 may make the next trial of t: what the other
    // warps still need of it is read before.  (The solve writes none of the
    // tables they read; the next trial's are made behind the barrier above.)
    const bool home = cax == orig.xi && cay == orig.yi && t.xi == orig.xi && t.yi == orig.yi;
    const double h = t.p[PH], bg = t.p[PBG];
    fail = __syncthreads_or(fail);
    if (wid == 0) {
      const double dev = team_trial_sum(cfg, ws, delta, lane);
      const double se = tc.se;
      act = ACT_CONTINUE;
      if (!fail) {
        const double e1 = delta ? se + dev : dev;
        // change of the error, exact from the differential evaluation
        const double change = delta ? dev : e1 - se;
        if (delta ? (change > 0.0) : (e1 > se)) {
          if ((change / se) < cfg.tol) {
            status = CONVERGED;
            act = ACT_BREAK_ADDED;
          }
        } else {
          if ((-change / se) < cfg.tol) {
            status = CONVERGED;
          } else if (dbl_gt_pos(lambda, LAMBDA_MIN)) {
            lambda = LAMBDA_DOWN * lambda;
          }
          act = ACT_BREAK_ADDED;
        }
        error = e1;
        from_se = false;
      }
      if (act == ACT_CONTINUE) {
        if (lane == 0) ctr[fail ? C_NEGFI : C_NONDECR]++;
        its = orig.iterations;
        error = orig.error;
        from_se = false;
        lambda = lambda * LAMBDA_UP;
        status = fail ? ERROR : orig.status;
      }
    } else if constexpr (sizeof(T) == 4) {
      // the trial's change of the fit image, while warp 0 decides
      if (home) {
#pragma unroll 1
        for (int p = tid - 32; p < cfg.nroi; p += NT - 32) {
          int rx, ry;
          roi_rc(ws.b.roi, p, rx, ry);
          Q2 cf, cb;
          team_trial_contrib(cfg, fs, ws, h, bg, s, p, rx, ry, pix_index(cfg, orig.xi, orig.yi, rx, ry), cf, cb);
          ws.q1f[p] = cf.h - ws.q0f[p];
          ws.q1b[p] = cb.h - ws.q0b[p];
        }
      }
    }
  }

  // -- 3. write back: the net change of the fit image
  if (act == ACT_ESCAPE) return true;   // nothing was changed
  const bool added_end = act == ACT_BREAK_ADDED;
  const PeakRec& t = *ws.b.t;
  const bool same = added_end && t.xi == orig.xi && t.yi == orig.yi;
  const SplinePos s = team_pos<T>(cfg, t);
#pragma unroll 1
  for (int p = tid; p < cfg.nroi; p += NT) {
    int rx, ry;
    roi_rc(ws.b.roi, p, rx, ry);
    const long long k0 = pix_index(cfg, orig.xi, orig.yi, rx, ry);
    if (same) {
      Q2 cf, cb;
      if constexpr (sizeof(T) == 4) {
        cf = Q2{ws.q1f[p], 0};
        cb = Q2{ws.q1b[p], 0};
      } else {
        Q2 of, ob;
        team_trial_contrib(cfg, fs, ws, t.p[PH], t.p[PBG], s, p, rx, ry, k0, cf, cb);
        team_start_contrib(fs, ws, orig, p, ws.b.R[p], __ldg(fs.scmos + k0), of, ob);
        cf = q_sub(cf, of);
        cb = q_sub(cb, ob);
      }
      acc_red<W>(fs.f, fbase + k0, cf, +1);
      acc_red<W>(fs.bg, fbase + k0, cb, +1);
    } else {
      Q2 cf, cb;
      team_start_contrib(fs, ws, orig, p, __ldg(fs.rqe + k0), __ldg(fs.scmos + k0), cf, cb);
      acc_red<W>(fs.f, fbase + k0, cf, -1);
      acc_red<W>(fs.bg, fbase + k0, cb, -1);
      atomicAdd(fs.cnt + fbase + k0, -1);
      if (added_end) {
        const long long k1 = pix_index(cfg, t.xi, t.yi, rx, ry);
        team_trial_contrib(cfg, fs, ws, t.p[PH], t.p[PBG], s, p, rx, ry, k1, cf, cb);
        acc_red<W>(fs.f, fbase + k1, cf, +1);
        acc_red<W>(fs.bg, fbase + k1, cb, +1);
        atomicAdd(fs.cnt + fbase + k1, 1);
      }
    }
  }
  if (wid == 0) {
    // the record the step ends on
    PeakRec& e = added_end ? *ws.b.t : *ws.b.w;
    if (lane == 0) {
      e.lambda = lambda;
      e.error = from_se ? tc.se : error;
      e.status = status;
      e.iterations = its;
      e.added = orig.added - 1 + (added_end ? 1 : 0);
    }
    __syncwarp();
    if (lane < 8) reinterpret_cast<double2*>(recp)[lane] = reinterpret_cast<const double2*>(&e)[lane];
  } else if (wid == 1 && lane < NCOUNTERS) {
    ctr_out[lane] = ctr[lane];
  }
  return false;
}

}  // namespace sa
