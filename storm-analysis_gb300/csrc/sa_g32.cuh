// sa_g32.cuh -- the LM step of one peak in the FP32 engine for the Gaussian
// models (2dfixed, 2d, 3d, Z); a team of TEAM_WARPS warps (one CTA) per peak.
//
// Team split.  What bounds a step is the latency of its dependent chain, not
// any pipe, and a sweep is a chain of steps, so the step's work is spread over
// the team's warps without changing any sum: what belongs to one ROI pixel is
// computed by one thread (TEAM pixels at once) and left in shared memory, and
// the per-pixel terms are then accumulated by one warp per group of sums,
// lane l taking pixels l, l + 32, ... in order and the warp's tree closing
// the sum.  Every sum keeps one order whatever the team's size.
//
// Precision plan.  The step's Hessian, its FP32 LDL^T factor and the
// per-pixel model shape are FP32; what decides the step -- the gradient and
// the change of the MLE error between the start of the step and a trial --
// is carried in float-float ("ff", ~48 bits) from exact inputs:
//   * the fit image and a copy of the data are fixed point, so f - x is
//     exact and becomes an ff residual without rounding;
//   * the shape factors exp(-t^2 w) are evaluated in ff per ROI row and
//     column (2 * roi exponentials per table, ff_exp) and kept as ff pairs;
//   * the change of the error for a trial at the same ROI anchor is
//     summed per pixel as  df * t1 + 2 x (r - log1p r),  t1 = 2 (f0 - x)/f0,
//     r = df / f0, with df = h1 psf1 - h0 psf0 (+ background change) in ff:
//     the first-order term, whose pixel sum cancels near convergence, is ff;
//     the second-order term is positive and FP32.
// This keeps the accept / reject / converged decisions of the reference
// (multi_fit.c:1229-1318, evaluated there in FP64) except where they sit
// within ~1e-12 of a threshold.
#pragma once

#include "sa_device.cuh"

namespace sa {

// Barrier ID of `count` threads of the CTA (whole warps); arrive: without
// waiting for the others.
__device__ __forceinline__ void bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

enum { ACT_EVAL = 0, ACT_CONTINUE = 1, ACT_BREAK = 2, ACT_BREAK_ADDED = 3, ACT_ESCAPE = 4 };

// Per-axis Jacobian factors of pass 1 in tab1 (ff pairs, stride ts):
// a1 = 2 h wx t_x, a2 = -h t_x^2 (x gx for Z), b1 = 2 h wy t_y, b2 = -h t_y^2
// (x gy), so that with ps = rqe * psf the Jacobian row is
//   2dfixed [ps, ps a1, ps b1, rqe]            (dao_fit.c:48-105)
//   2d      [ps, ps a1, ps b1, ps (a2+b2), rqe] (:409-467)
//   3d      [ps, ps a1, ps a2, ps b1, ps b2, rqe] (:811-871)
//   Z       [ps, ps a1, ps b1, ps (a2+b2), rqe] (:883-958)
template <int M>
__device__ inline void g32_grad_axis(const ModelCfg& cfg, const float* par, float* g, int ts, int side, int lane) {
  constexpr bool one_width = (M == M_2DFIXED) || (M == M_2D);
  const ff o = gpar(par, side ? GP_YO : GP_XO), wd = gpar(par, side && !one_width ? GP_WY : GP_WX);
  const ff H = gpar(par, GP_H);
  const ff HW = ff_mul(ff{2.0f * H.h, 2.0f * H.l}, wd);   // 2 h w
  const ff N = (M == M_Z) ? ff_neg(ff_mul(H, gpar(par, side ? GP_GY : GP_GX))) : ff_neg(H);
  g += side * 4 * ts;
#pragma unroll 1
  for (int i = lane; i < cfg.roi; i += 32) {
    const ff t = ff_add_f(o, (float)i);
    ff v = ff_mul(HW, t);
    g[i] = v.h;
    g[ts + i] = v.l;
    v = ff_mul(N, ff_mul(t, t));
    g[2 * ts + i] = v.h;
    g[3 * ts + i] = v.l;
  }
}

// The normal equations of a step as float-float values, in the memory of
// ws.jh: hi parts at [0, 36), lo parts at [36, 72); gradient first, then
// the packed upper Hessian (hes_index).
__device__ __forceinline__ float* g32_jh(WarpWS<float>& ws) { return reinterpret_cast<float*>(ws.jh); }

__device__ __forceinline__ ff shfl_ff(ff v, int src) {
  return ff{__shfl_sync(0xffffffffu, v.h, src), __shfl_sync(0xffffffffu, v.l, src)};
}

// The FP64 Cholesky of the ff normal equations (lane 0), the rare path of
// solve_g32 (an FP32 pivot <= 0), with the arithmetic of solve_fp64_lane0 /
// chol_solve.  Its matrix lives in shared scratch s (MAX_JAC^2 + MAX_JAC
// doubles; the factor overwrites the lower triangle) and its loops are not
// unrolled, so it adds no registers to the step; an out-of-line call would
// make the compiler save the step's live registers to the stack around it.
__device__ inline int solve_g32_fallback(const float* jh, int k, double lam, double* s, double* out) {
  double* A = s;
  double* b = s + MAX_JAC * MAX_JAC;
  int id = k;
#pragma unroll 1
  for (int l = 0; l < k; l++) {
    b[l] = (double)jh[l] + (double)jh[36 + l];
#pragma unroll 1
    for (int m = l; m < k; m++) {
      const double v = (double)jh[id] + (double)jh[36 + id];
      A[l * MAX_JAC + m] = (l == m) ? (1.0 + lam) * v : v;
      id++;
    }
  }
#pragma unroll 1
  for (int j = 0; j < k; j++) {
    double d = A[j * MAX_JAC + j];
#pragma unroll 1
    for (int q = 0; q < j; q++) d = __dsub_rn(d, __dmul_rn(A[j * MAX_JAC + q], A[j * MAX_JAC + q]));
    if (!(d > 0.0)) return j + 1;
    d = sqrt(d);
    A[j * MAX_JAC + j] = d;
#pragma unroll 1
    for (int i = j + 1; i < k; i++) {
      double t = A[j * MAX_JAC + i];
#pragma unroll 1
      for (int q = 0; q < j; q++) t = __dsub_rn(t, __dmul_rn(A[i * MAX_JAC + q], A[j * MAX_JAC + q]));
      A[i * MAX_JAC + j] = t / d;
    }
  }
#pragma unroll 1
  for (int i = 0; i < k; i++) {
    double t = b[i];
#pragma unroll 1
    for (int q = 0; q < i; q++) t = __dsub_rn(t, __dmul_rn(A[i * MAX_JAC + q], b[q]));
    b[i] = t / A[i * MAX_JAC + i];
  }
#pragma unroll 1
  for (int i = k - 1; i >= 0; i--) {
    double t = b[i];
#pragma unroll 1
    for (int q = i + 1; q < k; q++) t = __dsub_rn(t, __dmul_rn(A[q * MAX_JAC + i], b[q]));
    b[i] = t / A[i * MAX_JAC + i];
  }
  int st = 0;
#pragma unroll 1
  for (int i = 0; i < k; i++) {
    out[i] = b[i];
    if (isnan(b[i])) st = 1;
  }
  return st;
}

// Damped solve (H + lam diag H) d = b of the FP32 Gaussian step
// (multi_fit.c:1174-1203 with dposv :1839-1883), FP32 instructions only.
// Every lane factors the Jacobi-scaled matrix (LDL^T) and substitutes on its
// own, so the factorisation needs no shuffles; the two refinements compute
// the residual in float-float a row per lane and gather it to every lane.
// A pivot <= 0 hands the system to the FP64 Cholesky on lane 0, which
// decides failure as dposv does.  Lane j < K returns component j of the
// solution in dl (the K conversions to double run lane-parallel); the
// status is returned on every lane.
template <int K>
__device__ inline int solve_g32(WarpWS<float>& ws, double lam, double& dl, int lane) {
  const float* jh = g32_jh(ws);
  const ff L1 = ff_from_double(1.0 + lam);
  float sc[K], D[K], R[K], L[K][K], c[K];
  int status = 0;
  dl = 0.0;
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int id = hes_index(K, i, i);
    const float d = ff_mul(L1, ff{jh[id], jh[36 + id]}).h;
    if (!(d > 1.0e-30f && d < 1.0e30f)) status = 2;
    sc[i] = rsqrtf(d);
  }
  if (status == 0) {
#pragma unroll
    for (int j = 0; j < K; j++) {
      const int idj = hes_index(K, j, j);
      float dj = (ff_mul(L1, ff{jh[idj], jh[36 + idj]}).h * sc[j]) * sc[j];
#pragma unroll
      for (int m = 0; m < j; m++) dj = fmaf(-L[j][m] * L[j][m], D[m], dj);
      if (!(dj > 0.0f)) status = 2;
      D[j] = dj;
      const float inv = __frcp_rn(dj);
      R[j] = inv;
#pragma unroll
      for (int i = j + 1; i < K; i++) {
        float t = (jh[hes_index(K, i, j)] * sc[i]) * sc[j];
#pragma unroll
        for (int m = 0; m < j; m++) t = fmaf(-L[i][m] * L[j][m], D[m], t);
        L[i][j] = t * inv;
      }
    }
  }
  if (status == 0) {
    // L D L^T x = c, c = scaled right-hand side; d = x * scale
    auto substitute = [&](float (&v)[K]) {
#pragma unroll
      for (int i = 0; i < K; i++) {
#pragma unroll
        for (int m = 0; m < i; m++) v[i] = fmaf(-L[i][m], v[m], v[i]);
      }
#pragma unroll
      for (int i = 0; i < K; i++) v[i] = v[i] * R[i];
#pragma unroll
      for (int i = K - 1; i >= 0; i--) {
#pragma unroll
        for (int m = i + 1; m < K; m++) v[i] = fmaf(-L[m][i], v[m], v[i]);
      }
    };
    ff x[K];
#pragma unroll
    for (int i = 0; i < K; i++) c[i] = jh[i] * sc[i];
    substitute(c);
#pragma unroll
    for (int i = 0; i < K; i++) x[i] = two_prod(c[i], sc[i]);
    for (int it = 0; it < 2; it++) {
      // residual of row `lane` in float-float, then every row to every lane
      ff res{0.0f, 0.0f};
      if (lane < K) {
        res = ff{jh[lane], jh[36 + lane]};
#pragma unroll
        for (int j = 0; j < K; j++) {
          const int id = hes_index(K, lane, j);
          const ff a{jh[id], jh[36 + id]};
          res = ff_sub(res, ff_mul(j == lane ? ff_mul(L1, a) : a, x[j]));
        }
      }
#pragma unroll
      for (int i = 0; i < K; i++) c[i] = __shfl_sync(0xffffffffu, res.h, i) * sc[i];
      substitute(c);
#pragma unroll
      for (int i = 0; i < K; i++) x[i] = ff_add(x[i], two_prod(c[i], sc[i]));
    }
    ff xl = x[0];
#pragma unroll
    for (int j = 1; j < K; j++)
      if (lane == j) xl = x[j];
    dl = ff_to_double(xl);
    if (__any_sync(0xffffffffu, lane < K && isnan(xl.h))) status = 1;   // multi_fit.c:1857-1863
  }
  if (status == 2) {   // the same on every lane (the factorisation is)
    // scratch: the trial tables, rebuilt after every solve
    double* scr = reinterpret_cast<double*>(ws.tab1);
    int st = 0;
    if (lane == 0) st = solve_g32_fallback(jh, K, lam, scr, scr + MAX_JAC * MAX_JAC + MAX_JAC);
    __syncwarp();
    status = __shfl_sync(0xffffffffu, st, 0);
    dl = scr[MAX_JAC * MAX_JAC + MAX_JAC + (lane < K ? lane : 0)];
    __syncwarp();
  }
  return status;
}

struct G32Pix {
  long long F, B, X;
  float2 x;   // the data X 2^-36 as a float-float pair
  int C;
};

__device__ __forceinline__ void g32_load(const ModelCfg& cfg, const FrameSet<float>& fs, long long fbase,
                                         const unsigned short* roi, int ax, int ay, int p, G32Pix& v) {
  int rx, ry;
  roi_rc(roi, p, rx, ry);
  const long long k = pix_index(cfg, ax, ay, rx, ry);
  v.F = __ldcg(fs.f + fbase + k);
  v.B = __ldcg(fs.bg + fbase + k);
  v.C = __ldcg(fs.cnt + fbase + k);
  v.X = __ldg(fs.xq + fbase + k);
  v.x = __ldg(fs.xff + fbase + k);
}

// What a ROI pixel's terms need that only the peak's own record and the
// camera decide (no fit image): rqe, ps = rqe psf (FP32 for the Hessian, its
// float-float value for the gradient left in uh / ul), H0 psf (float-float)
// and the start contribution's fixed-point words, which the write-back takes
// out.  Computed while the sweep waits for the step's predecessors.
template <int M>
__device__ __forceinline__ void g32_pixel_static(const ModelCfg& cfg, const FrameSet<float>& fs,
                                                 WarpWS<float>& ws, int p) {
  const int ts = ws.ts;
  const float* t0 = ws.tab0;
  int rx, ry;
  roi_rc(ws.roi, p, rx, ry);
  const long long k = pix_index(cfg, ws.orig->xi, ws.orig->yi, rx, ry);
  const float rq = cfg.rqe_one ? 1.0f : (float)__ldg(fs.rqe + k);
  const ff H0 = gpar(ws.par0, GP_H);
  const ff psf = g32_psf(t0, ts, rx, ry);
  const ff pr = ff_mul_f(psf, rq);
  const ff hp = ff_mul(H0, psf);
  ws.Rs[p] = rq;
  ws.uh[p] = pr.h;
  ws.ul[p] = pr.l;
  if constexpr (M == M_Z) {
    ws.ps[p] = pr.h;
    ws.psl[p] = pr.l;
  } else {
    ws.ps[p] = t0[rx] * t0[2 * ts + ry] * rq;
  }
  ws.hph[p] = hp.h;
  ws.hpl[p] = hp.l;
  if (cfg.rqe_one && cfg.scmos_zero) {
    // uniform calibration: rqe 1 and sCMOS 0 change no bit of g32_contrib
    ws.q0f[p] = fixed_from_ff_call(hp);
  } else {
    Q2 qf, qb;
    g32_contrib<true>(t0, ts, H0, gpar(ws.par0, GP_BG), rx, ry, rq, cfg.scmos_zero ? 0.0f : (float)__ldg(fs.scmos + k), qf, qb);
    ws.q0f[p] = qf.h;
    ws.q0b[p] = qb.h;
  }
}

// Per-pixel state of the step's start, from the loaded pixel: f0 = f + bg /
// cnt and rho = f0 - x, exact up to the division (multi_fit.c:143; the data
// are kept in fixed point for this), t1 = 2 rho / f0, the Hessian weight
// t2 = 2 x / f0^2, the start error term (as its two factors, dc * dr) and
// what the gradient's sums share: u = t1 rqe psf.
//
// For the Z model t2 is (2 - t1) / f0 in float-float, rounded once to
// FP32.  Evaluated from the FP32-rounded x and f0 it carries ~2e-7 relative
// error per pixel, and that alone changes the reference's iteration count of
// ~0.2 % of the peaks of the astigmatic sCMOS workload (FP64 oracle with the
// same roundings emulated: 99.8 % of the peaks within the position
// tolerance); rounded once, 99.95 %.  The other Gaussian models keep the
// FP32 quotient (their fits match the oracle to 1e-5 px with it).
template <int M>
__device__ __forceinline__ void g32_pixel_state(const G32Pix& v, int p, WarpWS<float>& ws, bool& fail) {
  // f0 = rho + x with the data's float-float copy: two int64 conversions
  // fewer per pixel than converting f as well
  const float vx = v.x.x;
  const float cf = fx_s22(v.C);
  const ff bgc = ff_div(ff_from_fixed(v.B), ff{cf, 0.0f});
  const ff rho = ff_add(ff_from_fixed(v.F - v.X), bgc);
  const ff f0 = ff_add(rho, ff{v.x.x, v.x.y});
  float dc = 0.0f, dr = 0.0f;
  if (!(f0.h > 0.0f)) {
    fail = true;
  } else {
    // dev_res(rho.h, vx) = (2 vx) * dr, multiplied where it is accumulated
    dc = 2.0f * vx;
    dr = r_minus_log1p(rho.h * rcp_approx(vx));
  }
  ws.dc[p] = dc;
  ws.dr[p] = dr;
  const ff t1 = ff_div(ff{2.0f * rho.h, 2.0f * rho.l}, f0);
  ws.t1h[p] = t1.h;
  ws.t1l[p] = t1.l;
  ws.f0g[p] = f0.h;
  if constexpr (M == M_Z) {
    ws.T2s[p] = ff_div(ff_sub(ff{2.0f, 0.0f}, t1), f0).h;
  } else {
    const float iv = rcp_approx(f0.h);
    ws.T2s[p] = (2.0f * vx) * (iv * iv);
  }
  const ff u = ff_mul(t1, ff{ws.uh[p], ws.ul[p]});
  ws.uh[p] = u.h;
  ws.ul[p] = u.l;
  ws.Cs[p] = cf;
}

// Pass 1a: the start state of the ROI's pixels into the workspace, two
// pixels per thread in flight (their L2 round trips overlap).
template <int M>
__device__ inline void g32_gather(const ModelCfg& cfg, const FrameSet<float>& fs, long long fbase,
                                  const PeakRec& o, WarpWS<float>& ws, int tid, bool& fail) {
#pragma unroll 1
#pragma unroll 1
  for (int p = tid; p < cfg.nroi; p += 2 * TEAM) {
    G32Pix a, b;
    g32_load(cfg, fs, fbase, ws.roi, o.xi, o.yi, p, a);
    const bool two = p + TEAM < cfg.nroi;
    if (two) g32_load(cfg, fs, fbase, ws.roi, o.xi, o.yi, p + TEAM, b);
#pragma unroll 1
    for (int i = 0; i < (two ? 2 : 1); i++) {
      g32_pixel_state<M>(a, p + i * TEAM, ws, fail);
      a = b;
    }
  }
}

// Pass 1b, the normal equations from the start state: each warp sums its
// share over the ROI and closes it with the warp's tree (ff gradient; the
// Hessian's FP32 products and sums, except for the astigmatic Z model,
// whose fits turn on it: its iteration counts change on ~0.1 % of the
// peaks of the sCMOS workload when the Hessian carries FP32 rounding
// (measured against the FP64 oracle), so there the Jacobian row is
// float-float, every product is exact (two_prod) and the sums are
// float-float).  Shares (about equal instruction counts): gradient entries
// 2 w and 2 w + 1 on warp w and the Hessian on warp 3; for Z the gradient on
// warp 0 and five Hessian entries on each other warp.
template <int M>
__device__ __forceinline__ constexpr int g32_k() {
  return (M == M_2DFIXED) ? 4 : ((M == M_3D) ? 6 : 5);
}

// The gradient's factor of entry l at a pixel: entry l is sum u * factor
// (l = 0: u itself; l = K - 1: t1 rqe).
template <int M>
__device__ __forceinline__ ff g32_grad_factor(const float* gt, int ts, int rx, int ry, int l) {
  const ff A1{gt[rx], gt[ts + rx]}, A2{gt[2 * ts + rx], gt[3 * ts + rx]};
  const ff B1{gt[4 * ts + ry], gt[5 * ts + ry]}, B2{gt[6 * ts + ry], gt[7 * ts + ry]};
  if constexpr (M == M_3D) return l == 1 ? A1 : l == 2 ? A2 : l == 3 ? B1 : B2;
  return l == 1 ? A1 : l == 2 ? B1 : ff_add(A2, B2);
}

// Gradient entries [L0, L1) (L1 - L0 <= 8) of this warp into jh.
template <int M, int L0, int L1>
__device__ inline void g32_grad_part(const ModelCfg& cfg, WarpWS<float>& ws, float* jh, int lane) {
  constexpr int K = g32_k<M>(), N = L1 - L0;
  const int ts = ws.ts;
  const float* gt = ws.tab1;
  ff g[N];
#pragma unroll
  for (int i = 0; i < N; i++) g[i] = ff{0.0f, 0.0f};
#pragma unroll 1
  for (int p = lane; p < cfg.nroi; p += 32) {
    int rx, ry;
    roi_rc(ws.roi, p, rx, ry);
    const ff u{ws.uh[p], ws.ul[p]};
#pragma unroll
    for (int l = L0; l < L1; l++) {
      if (l == 0) ff_acc(g[l - L0], u);
      else if (l == K - 1) ff_acc(g[l - L0], ff_mul_f(ff{ws.t1h[p], ws.t1l[p]}, ws.Rs[p]));
      else ff_acc(g[l - L0], ff_mul_raw(u, g32_grad_factor<M>(gt, ts, rx, ry, l)));
    }
  }
  if constexpr (N > 2) {
    ff v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = i < N ? fast_two_sum(g[i < N ? i : 0].h, g[i < N ? i : 0].l) : ff{0.0f, 0.0f};
    const ff s = warp_reduce8_ff(v, lane);
    const int i = reduce8_index(lane);
    if ((lane & 3) == 0 && i < N) {
      jh[L0 + i] = s.h;
      jh[36 + L0 + i] = s.l;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) {
      const ff s = warp_sum_ffv(fast_two_sum(g[i].h, g[i].l));
      if (lane == i) {
        jh[L0 + i] = s.h;
        jh[36 + L0 + i] = s.l;
      }
    }
  }
}

// The FP32 Hessian (all entries) of this warp into jh.
template <int M>
__device__ inline void g32_hess_part(const ModelCfg& cfg, WarpWS<float>& ws, float* jh, int lane) {
  constexpr int K = g32_k<M>(), nhes = K * (K + 1) / 2;
  const int ts = ws.ts;
  const float* gt = ws.tab1;
  float acc[32];
#pragma unroll
  for (int i = 0; i < 32; i++) acc[i] = 0.0f;
#pragma unroll 1
  for (int p = lane; p < cfg.nroi; p += 32) {
    int rx, ry;
    roi_rc(ws.roi, p, rx, ry);
    const float t2 = ws.T2s[p], rq = ws.Rs[p], ps = ws.ps[p];
    const float a1 = gt[rx], a2 = gt[2 * ts + rx], b1 = gt[4 * ts + ry], b2 = gt[6 * ts + ry];
    float jf[K];
    jf[0] = ps;
    if constexpr (M == M_3D) {
      jf[1] = ps * a1;
      jf[2] = ps * a2;
      jf[3] = ps * b1;
      jf[4] = ps * b2;
    } else {
      jf[1] = ps * a1;
      jf[2] = ps * b1;
      if constexpr (M != M_2DFIXED) jf[3] = ps * (a2 + b2);
    }
    jf[K - 1] = rq;
#pragma unroll
    for (int l = 0; l < K; l++) {
#pragma unroll
      for (int m = l; m < K; m++) acc[l * K - (l * (l - 1)) / 2 + (m - l)] += t2 * jf[l] * jf[m];
    }
  }
  const float hv = warp_transpose_sum32(acc, lane);
  if (lane < nhes) {
    jh[K + lane] = hv;
    jh[36 + K + lane] = 0.0f;
  }
}

// Hessian entries [5 (w - 1), 5 w) of the Z model (packed upper triangle of
// five rows) on warp w = 1, 2, 3, float-float: the lanes' hi and lo words
// are summed by the same tree and added at the end.
template <int W>
__device__ inline void g32_hess_part_z(const ModelCfg& cfg, WarpWS<float>& ws, float* jh, int lane) {
  constexpr int K = 5, E0 = 5 * (W - 1);
  const int ts = ws.ts;
  const float* gt = ws.tab1;
  float hi[5], lo[5];
#pragma unroll
  for (int i = 0; i < 5; i++) hi[i] = lo[i] = 0.0f;
#pragma unroll 1
  for (int p = lane; p < cfg.nroi; p += 32) {
    int rx, ry;
    roi_rc(ws.roi, p, rx, ry);
    const float t2 = ws.T2s[p];
    const ff ps{ws.ps[p], ws.psl[p]};
    const ff A1{gt[rx], gt[ts + rx]}, A2{gt[2 * ts + rx], gt[3 * ts + rx]};
    const ff B1{gt[4 * ts + ry], gt[5 * ts + ry]}, B2{gt[6 * ts + ry], gt[7 * ts + ry]};
    ff jf[K];
    jf[0] = ps;
    jf[1] = ff_mul(ps, A1);
    jf[2] = ff_mul(ps, B1);
    jf[3] = ff_mul(ps, ff_add(A2, B2));
    jf[4] = ff{ws.Rs[p], 0.0f};
#pragma unroll
    for (int l = 0; l < K; l++) {
      const ff u = ff_mul_f(jf[l], t2);
#pragma unroll
      for (int m = l; m < K; m++) {
        const int id = l * K - (l * (l - 1)) / 2 + (m - l) - E0;
        if (id >= 0 && id < 5) {
          const ff x = ff_mul_raw(u, jf[m]);
          const ff sh = two_sum(hi[id], x.h);
          hi[id] = sh.h;
          lo[id] = __fadd_rn(lo[id], __fadd_rn(sh.l, x.l));
        }
      }
    }
  }
  // hi words' totals on the lanes with bit 4 clear, lo words' on the others
  float v[16];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    v[i] = i < 5 ? hi[i < 5 ? i : 0] : 0.0f;
    v[8 + i] = i < 5 ? lo[i < 5 ? i : 0] : 0.0f;
  }
  const ff half = warp_reduce16_to_ff(v, lane);
  const ff tot = ff_add(half, shfl_xor_ff(half, 16));
  const int i = (lane >> 1) & 7;
  if ((lane & 17) == 0 && i < 5) {
    jh[K + E0 + i] = tot.h;
    jh[36 + K + E0 + i] = tot.l;
  }
}

// The start error of the step (this warp; every lane gets it).
__device__ __forceinline__ double g32_dev_sum(const ModelCfg& cfg, const WarpWS<float>& ws, int lane) {
  float devf = 0.0f;
#pragma unroll 1
  for (int p = lane; p < cfg.nroi; p += 32) devf = fmaf(ws.dc[p], ws.dr[p], devf);
  return warp_sum_ff(devf);
}

template <int M>
__device__ inline void g32_pass1(const ModelCfg& cfg, WarpWS<float>& ws, int w, int lane) {
  constexpr int K = g32_k<M>();
  float* jh = g32_jh(ws);
  if constexpr (M == M_Z) {
    if (w == 0) {
      g32_grad_part<M, 0, K>(cfg, ws, jh, lane);
    } else if (w == 1) {
      g32_hess_part_z<1>(cfg, ws, jh, lane);
    } else if (w == 2) {
      g32_hess_part_z<2>(cfg, ws, jh, lane);
    } else {
      g32_hess_part_z<3>(cfg, ws, jh, lane);
    }
  } else {
    if (w == 0) {
      g32_grad_part<M, 0, 2>(cfg, ws, jh, lane);
    } else if (w == 1) {
      g32_grad_part<M, 2, 4>(cfg, ws, jh, lane);
    } else if (w == 2) {
      if constexpr (K > 4) g32_grad_part<M, 4, K>(cfg, ws, jh, lane);
    } else {
      g32_hess_part<M>(cfg, ws, jh, lane);
    }
  }
}

// Change of the MLE error for a trial at the start anchor (see the header
// comment), the terms of the thread's pixels; the trial tables are in tab1.
// First-order term (ff product) in uh / ul, second-order term as the two
// factors dc * dr.
template <typename T>
__device__ inline void g32_delta(const ModelCfg& cfg, WarpWS<T>& ws, int tid, bool& fail) {
  const int ts = ws.ts;
  const ff H1 = gpar(ws.par1, GP_H);
  const ff DBG = gpar(ws.par1, GP_DBG);
#pragma unroll 1
  for (int p = tid; p < cfg.nroi; p += TEAM) {
    int rx, ry;
    roi_rc(ws.roi, p, rx, ry);
    const float rq = ws.Rs[p];
    const ff d = ff_mul_f(ff_sub(ff_mul(H1, g32_psf(ws.tab1, ts, rx, ry)), ff{ws.hph[p], ws.hpl[p]}), rq);
    const ff bgd = ff_div(ff_mul_f(DBG, rq), ff{ws.Cs[p], 0.0f});
    const ff df = ff_add(d, bgd);
    const float f0 = ws.f0g[p];
    if (!(f0 + df.h > 0.0f)) {
      fail = true;
    } else {
      const float t1h = ws.t1h[p];
      const ff m = ff_mul_raw(df, ff{t1h, ws.t1l[p]});
      ws.uh[p] = m.h;
      ws.ul[p] = m.l;
      // x = f0 (1 - t1 / 2); the second-order term is FP32 anyway
      const float xv = fmaf(-0.5f * t1h, f0, f0);
      ws.dc[p] = 2.0f * xv;
      ws.dr[p] = r_minus_log1p(df.h * rcp_approx(f0));
    }
  }
}

// The sum of g32_delta's terms (this warp; every lane gets it).
__device__ __forceinline__ double g32_delta_sum(const ModelCfg& cfg, const WarpWS<float>& ws, int lane) {
  ff s1{0.0f, 0.0f};
  float s2 = 0.0f;
#pragma unroll 1
  for (int p = lane; p < cfg.nroi; p += 32) {
    ff_acc(s1, ff{ws.uh[p], ws.ul[p]});
    s2 = fmaf(ws.dc[p], ws.dr[p], s2);
  }
  s1 = fast_two_sum(s1.h, s1.l);
  return ff_to_double(warp_sum_ffv(s1)) + warp_sum_ff(s2);
}

// Is ROI pixel (rx, ry) inside the circular ROI (multi_fit.c:1031-1060)?
// Exact in FP32: every term is a multiple of 1/4.
__device__ __forceinline__ bool in_roi(int rx, int ry, int roi) {
  if (rx < 0 || ry < 0 || rx >= roi || ry >= roi) return false;
  const float c = 0.5f * (float)roi;
  const float dx = (float)rx - c + 0.5f, dy = (float)ry - c + 0.5f;
  return dx * dx + dy * dy <= c * c;
}

// MLE error of a trial at another anchor (FP32 with the exact fixed-point
// residual), the terms of the thread's pixels as the two factors dc * dr.
// The peak is still in the fit image at its start anchor o; its
// contribution is taken out here, pixel by pixel, exactly as the write-back
// will take it out.
template <typename T>
__device__ inline void g32_absolute(const ModelCfg& cfg, const FrameSet<T>& fs, long long fbase,
                                    const PeakRec& o, const PeakRec& t, WarpWS<T>& ws, int tid, bool& fail) {
  const int ts = ws.ts;
  const float h1 = ws.par1[2 * GP_H], bg1 = ws.par1[2 * GP_BG];   // (float) of the doubles
  const ff H0 = gpar(ws.par0, GP_H), BG0 = gpar(ws.par0, GP_BG);
  const int dx = t.xi - o.xi, dy = t.yi - o.yi;
#pragma unroll 1
  for (int p = tid; p < cfg.nroi; p += TEAM) {
    int rx, ry;
    roi_rc(ws.roi, p, rx, ry);
    const long long k = pix_index(cfg, t.xi, t.yi, rx, ry);
    long long F = __ldcg(fs.f + fbase + k), B = __ldcg(fs.bg + fbase + k);
    int C = __ldcg(fs.cnt + fbase + k);
    const float xv = (float)__ldg(fs.x + fbase + k);
    const float rq = cfg.rqe_one ? 1.0f : (float)__ldg(fs.rqe + k);
    const float sc = cfg.scmos_zero ? 0.0f : (float)__ldg(fs.scmos + k);
    const long long Xq = __ldg(fs.xq + fbase + k);
    const int ox = rx + dx, oy = ry + dy;   // the same image pixel in the start ROI
    if (in_roi(ox, oy, cfg.roi)) {
      Q2 qf, qb;
      g32_contrib<true>(ws.tab0, ts, H0, BG0, ox, oy, rq, sc, qf, qb);
      F -= qf.h;
      B -= qb.h;
      C -= 1;
    }
    const float psf = g32_psf(ws.tab1, ts, rx, ry).h;
    const float res = fx_to_float(F - Xq) + h1 * psf * rq +
                      (fx_to_float(B) + bg1 * rq + sc) * rcp_approx(fx_s22(C + 1));
    if (!(xv + res > 0.0f)) {
      fail = true;
    } else {
      ws.dc[p] = 2.0f * xv;
      ws.dr[p] = r_minus_log1p(res * rcp_approx(xv));
    }
  }
}

// Delta slot j of model M -> its parameter (apply_update's order,
// dao_fit.c:1777-1880).
template <int M>
__device__ __forceinline__ int g32_delta_param(int j) {
  if constexpr (M == M_3D) return j == 0 ? PH : j == 1 ? PX : j == 2 ? PXW : j == 3 ? PY : j == 4 ? PYW : PBG;
  if constexpr (M == M_Z) return j == 0 ? PH : j == 1 ? PX : j == 2 ? PY : j == 3 ? PZ : PBG;
  if constexpr (M == M_2D) return j == 0 ? PH : j == 1 ? PX : j == 2 ? PY : j == 3 ? PXW : PBG;
  return j == 0 ? PH : j == 1 ? PX : j == 2 ? PY : PBG;
}

// Ordered comparisons of a double with a nonzero finite constant, and the
// sign test, on the integer pipe: an FP64 comparison takes 64 cycles of the
// FP64 pipe and these sit on the step's critical path.  Doubles of one sign
// order as their bit patterns do; NaN compares false.
__device__ __forceinline__ bool dbl_gt_pos(double v, double c) {   // v > c, c > 0
  const long long b = __double_as_longlong(v);
  return b > __double_as_longlong(c) && b <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool dbl_lt_neg(double v, double c) {   // v < c, c < 0
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b > (unsigned long long)__double_as_longlong(c) && b <= 0xfff0000000000000ULL;
}
__device__ __forceinline__ bool dbl_negative(double v) {           // v < 0
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b > 0x8000000000000000ULL && b <= 0xfff0000000000000ULL;
}
// float -> double without the FP64 pipe (exact; subnormals take the conversion).
__device__ __forceinline__ double f2d(float f) {
  const unsigned u = __float_as_uint(f), e = u & 0x7f800000u;
  if (e == 0u ? (u << 1) != 0u : e == 0x7f800000u) return (double)f;
  const unsigned hi = (u & 0x80000000u) | (e == 0u ? 0u : ((u & 0x7fffffffu) >> 3) + 0x38000000u);
  return __hiloint2double((int)hi, (int)(u << 29));
}
__device__ __forceinline__ ff ff_from_double_i(double d) {
  const float h = __double2float_rn(d);
  return ff{h, __double2float_rn(d - f2d(h))};
}

// The trial of model M from the step's start record (a trial always starts
// from it: a rejected one resets the peak, mFitResetPeak multi_fit.c:1788-1798):
// apply_update + check_for on the trial record t, and the trial's parameter
// slots, one parameter per lane of warp 0.  Lane j < K applies delta j (dl)
// with apply_update's double operations -- the Z range clamp and widths from z
// (dao_fit.c:1828-1880), the ROI re-anchor (mFitUpdate multi_fit.c:1933-1946),
// mFitCheck and the width clamps of daoCheck2D / daoCheck3D (:1061-1119) -- and
// fills its slot of par1 (g32_params' double operations) from the value in
// its register; lane 6 fills GP_DBG, lane 7 the 2d model's y width, lanes 8
// and 9 the Z model's widths.  Each FP64 instruction runs once for all.
// Returns check_for's code (0 ok, 1 margin, 2 negative height) on every lane.
template <int M>
__device__ inline int g32_trial(const ModelCfg& cfg, WarpWS<float>& ws, double dl, int lane) {
  constexpr int K = g32_k<M>();
  const PeakRec& o = *ws.orig;
  PeakRec& t = *ws.t;
  const bool act = lane < K;
  const int src = act ? lane : (lane == 6 ? K - 1 : (M == M_2D && lane == 7 ? 3 : 0));
  const int pi = g32_delta_param<M>(src);
  const double dj = __shfl_sync(0xffffffffu, dl, src);
  const double p0 = o.p[pi];
  double nv = p0 - dj;
  if constexpr (M == M_Z) {
    if (pi == PZ) {
      if (nv < cfg.zmin) nv = cfg.zmin;
      if (nv > cfg.zmax) nv = cfg.zmax;
    }
  }
  // re-anchor on the PX and PY lanes
  const bool axis = act && (pi == PX || pi == PY);
  int ai = (pi == PY) ? o.yi : o.xi;
  // d: the value the lane's slot converts -- the offset from the ROI anchor
  // on the axis lanes, the background change on lane 6
  double d = nv - (lane == 6 ? p0 : (pi == PY ? ws.anchor[1] : ws.anchor[0]));
  if (axis && (dbl_lt_neg(d, -0.5) || dbl_gt_pos(d, 1.5))) {
    ai = (int)floor(nv);
    d = nv - (double)ai;
  }
  // mFitCheck: the anchors in the image, a non-negative height
  const int lim = (pi == PY) ? (cfg.ny - cfg.roi) : (cfg.nx - cfg.roi);
  const bool margin = __any_sync(0xffffffffu, axis && ((ai < 0) || (ai >= lim)));
  const bool negh = __any_sync(0xffffffffu, act && pi == PH && dbl_negative(nv));
  // width clamps (used only when the check passes; the trial is dropped otherwise)
  double cv = nv;
  if constexpr (M == M_2D || M == M_3D) {
    if (lane != 7 && (pi == PXW || (M == M_3D && pi == PYW))) {
      if (cv < cfg.wmin) cv = cfg.wmin;
      else if (cv > cfg.wmax) cv = cfg.wmax;
    }
  }
  if (act) {
    t.p[pi] = cv;
    if (M == M_2D && pi == PXW) t.p[PYW] = nv;   // the unclamped x width
    if (pi == PX) t.xi = ai;
    if (pi == PY) t.yi = ai;
  }
  int slot = pi == PX ? GP_XO : pi == PY ? GP_YO : pi == PXW ? GP_WX : pi == PYW ? GP_WY : pi == PBG ? GP_BG : GP_H;
  bool put = act && !(M == M_Z && pi == PZ);
  double v = axis ? -d - cfg.xoff : cv;
  if (lane == 6) {
    slot = GP_DBG;
    put = true;
    v = d;
  } else if (M == M_2D && lane == 7) {
    slot = GP_WY;
    put = true;
  }
  if constexpr (M == M_Z) {
    // widths from the new z: wx on lane 8, wy on lane 9 (widths_from_z)
    const double z = __shfl_sync(0xffffffffu, nv, 3);   // delta 3 is PZ
    const bool sy = (lane == 9);
    const double c0 = sy ? cfg.wy[0] : cfg.wx[0], c1 = sy ? cfg.wy[1] : cfg.wx[1];
    const double c2 = sy ? cfg.wy[2] : cfg.wx[2], c3 = sy ? cfg.wy[3] : cfg.wx[3];
    const double c4 = sy ? cfg.wy[4] : cfg.wx[4];
    const double z0 = (z - c1) / c2;
    const double z1 = z0 * z0, z2 = z1 * z0, z3 = z2 * z0;
    const double tt = 1.0 + z1 + c3 * z2 + c4 * z3;
    const double wt = tt * tt, wv = 2.0 / (c0 * tt);
    if (lane == 8) {
      t.wxt = wt;
      t.p[PXW] = wv;
      slot = GP_WX;
    } else if (lane == 9) {
      t.wyt = wt;
      t.p[PYW] = wv;
      slot = GP_WY;
    }
    if (lane == 8 || lane == 9) {
      put = true;
      v = wv;
    }
  }
  const ff f = ff_from_double_i(v);
  if (put) {
    ws.par1[2 * slot] = f.h;
    ws.par1[2 * slot + 1] = f.l;
  }
  __syncwarp();
  return margin ? 1 : (negh ? 2 : 0);
}

// What the step of a peak needs before it reads the fit image: its record
// (ws.orig, and the records the step ends on, ws.w and ws.t), its shape tables
// (tab0) and Jacobian factors (tab1), its pixels' static terms.  Only the
// peak's own step changes its record, so this overlaps the sweep's dependency
// waits: the caller runs it on NW = 3 warps while the team's fourth one
// waits, or on all four.  The caller's next barrier orders the results for
// the team.
template <int M, int NW>
__device__ inline void g32_prologue(const ModelCfg& cfg, const FrameSet<float>& fs, const PeakRec* recp,
                                    WarpWS<float>& ws, int tid) {
  const int lane = tid & 31, w = tid >> 5;
  auto sync = []() { bar_sync(1, NW * 32); };
  if (w == 0) {
    if (lane < 8) {
      const double2 v = __ldcg(reinterpret_cast<const double2*>(recp) + lane);
      reinterpret_cast<double2*>(ws.orig)[lane] = v;
      reinterpret_cast<double2*>(ws.w)[lane] = v;
      reinterpret_cast<double2*>(ws.t)[lane] = v;
    }
    __syncwarp();
    g32_params(cfg, *ws.orig, nullptr, M == M_Z, ws.par0, lane);
  } else if (w == 1) {
    if (lane < NCOUNTERS) reinterpret_cast<int*>(ws.scratch)[lane] = 0;
  }
  sync();
  const float* par = ws.par0;
  if (w == 0) {
    if (lane < 2 * GP_N) ws.par1[lane] = par[lane];   // the slots a trial leaves as they are
    g32_table_axis(cfg, gpar(par, GP_XO), gpar(par, GP_WX), ws.tab0, ws.ts, lane);
  } else if (w == 1) {
    g32_table_axis(cfg, gpar(par, GP_YO), gpar(par, GP_WY), ws.tab0 + 2 * ws.ts, ws.ts, lane);
  } else if (w == 2) {
    g32_grad_axis<M>(cfg, par, ws.tab1, ws.ts, 0, lane);
    g32_grad_axis<M>(cfg, par, ws.tab1, ws.ts, 1, lane);
    if (lane < 2) ws.anchor[lane] = (double)(lane ? ws.orig->yi : ws.orig->xi);
  }
  sync();
#pragma unroll 1
  for (int p = tid; p < cfg.nroi; p += 32 * NW) g32_pixel_static<M>(cfg, fs, ws, p);
}

// The write-back's words of an accepted trial at the start anchor, one pixel:
// the change of the fit image (into q1f) and of the background sum (q1b;
// one value for all pixels with a uniform calibration).
__device__ __forceinline__ void g32_pixel_change(const ModelCfg& cfg, const FrameSet<float>& fs,
                                                 WarpWS<float>& ws, int p) {
  const int ts = ws.ts;
  int rx, ry;
  roi_rc(ws.roi, p, rx, ry);
  const ff H1 = gpar(ws.par1, GP_H);
  if (cfg.rqe_one && cfg.scmos_zero) {
    ws.q1f[p] = fixed_from_ff_call(ff_mul(H1, g32_psf(ws.tab1, ts, rx, ry))) - ws.q0f[p];
  } else {
    const long long k = pix_index(cfg, ws.orig->xi, ws.orig->yi, rx, ry);
    Q2 qf, qb;
    g32_contrib<true>(ws.tab1, ts, H1, gpar(ws.par1, GP_BG), rx, ry, ws.Rs[p],
                cfg.scmos_zero ? 0.0f : (float)__ldg(fs.scmos + k), qf, qb);
    ws.q1f[p] = qf.h - ws.q0f[p];
    ws.q1b[p] = qb.h - ws.q0b[p];
  }
}

// The step of a peak of Gaussian model M (cfg.model == M), after
// g32_prologue and a barrier (all threads of the team).  Warp 0 solves, sums
// the trial's error and decides; meanwhile the other warps sum the start
// error or prepare the write-back of the trial.  Returns true if the step
// escaped its footprint (nothing changed).
template <int M>
__device__ bool lm_step_g32(const ModelCfg& cfg, const FrameSet<float>& fs, long long fbase, PeakRec* recp,
                            bool unbounded, int dil, WarpWS<float>& ws, TeamCtl& tc, int* ctr_out, int tid) {
  const int lane = tid & 31, wid = tid >> 5;
  const PeakRec& orig = *ws.orig;
  constexpr int k = g32_k<M>();
  const int ts = ws.ts;

  // -- 1. starting error, gradient / Hessian (multi_fit.c:1107-1142).  The
  // reference subtracts the peak here (:1141) and adds the accepted trial
  // back.  No other team touches this ROI during the step, so the
  // subtraction is deferred to the write-back, which applies the net change
  // once; the trial evaluations account for it.
  bool fail = false;
  g32_gather<M>(cfg, fs, fbase, orig, ws, tid, fail);
  const bool fail0 = __syncthreads_or(fail);
  g32_pass1<M>(cfg, ws, wid, lane);
  __syncthreads();
  if (wid == 1) {
    // the start error and the convergence threshold (read after the trial's
    // barriers); a start with f <= 0 keeps the record's error
    double se = g32_dev_sum(cfg, ws, lane);
    if (fail0) se = orig.error;
    if (lane == 0) {
      tc.se = se;
      tc.small = se > 0.0 ? cfg.tol * se : -1.0;
      if (fail0) reinterpret_cast<int*>(ws.scratch)[C_STARTFAIL]++;
    }
  }

  // -- 2. LM loop (multi_fit.c:1145-1325); lane 0 of warp 0 holds the scalar
  // state of the working record: lambda, its, status and error (from_se: the
  // error is the step's start error).
  int* ctr = reinterpret_cast<int*>(ws.scratch);
  double lambda = orig.lambda, error = 0.0;
  int its = orig.iterations, status = orig.status;
  bool from_se = true;
  int act = ACT_CONTINUE;
  for (;;) {
    if (wid == 0) {
      // the next trial: solve, update and check, until one is to be
      // evaluated or the step ends
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
        double dl;
        const int info = solve_g32<k>(ws, lambda, dl, lane);
        if (info != 0) {
          if (lane == 0) ctr[C_DPOSV]++;
          status = ERROR;
          lambda = lambda * LAMBDA_UP;
          continue;
        }
        const int c = g32_trial<M>(cfg, ws, dl, lane);
        const PeakRec& t = *ws.t;
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
    if (wid == 0) g32_table_axis(cfg, gpar(ws.par1, GP_XO), gpar(ws.par1, GP_WX), ws.tab1, ts, lane);
    else if (wid == 1) g32_table_axis(cfg, gpar(ws.par1, GP_YO), gpar(ws.par1, GP_WY), ws.tab1 + 2 * ts, ts, lane);
    __syncthreads();
    const PeakRec& t = *ws.t;
    const bool is_delta = (t.xi == orig.xi) && (t.yi == orig.yi);
    fail = false;
    if (is_delta) g32_delta(cfg, ws, tid, fail);
    else g32_absolute(cfg, fs, fbase, orig, t, ws, tid, fail);
    fail = __syncthreads_or(fail);
    if (wid == 0) {
      double dev = is_delta ? g32_delta_sum(cfg, ws, lane) : g32_dev_sum(cfg, ws, lane);
      // A trial whose error overflows FP32 has an error astronomically above
      // the start error in the reference's FP64 too: reject it.
      if ((__double_as_longlong(dev) & 0x7fffffffffffffffLL) >= __double_as_longlong(1.0e300)) dev = 1.0e300;
      const double se = tc.se;
      const double change = is_delta ? dev : dev - se;
      // |change| / se < tol as a product for a positive start error (no
      // FP64 division on the step's critical path; the two forms differ
      // only within 1e-16 of the threshold, far below the engine's
      // float-float error change)
      const long long cb = __double_as_longlong(change), sb = __double_as_longlong(tc.small);
      const bool small = sb >= 0 ? (cb & 0x7fffffffffffffffLL) < sb : (fabs(change) / se < cfg.tol);
      if (fail || (cb > 0 && !small)) {
        if (lane == 0) ctr[fail ? C_NEGFI : C_NONDECR]++;
        its = orig.iterations;
        error = orig.error;
        from_se = false;
        lambda = lambda * LAMBDA_UP;
        status = fail ? ERROR : orig.status;
        act = ACT_CONTINUE;
      } else {
        error = is_delta ? se + dev : dev;
        from_se = false;
        if (small) status = CONVERGED;
        else if (dbl_gt_pos(lambda, LAMBDA_MIN)) lambda = LAMBDA_DOWN * lambda;
        act = ACT_BREAK_ADDED;
      }
      // The next trial writes the slots and may write the tables (the solver's
      // scratch) that the other warps read for the change: not before they
      // are done.  They are by now, or warp 0 would wait for them above.
      if (is_delta) bar_sync(2, TEAM);
    } else if (is_delta) {
#pragma unroll 1
      for (int p = tid - 32; p < cfg.nroi; p += TEAM - 32) g32_pixel_change(cfg, fs, ws, p);
      bar_arrive(2, TEAM);
    }
  }

  // -- 3. write back: the net change of the fit image (subtract the start
  // contribution, add the accepted one)
  if (act == ACT_ESCAPE) return true;   // nothing was changed
  const bool added_end = act == ACT_BREAK_ADDED;
  const PeakRec& t = *ws.t;
  // uniform calibration: BG * 1 + 0 at every pixel, quantised once
  const bool uniform = cfg.rqe_one && cfg.scmos_zero;
  const ff BG0 = gpar(ws.par0, GP_BG), BG1 = gpar(ws.par1, GP_BG);
  const long long b0 = fixed_from_ff_call(BG0), b1 = fixed_from_ff_call(BG1);
  if (added_end && t.xi == orig.xi && t.yi == orig.yi) {
    for (int p = tid; p < cfg.nroi; p += TEAM) {
      int rx, ry;
      roi_rc(ws.roi, p, rx, ry);
      const long long kk = fbase + pix_index(cfg, orig.xi, orig.yi, rx, ry);
      acc_red<1>(fs.f, kk, Q2{ws.q1f[p], 0}, +1);
      acc_red<1>(fs.bg, kk, Q2{uniform ? b1 - b0 : ws.q1b[p], 0}, +1);
    }
  } else {
#pragma unroll 1
    for (int p = tid; p < cfg.nroi; p += TEAM) {
      int rx, ry;
      roi_rc(ws.roi, p, rx, ry);
      const long long kk = fbase + pix_index(cfg, orig.xi, orig.yi, rx, ry);
      acc_red<1>(fs.f, kk, Q2{ws.q0f[p], 0}, -1);
      acc_red<1>(fs.bg, kk, Q2{uniform ? b0 : ws.q0b[p], 0}, -1);
      atomicAdd(fs.cnt + kk, -1);
    }
    if (added_end) {   // at another anchor
      const ff H1 = gpar(ws.par1, GP_H);
#pragma unroll 1
      for (int p = tid; p < cfg.nroi; p += TEAM) {
        int rx, ry;
        roi_rc(ws.roi, p, rx, ry);
        const long long k = pix_index(cfg, t.xi, t.yi, rx, ry);
        Q2 qf, qb;
        g32_contrib<true>(ws.tab1, ts, H1, BG1, rx, ry, cfg.rqe_one ? 1.0f : (float)__ldg(fs.rqe + k),
                    cfg.scmos_zero ? 0.0f : (float)__ldg(fs.scmos + k), qf, qb);
        acc_red<1>(fs.f, fbase + k, qf, +1);
        acc_red<1>(fs.bg, fbase + k, qb, +1);
        atomicAdd(fs.cnt + fbase + k, 1);
      }
    }
  }
  if (wid == 0) {
    // the record the step ends on
    PeakRec& e = added_end ? *ws.t : *ws.w;
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
