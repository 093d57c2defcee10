// sa_launch_impl.cuh -- definitions of the launchers; included once per
// pixel type by sa_launch_f32.cu / sa_launch_f64.cu.
#pragma once

#include "sa_kernels.cuh"
#include "sa_launch.h"

namespace sa {

constexpr int SWEEP_BLOCK = 128;    // 4 warps, one peak each (fewer where their workspaces do not fit)
constexpr int CTA_BLOCK = 1024;     // per-frame kernels
constexpr int AUX_BLOCK = 256;      // warp-per-peak auxiliary kernels without a workspace

// Threads of a warp-per-peak auxiliary CTA with a workspace per warp.
static inline int aux_block(const ModelCfg& cfg) { return 32 * aux_warps(cfg); }

// Shared bytes of the sweep CTA's ROI pixel table (after the workspaces).
static inline size_t roi_table_bytes(int nroi) { return ((size_t)nroi * 2 + 15) & ~(size_t)15; }

// The kernels of a configuration: the FP32 Gaussian models have one
// instantiation each, everything else shares the generic step.  team_*: the
// kernels that step a peak per CTA (null: none).
template <typename T>
struct Kernels {
  void (*sweep)(ModelCfg, FrameSet<T>) = k_sweep<T, -1>;
  void (*tail)(ModelCfg, FrameSet<T>, int) = k_tail<T, -1>;
  void (*team_sweep)(ModelCfg, FrameSet<T>) = nullptr;
  void (*team_tail)(ModelCfg, FrameSet<T>, int) = nullptr;
  int team_threads = 0;
  size_t team_bytes = 0;

  template <typename S>
  void team(const ModelCfg& cfg) {
    team_sweep = k_sweep_team<S>;
    team_tail = k_tail_team<S>;
    team_threads = S::THREADS;
    team_bytes = S::bytes(cfg);
  }
  template <int M>
  void g32(const ModelCfg& cfg) {
    sweep = k_sweep<T, M>;
    tail = k_tail<T, M>;
    team<StepG32<M>>(cfg);
  }
};

template <typename T>
static Kernels<T> kernels(const ModelCfg& cfg) {
  Kernels<T> k;
  if constexpr (sizeof(T) == 4) {
    switch (cfg.model) {
      case M_2DFIXED: k.template g32<M_2DFIXED>(cfg); break;
      case M_2D: k.template g32<M_2D>(cfg); break;
      case M_3D: k.template g32<M_3D>(cfg); break;
      case M_Z: k.template g32<M_Z>(cfg); break;
      default: k.template team<StepTeam<float, 1>>(cfg); break;
    }
  } else {
    if (is_fft(cfg.model)) k.template team<StepTeam<double, 2>>(cfg);
    else if (is_pupil(cfg.model)) k.template team<StepTeam<double, 3>>(cfg);
    else if (is_spline(cfg.model)) k.template team<StepTeam<double, 1>>(cfg);
    else k.template team<StepTeam<double, 0>>(cfg);
  }
  return k;
}

template <typename T>
cudaError_t Launch<T>::configure(const ModelCfg& cfg, Shapes* sh) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int nsm = 0, max_smem = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const Kernels<T> k = kernels<T>(cfg);
  const size_t ws = warp_ws_bytes<T>(cfg, cfg.nroi);
  // four warps per sweep CTA, or as many as fit where their workspaces
  // (large ROIs in the FP64 engine, the pupil model) do not
  int wpc = SWEEP_BLOCK / 32;
  while (wpc > 1 && ws * wpc + roi_table_bytes(cfg.nroi) > (size_t)max_smem) wpc--;
  sh->warps = wpc;
  sh->smem = ws * wpc + roi_table_bytes(cfg.nroi);
  const size_t ws0 = warp_ws_bytes<T>(cfg, 0);
  const size_t grid_bytes = (size_t)(cfg.gx * cfg.gy + 1) * sizeof(int);
  const size_t s_cta_ws = ws0 * (size_t)cta_ws_warps(cfg);
  sh->cta_smem = s_cta_ws > grid_bytes ? s_cta_ws : grid_bytes;
  sh->warp_smem = ws0 * (size_t)aux_warps(cfg);
  // The limit is a property of the kernel, shared by every handle of the
  // process (handles of different models and ROI sizes may run side by
  // side), so it is raised to the device maximum rather than to this
  // handle's need.
  auto raise_limit = [max_smem](const void* fn, size_t need) {
    cudaFuncAttributes a;
    cudaError_t r = cudaFuncGetAttributes(&a, fn);
    if (r != cudaSuccess) return r;
    const int room = max_smem - (int)a.sharedSizeBytes;
    if (room < (int)need) return cudaErrorInvalidConfiguration;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, room);
  };
  struct {
    const void* fn;
    size_t need;
  } const all[] = {{(const void*)k.sweep, sh->smem},
                   {(const void*)k.tail, ws + roi_table_bytes(cfg.nroi)},
                   {(const void*)k_between<T>, sh->cta_smem},
                   // the warp-per-peak auxiliary kernels (their workspace is above the
                   // default 48 KB for the FFT PSF model)
                   {(const void*)k_newpeaks<T>, sh->warp_smem},
                   {(const void*)k_newpeaks_finder<T>, sh->warp_smem},
                   {(const void*)k_peak_props<T>, sh->warp_smem},
                   {(const void*)k_set_status<T>, sh->warp_smem}};
  for (const auto& a : all) {
    e = raise_limit(a.fn, a.need);
    if (e != cudaSuccess) return e;
  }
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.sweep, 32 * wpc, sh->smem);
  if (e != cudaSuccess) return e;
  sh->grid = nsm * (per_sm < 1 ? 1 : per_sm);
  // the team kernels, where a team's workspace fits
  sh->team_smem = k.team_bytes + roi_table_bytes(cfg.nroi);
  sh->team_threads = k.team_threads;
  if (k.team_sweep && raise_limit((const void*)k.team_sweep, sh->team_smem) == cudaSuccess &&
      raise_limit((const void*)k.team_tail, sh->team_smem) == cudaSuccess) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.team_sweep, k.team_threads, sh->team_smem);
    if (e != cudaSuccess) return e;
    sh->team_grid = nsm * per_sm;
  }
  return cudaSuccess;
}

template <typename T>
cudaError_t Launch<T>::between(const ModelCfg& cfg, const FrameSet<T>& fs, const Shapes& sh, bool start_only,
                               FramePoll* poll, unsigned* poll_err, cudaStream_t s) {
  k_between<T><<<fs.F, CTA_BLOCK, sh.cta_smem, s>>>(cfg, fs, start_only ? 1 : 0, poll, poll_err);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::sweep(const ModelCfg& cfg, const FrameSet<T>& fs, const Shapes& sh, int grid, bool team,
                             cudaStream_t s) {
  const Kernels<T> k = kernels<T>(cfg);
  if (team) k.team_sweep<<<grid, k.team_threads, sh.team_smem, s>>>(cfg, fs);
  else k.sweep<<<grid, 32 * sh.warps, sh.smem, s>>>(cfg, fs);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::tail(const ModelCfg& cfg, const FrameSet<T>& fs, const Shapes& sh, int tail_peaks,
                            cudaStream_t s) {
  const Kernels<T> k = kernels<T>(cfg);
  if (sh.team_grid > 0) k.team_tail<<<fs.F, k.team_threads, sh.team_smem, s>>>(cfg, fs, tail_peaks);
  else k.tail<<<fs.F, 32, (sh.smem - roi_table_bytes(cfg.nroi)) / sh.warps + roi_table_bytes(cfg.nroi), s>>>(cfg, fs, tail_peaks);
  return cudaGetLastError();
}

static inline int grid_for(long long n, int block) {
  long long g = (n + block - 1) / block;
  if (g > 4096) g = 4096;
  if (g < 1) g = 1;
  return (int)g;
}

template <typename T>
cudaError_t Launch<T>::new_image(const FrameSet<T>& fs, const void* img, int bits, int frame0,
                                 int nframes, cudaStream_t s) {
  const int g = grid_for(fs.npix * nframes, 256);
  if (bits == 32) k_new_image<T, float><<<g, 256, 0, s>>>(fs, (const float*)img, frame0, nframes);
  else if (bits == 16) k_new_image<T, unsigned short><<<g, 256, 0, s>>>(fs, (const unsigned short*)img, frame0, nframes);
  else k_new_image<T, double><<<g, 256, 0, s>>>(fs, (const double*)img, frame0, nframes);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::new_background(const FrameSet<T>& fs, const void* bg, int bits, int frame0,
                                      int nframes, cudaStream_t s) {
  const int g = grid_for(fs.npix * nframes, 256);
  if (bits == 32) k_new_background<T, float><<<g, 256, 0, s>>>(fs, (const float*)bg, frame0, nframes);
  else k_new_background<T, double><<<g, 256, 0, s>>>(fs, (const double*)bg, frame0, nframes);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::new_peaks(const ModelCfg& cfg, const FrameSet<T>& fs, const double* rows,
                                 int ncol, int ptype, const int* slots, const int* frames, int n,
                                 int do_add, size_t warp_smem, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int g = grid_for((long long)n * 32, aux_block(cfg));
  k_newpeaks<T><<<g, aux_block(cfg), warp_smem, s>>>(cfg, fs, rows, ncol, ptype, slots, frames, n, do_add);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::new_peaks_finder(const ModelCfg& cfg, const FrameSet<T>& fs, const int* slots,
                                        const int* frame_first, const int* frame_n, int nframes,
                                        size_t warp_smem, cudaStream_t s) {
  if (nframes <= 0) return cudaSuccess;
  k_newpeaks_finder<T><<<nframes, aux_block(cfg), warp_smem, s>>>(cfg, fs, slots, frame_first, frame_n);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::peak_error(const ModelCfg& cfg, const FrameSet<T>& fs, const int* slots,
                                  const int* frames, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int g = grid_for((long long)n * 32, AUX_BLOCK);
  k_peak_error<T><<<g, AUX_BLOCK, 0, s>>>(cfg, fs, slots, frames, n);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::peak_props(const ModelCfg& cfg, const FrameSet<T>& fs, const int* slots,
                                  const int* frames, int n, double* sum, double* fg, double* bg,
                                  double* jac, size_t warp_smem, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int g = grid_for((long long)n * 32, aux_block(cfg));
  k_peak_props<T><<<g, aux_block(cfg), warp_smem, s>>>(cfg, fs, slots, frames, n, sum, fg, bg, jac);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::set_status(const ModelCfg& cfg, const FrameSet<T>& fs, const int* slots,
                                  const int* frames, const int* status, int n, size_t warp_smem,
                                  cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int g = grid_for((long long)n * 32, aux_block(cfg));
  k_set_status<T><<<g, aux_block(cfg), warp_smem, s>>>(cfg, fs, slots, frames, status, n);
  return cudaGetLastError();
}

template <typename T>
cudaError_t Launch<T>::fit_image(const FrameSet<T>& fs, int frame, double* out, int residual,
                                 cudaStream_t s) {
  const int g = grid_for(fs.npix, 256);
  k_fit_image<T><<<g, 256, 0, s>>>(fs, frame, out, residual);
  return cudaGetLastError();
}

}  // namespace sa
