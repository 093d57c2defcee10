// sa_mp.cu -- launchers of the multi-plane kernels (sa_mp.cuh).
#include <algorithm>

#include "sa_mp.cuh"
#include "sa_mp.h"

namespace sa {

int mp_ws_bytes(const ModelCfg& cfg) { return (int)warp_ws_bytes<double>(cfg, cfg.nroi); }

static size_t al16(size_t b) { return (b + 15) & ~(size_t)15; }

// k_mp_sweep: per warp a workspace and a shape grid, per team its coupling
// state, the channels, the window's list of groups.
static size_t mp_smem_sweep(const MPParams& p) {
  const size_t wstride = (size_t)p.ws_bytes + al16((size_t)p.grid_doubles * 8);
  return (size_t)p.nc * p.teams * wstride + al16(sizeof(MPTeam) * p.teams) + al16(sizeof(MPChan) * p.nc) +
         sizeof(int) * (p.window + 2 * p.nc * p.window + (p.window + 31) / 32 + 2);
}

// k_mp_newpeaks: one warp.
size_t mp_smem(const MPParams& p) { return (size_t)p.ws_bytes + al16(sizeof(MPShared)) + (size_t)p.nc * sizeof(MPChan); }

static int g_max_smem = 0;

static cudaError_t mp_limits() {
  static bool done = false;
  if (done) return cudaSuccess;
  int dev = 0, max_smem = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  for (const void* fn : {(const void*)k_mp_sweep, (const void*)k_mp_newpeaks}) {
    cudaFuncAttributes a;
    e = cudaFuncGetAttributes(&a, fn);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - (int)a.sharedSizeBytes);
    if (e != cudaSuccess) return e;
    if (fn == (const void*)k_mp_sweep) g_max_smem = max_smem - (int)a.sharedSizeBytes;
  }
  done = true;
  return cudaSuccess;
}

cudaError_t mp_sweep(const MPChan* d_chans, const MPParams& p, int frames, cudaStream_t s) {
  cudaError_t e = mp_limits();
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 1;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long n = std::max(frames, 1);
  MPParams q = p;
  // A frame's CTAs (a cluster) and the groups stepping at once.  A step is
  // bound by the SM's FP64 pipes and by its own chain, so a frame takes the
  // more SMs the fewer frames there are: 8 CTAs of 2 teams each while every
  // CTA finds an SM of its own, 4 of 2 while the SMs hold few of them, 2 of 4
  // up to a frame an SM, then one CTA of MP_TEAMS and fewer teams (with less
  // to wait for in each frame), at least 2.  Frames of 256 x 256, 200 groups,
  // fits in ms with CTAs x teams 1 x 8 / 2 x 4 / 4 x 2 / 8 x 2: one frame 54 /
  // 39 / 33 / 27, 64 frames 86 / 71 / 67 / 76, 110 frames 93 / 91 / 82 / 104,
  // 152 frames 103 / 102 / 122 / 132, 256 frames 160 / 156 / 168 / - (5 teams
  // of one CTA; 151 with 4).
  q.cl = 8LL * frames <= sms ? 8 : 4LL * frames <= 3LL * sms ? 4 : frames <= sms ? 2 : 1;
  const int most = q.cl == 8 ? MP_BATCH : MP_TEAMS;
  q.batch = p.teams > 0 ? std::min(p.teams, MP_TEAMS)
                        : (int)std::max(2LL, std::min((long long)most, (MP_TEAMS * sms + n - 1) / n));
  q.cl = std::min(q.cl, q.batch);
  q.window = MP_WINDOW;
  const size_t limit = (size_t)g_max_smem;
  const int max_teams = MP_MAXCH * 2 / q.nc;
  q.teams = std::min((q.batch + q.cl - 1) / q.cl, max_teams);
  // a shorter list, then fewer teams where the workspaces fill the shared
  // memory; none: too many planes of a large PSF
  while (mp_smem_sweep(q) > limit) {
    if (q.window > 16) q.window /= 2;
    else if (q.teams > 1) q.teams--, q.window = MP_WINDOW;
    else return cudaErrorInvalidConfiguration;
  }
  q.batch = std::min(q.batch, q.teams * q.cl);
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(frames * q.cl);
  lc.blockDim = dim3(32 * q.nc * q.teams);
  lc.dynamicSmemBytes = mp_smem_sweep(q);
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = q.cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = q.cl > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&lc, k_mp_sweep, d_chans, q);
}

cudaError_t mp_newpeaks(const MPChan* d_chans, const MPParams& p, int frames, cudaStream_t s) {
  cudaError_t e = mp_limits();
  if (e != cudaSuccess) return e;
  k_mp_newpeaks<<<frames, 32, mp_smem(p), s>>>(d_chans, p);
  return cudaGetLastError();
}

}  // namespace sa
