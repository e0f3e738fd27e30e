// me_units.cu -- unit kernels (synthesis, Voigt, SVD, initial guess) and the
// launch dispatch.  The inversion kernel itself lives in me_invert.cuh.
//
#include <cuda_runtime.h>

#include "me_device.cuh"
#include "me_kernels.h"

namespace me {

namespace {

}  // namespace

// ---------------------------------------------------------------------------
// Building blocks exposed for the unit entry points.
// ---------------------------------------------------------------------------


// Syntheses of npix parameter sets (and, JAC, their Jacobians).  A block takes
// `per` pixels: its first threads set them up (the terms that do not depend
// on the wavelength) in shared memory, then all its threads take points
// (pixel, wavelength) in the order of the output, so that stores run along the
// wavelengths.  One thread per pixel stored 8 bytes every 32 nl (288 nl with
// the Jacobian) and left most of the device idle on maps of a few thousand
// pixels.
// flags (nullable): pixels without bit 0 get zeros instead; their parameters,
// which nothing has written, are not read.
// Measured on a B200, one thread per pixel against this: 262144 profiles of 60
// wavelengths, FP32, 912 -> 288 us; 10007 FP64 Jacobians of 112 wavelengths 1600
// -> 533 us; 37 FP32 Jacobians 147 -> 20 us (host call included).  The large FP32
// map is bound by instruction issue (0.84 per cycle and scheduler, DRAM at 21 %).
constexpr int kSynthThreads = 128;
template <class T>
constexpr int kSynthPixels = sizeof(T) == sizeof(float) ? 32 : 16;  // most per block

template <class T>
struct SynthPixel {
  SynthCall<T> c;
  T yy, inv_y;
  T rden[sizeof(T) == sizeof(float) ? kRden : 1];
  bool live;
};

enum SynthMode { kPlain, kFilter, kFilterSplit };  // no filter; with one: see launch_synth_t

template <class T, bool JAC, int MODE>
__global__ void __launch_bounds__(kSynthThreads)
    synth_kernel(const __grid_constant__ DevPlan P, const double *par, const unsigned char *flags,
                 long long npix, int per, double step7, double *prof, double *jac) {
  __shared__ T s_tab[100];
  __shared__ SynthPixel<T> s_px[kSynthPixels<T>];
  VoigtK<T> K;
  voigt_block_setup<T>(K, P, s_tab);
  const long long first = blockIdx.x * (long long)per;
  const int here = (int)(npix - first < per ? npix - first : per);
  if ((int)threadIdx.x < here) {
    SynthPixel<T> &o = s_px[threadIdx.x];
    const long long i = first + threadIdx.x;
    o.live = !flags || (flags[i] & 1);
    if (o.live) {
      double mp[9], step[9];
#pragma unroll
      for (int k = 0; k < 9; k++) {
        mp[k] = par[i * 9 + k];
        step[k] = P.step[k];
      }
      step[7] = step7;
      SynthCall<T> c;
      synth_setup<T>(c, mp, P, step);
      voigt_prepare<T>(K, c.p5, o.rden, 1);
      o.c = c;
      o.yy = K.yy;
      o.inv_y = K.inv_y;
    }
  }
  __syncthreads();
  const int nl = P.nl;
  const T ones[4] = {T(1), T(1), T(1), T(1)};
  K.rstride = 1;
  if constexpr (MODE == kFilterSplit) {
    // a point is a sub-wavelength; entry e of an observed value (the profiles,
    // then the Jacobian's J[s][k]) is summed over its sub-wavelengths in
    // order, from zero, by one thread (part: its sum so far, when the points of
    // a wavelength straddle two batches)
    constexpr int E = JAC ? 40 : 4;
    __shared__ T s_pt[kSynthThreads * E];
    __shared__ T s_part[E];
    const int ns = P.nsub, tid = threadIdx.x, total = here * nl * ns;
    for (int p0 = 0; p0 < total; p0 += kSynthThreads) {
      const int e = p0 + tid;
      const int p = e < total ? e / (nl * ns) : 0;
      if (e < total && s_px[p].live) {
        const SynthPixel<T> &o = s_px[p];
        K.yy = o.yy;
        K.inv_y = o.inv_y;
        K.rden = o.rden;
        T ys[4], Jq[4][9];
        me_point<T, JAC>(o.c, shift_wf<T>(o.c, P, e - p * nl * ns), K, ones, ys,
                         JAC ? Jq : nullptr);
#pragma unroll
        for (int s = 0; s < 4; s++) s_pt[tid * E + s] = ys[s];
        if (JAC) {
#pragma unroll
          for (int s = 0; s < 4; s++)
#pragma unroll
            for (int k = 0; k < 9; k++) s_pt[tid * E + 4 + s * 9 + k] = Jq[s][k];
        }
      }
      __syncthreads();
      const int p1 = p0 + kSynthThreads < total ? p0 + kSynthThreads : total;
      const int w0 = p0 / ns, w1 = (p1 - 1) / ns;
      T carry = T(0);
      for (int u = tid; u < (w1 - w0 + 1) * E; u += kSynthThreads) {
        const int w = w0 + u / E, m = u % E;
        const int q0 = w * ns > p0 ? w * ns : p0;
        const int q1 = (w + 1) * ns < p1 ? (w + 1) * ns : p1;
        T v = q0 == w * ns ? T(0) : s_part[m];
        if (s_px[w / nl].live)
          for (int q = q0; q < q1; q++) v += T(P.sub_w[q - w * ns]) * s_pt[(q - p0) * E + m];
        else
          v = T(0);
        if (q1 < (w + 1) * ns) {
          carry = v;
          continue;
        }
        const size_t i = (size_t)(first + w / nl);
        const int iw = w % nl;
        if (m < 4)
          prof[(i * 4 + m) * nl + iw] = (double)v;
        else
          jac[(i * 36 + m - 4) * nl + iw] = (double)v;
      }
      __syncthreads();
      if (p1 < (w1 + 1) * ns) {
        for (int u = tid; u < (w1 - w0 + 1) * E; u += kSynthThreads)
          if (u / E == w1 - w0) s_part[u % E] = carry;
        __syncthreads();
      }
    }
    return;
  }
  for (int e = threadIdx.x; e < here * nl; e += kSynthThreads) {
    const int p = e / nl, iw = e - p * nl;
    const SynthPixel<T> &o = s_px[p];
    const size_t i = (size_t)(first + p);
    double *out = prof + i * 4 * nl + iw;
    if (!o.live) {
#pragma unroll
      for (int s = 0; s < 4; s++) out[s * nl] = 0.0;
      continue;
    }
    K.yy = o.yy;
    K.inv_y = o.inv_y;
    K.rden = o.rden;
    T syn[4], J[4][9];
    channel_point<T, JAC, MODE == kFilter>(o.c, P, K, ones, iw, syn, JAC ? J : nullptr);
#pragma unroll
    for (int s = 0; s < 4; s++) out[s * nl] = (double)syn[s];
    if (JAC) {
      double *jo = jac + i * 36 * nl + iw;
#pragma unroll
      for (int s = 0; s < 4; s++)
#pragma unroll
        for (int k = 0; k < 9; k++) jo[(s * 9 + k) * nl] = (double)J[s][k];
    }
  }
}

template <class T>
__global__ void voigt_kernel(const DevPlan P, const double *nu, const double *a, long long n,
                             double *H, double *L) {
  __shared__ T s_tab[100];
  __shared__ T s_rden[kRden * 256];
  VoigtK<T> K;
  voigt_block_setup<T>(K, P, s_tab);
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const T y = T(a[i]);
  voigt_prepare<T>(K, y, s_rden + threadIdx.x, blockDim.x);
  const HL<T> r = voigt<T>(T(nu[i]), y, erfcx_t<T>(y), K);
  H[i] = (double)r.h;
  L[i] = (double)r.l;
}

__global__ void svd_kernel(const double *a, long long nmat, int n, double *u, double *w,
                           double *v, int *limit_hits) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= nmat) return;
  double am[81], vv[81], ww[9];
  for (int k = 0; k < n * n; k++) am[k] = a[i * n * n + k];
  const int hit = gr_svd(am, n, ww, vv);
  for (int k = 0; k < n * n; k++) {
    u[i * n * n + k] = am[k];
    v[i * n * n + k] = vv[k];
  }
  for (int k = 0; k < n; k++) w[i * n + k] = ww[k];
  if (hit && limit_hits) atomicAdd(limit_hits, 1);
}

__global__ void init_guess_kernel(const DevPlan P, const double *prof, long long npix,
                                  double *guess, double *extra, int *status) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= npix) return;
  PixelInit o;
  const int st = init_guess(prof + (size_t)i * 4 * P.nl, P, o, false);
  status[i] = st;
  for (int k = 0; k < 9; k++) guess[i * 9 + k] = st ? 0.0 : o.guess[k];
  extra[i * 5 + 0] = st ? 0.0 : o.norm0;
  extra[i * 5 + 1] = st ? 0.0 : o.normp;
  extra[i * 5 + 2] = st ? 0.0 : o.l70;
  extra[i * 5 + 3] = st ? 0.0 : o.l71;
  extra[i * 5 + 4] = st ? 0.0 : o.step7;
}

// ---------------------------------------------------------------------------
// Queue order of a learned start.  A pixel whose start is far from its profile
// tends to need many LM iterations and restarts; queued late, it runs on alone
// at the end of the batch while the GPU idles.  The misfit of each pixel's
// start -- the run -1 parameters exactly as the queue sets them up (Init_Guess,
// the network's free parameters, the bounds fold) -- is Loss_Function's chi^2
// (Src/LM_FIT.c:150-156; weights / sqrt(norm0), Src/ME_SOLVER.c:410-441) on
// every `stride`-th wavelength.  Pixels are queued by descending misfit in
// quarter-octave buckets, by a stable counting sort, so the order, and with it
// every result, is reproducible.  A pixel's steps are the same in any order;
// which kernel runs each of them (full rounds, lane-split rounds, the tail
// kernel) depends on when it is queued, so results agree with pixel order to
// rounding.
// ---------------------------------------------------------------------------
template <class T, bool FILT>
__global__ void start_misfit_kernel(const DevPlan P, const double *prof, const double *init_par,
                                    long long npix, int stride, unsigned char *key) {
  __shared__ T s_tab[100];
  __shared__ T s_rden[kRden * 128];
  VoigtK<T> K;
  voigt_block_setup<T>(K, P, s_tab);
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= npix) return;
  const int nl = P.nl;
  const double *pp = prof + (size_t)i * 4 * nl;
  PixelInit pin;
  if (init_guess(pp, P, pin, true) || P.nruns <= 0) {
    key[i] = (unsigned char)(kOrderBuckets - 1);  // skipped by the queue: last
    return;
  }
  double q[9], step[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double v = init_par[(size_t)i * 9 + k];
    q[k] = (P.fixed[k] || !isfinite(v)) ? pin.guess[k] : v;
    step[k] = P.step[k];
  }
  bounds_fold(q, P, pin.l70, pin.l71);
  step[7] = pin.step7;
  const double isn = 1.0 / sqrt(pin.norm0);
  SynthCall<T> c;
  synth_setup<T>(c, q, P, step);
  voigt_prepare<T>(K, c.p5, s_rden + threadIdx.x, blockDim.x);
  const T ones[4] = {T(1), T(1), T(1), T(1)};
  double chi = 0.0;
  int used = 0;
  for (int iw = 0; iw < nl; iw += stride, used++) {
    T syn[4];
    channel_point<T, false, FILT>(c, P, K, ones, iw, syn, nullptr);
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const double rd = ((double)syn[s] - pp[s * nl + iw]) * P.weights[s] * isn;
      chi += rd * rd;
    }
  }
  chi /= 4.0 * used;
  // bucket 0: chi^2 >= 2^32 or not finite; a quarter octave per bucket below,
  // down to bucket kOrderBuckets - 2 (chi^2 < 2^0.5 and all below)
  int b = 0;
  if (chi < 4294967296.0) {
    b = (int)floor((32.0 - log2(fmax(chi, 1e-300))) * 4.0);
    b = b < 0 ? 0 : (b > kOrderBuckets - 2 ? kOrderBuckets - 2 : b);
  }
  key[i] = (unsigned char)b;
}

// Stable counting sort of pixel indices by an 8-bit key, in three launches:
// per-block histograms of contiguous chunks (bucket-major), an exclusive scan
// of them, and a scatter in which each block walks its chunk in index order.
__global__ void order_hist_kernel(const unsigned char *key, long long n, long long chunk,
                                  int *hist) {
  __shared__ int h[kOrderBuckets];
  for (int t = threadIdx.x; t < kOrderBuckets; t += blockDim.x) h[t] = 0;
  __syncthreads();
  const long long lo = blockIdx.x * chunk;
  const long long hi = lo + chunk < n ? lo + chunk : n;
  for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) atomicAdd(&h[key[i]], 1);
  __syncthreads();
  for (int t = threadIdx.x; t < kOrderBuckets; t += blockDim.x)
    hist[(size_t)t * gridDim.x + blockIdx.x] = h[t];
}

// exclusive prefix sums of hist[0..m) in place; one block of 1024 threads
__global__ void __launch_bounds__(1024) order_scan_kernel(int *hist, int m) {
  __shared__ int part[1024];
  const int t = threadIdx.x;
  const int per = (m + 1023) / 1024;
  const int lo = t * per, hi = lo + per < m ? lo + per : m;
  int sum = 0;
  for (int i = lo; i < hi; i++) sum += hist[i];
  part[t] = sum;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {  // inclusive scan of the segment sums
    const int v = t >= o ? part[t - o] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  int run = part[t] - sum;
  for (int i = lo; i < hi; i++) {
    const int v = hist[i];
    hist[i] = run;
    run += v;
  }
}

__global__ void __launch_bounds__(256) order_scatter_kernel(const unsigned char *key, long long n,
                                                            long long chunk, const int *offs,
                                                            long long *order, long long first) {
  __shared__ int base[kOrderBuckets];
  __shared__ int wcnt[8][kOrderBuckets];
  for (int t = threadIdx.x; t < kOrderBuckets; t += blockDim.x) {
    base[t] = offs[(size_t)t * gridDim.x + blockIdx.x];
    for (int w = 0; w < 8; w++) wcnt[w][t] = 0;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long lo = blockIdx.x * chunk;
  const long long hi = lo + chunk < n ? lo + chunk : n;
  for (long long r0 = lo; r0 < hi; r0 += 256) {
    const long long i = r0 + threadIdx.x;
    const bool in = i < hi;
    const int k = in ? (int)key[i] : kOrderBuckets + lane;  // absent lanes match nobody
    const unsigned peers = __match_any_sync(0xffffffffu, k);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    const bool leader = lane == __ffs(peers) - 1;
    if (in && leader) wcnt[warp][k] = __popc(peers);
    __syncthreads();
    if (in) {
      int pos = base[k] + rank;
      for (int w = 0; w < warp; w++) pos += wcnt[w][k];
      order[pos] = first + i;
    }
    __syncthreads();
    if (in && leader) {
      atomicAdd(&base[k], __popc(peers));
      wcnt[warp][k] = 0;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

#define ME_DECLARE_ROUNDS(SUF)                                                                   \
  int round_grid_##SUF(int which, int device);                                                  \
  cudaError_t launch_round_##SUF(const DevPlan &P, const InvertArgs &A, const Slots &S,          \
                                 int parity, const int grids[3], cudaStream_t st,                \
                                 cudaEvent_t *ev, int svd_lanes, const Overlap *ov);             \
  cudaError_t launch_round_grp_##SUF(int G, const DevPlan &P, const InvertArgs &A,               \
                                     const Slots &S, int parity, const int grids[3],             \
                                     cudaStream_t st, cudaEvent_t *ev, const Overlap *ov);       \
  cudaError_t launch_finish_##SUF(const DevPlan &P, const InvertArgs &A, const Slots &S,         \
                                  int parity, int *cursor, int grid, cudaStream_t st);
ME_DECLARE_ROUNDS(f32)
ME_DECLARE_ROUNDS(f64)
ME_DECLARE_ROUNDS(f32f)
ME_DECLARE_ROUNDS(f64f)

// the variant of a plan: synthesis precision, and the instrument filter or not
#define ME_PICK(FN, ...)                                                                   \
  (precision == 1 ? (P.nsub > 1 ? FN##_f64f(__VA_ARGS__) : FN##_f64(__VA_ARGS__))           \
                  : (P.nsub > 1 ? FN##_f32f(__VA_ARGS__) : FN##_f32(__VA_ARGS__)))

cudaError_t launch_finish(int precision, const DevPlan &P, const InvertArgs &A, const Slots &S,
                          int parity, int *cursor, int grid, cudaStream_t st) {
  return ME_PICK(launch_finish, P, A, S, parity, cursor, grid, st);
}

cudaError_t launch_round_grp(int precision, int G, const DevPlan &P, const InvertArgs &A,
                             const Slots &S, int parity, const int grids[3], cudaStream_t st,
                             cudaEvent_t *ev, const Overlap *ov) {
  return ME_PICK(launch_round_grp, G, P, A, S, parity, grids, st, ev, ov);
}

// grids of the unfiltered kernels (the filtered ones run grid-stride loops
// over the same grids).  Each precision and filter unit has its own SVD
// kernel, whose dynamic shared memory exceeds the default limit; the sizing of
// the SVD grid raises that limit, so it is done in the filtered unit of the
// precision too (a plan may take a filter after it is made).
int round_grid(int precision, int which, int device) {
  if (which == 2 || which == 3) {
    if (precision == 1)
      round_grid_f64f(which, device);
    else
      round_grid_f32f(which, device);
  }
  return precision == 1 ? round_grid_f64(which, device) : round_grid_f32(which, device);
}

cudaError_t launch_round(int precision, const DevPlan &P, const InvertArgs &A, const Slots &S,
                         int parity, const int grids[3], cudaStream_t st, cudaEvent_t *ev,
                         int svd_lanes, const Overlap *ov) {
  return ME_PICK(launch_round, P, A, S, parity, grids, st, ev, svd_lanes, ov);
}

// SMs of the current device
static long long device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 1;
  return sms > 0 ? sms : 1;
}

template <class T>
static void launch_synth_t(const DevPlan &P, const double *d_par, const unsigned char *d_flags,
                           long long npix, double step7, double *d_prof, double *d_jac,
                           cudaStream_t st) {
  // pixels per block: up to kSynthPixels, fewer while the grid has less than
  // four blocks per SM, so that a few pixels spread over the device; of the
  // upper half of that range, the count whose wavelengths leave the fewest of
  // the block's threads idle in its last pass (6 wavelengths: 21 pixels)
  const long long sms = device_sms();
  constexpr int kMost = kSynthPixels<T>;
  int per = kMost;
  while (per > 1 && (npix + per - 1) / per < sms * 4) per /= 2;
  auto used = [&](int n) {
    const int points = n * P.nl;
    return (double)points / ((points + kSynthThreads - 1) / kSynthThreads * kSynthThreads);
  };
  if (per == kMost)
    for (int n = kMost - 1; n >= kMost / 2; n--)
      if (used(n) > used(per) + 0.05) per = n;
  const unsigned g = (unsigned)((npix + per - 1) / per);
  // with a filter a point is a sub-wavelength, its terms staged in shared
  // memory; with enough wavelengths to fill the device a thread sums its
  // wavelength's sub-wavelengths itself, which stages nothing (Fe I 6173, 21
  // sub-wavelengths, FP32: 48087 pixels 121 us against 180, 32 pixels 32 us
  // against 18).  FP64 Jacobians are always split: 40 sums of doubles beside
  // the point's registers spill (17486 pixels 1231 us against 906)
  const int mode = P.nsub <= 1 ? kPlain
                   : npix * P.nl >= sms * (d_jac ? 512 : 1024) ? kFilter : kFilterSplit;
  auto go = [&](auto jac, auto m) {
    synth_kernel<T, jac.value, m.value><<<g, kSynthThreads, 0, st>>>(
        P, d_par, d_flags, npix, per, step7, d_prof, d_jac);
  };
  auto pick = [&](auto jac) {
    if (mode == kPlain)
      go(jac, std::integral_constant<int, kPlain>());
    else if constexpr (jac.value && sizeof(T) == sizeof(double))
      go(jac, std::integral_constant<int, kFilterSplit>());
    else if (mode == kFilter)
      go(jac, std::integral_constant<int, kFilter>());
    else
      go(jac, std::integral_constant<int, kFilterSplit>());
  };
  if (d_jac)
    pick(std::true_type());
  else
    pick(std::false_type());
}

cudaError_t launch_synth(int precision, const DevPlan &P, const double *d_par, long long npix,
                         double step7, double *d_prof, double *d_jac, cudaStream_t st) {
  if (npix <= 0) return cudaSuccess;
  if (precision == 1)
    launch_synth_t<double>(P, d_par, nullptr, npix, step7, d_prof, d_jac, st);
  else
    launch_synth_t<float>(P, d_par, nullptr, npix, step7, d_prof, d_jac, st);
  return cudaGetLastError();
}

cudaError_t launch_fit(int precision, const DevPlan &P, const double *d_fitpar,
                       const unsigned char *d_flags, long long npix, double *d_fit,
                       cudaStream_t st) {
  if (npix <= 0) return cudaSuccess;
  if (precision == 1)
    launch_synth_t<double>(P, d_fitpar, d_flags, npix, P.step[7], d_fit, nullptr, st);
  else
    launch_synth_t<float>(P, d_fitpar, d_flags, npix, P.step[7], d_fit, nullptr, st);
  return cudaGetLastError();
}

cudaError_t launch_voigt(int precision, const DevPlan &P, const double *d_nu, const double *d_a,
                         long long n, double *d_H, double *d_L, cudaStream_t st) {
  const int b = 256;
  const unsigned g = (unsigned)((n + b - 1) / b);
  if (g == 0) return cudaSuccess;
  if (precision == 1)
    voigt_kernel<double><<<g, b, 0, st>>>(P, d_nu, d_a, n, d_H, d_L);
  else
    voigt_kernel<float><<<g, b, 0, st>>>(P, d_nu, d_a, n, d_H, d_L);
  return cudaGetLastError();
}

// matrices per warp for one thread per matrix: the fewest (a power of two) for
// which eight warps per SM cover them at once; a warp's time is that of the
// longest of its matrices' sweeps
static int svd_per_warp(long long nmat) {
  const long long warps = device_sms() * 8;
  int per = 32;
  while (per > 1 && (nmat + per / 2 - 1) / (per / 2) <= warps) per /= 2;
  return per;
}

// The full decomposition of 9 x 9 matrices, one thread per matrix (gr_svd9_v),
// `per` matrices per warp.  Matrices come in, and V and U go out, through the
// tile that holds V in between (stride 81: no bank conflict).  20011 normal
// matrices 105 us, 537 us with one thread per matrix in local memory.
constexpr int kSvd9VWords = 32 * (81 + kSvd9Words + 16);
__global__ void __launch_bounds__(32) svd9_v_kernel(const double *a, long long nmat, int per,
                                                    double *u, double *w, double *v,
                                                    int *limit_hits) {
  extern __shared__ double sm[];
  double *tile = sm, *wr = sm + 32 * 81;
  const int t = threadIdx.x;
  const long long first = blockIdx.x * (long long)per;
  const int here = (int)(nmat - first < per ? nmat - first : per);
  for (int k = t; k < here * 81; k += 32) tile[k] = a[first * 81 + k];
  __syncwarp();
  double A[9][9];
  if (t < here) {
#pragma unroll
    for (int r = 0; r < 9; r++)
#pragma unroll
      for (int c = 0; c < 9; c++) A[r][c] = tile[t * 81 + r * 9 + c];
    const int hit = gr_svd9_v<32>(A, wr + t, wr + 9 * 32 + t, wr + 18 * 32 + t, wr + 34 * 32 + t,
                                  tile + t * 81);
    if (hit && limit_hits) atomicAdd(limit_hits, 1);
  }
  __syncwarp();
  for (int k = t; k < here * 81; k += 32) v[first * 81 + k] = tile[k];
  for (int k = t; k < here * 9; k += 32) w[first * 9 + k] = wr[(k % 9) * 32 + k / 9];
  __syncwarp();
  if (t < here) {
#pragma unroll
    for (int r = 0; r < 9; r++)
#pragma unroll
      for (int c = 0; c < 9; c++) tile[t * 81 + r * 9 + c] = A[r][c];
  }
  __syncwarp();
  for (int k = t; k < here * 81; k += 32) u[first * 81 + k] = tile[k];
}

cudaError_t launch_svd(const double *d_a, long long nmat, int n, double *d_u, double *d_w,
                       double *d_v, int *d_hits, cudaStream_t st) {
  if (nmat <= 0) return cudaSuccess;
  if (n == 9) {
    const int per = svd_per_warp(nmat);
    svd9_v_kernel<<<(unsigned)((nmat + per - 1) / per), 32, kSvd9VWords * sizeof(double), st>>>(
        d_a, nmat, per, d_u, d_w, d_v, d_hits);
    return cudaGetLastError();
  }
  const int b = 128;
  const unsigned g = (unsigned)((nmat + b - 1) / b);
  if (g == 0) return cudaSuccess;
  svd_kernel<<<g, b, 0, st>>>(d_a, nmat, n, d_u, d_w, d_v, d_hits);
  return cudaGetLastError();
}

// The trial-step solve's U-only decomposition (gr_svd_u, gr_svd_u_grp) of
// nmat n x n matrices: G = 1, one thread per matrix in a column of shared
// memory (stride 32), as svd_kernel of the rounds holds it; G > 1, a group of
// G lanes per matrix, row-major in shared memory, as svd_grp_kernel and the
// tail kernel hold it.  Blocks of 32 threads.
template <int G, bool FAST>
__global__ void __launch_bounds__(32) svd_u_kernel(const double *a, long long nmat, int n,
                                                   double *u, double *w, int *limit_hits) {
  constexpr int kPer = 32 / G;  // matrices per block
  constexpr int kWords = G == 1 ? 99 * 32 : kPer * 81;
  __shared__ double sm[kWords];
  const int t = threadIdx.x;
  const long long i = blockIdx.x * (long long)kPer + t / G;
  if (i >= nmat) return;  // uniform across each group
  const int nn = n * n;
  int hit;
  if constexpr (G == 1) {
    double *am = sm + t, *wm = sm + 81 * 32 + t, *rv = sm + 90 * 32 + t;
    for (int k = 0; k < nn; k++) am[k * 32] = a[i * nn + k];
    hit = gr_svd_u<32, FAST>(am, n, wm, rv);
    for (int k = 0; k < nn; k++) u[i * nn + k] = am[k * 32];
    for (int k = 0; k < n; k++) w[i * n + k] = wm[k * 32];
  } else {
    const int lane = t % G;
    const unsigned mask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (t & ~(G - 1)));
    double *am = sm + (t / G) * 81;
    for (int k = lane; k < nn; k += G) am[k] = a[i * nn + k];
    __syncwarp(mask);
    double wl[9];
    hit = gr_svd_u_grp<G, FAST>(am, n, wl, lane, mask);
    for (int k = lane; k < nn; k += G) u[i * nn + k] = am[k];
    if (lane == 0)
      for (int k = 0; k < n; k++) w[i * n + k] = wl[k];
  }
  if (hit && limit_hits && (G == 1 || t % G == 0)) atomicAdd(limit_hits, 1);
}

// The decomposition of 9 x 9 matrices, one thread per matrix in registers
// (gr_svd9), `per` matrices per warp: a warp's matrices come in and go out
// through shared memory, so that global memory is read and written in whole
// lines (stride 81: no bank conflict).
template <int FORM, bool FAST>
__global__ void __launch_bounds__(32) svd_u9_kernel(const double *a, long long nmat, int per,
                                                    double *u, double *w, int *limit_hits) {
  __shared__ double tile[32 * 81];
  __shared__ double wr[kSvd9Words * 32];
  const int t = threadIdx.x;
  const long long first = blockIdx.x * (long long)per;
  const int here = (int)(nmat - first < per ? nmat - first : per);
  for (int k = t; k < here * 81; k += 32) tile[k] = a[first * 81 + k];
  __syncwarp();
  if (t < here) {
    double A[9][9];
#pragma unroll
    for (int r = 0; r < 9; r++)
#pragma unroll
      for (int c = 0; c < 9; c++) A[r][c] = tile[t * 81 + r * 9 + c];
    const int hit = gr_svd9<FORM, FAST, 32>(A, wr + t, wr + 9 * 32 + t, wr + 18 * 32 + t);
#pragma unroll
    for (int r = 0; r < 9; r++)
#pragma unroll
      for (int c = 0; c < 9; c++) tile[t * 81 + r * 9 + c] = A[r][c];
    if (hit && limit_hits) atomicAdd(limit_hits, 1);
  }
  __syncwarp();
  for (int k = t; k < here * 81; k += 32) u[first * 81 + k] = tile[k];
  for (int k = t; k < here * 9; k += 32) w[first * 9 + k] = wr[(k % 9) * 32 + k / 9];
}

template <int FORM>
static void launch_svd_u9(const double *d_a, long long nmat, int fast, double *d_u, double *d_w,
                          int *d_hits, cudaStream_t st) {
  const int per = svd_per_warp(nmat);
  const unsigned g = (unsigned)((nmat + per - 1) / per);
  if (fast)
    svd_u9_kernel<FORM, true><<<g, 32, 0, st>>>(d_a, nmat, per, d_u, d_w, d_hits);
  else
    svd_u9_kernel<FORM, false><<<g, 32, 0, st>>>(d_a, nmat, per, d_u, d_w, d_hits);
}

template <int G>
static void launch_svd_u_g(const double *d_a, long long nmat, int n, int fast, double *d_u,
                           double *d_w, int *d_hits, cudaStream_t st) {
  const unsigned g = (unsigned)((nmat + 32 / G - 1) / (32 / G));
  if (fast)
    svd_u_kernel<G, true><<<g, 32, 0, st>>>(d_a, nmat, n, d_u, d_w, d_hits);
  else
    svd_u_kernel<G, false><<<g, 32, 0, st>>>(d_a, nmat, n, d_u, d_w, d_hits);
}

cudaError_t launch_svd_u(const double *d_a, long long nmat, int n, int lanes, int fast,
                         double *d_u, double *d_w, int *d_hits, cudaStream_t st) {
  if (nmat <= 0) return cudaSuccess;
  if (n == 9) {
    if (lanes == 1)
      launch_svd_u9<0>(d_a, nmat, fast, d_u, d_w, d_hits, st);
    else
      launch_svd_u9<1>(d_a, nmat, fast, d_u, d_w, d_hits, st);
    return cudaGetLastError();
  }
  switch (lanes) {
    case 1: launch_svd_u_g<1>(d_a, nmat, n, fast, d_u, d_w, d_hits, st); break;
    case 2: launch_svd_u_g<2>(d_a, nmat, n, fast, d_u, d_w, d_hits, st); break;
    case 4: launch_svd_u_g<4>(d_a, nmat, n, fast, d_u, d_w, d_hits, st); break;
    case 8: launch_svd_u_g<8>(d_a, nmat, n, fast, d_u, d_w, d_hits, st); break;
    case 16: launch_svd_u_g<16>(d_a, nmat, n, fast, d_u, d_w, d_hits, st); break;
    case 32: launch_svd_u_g<32>(d_a, nmat, n, fast, d_u, d_w, d_hits, st); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_order_by_key(const unsigned char *d_key, long long n, int *d_hist,
                                long long *d_order, cudaStream_t st, long long base) {
  if (n <= 0) return cudaSuccess;
  const long long chunk = n / kOrderBlocks + 1 > 1024 ? n / kOrderBlocks + 1 : 1024;
  const int nb = (int)((n + chunk - 1) / chunk);
  order_hist_kernel<<<nb, 256, 0, st>>>(d_key, n, chunk, d_hist);
  order_scan_kernel<<<1, 1024, 0, st>>>(d_hist, kOrderBuckets * nb);
  order_scatter_kernel<<<nb, 256, 0, st>>>(d_key, n, chunk, d_hist, d_order, base);
  return cudaGetLastError();
}

// Re-sort of the queue positions [first, first + n) of `list` by the pixels'
// misfit keys, stable (the streamed host entry point: once the whole map has
// arrived, the part of the queue not yet taken goes into one global order).
__global__ void tail_gather_kernel(const long long *list, long long first, long long n,
                                   const unsigned char *key, unsigned char *tkey,
                                   long long *tval) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long pix = list[first + i];
  tval[i] = pix;
  tkey[i] = key[pix];
}

__global__ void tail_scatter_kernel(long long *list, long long first, long long n,
                                    const long long *perm, const long long *tval) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  list[first + i] = tval[perm[i]];
}

cudaError_t launch_resort_tail(long long *d_list, long long first, long long n,
                               const unsigned char *d_key, unsigned char *d_tkey,
                               long long *d_tval, int *d_hist, long long *d_perm,
                               cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int b = 256;
  const unsigned g = (unsigned)((n + b - 1) / b);
  tail_gather_kernel<<<g, b, 0, st>>>(d_list, first, n, d_key, d_tkey, d_tval);
  cudaError_t e = launch_order_by_key(d_tkey, n, d_hist, d_perm, st, 0);
  if (e != cudaSuccess) return e;
  tail_scatter_kernel<<<g, b, 0, st>>>(d_list, first, n, d_perm, d_tval);
  return cudaGetLastError();
}

cudaError_t launch_start_order(int precision, const DevPlan &P, const double *d_prof,
                               const double *d_init, long long npix, unsigned char *d_key,
                               int *d_hist, long long *d_order, cudaStream_t st,
                               long long base) {
  if (npix <= 0) return cudaSuccess;
  const int b = 128;
  const unsigned g = (unsigned)((npix + b - 1) / b);
  // about 16 wavelengths of the grid
  const int stride = P.nl / 16 > 1 ? P.nl / 16 : 1;
  if (precision == 1) {
    if (P.nsub > 1)
      start_misfit_kernel<double, true><<<g, b, 0, st>>>(P, d_prof, d_init, npix, stride, d_key);
    else
      start_misfit_kernel<double, false><<<g, b, 0, st>>>(P, d_prof, d_init, npix, stride, d_key);
  } else {
    if (P.nsub > 1)
      start_misfit_kernel<float, true><<<g, b, 0, st>>>(P, d_prof, d_init, npix, stride, d_key);
    else
      start_misfit_kernel<float, false><<<g, b, 0, st>>>(P, d_prof, d_init, npix, stride, d_key);
  }
  return launch_order_by_key(d_key, npix, d_hist, d_order, st, base);
}

cudaError_t launch_init_guess(const DevPlan &P, const double *d_prof, long long npix,
                              double *d_guess, double *d_extra, int *d_status, cudaStream_t st) {
  const int b = 128;
  const unsigned g = (unsigned)((npix + b - 1) / b);
  if (g == 0) return cudaSuccess;
  init_guess_kernel<<<g, b, 0, st>>>(P, d_prof, npix, d_guess, d_extra, d_status);
  return cudaGetLastError();
}

}  // namespace me
