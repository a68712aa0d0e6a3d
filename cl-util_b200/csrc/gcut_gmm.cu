// T-links from two colour models, computed on the device (gc_tlinks_gmm).
//
// The reference scores each pixel under a foreground and a background Gaussian mixture
// (GMM.score, GMM.pyx:130-163, running score_buf / score_img2d, gmm.cl:373-491) and feeds
// the solver excess = scoreBg - scoreFg (test_GraphCut.py:44-47).  Here the two scores, their
// difference and the int32 rounding are one pass over the image: 4 bytes read and 4 written
// per pixel, the rest is float64 arithmetic on registers.
//
// The models are full-covariance (a diagonal model is the special case the reference fits).
// Each component is evaluated as c - 0.5 * |Li (x - mean)|^2 with Li the inverse Cholesky
// factor, every add and multiply rounded on its own in a fixed order (the __d*_rn intrinsics
// are never contracted into fused multiply-adds), so a float64 host evaluation in the same
// order gives the same bits up to the last-bit differences of exp and log.
#include <cmath>
#include <cstdio>

#include "gcut_internal.h"

namespace {

constexpr int kMaxComp = GC_GMM_MAX_COMPONENTS;
constexpr int kThreads = 128;
// Images below this take one pixel a thread and a copy of the code for each model: with at most
// five warps a scheduler the two models' chains side by side count more than the instruction
// cache.  k_tlinks_gmm with 4 components, this way and the other: 61 kpix 4.8 and 6.0 us, 120
// kpix 7.4 and 6.9, 200 kpix 10.2 and 9.3.
constexpr long long kSmallImage = 3 << 15;

struct GmmArgs {
  gc_gauss comp[2][kMaxComp];  // [0] foreground, [1] background
  int n[2];
  double scale;
  int clamp;
};

// log(w N(x | mean, S)) of one component.
__device__ __forceinline__ double component_log_density(const gc_gauss& g, double r, double gr,
                                                        double b) {
  const double d0 = __dsub_rn(r, g.mean[0]);
  const double d1 = __dsub_rn(gr, g.mean[1]);
  const double d2 = __dsub_rn(b, g.mean[2]);
  const double y0 = __dmul_rn(g.li[0], d0);
  const double y1 = __dadd_rn(__dmul_rn(g.li[1], d0), __dmul_rn(g.li[2], d1));
  const double y2 = __dadd_rn(__dadd_rn(__dmul_rn(g.li[3], d0), __dmul_rn(g.li[4], d1)),
                              __dmul_rn(g.li[5], d2));
  const double q = __dadd_rn(__dadd_rn(__dmul_rn(y0, y0), __dmul_rn(y1, y1)), __dmul_rn(y2, y2));
  return __fma_rn(-0.5, q, g.c);   // halving is exact: one rounding, as in c - 0.5 * q
}

// exp(x) for x below this is under 2^-57, so 1 plus up to seven such terms, added in any
// order, rounds to exactly 1 in float64.
constexpr double kNegligible = -40.0;

// exp(x) for x below this is under 2^-144, beyond the last bit of a sum of at least 1.
constexpr double kVanishing = -100.0;

// -log sum_k w_k N(x | mean_k, S_k) = -(m + log(sum_k exp(e_k - m))), m = max_k e_k, of PX
// pixels under a model of n <= KMAX components.
template <int KMAX, int PX>
__device__ __forceinline__ void mixture_scores(const gc_gauss* comp, int n, const double (&r)[PX],
                                               const double (&g)[PX], const double (&b)[PX],
                                               double (&s)[PX]) {
  double e[PX][KMAX], m[PX];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    if (k < n) {
      const gc_gauss c = comp[k];
#pragma unroll
      for (int j = 0; j < PX; ++j) {
        e[j][k] = component_log_density(c, r[j], g[j], b[j]);
        m[j] = k == 0 || e[j][k] > m[j] ? e[j][k] : m[j];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < PX; ++j) {
    const double low = __dadd_rn(m[j], kNegligible);
    int near = 0;
#pragma unroll
    for (int k = 0; k < KMAX; ++k) near += k < n && e[j][k] >= low;
    // Only the largest term counts: the sum is exactly exp(0) = 1 and log(1) = 0, which is
    // what the full evaluation below gives too; skipping it saves the exp and log calls.
    s[j] = -__dadd_rn(m[j], 0.0);
    if (near > 1) {
      double sum = 0.0;
#pragma unroll
      for (int k = 0; k < KMAX; ++k) {
        if (k < n) {
          const double d = __dsub_rn(e[j][k], m[j]);
          double v = d == 0.0 ? 1.0 : 0.0;   // exp(0)
          if (d < 0.0 && d >= kVanishing) v = exp(d);
          sum = __dadd_rn(sum, v);
        }
      }
      s[j] = -__dadd_rn(m[j], log(sum));
    }
  }
}

// KMAX: the larger of the two models' component counts, rounded up to 2, 4 or 8 (fewer
// registers for the common small models).  A thread takes PX pixels, a block's width apart;
// MODELS = 2 evaluates the two models side by side, 1 one after the other by the same code.
//
// Bound by the float64 pipe (about 300 instructions a pixel at 4 components, 35 us at
// 1920x1080) and the instruction cache: the two models inline, with an exponential a component,
// overflow it.  One copy of the code for both and two pixels a thread, so that a component's
// parameters are moved to registers once for both, take 51 us there where one pixel and both
// models inline took 76 (4 pixels: 65; one pixel, one copy: 54); 1 component 13 (21), 8 97 (125).
// Left out: the exponentials of the largest term (exp(0) = 1) and of terms under 2^-144.
template <int KMAX, int PX, int MODELS>
__global__ void __launch_bounds__(kThreads, 4)
k_tlinks_gmm(const uint32_t* __restrict__ rgba, int width, long long n, int pitch,
             const GmmArgs a, int32_t* __restrict__ excess) {
  for (long long base = (long long)blockIdx.x * kThreads * PX + threadIdx.x; base < n;
       base += (long long)gridDim.x * kThreads * PX) {
    double r[PX], g[PX], b[PX], s_fg[PX], s_bg[PX] = {};
#pragma unroll
    for (int j = 0; j < PX; ++j) {
      const long long i = base + j * kThreads;
      uint32_t px = 0;
      if (i < n) px = __ldg(rgba + (pitch == width ? i : i / width * pitch + i % width));
      r[j] = (double)(px & 0xFFu);
      g[j] = (double)((px >> 8) & 0xFFu);
      b[j] = (double)((px >> 16) & 0xFFu);
    }
#pragma unroll MODELS
    for (int q = 0; q < 2; ++q) {   // foreground, background
#pragma unroll
      for (int j = 0; j < PX; ++j) s_fg[j] = s_bg[j];
      mixture_scores<KMAX, PX>(a.comp[q], a.n[q], r, g, b, s_bg);
    }
#pragma unroll
    for (int j = 0; j < PX; ++j) {
      const long long i = base + j * kThreads;
      // the conversion rounds down and saturates; the clamp is at most 2^30
      const int t = __double2int_rd(__dadd_rn(__dmul_rn(a.scale, __dsub_rn(s_bg[j], s_fg[j])), 0.5));
      if (i < n) excess[i] = min(max(t, -a.clamp), a.clamp);
    }
  }
}

template <int KMAX, int PX, int MODELS>
void launch_tlinks(const uint32_t* rgba, int width, long long n, int pitch, const GmmArgs& a,
                   int32_t* excess, cudaStream_t s) {
  const long long blocks = (n + kThreads * PX - 1) / (kThreads * PX);
  const unsigned grid = (unsigned)(blocks < (1LL << 30) ? blocks : (1LL << 30));
  k_tlinks_gmm<KMAX, PX, MODELS><<<grid, kThreads, 0, s>>>(rgba, width, n, pitch, a, excess);
}

int tlinks_fail(const char* msg) { return gcut::set_last_error(GC_ERR_INVALID, msg); }

bool finite_within(double v, double bound) { return std::isfinite(v) && std::fabs(v) <= bound; }

int check_model(const gc_gauss* m, int n, const char* which) {
  static thread_local char buf[160];
  if (n < 1 || n > kMaxComp) {
    snprintf(buf, sizeof buf, "gc_tlinks_gmm: %s model needs 1..%d components", which, kMaxComp);
    return tlinks_fail(buf);
  }
  if (!m) {
    snprintf(buf, sizeof buf, "gc_tlinks_gmm: %s model is null", which);
    return tlinks_fail(buf);
  }
  for (int k = 0; k < n; ++k) {
    bool ok = finite_within(m[k].c, 0x1p64);
    for (int j = 0; j < 3; ++j) ok = ok && finite_within(m[k].mean[j], 0x1p32);
    for (int j = 0; j < 6; ++j) ok = ok && finite_within(m[k].li[j], 0x1p32);
    if (!ok) {
      snprintf(buf, sizeof buf,
               "gc_tlinks_gmm: %s component %d has a non-finite or out-of-range parameter", which, k);
      return tlinks_fail(buf);
    }
  }
  return GC_OK;
}

}  // namespace

extern "C" int gc_tlinks_gmm(const uint32_t* rgba, int width, int height, int pitch,
                             const gc_gauss* fg, int n_fg, const gc_gauss* bg, int n_bg,
                             double scale, int32_t clamp, int32_t* excess, void* stream) {
  gcut::set_last_error(GC_OK, "");
  if (width < 0 || height < 0) return tlinks_fail("gc_tlinks_gmm: negative size");
  if (pitch < width) return tlinks_fail("gc_tlinks_gmm: pitch < width");
  if (!finite_within(scale, 0x1p32)) return tlinks_fail("gc_tlinks_gmm: |scale| > 2^32 or not finite");
  if (clamp < 0 || clamp > (1 << 30)) return tlinks_fail("gc_tlinks_gmm: clamp outside [0, 2^30]");
  int r = check_model(fg, n_fg, "foreground");
  if (r != GC_OK) return r;
  r = check_model(bg, n_bg, "background");
  if (r != GC_OK) return r;
  const long long n = (long long)width * height;
  if (n == 0) return GC_OK;
  if (!rgba || !excess) return tlinks_fail("gc_tlinks_gmm: null image or output");

  GmmArgs a{};
  for (int k = 0; k < n_fg; ++k) a.comp[0][k] = fg[k];
  for (int k = 0; k < n_bg; ++k) a.comp[1][k] = bg[k];
  a.n[0] = n_fg;
  a.n[1] = n_bg;
  a.scale = scale;
  a.clamp = clamp;
  const int kmax = n_fg > n_bg ? n_fg : n_bg;
  cudaStream_t s = (cudaStream_t)stream;
  if (n < kSmallImage) {
    if (kmax <= 2) launch_tlinks<2, 1, 2>(rgba, width, n, pitch, a, excess, s);
    else if (kmax <= 4) launch_tlinks<4, 1, 2>(rgba, width, n, pitch, a, excess, s);
    else launch_tlinks<8, 1, 2>(rgba, width, n, pitch, a, excess, s);
  } else {
    if (kmax <= 2) launch_tlinks<2, 2, 1>(rgba, width, n, pitch, a, excess, s);
    else if (kmax <= 4) launch_tlinks<4, 2, 1>(rgba, width, n, pitch, a, excess, s);
    else launch_tlinks<8, 1, 1>(rgba, width, n, pitch, a, excess, s);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return gcut::set_last_error(GC_ERR_CUDA, cudaGetErrorString(e));
  return GC_OK;
}
