// Colour-model fit on the device (gc_gmm_fit): expectation-maximisation of a Gaussian mixture
// over pixel colours, the reference's GMM.fit (GMM.pyx:165-372; initA, em1, em2, eval and
// check_converge, gmm.cl:33-372), in float64.
//
// The reference runs every EM iteration as a chain of launches separated by host waits: em1
// writes per-sample responsibilities to global memory, em2 halves them log2(n) times, eval
// and check_converge sum the log-likelihood, and the host reads it back to decide whether
// to go on.  Here the whole fit is ONE launch of one thread-block cluster (16 blocks of 640
// threads where the device can place them, else 8):
//   * a lane evaluates a sample; the moment sums (responsibility times 1, x and x x^T, ten per
//     component) are a matrix product over the samples, done by the double-precision matrix
//     instruction (m8n8k4: components x samples times samples x moments), whose accumulators
//     hold the warp's sums: no accumulators per lane, no shuffles to add them up;
//   * the blocks read one another's sums through distributed shared memory, every block in
//     the same fixed order, so every block holds bit-identical totals and takes the same
//     decisions (no broadcast is needed, and a run is deterministic);
//   * one cluster barrier per iteration: the sums are double-buffered, so a block's next ones
//     do not overwrite what another still reads.
// All barriers are hardware cluster barriers that every thread of every block reaches the
// same number of times: the loop's exit decisions come from the identical totals.
//
// An iteration is a chain of latencies, not of work (10,000 samples and 4 components keep the
// double-precision units busy for 1.1 us): 6.5 us each, a 65-iteration fit 426 us on one B200,
// against 14 and 912 with 8 blocks of 256 threads, 40 sums a lane added up by shuffles, two
// cluster barriers and one thread making all components' next models.
#include <cooperative_groups.h>

#include <cmath>
#include <mutex>
#include <unordered_map>

#include "gcut_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr int kMaxK = GC_GMM_MAX_COMPONENTS;
constexpr int kThreads = 640;
constexpr int kWarps = kThreads / 32;
constexpr int kStats = 10;                   // per component: r, r x (3), r x x^T (6)
constexpr int kLsum = kMaxK * kStats;        // index of the log-likelihood sum
constexpr int kVals = kLsum + 1;
constexpr int kMaxCluster = 16;
constexpr int kRow = 36;                     // doubles per component row of s.r (32 and padding:
                                             // a fragment's reads fall into distinct banks)
constexpr double kLog2Pi = 1.8378770664093453;  // log(2 pi)

struct FitShared {
  double stats[2][kVals];       // this block's sums, read by the cluster's other blocks
  double tot[kVals];            // cluster totals (identical in every block)
  double part[kWarps][kMaxK * kStats + 2];   // per-warp sums ([80]: log-likelihood)
  double w[kMaxK], mu[kMaxK][3], S[kMaxK][6];   // current model (S: lower triangle)
  double c[kMaxK], li[kMaxK][6];                // its evaluation form
  double lprev, lcur;
  int stop, status, iterations, converged;
  double r[kWarps][8][kRow];    // responsibilities of a warp's 32 samples, a row per component
};

// Evaluation form of component k: c = log w - 0.5 (3 log 2pi + log det S) and Li, the
// inverse of the lower Cholesky factor of S.  Returns false when S is not positive definite.
__device__ bool component_form(FitShared& sh, int k) {
  const double* S = sh.S[k];
  const double l00 = sqrt(S[0]);
  const double l10 = S[1] / l00, l20 = S[3] / l00;
  const double d11 = S[2] - l10 * l10;
  const double l11 = sqrt(d11);
  const double l21 = (S[4] - l20 * l10) / l11;
  const double d22 = S[5] - l20 * l20 - l21 * l21;
  const double l22 = sqrt(d22);
  const double i00 = 1.0 / l00, i11 = 1.0 / l11, i22 = 1.0 / l22;
  const double i10 = -l10 * i00 * i11;
  const double i21 = -l21 * i11 * i22;
  const double i20 = -(l20 * i00 + l21 * i10) * i22;
  const double logdet = 2.0 * (log(l00) + log(l11) + log(l22));
  sh.c[k] = log(sh.w[k]) - 0.5 * (3.0 * kLog2Pi + logdet);
  sh.li[k][0] = i00; sh.li[k][1] = i10; sh.li[k][2] = i11;
  sh.li[k][3] = i20; sh.li[k][4] = i21; sh.li[k][5] = i22;
  return S[0] > 0.0 && d11 > 0.0 && d22 > 0.0 && isfinite(logdet);
}

// M-step of component k from the cluster totals (em2, gmm.cl:183-312): weight N_k / sum N,
// mean sum r x / N_k, covariance sum r x x^T / N_k - mean mean^T + min_covar I.
__device__ void m_step(FitShared& sh, int k, int K, double min_covar, int full) {
  double sum_n = 0.0;
  for (int j = 0; j < K; ++j) sum_n += sh.tot[j * kStats];
  const double* t = sh.tot + k * kStats;
  const double nk = t[0];
  if (!(nk > 0.0)) {  // no responsibility left: weight 0, the rest unchanged
    sh.w[k] = 0.0;
    return;
  }
  sh.w[k] = nk / sum_n;
  const double m0 = t[1] / nk, m1 = t[2] / nk, m2 = t[3] / nk;
  sh.mu[k][0] = m0; sh.mu[k][1] = m1; sh.mu[k][2] = m2;
  double* S = sh.S[k];
  S[0] = t[4] / nk - m0 * m0 + min_covar;
  S[2] = t[6] / nk - m1 * m1 + min_covar;
  S[5] = t[9] / nk - m2 * m2 + min_covar;
  if (full) {
    S[1] = t[5] / nk - m1 * m0;
    S[3] = t[7] / nk - m2 * m0;
    S[4] = t[8] / nk - m2 * m1;
  } else {
    S[1] = S[3] = S[4] = 0.0;
  }
}

// D += A B for 8 x 4 by 4 x 8 doubles: lane l holds A[l / 4][l % 4], B[l % 4][l / 4] and
// D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

// Moment f of a colour (1, R, G, B, RR, GR, GG, BR, BG, BB): the product of two of 1, R, G, B,
// an integer below 2^16.  ca, cb: bit offsets of the factors in the word, negative for 1.
__device__ __forceinline__ double moment(uint32_t px, int ca, int cb) {
  const int a = ca < 0 ? 1 : (int)((px >> ca) & 255u), b = cb < 0 ? 1 : (int)((px >> cb) & 255u);
  return (double)(a * b);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// One cluster of blocks.  KMAX: the component count rounded up to 2, 4 or 8.  FULL: full
// covariances (else the off-diagonal factors are 0 and left out).
template <int KMAX, bool FULL>
__global__ void __launch_bounds__(kThreads, 1)
k_gmm_fit(const uint32_t* __restrict__ samples, int n, int K, int max_iter, double tol,
          double min_covar, double init_covar, gc_gmm_fit_result* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char fit_smem[];
  FitShared& sh = *reinterpret_cast<FitShared*>(fit_smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int stride = ranks * kThreads;

  // initA (gmm.cl:33-72): evenly spaced samples as means.  Its green channel goes through
  // the mask 0xFF0 (gmm.cl:54), a typo for 0xFF00; the full green byte is used here.
  if (tid < K) {
    const int k = tid;
    const int idx = K > 1 ? (int)((long long)k * (n - 1) / (K - 1)) : 0;
    const uint32_t px = samples[idx];
    sh.w[k] = 1.0 / K;
    sh.mu[k][0] = (double)(px & 0xFFu);
    sh.mu[k][1] = (double)((px >> 8) & 0xFFu);
    sh.mu[k][2] = (double)((px >> 16) & 0xFFu);
    double* S = sh.S[k];
    S[0] = S[2] = S[5] = init_covar;
    S[1] = S[3] = S[4] = 0.0;
  }
  if (tid == 0) {
    sh.lprev = sh.lcur = 0.0;
    sh.stop = sh.status = sh.iterations = sh.converged = 0;
  }
  for (int i = tid; i < kWarps * 8 * kRow; i += kThreads) (&sh.r[0][0][0])[i] = 0.0;   // rows >= K stay 0
  __syncthreads();
  if (tid < K && !component_form(sh, tid)) sh.status = 1;
  __syncthreads();

  // the moments this lane feeds to the matrix instruction: f = lane / 4, and 8 + lane / 4
  // (two of them; the others are 0)
  const int f = lane >> 2;
  const int ca = f == 0 ? -1 : f == 1 ? 0 : f == 2 ? 8 : f == 3 ? 16 : f == 4 ? 0 : f == 7 ? 16 : 8;
  const int cb = f < 4 ? -1 : f == 6 ? 8 : 0;
  const int cb2 = f == 0 ? 8 : 16;   // f = 8: B G; f = 9: B B
  const double (*const rw)[kRow] = sh.r[warp];

  for (int t = 0; !sh.status; ++t) {   // the same in every block: totals and models are identical
    const int buf = t & 1;
    // E-step (em1): responsibilities and their moment sums
    double d1[2] = {0.0, 0.0}, d2[2] = {0.0, 0.0}, lsum = 0.0;
    // (unsigned: the index passes n, which may be near 2^31, by up to a stride)
    for (unsigned i0 = rank * kThreads + warp * 32; i0 < (unsigned)n; i0 += stride) {   // warp-uniform
      const unsigned i = i0 + lane;
      // lanes past the end repeat the last sample and count 0 times: 0 times the responsibilities
      // of any other colour need not be 0, where no component is within reach of it
      const uint32_t px = samples[i < (unsigned)n ? i : (unsigned)n - 1];
      const double x0 = (double)(px & 0xFFu), x1 = (double)((px >> 8) & 0xFFu),
                   x2 = (double)((px >> 16) & 0xFFu);
      double e[KMAX];
      double m = -INFINITY;
#pragma unroll
      for (int k = 0; k < KMAX; ++k) {
        if (k < K) {
          const double q0 = x0 - sh.mu[k][0], q1 = x1 - sh.mu[k][1], q2 = x2 - sh.mu[k][2];
          const double* L = sh.li[k];
          const double y0 = L[0] * q0;
          const double y1 = FULL ? L[1] * q0 + L[2] * q1 : L[2] * q1;
          const double y2 = FULL ? L[3] * q0 + L[4] * q1 + L[5] * q2 : L[5] * q2;
          e[k] = sh.c[k] - 0.5 * (y0 * y0 + y1 * y1 + y2 * y2);
          m = fmax(m, e[k]);
        }
      }
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K) {
          e[k] = exp(e[k] - m);
          s += e[k];
        }
      if (i < (unsigned)n) lsum += m + log(s);
      const double inv = i < (unsigned)n ? 1.0 / s : 0.0;
      __syncwarp();   // the last step's reads of the rows
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K) sh.r[warp][k][lane] = e[k] * inv;
      __syncwarp();
#pragma unroll
      for (int g = 0; g < 8; ++g) {   // four samples a step
        const int src = 4 * g + (lane & 3);
        const double a = rw[f][src];
        const uint32_t q = __shfl_sync(0xffffffffu, px, src);
        mma_f64(d1, a, moment(q, ca, cb));
        mma_f64(d2, a, f < 2 ? moment(q, 16, cb2) : 0.0);
      }
    }
    lsum = warp_sum(lsum);
    {   // D[k][j]: component k = lane / 4, moments 2 (lane % 4) + {0, 1} of each product
      double* const p = sh.part[warp] + (lane >> 2) * kStats;
      const int j = 2 * (lane & 3);
      p[j] = d1[0];
      p[j + 1] = d1[1];
      if (j == 0) {
        p[8] = d2[0];
        p[9] = d2[1];
      }
      if (lane == 0) sh.part[warp][kLsum] = lsum;
    }
    __syncthreads();
    // block sums: four lanes a value, each a quarter of the warps, then in order
    if (tid < 4 * kVals) {
      const int v = tid >> 2, part = tid & 3;
      double a = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps / 4; ++w) a += sh.part[part * (kWarps / 4) + w][v];
      const unsigned mask = 15u << (lane & ~3);   // the value's four lanes
      a += __shfl_xor_sync(mask, a, 1);
      a += __shfl_xor_sync(mask, a, 2);
      if (part == 0) sh.stats[buf][v] = a;
    }
    cluster.sync();  // every block's sums are written

    // cluster totals (em2's reduction): every block adds the blocks' sums in rank order
    if (tid < 4 * kVals) {
      const int v = tid >> 2, part = tid & 3;
      double a = 0.0;
      for (int r = part * (ranks / 4); r < (part + 1) * (ranks / 4); ++r)
        a += cluster.map_shared_rank(&sh.stats[buf][0], r)[v];
      const unsigned mask = 15u << (lane & ~3);   // the value's four lanes
      a += __shfl_xor_sync(mask, a, 1);
      a += __shfl_xor_sync(mask, a, 2);
      if (part == 0) sh.tot[v] = a;
    }
    __syncthreads();
    // eval + check_converge (GMM.pyx:283-329): the sum just formed is L of the model that
    // produced the responsibilities, i.e. of iteration t - 1.  Thread k decides for itself and
    // makes the next model's component k.
    if (tid < K) {
      const double L = sh.tot[kLsum], lprev = sh.lprev;
      const bool conv = t >= 1 && t - 1 > 1 && fabs(L - lprev) < tol;
      const bool stop = conv || t == max_iter;
      __syncwarp((1u << K) - 1u);   // every one has read lprev
      if (tid == 0) {
        if (conv) sh.converged = 1;
        if (t >= 1) sh.lprev = L;
        sh.lcur = L;
        sh.iterations = t;
        sh.stop = stop;
      }
      if (!stop) {
        m_step(sh, tid, K, min_covar, FULL);
        if (!component_form(sh, tid)) sh.status = 1;
      }
    }
    __syncthreads();
    if (sh.stop) break;
  }
  cluster.sync();  // no block leaves while another reads its sums

  if (rank == 0 && tid == 0) {
    for (int k = 0; k < kMaxK; ++k) {
      const bool on = k < K;
      out->weights[k] = on ? sh.w[k] : 0.0;
      for (int j = 0; j < 3; ++j) out->means[k][j] = on ? sh.mu[k][j] : 0.0;
      for (int j = 0; j < 6; ++j) out->covars[k][j] = on ? sh.S[k][j] : 0.0;
    }
    // the evaluation form belongs to the returned model: the loop stops before an M-step
    for (int k = 0; k < kMaxK; ++k) {
      const bool on = k < K && !sh.status;
      out->components[k].c = on ? sh.c[k] : 0.0;
      for (int j = 0; j < 3; ++j) out->components[k].mean[j] = on ? sh.mu[k][j] : 0.0;
      for (int j = 0; j < 6; ++j) out->components[k].li[j] = on ? sh.li[k][j] : 0.0;
    }
    out->log_likelihood = sh.lcur;
    out->iterations = sh.iterations;
    out->converged = sh.converged;
    out->status = sh.status;
    out->n_components = K;
  }
}

int fit_fail(const char* msg) { return gcut::set_last_error(GC_ERR_INVALID, msg); }

// Launches the fit on the larger cluster the device can place (16 blocks is beyond the portable
// 8; whether they fit beside what else runs is the scheduler's business, as for any launch).
template <int KMAX, bool FULL>
cudaError_t launch_fit(const uint32_t* samples, int n, int K, int max_iter, double tol,
                       double min_covar, double init_covar, gc_gmm_fit_result* out, cudaStream_t s) {
  static std::mutex mu;
  static std::unordered_map<int, int> cluster_of;   // per device; 0: could not be set up
  const auto kernel = k_gmm_fit<KMAX, FULL>;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(FitShared);
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int cluster = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cluster_of.find(dev);
    if (it == cluster_of.end()) {
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FitShared));
      if (e != cudaSuccess) return e;
      int fit = 0, clusters = 0;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        attr.val.clusterDim.x = kMaxCluster;
        cfg.gridDim = dim3(kMaxCluster);
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0) fit = kMaxCluster;
      }
      cudaGetLastError();   // (a refusal above only means the portable size)
      it = cluster_of.emplace(dev, fit ? fit : 8).first;
    }
    cluster = it->second;
  }
  attr.val.clusterDim.x = cluster;
  cfg.gridDim = dim3(cluster);
  return cudaLaunchKernelEx(&cfg, kernel, samples, n, K, max_iter, tol, min_covar, init_covar, out);
}

template <int KMAX>
cudaError_t launch_fit(bool full, const uint32_t* samples, int n, int K, int max_iter, double tol,
                       double min_covar, double init_covar, gc_gmm_fit_result* out, cudaStream_t s) {
  return full ? launch_fit<KMAX, true>(samples, n, K, max_iter, tol, min_covar, init_covar, out, s)
              : launch_fit<KMAX, false>(samples, n, K, max_iter, tol, min_covar, init_covar, out, s);
}

}  // namespace

extern "C" int gc_gmm_fit(const uint32_t* samples, int n, int n_components, int max_iterations,
                          double tolerance, double min_covar, double init_covar,
                          int full_covariance, gc_gmm_fit_result* result, void* stream) {
  gcut::set_last_error(GC_OK, "");
  if (n_components < 1 || n_components > kMaxK)
    return fit_fail("gc_gmm_fit: n_components must be 1..GC_GMM_MAX_COMPONENTS");
  if (n < n_components) return fit_fail("gc_gmm_fit: fewer samples than components");
  if (max_iterations < 1 || max_iterations > 100000)
    return fit_fail("gc_gmm_fit: max_iterations must be 1..100000");
  if (!std::isfinite(tolerance) || tolerance < 0.0) return fit_fail("gc_gmm_fit: bad tolerance");
  if (!std::isfinite(min_covar) || min_covar < 0.0) return fit_fail("gc_gmm_fit: bad min_covar");
  if (!std::isfinite(init_covar) || !(init_covar > 0.0))
    return fit_fail("gc_gmm_fit: init_covar must be > 0");
  if (!samples || !result) return fit_fail("gc_gmm_fit: null samples or result");
  cudaStream_t s = (cudaStream_t)stream;
  const bool full = full_covariance != 0;
  const cudaError_t e =
      n_components <= 2 ? launch_fit<2>(full, samples, n, n_components, max_iterations, tolerance, min_covar, init_covar, result, s)
      : n_components <= 4 ? launch_fit<4>(full, samples, n, n_components, max_iterations, tolerance, min_covar, init_covar, result, s)
                          : launch_fit<8>(full, samples, n, n_components, max_iterations, tolerance, min_covar, init_covar, result, s);
  if (e != cudaSuccess) return gcut::set_last_error(GC_ERR_CUDA, cudaGetErrorString(e));
  return GC_OK;
}
