// Search-side kernels around the surrogate: the synchrony feature of a
// batch of simulated trajectories, the candidates' network inputs, and the
// ensemble's ranking score.  C ABI: device pointers and a stream.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "dense_b200_surrogate.h"

#include <cooperative_groups.h>

#include <cmath>
#include <cstdint>

#if defined(__GNUC__)
#define FEATURES_API extern "C" __attribute__((visibility("default")))
#else
#define FEATURES_API extern "C"
#endif

namespace {

constexpr int kSyncThreads = 512;
constexpr int kMaxSyncCells = 1024;
constexpr int kSyncGroups = kSyncThreads / 32;
constexpr int kSyncInv = 64;
// Bytes of the trajectories in flight (two CTAs per SM) that the 126 MB L2
// keeps between the kernel's two passes.
constexpr int64_t kSyncL2 = int64_t(80) << 20;

__device__ __forceinline__ double quiet_nan() { return __longlong_as_double(0x7FF8000000000000LL); }

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) t += red[i];  // warps in order
  return t;
}

// Mean pairwise Pearson correlation across the cells of each set's
// trajectory X[set][t][cell] (t < counts[set]; cells contiguous), cells
// with a constant trace left out:
//   sum_{i != j} <z_i, z_j> = |sum_i z_i|^2 - n  for unit, zero-mean z_i,
// divided by n (n - 1); NaN when fewer than two cells remain.
//
// Two passes over the samples: the cells' means and squared deviations
// (blocks of eight samples two-pass in registers, joined by the pairwise
// update of Chan, Golub and LeVeque, 1983, which keeps the two-pass
// accuracy), then per sample the sum of z over the cells.  A set's samples
// (600 x 200 doubles: 0.96 MB) are shared by a cluster of CTAs, as many as
// keep the sets in flight within the L2 cache, so that the second pass does
// not go back to HBM; the CTAs' statistics meet in distributed shared
// memory, joined in rank order.  1500 sets x 600 x 200, 1.44 GB: 0.54 ms (2.7 TB/s
// from HBM, 5.4 TB/s read), bound by issue (45 %) and the barriers between
// the passes; with one CTA per set and three passes, every one from HBM,
// 1.17 ms.  (Slices of the samples kept in shared memory, 8 or 16 CTAs a
// set, took 1.6 ms: the exchange and the reductions of so many CTAs cost
// more than the reads they save.)
struct CellStats {
  double n, mean, m2;
  __device__ __forceinline__ void join(double bn, double bmean, double bm2) {
    if (bn <= 0.0) return;
    if (n <= 0.0) {  // (the update's square of bmean may be out of range)
      n = bn;
      mean = bmean;
      m2 = bm2;
      return;
    }
    const double total = n + bn, w = bn / total, d = bmean - mean;
    mean += d * w;
    m2 += bm2 + d * d * (n * w);
    n = total;
  }
};

__global__ void __launch_bounds__(kSyncThreads, 2) synchrony_kernel(const double* __restrict__ X, int64_t set_stride,
                                                                    int64_t sample_stride, int cells,
                                                                    const int* __restrict__ counts,
                                                                    double* __restrict__ out) {
  __shared__ double red[kSyncThreads / 32];
  extern __shared__ double sy_dyn[];
  __shared__ double s_n[kSyncGroups];                       // samples of each thread group
  const int threads = blockDim.x, wide = max(threads, cells);
  double* s_mean = sy_dyn;                                  // the groups' statistics, [group][cell]
  double* s_m2 = s_mean + wide;
  double* r_mean = s_m2 + wide;                             // this rank's, read by the others
  double* r_m2 = r_mean + cells;
  double* centre = r_m2 + cells;                            // the cells' means over every rank
  __shared__ int share_top;
  __shared__ double share_sq;
  __shared__ unsigned long long share_bits;
  __shared__ double s_inv[kSyncInv];                        // 1 / (k + 1)
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int set = blockIdx.x / ranks;
  const int T = counts[set];
  const int per = T > 0 ? (T + ranks - 1) / ranks : 0;
  const int t0 = min(T, rank * per), rows = max(0, min(T, t0 + per) - t0);
  const double* x = X + set * set_stride + t0 * sample_stride;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int warps = threads >> 5;

  // pass 1: rows dealt over thread groups of `width` threads, eight
  // neighbouring rows at a time
  int width = 32;
  while (width < cells && width < threads) width *= 2;
  const int groups = threads / width, grp = tid / width, first = tid % width;
  // largest magnitude, to the 20 mantissa bits of its upper word (exactly
  // below, where the rest decides); infinities and NaN lie above all
  int top = 0;
  auto magnitude = [&](double v) { top = max(top, __double2hiint(v) & 0x7fffffff); };
  for (int i = tid; i < kSyncInv; i += threads) s_inv[i] = 1.0 / (i + 1);
  if (tid == 0) share_top = 0;
  __syncthreads();
  for (int c = first; c < cells; c += width) {
    const double* p = x + c + static_cast<int64_t>(grp) * 8 * sample_stride;
    const int64_t hop = static_cast<int64_t>(groups) * 8 * sample_stride;
    double mean = 0.0, m2 = 0.0;
    int t = grp * 8, k = 0;  // k whole blocks joined
    for (; t + 8 <= rows; t += groups * 8, p += hop, ++k) {
      double v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = p[j * sample_stride];
      const double m = (((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]))) * 0.125;
      double q0 = 0.0, q1 = 0.0;
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        magnitude(v[j]);
        magnitude(v[j + 1]);
        const double d0 = v[j] - m, d1 = v[j + 1] - m;
        q0 += d0 * d0;
        q1 += d1 * d1;
      }
      // CellStats::join of equal blocks: k blocks and one more
      const double w = k < kSyncInv ? s_inv[k] : 1.0 / (k + 1), d = m - mean;
      mean += d * w;
      m2 += (q0 + q1) + (k > 0 ? d * d * (8.0 * k * w) : 0.0);
    }
    CellStats st{8.0 * k, mean, m2};
    for (int j = 0; t + j < rows && j < 8; ++j) {
      const double v = p[j * sample_stride];
      magnitude(v);
      st.join(1.0, v, 0.0);
    }
    s_mean[grp * width + c] = st.mean;  // (one group when cells > width)
    s_m2[grp * width + c] = st.m2;
    if (c == 0) s_n[grp] = st.n;
  }
  __syncthreads();
  for (int c = tid; c < cells; c += threads) {
    CellStats st{0.0, 0.0, 0.0};
    for (int g = 0; g < groups; ++g) st.join(s_n[g], s_mean[g * width + c], s_m2[g * width + c]);
    r_mean[c] = st.mean;
    r_m2[c] = st.m2;
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) atomicMax(&share_top, top);
  cluster.sync();
  for (int k = 0; k < ranks; ++k) top = max(top, *cluster.map_shared_rank(&share_top, k));
  // The largest magnitude scales the threshold of a constant trace.  Between
  // the least and the greatest value of its upper word no norm lies but by
  // rare chance: then it is looked up exactly (every CTA of the cluster has
  // the same norms and comes to the same decision).  With an infinite or NaN
  // sample no cell counts (the comparison fails).
  double largest = __hiloint2double(top, 0);
  const double most = __hiloint2double(top, -1);
  auto counts_with = [](double nrm, double magnitude_) { return nrm > 1e-12 * (1.0 + magnitude_); };
  bool unsure = false;
  for (int c = tid; c < cells; c += threads) {
    CellStats st{0.0, 0.0, 0.0};
    for (int k = 0; k < ranks; ++k) {
      const int rk = max(0, min(T, k * per + per) - min(T, k * per));
      st.join(rk, cluster.map_shared_rank(r_mean, k)[c], cluster.map_shared_rank(r_m2, k)[c]);
    }
    const double nrm = sqrt(st.m2);
    centre[c] = st.mean;
    s_mean[c] = nrm;  // the groups' statistics are done with
    unsure = unsure || (counts_with(nrm, largest) && !counts_with(nrm, most));
  }
  if (__syncthreads_or(unsure) && top < 0x7ff00000) {
    unsigned long long bits = 0;
    const double* all = X + set * set_stride;
    for (int64_t i = tid; i < static_cast<int64_t>(T) * cells; i += threads)
      bits = max(bits, __double_as_longlong(all[i / cells * sample_stride + i % cells]) & 0x7fffffffffffffffull);
    if (tid == 0) share_bits = 0;
    __syncthreads();
    atomicMax(&share_bits, bits);
    __syncthreads();
    largest = __longlong_as_double(share_bits);
  }
  // the norms (0: left out) and their reciprocals (a norm out of range:
  // quotients of 0)
  double n_ok = 0.0;
  for (int c = tid; c < cells; c += threads) {
    const double nrm = s_mean[c];
    const bool ok = counts_with(nrm, largest);
    s_mean[c] = ok ? (isinf(nrm) ? 1.0 : nrm) : 0.0;
    s_m2[c] = ok ? 1.0 / nrm : 0.0;
    n_ok += ok ? 1.0 : 0.0;
  }
  const double n = block_sum(n_ok, red);  // (its barriers also publish the norms)

  // pass 2: a warp per four samples; the quotient from the reciprocal with
  // one FMA correction (its error stays below one ulp of the division's)
  double s2 = 0.0;
  for (int t = 4 * warp; t < rows; t += 4 * warps) {
    const int live = min(4, rows - t);
    const double* p = x + static_cast<int64_t>(t) * sample_stride;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int c = lane; c < cells; c += 32) {
      double v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = p[(j < live ? j : 0) * sample_stride + c];
      const double m = centre[c], nrm = s_mean[c], inv = s_m2[c];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double d = v[j] - m, q = d * inv;
        s[j] += __fma_rn(__fma_rn(-q, nrm, d), inv, q);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
      if (j < live) s2 += s[j] * s[j];
    }
  }
  const double mine = block_sum(lane == 0 ? s2 : 0.0, red);
  if (tid == 0) share_sq = mine;
  cluster.sync();
  if (rank == 0 && tid == 0) {
    double total = 0.0;
    for (int k = 0; k < ranks; ++k) total += *cluster.map_shared_rank(&share_sq, k);
    out[set] = n >= 2.0 ? (total - n) / (n * (n - 1.0)) : quiet_nan();
  }
  cluster.sync();  // every rank's shared memory stays until rank 0 has read it
}

// Network inputs of candidates P[r][ldp] (float64 parameters):
// Xb[r][j] = BF16(float32(log(P[r][idx[j]] / tmpl[j]) / log_spread)) for
// j < k, zeros in the padding columns and in rows n..Bp-1.
__global__ void encode_kernel(const double* __restrict__ P, int ldp, int n, const int* __restrict__ idx,
                              const double* __restrict__ tmpl, int k, double log_spread, __nv_bfloat16* __restrict__ Xb,
                              int in_pad, int Bp) {
  const int64_t total = static_cast<int64_t>(Bp) * in_pad;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / in_pad), j = static_cast<int>(i % in_pad);
    float v = 0.f;
    if (r < n && j < k) v = static_cast<float>(log(P[static_cast<int64_t>(r) * ldp + idx[j]] / tmpl[j]) / log_spread);
    Xb[i] = __float2bfloat16(v);
  }
}

// acc = Y (first network) or acc + Y, in float32, over [n][nout].
__global__ void ensemble_accumulate_kernel(const float* __restrict__ Y, int ldy, int n, int nout,
                                           float* __restrict__ acc, int first) {
  const int64_t total = static_cast<int64_t>(n) * nout;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / nout), c = static_cast<int>(i % nout);
    const float y = Y[static_cast<int64_t>(r) * ldy + c];
    acc[i] = first ? y : __fadd_rn(acc[i], y);
  }
}

// The ranking score of each candidate from the ensemble sum acc[n][nout]
// (outputs: log period, log amplitude, synchrony, oscillation indicator,
// acceptance indicator): y = (acc / nets) * sd + mu in float32, then in
// float64  y4 + w * (-|exp(clamp(y0, -10, 10)) - period| / tol
//                    + 0.5 clamp((y1 - log amp_min) / ramp + 0.5, 0, 1)
//                    + 0.5 clamp(y3, 0, 1)).
struct ScoreParams {
  float mu[8], sd[8];
  float nets;
  double weight, period, tol, log_amp_min, ramp;
};

__global__ void score_kernel(const float* __restrict__ acc, int n, int nout, const ScoreParams sp,
                             double* __restrict__ out) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    double y[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const float a = __fdiv_rn(acc[static_cast<int64_t>(r) * nout + j], sp.nets);
      y[j] = static_cast<double>(__fadd_rn(__fmul_rn(a, sp.sd[j]), sp.mu[j]));
    }
    const double per = exp(fmin(fmax(y[0], -10.0), 10.0));
    const double amp_term = fmin(fmax((y[1] - sp.log_amp_min) / sp.ramp + 0.5, 0.0), 1.0);
    const double osc_term = fmin(fmax(y[3], 0.0), 1.0);
    const double region = -fabs(per - sp.period) / sp.tol + 0.5 * amp_term + 0.5 * osc_term;
    out[r] = y[4] + sp.weight * region;
  }
}

int blocks_for(int64_t n) {
  const int64_t b = (n + 255) / 256;
  return static_cast<int>(b < 4096 ? (b > 0 ? b : 1) : 4096);
}

}  // namespace

FEATURES_API int dense_features_synchrony(const double* X, int64_t set_stride, int64_t sample_stride, int cells,
                                          const int* counts, int n_sets, double* out, void* stream) {
  if (n_sets < 0 || cells < 0 || cells > kMaxSyncCells) return 1;
  if (n_sets == 0) return 0;
  // the most samples a set can have in this layout (unknown, taken as few,
  // when the sets are not the outer dimension)
  const int64_t cap = sample_stride > 0 && set_stride >= sample_stride ? set_stride / sample_stride : 0;
  int ranks = 1;
  while (ranks < 8 && (296 / ranks * cap * cells * 8 > kSyncL2 ||
                       (static_cast<int64_t>(n_sets) * ranks < 296 && cap / ranks > 32)))
    ranks *= 2;
  // threads by a CTA's share of a set: the fixed part (reductions, exchange)
  // of 512 threads outweighs small sets (1500 sets x 50 x 20: 53 us with 512,
  // 32 us with 128; 700 sets x 100 x 200 with 256: 62 us either way; the
  // largest shares want all 512: 0.54 ms against 0.64 ms with 256)
  const int64_t share = cap * cells / ranks;
  const int threads = cap == 0 || share >= 16384 ? kSyncThreads : (share >= 4096 ? 256 : 128);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = ranks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(n_sets * ranks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = sizeof(double) * (2 * (threads > cells ? threads : cells) + 3 * cells);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, synchrony_kernel, X, set_stride, sample_stride, cells, counts, out);
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : 2;
}

FEATURES_API int dense_features_encode(const double* P, int ldp, int n, const int* idx, const double* tmpl, int k,
                                       double log_spread, void* Xb, int in_pad, int Bp, void* stream) {
  if (n < 0 || Bp < n || k > in_pad || k < 0 || !(log_spread != 0.0)) return 1;
  encode_kernel<<<blocks_for(static_cast<int64_t>(Bp) * in_pad), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      P, ldp, n, idx, tmpl, k, log_spread, static_cast<__nv_bfloat16*>(Xb), in_pad, Bp);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

FEATURES_API int dense_features_ensemble_accumulate(const float* Y, int ldy, int n, int nout, float* acc, int first,
                                                    void* stream) {
  if (n < 0 || nout <= 0 || ldy < nout) return 1;
  ensemble_accumulate_kernel<<<blocks_for(static_cast<int64_t>(n) * nout), 256, 0,
                               static_cast<cudaStream_t>(stream)>>>(Y, ldy, n, nout, acc, first);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// mu and sd (nout floats each) are host arrays.
FEATURES_API int dense_features_score(const float* acc, int n, int nout, int nets, const float* mu, const float* sd,
                                      double weight, double period, double tol, double amp_min, double ramp,
                                      double* out, void* stream) {
  if (n < 0 || nout < 5 || nout > 8 || nets <= 0 || !(amp_min > 0.0) || !(tol > 0.0) || !(ramp > 0.0)) return 1;
  ScoreParams sp{};
  for (int j = 0; j < nout; ++j) {
    sp.mu[j] = mu[j];
    sp.sd[j] = sd[j];
  }
  sp.nets = static_cast<float>(nets);
  sp.weight = weight;
  sp.period = period;
  sp.tol = tol;
  sp.log_amp_min = std::log(amp_min);
  sp.ramp = ramp;
  score_kernel<<<blocks_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(acc, n, nout, sp, out);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
