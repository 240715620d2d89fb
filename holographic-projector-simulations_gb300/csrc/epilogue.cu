// epilogue.cu -- deterministic cross-CTA reductions and the output semantics.
//
//   launch_reduce          sum of per-split partials in split order, scattered
//                          back to the caller's target order; replaces the
//                          reference's cublasZgemv row sum (cuda/kernel.cu:179-195)
//   launch_max_abs / launch_normalize_polar
//                          normalize_amp<false> + polar output
//                          (cuda/transform.cu:106-139, 376, 402-405)
//   launch_reference_wave  amplitude-only projector (cuda/transform.cu:379-395)
//   launch_complex_to_polar / launch_adjoint_epilogue   the adjoint's ends
//   launch_intensity_loss / launch_intensity_grad       the loss of a phase-only hologram
#include <float.h>

#include <algorithm>

#include "internal.cuh"
#include "ptx.cuh"

namespace holo {
namespace {

__global__ void __launch_bounds__(256) k_reduce(const double2 *__restrict__ partial, int splits,
                                                int M, const int32_t *__restrict__ order,
                                                double2 *__restrict__ y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
    double re = 0.0, im = 0.0;
    for (int s = 0; s < splits; ++s) {
      const double2 v = partial[(size_t)s * M + i];
      re += v.x;
      im += v.y;
    }
    y[order ? order[i] : i] = make_double2(re, im);
  }
}

__global__ void __launch_bounds__(256) k_reduce_batched(const SplitProblem *__restrict__ probs,
                                                        const int *__restrict__ offsets,
                                                        int n_probs, int total) {
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
    // problem p with offsets[p] <= g < offsets[p + 1]
    int lo = 0, hi = n_probs;
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (offsets[mid] <= g) lo = mid; else hi = mid;
    }
    const SplitProblem &P = probs[lo];
    if (P.splits == 1) continue;
    const int i = g - offsets[lo];
    double re = 0.0, im = 0.0;
    for (int s = 0; s < P.splits; ++s) {
      const double2 v = P.partial[(size_t)s * P.M + i];
      re += v.x;
      im += v.y;
    }
    P.y[P.order_t[i]] = make_double2(re, im);
  }
}

__device__ __forceinline__ bool fast_polar(double x, double y, const fixed::PolarEntry *table,
                                           double *modulus, double *angle) {
  return fixed::polar(x, y, table, [](float v, float u) { return atan2f(v, u); },
                      [](float v) { return ptx::rcp_approx(v); },
                      [](float v) { return ptx::rsqrt_approx(v); }, modulus, angle);
}

// Modulus and angle of what fast_polar leaves; zeros, which whole dark fields hold, without the
// ~90 FP64 operations of a hypot and an atan2 (a normalisation of 2^20 zeros: 226 us with both
// alone, 237 us with fast_polar tried before them, 86 us here).
__device__ __forceinline__ void slow_polar(double x, double y, double *modulus, double *angle) {
  if (x == 0.0 && y == 0.0) {
    *modulus = 0.0;
    *angle = signbit(x) ? copysign(3.14159265358979323846, y) : y;
  } else {
    *modulus = hypot(x, y);
    *angle = atan2(y, x);
  }
}

// The largest modulus.  Bound by the FP64 pipe: the squares' sum (2 operations instead of
// hypot's ~35) of every value first, then hypot only of those within 2^-40 of the block's largest
// sum, which the largest hypot is among; a block whose sums leave the safe range takes hypot
// for all.  512 values a block, not 2048: 512^2 values take 12 us.  With the kernel below, a
// normalisation of 1024^2 values took 249 us as a call before both, 142 us now.
constexpr int kMaxPerBlock = 512;
__global__ void __launch_bounds__(256) k_max_abs_partial(const double2 *__restrict__ y, int M,
                                                         double *__restrict__ partial) {
  __shared__ double s[256];
  const int step = gridDim.x * blockDim.x, first = blockIdx.x * blockDim.x + threadIdx.x;
  double most = 0.0;
  bool odd = false;
  for (int i = first; i < M; i += step) {
    const double q = fma(y[i].x, y[i].x, y[i].y * y[i].y);
    odd = odd || !(q < 1e300);
    most = q > most ? q : most;
  }
  s[threadIdx.x] = most;
  odd = __syncthreads_or(odd);
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] = fmax(s[threadIdx.x], s[threadIdx.x + w]);
    __syncthreads();
  }
  const double limit = odd || s[0] < 1e-280 ? -1.0 : s[0] * (1.0 - 0x1p-40);
  __syncthreads();
  double m = 0.0;
  if (!(most < limit))  // none of this thread's values otherwise
    for (int i = first; i < M; i += step)
      if (!(fma(y[i].x, y[i].x, y[i].y * y[i].y) < limit) && !(y[i].x == 0.0 && y[i].y == 0.0))
        m = fmax(m, hypot(y[i].x, y[i].y));
  s[threadIdx.x] = m;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] = fmax(s[threadIdx.x], s[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

__global__ void __launch_bounds__(256) k_max_final(const double *__restrict__ partial, int n,
                                                   double *__restrict__ out) {
  __shared__ double s[256];
  double m = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, partial[i]);
  s[threadIdx.x] = m;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] = fmax(s[threadIdx.x], s[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = s[0];
}

// Bound by the FP64 pipe (27 operations a value, fixed::polar, instead of ~130 of two quotients,
// hypot and atan2): 512^2 values take 21 us.  modulus / max by the
// reciprocal and one correction, as exact as the quotient.
__global__ void __launch_bounds__(256) k_normalize_polar(const double2 *__restrict__ y, int M,
                                                         const double *__restrict__ max_abs,
                                                         const fixed::PolarEntry *__restrict__ table,
                                                         double *__restrict__ amp,
                                                         double *__restrict__ phase) {
  __shared__ double inverse;
  const double mx = *max_abs;
  const bool scale = !(mx < 1e-6);  // below 1e-6 the reference leaves y unnormalised
  const double div = scale ? mx : 1.0;
  if (threadIdx.x == 0) inverse = 1.0 / div;
  __syncthreads();
  const double inv = inverse;
  const bool fast = div < 1e100;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
    double re = y[i].x, im = y[i].y, m, a;
    if (fast && fast_polar(re, im, table, &m, &a)) {
      const double q = m * inv;
      m = fma(fma(-q, div, m), inv, q);
    } else {
      if (scale) {
        re = __ddiv_rn(re, mx);
        im = __ddiv_rn(im, mx);
      }
      slow_polar(re, im, &m, &a);
    }
    amp[i] = m;
    phase[i] = a;
  }
}

__global__ void __launch_bounds__(256) k_complex_to_polar(const double2 *__restrict__ g, int M,
                                                          const fixed::PolarEntry *__restrict__ table,
                                                          double *__restrict__ amp,
                                                          double *__restrict__ phase) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
    double m, a;
    if (!fast_polar(g[i].x, g[i].y, table, &m, &a)) slow_polar(g[i].x, g[i].y, &m, &a);
    amp[i] = m;
    phase[i] = a;
  }
}

// Bound by the FP64 pipe: sine and cosine of the phase as fixed-point numbers (fp64_fixed.cuh), 9
// operations with the products instead of ~60: 1024^2 sources take 23 us.  With the polar form
// of the gradient it took a step of 1024^2 -> 512^2 from 2192 to 2141 us.
__global__ void __launch_bounds__(256) k_adjoint_epilogue(const double2 *__restrict__ h,
                                                          const double *__restrict__ amp,
                                                          const double *__restrict__ phase,
                                                          int N, const fixed::TrigEntry *__restrict__ trig,
                                                          const fixed::TurnWords *__restrict__ words,
                                                          double *__restrict__ grad_amp,
                                                          double *__restrict__ grad_phase) {
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    double sp, cp;
    const double ph = phase[n];
    const uint32_t hi = (uint32_t)__double2hiint(ph);
    const uint32_t e = ((hi >> 20) & 0x7ffu) - (uint32_t)(1023 + fixed::kTurnLow);
    if (e < (uint32_t)fixed::kTurnEntries) {
      const uint4 k = *reinterpret_cast<const uint4 *>(&words[e]);
      const uint64_t t = fixed::turns(hi, (uint32_t)__double2loint(ph), k.x, k.y, k.z, k.w);
      const uint32_t index = fixed::trig_index(t);
      int64_t c, s;
      fixed::cos_sin(t, index, trig[index & (fixed::kTrigEntries - 1)], &c, &s);
      cp = (double)c * 0x1p-62;
      sp = (double)s * 0x1p-62;
    } else {
      sincos(ph, &sp, &cp);
    }
    // w = e^{i phi} conj(H)
    const double wr = cp * h[n].x + sp * h[n].y;
    const double wi = sp * h[n].x - cp * h[n].y;
    grad_amp[n] = wr;
    grad_phase[n] = -amp[n] * wi;
  }
}

__global__ void __launch_bounds__(256) k_reference_wave(const double2 *__restrict__ y,
                                                        const double2 *__restrict__ y_ref, int M,
                                                        const double *__restrict__ max_y,
                                                        const double *__restrict__ max_ref,
                                                        double *__restrict__ amp,
                                                        double *__restrict__ phase) {
  const double my = *max_y, mr = *max_ref;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
    double yr = y[i].x, yi = y[i].y, rr = y_ref[i].x, ri = y_ref[i].y;
    if (!(my < 1e-6)) { yr = __ddiv_rn(yr, my); yi = __ddiv_rn(yi, my); }
    if (!(mr < 1e-6)) { rr = __ddiv_rn(rr, mr); ri = __ddiv_rn(ri, mr); }
    // interference, then the phase of the reference wave (the projector only
    // modulates amplitude): y = from_polar(|y + y_ref|, angle(y_ref))
    const double a = hypot(yr + rr, yi + ri);
    const double p = atan2(ri, rr);
    double sp, cp;
    sincos(p, &sp, &cp);
    const double tr = a * cp, ti = a * sp;
    amp[i] = hypot(tr, ti);
    phase[i] = atan2(ti, tr);
  }
}

// ---- mean((I / mean I - target)^2), I = |z|^2, and its gradient in z ------------------------
// Two passes over z (16 bytes a target) with sums per block in a fixed order: every block of the
// second reads the first's partial sums, so nothing waits for the host.  Latency bound at
// 256^2 targets, memory at 1024^2.  As separate array operations the loss and its gradient were
// 31 launches, three of them reductions in one block of 27 us: a gradient step of 256^2 ->
// 256^2 took 920 us with them and 541 us with these four; of 1024^2 -> 512^2 2320 and 2192 us.
constexpr int kLossThreads = 256;

__device__ double2 block_sum2(double2 v, double2 *shared) {
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, o);
    v.y += __shfl_down_sync(0xffffffffu, v.y, o);
  }
  if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = v;
  __syncthreads();
  double2 t = make_double2(0.0, 0.0);
  for (int w = 0; w < kLossThreads / 32; ++w) {
    t.x += shared[w].x;
    t.y += shared[w].y;
  }
  __syncthreads();
  return t;
}

__device__ double intensity(double2 z) { return fma(z.x, z.x, z.y * z.y); }
// I / mean by the mean's reciprocal, where that is a normal number
__device__ double relative(double inten, double mean, double inv) {
  return inv > 1e-300 && inv < 1e300 ? inten * inv : inten / mean;
}

__global__ void __launch_bounds__(kLossThreads) k_loss_mean(const double2 *__restrict__ z, int M,
                                                            double *__restrict__ partial) {
  __shared__ double2 shared[kLossThreads / 32];
  double2 sum = make_double2(0.0, 0.0);
  for (int i = blockIdx.x * kLossThreads + threadIdx.x; i < M; i += gridDim.x * kLossThreads)
    sum.x += intensity(z[i]);
  sum = block_sum2(sum, shared);
  if (threadIdx.x == 0) partial[blockIdx.x] = sum.x;
}

__global__ void __launch_bounds__(kLossThreads)
    k_loss_terms(const double2 *__restrict__ z, const double *__restrict__ target, int M,
                 const double *__restrict__ partial, double2 *__restrict__ sums,
                 double *__restrict__ diff, double *__restrict__ stats) {
  __shared__ double2 shared[kLossThreads / 32];
  double2 sum = make_double2(0.0, 0.0);
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kLossThreads) sum.x += partial[i];
  const double mean = block_sum2(sum, shared).x / M, inv = 1.0 / mean;
  sum = make_double2(0.0, 0.0);
  for (int i = blockIdx.x * kLossThreads + threadIdx.x; i < M; i += gridDim.x * kLossThreads) {
    const double n = relative(intensity(z[i]), mean, inv), d = n - target[i];
    if (diff) diff[i] = d;
    sum.x = fma(d, d, sum.x);
    sum.y = fma(d, n, sum.y);
  }
  sum = block_sum2(sum, shared);
  if (threadIdx.x == 0) {
    sums[blockIdx.x] = sum;
    if (blockIdx.x == 0) stats[0] = mean;
  }
}

__global__ void __launch_bounds__(kLossThreads) k_loss_final(const double2 *__restrict__ sums,
                                                             int blocks, int M,
                                                             double *__restrict__ loss,
                                                             double *__restrict__ stats) {
  __shared__ double2 shared[kLossThreads / 32];
  double2 sum = make_double2(0.0, 0.0);
  for (int i = threadIdx.x; i < blocks; i += kLossThreads) {
    sum.x += sums[i].x;
    sum.y += sums[i].y;
  }
  sum = block_sum2(sum, shared);
  if (threadIdx.x == 0) {
    *loss = sum.x / M;
    stats[1] = sum.y / M;
  }
}

// dL / dI_i = 2 / (M mean) (d_i - mean(d I / mean I)), dI / dz = 2 z
__global__ void __launch_bounds__(kLossThreads)
    k_loss_grad(const double2 *__restrict__ z, const double *__restrict__ diff, int M,
                const double *__restrict__ stats, const double *__restrict__ grad,
                double2 *__restrict__ out) {
  const double mean = stats[0], shift = stats[1], scale = 4.0 * *grad / M / mean;
  for (int i = blockIdx.x * kLossThreads + threadIdx.x; i < M; i += gridDim.x * kLossThreads) {
    const double g = scale * (diff[i] - shift);
    out[i] = make_double2(g * z[i].x, g * z[i].y);
  }
}

int blocks_for(int n) {
  int g = (n + 255) / 256;
  return g < 1 ? 1 : (g > 8192 ? 8192 : g);
}

}  // namespace

int epilogue_preload() {
  cudaFuncAttributes a;
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_reduce));
  return HOLO_OK;
}

int launch_reduce(const double2 *partial, int splits, int M, const int32_t *order, double2 *y,
                  cudaStream_t s) {
  if (M <= 0) return HOLO_OK;
  k_reduce<<<blocks_for(M), 256, 0, s>>>(partial, splits, M, order, y); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_reduce_batched(const SplitProblem *probs_dev, const int *prob_offsets, int n_probs,
                          int total_targets, cudaStream_t s) {
  if (total_targets <= 0) return HOLO_OK;
  k_reduce_batched<<<blocks_for(total_targets), 256, 0, s>>>(probs_dev, prob_offsets, n_probs,
                                                             total_targets); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_max_abs(const double2 *y, int M, double *partials, int n_partials, double *max_out,
                   cudaStream_t s) {
  int nb = (M + kMaxPerBlock - 1) / kMaxPerBlock;
  nb = nb < 1 ? 1 : (nb > n_partials ? n_partials : nb);
  k_max_abs_partial<<<nb, 256, 0, s>>>(y, M, partials); note_launches(1);
  k_max_final<<<1, 256, 0, s>>>(partials, nb, max_out); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_normalize_polar(const double2 *y, int M, const double *max_abs,
                           const fixed::PolarEntry *table, double *amp, double *phase,
                           cudaStream_t s) {
  if (M <= 0) return HOLO_OK;
  k_normalize_polar<<<blocks_for(M), 256, 0, s>>>(y, M, max_abs, table, amp, phase); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_complex_to_polar(const double2 *g, int M, const fixed::PolarEntry *table, double *amp,
                            double *phase, cudaStream_t s) {
  if (M <= 0) return HOLO_OK;
  k_complex_to_polar<<<blocks_for(M), 256, 0, s>>>(g, M, table, amp, phase); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_adjoint_epilogue(const double2 *h, const double *amp, const double *phase, int N,
                            const fixed::TrigEntry *trig, const fixed::TurnWords *words,
                            double *grad_amp, double *grad_phase, cudaStream_t s) {
  if (N <= 0) return HOLO_OK;
  k_adjoint_epilogue<<<blocks_for(N), 256, 0, s>>>(h, amp, phase, N, trig, words, grad_amp, grad_phase); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_intensity_loss(const double2 *z, const double *target, int M, double *loss, double *diff,
                          double *work, cudaStream_t s) {
  static_assert(HOLO_INTENSITY_WORK == 2 + 3 * 512, "two statistics, then the blocks' sums");
  if (M <= 0) return HOLO_OK;
  const int nb = std::min((M + 4 * kLossThreads - 1) / (4 * kLossThreads), 512);
  double2 *sums = reinterpret_cast<double2 *>(work + 2);
  double *partial = work + 2 + 2 * 512;
  k_loss_mean<<<nb, kLossThreads, 0, s>>>(z, M, partial); note_launches(1);
  k_loss_terms<<<nb, kLossThreads, 0, s>>>(z, target, M, partial, sums, diff, work); note_launches(1);
  k_loss_final<<<1, kLossThreads, 0, s>>>(sums, nb, M, loss, work); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_intensity_grad(const double2 *z, const double *diff, int M, const double *work,
                          const double *grad, double2 *out, cudaStream_t s) {
  if (M <= 0) return HOLO_OK;
  k_loss_grad<<<blocks_for(M), kLossThreads, 0, s>>>(z, diff, M, work, grad, out); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_reference_wave(double2 *y, const double2 *y_ref, int M, const double *max_y,
                          const double *max_ref, double *amp_out, double *phase_out,
                          cudaStream_t s) {
  if (M <= 0) return HOLO_OK;
  k_reference_wave<<<blocks_for(M), 256, 0, s>>>(y, y_ref, M, max_y, max_ref, amp_out,
                                                 phase_out); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

}  // namespace holo
