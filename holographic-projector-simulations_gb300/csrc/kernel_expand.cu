// kernel_expand.cu -- HOLO_SPLIT32 sums between clusters of points by separable expansions.
//
// The brute-force sum of superposition::per_block (cuda/superposition.cu:59-154) over every
// pair of a target cluster T (centre T0) and a source cluster S (centre S0), regrouped.  With
// D = T0 - S0, r0 = |D|, t' = t - T0, s' = s - S0 the phase of a pair splits into
//   r = |D + t' - s'| = alpha(t) + beta(s) + psi(t, s),
//   alpha = |D + t'|,  beta = |D - s'| - r0,  psi = r - alpha - beta,
// where alpha and beta belong to one point and psi, the mixed part, is small and smooth: its
// leading term is -(t'_perp . s'_perp) / r0, a few radians over clusters of thousands of
// points.  G(t, s) = e^{i s k psi} / r is therefore interpolated in both points on px x py
// Chebyshev nodes of the clusters' boxes (at most 128 of them), and the sum over the pair
// of clusters becomes
//   moments    mu_ab = sum_s T_a(x_s) T_b(y_s) a_s e^{i (phi_s + s k beta(s))}
//   translate  nu    = M G M^T mu   (M: Chebyshev coefficients of the nodal interpolant)
//   targets    y_t  += e^{i s k alpha(t)} sum_ab T_a(x_t) T_b(y_t) nu_ab:
// (ns + nt) point evaluations and 128^2 node pairs instead of ns nt pairs.  Moments and
// targets are products of a matrix of node weights (one row of T_a T_b per point) with one
// column pair (re, im) per partner cluster: they run on the tensor cores (tcgen05 kind::tf32
// as three products of TF32 splits, ~2^-21), while the CUDA cores form the phases, in the
// float-float arithmetic of the pair kernels (split_frame.cuh).
//
// Truncation: for e^{i z x} on [-1, 1] the p-node interpolant is off by at most
// 2 (z / 2)^p / p!; expand_choose (expand_plan.cu) takes the cheapest cluster sizes for which
// that stays below 8e-7 along each axis, which measured 2.5e-7 of the field's norm or less.
//
// The TF32 accumulator of an MMA drops bits of the running sum at every step, a bias that
// grows with the length of the chain: the moments kernel moves its accumulator to FP32
// registers every 64 sources and keeps the small cross products of the splits in an
// accumulator of their own; the target kernel adds the cross products and the high
// orders, which are small, before the low ones.
#include <algorithm>

#include "internal.cuh"
#include "ptx.cuh"

namespace holo {
namespace {

#include "split_frame.cuh"
#include "tc_operand.cuh"

constexpr int kNodes = kExpandNodes;  // node slots of a cluster: rows of the weight matrices
constexpr int kMaxP = 16;             // nodes along one axis
constexpr int kGroupT = 64;           // target clusters per moments block (128 MMA columns)
constexpr int kChunk = 16;            // sources per operand stage of the moments kernel
constexpr int kSuper = 64;            // sources staged, and summed in the MMA accumulator, at once
constexpr int kBlockT = 128;          // targets per block of the target kernel
constexpr int kGroupS = 32;           // source clusters per MMA of the target kernel (64 columns)
constexpr int kHalfFloats = 8192;     // one staged half (64 nodes, hi and lo) of nu: 32 KB

// Block -> (problem, block of it): the last problem whose first block is <= b.
template <bool BATCHED>
__device__ __forceinline__ const ExpandProblem &find_problem(const ExpandProblem &P0,
                                                             const ExpandProblem *probs,
                                                             const int *offs, int n, int *item) {
  if (!BATCHED) {
    *item = blockIdx.x;
    return P0;
  }
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (offs[mid] <= (int)blockIdx.x) lo = mid; else hi = mid;
  }
  *item = blockIdx.x - offs[lo];
  return probs[lo];
}

// FP32 frame of one cluster pair as the kernels read it: (s k e hi, r0) (s k e lo, b0 hi)
// (e, b0 lo) with b0 = s k r0 mod 2 pi, and the axes e1, e2.
__device__ __forceinline__ void store_frame(const ExpandProblem &P, int pair, const Frame &f) {
  float4 *q = reinterpret_cast<float4 *>(P.frames + 12 * (size_t)pair);
  q[0] = make_float4(f.ah[0], f.ah[1], f.ah[2], f.r0f);
  q[1] = make_float4(f.al[0], f.al[1], f.al[2], f.b0h);
  q[2] = make_float4(f.ef[0], f.ef[1], f.ef[2], f.b0l);
  float4 *b = reinterpret_cast<float4 *>(P.basis + 8 * (size_t)pair);
  b[0] = make_float4(f.e1[0], f.e1[1], f.e1[2], 0.f);
  b[1] = make_float4(f.e2[0], f.e2[1], f.e2[2], 0.f);
}

// a = ah + al plus b = bh + bl as a float-float pair.
__device__ __forceinline__ void add_ff(float ah, float al, float bh, float bl, float &h, float &l) {
  float s, e;
  two_sum(ah, bh, s, e);
  e = __fadd_rn(e, __fadd_rn(al, bl));
  h = __fadd_rn(s, e);
  l = __fsub_rn(e, __fsub_rn(h, s));
}

// s k rho of r = q + rho, rho = c / (q + r), c = |perpendicular offset|^2, to c^2:
// kap (c / q) (1 - c / 4q^2), kap = s k / 2 (the next term, c^3 / 16 q^5, is below 1e-7 rad where
// expand_choose admits the clusters).
__device__ __forceinline__ float curvature(float kap, float c, float q) {
  const float iq = ptx::rcp_approx(q), h = c * iq;
  return kap * h * fmaf(-0.25f * h, iq, 1.f);
}

// Mean error of cos.approx over a turn (GB300, 6.7e7 uniform angles; sin.approx has none).  Over
// sources of random phase every other error averages out, but this one adds up: over a
// cluster of 4096 it is sqrt(4096) 4e-8 = 2.6e-6 of the moment, more than all the rest
// (1.5e-6 of the 512^2 -> 1024^2 field with it, 6e-7 without).
constexpr float kCosBias = 4.034e-8f;

// (S + E + c) mod 2 pi for the curvature term c of some radians, |S| < 2^16: the turns are counted
// with c included and c is added where the reduced sum is small, so that the result stays
// within about [-pi, pi], where sin.approx is at its most exact (its product with 1 / 2 pi rounds
// by up to 7e-7 rad beyond a turn).
__device__ __forceinline__ float reduce_two_pi_with(float S, float E, float c) {
  const float n = __fsub_rn(fmaf(__fadd_rn(S, c), 0.159154943f, 12582912.0f), 12582912.0f);
  float r = __fadd_rn(fmaf(-n, 6.28125f, S), c);
  r = fmaf(-n, 1.935307169e-3f, r);   // fl32(2 pi - C1)
  r = fmaf(-n, 1.025313168e-11f, r);  // fl32(2 pi - C1 - C2)
  return __fadd_rn(r, E);
}

// Amplitudes that a block of the set-up looks at, and the blocks for n of them.
constexpr int kTopBlock = 4096;
__host__ __device__ __forceinline__ int top_blocks(int n) { return (n + kTopBlock - 1) / kTopBlock; }

// Exponent field of the power of two that the amplitudes are divided by, from the bits of the
// largest: moments, nodal weights and coefficients then stay far from the ends of the FP32
// range, whatever unit the caller's amplitudes are in (a low TF32 part of 1e-36 would be a
// subnormal of a few bits).  Powers of two: no other rounding than without.
__device__ __forceinline__ int scale_field(uint32_t top) {
  const int e = (int)(top >> 23);
  return top == 0u || e == 255 ? 127 : min(max(e, 1), 253);
}

// x times the scale, in its exponent (a product would take the FP64 pipe); a sum of two floats and
// a float's power of two stay far from the ends of the FP64 range.
__device__ __forceinline__ double scaled(double x, uint32_t field) {
  const int hi = __double2hiint(x), e = hi & 0x7ff00000;
  return e == 0 || e == 0x7ff00000
             ? x
             : __hiloint2double(hi + (((int)field - 127) << 20), __double2loint(x));
}

// ---- set-up: frames of all cluster pairs, largest amplitudes, offsets of the variant's tile centres from the
// cluster centres, Chebyshev tables ----
// Bound by the FP64 pipe's latency (a frame is ~150 dependent FP64 operations): one thread
// per pair, so a few thousand pairs run in the time of one.
template <bool BATCHED>
__global__ void __launch_bounds__(128) k_expand_setup(const ExpandProblem P0,
                                                      const ExpandProblem *__restrict__ probs,
                                                      const int *__restrict__ offs, int n_probs) {
  int item;
  const ExpandProblem &P = find_problem<BATCHED>(P0, probs, offs, n_probs, &item);
  const int tops = top_blocks(P.N);
  if (item < tops) {  // the largest of kTopBlock amplitudes (their bits order like the values)
    __shared__ uint32_t most[4];
    uint32_t m = 0;
    const int first = item * kTopBlock, last = min(P.N, first + kTopBlock);
    for (int j = first + threadIdx.x; j < last; j += 128)
      m = max(m, __float_as_uint(P.apf_s[j].y) & 0x7fffffffu);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) most[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) P.tops[item] = max(max(most[0], most[1]), max(most[2], most[3]));
    return;
  }
  int i = (item - tops) * blockDim.x + threadIdx.x;
  const int pairs = P.nTs * P.nS;
  if (i < pairs) {
    const int T = P.t0 + i / P.nS, S = i % P.nS;
    Frame f;
    build_frame(&f, P.box_t + 6 * (size_t)T, P.box_s + 6 * (size_t)S, P.sk);
    store_frame(P, i, f);
    return;
  }
  i -= pairs;
  const int leaves_s = box_count(P.N, 0), leaves_t = box_count(P.M, 0);
  if (i < leaves_s + leaves_t) {
    const bool src = i < leaves_s;
    const int j = src ? i : i - leaves_s;
    const double *c = src ? P.tiles_s + 6 * (size_t)(j * kLeafTile / P.cs)
                          : P.tiles_t + 6 * (size_t)(j * kLeafTile / P.tt);
    const double *b = src ? P.box_s + 6 * (size_t)(j * kLeafTile / P.ns)
                          : P.box_t + 6 * (size_t)(j * kLeafTile / P.nt);
    float *o = (src ? P.shift_s : P.shift_t) + 8 * (size_t)j;
    for (int d = 0; d < 3; ++d) {
      const double x = c[d] - b[d];
      o[d] = (float)x;
      o[4 + d] = (float)(x - (double)o[d]);
    }
    return;
  }
  i -= leaves_s + leaves_t;
  if (i < P.nS + P.nT) {
    const bool src = i < P.nS;
    const int j = src ? i : i - P.nS;
    const double *b = (src ? P.box_s : P.box_t) + 6 * (size_t)j;
    const float hx = (float)b[3 + P.ax], hy = (float)b[3 + P.ay];
    reinterpret_cast<float4 *>(src ? P.half_s : P.half_t)[j] =
        make_float4(hx, hy, hx > 0.f ? 1.f / hx : 0.f, hy > 0.f ? 1.f / hy : 0.f);
    return;
  }
  i -= P.nS + P.nT;
  if (i < 2 * kMaxP * kMaxP) {
    // M[a][j] = (2 - delta_a0) / p cos(pi a (2 j + 1) / 2p); row kMaxP^2 + j: node j
    const int axis = i / (kMaxP * kMaxP), a = i % (kMaxP * kMaxP) / kMaxP, j = i % kMaxP;
    const int p = axis ? P.py : P.px;
    float *tab = P.cheb + axis * (kMaxP * kMaxP + kMaxP);
    if (a < p && j < p)
      tab[a * kMaxP + j] = (a ? 2.f : 1.f) / (float)p *
                           cospif((float)((a * (2 * j + 1)) % (4 * p)) / (float)(2 * p));
    if (a == 0 && j < p) tab[kMaxP * kMaxP + j] = cospif((float)(2 * j + 1) / (float)(2 * p));
  }
}

// Float offset of record i of tile-ordered point arrays relative to its cluster's centre.  The
// shifts are per 256 points, so that tiles need not nest in the clusters (those of 768 do not).
__device__ __forceinline__ void cluster_offset(const float *geo, const float *shift, int i,
                                               float h[3], float l[3]) {
  const float2 *g = reinterpret_cast<const float2 *>(geo + 6 * (size_t)i);
  const float4 *s = reinterpret_cast<const float4 *>(shift + 8 * (size_t)(i / kLeafTile));
  const float2 g0 = g[0], g1 = g[1], g2 = g[2];
  const float4 sh = s[0], sl = s[1];
  add_ff(g0.x, g1.y, sh.x, sl.x, h[0], l[0]);
  add_ff(g0.y, g2.x, sh.y, sl.y, h[1], l[1]);
  add_ff(g1.x, g2.y, sh.z, sl.z, h[2], l[2]);
}

__device__ __forceinline__ float pick(const float v[3], int axis) {
  return axis == 0 ? v[0] : axis == 1 ? v[1] : v[2];
}

// T_0 .. T_{p-1}(x) to out[k * stride].
__device__ __forceinline__ void cheb_row(float x, int p, float *out, int stride) {
  float t0 = 1.f, t1 = x;
  for (int k = 0; k < p; ++k) {
    out[k * stride] = t0;
    const float t2 = fmaf(2.f * x, t1, -t0);
    t0 = t1;
    t1 = t2;
  }
}

// ---- moments -------------------------------------------------------------------------------
// One block: source cluster S, 64 target clusters, a share of S's sources; D[node][column] =
// sum over sources of weight x (re | im of a e^{i (phi + s k beta)}) for 64 + 64 columns.
// Per 16 sources every thread forms four sources' phasors for its target cluster (its frame
// stays in registers) and eight products T_a T_b of its node row, both split into TF32 parts,
// into one of two operand stages; one thread then issues the stage's six MMAs, and the other
// stage is filled while they run.
constexpr int kChebStride = kSuper + 4;  // 16-byte loads of eight rows hit eight bank groups
struct MomentsSmem {
  static constexpr size_t a = 0;                                // float [2][hi, lo][128*16]
  static constexpr size_t b = a + 4 * kNodes * kChunk * 4;      // float [2][hi, lo][128*16]
  static constexpr size_t cheb = b + 4 * 2 * kGroupT * kChunk * 4;  // float [2][16][68]
  static constexpr size_t rec = cheb + 2 * kMaxP * kChebStride * 4;  // float [9][64]
  static constexpr size_t bars = rec + 9 * kSuper * 4;          // uint64 [3]
  static constexpr size_t misc = bars + 4 * 8;                  // uint32 taddr, abort, spoilt, unscale
  static constexpr size_t bytes = misc + 16;
};
constexpr int kMomThreads = 256;

template <bool BATCHED>
__global__ void __launch_bounds__(kMomThreads, 2)
    k_expand_moments(const ExpandProblem P0, const ExpandProblem *__restrict__ probs,
                     const int *__restrict__ offs, int n_probs, int *err) {
  extern __shared__ __align__(128) unsigned char smem[];
  using L = MomentsSmem;
  constexpr int kStage = 2 * kNodes * kChunk;  // floats of one operand stage (hi, lo)
  float *sa = reinterpret_cast<float *>(smem + L::a), *sb = reinterpret_cast<float *>(smem + L::b);
  float *cheb = reinterpret_cast<float *>(smem + L::cheb);
  float *rec = reinterpret_cast<float *>(smem + L::rec);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::bars);  // free[2], full
  uint32_t *taddr_slot = reinterpret_cast<uint32_t *>(smem + L::misc);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L::misc + 4);
  volatile int *spoilt = reinterpret_cast<volatile int *>(smem + L::misc + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int b = 0; b < 3; ++b) ptx::mbar_init(&bars[b], 1);
    *abort_flag = 0;
    *spoilt = 0;
    ptx::fence_barrier_init();
  }
  if (warp == 0) ptx::tmem_alloc(taddr_slot, 256);

  int item;
  const ExpandProblem &P = find_problem<BATCHED>(P0, probs, offs, n_probs, &item);
  const int ks = item % P.ksplit, nTG = (P.nTs + kGroupT - 1) / kGroupT;
  const int tg = item / P.ksplit % nTG, S = item / P.ksplit / nTG;
  const int first = S * P.ns, count = min(P.ns, P.N - first);
  const int n_super = (count + kSuper - 1) / kSuper;
  const int sc0 = (int)((long long)n_super * ks / P.ksplit);
  const int sc1 = (int)((long long)n_super * (ks + 1) / P.ksplit);
  const int px = P.px, py = P.py, np = px * py;
  const float4 half = reinterpret_cast<const float4 *>(P.half_s)[S];
  const float kap = P.kap;
  // the sum's scale, for the staging threads; its exponent field for the target kernel
  float *unscale = reinterpret_cast<float *>(smem + L::misc + 12);
  if (warp == 1) {
    uint32_t m = 0;
    const int tops = top_blocks(P.N);
    for (int b = lane; b < tops; b += 32) m = max(m, P.tops[b]);
    const int e = scale_field(__reduce_max_sync(0xffffffffu, m));
    if (lane == 0) {
      *unscale = __uint_as_float((uint32_t)(254 - e) << 23);
      if (item == 0) P.tops[tops] = (uint32_t)e;
    }
  }

  // this thread's target cluster and its share of a chunk's sources
  const int tq = tid & (kGroupT - 1), quad = tid >> 6, Tl = tg * kGroupT + tq;
  float ah[3] = {0.f, 0.f, 0.f}, al[3] = {0.f, 0.f, 0.f}, ef[3] = {0.f, 0.f, 0.f}, r0 = 1.f;
  if (Tl < P.nTs) {
    const float4 *f = reinterpret_cast<const float4 *>(P.frames + 12 * ((size_t)Tl * P.nS + S));
    const float4 f0 = f[0], f1 = f[1], f2 = f[2];
    ah[0] = f0.x; ah[1] = f0.y; ah[2] = f0.z; r0 = f0.w;
    al[0] = f1.x; al[1] = f1.y; al[2] = f1.z;
    ef[0] = f2.x; ef[1] = f2.y; ef[2] = f2.z;
  }
  // this thread's node row (a, b) of the weight operand and its half of a chunk's sources
  const int row = tid & (kNodes - 1), khalf = tid >> 7;
  const float rmask = row < np ? 1.f : 0.f;
  const float *tab_x = cheb + (row < np ? row / py : 0) * kChebStride;
  const float *tab_y = cheb + (kMaxP + (row < np ? row % py : 0)) * kChebStride;

  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tbase = *taddr_slot;
  constexpr uint32_t idesc = ptx::tc_idesc_tf32(kNodes, 2 * kGroupT);
  // accumulators of this thread: node 32 (warp % 4) + lane, target clusters 32 (warp / 4) ..
  const uint32_t trow = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(32 * (warp >> 2));
  float acc_re[32], acc_im[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) acc_re[j] = acc_im[j] = 0.f;
  auto flush = [&](uint32_t col) {
    uint32_t v[16];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      ptx::tmem_ld16_nowait(trow + col + (uint32_t)(16 * (h & 1) + kGroupT * (h >> 1)), v);
      ptx::tmem_wait16(v);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (h < 2)
          acc_re[16 * h + j] += __uint_as_float(v[j]);
        else
          acc_im[16 * (h - 2) + j] += __uint_as_float(v[j]);
      }
    }
  };

  int g = 0;  // operand stages filled so far
  for (int sc = sc0; sc < sc1; ++sc) {
    // ---- stage 64 sources: offsets from the cluster centre, weights' factors ----
    __syncthreads();
    if (tid < 2 * kSuper) {
      const int i = tid & (kSuper - 1), axis = tid >> 6, idx = first + sc * kSuper + i;
      float h[3] = {0.f, 0.f, 0.f}, l[3] = {0.f, 0.f, 0.f};
      float2 pa = make_float2(0.f, 0.f);
      if (idx < P.N) {
        cluster_offset(P.geo_s, P.shift_s, idx, h, l);
        pa = P.apf_s[idx];
      }
      // a source that is not finite spoils the cluster's moments; it is looked for here, once
      // a source, because the splits into TF32 parts below turn a NaN into a zero
      const float zero = fmaf(0.f, h[0], fmaf(0.f, h[1], fmaf(0.f, h[2], fmaf(0.f, pa.x, 0.f * pa.y))));
      if (!(zero == 0.f)) *spoilt = 1;
      if (axis == 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          rec[d * kSuper + i] = h[d];
          rec[(3 + d) * kSuper + i] = l[d];
        }
        rec[6 * kSuper + i] = fmaf(h[0], h[0], fmaf(h[1], h[1], h[2] * h[2]));
        rec[7 * kSuper + i] = pa.x;
        rec[8 * kSuper + i] = pa.y * *unscale;
        cheb_row(pick(h, P.ax) * half.z, px, cheb + i, kChebStride);
      } else {
        cheb_row(pick(h, P.ay) * half.w, py, cheb + kMaxP * kChebStride + i, kChebStride);
      }
    }
    __syncthreads();
    for (int c = 0; c < kSuper / kChunk; ++c, ++g) {
      const int st = g & 1;
      float *a_hi = sa + st * kStage, *a_lo = a_hi + kNodes * kChunk;
      float *b_hi = sb + st * kStage, *b_lo = b_hi + kNodes * kChunk;
      if (g >= 2) tc_wait(&bars[st], ((g >> 1) - 1) & 1u, abort_flag, err);
      // ---- four phasors: sources 4 quad .. of the chunk for this thread's target cluster ----
      {
        float q[9][4];
#pragma unroll
        for (int f = 0; f < 9; ++f) {
          const float4 v = *reinterpret_cast<const float4 *>(rec + f * kSuper + kChunk * c + 4 * quad);
          q[f][0] = v.x; q[f][1] = v.y; q[f][2] = v.z; q[f][3] = v.w;
        }
        float re[4], im[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float th[3] = {q[0][j], q[1][j], q[2][j]}, tl[3] = {q[3][j], q[4][j], q[5][j]};
          float s, e, s2, e2;
          dot3_ff(ah, al, th, tl, s, e);
          two_sum(q[7][j], -s, s2, e2);
          const float ps = fmaf(ef[0], th[0], fmaf(ef[1], th[1], ef[2] * th[2]));
          const float ph = reduce_two_pi_with(
              s2, __fsub_rn(e2, e), curvature(kap, fmaf(-ps, ps, q[6][j]), r0 - ps));
          re[j] = fmaf(q[8][j], ptx::cos_approx(ph), -kCosBias * q[8][j]);
          im[j] = q[8][j] * ptx::sin_approx(ph);
        }
        const int o = (quad >> 1) * (2 * kGroupT * kTcK) + 32 * (quad & 1);
        const int ore = o + tc_off(tq, 0), oim = o + tc_off(kGroupT + tq, 0);
        float hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          hi[j] = ptx::to_tf32_int(re[j]);
          lo[j] = ptx::to_tf32_int(__fsub_rn(re[j], hi[j]));
        }
        *reinterpret_cast<float4 *>(b_hi + ore) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4 *>(b_lo + ore) = make_float4(lo[0], lo[1], lo[2], lo[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          hi[j] = ptx::to_tf32_int(im[j]);
          lo[j] = ptx::to_tf32_int(__fsub_rn(im[j], hi[j]));
        }
        *reinterpret_cast<float4 *>(b_hi + oim) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4 *>(b_lo + oim) = make_float4(lo[0], lo[1], lo[2], lo[3]);
      }
      // ---- eight weights: node row `row`, sources 8 khalf .. of the chunk ----
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = kChunk * c + 8 * khalf + 4 * h;
        const float4 x = *reinterpret_cast<const float4 *>(tab_x + k);
        const float4 y = *reinterpret_cast<const float4 *>(tab_y + k);
        const float w[4] = {rmask * x.x * y.x, rmask * x.y * y.y, rmask * x.z * y.z,
                            rmask * x.w * y.w};
        float hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          hi[j] = ptx::to_tf32_int(w[j]);
          lo[j] = ptx::to_tf32_int(__fsub_rn(w[j], hi[j]));
        }
        const int o = khalf * (kNodes * kTcK) + tc_off(row, 4 * h);
        *reinterpret_cast<float4 *>(a_hi + o) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4 *>(a_lo + o) = make_float4(lo[0], lo[1], lo[2], lo[3]);
      }
      ptx::fence_proxy_async_smem();
      ptx::tc_fence_before();
      __syncthreads();
      if (tid == 0 && !*abort_flag) {
        ptx::tc_fence_after();
#pragma unroll
        for (int k = 0; k < kChunk / kTcK; ++k) {
          const uint64_t dah = ptx::tc_smem_desc(a_hi + k * kNodes * kTcK, kTcLbo, kTcSbo);
          const uint64_t dal = ptx::tc_smem_desc(a_lo + k * kNodes * kTcK, kTcLbo, kTcSbo);
          const uint64_t dbh = ptx::tc_smem_desc(b_hi + k * kNodes * kTcK, kTcLbo, kTcSbo);
          const uint64_t dbl = ptx::tc_smem_desc(b_lo + k * kNodes * kTcK, kTcLbo, kTcSbo);
          ptx::tc_mma_tf32(tbase, dah, dbh, idesc, c > 0 || k > 0);
          ptx::tc_mma_tf32(tbase + 128, dah, dbl, idesc, g > 0 || k > 0);
          ptx::tc_mma_tf32(tbase + 128, dal, dbh, idesc, 1u);
        }
        ptx::tc_commit(&bars[st]);
        if (c == kSuper / kChunk - 1) ptx::tc_commit(&bars[2]);
      }
    }
    // ---- the 64 sources' sums into registers (the next MMA overwrites them after the
    // barrier that follows these loads) ----
    if (__all_sync(0xffffffffu, tc_wait(&bars[2], (sc - sc0) & 1u, abort_flag, err))) {
      ptx::tc_fence_after();
      flush(0);
      ptx::tc_fence_before();
    }
  }
  if (sc1 > sc0 && !*abort_flag) {
    __syncwarp();
    ptx::tc_fence_after();
    flush(128);
  }
  const int node = 32 * (warp & 3) + lane;
  // (every staging is behind a barrier of its chunks)
  const float nan = *spoilt ? __int_as_float(0x7fffffff) : 0.f;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const int T = tg * kGroupT + 32 * (warp >> 2) + j;
    if (T < P.nTs)
      P.moments[((size_t)ks * P.nTs * P.nS + (size_t)T * P.nS + S) * kNodes + node] =
          make_float2(acc_re[j] + nan, acc_im[j] + nan);
  }
  // every commit has arrived before the block ends
  if (tid == 0)
    for (int b = 0; b < 2; ++b)
      if (g > b) ptx::mbar_wait_bounded(&bars[b], ((g - 1 - b) >> 1) & 1u, kWaitCycles);
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  if (warp == 0) ptx::tmem_dealloc(tbase, 256);
}

// x rounded to TF32; NaN and infinities as they are (to_tf32_int's carry runs a NaN's fraction over
// into the sign: -0).
__device__ __forceinline__ float tf32_or_nonfinite(float x) {
  return __fsub_rn(x, x) == 0.f ? ptx::to_tf32_int(x) : x;
}

// ---- translate -----------------------------------------------------------------------------
// One block per cluster pair, one thread per node: moments to nodal weights, the px py x px py
// products with G formed on the fly (one reciprocal, sine and cosine per node pair: bound by
// the MUFU and FP32 pipes together), then back to Chebyshev coefficients, written as the TF32
// operand that the target kernel stages.
template <bool BATCHED>
__global__ void __launch_bounds__(kNodes) k_expand_translate(
    const ExpandProblem P0, const ExpandProblem *__restrict__ probs, const int *__restrict__ offs,
    int n_probs) {
  __shared__ float2 va[kNodes], vb[kNodes];
  __shared__ float tab[2][kMaxP * kMaxP + kMaxP];
  __shared__ float4 node_a[kNodes], node_b[kNodes];
  int item;
  const ExpandProblem &P = find_problem<BATCHED>(P0, probs, offs, n_probs, &item);
  const int Tl = item / P.nS, S = item % P.nS, n = threadIdx.x;
  const int px = P.px, py = P.py, np = px * py;
  const size_t pairs = (size_t)P.nTs * P.nS;
  for (int i = n; i < 2 * (kMaxP * kMaxP + kMaxP); i += kNodes)
    tab[i / (kMaxP * kMaxP + kMaxP)][i % (kMaxP * kMaxP + kMaxP)] = P.cheb[i];
  float2 mu = make_float2(0.f, 0.f);
  for (int k = 0; k < P.ksplit; ++k) {
    const float2 v = P.moments[(k * pairs + item) * kNodes + n];
    mu.x += v.x;
    mu.y += v.y;
  }
  va[n] = mu;
  const float4 *f = reinterpret_cast<const float4 *>(P.frames + 12 * (size_t)item);
  const float4 *fb = reinterpret_cast<const float4 *>(P.basis + 8 * (size_t)item);
  const float4 f0 = f[0], f2 = f[2], f3 = fb[0], f4 = fb[1];
  const float kap = P.kap, r0 = f0.w;
  const int a = n / py, b = n % py;  // Chebyshev order or node along each axis
  const float *mx = tab[0], *my = tab[1];
  __syncthreads();
  // nodal weights: M^T mu M, one axis at a time
  if (n < np) {
    float2 s = make_float2(0.f, 0.f);
    for (int j = 0; j < py; ++j) {
      const float m = my[j * kMaxP + b];
      const float2 v = va[a * py + j];
      s.x = fmaf(m, v.x, s.x);
      s.y = fmaf(m, v.y, s.y);
    }
    vb[n] = s;
  }
  __syncthreads();
  // node n of both clusters: offsets in the pair's frame
  float tx = 0.f, ty = 0.f, tz = 0.f, ct = 0.f, rt = 0.f;
  if (n < np) {
    float2 s = make_float2(0.f, 0.f);
    for (int i = 0; i < px; ++i) {
      const float m = mx[i * kMaxP + a];
      const float2 v = vb[i * py + b];
      s.x = fmaf(m, v.x, s.x);
      s.y = fmaf(m, v.y, s.y);
    }
    const float x = mx[kMaxP * kMaxP + a], y = my[kMaxP * kMaxP + b];
    const float ex[3] = {f2.x, f2.y, f2.z}, e1[3] = {f3.x, f3.y, f3.z}, e2[3] = {f4.x, f4.y, f4.z};
    const float4 ht = reinterpret_cast<const float4 *>(P.half_t)[P.t0 + Tl];
    const float4 hs = reinterpret_cast<const float4 *>(P.half_s)[S];
    const float ux = x * ht.x, uy = y * ht.y;
    const float e1x = pick(e1, P.ax), e1y = pick(e1, P.ay), e2x = pick(e2, P.ax);
    const float e2y = pick(e2, P.ay), exx = pick(ex, P.ax), exy = pick(ex, P.ay);
    tx = fmaf(e1x, ux, e1y * uy);
    ty = fmaf(e2x, ux, e2y * uy);
    tz = fmaf(exx, ux, exy * uy);
    ct = fmaf(tx, tx, ty * ty);
    rt = curvature(kap, ct, r0 + tz);
    const float wx = x * hs.x, wy = y * hs.y;
    const float sx = fmaf(e1x, wx, e1y * wy), sy = fmaf(e2x, wx, e2y * wy);
    const float sz = fmaf(exx, wx, exy * wy), cs = fmaf(sx, sx, sy * sy);
    node_a[n] = make_float4(-2.f * sx, -2.f * sy, sz, cs);
    node_b[n] = make_float4(s.x, s.y, curvature(kap, cs, r0 - sz), 0.f);
  }
  __syncthreads();
  // V_n = sum_j e^{i s k psi} / r W_j, psi = c u - c_t u_t - c_s u_s with c = c_t + c_s - 2 t.s
  // (the same regrouped into small differences, -2 t.s u + c_t (u - u_t) + c_s (u - u_s), took 16 %
  // longer and was no more exact in the field)
  float vre = 0.f, vim = 0.f;
  const float qt = r0 + tz;
#pragma unroll 4
  for (int j = 0; j < np; ++j) {
    const float4 s = node_a[j], w = node_b[j];
    const float c = fmaf(tx, s.x, fmaf(ty, s.y, ct + s.w)), iq = ptx::rcp_approx(qt - s.z);
    const float h = c * iq;
    const float psi = kap * h * fmaf(-0.25f * h, iq, 1.f) - rt - w.z;
    const float ir = iq * fmaf(-0.5f * h, iq, 1.f);  // 1 / r to c / q^2
    const float cr = ir * ptx::cos_approx(psi), ci = ir * ptx::sin_approx(psi);
    vre = fmaf(cr, w.x, fmaf(-ci, w.y, vre));
    vim = fmaf(cr, w.y, fmaf(ci, w.x, vim));
  }
  va[n] = make_float2(vre, vim);
  __syncthreads();
  // Chebyshev coefficients of the nodal values: M V M^T
  if (n < np) {
    float2 s = make_float2(0.f, 0.f);
    for (int i = 0; i < px; ++i) {
      const float m = mx[a * kMaxP + i];
      const float2 v = va[i * py + b];
      s.x = fmaf(m, v.x, s.x);
      s.y = fmaf(m, v.y, s.y);
    }
    vb[n] = s;
  }
  __syncthreads();
  // thread n: the coefficient of slot n of the MMA depth
  float2 nu = make_float2(0.f, 0.f);
  if (n < 4 * P.n_quads) {
    const uint32_t quad = P.quads[n >> 2];
    const int one = (quad >> 8) & 255, four = 4 * (quad & 255) + (n & 3);
    const int oa = quad >> 16 ? four : one, ob = quad >> 16 ? one : four;
    if (oa < px && ob < py)
      for (int j = 0; j < py; ++j) {
        const float m = my[ob * kMaxP + j];
        const float2 v = vb[oa * py + j];
        nu.x = fmaf(m, v.x, nu.x);
        nu.y = fmaf(m, v.y, nu.y);
      }
  }
  // operand rows S % 32 (re), 32 + S % 32 (im) and, 64 rows on, their TF32 remainders; depth n
  const int nSG = (P.nS + kGroupS - 1) / kGroupS, row = S % kGroupS;
  float *o = P.coeffs + ((size_t)Tl * nSG + S / kGroupS) * 2 * kHalfFloats +
             (size_t)(n >> 3) * (4 * kGroupS * kTcK);
  const float rh = tf32_or_nonfinite(nu.x), ih = tf32_or_nonfinite(nu.y);
  o[tc_off(row, n & 7)] = rh;
  o[tc_off(kGroupS + row, n & 7)] = ih;
  o[tc_off(2 * kGroupS + row, n & 7)] = tf32_or_nonfinite(__fsub_rn(nu.x, rh));
  o[tc_off(3 * kGroupS + row, n & 7)] = tf32_or_nonfinite(__fsub_rn(nu.y, ih));
}

// ---- targets -------------------------------------------------------------------------------
// Work items are blocks of 128 targets of one cluster against a share of the source clusters:
// D[target][column] = sum over nodes of weight x coefficient, 32 clusters (32 + 32 columns)
// at a time.  Persistent CTAs, one per SM, with a role per warp so that an item's weights are
// built and its coefficients fetched while the previous item's phases are formed:
//   builders (8 warps)   the weights of the next item's targets into tensor memory (the MMAs' A
//                        operand, both TF32 parts) once the MMAs of this one are complete,
//                        the targets' offsets, and the results of the item before
//   load warp            coefficients (halves of 64 nodes) and frames by bulk copies
//   MMA warp             one thread issues the products into one of two TMEM buffers
//   consumers (16 warps) read D, rotate by e^{i s k alpha}, sum: each thread one target and
//                        8 clusters of every 32
// Bound by issue slots: an item of 64 source clusters takes 13,300 clocks (512^2 -> 1024^2: 54 items
// a CTA, 0.37 ms, ncu: 65 % of the slots issue), most of them the consumers' FP32 work; a block
// per item without roles took 12,000 clocks of set-up and tail per item beside that.  Hand-offs are mbarrier phases; those a waiter may trail by two items come in
// pairs.
struct TargetsSmem {
  static constexpr int kStages = 4;                                 // halves of coefficients
  static constexpr size_t b = 0;                                    // float [4][kHalfFloats]
  static constexpr size_t quad = b + kStages * kHalfFloats * 4;     // float4 [8][128]: four orders
  static constexpr size_t cheb = quad + 8 * kBlockT * 16;           // float [24][128]
  static constexpr size_t rec = cheb + 24 * kBlockT * 4;            // float [2][7][128]
  static constexpr size_t part = rec + 2 * 7 * kBlockT * 4;         // float4 [4][128]
  static constexpr size_t frames = part + 4 * kBlockT * 16;         // float [2][32][12]
  static constexpr size_t bars = frames + 2 * kGroupS * 12 * 4;     // uint64 [21]
  static constexpr size_t misc = bars + 22 * 8;                     // uint32 taddr, abort
  static constexpr size_t bytes = misc + 16;
};
static_assert(TargetsSmem::bytes <= 227 * 1024, "target kernel: shared memory");
constexpr int kTgtConsumers = 16, kTgtBuilders = 8;
constexpr int kTgtThreads = 32 * (kTgtConsumers + 2 + kTgtBuilders);

template <bool BATCHED>
__global__ void __launch_bounds__(kTgtThreads, 1)
    k_expand_targets(const ExpandProblem P0, const ExpandProblem *__restrict__ probs,
                     const int *__restrict__ offs, int n_items, int *err) {
  extern __shared__ __align__(128) unsigned char smem[];
  using L = TargetsSmem;
  constexpr int kStages = L::kStages;
  float *sb = reinterpret_cast<float *>(smem + L::b);
  float4 *squad = reinterpret_cast<float4 *>(smem + L::quad);
  float *cheb = reinterpret_cast<float *>(smem + L::cheb);
  float *srec = reinterpret_cast<float *>(smem + L::rec);
  float4 *part = reinterpret_cast<float4 *>(smem + L::part);
  float *sframes = reinterpret_cast<float *>(smem + L::frames);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::bars);
  uint64_t *bfull = bars, *bfree = bars + 4, *dfull = bars + 8, *dfree = bars + 10,
           *ffull = bars + 12, *ffree = bars + 14, *a_ready = bars + 16, *a_free = bars + 18,
           *parts_ready = bars + 19, *parts_free = bars + 20;
  uint32_t *taddr_slot = reinterpret_cast<uint32_t *>(smem + L::misc);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L::misc + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool consumer = warp < kTgtConsumers, mma_warp = warp == kTgtConsumers,
             load_warp = warp == kTgtConsumers + 1;
  if (tid == 0) {
    for (int b = 0; b < kStages; ++b) {
      ptx::mbar_init(&bfull[b], 1);
      ptx::mbar_init(&bfree[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&dfull[b], 1);
      ptx::mbar_init(&dfree[b], kTgtConsumers);
      ptx::mbar_init(&ffull[b], 1);
      ptx::mbar_init(&ffree[b], kTgtConsumers);
      ptx::mbar_init(&a_ready[b], 32 * kTgtBuilders);
    }
    ptx::mbar_init(a_free, 1);
    ptx::mbar_init(parts_ready, kTgtConsumers);
    ptx::mbar_init(parts_free, kBlockT);
    *abort_flag = 0;
    ptx::fence_barrier_init();
  }
  if (mma_warp) ptx::tmem_alloc(taddr_slot, 512);  // D[2] 128 columns, weights hi and lo 128
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tbase = *taddr_slot;

  // item -> problem (items of a CTA only go up, so the search goes on from the last one),
  // target cluster (of the slab), first target, source cluster groups [g0, g1)
  int prob = 0, first = 0, next = BATCHED ? offs[1] : n_items;
  struct Item {
    int Tl, m0, sp, nSG, g0, g1;
  };
  auto locate = [&](int item, Item &w) -> const ExpandProblem & {
    if (BATCHED)
      while (item >= next) {
        first = next;
        ++prob;
        next = offs[prob + 1];
      }
    const ExpandProblem &P = BATCHED ? probs[prob] : P0;
    const int blk = (item - first) / P.ssplit;
    w.sp = (item - first) % P.ssplit;
    w.m0 = P.t0 * P.nt + blk * kBlockT;
    w.Tl = blk * kBlockT / P.nt;
    w.nSG = (P.nS + kGroupS - 1) / kGroupS;
    w.g0 = (int)((long long)w.nSG * w.sp / P.ssplit);
    w.g1 = (int)((long long)w.nSG * (w.sp + 1) / P.ssplit);
    return P;
  };

  Item w;
  if (mma_warp) {
    const uint32_t leader = lane == 0;
    constexpr uint32_t idesc = ptx::tc_idesc_tf32(kBlockT, 4 * kGroupS);
    constexpr uint32_t idesc_lo = ptx::tc_idesc_tf32(kBlockT, 2 * kGroupS);
    // one k step of 8 nodes further: 8 columns of weights, 4096 bytes of coefficients
    constexpr uint64_t kStepB = 4 * kGroupS * kTcK * 4 / 16;
    const uint32_t ta = tbase + 256;
    const uint64_t db0 = ptx::tc_smem_desc(sb, kTcLbo, kTcSbo);
    uint32_t hc = 0, gc = 0, it = 0;  // halves, groups and items so far
    for (int item = blockIdx.x; item < n_items; item += gridDim.x, ++it) {
      const ExpandProblem &P = locate(item, w);
      const int steps = (P.n_quads + 1) / 2;
      if (!tc_wait(&a_ready[it & 1], (it >> 1) & 1u, abort_flag, err)) break;
      for (int g = w.g0; g < w.g1 && !*abort_flag; ++g, ++gc) {
        const uint32_t d = gc & 1, dt = tbase + 4 * kGroupS * d;
        if (gc >= 2 && !tc_wait(&dfree[d], ((gc >> 1) - 1) & 1u, abort_flag, err)) break;
        uint32_t acc = 0;
        for (int half = steps > 8; half >= 0; --half, ++hc) {
          const uint32_t st = hc % kStages;
          if (!tc_wait(&bfull[st], (hc / kStages) & 1u, abort_flag, err)) break;
          ptx::tc_fence_after();
          const uint64_t b = db0 + st * (kHalfFloats * 4 / 16);
          const uint32_t a = ta + 64 * half;
          const int n = min(8, steps - 8 * half);
#pragma unroll
          for (int k = 7; k >= 0; --k) {
            if (k >= n) continue;
            // hi x (hi | lo), then lo x hi onto the second product
            ptx::tc_mma_tf32_ta(dt, a + 8 * k, b + k * kStepB, idesc, acc, leader);
            ptx::tc_mma_tf32_ta(dt + 2 * kGroupS, a + 128 + 8 * k, b + k * kStepB, idesc_lo, 1u, leader);
            acc = 1u;
          }
          ptx::tc_commit(&bfree[st], leader);
        }
        ptx::tc_commit(&dfull[d], leader);
      }
      ptx::tc_commit(a_free, leader);
    }
    // the MMAs in flight end before the CTA does
    if (it > 0) ptx::mbar_wait_bounded(a_free, (it - 1) & 1u, kWaitCycles);
    for (uint32_t h = hc > kStages ? hc - kStages : 0; h < hc; ++h)
      ptx::mbar_wait_bounded(&bfree[h % kStages], (h / kStages) & 1u, kWaitCycles);
    __syncwarp();
  } else if (load_warp) {
    if (lane == 0) {
      uint32_t hc = 0, gc = 0;
      for (int item = blockIdx.x; item < n_items && !*abort_flag; item += gridDim.x) {
        const ExpandProblem &P = locate(item, w);
        const int steps = (P.n_quads + 1) / 2;
        for (int g = w.g0; g < w.g1 && !*abort_flag; ++g, ++gc) {
          const uint32_t d = gc & 1;
          if (gc >= 2 && !tc_wait(&ffree[d], ((gc >> 1) - 1) & 1u, abort_flag, err)) break;
          const uint32_t bytes = 48 * min(kGroupS, P.nS - g * kGroupS);
          ptx::mbar_arrive_expect_tx(&ffull[d], bytes);
          ptx::bulk_g2s(sframes + d * kGroupS * 12,
                        P.frames + 12 * ((size_t)w.Tl * P.nS + g * kGroupS), bytes, &ffull[d]);
          for (int half = steps > 8; half >= 0; --half, ++hc) {
            const uint32_t st = hc % kStages, bytes_b = 4 * 4 * kGroupS * kTcK * min(8, steps - 8 * half);
            if (hc >= kStages && !tc_wait(&bfree[st], (hc / kStages - 1) & 1u, abort_flag, err)) break;
            ptx::mbar_arrive_expect_tx(&bfull[st], bytes_b);
            ptx::bulk_g2s(sb + st * kHalfFloats,
                          P.coeffs + (((size_t)w.Tl * w.nSG + g) * 2 + half) * kHalfFloats, bytes_b,
                          &bfull[st]);
          }
        }
      }
      // and so do the copies
      for (uint32_t h = hc > kStages ? hc - kStages : 0; h < hc; ++h)
        ptx::mbar_wait_bounded(&bfull[h % kStages], (h / kStages) & 1u, kWaitCycles);
      for (uint32_t g = gc > 2 ? gc - 2 : 0; g < gc; ++g)
        ptx::mbar_wait_bounded(&ffull[g & 1], (g >> 1) & 1u, kWaitCycles);
    }
    __syncwarp();
  } else if (consumer) {
    const int cg = warp >> 2, row = 32 * (warp & 3) + lane;
    const uint32_t trow = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(8 * cg);
    uint32_t gc = 0, it = 0;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x, ++it) {
      const ExpandProblem &P = locate(item, w);
      const float kap = P.kap;
      const int nS = P.nS;
      if (!__all_sync(0xffffffffu, tc_wait(&a_ready[it & 1], (it >> 1) & 1u, abort_flag, err))) break;
      const float *r = srec + (it & 1) * 7 * kBlockT + row;
      const float th[3] = {r[0], r[kBlockT], r[2 * kBlockT]};
      const float tl[3] = {r[3 * kBlockT], r[4 * kBlockT], r[5 * kBlockT]};
      const float t2 = r[6 * kBlockT];
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);  // (re hi, re lo, im hi, im lo)
      bool ok = true;
      for (int g = w.g0; g < w.g1; ++g, ++gc) {
        const uint32_t d = gc & 1, ph2 = (gc >> 1) & 1u;
        const int left = min(8, nS - g * kGroupS - 8 * cg);
        ok = __all_sync(0xffffffffu, tc_wait(&dfull[d], ph2, abort_flag, err) &&
                                         tc_wait(&ffull[d], ph2, abort_flag, err));
        if (!ok) break;
        ptx::tc_fence_after();
        uint32_t vr[8], vi[8], wr[8], wi[8];
        ptx::tmem_ld8_nowait(trow + 4 * kGroupS * d, vr);
        ptx::tmem_ld8_nowait(trow + 4 * kGroupS * d + kGroupS, vi);
        ptx::tmem_ld8_nowait(trow + 4 * kGroupS * d + 2 * kGroupS, wr);
        ptx::tmem_ld8_nowait(trow + 4 * kGroupS * d + 3 * kGroupS, wi);
        ptx::tmem_wait8(vr);
        ptx::tmem_wait8(vi);
        ptx::tmem_wait8(wr);
        ptx::tmem_wait8(wi);
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&dfree[d]);
        const float4 *f = reinterpret_cast<const float4 *>(sframes + (d * kGroupS + 8 * cg) * 12);
        float gr = 0.f, gim = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (j < left) {
            const float4 f0 = f[3 * j], f1 = f[3 * j + 1], f2 = f[3 * j + 2];
            const float ah[3] = {f0.x, f0.y, f0.z}, al[3] = {f1.x, f1.y, f1.z};
            float s, e, s2, e2;
            dot3_ff(ah, al, th, tl, s, e);
            two_sum(s, f1.w, s2, e2);
            const float tz = fmaf(f2.x, th[0], fmaf(f2.y, th[1], f2.z * th[2]));
            const float ph =
                reduce_two_pi_with(s2, __fadd_rn(__fadd_rn(e, e2), f2.w),
                                   curvature(kap, fmaf(-tz, tz, t2), f0.w + tz));
            const float cr = ptx::cos_approx(ph), sr = ptx::sin_approx(ph);
            const float re = __uint_as_float(vr[j]) + __uint_as_float(wr[j]);
            const float im = __uint_as_float(vi[j]) + __uint_as_float(wi[j]);
            gr = fmaf(re, cr, fmaf(-im, sr, gr));
            gim = fmaf(re, sr, fmaf(im, cr, gim));
          }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&ffree[d]);
        float h, e;
        two_sum(sum.x, gr, h, e);
        sum.x = h;
        sum.y = __fadd_rn(sum.y, e);
        two_sum(sum.z, gim, h, e);
        sum.z = h;
        sum.w = __fadd_rn(sum.w, e);
      }
      if (!ok) break;
      if (it > 0 &&
          !__all_sync(0xffffffffu, tc_wait(parts_free, (it - 1) & 1u, abort_flag, err)))
        break;
      part[cg * kBlockT + row] = sum;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(parts_ready);
    }
  } else {
    // ---- builders: thread (row, half): 64 nodes of one target's weights.  After a timeout
    // they go on (every wait then returns at once): their barrier needs all of them ----
    // (a warp reaches the 32 TMEM lanes of its index mod 4: rows follow from that)
    const int bt = tid - 32 * (kTgtConsumers + 2), row = 32 * (warp & 3) + lane, half = bt >> 7;
    auto bar_builders = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    static_assert(32 * kTgtBuilders == 256, "builders' named barrier");
    uint32_t it = 0;
    // the four warps of a target add their clusters' sums; results of an item
    int out_t = -1, out_sp = 0;
    const ExpandProblem *out_p = nullptr;
    auto write_out = [&](uint32_t i) {
      if (half) return;
      const int order = out_t >= 0 && out_p->ssplit == 1 ? out_p->order_t[out_t] : 0;
      const uint32_t field = out_t >= 0 ? out_p->tops[top_blocks(out_p->N)] : 127u;
      if (!tc_wait(parts_ready, i & 1u, abort_flag, err)) return;
      float4 s = part[row];
#pragma unroll
      for (int c = 1; c < 4; ++c) {
        const float4 v = part[c * kBlockT + row];
        float h, e;
        two_sum(s.x, v.x, h, e);
        s.x = h;
        s.y = __fadd_rn(s.y, __fadd_rn(v.y, e));
        two_sum(s.z, v.z, h, e);
        s.z = h;
        s.w = __fadd_rn(s.w, __fadd_rn(v.w, e));
      }
      ptx::mbar_arrive(parts_free);
      if (out_t >= 0) {
        const double2 v = make_double2(scaled((double)s.x + (double)s.y, field),
                                       scaled((double)s.z + (double)s.w, field));
        if (out_p->ssplit == 1)
          out_p->y[order] = v;
        else
          out_p->partial[(size_t)out_sp * out_p->M + out_t] = v;
      }
    };
    for (int item = blockIdx.x; item < n_items; item += gridDim.x, ++it) {
      const ExpandProblem &P = locate(item, w);
      const int px = P.px, py = P.py, np = px * py, t = w.m0 + row;
      float th[3] = {0.f, 0.f, 0.f}, tl[3] = {0.f, 0.f, 0.f};
      if (t < P.M) cluster_offset(P.geo_t, P.shift_t, t, th, tl);
      const float4 hx = reinterpret_cast<const float4 *>(P.half_t)[P.t0 + w.Tl];
      // the builders' reads of the last item's factors are behind the barrier below; its
      // records' buffer was released with the parts of item - 2
      {
        // T_0 .. T_{p-1} along one axis, as scalars and as fours (zero past the last)
        const int p = half ? py : px;
        const float x = half ? pick(th, P.ay) * hx.w : pick(th, P.ax) * hx.z;
        float *o = cheb + (half ? px : 0) * kBlockT + row;
        float4 *q = squad + (half ? 0 : 4) * kBlockT + row;
        float t0 = 1.f, t1 = x;
        for (int k = 0; k < p; k += 4) {
          float v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            v[j] = k + j < p ? t0 : 0.f;
            if (k + j < p) o[(k + j) * kBlockT] = t0;
            const float t2 = fmaf(2.f * x, t1, -t0);
            t0 = t1;
            t1 = t2;
          }
          q[(k / 4) * kBlockT] = make_float4(v[0], v[1], v[2], v[3]);
        }
      }
      if (half == 0) {
        float *r = srec + (it & 1) * 7 * kBlockT + row;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          r[d * kBlockT] = th[d];
          r[(3 + d) * kBlockT] = tl[d];
        }
        r[6 * kBlockT] = fmaf(th[0], th[0], fmaf(th[1], th[1], th[2] * th[2]));
      }
      bar_builders();
      if (it > 0) tc_wait(a_free, (it - 1) & 1u, abort_flag, err);
      ptx::tc_fence_after();
      // two quads (8 columns) at a time: one factor times four; the tensor cores drop the low
      // 13 bits, so the product itself is the high part and what it loses, rounded, the low
      const uint32_t acol = tbase + 256 + ((uint32_t)(32 * (warp & 3)) << 16);
      const int q1 = min(16 * half + 16, (P.n_quads + 1) / 2 * 2);
      for (int q = 16 * half; q < q1; q += 2) {
        float hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t c = P.quads[q + j];
          const bool along_x = c >> 16;
          const float s = cheb[((along_x ? px : 0) + (int)((c >> 8) & 255)) * kBlockT + row];
          const float4 f = squad[((along_x ? 4 : 0) + (int)(c & 255)) * kBlockT + row];
          const float v[4] = {s * f.x, s * f.y, s * f.z, s * f.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            hi[4 * j + e] = v[e];
            const float r = __fsub_rn(v[e], __uint_as_float(__float_as_uint(v[e]) & 0xffffe000u));
            lo[4 * j + e] = __uint_as_float(__float_as_uint(r) + 0x1000u);
          }
        }
        ptx::tmem_st8(acol + 4 * q, hi);
        ptx::tmem_st8(acol + 128 + 4 * q, lo);
      }
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      ptx::mbar_arrive(&a_ready[it & 1]);
      if (it > 0) write_out(it - 1);
      bar_builders();  // the factors are rewritten next; both halves of the results are out
      out_t = t < P.M ? t : -1;
      out_sp = w.sp;
      out_p = &P;
    }
    if (it > 0) write_out(it - 1);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  if (mma_warp) ptx::tmem_dealloc(tbase, 512);
}

}  // namespace

void expand_blocks(const ExpandProblem &p, int blocks[4]) {
  const long long n = (long long)p.nTs * p.nS + box_count(p.N, 0) + box_count(p.M, 0) +
                      p.nS + p.nT + 2 * kMaxP * kMaxP;
  blocks[0] = top_blocks(p.N) + (int)((n + 127) / 128);
  blocks[1] = p.nS * ((p.nTs + kGroupT - 1) / kGroupT) * p.ksplit;
  blocks[2] = p.nS * p.nTs;
  const long long m0 = (long long)p.t0 * p.nt, m1 = (long long)(p.t0 + p.nTs) * p.nt;
  const long long m = (m1 < p.M ? m1 : p.M) - m0;
  blocks[3] = (int)((m + kBlockT - 1) / kBlockT) * p.ssplit;
}

template <bool BATCHED>
static int launch_all(const ExpandProblem &p, const ExpandProblem *probs, const int *offs,
                      const int *blocks, int n, int sms, int *err, cudaStream_t s) {
  HOLO_TRY((kernel_setup<k_expand_moments<BATCHED>>(kMomThreads, (int)MomentsSmem::bytes, nullptr)));
  HOLO_TRY((kernel_setup<k_expand_targets<BATCHED>>(kTgtThreads, (int)TargetsSmem::bytes, nullptr)));
  const int step = BATCHED ? n + 1 : 0;
  k_expand_setup<BATCHED><<<blocks[0], 128, 0, s>>>(p, probs, offs, n);
  k_expand_moments<BATCHED><<<blocks[1], kMomThreads, MomentsSmem::bytes, s>>>(p, probs, offs + step,
                                                                              n, err);
  k_expand_translate<BATCHED><<<blocks[2], kNodes, 0, s>>>(p, probs, offs + 2 * step, n);
  k_expand_targets<BATCHED><<<std::min(blocks[3], sms), kTgtThreads, TargetsSmem::bytes, s>>>(
      p, probs, offs + 3 * step, blocks[3], err);
  note_launches(4);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_expand(const ExpandProblem &p, int sms, int *err, cudaStream_t s) {
  int blocks[4];
  expand_blocks(p, blocks);
  return launch_all<false>(p, nullptr, nullptr, blocks, 1, sms, err, s);
}

int launch_expand_batched(const ExpandProblem *probs_dev, const int *offs_dev, const int *totals,
                          int n, int sms, int *err, cudaStream_t s) {
  if (n <= 0) return HOLO_OK;
  return launch_all<true>(ExpandProblem{}, probs_dev, offs_dev, totals, n, sms, err, s);
}

}  // namespace holo
