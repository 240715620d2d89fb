// expand_plan.cu -- when and how a HOLO_SPLIT32 sum runs by cluster expansions
// (kernel_expand.cu), and its launches.
#include <math.h>

#include <algorithm>

#include "expand_plan.h"

namespace holo {

namespace {

// Largest error of the p-node Chebyshev interpolant of e^{i z x}, |x| <= 1.
double truncation(double z, int p) {
  double e = 2.0;
  for (int j = 1; j <= p; ++j) e *= 0.5 * z / j;
  return e;
}

// Interpolation error admitted along each axis of each cluster: at 8e-7 the whole field was
// within 2.5e-7 of its norm (four axes, but the worst case sits at the boxes' corners).
constexpr double kTruncation = 8e-7;

// Nodes for a mixed phase of z radians and a relative change eta of 1/r across the box; 0: too
// many.
int nodes_for(double z, double eta) {
  for (int p = 1; p <= 16; ++p)
    if (truncation(z, p) <= kTruncation && 2.0 * pow(0.5 * eta, p) <= kTruncation) return p;
  return 0;
}

}  // namespace

ExpandChoice expand_choose(const BoxStats &src, const BoxStats &tgt, int N, int M, int least_s,
                           int least_t, double k, double direct_seconds, double launches,
                           int sm_count) {
  ExpandChoice best;
  double gap2 = 0.0, e[3];
  for (int d = 0; d < 3; ++d) {
    const double g = std::max(0.0, std::max(src.lo[d] - tgt.hi[d], tgt.lo[d] - src.hi[d]));
    gap2 += g * g;
  }
  const double gap = sqrt(gap2);
  if (!(gap > 0.0)) return best;
  for (int d = 0; d < 3; ++d) {
    const double span = std::max(fabs(tgt.hi[d] - src.lo[d]), fabs(src.hi[d] - tgt.lo[d]));
    e[d] = std::min(1.0, span / gap);  // largest direction component of any pair
  }
  double best_s = direct_seconds;
  for (int ls = least_s; ls < kBoxLevels; ++ls) {
    if (ls > least_s && (256 << (ls - 1)) >= N) break;
    for (int lt = least_t; lt < kBoxLevels; ++lt) {
      if (lt > least_t && (256 << (lt - 1)) >= M) break;
      const double hs = src.h[ls], ht = tgt.h[lt], rel = (hs + ht) / gap;
      if (!(rel < 0.03)) continue;  // 1/r is taken to (c / r^2)^1: 3/8 rel^4 < 3e-7 left out
      // the axis along which both sets' clusters are flat
      int f = 0;
      for (int d = 1; d < 3; ++d)
        if (src.hd[ls][d] + tgt.hd[lt][d] < src.hd[ls][f] + tgt.hd[lt][f]) f = d;
      if (!(k * src.hd[ls][f] * ht / gap < 1e-7 && k * tgt.hd[lt][f] * hs / gap < 1e-7)) continue;
      // FP32 rounding of the curvature term, (hs + ht)^2 / 2r, and its truncated series
      const double c = (hs + ht) * (hs + ht) / gap;
      if (!(k * c * ldexp(1.0, -23) < 2e-6 && k * c * pow(rel, 4) / 16.0 < 1e-7)) continue;
      ExpandChoice ch;
      ch.ls = ls;
      ch.lt = lt;
      ch.ax = f == 0 ? 1 : 0;
      ch.ay = f == 2 ? 1 : 2;
      auto nodes = [&](int a, int b) {
        // along axis a the mixed phase is bilinear, k s_a t_a / r, plus what the direction
        // mixes in from axis b and the cubic terms
        const double exy = std::min(0.5, e[a] * e[b]), slope = 1.5 * (e[a] + rel) / (gap * gap);
        const double zs = k * src.hd[ls][a] * ((tgt.hd[lt][a] + exy * tgt.hd[lt][b]) / gap +
                                               slope * ht * (hs + ht));
        const double zt = k * tgt.hd[lt][a] * ((src.hd[ls][a] + exy * src.hd[ls][b]) / gap +
                                               slope * hs * (hs + ht));
        const double eta = std::max(src.hd[ls][a], tgt.hd[lt][a]) * (e[a] + rel) / gap;
        return nodes_for(std::max(zs, zt), eta);
      };
      ch.px = nodes(ch.ax, ch.ay);
      ch.py = nodes(ch.ay, ch.ax);
      if (!ch.px || !ch.py || ch.px * ch.py > kExpandNodes) continue;
      const double nS = box_count(N, ls), nT = box_count(M, lt);
      // SM clocks per unit of work, measured (kernel_expand.cu)
      const double clocks = kMomentClocks * (double)N * ceil(nT / 64) * 64 +
                            kTargetClocks * ceil((double)M / 128) * 128 * ceil(nS / 32) * 32 +
                            kNodePairClocks * nS * nT * 128.0 * ch.px * ch.py;
      const double seconds = launches + clocks / (sm_count * 1.9e9);
      if (seconds < best_s) {
        best_s = seconds;
        best = ch;
        best.use = true;
        best.seconds = seconds;
      }
    }
  }
  return best;
}

ExpandProblem expand_describe(holo_plan_s *p, const ExpandChoice &ch, double sk, double2 *y,
                              double share, ExpandScratch &tmp) {
  const Variant V = split_variant(p->variant);
  ExpandProblem P{};
  P.geo_s = p->geo_s;
  P.geo_t = p->geo_t;
  P.tiles_s = p->tiles_s;
  P.tiles_t = p->tiles_t;
  P.box_s = p->boxes_s + 6 * box_offset(p->N, ch.ls);
  P.box_t = p->boxes_t + 6 * box_offset(p->M, ch.lt);
  P.order_t = p->order_t;
  P.y = y;
  P.N = p->N;
  P.M = p->M;
  P.cs = V.cs;
  P.tt = V.tt();
  P.cs_log2 = 8 + box_level(P.cs);
  P.tt_log2 = 8 + box_level(P.tt);
  P.ns = 256 << ch.ls;
  P.nt = 256 << ch.lt;
  P.nS = box_count(P.N, ch.ls);
  P.nT = box_count(P.M, ch.lt);
  P.px = ch.px;
  P.py = ch.py;
  P.ax = ch.ax;
  P.ay = ch.ay;
  P.sk = sk;
  P.kap = (float)(0.5 * sk);
  // target clusters per launch: at most 1 GiB of frames, moments and coefficients
  const int groups_s = (P.nS + 31) / 32;
  const size_t row = (size_t)P.nS * (80 + 4 * 1024) + (size_t)groups_s * 65536;
  const size_t most = std::max<size_t>(1, ((size_t)1 << 30) / row);
  P.slab = most >= (size_t)P.nT ? P.nT : most >= 64 ? (int)(most / 64 * 64) : (int)most;
  // enough moments blocks for three waves of two per SM, enough target blocks for two of one
  const int sms = std::max(1, (int)(share * p->h->sm_count));
  const int mom = P.nS * ((P.slab + 63) / 64);
  P.ksplit = std::max(1, std::min({(6 * sms + mom - 1) / mom, P.ns / 64, 8}));
  const int blocks = (int)(((long long)P.slab * P.nt + 127) / 128);
  const int tgt = std::min(blocks, (P.M + 127) / 128);
  P.ssplit = std::max(1, std::min((2 * sms + tgt - 1) / tgt, groups_s));
  const size_t pairs = (size_t)P.slab * P.nS;
  P.apf_s = tmp.take<float2>(p->n_pad);
  P.frames = tmp.take<float>(12 * pairs);
  P.basis = tmp.take<float>(8 * pairs);
  P.half_s = tmp.take<float>(4 * (size_t)P.nS);
  P.half_t = tmp.take<float>(4 * (size_t)P.nT);
  P.shift_s = tmp.take<float>(8 * (size_t)((P.N + P.cs - 1) / P.cs));
  P.shift_t = tmp.take<float>(8 * (size_t)((P.M + P.tt - 1) / P.tt));
  P.cheb = tmp.take<float>(2 * (16 * 16 + 16));
  P.moments = tmp.take<float2>((size_t)P.ksplit * pairs * kExpandNodes);
  P.coeffs = tmp.take<float>((size_t)P.slab * groups_s * 16384);
  P.partial = P.ssplit > 1 ? tmp.take<double2>((size_t)P.ssplit * P.M) : nullptr;
  return P;
}

int expand_execute(holo_plan_s *p, const ExpandChoice &ch, double sk, const double *amp,
                   const double *phase, double2 *y, cudaStream_t s) {
  ExpandScratch size;
  expand_describe(p, ch, sk, y, 1.0, size);
  struct Buffer {
    void *p;
    cudaStream_t s;
    ~Buffer() { pool_free(p, s); }
  } buf{pool_alloc(p->h, size.bytes, s), s};
  if (!buf.p) return fail(HOLO_ERR_ALLOC, "expansion scratch of %zu bytes", size.bytes);
  ExpandScratch tmp;
  tmp.base = static_cast<unsigned char *>(buf.p);
  ExpandProblem P = expand_describe(p, ch, sk, y, 1.0, tmp);
  HOLO_TRY(launch_gather_apf(amp, phase, p->order_s, p->N, p->n_pad, const_cast<float2 *>(P.apf_s), s));
  HOLO_TRY(profile_mark(p->h, s, true));
  for (P.t0 = 0; P.t0 < P.nT; P.t0 += P.slab) {
    P.nTs = std::min(P.slab, P.nT - P.t0);
    HOLO_TRY(launch_expand(P, p->h->dev_err, s));
  }
  if (P.ssplit > 1) HOLO_TRY(launch_reduce(P.partial, P.ssplit, P.M, P.order_t, y, s));
  return profile_mark(p->h, s, false);
}

}  // namespace holo
