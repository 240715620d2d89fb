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

// Shares of a cluster's sources, and of the source clusters, that give every SM work: three
// waves of two moments blocks, two target items.
static int moment_shares(int nS, int nT, int ns, int sms) {
  const int blocks = nS * ((nT + 63) / 64);
  return std::max(1, std::min({(6 * sms + blocks - 1) / blocks, ns / 64, 32}));
}
static int target_shares(int nS, int M, int sms) {
  const int blocks = (M + 127) / 128;
  return std::max(1, std::min((2 * sms + blocks - 1) / blocks, (nS + 31) / 32));
}

// SM clocks that the three kernels take (GB300, the constants of expand_plan.h): whole waves of
// moments blocks, of target items and of translation blocks.
static double expand_clocks(const ExpandChoice &ch, int N, int M, int sms) {
  const int ns = 256 << ch.ls, nS = box_count(N, ch.ls), nT = box_count(M, ch.lt);
  const int ksplit = moment_shares(nS, nT, ns, sms), ssplit = target_shares(nS, M, sms);
  const double blocks = (double)nS * ((nT + 63) / 64) * ksplit;
  const double stages = ceil(ceil(std::min(ns, N) / 64.0) / ksplit);
  const double moments = kMomentStage * stages * (blocks <= sms ? 1.0 : 2.0 * ceil(blocks / (2.0 * sms)));
  const double items = ceil((M + 127) / 128 * (double)ssplit / sms);
  const double targets = items * (kTargetItem + kTargetGroup * ceil((nS + 31) / 32 / (double)ssplit));
  const double translate = std::max(kNodePairClocks * 128.0 * ch.px * ch.py * nS * nT / sms,
                                    kTranslateLatency * ch.px * ch.py);
  return moments + targets + translate;
}

int expand_quads(int px, int py, uint32_t *quads) {
  const int qx = px / 4, rx = px % 4, qy = py / 4;
  int n = 0;
  auto add = [&](uint32_t which, uint32_t scalar, uint32_t quad) {
    if (quads && n < 32) quads[n] = which << 16 | scalar << 8 | quad;
    ++n;
  };
  for (int a = 0; a < px; ++a)
    for (int q = 0; q < qy; ++q) add(0, a, q);
  for (int b = 4 * qy; b < py; ++b) {
    for (int q = 0; q < qx; ++q) add(1, b, q);
  }
  if (rx)
    for (int b = 4 * qy; b < py; ++b) add(1, b, qx);
  return n;
}

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
      if (!(k * c * ldexp(1.0, -23) < 3e-6 && k * c * pow(rel, 4) / 16.0 < 1e-7)) continue;
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
      if (expand_quads(ch.px, ch.py, nullptr) > 32) {
        std::swap(ch.px, ch.py);
        std::swap(ch.ax, ch.ay);
        if (expand_quads(ch.px, ch.py, nullptr) > 32) continue;
      }
      const double seconds = launches + expand_clocks(ch, N, M, sm_count) / 1.9e9;
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
                              double share, size_t slab_bytes, ExpandScratch &keep,
                              ExpandScratch &tmp) {
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
  P.ns = 256 << ch.ls;
  P.nt = 256 << ch.lt;
  P.nS = box_count(P.N, ch.ls);
  P.nT = box_count(P.M, ch.lt);
  P.px = ch.px;
  P.py = ch.py;
  P.ax = ch.ax;
  P.ay = ch.ay;
  P.n_quads = expand_quads(P.px, P.py, P.quads);
  P.sk = sk;
  P.kap = (float)(0.5 * sk);
  // target clusters per launch: at most slab_bytes of frames, moments and coefficients
  const int groups_s = (P.nS + 31) / 32;
  const size_t row = (size_t)P.nS * (80 + 4 * 1024) + (size_t)groups_s * 65536;
  const size_t most = std::max<size_t>(1, slab_bytes / row);
  P.slab = most >= (size_t)P.nT ? P.nT : most >= 64 ? (int)(most / 64 * 64) : (int)most;
  const int sms = std::max(1, (int)(share * p->h->sm_count));
  P.ksplit = moment_shares(P.nS, P.slab, P.ns, sms);
  P.ssplit = target_shares(P.nS, std::min(P.slab * P.nt, P.M), sms);
  const size_t pairs = (size_t)P.slab * P.nS;
  P.apf_s = keep.take<float2>(p->n_pad);
  P.frames = tmp.take<float>(12 * pairs);
  P.basis = tmp.take<float>(8 * pairs);
  P.half_s = tmp.take<float>(4 * (size_t)P.nS);
  P.half_t = tmp.take<float>(4 * (size_t)P.nT);
  P.shift_s = tmp.take<float>(8 * (size_t)box_count(P.N, 0));
  P.shift_t = tmp.take<float>(8 * (size_t)box_count(P.M, 0));
  P.cheb = tmp.take<float>(2 * (16 * 16 + 16));
  P.tops = tmp.take<uint32_t>((size_t)(P.N + 4095) / 4096 + 1);
  P.moments = tmp.take<float2>((size_t)P.ksplit * pairs * kExpandNodes);
  P.coeffs = tmp.take<float>((size_t)P.slab * groups_s * 16384);
  P.partial = P.ssplit > 1 ? keep.take<double2>((size_t)P.ssplit * P.M) : nullptr;
  return P;
}

int expand_execute(holo_plan_s *p, const ExpandChoice &ch, double sk, const double *amp,
                   const double *phase, double2 *y, cudaStream_t s) {
  struct Buffer {
    void *p;
    cudaStream_t s;
    ~Buffer() { pool_free(p, s); }
  } buf{nullptr, s};
  // smaller slabs where the device has no room for those of kSlabBytes
  size_t slab = kSlabBytes, bytes = 0;
  for (; !buf.p && slab >= kLeastSlabBytes; slab /= 8) {
    ExpandScratch size;
    expand_describe(p, ch, sk, y, 1.0, slab, size, size);
    bytes = size.bytes;
    buf.p = pool_alloc(p->h, bytes, s);
    if (buf.p) break;
  }
  if (!buf.p) return fail(HOLO_ERR_ALLOC, "expansion scratch of %zu bytes", bytes);
  ExpandScratch tmp;
  tmp.base = static_cast<unsigned char *>(buf.p);
  ExpandProblem P = expand_describe(p, ch, sk, y, 1.0, slab, tmp, tmp);
  HOLO_TRY(launch_gather_apf(amp, phase, p->order_s, p->N, p->n_pad, const_cast<float2 *>(P.apf_s), s));
  HOLO_TRY(profile_mark(p->h, s, true));
  for (P.t0 = 0; P.t0 < P.nT; P.t0 += P.slab) {
    P.nTs = std::min(P.slab, P.nT - P.t0);
    HOLO_TRY(launch_expand(P, p->h->sm_count, p->h->dev_err, s));
  }
  if (P.ssplit > 1) HOLO_TRY(launch_reduce(P.partial, P.ssplit, P.M, P.order_t, y, s));
  return profile_mark(p->h, s, false);
}

}  // namespace holo
