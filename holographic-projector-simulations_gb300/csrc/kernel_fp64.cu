// kernel_fp64.cu -- plain FP64 Huygens superposition (HOLO_FP64).
//
// Term for term the reference's FP64 path: phasor_displacement<dir>
// (cuda/superposition.cu:35-51) with norm3d_host (cuda/kernel.cu:95-99) and
// from_polar (cuda/kernel.cu:158-166).  Every product, sum, square root and
// quotient is rounded separately (explicit __d*_rn intrinsics, no FMA
// contraction), so each term equals the CPU oracle's bit for bit up to the
// last-ulp difference of sin/cos; only the order of the additions differs.
//
// Organisation (replacing per_block + cublasZgemv row sums,
// cuda/superposition.cu:59-154, cuda/kernel.cu:179-195): persistent CTAs over
// (target tile, source split) items; source tiles of CS points are staged in
// shared memory by TMA bulk copies (double-buffered, mbarrier-tracked); each
// thread owns R targets in registers; splits of the source range are reduced
// afterwards in a fixed order (deterministic, no atomics).
#include <type_traits>

#include "internal.cuh"
#include "ptx.cuh"

namespace holo {
namespace {

template <int THREADS, int R, int CS>
struct Fp64Smem {
  static constexpr size_t raw_pos = 0;                                     // double [2][CS*3]
  static constexpr size_t raw_ap = raw_pos + 2 * CS * 3 * sizeof(double);  // double2 [2][CS]
  static constexpr size_t bar = raw_ap + 2 * CS * sizeof(double2);         // uint64 [2]
  static constexpr size_t bytes = bar + 2 * sizeof(uint64_t);
};

// MINB: CTAs per SM the register allocation must leave room for (the FP64 pipe
// needs enough resident warps to hide the latency of its MUFU-seeded sqrt,
// division and sin/cos sequences).
template <int THREADS, int R, int CS, int MINB, bool CONST>
__global__ void __launch_bounds__(THREADS, MINB)
    k_fp64(const Fp64Problem P, int n_items, int *err) {
  extern __shared__ __align__(128) unsigned char smem[];
  using L = Fp64Smem<THREADS, R, CS>;
  constexpr int TT = THREADS * R;
  double *raw_pos = reinterpret_cast<double *>(smem + L::raw_pos);
  double2 *raw_ap = reinterpret_cast<double2 *>(smem + L::raw_ap);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L::bar);
  const int tid = threadIdx.x;
  if (tid == 0) {
    ptx::mbar_init(&bar[0], 1);
    ptx::mbar_init(&bar[1], 1);
    ptx::fence_barrier_init();
  }
  __syncthreads();
  uint32_t par[2] = {0u, 0u};

  auto issue = [&](int j, int buf) {
    ptx::mbar_arrive_expect_tx(&bar[buf], CS * (3 * sizeof(double) + sizeof(double2)));
    ptx::bulk_g2s(raw_pos + buf * CS * 3, P.pos_s + (size_t)j * CS * 3,
                  CS * 3 * sizeof(double), &bar[buf]);
    ptx::bulk_g2s(raw_ap + buf * CS, P.ap_s + (size_t)j * CS, CS * sizeof(double2),
                  &bar[buf]);
  };

  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int tt = item / P.splits;
    const int split = item % P.splits;
    const int sb = (int)(((long long)P.n_stiles * split) / P.splits);
    const int se = (int)(((long long)P.n_stiles * (split + 1)) / P.splits);

    double vx[R], vy[R], vz[R], re[R], im[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ti = tt * TT + tid + r * THREADS;
      const bool ok = ti < P.M;
      vx[r] = ok ? P.pos_t[3 * (size_t)ti] : 0.0;
      vy[r] = ok ? P.pos_t[3 * (size_t)ti + 1] : 0.0;
      vz[r] = ok ? P.pos_t[3 * (size_t)ti + 2] : 1.0;
      re[r] = 0.0;
      im[r] = 0.0;
    }
    if (tid == 0 && sb < se) issue(sb, 0);

    for (int j = sb; j < se; ++j) {
      const int buf = (j - sb) & 1;
      if (tid == 0 && j + 1 < se) issue(j + 1, buf ^ 1);
      const bool ok = ptx::mbar_wait_bounded(&bar[buf], par[buf], kWaitCycles);
      par[buf] ^= 1u;
      if (!__syncthreads_and(ok)) {
        if (tid == 0) atomicExch(err, kDevErrTimeout);
        return;
      }
      const double *sp = raw_pos + buf * CS * 3;
      const double2 *sa = raw_ap + buf * CS;
      const int count = min(CS, P.N - j * CS);
      for (int s = 0; s < count; ++s) {
        const double ux = sp[3 * s], uy = sp[3 * s + 1], uz = sp[3 * s + 2];
        const double2 a2 = sa[s];  // (phase, amp)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (CONST) {
            re[r] = __dadd_rn(re[r], 1.0);
          } else {
            const double a = __dsub_rn(vx[r], ux);
            const double b = __dsub_rn(vy[r], uy);
            const double c = __dsub_rn(vz[r], uz);
            const double ss = __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
            const double dist = __dsqrt_rn(ss);
            const double kr = __dmul_rn(dist, P.k);
            const double ph = P.sign > 0 ? __dadd_rn(a2.x, kr) : __dsub_rn(a2.x, kr);
            const double rr = __ddiv_rn(a2.y, dist);
            double sn, cs;
            sincos(ph, &sn, &cs);
            re[r] = __dadd_rn(re[r], __dmul_rn(rr, cs));
            im[r] = __dadd_rn(im[r], __dmul_rn(rr, sn));
          }
        }
      }
      __syncthreads();  // buffer `buf` is refilled two tiles later
    }

#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ti = tt * TT + tid + r * THREADS;
      if (ti < P.M) {
        const double2 v = make_double2(re[r], im[r]);
        if (P.splits == 1)
          P.y[ti] = v;
        else
          P.partial[(size_t)split * P.M + ti] = v;
      }
    }
  }
}

// ---- the same terms on the integer and FP32 pipes (fp64_fixed.cuh) ------------------------
// The FP64 pipe keeps 6.5 to 10 operations a pair instead of 56: the
// differences, their squares and sums (shared between a thread's four consecutive targets
// where they agree in a coordinate, as the rows of a lattice do: `share`), the product
// distance x k and the sum phase + that.  Bit for bit the other kernel's phases; amplitude /
// distance, sine and cosine are exact to 2^-55 or better and their products are summed as
// 64-bit integers, a tile of sources at a time, to 2^-54 of the target's own term of the tile's
// largest amplitude, whose distance sets the target's scale.  A pair out of the fixed-point
// ranges (a zero, infinite or NaN value, a distance four times under the one that set the
// scale, a phase beyond 2^43) takes the FP64 operations instead.
// Measured (GB300, 1000 sources -> 512^2 lattice targets): 4.35 ms against 30.0 ms (variant 0); the
// same with targets jittered, so that no coordinate is shared, 5.2 ms; with registers for 4 or
// 3 CTAs per SM instead of 5 4.6 ms, 2 targets a thread 4.9 ms, 8 4.6 ms.  Bound by the FP64
// pipe: 7.1 of its slots a pair at 0.92 of the rate a pure DFMA stream reaches (ncu: pipe 78 %
// active, issue slots 55 % for 319 instructions a pair).  One scale for a thread's four targets
// and one rounding for all sources took 4.28 ms and lost the bits that targets farther from a
// tile's brightest source than the first one need.
// One target a thread (variant 7) is for problems that would not fill the GPU: a whole call
// of 64 -> 64^2 0.10 ms against 0.24, of 256 -> 128^2 0.19 against 0.24, but of 1000 ->
// 128^2 0.44 against 0.37.
constexpr int kFixThreads = 128;
template <int CS>
struct FixSmem {
  static constexpr size_t trig = 0;                                        // TrigEntry [1024]
  static constexpr size_t turns = trig + fixed::kTrigEntries * sizeof(fixed::TrigEntry);
  static constexpr size_t pos = turns + fixed::kTurnEntries * sizeof(fixed::TurnWords);
  static constexpr size_t ap = pos + 2 * CS * 3 * sizeof(double);      // double2 [2][CS]
  static constexpr size_t amp = ap + 2 * CS * sizeof(double2);         // int64 [CS]
  static constexpr size_t bar = amp + CS * 8;                          // uint64 [3]
  static constexpr size_t bytes = bar + 3 * 8;
};
static_assert(sizeof(fixed::TrigEntry) == 32 && sizeof(fixed::TurnWords) == 16, "table layout");

template <int R, int CS, int MINB>
__global__ void __launch_bounds__(kFixThreads, MINB)
    k_fp64_fixed(const Fp64Problem P, int n_items, int *err) {
  extern __shared__ __align__(128) unsigned char smem[];
  using L = FixSmem<CS>;
  constexpr int TT = kFixThreads * R;
  fixed::TrigEntry *trig = reinterpret_cast<fixed::TrigEntry *>(smem + L::trig);
  fixed::TurnWords *turns = reinterpret_cast<fixed::TurnWords *>(smem + L::turns);
  double *raw_pos = reinterpret_cast<double *>(smem + L::pos);
  double2 *raw_ap = reinterpret_cast<double2 *>(smem + L::ap);
  long long *samp = reinterpret_cast<long long *>(smem + L::amp);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L::bar);
  static_assert(CS == 16 || CS == 64, "the amplitudes' reduction");
  __shared__ int s_exp[2];
  const int tid = threadIdx.x;
  constexpr uint32_t kTables = fixed::kTrigEntries * sizeof(fixed::TrigEntry),
                     kTurns = fixed::kTurnEntries * sizeof(fixed::TurnWords);
  if (tid == 0) {
    for (int b = 0; b < 3; ++b) ptx::mbar_init(&bar[b], 1);
    ptx::fence_barrier_init();
    ptx::mbar_arrive_expect_tx(&bar[2], kTables + kTurns);
    ptx::bulk_g2s(trig, P.trig, kTables, &bar[2]);
    ptx::bulk_g2s(turns, P.turns, kTurns, &bar[2]);
  }
  __syncthreads();
  const bool tables = ptx::mbar_wait_bounded(&bar[2], 0u, kWaitCycles);
  if (!__syncthreads_and(tables)) {
    if (tid == 0) atomicExch(err, kDevErrTimeout);
    return;
  }
  uint32_t par[2] = {0u, 0u};
  auto issue = [&](int j, int buf) {
    ptx::mbar_arrive_expect_tx(&bar[buf], CS * (3 * sizeof(double) + sizeof(double2)));
    ptx::bulk_g2s(raw_pos + buf * CS * 3, P.pos_s + (size_t)j * CS * 3, CS * 3 * sizeof(double),
                  &bar[buf]);
    ptx::bulk_g2s(raw_ap + buf * CS, P.ap_s + (size_t)j * CS, CS * sizeof(double2), &bar[buf]);
  };
  const double sk = P.sign > 0 ? P.k : -P.k;  // RN(phi - RN(r k)) = RN(phi + RN(r (-k)))

  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int tt = item / P.splits, split = item % P.splits;
    const int sb = (int)(((long long)P.n_stiles * split) / P.splits);
    const int se = (int)(((long long)P.n_stiles * (split + 1)) / P.splits);
    const int t0 = tt * TT + tid * R;
    double vx[R], vy[R], vz[R], re[R], im[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ti = t0 + r;
      const bool ok = ti < P.M;
      vx[r] = ok ? P.pos_t[3 * (size_t)ti] : (r ? vx[0] : 0.0);
      vy[r] = ok ? P.pos_t[3 * (size_t)ti + 1] : (r ? vy[0] : 0.0);
      vz[r] = ok ? P.pos_t[3 * (size_t)ti + 2] : (r ? vz[0] : 1.0);
      re[r] = 0.0;
      im[r] = 0.0;
    }
    // coordinates that every thread's targets share (bit for bit)
    bool same[3] = {true, true, true};
#pragma unroll
    for (int r = 1; r < R; ++r) {
      same[0] = same[0] && __double_as_longlong(vx[r]) == __double_as_longlong(vx[0]);
      same[1] = same[1] && __double_as_longlong(vy[r]) == __double_as_longlong(vy[0]);
      same[2] = same[2] && __double_as_longlong(vz[r]) == __double_as_longlong(vz[0]);
    }
    bool share[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) share[d] = __syncthreads_and(same[d]);
    if (tid == 0 && sb < se) issue(sb, 0);

    for (int j = sb; j < se; ++j) {
      const int buf = (j - sb) & 1;
      if (tid == 0 && j + 1 < se) issue(j + 1, buf ^ 1);
      const bool ok_wait = ptx::mbar_wait_bounded(&bar[buf], par[buf], kWaitCycles);
      par[buf] ^= 1u;
      if (!__syncthreads_and(ok_wait)) {
        if (tid == 0) atomicExch(err, kDevErrTimeout);
        return;
      }
      const double *sp = raw_pos + buf * CS * 3;
      const double2 *sa = raw_ap + buf * CS;
      const int count = min(CS, P.N - j * CS);
      // amplitudes of the tile in units of its largest one's exponent: amp = A 2^(ea - 1084)
      if (tid < 64) {
        const long long a = tid < count ? __double_as_longlong(sa[tid].y) : 0;
        const int e = (int)(a >> 52) & 0x7ff;
        // 4095 marks what has no place here: a subnormal, an infinity, a NaN
        const bool bad = e == 0x7ff || (e == 0 && (a & 0x7fffffffffffffffLL) != 0);
        const int top = __reduce_max_sync(0xffffffffu, (bad ? 4095 : e) << 6 | tid);
        if ((tid & 31) == 0) s_exp[tid >> 5] = top;
      }
      __syncthreads();
      const int key = max(s_exp[0], s_exp[1]), top = min(key & 63, count - 1);
      const int ea = key >= 64 ? key >> 6 : 1023;  // all zero: any scale
      if (tid < CS) {
        const long long a = tid < count ? __double_as_longlong(sa[tid].y) : 0;
        const int e = (int)(a >> 52) & 0x7ff, down = ea - e;
        const long long m = ((a & 0xfffffffffffffLL) | (1LL << 52)) << 9;
        const long long f = e == 0 || down > 62 ? 0 : m >> down;
        samp[tid] = a < 0 ? -f : f;
      }
      __syncthreads();
      // exponent field of the unit of sums scaled by 2^-q
      auto unit_exp = [&](int q) { return ea - 1078 - q + 1023; };
      // the sources of this tile; mask: coordinates that the targets of each thread share
      auto sum_tile = [&](auto mask) {
        constexpr bool SX = decltype(mask)::value & 1, SY = decltype(mask)::value & 2,
                       SZ = decltype(mask)::value & 4;
        // the scale of each target: a quarter of its distance from the tile's brightest source,
        // where that is well inside the exponent range; kNoScale sends every pair of the target
        // to the FP64 operations
        constexpr int kNoScale = -100000;
        int qref[R];
        long long fr[R], fi[R];
        uint32_t made = 0;  // products formed, a byte for each target: each rounds down
        {
          const double ux = sp[3 * top], uy = sp[3 * top + 1], uz = sp[3 * top + 2];
          double both = 0.0;  // what the targets share
          if (SX) { const double d = vx[0] - ux; both = d * d; }
          if (SY) { const double d = vy[0] - uy; both = fma(d, d, both); }
          if (SZ) { const double d = vz[0] - uz; both = fma(d, d, both); }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            double ss = both;
            if (!SX) { const double d = vx[r] - ux; ss = fma(d, d, ss); }
            if (!SY) { const double d = vy[r] - uy; ss = fma(d, d, ss); }
            if (!SZ) { const double d = vz[r] - uz; ss = fma(d, d, ss); }
            const uint32_t hi = (uint32_t)__double2hiint(ss);
            const int q = (((int)(hi >> 20) - 1023) >> 1) - 2, es = unit_exp(q);
            const bool in = hi - (200u << 20) < (1600u << 20) && ea > 200 && ea < 2047;
            qref[r] = in && es > 0 && es < 2046 ? q : kNoScale;
            fr[r] = fi[r] = 0;
          }
        }
        for (int s = 0; s < count; ++s) {
          const double ux = sp[3 * s], uy = sp[3 * s + 1], uz = sp[3 * s + 2];
          const double phi = sa[s].x;
          const long long am = samp[s];
          double xx = 0.0, yy = 0.0, zz = 0.0;
          if (SX) { const double d = __dsub_rn(vx[0], ux); xx = __dmul_rn(d, d); }
          if (SY) { const double d = __dsub_rn(vy[0], uy); yy = __dmul_rn(d, d); }
          if (SZ) { const double d = __dsub_rn(vz[0], uz); zz = __dmul_rn(d, d); }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (!SX) { const double d = __dsub_rn(vx[r], ux); xx = __dmul_rn(d, d); }
            if (!SY) { const double d = __dsub_rn(vy[r], uy); yy = __dmul_rn(d, d); }
            if (!SZ) { const double d = __dsub_rn(vz[r], uz); zz = __dmul_rn(d, d); }
            const double ss = __dadd_rn(__dadd_rn(xx, yy), zz);
            const uint32_t hi = (uint32_t)__double2hiint(ss);
            const fixed::Root rt = fixed::root(hi, (uint32_t)__double2loint(ss),
                                               [](float x) { return ptx::rsqrt_approx(x); });
            const double dist = __hiloint2double((int)(rt.d >> 32) + ((rt.q + 1022) << 20), (int)rt.d);
            const double ph = __dadd_rn(phi, __dmul_rn(dist, sk));
            const uint32_t hp = (uint32_t)__double2hiint(ph);
            const uint32_t te = ((hp >> 20) & 0x7ffu) - (uint32_t)(1023 + fixed::kTurnLow);
            const uint32_t down = (uint32_t)(rt.q - qref[r]);
            const bool fast = hi - (200u << 20) < (1600u << 20) && down <= 40u &&
                              te < (uint32_t)fixed::kTurnEntries;
            if (fast) {
              const uint4 k = *reinterpret_cast<const uint4 *>(&turns[te]);
              const uint64_t t = fixed::turns(hp, (uint32_t)__double2loint(ph), k.x, k.y, k.z, k.w);
              const uint32_t index = fixed::trig_index(t);
              const fixed::TrigEntry &E = trig[index & (fixed::kTrigEntries - 1)];
              int64_t c, sn;
              fixed::cos_sin(t, index, E, &c, &sn);
              const int64_t w = fixed::mulhi64(am, fixed::reciprocal(rt)) >> (down + 2);
              fr[r] += fixed::mulhi64(w, c);
              fi[r] += fixed::mulhi64(w, sn);
              made += w != 0 ? 1u << (8 * r) : 0u;
            } else {
              const double d = __dsqrt_rn(ss);
              const double kr = __dmul_rn(d, P.k);
              const double p = P.sign > 0 ? __dadd_rn(phi, kr) : __dsub_rn(phi, kr);
              const double w = __ddiv_rn(sa[s].y, d);
              double sn, cs;
              sincos(p, &sn, &cs);
              re[r] = __dadd_rn(re[r], __dmul_rn(w, cs));
              im[r] = __dadd_rn(im[r], __dmul_rn(w, sn));
            }
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (qref[r] == kNoScale) continue;
          const double unit = __hiloint2double(unit_exp(qref[r]) << 20, 0);
          const long long up = (long long)((made >> (8 * r) & 255u) + 1u) >> 1;
          re[r] = fma((double)(fr[r] + up), unit, re[r]);
          im[r] = fma((double)(fi[r] + up), unit, im[r]);
        }
      };
      if (R == 1) sum_tile(std::integral_constant<int, 7>{});
      else if (share[2] && share[0]) sum_tile(std::integral_constant<int, 5>{});
      else if (share[2] && share[1]) sum_tile(std::integral_constant<int, 6>{});
      else if (share[2]) sum_tile(std::integral_constant<int, 4>{});
      else sum_tile(std::integral_constant<int, 0>{});
      __syncthreads();  // buffer `buf` is refilled two tiles later, the amplitudes at once
    }

#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ti = t0 + r;
      if (ti < P.M) {
        const double2 v = make_double2(re[r], im[r]);
        if (P.splits == 1)
          P.y[ti] = v;
        else
          P.partial[(size_t)split * P.M + ti] = v;
      }
    }
  }
}

constexpr Variant kVariants[] = {
    {128, 4, 256},  // 0
    {256, 2, 256},  // 1
    {128, 2, 256},  // 2
    {64, 4, 256},   // 3
    {128, 2, 256},  // 4: registers for 8 CTAs per SM
    {128, 1, 256},  // 5: registers for 12 CTAs per SM
    {kFixThreads, 4, 64},  // 6: the fixed-point kernel
    {kFixThreads, 1, 16},  // 7: the same, one target per thread, 16 sources a tile
};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

template <int THREADS, int R, int CS, int MINB>
int launch_variant(const Fp64Problem &p, int grid, bool cst, int *err, cudaStream_t s) {
  using L = Fp64Smem<THREADS, R, CS>;
  const int n_items = p.n_ttiles * p.splits;
  if (n_items <= 0) return HOLO_OK;
  if (cst) {
    auto kern = k_fp64<THREADS, R, CS, MINB, true>;
    HOLO_TRY((kernel_setup<k_fp64<THREADS, R, CS, MINB, true>>(THREADS, (int)L::bytes, nullptr)));
    kern<<<grid, THREADS, L::bytes, s>>>(p, n_items, err); note_launches(1);
  } else {
    auto kern = k_fp64<THREADS, R, CS, MINB, false>;
    HOLO_TRY((kernel_setup<k_fp64<THREADS, R, CS, MINB, false>>(THREADS, (int)L::bytes, nullptr)));
    kern<<<grid, THREADS, L::bytes, s>>>(p, n_items, err); note_launches(1);
  }
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

template <int THREADS, int R, int CS, int MINB>
int occupancy_variant(int *out) {
  using L = Fp64Smem<THREADS, R, CS>;
  return kernel_setup<k_fp64<THREADS, R, CS, MINB, false>>(THREADS, (int)L::bytes, out);
}

template <int R, int CS, int MINB>
int launch_fixed(const Fp64Problem &p, int grid, bool cst, int *err, cudaStream_t s) {
  if (cst)  // every term 1: nothing to compute (same tiles, the plain kernel)
    return launch_variant<kFixThreads, R, CS, 1>(p, grid, true, err, s);
  const int n_items = p.n_ttiles * p.splits;
  if (n_items <= 0) return HOLO_OK;
  HOLO_TRY((kernel_setup<k_fp64_fixed<R, CS, MINB>>(kFixThreads, (int)FixSmem<CS>::bytes, nullptr)));
  k_fp64_fixed<R, CS, MINB><<<grid, kFixThreads, FixSmem<CS>::bytes, s>>>(p, n_items, err); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

}  // namespace

int fp64_variant_count() { return kNumVariants; }
Variant fp64_variant(int i) { return kVariants[i]; }

#define HOLO_FP64_DISPATCH(V, CALL)                                        \
  switch (V) {                                                             \
    case 0: return CALL(128, 4, 256, 1);                                   \
    case 1: return CALL(256, 2, 256, 1);                                   \
    case 2: return CALL(128, 2, 256, 1);                                   \
    case 3: return CALL(64, 4, 256, 1);                                    \
    case 4: return CALL(128, 2, 256, 8);                                   \
    case 5: return CALL(128, 1, 256, 12);                                  \
    default: return fail(HOLO_ERR_INVALID, "unknown fp64 variant %d", V);  \
  }

int launch_fp64(const Fp64Problem &p, int variant, int grid, bool const_phase, int *err,
                cudaStream_t s) {
  if (variant == 6) return launch_fixed<4, 64, 5>(p, grid, const_phase, err, s);
  if (variant == 7) return launch_fixed<1, 16, 5>(p, grid, const_phase, err, s);
#define CALL(T, R, C, B) launch_variant<T, R, C, B>(p, grid, const_phase, err, s)
  HOLO_FP64_DISPATCH(variant, CALL)
#undef CALL
}

int fp64_occupancy(int variant, int *ctas_per_sm) {
  if (variant == 6)
    return kernel_setup<k_fp64_fixed<4, 64, 5>>(kFixThreads, (int)FixSmem<64>::bytes, ctas_per_sm);
  if (variant == 7)
    return kernel_setup<k_fp64_fixed<1, 16, 5>>(kFixThreads, (int)FixSmem<16>::bytes, ctas_per_sm);
#define CALL(T, R, C, B) occupancy_variant<T, R, C, B>(ctas_per_sm)
  HOLO_FP64_DISPATCH(variant, CALL)
#undef CALL
}

}  // namespace holo
