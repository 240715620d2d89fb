// tiler.cu -- spatial tiling of a point set on the device.
//
// The split-precision kernels need every tile of consecutive points to be
// spatially compact: their FP32 arithmetic is relative to the tile centre, and
// the planner's error bound grows with the square of the widest tile.  The
// reference keeps points in file order (its square-tile reorder,
// cuda/reorder.cu:1-92, is never called).  Two tilings:
//   Hilbert: one stable counting sort by the Hilbert index of a 64 x 64 cell grid
//     over the two widest axes -- cheap, and exact squares on power-of-two grids,
//     but runs of the curve can be L-shaped or long for other point counts;
//   packed: super tiles of 8192 by sort-tile-recursive strips (stable counting
//     sorts by the quantised widest axis, then the second axis, then the strip),
//     each bisected in shared memory down to tiles of 256 by splitting off
//     power-of-two prefixes, so every tile of 256, 512 or 1024 points is one
//     bisection segment of nearly square extent -- about twice the planning
//     time, used where the Hilbert tiles' error bound rules out the fastest kernel.
// All sorts are stable and ties keep input order: each order is deterministic
// and does not depend on the tile size.
#include <algorithm>

#include "internal.cuh"

namespace holo {
namespace {

// Doubles as 64-bit integers of the same order (NaN excluded): minima and maxima run on the
// integer pipe, where FP64 compares would take a pair of the few FP64 lanes each.
__device__ __forceinline__ long long ordered64(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double from_ordered64(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}
constexpr long long kOrderedMax = 0x7fefffffffffffffLL;   // ordered64(DBL_MAX)
constexpr long long kOrderedMin = ~0x7fefffffffffffffLL;  // ordered64(-DBL_MAX)

struct Box64 {
  long long lo[3], hi[3];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = kOrderedMax;
      hi[d] = kOrderedMin;
    }
  }
  __device__ __forceinline__ void add(double x, double y, double z) {
    const double p[3] = {x, y, z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const long long k = ordered64(p[d]);
      if ((__double_as_longlong(p[d]) & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL) {  // not NaN
        lo[d] = min(lo[d], k);
        hi[d] = max(hi[d], k);
      }
    }
  }
  __device__ __forceinline__ void warp_reduce() {
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        lo[d] = min(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = max(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
  }
};

// One or two point sets that a launch of the Hilbert tiling handles (blockIdx.y).
struct SortSet {
  const double *pos;
  int n, parts;         // points; blocks of the box reduction
  long long *box;       // [parts][6] ordered keys
  uint16_t *keys;
  uint32_t *hist;       // [blocks of kSortBlock][kCells]
  uint32_t *totals;     // [kCells]
  int32_t *order;
};
struct SortSets {
  SortSet s[2];
};

// Box of 8 points per thread and block, and zeros for the histogram of the next kernel.
__global__ void __launch_bounds__(256) k_box_parts(const SortSets sets) {
  const SortSet &S = sets.s[blockIdx.y];
  if ((int)blockIdx.x >= S.parts) return;
  __shared__ Box64 w[8];
  const int step = S.parts * 256, at = blockIdx.x * 256 + threadIdx.x;
  Box64 b;
  b.clear();
  for (int i = at; i < S.n; i += step) {
    const double *p = S.pos + 3 * (size_t)i;
    b.add(p[0], p[1], p[2]);
  }
  const size_t cells = (size_t)((S.n + kSortBlock - 1) / kSortBlock) * (kCells / 4);
  if (S.hist)
    for (size_t c = at; c < cells; c += step)
      reinterpret_cast<uint4 *>(S.hist)[c] = make_uint4(0u, 0u, 0u, 0u);
  b.warp_reduce();
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x < 6) {
    const int d = threadIdx.x % 3;
    long long v = threadIdx.x < 3 ? w[0].lo[d] : w[0].hi[d];
    for (int j = 1; j < 8; ++j) v = threadIdx.x < 3 ? min(v, w[j].lo[d]) : max(v, w[j].hi[d]);
    S.box[6 * blockIdx.x + threadIdx.x] = v;
  }
}

// The whole box from the parts, by warps 0 .. 5 of a block, into shared memory (lo, hi).
__device__ __forceinline__ void reduce_box_parts(const long long *box, int parts, double *out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 6) {
    long long v = warp < 3 ? kOrderedMax : kOrderedMin;
    for (int b = lane; b < parts; b += 32)
      v = warp < 3 ? min(v, box[6 * b + warp]) : max(v, box[6 * b + warp]);
    for (int o = 16; o > 0; o >>= 1) {
      const long long x = __shfl_xor_sync(0xffffffffu, v, o);
      v = warp < 3 ? min(v, x) : max(v, x);
    }
    if (lane == 0) out[warp] = from_ordered64(v);
  }
}

__global__ void __launch_bounds__(256) k_bbox_final(const long long *__restrict__ box, int parts,
                                                    double *__restrict__ bbox) {
  reduce_box_parts(box, parts, bbox);
}

constexpr int kHilbertCells = 64;  // cells per axis of the Hilbert tiling (kCells in all)
static_assert(kHilbertCells * kHilbertCells == kCells, "Hilbert cells fill the sort's bins");

// Hilbert index of cell (x, y) on an n x n grid (n a power of two): the
// classic quadrant-rotation construction of the curve.
__device__ __forceinline__ uint32_t hilbert_xy2d(int n, int x, int y) {
  uint32_t d = 0;
  for (int s = n / 2; s > 0; s /= 2) {
    const int rx = (x & s) > 0;
    const int ry = (y & s) > 0;
    d += (uint32_t)s * (uint32_t)s * (uint32_t)((3 * rx) ^ ry);
    if (ry == 0) {
      if (rx == 1) {
        x = n - 1 - x;
        y = n - 1 - y;
      }
      const int t = x;
      x = y;
      y = t;
    }
  }
  return d;
}

// The two widest axes of a bounding box (lo[3], hi[3]), widest first.
__device__ __forceinline__ void widest_axes(const double *bbox, int *a0, int *a1) {
  double ext[3];
  for (int d = 0; d < 3; ++d) ext[d] = bbox[3 + d] - bbox[d];
  int x = 0, y = 1, z = 2;  // sort axes by extent, descending
  if (ext[y] > ext[x]) { int t = x; x = y; y = t; }
  if (ext[z] > ext[y]) { int t = y; y = z; z = t; }
  if (ext[y] > ext[x]) { int t = x; x = y; y = t; }
  *a0 = x;
  *a1 = y;
}

// Hilbert cell of every point and the histogram of each kSortBlock points.  Bound by the FP64
// pipe (two subtractions, products and conversions a point), so the box, the cell axes and
// the scales are worked out once per block of 1024 points, not per thread (18.8 us for
// 262,144 points and 5.1 us for 16,384 before, 12 us for both here).
__global__ void __launch_bounds__(256) k_cell_keys(const SortSets sets) {
  const SortSet &S = sets.s[blockIdx.y];
  const int i0 = blockIdx.x * 1024;
  if (i0 >= S.n) return;
  __shared__ double box[6], scale[2], low[2];
  __shared__ int axis[2];
  reduce_box_parts(S.box, S.parts, box);
  __syncthreads();
  if (threadIdx.x == 0) {
    widest_axes(box, &axis[0], &axis[1]);
    for (int a = 0; a < 2; ++a) {
      const double ext = box[3 + axis[a]] - box[axis[a]];
      scale[a] = ext > 0 ? kHilbertCells / ext : 0.0;
      low[a] = box[axis[a]];
    }
  }
  __syncthreads();
  const int a0 = axis[0], a1 = axis[1], lane = threadIdx.x & 31;
  const double l0 = low[0], l1 = low[1], s0 = scale[0], s1 = scale[1];
  uint32_t *hist = S.hist + (size_t)(i0 / kSortBlock) * kCells;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = i0 + 256 * k + threadIdx.x;
    int key = kCells;  // sentinel past the end
    if (i < S.n) {
      const double *p = S.pos + 3 * (size_t)i;
      int cx = (int)((p[a0] - l0) * s0);
      int cy = (int)((p[a1] - l1) * s1);
      cx = min(max(cx, 0), kHilbertCells - 1);
      cy = min(max(cy, 0), kHilbertCells - 1);
      key = (int)hilbert_xy2d(kHilbertCells, cx, cy);
      S.keys[i] = (uint16_t)key;
    }
    // runs of one cell (a lattice's rows) in one addition
    const uint32_t peers = __match_any_sync(0xffffffffu, key);
    if (i < S.n && (__ffs(peers) - 1) == lane) atomicAdd(&hist[key], __popc(peers));
  }
}

// Points per strip: about sqrt(#super tiles / aspect) strips make the super tiles
// square; the count is a multiple of the super tile so strips end on super-tile
// boundaries.  Every thread computes the same value from the box.
__device__ __forceinline__ long long strip_points(const double *bbox, int n) {
  int a0, a1;
  widest_axes(bbox, &a0, &a1);
  const double e0 = bbox[3 + a0] - bbox[a0], e1 = bbox[3 + a1] - bbox[a1];
  const long long nsup = (n + kSuperTile - 1) / kSuperTile;
  const double aspect = e0 > 0.0 ? fmax(e1 / e0, 1e-9) : 1.0;
  long long strips = llround(sqrt((double)nsup / aspect));
  strips = max(1LL, min(strips, min(nsup, (long long)kCells)));
  return (nsup + strips - 1) / strips * kSuperTile;
}

// Key of every point: its coordinate along the widest (axis 0) or the second widest
// (axis 1) axis of the box, quantised to kCells bins.
__global__ void __launch_bounds__(256) k_axis_keys(const double *__restrict__ pos, int n,
                                                   const double *__restrict__ bbox, int which,
                                                   uint16_t *__restrict__ keys) {
  int a0, a1;
  widest_axes(bbox, &a0, &a1);
  const int a = which ? a1 : a0;
  const double ext = bbox[3 + a] - bbox[a];
  const double sc = ext > 0.0 ? kCells / ext : 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int c = (int)((pos[3 * (size_t)i + a] - bbox[a]) * sc);
    keys[i] = (uint16_t)min(max(c, 0), kCells - 1);
  }
}

// strip[order_x[r]] = r / (points per strip): the strip of each point by its rank
// along the widest axis.
__global__ void __launch_bounds__(256) k_strip_keys(const int32_t *__restrict__ order_x, int n,
                                                    const double *__restrict__ bbox,
                                                    uint16_t *__restrict__ strip) {
  const long long per = strip_points(bbox, n);
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    strip[order_x[r]] = (uint16_t)(r / per);
}

// out[r] = src[perm[r]]
__global__ void __launch_bounds__(256) k_permute_keys(const uint16_t *__restrict__ src,
                                                      const int32_t *__restrict__ perm, int n,
                                                      uint16_t *__restrict__ out) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    out[r] = src[perm[r]];
}

// out[r] = a[b[r]]
__global__ void __launch_bounds__(256) k_compose(const int32_t *__restrict__ a,
                                                 const int32_t *__restrict__ b, int n,
                                                 int32_t *__restrict__ out) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    out[r] = a[b[r]];
}

__device__ __forceinline__ uint32_t ordered_bits(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Segment holding position i of a super tile of nl points after `level` splits:
// a segment longer than kLeafTile splits off its largest power-of-two prefix, so
// every split point is a multiple of each smaller tile size (256, 512, 1024).
__device__ __forceinline__ void bisect_segment(int i, int nl, int level, int *start, int *len) {
  int s = 0, l = nl;
  for (int k = 0; k < level && l > kLeafTile; ++k) {
    const int unit = 1 << (31 - __clz(l - 1));  // largest power of two below l
    if (i < s + unit) {
      l = unit;
    } else {
      s += unit;
      l -= unit;
    }
  }
  *start = s;
  *len = l;
}

// Compare-exchange of the bitonic network on a pair whose lower index is `lo_i`:
// keep the smaller key at the lower index when (lo_i & k) == 0, else the larger.
__device__ __forceinline__ uint64_t bitonic_keep(uint64_t mine, uint64_t other, bool lower,
                                                 bool ascending) {
  const uint64_t mn = mine < other ? mine : other, mx = mine < other ? other : mine;
  return (lower == ascending) ? mn : mx;
}

// The in-register stages (partner distance J < 8) of the network below.
template <int J>
__device__ __forceinline__ void bitonic_reg_stage(uint64_t (&v)[8], int t, int k) {
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (e & J) continue;
    const uint64_t a = v[e], b = v[e | J];
    if ((a > b) == (((8 * t + e) & k) == 0)) {
      v[e] = b;
      v[e | J] = a;
    }
  }
}

// Bitonic sort of kSuperTile keys, 8 consecutive keys per thread (1024 threads):
// partner distance j < 8 within a thread's registers, 8 <= j < 256 by warp
// shuffles, j >= 256 through shared memory (element i at (i % 8) * 1024 + i / 8, so
// a warp's accesses are consecutive).  Sorts each aligned block of kmax keys (a
// power of two) ascending: the merge phases stop at kmax, whose phase runs
// ascending everywhere.
__device__ void bitonic_sort_8192(uint64_t (&v)[8], uint64_t *sh, int kmax) {
  const int t = threadIdx.x;
  for (int k = 2; k <= kmax; k <<= 1) {
    const int kd = k == kmax ? 2 * kSuperTile : k;  // (i & kd) == 0: ascending
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 256) {
#pragma unroll
        for (int e = 0; e < 8; ++e) sh[e * 1024 + t] = v[e];
        __syncthreads();
        const int pt = t ^ (j >> 3);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int i = 8 * t + e;
          v[e] = bitonic_keep(v[e], sh[e * 1024 + pt], (t & (j >> 3)) == 0, (i & kd) == 0);
        }
        __syncthreads();
      } else if (j >= 8) {
        const int m = j >> 3;  // partner lane offset (< 32)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int i = 8 * t + e;
          const uint64_t o = __shfl_xor_sync(0xffffffffu, v[e], m);
          v[e] = bitonic_keep(v[e], o, (t & m) == 0, (i & kd) == 0);
        }
      } else if (j == 4) {
        bitonic_reg_stage<4>(v, t, kd);
      } else if (j == 2) {
        bitonic_reg_stage<2>(v, t, kd);
      } else {
        bitonic_reg_stage<1>(v, t, kd);
      }
    }
  }
}

// Recursive bisection of each super tile of kSuperTile consecutive points of
// `order` (in place): at each of five levels every segment longer than kLeafTile
// is sorted along the widest axis of its own box and split off at its largest
// power-of-two prefix, so tiles of 256, 512 and 1024 points are each one segment,
// of nearly square extent.  One bitonic sort of 64-bit keys (segment start,
// coordinate, position) per level keeps segments in place and ties in order.
__global__ void __launch_bounds__(1024) k_local_bisect(const double *__restrict__ pos, int n,
                                                       int32_t *__restrict__ order) {
  extern __shared__ __align__(16) unsigned char bsm[];
  uint64_t *sh = reinterpret_cast<uint64_t *>(bsm);                     // [kSuperTile]
  int32_t *idx = reinterpret_cast<int32_t *>(sh + kSuperTile);          // [2][kSuperTile]
  __shared__ uint32_t box[kSuperTile / kLeafTile][6];                   // ordered min, max
  __shared__ double ref[3];  // coordinates relative to the tile's first point, as floats
  __shared__ int kmax;       // sort blocks of this level: each segment lies in one
  const int t = threadIdx.x;
  const int base = blockIdx.x * kSuperTile;
  const int nl = min(kSuperTile, n - base);
  for (int i = t; i < nl; i += blockDim.x) idx[i] = order[base + i];
  if (t < 3) ref[t] = pos[3 * (size_t)order[base] + t];
  int cur = 0;
  for (int level = 0; level < 5; ++level) {
    for (int c = t; c < (kSuperTile / kLeafTile) * 6; c += blockDim.x)
      box[c / 6][c % 6] = (c % 6) < 3 ? 0xffffffffu : 0u;
    if (t == 0) kmax = 2;
    __syncthreads();
    // a warp's 256 consecutive positions lie in one segment (segments longer than
    // kLeafTile start at multiples of it): reduce in the warp, one atomic per warp
    int st[8], ln[8];
    uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    int blk = 2;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 8 * t + e;
      st[e] = 0;
      ln[e] = 0;
      if (i >= nl) continue;
      bisect_segment(i, nl, level, &st[e], &ln[e]);
      // smallest aligned power-of-two block holding the whole segment
      const int last = st[e] + ln[e] - 1;
      const int b = ln[e] > 1 ? 2 << (31 - __clz(st[e] ^ last)) : 2;
      blk = max(blk, b);
      if (ln[e] > kLeafTile) {
        const double *p = pos + 3 * (size_t)idx[cur * kSuperTile + i];
        for (int d = 0; d < 3; ++d) {
          const uint32_t o = ordered_bits((float)(p[d] - ref[d]));
          mn[d] = min(mn[d], o);
          mx[d] = max(mx[d], o);
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      for (int d = 0; d < 3; ++d) {
        mn[d] = min(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
        mx[d] = max(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
      }
      blk = max(blk, __shfl_xor_sync(0xffffffffu, blk, o));
    }
    if ((t & 31) == 0) {
      const int i0 = 8 * t;  // the warp's first position
      if (i0 < nl && ln[0] > kLeafTile)
        for (int d = 0; d < 3; ++d) {
          atomicMin(&box[st[0] / kLeafTile][d], mn[d]);
          atomicMax(&box[st[0] / kLeafTile][3 + d], mx[d]);
        }
      atomicMax(&kmax, blk);
    }
    __syncthreads();
    uint64_t v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 8 * t + e;
      uint64_t k = ~0ull;  // padding sorts last
      if (i < nl) {
        uint32_t c = 0;
        if (ln[e] > kLeafTile) {
          const uint32_t *b = box[st[e] / kLeafTile];
          int a = 0;
          float ext = -1.f;
          for (int d = 0; d < 3; ++d) {
            const float ed = from_ordered_bits(b[3 + d]) - from_ordered_bits(b[d]);
            if (ed > ext) {
              ext = ed;
              a = d;
            }
          }
          c = ordered_bits((float)(pos[3 * (size_t)idx[cur * kSuperTile + i] + a] - ref[a]));
        }
        k = ((uint64_t)st[e] << 45) | ((uint64_t)c << 13) | (uint64_t)i;
      }
      v[e] = k;
    }
    bitonic_sort_8192(v, sh, kmax);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = 8 * t + e;
      if (i < nl)
        idx[(cur ^ 1) * kSuperTile + i] = idx[cur * kSuperTile + (int)(v[e] & (kSuperTile - 1))];
    }
    cur ^= 1;
    __syncthreads();
  }
  for (int i = t; i < nl; i += blockDim.x) order[base + i] = idx[cur * kSuperTile + i];
}

// Per-block histogram of given keys (the packed tiling's sorts): hist[blk][cell].
__global__ void __launch_bounds__(256) k_hist(const SortSets sets) {
  const SortSet &S = sets.s[blockIdx.y];
  __shared__ uint32_t h[kCells];
  for (int c = threadIdx.x; c < kCells; c += blockDim.x) h[c] = 0;
  __syncthreads();
  const int i0 = blockIdx.x * kSortBlock;
  const int i1 = min(S.n, i0 + kSortBlock);
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) atomicAdd(&h[S.keys[i]], 1u);
  __syncthreads();
  for (int c = threadIdx.x; c < kCells; c += blockDim.x)
    S.hist[(size_t)blockIdx.x * kCells + c] = h[c];
}

// Per cell: the exclusive prefix of its counts over the blocks (in place) and their total.
__global__ void __launch_bounds__(128) k_scan_cells(const SortSets sets) {
  const SortSet &S = sets.s[blockIdx.y];
  const int cell = blockIdx.x * blockDim.x + threadIdx.x;
  const int nblk = (S.n + kSortBlock - 1) / kSortBlock;
  uint32_t run = 0, *h = S.hist + cell;
  int b = 0;
  for (; b + 8 <= nblk; b += 8) {
    uint32_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = h[(size_t)(b + j) * kCells];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      h[(size_t)(b + j) * kCells] = run;
      run += v[j];
    }
  }
  for (; b < nblk; ++b) {
    const uint32_t v = h[(size_t)b * kCells];
    h[(size_t)b * kCells] = run;
    run += v;
  }
  S.totals[cell] = run;
}

// Stable scatter of kSortBlock points by their cells.  Eight warps take 512 consecutive
// points each: a first walk, 32 points at a time, ranks every point among the earlier
// points of its cell in the warp (match.any), a prefix over the warps and the scanned
// totals turns the warps' counts into positions, and a last pass writes the order.  Bound by
// the latency of those dependent shared-memory updates: 16 here, 128 for one warp walking
// all 4096 points, which took 42 us for 262,144 points and 42 us for 16,384 (both sets
// in one launch of this kernel: 10 us, GB300).
constexpr int kScatWarps = 8, kScatSteps = kSortBlock / (32 * kScatWarps);
constexpr int kScatSmem = kScatWarps * kCells * 2 + kCells * 4;

__global__ void __launch_bounds__(32 * kScatWarps) k_scatter(const SortSets sets) {
  extern __shared__ __align__(16) unsigned char ssm[];
  uint16_t *cnt = reinterpret_cast<uint16_t *>(ssm);                            // [warp][cell]
  uint32_t *first = reinterpret_cast<uint32_t *>(ssm + kScatWarps * kCells * 2);  // [cell]
  __shared__ uint32_t warp_sum[kScatWarps];
  const SortSet &S = sets.s[blockIdx.y];
  const int i0 = blockIdx.x * kSortBlock;
  if (i0 >= S.n) return;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int c = t; c < kScatWarps * kCells * 2 / 16; c += 32 * kScatWarps)
    reinterpret_cast<uint4 *>(cnt)[c] = make_uint4(0u, 0u, 0u, 0u);
  // cells' first positions: exclusive scan of the totals (16 cells per thread) ...
  uint32_t v[16], sum = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 q = reinterpret_cast<const uint4 *>(S.totals)[4 * t + j];
    v[4 * j] = q.x; v[4 * j + 1] = q.y; v[4 * j + 2] = q.z; v[4 * j + 3] = q.w;
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) sum += v[j];
  uint32_t incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  uint32_t run = incl - sum;
  for (int w = 0; w < warp; ++w) run += warp_sum[w];
  // ... plus the points of earlier blocks
  const uint4 *before = reinterpret_cast<const uint4 *>(S.hist + (size_t)blockIdx.x * kCells);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 q = before[4 * t + j];
    uint4 f;
    f.x = run + q.x; run += v[4 * j];
    f.y = run + q.y; run += v[4 * j + 1];
    f.z = run + q.z; run += v[4 * j + 2];
    f.w = run + q.w; run += v[4 * j + 3];
    reinterpret_cast<uint4 *>(first)[4 * t + j] = f;
  }
  // ranks within each warp's points (cell << 16 | rank; 0xffffffff: past the end)
  uint32_t item[kScatSteps];
  uint16_t *mine = cnt + warp * kCells;
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < kScatSteps; ++k) {
    const int i = i0 + warp * (32 * kScatSteps) + 32 * k + lane;
    item[k] = i < S.n ? (uint32_t)S.keys[i] << 16 : 0xffffffffu;
  }
#pragma unroll
  for (int k = 0; k < kScatSteps; ++k) {
    const uint32_t key = item[k] >> 16, peers = __match_any_sync(0xffffffffu, key);
    const uint32_t prev = key < (uint32_t)kCells ? mine[key] : 0u;
    __syncwarp();
    if (key < (uint32_t)kCells) {
      item[k] |= prev + __popc(peers & lt);
      if ((peers >> lane) == 1u) mine[key] = (uint16_t)(prev + __popc(peers));  // highest lane
    }
    __syncwarp();
  }
  __syncthreads();
  // counts of the earlier warps, eight cells at a time (each count fits 13 bits)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = t + 256 * h;
    uint4 acc = make_uint4(0u, 0u, 0u, 0u);
    for (int w = 0; w < kScatWarps; ++w) {
      uint4 *q = reinterpret_cast<uint4 *>(cnt + w * kCells) + c;
      const uint4 x = *q;
      *q = acc;
      acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kScatSteps; ++k) {
    const uint32_t key = item[k] >> 16;
    if (key < (uint32_t)kCells)
      S.order[first[key] + mine[key] + (item[k] & 0xffffu)] =
          i0 + warp * (32 * kScatSteps) + 32 * k + lane;
  }
}

__global__ void __launch_bounds__(256) k_gather_pos(const double *__restrict__ pos,
                                                    const int32_t *__restrict__ order, int n,
                                                    int n_pad, double *__restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pad; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const size_t j = 3 * (size_t)(order ? order[i] : i);
      out[3 * (size_t)i] = pos[j];
      out[3 * (size_t)i + 1] = pos[j + 1];
      out[3 * (size_t)i + 2] = pos[j + 2];
    } else {
      out[3 * (size_t)i] = 0.0;
      out[3 * (size_t)i + 1] = 0.0;
      out[3 * (size_t)i + 2] = 0.0;
    }
  }
}

__global__ void __launch_bounds__(256) k_tile_bbox(const double *__restrict__ pos, int n,
                                                   int tile, double *__restrict__ tiles) {
  __shared__ Box64 w[8];
  const int i0 = blockIdx.x * tile;
  const int i1 = min(n, i0 + tile);
  Box64 b;
  b.clear();
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const double *p = pos + 3 * (size_t)i;
    b.add(p[0], p[1], p[2]);
  }
  b.warp_reduce();
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x < 3) {
    const int d = threadIdx.x;
    long long lo = w[0].lo[d], hi = w[0].hi[d];
    for (int j = 1; j < 8; ++j) {
      lo = min(lo, w[j].lo[d]);
      hi = max(hi, w[j].hi[d]);
    }
    tiles[6 * blockIdx.x + d] = 0.5 * (from_ordered64(lo) + from_ordered64(hi));
    tiles[6 * blockIdx.x + 3 + d] = 0.5 * (from_ordered64(hi) - from_ordered64(lo));
  }
}

// Points in tile order (zeros past the end up to n_pad), the boxes of the tiles of 256 .. 8192
// points of one super tile (levels 0 .. 5), and the super tile's part of their statistics.
// One warp per leaf of 256 points; the box of a longer tile merges its leaves' keys.  The
// FP64 operations left, two conversions of a box and its diagonal, are spread over lanes.
struct GatherSet {
  const double *pos;
  const int32_t *order;
  int n, n_pad;
  double *out, *boxes;
  BoxStats *parts;   // per super tile
  BoxStats *stats;   // of the whole set
};
struct GatherSets {
  GatherSet s[2];
};
__global__ void __launch_bounds__(1024) k_gather_boxes(const GatherSets sets) {
  constexpr int kLeaves = kSuperTile / kLeafTile;
  __shared__ long long leaf[kLeaves][6];
  __shared__ double box[2 * kLeaves][6];
  const GatherSet &S = sets.s[blockIdx.y];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, base = blockIdx.x * kSuperTile, n = S.n;
  if (base >= S.n_pad) return;
  Box64 b;
  b.clear();
  // all of a thread's points are asked for before the first is stored: a store between two
  // loads would make the second wait for it (the compiler cannot tell the arrays apart).  10007
  // and 50021 points in 17 us against 21, 2^20 in 28 against 31
  constexpr int kSteps = kLeafTile / 32, kAhead = 4;
  const int first = base + warp * kLeafTile + lane;
  int32_t at[kSteps];
#pragma unroll
  for (int k = 0; k < kSteps; ++k) at[k] = first + 32 * k < n ? S.order[first + 32 * k] : 0;
#pragma unroll
  for (int h = 0; h < kSteps; h += kAhead) {
    double v[kAhead][3];
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
#pragma unroll
      for (int d = 0; d < 3; ++d)
        v[k][d] = first + 32 * (h + k) < n ? S.pos[3 * (size_t)at[h + k] + d] : 0.0;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int i = first + 32 * (h + k);
      if (i < n) b.add(v[k][0], v[k][1], v[k][2]);
      if (i < S.n_pad) {
        double *o = S.out + 3 * (size_t)i;
        o[0] = v[k][0]; o[1] = v[k][1]; o[2] = v[k][2];
      }
    }
  }
  if (base >= n) return;
  b.warp_reduce();
  if (lane < 6) leaf[warp][lane] = lane < 3 ? (lane == 0 ? b.lo[0] : lane == 1 ? b.lo[1] : b.lo[2])
                                            : (lane == 3 ? b.hi[0] : lane == 4 ? b.hi[1] : b.hi[2]);
  __syncthreads();
  // thread t: axis t % 3 of tile t / 3 of the super tile's 63
  if (t < 3 * (2 * kLeaves - 1)) {
    const int d = t % 3;
    int level = 0, tile = t / 3;
    while (tile >= (kLeaves >> level)) tile -= kLeaves >> level++;
    const int size = kLeafTile << level;
    if (base + tile * size < n) {
      size_t at = blockIdx.x * (size_t)(kSuperTile / size) + tile;
      for (int l = 0; l < level; ++l) at += (n + (kLeafTile << l) - 1) / (kLeafTile << l);
      long long lo = kOrderedMax, hi = kOrderedMin;
      for (int f = tile << level; f < (tile + 1) << level; ++f) {
        lo = min(lo, leaf[f][d]);
        hi = max(hi, leaf[f][3 + d]);
      }
      const double c = 0.5 * (from_ordered64(lo) + from_ordered64(hi));
      const double h = 0.5 * (from_ordered64(hi) - from_ordered64(lo));
      S.boxes[6 * at + d] = c;
      S.boxes[6 * at + 3 + d] = h;
      box[t / 3][d] = c;
      box[t / 3][3 + d] = h;
    }
  }
  __syncthreads();
  // warp l: the largest half extents of level l, a lane per tile; the super tile's own box
  // comes from the last level
  if (warp < kBoxLevels) {
    BoxStats &o = S.parts[blockIdx.x];
    int first = 0;
    for (int l = 0; l < warp; ++l) first += kLeaves >> l;
    const bool in = lane < (kLeaves >> warp) && base + lane * (kLeafTile << warp) < n;
    double h2 = 0.0;
    long long m[4];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double e = in ? box[first + lane][3 + d] : 0.0;
      m[d] = in ? ordered64(e) : 0;
      h2 = __dadd_rn(h2, __dmul_rn(e, e));
    }
    m[3] = in ? ordered64(__dsqrt_rn(h2)) : 0;
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
      for (int d = 0; d < 4; ++d) m[d] = max(m[d], __shfl_xor_sync(0xffffffffu, m[d], s));
    if (lane < 3) o.hd[warp][lane] = from_ordered64(lane == 0 ? m[0] : lane == 1 ? m[1] : m[2]);
    if (lane == 3) o.h[warp] = from_ordered64(m[3]);
    if (warp == kBoxLevels - 1 && lane < 3) {
      o.lo[lane] = box[first][lane] - box[first][3 + lane];
      o.hi[lane] = box[first][lane] + box[first][3 + lane];
    }
  }
}

// All super tiles' statistics into one: warp j reduces entry j (minimum for lo, else maximum).
__global__ void __launch_bounds__(1024) k_box_stats(const GatherSets sets) {
  const GatherSet &S = sets.s[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = (S.n + kSuperTile - 1) / kSuperTile;
  if (warp >= kBoxStatDoubles || nb == 0) return;
  const bool low = warp < 3;
  long long v = low ? kOrderedMax : warp < 6 ? kOrderedMin : 0;
  for (int b = lane; b < nb; b += 32) {
    const long long x = ordered64(reinterpret_cast<const double *>(S.parts + b)[warp]);
    v = low ? min(v, x) : max(v, x);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const long long x = __shfl_xor_sync(0xffffffffu, v, o);
    v = low ? min(v, x) : max(v, x);
  }
  if (lane == 0) reinterpret_cast<double *>(S.stats)[warp] = from_ordered64(v);
}
static_assert(kBoxStatDoubles <= 32 && (kLeafTile << (kBoxLevels - 1)) == kSuperTile,
              "one warp per statistic, the last level is the super tile");

__global__ void __launch_bounds__(256) k_gather_ap(const double *__restrict__ amp,
                                                   const double *__restrict__ phase,
                                                   const int32_t *__restrict__ order, int n,
                                                   int n_pad, double2 *__restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pad; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const int j = order ? order[i] : i;
      out[i] = make_double2(phase[j], amp[j]);
    } else {
      out[i] = make_double2(0.0, 0.0);
    }
  }
}

// r as the nearest float and what that leaves, rounded to a float: by its bits where both are
// normal numbers (conversions from and to FP64 run at the FP64 pipe's rate, 4 of them and a
// subtraction a coordinate).
__device__ __forceinline__ void split_float(double r, float *hi, float *lo) {
  const uint32_t h = (uint32_t)__double2hiint(r), l = (uint32_t)__double2loint(r);
  const int e = (int)((h >> 20) & 0x7ffu) - 1023;
  if (e >= -60 && e <= 60) {
    const uint32_t near = (l >> 28) & 1u, sign = h & 0x80000000u;
    *hi = __uint_as_float((sign | (uint32_t)(e + 127) << 23 | (h & 0xfffffu) << 3 | l >> 29) + near);
    const int rest = (int)(l & 0x1fffffffu) - (int)(near << 29);  // of 2^(e - 52)
    *lo = __int2float_rn(rest) * __uint_as_float(sign | (uint32_t)(e - 52 + 127) << 23);
  } else if (r == 0.0) {
    *hi = *lo = 0.f;
  } else {
    *hi = (float)r;
    *lo = (float)(r - (double)*hi);
  }
}

// Offsets of tile-ordered points from their tile's centre as float-float pairs:
// out[6 i .. 6 i + 2] = hi = fl32(p - c), out[6 i + 3 .. 6 i + 5] = lo =
// fl32((p - c) - hi); zeros for the padding i >= n.  Bound by memory (48 bytes a point) once the
// split is not FP64 work: 2^20 + 2^18 points in 26 us, one launch, against 42 in two.
__global__ void __launch_bounds__(256) k_rel_hilo(const RelSets sets) {
  const RelSet &S = sets.s[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n_out; i += gridDim.x * blockDim.x) {
    float *o = S.out + 6 * (size_t)i;
    float hi[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f};
    if (i < S.n) {
      const double *c = S.tiles + 6 * (size_t)(i / S.tile), *p = S.pos + 3 * (size_t)i;
#pragma unroll
      for (int d = 0; d < 3; ++d) split_float(p[d] - c[d], &hi[d], &lo[d]);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      o[d] = hi[d];
      o[3 + d] = lo[d];
    }
  }
}

// (phase reduced to [-pi, pi], amplitude) in float, tile order.
__device__ __forceinline__ float2 apf_record(const double *amp, const double *phase,
                                             const int32_t *order, int n, int i) {
  if (i >= n) return make_float2(0.f, 0.f);
  const int j = order ? order[i] : i;
  const double p = phase[j];
  const double q = rint(p * kInvTwoPi);  // two-constant Cody-Waite reduction
  const double r = fma(-q, kTwoPiLo, fma(-q, kTwoPiHi, p));
  return make_float2((float)r, (float)amp[j]);
}
__global__ void __launch_bounds__(256) k_gather_apf(const double *__restrict__ amp,
                                                    const double *__restrict__ phase,
                                                    const int32_t *__restrict__ order, int n,
                                                    int n_pad, float2 *__restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pad; i += gridDim.x * blockDim.x)
    out[i] = apf_record(amp, phase, order, n, i);
}
__global__ void __launch_bounds__(256) k_gather_apf_batched(const GatherApf *__restrict__ sets,
                                                            int n_sets) {
  int lo = 0, hi = n_sets;  // the last set whose first block is <= this one
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (sets[mid].first <= (int)blockIdx.x) lo = mid; else hi = mid;
  }
  const GatherApf G = sets[lo];
  const int i0 = (blockIdx.x - G.first) * 1024 + threadIdx.x;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = i0 + 256 * k;
    if (i < G.n_pad) G.out[i] = apf_record(G.amp, G.phase, G.order, G.n, i);
  }
}

__global__ void __launch_bounds__(256) k_iota(int32_t *__restrict__ order, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    order[i] = i;
}

int grid_for(int n, int per_block, int cap) {
  int g = (n + per_block - 1) / per_block;
  return g < 1 ? 1 : (g > cap ? cap : g);
}

}  // namespace

size_t sort_hist_entries(int n) {
  const size_t nblk = (size_t)((n + kSortBlock - 1) / kSortBlock);
  return (nblk ? nblk : 1) * kCells;
}

static SortSet sort_set(const double *pos, int n, int32_t *order, const TileScratch &t) {
  SortSet S{};
  S.pos = pos;
  S.n = n;
  S.parts = grid_for(n, 256 * 8, 152);
  S.box = reinterpret_cast<long long *>(t.bbox_scratch);
  S.keys = t.keys;
  S.hist = t.hist;
  S.totals = t.scan;
  S.order = order;
  return S;
}

// Stable counting sort by S.keys (< kCells) into S.order (indices 0..n-1) of one or two
// sets; `counted`: their histograms are filled already.
static int counting_sort(const SortSets &sets, int count, bool counted, cudaStream_t s) {
  int nblk = 0;
  for (int i = 0; i < count; ++i) nblk = std::max(nblk, (sets.s[i].n + kSortBlock - 1) / kSortBlock);
  if (nblk > 4096) return fail(HOLO_ERR_INVALID, "point set too large for the tiler");
  HOLO_TRY(kernel_setup<k_scatter>(32 * kScatWarps, kScatSmem, nullptr));
  if (!counted) {
    k_hist<<<dim3(nblk, count), 256, 0, s>>>(sets); note_launches(1);
  }
  k_scan_cells<<<dim3(kCells / 128, count), 128, 0, s>>>(sets); note_launches(1);
  k_scatter<<<dim3(nblk, count), 32 * kScatWarps, kScatSmem, s>>>(sets); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

static int hilbert_order(const SortSets &sets, int count, cudaStream_t s) {
  int parts = 0, n = 0;
  for (int i = 0; i < count; ++i) {
    parts = std::max(parts, sets.s[i].parts);
    n = std::max(n, sets.s[i].n);
  }
  k_box_parts<<<dim3(parts, count), 256, 0, s>>>(sets); note_launches(1);
  k_cell_keys<<<dim3((n + 1023) / 1024, count), 256, 0, s>>>(sets); note_launches(1);
  return counting_sort(sets, count, true, s);
}

static int packed_order(const double *pos, int n, int32_t *order, const TileScratch &t,
                        cudaStream_t s) {
  constexpr int kBisectSmem = kSuperTile * (8 + 2 * 4);
  HOLO_TRY(kernel_setup<k_local_bisect>(1024, kBisectSmem, nullptr));
  if (n <= kSuperTile) {
    HOLO_TRY(launch_iota(order, n, s));
  } else {
    SortSets sets{};
    SortSet &S = sets.s[0];
    S = sort_set(pos, n, t.tmp_a, t);
    S.hist = nullptr;  // counted by k_hist
    k_box_parts<<<dim3(S.parts, 1), 256, 0, s>>>(sets); note_launches(1);
    k_bbox_final<<<1, 256, 0, s>>>(S.box, S.parts, t.bbox); note_launches(1);
    S.hist = t.hist;
    const int g = grid_for(n, 256, 8192);
    // order along the widest axis -> each point's strip
    k_axis_keys<<<g, 256, 0, s>>>(pos, n, t.bbox, 0, t.keys); note_launches(1);
    HOLO_TRY(counting_sort(sets, 1, false, s));
    k_strip_keys<<<g, 256, 0, s>>>(t.tmp_a, n, t.bbox, t.keys2); note_launches(1);
    // along the second axis, then (stably) by strip
    k_axis_keys<<<g, 256, 0, s>>>(pos, n, t.bbox, 1, t.keys); note_launches(1);
    S.order = t.tmp_b;
    HOLO_TRY(counting_sort(sets, 1, false, s));
    k_permute_keys<<<g, 256, 0, s>>>(t.keys2, t.tmp_b, n, t.keys); note_launches(1);
    S.order = t.tmp_a;
    HOLO_TRY(counting_sort(sets, 1, false, s));
    k_compose<<<g, 256, 0, s>>>(t.tmp_b, t.tmp_a, n, order); note_launches(1);
  }
  k_local_bisect<<<(n + kSuperTile - 1) / kSuperTile, 1024, kBisectSmem, s>>>(pos, n, order);
  note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int tile_order(const double *pos, int n, int32_t *order, const TileScratch &t, cudaStream_t s,
               int tiling) {
  if (n <= 0) return HOLO_OK;
  if (tiling == kTilePacked) return packed_order(pos, n, order, t, s);
  SortSets sets{};
  sets.s[0] = sort_set(pos, n, order, t);
  return hilbert_order(sets, 1, s);
}

int tile_sets(const TileSet *set, int count, int tiling, cudaStream_t s) {
  SortSets sets{};
  int sorted = 0;
  for (int i = 0; i < count; ++i) {
    if (set[i].known) {
      HOLO_CUDA(cudaMemcpyAsync(set[i].order, set[i].known, (size_t)set[i].n * sizeof(int32_t),
                                cudaMemcpyDeviceToDevice, s));
    } else if (tiling == kTilePacked) {
      HOLO_TRY(packed_order(set[i].pos, set[i].n, set[i].order, set[i].scratch, s));
    } else {
      sets.s[sorted++] = sort_set(set[i].pos, set[i].n, set[i].order, set[i].scratch);
    }
  }
  if (sorted) HOLO_TRY(hilbert_order(sets, sorted, s));
  GatherSets g{};
  int supers = 1;
  for (int i = 0; i < count; ++i) {
    g.s[i] = {set[i].pos, set[i].order, set[i].n, set[i].n_pad, set[i].pos_sorted, set[i].boxes,
              set[i].parts, set[i].stats};
    supers = std::max(supers, (set[i].n_pad + kSuperTile - 1) / kSuperTile);
  }
  k_gather_boxes<<<dim3(supers, count), 1024, 0, s>>>(g); note_launches(1);
  k_box_stats<<<count, 1024, 0, s>>>(g); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_gather_pos(const double *pos, const int32_t *order, int n, int n_pad, double *out,
                      cudaStream_t s) {
  if (n_pad <= 0) return HOLO_OK;
  k_gather_pos<<<grid_for(n_pad, 256, 8192), 256, 0, s>>>(pos, order, n, n_pad, out); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_pack_pos(const double *pos, int n, int n_pad, double *out, cudaStream_t s) {
  return launch_gather_pos(pos, nullptr, n, n_pad, out, s);
}

int launch_tile_bbox(const double *pos_sorted, int n, int tile, double *tiles, cudaStream_t s) {
  if (n <= 0) return HOLO_OK;
  const int nt = (n + tile - 1) / tile;
  k_tile_bbox<<<nt, 256, 0, s>>>(pos_sorted, n, tile, tiles); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_gather_ap(const double *amp, const double *phase, const int32_t *order, int n,
                     int n_pad, double2 *out, cudaStream_t s) {
  if (n_pad <= 0) return HOLO_OK;
  k_gather_ap<<<grid_for(n_pad, 256, 8192), 256, 0, s>>>(amp, phase, order, n, n_pad, out); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_pack_ap(const double *amp, const double *phase, int n, int n_pad, double2 *out,
                   cudaStream_t s) {
  return launch_gather_ap(amp, phase, nullptr, n, n_pad, out, s);
}

int launch_rel_hilo(const RelSet *set, int count, cudaStream_t s) {
  RelSets sets{};
  int most = 0;
  for (int i = 0; i < count; ++i) {
    sets.s[i] = set[i];
    most = std::max(most, set[i].n_out);
  }
  if (most <= 0) return HOLO_OK;
  k_rel_hilo<<<dim3(grid_for(most, 256, 8192), count), 256, 0, s>>>(sets); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_gather_apf(const double *amp, const double *phase, const int32_t *order, int n,
                      int n_pad, float2 *out, cudaStream_t s) {
  if (n_pad <= 0) return HOLO_OK;
  k_gather_apf<<<grid_for(n_pad, 256, 8192), 256, 0, s>>>(amp, phase, order, n, n_pad, out); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int launch_gather_apf_batched(const GatherApf *sets_dev, int n_sets, int blocks, cudaStream_t s) {
  if (n_sets <= 0 || blocks <= 0) return HOLO_OK;
  k_gather_apf_batched<<<blocks, 256, 0, s>>>(sets_dev, n_sets); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

int tiler_preload_hilbert() {
  cudaFuncAttributes a;
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_box_parts));
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_cell_keys));
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_scan_cells));
  HOLO_TRY(kernel_setup<k_scatter>(32 * kScatWarps, kScatSmem, nullptr));
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_gather_pos));
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_tile_bbox));
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_rel_hilo));
  HOLO_CUDA(cudaFuncGetAttributes(&a, k_gather_apf));
  return HOLO_OK;
}

int launch_iota(int32_t *order, int n, cudaStream_t s) {
  if (n <= 0) return HOLO_OK;
  k_iota<<<grid_for(n, 256, 8192), 256, 0, s>>>(order, n); note_launches(1);
  HOLO_CUDA(cudaGetLastError());
  return HOLO_OK;
}

}  // namespace holo
