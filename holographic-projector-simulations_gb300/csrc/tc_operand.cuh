// tc_operand.cuh -- shared-memory operands of the tf32 tensor-core kernels (kernel_tc.cu:
// the per-pair phase; kernel_expand.cu: the cluster expansions) and their bounded waits.
// Included inside an anonymous namespace of holo.
#pragma once

constexpr int kTcM = 128, kTcK = 8;             // rows and depth of one MMA
constexpr uint32_t kTcLbo = 128, kTcSbo = 256;  // operand layout (bytes), see tc_off

// Float offset of element (row r, feature k) of a K-major tf32 operand with K = 8:
// core matrices of 8 rows x 4 features (16 B rows, 128 B), the two along K 128 B
// apart (LBO), 8-row groups 256 B apart (SBO).  Rows of one 128- or 256-row block
// are contiguous, so block b starts at row 128 b / 256 b.
__host__ __device__ __forceinline__ int tc_off(int r, int k) {
  return (r >> 3) * 64 + (k >> 2) * 32 + (r & 7) * 4 + (k & 3);
}

// Row r of an operand pair (hi, lo): the 8 features split into TF32 high parts and
// TF32 remainders, written as four 16-byte stores (features 0-3 and 4-7 of a row
// are contiguous; eight consecutive rows fill 128 bytes, so a warp's stores are
// free of bank conflicts).
__device__ __forceinline__ void store_row_split(float *hi, float *lo, int r, const float *x) {
  float h[kTcK], l[kTcK];
#pragma unroll
  for (int k = 0; k < kTcK; ++k) {
    h[k] = ptx::to_tf32_int(x[k]);
    l[k] = ptx::to_tf32_int(__fsub_rn(x[k], h[k]));
  }
  *reinterpret_cast<float4 *>(hi + tc_off(r, 0)) = make_float4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<float4 *>(hi + tc_off(r, 4)) = make_float4(h[4], h[5], h[6], h[7]);
  *reinterpret_cast<float4 *>(lo + tc_off(r, 0)) = make_float4(l[0], l[1], l[2], l[3]);
  *reinterpret_cast<float4 *>(lo + tc_off(r, 4)) = make_float4(l[4], l[5], l[6], l[7]);
}

// Bounded wait that gives up at once when the CTA has aborted; sleep_ns > 0: poll with
// that much sleep in between.
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                        int *err, unsigned sleep_ns = 0) {
  if (*abort_flag) return false;
  if (sleep_ns ? ptx::mbar_wait_bounded_sleep(bar, parity, kWaitCycles, sleep_ns)
               : ptx::mbar_wait_bounded(bar, parity, kWaitCycles))
    return true;
  *abort_flag = 1;
  atomicExch(err, kDevErrTimeout);
  return false;
}
