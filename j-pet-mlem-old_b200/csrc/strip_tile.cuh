// Device pieces shared by the tile kernels (strip_kernels.cu, strip_pairs.cu).
#pragma once

#include "strip_internal.h"
#include "strip_device.cuh"

namespace stripmlem {

namespace {

constexpr unsigned kFull = 0xffffffffu;
// Tile kernels whose shared-memory windows leave room for one CTA per SM
// run 1024-thread CTAs (32 warps, 64 registers each), so the SM keeps as
// many resident warps as with two 512-thread CTAs.
constexpr int kWideThreads = 1024;
constexpr int kMaxWarps = kWideThreads / 32;

__device__ __forceinline__ EventPack pack_event(const EventF& e) {
  return EventPack{e.tan, e.y, e.z, e.sec, (unsigned)e.tlx | ((unsigned)e.brx << 16),
                   (unsigned)e.tly | ((unsigned)e.bry << 16)};
}

// Accumulation of the per-row partial sums of D_e within a lane.
template <int ACC>
struct RowSum;
template <>
struct RowSum<STRIP_ACCUM_FP32> {
  float s = 0.0f;
  __device__ __forceinline__ void add(float x) { s += x; }
  __device__ __forceinline__ double total() const { return (double)s; }
};
template <>
struct RowSum<STRIP_ACCUM_KAHAN> {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const float yv = __fsub_rn(x, c);
    const float t = __fadd_rn(s, yv);
    c = __fsub_rn(__fsub_rn(t, s), yv);
    s = t;
  }
  __device__ __forceinline__ double total() const {
    return (double)s - (double)c;
  }
};
template <>
struct RowSum<STRIP_ACCUM_FP64> {
  double s = 0.0;
  __device__ __forceinline__ void add(float x) { s += (double)x; }
  __device__ __forceinline__ double total() const { return s; }
};

// Shared-memory access by 32-bit shared-space byte address: the walks below
// advance one address register per step and let the loads and atomics use
// immediate offsets.
__device__ __forceinline__ float lds32(uint32_t addr) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void red_shared_add(uint32_t addr, unsigned v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Per-CTA state of the work item in flight: the unweighted window's
// fixed-point budget (units of 2^8), the item's sum of 1 / D_e, and the
// events the unweighted window had no room for (bit i: event begin + i).
constexpr unsigned kBudgetUnits = (unsigned)(kFixedBudget / 256.0f);
__shared__ unsigned s_fx_budget;
__shared__ float s_item_rsum;
__shared__ unsigned s_fb_bits[kMaxItemEvents / 32];
__shared__ int s_fb_n;

// Fixed-point scale of an adjoint work item: every addend is K_j w_e with
// K_j <= a.kbound (the GaussianKernel's bound, E <= 1 and a'Sa >= 2 R^2 ipsz)
// and |w_e| <= W, the item's largest weight, so with B = kbound * W the
// scale 2^s keeps each addend below 2^22 and the item's sum below 2^31.
// *negative: whether any weight is below zero.
__device__ int adjoint_shift(const LaunchArgs& a, const WorkItem& it, int lane,
                             bool* negative = nullptr) {
  __shared__ float s_wmax[kMaxWarps];
  __shared__ int s_shift;
  float m = 0.0f;
  bool neg = false;
  for (int64_t i = it.begin + threadIdx.x; i < it.begin + it.count;
       i += blockDim.x) {
    const float w = a.wf_in[i];
    m = fmaxf(m, fabsf(w));
    neg |= !(w >= 0.0f);  // NaN too
  }
  if (negative) *negative = __syncthreads_or(neg);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(kFull, m, o));
  if (lane == 0) s_wmax[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float W = 0.0f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) W = fmaxf(W, s_wmax[i]);
    const float B = a.kbound * W * 1.0001f;
    const float n = (float)it.count + (float)(it.count >> 7) + 1.0f;
    const float lim = fminf(4194304.0f, 2147483648.0f / n);
    int sh = 0;
    if (B > 0.0f && B < 3.0e38f)
      sh = (int)floorf(log2f(lim / B)) - 1;
    s_shift = max(-120, min(120, sh));
  }
  __syncthreads();
  return s_shift;
}

// f(row, column) over a window of wyn rows and wxn columns.  Column-major, a warp
// takes 8 rows x 4 columns at a time: 4-way shared-memory conflicts (a row of
// 32 columns: 32-way) and whole sectors of the image in L1; row-major, the rows
// one after the other.
template <bool COLUMNS, class F>
__device__ __forceinline__ void each_pixel(int wxn, int wyn, int lane, F&& f) {
  if constexpr (COLUMNS) {
    const int n_ct = (wxn + 3) >> 2, n_t = n_ct * ((wyn + 7) >> 3);
    for (int t = threadIdx.x >> 5; t < n_t; t += blockDim.x >> 5) {
      const int rt = t / n_ct, r = 8 * rt + (lane & 7), c = 4 * (t - rt * n_ct) + (lane >> 3);
      if (r < wyn && c < wxn) f(r, c);
    }
  } else {
    for (int q = threadIdx.x; q < wxn * wyn; q += blockDim.x) {
      const int r = q / wxn;
      f(r, q - r * wxn);
    }
  }
}

// Sum of v over the CTA, returned to every thread (two barriers).
__device__ __forceinline__ float block_sum(float v) {
  __shared__ float s_part[kMaxWarps];
  __shared__ float s_total;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_part[w];
    s_total = t;
  }
  __syncthreads();
  return s_total;
}

}  // namespace

}  // namespace stripmlem
