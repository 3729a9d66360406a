// The 3D hybrid MLEM iteration on sm_100a: k_mlem, and the windowed kernels
// below it for dense event lists.
//
// k_mlem: one warp per frame event.  The event's voxels are its LOR pixel infos
// [info_begin, info_end) times its planes [plane_begin, plane_end); the warp
// walks them flattened with the plane fastest.  The volume is held on the
// device with the plane index fastest (z-fast: voxel (x, y, z) at
// (x + n_c y) n_p + z), so a warp's image reads and accumulator atomics fall
// on a few contiguous sectors; the boundary layout (x fastest) is restored
// by launch_from_zfast.
//
// Per voxel (GaussianKernel::normalized, src/2d/strip/gaussian_kernel.h:
// 51-105, in the frame of the event's LOR):
//   K = c / sqrt(a' S a) exp(-b' S b / 2) / sens(z, up),
//   sens = (atan u - atan v) / pi,  weight = K w rho,  D += weight s.
// Everything that depends on the pixel only (c / sqrt(a' S a) w, (up_p - up)
// tan, the b_r term, 1 / (R -+ up_p), the pixel's sensitivity and its base
// index) is computed once per pixel into the warp's shared memory; per voxel
// remain z, the two ratios of the sensitivity (from z exactly as the
// reference forms them, so the decisions sens <= 0 at z = +-L/2 are the
// reference's), one exp2, the arctangent difference atan u - atan v =
// atan2(u - v, 1 + u v) by atan2_pos below, and an image load.  (A table of
// 1 / sens per pixel info and plane -- it depends on the LOR, the pixel and
// the plane only -- was slower: 414 against 252 ms per iteration on the
// big-barrel workload, the walk waiting on its HBM loads; with the events in
// LOR order, so that the rows in use stay in L2, still 279 against 204 ms.)
// Pass 1 keeps each
// voxel's weight in a per-warp shared cache (first kCache voxels) and the
// next kSpill in a per-warp slab of global memory (written and read back by
// the same warp within microseconds, so it stays in L2); pass 2
// scatters weight / D with one red.global.add.f32 per voxel, reading the
// cache or recomputing past it.
#include <algorithm>
#include <climits>
#include <cmath>

#include "hybrid_internal.h"

namespace hybridmlem {

namespace {

// Launch shape and per-warp cache (compile-time tuning constants).
#ifndef HYBRID_WARPS
#define HYBRID_WARPS 8
#endif
#ifndef HYBRID_CACHE
#define HYBRID_CACHE 2048
#endif
#ifndef HYBRID_BLOCKS_PER_SM
#define HYBRID_BLOCKS_PER_SM 3
#endif
#ifndef HYBRID_SPILL
#define HYBRID_SPILL 16384
#endif
#ifndef HYBRID_UNROLL
#define HYBRID_UNROLL 1
#endif
#ifndef HYBRID_UNROLL2
#define HYBRID_UNROLL2 1
#endif
constexpr int kWarps = HYBRID_WARPS;
constexpr int kThreads = kWarps * 32;
constexpr int kCache = HYBRID_CACHE;          // cached voxel weights per warp
constexpr int kSpill = HYBRID_SPILL;          // further weights per warp in global memory
constexpr int kBlocksPerSm = HYBRID_BLOCKS_PER_SM;
constexpr int kUnroll = HYBRID_UNROLL;           // pass-1 voxel-loop unroll
constexpr int kUnroll2 = HYBRID_UNROLL2;         // pass-2 voxel-loop unroll

// atan2(a, b) for a > 0, in (0, pi): the quotient of the smaller by the
// larger of a and |b| (fast division) folded into [0, 1], an odd polynomial
// t P(t^2) of degree 15 for atan on [0, 1], then the quadrant.  The
// coefficients come from tests/golden/fit_atan.py: Lawson's iteratively
// reweighted least squares toward the minimax absolute error (3.75e-8 in
// exact arithmetic, 1.2e-7 evaluated in binary32), rounded to binary32.
// The reference's atanf(u) - atanf(v) carries about the same binary32
// rounding.
__device__ __forceinline__ float atan2_pos(float a, float b) {
  const float ab = fabsf(b);
  const float mx = fmaxf(a, ab), mn = fminf(a, ab);
  const float t = __fdividef(mn, mx);
  const float s = t * t;
  float p = -0.0040545654483139515f;
  p = fmaf(p, s, 0.021862952038645744f);
  p = fmaf(p, s, -0.0559123195707798f);
  p = fmaf(p, s, 0.0964219719171524f);
  p = fmaf(p, s, -0.1390862911939621f);
  p = fmaf(p, s, 0.19946566224098206f);
  p = fmaf(p, s, -0.33329859375953674f);
  p = fmaf(p, s, 0.9999993443489075f);
  float r = t * p;
  if (a > ab) r = 1.5707963267948966f - r;
  if (b < 0.0f) r = 3.14159265358979f - r;
  return r;
}

// z of plane iz (VoxelGrid::center_z_at, voxel_grid.h:38-40).
__device__ __forceinline__ float plane_z(const GridF& g, int iz) {
  return ((float)iz + 0.5f) * g.p + g.z_left;
}

// pi / (pi sens) of a voxel at z for a pixel at up_p in a LOR of half length
// R (GaussianKernel::sensitivity, gaussian_kernel.h:139-148, with the two
// quotients as products by 1 / (R -+ up_p)); 0 where sens <= 0.  The signs
// of the two ratios, hence the decision sens <= 0, are the reference's.
__device__ __forceinline__ float inv_sens(float half_L, float z, float ra, float rb) {
  const float lmz = half_L - z, lpz = half_L + z;
  const float u = fminf(lmz * ra, lpz * rb);
  const float v = fmaxf(-lpz * ra, -lmz * rb);
  const float a = u - v;
  if (!(a > 0.0f)) return 0.0f;
  return __fdividef(3.14159265358979f, atan2_pos(a, fmaf(u, v, 1.0f)));
}

__device__ __forceinline__ float proj_up(const GridF& g, short2 p, float4 md) {
  const float cx = g.llc_x + (float)p.x * g.p;
  const float cy = g.llc_y + (float)p.y * g.p;
  return (cx - md.x) * md.z + (cy - md.y) * md.w;
}

// Event-dependent pixel terms of one chunk of 32 pixel infos.
struct PixelData {
  float4 t[32];    // c / sqrt(a' S a) w, (up_p - up) tan, b_r S_dl b_r, s
  float2 r[32];    // 1 / (R - up_p), 1 / (R + up_p)
  int base[32];    // z-fast index of plane 0
};

struct WarpSmem {
  PixelData px;
  float cache[kCache];
};

__device__ __forceinline__ void load_pixels(const GridF& g, const GeometryDev& geo,
                                            const float* __restrict__ sens, const Frame& f,
                                            float4 md, float R, int c0, int n_pix, int lane,
                                            PixelData& px) {
  const int k = c0 + lane;
  if (k < n_pix) {
    const int64_t info = (int64_t)f.info_begin + k;
    const short2 p = geo.pix[info];
    const float w = geo.w[info];
    const float upp = proj_up(g, p, md);
    const float dy = upp - f.up;
    const float yp = dy + f.up;
    const float sec_sq = f.sec * f.sec;
    const float ap = -(yp - R) * sec_sq;
    const float aq = -(yp + R) * sec_sq;
    const float ar = -2.0f * yp * f.sec * f.tan;
    const float aca = ap * g.ipz * ap + aq * g.ipz * aq + ar * g.ipdl * ar;
    const float br = -2.0f * dy * f.sec;
    const int pidx = p.x + g.nc * p.y;
    px.t[lane] = make_float4(g.norm_c * rsqrtf(aca) * w, dy * f.tan, br * g.ipdl * br,
                             sens[pidx]);
    px.r[lane] = make_float2(__frcp_rn(R - upp), __frcp_rn(R + upp));
    px.base[lane] = pidx * g.np;
  }
  __syncwarp();
}

// K w (without rho) of voxel (pixel j of the chunk, plane iz).
__device__ __forceinline__ float voxel_kw(const GridF& g, const Frame& f, const PixelData& px,
                                          int j, int iz, float half_L) {
  const float4 t4 = px.t[j];
  const float z = plane_z(g, iz);
  const float2 r = px.r[j];
  const float is = inv_sens(half_L, z, r.x, r.y);
  if (is == 0.0f) return 0.0f;
  const float bpq = (z - f.right) - t4.y;
  const float t = bpq * g.ipz * bpq;
  const float bcb = (t + t) + t4.z;
  return t4.x * exp2f(-0.7213475204444817f * bcb) * is;  // exp(-bcb / 2)
}

// Events frames[0 .. n_frames) and then the *n_list events that the windowed
// kernels left to this one (list; both null without windows).
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
k_mlem(const GridF g, const GeometryDev geo, const float* __restrict__ sens,
       const Frame* __restrict__ frames, int64_t n_frames, const Frame* __restrict__ win_frames,
       const int32_t* __restrict__ list, const int32_t* __restrict__ n_list,
       const float* __restrict__ rho_t, float* acc_t, float* spill) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  WarpSmem& sm = reinterpret_cast<WarpSmem*>(smem_raw)[wib];
  float* slab = spill + ((int64_t)blockIdx.x * kWarps + wib) * kSpill;
  const float half_L = g.L / 2;
  // grid-stride over the events (in LOR order: the warps resident at one
  // time work on a few LORs, whose pixel infos and image lines stay in L2)
  const int64_t n_warps = (int64_t)gridDim.x * kWarps;
  const int64_t n_all = n_frames + (n_list ? *n_list : 0);
  for (int64_t e = (int64_t)blockIdx.x * kWarps + wib; e < n_all; e += n_warps) {
    const Frame f = e < n_frames ? frames[e] : win_frames[list[e - n_frames]];
    const int n_pix = f.info_end - f.info_begin;
    const int n_pl = f.plane_end - f.plane_begin;
    if (n_pix <= 0 || n_pl <= 0) continue;
    const float4 md = geo.lor_md[f.lor];
    const float R = geo.lor_len[f.lor] / 2;
    const int q = 32 / n_pl, r = 32 - q * n_pl;
    const int j0 = lane / n_pl, pz0 = lane - j0 * n_pl;
    // pass 1: weights and the denominator
    float d = 0.0f;
    for (int c0 = 0; c0 < n_pix; c0 += 32) {
      load_pixels(g, geo, sens, f, md, R, c0, n_pix, lane, sm.px);
      const int nv = min(32, n_pix - c0) * n_pl;
      const int base = c0 * n_pl;
      int j = j0, pz = pz0;
#pragma unroll kUnroll
      for (int v = lane; v < nv; v += 32) {
        const int iz = f.plane_begin + pz;
        // the image load goes out first; the kernel arithmetic hides it
        const float rho = __ldg(rho_t + sm.px.base[j] + iz);
        float wgt = voxel_kw(g, f, sm.px, j, iz, half_L);
        if (wgt != 0.0f) {
          wgt *= rho;
          d = fmaf(wgt, sm.px.t[j].w, d);
        }
        const int fv = base + v;
        if (fv < kCache)
          sm.cache[fv] = wgt;
        else if (fv < kCache + kSpill)
          slab[fv - kCache] = wgt;
        j += q;
        pz += r;
        if (pz >= n_pl) {
          pz -= n_pl;
          ++j;
        }
      }
      __syncwarp();
    }
    double dd = d;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dd += __shfl_xor_sync(0xffffffffu, dd, o);
    if (!(dd > 0.0)) continue;
    const float inv = (float)(1.0 / dd);
    // pass 2: scatter weight / D
    for (int c0 = 0; c0 < n_pix; c0 += 32) {
      const int base = c0 * n_pl;
      const int nv = min(32, n_pix - c0) * n_pl;
      if (base + nv <= kCache + kSpill) {
        if (c0 + lane < n_pix) {
          const short2 p = geo.pix[(int64_t)f.info_begin + c0 + lane];
          sm.px.base[lane] = (p.x + g.nc * p.y) * g.np;
        }
        __syncwarp();
      } else {
        load_pixels(g, geo, sens, f, md, R, c0, n_pix, lane, sm.px);
      }
      int j = j0, pz = pz0;
#pragma unroll kUnroll2
      for (int v = lane; v < nv; v += 32) {
        const int iz = f.plane_begin + pz;
        const int vi = sm.px.base[j] + iz;
        const int fv = base + v;
        float wgt;
        if (fv < kCache) {
          wgt = sm.cache[fv];
        } else if (fv < kCache + kSpill) {
          wgt = slab[fv - kCache];
        } else {
          const float rho = __ldg(rho_t + vi);
          wgt = voxel_kw(g, f, sm.px, j, iz, half_L) * rho;
        }
        if (wgt != 0.0f) atomicAdd(acc_t + vi, wgt * inv);
        j += q;
        pz += r;
        if (pz >= n_pl) {
          pz -= n_pl;
          ++j;
        }
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------
// Windowed MLEM.  Within a LOR everything per voxel but the event's Gaussian
// -- the pixel weight, the angular sensitivity, the image -- depends on
// (pixel info, plane) only.  So the work is cut into tasks of 64 consecutive
// pixel infos x the planes of the events of one LOR and plane slab; a warp
// owns a task: it computes V = w / sens(z, up) * rho once per window entry
// into shared memory, and walks all events of the slab that touch its infos.
// What remains per event and voxel is the Gaussian along z, advanced by the
// two-multiply recurrence E <- E S, S <- S q from the event's middle plane
// both ways (the error grows with the distance from the anchor, where the
// values are smallest); a lane holds two neighbouring infos, so one 8-byte
// shared load and packed f32x2 arithmetic serve both.
//   k_win_project  D_e partials of the task's infos: binary32 per lane,
//                  binary64 across lanes and (global reductions) tasks
//   k_win_invert   1 / D_e, and the list of events left to k_mlem
//   k_win_back     acc[plane][info] += E c / sqrt(a'Sa) / D_e in binary32:
//                  the warp owns its entries, so plain read-modify-writes
//                  replace atomics; then acc * V goes to the volume with one
//                  reduction per touched entry instead of one per event and
//                  voxel
// Big barrel, 1e7 responses (3.58e10 voxels), ms per iteration: k_mlem 205
// (144 thread instructions a voxel), this 32.3 (20; issue-active 67 / 62 %,
// packed multiplies 52 / 44 % of the FMA pipe; a quarter of the instructions
// compute V).  Two kernels around D_e, not one CTA per window with barriers:
// the infos of an event span three or four warps whose loads differ with the
// events' positions, and a barrier-synchronised form issued 33 % of the time
// (66 ms).  Also measured: V's arithmetic one row at a time 36.7; two events
// of the same middle plane walked together 32.6 (fewer shared loads, but the
// set-up per event and V are what is left).
//
// Events outside the safe range of the recurrence (an anchor exponent below
// 2^-100, D_e outside [1e-25, 1e25] or not finite) go to `list` and k_mlem
// evaluates them voxel by voxel, so dropped and extreme events stay what they
// were.
constexpr int kWinStride = 66;  // words between planes: 64 infos + 2 (lane =
                                // plane stores of row pairs hit all banks)
constexpr int kWinWarps = 4;  // per CTA (they share nothing)
constexpr int kWinCtas = 4;   // per SM
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsq(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }

struct WinConst {
  float c1, r1, r0, q;  // the Gaussian along z at the plane pitch
};
__device__ __forceinline__ WinConst win_const(const GridF& g) {
  WinConst k;
  k.c1 = -kLog2e * g.ipz;
  k.r1 = 2.0f * k.c1 * g.p;
  k.r0 = k.c1 * g.p * g.p;
  k.q = exp2f(2.0f * k.c1 * g.p * g.p);
  return k;
}

// The frame events' window form (WinEvent in hybrid_internal.h).
__global__ void k_win_events(const GridF g, const GeometryDev geo,
                             const Frame* __restrict__ frames, int32_t n, WinEvent* out) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Frame f = frames[i];
    const float R = geo.lor_len[f.lor] / 2;
    const int planes = f.plane_end - f.plane_begin, pm = f.plane_begin + (planes >> 1);
    const float s2 = f.sec * f.sec, s4 = s2 * s2;
    WinEvent v;
    v.up = f.up;
    v.tan = f.tan;
    v.zc = plane_z(g, pm) - f.right;
    v.cd = -2.0f * kLog2e * g.ipdl * s2;
    v.na = 2.0f * g.ipz * s4 + 4.0f * g.ipdl * s2 * (f.tan * f.tan);
    v.nb = 2.0f * g.ipz * s4 * (R * R);
    v.info_begin = f.info_begin;
    v.shape = (unsigned)(f.info_end - f.info_begin) | (unsigned)planes << kWinRowBits |
              (unsigned)pm << (kWinRowBits + kWinPlaneBits);
    out[i] = v;
  }
}

// A lane's two infos of a task: constants of the LOR's pixels.
struct WinRows {
  float2 upp, upp2, ra, rb, w, s;
  int g0, g1;  // z-fast index of the window's first plane
};

__device__ __forceinline__ WinRows win_load_rows(const GridF& g, const GeometryDev& geo,
                                                 const float* __restrict__ sens,
                                                 int lor, int row0, int n_rows, int p0,
                                                 int lane) {
  WinRows r;
  r.upp = r.ra = r.rb = r.w = r.s = make_float2(0.0f, 0.0f);
  r.g0 = r.g1 = 0;
  const float4 md = geo.lor_md[lor];
  const float R = geo.lor_len[lor] / 2;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (2 * lane + h < n_rows) {
      const int64_t info = (int64_t)row0 + 2 * lane + h;
      const short2 p = geo.pix[info];
      const int pidx = p.x + g.nc * p.y;
      const float u = proj_up(g, p, md), wt = geo.w[info], sv = sens[pidx];
      const float a = __frcp_rn(R - u), b = __frcp_rn(R + u);
      if (h == 0) {
        r.upp.x = u; r.w.x = wt; r.s.x = sv; r.ra.x = a; r.rb.x = b;
        r.g0 = pidx * g.np + p0;
      } else {
        r.upp.y = u; r.w.y = wt; r.s.y = sv; r.ra.y = a; r.rb.y = b;
        r.g1 = pidx * g.np + p0;
      }
    }
  }
  r.upp2 = __fmul2_rn(r.upp, r.upp);
  return r;
}

__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// inv_sens of two pixels at the plane with half_L - z = lm and half_L + z =
// lp, times m: atan2_pos in packed arithmetic (the same coefficients).
__device__ __forceinline__ float2 inv_sens2(float lm, float lp, float2 ra, float2 rb, float2 m) {
  constexpr float kAtan[8] = {-0.0040545654483139515f, 0.021862952038645744f, -0.0559123195707798f, 0.0964219719171524f,
                              -0.1390862911939621f, 0.19946566224098206f, -0.33329859375953674f, 0.9999993443489075f};
  const float2 x0 = __fmul2_rn(dup(lm), ra), x1 = __fmul2_rn(dup(lp), rb);
  const float2 y0 = __fmul2_rn(dup(-lp), ra), y1 = __fmul2_rn(dup(-lm), rb);
  const float2 u = make_float2(fminf(x0.x, x1.x), fminf(x0.y, x1.y));
  const float2 v = make_float2(fmaxf(y0.x, y1.x), fmaxf(y0.y, y1.y));
  const float2 a = __fadd2_rn(u, make_float2(-v.x, -v.y));
  const float2 b = __ffma2_rn(u, v, dup(1.0f));
  const float2 ab = make_float2(fabsf(b.x), fabsf(b.y));
  const float2 t = __fmul2_rn(make_float2(fminf(a.x, ab.x), fminf(a.y, ab.y)),
                              make_float2(rcp(fmaxf(a.x, ab.x)), rcp(fmaxf(a.y, ab.y))));
  const float2 s = __fmul2_rn(t, t);
  float2 p = dup(kAtan[0]);
#pragma unroll
  for (int i = 1; i < 8; ++i) p = __ffma2_rn(p, s, dup(kAtan[i]));
  float2 r = __fmul2_rn(t, p);
  if (a.x > ab.x) r.x = 1.5707963267948966f - r.x;
  if (a.y > ab.y) r.y = 1.5707963267948966f - r.y;
  if (b.x < 0.0f) r.x = 3.14159265358979f - r.x;
  if (b.y < 0.0f) r.y = 3.14159265358979f - r.y;
  const float2 o = __fmul2_rn(__fmul2_rn(m, dup(3.14159265358979f)),
                              make_float2(rcp(r.x), rcp(r.y)));
  return make_float2(a.x > 0.0f ? o.x : 0.0f, a.y > 0.0f ? o.y : 0.0f);
}

// Calls f(L, p, V of infos 2 L and 2 L + 1, their image indices) for the
// entries of planes [p0, p1) of the window, lanes along the planes (coalesced
// image accesses).
template <class F>
__device__ __forceinline__ void win_entries(const GridF& g, const WinRows& r, int p0, int n_pl,
                                            int n_rows, const float* __restrict__ rho_t, int lane,
                                            F&& f) {
  const float half_L = g.L / 2;
#pragma unroll 2
  for (int L = 0; 2 * L < n_rows; ++L) {
    const float2 ra = make_float2(__shfl_sync(~0u, r.ra.x, L), __shfl_sync(~0u, r.ra.y, L));
    const float2 rb = make_float2(__shfl_sync(~0u, r.rb.x, L), __shfl_sync(~0u, r.rb.y, L));
    const float2 w = make_float2(__shfl_sync(~0u, r.w.x, L), __shfl_sync(~0u, r.w.y, L));
    const int g0 = __shfl_sync(~0u, r.g0, L);
    // an odd window's last pair reads the same pixel twice; its weight is 0
    const int g1 = 2 * L + 1 < n_rows ? __shfl_sync(~0u, r.g1, L) : g0;
    for (int p = lane; p < n_pl; p += 32) {
      const float2 x = make_float2(__ldg(rho_t + g0 + p), __ldg(rho_t + g1 + p));
      const float z = plane_z(g, p0 + p);
      f(L, p, __fmul2_rn(inv_sens2(half_L - z, half_L + z, ra, rb, w), x), g0 + p, g1 + p);
    }
  }
}

// The rows' Gaussian constants of an event: K (with 1 / sqrt(a'Sa)) at the
// anchor plane, its ratios upwards and downwards; arg: the exponents.
__device__ __forceinline__ void win_gauss(const WinConst& k, const WinEvent& e, const WinRows& r,
                                          float2& K, float2& Su, float2& Sd, float2& arg) {
  const float2 dy = __fadd2_rn(r.upp, dup(-e.up));
  const float2 t = __ffma2_rn(dy, dup(-e.tan), dup(e.zc));
  const float2 norm = __ffma2_rn(r.upp2, dup(e.na), dup(e.nb));
  arg = __ffma2_rn(__fmul2_rn(t, dup(k.c1)), t, __fmul2_rn(__fmul2_rn(dy, dup(e.cd)), dy));
  const float2 au = __ffma2_rn(t, dup(k.r1), dup(k.r0));
  const float2 ad = __ffma2_rn(t, dup(-k.r1), dup(k.r0));
  K = __fmul2_rn(make_float2(rsq(norm.x), rsq(norm.y)), make_float2(ex2(arg.x), ex2(arg.y)));
  Su = make_float2(ex2(au.x), ex2(au.y));
  Sd = make_float2(ex2(ad.x), ex2(ad.y));
}

// The event's share of a task: rows [rb, re) of the 64, anchor plane pm
// (window-relative), nd planes below it and nu from it on.
struct WinSpan {
  int rb, re, pm, nd, nu;
};
__device__ __forceinline__ WinSpan win_span(const WinEvent& e, int row0, int p0) {
  WinSpan s;
  s.rb = e.info_begin - row0;
  s.re = s.rb + (int)(e.shape & ((1u << kWinRowBits) - 1));
  const int planes = (int)((e.shape >> kWinRowBits) & ((1u << kWinPlaneBits) - 1));
  s.pm = (int)(e.shape >> (kWinRowBits + kWinPlaneBits)) - p0;
  s.nd = planes >> 1;
  s.nu = planes - s.nd;
  return s;
}

// Walks the item's events 32 at a time (each lane loads one into the warp's
// shared copy) and calls f(event index, event, its lane) for those that touch
// rows [row0, row0 + 64) and whose `use` is non-zero.
template <class Use, class F>
__device__ __forceinline__ void win_walk(const WinEvent* __restrict__ events, const WinItem& it,
                                         int row0, WinEvent* s_ev, int lane, Use&& use, F&& f) {
  for (int eb = it.e0; eb < it.e1; eb += 32) {
    bool hit = false;
    __syncwarp();  // the previous block's events are done with
    if (eb + lane < it.e1) {
      const WinEvent v = events[eb + lane];
      const int rb = v.info_begin - row0;
      hit = rb < 64 && rb + (int)(v.shape & ((1u << kWinRowBits) - 1)) > 0 && use(eb + lane);
      s_ev[lane] = v;
    }
    unsigned todo = __ballot_sync(~0u, hit);
    __syncwarp();
    for (; todo; todo &= todo - 1) {
      const int j = __ffs(todo) - 1;
      f(eb + j, s_ev[j], j);
    }
  }
}

struct WinArgs {
  GridF g;
  GeometryDev geo;
  const float* sens;
  const WinEvent* events;
  const WinItem* items;
  const WinTask* tasks;
  int n_tasks;
  int planes;         // of a window buffer
  int* counter;       // next task
  const float* rho_t;
  double* D;          // per event
  const float* inv;   // per event, k_win_back
  float* acc_t;
};

__device__ __forceinline__ int next_task(int* counter, int lane) {
  int t = 0;
  if (lane == 0) t = atomicAdd(counter, 1);
  return __shfl_sync(~0u, t, 0);
}

// Adds the lanes' sums of the n (<= 8) events in s_red[event][33] into D of
// the events' ids (event i's in lanes 4 i .. 4 i + 3).
__device__ __forceinline__ void win_reduce(const float* s_red, int n, int id, int lane,
                                           double* D) {
  __syncwarp();
  const float* v = s_red + (lane >> 2) * 33 + (lane & 3) * 8;
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) s += (double)v[i];
  s += __shfl_xor_sync(~0u, s, 1);
  s += __shfl_xor_sync(~0u, s, 2);
  if ((lane & 3) == 0 && (lane >> 2) < n) atomicAdd(D + id, s);
  __syncwarp();
}

__global__ void __launch_bounds__(32 * kWinWarps, kWinCtas)
k_win_project(const __grid_constant__ WinArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  WinEvent* s_ev = reinterpret_cast<WinEvent*>(smem_raw) + 32 * w;
  float* s_red = reinterpret_cast<float*>(smem_raw + kWinWarps * 32 * sizeof(WinEvent)) +
                 8 * 33 * w;
  float* win = reinterpret_cast<float*>(smem_raw + kWinWarps * 32 * sizeof(WinEvent)) +
               kWinWarps * 8 * 33 + w * a.planes * kWinStride;
  const WinConst k = win_const(a.g);
  const float2 Q = dup(k.q);
  const float* const mine = win + 2 * lane;
  for (;;) {
    const int t = next_task(a.counter, lane);
    if (t >= a.n_tasks) break;
    const WinTask task = a.tasks[t];
    const WinItem it = a.items[task.item];
    const int row0 = task.row0, p0 = task.p0, n_pl = task.p1 - task.p0;
    const int n_rows = min(64, it.i1 - row0);
    const WinRows r = win_load_rows(a.g, a.geo, a.sens, it.lor, row0, n_rows, p0, lane);
    __syncwarp();  // the previous task's window is done with
    win_entries(a.g, r, p0, n_pl, n_rows, a.rho_t, lane,
                [&](int L, int p, float2 V, int, int) {
                  *reinterpret_cast<float2*>(win + p * kWinStride + 2 * L) = V;
                });
    __syncwarp();
    int n_red = 0, red_id = 0;  // events in s_red; the one this lane adds up
    win_walk(a.events, it, row0, s_ev, lane, [](int) { return true; },
             [&](int ei, const WinEvent& e, int) {
      const WinSpan s = win_span(e, row0, p0);
      float2 K, Su, Sd, arg;
      win_gauss(k, e, r, K, Su, Sd, arg);
      float2 Pu = K, Pd = __fmul2_rn(K, Sd);
      Sd = __fmul2_rn(Sd, Q);
      float2 A = make_float2(0.0f, 0.0f), B = A;
      const float* au = mine + s.pm * kWinStride;
      const float* ad = au - kWinStride;
#pragma unroll 2
      for (int j = 0; j < s.nd; ++j, au += kWinStride, ad -= kWinStride) {
        A = __ffma2_rn(Pu, *reinterpret_cast<const float2*>(au), A);
        B = __ffma2_rn(Pd, *reinterpret_cast<const float2*>(ad), B);
        Pu = __fmul2_rn(Pu, Su);
        Pd = __fmul2_rn(Pd, Sd);
        Su = __fmul2_rn(Su, Q);
        Sd = __fmul2_rn(Sd, Q);
      }
      if (s.nu > s.nd) A = __ffma2_rn(Pu, *reinterpret_cast<const float2*>(au), A);
      A = __fadd2_rn(A, B);
      // rows of other events hold garbage: select, do not multiply by zero
      const int r0 = 2 * lane;
      const bool in0 = r0 >= s.rb && r0 < s.re, in1 = r0 + 1 >= s.rb && r0 + 1 < s.re;
      float d = in0 ? A.x * r.s.x : 0.0f;
      if (in1) d = fmaf(A.y, r.s.y, d);
      if ((in0 && !(arg.x > -100.0f)) || (in1 && !(arg.y > -100.0f))) d = NAN;
      // the lanes' sums wait in shared memory until eight events can be
      // added up together, four lanes each (five double shuffles per event
      // otherwise)
      s_red[n_red * 33 + lane] = d;
      if ((lane >> 2) == n_red) red_id = ei;
      if (++n_red == 8) {
        win_reduce(s_red, 8, red_id, lane, a.D);
        n_red = 0;
      }
    });
    win_reduce(s_red, n_red, red_id, lane, a.D);
  }
}

// inv_e = c / D_e (0: no scatter here); D_e <- 0 for the next iteration.
__global__ void k_win_invert(double* D, int32_t n, float norm_c, float* inv, int32_t* list,
                             int32_t* n_list) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double d = D[i], Dn = d * (double)norm_c;
    D[i] = 0.0;
    const bool safe = Dn > 1e-25 && Dn < 1e25;
    inv[i] = safe ? (float)(1.0 / d) : 0.0f;
    if (!safe) list[atomicAdd(n_list, 1)] = i;
  }
}

__global__ void __launch_bounds__(32 * kWinWarps, kWinCtas)
k_win_back(const __grid_constant__ WinArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  WinEvent* s_ev = reinterpret_cast<WinEvent*>(smem_raw) + 32 * w;
  float* win = reinterpret_cast<float*>(smem_raw + kWinWarps * 32 * sizeof(WinEvent)) +
               w * a.planes * kWinStride;
  const WinConst k = win_const(a.g);
  const float2 Q = dup(k.q);
  float* const mine = win + 2 * lane;
  for (;;) {
    const int t = next_task(a.counter, lane);
    if (t >= a.n_tasks) break;
    const WinTask task = a.tasks[t];
    const WinItem it = a.items[task.item];
    const int row0 = task.row0, p0 = task.p0, n_pl = task.p1 - task.p0;
    const int n_rows = min(64, it.i1 - row0);
    const WinRows r = win_load_rows(a.g, a.geo, a.sens, it.lor, row0, n_rows, p0, lane);
    __syncwarp();  // the previous task's window is flushed
    for (int p = 0; p < n_pl; ++p)
      *reinterpret_cast<float2*>(mine + p * kWinStride) = make_float2(0.0f, 0.0f);
    float my_inv = 0.0f;
    win_walk(a.events, it, row0, s_ev, lane,
             [&](int ei) {
               my_inv = a.inv[ei];
               return my_inv != 0.0f;
             },
             [&](int, const WinEvent& e, int j) {
      const WinSpan s = win_span(e, row0, p0);
      const float inv = __shfl_sync(~0u, my_inv, j);
      float2 K, Su, Sd, arg;
      win_gauss(k, e, r, K, Su, Sd, arg);
      // rows of other events: zeros throughout (their ratios may be inf)
      const int r0 = 2 * lane;
      const bool in0 = r0 >= s.rb && r0 < s.re, in1 = r0 + 1 >= s.rb && r0 + 1 < s.re;
      K = make_float2(in0 ? K.x * inv : 0.0f, in1 ? K.y * inv : 0.0f);
      Su = make_float2(in0 ? Su.x : 0.0f, in1 ? Su.y : 0.0f);
      Sd = make_float2(in0 ? Sd.x : 0.0f, in1 ? Sd.y : 0.0f);
      float2 Pu = K, Pd = __fmul2_rn(K, Sd);
      Sd = __fmul2_rn(Sd, Q);
      float* au = mine + s.pm * kWinStride;
      float* ad = au - kWinStride;
#pragma unroll 2
      for (int i = 0; i < s.nd; ++i, au += kWinStride, ad -= kWinStride) {
        float2* xu = reinterpret_cast<float2*>(au);
        float2* xd = reinterpret_cast<float2*>(ad);
        const float2 yu = *xu, yd = *xd;
        *xu = __fadd2_rn(yu, Pu);
        *xd = __fadd2_rn(yd, Pd);
        Pu = __fmul2_rn(Pu, Su);
        Pd = __fmul2_rn(Pd, Sd);
        Su = __fmul2_rn(Su, Q);
        Sd = __fmul2_rn(Sd, Q);
      }
      if (s.nu > s.nd) {
        float2* xu = reinterpret_cast<float2*>(au);
        *xu = __fadd2_rn(*xu, Pu);
      }
    });
    __syncwarp();
    win_entries(a.g, r, p0, n_pl, n_rows, a.rho_t, lane,
                [&](int L, int p, float2 V, int i0, int i1) {
                  const float2 x =
                      *reinterpret_cast<const float2*>(win + p * kWinStride + 2 * L);
                  const float c0 = x.x != 0.0f ? x.x * V.x : 0.0f;
                  const float c1 = x.y != 0.0f ? x.y * V.y : 0.0f;
                  if (c0 != 0.0f) atomicAdd(a.acc_t + i0, c0);
                  if (c1 != 0.0f) atomicAdd(a.acc_t + i1, c1);
                });
  }
}

// Boundary layout (x fastest, plane slowest) <-> z-fast layout.
__global__ void k_to_zfast(const GridF g, const float* __restrict__ rho, float* rho_t) {
  const int64_t n = (int64_t)g.n_pixels * g.np;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pidx = i % g.n_pixels, z = i / g.n_pixels;
    rho_t[pidx * g.np + z] = rho[i];
  }
}

__global__ void k_from_zfast(const GridF g, const float* __restrict__ rho_t, float* rho) {
  const int64_t n = (int64_t)g.n_pixels * g.np;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pidx = i % g.n_pixels, z = i / g.n_pixels;
    rho[i] = rho_t[pidx * g.np + z];
  }
}

// Totals of the frame events' pixel infos and voxels (out[0], out[1]) and the
// largest event's (out[2] infos, out[3] planes).
__global__ void k_event_counts(const Frame* __restrict__ frames, int64_t n,
                               unsigned long long* out) {
  unsigned long long a = 0, b = 0;
  int mr = 0, mp = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Frame f = frames[i];
    const int np = f.info_end - f.info_begin, nz = f.plane_end - f.plane_begin;
    a += np > 0 ? np : 0;
    b += (np > 0 && nz > 0) ? (unsigned long long)np * nz : 0ull;
    mr = max(mr, np);
    mp = max(mp, nz);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    mr = max(mr, __shfl_xor_sync(0xffffffffu, mr, o));
    mp = max(mp, __shfl_xor_sync(0xffffffffu, mp, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out, a);
    atomicAdd(out + 1, b);
    atomicMax(out + 2, (unsigned long long)mr);
    atomicMax(out + 3, (unsigned long long)mp);
  }
}

int grid_for(int64_t n) {
  const int64_t b = (n + 255) / 256;
  return (int)(b < 148 * 32 ? (b > 0 ? b : 1) : 148 * 32);
}

}  // namespace

int mlem_blocks_per_sm() { return kBlocksPerSm; }

void launch_to_zfast(const GridF& g, const float* rho, float* rho_t, cudaStream_t st) {
  k_to_zfast<<<grid_for((int64_t)g.n_pixels * g.np), 256, 0, st>>>(g, rho, rho_t);
}

void launch_from_zfast(const GridF& g, const float* rho_t, float* rho, cudaStream_t st) {
  k_from_zfast<<<grid_for((int64_t)g.n_pixels * g.np), 256, 0, st>>>(g, rho_t, rho);
}

size_t mlem_spill_floats(int n_blocks) { return (size_t)n_blocks * kWarps * kSpill; }

void launch_mlem(const GridF& g, const GeometryDev& geo, const float* sens, const Frame* frames,
                 int64_t n_frames, const Frame* win_frames, const int32_t* list,
                 const int32_t* n_list, const float* rho_t, float* acc_t, float* spill,
                 int n_blocks, cudaStream_t st) {
  const int smem = (int)sizeof(WarpSmem) * kWarps;
  cudaFuncSetAttribute(k_mlem, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k_mlem<<<n_blocks, kThreads, smem, st>>>(g, geo, sens, frames, n_frames, win_frames, list,
                                           n_list, rho_t, acc_t, spill);
}

namespace {
int win_smem(int planes) {
  return kWinWarps * (32 * (int)sizeof(WinEvent) + 8 * 33 * (int)sizeof(float) +
                      planes * kWinStride * (int)sizeof(float));
}
}  // namespace

WinPlan plan_windows(const GridF& g, int max_planes) {
  WinPlan w{};
  const float sz = 1.0f / sqrtf(g.ipz);
  // the recurrence's ratios stay finite up to planes of 4 sigma_z; the event
  // words hold kWinPmBits of plane index
  if (max_planes <= 0 || !(g.p <= 4.0f * sz) || g.np >= (1 << kWinPmBits)) return w;
  const int budget = (233472 / kWinCtas - 1024) / kWinWarps;
  int planes = (budget - win_smem(0) / kWinWarps) / (kWinStride * (int)sizeof(float));
  planes = std::min(planes, std::min(64, (int)g.np));
  w.planes = planes;
  w.max_planes = planes >= g.np ? planes : std::min(max_planes, planes - 4);
  w.tile_planes = planes >= g.np ? g.np : planes - w.max_planes + 1;
  w.n_slabs = g.np / w.tile_planes + 1;
  return w;
}

void launch_win_events(const GridF& g, const GeometryDev& geo, const Frame* frames, int32_t n,
                       WinEvent* out, cudaStream_t st) {
  k_win_events<<<grid_for(n), 256, 0, st>>>(g, geo, frames, n, out);
}

void launch_mlem_win(const GridF& g, const GeometryDev& geo, const float* sens,
                     const WinSet& ws, const float* rho_t, float* acc_t, int n_sm,
                     cudaStream_t st) {
  WinArgs a{};
  a.g = g;
  a.geo = geo;
  a.sens = sens;
  a.events = ws.events;
  a.items = ws.items;
  a.tasks = ws.tasks;
  a.n_tasks = ws.n_tasks;
  a.planes = ws.plan.planes;
  a.rho_t = rho_t;
  a.D = ws.D;
  a.inv = ws.inv;
  a.acc_t = acc_t;
  const int smem = win_smem(ws.plan.planes);
  cudaFuncSetAttribute(k_win_project, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaFuncSetAttribute(k_win_back, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const int grid = std::min((ws.n_tasks + kWinWarps - 1) / kWinWarps, n_sm * kWinCtas);
  a.counter = ws.counters;
  k_win_project<<<grid, 32 * kWinWarps, smem, st>>>(a);
  k_win_invert<<<grid_for(ws.n_events), 256, 0, st>>>(ws.D, ws.n_events, g.norm_c, ws.inv, ws.list,
                                                    ws.counters + 2);
  a.counter = ws.counters + 1;
  k_win_back<<<grid, 32 * kWinWarps, smem, st>>>(a);
}

void launch_event_counts(const Frame* frames, int64_t n, unsigned long long* out4,
                         cudaStream_t st) {
  cudaMemsetAsync(out4, 0, 4 * sizeof(unsigned long long), st);
  k_event_counts<<<grid_for(n), 256, 0, st>>>(frames, n, out4);
}

namespace {
// The kernel's arctangent (which = 0) or CUDA's atan2f (which = 1) on n
// argument pairs: the test hook that bounds atan2_pos's error.
__global__ void k_atan2_probe(const float* a, const float* b, int64_t n, int which,
                              float* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = which == 0 ? atan2_pos(a[i], b[i]) : atan2f(a[i], b[i]);
}
}  // namespace

cudaError_t launch_atan2_probe(const float* a, const float* b, int64_t n, int which,
                               float* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_atan2_probe<<<grid_for(n), 256, 0, st>>>(a, b, n, which, out);
  return cudaGetLastError();
}

}  // namespace hybridmlem
