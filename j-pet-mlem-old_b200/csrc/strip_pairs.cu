// The tile kernels of the GaussianKernel over column-major windows (MLEM,
// forward, adjoint, sigma gradient): row pairs in packed f32x2 arithmetic.
//
// An event is worked on by a group of LPE lanes (8 or 16: four or two events
// per warp).  Its box rows are paired from the middle out -- rows mid + k and
// mid - 1 - k -- and lane l of the group owns, in block b, pair LPE b + l.
// The two rows of a pair lie symmetrically about the event's centre, so their
// runs are equally long to within a pixel or two, and everything about them is
// one f32x2 operation: the exact set arithmetic, the closed-form run ends,
// the kernel constants, and the walks E <- E R, R <- R q (a step is one pixel
// of each row).  Bound by instruction issue (79 % issue-active, the FMA pipe at
// 51 %, the shared-memory pipe at 61 %).  With one row per lane the set-up of the
// rows was a third of the MLEM kernel; warp instructions an event at the 800 x
// 400 benchmark 928 -> 767, 4e6 events 4.39 -> 3.47 ms a pass (forward 2.31 -> 1.93, adjoint 2.65 ->
// 2.22).  Sixteen lanes an event issue more (943; they serve boxes above 80
// rows), and 384 threads of 80 registers without spills run slower (4.1 ms).
//
// Exactness.  The pixel sets are decided by binary32 operations rounded one by
// one (strip_device.cuh).  ptxas fuses a packed multiply and a packed add into
// a fused multiply-add even where both say .rn, so the exact products are
// written as fma(a, b, -0) with a -0 that the compiler cannot see
// (PairConst::nzero): a * b rounded once, whatever follows.
//
// Accuracy.  q (the ratio of neighbouring ratios) would enter pixel j of a run
// with its rounding error times j (j - 1) / 2.  The ratios advance by
// R <- R + R (q - 1), one fused operation with q - 1 rounded: the error is
// smaller by |q - 1| (0.08 at sigma_z = 5 pixels).  Below q = 1/2 it is larger,
// and steep sigmas go to k_tile (pair_const_ok).  (Not in the sigma gradient,
// which keeps the one-row kernel's steps.)
//
// Backprojection window: unsigned 32-bit fixed point as in strip_kernels.cu
// (fixed_shift and the unweighted windows of strip_internal.h).  An addend
// below 2^24 is converted by multiplying with 2^-149: the bits of the
// subnormal product are the addend rounded to an integer, so the conversion of
// two pixels is one packed multiply (denormals run at full rate) instead of
// two conversions on the quarter-rate pipe.  Items of few events, whose
// addends are larger, take cvt.rni.
#include <algorithm>
#include <type_traits>

#include "strip_internal.h"
#include "strip_kernel_eval.cuh"
#include "strip_rows.cuh"
#include "strip_tile.cuh"

namespace stripmlem {

namespace {

constexpr int kPairThreads = 512;
constexpr int kPairWide = 2 * kPairThreads;  // one CTA per SM
// Steps a turn of the walks' loops: four, but two for the MLEM kernel's sums
// (4e6 events at the 800 x 400 benchmark: 3.42 ms a pass against 3.60 with
// four; eight everywhere 3.97, one 4.38).
constexpr int kUnroll = 4;
__host__ __device__ constexpr int sum_unroll(int op) { return op == OP_MLEM ? 2 : kUnroll; }

__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }
// a * b, rounded, never fused with what follows
__device__ __forceinline__ float2 xmul(float2 a, float2 b, float2 nzero) {
  return __ffma2_rn(a, b, nzero);
}

// An event's constants over its rows.
struct PairEvent {
  float A, B;            // of the exact set arithmetic
  float ny, nz;          // -y, -z
  float tan, tanp, x0;   // tan, tan / pw, centre column
  float nk4;             // hw^2 = c9 + nk4 dy^2 (pixels^2)
  float na, nb, cd;      // GaussEvent, norm in units of kc^2
  float cmin, cend;      // box columns [cmin, cend)
  float fm;              // row of pair 0's lower row (mid), as float
  int n_a, n_b;          // rows of the two sides: pairs k < n_a, k < n_b
  int row_a;             // mid - wy0
};

__device__ __forceinline__ PairEvent pair_event(const ScannerF& s, const PairConst& c,
                                                const EventPack& m, int wy0) {
  PairEvent e;
  const int tlx = m.x & 0xFFFF, brx = m.x >> 16, tly = m.yb & 0xFFFF, bry = m.yb >> 16;
  const int H = bry > tly && brx > tlx ? bry - tly : 0;
  const int mid = tly + (H >> 1);
  e.n_a = H - (H >> 1);
  e.n_b = H >> 1;
  e.row_a = mid - wy0;
  e.fm = (float)mid;
  e.cmin = (float)tlx;
  e.cend = (float)brx;
  // gaussian_kernel.h:120-122, as event_setup
  const float tt = __fmul_rn(m.tan, m.tan);
  e.A = __fadd_rn(__fmul_rn(__fmul_rn(__fmul_rn(4.0f, m.sec), m.sec), s.ipsdl),
                  __fmul_rn(__fmul_rn(2.0f, tt), s.ipsz));
  e.B = __fmul_rn(__fmul_rn(-4.0f, m.tan), s.ipsz);
  e.ny = -m.y;
  e.nz = -m.z;
  e.tan = m.tan;
  e.tanp = m.tan * s.inv_pw;
  e.x0 = (m.z - s.tl_z_half_w) * s.inv_pw;
  const float s2 = m.sec * m.sec, s4 = s2 * s2;
  e.nk4 = s2 * c.nk4;
  e.na = fmaf(c.na4, s4, c.na2 * s2 * tt);
  e.nb = c.nb4 * s4;
  e.cd = c.cd * s2;
  return e;
}

// A pair of rows: the Gaussians' first values and ratios, and the runs packed
// as col_a | len_a << 8 | col_b << 16 | len_b << 24 (window columns; windows
// are at most 225 columns wide).
struct PairRow {
  float2 K0, R0;
  unsigned run;
  float2 dy, lo;  // sigma gradient: the rows' distances from y, the runs' first columns
};

// Pair k of the event, f32x2 = (row mid + k, row mid - 1 - k).
template <bool GRAD = false>
__device__ __forceinline__ PairRow pair_row(const ScannerF& s, const PairConst& c,
                                            const PairEvent& e, int k, float mw) {
  const float kf = (float)k;
  const float2 nzero = dup(c.nzero);
  const float2 iy = __fadd2_rn(make_float2(e.fm, e.fm - 1.0f), make_float2(kf, -kf));
  // row_set (strip_device.cuh), exact
  const float2 py = __fadd2_rn(dup(s.tl_y_half_h), xmul(iy, dup(-s.ph), nzero));
  const float2 dy = __fadd2_rn(py, dup(e.ny));
  const float2 Ady2 = xmul(xmul(dup(e.A), dy, nzero), dy, nzero);
  const float2 Bdy = xmul(dup(e.B), dy, nzero);
  // the closed-form ends (row_run, strip_rows.cuh)
  const float2 dd = __fmul2_rn(dy, dy);
  const float2 u = __ffma2_rn(dup(e.nk4), dd, dup(c.c9));
  const float2 hw = make_float2(sqrt_approx(fmaxf(u.x, 0.0f)), sqrt_approx(fmaxf(u.y, 0.0f)));
  float2 xv = __ffma2_rn(dup(e.tanp), dy, dup(e.x0));
  // a centre far left of the box, or NaN: an empty row either way (the
  // ellipse cannot reach the box from there); far right or inf ends empty
  xv = make_float2(fmaxf(xv.x, -1e5f), fmaxf(xv.y, -1e5f));
  const float2 M = dup(12582912.0f), nM = dup(-12582912.0f);
  const float2 ml = __fadd2_rn(__fadd2_rn(__ffma2_rn(hw, dup(-1.0f), xv), M), nM);
  const float2 mh = __fadd2_rn(__fadd2_rn(__fadd2_rn(xv, hw), M), nM);
  auto q_at = [&](float2 col) {  // row_q of the pixel column, exact
    const float2 pz = __fadd2_rn(dup(s.tl_z_half_w), xmul(col, dup(s.pw), nzero));
    const float2 dz = __fadd2_rn(pz, dup(e.nz));
    return __fadd2_rn(__fadd2_rn(Ady2, xmul(Bdy, dz, nzero)),
                      xmul(xmul(dup(c.C), dz, nzero), dz, nzero));
  };
  const float2 ql = q_at(ml), qh = q_at(mh);
  float2 lo = make_float2(ql.x <= 9.0f ? ml.x : ml.x + 1.0f, ql.y <= 9.0f ? ml.y : ml.y + 1.0f);
  float2 end = make_float2(qh.x <= 9.0f ? mh.x + 1.0f : mh.x, qh.y <= 9.0f ? mh.y + 1.0f : mh.y);
  lo = make_float2(fmaxf(lo.x, e.cmin), fmaxf(lo.y, e.cmin));
  end = make_float2(fminf(end.x, e.cend), fminf(end.y, e.cend));
  const float2 len = __ffma2_rn(lo, dup(-1.0f), end);
  // col | len << 8 in the mantissa: 2^23 + (lo - wx0) + 256 len
  const float2 bits = __ffma2_rn(len, dup(256.0f), __fadd2_rn(lo, dup(mw)));
  PairRow r;
  const unsigned ra = len.x >= 1.0f && k < e.n_a ? __float_as_uint(bits.x) : 0u;
  const unsigned rb = len.y >= 1.0f && k < e.n_b ? __float_as_uint(bits.y) : 0u;
  r.run = __byte_perm(ra, rb, 0x5410);
  // kernel constants (GaussEvent::row)
  const float2 t0 = __fadd2_rn(__ffma2_rn(lo, dup(s.pw), dup(s.tl_z_half_w)), dup(e.nz));
  const float2 t = __ffma2_rn(dy, dup(-e.tan), t0);
  const float2 yp = __fadd2_rn(dy, dup(-e.ny));
  const float2 norm = __ffma2_rn(dup(e.na), __fmul2_rn(yp, yp), dup(e.nb));
  const float2 arg = __ffma2_rn(__fmul2_rn(dup(c.c1), t), t, __fmul2_rn(dup(e.cd), dd));
  const float2 ar = __ffma2_rn(t, dup(c.r1), dup(c.r0));
  r.K0 = __fmul2_rn(make_float2(rsqrt_approx(norm.x), rsqrt_approx(norm.y)),
                    make_float2(ex2_approx(arg.x), ex2_approx(arg.y)));
  r.R0 = make_float2(ex2_approx(ar.x), ex2_approx(ar.y));
  if constexpr (GRAD) {
    r.dy = dy;
    r.lo = lo;
  }
  return r;
}

// The two runs of a pair as shared-space addresses of their first pixels
// (relative to a window base) and lengths: n steps together, then m of the
// longer one (a if long_a).
template <int CS>
struct PairWalk {
  static constexpr uint32_t kColB = 4u * CS;  // bytes between columns
  uint32_t a, b;
  int n, m;
  bool long_a;
  __device__ __forceinline__ PairWalk(unsigned run, uint32_t base_a, uint32_t base_b) {
    const int la = (run >> 8) & 0xFF, lb = run >> 24;
    a = base_a + (run & 0xFFu) * kColB;
    b = base_b + ((run >> 16) & 0xFFu) * kColB;
    n = min(la, lb);
    m = max(la, lb) - n;
    long_a = la > lb;
  }
};

// The walks: the n steps in a loop, then (behind a __syncwarp: the lanes leave
// the loop at different steps) the longer row's next pixel and, where any lane
// has them -- tips and clipped boxes -- the rest.

// Adds the sums of K w over the pair's runs to `to`: each row's by itself to a
// binary64 sum, both rows' together otherwise.  (By itself to a compensated
// binary32 sum as well: 1 % of an MLEM pass, 1.5 % with the two in packed
// arithmetic, and no smaller an error: what a row's own steps round is as much.)
template <int UNROLL, int ACC, int CS>
__device__ __forceinline__ void pair_sum(float2 P, float2 S, float2 Q, PairWalk<CS> w,
                                         RowSum<ACC>& to) {
  constexpr uint32_t kColB = PairWalk<CS>::kColB;
  float2 A = make_float2(0.0f, 0.0f);
#pragma unroll UNROLL
  for (int j = w.n; j > 0; --j, w.a += kColB, w.b += kColB) {
    A = __ffma2_rn(P, make_float2(lds32(w.a), lds32(w.b)), A);
    P = __fmul2_rn(P, S);
    S = __ffma2_rn(S, Q, S);
  }
  __syncwarp();
  constexpr bool kRows = ACC == STRIP_ACCUM_FP64;
  float sum = kRows ? (w.long_a ? A.x : A.y) : A.x + A.y;
  if (kRows) to.add(w.long_a ? A.y : A.x);
  uint32_t p = w.long_a ? w.a : w.b;
  float x = w.long_a ? P.x : P.y;
  if (w.m > 0) sum = fmaf(x, lds32(p), sum);
  if (__any_sync(kFull, w.m > 1)) {
    float r = w.long_a ? S.x : S.y;
#pragma unroll 1
    for (int j = w.m - 1; j > 0; --j) {
      x *= r;
      r = fmaf(r, Q.x, r);
      p += kColB;
      sum = fmaf(x, lds32(p), sum);
    }
    __syncwarp();
  }
  to.add(sum);
}

// Sums of K w and K w t^2 over the pair's runs (the sigma gradient); t: the
// distances of the runs' first pixels from the rows' centres.  2e6 events at
// 400 x 400, sigma_z 8, sigma_dl 30 mm: 6.5 ms with one event per warp, one
// row per lane and two global binary64 reductions per event on the same two
// words; 2.7 ms here, with the sums kept in the lanes over the item's events.
template <int CS>
__device__ __forceinline__ void pair_moments(float2 P, float2 S, float2 Q, float2 t, float pw,
                                             PairWalk<CS> w, float2& s0, float2& s2) {
  constexpr uint32_t kColB = PairWalk<CS>::kColB;
  s0 = s2 = make_float2(0.0f, 0.0f);
  const float2 dt = dup(pw), t0 = t;
  float2 at = make_float2(0.0f, 0.0f);  // steps taken
#pragma unroll kUnroll
  for (int j = w.n; j > 0; --j, w.a += kColB, w.b += kColB) {
    const float2 x = __fmul2_rn(P, make_float2(lds32(w.a), lds32(w.b)));
    s0 = __fadd2_rn(s0, x);
    s2 = __ffma2_rn(__fmul2_rn(x, t), t, s2);
    at = __fadd2_rn(at, dup(1.0f));
    t = __ffma2_rn(at, dt, t0);
    P = __fmul2_rn(P, S);
    S = __fmul2_rn(S, Q);
  }
  __syncwarp();
  if (__any_sync(kFull, w.m > 0)) {
    uint32_t p = w.long_a ? w.a : w.b;
    float x = w.long_a ? P.x : P.y, r = w.long_a ? S.x : S.y, u = w.long_a ? t.x : t.y;
    float a0 = 0.0f, a2 = 0.0f;
#pragma unroll 1
    for (int j = w.m; j > 0; --j) {
      const float v = x * lds32(p);
      a0 += v;
      a2 = fmaf(v * u, u, a2);
      u += pw;
      x *= r;
      r *= Q.x;
      p += kColB;
    }
    if (w.long_a) {
      s0.x += a0;
      s2.x += a2;
    } else {
      s0.y += a0;
      s2.y += a2;
    }
    __syncwarp();
  }
}

// How the backprojection turns a value into window units: K (times the image)
// by the subnormal product or cvt.rni, or signed by the 1.5 * 2^23 addend.
enum { kAddSubnormal, kAddCvt, kAddWeightedSubnormal, kAddWeightedCvt, kAddSigned };

// acc += K (in window units: P carries the event's factor) over the pair's
// runs; w: addresses in the accumulator window, off: from there to the image
// window.
template <int ADD, int CS>
__device__ __forceinline__ void pair_scatter(float2 P, float2 S, float2 Q, PairWalk<CS> w,
                                             uint32_t off) {
  constexpr uint32_t kColB = PairWalk<CS>::kColB;
  constexpr bool kWeighted = ADD == kAddWeightedSubnormal || ADD == kAddWeightedCvt;
  constexpr bool kSub = ADD == kAddSubnormal || ADD == kAddWeightedSubnormal;
  const float tiny = __uint_as_float(1u);  // 2^-149
  const float magic = 12582912.0f;
  const unsigned magic_bits = 0x4B400000u;
#pragma unroll kUnroll
  for (int j = w.n; j > 0; --j, w.a += kColB, w.b += kColB) {
    float2 x = P;
    if constexpr (kWeighted)
      x = __fmul2_rn(x, make_float2(lds32(w.a + off), lds32(w.b + off)));
    if constexpr (kSub) {
      x = __fmul2_rn(x, dup(tiny));
      red_shared_add(w.a, __float_as_uint(x.x));
      red_shared_add(w.b, __float_as_uint(x.y));
    } else if constexpr (ADD == kAddSigned) {
      x = __fadd2_rn(x, dup(magic));
      red_shared_add(w.a, __float_as_uint(x.x) - magic_bits);
      red_shared_add(w.b, __float_as_uint(x.y) - magic_bits);
    } else {
      red_shared_add(w.a, __float2uint_rn(x.x));
      red_shared_add(w.b, __float2uint_rn(x.y));
    }
    P = __fmul2_rn(P, S);
    S = __ffma2_rn(S, Q, S);
  }
  __syncwarp();
  auto put = [&](uint32_t p, float x) {  // one pixel
    if constexpr (kWeighted) x *= lds32(p + off);
    const unsigned v = kSub                ? __float_as_uint(x * tiny)
                       : ADD == kAddSigned ? __float_as_uint(x + magic) - magic_bits
                                           : __float2uint_rn(x);
    red_shared_add(p, v);
  };
  uint32_t p = w.long_a ? w.a : w.b;
  float x = w.long_a ? P.x : P.y;
  if (w.m > 0) put(p, x);
  if (__any_sync(kFull, w.m > 1)) {
    float r = w.long_a ? S.x : S.y;
#pragma unroll 1
    for (int j = w.m - 1; j > 0; --j) {
      x *= r;
      r = fmaf(r, Q.x, r);
      p += kColB;
      put(p, x);
    }
    __syncwarp();
  }
}

// A work item's window in shared memory.
struct PairWin {
  uint32_t w, acc;   // shared-space addresses of the image and the accumulator
  int wx0, wy0;
  float unit;        // window units per K / D (MLEM) or K w (adjoint)
};

// The events of a work item.  Warps take groups of `grab` events from the
// item's counter.  MLEM: WEIGHTED adds K rho / D, else K / D, with the events
// that the conversion or the window's budget has no room for marked in
// s_fb_bits; `only`: the marked events (unmarked as they find room).
template <int OP, int ACC, int LPE, int NB, int CS, bool WEIGHTED, int ADD>
__device__ __forceinline__ void pair_item(const LaunchArgs& a, const WorkItem& it,
                                          const PairWin& win, int lane, int grab,
                                          int* next_group, const unsigned* only,
                                          double* grad = nullptr) {
  constexpr int kPer = 32 / LPE;
  constexpr int kBlocks = OP == OP_MLEM ? NB : 1;  // kept for pass 2
  const int grp = lane / LPE, sub = lane & (LPE - 1);
  const float2 Q = dup(a.pc.qm1);
  const float mw = 8388608.0f - (float)win.wx0;
  float rsum = 0.0f;
  for (;;) {
    int g = 0;
    if (lane == 0) g = atomicAdd(next_group, 1);
    g = __shfl_sync(kFull, g, 0);
    const int g0 = g * grab, g1 = min(g0 + grab, it.count);
    if (g0 >= it.count) break;
    for (int j = g0 + grp; j - grp < g1; j += kPer) {
      bool has = j < g1;
      if (only && has) has = (only[j >> 5] >> (j & 31)) & 1u;
      if (only && !__any_sync(kFull, has)) continue;
      EventPack m = a.packs[it.begin + (has ? j : g0)];
      if (!has) m.yb = 0u;  // no rows
      const PairEvent e = pair_event(a.s, a.pc, m, win.wy0);
      // blocks of the warp's tallest event (a warp reduction: the branches on
      // it are uniform to the compiler too)
      const int nb = ((int)__reduce_max_sync(kFull, (unsigned)e.n_a) + LPE - 1) / LPE;
      // this lane's rows of block 0; block b lies 4 LPE b bytes further out
      const uint32_t ra = 4u * (uint32_t)(e.row_a + sub);
      const uint32_t rb = 4u * (uint32_t)(e.row_a - 1 - sub);
      if constexpr (OP == OP_ADJOINT) {
        const float wf = has ? a.wf_in[it.begin + j] * win.unit : 0.0f;
        if (!__any_sync(kFull, wf != 0.0f)) continue;
        for (int b = 0; b < nb; ++b) {
          PairRow r = pair_row(a.s, a.pc, e, LPE * b + sub, mw);
          if (wf == 0.0f) r.run = 0u;
          pair_scatter<ADD, CS>(__fmul2_rn(r.K0, dup(wf)), r.R0, Q,
                                   PairWalk<CS>(r.run, win.acc + ra + 4u * LPE * b,
                                            win.acc + rb - 4u * LPE * b), 0u);
        }
        continue;
      }
      if constexpr (OP == OP_GRAD) {
        // The lane adds up its rows of all its events in binary64.  A row's
        // values and steps are the one-row kernel's (grad_event): its sums
        // cancel to a few hundredths of their terms, so that other roundings
        // of the same row -- of q above all, 3e-5 at sigma_z of 10 pixels --
        // would set the two kernels' gradients apart by more than 2e-5.
        const double w = has ? a.w_in[a.perm[it.begin + j]] : 0.0;
        if (!__any_sync(kFull, w != 0.0)) continue;
        for (int b = 0; b < nb; ++b) {
          PairRow r = pair_row<true>(a.s, a.pc, e, LPE * b + sub, mw);
          if (w == 0.0) r.run = 0u;
          GaussGradRow ga, gb;
          ga.init(a.k, a.s.R, m.y, m.tan, m.sec, r.dy.x);
          gb.init(a.k, a.s.R, m.y, m.tan, m.sec, r.dy.y);
          const float2 t = make_float2(fmaf(r.lo.x, a.s.pw, a.s.tl_z_half_w) - m.z - ga.dytan,
                                       fmaf(r.lo.y, a.s.pw, a.s.tl_z_half_w) - m.z - gb.dytan);
          const float2 K0 = make_float2(ex2_approx(fmaf(a.k.c1 * t.x, t.x, ga.c0)),
                                        ex2_approx(fmaf(a.k.c1 * t.y, t.y, gb.c0)));
          const float2 R0 = make_float2(ex2_approx(fmaf(a.k.r1, t.x, a.k.r0)),
                                        ex2_approx(fmaf(a.k.r1, t.y, a.k.r0)));
          float2 s0, s2;
          pair_moments<CS>(K0, R0, dup(a.k.q), t, a.s.pw,
                           PairWalk<CS>(r.run, win.w + ra + 4u * LPE * b,
                                        win.w + rb - 4u * LPE * b), s0, s2);
          auto row = [&](const GaussGradRow& g, float s0, float s2) {
            // rows without pixels have any pref, fz and fdl
            if (s0 != 0.0f || s2 != 0.0f) {
              grad[0] += w * (double)(g.pref * fmaf(g.fz, s0, 2.0f * a.k.ipsz * s2));
              grad[1] += w * (double)(g.pref * g.fdl * s0);
            }
          };
          row(ga, s0.x, s2.x);
          row(gb, s0.y, s2.y);
        }
        continue;
      }
      RowSum<ACC> sum;
      PairRow rows[kBlocks];
      if constexpr (OP == OP_FORWARD) {
        for (int b = 0; b < nb; ++b) {
          const PairRow r = pair_row(a.s, a.pc, e, LPE * b + sub, mw);
          pair_sum<sum_unroll(OP)>(r.K0, r.R0, Q,
                                   PairWalk<CS>(r.run, win.w + ra + 4u * LPE * b,
                                                win.w + rb - 4u * LPE * b), sum);
        }
      } else {
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          if (b < nb) {
            rows[b] = pair_row(a.s, a.pc, e, LPE * b + sub, mw);
            pair_sum<sum_unroll(OP)>(rows[b].K0, rows[b].R0, Q,
                                     PairWalk<CS>(rows[b].run, win.w + ra + 4u * LPE * b,
                                                  win.w + rb - 4u * LPE * b), sum);
          }
        }
      }
      double D = sum.total();
#pragma unroll
      for (int o = LPE / 2; o > 0; o >>= 1) D += __shfl_xor_sync(kFull, D, o);
      if constexpr (OP == OP_FORWARD) {
        if (sub == 0 && e.n_a > 0) a.y_out[a.perm[it.begin + j]] = D;
        continue;
      }
      // reconstruction.h:290 -- an all-zero denominator contributes nothing
      bool go = e.n_a > 0 && D > 0.0;
      const float scale = go ? rcp_approx((float)D) : 0.0f;
      if constexpr (!WEIGHTED) {
        // reserve the event's largest addend, kbound * unit / D (rounded up, in
        // units of 2^8), from the item's fixed-point budget
        const float need = a.kbound * scale * win.unit;
        int ok = 0;
        // the subnormal conversion takes addends below 2^24
        if (sub == 0 && go && need < (ADD == kAddSubnormal ? 16000000.0f : kFixedBudget)) {
          const unsigned nu = (unsigned)(need * (1.0f / 256.0f)) + 1u;
          const unsigned old = atomicAdd(&s_fx_budget, nu);
          ok = old + nu <= kBudgetUnits;
          if (!ok) atomicSub(&s_fx_budget, nu);
        }
        ok = __shfl_sync(kFull, ok, lane & ~(LPE - 1));
        // an event without room is marked: it runs again, first (`only`) with
        // the other conversion, then in a weighted window
        if (go && sub == 0 && (only ? ok : !ok)) {
          atomicXor(&s_fb_bits[j >> 5], 1u << (j & 31));
          atomicAdd(&s_fb_n, only ? -1 : 1);
        }
        go = go && ok;
      }
      rsum += scale;
      if (!__any_sync(kFull, go)) continue;
      // the event's factor in the window's units (clamped: a denominator so
      // small that 1 / D overflows still scatters finite values)
      const float2 sc = dup(WEIGHTED ? fminf(scale * win.unit, 3.0e38f) : scale * win.unit);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        if (b < nb)
          pair_scatter<ADD, CS>(__fmul2_rn(rows[b].K0, sc), rows[b].R0, Q,
                            PairWalk<CS>(go ? rows[b].run : 0u, win.acc + ra + 4u * LPE * b,
                                     win.acc + rb - 4u * LPE * b),
                            win.w - win.acc);
      }
    }
  }
  if (OP == OP_MLEM && !only && sub == 0 && rsum != 0.0f) atomicAdd(&s_item_rsum, rsum);
}

// One work item on the whole CTA: stage the window, run the events, flush.
// `index` is the item's index among the launch's items (its statistic in
// a.item_hist).  The caller synchronises before the shared memory is reused.
template <int OP, int ACC, int LPE, int NB, int CS>
__device__ __forceinline__ void pair_tile_item(const LaunchArgs& a, const WorkItem it, int index,
                                               char* smem_raw, int* s_next_group) {
  constexpr bool kReads = OP != OP_ADJOINT, kWrites = OP == OP_MLEM || OP == OP_ADJOINT;
  int wx0, wy0, wx1, wy1;
  tile_window(a.t, a.s.n_z, a.s.n_y, it.tile, wx0, wy0, wx1, wy1);
  const int wxn = wx1 - wx0, wyn = wy1 - wy0;
  float* s_w = reinterpret_cast<float*>(smem_raw);
  // the adjoint reads no image: its accumulator is the only window
  float* s_acc = OP == OP_ADJOINT ? s_w : s_w + a.t.WXmax * CS;
  if (threadIdx.x == 0) {
    *s_next_group = 0;
    s_fx_budget = 0u;
    s_item_rsum = 0.0f;
    s_fb_n = 0;
  }
  if (OP == OP_MLEM)
    for (int q = threadIdx.x; q < kMaxItemEvents / 32; q += blockDim.x) s_fb_bits[q] = 0u;
  const int lane = threadIdx.x & 31;
  float wsum = 0.0f;
  float wmin = 0.0f;  // the least pixel below zero
  each_pixel<true>(wxn, wyn, lane, [&](int r, int c) {
    if (kReads) {
      const float v = a.rho[(int64_t)(wy0 + r) * a.s.n_z + wx0 + c];
      s_w[c * CS + r] = v;
      if (OP == OP_MLEM) {
        wsum += v;
        wmin = fminf(wmin, v);
      }
    }
    if (kWrites) s_acc[c * CS + r] = 0.0f;
  });
  bool negative = false;
  if constexpr (OP == OP_MLEM)
    negative = __syncthreads_or(wmin < 0.0f);
  else
    __syncthreads();
  PairWin win{(uint32_t)__cvta_generic_to_shared(s_w), (uint32_t)__cvta_generic_to_shared(s_acc),
              wx0, wy0, 1.0f};
  // groups of events per counter step: fewer for small items, so that every
  // warp has some
  constexpr int kPer = 32 / LPE;
  const int share = it.count / (int)(blockDim.x >> 5);
  const int grab = max(kPer, min(a.grab, share) / kPer * kPer);
  // Adds the window accumulator (fixed point at scale 2^fshift, times the
  // image value for an unweighted window, which is zeroed on the way) into
  // the global binary64 accumulator.
  auto flush = [&](int fshift, bool unweighted) {
    const double per = exp2((double)-fshift);
    each_pixel<true>(wxn, wyn, lane, [&](int r, int c) {
      const int wi = c * CS + r;
      const unsigned raw = __float_as_uint(s_acc[wi]);
      double v = (OP == OP_ADJOINT ? (double)(int)raw : (double)raw) * per;
      if (unweighted) {
        v *= (double)s_w[wi];
        s_acc[wi] = 0.0f;
      }
      if (v != 0.0) atomicAdd(a.acc + (int64_t)(wy0 + r) * a.s.n_z + wx0 + c, v);
    });
  };
  if constexpr (OP == OP_GRAD) {
    double grad[2] = {0.0, 0.0};
    pair_item<OP, ACC, LPE, NB, CS, false, kAddSigned>(a, it, win, lane, grab, s_next_group, nullptr,
                                                   grad);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      grad[0] += __shfl_xor_sync(kFull, grad[0], o);
      grad[1] += __shfl_xor_sync(kFull, grad[1], o);
    }
    if (lane == 0) {
      atomicAdd(a.grad_out, grad[0] / a.sz);
      atomicAdd(a.grad_out + 1, grad[1] / a.sdl);
    }
  } else if constexpr (OP == OP_FORWARD) {
    pair_item<OP, ACC, LPE, NB, CS, false, kAddSigned>(a, it, win, lane, grab, s_next_group, nullptr);
  } else if constexpr (OP == OP_ADJOINT) {
    // addends below 2^22 (adjoint_shift); without negative weights the
    // subnormal conversion gives the same integers without the subtractions
    const int fshift = adjoint_shift(a, it, lane, &negative);
    win.unit = exp2f((float)fshift);
    if (negative)
      pair_item<OP, ACC, LPE, NB, CS, false, kAddSigned>(a, it, win, lane, grab, s_next_group,
                                                     nullptr);
    else
      pair_item<OP, ACC, LPE, NB, CS, false, kAddSubnormal>(a, it, win, lane, grab, s_next_group,
                                                        nullptr);
    __syncthreads();
    flush(fshift, false);
  } else {
    // the unweighted window once the item has a statistic, else weighted
    const float wmean = block_sum(wsum) / (float)(wxn * wyn);
    const float hist = a.item_hist ? a.item_hist[index] : 0.0f;
    const float B = hist / wmean;  // this pass's sum of 1 / D_e, estimated
    const float lim = 1073741824.0f / (a.kbound * B);  // 2^30 / (kbound B)
    int fshift = 0;
    bool unweighted = false;
    if (hist > 0.0f && wmean > 0.0f && B > 0.0f && B < 3.0e38f && lim > 0.0f && lim < 3.0e38f) {
      fshift = (int)floorf(log2f(lim));
      unweighted = fshift >= -120 && fshift <= 120;
    }
    int n_weighted = it.count;
    const unsigned* only = nullptr;
    if (unweighted) {
      win.unit = exp2f((float)fshift);
      // with 512 events and more the mean addend is at most 2^21, so few meet
      // the subnormal conversion's 2^24 (3 in 1e5 at the benchmark; they run
      // again by cvt.rni); smaller items have larger ones
      bool late = false;
      if (it.count >= 512) {
        pair_item<OP, ACC, LPE, NB, CS, false, kAddSubnormal>(a, it, win, lane, grab, s_next_group,
                                                          nullptr);
        __syncthreads();
        late = s_fb_n > 0;
        __syncthreads();
        if (late) {
          if (threadIdx.x == 0) *s_next_group = 0;
          __syncthreads();
        }
      }
      if (it.count < 512 || late)
        pair_item<OP, ACC, LPE, NB, CS, false, kAddCvt>(a, it, win, lane, grab, s_next_group,
                                                    late ? s_fb_bits : nullptr);
      __syncthreads();
      flush(fshift, true);
      n_weighted = s_fb_n;  // the events that found no room
      only = s_fb_bits;
      if (n_weighted > 0) {
        __syncthreads();  // the flush has zeroed the window accumulator
        if (threadIdx.x == 0) {
          *s_next_group = 0;
          if (a.n_fallback) atomicAdd(a.n_fallback, (unsigned long long)n_weighted);
        }
        __syncthreads();
      }
    }
    if (n_weighted > 0) {
      const int fs = fixed_shift(n_weighted);
      win.unit = exp2f((float)fs);
      // K rho / D <= 1: addends up to the unit; over pixels below zero, infinite
      // (updates can make some) or NaN they may be anything, which cvt.rni clamps
      if (fs <= 23 && !negative && wmean <= 3.402823466e38f)
        pair_item<OP, ACC, LPE, NB, CS, true, kAddWeightedSubnormal>(a, it, win, lane, grab,
                                                                 s_next_group, only);
      else
        pair_item<OP, ACC, LPE, NB, CS, true, kAddWeightedCvt>(a, it, win, lane, grab, s_next_group,
                                                           only);
      __syncthreads();
      flush(fs, false);
    }
    if (threadIdx.x == 0 && a.item_hist) a.item_hist[index] = s_item_rsum * wmean;
  }
}

template <int OP, int ACC, int THREADS, int LPE, int NB, int CS>
__global__ void __launch_bounds__(THREADS, THREADS == kPairWide ? 1 : 2)
    k_pair_tile(const __grid_constant__ LaunchArgs a) {
  extern __shared__ __align__(16) char smem_raw[];
  __shared__ int s_next_group;
  pair_tile_item<OP, ACC, LPE, NB, CS>(a, a.items[blockIdx.x], blockIdx.x, smem_raw, &s_next_group);
}

// Blocks of row pairs held through both passes: 5 blocks of 8 pairs (80 rows)
// or 4 of 16 (128 rows).  Boxes of at most 80 rows take 8 lanes an event; the
// windows of taller ones have the tall column stride where they need it
// (choose_tiling).
constexpr int kBlocks8 = 5, kBlocks16 = 4;
static_assert(16 * kBlocks8 == kPairRows8 && 32 * kBlocks16 == kPairRows16, "row-pair layouts");

template <int OP, int ACC, int LPE, int NB, int CS>
cudaError_t launch_pair_lpe(const LaunchArgs& a, cudaStream_t st) {
  const int smem = a.t.smem_bytes / 2 * (OP == OP_MLEM ? 2 : 1);
  const bool wide = smem > kNarrowSmemBytes;  // one CTA per SM
  auto fn = wide ? k_pair_tile<OP, ACC, kPairWide, LPE, NB, CS>
                 : k_pair_tile<OP, ACC, kPairThreads, LPE, NB, CS>;
  cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return err;
  fn<<<a.n_items, wide ? kPairWide : kPairThreads, smem, st>>>(a);
  return cudaGetLastError();
}

template <int OP, int ACC>
cudaError_t launch_pair_t(const LaunchArgs& a, cudaStream_t st) {
  const bool tall = a.t.cs == kTallStride;
  if constexpr (OP == OP_MLEM) {
    if (tall) return launch_pair_lpe<OP, ACC, 16, kBlocks16, kTallStride>(a, st);
    if (a.t.max_rows > kPairRows8)
      return launch_pair_lpe<OP, ACC, 16, kBlocks16, kColumnStride>(a, st);
  } else {
    if (tall) return launch_pair_lpe<OP, ACC, 8, kBlocks8, kTallStride>(a, st);
  }
  return launch_pair_lpe<OP, ACC, 8, kBlocks8, kColumnStride>(a, st);
}

template <int OP>
cudaError_t launch_pair_op(int accum, const LaunchArgs& a, cudaStream_t st) {
  if (accum == STRIP_ACCUM_FP32) return launch_pair_t<OP, STRIP_ACCUM_FP32>(a, st);
  if (accum == STRIP_ACCUM_FP64) return launch_pair_t<OP, STRIP_ACCUM_FP64>(a, st);
  return launch_pair_t<OP, STRIP_ACCUM_KAHAN>(a, st);
}

}  // namespace

namespace {

// Persistent form over the work items of several reconstructions: a CTA takes
// item after item from a global counter; item i belongs to member
// items[i].member, whose arguments live in the kernel's parameter space.
template <int ACC, int THREADS, int LPE, int NB, int CS>
__global__ void __launch_bounds__(THREADS, THREADS == kPairWide ? 1 : 2)
    k_pair_batch(const __grid_constant__ BatchArgs b, const BatchItem* items, int n_items,
                 int* counter) {
  extern __shared__ __align__(16) char smem_raw[];
  __shared__ int s_next_group;
  __shared__ int s_item;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int i = s_item;
    if (i >= n_items) break;
    const BatchItem bi = items[i];
    pair_tile_item<OP_MLEM, ACC, LPE, NB, CS>(b.member[bi.member],
                                          WorkItem{bi.tile, bi.count, bi.begin}, bi.index,
                                          smem_raw, &s_next_group);
    __syncthreads();  // before the next item's window overwrites this one
  }
}

template <int THREADS, int LPE, int NB, int CS, class F>
cudaError_t with_pair_batch_t(int accum, F&& pick) {
  if (accum == STRIP_ACCUM_FP32) return pick(k_pair_batch<STRIP_ACCUM_FP32, THREADS, LPE, NB, CS>);
  if (accum == STRIP_ACCUM_FP64) return pick(k_pair_batch<STRIP_ACCUM_FP64, THREADS, LPE, NB, CS>);
  return pick(k_pair_batch<STRIP_ACCUM_KAHAN, THREADS, LPE, NB, CS>);
}

template <int LPE, int NB, int CS, class F>
cudaError_t with_pair_batch_w(int accum, int smem_bytes, F&& pick) {
  return smem_bytes > kNarrowSmemBytes ? with_pair_batch_t<kPairWide, LPE, NB, CS>(accum, pick)
                                       : with_pair_batch_t<kPairThreads, LPE, NB, CS>(accum, pick);
}

template <class F>
cudaError_t with_pair_batch(int accum, int smem_bytes, int max_rows, int windows, F&& pick) {
  if (windows == kPairTall)
    return with_pair_batch_w<16, kBlocks16, kTallStride>(accum, smem_bytes, pick);
  if (max_rows > kPairRows8)
    return with_pair_batch_w<16, kBlocks16, kColumnStride>(accum, smem_bytes, pick);
  return with_pair_batch_w<8, kBlocks8, kColumnStride>(accum, smem_bytes, pick);
}

// The events' packs, one event per thread.  Memory bound: 36 bytes an event.
__global__ void k_event_packs(ScannerF s, const float* __restrict__ zu,
                              const float* __restrict__ zd, const float* __restrict__ dl,
                              int64_t n, EventPack* packs) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  EventF e;
  event_setup(s, zu[i], zd[i], dl[i], e);
  packs[i] = pack_event(e);
}

}  // namespace

cudaError_t launch_event_packs(const ScannerF& s, const float* zu, const float* zd,
                               const float* dl, int64_t n, EventPack* packs, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_event_packs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s, zu, zd, dl, n, packs);
  return cudaGetLastError();
}

cudaError_t pair_batch_reserve_smem(int accum, int smem_bytes, int max_rows, int windows) {
  return with_pair_batch(accum, smem_bytes, max_rows, windows, [&](auto fn) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  });
}

cudaError_t launch_pair_batch(int accum, const BatchArgs& b, const BatchItem* items, int n_items,
                              int* counter, int smem_bytes, int max_rows, int windows,
                              int sm_count,                               cudaStream_t st) {
  const bool wide = smem_bytes > kNarrowSmemBytes;
  return with_pair_batch(accum, smem_bytes, max_rows, windows, [&](auto fn) -> cudaError_t {
    const int grid = std::min(n_items, sm_count * (wide ? 1 : 2));
    fn<<<grid, wide ? kPairWide : kPairThreads, smem_bytes, st>>>(b, items, n_items, counter);
    return cudaGetLastError();
  });
}

cudaError_t launch_pair_tile(int op, int accum, const LaunchArgs& a, cudaStream_t st) {
  switch (op) {
    case OP_MLEM:
      return launch_pair_op<OP_MLEM>(accum, a, st);
    case OP_FORWARD:
      return launch_pair_op<OP_FORWARD>(accum, a, st);
    case OP_ADJOINT:  // no per-event sums: one form
      return launch_pair_t<OP_ADJOINT, STRIP_ACCUM_FP32>(a, st);
    case OP_GRAD:
      return launch_pair_t<OP_GRAD, STRIP_ACCUM_FP32>(a, st);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace stripmlem
