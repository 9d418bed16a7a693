// itr_device.cuh — per-face and per-cell arithmetic of the first-order FV step, on sm_100a.
//
// Operation order follows crates/itr-hydro/src/numerics.rs exactly (every product and sum
// in the same association), and the library is compiled with -fmad=false, IEEE division
// and square root and no flush-to-zero, so each value here has the same bits as the
// reference's f32 kernel (the reference's rule: IEEE + - * / sqrt only, spec.md:618).
//   rcbrt        crates/itr-core/src/real.rs:116-130
//   cell_vel     numerics.rs:36-43
//   hll          numerics.rs:56-93
//   face_signed  numerics.rs:95-112
//   face_crest   numerics.rs:114-129
//   update_cell  numerics.rs:144-213 (flux_update + sources)
// NaN semantics of max/min/abs are the reference's (real.rs:38-58), not fmaxf/fabsf.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>
#include "itr_math.h"

namespace itr {

#define ITR_DEV __device__ __forceinline__

ITR_DEV float rmax(float a, float b) { return a > b ? a : b; }
ITR_DEV float rmin(float a, float b) { return a < b ? a : b; }
ITR_DEV float rabs(float a) { return a < 0.0f ? -a : a; }
ITR_DEV float canon(float a) { return a == 0.0f ? 0.0f : a; }

// x^(-1/3): bit seed 0x54A23280 - bits/3 and three short-chain Newton steps.
ITR_DEV float rcbrt(float x) {
  uint32_t bits = __float_as_uint(x);
  float r = __uint_as_float(0x54A23280u - bits / 3u);
  const float x3 = x * (float)(1.0 / 3.0);
  const float c43 = (float)(4.0 * (1.0 / 3.0));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    float r2 = r * r;
    r = r * c43 - x3 * (r2 * r2);
  }
  return r;
}

// Step constants, all rounded once from f64 (solver.rs:269-285).
struct StepK {
  float g, g_half, dt, dtdx, dtdy, inv_dx, inv_dy, h_dry, heps2, q_min, rain, cap;
  float nz;   // -0.0f read from the kernel parameters at run time (see mul2)
  unsigned exact;   // 1: this step through the scalar path (state or parameters not known to be bounded, or checking)
};

// A face flux tuple: mass, normal momentum seen from the low-index (n_l) and high-index
// (n_r) cell with the hydrostatic pressure correction folded in, tangential momentum.
struct FaceF { float m, nl, nr, t; };

// Desingularised velocity and celerity of a cell.
// 1/x rounded to nearest (IEEE): the same value as 1.0f / x compiled with IEEE division,
// through the reciprocal instruction path.
ITR_DEV float rcp(float x) { return __frcp_rn(x); }

// IEEE square root with zero kept off the instruction's special-case path: sqrt(+-0) is
// +-0 exactly, so returning x for x == 0 gives the same bits as sqrtf(x) for every input,
// while dry faces and cells (reduced depth 0) stay on the fast path.
ITR_DEV float sqrt_rn(float x) {
  const bool z = x == 0.0f;
  const float r = sqrtf(z ? 1.0f : x);
  return z ? x : r;
}

// The special operations of the scalar path: Exact for every operand; Fast without branches, the same
// bits for operands in the ranges that rcp2 and sqrt2 (below) state, which hold in a step from a
// bounded state (StepK::exact == 0). Fast::div: a y with y = 1 / b rounded, corrected twice by the
// exact residual (as div_rn), b in rcp2's range and not above 2^62; a small |a| (adjoints at the fringe of their domain
// of dependence) is scaled by 2^64 and back, which keeps the residual a normal number (|a / b| below 2^63 there:
// the derivative of u at h = 0 reaches 2 / h_eps^2). A quotient
// that overflows, or of an infinity or NaN, is returned before the correction (infinity - infinity); one
// below 2^-126 is rounded a second time on its way back, and may then lie one 2^-149 beside the IEEE
// result. The adjoint's divisors: celerities and |q|, 2^-76 .. 2^40; h^2 above h_eps^2; and h_eps^4 up
// to 4 h_eps^4, which asks for h_eps of 2^-31 or more (RunParams::adj_scalar).
struct Exact {
  static ITR_DEV float rcp(float x) { return itr::rcp(x); }
  static ITR_DEV float sqrt(float x) { return sqrt_rn(x); }
  static ITR_DEV float div(float a, float b) { return a / b; }
};
ITR_DEV float rcp_est(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
ITR_DEV float rsqrt_est(float x) { float r; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
struct Fast {
  static ITR_DEV float rcp(float x) {
    const float y = rcp_est(x);
    return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
  }
  static ITR_DEV float sqrt(float x) {
    const float xs = 0x1p48f * x, y = rsqrt_est(xs + 0x1p-126f);
    const float s = xs * y;
    return __fmaf_rn(__fmaf_rn(-s, s, xs), 0x1p-25f * y, 0x1p-24f * s);
  }
  static ITR_DEV float div(float a, float b) {
    const bool tiny = fabsf(a) < 0x1p-60f;
    const float y = rcp(b), as = a * (tiny ? 0x1p64f : 1.0f);
    const float q = as * y;
    const bool finite = fabsf(q) <= 0x1.fffffep127f;
    float r = __fmaf_rn(__fmaf_rn(-b, q, as), y, q);
    r = __fmaf_rn(__fmaf_rn(-b, r, as), y, r);
    return (finite ? r : q) * (tiny ? 0x1p-64f : 1.0f);
  }
};

template <class F = Exact>
ITR_DEV void cell_vel(float h, float qx, float qy, float g, float heps2, float& u, float& v, float& c) {
  float h2 = h * h;
  float inv = F::rcp(h2 + rmax(h2, heps2));
  float t = (h + h) * inv;
  u = qx * t;
  v = qy * t;
  c = F::sqrt(g * h);
}

// HLL flux with two-rarefaction wave speeds; dry-dry faces give exactly zero.
template <class F = Exact>
ITR_DEV FaceF hll(float hl, float ul, float tl, float cl, float hr, float ur, float tr, float cr, float g_half) {
  const bool dry_l = !(hl > 0.0f);
  const bool dry_r = !(hr > 0.0f);
  float ustar = 0.5f * (ul + ur) + cl - cr;
  float cstar = 0.5f * (cl + cr) + 0.25f * (ul - ur);
  float slw = rmin(ul - cl, ustar - cstar);
  float srw = rmax(ur + cr, ustar + cstar);
  float sl = dry_l ? ur - 2.0f * cr : (dry_r ? ul - cl : slw);
  float sr = dry_l ? ur + cr : (dry_r ? ul + 2.0f * cl : srw);
  float ml = hl * ul;
  float mr = hr * ur;
  float pl_ = g_half * hl * hl;
  float pr_ = g_half * hr * hr;
  float pl = ml * ul + pl_;
  float pr = mr * ur + pr_;
  const bool both_dry = dry_l && dry_r;
  const bool use_l = sl >= 0.0f;
  const bool use_r = sr <= 0.0f;
  float den = (both_dry || use_l || use_r) ? 1.0f : sr - sl;
  float inv = F::rcp(den);
  float slsr = sl * sr;
  float fm_star = (sr * ml - sl * mr + slsr * (hr - hl)) * inv;
  float fn_star = (sr * pl - sl * pr + slsr * (mr - ml)) * inv;
  float fm = both_dry ? 0.0f : (use_l ? ml : (use_r ? mr : fm_star));
  float fn = both_dry ? 0.0f : (use_l ? pl : (use_r ? pr : fn_star));
  float ft = fm * (fm > 0.0f ? tl : tr);
  FaceF f;
  f.m = fm; f.nl = fn - pl_; f.nr = fn - pr_; f.t = ft;
  return f;
}

// Signed-jump face (dz = z_R - z_L): one reduced side, one square root. `normal_x` picks
// which velocity component is normal. (ul,vl,cl) are the left/top cell's velocity.
template <bool NORMAL_X, class F>
ITR_DEV FaceF face_signed(float hl, float ul, float vl, float cl, float hr, float ur, float vr, float cr,
                          float dz, float g, float g_half) {
  const bool pos = dz > 0.0f;
  float hsl = rmax(hl - rmax(dz, 0.0f), 0.0f);
  float hsr = rmax(hr - rmax(-dz, 0.0f), 0.0f);
  float hred = pos ? hsl : hsr;
  float cred = F::sqrt(g * hred);
  float csl = pos ? cred : cl;
  float csr = pos ? cr : cred;
  if (NORMAL_X) return hll<F>(hsl, ul, vl, csl, hsr, ur, vr, csr, g_half);
  return hll<F>(hsl, vl, ul, csl, hsr, vr, ur, csr, g_half);
}

// Crest face: two non-negative jumps d_l = z_f - z_L, d_r = z_f - z_R.
template <bool NORMAL_X, class F>
ITR_DEV FaceF face_crest(float hl, float ul, float vl, float cl, float hr, float ur, float vr, float cr,
                         float d_l, float d_r, float g, float g_half) {
  float hsl = rmax(hl - d_l, 0.0f);
  float hsr = rmax(hr - d_r, 0.0f);
  float csl = d_l > 0.0f ? F::sqrt(g * hsl) : cl;
  float csr = d_r > 0.0f ? F::sqrt(g * hsr) : cr;
  if (NORMAL_X) return hll<F>(hsl, ul, vl, csl, hsr, ur, vr, csr, g_half);
  return hll<F>(hsl, vl, ul, csl, hsr, vr, ur, csr, g_half);
}

template <bool NORMAL_X, bool CREST, class F = Exact>
ITR_DEV FaceF face(float hl, float ul, float vl, float cl, float hr, float ur, float vr, float cr,
                   float d0, float d1, const StepK& k) {
  if (CREST) return face_crest<NORMAL_X, F>(hl, ul, vl, cl, hr, ur, vr, cr, d0, d1, k.g, k.g_half);
  return face_signed<NORMAL_X, F>(hl, ul, vl, cl, hr, ur, vr, cr, d0, k.g, k.g_half);
}

// Result of one cell update. c is sqrt(g*h) of the new depth, which is also the next
// step's celerity (h is never -0 here, so sqrt(g*h) of the stored value is the same bits).
struct CellNew {
  float h, qx, qy, s, infil, fix, c;
  bool bad;
};

// flux_update then sources (numerics.rs:144-195).
ITR_DEV CellNew update_cell(float h, float qx, float qy, const FaceF& w, const FaceF& e, const FaceF& n,
                            const FaceF& s, float wet, float gn2, const StepK& k) {
  float h1 = h - k.dtdx * (e.m - w.m) - k.dtdy * (s.m - n.m);
  float qx1 = qx - k.dtdx * (e.nl - w.nr) - k.dtdy * (s.t - n.t);
  float qy1 = qy - k.dtdx * (e.t - w.t) - k.dtdy * (s.nl - n.nr);
  CellNew o;
  bool bad = !(h1 >= -k.h_dry);
  o.fix = h1 < 0.0f ? -h1 : 0.0f;
  if (h1 < 0.0f) h1 = 0.0f;
  float h2 = h1 + k.rain * wet;
  o.infil = rmin(k.cap * wet, h2);
  float h3 = h2 - o.infil;
  const bool dry = h3 < k.h_dry;
  float r = rcbrt(dry ? 1.0f : h3);
  float r3 = r * r * r;
  float r7 = r3 * r3 * r;
  float qm = sqrt_rn(qx1 * qx1 + qy1 * qy1);
  float inv = rcp(1.0f + k.dt * gn2 * qm * r7);
  float keep = dry ? 0.0f : 1.0f;
  float qx2 = qx1 * inv * keep;
  float qy2 = qy1 * inv * keep;
  if (rabs(qx2) < k.q_min) qx2 = 0.0f;
  if (rabs(qy2) < k.q_min) qy2 = 0.0f;
  float c = sqrt_rn(k.g * h3);
  o.s = (rabs(qx2) * r3 + c) * k.inv_dx + (rabs(qy2) * r3 + c) * k.inv_dy;
  o.bad = bad || !(qm == qm);
  o.h = canon(h3);
  o.qx = canon(qx2);
  o.qy = canon(qy2);
  o.c = c;
  return o;
}

// ------------------------------------------------------------------ time integrator ----
// Hyetograph (scenario.rs:526-586) and the f64 step rule of solver.rs:449-489, evaluated by
// every thread of a design redundantly (identical inputs, identical bits).
constexpr int kMaxRain = 32;

// One linear piece of the rate: r0 + dr (x - t0) / den for x <= end (rden = 1 / den rounded). Piece 0 is
// the constant before the first point, piece n the constant after the last.
struct RainSeg { double t0, r0, dr, den, rden, end; };

struct Rain {
  int n;
  double t[kMaxRain];
  double r[kMaxRain];
  RainSeg seg[kMaxRain + 1];
};

// a / b rounded to nearest from y = 1 / b rounded to nearest, as fused multiply-adds: a y is within two
// units of the last place, one correction by the exact residual makes it faithful, a second one
// rounds it right (P. Markstein, IBM J. Res. Dev. 34(1), 1990; Muller et al., Handbook of
// Floating-Point Arithmetic, 2nd ed., 2018, ch. 4). Operands and quotient in the normal range, or a = 0.
ITR_DEV double div_rn(double a, double b, double y) {
  double q = a * y;
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}
// The same for a b that is an f32 above 0: the reciprocal by Newton steps from the hardware's estimate.
// The last step starts within a unit of 1 / b, so it rounds it right unless b's 53-bit significand is
// all ones (same sources), which an f32's is not.
ITR_DEV double div_by_f32(double a, double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
#pragma unroll
  for (int i = 0; i < 3; ++i) y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
  return div_rn(a, b, y);
}

ITR_DEV double rain_rate(const Rain& R, double x) {
  if (R.n == 0) return 0.0;
  if (x <= R.t[0]) return R.r[0];
  for (int k = 0; k + 1 < R.n; ++k) {
    if (x <= R.t[k + 1]) {
      double t0 = R.t[k], r0 = R.r[k], t1 = R.t[k + 1], r1 = R.r[k + 1];
      if (t1 == t0) return r1;
      return r0 + (r1 - r0) * (x - t0) / (t1 - t0);
    }
  }
  return R.r[R.n - 1];
}

ITR_DEV double rain_integral(const Rain& R, double a, double b) {
  if (b <= a) return 0.0;
  if (R.n == 0) return 0.0;
  double total = 0.0, tt = a, rr = rain_rate(R, a);
  for (int k = 0; k < R.n; ++k) {
    double tk = R.t[k];
    if (tk > a && tk < b) {
      double rk = rain_rate(R, tk);
      total += 0.5 * (rr + rk) * (tk - tt);
      tt = tk;
      rr = rk;
    }
  }
  double rb = rain_rate(R, b);
  total += 0.5 * (rr + rb) * (b - tt);
  return total;
}

// Inflow boundaries (Ghost::Inflow, boundary.rs:26-31,45-50,66-71). The inflow cells of a
// grid fall into groups, one per distinct (hydrograph, 1 / segment length) pair; a group's
// discharge per unit width q = rate(t) * inv_len * inflow_scale and its critical depth
// (q^2/g)^(1/3) are the same for all its cells, so they are evaluated once per design and
// step and the cells read them.
constexpr int kMaxInflow = 8;       // groups
constexpr int kMaxInflowPts = 64;   // hydrograph points over all groups

struct Inflow {
  int n;                        // groups (0: no inflow cells)
  int off[kMaxInflow + 1];      // group g's hydrograph points are [off[g], off[g+1])
  double inv_len[kMaxInflow];   // 1 / segment length [1/m]
  double scale;                 // SolverParams::inflow_scale
  double t[kMaxInflowPts];      // time [s]
  double q[kMaxInflowPts];      // discharge [m^3/s]
};

// Real::rcbrt for f64 (crates/itr-core/src/real.rs:81-95): the f32 seed constant moved to
// the f64 exponent and mantissa, then four short-chain Newton steps.
ITR_DEV double rcbrt_d(double x) {
  const unsigned long long K = 0x5540000000000000ull - (0x8782Bull << 29);
  double r = __longlong_as_double((long long)(K - (unsigned long long)__double_as_longlong(x) / 3ull));
  const double third = 1.0 / 3.0;
  const double x3 = x * third;
  const double c43 = 4.0 * third;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    double r2 = r * r;
    r = r * c43 - x3 * (r2 * r2);
  }
  return r;
}

// Hyetograph::rate (scenario.rs:561-570) over points [a, b) of the inflow table; the same
// arithmetic as rain_rate.
ITR_DEV double inflow_rate(const Inflow& F, int a, int b, double x) {
  if (b <= a) return 0.0;
  if (x <= F.t[a]) return F.q[a];
  for (int k = a; k + 1 < b; ++k) {
    if (x <= F.t[k + 1]) {
      double t0 = F.t[k], r0 = F.q[k], t1 = F.t[k + 1], r1 = F.q[k + 1];
      if (t1 == t0) return r1;
      return r0 + (r1 - r0) * (x - t0) / (t1 - t0);
    }
  }
  return F.q[b - 1];
}

// Group g at time t (the start of a step): x = f32 of the discharge per unit width q, and
// y = f32 of the critical depth x * rcbrt(x) * rcbrt(x), x = q^2 / g, in f64 (boundary.rs:
// 27-31). A ghost's depth is f32(max(h, crit)) = max(h, f32(crit)) since rounding is
// monotone and h is already an f32; its normal discharge f32(+-q) = +-f32(q).
ITR_DEV float2 inflow_values(const Inflow& F, int g, double t, double gacc) {
  const double q = inflow_rate(F, F.off[g], F.off[g + 1], t) * F.inv_len[g] * F.scale;
  const double x = q * q / gacc;
  double crit = 0.0;
  if (x > 0.0) {
    const double r = rcbrt_d(x);
    crit = x * r * r;
  }
  return make_float2((float)q, (float)crit);
}

// Ghost state from the interior cell (h, qx, qy) behind it (boundary.rs:36-87), for device
// boundary codes: 0 wall (normal momentum mirrored), 1 transmissive (copy), 2 stage (the
// design's stage depth hstage, momentum copied), 3 + g inflow group g (depth max(h, crit),
// inward normal discharge, zero tangential discharge; inf = inflow_values of the group).
// NX: the ghost lies across an x-normal face (west or east); inward_pos: west or north side.
template <bool NX>
ITR_DEV void ghost_state(int code, float& h, float& qx, float& qy, float hstage, float2 inf, bool inward_pos) {
  if (code == 0) {
    if (NX) qx = -qx; else qy = -qy;
  } else if (code == 2) {
    h = hstage;
  } else if (code >= 3) {
    h = h > inf.y ? h : inf.y;   // NaN h gives the critical depth, as f64::max does
    const float qn = inward_pos ? inf.x : -inf.x;
    if (NX) { qx = qn; qy = 0.0f; } else { qx = 0.0f; qy = qn; }
  }
}

// Ghost wetness of the padded rows for a step whose inflow group values are `inf` (the dry-row
// test of step_fused, kernel.rs:590-612, takes a row with a wet ghost as wet): a stage ghost
// holds water when its depth is > 0, an inflow ghost when the group's critical depth is > 0;
// wall and transmissive ghosts copy their interior cell, so they hold water only beside a wet
// row and need no flag. gw[j], j = 0 .. ny + 1 (0 and ny + 1: the north and south ghost rows,
// 1 .. ny: the west and east ghosts of grid row j - 1). bc: device codes (2 stage, 3 + group
// inflow) north[nx], south[nx], west[ny], east[ny]; bh: stage depths indexed like bc (or NULL).
// One warp, all 32 lanes.
ITR_DEV void ghost_row_wet(const uint8_t* bc, int nx, int ny, const float* bh, const float2* inf, uint8_t* gw, int lane) {
  auto wet = [&](int p) -> bool {
    const int code = bc[p];
    return (code == 2 && bh && bh[p] > 0.0f) || (code >= 3 && inf[code - 3].y > 0.0f);
  };
  for (int e = 0; e < 2; ++e) {   // the north and south ghost rows
    bool w = false;
    for (int c = lane; c < nx; c += 32) w = w || wet(e * nx + c);
    w = __any_sync(0xffffffffu, w);
    if (lane == 0) gw[e == 0 ? 0 : ny + 1] = w ? 1 : 0;
  }
  for (int j = 1 + lane; j <= ny; j += 32) gw[j] = (wet(2 * nx + j - 1) || wet(2 * nx + ny + j - 1)) ? 1 : 0;
}

// Run-wide scalars of one call.
struct RunParams {
  double duration, sync, cfl, dt_max, h_dry, h_eps, infil, initial_depth;
  double dx, dy, g, area, wet_count;
  uint32_t n_sync;
  int skip_dry;
  int rain_sorted;   // breakpoints non-decreasing in time
  int rain_pieces;   // ... and all numbers within div_rn's range: one piece at a time is the general integral's bits
  Rain rain;
  Inflow inflow;
  // step-invariant f32 constants (solver.rs:269-285), rounded once on the host
  float g_f, g_half_f, inv_dx_f, inv_dy_f, h_dry_f, heps2_f, q_min_f;
  double rdx, rdy;   // 1 / dx, 1 / dy rounded (div_rn)
  float nz;   // -0.0f, supplied at run time (see mul2)
  unsigned adj_scalar;   // 1: the adjoint's divisors leave the range of Fast::div (its backward steps take Exact)
  float s_safe;   // largest wave rate of a state whose step may take the branch-free roots (safe_rate_limit)
};

// Whether a state with this largest wave rate (|u| + c) / dx + (|v| + c) / dy is bounded (NaN is not).
ITR_DEV bool state_safe(const RunParams& P, float smax) { return smax <= P.s_safe; }
// The same of an initial depth (at rest): finite, not negative (-0 neither), celerity within the limit.
ITR_DEV bool depth_safe(const RunParams& P, float h) {
  return !(__float_as_uint(h) >> 31) && sqrtf(P.g_f * h) * (P.inv_dx_f + P.inv_dy_f) <= P.s_safe;
}
// A crest jump is a height above a cell; a negative one would deepen the water.
ITR_DEV bool jump_safe(float d) { return !(d < 0.0f); }
// A stage ghost's depth (boundary code 2): 0, or not so small that the momentum it copies becomes a huge velocity.
ITR_DEV bool stage_safe(int code, float hs) { return code != 2 || hs == 0.0f || (hs >= 0x1p-15f && hs <= 1024.0f); }

ITR_DEV double dmin_num(double a, double b) { return a < b ? a : b; }  // operands never NaN here

// One step's scalar schedule from the previous state of the integrator.
struct StepPlan {
  double dt, t_new, rain;
  bool hits;
};

// The step's schedule (solver.rs:449-489) as straight-line arithmetic. dt_pick: the dt before the clip to
// the sync instant t_sync (t_hit: the start from which a step is clipped). The rate at the
// step's start is known from the step before; while no breakpoint lies inside the step the integral is
// one trapezoid of the piece `seg`, else (or for a storm that is not sorted, or whose numbers leave div_rn's
// range: RunParams::rain_pieces) `rare` is set and the general integral replaces s.rain.
ITR_DEV double rain_piece(const RainSeg& g, double x) { return g.r0 + div_rn(g.dr * (x - g.t0), g.den, g.rden); }
ITR_DEV StepPlan plan_step_fast(const RunParams& P, double t, double t_sync, double t_hit, double dt_pick, double rate_t, int seg,
                                bool& rare) {
  StepPlan s;
  s.hits = t + dt_pick >= t_hit;
  s.dt = s.hits ? t_sync - t : dt_pick;
  const double b = t + s.dt;
  s.rain = 0.5 * (rate_t + rain_piece(P.rain.seg[seg], b)) * (b - t);
  rare = b > P.rain.seg[seg].end || !P.rain_pieces;
  s.t_new = s.hits ? t_sync : b;
  return s;
}

// Per-step constants from the host-rounded invariants and this step's dt and rain.
// BOUNDED: a step whose state and parameters are known to be bounded (StepK::exact 0), and with them dt, dx and dy.
template <bool BOUNDED = false>
ITR_DEV StepK step_consts(const RunParams& P, double dt, double rain) {
  StepK k;
  k.g = P.g_f; k.g_half = P.g_half_f; k.inv_dx = P.inv_dx_f; k.inv_dy = P.inv_dy_f;
  k.h_dry = P.h_dry_f; k.heps2 = P.heps2_f; k.q_min = P.q_min_f;
  k.dt = (float)dt;
  const bool bounded = BOUNDED || P.s_safe >= 0.0f;   // (div_rn's range)
  k.dtdx = (float)(bounded ? div_rn(dt, P.dx, P.rdx) : dt / P.dx);
  k.dtdy = (float)(bounded ? div_rn(dt, P.dy, P.rdy) : dt / P.dy);
  k.rain = (float)rain;
  k.cap = (float)(P.infil * dt);
  k.nz = P.nz;
  k.exact = 0u;
  return k;
}

// Objective on the device (objective.rs:94-149), for the incumbent abort and J.
struct DevObjective {
  int n_assets;
  const int* asset_off;
  const int* asset_pos;
  const double* asset_thr;
  const double* asset_w;
  int n_guard;
  const int* guard_pos;
  const double* baseline;  // per monitor or null
  double tol, tau, cut_cost, fill_cost, earth_w;
  int require, guard_abort, has_incumbent;
  double incumbent;
  int enabled;
};

// Per-design scalar results written by the kernels.
// A design's warm start (Solver::run_impl from a Checkpoint, solver.rs:354-378): the
// baseline's state at a checkpoint and its integrator there. state == NULL: cold start.
struct WarmStart {
  const float* state;   // [4][nx*ny]: h, qx, qy, running peak depth
  double t, dt_cfl, acc_rain, v0, volume, rel_res;
  double tot_infil, tot_fix, tot_in, tot_out;   // ledger totals (infil, fix per unit area)
  unsigned long long step;
  unsigned sync_index;
  int n_rows;
};

struct DesignOut {
  unsigned long long steps;
  double t_end;
  unsigned int sync_count;
  int status;
  unsigned int breach_cell;
  unsigned int breach_sync;
  double violation;
  double lower_bound;
  double v0;
  double volume;
  double rel_residual;
  int n_rows;
  int pad;
  unsigned long long rows_skipped;   // dry rows skipped (kernel.rs:605-612)
};

}  // namespace itr

// --------------------------------------------------------------- two cells at once ----
// The same arithmetic on pairs of cells: adds and multiplies are paired FP32 instructions,
// compares, selects and the estimates behind square roots and reciprocals are done per
// component. Association order is the scalar code's, so each component has the same bits as the
// scalar path (and as the reference's f32 kernel).
//
// Two forms. The *_exact functions call the scalar path, right for every input. The others run
// branch-free square roots and reciprocals whose operands must lie in stated ranges; a kernel
// takes them for a whole step when StepK::exact is 0, which the integrator sets only when the
// state it starts from and the run's parameters are bounded (safe_rate_limit below).
namespace itr {

struct B2 { bool x, y; };
struct Face2 { float2 m, nl, nr, t; };

ITR_DEV float2 f2(float a) { return make_float2(a, a); }
// Packed FP32 pairs through PTX with an explicit .rn rounding modifier.
ITR_DEV unsigned long long pk2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
ITR_DEV float2 upk2(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
ITR_DEV float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk2(a)), "l"(pk2(b)));
  return upk2(r);
}
ITR_DEV float2 sub2(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk2(a)), "l"(pk2(b)));
  return upk2(r);
}
// Paired product as fma(a, b, -0): exactly round(a*b) for every input (x + -0 == x, zeros
// keep their sign). mul.rn.f32x2 followed by an add is fused on sm_100a in spite of its .rn
// (measured: 42 % of random a*b+c differ from the twice-rounded value), and so is an fma whose
// -0 is a compile-time constant; -0 is therefore the kernel parameter StepK::nz.
ITR_DEV float2 mul2(float2 a, float2 b, float nz) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk2(a)), "l"(pk2(b)), "l"(pk2(make_float2(nz, nz))));
  return upk2(r);
}
// The plain paired product, for results that no addition reads (only products, estimates and
// selects of these) and for exact ones (a power of two), where fusing changes nothing.
ITR_DEV float2 mulp2(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk2(a)), "l"(pk2(b)));
  return upk2(r);
}
ITR_DEV float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk2(a)), "l"(pk2(b)), "l"(pk2(c)));
  return upk2(r);
}
// Products, sums and fused products with a constant or a value shared by all lanes, per component: the
// pair instruction would hold the constant in a register pair of each lane.
ITR_DEV float2 mulc2(float c, float2 a) { return make_float2(__fmul_rn(c, a.x), __fmul_rn(c, a.y)); }
ITR_DEV float2 addc2(float2 a, float c) { return make_float2(__fadd_rn(a.x, c), __fadd_rn(a.y, c)); }
ITR_DEV float2 fmac2(float c, float2 a, float2 b) { return make_float2(__fmaf_rn(c, a.x, b.x), __fmaf_rn(c, a.y, b.y)); }
ITR_DEV float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
ITR_DEV float2 sel2(B2 c, float2 a, float2 b) { return make_float2(c.x ? a.x : b.x, c.y ? a.y : b.y); }
ITR_DEV float2 max2(float2 a, float2 b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
ITR_DEV float2 min2(float2 a, float2 b) { return make_float2(fminf(a.x, b.x), fminf(a.y, b.y)); }
// max(a, 0) with the reference's NaN rule (a > 0 ? a : 0): the hardware maximum with +0 gives
// the same bits for all 2^32 inputs of each component.
ITR_DEV float2 max2z(float2 a) { return make_float2(fmaxf(a.x, 0.0f), fmaxf(a.y, 0.0f)); }
ITR_DEV B2 gt2(float2 a, float b) { return B2{a.x > b, a.y > b}; }

// 1/x for |x| in [2^-125, 2^126): one Newton step from the hardware estimate (textbook FMA
// refinement: P. Markstein, IBM J. Res. Dev. 34(1), 1990; J.-M. Muller et al., Handbook of
// Floating-Point Arithmetic, 2nd ed., 2018, ch. 4): y = est(1/x); e = fma(-x, y, 1); y + y e.
// Equal to CUDA's IEEE reciprocal on every 32-bit input of that range (tests/test_special_ops.py).
ITR_DEV float2 rcp2(float2 x) {
  const float2 y = make_float2(rcp_est(x.x), rcp_est(x.y));
  const float2 e = make_float2(__fmaf_rn(-x.x, y.x, 1.0f), __fmaf_rn(-x.y, y.y, 1.0f));
  return fma2(y, e, y);
}
// sqrt(x) for x = +0 or x in [2^-149, 2^80): one Newton step from the hardware estimate of
// 1/sqrt (same sources: s = x y, d = fma(-s, s, x), s + d (y / 2)), on x 2^48 so that the
// residual d is exact for the smallest subnormals too (wetting fronts have depths down to them).
// The 2^-126 added for the estimate alone keeps it finite at 0 and vanishes in rounding
// elsewhere. Equal to CUDA's IEEE square root on every 32-bit input of that range (tests/test_special_ops.py);
// about half its time, and without the branch that would end the basic block.
ITR_DEV float2 sqrt2(float2 x) {
  const float2 xs = mulc2(0x1p48f, x);
  const float2 xt = addc2(xs, 0x1p-126f);
  const float2 y = make_float2(rsqrt_est(xt.x), rsqrt_est(xt.y));
  const float2 s = mulp2(xs, y), h = mulc2(0x1p-25f, y);
  return fma2(fma2(neg2(s), s, xs), h, mulc2(0x1p-24f, s));
}

ITR_DEV float2 rcbrt2(float2 x, float nz) {
  float2 r = make_float2(__uint_as_float(0x54A23280u - __float_as_uint(x.x) / 3u),
                         __uint_as_float(0x54A23280u - __float_as_uint(x.y) / 3u));
  const float2 x3 = mulc2((float)(1.0 / 3.0), x);
  const float c43 = (float)(4.0 * (1.0 / 3.0));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float2 r2 = mulp2(r, r);
    r = sub2(mulc2(c43, r), mul2(x3, mulp2(r2, r2), nz));
  }
  return r;
}

// hll (numerics.rs:56-93) on two faces with finite, bounded states. Three places differ from the
// scalar text and give the same bits: 0.5 a + b and 2 a + b as one fma (the product is exact
// unless |a| < 2^-125, where it vanishes beside b: a wet side's celerity is above 2^-73); min and
// max as instructions (the sign of a zero wave speed is not read); and no test for two dry
// sides: their celerities are 0, so the wave speeds are equal and one of the upwind fluxes, a
// zero, is taken (its sign is lost in the cell update, whose states are never -0).
ITR_DEV Face2 hll2(float2 hl, float2 ul, float2 tl, float2 cl, float2 hr, float2 ur, float2 tr, float2 cr, float g_half, float nz) {
  const float NZ = nz;
  const B2 wet_l = gt2(hl, 0.0f), wet_r = gt2(hr, 0.0f);
  const float2 ustar = sub2(fmac2(0.5f, add2(ul, ur), cl), cr);
  const float2 cstar = fmac2(0.25f, sub2(ul, ur), mulc2(0.5f, add2(cl, cr)));
  const float2 ul_cl = sub2(ul, cl);
  const float2 ur_cr = add2(ur, cr);
  const float2 slw = min2(ul_cl, sub2(ustar, cstar));
  const float2 srw = max2(ur_cr, add2(ustar, cstar));
  const float2 sl = sel2(wet_l, sel2(wet_r, slw, ul_cl), fmac2(-2.0f, cr, ur));
  const float2 sr = sel2(wet_l, sel2(wet_r, srw, fmac2(2.0f, cl, ul)), ur_cr);
  const float2 ml = mul2(hl, ul, NZ);
  const float2 mr = mul2(hr, ur, NZ);
  const float2 pl_ = mul2(mulc2(g_half, hl), hl, NZ);
  const float2 pr_ = mul2(mulc2(g_half, hr), hr, NZ);
  const float2 pl = add2(mul2(ml, ul, NZ), pl_);
  const float2 pr = add2(mul2(mr, ur, NZ), pr_);
  const B2 use_l = B2{sl.x >= 0.0f, sl.y >= 0.0f}, use_r = B2{sr.x <= 0.0f, sr.y <= 0.0f};
  const float2 inv = rcp2(sub2(sr, sl));   // (not read where an upwind flux is taken)
  const float2 slsr = mulp2(sl, sr);
  const float2 fm_star = mul2(add2(sub2(mul2(sr, ml, NZ), mul2(sl, mr, NZ)), mul2(slsr, sub2(hr, hl), NZ)), inv, NZ);
  const float2 fn_star = mul2(add2(sub2(mul2(sr, pl, NZ), mul2(sl, pr, NZ)), mul2(slsr, sub2(mr, ml), NZ)), inv, NZ);
  const float2 fm = sel2(use_l, ml, sel2(use_r, mr, fm_star));
  const float2 fn = sel2(use_l, pl, sel2(use_r, pr, fn_star));
  Face2 f;
  f.m = fm;
  f.nl = sub2(fn, pl_);
  f.nr = sub2(fn, pr_);
  f.t = mul2(fm, sel2(gt2(fm, 0.0f), tl, tr), NZ);
  return f;
}

// face_signed / face_crest (numerics.rs:95-129) on two faces; (ul,vl,cl) of the low side.
template <bool NORMAL_X, bool CREST>
ITR_DEV Face2 face2(float2 hl, float2 ul, float2 vl, float2 cl, float2 hr, float2 ur, float2 vr, float2 cr,
                    float2 d0, float2 d1, const StepK& k) {
  const float NZ = k.nz;
  float2 hsl, hsr, csl, csr;
  if (!CREST) {
    const B2 pos = gt2(d0, 0.0f);
    hsl = max2z(sub2(hl, max2z(d0)));
    hsr = max2z(sub2(hr, max2z(neg2(d0))));
    const float2 cred = sqrt2(mulc2(k.g, sel2(pos, hsl, hsr)));
    csl = sel2(pos, cred, cl);
    csr = sel2(pos, cr, cred);
  } else {
    hsl = max2z(sub2(hl, d0));
    hsr = max2z(sub2(hr, d1));
    const B2 pl = gt2(d0, 0.0f), pr = gt2(d1, 0.0f);
    const float2 sl = sqrt2(mulc2(k.g, hsl)), sr = sqrt2(mulc2(k.g, hsr));
    csl = sel2(pl, sl, cl);
    csr = sel2(pr, sr, cr);
  }
  if (NORMAL_X) return hll2(hsl, ul, vl, csl, hsr, ur, vr, csr, k.g_half, NZ);
  return hll2(hsl, vl, ul, csl, hsr, vr, ur, csr, k.g_half, NZ);
}

// low: the depth before the positivity fix; a cell is unhealthy when low < -h_dry.
struct CellNew2 {
  float2 h, qx, qy, s, infil, fix, c, low;
};

// The step's dt / dx, dt / dy and the grid's 1 / dx, 1 / dy per component: 0 for a component whose
// cell stays as it is and adds nothing to the step's sums (a lane's idle columns).
struct UpdK { float2 dtdx, dtdy, inv_dx, inv_dy; };

// flux_update then sources (numerics.rs:144-195) on two cells with finite, bounded states.
// Momentum: the reference multiplies by keep = 0 where the new depth is below h_dry and then
// flushes |q| < q_min to 0; both are one select here (a dry cell's q is 0 either way).
ITR_DEV CellNew2 update_cell2(float2 h, float2 qx, float2 qy, const Face2& w, const Face2& e, const Face2& n,
                              const Face2& s, float2 wet, float2 gn2, const StepK& k, const UpdK& uk) {
  const float NZ = k.nz;
  const float2 dtdx = uk.dtdx, dtdy = uk.dtdy;
  CellNew2 o;
  const float2 h1 = sub2(sub2(h, mul2(dtdx, sub2(e.m, w.m), NZ)), mul2(dtdy, sub2(s.m, n.m), NZ));
  const float2 qx1 = sub2(sub2(qx, mul2(dtdx, sub2(e.nl, w.nr), NZ)), mul2(dtdy, sub2(s.t, n.t), NZ));
  const float2 qy1 = sub2(sub2(qy, mul2(dtdx, sub2(e.t, w.t), NZ)), mul2(dtdy, sub2(s.nl, n.nr), NZ));
  o.low = h1;
  const float2 hc = max2z(h1);
  o.fix = sub2(hc, h1);
  const float2 h2 = add2(hc, mulc2(k.rain, wet));
  o.infil = min2(mulc2(k.cap, wet), h2);
  const float2 h3 = sub2(h2, o.infil);
  const B2 dry = B2{h3.x < k.h_dry, h3.y < k.h_dry};
  const float2 r = rcbrt2(sel2(dry, f2(1.0f), h3), NZ);
  const float2 r3 = mulp2(mulp2(r, r), r);
  const float2 r7 = mulp2(mulp2(r3, r3), r);
  const float2 qm = sqrt2(add2(mul2(qx1, qx1, NZ), mul2(qy1, qy1, NZ)));
  const float2 inv = rcp2(addc2(mul2(mulp2(mulc2(k.dt, gn2), qm), r7, NZ), 1.0f));
  const float2 tx = mulp2(qx1, inv), ty = mulp2(qy1, inv);
  o.qx = make_float2(fabsf(tx.x) >= k.q_min && !dry.x ? tx.x : 0.0f, fabsf(tx.y) >= k.q_min && !dry.y ? tx.y : 0.0f);
  o.qy = make_float2(fabsf(ty.x) >= k.q_min && !dry.x ? ty.x : 0.0f, fabsf(ty.y) >= k.q_min && !dry.y ? ty.y : 0.0f);
  const float2 c = sqrt2(mulc2(k.g, h3));
  const float2 ax = mul2(o.qx, r3, NZ), ay = mul2(o.qy, r3, NZ);   // |q| r3 = |q r3|
  const float2 sx = make_float2(fabsf(ax.x) + c.x, fabsf(ax.y) + c.y), sy = make_float2(fabsf(ay.x) + c.x, fabsf(ay.y) + c.y);
  o.s = add2(mul2(sx, uk.inv_dx, NZ), mul2(sy, uk.inv_dy, NZ));
  o.h = addc2(h3, 0.0f);   // canon: -0 becomes +0
  o.c = c;
  return o;
}

// Paired desingularised velocity and celerity (cell_vel on two cells).
ITR_DEV void vel2(float2 h, float2 qx, float2 qy, const StepK& k, float2& u, float2& v) {
  const float2 h2 = mul2(h, h, k.nz);
  const float2 t = mulp2(add2(h, h), rcp2(add2(h2, make_float2(fmaxf(h2.x, k.heps2), fmaxf(h2.y, k.heps2)))));
  u = mul2(qx, t, k.nz);
  v = mul2(qy, t, k.nz);
}
ITR_DEV float2 cel2(float2 h, const StepK& k) { return sqrt2(mulc2(k.g, h)); }

// The same through the scalar path, for steps with StepK::exact set (rare: not inlined).
ITR_DEV Face2 face2_of(const FaceF& a, const FaceF& b) {
  Face2 f;
  f.m = make_float2(a.m, b.m); f.nl = make_float2(a.nl, b.nl); f.nr = make_float2(a.nr, b.nr); f.t = make_float2(a.t, b.t);
  return f;
}
ITR_DEV FaceF fx_(const Face2& f) { FaceF r; r.m = f.m.x; r.nl = f.nl.x; r.nr = f.nr.x; r.t = f.t.x; return r; }
ITR_DEV FaceF fy_(const Face2& f) { FaceF r; r.m = f.m.y; r.nl = f.nl.y; r.nr = f.nr.y; r.t = f.t.y; return r; }

template <bool NORMAL_X, bool CREST>
__device__ __noinline__ Face2 face2_exact(float2 hl, float2 ul, float2 vl, float2 cl, float2 hr, float2 ur, float2 vr, float2 cr,
                                          float2 d0, float2 d1, StepK k) {
  return face2_of(face<NORMAL_X, CREST>(hl.x, ul.x, vl.x, cl.x, hr.x, ur.x, vr.x, cr.x, d0.x, d1.x, k),
                  face<NORMAL_X, CREST>(hl.y, ul.y, vl.y, cl.y, hr.y, ur.y, vr.y, cr.y, d0.y, d1.y, k));
}
// low: -infinity for an unhealthy cell (a NaN is not below -h_dry).
static __device__ __noinline__ CellNew2 update_cell2_exact(float2 h, float2 qx, float2 qy, Face2 w, Face2 e, Face2 n, Face2 s,
                                                           float2 wet, float2 gn2, StepK k) {
  const CellNew a = update_cell(h.x, qx.x, qy.x, fx_(w), fx_(e), fx_(n), fx_(s), wet.x, gn2.x, k);
  const CellNew b = update_cell(h.y, qx.y, qy.y, fy_(w), fy_(e), fy_(n), fy_(s), wet.y, gn2.y, k);
  CellNew2 o;
  o.h = make_float2(a.h, b.h); o.qx = make_float2(a.qx, b.qx); o.qy = make_float2(a.qy, b.qy); o.s = make_float2(a.s, b.s);
  o.infil = make_float2(a.infil, b.infil); o.fix = make_float2(a.fix, b.fix); o.c = make_float2(a.c, b.c);
  const float inf = __int_as_float(0x7f800000);
  o.low = make_float2(a.bad ? -inf : 0.0f, b.bad ? -inf : 0.0f);
  return o;
}
struct Vel2 { float2 u, v, c; };
static __device__ __noinline__ Vel2 vel2_exact(float2 h, float2 qx, float2 qy, float g, float heps2) {
  Vel2 o;
  cell_vel(h.x, qx.x, qy.x, g, heps2, o.u.x, o.v.x, o.c.x);
  cell_vel(h.y, qx.y, qy.y, g, heps2, o.u.y, o.v.y, o.c.y);
  return o;
}

}  // namespace itr
