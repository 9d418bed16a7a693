// itr_band.cuh — forward step for grids whose state lives in HBM: a row-band sweep.
//
// The design's state stays in the ping-pong planes of the tiled path (PlainArgs: H, QX, QY
// [2][nx*ny], running peaks PK), the integrator in its control block (PlainCtl, advanced by
// plain_finalize_body in the last block, or by k_plain_finalize_locked); only the per-step update differs from k_plain_update. It is the row
// sweep of the cluster kernel (itr_batched.cuh) and of the reference's fused CPU kernel
// (crates/itr-hydro/src/kernel.rs:637-697), laid out for a state that is read from HBM:
//   * a warp owns a segment of 64 columns of a band of kBandRows rows; lane l holds the two
//     adjacent columns 64 s + 2 l and 64 s + 2 l + 1, whose faces and cell updates run as
//     paired FP32 instructions (face2 / update_cell2), every value bit-identical to the
//     scalar arithmetic;
//   * each face is computed once: the west x-face of each column and the south y-face of
//     each row of the band, the north y-face of a row carried in registers from the row
//     above. The east face of a column is the next column's west face (own register or a
//     shuffle from lane + 1). The two x-faces on the segment's edges (columns 64 s and
//     64 s + 64) are computed by the warp for all rows of the band at once before the sweep
//     (one paired face per lane) and kept in shared memory, so no warp waits on another;
//     the only faces computed twice are those edges and the band's top y-face row:
//     (1 + 1/32) x (1 + 1/64) of the faces, against 1.27 for a 16x16 tile with an 18x18 halo;
//   * velocities and celerity of a cell are computed once per step, when its row is loaded;
//   * the old state is read-only during a step (ping-pong), so warps never synchronise with
//     each other inside a step: row r + 1 is loaded while row r is updated, and the only
//     block barrier is the final reduction of the per-block partials.
// What bounds it: the row arithmetic, issue and dependent instructions at 12 warps an SM (61 % of the issue
// slots; a step of 16 designs of 1024 x 1024 moves 48 B per cell in 0.30 ms, 2.7 TB/s). So a row's inputs come as two records
// (jumps, wet | g n^2) of 16 B per pair, the columns past the grid are masked once per step instead of
// once per row, a row's ghosts are filled in when it is used (filled in at the load they made every
// row wait for memory: 285 ms against 238 ms of 16 designs x 959 steps; the layout with separate arrays
// took 256 ms), and the last block of a design advances its integrator, so that a step is one
// launch: one design of 1024 x 1024, 681 steps, 21.5 ms -> 19.3 ms.
// Outputs are k_plain_update's: the new plane, PK (and the argmax state index tpk), the
// per-block partials [kPart] in the finalize's layout, and the atomic smax / bad words.
// TAPE: the adjoint's replay of a recorded step (itr_adjoint_band.cuh): the same update, writing
// only the new plane (no peaks, partials, CFL maximum, health word or row flags).
#pragma once
#include <cmath>
#include "itr_plain.cuh"
#include "itr_batched.cuh"

namespace itr {

constexpr int kBandRows = 32;    // most rows per band (= lanes: one pre-pass edge face per lane)
constexpr int kBandWarps = 4;    // warps (64-column segments) per block

struct BandGeom {
  int ns;      // 64-column segments per row
  int wpb;     // warps per block
  int rows;    // rows per band
  int gx, gy;  // blocks per design: segment groups x bands
};

__host__ __device__ inline BandGeom band_geom(int nx, int ny, int rows) {
  BandGeom b;
  b.ns = (nx + 63) / 64;
  b.wpb = b.ns < kBandWarps ? b.ns : kBandWarps;
  b.rows = rows;
  b.gx = (b.ns + b.wpb - 1) / b.wpb;
  b.gy = (ny + rows - 1) / rows;
  return b;
}

// Rows per band. Every warp sweeps one band segment, all warps about equally long, so a launch
// takes ceil(warps / resident) rounds of the SMs (12 warps resident per SM: 3 blocks of 4
// warps, the register budget at which nothing spills, measured 7-8 % faster than 4 blocks
// with spills). The chosen height maximises the busy fraction of those rounds times
// R / (R + 1), the share of y-faces computed once (each band recomputes its top y-face row).
inline int band_rows_for(int nx, int ny, int n_designs, int sm_count) {
  const double resident = 12.0 * (sm_count > 0 ? sm_count : 148);
  int best = kBandRows;
  double best_score = -1.0;
  for (int rows = kBandRows; rows >= 6; --rows) {
    const BandGeom b = band_geom(nx, ny, rows);
    const double warps = (double)n_designs * b.ns * b.gy;
    const double rounds = std::ceil(warps / resident);
    const double score = warps / (rounds * resident) * rows / (rows + 1.0);
    if (score > best_score + 1e-9) { best_score = score; best = rows; }
  }
  return best;
}

// A row's pair of cells with its velocities and celerity. EX: through the scalar path.
template <bool EX>
ITR_DEV Cell2 cells_of(float2 h, float2 qx, float2 qy, const StepK& k) {
  Cell2 r;
  r.h = h; r.qx = qx; r.qy = qy;
  if constexpr (EX) {
    const Vel2 w = vel2_exact(h, qx, qy, k.g, k.heps2);
    r.u = w.u; r.v = w.v; r.c = w.c;
  } else {
    vel2(h, qx, qy, k, r.u, r.v);
    r.c = cel2(h, k);
  }
  return r;
}
template <bool EX, bool NORMAL_X, bool CREST>
ITR_DEV Face2 band_face(const Cell2& a, const Cell2& b, float2 d0, float2 d1, const StepK& k) {
  if constexpr (EX) return face2_exact<NORMAL_X, CREST>(a.h, a.u, a.v, a.c, b.h, b.u, b.v, b.c, d0, d1, k);
  else return face2<NORMAL_X, CREST>(a.h, a.u, a.v, a.c, b.h, b.u, b.v, b.c, d0, d1, k);
}

// Old state of cell (r, c) of the design; c == nx gives the east ghost of (r, nx - 1), c == -1
// the west ghost of (r, 0), r == -1 / ny the north / south ghost of (0, c) / (ny - 1, c)
// (boundary.rs:36-87; BND: stage and inflow ghosts through ghost_state). Anything else
// outside the grid (lanes past the last column) is still water on a flat bed.
template <bool BND>
ITR_DEV void band_cell(const PlainArgs& A, const PlainDesign& D, const float2* inf, size_t plane, int r, int c, float& h,
                       float& qx, float& qy) {
  const int nx = A.nx, ny = A.ny;
  h = 0.0f; qx = 0.0f; qy = 0.0f;
  const bool gxw = c == -1, gxe = c == nx, gyn = r == -1, gys = r == ny;
  if (c < -1 || c > nx || r < -1 || r > ny || ((gxw || gxe) && (gyn || gys))) return;
  const int sr = gyn ? 0 : (gys ? ny - 1 : r), sc = gxw ? 0 : (gxe ? nx - 1 : c);
  const size_t i = plane + (size_t)sr * nx + sc;
  h = D.H[i]; qx = D.QX[i]; qy = D.QY[i];
  if (!(gxw || gxe || gyn || gys)) return;
  const int p = gxw ? 2 * nx + sr : gxe ? 2 * nx + ny + sr : gyn ? sc : nx + sc;
  const int code = A.bc[p];
  if (!BND) {
    if (code == 0) { if (gxw || gxe) qx = -qx; else qy = -qy; }
    return;
  }
  const float hs = code == 2 ? D.bh[p] : 0.0f;
  const float2 fi = code >= 3 ? inf[code - 3] : make_float2(0.0f, 0.0f);
  if (gxw || gxe) ghost_state<true>(code, h, qx, qy, hs, fi, gxw);
  else ghost_state<false>(code, h, qx, qy, hs, fi, gyn);
}

// Raw (not yet velocity-complemented) state of the lane's two cells of a row.
struct Raw2 { float2 h, qx, qy; };

// Sums of one warp's sweep (one step): the finalize's partials, the largest wave rate, the lowest
// depth before the positivity fix, and whether a cell left the bounds of the branch-free step
// (looked for on the scalar path only: a step from a bounded state stays finite, and its largest
// wave rate tells).
struct BandAcc {
  float smax = 0.0f, low = 0.0f;
  bool uns = false;
  double infil = 0.0, fix = 0.0, in = 0.0, out = 0.0, vol = 0.0, ytop = 0.0, ybot = 0.0;
};

// A warp's segment of one band. EX: every root and reciprocal through the scalar path (k.exact).
// SKIP: with the dry-row test (only launched where the storm leaves a rain-free step).
template <bool EX, bool CREST, bool BND, bool TAPE, bool SKIP>
ITR_DEV void band_sweep(const PlainArgs& A, const PlainDesign& D, const PlainCtl& cl, const StepK& k, int d, int s, int r0, int r1,
                        float4* edge_w, float4* edge_e, BandAcc& acc) {
  const int par = cl.par;
  const bool hits = cl.pl.hits;
  const double dt_dy = cl.pl.dt * A.P.dy;
  const int nx = A.nx, ny = A.ny, nxp1 = nx + 1;
  const size_t N = (size_t)nx * ny, plane = A.plane_stride ? A.plane_stride : N;
  const size_t pin = (size_t)par * plane, pout = (size_t)(par ^ 1) * plane;
  const float2* inf = cl.inf;
  const int lane = threadIdx.x & 31;
  const int L = r1 - r0;
  const int cw = 64 * s, ce = cw + 64;              // the segment's edge x-faces
  // The lane's pair of columns; a pair past the grid reads the last one, whose mirror is the east ghost.
  const int P2 = pairs(nx), PJ = P2 + 2, p = 32 * s + lane, pl = p < P2 ? p : P2 - 1;
  const int c0 = 2 * p;
  const bool even = (nx & 1) == 0;                   // pairs are 8-byte aligned in every plane
  const bool v0 = p < P2, v1 = c0 + 1 < nx;         // cells of the lane
  const bool y_in = 2 * pl + 1 < nx;                 // the pair read has two cells
  const bool mir_x = even && p >= P2, mir_y = !even && p >= P2 - 1;   // ghost from the pair's other column
  const bool edge = mir_x || mir_y;
  const bool last_seg = ce > nx;                    // the east domain edge lies inside this segment
  const float2 mask = make_float2(v0 ? 1.0f : 0.0f, v1 ? 1.0f : 0.0f);
  const int jr = p + 1 <= P2 + 1 ? p + 1 : 0, gr = v0 ? p + 1 : 0;    // the pair's records (0: zeros)
  const float4* const Jl = A.J + (size_t)d * (ny + 1) * PJ + jr;
  const float4* const J2l = CREST ? A.J2 + (size_t)d * (ny + 1) * PJ + jr : nullptr;
  const float4* const Gl = A.G + gr;

  // Dry-row skipping (kernel.rs:605-612): with no rain this step, grid row r is skipped when
  // padded rows r, r + 1, r + 2 (grid rows r - 1, r, r + 1 and their ghosts) held no water
  // in the old state. Its faces are then exactly 0 and its cells keep their (zero) state, so
  // skipping changes no result. Bit p of skipm: grid row r0 + p; bit i of m: padded row r0 + i.
  unsigned long long skipm = 0ull;
  const unsigned* rw_old = SKIP ? D.rowwet + (size_t)par * (ny + 2) : nullptr;
  unsigned* rw_new = SKIP ? D.rowwet + (size_t)(par ^ 1) * (ny + 2) : nullptr;
  if (SKIP && !(k.rain > 0.0f)) {
    const int ja = r0 + lane, jb = r0 + 32 + lane;
    const bool da = ja <= ny + 1 && plain_row_dry(rw_old, D.gwet, ja);
    const bool db = lane < 2 && jb <= ny + 1 && plain_row_dry(rw_old, D.gwet, jb);
    const unsigned long long m =
        (unsigned long long)__ballot_sync(0xffffffffu, da) | ((unsigned long long)__ballot_sync(0xffffffffu, db) << 32);
    skipm = m & (m >> 1) & (m >> 2);
  }
  // Rows the sweep needs: row p is updated unless skipped, and its state and inputs are also
  // read for the next row's west faces; need(p) is false when rows p and p + 1 (or the band's
  // end) are both skipped, and then nothing of row p is loaded.
  auto skipped = [&](int q) -> bool { return SKIP && (q >= L || ((skipm >> q) & 1ull)); };
  auto need = [&](int q) -> bool { return !SKIP || !(skipped(q) && skipped(q + 1)); };

  // A row's raw state: the pair of the nearest grid row, and what the loads leave out (the rows
  // beyond the domain's edges, the column beyond the east edge). The second half waits for the loads, so it
  // runs when the row is used, a row of arithmetic after they were issued.
  auto load_row = [&](int r) -> Raw2 {
    const int rr = r < 0 ? 0 : r >= ny ? ny - 1 : r;
    const size_t i = pin + (size_t)rr * nx + 2 * pl;
    Raw2 o;
    if (even) {
      o.h = *reinterpret_cast<const float2*>(D.H + i);
      o.qx = *reinterpret_cast<const float2*>(D.QX + i);
      o.qy = *reinterpret_cast<const float2*>(D.QY + i);
    } else {
      o.h = make_float2(D.H[i], y_in ? D.H[i + 1] : 0.0f);
      o.qx = make_float2(D.QX[i], y_in ? D.QX[i + 1] : 0.0f);
      o.qy = make_float2(D.QY[i], y_in ? D.QY[i + 1] : 0.0f);
    }
    return o;
  };
  auto ghosts = [&](Raw2& o, int r) {
    if (r < 0 || r >= ny) {   // north or south ghost row (its east ghost is not read)
      for (int e = 0; e < 2; ++e) {
        float &h = e ? o.h.y : o.h.x, &qx = e ? o.qx.y : o.qx.x, &qy = e ? o.qy.y : o.qy.x;
        const int pos = (r < 0 ? 0 : nx) + 2 * pl + e;
        const int code = e == 0 || y_in ? A.bc[pos] : 1;
        const float hs = BND && code == 2 ? D.bh[pos] : 0.0f;
        const float2 fi = BND && code >= 3 ? inf[code - 3] : make_float2(0.0f, 0.0f);
        ghost_state<false>(code, h, qx, qy, hs, fi, r < 0);
      }
    } else if (edge) {
      float h = mir_x ? o.h.y : o.h.x, qx = mir_x ? o.qx.y : o.qx.x, qy = mir_x ? o.qy.y : o.qy.x;
      const int pos = 2 * nx + ny + r, code = A.bc[pos];
      const float hs = BND && code == 2 ? D.bh[pos] : 0.0f;
      const float2 fi = BND && code >= 3 ? inf[code - 3] : make_float2(0.0f, 0.0f);
      ghost_state<true>(code, h, qx, qy, hs, fi, false);
      if (mir_x) { o.h.x = h; o.qx.x = qx; o.qy.x = qy; } else { o.h.y = h; o.qx.y = qx; o.qy.y = qy; }
    }
  };

  // ---- pre-pass: the segment's two edge x-faces of every row of the band (skipped rows:
  //      zero faces, which they are) ----
  {
    const int r = r0 + lane;
    Raw2 lf, rt;
    float2 d0 = f2(0.0f), d1 = f2(0.0f);
    lf.h = lf.qx = lf.qy = rt.h = rt.qx = rt.qy = f2(0.0f);
    if (r < r1 && !skipped(lane)) {
      band_cell<BND>(A, D, inf, pin, r, cw - 1, lf.h.x, lf.qx.x, lf.qy.x);
      band_cell<BND>(A, D, inf, pin, r, cw, rt.h.x, rt.qx.x, rt.qy.x);
      if (ce <= nx) {
        band_cell<BND>(A, D, inf, pin, r, ce - 1, lf.h.y, lf.qx.y, lf.qy.y);
        band_cell<BND>(A, D, inf, pin, r, ce, rt.h.y, rt.qx.y, rt.qy.y);
      }
      const size_t xo = (size_t)r * nxp1;
      d0.x = D.dzx[xo + cw];
      d0.y = ce <= nx ? D.dzx[xo + ce] : 0.0f;
      if (CREST) { d1.x = D.dzx2[xo + cw]; d1.y = ce <= nx ? D.dzx2[xo + ce] : 0.0f; }
    }
    const Cell2 a = cells_of<EX>(lf.h, lf.qx, lf.qy, k), b = cells_of<EX>(rt.h, rt.qx, rt.qy, k);
    const Face2 f = band_face<EX, true, CREST>(a, b, d0, d1, k);
    edge_w[lane] = f4(fx_(f));
    edge_e[lane] = f4(fy_(f));
    // x_boundary (kernel.rs:435-450): the west domain face of every row, per face
    if (!TAPE && s == 0 && r < r1) {
      const double vw = (double)f.m.x * dt_dy;
      if (vw > 0.0) acc.in += vw; else acc.out -= vw;
    }
    if (!TAPE && ce == nx && r < r1) {   // the east domain face is this segment's edge
      const double ve = (double)f.m.y * dt_dy;
      if (ve > 0.0) acc.out += ve; else acc.in -= ve;
    }
  }
  __syncwarp();

  // ---- row sweep ----
  UpdK uk;
  uk.dtdx = mulc2(k.dtdx, mask); uk.dtdy = mulc2(k.dtdy, mask); uk.inv_dx = mulc2(k.inv_dx, mask); uk.inv_dy = mulc2(k.inv_dy, mask);
  auto xfaces = [&](const Cell2& c, float2 j, float2 j2, int q) -> Face2 {
    // west faces of the lane's two columns: (c0 - 1 | c0) and (c0 | c0 + 1); lane 0's first
    // one is the segment's west edge face from the pre-pass
    Cell2 left;
    left.h = west2(c.h); left.u = west2(c.u); left.v = west2(c.v); left.c = west2(c.c);
    left.qx = left.qy = f2(0.0f);
    Face2 f = band_face<EX, true, CREST>(left, c, j, j2, k);
    if (lane == 0) {
      const FaceF w = ff(edge_w[q]);
      f.m.x = w.m; f.nl.x = w.nl; f.nr.x = w.nr; f.t.x = w.t;
    }
    return f;
  };
  const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  Cell2 cur{}, nxt{};
  Face2 fN{}, fW{};
  if (!skipped(0)) {
    Raw2 ta = load_row(r0 - 1), ca = load_row(r0);   // the row above the band and its first
    ghosts(ta, r0 - 1);
    ghosts(ca, r0);
    const Cell2 top = cells_of<EX>(ta.h, ta.qx, ta.qy, k);
    cur = cells_of<EX>(ca.h, ca.qx, ca.qy, k);
    const float4 j = __ldg(Jl + (size_t)r0 * PJ), j2 = CREST ? __ldg(J2l + (size_t)r0 * PJ) : zero4;
    fN = band_face<EX, false, CREST>(top, cur, lo2(j), lo2(j2), k);
    fW = xfaces(cur, hi2(j), hi2(j2), 0);
    if (!TAPE && r0 == 0)   // y_boundary top (kernel.rs:452-472): summed over the row first
      acc.ytop += (v0 ? (double)fN.m.x : 0.0) + (v1 ? (double)fN.m.y : 0.0);
  }
  // inputs of row r, the jumps below it and west of row r + 1
  float4 jn = zero4, jn2 = zero4, gn = zero4;
  float2 pn = f2(0.0f);
  Raw2 raw;
  raw.h = raw.qx = raw.qy = f2(0.0f);
  auto load_in = [&](int r) {
    jn = __ldg(Jl + (size_t)(r + 1) * PJ);
    if (CREST) jn2 = __ldg(J2l + (size_t)(r + 1) * PJ);
    gn = __ldg(Gl + (size_t)r * PJ);
    if (!TAPE) {
      const size_t i = (size_t)r * nx + 2 * pl;
      if (even) pn = *reinterpret_cast<const float2*>(D.PK + i);
      else pn = make_float2(D.PK[i], y_in ? D.PK[i + 1] : 0.0f);
    }
    raw = load_row(r + 1);
  };
  if (need(0)) load_in(r0);
#pragma unroll 1
  for (int q = 0; q < L; ++q) {
    const int r = r0 + q;
    const float4 j = jn, j2 = jn2, g = gn;
    const float2 pk = pn;
    if (need(q)) {
      ghosts(raw, r + 1);
      nxt = cells_of<EX>(raw.h, raw.qx, raw.qy, k);
    }
    if (q + 1 < L && need(q + 1)) load_in(r + 1);   // next row's operands, in flight while this row is updated
    Face2 fWn{};
    const size_t ci = (size_t)r * nx + c0;
    if (SKIP && skipped(q)) {   // a dry row between dry rows: zero faces, the (zero) state carried over
      if (!skipped(q + 1)) fWn = xfaces(nxt, hi2(j), hi2(j2), q + 1);
      if (v0) { D.H[pout + ci] = 0.0f; D.QX[pout + ci] = 0.0f; D.QY[pout + ci] = 0.0f; }
      if (v1) { D.H[pout + ci + 1] = 0.0f; D.QX[pout + ci + 1] = 0.0f; D.QY[pout + ci + 1] = 0.0f; }
      cur = nxt; fN = Face2{}; fW = fWn;
      continue;
    }
    const Face2 fS = band_face<EX, false, CREST>(cur, nxt, lo2(j), lo2(j2), k);
    // (the row after the band's last is faced too, and not read: one straight-line body)
    fWn = xfaces(nxt, hi2(j), hi2(j2), q + 1 < L ? q + 1 : q);
    // east faces: the second column's west face, and lane + 1's first (lane 31: the edge)
    Face2 fE;
    fE.m = east2(fW.m); fE.nl = east2(fW.nl); fE.nr = east2(fW.nr); fE.t = east2(fW.t);
    if (lane == 31) {
      const FaceF e = ff(edge_e[q]);
      fE.m.y = e.m; fE.nl.y = e.nl; fE.nr.y = e.nr; fE.t.y = e.t;
    }
    CellNew2 o;
    if constexpr (EX) {
      o = update_cell2_exact(cur.h, cur.qx, cur.qy, fW, fE, fN, fS, lo2(g), hi2(g), k);
      if (!v0) { o.s.x = o.low.x = o.infil.x = o.fix.x = 0.0f; }   // (idle columns need not be finite here)
      if (!v1) { o.s.y = o.low.y = o.infil.y = o.fix.y = 0.0f; }
      acc.uns = acc.uns || !state_safe(A.P, o.s.x) || !state_safe(A.P, o.s.y);
    } else {
      o = update_cell2(cur.h, cur.qx, cur.qy, fW, fE, fN, fS, lo2(g), hi2(g), k, uk);
    }
    if (even) {
      if (v0) {
        *reinterpret_cast<float2*>(D.H + pout + ci) = o.h;
        *reinterpret_cast<float2*>(D.QX + pout + ci) = o.qx;
        *reinterpret_cast<float2*>(D.QY + pout + ci) = o.qy;
      }
    } else {
      if (v0) { D.H[pout + ci] = o.h.x; D.QX[pout + ci] = o.qx.x; D.QY[pout + ci] = o.qy.x; }
      if (v1) { D.H[pout + ci + 1] = o.h.y; D.QX[pout + ci + 1] = o.qx.y; D.QY[pout + ci + 1] = o.qy.y; }
    }
    if constexpr (!TAPE) {
      const bool up0 = v0 && o.h.x > pk.x, up1 = v1 && o.h.y > pk.y;
      if (up0) D.PK[ci] = o.h.x;
      if (up1) D.PK[ci + 1] = o.h.y;
      if (D.tpk) {   // the state that raised the peak last
        if (up0) D.tpk[ci] = (unsigned)(cl.step + 1);
        if (up1) D.tpk[ci + 1] = (unsigned)(cl.step + 1);
      }
      acc.smax = fmaxf(acc.smax, fmaxf(o.s.x, o.s.y));
      acc.low = fminf(acc.low, fminf(o.low.x, o.low.y));
      // row partials: f32 over the lane's pair, f64 across rows
      acc.infil += (double)(o.infil.x + o.infil.y);
      acc.fix += (double)(o.fix.x + o.fix.y);
      if (hits) acc.vol += (v0 ? (double)o.h.x : 0.0) + (v1 ? (double)o.h.y : 0.0);
      if (last_seg) {   // x_boundary: the east domain face inside this segment (kernel.rs:435-450)
        if (c0 == nx - 1 || c0 == nx - 2) {
          const double ve = (double)(c0 == nx - 1 ? fE.m.x : fE.m.y) * dt_dy;
          if (ve > 0.0) acc.out += ve; else acc.in -= ve;
        }
      }
      if (r == ny - 1) acc.ybot += (v0 ? (double)fS.m.x : 0.0) + (v1 ? (double)fS.m.y : 0.0);
      if (SKIP && __any_sync(0xffffffffu, (v0 && o.h.x > 0.0f) || (v1 && o.h.y > 0.0f)) && lane == 0)
        rw_new[r + 1] = 1u;   // the row holds water in the new state (every writer stores 1)
    }
    cur = nxt; fN = fS; fW = fWn;
  }
}

// One step of every design: bands of rows x groups of segments x designs. fin: the last block of a
// design to finish its band advances the design's integrator (plain_finalize_body), instead of a
// launch of its own.
template <bool CREST, bool BND, bool TAPE, bool SKIP>
__global__ void __launch_bounds__(kBandWarps * 32, 3) k_band(const PlainArgs A, int fin) {
  __shared__ float4 edge_w[kBandWarps][kBandRows], edge_e[kBandWarps][kBandRows];
  __shared__ float wmax[kBandWarps];
  __shared__ unsigned wbad[kBandWarps];
  __shared__ double wsum[kBandWarps][kPart];
  __shared__ unsigned s_last;
  const int nblk = gridDim.x * gridDim.y, d = blockIdx.z;
  const PlainDesign D = plain_design(A, d, nblk);
  const PlainCtl& cl = *D.ctl;
  if (cl.done) return;
  const StepK k = cl.k;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int s = blockIdx.x * wpb + wid;             // this warp's segment
  const int R = A.band_rows;                          // rows per band, <= kBandRows
  const int r0 = blockIdx.y * R;
  const int r1 = r0 + R < A.ny ? r0 + R : A.ny;
  BandAcc t;
  if (s < (A.nx + 63) / 64) {
    if (!k.exact) band_sweep<false, CREST, BND, TAPE, SKIP>(A, D, cl, k, d, s, r0, r1, edge_w[wid], edge_e[wid], t);
    else band_sweep<true, CREST, BND, TAPE, SKIP>(A, D, cl, k, d, s, r0, r1, edge_w[wid], edge_e[wid], t);
  }
  if constexpr (TAPE) return;
  // ---- block reduction into the finalize's partials (fixed order). What only some blocks or steps
  //      have (the edges' fluxes, the volume of a sync step) is summed only there. ----
  const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(t.smax));
  const bool low = t.low < -k.h_dry || __float_as_uint(t.low) == 0xff800000u;
  const unsigned b = (__any_sync(0xffffffffu, low) ? 1u : 0u) | (__any_sync(0xffffffffu, t.uns) ? 2u : 0u);
  const bool xedge = blockIdx.x == 0 || blockIdx.x == gridDim.x - 1, yedge = r0 == 0 || r1 == A.ny;
  double acc[kPart] = {t.infil, t.fix, t.in, t.out, t.vol, t.ytop, t.ybot};
#pragma unroll
  for (int j = 0; j < kPart; ++j)
    if (j < 2 || ((j == 2 || j == 3) && xedge) || (j == 4 && cl.pl.hits) || (j > 4 && yedge)) acc[j] = warp_sum_d(acc[j]);
  if (lane == 0) {
    wmax[wid] = __uint_as_float(m); wbad[wid] = b;
    for (int j = 0; j < kPart; ++j) wsum[wid][j] = acc[j];
  }
  __syncthreads();
  if (wid == 0) {
    if (lane == 0) {
      float mm = 0.0f; unsigned bb = 0u;
      for (int w = 0; w < wpb; ++w) { mm = fmaxf(mm, wmax[w]); bb |= wbad[w]; }
      if (mm > 0.0f) atomicMax(&D.ctl->smax_bits, __float_as_uint(mm));
      if (bb) atomicOr(&D.ctl->bad, bb);
    }
    if (lane < kPart) {
      double ss = 0.0;
      for (int w = 0; w < wpb; ++w) ss += wsum[w][lane];
      D.part[((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kPart + lane] = ss;
    }
  }
  if (!fin) return;
  // the design's last block: its partials, maxima and row flags are in memory before the count
  if (SKIP || wid == 0) __threadfence();   // (the threads that wrote them)
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicInc(A.arrive + d, (unsigned)nblk - 1u) == (unsigned)nblk - 1u ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  plain_finalize_body<false>(A, d, nblk, 0);
}

}  // namespace itr
