// itr_batched.cuh — the batched forward operator: one design per thread-block cluster.
//
// Replaces the reference's per-step `update` + `finalize` dispatch pair and its 64-step host
// polling (crates/itr-gpu/src/shader.wgsl:135-365, crates/itr-gpu/src/lib.rs:302-328) with a
// single persistent launch over the whole population: every cluster owns one design for the
// whole simulated storm and never leaves the SM between steps.
//
// Layout on chip. The design's rows are split into bands, one per CTA of the cluster; a band's
// state stays in shared memory until the run ends. A lane works on two adjacent columns (a pair)
// with paired FP32 instructions (itr_device.cuh, face2 / update_cell2), and the state is stored
// as the pairs the arithmetic reads, so a row costs three 16-byte loads and three 16-byte stores a
// lane and no register moves: A = (h0 h1 u0 u1), B = (v0 v1 c0 c1), Q = (qx0 qx1 qy0 qy1),
// running peaks (p0 p1). The inputs are packed alike once per call (k_pack_inputs): J = a row's
// north y-face and west x-face jumps of a pair, G = its wet and g n^2, read straight from L2 one
// row ahead.
//
// A CTA's band is cut into S strips of rows and W windows of at most 30 pairs; a warp sweeps one
// strip of one window row by row, the reference's fused in-place row sweep (crates/itr-hydro/src/
// kernel.rs:637-697): the north y-face of a row is carried in registers from the row above, the
// west x-faces of the next row are computed one row early, and the east face of a column is the
// west face of the next one (own register or a shuffle). Lanes 1 .. 30 own their pairs, lanes 0
// and 31 hold the neighbouring windows' nearest pairs, so every face a window needs is computed in
// it. The first and last row of a strip likewise: the y-faces on a strip's edges are computed by
// both strips (or CTAs) beside them. What a neighbour reads, the pairs on either side of a window
// boundary and the rows on either side of a strip boundary, is kept twice, for even and odd steps:
// a warp reads its neighbour's old state whatever row the neighbour has reached, and no warp waits
// for another during a step. Domain edges: the ghost column is a mirror of the last column, made in
// registers as the row is loaded. Velocities and celerity are stored with the state when a cell
// is updated, so each is computed once per cell-step.
// Lanes that own nothing compute on bounded neighbour values with dt / dx, dt / dy, 1 / dx, 1 / dy and
// the inputs 0, so their cells stay as they are and add nothing to the step's sums: the row body
// has no per-lane branch.
//
// Synchronisation per step: one full cluster barrier, for the CFL reduction, whose maximum and
// health flags go through a shared-memory atomic per warp and a DSMEM read of every CTA's slot.
// The f64 time integrator (dt rule, sync clipping, exact rain integral, solver.rs:449-489) runs
// in every thread redundantly on identical inputs, so no broadcast is needed.
//
// Ledgers: infiltration and positivity fix are summed per lane in f64 over the steps; the per-face
// boundary mass fluxes of a step go to shared memory, where one warp adds them to f64 sums of its
// lanes. At sync points these are reduced in a fixed order, and the volume, the ledger row, the
// guard test (objective.rs:130-145) and the incumbent lower bound (objective.rs:146-149) are
// evaluated on the device, so an aborted design stops at once.
#pragma once
#include <cooperative_groups.h>
#include "itr_device.cuh"

namespace itr {
namespace cg = cooperative_groups;

// Scalars of one CTA at a sync snapshot of a baseline-locked run (the Checkpoint of
// solver.rs:78-92 that the fallback restores): the integrator, which is the same in every
// CTA of a design, and this CTA's f64 ledger totals.
struct LockedSnap {
  double t, dt_cfl, s_cur, acc_rain, volume, rel_res;
  double led[4];
  unsigned long long step, skipped;   // skipped: dry rows of this CTA so far
  unsigned sync_index;
  int n_rows;
};

struct BatchArgs {
  RunParams P;
  int nx, ny, mode;
  int C;          // CTAs per design (cluster size)
  int W, S;       // windows (warps) per strip row, strips per CTA
  int n_designs;
  // packed inputs (k_pack_inputs), rows of pairs() + 2 records: record p + 1 is the pair of columns
  // 2 p, 2 p + 1, records 0 and pairs() + 1 the columns beside the grid
  const float4* G;    // ny rows: wet, wet, g n^2, g n^2
  const float4* J;    // per design ny + 1 rows f: y-face f of the two columns, west x-faces of row f
  const float4* J2;   // crest: the second jumps
  const unsigned* never;   // per design: 1 = an input out of the bounds of the branch-free step
  const uint8_t* bc;  // north[nx], south[nx], west[ny], east[ny]; device codes (ghost_state)
  const float* bh;    // stage-ghost depths, n_designs * [2 nx + 2 ny] indexed like bc, or NULL
  const float* h0;    // n_designs * nx*ny
  const double* cut;  // n_designs
  const double* fill; // n_designs
  int n_mon;
  const unsigned* mon_cells;
  DevObjective obj;
  float* peak_out;    // n_designs * nx*ny
  float* depth_out;   // n_designs * nx*ny
  double* ledger_out; // n_designs * max_rows * 8
  int max_rows;
  DesignOut* out;     // n_designs
  unsigned long long max_steps;
  unsigned exact;     // 1: every step through the scalar path (checking)
  unsigned wait_limit;   // try_wait rounds of a single-CTA design's barrier wait before status 5
  unsigned stall_test;   // 1: that barrier expects one arrival more than the CTA makes (timeout test)
  const WarmStart* warm;   // optional, per design (state NULL: cold start)
  // Baseline-locked dt (SolverParams::locked_dt / cfl_hard, solver.rs:42-46); read only by the
  // LOCKED instantiation, which is launched when locked_dt is set.
  const double* locked_dt;   // n_locked dts of the baseline, shared by every design
  unsigned long long n_locked;
  double cfl_hard;
  float4* snap;              // sync snapshot of every CTA's state, n_designs * C * SmemPlan::state bytes
  LockedSnap* snap_s;        // n_designs * C records
  double* fallback_t;        // n_designs: time the run fell back to adaptive dt, -1 for none
};

__host__ __device__ inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

ITR_DEV unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Column pairs of a row, windows of a strip row (30 own pairs a warp at most) and pairs per window.
__host__ __device__ inline int pairs(int nx) { return (nx + 1) / 2; }
__host__ __device__ inline int windows(int nx) { return (pairs(nx) + 29) / 30; }

// Shared-memory plan of one CTA. Every CTA of a cluster uses the plan of the largest band,
// so an offset names the same array in every CTA (DSMEM maps local pointers to peers).
struct SmemPlan {
  size_t a, b, q, pk, state, bx, by, sg, led, slot, red, mbar, inf, wf, gwf, nsk, total;
};

__host__ __device__ inline SmemPlan smem_plan(int nr_max, int nx, int S, int W, int nwarps, int bnd, int ny) {
  SmemPlan p;
  const size_t P2 = pairs(nx), RS = P2 + 2 * (W - 1);
  size_t o = 0;
  const size_t rows = nr_max + 2 * S;              // the strips' first and last rows twice
  p.a = o;   o += rows * RS * 16;                  // float4 h0 h1 u0 u1 (boundary pairs twice)
  p.b = o;   o += rows * RS * 16;                  // float4 v0 v1 c0 c1
  p.q = o;   o += nr_max * P2 * 16;                // float4 qx0 qx1 qy0 qy1
  p.pk = o;  o += nr_max * P2 * 8;                 // float2 peak depth
  o = align_up(o, 16);
  p.state = o;
  p.by = o;  o += (size_t)2 * 2 * P2 * 8;          // top/bottom boundary mass flux [2 parity][2][2 P2]
  p.bx = o;  o += (size_t)2 * nr_max * 4;          // west/east boundary mass flux of a step [2][nr]
  p.sg = o;  o += (size_t)2 * nr_max * 4;          // west/east wall signs (-1 wall, 1 copy) [2][nr]
  o = align_up(o, 16);
  p.led = o;  o += 4 * 8;                          // f64 totals up to the last sync: infil, fix, in, out
  p.slot = o; o += 3 * 8;                          // (smax bits, flags) of a step [3 in turn]
  p.red = o;  o += (size_t)nwarps * 8 * 8;         // f64 reductions at sync points
  p.mbar = o; o += 16;
  p.inf = o;  o += bnd ? (size_t)2 * kMaxInflow * 8 : 0;   // float2 inflow values [2 parity][groups]
  p.wf = o;   o += (size_t)2 * nr_max * W;           // row wetness bytes [2 parity][nr_max][W]
  p.gwf = o;  o += bnd ? (size_t)2 * (ny + 2) : 0;    // ghost wetness [2 parity][ny + 2 padded rows]
  o = align_up(o, 8);
  p.nsk = o;  o += 8;                                 // rows skipped by this CTA
  p.total = align_up(o, 16);
  return p;
}

ITR_DEV void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
ITR_DEV void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

ITR_DEV void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
ITR_DEV void mbar_arrive(unsigned long long* bar) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.release.cta.shared::cta.b64 st, [%0]; }" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait on phase `parity`: at most `limit` try_wait rounds; returns false if the
// bound ran out.
ITR_DEV bool mbar_wait(unsigned long long* bar, unsigned parity, unsigned limit) {
  for (unsigned it = 0; it < limit; ++it) {
    unsigned ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Self-checking build (-DITR_CHECKED): every shared, distributed-shared and global index
// is checked against its array; the first violation is recorded in g_itr_err (code, index,
// block, thread) and the access is redirected to element 0 instead of faulting.
#ifdef ITR_CHECKED
__device__ unsigned long long g_itr_err[4];
ITR_DEV long long chk(long long i, long long lim, int code) {
  if (i < 0 || i >= lim) {
    if (atomicCAS(&g_itr_err[0], 0ull, (unsigned long long)code) == 0ull) {
      g_itr_err[1] = (unsigned long long)i; g_itr_err[2] = blockIdx.x; g_itr_err[3] = threadIdx.x;
    }
    return 0;
  }
  return i;
}
#define CK(i, lim, code) ((int)chk((long long)(i), (long long)(lim), (code)))
#else
#define CK(i, lim, code) (i)
#endif

struct Smem {
  float4 *A, *B, *Q;
  float2* PK;
  float* BX;       // [2 side][nr_max]
  float* BY;       // [2 parity][2 side][2 P2]
  float* SG;       // [2 side][nr_max]
  double* LED;     // [4]
  uint2* slot;     // [3], step n's in slot n mod 3
  double* red;     // [nwarps][8]
  unsigned long long* mbar;
  float2* INF;     // inflow group values [2 parity][kMaxInflow] (stage/inflow grids only)
  uint8_t* WF;     // [2 parity][nr_max][W]: the warp's columns of the row held water (state of that parity)
  uint8_t* GWF;    // [2 parity][ny + 2]: a stage / inflow ghost of padded row j holds water (BND)
  unsigned long long* NSK;
  int nab, npk;   // bounds (checked build)
};

ITR_DEV float4 f4(const FaceF& f) { return make_float4(f.m, f.nl, f.nr, f.t); }
ITR_DEV FaceF ff(const float4& v) { FaceF f; f.m = v.x; f.nl = v.y; f.nr = v.z; f.t = v.w; return f; }

ITR_DEV double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Barrier over the design: the cluster's, or the CTA's for single-CTA designs.
template <bool CLUSTERED>
ITR_DEV void design_bar() {
  if (CLUSTERED) { cluster_arrive(); cluster_wait(); } else __syncthreads();
}

// Map a pointer into shared memory to the same offset in CTA `rank` of the cluster.
template <class T> ITR_DEV T* remote(T* p, int rank) {
  return cg::this_cluster().map_shared_rank(p, (unsigned)rank);
}

// A lane's pair of cells.
struct Cell2 { float2 h, qx, qy, u, v, c; };
struct Cell { float h, qx, qy, u, v, c; };

ITR_DEV float2 lo2(float4 a) { return make_float2(a.x, a.y); }
ITR_DEV float2 hi2(float4 a) { return make_float2(a.z, a.w); }
ITR_DEV float4 cat4(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }

// The pair one column to the west: the west lane's second column and this lane's first.
ITR_DEV float2 west2(float2 a) { return make_float2(__shfl_up_sync(0xffffffffu, a.y, 1), a.x); }
// The pair one column to the east.
ITR_DEV float2 east2(float2 a) { return make_float2(a.y, __shfl_down_sync(0xffffffffu, a.x, 1)); }

// Ghost cells (boundary.rs:36-87) from the interior cell c behind them: a wall mirrors the
// normal momentum (so the normal velocity flips sign exactly), a transmissive edge copies
// the cell. BND (the grid has stage or inflow cells): a stage or inflow ghost takes its
// state from ghost_state and its velocities and celerity from cell_vel, as every padded
// cell's do in the reference's velocity pass. NX: across an x-normal face; pos: index in
// bc / bh; inward_pos: west or north side.
template <bool BND, bool NX>
ITR_DEV Cell ghost_cell(Cell c, int code, const float* bh, int pos, const float2* inf, bool inward_pos, float g,
                        float heps2) {
  if (!BND || code < 2) {
    if (code == 0) {
      if (NX) { c.qx = -c.qx; c.u = -c.u; } else { c.qy = -c.qy; c.v = -c.v; }
    }
    return c;
  }
  const float hs = code == 2 ? bh[pos] : 0.0f;
  const float2 fi = code >= 3 ? inf[code - 3] : make_float2(0.0f, 0.0f);
  ghost_state<NX>(code, c.h, c.qx, c.qy, hs, fi, inward_pos);
  cell_vel(c.h, c.qx, c.qy, g, heps2, c.u, c.v, c.c);
  return c;
}
ITR_DEV Cell cx(const Cell2& a) { Cell c; c.h = a.h.x; c.qx = a.qx.x; c.qy = a.qy.x; c.u = a.u.x; c.v = a.v.x; c.c = a.c.x; return c; }
ITR_DEV Cell cy(const Cell2& a) { Cell c; c.h = a.h.y; c.qx = a.qx.y; c.qy = a.qy.y; c.u = a.u.y; c.v = a.v.y; c.c = a.c.y; return c; }
ITR_DEV Cell2 cell2_of(const Cell& a, const Cell& b) {
  Cell2 r;
  r.h = make_float2(a.h, b.h); r.qx = make_float2(a.qx, b.qx); r.qy = make_float2(a.qy, b.qy);
  r.u = make_float2(a.u, b.u); r.v = make_float2(a.v, b.v); r.c = make_float2(a.c, b.c);
  return r;
}

// Sync snapshot of one CTA of a baseline-locked run: its state and peaks (n16 16-byte words of
// shared memory) and, by thread 0, the integrator scalars and the CTA's ledger totals into
// record `rec`. Ends with a CTA barrier, so no thread writes the state of the next step before
// all of it is saved.
ITR_DEV void locked_save(const BatchArgs& A, const Smem& sm, int n16, size_t rec, double t, double dt_cfl, double s_cur,
                         double acc_rain, double volume, double rel_res, unsigned long long step, unsigned sync_index, int n_rows) {
  for (int i = threadIdx.x; i < n16; i += blockDim.x) A.snap[rec * n16 + i] = sm.A[i];
  if (threadIdx.x == 0) {
    LockedSnap& o = A.snap_s[rec];
    o.t = t; o.dt_cfl = dt_cfl; o.s_cur = s_cur; o.acc_rain = acc_rain; o.volume = volume; o.rel_res = rel_res;
    for (int j = 0; j < 4; ++j) o.led[j] = sm.LED[j];
    o.step = step; o.skipped = *sm.NSK; o.sync_index = sync_index; o.n_rows = n_rows;
  }
  __syncthreads();
}

// SKIP: the dry-row test of rain-free steps (kernel.rs:605-612) and the row wetness flags it
// reads. The host launches the SKIP instantiation when params.skip_dry is set and the storm
// has a rain-free interval inside the run; every other run has no rain-free step, where the
// test never skips, and takes the instantiation without the bookkeeping (same results).
template <bool CREST, bool CLUSTERED, int MAXT, bool BND, bool LOCKED = false, bool SKIP = false>
__global__ void __launch_bounds__(MAXT, 1) k_batched(const BatchArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool kAhead = !SKIP && MAXT <= 256;   // faces a row ahead of the updates (needs the 255 registers of 8 warps per SM)
  const int C = A.C;
  const int q = CLUSTERED ? (int)cg::this_cluster().block_rank() : 0;
  const int d = blockIdx.x / C;
  if (d >= A.n_designs) return;   // whole clusters only (grid is a multiple of C)
  const int nx = A.nx, ny = A.ny;
  const int ra = (int)((long long)q * ny / C), rb = (int)((long long)(q + 1) * ny / C);
  const int nr = rb - ra;
  const int nr_max = (ny + C - 1) / C;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nwarps = blockDim.x >> 5;
  const int W = A.W, S = A.S;
  const int s = wid / W, wis = wid % W;   // strip and window of this warp (every warp has one)
  // strip rows (global row indices; S <= the fewest rows of a CTA, so every strip has one)
  const int r0 = ra + (int)((long long)s * nr / S), r1 = ra + (int)((long long)(s + 1) * nr / S);
  const int L = r1 - r0, lr0 = r0 - ra;

  // ---- the lane's pair ----
  const int P2 = pairs(nx), PW = (P2 + W - 1) / W, RS = P2 + 2 * (W - 1), PJ = P2 + 2;
  const int pf = wis * PW, cnt = PW < P2 - pf ? PW : P2 - pf;   // own pairs pf .. pf + cnt - 1, lanes 1 .. cnt
  const int p = pf + lane - 1;
  const bool own = lane >= 1 && lane <= cnt;
  const bool odd = nx & 1, wlast = wis == W - 1;
  const bool west_g = wis == 0 && lane == 0;           // second column: the west ghost, mirrored from pair 0's first
  const bool east_g = wlast && !odd && lane == cnt + 1;   // first column: the east ghost, mirrored from the last pair's second
  const bool east_y = wlast && odd && lane == cnt;        // second column of the last pair: the east ghost, mirrored from its first
  const bool mir_y = west_g || east_y;
  const bool own_y = own && !east_y;
  // The pair it reads (a ghost lane its mirror; a lane past the window's neighbour any own pair)
  // and where that is kept on even and odd steps.
  const int ps = west_g || lane > cnt + 1 ? pf : (p >= P2 ? P2 - 1 : p);
  auto alt_of = [&](int pp) -> int {
    const int w = pp / PW, f = w * PW, c = PW < P2 - f ? PW : P2 - f;
    if (w > 0 && pp == f) return P2 + 2 * (w - 1) + 1;
    if (w < W - 1 && pp == f + c - 1) return P2 + 2 * w;
    return pp;
  };
  const int slot_e = ps, slot_o = alt_of(ps);
  // Where row lr of a CTA with n rows is kept on odd steps: the first and last row of strip s in
  // row nr_max + 2 s (+ 1).
  auto row_odd = [&](int lr, int n) -> int {
    const int st = ((lr + 1) * S - 1) / n, a = st * n / S, b = (st + 1) * n / S;
    return lr == a ? nr_max + 2 * st : lr == b - 1 ? nr_max + 2 * st + 1 : lr;
  };
  const float2 mask = make_float2(own ? 1.0f : 0.0f, own_y ? 1.0f : 0.0f);
  const int jx = lane <= cnt + 1 ? p + 1 : 0;   // record of the pair's jumps (0: zeros), p >= -1
  const int gx = own ? p + 1 : 0;               // of its wet and g n^2

  const SmemPlan pl_s = smem_plan(nr_max, nx, S, W, nwarps, BND ? 1 : 0, ny);
  Smem sm;
  sm.A = reinterpret_cast<float4*>(smem_raw + pl_s.a);
  sm.B = reinterpret_cast<float4*>(smem_raw + pl_s.b);
  sm.Q = reinterpret_cast<float4*>(smem_raw + pl_s.q);
  sm.PK = reinterpret_cast<float2*>(smem_raw + pl_s.pk);
  sm.BX = reinterpret_cast<float*>(smem_raw + pl_s.bx);
  sm.BY = reinterpret_cast<float*>(smem_raw + pl_s.by);
  sm.SG = reinterpret_cast<float*>(smem_raw + pl_s.sg);
  sm.LED = reinterpret_cast<double*>(smem_raw + pl_s.led);
  sm.slot = reinterpret_cast<uint2*>(smem_raw + pl_s.slot);
  sm.red = reinterpret_cast<double*>(smem_raw + pl_s.red);
  sm.mbar = reinterpret_cast<unsigned long long*>(smem_raw + pl_s.mbar);
  sm.INF = reinterpret_cast<float2*>(smem_raw + pl_s.inf);
  sm.WF = reinterpret_cast<uint8_t*>(smem_raw + pl_s.wf);
  sm.GWF = reinterpret_cast<uint8_t*>(smem_raw + pl_s.gwf);
  sm.NSK = reinterpret_cast<unsigned long long*>(smem_raw + pl_s.nsk);
  sm.nab = (nr_max + 2 * S) * RS; sm.npk = nr_max * P2;
  const RunParams& P = A.P;
  const size_t cell0_off = (size_t)d * nx * ny;
  const int bc_w = 2 * nx, bc_e = 2 * nx + ny, bc_n = 0, bc_s = nx, nbc = 2 * nx + 2 * ny;
  const float* const bh = BND ? A.bh + (size_t)d * nbc : nullptr;   // this design's stage depths
  const float4* const Jl = A.J + (size_t)d * (ny + 1) * PJ + jx;
  const float4* const J2l = CREST ? A.J2 + (size_t)d * (ny + 1) * PJ + jx : nullptr;
  const float4* const Gl = A.G + gx;

  // ---------------------------------------------------------------- initial state ----
  // (or a warm start: the baseline's state, peaks and integrator at a checkpoint)
  const WarmStart* WS = (A.warm && A.warm[d].state) ? &A.warm[d] : nullptr;
  const double t_start = WS ? WS->t : 0.0;
  double s0_l = 0.0, v0_l = 0.0;
  bool uns_i = false;   // an initial depth out of the bounds of the branch-free step
  for (int idx = tid; idx < nr * P2; idx += blockDim.x) {
    const int lr = idx / P2, pp = idx % P2;
    Cell c[2];
    float pk[2];
    for (int e = 0; e < 2; ++e) {
      const int col = 2 * pp + e;
      c[e].h = c[e].qx = c[e].qy = 0.0f;
      pk[e] = 0.0f;
      if (col < nx) {
        const size_t i = (size_t)(ra + lr) * nx + col, NN = (size_t)nx * ny;
        if (WS) {
          c[e].h = WS->state[i]; c[e].qx = WS->state[NN + i]; c[e].qy = WS->state[2 * NN + i]; pk[e] = WS->state[3 * NN + i];
        } else {
          c[e].h = A.h0[cell0_off + i];
          uns_i = uns_i || !depth_safe(P, c[e].h);
          const double hd = (double)c[e].h;
          v0_l += hd;
          if (hd > P.h_dry) {  // initial_smax (solver.rs:314-332) with q = 0
            const double cd = sqrt(P.g * hd);
            const double rr = (0.0 / hd + cd) / P.dx + (0.0 / hd + cd) / P.dy;
            s0_l = s0_l > rr ? s0_l : rr;
          }
        }
      }
      cell_vel(c[e].h, c[e].qx, c[e].qy, P.g_f, P.heps2_f, c[e].u, c[e].v, c[e].c);
    }
    const float4 a = make_float4(c[0].h, c[1].h, c[0].u, c[1].u), b = make_float4(c[0].v, c[1].v, c[0].c, c[1].c);
    const int e = lr * RS + pp, o = row_odd(lr, nr) * RS + alt_of(pp);
    sm.A[CK(e, sm.nab, 1)] = a; sm.B[e] = b;
    sm.A[CK(o, sm.nab, 1)] = a; sm.B[o] = b;
    sm.Q[CK(idx, sm.npk, 2)] = make_float4(c[0].qx, c[1].qx, c[0].qy, c[1].qy);
    sm.PK[idx] = make_float2(pk[0], pk[1]);
  }
  for (int i = tid; i < nr; i += blockDim.x) {
    sm.SG[i] = A.bc[bc_w + ra + i] == 0 ? -1.0f : 1.0f;
    sm.SG[nr_max + i] = A.bc[bc_e + ra + i] == 0 ? -1.0f : 1.0f;
  }
  if (tid < 3) sm.slot[tid] = make_uint2(0u, 0u);
  if (tid < 4) {
    const bool w = WS && q == 0;   // a warm start's totals so far
    sm.LED[tid] = !w ? 0.0 : tid == 0 ? WS->tot_infil : tid == 1 ? WS->tot_fix : tid == 2 ? WS->tot_in : WS->tot_out;
  }
  if (tid == 0) *sm.NSK = 0ull;
  if (tid == 0) mbar_init(sm.mbar, blockDim.x + (A.stall_test ? 1u : 0u));
  // inflow ghosts of step 0 (at t = 0), and the ghost wetness the dry-row test reads; each
  // later step's are written one step ahead
  if (BND && wid == nwarps - 1) {
    const int par = WS ? (int)(WS->step & 1ull) : 0;
    if (lane < P.inflow.n) sm.INF[par * kMaxInflow + lane] = inflow_values(P.inflow, lane, t_start, P.g);
    __syncwarp();
    if (SKIP) ghost_row_wet(A.bc, nx, ny, bh, sm.INF + par * kMaxInflow, sm.GWF + par * (ny + 2), lane);
  }
  {
    double sw = s0_l;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { double t = __shfl_xor_sync(0xffffffffu, sw, o); sw = sw > t ? sw : t; }
    const double vw = warp_sum_d(v0_l);
    const bool un = __any_sync(0xffffffffu, uns_i);
    if (lane == 0) { sm.red[wid * 8 + 0] = sw; sm.red[wid * 8 + 1] = vw; sm.red[wid * 8 + 2] = un ? 1.0 : 0.0; }
  }
  design_bar<CLUSTERED>();
  // Row wetness flags of the CTA's rows from the state of parity `par` in shared memory (init_state's
  // rule: a row is dry when every depth is 0): entry 0 of a row holds the flag, the others are cleared.
  auto row_flags = [&](int par) {
    for (int lr = wid; lr < nr; lr += nwarps) {
      bool w = false;
      for (int c = lane; c < nx; c += 32) {
        const float4 a = sm.A[par ? row_odd(lr, nr) * RS + alt_of(c >> 1) : lr * RS + (c >> 1)];
        w = w || ((c & 1) ? a.y : a.x) != 0.0f;
      }
      w = __any_sync(0xffffffffu, w);
      uint8_t* e = sm.WF + ((size_t)par * nr_max + lr) * W;
      for (int k = lane; k < W; k += 32) e[k] = (k == 0 && w) ? 1 : 0;
    }
  };
  if (SKIP) row_flags(WS ? (int)(WS->step & 1ull) : 0);
  // f64 sums over the warps of every CTA of the design: entry j of each warp's 8 in `red`
  // (the same lane order and butterfly in every warp: identical in every thread)
  auto total = [&](int j) -> double {
    double v = 0.0;
    for (int e = lane; e < C * nwarps; e += 32) {
      const double* rr = CLUSTERED ? remote(sm.red, e / nwarps) : sm.red;
      v += rr[(e % nwarps) * 8 + j];
    }
    return warp_sum_d(v);
  };
  double s0 = 0.0;
  for (int e = lane; e < C * nwarps; e += 32) {
    const double* rr = CLUSTERED ? remote(sm.red, e / nwarps) : sm.red;
    const double a = rr[(e % nwarps) * 8];
    s0 = s0 > a ? s0 : a;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { const double a = __shfl_xor_sync(0xffffffffu, s0, o); s0 = s0 > a ? s0 : a; }
  const double v0 = WS ? WS->v0 : total(1) * P.area;
  const bool uns_0 = total(2) > 0.0;
  design_bar<CLUSTERED>();   // red reused below

  // ------------------------------------------------------------------ integrator ----
  double t = t_start;
  unsigned long long step = WS ? WS->step : 0ull;
  unsigned sync_index = WS ? WS->sync_index : 0u;
  double dt_cfl = WS ? WS->dt_cfl : (s0 > 0.0 ? dmin_num(P.cfl / s0, P.dt_max) : P.dt_max);
  double acc_rain = WS ? WS->acc_rain : 0.0;
  // Scalar-path steps: always (checking, an input out of bounds), or until the state is known to be
  // bounded (a warm start's from the dt its wave rate gave).
  const bool always_exact = A.exact != 0u || A.never[d] != 0u;
  bool unsafe = WS ? !(P.cfl <= 0.99 * (double)P.s_safe * dt_cfl) : uns_0;
  int status = 0;
  int sc = 0;            // the step's slot of the CFL reduction
  unsigned phase = 0u;   // single-CTA designs: phase of the step's closing barrier
  unsigned breach_cell = 0, breach_sync = 0;
  double violation = 0.0, lower_bound = 0.0, volume = WS ? WS->volume : v0, rel_res = WS ? WS->rel_res : 0.0;
  int n_rows = WS ? WS->n_rows : 0;
  // the current sync instant, the latest start of a step that is clipped to it, and the storm's piece
  // and rate at t
  double t_sync = 0.0, t_hit = 0.0, rate_t = 0.0, smax = 0.0;
  int seg = 0;
  auto next_sync = [&]() {
    t_sync = dmin_num((double)(sync_index + 1) * P.sync, P.duration);
    t_hit = t_sync - 1e-9 * P.sync;
  };
  auto rain_at_t = [&](double x) {   // (t only grows, but for a locked run's return to its snapshot)
    while (P.rain_pieces && x > P.rain.seg[seg].end) ++seg;
    rate_t = rain_piece(P.rain.seg[seg], x);
  };
  next_sync();
  rain_at_t(t);
  bool have_smax = false;   // dt_cfl below is the start's; later steps take cfl / smax
  // f64 sums since the last sync: infiltration and positivity fix of this lane's cells; edge inflow
  // and outflow (lanes of warp 0)
  double sum_infil = 0.0, sum_fix = 0.0, sum_in = 0.0, sum_out = 0.0;

  const float2* inf_cur = sm.INF;   // this step's inflow group values (parity slot)
  unsigned gw_even = ~0u, gw_odd = ~0u;   // inflow groups that flow (a bit each) in the ghost wetness of each parity slot; ~0: not known
  const int top_odd = row_odd(lr0, nr), bot_odd = row_odd(lr0 + L - 1, nr);
  // The lane's pair in the rows above the strip's first and below its last, on even and odd steps: in
  // this CTA or the next one (unused at the domain's edges). B lies nab words after A everywhere.
  const float4 *up_e = sm.A, *up_o = sm.A, *dn_e = sm.A, *dn_o = sm.A;
  auto find_beside = [&](int r, const float4*& pe, const float4*& po) {
    const float4* pa = sm.A;
    int lr = r - ra, n = nr;
    if (CLUSTERED && (r < ra || r >= rb)) {
      const int qq = r < ra ? q - 1 : q + 1, a = (int)((long long)qq * ny / C);
      pa = remote(sm.A, qq);
      lr = r - a; n = (int)((long long)(qq + 1) * ny / C) - a;
    }
    pe = pa + CK(lr * RS + slot_e, sm.nab, 4);
    po = pa + CK(row_odd(lr, n) * RS + slot_o, sm.nab, 4);
  };
  if (r0 > 0) find_beside(r0 - 1, up_e, up_o);
  if (r1 < ny) find_beside(r1, dn_e, dn_o);
  auto pair_at = [&](const float4* pa) -> Cell2 {
    const float4 a = pa[0], b = pa[sm.nab];
    Cell2 c;
    c.h = lo2(a); c.u = hi2(a); c.v = lo2(b); c.c = hi2(b);
    return c;
  };
  int rd = slot_e, wr = slot_o;     // where the lane's pair is read and written this step
  // The lane's pair of row lr (global r, kept in row `row`) with its x ghosts.
  auto load_pair = [&](int row, int lr, int r) -> Cell2 {
    const int i = CK(row * RS + rd, sm.nab, 3);
    const float4 a = sm.A[i], b = sm.B[i];
    const float sg = sm.SG[(lane == 0 ? 0 : nr_max) + lr];
    Cell2 c;
    c.h = lo2(a); c.u = hi2(a); c.v = lo2(b); c.c = hi2(b);
    c.qx = c.qy = f2(0.0f);
    if (BND && (west_g || east_g || east_y)) {
      const int pos = west_g ? bc_w + r : bc_e + r;
      const int code = A.bc[CK(pos, nbc, 13)];
      if (code >= 2) {   // stage or inflow: from the momentum of the cell it mirrors
        const float4 m = sm.Q[lr * P2 + ps];
        Cell g;
        g.h = east_g ? c.h.y : c.h.x; g.qx = east_g ? m.y : m.x; g.qy = east_g ? m.w : m.z;
        g.u = g.v = g.c = 0.0f;
        g = ghost_cell<true, true>(g, code, bh, pos, inf_cur, west_g, P.g_f, P.heps2_f);
        if (mir_y) { c.h.y = g.h; c.u.y = g.u; c.v.y = g.v; c.c.y = g.c; }
        else { c.h.x = g.h; c.u.x = g.u; c.v.x = g.v; c.c.x = g.c; }
        return c;
      }
    }
    const float ux = sg * c.u.x, uy = sg * c.u.y;
    c.h.y = mir_y ? c.h.x : c.h.y; c.u.y = mir_y ? ux : c.u.y; c.v.y = mir_y ? c.v.x : c.v.y; c.c.y = mir_y ? c.c.x : c.c.y;
    c.h.x = east_g ? c.h.y : c.h.x; c.u.x = east_g ? uy : c.u.x; c.v.x = east_g ? c.v.y : c.v.x; c.c.x = east_g ? c.c.y : c.c.x;
    return c;
  };
  // The north or south ghost row beside row lr (only an own pair's columns matter).
  auto ghost_row = [&](const Cell2& c0, int lr, bool north) -> Cell2 {
    Cell2 c = c0;
    if (!own) return c;
    const float4 m = sm.Q[CK(lr * P2 + p, sm.npk, 15)];
    c.qx = lo2(m); c.qy = hi2(m);
    const int pos = (north ? bc_n : bc_s) + 2 * p;
    const Cell gx_ = ghost_cell<BND, false>(cx(c), A.bc[CK(pos, nbc, 16)], bh, pos, inf_cur, north, P.g_f, P.heps2_f);
    Cell gy_ = cy(c);
    if (own_y) gy_ = ghost_cell<BND, false>(gy_, A.bc[CK(pos + 1, nbc, 16)], bh, pos + 1, inf_cur, north, P.g_f, P.heps2_f);
    return cell2_of(gx_, gy_);
  };

  // ---- baseline-locked dt (solver.rs:436-483, 611-614) ----
  // Each step takes the baseline's dt while dt * smax of the current state stays within
  // cfl_hard. At the first step where it would not (or the schedule has run out), every CTA
  // restores its rows and scalars from the last sync snapshot and the run continues with the
  // adaptive dt. smax, the step and the schedule are the same in every thread of the cluster,
  // so the decision is uniform.
  bool locked_live = LOCKED;
  double s_cur = s0;
  const int n16 = (int)(pl_s.state / 16);
  if constexpr (LOCKED) {
    if (q == 0 && tid == 0) A.fallback_t[d] = -1.0;
    locked_save(A, sm, n16, (size_t)d * C + q, t, dt_cfl, s_cur, acc_rain, volume, rel_res, step, sync_index, n_rows);
  }

  while (t < P.duration && sync_index < P.n_sync) {
    if (step >= A.max_steps) { status = 4; break; }
    bool use_lock = false;
    double dt_lock = 0.0;
    if constexpr (LOCKED) {
      if (locked_live) {
        if (step < A.n_locked && A.locked_dt[step] * s_cur <= A.cfl_hard) {
          use_lock = true;
          dt_lock = A.locked_dt[step];
        } else {
          design_bar<CLUSTERED>();   // every CTA has finished reading this CTA's shared memory
          const size_t rec = (size_t)d * C + q;
          for (int i = tid; i < n16; i += blockDim.x) sm.A[i] = A.snap[rec * n16 + i];
          const LockedSnap& o = A.snap_s[rec];
          t = o.t; dt_cfl = o.dt_cfl; s_cur = o.s_cur; acc_rain = o.acc_rain; volume = o.volume; rel_res = o.rel_res;
          step = o.step; sync_index = o.sync_index; n_rows = o.n_rows;
          if (tid < 4) sm.LED[tid] = o.led[tid];
          if (SKIP && tid == 0) *sm.NSK = o.skipped;
          if (tid < 3) sm.slot[tid] = make_uint2(0u, 0u);
          sum_infil = sum_fix = sum_in = sum_out = 0.0;
          seg = 0; have_smax = false;
          next_sync(); rain_at_t(t);
          const int par = (int)(step & 1ull);
          if (BND && wid == nwarps - 1) {
            if (lane < P.inflow.n) sm.INF[par * kMaxInflow + lane] = inflow_values(P.inflow, lane, t, P.g);
            __syncwarp();
            if (SKIP) {
              ghost_row_wet(A.bc, nx, ny, bh, sm.INF + par * kMaxInflow, sm.GWF + par * (ny + 2), lane);
              gw_even = gw_odd = ~0u;
            }
          }
          if (SKIP) {
            __syncthreads();   // the restored rows complete before their flags are taken
            row_flags(par);
          }
          if (q == 0 && tid == 0) A.fallback_t[d] = t;
          locked_live = false;
          unsafe = true;   // (the snapshot's bound is not kept: one step through the scalar path)
          design_bar<CLUSTERED>();   // the restored state of every CTA visible before the next step
          continue;
        }
      }
    }
    const int sp = (int)(step & 1ull);
    rd = sp ? slot_o : slot_e;
    wr = sp ? slot_e : slot_o;
    // rows of the strip's first and last row as read and as written this step
    const int top_rd = sp ? top_odd : lr0, top_wr = sp ? lr0 : top_odd;
    const int bot_rd = sp ? bot_odd : lr0 + L - 1, bot_wr = sp ? lr0 + L - 1 : bot_odd;
    if (BND) inf_cur = sm.INF + sp * kMaxInflow;
    float smax_l = 0.0f, low_l = 0.0f;
    float2 infil_l = f2(0.0f), fix_l = f2(0.0f);
    bool uns_l = false;

    // ---- strip pre-phase: first row, its west faces, the strip's top y-faces ----
    float4 jc = __ldg(Jl + (size_t)r0 * PJ);
    float4 jc2 = CREST ? __ldg(J2l + (size_t)r0 * PJ) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    Cell2 cur = load_pair(top_rd, lr0, r0);
    Face2 fW, fN;
    StepPlan pl;
    StepK k;
    bool rare;
    {
      // the cells above the strip's first row: the ghost row, or the last row of the strip or CTA above
      const Cell2 above = r0 == 0 ? ghost_row(cur, lr0, true) : pair_at(sp ? up_o : up_e);
      const float2 lh = west2(cur.h), lu = west2(cur.u), lv = west2(cur.v), lc = west2(cur.c);
      // The dt chain in f64 and the strip's first faces need nothing from each other: both stand in one
      // straight-line block, so the faces fill the chain's latency.
      if (!(always_exact || unsafe)) {
        const double q_cfl = div_by_f32(P.cfl, smax);
        if (have_smax) dt_cfl = smax > 0.0 ? q_cfl : P.dt_max;
        const double dt_pick = use_lock ? dt_lock : dmin_num(dt_cfl, P.dt_max);
        pl = plan_step_fast(P, t, t_sync, t_hit, dt_pick, rate_t, seg, rare);
        k = step_consts<true>(P, pl.dt, pl.rain);
        fW = face2<true, CREST>(lh, lu, lv, lc, cur.h, cur.u, cur.v, cur.c, hi2(jc), hi2(jc2), k);
        fN = face2<false, CREST>(above.h, above.u, above.v, above.c, cur.h, cur.u, cur.v, cur.c, lo2(jc), lo2(jc2), k);
      } else {
        if (have_smax) dt_cfl = smax > 0.0 ? P.cfl / smax : P.dt_max;
        const double dt_pick = use_lock ? dt_lock : dmin_num(dt_cfl, P.dt_max);
        pl = plan_step_fast(P, t, t_sync, t_hit, dt_pick, rate_t, seg, rare);
        k = step_consts(P, pl.dt, pl.rain);
        k.exact = 1u;
        fW = face2_exact<true, CREST>(lh, lu, lv, lc, cur.h, cur.u, cur.v, cur.c, hi2(jc), hi2(jc2), k);
        fN = face2_exact<false, CREST>(above.h, above.u, above.v, above.c, cur.h, cur.u, cur.v, cur.c, lo2(jc), lo2(jc2), k);
      }
      if (rare) {   // a breakpoint of the storm inside the step
        pl.rain = rain_integral(P.rain, t, t + pl.dt);
        k.rain = (float)pl.rain;
      }
      if (r0 == 0 && own) {   // y_boundary top (kernel.rs:452-472)
        *reinterpret_cast<float2*>(sm.BY + (sp * 2 + 0) * 2 * P2 + 2 * p) = fN.m;
      }
    }

    if (BND) {
      // the next step's inflow ghosts, at its start time (slot read after this step's
      // closing barrier; the other slot's readers finished before the previous one)
      if (wid == nwarps - 1) {
        if (lane < P.inflow.n) sm.INF[(sp ^ 1) * kMaxInflow + lane] = inflow_values(P.inflow, lane, pl.t_new, P.g);
        if (SKIP) {
          // (the ghosts' wetness changes only with the groups that flow: going over the edge cells again each step
          // was up to 17 us of it on wide grids)
          __syncwarp();
          const unsigned flows = __ballot_sync(0xffffffffu, lane < P.inflow.n && sm.INF[(sp ^ 1) * kMaxInflow + (lane & (kMaxInflow - 1))].y > 0.0f);
          if (flows != (sp ? gw_even : gw_odd)) {
            ghost_row_wet(A.bc, nx, ny, bh, sm.INF + (sp ^ 1) * kMaxInflow, sm.GWF + (sp ^ 1) * (ny + 2), lane);
            (sp ? gw_even : gw_odd) = flows;
          }
        }
      }
    }
    UpdK uk;
    uk.dtdx = mulp2(f2(k.dtdx), mask); uk.dtdy = mulp2(f2(k.dtdy), mask);
    uk.inv_dx = mulp2(f2(k.inv_dx), mask); uk.inv_dy = mulp2(f2(k.inv_dy), mask);

    // ---- dry-row skipping (kernel.rs:605-612) ----
    // With no rain this step, grid row r is skipped when rows r - 1, r, r + 1 held no water in
    // the old state (flags of parity sp, written during the previous step; the rows beside the
    // CTA's band through DSMEM) and no stage or inflow ghost of theirs holds water. Its faces
    // are exactly 0 and its cells keep their zero state: skipping changes no result. The
    // decision depends only on shared flags, so every warp of a strip takes it alike.
    const bool try_skip = SKIP && !(k.rain > 0.0f);
    auto row_dry = [&](int j) -> bool {   // grid row j in [-1, ny]
      bool dr = !BND || sm.GWF[sp * (ny + 2) + j + 1] == 0;
      if (j < 0 || j >= ny) return dr;
      const uint8_t* wf = sm.WF;
      int lj = j - ra;
      if (CLUSTERED && (j < ra || j >= rb)) {
        const int qq = j < ra ? q - 1 : q + 1;
        wf = remote(sm.WF, qq);
        lj = j - (int)((long long)qq * ny / C);
      }
      const uint8_t* e = wf + ((size_t)sp * nr_max + lj) * W;
      for (int w = 0; w < W; ++w) dr = dr && e[w] == 0;
      return dr;
    };
    // Bit i of dmask: grid row r0 - 1 + mbase + i is dry, for the rows up to r0 + L, one row
    // per lane and ballot (64 rows per fill; a strip longer than 61 rows refills as it goes).
    unsigned long long dmask = 0ull;
    int mbase = 0;
    auto fill_mask = [&](int from) {
      const int ja = r0 - 1 + from + lane, jb = ja + 32, jmax = r0 + L;
      const bool da = ja <= jmax && row_dry(ja);
      const bool db = jb <= jmax && row_dry(jb);
      dmask = (unsigned long long)__ballot_sync(0xffffffffu, da) | ((unsigned long long)__ballot_sync(0xffffffffu, db) << 32);
      mbase = from;
    };
    if (try_skip) fill_mask(0);

    const bool bottom = s + 1 >= S && q + 1 >= C;   // the strip's last row is the domain's
    // An updated (or skipped) row's results.
    auto put_row = [&](int row, int lr, const CellNew2& o, float2 u, float2 v) {
      smax_l = fmaxf(smax_l, fmaxf(o.s.x, o.s.y));
      low_l = fminf(low_l, fminf(o.low.x, o.low.y));
      infil_l = add2(infil_l, o.infil);
      fix_l = add2(fix_l, o.fix);
      if (own) {
        const int i = CK(row * RS + wr, sm.nab, 6), m = CK(lr * P2 + p, sm.npk, 7);
        sm.A[i] = cat4(o.h, u);
        sm.B[i] = cat4(v, o.c);
        sm.Q[m] = cat4(o.qx, o.qy);
        const float2 pk = sm.PK[m];
        sm.PK[m] = make_float2(fmaxf(pk.x, o.h.x), fmaxf(pk.y, o.h.y));
      }
      if (SKIP) {   // the window's columns of this row hold water in the new state (read next step)
        const bool wet_any = __any_sync(0xffffffffu, (own && o.h.x > 0.0f) || (own_y && o.h.y > 0.0f));
        if (lane == 0) sm.WF[((size_t)(sp ^ 1) * nr_max + lr) * W + wis] = wet_any ? 1 : 0;
      }
    };
    auto skip_row = [&](int row, int lr) {   // a dry row between dry rows: nothing to update
      if (own) {
        const int i = row * RS + wr;
        sm.A[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        sm.B[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
      if (wis == 0 && lane == 1) sm.BX[lr] = 0.0f;
      if (east_g || east_y) sm.BX[nr_max + lr] = 0.0f;
      if (lane == 0) sm.WF[((size_t)(sp ^ 1) * nr_max + lr) * W + wis] = 0;
      if (lane == 0 && wis == 0) atomicAdd(sm.NSK, 1ull);   // once per skipped row (rain-free steps only)
    };
    // x_boundary (kernel.rs:435-450): mass flux of the west and east domain faces
    // (one lane has both of a single column's)
    const bool bx_w = wis == 0 && lane == 1, bx_e = east_g || east_y, bx_2 = bx_w && bx_e, sec = east_y && !bx_w;
    float* const bx = sm.BX + (bx_w ? 0 : nr_max);
    auto put_edges = [&](int lr, const Face2& f) {
      if (bx_w || bx_e) bx[lr] = sec ? f.m.y : f.m.x;
      if (bx_2) bx[nr_max + lr] = f.m.y;
    };
    // The update of one row on the scalar path: lanes' idle columns are left out one by one (in an
    // unbounded state their values need not be finite).
    auto exact_row = [&](const Cell2& c, const Face2& w, const Face2& e, const Face2& n, const Face2& so, float4 g, float2& u, float2& v) -> CellNew2 {
      CellNew2 o = update_cell2_exact(c.h, c.qx, c.qy, w, e, n, so, lo2(g), hi2(g), k);
      const Vel2 x = vel2_exact(o.h, o.qx, o.qy, P.g_f, P.heps2_f);
      u = x.u; v = x.v;
      if (!own) { o.s.x = o.low.x = o.infil.x = o.fix.x = 0.0f; }
      if (!own_y) { o.s.y = o.low.y = o.infil.y = o.fix.y = 0.0f; }
      uns_l = uns_l || !state_safe(P, o.s.x) || !state_safe(P, o.s.y);
      return o;
    };

    // ---- row sweep ----
    jc = __ldg(Jl + (size_t)(r0 + 1) * PJ);
    if (CREST) jc2 = __ldg(J2l + (size_t)(r0 + 1) * PJ);
    float4 gc = __ldg(Gl + (size_t)r0 * PJ);
    if (kAhead && !k.exact) {
      // The update of a row is one long dependent chain (its roots, reciprocals and Newton steps), the faces of the next
      // row another: the faces run one row ahead of the update, in one block, so the two chains fill
      // each other's latency.
      auto update_row = [&](int row, int lr, float2 h, const Face2& w, const Face2& n, const Face2& so, float4 g) {
        const float4 m = sm.Q[CK(lr * P2 + ps, sm.npk, 8)];
        Face2 e;
        e.m = east2(w.m); e.nl = east2(w.nl); e.nr = east2(w.nr); e.t = east2(w.t);
        const CellNew2 o = update_cell2(h, lo2(m), hi2(m), w, e, n, so, lo2(g), hi2(g), k, uk);
        float2 u, v;
        vel2(o.h, o.qx, o.qy, k, u, v);
        put_edges(lr, w);
        put_row(row, lr, o, u, v);
      };
      // faces below row i and west of row i + 1
      auto next_faces = [&](int i, Cell2& nxt, Face2& fS, Face2& fWn) {
        nxt = load_pair(i == L - 2 ? bot_rd : lr0 + i + 1, lr0 + i + 1, r0 + i + 1);
        const float2 lh = west2(nxt.h), lu = west2(nxt.u), lv = west2(nxt.v), lc = west2(nxt.c);
        fS = face2<false, CREST>(cur.h, cur.u, cur.v, cur.c, nxt.h, nxt.u, nxt.v, nxt.c, lo2(jc), lo2(jc2), k);
        fWn = face2<true, CREST>(lh, lu, lv, lc, nxt.h, nxt.u, nxt.v, nxt.c, hi2(jc), hi2(jc2), k);
      };
      const bool two = L > 1;
      float2 ph = f2(0.0f);
      Face2 pW{}, pN{};
      float4 pg = gc;
      Cell2 nxt;
      Face2 fS, fWn;
      auto shift = [&](float4 jn, float4 jn2, float4 gn) {
        ph = cur.h; pW = fW; pN = fN; pg = gc;
        cur = nxt; fN = fS; fW = fWn;
        jc = jn; jc2 = jn2; gc = gn;
      };
      auto inputs = [&](int i, float4& jn, float4& jn2, float4& gn) {   // of the row after row i
        jn = __ldg(Jl + (size_t)(r0 + i + 2) * PJ);
        jn2 = CREST ? __ldg(J2l + (size_t)(r0 + i + 2) * PJ) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        gn = __ldg(Gl + (size_t)(r0 + i + 1) * PJ);
      };
      if (two) {
        float4 jn, jn2, gn;
        inputs(0, jn, jn2, gn);
        next_faces(0, nxt, fS, fWn);
        shift(jn, jn2, gn);
      }
#pragma unroll 3
      for (int i = 1; i < L - 1; ++i) {
        float4 jn, jn2, gn;
        inputs(i, jn, jn2, gn);
        next_faces(i, nxt, fS, fWn);
        update_row(i == 1 ? top_wr : lr0 + i - 1, lr0 + i - 1, ph, pW, pN, fN, pg);
        shift(jn, jn2, gn);
        __syncwarp();
      }
      const Cell2 below = bottom ? ghost_row(cur, lr0 + L - 1, false) : pair_at(sp ? dn_o : dn_e);
      fS = face2<false, CREST>(cur.h, cur.u, cur.v, cur.c, below.h, below.u, below.v, below.c, lo2(jc), lo2(jc2), k);
      // y_boundary bottom (kernel.rs:452-472)
      if (bottom && own) *reinterpret_cast<float2*>(sm.BY + (sp * 2 + 1) * 2 * P2 + 2 * p) = fS.m;
      if (two) update_row(L == 2 ? top_wr : lr0 + L - 2, lr0 + L - 2, ph, pW, pN, fN, pg);
      update_row(two ? bot_wr : top_wr, lr0 + L - 1, cur.h, fW, fN, fS, gc);
    } else {
    // dry rows, or the scalar path: row by row; every row but the strip's last
#pragma unroll 1
    for (int i = 0; i < L - 1; ++i) {
      const int r = r0 + i, lr = lr0 + i;
      const int row_wr = i == 0 ? top_wr : lr, row_nxt = i == L - 2 ? bot_rd : lr + 1;
      // the next row's inputs, in flight while this row is updated
      const float4 jn = __ldg(Jl + (size_t)(r + 2) * PJ), gn = __ldg(Gl + (size_t)(r + 1) * PJ);
      const float4 jn2 = CREST ? __ldg(J2l + (size_t)(r + 2) * PJ) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      bool skip = false, skip_next = false;
      if (try_skip) {
        if (i - mbase > 60) fill_mask(i);
        const int b = i - mbase;   // bits b, b + 1, b + 2: rows r - 1, r, r + 1
        skip = ((dmask >> b) & 7ull) == 7ull;
        skip_next = ((dmask >> (b + 1)) & 7ull) == 7ull;
      }
      Cell2 nxt{};
      Face2 fS{}, fWn{};
      if (SKIP && skip) {
        if (!skip_next) {   // the next row's west faces
          nxt = load_pair(row_nxt, lr + 1, r + 1);
          const float2 lh = west2(nxt.h), lu = west2(nxt.u), lv = west2(nxt.v), lc = west2(nxt.c);
          fWn = k.exact ? face2_exact<true, CREST>(lh, lu, lv, lc, nxt.h, nxt.u, nxt.v, nxt.c, hi2(jc), hi2(jc2), k)
                        : face2<true, CREST>(lh, lu, lv, lc, nxt.h, nxt.u, nxt.v, nxt.c, hi2(jc), hi2(jc2), k);
        }
        skip_row(row_wr, lr);
      } else {
        nxt = load_pair(row_nxt, lr + 1, r + 1);
        const float4 m = sm.Q[CK(lr * P2 + ps, sm.npk, 8)];
        cur.qx = lo2(m); cur.qy = hi2(m);
        const float2 lh = west2(nxt.h), lu = west2(nxt.u), lv = west2(nxt.v), lc = west2(nxt.c);
        Face2 fE;
        fE.m = east2(fW.m); fE.nl = east2(fW.nl); fE.nr = east2(fW.nr); fE.t = east2(fW.t);
        CellNew2 o;
        float2 u, v;
        if (!k.exact) {
          fS = face2<false, CREST>(cur.h, cur.u, cur.v, cur.c, nxt.h, nxt.u, nxt.v, nxt.c, lo2(jc), lo2(jc2), k);
          fWn = face2<true, CREST>(lh, lu, lv, lc, nxt.h, nxt.u, nxt.v, nxt.c, hi2(jc), hi2(jc2), k);
          o = update_cell2(cur.h, cur.qx, cur.qy, fW, fE, fN, fS, lo2(gc), hi2(gc), k, uk);
          vel2(o.h, o.qx, o.qy, k, u, v);
        } else {
          fS = face2_exact<false, CREST>(cur.h, cur.u, cur.v, cur.c, nxt.h, nxt.u, nxt.v, nxt.c, lo2(jc), lo2(jc2), k);
          fWn = face2_exact<true, CREST>(lh, lu, lv, lc, nxt.h, nxt.u, nxt.v, nxt.c, hi2(jc), hi2(jc2), k);
          o = exact_row(cur, fW, fE, fN, fS, gc, u, v);
        }
        put_edges(lr, fW);
        put_row(row_wr, lr, o, u, v);
      }
      cur = nxt; fN = fS; fW = fWn;
      jc = jn; gc = gn; jc2 = jn2;
      __syncwarp();
    }
    // ---- the strip's last row: below it the south ghost row, or the first row of the strip or CTA below ----
    {
      const int lr = lr0 + L - 1, row_wr = L == 1 ? top_wr : bot_wr;
      bool skip = false;
      if (try_skip) {
        if (L - 1 - mbase > 60) fill_mask(L - 1);
        skip = ((dmask >> (L - 1 - mbase)) & 7ull) == 7ull;
      }
      if (SKIP && skip) {
        skip_row(row_wr, lr);
        if (bottom && own) *reinterpret_cast<float2*>(sm.BY + (sp * 2 + 1) * 2 * P2 + 2 * p) = f2(0.0f);
      } else {
        const float4 m = sm.Q[CK(lr * P2 + ps, sm.npk, 8)];
        cur.qx = lo2(m); cur.qy = hi2(m);
        Face2 fE, fS;
        fE.m = east2(fW.m); fE.nl = east2(fW.nl); fE.nr = east2(fW.nr); fE.t = east2(fW.t);
        const Cell2 b = bottom ? ghost_row(cur, lr, false) : pair_at(sp ? dn_o : dn_e);
        CellNew2 o;
        float2 u, v;
        if (!k.exact) {
          fS = face2<false, CREST>(cur.h, cur.u, cur.v, cur.c, b.h, b.u, b.v, b.c, lo2(jc), lo2(jc2), k);
          o = update_cell2(cur.h, cur.qx, cur.qy, fW, fE, fN, fS, lo2(gc), hi2(gc), k, uk);
          vel2(o.h, o.qx, o.qy, k, u, v);
        } else {
          fS = face2_exact<false, CREST>(cur.h, cur.u, cur.v, cur.c, b.h, b.u, b.v, b.c, lo2(jc), lo2(jc2), k);
          o = exact_row(cur, fW, fE, fN, fS, gc, u, v);
        }
        // y_boundary bottom (kernel.rs:452-472)
        if (bottom && own) *reinterpret_cast<float2*>(sm.BY + (sp * 2 + 1) * 2 * P2 + 2 * p) = fS.m;
        put_edges(lr, fW);
        put_row(row_wr, lr, o, u, v);
      }
    }
    }
    // ---- end of step: CFL max and health ----
    {
      const bool bad_l = low_l < -k.h_dry || __float_as_uint(low_l) == 0xff800000u;
      const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(smax_l));
      const unsigned b = (__any_sync(0xffffffffu, bad_l) ? 1u : 0u) | (__any_sync(0xffffffffu, uns_l) ? 2u : 0u);
      if (lane == 0) {
        atomicMax(&sm.slot[sc].x, m);
        if (b) atomicOr(&sm.slot[sc].y, b);
      }
      // this strip's edge fluxes of the step (written by this warp)
      const double dt_dy = pl.dt * P.dy;
      __syncwarp();
      if (wis == 0 || wlast)
        for (int j = lane; j < L; j += 32) {
          if (wis == 0) {
            const double vw = (double)sm.BX[lr0 + j] * dt_dy;            // west: inflow when m > 0
            if (vw > 0.0) sum_in += vw; else sum_out -= vw;
          }
          if (wlast) {
            const double ve = (double)sm.BX[nr_max + lr0 + j] * dt_dy;   // east: outflow when m > 0
            if (ve > 0.0) sum_out += ve; else sum_in -= ve;
          }
        }
      sum_infil += (double)(infil_l.x + infil_l.y);
      sum_fix += (double)(fix_l.x + fix_l.y);
    }
    rain_at_t(pl.t_new);   // (before the barrier: it needs nothing of this step's state)
    if (CLUSTERED) {
      design_bar<CLUSTERED>();
    } else {
      // single-CTA designs: a bounded wait; if it runs out the whole CTA leaves together
      mbar_arrive(sm.mbar);
      const bool ok = mbar_wait(sm.mbar, phase & 1u, A.wait_limit);
      phase += 1u;
      if (__syncthreads_or(ok ? 0 : 1)) { status = 5; break; }
    }
    // every CTA's slot, one per lane
    uint2 sl = make_uint2(0u, 0u);
    if (lane < C) sl = (CLUSTERED ? remote(sm.slot, lane) : sm.slot)[sc];
    const unsigned smax_bits = __reduce_max_sync(0xffffffffu, sl.x), badv = __reduce_or_sync(0xffffffffu, sl.y);
    if (wid == 0) {
      const double dt_dx = pl.dt * P.dx;
      // y_boundary (kernel.rs:452-472): a y-edge's mass fluxes are summed over the row first
      // (FixedSum<f64>: lane (col + 1) & 15 in column order, then the pairwise tree, which
      // the butterfly over lanes 0-15 reproduces), then split: the top edge is inflow when
      // the net flux is > 0, the bottom edge outflow
      for (int side = 0; side < 2; ++side) {
        if (side == 0 ? q != 0 : q != C - 1) continue;
        // (an edge without flow, a wall, adds nothing)
        bool flow = false;
        for (int j = lane; j < nx; j += 32) flow = flow || sm.BY[(sp * 2 + side) * 2 * P2 + j] != 0.0f;
        if (!__any_sync(0xffffffffu, flow)) continue;
        double acc16 = 0.0;
        if (lane < 16)
          for (int j = (lane + 15) & 15; j < nx; j += 16) acc16 += (double)sm.BY[(sp * 2 + side) * 2 * P2 + j];
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) acc16 += __shfl_xor_sync(0xffffffffu, acc16, o);
        const double v = acc16 * dt_dx;
        if (lane == 0) {
          if (side == 0) { if (v > 0.0) sum_in += v; else sum_out -= v; }
          else { if (v > 0.0) sum_out += v; else sum_in -= v; }
        }
      }
    }
    // Slots in turn: the one cleared here, step n + 2's, was read after step n - 1's barrier by threads that
    // have since arrived at step n's, and is next written after step n + 1's, which this thread arrives at
    // with the clear behind it. (Of two slots, the next step's would be cleared beside its writers.)
    if (tid == 0) sm.slot[sc == 0 ? 2 : sc - 1] = make_uint2(0u, 0u);
    sc = sc == 2 ? 0 : sc + 1;
    smax = (double)__uint_as_float(smax_bits);
    have_smax = true;
    step += 1;
    t = pl.t_new;
    acc_rain += pl.rain * P.area * P.wet_count;
    if (badv & 1u) { status = 3; break; }
    unsafe = !state_safe(P, __uint_as_float(smax_bits)) || (badv & 2u) != 0u;
    if constexpr (LOCKED) s_cur = smax;
    if (pl.hits) {
      // ---- sync point: volume, ledger row, guard and incumbent tests ----
      sync_index += 1;
      next_sync();
      double vol_l = 0.0;
      const int par = (int)(step & 1ull);
      for (int idx = tid; idx < nr * P2; idx += blockDim.x) {
        const int lr = idx / P2, pp = idx % P2;
        const float4 a = sm.A[par ? row_odd(lr, nr) * RS + alt_of(pp) : lr * RS + pp];
        vol_l += (double)a.x + (2 * pp + 1 < nx ? (double)a.y : 0.0);
      }
      const double ws[5] = {warp_sum_d(vol_l), warp_sum_d(sum_infil), warp_sum_d(sum_fix), warp_sum_d(sum_in), warp_sum_d(sum_out)};
      if (lane == 0)
        for (int j = 0; j < 5; ++j) sm.red[wid * 8 + j] = ws[j];
      design_bar<CLUSTERED>();   // volume partials and ledger sums of every CTA visible
      double tot[5];
      for (int j = 0; j < 5; ++j) tot[j] = total(j);
      for (int qq = 0; qq < C; ++qq) {   // and the totals up to the last sync
        const double* lg = CLUSTERED ? remote(sm.LED, qq) : sm.LED;
        for (int j = 0; j < 4; ++j) tot[1 + j] += lg[j];
      }
      const double v = tot[0] * P.area;
      const double infil = tot[1] * P.area, fix = tot[2] * P.area;
      const double expected = v0 + acc_rain + tot[3] - tot[4] - infil + fix;
      volume = v;
      const double gross = v0 + acc_rain + tot[3];
      rel_res = fabs(v - expected) / (gross > 1e-300 ? gross : 1e-300);
      if (q == 0 && tid == 0 && n_rows < A.max_rows && A.ledger_out) {
        double* o = A.ledger_out + ((size_t)d * A.max_rows + n_rows) * 8;
        o[0] = t; o[1] = v; o[2] = acc_rain; o[3] = tot[3]; o[4] = tot[4]; o[5] = infil; o[6] = fix; o[7] = v - expected;
      }
      n_rows += 1;
      // guard breach (objective.rs:132-145) and incumbent bound (objective.rs:147-149).
      // Every warp decides from the same peaks; the barrier below comes before any thread
      // acts, so no warp writes next-step peaks (or red, LED) while another still reads them.
      const DevObjective& ob = A.obj;
      int decision = 0;
      if (ob.enabled) {
        auto peak_of = [&](int mpos) -> double {
          const unsigned cell = A.mon_cells[mpos];
          const int rr_ = (int)(cell / (unsigned)nx), cc_ = (int)(cell % (unsigned)nx);
          int owner = 0;
          while (owner + 1 < C && rr_ >= (int)((long long)(owner + 1) * ny / C)) ++owner;
          const int ra_o = (int)((long long)owner * ny / C);
          const float2* pk = CLUSTERED ? remote(sm.PK, owner) : sm.PK;
          return (double)reinterpret_cast<const float*>(pk + CK((rr_ - ra_o) * P2 + (cc_ >> 1), sm.npk, 21))[cc_ & 1];
        };
        if (ob.guard_abort && ob.require && ob.baseline) {
          double best = 0.0; int bk = -1;
          for (int g0 = 0; g0 < ob.n_guard; g0 += 32) {
            const int gk = g0 + lane;
            double w = 0.0; int kk = -1;
            if (gk < ob.n_guard) {
              const int mp = ob.guard_pos[gk];
              w = peak_of(mp) - ob.baseline[mp] - ob.tol;
              if (w > 0.0) kk = gk;
            }
            // warp argmax, first index on ties
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              const double w2 = __shfl_xor_sync(0xffffffffu, w, o);
              const int k2 = __shfl_xor_sync(0xffffffffu, kk, o);
              const bool take = (k2 >= 0) && (kk < 0 || w2 > w || (w2 == w && k2 < kk));
              if (take) { w = w2; kk = k2; }
            }
            if (kk >= 0 && (bk < 0 || w > best)) { best = w; bk = kk; }
          }
          if (bk >= 0) {
            decision = 1;
            breach_cell = A.mon_cells[ob.guard_pos[bk]];
            breach_sync = sync_index;
            violation = best;
          }
        }
        if (decision == 0 && ob.has_incumbent) {
          double jr = 0.0;
          for (int a = 0; a < ob.n_assets; ++a) {
            double pkv = 0.0;
            for (int m = ob.asset_off[a] + lane; m < ob.asset_off[a + 1]; m += 32) {
              const double x = peak_of(ob.asset_pos[m]);
              pkv = pkv > x ? pkv : x;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { const double x = __shfl_xor_sync(0xffffffffu, pkv, o); pkv = pkv > x ? pkv : x; }
            jr += ob.asset_w[a] * ob.tau * itr_math::softplus((pkv - ob.asset_thr[a]) / ob.tau);
          }
          const double je = ob.cut_cost * A.cut[d] + ob.fill_cost * A.fill[d];
          const double lb = jr + ob.earth_w * je;
          if (lb >= ob.incumbent) { decision = 2; lower_bound = lb; }
        }
      }
      design_bar<CLUSTERED>();
      // this CTA's share joins its totals; the lanes' sums start again
      if (tid < 4) {
        double add = 0.0;
        for (int w = 0; w < nwarps; ++w) add += sm.red[w * 8 + 1 + tid];
        sm.LED[tid] += add;
      }
      sum_infil = sum_fix = sum_in = sum_out = 0.0;
      if (decision != 0) { status = decision; break; }
      if constexpr (LOCKED) {
        if (locked_live) {
          __syncthreads();   // LED complete
          dt_cfl = smax > 0.0 ? P.cfl / smax : P.dt_max;
          locked_save(A, sm, n16, (size_t)d * C + q, t, dt_cfl, s_cur, acc_rain, volume, rel_res, step, sync_index, n_rows);
        }
      }
    }
  }

  // ---------------------------------------------------------------- outputs ----------
  // All CTAs of the cluster leave the loop at the same step (identical decisions).
  design_bar<CLUSTERED>();
  const int par = (int)(step & 1ull);
  for (int idx = tid; idx < nr * nx; idx += blockDim.x) {
    const int lr = idx / nx, c = idx % nx, pp = c >> 1;
    const size_t g = cell0_off + (size_t)ra * nx + idx;
    const float4 a = sm.A[par ? row_odd(lr, nr) * RS + alt_of(pp) : lr * RS + pp];
    const float2 pk = sm.PK[lr * P2 + pp];
    A.depth_out[g] = (c & 1) ? a.y : a.x;
    A.peak_out[g] = (c & 1) ? pk.y : pk.x;
  }
  if (q == 0 && tid == 0) {
    DesignOut o;
    o.steps = step; o.t_end = t; o.sync_count = sync_index; o.status = status;
    o.breach_cell = breach_cell; o.breach_sync = breach_sync; o.violation = violation;
    o.lower_bound = lower_bound; o.v0 = v0; o.volume = volume; o.rel_residual = rel_res;
    o.n_rows = n_rows; o.pad = 0;
    unsigned long long tot_skip = 0ull;
    if (SKIP)
      for (int qq = 0; qq < C; ++qq) tot_skip += CLUSTERED ? *remote(sm.NSK, qq) : *sm.NSK;
    o.rows_skipped = tot_skip;
    A.out[d] = o;
  }
  // keep every CTA's shared memory alive until all remote reads are done
  if (CLUSTERED) { cluster_arrive(); cluster_wait(); }
}

}  // namespace itr
