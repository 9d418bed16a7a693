// itr_design.cuh — designs materialised on the device: primitives -> dz -> cell levels ->
// face jumps, for a fidelity level 1 grid (signed faces).
//
// Restates, per design and in f64:
//   * Primitive::profile (crates/itr-core/src/design.rs:107-134): distance to the primitive's
//     segment over half its width, (1 - s^2)^2 ridge or a flat-bottomed cut;
//   * DesignSpace::materialize (design.rs:316-385): 4x4 sub-sample quadrature per cell in the
//     union bounding box of the primitives, sum of height * mean profile over primitives,
//     masked by the editable cells, clamped to +-max_abs_dz; cut and fill volumes summed
//     over the box in row-major order;
//   * PreparedTerrain::apply_edit (crates/itr-hydro/src/terrain.rs:460-505) at level 1: cell
//     level z + dz (walls stay at z_wall) and every interior face jump f32(z_right - z_left),
//     the jumps of TerrainBase::build (terrain.rs:276-289) on the edited levels.
// The host evaluates each primitive's segment end points (sin and cos of its angle) with the
// same libm calls the reference makes, so every value here is an IEEE f64 add, multiply,
// divide or square root in the reference's order: the jumps equal the host path's bit for bit.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace itr {

// One primitive with its segment end points (Primitive::segment, design.rs:101-106).
struct MatPrim {
  double x0, y0, x1, y1;   // segment end points (equal for a mound)
  double width, height;
  double length;           // Primitive::length (the adjoint chain's d(end point)/dL)
  int kind;                // 0 berm, 1 swale, 2 cut, 3 mound
  int pad;
};

// One design: primitives [p0, p1) and the union bounding box, columns [c0, c1), rows [r0, r1)
// (empty when c0 >= c1 or r0 >= r1).
struct MatDesign {
  int p0, p1;
  int c0, r0, c1, r1;
};

struct MatArgs {
  int nx, ny, n;
  double ox, oy, dx, dy;   // GeoTransform of the grid
  double z_wall, max_abs_dz;
  const double* z;         // nx*ny base levels (walls at z_wall)
  const uint8_t* wall;     // nx*ny
  const uint8_t* editable; // nx*ny
  const MatPrim* prims;
  const MatDesign* des;
  double* dz;              // n * nx*ny
  double* ze;              // n * nx*ny edited levels
  float* dzx;              // n * ny*(nx+1)
  float* dzy;              // n * (ny+1)*nx
  double* cut;             // n
  double* fill;            // n
  const uint8_t* bc;       // boundary codes (ITR_BC_*) when stage depths are wanted, else NULL
  const double* stage;     // stage levels, indexed like bc
  float* bh;               // n * (2nx+2ny) stage-ghost depths
};

// Distance of (x, y) from the primitive's segment.
__device__ __forceinline__ double mat_distance(const MatPrim& p, double x, double y) {
  const double vx = p.x1 - p.x0, vy = p.y1 - p.y0;
  const double l2 = vx * vx + vy * vy;
  double t = 0.0;
  if (l2 > 0.0) {
    t = ((x - p.x0) * vx + (y - p.y0) * vy) / l2;
    t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
  }
  const double px = p.x0 + t * vx - x, py = p.y0 + t * vy - y;
  return sqrt(px * px + py * py);
}

// Primitive::profile (design.rs:107-134).
__device__ __forceinline__ double mat_profile(const MatPrim& p, double x, double y) {
  const double d = mat_distance(p, x, y);
  const double s = d / (0.5 * p.width);
  if (s >= 1.0) return 0.0;
  if (p.kind == 2) {   // cut: flat bottom, then a (1 - u^2)^2 bank
    if (s <= 0.5) return 1.0;
    const double u = (s - 0.5) / 0.5;
    const double w = 1.0 - u * u;
    return w * w;
  }
  const double w = 1.0 - s * s;
  return w * w;
}

// Every sub-sample of the cell centred on (x, y) lies outside the primitive, where its profile is 0: the
// samples are within 0.375 (dx + dy) of the centre, and 1e-9 of the coordinates' size covers the
// rounding. False for anything not a number, a negative width or an infinite height (0 times that).
__device__ __forceinline__ bool mat_outside(const MatPrim& p, double x, double y, double dx, double dy) {
  const double reach = 0.5 * p.width + 0.4 * (dx + dy) +
                       1e-9 * (fabs(x) + fabs(y) + fabs(p.x0) + fabs(p.y0) + fabs(p.x1) + fabs(p.y1));
  return p.width >= 0.0 && fabs(p.height) < 1e300 && mat_distance(p, x, y) > reach;
}

// dz and the edited level of every cell of every design (grid: cells / 256 x designs). Bound by f64
// divisions and square roots, 16 profiles per cell and primitive; the union box of a design is mostly
// outside any one primitive, and there one distance says that its sum is 0.
__global__ void k_materialize(const MatArgs M) {
  const int d = blockIdx.y;
  const size_t N = (size_t)M.nx * M.ny;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int r = (int)(i / M.nx), c = (int)(i % M.nx);
  const MatDesign D = M.des[d];
  double dz = 0.0;
  if (c >= D.c0 && c < D.c1 && r >= D.r0 && r < D.r1 && M.editable[i]) {
    double acc = 0.0;
    for (int q = D.p0; q < D.p1; ++q) {
      const MatPrim p = M.prims[q];
      if (p.height == 0.0 || mat_outside(p, M.ox + ((double)c + 0.5) * M.dx, M.oy - ((double)r + 0.5) * M.dy, M.dx, M.dy)) continue;
      double s = 0.0;
      for (int sy = 0; sy < 4; ++sy)
        for (int sx = 0; sx < 4; ++sx) {
          const double x = M.ox + ((double)c + ((double)sx + 0.5) / 4.0) * M.dx;
          const double y = M.oy - ((double)r + ((double)sy + 0.5) / 4.0) * M.dy;
          s += mat_profile(p, x, y);
        }
      acc += p.height * s * (1.0 / 16.0);
    }
    dz = acc < -M.max_abs_dz ? -M.max_abs_dz : (acc > M.max_abs_dz ? M.max_abs_dz : acc);
  }
  M.dz[(size_t)d * N + i] = dz;
  M.ze[(size_t)d * N + i] = M.wall[i] ? M.z_wall : M.z[i] + dz;
}

// Face jumps of the edited levels (domain-edge faces 0), and the stage ghosts' depths
// f32(max(stage - z, 0)) behind stage cells (grid: max(ny*(nx+1), (ny+1)*nx) / 256 x designs).
__global__ void k_mat_jumps(const MatArgs M) {
  const int d = blockIdx.y;
  const int nx = M.nx, ny = M.ny;
  const size_t N = (size_t)nx * ny;
  const double* ze = M.ze + (size_t)d * N;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < (size_t)ny * (nx + 1)) {
    const int r = (int)(i / (nx + 1)), f = (int)(i % (nx + 1));
    M.dzx[(size_t)d * ny * (nx + 1) + i] =
        (f >= 1 && f <= nx - 1) ? (float)(ze[(size_t)r * nx + f] - ze[(size_t)r * nx + f - 1]) : 0.0f;
  }
  if (i < (size_t)(ny + 1) * nx) {
    const int f = (int)(i / nx), c = (int)(i % nx);
    M.dzy[(size_t)d * (ny + 1) * nx + i] =
        (f >= 1 && f <= ny - 1) ? (float)(ze[(size_t)f * nx + c] - ze[(size_t)(f - 1) * nx + c]) : 0.0f;
  }
  const size_t NB = 2 * (size_t)(nx + ny);
  if (M.bh && i < NB) {
    // boundary cell i: north[nx], south[nx], west[ny], east[ny]
    size_t cell;
    if (i < (size_t)nx) cell = i;
    else if (i < 2 * (size_t)nx) cell = (size_t)(ny - 1) * nx + (i - nx);
    else if (i < 2 * (size_t)nx + ny) cell = (i - 2 * (size_t)nx) * nx;
    else cell = (i - 2 * (size_t)nx - ny) * nx + nx - 1;
    float h = 0.0f;
    if (M.bc[i] == 2) {
      const double v = M.stage[i] - ze[cell];
      h = (float)(v > 0.0 ? v : 0.0);
    }
    M.bh[(size_t)d * NB + i] = h;
  }
}

// Cut and fill volumes of each design's edit (design.rs:376-383), summed over its bounding
// box in row-major order as the reference does: a chain of f64 additions per volume, bit for bit. What
// bounds it is that chain, so only it is serial. One block per design takes the box in chunks of
// kVolChunk cells: every thread loads its cells and forms the products, the ones that are not 0
// (adding 0 changes nothing) are listed in order by ballots and counts, raised cells from the front and
// lowered ones from the back, and two threads of different warps add up the two lists while
// the other warps load the next chunk. With one warp per design walking the
// whole box, and every sample of every primitive evaluated, the materialisation of 16 designs of
// 1024 x 1024 took 18.9 ms; now 1.1 ms.
constexpr int kVolThreads = 512, kVolChunk = 8 * kVolThreads;

__global__ void __launch_bounds__(kVolThreads) k_mat_volumes(const MatArgs M) {
  __shared__ double list[kVolChunk];
  __shared__ int count[2][kVolThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, d = blockIdx.x;
  const MatDesign D = M.des[d];
  const double* dz = M.dz + (size_t)d * M.nx * M.ny;
  const double a = M.dx * M.dy;
  const int w = D.c1 > D.c0 ? D.c1 - D.c0 : 0, h = D.r1 > D.r0 ? D.r1 - D.r0 : 0, total = w * h;   // (at most 2^30 cells)
  const unsigned below = (1u << lane) - 1u;
  double sum = 0.0;   // thread 0: fill, thread 32: cut
  for (int base = 0; base < total; base += kVolChunk) {
    double p[8];
    unsigned up[8], dn[8];
    int nu = 0, nd = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int i = base + 256 * wid + 32 * k + lane;
      const double v = i < total ? dz[(size_t)(D.r0 + i / w) * M.nx + D.c0 + i % w] : 0.0;
      p[k] = v * a;
      up[k] = __ballot_sync(0xffffffffu, p[k] != 0.0 && v > 0.0);
      dn[k] = __ballot_sync(0xffffffffu, p[k] != 0.0 && !(v > 0.0));
      nu += __popc(up[k]); nd += __popc(dn[k]);
    }
    if (lane == 0) { count[0][wid] = nu; count[1][wid] = nd; }
    __syncthreads();   // (and the lists of the last chunk are summed)
    int ou = 0, od = 0, tu = 0, td = 0;
    for (int q = 0; q < kVolThreads / 32; ++q) {
      const int cu = count[0][q], cd = count[1][q];
      if (q < wid) { ou += cu; od += cd; }
      tu += cu; td += cd;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (up[k] >> lane & 1u) list[ou + __popc(up[k] & below)] = p[k];
      if (dn[k] >> lane & 1u) list[kVolChunk - 1 - (od + __popc(dn[k] & below))] = p[k];
      ou += __popc(up[k]); od += __popc(dn[k]);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 8
      for (int i = 0; i < tu; ++i) sum += list[i];
    } else if (threadIdx.x == 32) {
#pragma unroll 8
      for (int i = 0; i < td; ++i) sum -= list[kVolChunk - 1 - i];
    }
  }
  if (threadIdx.x == 0) M.fill[d] = sum;
  else if (threadIdx.x == 32) M.cut[d] = sum;
}

// ---- the design chain of the adjoint: dJ/d(height, width, length) per primitive ----
// dJ/d(dz) per cell from the face-jump gradients (level 1: each interior jump is the
// difference of its two cells' levels, the edge jumps stay 0, walls keep z_wall), then per
// primitive the derivative of the materialisation, written out from Primitive::profile
// (design.rs:107-134), contracted with it, plus the earthwork term lambda (cut_cost dV_cut +
// fill_cost dV_fill) (objective.rs:95-128).

// dJ/d(dz) of every cell of every design (grid: cells / 256 x designs).
__global__ void k_mat_gdz(int nx, int ny, const double* gx, const double* gy, const uint8_t* wall, double* gdz) {
  const int d = blockIdx.y;
  const size_t N = (size_t)nx * ny;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int r = (int)(i / nx), c = (int)(i % nx);
  const double* X = gx + (size_t)d * ny * (nx + 1) + (size_t)r * (nx + 1);
  const double* Y = gy + (size_t)d * (ny + 1) * nx;
  const double a = (c >= 1) ? X[c] : 0.0, b = (c + 1 <= nx - 1) ? X[c + 1] : 0.0;
  const double e = (r >= 1) ? Y[(size_t)r * nx + c] : 0.0, f = (r + 1 <= ny - 1) ? Y[(size_t)(r + 1) * nx + c] : 0.0;
  gdz[(size_t)d * N + i] = wall[i] ? 0.0 : ((a - b) + e) - f;
}

// The profile at (x, y) and its derivatives with respect to the primitive's width and length
// at fixed centre and angle. With s = d / (w / 2):
//   ridge P = (1 - s^2)^2, dP/ds = -4 s (1 - s^2);
//   cut   P = 1 for s <= 1/2, else (1 - u^2)^2 with u = 2 s - 1, dP/ds = -8 u (1 - u^2);
//   ds/dw = -s / w;  ds/dL = (2 / w) dd/dL, dd/dL = 0 beside the segment and, beyond an end,
//   the end's displacement (+-(cos a, sin a) / 2 per unit length) projected on the unit
//   vector from the sample to it.
__device__ __forceinline__ void mat_profile_d(const MatPrim& p, double x, double y, double& P, double& dw, double& dl) {
  P = 0.0; dw = 0.0; dl = 0.0;
  const double vx = p.x1 - p.x0, vy = p.y1 - p.y0;
  const double l2 = vx * vx + vy * vy;
  double t = 0.0;
  int end = 0;
  if (l2 > 0.0) {
    t = ((x - p.x0) * vx + (y - p.y0) * vy) / l2;
    if (t < 0.0) { t = 0.0; end = -1; }
    else if (t > 1.0) { t = 1.0; end = 1; }
  }
  const double px = p.x0 + t * vx - x, py = p.y0 + t * vy - y;
  const double d = sqrt(px * px + py * py);
  const double half = 0.5 * p.width;
  const double s = d / half;
  if (s >= 1.0) return;
  double dPds;
  if (p.kind == 2) {
    if (s <= 0.5) { P = 1.0; dPds = 0.0; }
    else { const double u = (s - 0.5) / 0.5, w = 1.0 - u * u; P = w * w; dPds = -8.0 * u * w; }
  } else {
    const double w = 1.0 - s * s;
    P = w * w; dPds = -4.0 * s * w;
  }
  dw = dPds * (-s / p.width);
  if (end != 0 && d > 0.0 && p.kind != 3 && p.length > 0.0) {
    const double ex = vx / (2.0 * p.length), ey = vy / (2.0 * p.length);
    dl = dPds * ((double)end * (px * ex + py * ey) / d) / half;
  }
}

// One primitive of one design: its own box of cells (materialize's box of that primitive).
struct MatJob {
  int design, prim;           // prim indexes the job's primitive table
  int c0, r0, c1, r1;
  int out;                    // output index (3 per primitive: height, width, length)
  int pad;
};

// Over a primitive's box, d(dz)/d(height, width, length) of every editable cell
// whose dz is not clamped, contracted with dJ/d(dz) plus the earthwork weight (the side of 0
// the cell's dz lies on; the mean of both sides at 0, as a central difference would see it). Bound by
// f64 divisions and square roots, as k_materialize, and like there most of a slanted box is outside the
// primitive. Blocks: primitives x slices of the box's cells (few primitives would leave the device
// idle: mat_dgrad_slices), each slice's sums at part + slice * stride; k_mat_dgrad_sum adds
// them in order.
inline int mat_dgrad_slices(int jobs, int sm_count) {
  const int s = 4 * (sm_count > 0 ? sm_count : 148) / (jobs > 0 ? jobs : 1);
  return s < 1 ? 1 : s > 64 ? 64 : s;
}
__global__ void k_mat_dgrad_sum(const double* part, int slices, int n, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double t = 0.0;
  for (int s = 0; s < slices; ++s) t += part[(size_t)s * n + i];
  out[i] = t;
}

__global__ void k_mat_dgrad(const MatArgs M, const MatPrim* jp, const MatJob* jobs, const double* dz, const double* gdz,
                            double earth_w, double cut_cost, double fill_cost, double* part, int stride) {
  const MatJob J = jobs[blockIdx.x];
  const MatPrim p = jp[J.prim];
  const int w = J.c1 - J.c0, h = J.r1 - J.r0;
  const size_t N = (size_t)M.nx * M.ny;
  const double area = M.dx * M.dy;
  double s[3] = {0, 0, 0};
  for (long long k = (long long)blockIdx.y * blockDim.x + threadIdx.x; w > 0 && h > 0 && k < (long long)w * h;
       k += (long long)gridDim.y * blockDim.x) {
    const int r = J.r0 + (int)(k / w), c = J.c0 + (int)(k % w);
    const size_t i = (size_t)r * M.nx + c;
    const double z = dz[(size_t)J.design * N + i];
    if (!M.editable[i] || !(z > -M.max_abs_dz && z < M.max_abs_dz)) continue;
    const double we = area * (z > 0.0 ? fill_cost : (z < 0.0 ? -cut_cost : 0.5 * (fill_cost - cut_cost)));
    const double g = gdz[(size_t)J.design * N + i] + earth_w * we;
    if (fabs(g) < 1e300 && mat_outside(p, M.ox + ((double)c + 0.5) * M.dx, M.oy - ((double)r + 0.5) * M.dy, M.dx, M.dy)) continue;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (int sy = 0; sy < 4; ++sy)
      for (int sx = 0; sx < 4; ++sx) {
        const double x = M.ox + ((double)c + ((double)sx + 0.5) / 4.0) * M.dx;
        const double y = M.oy - ((double)r + ((double)sy + 0.5) / 4.0) * M.dy;
        double P, dw, dl;
        mat_profile_d(p, x, y, P, dw, dl);
        a0 += P; a1 += dw; a2 += dl;
      }
    s[0] += g * a0 * (1.0 / 16.0);
    s[1] += g * p.height * a1 * (1.0 / 16.0);
    s[2] += g * p.height * a2 * (1.0 / 16.0);
  }
  __shared__ double red[32][3];
  for (int j = 0; j < 3; ++j)
    for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
  if ((threadIdx.x & 31) == 0)
    for (int j = 0; j < 3; ++j) red[threadIdx.x >> 5][j] = s[j];
  __syncthreads();
  if (threadIdx.x == 0) {
    double t[3] = {0, 0, 0};
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q)
      for (int j = 0; j < 3; ++j) t[j] += red[q][j];
    for (int j = 0; j < 3; ++j) part[(size_t)blockIdx.y * stride + J.out + j] = t[j];
  }
}

}  // namespace itr
