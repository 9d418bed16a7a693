// itr_pack.cuh — the inputs of the cluster kernel as its lanes read them (BatchArgs::G, J, J2).
//
// A record holds the operands of one pair of columns of one row: wet and g n^2 in G (shared by
// the designs), in J the jumps of the two north y-faces and of the two west x-faces. A lane then
// reads a row's operands with two 16-byte loads; from the caller's separate arrays, whose rows of
// nx + 1 floats are not aligned to pairs, it took eight 4-byte copies and their addresses. One pass
// over the inputs per call. Columns and faces outside the grid get zeros.
#pragma once
#include "itr_batched.cuh"

namespace itr {

struct PackArgs {
  int nx, ny, n;
  const float *wet, *gn2, *dzx, *dzy, *dzx2, *dzy2;   // as itr_grid / itr_design (dzx2, dzy2: crest only)
  const uint8_t* bc;
  const float* bh;      // stage-ghost depths per design, or NULL
  float4 *G, *J, *J2;
  unsigned* never;      // per design, zeroed: set when a crest jump or a stage depth is out of bounds
};

// Blocks of records x designs (more designs than a grid's y extent holds take turns).
__global__ void k_pack_inputs(const PackArgs A) {
  const int nx = A.nx, ny = A.ny, PJ = pairs(nx) + 2;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int f = i / PJ, c = 2 * (i % PJ - 1);   // face row and first column of the record
  auto at = [](const float* a, int row, int stride, int col, bool in) { return in ? a[(size_t)row * stride + col] : 0.0f; };
  const bool y0 = c >= 0 && c < nx, y1 = c + 1 >= 0 && c + 1 < nx;
  const bool x0 = f < ny && c >= 0 && c <= nx, x1 = f < ny && c + 1 >= 0 && c + 1 <= nx;
  for (int d = blockIdx.y; d < A.n; d += gridDim.y) {
    if (A.bh && blockIdx.x == 0) {
      const int nbc = 2 * (nx + ny);
      for (int b = threadIdx.x; b < nbc; b += blockDim.x)
        if (!stage_safe(A.bc[b], A.bh[(size_t)d * nbc + b])) A.never[d] = 1u;
    }
    if (i >= (ny + 1) * PJ) continue;
    const float* x = A.dzx + (size_t)d * ny * (nx + 1);
    const float* y = A.dzy + (size_t)d * (ny + 1) * nx;
    const float4 j = make_float4(at(y, f, nx, c, y0), at(y, f, nx, c + 1, y1), at(x, f, nx + 1, c, x0), at(x, f, nx + 1, c + 1, x1));
    A.J[(size_t)d * (ny + 1) * PJ + i] = j;
    if (A.J2) {
      const float* x2 = A.dzx2 + (size_t)d * ny * (nx + 1);
      const float* y2 = A.dzy2 + (size_t)d * (ny + 1) * nx;
      const float4 k = make_float4(at(y2, f, nx, c, y0), at(y2, f, nx, c + 1, y1), at(x2, f, nx + 1, c, x0), at(x2, f, nx + 1, c + 1, x1));
      A.J2[(size_t)d * (ny + 1) * PJ + i] = k;
      if (!(jump_safe(j.x) && jump_safe(j.y) && jump_safe(j.z) && jump_safe(j.w) && jump_safe(k.x) && jump_safe(k.y) && jump_safe(k.z) &&
            jump_safe(k.w)))
        A.never[d] = 1u;
    }
    if (d == 0 && f < ny)
      A.G[i] = make_float4(at(A.wet, f, nx, c, y0), at(A.wet, f, nx, c + 1, y1), at(A.gn2, f, nx, c, y0), at(A.gn2, f, nx, c + 1, y1));
  }
}

// Start depths of every design: hinit on wet cells (init_state, solver.rs:381-390). Blocks of cells x designs.
__global__ void k_fill_start(const float* wet, size_t N, int n, float hinit, float* h0) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const float h = wet[i] != 0.0f ? hinit : 0.0f;
  for (int d = blockIdx.y; d < n; d += gridDim.y) h0[(size_t)d * N + i] = h;
}

}  // namespace itr
