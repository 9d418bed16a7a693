// Counts where the branch-free operations of itr_device.cuh differ from CUDA's IEEE-rounded ones over the operands
// that their comments state. Built and called by test_special_ops.py, with the library's floating-point flags.
#include "itr_device.cuh"

using namespace itr;

namespace {

enum { kRcp, kRcpScalar, kSqrt, kSqrtScalar, kDiv, kDivSub, kDivRn, kDivF32, kMulAdd, kCounts };

__device__ unsigned long long hash64(unsigned long long x) {   // splitmix64 (Steele, Lea, Flood 2014)
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
// sign, an exponent in [lo, hi] and a significand, the last bits' edges among them
__device__ float some_f32(unsigned long long h, int lo, int hi) {
  const unsigned kind = (unsigned)(h >> 60), m = kind < 2 ? 0u : kind < 4 ? 0x7fffffu : kind < 5 ? 1u : (unsigned)(h & 0x7fffffu);
  const int e = lo + (int)((h >> 24 & 0xffffu) % (unsigned)(hi - lo + 1));
  return __uint_as_float((unsigned)(h >> 59 & 1u) << 31 | (unsigned)(e + 127) << 23 | m);
}
__device__ double some_f64(unsigned long long h, unsigned long long g, int lo, int hi) {
  const unsigned kind = (unsigned)(g >> 60);
  const unsigned long long m = kind < 1 ? 0ull : kind < 2 ? 0xfffffffffffffull : h & 0xfffffffffffffull;
  const int e = lo + (int)((g & 0xffffu) % (unsigned)(hi - lo + 1));
  return __longlong_as_double((long long)((unsigned long long)(g >> 59 & 1u) << 63 | (unsigned long long)(e + 1023) << 52 | m));
}

// Every 32-bit pattern, paired with another pattern of the range.
__global__ void over_floats(unsigned long long* n) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long bad[4] = {0, 0, 0, 0};
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < 1ull << 32; i += stride) {
    const float x = __uint_as_float((unsigned)i);
    if (fabsf(x) >= 0x1p-125f && fabsf(x) < 0x1p126f) {
      const float z = some_f32(hash64(i), -125, 125);
      const float2 r = rcp2(make_float2(x, z));
      bad[0] += !same(r.x, __frcp_rn(x)) + !same(r.y, __frcp_rn(z));
      bad[1] += !same(Fast::rcp(x), __frcp_rn(x));
    }
    if (x < 0x1p80f && !((unsigned)i >> 31)) {
      const float z = fabsf(some_f32(hash64(i), -126, 79));
      const float2 r = sqrt2(make_float2(z, x));
      bad[2] += !same(r.x, __fsqrt_rn(z)) + !same(r.y, __fsqrt_rn(x));
      bad[3] += !same(Fast::sqrt(x), __fsqrt_rn(x)) + !same(sqrt_rn(x), __fsqrt_rn(x));
    }
  }
  for (int k = 0; k < 4; ++k) if (bad[k]) atomicAdd(n + k, bad[k]);
}

__global__ void over_samples(unsigned long long* n, unsigned long long samples, float nz) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long bad[kCounts] = {};
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < samples; i += stride) {
    const unsigned long long h = hash64(4 * i), g = hash64(4 * i + 1), u = hash64(4 * i + 2), v = hash64(4 * i + 3);
    {   // Fast::div: divisors 2^-125 .. 2^62; quotients below 2^127, of a scaled dividend below 2^63
      const float a = (h & 255) == 0 ? (g & 1 ? 0.0f : __uint_as_float(0x7f800000u + (unsigned)(g & 2))) : some_f32(h, -126, 126), b = some_f32(g, -125, 61);
      const float q = __fdiv_rn(a, b), r = Fast::div(a, b);
      const float most = fabsf(a) < 0x1p-60f ? 0x1p63f : 0x1p127f;
      if (q == 0.0f || !(fabsf(q) < 0x1p-126f)) { if (!(fabsf(q) >= most) || isinf(a)) bad[kDiv] += !same(q, r); }
      else bad[kDivSub] += !(fabsf(q - r) <= 0x1p-149f);
    }
    {   // div_rn
      const double a = (h & 255) == 0 ? 0.0 : some_f64(h, u, -400, 300), b = some_f64(g, v, -250, 250);
      bad[kDivRn] += div_rn(a, b, __drcp_rn(b)) != __ddiv_rn(a, b);
      const double s = (double)fabsf(some_f32(v, -126, 127));
      bad[kDivF32] += div_by_f32(fabs(some_f64(u, h, -200, 200)), s) != __ddiv_rn(fabs(some_f64(u, h, -200, 200)), s);
    }
    {   // a paired product and sum round twice
      const float2 a = make_float2(some_f32(h, -40, 40), some_f32(g, -40, 40)), b = make_float2(some_f32(u, -40, 40), some_f32(v, -40, 40));
      const float2 c = make_float2(some_f32(h ^ v, -40, 40), -__fmul_rn(a.y, b.y) * (1.0f + 0x1p-23f * (float)(g & 7u)));
      const float2 r = add2(mul2(a, b, nz), c), s = sub2(c, mul2(a, b, nz));
      bad[kMulAdd] += !same(r.x, __fadd_rn(__fmul_rn(a.x, b.x), c.x)) + !same(r.y, __fadd_rn(__fmul_rn(a.y, b.y), c.y));
      bad[kMulAdd] += !same(s.x, __fsub_rn(c.x, __fmul_rn(a.x, b.x))) + !same(s.y, __fsub_rn(c.y, __fmul_rn(a.y, b.y)));
    }
  }
  for (int k = 0; k < kCounts; ++k) if (bad[k]) atomicAdd(n + k, bad[k]);
}

}  // namespace

extern "C" int special_ops(unsigned long long* counts, unsigned long long samples) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, kCounts * 8) != cudaSuccess) return 1;
  cudaMemset(d, 0, kCounts * 8);
  over_floats<<<148 * 8, 256>>>(d);
  over_samples<<<148 * 8, 256>>>(d, samples, -0.0f);
  const cudaError_t e = cudaMemcpy(counts, d, kCounts * 8, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}
