// Bitwise check of mf_ieee64.cuh against the FP64 instructions: counts of
// results that differ, for every leading 24 bits of a significand (the
// approximation's whole domain) with seeded low bits and exponents, for
// quotients and roots next to representable numbers, and for every pair of
// special values.
#include <cstdio>
#include <cstdint>
#include <cmath>
#include <cuda_runtime.h>

#include "mf_ieee64.cuh"

using namespace mf::ieee64;

__device__ uint64_t mix(uint64_t h) {
  h = (h ^ (h >> 30)) * 0xBF58476D1CE4E5B9ull;
  h = (h ^ (h >> 27)) * 0x94D049BB133111EBull;
  return h ^ (h >> 31);
}
__device__ double bits(uint64_t u) { return __longlong_as_double((long long)u); }
__device__ bool same(double a, double b) {
  return (__double_as_longlong(a) == __double_as_longlong(b)) || (isnan(a) && isnan(b));
}
__device__ double ref_minmod(double a, double b) {
  const double s = copysign(1.0, a);
  return s * fmax(0.0, fmin(fabs(a), s * b));
}

// out: div, root, comparisons, max/min, scale, minmod, mul
__device__ void one(double a, double b, unsigned* out) {
  if (!same(mul(a, b), __dmul_rn(a, b))) atomicAdd(&out[6], 1u);
  if (!same(div(a, b), __ddiv_rn(a, b))) atomicAdd(&out[0], 1u);
  if (!same(root(b), __dsqrt_rn(b))) atomicAdd(&out[1], 1u);
  if (lt(a, b) != (a < b) || le(a, b) != (a <= b)) atomicAdd(&out[2], 1u);
  const double x = maxnum(a, b), y = fmax(a, b), z = minnum(a, b), w = fmin(a, b);
  if (!(x == y || (isnan(x) && isnan(y))) || !(z == w || (isnan(z) && isnan(w))))
    atomicAdd(&out[3], 1u);
  if (!same(half(a), 0.5 * a) || !same(scale<-2>(a), 0.25 * a) || !same(scale<1>(a), a + a) ||
      !same(scale<6>(a), 64.0 * a) || !same(absval(a), fabs(a)) || !same(flip(a, ~0u), -a))
    atomicAdd(&out[4], 1u);
  if (!isnan(a) && !isnan(b) && minmod(a, b) != ref_minmod(a, b)) atomicAdd(&out[5], 1u);
}

__global__ void k_check(unsigned* out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 leading fraction bits
  for (int m = 0; m < 8; ++m) {
    const uint64_t r = mix(i * 8ull + m), s = mix(r + 12345);
    // b: fraction bits i, low bits random, all zero or all one
    const uint64_t low = (m & 3) == 1 ? 0 : (m & 3) == 2 ? 0x1fffffffull : (r & 0x1fffffffull);
    const uint64_t frac = ((uint64_t)(i & 0x7fffffu) << 29) | low;
    const int span = (m < 4) ? 60 : 1000;
    const double b = bits(((uint64_t)(1023 - span + (int)(s % (2 * span))) << 52) | frac);
    double a = bits((r & 0x800fffffffffffffull) |
                    ((uint64_t)(1023 - span + (int)((s >> 20) % (2 * span))) << 52));
    if (m == 3) a = nextafter(a * b, (s & 1) ? 1e308 : -1e308);  // quotient next to a number
    if (m == 5) a = b;
    if (m == 6) a = nextafter(b, (s & 1) ? 1e308 : 0.0);
    // products near the rounding's half-way points: few significant bits
    if (m == 7) one(bits(__double_as_longlong(a) & 0xfffffffff8000000ull),
                    bits((__double_as_longlong(b) & 0xfffffffffc000000ull) | ((s >> 40) & 3)), out);
    one(a, b, out);
    const double q = b * b;  // root next to a number
    if (!same(root(nextafter(q, (s & 1) ? 1e308 : 0.0)), __dsqrt_rn(nextafter(q, (s & 1) ? 1e308 : 0.0))) ||
        !same(root(q), __dsqrt_rn(q)))
      atomicAdd(&out[1], 1u);
  }
}

__global__ void k_special(unsigned* out) {
  const uint64_t v[20] = {0ull, 0x8000000000000000ull, 1ull, 0x8000000000000001ull,
                          0x000fffffffffffffull, 0x0010000000000000ull, 0x0010000000000001ull,
                          0x0020000000000000ull, 0x7fefffffffffffffull, 0xffefffffffffffffull,
                          0x7ff0000000000000ull, 0xfff0000000000000ull, 0x7ff8000000000000ull,
                          0xfff8000000000001ull, 0x3ff0000000000000ull, 0xbff0000000000000ull,
                          0x3fefffffffffffffull, 0x4000000000000001ull, 0x7fe0000000000000ull,
                          0x0340000000000003ull};
  for (int p = 0; p < 20; ++p)
    for (int q = 0; q < 20; ++q) one(bits(v[p]), bits(v[q]), out);
}

int main() {
  unsigned *d, h[7];
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 2;
  cudaMemset(d, 0, sizeof(h));
  k_check<<<(1 << 23) / 256, 256>>>(d);
  k_special<<<1, 1>>>(d);
  const cudaError_t e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
  printf("div %u\nroot %u\ncompare %u\nmaxmin %u\nscale %u\nminmod %u\nmul %u\nstatus %s\n", h[0],
         h[1], h[2], h[3], h[4], h[5], h[6], cudaGetErrorString(e));
  return e == cudaSuccess ? 0 : 1;
}
