// minmod, the maxima and the comparisons of mf_ieee64.cuh against the FP64
// forms for every pair of special values, NaN of either sign and kind among
// them: counts of results that differ in a bit (or, for a NaN, in being one).
#include <cstdio>
#include <cstdint>
#include <cmath>
#include <cuda_runtime.h>

#include "mf_ieee64.cuh"

using namespace mf::ieee64;

__device__ double bits(uint64_t u) { return __longlong_as_double((long long)u); }
__device__ bool same(double a, double b) {
  return (__double_as_longlong(a) == __double_as_longlong(b)) || (isnan(a) && isnan(b));
}
__device__ double ref_minmod(double a, double b) {
  const double s = copysign(1.0, a);
  return s * fmax(0.0, fmin(fabs(a), s * b));
}

__global__ void k_check(const uint64_t* v, int quiet, unsigned* out) {
  const int p = threadIdx.x, q = blockIdx.x;
  const double a = bits(v[p]), b = bits(v[q]);
  // differences of the state: never a signalling NaN
  if (p < quiet && q < quiet && !same(minmod(a, b), ref_minmod(a, b))) atomicAdd(&out[0], 1u);
  const double x = maxnum(a, b), y = fmax(a, b), z = minnum(a, b), w = fmin(a, b);
  if (!(x == y || (isnan(x) && isnan(y))) || !(z == w || (isnan(z) && isnan(w))))
    atomicAdd(&out[1], 1u);
  if (lt(a, b) != (a < b) || le(a, b) != (a <= b)) atomicAdd(&out[2], 1u);
}

int main() {
  const uint64_t v[22] = {0ull, 0x8000000000000000ull, 1ull, 0x8000000000000001ull,
                          0x0010000000000000ull, 0x3ff0000000000000ull, 0xbff0000000000000ull,
                          0x4000000000000001ull, 0xc000000000000001ull, 0x7fefffffffffffffull,
                          0xffefffffffffffffull, 0x7ff0000000000000ull, 0xfff0000000000000ull,
                          0x7ff8000000000000ull, 0xfff8000000000000ull, 0x7fffffffffffffffull,
                          0xffffffffffffffffull, 0x7ff8000000000001ull,
                          // signalling: payload in the high, then the low word
                          0x7ff0000100000000ull, 0xfff4000000000000ull, 0x7ff0000000000001ull,
                          0xfff00000ffffffffull};
  uint64_t* d = nullptr;
  unsigned *o = nullptr, h[3];
  if (cudaMalloc(&d, sizeof(v)) != cudaSuccess || cudaMalloc(&o, sizeof(h)) != cudaSuccess)
    return 2;
  cudaMemcpy(d, v, sizeof(v), cudaMemcpyHostToDevice);
  cudaMemset(o, 0, sizeof(h));
  k_check<<<22, 22>>>(d, 18, o);
  const cudaError_t e = cudaMemcpy(h, o, sizeof(h), cudaMemcpyDeviceToHost);
  printf("minmod %u\nmaxmin %u\ncompare %u\nstatus %s\n", h[0], h[1], h[2], cudaGetErrorString(e));
  return e == cudaSuccess ? 0 : 1;
}
