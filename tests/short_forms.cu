// The straight-line roots and reciprocals of fp_elements.cuh against CUDA's
// correctly rounded ones: counts of differing values, one "name count" a line
// (run by test_gpu_short_forms.py).
#include <cstdio>

#include "fp_internal.cuh"
#include "fp_elements.cuh"

using namespace fpb;

__device__ unsigned long long mix(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
__device__ int ulps(double a, double b) {
  const long long d = llabs(__double_as_longlong(a) - __double_as_longlong(b));
  return d > 1000 ? 1000 : (int)d;
}
// random mantissas (ones: the last 16 below all ones) of the exponents lo .. hi - 1
__global__ void f64(int lo, int hi, bool ones, int per, unsigned long long* out) {
  const unsigned long long id = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  int n[4] = {}, far = 0;
  for (int i = 0; i < per; ++i) {
    const unsigned long long h = mix(id * per + i), e = mix(h) % (unsigned)(hi - lo);
    const unsigned long long man = ones ? 0xfffffffffffffull - (h & 15) : h & 0xfffffffffffffull;
    const double d = __longlong_as_double((long long)((e + lo + 1023) << 52 | man));
    const double got[4] = {near_rcp(d), newton_rcp(-d), near_inv(d, 0.0), near_inv(d, 1e-8)};
    const double ref[4] = {__drcp_rn(d), __drcp_rn(-d), __drcp_rn(__dsqrt_rn(d)), __drcp_rn(__dsqrt_rn(d) + 1e-8)};
    for (int k = 0; k < 4; ++k) {
      n[k] += got[k] != ref[k];
      far += ulps(got[k], ref[k]) > 1;
    }
  }
  for (int k = 0; k < 4; ++k) atomicAdd(out + k, (unsigned long long)n[k]);
  atomicAdd(out + 4, (unsigned long long)far);
}
// every FP32 value of the exponents -100 .. 99
__global__ void f32(unsigned long long* out) {
  const unsigned first = (unsigned)(127 - 100) << 23, last = (unsigned)(127 + 100) << 23;
  int r = 0, s = 0;
  for (unsigned b = first + blockIdx.x * blockDim.x + threadIdx.x; b < last; b += gridDim.x * blockDim.x) {
    const float x = __uint_as_float(b);
    r += exact_rcp<true>(x) != __frcp_rn(x);
    s += exact_sqrt<true>(x) != __fsqrt_rn(x);
  }
  atomicAdd(out, (unsigned long long)r);
  atomicAdd(out + 1, (unsigned long long)s);
}

int main() {
  unsigned long long* n;
  if (cudaMallocManaged(&n, 5 * sizeof(*n))) return 1;
  const char* names[5] = {"rcp64", "rcp64_negative", "inv64", "inv64_offset", "far64"};
  for (int ones = 0; ones < 2; ++ones) {
    for (int k = 0; k < 5; ++k) n[k] = 0;
    f64<<<148 * 8, 256>>>(-990, 990, ones, ones ? 100 : 2000, n);
    if (cudaDeviceSynchronize()) return 1;
    for (int k = 0; k < 5; ++k) printf("%s%s %llu\n", names[k], ones ? "_ones" : "", n[k]);
  }
  n[0] = n[1] = 0;
  f32<<<148 * 8, 256>>>(n);
  if (cudaDeviceSynchronize()) return 1;
  printf("rcp32 %llu\nsqrt32 %llu\n", n[0], n[1]);
  return 0;
}
