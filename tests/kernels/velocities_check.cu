// Test kernel: the library's velocities (ymkh_common.cuh: px / n and pz / n
// through one reciprocal) against the IEEE divisions, bit for bit.
// Built by tests/test_gpu_fct_strip.py with nvcc; not part of the library.
#include "ymkh_common.cuh"

namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {  // splitmix64 finaliser
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double number(unsigned long long h, int e_lo, int e_n, bool all_ones) {
  const unsigned long long mant = all_ones ? 0x000FFFFFFFFFFFFFull - (h & 7) : h & 0x000FFFFFFFFFFFFFull;
  const unsigned long long e = (unsigned long long)(1023 + e_lo) + mix64(h) % (unsigned long long)e_n;
  return __longlong_as_double((long long)(((h >> 63) << 63) | (e << 52) | mant));
}

// n >= 0.05 (the density floor) but in kind 5.  kind 0: n near 1, momenta of any
// size; 1: n of any size up to 2^100; 2: momenta that put the quotient on or
// beside a double; 3: n with an all-ones mantissa; 4: special momenta and n;
// 5: n down to the 1e-10 of the field update.
__global__ void check(unsigned long long seed, long long count, int kind, unsigned long long* bad, double* first) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += stride) {
    const unsigned long long h = mix64(seed ^ mix64((unsigned long long)i)), g = mix64(h + 1), k = mix64(g + 1);
    double n = fabs(number(h, kind == 5 ? -33 : -4, kind == 1 ? 104 : (kind == 5 ? 40 : 8), kind == 3));
    double a = number(g, -1000, 2000, false), b = number(k, -40, 60, false);
    if (kind == 2) {
      a = number(g, -300, 600, false) * n;
      b = __longlong_as_double(__double_as_longlong(b * n) + ((k >> 1) & 1 ? 1 : -1));
    }
    if (kind == 4) {
      const double sp[12] = {0.0, -0.0, 0x1p-1070, -0x1p-1022, 0x1p-801, -0x1p-800, 0x1p900, 0x1p1020,
                             __longlong_as_double(0x7FF0000000000000ll), __longlong_as_double(0xFFF0000000000000ll),
                             __longlong_as_double(0x7FF8000000000000ll), 1.0};
      const double sn[4] = {0.05, 1.0, 0x1.8p91, __longlong_as_double(0x7FF0000000000000ll)};
      a = sp[i % 12];
      b = sp[(i / 12) % 12];
      n = sn[(i / 144) % 4];
    }
    n = fmax(n, kind == 5 ? 1e-10 : 0.05);
    double u, v;
    ymkh::velocities(n, a, b, u, v);
    const double wu = a / n, wv = b / n;
    const bool same = (__double_as_longlong(u) == __double_as_longlong(wu) || (u != u && wu != wu)) &&
                      (__double_as_longlong(v) == __double_as_longlong(wv) || (v != v && wv != wv));
    if (!same && atomicAdd(bad, 1ull) == 0ull) {
      first[0] = n;
      first[1] = a;
    }
  }
}

}  // namespace

extern "C" int velocities_check(unsigned long long seed, long long count, int kind, unsigned long long* host_bad,
                                double* host_first) {
  unsigned long long* d_bad = nullptr;
  double* d_first = nullptr;
  if (cudaMalloc(&d_bad, sizeof(unsigned long long)) != cudaSuccess) return 1;
  if (cudaMalloc(&d_first, 2 * sizeof(double)) != cudaSuccess) return 1;
  cudaMemset(d_bad, 0, sizeof(unsigned long long));
  cudaMemset(d_first, 0, 2 * sizeof(double));
  check<<<148 * 8, 256>>>(seed, count, kind, d_bad, d_first);
  if (cudaMemcpy(host_bad, d_bad, sizeof(unsigned long long), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  if (cudaMemcpy(host_first, d_first, 2 * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  cudaFree(d_bad);
  cudaFree(d_first);
  return 0;
}
