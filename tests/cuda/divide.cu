// The sweeps' division by a divisor known ahead against the correctly rounded
// division, bit for bit: random operands over all exponents, and dividends that
// put the quotient next to the middle of two doubles.  Test infrastructure only.
#include "../../seldon_b200/csrc/sweep.cuh"

namespace {

__device__ unsigned long long mix(unsigned long long x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

// sign and mantissa from r, exponent within e of 1 (all of them with e = 0)
__device__ double draw(unsigned long long r, int e) {
  const unsigned long long field = e ? 1023ull - e + mix(r) % (2ull * e + 1) : mix(r) & 2047ull;
  return __longlong_as_double((long long)((r & 0x800fffffffffffffull) | field << 52));
}

__global__ void compare(unsigned long long seed, long long n, unsigned long long* bad, double* first) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long r = mix(seed + (unsigned long long)i), q = mix(r + 1);
    const int kind = (int)(i & 3);  // two in four: near a middle; one within the range of both
    const int e = kind == 3 ? 0 : kind == 2 ? 420 : 150;
    const double b = draw(r, e);
    double a = draw(q, e);
    if (kind < 2) {
      // b (c + ulp / 2) to the nearest double, or a neighbour
      const double c = draw(q, 20), half = __dmul_rn(c, 0x1p-53);
      a = __fma_rn(b, c, __dmul_rn(b, half));
      if (kind == 1) a = __longlong_as_double(__double_as_longlong(a) + (long long)(q % 3) - 1);
    }
    const double want = __ddiv_rn(a, b), got = sb2::Divisor(b).divide(a);
    if (__double_as_longlong(want) != __double_as_longlong(got) && !(want != want && got != got)) {
      if (atomicAdd(bad, 1ull) == 0) {
        first[0] = a;
        first[1] = b;
      }
    }
  }
}

}  // namespace

extern "C" int compare_division(unsigned long long seed, long long n, unsigned long long* bad, double* first) {
  char* d = nullptr;
  if (cudaMalloc(&d, 32) != cudaSuccess) return -1;
  cudaError_t e = cudaMemset(d, 0, 32);
  if (e == cudaSuccess) {
    compare<<<1184, 256>>>(seed, n, reinterpret_cast<unsigned long long*>(d), reinterpret_cast<double*>(d + 8));
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(bad, d, sizeof(*bad), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(first, d + 8, 2 * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : -2;
}
