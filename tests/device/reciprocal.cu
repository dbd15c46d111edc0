// Compares reciprocal() with the division over n values of d: prints the
// largest difference in units of the last place and how many differ.
#include <cstdio>
#include <cstdlib>

#include "../../dim2d_finite_volume_b200/csrc/dim2d_physics.cuh"

__device__ unsigned long long g_differ, g_most;

// splitmix64
__device__ unsigned long long bits_of(unsigned long long i) {
  unsigned long long z = i * 0x9e3779b97f4a7c15ull + 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// kind 0: any sign, exponents -1020 .. 1020; 1: rho (3 - rho) for rho in (0, 3);
// 2: rows of neighbours of the powers of two
__global__ void k_compare(int kind, unsigned long long n) {
  const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += step) {
    const unsigned long long r = bits_of(i), mantissa = r & 0xfffffffffffffull;
    double d;
    if (kind == 0) {
      const unsigned long long e = 3 + (r >> 52) % 2041;
      d = __longlong_as_double((long long)((r & 0x8000000000000000ull) | e << 52 | mantissa));
    } else if (kind == 1) {
      const double rho = 3.0 * ((double)(r >> 11) + 0.5) * 0x1p-53;
      d = rho * (3.0 - rho);
    } else {
      d = __longlong_as_double((long long)(((3 + i / 64 % 2041) << 52) + i % 64 - 32));
    }
    const long long a = __double_as_longlong(dim2d::reciprocal(d));
    const long long b = __double_as_longlong(1.0 / d);
    const unsigned long long off = a > b ? a - b : b - a;
    if (off) {
      atomicAdd(&g_differ, 1ull);
      atomicMax(&g_most, off);
    }
  }
}

int main(int, char** argv) {
  const int kind = atoi(argv[1]);
  const unsigned long long n = strtoull(argv[2], nullptr, 10);
  k_compare<<<1024, 256>>>(kind, n);
  unsigned long long differ = 0, most = 0;
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(&differ, g_differ, sizeof differ);
  if (e == cudaSuccess) e = cudaMemcpyFromSymbol(&most, g_most, sizeof most);
  printf("%s %llu %llu\n", cudaGetErrorString(e), differ, most);
  return e == cudaSuccess ? 0 : 1;
}
