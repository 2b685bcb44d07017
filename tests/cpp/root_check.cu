// Compares the corrected root, the energy's root and the projection multiplier
// with the general operations of the device (sqrtf and the division, rounded to
// nearest) and prints the number of differences of each:
//   roots   every float of the exponents that the corrected root is used for
//   energy  every float from +0 to the last NaN
//   mults   pairs (h, lim): random bits, the bound near the root, and the roots
//           whose mantissas are the exceptional ones
#include <cstdio>

#include "hmf_multiplier.cuh"
#include "hmf_post.cuh"

using namespace hmf;

__device__ bool differ(float a, float b) {
  return __float_as_uint(a) != __float_as_uint(b) && !(a != a && b != b);
}

__device__ void report(unsigned long long mine, unsigned long long* count) {
  if (mine) atomicAdd(count, mine);
}

__global__ void check_roots(unsigned long long* count) {
  unsigned long long bad = 0;
  for (unsigned b = kMultLo + blockIdx.x * blockDim.x + threadIdx.x; b < kMultHi; b += gridDim.x * blockDim.x) {
    const float h = __uint_as_float(b);
    float y;
    bad += differ(corrected_root(h, y), sqrtf(h));
  }
  report(bad, count);
}

__global__ void check_energy(unsigned long long* count) {
  unsigned long long bad = 0;
  for (unsigned b = blockIdx.x * blockDim.x + threadIdx.x; b < 0x80000000u; b += gridDim.x * blockDim.x)
    bad += differ(energy_root(__uint_as_float(b)), sqrtf(__uint_as_float(b)));
  report(bad, count);
}

__device__ unsigned long long mix(unsigned long long x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__global__ void check_multipliers(unsigned long long pairs, unsigned long long* count, unsigned long long* used) {
  unsigned long long bad = 0, n = 0;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += stride) {
    const unsigned long long r = mix(i);
    unsigned hb = kMultLo + (unsigned)((r & 0xffffffffu) % (kMultHi - kMultLo));
    if ((i & 7) == 7) hb = (hb & ~0x7fffffu) | (0x7fffffu - (unsigned)(r >> 60));  // the last mantissas
    const float h = __uint_as_float(hb);
    unsigned lb = kMultLo + (unsigned)((r >> 32) % (kMultHi - kMultLo));
    if (i & 1) lb = __float_as_uint(sqrtf(h)) - 2u + (unsigned)((r >> 40) & 3u);  // the bound near the root
    const float lim = __uint_as_float(lb);
    if (multiplier_unsafe(h, lim)) continue;
    const float F = sqrtf(h);
    float root;
    const float q = multiplier_root(h, lim, root);
    bad += differ(multiplier_fast(h, lim), F > lim ? lim / F : 1.0f) + (F > lim && differ(q, lim / F));
    ++n;
  }
  report(bad, count);
  report(n, used);
}

int main() {
  unsigned long long* d = nullptr;
  unsigned long long h[4] = {0, 0, 0, 0};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 1;
  const int blocks = 152 * 8;
  const unsigned long long pairs = 4ull << 30;
  check_roots<<<blocks, 256>>>(d);
  check_energy<<<blocks, 256>>>(d + 1);
  check_multipliers<<<blocks, 256>>>(pairs, d + 2, d + 3);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  std::printf("roots %llu energy %llu mults %llu of %llu\n", h[0], h[1], h[2], h[3]);
  cudaFree(d);
  return 0;
}
