// SPDX-License-Identifier: MPL-2.0
// The mean shift's quotients (meanshift_fast.cuh) against the division, bit for bit:
// quotient over random and edge operands, over(d2, window(h2)) for windows of any
// size through the weight 1 - x it is used in.  Prints the mismatches of each and how many were compared.
#include "meanshift_fast.cuh"

#include <cstdio>
#include <cstring>
#include <vector>

using namespace sym;

__host__ __device__ uint64_t mix(uint64_t z) {  // splitmix64
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

// The bounds of quotient's range, their neighbours, zeros, subnormals, the largest
// values, infinities and NaN.
constexpr int kEdges = 22;
__device__ float edge(int i) {
  const float at[6] = {1e-20f, 1e-14f, 1e12f, 1e20f, 1.17549435e-38f, 1.f};
  if (i < 18) return __uint_as_float(__float_as_uint(at[i / 3]) + i % 3 - 1);
  const float more[4] = {0.f, 1e-45f, INFINITY, NAN};
  return more[i - 18];
}

constexpr int kWindows = 1 << 16;

__global__ void check(uint64_t n, const float *h2s, const Window<float> *windows, unsigned long long *bad) {
  const uint64_t at = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x, step = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = at; i < n; i += step) {
    const uint64_t z = mix(i);
    uint32_t ua = uint32_t(z), ub = uint32_t(z >> 32);
    if (i & 1) {  // exponents in the range of the residual form
      ua = (ua & 0x807fffffu) | ((70 + (ua >> 24) % 110) << 23);
      ub = (ub & 0x807fffffu) | ((85 + (ub >> 24) % 80) << 23);
    }
    const float a = __uint_as_float(ua), b = __uint_as_float(ub);
    if (!same(quotient(a, b), a / b)) atomicAdd(&bad[0], 1ull);
    // a vote anywhere within it (or far inside)
    const float h2 = h2s[i % kWindows];
    const float in = i & 2 ? float(mix(z + 1) >> 40) * 0x1p-24f : __uint_as_float(uint32_t(mix(z + 1)) % 0x3f800000u);
    const float d2 = h2 < INFINITY ? h2 * in : fabsf(a);
    if (d2 < h2 && !same(1.f - over(d2, windows[i % kWindows]), 1.f - d2 / h2)) atomicAdd(&bad[1], 1ull);
  }
  for (uint64_t i = at; i < 4 * kEdges * kEdges; i += step) {
    const float a = edge(int(i / 4 / kEdges)) * (i & 1 ? -1.f : 1.f);
    const float b = edge(int(i / 4 % kEdges)) * (i & 2 ? -1.f : 1.f);
    if (!same(quotient(a, b), a / b)) atomicAdd(&bad[0], 1ull);
  }
}

int main() {
  const uint64_t n = 1ull << 26;
  std::vector<float> h2(kWindows);
  std::vector<Window<float>> win(kWindows);
  for (int i = 0; i < kWindows; ++i) {  // every exponent, subnormals among them, and infinity
    const uint32_t bits = i ? uint32_t(mix(i)) % 0x7f800000u : 0x7f800000u;
    std::memcpy(&h2[i], &bits, 4);
    win[i] = window(h2[i]);
  }
  unsigned long long *bad, host[2] = {~0ull, ~0ull};
  float *dh;
  Window<float> *dw;
  if (cudaMalloc(&bad, 16) || cudaMemset(bad, 0, 16) || cudaMalloc(&dh, 4 * kWindows) ||
      cudaMalloc(&dw, sizeof(Window<float>) * kWindows) ||
      cudaMemcpy(dh, h2.data(), 4 * kWindows, cudaMemcpyHostToDevice) ||
      cudaMemcpy(dw, win.data(), sizeof(Window<float>) * kWindows, cudaMemcpyHostToDevice))
    return 1;
  check<<<152 * 4, 256>>>(n, dh, dw, bad);
  if (cudaDeviceSynchronize() || cudaMemcpy(host, bad, 16, cudaMemcpyDeviceToHost)) return 1;
  std::printf("%llu %llu of %llu\n", host[0], host[1], (unsigned long long)n);
  return host[0] || host[1] ? 2 : 0;
}
