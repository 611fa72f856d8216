// The six digits of float-float values (ex_ff_digits): each within BF16's exact
// integers (256; the first 128) and their sum within half a unit of the last
// digit of the value, for uniform and wide-ranging values and for values
// whose second remainder is a tie with a low half beside it.
#include <cstdio>

#include "exact_gemm.cuh"

using namespace sigma;

__global__ void check(int n, int* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long s = (unsigned long long)(i + 1) * 0x9E3779B97F4A7C15ull;
  auto uni = [&]() {  // [0, 1)
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(s >> 11) * 0x1p-53;
  };
  double x;
  const int kind = i % 3;
  if (kind == 0)
    x = 2.0 * uni() - 1.0;
  else if (kind == 1)
    x = (2.0 * uni() - 1.0) * exp2(-50.0 * uni());
  else
    x = (64 + (int)(63 * uni()) + ((int)(511 * uni()) - 255 + 0.5) / 512.0) / 128.0 + (2.0 * uni() - 1.0) * 0x1p-25;
  if (i & 8) x = -x;
  const float hi = (float)x, lo = (float)(x - (double)hi);
  const int e = i % 7 - 3;  // units of 2^e
  const float f = exp2f((float)e);
  float2 d[6];
  ex_ff_digits(make_float2(hi * f, -hi * f), make_float2(lo * f, -lo * f), -exp2f((float)(7 - e)), d);
  double a = 0.0, b = 0.0, w = 0x1p-7;
  bool ok = fabsf(d[0].x) <= 128.f;
  for (int k = 0; k < 6; ++k, w *= 0x1p-9) {
    a += d[k].x * w;
    b += d[k].y * w;
    ok = ok && fabsf(d[k].x) <= 256.f && d[k].x == rintf(d[k].x) && d[k].y == -d[k].x;
  }
  const double v = (double)hi + (double)lo;
  if (!ok || fabs(a - v) > 0x1.1p-53 || fabs(b + v) > 0x1.1p-53) atomicAdd(bad, 1);
}

int main() {
  int *bad = nullptr, h = -1;
  const int n = 3 << 20;
  if (cudaMalloc(&bad, sizeof(int)) != cudaSuccess) return 2;
  cudaMemset(bad, 0, sizeof(int));
  check<<<n / 256, 256>>>(n, bad);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  cudaMemcpy(&h, bad, sizeof(int), cudaMemcpyDeviceToHost);
  printf("%d bad\n", h);
  return h != 0;
}
