// phasor() (csrc/phasor.cuh) of the FP32 arguments on standard input, two a lane
// pair: writes (re, im) of each to standard output.
#include <cstdio>
#include <vector>

#include "phasor.cuh"

__global__ void run(const float2 *x, int n, float4 *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const sfxc::cpair e = sfxc::phasor(x[i].x, x[i].y);
  out[i] = make_float4(e.re.x, e.im.x, e.re.y, e.im.y);
}

int main() {
  std::vector<float> x;
  float buf[4096];
  for (size_t n; (n = fread(buf, 4, 4096, stdin)) > 0;) x.insert(x.end(), buf, buf + n);
  const int pairs = (int)(x.size() / 2);
  if (pairs == 0) return 1;
  float2 *d;
  float4 *o;
  std::vector<float4> h(pairs);
  if (cudaMalloc(&d, pairs * sizeof(float2)) || cudaMalloc(&o, pairs * sizeof(float4)) ||
      cudaMemcpy(d, x.data(), pairs * sizeof(float2), cudaMemcpyHostToDevice))
    return 2;
  run<<<(pairs + 255) / 256, 256>>>(d, pairs, o);
  if (cudaMemcpy(h.data(), o, pairs * sizeof(float4), cudaMemcpyDeviceToHost)) return 3;
  return fwrite(h.data(), sizeof(float4), pairs, stdout) == (size_t)pairs ? 0 : 4;
}
