// The rectilinear march's quotients against CUDA's division: for pairs counted
// out of `seed`, how many differ.
#include "../ascent_gb300/csrc/gvr_march_device.cuh"

namespace {
__device__ unsigned mix(unsigned long long x)
{
  x ^= x >> 33; x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull;
  return (unsigned)(x ^ x >> 33);
}

// b = 1.m 2^e for e in [lo, hi], a up to 38 powers of two below b
__global__ void differ(unsigned long long seed, long long n, int lo, int hi, unsigned long long *count)
{
  unsigned bad = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const unsigned u = mix(seed + 3 * i), v = mix(seed + 3 * i + 1), w = mix(seed + 3 * i + 2);
    const float b = scalbnf(1.f + (float)(u & 0x7fffff) * 0x1p-23f, lo + (int)(w % (unsigned)(hi - lo + 1)));
    float a = scalbnf((1.f + (float)(v & 0x7fffff) * 0x1p-23f) * b, -(int)(w >> 16 & 31) - (int)(w >> 21 & 7));
    if (w >> 28 == 0) a = w >> 24 & 1 ? b : 0.f;
    if (a > b) a = b;
    bad += gvr::div_by(a, b, 1.0f / b) != a / b;
  }
  if (bad) atomicAdd(count, (unsigned long long)bad);
}
}  // namespace

extern "C" __attribute__((visibility("default"))) long long differing(unsigned long long seed, long long n, int lo, int hi)
{
  unsigned long long *d = nullptr, h = ~0ull;
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof(h));
  differ<<<152 * 8, 256>>>(seed, n, lo, hi, d);
  cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaGetLastError();
  cudaFree(d);
  return e == cudaSuccess ? (long long)h : -1;
}
