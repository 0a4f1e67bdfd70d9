// Counts where the branch-free division, reciprocal and square root of Adam differ from CUDA's correctly
// rounded ones.  Built and driven by test_adam_arithmetic_gpu.py.
#include "../raf_b200/csrc/update_core.cuh"

using namespace rafb200;

struct Found {
  unsigned long long count;
  float a, b;  // operands of one of them
};

__device__ void report(Found* f, float a, float b) {
  if (atomicAdd(&f->count, 1ull) == 0ull) {
    f->a = a;
    f->b = b;
  }
}

// Every significand at exponents [lo, hi]: one float per thread, `which` 0 = reciprocal, 1 = square root.
__global__ void significands(int which, int lo, int hi, Found* f) {
  const long long total = (long long)(hi - lo + 1) << 23;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float(((unsigned)(lo + (int)(i >> 23) + 127) << 23) | (unsigned)(i & 0x7fffff));
    const float got = which ? sqrt_rn(x) : rcp_rn(x);
    const float want = which ? __fsqrt_rn(x) : __frcp_rn(x);
    if (__float_as_uint(got) != __float_as_uint(want)) report(f, x, 0.f);
  }
}

__device__ unsigned mix(unsigned long long x) {  // splitmix64, Steele, Lea and Flood (2014)
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return (unsigned)((x ^ (x >> 31)) >> 16);
}

// Quotients a / b with the exponents of a and b in the given ranges.  Every other a is the float next to
// (q + half a unit) * b for a random q: a quotient that lies as near to the middle of two floats as one can.
__global__ void quotients(int a_lo, int a_hi, int b_lo, int b_hi, long long n, Found* f) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const unsigned r0 = mix(4 * i), r1 = mix(4 * i + 1), r2 = mix(4 * i + 2);
    const int ea = a_lo + (int)(r2 % (unsigned)(a_hi - a_lo + 1)), eb = b_lo + (int)((r2 >> 12) % (unsigned)(b_hi - b_lo + 1));
    const float b = __uint_as_float(((unsigned)(eb + 127) << 23) | (r0 & 0x7fffff));
    float a = __uint_as_float(((unsigned)(ea + 127) << 23) | (r1 & 0x7fffff));
    if (i & 1) {
      const double q = (double)__uint_as_float((127u << 23) | (r1 & 0x7fffff)) + 0x1p-24;
      const float near = (float)(q * (double)__uint_as_float((127u << 23) | (r0 & 0x7fffff)));  // in [1, 4)
      a = near * __uint_as_float((unsigned)(ea - (near >= 2.f ? 1 : 0) + 127) << 23);
    }
    if ((r0 >> 30) & 1) a = -a;
    const float got = div_by(a, b, __frcp_rn(b)), want = __fdiv_rn(a, b);
    if (__float_as_uint(got) != __float_as_uint(want)) report(f, a, b);
  }
}

static int finish(Found* dev, Found* out) {
  cudaError_t rc = cudaMemcpy(out, dev, sizeof(Found), cudaMemcpyDeviceToHost);
  cudaFree(dev);
  return (int)rc;
}

extern "C" __attribute__((visibility("default"))) int check_significands(int which, int lo, int hi, Found* out) {
  Found* dev;
  if (cudaMalloc(&dev, sizeof(Found)) != cudaSuccess || cudaMemset(dev, 0, sizeof(Found)) != cudaSuccess) return -1;
  significands<<<148 * 8, 256>>>(which, lo, hi, dev);
  return finish(dev, out);
}

extern "C" __attribute__((visibility("default"))) int check_quotients(int a_lo, int a_hi, int b_lo, int b_hi, long long n, Found* out) {
  Found* dev;
  if (cudaMalloc(&dev, sizeof(Found)) != cudaSuccess || cudaMemset(dev, 0, sizeof(Found)) != cudaSuccess) return -1;
  quotients<<<148 * 8, 256>>>(a_lo, a_hi, b_lo, b_hi, n, dev);
  return finish(dev, out);
}
