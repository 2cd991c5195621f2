// The cell update's branch-free reciprocal, quotient, root and third
// (csrc/lattice.cuh) beside the correctly rounded operations of CUDA, for the
// tests: counts the inputs for which the bits differ and keeps the first one.
#include <cstdint>

#include "../openludwig_b200/csrc/lattice.cuh"

namespace {

__device__ uint32_t hash(uint32_t x) {  // Wellons' lowbias32
  x = (x ^ (x >> 16)) * 0x7feb352du;
  x = (x ^ (x >> 15)) * 0x846ca68bu;
  return x ^ (x >> 16);
}

__device__ void both(int op, float a, float b, float &got, float &want) {
  switch (op) {
    case 0: got = ol::recip_nr(a); want = __frcp_rn(a); break;
    case 1: got = ol::sqrt_nr(a); want = __fsqrt_rn(a); break;
    case 2: got = ol::third_of(a); want = __fdiv_rn(a, 3.0f); break;
    default: got = ol::quotient_nr(a, b); want = __fdiv_rn(a, b); break;
  }
}

// op 0..2: all n floats from the bit pattern first on.  op 3: n pseudo-random
// pairs, the exponents of both operands in [64, 192).
__global__ void k_compare(int op, uint32_t first, uint32_t n, unsigned long long *bad,
                          uint32_t *example) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    float a = __uint_as_float(first + (uint32_t)i), b = 1.0f, got, want;
    if (op == 3) {
      a = __uint_as_float(hash(2u * (uint32_t)i + first) % 0x40000000u + 0x20000000u);
      b = __uint_as_float(hash(2u * (uint32_t)i + 1u + first) % 0x40000000u + 0x20000000u);
    }
    both(op, a, b, got, want);
    if (__float_as_uint(got) != __float_as_uint(want) && atomicAdd(bad, 1ull) == 0) {
      example[0] = __float_as_uint(a);
      example[1] = __float_as_uint(b);
    }
  }
}

__global__ void k_values(int op, const float *a, const float *b, int n, float *got, float *want) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) both(op, a[i], b[i], got[i], want[i]);
}

}  // namespace

// Device pointers; the null stream.  Returns the launch's CUDA status.
extern "C" int olp_compare(int op, uint32_t first, uint32_t n, unsigned long long *bad,
                           uint32_t *example) {
  k_compare<<<1184, 256>>>(op, first, n, bad, example);
  return (int)cudaDeviceSynchronize();
}
extern "C" int olp_values(int op, const float *a, const float *b, int n, float *got, float *want) {
  k_values<<<(n + 127) / 128, 128>>>(op, a, b, n, got, want);
  return (int)cudaDeviceSynchronize();
}
