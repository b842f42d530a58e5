// Test infrastructure only: the fused epilogues' SiLU, its derivative and their
// division (chaos_oneapi_b200/csrc/mlp_fused.h) against the plain functions and
// the `/` operator on every 32-bit float.  Built and run by
// tests/test_gpu_silu.py; never linked into the library.
//
// Prints one line per comparison: name, values compared, values that differ
// (NaN equals NaN), largest difference in units of the last place.
#include <cstdio>
#include <cstring>

#include "../../chaos_oneapi_b200/csrc/mlp_fused.h"

using namespace chaos::mlp;

struct Count {
  unsigned long long seen, differ, ulps;
};
enum { kSilu, kSiluAlone, kDsilu, kQuotient, kReciprocal, kCounts };
__device__ Count counts[kCounts];

// Floats in order, as consecutive integers.
__device__ long long rank_of(float x) {
  const int b = __float_as_int(x);
  return b < 0 ? -(long long)(b & 0x7fffffff) : b;
}
__device__ void compare(Count &c, float got, float want) {
  c.seen++;
  if (got == want ? __float_as_int(got) == __float_as_int(want) : isnan(got) && isnan(want)) return;
  c.differ++;
  const unsigned long long d = isnan(got) || isnan(want)
                                   ? 1ull << 32
                                   : (unsigned long long)llabs(rank_of(got) - rank_of(want));
  if (d > c.ulps) c.ulps = d;
}

// 16 consecutive bit patterns per chunk, as a thread of the epilogues holds 16
// columns.
__global__ void check_kernel() {
  Count c[kCounts] = {};
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       i < (1ull << 28); i += (unsigned long long)gridDim.x * blockDim.x) {
    float x[16], s[16], ds[16], u[16];
    for (int j = 0; j < 16; j++) {
      x[j] = __int_as_float((int)(unsigned)(i * 16 + j));
      s[j] = ds[j] = x[j];
      u[j] = 1.f + 0.0625f * j;
    }
    silu_chunk(s);
    dsilu_chunk(u, ds);
    for (int j = 0; j < 16; j++) {
      compare(c[kSilu], s[j], silu(x[j]));
      compare(c[kDsilu], ds[j], u[j] * dsilu(x[j]));
      float one[1] = {x[j]};
      silu_chunk(one);
      compare(c[kSiluAlone], one[0], silu(x[j]));
      const float d = one_plus_exp_neg(x[j]);
      if (d < kFastDivLimit && !isinf(x[j])) compare(c[kQuotient], divide_above_one(x[j], d), x[j] / d);
      if (x[j] >= 1.f && x[j] < kFastDivLimit)
        compare(c[kReciprocal], divide_above_one(1.f, x[j]), 1.f / x[j]);
    }
  }
  for (int k = 0; k < kCounts; k++) {
    atomicAdd(&counts[k].seen, c[k].seen);
    atomicAdd(&counts[k].differ, c[k].differ);
    atomicMax(&counts[k].ulps, c[k].ulps);
  }
}

int main() {
  check_kernel<<<148 * 8, 256>>>();
  Count c[kCounts];
  const cudaError_t e = cudaMemcpyFromSymbol(c, counts, sizeof c);
  if (e != cudaSuccess) {
    std::fprintf(stderr, "%s\n", cudaGetErrorString(e));
    return 1;
  }
  const char *name[kCounts] = {"silu", "silu_alone", "dsilu", "quotient", "reciprocal"};
  for (int k = 0; k < kCounts; k++)
    std::printf("%s %llu %llu %llu\n", name[k], c[k].seen, c[k].differ, c[k].ulps);
  return 0;
}
