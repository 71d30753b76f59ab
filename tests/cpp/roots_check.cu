// roots.cuh against the correctly rounded functions, for every float of its ranges:
// prints the number of floats compared and of those that differ, by function.
#include <cstdio>
#include <cstring>

#include "../../mosaic-art-rust_gb300/csrc/roots.cuh"

namespace {
using namespace mg;
using Count = unsigned long long;

__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

// Every float of [lo, hi] (as bits) through each function; the pairs' other half
// takes the range from its other end.
__global__ void compare(int function, unsigned lo, unsigned hi, Count* differing) {
  Count bad = 0;
  for (Count i = (Count)lo + blockIdx.x * blockDim.x + threadIdx.x; i <= hi; i += (Count)gridDim.x * blockDim.x) {
    const float a = __uint_as_float((unsigned)i), b = __uint_as_float((unsigned)(lo + (hi - i)));
    if (function == 0) {
      bad += !same(rcp_in_range(a), __frcp_rn(a));
    } else if (function == 1) {
      const float2 r = rcp2_in_range(make_float2(a, b));
      bad += !same(r.x, __frcp_rn(a));
      bad += !same(r.y, __frcp_rn(b));
    } else if (function == 2) {
      bad += !same(weight_of_sq(a), __frcp_rn(__fadd_rn(__fsqrt_rn(a), 1.0f)));
    } else {
      const float2 r = weight_of_sq2(a, b);
      bad += !same(r.x, __frcp_rn(__fadd_rn(__fsqrt_rn(a), 1.0f)));
      bad += !same(r.y, __frcp_rn(__fadd_rn(__fsqrt_rn(b), 1.0f)));
    }
  }
  if (bad) atomicAdd(differing, bad);
}

unsigned bits(float f) {
  unsigned u;
  memcpy(&u, &f, 4);
  return u;
}
}  // namespace

int main() {
  const struct {
    const char* name;
    int function;
    unsigned lo, hi;
  } checks[] = {{"rcp_in_range", 0, bits(1.0f), bits(1e30f)},
                {"rcp2_in_range", 1, (127u - 67u) << 23, bits(4.0f) - 1u},
                {"weight_of_sq", 2, 0u, 0x7FFFFFFFu},  // zero, subnormals, infinity and NaN, too
                {"weight_of_sq2", 3, 0u, 0x7FFFFFFFu}};
  Count* d = nullptr;
  int failed = 0;
  if (cudaMalloc(&d, sizeof(Count)) != cudaSuccess) return 2;
  for (const auto& c : checks) {
    Count bad = 0;
    cudaMemset(d, 0, sizeof(Count));
    compare<<<1216, 256>>>(c.function, c.lo, c.hi, d);
    if (cudaMemcpy(&bad, d, sizeof(Count), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%s %llu floats, differing %llu\n", c.name, (Count)c.hi - c.lo + 1, bad);
    failed |= bad != 0;
  }
  return failed;
}
