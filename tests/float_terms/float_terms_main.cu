// The float nodal dS's quotient and logarithm (common.cuh) against CUDA's
// correctly rounded division and the scalar logarithm, on the device.
//   quot LO COUNT [LO COUNT ..]   quot_rn(x, p) == __fdiv_rn(x, p) for every mantissa x and
//                   the mantissas p = LO .. LO + COUNT - 1 (of 2^23 each; the
//                   quotient's rounding does not depend on the exponents)
//   range SEED      the same for random counts x < 2^24 and products of two
//                   degrees p < 2^48, and ref_term_nz against ref_term there
//   log             ref_logf_quot(x) == ref_logf(x) for every float x in
//                   [2^-48, 2^24)
// Prints the number of differences.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "common.cuh"

using namespace usap;

namespace {

__global__ void k_quot(unsigned lo, unsigned long long* bad) {
  const float p = __uint_as_float(0x3f800000u | (lo + blockIdx.y));
  unsigned n = 0;
  for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 23); m += gridDim.x * blockDim.x) {
    const float x = __uint_as_float(0x3f800000u | m);
    n += __float_as_uint(quot_rn(x, p)) != __float_as_uint(__fdiv_rn(x, p));
  }
  if (n) atomicAdd(bad, static_cast<unsigned long long>(n));
}

__global__ void k_range(uint64_t seed, unsigned long long* bad) {
  ref_tab_fill();
  __syncthreads();
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned n = 0;
  for (unsigned i = 0; i < 256; i++) {
    const Draws d = philox(t, i, 0, 0, seed);
    // degrees of any size below 2^24; the count is at most the smaller one
    const int da = 1 + static_cast<int>(draw_below(d.x0, 1 << (1 + i % 24)) % ((1 << 24) - 1));
    const int db = 1 + static_cast<int>(draw_below(d.x1, 1 << (1 + (i / 8) % 24)) % ((1 << 24) - 1));
    const int x = 1 + static_cast<int>(draw_below(d.x2, da < db ? da : db));
    const float xf = __int2float_rn(x), pf = __ll2float_rn(static_cast<long long>(da) * db);
    n += __float_as_uint(quot_rn(xf, pf)) != __float_as_uint(__fdiv_rn(xf, pf));
    n += __float_as_uint(ref_term_nz(x, ref_factor(da), ref_factor(db))) !=
         __float_as_uint(ref_term(x, static_cast<long long>(da) * db));
    n += ref_term_nz(0, ref_factor(da), ref_factor(i & 1 ? 0 : db)) != 0.0f;
  }
  if (n) atomicAdd(bad, static_cast<unsigned long long>(n));
}

__global__ void k_log(unsigned long long* bad) {
  ref_tab_fill();
  __syncthreads();
  const unsigned first = (127u - 48u) << 23, last = (127u + 24u) << 23;
  unsigned n = 0;
  for (unsigned u = first + blockIdx.x * blockDim.x + threadIdx.x; u < last; u += gridDim.x * blockDim.x) {
    const float x = __uint_as_float(u);
    n += __float_as_uint(ref_logf_quot(x)) != __float_as_uint(ref_logf(x));
  }
  if (n) atomicAdd(bad, static_cast<unsigned long long>(n));
}

}  // namespace

int main(int argc, char** argv) {
  unsigned long long *bad = nullptr, h = 0;
  if (argc < 2 || cudaMalloc(&bad, sizeof(h)) != cudaSuccess) return 2;
  cudaMemset(bad, 0, sizeof(h));
  if (!std::strcmp(argv[1], "quot") && argc % 2 == 0) {
    for (int i = 2; i < argc; i += 2) {
      const unsigned lo = std::strtoul(argv[i], nullptr, 10), count = std::strtoul(argv[i + 1], nullptr, 10);
      if (lo >= 1u << 23 || count > (1u << 23) - lo) return 2;
      for (unsigned p = lo; p < lo + count; p += 4096) {   // 30 ms a launch
        const unsigned k = lo + count - p < 4096 ? lo + count - p : 4096;
        k_quot<<<dim3(32, k), 256>>>(p, bad);
      }
    }
  } else if (!std::strcmp(argv[1], "range") && argc == 3) {
    k_range<<<148 * 8, 256>>>(std::strtoull(argv[2], nullptr, 10), bad);
  } else if (!std::strcmp(argv[1], "log")) {
    k_log<<<148 * 8, 256>>>(bad);
  } else {
    return 2;
  }
  if (cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  std::printf("%llu\n", h);
  cudaFree(bad);
  return 0;
}
