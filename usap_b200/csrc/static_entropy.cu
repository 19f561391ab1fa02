// usap_entropy_static: the description length of a partition computed in a
// fixed, file-scope device scratch array, with no allocation of any kind.
//
// Some callers cannot allocate when they need the score: a host framework
// whose own allocator has already reserved the device memory it may use
// (a cudaMalloc of ours would fail or push it past its budget), and a
// latency-sensitive loop that cannot take the device-wide synchronisation
// that cudaMalloc/cudaFree imply.  For them this entry point reads
// device-resident edges and block ids and writes the Q32 value to a device
// pointer, in the caller's stream order, using only the array below.
//
// The score is the one usap_op_entropy returns (model term of
// _compute_overall_entropy, graph_parallel.hpp:1314-1316, minus the data term
// summed over the dense block matrix, :1297-1312), term for term: the same
// glibc log table, the same rounding of each term and an order-independent
// int64 sum, so the two agree exactly.
#include <cstdint>
#include <cmath>
#include <climits>
#include <mutex>

#include "../../include/usap.h"
#include "common.cuh"
#include "engine.h"
#include "job.h"

namespace usap {
namespace {

constexpr int kStaticMaxBlocks = USAP_STATIC_MAX_BLOCKS;
constexpr int64_t kStaticMaxWeight = USAP_STATIC_MAX_WEIGHT;
constexpr int kStaticMaxDevices = 64;
constexpr int kThreads = 256;

constexpr size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

// regions of the scratch array (what a call clears lies together: the
// counters and M, and before them the degrees)
constexpr size_t kLogOff = 0;                                                // L[0..W]
constexpr size_t kDoutOff = align256(kLogOff + sizeof(double) * (kStaticMaxWeight + 1));
constexpr size_t kDinOff = align256(kDoutOff + sizeof(int32_t) * kStaticMaxBlocks);
constexpr size_t kCtrOff = align256(kDinOff + sizeof(int32_t) * kStaticMaxBlocks);
constexpr size_t kMOff = kCtrOff + 256;

struct StaticCounters {
  unsigned long long acc;    // data term, Q32, two's complement
  unsigned long long wsum;   // total edge weight seen
  int bad;                   // an input failed a device-side check
  unsigned done;             // CTAs of the last kernel that are through
};
static_assert(sizeof(StaticCounters) <= 256, "counters outgrow their region");

constexpr size_t kScratchBytes = align256(kMOff + sizeof(int32_t) * kStaticMaxBlocks * kStaticMaxBlocks);

// One array per device, shared by every call on that device.  The log table
// at its head is written once at set-up; the rest is cleared by each call.
static __device__ __align__(256) unsigned char g_static_scratch[kScratchBytes];

struct StaticView {
  const double* L;
  int32_t* M;        // B x B, row stride B
  int32_t* dout;
  int32_t* din;
  StaticCounters* ctr;
};

StaticView view_of(unsigned char* base) {
  return StaticView{reinterpret_cast<const double*>(base + kLogOff),
                    reinterpret_cast<int32_t*>(base + kMOff),
                    reinterpret_cast<int32_t*>(base + kDoutOff),
                    reinterpret_cast<int32_t*>(base + kDinOff),
                    reinterpret_cast<StaticCounters*>(base + kCtrOff)};
}

// The build is bound by atomics on few addresses: all edges of a partition of
// 19 blocks add to 361 cells, most of them to the 19 diagonal ones, and to 38
// degrees.  So each CTA counts its kBuildEdges edges in shared memory and adds
// only what it found: up to kSmallBlocks blocks the whole matrix (48 KB of
// shared memory hold 104 x 104), whose row and column sums are the degrees;
// above, the degrees alone (the cells are then at least 11 k addresses).
// Four edges per thread keep their loads in flight together, and a CTA's
// flush stands for four times the edges.  79000 edges, 19 blocks: 50 us with
// an atomic per edge and address in four launches, 11 us in a memset and one
// launch.
constexpr int kBuildThreads = 1024;
constexpr int kEdgesPerThread = 4;
constexpr int kBuildEdges = kBuildThreads * kEdgesPerThread;
constexpr int kSmallBlocks = 104;
constexpr int kEntropyCtas = 148 * 4;

// adds the edges of this CTA: ids outside [0, n) or [0, B) and negative
// weights are recorded, not followed
template <class AddFn>
__device__ __forceinline__ void add_edges(const StaticView& v, const int32_t* __restrict__ src,
                                          const int32_t* __restrict__ dst, const int32_t* __restrict__ w, int64_t e,
                                          int32_t n, const int32_t* __restrict__ part, int B, AddFn add) {
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * kBuildEdges + threadIdx.x;
  int32_t a[kEdgesPerThread], b[kEdgesPerThread], x[kEdgesPerThread], r[kEdgesPerThread], s[kEdgesPerThread];
#pragma unroll
  for (int k = 0; k < kEdgesPerThread; k++) {
    const int64_t i = i0 + k * kBuildThreads;
    const bool in = i < e;
    a[k] = in ? __ldg(src + i) : 0;
    b[k] = in ? __ldg(dst + i) : 0;
    x[k] = !in ? 0 : w ? __ldg(w + i) : 1;
  }
  bool bad = false;
#pragma unroll
  for (int k = 0; k < kEdgesPerThread; k++) {
    const bool in = i0 + k * kBuildThreads < e;
    const bool ok = in && a[k] >= 0 && a[k] < n && b[k] >= 0 && b[k] < n && x[k] >= 0;
    bad |= in && !ok;
    r[k] = ok ? __ldg(part + a[k]) : -1;
    s[k] = ok ? __ldg(part + b[k]) : -1;
    if (ok && (r[k] < 0 || r[k] >= B || s[k] < 0 || s[k] >= B)) {
      bad = true;
      r[k] = -1;
    }
  }
  long long wt = 0;
#pragma unroll
  for (int k = 0; k < kEdgesPerThread; k++)
    if (r[k] >= 0 && x[k] > 0) {
      wt += x[k];
      add(r[k], s[k], x[k]);
    }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&v.ctr->bad, 1);
  wt = warp_sum_ll(wt);
  if ((threadIdx.x & 31) == 0 && wt) atomicAdd(&v.ctr->wsum, static_cast<unsigned long long>(wt));
}

// one cell's part of the data term; a count or degree outside the log table
// is recorded instead of read
__device__ __forceinline__ long long cell_term(const double* L, int m, int di, int dr, bool* bad) {
  if (m < 0 || m > kStaticMaxWeight || di <= 0 || di > kStaticMaxWeight || dr <= 0 || dr > kStaticMaxWeight) {
    *bad = true;
    return 0;
  }
  return q32(g_term(L, m, di, dr));
}

// model term (saturated on the host) plus data term, saturated
__device__ __forceinline__ void write_result(bool bad, long long model_q, unsigned long long acc, int64_t* S_q) {
  const long long b = -static_cast<long long>(acc);
  long long r = static_cast<long long>(static_cast<unsigned long long>(model_q) + static_cast<unsigned long long>(b));
  if ((model_q > 0 && b > 0 && r < 0) || (model_q < 0 && b < 0 && r >= 0)) r = model_q > 0 ? LLONG_MAX : LLONG_MIN;
  *S_q = bad ? static_cast<int64_t>(LLONG_MIN) : r;
}

// true in every thread of the CTA that arrives last; what the others wrote
// before is then visible (to loads that bypass L1)
__device__ __forceinline__ bool last_cta(StaticCounters* ctr, int* s_last) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *s_last = atomicAdd(&ctr->done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!*s_last) return false;
  __threadfence();
  return true;
}

__device__ __forceinline__ bool inputs_bad(const StaticCounters* ctr) {
  return __ldcg(&ctr->bad) || __ldcg(&ctr->wsum) > static_cast<unsigned long long>(kStaticMaxWeight);
}

// B <= kSmallBlocks: counts, and in the last CTA the data term and the result
__global__ void __launch_bounds__(kBuildThreads) k_static_small(StaticView v, const int32_t* __restrict__ src,
                                                                const int32_t* __restrict__ dst,
                                                                const int32_t* __restrict__ w, int64_t e, int32_t n,
                                                                const int32_t* __restrict__ part, int B,
                                                                long long model_q, int64_t* S_q) {
  __shared__ int32_t s_M[kSmallBlocks * kSmallBlocks];
  __shared__ int32_t s_out[kSmallBlocks], s_in[kSmallBlocks];
  __shared__ unsigned long long s_acc;
  __shared__ int s_last, s_bad;
  const int cells = B * B;
  for (int c = threadIdx.x; c < cells; c += kBuildThreads) s_M[c] = 0;
  __syncthreads();
  add_edges(v, src, dst, w, e, n, part, B, [&](int r, int s, int x) { atomicAdd(s_M + r * B + s, x); });
  __syncthreads();
  for (int c = threadIdx.x; c < cells; c += kBuildThreads)
    if (s_M[c]) atomicAdd(v.M + c, s_M[c]);
  if (!last_cta(v.ctr, &s_last)) return;
  if (threadIdx.x < B) s_out[threadIdx.x] = s_in[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    s_acc = 0;
    s_bad = inputs_bad(v.ctr);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < cells; c += kBuildThreads) {
    const int m = __ldcg(v.M + c);
    s_M[c] = m;
    if (m) {
      const int i = c / B;
      atomicAdd(s_out + i, m);
      atomicAdd(s_in + (c - i * B), m);
    }
  }
  __syncthreads();
  long long sum = 0;
  bool bad = false;
  for (int c = threadIdx.x; c < cells; c += kBuildThreads) {
    const int m = s_M[c], i = c / B;
    if (m) sum += cell_term(v.L, m, s_in[c - i * B], s_out[i], &bad);
  }
  sum = warp_sum_ll(sum);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&s_acc, static_cast<unsigned long long>(sum));
  if (bad) s_bad = 1;
  __syncthreads();
  if (threadIdx.x == 0) write_result(s_bad != 0, model_q, s_acc, S_q);
}

// B > kSmallBlocks: the cells straight to global memory, the degrees by way of shared memory
__global__ void __launch_bounds__(kBuildThreads) k_static_build(StaticView v, const int32_t* __restrict__ src,
                                                                const int32_t* __restrict__ dst,
                                                                const int32_t* __restrict__ w, int64_t e, int32_t n,
                                                                const int32_t* __restrict__ part, int B) {
  __shared__ int32_t s_out[kStaticMaxBlocks], s_in[kStaticMaxBlocks];
  for (int c = threadIdx.x; c < B; c += kBuildThreads) s_out[c] = s_in[c] = 0;
  __syncthreads();
  add_edges(v, src, dst, w, e, n, part, B, [&](int r, int s, int x) {
    atomicAdd(v.M + r * B + s, x);
    atomicAdd(s_out + r, x);
    atomicAdd(s_in + s, x);
  });
  __syncthreads();
  for (int c = threadIdx.x; c < B; c += kBuildThreads) {
    if (s_out[c]) atomicAdd(v.dout + c, s_out[c]);
    if (s_in[c]) atomicAdd(v.din + c, s_in[c]);
  }
}

// data term over the B x B cells; the last CTA writes the result
__global__ void __launch_bounds__(kThreads) k_static_entropy(StaticView v, int B, long long model_q, int64_t* S_q) {
  __shared__ unsigned long long s_acc;
  __shared__ int s_last;
  if (threadIdx.x == 0) s_acc = 0;
  __syncthreads();
  long long sum = 0;
  bool bad = false;
  const int cells = B * B, stride = gridDim.x * kThreads;
  for (int c = blockIdx.x * kThreads + threadIdx.x; c < cells; c += stride) {
    const int m = v.M[c];
    if (!m) continue;
    const int i = c / B;
    sum += cell_term(v.L, m, v.din[c - i * B], v.dout[i], &bad);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&v.ctr->bad, 1);
  sum = warp_sum_ll(sum);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&s_acc, static_cast<unsigned long long>(sum));
  __syncthreads();
  if (threadIdx.x == 0 && s_acc) atomicAdd(&v.ctr->acc, s_acc);
  if (!last_cta(v.ctr, &s_last)) return;
  if (threadIdx.x == 0) write_result(inputs_bad(v.ctr), model_q, __ldcg(&v.ctr->acc), S_q);
}

std::mutex g_setup_mu;
unsigned char* g_scratch_ptr[kStaticMaxDevices] = {};

// Once per device, with that device current: the address of the array and
// the log table in its first region.  Copies go through a stack buffer.
unsigned char* scratch_for(int dev) {
  std::lock_guard<std::mutex> lk(g_setup_mu);
  if (g_scratch_ptr[dev]) return g_scratch_ptr[dev];
  void* ptr = nullptr;
  USAP_CUDA(cudaGetSymbolAddress(&ptr, g_static_scratch));
  unsigned char* base = static_cast<unsigned char*>(ptr);
  constexpr int64_t kChunk = 4096;
  double buf[kChunk];
  for (int64_t k0 = 0; k0 <= kStaticMaxWeight; k0 += kChunk) {
    const int64_t k1 = std::min<int64_t>(kStaticMaxWeight + 1, k0 + kChunk);
    for (int64_t k = k0; k < k1; k++) buf[k - k0] = k == 0 ? -INFINITY : std::log(static_cast<double>(k));
    USAP_CUDA(cudaMemcpy(base + kLogOff + sizeof(double) * k0, buf, sizeof(double) * (k1 - k0),
                         cudaMemcpyHostToDevice));
  }
  // a copy from pageable memory may return before it lands; the first call's
  // kernels can run on a non-blocking stream, so wait for the table here
  USAP_CUDA(cudaDeviceSynchronize());
  g_scratch_ptr[dev] = base;
  return base;
}

void entropy_static(const int32_t* src, const int32_t* dst, const int32_t* weight, int64_t e,
                    int32_t n, const int32_t* part, int32_t B, int64_t* S_q, cudaStream_t st) {
  if (!src || !dst || !part || !S_q) throw Error(USAP_ERR_INVALID, "null device pointer");
  if (n < 1 || e < 1) throw Error(USAP_ERR_INVALID, "need n >= 1 and e >= 1");
  if (B < 1) throw Error(USAP_ERR_INVALID, "need B >= 1");
  if (B > kStaticMaxBlocks)
    throw Error(USAP_ERR_LIMIT, "B = " + std::to_string(B) + " exceeds the static scratch limit of " +
                                    std::to_string(kStaticMaxBlocks) + " blocks");
  if (e > kStaticMaxWeight)
    throw Error(USAP_ERR_LIMIT, "e = " + std::to_string(e) + " exceeds the static scratch limit of " +
                                    std::to_string(kStaticMaxWeight) + " edges");
  int dev = -1;
  USAP_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kStaticMaxDevices) throw Error(USAP_ERR_INVALID, "device index out of range");
  int major = 0;
  USAP_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  if (major != 10) throw Error(USAP_ERR_NO_DEVICE, "current device is not sm_100 class");
  unsigned char* base = scratch_for(dev);
  const StaticView v = view_of(base);
  const long long model_q = q32_host(model_S(n, e, B));
  const int cells = B * B;
  const unsigned ctas = static_cast<unsigned>((e + kBuildEdges - 1) / kBuildEdges);
  const bool small = B <= kSmallBlocks;
  const size_t clear = small ? kCtrOff : kDoutOff;
  USAP_CUDA(cudaMemsetAsync(base + clear, 0, kMOff + sizeof(int32_t) * cells - clear, st));
  if (small) {
    k_static_small<<<ctas, kBuildThreads, 0, st>>>(v, src, dst, weight, e, n, part, B, model_q, S_q);
    USAP_LAUNCHED();
    return;
  }
  k_static_build<<<ctas, kBuildThreads, 0, st>>>(v, src, dst, weight, e, n, part, B);
  USAP_LAUNCHED();
  k_static_entropy<<<std::min((cells + kThreads - 1) / kThreads, kEntropyCtas), kThreads, 0, st>>>(v, B, model_q, S_q);
  USAP_LAUNCHED();
}

}  // namespace
}  // namespace usap

extern "C" usap_status usap_entropy_static(const int32_t* src, const int32_t* dst,
                                           const int32_t* weight, int64_t e, int32_t n,
                                           const int32_t* part, int32_t B, int64_t* S_q,
                                           void* stream) {
  return usap::call_guarded([&] {
    usap::entropy_static(src, dst, weight, e, n, part, B, S_q, static_cast<cudaStream_t>(stream));
  });
}
