// Partition scores on the device (bf::evaluate, include/evaluate.hpp:18-266):
// the contingency table, its row and column sums, the exact pair counts and
// the fixed-point information sums of eval_common.h, from device arrays of
// truth and given labels.  Only the sums (and, for the matching accuracy,
// the table when both sides have at most 2048 blocks) come back to the host,
// which forms the scores exactly as the host version does.  The device's part
// is a few microseconds: a call is bound by its launches, copies and the
// host's matching, so small tables take one host round trip, and the log
// table is the one the device keeps for its graphs (50000 vertices: 264 us with
// two round trips and the table copied by every call, 202 us now).
#include <algorithm>
#include <climits>
#include <cstddef>
#include <vector>

#include "eval_common.h"
#include "job.h"

namespace usap {

namespace {

constexpr int kThreads = 256;
constexpr int64_t kMaxCells = int64_t(1) << 26;   // dense table limit (256 MiB of counts)

constexpr int kCountThreads = 1024;
// The counts contend for few addresses (44 x 57 cells and 101 sums for 50000
// vertices), so up to kSmallCells cells each CTA counts kCountItems vertices
// in shared memory, takes the row and column sums from its cells and adds
// what is not zero.  Above, the table is wide enough for global atomics.
constexpr int kSmallCells = 8192;
constexpr int kCountItems = 4 * kCountThreads;
// b1 * b2 <= kSmallCells, so b1 + b2 <= kSmallCells + 1
constexpr size_t kSmallSmem = sizeof(unsigned) * (2 * kSmallCells + 1);

struct LabelInfo {
  int b1, b2, bad;            // blocks (largest label + 1) of truth and given
  unsigned long long known;   // vertices with truth >= 0
};

// header of a call's device buffer, and of what comes back to the host
struct EvalHead {
  LabelInfo info;
  EvalSums sums;
};

// a table the small path counts
__host__ __device__ __forceinline__ bool eval_small(const LabelInfo& i) {
  return !i.bad && i.b1 > 0 && i.b2 > 0 && i.known >= 2 && static_cast<long long>(i.b1) * i.b2 <= kSmallCells;
}

__global__ void __launch_bounds__(kCountThreads) k_eval_labels(int64_t n, const int32_t* __restrict__ truth,
                                                               const int32_t* __restrict__ given, LabelInfo* info) {
  __shared__ int s_b1, s_b2, s_bad;
  __shared__ unsigned long long s_known;
  if (threadIdx.x == 0) {
    s_b1 = s_b2 = s_bad = 0;
    s_known = 0;
  }
  __syncthreads();
  int mt = -1, mg = -1, bad = 0;
  unsigned known = 0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int t = truth[i], g = given[i];
    if (g < 0 || t < -1) bad = 1;
    mt = max(mt, t);
    mg = max(mg, g);
    known += t >= 0;
  }
  mt = __reduce_max_sync(0xffffffffu, mt);
  mg = __reduce_max_sync(0xffffffffu, mg);
  bad = __any_sync(0xffffffffu, bad);
  known = __reduce_add_sync(0xffffffffu, known);
  if ((threadIdx.x & 31) == 0) {
    // a label of 2^31 - 1 has no count of blocks
    if (mt == INT_MAX || mg == INT_MAX) bad |= 2;
    atomicMax(&s_b1, mt == INT_MAX ? 0 : mt + 1);
    atomicMax(&s_b2, mg == INT_MAX ? 0 : mg + 1);
    if (bad) atomicOr(&s_bad, bad);
    atomicAdd(&s_known, static_cast<unsigned long long>(known));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&info->b1, s_b1);
    atomicMax(&info->b2, s_b2);
    if (s_bad) atomicOr(&info->bad, s_bad);
    if (s_known) atomicAdd(&info->known, s_known);
  }
}
// small path: counts of the table (row-major b1 x b2) and its row and column
// sums; sizes are read from what k_eval_labels found, so that nothing waits
// for the host in between
__global__ void __launch_bounds__(kCountThreads) k_eval_count_small(int64_t n, const int32_t* __restrict__ truth,
                                                                    const int32_t* __restrict__ given,
                                                                    const LabelInfo* __restrict__ info,
                                                                    unsigned* __restrict__ table,
                                                                    unsigned* __restrict__ rows,
                                                                    unsigned* __restrict__ cols) {
  extern __shared__ unsigned s_tab[];
  const LabelInfo li = *info;
  if (!eval_small(li)) return;
  const int b1 = li.b1, b2 = li.b2, cells = b1 * b2;
  unsigned* s_rows = s_tab + cells;
  unsigned* s_cols = s_rows + b1;
  for (int i = threadIdx.x; i < cells + b1 + b2; i += kCountThreads) s_tab[i] = 0;
  __syncthreads();
  for (int64_t i0 = blockIdx.x * static_cast<int64_t>(kCountItems) + threadIdx.x; i0 < n;
       i0 += gridDim.x * static_cast<int64_t>(kCountItems)) {
    int t[4], g[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int64_t i = i0 + k * kCountThreads;
      t[k] = i < n ? __ldg(truth + i) : -1;
      g[k] = i < n ? __ldg(given + i) : 0;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (t[k] >= 0) atomicAdd(s_tab + t[k] * b2 + g[k], 1u);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < cells; c += kCountThreads) {
    const unsigned x = s_tab[c];
    if (!x) continue;
    const int i = c / b2;
    atomicAdd(table + c, x);
    atomicAdd(s_rows + i, x);
    atomicAdd(s_cols + (c - i * b2), x);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < b1; i += kCountThreads)
    if (s_rows[i]) atomicAdd(rows + i, s_rows[i]);
  for (int j = threadIdx.x; j < b2; j += kCountThreads)
    if (s_cols[j]) atomicAdd(cols + j, s_cols[j]);
}

// the same by global atomics
__global__ void k_eval_count(int64_t n, const int32_t* __restrict__ truth, const int32_t* __restrict__ given, int b2,
                             unsigned* __restrict__ table, unsigned* __restrict__ rows, unsigned* __restrict__ cols) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int t = truth[i];
    if (t < 0) continue;
    const int g = given[i];
    atomicAdd(table + static_cast<int64_t>(t) * b2 + g, 1u);
    atomicAdd(rows + t, 1u);
    atomicAdd(cols + g, 1u);
  }
}

// the exact sums over cells (items [0, cells)), rows and columns of the
// table that `info` describes
__global__ void __launch_bounds__(kThreads) k_eval_sums(const LabelInfo* __restrict__ info, bool small,
                                                        const unsigned* __restrict__ table,
                                                        const unsigned* __restrict__ rows,
                                                        const unsigned* __restrict__ cols,
                                                        const double* __restrict__ L, EvalSums* out) {
  const LabelInfo li = *info;
  if (small && !eval_small(li)) return;
  const int b1 = li.b1, b2 = li.b2;
  const long long N = static_cast<long long>(li.known);
  const long long cells = static_cast<long long>(b1) * b2;
  const long long total = cells + b1 + b2;
  if (blockIdx.x * static_cast<long long>(kThreads) >= total) return;
  __shared__ unsigned long long sh[13];
  if (threadIdx.x < 13) sh[threadIdx.x] = 0;
  __syncthreads();
  const double dN = static_cast<double>(N), LN = __ldg(L + N);
  long long sq = 0, same = 0, hgt = 0, htg = 0, mi = 0, sr = 0, s1 = 0, sc = 0, s2 = 0, h1 = 0, h2 = 0, nb1 = 0,
            nb2 = 0;
  for (long long x = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; x < total;
       x += static_cast<long long>(gridDim.x) * blockDim.x) {
    if (x < cells) {
      const long long c = table[x];
      if (!c) continue;
      const int i = static_cast<int>(x / b2), j = static_cast<int>(x - static_cast<long long>(i) * b2);
      const long long r = rows[i], s = cols[j];
      const double Lc = __ldg(L + c), Lr = __ldg(L + r), Ls = __ldg(L + s);
      sq += c * c;
      same += c * (c - 1) / 2;
      hgt += ev_term(c, dN, Lc, Lr);
      htg += ev_term(c, dN, Lc, Ls);
      mi += ev_mi_term(c, dN, Lc, LN, Lr, Ls);
    } else if (x < cells + b1) {
      const long long r = rows[x - cells];
      if (!r) continue;
      sr += r * r;
      s1 += r * (r - 1) / 2;
      nb1++;
      h1 += ev_term(r, dN, __ldg(L + r), LN);
    } else {
      const long long s = cols[x - cells - b1];
      if (!s) continue;
      sc += s * s;
      s2 += s * (s - 1) / 2;
      nb2++;
      h2 += ev_term(s, dN, __ldg(L + s), LN);
    }
  }
  const long long vals[13] = {sq, same, hgt, htg, mi, sr, s1, sc, s2, h1, h2, nb1, nb2};
#pragma unroll
  for (int k = 0; k < 13; k++) {
    const long long t = warp_sum_ll(vals[k]);
    if ((threadIdx.x & 31) == 0 && t) atomicAdd(sh + k, static_cast<unsigned long long>(t));
  }
  __syncthreads();
  if (threadIdx.x < 13 && sh[threadIdx.x]) {
    int64_t* const dst[13] = {&out->sq, &out->same, &out->h_gt_q, &out->h_tg_q, &out->mi_q, &out->sr, &out->s1,
                              &out->sc, &out->s2, &out->h_truth_q, &out->h_given_q, &out->nb_truth, &out->nb_given};
    atomicAdd(reinterpret_cast<unsigned long long*>(dst[threadIdx.x]), sh[threadIdx.x]);
  }
}

int grid_for(int64_t items) {
  int64_t b = (items + kThreads - 1) / kThreads;
  if (b > 148 * 8) b = 148 * 8;
  return static_cast<int>(b < 1 ? 1 : b);
}

int count_grid(int64_t n) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + kCountItems - 1) / kCountItems, 148 * 2)));
}

// Vertices below which a call's scores are enqueued at once and read the
// device's shared log table, which they grow up to that many entries (64 MiB on
// the device).  Above, a call learns first how many vertices count, and brings
// a larger table than that in memory of its own: the device passes take
// milliseconds there, and the shared table lives as long as the process.
constexpr int64_t kSharedLogs = int64_t(1) << 22;

}  // namespace

void evaluate_device(const int32_t* truth, const int32_t* given, int64_t n, int device, usap_scores* s) {
  if (n < 2) throw Error(USAP_ERR_INVALID, "need at least two labelled vertices");
  USAP_CUDA(cudaSetDevice(device));
  pool_configure(device);
  cudaStream_t st = nullptr;
  USAP_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  struct Cleanup {
    cudaStream_t st;
    std::vector<void*> bufs;
    ~Cleanup() {
      for (void* p : bufs) cudaFreeAsync(p, st);
      cudaStreamSynchronize(st);
      cudaStreamDestroy(st);
    }
  } cl{st, {}};
  auto alloc = [&](size_t bytes) {
    void* p = dev_alloc(bytes, st);
    cl.bufs.push_back(p);
    return p;
  };
  // small tables: labels, counts and sums are enqueued together, and the
  // header and the table come back in one copy; a larger table (known only
  // then) takes the general kernels and a second round trip
  struct Back {
    EvalHead head;
    unsigned table[kSmallCells];
  };
  unsigned char* base = static_cast<unsigned char*>(alloc(sizeof(Back) + sizeof(unsigned) * 2 * kSmallCells));
  EvalHead* head = reinterpret_cast<EvalHead*>(base);
  unsigned* table = reinterpret_cast<unsigned*>(base + offsetof(Back, table));
  unsigned* rows = table + kSmallCells;
  unsigned* cols = rows + kSmallCells;
  USAP_CUDA(cudaMemsetAsync(base, 0, sizeof(Back) + sizeof(unsigned) * 2 * kSmallCells, st));
  k_eval_labels<<<count_grid(n), kCountThreads, 0, st>>>(n, truth, given, &head->info);
  USAP_LAUNCHED();
  std::shared_ptr<const DeviceLogTable> logs;
  std::shared_ptr<const std::vector<double>> Lp;
  auto logs_to = [&](int64_t k) -> const double* {
    if (k < kSharedLogs) {
      logs = device_log_table(device, k, nullptr, kSharedLogs);
      return logs->L;
    }
    Lp = log_table(k);
    double* up = static_cast<double*>(alloc(sizeof(double) * (k + 1)));
    USAP_CUDA(cudaMemcpyAsync(up, Lp->data(), sizeof(double) * (k + 1), cudaMemcpyHostToDevice, st));
    return up;
  };
  const double* L = nullptr;
  Back back;
  auto small_scores = [&](int64_t k) {   // log k of every count needed
    USAP_CUDA(cudaFuncSetAttribute(k_eval_count_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(kSmallSmem)));
    k_eval_count_small<<<count_grid(n), kCountThreads, kSmallSmem, st>>>(n, truth, given, &head->info, table, rows,
                                                                         cols);
    USAP_LAUNCHED();
    L = logs_to(k);
    k_eval_sums<<<grid_for(2 * kSmallCells + 1), kThreads, 0, st>>>(&head->info, true, table, rows, cols, L,
                                                                    &head->sums);
    USAP_LAUNCHED();
    USAP_CUDA(cudaMemcpyAsync(&back, base, sizeof(back), cudaMemcpyDeviceToHost, st));
    USAP_CUDA(cudaStreamSynchronize(st));
  };
  const bool at_once = n < kSharedLogs;
  if (at_once) {
    small_scores(n);
  } else {
    USAP_CUDA(cudaMemcpyAsync(&back.head, head, sizeof(EvalHead), cudaMemcpyDeviceToHost, st));
    USAP_CUDA(cudaStreamSynchronize(st));
  }
  const LabelInfo li = back.head.info;
  if (li.bad & 1) throw Error(USAP_ERR_INVALID, "given labels must be >= 0 and truth labels >= -1");
  const int b1 = li.b1, b2 = li.b2;
  const int64_t N = static_cast<int64_t>(li.known);
  if (li.bad || b1 <= 0 || b2 <= 0 || N < 2)
    throw Error(USAP_ERR_INVALID, "need at least two vertices with known truth");
  const int64_t cells = static_cast<int64_t>(b1) * b2;
  if (cells > kMaxCells) throw Error(USAP_ERR_LIMIT, "contingency table above 2^26 cells");
  const int m = b1 > b2 ? b1 : b2;
  if (!at_once) {
    if (eval_small(li)) small_scores(N);
    else L = logs_to(N);
  }
  EvalSums e = back.head.sums;
  std::vector<unsigned> big;
  const unsigned* t = back.table;
  if (!eval_small(li)) {
    table = static_cast<unsigned*>(alloc(sizeof(unsigned) * (cells + b1 + b2)));
    rows = table + cells;
    cols = rows + b1;
    USAP_CUDA(cudaMemsetAsync(table, 0, sizeof(unsigned) * (cells + b1 + b2), st));
    k_eval_count<<<grid_for(n), kThreads, 0, st>>>(n, truth, given, b2, table, rows, cols);
    USAP_LAUNCHED();
    k_eval_sums<<<grid_for(cells + b1 + b2), kThreads, 0, st>>>(&head->info, false, table, rows, cols, L, &head->sums);
    USAP_LAUNCHED();
    USAP_CUDA(cudaMemcpyAsync(&e, &head->sums, sizeof(e), cudaMemcpyDeviceToHost, st));
    if (m <= 2048) {
      big.resize(static_cast<size_t>(cells));
      USAP_CUDA(cudaMemcpyAsync(big.data(), table, sizeof(unsigned) * cells, cudaMemcpyDeviceToHost, st));
      t = big.data();
    }
    USAP_CUDA(cudaStreamSynchronize(st));
  }
  e.N = N;
  scores_from_sums(e, s);
  if (m <= 2048) {
    std::vector<int64_t> t64(t, t + cells);
    s->accuracy = matching_accuracy(t64.data(), b1, b2, N);
  } else {
    s->accuracy = std::nan("");
  }
}

}  // namespace usap
