// Batched nodal update.
//
// Reference: the nodal_move task (graph_parallel.hpp:406-431) runs
// _propose_new_partition_nodal (:990-1222) for every vertex of a contiguous
// batch against the batch-start state, O(deg + B) per vertex (four length-B
// scratch rows are cleared and scanned); the update task (:433-458) applies
// the buffered moves, rebuilds M from scratch and tests convergence.
//
// Here one warp proposes for one vertex (one CTA for vertices of a degree
// above kHubDegree or kBatchHubDegree, so a hub does not set the batch's tail;
// up to that, and in precision 3 mostly beyond, a warp is faster).  The target is
// drawn in block-id order: on the dense tile through per-row chunk sums of
// M[u,:]+M[:,u] (chunks of 128 blocks, kept current by the same delta
// updates as M), on the sparse views by binary search of cumulative counts.
// The vertex's neighbour blocks are aggregated in an open-addressed hash in
// shared memory (global memory for the largest hubs), so dS costs O(deg)
// lookups: each distinct neighbour block b gives the changed entries
// M[r,b], M[s,b] (out-neighbours) or M[b,r], M[b,s] (in-neighbours); the
// entries a move leaves unchanged contribute count * (log new degree - log
// old degree), with the counts known exactly from the degrees.  The
// reference's rule that in-edges from blocks r and s do not adjust the 2x2
// row entries (the adjustment is commented out at :1135-1142) and that
// column sums skip i in {r,s} is kept.  Accepted moves are written to
// move_to[]; they are applied to the dense tile by +/-w deltas (exact
// integers, so order does not matter) and committed together with the
// partition.  The convergence bookkeeping of the update task runs on the
// device, so batches and sweeps queue without host round trips.
//
// Two schedules run the same device code.  Per batch launches: a proposal
// kernel (hubs in a second kernel on a side stream) and an apply kernel.
// Persistent: one cooperative launch runs a stage's whole nodal phase,
// one 768-thread CTA per SM, with grid barriers between entropy, sweep
// start, proposals and apply; it removes the launch gaps that otherwise
// cost about half of each batch.  There each CTA applies the moves it
// accepted itself (listed in shared memory while proposing), and for small
// B the proposals read a per-batch copy of the tile in shared memory.  In
// precision 3 a wave's proposals are only drawn by their warps; the CTA then
// evaluates their float dS together.
// State written inside that kernel (the partition, M, degrees, chunk sums,
// moves) is otherwise read through L2 (ld.cg); the non-coherent path is
// used only for data that no phase writes.  The phases
// of concurrent solves run side by side, each on fewer CTAs.
#include <cmath>
#include <mutex>
#include <type_traits>

#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>

#include "common.cuh"
#include "engine.h"

namespace cg = cooperative_groups;

namespace usap {

namespace {

// Load policies for the state a nodal batch reads: the partition, the
// block degrees and M.  LdNC (ld.global.nc) when the state is read-only
// for the whole launch; LdCG (L2, coherent) in the persistent kernel,
// whose later phases read what earlier phases wrote.
struct LdNC {
  template <class T>
  __device__ __forceinline__ static T ld(const T* p) { return __ldg(p); }
};
struct LdCG {
  template <class T>
  __device__ __forceinline__ static T ld(const T* p) { return __ldcg(p); }
};

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kHCap = 256;          // shared-memory hash slots per warp
constexpr int kChunk = 128;         // blocks per chunk sum of a dense row
constexpr int kHubThreads = 512;    // threads of a hub CTA
constexpr int kHubWarps = kHubThreads / 32;

// A group of G lanes of one warp (G = 16: a half-warp; G = 32: the warp)
// working on one vertex.  Shuffles use width G; ballots are returned as G
// bits of the caller's group.
template <int G>
struct Grp {
  int gl;          // lane within the group
  int base;        // first warp lane of the group
  unsigned mask;   // the group's lanes
  __device__ __forceinline__ explicit Grp(int lane)
      : gl(lane & (G - 1)), base(lane & ~(G - 1)),
        mask(G == 32 ? 0xffffffffu : (((1u << (G & 31)) - 1u) << (lane & ~(G - 1)))) {}
  __device__ __forceinline__ unsigned ballot(bool p) const { return __ballot_sync(mask, p) >> base; }
  __device__ __forceinline__ bool any(bool p) const { return __any_sync(mask, p) != 0; }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  template <class T>
  __device__ __forceinline__ T shfl(T v, int src) const { return __shfl_sync(mask, v, src, G); }
  template <class T>
  __device__ __forceinline__ T sum(T v) const {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, G);
    return v;
  }
  // compensated FP32 sum over the group; every lane gets the same value
  __device__ __forceinline__ FF ffsum(FF f) const {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
      f = ff_add(f, FF{__shfl_xor_sync(mask, f.hi, o, G), __shfl_xor_sync(mask, f.lo, o, G)});
    return f;
  }
  template <class T>
  __device__ __forceinline__ T incl_scan(T v) const {
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const T n = __shfl_up_sync(mask, v, o, G);
      if (gl >= o) v += n;
    }
    return v;
  }
};

// P (precision mode 1 or 2): dS is also evaluated in FP32 and decisions
// are taken on that value; the exact FP64 value is kept beside it.
// Ld loads the partition, LdT the tile state (M, Mt, chunk sums, block
// degrees): the persistent kernel may read the latter from a per-batch
// copy in shared memory.
template <class LD, int P = 0, class LDT = LD>
struct DenseOpsT {
  using Ld = LD;
  using LdT = LDT;
  static constexpr int kP = P;
  DenseView v;
  int B;
  __device__ __forceinline__ int get(int x, int y) const {
    return LDT::ld(v.M + static_cast<long long>(x) * v.ld + y);
  }
  // M[y, x], read from row x of the transposed tile (coalesced over y)
  __device__ __forceinline__ int get_t(int x, int y) const {
    return LDT::ld(v.Mt + static_cast<long long>(x) * v.ld + y);
  }
  // first block i (block-id order) whose cumulative M[u,i]+M[i,u] exceeds t:
  // a group scan over the row's chunk sums, then over the 128 entries of the
  // chosen chunk (128 / G per lane, 16-byte loads; rows are padded to ld, a
  // multiple of 4, with zeros)
  template <int G>
  __device__ __forceinline__ int sym_sample(int u, long long t, const Grp<G>& g, int* scanned) const {
    constexpr int PER = kChunk / G;
    const int nch = (B + kChunk - 1) / kChunk;
    const int* cs = v.CS + static_cast<long long>(u) * v.cld;
    long long run = 0;
    int c = nch - 1;
    for (int base = 0; base < nch; base += G) {
      const int cc = base + g.gl;
      const int val = cc < nch ? LDT::ld(cs + cc) : 0;
      const int incl = g.incl_scan(val);
      const int total = g.shfl(incl, G - 1);
      if (run + total > t) {
        const unsigned m = g.ballot(run + incl > t);
        const int l = __ffs(m) - 1;
        c = base + l;
        run += g.shfl(incl - val, l);
        break;
      }
      run += total;
    }
    const int i0 = c * kChunk + g.gl * PER;
    int pr[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) pr[k] = 0;
    const int* mrow = v.M + static_cast<long long>(u) * v.ld;
    const int* trow = v.Mt + static_cast<long long>(u) * v.ld;
#pragma unroll
    for (int q = 0; q < PER / 4; q++) {
      const int i = i0 + 4 * q;
      const int prev = q ? pr[4 * q - 1] : 0;
      if (i < B) {
        const int4 a = LDT::ld(reinterpret_cast<const int4*>(mrow + i));
        const int4 b = LDT::ld(reinterpret_cast<const int4*>(trow + i));
        pr[4 * q] = prev + a.x + b.x;
        pr[4 * q + 1] = pr[4 * q] + a.y + b.y;
        pr[4 * q + 2] = pr[4 * q + 1] + a.z + b.z;
        pr[4 * q + 3] = pr[4 * q + 2] + a.w + b.w;
      } else {
        pr[4 * q] = pr[4 * q + 1] = pr[4 * q + 2] = pr[4 * q + 3] = prev;
      }
    }
    const int last = pr[PER - 1];
    const int incl = g.incl_scan(last);
    const long long before = run + incl - last;
    const unsigned m = g.ballot(run + incl > t);
    const int l = m ? __ffs(m) - 1 : G - 1;
    int k = PER - 1;
#pragma unroll
    for (int kk = PER - 2; kk >= 0; kk--)
      if (before + pr[kk] > t) k = kk;
    *scanned += nch + kChunk;
    const int i = c * kChunk + l * PER + g.shfl(k, l);
    return i < B ? i : B - 1;
  }
};

template <int P = 0>
struct SortedOpsT {
  using Ld = LdNC;
  using LdT = LdNC;
  static constexpr int kP = P;
  SortedView v;
  int B;
  __device__ __forceinline__ int get(int x, int y) const {
    int lo = __ldg(v.rowptr + x), hi = __ldg(v.rowptr + x + 1);
    int p = find_sorted(v.col, lo, hi, y);
    return p >= 0 ? __ldg(v.val + p) : 0;
  }
  __device__ __forceinline__ int get_t(int x, int y) const { return get(y, x); }
  template <int G>
  __device__ __forceinline__ int sym_sample(int u, long long t, const Grp<G>&, int* scanned) const {
    int lo = __ldg(v.symptr + u), hi = __ldg(v.symptr + u + 1);
    long long base = lo > 0 ? __ldg(v.symcum + lo - 1) : 0;
    int j = upper_bound_i(v.symcum, lo, hi, t + base);
    if (j >= hi) j = hi - 1;   // t is below the row total; defensive clamp
    *scanned += 32 - __clz(hi - lo + 1);
    return __ldg(v.symcol + j);
  }
};

using DenseOps = DenseOpsT<LdNC>;
using SortedOps = SortedOpsT<0>;

__device__ __forceinline__ unsigned hash_slot(int b, int lg) {
  return (static_cast<unsigned>(b) * 0x9E3779B1u) >> (32 - lg);
}

__device__ __forceinline__ int table_lookup_wo(const int* key, const int* wo, int cap, int lg, int b) {
  unsigned h = hash_slot(b, lg);
  while (true) {
    int k = key[h];
    if (k == b) return wo[h];
    if (k == -1) return 0;
    h = (h + 1) & (cap - 1);
  }
}

__device__ __forceinline__ void table_insert(int* key, int* two, int* twi, int cap, int lg, int b,
                                             int ww, bool is_out) {
  unsigned h = hash_slot(b, lg);
  while (true) {
    int prev = atomicCAS(key + h, -1, b);
    if (prev == -1 || prev == b) break;
    h = (h + 1) & (cap - 1);
  }
  atomicAdd(is_out ? two + h : twi + h, ww);
}

struct VertexInfo {
  int r;
  long long kout, kin;
  int o0, dego, i0, degi;
};

template <class Ops>
__device__ __forceinline__ VertexInfo vertex_info(const NodalArgs& a, int v) {
  VertexInfo vi;
  vi.r = Ops::Ld::ld(a.part + v);
  vi.kout = __ldg(a.kout + v);
  vi.kin = __ldg(a.kin + v);
  vi.o0 = __ldg(a.out_ptr + v);
  vi.dego = __ldg(a.out_ptr + v + 1) - vi.o0;
  vi.i0 = __ldg(a.in_ptr + v);
  vi.degi = __ldg(a.in_ptr + v + 1) - vi.i0;
  return vi;
}

// target block once the chosen neighbour's block u is known
// (warp-collective): with probability B / (d_u + B) a uniform block, else
// a block drawn from row + column u of M
template <class Ops, int G>
__device__ __forceinline__ int target_from(const NodalArgs& a, const Ops& ops, const Draws& x, int u,
                                           const Grp<G>& g, int* scanned) {
  const long long dau = static_cast<long long>(Ops::LdT::ld(a.dout + u)) + Ops::LdT::ld(a.din + u);
  if (accept_uniform(x.x1, dau, a.B)) return static_cast<int>(draw_below(x.x2, a.B));
  return ops.template sym_sample<G>(u, draw_below(x.x2, dau), g, scanned);
}

// target block of the proposal for v (warp-collective), reading the
// vertex's adjacency from memory; used for hubs
template <class Ops>
__device__ __forceinline__ int propose_target(const NodalArgs& a, const Ops& ops, const Draws& x,
                                              const VertexInfo& vi, int lane, int* scanned) {
  const Grp<32> g(lane);
  const long long k = vi.kout + vi.kin;
  if (k == 0) return static_cast<int>(draw_below(x.x2, a.B));
  const long long t = draw_below(x.x0, k);
  const int deg = vi.dego + vi.degi;
  int j;
  if (a.unit) {
    j = static_cast<int>(t);
  } else {   // weighted: first neighbour whose cumulative weight exceeds t
    long long run = 0;
    j = deg - 1;
    for (int base = 0; base < deg; base += 32) {
      const int jj = base + lane;
      long long ww = 0;
      if (jj < deg) ww = jj < vi.dego ? __ldg(a.out_w + vi.o0 + jj) : __ldg(a.in_w + vi.i0 + jj - vi.dego);
      const long long incl = warp_incl_scan_ll(ww, lane);
      const long long total = __shfl_sync(0xffffffffu, incl, 31);
      if (run + total > t) {
        const unsigned m = __ballot_sync(0xffffffffu, run + incl > t);
        j = base + __ffs(m) - 1;
        break;
      }
      run += total;
    }
  }
  const int nbr = j < vi.dego ? __ldg(a.out_idx + vi.o0 + j) : __ldg(a.in_idx + vi.i0 + j - vi.dego);
  return target_from(a, ops, x, Ops::Ld::ld(a.part + nbr), g, scanned);
}

struct TermSums {
  long long acc;
  int sXR, sXS, sYR, sYS;
  FF f;   // FP32 value of the same terms (precision modes 1, 2)
};

// log of the degrees of r and s before and after the move
struct DegLogs {
  double r_out, s_out, r_out_n, s_out_n, r_in, s_in, r_in_n, s_in_n;
  FF fr_out, fs_out, fr_out_n, fs_out_n, fr_in, fs_in, fr_in_n, fs_in_n;   // precision modes 1, 2
};

template <int P>
__device__ __forceinline__ DegLogs deg_logs(const NodalArgs& a, long long dr_out, long long dr_in, long long ds_out,
                                            long long ds_in, long long kout, long long kin) {
  const double* __restrict__ L = a.L;
  DegLogs d{__ldg(L + dr_out), __ldg(L + ds_out), __ldg(L + dr_out - kout), __ldg(L + ds_out + kout),
            __ldg(L + dr_in),  __ldg(L + ds_in),  __ldg(L + dr_in - kin),   __ldg(L + ds_in + kin)};
  if constexpr (kPairTerms<P>) {
    const float2* __restrict__ T = a.L2;
    d.fr_out = ld_ff(T, dr_out);
    d.fs_out = ld_ff(T, ds_out);
    d.fr_out_n = ld_ff(T, dr_out - kout);
    d.fs_out_n = ld_ff(T, ds_out + kout);
    d.fr_in = ld_ff(T, dr_in);
    d.fs_in = ld_ff(T, ds_in);
    d.fr_in_n = ld_ff(T, dr_in - kin);
    d.fs_in_n = ld_ff(T, ds_in + kin);
  }
  return d;
}

// g(x, d1, d2) = x * ((L[x] - L[d1]) - L[d2]) from loaded log values,
// rounded exactly as g_term rounds it
__device__ __forceinline__ double g_val(long long x, double Lx, double L1, double L2) {
  if (x == 0) return 0.0;
  return __dmul_rn(static_cast<double>(x), __dsub_rn(__dsub_rn(Lx, L1), L2));
}

// dS terms of one aggregated neighbour block b (b not in {r, s}): v sends
// wo to b and receives wi from b
// the four terms of one changed pair of entries: + g(X) + g(Y) - g(X - w) - g(Y + w)
// (row entries M[r|s, b]: g(x, d_in[b], d_out[r|s]); column entries
// M[b, r|s]: g(x, d_in[r|s], d_out[b])); b's degree index is D
template <int P>
__device__ __forceinline__ void pair_terms(const NodalArgs& a, int X, int Y, int w, int D, const DegLogs& dl,
                                           bool col, TermSums& ts) {
  const double* __restrict__ L = a.L;
  const double LD = __ldg(L + D);
  const double a0 = col ? dl.r_in : dl.r_out, b0 = col ? dl.s_in : dl.s_out;
  const double a1 = col ? dl.r_in_n : dl.r_out_n, b1 = col ? dl.s_in_n : dl.s_out_n;
  const double LX = __ldg(L + X), LY = __ldg(L + Y), LXn = __ldg(L + X - w), LYn = __ldg(L + Y + w);
  ts.acc += q32(g_val(X, LX, col ? a0 : LD, col ? LD : a0));
  ts.acc += q32(g_val(Y, LY, col ? b0 : LD, col ? LD : b0));
  ts.acc -= q32(g_val(X - w, LXn, col ? a1 : LD, col ? LD : a1));
  ts.acc -= q32(g_val(Y + w, LYn, col ? b1 : LD, col ? LD : b1));
  if constexpr (kPairTerms<P>) {
    const float2* __restrict__ T = a.L2;
    const FF fD = ld_ff(T, D);
    const FF fa0 = col ? dl.fr_in : dl.fr_out, fb0 = col ? dl.fs_in : dl.fs_out;
    const FF fa1 = col ? dl.fr_in_n : dl.fr_out_n, fb1 = col ? dl.fs_in_n : dl.fs_out_n;
    ts.f = ff_add(ts.f, g_ff<P>(X, ld_ff(T, X), col ? fa0 : fD, col ? fD : fa0));
    ts.f = ff_add(ts.f, g_ff<P>(Y, ld_ff(T, Y), col ? fb0 : fD, col ? fD : fb0));
    ts.f = ff_sub(ts.f, g_ff<P>(X - w, ld_ff(T, X - w), col ? fa1 : fD, col ? fD : fa1));
    ts.f = ff_sub(ts.f, g_ff<P>(Y + w, ld_ff(T, Y + w), col ? fb1 : fD, col ? fD : fb1));
  }
}

template <class Ops>
__device__ __forceinline__ void slot_terms(const NodalArgs& a, const Ops& ops, int r, int s, int b, int wo,
                                           int wi, const DegLogs& dl, TermSums& ts) {
  if (wo > 0) {
    const int R = ops.get(r, b), S = ops.get(s, b);
    pair_terms<Ops::kP>(a, R, S, wo, Ops::LdT::ld(a.din + b), dl, false, ts);
    ts.sXR += R;
    ts.sXS += S;
  }
  if (wi > 0) {
    const int R = ops.get(b, r), S = ops.get(b, s);
    pair_terms<Ops::kP>(a, R, S, wi, Ops::LdT::ld(a.dout + b), dl, true, ts);
    ts.sYR += R;
    ts.sYS += S;
  }
}

// slot_terms from values already loaded: R = M[r,b], S = M[s,b], Di =
// d_in[b] (if wo > 0) and Rc = M[b,r], Sc = M[b,s], Do = d_out[b] (if wi > 0)
template <int P>
__device__ __forceinline__ void slot_terms_vals(const NodalArgs& a, int R, int S, int Rc, int Sc, int Di, int Do,
                                                int wo, int wi, const DegLogs& dl, TermSums& ts) {
  if (wo > 0) {
    pair_terms<P>(a, R, S, wo, Di, dl, false, ts);
    ts.sXR += R;
    ts.sXS += S;
  }
  if (wi > 0) {
    pair_terms<P>(a, Rc, Sc, wi, Do, dl, true, ts);
    ts.sYR += Rc;
    ts.sYS += Sc;
  }
}

// The 2x2 terms and the entries the move leaves unchanged, one term per
// lane (lanes 0-11), added to the warp-summed neighbour terms `ts`.  The
// four new 2x2 terms are subtracted; a -inf among them sets *ninf and is
// left out of the sum (the reference's dS is then -inf).  Every lane
// returns the same result.  P > 0: `fpart` is this lane's part of the
// FP32 sum of the neighbour terms; the group's FP32 dS goes to *f.
template <int G, int P = 0>
__device__ __forceinline__ long long finalize_grp(const NodalArgs& a, const Grp<G>& g, const TermSums& ts,
                                                   long long Rr, long long Rs, long long Sr, long long Ss,
                                                   long long wor, long long wos, long long dr_out,
                                                   long long dr_in, long long ds_out, long long ds_in,
                                                   long long kout, long long kin, int* ninf, FF fpart, double* f) {
  const double* __restrict__ L = a.L;
  const long long dr_out_n = dr_out - kout, ds_out_n = ds_out + kout;
  const long long dr_in_n = dr_in - kin, ds_in_n = ds_in + kin;
  // g lanes: mult * ((L[i0] - L[i1]) - L[i2]); coefficient lanes: mult * (L[i0] - L[i1])
  long long mult = 0, i0 = 0, i1 = 0, i2 = 0;
  bool coef = false, neg = false;
  switch (g.gl) {
    case 0: mult = Rr; i0 = Rr; i1 = dr_in; i2 = dr_out; break;
    case 1: mult = Rs; i0 = Rs; i1 = ds_in; i2 = dr_out; break;
    case 2: mult = Sr; i0 = Sr; i1 = dr_in; i2 = ds_out; break;
    case 3: mult = Ss; i0 = Ss; i1 = ds_in; i2 = ds_out; break;
    case 4: mult = Rr - wor; i0 = mult; i1 = dr_in_n; i2 = dr_out_n; neg = true; break;
    case 5: mult = Rs - wos; i0 = mult; i1 = ds_in_n; i2 = dr_out_n; neg = true; break;
    case 6: mult = Sr + wor; i0 = mult; i1 = dr_in_n; i2 = ds_out_n; neg = true; break;
    case 7: mult = Ss + wos; i0 = mult; i1 = ds_in_n; i2 = ds_out_n; neg = true; break;
    case 8: mult = dr_out - Rr - Rs - ts.sXR; i0 = dr_out_n; i1 = dr_out; coef = true; break;
    case 9: mult = ds_out - Sr - Ss - ts.sXS; i0 = ds_out_n; i1 = ds_out; coef = true; break;
    case 10: mult = dr_in - Rr - Sr - ts.sYR; i0 = dr_in_n; i1 = dr_in; coef = true; break;
    case 11: mult = ds_in - Rs - Ss - ts.sYS; i0 = ds_in_n; i1 = ds_in; coef = true; break;
    default: break;
  }
  const double La = __ldg(L + i0), Lb = __ldg(L + i1), Lc = __ldg(L + i2);
  double t = 0.0;
  if (mult != 0) {
    const double d = __dsub_rn(La, Lb);
    t = __dmul_rn(static_cast<double>(mult), coef ? d : __dsub_rn(d, Lc));
  }
  const bool inf = neg && isinf(t);
  long long q = inf ? 0 : q32(t);
  if (neg) q = -q;
  *ninf = g.any(inf) ? 1 : 0;
  if constexpr (kPairTerms<P>) {
    FF t32{0.0f, 0.0f};
    if (mult != 0 && !inf) {
      const FF A = ld_ff(a.L2, i0), Bv = ld_ff(a.L2, i1);
      t32 = coef ? coef_ff<P>(mult, A, Bv) : g_ff<P>(mult, A, Bv, ld_ff(a.L2, i2));
    }
    fpart = ff_add(fpart, neg ? ff_neg(t32) : t32);
    *f = ff_value(g.ffsum(fpart));
  }
  return ts.acc + g.sum(q);
}

// Precision mode 3: the reference's single-precision dS of v (block r)
// moving to s, _propose_new_partition_nodal (graph_parallel.hpp:1066-1215),
// in its float arithmetic and term order:
//  1. the old terms of rows r, s and (i not in {r, s}) columns r, s, block
//     by block (:1096-1114);
//  2. the four new 2x2 terms, the row entries adjusted by v's out-edges only
//     (:1180-1195; the in-edge adjustment is commented out at :1135-1142);
//  3. the new terms of rows and columns for i not in {r, s} (:1196-1215),
//     the entries adjusted by v's out-weight (rows) and in-weight (columns)
//     towards block i, from the vertex's neighbour-block weights.
// The terms can be evaluated in any order, but float addition does not
// reassociate, so they are added one after the other, in the reference's
// order, to one accumulator.  The persistent kernels evaluate the terms of
// all of a CTA's proposals together and give every chain a thread
// (coop_eval, coop_eval_sparse); ref32_eval is the form of a single warp,
// for the per-batch kernels.  Adding a zero term (an empty cell) leaves the
// float sum unchanged: the accumulator starts at +0 and round-to-nearest
// never makes it -0, so x + 0 = x holds for every value it takes (infinities
// and NaN included).
//
// One round of a warp's chain: lane l's four terms (block base + l) are
// staged in buf[4 l .. 4 l + 3] (buf: 4 G floats of shared memory, 16-byte
// aligned), and every lane then adds (or subtracts) all 4 G of them to its
// copy of the accumulator in that order.
template <int G>
__device__ __forceinline__ float ref32_accumulate(float dS, int gl, float t0, float t1, float t2, float t3, bool sub,
                                                  float* buf) {
  reinterpret_cast<float4*>(buf)[gl] = make_float4(t0, t1, t2, t3);
  __syncwarp();
#pragma unroll 8
  for (int j = 0; j < G; j++) {
    const float4 q = reinterpret_cast<const float4*>(buf)[j];
    if (sub) dS = __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(dS, q.x), q.y), q.z), q.w);
    else dS = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(dS, q.x), q.y), q.z), q.w);
  }
  __syncwarp();   // the next round overwrites buf
  return dS;
}

// How a group keeps its vertex's out- and in-weight towards each block:
// hashed by block (key, then out-, then in-weights), or in an array over all
// blocks, whose update is one addition and whose lookup one load
constexpr int kNbrHash = 0;
constexpr int kNbr8 = 1;    // 2 bytes a block: out, in (unit weights, degree <= 255)
constexpr int kNbr16 = 2;   // 4 bytes a block: out, in

// A proposal: v moves from block r to s.  In precision 3 it lies in shared
// memory until its float dS is evaluated.
struct __align__(16) Pend {
  int mode;        // kNbr*
  bool hub;        // its chunks are not listed
  const int* tab;  // v's neighbour-block weights (kNbr8, kNbr16), or the hash's keys
  const int *two, *twi;   // the hash's out- and in-weights
  float4 fo, fn;   // degree factors of rows r, s and columns r, s, old and new state
  int v, r, s, deg, scanned, noccupied;
  int dr_out, dr_in, ds_out, ds_in, kout, kin;
  int Rr, Rs, Sr, Ss, wor, wos;
  int cap, lg;     // the group's neighbour-block table
  long long acc;   // the exact value beside it (shadow)
  int ninf;
};

// the proposals of a CTA that are evaluated together
constexpr int kMaxPend = 48;   // two per warp and wave
constexpr int kSlot = 256;     // floats of a slot of coop_eval_sparse: 64 blocks x 4 rows
constexpr int kMaxSlots = 48;
struct PendList {
  Pend p[kMaxPend];
  int n;
};

// v's out- and in-weight towards block i
__device__ __forceinline__ void nbr_weights(const Pend& q, int i, int* wo, int* wi) {
  if (q.mode == kNbr8) {
    const unsigned w = reinterpret_cast<const unsigned short*>(q.tab)[i];
    *wo = w & 0xff;
    *wi = w >> 8;
  } else if (q.mode == kNbr16) {
    const unsigned w = q.tab[i];
    *wo = w & 0xffff;
    *wi = w >> 16;
  } else {
    unsigned h = hash_slot(i, q.lg);
    int k;
    while ((k = q.tab[h]) != i && k != -1) h = (h + 1) & (q.cap - 1);   // (a free slot holds no weights)
    *wo = q.two[h];
    *wi = q.twi[h];
  }
}

__device__ __forceinline__ void set_factors(Pend& q) {
  q.fo = make_float4(ref_factor(q.dr_out), ref_factor(q.ds_out), ref_factor(q.dr_in), ref_factor(q.ds_in));
  q.fn = make_float4(ref_factor(q.dr_out - q.kout), ref_factor(q.ds_out + q.kout), ref_factor(q.dr_in - q.kin),
                     ref_factor(q.ds_in + q.kin));
}

// the four new 2x2 terms (subtracted, in this order)
__device__ __forceinline__ void corner_terms(const Pend& q, float* c0, float* c1, float* c2, float* c3) {
  const int dor_n = q.dr_out - q.kout, dos_n = q.ds_out + q.kout;
  const int dir_n = q.dr_in - q.kin, dis_n = q.ds_in + q.kin;
  const int rr_r = q.Rr - q.wor, rr_s = q.Rs - q.wos, sr_r = q.Sr + q.wor, sr_s = q.Ss + q.wos;
  *c0 = rr_r ? ref_term(rr_r, static_cast<long long>(dir_n) * dor_n) : 0.0f;
  *c1 = rr_s ? ref_term(rr_s, static_cast<long long>(dis_n) * dor_n) : 0.0f;
  *c2 = sr_r ? ref_term(sr_r, static_cast<long long>(dir_n) * dos_n) : 0.0f;
  *c3 = sr_s ? ref_term(sr_s, static_cast<long long>(dis_n) * dos_n) : 0.0f;
}

__device__ __forceinline__ float ref32_corner(float dS, const Pend& q) {
  float c0, c1, c2, c3;
  corner_terms(q, &c0, &c1, &c2, &c3);
  return __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(dS, c0), c1), c2), c3);
}

// (not inlined: it runs after the group's other work is done, and a call
// gives it the registers the proposal code held.)
template <class Ops, int G>
__device__ __noinline__ float ref32_nodal(const Ops ops, const int32_t* __restrict__ din_p,
                                          const int32_t* __restrict__ dout_p, const float* Trow,
                                          const float* Tcol, int tld, const Pend& q, const int* key, const int* two,
                                          const int* twi, float* buf) {
  using LDT = typename Ops::LdT;
  const Grp<G> g(static_cast<int>(threadIdx.x & 31));
  const int B = ops.B, r = q.r, s = q.s;
  const int cap = q.cap, lg = q.lg;
  float dS = 0.0f;
  // Every round first issues the loads of the next round (pure reads of the
  // batch-start state), so that their L2 latency overlaps this round's
  // terms and chain.
  if (Trow) {
    // the old-state terms from the batch's tables (written in this launch: L2
    // loads).  Per-batch launches have none; the branch stays because the
    // compiler's code for the rounds below is slower without it (N = 20000, 97 ms
    // a solve with it, 112 ms without; a dozen other ways to write the rounds
    // took 111 to 116 ms)
    const float* tr = Trow + static_cast<long long>(r) * tld;
    const float* ts = Trow + static_cast<long long>(s) * tld;
    const float* cr = Tcol + static_cast<long long>(r) * tld;
    const float* cs = Tcol + static_cast<long long>(s) * tld;
    float n0, n1, n2, n3;
    auto tload = [&](int i) {
      const bool in = i < B, col = in && i != r && i != s;
      n0 = in ? __ldcg(tr + i) : 0.0f;
      n1 = in ? __ldcg(ts + i) : 0.0f;
      n2 = col ? __ldcg(cr + i) : 0.0f;
      n3 = col ? __ldcg(cs + i) : 0.0f;
    };
    tload(g.gl);
    for (int base = 0; base < B; base += G) {
      const float t0 = n0, t1 = n1, t2 = n2, t3 = n3;
      tload(base + G + g.gl);
      dS = ref32_accumulate<G>(dS, g.gl, t0, t1, t2, t3, false, buf);
    }
  }
  // a round's entries of rows r, s (R, S), columns r, s (Rc, Sc) and the
  // degrees of its block (d_in: di, d_out: dn)
  int nR, nS, nRc, nSc, ndi, ndn;
  if (!Trow) {
    const float dor = q.fo.x, dos = q.fo.y, dir = q.fo.z, dis = q.fo.w;
    auto oload = [&](int i) {
      nR = nS = nRc = nSc = ndi = ndn = 0;
      if (i < B) {
        nR = ops.get(r, i);
        nS = ops.get(s, i);
        if (i != r && i != s) {   // columns skip i in {r, s}
          nRc = ops.get_t(r, i);
          nSc = ops.get_t(s, i);
        }
        ndi = LDT::ld(din_p + i);
        ndn = LDT::ld(dout_p + i);
      }
    };
    oload(g.gl);
    for (int base = 0; base < B; base += G) {
      const int R = nR, S = nS, Rc = nRc, Sc = nSc;
      const float di = ref_factor(ndi), dn = ref_factor(ndn);
      oload(base + G + g.gl);
      if (!__any_sync(0xffffffffu, (R | S | Rc | Sc) != 0)) continue;
      const float t0 = ref_term_nz(R, di, dor);
      const float t1 = ref_term_nz(S, di, dos);
      const float t2 = ref_term_nz(Rc, dn, dir);
      const float t3 = ref_term_nz(Sc, dn, dis);
      dS = ref32_accumulate<G>(dS, g.gl, t0, t1, t2, t3, false, buf);
    }
  }
  dS = ref32_corner(dS, q);
  const float dor_n = q.fn.x, dos_n = q.fn.y, dir_n = q.fn.z, dis_n = q.fn.w;
  auto nload = [&](int i) {
    nR = nS = nRc = nSc = ndi = ndn = 0;
    if (i < B && i != r && i != s) {
      nR = ops.get(r, i);
      nS = ops.get(s, i);
      nRc = ops.get_t(r, i);
      nSc = ops.get_t(s, i);
      ndi = LDT::ld(din_p + i);
      ndn = LDT::ld(dout_p + i);
    }
  };
  nload(g.gl);
  for (int base = 0; base < B; base += G) {
    int R = nR, S = nS, Rc = nRc, Sc = nSc;
    const float di = ref_factor(ndi), dn = ref_factor(ndn);
    nload(base + G + g.gl);
    const int i = base + g.gl;
    // v's edges towards block i are part of M[r,i] (out) and M[i,r] (in)
    if (R > 0) {
      const int w = table_lookup_wo(key, two, cap, lg, i);
      R -= w;
      S += w;
    }
    if (Rc > 0) {
      const int w = table_lookup_wo(key, twi, cap, lg, i);
      Rc -= w;
      Sc += w;
    }
    if (!__any_sync(0xffffffffu, (R | S | Rc | Sc) != 0)) continue;
    // (all four evaluated, the empty ones discarded: no branches, so the
    // four evaluations overlap)
    const float u0 = ref_term_nz(R, di, dor_n);
    const float u1 = ref_term_nz(S, di, dos_n);
    const float u2 = ref_term_nz(Rc, dn, dir_n);
    const float u3 = ref_term_nz(Sc, dn, dis_n);
    dS = ref32_accumulate<G>(dS, g.gl, u0, u1, u2, u3, true, buf);
  }
  return dS;
}

// The float dS of a proposal by a whole warp, hashed neighbour blocks (buf:
// 128 floats).
template <class Ops>
__device__ __forceinline__ float ref32_eval(const NodalArgs& a, const Ops& ops, const Pend& q, const int* key,
                                            const int* two, const int* twi, float* buf) {
  return ref32_nodal<Ops, 32>(ops, a.din, a.dout, a.Trow, a.Tcol, a.tld, q, key, two, twi, buf);
}

// per-vertex outputs of a decided proposal; returns whether it is accepted
// (on the FP32 pair's value f in precision modes 1, 2, else on the exact
// FP64 value acc)
template <int P>
__device__ __forceinline__ bool emit(const NodalArgs& a, int v, int r, int s, long long acc, double f, int ninf) {
  const bool accept = ninf || (P > 0 ? f < 0.0 : acc < 0);
  a.move_to[v] = accept ? s : -1;
  a.from[v] = r;
  if (a.prop_s) {
    a.prop_s[v - a.beg] = s;
    a.prop_q[v - a.beg] = acc;
    a.prop_ninf[v - a.beg] = ninf;
    if (P > 0 && a.prop_f) a.prop_f[v - a.beg] = f;
  }
  return accept;
}

__device__ __forceinline__ void record_stay(const NodalArgs& a, int v, int r) {
  a.move_to[v] = -1;
  a.from[v] = r;
  if (a.prop_s) {
    a.prop_s[v - a.beg] = -1;
    a.prop_q[v - a.beg] = 0;
    a.prop_ninf[v - a.beg] = 0;
    if (a.prop_f) a.prop_f[v - a.beg] = 0.0;
  }
}

// accepted dS, moves and near-threshold proposals of one CTA, added to the
// control block once at the end of the kernel
// (the accepted dS summed for the convergence test is the exact FP64 value
// in precision modes 1 and 2, the reference's float value in mode 3)
struct CtaTally {
  unsigned long long cum, moves, near;
  int ninf;
  F32Tally f32;
  // persistent kernel: the edge chunks {v, chunk} of the CTA's accepted
  // moves, so that its apply pass visits only those (null elsewhere); *nown
  // counts past own_cap when the list overflows
  int2* own;
  int* nown;
  int own_cap;
};

// the accepted dS that the convergence test sums: the exact value, or in
// precision mode 3 the reference's float value (its update task sums the
// float dS it accepted, graph_parallel.hpp:428-434), in Q32
// |dS| <= 1e-9 for the value that decides: the exact one (Q32), or in
// precision 3 the float one
template <int P>
__device__ __forceinline__ bool near_threshold(long long acc, double f, int ninf) {
  if constexpr (P == 3) return !isinf(f) && fabs(f) <= 1e-9;
  return !ninf && acc <= kNearQ && acc >= -kNearQ;
}

template <int P>
__device__ __forceinline__ long long summed_dq(long long acc, double f) {
  if constexpr (P == 3) return q32(f);
  return acc;
}

template <int P>
__device__ __forceinline__ void tally(CtaTally* t, bool accept, long long acc, double f, int ninf, bool shadow) {
  if (accept) {
    if (ninf) atomicOr(&t->ninf, 1);
    else atomicAdd(&t->cum, static_cast<unsigned long long>(summed_dq<P>(acc, f)));
    atomicAdd(&t->moves, 1ull);
  }
  if (near_threshold<P>(acc, f, ninf)) atomicAdd(&t->near, 1ull);
  if constexpr (P > 0) {
    if (shadow && !ninf) f32_tally(&t->f32, f, acc);
  }
}

// the same straight into the control block (one proposal per CTA)
template <int P>
__device__ __forceinline__ void tally_ctl(NodalCtl* c, bool accept, long long acc, double f, int ninf,
                                          bool shadow) {
  if (accept) {
    if (ninf) atomicOr(&c->cum_ninf, 1);
    else atomicAdd(&c->cum_q, static_cast<unsigned long long>(summed_dq<P>(acc, f)));
    atomicAdd(&c->moves, 1ull);
  }
  if (near_threshold<P>(acc, f, ninf)) atomicAdd(&c->near, 1ull);
  if constexpr (P > 0) {
    if (shadow && !ninf) f32_tally(&c->f32, f, acc);
  }
}

__device__ __forceinline__ void tally_flush(const CtaTally* t, NodalCtl* ctl) {
  if (t->ninf) atomicOr(&ctl->cum_ninf, 1);
  if (t->cum) atomicAdd(&ctl->cum_q, t->cum);
  if (t->moves) atomicAdd(&ctl->moves, t->moves);
  if (t->near) atomicAdd(&ctl->near, t->near);
  f32_tally_flush(&t->f32, &ctl->f32);
}

// The outcome of a decided proposal (one lane of its group): written out,
// tallied, and its edge chunks listed for the CTA's apply pass.
template <class Ops>
__device__ __forceinline__ void close_vertex(const NodalArgs& a, const Pend& q, double f, CtaTally* tl,
                                             unsigned long long* my_bytes) {
  const bool shadow = Ops::kP != 3 || a.shadow;
  // without the shadow the -inf of a new-state term x log(x / 0) comes
  // from the float sum itself (the term is +inf there, and every new-state
  // term is subtracted)
  const int ninf = shadow ? q.ninf : (isinf(f) && f < 0.0 ? 1 : 0);
  const bool moved = emit<Ops::kP>(a, q.v, q.r, q.s, q.acc, f, ninf);
  tally<Ops::kP>(tl, moved, q.acc, f, ninf, shadow);
  if (moved && tl->own && !q.hub) {
    const int nch = q.deg > 32 ? (q.deg + 31) >> 5 : 1;   // the vertex's chunks (one even without edges)
    const int i0 = atomicAdd(tl->nown, nch);
    for (int c = 0; c < nch; c++)
      if (i0 + c < tl->own_cap) tl->own[i0 + c] = make_int2(q.v, c);
  }
  // precision 3 also reads, for the old-state and again for the new-state
  // terms, rows r and s and columns r and s of M and both degree arrays:
  // 2 x 24 bytes per block, as the reference's O(B) loops do
  if (a.stats)
    *my_bytes += 8 + 8ull * q.deg + 48ull * q.noccupied + 48 + 8ull * q.scanned + (Ops::kP == 3 ? 48ull * a.B : 0ull);
}

// Proposal for one vertex of degree <= KN * G by a group of G lanes (a
// warp, G = 32, or a half-warp, G = 16).  Each lane loads up to KN
// neighbours at once (ids, then their blocks) and keeps them in registers:
// the weights by neighbour block and the target draw (whose chosen neighbour
// is among them) come from the same loads.  tab: the group's 24 * G ints
// (hashed: 8 * G slots of key, out- and in-weight); list: KN * G ints.  With
// a.hub_units a warp also takes larger degrees, in steps of KN * G
// neighbours.  Closes the proposal, or in precision 3 leaves it in shared
// memory (the next entry of *pl, or *slot without a list) for
// its float dS to be evaluated; returns whether it did.
template <int KN, class Ops, int G>
__device__ __forceinline__ bool group_vertex(const NodalArgs& a, const Ops& ops, int v, uint32_t itr, int* tab,
                                             int* list, CtaTally* tl, const Grp<G>& g, unsigned long long* my_bytes,
                                             Pend* slot, PendList* pl) {
  using LD = typename Ops::Ld;
  using LDT = typename Ops::LdT;
  int *key = tab, *two = tab + 8 * G, *twi = tab + 16 * G;
  const unsigned lanes_below = (1u << g.gl) - 1u;
  const VertexInfo vi = vertex_info<Ops>(a, v);
  const int deg = vi.dego + vi.degi;
  const bool big = deg > KN * G;
  if (big && !(Ops::kP == 3 && G == 32 && a.hub_units)) return false;   // proposed by a larger group or a whole CTA
  const int r = vi.r;
  const Draws x = philox(static_cast<uint32_t>(v), itr, a.stage, kTagNodal, a.seed);
  const long long dr_out = LDT::ld(a.dout + r), dr_in = LDT::ld(a.din + r);
  int mode = kNbrHash;
  if (Ops::kP == 3 && a.coop && !a.shadow) {
    if (a.unit && deg <= 255 && a.B <= 48 * G) mode = kNbr8;
    else if (a.B <= 24 * G && vi.kout < 65536 && vi.kin < 65536) mode = kNbr16;
  }
  // at most 8 * G slots, of which a quarter stays free (deg <= 6 * G)
  int lg = 5;
  while ((1 << lg) < 2 * deg && (1 << lg) < 8 * G) lg++;
  const int cap = 1 << lg;
  if (mode == kNbrHash) {
    for (int i = g.gl; i < cap; i += G) {
      key[i] = -1;
      two[i] = 0;
      twi[i] = 0;
    }
  } else {
    const int words = mode == kNbr8 ? (a.B + 1) >> 1 : a.B;
    for (int i = g.gl; i < words; i += G) tab[i] = 0;
  }
  g.sync();
  auto insert = [&](int b, int w, bool is_out) {
    if (mode == kNbrHash) table_insert(key, two, twi, cap, lg, b, w, is_out);
    else if (mode == kNbr8) atomicAdd(reinterpret_cast<unsigned*>(tab) + (b >> 1), 1u << (((b & 1) << 4) | (is_out ? 0 : 8)));
    else atomicAdd(reinterpret_cast<unsigned*>(tab) + b, static_cast<unsigned>(w) << (is_out ? 0 : 16));
  };
  int nb[KN], wv[KN], pb[KN];
  // neighbours j0 + gl + G k of the out-list followed by the in-list
  auto load_nbrs = [&](int j0) {
#pragma unroll
    for (int k = 0; k < KN; k++) {
      const int j = j0 + g.gl + G * k;
      nb[k] = 0;
      wv[k] = 0;
      if (j < deg) {
        const bool is_out = j < vi.dego;
        nb[k] = is_out ? __ldg(a.out_idx + vi.o0 + j) : __ldg(a.in_idx + vi.i0 + j - vi.dego);
        wv[k] = a.unit ? 1 : (is_out ? __ldg(a.out_w + vi.o0 + j) : __ldg(a.in_w + vi.i0 + j - vi.dego));
      }
    }
#pragma unroll
    for (int k = 0; k < KN; k++) pb[k] = j0 + g.gl + G * k < deg ? LD::ld(a.part + nb[k]) : 0;
#pragma unroll
    for (int k = 0; k < KN; k++) {
      const int j = j0 + g.gl + G * k;
      if (j < deg) insert(pb[k], wv[k], j < vi.dego);
    }
  };
  load_nbrs(0);
  // the target: neighbour position j by weight, its block from registers
  int scanned = 0;
  int s;
  const long long ktot = vi.kout + vi.kin;
  if (ktot == 0) {
    s = static_cast<int>(draw_below(x.x2, a.B));
  } else if (Ops::kP == 3 && G == 32 && big) {
    for (int j0 = KN * G; j0 < deg; j0 += KN * G) load_nbrs(j0);
    s = propose_target(a, ops, x, vi, g.gl, &scanned);
  } else {
    const long long t = draw_below(x.x0, ktot);
    int j;
    if (a.unit) {
      j = static_cast<int>(t);
    } else {
      long long run = 0;
      j = deg - 1;
#pragma unroll
      for (int k = 0; k < KN; k++) {
        if (G * k >= deg) break;
        const long long ww = g.gl + G * k < deg ? wv[k] : 0;
        const long long incl = g.incl_scan(ww);
        const long long total = g.shfl(incl, G - 1);
        if (run + total > t) {
          const unsigned m = g.ballot(run + incl > t);
          j = G * k + __ffs(m) - 1;
          break;
        }
        run += total;
      }
    }
    const int kq = j / G;
    int pj = pb[0];
#pragma unroll
    for (int k = 1; k < KN; k++) pj = kq == k ? pb[k] : pj;
    s = target_from(a, ops, x, g.shfl(pj, j & (G - 1)), g, &scanned);
  }
  g.sync();
  if (s == r) {
    if (g.gl == 0) {
      record_stay(a, v, r);
      if (a.stats) *my_bytes += 8 + 8ull * deg + 8ull * scanned;
    }
    g.sync();
    return false;
  }
  const long long ds_out = LDT::ld(a.dout + s), ds_in = LDT::ld(a.din + s);
  int e4 = 0;
  if (g.gl < 4) e4 = ops.get(g.gl < 2 ? r : s, (g.gl & 1) ? s : r);
  // the exact FP64 dS (decides in precision 0; in the others the shadow
  // value the FP32 decision is compared with, skipped in precision 3
  // unless asked for)
  const bool shadow = Ops::kP != 3 || a.shadow;
  int ninf = 0, noccupied = 0;
  double f = 0.0;
  long long acc = 0;
  if (shadow) {
    const DegLogs dl = deg_logs<Ops::kP>(a, dr_out, dr_in, ds_out, ds_in, vi.kout, vi.kin);
    // compact the occupied slots so that each lane takes about one block
    int nlist = 0;
    for (int base = 0; base < cap; base += G) {
      const int i = base + g.gl;
      const int b = i < cap ? key[i] : -1;
      const unsigned occ = g.ballot(b >= 0);
      const bool use = b >= 0 && b != r && b != s;
      const unsigned mu = g.ballot(use);
      if (use) list[nlist + __popc(mu & lanes_below)] = i;
      nlist += __popc(mu);
      noccupied += __popc(occ);
    }
    g.sync();
    // each lane has at most KN slots (nlist <= KN * G): their M entries
    // and degrees are loaded in rounds of two, then the log terms
    TermSums ts{0, 0, 0, 0, 0};
#pragma unroll
    for (int k0 = 0; k0 < KN; k0 += 2) {
      int R[2], S[2], Rc[2], Sc[2], Di[2], Do[2], wo[2], wi[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int t = g.gl + G * (k0 + k);
        R[k] = S[k] = Rc[k] = Sc[k] = Di[k] = Do[k] = wo[k] = wi[k] = 0;
        if (t < nlist) {
          const int i = list[t];
          const int b = key[i];
          wo[k] = two[i];
          wi[k] = twi[i];
          if (wo[k] > 0) {
            R[k] = ops.get(r, b);
            S[k] = ops.get(s, b);
            Di[k] = LDT::ld(a.din + b);
          }
          if (wi[k] > 0) {
            Rc[k] = ops.get(b, r);
            Sc[k] = ops.get(b, s);
            Do[k] = LDT::ld(a.dout + b);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 2; k++)
        slot_terms_vals<Ops::kP>(a, R[k], S[k], Rc[k], Sc[k], Di[k], Do[k], wo[k], wi[k], dl, ts);
    }
    ts.acc = g.sum(ts.acc);
    ts.sXR = g.sum(ts.sXR);
    ts.sXS = g.sum(ts.sXS);
    ts.sYR = g.sum(ts.sYR);
    ts.sYS = g.sum(ts.sYS);
    const long long Rr = g.shfl(e4, 0), Rs = g.shfl(e4, 1);
    const long long Sr = g.shfl(e4, 2), Ss = g.shfl(e4, 3);
    const long long wor = table_lookup_wo(key, two, cap, lg, r);
    const long long wos = table_lookup_wo(key, two, cap, lg, s);
    acc = finalize_grp<G, Ops::kP>(a, g, ts, Rr, Rs, Sr, Ss, wor, wos, dr_out, dr_in, ds_out, ds_in, vi.kout,
                                   vi.kin, &ninf, ts.f, &f);
  }
  if constexpr (Ops::kP == 3) {
    const int e0 = g.shfl(e4, 0), e1 = g.shfl(e4, 1), e2 = g.shfl(e4, 2), e3 = g.shfl(e4, 3);
    if (g.gl == 0) {
      Pend& q = pl ? pl->p[atomicAdd(&pl->n, 1)] : *slot;
      q.mode = mode;
      q.hub = false;
      q.tab = key;
      q.two = two;
      q.twi = twi;
      q.v = v;
      q.r = r;
      q.s = s;
      q.deg = deg;
      q.scanned = scanned;
      q.noccupied = noccupied;
      q.acc = acc;
      q.ninf = ninf;
      q.cap = cap;
      q.lg = lg;
      q.dr_out = static_cast<int>(dr_out);
      q.dr_in = static_cast<int>(dr_in);
      q.ds_out = static_cast<int>(ds_out);
      q.ds_in = static_cast<int>(ds_in);
      q.kout = static_cast<int>(vi.kout);
      q.kin = static_cast<int>(vi.kin);
      q.Rr = e0;
      q.Rs = e1;
      q.Sr = e2;
      q.Ss = e3;
      int unused;
      nbr_weights(q, r, &q.wor, &unused);
      nbr_weights(q, s, &q.wos, &unused);
      set_factors(q);
    }
    g.sync();
    return true;
  } else {
    Pend q{};
    q.v = v;
    q.r = r;
    q.s = s;
    q.deg = deg;
    q.scanned = scanned;
    q.noccupied = noccupied;
    q.acc = acc;
    q.ninf = ninf;
    if (g.gl == 0) close_vertex<Ops>(a, q, f, tl, my_bytes);
    g.sync();
    return false;
  }
}

// One warp per vertex of degree <= kBatchHubDegree; 4 CTAs per SM, so that a
// lane's neighbours stay in registers (5 spilled: N = 20000, 113 ms a solve
// against 101 ms).  The float dS evaluates whole rows: the packing of coop_eval_sparse saves terms but
// adds latency to a warp that has a proposal of its own, and its queue takes
// shared memory from the L1 (N = 20000, per-batch launches:
// 141 ms a solve with it up to two edges a cell, 111 ms without; N = 50000: 251
// and 221 ms; N = 3000 from one block per vertex: 245 and 235 ms).
template <class Ops>
__global__ void __launch_bounds__(kThreads, 4) k_nodal_propose(NodalArgs a, Ops ops) {
  __shared__ int s_tab[kWarps][3 * kHCap];
  // occupied slots other than r, s; then the float dS's terms
  __shared__ __align__(16) int s_list[kWarps][kBatchHubDegree];
  __shared__ Pend s_pend[Ops::kP == 3 ? kWarps : 1];
  __shared__ CtaTally s_tally;
  if (a.ctl->done) return;   // written by earlier launches only
  const uint32_t itr = static_cast<uint32_t>(a.ctl->itr);
  if (threadIdx.x == 0) s_tally = CtaTally{0, 0, 0, 0};
  if constexpr (Ops::kP == 3) ref_tab_fill();
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nwarps = gridDim.x * kWarps;
  unsigned long long my_bytes = 0;
  for (int v = a.beg + blockIdx.x * kWarps + wib; v < a.end; v += nwarps) {
    int* const tab = s_tab[wib];
    const bool live = group_vertex<kBatchHubDegree / 32>(a, ops, v, itr, tab, s_list[wib], &s_tally, Grp<32>(lane),
                                                         &my_bytes, Ops::kP == 3 ? s_pend + wib : nullptr, nullptr);
    if constexpr (Ops::kP == 3) {
      if (live) {   // warp-uniform
        const float f = ref32_eval(a, ops, s_pend[wib], tab, tab + kHCap, tab + 2 * kHCap,
                                   reinterpret_cast<float*>(s_list[wib]));
        if (lane == 0) close_vertex<Ops>(a, s_pend[wib], f, &s_tally, &my_bytes);
        __syncwarp();
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) tally_flush(&s_tally, a.ctl);
  if (a.stats && lane == 0 && my_bytes) atomicAdd(&a.ctl->bytes, my_bytes);
}

template <int NW>
struct HubShared {
  long long acc[NW];
  int sum[5][NW];
  float fhi[NW], flo[NW];   // FP32 partial sums (precision modes 1, 2)
  int target, scanned;
  Pend pend;   // precision 3, without a list
};

// Proposal for one vertex of a larger degree by a whole CTA of NT
// threads.  The last warp draws the target while the others fill the hash
// of neighbour blocks (at most min(deg, B) entries: in `stab`, a shared
// region of `scap` slots per array, or beyond that in the vertex's global
// region; with a list, precision 3, the arrays follow one another from the
// region's end); each thread loads four neighbours at once, and up to four
// occupied slots at once for the terms.  In precision 3 the proposal is left
// in pl's first entry, or, without a list, warp 0 evaluates
// its float dS (chain: 128 floats).
template <class Ops, int NT>
__device__ __forceinline__ void hub_vertex(const NodalArgs& a, const Ops& ops, int v, uint32_t itr, int* stab,
                                           int scap, HubShared<NT / 32>* sh, unsigned long long* my_bytes,
                                           float* chain, PendList* pl) {
  using LD = typename Ops::Ld;
  using LDT = typename Ops::LdT;
  constexpr int NW = NT / 32;
  constexpr int kIns = NT - 32;   // threads that fill the table
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const VertexInfo vi = vertex_info<Ops>(a, v);
  const int deg = vi.dego + vi.degi;
  const int r = vi.r;
  const int distinct_max = deg < a.B ? deg : a.B;
  int lg = 5;
  while ((1 << lg) < 2 * distinct_max) lg++;
  const int cap = 1 << lg;
  int *key, *two, *twi;
  if (cap <= scap) {
    key = stab;
    two = stab + scap;
    twi = stab + 2 * scap;
    if (Ops::kP == 3 && pl) {   // what precedes them is free for the float dS
      key = stab + 3 * (scap - cap);
      two = key + cap;
      twi = two + cap;
    }
  } else {
    const long long off = __ldg(a.hi_off + v);
    key = a.hkey + off;
    two = a.hwo + off;
    twi = a.hwi + off;
  }
  for (int i = threadIdx.x; i < cap; i += NT) {
    key[i] = -1;
    two[i] = 0;
    twi[i] = 0;
  }
  __syncthreads();
  if (wib == NW - 1) {
    const Draws x = philox(static_cast<uint32_t>(v), itr, a.stage, kTagNodal, a.seed);
    int scanned = 0;
    const int st = propose_target(a, ops, x, vi, lane, &scanned);
    if (lane == 0) {
      sh->target = st;
      sh->scanned = scanned;
    }
  } else {
    for (int j0 = threadIdx.x; j0 < deg; j0 += 4 * kIns) {
      int nb[4], wv[4], pb[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int j = j0 + k * kIns;
        nb[k] = 0;
        wv[k] = 0;
        if (j < deg) {
          const bool is_out = j < vi.dego;
          nb[k] = is_out ? __ldg(a.out_idx + vi.o0 + j) : __ldg(a.in_idx + vi.i0 + j - vi.dego);
          wv[k] = a.unit ? 1 : (is_out ? __ldg(a.out_w + vi.o0 + j) : __ldg(a.in_w + vi.i0 + j - vi.dego));
        }
      }
#pragma unroll
      for (int k = 0; k < 4; k++) pb[k] = j0 + k * kIns < deg ? LD::ld(a.part + nb[k]) : 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int j = j0 + k * kIns;
        if (j < deg) table_insert(key, two, twi, cap, lg, pb[k], wv[k], j < vi.dego);
      }
    }
  }
  __syncthreads();
  const int s = sh->target;
  if (s == r) {
    if (threadIdx.x == 0) {
      record_stay(a, v, r);
      if (a.stats) *my_bytes += 8 + 8ull * deg + 8ull * sh->scanned;
    }
    __syncthreads();
    return;
  }
  const long long dr_out = LDT::ld(a.dout + r), dr_in = LDT::ld(a.din + r);
  const long long ds_out = LDT::ld(a.dout + s), ds_in = LDT::ld(a.din + s);
  const DegLogs dl = deg_logs<Ops::kP>(a, dr_out, dr_in, ds_out, ds_in, vi.kout, vi.kin);
  TermSums ts{0, 0, 0, 0, 0};
  int nocc = 0;
  for (int i = threadIdx.x; i < cap;) {
    int sl[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      sl[k] = -1;
      while (i < cap) {
        const int b = key[i];
        i += NT;
        if (b < 0) continue;
        nocc++;
        if (b != r && b != s) {
          sl[k] = i - NT;
          break;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (sl[k] >= 0) slot_terms(a, ops, r, s, key[sl[k]], two[sl[k]], twi[sl[k]], dl, ts);
  }
  ts.acc = warp_sum_ll(ts.acc);
  ts.sXR = warp_sum_i(ts.sXR);
  ts.sXS = warp_sum_i(ts.sXS);
  ts.sYR = warp_sum_i(ts.sYR);
  ts.sYS = warp_sum_i(ts.sYS);
  nocc = warp_sum_i(nocc);
  if constexpr (kPairTerms<Ops::kP>) ts.f = Grp<32>(lane).ffsum(ts.f);
  if (lane == 0) {
    sh->acc[wib] = ts.acc;
    sh->fhi[wib] = ts.f.hi;
    sh->flo[wib] = ts.f.lo;
    sh->sum[0][wib] = ts.sXR;
    sh->sum[1][wib] = ts.sXS;
    sh->sum[2][wib] = ts.sYR;
    sh->sum[3][wib] = ts.sYS;
    sh->sum[4][wib] = nocc;
  }
  __syncthreads();
  if (wib == 0) {
    TermSums tot{0, 0, 0, 0, 0};
    int occ = 0;
    FF fpart{0.0f, 0.0f};
    if (lane < NW) {
      fpart = FF{sh->fhi[lane], sh->flo[lane]};
      tot.acc = sh->acc[lane];
      tot.sXR = sh->sum[0][lane];
      tot.sXS = sh->sum[1][lane];
      tot.sYR = sh->sum[2][lane];
      tot.sYS = sh->sum[3][lane];
      occ = sh->sum[4][lane];
    }
    tot.acc = warp_sum_ll(tot.acc);
    tot.sXR = warp_sum_i(tot.sXR);
    tot.sXS = warp_sum_i(tot.sXS);
    tot.sYR = warp_sum_i(tot.sYR);
    tot.sYS = warp_sum_i(tot.sYS);
    occ = warp_sum_i(occ);
    int e4 = 0;
    if (lane < 4) e4 = ops.get(lane < 2 ? r : s, (lane & 1) ? s : r);
    const long long Rr = __shfl_sync(0xffffffffu, e4, 0), Rs = __shfl_sync(0xffffffffu, e4, 1);
    const long long Sr = __shfl_sync(0xffffffffu, e4, 2), Ss = __shfl_sync(0xffffffffu, e4, 3);
    const long long wor = table_lookup_wo(key, two, cap, lg, r);
    const long long wos = table_lookup_wo(key, two, cap, lg, s);
    int ninf;
    double f = 0.0;
    const long long acc = finalize_grp<32, Ops::kP>(a, Grp<32>(lane), tot, Rr, Rs, Sr, Ss, wor, wos, dr_out,
                                                    dr_in, ds_out, ds_in, vi.kout, vi.kin, &ninf, fpart, &f);
    if constexpr (Ops::kP == 3) {
      Pend& q = pl ? pl->p[0] : sh->pend;
      if (lane == 0) {
        q.mode = kNbrHash;
        q.hub = true;
        q.tab = key;
        q.two = two;
        q.twi = twi;
        q.v = v;
        q.deg = deg;
        q.scanned = sh->scanned;
        q.noccupied = occ;
        q.acc = acc;
        q.ninf = ninf;
        q.r = r;
        q.s = s;
        q.dr_out = static_cast<int>(dr_out);
        q.dr_in = static_cast<int>(dr_in);
        q.ds_out = static_cast<int>(ds_out);
        q.ds_in = static_cast<int>(ds_in);
        q.kout = static_cast<int>(vi.kout);
        q.kin = static_cast<int>(vi.kin);
        q.Rr = static_cast<int>(Rr);
        q.Rs = static_cast<int>(Rs);
        q.Sr = static_cast<int>(Sr);
        q.Ss = static_cast<int>(Ss);
        q.wor = static_cast<int>(wor);
        q.wos = static_cast<int>(wos);
        q.cap = cap;
        q.lg = lg;
        set_factors(q);
        if (pl) pl->n = 1;
      }
      __syncwarp();
      if (!pl)
        f = ref32_eval(a, ops, q, key, two, twi, chain);
    }
    // (a hub's exact value is a CTA-parallel sum over its slots and is
    // always evaluated; without the shadow it is not reported, as for the
    // other vertices)
    const bool shadow = Ops::kP != 3 || a.shadow;
    if (!shadow) ninf = isinf(f) && f < 0.0 ? 1 : 0;
    if (lane == 0 && !(Ops::kP == 3 && pl)) {
      tally_ctl<Ops::kP>(a.ctl, emit<Ops::kP>(a, v, r, s, acc, f, ninf), acc, f, ninf, shadow);
      if (a.stats)
        *my_bytes += 8 + 8ull * deg + 48ull * occ + 48 + 8ull * sh->scanned + (Ops::kP == 3 ? 48ull * a.B : 0ull);
    }
  }
  __syncthreads();
}

// one CTA per vertex of degree > kBatchHubDegree, hash in dynamic shared memory
// (`smem_cap` slots per array) or the vertex's global region
template <class Ops>
__global__ void __launch_bounds__(kHubThreads) k_nodal_propose_hub(NodalArgs a, Ops ops, const int32_t* hubs,
                                                                  int hub_lo, int hub_hi, int smem_cap) {
  extern __shared__ __align__(16) int dyn[];
  __shared__ HubShared<kHubWarps> sh;
  __shared__ __align__(16) float s_chain[Ops::kP == 3 ? 128 : 1];
  if (a.ctl->done) return;
  const uint32_t itr = static_cast<uint32_t>(a.ctl->itr);
  unsigned long long my_bytes = 0;
  if constexpr (Ops::kP == 3) {
    ref_tab_fill();
    __syncthreads();
  }
  for (int h = hub_lo + blockIdx.x; h < hub_hi; h += gridDim.x)
    hub_vertex<Ops, kHubThreads>(a, ops, __ldg(hubs + h), itr, dyn, smem_cap, &sh, &my_bytes, s_chain, nullptr);
  if (a.stats && threadIdx.x == 0 && my_bytes) atomicAdd(&a.ctl->bytes, my_bytes);
}

// --- block-merge proposals on the dense tile ------------------------------------
// The block_merge task (graph_parallel.hpp:349-368, _propose_new_partition_block
// :761-988) for B <= dense_max, reading the tile the nodal phase keeps (M, its
// transpose, the chunk sums) instead of sorted sparse views.  Draws, candidate
// order and the Q32 terms are those of the sparse kernel (kernels_merge.cu):
// the symmetric row M[u,:]+M[:,u] is walked in block-id order through the
// chunk sums, and the rows and columns of r and s are scanned whole, every
// column where both are non-zero giving one h term.

// sum of M[u,i] + M[i,u] over i < r (warp-collective, every lane returns it)
__device__ __forceinline__ long long sym_prefix(const DenseView& v, int u, int r, int lane) {
  const int c = r / kChunk;
  long long acc = 0;
  const int* cs = v.CS + static_cast<long long>(u) * v.cld;
  for (int q = lane; q < c; q += 32) acc += __ldg(cs + q);
  const int* mrow = v.M + static_cast<long long>(u) * v.ld;
  const int* trow = v.Mt + static_cast<long long>(u) * v.ld;
  for (int i = c * kChunk + lane; i < r; i += 32) acc += __ldg(mrow + i) + __ldg(trow + i);
  return warp_sum_ll(acc);
}

template <int P>
__global__ void __launch_bounds__(kThreads) k_merge_propose_dense(DenseView v, MergeArgs a) {
  constexpr bool F32 = P > 0;
  __shared__ F32Tally s_f32;
  if (F32) {
    if (threadIdx.x == 0) s_f32 = F32Tally{0, 0, 0, 0.0};
    __syncthreads();
  }
  const int lane = threadIdx.x & 31;
  const DenseOps ops{v, a.B};
  const Grp<32> g(lane);
  const long long items = static_cast<long long>(a.B) * a.K;
  const long long nwarps = static_cast<long long>(gridDim.x) * kWarps;
  for (long long item = static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5); item < items;
       item += nwarps) {
    const int r = static_cast<int>(item / a.K), k = static_cast<int>(item - static_cast<long long>(r) * a.K);
    const int B = a.B;
    const Draws x = philox(static_cast<uint32_t>(r), static_cast<uint32_t>(k), a.stage, kTagMerge, a.seed);
    const long long dr_out = __ldg(a.dout + r), dr_in = __ldg(a.din + r);
    const long long ka = dr_out + dr_in;
    int s;
    int scanned = 0;
    if (ka == 0) {
      s = static_cast<int>(draw_below(x.x2, B));
    } else {
      const int u = ops.sym_sample(r, static_cast<long long>(draw_below(x.x0, ka)), g, &scanned);
      const long long dau = static_cast<long long>(__ldg(a.dout + u)) + __ldg(a.din + u);
      if (accept_uniform(x.x1, dau, B)) {
        s = skip_r(static_cast<int>(draw_below(x.x2, B)), r, B);
      } else {
        // the multinomial over row u with r left out
        const long long c_ur = static_cast<long long>(ops.get(u, r)) + ops.get(r, u);
        const long long before = sym_prefix(v, u, r, lane);
        const long long wsum = dau - c_ur;
        if (wsum == 0) {
          s = skip_r(static_cast<int>(draw_below(x.x2, B)), r, B);
        } else {
          long long t2 = draw_below(x.x2, wsum);
          if (c_ur > 0 && t2 >= before) t2 += c_ur;
          s = ops.sym_sample(u, t2, g, &scanned);
        }
      }
    }
    // --- dS of merging r into s ---
    const long long ds_out = __ldg(a.dout + s), ds_in = __ldg(a.din + s);
    const long long ds_out_n = ds_out + dr_out, ds_in_n = ds_in + dr_in;
    int e4 = 0;
    if (lane < 4) e4 = ops.get(lane < 2 ? r : s, (lane & 1) ? s : r);
    const long long Mrr = __shfl_sync(0xffffffffu, e4, 0), Mrs = __shfl_sync(0xffffffffu, e4, 1);
    const long long Msr = __shfl_sync(0xffffffffu, e4, 2), Mss = __shfl_sync(0xffffffffu, e4, 3);
    long long acc = 0;
    FF f{0.0f, 0.0f};
    // rows r and s (M) and columns r and s (rows of Mt): columns i not in
    // {r, s} where both entries are non-zero
    const int* mr = v.M + static_cast<long long>(r) * v.ld;
    const int* ms = v.M + static_cast<long long>(s) * v.ld;
    const int* tr = v.Mt + static_cast<long long>(r) * v.ld;
    const int* ts = v.Mt + static_cast<long long>(s) * v.ld;
    for (int i = lane; i < B; i += 32) {
      if (i == r || i == s) continue;
      const int xr = __ldg(mr + i), xs = __ldg(ms + i);
      if (xr > 0 && xs > 0) {
        acc += q32(h_term(a.L, xr, xs));
        if constexpr (F32) f = ff_add(f, h_term_ff<P>(a.L2, xr, xs));
      }
      const int yr = __ldg(tr + i), ys = __ldg(ts + i);
      if (yr > 0 && ys > 0) {
        acc += q32(h_term(a.L, yr, ys));
        if constexpr (F32) f = ff_add(f, h_term_ff<P>(a.L2, yr, ys));
      }
    }
    acc = warp_sum_ll(acc);
    if constexpr (F32) f = g.ffsum(f);
    if (lane == 0) {
      acc += q32(g_term(a.L, Mrr, dr_in, dr_out));
      acc += q32(g_term(a.L, Mrs, ds_in, dr_out));
      acc += q32(g_term(a.L, Msr, dr_in, ds_out));
      acc += q32(g_term(a.L, Mss, ds_in, ds_out));
      acc -= q32(g_term(a.L, Mrr + Mrs + Msr + Mss, ds_in_n, ds_out_n));
      long long Ar, As, Cr, Cs;
      if (s != r) {
        Ar = dr_out - Mrr - Mrs;
        As = ds_out - Msr - Mss;
        Cr = dr_in - Mrr - Msr;
        Cs = ds_in - Mrs - Mss;
      } else {
        Ar = As = dr_out - Mrr;
        Cr = Cs = dr_in - Mrr;
      }
      acc += q32(coef_term(a.L, Ar, ds_out_n, dr_out));
      acc += q32(coef_term(a.L, As, ds_out_n, ds_out));
      acc += q32(coef_term(a.L, Cr, ds_in_n, dr_in));
      acc += q32(coef_term(a.L, Cs, ds_in_n, ds_in));
      a.prop_s[item] = s;
      if constexpr (F32) {
        const float2* __restrict__ T = a.L2;
        f = ff_add(f, g_term_ff<P>(T, Mrr, dr_in, dr_out));
        f = ff_add(f, g_term_ff<P>(T, Mrs, ds_in, dr_out));
        f = ff_add(f, g_term_ff<P>(T, Msr, dr_in, ds_out));
        f = ff_add(f, g_term_ff<P>(T, Mss, ds_in, ds_out));
        f = ff_sub(f, g_term_ff<P>(T, Mrr + Mrs + Msr + Mss, ds_in_n, ds_out_n));
        f = ff_add(f, coef_ff<P>(Ar, ld_ff(T, ds_out_n), ld_ff(T, dr_out)));
        f = ff_add(f, coef_ff<P>(As, ld_ff(T, ds_out_n), ld_ff(T, ds_out)));
        f = ff_add(f, coef_ff<P>(Cr, ld_ff(T, ds_in_n), ld_ff(T, dr_in)));
        f = ff_add(f, coef_ff<P>(Cs, ld_ff(T, ds_in_n), ld_ff(T, ds_in)));
        const double fv = ff_value(f);
        a.prop_q[item] = q32(fv);
        a.prop_x[item] = acc;
        a.prop_f[item] = fv;
        const double err = f32_err(fv, acc);
        atomicAdd(&s_f32.evals, 1ull);
        atomicMax(&s_f32.err_max, static_cast<unsigned long long>(__double_as_longlong(err)));
        atomicAdd(&s_f32.err_sum, err);
      } else {
        a.prop_q[item] = acc;
      }
    }
  }
  if (F32) {
    __syncthreads();
    if (threadIdx.x == 0) f32_tally_flush(&s_f32, a.f32);
  }
}

// chunk sums CS[u][c] = sum over the chunk's blocks i of M[u,i] + M[i,u]
__global__ void __launch_bounds__(kThreads) k_chunk_sums(int B, int ld, const int* __restrict__ M,
                                                        const int* __restrict__ Mt, int cld,
                                                        int* __restrict__ CS) {
  const int lane = threadIdx.x & 31;
  const int nch = (B + kChunk - 1) / kChunk;
  const long long items = static_cast<long long>(B) * nch;
  const long long nwarps = static_cast<long long>(gridDim.x) * kWarps;
  for (long long it = static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5); it < items;
       it += nwarps) {
    const int u = static_cast<int>(it / nch), c = static_cast<int>(it - static_cast<long long>(u) * nch);
    const int i0 = c * kChunk + lane * 4;
    int sum = 0;
    if (i0 < B) {
      const int4 a = *reinterpret_cast<const int4*>(M + static_cast<long long>(u) * ld + i0);
      const int4 b = *reinterpret_cast<const int4*>(Mt + static_cast<long long>(u) * ld + i0);
      sum = a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w;
    }
    sum = warp_sum_i(sum);
    if (lane == 0) CS[static_cast<long long>(u) * cld + c] = sum;
  }
}

// update (:433-458), second half: the sweep's cumulative dS is recorded for
// this sweep and added to S after every batch (as the reference does), then
// the convergence test -mean < thr * S ends the nodal phase.  One thread.
// The control block is read at once through L2 (ld.cg: the persistent
// kernel calls this after other CTAs wrote it), then written back.
__device__ __forceinline__ bool ctl_batch_end(NodalCtl* ctl, const CtlArgs& c) {
  const int done = __ldcg(&ctl->done);
  const long long cum = static_cast<long long>(__ldcg(&ctl->cum_q));
  const int itr = __ldcg(&ctl->itr);
  const int cum_ninf = __ldcg(&ctl->cum_ninf);
  const long long S_q = __ldcg(&ctl->S_q) + cum;
  const int S_ninf = __ldcg(&ctl->S_ninf) | cum_ninf;
  const unsigned long long batches = __ldcg(&ctl->batches);
  const unsigned long long proposals = __ldcg(&ctl->proposals);
  const unsigned long long edge_visits = __ldcg(&ctl->edge_visits);
  const double mean = __ldcg(&ctl->mean);
  if (done) return true;
  c.ide_q[itr] = cum;
  c.ide_n[itr] = cum_ninf;
  ctl->S_q = S_q;
  ctl->S_ninf = S_ninf;
  ctl->batches = batches + 1;
  ctl->proposals = proposals + static_cast<unsigned long long>(c.batch_vertices);
  ctl->edge_visits = edge_visits + static_cast<unsigned long long>(c.batch_edges);
  if (itr >= c.W - 1) {
    const double S_d = S_ninf ? -INFINITY : c.model_d + static_cast<double>(S_q) / kQ32;
    if (-mean < c.thr * S_d) {
      ctl->done = 1;
      return true;
    }
  }
  return false;
}

// prepare_batch (:381-395): the data term of S from the entropy
// accumulator (the model term is added where S is compared), the moving
// average of the previous sweeps' dS, and a fresh cumulative sum for this
// sweep.  One thread; reads as in ctl_batch_end.
__device__ __forceinline__ void ctl_sweep_start(NodalCtl* ctl, int W,
                                                const long long* ide_q, const int* ide_n) {
  const int done = __ldcg(&ctl->done);
  const unsigned long long sweeps = __ldcg(&ctl->sweeps);
  const unsigned long long eacc = __ldcg(&ctl->entropy_acc);
  if (done) return;
  const int itr = static_cast<int>(sweeps);
  double mean = 0.0;
  if (itr >= W - 1) {
    long long sum = 0;
    int ninf = 0;
    for (int i = itr - W + 1; i < itr; i++) {
      sum += __ldcg(ide_q + i);
      ninf |= __ldcg(ide_n + i);
    }
    mean = ninf ? -INFINITY : (static_cast<double>(sum) / kQ32) / static_cast<double>(W - 1);
  }
  ctl->itr = itr;
  ctl->S_q = -static_cast<long long>(eacc);
  ctl->S_ninf = 0;
  ctl->mean = mean;
  ctl->cum_q = 0;
  ctl->cum_ninf = 0;
  ctl->sweeps = sweeps + 1;
}

struct LdPlain {
  template <class T>
  __device__ __forceinline__ static T ld(const T* p) { return *p; }
};

// Accumulation of one CTA's tile deltas during an apply pass, in one of
// three modes.  All sums are exact integers, so the order of the updates
// does not matter.
//  kDeltaHashed: open-addressed tables in shared memory; `mkey/mval` hold
//    M[a][b] += d under the key a * ld + b; at the flush each entry updates
//    M and Mt and feeds the chunk sums of rows a and b, which are
//    accumulated in `ckey/cval` (key row * cld + chunk) and flushed last.  A
//    table that is full passes the update straight to global memory.
//  kDeltaDense (B * B <= the table region): a dense B x B array of deltas in
//    `mkey` (row stride dB = B) and the chunk-sum deltas in `ckey` (row *
//    cld + chunk); no probing, and a flush that scans B * B cells.  For
//    small B, where every CTA's updates fall on a few hundred cells and
//    global atomics would queue on them.
//  kDeltaGlobal: every update straight to M, Mt and the chunk sums; for
//    large B the updates spread over many cells and the per-CTA tables cost
//    more (clear, probes, flush) than they save.
constexpr int kDeltaHashed = 0, kDeltaGlobal = 1, kDeltaDense = 2;
struct DeltaTables {
  int *mkey, *mval, *ckey, *cval;
  int mlg, clg;   // capacities 1 << mlg, 1 << clg
  int mode = kDeltaHashed;
  int dB = 0;     // kDeltaDense: B
};

// Adds d under key k; false when no slot was found within kProbeMax probes
// (the caller then adds straight to global memory), so a nearly full table
// costs a bounded number of probes per insert.
constexpr int kProbeMax = 32;

__device__ __forceinline__ bool table_add(int* key, int* val, int lg, int k, int d) {
  const int cap = 1 << lg;
  unsigned h = hash_slot(k, lg);
  const int probes = cap < kProbeMax ? cap : kProbeMax;
  for (int probe = 0; probe < probes; probe++) {
    const int prev = atomicCAS(key + h, -1, k);
    if (prev == -1 || prev == k) {
      atomicAdd(val + h, d);
      return true;
    }
    h = (h + 1) & (cap - 1);
  }
  return false;
}

__device__ __forceinline__ void cs_add(const DeltaTables& t, int* CS, int key, int d) {
  if (!table_add(t.ckey, t.cval, t.clg, key, d)) atomicAdd(CS + key, d);
}

__device__ __forceinline__ void tile_add(const DeltaTables& t, int* M, int* Mt, int* CS, int ld, int cld, int x,
                                         int y, int d) {
  if (t.mode == kDeltaDense) {
    atomicAdd(t.mkey + x * t.dB + y, d);
    atomicAdd(t.ckey + x * cld + y / kChunk, d);
    atomicAdd(t.ckey + y * cld + x / kChunk, d);
    return;
  }
  if (t.mode == kDeltaGlobal) {
    atomicAdd(M + static_cast<long long>(x) * ld + y, d);
    atomicAdd(Mt + static_cast<long long>(y) * ld + x, d);
    atomicAdd(CS + x * cld + y / kChunk, d);
    atomicAdd(CS + y * cld + x / kChunk, d);
    return;
  }
  if (table_add(t.mkey, t.mval, t.mlg, x * ld + y, d)) return;
  atomicAdd(M + static_cast<long long>(x) * ld + y, d);
  atomicAdd(Mt + static_cast<long long>(y) * ld + x, d);
  cs_add(t, CS, x * cld + y / kChunk, d);
  cs_add(t, CS, y * cld + x / kChunk, d);
}

__device__ __forceinline__ void tables_clear(const DeltaTables& t) {
  for (int i = threadIdx.x; i < (1 << t.mlg); i += blockDim.x) {
    t.mkey[i] = -1;
    t.mval[i] = 0;
  }
  for (int i = threadIdx.x; i < (1 << t.clg); i += blockDim.x) {
    t.ckey[i] = -1;
    t.cval[i] = 0;
  }
}

// writes the CTA's accumulated deltas to the tile (CTA-collective; the
// tables are cleared again on the way)
__device__ __forceinline__ void tables_flush(const DeltaTables& t, int* M, int* Mt, int* CS, int ld, int cld) {
  __syncthreads();
  for (int i = threadIdx.x; i < (1 << t.mlg); i += blockDim.x) {
    const int k = t.mkey[i];
    if (k < 0) continue;
    const int d = t.mval[i];
    t.mkey[i] = -1;
    t.mval[i] = 0;
    if (d == 0) continue;
    const int x = k / ld, y = k - x * ld;
    atomicAdd(M + static_cast<long long>(x) * ld + y, d);
    atomicAdd(Mt + static_cast<long long>(y) * ld + x, d);
    cs_add(t, CS, x * cld + y / kChunk, d);
    cs_add(t, CS, y * cld + x / kChunk, d);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < (1 << t.clg); i += blockDim.x) {
    const int k = t.ckey[i];
    if (k < 0) continue;
    const int d = t.cval[i];
    t.ckey[i] = -1;
    t.cval[i] = 0;
    if (d) atomicAdd(CS + k, d);
  }
  __syncthreads();
}

// kDeltaDense: zero the B x B deltas and the B * cld chunk-sum deltas
__device__ __forceinline__ void dense_clear(const DeltaTables& t, int cld) {
  const int nm = t.dB * t.dB, nc = t.dB * cld;
  for (int i = threadIdx.x; i < nm; i += blockDim.x) t.mkey[i] = 0;
  for (int i = threadIdx.x; i < nc; i += blockDim.x) t.ckey[i] = 0;
}

// kDeltaDense: writes the non-zero deltas to M, Mt and the chunk sums (whose
// layout row * cld + chunk the dense array shares) and zeroes them
// (CTA-collective)
__device__ __forceinline__ void dense_flush(const DeltaTables& t, int* M, int* Mt, int* CS, int ld, int cld) {
  __syncthreads();
  const int B = t.dB, nm = B * B, nc = B * cld;
  for (int i = threadIdx.x; i < nm; i += blockDim.x) {
    const int d = t.mkey[i];
    if (d == 0) continue;
    t.mkey[i] = 0;
    const int x = i / B, y = i - x * B;
    atomicAdd(M + static_cast<long long>(x) * ld + y, d);
    atomicAdd(Mt + static_cast<long long>(y) * ld + x, d);
  }
  for (int i = threadIdx.x; i < nc; i += blockDim.x) {
    const int d = t.ckey[i];
    if (d == 0) continue;
    t.ckey[i] = 0;
    atomicAdd(CS + i, d);
  }
}

// Applies and commits the moves of one 32-edge chunk of a batch vertex
// (warp-collective).  A chunk whose vertex did not move returns at once.
// Old blocks of batch vertices come from `from`, so part[] is committed in
// the same pass: part is read only for vertices outside [beg, end).  An
// edge between two moved vertices is applied once, from its source's
// out-list.  LDM loads move_to/from, LDP the partition.  Tile deltas go to
// the CTA's tables.
template <class LDM, class LDP>
__device__ __forceinline__ void apply_chunk(int2 ch, const GraphDev& g, int32_t* part, const int32_t* move_to,
                                            const int32_t* from, int beg, int end, const DeltaTables& t, int ld,
                                            int* M, int* Mt, int cld, int* CS, int32_t* dout, int32_t* din,
                                            int lane) {
  const int v = ch.x;
  const int s = LDM::ld(move_to + v);
  if (s < 0) return;   // warp-uniform
  const int r = LDM::ld(from + v);
  const int o0 = __ldg(g.out_ptr + v), dego = __ldg(g.out_ptr + v + 1) - o0;
  const int i0 = __ldg(g.in_ptr + v), degi = __ldg(g.in_ptr + v + 1) - i0;
  if (ch.y == 0 && lane == 0) {
    part[v] = s;
    const int ko = __ldg(g.kout + v), ki = __ldg(g.kin + v);
    atomicSub(dout + r, ko);
    atomicAdd(dout + s, ko);
    atomicSub(din + r, ki);
    atomicAdd(din + s, ki);
  }
  const unsigned span = static_cast<unsigned>(end - beg);
  const int j = ch.y * 32 + lane;
  if (j >= dego + degi) return;
  const bool is_out = j < dego;
  const int y = is_out ? __ldg(g.out_idx + o0 + j) : __ldg(g.in_idx + i0 + j - dego);
  int w = 1;
  if (is_out ? g.out_w != nullptr : g.in_w != nullptr)
    w = is_out ? __ldg(g.out_w + o0 + j) : __ldg(g.in_w + i0 + j - dego);
  const bool inb = static_cast<unsigned>(y - beg) < span;
  const int my = inb ? LDM::ld(move_to + y) : -1;
  const int oy = inb ? LDM::ld(from + y) : LDP::ld(part + y);
  if (is_out) {
    tile_add(t, M, Mt, CS, ld, cld, r, oy, -w);
    tile_add(t, M, Mt, CS, ld, cld, s, my >= 0 ? my : oy, w);
  } else if (my < 0) {
    tile_add(t, M, Mt, CS, ld, cld, oy, r, -w);
    tile_add(t, M, Mt, CS, ld, cld, oy, s, w);
  }
}

constexpr int kApplyMLg = 11;   // per-CTA delta tables of the apply kernel
constexpr int kApplyCLg = 10;

// apply + commit of one batch on the dense tile, one warp per chunk
// ([c0, c1) of g.chunks); the last CTA to finish runs the batch-end
// bookkeeping
__global__ void __launch_bounds__(kThreads) k_nodal_apply_commit(GraphDev g, int64_t c0, int64_t c1, int32_t* part,
                                                                 const int32_t* __restrict__ move_to,
                                                                 const int32_t* __restrict__ from, int beg, int end,
                                                                 int ld, int* __restrict__ M, int* __restrict__ Mt,
                                                                 int cld, int* __restrict__ CS,
                                                                 int32_t* __restrict__ dout, int32_t* __restrict__ din,
                                                                 NodalCtl* ctl, CtlArgs c) {
  __shared__ int s_mkey[1 << kApplyMLg], s_mval[1 << kApplyMLg];
  __shared__ int s_ckey[1 << kApplyCLg], s_cval[1 << kApplyCLg];
  if (ctl->done) return;   // set only by the last CTA below, after every CTA passed here
  const DeltaTables t{s_mkey, s_mval, s_ckey, s_cval, kApplyMLg, kApplyCLg};
  tables_clear(t);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t nw = static_cast<int64_t>(gridDim.x) * kWarps;
  for (int64_t q = c0 + static_cast<int64_t>(blockIdx.x) * kWarps + (threadIdx.x >> 5); q < c1; q += nw)
    apply_chunk<LdNC, LdPlain>(__ldg(g.chunks + q), g, part, move_to, from, beg, end, t, ld, M, Mt, cld, CS, dout,
                               din, lane);
  tables_flush(t, M, Mt, CS, ld, cld);
  if (c.active) {
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned done_ctas = atomicAdd(&ctl->apply_done, 1u);
      if (done_ctas == gridDim.x - 1) {
        __threadfence();
        ctl_batch_end(ctl, c);
        ctl->apply_done = 0;
      }
    }
  }
}

// commits the batch's moves (degrees, partition) and runs the batch-end
// bookkeeping in one launch (sorted views, which are rebuilt per batch)
__global__ void k_nodal_commit(int32_t* __restrict__ part, int32_t* __restrict__ move_to,
                               const int32_t* __restrict__ kout, const int32_t* __restrict__ kin,
                               int beg, int end, int update_degrees, int32_t* __restrict__ dout,
                               int32_t* __restrict__ din, NodalCtl* ctl, CtlArgs c) {
  if (c.active && blockIdx.x == 0 && threadIdx.x == 0) ctl_batch_end(ctl, c);
  int stride = gridDim.x * blockDim.x;
  for (int v = beg + blockIdx.x * blockDim.x + threadIdx.x; v < end; v += stride) {
    const int s = move_to[v];
    if (s < 0) continue;
    const int r = part[v];
    if (update_degrees) {
      atomicSub(dout + r, kout[v]);
      atomicAdd(dout + s, kout[v]);
      atomicSub(din + r, kin[v]);
      atomicAdd(din + s, kin[v]);
    }
    part[v] = s;
    move_to[v] = -1;
  }
}

__global__ void k_ctl_sweep_start(NodalCtl* ctl, int W, const long long* ide_q,
                                  const int* ide_n) {
  ctl_sweep_start(ctl, W, ide_q, ide_n);
}

// --- persistent nodal phase ----------------------------------------------------
constexpr int kPThreads = 768;    // one CTA per SM (80 registers a thread)
constexpr int kPWarps = kPThreads / 32;
constexpr int kUnitWarp = -2;     // work unit of one vertex of degree <= kHubDegree
constexpr int kPHubLg = 13;
constexpr int kPHubSlots = 1 << kPHubLg;  // hub table slots in shared memory; larger hub tables are global
constexpr int kDeltaGlobalMinB = 256;     // from this B the phase kernel's apply writes straight to global memory
// The proposals of the phase kernel read the tile from shared memory up to
// this B: after a hub table of kSnapSlots slots per array come M and Mt (B x
// ld each, ld = B rounded up to 4), chunk sums and degrees; the rest of the
// hub region stages the cooperative float dS
constexpr int kSnapMaxB = 88;
constexpr int kSnapSlots = 256;   // >= a hub table's capacity for B <= kSnapMaxB (2 * B rounded up to a power of 2)
static_assert(kBatchHubDegree >= 128, "the float dS's terms outgrow a warp's list");
static_assert(kMaxPend == 2 * kPWarps, "a wave's proposals outgrow the list");
static_assert(3 * kSnapSlots + 2 * kSnapMaxB * kSnapMaxB + 3 * kSnapMaxB + 2 * kMaxPend * (4 * 16 + 4) <= 3 * kPHubSlots,
              "chunks of 16 blocks of a full list fit beside the tile copy");
static_assert(2 * kSnapMaxB <= kSnapSlots && kSnapMaxB <= kChunk, "hub tables or chunk sums outgrow the layout");
static_assert(kPHubSlots == 2 * kPhaseHubSlots, "hub regions are assigned for tables beyond this size");
constexpr unsigned long long kBarrierTimeoutNs = 200ull * 1000ull * 1000ull;
// dynamic shared memory: per-warp tables and lists, then the hub table
constexpr size_t kPWarpInts = 3 * kHCap + kHubDegree;
static_assert(kMaxPend <= kMaxSlots && 2 * kMaxSlots * kSlot <= 3 * kPHubSlots,
              "a step of a full list on a sparse tile outgrows the hub region");
constexpr size_t kPSmemBytes = sizeof(int) * (kPWarps * kPWarpInts + 3 * kPHubSlots);

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add64(unsigned long long* p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

constexpr unsigned long long kBarDone = 1ull << 32;   // bits 32..47: done arrivals
constexpr unsigned long long kBarOvf = 1ull << 48;    // bits 48..63: overflow arrivals (mod 2^16)

// Grid-wide barrier of the persistent kernel (all CTAs are co-resident:
// cooperative launch).  ctl->bar counts arrivals over the whole launch in
// its low 32 bits; barrier number k is passed once it reaches
// k * gridDim.x (`target`, advanced here).  After __syncthreads, thread 0
// adds its arrival with release semantics (publishing the CTA's writes)
// and waits with acquire loads.  The arrival may also carry kBarDone or
// kBarOvf, which every CTA then sees in the same load; *s_ovf (if given)
// receives the overflow count.  A wait gives up after kBarrierTimeoutNs and
// sets bar_err.  Returns -1 on error (every CTA then leaves at its next
// barrier), else 1 if kBarDone is set, else 0.
// Wait limit of a grid barrier and the failure-injection switch: a CTA
// with `hold` set never arrives, so every wait of the launch runs out.
struct BarrierOpts {
  unsigned long long timeout_ns = kBarrierTimeoutNs;
  bool hold = false;
};

template <class CtlT>
__device__ __forceinline__ int grid_barrier(CtlT* ctl, unsigned* target, bool publish_done, int* s_state,
                                            bool publish_ovf = false, unsigned* s_ovf = nullptr,
                                            BarrierOpts bo = BarrierOpts{}) {
  *target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    // a CTA told to withhold its arrival (failure injection) still waits,
    // so that every CTA leaves through the timeout below
    if (!bo.hold)
      red_release_add64(&ctl->bar, (publish_done ? 1ull + kBarDone : 1ull) + (publish_ovf ? kBarOvf : 0ull));
    const unsigned long long t0 = global_ns();
    unsigned spins = 0;
    int st;
    for (;;) {
      const unsigned long long v = ld_acquire64(&ctl->bar);
      if (static_cast<unsigned>(v) >= *target) {
        st = ((v >> 32) & 0xffffull) ? 1 : 0;
        if (s_ovf) *s_ovf = static_cast<unsigned>(v >> 48);
        break;
      }
      if ((++spins & 63u) == 0) {
        if (*reinterpret_cast<volatile int*>(&ctl->bar_err)) {
          st = -1;
          break;
        }
        if (global_ns() - t0 > bo.timeout_ns) {
          atomicExch(&ctl->bar_err, 1);
          st = -1;
          break;
        }
      }
    }
    *s_state = st;
  }
  __syncthreads();
  return *s_state;
}

// One stage's nodal phase in one cooperative launch: up to `maxitr` sweeps,
// each an entropy pass, the sweep-start bookkeeping, and for every batch a
// proposal pass (hubs first, one per CTA; then warp-per-vertex, first one
// vertex per warp of the CTAs without a hub, the rest handed out by a
// counter) and an apply pass, during which one thread runs the batch-end
// bookkeeping.  Each CTA applies the moves it accepted itself: the chunks
// of its moved work-unit vertices (listed in shared memory during the
// proposals) and of its moved hubs.  If any CTA's list overflowed (it
// announces that with its barrier arrival, so every CTA learns it from the
// same barrier load), every CTA instead scans all of the batch's edge
// chunks, skipping vertices that did not move.  Tile deltas accumulate per
// CTA as DeltaTables' mode for this B says.  Leaves when the convergence
// test sets `done`.
constexpr int kOwnCap = 1024;   // chunk entries of a CTA's own-move list

// algorithmic bytes of an applied chunk: per edge of a moved vertex its
// neighbour's id and block (8) and the two updated entries of M (16)
__device__ __forceinline__ unsigned long long apply_bytes(const NodalArgs& a, int2 ch) {
  if (__ldcg(a.move_to + ch.x) < 0) return 0;
  const int deg = (__ldg(a.out_ptr + ch.x + 1) - __ldg(a.out_ptr + ch.x)) +
                  (__ldg(a.in_ptr + ch.x + 1) - __ldg(a.in_ptr + ch.x));
  return 24ull * static_cast<unsigned long long>(max(0, min(32, deg - 32 * ch.y)));
}
// --- float dS of a CTA's proposals, evaluated together ---------------------------
// Every proposal needs up to 8 B terms added one after the other: evaluating
// a term takes about 60 issue slots a warp, adding it 4 cycles of one thread's
// dependent latency.  All warps but one evaluate terms, for a chunk of blocks
// of every proposal at a time, into one of two staging areas in shared
// memory, while the last warp, a thread per proposal, adds the chunk before.
// So the additions of up to 32 chains issue together (a warp per chain
// repeats its additions in every lane), the work of a wave is spread over the
// CTA whatever its number of proposals, and a small batch has 23 warps on its
// few.  It is bound by the issue of the evaluating warps; with few proposals
// and a large B by the chain.  A batch of N = 50000 (34 proposals a CTA) took
// 69 us at B = 382 against 143 us with a chain per half-warp, 27 us against
// 35 us at B = 48; one of N = 5000 (8 a CTA) 28 us against 37 us at B = 151.

// the four terms of block i of proposal q, old-state or new-state
template <class Ops>
__device__ __forceinline__ float4 coop_cell(const NodalArgs& a, const Ops& ops, const Pend& q, int i, bool fresh) {
  using LDT = typename Ops::LdT;
  const int r = q.r, s = q.s;
  const bool rs = i == r || i == s;
  const unsigned ro = static_cast<unsigned>(r) * ops.v.ld + i, so = static_cast<unsigned>(s) * ops.v.ld + i;
  if (!fresh && a.Trow)
    return make_float4(__ldcg(a.Trow + ro), __ldcg(a.Trow + so), rs ? 0.0f : __ldcg(a.Tcol + ro),
                       rs ? 0.0f : __ldcg(a.Tcol + so));
  if (fresh && rs) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  int R = LDT::ld(ops.v.M + ro), S = LDT::ld(ops.v.M + so), Rc = 0, Sc = 0;
  if (!rs) {   // columns skip i in {r, s}
    Rc = LDT::ld(ops.v.Mt + ro);
    Sc = LDT::ld(ops.v.Mt + so);
  }
  const float di = ref_factor(LDT::ld(a.din + i)), dn = ref_factor(LDT::ld(a.dout + i));
  const float4 f = fresh ? q.fn : q.fo;
  if (fresh) {   // v's edges towards block i are part of M[r,i] (out) and M[i,r] (in)
    int wo, wi;
    nbr_weights(q, i, &wo, &wi);
    R -= wo;
    S += wo;
    Rc -= wi;
    Sc += wi;
  }
  return make_float4(ref_term_nz(R, di, f.x), ref_term_nz(S, di, f.y), ref_term_nz(Rc, dn, f.z),
                     ref_term_nz(Sc, dn, f.w));
}

// The float dS of the listed proposals, handed to close(q, f) by one thread
// each (CTA-collective).  stage: `room` floats.
template <int NT, class Ops, class CloseFn>
__device__ __forceinline__ void coop_eval(const NodalArgs& a, const Ops& ops, const PendList& pl, float* stage,
                                          int room, CloseFn close) {
  constexpr int NW = NT / 32;
  const int np = pl.n;
  if (np == 0) return;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nc = np > 32 ? 2 : 1;        // warps that add: a proposal per lane
  const int nprod = NT - 32 * nc;        // threads that evaluate
  const bool adds = wib >= NW - nc;
  const int mine = (wib - (NW - nc)) * 32 + lane;
  // chunks of CB blocks, equal shares of B: at most about four
  // cells per evaluating thread, so that the last chunk's additions, which
  // overlap nothing, stay short, and both buffers within the room.  (A row of
  // the staging area is an odd number of 16-byte words: no bank conflicts
  // among the adding lanes.)
  const int most = max(8, min(4 * nprod / np, (room / (8 * np) - 1) & ~1));
  const int B = a.B, nch = (B + most - 1) / most;
  const int CB = ((B + nch - 1) / nch + 1) & ~1, stride = 4 * CB + 4;
  float dS = 0.0f, c0 = 0.0f, c1 = 0.0f, c2 = 0.0f, c3 = 0.0f;
  const bool has = adds && mine < np;
  if (has) corner_terms(pl.p[mine], &c0, &c1, &c2, &c3);   // due between the passes
  const int ks = threadIdx.x / CB, os = threadIdx.x - ks * CB;
  const int dk = nprod / CB, dr = nprod - dk * CB;   // from one of a thread's cells to its next
  for (int t = 0; t <= 2 * nch; t++) {
    if (!adds) {
      if (t < 2 * nch) {
        const bool fresh = t >= nch;
        const int b0 = (fresh ? t - nch : t) * CB;
        float* st = stage + (t & 1) * np * stride;
        int k = ks, o = os;
        while (k < np) {
          if (b0 + o < B)
            *reinterpret_cast<float4*>(st + k * stride + 4 * o) = coop_cell(a, ops, pl.p[k], b0 + o, fresh);
          k += dk;
          o += dr;
          if (o >= CB) {
            o -= CB;
            k++;
          }
        }
      }
    } else if (has && t > 0) {
      const bool fresh = t > nch;
      const int b0 = (fresh ? t - 1 - nch : t - 1) * CB;
      const int n = min(CB, B - b0);
      const float4* st = reinterpret_cast<const float4*>(stage + ((t - 1) & 1) * np * stride + mine * stride);
      if (!fresh) {
#pragma unroll 8
        for (int j = 0; j < n; j++) {
          const float4 q = st[j];
          dS = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(dS, q.x), q.y), q.z), q.w);
        }
      } else {
        if (t == nch + 1) dS = __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(dS, c0), c1), c2), c3);
#pragma unroll 8
        for (int j = 0; j < n; j++) {
          const float4 q = st[j];
          dS = __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(dS, q.x), q.y), q.z), q.w);
        }
      }
    }
    __syncthreads();
  }
  if (has) close(pl.p[mine], dS);
}

// The same on a tile with many empty cells.  A warp takes a proposal's 64
// blocks at a time: it packs the non-zero cells of the four rows, in the
// chain's order, into a slot of the staging area, and its lanes then replace
// each packed cell by its term, so an empty cell costs a compare instead of
// a term and an addition.  A packed cell holds the count (below 2^24) under
// its number among the 256; the block's degree comes from the lane that
// loaded it.  The loads of a warp's next 64 blocks are issued before it works
// on these.  Bound by the issue of the scan (about 400 slots for 64 blocks).
// N = 4999, B = 2500 (1.3% of the cells filled): 53 us a batch against 241 us
// with whole rows evaluated; N = 50000, B = 3052 (8%): 468 against 941 us.
struct SlotCounts {
  int n[2][kMaxSlots];
};

template <int NT, class Ops, class CloseFn>
__device__ __forceinline__ void coop_eval_sparse(const NodalArgs& a, const Ops& ops, const PendList& pl, float* stage,
                                                 int room, SlotCounts* sc, CloseFn close) {
  constexpr int NW = NT / 32;
  const int np = pl.n;
  if (np == 0) return;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nc = np > 32 ? 2 : 1;
  const int pw = NW - nc;
  const bool adds = wib >= pw;
  const int mine = (wib - pw) * 32 + lane;
  const int B = a.B, nch = (B + 63) >> 6;
  // m chunks of every proposal per step, in two sets of np * m slots
  const int m = min(nch, max(1, min(kMaxSlots, room / (2 * kSlot)) / np));
  const int nst = (nch + m - 1) / m, per = np * m;
  float dS = 0.0f, c0 = 0.0f, c1 = 0.0f, c2 = 0.0f, c3 = 0.0f;
  const bool has = adds && mine < np;
  if (has) corner_terms(pl.p[mine], &c0, &c1, &c2, &c3);
  // a warp's items of a step: slots wib, wib + pw, wib + 2 pw (< per); slot
  // x is chunk x / np of the step, proposal x % np
  int2 nx[6];
  auto load = [&](int t, int k, int c) {
#pragma unroll
    for (int j = 0; j < 6; j++) nx[j] = make_int2(0, 0);
    if (t >= 2 * nst) return;
    const Pend& q = pl.p[k];
    const int i = (((t >= nst ? t - nst : t) * m + c) << 6) + 2 * lane;
    if (i >= B) return;
    // (rows and degree arrays are readable up to an even number of blocks)
    const unsigned r = static_cast<unsigned>(q.r) * ops.v.ld + i, s = static_cast<unsigned>(q.s) * ops.v.ld + i;
    nx[0] = __ldcg(reinterpret_cast<const int2*>(ops.v.M + r));
    nx[1] = __ldcg(reinterpret_cast<const int2*>(ops.v.M + s));
    nx[2] = __ldcg(reinterpret_cast<const int2*>(ops.v.Mt + r));
    nx[3] = __ldcg(reinterpret_cast<const int2*>(ops.v.Mt + s));
    nx[4] = __ldcg(reinterpret_cast<const int2*>(a.din + i));
    nx[5] = __ldcg(reinterpret_cast<const int2*>(a.dout + i));
  };
  const unsigned lanes_below = (1u << lane) - 1u;
  const int k0 = wib % np, step_k = pw % np, c0x = wib / np, step_c = pw / np;
  if (!adds && wib < per) load(0, k0, c0x);
  for (int t = 0; t <= 2 * nst; t++) {
    if (!adds) {
      if (t < 2 * nst) {
        const bool fresh = t >= nst;
        int k1 = k0, c1 = c0x;
        for (int x = wib; x < per; x += pw) {
          const int kx = k1, cx = c1;
          const Pend& q = pl.p[kx];
          const int i = (((fresh ? t - nst : t) * m + cx) << 6) + 2 * lane;
          int c[8] = {nx[0].x, nx[1].x, nx[2].x, nx[3].x, nx[0].y, nx[1].y, nx[2].y, nx[3].y};
          const int di0 = nx[4].x, di1 = nx[4].y, dn0 = nx[5].x, dn1 = nx[5].y;
          k1 += step_k;
          c1 += step_c;
          if (k1 >= np) {
            k1 -= np;
            c1++;
          }
          if (x + pw < per) load(t, k1, c1);
          else load(t + 1, k0, c0x);
          if (!__any_sync(0xffffffffu, (c[0] | c[1] | c[2] | c[3] | c[4] | c[5] | c[6] | c[7]) != 0)) {
            if (lane == 0) sc->n[t & 1][x] = 0;
            continue;
          }
          const int r = q.r, s = q.s;
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const bool rs = i + k == r || i + k == s;   // columns (new: rows too) skip blocks r and s
            if (rs) c[4 * k + 2] = c[4 * k + 3] = 0;
            if (fresh) {
              if (rs) c[4 * k] = c[4 * k + 1] = 0;
              // v's edges towards block i are part of M[r,i] (out) and M[i,r] (in)
              if ((c[4 * k] | c[4 * k + 2]) != 0) {
                int wo, wi;
                nbr_weights(q, i + k, &wo, &wi);
                c[4 * k] -= wo;
                c[4 * k + 1] += wo;
                c[4 * k + 2] -= wi;
                c[4 * k + 3] += wi;
              }
            }
          }
          int total = 0, at = 0;   // non-zero cells in all, and in the lanes below
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const unsigned nz = __ballot_sync(0xffffffffu, c[k] != 0);
            total += __popc(nz);
            at += __popc(nz & lanes_below);
          }
          // a slot's 16-byte words are permuted by the proposal's number, so
          // that the adding lanes, at the same place of their slots, read
          // different banks
          int* slot = reinterpret_cast<int*>(stage) + ((t & 1) * per + x) * kSlot;
          const int sw = (kx & 7) << 2;
          {
#pragma unroll
            for (int k = 0; k < 8; k++)
              if (c[k]) slot[at++ ^ sw] = c[k] | static_cast<int>(static_cast<unsigned>(8 * lane + k) << 24);
          }
          __syncwarp();
          const float4 ff = fresh ? q.fn : q.fo;
          for (int e0 = 0; e0 < total; e0 += 32) {
            const int e = e0 + lane;
            const unsigned w = e < total ? slot[e ^ sw] : 0u;
            const int from = w >> 27, k = (w >> 24) & 7, j = k & 3;   // lane, cell of the lane, row
            const int a0 = __shfl_sync(0xffffffffu, di0, from), a1 = __shfl_sync(0xffffffffu, di1, from);
            const int b0 = __shfl_sync(0xffffffffu, dn0, from), b1 = __shfl_sync(0xffffffffu, dn1, from);
            const int d = (j & 2) ? ((k & 4) ? b1 : b0) : ((k & 4) ? a1 : a0);
            const float fa = (j & 1) ? ff.y : ff.x, fb = (j & 1) ? ff.w : ff.z;
            const float term = ref_term_nz(static_cast<int>(w & 0xffffffu), ref_factor(d), (j & 2) ? fb : fa);
            if (e < ((total + 3) & ~3)) slot[e ^ sw] = __float_as_int(term);   // zeros up to a multiple of 4
          }
          if (lane == 0) sc->n[t & 1][x] = total;
        }
      }
    } else if (has && t > 0) {
      const bool fresh = t > nst;
      if (t == nst + 1) dS = __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(dS, c0), c1), c2), c3);
      const int sw = mine & 7;
      for (int x = mine; x < per; x += np) {
        const int n = (sc->n[(t - 1) & 1][x] + 3) >> 2;
        const float4* st = reinterpret_cast<const float4*>(stage + (((t - 1) & 1) * per + x) * kSlot);
        if (!fresh) {
#pragma unroll 4
          for (int j = 0; j < n; j++) {
            const float4 q = st[j ^ sw];
            dS = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(dS, q.x), q.y), q.z), q.w);
          }
        } else {
#pragma unroll 4
          for (int j = 0; j < n; j++) {
            const float4 q = st[j ^ sw];
            dS = __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(dS, q.x), q.y), q.z), q.w);
          }
        }
      }
    }
    __syncthreads();
  }
  if (has) close(pl.p[mine], dS);
}

// One work unit of the persistent kernels: two vertices of degree <= 64
// (a half-warp each; un.y = -1 when there is only one) or one vertex
// (the whole warp, un.y = kUnitWarp).  wtab: the warp's shared-memory
// tables.  In precision 3 the proposals go to `pl`.
template <class Ops>
__device__ __forceinline__ void unit_vertices(const NodalArgs& a, const Ops& ops, int2 un, uint32_t itr, int* wtab,
                                              CtaTally* tl, int lane, unsigned long long* my_bytes, PendList* pl) {
  int* list = wtab + 3 * kHCap;
  if (un.y == kUnitWarp) {
    group_vertex<kHubDegree / 32>(a, ops, un.x, itr, wtab, list, tl, Grp<32>(lane), my_bytes, nullptr, pl);
  } else {
    const int h = lane >> 4;
    const int vv = h ? un.y : un.x;
    if (vv >= 0)
      group_vertex<kPairDegree / 16>(a, ops, vv, itr, wtab + h * (3 * kHCap / 2), list + h * kPairDegree, tl,
                                     Grp<16>(lane), my_bytes, nullptr, pl);
  }
  __syncwarp();
}

// item x of the two tables of `cells` cells each
__device__ __forceinline__ void ref32_table_cell(unsigned x, unsigned cells, int B, int ld, const int* M, const int* Mt,
                                                 const int32_t* din, const int32_t* dout, float* Trow, float* Tcol) {
  const bool col = x >= cells;
  const unsigned c = col ? x - cells : x;
  const unsigned b = c / ld, i = c - b * ld;
  float t = 0.0f;
  if (i < static_cast<unsigned>(B)) {
    const int m = __ldcg((col ? Mt : M) + c);
    t = ref_term_nz(m, ref_factor(__ldcg((col ? dout : din) + i)), ref_factor(__ldcg((col ? din : dout) + b)));
  }
  __stcg((col ? Tcol : Trow) + c, t);
}

// Precision mode 3: the reference's old-state dS terms of every tile cell
// for the batch about to be proposed (grid-collective; they depend on the
// cell and its blocks' degrees only, not on the proposing vertex):
//   Trow[b, i] = M[b,i] log(M[b,i] / (d_in[i] d_out[b]))
//   Tcol[b, i] = M[i,b] log(M[i,b] / (d_out[i] d_in[b]))
// in the reference's float arithmetic (ref_term), 0 for empty cells.
__device__ __forceinline__ void ref32_tables_pass(int B, int ld, const int* M, const int* Mt, const int32_t* din,
                                                  const int32_t* dout, float* Trow, float* Tcol) {
  const unsigned cells = static_cast<unsigned>(B) * ld;   // (the tables serve B <= 16384)
  for (unsigned x = blockIdx.x * blockDim.x + threadIdx.x; x < 2 * cells; x += gridDim.x * blockDim.x)
    ref32_table_cell(x, cells, B, ld, M, Mt, din, dout, Trow, Tcol);
}

template <int P, bool kSnap>
__global__ void __launch_bounds__(kPThreads, 1) k_nodal_phase(PhaseArgs p) {
  extern __shared__ __align__(16) int dyn[];
  __shared__ CtaTally s_tally;
  __shared__ HubShared<kPWarps> sh;
  __shared__ int s_base, s_state;
  __shared__ unsigned s_ovf;
  __shared__ int2 s_own[kOwnCap];
  __shared__ int s_nown;
  __shared__ PendList s_pl;
  __shared__ SlotCounts s_sc;
  using Ops = DenseOpsT<LdCG, P, std::conditional_t<kSnap, LdPlain, LdCG>>;
  NodalCtl* ctl = p.a.ctl;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int gw = blockIdx.x * kPWarps + wib;
  const int nw = gridDim.x * kPWarps;
  int* wtab = dyn + wib * kPWarpInts;
  int* htab = dyn + kPWarps * kPWarpInts;   // hub region: hub tables and staging during proposals, delta tables during apply
  int* hubtab = htab + 3 * kPhaseHubSlots;  // its second half: a hub's table
  // kSnap (B <= kSnapMaxB): the proposals read M, Mt, the chunk sums and the
  // block degrees from a copy in shared memory, taken at every batch start;
  // it shares the hub table's region (a hub's table then needs at most
  // kSnapSlots slots per array)
  int* sM = htab + 3 * kSnapSlots;
  int* sMt = sM + p.a.B * p.v.ld;
  int* sCS = sMt + p.a.B * p.v.ld;
  int* sdin = sCS + p.a.B;
  int* sdout = sdin + p.a.B;
  const int snap_ints = 3 * kSnapSlots + 2 * p.a.B * p.v.ld + ((3 * p.a.B + 3) & ~3);   // a multiple of 4
  DenseView vs = p.v;
  if (kSnap) {
    vs.M = sM;
    vs.Mt = sMt;
    vs.CS = sCS;
  }
  const Ops ops{vs, p.a.B};
  BarrierOpts bo;
  bo.timeout_ns = p.bar_timeout_ns ? p.bar_timeout_ns : kBarrierTimeoutNs;
  bo.hold = static_cast<int>(blockIdx.x) == p.bar_hold;
  // dense deltas in the first 2 * kPHubSlots ints, chunk-sum deltas (B <= 128: B entries) after them
  const int mode = p.a.B >= kDeltaGlobalMinB ? kDeltaGlobal
                   : (p.a.B * p.a.B <= 2 * kPHubSlots ? kDeltaDense : kDeltaHashed);
  const DeltaTables dt{htab, htab + kPHubSlots, htab + 2 * kPHubSlots, htab + 2 * kPHubSlots + kPHubSlots / 2,
                       kPHubLg, kPHubLg - 1, mode, p.a.B};
  const int B = p.a.B;
  unsigned ovf_seen = 0;   // overflow count at the previous proposal barrier
  const int64_t cells = static_cast<int64_t>(B) * B;
  unsigned target = 0;
  unsigned long long my_bytes = 0;
  bool converged = false;
  if constexpr (P == 3) ref_tab_fill();   // (grid barriers lie before its first use)
  for (int sw = 0; sw < p.maxitr; sw++) {
    // data term of S for this sweep (the entropy kernel's sum)
    {
      long long acc = 0;
      unsigned long long seen = 0, nz = 0;
      for (int64_t c = static_cast<int64_t>(blockIdx.x) * kPThreads + threadIdx.x; c < cells;
           c += static_cast<int64_t>(gridDim.x) * kPThreads) {
        const int i = static_cast<int>(c / B), j = static_cast<int>(c - static_cast<int64_t>(i) * B);
        const int m = __ldcg(p.v.M + static_cast<int64_t>(i) * p.v.ld + j);
        seen++;
        if (m) {
          nz++;
          acc += q32(g_term(p.a.L, m, __ldcg(p.din + j), __ldcg(p.dout + i)));
        }
      }
      // algorithmic bytes: every cell of the tile, two degrees per nonzero
      if (p.a.stats) my_bytes += 4 * seen + 8 * nz;
      acc = warp_sum_ll(acc);
      if (lane == 0 && acc) atomicAdd(&ctl->entropy_acc, static_cast<unsigned long long>(acc));
    }
    if (grid_barrier(ctl, &target, false, &s_state, false, nullptr, bo) < 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctl_sweep_start(ctl, p.W, p.ide_q, p.ide_n);
      ctl->entropy_acc = 0;
    }
    if (grid_barrier(ctl, &target, false, &s_state, false, nullptr, bo) < 0) return;
    const uint32_t itr = static_cast<uint32_t>(sw);   // ctl->sweeps before this sweep started
    for (int bi = 0; bi * p.bs < p.n; bi++) {
      NodalArgs a = p.a;
      a.beg = bi * p.bs;
      a.end = a.beg + p.bs < p.n ? a.beg + p.bs : p.n;
      const int count = a.end - a.beg;
      if constexpr (P == 3) {
        if (p.a.Trow) {   // the batch's old-state terms, before anyone proposes
          ref32_tables_pass(B, p.a.tld, p.v.M, p.v.Mt, p.din, p.dout, p.a.Trow, p.a.Tcol);
          if (grid_barrier(ctl, &target, false, &s_state, false, nullptr, bo) < 0) return;
        }
      }
      if (kSnap) {
        // the tile as the previous batch left it (rows padded to ld with
        // zeros; cld = 1)
        const int n4 = B * p.v.ld / 4;
        for (int i = threadIdx.x; i < n4; i += kPThreads) {
          reinterpret_cast<int4*>(sM)[i] = __ldcg(reinterpret_cast<const int4*>(p.v.M) + i);
          reinterpret_cast<int4*>(sMt)[i] = __ldcg(reinterpret_cast<const int4*>(p.v.Mt) + i);
        }
        for (int i = threadIdx.x; i < B; i += kPThreads) {
          sCS[i] = __ldcg(p.v.CS + i);
          sdin[i] = __ldcg(p.din + i);
          sdout[i] = __ldcg(p.dout + i);
        }
        a.din = sdin;
        a.dout = sdout;
        __syncthreads();
      }
      // proposals
      if (threadIdx.x == 0) {
        s_tally = CtaTally{0, 0, 0, 0};
        s_tally.own = s_own;
        s_tally.nown = &s_nown;
        s_tally.own_cap = kOwnCap;
        s_nown = 0;
        s_pl.n = 0;
      }
      __syncthreads();
      const int hub_lo = __ldg(p.batch_hub + bi);
      const int hub_hi = P == 3 && p.a.hub_units ? hub_lo : __ldg(p.batch_hub + bi + 1);   // proposed by CTAs
      const int hcta = min(hub_hi - hub_lo, static_cast<int>(gridDim.x));
      // work units: two vertices of degree <= 64 (a half-warp each) or one
      // vertex (a warp)
      const int u_lo = __ldg(p.unit_ptr + bi), nun = __ldg(p.unit_ptr + bi + 1) - u_lo;
      const int extra = P == 3 && p.a.hub_units ? __ldg(p.batch_hub + bi + 1) - hub_lo : 0;   // hubs as units
      const int first = (gridDim.x - hcta) * kPWarps;   // units handed out without the counter
      // waves of proposals: the CTA's hubs, one each; then one unit per warp,
      // dealt in turn to the CTAs without a hub; then, where units are left,
      // kPWarps per step of a counter
      int h = hub_lo + blockIdx.x;
      for (bool dealt = false;;) {
        int taken = 0;   // ints at the end of the hub region that hold a hub's table
        if (h < hub_hi) {
          hub_vertex<Ops, kPThreads>(a, ops, __ldg(p.hubs + h), itr, kSnap ? htab : hubtab,
                                     kSnap ? kSnapSlots : kPhaseHubSlots, &sh, &my_bytes, nullptr, &s_pl);
          if (P == 3 && !kSnap && s_pl.p[0].cap <= kPhaseHubSlots) taken = 3 * s_pl.p[0].cap;
          h += gridDim.x;
        } else {
          int i = nun + extra;
          if (!dealt) {
            dealt = true;
            if (static_cast<int>(blockIdx.x) >= hcta) i = wib * (gridDim.x - hcta) + (blockIdx.x - hcta);
          } else {
            if (first >= nun + extra) break;
            __syncthreads();
            if (threadIdx.x == 0) s_base = first + static_cast<int>(atomicAdd(&ctl->vnext, static_cast<unsigned>(kPWarps)));
            __syncthreads();
            if (s_base >= nun + extra) break;
            i = s_base + wib;
          }
          if (i < nun + extra) {
            const int2 un = i < nun ? __ldg(p.units + u_lo + i) : make_int2(__ldg(p.hubs + hub_lo + i - nun), kUnitWarp);
            unit_vertices(a, ops, un, itr, wtab, &s_tally, lane, &my_bytes, &s_pl);
          }
        }
        if constexpr (P == 3) {   // the float dS of the wave's proposals
          __syncthreads();
          float* stage = reinterpret_cast<float*>(htab + (kSnap ? snap_ints : 0));
          const int room = 3 * kPHubSlots - (kSnap ? snap_ints : 0) - taken;
          const auto close = [&](const Pend& q, float f) { close_vertex<Ops>(a, q, f, &s_tally, &my_bytes); };
          if (!kSnap && a.sparse) coop_eval_sparse<kPThreads>(a, ops, s_pl, stage, room, &s_sc, close);
          else coop_eval<kPThreads>(a, ops, s_pl, stage, room, close);
          __syncthreads();
          if (threadIdx.x == 0) s_pl.n = 0;
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) tally_flush(&s_tally, ctl);
      const int nown = s_nown;
      if (grid_barrier(ctl, &target, false, &s_state, nown > kOwnCap, &s_ovf, bo) < 0) return;
      // every CTA reads the same count here: the next overflow arrivals come
      // after the next proposal pass, which no CTA starts before all passed
      // the apply barrier below
      const bool scan_all = s_ovf != ovf_seen;
      ovf_seen = s_ovf;
      if (dt.mode == kDeltaDense) dense_clear(dt, p.v.cld);
      else if (dt.mode == kDeltaHashed) tables_clear(dt);
      // apply + commit; one thread closes the batch meanwhile
      bool done = false;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        const long long edges = (static_cast<long long>(__ldg(p.a.out_ptr + a.end)) - __ldg(p.a.out_ptr + a.beg)) +
                                (static_cast<long long>(__ldg(p.a.in_ptr + a.end)) - __ldg(p.a.in_ptr + a.beg));
        const CtlArgs ca{1, p.W, p.thr, p.model_d, p.ide_q, p.ide_n, count, edges};
        done = ctl_batch_end(ctl, ca);
        ctl->vnext = 0;
        if (scan_all) ctl->apply_scans++;
      }
      __syncthreads();
      {
        // own moves (chunk k of the CTA's list), or every chunk of the batch
        const int64_t cb = scan_all ? __ldg(p.chunk_ptr + a.beg) : 0;
        const int64_t k1 = scan_all ? __ldg(p.chunk_ptr + a.end) : nown;
        const int step = scan_all ? nw : kPWarps;
        for (int64_t k = (scan_all ? cb + gw : wib); k < k1; k += step) {
          const int2 ch = scan_all ? __ldg(p.g.chunks + k) : s_own[k];
          apply_chunk<LdCG, LdCG>(ch, p.g, p.part, a.move_to, a.from, a.beg, a.end, dt, p.v.ld, p.M, p.Mt,
                                  p.v.cld, p.CS, p.dout, p.din, lane);
          if (p.a.stats && lane == 0) my_bytes += apply_bytes(p.a, ch);
        }
      }
      // the CTA's moved hubs, whose chunks are not listed
      for (int h = hub_lo + blockIdx.x; !scan_all && h < hub_hi; h += gridDim.x) {
        const int v = __ldg(p.hubs + h);
        if (__ldcg(a.move_to + v) < 0) continue;   // CTA-uniform
        const int64_t q1 = __ldg(p.chunk_ptr + v + 1);
        for (int64_t q = __ldg(p.chunk_ptr + v) + wib; q < q1; q += kPWarps) {
          const int2 ch = __ldg(p.g.chunks + q);
          apply_chunk<LdCG, LdCG>(ch, p.g, p.part, a.move_to, a.from, a.beg, a.end, dt, p.v.ld, p.M, p.Mt,
                                  p.v.cld, p.CS, p.dout, p.din, lane);
          if (p.a.stats && lane == 0) my_bytes += apply_bytes(p.a, ch);
        }
      }
      if (dt.mode == kDeltaDense) dense_flush(dt, p.M, p.Mt, p.CS, p.v.ld, p.v.cld);
      else if (dt.mode == kDeltaHashed) tables_flush(dt, p.M, p.Mt, p.CS, p.v.ld, p.v.cld);
      const int st = grid_barrier(ctl, &target, done, &s_state, false, nullptr, bo);
      if (st < 0) return;   // a barrier failed
      if (st > 0) {         // converged
        converged = true;
        break;
      }
    }
    if (converged) break;
  }
  // the data term of the final state (the stage's description length),
  // read by the host with the control block; entropy_acc was cleared at
  // the last sweep start
  {
    long long acc = 0;
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * kPThreads + threadIdx.x; c < cells;
         c += static_cast<int64_t>(gridDim.x) * kPThreads) {
      const int i = static_cast<int>(c / B), j = static_cast<int>(c - static_cast<int64_t>(i) * B);
      const int m = __ldcg(p.v.M + static_cast<int64_t>(i) * p.v.ld + j);
      if (m) acc += q32(g_term(p.a.L, m, __ldcg(p.din + j), __ldcg(p.dout + i)));
    }
    acc = warp_sum_ll(acc);
    if (lane == 0 && acc) atomicAdd(&ctl->entropy_acc, static_cast<unsigned long long>(acc));
  }
  if (p.a.stats && my_bytes) atomicAdd(&ctl->bytes, my_bytes);
}

// the hub CTAs run on a second stream, concurrently with the warp kernel
template <class Ops>
void launch_propose(const NodalArgs& a, Ops ops, const HubList& hubs, const StreamPair& sp) {
  const int count = a.end - a.beg;
  if (count <= 0) return;
  const bool has_hubs = hubs.hi > hubs.lo;
  const bool fork = has_hubs && sp.side != sp.main;   // hubs overlap the warp kernel on the side stream
  if (fork) {
    USAP_CUDA(cudaEventRecord(sp.fork, sp.main));
    USAP_CUDA(cudaStreamWaitEvent(sp.side, sp.fork, 0));
  }
  if (has_hubs) {
    const size_t smem = sizeof(int) * 3 * static_cast<size_t>(hubs.smem_cap);
    k_nodal_propose_hub<Ops><<<hubs.hi - hubs.lo, kHubThreads, smem, sp.side>>>(a, ops, hubs.ids, hubs.lo,
                                                                                hubs.hi, hubs.smem_cap);
    USAP_LAUNCHED();
  }
  int blocks = (count + kWarps - 1) / kWarps;
  if (blocks > 148 * 8) blocks = 148 * 8;
  k_nodal_propose<Ops><<<blocks, kThreads, 0, sp.main>>>(a, ops);
  USAP_LAUNCHED();
  if (fork) {
    USAP_CUDA(cudaEventRecord(sp.join, sp.side));
    USAP_CUDA(cudaStreamWaitEvent(sp.main, sp.join, 0));
  }
}

}  // namespace

namespace {
int g_phase_grid[64];
}

// dynamic shared memory limits, set once per device, and the grid of the
// persistent kernel (CTAs per SM that fit x SMs; 0 if the device cannot
// run it cooperatively)
void nodal_configure(int device) {
  static std::once_flag once[64];
  if (device < 0 || device >= 64) return;
  std::call_once(once[device], [device] {
    const int smem = static_cast<int>(sizeof(int) * 3 * kHubSmemSlots);
    const int psmem = static_cast<int>(kPSmemBytes);
    int coop = 0, sms = 0;
    USAP_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
    USAP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    // one grid for every precision mode: the fewest co-resident CTAs
    int per_phase = 1 << 30;
    auto configure = [&](auto tag) {
      constexpr int P = decltype(tag)::value;
      USAP_CUDA(cudaFuncSetAttribute(k_nodal_propose_hub<DenseOpsT<LdNC, P>>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      USAP_CUDA(cudaFuncSetAttribute(k_nodal_propose_hub<SortedOpsT<P>>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      USAP_CUDA(cudaFuncSetAttribute(k_nodal_phase<P, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, psmem));
      USAP_CUDA(cudaFuncSetAttribute(k_nodal_phase<P, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, psmem));
      int a = 0, a2 = 0;
      USAP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_nodal_phase<P, false>, kPThreads, kPSmemBytes));
      USAP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a2, k_nodal_phase<P, true>, kPThreads, kPSmemBytes));
      per_phase = std::min(per_phase, std::min(a, a2));
    };
    configure(std::integral_constant<int, 0>{});
    configure(std::integral_constant<int, 1>{});
    configure(std::integral_constant<int, 2>{});
    configure(std::integral_constant<int, 3>{});
    g_phase_grid[device] = coop ? per_phase * sms : 0;
  });
}

int nodal_phase_grid(int device) {
  if (device < 0 || device >= 64) return 0;
  nodal_configure(device);
  return g_phase_grid[device];
}

// The line: per 64 blocks packing costs what it saves when about a fifth of
// the cells are filled (batches of N = 20000 at B = 1227, e = 0.2 cells: 91 us
// packed, 87 us whole; N = 50000 at B = 1526, 0.33: 385 against 294 us; N = 4999
// at B = 625, 0.2: 26 against 33 us).
bool float_ds_sparse(int64_t e, int32_t B) { return B > kSnapMaxB && 5 * e < static_cast<int64_t>(B) * B; }

int nodal_phase_warps() { return kPWarps; }

// the apply pass keys a tile cell as x * ld + y in 31 bits
int nodal_phase_max_blocks() { return 32768; }

// the cooperative kernel of precision mode `prec` (0, 1, 2, 3);
// snap: the variant that copies the tile into shared memory (B <= kSnapMaxB)
static const void* phase_kernel(int prec, bool snap) {
  if (snap) {
    if (prec == 1) return reinterpret_cast<const void*>(k_nodal_phase<1, true>);
    if (prec == 2) return reinterpret_cast<const void*>(k_nodal_phase<2, true>);
    if (prec == 3) return reinterpret_cast<const void*>(k_nodal_phase<3, true>);
    return reinterpret_cast<const void*>(k_nodal_phase<0, true>);
  }
  if (prec == 1) return reinterpret_cast<const void*>(k_nodal_phase<1, false>);
  if (prec == 2) return reinterpret_cast<const void*>(k_nodal_phase<2, false>);
  if (prec == 3) return reinterpret_cast<const void*>(k_nodal_phase<3, false>);
  return reinterpret_cast<const void*>(k_nodal_phase<0, false>);
}

void launch_nodal_phase(const PhaseArgs& p, int grid, cudaStream_t st) {
  PhaseArgs args = p;
  void* kargs[] = {&args};
  const void* fn = phase_kernel(p.a.prec, p.a.B <= kSnapMaxB);
  USAP_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kPThreads), kargs, kPSmemBytes, st));
  USAP_LAUNCHED();
}

void launch_nodal_propose_dense(const NodalArgs& a, DenseView v, const HubList& hubs,
                                const StreamPair& sp) {
  if (a.prec == 1) launch_propose(a, DenseOpsT<LdNC, 1>{v, a.B}, hubs, sp);
  else if (a.prec == 2) launch_propose(a, DenseOpsT<LdNC, 2>{v, a.B}, hubs, sp);
  else if (a.prec == 3) launch_propose(a, DenseOpsT<LdNC, 3>{v, a.B}, hubs, sp);
  else launch_propose(a, DenseOps{v, a.B}, hubs, sp);
}

void launch_nodal_propose_sorted(const NodalArgs& a, SortedView v, const HubList& hubs,
                                 const StreamPair& sp) {
  if (a.prec == 1) launch_propose(a, SortedOpsT<1>{v, a.B}, hubs, sp);
  else if (a.prec == 2) launch_propose(a, SortedOpsT<2>{v, a.B}, hubs, sp);
  else if (a.prec == 3) launch_propose(a, SortedOpsT<3>{v, a.B}, hubs, sp);
  else launch_propose(a, SortedOps{v, a.B}, hubs, sp);
}

void launch_merge_propose_dense(DenseView v, const MergeArgs& a, cudaStream_t st) {
  long long items = static_cast<long long>(a.B) * a.K;
  long long blocks = (items + kWarps - 1) / kWarps;
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  if (a.prec == 1) k_merge_propose_dense<1><<<static_cast<int>(blocks), kThreads, 0, st>>>(v, a);
  else if (a.prec == 2) k_merge_propose_dense<2><<<static_cast<int>(blocks), kThreads, 0, st>>>(v, a);
  else k_merge_propose_dense<0><<<static_cast<int>(blocks), kThreads, 0, st>>>(v, a);
  USAP_LAUNCHED();
}

void launch_chunk_sums(int B, DenseView v, int* CS, cudaStream_t st) {
  const int nch = (B + kChunk - 1) / kChunk;
  long long items = static_cast<long long>(B) * nch;
  long long blocks = (items + kWarps - 1) / kWarps;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) blocks = 1;
  k_chunk_sums<<<static_cast<int>(blocks), kThreads, 0, st>>>(B, v.ld, v.M, v.Mt, v.cld, CS);
  USAP_LAUNCHED();
}

void launch_nodal_apply_commit_dense(const GraphDev& g, int32_t* part, const int32_t* move_to,
                                     const int32_t* from, int beg, int end, int64_t c0, int64_t c1,
                                     int ld, int* M, int* Mt, int cld, int* CS, int32_t* dout,
                                     int32_t* din, NodalCtl* ctl, const CtlArgs& c, cudaStream_t st) {
  const int64_t items = c1 - c0;
  if (items <= 0) return;
  int64_t blocks = (items + kWarps - 1) / kWarps;
  if (blocks > 148 * 8) blocks = 148 * 8;
  k_nodal_apply_commit<<<static_cast<int>(blocks), kThreads, 0, st>>>(g, c0, c1, part, move_to, from, beg, end, ld,
                                                                      M, Mt, cld, CS, dout, din, ctl, c);
  USAP_LAUNCHED();
}

void launch_nodal_commit(const GraphDev& g, int32_t* part, int32_t* move_to, int beg, int end,
                         int update_degrees, int32_t* dout, int32_t* din, NodalCtl* ctl,
                         const CtlArgs& c, cudaStream_t st) {
  int count = end - beg;
  int blocks = (count + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  k_nodal_commit<<<blocks, 256, 0, st>>>(part, move_to, g.kout, g.kin, beg, end, update_degrees, dout,
                                         din, ctl, c);
  USAP_LAUNCHED();
}

void launch_ctl_sweep_start(NodalCtl* ctl, int W, const long long* ide_q,
                            const int* ide_n, cudaStream_t st) {
  k_ctl_sweep_start<<<1, 1, 0, st>>>(ctl, W, ide_q, ide_n);
  USAP_LAUNCHED();
}


}  // namespace usap
