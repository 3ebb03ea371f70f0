// K4: chained supernodal triangular solves through all diurnal bins in one
// persistent launch.
//
// Replaces the reference's eight sequential lu.solve calls per monodromy
// application (apply_monodromy, orbit/core/orbit.py:99-107; compute_s,
// orbit.py:110-120; the recovery sweep orbit.py:188-193) and their
// transposed twins (orbit/core/orbit_adjoint.py:36-67, 127-134).
//
// Work is a static list of tasks (bin, supernode, row chunk, orbit), ordered
// bin by bin: the forward sweep from the leaves to the root, then the
// backward sweep from the root to the leaves.  CTAs claim tasks in that order
// from an atomic counter and wait (bounded spin, acquire loads) only on the
// per-supernode completion counters of the tasks a task reads from: its
// children's update vectors, the previous bin's solution on its own rows, or
// its parent's backward result.  Since every dependency precedes its
// dependant in claim order and the grid is sized to be co-resident, the
// earliest unfinished task can always run.  A wait that exceeds its
// iteration limit sets ORBIT_ERR_TIMEOUT in the status word and every CTA
// leaves the loop.
//
// Ordering: a task's results are written by all its threads, then a block
// barrier, then one thread's red.release.gpu on the completion counter; the
// consumer's thread polls with ld.acquire.gpu, then a block barrier, then all
// its threads read.  Release and acquire are cumulative over the barriers'
// CTA-scope ordering, so no separate fence is needed on either side.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "handles.h"

namespace orbit {

namespace {

#ifndef ORBIT_SOLVE_THREADS
#define ORBIT_SOLVE_THREADS 128
#endif
// Blocks per SM the counter kernels are compiled for, per precision: many hide
// more of the per-task latency of launches that fill the GPU (FP32 10 with 48
// registers, FP64 7 with 72), fewer leave registers for the loads in flight of
// the others.  Sums do not depend on it.  8 bins, ms, many / few, with the factor
// entries of one bin of all orbits:
//   FP32 80x72x15: 1 orbit (52 M) 1.48 / 1.32, 4 (208 M) 2.67 / 2.54, 8 (416 M) 4.36 /
//   4.19, 10 (520 M) 5.07 / 5.15, 12 5.94 / 6.15; 60x54x15: 4 (105 M) 1.99 / 1.70, 12
//   (315 M) 3.69 / 3.33, 16 (420 M) 4.35 / 4.24, 24 (631 M) 6.33 / 6.39; 40x36x15: 24
//   (219 M) 3.05 / 2.75, 48 (439 M) 4.85 / 5.01.
//   FP64 60x54x15: 2 (53 M) 1.64 / 1.55, 4 (105 M) 2.41 / 2.30, 8 (210 M) 4.41 / 4.08, 12
//   (315 M) 5.30 / 5.29; 40x36x15: 10 (91 M) 3.40 / 3.10, 24 (219 M) 4.35 / 4.22;
//   64x60x15: 4 (134 M) 2.88 / 2.74, 6 (201 M) 3.63 / 3.80.  80x72x15, whose tree is
//   larger: 1 (52 M) 1.75 / 1.67, 2 (104 M) 2.59 / 2.67, 3 3.30 / 3.21, 4 (207 M) 3.94 /
//   4.06, 6 5.73 / 5.93.
// So the line lies at 1.6 GB a bin (400 M and 200 M entries) and, for FP64 trees of
// more than 40 M entries, at 0.6 GB, between one orbit and two.
constexpr int kChainBlocks[2] = {10, 7}, kChainBlocksFew[2] = {8, 6};  // FP32, FP64
inline double chain_many_bytes(const Symbolic& S, bool fp64) {
  return fp64 && S.fac_nnz > 40000000 ? 0.6e9 : 1.6e9;
}
constexpr int kSolveThreads = ORBIT_SOLVE_THREADS;
constexpr int kMaxPhases = 96;  // 2 x tree levels
constexpr int kWarps = kSolveThreads / 32;

template <typename T>
struct ChainDev {
  const int32_t *first, *n, *m, *parent, *child, *uidx, *rel, *ldn, *ldm;
  const int32_t* ginv;      // inverse extend-add maps, 2 x (n + m) per supernode
  const int64_t* ginv_off;
  const int32_t *nch_f, *nch_b, *level;
  int sub_front;  // per-warp vector capacity for subtree tasks
  const int64_t *uoff, *fac_off, *woff;
  const int4* items;
  const int32_t* phase_off;
  int nphase, items_per_bin, nsuper;
  int64_t N, fac_size, w_size;
  const T* factors;
  double* X;
  const double* E;
  double escale;
  double* Y;
  double* W;
  int* counters;
  int* task_counter;
  int* status;
  const int* orbit_ids;
  const int* set_of;  // factor set of each solve slot
  int n_bins;
  int B, tau0, tau1, trans;
  int Borb;  // multi-RHS kernel: right-hand sides in the launch (B counts their groups)
  int total;
  long long spin_limit;
  int never_ready;  // self-test: the first task waits for a count nothing reaches
  int prefetch;     // L2 prefetch of each task's factor rows before its dependency wait
  int stream_ef;    // factor rows read once per launch: evict-first loads
  int64_t prefetch_bytes;  // at most this many bytes of a task's rows are prefetched
  unsigned spin_ns;  // longest sleep between polls of a completion counter
  int ngroups;  // task groups (orbits or right-hand-side groups) split into ngroups ...
  int goff;     // ... whose phase sequences start goff phases apart
  // tagged results of the dataflow kernels (see Entry): per orbit w_size
  // update entries, N forward results, N solutions; bin tau's carry tag0 + tau
  void *WF, *YF, *XF;
  unsigned tag0;
  const FlowRec* recs;  // tasks of the row-oriented dataflow kernel
};

// Claim order.  A launch's work is nb bins x nphase phases (fwd leaves->root,
// bwd root->leaves) for B task groups (single orbits, or groups of
// right-hand sides).  The groups are split into D.ngroups sets; set gr runs its
// global phase g = bin * nphase + phase at slot g + gr * D.goff, and tasks are
// claimed slot by slot (set, then group, then item within a slot).  With one
// set this is the plain bin / phase / group order; with several, the sets reach
// the few large tasks at the top of the tree at different times, so tasks of
// the other sets fill the GPU meanwhile.  Every dependency lies inside one
// group (earlier phase or bin of the same orbit), so it is still claimed
// earlier, and the earliest unfinished task can always run.
constexpr int kMaxSlots = 9 * kMaxPhases + 1;
constexpr int kMaxSets = 8;

// Shared tables of the claim order: first task of every slot, first group of
// every set, task count of every phase.
struct SlotTables {
  int slot[kMaxSlots];
  int set_first[kMaxSets + 1];
  int cnt[kMaxPhases];
  int nslot, G;
};

template <typename T>
__device__ __forceinline__ void build_slots(const ChainDev<T>& D, SlotTables& S) {
  const int nb = D.total / (D.items_per_bin * D.B);
  const int G = nb * D.nphase;
  const int nslot = G + (D.ngroups - 1) * D.goff;
  for (int i = threadIdx.x; i < D.nphase; i += blockDim.x) S.cnt[i] = D.phase_off[i + 1] - D.phase_off[i];
  for (int i = threadIdx.x; i <= D.ngroups; i += blockDim.x) S.set_first[i] = (int)(((int64_t)i * D.B) / D.ngroups);
  __syncthreads();
  for (int sg = threadIdx.x; sg < nslot; sg += blockDim.x) {
    int sz = 0;
    for (int gr = 0; gr < D.ngroups; ++gr) {
      const int g = sg - gr * D.goff;
      if (g >= 0 && g < G) sz += S.cnt[g % D.nphase] * (S.set_first[gr + 1] - S.set_first[gr]);
    }
    S.slot[sg + 1] = sz;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    S.slot[0] = 0;
    for (int sg = 1; sg <= nslot; ++sg) S.slot[sg] += S.slot[sg - 1];
    S.nslot = nslot;
    S.G = G;
  }
  __syncthreads();
}

// Task t of slot lo -> bin q (0-based in the launch), phase p, group index gi, item index.
template <typename T>
__device__ __forceinline__ void slot_task(const ChainDev<T>& D, const SlotTables& S, int t, int lo, int& q, int& p,
                                          int& gi, int& item) {
  int rem = t - S.slot[lo];
  for (int gr = 0; gr < D.ngroups; ++gr) {
    const int g = lo - gr * D.goff;
    if (g < 0 || g >= S.G) continue;
    const int pp = g % D.nphase;
    const int cnt = S.cnt[pp];
    const int sz = cnt * (S.set_first[gr + 1] - S.set_first[gr]);
    if (rem < sz) {
      const int k = rem / cnt;
      q = g / D.nphase;
      p = pp;
      gi = S.set_first[gr] + k;
      item = D.phase_off[pp] + (rem - k * cnt);
      return;
    }
    rem -= sz;
  }
  q = p = gi = item = 0;  // not reached for t < total
}

// Task t -> bin q (0-based in the launch), phase p, group index gi, item index.
template <typename T>
__device__ __forceinline__ void decode_task(const ChainDev<T>& D, const SlotTables& S, int t, int& q, int& p,
                                            int& gi, int& item) {
  int lo = 0, hi = S.nslot;  // slot with slot[lo] <= t < slot[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (S.slot[mid] <= t) lo = mid;
    else hi = mid;
  }
  slot_task(D, S, t, lo, q, p, gi, item);
}

// Bounded spin on a completion counter: sleeps between polls double from
// 32 ns up to max_ns; `limit` polls at most, then ORBIT_ERR_TIMEOUT.
__device__ __forceinline__ bool wait_ge(const int* p, int target, int* status, long long limit,
                                        unsigned max_ns = 1024) {
  long long it = 0;
  unsigned ns = 32;
  while (ld_acquire(p) < target) {
    if (ld_volatile(status) != 0) return false;
    if (++it > limit) {
      raise_status(status, ORBIT_ERR_TIMEOUT);
      return false;
    }
    __nanosleep(ns);
    if (ns < max_ns) ns <<= 1;
  }
  return true;
}

// Vector types for 16-byte loads of factor rows (rows start 16-byte aligned:
// every leading dimension and block offset is a multiple of 4 elements).
template <typename T> struct Vec16;
template <> struct Vec16<float> { using type = float4; static constexpr int w = 4; };
template <> struct Vec16<double> { using type = double2; static constexpr int w = 2; };

__device__ __forceinline__ float dot16(const float4& a, const float* v) {
  return a.x * v[0] + a.y * v[1] + a.z * v[2] + a.w * v[3];
}
__device__ __forceinline__ double dot16(const double2& a, const double* v) {
  return a.x * v[0] + a.y * v[1];
}

// 16-byte loads in flight per lane in the row dot products of the chained
// solves, per precision.  FP32 6 (7.21 ms at 4, 6.94 at 6, 7.05 at 7 for the
// 12-orbit chain when it was chosen; a row's lanes, and with them the order of
// its sum, follow from it).  FP64 8: with the rows' ends in the first round, 6 / 8
// / 10 / 12 give 1.73 / 1.73 / 1.88 / 1.93 ms for one orbit of the 80x72x15 grid at
// 6 to 7 blocks per SM (10 and 12 spill), 2.63 / 2.35 / 2.62 / 2.77 for four of the
// 60x54x15 grid.
#ifndef ORBIT_SOLVE_DEPTH_FP32
#define ORBIT_SOLVE_DEPTH_FP32 6
#endif
#ifndef ORBIT_SOLVE_DEPTH_FP64
#define ORBIT_SOLVE_DEPTH_FP64 8
#endif
template <typename T> struct Depth { static constexpr int value = sizeof(T) == 4 ? ORBIT_SOLVE_DEPTH_FP32 : ORBIT_SOLVE_DEPTH_FP64; };

// Factor rows that a launch reads once (every solve slot has its own factor
// set) are loaded under an L2 evict-first policy, so that they do not push out
// the lines the tasks' prefetches brought in, nor the solution vectors; where
// slots share a set the rows are reused from L2 and load under the normal
// policy (the many-right-hand-side kernel keeps plain loads).  Measured on the
// 80x72x15 grid (8 bins, CUDA events): the 12-orbit FP32 chain 6.44-6.50 ms
// with evict-first against 6.58-6.62 without a hint, 6.54 with no L1
// allocation (alone or with evict-first), 6.57 with evict-last prefetches;
// the single-orbit FP64 chain unchanged (1.72 ms); evict-first in the 64-RHS
// kernels, where the groups share one set: 24.6 vs 20.9 ms transposed and
// 22.0 vs 20.7 ms forward.
__device__ __forceinline__ uint64_t stream_policy(bool evict_first) {
  uint64_t pol;
  if (evict_first) asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  else asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}

__device__ __forceinline__ float4 ld_stream(const float4* p, uint64_t pol) {
  float4 x;
  asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "l"(p), "l"(pol));
  return x;
}

__device__ __forceinline__ float2 ld_stream(const float2* p, uint64_t pol) {
  float2 x;
  asm("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(x.x), "=f"(x.y) : "l"(p), "l"(pol));
  return x;
}

__device__ __forceinline__ float ld_stream(const float* p, uint64_t pol) {
  float x;
  asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(x) : "l"(p), "l"(pol));
  return x;
}

__device__ __forceinline__ double2 ld_stream(const double2* p, uint64_t pol) {
  double2 x;
  asm("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(x.x), "=d"(x.y) : "l"(p), "l"(pol));
  return x;
}

// Factor rows in global memory, streamed under a cache policy, or staged in
// shared memory.
struct GlobalRow {
  uint64_t pol;
  template <typename V> __device__ __forceinline__ V vec(const V* p) const { return ld_stream(p, pol); }
  template <typename T> __device__ __forceinline__ T one(const T* p) const { return __ldg(p); }
};
struct SharedRow {
  template <typename V> __device__ __forceinline__ V vec(const V* p) const { return *p; }
  template <typename T> __device__ __forceinline__ T one(const T* p) const { return *p; }
};

// Per-lane partial of sum_{j0 <= j < j1} a[j] v[j] for a group of G lanes
// (gl = lane within the group; a 16-byte aligned at j = 0, v in shared memory,
// 16-byte aligned).  16-byte loads, up to U in flight per lane, the guarded loads
// of a round issued before any of them is used.  The unaligned ends (fewer than
// 4 elements, so at most one per lane) are read together with the first round:
// one memory latency for a row of up to U G vectors, where the ends used to cost
// one each (8 bins, ms: FP32, 12 orbits, 80x72x15 6.55 -> 6.03, 60x54x15 4.55 -> 3.77; one orbit of the
// 24x20x15 grid from shared memory 0.51 -> 0.45).
template <typename T, int G = 32, int U = Depth<T>::value, typename Row = GlobalRow>
__device__ __forceinline__ T dot_seg(const T* __restrict__ a, const T* v, int j0, int j1, int gl, const Row& row) {
  using V = typename Vec16<T>::type;
  constexpr int W = Vec16<T>::w;
  static_assert(G >= W, "one end element per lane");
  T acc0 = T(0), acc1 = T(0), acc2 = T(0), acc3 = T(0);
  // [j0, ja) scalar head up to the first aligned index, [ja, jb) 16-byte
  // vectors, [jb, j1) scalar tail
  const int ja = min((j0 + W - 1) / W * W, j1);
  const int jb = max(ja, j1 / W * W);
  const int nv1 = jb / W;
  const V* a4 = reinterpret_cast<const V*>(a);
  const bool head = j0 + gl < ja, tail = jb + gl < j1;
  T h = T(0), t = T(0);
  if (head) h = row.one(a + j0 + gl);
  if (tail) t = row.one(a + jb + gl);
  int k = ja / W + gl;
  V x[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    x[u] = V{};
    if (k + u * G < nv1) x[u] = row.vec(a4 + k + u * G);
  }
  if (head) acc0 = fma(h, v[j0 + gl], acc0);
  while (k < nv1) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || k + u * G < nv1) {
        const T d = dot16(x[u], v + (k + u * G) * W);
        if ((u & 3) == 0) acc0 += d;
        else if ((u & 3) == 1) acc1 += d;
        else if ((u & 3) == 2) acc2 += d;
        else acc3 += d;
      }
    k += U * G;
    if (k < nv1) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        x[u] = V{};
        if (u == 0 || k + u * G < nv1) x[u] = row.vec(a4 + k + u * G);
      }
    }
  }
  if (tail) acc1 = fma(t, v[jb + gl], acc1);
  return (acc0 + acc1) + (acc2 + acc3);
}

// Rows [r0, r1) of a row-major block as dot products, G lanes per row, so a
// warp works on 32 / G rows at once; warps wid, wid + nw, ... of the caller
// take successive row groups.  partial(g, i, gl) is a lane's share of row i
// (g is G as a std::integral_constant, for the matching dot_seg stride);
// store(i, sum) runs on the group's first lane.  The trip count is uniform
// across the warp (the shuffles are warp-wide).
template <int G, typename T, typename P, typename S>
__device__ __forceinline__ void grouped_rows(int r0, int r1, int wid, int nw, P&& partial, S&& store) {
  constexpr int R = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), gr = lane / G;
  for (int i0 = r0 + wid * R; i0 < r1; i0 += nw * R) {
    const int i = i0 + gr;
    T acc = i < r1 ? partial(std::integral_constant<int, G>(), i, gl) : T(0);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (i < r1 && gl == 0) store(i, acc);
  }
}

// Lanes per row from the longest row of the range: about U 16-byte vectors
// per lane (U loads in flight), between 4 and 32 lanes.
template <typename T, int U = 4>
__device__ __forceinline__ int group_lanes(int maxlen) {
  const int nv = (maxlen + Vec16<T>::w - 1) / Vec16<T>::w;
  return nv <= 4 * U ? 4 : nv <= 8 * U ? 8 : nv <= 16 * U ? 16 : 32;
}

#define ORBIT_GROUPED_ROWS(T, G_, r0, r1, wid, nw, partial, store)           \
  do {                                                                      \
    switch (G_) {                                                           \
      case 4: grouped_rows<4, T>(r0, r1, wid, nw, partial, store); break;   \
      case 8: grouped_rows<8, T>(r0, r1, wid, nw, partial, store); break;   \
      case 16: grouped_rows<16, T>(r0, r1, wid, nw, partial, store); break; \
      default: grouped_rows<32, T>(r0, r1, wid, nw, partial, store); break; \
    }                                                                       \
  } while (0)

// Column-oriented partial dot product of the transposed sweeps with whole-subtree
// tasks: this warp's share (rows i0 + warp, i0 + warp + kWarps, ... below i1) of
// sum_i a[i * stride] v[i], added to acc, with four loads in flight (lanes hold
// consecutive columns, so every row step is one coalesced read per warp).
template <typename T>
__device__ __forceinline__ T col_dot(const T* __restrict__ a, int64_t stride, int i0, int i1, const T* v, T acc) {
  int i = i0 + (threadIdx.x >> 5);
  for (; i + 3 * kWarps < i1; i += 4 * kWarps) {
    const T x0 = __ldg(a + (int64_t)i * stride);
    const T x1 = __ldg(a + (int64_t)(i + kWarps) * stride);
    const T x2 = __ldg(a + (int64_t)(i + 2 * kWarps) * stride);
    const T x3 = __ldg(a + (int64_t)(i + 3 * kWarps) * stride);
    acc = fma(x0, v[i], acc);
    acc = fma(x1, v[i + kWarps], acc);
    acc = fma(x2, v[i + 2 * kWarps], acc);
    acc = fma(x3, v[i + 3 * kWarps], acc);
  }
  for (; i < i1; i += kWarps) acc = fma(__ldg(a + (int64_t)i * stride), v[i], acc);
  return acc;
}

// Forward step of one supernode (L, or U^T when trans) for output rows
// [r0, r1): gathers its right-hand side (own entries of Xin, plus forcing) and
// the children's update vectors into `vec`, then one dense GEMV.  Ends with a
// block barrier.
template <typename T>
__device__ __forceinline__ void fwd_node(const ChainDev<T>& D, int o, int tau, int s, int r0, int r1, bool trans,
                                         T* vec, T* red) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t N = D.N;
  const int n = D.n[s], m = D.m[s], first = D.first[s];
  const int ldn = D.ldn[s], ldm = D.ldm[s];
  const T* SQ = D.factors + ((int64_t)D.set_of[o] * D.n_bins + tau) * D.fac_size + D.fac_off[s];
  const uint64_t pol = stream_policy(D.stream_ef != 0);
  double* Yo = D.Y + (int64_t)o * N;
  double* Wo = D.W + (int64_t)o * D.w_size;
  const int bin_in = trans ? tau + 1 : tau;
  const double* Xin = D.X + ((int64_t)o * 9 + bin_in) * N;
  const double* Ein = nullptr;
  if (D.E) {
    if (!trans) Ein = D.E + ((int64_t)o * 8 + tau) * N;
    else if (tau + 1 < D.tau1) Ein = D.E + ((int64_t)o * 8 + tau + 1) * N;
  }
  // Rows (or columns) [r0, r1) read vec on [0, min(r1, n)) and on
  // [max(r0, n), r1): only that part is gathered, in one pass, each position
  // pulling its own entry and the children's update entries that land on it
  // (inverse extend-add maps, -1 where a child contributes nothing).
  const int lo_end = min(r1, n), hi0 = max(r0, n);
  const int w = n + m;
  const int32_t* g0 = D.ginv + D.ginv_off[s];
  const int32_t* g1 = g0 + w;
  const int c0 = D.child[2 * s], c1 = D.child[2 * s + 1];
  const double* W0 = c0 >= 0 ? Wo + D.woff[c0] : nullptr;
  const double* W1 = c1 >= 0 ? Wo + D.woff[c1] : nullptr;
  for (int i = tid; i < lo_end; i += kSolveThreads) {
    double v = Xin[first + i];
    if (Ein) v += D.escale * Ein[first + i];
    const int u0 = g0[i], u1 = g1[i];
    if (u0 >= 0) v += W0[u0];
    if (u1 >= 0) v += W1[u1];
    vec[i] = (T)v;
  }
  for (int i = hi0 + tid; i < r1; i += kSolveThreads) {
    double v = 0.0;
    const int u0 = g0[i], u1 = g1[i];
    if (u0 >= 0) v += W0[u0];
    if (u1 >= 0) v += W1[u1];
    vec[i] = (T)v;
  }
  __syncthreads();
  if (!trans) {
    // rows of [SQ; Pb]: row i < n uses the strict lower part (unit diagonal)
    const int64_t woff = D.woff[s];
    auto partial = [&](auto g, int i, int gl) {
      return dot_seg<T, decltype(g)::value>(SQ + (int64_t)i * ldn, vec, 0, i < n ? i : n, gl, GlobalRow{pol});
    };
    auto store = [&](int i, T acc) {
      if (i < n) Yo[first + i] = (double)(vec[i] + acc);
      else Wo[woff + (i - n)] = (double)(vec[i] + acc);
    };
    const int G = group_lanes<T, Depth<T>::value>(min(r1 - 1, n));
    ORBIT_GROUPED_ROWS(T, G, r0, r1, warp, kWarps, partial, store);
  } else {
    // columns of [upper(SQ) | Qr]
    const T* Qr = SQ + (int64_t)(n + m) * ldn;
    for (int cb = r0; cb < r1; cb += 32) {
      const int c = cb + lane;
      T acc = T(0);
      if (c < r1) acc = c < n ? col_dot(SQ + c, ldn, 0, c + 1, vec, acc) : col_dot(Qr + (c - n), ldm, 0, n, vec, acc);
      red[warp * 32 + lane] = acc;
      __syncthreads();
      if (warp == 0 && c < r1) {
        T sum = T(0);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) sum += red[w * 32 + lane];
        if (c < n) Yo[first + c] = (double)sum;
        else Wo[D.woff[s] + (c - n)] = (double)(vec[c] + sum);
      }
      __syncthreads();
    }
  }
  __syncthreads();
}

// Backward step of one supernode (U, or L^T when trans) for rows [r0, r1):
// own forward result plus the ancestors' solution; the ancestor part of `vec`
// starts at the next 4-element boundary after the own part so both segments
// can be read with 16-byte loads.  Ends with a block barrier.
template <typename T>
__device__ __forceinline__ void bwd_node(const ChainDev<T>& D, int o, int tau, int s, int r0, int r1, bool trans,
                                         T* vec, T* red) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t N = D.N;
  const int n = D.n[s], m = D.m[s], first = D.first[s];
  const int ldn = D.ldn[s], ldm = D.ldm[s];
  const int n0pad = (n + 3) & ~3;
  const T* SQ = D.factors + ((int64_t)D.set_of[o] * D.n_bins + tau) * D.fac_size + D.fac_off[s];
  const uint64_t pol = stream_policy(D.stream_ef != 0);
  const double* Yo = D.Y + (int64_t)o * N;
  const int bin_out = trans ? tau : tau + 1;
  double* Xout = D.X + ((int64_t)o * 9 + bin_out) * N;
  const int32_t* ui = D.uidx + D.uoff[s];
  // rows (or columns) [r0, r1) read the own part of vec from r0 on
  for (int i = r0 + tid; i < n; i += kSolveThreads) vec[i] = (T)Yo[first + i];
  for (int u = tid; u < m; u += kSolveThreads) vec[n0pad + u] = (T)Xout[ui[u]];
  __syncthreads();
  if (!trans) {
    const T* Qr = SQ + (int64_t)(n + m) * ldn;
    auto partial = [&](auto g, int i, int gl) {
      constexpr int G = decltype(g)::value;
      return dot_seg<T, G>(SQ + (int64_t)i * ldn, vec, i, n, gl, GlobalRow{pol}) +
             dot_seg<T, G>(Qr + (int64_t)i * ldm, vec + n0pad, 0, m, gl, GlobalRow{pol});
    };
    auto store = [&](int i, T acc) { Xout[first + i] = (double)acc; };
    const int G = group_lanes<T, Depth<T>::value>(n - r0 + m);
    ORBIT_GROUPED_ROWS(T, G, r0, r1, warp, kWarps, partial, store);
  } else {
    // columns of [SQ_strict_lower ; Pb] with unit diagonal
    const T* Pb = SQ + (int64_t)n * ldn;
    for (int cb = r0; cb < r1; cb += 32) {
      const int c = cb + lane;
      T acc = T(0);
      if (c < r1) acc = col_dot(Pb + c, ldn, 0, m, vec + n0pad, col_dot(SQ + c, ldn, c + 1, n, vec, acc));
      red[warp * 32 + lane] = acc;
      __syncthreads();
      if (warp == 0 && c < r1) {
        T sum = vec[c];
#pragma unroll
        for (int w = 0; w < kWarps; ++w) sum += red[w * 32 + lane];
        Xout[first + c] = (double)sum;
      }
      __syncthreads();
    }
  }
  __syncthreads();
}

// Warp-level forward step of one small supernode (inside a subtree task).
template <typename T>
__device__ void fwd_node_warp(const ChainDev<T>& D, int o, int tau, int s, bool trans, T* v) {
  const int lane = threadIdx.x & 31;
  const int64_t N = D.N;
  const int n = D.n[s], m = D.m[s], first = D.first[s];
  const int ldn = D.ldn[s], ldm = D.ldm[s];
  const T* SQ = D.factors + ((int64_t)D.set_of[o] * D.n_bins + tau) * D.fac_size + D.fac_off[s];
  const uint64_t pol = stream_policy(D.stream_ef != 0);
  double* Yo = D.Y + (int64_t)o * N;
  double* Wo = D.W + (int64_t)o * D.w_size;
  const int bin_in = trans ? tau + 1 : tau;
  const double* Xin = D.X + ((int64_t)o * 9 + bin_in) * N;
  const double* Ein = nullptr;
  if (D.E) {
    if (!trans) Ein = D.E + ((int64_t)o * 8 + tau) * N;
    else if (tau + 1 < D.tau1) Ein = D.E + ((int64_t)o * 8 + tau + 1) * N;
  }
  for (int i = lane; i < n + m; i += 32) {
    double x = 0.0;
    if (i < n) {
      x = Xin[first + i];
      if (Ein) x += D.escale * Ein[first + i];
    }
    v[i] = (T)x;
  }
  for (int q2 = 0; q2 < 2; ++q2) {
    __syncwarp();
    const int c = D.child[2 * s + q2];
    if (c < 0) continue;
    const int mc = D.m[c];
    const int32_t* rel = D.rel + D.uoff[c];
    const double* wc = Wo + D.woff[c];
    for (int j = lane; j < mc; j += 32) v[rel[j]] += (T)wc[j];
  }
  __syncwarp();
  const int64_t woff = D.woff[s];
  if (!trans) {
    if (n <= 64) {
      for (int i = lane; i < n + m; i += 32) {
        const int len = i < n ? i : n;
        const T* row = SQ + (int64_t)i * ldn;
        T acc = T(0);
        for (int j = 0; j < len; ++j) acc = fma(__ldg(row + j), v[j], acc);
        if (i < n) Yo[first + i] = (double)(v[i] + acc);
        else Wo[woff + (i - n)] = (double)(v[i] + acc);
      }
    } else {
      auto partial = [&](auto g, int i, int gl) {
        return dot_seg<T, decltype(g)::value>(SQ + (int64_t)i * ldn, v, 0, i < n ? i : n, gl, GlobalRow{pol});
      };
      auto store = [&](int i, T acc) {
        if (i < n) Yo[first + i] = (double)(v[i] + acc);
        else Wo[woff + (i - n)] = (double)(v[i] + acc);
      };
      const int G = group_lanes<T>(n);
      ORBIT_GROUPED_ROWS(T, G, 0, n + m, 0, 1, partial, store);
    }
  } else {
    const T* Qr = SQ + (int64_t)(n + m) * ldn;
    for (int c = lane; c < n + m; c += 32) {
      T acc = T(0);
      if (c < n) {
        for (int i = 0; i <= c; ++i) acc = fma(__ldg(SQ + (int64_t)i * ldn + c), v[i], acc);
        Yo[first + c] = (double)acc;
      } else {
        const int u = c - n;
        for (int i = 0; i < n; ++i) acc = fma(__ldg(Qr + (int64_t)i * ldm + u), v[i], acc);
        Wo[woff + u] = (double)(v[c] + acc);
      }
    }
  }
  __syncwarp();
}

// Warp-level backward step of one small supernode (inside a subtree task).
template <typename T>
__device__ void bwd_node_warp(const ChainDev<T>& D, int o, int tau, int s, bool trans, T* v) {
  const int lane = threadIdx.x & 31;
  const int64_t N = D.N;
  const int n = D.n[s], m = D.m[s], first = D.first[s];
  const int ldn = D.ldn[s], ldm = D.ldm[s];
  const int n0pad = (n + 3) & ~3;
  const T* SQ = D.factors + ((int64_t)D.set_of[o] * D.n_bins + tau) * D.fac_size + D.fac_off[s];
  const uint64_t pol = stream_policy(D.stream_ef != 0);
  const double* Yo = D.Y + (int64_t)o * N;
  const int bin_out = trans ? tau : tau + 1;
  double* Xout = D.X + ((int64_t)o * 9 + bin_out) * N;
  const int32_t* ui = D.uidx + D.uoff[s];
  for (int i = lane; i < n; i += 32) v[i] = (T)Yo[first + i];
  for (int u = lane; u < m; u += 32) v[n0pad + u] = (T)Xout[ui[u]];
  __syncwarp();
  if (!trans) {
    const T* Qr = SQ + (int64_t)(n + m) * ldn;
    auto partial = [&](auto g, int i, int gl) {
      constexpr int G = decltype(g)::value;
      return dot_seg<T, G>(SQ + (int64_t)i * ldn, v, i, n, gl, GlobalRow{pol}) +
             dot_seg<T, G>(Qr + (int64_t)i * ldm, v + n0pad, 0, m, gl, GlobalRow{pol});
    };
    auto store = [&](int i, T acc) { Xout[first + i] = (double)acc; };
    const int G = group_lanes<T>(n + m);
    ORBIT_GROUPED_ROWS(T, G, 0, n, 0, 1, partial, store);
  } else {
    const T* Pb = SQ + (int64_t)n * ldn;
    for (int c = lane; c < n; c += 32) {
      T acc = v[c];
      for (int i = c + 1; i < n; ++i) acc = fma(__ldg(SQ + (int64_t)i * ldn + c), v[i], acc);
      for (int u = 0; u < m; ++u) acc = fma(__ldg(Pb + (int64_t)u * ldn + c), v[n0pad + u], acc);
      Xout[first + c] = (double)acc;
    }
  }
  __syncwarp();
}

// One instantiation per sweep direction (TR: transposed) and per schedule
// kind (SUB: the schedule has whole-subtree tasks), so that each kernel
// carries only the code its tasks run; FEW: fewer blocks per SM.
template <typename T, bool TR, bool SUB, bool FEW>
__global__ void __launch_bounds__(kSolveThreads, (FEW ? kChainBlocksFew : kChainBlocks)[sizeof(T) == 8]) k_chain(ChainDev<T> D) {
  extern __shared__ unsigned char smem_raw[];
  T* red = reinterpret_cast<T*>(smem_raw);      // kWarps * 32
  T* vec = red + kWarps * 32;                    // front-sized vector
  __shared__ int s_task;
  __shared__ int s_ok;   // status word clean at the claim
  __shared__ int s_dep;  // dependency wait succeeded
  __shared__ SlotTables s_tab;
  const int tid = threadIdx.x;
  build_slots(D, s_tab);
  for (;;) {
    if (tid == 0) {
      s_task = atomicAdd(D.task_counter, 1);
      s_ok = ld_volatile(D.status) == 0;
    }
    __syncthreads();
    const int t = s_task;
    if (t >= D.total || !s_ok) break;
    int q, p, oi, item;
    decode_task(D, s_tab, t, q, p, oi, item);
    const int tau = TR ? (D.tau1 - 1 - q) : (D.tau0 + q);
    const int4 it = D.items[item];
    const int o = D.orbit_ids[oi];
    const int s = it.x, kind = it.w;
    const bool fwd = (kind & 1) == 0;        // kinds 0, 2, 4, 6
    const bool trans = TR;                   // kinds 2, 3, 6, 7
    const bool subtree = SUB && kind >= 4;
    int* cbase = D.counters + (int64_t)o * 8 * 2 * D.nsuper;
    // The factor rows of a row-chunk task do not depend on other tasks: ask L2
    // for them before waiting (forward: whole rows of [SQ; Pb]; backward: the
    // upper part of the SQ rows and the Qr rows), one request per 128 bytes.
    // Off for FP64 at large batches, where the launch is throughput-bound and
    // the requests only cost issue slots.
    if (D.prefetch && (kind == 0 || kind == 1)) {
      const int n_s = D.n[s], ldn_s = D.ldn[s];
      const T* SQ = D.factors + ((int64_t)D.set_of[o] * D.n_bins + tau) * D.fac_size + D.fac_off[s];
      constexpr int L = 128 / sizeof(T);
      if (kind == 0) {
        const char* a = reinterpret_cast<const char*>(SQ + (int64_t)it.y * ldn_s);
        const int64_t bytes = min((int64_t)(it.z - it.y) * ldn_s * (int64_t)sizeof(T), D.prefetch_bytes);
        for (int64_t q = (int64_t)tid * 128; q < bytes; q += (int64_t)kSolveThreads * 128)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a + q));
      } else {
        const int ldm_s = D.ldm[s], m_s = D.m[s];
        const T* Qr = SQ + (int64_t)(n_s + m_s) * ldn_s;
        const int64_t row_bytes = (int64_t)(n_s + m_s) * sizeof(T);
        const int i_end = (int)min((int64_t)it.z, it.y + max((int64_t)1, D.prefetch_bytes / row_bytes));
        for (int i = it.y + (tid >> 3); i < i_end; i += kSolveThreads / 8) {
          const T* row = SQ + (int64_t)i * ldn_s;
          for (int c = (i & ~(L - 1)) + (tid & 7) * L; c < n_s; c += 8 * L)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(row + c));
          const T* qrow = Qr + (int64_t)i * ldm_s;
          for (int c = (tid & 7) * L; c < m_s; c += 8 * L) asm volatile("prefetch.global.L2 [%0];" ::"l"(qrow + c));
        }
      }
    }
    // ---- dependencies ----
    if (tid == 0) {
      bool ok = true;
      if (D.never_ready && t == 0)
        ok = wait_ge(cbase + (tau * 2 + 0) * D.nsuper + s, 0x7fffffff, D.status, D.spin_limit, D.spin_ns);
      if (!ok) {
      } else if (fwd) {
        if (!subtree)
          for (int q2 = 0; q2 < 2 && ok; ++q2) {
            const int c = D.child[2 * s + q2];
            if (c >= 0) ok = wait_ge(cbase + (tau * 2 + 0) * D.nsuper + c, D.nch_f[c], D.status, D.spin_limit, D.spin_ns);
          }
        if (ok && !trans && tau > D.tau0)
          ok = wait_ge(cbase + ((tau - 1) * 2 + 1) * D.nsuper + s, D.nch_b[s], D.status, D.spin_limit, D.spin_ns);
        if (ok && trans && tau < D.tau1 - 1)
          ok = wait_ge(cbase + ((tau + 1) * 2 + 1) * D.nsuper + s, D.nch_b[s], D.status, D.spin_limit, D.spin_ns);
      } else {
        const int par = D.parent[s];
        if (par < 0)
          ok = wait_ge(cbase + (tau * 2 + 0) * D.nsuper + s, D.nch_f[s], D.status, D.spin_limit, D.spin_ns);
        else
          ok = wait_ge(cbase + (tau * 2 + 1) * D.nsuper + par, D.nch_b[par], D.status, D.spin_limit, D.spin_ns);
      }
      s_dep = ok;
    }
    __syncthreads();
    if (!s_dep) break;
    if (!subtree) {
      if (fwd) fwd_node(D, o, tau, s, it.y, it.z, trans, vec, red);
      else bwd_node(D, o, tau, s, it.y, it.z, trans, vec, red);
    } else {
      // Whole subtree in this CTA: depth by depth (deepest first for the
      // forward sweep, root first for the backward sweep), the supernodes of
      // one depth spread over the warps, one warp per supernode.
      const int warp = threadIdx.x >> 5;
      T* wv = vec + warp * ((D.sub_front + 7) & ~3);
      const int d0 = it.y;
      const int top = D.level[s];
      int deep = top;
      for (int d = d0; d <= s; ++d) deep = max(deep, D.level[d]);
      for (int q3 = 0; q3 <= deep - top; ++q3) {
        const int lev = fwd ? deep - q3 : top + q3;
        int k = 0;
        for (int d = d0; d <= s; ++d) {
          if (D.level[d] != lev) continue;
          if ((k++ & (kWarps - 1)) != warp) continue;
          if (fwd) fwd_node_warp(D, o, tau, d, trans, wv);
          else bwd_node_warp(D, o, tau, d, trans, wv);
        }
        __syncthreads();
      }
    }
    if (tid == 0) {
      red_release_add(cbase + (tau * 2 + (fwd ? 0 : 1)) * D.nsuper + s, 1);
    }
  }
}

// ---- dataflow kernel ----
//
// One right-hand side per task, no completion counters: every value that one
// task hands to another (update entries W, forward results Y, solutions X) is
// stored together with a tag that names its launch and bin, so a consumer
// polls the very loads of its gather until the tags match.  Against a
// completion counter per supernode this takes the block barrier, the release
// and the separate acquire polls out of every step of the dependency chain,
// and a task starts as soon as the rows that it reads are there rather than
// when all chunks of the supernode are.
//
// An entry is published by one access that cannot tear: FP32 values as
// {value, tag} in 64 bits, FP64 values as two such halves {low, tag} {high,
// tag}, each valid by itself.  No fence orders different entries, and none is
// needed: each is checked by its own tag.
//
// The buffers hold one bin and are overwritten by the next one.  That is safe
// because a task overwrites an entry only after reads that depend on every
// reader of the old one: forward rows of bin t + 1 read the supernode's own
// solution of bin t, which was computed from its forward results and from all
// its ancestors' solutions, and those from every update entry of the
// supernodes below them (a child's update set contains all rows of its
// parent's separator, which the analysis checks).
template <typename T> struct Entry;
template <> struct Entry<float> {
  unsigned long long a;
};
template <> struct __align__(16) Entry<double> {
  unsigned long long a, b;
};

__device__ __forceinline__ bool ld_entry(const Entry<float>* p, unsigned tag, float& v) {
  unsigned long long a;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  v = __uint_as_float((unsigned)a);
  return (unsigned)(a >> 32) == tag;
}
__device__ __forceinline__ bool ld_entry(const Entry<double>* p, unsigned tag, double& v) {
  unsigned long long a, b;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  v = __hiloint2double((int)(unsigned)b, (int)(unsigned)a);
  return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}
__device__ __forceinline__ void st_entry(Entry<float>* p, unsigned tag, float v) {
  const unsigned long long a = ((unsigned long long)tag << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(a) : "memory");
}
__device__ __forceinline__ void st_entry(Entry<double>* p, unsigned tag, double v) {
  const unsigned long long t = (unsigned long long)tag << 32;
  const unsigned long long a = t | (unsigned)__double2loint(v), b = t | (unsigned)__double2hiint(v);
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}

// This lane's spin on one entry, bounded as wait_ge.
template <typename T>
__device__ __noinline__ bool spin_entry(const Entry<T>* p, unsigned tag, int* status, long long limit,
                                        unsigned max_ns) {
  unsigned ns = 32;
  T v;
  for (long long it = 0; !ld_entry(p, tag, v); ++it) {
    if ((it & 7) == 7 && ld_volatile(status) != 0) return false;
    if (it > limit) {
      raise_status(status, ORBIT_ERR_TIMEOUT);
      return false;
    }
    __nanosleep(ns);
    if (ns < max_ns) ns <<= 1;
  }
  return true;
}

// Gathers cnt positions into shared memory, position q by thread q mod NT,
// U positions per thread in flight.  load(q, entries[S], tags) issues the
// position's loads and returns a pointer to a missing entry (null when all were
// there, after storing the position's value).  Positions whose entries are not
// there yet are read again after one lane of the warp has seen its first
// missing entry arrive, so that waiting warps poll one address each.  False
// when a wait was given up (uniform over the warp).
template <typename T, int NT, int U, typename Load>
__device__ __forceinline__ bool flow_gather(int cnt, int* status, long long limit, unsigned max_ns, Load&& load) {
  constexpr int kWindow = flow_window(U);
  for (int base = 0; base < cnt; base += kWindow * NT) {
    const FlowShare sh = flow_share(cnt, base, (int)threadIdx.x, NT, kWindow);
    unsigned todo = sh.mine == 32 ? 0xffffffffu : (1u << sh.mine) - 1u;
    for (;;) {
      const Entry<T>* miss = nullptr;
      unsigned miss_tag = 0;
      for (int j = 0; j < sh.most; j += U) load(base + j * NT + (int)threadIdx.x, j, todo, miss, miss_tag);
      const unsigned bad = __ballot_sync(0xffffffffu, todo != 0);
      if (!bad) break;
      bool ok = true;
      if ((int)(threadIdx.x & 31) == __ffs(bad) - 1) ok = spin_entry<T>(miss, miss_tag, status, limit, max_ns);
      if (!__all_sync(0xffffffffu, ok)) return false;
    }
  }
  return true;
}

// Right-hand side of a forward task (rows or columns [r0, r1) of supernode
// s): vec on [0, min(r1, n)) and [max(r0, n), r1), own entries of the previous
// bin's solution (or of the launch's input) plus forcing and the children's
// update entries.
template <typename T, bool TR, int NT, int U>
__device__ __forceinline__ bool flow_gather_fwd(const ChainDev<T>& D, int o, int tau, int64_t ginv_off, int w0, int w1,
                                                int n, int m, int first, int r0, int r1, T* vec) {
  const int64_t N = D.N;
  const bool first_bin = TR ? tau == D.tau1 - 1 : tau == D.tau0;
  const int bin_in = TR ? tau + 1 : tau;
  const double* Xin = D.X + ((int64_t)o * 9 + bin_in) * N + first;
  const Entry<T>* XFo = static_cast<const Entry<T>*>(D.XF) + (int64_t)o * N + first;
  const double* Ein = nullptr;
  if (D.E) {
    if (!TR) Ein = D.E + ((int64_t)o * 8 + tau) * N + first;
    else if (tau + 1 < D.tau1) Ein = D.E + ((int64_t)o * 8 + tau + 1) * N + first;
  }
  const int lo_end = min(r1, n), hi0 = max(r0, n);
  const int cnt = lo_end + max(0, r1 - hi0);
  const int w = n + m;
  const int32_t* g0 = D.ginv + ginv_off;
  const Entry<T>* Wo = static_cast<const Entry<T>*>(D.WF) + (int64_t)o * D.w_size;
  const Entry<T>* W0 = Wo + max(w0, 0);  // not read where a child contributes nothing
  const Entry<T>* W1 = Wo + max(w1, 0);
  const unsigned tw = D.tag0 + tau, tx = TR ? tw + 1 : tw - 1;
  return flow_gather<T, NT, U>(
      cnt, D.status, D.spin_limit, D.spin_ns,
      [&](int q0, int j, unsigned& todo, const Entry<T>*& miss, unsigned& miss_tag) {
        int u0[U], u1[U];
        T x[U], a0[U], a1[U];
        double xd[U], e[U];
        unsigned got = 0;  // bits 3u: x, 3u + 1: child 0, 3u + 2: child 1
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool act = (todo >> (j + u)) & 1u;
          const int q = q0 + u * NT, i = q < lo_end ? q : q - lo_end + hi0;
          u0[u] = act ? g0[i] : -1;
          u1[u] = act ? g0[w + i] : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool act = (todo >> (j + u)) & 1u;
          const int i = q0 + u * NT;  // own positions are the first lo_end
          const bool own = act && i < lo_end;
          xd[u] = e[u] = 0.0;
          x[u] = a0[u] = a1[u] = T(0);
          if (own && first_bin) xd[u] = Xin[i];
          if (own && Ein) e[u] = Ein[i];
          if (!(own && !first_bin) || ld_entry(XFo + i, tx, x[u])) got |= 1u << (3 * u);
          if (u0[u] < 0 || ld_entry(W0 + u0[u], tw, a0[u])) got |= 2u << (3 * u);
          if (u1[u] < 0 || ld_entry(W1 + u1[u], tw, a1[u])) got |= 4u << (3 * u);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!((todo >> (j + u)) & 1u)) continue;
          const int q = q0 + u * NT, i = q < lo_end ? q : q - lo_end + hi0;
          if (((got >> (3 * u)) & 7u) == 7u) {
            double v = first_bin ? xd[u] : (double)x[u];
            if (Ein) v += D.escale * e[u];
            v += (double)a0[u];
            v += (double)a1[u];
            vec[i] = (T)v;
            todo &= ~(1u << (j + u));
          } else if (!miss) {
            const bool mx = !((got >> (3 * u)) & 1u);
            miss = mx ? XFo + q : !((got >> (3 * u)) & 2u) ? W0 + u0[u] : W1 + u1[u];
            miss_tag = mx ? tx : tw;
          }
        }
      });
}

// Inputs of a backward task: own forward results from r0 on, then (at vec +
// anc) the ancestors' solutions.
template <typename T, int NT, int U>
__device__ __forceinline__ bool flow_gather_bwd(const ChainDev<T>& D, int o, int tau, int64_t uoff, int n, int m,
                                                int first, int r0, int anc, T* vec) {
  const Entry<T>* Yo = static_cast<const Entry<T>*>(D.YF) + (int64_t)o * D.N + first + r0;
  const Entry<T>* XFo = static_cast<const Entry<T>*>(D.XF) + (int64_t)o * D.N;
  const int32_t* ui = D.uidx + uoff;
  const unsigned tag = D.tag0 + tau;
  const int own = n - r0, cnt = own + m;
  return flow_gather<T, NT, U>(
      cnt, D.status, D.spin_limit, D.spin_ns,
      [&](int q0, int j, unsigned& todo, const Entry<T>*& miss, unsigned& miss_tag) {
        int at[U];
        T v[U];
        unsigned got = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int q = q0 + u * NT;
          at[u] = ((todo >> (j + u)) & 1u) && q >= own ? ui[q - own] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int q = q0 + u * NT;
          v[u] = T(0);
          if ((todo >> (j + u)) & 1u)
            if (ld_entry(q < own ? Yo + q : XFo + at[u], tag, v[u])) got |= 1u << u;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!((todo >> (j + u)) & 1u)) continue;
          const int q = q0 + u * NT;
          if ((got >> u) & 1u) {
            vec[q < own ? r0 + q : anc + q - own] = v[u];
            todo &= ~(1u << (j + u));
          } else if (!miss) {
            miss = q < own ? Yo + q : XFo + at[u];
            miss_tag = tag;
          }
        }
      });
}

// Column sums of the transposed FP64 sweeps.  A column's sum is sixteen chains of
// fused multiply-adds, chain p over the rows congruent to p mod 16 of its block
// (U^T: SQ, or Qr; L^T: [SQ; Pb]) in increasing order; chains 4 w .. 4 w + 3 are
// added in pairs, the four sums of w in order.  The order fixes the rounding
// whatever the chunk, the lanes per row or the kernel (k_flow_t, k_chain_multi),
// so that a receptor's result does not depend on the batch that it is solved in.
constexpr int kColClasses = 16;

// For a row-major block (16-byte aligned at column c0, LPR vectors wide), sum over
// rows [i0, i1) (i0 a multiple of 16) of a[i][c] v[i], terms outside the triangle
// left out (TRI 1: i <= c, 2: i > c; c counted from the block's first column).  LPR lanes hold one
// row's vectors, so the block's 128 threads read 4 * 32 / LPR rows per step with U
// 16-byte loads in flight per lane, where one column per lane would have four
// 4-byte ones.  Warp w takes the chains 4 w .. 4 w + 3, LPR / 8 of them per lane.
template <int LPR, int TRI, int U>
__device__ __forceinline__ void col_part(const double* __restrict__ a, int64_t ld, int c0, int i0, int i1,
                                         const double* v, uint64_t pol, double (&acc)[LPR / 8][2]) {
  constexpr int Q = LPR / 8;
  const int lane = threadIdx.x & 31;
  const int c = c0 + (lane % LPR) * 2;
  const double* base = a + c;
  for (int i = i0 + (threadIdx.x >> 5) * 4 + lane / LPR * Q; i < i1; i += U / Q * kColClasses) {
    double2 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = i + u / Q * kColClasses + u % Q;
      x[u] = double2{};
      if (u == 0 || r < i1) x[u] = ld_stream(reinterpret_cast<const double2*>(base + (int64_t)r * ld), pol);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = i + u / Q * kColClasses + u % Q;
      if (u == 0 || r < i1) {
        const double b = v[r];
        if (TRI == 0 || (TRI == 1 ? r <= c : r > c)) acc[u % Q][0] = fma(x[u].x, b, acc[u % Q][0]);
        if (TRI == 0 || (TRI == 1 ? r <= c + 1 : r > c + 1)) acc[u % Q][1] = fma(x[u].y, b, acc[u % Q][1]);
      }
    }
  }
}

// Sum of the chains; red: kWarps x LPR * 2.  The thread c < LPR * 2 returns column
// c's sum.  Two block barriers.
template <int LPR>
__device__ __forceinline__ double col_reduce(double (&acc)[LPR / 8][2], double* red) {
  constexpr int CB = LPR * 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    double x = acc[0][k];
    if constexpr (LPR == 16) x += acc[1][k];
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane < LPR) red[warp * CB + lane * 2 + k] = x;
  }
  __syncthreads();
  double sum = 0.0;
  if (threadIdx.x < CB)
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sum += red[w * CB + threadIdx.x];
  __syncthreads();
  return sum;
}

// Results of a transposed task's column c (fwd: sum over the columns of U; bwd:
// including the unit diagonal's own value).
template <typename T>
__device__ __forceinline__ void flow_put_col(const ChainDev<T>& D, bool fwd, int o, int tau, int s, int n, int first,
                                             int c, T own, T sum) {
  const unsigned tag = D.tag0 + tau;
  if (!fwd) {
    st_entry(static_cast<Entry<T>*>(D.XF) + (int64_t)o * D.N + first + c, tag, sum);
    D.X[((int64_t)o * 9 + tau) * D.N + first + c] = (double)sum;
  } else if (c < n) {
    st_entry(static_cast<Entry<T>*>(D.YF) + (int64_t)o * D.N + first + c, tag, sum);
  } else {
    st_entry(static_cast<Entry<T>*>(D.WF) + (int64_t)o * D.w_size + D.woff[s] + (c - n), tag, own + sum);
  }
}

// Column blocks of a transposed FP32 task.  A column's sum is four chains of
// fused multiply-adds, chain w over every fourth row in increasing order, which
// are added in order at the end (forward: rows w, w + 4, ...; backward: rows
// c + 1 + w, ... of the triangle, then rows w, ... of the ancestors' panel): the
// order fixes the rounding whatever the chunk, so that loosely converged
// solves do not depend on it.  Warp w takes the rows congruent to w; in the
// backward triangle its lane of column c then holds chain (w - c - 1) mod 4,
// and the chains change warps through shared memory before the panel.  VEC
// consecutive columns per lane, U loads of VEC values in flight.
template <int VEC, int U>
__device__ __forceinline__ void col_chain(const float* __restrict__ a, int64_t ld, int i0, int i1, const float* v,
                                          uint64_t pol, float (&acc)[VEC]) {
  using V = typename std::conditional<VEC == 4, float4, typename std::conditional<VEC == 2, float2, float>::type>::type;
  for (int i = i0; i < i1; i += U * kWarps) {
    V x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      x[u] = V{};
      if (u == 0 || i + u * kWarps < i1) x[u] = ld_stream(reinterpret_cast<const V*>(a + (int64_t)(i + u * kWarps) * ld), pol);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || i + u * kWarps < i1) {
        const float b = v[i + u * kWarps];
        const float* xe = reinterpret_cast<const float*>(&x[u]);
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[k] = fmaf(xe[k], b, acc[k]);
      }
  }
}
// The same over the few rows that cross the triangle's diagonal: row i counts
// for column c + k when i <= c + k (LOW false) or i > c + k (LOW true).
template <int VEC, bool LOW>
__device__ __forceinline__ void col_chain_diag(const float* __restrict__ a, int64_t ld, int c, int i0, int i1,
                                               const float* v, float (&acc)[VEC]) {
#pragma unroll 4
  for (int i = i0; i < i1; i += kWarps) {
    const float b = v[i];
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      const bool in = LOW ? i > c + k : i <= c + k;
      const float x = in ? __ldg(a + (int64_t)i * ld + k) : 0.f;
      if (in) acc[k] = fmaf(x, b, acc[k]);
    }
  }
}

template <int VEC>
__device__ __forceinline__ void flow_chains(const ChainDev<float>& D, bool fwd, int o, int tau, int s, int n, int m,
                                            int first, int r0, int r1, const float* SQ, const float* vec, float* red,
                                            uint64_t pol) {
  constexpr int CB = 32 * VEC, U = 32 / VEC;
  const int ldn = D.ldn[s], ldm = D.ldm[s];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // first row >= i congruent to this warp
  auto from = [&](int i) { return i + ((warp - i) & (kWarps - 1)); };
  for (int cb = r0; cb < r1; cb += CB) {
    const int cend = min(cb + CB, r1), c = cb + lane * VEC;
    float acc[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc[k] = 0.f;
    if (fwd) {
      if (c < cend) {
        if (cb < n) {
          col_chain<VEC, U>(SQ + c, ldn, warp, cb, vec, pol, acc);
          col_chain_diag<VEC, false>(SQ + c, ldn, c, from(cb), cend, vec, acc);
        } else {
          col_chain<VEC, U>(SQ + (int64_t)(n + m) * ldn + (c - n), ldm, warp, n, vec, pol, acc);
        }
      }
    } else {
      const int d1 = min(cb + CB, n);  // rows beyond the diagonal's block
      if (c < cend) {
        col_chain_diag<VEC, true>(SQ + c, ldn, c, from(cb + 1), d1, vec, acc);
        col_chain<VEC, U>(SQ + c, ldn, from(d1), n, vec, pol, acc);
      }
#pragma unroll
      for (int k = 0; k < VEC; ++k) red[((warp - c - k - 1) & (kWarps - 1)) * CB + lane * VEC + k] = acc[k];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < VEC; ++k) acc[k] = red[warp * CB + lane * VEC + k];
      if (c < cend) col_chain<VEC, U>(SQ + (int64_t)n * ldn + c, ldn, warp, m, vec + n, pol, acc);
    }
    // each thread overwrites only what it read itself
#pragma unroll
    for (int k = 0; k < VEC; ++k) red[warp * CB + lane * VEC + k] = acc[k];
    __syncthreads();
    if (threadIdx.x < CB && cb + (int)threadIdx.x < cend) {
      const int cc = cb + threadIdx.x;
      float sum = fwd ? 0.f : vec[cc];
#pragma unroll
      for (int w = 0; w < kWarps; ++w) sum += red[w * CB + threadIdx.x];
      flow_put_col<float>(D, fwd, o, tau, s, n, first, cc, fwd && cc >= n ? vec[cc] : 0.f, sum);
    }
    __syncthreads();
  }
}

// Column blocks [cb, cb + 2 LPR) of a transposed FP64 task (its chunk starts at a
// multiple of 16 columns of SQ or of Qr).
template <int LPR>
__device__ __forceinline__ void flow_cols(const ChainDev<double>& D, bool fwd, int o, int tau, int s, int n, int m,
                                          int first, int r0, int r1, const double* SQ, const double* vec, double* red,
                                          uint64_t pol) {
  constexpr int CB = LPR * 2, U = 6;
  const int ldn = D.ldn[s], ldm = D.ldm[s];
  for (int cb = r0; cb < r1; cb += CB) {
    double acc[LPR / 8][2] = {};
    const int cend = min(cb + CB, r1);
    // lanes whose vector starts at or beyond the row's padded end read nothing
    const int cl = (threadIdx.x & 31) % LPR;
    if (fwd) {
      if (cb < n) {  // U^T: rows i <= c
        if (cb + cl * 2 < ldn) {
          col_part<LPR, 0, U>(SQ, ldn, cb, 0, cb, vec, pol, acc);
          col_part<LPR, 1, U>(SQ, ldn, cb, cb, min(cend, n), vec, pol, acc);
        }
      } else if (cb - n + cl * 2 < ldm) {
        col_part<LPR, 0, U>(SQ + (int64_t)(n + m) * ldn, ldm, cb - n, 0, n, vec, pol, acc);
      }
    } else if (cb + cl * 2 < ldn) {  // L^T, unit diagonal; [SQ; Pb] is one block of n + m rows
      col_part<LPR, 2, U>(SQ, ldn, cb, cb, min(cb + CB, n + m), vec, pol, acc);
      col_part<LPR, 0, U>(SQ, ldn, cb, cb + CB, n + m, vec, pol, acc);
    }
    const double sum = col_reduce<LPR>(acc, red);
    const int c = cb + threadIdx.x;
    if (threadIdx.x < CB && c < cend)
      flow_put_col<double>(D, fwd, o, tau, s, n, first, c, fwd && c >= n ? vec[c] : 0.0, fwd ? sum : vec[c] + sum);
  }
}

// Asynchronous copy of 16 bytes of factor values into shared memory under a
// cache policy (past L1).
__device__ __forceinline__ void stage16(void* dst, const void* src, uint64_t pol) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "l"(pol)
               : "memory");
}

// Stages columns [c0(r), c1(r)) of the rows r = 0 .. rows - 1 of a row-major
// block (16-byte aligned bounds, in vectors; at most nv of them), row r at
// dst + r * stride; as many lanes per row as it has vectors, up to a warp.
template <typename T, int NW, typename C0, typename C1>
__device__ __forceinline__ void stage_rows(T* dst, int stride, const T* src, int64_t ld, int rows, int nv,
                                           uint64_t pol, C0&& c0, C1&& c1) {
  constexpr int W = Vec16<T>::w;
  const int lg = nv >= 32 ? 5 : nv <= 1 ? 0 : 32 - __clz(nv - 1);
  const int per = 32 >> lg, lane = threadIdx.x & 31, gl = lane & ((1 << lg) - 1);
  for (int r = (threadIdx.x >> 5) * per + (lane >> lg); r < rows; r += NW * per) {
    const T* a = src + (int64_t)r * ld;
    T* d = dst + r * stride;
    for (int k = c0(r) + gl; k < c1(r); k += 1 << lg) stage16(d + k * W, a + k * W, pol);
  }
}

// A block's claimed task: index (the launch's total or more: none), bin in
// claim order, orbit, its factor set, and the task's record.
struct __align__(16) FlowClaim {  // written as 16-byte vectors
  FlowRec rec;
  int t, q, gi, o, set;
};

// A whole warp claims the next task and writes it to shared memory.  slot: of
// the last claimed task; K right-hand sides per group.
template <typename T>
__device__ __forceinline__ void flow_claim(const ChainDev<T>& D, const SlotTables& tab, FlowClaim& c, int& slot,
                                           int K = 1) {
  const int lane = threadIdx.x & 31;
  int t = 0;
  if (lane == 0) {
    t = atomicAdd(D.task_counter, 1);
    if (ld_volatile(D.status) != 0) t = D.total;
  }
  t = __shfl_sync(0xffffffffu, t, 0);
  if (t < D.total) {
    while (tab.slot[slot + 1] <= t) ++slot;
    int q, ph, gi, item;
    slot_task(D, tab, t, slot, q, ph, gi, item);
    if (lane < 4) reinterpret_cast<int4*>(&c.rec)[lane] = __ldg(reinterpret_cast<const int4*>(D.recs + item) + lane);
    if (lane == 4) {
      const int o = D.orbit_ids[gi * K];
      c.q = q;
      c.gi = gi;
      c.o = o;
      c.set = D.set_of[o];
    }
  }
  if (lane == 5) c.t = t;
}

// Row-oriented sweeps of launches bound by their dependency chain.  A task's
// factor rows, which do not depend on other tasks, are copied into shared
// memory as soon as the task is claimed, all of them in flight at once, while
// the gather waits for its inputs; the dot products then run from shared
// memory, where a row's unaligned ends and short rounds cost no memory latency
// each.  (From global memory, with the rows prefetched into L2, the products
// took 3 to 6 us of the 7 us that a step of the 24x20x15 grid's chain lasted;
// from shared memory 1 to 1.5 of 3.5.)  A launch that fills the GPU is faster
// on k_chain, which spends fewer instructions per byte and has more blocks per
// SM (12 FP32 orbits of the 80x72x15 grid: 6.5 ms against 10.6).
template <typename T>
__global__ void __launch_bounds__(kSolveThreads, 5)
    k_flow(ChainDev<T> D) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* stage = reinterpret_cast<T*>(smem_raw);        // kStageBytes
  T* vec = stage + kStageBytes / (int)sizeof(T);      // front-sized vector
  __shared__ __align__(16) FlowClaim s_claim;
  __shared__ SlotTables s_tab;
  constexpr int W = Vec16<T>::w;
  const int tid = threadIdx.x, warp = tid >> 5;
  build_slots(D, s_tab);
  const uint64_t pol = stream_policy(D.stream_ef != 0);
  for (int slot = 0;;) {
    if (tid < 32) flow_claim(D, s_tab, s_claim, slot);
    __syncthreads();
    const int t = s_claim.t;
    if (t >= D.total) break;
    const int tau = D.tau0 + s_claim.q, o = s_claim.o;
    const FlowRec& C = s_claim.rec;
    const int r0 = C.r0, r1 = C.r1, n = C.n, m = C.m, ldn = C.ldn, ldm = C.ldm, kind = C.kind_len & 255;
    const T* SQ = D.factors + ((int64_t)s_claim.set * D.n_bins + tau) * D.fac_size + C.fac_off;
    const T* Qr = SQ + (int64_t)(n + m) * ldn;
    const int stride = (int)staged_row(kind, r0, r1, n, ldn, ldm);
    // a single row may be longer than the stage: it is read from global memory
    const bool staged = (int64_t)(r1 - r0) * stride * (int64_t)sizeof(T) <= kStageBytes;
    const int a0 = r0 & ~3;  // first staged column of a backward task
    if (staged) {
      if (kind == 0) {
        stage_rows<T, kWarps>(stage, stride, SQ + (int64_t)r0 * ldn, ldn, r1 - r0, stride / W, pol, [](int) { return 0; },
                   [&](int r) { return (min(r0 + r, n) + W - 1) / W; });
      } else {
        stage_rows<T, kWarps>(stage, stride, SQ + (int64_t)r0 * ldn + a0, ldn, r1 - r0, (ldn - a0) / W, pol,
                   [&](int r) { return (r0 + r - a0) / W; }, [&](int) { return (n - a0 + W - 1) / W; });
        if (m > 0)
          stage_rows<T, kWarps>(stage + ldn - a0, stride, Qr + (int64_t)r0 * ldm, ldm, r1 - r0, ldm / W, pol,
                     [](int) { return 0; }, [&](int) { return (m + W - 1) / W; });
      }
    }
    const int anc = (n + 3) & ~3;  // ancestors' part of vec in a backward task
    bool ok = true;
    if (D.never_ready && t == 0)
      ok = spin_entry<T>(static_cast<const Entry<T>*>(D.YF), 0xffffffffu, D.status, D.spin_limit, D.spin_ns);
    constexpr int UF = sizeof(T) == 4 ? 4 : 3, UB = sizeof(T) == 4 ? 8 : 6;
    if (ok)
      ok = kind == 0 ? flow_gather_fwd<T, false, kSolveThreads, UF>(D, o, tau, C.map_off, C.w0, C.w1, n, m, C.first,
                                                                    r0, r1, vec)
                     : flow_gather_bwd<T, kSolveThreads, UB>(D, o, tau, C.map_off, n, m, C.first, r0, anc, vec);
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!__syncthreads_and(ok ? 1 : 0)) break;
    const unsigned tag = D.tag0 + tau;
    const int G = group_lanes<T, Depth<T>::value>(C.kind_len >> 8);
    constexpr int US = sizeof(T) == 4 ? Depth<T>::value : 4;  // FP32: the order of a row's sum follows from it
    if (kind == 0) {
      // rows of [SQ; Pb]: row i < n uses the strict lower part (unit diagonal)
      Entry<T>* Yo = static_cast<Entry<T>*>(D.YF) + (int64_t)o * D.N + C.first;
      Entry<T>* Wo = static_cast<Entry<T>*>(D.WF) + (int64_t)o * D.w_size + C.woff - n;
      auto store = [&](int i, T acc) { st_entry(i < n ? Yo + i : Wo + i, tag, vec[i] + acc); };
      if (staged) {
        auto partial = [&](auto g, int i, int gl) {
          return dot_seg<T, decltype(g)::value, US>(stage + (i - r0) * stride, vec, 0, i < n ? i : n, gl, SharedRow());
        };
        ORBIT_GROUPED_ROWS(T, G, r0, r1, warp, kWarps, partial, store);
      } else {
        auto partial = [&](auto g, int i, int gl) {
          return dot_seg<T, decltype(g)::value, US>(SQ + (int64_t)i * ldn, vec, 0, i < n ? i : n, gl, GlobalRow{pol});
        };
        ORBIT_GROUPED_ROWS(T, G, r0, r1, warp, kWarps, partial, store);
      }
    } else {
      Entry<T>* Xo = static_cast<Entry<T>*>(D.XF) + (int64_t)o * D.N + C.first;
      double* Xout = D.X + ((int64_t)o * 9 + tau + 1) * D.N + C.first;
      auto store = [&](int i, T acc) {
        st_entry(Xo + i, tag, acc);
        Xout[i] = (double)acc;
      };
      if (staged) {
        auto partial = [&](auto g, int i, int gl) {
          constexpr int Gv = decltype(g)::value;
          const T* row = stage + (i - r0) * stride;
          return dot_seg<T, Gv, US>(row - a0, vec, i, n, gl, SharedRow()) +
                 dot_seg<T, Gv, US>(row + (ldn - a0), vec + anc, 0, m, gl, SharedRow());
        };
        ORBIT_GROUPED_ROWS(T, G, r0, r1, warp, kWarps, partial, store);
      } else {
        auto partial = [&](auto g, int i, int gl) {
          constexpr int Gv = decltype(g)::value;
          return dot_seg<T, Gv, US>(SQ + (int64_t)i * ldn, vec, i, n, gl, GlobalRow{pol}) +
                 dot_seg<T, Gv, US>(Qr + (int64_t)i * ldm, vec + anc, 0, m, gl, GlobalRow{pol});
        };
        ORBIT_GROUPED_ROWS(T, G, r0, r1, warp, kWarps, partial, store);
      }
    }
    __syncthreads();
  }
}

// Column-oriented (transposed) sweeps.  Bound by the latency of the loads along
// a column (each stage of the dependency chain walks columns of up to n + m
// rows), so the loads in flight decide: 32 values per lane in FP32 at 7 blocks
// per SM (16 at 8 blocks, 1 / 4 / 12 orbits of the 40x36x15 grid: 1.49 / 1.93 /
// 2.58 ms; 32: 1.31 / 1.79 / 2.71), 12 in FP64.  Against one column per lane with
// four loads in flight and a completion counter per supernode: 40x36x15 FP32
// 1 / 12 orbits 3.25 / 5.03 -> 1.31 / 2.71 ms, FP64 1 orbit 2.38 -> 0.92;
// 80x72x15 FP32 12 orbits 11.5 -> 9.1, FP64 1 orbit 4.22 -> 1.82.
template <typename T>
__global__ void __launch_bounds__(kSolveThreads, 7) k_flow_t(ChainDev<T> D) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* red = reinterpret_cast<T*>(smem_raw);                      // kWarps * 32 (FP32: * 4)
  T* vec = red + kWarps * 32 * (sizeof(T) == 4 ? 4 : 1);          // front-sized vector
  __shared__ __align__(16) FlowClaim s_claim;
  __shared__ SlotTables s_tab;
  const int tid = threadIdx.x;
  build_slots(D, s_tab);
  const uint64_t pol = stream_policy(D.stream_ef != 0);
  for (int slot = 0;;) {
    if (tid < 32) flow_claim(D, s_tab, s_claim, slot);
    __syncthreads();
    const int t = s_claim.t;
    if (t >= D.total) break;
    const int tau = D.tau1 - 1 - s_claim.q, o = s_claim.o;
    const FlowRec& C = s_claim.rec;
    const int s = C.s, r0 = C.r0, r1 = C.r1, n = C.n, m = C.m, first = C.first, ldn = C.ldn;
    const bool fwd = C.kind_len == 2;
    const T* SQ = D.factors + ((int64_t)s_claim.set * D.n_bins + tau) * D.fac_size + C.fac_off;
    // The factor values do not depend on other tasks: ask L2 for them before
    // waiting, one request per 128 bytes of a row's segment.
    if (D.prefetch) {
      constexpr int L = 128 / sizeof(T);
      const bool sq = !fwd || r0 < n;
      const int ld = sq ? ldn : C.ldm;
      const T* a = sq ? SQ + r0 : SQ + (int64_t)(n + m) * ldn + (r0 - n);
      const int i0 = fwd ? 0 : r0, i1 = !fwd ? n + m : sq ? min(r1, n) : n;
      const int segs = ((r1 - r0) + L - 1) / L;
      const int rows = (int)min((int64_t)(i1 - i0), D.prefetch_bytes / (128 * segs));
      for (int b = tid; b < rows * segs; b += kSolveThreads)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a + (int64_t)(i0 + b / segs) * ld + min((b % segs) * L, r1 - r0 - 1)));
    }
    bool ok = true;
    if (D.never_ready && t == 0)
      ok = spin_entry<T>(static_cast<const Entry<T>*>(D.YF), 0xffffffffu, D.status, D.spin_limit, D.spin_ns);
    if (ok)
      ok = fwd ? flow_gather_fwd<T, true, kSolveThreads, sizeof(T) == 4 ? 4 : 3>(D, o, tau, C.map_off, C.w0, C.w1, n, m,
                                                                                 first, r0, r1, vec)
               : flow_gather_bwd<T, kSolveThreads, sizeof(T) == 4 ? 8 : 6>(D, o, tau, C.map_off, n, m, first, r0, n, vec);
    if (!__syncthreads_and(ok ? 1 : 0)) break;
    if constexpr (sizeof(T) == 4) {
      if (r1 - r0 >= 128) flow_chains<4>(D, fwd, o, tau, s, n, m, first, r0, r1, SQ, vec, red, pol);
      else if (r1 - r0 >= 64) flow_chains<2>(D, fwd, o, tau, s, n, m, first, r0, r1, SQ, vec, red, pol);
      else flow_chains<1>(D, fwd, o, tau, s, n, m, first, r0, r1, SQ, vec, red, pol);
    } else {
      if (r1 - r0 <= 16) flow_cols<8>(D, fwd, o, tau, s, n, m, first, r0, r1, SQ, vec, red, pol);
      else flow_cols<16>(D, fwd, o, tau, s, n, m, first, r0, r1, SQ, vec, red, pol);
    }
    __syncthreads();  // the record is read until here
  }
}

// ---- many FP64 right-hand sides on one factor set ----
//
// When every solve slot of an FP64 handle maps onto the same factor set (marginal
// perturbations or adjoint receptors of one operator), each task serves a
// group of K right-hand sides: one claim, one dependency wait (on the group's
// counters) and one barrier sequence, and every factor row loaded once is
// multiplied against the K gathered vectors.  Transposed sums have the order of
// k_flow_t's (16 right-hand sides of the 40x36x15 grid, a transposed sweep: 4.68
// ms with each lane's rows starting at its own column, 3.89 with the warp's rows
// together).

template <typename T, int G, int K>
__device__ __forceinline__ void dot_seg_multi(const T* __restrict__ a, const T* v, int vcap, int nk, int j0, int j1,
                                              int gl, T (&acc)[K]) {
  using V = typename Vec16<T>::type;
  constexpr int W = Vec16<T>::w;
  const int ja = min((j0 + W - 1) / W * W, j1);
  const int jb = max(ja, j1 / W * W);
  for (int j = j0 + gl; j < ja; j += G) {
    const T x = __ldg(a + j);
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k < nk) acc[k] = fma(x, v[k * vcap + j], acc[k]);
  }
  const V* a4 = reinterpret_cast<const V*>(a);
  const int nv0 = ja / W, nv1 = jb / W;
  for (int kk = nv0 + gl; kk < nv1; kk += 2 * G) {
    const bool b1 = kk + G < nv1;
    V x1 = {};
    const V x0 = __ldg(a4 + kk);
    if (b1) x1 = __ldg(a4 + kk + G);
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k < nk) {
        acc[k] += dot16(x0, v + k * vcap + kk * W);
        if (b1) acc[k] += dot16(x1, v + k * vcap + (kk + G) * W);
      }
  }
  for (int j = jb + gl; j < j1; j += G) {
    const T x = __ldg(a + j);
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k < nk) acc[k] = fma(x, v[k * vcap + j], acc[k]);
  }
}

// This warp's four chains of a column (see col_part), for K right-hand sides, and
// their sum: a at row 0 of the column's block, v by its rows.
template <typename T, int K>
__device__ __forceinline__ void col_dot_multi(const T* __restrict__ a, int64_t stride, int i0, int i1, const T* v,
                                              int vcap, int nk, T (&sum)[K]) {
  T acc[4][K] = {};
  int i = (i0 & ~(kColClasses - 1)) + (threadIdx.x >> 5) * 4;
  auto rows = [&](bool ends) {
    T x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      x[q] = !ends || (i + q >= i0 && i + q < i1) ? __ldg(a + (int64_t)(i + q) * stride) : T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (!ends || (i + q >= i0 && i + q < i1))
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (k < nk) acc[q][k] = fma(x[q], v[k * vcap + i + q], acc[q][k]);
    i += kColClasses;
  };
  if (i < i0) rows(true);  // no rows of it where i + 4 <= i0
  while (i + 4 <= i1) rows(false);
  if (i < i1) rows(true);
#pragma unroll
  for (int k = 0; k < K; ++k) sum[k] = (acc[0][k] + acc[1][k]) + (acc[2][k] + acc[3][k]);
}

template <int G, int K, typename T, typename P, typename S>
__device__ __forceinline__ void grouped_rows_multi(int r0, int r1, int wid, int nw, P&& partial, S&& store) {
  constexpr int R = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), gr = lane / G;
  for (int i0 = r0 + wid * R; i0 < r1; i0 += nw * R) {
    const int i = i0 + gr;
    T acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = T(0);
    if (i < r1) partial(std::integral_constant<int, G>(), i, gl, acc);
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (i < r1 && gl == 0) store(i, acc);
  }
}

#define ORBIT_GROUPED_ROWS_MULTI(T, K, G_, r0, r1, wid, nw, partial, store)            \
  do {                                                                                \
    switch (G_) {                                                                     \
      case 4: grouped_rows_multi<4, K, T>(r0, r1, wid, nw, partial, store); break;    \
      case 8: grouped_rows_multi<8, K, T>(r0, r1, wid, nw, partial, store); break;    \
      case 16: grouped_rows_multi<16, K, T>(r0, r1, wid, nw, partial, store); break;  \
      default: grouped_rows_multi<32, K, T>(r0, r1, wid, nw, partial, store); break;  \
    }                                                                                 \
  } while (0)

template <typename T, int K>
__global__ void __launch_bounds__(kSolveThreads, kChainBlocks[sizeof(T) == 8]) k_chain_multi(ChainDev<T> D, int vcap) {
  extern __shared__ unsigned char smem_raw[];
  T* vbuf = reinterpret_cast<T*>(smem_raw);  // K vectors of vcap
  T* red = vbuf + (int64_t)K * vcap;          // K x kWarps x 32 (transposed sweeps)
  __shared__ int s_task;
  __shared__ int s_ok;   // status word clean at the claim
  __shared__ int s_dep;  // dependency wait succeeded
  __shared__ SlotTables s_tab;
  const int tid = threadIdx.x, warp = tid >> 5;
  build_slots(D, s_tab);
  for (;;) {
    if (tid == 0) {
      s_task = atomicAdd(D.task_counter, 1);
      s_ok = ld_volatile(D.status) == 0;
    }
    __syncthreads();
    const int t = s_task;
    if (t >= D.total || !s_ok) break;
    int q, pph, gi, item;
    decode_task(D, s_tab, t, q, pph, gi, item);
    const int tau = D.trans ? (D.tau1 - 1 - q) : (D.tau0 + q);
    const int4 it = D.items[item];
    const int s = it.x, kind = it.w, r0 = it.y, r1 = it.z;
    const int nk = min(K, D.Borb - gi * K);
    int o[K];
#pragma unroll
    for (int k = 0; k < K; ++k) o[k] = D.orbit_ids[gi * K + (k < nk ? k : 0)];
    int* cbase = D.counters + (int64_t)o[0] * 8 * 2 * D.nsuper;  // the group's counters
    const int n = D.n[s], m = D.m[s], first = D.first[s], ldn = D.ldn[s], ldm = D.ldm[s];
    const T* SQ = D.factors + ((int64_t)D.set_of[o[0]] * D.n_bins + tau) * D.fac_size + D.fac_off[s];
    if (D.prefetch) {
      if (kind == 0) {
        const char* a = reinterpret_cast<const char*>(SQ + (int64_t)r0 * ldn);
        const int64_t bytes = min((int64_t)(r1 - r0) * ldn * (int64_t)sizeof(T), D.prefetch_bytes);
        for (int64_t q2 = (int64_t)tid * 128; q2 < bytes; q2 += (int64_t)kSolveThreads * 128)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a + q2));
      }
    }
    if (tid == 0) {
      bool ok = true;
      if (kind == 0 || kind == 2) {
        for (int q2 = 0; q2 < 2 && ok; ++q2) {
          const int c = D.child[2 * s + q2];
          if (c >= 0) ok = wait_ge(cbase + (tau * 2 + 0) * D.nsuper + c, D.nch_f[c], D.status, D.spin_limit, D.spin_ns);
        }
        if (ok && kind == 0 && tau > D.tau0)
          ok = wait_ge(cbase + ((tau - 1) * 2 + 1) * D.nsuper + s, D.nch_b[s], D.status, D.spin_limit, D.spin_ns);
        if (ok && kind == 2 && tau < D.tau1 - 1)
          ok = wait_ge(cbase + ((tau + 1) * 2 + 1) * D.nsuper + s, D.nch_b[s], D.status, D.spin_limit, D.spin_ns);
      } else {
        const int par = D.parent[s];
        if (par < 0) ok = wait_ge(cbase + (tau * 2 + 0) * D.nsuper + s, D.nch_f[s], D.status, D.spin_limit, D.spin_ns);
        else ok = wait_ge(cbase + (tau * 2 + 1) * D.nsuper + par, D.nch_b[par], D.status, D.spin_limit, D.spin_ns);
      }
      s_dep = ok;
    }
    __syncthreads();
    if (!s_dep) break;
    const int n0pad = (n + 3) & ~3;
    const int lane = tid & 31;
    if (kind == 2) {
      // transposed forward (U^T, then the update columns): gather over
      // [0, min(r1, n)) and [max(r0, n), r1) as the forward rows do, then
      // columns [r0, r1) of [upper(SQ) | Qr], each factor element used for
      // the K vectors
      const int lo_end = min(r1, n), hi0 = max(r0, n), w = n + m;
      const int32_t* g0 = D.ginv + D.ginv_off[s];
      const int32_t* g1 = g0 + w;
      const int c0 = D.child[2 * s], c1 = D.child[2 * s + 1];
      for (int k = 0; k < nk; ++k) {
        T* vec = vbuf + k * vcap;
        const double* Xin = D.X + ((int64_t)o[k] * 9 + tau + 1) * D.N;
        const double* Ein = (D.E && tau + 1 < D.tau1) ? D.E + ((int64_t)o[k] * 8 + tau + 1) * D.N : nullptr;
        const double* Wo = D.W + (int64_t)o[k] * D.w_size;
        const double* W0 = c0 >= 0 ? Wo + D.woff[c0] : nullptr;
        const double* W1 = c1 >= 0 ? Wo + D.woff[c1] : nullptr;
        for (int i = tid; i < lo_end; i += kSolveThreads) {
          double v = Xin[first + i];
          if (Ein) v += D.escale * Ein[first + i];
          const int u0 = g0[i], u1 = g1[i];
          if (u0 >= 0) v += W0[u0];
          if (u1 >= 0) v += W1[u1];
          vec[i] = (T)v;
        }
        for (int i = hi0 + tid; i < r1; i += kSolveThreads) {
          double v = 0.0;
          const int u0 = g0[i], u1 = g1[i];
          if (u0 >= 0) v += W0[u0];
          if (u1 >= 0) v += W1[u1];
          vec[i] = (T)v;
        }
      }
      __syncthreads();
      const T* Qr = SQ + (int64_t)(n + m) * ldn;
      const int64_t woff = D.woff[s];
      for (int cb = r0; cb < r1; cb += 32) {
        const int c = cb + lane;
        T acc[K];
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = T(0);
        if (c < r1) {
          if (c < n) col_dot_multi<T, K>(SQ + c, ldn, 0, c + 1, vbuf, vcap, nk, acc);
          else col_dot_multi<T, K>(Qr + (c - n), ldm, 0, n, vbuf, vcap, nk, acc);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) red[(k * kWarps + warp) * 32 + lane] = acc[k];
        __syncthreads();
        if (warp == 0 && c < r1) {
          for (int k = 0; k < nk; ++k) {
            T sum = T(0);
#pragma unroll
            for (int w2 = 0; w2 < kWarps; ++w2) sum += red[(k * kWarps + w2) * 32 + lane];
            if (c < n) D.Y[(int64_t)o[k] * D.N + first + c] = (double)sum;
            else D.W[(int64_t)o[k] * D.w_size + woff + (c - n)] = (double)(vbuf[k * vcap + c] + sum);
          }
        }
        __syncthreads();
      }
    } else if (kind == 3) {
      // transposed backward (L^T with unit diagonal): columns [r0, r1) of
      // [strict lower(SQ) ; Pb] against the own forward results and the
      // ancestors' solution
      const int32_t* ui = D.uidx + D.uoff[s];
      for (int k = 0; k < nk; ++k) {
        T* vec = vbuf + k * vcap;
        const double* Yo = D.Y + (int64_t)o[k] * D.N;
        const double* Xout = D.X + ((int64_t)o[k] * 9 + tau) * D.N;
        for (int i = r0 + tid; i < n; i += kSolveThreads) vec[i] = (T)Yo[first + i];
        for (int u = tid; u < m; u += kSolveThreads) vec[n + u] = (T)Xout[ui[u]];
      }
      __syncthreads();
      for (int cb = r0; cb < r1; cb += 32) {
        const int c = cb + lane;
        T acc[K];
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = T(0);
        if (c < r1) col_dot_multi<T, K>(SQ + c, ldn, c + 1, n + m, vbuf, vcap, nk, acc);
#pragma unroll
        for (int k = 0; k < K; ++k) red[(k * kWarps + warp) * 32 + lane] = acc[k];
        __syncthreads();
        if (warp == 0 && c < r1) {
          for (int k = 0; k < nk; ++k) {
            T sum = T(0);
#pragma unroll
            for (int w2 = 0; w2 < kWarps; ++w2) sum += red[(k * kWarps + w2) * 32 + lane];
            D.X[((int64_t)o[k] * 9 + tau) * D.N + first + c] = (double)(vbuf[k * vcap + c] + sum);
          }
        }
        __syncthreads();
      }
    } else if (kind == 0) {
      // gather each right-hand side's vector over the range the rows read
      const int lo_end = min(r1, n), hi0 = max(r0, n), w = n + m;
      const int32_t* g0 = D.ginv + D.ginv_off[s];
      const int32_t* g1 = g0 + w;
      const int c0 = D.child[2 * s], c1 = D.child[2 * s + 1];
      for (int k = 0; k < nk; ++k) {
        T* vec = vbuf + k * vcap;
        const double* Xin = D.X + ((int64_t)o[k] * 9 + tau) * D.N;
        const double* Ein = D.E ? D.E + ((int64_t)o[k] * 8 + tau) * D.N : nullptr;
        const double* Wo = D.W + (int64_t)o[k] * D.w_size;
        const double* W0 = c0 >= 0 ? Wo + D.woff[c0] : nullptr;
        const double* W1 = c1 >= 0 ? Wo + D.woff[c1] : nullptr;
        for (int i = tid; i < lo_end; i += kSolveThreads) {
          double v = Xin[first + i];
          if (Ein) v += D.escale * Ein[first + i];
          const int u0 = g0[i], u1 = g1[i];
          if (u0 >= 0) v += W0[u0];
          if (u1 >= 0) v += W1[u1];
          vec[i] = (T)v;
        }
        for (int i = hi0 + tid; i < r1; i += kSolveThreads) {
          double v = 0.0;
          const int u0 = g0[i], u1 = g1[i];
          if (u0 >= 0) v += W0[u0];
          if (u1 >= 0) v += W1[u1];
          vec[i] = (T)v;
        }
      }
      __syncthreads();
      const int64_t woff = D.woff[s];
      auto partial = [&](auto g, int i, int gl, T(&acc)[K]) {
        dot_seg_multi<T, decltype(g)::value, K>(SQ + (int64_t)i * ldn, vbuf, vcap, nk, 0, i < n ? i : n, gl, acc);
      };
      auto store = [&](int i, T(&acc)[K]) {
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (k < nk) {
            const double y = (double)(vbuf[k * vcap + i] + acc[k]);
            if (i < n) D.Y[(int64_t)o[k] * D.N + first + i] = y;
            else D.W[(int64_t)o[k] * D.w_size + woff + (i - n)] = y;
          }
      };
      const int Gl = group_lanes<T>(min(r1 - 1, n));
      ORBIT_GROUPED_ROWS_MULTI(T, K, Gl, r0, r1, warp, kWarps, partial, store);
    } else {
      const int32_t* ui = D.uidx + D.uoff[s];
      for (int k = 0; k < nk; ++k) {
        T* vec = vbuf + k * vcap;
        const double* Yo = D.Y + (int64_t)o[k] * D.N;
        const double* Xout = D.X + ((int64_t)o[k] * 9 + tau + 1) * D.N;
        for (int i = r0 + tid; i < n; i += kSolveThreads) vec[i] = (T)Yo[first + i];
        for (int u = tid; u < m; u += kSolveThreads) vec[n0pad + u] = (T)Xout[ui[u]];
      }
      __syncthreads();
      const T* Qr = SQ + (int64_t)(n + m) * ldn;
      auto partial = [&](auto g, int i, int gl, T(&acc)[K]) {
        constexpr int Gv = decltype(g)::value;
        dot_seg_multi<T, Gv, K>(SQ + (int64_t)i * ldn, vbuf, vcap, nk, i, n, gl, acc);
        dot_seg_multi<T, Gv, K>(Qr + (int64_t)i * ldm, vbuf + n0pad, vcap, nk, 0, m, gl, acc);
      };
      auto store = [&](int i, T(&acc)[K]) {
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (k < nk) D.X[((int64_t)o[k] * 9 + tau + 1) * D.N + first + i] = (double)acc[k];
      };
      const int Gl = group_lanes<T>(n - r0 + m);
      ORBIT_GROUPED_ROWS_MULTI(T, K, Gl, r0, r1, warp, kWarps, partial, store);
    }
    __syncthreads();
    if (tid == 0) {
      red_release_add(cbase + (tau * 2 + ((kind == 0 || kind == 2) ? 0 : 1)) * D.nsuper + s, 1);
    }
  }
}

// ---- many right-hand sides on one FP32 factor set ----
//
// K right-hand sides (4, 8 or 16) per task, interleaved: update entries,
// forward results and solutions are handed on as [position][K] floats, so that
// a gather reads one position's K values with 16-byte loads, and a factor value
// read once is used K times.  Bound by the shared-memory reads of the K vectors
// (16 bytes per 4 multiply-adds and row): four rows (or two columns) per lane
// share each of them, and the multiply-adds run two right-hand sides per
// instruction.  A right-hand side's sums have one order whatever K is.  Of a row:
// G lanes (from its chunk in the schedule of groups of four), each with every Gth
// vector of four entries, a vector's products added up (second, first, third,
// fourth) before they join the lane's sum, then a butterfly over the lanes.  Of a
// column: the four chains of flow_chains.
//
// What is left is latency (the wait, the gather and the barriers around them) at
// two blocks per SM, which the vectors of the largest fronts allow: 41 % of the
// issue slots used, transposed 33 %.  80x72x15 grid, 8 bins, 64 right-hand sides, a
// sweep against groups of four with one row (column) per lane: 18.0 -> 8.0 ms,
// transposed 17.4 -> 9.1 ms.
constexpr int kMultiThreads = 256;
constexpr int kMultiWarps = kMultiThreads / 32;
constexpr size_t kMultiSmem = 108 * 1024;  // two blocks per SM

struct MultiDev {
  ChainDev<float> C;
  float *W, *Y, *X;  // per group w_size x K, N x K, N x K
  const int32_t *nch_f, *nch_b;
  int smem_floats;  // dynamic shared memory of a block
};

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void unpack2(unsigned long long d, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(d));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// 16-byte chunk (right-hand sides 4 kq .. 4 kq + 3) of position j in the shared
// vectors: blocks of four positions, the chunks of a block permuted so that
// lanes reading the same chunk of eight consecutive blocks meet no bank twice.
template <int K>
__device__ __forceinline__ int multi_chunk(int j, int kq) {
  constexpr int QC = K / 4;
  const int jq = j >> 2, c = (j & 3) * QC + kq;
  return jq * 4 * QC + (QC == 1 ? c ^ ((jq >> 1) & 3) : c ^ (jq & 7));
}

// Forward right-hand side of the positions [0, min(r1, n)) and, from position
// `low` on, [max(r0, n), r1): own entries of the previous bin's solution (or of
// the launch's input) plus forcing and the children's update entries, K vectors.
template <int K, bool TR>
__device__ __forceinline__ void multi_gather_fwd(const MultiDev& M, const FlowRec& R, int gi, const int* o, int tau,
                                                 int r0, int r1, int low, float4* V) {
  const ChainDev<float>& D = M.C;
  constexpr int QC = K / 4;
  const int n = R.n, first = R.first, w = n + R.m;
  const bool first_bin = TR ? tau == D.tau1 - 1 : tau == D.tau0;
  const int bin_in = TR ? tau + 1 : tau;
  const int bin_e = TR ? tau + 1 : tau;
  const bool forced = D.E && (!TR || tau + 1 < D.tau1);
  const float4* Xg = reinterpret_cast<const float4*>(M.X + (int64_t)gi * D.N * K) + (int64_t)first * QC;
  const float4* Wg = reinterpret_cast<const float4*>(M.W + (int64_t)gi * D.w_size * K);
  const int32_t* g0 = D.ginv + R.map_off;
  const float4* W0 = Wg + (int64_t)max(R.w0, 0) * QC;
  const float4* W1 = Wg + (int64_t)max(R.w1, 0) * QC;
  const int lo_end = min(r1, n), hi0 = max(r0, n);
  const int cnt = lo_end + max(0, r1 - hi0);
#pragma unroll 2
  for (int idx = threadIdx.x; idx < cnt * QC; idx += kMultiThreads) {
    const int q = idx / QC, kq = idx % QC;
    const int i = q < lo_end ? q : q - lo_end + hi0;
    const int u0 = g0[i], u1 = g0[w + i];
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), a = x, b = x;
    if (u0 >= 0) a = __ldcg(W0 + (int64_t)u0 * QC + kq);
    if (u1 >= 0) b = __ldcg(W1 + (int64_t)u1 * QC + kq);
    if (i < n) {
      if (first_bin) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = D.X[((int64_t)o[4 * kq + k] * 9 + bin_in) * D.N + first + i];
      } else {
        x = __ldcg(Xg + (int64_t)i * QC + kq);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
      }
      if (forced)
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] += D.escale * D.E[((int64_t)o[4 * kq + k] * 8 + bin_e) * D.N + first + i];
    }
    if (u0 >= 0) { v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w; }
    if (u1 >= 0) { v[0] += b.x; v[1] += b.y; v[2] += b.z; v[3] += b.w; }
    V[multi_chunk<K>(q < lo_end ? q : low + q - lo_end, kq)] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
  }
}

// Positions [at, at + cnt) of the shared vectors from [position][K] arrays:
// src + idx(q) for q < cnt.
template <int K, typename Idx>
__device__ __forceinline__ void multi_gather(const float* src, int at, int cnt, float4* V, Idx&& idx) {
  constexpr int QC = K / 4;
  const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll 4
  for (int e = threadIdx.x; e < cnt * QC; e += kMultiThreads) {
    const int q = e / QC, kq = e % QC;
    V[multi_chunk<K>(at + q, kq)] = __ldcg(s4 + (int64_t)idx(q) * QC + kq);
  }
}

// acc[r][:] += (4 factor values a[r] of one vector) . (block jq of the shared
// vectors) for NR rows and the KW right-hand sides from 4 k0 on.  The value pairs
// of the factor entries are formed once for all of them.
template <int K, int KW, int NR>
__device__ __forceinline__ void multi_block(const float4* V, int jq, int k0, const float4 (&a)[NR],
                                            unsigned long long (&acc)[NR][KW / 2]) {
  unsigned long long p[NR][4];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    p[r][0] = pack2(a[r].x, a[r].x);
    p[r][1] = pack2(a[r].y, a[r].y);
    p[r][2] = pack2(a[r].z, a[r].z);
    p[r][3] = pack2(a[r].w, a[r].w);
  }
#pragma unroll
  for (int kq = 0; kq < KW / 4; ++kq) {
    unsigned long long v[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(V + multi_chunk<K>(4 * jq + j, k0 + kq));
      v[j][0] = t.x;
      v[j][1] = t.y;
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        acc[r][2 * kq + h] =
            add2(acc[r][2 * kq + h],
                 fma2(p[r][3], v[3][h], fma2(p[r][2], v[2][h], fma2(p[r][0], v[0][h], mul2(p[r][1], v[1][h])))));
  }
}

// acc[:] += x v[j] for one position j.
template <int K, int KW>
__device__ __forceinline__ void multi_one(const float4* V, int j, int k0, float x, unsigned long long (&acc)[KW / 2]) {
  const unsigned long long xx = pack2(x, x);
#pragma unroll
  for (int kq = 0; kq < KW / 4; ++kq) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(V + multi_chunk<K>(j, k0 + kq));
    acc[2 * kq] = fma2(xx, t.x, acc[2 * kq]);
    acc[2 * kq + 1] = fma2(xx, t.y, acc[2 * kq + 1]);
  }
}

// Sums over the G lanes of a group, the pairs of a butterfly, each lane keeping
// its share: values [4 rows][K] flat, on return 4 K / G of them from index
// `base` on.
template <int G, int K>
__device__ __forceinline__ int multi_reduce(unsigned long long (&acc)[4][K / 2], int gl, float (&v)[4 * K]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int h = 0; h < K / 2; ++h) unpack2(acc[r][h], v[r * K + 2 * h], v[r * K + 2 * h + 1]);
  int base = 0;
  int cnt = 4 * K;
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    // below one value per lane the rest of the group adds up the same values
    if (cnt > 1) {
      cnt >>= 1;
      const bool up = (gl & o) != 0;
#pragma unroll
      for (int q = 0; q < 2 * K; ++q)
        if (q < cnt) {
          const float mine = up ? v[q + cnt] : v[q], other = up ? v[q] : v[q + cnt];
          v[q] = mine + __shfl_xor_sync(0xffffffffu, other, o);
        }
      base += up ? cnt : 0;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return base;
}

// Row quads [4 q, 4 q + 4) of a task's rows [b0, b1), G lanes each; column j of
// row i at A0[(i - b0) * lda + j], of its ancestors' panel at B0[(i - b0) * ldb + j]
// (staged, or in global memory).  Forward: vectors from position 0, the rows'
// own values beyond n at `low`, from row `own0` on.  Backward: vectors of the
// own part at position j - at0, of the ancestors at `low`.
template <int G, int K, bool FWD>
__device__ __forceinline__ void multi_rows(const MultiDev& M, const FlowRec& R, int gi, const int* o, int nk, int tau,
                                           int b0, int b1, const float* A0, int lda, const float* B0, int ldb, int at0,
                                           int low, int own0, const float4* V) {
  const ChainDev<float>& D = M.C;
  const int n = R.n, m = R.m, first = R.first;
  // a warp takes up to 8 of the right-hand sides
  constexpr int KW = K < 8 ? K : 8, HALVES = K / KW;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), warp = threadIdx.x >> 5;
  const int k0 = (warp % HALVES) * (KW / 4);
  constexpr int per = 32 / G, sets = kMultiWarps / HALVES, NV = 4 * KW / G > 0 ? 4 * KW / G : 1;
  const int q0 = b0 >> 2, q1 = (b1 + 3) >> 2;
  for (int qb = q0 + (warp / HALVES) * per; qb < q1; qb += sets * per) {
    const int qd = qb + lane / G, i0 = 4 * qd;
    unsigned rows = 0;  // of the quad, in this batch; the others' sums are not stored
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (i0 + r >= b0 && i0 + r < b1) rows |= 1u << r;
    unsigned long long acc[4][KW / 2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int h = 0; h < KW / 2; ++h) acc[r][h] = 0ull;
    auto quad = [&](const float* p, int ld, int kk, float4 (&a)[4]) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        a[r] = (rows >> r) & 1u ? *(reinterpret_cast<const float4*>(p + r * ld) + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    const float* A = A0 + (int64_t)(i0 - b0) * lda;
    if (FWD) {
      if (rows) {
        const int nv1 = min(i0, n) >> 2;  // the quad's rows share their whole vectors
        for (int kk = gl; kk < nv1; kk += G) {
          float4 a[4];
          quad(A, lda, kk, a);
          multi_block<K, KW, 4>(V, kk, k0, a, acc);
        }
        const int j = 4 * nv1 + gl;
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (((rows >> r) & 1u) && j < min(i0 + r, n)) multi_one<K, KW>(V, j, k0, A[r * lda + j], acc[r]);
      }
    } else {
      // Upper triangle: row r's whole vectors start at ceil(i / 4), the quad's
      // first row one block before the others; lanes are aligned to the
      // others, and the first row's sums move one lane on afterwards.
      const int nvn = n >> 2;
      if (rows) {
#pragma unroll
        for (int r = 1; r < 4; ++r) {
          const int j = i0 + r + gl;
          if (((rows >> r) & 1u) && j < min(i0 + 4, n)) multi_one<K, KW>(V, j - at0, k0, A[r * lda + j], acc[r]);
        }
        if (gl == G - 1 && (rows & 1u) && qd < nvn) {
          const float4 a1[1] = {*(reinterpret_cast<const float4*>(A) + qd)};
          unsigned long long c1[1][KW / 2];
#pragma unroll
          for (int h = 0; h < KW / 2; ++h) c1[0][h] = acc[0][h];
          multi_block<K, KW, 1>(V, qd - (at0 >> 2), k0, a1, c1);
#pragma unroll
          for (int h = 0; h < KW / 2; ++h) acc[0][h] = c1[0][h];
        }
        for (int kk = qd + 1 + gl; kk < nvn; kk += G) {
          float4 a[4];
          quad(A, lda, kk, a);
          multi_block<K, KW, 4>(V, kk - (at0 >> 2), k0, a, acc);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          // lane of the row's own order that this lane stands for
          const int jb = max(r == 0 ? i0 : min(i0 + 4, n), nvn * 4), j = jb + (r == 0 ? (gl + 1) & (G - 1) : gl);
          if (((rows >> r) & 1u) && j < n) multi_one<K, KW>(V, j - at0, k0, A[r * lda + j], acc[r]);
        }
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < KW / 2; ++h)
        acc[0][h] = __shfl_sync(0xffffffffu, acc[0][h], (lane & ~(G - 1)) | ((gl - 1) & (G - 1)));
      if (rows) {
        const float* B = B0 + (int64_t)(i0 - b0) * ldb;
        const int nv = m >> 2;
        for (int kk = gl; kk < nv; kk += G) {
          float4 a[4];
          quad(B, ldb, kk, a);
          multi_block<K, KW, 4>(V, (low >> 2) + kk, k0, a, acc);
        }
        const int j = 4 * nv + gl;
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (((rows >> r) & 1u) && j < m) multi_one<K, KW>(V, low + j, k0, B[r * ldb + j], acc[r]);
      }
    }
    __syncwarp();
    float v[4 * KW];
    const int base = multi_reduce<G, KW>(acc, gl, v);
    // this lane's share: NV consecutive right-hand sides of one row
    const int r = base / KW, k = 4 * k0 + base % KW, i = i0 + r;
    if ((rows >> r) & 1u) {
      float* out;
      if (FWD) {
        const int at = i < n ? i : low + i - own0;
#pragma unroll
        for (int e = 0; e < NV; ++e)
          v[e] = reinterpret_cast<const float*>(V + multi_chunk<K>(at, (k + e) >> 2))[(k + e) & 3] + v[e];
        out = i < n ? M.Y + ((int64_t)gi * D.N + first + i) * K + k
                    : M.W + ((int64_t)gi * D.w_size + R.woff + (i - n)) * K + k;
      } else {
        out = M.X + ((int64_t)gi * D.N + first + i) * K + k;
        double* X = D.X + (int64_t)(tau + 1) * D.N + first + i;
#pragma unroll
        for (int e = 0; e < NV; ++e)
          if (k + e < nk) X[(int64_t)o[k + e] * 9 * D.N] = (double)v[e];
      }
      if constexpr (NV >= 4) {
#pragma unroll
        for (int e = 0; e < NV; e += 4)
          *reinterpret_cast<float4*>(out + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
      } else if constexpr (NV == 2) {
        *reinterpret_cast<float2*>(out) = make_float2(v[0], v[1]);
      } else {
        out[0] = v[0];
      }
    }
  }
}

// Column chains of a transposed task (see flow_chains) for K right-hand sides,
// VEC columns per lane: rows i0, i0 + 4, ... below i1 of a (at this lane's first
// column), positions i - at0 of the shared vectors.  DIAG: row i counts for
// column c + q when i <= c + q (1) or i > c + q (2).
template <int K, int VEC, int DIAG, int U>
__device__ __forceinline__ void multi_chain(const float* __restrict__ a, int64_t ld, int c, int i0, int i1,
                                            const float4* V, int at0, unsigned long long (&acc)[VEC][K / 2]) {
  using T = typename std::conditional<VEC == 2, float2, float>::type;
  for (int i = i0; i < i1; i += 4 * U) {
    T x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      x[u] = T{};
      if (u == 0 || i + 4 * u < i1) x[u] = __ldg(reinterpret_cast<const T*>(a + (int64_t)(i + 4 * u) * ld));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = i + 4 * u;
      if (u == 0 || r < i1) {
        const float* xe = reinterpret_cast<const float*>(&x[u]);
#pragma unroll
        for (int kq = 0; kq < K / 4; ++kq) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(V + multi_chunk<K>(r - at0, kq));
#pragma unroll
          for (int q = 0; q < VEC; ++q) {
            const unsigned long long xx = pack2(xe[q], xe[q]);
            const unsigned long long s0 = fma2(xx, t.x, acc[q][2 * kq]), s1 = fma2(xx, t.y, acc[q][2 * kq + 1]);
            const bool in = DIAG == 0 || (DIAG == 1 ? r <= c + q : r > c + q);
            if (in) {
              acc[q][2 * kq] = s0;
              acc[q][2 * kq + 1] = s1;
            }
          }
        }
      }
    }
  }
}

// Transposed task: columns [r0, r1) in pairs of blocks of 32 VEC, the first of a
// pair by warps 0-3, the second by warps 4-7, warp w of a half on the rows
// congruent to w.  The chains change warps, and are added up, through the
// shared memory behind the vectors, or over them where that is full (then the
// task is one pair, and a backward one gathers the ancestors' solution once its
// own part is used up).
template <int K, int VEC>
__device__ __forceinline__ void multi_cols(const MultiDev& M, const FlowRec& R, int gi, const int* o, int nk, int tau,
                                           const float* SQ, float4* V) {
  const ChainDev<float>& D = M.C;
  constexpr int CB = 32 * VEC, U = 8, QC = K / 4;  // U 4 / 8 / 12 / 16: 10.5 / 9.5 / 9.9 / 10.5 ms a sweep of dense vectors
  const bool fwd = R.kind_len == 2;
  const int r0 = R.r0, r1 = R.r1, n = R.n, m = R.m, first = R.first, ldn = R.ldn, ldm = R.ldm;
  const int lane = threadIdx.x & 31, half = threadIdx.x >> 7, w = (threadIdx.x >> 5) & 3, ht = threadIdx.x & 127;
  const int at0 = fwd ? 0 : r0 & ~3;
  const int low = fwd ? 0 : (n - at0 + 3) & ~3;  // ancestors' part, where it has room of its own
  const int blocks = (((fwd ? min(r1, n) : low + m) + 3) >> 2) * K;  // 16-byte chunks of all vectors
  const bool both = (blocks + 2 * 4 * QC * CB) * 4 <= M.smem_floats;
  // [class][right-hand-side quad][column] of this half
  ulonglong2* red = reinterpret_cast<ulonglong2*>(both ? V + blocks : V) + half * 4 * QC * CB;
  const float* Yg = M.Y + ((int64_t)gi * D.N + first) * K;
  const float* Xg = M.X + (int64_t)gi * D.N * K;
  const int32_t* ui = D.uidx + (fwd ? 0 : R.map_off);
  if (fwd) multi_gather_fwd<K, true>(M, R, gi, o, tau, 0, min(r1, n), 0, V);
  else multi_gather<K>(Yg, r0 - at0, n - r0, V, [&](int q) { return r0 + q; });
  if (!fwd && both) multi_gather<K>(Xg, low, m, V, [&](int q) { return ui[q]; });
  __syncthreads();
  auto from = [&](int i) { return i + ((w - i) & 3); };
  for (int pair = r0; pair < r1; pair += 2 * CB) {
  const int cb = pair + half * CB;
  const bool on = cb < r1;
  const int cend = min(cb + CB, r1), c = cb + lane * VEC;
  unsigned long long acc[VEC][K / 2];
#pragma unroll
  for (int q = 0; q < VEC; ++q)
#pragma unroll
    for (int h = 0; h < K / 2; ++h) acc[q][h] = 0ull;
  if (fwd) {
    if (on && c < cend) {
      if (cb < n) {
        multi_chain<K, VEC, 0, U>(SQ + c, ldn, c, w, cb, V, 0, acc);
        multi_chain<K, VEC, 1, U>(SQ + c, ldn, c, from(cb), cend, V, 0, acc);
      } else {
        multi_chain<K, VEC, 0, U>(SQ + (int64_t)(n + m) * ldn + (c - n), ldm, c, w, n, V, 0, acc);
      }
    }
  } else {
    const int d1 = min(cb + CB, n);
    if (on && c < cend) {
      multi_chain<K, VEC, 2, U>(SQ + c, ldn, c, from(cb + 1), d1, V, at0, acc);
      multi_chain<K, VEC, 0, U>(SQ + c, ldn, c, from(d1), n, V, at0, acc);
    }
    if (!both) __syncthreads();
    // the triangle's chain (w - c - 1) mod 4 of a column goes on in that warp
#pragma unroll
    for (int kq = 0; kq < QC; ++kq)
#pragma unroll
      for (int q = 0; q < VEC; ++q)
        red[(((w - c - q - 1) & 3) * QC + kq) * CB + lane * VEC + q] = make_ulonglong2(acc[q][2 * kq], acc[q][2 * kq + 1]);
    __syncthreads();
#pragma unroll
    for (int kq = 0; kq < QC; ++kq)
#pragma unroll
      for (int q = 0; q < VEC; ++q) {
        const ulonglong2 t = red[(w * QC + kq) * CB + lane * VEC + q];
        acc[q][2 * kq] = t.x;
        acc[q][2 * kq + 1] = t.y;
      }
    if (!both) {
      __syncthreads();
      multi_gather<K>(Xg, 0, m, V, [&](int q) { return ui[q]; });
      __syncthreads();
    }
    // position of ancestor row i is i (+ low)
    if (on && c < cend)
      multi_chain<K, VEC, 0, U>(SQ + (int64_t)n * ldn + c, ldn, c, w, m, V, both ? -low : 0, acc);
  }
  if (!both) __syncthreads();
  // the four chains of a column, added in order to its own value
#pragma unroll
  for (int kq = 0; kq < QC; ++kq)
#pragma unroll
    for (int q = 0; q < VEC; ++q)
      red[(w * QC + kq) * CB + lane * VEC + q] = make_ulonglong2(acc[q][2 * kq], acc[q][2 * kq + 1]);
  __syncthreads();
  const float4* part = reinterpret_cast<const float4*>(red);
  const int32_t* g0 = D.ginv + (fwd ? R.map_off : 0);
  for (int e = on ? ht : CB * QC; e < CB * QC; e += 128) {
    const int cc = cb + e / QC, kq = e % QC;
    if (cc >= cend) continue;
    float4* Y = reinterpret_cast<float4*>(M.Y + ((int64_t)gi * D.N + first + cc) * K) + kq;
    float4 sum = fwd ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcg(Y);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 t = part[(q * QC + kq) * CB + cc - cb];
      sum.x += t.x; sum.y += t.y; sum.z += t.z; sum.w += t.w;
    }
    if (!fwd) {
      *(reinterpret_cast<float4*>(M.X + ((int64_t)gi * D.N + first + cc) * K) + kq) = sum;
      double* X = D.X + (int64_t)tau * D.N + first + cc;
      const float x[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * kq + k < nk) X[(int64_t)o[4 * kq + k] * 9 * D.N] = (double)x[k];
    } else if (cc < n) {
      *Y = sum;
    } else {
      const int u0 = g0[cc], u1 = g0[n + m + cc];
      const float4* Wg = reinterpret_cast<const float4*>(M.W + (int64_t)gi * D.w_size * K) + kq;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
      if (u0 >= 0) x = __ldcg(Wg + ((int64_t)R.w0 + u0) * QC);
      if (u1 >= 0) y = __ldcg(Wg + ((int64_t)R.w1 + u1) * QC);
      sum.x += (float)((double)x.x + (double)y.x);
      sum.y += (float)((double)x.y + (double)y.y);
      sum.z += (float)((double)x.z + (double)y.z);
      sum.w += (float)((double)x.w + (double)y.w);
      *(reinterpret_cast<float4*>(M.W + ((int64_t)gi * D.w_size + R.woff + (cc - n)) * K) + kq) = sum;
    }
  }
  if (pair + 2 * CB < r1) __syncthreads();  // the chains' space is free
  }
}

// A task's factor rows are staged in what the vectors leave of the block's
// shared memory, all at once where they fit, else in batches of row quads; the
// first batch is in flight during the dependency wait and the gather.  Where not
// even a quad fits (the largest fronts) the rows are read from L2.
template <int K, bool TR>
__global__ void __launch_bounds__(kMultiThreads, 2) k_multi(MultiDev M) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* V = reinterpret_cast<float4*>(smem_raw);
  const ChainDev<float>& D = M.C;
  __shared__ __align__(16) FlowClaim s_claims[2];  // the current task and the next
  __shared__ int s_dep, s_o[K];
  __shared__ SlotTables s_tab;
  const int tid = threadIdx.x, lane = tid & 31;
  build_slots(D, s_tab);
  const uint64_t pol = stream_policy(false);
  // The last warp claims the next task during the gather of the current one, which
  // takes the claim's 1.7 us off a task's 12 (every dependency is claimed earlier,
  // so the earliest unfinished task is still the current one of its block).
  const bool claimer = tid >= kMultiThreads - 32;
  int slot = 0;
  if (claimer) flow_claim(D, s_tab, s_claims[0], slot, K);
  for (int cur = 0;; cur ^= 1) {
    __syncthreads();
    const FlowClaim& s_claim = s_claims[cur];
    const int t = s_claim.t;
    if (t >= D.total) break;
    const FlowRec& R = s_claim.rec;
    const int tau = TR ? (D.tau1 - 1 - s_claim.q) : (D.tau0 + s_claim.q);
    const int gi = s_claim.gi, o0 = s_claim.o;
    const int s = R.s, r0 = R.r0, r1 = R.r1, kind = R.kind_len & 255, n = R.n, m = R.m, ldn = R.ldn, ldm = R.ldm;
    const int nk = min(K, D.Borb - gi * K);
    if (tid >= 32 && tid < 32 + K) s_o[tid - 32] = D.orbit_ids[gi * K + (tid - 32 < nk ? tid - 32 : 0)];
    int* cbase = D.counters + (int64_t)o0 * 8 * 2 * D.nsuper;  // the group's counters
    const float* SQ = D.factors + ((int64_t)s_claim.set * D.n_bins + tau) * D.fac_size + R.fac_off;
    const float* Qr = SQ + (int64_t)(n + m) * ldn;
    // rows: shared positions of the vectors, and the stage behind them
    const int at0 = kind == 0 ? 0 : r0 & ~3;
    const int low = kind == 0 ? (min(r1, n) + 3) & ~3 : ((n + 3) & ~3) - at0;
    const int own0 = max(r0, n);
    const int positions = kind == 0 ? low + max(0, r1 - own0) : low + m;
    float* stage = reinterpret_cast<float*>(V + (positions + 3) / 4 * K);
    const int room = (M.smem_floats - (positions + 3) / 4 * 4 * K);
    const int stride = TR ? 0 : (int)staged_row(kind, r0, r1, n, ldn, ldm);
    const bool staged = !TR && room >= 4 * stride;
    // rows a batch holds, its end on a quad boundary
    auto batch_end = [&](int b0) { return staged ? min(r1, (b0 + room / max(stride, 4)) & ~3) : r1; };
    auto stage_batch = [&](int b0, int b1) {
      if (kind == 0) {
        stage_rows<float, kMultiWarps>(stage, stride, SQ + (int64_t)b0 * ldn, ldn, b1 - b0, stride / 4, pol,
                                       [](int) { return 0; }, [&](int r) { return (min(b0 + r, n) + 3) / 4; });
      } else {
        stage_rows<float, kMultiWarps>(stage, stride, SQ + (int64_t)b0 * ldn + at0, ldn, b1 - b0, (ldn - at0) / 4, pol,
                                       [&](int r) { return (b0 + r - at0) / 4; },
                                       [&](int) { return (n - at0 + 3) / 4; });
        if (m > 0)
          stage_rows<float, kMultiWarps>(stage + ldn - at0, stride, Qr + (int64_t)b0 * ldm, ldm, b1 - b0, ldm / 4, pol,
                                         [](int) { return 0; }, [&](int) { return (m + 3) / 4; });
      }
    };
    int b0 = r0, b1 = TR ? r0 : batch_end(r0);
    if (staged) {
      stage_batch(b0, b1);
    } else if (!TR) {
      const float* a = kind == 0 ? SQ + (int64_t)r0 * ldn : Qr + (int64_t)r0 * ldm;
      const int64_t bytes = (int64_t)(r1 - r0) * (kind == 0 ? ldn : ldm) * (int64_t)sizeof(float);
      for (int64_t b = (int64_t)tid * 128; b < bytes; b += (int64_t)kMultiThreads * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(a) + b));
    } else {
      // ask L2 for the columns before waiting
      const bool sq = kind == 3 || r0 < n;
      const int ld = sq ? ldn : ldm;
      const float* a = sq ? SQ + r0 : Qr + (r0 - n);
      const int i0 = kind == 2 ? 0 : r0, i1 = kind == 3 ? n + m : sq ? min(r1, n) : n;
      const int segs = (r1 - r0 + 31) / 32;
      for (int b = tid; b < segs * (i1 - i0); b += kMultiThreads)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a + (int64_t)(i0 + b / segs) * ld + min((b % segs) * 32, r1 - r0 - 1)));
    }
    if (tid < 32) {
      // up to three counters, one lane each
      const int* p = nullptr;
      int want = 0;
      if ((kind & 1) == 0) {
        const int c = lane < 2 ? D.child[2 * s + lane] : -1;
        const int prev = TR ? tau + 1 : tau - 1;
        if (c >= 0) {
          p = cbase + (tau * 2 + 0) * D.nsuper + c;
          want = M.nch_f[c];
        } else if (lane == 2 && (TR ? tau < D.tau1 - 1 : tau > D.tau0)) {
          p = cbase + (prev * 2 + 1) * D.nsuper + s;
          want = M.nch_b[s];
        }
      } else if (lane == 0) {
        const int par = D.parent[s];
        p = cbase + (par < 0 ? (tau * 2 + 0) * D.nsuper + s : (tau * 2 + 1) * D.nsuper + par);
        want = par < 0 ? M.nch_f[s] : M.nch_b[par];
      }
      const bool ok = !p || wait_ge(p, want, D.status, D.spin_limit, D.spin_ns);
      const bool all = __all_sync(0xffffffffu, ok);
      if (lane == 0) s_dep = all;
    }
    __syncthreads();
    if (!s_dep) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      break;
    }
    if (claimer) flow_claim(D, s_tab, s_claims[cur ^ 1], slot, K);
    if (TR) {
      if (r1 - r0 > 64) multi_cols<K, 2>(M, R, gi, s_o, nk, tau, SQ, V);
      else multi_cols<K, 1>(M, R, gi, s_o, nk, tau, SQ, V);
    } else {
      if (kind == 0) {
        multi_gather_fwd<K, false>(M, R, gi, s_o, tau, r0, r1, low, V);
      } else {
        const int32_t* ui = D.uidx + R.map_off;
        multi_gather<K>(M.Y + ((int64_t)gi * D.N + R.first) * K, r0 - at0, n - r0, V, [&](int q2) { return r0 + q2; });
        multi_gather<K>(M.X + (int64_t)gi * D.N * K, low, m, V, [&](int q2) { return ui[q2]; });
      }
      const int G = group_lanes<float>(R.kind_len >> 8);
      const float* A0 = staged ? stage - at0 : SQ + (int64_t)r0 * ldn;
      const float* B0 = staged ? stage + ldn - at0 : Qr + (int64_t)r0 * ldm;
      const int lda = staged ? stride : ldn, ldb = staged ? stride : ldm;
      for (;;) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (kind == 0) {
          switch (G) {
            case 4: multi_rows<4, K, true>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
            case 8: multi_rows<8, K, true>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
            case 16: multi_rows<16, K, true>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
            default: multi_rows<32, K, true>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
          }
        } else {
          switch (G) {
            case 4: multi_rows<4, K, false>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
            case 8: multi_rows<8, K, false>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
            case 16: multi_rows<16, K, false>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
            default: multi_rows<32, K, false>(M, R, gi, s_o, nk, tau, b0, b1, A0, lda, B0, ldb, at0, low, own0, V); break;
          }
        }
        if (b1 >= r1) break;
        __syncthreads();  // the stage is free
        b0 = b1;
        b1 = batch_end(b0);
        stage_batch(b0, b1);
      }
    }
    __syncthreads();
    if (tid == 0) red_release_add(cbase + (tau * 2 + (kind & 1)) * D.nsuper + s, 1);
  }
}

// x[tau0] += escale * E[tau0] (forcing of the transposed chain's last bin)
__global__ void k_add_forcing(double* X, const double* E, const int* orbit_ids, int64_t N, int tau0,
                              double escale) {
  const int o = orbit_ids[blockIdx.y];
  double* x = X + ((int64_t)o * 9 + tau0) * N;
  const double* e = E + ((int64_t)o * 8 + tau0) * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
    x[i] += escale * e[i];
}

// Bytes of each task's factor rows prefetched into L2 before its dependency
// wait at large batches: the first 48 KB (ORBIT_B200_PREFETCH_KB; 0 = the
// whole task).  With every resident CTA prefetching whole backward tasks (up
// to 64 KB at the large-batch schedule) the prefetched lines can outgrow L2
// and be fetched twice; with the evict-first row loads the 12-orbit FP32
// chain took 6.43 ms with a 48 KB window, 6.46 with 32 KB, 6.49 with 64 KB,
// 6.50 with 24 KB, 6.57 with 16 KB and 6.67 with whole tasks, while at 1 and
// 4 orbits whole tasks were fastest.
int64_t prefetch_limit_bytes() {
  static const int64_t b = [] {
    const char* e = std::getenv("ORBIT_B200_PREFETCH_KB");
    const long long kb = e ? std::atoll(e) : 48;
    return kb > 0 ? (int64_t)kb * 1024 : (int64_t)1 << 40;
  }();
  return b;
}

// Sets of task groups whose phase sequences are staggered in the claim
// order (ORBIT_B200_CHAIN_SETS, default 2; 1 = all groups in lockstep):
// measured 7.49 vs 7.62 ms for the 12-orbit FP32 chain, 12.5 vs 13.3 ms FP64,
// identical results; 3 and 4 sets were slower.
int chain_phase_sets() {
  static const int v = [] {
    const char* e = std::getenv("ORBIT_B200_CHAIN_SETS");
    const int k = e ? std::atoi(e) : 2;
    return std::max(1, std::min(k, kMaxSets));
  }();
  return v;
}

// Longest sleep between polls of a completion counter (ORBIT_B200_SPIN_NS,
// default 256 ns: 2.65 vs 2.77 ms for a single-orbit FP64 chain against a
// 1 us cap, no change at 12 orbits; 4 us was slower).
// Phases between the starts of successive staggered sets (ORBIT_B200_CHAIN_GOFF;
// unset or 0: the phases of one bin divided by the number of sets).  Any
// offset keeps every dependency claimed before its dependant (dependencies stay
// inside one orbit, hence inside one set); the last set starts at most one
// bin's phases after the first, which bounds the claim-slot table.
int chain_set_offset(int nphase, int nsets) {
  static const int v = [] {
    const char* e = std::getenv("ORBIT_B200_CHAIN_GOFF");
    return e ? std::atoi(e) : 0;
  }();
  const int g = v > 0 ? v : nphase / std::max(1, nsets);
  return std::max(1, std::min(g, nphase / std::max(1, nsets - 1)));
}

unsigned chain_spin_ns() {
  static const unsigned v = [] {
    const char* e = std::getenv("ORBIT_B200_SPIN_NS");
    const long k = e ? std::atol(e) : 256;
    return (unsigned)std::max(32L, std::min(k, 8192L));
  }();
  return v;
}

// The FP32 many-right-hand-side kernels on a prepared launch: groups of K.
int launch_multi(orbit_factor_s* f, const ChainDev<float>& C, int K, const DevSym::Flow& p, int B, int trans,
                 double* X, const int* d_orbit_ids, int tau0, const double* E, double escale, int sms,
                 cudaStream_t st) {
  const Symbolic& S = f->sym->S;
  MultiDev M;
  M.C = C;
  const int64_t groups = (B + K - 1) / K;
  M.W = f->multi;
  M.Y = M.W + groups * S.w_size * K;
  M.X = M.Y + groups * S.N * K;
  M.nch_f = trans ? p.nch_f : C.nch_f;
  M.nch_b = trans ? p.nch_b : C.nch_b;
  M.C.recs = p.recs;
  M.C.phase_off = p.phase_off;
  M.C.items_per_bin = p.items_per_bin;
  M.C.total = (C.tau1 - C.tau0) * p.items_per_bin * C.B;
  const void* fn = K == 16 ? (trans ? (const void*)k_multi<16, true> : (const void*)k_multi<16, false>)
                   : K == 8 ? (trans ? (const void*)k_multi<8, true> : (const void*)k_multi<8, false>)
                            : (trans ? (const void*)k_multi<4, true> : (const void*)k_multi<4, false>);
  const size_t vectors = ((size_t)(trans ? S.max_nm : S.max_front) + 16) / 4 * 4 * K * sizeof(float);
  // columns: the partial chains of two blocks of 64 columns
  const size_t smem = std::max<size_t>(trans ? 3 * 4 * 64 * K * sizeof(float) : kMultiSmem, vectors);
  M.smem_floats = (int)(smem / sizeof(float));
  if (int r = allow_max_smem(fn)) return r;
  int occ = 0;
  ORBIT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kMultiThreads, smem));
  if (occ < 1) {
    set_last_error("chain kernel cannot be resident");
    return ORBIT_ERR_INTERNAL;
  }
  const int grid = std::min(sms * occ, M.C.total);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (f->prof_on) {
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
  }
  void* args[] = {&M};
  ORBIT_CUDA_TRY(cudaLaunchKernel(fn, dim3(grid), dim3(kMultiThreads), args, smem, st));
  note_launch();
  if (f->prof_on) {
    cudaEventRecord(e1, st);
    f->prof_chain.push_back({e0, e1});
    f->prof_chain_bytes += (double)B * (C.tau1 - C.tau0) * S.fac_nnz * sizeof(float);
  }
  if (trans && E) {
    dim3 g((unsigned)((S.N + 255) / 256), B);
    k_add_forcing<<<g, 256, 0, st>>>(X, E, d_orbit_ids, S.N, tau0, escale);
    note_launch();
    ORBIT_CUDA_TRY(cudaGetLastError());
  }
  return ORBIT_OK;
}

// Which kernel, chunk schedule and dataflow table (kFlowKinds: none) a launch of
// B slots takes.
struct SweepRoute {
  bool multi, flow, rows;  // many right-hand sides per task; tagged values; of row chunks
  int K, groups;           // right-hand sides per task, task groups per (node chunk, bin)
  int ks;
  FlowKind kind;
  int k;
};

SweepRoute sweep_route(const orbit_factor_s* f, int B, int trans, bool never_ready) {
  const Symbolic& S = f->sym->S;
  const bool fp32 = f->precision == ORBIT_PREC_FP32, sub = S.max_sub_front > 0;
  SweepRoute r;
  // Right-hand sides on one factor set go through the multi-RHS kernels in
  // groups of K (row-chunk tasks, forward and transposed sweeps).
  r.multi = !never_ready && f->n_sets == 1 && B >= 2 && !sub;
  // group size: FP64 2, FP32 the batch's, while its vectors leave a block resident
  r.K = !r.multi ? 1 : !fp32 ? 2 : B > 8 ? 16 : B > 4 ? 8 : 4;
  while (r.K > 4 && (size_t)(S.max_front + 16) * r.K * sizeof(float) > 215000) r.K /= 2;
  r.groups = (B + r.K - 1) / r.K;
  // dataflow kernels: the transposed sweeps, and the others of launches bound
  // by their dependency chain
  r.flow = !r.multi && !sub && (trans || never_ready || chain_bound(S, r.groups));
  r.rows = r.flow && !trans;
  // Schedule by batch size: small chunks shorten one orbit's critical path,
  // large ones cut per-task overhead when many orbits fill the GPU.  The
  // transposed dataflow sweeps, whose sums do not depend on the chunks, go by
  // the factor entries that one bin's sweep of all groups reads instead (2 and
  // 6 groups of the 80x72x15 grid's 52 M).
  // (The FP32 many-right-hand-side rows keep the schedule of groups of four,
  // from which their lanes per row, and so the order of their sums, follow.)
  const int Bs = r.multi && fp32 ? (B + 3) / 4 : r.groups;
  const int64_t bin_elems = (int64_t)Bs * S.fac_nnz;
  r.ks = r.flow && trans ? (bin_elems <= 110000000 && !fp32 ? 0 : bin_elems <= 330000000 ? 1 : 2)
                         : (Bs < kSchedGroups[1] ? 0 : Bs < kSchedGroups[2] ? 1 : 2);
  const bool wide = r.multi && trans;
  r.kind = r.multi ? (!fp32 ? kFlowKinds : wide ? kFlowWide : kFlowWhole)
           : !r.flow ? kFlowKinds : trans ? kFlowColumns : fp32 ? kFlowRows32 : kFlowRows64;
  r.k = wide ? 0 : r.ks;
  return r;
}

// The launch's dataflow table (null where it takes none) and the handle's
// buffers for it.
int sweep_resources(orbit_factor_s* f, const SweepRoute& r, cudaStream_t st, const DevSym::Flow** table) {
  *table = nullptr;
  if (r.kind == kFlowKinds) return ORBIT_OK;
  if (int rc = sweep_buffers(f, r.multi)) return rc;
  return flow_table(f->sym, r.kind, r.k, st, table);
}

template <typename T>
int launch_chain_t(orbit_factor_s* f, double* X, int B, const int* d_orbit_ids, int trans, int tau0,
                   int tau1, const double* E, double escale, cudaStream_t st, bool never_ready = false) {
  orbit_symbolic_s* sy = f->sym;
  const Symbolic& S = sy->S;
  ChainDev<T> D;
  D.first = sy->d.first; D.n = sy->d.n; D.m = sy->d.m; D.parent = sy->d.parent;
  D.child = sy->d.child; D.uidx = sy->d.uidx; D.rel = sy->d.rel; D.ldn = sy->d.ldn; D.ldm = sy->d.ldm;
  D.ginv = sy->d.ginv; D.ginv_off = sy->d.ginv_off;
  const SweepRoute r = sweep_route(f, B, trans, never_ready);
  const DevSym::Flow* table = nullptr;
  if (int rc = sweep_resources(f, r, st, &table)) return rc;
  const bool multi = r.multi, flow = r.flow, rows = r.rows, sub = S.max_sub_front > 0;
  const int Bt = r.groups, ks = r.ks;
  constexpr int KM = 2;  // FP64 group size
  const SolveSched& Q = S.sched[ks];
  const auto& q = sy->d.sched[ks];
  D.nch_f = trans ? q.nchunk_fwdT : q.nchunk_fwd;
  D.nch_b = trans ? q.nchunk_bwdT : q.nchunk_bwd;
  D.level = sy->d.level;
  D.sub_front = S.max_sub_front;
  D.uoff = sy->d.uoff; D.fac_off = sy->d.fac_off; D.woff = sy->d.woff;
  D.items = trans ? q.sitems + Q.items_per_bin : q.sitems;
  D.phase_off = trans ? q.phase_offT : q.phase_off;
  D.items_per_bin = trans ? Q.items_per_binT : Q.items_per_bin;
  if (flow) {
    D.recs = table->recs;
    D.phase_off = table->phase_off;
    D.items_per_bin = table->items_per_bin;
  }
  D.nphase = 2 * S.nlevels;
  if (D.nphase > kMaxPhases) {
    set_last_error("chained solve: supernode tree deeper than the kernel's phase table");
    return ORBIT_ERR_INTERNAL;
  }
  D.nsuper = S.nsuper;
  D.N = S.N; D.fac_size = S.fac_size; D.w_size = S.w_size;
  D.factors = reinterpret_cast<const T*>(f->factors);
  D.X = X; D.E = E; D.escale = escale; D.Y = f->Ybuf; D.W = f->Wbuf;
  D.counters = f->counters; D.task_counter = f->task_counter; D.status = f->status;
  D.orbit_ids = d_orbit_ids; D.B = Bt; D.Borb = B; D.tau0 = tau0; D.tau1 = tau1; D.trans = trans;
  D.set_of = f->set_of; D.n_bins = f->n_bins;
  D.total = (tau1 - tau0) * D.items_per_bin * Bt;
  D.spin_limit = never_ready ? 20000LL : 4000000LL;  // bounded: a few seconds of sleeps (<= 1 us each)
  D.never_ready = never_ready ? 1 : 0;
  D.prefetch = (sizeof(T) == 4 || B <= 6) ? 1 : 0;
  // the window bounds the prefetch only where the prefetched lines of all
  // resident CTAs outgrow L2 (large batches); small batches prefetch whole tasks
  D.prefetch_bytes = Bt > 6 ? prefetch_limit_bytes() : ((int64_t)1 << 40);
  // evict-first factor loads only where no two solve slots share a factor set
  D.stream_ef = 1;
  {
    std::vector<char> seen((size_t)std::max(f->n_sets, 1), 0);
    for (int o = 0; o < f->n_orbits && D.stream_ef; ++o) {
      const int st_o = f->h_set_of[o];
      if (st_o < 0 || st_o >= f->n_sets || seen[st_o]) D.stream_ef = 0;
      else seen[st_o] = 1;
    }
  }
  D.spin_ns = chain_spin_ns();
  D.ngroups = std::max(1, std::min(Bt, chain_phase_sets()));
  D.goff = D.ngroups > 1 ? chain_set_offset(D.nphase, D.ngroups) : 0;
  if (D.total <= 0) return ORBIT_OK;
  if (flow) {
    // tags of this launch: 16 per launch, never 0 or all ones; a handle's
    // buffers are cleared, on this stream, each time its 28-bit launch count
    // starts over, the first launch being one of those
    unsigned seq = (f->flow_seq + 1) & 0x0fffffffu;
    if (seq == 0) {
      ORBIT_CUDA_TRY(cudaMemsetAsync(f->flow, 0, 2 * sizeof(T) * (size_t)f->n_orbits * (S.w_size + 2 * S.N), st));
      seq = 1;
    }
    f->flow_seq = seq;
    D.tag0 = f->flow_seq * 16u + 1u;
    const size_t eb = sizeof(Entry<T>);
    unsigned char* p = f->flow;
    D.WF = p; p += eb * (size_t)f->n_orbits * S.w_size;
    D.YF = p; p += eb * (size_t)f->n_orbits * S.N;
    D.XF = p;
  } else {
    ORBIT_CUDA_TRY(cudaMemsetAsync(f->counters, 0, sizeof(int) * (size_t)f->n_orbits * 16 * S.nsuper, st));
  }
  ORBIT_CUDA_TRY(cudaMemsetAsync(f->task_counter, 0, sizeof(int), st));
  const size_t smem =
      rows ? kStageBytes + sizeof(T) * ((size_t)S.max_front + 8)
           : sizeof(T) * ((size_t)kWarps * 32 * (flow && sizeof(T) == 4 ? 4 : 1) +
                          std::max<size_t>(S.max_front + 8, (size_t)kWarps * ((S.max_sub_front + 7) & ~3)) + 8);
  const bool few = (double)Bt * S.fac_nnz * sizeof(T) <= chain_many_bytes(S, sizeof(T) == 8);
  const void* kfn = rows    ? (const void*)k_flow<T>
                    : flow  ? (const void*)k_flow_t<T>
                    : !sub  ? (few ? (const void*)k_chain<T, false, false, true> : (const void*)k_chain<T, false, false, false>)
                    : trans ? (const void*)k_chain<T, true, true, false>
                            : (const void*)k_chain<T, false, true, false>;
  {
    int r0 = allow_max_smem(kfn);
    if (r0) return r0;
  }
  int dev = 0, sms = 0, occ = 0;
  ORBIT_CUDA_TRY(cudaGetDevice(&dev));
  ORBIT_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if constexpr (sizeof(T) == 4)
    if (multi) return launch_multi(f, D, r.K, *table, B, trans, X, d_orbit_ids, tau0, E, escale, sms, st);
  if constexpr (sizeof(T) == 8) if (multi) {
    const int vcap = (S.max_front + 8 + 3) & ~3;
    const size_t msmem = sizeof(T) * ((size_t)KM * vcap + (size_t)KM * kWarps * 32);
    {
      int r0 = allow_max_smem((const void*)k_chain_multi<T, KM>);
      if (r0) return r0;
    }
    ORBIT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_chain_multi<T, KM>, kSolveThreads, msmem));
    if (occ < 1) {
      set_last_error("chain kernel cannot be resident");
      return ORBIT_ERR_INTERNAL;
    }
    int grid = sms * occ;
    if (grid > D.total) grid = D.total;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (f->prof_on) {
      cudaEventCreate(&e0);
      cudaEventCreate(&e1);
      cudaEventRecord(e0, st);
    }
    k_chain_multi<T, KM><<<grid, kSolveThreads, msmem, st>>>(D, vcap);
    note_launch();
    if (f->prof_on) {
      cudaEventRecord(e1, st);
      f->prof_chain.push_back({e0, e1});
      f->prof_chain_bytes += (double)B * (tau1 - tau0) * S.fac_nnz * sizeof(T);
    }
    ORBIT_CUDA_TRY(cudaGetLastError());
    if (trans && E) {
      dim3 g((unsigned)((S.N + 255) / 256), B);
      k_add_forcing<<<g, 256, 0, st>>>(X, E, d_orbit_ids, S.N, tau0, escale);
      note_launch();
      ORBIT_CUDA_TRY(cudaGetLastError());
    }
    return ORBIT_OK;
  }
  ORBIT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kfn, kSolveThreads, smem));
  if (occ < 1) {
    set_last_error("chain kernel cannot be resident");
    return ORBIT_ERR_INTERNAL;
  }
  int grid = sms * occ;
  if (grid > D.total) grid = D.total;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (f->prof_on) {
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
  }
  if (rows) k_flow<T><<<grid, kSolveThreads, smem, st>>>(D);
  else if (flow) k_flow_t<T><<<grid, kSolveThreads, smem, st>>>(D);
  else if (!sub && few) k_chain<T, false, false, true><<<grid, kSolveThreads, smem, st>>>(D);
  else if (!sub) k_chain<T, false, false, false><<<grid, kSolveThreads, smem, st>>>(D);
  else if (trans) k_chain<T, true, true, false><<<grid, kSolveThreads, smem, st>>>(D);
  else k_chain<T, false, true, false><<<grid, kSolveThreads, smem, st>>>(D);
  note_launch();
  if (f->prof_on) {
    cudaEventRecord(e1, st);
    f->prof_chain.push_back({e0, e1});
    f->prof_chain_bytes += (double)B * (tau1 - tau0) * S.fac_nnz * sizeof(T);
  }
  ORBIT_CUDA_TRY(cudaGetLastError());
  if (trans && E) {
    dim3 g((unsigned)((S.N + 255) / 256), B);
    k_add_forcing<<<g, 256, 0, st>>>(X, E, d_orbit_ids, S.N, tau0, escale);
    note_launch();
    ORBIT_CUDA_TRY(cudaGetLastError());
  }
  return ORBIT_OK;
}

}  // namespace

int prepare_sweeps(orbit_factor_s* f, int B, int trans, cudaStream_t st) {
  const DevSym::Flow* table = nullptr;
  return sweep_resources(f, sweep_route(f, B, trans, false), st, &table);
}

// Run the chain on f->X (per orbit 9 vectors in permuted order).  Forward:
// reads X[tau0], writes X[tau0+1..tau1].  Transposed: reads X[tau1], writes
// X[tau1-1..tau0].  E (permuted, per orbit 8 vectors) may be null.
int launch_chain_x(orbit_factor_s* f, double* X, int B, const int* d_orbit_ids, int trans, int tau0,
                   int tau1, const double* E, double escale, cudaStream_t st) {
  if (f->precision == ORBIT_PREC_FP32)
    return launch_chain_t<float>(f, X, B, d_orbit_ids, trans, tau0, tau1, E, escale, st);
  return launch_chain_t<double>(f, X, B, d_orbit_ids, trans, tau0, tau1, E, escale, st);
}

int launch_chain(orbit_factor_s* f, int B, const int* d_orbit_ids, int trans, int tau0, int tau1,
                 const double* E, double escale, cudaStream_t st) {
  return launch_chain_x(f, f->X, B, d_orbit_ids, trans, tau0, tau1, E, escale, st);
}

// One chain launch whose first task waits for a completion count that is
// never reached: exercises the bounded wait, the status word and the orderly
// exit of every CTA.
int chain_wait_selftest(orbit_factor_s* f, const int* d_orbit_ids, cudaStream_t st) {
  ORBIT_CUDA_TRY(cudaMemsetAsync(f->status, 0, sizeof(int), st));
  int rc = f->precision == ORBIT_PREC_FP32
               ? launch_chain_t<float>(f, f->X, 1, d_orbit_ids, 0, 0, f->n_bins, nullptr, 0.0, st, true)
               : launch_chain_t<double>(f, f->X, 1, d_orbit_ids, 0, 0, f->n_bins, nullptr, 0.0, st, true);
  if (rc) return rc;
  ORBIT_CUDA_TRY(cudaMemcpyAsync(f->h_status, f->status, sizeof(int), cudaMemcpyDeviceToHost, st));
  ORBIT_CUDA_TRY(cudaStreamSynchronize(st));
  const int code = *f->h_status;
  ORBIT_CUDA_TRY(cudaMemsetAsync(f->status, 0, sizeof(int), st));
  ORBIT_CUDA_TRY(cudaStreamSynchronize(st));
  return code;
}

}  // namespace orbit
