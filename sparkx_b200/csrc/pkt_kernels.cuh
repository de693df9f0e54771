// Device kernels of the B200 PKT k-truss engine (sm_100a).
//
// One "union" CSR holds every graph of a launch as a disjoint union (vertex
// ids, slots and edge ids offset per member), so the preparation kernels
// (narrowing, orientation, support, finalize) see a single graph.  The peel
// runs a per-member state machine: each member has its own level, phase and
// frontier, and one device "wave" advances every member by one step (a level
// scan or one PKT sub-level).  A single graph is a union of one.
//
// Layout in HBM (u32 indices: width < 2^32, m < 2^28 per member):
//   off[n+1], nbr[width]        narrowed CSR, rows sorted ascending
//   row0[width] (u64)           the same rows as (name | edge id << 32) pairs, in
//                               slot order (edge id 0xFFFFFFFF: self-loop); a
//                               vertex's name is off[v], ascending with its id
//   dplus[n], opos[n+1]         degree-ordered out-degree and its prefix
//   ocol[m], osrc[m]            oriented edge e = (osrc[e] -> ocol[e]); e is the
//                               undirected edge id; rank(osrc) < rank(ocol)
//   es[m] (int2)                per edge {support / PKT level, tag}: the tag is
//                               the wave at which the edge is processed
//                               (0xFFFFFFFF: not yet queued); one 8-byte word so
//                               a triangle's two other edges cost two sectors
//   act[2][m], q[2][m] (u64)    per-member active lists and frontier queues,
//   qd[2][m] (uint4)            with each queued edge's row descriptor;
//                               segment [eb_g, eb_g + m_g) for member g
//   working CSR (off, row)      the peel's view: row0 at first, then rebuilt
//                               without processed edges whenever the live
//                               edges fill at most 76% of it (two ping-pong
//                               buffers)
//   rank index (u64)            per row of the working CSR: where its names lie
//                               (see rank_find); rebuilt with the rows
//   vinfo[n] (u64)              per vertex: the header of its row's rank index
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace sparx {

constexpr uint32_t kInvalid = 0xFFFFFFFFu;
constexpr uint32_t kTagActive = 0xFFFFFFFFu;
constexpr int kWorkBits = 36;  // packed queue counter: (count << 36) | work
constexpr unsigned long long kWorkMask = (1ull << kWorkBits) - 1;
constexpr int kEidBits = 28;   // queue entry: (wstart << 28) | local eid
constexpr uint32_t kEidMask = (1u << kEidBits) - 1;
constexpr unsigned kFull = 0xFFFFFFFFu;

// error flags (device bitmask)
enum : uint32_t {
  kErrRange = 1u,       // neighbour id >= n
  kErrUnsorted = 2u,    // row not ascending
  kErrMulti = 4u,       // duplicate slot
  kErrAsym = 8u,        // reverse slot missing
  kErrOverflowU8 = 16u, // truss > 255 with 8-bit output / level 255 in u8 mode
  kErrCapacity = 32u,   // packed counter or queue capacity exceeded
  kErrTimeout = 64u,    // device time budget exhausted
  kErrOffsets = 128u,   // offsets not monotone / wrong total
  kErrWaves = 256u,     // wave bound exceeded (no progress)
  kErrInternal = 512u,  // inconsistent wave layout (a device loop refused to spin)
};

enum : uint32_t { kPhaseScan0 = 0, kPhaseScan = 1, kPhaseProc = 2, kPhaseDone = 3 };

struct Union {  // the prepared concatenated graph, as the peel sees it
  const uint32_t* off;             // working row offsets
  const unsigned long long* row;   // working rows: (name | edge id << 32)
  const uint32_t* opos;
  const uint32_t* ocol;
  const uint32_t* osrc;
  int2* es;
  uint32_t* act[2];
  unsigned long long* q[2];
  uint4* qd[2];                    // per queue entry {short row start, length, long row begin, end}
  const unsigned long long* rpool; // rank index of the working rows (nullptr = none)
  const unsigned long long* vinfo; // per vertex: its row's index header {smallest name, scale}, scale 0: none
  uint2* qh[2];                    // per queue entry: the longer row's index header (nullptr = no index)
  uint32_t n;
  uint32_t m;
  uint32_t width;
  uint32_t G;
};

// The peel's arrays that stay where they are for a whole run.  The wave
// kernel takes them as a by-value parameter, so the compiler can re-read any
// of them from the parameter bank instead of holding (or spilling) it; only
// the working rows, which a compaction replaces, are read from the Union.
struct PeelArrays {
  const uint32_t* ocol;
  const uint32_t* osrc;
  int2* es;
  uint32_t* act0;
  uint32_t* act1;
  unsigned long long* q0;
  unsigned long long* q1;
  uint4* qd0;
  uint4* qd1;
  const uint32_t* mu;    // multigraphs: multiplicity per edge id (nullptr: simple graph)
  const unsigned long long* rpool;
  uint2* qh0;
  uint2* qh1;
};

// Field-by-field copy of a device-resident Union into registers (a struct
// copy would land in local memory).
struct UnionRegs {
  const uint32_t* __restrict__ off;
  const unsigned long long* __restrict__ row;
  const uint32_t* __restrict__ ocol;
  const uint32_t* __restrict__ osrc;
  int2* es;
  uint32_t* act0;
  uint32_t* act1;
  unsigned long long* q0;
  unsigned long long* q1;
  uint4* qd0;
  uint4* qd1;
  const uint32_t* __restrict__ mu;
  const unsigned long long* __restrict__ rpool;
  uint2* qh0;
  uint2* qh1;
  const unsigned long long* __restrict__ vinfo;
  __device__ __forceinline__ explicit UnionRegs(const Union* p)
      : off(p->off), row(p->row), ocol(p->ocol), osrc(p->osrc), es(p->es),
        act0(p->act[0]), act1(p->act[1]), q0(p->q[0]), q1(p->q[1]),
        qd0(p->qd[0]), qd1(p->qd[1]), mu(nullptr), rpool(p->rpool), qh0(p->qh[0]), qh1(p->qh[1]), vinfo(p->vinfo) {}
  __device__ __forceinline__ UnionRegs(const Union* p, const PeelArrays& a)
      : off(p->off), row(p->row), ocol(a.ocol), osrc(a.osrc), es(a.es),
        act0(a.act0), act1(a.act1), q0(a.q0), q1(a.q1),
        qd0(a.qd0), qd1(a.qd1), mu(a.mu), rpool(a.rpool), qh0(a.qh0), qh1(a.qh1), vinfo(nullptr) {}
};

// Open-addressed hash tables of oriented lists (a tuned option of the support
// pass): 2^(1 + ceil(log2 d)) entries (at most 4d, so at 4 * the list's start
// consecutive tables never overlap), probed linearly from a multiplicative
// hash of the name; an empty entry is all ones.
__device__ __forceinline__ uint32_t hash_log2cap(uint32_t d) { return 1u + (d > 1 ? 32u - __clz(d - 1) : 0u); }
__device__ __forceinline__ uint32_t hash_first(uint32_t w, uint32_t lg) { return (w * 0x9E3779B1u) >> (32 - lg); }

struct Member {  // static per-member ranges
  uint32_t vb, n;   // vertices [vb, vb + n)
  uint32_t sb, w;   // slots [sb, sb + w)
  uint32_t eb, m;   // edge ids [eb, eb + m)
};

struct MemberState {  // dynamic per-member peel state
  uint32_t phase, level, act_sel, q_sel;
  uint32_t act_count;
  uint32_t kept;            // wave accumulator: active edges kept by a scan
  uint32_t min_kept;        // wave accumulator: min support among kept
  uint32_t processed;       // edges whose truss is fixed
  unsigned long long curr;  // packed (count << 36 | work) of the frontier being processed
  unsigned long long next;  // wave accumulator: frontier being built
  uint32_t levels, max_level, waves, pad;
};

struct Control {
  uint32_t G;
  uint32_t wave;       // current wave number (>= 1)
  uint32_t done;
  uint32_t err;
  unsigned long long total_work;
  unsigned long long max_waves;
  unsigned long long t_start;
  unsigned long long timeout_ns;
  unsigned long long waves_run;
  // work counters (roofline accounting)
  unsigned long long el_proc;     // frontier elements searched
  unsigned long long el_scan;     // active-list entries scanned
  unsigned long long hits;        // triangles found by frontier elements
  unsigned long long edges_proc;  // frontier edges processed
  unsigned long long csr_slots;   // entries in the working rows
  unsigned long long compact_min; // do not compact working rows smaller than this
  unsigned long long compact_el;  // el_proc at the last compaction
  uint32_t exit_reason;           // why the loop stopped: kExit*
  uint32_t blocks_done;           // wave blocks finished (the last one plans the next wave)
  uint32_t compactions;
  uint32_t compact_pct;           // compact when live entries fill at most this % of the working rows
  uint32_t pad0;
  unsigned long long merge_iters; // groups of 32 elements inside one frontier edge
  unsigned long long lane_iters;  // groups of 32 elements over several edges
  // optional wave trace: per planned wave {start time (ns), work, members in
  // a frontier step, members in a scan}; nullptr = off
  ulonglong4* trace;
  unsigned long long trace_cap;
  // served unions: stop when a member finishes (its result can go out at
  // once), and when the host-mapped word `admit` is set (requests wait to
  // join); nullptr / 0 = off
  const volatile uint32_t* admit;
  uint32_t notify_done;
  uint32_t pad1;
};

enum : uint32_t { kExitNone = 0, kExitDone = 1, kExitCompact = 2, kExitError = 3, kExitMember = 4, kExitAdmit = 5 };

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ uint32_t deg_of(const uint32_t* off, uint32_t v) {
  return __ldg(off + v + 1) - __ldg(off + v);
}

// degree order, ties by id: the orientation rank
__device__ __forceinline__ bool rank_less(uint32_t du, uint32_t u, uint32_t dv, uint32_t v) {
  return du < dv || (du == dv && u < v);
}

// lower_bound of x in sorted a[lo, hi)
__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* __restrict__ a, uint32_t lo,
                                                    uint32_t hi, uint32_t x) {
  while (lo < hi) {
    uint32_t mid = lo + ((hi - lo) >> 1);
    if (__ldg(a + mid) < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Position of name w in the sorted row pairs [lo, hi) or kInvalid (rows without
// a rank index).  Names inside a row are spread close to evenly, so
// up to three interpolation probes narrow a long row before the binary search:
// on a 160k-entry hub row that is ~6 dependent loads instead of ~17.
__device__ __forceinline__ uint32_t find_in_row(const unsigned long long* __restrict__ row, uint32_t lo,
                                                uint32_t hi, uint32_t w) {
#pragma unroll 1
  for (int it = 0; it < 3 && hi - lo > 48; ++it) {
    const uint32_t a = (uint32_t)__ldg(row + lo), b = (uint32_t)__ldg(row + hi - 1);
    if (w < a || w > b) return kInvalid;
    // fraction in [0, 1); the clamp keeps g in [lo, hi - 1] whatever the rounding
    const float frac = __fdividef((float)(w - a), (float)(b - a) + 1.0f);
    const uint32_t span = hi - 1 - lo;
    const uint32_t g = lo + min(span, (uint32_t)(frac * (float)span));
    const uint32_t x = (uint32_t)__ldg(row + g);
    if (x == w) return g;
    if (x < w) lo = g + 1; else hi = g;
  }
  const uint32_t end = hi;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if ((uint32_t)__ldg(row + mid) < w) lo = mid + 1; else hi = mid;
  }
  return (lo < end && (uint32_t)__ldg(row + lo) == w) ? lo : kInvalid;
}

// Warp-cooperative search over a non-decreasing key(x): the largest x in [lo, hi]
// with key(x) <= t, given key(lo) <= t.  Each step gathers 32 evenly spaced keys
// with one load per lane and keeps the stretch between the two samples that
// bracket the target, so a span of n entries costs ceil(log32 n) + 1 dependent
// gathers instead of log2 n dependent loads.  All lanes must call it with the
// same arguments.
template <class KeyF>
__device__ __forceinline__ uint32_t warp_last_le(const KeyF& key, uint32_t lo, uint32_t hi,
                                                 unsigned long long t) {
  const uint32_t lane = lane_id();
  while (hi - lo >= 32) {
    const uint32_t step = (hi - lo) / 32 + 1;
    const unsigned long long s = (unsigned long long)lo + (unsigned long long)lane * step;
    const bool le = s <= hi && key((uint32_t)s) <= t;
    const uint32_t b = __ballot_sync(kFull, le) | 1u;  // key(lo) <= t
    const uint32_t tl = 31 - __clz(b);
    lo += tl * step;
    hi = min(hi, lo + step - 1);
  }
  const bool le = lo + lane <= hi && key(lo + lane) <= t;
  const uint32_t b = __ballot_sync(kFull, le) | 1u;
  return lo + 31 - __clz(b);
}

struct PrefKey {
  const unsigned long long* p;
  __device__ __forceinline__ unsigned long long operator()(uint32_t x) const { return p[x]; }
};

__device__ __forceinline__ unsigned long long warp_incl_scan(unsigned long long v) {
  const uint32_t lane = lane_id();
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long o = __shfl_up_sync(kFull, v, d);
    if (lane >= (uint32_t)d) v += o;
  }
  return v;
}

// ---------------------------------------------------------------------------
// Kernel A: ids and offsets in, checked (u64 ids are narrowed by the host as it
// fills the staging buffers).

// u32 ids: range check, optionally copying with a base shift (dst may be null)
__global__ void k_range_ids(const uint32_t* __restrict__ ids, uint32_t* __restrict__ dst,
                            unsigned long long count, uint32_t n_limit, uint32_t base,
                            uint32_t* __restrict__ err) {
  unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  bool bad = false;
  for (; i < count; i += stride) {
    uint32_t x = __ldg(ids + i);
    bad |= x >= n_limit;
    if (dst) dst[i] = x + base;
  }
  if (bad) atomicOr(err, kErrRange);
}

// offsets u64 -> u32 (+ a member's slot base), checking monotonicity inside
// this chunk; first/last values are checked when first_expect / last_expect
// are >= 0 (device inputs), else by the host.
__global__ void k_narrow_offsets(const unsigned long long* __restrict__ src, uint32_t* __restrict__ dst,
                                 uint32_t count, uint32_t slot_base, long long first_expect,
                                 long long last_expect, uint32_t* __restrict__ err) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t stride = gridDim.x * blockDim.x;
  bool bad = false;
  for (; i < count; i += stride) {
    const unsigned long long x = src[i];
    if (i == 0 && first_expect >= 0) bad |= x != (unsigned long long)first_expect;
    if (i + 1 == count && last_expect >= 0) bad |= x != (unsigned long long)last_expect;
    if (i + 1 < count) bad |= src[i + 1] < x;
    dst[i] = (uint32_t)x + slot_base;
  }
  if (bad) atomicOr(err, kErrOffsets);
}


// A device-resident CSR in one launch: offsets narrowed and checked as by
// k_narrow_offsets (first 0, last `width`), ids checked as by k_range_ids.
__global__ void k_check_csr(const unsigned long long* __restrict__ src, uint32_t* __restrict__ off, uint32_t n,
                            const uint32_t* __restrict__ ids, unsigned long long width, uint32_t* __restrict__ err) {
  const unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  bool bad = t == 0 && (__ldg(src) != 0 || __ldg(src + n) != width), range = false;
#pragma unroll 4
  for (unsigned long long i = t; i < n; i += stride) {
    const unsigned long long x = __ldg(src + i);
    bad |= __ldg(src + i + 1) < x;
    off[i] = (uint32_t)x;
  }
  if (t == 0) off[n] = (uint32_t)width;  // as checked above
  // ids four at a time where the caller's array allows it
  const unsigned long long quads = ((uintptr_t)ids & 15) == 0 ? width / 4 : 0;
  const uint4* id4 = reinterpret_cast<const uint4*>(ids);
#pragma unroll 4
  for (unsigned long long i = t; i < quads; i += stride) {
    const uint4 v = __ldg(id4 + i);
    range |= v.x >= n || v.y >= n || v.z >= n || v.w >= n;
  }
  for (unsigned long long i = 4 * quads + t; i < width; i += stride) range |= __ldg(ids + i) >= n;
  if (bad) atomicOr(err, kErrOffsets);
  if (range) atomicOr(err, kErrRange);
}

// The input checks' verdict: kernels behind them that follow offsets or ids do
// nothing on a flagged input (the host reads the flags once, with the counts).
__device__ __forceinline__ bool bad_input(const uint32_t* err) { return __ldcg(err) & (kErrOffsets | kErrRange); }

// ---------------------------------------------------------------------------
// Exclusive scan across the block (all threads call it); `total` is the
// block sum.  smem_warp holds one value per warp.
template <class T>
__device__ __forceinline__ T block_exclusive_scan(T x, T* smem_warp, T& total) {
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  T v = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    T o = __shfl_up_sync(kFull, v, d);
    if (lane >= (uint32_t)d) v += o;
  }
  if (lane == 31) smem_warp[wid] = v;
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    T w = lane < (uint32_t)nw ? smem_warp[lane] : T(0);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      T o = __shfl_up_sync(kFull, w, d);
      if (lane >= (uint32_t)d) w += o;
    }
    if (lane < (uint32_t)nw) smem_warp[lane] = w;
  }
  __syncthreads();
  T warp_off = wid ? smem_warp[wid - 1] : T(0);
  total = smem_warp[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_off + v - x;
}

// Row kernels take 32 consecutive vertices per warp: a row of at most
// kLaneRow entries is walked by its own lane, longer rows by the whole warp
// one at a time, so low-degree vertices (most of a skewed graph) keep all
// lanes busy.
constexpr uint32_t kLaneRow = 32;

// Rows longer than kWarpRow entries are oriented by a block each (over the list
// k_degree_stats builds); the others by their lane or their warp.
constexpr uint32_t kWarpRow = 2048;

// One pass over the offsets: the rows the orientation gives a block each, the
// largest degree and the slots in rows of degree >= 256 (the degree signature
// the tuning is keyed on).  Sums stay in registers: a histogram in shared memory
// was 2.0 of the de Bruijn graph's 5.1 ms, all its vertices in two buckets.
constexpr uint32_t kHeavyRow = 256;
__global__ void __launch_bounds__(256) k_degree_stats(const uint32_t* __restrict__ off, uint32_t n,
                                                      uint32_t* __restrict__ list, uint32_t* __restrict__ count,
                                                      uint32_t* __restrict__ dmax,
                                                      unsigned long long* __restrict__ heavy,
                                                      const uint32_t* err) {
  if (bad_input(err)) return;
  uint32_t mx = 0;
  unsigned long long hv = 0;
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    const uint32_t d = __ldg(off + u + 1) - __ldg(off + u);
    mx = max(mx, d);
    if (d >= kHeavyRow) hv += d;
    if (d > kWarpRow) list[atomicAdd(count, 1u)] = u;
  }
  __shared__ unsigned long long s_hv[8];
  __shared__ uint32_t s_mx[8];
  mx = __reduce_max_sync(kFull, mx);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) hv += __shfl_xor_sync(kFull, hv, d);
  if (lane_id() == 0) {
    s_mx[threadIdx.x >> 5] = mx;
    s_hv[threadIdx.x >> 5] = hv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < blockDim.x / 32; ++w) {
      mx = max(mx, s_mx[w]);
      hv += s_hv[w];
    }
    if (mx) atomicMax(dmax, mx);
    if (hv) atomicAdd(heavy, hv);
  }
}

// Entries of a row read side by side by a lane (or a warp): what bounds the two
// passes over the rows is the latency of an entry and then its vertex's offsets.
// One / two / four: R-MAT-19 (with its degree-ordered copy) 1.78 / 1.50 / 1.35 ms of
// orientation, R-MAT-17 285 / 230 / 225 us, ER n = 10^5, m = 10^6 121 / 118 / 117.
constexpr int kOrientWays = 4;

// Kernel B1: per-row validation + oriented out-degree.
//   rows strictly ascending (equal -> multigraph), counts self-loops, and
//   dplus[u] = #{v in N(u): v != u, rank(u) < rank(v)}.
__global__ void __launch_bounds__(256) k_orient_count(const uint32_t* __restrict__ off,
                                                      const uint32_t* __restrict__ nbr, uint32_t n,
                                                      uint32_t* __restrict__ dplus,
                                                      unsigned long long* __restrict__ self_loops,
                                                      uint32_t* __restrict__ err,
                                                      uint32_t* __restrict__ max_dplus,
                                                      const uint32_t* __restrict__ big_list,
                                                      const uint32_t* __restrict__ big_count) {
  // (this kernel itself raises kErrRange only where the checks before it did)
  if (bad_input(err)) return;
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  uint32_t flags = 0, mxd = 0;
  unsigned long long selfc = 0;
  for (uint32_t base = warp * 32; base < n; base += nwarps * 32) {
    const uint32_t u = base + lane;
    uint32_t b = 0, e = 0;
    if (u < n) { b = __ldg(off + u); e = __ldg(off + u + 1); }
    uint32_t cnt = 0;
    if (u < n && e - b <= kLaneRow) {
      uint32_t prev = 0;
      for (uint32_t s = b; s < e; s += kOrientWays) {
        uint32_t vs[kOrientWays], dv[kOrientWays];
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) vs[i] = s + i < e ? __ldg(nbr + s + i) : kInvalid;
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) dv[i] = vs[i] < n ? deg_of(off, vs[i]) : 0u;
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          if (s + i >= e) break;
          const uint32_t v = vs[i];
          if (s + i > b && prev < n) {  // the pair (prev, v), judged as the warp path does
            if (v == prev) flags |= kErrMulti;
            else if (v < prev) flags |= kErrUnsorted;
          }
          prev = v;
          if (v >= n) { flags |= kErrRange; continue; }
          if (v == u) { selfc++; continue; }
          cnt += rank_less(e - b, u, dv[i], v);
        }
      }
    }
    const bool blk = u < n && e - b > kWarpRow;  // counted below, a block per row
    unsigned big = __ballot_sync(kFull, u < n && e - b > kLaneRow && !blk);
    while (big) {
      const int j = __ffs(big) - 1;
      big &= big - 1;
      const uint32_t bu = base + j, bb = __shfl_sync(kFull, b, j), be = __shfl_sync(kFull, e, j);
      const uint32_t du = be - bb;
      uint32_t c = 0;
      for (uint32_t s0 = bb + lane; s0 < be; s0 += 32 * kOrientWays) {
        uint32_t vs[kOrientWays], nx[kOrientWays], dv[kOrientWays];
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          const uint32_t s = s0 + 32 * i;
          vs[i] = s < be ? __ldg(nbr + s) : kInvalid;
          nx[i] = s < be && s + 1 < be ? __ldg(nbr + s + 1) : kInvalid;
        }
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) dv[i] = vs[i] < n ? deg_of(off, vs[i]) : 0u;
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          const uint32_t s = s0 + 32 * i, v = vs[i];
          if (s >= be) break;
          if (v >= n) { flags |= kErrRange; continue; }
          if (s + 1 < be) {
            if (nx[i] == v) flags |= kErrMulti;
            else if (nx[i] < v) flags |= kErrUnsorted;
          }
          if (v == bu) { selfc++; continue; }
          c += rank_less(du, bu, dv[i], v);
        }
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) c += __shfl_xor_sync(kFull, c, d);
      if (lane == (uint32_t)j) cnt = c;
    }
    if (u < n && !blk) {
      dplus[u] = cnt;
      mxd = max(mxd, cnt);
    }
  }
  // rows longer than kWarpRow: block-wide, one row at a time
  __shared__ unsigned long long s_red[32];
  const uint32_t nbig = *big_count;
  for (uint32_t r = blockIdx.x; r < nbig; r += gridDim.x) {
    const uint32_t bu = big_list[r];
    const uint32_t bb = __ldg(off + bu), be = __ldg(off + bu + 1), du = be - bb;
    unsigned long long c = 0;
    for (uint32_t s = bb + threadIdx.x; s < be; s += blockDim.x) {
      const uint32_t v = __ldg(nbr + s);
      if (v >= n) { flags |= kErrRange; continue; }
      if (s + 1 < be) {
        const uint32_t nx = __ldg(nbr + s + 1);
        if (nx == v) flags |= kErrMulti;
        else if (nx < v) flags |= kErrUnsorted;
      }
      if (v == bu) { selfc++; continue; }
      c += rank_less(du, bu, deg_of(off, v), v);
    }
    unsigned long long total;
    block_exclusive_scan<unsigned long long>(c, s_red, total);
    if (threadIdx.x == 0) {
      dplus[bu] = (uint32_t)total;
      mxd = max(mxd, (uint32_t)total);
    }
  }
  if (flags) atomicOr(err, flags);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    selfc += __shfl_down_sync(kFull, selfc, d);
    mxd = max(mxd, __shfl_down_sync(kFull, mxd, d));
  }
  if (lane == 0 && selfc) atomicAdd(self_loops, selfc);
  if (lane == 0 && mxd) atomicMax(max_dplus, mxd);
}

// The same for rows that were checked already and are oriented by id alone (the
// relabelled copy, whose ids ascend with the degree's power of two): an out-list
// is the row's part after u, so a search of the row gives its length (R-MAT-22 60 us,
// the pass over the slots with their degrees 1060).
__global__ void __launch_bounds__(256) k_orient_count_by_id(const uint32_t* __restrict__ off,
                                                            const uint32_t* __restrict__ nbr, uint32_t n,
                                                            uint32_t* __restrict__ dplus,
                                                            unsigned long long* __restrict__ self_loops,
                                                            uint32_t* __restrict__ max_dplus) {
  uint32_t selfc = 0, mxd = 0;
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    const uint32_t e = __ldg(off + u + 1);
    uint32_t p = lower_bound_u32(nbr, __ldg(off + u), e, u);
    if (p < e && __ldg(nbr + p) == u) {
      ++selfc;
      ++p;
    }
    dplus[u] = e - p;
    mxd = max(mxd, e - p);
  }
  selfc = __reduce_add_sync(kFull, selfc);
  mxd = __reduce_max_sync(kFull, mxd);
  if (lane_id() == 0 && selfc) atomicAdd(self_loops, (unsigned long long)selfc);
  if (lane_id() == 0 && mxd) atomicMax(max_dplus, mxd);
}

// Kernel B2: fill oriented lists (kept in id order) and, for each vertex's
// out-slots, the (name | edge id << 32) pair of row0; self-loop slots get edge id
// 0xFFFFFFFF.  In-slots get their name; their edge id is left to B3: owner[s] = u
// marks them (kInvalid for the others).  `oname` (nullptr: not wanted) takes the out-slots' names (the
// rank index's keys, off[v]).  kById: oriented by id instead of (degree, id).
__device__ __forceinline__ unsigned long long make_pair(uint32_t name, uint32_t e) {
  return (unsigned long long)name | ((unsigned long long)e << 32);
}

// the two halves of a pair
__device__ __forceinline__ uint32_t& pair_name(unsigned long long* row, unsigned long long s) {
  return reinterpret_cast<uint32_t*>(row)[2 * s];
}
__device__ __forceinline__ uint32_t& pair_eid(unsigned long long* row, unsigned long long s) {
  return reinterpret_cast<uint32_t*>(row)[2 * s + 1];
}

template <bool kById>
__global__ void __launch_bounds__(256) k_orient_fill(const uint32_t* __restrict__ off,
                                                     const uint32_t* __restrict__ nbr, uint32_t n,
                                                     const uint32_t* __restrict__ opos,
                                                     uint32_t* __restrict__ ocol,
                                                     uint32_t* __restrict__ osrc,
                                                     unsigned long long* __restrict__ row0,
                                                     uint32_t* __restrict__ owner,
                                                     const uint32_t* __restrict__ big_list,
                                                     const uint32_t* __restrict__ big_count,
                                                     uint32_t* __restrict__ oname) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t base0 = warp * 32; base0 < n; base0 += nwarps * 32) {
    const uint32_t u = base0 + lane;
    uint32_t b = 0, e = 0;
    if (u < n) { b = __ldg(off + u); e = __ldg(off + u + 1); }
    if (u < n && e - b <= kLaneRow) {
      uint32_t p = __ldg(opos + u);
      for (uint32_t s0 = b; s0 < e; s0 += kOrientWays) {
        uint32_t vs[kOrientWays], names[kOrientWays], ends[kOrientWays];
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) vs[i] = s0 + i < e ? __ldg(nbr + s0 + i) : kInvalid;
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          names[i] = vs[i] < n ? __ldg(off + vs[i]) : 0u;
          ends[i] = !kById && vs[i] < n ? __ldg(off + vs[i] + 1) : 0u;
        }
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          const uint32_t s = s0 + i, v = vs[i], name = names[i];
          if (s >= e) break;
          uint32_t own = kInvalid;
          if (v == u || v >= n) {
            row0[s] = make_pair(name, kInvalid);
          } else if (kById ? u < v : rank_less(e - b, u, ends[i] - name, v)) {
            ocol[p] = v;
            osrc[p] = u;
            if (oname) oname[p] = name;
            row0[s] = make_pair(name, p);
            ++p;
          } else {
            own = u;
            pair_name(row0, s) = name;
          }
          owner[s] = own;
        }
      }
    }
    unsigned big = __ballot_sync(kFull, u < n && e - b > kLaneRow && e - b <= kWarpRow);
    while (big) {
      const int j = __ffs(big) - 1;
      big &= big - 1;
      const uint32_t bu = base0 + j, bb = __shfl_sync(kFull, b, j), be = __shfl_sync(kFull, e, j);
      const uint32_t du = be - bb;
      uint32_t p0 = __ldg(opos + bu);
      for (uint32_t s0 = bb; s0 < be; s0 += 32 * kOrientWays) {
        uint32_t vs[kOrientWays], names[kOrientWays], ends[kOrientWays];
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          const uint32_t s = s0 + 32 * i + lane;
          vs[i] = s < be ? __ldg(nbr + s) : kInvalid;
        }
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          names[i] = vs[i] < n ? __ldg(off + vs[i]) : 0u;
          ends[i] = !kById && vs[i] < n ? __ldg(off + vs[i] + 1) : 0u;
        }
#pragma unroll
        for (int i = 0; i < kOrientWays; ++i) {
          const uint32_t s = s0 + 32 * i + lane, v = vs[i], name = names[i];
          bool out = false;
          if (s < be) {
            uint32_t own = kInvalid;
            if (v == bu || v >= n) row0[s] = make_pair(name, kInvalid);
            else if (kById ? bu < v : rank_less(du, bu, ends[i] - name, v)) out = true;
            else { own = bu; pair_name(row0, s) = name; }
            owner[s] = own;
          }
          const unsigned bal = __ballot_sync(kFull, out);
          if (out) {
            const uint32_t p = p0 + __popc(bal & ((1u << lane) - 1));
            ocol[p] = v;
            osrc[p] = bu;
            if (oname) oname[p] = name;
            row0[s] = make_pair(name, p);
          }
          p0 += __popc(bal);
        }
      }
    }
  }
  // rows longer than kWarpRow: a block per row, out-slots placed in order by
  // a block-wide scan over chunks of four consecutive slots per thread
  __shared__ uint32_t s_scan[32];
  const uint32_t nbig = *big_count;
  for (uint32_t r = blockIdx.x; r < nbig; r += gridDim.x) {
    const uint32_t bu = big_list[r];
    const uint32_t bb = __ldg(off + bu), be = __ldg(off + bu + 1), du = be - bb;
    uint32_t p0 = __ldg(opos + bu);
    for (uint32_t base = bb; base < be; base += 4 * blockDim.x) {
      const uint32_t s0 = base + 4 * threadIdx.x;
      uint32_t v[4], name[4], outm = 0, nout = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i] = name[i] = 0;
        const uint32_t s = s0 + i;
        if (s < be) {
          v[i] = __ldg(nbr + s);
          uint32_t own = kInvalid;
          if (v[i] < n) name[i] = __ldg(off + v[i]);
          if (v[i] == bu || v[i] >= n) row0[s] = make_pair(name[i], kInvalid);
          else if (kById ? bu < v[i] : rank_less(du, bu, __ldg(off + v[i] + 1) - name[i], v[i])) { outm |= 1u << i; ++nout; }
          else { own = bu; pair_name(row0, s) = name[i]; }
          owner[s] = own;
        }
      }
      uint32_t total;
      uint32_t p = p0 + block_exclusive_scan<uint32_t>(nout, s_scan, total);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (outm & (1u << i)) {
          ocol[p] = v[i];
          osrc[p] = bu;
          if (oname) oname[p] = name[i];
          row0[s0 + i] = make_pair(name[i], p);
          ++p;
        }
      p0 += total;
    }
  }
}

// Kernel B3: in-slots (owner[s] = u: rank(v) < rank(u)) take the id of v's
// out-slot to u, found by binary search in v's oriented list; slot-parallel.
// Missing -> asymmetric.
__global__ void __launch_bounds__(256) k_orient_reverse(const uint32_t* __restrict__ nbr,
                                                        const uint32_t* __restrict__ owner,
                                                        unsigned long long width,
                                                        const uint32_t* __restrict__ opos,
                                                        const uint32_t* __restrict__ ocol,
                                                        unsigned long long* __restrict__ row0,
                                                        uint32_t* __restrict__ err) {
  bool bad = false;
  for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < width;
       s += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t u = __ldg(owner + s);
    if (u == kInvalid) continue;
    const uint32_t v = __ldg(nbr + s);
    const uint32_t lo = __ldg(opos + v), hi = __ldg(opos + v + 1);
    const uint32_t p = lower_bound_u32(ocol, lo, hi, u);
    if (p < hi && __ldg(ocol + p) == u) {
      pair_eid(row0, s) = p;
    } else {
      pair_eid(row0, s) = kInvalid;
      bad = true;
    }
  }
  if (bad) atomicOr(err, kErrAsym);
}

// ---------------------------------------------------------------------------
// Exclusive scans (reduce-then-scan, 3 kernels), with the input produced by a
// functor so work values need not be materialised.
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;


template <class T, class F>
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(F f, unsigned long long count, T* tile_sums) {
  __shared__ T sw[32];
  const unsigned long long base = (unsigned long long)blockIdx.x * kScanTile;
  T acc = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    unsigned long long i = base + (unsigned long long)j * kScanThreads + threadIdx.x;
    if (i < count) acc += f(i);
  }
  T total;
  block_exclusive_scan<T>(acc, sw, total);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(T* tile_sums, unsigned long long tiles, T* grand_total) {
  __shared__ T sw[32];
  T carry = 0;
  for (unsigned long long b = 0; b < tiles; b += kScanThreads) {
    unsigned long long i = b + threadIdx.x;
    T x = i < tiles ? tile_sums[i] : T(0);
    T total;
    T ex = block_exclusive_scan<T>(x, sw, total);
    if (i < tiles) tile_sums[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) *grand_total = carry;
}

// out[i] = exclusive prefix; out[count] = total
template <class T, class F>
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(F f, unsigned long long count, const T* tile_offsets,
                                                             T* out) {
  __shared__ T sw[32];
  const unsigned long long base = (unsigned long long)blockIdx.x * kScanTile;
  // each thread owns kScanItems consecutive items
  const unsigned long long my = base + (unsigned long long)threadIdx.x * kScanItems;
  T vals[kScanItems];
  T acc = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    unsigned long long i = my + j;
    vals[j] = i < count ? f(i) : T(0);
    acc += vals[j];
  }
  T total;
  T ex = block_exclusive_scan<T>(acc, sw, total) + tile_offsets[blockIdx.x];
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    unsigned long long i = my + j;
    if (i < count) out[i] = ex;
    ex += vals[j];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[count] = ex;
}

struct LoadU32 {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator()(unsigned long long i) const { return __ldg(p + i); }
};

// support work of oriented edge e = (a -> b): min(d+(a), d+(b)); by id, an element
// of N+(a) that lies in N+(b) comes after b in N+(a), so only those are searched:
// 0.62 of the elements on R-MAT-19 and -22, whose pass goes from 41.9 to 32.2 ms
// (the credits and the shorter runs stay)
template <bool kById>
struct SupportWork {
  const uint32_t* opos;
  const uint32_t* osrc;
  const uint32_t* ocol;
  __device__ __forceinline__ unsigned long long operator()(unsigned long long e) const {
    uint32_t a = __ldg(osrc + e), b = __ldg(ocol + e);
    uint32_t da = __ldg(opos + a + 1) - (kById ? (uint32_t)e + 1 : __ldg(opos + a));
    uint32_t db = __ldg(opos + b + 1) - __ldg(opos + b);
    return min(da, db);
  }
};

// ---------------------------------------------------------------------------
// Rank index of a sorted list (or row) of d entries: 2^lg buckets, lg =
// ceil(log2 d) + 3, of the entries' names, mapped linearly from the list's own
// smallest and largest name; 32 buckets share one 8-byte word {occupied
// buckets, position of the first entry at or past the word's first bucket}.
// A search costs one word; nine in ten absent names end there (8 to 16 buckets
// per entry), a present one is at the position plus the occupied buckets below
// it (later only when two entries share a bucket, found by a binary search of
// the word's entries, so a badly clustered list costs no more than before).
// Names are a vertex's offset in the CSR: ascending with the id, and spread as
// evenly as the slots are, whatever the degrees of neighbouring ids, which is
// what the linear map needs (ids sorted by degree would fill few buckets).
// Consecutive elements of an edge ask ascending names, so a warp's 32 searches
// fall on neighbouring words and neighbouring entries, as a merge's would.
// Words lie at the list's start in the pool (fewer than d of them); the header
// is {smallest name, scale}, scale 0: no index.  kRankFine in the scale (which
// stays below it: 8 names span at least 7): twice the buckets, for hubs.
constexpr uint32_t kRankFine = 0x80000000u;
__device__ __forceinline__ uint32_t rank_shift(uint32_t d, uint32_t scale) {  // 32 - lg
  return 30 - hash_log2cap(d) - (scale >> 31);
}
__device__ __forceinline__ uint32_t rank_bucket(uint32_t name, uint32_t mn, uint32_t scale, uint32_t sh) {
  return ((name - mn) * (scale & ~kRankFine)) >> sh;
}
__device__ __forceinline__ uint32_t list_name(uint32_t x) { return x; }
__device__ __forceinline__ uint32_t list_name(unsigned long long x) { return (uint32_t)x; }

// The entry at p is below `name`, whose bucket (in a word starting at `words`)
// is bk: entries that share a bucket precede it.  Mostly it is the next one;
// else a binary search of the word's entries finds it.
template <class E>
__device__ __forceinline__ uint32_t rank_later(const E* __restrict__ arr, uint32_t p, uint32_t le,
                                               const unsigned long long* __restrict__ words, uint32_t bk, uint32_t sh,
                                               uint32_t name, E* en) {
  if (++p >= le) return kInvalid;
  *en = __ldg(arr + p);
  if (list_name(*en) < name) {
    const uint32_t j = (bk >> 5) + 1;
    const uint32_t end = j == (1u << (27 - sh)) ? le : (uint32_t)(__ldg(words + j) >> 32);
    uint32_t hi = end;
    ++p;
    while (p < hi) {
      const uint32_t mid = p + ((hi - p) >> 1);
      if (list_name(__ldg(arr + mid)) < name) p = mid + 1; else hi = mid;
    }
    if (p >= end) return kInvalid;
    *en = __ldg(arr + p);
  }
  return list_name(*en) == name ? p : kInvalid;
}

// Position of `name` in the indexed list arr[lb, le) or kInvalid; *en: the entry.
// `name` may lie outside the list's range: its bucket is then arbitrary (but
// within the 2^lg), and the entry's own name decides.
template <class E>
__device__ __forceinline__ uint32_t rank_find(const unsigned long long* __restrict__ pool,
                                              const E* __restrict__ arr, uint32_t lb, uint32_t le, uint32_t mn,
                                              uint32_t scale, uint32_t name, E* en) {
  const uint32_t sh = rank_shift(le - lb, scale);
  const uint32_t bk = rank_bucket(name, mn, scale, sh);
  const unsigned long long* words = pool + lb;
  const unsigned long long w = __ldg(words + (bk >> 5));
  const uint32_t bits = (uint32_t)w, bit = 1u << (bk & 31);
  if (!(bits & bit)) return kInvalid;
  const uint32_t p = (uint32_t)(w >> 32) + __popc(bits & (bit - 1));
  *en = __ldg(arr + p);
  const uint32_t x = list_name(*en);
  if (x < name) return rank_later(arr, p, le, words, bk, sh, name, en);
  return x == name ? p : kInvalid;
}

// Entry p of the list [b, e): the first entry of each word writes it, with the
// empty words before it; the last entry writes the empty words after it.  Every
// word is written once, by one thread, so the pool needs no clearing.
template <class E>
__device__ __forceinline__ void rank_emit(const E* __restrict__ arr, uint32_t b, uint32_t e, uint32_t p, uint32_t mn,
                                          uint32_t scale, unsigned long long* __restrict__ pool) {
  const uint32_t sh = rank_shift(e - b, scale);
  unsigned long long* wp = pool + b;
  uint32_t bk = rank_bucket(list_name(__ldg(arr + p)), mn, scale, sh);
  const uint32_t j = bk >> 5;
  // words this entry is the first at or past: (word of the entry before, j]
  uint32_t k = p == b ? 0u : (rank_bucket(list_name(__ldg(arr + p - 1)), mn, scale, sh) >> 5) + 1;
  if (k <= j) {
    for (; k < j; ++k) wp[k] = (unsigned long long)p << 32;
    uint32_t bits = 0;
    for (uint32_t q = p; (bk >> 5) == j;) {
      bits |= 1u << (bk & 31);
      if (++q == e) break;
      bk = rank_bucket(list_name(__ldg(arr + q)), mn, scale, sh);
    }
    wp[j] = bits | ((unsigned long long)p << 32);
  }
  if (p + 1 == e)
    for (k = j + 1; k < (1u << (27 - sh)); ++k) wp[k] = (unsigned long long)e << 32;
}

// Headers of all lists and the words of those of at least `min_len` entries
// (>= 8), 32 lists per warp: each qualifying list is walked by the whole warp.
// Lists longer than kRankWarpList are cut into chunks of kRankChunk entries for
// k_rank_index_chunks: with degree-ordered vertices the long lists are
// neighbours, and one warp walking 32 of 2000 entries held up the pass.  Rows of
// vertices of original degree (off0) >= fine_min > 0 get the fine index, down to
// 8 entries left; `fine_count` (or nullptr) counts them.
constexpr uint32_t kRankWarpList = 128;
constexpr uint32_t kRankChunk = 1024;
// chunks listed for lists of `w` entries together
__host__ __device__ constexpr unsigned long long rank_chunks_max(unsigned long long w) {
  return w / kRankWarpList + w / kRankChunk + 1;
}
template <class E>
__global__ void __launch_bounds__(256) k_rank_index(const uint32_t* __restrict__ off, uint32_t n, uint32_t min_len,
                                                    const E* __restrict__ arr, unsigned long long* __restrict__ pool,
                                                    unsigned long long* __restrict__ hdr,
                                                    uint2* __restrict__ chunks, uint32_t* __restrict__ chunk_count,
                                                    const uint32_t* __restrict__ off0, uint32_t fine_min,
                                                    uint32_t* __restrict__ fine_count) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t u0 = warp * 32; u0 < n; u0 += nwarps * 32) {
    const uint32_t u = u0 + lane;
    uint32_t b = 0, e = 0, mn = 0, scale = 0;
    if (u < n) {
      b = __ldg(off + u);
      e = __ldg(off + u + 1);
      const bool fine = fine_min && __ldg(off0 + u + 1) - __ldg(off0 + u) >= fine_min;
      if (e - b >= (fine ? 8u : min_len)) {
        mn = list_name(__ldg(arr + b));
        scale = 0xFFFFFFFFu / max(list_name(__ldg(arr + e - 1)) - mn, 1u);
        if (fine) {
          scale |= kRankFine;
          if (fine_count) atomicAdd(fine_count, 1u);
        }
      }
      hdr[u] = mn | ((unsigned long long)scale << 32);
    }
    const bool large = scale && e - b > kRankWarpList;
    if (large) {
      const uint32_t k = (e - b + kRankChunk - 1) / kRankChunk;
      const uint32_t at = atomicAdd(chunk_count, k);
      for (uint32_t x = 0; x < k; ++x) chunks[at + x] = make_uint2(u, x);
    }
    unsigned todo = __ballot_sync(kFull, scale && !large);
    while (todo) {
      const int j = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t rb = __shfl_sync(kFull, b, j), re = __shfl_sync(kFull, e, j);
      const uint32_t rm = __shfl_sync(kFull, mn, j), rs = __shfl_sync(kFull, scale, j);
      for (uint32_t p = rb + lane; p < re; p += 32) rank_emit(arr, rb, re, p, rm, rs, pool);
    }
  }
}

template <class E>
__global__ void __launch_bounds__(256) k_rank_index_chunks(const uint32_t* __restrict__ off,
                                                           const E* __restrict__ arr,
                                                           unsigned long long* __restrict__ pool,
                                                           const unsigned long long* __restrict__ hdr,
                                                           const uint2* __restrict__ chunks,
                                                           const uint32_t* __restrict__ chunk_count) {
  const uint32_t nc = *chunk_count;
  for (uint32_t i = blockIdx.x; i < nc; i += gridDim.x) {
    const uint2 c = chunks[i];
    const uint32_t b = __ldg(off + c.x), e = __ldg(off + c.x + 1);
    const unsigned long long h = hdr[c.x];
    const uint32_t end = min(e, b + (c.y + 1) * kRankChunk);
    for (uint32_t p = b + c.y * kRankChunk + threadIdx.x; p < end; p += blockDim.x)
      rank_emit(arr, b, e, p, (uint32_t)h, (uint32_t)(h >> 32), pool);
  }
}

// ---------------------------------------------------------------------------
// Kernel C (balanced form): per oriented edge e = (a -> b), each element of the
// shorter of N+(a), N+(b) is searched in the longer; a hit c closes the
// triangle (a, b, c), credited on e, (a -> c) and (b -> c).  Work elements are
// spread evenly over warps through the exclusive prefix `spref`; a warp owns a
// contiguous chunk and walks it 32 elements at a time.
template <class StartF>
__device__ __forceinline__ uint32_t window_find(const StartF& start, uint32_t i, uint32_t count,
                                                unsigned long long j, bool valid);

// What bounds it: issue slots (61% busy) and the latency of its three dependent
// loads (element, word, entry); the credits are a tenth of it (R-MAT-20 9.1 ms
// with them, 8.2 without).  Hence the most warps (8 blocks of 256 threads per
// SM, 32 registers), and a run of at least kSupRun elements of one edge goes
// kSupWays groups of 32 at a time with its loads side by side.  R-MAT-22 as it runs,
// on its copy oriented by id: 7.2 G elements, 32.8 ms.  The choices were measured
// on the copy oriented by degree (11.8 G elements): 40.3 ms; 42.7 / 44.0 / 43.6 at
// 7 / 6 / 5 blocks with 2 / 2 / 3 groups in flight; one group 50.0; 4 to 8 buckets
// per entry instead of 8 to 16 45; binary searches narrowed through 64 samples of
// the longer list, which the index replaced, 80.0.  R-MAT-20 15.0 -> 8.5 ms.
constexpr int kSupBlocks = 8;
constexpr int kSupRun = 24;
constexpr int kSupWays = 2;

// kMulti (multigraphs, `mu` = multiplicity per edge id): a triangle of pairs
// (e, f, h) stands for mu_e * mu_f * mu_h triangles of copies, so a copy of e
// is credited mu_f * mu_h (each hit lane adds its own product; the one-atomic
// run credit of the simple form is for unit weights only).
//
// kHash: out-lists of at least hash_min entries have an open-addressed table
// of (name | position << 32) at 4 * their start in `hpool` (k_table_fill with
// OutListSource, the same layout as the peel's row tables), probed instead of
// searched.
__device__ __forceinline__ uint32_t probe_list(const unsigned long long* __restrict__ hpool, uint32_t lb,
                                               uint32_t len, uint32_t c) {
  const uint32_t lg = hash_log2cap(len), mask = (1u << lg) - 1;
  const unsigned long long* tb = hpool + 4ull * lb;
  uint32_t at = hash_first(c, lg);
#pragma unroll 1
  for (uint32_t it = 0; it <= mask; ++it) {
    const unsigned long long en = __ldg(tb + at);
    const uint32_t id = (uint32_t)en;
    if (id == c) return (uint32_t)(en >> 32);
    if (id == kInvalid) return kInvalid;
    at = (at + 1) & mask;
  }
  return kInvalid;
}

// Credit of one hit (f, h: positions of c in the two lists) of edge e.
__device__ __forceinline__ void credit_multi(int2* __restrict__ es, const uint32_t* __restrict__ mu, uint32_t e,
                                             uint32_t f, uint32_t h, unsigned long long* found) {
  const uint32_t me = __ldg(mu + e), mf = __ldg(mu + f), mh = __ldg(mu + h);
  atomicAdd(&es[f].x, (int)(me * mh));
  atomicAdd(&es[h].x, (int)(me * mf));
  atomicAdd(&es[e].x, (int)(mf * mh));
  *found += (unsigned long long)me * mf * mh;
}

// `oname`: the lists' keys, ascending in each list (the ids themselves when
// there is no index); `hdr` / `pool`: rank index of the lists of at least
// rank_min entries (hdr nullptr: none).
//
// kById: the graph is oriented by id (see SupportWork), and N+(a) takes part as
// its entries after b where it is the shorter list.
template <bool kMulti, bool kHash, bool kById>
__global__ void __launch_bounds__(256, kSupBlocks) k_support_balanced(
    const uint32_t* __restrict__ opos, const uint32_t* __restrict__ ocol,
    const uint32_t* __restrict__ osrc, const uint32_t* __restrict__ oname,
    const unsigned long long* __restrict__ spref, uint32_t m,
    int2* __restrict__ es, unsigned long long* __restrict__ tri_total,
    const uint32_t* __restrict__ mu, uint32_t rank_min, const unsigned long long* __restrict__ hdr,
    const unsigned long long* __restrict__ pool, const unsigned long long* __restrict__ hpool,
    uint32_t hash_min) {
  const uint32_t lane = lane_id();
  const unsigned long long total = spref[m];
  const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  unsigned long long ch = total / (nwarps * 4);
  ch = min(max((ch + 31) & ~31ull, 32ull), 4096ull);
  const PrefKey ps{spref};
  unsigned long long found_total = 0;
  for (unsigned long long c0 = warp * ch; c0 < total; c0 += nwarps * ch) {
    const unsigned long long kend = min(c0 + ch, total);
    uint32_t i = warp_last_le(PrefKey{spref}, 0, m - 1, c0);
    for (unsigned long long kb = c0; kb < kend;) {
      // edge i owns element kb (or has none left: then some later edge does)
      const unsigned long long e_start = spref[i], e_end = min(kend, spref[i + 1]);
      if (e_end >= kb + kSupRun) {
        // the rest of a long edge: its lists are the same for the whole warp
        const uint32_t a = __ldg(osrc + i), b = __ldg(ocol + i);
        const uint32_t ab = __ldg(opos + a), ae = __ldg(opos + a + 1);
        const uint32_t bb = __ldg(opos + b), be = __ldg(opos + b + 1);
        const uint32_t as = kById ? i + 1 : ab;  // the elements of N+(a)
        const bool a_short = ae - as <= be - bb;
        const uint32_t flb = a_short ? bb : ab, fle = a_short ? be : ae;
        const unsigned long long fh = hdr && fle - flb >= rank_min ? __ldg(hdr + (a_short ? b : a)) : 0ull;
        const uint32_t mn = (uint32_t)fh, scale = (uint32_t)(fh >> 32);
        const bool hashed = kHash && fle - flb >= hash_min;
        const uint32_t f0 = (a_short ? as : bb) + (uint32_t)(kb - e_start);
        const uint32_t f1 = f0 + (uint32_t)(e_end - kb);
        int cnt = 0;
        auto credit = [&](uint32_t f, uint32_t q) {
          if (kMulti) {
            credit_multi(es, mu, i, f, q, &found_total);
          } else {
            atomicAdd(&es[f].x, 1);
            atomicAdd(&es[q].x, 1);
            ++cnt;
          }
        };
        if (scale && !hashed) {
          // kSupWays groups of 32 at a time: their words, then their entries,
          // are loaded together
          const uint32_t sh = rank_shift(fle - flb, scale);
          const unsigned long long* words = pool + flb;
          for (uint32_t f = f0 + lane; f < f1; f += 32 * kSupWays) {
            uint32_t c[kSupWays], p[kSupWays], x[kSupWays];
            unsigned long long w[kSupWays];
#pragma unroll
            for (int j = 0; j < kSupWays; ++j) c[j] = f + 32 * j < f1 ? __ldg(oname + f + 32 * j) : mn;
#pragma unroll
            for (int j = 0; j < kSupWays; ++j) {
              p[j] = ((c[j] - mn) * scale) >> sh;
              w[j] = __ldg(words + (p[j] >> 5));
            }
#pragma unroll
            for (int j = 0; j < kSupWays; ++j) {
              const uint32_t bit = 1u << (p[j] & 31);
              const bool maybe = ((uint32_t)w[j] & bit) && f + 32 * j < f1;
              p[j] = maybe ? (uint32_t)(w[j] >> 32) + __popc((uint32_t)w[j] & (bit - 1)) : kInvalid;
              x[j] = maybe ? __ldg(oname + p[j]) : 0xFFFFFFFFu;
            }
#pragma unroll
            for (int j = 0; j < kSupWays; ++j) {
              if (x[j] < c[j]) p[j] = rank_later(oname, p[j], fle, words, ((c[j] - mn) * scale) >> sh, sh, c[j], &x[j]);
              if (x[j] == c[j] && p[j] != kInvalid) credit(f + 32 * j, p[j]);
            }
          }
        } else {
          for (uint32_t f = f0 + lane; f < f1; f += 32) {
            const uint32_t c = __ldg(oname + f);
            if (hashed) {
              const uint32_t q = probe_list(hpool, flb, fle - flb, c);
              if (q != kInvalid) credit(f, q);
            } else {
              const uint32_t q = lower_bound_u32(oname, flb, fle, c);
              if (q < fle && __ldg(oname + q) == c) credit(f, q);
            }
          }
        }
        if (!kMulti) {  // the edge's own credit, once per run
          found_total += cnt;
          cnt = __reduce_add_sync(kFull, cnt);
          if (lane == 0 && cnt) atomicAdd(&es[i].x, cnt);
        }
        kb = e_end;
        i = min(i + 1, m - 1);
        continue;
      }
      // short edges: 32 elements, each lane finds its own edge and lists
      const unsigned long long k = kb + lane;
      const bool valid = k < kend;
      const uint32_t e = window_find(ps, i, m, k, valid);
      const uint32_t last = (uint32_t)min(31ull, kend - 1 - kb);
      const uint32_t e_last = __shfl_sync(kFull, e, last);
      uint32_t o = 0, sb = 0, lb = 0, le = 0, lv = 0;
      if (valid) {
        o = (uint32_t)(k - spref[e]);
        const uint32_t a = __ldg(osrc + e), b = __ldg(ocol + e);
        const uint32_t ab = __ldg(opos + a), ae = __ldg(opos + a + 1);
        const uint32_t bb = __ldg(opos + b), be = __ldg(opos + b + 1);
        const uint32_t as = kById ? e + 1 : ab;
        if (ae - as <= be - bb) { sb = as; lb = bb; le = be; lv = b; }
        else { sb = bb; lb = ab; le = ae; lv = a; }
      }
      uint32_t p = kInvalid;  // position of c in the longer list
      if (valid) {
        const uint32_t c = __ldg(oname + sb + o);
        if (kHash && le - lb >= hash_min) {
          p = probe_list(hpool, lb, le - lb, c);
        } else if (hdr && le - lb >= rank_min) {
          const unsigned long long h = __ldg(hdr + lv);
          uint32_t en;
          p = rank_find(pool, oname, lb, le, (uint32_t)h, (uint32_t)(h >> 32), c, &en);
        } else {
          const uint32_t q = lower_bound_u32(oname, lb, le, c);
          if (q < le && __ldg(oname + q) == c) p = q;
        }
      }
      const bool hit = valid && p != kInvalid;
      if (kMulti) {
        if (hit) credit_multi(es, mu, e, sb + o, p, &found_total);
      } else {
        if (hit) {
          atomicAdd(&es[sb + o].x, 1);
          atomicAdd(&es[p].x, 1);
          found_total++;
        }
        // credit e once per run of lanes sharing it
        const unsigned hits = __ballot_sync(kFull, hit);
        const unsigned grp = __match_any_sync(kFull, valid ? e : kInvalid);
        if (valid && lane == (uint32_t)(__ffs(grp) - 1)) {
          const int cnt = __popc(grp & hits);
          if (cnt) atomicAdd(&es[e].x, cnt);
        }
      }
      i = e_last;
      kb += 32;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) found_total += __shfl_down_sync(kFull, found_total, d);
  if (lane == 0 && found_total) atomicAdd(tri_total, found_total);
}

// Kernel C (pair form): every oriented list is short (at most kPairList entries),
// so a thread walks its edge's two lists side by side; no prefix over the edges
// and no searches.  Bound by the gathers of the two lists (a sector each) and the
// edges' 24 bytes: de Bruijn graph (24.7 M edges, lists of 4 at most) 0.23 ms against
// 0.76 balanced, ER n = 10^5, m = 10^6 79 against 126 us, n = 10^6, m = 10^7 0.55
// against 0.90 ms; with lists of up to 64 entries (m = 2 M) 0.20 against 0.36 ms.
constexpr uint32_t kPairList = 64;
template <bool kMulti>
__global__ void __launch_bounds__(256) k_support_pairs(const uint32_t* __restrict__ opos,
                                                       const uint32_t* __restrict__ ocol,
                                                       const uint32_t* __restrict__ osrc, uint32_t m,
                                                       int2* __restrict__ es,
                                                       unsigned long long* __restrict__ tri_total,
                                                       unsigned long long* __restrict__ elements,
                                                       const uint32_t* __restrict__ mu) {
  unsigned long long found = 0, els = 0;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
    const uint32_t a = __ldg(osrc + e), b = __ldg(ocol + e);
    uint32_t i = __ldg(opos + a), j = __ldg(opos + b);
    const uint32_t ie = __ldg(opos + a + 1), je = __ldg(opos + b + 1);
    els += min(ie - i, je - j);
    int cnt = 0;
    if (i < ie && j < je) {
      uint32_t x = __ldg(ocol + i), y = __ldg(ocol + j);
      for (;;) {
        if (x == y) {
          if (kMulti) {
            credit_multi(es, mu, e, i, j, &found);
          } else {
            atomicAdd(&es[i].x, 1);
            atomicAdd(&es[j].x, 1);
            ++cnt;
          }
        }
        const bool both = x == y;
        if (x < y || both) {
          if (++i == ie) break;
          x = __ldg(ocol + i);
        }
        if (y < x || both) {  // x may have moved on: it is then above the old y, or y is still behind it
          if (++j == je) break;
          y = __ldg(ocol + j);
        }
      }
    }
    if (!kMulti && cnt) {
      atomicAdd(&es[e].x, cnt);
      found += cnt;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    found += __shfl_xor_sync(kFull, found, d);
    els += __shfl_xor_sync(kFull, els, d);
  }
  if (lane_id() == 0) {
    if (found) atomicAdd(tri_total, found);
    if (els) atomicAdd(elements, els);
  }
}

// ---------------------------------------------------------------------------
// Kernel C (vertex form).  Each triangle a < b < c (orientation rank) is found
// once, from its lowest vertex a: N+(a) is hashed into shared memory, then the
// out-lists N+(b) of every b in N+(a) are streamed with coalesced loads and
// probed against the table.  Of the three credits, (a -> b) and (a -> c) land
// in shared-memory counters for a's out-list, flushed once per vertex; only
// (b -> c) is a global atomic.  Light vertices (out-degree <= kLightMax) take
// one warp each; heavier ones one CTA each (k_support_heavy).
constexpr int kLightMax = 64;
constexpr int kLightSlots = 128;

__device__ __forceinline__ uint32_t hash_slot(uint32_t c, uint32_t shift) {
  return (c * 0x9E3779B1u) >> shift;
}

// insert key c -> j (table has >= 2x slots, so a free slot always exists)
__device__ __forceinline__ void table_insert(uint32_t* keys, uint16_t* vals, uint32_t mask, uint32_t shift,
                                             uint32_t c, uint32_t j) {
  uint32_t h = hash_slot(c, shift);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const uint32_t old = atomicCAS(keys + h, kInvalid, c);
    if (old == kInvalid) { vals[h] = (uint16_t)j; return; }
    h = (h + 1) & mask;
  }
}

__device__ __forceinline__ uint32_t table_find(const uint32_t* keys, const uint16_t* vals, uint32_t mask,
                                               uint32_t shift, uint32_t c) {
  uint32_t h = hash_slot(c, shift);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const uint32_t k = keys[h];
    if (k == c) return vals[h];
    if (k == kInvalid) return kInvalid;
    h = (h + 1) & mask;
  }
  return kInvalid;
}

__device__ __forceinline__ uint32_t log2_pow2(uint32_t t) { return 31 - __clz(t); }

__global__ void __launch_bounds__(256) k_support_light(const uint32_t* __restrict__ opos,
                                                       const uint32_t* __restrict__ ocol, uint32_t n,
                                                       int2* __restrict__ es, unsigned long long* __restrict__ tri_total,
                                                       uint32_t* __restrict__ heavy_list,
                                                       uint32_t* __restrict__ heavy_count,
                                                       uint32_t* __restrict__ vcursor) {
  __shared__ uint32_t s_key[8][kLightSlots];
  __shared__ uint16_t s_val[8][kLightSlots];
  __shared__ uint32_t s_cnt[8][kLightMax];
  const uint32_t lane = lane_id(), wib = threadIdx.x >> 5;
  uint32_t* keys = s_key[wib];
  uint16_t* vals = s_val[wib];
  uint32_t* cnt = s_cnt[wib];
  unsigned long long tri = 0;
  for (;;) {
    uint32_t v0 = 0;
    if (lane == 0) v0 = atomicAdd(vcursor, 32u);
    v0 = __shfl_sync(kFull, v0, 0);
    if (v0 >= n) break;
    const uint32_t va = v0 + lane;
    const uint32_t dv = va < n ? __ldg(opos + va + 1) - __ldg(opos + va) : 0u;
    const bool heavy = dv > (uint32_t)kLightMax;
    const unsigned hb = __ballot_sync(kFull, heavy);
    if (hb) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(heavy_count, (uint32_t)__popc(hb));
      at = __shfl_sync(kFull, at, 0);
      if (heavy) heavy_list[at + __popc(hb & ((1u << lane) - 1))] = va;
    }
    unsigned todo = __ballot_sync(kFull, dv >= 2 && !heavy);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t a = v0 + src;
      const uint32_t da = __shfl_sync(kFull, dv, src);
      const uint32_t base = __ldg(opos + a);
      uint32_t T = 8;
      while (T < 2 * da) T <<= 1;
      const uint32_t mask = T - 1, shift = 32 - log2_pow2(T);
      for (uint32_t s = lane; s < T; s += 32) keys[s] = kInvalid;
      if (lane < da) cnt[lane] = 0;
      if (lane + 32 < da) cnt[lane + 32] = 0;
      __syncwarp();
      const uint32_t b0 = lane < da ? __ldg(ocol + base + lane) : kInvalid;
      const uint32_t b1 = lane + 32 < da ? __ldg(ocol + base + lane + 32) : kInvalid;
      if (b0 != kInvalid) table_insert(keys, vals, mask, shift, b0, lane);
      if (b1 != kInvalid) table_insert(keys, vals, mask, shift, b1, lane + 32);
      // out-lists of the b's: start and length, exclusive prefix over lengths
      const uint32_t p0 = b0 != kInvalid ? __ldg(opos + b0) : 0u;
      const uint32_t l0 = b0 != kInvalid ? __ldg(opos + b0 + 1) - p0 : 0u;
      const uint32_t p1 = b1 != kInvalid ? __ldg(opos + b1) : 0u;
      const uint32_t l1 = b1 != kInvalid ? __ldg(opos + b1 + 1) - p1 : 0u;
      const uint32_t i0 = (uint32_t)warp_incl_scan(l0), t0 = __shfl_sync(kFull, i0, 31);
      const uint32_t i1 = (uint32_t)warp_incl_scan(l1) + t0, total = __shfl_sync(kFull, i1, 31);
      // exclusive starts; entries past the list never match (start = max)
      const uint32_t x0 = lane < da ? i0 - l0 : kInvalid;
      const uint32_t x1 = lane + 32 < da ? i1 - l1 : kInvalid;
      __syncwarp();
      for (uint32_t f0 = 0; f0 < total; f0 += 32) {
        const uint32_t f = f0 + lane;
        // entry owning f: largest index with start <= f, over 64 entries
        uint32_t t = 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
          const uint32_t cand = __shfl_sync(kFull, x0, t + d);
          if (cand <= f) t += d;
        }
        uint32_t u = 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
          const uint32_t cand = __shfl_sync(kFull, x1, u + d);
          if (cand <= f) u += d;
        }
        const uint32_t x1_0 = __shfl_sync(kFull, x1, 0);
        const uint32_t xt = __shfl_sync(kFull, x0, t), pt = __shfl_sync(kFull, p0, t);
        const uint32_t xu = __shfl_sync(kFull, x1, u), pu = __shfl_sync(kFull, p1, u);
        const bool hi = x1_0 <= f;  // entry index >= 32
        const uint32_t i = hi ? 32 + u : t;
        const uint32_t start = hi ? xu : xt, pos = hi ? pu : pt;
        bool hit = false;
        if (f < total) {
          const uint32_t at = pos + (f - start);
          const uint32_t c = __ldg(ocol + at);
          const uint32_t j = table_find(keys, vals, mask, shift, c);
          if (j != kInvalid) {
            hit = true;
            atomicAdd(cnt + j, 1u);    // a -> c
            atomicAdd(cnt + i, 1u);    // a -> b
            atomicAdd(&es[at].x, 1);   // b -> c
          }
        }
        tri += hit;
      }
      __syncwarp();
      if (lane < da && cnt[lane]) atomicAdd(&es[base + lane].x, (int)cnt[lane]);
      if (lane + 32 < da && cnt[lane + 32]) atomicAdd(&es[base + lane + 32].x, (int)cnt[lane + 32]);
      __syncwarp();
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) tri += __shfl_down_sync(kFull, tri, d);
  if (lane == 0 && tri) atomicAdd(tri_total, tri);
}

// Heavy vertices: one CTA each, table of `slots` entries in dynamic shared
// memory (slots >= 2 * max out-degree), lists of the b's staged in shared memory.
__global__ void __launch_bounds__(256) k_support_heavy(const uint32_t* __restrict__ opos,
                                                       const uint32_t* __restrict__ ocol,
                                                       int2* __restrict__ es, unsigned long long* __restrict__ tri_total,
                                                       const uint32_t* __restrict__ heavy_list,
                                                       const uint32_t* __restrict__ heavy_count,
                                                       uint32_t* __restrict__ hcursor, uint32_t slots,
                                                       uint32_t max_deg) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* keys = (uint32_t*)smem;                       // slots
  uint32_t* cnt = keys + slots;                           // max_deg
  uint32_t* pre = cnt + max_deg;                          // max_deg + 1 exclusive starts
  uint32_t* bpos = pre + max_deg + 1;                     // max_deg list starts
  uint16_t* vals = (uint16_t*)(bpos + max_deg);           // slots
  __shared__ uint32_t s_a, s_sum[32];
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t nheavy = *heavy_count;
  unsigned long long tri = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      const uint32_t h = atomicAdd(hcursor, 1u);
      s_a = h < nheavy ? heavy_list[h] : kInvalid;
    }
    __syncthreads();
    const uint32_t a = s_a;
    if (a == kInvalid) break;
    const uint32_t base = __ldg(opos + a), d = __ldg(opos + a + 1) - base;
    uint32_t T = 8;
    while (T < 2 * d) T <<= 1;
    const uint32_t mask = T - 1, shift = 32 - log2_pow2(T);
    for (uint32_t s = threadIdx.x; s < T; s += blockDim.x) keys[s] = kInvalid;
    for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    // insert N+(a), record the b lists, exclusive prefix of their lengths
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < d; i0 += blockDim.x) {
      const uint32_t i = i0 + threadIdx.x;
      uint32_t len = 0;
      if (i < d) {
        const uint32_t b = __ldg(ocol + base + i);
        table_insert(keys, vals, mask, shift, b, i);
        const uint32_t pb = __ldg(opos + b);
        len = __ldg(opos + b + 1) - pb;
        bpos[i] = pb;
      }
      uint32_t total;
      const uint32_t ex = block_exclusive_scan<uint32_t>(len, s_sum, total);
      if (i < d) pre[i] = carry + ex;
      carry += total;
    }
    if (threadIdx.x == 0) pre[d] = carry;
    __syncthreads();
    const uint32_t total = carry;
    for (uint32_t f0 = wid * 32; f0 < total; f0 += nw * 32) {
      const uint32_t f = f0 + lane;
      if (f < total) {
        // entry owning f: largest i with pre[i] <= f (entries with no out-list
        // share their start with the next entry and are skipped)
        uint32_t lo = 0, hi = d - 1;
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          if (pre[mid] <= f) lo = mid; else hi = mid - 1;
        }
        const uint32_t at = bpos[lo] + (f - pre[lo]);
        const uint32_t c = __ldg(ocol + at);
        const uint32_t j = table_find(keys, vals, mask, shift, c);
        if (j != kInvalid) {
          atomicAdd(cnt + j, 1u);
          atomicAdd(cnt + lo, 1u);
          atomicAdd(&es[at].x, 1);
          ++tri;
        }
      }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < d; i += blockDim.x)
      if (cnt[i]) atomicAdd(&es[base + i].x, (int)cnt[i]);
    __syncthreads();
  }
#pragma unroll
  for (int dd = 16; dd > 0; dd >>= 1) tri += __shfl_down_sync(kFull, tri, dd);
  if (lane == 0 && tri) atomicAdd(tri_total, tri);
}

// dynamic shared memory of k_support_heavy for a given max out-degree
__host__ __device__ inline size_t heavy_smem_bytes(uint32_t slots, uint32_t max_deg) {
  return (size_t)slots * 4 + (size_t)max_deg * 4 * 3 + 4 + (size_t)slots * 2;
}

// ---------------------------------------------------------------------------
// Peel setup: u8 wrap (u8 mode), per-member triangle sums and max support,
// tags cleared, identity active lists (local ids inside each member's segment).
// Per-lane running sums are flushed when the member changes, then reduced per
// warp, so a single member costs one atomic per warp.
__device__ __forceinline__ void flush_member_stats(uint32_t g, unsigned long long sum, uint32_t mx,
                                                   unsigned long long* mem_tri, uint32_t* mem_maxsup) {
  if (g == kInvalid) return;
  if (sum) atomicAdd(mem_tri + g, sum);
  if (mx) atomicMax(mem_maxsup + g, mx);
}

// Multigraphs (mu != nullptr): a pair's support is per copy, so its triangle
// credits are support * mu; a support that wrapped past 2^31 is a capacity error.
// Edges [e_begin, m): all of them, or those of members that join a served union.
__global__ void __launch_bounds__(256) k_peel_setup(const Union* __restrict__ Up, const Member* __restrict__ mem,
                                                    int u8mode, unsigned long long* __restrict__ mem_tri,
                                                    uint32_t* __restrict__ mem_maxsup,
                                                    const uint32_t* __restrict__ mu, uint32_t* __restrict__ err,
                                                    uint32_t e_begin = 0) {
  const Union U = *Up;
  const uint32_t G = U.G;
  uint32_t cur = kInvalid;
  unsigned long long sum = 0;
  uint32_t mx = 0;
  for (uint32_t e = e_begin + blockIdx.x * blockDim.x + threadIdx.x; e < U.m; e += gridDim.x * blockDim.x) {
    uint32_t g = 0;
    if (G > 1) {
      uint32_t lo = 0, hi = G - 1;
      while (lo < hi) {
        uint32_t mid = (lo + hi + 1) >> 1;
        if (mem[mid].eb <= e) lo = mid; else hi = mid - 1;
      }
      g = lo;
    }
    if (g != cur) {
      flush_member_stats(cur, sum, mx, mem_tri, mem_maxsup);
      cur = g; sum = 0; mx = 0;
    }
    int32_t s = U.es[e].x;
    if (mu) {
      if (s < 0) atomicOr(err, kErrCapacity);
      sum += (unsigned long long)(uint32_t)s * __ldg(mu + e);
    } else {
      sum += (unsigned long long)s;
    }
    if (u8mode) s &= 0xFF;
    U.es[e] = make_int2(s, (int)kTagActive);
    mx = max(mx, (uint32_t)s);
    U.act[0][e] = e - mem[g].eb;
  }
  // warp reduction when every lane ends on the same member
  const unsigned same = __match_any_sync(kFull, cur);
  if (same == kFull) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      sum += __shfl_down_sync(kFull, sum, d);
      mx = max(mx, __shfl_down_sync(kFull, mx, d));
    }
    if (lane_id() == 0) flush_member_stats(cur, sum, mx, mem_tri, mem_maxsup);
  } else {
    flush_member_stats(cur, sum, mx, mem_tri, mem_maxsup);
  }
}

// first wave: every member scans all its edges at level 0
__global__ void k_peel_init(const Member* __restrict__ mem, MemberState* __restrict__ st, Control* ctl,
                            unsigned long long* __restrict__ wpref, uint32_t G) {
  // single block: prefix of m_g
  __shared__ unsigned long long sw[32];
  unsigned long long carry = 0;
  for (uint32_t b = 0; b < G; b += blockDim.x) {
    const uint32_t g = b + threadIdx.x;
    unsigned long long w = 0;
    if (g < G) {
      MemberState s{};
      s.phase = mem[g].m ? kPhaseScan0 : kPhaseDone;
      s.act_count = mem[g].m;
      s.min_kept = 0xFFFFFFFFu;
      st[g] = s;
      w = s.phase == kPhaseDone ? 0 : mem[g].m;
    }
    unsigned long long total;
    unsigned long long ex = block_exclusive_scan<unsigned long long>(w, sw, total);
    if (g < G) wpref[g] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) {
    wpref[G] = carry;
    ctl->total_work = carry;
    ctl->wave = 1;
    ctl->done = carry == 0;
    ctl->waves_run = 0;
    ctl->el_scan = carry;
    ctl->t_start = globaltimer();
  }
}

// A single graph's peel state in one launch: the union, its member and the loop
// control (by value), the member's sums cleared, its first wave the level-0 scan.
__global__ void k_peel_begin(Union U, Union* dU, Member M, Member* mem, Control c, Control* ctl, MemberState* st,
                             unsigned long long* wpref, unsigned long long* mem_tri, uint32_t* mem_maxsup) {
  *dU = U;
  *mem = M;
  *mem_tri = 0;
  *mem_maxsup = 0;
  MemberState s{};
  s.phase = M.m ? kPhaseScan0 : kPhaseDone;
  s.act_count = M.m;
  s.min_kept = 0xFFFFFFFFu;
  *st = s;
  wpref[0] = 0;
  wpref[1] = M.m;
  c.total_work = M.m;
  c.wave = 1;
  c.done = M.m == 0;
  c.el_scan = M.m;
  c.t_start = globaltimer();
  *ctl = c;
}

struct WaveArgs {
  const Union* Up;     // working rows (replaced by compactions)
  PeelArrays arr;      // everything else the wave reads, by value
  const Member* mem;
  MemberState* st;
  Control* ctl;
  unsigned long long* wpref;
  uint32_t* err;
  cudaGraphConditionalHandle handle;  // WHILE condition of the peel graph
  int use_handle;                     // 0: waves are launched by the host
};

// Rows of frontier edge x in the working CSR: {shorter row start, its length,
// longer row begin, longer row end}.  The length is the edge's work.  *hq: the
// longer row's index header, or {0, 0}.
__device__ __forceinline__ uint4 edge_desc(const UnionRegs& U, uint32_t x, uint2* hq) {
  const uint32_t u = __ldg(U.osrc + x), v = __ldg(U.ocol + x);
  // row bounds and both rows' index headers, all in one round of loads
  const uint32_t ub = __ldg(U.off + u), ue = __ldg(U.off + u + 1);
  const uint32_t vb = __ldg(U.off + v), ve = __ldg(U.off + v + 1);
  const unsigned long long iu = U.vinfo ? __ldg(U.vinfo + u) : 0ull, iv = U.vinfo ? __ldg(U.vinfo + v) : 0ull;
  const bool u_short = ue - ub <= ve - vb;
  const unsigned long long li = u_short ? iv : iu;
  *hq = make_uint2((uint32_t)li, (uint32_t)(li >> 32));
  return u_short ? make_uint4(ub, ue - ub, vb, ve) : make_uint4(vb, ve - vb, ub, ue);
}

// PKT sub-level rule for one triangle (e, f, h) of frontier edge e at level l,
// wave W (pkt.rs:409-479 restated on undirected edge ids):
//   f or h processed (tag < W)         -> nothing
//   both above l                        -> charge both
//   only f above l                      -> charge f unless h is in this frontier
//                                          with a smaller id than e
//   only h above l                      -> symmetric
// A charge that takes the support from above l to l or below queues the edge
// for the next sub-level; a charge that goes below l is restored to l.
//
// A charge is 1 in a simple graph.  In a multigraph (kMulti) a triangle of
// pairs stands for mu_e * mu_f * mu_h triangles of copies, and peeling e
// removes mu_e * mu_h of them from each copy of f (mu_e * mu_f from h): the
// charge is that product, applied at once.
template <bool kMulti>
__device__ __forceinline__ void pkt_rule(const UnionRegs& U, uint32_t e, uint32_t f, int2 es_f, uint32_t h, int2 es_h,
                                         uint32_t l, uint32_t W, bool& pf, bool& ph) {
  pf = ph = false;
  const uint32_t tf = (uint32_t)es_f.y, th = (uint32_t)es_h.y;
  if (tf < W || th < W) return;
  const int32_t sf = es_f.x, sh = es_h.x;
  const int32_t L = (int32_t)l;
  bool df = false, dh = false;
  if (sf > L && sh > L) { df = true; dh = true; }
  else if (sf > L) df = (e < h) || (th != W);
  else if (sh > L) dh = (e < f) || (tf != W);
  int32_t cf = 1, ch = 1;
  if (kMulti && (df || dh)) {
    const int32_t me = (int32_t)__ldg(U.mu + e), mf = (int32_t)__ldg(U.mu + f), mh = (int32_t)__ldg(U.mu + h);
    cf = me * mh;
    ch = me * mf;
  }
  if (df) {
    int32_t prev = atomicSub(&U.es[f].x, cf);
    if (prev > L && prev - cf <= L) pf = true;
    if (prev - cf < L) atomicMax(&U.es[f].x, L);
  }
  if (dh) {
    int32_t prev = atomicSub(&U.es[h].x, ch);
    if (prev > L && prev - ch <= L) ph = true;
    if (prev - ch < L) atomicMax(&U.es[h].x, L);
  }
}

// Entry lookup for a warp iteration over consecutive work indices.  `start(x)`
// is the (non-decreasing) first work index of entry x; entry `i` owns the
// iteration's first element.  Each lane finds the largest x with
// start(x) <= j among entries i .. i+31 with a 5-step shuffle search; a lane
// whose entry lies beyond the window (only possible when entries own no work)
// falls back to a binary search in memory.
template <class StartF>
__device__ __forceinline__ uint32_t window_find(const StartF& start, uint32_t i, uint32_t count,
                                                unsigned long long j, bool valid) {
  const uint32_t lane = lane_id();
  const unsigned long long st = (i + lane < count) ? start(i + lane) : ~0ull;
  uint32_t t = 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const unsigned long long cand = __shfl_sync(kFull, st, t + d);
    if (cand <= j) t += d;
  }
  uint32_t x = i + t;
  if (valid && t == 31 && x + 1 < count && start(x + 1) <= j) {
    uint32_t lo = x + 1, hi = count - 1;
    while (lo < hi) {
      uint32_t mid = lo + ((hi - lo + 1) >> 1);
      if (start(mid) <= j) lo = mid; else hi = mid - 1;
    }
    x = lo;
  }
  return x;
}

struct QueueStart {
  const unsigned long long* q;
  __device__ __forceinline__ unsigned long long operator()(uint32_t x) const { return q[x] >> kEidBits; }
};

// Per-warp staging of frontier pushes in shared memory: edge ids are gathered
// across iterations and published with one 64-bit atomic (count and work) per
// kPushBuf entries, instead of one per iteration on a single hot counter.  The
// row descriptors of the staged edges are looked up at publication, all lanes
// at once, so those dependent loads stay off the per-iteration path.
constexpr int kPushBuf = 64;
constexpr int kWaveThreads = 128;
// Resident blocks per SM, which sets the register budget (40): with the found
// triangles staged the search no longer needs the last 16 warps an SM holds, and
// spills less.  Calls at 48 / 64 warps per SM, when that was chosen: R-MAT-22
// 285.9 / 284.8 ms, R-MAT-19 47.0 / 48.4, R-MAT-16 15.2 / 16.4.
constexpr int kWaveBlocksPerSm = 12;
constexpr int kWaveWarps = kWaveThreads / 32;
constexpr int kTailThreads = 512;  // threads per block of the small waves' cluster (1024: R-MAT-12 6% slower)
// slots of the per-warp loop state in shared memory (k_wave)
enum : int { kCtxJb = 0, kCtxSegEnd = 1, kCtxKend = 2 };
enum : int { kCtxEb = 0, kCtxM, kCtxLevel, kCtxQsel, kCtxQcount, kCtxSegLen, kCtxG, kCtxW };
// kept active-list entries staged per warp before one atomic reserves their
// place: every kept entry of a large scan goes through one counter per member
constexpr int kKeepBuf = 256;
// A run of at least kWaveRun elements of one frontier edge goes kWaveWays groups
// of 32 at a time, their row entries, index words and found entries loaded side
// by side: the wave waits for memory (19 long-scoreboard stall cycles per issue in
// a large wave, DRAM at 28%), so loads in flight count (R-MAT-22's peel 277 ms
// with one group, 257 with two).  Three and four spill (233 and 241 ms against 231,
// once the found triangles were staged).
constexpr int kWaveWays = 2;
constexpr uint32_t kWaveRun = 24;

struct PushStage {
  uint32_t* eid;  // this warp's kPushBuf staged edges
  uint32_t n;     // warp-uniform fill
};

// Publication of a warp's staged pushes.  Not inlined: it runs once per
// kPushBuf pushes, and as a call its temporaries (two row descriptors, hash
// descriptors, scans) stay out of the element loop's register budget.  It
// reads the union's arrays from the device-resident Union.
__device__ __noinline__ void push_flush_cold(const uint32_t* eid, uint32_t n, const Union* Up, uint32_t eb,
                                             uint32_t m, MemberState* st, uint32_t* err, uint32_t q_sel) {
  const UnionRegs U(Up);
  // the queue being built (q_sel names the one being processed)
  unsigned long long* qnext = q_sel ? U.q0 : U.q1;
  uint4* qdnext = q_sel ? U.qd0 : U.qd1;
  uint2* qhnext = q_sel ? U.qh0 : U.qh1;
  const Member M{0, 0, 0, 0, eb, m};
  const uint32_t lane = lane_id();
  const uint32_t x0 = lane < n ? eid[lane] : 0u, x1 = lane + 32 < n ? eid[lane + 32] : 0u;
  uint2 h0 = make_uint2(0, 0), h1 = make_uint2(0, 0);
  const uint4 d0 = lane < n ? edge_desc(U, x0, &h0) : make_uint4(0, 0, 0, 0);
  const uint4 d1 = lane + 32 < n ? edge_desc(U, x1, &h1) : make_uint4(0, 0, 0, 0);
  const unsigned long long p0 = warp_incl_scan(d0.y), p1 = warp_incl_scan(d1.y);
  const unsigned long long t0 = __shfl_sync(kFull, p0, 31), t1 = __shfl_sync(kFull, p1, 31);
  unsigned long long old = 0;
  if (lane == 0) {
    old = atomicAdd(&st->next, ((unsigned long long)n << kWorkBits) | (t0 + t1));
    if ((old & kWorkMask) + t0 + t1 > kWorkMask) atomicOr(err, kErrCapacity);
  }
  old = __shfl_sync(kFull, old, 0);
  const unsigned long long pos = old >> kWorkBits, ws = old & kWorkMask;
  if (lane < n) {
    if (pos + lane < M.m) {
      qnext[M.eb + pos + lane] = ((ws + p0 - d0.y) << kEidBits) | (x0 - M.eb);
      qdnext[M.eb + pos + lane] = d0;
      if (U.qh0) qhnext[M.eb + pos + lane] = h0;
    } else {
      atomicOr(err, kErrCapacity);
    }
  }
  if (lane + 32 < n) {
    if (pos + 32 + lane < M.m) {
      qnext[M.eb + pos + 32 + lane] = ((ws + t0 + p1 - d1.y) << kEidBits) | (x1 - M.eb);
      qdnext[M.eb + pos + 32 + lane] = d1;
      if (U.qh0) qhnext[M.eb + pos + 32 + lane] = h1;
    } else {
      atomicOr(err, kErrCapacity);
    }
  }
}

__device__ __forceinline__ void push_flush(PushStage& ps, const Union* Up, uint32_t eb, uint32_t m, MemberState* st,
                                           uint32_t* err, uint32_t q_sel) {
  __syncwarp();
  if (ps.n == 0) return;
  push_flush_cold(ps.eid, ps.n, Up, eb, m, st, err, q_sel);
  ps.n = 0;
  __syncwarp();
}

// Queue edge x (union eid) for wave W + 1.  All lanes call it.
__device__ __forceinline__ void push_edge(PushStage& ps, const UnionRegs& U, const Union* Up, uint32_t eb,
                                          uint32_t m, MemberState* st, uint32_t* err, uint32_t q_sel, bool want,
                                          uint32_t x, uint32_t W) {
  const unsigned bal = __ballot_sync(kFull, want);
  if (!bal) return;
  const uint32_t k = __popc(bal);
  if (ps.n + k > kPushBuf) push_flush(ps, Up, eb, m, st, err, q_sel);
  if (want) {
    U.es[x].y = (int)(W + 1);
    ps.eid[ps.n + __popc(bal & ((1u << lane_id()) - 1))] = x;
  }
  ps.n += k;
}

// Member state read past L1: the planner runs in the wave kernel's last
// block, whose L1 may hold lines that other blocks changed by atomics.
__device__ __forceinline__ MemberState load_state_cg(const MemberState* p) {
  static_assert(sizeof(MemberState) % 16 == 0, "MemberState is read as uint4 words");
  MemberState s;
  const uint4* src = reinterpret_cast<const uint4*>(p);
  uint4* dst = reinterpret_cast<uint4*>(&s);
#pragma unroll
  for (int i = 0; i < (int)(sizeof(MemberState) / 16); ++i) dst[i] = __ldcg(src + i);
  return s;
}

struct PlanShared {
  unsigned long long sw[32];
  uint32_t live;
  uint32_t newly_done;  // members that finished in this wave
  unsigned long long proc, scan, edges, live_edges;
};

// A member's state after the wave that just ran; returns the next wave's work.
__device__ __forceinline__ unsigned long long advance_member(MemberState& s, uint32_t m) {
  const unsigned long long cnt = s.next >> kWorkBits;
  switch (s.phase) {
    case kPhaseScan0:
      s.act_sel ^= 1u;
      s.act_count = s.kept;
      s.kept = 0;
      if (s.processed >= m) s.phase = kPhaseDone;
      else { s.level = s.min_kept; s.min_kept = 0xFFFFFFFFu; s.phase = kPhaseScan; }
      break;
    case kPhaseScan:
      s.act_sel ^= 1u;
      s.act_count = s.kept;
      s.kept = 0;
      if (cnt) {
        s.curr = s.next;
        s.next = 0;
        s.q_sel ^= 1u;
        s.phase = kPhaseProc;
        s.levels++;
        s.max_level = s.level;
      } else if (s.act_count == 0) {
        s.phase = kPhaseDone;
      } else {
        s.level = s.min_kept;  // no edge at this level: jump to the next occupied one
      }
      s.min_kept = 0xFFFFFFFFu;
      break;
    case kPhaseProc:
      s.processed += (uint32_t)(s.curr >> kWorkBits);
      if (cnt) {
        s.curr = s.next;
        s.next = 0;
        s.q_sel ^= 1u;
      } else {
        s.curr = 0;
        if (s.processed >= m) s.phase = kPhaseDone;
        else { s.level += 1; s.phase = kPhaseScan; s.min_kept = 0xFFFFFFFFu; }
      }
      break;
    default:
      return 0;
  }
  if (s.phase != kPhaseDone) s.waves++;
  return s.phase == kPhaseDone ? 0 : s.phase == kPhaseProc ? s.curr & kWorkMask : s.act_count;
}

// The loop's side of a planned wave: work counters, the bounds, and whether the
// loop stops here.  One thread calls it; returns ctl->done.
// 1, 2 and 8 measured alike on R-MAT-19, R-MAT-22 and the mix of 24 graphs.
constexpr unsigned long long kCompactPay = 2;

struct WavePlan {
  unsigned long long total, proc, scan, edges, live_edges;
  uint32_t live, newly_done;
};
__device__ __forceinline__ uint32_t plan_commit(Control* ctl, uint32_t* __restrict__ err, const WavePlan& P) {
  // one round of loads, then one of stores
  const unsigned long long waves = ctl->waves_run + 1, max_waves = ctl->max_waves, t_start = ctl->t_start,
                           timeout = ctl->timeout_ns, el_proc = ctl->el_proc, el_scan = ctl->el_scan,
                           edges = ctl->edges_proc, slots = ctl->csr_slots, compact_min = ctl->compact_min,
                           compact_el = ctl->compact_el;
  const uint32_t wave = ctl->wave, pct = ctl->compact_pct, notify = ctl->notify_done;
  const volatile uint32_t* admit = ctl->admit;
  ulonglong4* trace = ctl->trace;
  const uint32_t e = __ldcg(err);
  if (trace && waves - 1 < ctl->trace_cap) trace[waves - 1] = make_ulonglong4(globaltimer(), P.total, P.proc, P.scan);
  ctl->el_proc = el_proc + P.proc;
  ctl->el_scan = el_scan + P.scan;
  ctl->edges_proc = edges + P.edges;
  ctl->total_work = P.total;
  ctl->wave = wave + 1;
  ctl->waves_run = waves;
  uint32_t done = 0, reason = kExitNone;
  if (P.live == 0) { done = 1; reason = kExitDone; }
  if (e) { done = 1; reason = kExitError; }
  if (waves > max_waves) { atomicOr(err, kErrWaves); done = 1; reason = kExitError; }
  if (globaltimer() - t_start > timeout) { atomicOr(err, kErrTimeout); done = 1; reason = kExitError; }
  // live edges fill at most compact_pct % of the working rows (76 unless
  // tuned): stop so the host can compact them (a compaction is a few passes
  // over the rows, which the shorter rows repay at this fill: R-MAT-22 276.4 ms,
  // 85% 281.4, 70% 281.9, 90% 283.5)
  // ... once the waves since the last one have searched at least a kCompactPay-th
  // as many elements as it would move: a graph whose peel ends in a few small
  // waves (de Bruijn: 305 elements, 49 M slots, 0.6 of its 5.2 ms) never pays it
  if (!done && slots >= compact_min && 200 * P.live_edges <= (unsigned long long)pct * slots &&
      kCompactPay * (el_proc + P.proc - compact_el) >= slots) {
    done = 1;
    reason = kExitCompact;
  }
  if (!done && notify && P.newly_done) { done = 1; reason = kExitMember; }
  if (!done && admit && *admit) { done = 1; reason = kExitAdmit; }
  ctl->done = done;
  ctl->exit_reason = reason;
  return done;
}

// Planner: one block advances every member's state machine after a wave and
// lays out the next wave's work; sets the CUDA-graph loop condition.  Runs in
// the last block of each wave (see k_wave), after every other block's writes.
// Up to 32 members are planned by one warp: no block scans and no barriers, and
// the loads go out in one round (a small wave spent 2.0 of its 8.1 us here).
__device__ __forceinline__ void plan_wave(const Member* __restrict__ mem, MemberState* __restrict__ st,
                                          Control* ctl, unsigned long long* __restrict__ wpref,
                                          uint32_t* __restrict__ err, cudaGraphConditionalHandle handle,
                                          int use_handle, PlanShared& ps, uint32_t G, bool was_done) {
  if (was_done) {
    // the loop is stopped (host-launched waves keep coming until the host
    // looks): the planned wave must survive untouched for a resume
    if (threadIdx.x == 0 && use_handle) cudaGraphSetConditional(handle, 0u);
    return;
  }
  if (G <= 32) {
    if (threadIdx.x >= 32) return;
    const uint32_t g = threadIdx.x;
    MemberState s{};
    s.phase = kPhaseDone;
    uint32_t m = 0;
    if (g < G) {
      s = load_state_cg(st + g);
      m = mem[g].m;
    }
    const uint32_t before = s.phase;
    const unsigned long long w = advance_member(s, m);
    const bool live = s.phase != kPhaseDone, proc = s.phase == kPhaseProc;
    if (g < G) st[g] = s;
    WavePlan P{};
    if (G == 1) {
      if (g > 0) return;
      P.total = w;
      P.proc = proc ? w : 0;
      P.edges = proc ? s.curr >> kWorkBits : 0;
      P.live_edges = live ? m - s.processed : 0;
      P.live = live;
      P.newly_done = !live && before != kPhaseDone;
      wpref[0] = 0;
      wpref[1] = w;
    } else {
      const unsigned long long incl = warp_incl_scan(w);
      if (g < G) wpref[g] = incl - w;
      P.total = __shfl_sync(kFull, incl, 31);
      // frontier edges of a union stay below 2^32 (edge ids are 32-bit), live edges too
      P.edges = __reduce_add_sync(kFull, proc ? (uint32_t)(s.curr >> kWorkBits) : 0u);
      P.live_edges = __reduce_add_sync(kFull, live ? m - s.processed : 0u);
      P.live = __popc(__ballot_sync(kFull, live));
      P.newly_done = __popc(__ballot_sync(kFull, !live && before != kPhaseDone));
      P.proc = proc ? w : 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) P.proc += __shfl_xor_sync(kFull, P.proc, d);
      if (g > 0) return;
      wpref[G] = P.total;
    }
    P.scan = P.total - P.proc;
    const uint32_t done = plan_commit(ctl, err, P);
    if (use_handle) cudaGraphSetConditional(handle, done ? 0u : 1u);
    return;
  }
  unsigned long long* sw = ps.sw;
  if (threadIdx.x == 0) { ps.live = 0; ps.proc = 0; ps.scan = 0; ps.edges = 0; ps.live_edges = 0; ps.newly_done = 0; }
  __syncthreads();
  unsigned long long carry = 0;
  for (uint32_t b = 0; b < G; b += blockDim.x) {
    const uint32_t g = b + threadIdx.x;
    unsigned long long w = 0;
    if (g < G) {
      MemberState s = load_state_cg(st + g);
      const uint32_t m = mem[g].m, before = s.phase;
      w = advance_member(s, m);
      st[g] = s;
      if (s.phase == kPhaseProc) {
        atomicAdd(&ps.proc, w);
        atomicAdd(&ps.edges, s.curr >> kWorkBits);
      } else if (w) {
        atomicAdd(&ps.scan, w);
      }
      if (s.phase != kPhaseDone) {
        atomicAdd(&ps.live, 1u);
        atomicAdd(&ps.live_edges, (unsigned long long)(m - s.processed));
      } else if (before != kPhaseDone) {
        atomicAdd(&ps.newly_done, 1u);
      }
    }
    unsigned long long total;
    unsigned long long ex = block_exclusive_scan<unsigned long long>(w, sw, total);
    if (g < G) wpref[g] = carry + ex;
    carry += total;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    wpref[G] = carry;
    const uint32_t done =
        plan_commit(ctl, err, WavePlan{carry, ps.proc, ps.scan, ps.edges, ps.live_edges, ps.live, ps.newly_done});
    if (use_handle) cudaGraphSetConditional(handle, done ? 0u : 1u);
  }
}

// One member's segment of a level scan (kPhaseScan0 / kPhaseScan): active
// entry j of the segment is kept (support above the level), queued for this
// level, or dropped (processed).  Not inlined: its staging state stays out of
// the frontier loop's register budget.  Publishes its pushes before returning.
// Four groups of 32 entries at a time: what bounds a scan is its instructions and
// the two dependent loads per entry (R-MAT-22's scans 33 -> 26 ms, its largest 168
// -> 132 us for 19 M entries; two groups 29 ms, a stage of 384 entries 28).
constexpr int kScanWays = 4;
__device__ __noinline__ void wave_scan_segment(const Union* Up, MemberState* st, uint32_t eb, uint32_t m,
                                               uint32_t phase, uint32_t level, uint32_t act_sel, uint32_t q_sel,
                                               uint32_t W, uint32_t a0, uint32_t seg_len, uint32_t* keepbuf,
                                               uint32_t* push_eid, uint32_t* err) {
  const UnionRegs U(Up);
  const uint32_t lane = lane_id();
  PushStage ps{push_eid, 0};
  const uint32_t* act = act_sel ? U.act1 : U.act0;
  uint32_t* act_out = act_sel ? U.act0 : U.act1;
  const bool first = phase == kPhaseScan0;
  uint32_t nkeep = 0, nzero = 0, mn = 0xFFFFFFFFu;
  act += eb + a0;
  for (uint32_t r = 0; r < seg_len; r += 32 * kScanWays) {
    // kScanWays groups of 32 entries: their ids, then their states, side by side
    uint32_t le[kScanWays];
    int2 se[kScanWays];
#pragma unroll
    for (int j = 0; j < kScanWays; ++j) le[j] = r + 32 * j + lane < seg_len ? act[r + 32 * j + lane] : kInvalid;
#pragma unroll
    for (int j = 0; j < kScanWays; ++j) se[j] = le[j] != kInvalid ? U.es[eb + le[j]] : make_int2(0, 0);
    if (nkeep + 32 * kScanWays > kKeepBuf) {
      __syncwarp();
      uint32_t old = 0;
      if (lane == 0) old = atomicAdd(&st->kept, nkeep);
      old = __shfl_sync(kFull, old, 0);
      for (uint32_t t = lane; t < nkeep; t += 32) act_out[eb + old + t] = keepbuf[t];
      nkeep = 0;
      __syncwarp();
    }
    bool queue[kScanWays], any = false;
#pragma unroll
    for (int j = 0; j < kScanWays; ++j) {
      const int32_t s = se[j].x;
      // processed edges leave the active list (the first scan: those without support)
      const bool live = le[j] != kInvalid && (first ? s != 0 : (uint32_t)se[j].y == kTagActive);
      queue[j] = live && !first && s <= (int32_t)level;
      const bool keep = live && !queue[j];
      if (keep) mn = min(mn, (uint32_t)s);
      if (first && le[j] != kInvalid && !live) {
        U.es[eb + le[j]].y = 0;
        ++nzero;
      }
      any |= queue[j];
      const unsigned kb = __ballot_sync(kFull, keep);
      if (keep) keepbuf[nkeep + __popc(kb & ((1u << lane) - 1))] = le[j];
      nkeep += __popc(kb);
    }
    if (__any_sync(kFull, any)) {
#pragma unroll
      for (int j = 0; j < kScanWays; ++j)
        push_edge(ps, U, Up, eb, m, st, err, q_sel, queue[j], eb + le[j], W);
    }
  }
  __syncwarp();
  if (nkeep) {
    uint32_t old = 0;
    if (lane == 0) old = atomicAdd(&st->kept, nkeep);
    old = __shfl_sync(kFull, old, 0);
    for (uint32_t t = lane; t < nkeep; t += 32) act_out[eb + old + t] = keepbuf[t];
  }
  nzero = __reduce_add_sync(kFull, nzero);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mn = min(mn, __shfl_xor_sync(kFull, mn, d));
  if (lane == 0) {
    if (mn != 0xFFFFFFFFu) atomicMin(&st->min_kept, mn);
    if (nzero) atomicAdd(&st->processed, nzero);
  }
  __syncwarp();
  push_flush(ps, Up, eb, m, st, err, q_sel);
}

// Kernel D: one peel wave.  The wave's work (all members' scan elements and
// frontier elements, laid out by `wpref`) is cut into warp-sized chunks; a
// warp walks its chunk member by member, 32 consecutive elements per
// iteration, so every iteration belongs to one member.
//   scan element j      active-list entry j: processed -> dropped; support
//                       <= level -> queued for this level; else kept
//   frontier element j  element o of the shorter working row of frontier
//                       edge e, searched in the longer row; a hit is a triangle
// The search is one word of the longer row's rank index for most absent names
// and one entry more for the others; it replaced a row merge (similar lengths),
// per-row hash tables and dense hub maps, whose probes were random DRAM sectors:
// R-MAT-22's peel 315 -> 257 ms, its first large wave 0.87 -> 0.68 ms on R-MAT-20
// with 0.60 -> 0.36 G instructions and 2.7 -> 1.4 GB read.  The index is rebuilt
// with the rows at every compaction, so it shrinks with what is left.
constexpr int kHitBuf = 64;  // found triangles staged per warp: fewer than 32, and 32 of a group

template <int kWarps>
struct WaveShared {
  uint32_t push_eid[kWarps][kPushBuf];
  uint32_t keep[kWarps][kKeepBuf];
  uint32_t hit_e[kWarps][kHitBuf], hit_f[kWarps][kHitBuf], hit_h[kWarps][kHitBuf];
  // work counters (per warp: hits, groups of 32 elements inside one edge, groups
  // over several edges), here rather than in registers held across the loop;
  // lane 0 adds to them
  uint32_t cnt[3][kWarps];
  // warp-uniform state of the frontier loop, read back where it is used: held
  // in registers it was spilled to local memory, whose lines the loop's random
  // row and state loads evict from L1
  unsigned long long w64[kWarps][3];  // kCtxJb, kCtxSegEnd, kCtxKend
  uint32_t w32[kWarps][8];            // kCtxEb .. kCtxW
};

// What a small wave's warps need of member 0, read in the same round of loads as
// the control: a single graph's wave then starts one L2 round trip earlier (a wave
// over the whole chip loses more to the registers this holds: R-MAT-19 2% slower).
struct WaveHead {
  uint4 s;                  // phase, level, act_sel, q_sel
  unsigned long long curr;
  Member M;
};
__device__ __forceinline__ WaveHead wave_head(const WaveArgs& a) {
  const uint4* st = reinterpret_cast<const uint4*>(a.st);
  WaveHead h;
  h.s = __ldcg(st);
  h.curr = __ldcg(reinterpret_cast<const unsigned long long*>(st + 2));
  h.M = a.mem[0];
  return h;
}
static_assert(offsetof(MemberState, phase) == 0 && offsetof(MemberState, q_sel) == 12 &&
                  offsetof(MemberState, curr) == 32, "wave_head reads MemberState as uint4 words");

// This warp's share of wave W (warp `warp` of `nwarps`).  kTail (small waves): a
// warp's queue window brings its entries' row descriptors along, 24 bytes more per
// entry for a round trip less.
template <bool kMulti, bool kTail, int kWarps>
__device__ __forceinline__ void wave_work(const WaveArgs& a, WaveShared<kWarps>& sh, unsigned long long total,
                                          uint32_t W, uint32_t G, const WaveHead& head, unsigned long long warp,
                                          unsigned long long nwarps) {
  const uint32_t lane = lane_id();
  const uint32_t wib = threadIdx.x >> 5;
  const UnionRegs U(a.Up, a.arr);
  // one chunk per warp: finer chunks (handed out by a block counter too: R-MAT-22
  // 303 -> 321 to 361 ms with 1 to 8 pieces per warp) measured slower, the search
  // for a chunk's first entry is paid once per warp; ch * nwarps >= total, so the chunk below is the warp's only one
  const unsigned long long ch = max(((total + nwarps - 1) / nwarps + 31) & ~31ull, 32ull);
  PushStage ps{sh.push_eid[wib], 0};
  volatile unsigned long long* const w64 = sh.w64[wib];
  volatile uint32_t* const w32 = sh.w32[wib];

  if (warp * ch < total) {
    const unsigned long long c0 = warp * ch;
    if (lane == 0) w64[kCtxKend] = min(c0 + ch, total);
    __syncwarp();
    unsigned long long k = c0;
    uint32_t g = G > 1 ? warp_last_le(PrefKey{a.wpref}, 0, G - 1, k) : 0;
    while (k < w64[kCtxKend]) {
      const unsigned long long kend = w64[kCtxKend];
      while (g + 1 < G && a.wpref[g + 1] <= k) ++g;
      const unsigned long long mbeg = G > 1 ? a.wpref[g] : 0ull;
      // a segment spans < 2^31 elements, so offsets inside it are 32-bit
      const unsigned long long seg_end = min(min(kend, G > 1 ? a.wpref[g + 1] : total), k + (1ull << 31));
      if (seg_end <= k || mbeg > k) {  // layout does not cover k: stop rather than spin
        if (lane == 0) atomicOr(a.err, kErrInternal);
        break;
      }
      MemberState* st = a.st + g;
      const bool ready = kTail && G == 1;  // the head brought it
      const Member M = ready ? head.M : a.mem[g];
      const uint32_t phase = ready ? head.s.x : st->phase, level = ready ? head.s.y : st->level,
                     act_sel = ready ? head.s.z : st->act_sel, q_sel = ready ? head.s.w : st->q_sel;
      if (phase == kPhaseProc) {
        const uint32_t qcount0 = (uint32_t)((ready ? head.curr : st->curr) >> kWorkBits);
        if (qcount0 == 0) {
          if (lane == 0) atomicOr(a.err, kErrInternal);
          k = seg_end;
          continue;
        }
        const uint32_t i0 =
            warp_last_le(QueueStart{(q_sel ? U.q1 : U.q0) + M.eb}, 0, qcount0 - 1, k - mbeg);
        __syncwarp();
        if (lane == 0) {
          // element j (member-relative) = jb + r + lane; r counts the segment
          w64[kCtxJb] = k - mbeg;
          w64[kCtxSegEnd] = seg_end;
          w32[kCtxEb] = M.eb;
          w32[kCtxM] = M.m;
          w32[kCtxLevel] = level;
          w32[kCtxQsel] = q_sel;
          w32[kCtxQcount] = qcount0;
          w32[kCtxSegLen] = (uint32_t)(seg_end - k);
          w32[kCtxG] = g;
          w32[kCtxW] = W;
        }
        __syncwarp();
        uint32_t i = i0;
        uint32_t found = 0, nhit = 0;
        // the rule for hits [at, at + 32) of the stage, lanes in `on`
        auto resolve = [&](uint32_t at, unsigned on) {
          bool pf = false, ph = false;
          uint32_t rf = 0, rh = 0;
          if (on >> lane & 1) {
            const uint32_t re = sh.hit_e[wib][at + lane];
            rf = sh.hit_f[wib][at + lane];
            rh = sh.hit_h[wib][at + lane];
            const int2 s_f = U.es[rf], s_h = U.es[rh];
            pkt_rule<kMulti>(U, re, rf, s_f, rh, s_h, w32[kCtxLevel], w32[kCtxW], pf, ph);
          }
          if (__any_sync(kFull, pf || ph)) {
            push_edge(ps, U, a.Up, w32[kCtxEb], w32[kCtxM], a.st + w32[kCtxG], a.err, w32[kCtxQsel], pf, rf,
                      w32[kCtxW]);
            push_edge(ps, U, a.Up, w32[kCtxEb], w32[kCtxM], a.st + w32[kCtxG], a.err, w32[kCtxQsel], ph, rh,
                      w32[kCtxW]);
          }
        };
        for (uint32_t r = 0; r < w32[kCtxSegLen];) {
          const uint32_t seg_len = w32[kCtxSegLen];
          const uint32_t qcount = w32[kCtxQcount];
          // the window's entries, loaded once: each lane picks its own by a
          // shuffle search on the work starts (entries own >= 1 element, so
          // 32 consecutive elements span at most 32 entries).  The search runs
          // on 32-bit distances from the iteration's first element jr: the
          // window's first entry owns element jr - 1 or jr and an entry's work
          // is below 2^31, so every distance lies in (-2^31, 2^31); entries
          // past the queue's end clamp to the most negative.  Lane l's
          // element jr + l lies in entry x iff jr - start(x) >= -l.
          const unsigned long long jr = w64[kCtxJb] + r;
          const unsigned long long qv =
              (i + lane < qcount) ? ((w32[kCtxQsel] ? U.q1 : U.q0) + w32[kCtxEb])[i + lane] : ~0ull;
          uint4 wd = make_uint4(0, 0, 0, 0);
          uint2 wh = make_uint2(0, 0);
          if (kTail && i + lane < qcount) {
            wd = ((w32[kCtxQsel] ? U.qd1 : U.qd0) + w32[kCtxEb])[i + lane];
            if (U.qh0) wh = ((w32[kCtxQsel] ? U.qh1 : U.qh0) + w32[kCtxEb])[i + lane];
          }
          const int32_t dq = (int32_t)max((long long)(jr - (qv >> kEidBits)), (long long)INT32_MIN);
          // elements of entry i from jr on (an end past the queue is 2^31)
          const uint32_t rem = min(seg_len - r, 0u - (uint32_t)__shfl_sync(kFull, dq, 1));
          bool valid;
          uint32_t e = 0, o = 0;
          uint4 dsc = make_uint4(0, 0, 0, 0);
          uint2 hq = make_uint2(0, 0);
          uint32_t o_end;       // the lane's elements o, o + 32, ... below o_end
          const bool run = (int32_t)rem >= (int32_t)kWaveRun;
          const uint32_t i_win = i;
          uint32_t x = i;
          if (run) {
            // the rest of entry i: one edge, the same rows for the whole warp
            e = w32[kCtxEb] + __shfl_sync(kFull, (uint32_t)qv & kEidMask, 0);
            o = (uint32_t)__shfl_sync(kFull, dq, 0) + lane;
            valid = true;
            o_end = o - lane + rem;
            r += rem;
            i += 1;
            if (lane == 0) sh.cnt[1][wib] += (rem + 31) / 32;
          } else {
            uint32_t t = 0;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
              const int32_t cand = __shfl_sync(kFull, dq, t + d);
              if (cand >= -(int32_t)lane) t += d;
            }
            o = (uint32_t)(__shfl_sync(kFull, dq, t) + (int32_t)lane);
            e = w32[kCtxEb] + __shfl_sync(kFull, (uint32_t)qv & kEidMask, t);
            x = i + t;
            const uint32_t last = min(31u, seg_len - 1 - r);
            i = __shfl_sync(kFull, x, last);
            valid = r + lane < seg_len;
            o_end = o + 1;
            r += 32;
            if (lane == 0) sh.cnt[2][wib]++;
          }
          if (kTail) {
            const int src = (int)(x - i_win);
            dsc = make_uint4(__shfl_sync(kFull, wd.x, src), __shfl_sync(kFull, wd.y, src),
                             __shfl_sync(kFull, wd.z, src), __shfl_sync(kFull, wd.w, src));
            hq = make_uint2(__shfl_sync(kFull, wh.x, src), __shfl_sync(kFull, wh.y, src));
          } else if (valid) {
            dsc = ((w32[kCtxQsel] ? U.qd1 : U.qd0) + w32[kCtxEb])[x];
            if (U.qh0) hq = ((w32[kCtxQsel] ? U.qh1 : U.qh0) + w32[kCtxEb])[x];
          }
          // rows may have been compacted since the entry's work was counted
          o_end = valid ? min(o_end, dsc.y) : 0u;
          const unsigned long long* words = U.rpool + dsc.z;
          const uint32_t shift = rank_shift(dsc.w - dsc.z, hq.y);
          hq.y &= ~kRankFine;
          // warp-uniform trips: all lanes of a run share o_end; otherwise one trip
          const uint32_t o0 = o - lane;
          for (uint32_t og = 0; run ? o0 + og < o_end : og == 0; og += 32 * kWaveWays, o += 32 * kWaveWays) {
            uint32_t w[kWaveWays], f[kWaveWays], h[kWaveWays];
            unsigned long long en[kWaveWays];
#pragma unroll
            for (int j = 0; j < kWaveWays; ++j) {
              en[j] = o + 32 * j < o_end ? __ldg(U.row + dsc.x + o + 32 * j) : ~0ull;
              h[j] = kInvalid;
            }
            // f == kInvalid: a self-loop entry.  The frontier edge's own entry needs
            // no check: its name is the longer row's vertex, which that row holds
            // only as a self-loop (h == kInvalid).
            if (hq.y) {
              // the longer row's rank index: its words, then its entries, side by side
              uint32_t bk[kWaveWays];
#pragma unroll
              for (int j = 0; j < kWaveWays; ++j) {
                w[j] = (uint32_t)en[j];
                f[j] = (uint32_t)(en[j] >> 32);
                bk[j] = ((w[j] - hq.x) * hq.y) >> shift;
                en[j] = f[j] != kInvalid ? __ldg(words + (bk[j] >> 5)) : 0ull;
              }
#pragma unroll
              for (int j = 0; j < kWaveWays; ++j) {
                const uint32_t bit = 1u << (bk[j] & 31);
                if ((uint32_t)en[j] & bit) {
                  uint32_t p = (uint32_t)(en[j] >> 32) + __popc((uint32_t)en[j] & (bit - 1));
                  unsigned long long at = __ldg(U.row + p);
                  if ((uint32_t)at < w[j]) p = rank_later(U.row, p, dsc.w, words, bk[j], shift, w[j], &at);
                  if (p != kInvalid && (uint32_t)at == w[j]) h[j] = (uint32_t)(at >> 32);
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < kWaveWays; ++j) {
                w[j] = (uint32_t)en[j];
                f[j] = (uint32_t)(en[j] >> 32);
                if (f[j] != kInvalid) {
                  const uint32_t p = find_in_row(U.row, dsc.z, dsc.w, w[j]);
                  if (p != kInvalid) h[j] = (uint32_t)(__ldg(U.row + p) >> 32);
                }
              }
            }
            // found triangles gather in the warp's stage and are resolved 32 at a
            // time, so that the rule runs on full warps (a third of the elements
            // are hits on R-MAT)
#pragma unroll
            for (int j = 0; j < kWaveWays; ++j) {
              const unsigned hb = __ballot_sync(kFull, h[j] != kInvalid);
              if (hb == 0) continue;
              const uint32_t at = nhit + __popc(hb & ((1u << lane) - 1));
              if (h[j] != kInvalid) {
                sh.hit_e[wib][at] = e;
                sh.hit_f[wib][at] = f[j];
                sh.hit_h[wib][at] = h[j];
              }
              nhit += __popc(hb);
              found += __popc(hb);
              if (nhit >= 32) {
                __syncwarp();
                nhit -= 32;
                resolve(nhit, kFull);
                __syncwarp();
              }
            }
          }
        }
        if (nhit) {
          __syncwarp();
          resolve(0, nhit == 32 ? kFull : (1u << nhit) - 1);
          nhit = 0;
          __syncwarp();
        }
        if (lane == 0) sh.cnt[0][wib] += found;
        // entries belong to this member: publish before moving on
        push_flush(ps, a.Up, w32[kCtxEb], w32[kCtxM], a.st + w32[kCtxG], a.err, w32[kCtxQsel]);
        k = w64[kCtxSegEnd];
        g = w32[kCtxG];
        continue;
      } else if (phase == kPhaseScan0 || phase == kPhaseScan) {
        // active-list positions are below the member's edge count (< 2^28)
        wave_scan_segment(a.Up, st, M.eb, M.m, phase, level, act_sel, q_sel, W, (uint32_t)(k - mbeg),
                          (uint32_t)(seg_end - k), sh.keep[wib], ps.eid, a.err);
      }
      push_flush(ps, a.Up, M.eb, M.m, st, a.err, q_sel);  // entries belong to this member: publish before moving on
      k = seg_end;
    }
  }
}

// Work counters: summed per block, then one atomic per counter and block
// (per-warp atomics on three addresses serialise on large waves).  All threads
// call it, after a block barrier.
template <int kWarps>
__device__ __forceinline__ void flush_counts(const WaveArgs& a, const WaveShared<kWarps>& sh) {
  if (threadIdx.x < 3) {
    unsigned long long sum = 0;
#pragma unroll 8
    for (int w = 0; w < kWarps; ++w) sum += sh.cnt[threadIdx.x][w];
    unsigned long long* dst = threadIdx.x == 0 ? &a.ctl->hits
                              : threadIdx.x == 1 ? &a.ctl->merge_iters : &a.ctl->lane_iters;
    if (sum) atomicAdd(dst, sum);
  }
}

template <bool kMulti>
__global__ void __launch_bounds__(kWaveThreads, kWaveBlocksPerSm) k_wave(WaveArgs a) {
  __shared__ WaveShared<kWaveWarps> sh;
  const uint32_t lane = lane_id();
  if (lane < 3) sh.cnt[lane][threadIdx.x >> 5] = 0;
  __syncwarp();
  // a stopped loop (host-launched waves run on until the host looks) does no
  // work, but its blocks still hand over to the planner
  wave_work<kMulti, false>(a, sh, a.ctl->done ? 0ull : a.ctl->total_work, a.ctl->wave, a.ctl->G, WaveHead{},
                    ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                    ((unsigned long long)gridDim.x * blockDim.x) >> 5);
  __syncthreads();
  flush_counts(a, sh);
  // the last block to finish plans the next wave (threadfence-reduction
  // pattern: every thread fences its writes, the block takes a ticket; the
  // block holding the last ticket sees every other block's writes)
  __shared__ uint32_t s_last;
  __shared__ PlanShared s_plan;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&a.ctl->blocks_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (s_last) {
    __threadfence();
    plan_wave(a.mem, a.st, a.ctl, a.wpref, a.err, a.handle, a.use_handle, s_plan, a.ctl->G, a.ctl->done);
    if (threadIdx.x == 0) a.ctl->blocks_done = 0;
  }
}

// Small waves in one launch: a single thread-block cluster runs wave after wave
// while the planned one has at most `max_work` elements, its blocks meeting at
// the cluster's hardware barrier instead of at a kernel boundary, and block 0
// planning between two of them.  A wave of 100 elements takes 7 us here, 13 to 14
// as a kernel over the whole chip (launch gap 3, block start 1, ticket 2); what is
// left is its chain of dependent round trips to L2.  The barrier's release and
// acquire order the waves' memory; everything a wave reads through the read-only
// path (rows, index, edges) does not change between compactions.  Every block
// leaves the loop on the same values, read after the same barrier, and the
// planner's bounds (waves, time) end it as they end the loop of k_wave.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <bool kMulti>
__global__ void __launch_bounds__(kTailThreads, 1) k_wave_tail(WaveArgs a, unsigned long long max_work) {
  __shared__ WaveShared<kTailThreads / 32> sh;
  __shared__ PlanShared s_plan;
  const uint32_t wib = threadIdx.x >> 5;
  if (lane_id() < 3) sh.cnt[lane_id()][wib] = 0;
  __syncwarp();
  for (;;) {
    const unsigned long long total = __ldcg(&a.ctl->total_work);
    const uint32_t W = __ldcg(&a.ctl->wave);
    const uint32_t G = __ldcg(&a.ctl->G);
    const WaveHead head = wave_head(a);
    if (__ldcg(&a.ctl->done) || total > max_work) break;
    wave_work<kMulti, true>(a, sh, total, W, G, head, wib * gridDim.x + blockIdx.x, (kTailThreads / 32) * gridDim.x);
    __syncwarp();
    cluster_barrier();
    if (blockIdx.x == 0) plan_wave(a.mem, a.st, a.ctl, a.wpref, a.err, a.handle, 0, s_plan, G, false);
    __syncwarp();
    cluster_barrier();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.use_handle)
    cudaGraphSetConditional(a.handle, __ldcg(&a.ctl->done) ? 0u : 1u);
  __syncthreads();
  flush_counts(a, sh);
}

// Working-row compaction (between waves): keep the entries whose edge is not
// processed (tag >= the next wave).  The edges' states are first condensed
// into a bitmap (one bit per edge, small enough to stay in L2); the rows are then
// one flat array whose kept entries move up, whatever rows they belong to, so no
// row's length matters: with a lane, a warp or a block per row the passes waited
// for warps whose 32 neighbouring rows were all long (degree-ordered vertices):
// the 28 compactions of R-MAT-22 20 -> 5 ms, mix of 24 graphs 212 -> 192 ms.  Bound
// by the bitmap's lookups (one per slot, L2) and 24 bytes of HBM per slot.
//   k_compact_mark     edges -> bitmap
//   k_compact_count    slots -> bitmap, kept slots per tile (then scanned)
//   k_compact_move     kept entries to their new place, kept slots before each
//                      32-slot word
//   k_compact_offsets  each row's start: the kept slots before its old start
__global__ void __launch_bounds__(256) k_compact_mark(const int2* __restrict__ es, uint32_t m,
                                                      const Control* ctl, uint32_t* __restrict__ alive) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t W = ctl->wave;
  const uint32_t words = (m + 31) / 32;
  for (uint32_t i = warp; i < words; i += nwarps) {
    const uint32_t x = i * 32 + lane;
    const bool live = x < m && (uint32_t)__ldg(&es[x].y) >= W;
    const uint32_t bits = __ballot_sync(kFull, live);
    if (lane == 0) alive[i] = bits;
  }
}

__device__ __forceinline__ bool is_alive(const uint32_t* __restrict__ alive, uint32_t x) {
  return x != kInvalid && ((__ldg(alive + (x >> 5)) >> (x & 31)) & 1u);
}

constexpr uint32_t kCompactTile = 8192;  // slots per block of 256 threads: a 32-slot word each

__global__ void __launch_bounds__(256) k_compact_count(const unsigned long long* __restrict__ row,
                                                       unsigned long long slots,
                                                       const uint32_t* __restrict__ alive,
                                                       uint32_t* __restrict__ kept, uint32_t* __restrict__ tiles) {
  __shared__ uint32_t s_sum[8];
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  const unsigned long long base = (unsigned long long)blockIdx.x * kCompactTile;
  uint32_t sum = 0;
#pragma unroll 8
  for (uint32_t x = wid; x < kCompactTile / 32; x += 8) {
    const unsigned long long i = base + 32 * x + lane;
    const bool k = i < slots && is_alive(alive, (uint32_t)(__ldg(row + i) >> 32));
    const uint32_t bits = __ballot_sync(kFull, k);
    if (lane == 0 && base + 32 * x < slots) kept[(base >> 5) + x] = bits;
    sum += __popc(bits);
  }
  if (lane == 0) s_sum[wid] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += s_sum[w];
    tiles[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(256) k_compact_move(const unsigned long long* __restrict__ row,
                                                      unsigned long long slots,
                                                      const uint32_t* __restrict__ kept,
                                                      const uint32_t* __restrict__ tiles,
                                                      uint32_t* __restrict__ before,
                                                      unsigned long long* __restrict__ row2) {
  __shared__ uint32_t s_scan[32], s_bits[256], s_at[256];
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  const unsigned long long base = (unsigned long long)blockIdx.x * kCompactTile;
  const unsigned long long word = (base >> 5) + threadIdx.x;
  const uint32_t bits = 32 * word < slots ? __ldg(kept + word) : 0u;
  uint32_t total;
  const uint32_t at = __ldg(tiles + blockIdx.x) + block_exclusive_scan<uint32_t>(__popc(bits), s_scan, total);
  if (32 * word < slots) before[word] = at;
  s_bits[threadIdx.x] = bits;
  s_at[threadIdx.x] = at;
  __syncthreads();
#pragma unroll 8
  for (uint32_t x = wid; x < kCompactTile / 32; x += 8) {
    const uint32_t m = s_bits[x];
    if (m >> lane & 1) row2[s_at[x] + __popc(m & ((1u << lane) - 1))] = __ldg(row + base + 32 * x + lane);
  }
}

// `total`: kept slots (a row may start at the array's end)
__global__ void __launch_bounds__(256) k_compact_offsets(const uint32_t* __restrict__ off, uint32_t n,
                                                         unsigned long long slots,
                                                         const uint32_t* __restrict__ kept,
                                                         const uint32_t* __restrict__ before,
                                                         const uint32_t* __restrict__ total,
                                                         uint32_t* __restrict__ off2) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u <= n; u += gridDim.x * blockDim.x) {
    const uint32_t s = __ldg(off + u);
    off2[u] = s < slots ? __ldg(before + (s >> 5)) + __popc(__ldg(kept + (s >> 5)) & ((1u << (s & 31)) - 1)) : *total;
  }
}

// After a compaction the rows moved: rebuild the descriptors of every queued
// frontier.  `per` blocks share a member (block b serves member b / per), so
// one large frontier is spread over the whole GPU.
__global__ void __launch_bounds__(256) k_refresh_desc(const Union* __restrict__ Up,
                                                      const Member* __restrict__ mem,
                                                      const MemberState* __restrict__ st, uint32_t G,
                                                      uint32_t per) {
  const UnionRegs U(Up);
  const uint32_t g = blockIdx.x / per, part = blockIdx.x % per;
  if (g >= G) return;
  const MemberState s = st[g];
  if (s.phase != kPhaseProc) return;
  const uint32_t cnt = (uint32_t)(s.curr >> kWorkBits);
  const Member M = mem[g];
  const unsigned long long* q = (s.q_sel ? U.q1 : U.q0) + M.eb;
  uint4* qd = (s.q_sel ? U.qd1 : U.qd0) + M.eb;
  uint2* qh = U.qh0 ? (s.q_sel ? U.qh1 : U.qh0) + M.eb : nullptr;
  for (uint32_t x = part * blockDim.x + threadIdx.x; x < cnt; x += per * blockDim.x) {
    uint2 hq;
    qd[x] = edge_desc(U, M.eb + (uint32_t)(q[x] & kEidMask), &hq);
    if (qh) qh[x] = hq;
  }
}

// Publish the compacted rows and resume the loop.
__global__ void k_compact_commit(Union* U, const uint32_t* off2, const unsigned long long* row2,
                                 const uint32_t* new_slots, Control* ctl) {
  U->off = off2;
  U->row = row2;
  ctl->csr_slots = *new_slots;
  ctl->compactions += 1;
  ctl->compact_el = ctl->el_proc;
  ctl->exit_reason = kExitNone;
  ctl->done = 0;
}


// Kernel E: truss per slot = level + 2 (pkt.rs:524-526); self-loop slots 2.
// Multigraphs: `smap` takes each slot of the caller's CSR to its pair's slot
// in the deduplicated rows (nullptr: the rows are the caller's).
template <typename OutT>
__global__ void k_finalize(const unsigned long long* __restrict__ row0, const int2* __restrict__ es,
                           unsigned long long width, OutT* __restrict__ out, int u8mode, int out8,
                           uint32_t* __restrict__ kmax, uint32_t* __restrict__ err,
                           const uint32_t* __restrict__ smap) {
  unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  uint32_t mx = 0;
  bool ovf = false;
  for (; i < width; i += stride) {
    const uint32_t e = (uint32_t)(__ldg(row0 + (smap ? __ldg(smap + i) : i)) >> 32);
    uint32_t t = 2;
    if (e != kInvalid) {
      const uint32_t s = (uint32_t)__ldg(&es[e].x);
      t = s + 2;
      if (u8mode) { ovf |= s >= 255; t &= 0xFFu; }
      else if (out8) ovf |= t > 255;
    }
    mx = max(mx, t);
    out[i] = (OutT)t;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mx = max(mx, __shfl_down_sync(__activemask(), mx, d));
  if ((threadIdx.x & 31) == 0) atomicMax(kmax, mx);
  if (ovf) atomicOr(err, kErrOverflowU8);
}

// support per slot (Triangles::new layout): sup of the slot's edge, 0 for self-loops
// ---------------------------------------------------------------------------
// k-core decomposition (the peel of liu_et_al.rs:190-420, level-synchronous):
// degree = row length (mod 256 in u8 mode, the reference's AtomicU8); vertices
// with degree 0 get core 0; at level k every live vertex with degree <= k is
// peeled with core k, and peeling it decrements each neighbour's degree only
// while that degree exceeds k; a neighbour whose degree drops from k + 1 to k
// joins the next sub-level.  The result does not depend on the order.
//
// The level loop runs on the device: one wave is either the scan of level k (live
// vertices of degree <= k join the frontier, the smallest degree left is
// recorded) or one sub-level, and the last block of each wave advances the state
// (the next sub-level, the next level, or a jump past empty levels to the
// smallest degree left) and sets the CUDA-graph loop condition.  Bounded by a
// wave count and the device clock, like the PKT peel.
//
// A sub-level's work is the frontier's row entries, spread evenly over the warps
// through each queue entry's work start: with a warp per frontier vertex one hub
// row of 10^5 entries was 3,000 round trips of one warp (R-MAT-20 42 ms of
// peel, 7.5 now).  Small waves run in one cluster (k_kcore_tail), as the PKT peel's do.
__global__ void __launch_bounds__(256) k_kcore_init(const uint32_t* __restrict__ off, uint32_t n, int u8mode,
                                                    uint32_t* __restrict__ deg, uint32_t* __restrict__ alive,
                                                    uint32_t* __restrict__ core,
                                                    unsigned long long* __restrict__ remaining) {
  uint32_t live = 0;
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    const uint32_t d = __ldg(off + u + 1) - __ldg(off + u);
    deg[u] = u8mode ? (d & 0xFFu) : d;
    alive[u] = d != 0;
    core[u] = 0;
    live += d != 0;
  }
  live = __reduce_add_sync(kFull, live);
  if (lane_id() == 0 && live) atomicAdd(remaining, (unsigned long long)live);
}

struct KcState {
  uint32_t phase;        // 0 scan, 1 sub-level, 2 done
  uint32_t k;
  uint32_t min_left;     // wave accumulator (scan): smallest degree above k
  uint32_t sel;          // queue holding the frontier
  uint32_t levels, subs, kmax;
  uint32_t blocks_done;
  uint32_t err;
  uint32_t pad;
  unsigned long long curr;       // frontier of the sub-level to run: vertices << 32 | row entries
  unsigned long long next;       // wave accumulator: frontier being built
  unsigned long long remaining;  // live vertices
  unsigned long long waves_run, max_waves, t_start, timeout_ns;
};

__global__ void k_kcore_start(KcState* st, unsigned long long max_waves, unsigned long long timeout_ns) {
  st->phase = st->remaining ? 0u : 2u;
  st->k = 1;
  st->curr = 0;
  st->next = 0;
  st->min_left = 0xFFFFFFFFu;
  st->sel = 0;
  st->max_waves = max_waves;
  st->timeout_ns = timeout_ns;
  st->t_start = globaltimer();
}

struct KcArgs {
  const uint32_t* off;
  const uint32_t* nbr;
  uint32_t n;
  uint32_t* deg;
  uint32_t* alive;
  uint32_t* core;
  unsigned long long* q0;  // queue entries: first row entry in the frontier << 32 | vertex
  unsigned long long* q1;
  KcState* st;
  cudaGraphConditionalHandle handle;
  int use_handle;
};

// The lanes that `take` put their vertex v (core k) into the frontier being built.
__device__ __forceinline__ void kc_push(const KcArgs& a, unsigned long long* next, bool take, uint32_t v, uint32_t k) {
  const unsigned bal = __ballot_sync(kFull, take);
  if (!bal) return;
  uint32_t len = 0;
  if (take) {
    a.alive[v] = 0;
    a.core[v] = k;
    len = __ldg(a.off + v + 1) - __ldg(a.off + v);
  }
  uint32_t incl = len;  // a frontier's entries stay below the slot count, 2^32
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(kFull, incl, d);
    if (lane_id() >= (uint32_t)d) incl += o;
  }
  unsigned long long old = 0;
  if (lane_id() == 31) old = atomicAdd(&a.st->next, ((unsigned long long)__popc(bal) << 32) | incl);
  old = __shfl_sync(kFull, old, 31);
  if (take)
    next[(uint32_t)(old >> 32) + __popc(bal & ((1u << lane_id()) - 1))] =
        ((unsigned long long)((uint32_t)old + incl - len) << 32) | v;
}

struct KcStart {
  const unsigned long long* q;
  __device__ __forceinline__ unsigned long long operator()(uint32_t x) const { return q[x] >> 32; }
};

// One wave's share of warp `warp` of `nwarps`.
__device__ __forceinline__ void kc_work(const KcArgs& a, uint32_t phase, uint32_t k, uint32_t sel,
                                        unsigned long long curr, uint32_t warp, uint32_t nwarps) {
  const uint32_t lane = lane_id();
  if (phase == 0) {
    unsigned long long* frontier = sel ? a.q1 : a.q0;
    uint32_t mn = 0xFFFFFFFFu;
    for (unsigned long long b = 32ull * warp; b < a.n; b += 32ull * nwarps) {
      const uint32_t u = (uint32_t)b + lane;
      bool take = false;
      if (b + lane < a.n && a.alive[u]) {
        const uint32_t d = a.deg[u];
        take = d <= k;
        if (!take) mn = min(mn, d);
      }
      kc_push(a, frontier, take, u, k);
    }
    mn = __reduce_min_sync(kFull, mn);
    if (lane == 0 && mn != 0xFFFFFFFFu) atomicMin(&a.st->min_left, mn);
  } else if (phase == 1) {
    const unsigned long long* q = sel ? a.q1 : a.q0;
    unsigned long long* next = sel ? a.q0 : a.q1;
    const uint32_t count = (uint32_t)(curr >> 32), total = (uint32_t)curr;
    // one chunk per warp, 32 consecutive entries per step
    const unsigned long long ch = max(((total + nwarps - 1ull) / nwarps + 31) & ~31ull, 32ull);
    if (warp * ch >= total || count == 0) return;
    const uint32_t kend = (uint32_t)min((warp + 1) * ch, (unsigned long long)total);
    uint32_t i = warp_last_le(KcStart{q}, 0, count - 1, warp * ch);
    for (uint32_t j0 = (uint32_t)(warp * ch); j0 < kend; j0 += 32) {
      // each lane's entry among the 32 from i on (every row has an entry, and the
      // window's first one owns element j0: 32 elements span at most 32 of them)
      const unsigned long long qv = i + lane < count ? q[i + lane] : ~0ull;
      const uint32_t start = (uint32_t)(qv >> 32), j = j0 + lane;
      uint32_t t = 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
        if (__shfl_sync(kFull, start, t + d) <= j) t += d;
      const uint32_t u = __shfl_sync(kFull, (uint32_t)qv, t), at = __shfl_sync(kFull, start, t);
      // on to the owner of j0 + 32: the last lane's entry, or the one after it where
      // that starts there (past the window after 32 rows of one entry)
      const uint32_t tl = __shfl_sync(kFull, t, min(31u, kend - 1 - j0));
      const uint32_t after = tl < 31 ? __shfl_sync(kFull, start, tl + 1)
                             : i + 32 < count ? (uint32_t)(q[i + 32] >> 32) : 0xFFFFFFFFu;
      i += tl + (after <= j0 + 32);
      bool push = false;
      uint32_t v = 0;
      if (j < kend) {
        v = __ldg(a.nbr + __ldg(a.off + u) + (j - at));
        // a degree at or below k belongs to a peeled vertex or one of this
        // level's: it is left alone.  Of the decrements that race past k + 1 one
        // sees it, and the vertex is no longer live for the others.
        if (*(volatile uint32_t*)(a.deg + v) > k) push = atomicSub(a.deg + v, 1u) == k + 1;
      }
      kc_push(a, next, push, v, k);
    }
  }
}

// After a wave: the next one, or the end.  One thread.
__device__ __forceinline__ bool kc_plan(KcState* st) {
  const uint32_t phase = st->phase, k = st->k;
  bool done = phase == 2;
  if (done) return true;
  const unsigned long long next = __ldcg(&st->next);
  if (phase == 0) {
    if (next) {
      st->curr = next;
      st->phase = 1;
      st->levels += 1;
      st->kmax = k;
    } else {
      const uint32_t ml = __ldcg(&st->min_left);
      if (ml == 0xFFFFFFFFu) { st->err |= kErrInternal; done = true; }  // live vertices, none found
      else st->k = max(k + 1, ml);
    }
  } else {
    st->remaining -= min(st->remaining, st->curr >> 32);
    st->subs += 1;
    st->curr = next;
    if (next) {
      st->sel ^= 1u;
    } else {
      st->k = k + 1;
      st->phase = 0;
    }
  }
  st->next = 0;
  st->min_left = 0xFFFFFFFFu;
  st->waves_run += 1;
  if (st->remaining == 0 && st->phase == 0) done = true;
  if (st->waves_run > st->max_waves) { st->err |= kErrWaves; done = true; }
  if (globaltimer() - st->t_start > st->timeout_ns) { st->err |= kErrTimeout; done = true; }
  if (done) st->phase = 2;
  return done;
}

__global__ void __launch_bounds__(256) k_kcore_wave(KcArgs a) {
  kc_work(a, a.st->phase, a.st->k, a.st->sel, a.st->curr, (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
          (gridDim.x * blockDim.x) >> 5);
  // the last block to finish plans the next wave
  __shared__ uint32_t s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&a.st->blocks_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last || threadIdx.x != 0) return;
  __threadfence();
  a.st->blocks_done = 0;
  const bool done = kc_plan(a.st);
  if (a.use_handle) cudaGraphSetConditional(a.handle, done ? 0u : 1u);
}

// Small waves in one cluster (see k_wave_tail): sub-levels of at most `max_work`
// row entries, and scans of graphs of at most that many vertices.
__global__ void __launch_bounds__(kTailThreads, 1) k_kcore_tail(KcArgs a, uint32_t max_work) {
  for (;;) {
    const uint32_t phase = __ldcg(&a.st->phase), k = __ldcg(&a.st->k), sel = __ldcg(&a.st->sel);
    const unsigned long long curr = __ldcg(&a.st->curr);
    if (phase == 2 || (phase == 0 ? a.n : (uint32_t)curr) > max_work) break;
    kc_work(a, phase, k, sel, curr, (threadIdx.x >> 5) * gridDim.x + blockIdx.x, (kTailThreads / 32) * gridDim.x);
    __syncwarp();
    cluster_barrier();
    if (blockIdx.x == 0 && threadIdx.x == 0) kc_plan(a.st);
    __syncwarp();
    cluster_barrier();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.use_handle)
    cudaGraphSetConditional(a.handle, __ldcg(&a.st->phase) == 2 ? 0u : 1u);
}

template <typename OutT>
__global__ void k_kcore_out(const uint32_t* __restrict__ core, uint32_t n, OutT* __restrict__ out) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x)
    out[u] = (OutT)core[u];
}

// Local clustering coefficient per vertex, and the sums behind the average and
// the transitivity, from the edge supports (clustering_coefficient.rs:93-190
// restated): with d = |N(u)| (distinct neighbours; a self-loop counts),
// possible(u) = d(d - 1)/2 for d > 1, t(u) = ceil(sum of u's slot supports /
// 2) = triangles at u, local(u) = t(u) / possible(u) or 0.  Slot supports are
// reduced mod 256 in u8 mode, as the reference's AtomicU8 counts are.  Rows
// of up to kLaneRow entries per lane, longer rows per warp, those of more than
// kWarpRow (`big_list`) per block.
__device__ __forceinline__ uint32_t slot_support(unsigned long long pr, const int2* __restrict__ es,
                                                 int u8mode) {
  const uint32_t e = (uint32_t)(pr >> 32);
  const uint32_t s = e == kInvalid ? 0u : (uint32_t)__ldg(&es[e].x);
  return u8mode ? (s & 0xFFu) : s;
}

// Supports of the slots s, s + step, .. below e, four at a time: their pairs, then
// their edges' supports, are loaded together.
__device__ __forceinline__ unsigned long long row_support(unsigned long long s, uint32_t e, uint32_t step,
                                                          const unsigned long long* __restrict__ row0,
                                                          const int2* __restrict__ es, int u8mode,
                                                          const uint32_t* __restrict__ mult) {
  unsigned long long c = 0;
  for (; s < e; s += 4 * step) {
    unsigned long long pr[4];
    uint32_t sup[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) pr[j] = s + j * step < e ? __ldg(row0 + s + j * step) : ~0ull;
#pragma unroll
    for (int j = 0; j < 4; ++j) sup[j] = slot_support(pr[j], es, u8mode);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      c += (unsigned long long)sup[j] * (mult && s + j * step < e ? __ldg(mult + s + j * step) : 1u);
  }
  return c;
}

// What bounds it: the two dependent loads of a slot; a warp walking hub rows 32
// slots at a time was the whole pass (R-MAT-17, 3.7 M slots: 363 us, now 58).
//
// Multigraphs: the rows are the deduplicated ones (so d counts distinct
// neighbours, the reference's HashSet) and `mult` gives each slot's copies,
// every copy carrying the pair's support.
__global__ void __launch_bounds__(256) k_clustering(const uint32_t* __restrict__ off,
                                                    const unsigned long long* __restrict__ row0,
                                                    const int2* __restrict__ es, uint32_t n, int u8mode,
                                                    double* __restrict__ local, double* __restrict__ sum_possible,
                                                    double* __restrict__ sum_local,
                                                    unsigned long long* __restrict__ sum_slots,
                                                    const uint32_t* __restrict__ mult,
                                                    const uint32_t* __restrict__ big_list,
                                                    const uint32_t* __restrict__ big_count) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  double acc_p = 0.0, acc_l = 0.0;
  unsigned long long acc_s = 0;
  auto vertex = [&](uint32_t u, uint32_t d, unsigned long long ts) {
    const double possible = d > 1 ? (double)d * (double)(d - 1) / 2.0 : 0.0;
    const double tri = (double)((ts + 1) / 2);
    const double loc = possible > 0.0 ? tri / possible : 0.0;
    local[u] = loc;
    acc_p += possible;
    acc_l += loc;
    acc_s += ts;
  };
  __shared__ unsigned long long s_red[32];
  const uint32_t nbig = *big_count;
  for (uint32_t r = blockIdx.x; r < nbig; r += gridDim.x) {
    const uint32_t u = big_list[r], b = __ldg(off + u), e = __ldg(off + u + 1);
    unsigned long long ts;
    block_exclusive_scan<unsigned long long>(
        row_support((unsigned long long)b + threadIdx.x, e, blockDim.x, row0, es, u8mode, mult), s_red, ts);
    if (threadIdx.x == 0) vertex(u, e - b, ts);
  }
  for (uint32_t base = warp * 32; base < n; base += nwarps * 32) {
    const uint32_t u = base + lane;
    uint32_t b = 0, e = 0;
    if (u < n) { b = __ldg(off + u); e = __ldg(off + u + 1); }
    unsigned long long ts = 0;
    if (u < n && e - b <= kLaneRow) ts = row_support(b, e, 1, row0, es, u8mode, mult);
    const bool blk = e - b > kWarpRow;
    unsigned big = __ballot_sync(kFull, u < n && e - b > kLaneRow && !blk);
    while (big) {
      const int j = __ffs(big) - 1;
      big &= big - 1;
      const uint32_t bb = __shfl_sync(kFull, b, j), be = __shfl_sync(kFull, e, j);
      unsigned long long c = row_support((unsigned long long)bb + lane, be, 32, row0, es, u8mode, mult);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) c += __shfl_xor_sync(kFull, c, d);
      if (lane == (uint32_t)j) ts = c;
    }
    if (u < n && !blk) vertex(u, e - b, ts);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    acc_p += __shfl_xor_sync(kFull, acc_p, d);
    acc_l += __shfl_xor_sync(kFull, acc_l, d);
    acc_s += __shfl_xor_sync(kFull, acc_s, d);
  }
  if (lane == 0) {
    if (acc_p != 0.0) atomicAdd(sum_possible, acc_p);
    if (acc_l != 0.0) atomicAdd(sum_local, acc_l);
    if (acc_s) atomicAdd(sum_slots, acc_s);
  }
}

__global__ void k_support_slots(const unsigned long long* __restrict__ row0, const int2* __restrict__ es,
                                unsigned long long width, uint32_t* __restrict__ out, int u8mode,
                                const uint32_t* __restrict__ smap) {
  unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (; i < width; i += stride) {
    const uint32_t e = (uint32_t)(__ldg(row0 + (smap ? __ldg(smap + i) : i)) >> 32);
    uint32_t s = e == kInvalid ? 0u : (uint32_t)__ldg(&es[e].x);
    out[i] = u8mode ? (s & 0xFFu) : s;
  }
}

// ---------------------------------------------------------------------------
// Multigraphs (the reference's OneOrMany paths, impl_csc.rs:154-215,
// triangles.rs:172-224, pkt.rs:373-395): parallel edges are equal neighbour
// ids side by side in a row.  All copies of a pair are interchangeable, so
// they share one truss number; the engine reduces each row to its distinct
// neighbours with a multiplicity per slot, runs the weighted support and peel
// on those rows, and maps every caller slot back to its pair.  A warp per row
// (cold path: only multigraphs take it).
//   k_dedupe_count  distinct neighbours per row
//   k_dedupe_fill   deduplicated rows, copies per slot, caller slot -> slot
//   k_mult_out      multiplicity per edge id, from each pair's out-slot
//   k_mult_check    an in-slot must agree (else the CSR is not symmetric)
__global__ void __launch_bounds__(256) k_dedupe_count(const uint32_t* __restrict__ off,
                                                      const uint32_t* __restrict__ nbr, uint32_t n,
                                                      uint32_t* __restrict__ dcount) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t u = warp; u < n; u += nwarps) {
    const uint32_t b = __ldg(off + u), e = __ldg(off + u + 1);
    uint32_t c = 0;
    for (uint32_t s0 = b; s0 < e; s0 += 32) {
      const uint32_t s = s0 + lane;
      const bool head = s < e && (s == b || __ldg(nbr + s) != __ldg(nbr + s - 1));
      c += __popc(__ballot_sync(kFull, head));
    }
    if (lane == 0) dcount[u] = c;
  }
}

__global__ void __launch_bounds__(256) k_dedupe_fill(const uint32_t* __restrict__ off,
                                                     const uint32_t* __restrict__ nbr, uint32_t n,
                                                     const uint32_t* __restrict__ off2,
                                                     uint32_t* __restrict__ nbr2, uint32_t* __restrict__ mult2,
                                                     uint32_t* __restrict__ smap, uint32_t* __restrict__ err) {
  const uint32_t lane = lane_id();
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t u = warp; u < n; u += nwarps) {
    const uint32_t b = __ldg(off + u), e = __ldg(off + u + 1);
    uint32_t p0 = __ldg(off2 + u);  // slot of the run before this chunk's first head, + 1
    for (uint32_t s0 = b; s0 < e; s0 += 32) {
      const uint32_t s = s0 + lane;
      const uint32_t v = s < e ? __ldg(nbr + s) : 0u;
      const bool head = s < e && (s == b || v != __ldg(nbr + s - 1));
      const unsigned hb = __ballot_sync(kFull, head);
      // the run holding slot s: heads up to and including this lane
      const uint32_t pos = p0 + __popc(hb & (0xFFFFFFFFu >> (31 - lane))) - 1;
      if (s < e) {
        if (head) nbr2[pos] = v;
        smap[s] = pos;
        const uint32_t c = atomicAdd(mult2 + pos, 1u);
        if (c == 0xFFFFu) atomicOr(err, kErrCapacity);  // more than 65535 copies of one pair
      }
      p0 += __popc(hb);
    }
  }
}

__global__ void __launch_bounds__(256) k_mult_out(const unsigned long long* __restrict__ row0,
                                                  const uint32_t* __restrict__ owner,
                                                  const uint32_t* __restrict__ mult2, unsigned long long width,
                                                  uint32_t* __restrict__ mu) {
  for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < width;
       s += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t e = (uint32_t)(__ldg(row0 + s) >> 32);
    if (e != kInvalid && __ldg(owner + s) == kInvalid) mu[e] = __ldg(mult2 + s);
  }
}

__global__ void __launch_bounds__(256) k_mult_check(const unsigned long long* __restrict__ row0,
                                                    const uint32_t* __restrict__ owner,
                                                    const uint32_t* __restrict__ mult2, unsigned long long width,
                                                    const uint32_t* __restrict__ mu, uint32_t* __restrict__ err) {
  bool bad = false;
  for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < width;
       s += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t e = (uint32_t)(__ldg(row0 + s) >> 32);
    if (e != kInvalid && __ldg(owner + s) != kInvalid) bad |= __ldg(mu + e) != __ldg(mult2 + s);
  }
  if (bad) atomicOr(err, kErrAsym);
}

// ---------------------------------------------------------------------------
// Served unions: members join a running peel between graph launches.  Their
// graphs are prepared (narrowed, oriented, supported) as a union of their own,
// then copied behind the running union's vertices, slots and edge ids with
// the ids shifted; their states start at the level-0 scan.
__global__ void k_shift_u32(uint32_t* __restrict__ dst, const uint32_t* __restrict__ src,
                            unsigned long long count, uint32_t add) {
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (unsigned long long)gridDim.x * blockDim.x)
    dst[i] = src[i] + add;
}

// row pairs (name | edge id << 32): name + name_add, edge id + eid_add (self-loops keep kInvalid)
__global__ void k_shift_pairs(unsigned long long* __restrict__ dst, const unsigned long long* __restrict__ src,
                              unsigned long long count, uint32_t name_add, uint32_t eid_add) {
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long pr = src[i];
    const uint32_t name = (uint32_t)pr + name_add, e = (uint32_t)(pr >> 32);
    dst[i] = make_pair(name, e == kInvalid ? kInvalid : e + eid_add);
  }
}

// new members' states (the first wave of a member is its level-0 scan)
__global__ void k_member_init(const Member* __restrict__ mem, MemberState* __restrict__ st, uint32_t g0,
                              uint32_t g1) {
  for (uint32_t g = g0 + blockIdx.x * blockDim.x + threadIdx.x; g < g1; g += gridDim.x * blockDim.x) {
    MemberState s{};
    s.phase = mem[g].m ? kPhaseScan0 : kPhaseDone;
    s.act_count = mem[g].m;
    s.min_kept = 0xFFFFFFFFu;
    st[g] = s;
  }
}

// members joined: the union's member count, wave bound and working-row size grow
__global__ void k_ctl_join(Control* ctl, uint32_t G, unsigned long long add_waves, unsigned long long add_slots) {
  ctl->G = G;
  ctl->max_waves += add_waves;
  ctl->csr_slots += add_slots;
}

// One block: the pending wave's layout again (after members joined), no state
// transitions; restarts the time budget and the loop.
__global__ void k_replan(const Member* __restrict__ mem, const MemberState* __restrict__ st, Control* ctl,
                         unsigned long long* __restrict__ wpref) {
  __shared__ unsigned long long sw[32];
  const uint32_t G = ctl->G;
  unsigned long long carry = 0;
  for (uint32_t b = 0; b < G; b += blockDim.x) {
    const uint32_t g = b + threadIdx.x;
    unsigned long long w = 0;
    if (g < G) {
      const MemberState s = st[g];
      if (s.phase == kPhaseScan0 || s.phase == kPhaseScan) w = s.act_count;
      else if (s.phase == kPhaseProc) w = s.curr & kWorkMask;
    }
    unsigned long long total;
    const unsigned long long ex = block_exclusive_scan<unsigned long long>(w, sw, total);
    if (g < G) wpref[g] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) {
    wpref[G] = carry;
    ctl->total_work = carry;
    ctl->t_start = globaltimer();
    ctl->done = 0;
    ctl->exit_reason = kExitNone;
  }
}

// Hash tables per oriented list (see hash_log2cap; a tuned option of the support
// pass): the lists of at least `min_len` entries get an open-addressed table of
// 2^(1+ceil(log2 d)) 8-byte entries at 4 * the list's start in `pool`.  A warp
// reads the lengths of 32 consecutive lists at once and builds each qualifying
// table in turn in its own slice of shared memory (cleared, filled by
// compare-and-swap, then stored coalesced).  Lists whose table is larger than
// the slice are listed for k_table_fill_big, a block per list, which builds them
// in place.  Every table is written whole, so the pool needs no clearing
// beforehand; entries outside the tables are never read.
constexpr uint32_t kTableSmem = 1024;  // entries per warp (8 KB)
constexpr int kTableWarps = 4;

// support: (name | position << 32) from the oriented out-lists
struct OutListSource {
  const uint32_t* oname;
  __device__ __forceinline__ unsigned long long operator()(uint32_t j) const {
    return (unsigned long long)__ldg(oname + j) | ((unsigned long long)j << 32);
  }
};

template <class Source>
__global__ void __launch_bounds__(kTableWarps * 32) k_table_fill(const uint32_t* __restrict__ off, uint32_t n,
                                                                  uint32_t min_len,
                                                                  Source src, unsigned long long* __restrict__ pool,
                                                                  uint32_t* __restrict__ big, uint32_t* big_count) {
  __shared__ unsigned long long s_tab[kTableWarps][kTableSmem];
  const uint32_t lane = lane_id();
  unsigned long long* st = s_tab[threadIdx.x >> 5];
  const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  for (unsigned long long u0 = warp * 32; u0 < n; u0 += nwarps * 32) {
    const unsigned long long u = u0 + lane;
    uint32_t b = 0, d = 0;
    bool want = false;
    if (u < n) {
      b = __ldg(off + u);
      d = __ldg(off + u + 1) - b;
      want = d >= min_len;
    }
    const bool large = want && hash_log2cap(d) > 31 - __clz(kTableSmem);
    if (large) big[atomicAdd(big_count, 1u)] = (uint32_t)u;
    unsigned todo = __ballot_sync(kFull, want && !large);
    while (todo) {
      const int r = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t rb = __shfl_sync(kFull, b, r), rd = __shfl_sync(kFull, d, r);
      const uint32_t lg = hash_log2cap(rd), cap = 1u << lg, mask = cap - 1;
      for (uint32_t i = lane; i < cap; i += 32) st[i] = ~0ull;
      __syncwarp();
      for (uint32_t x = rb + lane; x < rb + rd; x += 32) {
        const unsigned long long en = src(x);
        if (en == ~0ull) continue;
        uint32_t at = hash_first((uint32_t)en, lg);
        for (uint32_t it = 0; it <= mask; ++it) {
          if (atomicCAS(st + at, ~0ull, en) == ~0ull) break;
          at = (at + 1) & mask;
        }
      }
      __syncwarp();
      unsigned long long* tb = pool + 4ull * rb;
      for (uint32_t i = lane; i < cap; i += 32) tb[i] = st[i];
      __syncwarp();
    }
  }
}

// The listed rows (tables larger than a warp's slice): a block per row, the
// table cleared and filled in place by all its threads.
template <class Source>
__global__ void __launch_bounds__(256) k_table_fill_big(const uint32_t* __restrict__ off,
                                                        const uint32_t* __restrict__ big,
                                                        const uint32_t* __restrict__ big_count, Source src,
                                                        unsigned long long* __restrict__ pool) {
  const uint32_t nb = *big_count;
  for (uint32_t i = blockIdx.x; i < nb; i += gridDim.x) {
    const uint32_t u = big[i];
    const uint32_t rb = __ldg(off + u), rd = __ldg(off + u + 1) - rb;
    const uint32_t lg = hash_log2cap(rd), cap = 1u << lg, mask = cap - 1;
    unsigned long long* tb = pool + 4ull * rb;
    for (uint32_t j = threadIdx.x; j < cap; j += blockDim.x) tb[j] = ~0ull;
    __syncthreads();
    for (uint32_t x = rb + threadIdx.x; x < rb + rd; x += blockDim.x) {
      const unsigned long long en = src(x);
      if (en == ~0ull) continue;
      uint32_t at = hash_first((uint32_t)en, lg);
      for (uint32_t it = 0; it <= mask; ++it) {
        if (atomicCAS(tb + at, ~0ull, en) == ~0ull) break;
        at = (at + 1) & mask;
      }
    }
    __syncthreads();
  }
}

}  // namespace sparx
