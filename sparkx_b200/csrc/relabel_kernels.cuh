// Vertex relabelling for locality: vertices take new ids in (floor(log2
// degree), id) order, within their own graph's id range in a union, and the
// CSR is rebuilt on them; the caller's
// slot s maps to the new slot rmap[s].  Rows are sorted by id, and within a
// degree bucket the new ids keep the old order, so each new row is the old
// row stably partitioned by its neighbours' buckets: no sort of the slots is
// needed.  Edges of similar-degree vertices sit together, so the peel's random
// state and row reads fall on far fewer lines, and the copy is oriented by id
// alone, which shortens the support pass's searches: R-MAT-22 (orientation +
// support + peel) 6.3 + 50.8 + 249.9 -> 9.0 + 31.1 + 215.6 ms, R-MAT-21 with edge
// factor 12 2.0 + 14.2 + 87.7 -> 4.4 + 8.8 + 82.4.
//   k_vertex_keys       ((member << 5 | bucket) << 32 | id) per vertex, for the
//                       radix passes (one for a single graph)
//   k_vertex_order      new id and new degree per vertex
//   k_relabel_rows      a warp per row of at most kRelabelWarpRow entries
//   k_relabel_rows_big  a block per longer row (the listed big rows)
// Both row kernels count the row's entries per bucket, scan the 32 counts,
// then place the entries chunk by chunk in their order: an entry's place is
// its bucket's cursor plus the same-bucket entries before it in the chunk.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sparx {

constexpr uint32_t kRelabelWarpRow = 2048;  // longer rows: a block each (the orientation's big-row list)

__device__ __forceinline__ uint32_t degree_bucket(uint32_t d) { return d > 1 ? 31u - __clz(d) : 0u; }

// Keys ((member << 5 | bucket) << 32 | id): in a union of G graphs (members
// by ascending first vertex `vb`) every vertex keeps to its member's id range.
__global__ void __launch_bounds__(256) k_vertex_keys(const uint32_t* __restrict__ off, uint32_t n,
                                                     const uint32_t* __restrict__ member_vb, uint32_t G,
                                                     unsigned long long* __restrict__ keys,
                                                     uint8_t* __restrict__ bucket) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    const uint32_t b = degree_bucket(__ldg(off + u + 1) - __ldg(off + u));
    uint32_t lo = 0, hi = G - 1;  // the last member whose first vertex is <= u
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (__ldg(member_vb + mid) <= u) lo = mid; else hi = mid - 1;
    }
    keys[u] = ((unsigned long long)((lo << 5) | b) << 32) | u;
    bucket[u] = (uint8_t)b;
  }
}

__global__ void __launch_bounds__(256) k_vertex_order(const unsigned long long* __restrict__ sorted,
                                                      const uint32_t* __restrict__ off, uint32_t n,
                                                      uint32_t* __restrict__ newid, uint32_t* __restrict__ deg_new) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const uint32_t u = (uint32_t)sorted[p];
    newid[u] = p;
    deg_new[p] = __ldg(off + u + 1) - __ldg(off + u);
  }
}

// Entries of a row a lane holds at a time: their buckets and new ids are loaded side
// by side.
constexpr int kRelabelWays = 4;

struct RelabelEntries {
  uint32_t v[kRelabelWays], bk[kRelabelWays];  // bucket 32: no entry
  __device__ __forceinline__ void load(const uint32_t* __restrict__ nbr, const uint8_t* __restrict__ bucket,
                                       unsigned long long s0, uint32_t e) {
#pragma unroll
    for (int q = 0; q < kRelabelWays; ++q) v[q] = s0 + 32 * q < e ? __ldg(nbr + s0 + 32 * q) : 0u;
#pragma unroll
    for (int q = 0; q < kRelabelWays; ++q) bk[q] = s0 + 32 * q < e ? bucket[v[q]] : 32u;
  }
  __device__ __forceinline__ void count(uint32_t* cnt) const {
#pragma unroll
    for (int q = 0; q < kRelabelWays; ++q)
      if (bk[q] < 32u) atomicAdd(&cnt[bk[q]], 1u);
  }
};

// exclusive scan over the warp
__device__ __forceinline__ uint32_t relabel_scan(uint32_t c) {
  uint32_t x = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if ((threadIdx.x & 31) >= (uint32_t)d) x += y;
  }
  return x - c;
}

// Rows of at most kRelabelWarpRow entries, a warp each (rows over it are
// k_relabel_rows_big's).  Bound by the chain offsets -> entry -> bucket -> counts ->
// place: a warp reads the bounds and new places of 32 rows at once, and rows of up to
// 128 entries stay in registers between counting and placing (R-MAT-22 1440 -> 1200 us).
__global__ void __launch_bounds__(256) k_relabel_rows(const uint32_t* __restrict__ off,
                                                      const uint32_t* __restrict__ nbr, uint32_t n,
                                                      const uint32_t* __restrict__ newid,
                                                      const uint8_t* __restrict__ bucket,
                                                      const uint32_t* __restrict__ off_new,
                                                      uint32_t* __restrict__ nbr_new, uint32_t* __restrict__ rmap) {
  __shared__ uint32_t s_cur[8][32];
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  uint32_t* cur = s_cur[wib];  // the row's bucket counts, then the buckets' cursors
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = (gridDim.x * blockDim.x) >> 5;
  constexpr uint32_t kStep = 32 * kRelabelWays;
  for (unsigned long long u0 = warp; u0 < n; u0 += 32 * nwarps) {
    const unsigned long long mine = u0 + lane * nwarps;  // a warp's rows are nwarps apart
    uint32_t mb = 0, me = 0, mbase = 0;
    if (mine < n) {
      mb = __ldg(off + mine);
      me = __ldg(off + mine + 1);
      mbase = __ldg(off_new + __ldg(newid + mine));
    }
    unsigned todo = __ballot_sync(0xFFFFFFFFu, me > mb && me - mb <= kRelabelWarpRow);
    while (todo) {
      const int j = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t b = __shfl_sync(0xFFFFFFFFu, mb, j), e = __shfl_sync(0xFFFFFFFFu, me, j);
      const uint32_t base = __shfl_sync(0xFFFFFFFFu, mbase, j);
      // per-bucket counts of the row, then their exclusive scan (lane = bucket)
      RelabelEntries E;
      cur[lane] = 0;
      __syncwarp();
      for (unsigned long long s0 = b; s0 < e; s0 += kStep) {
        E.load(nbr, bucket, s0 + lane, e);
        E.count(cur);
      }
      __syncwarp();
      const uint32_t c = cur[lane];
      const uint32_t at0 = base + relabel_scan(c);
      __syncwarp();
      cur[lane] = at0;
      __syncwarp();
      for (unsigned long long s0 = b; s0 < e; s0 += kStep) {
        if (e - b > kStep) E.load(nbr, bucket, s0 + lane, e);
        uint32_t to[kRelabelWays];
#pragma unroll
        for (int q = 0; q < kRelabelWays; ++q) to[q] = E.bk[q] < 32u ? __ldg(newid + E.v[q]) : 0u;
#pragma unroll
        for (int q = 0; q < kRelabelWays; ++q) {
          if (s0 + 32 * q >= e) break;
          const bool valid = E.bk[q] < 32u;
          const unsigned same = __match_any_sync(0xFFFFFFFFu, E.bk[q]);
          const uint32_t rank = __popc(same & ((1u << lane) - 1));
          uint32_t at = 0;
          if (valid) at = cur[E.bk[q]] + rank;
          __syncwarp();
          if (valid) {
            nbr_new[at] = to[q];
            rmap[s0 + 32 * q + lane] = at;
            if (rank == 0) cur[E.bk[q]] += __popc(same);
          }
          __syncwarp();
        }
      }
    }
  }
}

// The listed rows longer than kRelabelWarpRow, a block of 256 each, in rounds of 1024
// entries: a warp ranks its 128 consecutive ones by itself, then the warps' bucket
// counts become places.  The longest row is the pass: R-MAT-22 (130 thousand entries) 1570 us in
// rounds of 256 with three barriers, now 900.
__global__ void __launch_bounds__(256) k_relabel_rows_big(const uint32_t* __restrict__ off,
                                                          const uint32_t* __restrict__ nbr,
                                                          const uint32_t* __restrict__ list,
                                                          const uint32_t* __restrict__ count,
                                                          const uint32_t* __restrict__ newid,
                                                          const uint8_t* __restrict__ bucket,
                                                          const uint32_t* __restrict__ off_new,
                                                          uint32_t* __restrict__ nbr_new, uint32_t* __restrict__ rmap) {
  __shared__ uint32_t s_cnt[32];
  __shared__ uint32_t s_wc[8][32];
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t nbig = *count;
  const uint32_t warp_at = wib * 32 * kRelabelWays + lane;
  constexpr uint32_t kRound = 256 * kRelabelWays;
  for (uint32_t r = blockIdx.x; r < nbig; r += gridDim.x) {
    const uint32_t u = list[r];
    const uint32_t b = __ldg(off + u), e = __ldg(off + u + 1);
    RelabelEntries E;
    if (threadIdx.x < 32) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    for (unsigned long long s0 = b; s0 < e; s0 += kRound) {
      E.load(nbr, bucket, s0 + warp_at, e);
      E.count(s_cnt);
    }
    __syncthreads();
    uint32_t run = 0;  // of the first warp's lanes: their bucket's next place
    if (threadIdx.x < 32) run = __ldg(off_new + __ldg(newid + u)) + relabel_scan(s_cnt[threadIdx.x]);
    for (unsigned long long s0 = b; s0 < e; s0 += kRound) {
      // a warp's row of counts is its own until the first barrier and after the second
      s_wc[wib][lane] = 0;
      E.load(nbr, bucket, s0 + warp_at, e);
      uint32_t to[kRelabelWays], rank[kRelabelWays];
#pragma unroll
      for (int q = 0; q < kRelabelWays; ++q) to[q] = E.bk[q] < 32u ? __ldg(newid + E.v[q]) : 0u;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < kRelabelWays; ++q) {
        const unsigned same = __match_any_sync(0xFFFFFFFFu, E.bk[q]);
        const uint32_t lower = __popc(same & ((1u << lane) - 1));
        const uint32_t seen = E.bk[q] < 32u ? s_wc[wib][E.bk[q]] : 0u;
        rank[q] = seen + lower;
        __syncwarp();
        if (E.bk[q] < 32u && lower == 0) s_wc[wib][E.bk[q]] = seen + __popc(same);
        __syncwarp();
      }
      __syncthreads();
      if (threadIdx.x < 32) {
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          const uint32_t c = s_wc[w][threadIdx.x];
          s_wc[w][threadIdx.x] = run;
          run += c;
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kRelabelWays; ++q)
        if (E.bk[q] < 32u) {
          const uint32_t at = s_wc[wib][E.bk[q]] + rank[q];
          nbr_new[at] = to[q];
          rmap[s0 + warp_at + 32 * q] = at;
        }
      __syncwarp();
    }
    __syncthreads();  // s_cnt of the next row
  }
}

}  // namespace sparx
