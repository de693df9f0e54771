// MatrixMarket text -> CSR on the GPU (the input side of the path): the
// reference's GraphCache::from_mtx_file (graph/cache/parser_mtx/mod.rs:34-162)
// parses entry lines with host threads (parser_mtx/producers.rs:139-240),
// counts degrees, scatters neighbours and sorts every row
// (graph/cache/impl_sort.rs:10-51).  Here the body of the file is one device
// buffer:
//   k_mtx_count_lines / k_mtx_fill_lines   line starts (a byte after '\n')
//   k_mtx_parse                             per line: skip blank and '%' lines
//                                           and lines with fewer than two
//                                           tokens, parse i j (1-based), flag
//                                           0 or out-of-range indices; entry
//                                           (i-1, j-1) and the number of keys
//   k_mtx_emit                              the entry and, for a symmetric
//                                           header and i != j, the mirror, as
//                                           keys row << bits | column (bits:
//                                           of a vertex id)
//   k_radix_hist / k_radix_scatter          stable LSD radix sort of the keys
//                                           (8-bit digits): sorted keys are the
//                                           CSR rows in order, each ascending
//   k_mtx_rows                              row lengths -> offsets (scanned),
//                                           columns -> neighbours
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sparx {

enum : uint32_t {
  kMtxZeroIndex = 1u,    // an index of 0 (MatrixMarket is 1-based)
  kMtxOutOfRange = 2u,   // an index beyond the size line
  kMtxBadNumber = 4u,    // a token that is not an unsigned integer
};

// Rust's char::is_whitespace on ASCII (what str::trim and split_whitespace use)
__device__ __forceinline__ bool mtx_space(unsigned char c) {
  return c == ' ' || c == '\t' || c == '\n' || c == '\r' || c == 0x0B || c == 0x0C;
}

__device__ __forceinline__ bool line_start(const unsigned char* __restrict__ body, unsigned long long p) {
  return p == 0 || body[p - 1] == '\n';
}

// line starts per 16-byte chunk: the '\n' among the byte before it and its first
// 15, read as one 16-byte word (`body` is aligned; a byte at a time the two passes of
// the scan took 130 us for 25 MB, so 34)
struct MtxLineCount {
  const unsigned char* body;
  unsigned long long len;
  __device__ __forceinline__ unsigned long long operator()(unsigned long long c) const {
    const unsigned long long b = c * 16;
    if (b + 16 > len) {
      unsigned long long n = 0;
      for (unsigned long long p = b; p < len; ++p) n += line_start(body, p);
      return n;
    }
    const uint4 w = __ldg((const uint4*)(body + b));
    constexpr uint32_t nl = 0x0A0A0A0Au;
    // 8 bits set per equal byte; the chunk's last byte starts the next chunk's line
    const uint32_t bits = __popc(__vcmpeq4(w.x, nl)) + __popc(__vcmpeq4(w.y, nl)) + __popc(__vcmpeq4(w.z, nl)) +
                          __popc(__vcmpeq4(w.w, nl) & 0x00FFFFFFu);
    return (bits >> 3) + line_start(body, b);
  }
};

__global__ void __launch_bounds__(256) k_mtx_fill_lines(const unsigned char* __restrict__ body,
                                                        unsigned long long len,
                                                        const unsigned long long* __restrict__ chunk_pref,
                                                        unsigned long long* __restrict__ starts) {
  const unsigned long long chunks = (len + 15) / 16;
  for (unsigned long long c = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; c < chunks;
       c += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long at = chunk_pref[c];
    const unsigned long long b = c * 16, e = min(b + 16, len);
    for (unsigned long long p = b; p < e; ++p)
      if (line_start(body, p)) starts[at++] = p;
  }
}

// Unsigned decimal token at [p, e): Rust's usize::from_str (an optional '+',
// then digits; anything else, or a value past 64 bits, fails).
__device__ __forceinline__ bool mtx_number(const unsigned char* __restrict__ body, unsigned long long p,
                                           unsigned long long e, unsigned long long* out) {
  if (p < e && body[p] == '+') ++p;
  if (p >= e) return false;
  unsigned long long v = 0;
  for (; p < e; ++p) {
    const unsigned c = body[p] - '0';
    if (c > 9) return false;
    if (v > (~0ull - c) / 10) return false;
    v = v * 10 + c;
  }
  *out = v;
  return true;
}

// One thread per line: its keys counted into `count`, its entry (row << 32 | column)
// into `entry`, error flags with the first failing line.  Bound by the byte loads
// of a line (each thread its own sectors); a second parse to emit the keys took as
// long again as this one (63 us for 1.85 M lines), reading the entry back takes 12.
__global__ void __launch_bounds__(256) k_mtx_parse(const unsigned char* __restrict__ body,
                                                   unsigned long long len,
                                                   const unsigned long long* __restrict__ starts,
                                                   unsigned long long lines, unsigned long long n, int symmetric,
                                                   uint32_t* __restrict__ count,
                                                   unsigned long long* __restrict__ entry, uint32_t* __restrict__ err,
                                                   unsigned long long* __restrict__ bad_line) {
  for (unsigned long long l = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; l < lines;
       l += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long p = starts[l];
    // the next line starts after this one's '\n'; the last line may lack its own
    const unsigned long long end = l + 1 < lines ? starts[l + 1] - 1 : len - (body[len - 1] == '\n');
    while (p < end && mtx_space(body[p])) ++p;  // trim
    uint32_t edges = 0, flags = 0;
    unsigned long long i = 0, j = 0;
    if (p < end && body[p] != '%') {
      unsigned long long t0 = p;
      while (p < end && !mtx_space(body[p])) ++p;
      const unsigned long long t0e = p;
      while (p < end && mtx_space(body[p])) ++p;
      const unsigned long long t1 = p;
      while (p < end && !mtx_space(body[p])) ++p;
      const unsigned long long t1e = p;
      if (t1 < t1e) {  // two tokens (fewer: the line is skipped)
        if (!mtx_number(body, t0, t0e, &i) || !mtx_number(body, t1, t1e, &j)) flags |= kMtxBadNumber;
        else if (i == 0 || j == 0) flags |= kMtxZeroIndex;
        else if (i > n || j > n) flags |= kMtxOutOfRange;
        else edges = (symmetric && i != j) ? 2u : 1u;
      }
    }
    count[l] = edges;
    if (edges) entry[l] = ((i - 1) << 32) | (j - 1);
    if (flags) {
      atomicOr(err, flags);
      atomicMin(bad_line, l);
    }
  }
}

// The lines' keys, row << bits | column, at their places `at`.
__global__ void __launch_bounds__(256) k_mtx_emit(const uint32_t* __restrict__ count,
                                                  const unsigned long long* __restrict__ entry,
                                                  const unsigned long long* __restrict__ at, unsigned long long lines,
                                                  int bits, unsigned long long* __restrict__ keys) {
  for (unsigned long long l = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; l < lines;
       l += (unsigned long long)gridDim.x * blockDim.x) {
    const uint32_t edges = count[l];
    if (!edges) continue;
    const unsigned long long o = at[l], i = entry[l] >> 32, j = entry[l] & 0xFFFFFFFFull;
    keys[o] = (i << bits) | j;
    if (edges == 2) keys[o + 1] = (j << bits) | i;
  }
}

struct LoadCount {
  const uint32_t* p;
  __device__ __forceinline__ unsigned long long operator()(unsigned long long i) const { return p[i]; }
};

// ---------------------------------------------------------------------------
// Stable LSD radix sort of u64 keys, 8 bits per pass.  Each block owns a
// contiguous segment; hist[d * blocks + b] counts digit d in block b's segment,
// its exclusive scan (digit-major) gives every (digit, block) its output start,
// and the scatter places the segment's keys in order: items go through in rounds
// of kRadixRound, a warp taking 32 * kRadixItems consecutive ones in groups of 32
// (match + popcount of the lower lanes, after what the warp's earlier groups had of
// the digit); then the warps' counts become starts.  Two barriers per round of 1024
// instead of three per 256: 3.7 M keys 38 -> 29 us a pass (60 MB, 9 us at the copy
// bandwidth; what is left is the scattered 8-byte stores and the rounds' latency).
constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixItems = 4;
constexpr int kRadixRound = kRadixThreads * kRadixItems;

__device__ __forceinline__ unsigned long long radix_segment(unsigned long long count, uint32_t blocks, uint32_t b) {
  const unsigned long long per = (count + blocks - 1) / blocks;
  return min(count, per * b);
}

__global__ void __launch_bounds__(kRadixThreads) k_radix_hist(const unsigned long long* __restrict__ keys,
                                                              unsigned long long count, int shift,
                                                              uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const unsigned long long b0 = radix_segment(count, gridDim.x, blockIdx.x);
  const unsigned long long b1 = radix_segment(count, gridDim.x, blockIdx.x + 1);
  for (unsigned long long i = b0 + threadIdx.x; i < b1; i += kRadixThreads)
    atomicAdd(&h[(keys[i] >> shift) & 0xFF], 1u);
  __syncthreads();
  hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// kPay: a u32 payload travels with each key (pin -> pout), in the same order.
template <bool kPay>
__global__ void __launch_bounds__(kRadixThreads) k_radix_scatter(const unsigned long long* __restrict__ in,
                                                                 unsigned long long* __restrict__ out,
                                                                 unsigned long long count, int shift,
                                                                 const uint32_t* __restrict__ start,
                                                                 const uint32_t* __restrict__ pin,
                                                                 uint32_t* __restrict__ pout) {
  __shared__ uint32_t warp_cnt[kRadixWarps][256];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t run = start[threadIdx.x * gridDim.x + blockIdx.x];  // this thread's digit's next place
  const unsigned long long b0 = radix_segment(count, gridDim.x, blockIdx.x);
  const unsigned long long b1 = radix_segment(count, gridDim.x, blockIdx.x + 1);
  for (unsigned long long r = b0; r < b1; r += kRadixRound) {
    // a warp's row of counts is its own until the first barrier and after the second
    for (uint32_t x = lane; x < 256; x += 32) warp_cnt[wid][x] = 0;
    const unsigned long long w0 = r + wid * (32 * kRadixItems) + lane;
    unsigned long long k[kRadixItems];
    uint32_t pl[kRadixItems], d[kRadixItems], rank[kRadixItems];
#pragma unroll
    for (int q = 0; q < kRadixItems; ++q) {
      const bool valid = w0 + 32 * q < b1;
      k[q] = valid ? in[w0 + 32 * q] : 0ull;
      pl[q] = kPay && valid ? pin[w0 + 32 * q] : 0u;
      d[q] = valid ? (uint32_t)((k[q] >> shift) & 0xFF) : 256u;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kRadixItems; ++q) {
      const unsigned same = __match_any_sync(0xFFFFFFFFu, d[q]);
      const uint32_t lower = __popc(same & ((1u << lane) - 1));
      const uint32_t seen = d[q] < 256 ? warp_cnt[wid][d[q]] : 0u;
      rank[q] = seen + lower;
      __syncwarp();
      if (d[q] < 256 && lower == 0) warp_cnt[wid][d[q]] = seen + __popc(same);
      __syncwarp();
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kRadixWarps; ++w) {
      const uint32_t c = warp_cnt[w][threadIdx.x];
      warp_cnt[w][threadIdx.x] = run;
      run += c;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kRadixItems; ++q)
      if (d[q] < 256) {
        const uint32_t to = warp_cnt[wid][d[q]] + rank[q];
        out[to] = k[q];
        if (kPay) pout[to] = pl[q];
      }
    __syncwarp();
  }
}

// Row lengths and neighbours from the sorted keys (rows are contiguous runs of equal
// row parts): a warp adds each of its runs once (14 us for 3.7 M keys; an atomic per key and
// the columns in a pass of their own 65).
__global__ void __launch_bounds__(256) k_mtx_rows(const unsigned long long* __restrict__ keys, unsigned long long count,
                                                  int bits, uint32_t* __restrict__ deg,
                                                  unsigned long long* __restrict__ nbr) {
  const uint32_t lane = threadIdx.x & 31;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i0 = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < count;
       i0 += stride) {
    const unsigned long long i = i0 + lane;
    const bool valid = i < count;
    const unsigned long long k = valid ? keys[i] : ~0ull;
    const unsigned long long row = valid ? k >> bits : ~0ull;
    const unsigned long long prev = __shfl_up_sync(0xFFFFFFFFu, row, 1);
    const unsigned heads = __ballot_sync(0xFFFFFFFFu, lane == 0 || row != prev);
    if (valid) {
      nbr[i] = k & ((1ull << bits) - 1);
      if ((heads >> lane) & 1) {
        const unsigned later = lane < 31 ? heads >> (lane + 1) : 0u;  // the next head ends this run
        const uint32_t to = later ? lane + __ffs(later) : 32u;
        const uint32_t last = (uint32_t)min(32ull, count - i0);
        atomicAdd(&deg[row], min(to, last) - lane);
      }
    }
  }
}

}  // namespace sparx
