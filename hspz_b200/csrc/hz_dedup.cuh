// dedup_and_order (src/hsp.rs:94-126) on the device, for every dedup scope
// of a wave at once.
//
// The raw HSPs of a wave carry their scope.  They are ordered by (scope,
// diagonal, ref_start, len, score descending) -- hspComp within each scope.  A
// record is kept when it starts its scope or is not contained in the previous
// INPUT record (hspEqual compares against the previous element, not the last
// kept one).  The kept records are then ordered by (scope, query_start,
// ref_start, len, score descending) -- hspCompLastz within each scope.  Both
// orders are total over the four fields, so any sort gives the reference's
// stable sorts.
//
// Most raw HSPs are copies: every seed of a homologous stretch finds the same
// one.  A copy follows its original in the first order and is contained in
// it, and the record after both is compared with the same fields either way,
// so exact copies are taken out first, by a hash set (unique_kernel); 630 000
// raw HSPs of a 16 Mbp batch are 2 500 different ones.
//
// The sorts are merge sorts of record indices: blocks sort tiles of kSortTile
// records in shared memory, then passes merge pairs of sorted runs, a block
// per kSortTile outputs.  Each is bound by latency at these sizes (~11 us a
// pass at 200 000 records), so what counts is their number: one block sort and
// log2(n / kSortTile) passes, where an 8-bit radix sort of the five fields
// takes 20 passes of five launches.  Both sorts, filter and output of 200 003
// records: 1078 us by radix sorts, 203 us; 2048 records 56 us.  A batch's
// 105 000 raw HSPs (900 kept): 1.06 ms, 0.08 with the set.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "hz_device.cuh"

namespace hz {

// Output record of a wave: the scope and the HSP.
struct ScopedHspOut {
  uint32_t scope;
  SegmentPair h;
};

// An HSP of a caller's buffer, which need only be 4-byte aligned.
struct PlainHsp {
  uint32_t ref_start, query_start, len;
  int32_t score;
};
__device__ __forceinline__ SegmentPair load_hsp(const SegmentPair *p) { return *p; }
__device__ __forceinline__ SegmentPair load_hsp(const PlainHsp *p) {
  return SegmentPair{p->ref_start, p->query_start, p->len, p->score};
}

// hspEqual (src/hsp.rs:83-87): same diagonal and one [start, start+len]
// reference interval inside the other, with wrapping ends.
__device__ __forceinline__ bool contained_dev(const SegmentPair &x, const SegmentPair &y) {
  uint32_t xe = x.ref_start + x.len, ye = y.ref_start + y.len;
  return (x.ref_start - x.query_start) == (y.ref_start - y.query_start) &&
         ((x.ref_start >= y.ref_start && xe <= ye) || (y.ref_start >= x.ref_start && ye <= xe));
}

// ---------------------------------------------------------------------------
// Exact copies out.  table: `slots` words (at least twice the records),
// zeroed; an entry is a record's index + 1.  The first of equal records to
// claim an entry is one of the distinct ones: its index goes to out, *n_out
// counts them, and the first `n_head` go to head as well.
__device__ __forceinline__ uint32_t hsp_hash(const SegmentPair &h, uint32_t scope) {
  uint32_t x = h.ref_start * 0x9E3779B1u ^ (h.query_start + 0x85EBCA6Bu) * 0xC2B2AE35u;
  x = (x ^ x >> 15) * 0x2C1B3C6Du ^ h.len * 0x297A2D39u ^ (uint32_t)h.score * 0x165667B1u ^ scope * 0x27D4EB2Fu;
  x = (x ^ x >> 13) * 0x85EBCA77u;
  return x ^ x >> 16;
}

__global__ void __launch_bounds__(256) unique_kernel(const SegmentPair *__restrict__ raw,
                                                     const uint32_t *__restrict__ raw_scope,
                                                     const uint32_t *__restrict__ n_raw, uint32_t cap,
                                                     uint32_t *table, uint32_t slots, uint32_t *__restrict__ out,
                                                     uint32_t *n_out, ScopedHspOut *__restrict__ head,
                                                     uint32_t n_head) {
  const uint32_t n = min(*n_raw, cap);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const SegmentPair h = raw[i];
    const uint32_t scope = raw_scope[i];
    bool first = false;
    uint32_t at = (uint32_t)(((unsigned long long)hsp_hash(h, scope) * slots) >> 32);
    while (true) {
      // most entries met are taken: look before claiming
      uint32_t e = *(volatile uint32_t *)&table[at];
      if (!e) {
        e = atomicCAS(&table[at], 0u, i + 1);
        if (!e) {
          first = true;
          break;
        }
      }
      const SegmentPair o = raw[e - 1];
      if (o.ref_start == h.ref_start && o.query_start == h.query_start && o.len == h.len && o.score == h.score &&
          raw_scope[e - 1] == scope)
        break;
      at = at + 1 < slots ? at + 1 : 0u;
    }
    if (first) {
      const uint32_t k = atomicAdd(n_out, 1u);
      out[k] = i;
      if (k < n_head) head[k] = ScopedHspOut{scope, h};
    }
  }
}

// ---------------------------------------------------------------------------
// Sort keys: five words, most significant first.

enum DedupOrder : int { kByDiagonal, kByLastz };

struct DedupKey {
  unsigned long long a, b;
  uint32_t c;
};
__device__ __forceinline__ bool key_less(const DedupKey &x, const DedupKey &y) {
  return x.a != y.a ? x.a < y.a : x.b != y.b ? x.b < y.b : x.c < y.c;
}
template <int ORDER> __device__ __forceinline__ DedupKey key_of(const SegmentPair &h, uint32_t scope) {
  const uint32_t second = ORDER == kByDiagonal ? h.ref_start - h.query_start  // wrapping u32 diagonal (src/hsp.rs:49-51)
                                               : h.query_start;
  return DedupKey{(unsigned long long)scope << 32 | second, (unsigned long long)h.ref_start << 32 | h.len,
                  ~((uint32_t)h.score ^ 0x80000000u)};  // larger score sorts first
}

// Few records per thread: the merges inside a tile are chains of shared-memory
// reads, and 1024 threads of two records shorten them (200 003 records: 203 us
// against 218 with 512 threads and 287 with 256).
constexpr int kSortThreads = 1024;
constexpr int kSortItems = 2;
constexpr uint32_t kSortTile = kSortThreads * kSortItems;  // 2048

// A tile's keys in shared memory (kept in place) for sorts of their slots.
struct SortTile {
  unsigned long long a[kSortTile], b[kSortTile];
  uint32_t c[kSortTile];
  uint16_t ord[kSortTile];
  __device__ __forceinline__ bool less(uint32_t x, uint32_t y) const {
    if (a[x] != a[y]) return a[x] < a[y];
    if (b[x] != b[y]) return b[x] < b[y];
    return c[x] < c[y];
  }
  __device__ __forceinline__ void put(uint32_t i, const DedupKey &k) {
    a[i] = k.a;
    b[i] = k.b;
    c[i] = k.c;
  }
};

// How many of the first `diag` outputs of merging tile slots A[0, na) and
// B[0, nb) (both sorted) come from A; equal keys take A first.
template <typename L> __device__ __forceinline__ uint32_t merge_split(uint32_t diag, uint32_t na, uint32_t nb, L b_before_a) {
  uint32_t lo = diag > nb ? diag - nb : 0u, hi = min(diag, na);
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (b_before_a(mid, diag - 1 - mid)) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// Records a sort reads: their buffer, scopes (null: all 0), the indices to
// sort (null: 0, 1, ...) and their number on the device (null: n).
template <typename H> struct SortArgs {
  const H *recs;
  const uint32_t *scope;
  const uint32_t *idx;
  const uint32_t *n_dev;
  uint32_t n;
  uint32_t *out;
  __device__ __forceinline__ uint32_t count() const { return n_dev ? *n_dev : n; }
  template <int ORDER> __device__ __forceinline__ DedupKey key(uint32_t i) const {
    return key_of<ORDER>(load_hsp(recs + i), scope ? scope[i] : 0u);
  }
};

// Sorts each tile of kSortTile indices.
template <int ORDER, typename H> __global__ void __launch_bounds__(kSortThreads) sort_tiles_kernel(SortArgs<H> s) {
  __shared__ SortTile t;
  const uint32_t n = s.count(), base = blockIdx.x * kSortTile;
  if (base >= n) return;
  const uint32_t m = min(n - base, kSortTile), tid = threadIdx.x;
  uint32_t src[kSortItems];
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    const uint32_t p = i * kSortThreads + tid;
    src[i] = p < m ? (s.idx ? s.idx[base + p] : base + p) : 0u;
  }
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    const uint32_t p = i * kSortThreads + tid;
    t.put(p, p < m ? s.template key<ORDER>(src[i]) : DedupKey{~0ull, ~0ull, ~0u});
  }
  __syncthreads();
  // each thread's slots in registers (insertion), then merges of
  // doubling width; slots past m hold the largest key and stay last
  uint16_t o[kSortItems];
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    o[i] = (uint16_t)(tid * kSortItems + i);
#pragma unroll
    for (int j = i; j > 0; j--)
      if (t.less(o[j], o[j - 1])) {
        const uint16_t x = o[j];
        o[j] = o[j - 1];
        o[j - 1] = x;
      }
  }
  for (uint32_t width = kSortItems; width < kSortTile; width *= 2) {
#pragma unroll
    for (int i = 0; i < kSortItems; i++) t.ord[tid * kSortItems + i] = o[i];
    __syncthreads();
    if (width < m) {
      const uint32_t at = tid * kSortItems, pair = at & ~(2 * width - 1);
      const uint16_t *A = t.ord + pair, *B = A + width;
      uint32_t x = merge_split(at - pair, width, width,
                               [&](uint32_t i, uint32_t j) { return t.less(B[j], A[i]); });
      uint32_t y = at - pair - x;
#pragma unroll
      for (int i = 0; i < kSortItems; i++) {
        const bool b = x >= width || (y < width && t.less(B[y], A[x]));
        o[i] = b ? B[y++] : A[x++];
      }
    }
    __syncthreads();
  }
  // the sorted slots' indices (the slots' own are still in the registers)
#pragma unroll
  for (int i = 0; i < kSortItems; i++) t.c[i * kSortThreads + tid] = src[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    const uint32_t p = tid * kSortItems + i;
    if (p < m) s.out[base + p] = t.c[o[i]];
  }
}

// One pass: merges sorted runs [2 r run, ...) of `run` indices in pairs, a
// block per kSortTile outputs.  Does nothing once one run holds them all.
template <int ORDER, typename H>
__global__ void __launch_bounds__(kSortThreads) merge_runs_kernel(SortArgs<H> s, uint32_t run) {
  __shared__ SortTile t;
  __shared__ uint32_t split[2];
  const uint32_t n = s.count(), base = blockIdx.x * kSortTile;
  if (run >= n || base >= n) return;
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t pair = base / (2 * run) * (2 * run);
  const uint32_t na = min(run, n - pair), nb = min(run, n - pair - na);
  const uint32_t *A = s.idx + pair, *B = A + na;
  const uint32_t d0 = base - pair, d1 = min(d0 + kSortTile, na + nb);
  if (tid < 64) {
    // warps 0 and 1 find the block's two splits, 32 probes at a time
    const uint32_t diag = tid < 32 ? d0 : d1;
    uint32_t lo = diag > nb ? diag - nb : 0u, hi = min(diag, na);  // the answer lies in [lo, hi]
    while (lo < hi) {
      const uint32_t step = (hi - lo + 31) / 32, mid = lo + lane * step;
      bool b_first = true;  // B[diag - 1 - mid] before A[mid]: the answer is at most mid
      if (mid < hi)
        b_first = key_less(s.template key<ORDER>(B[diag - 1 - mid]), s.template key<ORDER>(A[mid]));
      const uint32_t yes = __ballot_sync(0xffffffffu, b_first);
      const uint32_t k = yes ? (uint32_t)(__ffs((int)yes) - 1) : 32u;  // the first probe at or past the answer
      const uint32_t new_hi = k < 32 ? min(hi, lo + k * step) : hi;
      if (k) lo = min(lo + (k - 1) * step + 1, new_hi);
      hi = new_hi;
    }
    if (lane == 0) split[tid >> 5] = lo;
  }
  __syncthreads();
  const uint32_t a0 = split[0], a1 = split[1], b0 = d0 - a0, b1 = d1 - a1;
  const uint32_t ma = a1 - a0, mb = b1 - b0, m = ma + mb;
  uint32_t src[kSortItems];
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    const uint32_t p = i * kSortThreads + tid;
    src[i] = p < ma ? A[a0 + p] : p < m ? B[b0 + p - ma] : 0u;
  }
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    const uint32_t p = i * kSortThreads + tid;
    if (p < m) t.put(p, s.template key<ORDER>(src[i]));
  }
  __syncthreads();
  uint32_t o[kSortItems];
  const uint32_t at = min(tid * kSortItems, m);
  uint32_t x = merge_split(at, ma, mb, [&](uint32_t i, uint32_t j) { return t.less(ma + j, i); });
  uint32_t y = at - x;
#pragma unroll
  for (int i = 0; i < kSortItems; i++) {
    o[i] = 0;
    if (at + i < m) {
      const bool b = x >= ma || (y < mb && t.less(ma + y, x));
      o[i] = b ? ma + y++ : x++;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSortItems; i++) t.c[i * kSortThreads + tid] = src[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kSortItems; i++)
    if (at + i < m) s.out[base + at + i] = t.c[o[i]];
}

// Merge passes that sort n records, and whether the result ends in the second
// of the two buffers the passes alternate between.
__host__ __device__ inline int merge_passes(uint32_t n) {
  int p = 0;
  for (unsigned long long run = kSortTile; run < n; run *= 2) p++;
  return p;
}

// Sorts the indices src.idx (null: 0, 1, ...) into *a, or into *b after an odd
// number of passes.  With a device count the launches are those of src.n, the
// largest it can be, and the buffer follows from the count (merge_passes).
// Returns the launches.
template <int ORDER, typename H>
inline int sort_indices(SortArgs<H> s, uint32_t *a, uint32_t *b, cudaStream_t st) {
  const unsigned blocks = (s.n + kSortTile - 1) / kSortTile;
  s.out = a;
  sort_tiles_kernel<ORDER, H><<<blocks, kSortThreads, 0, st>>>(s);
  const int passes = merge_passes(s.n);
  uint32_t run = kSortTile;
  for (int p = 0; p < passes; p++, run *= 2) {
    s.idx = a;
    s.out = b;
    merge_runs_kernel<ORDER, H><<<blocks, kSortThreads, 0, st>>>(s, run);
    uint32_t *x = a;
    a = b;
    b = x;
  }
  return 1 + passes;
}

// The records (sorted by diagonal) that are kept: their indices to kept, in
// any order, their number to *n_kept (zeroed by the caller).
template <typename H>
__global__ void __launch_bounds__(256) keep_kernel(SortArgs<H> s, uint32_t *__restrict__ kept, uint32_t *n_kept) {
  const uint32_t n = s.count(), stride = gridDim.x * blockDim.x;
  for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += stride) {
    const uint32_t i = i0 + threadIdx.x;
    bool k = false;
    uint32_t r = 0;
    if (i < n) {
      r = s.idx[i];
      k = true;
      if (i > 0) {
        const uint32_t q = s.idx[i - 1];
        k = (s.scope && s.scope[q] != s.scope[r]) || !contained_dev(load_hsp(s.recs + q), load_hsp(s.recs + r));
      }
    }
    const uint32_t b = __ballot_sync(0xffffffffu, k);
    uint32_t at = 0;
    if ((threadIdx.x & 31) == 0 && b) at = atomicAdd(n_kept, (uint32_t)__popc(b));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (k) kept[at + (uint32_t)__popc(b & lanemask_lt())] = r;
  }
}

// The records of a list of indices.
__global__ void gather_scoped_kernel(const SegmentPair *__restrict__ raw, const uint32_t *__restrict__ raw_scope,
                                     const uint32_t *__restrict__ idx, uint32_t n, ScopedHspOut *__restrict__ out) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint32_t r = idx[i];
    out[i] = ScopedHspOut{raw_scope[r], raw[r]};
  }
}

// The kept records in order, from the buffer their sort ended in.
__global__ void emit_scoped_kernel(const SegmentPair *__restrict__ raw, const uint32_t *__restrict__ raw_scope,
                                   const uint32_t *__restrict__ a, const uint32_t *__restrict__ b,
                                   const uint32_t *__restrict__ n_kept, ScopedHspOut *__restrict__ out) {
  const uint32_t n = *n_kept;
  const uint32_t *perm = merge_passes(n) & 1 ? b : a;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint32_t r = perm[i];
    out[i] = ScopedHspOut{raw_scope[r], raw[r]};
  }
}
__global__ void emit_plain_kernel(const PlainHsp *__restrict__ in, const uint32_t *__restrict__ a,
                                  const uint32_t *__restrict__ b, const uint32_t *__restrict__ n_kept,
                                  PlainHsp *__restrict__ out, uint32_t *__restrict__ n_out) {
  const uint32_t n = *n_kept;
  const uint32_t *perm = merge_passes(n) & 1 ? b : a;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = in[perm[i]];
  if (blockIdx.x == 0 && threadIdx.x == 0) *n_out = n;
}

}  // namespace hz
