// Device-wide scans (reduce-then-scan, three launches, no inter-block waits)
// and a stable LSD radix sort of (u32 key, u32 value) pairs built on them, for
// the on-device seed-table build.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "hz_device.cuh"

namespace hz {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

// Sum of one or two u32 streams.
template <typename T> struct Sum;
template <> struct Sum<uint32_t> {
  __device__ __forceinline__ static uint32_t zero() { return 0u; }
  __device__ __forceinline__ static uint32_t add(uint32_t a, uint32_t b) { return a + b; }
  __device__ __forceinline__ static uint32_t shfl_up(uint32_t v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
};
template <> struct Sum<uint2> {
  __device__ __forceinline__ static uint2 zero() { return make_uint2(0u, 0u); }
  __device__ __forceinline__ static uint2 add(uint2 a, uint2 b) { return make_uint2(a.x + b.x, a.y + b.y); }
  __device__ __forceinline__ static uint2 shfl_up(uint2 v, int d) {
    return make_uint2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
  }
};

// A 64-bit hit count paired with a 32-bit position count.
struct HitNz {
  unsigned long long h;
  uint32_t n;
};
template <> struct Sum<HitNz> {
  __device__ __forceinline__ static HitNz zero() { return HitNz{0ull, 0u}; }
  __device__ __forceinline__ static HitNz add(HitNz a, HitNz b) { return HitNz{a.h + b.h, a.n + b.n}; }
  __device__ __forceinline__ static HitNz shfl_up(HitNz v, int d) {
    return HitNz{__shfl_up_sync(0xffffffffu, v.h, d), __shfl_up_sync(0xffffffffu, v.n, d)};
  }
};

// A maximum, for scans that carry the last value seen in ascending data.
struct MaxU32 {
  uint32_t v;
};
template <> struct Sum<MaxU32> {
  __device__ __forceinline__ static MaxU32 zero() { return MaxU32{0u}; }
  __device__ __forceinline__ static MaxU32 add(MaxU32 a, MaxU32 b) { return MaxU32{max(a.v, b.v)}; }
  __device__ __forceinline__ static MaxU32 shfl_up(MaxU32 v, int d) {
    return MaxU32{__shfl_up_sync(0xffffffffu, v.v, d)};
  }
};

// Exclusive block scan of one value per thread; returns the exclusive prefix
// and writes the block total to *total.
template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T *total) {
  __shared__ T warp_tot[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    T up = Sum<T>::shfl_up(incl, d);
    if (lane >= d) incl = Sum<T>::add(incl, up);
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    T w = lane < kScanThreads / 32 ? warp_tot[lane] : Sum<T>::zero();
    T wi = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      T up = Sum<T>::shfl_up(wi, d);
      if (lane >= d) wi = Sum<T>::add(wi, up);
    }
    if (lane < kScanThreads / 32) warp_tot[lane] = wi;  // inclusive warp prefix
  }
  __syncthreads();
  T before = warp == 0 ? Sum<T>::zero() : warp_tot[warp - 1];
  *total = warp_tot[kScanThreads / 32 - 1];
  __syncthreads();
  // exclusive = before + incl - v  (as add of the exclusive lane prefix)
  T lane_excl = Sum<T>::shfl_up(incl, 1);
  if (lane == 0) lane_excl = Sum<T>::zero();
  return Sum<T>::add(before, lane_excl);
}

// Pass 1: per-tile totals.
template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const T *__restrict__ in, uint64_t n,
                                                                   T *__restrict__ partial) {
  uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
  T acc = Sum<T>::zero();
#pragma unroll
  for (int i = 0; i < kScanItems; i++)
    if (base + i < n) acc = Sum<T>::add(acc, in[base + i]);
  T tot;
  block_exclusive_scan<T>(acc, &tot);
  if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

// Pass 2: exclusive scan of the tile totals in one block (any count), total
// into *grand.
template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_partials_kernel(T *partial, uint64_t n, T *grand) {
  T carry = Sum<T>::zero();
  for (uint64_t off = 0; off < n; off += kScanTile) {
    uint64_t base = off + (uint64_t)threadIdx.x * kScanItems;
    T v[kScanItems];
    T acc = Sum<T>::zero();
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
      v[i] = base + i < n ? partial[base + i] : Sum<T>::zero();
      acc = Sum<T>::add(acc, v[i]);
    }
    T tot;
    T ex = Sum<T>::add(carry, block_exclusive_scan<T>(acc, &tot));
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
      if (base + i < n) partial[base + i] = ex;
      ex = Sum<T>::add(ex, v[i]);
    }
    carry = Sum<T>::add(carry, tot);
  }
  if (threadIdx.x == 0 && grand) *grand = carry;
}

// Pass 3: per-tile exclusive or inclusive scan plus the tile offset.
template <typename T, bool INCLUSIVE = false>
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const T *__restrict__ in, uint64_t n,
                                                                  const T *__restrict__ partial,
                                                                  T *__restrict__ out) {
  uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
  T v[kScanItems];
  T acc = Sum<T>::zero();
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    v[i] = base + i < n ? in[base + i] : Sum<T>::zero();
    acc = Sum<T>::add(acc, v[i]);
  }
  T tot;
  T ex = Sum<T>::add(partial[blockIdx.x], block_exclusive_scan<T>(acc, &tot));
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    const T next = Sum<T>::add(ex, v[i]);
    if (base + i < n) out[base + i] = INCLUSIVE ? next : ex;
    ex = next;
  }
}

inline uint64_t scan_tiles(uint64_t n) { return (n + kScanTile - 1) / kScanTile; }

// Exclusive scan of n elements from `in` to `out` (may alias); `partial`
// needs scan_tiles(n) elements; the grand total lands in *grand (device).
template <typename T>
inline void exclusive_scan(const T *in, T *out, uint64_t n, T *partial, T *grand, cudaStream_t s) {
  uint64_t tiles = scan_tiles(n);
  if (n == 0) {
    cudaMemsetAsync(grand, 0, sizeof(T), s);
    return;
  }
  scan_reduce_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, partial);
  scan_partials_kernel<T><<<1, kScanThreads, 0, s>>>(partial, tiles, grand);
  scan_apply_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, partial, out);
}

// Inclusive scan in place.
template <typename T> inline void inclusive_scan(T *data, uint64_t n, T *partial, cudaStream_t s) {
  const uint64_t tiles = scan_tiles(n);
  if (n == 0) return;
  scan_reduce_kernel<T><<<(unsigned)tiles, kScanThreads, 0, s>>>(data, n, partial);
  scan_partials_kernel<T><<<1, kScanThreads, 0, s>>>(partial, tiles, (T *)nullptr);
  scan_apply_kernel<T, true><<<(unsigned)tiles, kScanThreads, 0, s>>>(data, n, partial, data);
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, value) pairs, 8-bit digits.

constexpr int kRadixThreads = 256;
constexpr int kRadixItems = 16;
constexpr int kRadixTile = kRadixThreads * kRadixItems;  // 4096
constexpr int kRadixBins = 256;

// Digit histogram of each tile, stored digit-major: hist[d * tiles + tile].
__global__ void __launch_bounds__(kRadixThreads) radix_hist_kernel(const uint32_t *__restrict__ keys, uint64_t n,
                                                                   int shift, uint32_t *__restrict__ hist,
                                                                   uint64_t tiles) {
  __shared__ uint32_t h[kRadixBins];
  h[threadIdx.x] = 0;
  __syncthreads();
  uint64_t base = (uint64_t)blockIdx.x * kRadixTile;
  for (int i = 0; i < kRadixItems; i++) {
    uint64_t e = base + (uint64_t)i * kRadixThreads + threadIdx.x;
    if (e < n) atomicAdd(&h[(keys[e] >> shift) & 0xFF], 1u);
  }
  __syncthreads();
  hist[(uint64_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of a tile, in element order: a warp takes 512 consecutive
// elements, 32 at a time.  An element's rank among its digit is the warp's
// count so far plus its earlier peers in the round; the warps' counts and the
// digits' totals are scanned once per tile, the tile is put in order in shared
// memory, and its runs (16 elements of a digit on average) go out side by
// side.  FIRST: the keys are the k-mers of all strided positions, invalid ones
// (kInvalidKmer) left out, and an element's value is its position.  16 M
// pairs: 0.31 ms a pass with a block-wide round of ranks per 256 elements and
// a scattered store each, 0.17 here.
template <bool FIRST>
__global__ void __launch_bounds__(kRadixThreads) radix_scatter_kernel(
    const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals, uint64_t n, int shift,
    const uint32_t *__restrict__ offsets, uint64_t tiles, uint32_t *__restrict__ keys_out,
    uint32_t *__restrict__ vals_out, uint64_t start, uint32_t step) {
  constexpr int W = kRadixThreads / 32;
  __shared__ uint32_t cnt[W][kRadixBins];  // per warp: the digit's count so far, then what earlier warps hold
  __shared__ uint32_t first[kRadixBins];   // the digit's first place in the ordered tile
  __shared__ uint32_t goff[kRadixBins];    // its place in the output less that
  __shared__ uint32_t warp_tot[W];
  __shared__ uint32_t sk[kRadixTile], sv[kRadixTile];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int w = 0; w < W; w++) cnt[w][threadIdx.x] = 0;
  const uint64_t base = (uint64_t)blockIdx.x * kRadixTile + warp * (kRadixTile / W);
  uint32_t k[kRadixItems], v[kRadixItems], rank[kRadixItems];
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const uint64_t e = base + (uint32_t)i * 32 + lane;
    k[i] = e < n ? keys[e] : kInvalidKmer;
    v[i] = FIRST ? (uint32_t)(start + e * step) : e < n ? vals[e] : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const uint64_t e = base + (uint32_t)i * 32 + lane;
    const bool ok = e < n && (!FIRST || k[i] != kInvalidKmer);
    const uint32_t d = ok ? (k[i] >> shift) & 0xFFu : 0x100u;  // left-out lanes form their own group
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    rank[i] = ok ? cnt[warp][d] + __popc(peers & lanemask_lt()) : 0xFFFFFFFFu;
    __syncwarp();
    if (ok && (peers & lanemask_lt()) == 0) cnt[warp][d] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  uint32_t total = 0;
#pragma unroll
  for (int w = 0; w < W; w++) {
    const uint32_t c = cnt[w][threadIdx.x];
    cnt[w][threadIdx.x] = total;
    total += c;
  }
  uint32_t incl = total;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= (uint32_t)d) incl += up;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  uint32_t before = incl - total, all = 0;
#pragma unroll
  for (int w = 0; w < W; w++) {
    if ((uint32_t)w < warp) before += warp_tot[w];
    all += warp_tot[w];
  }
  first[threadIdx.x] = before;
  goff[threadIdx.x] = offsets[(uint64_t)threadIdx.x * tiles + blockIdx.x] - before;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRadixItems; i++)
    if (rank[i] != 0xFFFFFFFFu) {
      const uint32_t d = (k[i] >> shift) & 0xFFu, at = first[d] + cnt[warp][d] + rank[i];
      sk[at] = k[i];
      sv[at] = v[i];
    }
  __syncthreads();
  for (uint32_t p = threadIdx.x; p < all; p += kRadixThreads) {
    const uint32_t key = sk[p], dst = goff[(key >> shift) & 0xFFu] + p;
    keys_out[dst] = key;
    vals_out[dst] = sv[p];
  }
}

}  // namespace hz
