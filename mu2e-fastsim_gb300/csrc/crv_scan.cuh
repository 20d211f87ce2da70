// Device-wide exclusive prefix sums over values that a source computes and places: one launch (a tile of items), two
// (block sums; prefixes) or three (with a scan of the block sums between them).
//
// A source S has a value type V (long long, or Two for two sums in one pass), item(i), the value of item i, and
// put(i, v, before), which takes item i's value and the sum of the values before it.  Flags (S::FLAG) have values 0
// and 1 only.  So what a caller does around a prefix sum (finding the heads of runs, filling the rows they start) is
// done in the sum's own passes, and neither the values nor the prefixes cross memory unless a later kernel reads them.
// What has to happen to the sum itself (a check against a capacity, a count passed on) is the end of the last pass.
//
// Bound by the reads of the source where n is large and by launches where it is small.  With kernels of their own around
// a three-launch sum of stored int32 values, the sums and what surrounds them took 85 of the 122 kernel and fill nodes of
// a chain graph; now 25 of 50.  All kernels of a chain: 665 -> 538 us at 16 events, 78.6 -> 75.1 ms at 65,536 (runs of
// equal labels in 265 million charges: 3.4 -> 1.04 ms, 4.2 GB of labels read twice at 4.1 TB/s).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "crv_launch.h"

namespace crv {

constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;                        // items per thread of a tile
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
// Between one tile and this many items a thread takes one item: eight in a row leave most SMs without a block, and a
// source whose put loads through an index does so eight times in a row (16 events, 43,000 rows of room: placing the
// waveforms 11.2 -> 4.3 us, the hits 10.4 -> 3.9 us).
constexpr long long SCAN_SINGLES = 512 * 304;
constexpr int SCAN_WARPS = SCAN_THREADS / 32;
// Up to this many tiles every block adds up the sums of the tiles before it by itself (at most 4 loads per thread);
// beyond, where that would read more than the items themselves, one block scans them in a launch of its own.
constexpr long long SCAN_SELF_TILES = 2048;

// effective length: the host bound n, or the device count *n_dev when it is smaller (arrays sized by an upper bound)
__device__ __forceinline__ long long scan_len(long long n, const long long* n_dev) { return bounded_count(n, n_dev); }

// two sums in one pass
struct Two {
  long long a, b;
};
__device__ __forceinline__ Two operator+(const Two& x, const Two& y) { return {x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ Two operator-(const Two& x, const Two& y) { return {x.a - y.a, x.b - y.b}; }
__device__ __forceinline__ long long scan_up(long long v, int o) { return __shfl_up_sync(0xffffffffu, v, o); }
__device__ __forceinline__ Two scan_up(const Two& v, int o) { return {scan_up(v.a, o), scan_up(v.b, o)}; }
__device__ __forceinline__ long long scan_from(long long v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ Two scan_from(const Two& v, int l) { return {scan_from(v.a, l), scan_from(v.b, l)}; }
__device__ __forceinline__ long long part_of(const Two& v, int k) { return k ? v.b : v.a; }
__device__ __forceinline__ long long part_of(long long v, int) { return v; }

// inclusive sums over the lanes
template <typename V>
__device__ __forceinline__ V scan_lanes(V x) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V y = scan_up(x, o);
    if (int(threadIdx.x & 31) >= o) x = x + y;
  }
  return x;
}

// sum over the block, in every thread (red: SCAN_WARPS values, free on return)
template <typename V>
__device__ __forceinline__ V scan_block_sum(V x, V* red) {
  x = scan_lanes(x);
  if ((threadIdx.x & 31) == 31) red[threadIdx.x >> 5] = x;
  __syncthreads();
  V s{};
#pragma unroll
  for (int w = 0; w < SCAN_WARPS; ++w) s = s + red[w];
  __syncthreads();
  return s;
}

// off: plus the sums of the warps before warp w; returns it plus those of all warps
template <typename V>
__device__ __forceinline__ V scan_of_warps(const V* red, int w, V& off) {
  V sum = off;
#pragma unroll
  for (int q = 0; q < SCAN_WARPS; ++q) {
    if (q < w) off = off + red[q];
    sum = sum + red[q];
  }
  return sum;
}

// what is done with a sum once it is known, by one thread
struct ScanEnd {
  long long* total = nullptr;          // the sum; copy (may be null): a second place for it
  long long* copy = nullptr;
  Status* status = nullptr;            // set: a sum above cap raises CRV_ST_CAPACITY and need[slot]
  int slot = 0;
  long long cap = 0;
  long long* pass = nullptr;           // set: *pass = the sum (pass_n set: *pass_n), or 0 when the sum is above pass_cap
  const long long* pass_n = nullptr;
  long long pass_cap = 0;
  int* clear = nullptr;                // set: nclear counts from here are zeroed
  int nclear = 1;

  ScanEnd& check(Status* s, int need_slot, long long most) {
    status = s;
    slot = need_slot;
    cap = most;
    return *this;
  }
  ScanEnd& guard(long long* to, long long most, const long long* n = nullptr) {
    pass = to;
    pass_cap = most;
    pass_n = n;
    return *this;
  }
  __device__ __forceinline__ void operator()(long long sum) const {
    *total = sum;
    if (copy) *copy = sum;
    if (status && sum > cap) {
      set_flag(status, CRV_ST_CAPACITY);
      need_at_least(status, slot, sum);
    }
    if (clear)
      for (int k = 0; k < nclear; ++k) clear[k] = 0;
    if (pass) *pass = sum <= pass_cap ? (pass_n ? *pass_n : sum) : 0;
  }
};
inline ScanEnd scan_end(long long* total, void* copy = nullptr) {
  ScanEnd e;
  e.total = total;
  e.copy = reinterpret_cast<long long*>(copy);
  return e;
}
struct ScanEnds {
  ScanEnd e[2];
};

// sums of the tiles
template <typename S, int ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_sums(const __grid_constant__ S src, long long n,
                                                          const long long* __restrict__ n_dev,
                                                          typename S::V* __restrict__ part) {
  using V = typename S::V;
  __shared__ V red[SCAN_WARPS];
  n = scan_len(n, n_dev);
  for (long long tile = blockIdx.x; tile * (SCAN_THREADS * ITEMS) < n; tile += gridDim.x) {
    V s{};
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const long long i = tile * (SCAN_THREADS * ITEMS) + (long long)j * SCAN_THREADS + threadIdx.x;
      if (i < n) s = s + src.item(i);
    }
    s = scan_block_sum(s, red);
    if (threadIdx.x == 0) part[tile] = s;
  }
}

// exclusive scan, in place by one block, of the sums of the tiles that hold items
template <typename V>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_parts(V* __restrict__ part, long long n,
                                                           const long long* __restrict__ n_dev) {
  __shared__ V red[SCAN_WARPS];
  n = scan_len(n, n_dev);
  const long long nt = (n + SCAN_TILE - 1) / SCAN_TILE;
  V carry{};
  for (long long base = 0; base < nt; base += SCAN_TILE) {
    V v[SCAN_ITEMS], s{};
    const long long i0 = base + (long long)threadIdx.x * SCAN_ITEMS;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
      v[j] = i0 + j < nt ? part[i0 + j] : V{};
      s = s + v[j];
    }
    const V x = scan_lanes(s);
    if ((threadIdx.x & 31) == 31) red[threadIdx.x >> 5] = x;
    __syncthreads();
    V run = carry + (x - s);
#pragma unroll
    for (int w = 0; w < SCAN_WARPS; ++w) {
      if (w < int(threadIdx.x >> 5)) run = run + red[w];
      carry = carry + red[w];
    }
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
      if (i0 + j < nt) part[i0 + j] = run;
      run = run + v[j];
    }
    __syncthreads();
  }
}

// Prefixes of a tile: each warp takes ITEMS rows of 32 consecutive items (coalesced, all in flight at once), a lane
// one item of each row; a row's prefixes are shuffles, a flag row's one ballot.  scanned: part holds the sums of the
// tiles before each tile; else each block adds them up (no launch and no order between the blocks is needed for it).
template <typename S, int ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_put(const __grid_constant__ S src, long long n,
                                                         const long long* __restrict__ n_dev,
                                                         const typename S::V* __restrict__ part, int scanned,
                                                         const __grid_constant__ ScanEnds end) {
  using V = typename S::V;
  __shared__ V red[SCAN_WARPS];
  n = scan_len(n, n_dev);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // (tile 0 also when it holds no item: the end is still to be done)
  for (long long tile = blockIdx.x; tile * (SCAN_THREADS * ITEMS) < n || tile == 0; tile += gridDim.x) {
    const bool last = (tile + 1) * (SCAN_THREADS * ITEMS) >= n;
    V off{};
    if (scanned) {
      if (n > 0) off = part[tile];
    } else if (tile > 0) {
      for (int t = threadIdx.x; t < int(tile); t += SCAN_THREADS) off = off + part[t];
      off = scan_block_sum(off, red);
    }
    const long long i0 = tile * (SCAN_THREADS * ITEMS) + (long long)w * (32 * ITEMS) + lane;
    if constexpr (S::FLAG) {
      unsigned m[ITEMS];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        m[j] = __ballot_sync(0xffffffffu, i0 + 32 * j < n && src.item(i0 + 32 * j) != 0);
        cnt += __popc(m[j]);
      }
      if (lane == 0) red[w] = cnt;
      __syncthreads();
      const V sum = scan_of_warps(red, w, off);
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if ((m[j] >> lane) & 1u) src.put(i0 + 32 * j, 1, off + __popc(m[j] & ((1u << lane) - 1u)));
        off = off + __popc(m[j]);
      }
      if (last && threadIdx.x == 0) end.e[0](sum);
    } else {
      V x[ITEMS], e[ITEMS], run{};
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) x[j] = i0 + 32 * j < n ? src.item(i0 + 32 * j) : V{};
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const V s = scan_lanes(x[j]);
        e[j] = run + (s - x[j]);
        run = run + scan_from(s, 31);
      }
      if (lane == 0) red[w] = run;
      __syncthreads();
      const V sum = scan_of_warps(red, w, off);
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (i0 + 32 * j < n) src.put(i0 + 32 * j, x[j], off + e[j]);
      if (last && threadIdx.x < sizeof(V) / sizeof(long long)) end.e[threadIdx.x](part_of(sum, threadIdx.x));
    }
    __syncthreads();
  }
}

// out[i] = sum of in[j], j < i
template <typename T>
struct Column {
  using V = long long;
  static constexpr bool FLAG = false;
  const T* in;
  long long* out;
  __device__ __forceinline__ long long item(long long i) const { return (long long)in[i]; }
  __device__ __forceinline__ void put(long long i, long long, long long before) const { out[i] = before; }
};
template <typename T>
Column<T> column(const T* in, long long* out) {
  return {in, out};
}
// two columns at once
struct Columns {
  using V = Two;
  static constexpr bool FLAG = false;
  const int32_t *in_a, *in_b;
  long long *out_a, *out_b;
  __device__ __forceinline__ Two item(long long i) const { return {in_a[i], in_b[i]}; }
  __device__ __forceinline__ void put(long long i, const Two&, const Two& before) const {
    out_a[i] = before.a;
    out_b[i] = before.b;
  }
};

inline int scan_items(long long n) { return n > SCAN_TILE && n <= SCAN_SINGLES ? 1 : SCAN_ITEMS; }
inline long long scan_tiles(long long n) {
  const long long t = (long long)SCAN_THREADS * scan_items(n);
  return n > 0 ? (n + t - 1) / t : 1;
}

// Scratch of a sum over up to n items, in 8-byte words.  A sum over fewer items can have more tiles (of one item per
// thread), so beyond SCAN_SINGLES it is at least that many items' tiles: one scratch then serves every sum it is sized above.
inline long long scan_parts_len(long long n) {
  const long long t = scan_tiles(n), most = scan_tiles(SCAN_SINGLES);
  return 2 * (n > SCAN_SINGLES && t < most ? most : t);
}

template <int ITEMS, typename S>
void scan_launch(const S& src, long long n, const long long* n_dev, const ScanEnds& end, typename S::V* part, long long nb,
                 cudaStream_t s) {
  // at most 16 blocks an SM (four at a time), so that a bound far above the count starts few blocks that find nothing
  const long long most = (long long)device_info().sms * 16;
  const unsigned grid = (unsigned)(nb < most ? nb : most);
  if (nb > 1) {
    crv::Mark mark_("k_scan_sums", s);
    k_scan_sums<S, ITEMS><<<grid, SCAN_THREADS, 0, s>>>(src, n, n_dev, part);
  }
  if (nb > SCAN_SELF_TILES) {
    crv::Mark mark_("k_scan_parts", s);
    k_scan_parts<typename S::V><<<1, SCAN_THREADS, 0, s>>>(part, n, n_dev);
  }
  crv::Mark mark_("k_scan_put", s);
  k_scan_put<S, ITEMS><<<grid, SCAN_THREADS, 0, s>>>(src, n, n_dev, part, nb > SCAN_SELF_TILES ? 1 : 0, end);
}

// One sum over the source.  n_dev (may be null): device count of valid items when n is only an upper bound; items
// beyond it are neither read nor placed.  part: scratch of scan_parts_len(n) words.
template <typename S>
cudaError_t exclusive_scan(const S& src, long long n, const long long* n_dev, const ScanEnds& end, long long* part,
                           cudaStream_t s) {
  typename S::V* const p = reinterpret_cast<typename S::V*>(part);
  if (scan_items(n) == 1) scan_launch<1>(src, n, n_dev, end, p, scan_tiles(n), s);
  else scan_launch<SCAN_ITEMS>(src, n, n_dev, end, p, scan_tiles(n), s);
  return cudaGetLastError();
}
template <typename S>
cudaError_t exclusive_scan(const S& src, long long n, const long long* n_dev, const ScanEnd& end, long long* part,
                           cudaStream_t s) {
  return exclusive_scan(src, n, n_dev, ScanEnds{{end, ScanEnd{}}}, part, s);
}

}  // namespace crv
