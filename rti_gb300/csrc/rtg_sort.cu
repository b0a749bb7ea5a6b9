// rtg_sort.cu -- stable LSD radix sort of (uint32 key, uint32 value) pairs and
// exclusive prefix sums, used by the LBVH build (Morton order) and by the
// neighbour lists.  Neither runs inside a trace.
//
// Radix sort: 8-bit digits.  Up to kRsSmall pairs one block runs every pass.
// Longer arrays take one histogram launch for the digits of all passes, then
// one launch a pass: each tile ranks its keys by warp match masks, publishes
// its digit counts and adds up its predecessors' (decoupled look-back, Merrill
// and Garland 2016), so that no pass needs a scan of per-tile tables.  Bound by
// the latency of few small launches: the 98 k Morton keys of a trench took 12
// launches and 0.16 ms of a histogram, a scan and a scatter a pass in tiles of
// 4096 (25 blocks for 152 SMs); now 5 launches and tiles of 1024.
#include <cstdint>

#include "rtg_internal.cuh"

namespace rtg {

namespace {

constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsMaxPasses = 4;
// Tiles of 1024 up to 2^18 pairs (every SM has one), of 4096 beyond (fewer
// tiles to look back over).
constexpr int kRsItemsShort = 4, kRsItemsLong = 16;
constexpr int64_t kRsShort = (int64_t)1 << 18;
constexpr int kRsSmallThreads = 1024;
constexpr int kRsSmallItems = 4;
constexpr int64_t kRsSmall = (int64_t)kRsSmallThreads * kRsSmallItems;
// look-back words: the count in the low 30 bits, the state above
constexpr uint32_t kRsCount = 1u << 30, kRsPrefix = 2u << 30, kRsValue = (1u << 30) - 1u;
constexpr uint32_t kRsSpins = 1u << 22;  // look-back reads of one word before the tile gives up

// Digit counts of every pass: hist[pass][digit].
__global__ void __launch_bounds__(kRsThreads) rs_hist(const uint32_t* __restrict__ keys, int64_t n, int passes,
                                                       uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[kRsMaxPasses][256];
  const int tid = threadIdx.x;
  for (int p = 0; p < passes; ++p) h[p][tid] = 0;
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * kRsThreads + tid; i < n; i += (int64_t)gridDim.x * kRsThreads) {
    const uint32_t k = keys[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p)
    if (h[p][tid]) atomicAdd(&hist[256 * p + tid], h[p][tid]);
}

// Exclusive scan of one value per thread over the first 256 threads of the
// block (all threads call it; warp_sums holds 8 words).
__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t* warp_sums) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31 && warp < 8) warp_sums[warp] = x;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp && w < 8; ++w) before += warp_sums[w];
  __syncthreads();
  return before + x - v;
}

// One pass over one tile.  Tiles are numbered in the order in which their
// blocks start, so a tile only waits for tiles that already run.
template <int ITEMS>
__global__ void __launch_bounds__(kRsThreads) rs_pass(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                       uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                       int64_t n, int shift, const uint32_t* __restrict__ hist,
                                                       uint32_t* __restrict__ next_tile, volatile uint32_t* look,
                                                       unsigned long long* __restrict__ errors) {
  __shared__ uint32_t wcnt[kRsWarps][256];
  __shared__ uint32_t offs[256];
  __shared__ uint32_t warp_sums[8];
  __shared__ uint32_t s_tile, s_bad;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s_tile = atomicAdd(next_tile, 1u);
    s_bad = 0u;
  }
  for (int w = 0; w < kRsWarps; ++w) wcnt[w][tid] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const int64_t base = (int64_t)tile * (kRsThreads * ITEMS) + (int64_t)warp * (32 * ITEMS);
  const unsigned lt_mask = (1u << lane) - 1u;
  uint32_t key[ITEMS], rank[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int64_t i = base + r * 32 + lane;
    const bool valid = i < n;
    key[r] = valid ? kin[i] : 0u;
    const uint32_t d = valid ? ((key[r] >> shift) & 255u) : 256u;
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
    const uint32_t before = valid ? wcnt[warp][d] : 0u;
    rank[r] = before + (uint32_t)__popc(peers & lt_mask);
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = before + (uint32_t)__popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // digit tid: its count in this tile, and the warps' offsets within it
  uint32_t count = 0;
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) {
    const uint32_t c = wcnt[w][tid];
    wcnt[w][tid] = count;
    count += c;
  }
  volatile uint32_t* mine = look + (int64_t)tile * 256 + tid;
  *mine = count | (tile == 0 ? kRsPrefix : kRsCount);
  // eight predecessors at a time: their words come in one latency
  uint32_t before = 0;
  bool found = false;
  for (int64_t t = (int64_t)tile - 1; t >= 0 && !found; t -= 8) {
    uint32_t v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k] = kRsPrefix;  // before the first tile
      if (t - k >= 0) v[k] = look[(t - k) * 256 + tid];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (found) continue;
      for (uint32_t spin = 0; v[k] < kRsCount && spin < kRsSpins; ++spin) v[k] = look[(t - k) * 256 + tid];
      if (v[k] < kRsCount) s_bad = 1u;  // gave up: the sort fails as a whole
      before += v[k] & kRsValue;
      found = v[k] < kRsCount || v[k] >= kRsPrefix;
    }
  }
  if (tile != 0) *mine = ((before + count) & kRsValue) | kRsPrefix;
  const uint32_t start = scan256(hist[tid], warp_sums);
  offs[tid] = start + before;
  __syncthreads();
  if (s_bad) {
    if (tid == 0) atomicAdd(errors, 1ull);
    return;
  }
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int64_t i = base + r * 32 + lane;
    if (i >= n) continue;
    const uint32_t d = (key[r] >> shift) & 255u;
    const uint32_t pos = offs[d] + wcnt[warp][d] + rank[r];
    if (pos < (uint64_t)n) {
      kout[pos] = key[r];
      vout[pos] = vin[i];
    }
  }
}

// Every pass of a short array in one block.
__global__ void __launch_bounds__(kRsSmallThreads) rs_small(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1,
                                                             int n, int passes) {
  constexpr int kWarps = kRsSmallThreads / 32;
  __shared__ uint16_t wcnt[kWarps][256];
  __shared__ uint32_t offs[256];
  __shared__ uint32_t warp_sums[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  uint32_t *kin = k0, *vin = v0, *kout = k1, *vout = v1;
  for (int p = 0; p < passes; ++p) {
    const int shift = 8 * p;
    for (int j = lane; j < 256; j += 32) wcnt[warp][j] = 0;
    __syncwarp();
    uint32_t key[kRsSmallItems], val[kRsSmallItems], rank[kRsSmallItems];
#pragma unroll
    for (int r = 0; r < kRsSmallItems; ++r) {
      const int i = warp * (32 * kRsSmallItems) + r * 32 + lane;
      const bool valid = i < n;
      key[r] = valid ? kin[i] : 0u;
      val[r] = valid ? vin[i] : 0u;
      const uint32_t d = valid ? ((key[r] >> shift) & 255u) : 256u;
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
      const uint32_t before = valid ? wcnt[warp][d] : 0u;
      rank[r] = before + (uint32_t)__popc(peers & lt_mask);
      __syncwarp();
      if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = (uint16_t)(before + (uint32_t)__popc(peers));
      __syncwarp();
    }
    __syncthreads();
    uint32_t count = 0;
    if (tid < 256)
      for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = wcnt[w][tid];
        wcnt[w][tid] = (uint16_t)count;
        count += c;
      }
    const uint32_t start = scan256(count, warp_sums);
    if (tid < 256) offs[tid] = start;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRsSmallItems; ++r) {
      const int i = warp * (32 * kRsSmallItems) + r * 32 + lane;
      if (i >= n) continue;
      const uint32_t d = (key[r] >> shift) & 255u;
      const uint32_t pos = offs[d] + wcnt[warp][d] + rank[r];
      kout[pos] = key[r];
      vout[pos] = val[r];
    }
    __syncthreads();  // the outputs are complete before they become the inputs
    uint32_t* t = kin; kin = kout; kout = t;
    t = vin; vin = vout; vout = t;
  }
}

constexpr int kScanThreads = 1024;
constexpr int64_t kScanChunk = (int64_t)kScanThreads * 4;  // items one block scans in one step

// Exclusive scan of items [base, base + kScanChunk) of a, in place, after
// `carry`; returns the chunk's total.  All threads of the block call it.
template <typename T>
__device__ T scan_chunk(T* __restrict__ a, int64_t base, int64_t m, T carry, T* warp_sums) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = blockDim.x >> 5;
  T v[4];
  T s = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t i = base + (int64_t)tid * 4 + q;
    v[q] = i < m ? a[i] : (T)0;
    s += v[q];
  }
  // inclusive warp scan of the thread sums
  T x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nw ? warp_sums[lane] : (T)0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) warp_sums[lane] = w;
  }
  __syncthreads();
  T excl = carry + (warp > 0 ? warp_sums[warp - 1] : (T)0) + (x - s);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t i = base + (int64_t)tid * 4 + q;
    if (i < m) a[i] = excl;
    excl += v[q];
  }
  const T chunk_total = warp_sums[nw - 1];
  __syncthreads();  // warp_sums is reused by the next call
  return chunk_total;
}

// Single-block exclusive scan, in place, chunk after chunk.
template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_excl_kernel(T* __restrict__ a, int64_t m, T* total) {
  __shared__ T warp_sums[32];
  T carry = 0;
  for (int64_t base = 0; base < m; base += kScanChunk) carry += scan_chunk(a, base, m, carry, warp_sums);
  if (threadIdx.x == 0 && total) *total = carry;
}

// Multi-block scan, pass 1: the total of every chunk.
template <typename T>
__global__ void __launch_bounds__(kScanThreads) chunk_sum_kernel(const T* __restrict__ a, int64_t m,
                                                                 T* __restrict__ sums) {
  __shared__ T warp_sums[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = (int64_t)blockIdx.x * kScanChunk;
  T s = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t i = base + (int64_t)tid * 4 + q;
    if (i < m) s += a[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
  if (lane == 0) warp_sums[warp] = s;
  __syncthreads();
  if (warp == 0) {
    T w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : (T)0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xFFFFFFFFu, w, o);
    if (lane == 0) sums[blockIdx.x] = w;
  }
}

// Multi-block scan, pass 3: every chunk after its scanned offset (pass 2 is
// scan_excl_kernel over the chunk totals).
template <typename T>
__global__ void __launch_bounds__(kScanThreads) chunk_scan_kernel(T* __restrict__ a, int64_t m,
                                                                  const T* __restrict__ offsets) {
  __shared__ T warp_sums[32];
  scan_chunk(a, (int64_t)blockIdx.x * kScanChunk, m, offsets[blockIdx.x], warp_sums);
}

// Exclusive scan of m items in place (total into *d_total when given): one
// block for short arrays, three passes over chunks of kScanChunk otherwise.
template <typename T>
int exclusive_scan(rtg_context* ctx, T* d_a, int64_t m, T* d_total, cudaStream_t st) {
  if (m <= 0) return RTG_OK;
  if (m <= 4 * kScanChunk) {
    scan_excl_kernel<T><<<1, kScanThreads, 0, st>>>(d_a, m, d_total);
    RTG_CUDA(ctx, cudaGetLastError());
    return RTG_OK;
  }
  const int64_t nc = (m + kScanChunk - 1) / kScanChunk;
  DBuf<T> sums;
  RTG_TRY(talloc(ctx, sums, (size_t)nc, st, "scan chunk totals"));
  chunk_sum_kernel<T><<<(unsigned)nc, kScanThreads, 0, st>>>(d_a, m, sums.p);
  scan_excl_kernel<T><<<1, kScanThreads, 0, st>>>(sums.p, nc, d_total);
  chunk_scan_kernel<T><<<(unsigned)nc, kScanThreads, 0, st>>>(d_a, m, sums.p);
  const cudaError_t e = cudaGetLastError();
  tfree(sums, st);
  if (e != cudaSuccess) return check_cuda(ctx, e, "scan");
  return RTG_OK;
}

}  // namespace

int exclusive_scan_u32(rtg_context* ctx, uint32_t* d_a, int64_t m, uint32_t* d_total, cudaStream_t st) {
  return exclusive_scan<uint32_t>(ctx, d_a, m, d_total, st);
}

int exclusive_scan_i64(rtg_context* ctx, int64_t* d_a, int64_t m, int64_t* d_total, cudaStream_t st) {
  return exclusive_scan<long long>(ctx, (long long*)d_a, m, (long long*)d_total, st);
}

// Sorts (keys, vals) by the low `bits` (at most 32) bits of the keys, stably;
// n < 2^30.  Enqueues and returns: the results are in d_keys/d_vals once the
// stream gets there; d_tmp_keys/d_tmp_vals are scratch of the same length.  A
// sort that failed (a look-back that gave up) is counted in *d_errors and
// leaves positions unwritten.
int radix_sort_pairs(rtg_context* ctx, uint32_t* d_keys, uint32_t* d_vals, uint32_t* d_tmp_keys,
                     uint32_t* d_tmp_vals, int64_t n, int bits, unsigned long long* d_errors, cudaStream_t st) {
  if (n <= 1) return RTG_OK;
  const int passes = (bits + 7) / 8;
  if (n <= kRsSmall) {
    rs_small<<<1, kRsSmallThreads, 0, st>>>(d_keys, d_vals, d_tmp_keys, d_tmp_vals, (int)n, passes);
  } else {
    const bool shrt = n <= kRsShort;
    const int64_t tile = kRsThreads * (shrt ? kRsItemsShort : kRsItemsLong);
    const int64_t tiles = (n + tile - 1) / tile;
    // histograms | tile counters | look-back words, zeroed together
    const size_t head = 256 * kRsMaxPasses + kRsMaxPasses, words = head + (size_t)(256 * tiles * passes);
    DBuf<uint32_t> work;
    RTG_TRY(talloc(ctx, work, words, st, "radix sort"));
    cudaMemsetAsync(work.p, 0, words * sizeof(uint32_t), st);
    const int64_t hb = (n + kRsThreads * 8 - 1) / (kRsThreads * 8);  // at most four blocks for each of 152 SMs
    rs_hist<<<(unsigned)(hb < 608 ? hb : 608), kRsThreads, 0, st>>>(d_keys, n, passes, work.p);
    uint32_t *kin = d_keys, *vin = d_vals, *kout = d_tmp_keys, *vout = d_tmp_vals;
    for (int p = 0; p < passes; ++p) {
      uint32_t* look = work.p + head + (size_t)(256 * tiles * p);
      uint32_t* next = work.p + 256 * kRsMaxPasses + p;
      const uint32_t* hist = work.p + 256 * p;
      if (shrt)
        rs_pass<kRsItemsShort><<<(unsigned)tiles, kRsThreads, 0, st>>>(kin, vin, kout, vout, n, 8 * p, hist, next, look,
                                                                        d_errors);
      else
        rs_pass<kRsItemsLong><<<(unsigned)tiles, kRsThreads, 0, st>>>(kin, vin, kout, vout, n, 8 * p, hist, next, look,
                                                                       d_errors);
      uint32_t* t = kin; kin = kout; kout = t;
      t = vin; vin = vout; vout = t;
    }
    tfree(work, st);
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && (passes & 1)) {
    e = cudaMemcpyAsync(d_keys, d_tmp_keys, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_vals, d_tmp_vals, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
  }
  if (e != cudaSuccess) return check_cuda(ctx, e, "radix sort");
  return RTG_OK;
}

}  // namespace rtg
