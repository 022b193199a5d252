// Device radix sort of packed product states, prefix scans, segmented reduction, merge of
// sorted bases and batched binary search.  These replace the Python set/dict/sorted
// bookkeeping of upstream expand_basis (impurityModel/ed/finite.py:1696-1803) and the
// dict accumulation inside applyOp (finite.py:1355-1388).
#include <algorithm>

#include "common.cuh"

namespace edgpu {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// ---------------------------------------------------------------------------------------
// Exclusive scan of int64 (multi-level, reduce-then-scan)
// ---------------------------------------------------------------------------------------

__device__ __forceinline__ int64_t block_exclusive_scan(int64_t v, int64_t* warp_tot, int64_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    int64_t t = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int64_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nw) warp_tot[lane] = t;
  }
  __syncthreads();
  const int64_t before = warp ? warp_tot[warp - 1] : 0;
  total = warp_tot[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const int64_t* in, int64_t n, int64_t* partial) {
  __shared__ int64_t wt[32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n) s += in[base + k];
  int64_t total;
  block_exclusive_scan(s, wt, total);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_down_kernel(const int64_t* in, int64_t n, const int64_t* block_off,
                                                                 int64_t* out) {
  __shared__ int64_t wt[32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t v[kScanItems];
  int64_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    s += v[k];
  }
  int64_t total;
  int64_t run = block_exclusive_scan(s, wt, total) + (block_off ? block_off[blockIdx.x] : 0);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) {
    out[n] = (block_off ? block_off[blockIdx.x] : 0) + total;
  }
}

static size_t scan_ws_elems(int64_t n) {
  if (n <= kScanTile) return 0;
  const int64_t nb = (n + kScanTile - 1) / kScanTile;
  return (size_t)(nb + 1) + scan_ws_elems(nb);
}

static int scan_rec(const int64_t* in, int64_t* out, int64_t n, int64_t* ws, cudaStream_t s) {
  const int64_t nb = (n + kScanTile - 1) / kScanTile;
  if (nb <= 1) {
    scan_down_kernel<<<1, kScanThreads, 0, s>>>(in, n, nullptr, out); note_launch();
    return check_launch();
  }
  int64_t* partial = ws;
  int64_t* partial_scan = ws + nb + 1;
  (void)partial_scan;
  scan_reduce_kernel<<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, partial); note_launch();
  // Scan partial sums in place into a temp region after them: reuse a second level.
  int64_t* next_ws = ws + nb + 1;
  // The scan output of the partials needs nb + 1 entries; put it into `partial` itself via
  // a recursive call writing to the level's output buffer located in next level's space.
  int rc = scan_rec(partial, partial, nb, next_ws, s);
  if (rc) return rc;
  scan_down_kernel<<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, partial, out); note_launch();
  return check_launch();
}

// ---------------------------------------------------------------------------------------
// Radix sort (stable LSD, 8-bit digits) of W-word keys with a uint32 payload
// ---------------------------------------------------------------------------------------

constexpr int kSortWarps = 16;
constexpr int kSortThreads = kSortWarps * 32;
constexpr int kSortRounds = 8;
constexpr int kSortTile = kSortThreads * kSortRounds;

template <int W>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const uint64_t* keys, int64_t n, int q, int shift,
                                                                  int64_t* hist, int64_t nblocks) {
  __shared__ int h[256];
  for (int d = threadIdx.x; d < 256; d += blockDim.x) h[d] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
  for (int k = threadIdx.x; k < kSortTile; k += blockDim.x) {
    const int64_t i = base + k;
    if (i < n) {
      const int d = (int)((keys[i * W + q] >> shift) & 0xFF);
      atomicAdd(&h[d], 1);
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[(int64_t)d * nblocks + blockIdx.x] = h[d];
}

template <int W>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(const uint64_t* keys_in, const uint32_t* pay_in,
                                                                     uint64_t* keys_out, uint32_t* pay_out, int64_t n,
                                                                     int q, int shift, const int64_t* offs,
                                                                     int64_t nblocks) {
  __shared__ int cnt[kSortWarps][256];
  __shared__ int64_t gbase[256];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = threadIdx.x; k < kSortWarps * 256; k += blockDim.x) (&cnt[0][0])[k] = 0;
  __syncthreads();
  const int64_t wbase = (int64_t)blockIdx.x * kSortTile + (int64_t)warp * 32 * kSortRounds;
  const unsigned lt = (1u << lane) - 1u;
  for (int r = 0; r < kSortRounds; ++r) {
    const int64_t i = wbase + r * 32 + lane;
    const bool valid = i < n;
    const unsigned vmask = __ballot_sync(FULL, valid);
    if (valid) {
      const int d = (int)((keys_in[i * W + q] >> shift) & 0xFF);
      const unsigned peers = __match_any_sync(vmask, d);
      if (lane == __ffs(peers) - 1) cnt[warp][d] += __popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    const int d = threadIdx.x;
    int run = 0;
    for (int w = 0; w < kSortWarps; ++w) {
      const int t = cnt[w][d];
      cnt[w][d] = run;
      run += t;
    }
    gbase[d] = offs[(int64_t)d * nblocks + blockIdx.x];
  }
  __syncthreads();
  for (int r = 0; r < kSortRounds; ++r) {
    const int64_t i = wbase + r * 32 + lane;
    const bool valid = i < n;
    const unsigned vmask = __ballot_sync(FULL, valid);
    int d = 0;
    unsigned peers = 0;
    int rank = 0;
    if (valid) {
      d = (int)((keys_in[i * W + q] >> shift) & 0xFF);
      peers = __match_any_sync(vmask, d);
      rank = cnt[warp][d] + __popc(peers & lt);
    }
    __syncwarp();
    if (valid) {
      const int64_t dst = gbase[d] + rank;
#pragma unroll
      for (int k = 0; k < W; ++k) keys_out[dst * W + k] = keys_in[i * W + k];
      pay_out[dst] = pay_in[i];
      if (lane == __ffs(peers) - 1) cnt[warp][d] += __popc(peers);
    }
    __syncwarp();
  }
}

template <int W>
__global__ void vary_kernel(const uint64_t* keys, int64_t n, unsigned long long* out) {
  uint64_t acc[W];
  uint64_t k0[W];
#pragma unroll
  for (int q = 0; q < W; ++q) {
    acc[q] = 0;
    k0[q] = keys[q];
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int q = 0; q < W; ++q) acc[q] |= keys[i * W + q] ^ k0[q];
  }
#pragma unroll
  for (int q = 0; q < W; ++q) {
    uint64_t v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicOr(out + q, (unsigned long long)v);
  }
}

template <int W>
__global__ void copy_states_kernel(const uint64_t* src, const uint32_t* psrc, uint64_t* dst, uint32_t* pdst, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int q = 0; q < W; ++q) dst[i * W + q] = src[i * W + q];
    pdst[i] = psrc[i];
  }
}

template <int W>
__global__ void heads_kernel(const uint64_t* keys, int64_t n, int64_t* head) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    head[i] = (i == 0) ? 1 : (state_cmp_mm<W>(keys + i * W, keys + (i - 1) * W) != 0 ? 1 : 0);
  }
}

template <int W>
__global__ void segment_reduce_kernel(const uint64_t* keys, const uint32_t* payload, int64_t n,
                                      const int64_t* head_scan, const double2* vals, uint64_t* out_keys,
                                      uint32_t* out_first, double2* out_vals) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t o = head_scan[i];
    if (head_scan[i + 1] == o) continue;  // not a head
#pragma unroll
    for (int q = 0; q < W; ++q) out_keys[o * W + q] = keys[i * W + q];
    if (out_first) out_first[o] = payload[i];
    if (vals && out_vals) {
      double2 acc = vals[payload[i]];
      for (int64_t j = i + 1; j < n && head_scan[j + 1] == head_scan[j]; ++j) {
        const double2 v = vals[payload[j]];
        acc.x = __dadd_rn(acc.x, v.x);
        acc.y = __dadd_rn(acc.y, v.y);
      }
      out_vals[o] = acc;
    }
  }
}

template <int W>
__global__ void merge_kernel(const uint64_t* a, int64_t na, const uint64_t* b, int64_t nb, uint64_t* out) {
  const int64_t tot = na + nb;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (int64_t)gridDim.x * blockDim.x) {
    uint64_t key[W];
    int64_t pos;
    if (t < na) {
      load_state<W>(a + t * W, key);
      pos = t + lower_bound_state<W>(b, nb, key);
    } else {
      const int64_t k = t - na;
      load_state<W>(b + k * W, key);
      pos = k + lower_bound_state<W>(a, na, key);
    }
    store_state<W>(out + pos * W, key);
  }
}

template <int W>
__global__ void lookup_kernel(const uint64_t* basis, int64_t n, const uint64_t* query, int64_t nq, int64_t* out) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nq; t += (int64_t)gridDim.x * blockDim.x) {
    uint64_t key[W];
    load_state<W>(query + t * W, key);
    out[t] = find_state<W>(basis, n, key);
  }
}

inline unsigned grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)grid_cap() * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

}  // namespace edgpu

using namespace edgpu;

extern "C" size_t edgpu_scan_workspace(int64_t n) { return scan_ws_elems(n) * sizeof(int64_t) + 256; }

extern "C" int edgpu_scan_i64(const int64_t* in, int64_t* out, int64_t n, void* workspace, size_t workspace_bytes,
                              void* stream) {
  if (n < 0 || !out) return EDGPU_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    cudaMemsetAsync(out, 0, sizeof(int64_t), s);
    return check_launch();
  }
  if (!in) return EDGPU_ERR_ARG;
  if (workspace_bytes < edgpu_scan_workspace(n)) return EDGPU_ERR_WORKSPACE;
  return scan_rec(in, out, n, reinterpret_cast<int64_t*>(workspace), s);
}

namespace edgpu {

// ---------------------------------------------------------------------------------------
// Small inputs: one CTA sorts (key, original position) pairs in shared memory with a bitonic
// network (a total order, so the result is the stable sort), one launch instead of a
// histogram, scan and scatter launch per varying key byte.
// ---------------------------------------------------------------------------------------
constexpr int kSmallSortThreads = 1024;
constexpr size_t kSmallSortBytes = 160 * 1024;

inline int small_sort_pow2(int64_t n) {
  int p = 1;
  while (p < n) p <<= 1;
  return p;
}

inline bool small_sort_fits(int n_words, int64_t n) {
  return n <= 8192 && (size_t)small_sort_pow2(n) * (8 * (size_t)n_words + 4) <= kSmallSortBytes;
}

inline int small_sort_threads(int N) { return std::min(std::max(N / 2, 32), kSmallSortThreads); }

// The network on N keys in shared memory; POS: ties by position (a stable sort), else equal keys stay as they lie.
template <int W, bool POS>
__device__ __forceinline__ void small_network(uint64_t* k, uint32_t* idx, int N) {
  for (int size = 2; size <= N; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = threadIdx.x; t < (N >> 1); t += blockDim.x) {
        const int lo = 2 * t - (t & (stride - 1));
        const int hi = lo + stride;
        const bool up = (lo & size) == 0;
        int c = 0;
#pragma unroll
        for (int q = 0; q < W; ++q) {
          if (c == 0) {
            const uint64_t a = k[(size_t)lo * W + q], b = k[(size_t)hi * W + q];
            c = a < b ? -1 : (a > b ? 1 : 0);
          }
        }
        if (POS && c == 0) c = idx[lo] < idx[hi] ? -1 : 1;
        if (c != 0 && (c > 0) == up) {
#pragma unroll
          for (int q = 0; q < W; ++q) {
            const uint64_t tmp = k[(size_t)lo * W + q];
            k[(size_t)lo * W + q] = k[(size_t)hi * W + q];
            k[(size_t)hi * W + q] = tmp;
          }
          if (POS) {
            const uint32_t ti = idx[lo];
            idx[lo] = idx[hi];
            idx[hi] = ti;
          }
        }
      }
      __syncthreads();
    }
  }
}

template <int W>
__global__ void __launch_bounds__(kSmallSortThreads) small_sort_kernel(uint64_t* keys, uint32_t* payload, int n, int N) {
  extern __shared__ __align__(16) unsigned char sm[];
  uint64_t* k = reinterpret_cast<uint64_t*>(sm);
  uint32_t* idx = reinterpret_cast<uint32_t*>(k + (size_t)N * W);
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
#pragma unroll
    for (int q = 0; q < W; ++q) k[(size_t)i * W + q] = i < n ? keys[(size_t)i * W + q] : ~0ull;
    idx[i] = (uint32_t)i;  // padding sorts last: all-ones keys, positions >= n
  }
  __syncthreads();
  small_network<W, true>(k, idx, N);
  // payloads follow their keys: read every original payload before any write
  uint32_t pv[(8192 + kSmallSortThreads - 1) / kSmallSortThreads];
  int u = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) pv[u++] = payload[idx[i]];
  __syncthreads();
  u = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
#pragma unroll
    for (int q = 0; q < W; ++q) keys[(size_t)i * W + q] = k[(size_t)i * W + q];
    payload[i] = pv[u++];
  }
}

// The sorted unique keys in one launch: the network, then the segment heads counted a block of keys at a
// time.  As separate steps (copy, positions, sort, heads, two scans, compaction) a layer of a few hundred
// states cost seven launches of two or three microseconds each and their issue: the construction of a
// 360-state sector (three layers) 0.80 -> 0.67 ms.
template <int W>
__global__ void __launch_bounds__(kSmallSortThreads) small_unique_kernel(const uint64_t* __restrict__ keys, int n, int N,
                                                                         uint64_t* __restrict__ out,
                                                                         int64_t* __restrict__ count) {
  extern __shared__ __align__(16) unsigned char sm[];
  uint64_t* k = reinterpret_cast<uint64_t*>(sm);
  __shared__ int heads[kSmallSortThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int i = threadIdx.x; i < N; i += blockDim.x)
#pragma unroll
    for (int q = 0; q < W; ++q) k[(size_t)i * W + q] = i < n ? keys[(size_t)i * W + q] : ~0ull;  // padding sorts last
  __syncthreads();
  small_network<W, false>(k, nullptr, N);
  int base = 0;
  for (int i0 = 0; i0 < n; i0 += blockDim.x) {
    const int i = i0 + threadIdx.x;
    bool head = i < n;
    if (head && i > 0) {
      bool same = true;
#pragma unroll
      for (int q = 0; q < W; ++q) same = same && k[(size_t)i * W + q] == k[(size_t)(i - 1) * W + q];
      head = !same;
    }
    const unsigned b = __ballot_sync(0xffffffffu, head);
    if (lane == 0) heads[warp] = __popc(b);
    __syncthreads();
    int at = base + __popc(b & ((1u << lane) - 1u));
    for (int q = 0; q < warps; ++q) {
      if (q < warp) at += heads[q];
      base += heads[q];
    }
    if (head)
#pragma unroll
      for (int q = 0; q < W; ++q) out[(size_t)at * W + q] = k[(size_t)i * W + q];
    __syncthreads();  // heads is free
  }
  if (threadIdx.x == 0) *count = base;
}

}  // namespace edgpu

extern "C" int edgpu_sort_unique_fits(int n_words, int64_t n) {
  return n_words >= 1 && n_words <= EDGPU_MAX_WORDS && n >= 0 && small_sort_fits(n_words, n);
}

extern "C" int edgpu_sort_unique(int n_words, const uint64_t* keys, int64_t n, uint64_t* out, int64_t* count,
                                 void* stream) {
  if (n < 1 || !keys || !out || !count || !edgpu_sort_unique_fits(n_words, n)) return EDGPU_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int N = std::max(2, small_sort_pow2(n));
  const size_t smem = (size_t)N * 8 * (size_t)n_words;
  EDGPU_DISPATCH_W(n_words, {
    cudaFuncSetAttribute(small_unique_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    small_unique_kernel<W><<<1, small_sort_threads(N), smem, s>>>(keys, (int)n, N, out, count); note_launch();
  });
  return check_launch();
}

extern "C" size_t edgpu_sort_states_workspace(int n_words, int64_t n) {
  const int64_t nb = (n + kSortTile - 1) / kSortTile;
  const int64_t hist = 256 * (nb > 0 ? nb : 1);
  size_t bytes = 0;
  bytes += (size_t)n * n_words * sizeof(uint64_t);  // alternate keys
  bytes += (size_t)n * sizeof(uint32_t);            // alternate payload
  bytes = (bytes + 255) & ~(size_t)255;
  bytes += (size_t)hist * sizeof(int64_t);            // histogram
  bytes += (size_t)(hist + 1) * sizeof(int64_t);      // scanned offsets
  bytes += edgpu_scan_workspace(hist);
  return bytes + 512;
}

extern "C" int edgpu_vary_mask(int n_words, const uint64_t* keys, int64_t n, uint64_t* vary_out, void* stream) {
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS || !vary_out || n < 0) return EDGPU_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  cudaMemsetAsync(vary_out, 0, sizeof(uint64_t) * n_words, s);
  if (n == 0) return check_launch();
  EDGPU_DISPATCH_W(n_words, {
    vary_kernel<W><<<grid_for(n, 256), 256, 0, s>>>(keys, n, reinterpret_cast<unsigned long long*>(vary_out)); note_launch();
  });
  return check_launch();
}

extern "C" int edgpu_sort_states(int n_words, uint64_t* keys, uint32_t* payload, int64_t n, const uint64_t* vary_mask,
                                 void* workspace, size_t workspace_bytes, void* stream) {
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS || n < 0) return EDGPU_ERR_ARG;
  if (n <= 1) return EDGPU_OK;
  if (!keys || !payload) return EDGPU_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (small_sort_fits(n_words, n)) {
    const int N = small_sort_pow2(n);
    const size_t smem = (size_t)N * (8 * (size_t)n_words + 4);
    EDGPU_DISPATCH_W(n_words, {
      cudaFuncSetAttribute(small_sort_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      small_sort_kernel<W><<<1, small_sort_threads(N), smem, s>>>(keys, payload, (int)n, N); note_launch();
    });
    return check_launch();
  }
  if (workspace_bytes < edgpu_sort_states_workspace(n_words, n)) return EDGPU_ERR_WORKSPACE;
  const int64_t nb = (n + kSortTile - 1) / kSortTile;
  const int64_t hist_n = 256 * nb;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  size_t off = 0;
  uint64_t* keys_alt = reinterpret_cast<uint64_t*>(ws + off);
  off += (size_t)n * n_words * sizeof(uint64_t);
  uint32_t* pay_alt = reinterpret_cast<uint32_t*>(ws + off);
  off += (size_t)n * sizeof(uint32_t);
  off = (off + 255) & ~(size_t)255;
  int64_t* hist = reinterpret_cast<int64_t*>(ws + off);
  off += (size_t)hist_n * sizeof(int64_t);
  int64_t* offs = reinterpret_cast<int64_t*>(ws + off);
  off += (size_t)(hist_n + 1) * sizeof(int64_t);
  void* scan_ws = ws + off;
  const size_t scan_bytes = workspace_bytes - off;

  uint64_t* kin = keys;
  uint32_t* pin = payload;
  uint64_t* kout = keys_alt;
  uint32_t* pout = pay_alt;
  int rc = EDGPU_OK;
  for (int q = n_words - 1; q >= 0; --q) {
    for (int byte = 0; byte < 8; ++byte) {
      const int shift = 8 * byte;
      if (vary_mask && ((vary_mask[q] >> shift) & 0xFFull) == 0) continue;
      EDGPU_DISPATCH_W(n_words, {
        radix_hist_kernel<W><<<(unsigned)nb, kSortThreads, 0, s>>>(kin, n, q, shift, hist, nb); note_launch();
      });
      if ((rc = check_launch())) return rc;
      if ((rc = edgpu_scan_i64(hist, offs, hist_n, scan_ws, scan_bytes, stream))) return rc;
      EDGPU_DISPATCH_W(n_words, {
        radix_scatter_kernel<W><<<(unsigned)nb, kSortThreads, 0, s>>>(kin, pin, kout, pout, n, q, shift, offs, nb); note_launch();
      });
      if ((rc = check_launch())) return rc;
      uint64_t* tk = kin;
      kin = kout;
      kout = tk;
      uint32_t* tp = pin;
      pin = pout;
      pout = tp;
    }
  }
  if (kin != keys) {
    EDGPU_DISPATCH_W(n_words, { copy_states_kernel<W><<<grid_for(n, 256), 256, 0, s>>>(kin, pin, keys, payload, n); note_launch(); });
    rc = check_launch();
  }
  return rc;
}

extern "C" int edgpu_segment_heads(int n_words, const uint64_t* keys, int64_t n, int64_t* head, void* stream) {
  if (n < 0 || (n > 0 && (!keys || !head))) return EDGPU_ERR_ARG;
  if (n == 0) return EDGPU_OK;
  EDGPU_DISPATCH_W(n_words, { heads_kernel<W><<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(keys, n, head); note_launch(); });
  return check_launch();
}

extern "C" int edgpu_segment_reduce(int n_words, const uint64_t* keys, const uint32_t* payload, int64_t n,
                                    const int64_t* head_scan, const double* vals, uint64_t* out_keys,
                                    uint32_t* out_first, double* out_vals, void* stream) {
  if (n < 0 || (n > 0 && (!keys || !payload || !head_scan || !out_keys))) return EDGPU_ERR_ARG;
  if (n == 0) return EDGPU_OK;
  EDGPU_DISPATCH_W(n_words, {
    segment_reduce_kernel<W><<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
        keys, payload, n, head_scan, reinterpret_cast<const double2*>(vals), out_keys, out_first,
        reinterpret_cast<double2*>(out_vals)); note_launch();
  });
  return check_launch();
}

extern "C" int edgpu_merge_states(int n_words, const uint64_t* a, int64_t na, const uint64_t* b, int64_t nb,
                                  uint64_t* out, void* stream) {
  if (na < 0 || nb < 0 || !out) return EDGPU_ERR_ARG;
  if (na + nb == 0) return EDGPU_OK;
  EDGPU_DISPATCH_W(n_words, {
    merge_kernel<W><<<grid_for(na + nb, 256), 256, 0, (cudaStream_t)stream>>>(a, na, b, nb, out); note_launch();
  });
  return check_launch();
}

extern "C" int edgpu_lookup_states(int n_words, const uint64_t* basis, int64_t n_basis, const uint64_t* query,
                                   int64_t nq, int64_t* out_index, void* stream) {
  if (nq < 0 || n_basis < 0 || (nq > 0 && (!query || !out_index))) return EDGPU_ERR_ARG;
  if (nq == 0) return EDGPU_OK;
  EDGPU_DISPATCH_W(n_words, {
    lookup_kernel<W><<<grid_for(nq, 256), 256, 0, (cudaStream_t)stream>>>(basis, n_basis, query, nq, out_index); note_launch();
  });
  return check_launch();
}

namespace edgpu {

// ---------------------------------------------------------------------------------------
// Large inputs of nearly full or nearly empty states (edgpu_sort_states_packed).
//
// The states of a sector differ in a few orbitals out of hundreds, spread over every byte: 316
// spin-orbitals took 40 radix passes of 44 bytes a key (1.3 ms for 438 000 states).  Where every
// state has at most a few zeros (or ones) among the bits that vary at all, their positions,
// ascending, are the state: at the first bit in which two states differ one of them has its next
// zero there and the other one a later zero or none, so comparing the position lists (none = the
// largest) compares the states; for ones the order of the positions is turned round.  Three
// positions of 9 bits are four passes of 12 bytes, and one gather of the states at the end
// (0.12 ms there).
// ---------------------------------------------------------------------------------------

// out: [0, W) bits that vary, [W] smallest and [W + 1] largest number of ones, [W + 2, 2 W + 2) the
// first state.
template <int W>
__global__ void stats_kernel(const uint64_t* keys, int64_t n, unsigned long long* out) {
  uint64_t acc[W], k0[W];
  unsigned lo = 64 * W, hi = 0;
#pragma unroll
  for (int q = 0; q < W; ++q) {
    acc[q] = 0;
    k0[q] = keys[q];
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    unsigned c = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) {
      const uint64_t k = keys[i * W + q];
      acc[q] |= k ^ k0[q];
      c += __popcll(k);
    }
    lo = c < lo ? c : lo;
    hi = c > hi ? c : hi;
  }
  __shared__ unsigned long long sv[W];
  __shared__ unsigned slo, shi;
  if (threadIdx.x < W) sv[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    slo = 64 * W;
    shi = 0;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < W; ++q) {
    uint64_t v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicOr(&sv[q], (unsigned long long)v);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&slo, lo);
    atomicMax(&shi, hi);
  }
  __syncthreads();
  if (threadIdx.x < W && sv[threadIdx.x]) atomicOr(out + threadIdx.x, sv[threadIdx.x]);
  if (threadIdx.x == 0) {
    atomicMin(out + W, (unsigned long long)slo);
    atomicMax(out + W + 1, (unsigned long long)shi);
  }
  if (blockIdx.x == 0 && threadIdx.x < W) out[W + 2 + threadIdx.x] = keys[threadIdx.x];
}

struct VaryMask {
  uint64_t w[EDGPU_MAX_WORDS];
};

// The positions of the varying zeros (ones) as one key of `count` fields of `bits` bits.
template <int W>
__global__ void pack_kernel(const uint64_t* keys, int64_t n, VaryMask vary, int ones, int bits, int count,
                            uint64_t* packed, uint32_t* idx) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t none = (1ull << bits) - 1;
    uint64_t key = 0;
    int used = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) {
      const uint64_t k = keys[i * W + q];
      uint64_t z = (ones ? k : ~k) & vary.w[q];
      while (z && used < count) {
        const int p = __clzll(z);
        z &= ~(1ull << (63 - p));
        const uint64_t pos = (uint64_t)(64 * q + p);
        key = (key << bits) | (ones ? none - pos : pos);
        ++used;
      }
    }
    for (; used < count; ++used) key = (key << bits) | (ones ? 0ull : none);
    packed[i] = key;
    idx[i] = (uint32_t)i;
  }
}

template <int W>
__global__ void gather_states_kernel(const uint64_t* src, const uint32_t* psrc, const uint32_t* idx, uint64_t* dst,
                                     uint32_t* pdst, int64_t n) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n * W; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / W;
    const int q = (int)(t - i * W);
    const uint32_t from = idx[i];
    dst[t] = src[(int64_t)from * W + q];
    if (q == 0) pdst[i] = psrc[from];
  }
}

// How states with these statistics are packed: fields of `bits` bits, `count` of them (0: not at all).
struct Packing {
  int ones, bits, count;
};

Packing choose_packing(int W, const uint64_t* stats) {
  int fixed_ones = 0, vary_bytes = 0;
  for (int q = 0; q < W; ++q) {
    fixed_ones += __builtin_popcountll(stats[W + 2 + q] & ~stats[q]);
    for (int b = 0; b < 8; ++b) vary_bytes += ((stats[q] >> (8 * b)) & 0xFF) != 0;
  }
  int varying = 0;
  for (int q = 0; q < W; ++q) varying += __builtin_popcountll(stats[q]);
  Packing best{0, 0, 0};
  int bits = 1;
  while ((1 << bits) - 1 < 64 * W) ++bits;  // every position and "none"
  for (int ones = 0; ones < 2; ++ones) {
    // most ones (zeros) a state has among the varying bits
    const int count = ones ? (int)stats[W + 1] - fixed_ones : varying - ((int)stats[W] - fixed_ones);
    if (count < 1 || count * bits > 64) continue;
    if (best.count == 0 || count < best.count) best = Packing{ones, bits, count};
  }
  // passes of 12 bytes a key and a gather (three times the state) against passes of the whole state
  if (best.count && (best.count * best.bits + 7) / 8 * 12 + 3 * (8 * W + 4) >= vary_bytes * (8 * W + 4)) best.count = 0;
  return best;
}

}  // namespace edgpu

extern "C" int edgpu_state_stats(int n_words, const uint64_t* keys, int64_t n, uint64_t* stats, void* stream) {
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS || !keys || !stats || n < 1) return EDGPU_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemsetAsync(stats, 0, sizeof(uint64_t) * (2 * (size_t)n_words + 2), s) != cudaSuccess ||
      cudaMemsetAsync(stats + n_words, 0xFF, sizeof(uint64_t), s) != cudaSuccess)
    return EDGPU_ERR_CUDA;
  EDGPU_DISPATCH_W(n_words, {
    stats_kernel<W><<<grid_for(n, 1024), 256, 0, s>>>(keys, n, reinterpret_cast<unsigned long long*>(stats)); note_launch();
  });
  return check_launch();
}

extern "C" int edgpu_sort_packing(int n_words, const uint64_t* stats) {
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS || !stats) return -1;
  const Packing p = choose_packing(n_words, stats);
  return p.count * p.bits;
}

extern "C" size_t edgpu_sort_states_packed_workspace(int n_words, int64_t n) {
  const size_t a = edgpu_sort_states_workspace(n_words, n);
  const size_t b = ((size_t)n * (8 + 4 + 8 * (size_t)n_words + 4) + 1024) + edgpu_sort_states_workspace(1, n);
  return a > b ? a : b;
}

extern "C" int edgpu_sort_states_packed(int n_words, uint64_t* keys, uint32_t* payload, int64_t n,
                                        const uint64_t* stats, void* workspace, size_t workspace_bytes, void* stream) {
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS || n < 0) return EDGPU_ERR_ARG;
  if (n <= 1) return EDGPU_OK;
  if (!keys || !payload || !stats) return EDGPU_ERR_ARG;
  const Packing pk = choose_packing(n_words, stats);
  // small inputs are sorted in one CTA's shared memory whatever their bits
  if (pk.count == 0 || n >= (1ll << 32) || small_sort_fits(n_words, n) || small_sort_fits(1, n))
    return edgpu_sort_states(n_words, keys, payload, n, stats, workspace, workspace_bytes, stream);
  if (workspace_bytes < edgpu_sort_states_packed_workspace(n_words, n)) return EDGPU_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  size_t off = 0;
  auto carve = [&](size_t bytes) {
    unsigned char* p = ws + off;
    off += (bytes + 255) & ~(size_t)255;
    return p;
  };
  uint64_t* packed = reinterpret_cast<uint64_t*>(carve(8 * (size_t)n));
  uint64_t* src = reinterpret_cast<uint64_t*>(carve(8 * (size_t)n * n_words));
  uint32_t* idx = reinterpret_cast<uint32_t*>(carve(4 * (size_t)n));
  uint32_t* psrc = reinterpret_cast<uint32_t*>(carve(4 * (size_t)n));
  VaryMask vary{};
  for (int q = 0; q < n_words; ++q) vary.w[q] = stats[q];
  EDGPU_DISPATCH_W(n_words, {
    pack_kernel<W><<<grid_for(n, 256), 256, 0, s>>>(keys, n, vary, pk.ones, pk.bits, pk.count, packed, idx); note_launch();
  });
  int rc = check_launch();
  if (rc) return rc;
  const int total = pk.bits * pk.count;
  const uint64_t mask = total >= 64 ? ~0ull : (1ull << total) - 1;
  if ((rc = edgpu_sort_states(1, packed, idx, n, &mask, ws + off, workspace_bytes - off, stream))) return rc;
  if (cudaMemcpyAsync(src, keys, 8 * (size_t)n * n_words, cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(psrc, payload, 4 * (size_t)n, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return EDGPU_ERR_CUDA;
  EDGPU_DISPATCH_W(n_words, {
    gather_states_kernel<W><<<grid_for(n * W, 256), 256, 0, s>>>(src, psrc, idx, keys, payload, n); note_launch();
  });
  return check_launch();
}
