// Kernels of the scheduled and the paged H x (spmv.cu) and their launchers.  The shifted products (Y = H X +
// shift X, the float copies only) are kernels of their own, instantiated in spmv_shift.cu so that the two
// halves compile side by side.
#pragma once

#include <climits>

#include "common.cuh"
#include "pages.cuh"

namespace edgpu {

template <typename T>
struct Pack16;
template <>
struct Pack16<float> {
  using type = float4;
  static constexpr int runs = 2;
};
template <>
struct Pack16<double> {
  using type = double2;
  static constexpr int runs = 1;
};

// SHIFT: Y = H X + shift X, a kernel of its own here and below (only the float copies are shifted): with the
// shift as an argument alone the unshifted products took 2 to 12 % more (pages of 256 entries, 200 000 rows of
// 5 entries, R = 16: 14.4 -> 16.4 us).
template <typename T, bool VALC, int L, int U, bool SHIFT>
__global__ void spmv_sched_kernel(int64_t n_heavy, int64_t n, const int64_t* __restrict__ rp,
                                  const int32_t* __restrict__ col, const T* __restrict__ vals,
                                  const int32_t* __restrict__ sched, T shift,
                                  const typename Pack16<T>::type* __restrict__ X,
                                  typename Pack16<T>::type* __restrict__ Y) {
  using P = typename Pack16<T>::type;
  constexpr int RV = Pack16<T>::runs;
  constexpr int G = 32 / L;  // row groups per warp
  const int lane = threadIdx.x & 31;
  const int grp = lane / L, sub = lane - grp * L;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const bool heavy = warp < n_heavy;  // warp-uniform
  int64_t row = -1, e = 0, e1 = 0;
  int stride = 1;
  if (heavy) {
    row = __ldg(sched + warp);
    e = __ldg(rp + row) + grp;
    e1 = __ldg(rp + row + 1);
    stride = G;
  } else {
    const int64_t k = n_heavy + (warp - n_heavy) * G + grp;
    if (k < n) {
      row = __ldg(sched + k);
      e = __ldg(rp + row);
      e1 = __ldg(rp + row + 1);
    }
  }
  T ar[RV], ai[RV];
#pragma unroll
  for (int q = 0; q < RV; ++q) ar[q] = ai[q] = T(0);
  for (; e < e1; e += (int64_t)stride * U) {
    int c[U];
    T hr[U], hi[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t eu = e + (int64_t)u * stride;
      const bool ok = eu < e1;
      // the CSR is read once: streaming loads leave L2 to x
      c[u] = ok ? __ldcs(col + eu) : 0;
      if (VALC) {
        hr[u] = ok ? __ldcs(vals + 2 * eu) : T(0);
        hi[u] = ok ? __ldcs(vals + 2 * eu + 1) : T(0);
      } else {
        hr[u] = ok ? __ldcs(vals + eu) : T(0);
        hi[u] = T(0);
      }
    }
    P xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) xv[u] = (e + (int64_t)u * stride < e1) ? __ldg(X + (int64_t)c[u] * L + sub) : P{};
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const T* xs = reinterpret_cast<const T*>(&xv[u]);
#pragma unroll
      for (int q = 0; q < RV; ++q) {
        const T xr = xs[2 * q], xi = xs[2 * q + 1];
        ar[q] += hr[u] * xr;
        ai[q] += hr[u] * xi;
        if (VALC) {
          ar[q] -= hi[u] * xi;
          ai[q] += hi[u] * xr;
        }
      }
    }
  }
  if (heavy) {
#pragma unroll
    for (int o = L; o < 32; o <<= 1)
#pragma unroll
      for (int q = 0; q < RV; ++q) {
        ar[q] += __shfl_xor_sync(0xffffffffu, ar[q], o);
        ai[q] += __shfl_xor_sync(0xffffffffu, ai[q], o);
      }
    if (grp != 0) return;
  }
  if (row < 0) return;
  P out;
  T* os = reinterpret_cast<T*>(&out);
  // the row's x, when a multiple of it is added to the product: read last, for its registers
  const P own = SHIFT ? __ldg(X + row * L + sub) : P{};
  const T* xo = reinterpret_cast<const T*>(&own);
#pragma unroll
  for (int q = 0; q < RV; ++q) {
    os[2 * q] = SHIFT ? ar[q] + shift * xo[2 * q] : ar[q];
    os[2 * q + 1] = SHIFT ? ai[q] + shift * xo[2 * q + 1] : ai[q];
  }
  __stcs(Y + row * L + sub, out);
}

template <typename T, bool VALC, int L, bool SHIFT>
int launch_sched(const edgpu_csr* h, const T* vals, const int32_t* sched, int64_t n_heavy, int unroll, int block,
                 T shift, const void* x, void* y, cudaStream_t s) {
  using P = typename Pack16<T>::type;
  constexpr int G = 32 / L;
  const int64_t n = h->n;
  const int64_t warps = n_heavy + (n - n_heavy + G - 1) / G;
  const int64_t blocks = (warps * 32 + block - 1) / block;
  if (blocks > 0x7fffffffLL) return EDGPU_ERR_ARG;
  const P* X = reinterpret_cast<const P*>(x);
  P* Y = reinterpret_cast<P*>(y);
  auto kern = unroll == 4   ? spmv_sched_kernel<T, VALC, L, 4, SHIFT>
              : unroll == 8 ? spmv_sched_kernel<T, VALC, L, 8, SHIFT>
                            : spmv_sched_kernel<T, VALC, L, 2, SHIFT>;
  kern<<<(unsigned)blocks, block, 0, s>>>(n_heavy, n, h->row_ptr, h->col, vals, sched, shift, X, Y);
  note_launch();
  return check_launch();
}

template <typename T, bool VALC, bool SHIFT>
int dispatch_lanes(const edgpu_csr* h, const T* vals, const int32_t* sched, int64_t n_heavy, int unroll, int block,
                   T shift, const void* x, void* y, int L, cudaStream_t s) {
  switch (L) {
    case 1: return launch_sched<T, VALC, 1, SHIFT>(h, vals, sched, n_heavy, unroll, block, shift, x, y, s);
    case 2: return launch_sched<T, VALC, 2, SHIFT>(h, vals, sched, n_heavy, unroll, block, shift, x, y, s);
    case 4: return launch_sched<T, VALC, 4, SHIFT>(h, vals, sched, n_heavy, unroll, block, shift, x, y, s);
    case 8: return launch_sched<T, VALC, 8, SHIFT>(h, vals, sched, n_heavy, unroll, block, shift, x, y, s);
    case 16: return launch_sched<T, VALC, 16, SHIFT>(h, vals, sched, n_heavy, unroll, block, shift, x, y, s);
    case 32: return launch_sched<T, VALC, 32, SHIFT>(h, vals, sched, n_heavy, unroll, block, shift, x, y, s);
    default: return EDGPU_ERR_ARG;
  }
}

// ---------------------------------------------------------------------------------------
// Paged layout (edgpu_spmv_pages_build / edgpu_spmv_paged[_c64]).
//
// The rows of a schedule are cut into slices and packed whole, in schedule order, into
// fixed-size pages of CH entries.  A heavy row is a slice of its own whose entries are dealt
// to the C = 32 / L row groups of a warp in turn (group r takes entries r, r + C, ...); a
// light slice holds C consecutive light rows, one per group.  A page is a header column (C
// entries; the first holds the number of used columns), then per slice a header column
// (entry r: column -2 - row of group r, or INT_MIN for none, and a flag set for a heavy row)
// and the slice's entry columns (entry (k, r): column and value of the group's k-th entry,
// column -1 past its end).
//
// One warp serves one page: it copies the page into shared memory with cp.async (16-byte
// chunks, coalesced) and reads its columns as one stream, U columns per batch, so U gathers
// of x rows per lane are in flight whatever the slice boundaries; a slice header column
// closes the groups' previous rows (adding a heavy row's partial sums across the groups with
// xor shuffles) and opens the next.  The only memory latencies on a warp's path are the page
// copy and the gathers; the rows, columns and values come from shared memory.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16_hint(void* smem, const void* gmem, uint64_t pol) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// L2 eviction-priority policies (PTX createpolicy): x rows are gathered nnz times and should
// stay in L2; pages are read once.
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ float4 ldg_hint(const float4* ptr, uint64_t pol) {
  float4 v;
  asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ double2 ldg_hint(const double2* ptr, uint64_t pol) {
  double2 v;
  asm volatile("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;\n" : "=d"(v.x), "=d"(v.y) : "l"(ptr), "l"(pol));
  return v;
}

constexpr int kPageWarps = 4;  // warps (pages) per block of the paged kernel

template <typename T, bool VALC, int L, int U, int CH, bool PIPE, bool HINT, bool SHIFT>
__global__ void __launch_bounds__(32 * kPageWarps) spmv_pages_kernel(int64_t n_pages,
                                                                     const Ent<T, VALC>* __restrict__ pages, T shift,
                                                                     const typename Pack16<T>::type* __restrict__ X,
                                                                     typename Pack16<T>::type* __restrict__ Y) {
  using E = Ent<T, VALC>;
  using P = typename Pack16<T>::type;
  constexpr int RV = Pack16<T>::runs;
  constexpr int C = 32 / L;
  constexpr int CHUNKS = CH * (int)sizeof(E) / 16;  // 16-byte copies per page
  extern __shared__ __align__(16) unsigned char page_raw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int grp = lane / L, sub = lane - grp * L;
  const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (p >= n_pages) return;  // warp-uniform
  E* pg = reinterpret_cast<E*>(page_raw) + (size_t)wib * CH;
  uint64_t pol_x = 0;
  {
    const unsigned char* src = reinterpret_cast<const unsigned char*>(pages + p * CH);
    unsigned char* dst = reinterpret_cast<unsigned char*>(pg);
    if constexpr (HINT) {
      pol_x = l2_policy_evict_last();
      const uint64_t pol_p = l2_policy_evict_first();
#pragma unroll
      for (int k = lane; k < CHUNKS; k += 32) cp_async16_hint(dst + 16 * k, src + 16 * k, pol_p);
    } else {
#pragma unroll
      for (int k = lane; k < CHUNKS; k += 32) cp_async16(dst + 16 * k, src + 16 * k);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncwarp();
  }
  T ar[RV], ai[RV];
#pragma unroll
  for (int q = 0; q < RV; ++q) ar[q] = ai[q] = T(0);
  int64_t row = -1;
  bool heavy = false;
  auto flush = [&]() {  // called by the whole warp at the same column
    if (heavy) {
#pragma unroll
      for (int o = L; o < 32; o <<= 1)
#pragma unroll
        for (int q = 0; q < RV; ++q) {
          ar[q] += __shfl_xor_sync(0xffffffffu, ar[q], o);
          ai[q] += __shfl_xor_sync(0xffffffffu, ai[q], o);
        }
    }
    if (row >= 0 && (!heavy || grp == 0)) {
      P out;
      T* os = reinterpret_cast<T*>(&out);
      // read here and not with the row's header: four registers less, 10 blocks an SM instead of 9
      const P own = SHIFT ? __ldg(X + row * L + sub) : P{};
      const T* xo = reinterpret_cast<const T*>(&own);
#pragma unroll
      for (int q = 0; q < RV; ++q) {
        os[2 * q] = SHIFT ? ar[q] + shift * xo[2 * q] : ar[q];
        os[2 * q + 1] = SHIFT ? ai[q] + shift * xo[2 * q + 1] : ai[q];
      }
      __stcs(Y + row * L + sub, out);
    }
#pragma unroll
    for (int q = 0; q < RV; ++q) ar[q] = ai[q] = T(0);
  };
  const int ncols = pg[0].c;
  E en[U];
  P xv[U];
  // batch k: U columns from shared memory, then their gathers (issued before the previous
  // batch is consumed when PIPE, so two batches of gathers are in flight)
  auto fetch = [&](int k, E* e, P* x) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k + u < ncols) {
        e[u] = pg[(k + u) * C + grp];
      } else {
        e[u] = E{};
        e[u].c = -1;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if constexpr (HINT) {
        x[u] = e[u].c >= 0 ? ldg_hint(X + (int64_t)e[u].c * L + sub, pol_x) : P{};
      } else {
        x[u] = e[u].c >= 0 ? __ldg(X + (int64_t)e[u].c * L + sub) : P{};
      }
    }
  };
  auto consume = [&](const E* e, const P* x) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = e[u].c;
      if (c <= -2) {  // a slice header column (the same kind in every group)
        flush();
        row = c == INT_MIN ? -1 : (int64_t)(-2 - (int64_t)c);
        heavy = e[u].flag() != 0;
        continue;
      }
      if (c < 0) continue;
      const T* xs = reinterpret_cast<const T*>(&x[u]);
      T hr, hi = T(0);
      if constexpr (VALC) {
        hr = e[u].vr;
        hi = e[u].vi;
      } else {
        hr = e[u].v;
      }
#pragma unroll
      for (int q = 0; q < RV; ++q) {
        const T xr = xs[2 * q], xi = xs[2 * q + 1];
        ar[q] += hr * xr;
        ai[q] += hr * xi;
        if (VALC) {
          ar[q] -= hi * xi;
          ai[q] += hi * xr;
        }
      }
    }
  };
  if constexpr (PIPE) {
    E en2[U];
    P xv2[U];
    if (1 < ncols) fetch(1, en, xv);
    for (int k = 1; k < ncols; k += 2 * U) {
      if (k + U < ncols) fetch(k + U, en2, xv2);
      consume(en, xv);
      if (k + U >= ncols) break;
      if (k + 2 * U < ncols) fetch(k + 2 * U, en, xv);
      consume(en2, xv2);
    }
  } else {
    for (int k = 1; k < ncols; k += U) {
      fetch(k, en, xv);
      consume(en, xv);
    }
  }
  flush();
}

template <typename T, bool VALC, int L, int U, int CH, bool SHIFT>
int launch_pages_t(int64_t n_pages, const void* pages, T shift, const void* x, void* y, cudaStream_t s, int flags) {
  using P = typename Pack16<T>::type;
  using E = Ent<T, VALC>;
  auto kern = (flags & 1) ? ((flags & 2) ? spmv_pages_kernel<T, VALC, L, U, CH, true, true, SHIFT>
                                         : spmv_pages_kernel<T, VALC, L, U, CH, true, false, SHIFT>)
                          : ((flags & 2) ? spmv_pages_kernel<T, VALC, L, U, CH, false, true, SHIFT>
                                         : spmv_pages_kernel<T, VALC, L, U, CH, false, false, SHIFT>);
  const size_t smem = (size_t)kPageWarps * CH * sizeof(E);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    return EDGPU_ERR_CUDA;
  }
  const int64_t blocks = (n_pages + kPageWarps - 1) / kPageWarps;
  if (blocks > 0x7fffffffLL) return EDGPU_ERR_ARG;
  kern<<<(unsigned)blocks, 32 * kPageWarps, smem, s>>>(n_pages, reinterpret_cast<const E*>(pages), shift,
                                                        reinterpret_cast<const P*>(x), reinterpret_cast<P*>(y));
  note_launch();
  return check_launch();
}

// unroll: 4 or 8 gathers per lane per batch; flags bit 0: two batches in flight, bit 1: L2
// eviction hints (x rows evict-last, pages evict-first)
template <typename T, bool VALC, int L, bool SHIFT>
int launch_pages_l(int64_t n_pages, const void* pages, int CH, int unroll, int flags, T shift, const void* x, void* y,
                   cudaStream_t s) {
  if (CH == 256 && unroll == 4) return launch_pages_t<T, VALC, L, 4, 256, SHIFT>(n_pages, pages, shift, x, y, s, flags);
  if (CH == 256 && unroll == 8) return launch_pages_t<T, VALC, L, 8, 256, SHIFT>(n_pages, pages, shift, x, y, s, flags);
  if (CH == 512 && unroll == 4) return launch_pages_t<T, VALC, L, 4, 512, SHIFT>(n_pages, pages, shift, x, y, s, flags);
  if (CH == 512 && unroll == 8) return launch_pages_t<T, VALC, L, 8, 512, SHIFT>(n_pages, pages, shift, x, y, s, flags);
  if (CH == 1024 && unroll == 4) return launch_pages_t<T, VALC, L, 4, 1024, SHIFT>(n_pages, pages, shift, x, y, s, flags);
  if (CH == 1024 && unroll == 8) return launch_pages_t<T, VALC, L, 8, 1024, SHIFT>(n_pages, pages, shift, x, y, s, flags);
  return EDGPU_ERR_ARG;
}

template <typename T, bool VALC, bool SHIFT>
int launch_pages(int64_t n_pages, const void* pages, int CH, int unroll, int flags, int L, T shift, const void* x,
                 void* y, cudaStream_t s) {
  switch (L) {
    case 2: return launch_pages_l<T, VALC, 2, SHIFT>(n_pages, pages, CH, unroll, flags, shift, x, y, s);
    case 4: return launch_pages_l<T, VALC, 4, SHIFT>(n_pages, pages, CH, unroll, flags, shift, x, y, s);
    case 8: return launch_pages_l<T, VALC, 8, SHIFT>(n_pages, pages, CH, unroll, flags, shift, x, y, s);
    case 16: return launch_pages_l<T, VALC, 16, SHIFT>(n_pages, pages, CH, unroll, flags, shift, x, y, s);
    default: return EDGPU_ERR_ARG;
  }
}

extern template int dispatch_lanes<float, true, true>(const edgpu_csr*, const float*, const int32_t*, int64_t, int, int,
                                                      float, const void*, void*, int, cudaStream_t);
extern template int dispatch_lanes<float, false, true>(const edgpu_csr*, const float*, const int32_t*, int64_t, int,
                                                       int, float, const void*, void*, int, cudaStream_t);
extern template int launch_pages<float, true, true>(int64_t, const void*, int, int, int, int, float, const void*, void*,
                                                    cudaStream_t);
extern template int launch_pages<float, false, true>(int64_t, const void*, int, int, int, int, float, const void*,
                                                     void*, cudaStream_t);

}  // namespace edgpu
