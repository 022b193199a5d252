// Sparse H·v, batched Lanczos tridiagonalisation, Lanczos with full reorthogonalisation,
// Ritz/shifted-solve vector assembly and continued fractions.
//
// Upstream counterparts: get_tridiagonal_krylov_vectors (impurityModel/ed/finite.py:1897-1995),
// scipy eigsh in eigensystem (finite.py:105), BiCGSTAB in getRIXSmap (spectra.py:962,1080)
// and the continued fraction of getGreen (spectra.py:678-680).
//
// Vectors of a batch are stored [n][R] (run index fastest) so that the R threads of one
// row read the row's CSR entries once (broadcast) and gather x[col][0..R) contiguously.
// All reductions are deterministic: per-block partials in fixed order, summed in fixed order.
#include <algorithm>
#include <atomic>
#include <climits>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "common.cuh"
#include "df64.cuh"

namespace cg = cooperative_groups;

namespace edgpu {

template <typename T>
struct Cx;
template <>
struct Cx<double> {
  using V = double2;
};
template <>
struct Cx<float> {
  using V = float2;
};

__device__ __forceinline__ double2 ld(const double2* p) { return *p; }
__device__ __forceinline__ float2 ld(const float2* p) { return *p; }

struct RunTile {
  int rt;   // runs per block (blockDim.x)
  int rb;   // rows per block pass (blockDim.y)
  int nrb;  // row blocks (gridDim.x)
  int nrt;  // run tiles (gridDim.y)
};

inline RunTile make_tile(int64_t n, int R) {
  RunTile t;
  t.rt = R < 32 ? R : 32;
  t.rb = 256 / t.rt;
  if (t.rb < 1) t.rb = 1;
  t.nrt = (R + t.rt - 1) / t.rt;
  int64_t nrb = (n + t.rb - 1) / t.rb;
  // about 4 blocks per SM in total over the (row block, run tile) grid
  int64_t cap = ((int64_t)grid_cap() * 4 + t.nrt - 1) / t.nrt;
  if (cap < 1) cap = 1;
  if (nrb > cap) nrb = cap;
  if (nrb < 1) nrb = 1;
  t.nrb = (int)nrb;
  return t;
}

// y = H x and the per-block partials of Re<y, x>: one vector, a row per thread (blockDim.y of them).
template <bool VALC>
__global__ void spmv_alpha_kernel(int64_t n, const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                  const double* __restrict__ vals, const double2* __restrict__ x,
                                  double2* __restrict__ y, double* __restrict__ partial) {
  extern __shared__ double red[];
  const int ti = threadIdx.y;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.y + ti; i < n; i += (int64_t)gridDim.x * blockDim.y) {
    double yr = 0.0, yi = 0.0;
    const int64_t e1 = rp[i + 1];
    for (int64_t e = rp[i]; e < e1; ++e) {
      const double2 xv = x[col[e]];
      if (VALC) {
        const double hr = vals[2 * e], hi = vals[2 * e + 1];
        yr += hr * xv.x - hi * xv.y;
        yi += hr * xv.y + hi * xv.x;
      } else {
        const double h = vals[e];
        yr += h * xv.x;
        yi += h * xv.y;
      }
    }
    y[i] = make_double2(yr, yi);
    const double2 v = x[i];
    acc += yr * v.x + yi * v.y;
  }
  red[ti] = acc;
  __syncthreads();
  if (ti == 0) {
    double s = 0.0;
    for (int k = 0; k < (int)blockDim.y; ++k) s += red[k];
    partial[blockIdx.x] = s;
  }
}

// ---------------------------------------------------------------------------------------
// Grid-wide batched Lanczos (lanczos_impl): two launches per step on vectors kept unnormalised.
// Serves complex64 vectors, more runs or larger sectors than lanczos_grid_kernel below, and the
// allocation-free entry point (whose callers forbid what a cooperative launch might allocate in the driver).
//
// w_j is stored as it leaves the three-term update and v_j = w_j / beta_{j-1} is never formed:
// the first launch takes y = H w_j and the partial sums of <y, w_j>, the second
//   alpha_j = <y, w_j> / beta_{j-1}^2,
//   w_{j+1} = y / beta_{j-1} - (alpha_j / beta_{j-1}) w_j - (beta_{j-1} / beta_{j-2}) w_{j-1}
// with the partial sums of |w_{j+1}|^2, so the normalising pass over the vectors and its launch
// are gone.  What bounded the three-launch form on the 47 895-state sector (R = 3: 36 us each)
// was not the vectors but every block adding the other blocks' 564 partials one after another
// (dependent FP64 adds, ~64 cycles each on GB300) and one CSR entry in flight per thread; here
// a block's threads share the partials (four chains each, then a fixed tree) and each thread
// keeps kStepUnroll gathers in flight.  Per step 108 -> 33 us there, most of it FP64 issue (1300
// FP64 warp instructions an SM in the product, rows of 3 to 13 entries side by side in a warp).
// ---------------------------------------------------------------------------------------
constexpr int kStepUnroll = 4;
constexpr int kStepMaxThreads = 512;

// The tile of a batch: run tiles as make_tile, in blocks of 512 threads (at most two an SM) where
// there are rows for three quarters of those, else in blocks of 256.  Every block adds up all
// blocks' partials, and the FP64 pipe takes ~15 cycles a warp instruction: 304 blocks instead of
// 564 take the update from 15 to 12 us at n = 47 895, R = 3; 1024 threads (152 blocks) take it to 10
// but the product from 20 to 23, its phases no longer overlapping another block's.
inline RunTile make_step_tile(int64_t n, int R) {
  RunTile t = make_tile(n, R);
  const int rb = kStepMaxThreads / t.rt;
  const int64_t blocks = (n + rb - 1) / rb, cap = std::max(1, 2 * grid_cap() / t.nrt);
  if (2 * blocks * t.nrt >= 3 * grid_cap()) {
    t.rb = rb;
    t.nrb = (int)std::min(blocks, cap);
  }
  return t;
}

// Sum over the thread rows ti of the block's per-thread values (thread (tr, ti) holds run tr's
// part), in a fixed tree; valid for every thread of run tr after the call.  Synchronises.
__device__ __forceinline__ double tile_sum(double v, double* red) {
  const int tr = threadIdx.x, ti = threadIdx.y, rt = blockDim.x;
  __syncthreads();
  red[ti * rt + tr] = v;
  __syncthreads();
  for (int len = blockDim.y; len > 1;) {
    const int h = (len + 1) >> 1;
    if (ti + h < len) red[ti * rt + tr] += red[(ti + h) * rt + tr];
    __syncthreads();
    len = h;
  }
  return red[tr];
}

// Sum of run r's nb per-block partials p[b * R + r], shared by the block's thread rows.
__device__ __forceinline__ double tile_partials(const double* __restrict__ p, int nb, int R, int r, double* red) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  if (r < R) {
    const int step = blockDim.y;
    int b = threadIdx.y;
    for (; b + 3 * step < nb; b += 4 * step) {
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += p[(int64_t)(b + q * step) * R + r];
    }
    for (; b < nb; b += step) s[0] += p[(int64_t)b * R + r];
  }
  return tile_sum((s[0] + s[1]) + (s[2] + s[3]), red);
}

// A row's products, one thread per run, entries [e, e1) in steps of `stride`, kStepUnroll gathers
// in flight.
template <typename T, bool VALC>
__device__ __forceinline__ typename Cx<T>::V row_products(int64_t e, int64_t e1, int stride,
                                                          const int32_t* __restrict__ col,
                                                          const T* __restrict__ vals, int R, int r,
                                                          const typename Cx<T>::V* __restrict__ X) {
  using V = typename Cx<T>::V;
  T yr = 0, yi = 0;
  for (; e < e1; e += (int64_t)kStepUnroll * stride) {
    int c[kStepUnroll];
    T hr[kStepUnroll], hi[kStepUnroll];
#pragma unroll
    for (int u = 0; u < kStepUnroll; ++u) {
      const int64_t eu = e + (int64_t)u * stride;
      const bool ok = eu < e1;
      c[u] = ok ? __ldg(col + eu) : -1;
      hr[u] = ok ? __ldg(vals + (VALC ? 2 * eu : eu)) : T(0);
      hi[u] = VALC && ok ? __ldg(vals + 2 * eu + 1) : T(0);
    }
    V x[kStepUnroll];
#pragma unroll
    for (int u = 0; u < kStepUnroll; ++u)
      if (c[u] >= 0) x[u] = ld(X + (int64_t)c[u] * R + r);
#pragma unroll
    for (int u = 0; u < kStepUnroll; ++u) {
      if (c[u] < 0) break;
      yr += hr[u] * x[u].x;
      yi += hr[u] * x[u].y;
      if (VALC) {
        yr -= hi[u] * x[u].y;
        yi += hi[u] * x[u].x;
      }
    }
  }
  V y;
  y.x = yr;
  y.y = yi;
  return y;
}

// Rows longer than this are split among kStepSplit threads per run, after the others.  The sectors' first
// rows (few bath holes) are the long ones: 3045 of the 47 895 hold 43 % of the entries, about 65 each,
// against 7 in the others, and one thread's chain of 65 gathers was the launch's length.  Not with more
// than 32 runs: a warp is then one row of 32 runs, and there are warps enough beside the long ones.
// The block's threads meet only for the long rows: a barrier in every pass of 16 rows cost 200 000 rows and
// 100 runs 20 % against the row loop without one (6 steps 7.99 -> 6.12 ms; 47 895 rows of the
// 316-spin-orbital sector 2.83 -> 2.44, split rows given up too).
constexpr int kStepHeavy = 24;
constexpr int kStepSplit = 8;

// Y = H X, per-block partials of Re<Y, X> per run into pa.  Thread (tr, ti) takes run tr of row
// ti of the block's pass; consecutive rows go to different blocks (groups of `group` rows) so that
// the long rows, neighbours in the basis, spread over all SMs.  The first row block also turns
// the previous update's norm partials pb into beta[.][j - 1] (nothing else reads them).
template <typename T, bool VALC>
__global__ void __launch_bounds__(kStepMaxThreads, 2) step_spmm_kernel(int64_t n, const int64_t* __restrict__ rp,
                                                        const int32_t* __restrict__ col, const T* __restrict__ vals,
                                                        int R, int group, int heavy, const typename Cx<T>::V* __restrict__ X,
                                                        typename Cx<T>::V* __restrict__ Y, double* __restrict__ pa,
                                                        const double* __restrict__ pb, double* __restrict__ beta,
                                                        int K, int j, const int32_t* __restrict__ k_max,
                                                        int32_t* status) {
  using V = typename Cx<T>::V;
  extern __shared__ double red[];
  __shared__ int64_t heavy_row[kStepMaxThreads];
  __shared__ int warp_heavy[kStepMaxThreads / 32];
  __shared__ V part[kStepMaxThreads];
  const int tr = threadIdx.x, ti = threadIdx.y, rb = blockDim.y;
  const int tid = ti * blockDim.x + tr, lane = tid & 31, warp = tid >> 5;
  const int r = blockIdx.y * blockDim.x + tr;
  double acc = 0.0;
  const auto row_of = [&](int64_t base) {
    const int64_t lin = base + ti;
    return (lin / group * gridDim.x + blockIdx.x) * group + lin % group;
  };
  const auto more = [&](int64_t base) { return base / group * group * gridDim.x < n; };  // block-uniform; rb may cut a group
  bool any = false;
  for (int64_t base = 0; more(base); base += rb) {
    const int64_t i = row_of(base);
    if (i >= n) continue;
    const int64_t e0 = __ldg(rp + i), e1 = __ldg(rp + i + 1);
    if (e1 - e0 > heavy) {
      any = true;
    } else if (r < R) {
      const V v = ld(X + i * R + r);
      const V y = row_products<T, VALC>(e0, e1, 1, col, vals, R, r, X);
      Y[i * R + r] = y;
      acc += (double)y.x * (double)v.x + (double)y.y * (double)v.y;
    }
  }
  // the long rows after the others, pass by pass, listed in thread order: kStepSplit threads per run and row,
  // their parts added in a fixed order by the first of them
  const bool long_rows = __syncthreads_or(any);
  for (int64_t base = 0; long_rows && more(base); base += rb) {
    const int64_t i = row_of(base);
    const bool mine = tr == 0 && i < n && __ldg(rp + i + 1) - __ldg(rp + i) > heavy;
    const int nh = __syncthreads_count(mine);
    if (nh == 0) continue;
    const int in_warp = (int)(blockDim.x * blockDim.y) - 32 * warp;  // threads of this warp
    const unsigned bal = __ballot_sync(in_warp >= 32 ? 0xffffffffu : (1u << in_warp) - 1u, mine);
    if (lane == 0) warp_heavy[warp] = __popc(bal);
    __syncthreads();
    if (mine) {
      int at = __popc(bal & ((1u << lane) - 1u));
      for (int q = 0; q < warp; ++q) at += warp_heavy[q];
      heavy_row[at] = i;
    }
    __syncthreads();
    const int slots = rb / kStepSplit, slot = ti / kStepSplit, seg = ti % kStepSplit;
    for (int h0 = 0; h0 < nh; h0 += slots) {
      const bool on = slot < slots && h0 + slot < nh && r < R;
      const int64_t ih = on ? heavy_row[h0 + slot] : 0;
      if (on) part[tid] = row_products<T, VALC>(__ldg(rp + ih) + seg, __ldg(rp + ih + 1), kStepSplit, col, vals, R, r, X);
      __syncthreads();
      if (on && seg == 0) {
        V y = part[tid];
#pragma unroll
        for (int q = 1; q < kStepSplit; ++q) {
          const V p = part[tid + q * blockDim.x];
          y.x += p.x;
          y.y += p.y;
        }
        const V v = ld(X + ih * R + r);
        Y[ih * R + r] = y;
        acc += (double)y.x * (double)v.x + (double)y.y * (double)v.y;
      }
      __syncthreads();
    }
  }
  const double s = tile_sum(acc, red);
  if (ti == 0 && r < R) pa[(int64_t)blockIdx.x * R + r] = s;
  if (blockIdx.x != 0 || j == 0) return;
  const double bt = sqrt(tile_partials(pb, gridDim.x, R, r, red));
  if (ti == 0 && r < R) {
    beta[(int64_t)r * K + (j - 1)] = bt;
    if (k_max[r] > j && !(bt > 0.0)) atomicExch(status, (int32_t)(bt == 0.0 ? EDGPU_ERR_BREAKDOWN : EDGPU_ERR_NAN));
  }
}

// alpha_j and, unless it is the last step, w_{j+1} into the buffer of w_{j-1} with the per-block
// partials of its squared norm.  nb: row blocks of the launch that wrote pa (and of this one
// unless it is the last step's, which runs one row block per run tile).
constexpr int kUpdateUnroll = 2;

template <typename T>
__global__ void __launch_bounds__(kStepMaxThreads, 2) step_update_kernel(int64_t n, int R, const typename Cx<T>::V* __restrict__ Y,
                                                          const typename Cx<T>::V* __restrict__ Wc,
                                                          typename Cx<T>::V* __restrict__ Wp,
                                                          const double* __restrict__ pa, int nb,
                                                          const double* __restrict__ beta, double* __restrict__ alpha,
                                                          int K, int j, double* __restrict__ pb) {
  using V = typename Cx<T>::V;
  extern __shared__ double red[];
  __shared__ double coef[3][32];  // of y, w_j, w_{j-1}
  const int tr = threadIdx.x, ti = threadIdx.y;
  const int r = blockIdx.y * blockDim.x + tr;
  double b1 = 1.0, i1 = 1.0, i2 = 1.0;  // beta_{j-1}, 1 / beta_{j-1}, 1 / beta_{j-2}; 1 where there is none
  if (ti == 0 && r < R) {  // one warp divides, not the whole block
    // a run whose beta was 0 has ended: its vector stays 0
    if (j > 0) {
      b1 = beta[(int64_t)r * K + (j - 1)];
      i1 = b1 > 0.0 ? 1.0 / b1 : 0.0;
    }
    if (j > 1) {
      const double b2 = beta[(int64_t)r * K + (j - 2)];
      i2 = b2 > 0.0 ? 1.0 / b2 : 0.0;
    }
  }
  // the thread's first elements are in flight while the partials are summed
  const int64_t step = (int64_t)gridDim.x * blockDim.y;
  const int64_t first = (int64_t)blockIdx.x * blockDim.y + ti;
  V y[kUpdateUnroll], w[kUpdateUnroll], p[kUpdateUnroll];
  auto fetch = [&](int64_t i0) {
#pragma unroll
    for (int u = 0; u < kUpdateUnroll; ++u) {
      const int64_t i = i0 + u * step;
      if (i < n) {
        y[u] = ld(Y + i * R + r);
        w[u] = ld(Wc + i * R + r);
        if (j > 0) p[u] = Wp[i * R + r];
      }
    }
  };
  if (r < R && j + 1 < K) fetch(first);
  const double sa = tile_partials(pa, nb, R, r, red);
  if (ti == 0 && r < R) {
    const double a = sa * i1 * i1;
    if (blockIdx.x == 0) alpha[(int64_t)r * K + j] = a;
    coef[0][tr] = i1;
    coef[1][tr] = -a * i1;
    coef[2][tr] = j > 0 ? -b1 * i2 : 0.0;
  }
  if (j + 1 >= K) return;  // the same for the whole launch
  __syncthreads();
  double acc = 0.0;
  if (r < R) {
    const T cy = (T)coef[0][tr], cw = (T)coef[1][tr], cp = (T)coef[2][tr];
    for (int64_t i0 = first; i0 < n; i0 += kUpdateUnroll * step) {
      if (i0 != first) fetch(i0);
#pragma unroll
      for (int u = 0; u < kUpdateUnroll; ++u) {
        const int64_t i = i0 + u * step;
        if (i >= n) break;
        T re = cy * y[u].x + cw * w[u].x, im = cy * y[u].y + cw * w[u].y;
        if (j > 0) {
          re += cp * p[u].x;
          im += cp * p[u].y;
        }
        V o;
        o.x = re;
        o.y = im;
        Wp[i * R + r] = o;
        acc += (double)re * (double)re + (double)im * (double)im;
      }
    }
  }
  const double s = tile_sum(acc, red);
  if (ti == 0 && r < R) pb[(int64_t)blockIdx.x * R + r] = s;
}

__global__ void to_c64_kernel(const double2* in, float2* out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 v = in[i];
    out[i] = make_float2((float)v.x, (float)v.y);
  }
}

__global__ void copy_c128_kernel(const double2* in, double2* out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[i];
}

// ---------------------------------------------------------------------------------------
// Full reorthogonalisation: dots h[k] = <V_k, w>, k < m; then w -= sum_k h[k] V_k.
// ---------------------------------------------------------------------------------------
constexpr int kDotTile = 8;

__global__ void multidot_kernel(const double2* __restrict__ V, int m, int64_t n, const double2* __restrict__ w,
                                double2* __restrict__ partial) {
  __shared__ double2 red[kDotTile][256 / 32];
  const int k0 = blockIdx.y * kDotTile;
  double2 acc[kDotTile];
#pragma unroll
  for (int k = 0; k < kDotTile; ++k) acc[k] = make_double2(0.0, 0.0);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 x = w[i];
#pragma unroll
    for (int k = 0; k < kDotTile; ++k) {
      if (k0 + k < m) {
        const double2 v = V[(int64_t)(k0 + k) * n + i];
        acc[k].x += v.x * x.x + v.y * x.y;
        acc[k].y += v.x * x.y - v.y * x.x;
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < kDotTile; ++k) {
    double a = acc[k].x, b = acc[k].y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) red[k][warp] = make_double2(a, b);
  }
  __syncthreads();
  if (threadIdx.x < kDotTile && k0 + threadIdx.x < m) {
    double a = 0.0, b = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
      a += red[threadIdx.x][q].x;
      b += red[threadIdx.x][q].y;
    }
    partial[(int64_t)(k0 + threadIdx.x) * gridDim.x + blockIdx.x] = make_double2(a, b);
  }
}

__global__ void sum_partials_kernel(const double2* partial, int m, int nb, double2* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  double a = 0.0, b = 0.0;
  for (int q = 0; q < nb; ++q) {
    a += partial[(int64_t)k * nb + q].x;
    b += partial[(int64_t)k * nb + q].y;
  }
  out[k] = make_double2(a, b);
}

__global__ void subtract_proj_kernel(const double2* __restrict__ V, int m, int64_t n, const double2* __restrict__ h,
                                     double2* __restrict__ w) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double2 x = w[i];
#pragma unroll 8
    for (int k = 0; k < m; ++k) {
      const double2 c = h[k];
      const double2 v = V[(int64_t)k * n + i];
      x.x -= c.x * v.x - c.y * v.y;
      x.y -= c.x * v.y + c.y * v.x;
    }
    w[i] = x;
  }
}

// Single-run helpers for the reorthogonalised Lanczos (R == 1 specialisations).
__global__ void reorth_alpha_update_kernel(int64_t n, double2* w, const double2* vj, const double2* vjm1,
                                           const double* palpha, int nrb, double* alpha, const double* beta, int j,
                                           double* pnorm) {
  __shared__ double red[256];
  __shared__ double a_s;
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int b = 0; b < nrb; ++b) t += palpha[b];
    a_s = t;
    if (blockIdx.x == 0) alpha[j] = t;
  }
  __syncthreads();
  const double a = a_s;
  const double bp = (j > 0) ? beta[j - 1] : 0.0;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double2 y = w[i];
    const double2 c = vj[i];
    y.x -= a * c.x;
    y.y -= a * c.y;
    if (j > 0) {
      const double2 p = vjm1[i];
      y.x -= bp * p.x;
      y.y -= bp * p.y;
    }
    w[i] = y;
    acc += y.x * y.x + y.y * y.y;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < (int)blockDim.x; ++k) s += red[k];
    pnorm[blockIdx.x] = s;
  }
}

// h[k] = <V_k, w> for k < m: one block per k, whole vector, deterministic block tree.
__global__ void __launch_bounds__(256) dot_per_k_kernel(const double2* __restrict__ V, int m, int64_t n,
                                                        const double2* __restrict__ w, double2* __restrict__ h) {
  __shared__ double red_r[8], red_i[8];
  const int k = blockIdx.x;
  if (k >= m) return;
  const double2* vk = V + (int64_t)k * n;
  double hr = 0.0, hi = 0.0;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double2 v = vk[i], x = w[i];
    hr += v.x * x.x + v.y * x.y;
    hi += v.x * x.y - v.y * x.x;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    hr += __shfl_down_sync(0xffffffffu, hr, o);
    hi += __shfl_down_sync(0xffffffffu, hi, o);
  }
  if (lane == 0) {
    red_r[warp] = hr;
    red_i[warp] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
      a += red_r[q];
      b += red_i[q];
    }
    h[k] = make_double2(a, b);
  }
}

// w -= sum_k h[k] V_k, block = 32 rows x 8 k-residue classes (smem reduction over the 8);
// with_norm: per-block partial |w|^2 of the updated rows into pnorm[blockIdx.x].
__global__ void __launch_bounds__(256) project_out_kernel(const double2* __restrict__ V, int m, int64_t n,
                                                          const double2* __restrict__ h, double2* __restrict__ w,
                                                          double* __restrict__ pnorm, int with_norm) {
  __shared__ double2 part[8][32];
  __shared__ double nrm[32];
  const int ri = threadIdx.x & 31, kc = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 32 + ri;
  double2 acc = make_double2(0.0, 0.0);
  if (i < n) {
#pragma unroll 4
    for (int k = kc; k < m; k += 8) {
      const double2 c = h[k];
      const double2 v = V[(int64_t)k * n + i];
      acc.x += c.x * v.x - c.y * v.y;
      acc.y += c.x * v.y + c.y * v.x;
    }
  }
  part[kc][ri] = acc;
  __syncthreads();
  if (kc == 0) {
    double nr = 0.0;
    if (i < n) {
      double2 x = w[i];
      for (int q = 0; q < 8; ++q) {
        x.x -= part[q][ri].x;
        x.y -= part[q][ri].y;
      }
      w[i] = x;
      nr = x.x * x.x + x.y * x.y;
    }
    nrm[ri] = nr;
  }
  __syncthreads();
  if (with_norm && threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < 32; ++q) t += nrm[q];
    pnorm[blockIdx.x] = t;
  }
}

__global__ void norm_partial_kernel(int64_t n, const double2* w, double* pnorm) {
  __shared__ double red[256];
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 y = w[i];
    acc += y.x * y.x + y.y * y.y;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < (int)blockDim.x; ++k) s += red[k];
    pnorm[blockIdx.x] = s;
  }
}

__global__ void reorth_normalize_kernel(int64_t n, const double2* w, double2* vnext, const double* pnorm, int nb,
                                        double* beta, int j, int32_t* status) {
  __shared__ double bt_s;
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int b = 0; b < nb; ++b) s += pnorm[b];
    bt_s = sqrt(s);
    if (blockIdx.x == 0) {
      beta[j] = bt_s;
      if (!(bt_s > 0.0)) atomicExch(status, (int32_t)(bt_s == 0.0 ? EDGPU_ERR_BREAKDOWN : EDGPU_ERR_NAN));
    }
  }
  __syncthreads();
  const double bt = bt_s;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 y = w[i];
    vnext[i] = bt > 0.0 ? make_double2(y.x / bt, y.y / bt) : make_double2(0.0, 0.0);
  }
}

// X[m][i] = sum_k C[k][m] V[k][i]
__global__ void combine_kernel(const double2* __restrict__ V, int K, int64_t n, const double2* __restrict__ C, int M,
                               double2* __restrict__ X) {
  const int m = blockIdx.y;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double xr = 0.0, xi = 0.0;
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
      const double2 c = C[(int64_t)k * M + m];
      const double2 v = V[(int64_t)k * n + i];
      xr += c.x * v.x - c.y * v.y;
      xi += c.x * v.y + c.y * v.x;
    }
    X[(int64_t)m * n + i] = make_double2(xr, xi);
  }
}

// Continued fraction g = 1 / (d_0 - b_0^2 / (d_1 - b_1^2 / ...)), d_i = omega + e - a_i + i delta, for
// every (run, omega), as the ratio g = D_1 / D_0 of
//   D_i = d_i D_{i+1} - b_i^2 D_{i+2},  D_k = 1, D_{k+1} = 0:
// no division in the loop.  The kernel is bound by FP64 issue (GB300: ~15 cycles a warp
// instruction), so the count of FP64 operations a step is its time.  With D_i scaled by delta^-1 a
// step (SCALED) the imaginary part of d_i is 1 and a step takes five: s = omega/delta - (a_i -
// e)/delta, then s D_r - D_i - c D2_r and s D_i + D_r - c D2_i as two fused operations each, c =
// (b_i/delta)^2.  750 runs x 4000 points, up to 150 steps: 9.27 -> 3.52 ms,
// the FP64 pipe busy 95 % of the time.
// Below kCfracMinDelta the quotients would leave the range of the scaling, and the unscaled step
// (seven operations) runs.  (a_i - e)/delta and c are staged in shared memory by the block, so the
// common energy cancels before anything is rounded against omega.  The exponents of D are looked
// at every fourth step on the integer pipe and brought back to 1 when they leave +-300 bits;
// ratios do not change under that.
// A block holds rt = 128 / wt runs x wt omegas (wt: 128, or the power of two that holds all of
// them), kCfracStage coefficients of its runs at a time.
constexpr int kCfracThreads = 128;
constexpr int kCfracStage = 1024;  // (a, b^2) pairs staged per block: 16 KiB
constexpr double kCfracMinDelta = 1e-9;

template <bool SCALED>
__global__ void __launch_bounds__(kCfracThreads)
    cfrac_kernel(const double* __restrict__ alpha, const double* __restrict__ beta,
                 const int32_t* __restrict__ k_len, int K, int R, const double* __restrict__ omega, int n_omega,
                 double delta, const double* __restrict__ e, const double* __restrict__ scale, int wt, int tiles,
                 double2* __restrict__ g) {
  __shared__ double2 ab[kCfracStage];
  __shared__ int longest;
  const int tid = threadIdx.x, tx = tid % wt, ty = tid / wt, rt = kCfracThreads / wt;
  const int64_t r0 = (int64_t)(blockIdx.x / tiles) * rt;
  const int64_t r = r0 + ty;
  const int w = (int)(blockIdx.x % tiles) * wt + tx;
  const int chunk = kCfracStage / rt;  // a multiple of 4 (rt <= 128)
  const double id = SCALED ? 1.0 / delta : 1.0;
  int kl = 0;
  double zr = 0.0;
  if (r < R && w < n_omega) {
    kl = min(k_len[r], K);
    // the rounding of omega + e at e's size is upstream's; taking e off again is exact
    const double er = e[r];
    zr = ((omega[w] + er) - er) * id;
  }
  if (tid == 0) longest = 0;
  __syncthreads();
  if (tx == 0) atomicMax(&longest, kl);
  __syncthreads();
  const int kmax = longest;
  double2 d1 = make_double2(1.0, 0.0), d2 = make_double2(0.0, 0.0);  // D_{i+1}, D_{i+2}
  for (int c0 = (kmax - 1) / chunk * chunk; c0 >= 0 && kmax > 0; c0 -= chunk) {
    const int cn = min(chunk, kmax - c0);
    __syncthreads();
    for (int q = tid; q < rt * chunk; q += kCfracThreads) {
      const int64_t rq = r0 + q / chunk;
      const int i = q % chunk;
      if (rq < R && i < cn) {
        const double a = alpha[rq * K + c0 + i] - e[rq], b = beta[rq * K + c0 + i] * id;
        ab[q] = make_double2(a * id, -(b * b));  // negated here: a negation takes the FP64 pipe
      }
    }
    __syncthreads();
    const double2* mine = ab + ty * chunk;
    for (int i0 = (cn - 1) & ~3; i0 >= 0; i0 -= 4) {
#pragma unroll
      for (int u = 3; u >= 0; --u) {
        const int i = i0 + u;
        if (c0 + i < kl) {
          const double2 c = mine[i];
          const double s = zr - c.x, b2 = c0 + i + 1 < kl ? c.y : 0.0;  // the last beta is not part of it
          double2 d;
          if (SCALED) {
            d.x = fma(b2, d2.x, fma(s, d1.x, -d1.y));
            d.y = fma(b2, d2.y, fma(s, d1.y, d1.x));
          } else {
            d.x = fma(b2, d2.x, fma(s, d1.x, -(delta * d1.y)));
            d.y = fma(b2, d2.y, fma(s, d1.y, delta * d1.x));
          }
          d2 = d1;
          d1 = d;
        }
      }
      const int m = max(max(__double2hiint(d1.x) & 0x7fffffff, __double2hiint(d1.y) & 0x7fffffff),
                        max(__double2hiint(d2.x) & 0x7fffffff, __double2hiint(d2.y) & 0x7fffffff));
      const int ex = m >> 20;
      // when one lane has to, the warp does: the lanes then stay in step
      if (__any_sync(0xffffffffu, (ex > 1323 && ex < 2046) || (ex < 723 && ex > 0))) {
        const double f = ex > 0 && ex < 2046 ? __hiloint2double((2046 - ex) << 20, 0) : 1.0;
        d1.x *= f;
        d1.y *= f;
        d2.x *= f;
        d2.y *= f;
      }
    }
  }
  if (r >= R || w >= n_omega) return;
  double2 o = make_double2(0.0, 0.0);
  if (kl > 0) {
    // g = D_1 / (delta D_0); D_0 is d1 after the last step, D_1 the one before
    const double f = (scale ? scale[r] : 1.0) * id / (d1.x * d1.x + d1.y * d1.y);
    o = make_double2(f * (d2.x * d1.x + d2.y * d1.y), f * (d2.y * d1.x - d2.x * d1.y));
  }
  g[r * n_omega + w] = o;
}

bool small_fits(int64_t n, int precision);
int lanczos_small(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K, int precision,
                  double* alpha, double* beta, int32_t* status, void* ws, cudaStream_t s);

// Mixed form: a'[r][i] = float(alpha - e_r), b2[r][i] = float(beta^2) (FP64 subtraction
// first, so the large common energy cancels exactly), then the fraction in float32.
__global__ void cfrac_prep_kernel(const double* __restrict__ alpha, const double* __restrict__ beta,
                                  const int32_t* __restrict__ k_len, int K, int R, const double* __restrict__ e,
                                  float* __restrict__ ap, float* __restrict__ b2) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)R * K) return;
  const int r = (int)(t / K);
  ap[t] = (float)(alpha[t] - e[r]);
  b2[t] = (float)(beta[t] * beta[t]);
  (void)k_len;
}

__global__ void cfrac_f32_kernel(const float* __restrict__ ap, const float* __restrict__ b2,
                                 const int32_t* __restrict__ k_len, int K, int R, const double* __restrict__ omega,
                                 int n_omega, double delta, const double* __restrict__ scale, double2* __restrict__ g) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (int64_t)R * n_omega) return;
  const int r = (int)(tid / n_omega);
  const int w = (int)(tid % n_omega);
  const int kl = k_len[r];
  const float zr = (float)omega[w];
  const float zi = (float)delta;
  const float* a = ap + (int64_t)r * K;
  const float* b = b2 + (int64_t)r * K;
  float gr = 0.f, gi = 0.f;
  for (int i = kl - 1; i >= 0; --i) {
    float dr = zr - a[i], di = zi;
    if (i != kl - 1) {
      dr -= b[i] * gr;
      di -= b[i] * gi;
    }
    const float inv = 1.0f / (dr * dr + di * di);
    gr = dr * inv;
    gi = -di * inv;
  }
  const double s = scale ? scale[r] : 1.0;
  g[tid] = kl > 0 ? make_double2(s * (double)gr, s * (double)gi) : make_double2(0.0, 0.0);
}

inline unsigned grid_1d(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)grid_cap() * 8;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

// Row-parallel SpMM for y = H x with x, y [n][R]: thread = (row i, group g of RV runs),
// L = R / RV threads per row, one row per thread, 16-byte vector loads of x (float4 holds
// two complex64 runs, double2 one complex128 run) and UNROLL independent gathers in flight.
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  using type = float4;
  static constexpr int runs = 2;
};
template <>
struct Vec16<double> {
  using type = double2;
  static constexpr int runs = 1;
};

constexpr int kRowsThreads = 128;  // smaller blocks shorten the tail of ragged rows

// RV runs per thread: what 16 bytes hold, or one (8 bytes) for an odd number of complex64 runs.
// SHIFT: Y = H X + shift X.  A kernel of its own, its x read as the row is stored: the shift and the x held through
// the row cost the unshifted FP64 products registers and 10 to 28 % of their time (200 000 rows of 5
// entries, R = 3: 24.6 -> 29.6 us, R = 16: 94 -> 120).
template <typename T, bool VALC, int RV, bool SHIFT>
__global__ void __launch_bounds__(kRowsThreads) spmm_rows_kernel(int64_t n, const int64_t* __restrict__ rp,
                                                                 const int32_t* __restrict__ col,
                                                                 const T* __restrict__ vals, int R, int L, T shift,
                                                                 const typename Cx<T>::V* __restrict__ X,
                                                                 typename Cx<T>::V* __restrict__ Y) {
  using Q = std::conditional_t<RV == Vec16<T>::runs, typename Vec16<T>::type, typename Cx<T>::V>;
  constexpr int UNROLL = 8;
  const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = gt / L;
  const int g = (int)(gt - i * L);
  if (i >= n) return;
  const int64_t r0 = (int64_t)g * RV;
  T ar[RV], ai[RV];
#pragma unroll
  for (int q = 0; q < RV; ++q) ar[q] = ai[q] = 0;
  const int64_t e1 = __ldg(rp + i + 1);
  // Batches of UNROLL entries, the last one predicated: every row needs at most three
  // dependent memory round trips per batch (row pointers, CSR entries, gathers of x).
  for (int64_t e = __ldg(rp + i); e < e1; e += UNROLL) {
    int c[UNROLL];
    T hr[UNROLL], hi[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const bool ok = e + u < e1;
      // CSR entries are read once: streaming loads keep x resident in L2
      c[u] = ok ? __ldcs(col + e + u) : 0;
      if (VALC) {
        hr[u] = ok ? __ldcs(vals + 2 * (e + u)) : T(0);
        hi[u] = ok ? __ldcs(vals + 2 * (e + u) + 1) : T(0);
      } else {
        hr[u] = ok ? __ldcs(vals + e + u) : T(0);
        hi[u] = 0;
      }
    }
    Q xv[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      xv[u] = (e + u < e1) ? __ldg(reinterpret_cast<const Q*>(X + (int64_t)c[u] * R + r0)) : Q{};
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
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
  Q out;
  T* os = reinterpret_cast<T*>(&out);
  const Q own = SHIFT ? __ldg(reinterpret_cast<const Q*>(X + i * R + r0)) : Q{};
  const T* xo = reinterpret_cast<const T*>(&own);
#pragma unroll
  for (int q = 0; q < RV; ++q) {
    os[2 * q] = SHIFT ? ar[q] + shift * xo[2 * q] : ar[q];
    os[2 * q + 1] = SHIFT ? ai[q] + shift * xo[2 * q + 1] : ai[q];
  }
  __stcs(reinterpret_cast<Q*>(Y + i * R + r0), out);
}

template <typename T, int RV>
int launch_rows(const edgpu_csr* h, const T* val_c, const T* val_r, T shift, const typename Cx<T>::V* x,
                typename Cx<T>::V* y, int R, cudaStream_t s) {
  const int L = R / RV;
  const int64_t blocks = (h->n * (int64_t)L + kRowsThreads - 1) / kRowsThreads;
  if (blocks > 0x7fffffffLL) return EDGPU_ERR_ARG;
  auto kern = val_c ? spmm_rows_kernel<T, true, RV, false> : spmm_rows_kernel<T, false, RV, false>;
  if constexpr (sizeof(T) == 4)  // only the float copies are shifted
    if (shift != T(0)) kern = val_c ? spmm_rows_kernel<T, true, RV, true> : spmm_rows_kernel<T, false, RV, true>;
  kern<<<(unsigned)blocks, kRowsThreads, 0, s>>>(h->n, h->row_ptr, h->col, val_c ? val_c : val_r, R, L, shift, x, y);
  note_launch();
  return check_launch();
}

inline bool spmv_aligned(const void* x, const void* y) {
  return ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
}

// Optional per-kernel timing with CUDA events on the launching stream: kernel_ms[0..2] receive
// the summed durations of the SpMM and the update launches (host array; [2] is 0).
struct KernelTimer {
  double* out;
  std::vector<cudaEvent_t> ev[2];
  cudaStream_t s;
  KernelTimer(double* o, int K, cudaStream_t st) : out(o), s(st) {
    if (!out) return;
    for (int k = 0; k < 2; ++k) {
      ev[k].resize(2 * (size_t)K);
      for (auto& e : ev[k]) cudaEventCreate(&e);
    }
  }
  void mark(int kind, int j, int phase) {
    if (out) cudaEventRecord(ev[kind][2 * (size_t)j + phase], s);
  }
  void finish(int K) {
    if (!out) return;
    out[2] = 0.0;
    for (int k = 0; k < 2; ++k) {
      double tot = 0.0;
      for (int j = 0; j < K; ++j) {
        float ms = 0.f;
        cudaEventSynchronize(ev[k][2 * (size_t)j + 1]);
        if (cudaEventElapsedTime(&ms, ev[k][2 * (size_t)j], ev[k][2 * (size_t)j + 1]) == cudaSuccess) tot += ms;
      }
      out[k] = tot;
    }
    for (int k = 0; k < 2; ++k)
      for (auto& e : ev[k]) cudaEventDestroy(e);
  }
};

// The same recurrence in FP64 as one cooperative launch, for sectors whose rows fit in the SMs' shared
// memory.  A block of 1024 threads per SM takes the rows b, b + B, ... (the long ones are neighbours in
// the basis), sorts them by length and keeps their entries, y, w and v_{j-1} in shared memory for all
// steps; only the unscaled w = beta_{j-1} v_j goes through L2, for the other blocks' gathers.  Two or four
// threads per row and run; a warp's rows have nearly equal lengths.  Two grid barriers a step (after the
// partials of alpha_j and of beta_j^2), the sums of the blocks' partials by a warp per run in one
// fixed order.
// Bound by latency: of a step's 25 us for 3 runs of 47 895 rows with 458 223 entries the products' FP64
// issue is 4.4 (16 cycles a warp instruction), their phase 10 to 15 (the long rows, lanes idle beside rows of
// six entries), the barriers and sums the rest.
// 100 steps there: 2.54 ms.  40 steps of 1, 3, 8, 16 runs 0.81, 1.12, 1.82, 3.21 ms, in two launches a step 1.12,
// 1.56, 2.18, 3.21 (their gaps, H and the vectors read again); of 32 runs of 4300 short rows 1.59 and 1.35.
constexpr int kGridThreads = 1024;
constexpr int kGridRuns = kGridThreads / 32;
constexpr int kGridRows = 2048;  // rows of a block at most (their ranks take rows^2 / 1024 steps)

struct GridArgs {
  int64_t n;
  const int64_t* rp;
  const int32_t* col;
  const double* vals;
  const double2* v0;
  int R, K;
  int sub;      // threads per row and run
  int ent_cap;  // entries a block has room for
  double2 *A, *B;
  double *pa, *pb;
  const int32_t* k_max;
  double *alpha, *beta;
  int32_t* status;
};

// Shared memory of a block without the entries.
inline size_t grid_fixed_bytes(int64_t rows, int R) {
  return 3 * sizeof(double2) * (size_t)rows * R + sizeof(double) * kGridThreads +
         (sizeof(int) + 2 * sizeof(uint16_t)) * (size_t)rows + 16;
}

template <bool VALC>
__global__ void __launch_bounds__(kGridThreads, 1) lanczos_grid_kernel(GridArgs g) {
  cg::grid_group grid = cg::this_grid();
  const int B = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, R = g.R, K = g.K;
  const int mine = (int)((g.n - b + B - 1) / B), items = mine * R;
  const int most = (int)((g.n + B - 1) / B);
  extern __shared__ __align__(16) unsigned char sm[];
  double2* y = reinterpret_cast<double2*>(sm);  // [slot][run], as w and p
  double2* w = y + (size_t)most * R;
  double2* p = w + (size_t)most * R;
  double* red = reinterpret_cast<double*>(p + (size_t)most * R);
  double* eval = red + kGridThreads;
  int* ecol = reinterpret_cast<int*>(eval + (size_t)g.ent_cap * (VALC ? 2 : 1));
  int* eoff = ecol + g.ent_cap;                               // [mine] a slot's first entry
  uint16_t* len = reinterpret_cast<uint16_t*>(eoff + most);   // [mine]
  uint16_t* order = len + most;                               // [mine] slot's row b + B * order
  __shared__ double s_ib[kGridRuns], s_cy[kGridRuns], s_cw[kGridRuns], s_cp[kGridRuns], s_b[kGridRuns];
  __shared__ int s_fits;

  for (int k = tid; k < mine; k += kGridThreads) {
    const int64_t i = b + (int64_t)B * k, l = g.rp[i + 1] - g.rp[i];
    len[k] = (uint16_t)(l < 0xFFFF ? l : 0xFFFF);
  }
  __syncthreads();
  for (int k = tid; k < mine; k += kGridThreads) {
    const int l = len[k];
    int at = 0;
    for (int q = 0; q < mine; ++q) at += len[q] > l || (len[q] == l && q < k);
    order[at] = (uint16_t)k;
  }
  __syncthreads();
  if (warp == 0) {
    int at = 0;
    bool fits = true;
    for (int q0 = 0; q0 < mine; q0 += 32) {
      const int l = q0 + lane < mine ? len[order[q0 + lane]] : 0;
      int end = l;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += o;
      }
      if (q0 + lane < mine) eoff[q0 + lane] = at + end - l;
      at += __shfl_sync(0xffffffffu, end, 31);
      fits = fits && at <= g.ent_cap;
      if (!fits) break;
    }
    if (lane == 0) s_fits = fits;
  }
  __syncthreads();
  const bool fits = s_fits;
  if (!fits) {
    for (int s = tid; s < mine; s += kGridThreads) eoff[s] = 0;
  } else {
    for (int s = warp; s < mine; s += kGridThreads / 32) {
      const int64_t e0 = g.rp[b + (int64_t)B * order[s]];
      const int l = len[order[s]], at = eoff[s];
      for (int e = lane; e < l; e += 32) {
        ecol[at + e] = g.col[e0 + e];
        if (VALC) {
          eval[2 * (at + e)] = g.vals[2 * (e0 + e)];
          eval[2 * (at + e) + 1] = g.vals[2 * (e0 + e) + 1];
        } else {
          eval[at + e] = g.vals[e0 + e];
        }
      }
    }
  }
  // dense loops: a run per thread whatever the pass
  const int dense = kGridThreads / R * R, dr = tid % R;
  if (tid < dense)
    for (int q = tid; q < items; q += dense) {
      w[q] = g.v0[(b + (int64_t)B * order[q / R]) * R + dr];
      p[q] = make_double2(0.0, 0.0);
    }
  if (tid < R) {
    s_ib[tid] = 1.0;
    s_b[tid] = 0.0;
  }
  __syncthreads();

  // products: g.sub threads per row and run
  const int sub = g.sub, per = kGridThreads / (R * sub) * R, gi = tid / sub, gs = tid % sub;
  const int slot0 = gi / R, gr = gi % R, slots = per / R;

  // sums of a run: the last warps, whose rows are the shortest
  const int run = kGridThreads / 32 - 1 - warp;
  // this block's partial of a dense sum, a warp per run
  auto partial = [&](double v, double* out) {
    red[tid] = v;
    __syncthreads();
    if (run < R) {
      const int lim = items < dense ? items : dense;
      double s[4] = {0.0, 0.0, 0.0, 0.0};
      for (int k = run + R * lane; k < lim; k += 128 * R) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k + 32 * R * u < lim) s[u] += red[k + 32 * R * u];
      }
      double t = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) out[(int64_t)b * R + run] = t;
    }
    grid.sync();
  };
  // the sum of all blocks' partials of `run`
  auto total = [&](const double* part) -> double {
    double s = 0.0;
    for (int q = lane; q < B; q += 32) s += part[(int64_t)q * R + run];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  };

  const double2* cur = g.v0;
  for (int j = 0; j < K; ++j) {
    // ---- y = H w, alpha_j
    if (gi < per) {
      const double2* x = cur + gr;
      for (int slot = slot0; slot < mine; slot += slots) {
        const int k0 = order[slot];
        int l = len[k0];
        const int* ec = ecol + eoff[slot];
        const double* ev = eval + (VALC ? 2 : 1) * eoff[slot];
        if (!fits) {
          const int64_t i = b + (int64_t)B * k0, e0 = g.rp[i];
          l = (int)(g.rp[i + 1] - e0);
          ec = g.col + e0;
          ev = g.vals + (VALC ? 2 : 1) * e0;
        }
        double yr = 0.0, yi = 0.0;
        for (int e = gs; e < l; e += 4 * sub) {
          double2 xv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (e + u * sub < l) xv[u] = x[(int64_t)ec[e + u * sub] * R];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = e + u * sub;
            if (k < l) {
              const double hr = ev[VALC ? 2 * k : k];
              yr = fma(hr, xv[u].x, yr);
              yi = fma(hr, xv[u].y, yi);
              if (VALC) {
                const double hi = ev[2 * k + 1];
                yr = fma(-hi, xv[u].y, yr);
                yi = fma(hi, xv[u].x, yi);
              }
            }
          }
        }
        // the threads of a row and run: neighbours in a warp
        const unsigned group = ((1u << sub) - 1u) << (lane & ~(sub - 1));
        for (int o = sub >> 1; o > 0; o >>= 1) {
          yr += __shfl_xor_sync(group, yr, o);
          yi += __shfl_xor_sync(group, yi, o);
        }
        if (gs == 0) y[slot * R + gr] = make_double2(yr, yi);
      }
    }
    __syncthreads();
    double acc = 0.0;
    if (tid < dense)
      for (int q = tid; q < items; q += dense) acc = fma(y[q].y, w[q].y, fma(y[q].x, w[q].x, acc));
    partial(acc, g.pa);
    if (run < R) {
      const double ib = s_ib[run], a = total(g.pa) * ib * ib;
      if (lane == 0) {
        if (b == 0) g.alpha[(int64_t)run * K + j] = a;
        s_cy[run] = ib;
        s_cw[run] = -a * ib;
        s_cp[run] = -s_b[run];
      }
    }
    if (j + 1 >= K) break;  // identical in every block
    __syncthreads();
    // ---- w' = y / beta_{j-1} - alpha_j v_j - beta_{j-1} v_{j-1}, beta_j
    double2* nxt = j & 1 ? g.B : g.A;
    acc = 0.0;
    if (tid < dense) {
      const double cy = s_cy[dr], cw = s_cw[dr], cp = s_cp[dr];
      for (int q = tid, s = tid / R; q < items; q += dense, s += dense / R) {
        const double2 v = w[q], h = y[q], o = p[q];
        double2 x;
        x.x = fma(cp, o.x, fma(cw, v.x, cy * h.x));
        x.y = fma(cp, o.y, fma(cw, v.y, cy * h.y));
        p[q] = make_double2(v.x * cy, v.y * cy);
        w[q] = x;
        nxt[(b + (int64_t)B * order[s]) * R + dr] = x;
        acc = fma(x.y, x.y, fma(x.x, x.x, acc));
      }
    }
    partial(acc, g.pb);
    if (run < R) {
      const double t = total(g.pb);
      if (lane == 0) {
        const double bt = sqrt(t);
        s_b[run] = bt;
        s_ib[run] = bt > 0.0 ? 1.0 / bt : 0.0;  // a run whose beta is 0 has ended: its vector stays 0
        if (b == 0) {
          g.beta[(int64_t)run * K + j] = bt;
          if (g.k_max[run] > j + 1 && !(bt > 0.0))
            atomicExch(g.status, (int32_t)(bt == 0.0 ? EDGPU_ERR_BREAKDOWN : EDGPU_ERR_NAN));
        }
      }
    }
    cur = nxt;
  }
}

// Launches the cooperative form where the sector's vectors and entries fit in shared memory (without the
// entries 40 steps of 300 000 rows take 3.4 ms against 2.4 in two launches a step): false when the caller's two
// launches a step take the call, also where the launch is refused (a program that has only a part of the
// SMs cannot hold all blocks at once).
static bool launch_grid(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K, double* alpha,
                       double* beta, int32_t* status, unsigned char* ws, cudaStream_t s) {
  if (R > kGridRuns || (!h->val_c && !h->val_r)) return false;
  const int blocks = grid_cap();
  const int64_t most = (h->n + blocks - 1) / blocks;
  const bool cplx = h->val_c != nullptr;
  const size_t limit = 220 * 1024, per_entry = (cplx ? 16 : 8) + sizeof(int);
  if (h->n < blocks || most > kGridRows || grid_fixed_bytes(most, R) > limit) return false;
  GridArgs g{};
  const size_t room = (limit - grid_fixed_bytes(most, R)) / per_entry;
  if (room < (size_t)(h->nnz / blocks + h->nnz / blocks / 8 + 64)) return false;
  g.ent_cap = (int)std::min<size_t>(room, (size_t)(2 * (h->nnz / blocks) + 256)) & ~1;
  const size_t bytes = grid_fixed_bytes(most, R) + per_entry * (size_t)g.ent_cap;
  auto kern = cplx ? lanczos_grid_kernel<true> : lanczos_grid_kernel<false>;
  int dev = 0, coop = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kGridThreads, bytes) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return false;
  }
  // the same places in the workspace as the two launches a step: two vectors, the partials behind the third
  const size_t vec = (sizeof(double2) * (size_t)h->n * R + 255) & ~(size_t)255;
  const size_t part = (sizeof(double) * (size_t)blocks * R + 255) & ~(size_t)255;
  if (2 * part > vec) return false;  // pa and pb share the third vector's place
  g.n = h->n;
  g.rp = h->row_ptr;
  g.col = h->col;
  g.vals = cplx ? h->val_c : h->val_r;
  g.v0 = reinterpret_cast<const double2*>(v0);
  g.R = R;
  g.K = K;
  // The few long rows of a sector (65 entries, 9.6 on average) set the products' length: 40 steps of the
  // 316-spin-orbital sector take 1143, 864, 808 us with 1, 2, 4 threads a row for one run, 1349, 1114,
  // 1286 for 3 runs and 1930, 1822, 2542 for 8.
  g.sub = most * R <= 320 ? 4 : 2;
  g.A = reinterpret_cast<double2*>(ws);
  g.B = reinterpret_cast<double2*>(ws + vec);
  g.pa = reinterpret_cast<double*>(ws + 2 * vec);
  g.pb = reinterpret_cast<double*>(ws + 2 * vec + part);
  g.k_max = k_max;
  g.alpha = alpha;
  g.beta = beta;
  g.status = status;
  void* args[] = {&g};
  if (cudaLaunchCooperativeKernel((const void*)kern, blocks, kGridThreads, args, bytes, s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  note_launch();
  return true;
}

template <typename T>
int lanczos_impl(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K, double* alpha, double* beta,
                 int32_t* status, unsigned char* ws, size_t ws_bytes, cudaStream_t s, double* kernel_ms = nullptr) {
  using V = typename Cx<T>::V;
  const int64_t n = h->n;
  const int64_t nv = n * (int64_t)R;
  const RunTile t = make_step_tile(n, R);  // no more row blocks than the workspace was sized for
  size_t off = 0;
  auto carve = [&](size_t bytes) {
    unsigned char* p = ws + off;
    off += (bytes + 255) & ~(size_t)255;
    return p;
  };
  V* A = reinterpret_cast<V*>(carve(sizeof(V) * nv));
  V* B = reinterpret_cast<V*>(carve(sizeof(V) * nv));
  V* Wb = reinterpret_cast<V*>(carve(sizeof(V) * nv));
  double* pa = reinterpret_cast<double*>(carve(sizeof(double) * (size_t)t.nrb * R));
  double* pb = reinterpret_cast<double*>(carve(sizeof(double) * (size_t)t.nrb * R));
  if (off > ws_bytes) return EDGPU_ERR_WORKSPACE;
  if (sizeof(T) == 8)
    copy_c128_kernel<<<grid_1d(nv, 256), 256, 0, s>>>(reinterpret_cast<const double2*>(v0),
                                                       reinterpret_cast<double2*>(A), nv);
  else
    to_c64_kernel<<<grid_1d(nv, 256), 256, 0, s>>>(reinterpret_cast<const double2*>(v0),
                                                    reinterpret_cast<float2*>(A), nv); note_launch();
  int rc = check_launch();
  if (rc) return rc;
  dim3 grid(t.nrb, t.nrt), block(t.rt, t.rb);
  const size_t red = sizeof(double) * (size_t)t.rt * t.rb;
  const T* vals = nullptr;
  bool valc = false;
  if (sizeof(T) == 8) {
    valc = h->val_c != nullptr;
    vals = (const T*)(valc ? (const void*)h->val_c : (const void*)h->val_r);
  } else {
    valc = h->val_cf != nullptr;
    vals = (const T*)(valc ? (const void*)h->val_cf : (const void*)h->val_rf);
  }
  if (!vals) return EDGPU_ERR_ARG;
  V* Wc = A;
  V* Wp = B;
  // one pass over the rows: single rows dealt to the blocks; several: groups of 8, so that the
  // CSR of neighbouring rows is read by one block
  const int group = (int64_t)t.nrb * t.rb >= n ? 1 : 8;
  const int heavy = t.nrt > 1 ? INT_MAX : kStepHeavy;
  KernelTimer timer(kernel_ms, K, s);
  for (int j = 0; j < K; ++j) {
    timer.mark(0, j, 0);
    if (valc)
      step_spmm_kernel<T, true><<<grid, block, red, s>>>(n, h->row_ptr, h->col, vals, R, group, heavy, Wc, Wb, pa, pb, beta, K, j,
                                                         k_max, status);
    else
      step_spmm_kernel<T, false><<<grid, block, red, s>>>(n, h->row_ptr, h->col, vals, R, group, heavy, Wc, Wb, pa, pb, beta, K, j,
                                                          k_max, status);
    note_launch();
    timer.mark(0, j, 1);
    timer.mark(1, j, 0);
    const dim3 ugrid(j + 1 < K ? t.nrb : 1, t.nrt);  // the last step only adds up alpha
    step_update_kernel<T><<<ugrid, block, red, s>>>(n, R, Wb, Wc, Wp, pa, t.nrb, beta, alpha, K, j, pb);
    note_launch();
    timer.mark(1, j, 1);
    if ((rc = check_launch())) return rc;
    std::swap(Wc, Wp);
  }
  timer.finish(K);
  return EDGPU_OK;
}

// The milliseconds of what run() launches into kernel_ms[0] (the others 0) where kernel_ms is given.
template <typename F>
auto timed_whole(double* kernel_ms, cudaStream_t s, F&& run) {
  if (!kernel_ms) return run();
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, s);
  const auto rc = run();
  cudaEventRecord(e1, s);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  kernel_ms[0] = ms;
  kernel_ms[1] = kernel_ms[2] = 0.0;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return rc;
}

// Sectors beyond one SM's shared memory, the same for the timed entry point and the plain one: a timed run
// has the other's bits, and its time is of the kernels that the other runs.
static int lanczos_large(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K, int precision,
                         double* alpha, double* beta, int32_t* status, unsigned char* ws, size_t ws_bytes,
                         cudaStream_t s, double* kernel_ms = nullptr) {
  if (precision != 0) return lanczos_impl<float>(h, v0, R, k_max, K, alpha, beta, status, ws, ws_bytes, s, kernel_ms);
  if (timed_whole(kernel_ms, s, [&] { return launch_grid(h, v0, R, k_max, K, alpha, beta, status, ws, s); }))
    return check_launch();
  return lanczos_impl<double>(h, v0, R, k_max, K, alpha, beta, status, ws, ws_bytes, s, kernel_ms);
}

}  // namespace edgpu

using namespace edgpu;

extern "C" int edgpu_spmv(const edgpu_csr* h, const double* x, double* y, int R, void* stream) {
  if (!h || !x || !y || R < 1 || h->n < 0) return EDGPU_ERR_ARG;
  if (!h->val_c && !h->val_r) return EDGPU_ERR_ARG;
  if (h->n == 0) return EDGPU_OK;
  return launch_rows<double, 1>(h, h->val_c, h->val_r, 0.0, reinterpret_cast<const double2*>(x),
                                reinterpret_cast<double2*>(y), R, (cudaStream_t)stream);
}

extern "C" int edgpu_spmv_shift_c64(const edgpu_csr* h, float shift, const float* x, float* y, int R, void* stream) {
  if (!h || !x || !y || R < 1 || h->n < 0) return EDGPU_ERR_ARG;
  if (!h->val_cf && !h->val_rf) return EDGPU_ERR_ARG;
  if (h->n == 0) return EDGPU_OK;
  const float2* xc = reinterpret_cast<const float2*>(x);
  float2* yc = reinterpret_cast<float2*>(y);
  // two runs a thread; one where their number is odd or a pair is not 16 bytes aligned
  if (R % 2 == 0 && spmv_aligned(x, y))
    return launch_rows<float, 2>(h, h->val_cf, h->val_rf, shift, xc, yc, R, (cudaStream_t)stream);
  return launch_rows<float, 1>(h, h->val_cf, h->val_rf, shift, xc, yc, R, (cudaStream_t)stream);
}

extern "C" int edgpu_spmv_c64(const edgpu_csr* h, const float* x, float* y, int R, void* stream) {
  return edgpu_spmv_shift_c64(h, 0.f, x, y, R, stream);
}

extern "C" size_t edgpu_lanczos_workspace(int64_t n, int R, int K, int precision) {
  (void)K;
  const size_t vs = precision == 1 ? sizeof(float2) : sizeof(double2);
  RunTile t = make_tile(n > 0 ? n : 1, R > 0 ? R : 1);
  size_t b = 0;
  for (int k = 0; k < 3; ++k) b += ((vs * (size_t)n * R) + 255) & ~(size_t)255;
  b += 2 * (((sizeof(double) * (size_t)t.nrb * R) + 255) & ~(size_t)255);
  return b + 256;
}

// The df64 form (precision 3) exists for real H in the shared-memory path; everything else
// it asks for runs in FP64.
static int effective_precision(const edgpu_csr* h, int precision) {
  if (precision != 3) return precision;
  return (h->val_df && !h->val_c && small_fits(h->n, 3)) ? 3 : 0;
}

extern "C" int edgpu_lanczos(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K, int precision,
                             double* alpha, double* beta, int32_t* status_dev, void* workspace, size_t workspace_bytes,
                             void* stream) {
  if (!h || !v0 || R < 1 || K < 1 || !k_max || !alpha || !beta || !status_dev || h->n < 1) return EDGPU_ERR_ARG;
  if (precision < 0 || precision > 3 || precision == 2) return EDGPU_ERR_ARG;
  precision = effective_precision(h, precision);
  if (workspace_bytes < edgpu_lanczos_workspace(h->n, R, K, precision)) return EDGPU_ERR_WORKSPACE;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  if (small_fits(h->n, precision))
    return lanczos_small(h, v0, R, k_max, K, precision, alpha, beta, status_dev, ws, (cudaStream_t)stream);
  return lanczos_large(h, v0, R, k_max, K, precision, alpha, beta, status_dev, ws, workspace_bytes,
                       (cudaStream_t)stream);
}

extern "C" int edgpu_lanczos_timed(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K,
                                   int precision, double* alpha, double* beta, int32_t* status_dev, void* workspace,
                                   size_t workspace_bytes, void* stream, double* kernel_ms) {
  if (!h || !v0 || R < 1 || K < 1 || !k_max || !alpha || !beta || !status_dev || h->n < 1 || !kernel_ms)
    return EDGPU_ERR_ARG;
  if (precision < 0 || precision > 3 || precision == 2) return EDGPU_ERR_ARG;
  precision = effective_precision(h, precision);
  if (workspace_bytes < edgpu_lanczos_workspace(h->n, R, K, precision)) return EDGPU_ERR_WORKSPACE;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  cudaStream_t s = (cudaStream_t)stream;
  if (small_fits(h->n, precision))  // the whole recurrence (products, sums, updates) in one launch
    return timed_whole(kernel_ms, s, [&] {
      return lanczos_small(h, v0, R, k_max, K, precision, alpha, beta, status_dev, ws, s);
    });
  return lanczos_large(h, v0, R, k_max, K, precision, alpha, beta, status_dev, ws, workspace_bytes, s, kernel_ms);
}

namespace edgpu {
size_t reorth_coop_scratch_bytes();
int lanczos_reorth_coop(const edgpu_csr* h, const double* v0, int j0, int j1, int K_cap, double* Vd, double* wd,
                        double* alpha, double* beta, int32_t* status_dev, double* scratch, double2* hc,
                        cudaStream_t s);
}  // namespace edgpu
static std::atomic<int> g_reorth_fused{1};

extern "C" void edgpu_set_reorth_fused(int enabled) { g_reorth_fused.store(enabled ? 1 : 0); }

extern "C" size_t edgpu_lanczos_reorth_workspace(int64_t n, int K_cap) {
  const int64_t nrb = grid_1d(n > 0 ? n : 1, 256);
  size_t b = 0;
  b += sizeof(double2) * (size_t)n;                        // y
  b += sizeof(double) * (size_t)nrb * 2 + 512;             // alpha/norm partials
  b += sizeof(double2) * (size_t)(K_cap + 1) * nrb + 256;  // dot partials
  b += sizeof(double2) * (size_t)(K_cap + 1) + 256;        // h
  b += sizeof(double) * (size_t)((n + 31) / 32 + 1) + 256;  // projection-block norm partials
  b += reorth_coop_scratch_bytes() + 256;                   // per-block partials of the fused form
  return b + 1024;
}


extern "C" int edgpu_lanczos_reorth(const edgpu_csr* h, const double* v0, int j0, int j1, int K_cap, double* Vd,
                                    double* wd, double* alpha, double* beta, int32_t* status_dev, void* workspace,
                                    size_t workspace_bytes, void* stream) {
  if (!h || !Vd || !wd || !alpha || !beta || !status_dev || h->n < 1) return EDGPU_ERR_ARG;
  if (j0 < 0 || j1 > K_cap || j0 > j1) return EDGPU_ERR_ARG;
  if (j0 == 0 && !v0) return EDGPU_ERR_ARG;
  if (workspace_bytes < edgpu_lanczos_reorth_workspace(h->n, K_cap)) return EDGPU_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  if (j0 == j1) return EDGPU_OK;
  const int64_t n = h->n;
  double2* V = reinterpret_cast<double2*>(Vd);
  double2* w = reinterpret_cast<double2*>(wd);
  const unsigned nrb = grid_1d(n, 256);
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  size_t off = 0;
  auto carve = [&](size_t bytes) {
    unsigned char* p = ws + off;
    off += (bytes + 255) & ~(size_t)255;
    return p;
  };
  double* pa = reinterpret_cast<double*>(carve(sizeof(double) * nrb));
  double* pn = reinterpret_cast<double*>(carve(sizeof(double) * nrb));
  double2* pd = reinterpret_cast<double2*>(carve(sizeof(double2) * (size_t)(K_cap + 1) * nrb));
  double2* hc = reinterpret_cast<double2*>(carve(sizeof(double2) * (size_t)(K_cap + 1)));
  double* pnp = reinterpret_cast<double*>(carve(sizeof(double) * (size_t)((n + 31) / 32 + 1)));
  double* coop = reinterpret_cast<double*>(carve(reorth_coop_scratch_bytes()));
  if (off > workspace_bytes) return EDGPU_ERR_WORKSPACE;
  if (g_reorth_fused.load()) {
    const int rcc = lanczos_reorth_coop(h, v0, j0, j1, K_cap, Vd, wd, alpha, beta, status_dev, coop, hc, s);
    if (rcc >= 0) return rcc;
  }
  if (j0 == 0) {
    copy_c128_kernel<<<grid_1d(n, 256), 256, 0, s>>>(reinterpret_cast<const double2*>(v0), V, n);
    note_launch();
  }
  int rc = check_launch();
  if (rc) return rc;
  for (int j = j0; j < j1; ++j) {
    const double2* vj = V + (int64_t)j * n;
    // w = H v_j ; alpha partials
    dim3 grid(nrb, 1), block(1, 256);
    if (h->val_c)
      spmv_alpha_kernel<true><<<grid, block, sizeof(double) * 256, s>>>(n, h->row_ptr, h->col, h->val_c, vj, w, pa);
    else
      spmv_alpha_kernel<false><<<grid, block, sizeof(double) * 256, s>>>(n, h->row_ptr, h->col, h->val_r, vj, w, pa);
    note_launch();
    reorth_alpha_update_kernel<<<nrb, 256, 0, s>>>(n, w, vj, j > 0 ? V + (int64_t)(j - 1) * n : nullptr, pa, nrb,
                                                   alpha, beta, j, pn); note_launch();
    if ((rc = check_launch())) return rc;
    if (j + 1 >= K_cap) break;
    // two passes of classical Gram-Schmidt against V[0..j]; the second pass also forms the
    // per-block partial norms of the final w
    const int m = j + 1;
    const unsigned prb = (unsigned)((n + 31) / 32);
    for (int pass = 0; pass < 2; ++pass) {
      dot_per_k_kernel<<<m, 256, 0, s>>>(V, m, n, w, hc); note_launch();
      project_out_kernel<<<prb, 256, 0, s>>>(V, m, n, hc, w, pnp, pass == 1); note_launch();
    }
    reorth_normalize_kernel<<<nrb, 256, 0, s>>>(n, w, V + (int64_t)(j + 1) * n, pnp, (int)prb, beta, j, status_dev); note_launch();
    (void)pd;
    (void)pn;
    if ((rc = check_launch())) return rc;
  }
  return EDGPU_OK;
}

extern "C" int edgpu_combine(const double* V, int K, int64_t n, const double* C, int M, double* X, void* stream) {
  if (!V || !C || !X || K < 1 || M < 1 || n < 1) return EDGPU_ERR_ARG;
  dim3 grid(grid_1d(n, 256) > 64 ? 64 : grid_1d(n, 256), M);
  combine_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<const double2*>(V), K, n,
                                                        reinterpret_cast<const double2*>(C), M,
                                                        reinterpret_cast<double2*>(X)); note_launch();
  return check_launch();
}

extern "C" size_t edgpu_cfrac_f32_workspace(int K, int R) { return 2 * sizeof(float) * (size_t)K * R + 512; }

extern "C" int edgpu_cfrac_f32(const double* alpha, const double* beta, const int32_t* k_len, int K, int R,
                               const double* omega, int n_omega, double delta, const double* e, const double* scale,
                               double* g, void* workspace, size_t workspace_bytes, void* stream) {
  if (!alpha || !beta || !k_len || !omega || !e || !g || K < 1 || R < 0 || n_omega < 0) return EDGPU_ERR_ARG;
  const int64_t tot = (int64_t)R * n_omega;
  if (tot == 0) return EDGPU_OK;
  if (!workspace || workspace_bytes < edgpu_cfrac_f32_workspace(K, R)) return EDGPU_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  float* ap = reinterpret_cast<float*>(workspace);
  float* b2 = ap + (size_t)K * R;
  const int64_t tk = (int64_t)K * R;
  cfrac_prep_kernel<<<(unsigned)((tk + 255) / 256), 256, 0, s>>>(alpha, beta, k_len, K, R, e, ap, b2);
  note_launch();
  cfrac_f32_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(ap, b2, k_len, K, R, omega, n_omega, delta, scale,
                                                               reinterpret_cast<double2*>(g));
  note_launch();
  return check_launch();
}

extern "C" int edgpu_cfrac(const double* alpha, const double* beta, const int32_t* k_len, int K, int R,
                           const double* omega, int n_omega, double delta, const double* e, const double* scale,
                           double* g, void* stream) {
  if (!alpha || !beta || !k_len || !omega || !e || !g || K < 1 || R < 0 || n_omega < 0) return EDGPU_ERR_ARG;
  const int64_t tot = (int64_t)R * n_omega;
  if (tot == 0) return EDGPU_OK;
  int wt = kCfracThreads;
  while (wt > 1 && wt / 2 >= n_omega) wt >>= 1;
  const int rt = kCfracThreads / wt, tiles = (n_omega + wt - 1) / wt;
  const int64_t blocks = ((int64_t)R + rt - 1) / rt * tiles;
  if (blocks > 0x7fffffffLL) return EDGPU_ERR_ARG;
  auto kern = fabs(delta) >= kCfracMinDelta ? cfrac_kernel<true> : cfrac_kernel<false>;
  kern<<<(unsigned)blocks, kCfracThreads, 0, (cudaStream_t)stream>>>(alpha, beta, k_len, K, R, omega, n_omega, delta, e,
                                                                     scale, wt, tiles, reinterpret_cast<double2*>(g));
  note_launch();
  return check_launch();
}

// =======================================================================================
// Small sectors: one CTA per run, the whole Krylov loop in one persistent launch.
// =======================================================================================
namespace edgpu {

constexpr int kSmallThreads = 512;
constexpr int kSmallBatch = 8;  // CSR entries loaded together per row

// Deterministic block sum (fixed thread -> partial mapping and fixed tree).  The first `active`
// threads may hold a value; the other warps keep off the FP64 pipe (their sum is 0).  ROOT: one
// thread turns the sum into its root, returned instead, and red[33] into the root's reciprocal (0
// for 0 and NaN) -- by every thread of 16 warps these two took 6 400 cycles of FP64 issue.
template <bool ROOT>
__device__ __forceinline__ double block_sum(double v, double* red, int active) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (32 * warp < active) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    double t = lane < nw ? red[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) {
      if (ROOT) {
        const double b = sqrt(t);
        red[32] = b;
        red[33] = b > 0.0 ? 1.0 / b : 0.0;
      } else {
        red[32] = t;
      }
    }
  }
  __syncthreads();
  return red[32];
}

__device__ __forceinline__ double2 to_v(double2 a, double) { return a; }
__device__ __forceinline__ float2 to_v(double2 a, float) { return make_float2((float)a.x, (float)a.y); }

// Upstream's Lanczos recurrence (finite.py:1974-1992) for run r entirely in shared memory:
// x = v_j, p = v_{j-1}, y = H v_j then w.  One CTA per run, persistent over runs.
//
// Bound by FP64 issue (~16 cycles a warp instruction; two CTAs share an SM's pipe).  SLICED (real H):
// the products walk the rows by length on the sliced copy (slices_kernel), a warp's rows of nearly
// equal lengths and their entries side by side in memory, instead of 32 consecutive rows whose
// longest sets the pace (1.52 issue slots an entry on the 1770-row sector, 1.03 sliced).  Every row
// still adds its entries in their order, and alpha's per-thread sums run over the rows i = tid,
// tid + 512, ... after a barrier, so the bits are those of the unsliced form: a recurrence without
// reorthogonalisation turns rounding into visible changes.  750 runs x 150 steps of the 1770-row
// sector: 17.6 ms (19.2 from the CSR rows with the root in every thread; the 46.6 operations a row
// and step that these bits need issue in 15.9); 750 runs of a 200-row
// matrix 6.4 -> 4.3 ms, 9 runs of 600 rows 2.96 -> 2.46.
template <typename T, bool VALC, bool SLICED>
__global__ void __launch_bounds__(kSmallThreads) lanczos_small_kernel(
    int64_t n, const int64_t* __restrict__ rp, const int32_t* __restrict__ col, const T* __restrict__ vals,
    const int32_t* __restrict__ sinfo, const int32_t* __restrict__ soff, const int32_t* __restrict__ ecol,
    const T* __restrict__ eval, int R, const double2* __restrict__ v0, const int32_t* __restrict__ k_max, int K,
    double* __restrict__ alpha, double* __restrict__ beta, int32_t* status) {
  using V = typename Cx<T>::V;
  extern __shared__ __align__(16) unsigned char sm[];
  V* A = reinterpret_cast<V*>(sm);
  V* B = A + n;
  V* Cv = B + n;
  double* red = reinterpret_cast<double*>(Cv + n);
  const int tid = threadIdx.x, bs = blockDim.x;
  const int active = n < bs ? (int)n : bs;
  const bool sliced = SLICED && soff[0] >= 0;
  const int npad = (int)((n + 31) & ~(int64_t)31);
  for (int r = blockIdx.x; r < R; r += gridDim.x) {
    const int km = k_max[r];
    if (km <= 0) continue;
    for (int64_t i = tid; i < n; i += bs) {
      A[i] = to_v(v0[i * R + r], T(0));
      B[i] = to_v(make_double2(0.0, 0.0), T(0));
    }
    __syncthreads();
    V* x = A;
    V* p = B;
    V* y = Cv;
    double bprev = 0.0;
    for (int j = 0; j < km; ++j) {
      double acc = 0.0;
      if (SLICED && sliced) {
        for (int q = tid; q < npad; q += bs) {
          const int info = __ldg(sinfo + q);
          if (info < 0) continue;
          const int len = info >> 16;
          const int32_t* c = ecol + __ldg(soff + (q >> 5)) + (q & 31);
          const T* h = eval + (c - ecol);
          T yr = 0, yi = 0;
          for (int e = 0; e < len; e += kSmallBatch) {
            int cc[kSmallBatch];
            T hh[kSmallBatch];
#pragma unroll
            for (int u = 0; u < kSmallBatch; ++u) {
              const bool ok = e + u < len;
              cc[u] = ok ? __ldg(c + 32 * (e + u)) : 0;
              hh[u] = ok ? __ldg(h + 32 * (e + u)) : T(0);
            }
#pragma unroll
            for (int u = 0; u < kSmallBatch; ++u) {
              if (e + u < len) {
                const V xv = x[cc[u]];
                yr += hh[u] * xv.x;
                yi += hh[u] * xv.y;
              }
            }
          }
          V yv;
          yv.x = yr;
          yv.y = yi;
          y[info & 0xffff] = yv;
        }
        __syncthreads();
        for (int64_t i = tid; i < n; i += bs) {
          const V yv = y[i], xi = x[i];
          acc += (double)yv.x * (double)xi.x + (double)yv.y * (double)xi.y;
        }
      } else {
        for (int64_t i = tid; i < n; i += bs) {
          T yr = 0, yi = 0;
          const int64_t e1 = rp[i + 1];
          for (int64_t e = rp[i]; e < e1; ++e) {
            const V xv = x[col[e]];
            if (VALC) {
              const T hr = vals[2 * e], hi = vals[2 * e + 1];
              yr += hr * xv.x - hi * xv.y;
              yi += hr * xv.y + hi * xv.x;
            } else {
              const T h = vals[e];
              yr += h * xv.x;
              yi += h * xv.y;
            }
          }
          V yv;
          yv.x = yr;
          yv.y = yi;
          y[i] = yv;
          const V xi = x[i];
          acc += (double)yr * (double)xi.x + (double)yi * (double)xi.y;
        }
      }
      const double a = block_sum<false>(acc, red, active);
      if (tid == 0) alpha[(int64_t)r * K + j] = a;
      if (j + 1 == km) break;
      acc = 0.0;
      const T af = (T)a, bf = (T)bprev;
      for (int64_t i = tid; i < n; i += bs) {
        V w = y[i];
        const V xi = x[i];
        const V pi = p[i];
        w.x = (w.x - af * xi.x) - bf * pi.x;
        w.y = (w.y - af * xi.y) - bf * pi.y;
        y[i] = w;
        acc += (double)w.x * (double)w.x + (double)w.y * (double)w.y;
      }
      const double b = block_sum<true>(acc, red, active);
      if (tid == 0) {
        beta[(int64_t)r * K + j] = b;
        if (!(b > 0.0)) atomicExch(status, (int32_t)(b == 0.0 ? EDGPU_ERR_BREAKDOWN : EDGPU_ERR_NAN));
      }
      const T inv = (T)red[33];
      for (int64_t i = tid; i < n; i += bs) {
        const V w = y[i];
        V o;
        o.x = w.x * inv;
        o.y = w.y * inv;
        p[i] = o;  // overwrite v_{j-1} with v_{j+1}
      }
      __syncthreads();
      V* t = p;
      p = x;
      x = t;
      bprev = b;
    }
    __syncthreads();
  }
}

// The double-float recurrence with one shared-memory vector per run.  The H v_j pass
// gathers x = v_j from anywhere in the sector, but every other access to a vector touches
// only the thread's own rows (i = tid, tid + THREADS, ...), so v_{j-1} lives in a per-CTA
// slice of global memory (the Lanczos workspace; each element is read and written only by
// the thread that owns its row, so no fence is needed) and only x occupies shared memory.
// Pass 1 overwrites p = v_{j-1} with H v_j - beta_{j-1} v_{j-1} while summing
// alpha_j = v_j . H v_j from the same row values; pass 2, after the SpMV of every thread
// has finished (the alpha sum's barriers), forms w = p - alpha_j v_j, moves v_j into p and
// w into x; pass 3 normalises x in place.  (The subtractions run in the order
// (H v - beta p) - alpha v instead of upstream's (H v - alpha v) - beta p, a difference at
// the 2^-48 rounding level.)  At 16 + 4 bytes per row of shared memory (vector and cached
// row pointers) five or six CTAs fit on an SM, so a batch of runs the size of a RIXS map
// (hundreds of runs) runs as one wave.  Every thread forms beta and 1/beta itself from the
// broadcast sum (double-float square root and reciprocal, a few FP32 instructions), so no
// barrier publishes them; the last thread converts alpha and beta to FP64 for the outputs.
template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) lanczos_small_df_kernel(
    int64_t n, const int64_t* __restrict__ rp, const int32_t* __restrict__ col, const float2* __restrict__ hv, int R,
    const double2* __restrict__ v0, const int32_t* __restrict__ k_max, int K, double* __restrict__ alpha,
    double* __restrict__ beta, int32_t* status, float4* __restrict__ pbuf) {
  // vectors as float4 (re.hi, im.hi, re.lo, im.lo): .xy and .zw are the packed high and
  // low parts that the float2 instructions take directly
  extern __shared__ __align__(16) unsigned char sm[];
  float4* x = reinterpret_cast<float4*>(sm);
  dfl* red = reinterpret_cast<dfl*>(x + n);                // two reduction buffers
  int32_t* srp = reinterpret_cast<int32_t*>(red + kDfRed);  // row pointers, cached once
  float4* __restrict__ p = pbuf + (size_t)blockIdx.x * (size_t)n;
  constexpr int NW = THREADS / 32;
  const int tid = threadIdx.x;
  const dfl zero = {0.f, 0.f};
  for (int64_t i = tid; i <= n; i += THREADS) srp[i] = (int32_t)rp[i];
  for (int r = blockIdx.x; r < R; r += gridDim.x) {
    const int km = k_max[r];
    if (km <= 0) continue;
    for (int64_t i = tid; i < n; i += THREADS) {
      const double2 v = v0[i * R + r];
      const dfl re = df_split(v.x), im = df_split(v.y);
      x[i] = make_float4(re.hi, im.hi, re.lo, im.lo);
      p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    dfl bprev = zero;
    for (int j = 0; j < km; ++j) {
      const dfl nb = {-bprev.hi, -bprev.lo};
      dacc2 acc = {{0.f, 0.f}, {0.f, 0.f}};
      for (int64_t i = tid; i < n; i += THREADS) {
        const float4 pi = p[i];  // issued before the row's products, used after them
        dacc2 y = {{0.f, 0.f}, {0.f, 0.f}};
        const int e1 = srp[i + 1];
        for (int e = srp[i]; e < e1; e += kSmallBatch) {
          int c[kSmallBatch];
          float2 hh[kSmallBatch];
#pragma unroll
          for (int u = 0; u < kSmallBatch; ++u) {
            const bool ok = e + u < e1;
            c[u] = ok ? __ldg(col + e + u) : 0;
            hh[u] = ok ? __ldg(hv + e + u) : make_float2(0.f, 0.f);
          }
#pragma unroll
          for (int u = 0; u < kSmallBatch; ++u) {
            if (e + u < e1) {
              const float4 xv = x[c[u]];
              dacc2_fma(y, {hh[u].x, hh[u].y}, make_float2(xv.x, xv.y), make_float2(xv.z, xv.w));
            }
          }
        }
        const dfl2 h = dacc2_val(y);
        const float4 xi = x[i];
        dacc2_fma2(acc, h, make_float2(xi.x, xi.y), make_float2(xi.z, xi.w));
        const dfl2 w = df2_fma_s(h, {make_float2(pi.x, pi.y), make_float2(pi.z, pi.w)}, nb);
        p[i] = make_float4(w.hi.x, w.hi.y, w.lo.x, w.lo.y);
      }
      const dfl a = df_block_sum2<NW>(dacc2_total(acc), red);
      if (tid == THREADS - 1) alpha[(int64_t)r * K + j] = df_val(a);
      if (j + 1 == km) break;
      const dfl na = {-a.hi, -a.lo};
      acc = {{0.f, 0.f}, {0.f, 0.f}};
      for (int64_t i = tid; i < n; i += THREADS) {
        const float4 wv = p[i], xi = x[i];
        const dfl2 w = df2_fma_s({make_float2(wv.x, wv.y), make_float2(wv.z, wv.w)},
                                 {make_float2(xi.x, xi.y), make_float2(xi.z, xi.w)}, na);
        p[i] = xi;  // v_j: the next step's v_{j-1}
        x[i] = make_float4(w.hi.x, w.hi.y, w.lo.x, w.lo.y);
        dacc2_fma2(acc, w, w.hi, w.lo);
      }
      bprev = df_sqrt(df_block_sum2<NW>(dacc2_total(acc), red + 40));
      const dfl ib = bprev.hi > 0.f ? df_rcp(bprev) : zero;
      if (tid == THREADS - 1) {
        const double b = df_val(bprev);
        beta[(int64_t)r * K + j] = b;
        if (!(b > 0.0)) atomicExch(status, (int32_t)(b == 0.0 ? EDGPU_ERR_BREAKDOWN : EDGPU_ERR_NAN));
      }
      for (int64_t i = tid; i < n; i += THREADS) {
        const float4 wv = x[i];
        const dfl2 v = df2_mul_s({make_float2(wv.x, wv.y), make_float2(wv.z, wv.w)}, ib);
        x[i] = make_float4(v.hi.x, v.hi.y, v.lo.x, v.lo.y);
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

// Sliced layout of a CSR matrix for the one-CTA-per-run double-float Lanczos.  Rows are
// ordered by length, longest first (a stable counting sort, so equal lengths keep their
// order), and cut into slices of 32 consecutive slots, one slice per warp iteration; slice q
// stores entry e of its lane-th row at soff[q] + 32 e + lane, padded to the slice's longest
// row, so that a warp's loads of the e-th entries of its 32 rows are one contiguous 128-byte
// (columns) and 256-byte (values) line, and the rows of a warp have nearly equal lengths.
// sinfo[slot] = row | (length << 16), or -1 for the padding slots after the last row; the
// stored columns are slots too (the slot that holds the column's row), so the Lanczos kernel
// keeps its vector in slot order and touches a warp's own rows contiguously.
// Built by one CTA: the counting sort's histogram with atomics (order-free), the stable
// placement by warp 0 with __match_any_sync ranks, then the fill by every thread.  When the
// slices would need more than `cap` entries (possible only for rows with repeated columns)
// every slot gets length 0 and *status EDGPU_ERR_WORKSPACE, so nothing reads past the arrays.
// SLOTS = false (the FP64 kernel, which keeps its vectors in row order): stored columns are rows, and
// where the slices do not fit soff[0] becomes -1 and the caller's kernel reads the CSR arrays.
template <typename E, bool SLOTS>
__global__ void __launch_bounds__(1024) slices_kernel(int64_t n, const int64_t* __restrict__ rp,
                                                      const int32_t* __restrict__ col, const E* __restrict__ hv,
                                                      int32_t* __restrict__ sinfo, int32_t* __restrict__ soff,
                                                      int32_t* __restrict__ ecol, E* __restrict__ eval, int64_t cap,
                                                      int32_t* status) {
  extern __shared__ int32_t hist[];  // [n + 1] bucket offsets (row lengths 0..n)
  __shared__ int32_t s_max;
  __shared__ int32_t s_over;
  const int tid = threadIdx.x;
  const int npad = (int)((n + 31) & ~(int64_t)31), nslices = npad >> 5;
  if (tid == 0) {
    s_max = 0;
    s_over = 0;
  }
  __syncthreads();
  int lmax = 0;
  for (int64_t i = tid; i < n; i += blockDim.x) lmax = max(lmax, (int)(rp[i + 1] - rp[i]));
  atomicMax(&s_max, lmax);
  __syncthreads();
  if (!SLOTS && s_max > n) {
    if (tid == 0) soff[0] = -1;
    return;
  }
  if (s_max > n) {  // repeated columns: no sliced layout
    for (int q = tid; q < npad; q += blockDim.x) sinfo[q] = q < n ? q : -1;
    for (int q = tid; q <= nslices; q += blockDim.x) soff[q] = 0;
    if (tid == 0) atomicExch(status, (int32_t)EDGPU_ERR_WORKSPACE);
    return;
  }
  const int L = s_max;
  for (int k = tid; k <= L; k += blockDim.x) hist[k] = 0;
  __syncthreads();
  for (int64_t i = tid; i < n; i += blockDim.x) atomicAdd(&hist[L - (int)(rp[i + 1] - rp[i])], 1);
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int k = 0; k <= L; ++k) {
      const int c = hist[k];
      hist[k] = run;
      run += c;
    }
  }
  __syncthreads();
  if (tid < 32) {
    const unsigned lt = (1u << tid) - 1u;
    for (int64_t c0 = 0; c0 < n; c0 += 32) {
      const int64_t i = c0 + tid;
      const int len = i < n ? (int)(rp[i + 1] - rp[i]) : 0;
      const int key = i < n ? L - len : -1;
      const unsigned same = __match_any_sync(0xffffffffu, key);
      const int base = key >= 0 ? hist[key] : 0;
      if (i < n) sinfo[base + __popc(same & lt)] = (int32_t)i | (len << 16);
      __syncwarp();
      if (key >= 0 && (__ffs(same) - 1) == tid) hist[key] = base + __popc(same);
      __syncwarp();
    }
  }
  for (int q = (int)n + tid; q < npad; q += blockDim.x) sinfo[q] = -1;
  __syncthreads();
  // the bucket offsets are spent: hist becomes the slot of each row
  for (int q = tid; q < (int)n; q += blockDim.x) hist[sinfo[q] & 0xffff] = q;
  __syncthreads();
  if (tid == 0) {
    int64_t off = 0;
    soff[0] = 0;
    for (int q = 0; q < nslices; ++q) {
      off += 32 * (int64_t)(sinfo[32 * q] >> 16);  // the slice's first row is its longest
      soff[q + 1] = (int32_t)off;
    }
    if (off > cap) s_over = 1;
  }
  __syncthreads();
  if (!SLOTS && s_over) {
    if (tid == 0) soff[0] = -1;
    return;
  }
  if (s_over) {
    for (int q = tid; q < npad; q += blockDim.x) sinfo[q] = sinfo[q] < 0 ? -1 : (sinfo[q] & 0xffff);
    for (int q = tid; q <= nslices; q += blockDim.x) soff[q] = 0;
    if (tid == 0) atomicExch(status, (int32_t)EDGPU_ERR_WORKSPACE);
    return;
  }
  for (int q = tid; q < npad; q += blockDim.x) {
    const int info = sinfo[q];
    const int sl = q >> 5;
    const int m = (soff[sl + 1] - soff[sl]) >> 5;
    const int64_t base = soff[sl] + (q & 31);
    const int len = info < 0 ? 0 : (info >> 16);
    const int64_t e0 = info < 0 ? 0 : rp[info & 0xffff];
    for (int e = 0; e < m; ++e) {
      ecol[base + 32 * e] = e < len ? (SLOTS ? hist[col[e0 + e]] : col[e0 + e]) : 0;
      eval[base + 32 * e] = e < len ? hv[e0 + e] : E{};
    }
  }
}

// Entries the sliced layout can need: every slice but the first is no wider than the
// shortest row of the slice before it, so the padding beyond nnz is at most 32 times the
// longest row, itself at most n for rows without repeated columns.
static int64_t df_slices_cap(int64_t n, int64_t nnz) { return nnz + 32 * n; }

// lanczos_small_df_kernel on the sliced layout: thread tid walks the slots tid, tid +
// THREADS, ... (a warp takes whole slices), so its rows and their order follow the slots;
// both vectors are kept in slot order (the stored columns are slots), so every access but
// the H v gathers is contiguous.  The arithmetic of every row and vector element is that of
// lanczos_small_df_kernel; only the rows' assignment to threads, and so the order of the
// per-thread partial sums of alpha and beta, differ.
template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) lanczos_sliced_df_kernel(
    int64_t n, const int32_t* __restrict__ g_sinfo, const int32_t* __restrict__ g_soff,
    const int32_t* __restrict__ ecol, const float2* __restrict__ eval, int R, const double2* __restrict__ v0,
    const int32_t* __restrict__ k_max, int K, double* __restrict__ alpha, double* __restrict__ beta, int32_t* status,
    float4* __restrict__ pbuf) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int npad = (int)((n + 31) & ~(int64_t)31), nslices = npad >> 5;
  float4* x = reinterpret_cast<float4*>(sm);  // in slot order, zero in the padding slots
  dfl* red = reinterpret_cast<dfl*>(x + npad);
  int32_t* sinfo = reinterpret_cast<int32_t*>(red + kDfRed);
  int32_t* soff = sinfo + npad;
  float4* __restrict__ p = pbuf + (size_t)blockIdx.x * (size_t)npad;
  constexpr int NW = THREADS / 32;
  const int tid = threadIdx.x;
  const dfl zero = {0.f, 0.f};
  for (int q = tid; q < npad; q += THREADS) sinfo[q] = g_sinfo[q];
  for (int q = tid; q <= nslices; q += THREADS) soff[q] = g_soff[q];
  for (int r = blockIdx.x; r < R; r += gridDim.x) {
    const int km = k_max[r];
    if (km <= 0) continue;
    for (int q = tid; q < npad; q += THREADS) {
      const int info = sinfo[q];
      float4 xv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (info >= 0) {
        const double2 v = v0[(int64_t)(info & 0xffff) * R + r];
        const dfl re = df_split(v.x), im = df_split(v.y);
        xv = make_float4(re.hi, im.hi, re.lo, im.lo);
      }
      x[q] = xv;
      p[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    dfl bprev = zero;
    for (int j = 0; j < km; ++j) {
      const dfl nb = {-bprev.hi, -bprev.lo};
      dacc2 acc = {{0.f, 0.f}, {0.f, 0.f}};
      for (int q = tid; q < npad; q += THREADS) {
        const int info = sinfo[q];
        if (info < 0) continue;
        const float4 pq = p[q];
        const int len = info >> 16;
        const int64_t base = soff[q >> 5] + (q & 31);
        dacc2 y = {{0.f, 0.f}, {0.f, 0.f}};
        for (int e = 0; e < len; e += kSmallBatch) {
          int c[kSmallBatch];
          float2 hh[kSmallBatch];
#pragma unroll
          for (int u = 0; u < kSmallBatch; ++u) {
            const bool ok = e + u < len;
            c[u] = ok ? __ldg(ecol + base + 32 * (e + u)) : 0;
            hh[u] = ok ? __ldg(eval + base + 32 * (e + u)) : make_float2(0.f, 0.f);
          }
#pragma unroll
          for (int u = 0; u < kSmallBatch; ++u) {
            if (e + u < len) {
              const float4 xv = x[c[u]];
              dacc2_fma(y, {hh[u].x, hh[u].y}, make_float2(xv.x, xv.y), make_float2(xv.z, xv.w));
            }
          }
        }
        const dfl2 h = dacc2_val(y);
        const float4 xi = x[q];
        dacc2_fma2(acc, h, make_float2(xi.x, xi.y), make_float2(xi.z, xi.w));
        const dfl2 w = df2_fma_s(h, {make_float2(pq.x, pq.y), make_float2(pq.z, pq.w)}, nb);
        p[q] = make_float4(w.hi.x, w.hi.y, w.lo.x, w.lo.y);
      }
      const dfl a = df_block_sum2<NW>(dacc2_total(acc), red);
      if (tid == THREADS - 1) alpha[(int64_t)r * K + j] = df_val(a);
      if (j + 1 == km) break;
      const dfl na = {-a.hi, -a.lo};
      acc = {{0.f, 0.f}, {0.f, 0.f}};
      for (int q = tid; q < npad; q += THREADS) {
        if (sinfo[q] < 0) continue;
        const float4 wv = p[q], xi = x[q];
        const dfl2 w = df2_fma_s({make_float2(wv.x, wv.y), make_float2(wv.z, wv.w)},
                                 {make_float2(xi.x, xi.y), make_float2(xi.z, xi.w)}, na);
        p[q] = xi;  // v_j: the next step's v_{j-1}
        x[q] = make_float4(w.hi.x, w.hi.y, w.lo.x, w.lo.y);
        dacc2_fma2(acc, w, w.hi, w.lo);
      }
      bprev = df_sqrt(df_block_sum2<NW>(dacc2_total(acc), red + 40));
      const dfl ib = bprev.hi > 0.f ? df_rcp(bprev) : zero;
      if (tid == THREADS - 1) {
        const double b = df_val(bprev);
        beta[(int64_t)r * K + j] = b;
        if (!(b > 0.0)) atomicExch(status, (int32_t)(b == 0.0 ? EDGPU_ERR_BREAKDOWN : EDGPU_ERR_NAN));
      }
      for (int q = tid; q < npad; q += THREADS) {  // the padding slots stay zero
        const float4 wv = x[q];
        const dfl2 v = df2_mul_s({make_float2(wv.x, wv.y), make_float2(wv.z, wv.w)}, ib);
        x[q] = make_float4(v.hi.x, v.hi.y, v.lo.x, v.lo.y);
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

static size_t sliced_df_smem_bytes(int64_t n) {
  const int64_t npad = (n + 31) & ~(int64_t)31;
  return sizeof(float4) * (size_t)npad + kDfRed * sizeof(dfl) + sizeof(int32_t) * (size_t)(npad + npad / 32 + 1) + 16;
}

// Shared memory that decides whether a sector takes the one-CTA-per-run path (unchanged by
// the one-vector form of the double-float kernel, so that the same sectors take it).
size_t small_smem_bytes(int64_t n, int precision) {
  if (precision == 3)
    return 2 * sizeof(float4) * (size_t)n + kDfRed * sizeof(dfl) + sizeof(int32_t) * (size_t)(n + 1) + 16;
  const size_t v = precision == 1 ? sizeof(float2) : sizeof(double2);
  return 3 * v * (size_t)n + 68 * sizeof(double) + 16;
}

// Shared memory of one lanczos_small_df_kernel CTA: x, the reduction buffers, row pointers.
static size_t small_df_smem_bytes(int64_t n) {
  return sizeof(float4) * (size_t)n + kDfRed * sizeof(dfl) + sizeof(int32_t) * (size_t)(n + 1) + 16;
}

bool small_fits(int64_t n, int precision) { return small_smem_bytes(n, precision) <= 200 * 1024; }

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Entries the sliced copy of a real H is given in the FP64 form's workspace (beside its slot table);
// 0 where the smallest workspace edgpu_lanczos accepts for (n, R) cannot hold it, and for calls of
// fewer than eight steps a CTA slot, which do not repay the one-CTA launch that makes the copy:
// 152 runs of 1770 rows take 193 us sliced and 166 from the CSR rows at 2 steps, 434 and 447 at 8,
// 933 and 998 at 20; 750 runs of 2 steps 414 and 451.
static int64_t fp64_slices_cap(int64_t n, int64_t nnz, int R, int K) {
  const int64_t npad = (n + 31) & ~(int64_t)31, cap = nnz + nnz / 4 + 32 * 64;
  const size_t need = 256 + align256(4 * (size_t)npad) + align256(4 * (size_t)(npad / 32 + 1)) + align256(4 * (size_t)cap) +
                      align256(8 * (size_t)cap);
  const int64_t waves = (R + grid_cap() - 1) / grid_cap();
  return waves * K >= 8 && need <= 3 * sizeof(double2) * (size_t)n * R ? cap : 0;
}

template <typename T, bool VALC>
int launch_small(const edgpu_csr* h, const T* vals, const double* v0, int R, const int32_t* k_max, int K,
                 double* alpha, double* beta, int32_t* status, int precision, void* ws, cudaStream_t s) {
  const int64_t n = h->n;
  const size_t smem = small_smem_bytes(n, precision);
  int32_t *sinfo = nullptr, *soff = nullptr, *ecol = nullptr;
  T* eval = nullptr;
  auto kern = lanczos_small_kernel<T, VALC, false>;
  if constexpr (sizeof(T) == 8 && !VALC) {
    const int64_t cap = ws ? fp64_slices_cap(n, h->nnz, R, K) : 0;
    if (cap > 0) {
      unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
      const int64_t npad = (n + 31) & ~(int64_t)31;
      eval = reinterpret_cast<T*>(base);
      ecol = reinterpret_cast<int32_t*>(base + align256(8 * (size_t)cap));
      sinfo = reinterpret_cast<int32_t*>(reinterpret_cast<unsigned char*>(ecol) + align256(4 * (size_t)cap));
      soff = reinterpret_cast<int32_t*>(reinterpret_cast<unsigned char*>(sinfo) + align256(4 * (size_t)npad));
      const size_t hist_bytes = sizeof(int32_t) * (size_t)(n + 1);
      auto slices = slices_kernel<double, false>;
      cudaFuncSetAttribute(slices, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist_bytes);
      slices<<<1, 1024, hist_bytes, s>>>(n, h->row_ptr, h->col, vals, sinfo, soff, ecol, eval, cap, status);
      note_launch();
      kern = lanczos_small_kernel<T, VALC, true>;
    }
  }
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSmallThreads, smem);
  if (per_sm < 1) per_sm = 1;
  int grid = grid_cap() * per_sm;
  if (grid > R) grid = R;
  kern<<<grid, kSmallThreads, smem, s>>>(n, h->row_ptr, h->col, vals, sinfo, soff, ecol, eval, R,
                                         reinterpret_cast<const double2*>(v0), k_max, K, alpha, beta, status);
  note_launch();
  return check_launch();
}

// CTA slots per SM that the one-CTA-per-run double-float Lanczos leaves free (process-wide,
// default 0), so that kernels of a pipeline running concurrently on another stream find room
// on every SM instead of waiting for the persistent grid to drain.
static std::atomic<int> g_small_reserve{0};
extern "C" void edgpu_set_small_reserve(int slots) { g_small_reserve.store(slots > 0 ? slots : 0); }

// CTA size: the largest of 512, 256, 192, 160 and 128 threads (64 registers a thread at the
// occupancy each is compiled for) whose CTAs cover the R runs in the fewest waves with one
// slot per SM kept back.  It depends only on (n, R) and the GPU, never on the reserve, so a
// run's reduction order, and its result bits, do not change with concurrent work; the
// reserve only limits how many of the CTAs are resident at once.  On the 1770-row RIXS
// final-state sector with 750 runs this is 160 threads, five CTAs per SM, one wave.
// The sliced layout is used when the smallest workspace edgpu_lanczos accepts for (n, R, K)
// holds it next to the per-CTA vectors (a function of the problem only, so a given problem
// always takes the same path); otherwise the kernel reads the CSR arrays directly.
using SmallDfKern = void (*)(int64_t, const int64_t*, const int32_t*, const float2*, int, const double2*,
                             const int32_t*, int, double*, double*, int32_t*, float4*);
using SlicedDfKern = void (*)(int64_t, const int32_t*, const int32_t*, const int32_t*, const float2*, int,
                              const double2*, const int32_t*, int, double*, double*, int32_t*, float4*);
static const int kDfThreads[5] = {512, 256, 192, 160, 128};

// Process-wide CTA-size choice for the double-float one-CTA-per-run Lanczos (index into
// kDfThreads, or -1 for the rule below); set by the engine's autotuner around a call.
static std::atomic<int> g_df_cta{-1};
extern "C" void edgpu_set_lanczos_cta(int index) { g_df_cta.store(index >= 0 && index < 5 ? index : -1); }

static int pick_df_config(const void* const* kerns, size_t smem, int R, int* per_sm_out) {
  const int nsm = grid_cap();
  const int forced = g_df_cta.load();
  if (forced >= 0) {
    cudaFuncSetAttribute(kerns[forced], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kerns[forced], kDfThreads[forced], smem);
    if (per_sm >= 1) {
      *per_sm_out = per_sm;
      return forced;
    }
    cudaGetLastError();
  }
  int best = -1, best_waves = 0;
  for (int c = 0; c < 5; ++c) {
    cudaFuncSetAttribute(kerns[c], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kerns[c], kDfThreads[c], smem);
    if (per_sm < 1) continue;
    const int64_t slots = (int64_t)nsm * (per_sm > 1 ? per_sm - 1 : 1);
    const int waves = (int)((R + slots - 1) / slots);
    if (best < 0 || waves < best_waves) {
      best = c;
      best_waves = waves;
      *per_sm_out = per_sm;
    }
  }
  return best;
}

int launch_small_df(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K, double* alpha,
                    double* beta, int32_t* status, void* ws, cudaStream_t s) {
  static const SmallDfKern csr_kerns[5] = {lanczos_small_df_kernel<512, 2>, lanczos_small_df_kernel<256, 4>,
                                           lanczos_small_df_kernel<192, 5>, lanczos_small_df_kernel<160, 6>,
                                           lanczos_small_df_kernel<128, 8>};
  static const SlicedDfKern sl_kerns[5] = {lanczos_sliced_df_kernel<512, 2>, lanczos_sliced_df_kernel<256, 4>,
                                           lanczos_sliced_df_kernel<192, 5>, lanczos_sliced_df_kernel<160, 6>,
                                           lanczos_sliced_df_kernel<128, 8>};
  const int64_t n = h->n, nnz = h->nnz;
  const int64_t npad = (n + 31) & ~(int64_t)31, nslices = npad / 32;
  const int nsm = grid_cap();
  const int reserve = g_small_reserve.load();
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
  // sliced layout: per-CTA vectors, slot table, slice offsets, columns, values
  if (n <= 32767) {
    const size_t smem = sliced_df_smem_bytes(n);
    int per_sm = 1;
    const int c = pick_df_config(reinterpret_cast<const void* const*>(sl_kerns), smem, R, &per_sm);
    if (c >= 0) {
      int grid = nsm * (per_sm - reserve > 0 ? per_sm - reserve : 1);
      if (grid > R) grid = R;
      const int64_t cap = df_slices_cap(n, nnz);
      const size_t b_p = align256(sizeof(float4) * (size_t)npad * (size_t)(R < nsm * per_sm ? R : nsm * per_sm));
      const size_t b_info = align256(sizeof(int32_t) * (size_t)npad);
      const size_t b_off = align256(sizeof(int32_t) * (size_t)(nslices + 1));
      const size_t b_col = align256(sizeof(int32_t) * (size_t)cap);
      const size_t b_val = align256(sizeof(float2) * (size_t)cap);
      if (256 + b_p + b_info + b_off + b_col + b_val <= edgpu_lanczos_workspace(n, R, K, 3)) {
        float4* pbuf = reinterpret_cast<float4*>(base);
        int32_t* sinfo = reinterpret_cast<int32_t*>(base + b_p);
        int32_t* soff = reinterpret_cast<int32_t*>(base + b_p + b_info);
        int32_t* ecol = reinterpret_cast<int32_t*>(base + b_p + b_info + b_off);
        float2* eval = reinterpret_cast<float2*>(base + b_p + b_info + b_off + b_col);
        const size_t hist_bytes = sizeof(int32_t) * (size_t)(n + 1);
        auto slices = slices_kernel<float2, true>;
        cudaFuncSetAttribute(slices, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist_bytes);
        slices<<<1, 1024, hist_bytes, s>>>(n, h->row_ptr, h->col, reinterpret_cast<const float2*>(h->val_df),
                                                     sinfo, soff, ecol, eval, cap, status);
        note_launch();
        sl_kerns[c]<<<grid, kDfThreads[c], smem, s>>>(n, sinfo, soff, ecol, eval, R,
                                                       reinterpret_cast<const double2*>(v0), k_max, K, alpha, beta,
                                                       status, pbuf);
        note_launch();
        return check_launch();
      }
    }
  }
  const size_t smem = small_df_smem_bytes(n);
  int per_sm = 1;
  const int c = pick_df_config(reinterpret_cast<const void* const*>(csr_kerns), smem, R, &per_sm);
  if (c < 0) return EDGPU_ERR_ARG;
  int grid = nsm * (per_sm - reserve > 0 ? per_sm - reserve : 1);
  if (grid > R) grid = R;
  csr_kerns[c]<<<grid, kDfThreads[c], smem, s>>>(n, h->row_ptr, h->col, reinterpret_cast<const float2*>(h->val_df), R,
                                                 reinterpret_cast<const double2*>(v0), k_max, K, alpha, beta, status,
                                                 reinterpret_cast<float4*>(base));
  note_launch();
  return check_launch();
}

int lanczos_small(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K, int precision,
                  double* alpha, double* beta, int32_t* status, void* ws, cudaStream_t s) {
  if (precision == 3) {
    if (h->val_df && !h->val_c) return launch_small_df(h, v0, R, k_max, K, alpha, beta, status, ws, s);
    precision = 0;  // complex H: FP64
  }
  if (precision == 0) {
    if (h->val_c) return launch_small<double, true>(h, h->val_c, v0, R, k_max, K, alpha, beta, status, 0, ws, s);
    return launch_small<double, false>(h, h->val_r, v0, R, k_max, K, alpha, beta, status, 0, ws, s);
  }
  if (h->val_cf) return launch_small<float, true>(h, h->val_cf, v0, R, k_max, K, alpha, beta, status, 1, ws, s);
  if (!h->val_rf) return EDGPU_ERR_ARG;
  return launch_small<float, false>(h, h->val_rf, v0, R, k_max, K, alpha, beta, status, 1, ws, s);
}

// ---------------------------------------------------------------------------------------
// Shifted solves (z - H) x = y for many z from one Krylov space, CTA per right-hand side.
// The Lanczos vectors v_{j-1}, v_j and w live in shared memory; each v_j is also written to
// V[rhs][j][n] for assembling x(z) = |y| V (z - T)^{-1} e_1 afterwards.  No
// reorthogonalisation: the three-term relation H V = V T + b v e^T holds to rounding even
// after orthogonality is lost, so the residual estimate below stays valid and the loop
// simply runs until it is met.  Thread t < nz tracks shift z_t: LU pivots
// d_k = (z - a_k) - b_{k-1}^2 / d_{k-1} and the last component q_m of (z - T_m)^{-1} e_1,
// so the residual ||r|| / ||y|| = b_{m-1} |q_m| costs O(1) per step.
// Replaces upstream's per-energy BiCGSTAB (spectra.py:962,1080).
// ---------------------------------------------------------------------------------------
//
// FP64 form.  A step on one SM is bound by FP64 issue (~16 cycles a warp instruction) and its two
// sums, so what the instructions are spent on decides: rows go to the warps sorted by length (a
// warp's rows take as many entries as the longest of them), the sector's entries stay in shared
// memory where they fit (column-major slices of 32 rows), one thread takes the root and the
// reciprocal of beta (by all threads they were a quarter of the step), and the shifts' estimates
// run in warps of their own beside the next step's H v (a step past convergence does no harm: only
// the first m vectors are used).  360 rows, 15 right-hand sides, 50 shifts, ~490 steps:
// 5.52 -> 3.19 ms, 6.4 us a step, of which some 4 are FP64 issue.
constexpr int kShiftMaxThreads = 2 * kSmallThreads;

// Sum over the first `mw` warps (the others pass by), returned to every thread; red: 34 doubles.
// ROOT: red[32] becomes the root of the sum and red[33] its reciprocal (0 for 0).
template <bool ROOT>
__device__ __forceinline__ double main_sum(double v, double* red, int mw) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < mw) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
  }
  __syncthreads();
  if (warp == 0) {
    double t = lane < mw ? red[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) {
      if (ROOT) {
        const double s = sqrt(t);
        red[32] = s;
        red[33] = s > 0.0 ? 1.0 / s : 0.0;
      } else {
        red[32] = t;
      }
    }
  }
  __syncthreads();
  return red[32];
}

struct ShiftedArgs {
  int64_t n;
  const int64_t* rp;
  const int32_t* col;
  const double* vals;
  int n_rhs;
  const double2 *Y, *zs;
  int nz, k_cap;
  double tol;
  double2* V;
  double *alpha, *beta;
  int32_t* m_out;
  double* ynorm;
  int32_t* status;
  int main_threads;  // the others track the shifts
  int ent_cap;       // entries of the sliced copy that fit in shared memory
};

template <bool VALC>
__global__ void __launch_bounds__(kShiftMaxThreads) shifted_small_kernel(ShiftedArgs g) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int n = (int)g.n, M = g.main_threads, mw = M >> 5, nz = g.nz, k_cap = g.k_cap;
  const int npad = (n + 31) & ~31, slices = npad >> 5;
  double2* X = reinterpret_cast<double2*>(sm);
  double2* P = X + n;
  double2* Wv = P + n;
  double* red = reinterpret_cast<double*>(Wv + n);  // [34]
  double* sval = red + 34;
  uint16_t* scol = reinterpret_cast<uint16_t*>(sval + (size_t)g.ent_cap * (VALC ? 2 : 1));
  uint16_t* order = scol + g.ent_cap;               // [npad] row of each slot, 0xFFFF past the last
  uint16_t* len = order + npad;                     // [npad]
  __shared__ int soff[140];                         // slice starts in the copy
  __shared__ int sliced;
  const int tid = threadIdx.x, bs = blockDim.x;
  const bool is_main = tid < M;
  // rows by length, longest first, equal lengths in order
  for (int i = tid; i < n; i += bs) {
    const int64_t l = g.rp[i + 1] - g.rp[i];
    len[i] = (uint16_t)(l < 0xFFFF ? l : 0xFFFF);
  }
  for (int i = n + tid; i < npad; i += bs) {
    len[i] = 0;
    order[i] = 0xFFFF;
  }
  __syncthreads();
  for (int i = tid; i < n; i += bs) {
    const int l = len[i];
    int rank = 0;
    for (int q = 0; q < n; ++q) rank += len[q] > l || (len[q] == l && q < i);
    order[rank] = (uint16_t)i;
  }
  __syncthreads();
  if (tid == 0) {
    int at = 0;
    for (int q = 0; q < slices; ++q) {
      soff[q] = at;
      at += 32 * (int)len[order[32 * q]];
    }
    soff[slices] = at;
    sliced = at <= g.ent_cap;
  }
  __syncthreads();
  if (sliced) {
    for (int q = tid; q < npad; q += bs) {
      const int row = order[q], s = q >> 5, width = (soff[s + 1] - soff[s]) >> 5;
      const int l = row == 0xFFFF ? 0 : len[row];
      const int64_t e0 = row == 0xFFFF ? 0 : g.rp[row];
      for (int e = 0; e < width; ++e) {
        const int at = soff[s] + 32 * e + (q & 31);
        scol[at] = e < l ? (uint16_t)g.col[e0 + e] : 0;
        if (VALC) {
          sval[2 * at] = e < l ? g.vals[2 * (e0 + e)] : 0.0;
          sval[2 * at + 1] = e < l ? g.vals[2 * (e0 + e) + 1] : 0.0;
        } else {
          sval[at] = e < l ? g.vals[e0 + e] : 0.0;
        }
      }
    }
  }
  __syncthreads();
  for (int r = blockIdx.x; r < g.n_rhs; r += gridDim.x) {
    double2* Vr = g.V + (size_t)r * k_cap * n;
    const double2* y = g.Y + (size_t)r * n;
    double acc = 0.0;
    if (is_main)
      for (int i = tid; i < n; i += M) acc = fma(y[i].y, y[i].y, fma(y[i].x, y[i].x, acc));
    __syncthreads();  // red is free
    const double yn = main_sum<true>(acc, red, mw);
    const double iyn = red[33];
    if (tid == 0) g.ynorm[r] = yn;
    if (!(yn > 0.0)) {
      if (tid == 0) g.m_out[r] = 0;
      __syncthreads();
      continue;
    }
    if (is_main)
      for (int i = tid; i < n; i += M) {
        const double2 v = make_double2(y[i].x * iyn, y[i].y * iyn);
        X[i] = v;
        P[i] = make_double2(0.0, 0.0);
        Vr[i] = v;
      }
    __syncthreads();
    double2* x = X;
    double2* p = P;
    const int tz = tid - M;
    double2 z = make_double2(0.0, 0.0), id = make_double2(0.0, 0.0), q = make_double2(1.0, 0.0);
    if (tz >= 0 && tz < nz) z = g.zs[(size_t)r * nz + tz];
    // the shift's pivot and residual estimate for step k, from alpha_k, beta_{k-1} and beta_k
    auto track = [&](int k, double a, double b0, double b1) -> bool {
      if (tz < 0 || tz >= nz) return true;
      double2 d = make_double2(z.x - a, z.y), qn = make_double2(1.0, 0.0);
      if (k > 0) {
        const double b2 = b0 * b0;
        d.x -= b2 * id.x;
        d.y -= b2 * id.y;
        qn = make_double2(q.x * b0, q.y * b0);
      }
      const double rd = 1.0 / (d.x * d.x + d.y * d.y);
      id = make_double2(d.x * rd, -d.y * rd);
      q = make_double2(qn.x * id.x - qn.y * id.y, qn.x * id.y + qn.y * id.x);
      return b1 * sqrt(q.x * q.x + q.y * q.y) <= g.tol;
    };
    double a = 0.0, b = 0.0, bprev = 0.0;  // alpha_{j-1}, beta_{j-1}, beta_{j-2} at the top of step j
    int m = k_cap;
    for (int j = 0;; ++j) {
      bool ok = j > 0;
      acc = 0.0;
      if (is_main) {
        if (j < k_cap)
          for (int s = tid; s < npad; s += M) {
            const int row = order[s];
            if (row == 0xFFFF) continue;
            const int l = len[row];
            double yr = 0.0, yi = 0.0;
            if (sliced) {
              const int base = soff[s >> 5] + (s & 31);
#pragma unroll 4
              for (int e = 0; e < l; ++e) {
                const int at = base + 32 * e;
                const double2 xv = x[scol[at]];
                const double hr = sval[VALC ? 2 * at : at];
                yr = fma(hr, xv.x, yr);
                yi = fma(hr, xv.y, yi);
                if (VALC) {
                  const double hi = sval[2 * at + 1];
                  yr = fma(-hi, xv.y, yr);
                  yi = fma(hi, xv.x, yi);
                }
              }
            } else {
              const int64_t e1 = g.rp[row + 1];
#pragma unroll 4
              for (int64_t e = g.rp[row]; e < e1; ++e) {
                const double2 xv = x[g.col[e]];
                const double hr = g.vals[VALC ? 2 * e : e];
                yr = fma(hr, xv.x, yr);
                yi = fma(hr, xv.y, yi);
                if (VALC) {
                  const double hi = g.vals[2 * e + 1];
                  yr = fma(-hi, xv.y, yr);
                  yi = fma(hi, xv.x, yi);
                }
              }
            }
            Wv[row] = make_double2(yr, yi);
            acc = fma(yi, x[row].y, fma(yr, x[row].x, acc));
          }
      } else if (j > 0) {
        ok = track(j - 1, a, bprev, b);
      }
      const bool conv = __syncthreads_and(ok);
      if (conv || j == k_cap) {  // step j - 1 was the last
        m = j;
        if (tid == 0 && !conv) atomicExch(g.status, (int32_t)EDGPU_ERR_NOCONV);
        break;
      }
      bprev = b;
      a = main_sum<false>(acc, red, mw);
      if (tid == 0) g.alpha[(size_t)r * k_cap + j] = a;
      acc = 0.0;
      if (is_main)
        for (int i = tid; i < n; i += M) {
          double2 t = Wv[i];
          const double2 c = x[i], pv = p[i];
          t.x = fma(-bprev, pv.x, fma(-a, c.x, t.x));
          t.y = fma(-bprev, pv.y, fma(-a, c.y, t.y));
          Wv[i] = t;
          acc = fma(t.y, t.y, fma(t.x, t.x, acc));
        }
      __syncthreads();  // red is free
      b = main_sum<true>(acc, red, mw);
      const double ib = red[33];
      if (tid == 0) g.beta[(size_t)r * k_cap + j] = b;
      if (!(b > 0.0)) {  // the space is exhausted, or a NaN
        m = j + 1;
        if (tid == 0 && !(b >= 0.0)) atomicExch(g.status, (int32_t)EDGPU_ERR_NAN);
        break;
      }
      if (is_main) {
        double2* vn = Vr + (size_t)(j + 1) * n;
        for (int i = tid; i < n; i += M) {
          const double2 v = make_double2(Wv[i].x * ib, Wv[i].y * ib);
          p[i] = v;  // v_{j-1} is no longer needed: its buffer becomes v_{j+1}
          if (j + 1 < k_cap) vn[i] = v;
        }
      }
      __syncthreads();
      double2* t = p;
      p = x;
      x = t;
    }
    if (tid == 0) g.m_out[r] = m;
    __syncthreads();
  }
}

// The same recurrence with a right-hand side on a cluster of 2, 4 or 8 CTAs, for calls whose
// right-hand sides leave SMs idle (15 RIXS intermediate states on 152 SMs).
//
// On one CTA a step is bound by that SM's FP64 issue (16 cycles a warp instruction, of one lane or of
// 32).  Here the rows, sorted by length, are dealt to the row CTAs one by one; every CTA keeps the whole
// vector in shared memory for its gather and sends its rows of the next one to the others
// (distributed shared memory).  Few shifts (kOwnTrackers) are tracked by a CTA of their own, more of
// them by warps of every CTA.  What is left is latency, so a step has two cluster barriers and no more:
//   1  y = H w on the unscaled w = beta_{j-1} v_j, SUB lanes a row, a component per half of them,
//      and the partials of <w, y>, a partial per warp sent to every CTA.  Meanwhile a warp of the last
//      CTA takes the root of |w|^2 and its reciprocal, and the trackers the pivots of step j - 1.
//   2  one warp adds up alpha_j while the others form v_j and y - beta_{j-1} v_{j-1}; then
//      w' = y - alpha_j v_j - beta_{j-1} v_{j-1}, sent to every row CTA, and the partials of |w'|^2,
//      sent to the last CTA.  The trackers' verdict on step j - 1 arrives with them.
// Roots and reciprocals (~1500 dependent cycles each) and the trackers' ~3000 thus stay off the
// chain.  Every warp that adds up partials takes them in the same order, so that all CTAs take identical
// branches around the barriers.
// 15 right-hand sides, 50 shifts, ~480 steps: 360 states (15 RIXS intermediate states) 4.3 -> 2.9 ms for
// the whole solve; a random H of 3500 rows 38 -> 20; 70 right-hand sides of 360 rows (pairs) 6.1 -> 4.9.  A
// step of the 360 states is ~7000 cycles of latencies: 2 barriers of ~600, two sums over all lanes of
// ~1200 each, some 30 dependent FP64 operations of 64 and more.
constexpr int kClusterMax = 8;
constexpr int kOwnTrackers = 64;                                         // shifts of a tracking CTA at most
constexpr int kClusterWarps = kSmallThreads / 32;                        // main warps at most
constexpr int kClusterThreads = kSmallThreads + 32 + kSmallThreads / 2;  // and the sums', and the trackers

struct ClusterArgs {
  ShiftedArgs a;
  int passes;   // rounds of main_threads / SUB rows
  int rows_on;  // row CTAs: all of the cluster, or all but the last
};

// barrier of the first `threads` threads (the main warps and the one that sums)
__device__ __forceinline__ void cluster_bar(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

template <bool VALC, int SUB>
__global__ void __launch_bounds__(kClusterThreads) shifted_cluster_kernel(ClusterArgs ca) {
  const ShiftedArgs& g = ca.a;
  cg::cluster_group cl = cg::this_cluster();
  const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank(), RC = ca.rows_on;
  const int n = (int)g.n, M = g.main_threads, mw = M >> 5, nz = g.nz, k_cap = g.k_cap;
  constexpr int spw = 32 / SUB;  // rows of a warp
  const int passes = ca.passes, rpp = M / SUB, nsl = passes * mw;
  extern __shared__ __align__(16) unsigned char sm[];
  double2* A = reinterpret_cast<double2*>(sm);
  double2* B = A + n;
  double* own_y = reinterpret_cast<double*>(B + n);  // [passes][M] of this thread's components
  double* own_p = own_y + (size_t)passes * M;
  double* sval = own_p + (size_t)passes * M;
  uint16_t* scol = reinterpret_cast<uint16_t*>(sval + (size_t)g.ent_cap * (VALC ? 2 : 1));
  uint16_t* len = scol + g.ent_cap;  // [n]
  uint16_t* order = len + n;         // [passes * rpp] this CTA's rows, 0xFFFF past the last
  __shared__ double s_alpha[kClusterMax * kClusterWarps], s_norm[kClusterMax * kClusterWarps];
  __shared__ int s_ok[kClusterMax * kClusterWarps];
  __shared__ int soff[2 * kSmallThreads];
  __shared__ double s_a, s_b, s_ib, s_ib2;
  __shared__ int sliced;
  const int tid = threadIdx.x, bs = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const bool row_cta = rank < RC, last_cta = rank == CL - 1;
  const bool is_main = tid < M, is_sum = warp == mw;
  // trackers: every CTA's where they share the row CTAs, else the last CTA's
  const int tz = tid - M - 32, tw = (bs - M - 32) >> 5;
  const int tcs = RC == CL ? CL : 1, trank = RC == CL ? rank : 0;
  const bool is_track = tz >= 0 && (RC == CL || last_cta);
  const int zi = tz * tcs + trank;
  const int comp = SUB == 4 ? (lane >> 1) & 1 : lane & 1;            // 0: real part, 1: imaginary part
  const int d0 = SUB == 4 ? lane & 1 : 0, dstep = SUB == 4 ? 2 : 1;  // the CTAs this lane sends to

  // rows by length, longest first, equal lengths in order; slot s is row s / RC of CTA s % RC
  for (int i = tid; i < n; i += bs) {
    const int64_t l = g.rp[i + 1] - g.rp[i];
    len[i] = (uint16_t)(l < 0xFFFF ? l : 0xFFFF);
  }
  for (int q = tid; q < passes * rpp; q += bs) order[q] = 0xFFFF;
  cl.sync();
  for (int i = rank + CL * tid; i < n; i += CL * bs) {
    const int l = len[i];
    int at = 0;
    for (int q = 0; q < n; ++q) at += len[q] > l || (len[q] == l && q < i);
    cl.map_shared_rank(order, at % RC)[at / RC] = (uint16_t)i;
  }
  cl.sync();
  if (tid == 0) {
    int at = 0;
    for (int s = 0; s < nsl; ++s) {
      const int row = order[s * spw];
      soff[s] = at;
      if (row != 0xFFFF) at += 32 * ((len[row] + SUB - 1) / SUB);
      if (at > g.ent_cap) break;
    }
    soff[nsl] = at;
    sliced = at <= g.ent_cap;
  }
  __syncthreads();
  if (sliced) {
    for (int q = tid; q < 32 * nsl; q += bs) {
      const int s = q >> 5, row = order[s * spw + (q & 31) / SUB], width = (soff[s + 1] - soff[s]) >> 5;
      const int l = row == 0xFFFF ? 0 : len[row];
      const int64_t e0 = row == 0xFFFF ? 0 : g.rp[row];
      for (int e = 0; e < width; ++e) {
        const int at = soff[s] + 32 * e + (q & 31), k = e * SUB + q % SUB;
        scol[at] = k < l ? (uint16_t)g.col[e0 + k] : 0;
        if (VALC) {
          sval[2 * at] = k < l ? g.vals[2 * (e0 + k)] : 0.0;
          sval[2 * at + 1] = k < l ? g.vals[2 * (e0 + k) + 1] : 0.0;
        } else {
          sval[at] = k < l ? g.vals[e0 + k] : 0.0;
        }
      }
    }
  }
  __syncthreads();
  // a thread's row of the first pass
  const int row0 = is_main ? order[tid / SUB] : 0xFFFF;
  const int len0 = row0 != 0xFFFF ? len[row0] : 0, at0 = is_main && sliced ? soff[warp] + lane : 0;

  // the sum of a main warp's components (the lanes of one component carry equal values)
  auto warp_part = [&](double v) -> double {
#pragma unroll
    for (int o = 16; o >= (SUB == 4 ? 2 : 1); o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  auto total = [&](const double* slots) -> double {
    double v = 0.0;
    for (int k = lane; k < RC * mw; k += 32) v += slots[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  // |w| and its reciprocal, from the last CTA to every CTA: the root from the reciprocal by one
  // Newton step
  auto roots = [&](double* out) {
    const double w2 = total(s_norm);
    const double ib = w2 > 0.0 ? rsqrt(w2) : 0.0, h = w2 * ib;
    const double b = w2 < HUGE_VAL ? fma(fma(-h, h, w2), 0.5 * ib, h) : w2;
    if (lane < CL) {
      *cl.map_shared_rank(&s_ib, lane) = ib;
      *cl.map_shared_rank(&s_ib2, lane) = ib * ib;
      *cl.map_shared_rank(&s_b, lane) = b;
    }
    if (lane == 0) *out = b;
  };

  for (int r = blockIdx.x / CL; r < g.n_rhs; r += gridDim.x / CL) {
    double2* Vr = g.V + (size_t)r * k_cap * n;
    const double2* y = g.Y + (size_t)r * n;
    double2 *cur = A, *nxt = B;
    cl.sync();  // every CTA is done with the slots of the last right-hand side
    for (int i = tid; i < n; i += bs) cur[i] = y[i];
    if (is_main && row_cta) {
      double acc = 0.0;
      for (int ps = 0; ps < passes; ++ps) {
        const int row = ps ? order[ps * rpp + tid / SUB] : row0;
        if (row == 0xFFFF) continue;
        const double v = comp ? y[row].y : y[row].x;
        own_p[ps * M + tid] = 0.0;
        acc = fma(v, v, acc);
      }
      acc = warp_part(acc);
      if (lane == 0) cl.map_shared_rank(s_norm, CL - 1)[rank * mw + warp] = acc;
    }
    cl.sync();
    if (is_sum && last_cta) roots(g.ynorm + r);
    cl.sync();
    if (!(s_b > 0.0)) {
      if (rank == 0 && tid == 0) g.m_out[r] = 0;
      continue;
    }
    const double iyn = s_ib;
    for (int i = tid; i < n; i += bs) cur[i] = make_double2(cur[i].x * iyn, cur[i].y * iyn);
    __syncthreads();
    double2 z = make_double2(0.0, 0.0), id = make_double2(0.0, 0.0), q = make_double2(1.0, 0.0);
    if (is_track && zi < nz) z = g.zs[(size_t)r * nz + zi];
    double bt = 0.0;  // a tracker's beta_{j-2}
    int m = k_cap;
    for (int j = 0;; ++j) {
      // ---- 1
      if (is_main) {
        if (row_cta && j < k_cap) {
          double acc = 0.0;
          for (int ps = 0; ps < passes; ++ps) {
            const int row = ps ? order[ps * rpp + tid / SUB] : row0;
            double yr = 0.0, yi = 0.0, x = 0.0;
            if (row != 0xFFFF) {
              x = reinterpret_cast<const double*>(cur)[2 * row + comp];
              if (sliced) {
                const int l = ps ? len[row] : len0;
                int at = ps ? soff[ps * mw + warp] + lane : at0;
#pragma unroll 4
                for (int k = tid % SUB; k < l; k += SUB, at += 32) {
                  const double2 xv = cur[scol[at]];
                  const double hr = sval[VALC ? 2 * at : at];
                  yr = fma(hr, xv.x, yr);
                  yi = fma(hr, xv.y, yi);
                  if (VALC) {
                    const double hi = sval[2 * at + 1];
                    yr = fma(-hi, xv.y, yr);
                    yi = fma(hi, xv.x, yi);
                  }
                }
              } else {
                const int64_t e1 = g.rp[row + 1];
#pragma unroll 4
                for (int64_t e = g.rp[row] + tid % SUB; e < e1; e += SUB) {
                  const double2 xv = cur[g.col[e]];
                  const double hr = g.vals[VALC ? 2 * e : e];
                  yr = fma(hr, xv.x, yr);
                  yi = fma(hr, xv.y, yi);
                  if (VALC) {
                    const double hi = g.vals[2 * e + 1];
                    yr = fma(-hi, xv.y, yr);
                    yi = fma(hi, xv.x, yi);
                  }
                }
              }
            }
            double v = (comp ? yi : yr) + __shfl_xor_sync(0xffffffffu, comp ? yr : yi, SUB >> 1);
            if (SUB == 4) v += __shfl_xor_sync(0xffffffffu, v, 1);
            own_y[ps * M + tid] = v;
            acc = fma(v, x, acc);
          }
          acc = warp_part(acc);
          if (lane < CL) cl.map_shared_rank(s_alpha, lane)[rank * mw + warp] = acc;
        }
      } else if (is_sum) {
        if (last_cta && j > 0) roots(g.beta + (size_t)r * k_cap + j - 1);
      } else if (is_track && j > 0 && zi < nz) {
        // the shift's pivot and residual estimate for step j - 1, but for the factor beta_{j-1}
        double2 d = make_double2(z.x - s_a, z.y), qn = make_double2(1.0, 0.0);
        if (j > 1) {
          const double b2 = bt * bt;
          d.x -= b2 * id.x;
          d.y -= b2 * id.y;
          qn = make_double2(q.x * bt, q.y * bt);
        }
        const double rd = 1.0 / (d.x * d.x + d.y * d.y);
        id = make_double2(d.x * rd, -d.y * rd);
        q = make_double2(qn.x * id.x - qn.y * id.y, qn.x * id.y + qn.y * id.x);
      }
      cl.sync();
      const double b = s_b, ib = j > 0 ? s_ib : 1.0;  // beta_{j-1} and its reciprocal
      if (!(b > 0.0)) {  // the space is exhausted, or a NaN
        m = j;
        if (rank == 0 && tid == 0 && !(b >= 0.0)) atomicExch(g.status, (int32_t)EDGPU_ERR_NAN);
        break;
      }
      // ---- 2
      if (is_main) {
        if (row_cta && j < k_cap) {
          const double nb = j > 0 ? -b : 0.0;
          double* vj = reinterpret_cast<double*>(Vr + (size_t)j * n);
          for (int ps = 0; ps < passes; ++ps) {
            const int row = ps ? order[ps * rpp + tid / SUB] : row0, at = ps * M + tid;
            if (row == 0xFFFF) continue;
            const double v = reinterpret_cast<const double*>(cur)[2 * row + comp] * ib;
            own_y[at] = fma(nb, own_p[at], own_y[at] * ib);
            own_p[at] = v;
            if (d0 == 0) vj[2 * row + comp] = v;
          }
          cluster_bar(M + 32);
          const double na = -s_a;
          double acc = 0.0;
          for (int ps = 0; ps < passes; ++ps) {
            const int row = ps ? order[ps * rpp + tid / SUB] : row0, at = ps * M + tid;
            if (row == 0xFFFF) continue;
            const double w = fma(na, own_p[at], own_y[at]);
            acc = fma(w, w, acc);
            for (int d = d0; d < RC; d += dstep)
              reinterpret_cast<double*>(cl.map_shared_rank(nxt, d))[2 * row + comp] = w;
          }
          acc = warp_part(acc);
          if (lane == 0) cl.map_shared_rank(s_norm, CL - 1)[rank * mw + warp] = acc;
        }
      } else if (is_sum) {
        if (j < k_cap) {
          double a = total(s_alpha);
          if (j > 0) a *= s_ib2;
          if (lane == 0) {
            s_a = a;
            if (rank == 0) g.alpha[(size_t)r * k_cap + j] = a;
          }
          if (row_cta) cluster_bar(M + 32);
        }
      } else if (is_track && j > 0) {
        bt = b;
        const bool ok = __all_sync(0xffffffffu, zi >= nz || b * sqrt(q.x * q.x + q.y * q.y) <= g.tol);
        if (lane < CL) cl.map_shared_rank(s_ok, lane)[trank * tw + (tz >> 5)] = ok;
      }
      cl.sync();
      if (j > 0) {
        bool ok = true;
        for (int k = lane; k < tcs * tw; k += 32) ok = ok && s_ok[k];
        const bool conv = __all_sync(0xffffffffu, ok);
        if (conv || j == k_cap) {  // step j - 1 was the last
          m = j;
          if (rank == 0 && tid == 0 && !conv) atomicExch(g.status, (int32_t)EDGPU_ERR_NOCONV);
          break;
        }
      }
      double2* t = cur;
      cur = nxt;
      nxt = t;
    }
    if (rank == 0 && tid == 0) g.m_out[r] = m;
  }
  cl.sync();
}

// The same shifted solves in double-float arithmetic for a real H (values as hi/lo float
// pairs), two vectors per right-hand side as in lanczos_small_df_kernel, each v_j written
// to V[rhs][j] as float4 (re.hi, re.lo, im.hi, im.lo).  The residual estimate only decides
// when to stop, so its LU recurrence runs in FP32 (the pivots keep Im d_k >= Im z > 0, so
// it cannot break down); every thread forms beta and 1/beta from the broadcast sum, and the
// barrier that pools the per-shift verdicts is the only one beyond the two sums.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) shifted_small_df_kernel(
    int64_t n, const int64_t* __restrict__ rp, const int32_t* __restrict__ col, const float2* __restrict__ hv,
    int n_rhs, const double2* __restrict__ Y, const double2* __restrict__ zs, int nz, int k_cap, float tol,
    float4* __restrict__ V, double* __restrict__ alpha, double* __restrict__ beta, int32_t* __restrict__ m_out,
    double* __restrict__ ynorm_out, int32_t* status) {
  extern __shared__ __align__(16) unsigned char sm[];
  float4* A = reinterpret_cast<float4*>(sm);
  float4* B = A + n;
  dfl* red = reinterpret_cast<dfl*>(B + n);
  int32_t* srp = reinterpret_cast<int32_t*>(red + kDfRed);
  constexpr int NW = THREADS / 32;
  const int tid = threadIdx.x;
  const dfl zero = {0.f, 0.f};
  for (int64_t i = tid; i <= n; i += THREADS) srp[i] = (int32_t)rp[i];
  for (int r = blockIdx.x; r < n_rhs; r += gridDim.x) {
    float4* Vr = V + (size_t)r * k_cap * n;
    const double2* y = Y + (size_t)r * n;
    dacc acc = {0.f, 0.f};
    for (int64_t i = tid; i < n; i += THREADS) {
      const double2 v = y[i];
      const dfl re = df_split(v.x), im = df_split(v.y);
      A[i] = make_float4(re.hi, re.lo, im.hi, im.lo);
      dacc_fma(acc, re, re.hi, re.lo);
      dacc_fma(acc, im, im.hi, im.lo);
    }
    const dfl yn = df_sqrt(df_block_sum2<NW>(dacc_val(acc), red));
    if (tid == THREADS - 1) ynorm_out[r] = df_val(yn);
    if (!(yn.hi > 0.f)) {
      if (tid == 0) m_out[r] = 0;
      __syncthreads();
      continue;
    }
    const dfl iyn = df_rcp(yn);
    for (int64_t i = tid; i < n; i += THREADS) {
      const float4 w = A[i];
      const dfl vr = df_mul({w.x, w.y}, iyn), vi = df_mul({w.z, w.w}, iyn);
      const float4 v = make_float4(vr.hi, vr.lo, vi.hi, vi.lo);
      A[i] = v;
      B[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      Vr[i] = v;
    }
    __syncthreads();
    float4* x = A;
    float4* p = B;
    float2 z = make_float2(0.f, 0.f), d = make_float2(1.f, 0.f), q = make_float2(1.f, 0.f);
    if (tid < nz) {
      const double2 zd = zs[(size_t)r * nz + tid];
      z = make_float2((float)zd.x, (float)zd.y);
    }
    dfl bprev = zero;
    int m = k_cap;
    for (int j = 0; j < k_cap; ++j) {
      const dfl nb = {-bprev.hi, -bprev.lo};
      acc = {0.f, 0.f};
      for (int64_t i = tid; i < n; i += THREADS) {
        dacc yr = {0.f, 0.f}, yi = {0.f, 0.f};
        const int e1 = srp[i + 1];
        for (int e = srp[i]; e < e1; e += kSmallBatch) {
          int c[kSmallBatch];
          float2 hh[kSmallBatch];
#pragma unroll
          for (int u = 0; u < kSmallBatch; ++u) {
            const bool ok = e + u < e1;
            c[u] = ok ? __ldg(col + e + u) : 0;
            hh[u] = ok ? __ldg(hv + e + u) : make_float2(0.f, 0.f);
          }
#pragma unroll
          for (int u = 0; u < kSmallBatch; ++u) {
            if (e + u < e1) {
              const dfl h = {hh[u].x, hh[u].y};
              const float4 xv = x[c[u]];
              dacc_fma(yr, h, xv.x, xv.y);
              dacc_fma(yi, h, xv.z, xv.w);
            }
          }
        }
        const dfl hr = dacc_val(yr), hi = dacc_val(yi);
        const float4 xi = x[i], pi = p[i];
        dacc_fma(acc, hr, xi.x, xi.y);
        dacc_fma(acc, hi, xi.z, xi.w);
        const dfl wr = df_fma(hr, nb, {pi.x, pi.y}), wi = df_fma(hi, nb, {pi.z, pi.w});
        p[i] = make_float4(wr.hi, wr.lo, wi.hi, wi.lo);
      }
      const dfl a = df_block_sum2<NW>(dacc_val(acc), red);
      if (tid == THREADS - 1) alpha[(size_t)r * k_cap + j] = df_val(a);
      const dfl na = {-a.hi, -a.lo};
      acc = {0.f, 0.f};
      for (int64_t i = tid; i < n; i += THREADS) {
        const float4 w = p[i], xi = x[i];
        const dfl wr = df_fma({w.x, w.y}, na, {xi.x, xi.y});
        const dfl wi = df_fma({w.z, w.w}, na, {xi.z, xi.w});
        p[i] = make_float4(wr.hi, wr.lo, wi.hi, wi.lo);
        dacc_fma(acc, wr, wr.hi, wr.lo);
        dacc_fma(acc, wi, wi.hi, wi.lo);
      }
      const dfl b = df_sqrt(df_block_sum2<NW>(dacc_val(acc), red + 40));
      if (tid == THREADS - 1) beta[(size_t)r * k_cap + j] = df_val(b);
      bool ok = true;
      if (tid < nz) {
        const float af = a.hi, bp = bprev.hi;
        float2 dn = make_float2(z.x - af, z.y);
        if (j > 0) {
          const float rd = __fdiv_rn(bp * bp, d.x * d.x + d.y * d.y);
          dn.x -= rd * d.x;
          dn.y += rd * d.y;
        }
        const float2 qn = make_float2(j > 0 ? q.x * bp : 1.f, j > 0 ? q.y * bp : 0.f);
        const float rr = __fdiv_rn(1.f, dn.x * dn.x + dn.y * dn.y);
        q = make_float2((qn.x * dn.x + qn.y * dn.y) * rr, (qn.y * dn.x - qn.x * dn.y) * rr);
        d = dn;
        ok = b.hi * sqrtf(q.x * q.x + q.y * q.y) <= tol;
      }
      const bool conv = __syncthreads_and(ok);
      if (conv || !(b.hi > 0.f) || j + 1 == k_cap) {
        m = j + 1;
        if (tid == 0) {
          if (!(b.hi >= 0.f))
            atomicExch(status, (int32_t)EDGPU_ERR_NAN);
          else if (!conv && b.hi > 0.f)
            atomicExch(status, (int32_t)EDGPU_ERR_NOCONV);
        }
        break;
      }
      const dfl ib = df_rcp(b);
      float4* vn = Vr + (size_t)(j + 1) * n;
      for (int64_t i = tid; i < n; i += THREADS) {
        const float4 w = p[i];
        const dfl vr = df_mul({w.x, w.y}, ib), vi = df_mul({w.z, w.w}, ib);
        const float4 v = make_float4(vr.hi, vr.lo, vi.hi, vi.lo);
        p[i] = v;
        vn[i] = v;
      }
      __syncthreads();
      float4* t = p;
      p = x;
      x = t;
      bprev = b;
    }
    if (tid == 0) m_out[r] = m;
    __syncthreads();
  }
}

// coef[r][k][z] = ynorm_r * ((z - T_m)^{-1} e_1)_k, from the minors of z - T_m: with
//   theta_k = (z - a_k) theta_{k+1} - b_k^2 theta_{k+2}, theta_m = 1, theta_{m+1} = 0
// the solution is x_k = (b_0 ... b_{k-1}) theta_{k+1} / theta_0.  Neither product has a division, so
// the chain per step is two dependent multiply-adds instead of a reciprocal and two sweeps, and what
// follows the chains runs a component per thread over the whole chip (15 right-hand sides, 50
// shifts, ~490 steps: the sweeps of an elimination 0.56 ms, chains and components 0.19 ms).  Values
// are kept within +-300 bits of 1, the power of two taken out so far beside them.
__device__ __forceinline__ int exponent_of(double x) { return (__double2hiint(x) >> 20) & 0x7FF; }

// (z - a) t1 - b^2 t2
__device__ __forceinline__ double2 minor_step(double2 z, double a, double b, double2 t1, double2 t2) {
  const double dr = z.x - a, b2 = -(b * b);
  return make_double2(fma(dr, t1.x, fma(-z.y, t1.y, b2 * t2.x)), fma(dr, t1.y, fma(z.y, t1.x, b2 * t2.y)));
}

// Block per right-hand side: a thread per shift runs its chain, one of the last warp the products.
__global__ void __launch_bounds__(512) shifted_chain_kernel(const double* __restrict__ alpha,
                                                            const double* __restrict__ beta,
                                                            const int32_t* __restrict__ m_arr,
                                                            const double2* __restrict__ zs, int nz, int k_cap,
                                                            double2* __restrict__ theta, int* __restrict__ theta_exp,
                                                            double* __restrict__ prod, int* __restrict__ prod_exp) {
  extern __shared__ double ab[];
  const int r = blockIdx.x;
  const int m = m_arr[r];
  double* a = ab;
  double* b = ab + k_cap;
  for (int k = threadIdx.x; k < m; k += blockDim.x) {
    a[k] = alpha[(size_t)r * k_cap + k];
    b[k] = beta[(size_t)r * k_cap + k];
  }
  __syncthreads();
  const size_t base = (size_t)r * k_cap * nz;
  if (threadIdx.x >= blockDim.x - 32) {  // a warp of its own
    if (threadIdx.x != blockDim.x - 1) return;
    double p = 1.0;
    int e = 0;
    for (int k = 0; k < m; ++k) {
      prod[(size_t)r * k_cap + k] = p;
      prod_exp[(size_t)r * k_cap + k] = e;
      p *= b[k];
      const int ex = exponent_of(p);
      if ((ex > 1323 && ex < 2046) || (ex < 723 && ex > 0)) {
        p *= __hiloint2double((2046 - ex) << 20, 0);
        e += ex - 1023;
      }
    }
    return;
  }
  for (int zi = threadIdx.x; zi < nz; zi += blockDim.x - 32) {
    const double2 z = zs[(size_t)r * nz + zi];
    double2 t1 = make_double2(1.0, 0.0), t2 = make_double2(0.0, 0.0);
    int e = 0;
    // four steps between two looks at the exponents: what does not hang on the chain is ready early
    for (int k0 = (m - 1) & ~3; k0 >= 0; k0 -= 4) {
#pragma unroll
      for (int u = 3; u >= 0; --u) {
        const int k = k0 + u;
        if (k < m) {
          theta[base + (size_t)k * nz + zi] = t1;  // theta_{k+1}
          theta_exp[base + (size_t)k * nz + zi] = e;
          const double2 t = minor_step(z, a[k], b[k], t1, t2);
          t2 = t1;
          t1 = t;
        }
      }
      const int ex = max(max(exponent_of(t1.x), exponent_of(t1.y)), max(exponent_of(t2.x), exponent_of(t2.y)));
      if ((ex > 1323 && ex < 2046) || (ex < 723 && ex > 0)) {
        const double f = __hiloint2double((2046 - ex) << 20, 0);
        t1.x *= f;
        t1.y *= f;
        t2.x *= f;
        t2.y *= f;
        e += ex - 1023;
      }
    }
  }
}

// A component per thread; DF writes the coefficients as double-float pairs (float4).
template <bool DF>
__global__ void __launch_bounds__(256) shifted_coef_kernel(
    const double* __restrict__ alpha, const double* __restrict__ beta, const int32_t* __restrict__ m_arr,
    const double* __restrict__ ynorm, const double2* __restrict__ zs, int nz, int k_cap,
    const double2* __restrict__ theta, const int* __restrict__ theta_exp, const double* __restrict__ prod,
    const int* __restrict__ prod_exp, double2* __restrict__ coef, float4* __restrict__ coef_df) {
  const int r = blockIdx.y;
  const int m = m_arr[r];
  const size_t base = (size_t)r * k_cap * nz;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (int64_t)m * nz;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(t / nz), zi = (int)(t - (int64_t)k * nz);
    // theta_0 from theta_1 and theta_2, in theta_1's power of two
    const double2 t1 = theta[base + zi];
    const int e0 = theta_exp[base + zi];
    double2 t2 = make_double2(0.0, 0.0);
    if (m > 1) {
      const int d = theta_exp[base + nz + zi] - e0;
      t2 = theta[base + nz + zi];
      t2 = make_double2(ldexp(t2.x, d), ldexp(t2.y, d));
    }
    const double2 t0 = minor_step(zs[(size_t)r * nz + zi], alpha[(size_t)r * k_cap], beta[(size_t)r * k_cap], t1, t2);
    const double2 v = theta[base + t];
    const double s = ynorm[r] * prod[(size_t)r * k_cap + k] / (t0.x * t0.x + t0.y * t0.y);
    const int e = prod_exp[(size_t)r * k_cap + k] + theta_exp[base + t] - e0;
    const double2 o = make_double2(ldexp(s * fma(v.x, t0.x, v.y * t0.y), e), ldexp(s * fma(v.y, t0.x, -(v.x * t0.y)), e));
    if (DF) {
      const dfl re = df_split(o.x), im = df_split(o.y);
      coef_df[base + t] = make_float4(re.hi, re.lo, im.hi, im.lo);
    } else {
      coef[base + t] = o;
    }
  }
}

// X[r][z][i] = sum_k coef[r][k][z] V[r][k][i] (FP64): thread per row, kSumZ shifts per thread.  Bound
// by FP64 issue, so a complex product takes three multiply-adds instead of four: with
//   s1 += cr (vr + vi), s2 += vi (cr + ci), s3 += vr (ci - cr)
// the sums are re = s1 - s2, im = s1 + s3; vr + vi is formed once for all shifts, the coefficient
// sums once per block.  (Written as a sum of products the four compiled to six.)  15 x 50 sums of
// ~490 vectors of 360 rows: 1.60 -> 0.81 ms.  The rounding is bounded by |c| |v| and not by each component, so
// the smaller of a sum's real and imaginary parts is relatively less accurate than by four products; both errors
// lie far below the 1e-10 at which the solves stop.
constexpr int kSumZ = 4, kSumRows = 64, kSumStage = 64;
__global__ void __launch_bounds__(kSumRows) combine_batched_kernel(const double2* __restrict__ V,
                                                                   const double2* __restrict__ coef,
                                                                   const int32_t* __restrict__ m_arr, int64_t n,
                                                                   int nz, int k_cap, double2* __restrict__ X) {
  __shared__ double cs[kSumStage][kSumZ][3];
  const int r = blockIdx.z, z0 = blockIdx.y * kSumZ;
  const int m = m_arr[r];
  const double2* c = coef + (size_t)r * k_cap * nz;
  const double2* Vr = V + (size_t)r * k_cap * n;
  const int64_t i = (int64_t)blockIdx.x * kSumRows + threadIdx.x;
  double s1[kSumZ], s2[kSumZ], s3[kSumZ];
#pragma unroll
  for (int u = 0; u < kSumZ; ++u) s1[u] = s2[u] = s3[u] = 0.0;
  for (int k0 = 0; k0 < m; k0 += kSumStage) {
    const int kn = m - k0 < kSumStage ? m - k0 : kSumStage;
    __syncthreads();
    for (int t = threadIdx.x; t < kn * kSumZ; t += kSumRows) {
      const int k = t / kSumZ, u = t % kSumZ;
      const double2 v = z0 + u < nz ? c[(size_t)(k0 + k) * nz + z0 + u] : make_double2(0.0, 0.0);
      cs[k][u][0] = v.x;
      cs[k][u][1] = v.x + v.y;
      cs[k][u][2] = v.y - v.x;
    }
    __syncthreads();
    if (i < n) {
#pragma unroll 4
      for (int k = 0; k < kn; ++k) {
        const double2 v = Vr[(size_t)(k0 + k) * n + i];
        const double sum = v.x + v.y;
#pragma unroll
        for (int u = 0; u < kSumZ; ++u) {
          s1[u] = fma(cs[k][u][0], sum, s1[u]);
          s2[u] = fma(cs[k][u][1], v.y, s2[u]);
          s3[u] = fma(cs[k][u][2], v.x, s3[u]);
        }
      }
    }
  }
  if (i >= n) return;
#pragma unroll
  for (int u = 0; u < kSumZ; ++u)
    if (z0 + u < nz) X[((size_t)r * nz + z0 + u) * n + i] = make_double2(s1[u] - s2[u], s1[u] + s3[u]);
}

// The same in double-float: thread per row i, kCombineZ shifts per thread (V[k][i] read once
// for all of them), sums in double-float, FP64 only for the output.
constexpr int kCombineZ = 8;
__global__ void __launch_bounds__(128) combine_df_kernel(const float4* __restrict__ V, const float4* __restrict__ coef,
                                                         const int32_t* __restrict__ m_arr, int64_t n, int nz,
                                                         int k_cap, double2* __restrict__ X) {
  const int r = blockIdx.z;
  const int z0 = blockIdx.y * kCombineZ;
  const int m = m_arr[r];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float4* c = coef + (size_t)r * k_cap * nz;
  const float4* Vr = V + (size_t)r * k_cap * n;
  dacc xr[kCombineZ], xi[kCombineZ];
#pragma unroll
  for (int u = 0; u < kCombineZ; ++u) xr[u] = xi[u] = {0.f, 0.f};
  if (i < n) {
    for (int k = 0; k < m; ++k) {
      const float4 v = Vr[(size_t)k * n + i];
#pragma unroll
      for (int u = 0; u < kCombineZ; ++u) {
        const float4 ck = z0 + u < nz ? __ldg(c + (size_t)k * nz + z0 + u) : make_float4(0.f, 0.f, 0.f, 0.f);
        const dfl cr = {ck.x, ck.y}, ci = {ck.z, ck.w}, nci = {-ck.z, -ck.w};
        dacc_fma(xr[u], cr, v.x, v.y);
        dacc_fma(xr[u], nci, v.z, v.w);
        dacc_fma(xi[u], cr, v.z, v.w);
        dacc_fma(xi[u], ci, v.x, v.y);
      }
    }
#pragma unroll
    for (int u = 0; u < kCombineZ; ++u)
      if (z0 + u < nz) X[((size_t)r * nz + z0 + u) * n + i] = make_double2(df_val(dacc_val(xr[u])), df_val(dacc_val(xi[u])));
  }
}

}  // namespace edgpu

extern "C" size_t edgpu_shifted_solve_workspace(int64_t n, int n_rhs, int nz, int k_cap) {
  size_t b = 0;
  b += sizeof(double2) * (size_t)n_rhs * k_cap * n + 256;       // V
  b += 2 * sizeof(double) * (size_t)n_rhs * k_cap + 512;        // alpha, beta
  b += sizeof(int32_t) * (size_t)n_rhs + sizeof(double) * n_rhs + 512;
  b += 3 * sizeof(double2) * (size_t)n_rhs * nz * k_cap + 768;  // coefficients + Thomas scratch
  return b + 1024;
}

namespace {

// Launches the clusters where one of the sizes holds every right-hand side at once; false where
// none does (the caller's one-CTA form, which keeps every SM busy then) or is accepted.  A warp's worth of
// rows has nothing to share: 1 row takes 130 us on one CTA and 145 on a cluster, 33 rows 342 and 327.
bool launch_shifted_cluster(edgpu::ShiftedArgs g, bool cplx, int64_t nnz, cudaStream_t s) {
  using namespace edgpu;
  if (g.n <= 32) return false;
  const size_t per_entry = (cplx ? 16 : 8) + 2;
  for (int cl = kClusterMax; cl > 1; cl >>= 1) {
    if ((int64_t)g.n_rhs * cl > grid_cap()) continue;
    ClusterArgs c{};
    c.a = g;
    c.rows_on = cl > 2 && g.nz <= kOwnTrackers ? cl - 1 : cl;
    const int rows = (int)((g.n + c.rows_on - 1) / c.rows_on);
    const int sub = 4 * rows <= kSmallThreads ? 4 : 2;
    auto kern = sub == 4 ? (cplx ? shifted_cluster_kernel<true, 4> : shifted_cluster_kernel<false, 4>)
                         : (cplx ? shifted_cluster_kernel<true, 2> : shifted_cluster_kernel<false, 2>);
    c.a.main_threads = std::min(kSmallThreads, (sub * rows + 31) / 32 * 32);
    c.passes = (sub * rows + c.a.main_threads - 1) / c.a.main_threads;
    const int threads = c.a.main_threads + 32 + ((c.rows_on < cl ? g.nz : (g.nz + cl - 1) / cl) + 31) / 32 * 32;
    const size_t fixed = 2 * sizeof(double2) * (size_t)g.n + 2 * sizeof(double) * (size_t)c.passes * c.a.main_threads +
                         sizeof(uint16_t) * (size_t)(g.n + (int64_t)c.passes * c.a.main_threads / sub) + 16;
    if (fixed > 200 * 1024) continue;
    // a warp's rows have nearly equal lengths: room for half as many lanes without an entry again
    const int64_t want = (nnz / c.rows_on + 1) * 3 / 2 + (int64_t)sub * rows + 32;
    c.a.ent_cap = fixed + per_entry * (size_t)want <= 216 * 1024 ? (int)((want + 3) & ~(int64_t)3) : 0;
    const size_t bytes = fixed + per_entry * (size_t)c.a.ent_cap;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = cl;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(cl * g.n_rhs));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (fit < g.n_rhs) continue;
    if (cudaLaunchKernelEx(&cfg, kern, c) == cudaSuccess) return true;
    cudaGetLastError();
  }
  return false;
}

int shifted_solve_impl(const edgpu_csr* h, const double* Y, int n_rhs, const double* zs, int nz, int k_cap, double tol,
                       double* X, int32_t* m_out, int32_t* status_dev, void* workspace, size_t workspace_bytes,
                       cudaStream_t s, bool df) {
  using namespace edgpu;
  if (!h || !Y || !zs || !X || !m_out || !status_dev || n_rhs < 1 || nz < 1 || k_cap < 1 || h->n < 1)
    return EDGPU_ERR_ARG;
  if (nz > kSmallThreads) return EDGPU_ERR_ARG;
  if (df && (!h->val_df || h->val_c)) return EDGPU_ERR_ARG;
  if (workspace_bytes < edgpu_shifted_solve_workspace(h->n, n_rhs, nz, k_cap)) return EDGPU_ERR_WORKSPACE;
  const int64_t n = h->n;
  const size_t smem = df ? small_smem_bytes(n, 3) : 3 * sizeof(double2) * (size_t)n + 34 * sizeof(double) + 16;
  if (smem > 200 * 1024) return EDGPU_ERR_ARG;
  const size_t coef_smem = 2 * sizeof(double) * (size_t)k_cap;
  if (coef_smem > 200 * 1024) return EDGPU_ERR_ARG;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  size_t off = 0;
  auto carve = [&](size_t bytes) {
    unsigned char* p = ws + off;
    off += (bytes + 255) & ~(size_t)255;
    return p;
  };
  void* V = carve(sizeof(double2) * (size_t)n_rhs * k_cap * n);
  double* alpha = reinterpret_cast<double*>(carve(sizeof(double) * (size_t)n_rhs * k_cap));
  double* beta = reinterpret_cast<double*>(carve(sizeof(double) * (size_t)n_rhs * k_cap));
  double* yn = reinterpret_cast<double*>(carve(sizeof(double) * (size_t)n_rhs));
  const size_t cbytes = sizeof(double2) * (size_t)n_rhs * nz * k_cap;
  void* coef = carve(cbytes);
  double2* cp = reinterpret_cast<double2*>(carve(cbytes));
  double2* xs = reinterpret_cast<double2*>(carve(cbytes));
  if (off > workspace_bytes) return EDGPU_ERR_WORKSPACE;
  const double2* Yc = reinterpret_cast<const double2*>(Y);
  const double2* zc = reinterpret_cast<const double2*>(zs);
  int per_sm = 0;
  if (df) {
    auto kern = shifted_small_df_kernel<kSmallThreads>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSmallThreads, smem);
    if (per_sm < 1) per_sm = 1;
    const int grid = std::min(grid_cap() * per_sm, n_rhs);
    kern<<<grid, kSmallThreads, smem, s>>>(n, h->row_ptr, h->col, reinterpret_cast<const float2*>(h->val_df), n_rhs,
                                           Yc, zc, nz, k_cap, (float)tol, reinterpret_cast<float4*>(V), alpha, beta,
                                           m_out, yn, status_dev);
  } else {
    auto kern = h->val_c ? shifted_small_kernel<true> : shifted_small_kernel<false>;
    const int npad = (int)((n + 31) & ~(int64_t)31);
    ShiftedArgs g{};
    g.n = n;
    g.rp = h->row_ptr;
    g.col = h->col;
    g.vals = h->val_c ? h->val_c : h->val_r;
    g.n_rhs = n_rhs;
    g.Y = Yc;
    g.zs = zc;
    g.nz = nz;
    g.k_cap = k_cap;
    g.tol = tol;
    g.V = reinterpret_cast<double2*>(V);
    g.alpha = alpha;
    g.beta = beta;
    g.m_out = m_out;
    g.ynorm = yn;
    g.status = status_dev;
    const size_t per_entry = (h->val_c ? 16 : 8) + 2;
    if (!launch_shifted_cluster(g, h->val_c != nullptr, h->nnz, s)) {
      g.main_threads = std::min(kSmallThreads, npad);
      const int threads = g.main_threads + (nz + 31) / 32 * 32;
      // shared memory: vectors, sums, slots; the sliced entries when a third more than nnz of them fit
      const size_t fixed = 3 * sizeof(double2) * (size_t)n + 34 * sizeof(double) + 2 * sizeof(uint16_t) * (size_t)npad + 16;
      const int64_t want = h->nnz + h->nnz / 3 + 32;
      g.ent_cap = fixed + per_entry * (size_t)want <= 220 * 1024 ? (int)((want + 3) & ~(int64_t)3) : 0;
      const size_t bytes = fixed + per_entry * (size_t)g.ent_cap;
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, bytes);
      if (per_sm < 1) per_sm = 1;
      const int grid = std::min(grid_cap() * per_sm, n_rhs);
      kern<<<grid, threads, bytes, s>>>(g);
    }
  }
  note_launch();
  int rc = check_launch();
  if (rc) return rc;
  // the scratch of the coefficients: [products][their exponents][exponents of the minors]
  double* prod = reinterpret_cast<double*>(xs);
  int* prod_exp = reinterpret_cast<int*>(prod + (size_t)n_rhs * k_cap);
  int* theta_exp = prod_exp + (size_t)n_rhs * k_cap;
  cudaFuncSetAttribute(shifted_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)coef_smem);
  const int cthreads = std::min(512, (nz + 31) / 32 * 32 + 32);
  shifted_chain_kernel<<<n_rhs, cthreads, coef_smem, s>>>(alpha, beta, m_out, zc, nz, k_cap, cp, theta_exp, prod,
                                                          prod_exp);
  note_launch();
  const dim3 cgrid((unsigned)std::min<int64_t>(((int64_t)k_cap * nz + 255) / 256, grid_cap()), (unsigned)n_rhs);
  if (df)
    shifted_coef_kernel<true><<<cgrid, 256, 0, s>>>(alpha, beta, m_out, yn, zc, nz, k_cap, cp, theta_exp, prod,
                                                    prod_exp, nullptr, reinterpret_cast<float4*>(coef));
  else
    shifted_coef_kernel<false><<<cgrid, 256, 0, s>>>(alpha, beta, m_out, yn, zc, nz, k_cap, cp, theta_exp, prod,
                                                     prod_exp, reinterpret_cast<double2*>(coef), nullptr);
  note_launch();
  if (df) {
    dim3 g3((unsigned)((n + 127) / 128), (unsigned)((nz + kCombineZ - 1) / kCombineZ), (unsigned)n_rhs);
    combine_df_kernel<<<g3, 128, 0, s>>>(reinterpret_cast<const float4*>(V), reinterpret_cast<const float4*>(coef), m_out,
                                         n, nz, k_cap, reinterpret_cast<double2*>(X));
  } else {
    dim3 g3((unsigned)((n + kSumRows - 1) / kSumRows), (unsigned)((nz + kSumZ - 1) / kSumZ), (unsigned)n_rhs);
    combine_batched_kernel<<<g3, kSumRows, 0, s>>>(reinterpret_cast<const double2*>(V),
                                                   reinterpret_cast<const double2*>(coef), m_out, n, nz, k_cap,
                                                   reinterpret_cast<double2*>(X));
  }
  note_launch();
  return check_launch();
}

}  // namespace

extern "C" int edgpu_shifted_solve(const edgpu_csr* h, const double* Y, int n_rhs, const double* zs, int nz, int k_cap,
                                   double tol, double* X, int32_t* m_out, int32_t* status_dev, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  return shifted_solve_impl(h, Y, n_rhs, zs, nz, k_cap, tol, X, m_out, status_dev, workspace, workspace_bytes,
                            (cudaStream_t)stream, false);
}

extern "C" int edgpu_shifted_solve_df(const edgpu_csr* h, const double* Y, int n_rhs, const double* zs, int nz,
                                      int k_cap, double tol, double* X, int32_t* m_out, int32_t* status_dev,
                                      void* workspace, size_t workspace_bytes, void* stream) {
  return shifted_solve_impl(h, Y, n_rhs, zs, nz, k_cap, tol, X, m_out, status_dev, workspace, workspace_bytes,
                            (cudaStream_t)stream, true);
}

// =======================================================================================
// Allocation-free batched Lanczos (edgpu_lanczos_noalloc).
//
// For callers that cannot allocate device memory themselves.  The grid-wide batched
// Lanczos needs three [n][R] vectors and per-block partial sums as scratch; here that
// scratch is this file's static device array, which every GPU that loads the library
// holds until the process exits.  Host code must not hand the array's name to a kernel
// (in host code it is only a stand-in symbol): its device address is looked up once per
// device with cudaGetSymbolAddress, with that device current, and cached.
// =======================================================================================
#include <mutex>

static __device__ __align__(256) unsigned char g_lanczos_noalloc_scratch[EDGPU_LANCZOS_NOALLOC_BYTES];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kMaxDevices] = {};

int noalloc_scratch_address(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return EDGPU_ERR_CUDA;
  if (dev < 0 || dev >= kMaxDevices) return EDGPU_ERR_ARG;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_lanczos_noalloc_scratch) != cudaSuccess || !p) return EDGPU_ERR_CUDA;
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return EDGPU_OK;
}
}  // namespace

extern "C" int edgpu_lanczos_noalloc(const edgpu_csr* h, const double* v0, int R, const int32_t* k_max, int K,
                                     int precision, double* alpha, double* beta, int32_t* status_dev, void* stream) {
  if (!h || !v0 || R < 1 || K < 1 || !k_max || !alpha || !beta || !status_dev || h->n < 1) return EDGPU_ERR_ARG;
  // the same precision values as edgpu_lanczos accepts
  if (precision < 0 || precision > 3 || precision == 2) return EDGPU_ERR_ARG;
  if (precision == 3) precision = 0;  // the df64 form has no grid-wide variant
  if (precision == 0 && !h->val_c && !h->val_r) return EDGPU_ERR_ARG;
  if (precision != 0 && !h->val_cf && !h->val_rf) return EDGPU_ERR_ARG;
  if (edgpu_lanczos_workspace(h->n, R, K, precision) > (size_t)EDGPU_LANCZOS_NOALLOC_BYTES)
    return EDGPU_ERR_WORKSPACE;
  void* scratch = nullptr;
  const int rc = noalloc_scratch_address(&scratch);
  if (rc) return rc;
  unsigned char* ws = reinterpret_cast<unsigned char*>(scratch);
  const size_t bytes = (size_t)EDGPU_LANCZOS_NOALLOC_BYTES;
  cudaStream_t s = (cudaStream_t)stream;
  // Every buffer in the scratch is written before it is read (the start vectors are
  // copied in, v_{j-1} is first read after step 0 wrote it, partial sums are written by
  // the kernel that precedes their reader), so nothing has to be cleared between calls.
  if (precision == 0) return edgpu::lanczos_impl<double>(h, v0, R, k_max, K, alpha, beta, status_dev, ws, bytes, s);
  return edgpu::lanczos_impl<float>(h, v0, R, k_max, K, alpha, beta, status_dev, ws, bytes, s);
}

extern "C" size_t edgpu_lanczos_noalloc_bytes(void) { return (size_t)EDGPU_LANCZOS_NOALLOC_BYTES; }

extern "C" void edgpu_lanczos_noalloc_forget(void) {
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  for (int d = 0; d < kMaxDevices; ++d) g_noalloc_ptr[d] = nullptr;
}
