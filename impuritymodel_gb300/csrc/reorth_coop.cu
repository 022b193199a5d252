// Lanczos with full reorthogonalisation as one cooperative (grid-wide persistent) launch per
// chunk of steps.
//
// The per-step form issues seven launches per Krylov step (SpMV + alpha, alpha update, two
// Gram-Schmidt passes of dot + project, normalise).  Here one cooperative launch with one block
// of 1024 threads per SM runs the recurrence
//   w = H v_j, alpha_j = Re<v_j, w>, w -= alpha_j v_j + beta_{j-1} v_{j-1},
//   h = V^H w, w -= V h (again where the first pass removed more than half of |w|^2),
//   beta_j = |w|, v_{j+1} = w / beta_j
// in phases separated by grid barriers (cooperative_groups grid sync, ~1.2 us on GB300):
//   A  y = H v_j, a row per kSub lanes; v_j = w / beta_{j-1} is formed by the gather and written
//      to V[j] by the row's first lane; partials of alpha_j.
//   C  w' = y - alpha_j v_j - beta_{j-1} v_{j-1} and its products with V.  The blocks form a grid of
//      row chunks x vector groups: a block keeps its chunk of w' in shared memory and a warp
//      takes a vector's whole chunk, so that every SM has FP64 work whatever m and n are (a block
//      per vector left 152 - m SMs idle and a block's 8 warps on one long vector).
//   R  (many chunks only) h_k from its partials, block k % B.
//   D  w -= V h on each block's rows, lanes on rows and vector classes; partials of |w|^2.
// The second pass (C without the three-term update, R, D) runs only where Kahan's "twice is enough"
// test asks: after a pass that keeps |w| >= |w'| / sqrt(2), w is orthogonal to V to working
// precision.  In a Lanczos step w' is orthogonal to V up to rounding, so a step normally takes three
// or four barriers instead of seven, and half the FP64 work.
//
// Bound: FP64 issue (~16 cycles a warp instruction) in C and D on large sectors, barriers and L2
// round trips on small ones.  Measured (FP64, real H):
// 1770 states, some 100 vectors: 45 -> 24 us a step; 47 895 states: 305 -> 85 us, of which 37 and 30 in
// C and D (63 000 cycles each are their FP64 instructions).
// Scalars are summed from per-block partials in one fixed order by every block, so all
// blocks hold identical values and take identical branches around the grid barriers.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace edgpu {

constexpr int kCoopThreads = 1024;
constexpr int kCoopWarps = kCoopThreads / 32;
constexpr int kCoopMaxBlocks = 1024;
constexpr int64_t kCoopMaxN = 65536;
constexpr int kCoopChunkRows = 448;  // rows of a chunk at most (65 536 rows on 147 SMs or more)
constexpr int kCoopSmemH = 1024;     // coefficients kept in shared memory
constexpr int kCoopFewChunks = 16;   // up to here every block adds up the partials itself

size_t reorth_coop_scratch_bytes() { return 3 * sizeof(double) * kCoopMaxBlocks; }

// Sum over the block in a fixed order, valid in every thread; buf: kCoopWarps + 1 doubles that no
// one else uses until the next barrier.
__device__ __forceinline__ double coop_block_sum(double v, double* buf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // warps without a value (most of them on small sectors) keep off the FP64 pipe
  if (__any_sync(0xffffffffu, (__double_as_longlong(v) << 1) != 0)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  __syncthreads();
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double t = buf[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) buf[kCoopWarps] = t;
  }
  __syncthreads();
  return buf[kCoopWarps];
}

// Sums of p[0..cnt) and q[0..cnt) (q may be null) in one fixed order (lane-strided, then an xor tree),
// returned to every thread of the block; identical bits in every block.
__device__ __forceinline__ void coop_fixed_sums(const double* p, const double* q, int cnt, double* bcast, double& sp,
                                                double& sq) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  const double* src = warp == 0 ? p : (warp == 1 ? q : nullptr);
  if (src) {
    double s = 0.0;
    for (int k = lane; k < cnt; k += 32) s += src[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) bcast[warp] = s;
  }
  __syncthreads();
  sp = bcast[0];
  sq = q ? bcast[1] : 0.0;
}

// (re, im) += conj(v) x in four fused operations (as a sum of products it compiles to six)
__device__ __forceinline__ void conj_fma(double& re, double& im, double2 v, double2 x) {
  re = fma(v.x, x.x, re);
  im = fma(v.x, x.y, im);
  re = fma(v.y, x.y, re);
  im = fma(-v.y, x.x, im);
}

// (re, im) summed over the warp: the halves of the warp take one component each after the first
// exchange, five additions instead of ten; lane 0 has re, lane 16 im.
__device__ __forceinline__ double coop_warp_sum2(double re, double im, int lane) {
  const bool hi = lane >= 16;
  double t = (hi ? im : re) + __shfl_xor_sync(0xffffffffu, hi ? re : im, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

struct CoopArgs {
  int64_t n;
  const int64_t* rp;
  const int32_t* col;
  const double* vals;
  const double2* v0;
  int j0, j1, K_cap;
  double2 *V, *w, *y;
  double *alpha, *beta;
  int32_t* status;
  double *pa, *pn, *pw;  // per-block partials of alpha, |w|^2 and |w'|^2
  double2 *pd, *hc;      // [m][chunks] partials of h, h
  int chunks;            // row chunks of phase C
  int sub;               // lanes per row of phase A
};

template <bool VALC>
__global__ void __launch_bounds__(kCoopThreads, 1) lanczos_reorth_coop_kernel(CoopArgs g) {
  cg::grid_group grid = cg::this_grid();
  const int B = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int64_t n = g.n;
  const int64_t gtid = (int64_t)b * kCoopThreads + tid, gthreads = (int64_t)B * kCoopThreads;
  __shared__ double red[kCoopWarps + 1];
  __shared__ double bc[2];
  __shared__ double beta_s[2];  // beta_{j-1} and its reciprocal
  __shared__ double2 ws[kCoopChunkRows];  // this block's chunk of w in phase C
  __shared__ double2 hs[kCoopSmemH];
  __shared__ double2 part[kCoopThreads];
  double2* const V = g.V;
  double2* const w = g.w;
  double2* const y = g.y;

  // phase C: block b is chunk b % chunks, vector group b / chunks
  const int C = g.chunks, groups = B / C, vg = b / C;
  const int64_t crows = (n + C - 1) / C, c0 = (int64_t)(b % C) * crows;
  const int cn = (int)(vg < groups && c0 < n ? (n - c0 < crows ? n - c0 : crows) : 0);
  // phase D: this block's rows, a lane per row of RW-row tiles, the other lanes and warps on
  // further vector classes
  const int64_t drows = (n + B - 1) / B, d0 = (int64_t)b * drows;
  const int dn = (int)(d0 < n ? (n - d0 < drows ? n - d0 : drows) : 0);
  const int RW = drows <= 8 ? 8 : (drows <= 16 ? 16 : 32);

  if (g.j0 == 0)
    for (int64_t i = gtid; i < n; i += gthreads) V[i] = g.v0[i];
  // only one thread takes roots and reciprocals: ~12 FP64 instructions of 32 warps would be 3 us
  if (tid == 0) {
    const double bp = g.j0 > 0 ? g.beta[g.j0 - 1] : 0.0;
    beta_s[0] = bp;
    beta_s[1] = bp > 0.0 ? 1.0 / bp : 0.0;
  }
  grid.sync();

  // h_k = <v_k, w> of the block's chunk (in ws) for its vector group
  auto dots = [&](int m) {
    if (cn > 0) {
      // two vectors a warp while there are enough for that: each element of w is read once for both
      const int own = (m - vg + groups - 1) / groups;  // vectors of this group
      const int pair = own >= 2 * kCoopWarps ? 2 : 1;
      for (int q = warp * pair; q < own; q += kCoopWarps * pair) {
        const int k = vg + groups * q;
        const bool two = pair == 2 && q + 1 < own;
        const double2* v0 = V + (int64_t)k * n + c0;
        const double2* v1 = two ? v0 + (int64_t)groups * n : v0;
        double ar = 0.0, am = 0.0, br = 0.0, bm = 0.0;
        if (two) {
#pragma unroll 4
          for (int r = lane; r < cn; r += 32) {
            const double2 v = v0[r], u = v1[r], x = ws[r];
            conj_fma(ar, am, v, x);
            conj_fma(br, bm, u, x);
          }
        } else {
#pragma unroll 4
          for (int r = lane; r < cn; r += 32) {
            const double2 v = v0[r], x = ws[r];
            conj_fma(ar, am, v, x);
          }
        }
        double* out = reinterpret_cast<double*>(g.pd + (int64_t)k * C + b % C);
        const double t = coop_warp_sum2(ar, am, lane);
        if (lane == 0) out[0] = t;
        if (lane == 16) out[1] = t;
        if (two) {
          out += 2 * (int64_t)groups * C;
          const double s = coop_warp_sum2(br, bm, lane);
          if (lane == 0) out[0] = s;
          if (lane == 16) out[1] = s;
        }
      }
    }
    grid.sync();
  };

  // the coefficients into hs (or g.hc where there are too many for it)
  auto coefficients = [&](int m) {
    const bool reduce = C > kCoopFewChunks || m > kCoopSmemH;
    if (reduce) {
      for (int k = b + B * warp; k < m; k += B * kCoopWarps) {
        double hr = 0.0, hm = 0.0;
        for (int c = lane; c < C; c += 32) {
          const double2 v = g.pd[(int64_t)k * C + c];
          hr += v.x;
          hm += v.y;
        }
        const double t = coop_warp_sum2(hr, hm, lane);
        double* out = reinterpret_cast<double*>(g.hc + k);
        if (lane == 0) out[0] = t;
        if (lane == 16) out[1] = t;
      }
      grid.sync();
    }
    if (m <= kCoopSmemH) {
      for (int k = tid; k < m; k += kCoopThreads) {
        double2 h = make_double2(0.0, 0.0);
        if (reduce) {
          h = g.hc[k];
        } else {
          for (int c = 0; c < C; ++c) {
            const double2 v = g.pd[(int64_t)k * C + c];
            h.x += v.x;
            h.y += v.y;
          }
        }
        hs[k] = h;
      }
    }
    __syncthreads();
  };

  // w -= V h on the block's rows; this thread's part of |w|^2
  auto project = [&](int m) -> double {
    const double2* h = m <= kCoopSmemH ? hs : g.hc;
    double nrm = 0.0;
    const int tiles = (dn + RW - 1) / RW;
    for (int t0 = 0; t0 < tiles; t0 += kCoopWarps) {
      const int nt = tiles - t0 < kCoopWarps ? tiles - t0 : kCoopWarps;
      const int wc = kCoopWarps / nt;                     // warps per tile
      const int tile = warp % nt, cls = (warp / nt) * (32 / RW) + lane / RW;
      const int classes = wc * (32 / RW);
      const int r = (t0 + tile) * RW + lane % RW;
      const bool on = warp / nt < wc && r < dn;
      // the rows this thread finishes below, in flight during the products
      int L = 8;
      while (L > 1 && nt * RW * L > kCoopThreads) L >>= 1;
      const int row = tid / L, q0 = tid % L, rr = t0 * RW + row;
      const bool last = q0 == 0 && row < nt * RW && rr < dn;
      double2 x = make_double2(0.0, 0.0);
      if (last) x = w[d0 + rr];
      double ar = 0.0, am = 0.0;
      if (on) {
        const double2* v = V + d0 + r;
#pragma unroll 4
        for (int k = cls; k < m; k += classes) {
          const double2 c = h[k], u = v[(int64_t)k * n];
          ar = fma(c.x, u.x, ar);
          am = fma(c.x, u.y, am);
          ar = fma(-c.y, u.y, ar);
          am = fma(c.y, u.x, am);
        }
      }
      __syncthreads();
      if (warp / nt < wc) part[(cls * nt + tile) * RW + lane % RW] = make_double2(ar, am);
      __syncthreads();
      // a row's classes summed by up to eight threads, then their sums
      if (warp * 32 / L < nt * RW) {  // warp-uniform: L divides 32
        double sr = 0.0, sm = 0.0;
        if (row < nt * RW)
          for (int q = q0; q < classes; q += L) {
            const double2 s = part[q * nt * RW + row];
            sr += s.x;
            sm += s.y;
          }
        for (int o = L >> 1; o > 0; o >>= 1) {
          sr += __shfl_xor_sync(0xffffffffu, sr, o);
          sm += __shfl_xor_sync(0xffffffffu, sm, o);
        }
        if (last) {
          x.x -= sr;
          x.y -= sm;
          w[d0 + rr] = x;
          nrm = fma(x.y, x.y, fma(x.x, x.x, nrm));
        }
      }
    }
    return nrm;
  };

  for (int j = g.j0; j < g.j1; ++j) {
    // ---- A
    double2* const vj = V + (int64_t)j * n;
    const double2* const vjm1 = j > 0 ? V + (int64_t)(j - 1) * n : nullptr;
    const bool raw = j > g.j0;  // v_j = w / beta_{j-1} is not written yet
    const double bprev = beta_s[0], ib = beta_s[1];
    const double2* const xs = raw ? w : vj;
    // rows dealt to the blocks one by one (the long rows are neighbours); their products collect in
    // shared memory, and the scaling, alpha and the stores run a row per thread, since an FP64
    // instruction costs the same for one lane as for 32
    const int sub = tid % g.sub, per_pass = kCoopThreads / g.sub;
    const int mine = (int)((n - b + B - 1) / B);  // this block's rows b, b + B, ...
    double ap = 0.0;
    for (int r0 = 0; r0 < mine; r0 += per_pass) {
      const int lr = r0 + tid / g.sub;
      const int k = r0 + tid;
      const bool dense = tid < per_pass && k < mine;
      double2 v = make_double2(0.0, 0.0);
      if (dense) v = xs[b + (int64_t)B * k];  // in flight during the gather
      if (r0 + (tid - lane) / g.sub < mine) {  // some row for this warp
        double yr = 0.0, yi = 0.0;
        if (lr < mine) {
          const int64_t i = b + (int64_t)B * lr;
          const int64_t e1 = g.rp[i + 1];
#pragma unroll 4
          for (int64_t e = g.rp[i] + sub; e < e1; e += g.sub) {
            const double2 x = xs[g.col[e]];
            if (VALC) {
              const double hr = g.vals[2 * e], hm = g.vals[2 * e + 1];
              yr = fma(-hm, x.y, fma(hr, x.x, yr));
              yi = fma(hm, x.x, fma(hr, x.y, yi));
            } else {
              const double hr = g.vals[e];
              yr += hr * x.x;
              yi += hr * x.y;
            }
          }
        }
        for (int o = g.sub >> 1; o > 0; o >>= 1) {
          yr += __shfl_xor_sync(0xffffffffu, yr, o);
          yi += __shfl_xor_sync(0xffffffffu, yi, o);
        }
        if (sub == 0 && lr < mine) part[tid / g.sub] = make_double2(yr, yi);
      }
      __syncthreads();
      if (dense) {
        const int64_t i = b + (int64_t)B * k;
        double2 p = part[tid];
        if (raw) {
          p.x *= ib;
          p.y *= ib;
          v.x *= ib;
          v.y *= ib;
          vj[i] = v;
        }
        ap = fma(v.y, p.y, fma(v.x, p.x, ap));
        y[i] = p;
      }
      __syncthreads();
    }
    ap = coop_block_sum(ap, red);
    if (tid == 0) g.pa[b] = ap;
    grid.sync();
    // ---- C
    double a, unused;
    coop_fixed_sums(g.pa, nullptr, B, bc, a, unused);
    if (b == 0 && tid == 0) g.alpha[j] = a;
    if (j + 1 >= g.K_cap) return;  // identical in every block
    const int m = j + 1;
    {
      double nw = 0.0;
      for (int r = tid; r < cn; r += kCoopThreads) {
        const int64_t i = c0 + r;
        double2 x = y[i];
        const double2 c = vj[i];
        x.x -= a * c.x;
        x.y -= a * c.y;
        if (vjm1) {
          const double2 p = vjm1[i];
          x.x -= bprev * p.x;
          x.y -= bprev * p.y;
        }
        ws[r] = x;
        if (vg == 0) {
          w[i] = x;
          nw = fma(x.y, x.y, fma(x.x, x.x, nw));
        }
      }
      nw = coop_block_sum(nw, red);  // also the barrier before ws is read
      if (tid == 0) g.pw[b] = nw;
    }
    dots(m);
    coefficients(m);
    // ---- D
    double nrm = coop_block_sum(project(m), red);
    if (tid == 0) g.pn[b] = nrm;
    grid.sync();
    double before, after;
    coop_fixed_sums(g.pw, g.pn, B, bc, before, after);
    if (after < 0.5 * before) {  // identical in every block; false for NaN
      for (int r = tid; r < cn; r += kCoopThreads) ws[r] = w[c0 + r];
      __syncthreads();
      dots(m);
      coefficients(m);
      nrm = coop_block_sum(project(m), red);
      if (tid == 0) g.pn[b] = nrm;
      grid.sync();
      coop_fixed_sums(g.pn, nullptr, B, bc, after, unused);
    }
    if (tid == 0) {
      const double bt = sqrt(after);
      beta_s[0] = bt;
      beta_s[1] = 1.0 / bt;
      if (b == 0) {
        g.beta[j] = bt;
        if (!(bt > 0.0)) atomicExch(g.status, (int32_t)(bt == 0.0 ? EDGPU_ERR_BREAKDOWN : EDGPU_ERR_NAN));
      }
    }
    __syncthreads();
    if (!(beta_s[0] > 0.0)) return;  // identical in every block
  }
  // the vector the next chunk starts from
  if (g.j1 > g.j0) {
    double2* vn = V + (int64_t)g.j1 * n;
    const double ib = beta_s[1];  // as phase A forms it, so that the bits do not depend on the chunks
    for (int64_t i = gtid; i < n; i += gthreads) {
      const double2 x = w[i];
      vn[i] = make_double2(x.x * ib, x.y * ib);
    }
  }
}

// Returns -1 when the sector is outside the cooperative kernel's range or the device cannot
// co-schedule the grid (caller uses the per-step kernels), else a status.  y [n], pd [K_cap + 1]
// [blocks of 256 rows, at most 8 an SM] and hc [K_cap + 1] come from the caller's workspace.
int lanczos_reorth_coop(const edgpu_csr* h, const double* v0, int j0, int j1, int K_cap, double* Vd, double* wd,
                        double* alpha, double* beta, int32_t* status_dev, double* scratch, double2* y, double2* pd,
                        double2* hc, cudaStream_t s) {
  if (h->n > kCoopMaxN || (!h->val_c && !h->val_r)) return -1;
  int dev = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) {
    cudaGetLastError();
    return -1;
  }
  auto kern = h->val_c ? lanczos_reorth_coop_kernel<true> : lanczos_reorth_coop_kernel<false>;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kCoopThreads, 0) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return -1;
  }
  int blocks = grid_cap();  // one block per SM
  if (blocks > kCoopMaxBlocks) blocks = kCoopMaxBlocks;
  CoopArgs g{};
  g.n = h->n;
  g.rp = h->row_ptr;
  g.col = h->col;
  g.vals = h->val_c ? h->val_c : h->val_r;
  g.v0 = reinterpret_cast<const double2*>(v0);
  g.j0 = j0;
  g.j1 = j1;
  g.K_cap = K_cap;
  g.V = reinterpret_cast<double2*>(Vd);
  g.w = reinterpret_cast<double2*>(wd);
  g.y = y;
  g.alpha = alpha;
  g.beta = beta;
  g.status = status_dev;
  g.pa = scratch;
  g.pn = scratch + kCoopMaxBlocks;
  g.pw = scratch + 2 * kCoopMaxBlocks;
  g.pd = pd;
  g.hc = hc;
  const int64_t want = (h->n + 255) / 256;
  g.chunks = (int)(want < blocks ? want : blocks);
  if ((h->n + g.chunks - 1) / g.chunks > kCoopChunkRows) return -1;
  // eight lanes a row while every row is gathered in one pass, fewer (and fewer additions of partial
  // sums) on larger sectors
  g.sub = h->n * 8 <= (int64_t)blocks * kCoopThreads ? 8 : 4;
  void* args[] = {&g};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)kern, blocks, kCoopThreads, args, 0, s);
  note_launch();
  if (e != cudaSuccess) {
    cudaGetLastError();
    return EDGPU_ERR_CUDA;
  }
  return check_launch();
}

}  // namespace edgpu
