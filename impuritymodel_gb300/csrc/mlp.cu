// BF16 multilayer perceptron over occupation bitstrings on the 5th-generation tensor cores.
//
// The network ranks candidate product states during basis pruning (no counterpart in
// upstream impurityModel, whose expand_basis keeps every state of the closure,
// impurityModel/ed/finite.py:1696-1803).  Its GEMMs run on tcgen05 fed by the tensor memory
// accelerator: a producer thread keeps a ring of K tiles in flight (2-D bulk-tensor copies
// into shared memory, completion on one mbarrier per stage), and a second thread issues
// tcgen05.mma (kind::f16, BF16 operands, FP32 accumulator in tensor memory) on each tile as
// it lands, never waiting for the MMAs themselves; every tile's MMAs commit to the stage's
// second mbarrier, which hands the stage back to the producer for the tile S ahead.
// The accumulator is read back with tcgen05.ld for a fused epilogue (bias, ReLU, ReLU mask,
// transposed copies for the backward pass) with 16-byte stores.
//
// One primitive covers forward and backward: C[M][N] = A[M][K] * B[N][K]^T with A and B
// row-major ("K-major") BF16, K a multiple of 64, M a multiple of 128, N a multiple of 16.
// The tile width (256, 64 or 16 columns) is the widest that still gives most SMs a tile.
// Every mbarrier wait has an iteration limit after which the kernel records
// EDGPU_ERR_NOCONV, waits (bounded) for its copies and MMAs still in flight, frees its tensor
// memory and returns.
#include <cuda_bf16.h>

#include "common.cuh"
#include "tma.cuh"

namespace edgpu {

constexpr int kGemmThreads = 128;  // 4 warps: tensor-memory lanes 0-127 = tile rows
constexpr int kBM = 128, kBK = 64;
constexpr uint32_t kSwizzleAtom = 1024;  // 8 rows x 128 bytes: one repeat of the 128-byte swizzle
constexpr long long kWaitLimit = 1LL << 24;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of a K-major operand in the 128-byte swizzled layout: rows
// of 64 BF16 (128 bytes) one after another, the 16-byte chunks of row r permuted by XOR with
// r % 8, groups of 8 rows 1024 bytes apart (SBO); the leading-dimension offset is unused in
// this layout (encoded as 1).  `saddr` is the tile base (1024-byte aligned) plus 32 bytes per
// 16-column K step.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;                     // LBO (unused)
  d |= (uint64_t)(kSwizzleAtom >> 4) << 32;   // SBO
  d |= (uint64_t)1 << 46;                     // descriptor version of the tcgen05 family
  d |= (uint64_t)2 << 61;                     // 128-byte swizzle; base offset 0
  return d;
}

// Instruction descriptor of kind::f16: D F32, A and B BF16, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* m, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* m, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint64_t* m, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(m)), "r"(phase)
      : "memory");
  return ok != 0;
}

// Bounded wait for the given phase of the barrier; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* m, uint32_t phase) {
  for (long long t = 0; t < kWaitLimit; ++t)
    if (mbar_test(m, phase)) return true;
  return false;
}

// Box {64 columns, box rows} of the 2-D BF16 tensor `map` at (column x, row y) into dst,
// 128-byte swizzled.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The barrier's next phase completes once every tcgen05 operation this thread issued so far
// has completed.
__device__ __forceinline__ void mma_commit(uint64_t* m) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(m))
               : "memory");
}

// 16 consecutive FP32 columns of this thread's tensor-memory lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

enum GemmEpilogue : int {
  kEpiStoreF32 = 0,   // C (float) = acc
  kEpiBiasRelu = 1,   // Y = relu(acc + bias[col]) -> BF16 Y[row][col] and Yt[col][row]
  kEpiReluMask = 2,   // Y = acc * (mask[row][col] > 0) -> BF16 Y and Yt
};

struct GemmArgs {
  const __nv_bfloat16* A;  // [M][K]
  const __nv_bfloat16* B;  // [N][K]
  int M, N, K;
  float* C;                  // kEpiStoreF32: [M][N]
  const float* bias;         // kEpiBiasRelu: [N]
  const __nv_bfloat16* mask; // kEpiReluMask: [M][N]
  __nv_bfloat16* Y;          // [M][N]
  __nv_bfloat16* Yt;         // [N][M] (may be null)
  int32_t* status;
  int vec;                   // C, Y and mask 16-byte aligned: 16-byte row stores and loads
};

// Shared-memory ring of a 128 x BN tile.  One stage holds the K tile (64 columns) of A and of
// B, each one 2-D bulk-tensor box {64, rows} in the 128-byte swizzled layout (one 128-byte
// request per row), each 1024-byte aligned.  The narrow 16-column tiles run only where the
// grid is small (a few row tiles, long K: the weight gradients), so they keep 8 stages in
// flight; the wider ones 4 or 3 (two or one CTAs per SM).
template <int BN>
struct GemmTile {
  static constexpr int kStages = BN <= 16 ? 8 : (BN >= 256 ? 3 : 4);
  static constexpr uint32_t kABytes = kBM * kBK * 2;          // 16 KiB
  static constexpr uint32_t kBBytes = BN * kBK * 2;
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;  // a multiple of 1 KiB
  static constexpr uint32_t kCols = BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
  static constexpr size_t kSmem = (size_t)kStages * kStageBytes + 1024;  // + alignment of the ring
};

// One output tile, rows from m0 and columns from n0 (the whole CTA).
template <int EPI, int BN>
__device__ __forceinline__ void gemm_tile(const CUtensorMap* amap, const CUtensorMap* bmap, const GemmArgs& g, int m0,
                                          int n0) {
  using T = GemmTile<BN>;
  constexpr int S = T::kStages;
  extern __shared__ unsigned char sm[];
  __shared__ uint64_t full[S], empty[S], done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ring = (smem_u32(sm) + 1023u) & ~1023u;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(T::kCols)
                 : "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&done, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  const int ktiles = g.K / kBK;
  if (warp == 1) {
    if (lane == 0) {
      // producer: K tile t into stage t % S once the MMAs of tile t - S have released it
      int issued = 0;
      bool ok = true;
      for (int t = 0; t < ktiles; ++t) {
        const int s = t % S;
        if (t >= S && !mbar_wait(&empty[s], (uint32_t)(t / S - 1) & 1u)) {
          ok = false;
          break;
        }
        if (*reinterpret_cast<volatile int*>(&failed)) break;  // the MMA side gave up
        const uint32_t a = ring + (uint32_t)s * T::kStageBytes, b = a + T::kABytes;
        mbar_expect_tx(&full[s], T::kStageBytes);
        tma_load_2d(a, amap, t * kBK, m0, &full[s]);
        tma_load_2d(b, bmap, t * kBK, n0, &full[s]);
        ++issued;
      }
      if (!ok) atomicExch(&failed, 1);
      // every copy issued has landed before the CTA may exit (earlier tiles of a stage were
      // consumed before its last one was issued)
      for (int t = issued > S ? issued - S : 0; t < issued; ++t) mbar_wait(&full[t % S], (uint32_t)(t / S) & 1u);
    }
    __syncwarp();
  } else if (warp == 0) {
    if (lane == 0) {
      // MMA issuer: never waits for MMAs, so they queue back to back in the tensor pipe
      const uint32_t idesc = idesc_bf16(kBM, BN);
      bool ok = true;
      for (int kt = 0; kt < ktiles; ++kt) {
        const int s = kt % S;
        if (!mbar_wait(&full[s], (uint32_t)(kt / S) & 1u)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a = ring + (uint32_t)s * T::kStageBytes, b = a + T::kABytes;
#pragma unroll
        for (int k16 = 0; k16 < kBK / 16; ++k16)
          mma_bf16(tmem, smem_desc_sw128(a + (uint32_t)k16 * 32u), smem_desc_sw128(b + (uint32_t)k16 * 32u), idesc,
                   (kt > 0 || k16 > 0) ? 1u : 0u);
        mma_commit(&empty[s]);  // releases the stage to the producer once these MMAs are done
      }
      mma_commit(&done);
      if (!ok) atomicExch(&failed, 1);
    }
    __syncwarp();
  }
  if (!mbar_wait(&done, 0u)) atomicExch(&failed, 1);
  __syncthreads();
  tc_fence_after();
  if (failed) {
    if (tid == 0) atomicExch(g.status, (int32_t)EDGPU_ERR_NOCONV);
  } else {
    // epilogue: warp w owns tensor-memory lanes (= tile rows) 32w .. 32w+31; M % 128 == 0
    // and N % BN == 0, so every row and column of the tile exists
    const int row = m0 + warp * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    for (int c0 = 0; c0 < BN; c0 += 16) {
      float v[16];
      tmem_ld16(trow + (uint32_t)c0, v);
      const int col0 = n0 + c0;
      const int64_t off = (int64_t)row * g.N + col0;
      if (EPI == kEpiStoreF32) {
        if (g.vec) {
          float4* dst = reinterpret_cast<float4*>(g.C + off);
#pragma unroll
          for (int q = 0; q < 4; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q) g.C[off + q] = v[q];
        }
        continue;
      }
      if (EPI == kEpiBiasRelu) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = fmaxf(v[q] + g.bias[col0 + q], 0.0f);
      }
      if (EPI == kEpiReluMask) {
        uint32_t mw[8];
        if (g.vec) {
          const uint4* src = reinterpret_cast<const uint4*>(g.mask + off);
          const uint4 m_lo = src[0], m_hi = src[1];
          mw[0] = m_lo.x, mw[1] = m_lo.y, mw[2] = m_lo.z, mw[3] = m_lo.w;
          mw[4] = m_hi.x, mw[5] = m_hi.y, mw[6] = m_hi.z, mw[7] = m_hi.w;
        } else {
          const unsigned short* src = reinterpret_cast<const unsigned short*>(g.mask + off);
#pragma unroll
          for (int q = 0; q < 8; ++q) mw[q] = (uint32_t)src[2 * q] | ((uint32_t)src[2 * q + 1] << 16);
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const float m = __uint_as_float(((mw[q >> 1] >> (16 * (q & 1))) & 0xFFFFu) << 16);  // BF16 -> FP32
          v[q] = m > 0.0f ? v[q] : 0.0f;
        }
      }
      uint32_t pk[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
        pk[q] = *reinterpret_cast<const uint32_t*>(&h);
      }
      if (g.vec) {
        uint4* dst = reinterpret_cast<uint4*>(g.Y + off);
        dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      } else {
        unsigned short* dst = reinterpret_cast<unsigned short*>(g.Y + off);
#pragma unroll
        for (int q = 0; q < 16; ++q) dst[q] = (unsigned short)(pk[q >> 1] >> (16 * (q & 1)));
      }
      if (g.Yt) {
        unsigned short* dst = reinterpret_cast<unsigned short*>(g.Yt);
#pragma unroll
        for (int q = 0; q < 16; ++q)  // lanes write consecutive rows: 64-byte runs per warp
          dst[(int64_t)(col0 + q) * g.M + row] = (unsigned short)(pk[q >> 1] >> (16 * (q & 1)));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kCols) : "memory");
}

template <int EPI, int BN>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemm_bf16_tc_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap,
                        GemmArgs g) {
  gemm_tile<EPI, BN>(&amap, &bmap, g, blockIdx.x * kBM, blockIdx.y * BN);
}

// Two products in one launch (blockIdx.z): the weight gradients have 32 and 40 narrow tiles with long
// chains of K tiles (22 us each at 4096 rows), so that one after the other they leave most SMs idle.
template <int EPI, int BN>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap a0, const __grid_constant__ CUtensorMap b0, GemmArgs g0,
                          const __grid_constant__ CUtensorMap a1, const __grid_constant__ CUtensorMap b1,
                          GemmArgs g1) {
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
  if (blockIdx.z == 0) {
    if (m0 < g0.M && n0 < g0.N) gemm_tile<EPI, BN>(&a0, &b0, g0, m0, n0);
  } else {
    if (m0 < g1.M && n0 < g1.N) gemm_tile<EPI, BN>(&a1, &b1, g1, m0, n0);
  }
}

// [rows][K] row-major BF16 as a 2-D tensor map with box {64 columns, box_rows rows}, 128-byte
// swizzled in shared memory.
bool gemm_operand_map(CUtensorMap* map, const __nv_bfloat16* ptr, int K, int rows, int box_rows) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int EPI, int BN>
int launch_gemm(const GemmArgs& g, cudaStream_t s) {
  using T = GemmTile<BN>;
  alignas(64) CUtensorMap amap, bmap;
  if (!gemm_operand_map(&amap, g.A, g.K, g.M, kBM) || !gemm_operand_map(&bmap, g.B, g.K, g.N, BN))
    return EDGPU_ERR_CUDA;
  auto* kern = gemm_bf16_tc_kernel<EPI, BN>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::kSmem) != cudaSuccess)
    return EDGPU_ERR_CUDA;
  dim3 grid(g.M / kBM, g.N / BN);
  kern<<<grid, kGemmThreads, T::kSmem, s>>>(amap, bmap, g);
  note_launch();
  return check_launch();
}

// Widest tile (256, 64 or 16 columns dividing N) that still gives about four fifths of the SMs
// a tile; the narrowest that divides N otherwise.
int gemm_tile_width(int M, int N) {
  const int64_t want = (int64_t)grid_cap() * 4 / 5;
  for (int bn : {256, 64, 16})
    if (N % bn == 0 && (int64_t)(M / kBM) * (N / bn) >= want) return bn;
  return 16;
}

template <int EPI>
int launch_gemm_bn(const GemmArgs& g, cudaStream_t s) {
  switch (gemm_tile_width(g.M, g.N)) {
    case 256:
      return launch_gemm<EPI, 256>(g, s);
    case 64:
      return launch_gemm<EPI, 64>(g, s);
    default:
      return launch_gemm<EPI, 16>(g, s);
  }
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int gemm_bf16(int epi, GemmArgs g, cudaStream_t s) {
  if (!g.A || !g.B || !g.status || g.M < 1 || g.N < 16 || g.K < kBK || g.K % kBK || g.N % 16 || g.M % kBM)
    return EDGPU_ERR_ARG;
  if (g.N / 16 > 65535) return EDGPU_ERR_ARG;  // grid.y = N / tile width
  if (!aligned16(g.A) || !aligned16(g.B)) return EDGPU_ERR_ARG;
  switch (epi) {
    case kEpiStoreF32:
      if (!g.C) return EDGPU_ERR_ARG;
      g.vec = aligned16(g.C);
      return launch_gemm_bn<kEpiStoreF32>(g, s);
    case kEpiBiasRelu:
      if (!g.Y || !g.bias) return EDGPU_ERR_ARG;
      g.vec = aligned16(g.Y);
      return launch_gemm_bn<kEpiBiasRelu>(g, s);
    case kEpiReluMask:
      if (!g.Y || !g.mask) return EDGPU_ERR_ARG;
      g.vec = aligned16(g.Y) && aligned16(g.mask);
      return launch_gemm_bn<kEpiReluMask>(g, s);
    default:
      return EDGPU_ERR_ARG;
  }
}

// ---------------------------------------------------------------------------------------
// Network pieces around the GEMMs (CUDA cores): input bits, output head, bias gradients,
// Adam, BF16 copies of the weights.
// ---------------------------------------------------------------------------------------

// X[b][i] = occupation of spin-orbital i (bit 63 - i%64 of word i/64) for i < n_in, BF16;
// Xt = X^T when not null.
__global__ void mlp_bits_kernel(const uint64_t* __restrict__ states, int W, int64_t B, int n_in,
                                __nv_bfloat16* __restrict__ X, __nv_bfloat16* __restrict__ Xt) {
  const int64_t total = B * (int64_t)n_in;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / n_in;
    const int i = (int)(t - b * n_in);
    const int q = i >> 6;
    float v = 0.0f;
    if (q < W) v = (float)((states[b * W + q] >> (63 - (i & 63))) & 1ull);
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    X[t] = h;
    if (Xt) Xt[(int64_t)i * B + b] = h;
  }
}

// y[b] = sum_j H[b][j] w3[j] + b3 (warp per row, FP32)
__global__ void mlp_head_kernel(const __nv_bfloat16* __restrict__ H, const float* __restrict__ w3, const float* b3,
                                int64_t B, int n_h, float* __restrict__ y) {
  const int lane = threadIdx.x & 31;
  for (int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < B;
       b += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    float acc = 0.0f;
    for (int j = lane; j < n_h; j += 32) acc += __bfloat162float(H[b * n_h + j]) * w3[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) y[b] = acc + b3[0];
  }
}

// Mean-squared-error head backward: dy = 2 (y - t) / B; dH[b][j] = dy w3[j] (H[b][j] > 0)
// as BF16 dH and dHt; loss partials per block.
__global__ void mlp_head_backward_kernel(const __nv_bfloat16* __restrict__ H, const float* __restrict__ y,
                                         const float* __restrict__ target, const float* __restrict__ w3, int64_t B,
                                         int n_h, float* __restrict__ dy, __nv_bfloat16* __restrict__ dH,
                                         __nv_bfloat16* __restrict__ dHt) {
  const int64_t total = B * (int64_t)n_h;
  const float inv = 2.0f / (float)B;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / n_h;
    const int j = (int)(t - b * n_h);
    const float d = (y[b] - target[b]) * inv;
    if (j == 0) dy[b] = d;
    const float g = __bfloat162float(H[t]) > 0.0f ? d * w3[j] : 0.0f;
    const __nv_bfloat16 gb = __float2bfloat16_rn(g);
    dH[t] = gb;
    dHt[(int64_t)j * B + b] = gb;
  }
}

// out[r] = sum_c M[r][c] * (v ? v[c] : 1) for a row-major [rows][cols] BF16 matrix, block per
// row, fixed-order reduction (bias gradients from the transposed activations / deltas).
__global__ void mlp_row_dot_kernel(const __nv_bfloat16* __restrict__ M, int rows, int64_t cols,
                                   const float* __restrict__ v, float* __restrict__ out) {
  __shared__ float red[32];
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    float acc = 0.0f;
    for (int64_t c = threadIdx.x; c < cols; c += blockDim.x)
      acc += __bfloat162float(M[(int64_t)r * cols + c]) * (v ? v[c] : 1.0f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.0f;
      for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += red[q];
      out[r] = t;
    }
    __syncthreads();
  }
}

// Adam on a flat FP32 parameter vector (bias-corrected step size lr_t from the host).
__global__ void mlp_adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                                float* __restrict__ v, int64_t n, float lr_t, float beta1, float beta2, float eps) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = beta1 * m[i] + (1.0f - beta1) * gi;
    const float vi = beta2 * v[i] + (1.0f - beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr_t * mi / (sqrtf(vi) + eps);
  }
}

// BF16 copy of a row-major [rows][cols] FP32 matrix, and of its transpose when Wt is set.
__global__ void mlp_to_bf16_kernel(const float* __restrict__ Wf, int rows, int cols, __nv_bfloat16* __restrict__ Wb,
                                   __nv_bfloat16* __restrict__ Wt) {
  const int64_t total = (int64_t)rows * cols;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(t / cols), c = (int)(t - (int64_t)r * cols);
    const __nv_bfloat16 h = __float2bfloat16_rn(Wf[t]);
    if (Wb) Wb[t] = h;
    if (Wt) Wt[(int64_t)c * rows + r] = h;
  }
}

// ---------------------------------------------------------------------------------------
// Ranking states: the whole network in one launch, occupation words in, scores out.
//
// Layer by layer, ranking 462 120 states moved 2.2 GB through memory (the BF16 occupation matrix
// written and read, both hidden layers written and read) for 18 MB of states and 2 MB of scores:
// 0.86 ms, a third of it the expansion of bits into BF16.  Here a CTA takes tiles of 128 states (two
// at a time when there are more tiles than SMs) and nothing but the words, the weights and the
// scores crosses global memory:
//   * the threads expand each state's words into a row of the A operand in shared memory (one
//     word is one 64-column K tile; four bits at a time from a 16-entry table); the fifth K tile
//     takes the first one's place once that has been read, so that A and two weight tiles fit;
//   * the weights stream through a two-stage ring of K tiles (bulk-tensor copies, 32 KiB each),
//     each tile feeding the MMAs of both state tiles;
//   * the first layer's accumulator (tensor memory, 256 columns a tile) is read back, bias, ReLU,
//     BF16, into the same A buffer as layer two's operand;
//   * layer two's accumulator is read back, and the head's sum runs in the threads.
// The BF16 roundings and the order of the K steps are those of the layer-by-layer kernels; the
// head's FP32 sum runs in another order.  Time for 462 120 states: 0.86 -> 0.138 ms.  Bound: the
// phases of a pass follow one another (expansion 1.7k cycles, layer one 6.7k, epilogue, layer two
// 5.3k, epilogue; the MMAs alone 9.2k).  With 8 epilogue warps and the biases read through L1 the
// epilogues took 4.7k and 7-9k cycles; 16 warps with the biases in shared memory took 0.03 ms off.
// A third weight stage (in the room of the biases) gained nothing.
// Every wait has an iteration limit, as in the GEMM above.
// ---------------------------------------------------------------------------------------
constexpr int kRankIn = 320, kRankHidden = 256;
constexpr int kRankChunks1 = kRankIn / kBK, kRankChunks2 = kRankHidden / kBK;
constexpr int kRankEpiThreads = 512;                    // 16 warps
constexpr int kRankThreads = kRankEpiThreads + 64;      // + producer warp + MMA warp
constexpr int kRankMmaWarp = kRankEpiThreads / 32;
constexpr int kRankQuarter = kRankHidden / 4;           // columns of an epilogue thread
constexpr uint32_t kRankABytes = kBM * kBK * 2;         // one K tile of 128 states: 16 KiB
constexpr uint32_t kRankTileBytes = kRankChunks2 * kRankABytes;  // the fifth K tile follows the first in its place
constexpr uint32_t kRankStageBytes = kRankHidden * kBK * 2;
constexpr int kRankStages = 2;
constexpr size_t kRankSmem = 2 * (size_t)kRankTileBytes + kRankStages * (size_t)kRankStageBytes + 1024;

__device__ __forceinline__ void mbar_arrive(uint64_t* m) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(m)) : "memory");
}

// Shared-memory writes of this thread become visible to the tensor core and the copy engine.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// 16 consecutive FP32 columns of this thread's tensor-memory lane; the registers hold them after
// tmem_wait_ld.
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// Ties the registers of earlier loads to the wait, so that nothing reads them before it.
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16], uint32_t (&s)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 16; ++q) asm volatile("" : "+r"(r[q]), "+r"(s[q]));
}

// relu(v + b) of two columns as a BF16 pair.  The maximum is taken after the rounding (monotone, so
// the same value) to work on both at once; like fmaxf it makes a NaN 0.
__device__ __forceinline__ __nv_bfloat162 bias_relu2(uint32_t v0, uint32_t v1, float b0, float b1) {
  const float2 x = __fadd2_rn(make_float2(__uint_as_float(v0), __uint_as_float(v1)), make_float2(b0, b1));
  return __hmax2(__floats2bfloat162_rn(x.x, x.y), __float2bfloat162_rn(0.0f));
}

struct RankArgs {
  const uint64_t* states;  // [n][W]
  int W;
  int64_t n;
  const float *b1, *b2, *w3, *b3;
  float* y;
  int tiles;        // 128-state tiles per pass of a CTA: 1 or 2
  int64_t passes;   // over the whole launch
  int32_t* status;
};

__global__ void __launch_bounds__(kRankThreads, 1)
    mlp_rank_kernel(const __grid_constant__ CUtensorMap w1map, const __grid_constant__ CUtensorMap w2map, RankArgs g) {
  extern __shared__ unsigned char sm[];
  __shared__ uint64_t full[kRankStages], empty[kRankStages], a_full, acc_full, first_read, last_full, quarter_sums, drained;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  __shared__ uint2 nibble[16];
  __shared__ float part[3][2 * kBM];
  __shared__ __align__(16) float sb1[kRankHidden], sb2[kRankHidden], sw3[kRankHidden];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t abuf = (smem_u32(sm) + 1023u) & ~1023u;
  const uint32_t ring = abuf + 2 * kRankTileBytes;
  if (warp == kRankMmaWarp)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(512u)
                 : "memory");
  if (tid == 0) {
    for (int s = 0; s < kRankStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&a_full, kRankEpiThreads);
    mbar_init(&acc_full, 1);
    mbar_init(&first_read, 1);
    mbar_init(&last_full, kRankEpiThreads);
    mbar_init(&quarter_sums, kRankEpiThreads / 4 * 3);
    mbar_init(&drained, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 16)  // four occupation bits, first column in the highest, as four BF16
    nibble[tid] = make_uint2(((tid & 8) ? 0x3F80u : 0u) | ((tid & 4) ? 0x3F800000u : 0u),
                             ((tid & 2) ? 0x3F80u : 0u) | ((tid & 1) ? 0x3F800000u : 0u));
  for (int k = tid; k < kRankHidden; k += kRankThreads) {
    sb1[k] = g.b1[k];
    sb2[k] = g.b2[k];
    sw3[k] = g.w3[k];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  volatile int* gave_up = &failed;
  if (warp == kRankMmaWarp + 1) {
    if (lane == 0) {
      // producer: the K tiles of W1 then W2 for every pass
      int64_t it = 0;
      bool ok = true;
      for (int64_t p = blockIdx.x; ok && p < g.passes; p += gridDim.x) {
        for (int c = 0; c < kRankChunks1 + kRankChunks2; ++c, ++it) {
          const int s = (int)(it % kRankStages);
          if (it >= kRankStages && !mbar_wait(&empty[s], (uint32_t)(it / kRankStages - 1) & 1u)) ok = false;
          if (!ok || *gave_up) {
            ok = false;
            break;
          }
          mbar_expect_tx(&full[s], kRankStageBytes);
          const bool first = c < kRankChunks1;
          tma_load_2d(ring + (uint32_t)s * kRankStageBytes, first ? &w1map : &w2map,
                      (first ? c : c - kRankChunks1) * kBK, 0, &full[s]);
        }
      }
      if (!ok) atomicExch(&failed, 1);
      // every copy issued has landed before the CTA may exit
      for (int64_t t = it > kRankStages ? it - kRankStages : 0; t < it; ++t)
        mbar_wait(&full[t % kRankStages], (uint32_t)(t / kRankStages) & 1u);
    }
    __syncwarp();
  } else if (warp == kRankMmaWarp) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(kBM, kRankHidden);
      int64_t it = 0;
      uint32_t pass_phase = 0;
      bool ok = true;
      for (int64_t p = blockIdx.x; ok && p < g.passes; p += gridDim.x, pass_phase ^= 1u) {
        for (int layer = 0; ok && layer < 2; ++layer) {
          // the A operand is written and the accumulator's last contents have been read
          if (!mbar_wait(&a_full, (uint32_t)layer)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const int chunks = layer ? kRankChunks2 : kRankChunks1;
          for (int c = 0; c < chunks; ++c, ++it) {
            const int s = (int)(it % kRankStages);
            if (!mbar_wait(&full[s], (uint32_t)(it / kRankStages) & 1u) ||
                (c == kRankChunks2 && !mbar_wait(&last_full, pass_phase))) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t b = ring + (uint32_t)s * kRankStageBytes;
            for (int q = 0; q < g.tiles; ++q) {
              const uint32_t a = abuf + (uint32_t)q * kRankTileBytes + (uint32_t)(c % kRankChunks2) * kRankABytes;
#pragma unroll
              for (int k16 = 0; k16 < kBK / 16; ++k16)
                mma_bf16(tmem + (uint32_t)(q * kRankHidden), smem_desc_sw128(a + (uint32_t)k16 * 32u),
                         smem_desc_sw128(b + (uint32_t)k16 * 32u), idesc, (c > 0 || k16 > 0) ? 1u : 0u);
            }
            mma_commit(&empty[s]);
            if (layer == 0 && c == 0) mma_commit(&first_read);
          }
          if (ok) mma_commit(&acc_full);
        }
      }
      if (!ok) atomicExch(&failed, 1);
      // no MMA is in flight when the tensor memory is freed
      mma_commit(&drained);
      if (!mbar_wait(&drained, 0u)) atomicExch(&failed, 1);
    }
    __syncwarp();
  } else {
    // Expansion: threads tid and tid + 256 write state tid of the pass.  Epilogues: the thread reads
    // its warp's tensor-memory lane (a state of each tile) in 64 of the 256 columns, so that a bias
    // value is loaded once for two states, and four warps a scheduler hide the loads' latency.
    const int row = ((warp & 3) << 5) + lane, quarter = warp >> 2;
    const int xs = tid & (2 * kBM - 1), xhalf = tid / (2 * kBM);
    const uint32_t xrow = abuf + (uint32_t)(xs / kBM) * kRankTileBytes + (uint32_t)(xs % kBM) * 128u;
    const uint32_t hrow = abuf + (uint32_t)row * 128u + (uint32_t)quarter * kRankABytes;
    const uint32_t sw = (uint32_t)(row & 7), xsw = (uint32_t)(xs & 7);
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(quarter * kRankQuarter);
    const bool two = g.tiles == 2;
    uint32_t pass_phase = 0;
    bool ok = true;
    uint64_t words[3];  // two K tiles and the shared fifth of the thread's state, loaded a pass ahead
    auto fetch = [&](int64_t p) {
      const int64_t i = p * g.tiles * kBM + xs;
      const bool on = xs < g.tiles * kBM && p < g.passes && i < g.n;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int c = k < 2 ? 2 * xhalf + k : kRankChunks2;
        words[k] = on && c < g.W ? __ldg(g.states + i * g.W + c) : 0ull;
      }
    };
    // byte q of the word, from the top, is piece `piece` (16 bytes, eight columns) of the K tile
    auto expand = [&](uint64_t word, int q, int chunk, int piece) {
      const uint2 h = nibble[(word >> (60 - 8 * q)) & 15u], l = nibble[(word >> (56 - 8 * q)) & 15u];
      st_shared_v4(xrow + (uint32_t)chunk * kRankABytes + ((((uint32_t)piece) ^ xsw) << 4), h.x, h.y, l.x, l.y);
    };
    fetch(blockIdx.x);
    for (int64_t p = blockIdx.x; ok && p < g.passes; p += gridDim.x, pass_phase ^= 1u) {
      const int64_t base = p * g.tiles * kBM;
#pragma unroll
      for (int q = 0; q < 16; ++q) expand(words[q >> 3], q & 7, 2 * xhalf + (q >> 3), q & 7);
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(&a_full);
      // the fifth K tile takes the first one's place once the MMAs have read that
      ok = __all_sync(0xffffffffu, mbar_wait(&first_read, pass_phase) && !*gave_up);
      if (!ok) break;
#pragma unroll
      for (int q = 0; q < 4; ++q) expand(words[2] << (32 * xhalf), q, 0, q + 4 * xhalf);
      fence_async_smem();
      mbar_arrive(&last_full);
      fetch(p + gridDim.x);
      // one answer for the warp: its tensor-memory loads are collective
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full, 0u) && !*gave_up);
      if (!ok) break;
      tc_fence_after();
      for (int c0 = 0; c0 < kRankQuarter; c0 += 16) {
        uint32_t v[16], u[16];
        tmem_ld16_async(trow + (uint32_t)c0, v);
        if (two) tmem_ld16_async(trow + (uint32_t)(kRankHidden + c0), u);
        tmem_wait_ld(v, u);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float4* bias = reinterpret_cast<const float4*>(sb1 + quarter * kRankQuarter + c0 + 8 * q);
          const float4 bl = bias[0], bh = bias[1];
          const float bb[8] = {bl.x, bl.y, bl.z, bl.w, bh.x, bh.y, bh.z, bh.w};
          const uint32_t at = hrow + (((uint32_t)(c0 / 8 + q) ^ sw) << 4);
          uint32_t pk[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const __nv_bfloat162 h = bias_relu2(v[8 * q + 2 * k], v[8 * q + 2 * k + 1], bb[2 * k], bb[2 * k + 1]);
            pk[k] = *reinterpret_cast<const uint32_t*>(&h);
          }
          st_shared_v4(at, pk[0], pk[1], pk[2], pk[3]);
          if (two) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const __nv_bfloat162 h = bias_relu2(u[8 * q + 2 * k], u[8 * q + 2 * k + 1], bb[2 * k], bb[2 * k + 1]);
              pk[k] = *reinterpret_cast<const uint32_t*>(&h);
            }
            st_shared_v4(at + kRankTileBytes, pk[0], pk[1], pk[2], pk[3]);
          }
        }
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(&a_full);
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full, 1u) && !*gave_up);
      if (!ok) break;
      tc_fence_after();
      // head: eight partial sums a state in packed pairs, added up, then the four quarters
      float2 s[4], z[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) s[k] = z[k] = make_float2(0.0f, 0.0f);
      for (int c0 = 0; c0 < kRankQuarter; c0 += 16) {
        uint32_t v[16], u[16];
        tmem_ld16_async(trow + (uint32_t)c0, v);
        if (two) tmem_ld16_async(trow + (uint32_t)(kRankHidden + c0), u);
        tmem_wait_ld(v, u);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int at = quarter * kRankQuarter + c0 + 4 * q, k = 2 * (q & 1);
          const float4 b = *reinterpret_cast<const float4*>(sb2 + at), w = *reinterpret_cast<const float4*>(sw3 + at);
          const float2 w01 = make_float2(w.x, w.y), w23 = make_float2(w.z, w.w);
          s[k] = __ffma2_rn(__bfloat1622float2(bias_relu2(v[4 * q], v[4 * q + 1], b.x, b.y)), w01, s[k]);
          s[k + 1] = __ffma2_rn(__bfloat1622float2(bias_relu2(v[4 * q + 2], v[4 * q + 3], b.z, b.w)), w23, s[k + 1]);
          if (two) {
            z[k] = __ffma2_rn(__bfloat1622float2(bias_relu2(u[4 * q], u[4 * q + 1], b.x, b.y)), w01, z[k]);
            z[k + 1] = __ffma2_rn(__bfloat1622float2(bias_relu2(u[4 * q + 2], u[4 * q + 3], b.z, b.w)), w23, z[k + 1]);
          }
        }
      }
      const float2 ss = __fadd2_rn(__fadd2_rn(s[0], s[1]), __fadd2_rn(s[2], s[3]));
      const float2 zz = __fadd2_rn(__fadd2_rn(z[0], z[1]), __fadd2_rn(z[2], z[3]));
      if (quarter > 0) {
        part[quarter - 1][row] = ss.x + ss.y;
        part[quarter - 1][kBM + row] = zz.x + zz.y;
        mbar_arrive(&quarter_sums);
      } else {
        // one answer for the warp here too: a lane that gave up alone would be missing from the next vote
        ok = __all_sync(0xffffffffu, mbar_wait(&quarter_sums, pass_phase));
        if (!ok) break;
        const float b3 = __ldg(g.b3);
        if (base + row < g.n) g.y[base + row] = ((ss.x + ss.y) + part[0][row]) + (part[1][row] + part[2][row]) + b3;
        if (two && base + kBM + row < g.n)
          g.y[base + kBM + row] =
              ((zz.x + zz.y) + part[0][kBM + row]) + (part[1][kBM + row] + part[2][kBM + row]) + b3;
      }
      // the next pass writes part only after the first quarter has arrived on a_full again
    }
    if (!ok) atomicExch(&failed, 1);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (failed && tid == 0) atomicExch(g.status, (int32_t)EDGPU_ERR_NOCONV);
  if (warp == kRankMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

int mlp_rank(const RankArgs& args, const __nv_bfloat16* W1, const __nv_bfloat16* W2, cudaStream_t s) {
  RankArgs g = args;
  alignas(64) CUtensorMap w1map, w2map;
  if (!gemm_operand_map(&w1map, W1, kRankIn, kRankHidden, kRankHidden) ||
      !gemm_operand_map(&w2map, W2, kRankHidden, kRankHidden, kRankHidden))
    return EDGPU_ERR_CUDA;
  const int64_t tiles = (g.n + kBM - 1) / kBM;
  // two tiles a pass share each weight tile; with no more tiles than SMs one each is faster
  g.tiles = tiles > grid_cap() ? 2 : 1;
  g.passes = (tiles + g.tiles - 1) / g.tiles;
  if (cudaFuncSetAttribute(mlp_rank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRankSmem) != cudaSuccess)
    return EDGPU_ERR_CUDA;
  const unsigned grid = (unsigned)(g.passes < grid_cap() ? g.passes : grid_cap());
  mlp_rank_kernel<<<grid, kRankThreads, kRankSmem, s>>>(w1map, w2map, g);
  note_launch();
  return check_launch();
}

inline unsigned mlp_grid(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)grid_cap() * 8;
  return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

// ---------------------------------------------------------------------------------------
// One training step in eight launches (edgpu_mlp_train_step): what the layer-by-layer calls do, with
// the pieces around the GEMMs fused and issued from one call.  As single calls a step was 23
// launches, 0.138 ms on the device and 0.29 ms in the program (batch 4096); what the pieces compute,
// and in what order they add it up, is unchanged, except for the sum of dy (the gradient of b3) and the
// loss.  Eight batches of 4096: 2.26 -> 0.81 ms a call, 0.06 ms a step on the device (0.022 of it the
// weight gradients).
// ---------------------------------------------------------------------------------------
constexpr int kStepRows = 32;  // batch rows per block of the element-wise pieces

// X and X^T of the states idx[b] (or b): a row's words once into shared memory, 16-byte stores both ways.
__global__ void __launch_bounds__(256) mlp_step_bits_kernel(const uint64_t* __restrict__ states, int W,
                                                            const int64_t* __restrict__ idx, int64_t B,
                                                            __nv_bfloat16* __restrict__ X,
                                                            __nv_bfloat16* __restrict__ Xt) {
  constexpr int NW = kRankIn / 64;
  __shared__ uint64_t word[kStepRows][NW];
  __shared__ uint2 nibble[16];
  const int tid = threadIdx.x;
  const int64_t b0 = (int64_t)blockIdx.x * kStepRows;
  if (tid < 16)
    nibble[tid] = make_uint2(((tid & 8) ? 0x3F80u : 0u) | ((tid & 4) ? 0x3F800000u : 0u),
                             ((tid & 2) ? 0x3F80u : 0u) | ((tid & 1) ? 0x3F800000u : 0u));
  if (tid < kStepRows * NW) {
    const int r = tid / NW, q = tid % NW;
    const int64_t s = idx ? idx[b0 + r] : b0 + r;
    word[r][q] = q < W ? states[s * W + q] : 0ull;
  }
  __syncthreads();
  uint4* x = reinterpret_cast<uint4*>(X + b0 * kRankIn);
  for (int t = tid; t < kStepRows * kRankIn / 8; t += 256) {
    const int r = t / (kRankIn / 8), q = t % (kRankIn / 8);
    const uint32_t byte = (uint32_t)(word[r][q >> 3] >> (56 - 8 * (q & 7))) & 255u;
    const uint2 h = nibble[byte >> 4], l = nibble[byte & 15u];
    x[t] = make_uint4(h.x, h.y, l.x, l.y);
  }
  for (int t = tid; t < kRankIn * kStepRows / 8; t += 256) {
    const int i = t / (kStepRows / 8), g = t % (kStepRows / 8);
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t lo = (uint32_t)(word[8 * g + 2 * k][i >> 6] >> (63 - (i & 63))) & 1u;
      const uint32_t hi = (uint32_t)(word[8 * g + 2 * k + 1][i >> 6] >> (63 - (i & 63))) & 1u;
      v[k] = lo * 0x3F80u | hi * 0x3F800000u;
    }
    *reinterpret_cast<uint4*>(Xt + (int64_t)i * B + b0 + 8 * g) = make_uint4(v[0], v[1], v[2], v[3]);
  }
}

// Head forward and backward of kStepRows rows: scores, dy, dH2 and its transpose, the squared error.
__global__ void __launch_bounds__(256) mlp_step_head_kernel(const __nv_bfloat16* __restrict__ H,
                                                            const float* __restrict__ target,
                                                            const int64_t* __restrict__ idx,
                                                            const float* __restrict__ w3, const float* __restrict__ b3,
                                                            int64_t B, float* __restrict__ dy,
                                                            __nv_bfloat16* __restrict__ dH,
                                                            __nv_bfloat16* __restrict__ dHt,
                                                            float* __restrict__ err) {
  __shared__ __align__(16) __nv_bfloat16 h[kStepRows][kRankHidden + 8];
  __shared__ float w[kRankHidden], d[kStepRows], e2[kStepRows];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t b0 = (int64_t)blockIdx.x * kStepRows;
  w[tid] = w3[tid];
  for (int t = tid; t < kStepRows * kRankHidden / 8; t += 256) {
    const int r = t / (kRankHidden / 8), q = t % (kRankHidden / 8);
    *reinterpret_cast<uint4*>(&h[r][8 * q]) = reinterpret_cast<const uint4*>(H + (b0 + r) * kRankHidden)[q];
  }
  __syncthreads();
  const float inv = 2.0f / (float)B;
  for (int r = warp; r < kStepRows; r += 8) {
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < kRankHidden / 32; ++j) acc += __bfloat162float(h[r][32 * j + lane]) * w[32 * j + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const float y = acc + b3[0], diff = y - target[idx ? idx[b0 + r] : b0 + r];
      d[r] = diff * inv;
      e2[r] = diff * diff;
      dy[b0 + r] = d[r];
    }
  }
  __syncthreads();
  auto grad = [&](int r, int j) -> uint32_t {
    const float g = __bfloat162float(h[r][j]) > 0.0f ? d[r] * w[j] : 0.0f;
    const __nv_bfloat16 gb = __float2bfloat16_rn(g);
    return (uint32_t)*reinterpret_cast<const unsigned short*>(&gb);
  };
  for (int t = tid; t < kStepRows * kRankHidden / 8; t += 256) {
    const int r = t / (kRankHidden / 8), q = t % (kRankHidden / 8);
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = grad(r, 8 * q + 2 * k) | grad(r, 8 * q + 2 * k + 1) << 16;
    reinterpret_cast<uint4*>(dH + (b0 + r) * kRankHidden)[q] = make_uint4(v[0], v[1], v[2], v[3]);
  }
#pragma unroll
  for (int g = 0; g < kStepRows / 8; ++g) {  // column tid
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = grad(8 * g + 2 * k, tid) | grad(8 * g + 2 * k + 1, tid) << 16;
    *reinterpret_cast<uint4*>(dHt + (int64_t)tid * B + b0 + 8 * g) = make_uint4(v[0], v[1], v[2], v[3]);
  }
  if (warp == 0) {
    float s = e2[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) err[blockIdx.x] = s;
  }
}

__device__ __forceinline__ float block_sum256(float acc, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  float t = 0.0f;
  if (threadIdx.x == 0)
    for (int q = 0; q < 8; ++q) t += red[q];
  __syncthreads();
  return t;  // thread 0
}

// Gradients of w3, b2 and b1 (blockIdx.y 0, 1, 2; a row per block, the sums of mlp_row_dot_kernel), and
// in one more block those of b3 and the loss.
__global__ void __launch_bounds__(256) mlp_step_dots_kernel(const __nv_bfloat16* __restrict__ H2t,
                                                            const __nv_bfloat16* __restrict__ dH2t,
                                                            const __nv_bfloat16* __restrict__ dH1t,
                                                            const float* __restrict__ dy,
                                                            const float* __restrict__ err, int64_t B,
                                                            float* __restrict__ gw3, float* __restrict__ gb2,
                                                            float* __restrict__ gb1, float* __restrict__ gb3,
                                                            float* __restrict__ loss) {
  __shared__ float red[8];
  const int r = blockIdx.x;
  if (r == kRankHidden) {
    if (blockIdx.y != 0) return;
    float acc = 0.0f, e = 0.0f;
    for (int64_t c = threadIdx.x; c < B; c += 256) acc += dy[c];
    for (int64_t c = threadIdx.x; c < B / kStepRows; c += 256) e += err[c];
    const float s = block_sum256(acc, red), t = block_sum256(e, red);
    if (threadIdx.x == 0) {
      gb3[0] = s;
      loss[0] = t / (float)B;
    }
    return;
  }
  const __nv_bfloat16* M = (blockIdx.y == 0 ? H2t : (blockIdx.y == 1 ? dH2t : dH1t)) + (int64_t)r * B;
  float acc = 0.0f;
  if (blockIdx.y == 0) {
    for (int64_t c = threadIdx.x; c < B; c += 256) acc += __bfloat162float(M[c]) * dy[c];
  } else {
    for (int64_t c = threadIdx.x; c < B; c += 256) acc += __bfloat162float(M[c]);
  }
  const float s = block_sum256(acc, red);
  if (threadIdx.x == 0) (blockIdx.y == 0 ? gw3 : (blockIdx.y == 1 ? gb2 : gb1))[r] = s;
}

// Adam on the flat parameters (W1, b1, W2, b2, w3, b3) with the BF16 copies of W1, W2 and W2^T.
__global__ void __launch_bounds__(256) mlp_step_adam_kernel(float* __restrict__ p, const float* __restrict__ g,
                                                            float* __restrict__ m, float* __restrict__ v, int n,
                                                            float lr_t, float beta1, float beta2, float eps,
                                                            __nv_bfloat16* __restrict__ W1b,
                                                            __nv_bfloat16* __restrict__ W2b,
                                                            __nv_bfloat16* __restrict__ W2t) {
  constexpr int kW1 = kRankHidden * kRankIn, kW2 = kW1 + kRankHidden;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = beta1 * m[i] + (1.0f - beta1) * gi;
    const float vi = beta2 * v[i] + (1.0f - beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float x = p[i] - lr_t * mi / (sqrtf(vi) + eps);
    p[i] = x;
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    if (i < kW1) {
      W1b[i] = h;
    } else if (i >= kW2 && i < kW2 + kRankHidden * kRankHidden) {
      const int k = i - kW2;
      W2b[k] = h;
      W2t[(k % kRankHidden) * kRankHidden + k / kRankHidden] = h;
    }
  }
}

struct StepSpace {
  __nv_bfloat16 *X, *Xt, *H1, *H1t, *H2, *H2t, *dH2, *dH2t, *dH1, *dH1t;
  float *dy, *err;
  size_t bytes;
};

StepSpace step_space(void* ws, int64_t B) {
  StepSpace s{};
  unsigned char* base = reinterpret_cast<unsigned char*>(ws);
  auto carve = [&](size_t bytes) {
    unsigned char* q = base + s.bytes;
    s.bytes += (bytes + 255) & ~(size_t)255;
    return q;
  };
  auto matrix = [&](int cols) { return reinterpret_cast<__nv_bfloat16*>(carve(2 * (size_t)B * cols)); };
  s.X = matrix(kRankIn);
  s.Xt = matrix(kRankIn);
  for (__nv_bfloat16** q : {&s.H1, &s.H1t, &s.H2, &s.H2t, &s.dH2, &s.dH2t, &s.dH1, &s.dH1t}) *q = matrix(kRankHidden);
  s.dy = reinterpret_cast<float*>(carve(sizeof(float) * (size_t)B));
  s.err = reinterpret_cast<float*>(carve(sizeof(float) * (size_t)(B / kStepRows + 1)));
  return s;
}

}  // namespace edgpu

using namespace edgpu;

extern "C" int edgpu_gemm_bf16_epi(int epi, const void* A, const void* B, int M, int N, int K, float* C,
                                   const float* bias, const void* mask, void* Y, void* Yt, int32_t* status_dev,
                                   void* stream) {
  GemmArgs g{};
  g.A = reinterpret_cast<const __nv_bfloat16*>(A);
  g.B = reinterpret_cast<const __nv_bfloat16*>(B);
  g.M = M;
  g.N = N;
  g.K = K;
  g.C = C;
  g.bias = bias;
  g.mask = reinterpret_cast<const __nv_bfloat16*>(mask);
  g.Y = reinterpret_cast<__nv_bfloat16*>(Y);
  g.Yt = reinterpret_cast<__nv_bfloat16*>(Yt);
  g.status = status_dev;
  return gemm_bf16(epi, g, (cudaStream_t)stream);
}

extern "C" int edgpu_mlp_bits(const uint64_t* states, int W, int64_t B, int n_in, void* X, void* Xt, void* stream) {
  if (!states || W < 1 || B < 1 || n_in < 1 || !X) return EDGPU_ERR_ARG;
  mlp_bits_kernel<<<mlp_grid(B * n_in, 256), 256, 0, (cudaStream_t)stream>>>(
      states, W, B, n_in, reinterpret_cast<__nv_bfloat16*>(X), reinterpret_cast<__nv_bfloat16*>(Xt));
  note_launch();
  return check_launch();
}

extern "C" int edgpu_mlp_head(const void* H, const float* w3, const float* b3, int64_t B, int n_h, float* y,
                              void* stream) {
  if (!H || !w3 || !b3 || B < 1 || n_h < 1 || !y) return EDGPU_ERR_ARG;
  mlp_head_kernel<<<mlp_grid(B * 32, 256), 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(H), w3, b3, B, n_h, y);
  note_launch();
  return check_launch();
}

extern "C" int edgpu_mlp_rank(const uint64_t* states, int W, int64_t n, int n_in, int n_h, const void* W1,
                              const float* b1, const void* W2, const float* b2, const float* w3, const float* b3,
                              float* y, int32_t* status_dev, void* stream) {
  if (!states || W < 1 || n < 1 || !W1 || !b1 || !W2 || !b2 || !w3 || !b3 || !y || !status_dev) return EDGPU_ERR_ARG;
  if (n_in != kRankIn || n_h != kRankHidden) return EDGPU_ERR_ARG;
  if (!aligned16(W1) || !aligned16(W2)) return EDGPU_ERR_ARG;
  RankArgs g{};
  g.states = states;
  g.W = W;
  g.n = n;
  g.b1 = b1;
  g.b2 = b2;
  g.w3 = w3;
  g.b3 = b3;
  g.y = y;
  g.status = status_dev;
  return mlp_rank(g, reinterpret_cast<const __nv_bfloat16*>(W1), reinterpret_cast<const __nv_bfloat16*>(W2),
                  (cudaStream_t)stream);
}

extern "C" size_t edgpu_mlp_step_workspace(int64_t B) {
  return B < kBM || B % kBM ? 0 : step_space(nullptr, B).bytes + 256;
}

extern "C" int edgpu_mlp_train_step(const uint64_t* states, int W, const int64_t* idx, const float* target, int64_t B,
                                    int n_in, int n_h, float* P, float* G, float* m, float* v, void* W1b, void* W2b,
                                    void* W2t, float lr_t, float beta1, float beta2, float eps, float* loss,
                                    int32_t* status_dev, void* workspace, size_t workspace_bytes, void* stream) {
  if (!states || W < 1 || !target || B < kBM || B % kBM || B > 0x7fffffff || !P || !G || !m || !v) return EDGPU_ERR_ARG;
  if (n_in != kRankIn || n_h != kRankHidden || !W1b || !W2b || !W2t || !loss || !status_dev || !workspace)
    return EDGPU_ERR_ARG;
  if (workspace_bytes < edgpu_mlp_step_workspace(B)) return EDGPU_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  const StepSpace w = step_space(
      reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~(uintptr_t)255), B);
  constexpr int kW1 = kRankHidden * kRankIn, kW2 = kRankHidden * kRankHidden;
  const int ob1 = kW1, oW2 = ob1 + kRankHidden, ob2 = oW2 + kW2, ow3 = ob2 + kRankHidden, ob3 = ow3 + kRankHidden;
  auto bf = [](void* q) { return reinterpret_cast<__nv_bfloat16*>(q); };
  const int M = (int)B;
  const unsigned blocks = (unsigned)(B / kStepRows);
  int rc;
  mlp_step_bits_kernel<<<blocks, 256, 0, s>>>(states, W, idx, B, w.X, w.Xt);
  note_launch();
  auto layer = [&](const __nv_bfloat16* A, const __nv_bfloat16* Bm, int K, const float* bias,
                   const __nv_bfloat16* mask, __nv_bfloat16* Y, __nv_bfloat16* Yt) {
    GemmArgs g{};
    g.A = A;
    g.B = Bm;
    g.M = M;
    g.N = kRankHidden;
    g.K = K;
    g.bias = bias;
    g.mask = mask;
    g.Y = Y;
    g.Yt = Yt;
    g.status = status_dev;
    return gemm_bf16(mask ? kEpiReluMask : kEpiBiasRelu, g, s);
  };
  if ((rc = layer(w.X, bf(W1b), kRankIn, P + ob1, nullptr, w.H1, w.H1t))) return rc;
  if ((rc = layer(w.H1, bf(W2b), kRankHidden, P + ob2, nullptr, w.H2, w.H2t))) return rc;
  mlp_step_head_kernel<<<blocks, 256, 0, s>>>(w.H2, target, idx, P + ow3, P + ob3, B, w.dy, w.dH2, w.dH2t, w.err);
  note_launch();
  if ((rc = layer(w.dH2, bf(W2t), kRankHidden, nullptr, w.H1, w.dH1, w.dH1t))) return rc;
  // both weight gradients
  {
    constexpr int BN = 16;
    using T = GemmTile<BN>;
    GemmArgs g0{}, g1{};
    g0.M = g1.M = kRankHidden;
    g0.N = kRankHidden;
    g1.N = kRankIn;
    g0.K = g1.K = M;
    g0.C = G + oW2;
    g1.C = G;
    g0.status = g1.status = status_dev;
    g0.vec = aligned16(g0.C);
    g1.vec = aligned16(g1.C);
    alignas(64) CUtensorMap a0, b0, a1, b1;
    if (!gemm_operand_map(&a0, w.dH2t, M, kRankHidden, kBM) || !gemm_operand_map(&b0, w.H1t, M, kRankHidden, BN) ||
        !gemm_operand_map(&a1, w.dH1t, M, kRankHidden, kBM) || !gemm_operand_map(&b1, w.Xt, M, kRankIn, BN))
      return EDGPU_ERR_CUDA;
    auto* kern = gemm_bf16_pair_kernel<kEpiStoreF32, BN>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::kSmem) != cudaSuccess)
      return EDGPU_ERR_CUDA;
    kern<<<dim3(kRankHidden / kBM, kRankIn / BN, 2), kGemmThreads, T::kSmem, s>>>(a0, b0, g0, a1, b1, g1);
    note_launch();
  }
  mlp_step_dots_kernel<<<dim3(kRankHidden + 1, 3), 256, 0, s>>>(w.H2t, w.dH2t, w.dH1t, w.dy, w.err, B, G + ow3, G + ob2,
                                                               G + ob1, G + ob3, loss);
  note_launch();
  const int n = ob3 + 1;
  mlp_step_adam_kernel<<<(n + 255) / 256, 256, 0, s>>>(P, G, m, v, n, lr_t, beta1, beta2, eps, bf(W1b), bf(W2b), bf(W2t));
  note_launch();
  return check_launch();
}

extern "C" int edgpu_mlp_head_backward(const void* H, const float* y, const float* target, const float* w3,
                                       int64_t B, int n_h, float* dy, void* dH, void* dHt, void* stream) {
  if (!H || !y || !target || !w3 || B < 1 || n_h < 1 || !dy || !dH || !dHt) return EDGPU_ERR_ARG;
  mlp_head_backward_kernel<<<mlp_grid(B * n_h, 256), 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(H), y, target, w3, B, n_h, dy, reinterpret_cast<__nv_bfloat16*>(dH),
      reinterpret_cast<__nv_bfloat16*>(dHt));
  note_launch();
  return check_launch();
}

extern "C" int edgpu_mlp_row_dot(const void* M, int rows, int64_t cols, const float* v, float* out, void* stream) {
  if (!M || rows < 1 || cols < 1 || !out) return EDGPU_ERR_ARG;
  mlp_row_dot_kernel<<<rows < 4096 ? rows : 4096, 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(M), rows, cols, v, out);
  note_launch();
  return check_launch();
}

extern "C" int edgpu_mlp_adam(float* p, const float* g, float* m, float* v, int64_t n, float lr_t, float beta1,
                              float beta2, float eps, void* stream) {
  if (!p || !g || !m || !v || n < 1) return EDGPU_ERR_ARG;
  mlp_adam_kernel<<<mlp_grid(n, 256), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, lr_t, beta1, beta2, eps);
  note_launch();
  return check_launch();
}

extern "C" int edgpu_mlp_to_bf16(const float* Wf, int rows, int cols, void* Wb, void* Wt, void* stream) {
  if (!Wf || rows < 1 || cols < 1 || (!Wb && !Wt)) return EDGPU_ERR_ARG;
  mlp_to_bf16_kernel<<<mlp_grid((int64_t)rows * cols, 256), 256, 0, (cudaStream_t)stream>>>(
      Wf, rows, cols, reinterpret_cast<__nv_bfloat16*>(Wb), reinterpret_cast<__nv_bfloat16*>(Wt));
  note_launch();
  return check_launch();
}

extern "C" int edgpu_gemm_tile_width(int M, int N) {
  if (M < kBM || M % kBM || N < 16 || N % 16 || N / 16 > 65535) return 0;
  return gemm_tile_width(M, N);
}

extern "C" int edgpu_gemm_bf16(const void* A, const void* B, int M, int N, int K, float* C, int32_t* status_dev,
                               void* stream) {
  GemmArgs g{};
  g.A = reinterpret_cast<const __nv_bfloat16*>(A);
  g.B = reinterpret_cast<const __nv_bfloat16*>(B);
  g.M = M;
  g.N = N;
  g.K = K;
  g.C = C;
  g.status = status_dev;
  return gemm_bf16(kEpiStoreF32, g, (cudaStream_t)stream);
}
