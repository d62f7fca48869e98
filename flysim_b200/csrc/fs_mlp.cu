// Mean-field surrogate: a small MLP (BF16 weights and activations, FP32
// accumulation) trained and evaluated with hand-written 5th-generation
// tensor-core kernels.  It has no counterpart in the reference; it maps sweep
// parameters (per-group drive, excitatory and inhibitory gains) to
// per-region firing rates and a hyperactivity logit, and screens parameter
// grids whose candidates the simulator then verifies.
//
// GEMM: C[M x N] = A[M x K] . B[N x K]^T, A and B BF16 row-major (K
// contiguous).  One CTA per 128-row tile holds the whole K (<= 256) and N
// (<= 256) in shared memory in the no-swizzle K-major core-matrix layout
// (8 rows x 16 bytes per core matrix); one thread issues K/16 tcgen05.mma
// (kind::f16, BF16 x BF16 -> FP32) into a TMEM accumulator; tcgen05.commit
// arrives on an mbarrier; the four warps read their 32 TMEM lanes back
// (tcgen05.ld 32x32b) for a fused epilogue: bias, ReLU, the ReLU mask of the
// backward pass, FP32 / BF16 / transposed-BF16 outputs.
//
// Training: an epoch is one persistent launch, k_train, for networks whose
// weights are at most as many tiles of 128 x 16 as there are SMs beside its
// sixteen row CTAs (132 on 148 SMs: four layers of 256 x 256); larger ones replay
// a CUDA graph of one Adam step (forward GEMMs, loss, gradient GEMMs, bias sums,
// Adam updates; batch index and Adam step count live in device counters).
// Inference: k_forward, all layers in one launch.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <numeric>
#include <random>
#include <string>
#include <thread>
#include <utility>
#include <vector>
#include <sys/mman.h>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include "flysim_b200.h"
#include "fs_barrier.cuh"

namespace fsm {

typedef __nv_bfloat16 bf16;
constexpr int kThreads = 128;  // four warps: one quarter of the 128 TMEM lanes each
constexpr int kTileM = 128;
constexpr uint32_t kSpin = 1u << 26;  // bounded mbarrier wait

struct GemmArgs {
  const bf16 *A;
  int lda;
  const bf16 *B;
  int ldb;
  int M, N, K;
  const float *bias;  // [N] or null
  int relu;
  const bf16 *mask;   // [M x N]: output zeroed where mask <= 0 (ReLU backward), or null
  int ldm;
  float *Cf;          // FP32 [M x N] or null
  int ldcf;
  bf16 *Cb;           // BF16 [M x N] or null
  int ldcb;
  bf16 *Ct;           // BF16 [N x M] (transposed) or null
  int ldct;
  int *err;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor (no swizzle, K-major): `lbo` = bytes
// between the two 8-element K halves of a 16-wide K step, `sbo` = bytes
// between consecutive 8-row groups; descriptor version 1.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  return d;  // base offset 0, legacy LBO mode, layout type 0 (no swizzle)
}

// Instruction descriptor, kind::f16: D FP32, A and B BF16, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t M, uint32_t N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      :
      : "r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

constexpr int kKC = 64;   // K columns per load chunk (4 MMAs, one mbarrier)
constexpr int kCW = 64;   // output columns per epilogue chunk
constexpr int kSP = kCW + 4;  // staging row pitch (floats)
constexpr int kMaxChunks = 256 / kKC;

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < kSpin; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Grid: x over 128-row tiles, y over column tiles of g.N / gridDim.y columns.
// Operands arrive by TMA (cp.async.bulk.tensor, no swizzle): each 8-wide K
// column of a tile is one box of rows x 16 bytes, which is exactly a stack
// of K-major core matrices (8 rows x 16 bytes, 128 bytes apart), so one
// thread issues every box of the tile up front, K chunk by K chunk on its
// own mbarrier, and starts each chunk's MMAs as soon as it lands.  Rows past
// M are the TMA's zero fill.  The epilogue goes through shared memory
// (reusing the operand space once the accumulator is complete) so that
// every global store is coalesced.
__global__ void __launch_bounds__(kThreads) k_gemm_tn(const __grid_constant__ GemmArgs g,
                                                      const __grid_constant__ CUtensorMap ta,
                                                      const __grid_constant__ CUtensorMap tb) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int K = g.K, N = g.N / (int)gridDim.y, nkb = K >> 3;  // 8-wide K columns
  const int n0 = blockIdx.y * N;  // first column of this CTA
  uint8_t *sA = smem;                              // nkb boxes of 128 rows x 16 B
  uint8_t *sB = smem + (size_t)nkb * kTileM * 16;  // nkb boxes of N rows x 16 B
  const size_t opnd = (size_t)nkb * (kTileM + N) * 16, stage = (size_t)kTileM * kSP * 4;
  uint64_t *mbar = (uint64_t *)(smem + (opnd > stage ? opnd : stage));  // [0] MMA, [1..] K chunks
  uint32_t *tslot = (uint32_t *)(mbar + 1 + kMaxChunks);
  float *stg = (float *)smem;                      // epilogue staging [128][kSP]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * kTileM;
  const int nch = (K + kKC - 1) / kKC;
  uint32_t ncols = 32;
  while (ncols < (uint32_t)N) ncols <<= 1;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                 "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    for (int c = 0; c <= nch; c++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(mbar + c)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tslot;
  bool loads_ok = true;
  if (tid == 0) {
    // every box of the tile, chunk by chunk
    for (int c = 0; c < nch; c++) {
      const int kb0 = c * (kKC / 8), kb1 = min(nkb, kb0 + kKC / 8);
      const uint32_t bytes = (uint32_t)(kb1 - kb0) * (uint32_t)(kTileM + N) * 16u;
      const uint32_t bar = smem_u32(mbar + 1 + c);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
      for (int kb = kb0; kb < kb1; kb++) {
        tma_load_2d(smem_u32(sA + (size_t)kb * kTileM * 16), &ta, kb * 8, m0, bar);
        tma_load_2d(smem_u32(sB + (size_t)kb * N * 16), &tb, kb * 8, n0, bar);
      }
    }
    // MMAs as the chunks land: slab s (16 wide) = boxes 2s (LBO away: 2s+1)
    const uint32_t id = idesc_bf16(kTileM, (uint32_t)N);
    for (int c = 0; c < nch && loads_ok; c++) {
      loads_ok = mbar_wait(smem_u32(mbar + 1 + c), 0);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int s0 = c * (kKC / 16), s1 = min(K >> 4, s0 + kKC / 16);
      for (int sl = s0; sl < s1 && loads_ok; sl++) {
        const uint64_t ad = sdesc(smem_u32(sA + (size_t)(2 * sl) * kTileM * 16), kTileM * 16, 128);
        const uint64_t bd = sdesc(smem_u32(sB + (size_t)(2 * sl) * N * 16), (uint32_t)N * 16, 128);
        mma_bf16(tmem, ad, bd, id, sl > 0 ? 1u : 0u);
      }
    }
    if (!loads_ok) {
      if (g.err) atomicExch(g.err, 4);
      for (int c = 0; c < nch; c++) mbar_wait(smem_u32(mbar + 1 + c), 0);  // no copy outlives the CTA
    }
  }
  if (tid == 0)
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                     smem_u32(mbar))
                 : "memory");
  // wait for the accumulator (bounded); the commit covers every MMA issued
  const bool ok = mbar_wait(smem_u32(mbar), 0);
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (!ok) {
    if (g.err && tid == 0) atomicExch(g.err, 3);
  } else {
    const int rl = warp * 32 + lane;  // this thread's accumulator row
    for (int cc = 0; cc < N; cc += kCW) {
      const int cw = min(kCW, N - cc);
      // TMEM -> registers -> (bias, ReLU) -> staging
      for (int c0 = 0; c0 < cw; c0 += 16) {
        uint32_t v[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(cc + c0), v);
#pragma unroll
        for (int j = 0; j < 16; j++) {
          float x = __uint_as_float(v[j]);
          if (g.bias) x += g.bias[n0 + cc + c0 + j];
          if (g.relu) x = fmaxf(x, 0.0f);
          stg[rl * kSP + c0 + j] = x;
        }
      }
      __syncthreads();
      const int rows = min(kTileM, g.M - m0);
      // row-major outputs: 8 consecutive columns per thread, coalesced
      const int c8 = cw >> 3;
      for (int i = tid; i < rows * c8; i += kThreads) {
        const int r = i / c8, c = (i - r * c8) * 8;
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = stg[r * kSP + c + j];
        const size_t gc = (size_t)n0 + cc + c;
        if (g.mask) {
          const uint4 mv = *(const uint4 *)(g.mask + (size_t)(m0 + r) * g.ldm + gc);
          const bf16 *mb = (const bf16 *)&mv;
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (!(__bfloat162float(mb[j]) > 0.0f)) x[j] = 0.0f;
#pragma unroll
          for (int j = 0; j < 8; j++) stg[r * kSP + c + j] = x[j];  // masked values for the transposed store
        }
        if (g.Cf) {
          float4 *dst = (float4 *)(g.Cf + (size_t)(m0 + r) * g.ldcf + gc);
          dst[0] = make_float4(x[0], x[1], x[2], x[3]);
          dst[1] = make_float4(x[4], x[5], x[6], x[7]);
        }
        if (g.Cb) {
          uint4 o;
          bf16 *ob = (bf16 *)&o;
#pragma unroll
          for (int j = 0; j < 8; j++) ob[j] = __float2bfloat16_rn(x[j]);
          *(uint4 *)(g.Cb + (size_t)(m0 + r) * g.ldcb + gc) = o;
        }
      }
      if (g.Ct) {
        __syncthreads();
        // transposed: consecutive threads take consecutive rows of one column
        for (int i = tid; i < rows * cw; i += kThreads) {
          const int c = i / rows, r = i - c * rows;
          g.Ct[((size_t)n0 + cc + c) * g.ldct + m0 + r] = __float2bfloat16_rn(stg[r * kSP + c]);
        }
      }
      __syncthreads();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(ncols));
}

size_t gemm_smem(int N, int K) {
  const size_t opnd = (size_t)(K / 8) * (kTileM + N) * 16, stage = (size_t)kTileM * kSP * 4;
  return (opnd > stage ? opnd : stage) + 8 * (1 + kMaxChunks) + 16;
}

// 2-D tensor map of a row-major BF16 matrix (rows x cols, leading dimension
// ld elements) read in boxes of box_rows rows x 8 columns (16 bytes)
typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_fn = nullptr;

int make_map(CUtensorMap *map, const bf16 *ptr, int rows, int cols, int ld, int box_rows, std::string &err) {
  if (!encode_fn) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn ||
        q != cudaDriverEntryPointSuccess) {
      err = "gemm: cuTensorMapEncodeTiled is not available";
      return FS_ERR_CUDA;
    }
    encode_fn = (EncodeTiled)fn;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {8u, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUresult r = encode_fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)ptr, dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    err = "gemm: tensor map encoding failed (" + std::to_string((int)r) + ")";
    return FS_ERR_ARG;
  }
  return FS_OK;
}

bool gemm_attr_set = false;

// Checks the shape rules and launches one GEMM.
int gemm(const GemmArgs &g, cudaStream_t st, std::string &err) {
  if (g.N < 16 || g.N > 256 || g.N % 16 || g.K < 16 || g.K > 256 || g.K % 16 || g.M < 1 || g.lda % 8 ||
      g.ldb % 8 || ((uintptr_t)g.A & 15) || ((uintptr_t)g.B & 15) ||
      (g.Cf && (g.ldcf % 4 || ((uintptr_t)g.Cf & 15))) || (g.Cb && (g.ldcb % 8 || ((uintptr_t)g.Cb & 15))) ||
      (g.mask && (g.ldm % 8 || ((uintptr_t)g.mask & 15)))) {
    err = "gemm: N and K must be multiples of 16 in [16, 256], leading dimensions multiples of 8 (4 for "
          "FP32 output), operands and outputs 16-byte aligned";
    return FS_ERR_ARG;
  }
  if (!gemm_attr_set) {
    cudaFuncSetAttribute(k_gemm_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(256, 256));
    gemm_attr_set = true;
  }
  // column tiles of 64 when there are few row tiles (every GEMM of the framework
  // itself: batches of up to 256 rows), so that small-M GEMMs still spread over
  // the SMs; one column tile otherwise (checks of many rows)
  const int tiles = (g.M + kTileM - 1) / kTileM;
  const int ny = (g.N % 64 == 0 && tiles < 296) ? g.N / 64 : 1;
  const dim3 grid((g.M + kTileM - 1) / kTileM, ny);
  CUtensorMap ta, tb;
  int rc = make_map(&ta, g.A, g.M, g.K, g.lda, kTileM, err);
  if (!rc) rc = make_map(&tb, g.B, g.N, g.K, g.ldb, g.N / ny, err);
  if (rc) return rc;
  k_gemm_tn<<<grid, kThreads, gemm_smem(g.N / ny, g.K), st>>>(g, ta, tb);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("gemm launch: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  return FS_OK;
}

// ---- element-wise kernels of the MLP -----------------------------------------

// rows of x (FP32, `cols` wide; row r taken from perm[ctr*rows + r] when
// perm is given) -> BF16 X [rows x pcols] and optionally X^T [pcols x ldt]
__global__ void k_stage_x(const float *x, int rows, int cols, int pcols, const int *perm, const int *ctr, bf16 *X,
                          bf16 *XT, int ldt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * pcols) return;
  const int r = i / pcols, c = i - r * pcols;
  const size_t src = perm ? (size_t)perm[(size_t)(*ctr) * rows + r] : (size_t)r;
  const float v = c < cols ? x[src * cols + c] : 0.0f;
  const bf16 b = __float2bfloat16_rn(v);
  X[(size_t)r * pcols + c] = b;
  if (XT) XT[(size_t)c * ldt + r] = b;
}

__global__ void k_stage_t(const float *t, int rows, int cols, int pcols, const int *perm, const int *ctr, float *T) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * pcols) return;
  const int r = i / pcols, c = i - r * pcols;
  const size_t src = perm ? (size_t)perm[(size_t)(*ctr) * rows + r] : (size_t)r;
  T[i] = c < cols ? t[src * cols + c] : 0.0f;
}

// One output's loss and gradient: column c of nr regressions and a logit.
__device__ __forceinline__ void loss_element(float y, float t, int c, int nr, int rows, float &l, float &d) {
  l = d = 0.0f;
  if (c < nr) {
    const float e = y - t;
    d = 2.0f * e / (float)(nr * rows);
    l = e * e / (float)(nr * rows);
  } else if (c == nr) {
    const float p = 1.0f / (1.0f + expf(-y));
    d = (p - t) / (float)rows;
    l = (fmaxf(y, 0.0f) - y * t + log1pf(expf(-fabsf(y)))) / (float)rows;
  }
}

// Loss and output-layer gradient.  Columns [0, nr) regress log-rates (mean
// squared error averaged over nr columns and the rows), column nr is the
// hyperactivity logit (binary cross-entropy averaged over the rows); padded
// columns get zero gradient.
__global__ void k_loss(const float *Z, const float *T, int rows, int pcols, int nr, bf16 *dZ, bf16 *dZT, int ldt,
                       float *loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.0f;
  if (i < rows * pcols) {
    const int r = i / pcols, c = i - r * pcols;
    float d;
    loss_element(Z[i], T[i], c, nr, rows, l, d);
    const bf16 b = __float2bfloat16_rn(d);
    dZ[i] = b;
    dZT[(size_t)c * ldt + r] = b;
  }
  for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0 && l != 0.0f) atomicAdd(loss, l);
}

// bias gradient: row sums of dZ^T, one warp per output unit
__global__ void k_bias_grad(const bf16 *dZT, int ldt, int rows, int n, float *gb) {
  const int c = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= n) return;
  float s = 0.0f;
  for (int r = lane; r < rows; r += 32) s += __bfloat162float(dZT[(size_t)c * ldt + r]);
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) gb[c] = s;
}

// One weight's Adam update; c1, c2: the bias corrections of this step.
__device__ __forceinline__ void adam_update(float &w, float &m, float &v, float gi, float lr, float c1, float c2) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  m = __fmaf_rn(1.0f - b1, gi, __fmul_rn(b1, m));  // one contraction in every kernel
  v = __fmaf_rn(__fmul_rn(1.0f - b2, gi), gi, __fmul_rn(b2, v));
  // (a weight that never had a gradient: the step is exactly 0, and its
  // zero operands would take the divisions' slow path)
  if (m != 0.0f || v != 0.0f) w = w - lr * (m / c1) / (sqrtf(v / c2) + eps);
}
__device__ __forceinline__ void adam_corrections(int step, float &c1, float &c2) {
  const float t = (float)(step + 1);
  c1 = 1.0f - powf(0.9f, t);
  c2 = 1.0f - powf(0.999f, t);
}

// Adam on the FP32 master copy (step count from the device counter), then the
// BF16 copies W and W^T.
__global__ void k_adam(float *w, float *m, float *v, const float *g, int n, int rows, int cols, float lr,
                       const int *ctr, bf16 *Wb, bf16 *Wt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float c1, c2, wi = w[i], mi = m[i], vi = v[i];
  adam_corrections(ctr[1], c1, c2);
  adam_update(wi, mi, vi, g[i], lr, c1, c2);
  m[i] = mi;
  v[i] = vi;
  w[i] = wi;
  if (Wb) {
    const bf16 b = __float2bfloat16_rn(wi);
    Wb[i] = b;
    const int r = i / cols, c = i - r * cols;
    Wt[(size_t)c * rows + r] = b;
  }
}

__global__ void k_step_end(int *ctr) {
  ctr[0] += 1;  // batch within the epoch
  ctr[1] += 1;  // Adam step
}

// W's BF16 copies: row-major, transposed, and blocked (the order k_forward and
// k_train stream: 128 rows x 64 columns as eight boxes of 128 rows x 16 bytes)
__global__ void k_refresh(const float *w, int rows, int cols, bf16 *Wb, bf16 *Wt, bf16 *Wk) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * cols) return;
  const bf16 b = __float2bfloat16_rn(w[i]);
  Wb[i] = b;
  const int r = i / cols, c = i - r * cols;
  Wt[(size_t)c * rows + r] = b;
  Wk[(size_t)(r / 128 * ((cols + 63) / 64) + c / 64) * 8192 + (size_t)((c & 63) >> 3) * 1024 + (r & 127) * 8 + (c & 7)] = b;
}

// ---- persistent training kernel ----------------------------------------------
// One launch runs an epoch's Adam steps over batches of kBatch = 256 rows.  The
// network's row dependencies decide the split: given the weights, forward and
// backward of a row need no other row, so kRowCtas CTAs take kRowsCta = 16 rows
// each through all layers with no exchange; only the weight gradients sum over
// rows, and a CTA per 128 x 16 tile of a layer's weights forms its sum, keeps
// the tile's weights and Adam moments in registers for the launch and updates
// them.  Two grid barriers a step.
//
// Row CTAs: D[features x rows] = W . H^T, so an epilogue thread owns a feature
// with its 16 rows; it writes the next layer's operand to shared memory and the
// transposed activations the gradient tiles read with two coalesced 16-byte
// stores.  The weights (0.6 MB a step, more than shared memory) stream from L2
// through a ring of 16 KB chunks (two to a slot), contiguous in the blocked layout the tile
// CTAs write: [128 rows x 64 k] as eight boxes of 128 rows x 16 bytes, the
// no-swizzle K-major core-matrix order.  Every accumulator sums the same
// products over K in the same order as k_gemm_tn.
//
// The step this replaces was 28 graph nodes, each a launch of a few CTAs: 146 us
// for about 1 us of tensor work; now 22.6 us (surrogate, 32-256-256-256-59).
// What bounds it is the chain of small products (seven of them, each waits for
// its operand, its accumulator and its epilogue), the tile update (about 9,000
// cycles: load, product, Adam with its IEEE divisions, publication) and the
// two barriers (2,000 each).
constexpr int kBatch = 256;     // training rows per step
constexpr int kRowsCta = 16, kRowCtas = kBatch / kRowsCta;
constexpr int kMaxTrainL = 24;
constexpr int kTrThreads = 320;  // warps 0-7 epilogues, 8 copies, 9 MMAs
constexpr int kRing = 4;         // slots of two 16 KB chunks (a K chunk of up to two row tiles)
constexpr uint32_t kChunkB = 16384;
// Bytes between the 8-wide K boxes of a row CTA's operand ([K/8][16 rows][8] and
// 16 bytes of padding, so that the lanes of a feature store hit four times the
// banks)
constexpr uint32_t kHsBox = kRowsCta * 16 + 16;
constexpr int kTileN = 16;       // weight columns of a tile CTA

struct TrainLayer {
  int in, out;           // padded widths
  bf16 *Wk, *Wt;         // blocked W [out x in] and W^T [in x out]
  bf16 *HT;              // the layer's input, transposed: [in/kTileN][row/8][kTileN][8]
  bf16 *dZT;             // its output gradient, transposed: [out/128][row/8][128][8]
  float *W, *mW, *vW, *b, *mb, *vb;
};
struct TrainArgs {
  TrainLayer l[kMaxTrainL];
  int L, steps, din, dout, tiles;
  const float *x, *t;
  const int *perm;
  const uint32_t *tile;  // layer | out tile << 8 | in tile << 16
  float lr;
  float *loss;
  int *ctr;
  unsigned int *bar;
  int *err;
};

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// Waits (bounded) for the ring's copies in flight, so that a CTA that leaves after
// a wait gave up leaves none behind: slot, ph: the issuing thread's next slot and
// its round's parity (a slot never filled passes at once).
__device__ __forceinline__ void drain_ring(const uint64_t *full, int slots, uint32_t slot, uint32_t ph) {
  for (uint32_t c = 0; c < (uint32_t)slots; c++) mbar_wait(smem_u32(full + c), c < slot ? ph : ph ^ 1u);
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;\n" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ uint32_t bf2(float a, float b) {
  const __nv_bfloat162 v = __halves2bfloat162(__float2bfloat16_rn(a), __float2bfloat16_rn(b));
  return *(const uint32_t *)&v;
}

// barriers in shared memory
struct TrainBars {
  uint64_t full[kRing], empty[kRing], done;
  uint32_t tmem;
  int src[2][kRowsCta];
  int fail;
};

// The products of one step of a row CTA: forward layers, then backward ones.
template <class F>
__device__ __forceinline__ void for_stages(const TrainArgs &g, F &&f) {
  for (int l = 0; l < g.L; l++) f(l, false, g.l[l].Wk, g.l[l].out, g.l[l].in);
  for (int l = g.L - 1; l > 0; l--) f(l, true, g.l[l].Wt, g.l[l].in, g.l[l].out);
}

// Sixteen rows through the network (CTAs [0, kRowCtas)).
__device__ __forceinline__ void train_rows(const TrainArgs &g, uint8_t *smem, TrainBars &B) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = (int)blockIdx.x * kRowsCta, L = g.L;
  bf16 *Hs = (bf16 *)(smem + kRing * 2 * kChunkB);  // operand, K-major boxes kHsBox apart
  const uint32_t hs = smem_u32(Hs), tmem = B.tmem, done = smem_u32(&B.done);
  unsigned long long target = 0;
  uint32_t slot = 0, ph = 0;  // copies and MMAs: chunk slot and its round's parity
  uint32_t dph = 0;           // parity of `done`
  bool ok = true;
  const int p0 = g.l[0].in;
  // rows of step s and their inputs into the operand buffer
  auto rows_of = [&](int s) {
    if (tid < kRowsCta) B.src[s & 1][tid] = __ldg(g.perm + (size_t)s * kBatch + row0 + tid);
  };
  auto stage_x = [&](int s) {
    for (int e = tid; e < kRowsCta * p0; e += 256) {
      const int r = e / p0, c = e - r * p0;
      const float v = c < g.din ? __ldg(g.x + (size_t)B.src[s & 1][r] * g.din + c) : 0.0f;
      Hs[(c >> 3) * (kHsBox / 2) + r * 8 + (c & 7)] = __float2bfloat16_rn(v);
    }
  };
  auto leave = [&]() {
    if (warp == 8 && lane == 0) drain_ring(B.full, kRing, slot, ph);
  };
  rows_of(0);
  __syncthreads();
  if (tid < 256) stage_x(0);
  if (!fsd::grid_sync(g.bar, g.err, gridDim.x, target)) return;
  for (int s = 0; s < g.steps; s++) {
    if (warp == 8) {
      if (lane == 0) {
        fence_async();  // the tiles' weights, written before the barrier
        for_stages(g, [&](int, bool, const bf16 *W, int M, int K) {
          const uint8_t *src = (const uint8_t *)W;
          const uint32_t second = M > 128 ? (uint32_t)((K + 63) / 64) * kChunkB : 0u;  // the second row tile's chunks
          for (int k0 = 0; k0 < K && ok; k0 += 64, src += kChunkB) {
            const uint32_t bytes = (uint32_t)min(64, K - k0) * 256u, full = smem_u32(&B.full[slot]);
            const uint32_t dst = smem_u32(smem) + slot * 2 * kChunkB;
            ok = mbar_wait(smem_u32(&B.empty[slot]), ph ^ 1u);
            if (!ok) break;
            mbar_expect(full, second ? 2 * bytes : bytes);
            bulk_load(dst, src, bytes, full);
            if (second) bulk_load(dst + kChunkB, src + second, bytes, full);
            if (++slot == kRing) slot = 0, ph ^= 1u;
          }
        });
      }
    } else if (warp == 9) {
      // (the whole warp runs the loops, one elected lane issues: a product's
      // MMAs follow each other at 41 cycles, 32 of them W's reads from shared
      // memory, and at 75-80 from a branch that only one lane enters)
      const uint64_t ra = sdesc(smem_u32(smem), 2048, 128), rb = sdesc(hs, kHsBox, 128);
      constexpr uint32_t kB = 2 * kHsBox >> 4;  // descriptors advance by adding to the address field
      const uint32_t id = idesc_bf16(128, kRowsCta);
      for_stages(g, [&](int, bool, const bf16 *, int M, int K) {
        asm volatile("bar.sync 2, 288;\n" ::: "memory");  // the operand is in shared memory
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        for (int k0 = 0; k0 < K && ok; k0 += 64) {
          ok = mbar_wait(smem_u32(&B.full[slot]), ph);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint64_t a0 = ra + slot * (2 * kChunkB >> 4), a1 = a0 + (kChunkB >> 4);
          const uint64_t b = rb + (uint32_t)(k0 >> 4) * kB;
          const uint32_t acc = k0 > 0 ? 1u : 0u;
          if (elect_one()) {
            if (K - k0 >= 64 && M > 128) {
#pragma unroll
              for (int k = 0; k < 4; k++) {
                mma_bf16(tmem, a0 + k * 256, b + k * kB, id, k ? 1u : acc);
                mma_bf16(tmem + kRowsCta, a1 + k * 256, b + k * kB, id, k ? 1u : acc);
              }
            } else if (K - k0 >= 64) {
#pragma unroll
              for (int k = 0; k < 4; k++) mma_bf16(tmem, a0 + k * 256, b + k * kB, id, k ? 1u : acc);
            } else {
              for (int k = 0; k < (K - k0) >> 4; k++) {
                mma_bf16(tmem, a0 + k * 256, b + k * kB, id, k ? 1u : acc);
                if (M > 128) mma_bf16(tmem + kRowsCta, a1 + k * 256, b + k * kB, id, k ? 1u : acc);
              }
            }
            mma_commit(smem_u32(&B.empty[slot]));
            if (k0 + 64 >= K) mma_commit(done);
          }
          __syncwarp();
          if (++slot == kRing) slot = 0, ph ^= 1u;
        }
      });
    } else {
      const int f = (warp & 3) * 32 + lane + (warp >> 2) * 128;  // the thread's feature
      const int last = g.l[L - 1].out;
      fence_async_smem();
      asm volatile("bar.sync 2, 288;\n" ::: "memory");
      // while the first layer runs: the targets of output feature f, and the
      // input, transposed, for its layer's gradient
      // (eight rows of feature f & 127 where the output layer has one row tile)
      const bool split = last <= 128;
      const int ft = split ? f & 127 : f, rt = split ? (warp >> 2) * 8 : 0;
      float tt[kRowsCta];
#pragma unroll
      for (int r = 0; r < kRowsCta; r++)
        tt[r] = ft < g.dout && (r < 8 || !split) ? __ldg(g.t + (size_t)B.src[s & 1][rt + r] * g.dout + ft) : 0.0f;
      if (tid < p0) {
        uint32_t v[8];
#pragma unroll
        for (int r = 0; r < kRowsCta; r += 2)
          v[r >> 1] = (uint32_t) * (const uint16_t *)(Hs + (tid >> 3) * (kHsBox / 2) + r * 8 + (tid & 7)) |
                      (uint32_t) * (const uint16_t *)(Hs + (tid >> 3) * (kHsBox / 2) + (r + 1) * 8 + (tid & 7)) << 16;
        uint4 *dst = (uint4 *)(g.l[0].HT + (size_t)(tid / kTileN) * (kTileN * kBatch) +
                               (size_t)(row0 >> 3) * (kTileN * 8) + (tid % kTileN) * 8);
        dst[0] = make_uint4(v[0], v[1], v[2], v[3]);
        dst[kTileN] = make_uint4(v[4], v[5], v[6], v[7]);
      }
      asm volatile("bar.sync 3, 256;\n" ::: "memory");  // Hs is read before the next operand goes there
      float lsum = 0.0f;
      for_stages(g, [&](int l, bool back, const bf16 *, int M, int) {
        const TrainLayer &Y = g.l[l];
        const float bias = !back && f < M ? __ldcg(Y.b + f) : 0.0f;
        // backward: the input of layer l, whose sign is the ReLU's mask
        uint4 h0 = make_uint4(0, 0, 0, 0), h1 = h0;
        if (back && f < M) {
          const uint4 *src = (const uint4 *)(Y.HT + (size_t)(f / kTileN) * (kTileN * kBatch) +
                                             (size_t)(row0 >> 3) * (kTileN * 8) + (f % kTileN) * 8);
          h0 = __ldcg(src);
          h1 = __ldcg(src + kTileN);
        }
        ok = mbar_wait(done, dph) && ok;
        dph ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (!back && l + 1 == L && M <= 128) {
          // the output layer fills four warps' accumulator lanes: warps w and
          // w + 4 take eight rows each of the loss and its gradient
          const int fo = (warp & 3) * 32 + lane, h8 = warp >> 2;
          uint32_t a[8], v[4];
          tmem_ld8(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(h8 * 8), a);
          asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
          const float bo = fo < M ? __ldcg(Y.b + fo) : 0.0f;
          float x[8];
#pragma unroll
          for (int r = 0; r < 8; r++) {
            float lo;
            loss_element(__uint_as_float(a[r]) + bo, tt[r], fo, g.dout - 1, kBatch, lo, x[r]);
            lsum += lo;
          }
#pragma unroll
          for (int r = 0; r < 8; r += 2) v[r >> 1] = bf2(x[r], x[r + 1]);
          if (fo < M && L > 1) {
            uint16_t *h = (uint16_t *)(Hs + (fo >> 3) * (kHsBox / 2) + (fo & 7) + h8 * 64);
#pragma unroll
            for (int r = 0; r < 8; r++) h[r * 8] = (uint16_t)(v[r >> 1] >> (16 * (r & 1)));
          }
          fence_async_smem();
          if (L > 1) asm volatile("bar.sync 2, 288;\n" ::: "memory");
          if (fo < M)
            *(uint4 *)(Y.dZT + (size_t)((row0 >> 3) + h8) * 1024 + (size_t)fo * 8) = make_uint4(v[0], v[1], v[2], v[3]);
          return;
        }
        uint32_t v[8];
        if ((f & ~127) < M) {  // (whole warps)
          uint32_t a[16];
          tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * kRowsCta), a);
          asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
          float x[kRowsCta];
          const bf16 *m0 = (const bf16 *)&h0, *m1 = (const bf16 *)&h1;
#pragma unroll
          for (int r = 0; r < kRowsCta; r++) x[r] = __uint_as_float(a[r]);
          if (back) {
#pragma unroll
            for (int r = 0; r < kRowsCta; r++)
              if (!(__bfloat162float(r < 8 ? m0[r & 7] : m1[r & 7]) > 0.0f)) x[r] = 0.0f;
          } else if (l + 1 < L) {
#pragma unroll
            for (int r = 0; r < kRowsCta; r++) x[r] = fmaxf(x[r] + bias, 0.0f);
          } else {
#pragma unroll 4
            for (int r = 0; r < kRowsCta; r++) {
              float lo, d;
              loss_element(x[r] + bias, tt[r], f, g.dout - 1, kBatch, lo, d);
              lsum += lo;
              x[r] = d;
            }
          }
#pragma unroll
          for (int r = 0; r < kRowsCta; r += 2) v[r >> 1] = bf2(x[r], x[r + 1]);
          if (f < M && (!back || l > 1)) {  // the next stage's operand
            uint16_t *h = (uint16_t *)(Hs + (f >> 3) * (kHsBox / 2) + (f & 7));
#pragma unroll
            for (int r = 0; r < kRowsCta; r++) h[r * 8] = (uint16_t)(v[r >> 1] >> (16 * (r & 1)));
          }
        }
        fence_async_smem();
        if (!(back && l == 1) && L > 1) asm volatile("bar.sync 2, 288;\n" ::: "memory");
        // while the next stage runs: the next layer's input (forward), the
        // gradients of the output and of each layer's input, for the tiles
        if (f < M) {
          const bool act = !back && l + 1 < L;
          const int T = act ? kTileN : 128;
          bf16 *base = act ? g.l[l + 1].HT : back ? g.l[l - 1].dZT : Y.dZT;
          uint4 *dst = (uint4 *)(base + (size_t)(f / T) * (T * kBatch) + (size_t)(row0 >> 3) * (T * 8) +
                                 (size_t)(f % T) * 8);
          dst[0] = make_uint4(v[0], v[1], v[2], v[3]);
          dst[T] = make_uint4(v[4], v[5], v[6], v[7]);
        }
      });
      fence_async();  // the tiles read what was written above
      if ((split ? warp & 3 : warp) * 32 < last) {
        for (int o = 16; o; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if (lane == 0) atomicAdd(g.loss, lsum);
      }
    }
    if (!ok) B.fail = 1;
    if (!fsd::grid_sync(g.bar, g.err, gridDim.x, target)) return leave();  // activations and gradients are out
    if (B.fail) {
      if (tid == 0) atomicExch(g.err, 6);
      return leave();
    }
    if (s + 1 < g.steps) {  // while the tiles update
      rows_of(s + 1);
      __syncthreads();
      if (tid < 256) stage_x(s + 1);
    }
    if (!fsd::grid_sync(g.bar, g.err, gridDim.x, target)) return;  // the weights are updated
  }
}

// One tile of a layer's weights (CTAs from kRowCtas on): rows [128 mt, ...) of
// W [out x in], columns [kTileN nt, ...).
__device__ __forceinline__ void train_tile(const TrainArgs &g, uint8_t *smem, TrainBars &B) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kC = kTileN / 2;  // columns of a thread
  constexpr uint32_t kBc = kTileN * 128;  // bytes of H^T in a chunk of 64 rows
  const uint32_t code = __ldg(g.tile + blockIdx.x - kRowCtas);
  const TrainLayer &Y = g.l[code & 0xffu];
  const int mt = (int)(code >> 8) & 0xff, nt = (int)(code >> 16), NT = (Y.in + kTileN - 1) / kTileN;
  uint8_t *sA = smem, *sB = smem + 4 * kChunkB;        // dZ^T [32][128][8], H^T [32][kTileN][8]
  bf16 *tr = (bf16 *)(smem + 5 * kChunkB);             // the tile's W^T [kTileN in][128 out]
  const int o = mt * 128 + (warp & 3) * 32 + lane;     // the thread's weight row and kC columns
  const int i0 = nt * kTileN + (warp >> 2) * kC;
  const bool mine = tid < 256 && o < Y.out && i0 < Y.in;
  // biases: the row tile's are dealt to its column tiles, in a tile to the
  // warps; lane k of a warp has its k-th, row fb(k) of the row tile
  auto fb = [&](int k) { return nt + NT * (warp + 8 * k); };
  const int nb = tid < 256 ? max(0, (min(128, Y.out - mt * 128) - nt + NT * (8 - warp) - 1) / (NT * 8)) : 0;
  const int ob = mt * 128 + fb(lane);
  float w[kC], m[kC], v[kC], b = 0.0f, bm = 0.0f, bv = 0.0f;
#pragma unroll
  for (int k = 0; k < kC; k++) {
    const size_t e = (size_t)o * Y.in + i0 + k;
    w[k] = mine ? Y.W[e] : 0.0f;
    m[k] = mine ? Y.mW[e] : 0.0f;
    v[k] = mine ? Y.vW[e] : 0.0f;
  }
  if (lane < nb) b = Y.b[ob], bm = Y.mb[ob], bv = Y.vb[ob];
  // the BF16 copies, blocked (see above); the transposed one through shared
  // memory, eight rows of a column a thread
  auto publish = [&]() {
    if (tid < 256) {
      uint32_t p[kC / 2];
#pragma unroll
      for (int k = 0; k < kC; k += 2) p[k >> 1] = bf2(w[k], w[k + 1]);
      if (mine) {
        const int kc = (Y.in + 63) / 64;
        *(uint4 *)(Y.Wk + ((size_t)mt * kc + i0 / 64) * (kChunkB / 2) + (size_t)((i0 & 63) >> 3) * 1024 +
                   (size_t)(o & 127) * 8) = make_uint4(p[0], p[1], p[2], p[3]);
      }
#pragma unroll
      for (int k = 0; k < kC; k++)
        ((uint16_t *)tr)[((warp >> 2) * kC + k) * 128 + (o & 127)] = (uint16_t)(p[k >> 1] >> (16 * (k & 1)));
      asm volatile("bar.sync 3, 256;\n" ::: "memory");
      for (int q = tid; q < kTileN * 16; q += 256) {
        const int i = nt * kTileN + q % kTileN, oo = mt * 128 + q / kTileN * 8;
        if (i < Y.in && oo < Y.out) {
          const int kc = (Y.out + 63) / 64;
          *(uint4 *)(Y.Wt + ((size_t)(i / 128) * kc + oo / 64) * (kChunkB / 2) + (size_t)((oo & 63) >> 3) * 1024 +
                     (size_t)(i & 127) * 8) = *(const uint4 *)(tr + q % kTileN * 128 + q / kTileN * 8);
        }
      }
      if (lane < nb) Y.b[ob] = b;
      fence_async();
    }
  };
  static_assert(kC == 8, "a thread's columns are one 16-byte store");
  publish();
  unsigned long long target = 0;
  const int t0 = g.ctr[1];
  bool ok = true;
  if (!fsd::grid_sync(g.bar, g.err, gridDim.x, target)) return;
  for (int s = 0; s < g.steps; s++) {
    const uint32_t ph = (uint32_t)s & 1u;
    if (!fsd::grid_sync(g.bar, g.err, gridDim.x, target)) return;  // the step's gradients are out
    if (warp == 8) {
      if (lane == 0) {
        fence_async();
        for (int c = 0; c < 4; c++) {
          const uint32_t bar = smem_u32(&B.full[c]);
          mbar_expect(bar, kChunkB + kBc);
          bulk_load(smem_u32(sA + c * kChunkB), Y.dZT + (size_t)mt * (128 * kBatch) + (size_t)c * (kChunkB / 2), kChunkB,
                    bar);
          bulk_load(smem_u32(sB + c * kBc), (const uint8_t *)(Y.HT + (size_t)nt * (kTileN * kBatch)) + c * kBc, kBc,
                    bar);
        }
      }
    } else if (warp == 9) {
      if (lane == 0) {
        const uint64_t da = sdesc(smem_u32(sA), 2048, 128), db = sdesc(smem_u32(sB), kTileN * 16u, 128);
        for (int c = 0; c < 4 && ok; c++) {
          ok = mbar_wait(smem_u32(&B.full[c]), ph);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
          for (int k = 0; k < 4; k++)
            mma_bf16(B.tmem, da + (4 * c + k) * 256, db + (4 * c + k) * (kTileN * 2), idesc_bf16(128, kTileN),
                     c + k > 0 ? 1u : 0u);
        }
        mma_commit(smem_u32(&B.done));
      }
    } else {
      float c1, c2;
      adam_corrections(t0 + s, c1, c2);
      if (nb) {  // gradient of the biases: row sums of dZ^T, in k_bias_grad's order
        for (int c = 0; c < 4; c++) ok = mbar_wait(smem_u32(&B.full[c]), ph) && ok;
        float gb = 0.0f;
        for (int k = 0; k < nb; k++) {
          const bf16 *p = (const bf16 *)sA + fb(k) * 8 + (lane & 7);
          float a = 0.0f;
#pragma unroll
          for (int j = 0; j < 8; j++) a += __bfloat162float(p[(size_t)((lane >> 3) + 4 * j) * 1024]);
          for (int q = 16; q; q >>= 1) a += __shfl_xor_sync(0xffffffffu, a, q);
          if (lane == k) gb = a;
        }
        if (lane < nb) adam_update(b, bm, bv, gb, g.lr, c1, c2);
      }
      ok = mbar_wait(smem_u32(&B.done), ph) && ok;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      uint32_t a[kC];
      tmem_ld8(B.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * kC), a);
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      if (mine)
#pragma unroll
        for (int k = 0; k < kC; k++) adam_update(w[k], m[k], v[k], __uint_as_float(a[k]), g.lr, c1, c2);
      publish();
    }
    if (!ok) {
      B.fail = 1;
      if (warp == 9) drain_ring(B.full, 4, 4, ph);  // (its copies in flight; the copying lane does not wait)
    }
    if (!fsd::grid_sync(g.bar, g.err, gridDim.x, target)) return;
    if (B.fail) {
      if (tid == 0) atomicExch(g.err, 6);
      return;
    }
  }
#pragma unroll
  for (int k = 0; k < kC; k++) {
    const size_t e = (size_t)o * Y.in + i0 + k;
    if (mine) Y.W[e] = w[k], Y.mW[e] = m[k], Y.vW[e] = v[k];
  }
  if (lane < nb) Y.mb[ob] = bm, Y.vb[ob] = bv;
  if (blockIdx.x == kRowCtas && tid == 0) g.ctr[1] = t0 + g.steps;
}

__global__ void __launch_bounds__(kTrThreads, 1) k_train(const __grid_constant__ TrainArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ TrainBars B;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;\n" ::"r"(smem_u32(&B.tmem)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    for (int c = 0; c < kRing; c++) {
      mbar_init(smem_u32(&B.full[c]), 1);
      mbar_init(smem_u32(&B.empty[c]), 1);
    }
    mbar_init(smem_u32(&B.done), 1);
    B.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    fence_async();
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (blockIdx.x < kRowCtas) train_rows(g, smem, B);
  else train_tile(g, smem, B);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;\n" ::"r"(B.tmem));
}
constexpr int kTrainSmem = kRing * 2 * (int)kChunkB + 32 * (int)kHsBox;

// ---- inference kernel ----------------------------------------------------------
// R rows at a time through all layers in one CTA (the row CTAs' scheme of
// k_train): the inputs are rounded to BF16 on the way in, the weights stream
// from L2 in 16 KB chunks, the activations stay in shared memory and only the
// outputs are written.  A GEMM launch per layer moved every layer's
// activations through memory and padded the outputs.  R = 16 while 16-row tiles fit
// one wave of CTAs (a tile is a chain of products, so few rows want many CTAs),
// 64 beyond (the chunks of a tile serve four times the rows).  On the device
// 2,000 rows 48 -> 13 us, 8,192 rows 54 -> 20 us; a call is bound by the copies
// (2,000 rows 0.71 -> 0.13 ms, 400,000 rows 32 -> 7.8 ms).
struct FwdLayer {
  const bf16 *Wk;
  const float *b;
  int in, out;
};
constexpr int kFwdCached = 32;  // layers held in shared memory (deeper ones are read from L2)

template <int R>
constexpr uint32_t kFwdBox = R * 16 + 16;  // bytes between the K boxes of an operand, padded as kHsBox
template <int R>
constexpr int kFwdSmem = kRing * 2 * (int)kChunkB + 2 * 32 * (int)kFwdBox<R>;

template <int R>
__global__ void __launch_bounds__(kTrThreads, 1) k_forward(const FwdLayer *gl, int L, const float *x, float *y, int rows,
                                                          int din, int dout, int *err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ TrainBars B;
  __shared__ FwdLayer sl[kFwdCached];
  constexpr uint32_t kBox = kFwdBox<R>, kCols = 2 * R;
  constexpr int CH = R == 16 ? 8 : 16;  // rows of an epilogue pass
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  bf16 *Xs = (bf16 *)(smem + kRing * 2 * kChunkB), *Hs = Xs + 32 * (kBox / 2);  // operands of the first and the other layers
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&B.tmem)),
                 "r"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    for (int c = 0; c < kRing; c++) {
      mbar_init(smem_u32(&B.full[c]), 1);
      mbar_init(smem_u32(&B.empty[c]), 1);
    }
    mbar_init(smem_u32(&B.done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
    fence_async();
  }
  for (int l = tid; l < min(L, kFwdCached); l += kTrThreads) sl[l] = gl[l];
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = B.tmem, done = smem_u32(&B.done);
  const int tiles = (rows + R - 1) / R;
  uint32_t slot = 0, ph = 0, dph = 0;
  bool ok = true;
  auto layer = [&](int l) { return l < kFwdCached ? sl[l] : gl[l]; };
  if (warp == 8) {
    if (lane == 0) {
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x)
        for (int l = 0; l < L && ok; l++) {
          const FwdLayer Y = layer(l);
          const uint8_t *src = (const uint8_t *)Y.Wk;
          const uint32_t second = Y.out > 128 ? (uint32_t)((Y.in + 63) / 64) * kChunkB : 0u;
          for (int k0 = 0; k0 < Y.in && ok; k0 += 64, src += kChunkB) {
            const uint32_t bytes = (uint32_t)min(64, Y.in - k0) * 256u, full = smem_u32(&B.full[slot]);
            const uint32_t dst = smem_u32(smem) + slot * 2 * kChunkB;
            ok = mbar_wait(smem_u32(&B.empty[slot]), ph ^ 1u);
            if (!ok) break;
            mbar_expect(full, second ? 2 * bytes : bytes);
            bulk_load(dst, src, bytes, full);
            if (second) bulk_load(dst + kChunkB, src + second, bytes, full);
            if (++slot == kRing) slot = 0, ph ^= 1u;
          }
        }
      drain_ring(B.full, kRing, slot, ph);
    }
  } else if (warp == 9) {
    const uint64_t ra = sdesc(smem_u32(smem), 2048, 128);
    const uint64_t rx = sdesc(smem_u32(Xs), kBox, 128), rh = sdesc(smem_u32(Hs), kBox, 128);
    constexpr uint32_t kB = 2 * kBox >> 4;
    const uint32_t id = idesc_bf16(128, R);
    for (int t = blockIdx.x; t < tiles; t += gridDim.x)
      for (int l = 0; l < L; l++) {
        const FwdLayer Y = layer(l);
        asm volatile("bar.sync 2, 288;\n" ::: "memory");  // the operand is in shared memory
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        for (int k0 = 0; k0 < Y.in && ok; k0 += 64) {
          ok = mbar_wait(smem_u32(&B.full[slot]), ph);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint64_t a0 = ra + slot * (2 * kChunkB >> 4), a1 = a0 + (kChunkB >> 4);
          const uint64_t b = (l ? rh : rx) + (uint32_t)(k0 >> 4) * kB;
          const uint32_t acc = k0 > 0 ? 1u : 0u;
          if (elect_one()) {
            if (Y.in - k0 >= 64 && Y.out > 128) {
#pragma unroll
              for (int k = 0; k < 4; k++) {
                mma_bf16(tmem, a0 + k * 256, b + k * kB, id, k ? 1u : acc);
                mma_bf16(tmem + R, a1 + k * 256, b + k * kB, id, k ? 1u : acc);
              }
            } else {
              for (int k = 0; k < min(4, (Y.in - k0) >> 4); k++) {
                mma_bf16(tmem, a0 + k * 256, b + k * kB, id, k ? 1u : acc);
                if (Y.out > 128) mma_bf16(tmem + R, a1 + k * 256, b + k * kB, id, k ? 1u : acc);
              }
            }
            mma_commit(smem_u32(&B.empty[slot]));
            if (k0 + 64 >= Y.in) mma_commit(done);
          }
          __syncwarp();
          if (++slot == kRing) slot = 0, ph ^= 1u;
        }
      }
  } else {
    const int p0 = layer(0).in;
    auto stage_x = [&](int t) {
      for (int e = tid; e < R * p0; e += 256) {
        const int r = e / p0, c = e - r * p0;
        const float v = c < din && t * R + r < rows ? __ldg(x + (size_t)(t * R + r) * din + c) : 0.0f;
        Xs[(c >> 3) * (kBox / 2) + r * 8 + (c & 7)] = __float2bfloat16_rn(v);
      }
      fence_async_smem();
    };
    if ((int)blockIdx.x < tiles) {
      stage_x(blockIdx.x);
      asm volatile("bar.sync 2, 288;\n" ::: "memory");
    }
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      const bool more = t + (int)gridDim.x < tiles;
      for (int l = 0; l < L; l++) {
        const FwdLayer Y = layer(l);
        // the next tile's inputs, once the first layer's product is done
        if (l == 1 && more) stage_x(t + gridDim.x);
        const bool split = Y.out <= 128;  // one row tile: warps w and w + 4 take half the rows each
        const int f = (warp & 3) * 32 + lane + (split ? 0 : (warp >> 2) * 128);
        const int r0 = split ? (warp >> 2) * (R / 2) : 0, r1 = split ? r0 + R / 2 : R;
        const float bias = f < Y.out ? __ldg(Y.b + f) : 0.0f;
        ok = mbar_wait(done, dph) && ok;
        dph ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(split ? 0 : (warp >> 2) * R);
        if ((f & ~31) < Y.out) {  // (whole warps)
          for (int r = r0; r < r1; r += CH) {
            uint32_t a[CH];
            if constexpr (CH == 8) tmem_ld8(ta + (uint32_t)r, a);
            else tmem_ld16(ta + (uint32_t)r, a);
            if (l + 1 < L) {
              if (f < Y.out) {
                uint16_t *h = (uint16_t *)(Hs + (f >> 3) * (kBox / 2) + (f & 7) + r * 8);
#pragma unroll
                for (int q = 0; q < CH; q += 2) {
                  const uint32_t v = bf2(fmaxf(__uint_as_float(a[q]) + bias, 0.0f),
                                         fmaxf(__uint_as_float(a[q + 1]) + bias, 0.0f));
                  h[q * 8] = (uint16_t)v;
                  h[q * 8 + 8] = (uint16_t)(v >> 16);
                }
              }
            } else if (f < dout) {
#pragma unroll
              for (int q = 0; q < CH; q++)
                if (t * R + r + q < rows) y[(size_t)(t * R + r + q) * dout + f] = __uint_as_float(a[q]) + bias;
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        }
        if (L == 1 && more) stage_x(t + gridDim.x);
        fence_async_smem();
        if (l + 1 < L || more) asm volatile("bar.sync 2, 288;\n" ::: "memory");
      }
    }
  }
  if (!ok) atomicExch(err, 7);
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols));
}

inline int pad16(int x) { return (x + 15) / 16 * 16; }

constexpr int kChunk = 8192;    // inference rows of a lane's pass
constexpr int kLanes = 6;       // host threads (each its stream and pinned buffers) of a large inference

// A lane of forward(): stream, events, and device and page-locked buffers of
// `cap` bytes for a chunk's inputs and outputs.
struct FwdLane {
  int device = 0;
  size_t cap = 0;
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  char *dev = nullptr, *host = nullptr;
};

void free_lane(FwdLane &a) {
  if (a.st) cudaStreamSynchronize(a.st);
  if (a.dev) cudaFree(a.dev);
  if (a.host) {
    cudaHostUnregister(a.host);
    std::free(a.host);
  }
  if (a.e0) cudaEventDestroy(a.e0);
  if (a.e1) cudaEventDestroy(a.e1);
  if (a.st) cudaStreamDestroy(a.st);
  a = FwdLane();
}

constexpr size_t kPage = 2u << 20;  // lanes are whole huge pages

// Bytes of a lane for chunks of `need` bytes, of a network whose full chunks
// take `full`: rounded up, so that calls of growing size soon find their lane
// (a buffer of exactly the call's size made every larger call wait for a new
// one).  4 MB hold a full chunk of the surrogate.
size_t lane_bytes(size_t need, size_t full) {
  size_t cap = 4u << 20;
  while (cap < need) cap *= 2;
  return (std::min(cap, full) + kPage - 1) / kPage * kPage;
}

// A new lane on the current device (`device`).  Its host buffer is allocated
// and touched as huge pages before it is page-locked: 4 MB take 1.1 ms in all,
// cudaMallocHost alone 4 ms.
cudaError_t make_lane(int device, size_t cap, FwdLane &a) {
  a = FwdLane();
  a.device = device;
  a.cap = cap;
  char *h = (char *)std::aligned_alloc(kPage, cap);
  if (!h) return cudaErrorMemoryAllocation;
  madvise(h, cap, MADV_HUGEPAGE);
  for (size_t i = 0; i < cap; i += 4096) ((volatile char *)h)[i] = 0;
  cudaError_t e = cudaHostRegister(h, cap, cudaHostRegisterDefault);
  if (e == cudaSuccess) a.host = h;
  else std::free(h);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&a.st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&a.e0);
  if (e == cudaSuccess) e = cudaEventCreate(&a.e1);
  if (e == cudaSuccess) e = cudaMalloc((void **)&a.dev, cap);
  if (e != cudaSuccess) {
    free_lane(a);
    cudaGetLastError();  // (not the next launch's error)
  }
  return e;
}

// Idle lanes, shared by the networks of the process (a new network's first
// call would otherwise wait for page-locked memory); at most kLanes are kept,
// and none once the last network is destroyed.
struct LanePool {
  // Making a lane takes 1.1 ms, a chunk on one lane 0.4 ms: a call's second and
  // further lanes are made when calls that found too few have brought this many
  // chunks for each, so that a first call of a few chunks does not cost more
  // than it would on one lane (65,536 rows, first call: 19.7 ms with six
  // new lanes, 8.3 ms before there were lanes, 5.3 ms by this rule).
  static constexpr uint64_t kChunksPerLane = 8;
  std::mutex mu;
  std::vector<FwdLane> idle;
  uint64_t owed = 0;  // chunks of such calls
  int users = 0;
  LanePool() { idle.reserve(kLanes + 1); }
  void enter() {
    std::lock_guard<std::mutex> l(mu);
    users++;
  }
  void leave() {
    std::vector<FwdLane> drop;
    {
      std::lock_guard<std::mutex> l(mu);
      if (--users == 0) {
        drop = idle;
        idle.clear();
        owed = 0;
      }
    }
    for (FwdLane &a : drop) {
      cudaSetDevice(a.device);
      free_lane(a);
    }
  }
  // Up to `want` idle lanes of at least `cap` bytes on `device` for a call of
  // `chunks` chunks, the smallest first; returns how many more it may make.
  size_t take(int device, size_t cap, size_t want, uint64_t chunks, std::vector<FwdLane> &got) {
    std::lock_guard<std::mutex> l(mu);
    while (got.size() < want) {
      size_t k = idle.size();
      for (size_t i = 0; i < idle.size(); i++)
        if (idle[i].device == device && idle[i].cap >= cap && (k == idle.size() || idle[i].cap < idle[k].cap)) k = i;
      if (k == idle.size()) break;
      got.push_back(idle[k]);
      idle.erase(idle.begin() + (ptrdiff_t)k);
    }
    if (got.size() >= want) return 0;
    const size_t first = got.empty() ? 1 : 0;  // every call has one
    owed = std::min<uint64_t>(owed + chunks, kLanes * kChunksPerLane);
    const size_t more = (size_t)std::min<uint64_t>(want - got.size() - first, owed / kChunksPerLane);
    owed -= more * kChunksPerLane;
    return first + more;
  }
  void give(FwdLane &a) {
    if (!a.st) return;
    FwdLane drop;
    {
      std::lock_guard<std::mutex> l(mu);
      idle.push_back(a);
      if (idle.size() > (size_t)kLanes) {  // the smallest goes
        size_t k = 0;
        for (size_t i = 1; i < idle.size(); i++)
          if (idle[i].cap < idle[k].cap) k = i;
        drop = idle[k];
        idle.erase(idle.begin() + (ptrdiff_t)k);
      }
    }
    free_lane(drop);
  }
};
LanePool &lane_pool() {
  static LanePool *p = new LanePool();  // (never destroyed: networks may outlive static objects)
  return *p;
}

struct Mlp {
  int device = 0, sms = 148;
  cudaStream_t st = nullptr;
  std::vector<int> dims, pd;  // logical and padded (multiple of 16) widths
  int L = 0;
  std::vector<float *> W, b, mW, vW, mb, vb, gW, gb;
  std::vector<bf16 *> Wb, Wt, Wk;  // row-major, transposed, blocked (k_refresh)
  // training buffers (kBatch rows)
  bf16 *X = nullptr, *XT = nullptr;
  std::vector<bf16 *> H, HT, dZ, dZT;
  float *Zo = nullptr, *T = nullptr, *loss = nullptr, *xs = nullptr, *ts = nullptr;
  int *ctr = nullptr, *err = nullptr;
  FwdLayer *fl = nullptr;  // k_forward's layers
  cudaEvent_t fwd0 = nullptr;  // start of a forward()
  bool pooled = false;     // counted by the lane pool
  // k_train: its blocked buffers and tiles (lazily), grid barrier
  std::vector<TrainLayer> tl;
  uint32_t *tile = nullptr;
  int tiles = 0;
  unsigned int *bar = nullptr;
  // the training set on the device, kept (grown) across calls: fit() trains in
  // rounds on the same rows
  float *xall = nullptr, *tall = nullptr, *eloss = nullptr;
  int *perm = nullptr;           // the orders of two epochs
  cudaStream_t order_st = nullptr;  // copies an epoch's order while the last one runs
  cudaEvent_t order_ev = nullptr;   // it is there
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};  // start and end of the last even and odd epoch
  uint64_t cap_rows = 0;
  uint32_t cap_epochs = 0;
  std::vector<void *> allocs;
  float lr = 1e-3f;
};

template <class X>
int mal(Mlp *m, X **p, size_t n, std::string &err) {
  *p = nullptr;
  const size_t bytes = std::max<size_t>(n, 1) * sizeof(X);
  cudaError_t e = cudaMalloc((void **)p, bytes);
  if (e != cudaSuccess) {
    err = std::string("cudaMalloc: ") + cudaGetErrorString(e);
    return FS_ERR_NOMEM;
  }
  m->allocs.push_back(*p);
  e = cudaMemsetAsync(*p, 0, bytes, m->st);
  if (e != cudaSuccess) {
    err = std::string("cudaMemset: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  return FS_OK;
}

void release(Mlp *m, void *p) {
  if (!p) return;
  auto it = std::find(m->allocs.begin(), m->allocs.end(), p);
  if (it != m->allocs.end()) m->allocs.erase(it);
  cudaFree(p);
}

int check(Mlp *m, std::string &err) {
  cudaError_t e = cudaStreamSynchronize(m->st);
  if (e != cudaSuccess) {
    err = std::string("mlp kernels: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  int h = 0;
  cudaMemcpy(&h, m->err, 4, cudaMemcpyDeviceToHost);
  if (h) {
    err = "mlp: tensor-core accumulator wait gave up (device error word set)";
    return FS_ERR_TIMEOUT;
  }
  return FS_OK;
}

void destroy(Mlp *m) {
  if (!m) return;
  cudaSetDevice(m->device);
  if (m->st) cudaStreamSynchronize(m->st);
  if (m->order_st) cudaStreamSynchronize(m->order_st);
  for (void *p : m->allocs) cudaFree(p);
  if (m->order_st) cudaStreamDestroy(m->order_st);
  if (m->order_ev) cudaEventDestroy(m->order_ev);
  for (cudaEvent_t x : m->ev)
    if (x) cudaEventDestroy(x);
  if (m->fwd0) cudaEventDestroy(m->fwd0);
  if (m->st) cudaStreamDestroy(m->st);
  if (m->pooled) lane_pool().leave();
  delete m;
}

int create(const uint32_t *dims, uint32_t nd, int device, uint64_t seed, Mlp **out, std::string &err) {
  *out = nullptr;
  if (!dims || nd < 2) {
    err = "mlp: need at least an input and an output width";
    return FS_ERR_ARG;
  }
  for (uint32_t i = 0; i < nd; i++)
    if (dims[i] < 1 || dims[i] > 256) {
      err = "mlp: layer widths must be in [1, 256]";
      return FS_ERR_ARG;
    }
  if (dims[nd - 1] < 2) {
    err = "mlp: the output needs at least one rate and the hyperactivity logit";
    return FS_ERR_ARG;
  }
  Mlp *m = new Mlp();
  m->device = device;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&m->fwd0);
  if (e != cudaSuccess) {
    err = std::string("mlp: ") + cudaGetErrorString(e);
    destroy(m);
    return FS_ERR_CUDA;
  }
  if (!gemm_attr_set) {
    cudaFuncSetAttribute(k_gemm_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem(256, 256));
    gemm_attr_set = true;
  }
  for (uint32_t i = 0; i < nd; i++) {
    m->dims.push_back((int)dims[i]);
    m->pd.push_back(pad16((int)dims[i]));
  }
  m->L = (int)nd - 1;
  m->pooled = true;
  lane_pool().enter();
  cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device);
  int rc = mal(m, &m->err, 1, err);
  if (!rc) rc = mal(m, &m->ctr, 2, err);
  std::mt19937_64 gen(seed ? seed : 1);
  std::normal_distribution<double> nrm(0.0, 1.0);
  for (int l = 0; l < m->L && !rc; l++) {
    const int pi = m->pd[l], po = m->pd[l + 1], n = pi * po;
    float *w, *bb, *mw, *vw, *mbb, *vbb, *gw, *gbb;
    bf16 *wb, *wt, *wk;
    if ((rc = mal(m, &w, n, err)) || (rc = mal(m, &bb, po, err)) || (rc = mal(m, &mw, n, err)) ||
        (rc = mal(m, &vw, n, err)) || (rc = mal(m, &mbb, po, err)) || (rc = mal(m, &vbb, po, err)) ||
        (rc = mal(m, &gw, n, err)) || (rc = mal(m, &gbb, po, err)) || (rc = mal(m, &wb, n, err)) ||
        (rc = mal(m, &wt, n, err)) ||
        (rc = mal(m, &wk, (size_t)((po + 127) / 128) * ((pi + 63) / 64) * 8192, err)))
      break;
    m->W.push_back(w); m->b.push_back(bb); m->mW.push_back(mw); m->vW.push_back(vw);
    m->mb.push_back(mbb); m->vb.push_back(vbb); m->gW.push_back(gw); m->gb.push_back(gbb);
    m->Wb.push_back(wb); m->Wt.push_back(wt); m->Wk.push_back(wk);
    // He initialisation of the logical block; padding stays zero
    std::vector<float> hw(n, 0.0f);
    const double sc = std::sqrt(2.0 / m->dims[l]);
    for (int r = 0; r < m->dims[l + 1]; r++)
      for (int c = 0; c < m->dims[l]; c++) hw[(size_t)r * pi + c] = (float)(sc * nrm(gen));
    cudaMemcpyAsync(w, hw.data(), (size_t)n * 4, cudaMemcpyHostToDevice, m->st);
    k_refresh<<<(n + 255) / 256, 256, 0, m->st>>>(w, po, pi, wb, wt, wk);
    cudaStreamSynchronize(m->st);
  }
  if (!rc) rc = mal(m, &m->fl, m->L, err);
  if (!rc) {
    std::vector<FwdLayer> fl;
    for (int l = 0; l < m->L; l++) fl.push_back(FwdLayer{m->Wk[l], m->b[l], m->pd[l], m->pd[l + 1]});
    cudaMemcpyAsync(m->fl, fl.data(), fl.size() * sizeof(FwdLayer), cudaMemcpyHostToDevice, m->st);
    cudaStreamSynchronize(m->st);
  }
  if (!rc) rc = mal(m, &m->X, (size_t)kBatch * m->pd[0], err);
  if (!rc) rc = mal(m, &m->XT, (size_t)kBatch * m->pd[0], err);
  for (int l = 1; l <= m->L && !rc; l++) {
    bf16 *h, *ht, *dz, *dzt;
    const size_t n = (size_t)kBatch * m->pd[l];
    if ((rc = mal(m, &h, n, err)) || (rc = mal(m, &ht, n, err)) || (rc = mal(m, &dz, n, err)) ||
        (rc = mal(m, &dzt, n, err)))
      break;
    m->H.push_back(h); m->HT.push_back(ht); m->dZ.push_back(dz); m->dZT.push_back(dzt);
  }
  if (!rc) rc = mal(m, &m->Zo, (size_t)kBatch * m->pd[m->L], err);
  if (!rc) rc = mal(m, &m->T, (size_t)kBatch * m->pd[m->L], err);
  if (!rc) rc = mal(m, &m->loss, 1, err);
  if (!rc) rc = mal(m, &m->xs, (size_t)kBatch * m->dims[0], err);
  if (!rc) rc = mal(m, &m->ts, (size_t)kBatch * m->dims[m->L], err);
  if (!rc) rc = check(m, err);
  if (rc) {
    destroy(m);
    return rc;
  }
  *out = m;
  return FS_OK;
}

// forward over the `rows` staged rows of X (training buffers)
int forward_train(Mlp *m, int rows, std::string &err) {
  for (int l = 0; l < m->L; l++) {
    GemmArgs g{};
    g.A = l == 0 ? m->X : m->H[l - 1];
    g.lda = m->pd[l];
    g.B = m->Wb[l];
    g.ldb = m->pd[l];
    g.M = rows;
    g.N = m->pd[l + 1];
    g.K = m->pd[l];
    g.bias = m->b[l];
    g.err = m->err;
    if (l + 1 < m->L) {
      g.relu = 1;
      g.Cb = m->H[l];
      g.ldcb = m->pd[l + 1];
      g.Ct = m->HT[l];
      g.ldct = kBatch;
    } else {
      g.Cf = m->Zo;
      g.ldcf = m->pd[l + 1];
    }
    int rc = gemm(g, m->st, err);
    if (rc) return rc;
  }
  return FS_OK;
}

// loss and gradients of the staged batch; Adam step when `update`
int backward(Mlp *m, int rows, bool update, std::string &err) {
  const int L = m->L, po = m->pd[L];
  k_loss<<<(rows * po + 255) / 256, 256, 0, m->st>>>(m->Zo, m->T, rows, po, m->dims[L] - 1, m->dZ[L - 1],
                                                    m->dZT[L - 1], kBatch, m->loss);
  for (int l = L - 1; l >= 0; l--) {
    GemmArgs g{};  // dW_l = dZ_l^T . H_{l-1}
    g.A = m->dZT[l];
    g.lda = kBatch;
    g.B = l == 0 ? m->XT : m->HT[l - 1];
    g.ldb = kBatch;
    g.M = m->pd[l + 1];
    g.N = m->pd[l];
    g.K = rows;
    g.Cf = m->gW[l];
    g.ldcf = m->pd[l];
    g.err = m->err;
    int rc = gemm(g, m->st, err);
    if (rc) return rc;
    k_bias_grad<<<(m->pd[l + 1] + 7) / 8, 256, 0, m->st>>>(m->dZT[l], kBatch, rows, m->pd[l + 1], m->gb[l]);
    if (l > 0) {
      GemmArgs h{};  // dZ_{l-1} = (dZ_l . W_l) * (H_{l-1} > 0)
      h.A = m->dZ[l];
      h.lda = m->pd[l + 1];
      h.B = m->Wt[l];
      h.ldb = m->pd[l + 1];
      h.M = rows;
      h.N = m->pd[l];
      h.K = m->pd[l + 1];
      h.mask = m->H[l - 1];
      h.ldm = m->pd[l];
      h.Cb = m->dZ[l - 1];
      h.ldcb = m->pd[l];
      h.Ct = m->dZT[l - 1];
      h.ldct = kBatch;
      h.err = m->err;
      if ((rc = gemm(h, m->st, err))) return rc;
    }
  }
  if (update) {
    for (int l = 0; l < L; l++) {
      const int n = m->pd[l] * m->pd[l + 1];
      k_adam<<<(n + 255) / 256, 256, 0, m->st>>>(m->W[l], m->mW[l], m->vW[l], m->gW[l], n, m->pd[l + 1], m->pd[l],
                                                m->lr, m->ctr, m->Wb[l], m->Wt[l]);
      k_adam<<<(m->pd[l + 1] + 255) / 256, 256, 0, m->st>>>(m->b[l], m->mb[l], m->vb[l], m->gb[l], m->pd[l + 1], 1, 1,
                                                           m->lr, m->ctr, nullptr, nullptr);
    }
    k_step_end<<<1, 1, 0, m->st>>>(m->ctr);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("mlp backward: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  return FS_OK;
}

uint64_t param_count(const Mlp *m) {
  uint64_t n = 0;
  for (int l = 0; l < m->L; l++) n += (uint64_t)m->dims[l] * m->dims[l + 1] + m->dims[l + 1];
  return n;
}

// logical parameter vector (per layer: W [out x in] row-major, then b) <->
// padded device copies; `grads` reads the gradient buffers instead
int params_io(Mlp *m, float *out, const float *in, bool grads, std::string &err) {
  cudaStreamSynchronize(m->st);
  size_t o = 0;
  for (int l = 0; l < m->L; l++) {
    const int pi = m->pd[l], po = m->pd[l + 1], di = m->dims[l], dout = m->dims[l + 1];
    std::vector<float> w((size_t)pi * po, 0.0f), bb(po, 0.0f);
    float *dw = grads ? m->gW[l] : m->W[l], *db = grads ? m->gb[l] : m->b[l];
    if (!in) {
      cudaMemcpy(w.data(), dw, w.size() * 4, cudaMemcpyDeviceToHost);
      cudaMemcpy(bb.data(), db, bb.size() * 4, cudaMemcpyDeviceToHost);
    }
    for (int r = 0; r < dout; r++)
      for (int c = 0; c < di; c++) {
        if (in) w[(size_t)r * pi + c] = in[o + (size_t)r * di + c];
        else out[o + (size_t)r * di + c] = w[(size_t)r * pi + c];
      }
    o += (size_t)dout * di;
    for (int r = 0; r < dout; r++) {
      if (in) bb[r] = in[o + r];
      else out[o + r] = bb[r];
    }
    o += dout;
    if (in) {
      cudaMemcpy(dw, w.data(), w.size() * 4, cudaMemcpyHostToDevice);
      cudaMemcpy(db, bb.data(), bb.size() * 4, cudaMemcpyHostToDevice);
      k_refresh<<<(pi * po + 255) / 256, 256, 0, m->st>>>(m->W[l], po, pi, m->Wb[l], m->Wt[l],
                                                                  m->Wk[l]);
    }
  }
  return check(m, err);
}

// host rows -> the training buffers (X, X^T, T)
int stage_host(Mlp *m, const float *x, const float *t, int rows, std::string &err) {
  cudaMemcpyAsync(m->xs, x, (size_t)rows * m->dims[0] * 4, cudaMemcpyHostToDevice, m->st);
  k_stage_x<<<(rows * m->pd[0] + 255) / 256, 256, 0, m->st>>>(m->xs, rows, m->dims[0], m->pd[0], nullptr, nullptr,
                                                               m->X, m->XT, kBatch);
  if (t) {
    cudaMemcpyAsync(m->ts, t, (size_t)rows * m->dims[m->L] * 4, cudaMemcpyHostToDevice, m->st);
    k_stage_t<<<(rows * m->pd[m->L] + 255) / 256, 256, 0, m->st>>>(m->ts, rows, m->dims[m->L], m->pd[m->L], nullptr,
                                                                    nullptr, m->T);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("mlp staging: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  return FS_OK;
}

int grad(Mlp *m, const float *x, const float *t, int rows, float *g, float *loss, std::string &err) {
  if (rows < 16 || rows > kBatch || rows % 16) {
    err = "mlp grad: rows must be a multiple of 16 in [16, 256]";
    return FS_ERR_ARG;
  }
  int rc;
  cudaMemsetAsync(m->loss, 0, 4, m->st);
  if ((rc = stage_host(m, x, t, rows, err)) || (rc = forward_train(m, rows, err)) ||
      (rc = backward(m, rows, false, err)) || (rc = check(m, err)))
    return rc;
  if (loss) cudaMemcpy(loss, m->loss, 4, cudaMemcpyDeviceToHost);
  return params_io(m, g, nullptr, true, err);
}

// Rows [r0, r0 + n) of a call through lane a (n <= kChunk); host copies into
// and out of the pinned buffers by the calling thread.  ran: when its kernel
// ran, in ms after the event `from` (null: from its own start on).
cudaError_t forward_rows(Mlp *m, FwdLane &a, const float *x, float *y, uint64_t r0, int n,
                         cudaEvent_t from, std::pair<float, float> &ran) {
  const int di = m->dims[0], no = m->dims[m->L];
  const size_t bx = (size_t)n * di * 4, by = (size_t)n * no * 4, oy = (bx + 255) / 256 * 256;
  std::memcpy(a.host, x + r0 * di, bx);
  cudaError_t e = cudaMemcpyAsync(a.dev, a.host, bx, cudaMemcpyHostToDevice, a.st);
  if (e == cudaSuccess) e = cudaEventRecord(a.e0, a.st);
  if (e != cudaSuccess) return e;
  const float *dx = (const float *)a.dev;
  float *dy = (float *)(a.dev + oy);
  if ((n + 15) / 16 <= m->sms)
    k_forward<16><<<(n + 15) / 16, kTrThreads, kFwdSmem<16>, a.st>>>(m->fl, m->L, dx, dy, n, di, no, m->err);
  else
    k_forward<64><<<std::min((n + 63) / 64, m->sms), kTrThreads, kFwdSmem<64>, a.st>>>(m->fl, m->L, dx, dy, n, di, no,
                                                                                    m->err);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaEventRecord(a.e1, a.st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(a.host + oy, dy, by, cudaMemcpyDeviceToHost, a.st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(a.st);
  if (e != cudaSuccess) return e;
  std::memcpy(y + r0 * no, a.host + oy, by);
  if (from) e = cudaEventElapsedTime(&ran.first, from, a.e0);
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ran.second, from ? from : a.e0, a.e1);
  return e;
}

double total(const std::vector<std::pair<float, float>> &v) {
  double sum = 0.0;
  for (const auto &p : v) sum += p.second;
  return sum;
}

// Milliseconds that at least one of the intervals covers.
double covered(std::vector<std::pair<float, float>> &v) {
  std::sort(v.begin(), v.end());
  double sum = 0.0, end = 0.0;
  for (const auto &p : v) {
    sum += std::max(0.0, (double)p.second - std::max((double)p.first, end));
    end = std::max(end, (double)p.second);
  }
  return sum;
}

// Calls of more than one chunk run on several lanes, each with a host thread
// that takes the next chunk: the host copies, the two transfer directions and
// the kernels of different chunks overlap.
int forward(Mlp *m, const float *x, uint64_t rows, float *y, double *device_ms, std::string &err) {
  const uint64_t chunks = (rows + kChunk - 1) / kChunk, per = std::min<uint64_t>(rows, kChunk);
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t want = (size_t)std::max<uint64_t>(1, std::min<uint64_t>({(uint64_t)kLanes, chunks, (uint64_t)hw}));
  const size_t row = (size_t)(m->dims[0] + m->dims[m->L]) * 4, cap = lane_bytes(per * row + 256, kChunk * row + 256);
  cudaError_t e = cudaFuncSetAttribute(k_forward<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem<16>);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_forward<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem<64>);
  // (one lane's kernels follow each other: no common start is needed, whose
  // record and queries took 8 us of a call of 2,000 rows)
  if (e == cudaSuccess && want > 1) e = cudaEventRecord(m->fwd0, m->st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->st);  // weights and parameters are in place
  if (e != cudaSuccess) {
    err = std::string("mlp forward: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  std::vector<std::pair<float, float>> ran(chunks);
  std::vector<FwdLane> lane;
  lane.reserve(kLanes);
  // (new lanes one after the other before the work starts: made by the lanes'
  // own threads, each waited 3 ms for the driver's lock and held up the others)
  for (size_t more = lane_pool().take(m->device, cap, want, chunks, lane); more && e == cudaSuccess; more--) {
    FwdLane a;
    e = make_lane(m->device, cap, a);
    if (e == cudaSuccess) lane.push_back(a);
  }
  if (!lane.empty()) e = cudaSuccess;  // a lane that cannot be made is done without
  const size_t lanes = lane.size();
  std::atomic<uint64_t> next{0};
  std::vector<cudaError_t> res(lanes, cudaSuccess);
  auto work = [&](size_t w) {
    cudaError_t r = cudaSetDevice(m->device);
    for (uint64_t c; r == cudaSuccess && (c = next.fetch_add(1)) < chunks;)
      r = forward_rows(m, lane[w], x, y, c * kChunk, (int)std::min<uint64_t>(kChunk, rows - c * kChunk),
                       want > 1 ? m->fwd0 : nullptr, ran[c]);
    res[w] = r;
  };
  if (lanes) {
    std::vector<std::thread> th;
    try {
      for (size_t w = 1; w < lanes; w++) th.emplace_back(work, w);
    } catch (...) {  // fewer threads than lanes: the others take the chunks
    }
    work(0);
    for (std::thread &q : th) q.join();
  }
  for (size_t w = 0; w < lanes; w++) {
    lane_pool().give(lane[w]);
    if (e == cudaSuccess) e = res[w];
  }
  if (e != cudaSuccess) {
    err = std::string("mlp forward: ") + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? FS_ERR_NOMEM : FS_ERR_CUDA;
  }
  // (the lanes' kernels overlap and wait for each other; want = 1: one chunk at most,
  // or one host thread)
  if (device_ms) *device_ms = want > 1 ? covered(ran) : total(ran);
  return check(m, err);
}

// Buffers and tiles of k_train; m->tiles = -1: the network has more weight
// tiles than SMs beside the row CTAs (each tile's owner keeps it in registers).
int ensure_train(Mlp *m, std::string &err) {
  if (m->tiles) return FS_OK;
  std::vector<uint32_t> tile;
  for (int l = 0; l < m->L; l++)
    for (int mt = 0; mt * 128 < m->pd[l + 1]; mt++)
      for (int nt = 0; nt * kTileN < m->pd[l]; nt++) tile.push_back((uint32_t)(l | mt << 8 | nt << 16));
  int sms = 0, coop = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, m->device);
  if (m->L > kMaxTrainL || !coop || (int)tile.size() + kRowCtas > sms) {
    m->tiles = -1;
    return FS_OK;
  }
  // the blocked buffers are parts of one allocation (a dozen of their own took
  // longer than a small first call)
  std::vector<TrainLayer> tl(m->L);
  bf16 *buf = nullptr;
  size_t total = 0;
  for (int pass = 0; pass < 2; pass++) {
    size_t at = 0;
    const auto up = [](int v, int k) { return (size_t)((v + k - 1) / k); };
    const auto part = [&](size_t n) {
      bf16 *p = buf ? buf + at : nullptr;
      at += (n + 127) / 128 * 128;
      return p;
    };
    for (int l = 0; l < m->L; l++) {
      TrainLayer &y = tl[l];
      y.in = m->pd[l];
      y.out = m->pd[l + 1];
      y.Wk = m->Wk[l];
      y.Wt = part(up(y.in, 128) * up(y.out, 64) * (kChunkB / 2));
      y.HT = part(up(y.in, kTileN) * kTileN * kBatch);
      y.dZT = part(up(y.out, 128) * 128 * kBatch);
      y.W = m->W[l]; y.mW = m->mW[l]; y.vW = m->vW[l];
      y.b = m->b[l]; y.mb = m->mb[l]; y.vb = m->vb[l];
    }
    total = at;
    if (pass == 0) {
      int rc = mal(m, &buf, total, err);
      if (rc) return rc;
    }
  }
  int rc = FS_OK;
  if (!rc) rc = mal(m, &m->tile, tile.size(), err);
  if (!rc) rc = mal(m, &m->bar, 64, err);
  if (rc) return rc;
  cudaError_t e = cudaMemcpyAsync(m->tile, tile.data(), tile.size() * 4, cudaMemcpyHostToDevice, m->st);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->st);
  if (e != cudaSuccess) {
    err = std::string("mlp train set-up: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  m->tl = tl;
  m->tiles = (int)tile.size();
  return FS_OK;
}

// One Adam step, captured once and replayed (networks k_train does not take).
int capture_step(Mlp *m, const float *xall, const float *tall, const int *perm, cudaGraphExec_t *exec,
                 std::string &err) {
  cudaGraph_t graph = nullptr;
  int rc = FS_OK;
  cudaError_t e = cudaStreamBeginCapture(m->st, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    k_stage_x<<<(kBatch * m->pd[0] + 255) / 256, 256, 0, m->st>>>(xall, kBatch, m->dims[0], m->pd[0], perm, m->ctr,
                                                                   m->X, m->XT, kBatch);
    k_stage_t<<<(kBatch * m->pd[m->L] + 255) / 256, 256, 0, m->st>>>(tall, kBatch, m->dims[m->L], m->pd[m->L], perm,
                                                                      m->ctr, m->T);
    rc = forward_train(m, kBatch, err);
    if (!rc) rc = backward(m, kBatch, true, err);
    cudaError_t e2 = cudaStreamEndCapture(m->st, &graph);
    if (!rc && e2 != cudaSuccess) e = e2;
  }
  if (!rc && e == cudaSuccess) e = cudaGraphInstantiate(exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (!rc && e != cudaSuccess) {
    err = std::string("mlp train graph: ") + cudaGetErrorString(e);
    rc = FS_ERR_CUDA;
  }
  return rc;
}

// Device buffers for `rows` training rows and `epochs` epochs.
int ensure_rows(Mlp *m, uint64_t rows, uint32_t epochs, std::string &err) {
  int rc = FS_OK;
  if (rows > m->cap_rows) {
    m->cap_rows = 0;
    release(m, m->xall);
    release(m, m->tall);
    release(m, m->perm);
    m->xall = m->tall = nullptr;
    m->perm = nullptr;
    if ((rc = mal(m, &m->xall, rows * m->dims[0], err)) || (rc = mal(m, &m->tall, rows * m->dims[m->L], err)) ||
        (rc = mal(m, &m->perm, 2 * rows, err)))
      return rc;
    // (their zero fill, before another stream writes perm)
    if (cudaStreamSynchronize(m->st) != cudaSuccess) {
      err = "mlp train: buffers";
      return FS_ERR_CUDA;
    }
    m->cap_rows = rows;
  }
  if (epochs > m->cap_epochs) {
    m->cap_epochs = 0;
    release(m, m->eloss);
    m->eloss = nullptr;
    if ((rc = mal(m, &m->eloss, epochs, err))) return rc;
    m->cap_epochs = epochs;
  }
  cudaError_t e = cudaSuccess;
  for (cudaEvent_t &x : m->ev)
    if (!x && e == cudaSuccess) e = cudaEventCreate(&x);
  if (epochs > 1) {
    if (!m->order_st && e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->order_st, cudaStreamNonBlocking);
    if (!m->order_ev && e == cudaSuccess) e = cudaEventCreateWithFlags(&m->order_ev, cudaEventDisableTiming);
  }
  if (e != cudaSuccess) {
    err = std::string("mlp train: ") + cudaGetErrorString(e);
    return FS_ERR_CUDA;
  }
  return FS_OK;
}

int train(Mlp *m, const float *x, const float *t, uint64_t rows, uint32_t epochs, float lr, uint64_t seed,
          float *epoch_loss, double *device_ms, std::string &err) {
  const int steps = (int)(rows / kBatch);
  if (steps < 1) {
    err = "mlp train: need at least 256 rows";
    return FS_ERR_ARG;
  }
  m->lr = lr;
  int rc = ensure_train(m, err);
  if (!rc) rc = ensure_rows(m, rows, epochs, err);
  if (rc) return rc;
  cudaMemcpyAsync(m->xall, x, rows * m->dims[0] * 4, cudaMemcpyHostToDevice, m->st);
  cudaMemcpyAsync(m->tall, t, rows * m->dims[m->L] * 4, cudaMemcpyHostToDevice, m->st);
  cudaGraphExec_t exec = nullptr;
  if (m->tiles < 0 && (rc = capture_step(m, m->xall, m->tall, m->perm, &exec, err))) return rc;
  TrainArgs a{};
  for (size_t l = 0; l < m->tl.size(); l++) a.l[l] = m->tl[l];
  a.L = m->L;
  a.steps = steps;
  a.din = m->dims[0];
  a.dout = m->dims[m->L];
  a.tiles = m->tiles;
  a.x = m->xall;
  a.t = m->tall;
  a.tile = m->tile;
  a.lr = lr;
  a.ctr = m->ctr;
  a.bar = m->bar;
  a.err = m->err;
  std::mt19937_64 gen(seed ? seed : 1);
  cudaError_t e = cudaSuccess;
  auto ok = [&](cudaError_t r) {
    if (e == cudaSuccess) e = r;
    return e == cudaSuccess;
  };
  if (epochs) ok(cudaMemsetAsync(m->eloss, 0, (size_t)epochs * 4, m->st));
  double ms = 0.0;
  auto epoch_time = [&](uint32_t ep) {  // of an epoch that has ended
    float t = 0;
    if (ok(cudaEventElapsedTime(&t, m->ev[ep & 1u], m->ev[2 + (ep & 1u)]))) ms += t;
  };
  std::vector<int> order(rows);
  for (uint32_t ep = 0; ep < epochs && e == cudaSuccess; ep++) {
    // the host draws an epoch's order, and copies it on a stream of its own,
    // while the device runs the last one (pageable memory, staged by the copy:
    // page-locking its room cost a network's first call 2 ms); the captured step
    // has one place for it, behind the last epoch
    if (ep >= 2) {
      if (!ok(cudaEventSynchronize(m->ev[2 + (ep & 1u)]))) break;
      epoch_time(ep - 2);
    }
    std::iota(order.begin(), order.end(), 0);
    std::shuffle(order.begin(), order.end(), gen);
    const bool apart = !exec && epochs > 1;
    a.perm = m->perm + (apart ? (ep & 1u) * m->cap_rows : 0);
    const cudaStream_t cs = apart ? m->order_st : m->st;
    ok(cudaMemcpyAsync((void *)a.perm, order.data(), (size_t)steps * kBatch * 4, cudaMemcpyHostToDevice, cs));
    if (apart) {
      ok(cudaEventRecord(m->order_ev, cs));
      ok(cudaStreamWaitEvent(m->st, m->order_ev, 0));
    }
    if (exec) {
      ok(cudaMemsetAsync(m->ctr, 0, 4, m->st));  // batch index (the Adam count in ctr[1] runs on)
      ok(cudaMemsetAsync(m->loss, 0, 4, m->st));
      ok(cudaEventRecord(m->ev[ep & 1u], m->st));
      for (int s = 0; s < steps && e == cudaSuccess; s++) ok(cudaGraphLaunch(exec, m->st));
      ok(cudaEventRecord(m->ev[2 + (ep & 1u)], m->st));
      ok(cudaMemcpyAsync(m->eloss + ep, m->loss, 4, cudaMemcpyDeviceToDevice, m->st));
    } else {
      a.loss = m->eloss + ep;
      void *args[] = {&a};
      ok(cudaMemsetAsync(m->bar, 0, 8, m->st));
      ok(cudaEventRecord(m->ev[ep & 1u], m->st));
      if (e == cudaSuccess)
        ok(cudaLaunchCooperativeKernel((const void *)k_train, kRowCtas + m->tiles, kTrThreads, args, kTrainSmem, m->st));
      ok(cudaEventRecord(m->ev[2 + (ep & 1u)], m->st));
    }
  }
  for (int l = 0; l < m->L; l++) {  // the BF16 copies that inference and grad() read
    const int n = m->pd[l] * m->pd[l + 1];
    k_refresh<<<(n + 255) / 256, 256, 0, m->st>>>(m->W[l], m->pd[l + 1], m->pd[l], m->Wb[l], m->Wt[l], m->Wk[l]);
  }
  std::vector<float> el(epochs, 0.0f);
  if (epochs) ok(cudaMemcpyAsync(el.data(), m->eloss, (size_t)epochs * 4, cudaMemcpyDeviceToHost, m->st));
  rc = check(m, err);
  if (exec) cudaGraphExecDestroy(exec);
  if (!rc && e != cudaSuccess) {
    err = std::string("mlp train: ") + cudaGetErrorString(e);
    rc = FS_ERR_CUDA;
  }
  if (!rc)
    for (uint32_t ep = epochs > 2 ? epochs - 2 : 0; ep < epochs; ep++) epoch_time(ep);
  if (epoch_loss)
    for (uint32_t ep = 0; ep < epochs && !rc; ep++) epoch_loss[ep] = el[ep] / (float)steps;
  if (device_ms) *device_ms = ms;
  return rc;
}

}  // namespace fsm

// ---- C ABI ---------------------------------------------------------------------
struct fs_mlp {
  fsm::Mlp *m;
};

namespace {
thread_local std::string g_mlp_err;
int mlp_fail(int rc, const std::string &msg) {
  g_mlp_err = msg;
  return rc;
}
}  // namespace

extern "C" {

const char *fs_mlp_error(void) { return g_mlp_err.c_str(); }

int fs_mlp_create(const uint32_t *dims, uint32_t ndims, int device, uint64_t seed, fs_mlp **out) {
  if (!out) return mlp_fail(FS_ERR_ARG, "fs_mlp_create: out is NULL");
  *out = nullptr;
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) return mlp_fail(FS_ERR_NODEVICE, "fs_mlp_create: no CUDA device");
  if (device < 0 || device >= nd) return mlp_fail(FS_ERR_ARG, "fs_mlp_create: bad device ordinal");
  std::string err;
  fsm::Mlp *m = nullptr;
  int rc = fsm::create(dims, ndims, device, seed, &m, err);
  if (rc) return mlp_fail(rc, err);
  *out = new fs_mlp{m};
  return FS_OK;
}

int fs_mlp_destroy(fs_mlp *h) {
  if (!h) return FS_OK;
  fsm::destroy(h->m);
  delete h;
  return FS_OK;
}

uint64_t fs_mlp_param_count(const fs_mlp *h) { return h ? fsm::param_count(h->m) : 0; }

int fs_mlp_get_params(fs_mlp *h, float *params) {
  if (!h || !params) return mlp_fail(FS_ERR_ARG, "fs_mlp_get_params: null argument");
  cudaSetDevice(h->m->device);
  std::string err;
  int rc = fsm::params_io(h->m, params, nullptr, false, err);
  return rc ? mlp_fail(rc, err) : FS_OK;
}

int fs_mlp_set_params(fs_mlp *h, const float *params) {
  if (!h || !params) return mlp_fail(FS_ERR_ARG, "fs_mlp_set_params: null argument");
  cudaSetDevice(h->m->device);
  std::string err;
  int rc = fsm::params_io(h->m, nullptr, params, false, err);
  return rc ? mlp_fail(rc, err) : FS_OK;
}

int fs_mlp_forward(fs_mlp *h, const float *x, uint64_t rows, float *y, double *device_ms) {
  if (!h || (rows && (!x || !y))) return mlp_fail(FS_ERR_ARG, "fs_mlp_forward: null argument");
  cudaSetDevice(h->m->device);
  std::string err;
  int rc = fsm::forward(h->m, x, rows, y, device_ms, err);
  return rc ? mlp_fail(rc, err) : FS_OK;
}

int fs_mlp_grad(fs_mlp *h, const float *x, const float *t, uint32_t rows, float *grads, float *loss) {
  if (!h || !x || !t || !grads) return mlp_fail(FS_ERR_ARG, "fs_mlp_grad: null argument");
  cudaSetDevice(h->m->device);
  std::string err;
  int rc = fsm::grad(h->m, x, t, (int)rows, grads, loss, err);
  return rc ? mlp_fail(rc, err) : FS_OK;
}

int fs_mlp_train(fs_mlp *h, const float *x, const float *t, uint64_t rows, uint32_t epochs, float lr, uint64_t seed,
                 float *epoch_loss, double *device_ms) {
  if (!h || !x || !t) return mlp_fail(FS_ERR_ARG, "fs_mlp_train: null argument");
  cudaSetDevice(h->m->device);
  std::string err;
  int rc = fsm::train(h->m, x, t, rows, epochs, lr, seed, epoch_loss, device_ms, err);
  return rc ? mlp_fail(rc, err) : FS_OK;
}

int fs_mlp_gemm(const uint16_t *a, const uint16_t *b, uint32_t m, uint32_t n, uint32_t k, const float *bias,
                int relu, float *c) {
  if (!a || !b || !c) return mlp_fail(FS_ERR_ARG, "fs_mlp_gemm: null argument");
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) return mlp_fail(FS_ERR_NODEVICE, "fs_mlp_gemm: no CUDA device");
  fsm::GemmArgs g{};
  g.M = (int)m;
  g.N = (int)n;
  g.K = (int)k;
  g.lda = (int)k;
  g.ldb = (int)k;
  g.relu = relu;
  g.ldcf = (int)n;
  void *da = nullptr, *db = nullptr, *dc = nullptr, *dbias = nullptr;
  int *derr = nullptr;
  cudaError_t e = cudaMalloc(&da, (size_t)m * k * 2);
  if (e == cudaSuccess) e = cudaMalloc(&db, (size_t)n * k * 2);
  if (e == cudaSuccess) e = cudaMalloc(&dc, (size_t)m * n * 4);
  if (e == cudaSuccess && bias) e = cudaMalloc(&dbias, (size_t)n * 4);
  if (e == cudaSuccess) e = cudaMalloc(&derr, 4);
  int rc = FS_OK;
  std::string err;
  if (e == cudaSuccess) {
    cudaMemcpy(da, a, (size_t)m * k * 2, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, (size_t)n * k * 2, cudaMemcpyHostToDevice);
    if (bias) cudaMemcpy(dbias, bias, (size_t)n * 4, cudaMemcpyHostToDevice);
    cudaMemset(derr, 0, 4);
    g.A = (const fsm::bf16 *)da;
    g.B = (const fsm::bf16 *)db;
    g.Cf = (float *)dc;
    g.bias = (const float *)dbias;
    g.err = derr;
    rc = fsm::gemm(g, nullptr, err);
    if (!rc) {
      e = cudaDeviceSynchronize();
      int h = 0;
      if (e == cudaSuccess) e = cudaMemcpy(&h, derr, 4, cudaMemcpyDeviceToHost);
      if (e == cudaSuccess && h) rc = mlp_fail(FS_ERR_TIMEOUT, "fs_mlp_gemm: accumulator wait gave up");
      if (e == cudaSuccess && !rc) e = cudaMemcpy(c, dc, (size_t)m * n * 4, cudaMemcpyDeviceToHost);
    }
  }
  if (e != cudaSuccess && !rc) rc = mlp_fail(FS_ERR_CUDA, std::string("fs_mlp_gemm: ") + cudaGetErrorString(e));
  else if (rc && !err.empty()) mlp_fail(rc, err);
  cudaFree(da);
  cudaFree(db);
  cudaFree(dc);
  cudaFree(dbias);
  cudaFree(derr);
  return rc;
}

}  // extern "C"
