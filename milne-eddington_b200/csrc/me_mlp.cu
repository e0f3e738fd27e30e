// me_mlp.cu -- the learned initialiser: a small MLP that maps a normalised
// Stokes profile to the nine ME parameters, trained on the GPU on profiles the
// GPU forward model synthesises from seeded parameter draws plus noise.
//
//   features (4 nl)  ->  256 GELU  ->  256 GELU  ->  256 GELU  ->  10 outputs
//   outputs: B, cos(theta), sin(2 phi), cos(2 phi), v, Doppler width, a, eta0,
//            beta, S / I_max, each standardised with the training-set moments.
//
// Everything is hand-written here: the data synthesis, the BF16 tensor-core
// kernels (tcgen05.mma fed by TMA, FP32 accumulators in tensor memory: the whole
// inference of a map in one, a training step in two) and the separate GEMMs they
// grew from (tcgen05, or mma.sync m16n8k16 for shapes and settings that ask for
// it), Adam with FP32 master weights, and the decode that turns the outputs into
// per-pixel starting parameters for the LM.  The reference
// has no learned part; the plain LM with its restarts stays the fallback.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/me_b200.h"
#include "me_kernels.h"
#include "me_umma.cuh"

namespace me {
namespace mlp {

constexpr int kHidden = 256;
constexpr int kOut = 10;
constexpr int kLayers = 4;
constexpr int kOutRows = 32;  // rows of the last layer's weights (10 used, zeros past)
typedef __nv_bfloat16 bf16;

// ---------------------------------------------------------------------------
// GEMM: C[M x N] = A[M x R] * Bt[N x R]^T, A and Bt row-major BF16 with R
// contiguous (R % 32 == 0), FP32 accumulation on the tensor cores
// (mma.sync.m16n8k16.row.col.f32.bf16.bf16.f32).  Epilogue: + bias[n] (if
// given), store FP32 pre-activation Z (if given), then GELU (if gelu) into
// BF16 Y (if given) and/or FP32 Yf (if given).  CTA tile 64 x 64, 4 warps of
// 32 x 32, K steps of 32 through shared memory.
// ---------------------------------------------------------------------------
constexpr int kTM = 64, kTN = 64, kTK = 32;

__device__ __forceinline__ void mma_bf16(float c[4], const unsigned a[4], const unsigned b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float gelu_f(float z) {
  return 0.5f * z * (1.f + erff(z * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad(float z) {
  const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
  const float pdf = 0.3989422804014327f * __expf(-0.5f * z * z);
  return cdf + z * pdf;
}

__global__ void __launch_bounds__(128) gemm_kernel(const bf16 *__restrict__ A,
                                                   const bf16 *__restrict__ Bt, int M, int N,
                                                   int R, const float *__restrict__ bias,
                                                   float *__restrict__ Z, int gelu,
                                                   bf16 *__restrict__ Y, float *__restrict__ Yf) {
  __shared__ __align__(16) bf16 sA[kTM][kTK + 8];
  __shared__ __align__(16) bf16 sB[kTN][kTK + 8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * kTM, n0 = blockIdx.x * kTN;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int g = lane >> 2, t4 = lane & 3;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int k = 0; k < 4; k++) acc[i][j][k] = 0.f;
  // split-K: blockIdx.z takes R / gridDim.z of the reduction (a multiple of
  // kTK); partial sums are added into Yf, which the caller zeroes
  const int rz = R / (int)gridDim.z;
  const int kbeg = blockIdx.z * rz, kend = kbeg + rz;
  for (int k0 = kbeg; k0 < kend; k0 += kTK) {
    // 64 x 32 BF16 tiles: 128 threads x 16 elements (two 16-byte chunks) each
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int chunk = tid + c * 128;  // 256 chunks of 8 elements
      const int r = chunk >> 2, col = (chunk & 3) * 8;
      uint4 va = make_uint4(0, 0, 0, 0), vb = make_uint4(0, 0, 0, 0);
      if (m0 + r < M) va = *reinterpret_cast<const uint4 *>(A + (size_t)(m0 + r) * R + k0 + col);
      if (n0 + r < N) vb = *reinterpret_cast<const uint4 *>(Bt + (size_t)(n0 + r) * R + k0 + col);
      *reinterpret_cast<uint4 *>(&sA[r][col]) = va;
      *reinterpret_cast<uint4 *>(&sB[r][col]) = vb;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kTK; kk += 16) {
      unsigned af[2][4], bfr[4][2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int r = wm + i * 16 + g;
        af[i][0] = *reinterpret_cast<const unsigned *>(&sA[r][kk + t4 * 2]);
        af[i][1] = *reinterpret_cast<const unsigned *>(&sA[r + 8][kk + t4 * 2]);
        af[i][2] = *reinterpret_cast<const unsigned *>(&sA[r][kk + 8 + t4 * 2]);
        af[i][3] = *reinterpret_cast<const unsigned *>(&sA[r + 8][kk + 8 + t4 * 2]);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int n = wn + j * 8 + g;
        bfr[j][0] = *reinterpret_cast<const unsigned *>(&sB[n][kk + t4 * 2]);
        bfr[j][1] = *reinterpret_cast<const unsigned *>(&sB[n][kk + 8 + t4 * 2]);
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) mma_bf16(acc[i][j], af[i], bfr[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int m = m0 + wm + i * 16 + g + h * 8;
        if (m >= M) continue;
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int n = n0 + wn + j * 8 + t4 * 2 + e;
          if (n >= N) continue;
          float z = acc[i][j][h * 2 + e];
          if (gridDim.z > 1) {
            atomicAdd(Yf + (size_t)m * N + n, z);
            continue;
          }
          if (bias) z += bias[n];
          if (Z) Z[(size_t)m * N + n] = z;
          const float y = gelu ? gelu_f(z) : z;
          if (Y) Y[(size_t)m * N + n] = __float2bfloat16(y);
          if (Yf) Yf[(size_t)m * N + n] = y;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The same GEMM and epilogue on the sm_100a tensor cores.  A CTA owns a
// 128 x bn tile of C (bn = N up to 256, N % 16 == 0); TMA brings 128 x 64 and
// bn x 64 BF16 tiles of A and Bt into a two-stage ring of 128-byte-swizzled
// shared memory; thread 0 issues four tcgen05.mma (K = 16 each) per stage into
// an FP32 accumulator of bn tensor-memory columns and commits each stage to
// the mbarrier that frees it for the next load; after the last commit every
// warp reads its 32 accumulator rows with tcgen05.ld and applies the epilogue
// (bias, Z, GELU, Y, Yf, or split-K atomics) on 16-column chunks.  Waits are
// bounded: on expiry the CTA writes a code to *err (1: operand load, 2: stage
// release, 3: accumulator), drains what it issued, frees its tensor memory
// and leaves C unwritten.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void umma_tile(const CUtensorMap *tmA, const CUtensorMap *tmB, int m0,
                                          int n0, int bn, int kbeg, int rz, bool split, int M,
                                          int N, const float *__restrict__ bias,
                                          float *__restrict__ Z, int gelu, bf16 *__restrict__ Y,
                                          float *__restrict__ Yf, int *__restrict__ err) {
  using namespace me::umma;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t stB = (uint32_t)bn * kBK * 2;  // a multiple of 2048: bn % 16 == 0
  const uint32_t sA = base, sB = base + kStages * kStageA;
  const uint32_t bars = sB + kStages * stB;
  // full[s] = bars + 8 s, empty[s] = bars + 8 (kStages + s), done after them
  const uint32_t done = bars + 8 * 2 * kStages;
  uint32_t *misc = reinterpret_cast<uint32_t *>(smem_raw + (done + 8 - raw));
  volatile uint32_t *abort_flag = misc + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ncols = tmem_cols(bn);

  if (warp == 0) {
    tmem_alloc(smem_u32(misc), ncols);
    tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(bars + 8 * s, 1);
      mbar_init(bars + 8 * (kStages + s), 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];

  const int nk = (rz + kBK - 1) / kBK;
  const uint32_t tx = (uint32_t)(kBM + bn) * kBK * 2;

  if (warp == 0) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16_f32(kBM, bn);
      int code = 0, loaded = 0, kb = 0;
      for (; loaded < nk && loaded < kStages; loaded++) {
        const uint32_t full = bars + 8 * loaded;
        mbar_expect_tx(full, tx);
        tma_load_2d(sA + loaded * kStageA, tmA, full, kbeg + loaded * kBK, m0);
        tma_load_2d(sB + loaded * stB, tmB, full, kbeg + loaded * kBK, n0);
      }
      for (; kb < nk; kb++) {
        const int s = kb % kStages;
        if (!mbar_wait(bars + 8 * s, (uint32_t)(kb / kStages) & 1u)) {
          code = 1;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < kBK / 16; k++)
          umma_bf16(tmem, sw128_kmajor_desc(sA + s * kStageA + 32 * k),
                   sw128_kmajor_desc(sB + s * stB + 32 * k), idesc, (kb | k) != 0);
        mma_commit(bars + 8 * (kStages + s));
        // refill the stage of the previous k block once its MMAs have read it
        if (kb >= 1 && loaded < nk) {
          const int ls = loaded % kStages;  // == (kb - 1) % kStages
          if (!mbar_wait(bars + 8 * (kStages + ls), (uint32_t)(loaded / kStages - 1) & 1u)) {
            code = 2;
            break;
          }
          const uint32_t full = bars + 8 * ls;
          mbar_expect_tx(full, tx);
          tma_load_2d(sA + ls * kStageA, tmA, full, kbeg + loaded * kBK, m0);
          tma_load_2d(sB + ls * stB, tmB, full, kbeg + loaded * kBK, n0);
          loaded++;
        }
      }
      mma_commit(done);  // tracks every MMA issued above
      if (code) {
        // loads issued and not consumed: let them land before the CTA exits
        for (int j = kb; j < loaded; j++) mbar_wait(bars + 8 * (j % kStages), (uint32_t)(j / kStages) & 1u);
        *abort_flag = 1;
        atomicExch(err, code);
      }
    }
    __syncwarp();
  }
  if (!mbar_wait(done, 0)) {
    *abort_flag = 1;
    atomicExch(err, 3);
  }
  __syncthreads();
  tc_fence_after();
  if (!*abort_flag) {
    const int row = m0 + warp * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    for (int c = 0; c < bn; c += 16) {
      const int n = n0 + c;
      if (n >= N) break;  // the same for the whole warp
      float v[16];
      tmem_ld16(trow + (uint32_t)c, v);
      if (row >= M) continue;
      const size_t o = (size_t)row * N + n;
      if (split) {
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          atomicAdd(reinterpret_cast<float4 *>(Yf + o + j),
                    make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
        continue;
      }
      if (bias) {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] += __ldg(bias + n + j);
      }
      if (Z) {
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4 *>(Z + o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
      if (gelu) {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = gelu_f(v[j]);
      }
      if (Y) {
        uint32_t pk[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          pk[j] = *reinterpret_cast<const uint32_t *>(&h);
        }
        *reinterpret_cast<uint4 *>(Y + o) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4 *>(Y + o + 8) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
      if (Yf) {
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4 *>(Yf + o + j) =
              make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, ncols);
}

__global__ void __launch_bounds__(128, 1)
    umma_gemm_kernel(const __grid_constant__ CUtensorMap tmA,
                     const __grid_constant__ CUtensorMap tmB, int M, int N, int R, int bn,
                     const float *__restrict__ bias, float *__restrict__ Z, int gelu,
                     bf16 *__restrict__ Y, float *__restrict__ Yf, int *__restrict__ err) {
  const int rz = R / (int)gridDim.z;
  umma_tile(&tmA, &tmB, blockIdx.y * me::umma::kBM, blockIdx.x * bn, bn, blockIdx.z * rz, rz,
            gridDim.z > 1, M, N, bias, Z, gelu, Y, Yf, err);
}

// cuTensorMapEncodeTiled from the driver, looked up once through the runtime
// (the library does not link libcuda)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// Tensor map of a row-major BF16 matrix [rows][cols] read in boxes of
// box_rows x 64 with the 128-byte swizzle; boxes reaching past the matrix
// read zeros
bool tile_map(CUtensorMap *map, const bf16 *p, int rows, int cols, int box_rows) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(p) & 15) || (cols * 2) % 16 || box_rows < 1 ||
      box_rows > 256)
    return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {(cuuint32_t)me::umma::kBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16 *>(p), dims, strides, box,
             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Which GEMM runs: the tcgen05 kernel wherever its shape rules hold (N % 16 ==
// 0, each split-K share a multiple of 64, tensor maps encodable), else the
// mma.sync kernel; GemmPath::mma_sync forces the latter.
enum class GemmPath { tcgen05 = 0, mma_sync = 1 };

// Tensor maps already encoded for a model's buffers: a map is a function of
// (address, rows, columns, box rows) alone, so a hit is always valid.
struct TileMapCache {
  struct Entry {
    const void *p;
    int rows, cols, box_rows;
    CUtensorMap map;
  };
  std::vector<Entry> entries;
};

struct GemmCtx {
  GemmPath path = GemmPath::tcgen05;
  int *err = nullptr;             // device flag of the tcgen05 kernel's bounded waits
  long long *launches = nullptr;  // [2]: launches of each kernel, indexed by GemmPath
  TileMapCache *maps = nullptr;   // may be null (no caching)
};

bool cached_tile_map(TileMapCache *c, CUtensorMap *map, const bf16 *p, int rows, int cols,
                     int box_rows) {
  if (c)
    for (const TileMapCache::Entry &e : c->entries)
      if (e.p == p && e.rows == rows && e.cols == cols && e.box_rows == box_rows) {
        *map = e.map;
        return true;
      }
  if (!tile_map(map, p, rows, cols, box_rows)) return false;
  if (c) {
    if (c->entries.size() >= 256) c->entries.clear();
    c->entries.push_back({p, rows, cols, box_rows, *map});
  }
  return true;
}

// Per-device facts the launch needs, looked up once per device: the SM count
// and whether the kernel's shared-memory limit has been raised.
struct DeviceFacts {
  int sms = 0;
  bool smem_ok = false, pred_ok = false, step_ok = false;
};

bool predict_kernel_ready();  // (below, with the kernels)
bool step_kernels_ready();

const DeviceFacts &device_facts() {
  static DeviceFacts facts[64];
  static std::once_flag once[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    static const DeviceFacts none;
    return none;
  }
  std::call_once(once[dev], [dev]() {
    DeviceFacts f;
    if (cudaDeviceGetAttribute(&f.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      f.sms = 0;
    f.smem_ok = cudaFuncSetAttribute(umma_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     me::umma::kSmemMax) == cudaSuccess;
    f.pred_ok = predict_kernel_ready();
    f.step_ok = f.smem_ok && step_kernels_ready();
    facts[dev] = f;
  });
  return facts[dev];
}

// split > 1: R % (split * kTK) == 0, only Yf (zeroed by the caller), no
// epilogue.  Returns the kernel that ran.
GemmPath gemm(const GemmCtx &g, const bf16 *A, const bf16 *Bt, int M, int N, int R,
              const float *bias, float *Z, int gelu, bf16 *Y, float *Yf, cudaStream_t st,
              int split = 1) {
  if (g.path == GemmPath::tcgen05 && g.err && N % 16 == 0 && R % split == 0 &&
      (split == 1 || (R / split) % me::umma::kBK == 0)) {
    // column tile: all of N up to 256, halved (in multiples of 16, down to
    // 32) while the grid has fewer than two CTAs per SM, so that small
    // batches still spread over the GPU
    const DeviceFacts &dv = device_facts();
    int bn = N <= me::umma::kMaxBN ? N : me::umma::kMaxBN;
    const long long tiles_m = (M + me::umma::kBM - 1) / me::umma::kBM;
    while (bn > 32 && bn % 32 == 0 &&
           (long long)((N + bn - 1) / bn) * tiles_m * split < 2LL * dv.sms)
      bn /= 2;
    CUtensorMap ma, mb;
    if (dv.smem_ok && cached_tile_map(g.maps, &ma, A, M, R, me::umma::kBM) &&
        cached_tile_map(g.maps, &mb, Bt, N, R, bn)) {
      dim3 grid((N + bn - 1) / bn, (M + me::umma::kBM - 1) / me::umma::kBM, split);
      umma_gemm_kernel<<<grid, 128, me::umma::smem_bytes(bn), st>>>(ma, mb, M, N, R, bn, bias, Z,
                                                                    gelu, Y, Yf, g.err);
      if (g.launches) g.launches[(int)GemmPath::tcgen05]++;
      return GemmPath::tcgen05;
    }
  }
  dim3 grid((N + kTN - 1) / kTN, (M + kTM - 1) / kTM, split);
  gemm_kernel<<<grid, 128, 0, st>>>(A, Bt, M, N, R, bias, Z, gelu, Y, Yf);
  if (g.launches) g.launches[(int)GemmPath::mma_sync]++;
  return GemmPath::mma_sync;
}

// out[c][r] = in[r][c] (BF16), rows x cols
__global__ void transpose_kernel(const bf16 *in, int rows, int cols, bf16 *out) {
  __shared__ bf16 tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int r = by + i, c = bx + threadIdx.x;
    if (r < rows && c < cols) tile[i][threadIdx.x] = in[(size_t)r * cols + c];
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int c = bx + i, r = by + threadIdx.x;
    if (r < rows && c < cols) out[(size_t)c * rows + r] = tile[threadIdx.x][i];
  }
}

void transpose(const bf16 *in, int rows, int cols, bf16 *out, cudaStream_t st) {
  dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
  transpose_kernel<<<grid, block, 0, st>>>(in, rows, cols, out);
}

// ---------------------------------------------------------------------------
// Training data: parameter draws (Philox per sample) -> FP32 synthesis at the
// plan's grid -> noise -> normalised features (BF16) and encoded targets.
// ---------------------------------------------------------------------------
struct Prior {  // the training distribution
  float b_lo, b_hi, cost_lo, cost_hi, phi_lo, phi_hi, v_sigma, w_lo, w_hi, a_lo, a_hi, eta_lo,
      eta_hi, s, beta_lo, beta_hi, noise;
  // second population (B and eta0 ranges) drawn with probability mix
  float mix, mb_lo, mb_hi, meta_lo, meta_hi;
};

__device__ __forceinline__ void draws16(unsigned long long seed, long long i, float u[16]) {
#pragma unroll
  for (int blk = 0; blk < 4; blk++) {
    uint32_t c[4] = {(uint32_t)((unsigned long long)i & 0xffffffffu),
                     (uint32_t)((unsigned long long)i >> 32), 0x4D4C5000u, (uint32_t)blk};
    philox10(c, (uint32_t)(seed & 0xffffffffu), (uint32_t)(seed >> 32));
#pragma unroll
    for (int k = 0; k < 4; k++) u[blk * 4 + k] = ((float)c[k] + 0.5f) * 2.3283064365386963e-10f;
  }
}

// features of one profile: I / I_max - 1, Q, U, V / I_max (x 10), then the
// training-set standardisation (mean, inv_std); also returns I_max
__device__ __forceinline__ float feature_value(int s, float v, float imax_inv) {
  return s == 0 ? v * imax_inv - 1.f : 10.f * v * imax_inv;
}

// The training set leaves the synthesis in tiles of 128 samples, each value of a
// tile's samples side by side ([tile][column][128]): a thread makes a sample, so
// a warp's stores and the pass back over the profile are contiguous.  131,072
// samples of 60 wavelengths: 212 us, in rows 571; the moments of the features
// and targets and their standardisation (transposed in shared memory) 111, 349.
constexpr int kTile = 128;

__global__ void synth_train_kernel(const __grid_constant__ DevPlan P, Prior pr,
                                   unsigned long long seed, long long n, int ld, float *Xraw,
                                   float *Tgt) {
  __shared__ float s_tab[100];
  __shared__ float s_rden[kRden * kTile];
  VoigtK<float> K;
  voigt_block_setup<float>(K, P, s_tab);
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float u[16];
  draws16(seed, i, u);
  double par[9];
  const bool second = u[9] < pr.mix;  // u[9]: the population
  par[0] = second ? pr.mb_lo + (pr.mb_hi - pr.mb_lo) * u[0] : pr.b_lo + (pr.b_hi - pr.b_lo) * u[0];
  const double cost = pr.cost_lo + (pr.cost_hi - pr.cost_lo) * u[1];
  par[1] = acos(cost);
  par[2] = pr.phi_lo + (pr.phi_hi - pr.phi_lo) * u[2];
  // Box-Muller for v
  par[3] = pr.v_sigma * sqrt(-2.0 * log((double)u[3])) * cos(6.283185307179586 * u[4]);
  par[4] = pr.w_lo + (pr.w_hi - pr.w_lo) * u[5];
  par[5] = pr.a_lo + (pr.a_hi - pr.a_lo) * u[6];
  par[6] = second ? pr.meta_lo + (pr.meta_hi - pr.meta_lo) * u[7]
                  : pr.eta_lo + (pr.eta_hi - pr.eta_lo) * u[7];
  par[7] = pr.s;
  par[8] = pr.beta_lo + (pr.beta_hi - pr.beta_lo) * u[8];
  SynthCall<float> c;
  synth_setup<float>(c, par, P, P.step);
  voigt_prepare<float>(K, c.p5, s_rden + threadIdx.x, blockDim.x);
  const float ones[4] = {1.f, 1.f, 1.f, 1.f};
  const int nl = P.nl;
  // this sample's column of its tile: the profile, then the features
  float *xr = Xraw + (size_t)blockIdx.x * ld * kTile + threadIdx.x;
  float imax = 0.f;
  unsigned long long nseed = seed ^ 0x9E3779B97F4A7C15ull;
  for (int iw = 0; iw < nl; iw++) {
    float syn[4];
    if (P.nsub > 1)
      channel_point<float, false, true>(c, P, K, ones, iw, syn, nullptr);
    else
      channel_point<float, false, false>(c, P, K, ones, iw, syn, nullptr);
    // noise: 4 normals per wavelength from one Philox call
    uint32_t cc[4] = {(uint32_t)((unsigned long long)i & 0xffffffffu),
                      (uint32_t)((unsigned long long)i >> 32), (uint32_t)iw, 0x4E4F4953u};
    philox10(cc, (uint32_t)(nseed & 0xffffffffu), (uint32_t)(nseed >> 32));
#pragma unroll
    for (int s = 0; s < 4; s += 2) {
      const float u1 = ((float)cc[s] + 0.5f) * 2.3283064365386963e-10f;
      const float u2 = ((float)cc[s + 1] + 0.5f) * 2.3283064365386963e-10f;
      const float r = sqrtf(-2.f * logf(u1));
      float sn, cs;
      sincosf(6.2831853f * u2, &sn, &cs);
      syn[s] += pr.noise * r * cs;
      syn[s + 1] += pr.noise * r * sn;
    }
#pragma unroll
    for (int s = 0; s < 4; s++) xr[(size_t)(s * nl + iw) * kTile] = syn[s];
    imax = fmaxf(imax, syn[0]);
  }
  const float inv = 1.f / imax;
  for (int k = 0; k < 4 * nl; k++) {
    float *x = xr + (size_t)k * kTile;
    *x = feature_value(k < nl ? 0 : 1, *x, inv);
  }
  for (int k = 4 * nl; k < ld; k++) xr[(size_t)k * kTile] = 0.f;
  float *t = Tgt + (size_t)blockIdx.x * kOut * kTile + threadIdx.x;
  t[0 * kTile] = (float)par[0];
  t[1 * kTile] = (float)cost;
  t[2 * kTile] = (float)sin(2.0 * par[2]);
  t[3 * kTile] = (float)cos(2.0 * par[2]);
  t[4 * kTile] = (float)par[3];
  t[5 * kTile] = (float)par[4];
  t[6 * kTile] = (float)par[5];
  t[7 * kTile] = (float)par[6];
  t[8 * kTile] = (float)par[8];
  t[9 * kTile] = (float)(par[7] * inv);
}

// Sums and sums of squares of the columns of n tiled samples, in FP64: a warp
// per column and share of the tiles into part [gridDim.y][cols][2], added up in
// order by moments_sum_kernel.
__global__ void moments_kernel(const float *x, long long n, int cols, double *part) {
  const int col = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (col >= cols) return;
  double s = 0, s2 = 0;
  for (long long t = blockIdx.y; t * kTile < n; t += gridDim.y) {
    const float4 f = __ldg(reinterpret_cast<const float4 *>(
        x + ((size_t)t * cols + col) * kTile + lane * 4));
    const double v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (t * kTile + lane * 4 + e < n) {
        s += v[e];
        s2 += v[e] * v[e];
      }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if (lane == 0) {
    part[((size_t)blockIdx.y * cols + col) * 2] = s;
    part[((size_t)blockIdx.y * cols + col) * 2 + 1] = s2;
  }
}

__global__ void moments_sum_kernel(const double *part, int shares, int cols, double *sum) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * cols) return;
  double s = 0;
  for (int k = 0; k < shares; k++) s += part[(size_t)k * 2 * cols + i];
  sum[i] = s;
}

// (x - mean) * istd of tiled samples, 32 columns of a tile per CTA, as the BF16
// rows X [n][cols] (cols % 32 == 0)
__global__ void __launch_bounds__(256)
    standardise_kernel(const float *x, long long n, int cols, const float *mean,
                       const float *istd, bf16 *X) {
  __shared__ __nv_bfloat162 s_out[kTile][17];
  const int c0 = blockIdx.y * 32;
  for (int i = threadIdx.x; i < 16 * kTile; i += 256) {
    const int c = c0 + 2 * (i / kTile), r = i % kTile;
    const float *p = x + ((size_t)blockIdx.x * cols + c) * kTile + r;
    s_out[r][i / kTile] = __floats2bfloat162_rn((__ldg(p) - __ldg(mean + c)) * __ldg(istd + c),
                                                (__ldg(p + kTile) - __ldg(mean + c + 1)) *
                                                    __ldg(istd + c + 1));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * kTile; i += 256) {
    const long long r = (long long)blockIdx.x * kTile + i / 16;
    if (r < n)
      *reinterpret_cast<__nv_bfloat162 *>(X + (size_t)r * cols + c0 + 2 * (i % 16)) =
          s_out[i / 16][i % 16];
  }
}

// the same of tiled targets, as FP32 rows [n][kOut]
__global__ void standardise_targets_kernel(const float *x, long long n, const float *mean,
                                           const float *istd, float *T) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float *p = x + (size_t)(i / kTile) * kOut * kTile + i % kTile;
#pragma unroll
  for (int k = 0; k < kOut; k++) T[(size_t)i * kOut + k] = (p[k * kTile] - mean[k]) * istd[k];
}

// features of map profiles (FP64 [n][4][nl]) for inference, standardised:
// one warp per profile, each lane on pairs of consecutive features, so that a
// warp reads 512 contiguous bytes (16-byte loads when the profiles are 16-byte
// aligned, VEC) and writes 128 contiguous bytes per step.  Every value is the
// same expression of the same inputs as in the training features.
template <bool VEC>
__global__ void __launch_bounds__(256)
    map_features_kernel(const double *__restrict__ prof, long long n, int nl, int ld,
                        const float *__restrict__ mean, const float *__restrict__ istd, bf16 *X,
                        float *imax_out) {
  const long long i = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= n) return;  // the same for the whole warp
  const double *p = prof + (size_t)i * 4 * nl;
  double imax = 0.0;
  for (int iw = lane; iw < nl; iw += 32) imax = fmax(imax, p[iw]);
#pragma unroll
  for (int o = 16; o; o >>= 1) imax = fmax(imax, __shfl_xor_sync(0xffffffffu, imax, o));
  const float inv = imax > 0 ? (float)(1.0 / imax) : 0.f;
  __nv_bfloat162 *x = reinterpret_cast<__nv_bfloat162 *>(X + (size_t)i * ld);
  const int nf = 4 * nl;  // even, so a pair starting below nf ends below it
  for (int k = 2 * lane; k < ld; k += 64) {
    float v0 = 0.f, v1 = 0.f;  // the padding columns stay zero
    if (k < nf) {
      double q0, q1;
      if (VEC) {
        const double2 q = *reinterpret_cast<const double2 *>(p + k);
        q0 = q.x;
        q1 = q.y;
      } else {
        q0 = p[k];
        q1 = p[k + 1];
      }
      v0 = (feature_value(k / nl, (float)q0, inv) - mean[k]) * istd[k];
      v1 = (feature_value((k + 1) / nl, (float)q1, inv) - mean[k + 1]) * istd[k + 1];
    }
    x[k >> 1] = __floats2bfloat162_rn(v0, v1);
  }
  if (lane == 0) imax_out[i] = (float)imax;
}

// network outputs (standardised, one row y) -> the nine ME parameters p[9] (FP64)
__device__ __forceinline__ void decode_row(const float *y, const float *tmean, const float *tstd,
                                           float imax, double *p) {
  float t[kOut];
#pragma unroll
  for (int k = 0; k < kOut; k++) t[k] = y[k] * tstd[k] + tmean[k];
  p[0] = fmax((double)t[0], 0.0);
  p[1] = acos(fmin(fmax((double)t[1], -1.0), 1.0));
  double phi = 0.5 * atan2((double)t[2], (double)t[3]);
  if (phi < 0) phi += kPi;
  p[2] = phi;
  p[3] = t[4];
  p[4] = t[5];
  p[5] = t[6];
  p[6] = t[7];
  p[7] = (double)t[9] * imax;
  p[8] = t[8];
}

__global__ void decode_kernel(const float *Y, long long n, int ld, const float *tmean,
                              const float *tstd, const float *imax, double *par) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  decode_row(Y + (size_t)i * ld, tmean, tstd, imax[i], par + (size_t)i * 9);
}

// ---------------------------------------------------------------------------
// The whole inference of a map in one kernel: features, the four layers on the
// tensor cores, the decode.  A CTA holds two tiles of 128 profiles, each with
// eight working warps, which write the features, and after each layer the
// activations, as BF16 into the tile the next layer reads (K-major, 128-byte
// swizzle).  One more warp brings the weights in (TMA, 64 inputs of a layer per
// stage) and one issues the MMAs into each tile's 256 FP32 tensor-memory
// columns, for one tile while the other is in its epilogue: with the loads on
// the issuing lane, and half of N per instruction, a layer's MMAs took 7,100
// cycles, as they are 2,500.  Rows of more than 256 features go through the
// first layer in pieces of 256.  Nothing of a profile's activations leaves the
// SM.  The epilogues bound it, by their instructions: some 45 per GELU (erff,
// as in the separate kernels: its results are rounded to BF16, and another form
// would turn some of them), 69 of the 97 thousand cycles of a pair of tiles;
// the features take another 12, with the next pair's profiles asked into L2
// ahead of time (before that, and with a row's loads in pairs only, 40).
// The values are those of map_features_kernel, umma_gemm_kernel and
// decode_kernel, which did this in six launches with every layer's activations
// through memory.  Profiles of 60 wavelengths, there and here, us:
//   1: 46, 45;  1,000: 52, 47;  18,900: 89, 50;  37,889: 162, 96;  300,007: 920, 496
// and of 112: 18,900: 102, 55;  75,000: 311, 164.  Few profiles of more features
// go through the six launches all the same: see predict_separately.
// Waits are bounded.  The first to run out writes a code to *err (1: weights, 2: a
// free stage, 3: the accumulator) and raises the CTA's stop flag, at which all
// other waits end too.  The named barriers have no limit: every warp passes each
// of them once per phase with bar.sync, whatever its waits gave, so that none
// runs ahead and none is left behind.  Results are then left unwritten, and the
// CTA ends once its own copies have landed and its MMAs are done.
// ---------------------------------------------------------------------------
constexpr int kPredWarps = 8;  // per tile
constexpr int kPredThreads = (2 * kPredWarps + 2) * 32;
constexpr int kPredK = 256;                          // features per piece
constexpr int kPredBox = 128 * me::umma::kBK * 2;  // a box of weights
constexpr int kPredStage = 2 * kPredBox;           // 64 inputs of a layer
constexpr int kPredStages = 3;
constexpr int kPredA = (kPredK / me::umma::kBK) * me::umma::kStageA;
constexpr int kPredBars = 128;  // mbarriers, tensor-memory base, stop flag
constexpr int kPredSmem = 2 * kPredA + kPredStages * kPredStage + kPredBars + 2 * 128 * 4;

struct PredNet {
  const float *bias[kLayers];
  const float *fmean, *fistd, *tmean, *tstd;
};

// The limit of a kernel's waits and, for tests of what follows when one runs
// out, a kind of event that arrives nowhere: a barrier's address is taken here,
// once, so that it costs the loops nothing.
struct WaitRules {
  uint32_t tries = me::umma::kWaitTries;
  int drop = 0;  // 1: the loads of weights, 2: the MMAs' completion, 3: the stages' release
};

// mbar_wait for a CTA's roles: false, with the error and the stop flag raised,
// when it runs out.
__device__ __forceinline__ bool role_wait(uint32_t bar, uint32_t parity, const WaitRules &rules,
                                          volatile uint32_t *stop, int *err, int code) {
  if (me::umma::mbar_wait(bar, parity, rules.tries, stop)) return true;
  if (!*stop) atomicCAS(err, 0, code);
  *stop = 1;
  return false;
}

// values k and k + 1 (k even, so both or neither are in) of a profile
template <bool VEC>
__device__ __forceinline__ double2 load_pair(const double *p, bool in) {
  if (!in) return make_double2(0.0, 0.0);
  if (VEC) return __ldg(reinterpret_cast<const double2 *>(p));
  return make_double2(__ldg(p), __ldg(p + 1));
}

template <bool VEC>
__global__ void __launch_bounds__(kPredThreads, 1)
    mlp_predict_kernel(const __grid_constant__ CUtensorMap w0,
                       const __grid_constant__ CUtensorMap w1,
                       const __grid_constant__ CUtensorMap w2,
                       const __grid_constant__ CUtensorMap w3, const PredNet net,
                       const __grid_constant__ WaitRules rules,
                       const double *__restrict__ prof, long long n, int nl, int nip,
                       double *__restrict__ par, int *__restrict__ err) {
  using namespace me::umma;
  extern __shared__ __align__(1024) uint8_t pred_smem[];
  const uint32_t base = smem_u32(pred_smem);
  const uint32_t sW = base + 2 * kPredA, bars = sW + kPredStages * kPredStage;
  // full[s] = bars + 8 s, empty[s] after them, then done[tile], drain, and one for
  // each stage and tile that nothing waits for
  const uint32_t done = bars + 8 * 2 * kPredStages, drain = done + 16, spare = drain + 8;
  uint32_t *misc = reinterpret_cast<uint32_t *>(pred_smem + (spare + 8 * kPredStages - base));
  volatile uint32_t *stop = misc + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    tmem_alloc(smem_u32(misc), 512);
    tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < 3 * kPredStages + 3; s++) mbar_init(bars + 8 * s, 1);
    *stop = (base & 1023u) ? 1u : 0u;
    if (base & 1023u) atomicExch(err, 1);  // the tiles need their alignment
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const long long tiles = (n + kBM - 1) / kBM;
  const int pieces = (nip + kPredK - 1) / kPredK;
  const int last_blocks = (nip - (pieces - 1) * kPredK + kBK - 1) / kBK;
  // tile g of this CTA's k-th pair: blockIdx.x + (2 k + g) gridDim.x
  const long long mine0 = (tiles - 1 - blockIdx.x) / gridDim.x + 1;  // (grid <= tiles)

  // Stages of weights in the order the MMAs use them: per phase (a piece of the
  // first layer, or a layer) and tile, its blocks of 64 inputs.
  const int phases = pieces + 3;
  auto blocks_of = [&](int ph) { return ph == pieces - 1 ? last_blocks : 4; };
  if (warp == 2 * kPredWarps + 1) {
    if (lane == 0 && !*stop) {
      uint32_t st = 0, par = 1;  // parity that empty[st] waits for (fresh: passes)
      const uint32_t landed = rules.drop == 1 ? spare : bars;
      bool dead = false;
      for (int todo = (int)mine0; todo > 0 && !dead; todo -= 2) {
        if (VEC)  // the next pair's profiles into L2
          for (int g = 2; g < 4 && g < todo; g++) {
            const long long r = (blockIdx.x + (mine0 - todo + g) * gridDim.x) * kBM;
            l2_prefetch(prof + (size_t)r * 4 * nl,
                        (uint32_t)min((long long)kBM, n - r) * (uint32_t)nl * 32u);
          }
        for (int ph = 0; ph < phases && !dead; ph++)
          for (int g = 0; g < 2 && g < todo && !dead; g++)
            for (int kb = 0; kb < blocks_of(ph); kb++) {
              if (!role_wait(bars + 8 * (kPredStages + st), par, rules, stop, err, 2)) {
                dead = true;
                break;
              }
              const uint32_t full = landed + 8 * st, dst = sW + st * kPredStage;
              if (ph == phases - 1) {
                mbar_expect_tx(full, 32 * kBK * 2);
                tma_load_2d(dst, &w3, full, kb * kBK, 0);
              } else {
                const CUtensorMap *w = ph < pieces ? &w0 : ph == pieces ? &w1 : &w2;
                const int k = (ph < pieces ? ph * kPredK : 0) + kb * kBK;
                mbar_expect_tx(full, kPredStage);
                tma_load_2d(dst, w, full, k, 0);
                tma_load_2d(dst + kPredBox, w, full, k, 128);
              }
              if (++st == kPredStages) st = 0, par ^= 1;
            }
      }
      // the last copies, which no MMA may have read, land before the CTA ends
      for (uint32_t i = 0; i < kPredStages; i++)
        mbar_wait(landed + 8 * i, i < st ? par ^ 1 : par, rules.tries);
    }
    __syncwarp();
  } else if (warp == 2 * kPredWarps) {
    uint32_t st = 0, par = 0;
    const uint32_t freed = rules.drop == 3 ? spare : bars + 8 * kPredStages;
    const uint32_t ended = rules.drop == 2 ? spare : done;
    bool dead = *stop != 0;
    const uint64_t descW = sw128_kmajor_desc(sW);
    for (int todo = (int)mine0; todo > 0; todo -= 2)
      for (int ph = 0; ph < phases; ph++)
        for (int g = 0; g < 2 && g < todo; g++) {
          if (g == 0)
            asm volatile("bar.sync 1, %0;" ::"n"((kPredWarps + 1) * 32) : "memory");
          else
            asm volatile("bar.sync 2, %0;" ::"n"((kPredWarps + 1) * 32) : "memory");
          tc_fence_after();
          if (lane == 0 && !dead) {
            const uint32_t idesc = idesc_bf16_f32(kBM, ph == phases - 1 ? 32 : 256);
            uint64_t da = sw128_kmajor_desc(base + g * kPredA);
            const uint32_t d = tmem + (uint32_t)(g * 256);
            const int count = blocks_of(ph);
            const bool fresh = ph == 0 || ph >= pieces;
            for (int kb = 0; kb < count; kb++) {
              if (!role_wait(bars + 8 * st, par, rules, stop, err, 1)) {
                dead = true;
                break;
              }
              tc_fence_after();
              // (a slice's address enters its descriptor in units of 16 bytes)
              const uint64_t db = descW + (uint64_t)(st * (kPredStage >> 4));
              umma_bf16(d, da, db, idesc, !(fresh && kb == 0));
              umma_bf16(d, da + 2, db + 2, idesc, 1);
              umma_bf16(d, da + 4, db + 4, idesc, 1);
              umma_bf16(d, da + 6, db + 6, idesc, 1);
              mma_commit(freed + 8 * st);
              da += kStageA >> 4;
              if (++st == kPredStages) st = 0, par ^= 1;
            }
            if (!dead) mma_commit(ended + 8 * g);
          }
          __syncwarp();
        }
    if (lane == 0 && *stop) {  // what it issued ends before the CTA does
      mma_commit(drain);
      mbar_wait(drain, 0, rules.tries);
    }
    __syncwarp();
  } else {
    const int g = warp / kPredWarps, gw = warp % kPredWarps;
    uint8_t *tileA = pred_smem + g * kPredA;
    float *s_imax = reinterpret_cast<float *>(pred_smem + (bars + kPredBars - base)) + g * 128;
    uint32_t phase = 0;
    auto publish = [&]() {  // the A tile is written and the accumulator read
      fence_smem_to_async();
      tc_fence_before();
      if (g == 0)
        asm volatile("bar.sync 1, %0;" ::"n"((kPredWarps + 1) * 32) : "memory");
      else
        asm volatile("bar.sync 2, %0;" ::"n"((kPredWarps + 1) * 32) : "memory");
    };
    auto group_sync = [&]() {
      if (g == 0)
        asm volatile("bar.sync 3, %0;" ::"n"(kPredWarps * 32) : "memory");
      else
        asm volatile("bar.sync 4, %0;" ::"n"(kPredWarps * 32) : "memory");
    };
    auto finished = [&]() {  // this phase's MMAs are done
      role_wait(done + 8 * g, phase & 1u, rules, stop, err, 3);
      __syncwarp();
      phase++;
      tc_fence_after();
    };
    const int row = (gw & 3) * 32 + lane;  // this thread's row in the epilogues
    const uint32_t trow = tmem + (uint32_t)(g * 256) + ((uint32_t)((gw & 3) * 32) << 16);
    const int col0 = (gw >> 2) * 128;
    const int nf = 4 * nl;
    for (long long tile = blockIdx.x + (long long)g * gridDim.x; tile < tiles;
         tile += 2LL * gridDim.x) {
      const long long r0 = tile * kBM + gw * 16;  // this warp's rows of features
      const double *p0 = prof + (size_t)r0 * nf;
      // I_max, eight rows at a time: each lane's maxima, then a butterfly that
      // halves the rows a lane holds at each of its first three steps; lanes
      // 4 r .. 4 r + 3 end with row r's.
      float my_inv[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        double m[8];
#pragma unroll
        for (int r = 0; r < 8; r++) m[r] = 0.0;
#pragma unroll 1
        for (int k = 2 * lane; k < nl; k += 64) {
          double2 v[8];
#pragma unroll
          for (int r = 0; r < 8; r++)
            v[r] = load_pair<VEC>(p0 + (size_t)(8 * h + r) * nf + k, r0 + 8 * h + r < n);
          const bool both = k + 1 < nl;
#pragma unroll
          for (int r = 0; r < 8; r++) m[r] = fmax(fmax(m[r], v[r].x), both ? v[r].y : 0.0);
        }
#pragma unroll
        for (int w = 4; w; w >>= 1) {
          const bool up = lane & (4 * w);
#pragma unroll
          for (int r = 0; r < w; r++) {
            const double got = __shfl_xor_sync(0xffffffffu, up ? m[r] : m[r + w], 4 * w);
            m[r] = fmax(up ? m[r + w] : m[r], got);
          }
        }
        m[0] = fmax(m[0], __shfl_xor_sync(0xffffffffu, m[0], 2));
        m[0] = fmax(m[0], __shfl_xor_sync(0xffffffffu, m[0], 1));
        my_inv[h] = m[0] > 0 ? (float)(1.0 / m[0]) : 0.f;
        if (!(lane & 3)) s_imax[gw * 16 + 8 * h + (lane >> 2)] = (float)m[0];
      }
      for (int pc = 0; pc < pieces; pc++) {
        if (pc) finished();  // the piece before has been read
        const int blocks = pc < pieces - 1 ? kPredK / kBK : last_blocks;
#pragma unroll 1
        for (int b = 0; b < blocks; b++) {
          const int k = pc * kPredK + b * kBK + 2 * lane;
          const bool in = k < nf;
          double2 v[16];
#pragma unroll
          for (int r = 0; r < 16; r++)
            v[r] = load_pair<VEC>(p0 + (size_t)r * nf + k, in && r0 + r < n);
          float2 mean = make_float2(0.f, 0.f), istd = mean;
          if (in) {
            mean = __ldg(reinterpret_cast<const float2 *>(net.fmean + k));
            istd = __ldg(reinterpret_cast<const float2 *>(net.fistd + k));
          }
#pragma unroll
          for (int r = 0; r < 16; r++) {
            const float inv = __shfl_sync(0xffffffffu, my_inv[r >> 3], 4 * (r & 7));
            const float f0 =
                (feature_value(k < nl ? 0 : 1, (float)v[r].x, inv) - mean.x) * istd.x;
            const float f1 =
                (feature_value(k + 1 < nl ? 0 : 1, (float)v[r].y, inv) - mean.y) * istd.y;
            *reinterpret_cast<__nv_bfloat162 *>(
                tileA + sw128_offset(gw * 16 + r, b * kBK + 2 * lane)) =
                __floats2bfloat162_rn(in ? f0 : 0.f, in ? f1 : 0.f);  // (zeros in the padding)
          }
        }
        publish();
      }
      for (int l = 0; l < 3; l++) {
        finished();
        const float *bias = net.bias[l];
#pragma unroll 1
        for (int c = col0; c < col0 + 128; c += 16) {
          float bv[16], v[16];
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            const float4 f = __ldg(reinterpret_cast<const float4 *>(bias + c + j));
            bv[j] = f.x, bv[j + 1] = f.y, bv[j + 2] = f.z, bv[j + 3] = f.w;
          }
          tmem_ld16(trow + (uint32_t)c, v);
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] += bv[j];
          uint32_t pk[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(gelu_f(v[2 * j]), gelu_f(v[2 * j + 1]));
            pk[j] = *reinterpret_cast<const uint32_t *>(&h);
          }
          *reinterpret_cast<uint4 *>(tileA + sw128_offset(row, c)) =
              make_uint4(pk[0], pk[1], pk[2], pk[3]);
          *reinterpret_cast<uint4 *>(tileA + sw128_offset(row, c + 8)) =
              make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        publish();
      }
      finished();
      group_sync();  // s_imax is whole
      if (gw < 4) {
        float y[16];
        tmem_ld16(trow, y);
        const long long i = tile * kBM + row;
#pragma unroll
        for (int j = 0; j < kOut; j++) y[j] += __ldg(net.bias[3] + j);
        if (i < n && !*stop)
          decode_row(y, net.tmean, net.tstd, s_imax[row], par + (size_t)i * 9);
      }
      group_sync();  // the next tile's I_max must not overtake the decode
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

bool predict_kernel_ready() {
  const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
  return cudaFuncSetAttribute(mlp_predict_kernel<true>, a, kPredSmem) == cudaSuccess &&
         cudaFuncSetAttribute(mlp_predict_kernel<false>, a, kPredSmem) == cudaSuccess;
}

// ---------------------------------------------------------------------------
// A training step up to the gradients' operands in one kernel: the batch's
// gather, the forward pass, the loss and the backward pass to every layer's
// dZ.  A CTA takes 32 rows of the batch, so that a batch of 4096 fills 128 SMs,
// and computes each layer transposed: the weights are the 256 (two times 128)
// rows of the MMA and the batch rows its columns.  So a thread's accumulators
// are 16 batch rows of one neuron: the layer's output leaves for the weight
// gradient's transposed operand as 32-byte stores, the bias is one value, the
// bias gradient a sum in registers, and the pre-activations of the three hidden
// layers stay in registers until the backward pass asks for them.  The next
// operand is written to shared memory as in mlp_predict_kernel, whose warps of
// loads and of MMAs this has too; a layer's weights fill the four stages, so
// they arrive during the epilogue before them.  The values are those of
// gather_kernel, the GEMMs and their epilogues, mse_grad_kernel and
// gelu_back_kernel (which the mma.sync path runs), each rounded to BF16 at the
// same places.  A CTA's 32 us at a batch of 4096: gathering 2, the epilogues'
// instructions 12 (erff, and in the backward pass expf), the MMAs and the
// weights they wait for 11.  With mlp_wgrad_kernel (12 us) and adam_kernel (7)
// a step takes 55 us, as 44 launches it took 248; with a batch of 256, 48 (190);
// of 65,536, 520 (1,250).
// ---------------------------------------------------------------------------
constexpr int kStepRows = 32, kStepWarps = 16;
constexpr int kStepThreads = (kStepWarps + 2) * 32;
constexpr int kStepStages = 4;
constexpr int kStepBlock = kStepRows * me::umma::kBK * 2;  // 64 inputs of the batch rows
constexpr int kStepBars = 128;
constexpr int kStepSmem = kStepStages * kPredStage + 4 * kStepBlock + kStepBars;

struct StepMaps {
  CUtensorMap w[kLayers];  // W [dout][din]
  CUtensorMap t[kLayers];  // W^T [din][dout], layers 1..
};
struct StepNet {
  const float *bias[kLayers];
  bf16 *xt;               // [nip][B]: the batch, transposed
  bf16 *at[kLayers - 1];  // [256][B]: the hidden layers' outputs
  bf16 *dzt[kLayers];     // [dout][B]: dZ
  float *gb[kLayers];     // += the bias gradients
};

__device__ __forceinline__ uint32_t step_offset(int row, int k) {
  return (uint32_t)(k / me::umma::kBK) * kStepBlock + (uint32_t)row * 128 +
         ((((uint32_t)(k % me::umma::kBK) >> 3) ^ ((uint32_t)row & 7)) << 4) +
         ((uint32_t)k & 7) * 2;
}

__global__ void __launch_bounds__(kStepThreads, 1)
    mlp_step_kernel(const __grid_constant__ StepMaps maps, const __grid_constant__ StepNet net,
                    const __grid_constant__ WaitRules rules, const bf16 *__restrict__ X,
                    const long long *__restrict__ idx, const float *__restrict__ T, int B,
                    int nip, double *__restrict__ loss, int *__restrict__ err) {
  using namespace me::umma;
  extern __shared__ __align__(1024) uint8_t step_smem[];
  const uint32_t base = smem_u32(step_smem);
  uint8_t *tile = step_smem + kStepStages * kPredStage;
  const uint32_t sX = base + kStepStages * kPredStage, bars = sX + 4 * kStepBlock;
  // full[s] = bars + 8 s, empty[s] after them, then done, drain and the spare
  // ones; waits and barriers as in mlp_predict_kernel
  const uint32_t done = bars + 8 * 2 * kStepStages, drain = done + 8, spare = drain + 8;
  uint32_t *misc = reinterpret_cast<uint32_t *>(step_smem + (spare + 8 * kStepStages - base));
  volatile uint32_t *stop = misc + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    tmem_alloc(smem_u32(misc), 64);
    tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < 3 * kStepStages + 2; s++) mbar_init(bars + 8 * s, 1);
    *stop = (base & 1023u) ? 1u : 0u;
    if (base & 1023u) atomicExch(err, 1);  // the tiles need their alignment
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const int row0 = blockIdx.x * kStepRows;
  const int pieces = (nip + kPredK - 1) / kPredK;
  const int last_blocks = (nip - (pieces - 1) * kPredK + kBK - 1) / kBK;
  // phases: the first layer's pieces, layers 1 and 2, the outputs, then back
  // through the outputs' weights and layers 2 and 1
  const int phases = pieces + 6, out = pieces + 2;
  auto blocks_of = [&](int ph) { return ph == pieces - 1 ? last_blocks : ph == out + 1 ? 1 : 4; };

  if (warp == kStepWarps + 1) {
    if (lane == 0 && !*stop) {
      uint32_t st = 0, par = 1;  // parity that empty[st] waits for (fresh: passes)
      const uint32_t landed = rules.drop == 1 ? spare : bars;
      bool dead = false;
      for (int ph = 0; ph < phases && !dead; ph++) {
        const CUtensorMap *w = ph < pieces ? &maps.w[0]
                               : ph <= out ? &maps.w[ph - pieces + 1]
                                           : &maps.t[kLayers - (ph - out)];
        for (int kb = 0; kb < blocks_of(ph); kb++) {
          if (!role_wait(bars + 8 * (kStepStages + st), par, rules, stop, err, 2)) {
            dead = true;
            break;
          }
          const uint32_t full = landed + 8 * st, dst = base + st * kPredStage;
          const int k = (ph < pieces ? ph * kPredK : 0) + kb * kBK;
          mbar_expect_tx(full, ph == out ? 32 * kBK * 2 : kPredStage);
          tma_load_2d(dst, w, full, k, 0);
          if (ph != out) tma_load_2d(dst + kPredBox, w, full, k, 128);
          if (++st == kStepStages) st = 0, par ^= 1;
        }
      }
      // the last copies, which no MMA may have read, land before the CTA ends
      for (uint32_t i = 0; i < kStepStages; i++)
        mbar_wait(landed + 8 * i, i < st ? par ^ 1 : par, rules.tries);
    }
    __syncwarp();
  } else if (warp == kStepWarps) {
    uint32_t st = 0, par = 0;
    const uint32_t freed = rules.drop == 3 ? spare : bars + 8 * kStepStages;
    const uint32_t ended = rules.drop == 2 ? spare : done;
    bool dead = *stop != 0;
    const uint64_t descW = sw128_kmajor_desc(base);
    const uint32_t idesc = idesc_bf16_f32(kBM, kStepRows);
    for (int ph = 0; ph < phases; ph++) {
      asm volatile("bar.sync 1, %0;" ::"n"((kStepWarps + 1) * 32) : "memory");
      tc_fence_after();
      if (lane == 0 && !dead) {
        uint64_t db = sw128_kmajor_desc(sX);
        const int count = blocks_of(ph);
        const bool fresh = ph == 0 || ph >= pieces;
        for (int kb = 0; kb < count; kb++) {
          if (!role_wait(bars + 8 * st, par, rules, stop, err, 1)) {
            dead = true;
            break;
          }
          tc_fence_after();
          // (a slice's address enters its descriptor in units of 16 bytes)
          const uint64_t da = descW + (uint64_t)(st * (kPredStage >> 4));
          const int slices = ph == out + 1 ? kOutRows / 16 : 4;
          for (int k = 0; k < slices; k++) {  // (the halves in turn: each MMA waits for its
            const uint32_t add = !(fresh && kb == 0 && k == 0);  // accumulator's last)
            umma_bf16(tmem, da + 2 * k, db + 2 * k, idesc, add);
            if (ph != out)
              umma_bf16(tmem + kStepRows, da + (kPredBox >> 4) + 2 * k, db + 2 * k, idesc, add);
          }
          mma_commit(freed + 8 * st);
          db += kStepBlock >> 4;
          if (++st == kStepStages) st = 0, par ^= 1;
        }
        if (!dead) mma_commit(ended);
      }
      __syncwarp();
    }
    if (lane == 0 && *stop) {  // what it issued ends before the CTA does
      mma_commit(drain);
      mbar_wait(drain, 0, rules.tries);
    }
    __syncwarp();
  } else {
    uint32_t phase = 0;
    auto publish = [&]() {  // the operand is written and the accumulator read
      fence_smem_to_async();
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"((kStepWarps + 1) * 32) : "memory");
    };
    auto workers = [&]() {
      asm volatile("bar.sync 2, %0;" ::"n"(kStepWarps * 32) : "memory");
    };
    auto finished = [&]() {  // this phase's MMAs are done
      role_wait(done, phase & 1u, rules, stop, err, 3);
      __syncwarp();
      phase++;
      tc_fence_after();
    };
    // the batch
    for (int pc = 0; pc < pieces; pc++) {
      if (pc) finished();  // the piece before has been read
      const int blocks = pc < pieces - 1 ? 4 : last_blocks;
      for (int i = threadIdx.x; i < kStepRows * blocks * 8; i += kStepWarps * 32) {
        const int r = i / (blocks * 8), c = i % (blocks * 8), k = pc * kPredK + c * 8;
        uint4 v = make_uint4(0, 0, 0, 0);  // zeros past the features
        if (k < nip)
          v = __ldg(reinterpret_cast<const uint4 *>(X + (size_t)__ldg(idx + row0 + r) * nip + k));
        *reinterpret_cast<uint4 *>(tile + step_offset(r, c * 8)) = v;
      }
      publish();
      workers();
      for (int i = threadIdx.x; i < 2 * blocks * kBK; i += kStepWarps * 32) {
        const int c = i >> 1, r = (i & 1) * 16, k = pc * kPredK + c;
        if (k >= nip) continue;
        uint32_t pk[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
          pk[j] = *reinterpret_cast<const uint16_t *>(tile + step_offset(r + 2 * j, c)) |
                  (uint32_t)*reinterpret_cast<const uint16_t *>(
                      tile + step_offset(r + 2 * j + 1, c))
                      << 16;
        uint4 *o = reinterpret_cast<uint4 *>(net.xt + (size_t)k * B + row0 + r);
        o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
      workers();  // the tile has been read
    }
    // this thread's neuron and 16 batch rows
    const int neuron = ((warp >> 2) & 1) * 128 + (warp & 3) * 32 + lane, r16 = (warp >> 3) * 16;
    const uint32_t acc = tmem + (uint32_t)(((warp >> 2) & 1) * kStepRows + r16) +
                         ((uint32_t)((warp & 3) * 32) << 16);
    // BF16 values as the next operand, and then as the weight gradient's (a fence
    // for the first would wait for the second's stores)
    auto put_next = [&](const float v[16], int n) {
#pragma unroll
      for (int j = 0; j < 16; j++)
        *reinterpret_cast<bf16 *>(tile + step_offset(r16 + j, n)) = __float2bfloat16(v[j]);
    };
    auto put_grad = [&](const float v[16], bf16 *outT, int n) {
      uint32_t pk[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        pk[j] = *reinterpret_cast<const uint32_t *>(&h);
      }
      uint4 *o = reinterpret_cast<uint4 *>(outT + (size_t)n * B + row0 + r16);
      o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    };
    auto column_sum = [&](const float v[16]) {  // of the rounded values
      float t = 0.f;
#pragma unroll
      for (int j = 0; j < 16; j++) t += __bfloat162float(__float2bfloat16(v[j]));
      return t;
    };
    float z[kLayers - 1][16];
#pragma unroll
    for (int l = 0; l < kLayers - 1; l++) {
      const float b = __ldg(net.bias[l] + neuron);
      finished();
      tmem_ld16(acc, z[l]);
      float h[16];
#pragma unroll
      for (int j = 0; j < 16; j++) {
        z[l][j] += b;
        h[j] = gelu_f(z[l][j]);
      }
      put_next(h, neuron);
      publish();
      put_grad(h, net.at[l], neuron);
    }
    if ((warp & 7) == 0) {  // the outputs: lane's, 16 rows
      float v[16], t[16], sq = 0.f;
      const float b = __ldg(net.bias[kLayers - 1] + lane);
#pragma unroll
      for (int j = 0; j < 16; j++)
        t[j] = lane < kOut ? __ldg(T + (size_t)__ldg(idx + row0 + r16 + j) * kOut + lane) : 0.f;
      finished();
      tmem_ld16(acc, v);
#pragma unroll
      for (int j = 0; j < 16; j++) {
        float g = 0.f;
        if (lane < kOut) {
          const float d = v[j] + b - t[j];
          g = 2.f * d / (float)(B * kOut);
          sq += d * d;
        }
        v[j] = g;
      }
      put_next(v, lane);
      publish();
      put_grad(v, net.dzt[kLayers - 1], lane);
      atomicAdd(net.gb[kLayers - 1] + lane, column_sum(v));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (lane == 0) atomicAdd(loss, (double)sq / (double)(B * kOut));
    } else {
      finished();
      publish();
    }
#pragma unroll
    for (int l = kLayers - 2; l >= 0; l--) {
      float v[16];
      finished();
      tmem_ld16(acc, v);
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] *= gelu_grad(z[l][j]);
      if (l > 0) {
        put_next(v, neuron);
        publish();
      }
      put_grad(v, net.dzt[l], neuron);
      atomicAdd(net.gb[l] + neuron, column_sum(v));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 64);
}

// The weight gradients of all layers in one launch, dW_l [dout][din] += dZ_l^T
// [dout][B] times A_l^T [din][B], each a GEMM over the batch divided in `split`
// shares whose CTAs add into dW.  blockIdx.y: the share; blockIdx.x: the 128 x
// kGradN tiles of layer 0, then of the next layers.
constexpr int kGradN = 128;
struct GradMaps {
  CUtensorMap a[kLayers], b[kLayers];
};
struct GradNet {
  float *gw[kLayers];
  int m[kLayers], n[kLayers], tiles[kLayers];
};

__global__ void __launch_bounds__(128, 1)
    mlp_wgrad_kernel(const __grid_constant__ GradMaps maps,
                     const __grid_constant__ GradNet net, int B,
                     int *__restrict__ err) {
  int l = 0, t = blockIdx.x;
  while (l < kLayers - 1 && t >= net.tiles[l]) t -= net.tiles[l++];
  const int across = (net.n[l] + kGradN - 1) / kGradN;
  const int rz = B / (int)gridDim.y;
  umma_tile(&maps.a[l], &maps.b[l], t / across * me::umma::kBM, t % across * kGradN, kGradN,
            blockIdx.y * rz, rz, true, net.m[l], net.n[l], nullptr, nullptr, 0, nullptr,
            net.gw[l], err);
}

bool step_kernels_ready() {
  return cudaFuncSetAttribute(mlp_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kStepSmem) == cudaSuccess &&
         cudaFuncSetAttribute(mlp_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              me::umma::kSmemMax) == cudaSuccess;
}

// ---------------------------------------------------------------------------
// loss and optimiser
// ---------------------------------------------------------------------------
// dY = 2 (Y - T) / (rows * kOut) for the batch rows idx[0..rows) (T standardised,
// [n][kOut]); Y and dY have row stride ld, the columns past kOut get zero.
// loss += mean squared error of the batch.
__global__ void mse_grad_kernel(const float *Yf, int ld, const float *Tstd, const long long *idx,
                                int rows, bf16 *dYb, double *loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float sq = 0.f;
  if (i < rows * ld) {
    const int r = i / ld, k = i % ld;
    float gr = 0.f;
    if (k < kOut) {
      const float d = Yf[i] - Tstd[(size_t)idx[r] * kOut + k];
      gr = 2.f * d / (float)(rows * kOut);
      sq = d * d;
    }
    dYb[i] = __float2bfloat16(gr);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  __shared__ float part[32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += part[w];
    atomicAdd(loss, (double)t / (double)(rows * kOut));
  }
}

// dA_prev = dH * gelu'(Z): BF16 out
__global__ void gelu_back_kernel(const float *dH, const float *Z, long long n, bf16 *dZb) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  dZb[i] = __float2bfloat16(dH[i] * gelu_grad(Z[i]));
}

// db[c] += sum over a chunk of rows of dZ[r][c] (db zeroed before); grid
// (cols / 32, row chunks), block (32, 8)
__global__ void bias_grad_kernel(const bf16 *dZ, int rows, int cols, int rows_per_chunk,
                                 float *db) {
  const int c = blockIdx.x * 32 + threadIdx.x;
  const int r0 = blockIdx.y * rows_per_chunk;
  const int r1 = min(rows, r0 + rows_per_chunk);
  float s = 0.f;
  if (c < cols)
    for (int r = r0 + threadIdx.y; r < r1; r += 8) s += __bfloat162float(dZ[(size_t)r * cols + c]);
  __shared__ float part[8][33];
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) t += part[k][threadIdx.x];
    atomicAdd(db + c, t);
  }
}

// Adam (Kingma & Ba 2015) on all FP32 master parameters at once, refreshing the BF16
// weights and their transposes, and clearing the gradients for the next step.
// Parameters, moments and gradients have one layout of n floats; layer l's
// weights [rows][cols] start at off[l], its biases lie before off[l + 1].
struct AdamNet {
  float *w, *m, *v, *g;
  long long n, off[kLayers];
  int rows[kLayers], cols[kLayers];
  bf16 *wb[kLayers], *wbt[kLayers];
};

__global__ void adam_kernel(const __grid_constant__ AdamNet net, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= net.n) return;
  const float gi = net.g[i];
  net.g[i] = 0.f;
  const float mi = b1 * net.m[i] + (1.f - b1) * gi;
  const float vi = b2 * net.v[i] + (1.f - b2) * gi * gi;
  net.m[i] = mi;
  net.v[i] = vi;
  const float wi = net.w[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  net.w[i] = wi;
  int l = 0;
#pragma unroll
  for (int k = 1; k < kLayers; k++) l = i >= net.off[k] ? k : l;
  const int j = (int)(i - net.off[l]), cols = net.cols[l], rows = net.rows[l];
  if (j >= rows * cols) return;
  const bf16 h = __float2bfloat16(wi);
  net.wb[l][j] = h;
  net.wbt[l][(size_t)(j % cols) * rows + j / cols] = h;
}

// gather rows idx[] of X [n][cols] into Xb [rows][cols]
__global__ void gather_kernel(const bf16 *X, const long long *idx, int rows, int cols, bf16 *Xb) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)rows * cols) return;
  const int r = (int)(i / cols), c = (int)(i % cols);
  Xb[i] = X[(size_t)idx[r] * cols + c];
}

// a random permutation of [0, n) per epoch: Feistel network on the index
// space (cycle-walking), keyed per epoch
__device__ __forceinline__ unsigned long long feistel(unsigned long long x, int bits, uint32_t k0,
                                                      uint32_t k1) {
  const int half = (bits + 1) / 2;
  const unsigned long long mask = (1ull << half) - 1;
  unsigned long long l = x >> half, r = x & mask;
  for (int round = 0; round < 4; round++) {
    uint32_t c[4] = {(uint32_t)r, (uint32_t)round, 0x46454953u, 0};
    philox10(c, k0, k1);
    const unsigned long long f = c[0] & mask;
    const unsigned long long nl = r, nr = (l ^ f) & mask;
    l = nl;
    r = nr;
  }
  return (l << half) | r;
}

__global__ void permute_kernel(long long n, int bits, uint32_t k0, uint32_t k1, long long *perm) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long x = (unsigned long long)i;
  do {
    x = feistel(x, bits, k0, k1);
  } while (x >= (unsigned long long)n);
  perm[i] = (long long)x;
}

}  // namespace mlp
}  // namespace me

// ---------------------------------------------------------------------------
// Host side: model, training, inference, files (C ABI in include/me_b200.h).
// ---------------------------------------------------------------------------
namespace {

using namespace me::mlp;

constexpr int kOutPad = kOutRows;

struct DBuf {
  void *p = nullptr;
  size_t n = 0;
  bool own = true;
  DBuf() = default;
  DBuf(const DBuf &) = delete;
  DBuf &operator=(const DBuf &) = delete;
  ~DBuf() { release(); }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= n) return cudaSuccess;
    release();
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaSuccess)
      n = bytes;
    else
      p = nullptr;
    return e;
  }
  void view(void *q, size_t bytes) {  // a part of another buffer, which outlives this one
    release();
    p = q;
    n = bytes;
    own = false;
  }
  void release() {
    if (p && own) cudaFree(p);
    p = nullptr;
    n = 0;
    own = true;
  }
  template <class T>
  T *as() const {
    return static_cast<T *>(p);
  }
};

int fail(int code, const std::string &m) { return me::record_error(code, m.c_str()); }

#define MCK(call)                                                               \
  do {                                                                          \
    cudaError_t e_ = (call);                                                    \
    if (e_ != cudaSuccess)                                                      \
      return fail(ME_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Parts of one allocation, each on 256 bytes: ask for them, take the memory,
// and the buffers are views of it.
struct Arena {
  struct Part {
    DBuf *d;
    size_t off, bytes;
  };
  std::vector<Part> parts;
  size_t total = 0;
  void add(DBuf &d, size_t bytes) {
    parts.push_back({&d, total, bytes});
    total += (bytes + 255) / 256 * 256;
  }
  void place(void *p) const {
    for (const Part &q : parts) q.d->view(static_cast<char *>(p) + q.off, q.bytes);
  }
};

inline unsigned nblk(long long n, int b = 256) { return (unsigned)((n + b - 1) / b); }

}  // namespace

struct me_mlp {
  int device = 0;
  int nl = 0, nin = 0, nip = 0;  // grid size, features, padded input width
  int din[kLayers], dout[kLayers];
  // per layer: FP32 master W [dout][din] and b, BF16 W and W^T, Adam moments, gradients
  DBuf w[kLayers], b[kLayers], wb[kLayers], wbt[kLayers], mw[kLayers], vw[kLayers], mb[kLayers],
      vb[kLayers], gw[kLayers], gb[kLayers];
  DBuf fmean, fistd, tmean, tstd, tistd;  // feature and target standardisation (device)
  std::vector<float> h_fmean, h_fistd, h_tmean, h_tstd;
  long long adam_t = 0;
  // batch work buffers
  int cap = 0, step_cap = 0;
  DBuf xb, xbt, z[kLayers], a[kLayers], at[kLayers], yf, dyb, dybt, dh, dz, dzt;
  cudaEvent_t batch_used = nullptr;  // the last inference that used them
  DBuf sxt, sat[kLayers - 1], sdzt[kLayers];  // operands of the weight gradients (mlp_step_kernel)
  DBuf loss, imax;
  // the allocations that the buffers above are parts of; the parameters, their
  // moments and their gradients have one layout, of `flat` floats each
  DBuf model, batch, step;
  long long flat = 0;
  WaitRules waits;  // of the fused kernels (me_mlp_set_waits)
  // GEMM kernel choice and the tcgen05 kernel's error flag (device int)
  GemmPath gemm_path = GemmPath::tcgen05;
  DBuf gerr;
  long long gemm_launches[2] = {0, 0};
  TileMapCache maps;
  ~me_mlp() {
    if (batch_used) cudaEventDestroy(batch_used);
  }
};

namespace {

size_t wcount(const me_mlp *m, int l) { return (size_t)m->dout[l] * m->din[l]; }

GemmCtx ctx(me_mlp *m) {
  GemmCtx g;
  g.path = m->gemm_path;
  g.err = m->gerr.as<int>();
  g.launches = m->gemm_launches;
  g.maps = &m->maps;
  return g;
}

// reads and clears the tcgen05 GEMM's error flag (synchronises the device)
int gemm_status(me_mlp *m) {
  if (!m->gerr.p) return ME_OK;
  int e = 0;
  MCK(cudaMemcpy(&e, m->gerr.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (!e) return ME_OK;
  MCK(cudaMemset(m->gerr.p, 0, sizeof(int)));
  static const char *what[] = {"", "operand load", "stage release", "accumulator"};
  return fail(ME_ERR_CUDA, std::string("tensor-core GEMM: wait for the ") +
                               what[e >= 1 && e <= 3 ? e : 0] + " timed out");
}

long long param_count(const me_mlp *m) {
  long long n = 0;
  for (int l = 0; l < kLayers; l++) n += (long long)wcount(m, l) + m->dout[l];
  return n;
}

int ensure_batch(me_mlp *m, int B) {
  if (B <= m->cap) return ME_OK;
  const size_t r = (size_t)B;
  Arena a;
  a.add(m->xb, r * m->nip * 2);
  a.add(m->xbt, r * m->nip * 2);
  for (int l = 0; l < kLayers; l++) {
    a.add(m->z[l], r * m->dout[l] * 4);
    a.add(m->a[l], r * m->dout[l] * 2);
    a.add(m->at[l], r * m->dout[l] * 2);
  }
  a.add(m->yf, r * kOutPad * 4);
  a.add(m->dyb, r * kOutPad * 2);
  a.add(m->dybt, r * kOutPad * 2);
  a.add(m->dh, r * kHidden * 4);
  a.add(m->dz, r * kHidden * 2);
  a.add(m->dzt, r * kHidden * 2);
  a.add(m->imax, r * 4);
  m->cap = 0;
  MCK(m->batch.ensure(a.total));
  a.place(m->batch.p);
  m->cap = B;
  return ME_OK;
}

// the operands of the weight gradients of B rows, in `mem` where they fit
int ensure_step(me_mlp *m, int B, void *mem, size_t bytes) {
  if (!mem && B <= m->step_cap) return ME_OK;
  Arena a;
  a.add(m->sxt, (size_t)B * m->nip * 2);
  for (int l = 0; l < kLayers; l++) {
    if (l < kLayers - 1) a.add(m->sat[l], (size_t)B * m->dout[l] * 2);
    a.add(m->sdzt[l], (size_t)B * m->dout[l] * 2);
  }
  if (a.total <= bytes) {
    a.place(mem);
    return ME_OK;
  }
  m->step_cap = 0;
  MCK(m->step.ensure(a.total));
  a.place(m->step.p);
  m->step_cap = B;
  return ME_OK;
}

__global__ void init_weights_kernel(float *w, long long n, int din, int din_used, int dout_used,
                                    unsigned long long seed, float scale) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = (int)(i % din);
  const long long r = i / din;
  uint32_t cc[4] = {(uint32_t)i, (uint32_t)(i >> 32), 0x494E4954u, 0};
  me::philox10(cc, (uint32_t)seed, (uint32_t)(seed >> 32));
  const float u1 = ((float)cc[0] + 0.5f) * 2.3283064365386963e-10f;
  const float u2 = ((float)cc[1] + 0.5f) * 2.3283064365386963e-10f;
  const float g = sqrtf(-2.f * logf(u1)) * cosf(6.2831853f * u2);
  w[i] = (c < din_used && r < dout_used) ? scale * g : 0.f;
}

// BF16 copy of W [rows][cols] and of its transpose
__global__ void to_bf16_kernel(const float *w, long long n, int cols, int rows, bf16 *wb,
                               bf16 *wbt) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bf16 v = __float2bfloat16(w[i]);
  wb[i] = v;
  const long long r = i / cols, c = i % cols;
  wbt[(size_t)c * rows + r] = v;
}

__global__ void f32_to_bf16_kernel(const float *x, long long n, bf16 *y) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16(x[i]);
}

__global__ void iota_kernel(long long *idx, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) idx[i] = i;
}

int refresh_bf16(me_mlp *m, cudaStream_t st) {
  for (int l = 0; l < kLayers; l++) {
    const long long nw = (long long)wcount(m, l);
    to_bf16_kernel<<<nblk(nw), 256, 0, st>>>(m->w[l].as<float>(), nw, m->din[l], m->dout[l],
                                              m->wb[l].as<bf16>(), m->wbt[l].as<bf16>());
  }
  MCK(cudaGetLastError());
  return ME_OK;
}

int alloc_model(me_mlp *m, int nl) {
  m->nl = nl;
  m->nin = 4 * nl;
  m->nip = (m->nin + 31) / 32 * 32;
  const int din[kLayers] = {m->nip, kHidden, kHidden, kHidden};
  const int dout[kLayers] = {kHidden, kHidden, kHidden, kOutPad};
  for (int l = 0; l < kLayers; l++) {
    m->din[l] = din[l];
    m->dout[l] = dout[l];
  }
  Arena a;
  DBuf *const flat[4][2] = {{m->gw, m->gb}, {m->w, m->b}, {m->mw, m->mb}, {m->vw, m->vb}};
  for (auto &k : flat) {
    for (int l = 0; l < kLayers; l++) {
      a.add(k[0][l], wcount(m, l) * 4);
      a.add(k[1][l], dout[l] * 4);
    }
    if (!m->flat) m->flat = (long long)(a.total / 4);
  }
  for (int l = 0; l < kLayers; l++) {
    a.add(m->wb[l], wcount(m, l) * 2);
    a.add(m->wbt[l], wcount(m, l) * 2);
  }
  a.add(m->fmean, m->nip * 4);
  a.add(m->fistd, m->nip * 4);
  a.add(m->tmean, kOut * 4);
  a.add(m->tstd, kOut * 4);
  a.add(m->tistd, kOut * 4);
  a.add(m->gerr, sizeof(int));
  a.add(m->loss, sizeof(double));
  MCK(m->model.ensure(a.total));
  a.place(m->model.p);
  MCK(cudaMemset(m->model.p, 0, a.total));
  m->h_fmean.assign(m->nip, 0.f);
  m->h_fistd.assign(m->nip, 1.f);
  m->h_tmean.assign(kOut, 0.f);
  m->h_tstd.assign(kOut, 1.f);
  return ME_OK;
}

int upload_standardisation(me_mlp *m) {
  MCK(cudaMemcpy(m->fmean.p, m->h_fmean.data(), m->nip * 4, cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(m->fistd.p, m->h_fistd.data(), m->nip * 4, cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(m->tmean.p, m->h_tmean.data(), kOut * 4, cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(m->tstd.p, m->h_tstd.data(), kOut * 4, cudaMemcpyHostToDevice));
  return ME_OK;
}

// He initialisation (sqrt(2 / fan_in)) for the GELU layers, sqrt(1 / fan_in)
// for the output layer; zero biases; zero weights on the padding
int init_model(me_mlp *m, unsigned long long seed) {
  for (int l = 0; l < kLayers; l++) {
    const long long nw = (long long)wcount(m, l);
    const int din_used = l == 0 ? m->nin : m->din[l];
    const int dout_used = l == kLayers - 1 ? kOut : m->dout[l];
    const float scale = (l == kLayers - 1 ? 1.f : 1.41421356f) / sqrtf((float)din_used);
    init_weights_kernel<<<nblk(nw), 256>>>(m->w[l].as<float>(), nw, m->din[l], din_used,
                                           dout_used, seed * 131 + l, scale);
  }
  MCK(cudaGetLastError());
  return refresh_bf16(m, nullptr);
}

// forward pass of B rows of m->xb -> m->yf [B][32] FP32 (pre-activations
// kept in m->z when `keep`)
void forward(me_mlp *m, int B, bool keep, cudaStream_t st) {
  const bf16 *in = m->xb.as<bf16>();
  for (int l = 0; l < kLayers; l++) {
    const bool last = l == kLayers - 1;
    gemm(ctx(m), in, m->wb[l].as<bf16>(), B, m->dout[l], m->din[l], m->b[l].as<float>(),
         (!last && keep) ? m->z[l].as<float>() : nullptr, last ? 0 : 1,
         last ? nullptr : m->a[l].as<bf16>(), last ? m->yf.as<float>() : nullptr, st);
    in = m->a[l].as<bf16>();
  }
}

// backward from dY (m->dyb, BF16 [B][32]), added into m->gw / m->gb
void backward(me_mlp *m, int B, cudaStream_t st) {
  const bf16 *dcur = m->dyb.as<bf16>();  // dZ of layer l, BF16 [B][dout]
  for (int l = kLayers - 1; l >= 0; l--) {
    const int dout = m->dout[l], din = m->din[l];
    // dW [dout][din] = dZ^T A_prev: GEMM of dZ^T [dout][B] and A_prev^T [din][B]
    bf16 *dzt = l == kLayers - 1 ? m->dybt.as<bf16>() : m->dzt.as<bf16>();
    transpose(dcur, B, dout, dzt, st);
    const bf16 *aprev = l == 0 ? m->xb.as<bf16>() : m->a[l - 1].as<bf16>();
    bf16 *aprevt = l == 0 ? m->xbt.as<bf16>() : m->at[l - 1].as<bf16>();
    transpose(aprev, B, din, aprevt, st);
    int split = 1;
    while (split < 16 && B % (2 * split * kTK) == 0 && B / (2 * split) >= 256) split *= 2;
    gemm(ctx(m), dzt, aprevt, dout, din, B, nullptr, nullptr, 0, nullptr, m->gw[l].as<float>(), st, split);
    const int chunk = 256;
    bias_grad_kernel<<<dim3((dout + 31) / 32, (B + chunk - 1) / chunk), dim3(32, 8), 0, st>>>(
        dcur, B, dout, chunk, m->gb[l].as<float>());
    if (l == 0) break;
    // dA_prev [B][din] = dZ W: GEMM of dZ [B][dout] and W^T [din][dout]
    gemm(ctx(m), dcur, m->wbt[l].as<bf16>(), B, din, dout, nullptr, nullptr, 0, nullptr,
         m->dh.as<float>(), st);
    gelu_back_kernel<<<nblk((long long)B * din), 256, 0, st>>>(
        m->dh.as<float>(), m->z[l - 1].as<float>(), (long long)B * din, m->dz.as<bf16>());
    dcur = m->dz.as<bf16>();
  }
}

void adam_step(me_mlp *m, float lr, cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  m->adam_t++;
  const float c1 = (float)(1.0 / (1.0 - pow((double)b1, (double)m->adam_t)));
  const float c2 = (float)(1.0 / (1.0 - pow((double)b2, (double)m->adam_t)));
  AdamNet net;
  net.w = m->w[0].as<float>();
  net.m = m->mw[0].as<float>();
  net.v = m->vw[0].as<float>();
  net.g = m->gw[0].as<float>();
  net.n = m->flat;
  for (int l = 0; l < kLayers; l++) {
    net.off[l] = m->w[l].as<float>() - net.w;
    net.rows[l] = m->dout[l];
    net.cols[l] = m->din[l];
    net.wb[l] = m->wb[l].as<bf16>();
    net.wbt[l] = m->wbt[l].as<bf16>();
  }
  adam_kernel<<<nblk(m->flat), 256, 0, st>>>(net, lr, b1, b2, eps, c1, c2);
}

// The gradients of B rows in two kernels, where the tcgen05 kernels are chosen
// and can run (ok): the arguments of both, set up once for all steps.
struct StepPlan {
  bool ok = false;
  StepMaps maps;
  StepNet net;
  GradMaps gmaps;
  GradNet gnet;
  unsigned tiles = 0, split = 1;
};

bool step_fused(const me_mlp *m) {
  return m->gemm_path == GemmPath::tcgen05 && device_facts().step_ok;
}

void plan_step(me_mlp *m, int B, StepPlan *p) {
  memset(&p->maps, 0, sizeof(p->maps));
  for (int l = 0; l < kLayers; l++) {
    const bf16 *in = l ? m->sat[l - 1].as<bf16>() : m->sxt.as<bf16>();
    if (!cached_tile_map(&m->maps, &p->maps.w[l], m->wb[l].as<bf16>(), m->dout[l], m->din[l],
                         l < kLayers - 1 ? 128 : kOutPad) ||
        (l > 0 && !cached_tile_map(&m->maps, &p->maps.t[l], m->wbt[l].as<bf16>(), m->din[l],
                                   m->dout[l], 128)) ||
        !cached_tile_map(&m->maps, &p->gmaps.a[l], m->sdzt[l].as<bf16>(), m->dout[l], B,
                         me::umma::kBM) ||
        !cached_tile_map(&m->maps, &p->gmaps.b[l], in, m->din[l], B, kGradN))
      return;
    p->net.bias[l] = m->b[l].as<float>();
    if (l < kLayers - 1) p->net.at[l] = m->sat[l].as<bf16>();
    p->net.dzt[l] = m->sdzt[l].as<bf16>();
    p->net.gb[l] = m->gb[l].as<float>();
    p->gnet.gw[l] = m->gw[l].as<float>();
    p->gnet.m[l] = m->dout[l];
    p->gnet.n[l] = m->din[l];
    p->gnet.tiles[l] = ((m->dout[l] + me::umma::kBM - 1) / me::umma::kBM) *
                       ((m->din[l] + kGradN - 1) / kGradN);
    p->tiles += (unsigned)p->gnet.tiles[l];
  }
  p->net.xt = m->sxt.as<bf16>();
  while (p->split < 16 && B / (2 * p->split) >= 256) p->split *= 2;
  while (B % (p->split * me::umma::kBK)) p->split /= 2;  // (B % 256 == 0: ends at 4 or before)
  p->ok = true;
}

void run_step(me_mlp *m, const StepPlan &p, int B, const bf16 *X, const float *T,
              const long long *idx, cudaStream_t st) {
  mlp_step_kernel<<<B / kStepRows, kStepThreads, kStepSmem, st>>>(
      p.maps, p.net, m->waits, X, idx, T, B, m->nip, m->loss.as<double>(), m->gerr.as<int>());
  mlp_wgrad_kernel<<<dim3(p.tiles, p.split), 128, me::umma::smem_bytes(kGradN), st>>>(
      p.gmaps, p.gnet, B, m->gerr.as<int>());
  m->gemm_launches[(int)GemmPath::tcgen05] += kLayers + 2 * kLayers - 1;
}

// loss and gradients of the rows idx[0..B) of the standardised targets T
// (the batch features already in m->xb); loss accumulated into m->loss
void loss_grad(me_mlp *m, int B, const float *T, const long long *idx, cudaStream_t st) {
  forward(m, B, true, st);
  mse_grad_kernel<<<nblk((long long)B * kOutPad), 256, 0, st>>>(
      m->yf.as<float>(), kOutPad, T, idx, B, m->dyb.as<bf16>(), m->loss.as<double>());
  backward(m, B, st);
}

void prior_from(const me_mlp_train_params *tp, Prior &pr) {
  pr.b_lo = (float)tp->b_range[0];
  pr.b_hi = (float)tp->b_range[1];
  pr.cost_lo = (float)tp->cos_theta_range[0];
  pr.cost_hi = (float)tp->cos_theta_range[1];
  pr.phi_lo = (float)tp->phi_range[0];
  pr.phi_hi = (float)tp->phi_range[1];
  pr.v_sigma = (float)tp->v_sigma;
  pr.w_lo = (float)tp->doppler_range[0];
  pr.w_hi = (float)tp->doppler_range[1];
  pr.a_lo = (float)tp->damping_range[0];
  pr.a_hi = (float)tp->damping_range[1];
  pr.eta_lo = (float)tp->eta_range[0];
  pr.eta_hi = (float)tp->eta_range[1];
  pr.s = (float)tp->s;
  pr.beta_lo = (float)tp->beta_range[0];
  pr.beta_hi = (float)tp->beta_range[1];
  pr.noise = (float)tp->noise;
  pr.mix = (float)tp->mix_weight;
  pr.mb_lo = (float)tp->mix_b_range[0];
  pr.mb_hi = (float)tp->mix_b_range[1];
  pr.meta_lo = (float)tp->mix_eta_range[0];
  pr.meta_hi = (float)tp->mix_eta_range[1];
}

// Few profiles of many features: the separate kernels, whose features kernel has a
// warp per profile and a CTA per eight, where mlp_predict_kernel's CTA of 128
// takes them piece by piece.  Both sides, us for a call alone, separately and in
// one kernel: 1 profile of 112 wavelengths 47.8, 49.6; 128: 45.2, 50.4; 192: 49.0,
// 54.5; 512: 63.4, 84.8; 64 of 128: 48.3, 51.4; 128 of 128: 53.5, 52.8, and of 160:
// 55.1, 55.0; 3,000 of 193: 62.8, 63.3, and of 512: 88.7, 95.1; 5,000 of 256: 75.5,
// 67.8, and of 512: 106.9, 97.3.  The values are the same.
bool predict_separately(const me_mlp *m, long long npix) {
  return m->nip > 384 && npix <= (m->nip > 768 ? 3072 : 64);
}

}  // namespace

namespace me {
// plan constants with device grid pointers, and the plan's device (me_api.cu)
int plan_devplan(const me_plan *p, DevPlan *out, int *device);

int mlp_gemm_status(me_mlp *m) { return gemm_status(m); }

long long mlp_predict_launches(const me_mlp *m, long long npix) {
  return m->gemm_path == GemmPath::tcgen05 && device_facts().pred_ok &&
                 !predict_separately(m, npix)
             ? 1
             : kMlpPredLaunches * ((npix + kMlpPredChunk - 1) / kMlpPredChunk);
}
}  // namespace me

extern "C" int me_mlp_train_params_default(me_mlp_train_params *tp) {
  if (!tp) return fail(ME_ERR_ARG, "null argument");
  memset(tp, 0, sizeof(*tp));
  tp->samples = 1LL << 22;
  tp->epochs = 16;
  tp->batch = 4096;
  tp->lr = 1e-3;
  tp->seed = 20240607ULL;
  tp->b_range[0] = 0;
  tp->b_range[1] = 3000;
  tp->cos_theta_range[0] = -1;
  tp->cos_theta_range[1] = 1;
  tp->phi_range[0] = 0;
  tp->phi_range[1] = me::kPi;
  tp->v_sigma = 1.5;
  tp->doppler_range[0] = 150;
  tp->doppler_range[1] = 350;
  tp->damping_range[0] = 0.1;
  tp->damping_range[1] = 0.8;
  tp->eta_range[0] = 2;
  tp->eta_range[1] = 30;
  tp->s = 1.0;
  tp->beta_range[0] = 0.1;
  tp->beta_range[1] = 0.6;
  tp->noise = 1e-3;
  return ME_OK;
}

extern "C" void me_mlp_destroy(me_mlp *m) {
  if (!m) return;
  int cur = 0;
  cudaGetDevice(&cur);
  cudaSetDevice(m->device);
  delete m;
  cudaSetDevice(cur);
}

extern "C" int me_mlp_train(me_plan *plan, const me_mlp_train_params *tp, me_mlp **out,
                            double *final_loss) {
  if (!plan || !tp || !out) return fail(ME_ERR_ARG, "null argument");
  *out = nullptr;
  if (tp->batch < 256 || tp->batch % 256 || tp->samples < tp->batch || tp->epochs < 0 ||
      tp->samples > (1LL << 31) || !(tp->lr > 0))
    return fail(ME_ERR_ARG,
                "batch a multiple of 256, batch <= samples <= 2^31, epochs >= 0, lr > 0");
  if (tp->gemm != ME_GEMM_TCGEN05 && tp->gemm != ME_GEMM_MMA_SYNC)
    return fail(ME_ERR_ARG, "gemm must be ME_GEMM_TCGEN05 or ME_GEMM_MMA_SYNC");
  if (!(tp->mix_weight >= 0.0 && tp->mix_weight <= 1.0))
    return fail(ME_ERR_ARG, "mix_weight must lie in [0, 1]");
  me::DevPlan P;
  int device = 0;
  int rc = me::plan_devplan(plan, &P, &device);
  if (rc) return rc;
  MCK(cudaSetDevice(device));
  me_mlp *m = new me_mlp();
  m->device = device;
  m->gemm_path = tp->gemm == ME_GEMM_TCGEN05 ? GemmPath::tcgen05 : GemmPath::mma_sync;
  rc = alloc_model(m, P.nl);
  if (!rc) rc = init_model(m, tp->seed);
  if (rc) {
    delete m;
    return rc;
  }
  std::unique_ptr<me_mlp, void (*)(me_mlp *)> guard(m, me_mlp_destroy);
  cudaStream_t st = nullptr;
  const long long n = tp->samples;
  const int nip = m->nip;
  // ---- training set: FP32 synthesis on the plan's grid, then standardisation ----
  DBuf Xf, set, X, T;
  const size_t tiles = (size_t)((n + kTile - 1) / kTile);
  Arena parts;
  if (step_fused(m))  // (the other path gives the FP32 features back before its buffers)
    parts.add(Xf, tiles * kTile * nip * 4);
  else
    MCK(Xf.ensure(tiles * kTile * nip * 4));
  parts.add(X, (size_t)n * nip * 2);
  parts.add(T, (size_t)n * kOut * 4);
  MCK(set.ensure(parts.total));
  parts.place(set.p);
  Prior pr;
  prior_from(tp, pr);
  // The targets lie in X until the features take their place (n >= 256, so 64 n
  // bytes and more hold the tiles), the sums in the gradients.
  float *const traw = X.as<float>();
  synth_train_kernel<<<(unsigned)tiles, kTile, 0, st>>>(P, pr, tp->seed, n, nip, Xf.as<float>(),
                                                        traw);
  MCK(cudaGetLastError());
  {
    const int shares = (int)(tiles < 64 ? tiles : 64);
    double *const sums = m->gw[0].as<double>(), *const part = sums + 2 * nip;
    std::vector<double> a(2 * nip);
    auto moments = [&](const float *x, int cols) {
      moments_kernel<<<dim3((cols + 7) / 8, shares), 256, 0, st>>>(x, n, cols, part);
      moments_sum_kernel<<<nblk(2 * cols), 256, 0, st>>>(part, shares, cols, sums);
      return cudaMemcpy(a.data(), sums, 2 * cols * 8, cudaMemcpyDeviceToHost);
    };
    MCK(moments(Xf.as<float>(), nip));
    for (int c = 0; c < nip; c++) {
      const double mu = a[2 * c] / n, var = a[2 * c + 1] / n - mu * mu;
      m->h_fmean[c] = c < m->nin ? (float)mu : 0.f;
      m->h_fistd[c] = (c < m->nin && var > 1e-20) ? (float)(1.0 / sqrt(var)) : 0.f;
    }
    MCK(moments(traw, kOut));
    std::vector<float> tinv(kOut);
    for (int c = 0; c < kOut; c++) {
      const double mu = a[2 * c] / n, var = a[2 * c + 1] / n - mu * mu;
      m->h_tmean[c] = (float)mu;
      m->h_tstd[c] = var > 1e-20 ? (float)sqrt(var) : 1.f;
      tinv[c] = 1.f / m->h_tstd[c];
    }
    rc = upload_standardisation(m);
    if (rc) return rc;
    MCK(cudaMemcpy(m->tistd.p, tinv.data(), kOut * 4, cudaMemcpyHostToDevice));
    standardise_targets_kernel<<<nblk(n), 256, 0, st>>>(traw, n, m->tmean.as<float>(),
                                                        m->tistd.as<float>(), T.as<float>());
    standardise_kernel<<<dim3((unsigned)tiles, nip / 32), 256, 0, st>>>(
        Xf.as<float>(), n, nip, m->fmean.as<float>(), m->fistd.as<float>(), X.as<bf16>());
    MCK(cudaMemsetAsync(m->gw[0].p, 0, (size_t)m->flat * 4, st));
    MCK(cudaGetLastError());
  }
  // ---- Adam on shuffled batches ----
  // What follows lies where the FP32 features were, if it fits there; they are
  // not needed any more.
  const int B = tp->batch;
  DBuf perm;
  const size_t permb = ((size_t)n * sizeof(long long) + 255) / 256 * 256;  // <= Xf (nip >= 32)
  StepPlan sp;
  if (step_fused(m)) {
    perm.view(Xf.p, permb);
    rc = ensure_step(m, B, Xf.as<char>() + permb, Xf.n - permb);
    if (rc) return rc;
    plan_step(m, B, &sp);
  }
  if (!sp.ok) {
    MCK(cudaStreamSynchronize(st));
    Xf.release();
    rc = ensure_batch(m, B);
    if (rc) return rc;
    perm.view(nullptr, 0);
    MCK(perm.ensure((size_t)n * sizeof(long long)));
  }
  int bits = 1;
  while ((1LL << bits) < n) bits++;
  const long long steps = n / B;
  double last = 0.0;
  for (int ep = 0; ep < tp->epochs; ep++) {
    const unsigned long long k = tp->seed * 0x9E3779B97F4A7C15ull + 0x51ull * (ep + 1);
    permute_kernel<<<nblk(n), 256, 0, st>>>(n, bits, (uint32_t)k, (uint32_t)(k >> 32),
                                            perm.as<long long>());
    MCK(cudaMemsetAsync(m->loss.p, 0, sizeof(double), st));
    for (long long s = 0; s < steps; s++) {
      const long long *idx = perm.as<long long>() + s * B;
      if (sp.ok) {
        run_step(m, sp, B, X.as<bf16>(), T.as<float>(), idx, st);
      } else {
        gather_kernel<<<nblk((long long)B * nip), 256, 0, st>>>(X.as<bf16>(), idx, B, nip,
                                                                m->xb.as<bf16>());
        loss_grad(m, B, T.as<float>(), idx, st);
      }
      adam_step(m, (float)tp->lr, st);
    }
    MCK(cudaGetLastError());
    double l = 0;
    MCK(cudaMemcpyAsync(&l, m->loss.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    MCK(cudaStreamSynchronize(st));
    rc = gemm_status(m);
    if (rc) return rc;
    last = l / (double)steps;
  }
  // (what lay in the training set's memory goes with it)
  if (m->step_cap == 0) {
    m->sxt.release();
    for (DBuf &d : m->sat) d.release();
    for (DBuf &d : m->sdzt) d.release();
  }
  if (final_loss) *final_loss = last;
  *out = guard.release();
  return ME_OK;
}

// The inference in one kernel, where the tcgen05 kernels are chosen and can run;
// false: nothing was launched.
static bool predict_fused(me_mlp *m, const double *d_prof, long npix, double *d_par,
                          cudaStream_t st) {
  const DeviceFacts &dv = device_facts();
  if (m->gemm_path != GemmPath::tcgen05 || !m->gerr.p || !dv.pred_ok || dv.sms <= 0) return false;
  CUtensorMap w[kLayers];
  for (int l = 0; l < kLayers; l++)
    if (!cached_tile_map(&m->maps, &w[l], m->wb[l].as<bf16>(), m->dout[l], m->din[l],
                         l < kLayers - 1 ? 128 : kOutPad))
      return false;
  PredNet net;
  for (int l = 0; l < kLayers; l++) net.bias[l] = m->b[l].as<float>();
  net.fmean = m->fmean.as<float>();
  net.fistd = m->fistd.as<float>();
  net.tmean = m->tmean.as<float>();
  net.tstd = m->tstd.as<float>();
  const long long tiles = ((long long)npix + me::umma::kBM - 1) / me::umma::kBM;
  const unsigned grid = (unsigned)(tiles < dv.sms ? tiles : dv.sms);
  auto go = [&](auto kernel) {
    kernel<<<grid, kPredThreads, kPredSmem, st>>>(w[0], w[1], w[2], w[3], net, m->waits, d_prof,
                                                  npix, m->nl, m->nip, d_par, m->gerr.as<int>());
  };
  if ((reinterpret_cast<uintptr_t>(d_prof) & 15) == 0)
    go(mlp_predict_kernel<true>);
  else
    go(mlp_predict_kernel<false>);
  m->gemm_launches[(int)GemmPath::tcgen05] += kLayers;
  return true;
}

extern "C" int me_mlp_predict_device(me_mlp *m, const double *d_prof, long npix, double *d_par,
                                     void *stream) {
  if (!m || (npix > 0 && (!d_prof || !d_par)) || npix < 0)
    return fail(ME_ERR_ARG, "null argument");
  if (npix == 0) return ME_OK;
  MCK(cudaSetDevice(m->device));
  cudaStream_t st = (cudaStream_t)stream;
  // (the separate kernels share the initialiser's buffers, which a first call
  // allocates: not under capture, and in order from stream to stream)
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  const bool apart = predict_separately(m, npix) &&
                     cudaStreamIsCapturing(st, &capture) == cudaSuccess &&
                     capture == cudaStreamCaptureStatusNone;
  if (!apart && predict_fused(m, d_prof, npix, d_par, st)) {
    MCK(cudaGetLastError());
    if (!stream) {
      MCK(cudaStreamSynchronize(st));
      return gemm_status(m);
    }
    return ME_OK;
  }
  const int chunk = (int)(npix < me::kMlpPredChunk ? (npix + 255) / 256 * 256 : me::kMlpPredChunk);
  int rc = ensure_batch(m, chunk);
  if (rc) return rc;
  if (apart) {
    if (!m->batch_used) MCK(cudaEventCreateWithFlags(&m->batch_used, cudaEventDisableTiming));
    MCK(cudaStreamWaitEvent(st, m->batch_used, 0));
  }
  for (long long r0 = 0; r0 < npix; r0 += chunk) {
    const int rows = (int)((npix - r0) < chunk ? (npix - r0) : chunk);
    // a chunk starts 32 nl r0 bytes in, so its alignment is the base's
    if ((reinterpret_cast<uintptr_t>(d_prof) & 15) == 0)
      map_features_kernel<true><<<nblk(rows, 8), 256, 0, st>>>(
          d_prof + (size_t)r0 * 4 * m->nl, rows, m->nl, m->nip, m->fmean.as<float>(),
          m->fistd.as<float>(), m->xb.as<bf16>(), m->imax.as<float>());
    else
      map_features_kernel<false><<<nblk(rows, 8), 256, 0, st>>>(
          d_prof + (size_t)r0 * 4 * m->nl, rows, m->nl, m->nip, m->fmean.as<float>(),
          m->fistd.as<float>(), m->xb.as<bf16>(), m->imax.as<float>());
    forward(m, rows, false, st);
    decode_kernel<<<nblk(rows, 128), 128, 0, st>>>(m->yf.as<float>(), rows, kOutPad,
                                                   m->tmean.as<float>(), m->tstd.as<float>(),
                                                   m->imax.as<float>(), d_par + (size_t)r0 * 9);
  }
  MCK(cudaGetLastError());
  if (apart) MCK(cudaEventRecord(m->batch_used, st));
  if (!stream) {
    MCK(cudaStreamSynchronize(st));
    return gemm_status(m);
  }
  return ME_OK;
}

extern "C" int me_mlp_predict(me_mlp *m, const double *prof, long npix, double *par) {
  if (!m || (npix > 0 && (!prof || !par)) || npix < 0) return fail(ME_ERR_ARG, "null argument");
  if (npix == 0) return ME_OK;
  MCK(cudaSetDevice(m->device));
  DBuf dp, dq;
  MCK(dp.ensure((size_t)npix * 4 * m->nl * 8));
  MCK(dq.ensure((size_t)npix * 9 * 8));
  MCK(cudaMemcpy(dp.p, prof, (size_t)npix * 4 * m->nl * 8, cudaMemcpyHostToDevice));
  int rc = me_mlp_predict_device(m, dp.as<double>(), npix, dq.as<double>(), nullptr);
  if (rc) return rc;
  MCK(cudaMemcpy(par, dq.p, (size_t)npix * 9 * 8, cudaMemcpyDeviceToHost));
  return ME_OK;
}

extern "C" int me_mlp_shape(const me_mlp *m, int *nl, int *nin_pad, long long *nparams) {
  if (!m) return fail(ME_ERR_ARG, "null argument");
  if (nl) *nl = m->nl;
  if (nin_pad) *nin_pad = m->nip;
  if (nparams) *nparams = param_count(m);
  return ME_OK;
}

namespace {
// copies the parameters (or gradients) between a flat host array and the
// device, where they lie in the same order without gaps (alloc_model: every
// layer's sizes but the last bias's are multiples of 64 floats)
int copy_flat(const me_mlp *m, bool grads, float *host, bool to_host) {
  void *dev = grads ? m->gw[0].p : m->w[0].p;
  const size_t bytes = (size_t)param_count(m) * 4;
  if (to_host)
    MCK(cudaMemcpy(host, dev, bytes, cudaMemcpyDeviceToHost));
  else
    MCK(cudaMemcpy(dev, host, bytes, cudaMemcpyHostToDevice));
  return ME_OK;
}
}  // namespace

extern "C" int me_mlp_get_params(const me_mlp *m, float *params) {
  if (!m || !params) return fail(ME_ERR_ARG, "null argument");
  MCK(cudaSetDevice(m->device));
  return copy_flat(m, false, params, true);
}

extern "C" int me_mlp_set_params(me_mlp *m, const float *params) {
  if (!m || !params) return fail(ME_ERR_ARG, "null argument");
  MCK(cudaSetDevice(m->device));
  int rc = copy_flat(m, false, const_cast<float *>(params), false);
  if (rc) return rc;
  rc = refresh_bf16(m, nullptr);
  if (rc) return rc;
  MCK(cudaDeviceSynchronize());
  return ME_OK;
}

extern "C" int me_mlp_loss_grad(me_mlp *m, const float *x, const float *t, int rows, double *loss,
                                float *grad) {
  if (!m || !x || !t || !loss || !grad) return fail(ME_ERR_ARG, "null argument");
  if (rows < 256 || rows % 256) return fail(ME_ERR_ARG, "rows must be a positive multiple of 256");
  MCK(cudaSetDevice(m->device));
  int rc = ensure_batch(m, rows);
  if (rc) return rc;
  if (m->batch_used) MCK(cudaStreamWaitEvent(nullptr, m->batch_used, 0));
  DBuf xf, tf, idx;
  MCK(xf.ensure((size_t)rows * m->nip * 4));
  MCK(tf.ensure((size_t)rows * kOut * 4));
  MCK(idx.ensure((size_t)rows * 8));
  MCK(cudaMemcpy(xf.p, x, (size_t)rows * m->nip * 4, cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(tf.p, t, (size_t)rows * kOut * 4, cudaMemcpyHostToDevice));
  f32_to_bf16_kernel<<<nblk((long long)rows * m->nip), 256>>>(xf.as<float>(),
                                                               (long long)rows * m->nip,
                                                               m->xb.as<bf16>());
  iota_kernel<<<nblk(rows), 256>>>(idx.as<long long>(), rows);
  MCK(cudaMemset(m->loss.p, 0, sizeof(double)));
  MCK(cudaMemset(m->gw[0].p, 0, (size_t)m->flat * 4));
  StepPlan sp;
  if (step_fused(m)) {
    rc = ensure_step(m, rows, nullptr, 0);
    if (rc) return rc;
    plan_step(m, rows, &sp);
  }
  if (sp.ok)
    run_step(m, sp, rows, m->xb.as<bf16>(), tf.as<float>(), idx.as<long long>(), nullptr);
  else
    loss_grad(m, rows, tf.as<float>(), idx.as<long long>(), nullptr);
  MCK(cudaGetLastError());
  MCK(cudaDeviceSynchronize());
  rc = gemm_status(m);
  if (rc) return rc;
  MCK(cudaMemcpy(loss, m->loss.p, sizeof(double), cudaMemcpyDeviceToHost));
  return copy_flat(m, true, grad, true);
}

extern "C" int me_mlp_set_gemm(me_mlp *m, int path) {
  if (!m) return fail(ME_ERR_ARG, "null argument");
  if (path != ME_GEMM_TCGEN05 && path != ME_GEMM_MMA_SYNC)
    return fail(ME_ERR_ARG, "path must be ME_GEMM_TCGEN05 or ME_GEMM_MMA_SYNC");
  m->gemm_path = path == ME_GEMM_TCGEN05 ? GemmPath::tcgen05 : GemmPath::mma_sync;
  return ME_OK;
}

extern "C" int me_mlp_set_waits(me_mlp *m, unsigned tries, int drop) {
  if (!m) return fail(ME_ERR_ARG, "null argument");
  if (drop < 0 || drop > 3) return fail(ME_ERR_ARG, "drop must be 0 to 3");
  m->waits = WaitRules();
  if (tries) m->waits.tries = tries;
  m->waits.drop = drop;
  return ME_OK;
}

extern "C" int me_mlp_gemm_launches(const me_mlp *m, long long *tcgen05, long long *mma_sync) {
  if (!m) return fail(ME_ERR_ARG, "null argument");
  if (tcgen05) *tcgen05 = m->gemm_launches[(int)GemmPath::tcgen05];
  if (mma_sync) *mma_sync = m->gemm_launches[(int)GemmPath::mma_sync];
  return ME_OK;
}

extern "C" int me_gemm_bf16(int device, int path, const uint16_t *a, const uint16_t *bt, int m,
                            int n, int r, int split, const float *bias, int gelu, float *z,
                            float *y, int *ran) {
  if (!a || !bt || !y) return fail(ME_ERR_ARG, "null argument");
  if (path != ME_GEMM_TCGEN05 && path != ME_GEMM_MMA_SYNC)
    return fail(ME_ERR_ARG, "path must be ME_GEMM_TCGEN05 or ME_GEMM_MMA_SYNC");
  if (m < 1 || n < 1 || r < 32 || split < 1 || r % (32 * split))
    return fail(ME_ERR_ARG, "need m, n >= 1, r >= 32 and r % (32 split) == 0");
  if (split > 1 && (bias || gelu || z))
    return fail(ME_ERR_ARG, "a split reduction has no bias, GELU or z");
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0)
    return fail(ME_ERR_NODEVICE, "no CUDA device");
  if (device < 0 || device >= nd) return fail(ME_ERR_ARG, "device out of range");
  MCK(cudaSetDevice(device));
  DBuf da, db, dbias, dz, dy, derr;
  const size_t mr = (size_t)m * r, nr = (size_t)n * r, mn = (size_t)m * n;
  MCK(da.ensure(mr * 2));
  MCK(db.ensure(nr * 2));
  MCK(dy.ensure(mn * 4));
  MCK(derr.ensure(sizeof(int)));
  MCK(cudaMemcpy(da.p, a, mr * 2, cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(db.p, bt, nr * 2, cudaMemcpyHostToDevice));
  MCK(cudaMemset(dy.p, 0, mn * 4));
  MCK(cudaMemset(derr.p, 0, sizeof(int)));
  if (bias) {
    MCK(dbias.ensure((size_t)n * 4));
    MCK(cudaMemcpy(dbias.p, bias, (size_t)n * 4, cudaMemcpyHostToDevice));
  }
  if (z) MCK(dz.ensure(mn * 4));
  GemmCtx g;
  g.path = path == ME_GEMM_TCGEN05 ? GemmPath::tcgen05 : GemmPath::mma_sync;
  g.err = derr.as<int>();
  const GemmPath used = gemm(g, da.as<bf16>(), db.as<bf16>(), m, n, r, dbias.as<float>(),
                             dz.as<float>(), gelu, nullptr, dy.as<float>(), nullptr, split);
  if (ran) *ran = used == GemmPath::tcgen05 ? ME_GEMM_TCGEN05 : ME_GEMM_MMA_SYNC;
  MCK(cudaGetLastError());
  MCK(cudaDeviceSynchronize());
  int e = 0;
  MCK(cudaMemcpy(&e, derr.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) return fail(ME_ERR_CUDA, "tensor-core GEMM: a bounded wait timed out");
  MCK(cudaMemcpy(y, dy.p, mn * 4, cudaMemcpyDeviceToHost));
  if (z) MCK(cudaMemcpy(z, dz.p, mn * 4, cudaMemcpyDeviceToHost));
  return ME_OK;
}

// File: "MEMLP001", int32 nl, int32 nin_pad, float fmean[nin_pad],
// fistd[nin_pad], tmean[10], tstd[10], then the parameters as
// me_mlp_get_params lays them out (little-endian).
static const char kMagic[8] = {'M', 'E', 'M', 'L', 'P', '0', '0', '1'};

extern "C" int me_mlp_save(const me_mlp *m, const char *path) {
  if (!m || !path) return fail(ME_ERR_ARG, "null argument");
  MCK(cudaSetDevice(m->device));
  std::vector<float> prm((size_t)param_count(m));
  int rc = copy_flat(m, false, prm.data(), true);
  if (rc) return rc;
  FILE *f = fopen(path, "wb");
  if (!f) return fail(ME_ERR_IO, std::string("cannot write ") + path);
  const int32_t hdr[2] = {m->nl, m->nip};
  bool ok = fwrite(kMagic, 1, 8, f) == 8 && fwrite(hdr, 4, 2, f) == 2 &&
            fwrite(m->h_fmean.data(), 4, m->nip, f) == (size_t)m->nip &&
            fwrite(m->h_fistd.data(), 4, m->nip, f) == (size_t)m->nip &&
            fwrite(m->h_tmean.data(), 4, kOut, f) == (size_t)kOut &&
            fwrite(m->h_tstd.data(), 4, kOut, f) == (size_t)kOut &&
            fwrite(prm.data(), 4, prm.size(), f) == prm.size();
  ok = (fclose(f) == 0) && ok;
  if (!ok) return fail(ME_ERR_IO, std::string("short write to ") + path);
  return ME_OK;
}

extern "C" int me_mlp_load(const char *path, int device, me_mlp **out) {
  if (!path || !out) return fail(ME_ERR_ARG, "null argument");
  *out = nullptr;
  FILE *f = fopen(path, "rb");
  if (!f) return fail(ME_ERR_IO, std::string("cannot read ") + path);
  char magic[8];
  int32_t hdr[2];
  bool ok = fread(magic, 1, 8, f) == 8 && memcmp(magic, kMagic, 8) == 0 &&
            fread(hdr, 4, 2, f) == 2 && hdr[0] > 0 && hdr[0] <= ME_MAX_NL &&
            hdr[1] == (4 * hdr[0] + 31) / 32 * 32;
  if (!ok) {
    fclose(f);
    return fail(ME_ERR_FORMAT, std::string("not an initialiser file: ") + path);
  }
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd == 0) {
    fclose(f);
    return fail(ME_ERR_NODEVICE, "no CUDA device");
  }
  if (device < 0 || device >= nd) {
    fclose(f);
    return fail(ME_ERR_ARG, "device out of range");
  }
  cudaSetDevice(device);
  me_mlp *m = new me_mlp();
  m->device = device;
  std::unique_ptr<me_mlp, void (*)(me_mlp *)> guard(m, me_mlp_destroy);
  int rc = alloc_model(m, hdr[0]);
  if (rc) {
    fclose(f);
    return rc;
  }
  std::vector<float> prm((size_t)param_count(m));
  ok = fread(m->h_fmean.data(), 4, m->nip, f) == (size_t)m->nip &&
       fread(m->h_fistd.data(), 4, m->nip, f) == (size_t)m->nip &&
       fread(m->h_tmean.data(), 4, kOut, f) == (size_t)kOut &&
       fread(m->h_tstd.data(), 4, kOut, f) == (size_t)kOut &&
       fread(prm.data(), 4, prm.size(), f) == prm.size();
  fclose(f);
  if (!ok) return fail(ME_ERR_FORMAT, std::string("truncated initialiser file: ") + path);
  rc = upload_standardisation(m);
  if (!rc) rc = me_mlp_set_params(m, prm.data());
  if (rc) return rc;
  *out = guard.release();
  return ME_OK;
}
