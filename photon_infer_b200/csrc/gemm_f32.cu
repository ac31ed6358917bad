// True 32-bit matrix product for the float32 path: C[M,N] = A[M,K] * W[N,K]^T with
// plain FMA on the CUDA cores, no tensor-core mode of reduced precision.  Same
// contract as the reference's naive product (include/photon/ops/kernels/
// matmul_kernel.hpp:104-129: W is [out, in] row-major, no bias).
//
// Every output element is one chain of K fused multiply-adds in ascending k, so a
// row's result does not depend on M, on the kernel or tile it fell into or on the other rows:
// the float32 path gives identical bits for every way of cutting a request into steps.  So K is never
// split, and the kernels below differ only in how they bring the operands to the multiply-adds.
// Weights of 2^22 numbers, 1,024 rows and 2,048 columns and more do not come here but to gemm_f32_tc.cu (ops.sgemm_tc_supported).
#include "common.cuh"

__device__ __forceinline__ void sg_cp16(float* dst, const float* src, bool in) {      // nothing is read where `in` does not
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"                         // hold: the bytes become zero
               ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void sg_cp4(float* dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
               ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// ---------------------------------------------------------------- many rows: tiles of BM x BN
// A warp owns TM rows x all BN columns of the tile, lane l the columns l, l + 32 ..: a row's operand is one shared-memory
// broadcast for the whole warp, four values of k at a time, and the lanes' quads of W (rows 20 floats apart) do not conflict.
// Slabs of 16 k of both operands come by cp.async, as they lie, into a ring of SG_STAGES, so that three slabs are on
// their way while one is multiplied: with the next slab alone in flight a tile of 64 x 64 took half as long again.
// What bounds it: an outer product of registers issues 101 multiply-adds a cycle and SM (measured with nothing else in
// the loop; 83 with packed pairs, whose three 64-bit operands take three cycles to read), of which 2048 x 16384 x 2048
// reaches 79 % (46 TFLOP/s); 513 x 16384 x 2048 takes 868 us.
#define SG_BK 16
#define SG_LD (SG_BK + 4)
#define SG_STAGES 4

template <int BM, int BN, int TM, bool VEC>
__global__ void __launch_bounds__(BM / TM * 32)
sgemm_tile_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, long ldw,
                  float* __restrict__ C, long ldc, int M, int N, int K) {
  constexpr int TN = BN / 32, THREADS = BM / TM * 32;
  constexpr int STAGE = (BM + BN) * SG_LD;           // A's rows, then W's
  extern __shared__ __align__(16) float sg[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int slabs = (K + SG_BK - 1) / SG_BK;
  auto fetch = [&](int slab) {
    if (slab < slabs) {
      float* d = sg + (slab % SG_STAGES) * STAGE;
      const int k0 = slab * SG_BK;
      constexpr int PER = VEC ? SG_BK / 4 : SG_BK, W4 = VEC ? 4 : 1;   // copies per row, floats per copy
#pragma unroll
      for (int i = 0; i < (BM + BN) * PER / THREADS; ++i) {
        const int at = tid + i * THREADS;
        const int r = at / PER, k = k0 + at % PER * W4;
        const bool isa = r < BM;
        const bool in = k < K && (isa ? m0 + r < M : n0 + r - BM < N);
        const float* src = !in ? W : isa ? A + (size_t)(m0 + r) * lda + k : W + (size_t)(n0 + r - BM) * ldw + k;
        float* dst = d + r * SG_LD + at % PER * W4;
        if (VEC) sg_cp16(dst, src, in); else sg_cp4(dst, src, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  static_assert((BM + BN) * (SG_BK / 4) % THREADS == 0, "whole passes of copies");
#pragma unroll
  for (int s = 0; s < SG_STAGES - 1; ++s) fetch(s);
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int slab = 0; slab < slabs; ++slab) {
    asm volatile("cp.async.wait_group %0;" ::"n"(SG_STAGES - 2) : "memory");
    __syncthreads();                                 // this slab is there, and the stage before it is read no more
    fetch(slab + SG_STAGES - 1);
    const float* ar = sg + (slab % SG_STAGES) * STAGE + warp * TM * SG_LD;
    const float* wr = sg + (slab % SG_STAGES) * STAGE + (BM + lane) * SG_LD;
#pragma unroll
    for (int q = 0; q < SG_BK; q += 4) {
      float4 a[TM], w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(wr + j * 32 * SG_LD + q);
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(ar + i * SG_LD + q);
      // one value of k after the other: TM x TN chains stand between two links of one
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + warp * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + lane + j * 32;
      if (gn < N) C[(size_t)gm * ldc + gn] = acc[i][j];
    }
  }
}

// ---------------------------------------------------------------- few rows: W streams through once
// A block owns 16 rows of W and all rows of A (up to 8 MR): thread (m, n) carries the chains of rows m, m + 8 .. of A for
// its row of W.  Slabs of 128 k of both come by cp.async into a ring of SR_STAGES; the operands of the next SR_Q quads of k
// are read while the present ones are multiplied, so that the chain (a multiply-add every four cycles) waits for nothing
// but itself.  What bounds it: W's bytes where W is large (it is read once), else the chain.
#define SR_ROWS 16
#define SR_BK 128
#define SR_LD (SR_BK + 4)                            // rows start four banks apart: 16-byte reads of 8 rows do not conflict
#define SR_STAGES 4

template <int MR>
__global__ void __launch_bounds__(128)
sgemm_rows_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, long ldw,
                  float* __restrict__ C, long ldc, int M, int N, int K) {
  extern __shared__ __align__(16) float sr[];
  constexpr int STAGE = (SR_ROWS + 8 * MR) * SR_LD;  // W's rows, then A's
  constexpr int SR_Q = MR == 1 ? 4 : MR <= 4 ? 2 : 1;
  const int tid = threadIdx.x;
  const int n = tid & 15, m = tid >> 4;
  const int n0 = blockIdx.x * SR_ROWS;
  const int slabs = (K + SR_BK - 1) / SR_BK;
  auto fetch = [&](int slab) {
    if (slab < slabs) {
      float* d = sr + (slab % SR_STAGES) * STAGE;
      const int k0 = slab * SR_BK;
#pragma unroll
      for (int i = 0; i < (SR_ROWS + 8 * MR) * (SR_BK / 4) / 128; ++i) {
        const int at = tid + i * 128;
        const int r = at / (SR_BK / 4), q = (at % (SR_BK / 4)) * 4;
        const bool isw = r < SR_ROWS;
        const bool in = k0 + q < K && (isw ? n0 + r < N : r - SR_ROWS < M);
        const float* src = !in ? W : isw ? W + (size_t)(n0 + r) * ldw + k0 + q : A + (size_t)(r - SR_ROWS) * lda + k0 + q;
        sg_cp16(d + r * SR_LD + q, src, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < SR_STAGES - 1; ++s) fetch(s);
  float acc[MR];
#pragma unroll
  for (int i = 0; i < MR; ++i) acc[i] = 0.f;
  for (int slab = 0; slab < slabs; ++slab) {
    asm volatile("cp.async.wait_group %0;" ::"n"(SR_STAGES - 2) : "memory");
    __syncthreads();                                 // this slab is there, and the stage before it is read no more
    fetch(slab + SR_STAGES - 1);
    const float* wr = sr + (slab % SR_STAGES) * STAGE + n * SR_LD;
    const float* ar = sr + (slab % SR_STAGES) * STAGE + (SR_ROWS + m) * SR_LD;
    if (m >= M) continue;
    float4 w[2][SR_Q], a[2][SR_Q][MR];
    auto read = [&](int buf, int q0) {
#pragma unroll
      for (int q = 0; q < SR_Q; ++q) {
        w[buf][q] = *reinterpret_cast<const float4*>(wr + 4 * (q0 + q));
#pragma unroll
        for (int i = 0; i < MR; ++i) a[buf][q][i] = *reinterpret_cast<const float4*>(ar + i * 8 * SR_LD + 4 * (q0 + q));
      }
    };
    auto multiply = [&](int buf, int quads) {
#pragma unroll
      for (int q = 0; q < SR_Q; ++q) {
        if (q >= quads) break;
#pragma unroll
        for (int i = 0; i < MR; ++i) acc[i] = fmaf(a[buf][q][i].x, w[buf][q].x, acc[i]);
#pragma unroll
        for (int i = 0; i < MR; ++i) acc[i] = fmaf(a[buf][q][i].y, w[buf][q].y, acc[i]);
#pragma unroll
        for (int i = 0; i < MR; ++i) acc[i] = fmaf(a[buf][q][i].z, w[buf][q].z, acc[i]);
#pragma unroll
        for (int i = 0; i < MR; ++i) acc[i] = fmaf(a[buf][q][i].w, w[buf][q].w, acc[i]);
      }
    };
    const int left = (K - slab * SR_BK) / 4;         // quads of k from here on
    if (left >= SR_BK / 4) {
      read(0, 0);
#pragma unroll
      for (int g = 0; g < SR_BK / 4 / SR_Q; ++g) {
        if (g + 1 < SR_BK / 4 / SR_Q) read((g + 1) & 1, (g + 1) * SR_Q);
        multiply(g & 1, SR_Q);
      }
    } else {
      for (int q = 0; q < left; q += SR_Q) { read(0, q); multiply(0, left - q); }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < MR; ++i)
    if (m + 8 * i < M && n0 + n < N) C[(size_t)(m + 8 * i) * ldc + n0 + n] = acc[i];
}

template <int MR>
static int sgemm_rows_go(const float* A, long lda, const float* W, long ldw, float* C, long ldc, int M, int N, int K,
                         cudaStream_t stream) {
  const size_t smem = (size_t)SR_STAGES * (SR_ROWS + 8 * MR) * SR_LD * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(sgemm_rows_kernel<MR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  sgemm_rows_kernel<MR><<<(N + SR_ROWS - 1) / SR_ROWS, 128, smem, stream>>>(A, lda, W, ldw, C, ldc, M, N, K);
  return launch_status();
}

template <int BM, int BN, int TM, bool VEC>
static int sgemm_tile_go(const float* A, long lda, const float* W, long ldw, float* C, long ldc, int M, int N, int K,
                         cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return PHOTON_ERR_UNSUPPORTED;
  const size_t smem = (size_t)SG_STAGES * (BM + BN) * SG_LD * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(sgemm_tile_kernel<BM, BN, TM, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  sgemm_tile_kernel<BM, BN, TM, VEC><<<grid, BM / TM * 32, smem, stream>>>(A, lda, W, ldw, C, ldc, M, N, K);
  return launch_status();
}

PHOTON_API int photon_sgemm_nt(const float* A, long lda, const float* W, long ldw, float* C, long ldc,
                               int M, int N, int K, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return PHOTON_ERR_ARGUMENT;
  // 16-byte copies of both operands
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
  // Few rows: while the tiles' one round leaves most SMs idle.  A round of tiles takes 80 to 92 us per 2,048 of K whatever
  // N; the rows kernel grows with N (8 rows: 15 us at N = 2,048, 64 at 16,384; 16 rows: 19 and 104; 32 rows: 27 and 142).
  if (vec && M <= 64 && N <= (M <= 8 ? 1 << 20 : M <= 16 ? 12288 : M <= 32 ? 8192 : 4096)) {
    if (M <= 8) return sgemm_rows_go<1>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    if (M <= 16) return sgemm_rows_go<2>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    if (M <= 32) return sgemm_rows_go<4>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    return sgemm_rows_go<8>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  }
#define SG_GO(BM, BN, TM) (vec ? sgemm_tile_go<BM, BN, TM, true>(A, lda, W, ldw, C, ldc, M, N, K, stream) \
                               : sgemm_tile_go<BM, BN, TM, false>(A, lda, W, ldw, C, ldc, M, N, K, stream))
  // The tile, by its time per 2,048 of K as measured: `each` us for a tile on an SM that is full of them, `alone` more for
  // the first (64 x 128: 46 TFLOP/s with many tiles, 32 x 128: 43, 64 x 64: 39, but the smaller ones leave less of the last
  // round empty: 513 x 3072 takes 249, 187 and 202 us, 513 x 2048 x 8192 takes 543, 568 and 552, 128 x 3072 takes 138, 93 and 83).
  const long sms = photon_sm_count();
  auto cost = [&](long bm, long bn, double each, double alone) {
    const long tiles = ((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    return (double)((tiles + sms - 1) / sms) * each + alone;
  };
  const double c0 = cost(64, 128, 108.0, 30.0), c1 = cost(32, 128, 58.0, 35.0), c2 = cost(64, 64, 64.0, 19.0);
  if (c0 <= c1 && c0 <= c2) return SG_GO(64, 128, 16);
  if (c1 <= c2) return SG_GO(32, 128, 8);
  return SG_GO(64, 64, 8);
}
