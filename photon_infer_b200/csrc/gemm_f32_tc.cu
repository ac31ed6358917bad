// 32-bit matrix product of large weights on the fifth-generation tensor cores: C[M, N] = A[M, K] * W[N, K]^T, float in and out.
//
// A 32-bit number is the sum of three bfloat16 numbers, each what the ones before left (W's by cutting bits off, 8 + 8 + 8, the
// tokens' by rounding; exact down to 2^-110, where the third one's last bits leave bfloat16's range).  Of the nine products of such
// parts the six largest are formed.  Of a term w a with w and a in [1, 2), w's second and third parts are below 2^-7 and 2^-15, the tokens'
// 2^-8 and 2^-17 at most: the three products left out are below 2^-23 + 2^-24 + 2^-32 of it (2^-22.4), of either sign.  Six bfloat16
// products a term are still six times what the FP32 pipe does (1.6 PFLOP/s / 6 against 31 to 46 TFLOP/s of gemm_f32.cu's
// tiles).  Measured, 513 rows, against those: 3072 x 2048 46 us (190), 2048 x 2048 42 (141), 16384 x 2048 212 (870), 2048 x 8192
// 135 (545); one row, captured, weights from memory, 13, 10, 30 and 19 (12, 10, 31 and 34).  Error against 64 bits (rms, K = 2048): 1.1e-7, the chain's 8.1e-7.
// What bounds it: at 513 rows the products (1.1 PFLOP/s of bfloat16 with ragged tiles and a last round), with 69 KB a chunk
// and SM from L2 close behind; up to 64 rows W's bytes.
//
// The order of every sum depends on K alone, so a row of C has the same bits for every M, tile and split (the float32 path
// promises that for every way of cutting a request into steps):
//   * 64 of K are a chunk: in tensor memory, the five small products first, then the large one, whose additions the tensor
//     cores truncate: four of them, and the chunk is at most an eighth of the sum;
//   * chunks are added up in registers, rounded to nearest, in groups of ceil(K / 512) chunks (eight groups at most), and the
//     groups in ascending order.  Where tiles alone leave SMs idle, the groups are what is shared out over blocks: each
//     group's sum goes to scratch memory, and a kernel of its own adds them up.
// W lies on the instruction's M side for every M, as the A operand in tensor memory: sixteen warps read a 32-bit tile of W
// from shared memory (four threads a row), split it and store the parts with tcgen05.st, so that shared memory serves W's floats once
// and the products read only the tokens' parts from it.  Those (split once by a kernel of its own) come by TMA as the
// instruction's N side, 16 to 96 tokens.
//
// What is not finite: a part that is infinite or NaN makes every sum it meets non-finite, so an output that is finite is right,
// and one that is not is formed again as gemm_f32.cu forms it, a chain of multiply-adds over the numbers as they are.
//
// Every wait on an mbarrier is bounded; when one runs out the block raises an abort flag that all roles poll, records
// PHOTON_DEV_WAIT_TIMEOUT, waits (bounded) for its copies in flight, frees its tensor memory and returns.
#include "attention_tc.cuh"

#define FT_BM 128                     // features a tile
#define FT_BK 64                      // a chunk: 64 of K
#define FT_MAXT 96                    // tokens a tile, at most: 48 a thread, twice, stay in registers
#define FT_W_BYTES (FT_BM * FT_BK * 4)
#define FT_MAX_RING 6
#define FT_GROUPS 8
#define FT_FEW 16                     // tokens up to which one launch does all
#define FT_A_COLS 96                  // tensor memory columns of a chunk's parts of W
// Warps of a block: four that issue, those that split W (eight were slower with many tokens: waits in a row and half-rate bit
// operations), those that add the chunks up.  Up to FT_FEW tokens half as many, so that two blocks fit an SM.
template <bool FEW> struct FtShape {
  static constexpr int splitters = FEW ? 8 : 16, adders = FEW ? 4 : 8, threads = (4 + splitters + adders) * 32;
  static constexpr int d_cols = FEW ? 32 : 96, tmem_cols = FEW ? 256 : 512;     // of an accumulator; of all (a power of two)
};
#define FT_BAR_BYTES 512
#define FT_SMEM_LIMIT (227 * 1024)

__device__ __forceinline__ void ft_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// at_split2 by cutting bits off: 8 + 8 + 8 bits, all of them.
__device__ __forceinline__ void ft_cut2(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
  x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u); y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
  mid = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
  x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u); y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
  lo = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

// The chain of gemm_f32.cu, for outputs that are not finite.
__device__ __noinline__ float ft_chain(const float* a, const float* w, int K) {
  float acc = 0.f;
#pragma unroll 8
  for (int k = 0; k < K; ++k) acc = fmaf(__ldg(a + k), __ldg(w + k), acc);
  return acc;
}

__device__ __forceinline__ float ft_checked(float y, const float* a, const float* w, int K) {
  return fabsf(y) <= 3.402823466e38f ? y : ft_chain(a, w, K);
}

// ---------------------------------------------------------------- the tokens' parts: [3][M][Kp], zeros from K to Kp
template <bool VEC>
__global__ void __launch_bounds__(256)
ft_split_kernel(const float* __restrict__ A, long lda, int M, int K, int Kp, bf16* __restrict__ parts) {
  pdl_wait();
  // From here on all that came before is done, so the product's blocks may come and ask for W, which waits for nothing else; where this
  // grid is small, at once
  const bool small = gridDim.x <= 64;
  if (small) pdl_launch_dependents();
  const size_t plane = (size_t)M * Kp;
  const long quads = (long)M * (Kp / 4);
  for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < quads; i += (long)gridDim.x * 256) {
    const long m = i / (Kp / 4);
    const int k = (int)(i % (Kp / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* src = A + m * lda + k;
    if (VEC) {
      if (k < K) v = *reinterpret_cast<const float4*>(src);
    } else {
      if (k < K) v.x = src[0];
      if (k + 1 < K) v.y = src[1];
      if (k + 2 < K) v.z = src[2];
      if (k + 3 < K) v.w = src[3];
    }
    uint2 p[3];
    at_split2(v.x, v.y, p[0].x, p[1].x, p[2].x);
    at_split2(v.z, v.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
    for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(parts + j * plane + (size_t)m * Kp + k) = p[j];
  }
  if (!small) pdl_launch_dependents();
}

// Place in a ring: its stage and the parity of the turn, stepped without a division (a runtime modulus costs a role 200 to 300
// cycles a chunk).
struct FtPlace {
  int s = 0, turn = 0;
  __device__ __forceinline__ void step(int stages) { if (++s == stages) { s = 0; turn ^= 1; } }
};

__device__ __forceinline__ void ft_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
// A number in the shared memory of block `rank` of the cluster, at the place it has here.
__device__ __forceinline__ float ft_peer(const float* mine, int rank) {
  float v;
  asm volatile("{\n.reg .u32 a;\nmapa.shared::cluster.u32 a, %1, %2;\nld.shared::cluster.f32 %0, [a];\n}"
               : "=f"(v) : "r"(tc_smem(mine)), "r"(rank) : "memory");
  return v;
}

struct FtArgs {
  const float* A; long lda;
  const float* W; long ldw;
  float* C; long ldc;
  float* partial;                     // [groups][M][N], where the groups are shared out
  int* err;
  int M, N, K;
  int nt;                             // tokens a tile, a multiple of 16
  int token_tiles, splits;
  int chunks, group_chunks, groups;
  int w_stages, b_stages;
  int sum_bytes, vec;                 // FEW: shared memory of the groups' sums; whether A can be read 16 bytes at a time
};

// ---------------------------------------------------------------- the product: a block per tile of features x tokens x groups
// HC: columns (tokens) of a worker thread; two warps share a lane quarter and halve the tokens.
// FEW: at most 16 tokens, in one launch: the adders split the tokens as well, and the blocks that share out a tile's groups are a
// cluster, whose sums meet in shared memory.  It spares the host two launches of three (27 -> 13 us a call) and takes the
// GPU longer (a Llama 3.2 1B layer's four products with one row: 107 us, 88 in three launches; clusters of eight leave SMs idle, and the
// adders do more in a row), so it is for launches that are not captured.
template <int HC, bool FEW>
__global__ void __launch_bounds__(FtShape<FEW>::threads, FEW ? 2 : 1)
ft_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b, const FtArgs p) {
  using Shape = FtShape<FEW>;
  extern __shared__ unsigned char ft_dyn[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)ft_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* w_ring = base;
  const int part_bytes = p.nt * FT_BK * 2, b_bytes = 3 * part_bytes;
  unsigned char* b_ring = base + p.w_stages * FT_W_BYTES;
  float* sums = reinterpret_cast<float*>(b_ring + p.b_stages * b_bytes);               // FEW: [groups of the block][16][128]
  uint64_t* w_full = reinterpret_cast<uint64_t*>(b_ring + p.b_stages * b_bytes + (FEW ? p.sum_bytes : 0));
  uint64_t* w_empty = w_full + FT_MAX_RING;
  uint64_t* b_full = w_empty + FT_MAX_RING;
  uint64_t* b_empty = b_full + FT_MAX_RING;
  uint64_t* ready = b_empty + FT_MAX_RING;           // [2] the parts of a chunk of W lie in tensor memory, and the accumulator is read
  uint64_t* done = ready + 2;                        // [2] its products are done
  uint64_t* order = done + 2;                        // [2] the other issuer's products are issued
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(order + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // token tiles fastest: blocks that run together share W's tiles
  const int tt = blockIdx.x % p.token_tiles, rest = blockIdx.x / p.token_tiles;
  const int split = rest % p.splits, ft = rest / p.splits;
  const int n0 = ft * FT_BM, t0 = tt * p.nt;
  const int nt = min(p.nt, (p.M - t0 + 15) & ~15);   // the last tile of tokens is as narrow as what is left
  const int group0 = split * p.groups / p.splits, group1 = (split + 1) * p.groups / p.splits;
  const int chunk0 = group0 * p.group_chunks, chunk1 = min(p.chunks, group1 * p.group_chunks);

  auto load_w = [&](int c, int stage) {
#ifdef FT_TEST_NO_LOADS
    return;
#endif
    unsigned char* dst = w_ring + stage * FT_W_BYTES;
    tc_mbar_expect_tx(&w_full[stage], FT_W_BYTES);
    tc_tma_load(dst, &map_w, c * FT_BK, n0, &w_full[stage]);
    tc_tma_load(dst + FT_W_BYTES / 2, &map_w, c * FT_BK + 32, n0, &w_full[stage]);
  };
  if (warp == 0) {
    if (tc_elect()) {
      for (int s = 0; s < FT_MAX_RING; ++s) {
        tc_mbar_init(&w_full[s], 1); tc_mbar_init(&w_empty[s], Shape::splitters);
        tc_mbar_init(&b_full[s], FEW ? Shape::adders : 1); tc_mbar_init(&b_empty[s], 1);
      }
      for (int s = 0; s < 2; ++s) {
        tc_mbar_init(&ready[s], Shape::splitters + Shape::adders); tc_mbar_init(&done[s], 1); tc_mbar_init(&order[s], 1);
      }
      *abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      // W's first tiles, while the others set up; behind ft_split_kernel, which waits for all before it, they need not wait again
      if (FEW) pdl_wait();
      for (int s = 0; s < p.w_stages && chunk0 + s < chunk1; ++s) load_w(chunk0 + s, s);
    }
    __syncwarp();
  } else if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tmem_slot)), "n"(Shape::tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_a = tmem + (FEW ? 64 : 2 * Shape::d_cols);        // two accumulators, then two stages of W's parts

  // registers: 128 threads that only issue (40), 512 that split (48), 256 that hold sums (136): 64,512, as launched (896 x 72);
  // FEW: 128 x 32 + 256 x 64 + 128 x 96 = 32,768, as launched (512 x 64)
  if (warp < 4) {
  if (FEW) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;"); else asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
  if (warp == 0) {
    // ---------------- W's tiles, from the first turn on
    const bool elected = tc_elect();
    int it = min(p.w_stages, chunk1 - chunk0);
    FtPlace at;
    at.turn = 1;
    for (int c = chunk0 + p.w_stages; c < chunk1; ++c, ++it, at.step(p.w_stages)) {
      if (!tc_wait(&w_empty[at.s], at.turn ^ 1, abort_flag)) break;
      if (elected) load_w(c, at.s);
    }
    if (elected && *abort_flag)
      for (int j = (it > p.w_stages ? it - p.w_stages : 0); j < it; ++j)
        for (uint32_t i = 0; i < TC_WAIT_LIMIT && !tc_mbar_try(&w_full[j % p.w_stages], (j / p.w_stages) & 1); ++i) {}
    pdl_wait();
  } else if (warp == 1) {
    // ---------------- the tokens' parts
    pdl_wait();
    const bool elected = tc_elect();
    int it = 0;
    FtPlace at;
    for (int c = FEW ? chunk1 : chunk0; c < chunk1; ++c, ++it, at.step(p.b_stages)) {
      if (!tc_wait(&b_empty[at.s], at.turn ^ 1, abort_flag)) break;
      if (elected) {
        tc_mbar_expect_tx(&b_full[at.s], b_bytes);
        tc_tma_load3(b_ring + at.s * b_bytes, &map_b, c * FT_BK, t0, 0, &b_full[at.s]);
      }
    }
    if (elected && *abort_flag)
      for (int j = (it > p.b_stages ? it - p.b_stages : 0); j < it; ++j)
        for (uint32_t i = 0; i < TC_WAIT_LIMIT && !tc_mbar_try(&b_full[j % p.b_stages], (j / p.b_stages) & 1); ++i) {}
  } else {
    // ---------------- products: two warps, even and odd chunks (accumulators and parts of their own), each behind the other's.  A
    // barrier costs its waiter 100 to 250 cycles even when it is ready; so the next chunk's barriers are waited for while this
    // chunk's products are issued, and only the hand-over lies between them.
    pdl_wait();
    const bool elected = tc_elect();
    const int mine = warp - 2;
    const uint32_t idesc = tc_idesc(FT_BM, nt);
    const uint32_t d = tmem + mine * Shape::d_cols, a = tmem_a + mine * FT_A_COLS;
    // (part of W, part of the tokens), the smallest products first
    constexpr int PW[6] = {0, 2, 1, 0, 1, 0}, PB[6] = {2, 0, 1, 1, 0, 0};
    const uint64_t step = (uint64_t)(part_bytes >> 4);
    FtPlace at;
    int turn = 0;
    if (mine) at.step(p.b_stages);
    for (int c = chunk0 + mine; c < chunk1; c += 2, turn ^= 1) {
      if (!tc_wait(&b_full[at.s], at.turn, abort_flag)) break;
      if (!tc_wait(&ready[mine], turn, abort_flag)) break;
      if (!tc_wait(&order[mine], turn ^ mine ^ 1, abort_flag)) break;
      tc_fence_after();
      if (elected) {
        const uint64_t b0 = tc_desc(tc_smem(b_ring + at.s * b_bytes));
        const uint64_t b[3] = {b0, b0 + step, b0 + 2 * step};
#pragma unroll
        for (int j = 0; j < 6; ++j)
#pragma unroll
          for (int k = 0; k < FT_BK / 16; ++k)
            at_mma_ts(d, a + PW[j] * 32 + k * 8, b[PB[j]] + k * 2, idesc, (j > 0 || k > 0) ? 1u : 0u);
        tc_mbar_arrive(&order[mine ^ 1]);
        tc_commit(&done[mine]);
        tc_commit(&b_empty[at.s]);
      }
      at.step(p.b_stages);
      at.step(p.b_stages);
    }
    pdl_launch_dependents();
  }
  if (FEW && p.splits > 1) { ft_cluster_sync(); ft_cluster_sync(); }
  } else if (warp < 4 + Shape::splitters) {
    // ---------------- W's tile of a chunk into its parts: the warps of a lane quarter (a thread a row) share out the 64 of K, 16 a unit
    if (!FEW) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    constexpr int UNITS = 16 / Shape::splitters;
    const int unit0 = ((warp - 4) >> 2) * UNITS, r = (warp & 3) * 32 + lane;
    const uint32_t a0 = tmem_a + ((uint32_t)((warp & 3) * 32) << 16) + unit0 * 8;
    FtPlace at, two;
    for (int c = chunk0; c < chunk1; ++c, at.step(p.w_stages), two.step(2)) {
      if (!tc_wait_warp(&w_full[at.s], at.turn, abort_flag)) break;
      const unsigned char* row = w_ring + at.s * FT_W_BYTES + (unit0 >> 1) * (FT_W_BYTES / 2) + r * 128;
      uint32_t hi[UNITS][8], mid[UNITS][8], lo[UNITS][8];
#pragma unroll
      for (int u = 0; u < UNITS; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(row + (((((unit0 + u) & 1) * 4 + j) ^ (r & 7)) << 4));
          ft_cut2(v.x, v.y, hi[u][2 * j], mid[u][2 * j], lo[u][2 * j]);
          ft_cut2(v.z, v.w, hi[u][2 * j + 1], mid[u][2 * j + 1], lo[u][2 * j + 1]);
        }
      // all but the stores lies before the wait for the products that read this place
      if (!tc_wait_warp(&done[two.s], two.turn ^ 1, abort_flag)) break;
      tc_fence_after();
#pragma unroll
      for (int u = 0; u < UNITS; ++u) {
        const uint32_t a = a0 + two.s * FT_A_COLS + u * 8;
        ft_st8(a, hi[u]);
        ft_st8(a + 32, mid[u]);
        ft_st8(a + 64, lo[u]);
      }
      tc_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { tc_mbar_arrive(&ready[two.s]); tc_mbar_arrive(&w_empty[at.s]); }
    }
    pdl_wait();
    if (FEW && p.splits > 1) { ft_cluster_sync(); ft_cluster_sync(); }
  } else {
    // ---------------- sums: a thread a feature; two warps share a lane quarter and halve the tile's tokens (FEW: one has all)
    if (FEW) asm volatile("setmaxnreg.inc.sync.aligned.u32 96;"); else asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
    pdl_wait();
    const int quad = warp & 3, half = (warp - 4 - Shape::splitters) >> 2;
    const int r = quad * 32 + lane;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    const int col0 = half * (nt / 2), cols = FEW ? nt : nt / 2;
    float total[HC], group[HC];
    bool ok = true;
    int in_group = 0, groups_done = 0;

    auto finish_group = [&]() {
      if (FEW && p.splits > 1) {
#pragma unroll
        for (int j = 0; j < HC; ++j) if (j < cols) sums[(groups_done * FT_FEW + col0 + j) * FT_BM + r] = group[j];
      } else if (p.splits > 1) {
        if (n0 + r < p.N) {
          float* dst = p.partial + ((size_t)(group0 + groups_done) * p.M + t0 + col0) * p.N + n0 + r;
#pragma unroll
          for (int j = 0; j < HC; ++j)
            if (j < cols && t0 + col0 + j < p.M) __stcg(dst + (size_t)j * p.N, group[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < HC; ++j) total[j] = groups_done == 0 ? group[j] : total[j] + group[j];
      }
      ++groups_done;
      in_group = 0;
    };
    auto promote = [&](int it) {
      const int buf = it & 1;
      if (!tc_wait_warp(&done[buf], (it >> 1) & 1, abort_flag)) { ok = false; return; }
      tc_fence_after();
      constexpr int STEP = HC < 32 ? HC : HC == 32 ? 32 : 24;
#pragma unroll
      for (int q = 0; q < HC; q += STEP) {
        uint32_t v[STEP];
#pragma unroll
        for (int i = 0; i < STEP; i += 8) tc_ld8_issue(tmem + buf * Shape::d_cols + lanes + col0 + q + i, v + i);
        tc_ld_wait();
        if (q + STEP >= HC) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(&ready[buf]);
        }
        if (in_group == 0) {
#pragma unroll
          for (int j = 0; j < STEP; ++j) group[q + j] = __uint_as_float(v[j]);
        } else {
#pragma unroll
          for (int j = 0; j < STEP; ++j) group[q + j] += __uint_as_float(v[j]);
        }
      }
      if (++in_group == p.group_chunks) finish_group();
    };

    if (lane < 2) tc_mbar_arrive(&ready[lane]);      // both accumulators are free
    const int n = chunk1 - chunk0;
    if constexpr (FEW) {
      // a chunk's tokens, three chunks ahead of the sums; the numbers of four are on their way (under a stream of W a load takes as
      // long as two or three chunks).  A thread has four numbers of two tokens.
      const int w = threadIdx.x - (4 + Shape::splitters) * 32, row = w >> 4, quad4 = w & 15;
      auto fetch = [&](int c, int m) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        const int k = c * FT_BK + quad4 * 4;
        if (c < chunk1 && m < p.M && k < p.K) {       // K is a multiple of four
          const float* src = p.A + (size_t)m * p.lda + k;
          if (p.vec) v = *reinterpret_cast<const float4*>(src);
          else v = make_float4(src[0], src[1], src[2], src[3]);
        }
        return v;
      };
      float4 next[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) { next[i][0] = fetch(chunk0 + i, row); next[i][1] = fetch(chunk0 + i, row + 8); }
      FtPlace at;
      auto put = [&](int c, float4* slot) {
        if (!tc_wait_warp(&b_empty[at.s], at.turn ^ 1, abort_flag)) { ok = false; return; }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 v = slot[h];
          slot[h] = fetch(c + 4, row + 8 * h);
          uint2 q[3];
          at_split2(v.x, v.y, q[0].x, q[1].x, q[2].x);
          at_split2(v.z, v.w, q[0].y, q[1].y, q[2].y);
          // as TMA would lay them: 128 bytes a row, 16-byte pieces swizzled by the row
          unsigned char* dst = b_ring + at.s * b_bytes + (row + 8 * h) * 128 + (((quad4 >> 1) ^ (row & 7)) << 4) + (quad4 & 1) * 8;
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(dst + i * part_bytes) = q[i];
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&b_full[at.s]);
        at.step(p.b_stages);
      };
#pragma unroll
      for (int i = 0; i < 3; ++i) if (i < n && ok) put(chunk0 + i, next[i]);
      for (int it = 0; it < n && ok; it += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (ok && it + i + 3 < n) put(chunk0 + it + i + 3, next[(i + 3) & 3]);
          if (ok && it + i < n) promote(it + i);
        }
      }
    } else {
      for (int it = 0; it < n && ok; ++it) promote(it);
    }
    if (ok && in_group > 0) finish_group();

    if (FEW && p.splits > 1) {
      // every block of the cluster has its groups' sums in shared memory, and adds up a share of the tokens
      ft_cluster_sync();
      for (int t = split; t < p.M && n0 + r < p.N && !*abort_flag; t += p.splits) {
        float v[FT_GROUPS];
        int s = 0, g0 = 0;
#pragma unroll
        for (int g = 0; g < FT_GROUPS; ++g) {
          if (g >= p.groups) break;
          if (g == (s + 1) * p.groups / p.splits) { ++s; g0 = g; }
          v[g] = ft_peer(sums + ((g - g0) * FT_FEW + t) * FT_BM + r, s);
        }
        float y = v[0];
#pragma unroll
        for (int g = 1; g < FT_GROUPS; ++g) if (g < p.groups) y += v[g];
        p.C[(size_t)t * p.ldc + n0 + r] = ft_checked(y, p.A + (size_t)t * p.lda, p.W + (size_t)(n0 + r) * p.ldw, p.K);
      }
      ft_cluster_sync();                              // none leaves while another reads its sums
    } else if (p.splits == 1 && ok && n0 + r < p.N) {
      float* dst = p.C + (size_t)(t0 + col0) * p.ldc + n0 + r;
#pragma unroll
      for (int j = 0; j < HC; ++j)
        if (j < cols && t0 + col0 + j < p.M)
          dst[(size_t)j * p.ldc] = ft_checked(total[j], p.A + (size_t)(t0 + col0 + j) * p.lda, p.W + (size_t)(n0 + r) * p.ldw, p.K);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(Shape::tmem_cols) : "memory");
  }
  if (threadIdx.x == 0 && *abort_flag) report_error(p.err, PHOTON_DEV_WAIT_TIMEOUT, blockIdx.x, 0, 0);
}

// ---------------------------------------------------------------- the groups' sums, where blocks shared them out
__global__ void __launch_bounds__(256) ft_groups_kernel(const FtArgs p) {
  pdl_wait();
  const size_t plane = (size_t)p.M * p.N;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < plane; i += (size_t)gridDim.x * 256) {
    float g[FT_GROUPS];
#pragma unroll
    for (int j = 0; j < FT_GROUPS; ++j) g[j] = j < p.groups ? __ldcg(p.partial + j * plane + i) : 0.f;
    float y = g[0];
#pragma unroll
    for (int j = 1; j < FT_GROUPS; ++j) if (j < p.groups) y += g[j];
    const size_t m = i / p.N, n = i % p.N;
    p.C[m * p.ldc + n] = ft_checked(y, p.A + m * p.lda, p.W + n * p.ldw, p.K);
  }
  pdl_launch_dependents();
}

// ---------------------------------------------------------------- host side
namespace {
struct FtPlan { int nt, token_tiles, feature_tiles, splits, chunks, group_chunks, groups; };
}

// Tokens a tile and groups a block, by the time that they take in cycles of an SM.  A chunk of 64 of K is 24 products of nt / 2
// cycles each, W's 32 KB and the tokens' parts from L2 and the hand-overs (1,640 cycles measured up to 64 tokens, 1,960 at 96);
// what goes before and after is 6,000.
static FtPlan ft_plan(int M, int N, int K, bool few) {
  FtPlan b = {};
  b.chunks = (K + FT_BK - 1) / FT_BK;
  b.group_chunks = (b.chunks + FT_GROUPS - 1) / FT_GROUPS;
  b.groups = (b.chunks + b.group_chunks - 1) / b.group_chunks;
  b.feature_tiles = (N + FT_BM - 1) / FT_BM;
  const long sms = photon_sm_count();
  double best = 1e300;
  for (int nt = 16; nt <= FT_MAXT && nt < M + 16; nt += 16) {
    const long tt = (M + nt - 1) / nt;
    const double full = (double)((M + 15) / 16 * 16) / nt;                 // the last tile costs what it holds
    for (int s = 1; s <= b.groups; s = few ? 2 * s : s + 1) {
      const long blocks = b.feature_tiles * tt * s;
      // few tokens: two blocks an SM where the sums leave room for them, in clusters of s
      const long places = !few || s <= 2 ? sms : s == 4 ? 2 * 128 : 2 * 120;
      const double rounds = blocks <= 2 * places ? (double)((blocks + places - 1) / places) : b.feature_tiles * full * s / places + 0.5;
      const double chunk = nt > 64 ? 1000.0 + 10.0 * nt : 1640.0;
      double t = rounds * ((double)((b.groups + s - 1) / s * b.group_chunks) * chunk + 6000.0);
      if (s > 1) t += few ? 2000.0 : 5000.0 + (double)M * N * b.groups / sms / 8;
      if (t < best) { best = t; b.nt = nt; b.token_tiles = (int)tt; b.splits = s; }
    }
  }
  return b;
}

static long ft_parts_bytes(int M, int K) {
  const long Kp = ((long)K + FT_BK - 1) / FT_BK * FT_BK;
  return 3 * (long)M * Kp * 2;
}

// Rows that one round of launches takes; more go in several, so that the scratch has a bound.
#define FT_SLAB 4096

// Bytes of scratch that photon_sgemm_tc needs, 16-byte aligned; none with one_launch.
PHOTON_API long photon_sgemm_tc_scratch(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > FT_SLAB) {
    const long a = photon_sgemm_tc_scratch(FT_SLAB, N, K), b = photon_sgemm_tc_scratch(M % FT_SLAB, N, K);
    return a > b ? a : b;
  }
  const FtPlan b = ft_plan(M, N, K, false);
  return ft_parts_bytes(M, K) + (b.splits > 1 ? (long)b.groups * M * N * 4 : 0);
}

// Kernels that photon_sgemm_tc launches.
PHOTON_API int photon_sgemm_tc_launches(int M, int N, int K, int one_launch) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (one_launch) return 1;
  int n = 0;
  for (; M > 0; M -= FT_SLAB) n += ft_plan(M < FT_SLAB ? M : FT_SLAB, N, K, false).splits > 1 ? 3 : 2;
  return n;
}

template <int HC, bool FEW>
static int ft_go(const CUtensorMap& mw, const CUtensorMap& mb, const FtArgs& a, int blocks, size_t smem, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(ft_kernel<HC, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks); cfg.blockDim = dim3(FtShape<FEW>::threads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (FEW && a.splits > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = a.splits; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (photon_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  e = cudaLaunchKernelEx(&cfg, ft_kernel<HC, FEW>, mw, mb, a);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

PHOTON_API int photon_sgemm_tc(const float* A, long lda, const float* W, long ldw, float* C, long ldc, int M, int N, int K,
                               int one_launch, void* scratch, long scratch_bytes, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (one_launch && M > FT_FEW)) return PHOTON_ERR_ARGUMENT;
  if (K % 4 || ldw % 4 || ((uintptr_t)W & 15) || ((uintptr_t)scratch & 15)) return PHOTON_ERR_UNSUPPORTED;   // TMA
  for (; M > FT_SLAB; M -= FT_SLAB, A += (long)FT_SLAB * lda, C += (long)FT_SLAB * ldc) {
    const int st = photon_sgemm_tc(A, lda, W, ldw, C, ldc, FT_SLAB, N, K, 0, scratch, scratch_bytes, err, stream);
    if (st != 0) return st;
  }
  const bool few = one_launch != 0;
  const FtPlan b = ft_plan(M, N, K, few);
  const long blocks = (long)b.feature_tiles * b.token_tiles * b.splits;
  if (blocks > 0x7fffffffL) return PHOTON_ERR_UNSUPPORTED;
  const long need = few ? 0 : ft_parts_bytes(M, K) + (b.splits > 1 ? (long)b.groups * M * N * 4 : 0);
  if (scratch_bytes < need || (need > 0 && scratch == nullptr)) return PHOTON_ERR_ARGUMENT;
  const int Kp = b.chunks * FT_BK;
  bf16* parts = (bf16*)scratch;

  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return PHOTON_ERR_UNSUPPORTED;
  CUtensorMap mw = {}, mb = {};
  {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, strides[1] = {(cuuint64_t)ldw * 4};
    cuuint32_t box[2] = {32, FT_BM}, one[2] = {1, 1};
    if (fn(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return PHOTON_ERR_ARGUMENT;
  }
  FtArgs a = {};
  a.A = A; a.lda = lda; a.W = W; a.ldw = ldw; a.C = C; a.ldc = ldc; a.err = err;
  a.M = M; a.N = N; a.K = K; a.nt = b.nt; a.token_tiles = b.token_tiles; a.splits = b.splits;
  a.chunks = b.chunks; a.group_chunks = b.group_chunks; a.groups = b.groups;
  a.vec = lda % 4 == 0 && ((uintptr_t)A & 15) == 0;
  const int b_bytes = 3 * b.nt * FT_BK * 2, room = FT_SMEM_LIMIT - 1024 - FT_BAR_BYTES;
  if (few) {
    // two blocks an SM (113 KB each) but for a split in two; one with a deep ring where there are no more blocks than SMs
    a.b_stages = 4;
    a.sum_bytes = b.splits > 1 ? (b.groups + b.splits - 1) / b.splits * FT_FEW * FT_BM * 4 : 0;
    a.w_stages = b.splits == 1 && blocks <= photon_sm_count() ? 5 : 2;
    const size_t smem = (size_t)a.w_stages * FT_W_BYTES + (size_t)a.b_stages * b_bytes + a.sum_bytes + 1024 + FT_BAR_BYTES;
    return ft_go<16, true>(mw, mb, a, (int)blocks, smem, stream);
  }
  {
    cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)M, 3}, strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)M * Kp * 2};
    cuuint32_t box[3] = {FT_BK, (cuuint32_t)b.nt, 3}, one[3] = {1, 1, 1};
    if (fn(&mb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, parts, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return PHOTON_ERR_ARGUMENT;
  }
  const long quads = (long)M * (Kp / 4), want = (quads + 255) / 256, cap = 8L * photon_sm_count();
  const dim3 sgrid((unsigned)(want < cap ? want : cap));
  int st = a.vec ? launch_pdl(ft_split_kernel<true>, sgrid, dim3(256), 0, stream, A, lda, M, K, Kp, parts)
                 : launch_pdl(ft_split_kernel<false>, sgrid, dim3(256), 0, stream, A, lda, M, K, Kp, parts);
  if (st != 0) return st;
  a.partial = (float*)((unsigned char*)scratch + ft_parts_bytes(M, K));
  // as many stages of the tokens' parts as leave W three: a stage's load takes as long as a chunk's products or two
  a.w_stages = b.nt <= 64 ? 4 : 3;
  a.b_stages = (room - a.w_stages * FT_W_BYTES) / b_bytes;
  if (a.b_stages > FT_MAX_RING) {
    a.b_stages = FT_MAX_RING;
    a.w_stages = (room - a.b_stages * b_bytes) / FT_W_BYTES;
    if (a.w_stages > FT_MAX_RING) a.w_stages = FT_MAX_RING;
  }
  const size_t smem = (size_t)a.w_stages * FT_W_BYTES + (size_t)a.b_stages * b_bytes + 1024 + FT_BAR_BYTES;
  if (b.nt <= 16) st = ft_go<8, false>(mw, mb, a, (int)blocks, smem, stream);
  else if (b.nt <= 32) st = ft_go<16, false>(mw, mb, a, (int)blocks, smem, stream);
  else if (b.nt <= 64) st = ft_go<32, false>(mw, mb, a, (int)blocks, smem, stream);
  else st = ft_go<48, false>(mw, mb, a, (int)blocks, smem, stream);
  if (st != 0 || b.splits == 1) return st;
  const long each = ((long)M * N + 255) / 256;
  return launch_pdl(ft_groups_kernel, dim3((unsigned)(each < cap ? each : cap)), dim3(256), 0, stream, a);
}
