// Paged causal attention for prompt portions on the fifth-generation tensor cores
// (tcgen05, accumulators in tensor memory), bfloat16, heads of up to 128 numbers (a multiple of 8; tiles are 64 or 128
// wide, zeros behind the head), values of another width where VALUE_DIM says so.
//
// A block owns up to 128 query rows of one request that share a key/value head
// (row = token_in_step * GROUP + head_in_group, as in attention_flash.cu; floor(128 / GROUP)
// whole tokens) and walks the
// request's keys in tiles of 64 (AT_KT):
//   * warp 4 brings the rows of Q (one 3-D TMA box) and then the key and value tiles of the
//     paged cache (one TMA box per page part, the block table followed by the lanes of the
//     warp) into a ring of shared-memory stages, 128-byte swizzle;
//   * one thread of warp 5 issues S = Q K^T (tcgen05.mma, M 128, N 64) into one of two score
//     buffers in tensor memory, and O += P V (M 128, N = head size; V is read as it lies in
//     the cache, keys along the rows, through an MN-major descriptor);
//   * warps 0-3 own one row per thread: they read the scores with tcgen05.ld, keep the
//     running maximum and sum in 32-bit, write P = exp2(..) as bfloat16 back over the scores in
//     tensor memory (the second product takes its A operand from there), and rescale O in tensor memory only when
//     a row's maximum has grown by more than 2^8 since the last rescale (the sum and O stay
//     relative to the maximum in use, so the result is the same up to rounding).
// The scores of tile i + 1 are computed while the softmax of tile i runs.  (attention_tc_pairs_kernel below: two such tiles a block.)
//
// Formula: include/photon/ops/kernels/mha_kernel.hpp:188-229 (scores (q.k)/sqrt(d) for the
// keys up to the token's own position, softmax, weighted sum of values; head h uses
// key/value head h / (n_q/n_kv)), with an optional window.  The reference has no
// tensor-core attention (src/ops/kernels/cuda/paged_attention.cu:90-194).
//
// Keys beyond a row's position are masked by selection, so what their cache rows hold does not
// matter for the scores; their value rows are multiplied by P = 0, so the rows of the last tile
// that lie beyond the request's last key (not yet written, or left by an earlier owner of the
// page) are set to zero in shared memory before the product reads them.  Page parts wholly
// beyond the last key or before the window are not read at all (TMA zero fill).
//
// Every wait on an mbarrier is bounded.  When one runs out the block raises an abort flag
// that all roles poll, records PHOTON_DEV_WAIT_TIMEOUT, waits (bounded) for the copies it
// has in flight, frees its tensor memory and returns.
//
// Compiled per model with -DHEAD_DIM=<d> and, where a value has another width than a key, -DVALUE_DIM=<dv>.
#include "attention_tc.cuh"
#include <type_traits>
#include <math.h>

#ifndef HEAD_DIM
#define HEAD_DIM 64
#endif
#ifndef VALUE_DIM
#define VALUE_DIM HEAD_DIM
#endif
static_assert(HEAD_DIM % 8 == 0 && HEAD_DIM >= 16 && HEAD_DIM <= 128, "head size of the tcgen05 attention");
static_assert(VALUE_DIM % 8 == 0 && VALUE_DIM >= 16 && VALUE_DIM <= 128, "size of a value of the tcgen05 attention");

#define AT_ROWS 128
// Keys per tile.  -DAT_KT=128 (heads of 64 only: two stages of such tiles leave room for two blocks per SM) halves the
// hand-overs per key, but tensor memory then holds ONE score buffer beside O, so the scores of the next tile wait
// for P V of this one: measured 47.5 us against 38.6 us at 2,048 tokens, 522 against 427 us at 8,192.
#ifndef AT_KT
#define AT_KT 64
#endif
static_assert(AT_KT == 64 || (HEAD_DIM == 64 && VALUE_DIM == 64), "tiles of 128 keys only at heads of 64");
static_assert(AT_KT == 64 || AT_KT == 128, "keys per tile");
#define AT_NBUF (AT_KT == 128 ? 1 : 2)             // score buffers in tensor memory (128 columns in all)
#define AT_DH ((HEAD_DIM + 63) / 64)               // 64-wide halves of the head dimension
#define AT_VH ((VALUE_DIM + 63) / 64)              // ... and of a value
#ifndef AT_STAGES
#define AT_STAGES (AT_DH * AT_KT == 64 && AT_VH == 1 ? 3 : 2)   // two blocks per SM either way (81 KB, or 97 KB at heads of 128)
#endif
#ifndef AT_BLOCKS_PER_SM
#define AT_BLOCKS_PER_SM 2
#endif
#define AT_THREADS 192                             // warps 0-3: softmax, warp 4: TMA, warp 5: MMA + TMEM
#define AT_Q_BYTES (AT_ROWS * 128 * AT_DH)
#define AT_K_BYTES (AT_KT * 128 * AT_DH)           // one K tile
#define AT_V_BYTES (AT_KT * 128 * AT_VH)           // one V tile
#define AT_HALF_BYTES (AT_KT * 128)                // one 64-wide half of a K or V tile
#ifndef AT_P_TMEM
#define AT_P_TMEM 1                                // 1: P stays in tensor memory (it takes the place of the scores it came from)
#endif
#define AT_P_BYTES (AT_P_TMEM ? 0 : AT_ROWS * AT_KT * 2)
static_assert(AT_P_TMEM || AT_KT == 64, "P in shared memory only with tiles of 64 keys");
#define AT_STAGE_BYTES (AT_K_BYTES + AT_V_BYTES)
#define AT_SMEM_BYTES (AT_Q_BYTES + AT_STAGES * AT_STAGE_BYTES + 2 * AT_P_BYTES + 1024 + 256)
#define AT_TMEM_COLS 256                           // scores 2 x 64 or 1 x 128 columns, O from column 128
#define AT_O_COL 128
#define AT_RESCALE_STEP 8.0f                       // log2 units a maximum may lag behind before O is rescaled

struct AttnTcParams {
  bf16* out; long out_stride;                      // [T, n_q * dv]
  const int* block_table; int max_pages;           // [S, max_pages]
  const int* cu_tokens;                            // [S + 1]
  const int* positions;                            // [T]
  int n_kv, group, tile_rows, page_size, num_pages, box_rows, window, tiles_per_seq, num_seqs, total_rows;
  float scale_log2;                                // scale * log2(e); with bounded scores log2(e) alone
  int* err;
  // keep_first: with a window, keys 0 .. keep_first - 1 stay visible behind it.  sinks [n_q] (may be null): one more key
  // with this score and no value in a head's softmax.  softcap > 0: scores become softcap * tanh(score * cap_in), cap_in = scale / softcap.
  int keep_first;
  const float* sinks;
  float softcap, cap_in;
  const bf16* gate; long gate_stride;              // may be null: [T, n_q * dv]; every output is multiplied by sigmoid(gate)
};

// The grid has a block per `per` tiles of the requests that have tiles here (few rows: the split-key kernel takes the
// request), one request behind the other: every warp walks the requests, 32 at a time, to the one that holds the block's
// tiles.  A grid of (requests x tiles of the longest) was 8,528 blocks where 208 had work, a portion of 1,093
// tokens beside 40 decoded ones (24/8 heads of 128): 105 us, against 70 us without the empty blocks, each of which took
// the shared memory of a full one.
__device__ __forceinline__ bool at_find(const AttnTcParams& P, int per, int index, int& seq, int& before) {
  seq = 0; before = 0;                             // `before`: blocks of the requests in front of `seq`
  if (P.num_seqs <= 1) return true;
  const int lane = threadIdx.x & 31;
  int total = 0;
  for (int s0 = 0; s0 < P.num_seqs; s0 += 32) {
    const int s = s0 + lane;
    int n = 0;
    if (s < P.num_seqs) {
      const int r = (P.cu_tokens[s + 1] - P.cu_tokens[s]) * P.group;
      if (r > 16) n = (min((r + P.tile_rows - 1) / P.tile_rows, P.tiles_per_seq) + per - 1) / per;
    }
    int upto = n;                                  // inclusive sum over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, total + upto > index);
    if (hit != 0) {
      const int l = __ffs(hit) - 1;
      seq = s0 + l;
      before = total + __shfl_sync(0xffffffffu, upto - n, l);
      return true;
    }
    total += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

// The output of a row: its O divided by its sum, times the gate; columns of tensor memory from `o_addr` on.
__device__ __forceinline__ void at_write(const AttnTcParams& P, uint32_t o_addr, bool valid, int tok, int head, float m_used, float l) {
  // the sink's weight, relative to the maximum in use
  if (P.sinks && valid) l += exp2f(fmaf(P.sinks[head], 1.4426950408889634f, -m_used));
  const float inv = l > 0.f ? 1.f / l : 0.f;
  bf16* dst = P.out + (size_t)tok * P.out_stride + (size_t)head * VALUE_DIM;
  const bf16* gt = P.gate ? P.gate + (size_t)tok * P.gate_stride + (size_t)head * VALUE_DIM : nullptr;
#pragma unroll 1
  for (int cc = 0; cc < VALUE_DIM; cc += 32) {
    uint32_t ov[32];
    tc_ld32(o_addr + cc, ov);
    if (valid) {
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        if (VALUE_DIM % 32 != 0 && cc + j >= VALUE_DIM) continue;
        if (gt) {
          // eight gates of this row (16 bytes): the output times sigmoid(gate), folded into the numbers before `inv`
          const uint4 gz = *reinterpret_cast<const uint4*>(gt + cc + j);
          const __nv_bfloat162* gp = reinterpret_cast<const __nv_bfloat162*>(&gz);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 z = __bfloat1622float2(gp[u]);
            ov[j + 2 * u] = __float_as_uint(__fdividef(__uint_as_float(ov[j + 2 * u]), 1.0f + __expf(-z.x)));
            ov[j + 2 * u + 1] = __float_as_uint(__fdividef(__uint_as_float(ov[j + 2 * u + 1]), 1.0f + __expf(-z.y)));
          }
        }
        uint4 v4;
        v4.x = at_pack(__uint_as_float(ov[j]) * inv, __uint_as_float(ov[j + 1]) * inv);
        v4.y = at_pack(__uint_as_float(ov[j + 2]) * inv, __uint_as_float(ov[j + 3]) * inv);
        v4.z = at_pack(__uint_as_float(ov[j + 4]) * inv, __uint_as_float(ov[j + 5]) * inv);
        v4.w = at_pack(__uint_as_float(ov[j + 6]) * inv, __uint_as_float(ov[j + 7]) * inv);
        *reinterpret_cast<uint4*>(dst + cc + j) = v4;
      }
    }
  }
}

__global__ void __launch_bounds__(AT_THREADS, AT_BLOCKS_PER_SM)
attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const AttnTcParams P) {
  // ---- which rows: uniform for the block, before anything is set up
  const int g = blockIdx.x;
  const int G = P.group;
  pdl_wait();                                      // q, the cache and the step's tables come from kernels before
  int seq, before;
  if (!at_find(P, 1, (int)blockIdx.y, seq, before)) return;
  const int tok0 = P.cu_tokens[seq], ntok = P.cu_tokens[seq + 1] - tok0;
  const int rows = ntok * G;
  const int seq_tiles = min((rows + P.tile_rows - 1) / P.tile_rows, P.tiles_per_seq);
  const int qtile = seq_tiles - 1 - ((int)blockIdx.y - before);        // most keys first
  if (rows <= 16 || qtile < 0) return;
  const int row0 = qtile * P.tile_rows;            // tile_rows: the largest multiple of GROUP up to 128
  const int nrows = min(P.tile_rows, rows - row0);
  const int t_first = row0 / G, t_last = (row0 + nrows - 1) / G;
  const int pos_first = P.positions[tok0 + t_first], pos_last = P.positions[tok0 + t_last];
  const int key_lo = (P.window > 0 && pos_first - P.window + 1 > 0) ? pos_first - P.window + 1 : 0;
  // Key tiles: with kept first keys, the tiles that hold them and lie below the window's first tile come first;
  // i counts through both stretches and tile_of gives the key tile.
  const int tile_begin = key_lo / AT_KT;
  const int kept_tiles = (P.keep_first > 0 && key_lo > 0) ? min((P.keep_first + AT_KT - 1) / AT_KT, tile_begin) : 0;
  const int ntiles = kept_tiles + pos_last / AT_KT + 1 - tile_begin;
  auto tile_of = [&](int i) { return i < kept_tiles ? i : tile_begin + i - kept_tiles; };

  extern __shared__ unsigned char at_dyn[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)at_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = base;
  unsigned char* kv_s = q_s + AT_Q_BYTES;                              // AT_STAGES x (K tile | V tile)
  unsigned char* p_s = kv_s + AT_STAGES * AT_STAGE_BYTES;              // 2 x P
  uint64_t* bars = reinterpret_cast<uint64_t*>(p_s + 2 * AT_P_BYTES);
  uint64_t* q_full = bars;                          // TMA -> MMA
  uint64_t* k_full = bars + 1;                      // [AT_STAGES] TMA -> MMA
  uint64_t* v_full = k_full + AT_STAGES;            // [AT_STAGES] TMA -> MMA
  uint64_t* kv_empty = v_full + AT_STAGES;          // [AT_STAGES] MMA -> TMA
  uint64_t* s_full = kv_empty + AT_STAGES;          // [2] MMA -> softmax
  uint64_t* p_full = s_full + 2;                    // [2] softmax -> MMA (one arrival per warp)
  uint64_t* pv_done = p_full + 2;                   // [2] MMA -> softmax: P buffer free, O up to date
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tc_mbar_init(q_full, 1);
    for (int s = 0; s < AT_STAGES; ++s) { tc_mbar_init(&k_full[s], 1); tc_mbar_init(&v_full[s], 1); tc_mbar_init(&kv_empty[s], 1); }
    for (int b = 0; b < 2; ++b) { tc_mbar_init(&s_full[b], 1); tc_mbar_init(&p_full[b], 4); tc_mbar_init(&pv_done[b], 1); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tmem_slot)), "n"(AT_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 4) {
    // ---------------- producer
    const bool elected = tc_elect();
    if (elected) {
      tc_mbar_expect_tx(q_full, P.tile_rows * 128 * AT_DH);       // rows beyond tile_rows stay as they are: nobody uses them
#pragma unroll
      for (int h = 0; h < AT_DH; ++h)
        tc_tma_load3(q_s + h * (AT_ROWS * 128), &map_q, h * 64, g * G, tok0 + t_first, q_full);
    }
    const int* table = P.block_table + (size_t)seq * P.max_pages;
    const int boxes = AT_KT / P.box_rows;           // parts of a tile that may lie in different pages
    int issued = 0;
    for (int i = 0; i < ntiles; ++i) {
      const int s = i % AT_STAGES;
      // the page of this lane's part, looked up before the wait for a free stage
      int rowc = P.total_rows;                      // outside the map: the part is filled with zeros
      if (lane < boxes) {
        const int key = tile_of(i) * AT_KT + lane * P.box_rows;
        if (key <= pos_last && (key + P.box_rows - 1 >= key_lo || key < P.keep_first)) {
          const int pidx = key / P.page_size, slot = key - pidx * P.page_size;
          const int page = table[pidx];
          if (page < 0 || page >= P.num_pages) report_error(P.err, PHOTON_DEV_BAD_PAGE, tok0, key, page);
          else rowc = (page * P.n_kv + g) * P.page_size + slot;
        }
      }
      if (!__all_sync(0xffffffffu, tc_wait(&kv_empty[s], ((i / AT_STAGES) & 1) ^ 1, abort_flag))) break;
      if (elected) { tc_mbar_expect_tx(&k_full[s], AT_K_BYTES); tc_mbar_expect_tx(&v_full[s], AT_V_BYTES); }
      // one thread issues all parts: the lanes that know their pages would be served one by one, and slower
      unsigned char* kst = kv_s + s * AT_STAGE_BYTES;
      for (int part = 0; part < boxes; ++part, kst += P.box_rows * 128) {
        const int row = __shfl_sync(0xffffffffu, rowc, part);
        if (elected) {
#pragma unroll
          for (int h = 0; h < AT_DH; ++h) tc_tma_load(kst + h * AT_HALF_BYTES, &map_k, h * 64, row, &k_full[s]);
#pragma unroll
          for (int h = 0; h < AT_VH; ++h) tc_tma_load(kst + AT_K_BYTES + h * AT_HALF_BYTES, &map_v, h * 64, row, &v_full[s]);
        }
      }
      issued = i + 1;
    }
    if (elected && *abort_flag) {
      // copies already issued still write into this block's shared memory: wait for them, bounded
      for (uint32_t w = 0; w < TC_WAIT_LIMIT && !tc_mbar_try(q_full, 0); ++w) {}
      for (int j = (issued > AT_STAGES ? issued - AT_STAGES : 0); j < issued; ++j) {
        for (uint32_t w = 0; w < TC_WAIT_LIMIT && !tc_mbar_try(&k_full[j % AT_STAGES], (j / AT_STAGES) & 1); ++w) {}
        for (uint32_t w = 0; w < TC_WAIT_LIMIT && !tc_mbar_try(&v_full[j % AT_STAGES], (j / AT_STAGES) & 1); ++w) {}
      }
    }
  } else if (warp == 5) {
    // ---------------- MMA issuer: the warp waits, one of its lanes issues
    const bool elected = tc_elect();
    {
      const uint32_t idesc_s = tc_idesc(AT_ROWS, AT_KT);
      const uint32_t idesc_o = tc_idesc(AT_ROWS, 64 * AT_VH) | TC_IDESC_B_MN;
      const uint32_t q_addr = tc_smem(q_s);
      auto issue_scores = [&](int i) -> bool {
        const int s = i % AT_STAGES;
        if (!tc_wait(&k_full[s], (i / AT_STAGES) & 1, abort_flag)) return false;
        tc_fence_after();
        if (elected) {
          const uint32_t k_addr = tc_smem(kv_s + s * AT_STAGE_BYTES);
#pragma unroll
          for (int kk = 0; kk < (HEAD_DIM + 15) / 16; ++kk)
            tc_mma(tmem_base + (i % AT_NBUF) * AT_KT, tc_desc(q_addr + (kk >> 2) * (AT_ROWS * 128) + (kk & 3) * 32),
                   tc_desc(k_addr + (kk >> 2) * AT_HALF_BYTES + (kk & 3) * 32), idesc_s, kk > 0 ? 1u : 0u);
          tc_commit(&s_full[i % AT_NBUF]);
        }
        return true;
      };
      bool ok = tc_wait(q_full, 0, abort_flag);
      if (ok) ok = issue_scores(0);
      for (int i = 0; i < ntiles && ok; ++i) {
        // two score buffers: the next tile's scores are issued before this tile's P V; one buffer (P lies where the
        // scores were): after it, and the tensor core runs them in the order of issue
        if (AT_NBUF == 2 && i + 1 < ntiles) { ok = issue_scores(i + 1); if (!ok) break; }
        const int s = i % AT_STAGES;
        if (!tc_wait(&p_full[i % AT_NBUF], (i / AT_NBUF) & 1, abort_flag)) { ok = false; break; }
        if (!tc_wait(&v_full[s], (i / AT_STAGES) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        if (elected) {
          const uint32_t p_addr = tc_smem(p_s + (i & 1) * AT_P_BYTES);
          const uint32_t v_addr = tc_smem(kv_s + s * AT_STAGE_BYTES + AT_K_BYTES);
#pragma unroll
          for (int kk = 0; kk < AT_KT / 16; ++kk) {  // 16 keys: two groups of 8 rows of V
            if (AT_P_TMEM)                         // P: 8 columns of packed pairs per 16 keys, where the tile's scores were
              at_mma_ts(tmem_base + AT_O_COL, tmem_base + (i % AT_NBUF) * AT_KT + kk * 8, tc_desc_mn(v_addr + kk * 2048, AT_HALF_BYTES, 1024),
                        idesc_o, (i > 0 || kk > 0) ? 1u : 0u);
            else                                   // P: 32 bytes along a row of the swizzled tile in shared memory
              tc_mma(tmem_base + AT_O_COL, tc_desc(p_addr + kk * 32), tc_desc_mn(v_addr + kk * 2048, AT_HALF_BYTES, 1024),
                     idesc_o, (i > 0 || kk > 0) ? 1u : 0u);
          }
          tc_commit(&kv_empty[s]);
          tc_commit(&pv_done[i % AT_NBUF]);
        }
        if (AT_NBUF == 1 && i + 1 < ntiles) ok = issue_scores(i + 1);
      }
      pdl_launch_dependents();                      // all products of this block are issued
    }
  } else {
    // ---------------- softmax: thread = row
    const int r = threadIdx.x;                      // 0..127
    const int row = row0 + r;
    const bool valid = r < P.tile_rows && row < rows;
    // rows that nobody reads see every key: masking them would keep their warp busy at every tile (groups of 3: 2 rows of 128)
    const int pos = valid ? P.positions[tok0 + row / G] : 0x7fffffff;
    const int lo = (valid && P.window > 0 && pos - P.window + 1 > 0) ? pos - P.window + 1 : 0;
    const int kept = P.keep_first;
    const float cap = P.softcap, cap_in = P.cap_in * 2.8853900817779268f;     // tanh(x) = 1 - 2 / (2^(2 x log2 e) + 1)
    const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
    const float c = P.scale_log2;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    // the warp goes on or gives up together: tcgen05.ld/st need all of its lanes
    auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, tc_wait(bar, parity, abort_flag) ? 1 : 0) != 0;
    };
    for (int i = 0; i < ntiles; ++i) {
      const int b = i % AT_NBUF;
      if (!wait_all(&s_full[b], (i / AT_NBUF) & 1)) { ok = false; break; }
      tc_fence_after();
      const int key_base = tile_of(i) * AT_KT;
      const bool masked = !(key_base + AT_KT - 1 <= pos && key_base >= lo);
      // 64 scores of this row: keys key_base + 64 * half ..; those the row may not see become -inf
      uint32_t sv[64];
      auto load64 = [&](int half) {
        tc_ld32_issue(lane_addr + b * AT_KT + half * 64, sv);
        tc_ld32_issue(lane_addr + b * AT_KT + half * 64 + 32, sv + 32);
        tc_ld_wait();
        if (cap > 0.f) {
#pragma unroll
          for (int j = 0; j < 64; ++j) {
            const float e = at_exp2(__uint_as_float(sv[j]) * cap_in);
            sv[j] = __float_as_uint(cap - __fdividef(2.0f * cap, e + 1.0f));
          }
        }
        if (masked) {
#pragma unroll
          for (int j = 0; j < 64; ++j) {
            const int key = key_base + half * 64 + j;
            sv[j] = ((key >= lo || key < kept) && key <= pos) ? sv[j] : 0xff800000u;       // -inf
          }
        }
      };
      // first pass: the row's maximum, four independent chains of three-input maxima
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
      for (int half = 0; half < AT_KT / 64; ++half) {
        load64(half);
#pragma unroll
        for (int j = 0; j < 64; j += 8) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            mx4[u] = at_max3(mx4[u], __uint_as_float(sv[j + 2 * u]), __uint_as_float(sv[j + 2 * u + 1]));
        }
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // the maximum in use lags behind the true one by at most AT_RESCALE_STEP
      const float cand = fmaxf(m_used, mx * c);
      float factor = 1.f;
      const bool grow = cand > m_used + AT_RESCALE_STEP;          // also the first finite maximum
      if (grow) { factor = at_exp2(m_used - cand); m_used = cand; l *= factor; }
      const float sub = (m_used == -INFINITY) ? 0.f : m_used;
      // O rescale: the products of the tile before must have landed
      if (i > 0 && __any_sync(0xffffffffu, grow)) {
        if (!wait_all(&pv_done[(i - 1) % AT_NBUF], ((i - 1) / AT_NBUF) & 1)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int cc = 0; cc < VALUE_DIM; cc += 32) {
          uint32_t ov[32];
          tc_ld32(lane_addr + AT_O_COL + cc, ov);
#pragma unroll
          for (int j = 0; j < 32; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * factor);
          tc_st32(lane_addr + AT_O_COL + cc, ov);
        }
        tc_st_wait();
      }
      if (i == ntiles - 1 && pos_last - key_base + 1 < AT_KT) {
        // value rows beyond the request's last key: zeros instead of whatever the page holds
        const int nvalid = pos_last - key_base + 1, nzero = AT_KT - nvalid;
        const int s = i % AT_STAGES;
        if (!wait_all(&v_full[s], (i / AT_STAGES) & 1)) { ok = false; break; }
        unsigned char* vst = kv_s + s * AT_STAGE_BYTES + AT_K_BYTES;
        for (int e = r; e < nzero * 8 * AT_VH; e += AT_ROWS) {
          const int half = e / (nzero * 8), rem = e - half * (nzero * 8);
          *reinterpret_cast<uint4*>(vst + half * AT_HALF_BYTES + (nvalid + (rem >> 3)) * 128 + ((rem & 7) << 4)) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> the tensor core's reads
      }
      // second pass: P = exp2(score * c - max in use), 64 keys at a time (tiles of 128 keys: read again from tensor
      // memory, so that a row's scores never need 128 registers)
      float sum8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const float nsub = -sub;
#pragma unroll 1
      for (int half = 0; half < AT_KT / 64; ++half) {
        if (AT_KT > 64) load64(half);
        uint32_t pk[32];
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          float x0, x1;
          at_fma2(x0, x1, __uint_as_float(sv[j]), __uint_as_float(sv[j + 1]), c, nsub);
          const float p0 = at_exp2(x0), p1 = at_exp2(x1);
          at_add2(sum8[j & 6], sum8[(j & 6) + 1], p0, p1);
          pk[j >> 1] = at_pack(p0, p1);
        }
        if (AT_P_TMEM) {
          // P over the scores it came from: packed pairs, 32 columns per 64 keys.  With tiles of 128 keys the first
          // half's P covers scores already read, and the second half's scores (columns 64..127) are still whole.
          tc_st32(lane_addr + b * AT_KT + half * 32, pk);
        } else {
          // the P buffer is free once the products of tile i - 2 have read it
          if (i >= 2 && !wait_all(&pv_done[b], ((i - 2) >> 1) & 1)) { ok = false; break; }
          unsigned char* prow = p_s + b * AT_P_BYTES + r * 128;
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) {
            uint4 v4 = make_uint4(pk[ch * 4], pk[ch * 4 + 1], pk[ch * 4 + 2], pk[ch * 4 + 3]);
            *reinterpret_cast<uint4*>(prow + ((ch ^ (r & 7)) << 4)) = v4;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> the tensor core's reads
        }
      }
      if (!ok) break;
      l += ((sum8[0] + sum8[1]) + (sum8[2] + sum8[3])) + ((sum8[4] + sum8[5]) + (sum8[6] + sum8[7]));
      if (AT_P_TMEM) tc_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(&p_full[b]);
    }
    if (ok && ntiles > 0 && wait_all(&pv_done[(ntiles - 1) % AT_NBUF], ((ntiles - 1) / AT_NBUF) & 1)) {
      tc_fence_after();
      const int tk = valid ? row / G : 0, h = valid ? row - tk * G : 0;
      at_write(P, lane_addr + AT_O_COL, valid, tok0 + tk, g * G + h, m_used, l);
    }
  }
  // ---------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(AT_TMEM_COLS) : "memory");
  }
  if (threadIdx.x == 0 && *abort_flag) report_error(P.err, PHOTON_DEV_WAIT_TIMEOUT, blockIdx.x, blockIdx.y, 0);
}

// ---------------------------------------------------------------- two query tiles a block
// Heads of more than 64 numbers and long contexts: a block of 384 threads owns an SM and two tiles of 128 rows of one request and
// walks the keys that either sees in tiles of 128.  Scores have 128 columns a query tile (a product with N 64 reads 6 KB of
// shared memory in 48 cycles where 32 would do; N 128 takes 64 either way), and while one tile's softmax runs, the tensor cores
// work for the other:
//   * warp 8 brings key and value tiles into rings of their own;
//   * one thread of warp 9 issues, for the two query tiles in turn, O += P V in halves of 64 keys, each as soon as its P lies in
//     tensor memory, and the next S = Q K^T, which takes the place of that P (the tensor cores run products in the order of issue,
//     so scores that are there also say that the O before is);
//   * warps 0-3 and 4-7: the rows of a query tile each.  They have 232 registers (the launch gives 168, the other four warps
//     keep 40: 128 x 40 + 256 x 232 = 64,512 = 384 x 168), so that a row's 128 scores stay in registers.
// The first tile's products end with its own last key: a value that is not finite, of a token that only the second tile sees, meets
// weights of 0 there, and 0 times it would be NaN.  The 16 keys among which it ends come with zeros behind it from a place of their own
// (0.9 us a block: 2,048 tokens from the start 48.3 and 50.1).
// Bound by the softmax warps (3,700 cycles for a pair of tiles of 128 keys, of which the exponentials take 2,048 at 16 a cycle and SM and the
// products as many: both units are active for 55 % of the time).  2,048 tokens behind 14,336, 32/8 heads of 128: 657 us with a tile a block, 482 so (1,070 TFLOP/s);
// 2,048 from the start 54 and 50.  Heads of 64 gain nothing at any length (2,048 tokens 43 and 46 us; with columns of its own for P 42 and 48).
#if HEAD_DIM > 64
#define AP_KT 128
#define AP_THREADS 384
#define AP_K_BYTES (AP_KT * 128 * AT_DH)
#define AP_V_BYTES (AP_KT * 128 * AT_VH)
#define AP_HALF (AP_KT * 128)                      // one 64-wide half of a K or V tile
#define AP_STAGES 2
#define AP_EDGE_BYTES (AT_VH * 2048)                // 16 value rows
#define AP_SMEM_BYTES (2 * AT_Q_BYTES + AP_STAGES * (AP_K_BYTES + AP_V_BYTES) + AP_EDGE_BYTES + 1024 + 256)
static_assert(AP_SMEM_BYTES <= 227 * 1024, "shared memory of a block");
#define AP_O_COL 256                               // scores: 2 x 128 columns; O: 2 x 128

__global__ void __launch_bounds__(AP_THREADS, 1)
attention_tc_pairs_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                          const __grid_constant__ CUtensorMap map_v, const AttnTcParams P) {
  const int g = blockIdx.x;
  const int G = P.group;
  pdl_wait();                                      // q, the cache and the step's tables come from kernels before
  int seq, before;
  if (!at_find(P, 2, (int)blockIdx.y, seq, before)) return;
  const int tok0 = P.cu_tokens[seq], ntok = P.cu_tokens[seq + 1] - tok0;
  const int rows = ntok * G;
  const int seq_tiles = min((rows + P.tile_rows - 1) / P.tile_rows, P.tiles_per_seq);
  const int pair = (seq_tiles + 1) / 2 - 1 - ((int)blockIdx.y - before);           // most keys first
  if (rows <= 16 || pair < 0) return;
  const int row0 = pair * 2 * P.tile_rows;
  const int nq = 2 * pair + 1 < seq_tiles ? 2 : 1;
  const int tile_tokens = P.tile_rows / G;
  const int t_first = row0 / G, t_last = (min(row0 + nq * P.tile_rows, rows) - 1) / G;
  const int pos_first = P.positions[tok0 + t_first], pos_last = P.positions[tok0 + t_last];
  const int key_lo = (P.window > 0 && pos_first - P.window + 1 > 0) ? pos_first - P.window + 1 : 0;
  const int tile_begin = key_lo / AP_KT;
  const int kept_tiles = (P.keep_first > 0 && key_lo > 0) ? min((P.keep_first + AP_KT - 1) / AP_KT, tile_begin) : 0;
  const int ntiles = kept_tiles + pos_last / AP_KT + 1 - tile_begin;
  auto tile_of = [&](int i) { return i < kept_tiles ? i : tile_begin + i - kept_tiles; };
  // the tile of keys behind the last one that the first query tile sees, and that tile's keys before
  const int mid = nq == 2 ? P.positions[tok0 + t_first + tile_tokens - 1] + 1 : 0;
  const int mid_tile = nq == 2 ? kept_tiles + mid / AP_KT - tile_begin : ntiles, mid_keys = mid & (AP_KT - 1);

  extern __shared__ unsigned char at_dyn[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)at_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = base;
  unsigned char* k_s = q_s + 2 * AT_Q_BYTES;
  unsigned char* v_s = k_s + AP_STAGES * AP_K_BYTES;
  unsigned char* edge_s = v_s + AP_STAGES * AP_V_BYTES;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(edge_s + AP_EDGE_BYTES);
  uint64_t* k_full = q_full + 1;                    // [AP_STAGES] TMA -> MMA
  uint64_t* k_empty = k_full + AP_STAGES;           // [AP_STAGES] MMA -> TMA
  uint64_t* v_full = k_empty + AP_STAGES;
  uint64_t* v_empty = v_full + AP_STAGES;
  uint64_t* s_full = v_empty + AP_STAGES;           // [query tile] MMA -> softmax: the scores, and the O before
  uint64_t* p_full = s_full + 2;                    // [query tile][half] softmax -> MMA (one arrival per warp)
  uint64_t* o_full = p_full + 4;                    // [query tile] MMA -> softmax: all of O
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tc_mbar_init(q_full, 1);
    for (int s = 0; s < AP_STAGES; ++s) {
      tc_mbar_init(&k_full[s], 1); tc_mbar_init(&k_empty[s], 1); tc_mbar_init(&v_full[s], 1); tc_mbar_init(&v_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) { tc_mbar_init(&s_full[b], 1); tc_mbar_init(&o_full[b], 1); }
    for (int b = 0; b < 4; ++b) tc_mbar_init(&p_full[b], 4);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tmem_slot)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 8) {
      // ---------------- producer
      const bool elected = tc_elect();
      if (elected) {
        tc_mbar_expect_tx(q_full, nq * P.tile_rows * 128 * AT_DH);     // rows beyond tile_rows stay as they are: nobody uses them
        for (int j = 0; j < nq; ++j)
#pragma unroll
          for (int h = 0; h < AT_DH; ++h)
            tc_tma_load3(q_s + j * AT_Q_BYTES + h * (AT_ROWS * 128), &map_q, h * 64, g * G, tok0 + t_first + j * tile_tokens, q_full);
      }
      const int* table = P.block_table + (size_t)seq * P.max_pages;
      const int boxes = AP_KT / P.box_rows;         // parts of a tile that may lie in different pages
      // the row of this lane's part of a tile; outside the map: the part is filled with zeros
      auto row_of = [&](int i) {
        int rowc = P.total_rows;
        if (lane < boxes) {
          const int key = tile_of(i) * AP_KT + lane * P.box_rows;
          if (key <= pos_last && (key + P.box_rows - 1 >= key_lo || key < P.keep_first)) {
            const int pidx = key / P.page_size, slot = key - pidx * P.page_size;
            const int page = table[pidx];
            if (page < 0 || page >= P.num_pages) report_error(P.err, PHOTON_DEV_BAD_PAGE, tok0, key, page);
            else rowc = (page * P.n_kv + g) * P.page_size + slot;
          }
        }
        return rowc;
      };
      int kn = 0, vn = 0;                           // key and value tiles asked for so far
      auto load = [&](int n, unsigned char* ring, int bytes, int halves, const CUtensorMap* map, uint64_t* full, uint64_t* empty) -> bool {
        const int s = n % AP_STAGES, rowc = row_of(n);
        if (!__all_sync(0xffffffffu, tc_wait(&empty[s], ((n / AP_STAGES) & 1) ^ 1, abort_flag))) return false;
        if (elected) tc_mbar_expect_tx(&full[s], bytes);
        unsigned char* dst = ring + s * bytes;
        for (int part = 0; part < boxes; ++part, dst += P.box_rows * 128) {
          const int row = __shfl_sync(0xffffffffu, rowc, part);
          if (elected)
            for (int h = 0; h < halves; ++h) tc_tma_load(dst + h * AP_HALF, map, h * 64, row, &full[s]);
        }
        return true;
      };
      auto load_k = [&]() { const bool ok = load(kn, k_s, AP_K_BYTES, AT_DH, &map_k, k_full, k_empty); kn += ok; return ok; };
      auto load_v = [&]() { const bool ok = load(vn, v_s, AP_V_BYTES, AT_VH, &map_v, v_full, v_empty); vn += ok; return ok; };
      // in the order in which room appears: the scores of tile i free a key tile before the products of tile i free values
      bool ok = true;
      for (int n = 0; n < AP_STAGES && n < ntiles && ok; ++n) ok = load_k();
      for (int i = 0; i < ntiles && ok; ++i) {
        ok = load_v();
        if (ok && kn < ntiles) ok = load_k();
      }
      if (elected && *abort_flag) {
        // copies already issued still write into this block's shared memory: wait for them, bounded
        for (uint32_t w = 0; w < TC_WAIT_LIMIT && !tc_mbar_try(q_full, 0); ++w) {}
        for (int n = (kn > AP_STAGES ? kn - AP_STAGES : 0); n < kn; ++n)
          for (uint32_t w = 0; w < TC_WAIT_LIMIT && !tc_mbar_try(&k_full[n % AP_STAGES], (n / AP_STAGES) & 1); ++w) {}
        for (int n = (vn > AP_STAGES ? vn - AP_STAGES : 0); n < vn; ++n)
          for (uint32_t w = 0; w < TC_WAIT_LIMIT && !tc_mbar_try(&v_full[n % AP_STAGES], (n / AP_STAGES) & 1); ++w) {}
      }
    } else if (warp == 9) {
      // ---------------- MMA issuer: the warp waits, one of its lanes issues
      const bool elected = tc_elect();
      const uint32_t idesc_s = tc_idesc(AT_ROWS, AP_KT);
      const uint32_t idesc_o = tc_idesc(AT_ROWS, 64 * AT_VH) | TC_IDESC_B_MN;
      auto issue_scores = [&](int i, int j) -> bool {
        const int s = i % AP_STAGES;
        if (!tc_wait(&k_full[s], (i / AP_STAGES) & 1, abort_flag)) return false;
        tc_fence_after();
        if (elected) {
          const uint32_t q_addr = tc_smem(q_s + j * AT_Q_BYTES), k_addr = tc_smem(k_s + s * AP_K_BYTES);
#pragma unroll
          for (int kk = 0; kk < (HEAD_DIM + 15) / 16; ++kk)
            tc_mma(tmem + j * 128, tc_desc(q_addr + (kk >> 2) * (AT_ROWS * 128) + (kk & 3) * 32),
                   tc_desc(k_addr + (kk >> 2) * AP_HALF + (kk & 3) * 32), idesc_s, kk > 0 ? 1u : 0u);
          tc_commit(&s_full[j]);
          if (j == nq - 1) tc_commit(&k_empty[s]);
        }
        return true;
      };
      bool ok = tc_wait(q_full, 0, abort_flag);
      for (int j = 0; j < nq && ok; ++j) ok = issue_scores(0, j);
      // EDGE: the tiles of keys in which the first query tile ends, and behind.  In one loop with the others, whose products it kept from
      // issuing one behind the other, this took 15 % (2,048 tokens behind 14,336, 24/8 heads: 467 -> 540 us); it is rolled up because straight
      // code that a block meets once costs more to fetch than to run.
      auto products = [&](int i, auto edge) -> bool {
        constexpr bool EDGE = decltype(edge)::value;
        const int s = i % AP_STAGES;
        for (int j = 0; j < nq; ++j) {
          // the copy below needs all lanes; the vote alone would take 4 % where the tensor cores wait for the issue
          if (!(EDGE ? tc_wait_warp(&v_full[s], (i / AP_STAGES) & 1, abort_flag) : tc_wait(&v_full[s], (i / AP_STAGES) & 1, abort_flag))) return false;
          const uint32_t o = tmem + AP_O_COL + j * 128, p = tmem + j * 128;          // P: 8 columns of packed pairs for 16 keys, halves 32 apart
          const uint32_t v_addr = tc_smem(v_s + s * AP_V_BYTES);                     // 16 keys: two groups of 8 rows of V
          if (EDGE) {
            const int sees = j > 0 ? AP_KT : i == mid_tile ? mid_keys : 0;
            if (j == 0 && i == mid_tile && (mid_keys & 15)) {
              // the 16 values among which it ends
              const unsigned char* from = v_s + s * AP_V_BYTES + (mid_keys >> 4) * 2048;
#pragma unroll 1
              for (int e = lane; e < 128; e += 32)
#pragma unroll
                for (int h = 0; h < AT_VH; ++h)
                  *reinterpret_cast<uint4*>(edge_s + h * 2048 + e * 16) =
                      (e >> 3) < (mid_keys & 15) ? *reinterpret_cast<const uint4*>(from + h * AP_HALF + e * 16) : make_uint4(0, 0, 0, 0);
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic writes -> the tensor core's reads
              __syncwarp();
            }
#pragma unroll 1
            for (int kk = 0; kk < 8; ++kk) {
              if ((kk & 3) == 0) {
                if (!tc_wait(&p_full[2 * j + (kk >> 2)], i & 1, abort_flag)) return false;
                tc_fence_after();
              }
              if (elected && kk * 16 < sees)
                at_mma_ts(o, p + kk * 8, kk * 16 + 16 <= sees ? tc_desc_mn(v_addr + kk * 2048, AP_HALF, 1024) : tc_desc_mn(tc_smem(edge_s), 2048, 1024),
                          idesc_o, (i > 0 || kk > 0) ? 1u : 0u);
            }
          } else {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              if (!tc_wait(&p_full[2 * j + half], i & 1, abort_flag)) return false;
              tc_fence_after();
              if (elected)
#pragma unroll
                for (int kk = half * 4; kk < half * 4 + 4; ++kk)
                  at_mma_ts(o, p + kk * 8, tc_desc_mn(v_addr + kk * 2048, AP_HALF, 1024), idesc_o, (i > 0 || kk > 0) ? 1u : 0u);
            }
          }
          if (elected) {
            if (j == nq - 1) tc_commit(&v_empty[s]);
            if (i + 1 == ntiles) tc_commit(&o_full[j]);
          }
          if (i + 1 < ntiles && !issue_scores(i + 1, j)) return false;
        }
        return true;
      };
      int i = 0;
      for (; i < min(mid_tile, ntiles) && ok; ++i) ok = products(i, std::false_type());
      for (; i < ntiles && ok; ++i) ok = products(i, std::true_type());
      pdl_launch_dependents();                      // all products of this block are issued
    }
  } else {
    // ---------------- softmax: thread = row of query tile j
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    const int j = warp >> 2;
    const int r = threadIdx.x & 127;
    const int row = row0 + j * P.tile_rows + r;
    const bool valid = j < nq && r < P.tile_rows && row < rows;
    // rows that nobody reads see every key: masking them would keep their warp busy at every tile (groups of 3: 2 rows of 128)
    const int pos = valid ? P.positions[tok0 + row / G] : 0x7fffffff;
    const int lo = (valid && P.window > 0 && pos - P.window + 1 > 0) ? pos - P.window + 1 : 0;
    const int kept = P.keep_first;
    const float cap = P.softcap, cap_in = P.cap_in * 2.8853900817779268f;     // tanh(x) = 1 - 2 / (2^(2 x log2 e) + 1)
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t s_addr = lane_addr + j * 128, o_addr = lane_addr + AP_O_COL + j * 128;
    const float c = P.scale_log2;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    // the warp goes on or gives up together: tcgen05.ld/st need all of its lanes
    auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {
      return __all_sync(0xffffffffu, tc_wait(bar, parity, abort_flag) ? 1 : 0) != 0;
    };
    for (int i = 0; i < ntiles && j < nq; ++i) {
      if (!wait_all(&s_full[j], i & 1)) { ok = false; break; }
      tc_fence_after();
      const int key_base = tile_of(i) * AP_KT;
      uint32_t sv[AP_KT];
#pragma unroll
      for (int u = 0; u < AP_KT; u += 32) tc_ld32_issue(s_addr + u, sv + u);
      tc_ld_wait();
      if (cap > 0.f) {
#pragma unroll
        for (int u = 0; u < AP_KT; ++u) {
          const float e = at_exp2(__uint_as_float(sv[u]) * cap_in);
          sv[u] = __float_as_uint(cap - __fdividef(2.0f * cap, e + 1.0f));
        }
      }
      if (!(key_base + AP_KT - 1 <= pos && key_base >= lo)) {
        // keys this row does not see: those before offset a (but for the kept ones, before k) or behind offset b of the tile
        const int a = lo - key_base, b = pos - key_base, k = kept - key_base;
#pragma unroll
        for (int u = 0; u < AP_KT; ++u) sv[u] = ((u >= a || u < k) && u <= b) ? sv[u] : 0xff800000u;       // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int u = 0; u < AP_KT; u += 8) {
#pragma unroll
        for (int w = 0; w < 4; ++w) mx4[w] = at_max3(mx4[w], __uint_as_float(sv[u + 2 * w]), __uint_as_float(sv[u + 2 * w + 1]));
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // the maximum in use lags behind the true one by at most AT_RESCALE_STEP
      const float cand = fmaxf(m_used, mx * c);
      float factor = 1.f;
      const bool grow = cand > m_used + AT_RESCALE_STEP;          // also the first finite maximum
      if (grow) { factor = at_exp2(m_used - cand); m_used = cand; l *= factor; }
      const float nsub = (m_used == -INFINITY) ? 0.f : -m_used;
      // rescale O: the products of the tile before have landed, because they were issued before these scores
      if (i > 0 && __any_sync(0xffffffffu, grow)) {
#pragma unroll 1
        for (int cc = 0; cc < VALUE_DIM; cc += 32) {
          uint32_t ov[32];
          tc_ld32(o_addr + cc, ov);
#pragma unroll
          for (int u = 0; u < 32; ++u) ov[u] = __float_as_uint(__uint_as_float(ov[u]) * factor);
          tc_st32(o_addr + cc, ov);
        }
        tc_st_wait();
      }
      if (j == 0 && i == ntiles - 1 && pos_last - key_base + 1 < AP_KT) {
        // value rows beyond the request's last key: zeros instead of whatever the page holds.  The first tile's warps write them
        // before their P is ready, and the second tile's products are issued after the first's.
        const int nvalid = pos_last - key_base + 1, nzero = AP_KT - nvalid;
        const int s = i % AP_STAGES;
        if (!wait_all(&v_full[s], (i / AP_STAGES) & 1)) { ok = false; break; }
        unsigned char* vst = v_s + s * AP_V_BYTES;
        for (int e = r; e < nzero * 8 * AT_VH; e += AT_ROWS) {
          const int half = e / (nzero * 8), rem = e - half * (nzero * 8);
          *reinterpret_cast<uint4*>(vst + half * AP_HALF + (nvalid + (rem >> 3)) * 128 + ((rem & 7) << 4)) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> the tensor core's reads
      }
      // P = exp2(score * c - max in use), packed pairs over the scores they came from (32 columns per 64 keys)
      float sum8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t pk[32];
#pragma unroll
        for (int u = 0; u < 64; u += 2) {
          float x0, x1;
          at_fma2(x0, x1, __uint_as_float(sv[half * 64 + u]), __uint_as_float(sv[half * 64 + u + 1]), c, nsub);
          const float p0 = at_exp2(x0), p1 = at_exp2(x1);
          at_add2(sum8[u & 6], sum8[(u & 6) + 1], p0, p1);
          pk[u >> 1] = at_pack(p0, p1);
        }
        tc_st32(s_addr + half * 32, pk);
        tc_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&p_full[2 * j + half]);
      }
      l += ((sum8[0] + sum8[1]) + (sum8[2] + sum8[3])) + ((sum8[4] + sum8[5]) + (sum8[6] + sum8[7]));
    }
    if (ok && j < nq && ntiles > 0 && wait_all(&o_full[j], 0)) {
      tc_fence_after();
      const int tk = valid ? row / G : 0, h = valid ? row - tk * G : 0;
      at_write(P, o_addr, valid, tok0 + tk, g * G + h, m_used, l);
    }
  }
  // ---------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
  if (threadIdx.x == 0 && *abort_flag) report_error(P.err, PHOTON_DEV_WAIT_TIMEOUT, blockIdx.x, blockIdx.y, 0);
}

#endif

PHOTON_API int photon_attention_tc_head_dim() { return HEAD_DIM; }

// Runs the requests of the step that bring more than 16 rows (tokens x group); the others are left
// untouched.  q [T, n_q * d] with row stride q_stride, out [T, n_q * dv]; k_cache
// [num_pages, n_kv, page_size, d] and v_cache [num_pages, n_kv, page_size, dv] contiguous.  group at most 128, page_size a multiple of 8 that
// divides 64 or is a multiple of 64.
PHOTON_API int photon_attention_tc(const void* q, long q_stride, void* out, long out_stride, const void* k_cache,
                                   const void* v_cache, const int* block_table, int max_pages, const int* cu_tokens,
                                   const int* positions, int S, int max_tokens_per_seq, int T, int n_q, int n_kv, int d,
                                   int page_size, int num_pages, int window, float scale, int* err,
                                   cudaStream_t stream) {
  return photon_attention_tc_ex(q, q_stride, out, out_stride, k_cache, v_cache, block_table, max_pages, cu_tokens, positions,
                                S, max_tokens_per_seq, T, n_q, n_kv, d, page_size, num_pages, window, scale, err, 0, nullptr, 0.f,
                                nullptr, 0, stream);
}

// Whether blocks own two query tiles (attention_tc_pairs_kernel).  `keys`: of the longest request that runs here; `tiles`, `pairs`: blocks of
// one and of two tiles.  The pairs' keys cost less and their set-up more: us, one and two tiles a block, without a window
//   keys 4,096 and more: 64 tokens behind 4,096 73 and 71, 2,048 behind 14,336 675 and 512 (32/8 heads of 128), 512 behind 8,192 147 and 140 (24/8);
//   one tile a request, so that no block waits for two: 128 behind 1,536 33 and 29, 128 behind 512 16 and 15, 17 behind 512 15 and 16 (16/16);
//   more tiles than SMs: 1,024 behind 1,536 50 and 49, 1,024 behind 512 33 and 34 (32/8), 2,048 from the start 40 and 42 (16/16);
//   more than two an SM: 2,048 from the start 54 and 50 (32/8), 47 and 46 (24/8), 67 and 69 (40/2: 342 pairs, a third round);
//   fewer: 512 behind 2,048 48 and 49, 1,093 beside 40 decoded tokens 27 and 30 (24/8), 200 beside requests of 14,000 keys 12 and 17.
// Under a window both ends of a row's keys are masked: 2,048 tokens, windows of 128, 512 and 1,024 22 and 30, 34 and 41, 46 and 48; of
// 4,096 behind 8,192 160 and 153, 512 tokens there 74 and 76 (24/8: 76 and 79).  It counts for half of its keys, but with one tile a
// request (17 tokens under windows of 1,024 and 2,048: 23 and 23, 39 and 36).
#ifndef AT_PAIRS_KEYS
#define AT_PAIRS_KEYS 4096
#endif
static bool at_two_tiles(long keys, int window, int tiles_per_seq, long tiles, long pairs, int sms) {
  const bool cut = window > 0 && window < keys;
  const long seen = cut ? window / 2 : keys, full = AT_PAIRS_KEYS;
  if (seen >= full) return true;
  if (tiles_per_seq == 1) return (cut ? window : keys) >= full * 3 / 8;
  if (tiles <= sms) return false;
  return seen >= full * 5 / 8 || (seen >= full / 2 && tiles > 2 * sms && pairs <= 2 * sms);
}
// The rule alone, for a device of `sms` multiprocessors (heads of 64 and less always have one tile).
PHOTON_API int photon_attention_tc_two_tiles(long keys, int window, int tiles_per_seq, long tiles, long pairs, int sms) {
  return HEAD_DIM > 64 && at_two_tiles(keys, window, tiles_per_seq, tiles, pairs, sms);
}

// The same with kept first keys, sinks and bounded scores (see AttnTcParams), and an optional gate: bfloat16
// [T, n_q * dv] with row stride gate_stride (16-byte aligned rows); every output is multiplied by sigmoid(gate).
PHOTON_API int photon_attention_tc_ex(const void* q, long q_stride, void* out, long out_stride, const void* k_cache,
                                      const void* v_cache, const int* block_table, int max_pages, const int* cu_tokens,
                                      const int* positions, int S, int max_tokens_per_seq, int T, int n_q, int n_kv, int d,
                                      int page_size, int num_pages, int window, float scale, int* err, int keep_first,
                                      const float* sinks, float softcap, const void* gate, long gate_stride, cudaStream_t stream) {
  return photon_attention_tc_keys(q, q_stride, out, out_stride, k_cache, v_cache, block_table, max_pages, cu_tokens, positions, S,
                                  max_tokens_per_seq, T, n_q, n_kv, d, page_size, num_pages, window, scale, err, keep_first, sinks,
                                  softcap, gate, gate_stride, 0, stream);
}

// The same, told how many keys the longest request that runs here has, which decides between kernels; 0: not known (the block table's width
// where the step is one request, else few).
PHOTON_API int photon_attention_tc_keys(const void* q, long q_stride, void* out, long out_stride, const void* k_cache,
                                        const void* v_cache, const int* block_table, int max_pages, const int* cu_tokens,
                                        const int* positions, int S, int max_tokens_per_seq, int T, int n_q, int n_kv, int d,
                                        int page_size, int num_pages, int window, float scale, int* err, int keep_first,
                                        const float* sinks, float softcap, const void* gate, long gate_stride, int keys,
                                        cudaStream_t stream) {
  if (S <= 0 || T <= 0) return 0;
  if (keep_first < 0 || softcap < 0.f) return PHOTON_ERR_ARGUMENT;
  if (d != HEAD_DIM || n_kv <= 0 || n_q % n_kv || !(scale > 0.f)) return PHOTON_ERR_UNSUPPORTED;
  const int G = n_q / n_kv;
  if (G > AT_ROWS) return PHOTON_ERR_UNSUPPORTED;
  if (page_size < 8 || (page_size & 7) || !((AT_KT % page_size) == 0 || (page_size % AT_KT) == 0)) return PHOTON_ERR_UNSUPPORTED;
  if (((uintptr_t)q & 15) || (q_stride & 7) || ((uintptr_t)k_cache & 15) || ((uintptr_t)v_cache & 15) ||
      ((uintptr_t)out & 15) || (out_stride & 7))
    return PHOTON_ERR_ARGUMENT;
  const long total_rows = (long)num_pages * n_kv * page_size;
  if (total_rows > 0x7fffffffL || n_kv > 65535) return PHOTON_ERR_UNSUPPORTED;
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return PHOTON_ERR_UNSUPPORTED;
  const int box_rows = page_size < AT_KT ? page_size : AT_KT;
  CUtensorMap map_q, map_k, map_v;
  {
    cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)n_q, (cuuint64_t)T};
    cuuint64_t strides[2] = {(cuuint64_t)d * 2, (cuuint64_t)q_stride * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)(AT_ROWS / G)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(&map_q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return PHOTON_ERR_ARGUMENT;
  }
  int st = make_map(&map_k, k_cache, total_rows, d, d, box_rows);
  if (st != 0) return st;
  st = make_map(&map_v, v_cache, total_rows, VALUE_DIM, VALUE_DIM, box_rows);
  if (st != 0) return st;
  AttnTcParams P;
  P.out = (bf16*)out; P.out_stride = out_stride; P.block_table = block_table; P.max_pages = max_pages;
  P.cu_tokens = cu_tokens; P.positions = positions; P.n_kv = n_kv; P.group = G; P.tile_rows = (AT_ROWS / G) * G;
  P.page_size = page_size;
  P.num_pages = num_pages; P.box_rows = box_rows; P.window = window; P.total_rows = (int)total_rows;
  P.scale_log2 = scale * 1.4426950408889634f; P.err = err;
  P.keep_first = window > 0 ? keep_first : 0; P.sinks = sinks; P.softcap = softcap; P.cap_in = 0.f;
  if (softcap > 0.f) { P.cap_in = scale / softcap; P.scale_log2 = 1.4426950408889634f; }
  if (gate != nullptr && (((uintptr_t)gate & 15) || (gate_stride & 7))) return PHOTON_ERR_ARGUMENT;
  P.gate = (const bf16*)gate; P.gate_stride = gate_stride;
  const long rows = (long)max_tokens_per_seq * G;
  P.tiles_per_seq = (int)((rows + P.tile_rows - 1) / P.tile_rows);
  P.num_seqs = S;
  if ((long)S * P.tiles_per_seq > 65535) return PHOTON_ERR_UNSUPPORTED;
  static bool attr_done = false;
  if (!attr_done) {
    cudaError_t e1 = cudaFuncSetAttribute(attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM_BYTES);
    cudaError_t e2 = cudaFuncSetAttribute(attention_tc_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e1 != cudaSuccess) return (int)e1;
    if (e2 != cudaSuccess) return (int)e2;
    attr_done = true;
  }
  // tiles of all requests together: one partly filled tile for each of those with more than 16 rows
  const long part = (long)T * G / 17 < S ? (long)T * G / 17 : S;
  const long most = (long)T * G / P.tile_rows + part;
  dim3 grid(n_kv, (unsigned)(most < (long)S * P.tiles_per_seq ? most : (long)S * P.tiles_per_seq));
  if (S == 1) grid.y = P.tiles_per_seq;
  if (grid.y == 0) return 0;                        // no request of the step has more than 16 rows
#if HEAD_DIM > 64
  // a request's last tile may be alone in its block
  const unsigned y = (unsigned)(S == 1 ? (grid.y + 1) / 2 : (grid.y + (part < (long)grid.y ? part : (long)grid.y) + 1) / 2);
  const long longest = keys > 0 ? keys : S == 1 ? (long)max_pages * page_size : 0;
  if (at_two_tiles(longest, window, P.tiles_per_seq, (long)grid.y * n_kv, (long)y * n_kv, photon_sm_count())) {
    cudaError_t e = cudaFuncSetAttribute(attention_tc_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AP_SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    return launch_pdl(attention_tc_pairs_kernel, dim3(n_kv, y), dim3(AP_THREADS), (size_t)AP_SMEM_BYTES, stream, map_q, map_k, map_v, P);
  }
#endif
  return launch_pdl(attention_tc_kernel, grid, dim3(AT_THREADS), (size_t)AT_SMEM_BYTES, stream, map_q, map_k, map_v, P);
}
