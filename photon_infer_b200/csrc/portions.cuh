// Where a block's work lies among the long portions of a step.
#pragma once
#include "common.cuh"

struct Portion {
  int seq;      // the request; -1: no request holds the place
  int before;   // places of the long requests in front of it
  int rank;     // long requests in front of it
  int cut_before, cut_rank;     // the same two, counting only requests with more than one place
};

// The requests that bring at least `from` tokens stand one behind the other, with a place for every `size` tokens begun; the others
// have none.  Finds the request that holds place `at` (BY_RANK: the long request number `at`).  All lanes of a warp call it: they
// look at 32 requests at a time.
template <bool BY_RANK>
__device__ __forceinline__ Portion find_portion(const int* __restrict__ cu_tokens, int num_seqs, int from, int size, int at) {
  const int lane = threadIdx.x & 31;
  Portion p = {-1, 0, 0, 0, 0};
  for (int s0 = 0; s0 < num_seqs; s0 += 32) {
    const int s = s0 + lane;
    int n = s < num_seqs ? cu_tokens[s + 1] - cu_tokens[s] : 0;
    n = n > 0 && n >= from ? (n + size - 1) / size : 0;
    int upto = n;                                        // inclusive sum over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned longs = __ballot_sync(0xffffffffu, n > 0), cuts = __ballot_sync(0xffffffffu, n > 1);
    const int rank = p.rank + __popc(longs & ((1u << lane) - 1));
    const unsigned hit = __ballot_sync(0xffffffffu, n > 0 && (BY_RANK ? rank == at : p.before + upto > at));
    if (hit != 0) {
      const int l = __ffs(hit) - 1;
      p.seq = s0 + l;
      p.before += __shfl_sync(0xffffffffu, upto - n, l);
      p.rank = __shfl_sync(0xffffffffu, rank, l);
      p.cut_before += __reduce_add_sync(0xffffffffu, lane < l && n > 1 ? n : 0);
      p.cut_rank += __popc(cuts & ((1u << l) - 1));
      return p;
    }
    p.before += __shfl_sync(0xffffffffu, upto, 31);
    p.rank += __popc(longs);
    p.cut_before += __reduce_add_sync(0xffffffffu, n > 1 ? n : 0);
    p.cut_rank += __popc(cuts);
  }
  return p;
}
