// Pieces of C tokens counted through a step's sequences (first row, rows, position, slot) in their order, each with as many as its rows take; a sequence of
// fewer than `least` rows has none (least 0: every sequence has one, rows or not).  Only the rows of the whole step are known on the host, so launches are sized
// for the most that n sequences of `rows` rows can have, and a CTA finds its own here.  Called by whole warps.
#pragma once
#include "common.cuh"

namespace b200 {

__device__ __forceinline__ int seq_pieces(const int4& sq, int least, int C) { return sq.y >= least ? (max(sq.y, 1) + C - 1) / C : 0; }

// the sequence of piece `at` and the piece's number there; -1: there are not that many
__device__ __forceinline__ int seq_of_piece(const int4* seqs, int n_seqs, int least, int C, int at, int& piece) {
  if (n_seqs == 1) {
    piece = at;
    return at < seq_pieces(seqs[0], least, C) ? 0 : -1;
  }
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int s0 = 0; s0 < n_seqs; s0 += 32) {
    const int n = s0 + lane < n_seqs ? seq_pieces(seqs[s0 + lane], least, C) : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const unsigned past = __ballot_sync(0xffffffffu, before + incl > at);
    if (past) {
      const int w = __ffs(past) - 1;
      piece = at - before - __shfl_sync(0xffffffffu, incl - n, w);
      return s0 + w;
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  return -1;
}
// the z-th of the sequences that have pieces, and how many pieces lie before its own; -1: there are not that many
__device__ __forceinline__ int seq_with_pieces(const int4* seqs, int n_seqs, int least, int C, int z, int& before) {
  const int lane = threadIdx.x & 31;
  before = 0;
  for (int s0 = 0; s0 < n_seqs; s0 += 32) {
    const int n = s0 + lane < n_seqs ? seq_pieces(seqs[s0 + lane], least, C) : 0;
    const unsigned have = __ballot_sync(0xffffffffu, n > 0);
    if (z < __popc(have)) {
      const int w = (int)__fns(have, 0, z + 1);
      before += __reduce_add_sync(0xffffffffu, lane < w ? n : 0);
      return s0 + w;
    }
    z -= __popc(have);
    before += __reduce_add_sync(0xffffffffu, n);
  }
  return -1;
}

}  // namespace b200
