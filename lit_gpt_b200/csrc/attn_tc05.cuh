// Causal prompt attention on tcgen05 (attn_tc05.cu), called by the entry points of attn_prefill.cu for the cases without gate, distance
// bias, soft cap, shared key part or score planes.
#pragma once
#include "common.cuh"

namespace b200 {

struct AttnTc05Args {
  const __nv_bfloat16* q; const __nv_bfloat16* k; const __nv_bfloat16* v; __nv_bfloat16* y;   // q, k, v: rows on 16-byte boundaries
  int64_t q_b, q_h, q_r, k_b, k_h, k_r, v_b, v_h, v_r, y_b, y_r;                              // element strides: batch, head (group), row
  const int4* seqs;       // ragged: {first query row, rows, position of the first row, row of position 0 in k / v}; null: `pos` and T
  const void* pos; int pos64;
  int window;             // > 0 (ragged): row at position i sees keys i - window < j <= i
  const __nv_bfloat16* sink;
  int kv_first_row;       // ragged: the keys start at the sequence's first query row
  int T, n_head, n_groups, max_seq;   // ragged: T is the longest sequence's rows
  float scale_log2;
  int pairs;              // set by launch_attn_tc05: blocks of 256 query rows, one CTA's, before those of 128
};

cudaError_t launch_attn_tc05(const AttnTc05Args& a, int head_size, int batch, cudaStream_t st);

}  // namespace b200
