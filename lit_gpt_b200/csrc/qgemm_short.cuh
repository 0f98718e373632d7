// Prompt GEMM of up to 256 rows (qgemm_short.cu): what b200_qgemm asks of it.
#pragma once
#include "common.cuh"

namespace b200 {

struct ShortArgs {
  const uint8_t* packed[2];   // reference layout, as in GemmParams; [1]: the up projection beside the gate (gate / up pairs)
  const uint32_t* scale[2];
  const __nv_bfloat16* x;     // (M, K)
  const __nv_bfloat16* bias;  // (N) or null; no gate / up pair
  __nv_bfloat16* y;           // (M, N)
  float* partial;             // partial sums of tiles that two CTAs or more share (short_scratch_bytes)
  int64_t M, N, K;
  int qtype;
};

// ctas == 0: not a shape of this kernel.  `shared`: CTAs take equal ranges of all the k there is to do, tiles cut where a range ends; else whole tiles.
struct ShortPlan {
  int ctas;
  bool shared;
  double time;                // us, as modelled
};

bool short_takes(const ShortArgs& a, bool pair);                              // pointers and sizes
ShortPlan short_shape(int64_t N, int64_t K, bool shared);                      // the CTAs of either way, no time
ShortPlan short_plan(int64_t M, int64_t N, int64_t K, int qtype, bool pair, bool scratch);
size_t short_scratch_bytes(int64_t M, int64_t N, const ShortPlan& plan, bool pair);
cudaError_t launch_short(const ShortArgs& a, const ShortPlan& plan, bool pair, cudaStream_t st);

}  // namespace b200
