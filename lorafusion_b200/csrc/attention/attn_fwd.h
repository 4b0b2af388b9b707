// What the two forward kernels share on the host: their parameters, and the launch of the one for groups
// of a single query head.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace lf {

struct AttnFwdParams {
  const int4* tiles;
  int num_tiles;
  int Hq, Hkv;
  int q_col0, k_col0, v_col0;
  __nv_bfloat16* out;
  long long ldo;
  float* lse;
  long long M_total;
  float scale, scale_log2e;
  int pairs_per_cta;  // attn_fwd_kernel: head pairs of a group that one CTA walks (grid.y CTAs share a group)
  int* err;
};

// Hq == Hkv.  Returns 0 or a negative error code.
int launch_attn_fwd_one_head(const AttnFwdParams& p, const CUtensorMap& tm, cudaStream_t stream);

}  // namespace lf
