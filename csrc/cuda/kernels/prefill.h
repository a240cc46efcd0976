// Host interface of the prompt-side kernels (no torch dependency).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace ccl {

// Rotary embedding and KV append for whole prompts: `rows` = sequences x seq rows of the QKV projection, row b * seq + s
// holding n_heads q heads, n_kv_heads k heads and n_kv_heads v heads of position s (head_dim 128; n_heads may be 0 when
// only K and V were projected). q is rotated in place, k is rotated into the cache, v is copied into it.
struct RopeAppendParams {
  __nv_bfloat16* qkv;
  long long qkv_stride;      // elements, a multiple of 8
  __nv_bfloat16* k_cache;    // [sequences, n_kv_heads, max_seq, 128]
  __nv_bfloat16* v_cache;
  const float* cos;          // [>= seq, 64]
  const float* sin;
  int rows, seq, n_heads, n_kv_heads, max_seq;
};
cudaError_t rope_append(const RopeAppendParams& p, cudaStream_t stream);

}  // namespace ccl
