// Host interface of the one-rank forms of the gradient ops (no torch dependency).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ccl {

constexpr int kMaxCastTensors = 48;

// dst[off[i] + j] = scale * src[i][j]  (accumulate: += ) for n tensors of one dtype, in one launch.
struct CastTable {
  const void* src[kMaxCastTensors];
  uint64_t off[kMaxCastTensors];     // element offsets in dst
  uint64_t count[kMaxCastTensors];
  int n = 0;
  void* dst = nullptr;
  float scale = 1.f;
};
// in_dtype: bf16, f16 or f32 (comm dtypes); out_dtype: in_dtype or f32.
cudaError_t launch_cast_table(int in_dtype, int out_dtype, bool accumulate, const CastTable& t, cudaStream_t stream);

}  // namespace ccl
