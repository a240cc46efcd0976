// Gradient averaging / widening when there is nobody to reduce with: scale, cast and (optionally) accumulate a list of
// tensors into one flat buffer. Bound by memory: a bf16 gradient is read once and its fp32 shard read and written once,
// 10 bytes per parameter; as separate copy, scale and add launches it was 22.
#include "local_ops.h"

#include "collectives.h"
#include "comm.cuh"
#include "gemm.h"

#include <algorithm>

namespace ccl {
namespace {

constexpr int kThreads = 256;

template <typename TIn, typename TOut, bool ACC>
__global__ void __launch_bounds__(kThreads) cast_table_kernel(const __grid_constant__ CastTable t) {
  // No early start for the kernel behind it: GEMMs and the decode step fetch weights before they wait for their predecessor,
  // and what is cast here may be such weights (the copy that this kernel replaces started nobody early either).
  ptx::griddep_wait();
  const TIn* src = static_cast<const TIn*>(t.src[blockIdx.y]);
  TOut* dst = static_cast<TOut*>(t.dst) + t.off[blockIdx.y];
  const size_t n = t.count[blockIdx.y];
  const float scale = t.scale;
  constexpr int N = 16 / (int)sizeof(TIn);              // elements of one source vector
  constexpr int D = N * (int)sizeof(TOut) / 16;         // destination vectors for them (1 or 2)
  const bool aligned = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
  const size_t nv = aligned ? n / N : 0;
  const size_t step = (size_t)gridDim.x * kThreads;
  size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x;
  for (; i < nv; i += step) {
    Vec<TIn> x;
    *reinterpret_cast<uint4*>(&x) = ptx::ld_nc_v4(src + i * N);
    Vec<TOut> y[D];
    if (ACC) {
#pragma unroll
      for (int d = 0; d < D; ++d) *reinterpret_cast<uint4*>(&y[d]) = reinterpret_cast<const uint4*>(dst + i * N)[d];
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
      TOut& o = y[j / Vec<TOut>::kN].v[j % Vec<TOut>::kN];
      const float v = to_acc(x.v[j]) * scale;
      o = from_acc<TOut, float>(ACC ? to_acc(o) + v : v);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) reinterpret_cast<uint4*>(dst + i * N)[d] = *reinterpret_cast<const uint4*>(&y[d]);
  }
  for (size_t e = nv * N + (size_t)blockIdx.x * kThreads + threadIdx.x; e < n; e += step) {
    const float v = to_acc(src[e]) * scale;
    dst[e] = from_acc<TOut, float>(ACC ? to_acc(dst[e]) + v : v);
  }
}

template <typename TIn, typename TOut>
cudaError_t launch(bool accumulate, const CastTable& t, cudaStream_t stream) {
  uint64_t most = 0;
  for (int i = 0; i < t.n; ++i) most = std::max(most, t.count[i]);
  if (most == 0) return cudaSuccess;
  constexpr uint64_t kPerBlock = (uint64_t)kThreads * (16 / sizeof(TIn));
  // eight CTAs of 256 threads fill an SM; more of them would only queue
  const unsigned gx = (unsigned)std::min<uint64_t>((most + kPerBlock - 1) / kPerBlock, 8 * 148);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(gx, t.n, 1);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  cfg.attrs = attr;
  cfg.numAttrs = pdl_launch_attr(&attr[0]);
  cudaError_t e = accumulate ? cudaLaunchKernelEx(&cfg, cast_table_kernel<TIn, TOut, true>, t) : cudaLaunchKernelEx(&cfg, cast_table_kernel<TIn, TOut, false>, t);
  if (e == cudaSuccess) launch_count_add(1);
  return e;
}

}  // namespace

cudaError_t launch_cast_table(int in_dtype, int out_dtype, bool accumulate, const CastTable& t, cudaStream_t stream) {
  if (t.n < 0 || t.n > kMaxCastTensors) return cudaErrorInvalidValue;
  if (t.n == 0) return cudaSuccess;
  if (out_dtype == kF32) {
    if (in_dtype == kBF16) return launch<__nv_bfloat16, float>(accumulate, t, stream);
    if (in_dtype == kF16) return launch<__half, float>(accumulate, t, stream);
    if (in_dtype == kF32) return launch<float, float>(accumulate, t, stream);
  } else if (out_dtype == in_dtype) {
    if (in_dtype == kBF16) return launch<__nv_bfloat16, __nv_bfloat16>(accumulate, t, stream);
    if (in_dtype == kF16) return launch<__half, __half>(accumulate, t, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace ccl
