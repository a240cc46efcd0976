// Prompt-side rotary embedding and KV append, one pass over the QKV projection.
//
// Bound by memory: every q and k element is read once and written once, every v element copied. Eight threads share a head
// (two 16-byte pieces each, 64 dims apart, which is what the rotation pairs), so a warp moves whole 128-byte lines. Before,
// the same work was a dozen elementwise launches per layer: 1.47 ms of a layer at 16 x 1024 rows of 96 heads. It rounds
// where they did (tables and products in bf16), so that a prompt's cache keeps its values.
#include "prefill.h"

#include "gemm.h"
#include "ptx.cuh"

#include <stdint.h>

namespace ccl {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ void unpack8(const uint4& a, float (&f)[8]) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
    f[2 * i] = __low2float(h);
    f[2 * i + 1] = __high2float(h);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void __launch_bounds__(kThreads) rope_append_kernel(const RopeAppendParams p) {
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  const int heads = p.n_heads + 2 * p.n_kv_heads;
  const long long idx = (long long)blockIdx.x * kThreads + threadIdx.x;
  const int j = (int)(idx & 7);
  const long long hr = idx >> 3;
  const int row = (int)(hr / heads);
  if (row >= p.rows) return;
  const int head = (int)(hr - (long long)row * heads);
  const int b = row / p.seq, s = row - b * p.seq;
  __nv_bfloat16* src = p.qkv + (size_t)row * p.qkv_stride + (size_t)head * 128 + j * 8;
  uint4 lo = *reinterpret_cast<const uint4*>(src), hi = *reinterpret_cast<const uint4*>(src + 64);
  const bool is_v = head >= p.n_heads + p.n_kv_heads;
  if (!is_v) {
    float a[8], c[8], x[8], y[8];
    unpack8(lo, a);
    unpack8(hi, c);
    const float4* cr = reinterpret_cast<const float4*>(p.cos + (size_t)s * 64 + j * 8);
    const float4* sr = reinterpret_cast<const float4*>(p.sin + (size_t)s * 64 + j * 8);
    const float4 c0 = cr[0], c1 = cr[1], s0 = sr[0], s1 = sr[1];
    const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    auto r = [](float f) { return __bfloat162float(__float2bfloat16(f)); };
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float cb = r(cs[i]), sb = r(sn[i]);
      x[i] = r(a[i] * cb) - r(c[i] * sb);
      y[i] = r(c[i] * cb) + r(a[i] * sb);
    }
    lo = pack8(x);
    hi = pack8(y);
  }
  __nv_bfloat16* dst = src;
  if (head >= p.n_heads) {
    const int kvh = is_v ? head - p.n_heads - p.n_kv_heads : head - p.n_heads;
    dst = (is_v ? p.v_cache : p.k_cache) + (((size_t)b * p.n_kv_heads + kvh) * p.max_seq + s) * 128 + j * 8;
  }
  *reinterpret_cast<uint4*>(dst) = lo;
  *reinterpret_cast<uint4*>(dst + 64) = hi;
}

}  // namespace

cudaError_t rope_append(const RopeAppendParams& p, cudaStream_t stream) {
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const int heads = p.n_heads + 2 * p.n_kv_heads;
  if (p.rows <= 0 || p.seq <= 0 || p.seq > p.max_seq || p.rows % p.seq != 0 || p.n_kv_heads <= 0 || p.n_heads < 0) return cudaErrorInvalidValue;
  if (!aligned(p.qkv) || !aligned(p.k_cache) || !aligned(p.v_cache) || !aligned(p.cos) || !aligned(p.sin)) return cudaErrorInvalidValue;
  if (p.qkv_stride % 8 != 0 || p.qkv_stride < (long long)heads * 128) return cudaErrorInvalidValue;
  const long long threads = (long long)p.rows * heads * 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((threads + kThreads - 1) / kThreads), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  cfg.attrs = attr;
  cfg.numAttrs = pdl_launch_attr(&attr[0]);
  cudaError_t e = cudaLaunchKernelEx(&cfg, rope_append_kernel, p);
  if (e == cudaSuccess) launch_count_add(1);
  return e;
}

}  // namespace ccl
