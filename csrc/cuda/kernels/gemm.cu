// Host launcher of the tcgen05 bf16 GEMM: builds (and caches) the TMA tensor maps, picks tile
// width / pipeline depth / split-K cluster size, and launches the kernel from gemm_tcgen05.cuh.
#include "gemm.h"
#include "gemm_2sm.cuh"
#include "gemm_tcgen05.cuh"
#include "tma_desc.h"

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>

namespace ccl {

namespace {
std::atomic<uint64_t> g_launches{0};
}
bool pdl_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("CCL_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}
int pdl_launch_attr(cudaLaunchAttribute* attr) {
  if (!pdl_enabled()) return 0;
  attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr->val.programmaticStreamSerializationAllowed = 1;
  return 1;
}

uint64_t launch_count() { return g_launches.load(); }
void launch_count_add(uint64_t n) { g_launches.fetch_add(n); }
void launch_count_reset() { g_launches.store(0); }

namespace gemm {

template <int BN, bool DUAL, typename OutT>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                const Params p) {
  const int m0 = blockIdx.x * kBM;
  gemm_tile_body<BN, DUAL>(&tma_a, &tma_b, p, StoreEpilogue<OutT>{}, TileCoord{m0, m0, (int)blockIdx.y * BN});
}

// Operands of the row-major problem D[M, N] = A · B^T for the CTA-pair kernel.
struct Desc2 {
  const void *a, *b;
  int64_t M, N, K, lda, ldb;
  int b_tiled;
  int64_t b_packed_rows;
};

// Tile width for the CTA-pair kernel.
int pick_bn(int64_t M, int64_t N, bool dual, bool packed) {
  const int64_t mt = (M + 2 * kBM - 1) / (2 * kBM);
  double best = 1e30;
  int bn = 256;
  for (int w = 256; w >= 64; w -= (packed ? w / 2 : 32)) {
    const int64_t cols = dual ? w / 2 : w;
    if (dual && cols % 32 != 0) continue;
    const int64_t nt = (N + cols - 1) / cols;
    const int64_t waves = (mt * nt + 73) / 74;
    const double cost = (double)waves * std::max(2.0 * w, 256.0 + w);
    if (cost < best * 0.999) {
      best = cost;
      bn = w;
    }
  }
  return bn;
}

template <bool DUAL, typename OutT>
cudaError_t launch_2sm(const GemmDesc& d, const Desc2& q, int bn, cudaStream_t stream) {
  Params2 p{};
  p.M = (int)q.M;
  p.N = (int)q.N;
  p.K = (int)q.K;
  p.bn = bn;
  const int k_iters = (int)((q.K + kBK - 1) / kBK);
  p.m_tiles = (int)((q.M + 2 * kBM - 1) / (2 * kBM));
  const int cols = DUAL ? bn / 2 : bn;
  p.n_tiles = (int)((q.N + cols - 1) / cols);
  p.b_tiled = q.b_tiled;
  p.k_tiles = k_iters;
  p.dual_off = (int)d.dual_off;
  p.out = d.out;
  p.ldo = d.ldo;
  p.status = d.status;
  p.tma_out = (reinterpret_cast<uintptr_t>(d.out) & 15) == 0 && (d.ldo * (int64_t)sizeof(OutT)) % 16 == 0;
  CUtensorMap ta, tb, to;
  if (!tma::make_2d_bf16(&ta, q.a, (uint64_t)q.M, (uint64_t)q.K, (uint64_t)q.lda, kBM, kBK)) return cudaErrorInvalidValue;
  if (q.b_tiled) {
    if (!tma::make_2d_bf16(&tb, q.b, (uint64_t)q.b_packed_rows, (uint64_t)kBK, (uint64_t)kBK, bn / 2, kBK)) return cudaErrorInvalidValue;
  } else if (!tma::make_2d_bf16(&tb, q.b, (uint64_t)(DUAL ? d.dual_off + q.N : q.N), (uint64_t)q.K, (uint64_t)q.ldb, bn / 2, kBK)) {
    return cudaErrorInvalidValue;
  }
  if (p.tma_out) {
    if (!tma::make_2d_result(&to, d.out, (uint64_t)q.M, (uint64_t)q.N, (uint64_t)d.ldo, sizeof(OutT) == 4)) return cudaErrorInvalidValue;
  } else {
    to = ta;
  }
  auto kern = gemm_2sm_kernel<DUAL, OutT>;
  const size_t smem = smem_bytes_2sm();
  static DeviceOnce configured;
  if (configured.pending()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes_2sm());
    if (e != cudaSuccess) return e;
    configured.done();
  }
  const int total = p.m_tiles * p.n_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (total < 74 ? total : 74), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  cfg.attrs = attr;
  cfg.numAttrs = pdl_launch_attr(&attr[0]);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, tb, to, p);
  if (e == cudaSuccess) g_launches.fetch_add(1);
  return e;
}

cudaError_t dispatch_2sm(const GemmDesc& d, cudaStream_t stream) {
  Desc2 q{};
  q.K = d.K;
  if (d.trans_out) {  // out[n * ldo + m]: the rows of the result are B's
    q.a = d.b;
    q.M = d.N;
    q.lda = d.ldb;
    q.b = d.a;
    q.N = d.M;
    q.ldb = d.lda;
    q.b_tiled = d.a_tiled;
    q.b_packed_rows = d.a_packed_rows;
  } else {
    q.a = d.a;
    q.M = d.M;
    q.lda = d.lda;
    q.b = d.b;
    q.N = d.N;
    q.ldb = d.ldb;
  }
  // a given width counts result columns (dual: of each half)
  int bn = d.bn > 0 ? std::min(256, d.dual_off > 0 ? 2 * d.bn : d.bn) : pick_bn(q.M, q.N, d.dual_off > 0, q.b_tiled != 0);
  if (d.dual_off > 0) return d.out_fp32 ? launch_2sm<true, float>(d, q, bn, stream) : launch_2sm<true, __nv_bfloat16>(d, q, bn, stream);
  return d.out_fp32 ? launch_2sm<false, float>(d, q, bn, stream) : launch_2sm<false, __nv_bfloat16>(d, q, bn, stream);
}

// Pipeline depth for a given split: narrow (decode) tiles are memory-bound, so when one CTA per SM
// does not cover the grid the pipeline shrinks until two CTAs fit on an SM.
template <int BN, bool DUAL>
int stages_for(int64_t ctas, int k_iters, int splitk) {
  size_t budget = 200 * 1024;
  if (BN <= 32 && ctas > 148) budget = 104 * 1024;  // measured: 48/64/80 KB budgets were 0.2-6 % slower end to end
  int stages = kMaxStages;
  while (stages > 2 && smem_bytes<BN, DUAL>(stages, splitk) > budget) --stages;
  const int per = (k_iters + splitk - 1) / splitk;
  if (stages > per && per >= 2) stages = per;
  return stages;
}

template <int BN, bool DUAL, typename OutT>
cudaError_t launch(const GemmDesc& d, int splitk, cudaStream_t stream) {
  const int m_tiles = (int)((d.M + kBM - 1) / kBM);
  const int n_tiles = (int)((d.N + BN - 1) / BN);
  const int k_iters = (int)((d.K + kBK - 1) / kBK);

  constexpr size_t kSmemMax = 200 * 1024;
  auto kern = gemm_kernel<BN, DUAL, OutT>;
  static DeviceOnce configured;
  if (configured.pending()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax + 2048);
    if (e != cudaSuccess) return e;
    // the kernel keeps nothing in L1: give shared memory the whole array so that two CTAs fit
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    // split-K over 16 CTAs is one step beyond the portable cluster size
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    configured.done();
  }
  // split-K: bounded by the largest cluster and by the amount of K work per CTA
  if (splitk > 16) splitk = 16;
  while (splitk > 1 && k_iters / splitk < 2) --splitk;
  if (splitk > 8 && splitk < 16) splitk = 8;   // between the portable limit and 16: stay portable
  if (splitk < 1) splitk = 1;
  const int stages = stages_for<BN, DUAL>((int64_t)m_tiles * n_tiles * splitk, k_iters, splitk);
  const size_t smem = smem_bytes<BN, DUAL>(stages, splitk);

  CUtensorMap ta, tb;
  const int64_t a_rows = DUAL ? (d.dual_off + d.M) : d.M;
  if (d.a_tiled) {
    if (!tma::make_2d_bf16(&ta, d.a, (uint64_t)d.a_packed_rows, (uint64_t)kBK, (uint64_t)kBK, kBM, kBK))
      return cudaErrorInvalidValue;
  } else if (!tma::make_2d_bf16(&ta, d.a, (uint64_t)a_rows, (uint64_t)d.K, (uint64_t)d.lda, kBM, kBK)) {
    return cudaErrorInvalidValue;
  }
  if (!tma::make_2d_bf16(&tb, d.b, (uint64_t)d.N, (uint64_t)d.K, (uint64_t)d.ldb, BN, kBK))
    return cudaErrorInvalidValue;

  Params p;
  p.M = (int)d.M;
  p.N = (int)d.N;
  p.K = (int)d.K;
  p.out = d.out;
  p.ldo = d.ldo;
  p.trans_out = d.trans_out;
  p.dual_off = (int)d.dual_off;
  p.stages = stages;
  p.splitk = splitk;
  p.status = d.status;
  p.acquire_a = 0;
  p.a_tiled = d.a_tiled;
  p.a_static = d.a_tiled;  // packed operands are weights: nothing on the stream produces them
  p.a_packed = d.a_tiled ? d.a : nullptr;
  p.k_tiles = k_iters;

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(m_tiles, n_tiles, splitk);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = splitk;
  cfg.attrs = attr;
  cfg.numAttrs = 1 + pdl_launch_attr(&attr[1]);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, tb, p);
  if (e == cudaSuccess) g_launches.fetch_add(1);
  return e;
}

template <int BN>
cudaError_t dispatch_bn(const GemmDesc& d, int splitk, cudaStream_t s) {
  if (d.dual_off > 0) {
    if constexpr (BN <= 128) {
      return d.out_fp32 ? launch<BN, true, float>(d, splitk, s)
                        : launch<BN, true, __nv_bfloat16>(d, splitk, s);
    } else {
      return cudaErrorInvalidValue;
    }
  }
  return d.out_fp32 ? launch<BN, false, float>(d, splitk, s)
                    : launch<BN, false, __nv_bfloat16>(d, splitk, s);
}

}  // namespace gemm

cudaError_t gemm_bf16_tn(const GemmDesc& d, cudaStream_t stream) {
  if (!d.a || !d.b || !d.out || d.M <= 0 || d.N <= 0 || d.K <= 0) return cudaErrorInvalidValue;
  if ((!d.a_tiled && (d.lda % 8)) || (d.ldb % 8)) return cudaErrorInvalidValue;  // TMA strides: 16-byte multiples
  if ((reinterpret_cast<uintptr_t>(d.a) & 15) || (reinterpret_cast<uintptr_t>(d.b) & 15))
    return cudaErrorInvalidValue;
  // Many result rows: the CTA-pair kernel, whose result is row-major (with trans_out the rows are B's; a dual or packed A
  // can only be its B operand, so those need trans_out). Up to 64 columns the one-CTA kernel below stays the better one: it
  // streams A through narrow tiles and splits K (us, pairs / one CTA, at K = 4096 and 16384: 256 x 16 20.5 / 10.2 and 57.3 /
  // 14.3, 4096 x 16 24.6 / 16.4 and 69.6 / 36.9, 1024 x 64 22.5 / 16.4 and 59.4 / 34.8); from 65 on it has no split and took
  // 32.8 and 102.4 for 256 x 80 where pairs take 20.5 and 57.3.
  if (d.a_tiled && d.dual_off % gemm::kBM != 0) return cudaErrorInvalidValue;  // gate and up start on whole packed tiles
  const bool width_ok = d.bn == 0 || d.bn == 64 || d.bn == 128 || (d.bn == 256 && d.dual_off == 0) ||
                        (d.bn > 64 && d.bn < 256 && d.bn % 32 == 0 && !d.a_tiled && d.dual_off == 0);
  if (width_ok && d.splitk <= 1 && (d.trans_out ? d.N : d.M) > 128 &&
      (d.trans_out || (!d.a_tiled && d.dual_off == 0 && d.N > 64)))
    return gemm::dispatch_2sm(d, stream);
  int bn = d.bn;
  if (bn == 0) {
    if (d.N <= 16) bn = 16;
    else if (d.N <= 32) bn = 32;
    else if (d.N <= 64) bn = 64;
    else if (d.N <= 128 || d.dual_off > 0) bn = 128;
    else bn = 256;
  }
  int splitk = d.splitk;
  if (splitk == 0) {
    const int64_t tiles = ((d.M + 127) / 128) * ((d.N + bn - 1) / bn);
    const int64_t k_iters = (d.K + 63) / 64;
    splitk = 1;
    if (bn <= 32) {
      // memory-bound: the best split measured on B200 is the largest one that keeps the grid at
      // no more than ~264 CTAs (just under two per SM, leaving room for cluster placement inside
      // a GPC): 96 tiles -> 2, 86 SwiGLU tiles -> 3, 32 tiles -> 8, 250 tiles -> 1; one more step
      // (e.g. 96 tiles x 3 = 288 CTAs) no longer fits one wave and costs 40 %. At least 4 K-steps
      // stay in every CTA.
      splitk = (int)(264 / tiles);
      // few tiles (a tensor-parallel shard of a projection): clusters of 16 keep more SMs streaming weights
      // (measured at the shapes one rank of eight sees, batch 16: qkv 12 tiles 7.5 -> 6.9 us with 16; the SwiGLU
      // pair, whose CTAs stream two weight tiles per step, 10.9 -> 11.0 us, so it stays at 8)
      if (splitk > 8) splitk = (splitk >= 16 && d.dual_off == 0) ? 16 : 8;
      while (splitk > 1 && k_iters / splitk < 4) splitk = splitk == 16 ? 8 : splitk - 1;
      if (splitk < 1) splitk = 1;
    } else if (bn <= 64 && tiles < 148) {
      splitk = (int)(148 / tiles);
      if (splitk > 4) splitk = 4;
      if (splitk < 1) splitk = 1;
    }
  }
  switch (bn) {
    case 16: return gemm::dispatch_bn<16>(d, splitk, stream);
    case 32: return gemm::dispatch_bn<32>(d, splitk, stream);
    case 64: return gemm::dispatch_bn<64>(d, splitk, stream);
    case 128: return gemm::dispatch_bn<128>(d, splitk, stream);
    case 256: return gemm::dispatch_bn<256>(d, splitk, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ccl
