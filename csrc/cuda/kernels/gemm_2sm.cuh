// Compute-bound bf16 GEMM on CTA pairs:  D[M, N] = A[M, K] · B[N, K]^T, row-major result, fp32 accumulation.
//
// What bounds it: tensor throughput, and before that the 128 B/clk of shared memory that both the TMA writes and the
// MMA's operand reads go through. A 128 x 256 tile on one SM moves 48 KB in and 48 KB out per 512 MMA clocks, 192 B/clk:
// the one-CTA kernel stopped at 0.80 of cuBLAS for that reason. A pair of CTAs (cta_group::2) computes 256 x 256
// together, each holding half of A's rows and half of B's: 32 KB in and out per 512 clocks, 128 B/clk, and half the L2
// traffic per flop.
//
//   cluster of two CTAs, persistent over a list of 256 x bn tiles (bn a multiple of 32 chosen per problem, see
//   pick_bn in gemm.cu), 6 stages of (128 x 64 of A + bn/2 x 64 of B) per CTA
//     warp 0      TMA producer in both CTAs; all bytes of a stage are counted on the even CTA's barrier
//     warp 1      TMEM allocation; in the even CTA the MMA issuer (M = 256, N = bn), commits are multicast to both
//     warps 2..5  epilogue of this CTA's 128 rows: TMEM -> registers -> swizzled staging -> TMA store, while the
//                 accumulator's other half (2 x 256 TMEM columns) is already being filled for the next tile
//
// SwiGLU ("dual"): the even CTA loads bn/2 gate rows of B, the odd one the bn/2 up rows `dual_off` further down, so that
// accumulator columns [0, bn/2) are the gate and [bn/2, bn) the up projection of the same outputs, at no extra cost.
// B may be pre-packed in contiguous 128 x 64 tiles (weights, see gemm.h).
#pragma once
#include "gemm_tcgen05.cuh"

namespace ccl {
namespace gemm {

struct Params2 {
  int M, N, K;        // N: columns of the result
  int bn;             // accumulator columns of a tile; a tile covers bn result columns (dual: bn / 2)
  int m_tiles, n_tiles;
  int b_tiled;        // B is pre-packed: tile (nt, kt) at packed row (nt * k_tiles + kt) * 128
  int k_tiles;
  int dual_off;       // > 0: SwiGLU, row offset of the up projection
  int tma_out;        // 1: the result can be written with TMA stores (16-byte aligned base and row stride)
  void* out;
  long long ldo;
  int* status;
};

constexpr int kStage2 = 2 * kBM * kBK * 2;   // 128 rows of A and at most 128 rows of B per CTA
constexpr int kStaging2 = 4 * 2 * 4096;      // four epilogue warps, two 32 x 32 blocks each
constexpr int kStages2 = 6;

struct __align__(8) Barriers2 {
  uint64_t full[kStages2];
  uint64_t empty[kStages2];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  uint32_t failed;
};

__host__ __device__ constexpr size_t smem_bytes_2sm() {
  return 1024 + (size_t)kStages2 * kStage2 + kStaging2 + sizeof(Barriers2);
}

// Tiles that run at the same time share panels of A and B in L2: groups of 8 row tiles (2048 rows) walk the columns.
__device__ __forceinline__ void tile_of_2sm(int t, int m_tiles, int n_tiles, int& mt, int& nt) {
  constexpr int kGroupM = 8;
  const int in_group = kGroupM * n_tiles;
  const int gid = t / in_group;
  const int first_m = gid * kGroupM;
  const int gsm = (m_tiles - first_m) < kGroupM ? (m_tiles - first_m) : kGroupM;
  const int r = t - gid * in_group;
  mt = first_m + r % gsm;
  nt = r / gsm;
}

template <bool DUAL, typename OutT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_2sm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                    const __grid_constant__ CUtensorMap tma_out, const Params2 p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kABytes = kBM * kBK * 2;
  constexpr uint32_t kTmemCols = 512;
  uint8_t* staging = smem + (size_t)kStages2 * kStage2;
  Barriers2* bars = reinterpret_cast<Barriers2*>(staging + kStaging2);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const int cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const int total = p.m_tiles * p.n_tiles;
  const int k_iters = (p.K + kBK - 1) / kBK;
  const int bh = p.bn >> 1;                    // rows of B per CTA
  const int ncols = DUAL ? bh : p.bn;          // result columns of a tile

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages2; ++s) {
      ptx::mbar_init(&bars->full[s], 1);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&bars->tmem_full[b], 1);
      ptx::mbar_init(&bars->tmem_empty[b], 8);  // the four epilogue warps of both CTAs
    }
    bars->failed = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_2sm(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish_2sm();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_arrive();
  ptx::cluster_wait();
  ptx::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  ptx::griddep_launch_dependents();

  if (warp == 0) {
    if (ptx::elect_one()) {
      ptx::prefetch_tmap(&tma_a);
      ptx::prefetch_tmap(&tma_b);
      ptx::griddep_wait();
      const uint32_t stage_tx = 2u * (uint32_t)(kABytes + bh * kBK * 2);
      const uint32_t full0 = ptx::mapa(ptx::smem_u32(&bars->full[0]), 0);
      int s = 0;
      uint32_t phase = 1;  // the first pass over the ring finds it empty
      bool ok = true;
      for (int t = cluster; t < total && ok; t += n_clusters) {
        int mt, nt;
        tile_of_2sm(t, p.m_tiles, p.n_tiles, mt, nt);
        const int arow = mt * 2 * kBM + (int)rank * kBM;
        const int brow = DUAL ? nt * bh + (int)rank * p.dual_off : nt * p.bn + (int)rank * bh;
        const int bstep = p.b_tiled ? kBM : 0;
        int by = p.b_tiled ? (brow / kBM) * p.k_tiles * kBM + brow % kBM : brow;
        for (int k = 0; k < k_iters; ++k, by += bstep) {
          if (!ptx::mbar_wait(&bars->empty[s], phase)) {
            bars->failed = 1;
            if (p.status) atomicExch(p.status, 121);
            ok = false;
            break;
          }
          uint8_t* st = smem + s * kStage2;
          const uint32_t bar = full0 + s * 8;
          if (rank == 0) ptx::mbar_arrive_expect_tx(&bars->full[s], stage_tx);
          ptx::tma_load_2d_2sm(st, &tma_a, bar, k * kBK, arow);
          ptx::tma_load_2d_2sm(st + kABytes, &tma_b, bar, bstep ? 0 : k * kBK, by);
          if (++s == kStages2) {
            s = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && ptx::elect_one()) {
      ptx::griddep_wait();  // the first operands come after it: the time limits of the waits below start here
      const uint32_t idesc = ptx::make_idesc_bf16(2 * kBM, p.bn);
      // the loop below is one thread's serial chain: no divisions, and the descriptors only by addition
      const uint64_t desc_a0 = ptx::make_desc_sw128(ptx::smem_u32(smem));
      const uint64_t desc_b0 = ptx::make_desc_sw128(ptx::smem_u32(smem) + kABytes);
      int s = 0;
      uint32_t phase = 0;
      int i = 0;
      bool ok = true;
      for (int t = cluster; t < total && ok; t += n_clusters, ++i) {
        const int acc = i & 1;
        if (!ptx::mbar_wait(&bars->tmem_empty[acc], (((uint32_t)i >> 1) & 1) ^ 1)) {
          bars->failed = 1;
          if (p.status) atomicExch(p.status, 122);
          break;
        }
        ptx::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int k = 0; k < k_iters; ++k) {
          if (!ptx::mbar_wait(&bars->full[s], phase)) {
            bars->failed = 1;
            if (p.status) atomicExch(p.status, 123);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint64_t da = desc_a0 + (uint32_t)(s * (kStage2 >> 4)), db = desc_b0 + (uint32_t)(s * (kStage2 >> 4));
#pragma unroll
          for (int kk = 0; kk < kBK / 16; ++kk)
            ptx::umma_bf16_ss_2sm(d_tmem, da + kk * 2, db + kk * 2, idesc, (k > 0 || kk > 0) ? 1u : 0u);
          ptx::umma_commit_2sm(&bars->empty[s], 0x3);
          if (++s == kStages2) {
            s = 0;
            phase ^= 1;
          }
        }
        if (ok) ptx::umma_commit_2sm(&bars->tmem_full[acc], 0x3);
      }
    }
  } else {
    const int q = warp & 3;
    const uint32_t stage_buf = ptx::smem_u32(staging + q * 2 * 4096);
    constexpr int kOutBytes = 32 * (int)sizeof(OutT);        // one row of a 32-column block
    constexpr int kSwz = sizeof(OutT) == 2 ? 3 : 7;          // 64-byte or 128-byte swizzle
    ptx::griddep_wait();
    int i = 0;
    uint32_t nstore = 0;
    for (int t = cluster; t < total; t += n_clusters, ++i) {
      int mt, nt;
      tile_of_2sm(t, p.m_tiles, p.n_tiles, mt, nt);
      const int acc = i & 1;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->tmem_full[acc], ((uint32_t)i >> 1) & 1))) {
        bars->failed = 1;
        if (p.status) atomicExch(p.status, 124);
        break;
      }
      ptx::tc_fence_after();
      const int row0 = mt * 2 * kBM + (int)rank * kBM + q * 32;
      const int col0 = nt * ncols;
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * 256;
      for (int c = 0; c < ncols; c += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32b_x32(taddr + c, r);
        float v[32];
        if (DUAL) {
          uint32_t u[32];
          ptx::tmem_ld_32x32b_x32(taddr + bh + c, u);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = silu(__uint_as_float(r[j])) * __uint_as_float(u[j]);
        } else {
          ptx::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        }
        if (c + 32 >= ncols) {
          // the accumulator is in registers: the MMA of the next tile but one may overwrite it
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa(ptx::smem_u32(&bars->tmem_empty[acc]), 0));
        }
        if (row0 >= p.M || col0 + c >= p.N) continue;
        const uint32_t buf = stage_buf + (nstore & 1) * 4096;
        if (p.tma_out) {
          if (lane == 0) ptx::tma_store_wait_read<1>();  // the store before the last one has left its buffer
          __syncwarp();
        } else {
          __syncwarp();
        }
#pragma unroll
        for (int g = 0; g < kOutBytes / 16; ++g) {
          uint32_t w[4];
          if constexpr (sizeof(OutT) == 2) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * g + 2 * j], v[8 * g + 2 * j + 1]);
              w[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = __float_as_uint(v[4 * g + j]);
          }
          const int xr = sizeof(OutT) == 2 ? (lane >> 1) & kSwz : lane & kSwz;
          ptx::st_shared_v4(buf + lane * kOutBytes + ((g ^ xr) << 4), w[0], w[1], w[2], w[3]);
        }
        if (p.tma_out) {
          ptx::fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            ptx::tma_store_2d(&tma_out, staging + q * 2 * 4096 + (nstore & 1) * 4096, col0 + c, row0);
            ptx::tma_store_commit();
          }
        } else {
          // rows whose start is not 16-byte aligned: one row at a time, one column per lane
          __syncwarp();
          const uint8_t* sb = staging + q * 2 * 4096 + (nstore & 1) * 4096;
          OutT* out = static_cast<OutT*>(p.out);
          if (col0 + c + lane < p.N) {
            for (int rr = 0; rr < 32 && row0 + rr < p.M; ++rr) {
              const int byte = lane * (int)sizeof(OutT);
              const int xr = sizeof(OutT) == 2 ? (rr >> 1) & kSwz : rr & kSwz;
              out[(long long)(row0 + rr) * p.ldo + col0 + c + lane] =
                  *reinterpret_cast<const OutT*>(sb + rr * kOutBytes + (((byte >> 4) ^ xr) << 4) + (byte & 15));
            }
          }
        }
        ++nstore;
      }
    }
    if (p.tma_out && lane == 0) ptx::tma_store_wait_all();
  }
  __syncwarp();
  ptx::tc_fence_before();
  __syncthreads();
  // neither CTA may leave while the other can still arrive on its barriers or read its operands
  ptx::cluster_arrive();
  ptx::cluster_wait();
  if (warp == 1) ptx::tmem_dealloc_2sm(tmem_base, kTmemCols);
}

}  // namespace gemm
}  // namespace ccl
