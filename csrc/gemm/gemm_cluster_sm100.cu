// Products with few output tiles: the contraction is divided over a cluster of CTAs that share one output tile.
//
// What bounds such a product in gemm_sm100.cu is one SM's share of L2 bandwidth: a CTA streams its 32 KB of operands per K block at
// about 160 GB/s (0.2 us a block), so 12 tiles with K = 2048 leave 136 SMs idle and walk 32 blocks. Here the CTAs of a
// cluster (4 or 8) each take a run of K blocks, leave their fp32 partial tile in the shared memory of the CTAs that finish it
// (CTA r finishes rows 128 r / S .. of the tile; distributed shared memory, no global scratch, no cleared result and no atomics), and
// every CTA sums its rows over the ranks in rank order: the result does not depend on timing. The sum is the one a single CTA forms up to the
// association of S partial sums.
//
// 320 threads: warp 0 loads by TMA, warp 1 issues tcgen05.mma, warps 2..9 hand the accumulator (TMEM) over; all finish. Rows
// travel as 16-byte pieces, XOR-swizzled by their row so that a warp's 32 rows meet different banks.
#include "../common/launch.cuh"
#include "../common/tensormap.h"
#include "gemm_common.cuh"

namespace b200 {

constexpr int CL_BN = 128;

struct ClusterSmem {
  static constexpr int BN = CL_BN;
  static constexpr int A_BYTES = BM * TILE_K_BYTES;
  static constexpr int STAGE_BYTES = A_BYTES + BN * TILE_K_BYTES;
  static constexpr int STAGES = 4;
  static constexpr int RECV_BYTES = BM * BN * 4;                 // [S sources][128 / S rows][BN] partial sums
  static constexpr int TOTAL = STAGES * STAGE_BYTES + RECV_BYTES + 256 + 1024;
};

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ GemmParams p) {
  using S = ClusterSmem;
  using T = __nv_bfloat16;
  constexpr int BN = CL_BN;
  constexpr int BK = ElemTraits<T>::BK, STAGES = S::STAGES;
  constexpr int ATOM = TILE_K_BYTES / sizeof(T);
  constexpr int UMMA_K = UMMA_K_BYTES / sizeof(T), K_STEPS = BK / UMMA_K;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* recv = smem + STAGES * S::STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(recv + S::RECV_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int ranks = p.splits, rank = (int)cluster_ctarank();
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    mbar_init(acc_full, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, BN); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  cluster_sync_all();              // every CTA of the cluster runs: its shared memory may be written
  pdl_wait();

  const int n_blocks = (p.N + BN - 1) / BN, m_blocks = (p.M + BM - 1) / BM;
  const int tile = (int)blockIdx.x / ranks;
  const int b = tile / (m_blocks * n_blocks), r2 = tile % (m_blocks * n_blocks), mb = r2 / n_blocks, nb = r2 % n_blocks;
  const int num_kb = (p.K + BK - 1) / BK, per = (num_kb + ranks - 1) / ranks;
  const int kb0 = min(rank * per, num_kb), kb1 = min(kb0 + per, num_kb);

  if (warp == 0) {
    if (lane == 0) {
      const uint32_t tx_bytes = (A_MN ? S::A_BYTES : tile_box(p.M, BM) * TILE_K_BYTES) + (B_MN ? BN * TILE_K_BYTES : tile_box(p.N, BN) * TILE_K_BYTES);
      int stage = 0; uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ST_TIMEOUT_TMA_EMPTY)) break;
        uint8_t* sa = smem + stage * S::STAGE_BYTES;
        uint8_t* sb = sa + S::A_BYTES;
        mbar_expect_tx(&full_bar[stage], tx_bytes);
        if (!A_MN) {
          tma_load_3d(sa, &tmA, &full_bar[stage], kb * BK, mb * BM, b);
        } else {
#pragma unroll
          for (int a = 0; a < BM / ATOM; ++a) tma_load_3d(sa + a * (BK * TILE_K_BYTES), &tmA, &full_bar[stage], mb * BM + a * ATOM, kb * BK, b);
        }
        if (!B_MN) {
          tma_load_3d(sb, &tmB, &full_bar[stage], kb * BK, nb * BN, b);
        } else {
#pragma unroll
          for (int a = 0; a < BN / ATOM; ++a) tma_load_3d(sb + a * (BK * TILE_K_BYTES), &tmB, &full_bar[stage], nb * BN + a * ATOM, kb * BK, b);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(BM, BN, KindOf<T>::CF, KindOf<T>::AF, KindOf<T>::BF, A_MN ? 1u : 0u, B_MN ? 1u : 0u);
      int stage = 0; uint32_t phase = 0; bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase, p.status, ST_TIMEOUT_TMA_FULL)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t sa = smem_u32(smem + stage * S::STAGE_BYTES), sb = sa + S::A_BYTES;
#pragma unroll
        for (int k = 0; k < K_STEPS; ++k)
          umma_kind<T>(tmem_base, operand_desc<T, A_MN>(sa, k), operand_desc<T, B_MN>(sb, k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        tc_commit(&empty_bar[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) tc_commit(acc_full);
    }
    __syncwarp();
  } else {
    // this warp: rows 32 q .., columns chalf * BN / 2 ..; a row goes to the CTA that finishes it
    const int q = warp & 3, chalf = (warp - 2) >> 2, row = q * 32 + lane;
    const int rows_per = BM / ranks, dst = row / rows_per, lr = row % rows_per;
    const uint32_t out = cluster_map(smem_u32(recv), (uint32_t)dst) + (uint32_t)((rank * rows_per + lr) * (BN * 4));
    const bool has_k = kb0 < kb1;
    const bool ok = mbar_wait(acc_full, 0, p.status, ST_TIMEOUT_ACC_FULL);
    tc_fence_after_sync();
#pragma unroll
    for (int c = 0; c < BN / 2; c += 32) {
      uint32_t v[32];
      tmem_ld_x32(tmem_base + (uint32_t(q * 32) << 16) + chalf * (BN / 2) + c, v);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int chunk = (chalf * (BN / 2) + c) / 4 + j;
        const bool keep = has_k && ok;
        st_cluster_v4(out + (uint32_t)((chunk ^ (lr & 7)) << 4), keep ? v[4 * j] : 0u, keep ? v[4 * j + 1] : 0u, keep ? v[4 * j + 2] : 0u, keep ? v[4 * j + 3] : 0u);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();              // every partial row has arrived; nothing is written into another CTA from here on
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, BN); }

  const int rows_per = BM / ranks, row_first = mb * BM + rank * rows_per;
  const float alpha = p.alpha_ptr ? p.alpha * *p.alpha_ptr : p.alpha;
  const bool vec = p.vec_ok != 0;
  for (int i = threadIdx.x; i < rows_per * (BN / 4); i += GEMM_THREADS) {
    const int lr = i / (BN / 4), chunk = i % (BN / 4);
    const int row = row_first + lr, col = nb * BN + chunk * 4;
    if (row >= p.M || col >= p.N) continue;
    const uint8_t* src = recv + lr * (BN * 4) + ((chunk ^ (lr & 7)) << 4);
    const float4 u = *reinterpret_cast<const float4*>(src);
    float f[4] = {u.x, u.y, u.z, u.w};
    for (int r = 1; r < ranks; ++r) {
      const float4 w = *reinterpret_cast<const float4*>(src + r * rows_per * (BN * 4));
      f[0] += w.x; f[1] += w.y; f[2] += w.z; f[3] += w.w;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) f[j] *= alpha;
    const int n = min(4, p.N - col);
    if (p.bias) {
      if (p.bias_f32) {
        const float* bp = reinterpret_cast<const float*>(p.bias) + b * p.strideBias + col;
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < n) f[j] += bp[j];
      } else {
        const __nv_bfloat16* bp = reinterpret_cast<const __nv_bfloat16*>(p.bias) + b * p.strideBias + col;
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < n) f[j] += __bfloat162float(bp[j]);
      }
    }
    const long long at = (long long)b * p.strideC + (long long)row * p.ldc + col;
    if (p.aux_out) {
      __nv_bfloat16* ap = reinterpret_cast<__nv_bfloat16*>(p.aux_out) + at;
#pragma unroll
      for (int j = 0; j < 4; ++j) if (j < n) ap[j] = __float2bfloat16(f[j]);
    }
    if (p.act != ACT_NONE) {
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = act_fwd(f[j], p.act);
    }
    if (p.aux_in) {
      const __nv_bfloat16* ap = reinterpret_cast<const __nv_bfloat16*>(p.aux_in) + at;
#pragma unroll
      for (int j = 0; j < 4; ++j) if (j < n) f[j] *= act_bwd(__bfloat162float(ap[j]), p.dact);
    }
    if (p.residual) {
      const __nv_bfloat16* rp = reinterpret_cast<const __nv_bfloat16*>(p.residual) + (long long)b * p.strideR + (long long)row * p.ldr + col;
#pragma unroll
      for (int j = 0; j < 4; ++j) if (j < n) f[j] += __bfloat162float(rp[j]);
    }
    if (p.out_mode == OUT_BF16) {
      __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + at;
      if (vec && n == 4) *reinterpret_cast<uint2*>(cp) = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
      else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < n) cp[j] = __float2bfloat16(f[j]);
      }
    } else {
      float* cp = reinterpret_cast<float*>(p.C) + at;
      if (p.out_mode == OUT_F32) {
        if (vec && n == 4) *reinterpret_cast<float4*>(cp) = make_float4(f[0], f[1], f[2], f[3]);
        else {
#pragma unroll
          for (int j = 0; j < 4; ++j) if (j < n) cp[j] = f[j];
        }
      } else if (vec && n == 4) {
        atomicAdd(reinterpret_cast<float4*>(cp), make_float4(f[0], f[1], f[2], f[3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < n) atomicAdd(cp + j, f[j]);
      }
    }
  }
}

template <bool A_MN, bool B_MN>
static int cluster_set_attr() {
  static bool done = false;
  if (done) return 0;
  (void)cudaGetLastError();
  cudaError_t e = cudaFuncSetAttribute(gemm_cluster_kernel<A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, ClusterSmem::TOTAL);
  if (e != cudaSuccess) return (int)e;
  done = true;
  return 0;
}

template <bool A_MN, bool B_MN>
static int launch_cluster(const GemmArgs& a, int ranks, cudaStream_t stream) {
  using T = __nv_bfloat16;
  CUtensorMap tmA, tmB;
  int rc = operand_map<T, A_MN>(&tmA, a.A, a.M, a.K, a.batch, a.lda, a.strideA, BM);
  if (rc) return 100 + rc;
  rc = operand_map<T, B_MN>(&tmB, a.B, a.N, a.K, a.batch, a.ldb, a.strideB, CL_BN);
  if (rc) return 200 + rc;
  if (int e = cluster_set_attr<A_MN, B_MN>()) return 300 + e;
  GemmParams p = a.p;
  p.splits = ranks;
  const long long tiles = (long long)((p.M + BM - 1) / BM) * ((p.N + CL_BN - 1) / CL_BN) * p.batch;
  cudaError_t e = launch_pdl_cluster(gemm_cluster_kernel<A_MN, B_MN>, dim3((unsigned)(tiles * ranks)), dim3(GEMM_THREADS), ClusterSmem::TOTAL, ranks,
                                     stream, tmA, tmB, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

// CTAs per tile; 1: one CTA forms each sum. A cluster costs about 2 us (its CTAs start together, so the kernel's start hides less behind its
// predecessor, and the partial tiles cross); a K block costs 0.2 us. Device time in a chain of launches, one CTA a tile (64-wide tiles, the
// better of the two) against clusters of 8 / 4: 16 x 512 x 2048 10.0 / 7.7 us, 333 x 512 x 2048 10.6 / 8.4, with a residual 11.6 / 8.4,
// 333 x 512 x 8192 29.9 / 10.9; 333 x 1024 x 1024 7.4 / 8.4 and 333 x 512 x 512 5.7 / 7.5: below 24 blocks the cluster loses. About 100
// SMs are reached by clusters of 8 at once: more and a second wave begins (32 tiles in clusters of 8: 24 us). Clusters of 4 win alone up to
// 128 CTAs (1024 x 512 x 2048 10.8 / 9.7), but among a block's other launches, which they keep from starting early, 32 tiles lose: LM logits
// of 512 tokens (16 tiles) 1330 -> 1163 us, of 1024 tokens (32 tiles) 1478 -> 1566.
int gemm_cluster_ranks(const GemmArgs& a) {
  if (a.dtype != GEMM_BF16 || a.p.m_valid || a.p.k_valid || a.p.out_mode == OUT_I32 || a.K < 24 * 64) return 1;
  const long long tiles = (long long)((a.p.M + BM - 1) / BM) * ((a.p.N + CL_BN - 1) / CL_BN) * a.p.batch;
  return tiles * 8 <= 96 ? 8 : tiles * 4 <= 64 ? 4 : 1;
}

int gemm_cluster_launch(const GemmArgs& a, int ranks, cudaStream_t stream) {
  if (!a.a_mn && !a.b_mn) return launch_cluster<false, false>(a, ranks, stream);
  if (!a.a_mn && a.b_mn) return launch_cluster<false, true>(a, ranks, stream);
  if (a.a_mn && !a.b_mn) return launch_cluster<true, false>(a, ranks, stream);
  return launch_cluster<true, true>(a, ranks, stream);
}

int gemm_cluster_init() {
  return cluster_set_attr<false, false>() | cluster_set_attr<false, true>() | cluster_set_attr<true, false>() | cluster_set_attr<true, true>();
}

}  // namespace b200
