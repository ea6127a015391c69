// fp32 products too small for the tensor-core kernel: a few thousand to a few million multiply-adds, as in the layers of a
// small classifier. There the tcgen05 kernel is all latency (TMEM allocation, a TMA pipeline and a drain for one tile: 8-10 us
// whatever the size) and MN-major operands cost a transpose launch before it. Here a block of 256 threads owns 16 x 16 results:
// K is walked in chunks of 64 or 128 staged through shared memory K-major (either storage order of either operand is read coalesced
// and turned on the way), the next chunk's loads are in flight during the FMAs, and the chunk's K range is split over four
// groups of 64 threads whose 2 x 2 partial results are added at the end. Operands are cut to TF32 as the
// tensor cores read them (the low 13 mantissa bits dropped), so that a result does not depend on which kernel its size picks;
// their products are exact in fp32 and summed by fp32 FMAs.
// Operands are read past L1 (ld.cg): a block may be resident before the producer of an operand has finished (programmatic
// launch), and a line its SM's L1 still holds from the memory's previous use would be taken for the operand.
// Measured against the tensor-core path (with its transposes) in ops/gemm.py, where the rule for taking it is.
#include "../common/ptx.cuh"
#include "../common/launch.cuh"
#include "gemm_sm100.h"

namespace b200 {

constexpr int SG_T = 16;                                    // tile edge

__device__ __forceinline__ float sg_tf32(float v) { return __uint_as_float(__float_as_uint(v) & 0xffffe000u); }

// 16 rows x KC of an operand stored [rows][K] (MN false) or [K][rows] (MN true)
template <bool MN, int KC>
__device__ __forceinline__ void sg_load(const float* x, long long ld, int row0, int rows, int k0, int K, float (&v)[KC / 16]) {
#pragma unroll
  for (int i = 0; i < KC / 16; ++i) {
    const int e = i * 256 + threadIdx.x;
    const int r = row0 + (MN ? e % SG_T : e / KC), k = k0 + (MN ? e / SG_T : e % KC);
    v[i] = (r < rows && k < K) ? __ldcg(MN ? x + (long long)k * ld + r : x + (long long)r * ld + k) : 0.f;
  }
}
template <bool MN, int KC>
__device__ __forceinline__ void sg_put(float (*s)[KC + 4], const float (&v)[KC / 16]) {      // (padded rows: 16-byte reads of 8 rows hit 8 bank groups)
#pragma unroll
  for (int i = 0; i < KC / 16; ++i) {
    const int e = i * 256 + threadIdx.x;
    s[MN ? e % SG_T : e / KC][MN ? e / SG_T : e % KC] = sg_tf32(v[i]);     // (cut here: at the load it would wait for it)
  }
}

template <bool A_MN, bool B_MN, int KC>
__global__ void __launch_bounds__(256)
gemm_small_kernel(const float* A, long long lda, const float* B, long long ldb, GemmParams p) {
  __shared__ __align__(16) float sA[2][SG_T][KC + 4], sB[2][SG_T][KC + 4];
  __shared__ float4 s_part[3][64];
  const int tid = threadIdx.x, grp = tid >> 6, t = tid & 63;
  const int m0 = blockIdx.y * SG_T, n0 = blockIdx.x * SG_T;
  const int tm = t >> 3, tn = t & 7;                        // rows tm, tm + 8 and columns tn, tn + 8 of the tile
  pdl_trigger();
  pdl_wait();
  float acc[2][2] = {};
  float va[KC / 16], vb[KC / 16];
  sg_load<A_MN, KC>(A, lda, m0, p.M, 0, p.K, va);
  sg_load<B_MN, KC>(B, ldb, n0, p.N, 0, p.K, vb);
  int buf = 0;
  for (int k0 = 0; k0 < p.K; k0 += KC, buf ^= 1) {
    sg_put<A_MN, KC>(sA[buf], va);
    sg_put<B_MN, KC>(sB[buf], vb);
    __syncthreads();                                        // (one barrier a chunk: the other buffer was read before the last one)
    if (k0 + KC < p.K) {
      sg_load<A_MN, KC>(A, lda, m0, p.M, k0 + KC, p.K, va);
      sg_load<B_MN, KC>(B, ldb, n0, p.N, k0 + KC, p.K, vb);
    }
#pragma unroll
    for (int kk = 0; kk < KC / 4; kk += 4) {
      const int k = grp * (KC / 4) + kk;
      float4 a[2], b[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[i] = *reinterpret_cast<const float4*>(&sA[buf][tm + 8 * i][k]);
        b[i] = *reinterpret_cast<const float4*>(&sB[buf][tn + 8 * i][k]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]); acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]); acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
  }
  if (grp > 0) s_part[grp - 1][t] = make_float4(acc[0][0], acc[0][1], acc[1][0], acc[1][1]);
  __syncthreads();
  if (grp > 0) return;
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    const float4 v = s_part[g][t];
    acc[0][0] += v.x; acc[0][1] += v.y; acc[1][0] += v.z; acc[1][1] += v.w;
  }
  const float alpha = p.alpha_ptr ? p.alpha * __ldcg(p.alpha_ptr) : p.alpha;
  const float* bias = reinterpret_cast<const float*>(p.bias);
  float* C = reinterpret_cast<float*>(p.C);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int m = m0 + tm + 8 * i, n = n0 + tn + 8 * j;
      if (m >= p.M || n >= p.N) continue;
      float v = acc[i][j] * alpha;
      if (bias) v += __ldcg(bias + n);
      if (p.act == ACT_RELU) v = v > 0.f ? v : 0.f;
      if (p.out_mode == OUT_F32_ATOMIC) atomicAdd(C + m * p.ldc + n, v); else C[m * p.ldc + n] = v;
    }
}

}  // namespace b200

// C (+)= act(alpha A B^T + bias) for fp32 operands of any leading dimension, one matrix, fp32 result, fp32 or no bias,
// activation none or ReLU.
extern "C" int b200_gemm_small(const b200::GemmArgs* args, cudaStream_t st) {
  using namespace b200;
  const GemmArgs& a = *args;
  const GemmParams& p = a.p;
  if (p.M <= 0 || p.N <= 0) return 0;
  if (a.dtype != GEMM_F32 || p.batch != 1 || p.splits > 1 || (p.out_mode != OUT_F32 && p.out_mode != OUT_F32_ATOMIC) || (p.act != ACT_NONE && p.act != ACT_RELU) ||
      (p.bias && (!p.bias_f32 || p.strideBias)) || p.residual || p.aux_in || p.aux_out || p.row_scale || p.col_scale || p.m_valid || p.k_valid)
    return -3;
  const dim3 grid((p.N + SG_T - 1) / SG_T, (p.M + SG_T - 1) / SG_T), block(256);
  if (grid.y > 65535) return -3;
  const float* A = static_cast<const float*>(a.A); const float* B = static_cast<const float*>(a.B);
  // chunks of 128 halve the exposed load latencies of a long K; K <= 64 would compute on padding (256 x 784 x 32: 3.4 us with
  // chunks of 64, 5.7 with 128; 32 x 256 x 784: 7.8 and 7.1)
  const bool lng = p.K > 128;
  void (*fn)(const float*, long long, const float*, long long, GemmParams) =
      !a.a_mn ? (!a.b_mn ? (lng ? gemm_small_kernel<false, false, 128> : gemm_small_kernel<false, false, 64>)
                         : (lng ? gemm_small_kernel<false, true, 128> : gemm_small_kernel<false, true, 64>))
              : (!a.b_mn ? (lng ? gemm_small_kernel<true, false, 128> : gemm_small_kernel<true, false, 64>)
                         : (lng ? gemm_small_kernel<true, true, 128> : gemm_small_kernel<true, true, 64>));
  cudaError_t e = launch_pdl(fn, grid, block, 0, st, A, a.lda, B, a.ldb, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}
