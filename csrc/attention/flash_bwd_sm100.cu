// A2: FlashAttention backward on tcgen05 / TMEM (sm_100a), causal and non-causal, head_dim 64 / 128.
//
// Gradients of O = softmax(Q K^T * scale) V for an arbitrary upstream dO. (The reference's backward,
// rust-nn src/tensor.rs:1468-1554, assumes a uniform upstream gradient; the oracle here is autograd
// through dense fp32 softmax attention.)
//
// One CTA = one (batch, head, 128-key block), looping over the query blocks that see it. Everything is computed
// transposed (rows = keys), so that P^T can feed dV straight from tensor memory. Per query block:
//   S^T = K Q^T            dP^T = V dO^T                   (K-major x K-major)        -> TMEM
//   P = exp2(S c - lse)    dS = P (dP - delta)             P^T -> TMEM over S^T, dS^T -> one bf16 tile in shared memory
//   dV += P^T dO           dK += dS^T Q                    accumulate in TMEM for the whole loop
//   dQ  = dS K             (MN-major view of the dS^T tile) -> TMEM -> shared memory -> bulk fp32 add in L2
// What bounded the earlier form was its serial chain: all warps waited for S and dP, then the tensor cores waited for all
// warps, and dQ went out as 16-byte atomics to 32 different rows per instruction. Here the roles are separate warps joined
// by mbarriers: one thread issues the products, one warp loads, eight softmax warps (thread = one key x 64 queries) and
// four dQ warps, so that the exponentials of block i+1 run beside dK / dQ of block i. What bounds it now is shared-memory
// bandwidth (operands of the products, dS, the row statistics): P, and for head_dim 64 K and V, are A operands in TMEM,
// and dQ leaves as 8 KB bulk adds in a private layout ([32-row group][hd / 4][32][4]) that the staging stores write without
// bank conflicts (the same layout added from registers, 512 bytes per instruction, was slower: 884 against 737 us below).
// S of the next block is written over the P that dV has just read, and behind it in issue order. The PTX document orders products
// of one accumulator and shape, which these two are not: that the tensor core of a CTA executes one thread's products in issue
// order is an observation (every test and every repeated run agrees), not a promise. A commit and a wait between them would put
// the completion of dV on the chain of every block, which issuing S early is there to shorten.
// Every wait is bounded.
// Measured, kernel alone (B x H x S x hd, causal; earlier form -> this one): 4 x 16 x 4096 x 128 1371 -> 718 us (957 TFLOP/s),
// 4 x 16 x 4096 x 64 769 -> 449 us, 64 x 8 x 1024 x 64 507 -> 355 us; not causal, 16 x 8 x 577 x 64 92 -> 67 us.
#include <algorithm>
#include "../common/ptx.cuh"
#include "../common/launch.cuh"
#include "../common/tensormap.h"
#include "flash_sm100.h"

namespace b200 {

struct BwdParams {
  __nv_bfloat16* dk; long long dk_sb, dk_ss, dk_sh;
  __nv_bfloat16* dv; long long dv_sb, dv_ss, dv_sh;
  __nv_bfloat16* dq; long long dq_sb, dq_ss, dq_sh;      // written here when there is one key block, else by the conversion below
  float* dq_accum;
  const float* lse; const float* delta;
  int B, H, Sq, Skv;
  float scale, scale_log2;
  uint32_t* status;
  int global_order;       // schedule the first key block of ALL heads first (only while the operands of all heads fit L2-ish)
};

// delta[b,h,s] = sum_e dO[b,s,h,e] * O[b,s,h,e]; hd/8 lanes per row, one 16-byte load of each operand per lane. The same
// pass clears the dQ accumulator (`acc4` vectors of four floats). The kernels of this file may be resident before their
// predecessor has finished, so what it wrote is read past L1 (ld.cg), never through the read-only path.
__global__ void flash_delta_kernel(const __nv_bfloat16* o, long long o_sb, long long o_ss, long long o_sh,
                                   const __nv_bfloat16* d, long long d_sb, long long d_ss, long long d_sh,
                                   float* __restrict__ delta, float4* __restrict__ acc, long long acc4, int B, int H, int S, int hd) {
  pdl_trigger();
  pdl_wait();
  const int lpr = hd / 8;                                   // lanes per row: 8 (hd 64) or 16 (hd 128)
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long w = t / lpr;
  const int sub = (int)(t % lpr);
  const long long total = (long long)B * H * S;
  float sum = 0.f;
  // rows are enumerated [b][s][h] so that neighbouring lanes read neighbouring memory
  const int h = (int)(w % H); const long long r = w / H; const int s = (int)(r % S); const int b = (int)(r / S);
  if (w < total) {
    const uint4 a = __ldcg(reinterpret_cast<const uint4*>(o + b * o_sb + s * o_ss + h * o_sh + sub * 8));
    const uint4 c = __ldcg(reinterpret_cast<const uint4*>(d + b * d_sb + s * d_ss + h * d_sh + sub * 8));
    const float2 a0 = unpack_bf16x2(a.x), a1 = unpack_bf16x2(a.y), a2 = unpack_bf16x2(a.z), a3 = unpack_bf16x2(a.w);
    const float2 c0 = unpack_bf16x2(c.x), c1 = unpack_bf16x2(c.y), c2 = unpack_bf16x2(c.z), c3 = unpack_bf16x2(c.w);
    sum = a0.x * c0.x + a0.y * c0.y + a1.x * c1.x + a1.y * c1.y + a2.x * c2.x + a2.y * c2.y + a3.x * c3.x + a3.y * c3.y;
  }
  for (long long i = t; i < acc4; i += (long long)gridDim.x * blockDim.x) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int o2 = lpr >> 1; o2; o2 >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o2);
  if (w < total && sub == 0) delta[((long long)b * H + h) * S + s] = sum;
}

// dq[b,s,h,:] (bf16, strided) = scale * dq_accum. The accumulator is laid out the way the dQ warps hand it over: per (b, h) and
// 32 queries, [hd / 4 column groups][32 rows][4] fp32. A thread converts 16 columns of a row:
// its four reads are 16 bytes beside its neighbours', its write is a whole 32-byte sector.
__global__ void flash_dq_convert_kernel(const float* acc, __nv_bfloat16* __restrict__ dq, long long sb,
                                        long long ss, long long sh, float scale, int B, int S, int H, int hd) {
  pdl_trigger();
  pdl_wait();
  const int groups = hd / 16, parts = (S + 31) / 32;
  const long long total = (long long)B * H * parts * groups * 32;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += stride) {
    const int lane = (int)(i & 31); long long r = i >> 5;
    const int g = (int)(r % groups); r /= groups;              // r: (b, h, 32 queries)
    const long long bh = r / parts;
    const int s = (int)(r % parts) * 32 + lane;
    if (s >= S) continue;
    const float4* src = reinterpret_cast<const float4*>(acc + r * (32 * hd) + g * 512) + lane;
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 v = __ldcg(src + j * 32);
      o[2 * j] = pack_bf16x2(v.x * scale, v.y * scale); o[2 * j + 1] = pack_bf16x2(v.z * scale, v.w * scale);
    }
    uint4* dst = reinterpret_cast<uint4*>(dq + (bh / H) * sb + s * ss + (bh % H) * sh + g * 16);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]); dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
  }
}

// What differs by head_dim. 64 leaves TMEM columns for dQ and for operand copies of K and V (A operands of S and dP, which
// then read only Q and dO from shared memory). 128 fills TMEM with dK and dV: dQ overwrites dP once that has been read.
template <int HD>
struct BwdCfg {
  static constexpr bool ROOM = HD == 64;                   // TMEM has room beside S, dP, dK, dV
  static constexpr int SW = 8;                             // softmax warps
  static constexpr int SC = 128 / (SW / 4);                // query columns per softmax thread
  static constexpr int MMA_W = SW + 4, LOAD_W = SW + 5, STAT_W = SW + 6;     // after 4 dQ warps, one warp each
  static constexpr int THREADS = (SW + 7) * 32;
  static constexpr int TILE = 128 * HD * 2;                // one Q / dO / K / V tile
  static constexpr int Q_ST = HD == 64 ? 3 : 2;            // Q stages: S of block i+1 is wanted before dK of block i-1 is done
  static constexpr int DO_ST = HD == 64 ? 2 : 1;           // dO stages
  static constexpr int DS_ST = HD == 64 ? 2 : 1;           // dS stages
  static constexpr int DS = 128 * 128 * 2;                 // dS^T tile, bf16 [key][query]
  static constexpr int OFF_V = TILE, OFF_Q = 2 * TILE, OFF_DO = OFF_Q + Q_ST * TILE, OFF_DS = OFF_DO + DO_ST * TILE;
  static constexpr int STG = 4 * 8192;                     // dQ staging: 64 columns x 32 rows fp32 per warp
  static constexpr int OFF_STG = OFF_DS + DS_ST * DS, OFF_STAT = OFF_STG + STG, OFF_BAR = OFF_STAT + 4 * 128 * 4;
  static constexpr int SMEM = OFF_BAR + 26 * 8 + 16;
};
static_assert(BwdCfg<64>::SMEM <= 232448 && BwdCfg<128>::SMEM <= 232448, "shared memory of one SM");

template <int HD, bool CAUSAL>
__global__ void __launch_bounds__(BwdCfg<HD>::THREADS, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, BwdParams p) {
  using L = BwdCfg<HD>;
  constexpr int BLK = 128, KA = HD / 64, TILE = L::TILE;
  constexpr int Q_ST = L::Q_ST, DO_ST = L::DO_ST, DS_ST = L::DS_ST, SC = L::SC;
  constexpr bool ROOM = L::ROOM;
  constexpr uint32_t COL_S = 0, COL_DP = 128, COL_DK = 256, COL_DV = 256 + HD;
  constexpr uint32_t COL_DQ = ROOM ? 384 : COL_DP, COL_K = 448, COL_V = 480;        // (K, V copies only with ROOM)

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = smem + L::OFF_V;
  uint8_t* sQ = smem + L::OFF_Q;
  uint8_t* sdO = smem + L::OFF_DO;
  uint8_t* sdS = smem + L::OFF_DS;
  uint8_t* sStg = smem + L::OFF_STG;
  float* sL = reinterpret_cast<float*>(smem + L::OFF_STAT);     // [2][128] -lse in log2 units
  float* sD = sL + 2 * BLK;                                     // [2][128] -delta
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* kv_full = bars;            // 1
  uint64_t* q_full = bars + 1;         // Q_ST
  uint64_t* q_empty = bars + 4;        // Q_ST
  uint64_t* do_full = bars + 7;        // DO_ST
  uint64_t* do_empty = bars + 9;       // DO_ST
  uint64_t* st_full = bars + 11;       // 2: row statistics
  uint64_t* st_empty = bars + 13;      // 2
  uint64_t* s_full = bars + 15;
  uint64_t* kv_tmem = bars + 16;       // ROOM: the operand copies of K and V are in TMEM
  uint64_t* p_ready = bars + 17;
  uint64_t* dp_full = bars + 18;
  uint64_t* ds_ready = bars + 19;
  uint64_t* ds_empty = bars + 20;      // DS_ST
  uint64_t* dq_full = bars + 22;
  uint64_t* dq_empty = bars + 23;
  uint64_t* fin = bars + 24;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  pdl_trigger();
  const int n_kv_blocks = (p.Skv + BLK - 1) / BLK;
  const int m_blocks = (p.Sq + BLK - 1) / BLK;
  const int n_bh = p.B * p.H;
  // early key blocks (most work when causal) first: across all heads while their operands stay in L2, else per head
  const int bid = blockIdx.x;
  const int jb = p.global_order ? bid / n_bh : bid % n_kv_blocks;
  const int bh = p.global_order ? bid % n_bh : bid / n_kv_blocks;
  const int h = bh % p.H, b = bh / p.H;
  const int kv0 = jb * BLK;

  if ((smem_u32(smem) & 1023u) != 0) {
    if (tid == 0 && p.status) atomicCAS(p.status, 0u, (uint32_t)ST_BAD_ARGUMENT);
    return;
  }
  if (tid == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < Q_ST; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); }
    for (int s = 0; s < DO_ST; ++s) { mbar_init(&do_full[s], 1); mbar_init(&do_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&st_full[s], 32); mbar_init(&st_empty[s], L::SW); }
    mbar_init(s_full, 1); mbar_init(kv_tmem, L::SW); mbar_init(p_ready, L::SW); mbar_init(dp_full, 1);
    mbar_init(ds_ready, L::SW); for (int s = 0; s < DS_ST; ++s) mbar_init(&ds_empty[s], 1);
    mbar_init(dq_full, 1); mbar_init(dq_empty, 4); mbar_init(fin, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  const int i_start = CAUSAL ? jb : 0;
  const int n_iter = m_blocks - i_start;

  if (warp < L::SW) {
    // ------------------------------------------------------------------ softmax warps: thread = key row, SC of the queries
    const int quarter = warp & 3, cg = warp >> 2, row = quarter * 32 + lane, col0 = cg * SC;
    const int kv_row = kv0 + row;
    const uint32_t trow = tmem_base + (uint32_t(quarter * 32) << 16);
    const bool key_ok = kv_row < p.Skv;
    // 32 fp32 values -> bf16, into columns col0 + c*32 .. of this thread's row of a [128][128] tile
    auto put32 = [&](uint8_t* base, int c, const float* v) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int ch = (col0 >> 3) + c * 4 + g;                // 16-byte chunk of the row
        *reinterpret_cast<uint4*>(base + (ch >> 3) * (BLK * 128) + sw128_offset(row, ch & 7)) =
            make_uint4(pack_bf16x2(v[g * 8], v[g * 8 + 1]), pack_bf16x2(v[g * 8 + 2], v[g * 8 + 3]),
                       pack_bf16x2(v[g * 8 + 4], v[g * 8 + 5]), pack_bf16x2(v[g * 8 + 6], v[g * 8 + 7]));
      }
    };
    bool ok = true;
    if (ROOM && n_iter > 0) {                                  // the two column groups copy a row of K and of V
      ok = __all_sync(0xffffffffu, mbar_wait(kv_full, 0, p.status, ST_TIMEOUT_TMA_FULL));
      if (ok) {
        const uint8_t* src = cg == 0 ? sK : sV;
        uint32_t w[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 u = *reinterpret_cast<const uint4*>(src + sw128_offset(row, c));
          w[4 * c] = u.x; w[4 * c + 1] = u.y; w[4 * c + 2] = u.z; w[4 * c + 3] = u.w;
        }
        tmem_st_x32(trow + (cg == 0 ? COL_K : COL_V), w);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(kv_tmem);
      }
    }
    for (int it = 0; it < n_iter && ok; ++it) {
      const int st = it & 1;
      const int qc0 = (i_start + it) * BLK + col0;             // first query of this thread's columns
      float pr[SC];
      ok = mbar_wait(&st_full[st], (it >> 1) & 1, p.status, ST_TIMEOUT_GENERIC) && mbar_wait(s_full, it & 1, p.status, ST_TIMEOUT_ACC_FULL);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }               // (also brings the warp together for the TMEM loads)
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < SC / 32; ++c) tmem_ld_x32(trow + COL_S + col0 + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&pr[c * 32]));
      tmem_ld_wait();
      const float* l4 = sL + st * BLK + col0;
#pragma unroll
      for (int e = 0; e < SC; e += 4) {
        const float4 l = *reinterpret_cast<const float4*>(l4 + e);
        fma2_pair(pr[e], pr[e + 1], p.scale_log2, l.x, l.y);
        fma2_pair(pr[e + 2], pr[e + 3], p.scale_log2, l.z, l.w);
        pr[e] = ex2_approx(pr[e]); pr[e + 1] = ex2_approx(pr[e + 1]); pr[e + 2] = ex2_approx(pr[e + 2]); pr[e + 3] = ex2_approx(pr[e + 3]);
      }
      // queries past the end have -lse = -inf, so their P is already zero; keys past the end and later keys are masked here
      if (kv0 + BLK > p.Skv || (CAUSAL && qc0 < kv0 + BLK - 1)) {
        const int first = !key_ok ? SC : CAUSAL ? kv_row - qc0 : 0;            // columns below `first` do not see this key
#pragma unroll
        for (int e = 0; e < SC; ++e) if (e < first) pr[e] = 0.f;
      }
      {
        static_assert(SC == 64, "P of 64 queries is 32 TMEM columns");
        uint32_t pk[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) pk[e] = pack_bf16x2(pr[2 * e], pr[2 * e + 1]);
        tmem_st_x32(trow + COL_S + col0, pk);                  // over the S columns this thread has just read
        tmem_st_wait();
        tc_fence_before_sync();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      ok = mbar_wait(dp_full, it & 1, p.status, ST_TIMEOUT_ACC_FULL) &&
           (it < DS_ST || mbar_wait(&ds_empty[it % DS_ST], ((it / DS_ST) - 1) & 1, p.status, ST_TIMEOUT_TMA_EMPTY));
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc_fence_after_sync();
      const float* d4 = sD + st * BLK + col0;
#pragma unroll
      for (int c = 0; c < SC / 32; ++c) {
        float ds[32];
        tmem_ld_x32(trow + COL_DP + col0 + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&ds[0]));
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const float4 d = *reinterpret_cast<const float4*>(d4 + c * 32 + e);
          add2(ds[e], ds[e + 1], d.x, d.y); add2(ds[e + 2], ds[e + 3], d.z, d.w);
          mul2(ds[e], ds[e + 1], pr[c * 32 + e], pr[c * 32 + e + 1]); mul2(ds[e + 2], ds[e + 3], pr[c * 32 + e + 2], pr[c * 32 + e + 3]);
        }
        put32(sdS + (it % DS_ST) * L::DS, c, ds);
      }
      tc_fence_before_sync();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) { mbar_arrive(ds_ready); mbar_arrive(&st_empty[st]); }
    }
    // dK / dV: TMEM -> bf16 global, HD / (SW / 4) columns per thread
    constexpr int HH = HD / (L::SW / 4);
    __nv_bfloat16* dkp = p.dk + (long long)b * p.dk_sb + (long long)kv_row * p.dk_ss + (long long)h * p.dk_sh + cg * HH;
    __nv_bfloat16* dvp = p.dv + (long long)b * p.dv_sb + (long long)kv_row * p.dv_ss + (long long)h * p.dv_sh + cg * HH;
    if (n_iter <= 0) {                                         // a key block that no query sees: zero gradients
      if (key_ok)
        for (int e = 0; e < HH; e += 8) { *reinterpret_cast<uint4*>(dkp + e) = make_uint4(0, 0, 0, 0); *reinterpret_cast<uint4*>(dvp + e) = make_uint4(0, 0, 0, 0); }
    } else if (ok && __all_sync(0xffffffffu, mbar_wait(fin, 0, p.status, ST_TIMEOUT_ACC_FULL))) {
      tc_fence_after_sync();
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const float sc = w == 0 ? p.scale : 1.f;
        __nv_bfloat16* dst = w == 0 ? dkp : dvp;
        uint32_t v[HH];
#pragma unroll
        for (int c = 0; c < HH / 16; ++c) tmem_ld_x16(trow + (w == 0 ? COL_DK : COL_DV) + cg * HH + c * 16, *reinterpret_cast<uint32_t(*)[16]>(&v[c * 16]));
        tmem_ld_wait();
        if (key_ok) {
#pragma unroll
          for (int e = 0; e < HH; e += 8)
            *reinterpret_cast<uint4*>(dst + e) = make_uint4(
                pack_bf16x2(__uint_as_float(v[e]) * sc, __uint_as_float(v[e + 1]) * sc),
                pack_bf16x2(__uint_as_float(v[e + 2]) * sc, __uint_as_float(v[e + 3]) * sc),
                pack_bf16x2(__uint_as_float(v[e + 4]) * sc, __uint_as_float(v[e + 5]) * sc),
                pack_bf16x2(__uint_as_float(v[e + 6]) * sc, __uint_as_float(v[e + 7]) * sc));
        }
      }
    }
  } else if (warp < L::MMA_W) {
    // ------------------------------------------------------------------ dQ warps: TMEM -> staging -> one bulk add per warp and 64 columns
    const int quarter = warp & 3, parts = (p.Sq + 31) / 32;
    const bool whole = n_kv_blocks == 1;
    const uint32_t trow = tmem_base + (uint32_t(quarter * 32) << 16);
    uint8_t* stg = sStg + quarter * 8192;
    for (int it = 0; it < n_iter; ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(dq_full, it & 1, p.status, ST_TIMEOUT_ACC_FULL))) break;
      tc_fence_after_sync();
      const int part = (i_start + it) * 4 + quarter;           // 32 queries
      if (part >= parts) {                                     // past the end: nothing to add
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(dq_empty);
        continue;
      }
      float* dst = p.dq_accum + ((long long)bh * parts + part) * (32 * HD);
#pragma unroll
      for (int a = 0; a < KA; ++a) {
        uint32_t v[64];
        tmem_ld_x32(trow + COL_DQ + a * 64, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
        tmem_ld_x32(trow + COL_DQ + a * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
        tmem_ld_wait();
        if (a == KA - 1) {                                     // everything is in registers: the columns are free
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(dq_empty);
        }
        if (whole) {                                           // no other block adds to these rows
          const int q = part * 32 + lane;
          if (q < p.Sq) {
            uint4* out = reinterpret_cast<uint4*>(p.dq + (long long)b * p.dq_sb + (long long)q * p.dq_ss + (long long)h * p.dq_sh + a * 64);
#pragma unroll
            for (int e = 0; e < 64; e += 8)
              out[e / 8] = make_uint4(pack_bf16x2(__uint_as_float(v[e]) * p.scale, __uint_as_float(v[e + 1]) * p.scale),
                                      pack_bf16x2(__uint_as_float(v[e + 2]) * p.scale, __uint_as_float(v[e + 3]) * p.scale),
                                      pack_bf16x2(__uint_as_float(v[e + 4]) * p.scale, __uint_as_float(v[e + 5]) * p.scale),
                                      pack_bf16x2(__uint_as_float(v[e + 6]) * p.scale, __uint_as_float(v[e + 7]) * p.scale));
          }
          __syncwarp();
          continue;
        }
        if (lane == 0) tma_store_wait_read0();                 // the staging buffer's previous contents have been read
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 16; ++c)
          *reinterpret_cast<uint4*>(stg + (c * 32 + lane) * 16) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) { bulk_reduce_add_f32(dst + a * 2048, stg, 8192); tma_store_commit(); }
      }
    }
    if (lane == 0) tma_store_wait0();
  } else if (warp == L::MMA_W) {
    // ------------------------------------------------------------------ MMA warp: one thread issues every product
    if (n_iter > 0 && elect_one()) {
      constexpr uint32_t idesc_kk = make_idesc(BLK, BLK, CFMT_F32, FMT_BF16, FMT_BF16, 0, 0);   // S^T, dP^T
      constexpr uint32_t idesc_km = make_idesc(BLK, HD, CFMT_F32, FMT_BF16, FMT_BF16, 0, 1);    // dV, dK
      constexpr uint32_t idesc_mm = make_idesc(BLK, HD, CFMT_F32, FMT_BF16, FMT_BF16, 1, 1);    // dQ
      const uint32_t lK = sdesc_lo(smem_u32(sK), 0), lV = sdesc_lo(smem_u32(sV), 0), mK = sdesc_lo(smem_u32(sK), BLK * 128);
      auto xyT = [&](uint32_t d, uint32_t lx, uint32_t ly) {   // [128 keys][128 queries], both operands K-major
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t adv = (k >> 2) * (BLK * 128) + (k & 3) * 32;
          if (k == 0) umma_f16_c<false>(d, sdesc_at<1024>(lx, adv), sdesc_at<1024>(ly, adv), idesc_kk);
          else umma_f16_c<true>(d, sdesc_at<1024>(lx, adv), sdesc_at<1024>(ly, adv), idesc_kk);
        }
      };
      auto kvT = [&](uint32_t d, uint32_t a, uint32_t ly) {    // the same with the K or V operand from TMEM
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          if (k == 0) umma_f16_ta<false>(d, a + k * 8, sdesc_at<1024>(ly, k * 32), idesc_kk);
          else umma_f16_ta<true>(d, a + k * 8, sdesc_at<1024>(ly, k * 32), idesc_kk);
        }
      };
      auto s_of = [&](int it) {
        const uint32_t lQ = sdesc_lo(smem_u32(sQ + (it % Q_ST) * TILE), 0);
        if constexpr (ROOM) kvT(tmem_base + COL_S, tmem_base + COL_K, lQ); else xyT(tmem_base + COL_S, lK, lQ);
        tc_commit(s_full);
      };
      auto dp_of = [&](int it) {
        const uint32_t ldO = sdesc_lo(smem_u32(sdO + (it % DO_ST) * TILE), 0);
        if constexpr (ROOM) kvT(tmem_base + COL_DP, tmem_base + COL_V, ldO); else xyT(tmem_base + COL_DP, lV, ldO);
        tc_commit(dp_full);
      };
      auto dv_of = [&](int it) {                               // dV += P^T dO: 64 queries of P per 64 columns of S, in the first 32 of them
        const uint32_t m = sdesc_lo(smem_u32(sdO + (it % DO_ST) * TILE), BLK * 128);
#pragma unroll
        for (int k = 0; k < BLK / 16; ++k) {
          const uint32_t a = tmem_base + COL_S + (k >> 2) * 64 + (k & 3) * 8;
          if (k == 0 && it == 0) umma_f16_ta<false>(tmem_base + COL_DV, a, sdesc_at<1024>(m, k * 2048), idesc_km);
          else umma_f16_ta<true>(tmem_base + COL_DV, a, sdesc_at<1024>(m, k * 2048), idesc_km);
        }
      };
      auto dk_of = [&](int it) {                               // dK += dS^T Q
        const uint32_t ld = sdesc_lo(smem_u32(sdS + (it % DS_ST) * L::DS), 0), m = sdesc_lo(smem_u32(sQ + (it % Q_ST) * TILE), BLK * 128);
#pragma unroll
        for (int k = 0; k < BLK / 16; ++k) {
          const uint32_t adv = (k >> 2) * (BLK * 128) + (k & 3) * 32;
          if (k == 0 && it == 0) umma_f16_c<false>(tmem_base + COL_DK, sdesc_at<1024>(ld, adv), sdesc_at<1024>(m, k * 2048), idesc_km);
          else umma_f16_c<true>(tmem_base + COL_DK, sdesc_at<1024>(ld, adv), sdesc_at<1024>(m, k * 2048), idesc_km);
        }
      };
      auto dq_of = [&](int it) {                               // dQ = dS K: dS is the MN-major view of the dS^T tile
        const uint32_t md = sdesc_lo(smem_u32(sdS + (it % DS_ST) * L::DS), BLK * 128);
#pragma unroll
        for (int k = 0; k < BLK / 16; ++k) {
          if (k == 0) umma_f16_c<false>(tmem_base + COL_DQ, sdesc_at<1024>(md, k * 2048), sdesc_at<1024>(mK, k * 2048), idesc_mm);
          else umma_f16_c<true>(tmem_base + COL_DQ, sdesc_at<1024>(md, k * 2048), sdesc_at<1024>(mK, k * 2048), idesc_mm);
        }
        tc_commit(dq_full);
      };
      auto run = [&]() -> bool {
        if (!mbar_wait(kv_full, 0, p.status, ST_TIMEOUT_TMA_FULL) || !mbar_wait(&q_full[0], 0, p.status, ST_TIMEOUT_TMA_FULL)) return false;
        if (ROOM && !mbar_wait(kv_tmem, 0, p.status, ST_TIMEOUT_ACC_EMPTY)) return false;
        tc_fence_after_sync();
        s_of(0);
        if (!mbar_wait(&do_full[0], 0, p.status, ST_TIMEOUT_TMA_FULL)) return false;
        tc_fence_after_sync();
        dp_of(0);
        auto next_s = [&](int it) -> bool {
          if (!mbar_wait(&q_full[it % Q_ST], (it / Q_ST) & 1, p.status, ST_TIMEOUT_TMA_FULL)) return false;
          tc_fence_after_sync();
          s_of(it);
          return true;
        };
        auto next_dp = [&](int it) -> bool {
          if (!mbar_wait(&do_full[it % DO_ST], (it / DO_ST) & 1, p.status, ST_TIMEOUT_TMA_FULL)) return false;
          tc_fence_after_sync();
          dp_of(it);
          return true;
        };
        for (int it = 0; it < n_iter; ++it) {
          const bool more = it + 1 < n_iter;
          if (!mbar_wait(p_ready, it & 1, p.status, ST_TIMEOUT_ACC_EMPTY)) return false;
          tc_fence_after_sync();
          dv_of(it);
          tc_commit(&do_empty[it % DO_ST]);                    // dP and dV of this block were dO's readers
          if (more && !next_s(it + 1)) return false;           // over P of this block, behind dV in issue order (see the top)
          if (!mbar_wait(ds_ready, it & 1, p.status, ST_TIMEOUT_ACC_EMPTY)) return false;
          tc_fence_after_sync();
          if (ROOM) {                                          // dP keeps its own columns: first, it is what the softmax warps wait for
            if (more && !next_dp(it + 1)) return false;
            if (it > 0 && !mbar_wait(dq_empty, (it - 1) & 1, p.status, ST_TIMEOUT_ACC_EMPTY)) return false;
            tc_fence_after_sync();
          }
          dq_of(it);
          dk_of(it);
          tc_commit(&q_empty[it % Q_ST]);
          tc_commit(&ds_empty[it % DS_ST]);
          if (!ROOM && more) {                               // dP takes dQ's columns back
            if (!mbar_wait(dq_empty, it & 1, p.status, ST_TIMEOUT_ACC_EMPTY)) return false;
            if (!next_dp(it + 1)) return false;
          }
        }
        tc_commit(fin);
        return true;
      };
      if (!run()) { tc_commit(fin); mbar_wait(fin, 0, p.status, ST_TIMEOUT_ACC_FULL); }   // after an expired wait: let what was issued finish
    }
  } else if (warp == L::LOAD_W) {
    // ------------------------------------------------------------------ load warp: one thread, tiles by TMA
    if (lane == 0 && n_iter > 0) {
      auto tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int s0) {
#pragma unroll
        for (int a = 0; a < KA; ++a) tma_load_4d(dst + a * (BLK * 128), tm, bar, a * 64, h, s0, b);
      };
      int nq = 0, ndo = 0;                                     // tiles issued
      mbar_expect_tx(kv_full, 2 * TILE);
      tile(sK, &tmK, kv_full, kv0);
      tile(sV, &tmV, kv_full, kv0);
      for (int it = 0; it < n_iter; ++it) {
        const int qs = it % Q_ST, ds = it % DO_ST, q0 = (i_start + it) * BLK;
        if (it >= Q_ST && !mbar_wait(&q_empty[qs], ((it / Q_ST) - 1) & 1, p.status, ST_TIMEOUT_TMA_EMPTY)) break;
        mbar_expect_tx(&q_full[qs], TILE); tile(sQ + qs * TILE, &tmQ, &q_full[qs], q0); ++nq;
        if (it >= DO_ST && !mbar_wait(&do_empty[ds], ((it / DO_ST) - 1) & 1, p.status, ST_TIMEOUT_TMA_EMPTY)) break;
        mbar_expect_tx(&do_full[ds], TILE); tile(sdO + ds * TILE, &tmdO, &do_full[ds], q0); ++ndo;
      }
      // no copy may be in flight when the block leaves, whatever ended the loop: the last tile of each stage has landed
      mbar_wait(kv_full, 0, p.status, ST_TIMEOUT_TMA_FULL);
      for (int i = max(nq - Q_ST, 0); i < nq; ++i) mbar_wait(&q_full[i % Q_ST], (i / Q_ST) & 1, p.status, ST_TIMEOUT_TMA_FULL);
      for (int i = max(ndo - DO_ST, 0); i < ndo; ++i) mbar_wait(&do_full[i % DO_ST], (i / DO_ST) & 1, p.status, ST_TIMEOUT_TMA_FULL);
    }
  } else {
    // ------------------------------------------------------------------ statistics warp: -lse (log2 units) and -delta of a query block
    for (int it = 0; it < n_iter; ++it) {
      const int st = it & 1, q0 = (i_start + it) * BLK;
      float lv[4], dv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int q = q0 + k * 32 + lane;
        const long long idx = (long long)bh * p.Sq + q;
        lv[k] = q < p.Sq ? __ldcg(p.lse + idx) * -1.4426950408889634f : -INFINITY;
        dv[k] = q < p.Sq ? -__ldcg(p.delta + idx) : 0.f;
      }
      if (it >= 2 && !mbar_wait(&st_empty[st], ((it >> 1) - 1) & 1, p.status, ST_TIMEOUT_TMA_EMPTY)) break;
#pragma unroll
      for (int k = 0; k < 4; ++k) { sL[st * BLK + k * 32 + lane] = lv[k]; sD[st * BLK + k * 32 + lane] = dv[k]; }
      mbar_arrive(&st_full[st]);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc_fence_after_sync(); tmem_dealloc(tmem_base, 512); }
}

template <int HD, bool CAUSAL>
static int bwd_set_attr() {
  static bool done = false;
  if (done) return 0;
  constexpr int SMEM = BwdCfg<HD>::SMEM;
  (void)cudaGetLastError();
  if (cudaFuncSetAttribute(flash_bwd_kernel<HD, CAUSAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) return 1;
  done = true;
  return 0;
}

template <int HD, bool CAUSAL>
static int launch_bwd(const FlashArgs& a, cudaStream_t st) {
  CUtensorMap tmQ, tmK, tmV, tmdO;
  const auto BF = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const auto SW = CU_TENSOR_MAP_SWIZZLE_128B;
  if (make_tmap_attn(&tmQ, a.q.ptr, BF, 2, a.hd, a.H, a.Sq, a.B, a.q.sh, a.q.ss, a.q.sb, 64, 128, SW)) return 101;
  if (make_tmap_attn(&tmK, a.k.ptr, BF, 2, a.hd, a.H, a.Skv, a.B, a.k.sh, a.k.ss, a.k.sb, 64, 128, SW)) return 102;
  if (make_tmap_attn(&tmV, a.v.ptr, BF, 2, a.hd, a.H, a.Skv, a.B, a.v.sh, a.v.ss, a.v.sb, 64, 128, SW)) return 103;
  if (make_tmap_attn(&tmdO, a.dout.ptr, BF, 2, a.hd, a.H, a.Sq, a.B, a.dout.sh, a.dout.ss, a.dout.sb, 64, 128, SW)) return 104;
  constexpr int SMEM = BwdCfg<HD>::SMEM;
  auto kfn = flash_bwd_kernel<HD, CAUSAL>;
  if (bwd_set_attr<HD, CAUSAL>()) return 105;
  const long long rows = (long long)a.B * a.H * a.Sq;
  // one key block: its dQ is the whole of it and leaves as bf16, with no accumulator to clear, add to and convert (2048 x 16 x 16 x
  // 128 causal, forward + backward: 2776 -> 2088 us, scratch 2.5 -> 0.5 GB). Else the accumulator covers whole groups of 32 queries.
  const bool whole = a.Skv <= 128;
  if (!whole && !a.dq_accum) return -2;
  const long long acc_rows = whole ? 0 : (long long)a.B * a.H * ((a.Sq + 31) / 32 * 32);
  launch_pdl(flash_delta_kernel, dim3((unsigned)((rows * (a.hd / 8) + 255) / 256)), dim3(256), 0, st,
             (const __nv_bfloat16*)a.o.ptr, a.o.sb, a.o.ss, a.o.sh, (const __nv_bfloat16*)a.dout.ptr, a.dout.sb, a.dout.ss, a.dout.sh,
             a.delta, (float4*)a.dq_accum, acc_rows * (a.hd / 4), a.B, a.H, a.Sq, a.hd);
  BwdParams p;
  p.dk = (__nv_bfloat16*)a.dk.ptr; p.dk_sb = a.dk.sb; p.dk_ss = a.dk.ss; p.dk_sh = a.dk.sh;
  p.dv = (__nv_bfloat16*)a.dv.ptr; p.dv_sb = a.dv.sb; p.dv_ss = a.dv.ss; p.dv_sh = a.dv.sh;
  p.dq = (__nv_bfloat16*)a.dq.ptr; p.dq_sb = a.dq.sb; p.dq_ss = a.dq.ss; p.dq_sh = a.dq.sh;
  p.dq_accum = a.dq_accum; p.lse = a.lse; p.delta = a.delta;
  p.B = a.B; p.H = a.H; p.Sq = a.Sq; p.Skv = a.Skv;
  p.scale = a.scale; p.scale_log2 = a.scale * 1.4426950408889634f; p.status = a.status;
  p.global_order = ((long long)a.B * a.H * ((long long)a.Sq + a.Skv) * a.hd * 4 <= 64ll * 1024 * 1024) ? 1 : 0;
  const long long grid = (long long)((a.Skv + 127) / 128) * a.H * a.B;
  launch_pdl(kfn, dim3((unsigned)grid), dim3(BwdCfg<HD>::THREADS), SMEM, st, tmQ, tmK, tmV, tmdO, p);
  const long long g = std::min<long long>((acc_rows * (a.hd / 16) + 255) / 256, 148 * 16);
  if (!whole) launch_pdl(flash_dq_convert_kernel, dim3((unsigned)g), dim3(256), 0, st, (const float*)a.dq_accum, (__nv_bfloat16*)a.dq.ptr, a.dq.sb, a.dq.ss, a.dq.sh,
             a.scale, a.B, a.Sq, a.H, a.hd);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace b200

extern "C" int b200_flash_bwd_init() {
  using namespace b200;
  return bwd_set_attr<64, true>() | bwd_set_attr<64, false>() | bwd_set_attr<128, true>() | bwd_set_attr<128, false>();
}

extern "C" int b200_flash_bwd(const b200::FlashArgs* a, cudaStream_t st) {
  using namespace b200;
  if (a->B <= 0 || a->H <= 0 || a->Sq <= 0 || a->Skv <= 0) return 0;
  if (a->hd == 64) return a->causal ? launch_bwd<64, true>(*a, st) : launch_bwd<64, false>(*a, st);
  if (a->hd == 128) return a->causal ? launch_bwd<128, true>(*a, st) : launch_bwd<128, false>(*a, st);
  return -3;
}
