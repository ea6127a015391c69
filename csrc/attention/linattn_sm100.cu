// A3 / A4: causal linear attention, forward and backward, as fused chunk kernels on tcgen05 / TMEM (sm_100a).
//
//   out_t = phi(s q_t) . S_t / (phi(s q_t) . z_t + eps),   S_t = sum_{u<=t} phi(s k_u) (x) v_u,   z_t = sum_{u<=t} phi(s k_u)
//
// with phi = ELU + 1 or ReLU^2 (rust-nn src/linear_attention.rs:42-94). The reference runs the causal form as a
// per-token rank-1 recurrence and its backward stores every S_t (src/linear_attention.rs:214-266, 502-632). Here a CTA
// walks the sequence of one (batch, head), or one of `n_seg` segments of it, in chunks of 128 tokens (a token is a TMEM
// lane). Segments first take their totals (`state_only`), a small kernel sums them up, and the pass starts each segment from
// the sum: few heads leave most SMs idle otherwise. Per chunk, with Q~ = phi(sQ), K~ = phi(sK) formed in shared memory in place on the TMA tiles:
//
//   forward     A = mask(Q~ K~^T)            NUM = Q~ S + A V          den = rowsum(A) + Q~ . z        out = NUM / (den + eps)
//               S += K~^T V                  z += colsum(K~)
//   backward 1  (same direction, carries S, z again)      G = dO / D,  dden = -(dO . O) / D
//               dA = mask(G V^T + dden 1^T)  dQ~ = dA K~ + G S^T + dden (x) z
//   backward 2  (reverse direction, carries dS = sum_later Q~^T G and dz = sum_later Q~^T dden)
//               dV = mask(A)^T G + K~ dS     dK~ = mask(dA)^T Q~ + V dS^T + 1 (x) dz
//               dS += Q~^T G                 dz += Q~^T dden
//   then dQ = s phi'(sQ) dQ~, dK = s phi'(sK) dK~ in the epilogue.
//
// Every product is a tcgen05.mma with fp32 accumulation in TMEM. The running state stays in TMEM in fp32 for the whole
// sequence; where it enters a product as an operand it is written to shared memory as TWO bf16 tiles (value and
// rounding remainder) and multiplied twice, so the state contributes ~16 mantissa bits: dQ is a difference of two
// nearly equal terms (G S^T against dden z) and a single bf16 copy of S loses it. z and dz are applied in fp32 by the
// threads. The same natural [d_k][d_v] tile serves as MN-major B operand (x S) and as K-major B operand (x S^T).
// No state is ever stored per token or per chunk: both backward kernels recompute what they need from Q, K, V, dO, O
// and the saved denominators.
//
// What bounds the kernels is the chain of steps in a chunk (features, products, mask, products, results), two CTAs per SM at head size 64 and one at
// 128, not the tensor core (a fifth busy) or memory (half busy). So products that need no features (G V^T, G S^T, V dS^T) are issued before
// the features are formed, the forward forms a chunk's features while the products of the chunk before it run, and a warp reads and
// converts only the 32 x 32 blocks of a masked tile that it keeps. 8 x 16 x 16384 x 64 forward + backward 2272 -> 1989 us (ELU + 1),
// 2258 -> 1749 (ReLU^2, whose features cost less); 4 x 16 x 4096 x 128 765 -> 725 and 756 -> 632 us.
//
// `s_in` / `s_out` (optional) are the state before the first token and after the last one; a sequence-parallel rank
// passes the sum of the lower ranks' states in and hands its own total out. Every wait is bounded (status word).
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "linattn_sm100.h"

namespace b200 {

constexpr int LA_C = 128;                    // tokens per chunk = rows of every product = TMEM lanes
constexpr uint32_t LA_X_LBO = LA_C * 128;    // distance of a tile's 64-column atoms

__device__ __forceinline__ bool la_wait_flag(const uint32_t* f, uint32_t want, long long budget, uint32_t* status) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
    if ((int32_t)(v - want) >= 0) return true;
    if (clock64() - t0 > budget) { if (status) atomicCAS(status, 0u, (uint32_t)ST_TIMEOUT_PEER_FLAG); return false; }
    __nanosleep(64);
  }
}
__device__ __forceinline__ void la_set_flag(uint32_t* f, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(f), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t la_epoch(const LinAttnArgs& p) {
  return (p.sx.role != 0 && p.sx.world > 1) ? *reinterpret_cast<volatile const uint32_t*>(p.sx.words) + 1u : 0u;
}
// Main pass: the state this (batch, head) starts from. Without an exchange that is `fallback` (the caller's s_in / ds_in).
template <int HD>
__device__ __forceinline__ const float* la_consume(const LinAttnArgs& p, int bh, uint32_t epoch, const float* fallback) {
  const LaExchange& x = p.sx;
  if (x.role != 2 || x.world <= 1) return fallback;
  const int lo = x.dir == 0 ? 0 : x.rank + 1, hi = x.dir == 0 ? x.rank : x.world;       // the ranks whose totals flow in
  if (lo >= hi) return nullptr;
  constexpr int ST = HD * HD + HD;
  const int BH = p.B * p.H, tid = threadIdx.x;
  int good = 1;
  if (tid >= lo && tid < hi && !la_wait_flag(x.flags[x.rank] + (size_t)tid * BH + bh, epoch, x.wait_cycles, p.status)) good = 0;
  const bool ok = __syncthreads_and(good) != 0;
  float4* dst = reinterpret_cast<float4*>(x.prefix + (size_t)bh * ST);
  for (int i = tid; i < ST / 4; i += blockDim.x) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = lo; r < hi && ok; ++r) {
      const float4 v = __ldcv(reinterpret_cast<const float4*>(x.state[r] + ((size_t)(epoch & 1u) * BH + bh) * ST) + i);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    dst[i] = acc;
  }
  __threadfence_system();
  __syncthreads();
  if (tid >= lo && tid < hi) la_set_flag(x.acks[tid] + (size_t)x.rank * BH + bh, epoch);        // "I have read your total"
  return x.prefix;
}
// State pass: where this slice's totals go. With an exchange: this rank's symmetric buffer (after the consumers of the
// call two earlier have released it); `la_publish_end` then raises the flags at the consumers.
template <int HD>
__device__ __forceinline__ float* la_publish_begin(const LinAttnArgs& p, int bh, uint32_t epoch, float* fallback) {
  const LaExchange& x = p.sx;
  if (x.role != 1 || x.world <= 1) return fallback;
  constexpr int ST = HD * HD + HD;
  const int BH = p.B * p.H, tid = threadIdx.x;
  const int lo = x.dir == 0 ? x.rank + 1 : 0, hi = x.dir == 0 ? x.world : x.rank;       // the ranks that will read it
  if (tid >= lo && tid < hi) la_wait_flag(x.acks[x.rank] + (size_t)tid * BH + bh, epoch - 2u, x.wait_cycles, p.status);
  __syncthreads();
  return x.state[x.rank] + (size_t)(epoch & 1u) * BH * ST;
}
__device__ __forceinline__ void la_publish_end(const LinAttnArgs& p, int bh, uint32_t epoch) {
  const LaExchange& x = p.sx;
  if (x.role != 1 || x.world <= 1) return;
  const int BH = p.B * p.H, tid = threadIdx.x;
  const int lo = x.dir == 0 ? x.rank + 1 : 0, hi = x.dir == 0 ? x.world : x.rank;
  __threadfence_system();
  __syncthreads();
  if (tid >= lo && tid < hi) la_set_flag(x.flags[tid] + (size_t)x.rank * BH + bh, epoch);
}
// Main pass, last thing: the last CTA to get here advances the call counter.
__device__ __forceinline__ void la_retire(const LinAttnArgs& p, uint32_t epoch) {
  const LaExchange& x = p.sx;
  if (x.role != 2 || x.world <= 1 || threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(x.words + 1, 1u) == gridDim.x - 1) { x.words[1] = 0u; __threadfence(); x.words[0] = epoch; }
}

// The feature maps (KIND 0: ELU + 1, 1: ReLU^2) on pairs. Both sides of ELU + 1 are computed and one is selected: as a branch per element, the
// exponentials of one tile took 2550 cycles. (An overflowing exponential is never the selected side; a NaN is.)
__device__ __forceinline__ float la_exp(float x) { return ex2_approx(x * 1.4426950408889634f); }
template <int KIND>
__device__ __forceinline__ void la_phi2(float& x, float& y, float scale) {
  mul2(x, y, scale, scale);
  if constexpr (KIND == 0) {
    float ex = x, ey = y, px = x, py = y;
    mul2(ex, ey, 1.4426950408889634f, 1.4426950408889634f);
    add2(px, py, 1.f, 1.f);
    ex = ex2_approx(ex); ey = ex2_approx(ey);
    x = x > 0.f ? px : ex; y = y > 0.f ? py : ey;
  } else {
    x = fmaxf(x, 0.f); y = fmaxf(y, 0.f);                 // (0 for a NaN)
    mul2(x, y, x, y);
  }
}
template <int KIND>
__device__ __forceinline__ float la_dphi(float x) {
  if constexpr (KIND == 0) { const float e = la_exp(x); return x > 0.f ? 1.f : e; }
  else return x > 0.f ? 2.f * x : 0.f;
}
// One fp32 row of HD values -> bf16 "value" tile and bf16 "remainder" tile (row = thread), [rows][HD] swizzled atoms
// of `rows` rows each.
template <int HD>
__device__ __forceinline__ void la_write_hilo(uint8_t* hi, uint8_t* lo, int rows, int row, const float* v) {
#pragma unroll
  for (int g = 0; g < HD / 8; ++g) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = v[g * 8 + 2 * j], b = v[g * 8 + 2 * j + 1];
      const __nv_bfloat16 ah = __float2bfloat16_rn(a), bh = __float2bfloat16_rn(b);
      h[j] = pack_bf16x2(__bfloat162float(ah), __bfloat162float(bh));
      l[j] = pack_bf16x2(a - __bfloat162float(ah), b - __bfloat162float(bh));
    }
    const uint32_t off = (g >> 3) * (rows * 128) + sw128_offset(row, g & 7);
    *reinterpret_cast<uint4*>(hi + off) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(lo + off) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

template <int N>
__device__ __forceinline__ void la_tmem_row(uint32_t taddr, float* out) {
#pragma unroll
  for (int c = 0; c < N / 32; ++c) tmem_ld_x32(taddr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&out[c * 32]));
  tmem_ld_wait();
}

// ---- MMA issue helpers (one thread). All tiles: atoms of 64 columns, 128-byte rows, 128-byte swizzle.
// D[128 x 128] = X Y^T, both operands K-major [128][HD]
template <int HD>
__device__ __forceinline__ void la_mma_xyT(uint32_t d, const uint8_t* x, const uint8_t* y) {
  constexpr uint32_t idesc = make_idesc(128, 128, CFMT_F32, FMT_BF16, FMT_BF16, 0, 0);
  const uint32_t lx = sdesc_lo(smem_u32(x), 0), ly = sdesc_lo(smem_u32(y), 0);
#pragma unroll
  for (int k = 0; k < HD / 16; ++k) {
    const uint32_t adv = (k >> 2) * (LA_C * 128) + (k & 3) * 32;
    umma_f16(d, sdesc_at<1024>(lx, adv), sdesc_at<1024>(ly, adv), idesc, k > 0);
  }
}
// D[128 x HD] (+)= P W with P K-major [128][KT] (KT = 128 tokens or HD) and W MN-major: [KT rows][HD], atoms `w_lbo` apart
template <int HD, int KT>
__device__ __forceinline__ void la_mma_pw(uint32_t d, const uint8_t* p, const uint8_t* w, uint32_t w_lbo, bool acc) {
  constexpr uint32_t idesc = make_idesc(128, HD, CFMT_F32, FMT_BF16, FMT_BF16, 0, 1);
  const uint32_t lp = sdesc_lo(smem_u32(p), 0), lw = sdesc_lo(smem_u32(w), w_lbo);
#pragma unroll
  for (int k = 0; k < KT / 16; ++k) {
    const uint32_t advp = (k >> 2) * (LA_C * 128) + (k & 3) * 32;
    umma_f16(d, sdesc_at<1024>(lp, advp), sdesc_at<1024>(lw, k * 2048), idesc, acc || k > 0);
  }
}
// D[128 x HD] += P W over 128 tokens, P in TMEM as `la_put_half128` leaves it (`a`: its first column, + 32 for the remainders)
template <int HD>
__device__ __forceinline__ void la_mma_tw(uint32_t d, uint32_t a, const uint8_t* w) {
  constexpr uint32_t idesc = make_idesc(128, HD, CFMT_F32, FMT_BF16, FMT_BF16, 0, 1);
  const uint32_t lw = sdesc_lo(smem_u32(w), LA_C * 128);
#pragma unroll
  for (int k = 0; k < LA_C / 16; ++k) umma_f16_ta<true>(d, a + (k >> 2) * 64 + (k & 3) * 8, sdesc_at<1024>(lw, k * 2048), idesc);
}
// D[128 x HD] (+)= X W^T with X K-major [128][HD] and W K-major [HD rows][HD] (atoms of HD rows)
template <int HD>
__device__ __forceinline__ void la_mma_xwT(uint32_t d, const uint8_t* x, const uint8_t* w, bool acc) {
  constexpr uint32_t idesc = make_idesc(128, HD, CFMT_F32, FMT_BF16, FMT_BF16, 0, 0);
  const uint32_t lx = sdesc_lo(smem_u32(x), 0), lw = sdesc_lo(smem_u32(w), 0);
#pragma unroll
  for (int k = 0; k < HD / 16; ++k) {
    const uint32_t advx = (k >> 2) * (LA_C * 128) + (k & 3) * 32, advw = (k >> 2) * (HD * 128) + (k & 3) * 32;
    umma_f16(d, sdesc_at<1024>(lx, advx), sdesc_at<1024>(lw, advw), idesc, acc || k > 0);
  }
}
// State update D[128 (d_k, zero-padded) x HD] (+)= X^T W over the 128 tokens: X, W MN-major [128 tokens][HD].
// For HD = 64 X's second 64-column atom is the tile behind it (see LaSmem): rows 64..127 of D are not used.
template <int HD>
__device__ __forceinline__ void la_mma_xTw(uint32_t d, const uint8_t* x, const uint8_t* w, bool acc) {
  constexpr uint32_t idesc = make_idesc(128, HD, CFMT_F32, FMT_BF16, FMT_BF16, 1, 1);
  const uint32_t lx = sdesc_lo(smem_u32(x), LA_X_LBO), lw = sdesc_lo(smem_u32(w), LA_C * 128);
#pragma unroll
  for (int k = 0; k < LA_C / 16; ++k)
    umma_f16(d, sdesc_at<1024>(lx, k * 2048), sdesc_at<1024>(lw, k * 2048), idesc, acc || k > 0);
}

template <int HD>
struct LaSmem {
  static constexpr int TILE = LA_C * HD * 2;          // one [128][HD] operand tile
  static constexpr int ST = HD * HD * 2;              // one state tile [HD][HD]
  // Head size 64: 80 KB of tiles and 256 TMEM columns, so that two CTAs share an SM and one's elementwise work runs beside
  // the other's products and waits. The state update wants 128 rows where there are 64: its second 64-row atom is whatever
  // tile follows in shared memory, and rows 64..127 of the result are never read.
  static constexpr uint32_t TMEM = HD == 64 ? 256 : 512;
  static constexpr int CTAS = HD == 64 ? 2 : 1;
};

// ---------------------------------------------------------------------------------------------------- forward
// Thread mapping of the forward kernel: 8 warps. Warp w owns tile rows / TMEM lanes 32 (w & 3) .. + 31 (the lanes a warp
// may read) and column half w >> 2 of every row, so the elementwise work of a chunk is spread over twice the warps of a
// row-per-thread mapping and every scheduler has two warps to switch between (the kernel is bound by instruction
// latency, not by the tensor core: 4 k instructions per chunk and thread at ~5 cycles each with one warp per scheduler).
constexpr int LA_FWD_THREADS = 256;

// phi(scale * x) in place on this thread's half of its row (4 of the 8 16-byte chunks of every 64-column atom)
template <int HD, int KIND>
__device__ __forceinline__ void la_phi_half(uint8_t* tile, int row, int hf, int valid, float scale) {
#pragma unroll
  for (int a = 0; a < HD / 64; ++a)
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) {
      const int c = hf * 4 + c4;
      uint4* p = reinterpret_cast<uint4*>(tile + a * (LA_C * 128) + sw128_offset(row, c));
      uint4 u = *p;
      uint32_t* w = &u.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f = unpack_bf16x2(w[j]);
        la_phi2<KIND>(f.x, f.y, scale);
        w[j] = row < valid ? pack_bf16x2(f.x, f.y) : 0u;
      }
      *p = u;
    }
}
// this thread's half of (row . z)
template <int HD>
__device__ __forceinline__ float la_dot_half(const uint8_t* tile, int row, int hf, const float* z) {
  float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
  for (int a = 0; a < HD / 64; ++a)
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) {
      const int c = hf * 4 + c4;
      const uint4 u = *reinterpret_cast<const uint4*>(tile + a * (LA_C * 128) + sw128_offset(row, c));
      const uint32_t* w = &u.x;
      const float* zz = z + a * 64 + c * 8;
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(w[j]); acc0 = fmaf(f.x, zz[2 * j], acc0); acc1 = fmaf(f.y, zz[2 * j + 1], acc1); }
    }
  return acc0 + acc1;
}
// Columns 64 hf .. of this thread's row of a [128][128] fp32 tile in TMEM, masked, -> A operand over the same columns (`col` = 64 hf of the tile):
// the bf16 values in the first 32, the rounding remainders (REM) in the next 32. The masked tile enters its product as value + remainder like
// the state does where the result is a difference of nearly equal sums (one bf16 copy costs dQ ~2 %). A warp's 32 rows meet a 32-column
// block wholly kept, wholly dropped (not even read) or on the diagonal: LOWER keeps columns <= row, else columns >= row. `f(i, x)` gives the
// value that column 64 hf + i, which held x, enters with; `g` is given the pairs that are kept.
template <bool LOWER, bool REM, typename F, typename G>
__device__ __forceinline__ void la_mask_put(uint32_t col, int quad, int hf, int lane, F f, G g) {
  const int d0 = LOWER ? 2 * hf - quad : quad - 2 * hf, d1 = LOWER ? d0 + 1 : d0 - 1;       // < 0 kept, 0 diagonal, > 0 dropped
  // The remainders of the first block lie over the second: both are read first. Without remainders one after the other, in half the registers
  uint32_t v[REM ? 64 : 32];
  if constexpr (REM) {
    if (d0 <= 0) tmem_ld_x32(col, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
    if (d1 <= 0) tmem_ld_x32(col + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
    tmem_ld_wait();
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int d = k == 0 ? d0 : d1;
    uint32_t h[16], l[16];
    if (d > 0) {
#pragma unroll
      for (int i = 0; i < 16; ++i) h[i] = l[i] = 0u;
    } else {
      constexpr int V1 = REM ? 32 : 0;
      if constexpr (!REM) { tmem_ld_x32(col + 32 * k, *reinterpret_cast<uint32_t(*)[32]>(&v[0])); tmem_ld_wait(); }
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float x = f(32 * k + i, __uint_as_float(v[V1 * k + i])), y = f(32 * k + i + 1, __uint_as_float(v[V1 * k + i + 1]));
        if (d == 0) {
          if (LOWER ? i > lane : i < lane) x = 0.f;
          if (LOWER ? i + 1 > lane : i + 1 < lane) y = 0.f;
        }
        g(x, y);
        h[i / 2] = pack_bf16x2(x, y);
        if constexpr (REM) { const float2 r = unpack_bf16x2(h[i / 2]); l[i / 2] = pack_bf16x2(x - r.x, y - r.y); }
      }
    }
    tmem_st_x16(col + 16 * k, h);
    if constexpr (REM) tmem_st_x16(col + 32 + 16 * k, l);
  }
  tmem_st_wait();
}
// HD / 2 fp32 values = columns (HD / 2) hf .. of a state row -> value and remainder tiles ([rows][HD], atoms of `rows` rows)
template <int HD>
__device__ __forceinline__ void la_write_hilo_half(uint8_t* hi, uint8_t* lo, int rows, int row, int hf, const float* v) {
#pragma unroll
  for (int gg = 0; gg < HD / 16; ++gg) {
    const int g = hf * (HD / 16) + gg;
    uint32_t h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a = v[gg * 8 + 2 * j], b = v[gg * 8 + 2 * j + 1];
      h[j] = pack_bf16x2(a, b);
      const float2 r = unpack_bf16x2(h[j]);
      l[j] = pack_bf16x2(a - r.x, b - r.y);
    }
    const uint32_t off = (g >> 3) * (rows * 128) + sw128_offset(row, g & 7);
    *reinterpret_cast<uint4*>(hi + off) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(lo + off) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}
// partial column sum: rows [r0, r0 + n) of column k
__device__ __forceinline__ float la_colsum_rows(const uint8_t* tile, int k, int r0, int n) {
  const uint8_t* base = tile + (k >> 6) * (LA_C * 128) + (k & 7) * 2;
  const int chunk = (k & 63) >> 3;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 4
  for (int r = r0; r < r0 + n; r += 4) {
    s0 += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r, chunk)));
    s1 += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r + 1, chunk)));
    s2 += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r + 2, chunk)));
    s3 += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r + 3, chunk)));
  }
  return (s0 + s1) + (s2 + s3);
}

// 16-byte piece `i` (of HD / 16) of this thread's half row in a swizzled [128][HD] tile
template <int HD>
__device__ __forceinline__ uint4* la_half_piece(uint8_t* tile, int row, int hf, int i) {
  const int c = hf * (HD / 16) + i;
  return reinterpret_cast<uint4*>(tile + (c >> 3) * (LA_C * 128) + sw128_offset(row, c & 7));
}
// a finished [128][HD] tile to global memory (one thread; tokens past the end are clipped by the tensor map)
template <int HD>
__device__ __forceinline__ void la_store_tile(const CUtensorMap* tm, const uint8_t* tile, int h, int tok0, int b) {
#pragma unroll
  for (int a = 0; a < HD / 64; ++a) tma_store_4d(tm, tile + a * (LA_C * 128), a * 64, h, tok0, b);
}
template <int HD, int KIND>
__global__ void __launch_bounds__(LA_FWD_THREADS, LaSmem<HD>::CTAS)
linattn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmLo, const LinAttnArgs p) {
  using L = LaSmem<HD>;
  constexpr int KA = HD / 64;
  constexpr int HH = HD / 2;                  // columns of a HD-wide row per thread
  constexpr int ZP = LA_FWD_THREADS / HD;     // row groups of the column sums of K~ (4 or 2)
  constexpr uint32_t COL_A = 0, COL_NUM = 128, COL_S = 128 + HD;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + L::TILE;                 // 2 stages
  uint8_t* sV = sK + 2 * L::TILE;
  uint8_t* sShi = sV + L::TILE;
  uint8_t* sSlo = sShi + L::ST;
  float* sz = reinterpret_cast<float*>(sSlo + L::ST);               // [HD]
  float* s_part = sz + HD;                    // [2][128]: the halves' shares of a row's denominator
  float* s_zk = s_part + 2 * LA_C;            // [ZP][HD]: partial column sums of K~
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_zk + LA_FWD_THREADS);
  uint64_t* q_bar = bars; uint64_t* k_bar = bars + 1; uint64_t* v_bar = bars + 3; uint64_t* a_bar = bars + 4; uint64_t* b_bar = bars + 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int quad = warp & 3, hf = warp >> 2, row = quad * 32 + lane;
  const int bh = blockIdx.x / p.n_seg, seg = blockIdx.x % p.n_seg, b = bh / p.H, h = bh % p.H;
  const int c0 = seg * p.seg_chunks;           // first chunk of this CTA's segment
  const int n_chunks = min(p.seg_chunks, (p.S + LA_C - 1) / LA_C - c0);
  const bool full = !p.state_only;
  if (p.n_seg > 1 && !full && seg == p.n_seg - 1) return;      // nothing follows the last segment
  // ELU + 1 features sit near 1, where a bf16 copy of the masked tile loses what the later subtraction needs; ReLU^2
  // features are spread over the exponent range and a single copy is enough (0.3 % measured)
  constexpr bool rem = KIND == 0;
  if ((smem_u32(smem) & 1023u) != 0) { if (tid == 0 && p.status) atomicCAS(p.status, 0u, (uint32_t)ST_BAD_ARGUMENT); return; }
  if (tid == 0) {
    mbar_init(q_bar, 1); mbar_init(&k_bar[0], 1); mbar_init(&k_bar[1], 1); mbar_init(v_bar, 1); mbar_init(a_bar, 1); mbar_init(b_bar, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, L::TMEM); tmem_relinquish(); }
  // state before the first token: TMEM (fp32) and the two bf16 operand tiles
  const size_t st_stride = (size_t)HD * HD + HD;
  const uint32_t sx_epoch = la_epoch(p);
  const float* s_in = la_consume<HD>(p, bh, sx_epoch, p.s_in);       // the caller's state, or the lower ranks' totals
  if (tid < HD) {
    float s0[HD];
#pragma unroll
    for (int i = 0; i < HD; ++i) s0[i] = s_in ? s_in[blockIdx.x * st_stride + (size_t)tid * HD + i] : 0.f;
    la_write_hilo<HD>(sShi, sSlo, HD, tid, s0);
    sz[tid] = s_in ? s_in[blockIdx.x * st_stride + (size_t)HD * HD + tid] : 0.f;
  }
  tc_fence_before_sync();
  fence_proxy_async_smem();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t trow = tmem_base + (uint32_t(quad * 32) << 16);
  if (s_in && hf == 0) {                             // TMEM accesses are warp-wide: every lane stores (rows >= HD: zeros)
#pragma unroll
    for (int c = 0; c < HD / 32; ++c) {
      uint32_t r[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = row < HD ? __float_as_uint(s_in[blockIdx.x * st_stride + (size_t)row * HD + c * 32 + i]) : 0u;
      tmem_st_x32(trow + COL_S + c * 32, r);
    }
    tmem_st_wait();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();

  auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int chunk) {
    mbar_expect_tx(bar, L::TILE);
#pragma unroll
    for (int a = 0; a < KA; ++a) tma_load_4d(dst + a * (LA_C * 128), tm, bar, a * 64, h, (c0 + chunk) * LA_C, b);
  };
  if (tid == 0) {
    if (full) load(sQ, &tmQ, q_bar, 0);
    load(sK, &tmK, &k_bar[0], 0);
    load(sV, &tmV, v_bar, 0);
    if (n_chunks > 1) load(sK + L::TILE, &tmK, &k_bar[1], 1);
  }
  bool ok = true;
  const bool have_state0 = s_in != nullptr;
  // The features of a chunk are formed one chunk ahead, while the products of the chunk before it run
  auto phi = [&](int c) {
    if (full && !mbar_wait(q_bar, c & 1, p.status, ST_TIMEOUT_TMA_FULL)) ok = false;
    if (ok && !mbar_wait(&k_bar[c & 1], (c >> 1) & 1, p.status, ST_TIMEOUT_TMA_FULL)) ok = false;
    if (full) la_phi_half<HD, KIND>(sQ, row, hf, LA_C, p.scale);
    la_phi_half<HD, KIND>(sK + (c & 1) * L::TILE, row, hf, min(LA_C, p.S - (c0 + c) * LA_C), p.scale);
    fence_proxy_async_smem();
  };
  phi(0);
  if (__syncthreads_or(!ok)) ok = false;
  for (int c = 0; c < n_chunks && ok; ++c) {
    const int st = c & 1;
    uint8_t* sKc = sK + st * L::TILE;
    float den = p.eps;
    if (full) {
      if (warp == 0 && elect_one()) {
        tc_fence_after_sync();
        la_mma_xyT<HD>(tmem_base + COL_A, sQ, sKc);                                   // A = Q~ K~^T
        la_mma_pw<HD, HD>(tmem_base + COL_NUM, sQ, sShi, HD * 128, false);            // NUM = Q~ S (value + remainder)
        la_mma_pw<HD, HD>(tmem_base + COL_NUM, sQ, sSlo, HD * 128, true);
        tc_commit(a_bar);                                                             // covers every reader of Q~
      }
      // this half's share of Q~ . z in fp32 while the tensor core works
      float part = la_dot_half<HD>(sQ, row, hf, sz);
      if (!mbar_wait(a_bar, c & 1, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;
      if (__syncthreads_or(!ok)) { ok = false; break; }
      tc_fence_after_sync();
      if (tid == 0 && c + 1 < n_chunks) load(sQ, &tmQ, q_bar, c + 1);            // Q~ has been consumed
      float r0 = 0.f, r1 = 0.f;
      la_mask_put<true, rem>(trow + COL_A + hf * 64, quad, hf, lane, [](int, float x) { return x; }, [&](float x, float y) { add2(r0, r1, x, y); });
      s_part[hf * LA_C + row] = part + (r0 + r1);
      tc_fence_before_sync();
    }
    __syncthreads();
    if (full) den += s_part[row] + s_part[LA_C + row];        // both halves add in the same order
    if (warp == 0 && elect_one()) {
      ok = mbar_wait(v_bar, c & 1, p.status, ST_TIMEOUT_TMA_FULL);
      if (ok) {
        tc_fence_after_sync();
        if (full) {                                                                                    // NUM += A V (value + remainder)
          la_mma_tw<HD>(tmem_base + COL_NUM, tmem_base + COL_A, sV);
          if (rem) la_mma_tw<HD>(tmem_base + COL_NUM, tmem_base + COL_A + 32, sV);
        }
        la_mma_xTw<HD>(tmem_base + COL_S, sKc, sV, have_state0 || c > 0);                   // S += K~^T V
        tc_commit(b_bar);
      }
    }
    // z += colsum(K~) while the products run: ZP row groups per column, combined after the barrier below
    s_zk[tid] = la_colsum_rows(sKc, tid % HD, (tid / HD) * (LA_C / ZP), LA_C / ZP);
    if (c + 1 < n_chunks) phi(c + 1);
    if (!mbar_wait(b_bar, c & 1, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc_fence_after_sync();
    if (tid == 0 && !full) {                                                  // K~ and V of this chunk are free
      if (c + 1 < n_chunks) load(sV, &tmV, v_bar, c + 1);
      if (c + 2 < n_chunks) load(sKc, &tmK, &k_bar[st], c + 2);
    }
    if (full) {
      float num[HH];
      la_tmem_row<HH>(trow + COL_NUM + hf * HH, num);
      const int tok = (c0 + c) * LA_C + row;
      const float inv = 1.f / den;
      // O and its remainder leave as tiles: through V's and K~'s buffers, which this chunk is done with
#pragma unroll
      for (int i = 0; i < HH; i += 8) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float x = num[i + 2 * j] * inv, y = num[i + 2 * j + 1] * inv;
          hi[j] = pack_bf16x2(x, y);
          const float2 r = unpack_bf16x2(hi[j]);
          lo[j] = pack_bf16x2(x - r.x, y - r.y);
        }
        *la_half_piece<HD>(sV, row, hf, i / 8) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (p.o_lo.ptr) *la_half_piece<HD>(sKc, row, hf, i / 8) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      if (tok < p.S && p.den && hf == 0) p.den[((long long)b * p.H + h) * p.S + tok] = den;
    }
    if (tid < HD) {
      float zk = 0.f;
#pragma unroll
      for (int g = 0; g < ZP; ++g) zk += s_zk[g * HD + tid];
      sz[tid] += zk;
    }
    if (full && c + 1 < n_chunks && quad * 32 < HD) {                         // operand copies of the new state (warps that own state rows)
      float srow[HH];
      la_tmem_row<HH>(trow + COL_S + hf * HH, srow);
      if (row < HD) la_write_hilo_half<HD>(sShi, sSlo, HD, row, hf, srow);
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (full && tid == 0) {
      la_store_tile<HD>(&tmO, sV, h, (c0 + c) * LA_C, b);
      if (p.o_lo.ptr) la_store_tile<HD>(&tmLo, sKc, h, (c0 + c) * LA_C, b);
      tma_store_commit();
      if (c + 1 < n_chunks) {
        tma_store_wait_read0();
        load(sV, &tmV, v_bar, c + 1);
        if (c + 2 < n_chunks) load(sKc, &tmK, &k_bar[st], c + 2);
      }
    }
  }
  if (tid == 0) tma_store_wait0();
  float* s_out = la_publish_begin<HD>(p, bh, sx_epoch, p.s_out);      // the caller's buffer, or this rank's slot of the exchange
  const size_t out_idx = full ? bh : blockIdx.x;
  if (ok && s_out && hf == 0 && (!full || seg == p.n_seg - 1)) {
    tc_fence_after_sync();
    float srow[HD];
    la_tmem_row<HD>(trow + COL_S, srow);
    if (row < HD) {
#pragma unroll
      for (int i = 0; i < HD; i += 4)
        *reinterpret_cast<float4*>(s_out + out_idx * st_stride + (size_t)row * HD + i) = make_float4(srow[i], srow[i + 1], srow[i + 2], srow[i + 3]);
      s_out[out_idx * st_stride + (size_t)HD * HD + row] = sz[row];
    }
  }
  la_publish_end(p, bh, sx_epoch);
  la_retire(p, sx_epoch);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc_fence_after_sync(); tmem_dealloc(tmem_base, L::TMEM); }
}

// ---------------------------------------------------------------------------------------------------- backward helpers (8 warps)
// G = dO / D (bf16) and dden = -(G . O) per token, once for both gradient kernels and their state pass: formed inside them,
// the three dependent loads cost each chunk 5500 of its 16500 cycles; as a tile G is a TMA load that is under way early.
// hd / 8 lanes share a token; tokens are enumerated [b][s][h] so that neighbouring lanes read neighbouring memory.
__global__ void la_g_kernel(const LinAttnArgs p) {
  const int lpr = p.hd / 8;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long w = t / lpr;
  const int sub = (int)(t % lpr);
  const bool ok = w < (long long)p.B * p.H * p.S;
  const int h = (int)(w % p.H); const long long q = w / p.H; const int s = (int)(q % p.S); const int b = (int)(q / p.S);
  const long long idx = ((long long)b * p.H + h) * p.S + s;
  float dot = 0.f;
  if (ok) {
    auto at = [&](const AttnTensor& x) { return reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(x.ptr) + b * x.sb + s * x.ss + h * x.sh + sub * 8); };
    const uint4 du = *at(p.dout), ou = *at(p.o), lu = p.o_lo.ptr ? *at(p.o_lo) : make_uint4(0, 0, 0, 0);
    const float inv = 1.f / p.den[idx];
    const uint32_t* dw = &du.x; const uint32_t* ow = &ou.x; const uint32_t* lw = &lu.x;
    uint32_t g[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 d2 = unpack_bf16x2(dw[j]), o2 = unpack_bf16x2(ow[j]), l2 = unpack_bf16x2(lw[j]);
      // the SAME rounded G enters G V^T on the tensor core and the dot product here, so that the two halves of
      // dA = G . (V_s - O_t) see one dO; O carries its remainder
      g[j] = pack_bf16x2(d2.x * inv, d2.y * inv);
      const float2 gr = unpack_bf16x2(g[j]);
      dot = fmaf(gr.x, o2.x + l2.x, dot); dot = fmaf(gr.y, o2.y + l2.y, dot);
    }
    *at(p.g) = make_uint4(g[0], g[1], g[2], g[3]);
  }
  for (int o = lpr >> 1; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (ok && sub == 0) p.dden[idx] = -dot;
}
// scale * phi'(scale * x) * grad for this thread's half of a token, x the raw (bf16) row in the tile `x`, as bf16 into `dst`
template <int HD, int KIND>
__device__ __forceinline__ void la_put_dphi_half(uint8_t* x, uint8_t* dst, int row, int hf, const float* grad, float scale) {
#pragma unroll
  for (int i = 0; i < HD / 16; ++i) {
    const uint4 xu = *la_half_piece<HD>(x, row, hf, i);
    const uint32_t* xw = &xu.x;
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x2 = unpack_bf16x2(xw[j]);
      const float a = x2.x * scale, c = x2.y * scale;
      const float da = la_dphi<KIND>(a), dc = la_dphi<KIND>(c);
      o[j] = pack_bf16x2(grad[i * 8 + 2 * j] * da * scale, grad[i * 8 + 2 * j + 1] * dc * scale);
    }
    *la_half_piece<HD>(dst, row, hf, i) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}
// partial weighted column sum: sum over rows [r0, r0 + n) of w[r] * tile(r, k)
__device__ __forceinline__ float la_colsum_w_rows(const uint8_t* tile, int k, const float* w, int r0, int n) {
  const uint8_t* base = tile + (k >> 6) * (LA_C * 128) + (k & 7) * 2;
  const int chunk = (k & 63) >> 3;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 4
  for (int r = r0; r < r0 + n; r += 4) {
    s0 = fmaf(w[r], __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r, chunk))), s0);
    s1 = fmaf(w[r + 1], __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r + 1, chunk))), s1);
    s2 = fmaf(w[r + 2], __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r + 2, chunk))), s2);
    s3 = fmaf(w[r + 3], __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + sw128_offset(r + 3, chunk))), s3);
  }
  return (s0 + s1) + (s2 + s3);
}

// ---------------------------------------------------------------------------------------------------- backward 1: dQ
// Same 8-warp mapping as the forward: warp w owns rows 32 (w & 3) .. and column half w >> 2.
template <int HD, int KIND>
__global__ void __launch_bounds__(LA_FWD_THREADS, LaSmem<HD>::CTAS)
linattn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                      const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CUtensorMap tmDQ, const LinAttnArgs p) {
  using L = LaSmem<HD>;
  constexpr int KA = HD / 64;
  constexpr int HH = HD / 2;
  constexpr int ZP = LA_FWD_THREADS / HD;
  constexpr uint32_t COL_A = 0, COL_DQ = 128, COL_S = 128 + HD;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sG = smem;
  uint8_t* sK = sG + L::TILE;                 // 2 stages
  uint8_t* sV = sK + 2 * L::TILE;
  uint8_t* sQr = sV + L::TILE;                // raw Q: phi' needs it
  uint8_t* sShi = sQr + L::TILE;
  uint8_t* sSlo = sShi + L::ST;
  float* sz = reinterpret_cast<float*>(sSlo + L::ST);
  float* s_zk = sz + HD;                      // [256]: partial column sums of K~
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_zk + LA_FWD_THREADS);
  uint64_t* k_bar = bars; uint64_t* v_bar = bars + 2; uint64_t* a_bar = bars + 3; uint64_t* b_bar = bars + 4; uint64_t* q_bar = bars + 5; uint64_t* g_bar = bars + 6;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 7);

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int quad = warp & 3, hf = warp >> 2, row = quad * 32 + lane;
  const int bh = blockIdx.x / p.n_seg, seg = blockIdx.x % p.n_seg, b = bh / p.H, h = bh % p.H;
  const int c0 = seg * p.seg_chunks;           // first chunk of this CTA's segment
  const int n_chunks = min(p.seg_chunks, (p.S + LA_C - 1) / LA_C - c0);
  constexpr bool rem = KIND == 0;              // see the forward kernel
  if ((smem_u32(smem) & 1023u) != 0) { if (tid == 0 && p.status) atomicCAS(p.status, 0u, (uint32_t)ST_BAD_ARGUMENT); return; }
  if (tid == 0) {
    mbar_init(&k_bar[0], 1); mbar_init(&k_bar[1], 1); mbar_init(v_bar, 1); mbar_init(a_bar, 1); mbar_init(b_bar, 1); mbar_init(q_bar, 1); mbar_init(g_bar, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, L::TMEM); tmem_relinquish(); }
  const size_t st_stride = (size_t)HD * HD + HD;
  if (tid < HD) {
    float s0[HD];
#pragma unroll
    for (int i = 0; i < HD; ++i) s0[i] = p.s_in ? p.s_in[blockIdx.x * st_stride + (size_t)tid * HD + i] : 0.f;
    la_write_hilo<HD>(sShi, sSlo, HD, tid, s0);
    sz[tid] = p.s_in ? p.s_in[blockIdx.x * st_stride + (size_t)HD * HD + tid] : 0.f;
  }
  tc_fence_before_sync();
  fence_proxy_async_smem();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t trow = tmem_base + (uint32_t(quad * 32) << 16);
  if (p.s_in && hf == 0) {
#pragma unroll
    for (int c = 0; c < HD / 32; ++c) {
      uint32_t r[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = row < HD ? __float_as_uint(p.s_in[blockIdx.x * st_stride + (size_t)row * HD + c * 32 + i]) : 0u;
      tmem_st_x32(trow + COL_S + c * 32, r);
    }
    tmem_st_wait();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();

  auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int chunk) {
    mbar_expect_tx(bar, L::TILE);
#pragma unroll
    for (int a = 0; a < KA; ++a) tma_load_4d(dst + a * (LA_C * 128), tm, bar, a * 64, h, (c0 + chunk) * LA_C, b);
  };
  if (tid == 0) {
    load(sK, &tmK, &k_bar[0], 0);
    load(sV, &tmV, v_bar, 0);
    load(sQr, &tmQ, q_bar, 0);
    load(sG, &tmG, g_bar, 0);
    if (n_chunks > 1) load(sK + L::TILE, &tmK, &k_bar[1], 1);
  }
  const float* ddp = p.dden + ((long long)b * p.H + h) * p.S;
  float dden_next = c0 * LA_C + row < p.S ? ddp[c0 * LA_C + row] : 0.f;               // a chunk ahead
  bool ok = true;
  const bool have_state0 = p.s_in != nullptr;
  for (int c = 0; c < n_chunks; ++c) {
    const int st = c & 1;
    uint8_t* sKc = sK + st * L::TILE;
    const int valid = min(LA_C, p.S - (c0 + c) * LA_C);
    const float dden = dden_next;
    if (c + 1 < n_chunks) { const int t = (c0 + c + 1) * LA_C + row; dden_next = t < p.S ? ddp[t] : 0.f; }
    if (!mbar_wait(v_bar, c & 1, p.status, ST_TIMEOUT_TMA_FULL)) ok = false;
    if (ok && !mbar_wait(g_bar, c & 1, p.status, ST_TIMEOUT_TMA_FULL)) ok = false;
    if (__syncthreads_or(!ok)) { ok = false; break; }
    if (warp == 0 && elect_one()) {
      tc_fence_after_sync();
      la_mma_xyT<HD>(tmem_base + COL_A, sG, sV);                                      // T = G V^T
      la_mma_xwT<HD>(tmem_base + COL_DQ, sG, sShi, false);                            // dQ~ = G S^T (value + remainder)
      la_mma_xwT<HD>(tmem_base + COL_DQ, sG, sSlo, true);
      tc_commit(a_bar);
    }
    // K~ while the products that do without it run
    if (!mbar_wait(&k_bar[st], (c >> 1) & 1, p.status, ST_TIMEOUT_TMA_FULL)) ok = false;
    la_phi_half<HD, KIND>(sKc, row, hf, valid, p.scale);
    fence_proxy_async_smem();
    if (!mbar_wait(a_bar, c & 1, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc_fence_after_sync();
    if (tid == 0 && c + 1 < n_chunks) load(sG, &tmG, g_bar, c + 1);                   // both readers of G are done
    la_mask_put<true, rem>(trow + COL_A + hf * 64, quad, hf, lane, [&](int, float x) { return x + dden; }, [](float, float) {});
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0 && elect_one()) {
      tc_fence_after_sync();
      la_mma_tw<HD>(tmem_base + COL_DQ, tmem_base + COL_A, sKc);                      // dQ~ += dA K~ (value + remainder)
      if (rem) la_mma_tw<HD>(tmem_base + COL_DQ, tmem_base + COL_A + 32, sKc);
      la_mma_xTw<HD>(tmem_base + COL_S, sKc, sV, have_state0 || c > 0);    // S += K~^T V
      tc_commit(b_bar);
    }
    s_zk[tid] = la_colsum_rows(sKc, tid % HD, (tid / HD) * (LA_C / ZP), LA_C / ZP);
    if (!mbar_wait(b_bar, c & 1, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc_fence_after_sync();
    if (tid == 0 && c + 2 < n_chunks) load(sKc, &tmK, &k_bar[st], c + 2);
    if (!mbar_wait(q_bar, c & 1, p.status, ST_TIMEOUT_TMA_FULL)) ok = false;          // (landed long ago; its time-out ends the loop above)
    __syncwarp();
    {
      float dq[HH];
      la_tmem_row<HH>(trow + COL_DQ + hf * HH, dq);
#pragma unroll
      for (int i = 0; i < HH; ++i) dq[i] = fmaf(dden, sz[hf * HH + i], dq[i]);        // z of the chunks before this one
      la_put_dphi_half<HD, KIND>(sQr, sV, row, hf, dq, p.scale);                    // V's buffer takes the result
    }
    __syncthreads();                                                                  // every thread has read the old z
    if (tid < HD) {
      float zk = 0.f;
#pragma unroll
      for (int g = 0; g < ZP; ++g) zk += s_zk[g * HD + tid];
      sz[tid] += zk;
    }
    if (c + 1 < n_chunks && quad * 32 < HD) {
      float srow[HH];
      la_tmem_row<HH>(trow + COL_S + hf * HH, srow);
      if (row < HD) la_write_hilo_half<HD>(sShi, sSlo, HD, row, hf, srow);
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (tid == 0) {
      la_store_tile<HD>(&tmDQ, sV, h, (c0 + c) * LA_C, b);
      tma_store_commit();
      if (c + 1 < n_chunks) {
        load(sQr, &tmQ, q_bar, c + 1);
        tma_store_wait_read0();
        load(sV, &tmV, v_bar, c + 1);
      }
    }
  }
  if (tid == 0) tma_store_wait0();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc_fence_after_sync(); tmem_dealloc(tmem_base, L::TMEM); }
}

// ---------------------------------------------------------------------------------------------------- backward 2: dK, dV
template <int HD, int KIND>
__global__ void __launch_bounds__(LA_FWD_THREADS, LaSmem<HD>::CTAS)
linattn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmG, const __grid_constant__ CUtensorMap tmDK,
                       const __grid_constant__ CUtensorMap tmDV, const LinAttnArgs p) {
  using L = LaSmem<HD>;
  constexpr int KA = HD / 64;
  constexpr int HH = HD / 2;
  constexpr int ZP = LA_FWD_THREADS / HD;
  constexpr uint32_t COL_T = 0, COL_DV = 128, COL_DK = 128 + HD, COL_DS = HD == 64 ? COL_T : 128 + 2 * HD;
  // Head size 64 keeps dS in registers (a chunk's share goes through T's columns): 256 TMEM columns hold T, dV and dK
  constexpr bool DS_REG = HD == 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + L::TILE;
  uint8_t* sV = sK + L::TILE;
  uint8_t* sG = sV + L::TILE;
  uint8_t* sKr = sG + L::TILE;                 // raw K: phi' needs it
  uint8_t* sDhi = sKr + L::TILE;
  uint8_t* sDlo = sDhi + L::ST;
  float* sdz = reinterpret_cast<float*>(sDlo + L::ST);     // [HD]
  float* sdden = sdz + HD;                                  // [128]
  float* s_zk = sdden + LA_C;                               // [256]: partial column sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_zk + LA_FWD_THREADS);
  uint64_t* ld_bar = bars; uint64_t* t_bar = bars + 1; uint64_t* u_bar = bars + 2; uint64_t* b_bar = bars + 3;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int quad = warp & 3, hf = warp >> 2, row = quad * 32 + lane;
  const int bh = blockIdx.x / p.n_seg, seg = blockIdx.x % p.n_seg, b = bh / p.H, h = bh % p.H;
  const int c0 = seg * p.seg_chunks;           // first chunk of this CTA's segment
  const int n_chunks = min(p.seg_chunks, (p.S + LA_C - 1) / LA_C - c0);
  const bool full = !p.state_only;               // state_only: only dS / dz of this slice (reads Q, G, dden)
  if (p.n_seg > 1 && !full && seg == 0) return;  // nothing precedes the first segment
  if ((smem_u32(smem) & 1023u) != 0) { if (tid == 0 && p.status) atomicCAS(p.status, 0u, (uint32_t)ST_BAD_ARGUMENT); return; }
  if (tid == 0) {
    mbar_init(ld_bar, 1); mbar_init(t_bar, 1); mbar_init(u_bar, 1); mbar_init(b_bar, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, L::TMEM); tmem_relinquish(); }
  const size_t st_stride = (size_t)HD * HD + HD;
  const uint32_t sx_epoch = la_epoch(p);
  const float* ds_in = la_consume<HD>(p, bh, sx_epoch, p.ds_in);     // the caller's dS, or the higher ranks' totals
  if (tid < HD) {
    float s0[HD];
#pragma unroll
    for (int i = 0; i < HD; ++i) s0[i] = ds_in ? ds_in[blockIdx.x * st_stride + (size_t)tid * HD + i] : 0.f;
    la_write_hilo<HD>(sDhi, sDlo, HD, tid, s0);
    sdz[tid] = ds_in ? ds_in[blockIdx.x * st_stride + (size_t)HD * HD + tid] : 0.f;
  }
  tc_fence_before_sync();
  fence_proxy_async_smem();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t trow = tmem_base + (uint32_t(quad * 32) << 16);
  float ds_acc[DS_REG ? HH : 1];                                                      // DS_REG: this thread's half row of dS
  if (DS_REG) {
#pragma unroll
    for (int i = 0; i < (DS_REG ? HH : 1); ++i) ds_acc[i] = (ds_in && row < HD) ? ds_in[blockIdx.x * st_stride + (size_t)row * HD + hf * HH + i] : 0.f;
  }
  if (!DS_REG && ds_in && hf == 0) {
#pragma unroll
    for (int c = 0; c < HD / 32; ++c) {
      uint32_t r[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = row < HD ? __float_as_uint(ds_in[blockIdx.x * st_stride + (size_t)row * HD + c * 32 + i]) : 0u;
      tmem_st_x32(trow + COL_DS + c * 32, r);
    }
    tmem_st_wait();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();

  // The tiles of a chunk arrive on one barrier: Q and G as soon as the previous chunk's products are done, K (twice: phi' needs
  // it raw) and V once the results that leave through their buffers have been read
  auto load_qg = [&](int chunk) {
    mbar_expect_tx(ld_bar, (full ? 5 : 2) * L::TILE);
#pragma unroll
    for (int a = 0; a < KA; ++a) {
      tma_load_4d(sQ + a * (LA_C * 128), &tmQ, ld_bar, a * 64, h, (c0 + chunk) * LA_C, b);
      tma_load_4d(sG + a * (LA_C * 128), &tmG, ld_bar, a * 64, h, (c0 + chunk) * LA_C, b);
    }
  };
  auto load_kv = [&](int chunk) {
#pragma unroll
    for (int a = 0; a < KA; ++a) {
      tma_load_4d(sK + a * (LA_C * 128), &tmK, ld_bar, a * 64, h, (c0 + chunk) * LA_C, b);
      tma_load_4d(sKr + a * (LA_C * 128), &tmK, ld_bar, a * 64, h, (c0 + chunk) * LA_C, b);
      tma_load_4d(sV + a * (LA_C * 128), &tmV, ld_bar, a * 64, h, (c0 + chunk) * LA_C, b);
    }
  };
  if (tid == 0) { load_qg(n_chunks - 1); if (full) load_kv(n_chunks - 1); }
  const float* ddp = p.dden + ((long long)b * p.H + h) * p.S;
  auto dden_of = [&](int chunk) { const int t = (c0 + chunk) * LA_C + tid; return tid < LA_C && t < p.S ? ddp[t] : 0.f; };
  float dden_next = dden_of(n_chunks - 1);                                            // a chunk ahead
  bool ok = true;
  const bool have_state0 = ds_in != nullptr;
  for (int it = 0; it < n_chunks; ++it) {
    const int c = n_chunks - 1 - it;
    const int valid = min(LA_C, p.S - (c0 + c) * LA_C);
    if (tid < LA_C) sdden[tid] = dden_next;
    if (c > 0) dden_next = dden_of(c - 1);
    if (!mbar_wait(ld_bar, it & 1, p.status, ST_TIMEOUT_TMA_FULL)) ok = false;
    if (__syncthreads_or(!ok)) { ok = false; break; }
    if (full && warp == 0 && elect_one()) {                                           // the products that do without the features
      tc_fence_after_sync();
      la_mma_xyT<HD>(tmem_base + COL_T, sV, sG);                                      // (G V^T)^T = V G^T   [key][query]
      tc_commit(t_bar);
      la_mma_xwT<HD>(tmem_base + COL_DK, sV, sDhi, false);                            // dK~ = V dS^T (value + remainder)
      la_mma_xwT<HD>(tmem_base + COL_DK, sV, sDlo, true);
    }
    la_phi_half<HD, KIND>(sQ, row, hf, LA_C, p.scale);
    if (full) la_phi_half<HD, KIND>(sK, row, hf, valid, p.scale);
    fence_proxy_async_smem();
    if (full) {
      if (!mbar_wait(t_bar, 0, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;            // (two completions a chunk)
      if (__syncthreads_or(!ok)) { ok = false; break; }
      tc_fence_after_sync();
      // queries at or after this key
      la_mask_put<false, false>(trow + COL_T + hf * 64, quad, hf, lane, [&](int i, float x) { return x + sdden[hf * 64 + i]; }, [](float, float) {});
      tc_fence_before_sync();
      __syncthreads();
      if (warp == 0 && elect_one()) {
        tc_fence_after_sync();
        la_mma_tw<HD>(tmem_base + COL_DK, tmem_base + COL_T, sQ);                     // dK~ += mask(dA)^T Q~
        tc_commit(u_bar);
        // A^T = K~ Q~^T, over the tile that dK~ reads just before: in issue order, which is an observation (PTX
        // promises it for one accumulator and shape); waiting for dK~ here would add its completion to the chain of every chunk
        la_mma_xyT<HD>(tmem_base + COL_T, sK, sQ);
        tc_commit(t_bar);
        la_mma_pw<HD, HD>(tmem_base + COL_DV, sK, sDhi, HD * 128, false);             // dV = K~ dS (value + remainder)
        la_mma_pw<HD, HD>(tmem_base + COL_DV, sK, sDlo, HD * 128, true);
      }
      if (!mbar_wait(t_bar, 1, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;            // (u_bar has come by then: products are seen to execute in issue order)
      if (ok && !mbar_wait(u_bar, it & 1, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;
      if (__syncthreads_or(!ok)) { ok = false; break; }
      tc_fence_after_sync();
      la_mask_put<false, false>(trow + COL_T + hf * 64, quad, hf, lane, [](int, float x) { return x; }, [](float, float) {});
      tc_fence_before_sync();
    }
    __syncthreads();
    if (warp == 0 && elect_one()) {
      tc_fence_after_sync();
      if (full) la_mma_tw<HD>(tmem_base + COL_DV, tmem_base + COL_T, sG);             // dV += mask(A)^T G
      la_mma_xTw<HD>(tmem_base + COL_DS, sQ, sG, !DS_REG && (have_state0 || it > 0)); // dS += Q~^T G
      tc_commit(b_bar);
    }
    // dz += Q~^T dden in fp32: ZP row groups per column, combined after the barriers below
    s_zk[tid] = la_colsum_w_rows(sQ, tid % HD, sdden, (tid / HD) * (LA_C / ZP), LA_C / ZP);
    if (!mbar_wait(b_bar, it & 1, p.status, ST_TIMEOUT_ACC_FULL)) ok = false;
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc_fence_after_sync();
    if (tid == 0 && c > 0) load_qg(c - 1);
    if (full) {
      float g[HH];
      la_tmem_row<HH>(trow + COL_DV + hf * HH, g);
#pragma unroll
      for (int i = 0; i < HH; i += 8)                                                 // dV and dK leave through V's and K~'s buffers
        *la_half_piece<HD>(sV, row, hf, i / 8) = make_uint4(pack_bf16x2(g[i], g[i + 1]), pack_bf16x2(g[i + 2], g[i + 3]),
                                                            pack_bf16x2(g[i + 4], g[i + 5]), pack_bf16x2(g[i + 6], g[i + 7]));
      la_tmem_row<HH>(trow + COL_DK + hf * HH, g);
#pragma unroll
      for (int i = 0; i < HH; ++i) g[i] += sdz[hf * HH + i];                           // dz of the chunks after this one
      la_put_dphi_half<HD, KIND>(sKr, sK, row, hf, g, p.scale);
    }
    __syncthreads();                                                                  // every thread has read the old dz
    if (tid < HD) {
      float dzk = 0.f;
#pragma unroll
      for (int g = 0; g < ZP; ++g) dzk += s_zk[g * HD + tid];
      sdz[tid] += dzk;
    }
    if (quad * 32 < HD && (DS_REG || (full && c > 0))) {
      float srow[HH];
      la_tmem_row<HH>(trow + COL_DS + hf * HH, srow);
      if constexpr (DS_REG) {
#pragma unroll
        for (int i = 0; i < HH; ++i) srow[i] = ds_acc[i] += srow[i];
      }
      if (full && c > 0 && row < HD) la_write_hilo_half<HD>(sDhi, sDlo, HD, row, hf, srow);
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (full && tid == 0) {
      la_store_tile<HD>(&tmDV, sV, h, (c0 + c) * LA_C, b);
      la_store_tile<HD>(&tmDK, sK, h, (c0 + c) * LA_C, b);
      tma_store_commit();
      if (c > 0) { tma_store_wait_read0(); load_kv(c - 1); }
    }
  }
  if (tid == 0) tma_store_wait0();
  float* ds_out = la_publish_begin<HD>(p, bh, sx_epoch, p.ds_out);
  const size_t out_idx = full ? bh : blockIdx.x;
  if (ok && ds_out && (!full || seg == 0)) {
    tc_fence_after_sync();
    float srow[HH];
    if constexpr (DS_REG) {
#pragma unroll
      for (int i = 0; i < HH; ++i) srow[i] = ds_acc[i];
    } else {
      la_tmem_row<HH>(trow + COL_DS + hf * HH, srow);
    }
    if (row < HD) {
#pragma unroll
      for (int i = 0; i < HH; i += 4)
        *reinterpret_cast<float4*>(ds_out + out_idx * st_stride + (size_t)row * HD + hf * HH + i) = make_float4(srow[i], srow[i + 1], srow[i + 2], srow[i + 3]);
      if (hf == 0) ds_out[out_idx * st_stride + (size_t)HD * HD + row] = sdz[row];
    }
  }
  la_publish_end(p, bh, sx_epoch);
  la_retire(p, sx_epoch);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) { tc_fence_after_sync(); tmem_dealloc(tmem_base, L::TMEM); }
}

// ---------------------------------------------------------------------------------------------------- host side
template <int HD> constexpr int la_fwd_smem() { return 4 * LaSmem<HD>::TILE + 2 * LaSmem<HD>::ST + HD * 4 + 128; }
// the forward kernel also keeps [2][128] denominator shares and 256 partial column sums
template <int HD> constexpr int la_fwd8_smem() { return la_fwd_smem<HD>() + 2 * LA_C * 4 + LA_FWD_THREADS * 4; }
// dQ, dK / dV: a raw tile and partial column sums; dK / dV: [128] dden
template <int HD> constexpr int la_dq8_smem() { return la_fwd_smem<HD>() + LaSmem<HD>::TILE + LA_FWD_THREADS * 4; }
template <int HD> constexpr int la_dkv_smem() { return 5 * LaSmem<HD>::TILE + 2 * LaSmem<HD>::ST + (HD + LA_C) * 4 + LA_FWD_THREADS * 4 + 128; }

static int la_map(CUtensorMap* m, const LinAttnArgs& a, const AttnTensor& t) {
  return make_tmap_attn(m, t.ptr, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.hd, a.H, a.S, a.B, t.sh, t.ss, t.sb, 64, LA_C, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int HD, int KIND>
static int la_set_attrs() {
  static bool done = false;
  if (done) return 0;
  (void)cudaGetLastError();
  if (cudaFuncSetAttribute(linattn_fwd_kernel<HD, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, la_fwd8_smem<HD>()) != cudaSuccess) return 1;
  if (cudaFuncSetAttribute(linattn_bwd_dq_kernel<HD, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, la_dq8_smem<HD>()) != cudaSuccess) return 1;
  if (cudaFuncSetAttribute(linattn_bwd_dkv_kernel<HD, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, la_dkv_smem<HD>()) != cudaSuccess) return 1;
  done = true;
  return 0;
}

// The states between segments: in place, seg[bh][s] <- base[bh] + the totals of the segments before s (`reverse`: behind s).
__global__ void la_segment_prefix_kernel(float* __restrict__ seg, const float* __restrict__ base, int n_seg, int n, int reverse) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float* p = seg + (size_t)blockIdx.y * n_seg * n + i;
  float acc = base ? base[(size_t)blockIdx.y * n + i] : 0.f;
  for (int k0 = 0; k0 < n_seg; k0 += 8) {            // eight loads in flight: the sum is the only serial part
    float t[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)                      // (the last one's total was not taken)
      t[k] = k0 + k + 1 < n_seg ? p[(size_t)(reverse ? n_seg - 1 - k0 - k : k0 + k) * n] : 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k0 + k < n_seg) { p[(size_t)(reverse ? n_seg - 1 - k0 - k : k0 + k) * n] = acc; acc += t[k]; }
  }
}

template <int HD, int KIND>
static int la_launch(const LinAttnArgs& a, int which, cudaStream_t st) {
  if (la_set_attrs<HD, KIND>()) return 104;
  if (which == 4) {                                     // a whole backward: G pass, dQ, dK / dV
    if (int rc = la_launch<HD, KIND>(a, 3, st)) return rc;
    if (int rc = la_launch<HD, KIND>(a, 1, st)) return rc;
    LinAttnArgs t = a;
    t.seg = a.dseg;
    t.s_in = nullptr;
    return la_launch<HD, KIND>(t, 2, st);
  }
  if (which != 3 && a.n_seg > 1 && !a.state_only && a.s_in != a.seg && a.ds_in != a.seg) {
    // segments: their totals, the prefix over them (the forward's serves the dQ pass too), then the pass itself from there
    LinAttnArgs t = a;
    if (which != 1) {
      t.state_only = 1; t.s_in = t.ds_in = nullptr; t.s_out = t.ds_out = a.seg;
      if (int rc = la_launch<HD, KIND>(t, which, st)) return rc;
      constexpr int N = HD * HD + HD;
      la_segment_prefix_kernel<<<dim3((N + 255) / 256, a.B * a.H), 256, 0, st>>>(a.seg, which == 0 ? a.s_in : a.ds_in, a.n_seg, N, which == 2);
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return 400 + (int)e;
    }
    t = a;
    if (which == 2) t.ds_in = a.seg; else t.s_in = a.seg;
    return la_launch<HD, KIND>(t, which, st);
  }
  if (which == 3) {
    const long long n = (long long)a.B * a.H * a.S * (HD / 8);
    la_g_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : 400 + (int)e;
  }
  CUtensorMap tq, tk, tv, tg, t0, t1;                   // t0, t1: results
  const unsigned grid = (unsigned)(a.B * a.H * a.n_seg);
  if (la_map(&tk, a, a.k)) return 102;
  if (la_map(&tv, a, a.v)) return 103;
  tq = tg = t0 = t1 = tk;
  if (which != 0 && la_map(&tg, a, a.g)) return 104;
  const bool state = a.state_only != 0 && which != 1;
  if (!(which == 0 && state) && la_map(&tq, a, a.q)) return 101;
  if (which == 0) {
    if (!state && la_map(&t0, a, a.o)) return 105;
    if (!state && a.o_lo.ptr && la_map(&t1, a, a.o_lo)) return 106;
    linattn_fwd_kernel<HD, KIND><<<grid, LA_FWD_THREADS, la_fwd8_smem<HD>(), st>>>(tq, tk, tv, t0, t1, a);
  } else if (which == 1) {
    if (la_map(&t0, a, a.dq)) return 105;
    linattn_bwd_dq_kernel<HD, KIND><<<grid, LA_FWD_THREADS, la_dq8_smem<HD>(), st>>>(tq, tk, tv, tg, t0, a);
  } else {
    if (!state && (la_map(&t0, a, a.dk) || la_map(&t1, a, a.dv))) return 105;
    linattn_bwd_dkv_kernel<HD, KIND><<<grid, LA_FWD_THREADS, la_dkv_smem<HD>(), st>>>(tq, tk, tv, tg, t0, t1, a);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace b200

// which: 0 forward (or state-only pass), 4 backward; its parts: 3 G pass, then 1 dQ and 2 dK / dV. Causal form; hd 64 or 128; bf16.
extern "C" int b200_linattn(const b200::LinAttnArgs* a, int which, cudaStream_t st) {
  using namespace b200;
  if (a->B <= 0 || a->H <= 0 || a->S <= 0) return 0;
  if (which < 0 || which > 4 || (which == 4 && (a->state_only || a->sx.role != 0 || (a->n_seg > 1 && !a->dseg))) || (which > 0 && (!a->g.ptr || !a->dden)) || a->n_seg < 1 || (a->n_seg > 1 && (!a->seg || a->state_only || a->sx.role != 0))) return -2;
  if ((long long)a->n_seg * a->seg_chunks < (a->S + LA_C - 1) / LA_C || (long long)(a->n_seg - 1) * a->seg_chunks >= (a->S + LA_C - 1) / LA_C) return -2;
  if (a->hd == 64) return a->kind == 0 ? la_launch<64, 0>(*a, which, st) : la_launch<64, 1>(*a, which, st);
  if (a->hd == 128) return a->kind == 0 ? la_launch<128, 0>(*a, which, st) : la_launch<128, 1>(*a, which, st);
  return -3;
}
extern "C" int b200_linattn_init() { return b200::la_set_attrs<64, 0>() | b200::la_set_attrs<64, 1>() | b200::la_set_attrs<128, 0>() | b200::la_set_attrs<128, 1>(); }
