// The GEMM body for fp32 operands (as TF32, all four layouts) and 8-bit operands (K-major).
#include "gemm_body.cuh"

namespace b200 {

// TF32 tiles 64, 128 and 256 (a pair of CTAs on 256 x 256) wide: us that a launch takes besides its K loop, us a K block takes while the whole
// machine runs them, and what a transposed A / B adds to that (its 32-byte swizzle pieces are read more slowly). Fitted to products
// of 300 to 4096; the least sum is taken. 4096^3 254 us on 128-wide tiles, 193 on pairs (both transposed: 408 and 242); 1024^3
// with B transposed 15.9 us 128 wide, 12.9 us 64 wide; 2048 x 1024 x 512 8.9 us 128 wide, 12.7 on pairs.
static int f32_tile(const GemmArgs& a, int sms) {
  static constexpr struct { int bn; float base, block, a_mn, b_mn; } T[3] = {
      {64, 4.3f, 0.239f, 0.100f, 0.017f}, {128, 4.4f, 0.283f, 0.084f, 0.084f}, {256, 6.7f, 0.377f, 0.034f, 0.022f}};
  int best = 128; float least = 1e30f;
  for (const auto& t : T) {
    if (t.bn == 256 && (a.M < 256 || !pair_enabled())) continue;
    const long long bm = t.bn == 256 ? 256 : 128, slots = t.bn == 256 ? sms / 2 : sms;
    const long long tiles = ((a.M + bm - 1) / bm) * ((a.N + t.bn - 1) / t.bn) * a.batch * a.p.splits;
    const long long blocks = ((a.K + 31) / 32 + a.p.splits - 1) / a.p.splits;
    const float us = t.base + (float)((tiles + slots - 1) / slots * blocks) * (t.block + (a.a_mn ? t.a_mn : 0.f) + (a.b_mn ? t.b_mn : 0.f));
    if (us < least) { least = us; best = t.bn; }
  }
  return best;
}

static int launch_f32(const GemmArgs& a, int bn, cudaStream_t s, int sms) {
  if (bn == 0) bn = f32_tile(a, sms);
  if (bn == 256) {
    if (!a.a_mn && !a.b_mn) return launch_pair<float, false, false>(a, s, sms);
    if (!a.a_mn && a.b_mn) return launch_pair<float, false, true>(a, s, sms);
    if (a.a_mn && !a.b_mn) return launch_pair<float, true, false>(a, s, sms);
    return launch_pair<float, true, true>(a, s, sms);
  }
  return bn == 64 ? launch_major<float, 64>(a, s, sms) : launch_major<float, 128>(a, s, sms);
}

// Pairs of CTAs (bn 512) from one and a half waves of them: int8 4096^3 to bf16 56.4 -> 47.8 us, 2048 x 4096 x 4096 28.0 -> 27.4; with one
// wave, 1024 x 4096 x 4096, 17.1 -> 18.3, and with K = 1024 the results bind: 23.8 -> 26.2. 64-wide tiles while they run at once.
static int tile_8bit(const GemmArgs& a, int sms) {
  const long long m = (a.M + 127) / 128 * a.batch;
  if (m * ((a.N + 63) / 64) <= sms) return 64;
  if (pair_enabled() && a.K >= 2048 && (long long)((a.M + 255) / 256) * ((a.N + 255) / 256) * a.batch * 4 >= 3ll * sms) return 512;
  return m * ((a.N + 255) / 256) >= sms ? 256 : 128;
}

template <typename T>
static int launch_8bit(const GemmArgs& a, int bn, cudaStream_t s, int sms) {
  if (bn == 0) bn = tile_8bit(a, sms);
  if (bn == 512) return launch_pair<T, false, false>(a, s, sms);
  if (bn == 64) return launch_one<T, 64, false, false>(a, s, sms);
  return bn == 256 ? launch_one<T, 256, false, false>(a, s, sms) : launch_one<T, 128, false, false>(a, s, sms);
}

int gemm_kinds_launch(const GemmArgs& a, int bn, int num_sms, cudaStream_t stream) {
  switch (a.dtype) {
    case GEMM_F32: return launch_f32(a, bn, stream, num_sms);
    case GEMM_S8S8: return launch_8bit<s8s8_t>(a, bn, stream, num_sms);
    case GEMM_U8S8: return launch_8bit<u8s8_t>(a, bn, stream, num_sms);
    case GEMM_E4M3: return launch_8bit<e4m3_t>(a, bn, stream, num_sms);
    default: return -3;
  }
}

template <typename T>
static int init_8bit() { return gemm_set_attr<T, 64, false, false>() | gemm_set_attr<T, 128, false, false>() | gemm_set_attr<T, 256, false, false>() | pair_set_attr<T, false, false>(); }

int gemm_kinds_init() {
  int e = init_8bit<s8s8_t>() | init_8bit<u8s8_t>() | init_8bit<e4m3_t>();
#define B200_INIT_MAJOR(A, B) e |= gemm_set_attr<float, 64, A, B>() | gemm_set_attr<float, 128, A, B>() | pair_set_attr<float, A, B>();
  B200_INIT_MAJOR(false, false) B200_INIT_MAJOR(false, true) B200_INIT_MAJOR(true, false) B200_INIT_MAJOR(true, true)
#undef B200_INIT_MAJOR
  return e;
}

}  // namespace b200
