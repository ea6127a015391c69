// What the tcgen05 GEMM kernels share: tile constants, operand kinds, activations of the epilogue.
#pragma once
#include "../common/ptx.cuh"
#include "../common/tensormap.h"
#include "gemm_sm100.h"

namespace b200 {

constexpr int BM = 128;
constexpr int EPI_WARPS = 8;
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;   // TMA warp + MMA warp + epilogue warps
constexpr int TILE_K_BYTES = 128;  // one swizzle row
constexpr int UMMA_K_BYTES = 32;
constexpr int EPI_PANEL_BYTES = 32 * 128;   // per-warp staging panel: 32 rows x 128 bytes

template <typename T> struct ElemTraits;
template <> struct ElemTraits<__nv_bfloat16> {
  static constexpr int BK = 64;
  static constexpr uint32_t FMT = FMT_BF16;
  static constexpr bool TF32 = false;
};
template <> struct ElemTraits<float> {
  static constexpr int BK = 32;
  static constexpr uint32_t FMT = FMT_TF32;
  static constexpr bool TF32 = true;
};
// 8-bit operand tags (one byte each). The integer kinds accumulate in int32, fp8 in fp32; the
// epilogue turns either into fp32 and applies per-row (A) and per-column (B) dequantisation scales.
struct s8s8_t { int8_t v; };     // signed x signed      (quantised activations x quantised weights)
struct u8s8_t { uint8_t v; };    // unsigned A x signed B (the reference's igemm contract, src/int8.rs:222-234)
struct e4m3_t { uint8_t v; };    // fp8 e4m3 x e4m3
enum : int { KIND_F16 = 0, KIND_TF32 = 1, KIND_I8 = 2, KIND_F8 = 3 };
template <typename T> struct KindOf { static constexpr int v = ElemTraits<T>::TF32 ? KIND_TF32 : KIND_F16; static constexpr uint32_t AF = ElemTraits<T>::FMT, BF = ElemTraits<T>::FMT, CF = CFMT_F32; };
template <> struct ElemTraits<s8s8_t> { static constexpr int BK = 128; static constexpr uint32_t FMT = FMT_S8; static constexpr bool TF32 = false; };
template <> struct ElemTraits<u8s8_t> { static constexpr int BK = 128; static constexpr uint32_t FMT = FMT_S8; static constexpr bool TF32 = false; };
template <> struct ElemTraits<e4m3_t> { static constexpr int BK = 128; static constexpr uint32_t FMT = 0; static constexpr bool TF32 = false; };
template <> struct KindOf<s8s8_t> { static constexpr int v = KIND_I8; static constexpr uint32_t AF = FMT_S8, BF = FMT_S8, CF = CFMT_S32; };
template <> struct KindOf<u8s8_t> { static constexpr int v = KIND_I8; static constexpr uint32_t AF = FMT_U8, BF = FMT_S8, CF = CFMT_S32; };
template <> struct KindOf<e4m3_t> { static constexpr int v = KIND_F8; static constexpr uint32_t AF = 0, BF = 0, CF = CFMT_F32; };   // 0 = E4M3 in kind::f8f6f4

// hardware tanh (MUFU.TANH): relative error ~2^-11, far below bf16 output precision
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float act_fwd(float v, int act) {
  switch (act) {
    case ACT_RELU: return v > 0.f ? v : 0.f;
    case ACT_GELU: {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      float u = k0 * (v + k1 * v * v * v);
      return 0.5f * v * (1.f + tanh_fast(u));
    }
    case ACT_SILU: return v / (1.f + __expf(-v));
    case ACT_SIGMOID: return 1.f / (1.f + __expf(-v));
    case ACT_TANH: return tanh_fast(v);
    default: return v;
  }
}
// derivative of the activation, evaluated at the saved value `s`:
// the pre-activation for GELU/SiLU, the output for ReLU/sigmoid/tanh.
__device__ __forceinline__ float act_bwd(float s, int act) {
  switch (act) {
    case ACT_RELU: return s > 0.f ? 1.f : 0.f;
    case ACT_GELU: {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      float u = k0 * (s + k1 * s * s * s);
      float t = tanh_fast(u);
      float du = k0 * (1.f + 3.f * k1 * s * s);
      return 0.5f * (1.f + t) + 0.5f * s * (1.f - t * t) * du;
    }
    case ACT_SILU: {
      float sg = 1.f / (1.f + __expf(-s));
      return sg * (1.f + s * (1.f - sg));
    }
    case ACT_SIGMOID: return s * (1.f - s);
    case ACT_TANH: return 1.f - s * s;
    default: return 1.f;
  }
}

// ---------------------------------------------------------------------------- operands in shared memory
// K-major: rows of 128 bytes along K, 8-row groups 1024 B apart. MN-major: rows of 128 bytes along M / N per K index, K groups of 8 rows
// 1024 B apart (4 rows, 512 B, for 32-bit elements: their 128-byte swizzle moves 32-byte pieces over 4 rows), atoms of one row's width
// BK * 128 B apart.
template <typename T, bool MN>
__device__ __forceinline__ uint64_t operand_desc(uint32_t tile, int k) {
  constexpr uint32_t UMMA_K = UMMA_K_BYTES / sizeof(T);
  if constexpr (!MN) return make_sdesc_sw128(tile + k * UMMA_K_BYTES, 0, 1024);
  else if constexpr (sizeof(T) == 4) return make_sdesc_sw128_b32(tile + k * UMMA_K * TILE_K_BYTES, ElemTraits<T>::BK * TILE_K_BYTES, 512);
  else return make_sdesc_sw128(tile + k * UMMA_K * TILE_K_BYTES, ElemTraits<T>::BK * TILE_K_BYTES, 1024);
}

template <typename T>
__device__ __forceinline__ void umma_kind(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum) {
  if constexpr (KindOf<T>::v == KIND_TF32) umma_tf32(d, da, db, idesc, accum);
  else if constexpr (KindOf<T>::v == KIND_I8) umma_i8(d, da, db, idesc, accum);
  else if constexpr (KindOf<T>::v == KIND_F8) umma_f8(d, da, db, idesc, accum);
  else umma_f16(d, da, db, idesc, accum);
}

template <typename T>
__device__ __forceinline__ void umma_kind_pair(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum) {
  if constexpr (KindOf<T>::v == KIND_TF32) umma_tf32_pair(d, da, db, idesc, accum);
  else if constexpr (KindOf<T>::v == KIND_I8) umma_i8_pair(d, da, db, idesc, accum);
  else if constexpr (KindOf<T>::v == KIND_F8) umma_f8_pair(d, da, db, idesc, accum);
  else umma_f16_pair(d, da, db, idesc, accum);
}

template <typename T> struct DT;
template <> struct DT<__nv_bfloat16> { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16; };
template <> struct DT<float> { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_FLOAT32; };
template <> struct DT<s8s8_t> { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_UINT8; };
template <> struct DT<u8s8_t> { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_UINT8; };
template <> struct DT<e4m3_t> { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_UINT8; };

// Rows of a K-major tile that are copied: the copy engine also spends its time on rows past the end of a matrix (it fills them with zeros at the
// rate of any others, about 64 bytes a cycle), and what such a row of A or B holds only reaches rows or columns of the result that are not
// stored. 16 x 32000 x 512 11.7 -> 8.7 us.
__host__ __device__ constexpr int tile_box(int rows, int tile_rows) { return rows >= tile_rows ? tile_rows : (rows + 7) / 8 * 8; }

// Tensor map of an operand of `rows` rows and K columns (stored transposed when MN) for tiles of `tile_rows` rows.
// K-major: view [batch][rows][K], box {BK, tile_box(rows, tile_rows)}. MN-major: view [batch][K][rows], box {one 128-byte row, BK}.
template <typename T, bool MN>
inline int operand_map(CUtensorMap* m, const void* base, int rows, int K, int batch, long long ld, long long stride, int tile_rows) {
  constexpr int BK = ElemTraits<T>::BK, ATOM = TILE_K_BYTES / sizeof(T);
  if (!MN) return make_tmap_3d(m, base, DT<T>::v, sizeof(T), K, rows, batch, ld * sizeof(T), stride * sizeof(T), BK, tile_box(rows, tile_rows), CU_TENSOR_MAP_SWIZZLE_128B);
  return make_tmap_3d(m, base, DT<T>::v, sizeof(T), rows, K, batch, ld * sizeof(T), stride * sizeof(T), ATOM, BK,
                      sizeof(T) == 4 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B);
}

// gemm_cluster_sm100.cu
int gemm_cluster_ranks(const GemmArgs& a);
int gemm_cluster_launch(const GemmArgs& a, int ranks, cudaStream_t stream);
int gemm_cluster_init();
// gemm_kinds_sm100.cu: fp32 (as TF32) and 8-bit operands
int gemm_kinds_launch(const GemmArgs& a, int bn, int num_sms, cudaStream_t stream);
int gemm_kinds_init();

}  // namespace b200
