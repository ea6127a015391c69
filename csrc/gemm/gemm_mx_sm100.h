// Launch interface of the block-scaled product (plain C structs).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace b200 {

struct MxGemmArgs {
  const void* A; const void* B;        // element bytes, K-major
  const void* sfa; const void* sfb;    // scale chunks (see above); row blocks padded to a multiple of 256 rows
  void* C; long long ldc;              // [M, N] bf16 or fp32
  int M, N, K;
  int out_f32;
  float alpha;                         // product of the per-tensor scales (NVFP4) or 1
  int kind;
  const void* bias;                    // [N] bf16 or null, added in fp32
  uint32_t* status;
};

}  // namespace b200

extern "C" int b200_gemm_mx(const b200::MxGemmArgs* args, int num_sms, cudaStream_t stream);
extern "C" int b200_mx_quant(const void* x, int is_bf16, long long ldx, long long rows, int K, int kind, float tensor_scale, void* data,
                             void* sf, cudaStream_t st);
