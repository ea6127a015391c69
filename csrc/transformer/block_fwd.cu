// A pre-norm transformer block, forward only, as ONE call from the host: LayerNorm, QKV projection, flash attention, output
// projection, residual add + LayerNorm, GELU layer, second feed-forward layer with the residual. The launches are the ones
// ops/transformer.py makes one by one when it has to keep tensors for a backward; a prompt of a few hundred tokens takes
// 5 to 10 us on the GPU per launch, less than the 30 us that preparing a launch from Python took, so without gradients the
// whole sequence is issued here from one record of pointers (each launcher goes through launch_pdl).
#include <cmath>
#include "../attention/flash_sm100.h"
#include "../gemm/gemm_sm100.h"

extern "C" int b200_layernorm_fwd(const void* x, const float* gamma, const float* beta, void* y, float* mean, float* rstd, long long rows, int d,
                                  float eps, int is_bf16, cudaStream_t st);
extern "C" int b200_add_layernorm_fwd(const void* x, const void* res, const float* gamma, const float* beta, void* sum_out, void* y, float* mean,
                                      float* rstd, long long rows, int d, float eps, cudaStream_t st);
extern "C" int b200_binary(const void* a, const void* b, void* y, long long n, int op, long long period, int is_bf16, cudaStream_t st);

namespace b200 {

struct BlockArgs {
  // activations [T, d] and workspace, all bf16 and 16-byte aligned: h [T, d], qkv [T, 3d], o [T, d], y1 [T, d], a [T, ff]
  const void* x; void* y;
  void *h, *qkv, *o, *y1, *a;
  float *mean, *rstd, *lse;                      // fp32 [T], [T], [B, heads, S]
  const void *wqkv, *wo, *w1, *w2;               // bf16, K-major: [3d, d], [d, d], [ff, d], [d, ff]
  const float *g1, *be1, *g2, *be2, *bqkv, *bo, *b1, *b2;
  int B, S, d, ff, heads, causal, op_add, num_sms;
  float eps;
  uint32_t* status;
};

static int block_gemm(const BlockArgs& b, const void* A, int M, int K, const void* W, int N, const float* bias, int act, const void* residual, void* C, cudaStream_t st) {
  GemmArgs g = {};
  GemmParams& p = g.p;
  p.M = g.M = M; p.N = g.N = N; p.K = g.K = K; p.batch = g.batch = 1; p.splits = 0;
  p.C = C; p.ldc = N; p.strideC = (long long)M * N;
  p.bias = bias; p.bias_f32 = 1; p.bias_vec_ok = ((uintptr_t)bias % 16 == 0 && N % 4 == 0) ? 1 : 0;
  p.residual = residual; p.ldr = residual ? N : 0; p.strideR = residual ? (long long)M * N : 0; p.res_vec_ok = residual ? 1 : 0;
  p.alpha = 1.f; p.act = act; p.dact = ACT_NONE; p.out_mode = OUT_BF16; p.vec_ok = 1;          // widths are multiples of 8, buffers aligned
  p.status = b.status;
  g.A = A; g.lda = K; g.strideA = (long long)M * K; g.B = W; g.ldb = K; g.strideB = (long long)N * K;
  g.dtype = GEMM_BF16;
  return b200_gemm_launch(&g, 0, b.num_sms, st);
}

}  // namespace b200

// Returns 0, or the failing launch's code; *launches counts the kernels.
extern "C" int b200_block_fwd(const b200::BlockArgs* args, int* launches, cudaStream_t st) {
  using namespace b200;
  const BlockArgs& b = *args;
  const int T = b.B * b.S, d = b.d, hd = d / b.heads;
  int n = 7;
  if (int rc = b200_layernorm_fwd(b.x, b.g1, b.be1, b.h, b.mean, b.rstd, T, d, b.eps, 1, st)) return rc;
  if (int rc = block_gemm(b, b.h, T, d, b.wqkv, 3 * d, b.bqkv, ACT_NONE, nullptr, b.qkv, st)) return rc;
  FlashArgs f = {};
  char* qkv = static_cast<char*>(b.qkv);
  AttnTensor* part[3] = {&f.q, &f.k, &f.v};
  for (int i = 0; i < 3; ++i) *part[i] = {qkv + (size_t)i * d * 2, (long long)b.S * 3 * d, 3ll * d, hd};
  f.o = {b.o, (long long)b.S * d, d, hd};
  f.lse = b.lse; f.B = b.B; f.H = b.heads; f.Sq = f.Skv = b.S; f.hd = hd;
  f.scale = (float)(1.0 / sqrt((double)hd)); f.causal = b.causal; f.status = b.status;
  if (int rc = b200_flash_fwd(&f, st)) return rc;
  if (int rc = block_gemm(b, b.o, T, d, b.wo, d, b.bo, ACT_NONE, nullptr, b.h, st)) return rc;
  int rc = b200_add_layernorm_fwd(b.h, b.x, b.g2, b.be2, b.y1, b.o, b.mean, b.rstd, T, d, b.eps, st);
  if (rc == -1) {                                            // a width the fused kernel does not take: two kernels
    if ((rc = b200_binary(b.h, b.x, b.y1, (long long)T * d, b.op_add, 0, 1, st))) return rc;
    rc = b200_layernorm_fwd(b.y1, b.g2, b.be2, b.o, b.mean, b.rstd, T, d, b.eps, 1, st);
    ++n;
  }
  if (rc) return rc;
  if ((rc = block_gemm(b, b.o, T, d, b.w1, b.ff, b.b1, ACT_GELU, nullptr, b.a, st))) return rc;
  if ((rc = block_gemm(b, b.a, T, b.ff, b.w2, d, b.b2, ACT_NONE, b.y1, b.y, st))) return rc;
  *launches = n;
  return 0;
}
