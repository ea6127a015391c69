// G1, C entry points and the kernels built around one GEMM body: plain products, tensor-parallel products, the one-kernel
// MoE forward. The body and its launch code (launch_pdl) are in gemm_body.cuh; fp32 and 8-bit operands are instantiated in gemm_kinds_sm100.cu.
#include "gemm_body.cuh"

namespace b200 {

// ---------------------------------------------------------------------------- expert-parallel MoE layer, forward, ONE kernel
// dispatch (token rows stored into the owning rank's expert buffers over NVLink, slots claimed with remote atomics)
// -> cross-rank barrier -> grouped GEMM 1 (+bias, activation, saved pre-activation) over the real per-expert counts
// -> grid barrier -> grouped GEMM 2 into the peer-visible output buffer -> cross-rank barrier -> combine (weighted sum of
// the k expert rows of every token, read from the owners over NVLink) while the input buffer is saved for the backward
// and cleared -> cross-rank barrier. One persistent launch of one CTA per SM: the barriers inside it need every CTA
// resident. No host synchronisation, no NCCL; every wait is bounded by a clock budget and reports through the status word.
constexpr int MOEF_MAX_RANKS = 8;
struct MoeFusedArgs {
  const __nv_bfloat16* x; const int* idx; int* dest;        // [T, d], [T, k] expert ids, [T, k] global row ids (out)
  void* xbuf[MOEF_MAX_RANKS]; int* fill[MOEF_MAX_RANKS];     // every rank's expert input buffer [E_local, cap, d] and slot counters [E_local]
  const void* ybuf[MOEF_MAX_RANKS];                          // every rank's expert output buffer [E_local, cap, d]
  uint32_t* bar_flags[MOEF_MAX_RANKS];                       // cross-rank barrier flags (shared with the barrier kernel of the backward)
  uint32_t* bar_words;                                       // local: [0] cross-rank barriers passed so far
  uint32_t* sync;                                            // local: [0] CTA arrivals, [1] barrier generation
  const float* w; __nv_bfloat16* out;                        // [T, k] gate weights, [T, d] result
  __nv_bfloat16* xsave;                                      // copy of this rank's expert inputs for the weight gradient
  int* counts_out;                                           // [E_local] rows in use per local expert (for the backward)
  long long tokens, rows_per_rank, wait_cycles;
  int k, d, E_local, cap, rank, world;
  uint32_t* status;
};

__device__ __forceinline__ void moef_barrier(const MoeFusedArgs& a, uint32_t gen, uint32_t epoch, bool cross) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();                                  // this CTA's stores, peer stores included, are out
    const uint32_t old = atomicAdd(a.sync, 1u);
    if (old % gridDim.x == gridDim.x - 1) {                  // the last CTA to arrive speaks for the rank
      if (cross && a.world > 1) {
        for (int r = 0; r < a.world; ++r) st_release_sys_u32(a.bar_flags[r] + a.rank, epoch);
        for (int r = 0; r < a.world; ++r)
          if (!wait_flag<true>(a.bar_flags[a.rank] + r, epoch, a.wait_cycles, a.status, ST_TIMEOUT_PEER_FLAG)) break;
      }
      if (cross) { __threadfence_system(); a.bar_words[0] = epoch; }
      __threadfence();
      st_release_gpu_u32(a.sync + 1, gen);
    }
    wait_flag<false>(a.sync + 1, gen, 2 * a.wait_cycles, a.status, ST_TIMEOUT_GENERIC);
    __threadfence();
  }
  __syncthreads();
}

__global__ void __launch_bounds__(GEMM_THREADS, 1)
moe_fused_fwd_kernel(const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ GemmParams p1,
                     const __grid_constant__ OutMaps om1, const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2,
                     const __grid_constant__ GemmParams p2, const __grid_constant__ OutMaps om2, const __grid_constant__ MoeFusedArgs a) {
  const uint32_t gen0 = *reinterpret_cast<volatile const uint32_t*>(a.sync + 1);
  const uint32_t ep0 = *reinterpret_cast<volatile const uint32_t*>(a.bar_words);
  const int lane = threadIdx.x & 31;
  const long long warp_g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long row_vec = a.d / 8;                         // 16-byte vectors per row
  // ---- dispatch: one warp per (token, choice)
  for (long long wid = warp_g; wid < a.tokens * a.k; wid += n_warps) {
    const long long t = wid / a.k;
    const int e = a.idx[wid];
    const int owner = e / a.E_local, el = e % a.E_local;
    int slot = 0;
    if (lane == 0) slot = atomicAdd_system(a.fill[owner] + el, 1);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (slot >= a.cap) { if (lane == 0) a.dest[wid] = -1; continue; }
    if (lane == 0) a.dest[wid] = (owner * a.E_local + el) * a.cap + slot;
    const uint4* src = reinterpret_cast<const uint4*>(a.x + t * a.d);
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.xbuf[owner]) + ((long long)el * a.cap + slot) * a.d);
    for (long long i = lane; i < row_vec; i += 32) dst[i] = src[i];
  }
  moef_barrier(a, gen0 + 1, ep0 + 1, true);                  // every rank's rows and slot counts have landed
  fence_proxy_async_all();                                   // ... and are visible to the TMA loads below
  gemm_body<__nv_bfloat16, 256, false, false, TP_NONE, 1, true>(tmA1, tmB1, p1, nullptr, &om1);
  moef_barrier(a, gen0 + 2, 0u, false);                      // all of h is written
  fence_proxy_async_all();
  gemm_body<__nv_bfloat16, 256, false, false, TP_NONE, 1>(tmA2, tmB2, p2, nullptr, &om2);
  moef_barrier(a, gen0 + 3, ep0 + 2, true);                  // every rank's expert outputs are in place
  // ---- combine: one warp per token; rows may live on a peer
  for (long long t = warp_g; t < a.tokens; t += n_warps) {
    for (long long c = lane; c < row_vec; c += 32) {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int j = 0; j < a.k; ++j) {
        const int r = a.dest[t * a.k + j];
        if (r < 0) continue;
        const float wj = a.w[t * a.k + j];
        const int owner = (int)(r / a.rows_per_rank);
        const long long lr = r % a.rows_per_rank;
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(a.ybuf[owner]) + lr * a.d) + c);
        const __nv_bfloat162* hh = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int q = 0; q < 4; ++q) { const float2 f = __bfloat1622float2(hh[q]); acc[2 * q] += wj * f.x; acc[2 * q + 1] += wj * f.y; }
      }
      uint4 o;
      __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int q = 0; q < 4; ++q) oh[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
      *(reinterpret_cast<uint4*>(a.out + t * a.d) + c) = o;
    }
  }
  // ---- keep the expert inputs for the weight gradient and clear the buffer for the next layer (rows in use, rounded up to
  //      the 128-row tiles the backward's K loop covers; rows past a count are zero already and are saved as zeros)
  {
    uint4* xb = reinterpret_cast<uint4*>(a.xbuf[a.rank]);
    uint4* xs = reinterpret_cast<uint4*>(a.xsave);
    const int* fill = a.fill[a.rank];
    const long long total_rows = (long long)a.E_local * a.cap;
    for (long long row = warp_g; row < total_rows; row += n_warps) {
      const int e = (int)(row / a.cap), r = (int)(row % a.cap);
      const int cnt = min(*reinterpret_cast<volatile const int*>(fill + e), a.cap);
      if (r >= (cnt + 127) / 128 * 128) continue;
      for (long long i = lane; i < row_vec; i += 32) {
        const uint4 v = xb[row * row_vec + i];
        if (xs) xs[row * row_vec + i] = v;
        xb[row * row_vec + i] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }
  moef_barrier(a, gen0 + 4, 0u, false);                      // every CTA has read the slot counts
  if (blockIdx.x == 0)
    for (int e = threadIdx.x; e < a.E_local; e += blockDim.x) {
      int* f = a.fill[a.rank] + e;
      a.counts_out[e] = min(*reinterpret_cast<volatile int*>(f), a.cap);
      *f = 0;
    }
  moef_barrier(a, gen0 + 5, ep0 + 3, true);                  // peers have read my outputs; everyone's input buffers are clear
}

// bf16, K-major x K-major (the Linear forward layout) fused with its neighbouring collective
template <int BN, int TP>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tp_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ GemmParams p,
               const __grid_constant__ TpParams tp, const __grid_constant__ PeerMaps pm) {
  gemm_body<__nv_bfloat16, BN, false, false, TP>(tmA, tmB, p, &tp, nullptr, &pm);
}

template <int BN, int TP>
static int launch_tp(const GemmArgs& a, const TpParams& tp, cudaStream_t stream, int num_sms) {
  using T = __nv_bfloat16;
  using S = GemmSmem<T, BN, false, false>;
  CUtensorMap tmA, tmB;
  // A: TP_AG_GEMM multiplies out of the local staging copy [M, K]; TP_GEMM_RS out of the caller's A
  const void* aptr = (TP == TP_AG_GEMM) ? tp.stage_peer[tp.rank] : a.A;
  const long long lda = (TP == TP_AG_GEMM) ? a.K : a.lda;
  int rc = operand_map<T, false>(&tmA, aptr, a.M, a.K, 1, lda, (long long)a.M * lda, BM);
  if (rc) return 100 + rc;
  rc = operand_map<T, false>(&tmB, a.B, a.N, a.K, 1, a.ldb, (long long)a.N * a.ldb, BN);
  if (rc) return 200 + rc;
  static bool attr_done = false;
  if (!attr_done) {
    (void)cudaGetLastError();
    cudaError_t e = cudaFuncSetAttribute(gemm_tp_kernel<BN, TP>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_done = true;
  }
  // every CTA must be resident at once (CTAs wait on one another): one CTA per SM, grid <= SM count
  int grid = num_sms;
  if (TP == TP_AG_GEMM && grid - tp.copy_ctas < 1) return -6;
  PeerMaps pm;
  pm.use = 0;
  for (int r = 0; r < TP_MAX_WORLD; ++r) pm.m[r] = tmA;
  if (TP == TP_AG_GEMM) {
    static int tp_bulk = -1;
    if (tp_bulk < 0) { const char* e = getenv("B200NN_TP_BULK_GATHER"); tp_bulk = (e && e[0] == '0') ? 0 : 1; }
    if (tp_bulk && S::STAGE_BYTES >= 32 * 1024) pm.use = 2;
  }
  if (TP == TP_GEMM_RS && BN >= 128) {
    static int tp_tma = -1;
    if (tp_tma < 0) { const char* e = getenv("B200NN_TP_TMA_STORE"); tp_tma = (e && e[0] == '0') ? 0 : 1; }
    const unsigned long long rows_per_rank = (unsigned long long)tp.blocks_per_rank * BM, nb = (unsigned long long)a.p.N * 2;
    if (tp_tma && a.p.N % 8 == 0) {
      pm.use = 1;
      for (int r = 0; r < tp.world; ++r)
        if ((reinterpret_cast<uintptr_t>(tp.slots_peer[r]) & 15) ||
            make_tmap_3d(&pm.m[r], tp.slots_peer[r], DT<T>::v, sizeof(T), a.p.N, rows_per_rank, 2ull * tp.world, nb, rows_per_rank * nb, 64, 32,
                         CU_TENSOR_MAP_SWIZZLE_128B)) { pm.use = 0; break; }
    }
  }
  gemm_tp_kernel<BN, TP><<<grid, GEMM_THREADS, S::TOTAL, stream>>>(tmA, tmB, a.p, tp, pm);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}

}  // namespace b200

// Loads every GEMM variant and sets its attributes up front (called once after the library is loaded).
extern "C" int b200_gemm_init() {
  using namespace b200;
  int e = 0;
#define B200_INIT_BN(BN) \
  e |= gemm_set_attr<__nv_bfloat16, BN, false, false>(); e |= gemm_set_attr<__nv_bfloat16, BN, false, true>(); \
  e |= gemm_set_attr<__nv_bfloat16, BN, true, false>(); e |= gemm_set_attr<__nv_bfloat16, BN, true, true>();
  B200_INIT_BN(64) B200_INIT_BN(128) B200_INIT_BN(256)
#undef B200_INIT_BN
  e |= gemm_set_attr<__nv_bfloat16, 64, false, false, true>() | gemm_set_attr<__nv_bfloat16, 256, false, false, true>() | pair_set_attr<__nv_bfloat16, false, false, true>();
  e |= pair_set_attr<__nv_bfloat16, false, false>(); e |= pair_set_attr<__nv_bfloat16, false, true>(); e |= pair_set_attr<__nv_bfloat16, true, false>(); e |= pair_set_attr<__nv_bfloat16, true, true>();
  e |= gemm_cluster_init() | gemm_kinds_init();
  return e;
}

// 0: single-CTA tiles only; 1: 256 x 256 tiles on CTA pairs where they pay (default); 2: wherever M >= 256 and the tile is 256 wide
extern "C" int b200_gemm_set_pair(int mode) { b200::g_pair_mode = mode < 0 ? 0 : (mode > 2 ? 2 : mode); return 0; }

extern "C" int b200_gemm_set_tma_store(int on) { b200::g_tma_store = on ? 1 : 0; return 0; }

// Tiles of a bf16 product: bf16 results of up to 512 rows 64 columns while such tiles run at once, which shortens what a CTA loads and writes
// (device time, 64 / 128 wide: 333 x 2048 x 512 5.9 / 6.6 us, 512 x 512 x 512 5.6 / 6.4; 1024 x 1536 x 512 (192 tiles) 8.1 / 6.8), 256 once such
// tiles fill the machine. Alone, 64 columns also win at 1024 x 512 (5.8 / 6.5 us), but a chain of products that alternates between kernels pays
// about 3 us a change, and from 600 rows on a block's wider products are 128 wide: LM logits of 1024 tokens 1566 us mixed, 1480 all 128 wide;
// up to 512 tokens all of them are narrow: 1305 -> 1169 us.
static int bf16_tile(const b200::GemmArgs& a, int sms) {
  const long long m = (long long)((a.M + 127) / 128) * a.batch;
  if (a.N <= 64 || (a.p.out_mode == b200::OUT_BF16 && a.M <= 512 && m * ((a.N + 63) / 64) <= sms)) return 64;
  return a.N > 128 && m * ((a.N + 255) / 256) >= sms ? 256 : 128;
}

// bn: columns of a tile, 0 to leave the choice to the operands' rule
extern "C" int b200_gemm_launch(const b200::GemmArgs* args, int bn, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (args->p.M <= 0 || args->p.N <= 0 || args->p.batch <= 0) return 0;
  if (args->dtype != GEMM_BF16 && args->dtype != GEMM_F32 && (args->a_mn || args->b_mn)) return -4;   // 8-bit operands: K-major only (weights are stored [N,K] once at quantisation time)
  if (args->p.out_mode == OUT_I32 && args->dtype == GEMM_E4M3) return -5;
  GemmArgs a = *args;
  if (a.p.splits == 0) {                                     // left to the launcher
    a.p.splits = 1;
    const int ranks = gemm_cluster_ranks(a);
    if (ranks > 1) return gemm_cluster_launch(a, ranks, stream);
  }
  if (a.dtype != GEMM_BF16) return gemm_kinds_launch(a, bn, num_sms, stream);
  switch (bn ? bn : bf16_tile(a, num_sms)) {
    case 64: return launch_major<__nv_bfloat16, 64>(a, stream, num_sms);
    case 128: return launch_major<__nv_bfloat16, 128>(a, stream, num_sms);
    case 256: return launch_major<__nv_bfloat16, 256>(a, stream, num_sms);
    default: return -2;
  }
}

// Tensor-parallel GEMM (see TpParams). bf16 operands, both K-major, batch 1, no split-K, bf16 output.
extern "C" int b200_gemm_tp_launch(const b200::GemmArgs* args, const b200::TpParams* tp, int bn, int num_sms, cudaStream_t stream) {
  using namespace b200;
  const GemmArgs& a = *args;
  if (a.dtype != GEMM_BF16 || a.a_mn || a.b_mn || a.p.batch != 1 || a.p.splits != 1 || a.p.out_mode != OUT_BF16) return -3;
  if (tp->world < 1 || tp->world > TP_MAX_WORLD || tp->blocks_per_rank < 1 || a.p.M != tp->world * tp->blocks_per_rank * BM) return -7;
  if (a.p.K % 8 != 0 || a.p.N % 8 != 0) return -8;
  if (tp->mode == TP_AG_GEMM) {
    if (tp->world > 1 && tp->copy_ctas < 1) return -6;
    return bn == 256 ? launch_tp<256, TP_AG_GEMM>(a, *tp, stream, num_sms) : launch_tp<128, TP_AG_GEMM>(a, *tp, stream, num_sms);
  }
  if (tp->mode == TP_GEMM_RS) {
    if (a.p.ldc != a.p.N || !a.p.vec_ok || a.p.act != ACT_NONE || a.p.aux_out || a.p.aux_in) return -9;
    return bn == 256 ? launch_tp<256, TP_GEMM_RS>(a, *tp, stream, num_sms) : launch_tp<128, TP_GEMM_RS>(a, *tp, stream, num_sms);
  }
  return -2;
}

// One launch for the forward of an expert-parallel MoE layer (see moe_fused_fwd_kernel). g1 / g2 describe the two grouped
// GEMMs exactly as b200_gemm_launch would take them (bf16, both operands K-major, 256-wide tiles, no split-K, batch =
// local experts, m_valid = this rank's slot counters).
extern "C" int b200_moe_fused_fwd(const b200::GemmArgs* g1, const b200::GemmArgs* g2, const b200::MoeFusedArgs* fa, int num_sms, cudaStream_t stream) {
  using namespace b200;
  using T = __nv_bfloat16;
  using S = GemmSmem<T, 256, false, false>;
  constexpr int BN = 256;
  if (fa->world < 1 || fa->world > MOEF_MAX_RANKS || fa->d % 8) return -1;
  const GemmArgs* gs[2] = {g1, g2};
  CUtensorMap tmA[2], tmB[2];
  OutMaps om[2];
  for (int i = 0; i < 2; ++i) {
    const GemmArgs& a = *gs[i];
    if (a.dtype != GEMM_BF16 || a.a_mn || a.b_mn || a.p.splits != 1 || a.p.out_mode != OUT_BF16) return -3;
    int rc = operand_map<T, false>(&tmA[i], a.A, a.M, a.K, a.batch, a.lda, a.strideA, BM);
    if (rc) return 100 + rc;
    rc = operand_map<T, false>(&tmB[i], a.B, a.N, a.K, a.batch, a.ldb, a.strideB, BN);
    if (rc) return 200 + rc;
    om[i].c = tmA[i]; om[i].aux = tmA[i];
    make_out_maps(om[i], a.p, BN);
  }
  static bool attr_done = false;
  if (!attr_done) {
    (void)cudaGetLastError();
    cudaError_t e = cudaFuncSetAttribute(moe_fused_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL);
    if (e != cudaSuccess) return 300 + (int)e;
    attr_done = true;
  }
  // every CTA must be resident at once (CTAs wait on one another): one CTA per SM, grid = SM count, the same for every launch
  moe_fused_fwd_kernel<<<num_sms, GEMM_THREADS, S::TOTAL, stream>>>(tmA[0], tmB[0], g1->p, om[0], tmA[1], tmB[1], g2->p, om[1], *fa);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 400 + (int)e;
}
