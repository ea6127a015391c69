// Launch interface of the fused linear-attention kernels (plain C structs).
#pragma once
#include "flash_sm100.h"

namespace b200 {

// Sequence-parallel exchange of the slice totals, done by the attention kernels themselves over NVLink peer memory.
// The state pass of a rank (role 1) writes its total into its OWN symmetric buffer and then raises one flag per
// (consumer rank, batch x head); the main pass (role 2) of a consumer waits for the flags of the ranks it depends on,
// pulls their totals with plain peer loads in rank order (so every run sums in the same order), keeps the sum in
// `prefix` and acknowledges. A total is double-buffered by call parity and is only overwritten once every consumer has
// acknowledged the call two earlier. The call counter is a device word that the last CTA of the main pass advances,
// so a captured graph replays with fresh epochs. All waits are bounded.
constexpr int LA_MAX_WORLD = 8;
struct LaExchange {
  float* state[LA_MAX_WORLD];       // every rank's totals [2][B*H][hd*hd + hd] fp32 (peer-mapped)
  uint32_t* flags[LA_MAX_WORLD];    // every rank's arrival flags [world][B*H] (peer-mapped): flags[c][r * BH + bh] = epoch
  uint32_t* acks[LA_MAX_WORLD];     // every rank's release flags [world][B*H] (peer-mapped): acks[r][c * BH + bh] = epoch
  float* prefix;                    // local [B*H][hd*hd + hd]: the sum the main pass started from (the backward needs it again)
  uint32_t* words;                  // local: [0] calls so far, [1] retired CTAs of the main pass
  long long wait_cycles;
  int rank, world;                  // world <= 1: no exchange
  int dir;                          // 0: sum over the LOWER ranks (forward states), 1: over the HIGHER ranks (backward)
  int role;                         // 0: none, 1: publish this slice's total, 2: consume
};

struct LinAttnArgs {
  AttnTensor q, k, v, o;                     // bf16 [B, S, H, hd] (any strides, hd contiguous)
  AttnTensor dout, dq, dk, dv;               // backward
  AttnTensor g;                              // backward scratch, bf16: G = dO / D (written by the G pass, read by both gradient kernels)
  AttnTensor o_lo;                           // optional bf16 remainder O - bf16(O): written by forward, read by backward.
                                             // dden = -(dO . O) / D is one half of a difference of nearly equal terms
                                             // (S^T G against (G . O) z); 8 mantissa bits of O are not enough for it
  float* den;                                // [B, H, S] fp32: denominators incl. eps (written by forward, read by backward)
  float* dden;                               // backward scratch, [B, H, S] fp32: -(G . O)
  const float* s_in;                         // optional [B*H][hd*hd + hd] fp32: state (row-major [d_k][d_v]) then z
  float* s_out;                              // optional, same layout: state after the last token (forward / state pass)
  const float* ds_in;                        // backward 2, optional: dS, dz flowing in from the tokens after this slice
  float* ds_out;                             // backward 2, optional: dS, dz at the first token (for the slices before it)
  int B, H, S, hd;
  float scale, eps;
  int kind;                                  // 0: ELU + 1, 1: ReLU^2
  int state_only;                            // forward: only accumulate the state (reads K, V; writes s_out)
  uint32_t* status;
  float* seg;                                // n_seg > 1: [B*H][n_seg][hd*hd + hd] fp32 workspace for the states between segments
  int n_seg, seg_chunks;                     // the sequence is walked as n_seg segments of seg_chunks chunks by as many CTAs
  float* dseg;                               // whole backward, n_seg > 1: the workspace of dK / dV (`seg` holds the forward's states)
  LaExchange sx;
};

}  // namespace b200

extern "C" int b200_linattn(const b200::LinAttnArgs* a, int which, cudaStream_t st);
