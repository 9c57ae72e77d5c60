// Recurrences with one decay per head and token over prompts, in chunks of 128 tokens on tcgen05.
#pragma once

#include "hybrid.cuh"

namespace pace {

// Tokens in rows of `src`: head h reads its query at q_at + (h / per_group) q_step, its key likewise, its value at v_at + h vdim.
struct ChunkArgs {
  const __nv_bfloat16* src;
  int64_t src_stride;
  int q_at, k_at, v_at, q_step, per_group;
  const float* decay;                      // lightning: decay per head (silu of q, k and v); null: the state-space recurrence
  const __nv_bfloat16* dt_raw;
  int64_t dt_stride;
  const float *dt_bias, *neg_a, *d_skip;
  float* state;
  __nv_bfloat16* out;
  int64_t out_stride;
  int heads, dim, vdim;
  // scratch (chunk_umma_bytes) and the places of one round of launches
  int place0, places, v_blocks;
  float *add, *log_decay;
  unsigned char *tiles, *kv;
};

// Whether the chunks of 128 are the faster form of a step (segments: into how many the chunks of 64 would cut a sequence).
bool chunk_umma_pays(const pace_step_t& st, int heads, int vdim, bool lightning, int segments);
// Scratch of a step, 0 where they cannot be taken.
uint64_t chunk_umma_bytes(const pace_step_t& st, int heads, int dim, int vdim, bool lightning);
// False: not for these operands or this much scratch (the chunks of 64 take them).
bool chunk_umma_fits(const pace_step_t& st, const ChunkArgs& a, const void* workspace, uint64_t workspace_bytes);
int chunk_umma(const pace_step_t& st, ChunkArgs a, void* workspace, cudaStream_t s);

}  // namespace pace
