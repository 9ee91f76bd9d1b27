// What the attention kernels of bf16 ragged steps know about a layer (mixers_mma.cu, attend_portions.cu).
#pragma once
#include "mixers.cuh"
#include "mma.cuh"

namespace tmb {

struct AttendParams {
  const bf16* proj;
  bf16* k_pool;
  bf16* v_pool;
  bf16* out;
  float* part;
  unsigned* count;
  const float *q_norm, *k_norm;
  int proj_stride, out_stride, heads, kv_heads, dim, vdim, pool_dim, v_pool_dim, window, keep, splits, gate_at;
  int subs, sub_heads;      // query heads of one key head are served in `subs` units of up to `sub_heads`
  int q_head;               // elements from one query head to the next
  const int* context;       // portions whose keys and values are rows [.. + position] of k_pool and v_pool (see AttendContext), or null
  int context_stride;
  float scale_log2, sink_log2, eps;
  bool value_is_key, even;
  Rotary rotary;
  Blend blend;
  const float* sinks;
  __device__ float sink_of(int head) const { return sinks ? sinks[head] * 1.4426950408889634f : sink_log2; }
};

// Portions on tcgen05 tiles, keys and values through maps (AttentionArgs); `done` false: not for these, nothing was queued.
int AttendPortions(const Queue& q, const StepRows& r, const AttendParams& p, const CUtensorMap* k_map, const CUtensorMap* v_map, bool* done);
int PreparePortions();

}  // namespace tmb
