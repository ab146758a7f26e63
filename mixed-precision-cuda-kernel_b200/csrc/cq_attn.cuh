// The decode attention on mma.sync (cq_attn.cu), called by cq_attn_decode for the calls it takes.
#pragma once

#include "cq_common.cuh"

// Whether the kernel takes such a call (on 16-byte aligned buffers); step: with the step's rotation in the same launch.
bool cq_attn_mma_takes(int sequences, int n_heads, int n_kv_heads, int head_dim, int max_seq, bool step);
// k_new, v_new and the rotary tables: the step's rotation and cache write in the same launch (all 16-byte aligned).
// counters, part: the workspace as cq_attn_decode lays it out, partial results of up to `most` ranges per head.
int cq_attn_mma_launch(const void* q, const void* k_cache, const void* v_cache, const long long* position, void* out, int sequences,
                       int n_heads, int n_kv_heads, int head_dim, int max_seq, float scale, int most, unsigned int* counters,
                       float* part, cudaStream_t stream, const void* k_new = nullptr, const void* v_new = nullptr,
                       const float* cos_table = nullptr, const float* sin_table = nullptr);
