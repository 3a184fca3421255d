// One decoding step's attention: a few query rows against a key/value cache (see attention_decode.cu).
#pragma once
#include "common.cuh"

namespace mt {

struct DecodeStep {
  const void* q; void* k_cache; void* v_cache; void* o;
  mt_strides3 sq, sc, so;
  int64_t batch, heads, kv_heads, q_len, kv_len, head_dim;
  float scale;
  int causal_offset, dtype;
  // fused preparation (q_len = 1): append k_new / v_new at cache row append_slot (kv_len counts it),
  // after rotary embedding and QK-norm of q and k when the tables' rows are given
  int fused;
  const void* k_new; const void* v_new;
  mt_strides3 sk_new, sv_new;
  int64_t append_slot;
  const float* cos_row; const float* sin_row;
  float eps;
  int early_cache;      // rows held before this step were not written by the kernel just in front in the stream
};

int attn_decode_step(const DecodeStep& a, cudaStream_t st);
int kv_append(const void* k_new, const void* v_new, void* k_cache, void* v_cache, mt_strides3 sk, mt_strides3 sv,
              mt_strides3 scache, int64_t batch, int64_t heads, int64_t n_new, int64_t pos0, int64_t max_len,
              int64_t head_dim, int dtype, cudaStream_t st);

}  // namespace mt
