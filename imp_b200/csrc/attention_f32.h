// The float32 attention kernel of attention_f32.cu; arguments as imp_paged_attention_generic's.  IMP_ERR_UNSUPPORTED, with
// nothing launched, for head sizes other than 64, 128 and 256 and for rows that do not start on 16 bytes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

int imp_attention_f32(float* out, int64_t out_stride, const float* q, int64_t q_stride, const float* k_cache, const float* v_cache,
                      const int* block_table, int bt_stride, const int* seq_of_token, const int* positions, int n_tokens, int n_seqs,
                      int Hq, int Hkv, int Dh, int page_size, int num_pages, float scale, int window, int* status, cudaStream_t stream);
