// Causal attention of a prompt chunk (seq_flash.cu), head dimension 256.
#pragma once
#include "common.cuh"

int seq_flash_attention(const bf16* q, const bf16* qg, const bf16* k_cache, const bf16* v_cache, bf16* out, int tokens, int position0,
                        int capacity, int q_heads, int kv_heads, cudaStream_t stream);
