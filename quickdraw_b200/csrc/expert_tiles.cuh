// The grouped product with the weights decoded into tensor memory (expert_tiles.cu), for qd_nvfp4_grouped_matmul.
#pragma once
#include "common.cuh"

namespace qd {

struct ExpertTilesArgs {
    const void* x; const void* codes; const void* scales; const float* global;
    const int32_t* order; const int32_t* boundaries; const float* routing; bf16* y;
    int routes, experts, topk, out_features, in_features, by_token, scatter, global_per_expert;
    unsigned int* status;
};

// Whether the sizes and addresses are ones it takes (out_multiple: weight rows per item, 256; 128 of each bank in the SwiGLU form).
bool expert_tiles_cover(int experts, int out_features, int in_features, int out_multiple, const void* x, const void* codes, const void* scales);
int expert_tiles_matmul(const ExpertTilesArgs& a, cudaStream_t stream);

}  // namespace qd
