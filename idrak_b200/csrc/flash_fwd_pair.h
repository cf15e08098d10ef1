// The forward kernel with two query tiles per CTA (flash_fwd_pair.cu).
#pragma once
#include "flash_common.cuh"

namespace idrak {
bool flash_fwd_pair_wanted(const FlashParams& p, int D);
int flash_fwd_pair_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& p, cudaStream_t stream);
}  // namespace idrak
