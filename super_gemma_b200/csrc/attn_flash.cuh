// What the two flash prefill kernels of head_dim 128 share: the units they work on and the partials they leave.
#pragma once

#include <cuda.h>

#include "sgb_common.cuh"
#include "sgb_kernels.h"

namespace sgb {

struct FlashParams {
    const uint32_t* step;
    float* out;
    float* part_acc;     // pieces > 1: [row][piece][128] unnormalised O
    float* part_ml;      // pieces > 1: [row][piece][2] = running max (base-2 exponent units), sum
    uint32_t* status;
    uint32_t m_tokens;   // query tokens in the chunk
    uint32_t n_kv;
    uint32_t window;     // 0 = none
    uint32_t ring;       // TWO_SRC: ring slots
    float scale;
    uint32_t head_group; // kv heads whose query tiles are interleaved in launch order (divides n_kv)
};

// attn_prefill_long.cu: causal, one source, many keys per CTA; grid (units, 1, pieces) and the boxes below.
constexpr uint32_t LONG_BLOCK_N = 128;  // rows of a K or V box
cudaError_t launch_flash_long(const LaunchArgs& a, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashParams& prm,
                              uint32_t units, uint32_t pieces);

}  // namespace sgb
