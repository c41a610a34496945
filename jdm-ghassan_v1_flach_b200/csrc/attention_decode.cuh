// Decode attention on the tensor cores (attention_decode.cu).
#pragma once

#include "common.cuh"

namespace b200 {

constexpr int FLASH_MIN_T = 128;             // steps from which a prompt takes the tensor-core kernel (attention_flash.cu)

struct DecodeMmaArgs {
    const float* q = nullptr;                // [batch, H, hd]
    const uint16_t *kc = nullptr, *vc = nullptr;   // fp16 [rows, KV*hd]
    float* out = nullptr;                    // [batch, H, hd]
    float* part = nullptr;                   // [batch, H, splits, hd + 4]: o, m, l of each piece
    const int32_t* page_table = nullptr;     // [batch, max_pages] or null (ring)
    const int32_t* seq_lens = nullptr;       // [batch] or null
    int H = 0, KV = 0, hd = 0, group = 0, splits = 1;
    int cur_len = 0, j0 = 0;                 // ring: positions [j0, cur_len)
    int ring_start = 0, pinned = 0, ring_cap = 1;
    int max_pages = 0, page = 1;
    float scale = 1.0f;
    bool dry = false;                        // launch_pdl's flag: always a real launch here
};
bool attention_decode_mma_takes(const DecodeMmaArgs& a);
int attention_decode_mma(DecodeMmaArgs a, int batch, int max_len, float* fixed_part = nullptr, int64_t fixed_floats = 0);

}  // namespace b200
