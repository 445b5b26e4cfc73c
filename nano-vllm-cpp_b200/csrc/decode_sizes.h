// What a decode call of given sizes takes, for the layers above the C ABI that make such a call right away.
#pragma once

#include <cstddef>
#include <cstdint>

namespace nvk {

// Workspace of a call of exactly these sizes (nvk_decode_attention_workspace_bytes: of all smaller ones as well).
size_t decode_mma_workspace_needed(int64_t batch, int num_heads, int num_kv_heads, int head_dim, int64_t max_blocks, int block_size);

}  // namespace nvk
