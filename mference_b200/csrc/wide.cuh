// Expert FFN of a block of rows in fp32 accuracy: interface used by api.cu.
#pragma once

#include "common.cuh"

namespace mfb {

// For handles with the streaming arena and MFB_FLAG_PREFILL_TENSOR_CORE, whose scratch it uses (xs16, acts16, acts).
cudaError_t wide_init(const mfb_moe_config& c);
// a.partial[token * (top_k + 1) + rank, :] for every pair of a.sorted / a.groups: the routed pairs of n_tokens rows x, and behind
// them a shared pair per token where the layer has a shared expert.
cudaError_t wide_ffn(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const Arena& a, const void* x, uint32_t ldx, uint32_t n_tokens,
                     uint32_t max_groups);

}  // namespace mfb
