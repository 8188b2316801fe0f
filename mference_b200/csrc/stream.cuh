// Decode-time expert FFN, streaming form: interface used by api.cu.
#pragma once

#include <functional>

#include "common.cuh"

namespace mfb {

// What the path keeps in the handle besides Arena::acts, which holds the hidden activations.
struct StreamArena {
    uint8_t* base = nullptr;       // the allocation that holds the others
    // Either form of the rows lies in xr and the remainders behind it (xs likewise): fp16 numbers, or [tokens][4][d] digits (digits.cu).
    __half* xr = nullptr;          // [tokens][d] activations as fp16 times a power of two, in the routed codes' order
    __half* xs = nullptr;          // the same in the shared expert's order, where that differs
    __half *xr_rest = nullptr, *xs_rest = nullptr;   // [tokens][d] remainders of the rows that fp16 does not hold: marked ones
    float* unit = nullptr;         // [tokens] what turns a row's sums back (the row is scaled into the range of fp16); negative: a marked row
    __half* split = nullptr;       // [tokens * (top_k + 1)][2][f] hidden activations as heads and remainders, or [..][4][f] digits
    float2 *tr = nullptr, *ts = nullptr;   // [tokens][d / 32] at most: unit and sum of the scale groups of xr and xs (digits.cu)
    float2* th = nullptr;          // [tokens * (top_k + 1)][f / 32] at most: the same of the hidden rows
    uint32_t* hidden_max = nullptr;   // [tokens * (top_k + 1)] per sorted pair: bits of the largest hidden activation
    WorkTile* tiles = nullptr;
    uint32_t* n_tiles = nullptr;
    uint32_t* arrivals = nullptr;  // zero between calls (launch_row_route)
};

constexpr uint32_t STREAM_MAX_TOKENS = 64;
constexpr uint32_t STREAM_LONGEST = 6912;   // of d and f: two rows of so many elements, as heads and remainders, and two stages fit a CTA

bool stream_supported(const mfb_moe_config& c);
cudaError_t stream_alloc(const mfb_moe_config& c, StreamArena* a);
void stream_free(StreamArena* a);
// Activations of n_tokens rows into the arena; with norm_eps >= 0 the rows are RMS-normalised first and also stored in xn.
// pending: the rows are pending->y once its combination is made, which this does.
cudaError_t stream_prep(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const StreamArena& a, const void* x, uint32_t ldx,
                        uint32_t n_tokens, const __nv_bfloat16* norm_w, float norm_eps, void* xn, const PendingCombine* pending = nullptr);
// Work list of a sorted pair list (launch_route_small writes the same one).
uint32_t stream_tile_rows(const mfb_moe_config& c, uint32_t n_tokens);
uint32_t stream_shared_rows(const mfb_moe_config& c, uint32_t n_tokens);
cudaError_t stream_tiles(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const StreamArena& a, bool shared, uint32_t tile_rows,
                         uint32_t shared_rows, const mfb_group* groups, const uint32_t* n_groups);
// Both FFN phases over the work list: fp32 rows of `partial` per (token, rank slot).
cudaError_t stream_ffn(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const StreamArena& a, uint32_t n_tokens, bool shared,
                       const mfb_pair* sorted, float* acts, float* partial, int sm_count,
                       const std::function<cudaError_t()>& between = nullptr);   // called between the phases

}  // namespace mfb
