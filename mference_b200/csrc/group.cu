// Device-side sort of a routing table by (expert, token, rank) and the host-side grouping with the
// reference's validation.  Order and outputs follow PrefillMoEGrouping.groupTokenExpertPairs
// (Sources/Mference/Kernels/Prefill/MoE/PrefillMoEGrouping.swift:90-192): the reference sorts on the CPU
// after reading the whole table back; here a counting sort (per-chunk histogram, column scan, ordered
// scatter) produces the identical order without leaving the device and without atomics on global memory,
// so the result is deterministic.  Up to GROUP_BLOCK_MAX_PAIRS pairs are sorted by one block.
#include <algorithm>
#include <unordered_set>
#include <vector>

#include "common.cuh"

namespace mfb {

namespace {

constexpr uint32_t kNoExpert = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t pair_expert(const uint32_t* idx, uint32_t p, uint32_t n_pairs, uint32_t top_k,
                                                uint32_t slot_mask, uint32_t num_experts) {
    if (p >= n_pairs) return kNoExpert;
    if (!((slot_mask >> (p % top_k)) & 1u)) return kNoExpert;
    const uint32_t e = idx[p];
    return e < num_experts ? e : kNoExpert;
}

// One warp per chunk of GROUP_CHUNK consecutive (token-major) pairs: per-expert counts of the chunk.
__global__ void group_hist_kernel(const uint32_t* __restrict__ idx, uint32_t n_pairs, uint32_t top_k,
                                  uint32_t num_experts, uint32_t slot_mask, uint32_t n_chunks,
                                  uint32_t* __restrict__ chunk_hist) {
    extern __shared__ uint32_t sh[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t chunk = blockIdx.x * (blockDim.x >> 5) + warp;
    uint32_t* h = sh + warp * num_experts;
    for (uint32_t e = lane; e < num_experts; e += 32) h[e] = 0;
    __syncwarp();
    pdl_wait();
    pdl_release();
    if (chunk < n_chunks) {
        uint32_t e[GROUP_CHUNK / 32];
#pragma unroll
        for (uint32_t i = 0; i < GROUP_CHUNK / 32; ++i) e[i] = pair_expert(idx, chunk * GROUP_CHUNK + i * 32 + lane, n_pairs, top_k, slot_mask, num_experts);
#pragma unroll
        for (uint32_t i = 0; i < GROUP_CHUNK / 32; ++i)
            if (e[i] != kNoExpert) atomicAdd(&h[e[i]], 1u);
        __syncwarp();
        for (uint32_t e = lane; e < num_experts; e += 32) chunk_hist[(size_t)chunk * num_experts + e] = h[e];
    }
}

// One block per expert: exclusive scan of that expert's column of chunk_hist over the chunks; total -> counts.
__global__ void group_colscan_kernel(uint32_t* __restrict__ chunk_hist, uint32_t n_chunks, uint32_t num_experts,
                                     uint32_t* __restrict__ counts) {
    __shared__ uint32_t warp_sums[8];
    __shared__ uint32_t carry_s;
    const uint32_t e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry_s = 0;
    pdl_wait();
    pdl_release();
    __syncthreads();
    for (uint32_t base = 0; base < n_chunks; base += blockDim.x) {
        const uint32_t c = base + tid;
        const uint32_t v = c < n_chunks ? chunk_hist[(size_t)c * num_experts + e] : 0u;
        uint32_t incl = v;
        for (uint32_t off = 1; off < 32; off <<= 1) {
            const uint32_t n = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += n;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        uint32_t warp_base = 0;
        for (uint32_t w = 0; w < warp; ++w) warp_base += warp_sums[w];
        const uint32_t carry = carry_s;
        if (c < n_chunks) chunk_hist[(size_t)c * num_experts + e] = carry + warp_base + incl - v;
        __syncthreads();
        if (tid == blockDim.x - 1) carry_s = carry + warp_base + incl;
        __syncthreads();
    }
    if (tid == 0) counts[e] = carry_s;
}

// A block of THREADS: expert offsets (exclusive scan of the counts s_cnt in expert order, absent experts marked), the compacted group
// list and the optional shared-expert group over all tokens, a few neighbouring experts per thread.  s_first: every expert's offset, absent
// ones too, in shared memory.  Of the blocks that call it one writes.  Returns the number of pairs; s_first is complete behind the next
// barrier.  (One warp, 32 experts a round, took 8 dependent rounds for 256 experts; in a kernel of its own between the column scan and the
// scatter that was 5 us of the 24 us sort of 4096 x 8 pairs; calls of 2500 and 4096 skewed rows 316 -> 308 and 428 -> 424 us.)
template <uint32_t THREADS>
__device__ __forceinline__ uint32_t group_experts(const uint32_t* s_cnt, uint32_t num_experts, uint32_t n_tokens, int append_shared, bool write, uint32_t* s_first,
                                                  uint32_t* __restrict__ offsets, mfb_group* __restrict__ groups, uint32_t* __restrict__ n_groups) {
    constexpr uint32_t WARPS = THREADS / 32;
    __shared__ uint32_t s_sum[2][WARPS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per = (num_experts + THREADS - 1) / THREADS, e0 = threadIdx.x * per;
    uint32_t cnt = 0, live = 0;
    for (uint32_t e = e0; e < min(e0 + per, num_experts); ++e) { cnt += s_cnt[e]; live += s_cnt[e] ? 1u : 0u; }
    uint32_t ic = cnt, il = live;
    for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, ic, off), b = __shfl_up_sync(0xFFFFFFFFu, il, off);
        if (lane >= off) { ic += a; il += b; }
    }
    if (lane == 31) { s_sum[0][warp] = ic; s_sum[1][warp] = il; }
    __syncthreads();
    const uint32_t c = lane < WARPS ? s_sum[0][lane] : 0u, l = lane < WARPS ? s_sum[1][lane] : 0u;
    uint32_t run = ic - cnt + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? c : 0u), g = il - live + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? l : 0u);
    const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, c), ng = __reduce_add_sync(0xFFFFFFFFu, l);
    for (uint32_t e = e0; e < min(e0 + per, num_experts); ++e) {
        const uint32_t n = s_cnt[e];
        s_first[e] = run;
        if (write) {
            offsets[e] = n ? run : 0xFFFFFFFFu;
            if (n) {
                groups[g].expert = e;
                groups[g].pair_start = run;
                groups[g].pair_count = n;
            }
        }
        g += n ? 1u : 0u;
        run += n;
    }
    if (write && threadIdx.x == 0) {
        if (append_shared) {
            groups[ng].expert = num_experts;
            groups[ng].pair_start = total;
            groups[ng].pair_count = n_tokens;
        }
        *n_groups = ng + (append_shared ? 1u : 0u);
    }
    return total;
}

// The shared expert's rows behind the routed pairs: thread `at` of `threads`.
__device__ __forceinline__ void group_shared_rows(mfb_pair* __restrict__ sorted, uint32_t base, uint32_t n_tokens, uint32_t num_experts, uint32_t top_k, uint32_t at,
                                                  uint32_t threads) {
    for (uint32_t t = at; t < n_tokens; t += threads) {
        mfb_pair p;
        p.token = t; p.expert = num_experts; p.rank = top_k; p.weight_bits = 0x3C00u; /* fp16 1.0 */
        sorted[base + t] = p;
    }
}

// A routing table without a pair.
__global__ void group_empty_kernel(uint32_t num_experts, uint32_t n_tokens, uint32_t top_k, int append_shared, uint32_t* __restrict__ offsets,
                                   uint32_t* __restrict__ counts, mfb_group* __restrict__ groups, uint32_t* __restrict__ n_groups, mfb_pair* __restrict__ sorted) {
    __shared__ uint32_t s_cnt[MFB_MAX_EXPERTS], s_first[MFB_MAX_EXPERTS];
    pdl_wait();
    pdl_release();
    for (uint32_t e = threadIdx.x; e < num_experts; e += blockDim.x) { s_cnt[e] = 0u; counts[e] = 0u; }
    __syncthreads();
    group_experts<256>(s_cnt, num_experts, n_tokens, append_shared, true, s_first, offsets, groups, n_groups);
    if (append_shared) group_shared_rows(sorted, 0u, n_tokens, num_experts, top_k, threadIdx.x, blockDim.x);
}

// The whole sort in one block, for up to GROUP_BLOCK_MAX_PAIRS pairs: a warp per `part` consecutive pairs, eight per lane at
// most, all requested at once.  One walk over a warp's pairs gives their expert's count and each pair's rank within the warp's.
// Latency throughout: the kernels of the general form took 28 us for 203 x 8 pairs (eight dependent rounds per warp
// and a launch between any two steps), this one 10; beyond the limit one SM has too much to write.
constexpr uint32_t GROUP_BLOCK_WARPS = 32, GROUP_BLOCK_ROUNDS = 8, GROUP_BLOCK_MAX_PAIRS = GROUP_BLOCK_WARPS * GROUP_BLOCK_ROUNDS * 32;

__global__ void __launch_bounds__(GROUP_BLOCK_WARPS * 32) group_block_kernel(
    const uint32_t* __restrict__ idx, const uint16_t* __restrict__ route_w, uint32_t n_pairs, uint32_t part, uint32_t n_tokens, uint32_t top_k,
    uint32_t num_experts, uint32_t slot_mask, int append_shared, uint32_t* __restrict__ offsets, uint32_t* __restrict__ counts,
    mfb_group* __restrict__ groups, uint32_t* __restrict__ n_groups, mfb_pair* __restrict__ sorted, uint32_t* __restrict__ inv) {
    __shared__ uint32_t s_cnt[MFB_MAX_EXPERTS], s_first[MFB_MAX_EXPERTS];
    extern __shared__ uint16_t s_run[];   // [warp][expert]: the warp's pairs of the expert so far; then the earlier warps'
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint16_t* const run = s_run + warp * num_experts;
    for (uint32_t e = lane; e < num_experts; e += 32) run[e] = 0;
    __syncwarp();
    pdl_wait();
    pdl_release();
    const uint32_t first = warp * part, last = min(first + part, n_pairs);
    uint32_t expert[GROUP_BLOCK_ROUNDS], rank[GROUP_BLOCK_ROUNDS], weight[GROUP_BLOCK_ROUNDS];
#pragma unroll
    for (uint32_t i = 0; i < GROUP_BLOCK_ROUNDS; ++i) {
        const uint32_t p = first + i * 32 + lane;
        expert[i] = pair_expert(idx, p, last, top_k, slot_mask, num_experts);
        weight[i] = p < last && route_w ? (uint32_t)route_w[p] : 0u;
    }
#pragma unroll
    for (uint32_t i = 0; i < GROUP_BLOCK_ROUNDS; ++i) {
        if (i * 32 >= part) break;
        const uint32_t e = expert[i], peers = __match_any_sync(0xFFFFFFFFu, e), before = __popc(peers & ((1u << lane) - 1u));
        rank[i] = e != kNoExpert ? run[e] + before : 0u;
        __syncwarp();
        if (e != kNoExpert && before == 0) run[e] += (uint16_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < num_experts; e += blockDim.x) {
        uint32_t sum = 0;
#pragma unroll 8
        for (uint32_t w = 0; w < GROUP_BLOCK_WARPS; ++w) {
            const uint32_t c = s_run[w * num_experts + e];
            s_run[w * num_experts + e] = (uint16_t)sum;
            sum += c;
        }
        s_cnt[e] = sum;
        counts[e] = sum;
    }
    __syncthreads();
    const uint32_t total = group_experts<GROUP_BLOCK_WARPS * 32>(s_cnt, num_experts, n_tokens, append_shared, true, s_first, offsets, groups, n_groups);
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < GROUP_BLOCK_ROUNDS; ++i) {
        const uint32_t p = first + i * 32 + lane, e = expert[i];
        if (e == kNoExpert) continue;
        const uint32_t pos = s_first[e] + run[e] + rank[i];
        mfb_pair out;
        out.token = p / top_k; out.expert = e; out.rank = p % top_k; out.weight_bits = weight[i];
        sorted[pos] = out;
        if (inv) inv[p] = pos;
    }
    if (append_shared) group_shared_rows(sorted, total, n_tokens, num_experts, top_k, threadIdx.x, blockDim.x);
}

// One warp per chunk again: walk the chunk in order, 32 pairs per round; a pair's slot is its expert's
// offset + pairs of that expert in earlier chunks + earlier in this chunk.  Every block scans the counts for the offsets.
constexpr uint32_t SCATTER_WARPS = 4;
__global__ void __launch_bounds__(SCATTER_WARPS * 32) group_scatter_kernel(const uint32_t* __restrict__ idx, const uint16_t* __restrict__ route_w,
                                     uint32_t n_pairs, uint32_t n_tokens, uint32_t top_k, uint32_t num_experts, uint32_t slot_mask, int append_shared,
                                     uint32_t n_chunks, const uint32_t* __restrict__ chunk_hist, const uint32_t* __restrict__ counts,
                                     uint32_t* __restrict__ offsets, mfb_group* __restrict__ groups, uint32_t* __restrict__ n_groups,
                                     mfb_pair* __restrict__ sorted, uint32_t* __restrict__ inv) {
    extern __shared__ uint32_t sh[];
    uint32_t* s_off = sh;  // [num_experts] expert offsets, shared by the block; then the counts; then a row per warp
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = SCATTER_WARPS;
    uint32_t* s_cnt = sh + num_experts;
    uint32_t* run = sh + (2 + warp) * num_experts;
    pdl_wait();
    pdl_release();
    for (uint32_t e = threadIdx.x; e < num_experts; e += blockDim.x) s_cnt[e] = counts[e];
    __syncthreads();
    const uint32_t total = group_experts<SCATTER_WARPS * 32>(s_cnt, num_experts, n_tokens, append_shared, blockIdx.x == 0, s_off, offsets, groups, n_groups);
    __syncthreads();
    if (append_shared) group_shared_rows(sorted, total, n_tokens, num_experts, top_k, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    const uint32_t chunk = blockIdx.x * warps + warp;
    if (chunk >= n_chunks) return;
    uint32_t expert[GROUP_CHUNK / 32], weight[GROUP_CHUNK / 32];   // all requested at once: round by round they were eight round trips
#pragma unroll
    for (uint32_t i = 0; i < GROUP_CHUNK / 32; ++i) {
        const uint32_t p = chunk * GROUP_CHUNK + i * 32 + lane;
        expert[i] = pair_expert(idx, p, n_pairs, top_k, slot_mask, num_experts);
        weight[i] = p < n_pairs && route_w ? (uint32_t)route_w[p] : 0u;
    }
    for (uint32_t e = lane; e < num_experts; e += 32) run[e] = s_off[e] + chunk_hist[(size_t)chunk * num_experts + e];
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < GROUP_CHUNK / 32; ++i) {
        const uint32_t p = chunk * GROUP_CHUNK + i * 32 + lane, e = expert[i];
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, e);
        const uint32_t before = __popc(peers & ((1u << lane) - 1u));
        uint32_t pos = 0;
        if (e != kNoExpert) pos = run[e] + before;
        __syncwarp();
        if (e != kNoExpert && before == 0) run[e] += __popc(peers);
        __syncwarp();
        if (e != kNoExpert) {
            mfb_pair out;
            out.token = p / top_k; out.expert = e; out.rank = p % top_k;
            out.weight_bits = weight[i];
            sorted[pos] = out;
            if (inv) inv[p] = pos;
        }
    }
}

}  // namespace

cudaError_t launch_group(cudaStream_t s, const uint32_t* idx, const uint16_t* route_w, uint32_t n_tokens,
                         uint32_t top_k, uint32_t num_experts, uint32_t slot_mask, int append_shared,
                         Arena& a, mfb_pair* out_sorted, uint32_t* out_offsets,
                         uint32_t* out_counts, mfb_group* out_groups, uint32_t* out_n_groups, uint32_t* inv) {
    const uint32_t n_pairs = n_tokens * top_k;
    const uint32_t n_chunks = (n_pairs + GROUP_CHUNK - 1) / GROUP_CHUNK;
    const uint32_t warps = SCATTER_WARPS;
    const uint32_t blocks = (n_chunks + warps - 1) / warps;
    if (n_pairs > 0 && n_pairs <= GROUP_BLOCK_MAX_PAIRS) {
        const uint32_t part = (n_pairs + GROUP_BLOCK_WARPS * 32 - 1) / (GROUP_BLOCK_WARPS * 32) * 32;
        count_launches(1);
        return launch_dependent(group_block_kernel, dim3(1), dim3(GROUP_BLOCK_WARPS * 32), GROUP_BLOCK_WARPS * num_experts * sizeof(uint16_t), s, idx, route_w,
                                n_pairs, part, n_tokens, top_k, num_experts, slot_mask, append_shared, out_offsets, out_counts, out_groups, out_n_groups,
                                out_sorted, inv);
    }
    if (n_chunks == 0) {
        count_launches(1);
        return launch_dependent(group_empty_kernel, dim3(1), dim3(256), 0, s, num_experts, n_tokens, top_k, append_shared, out_offsets, out_counts, out_groups,
                                out_n_groups, out_sorted);
    }
    MFB_TRY(launch_dependent(group_hist_kernel, dim3(blocks), dim3(warps * 32), warps * num_experts * sizeof(uint32_t), s,
                             idx, n_pairs, top_k, num_experts, slot_mask, n_chunks, a.chunk_hist));
    MFB_TRY(launch_dependent(group_colscan_kernel, dim3(num_experts), dim3(256), 0, s, a.chunk_hist, n_chunks, num_experts, out_counts));
    MFB_TRY(launch_dependent(group_scatter_kernel, dim3(blocks), dim3(warps * 32), (warps + 2) * num_experts * sizeof(uint32_t), s, idx, route_w, n_pairs, n_tokens,
                             top_k, num_experts, slot_mask, append_shared, n_chunks, a.chunk_hist, out_counts, out_offsets, out_groups, out_n_groups, out_sorted, inv));
    count_launches(3);
    return cudaSuccess;
}

}  // namespace mfb

// ---------------------------------------------------------------------------------------------------------
// Host-side grouping (validation, sort keys, tiles) for callers that hold the routing table on the host.

extern "C" int32_t mfb_moe_group_host(const mfb_pair* pairs, int64_t n_pairs, int64_t query_count, int64_t top_k,
                                      int64_t num_experts, int64_t tile_expert_count, const uint64_t* expert_sort_keys,
                                      int64_t n_sort_keys, mfb_pair* out_sorted, uint32_t* out_offsets,
                                      uint32_t* out_counts, mfb_group* out_groups, uint32_t* out_n_groups,
                                      mfb_tile* out_tiles, uint32_t* out_n_tiles, uint32_t* err_a, uint32_t* err_b) {
    uint32_t dummy_a = 0, dummy_b = 0;
    if (!err_a) err_a = &dummy_a;
    if (!err_b) err_b = &dummy_b;
    *err_a = *err_b = 0;
    if (out_n_groups) *out_n_groups = 0;
    if (out_n_tiles) *out_n_tiles = 0;
    auto fail = [&](int32_t code, uint32_t a, uint32_t b, const char* what) {
        *err_a = a; *err_b = b;
        mfb::set_error("grouping: %s (%u, %u)", what, a, b);
        return code;
    };
    if (query_count < 0) return fail(MFB_ERR_GROUP_INVALID_QUERY_COUNT, (uint32_t)query_count, 0, "queryCount must be non-negative");
    if (top_k <= 0) return fail(MFB_ERR_GROUP_INVALID_TOP_K, (uint32_t)top_k, 0, "topK must be positive");
    if (num_experts <= 0) return fail(MFB_ERR_GROUP_INVALID_NUM_EXPERTS, (uint32_t)num_experts, 0, "numExperts must be positive");
    if (tile_expert_count < 1 || tile_expert_count > 16)
        return fail(MFB_ERR_GROUP_INVALID_TILE_EXPERT_COUNT, (uint32_t)tile_expert_count, 0, "tileExpertCount must be in 1...16");
    if (expert_sort_keys && n_sort_keys != num_experts)
        return fail(MFB_ERR_GROUP_SORT_KEY_COUNT_MISMATCH, (uint32_t)num_experts, (uint32_t)n_sort_keys, "expert sort key count");
    if (n_pairs != query_count * top_k)
        return fail(MFB_ERR_GROUP_PAIR_COUNT_MISMATCH, (uint32_t)(query_count * top_k), (uint32_t)n_pairs, "route pair count");
    if (!pairs && n_pairs > 0) return fail(MFB_ERR_INVALID_ARGUMENT, 0, 0, "pairs is NULL");

    std::unordered_set<uint64_t> seen;
    seen.reserve((size_t)n_pairs * 2 + 1);
    for (int64_t i = 0; i < n_pairs; ++i) {
        const mfb_pair& p = pairs[i];
        if (p.token >= (uint32_t)query_count) return fail(MFB_ERR_GROUP_TOKEN_OUT_OF_RANGE, p.token, 0, "route token out of range");
        if (p.rank >= (uint32_t)top_k) return fail(MFB_ERR_GROUP_RANK_OUT_OF_RANGE, p.rank, 0, "route rank out of range");
        if (p.expert >= (uint32_t)num_experts) return fail(MFB_ERR_GROUP_EXPERT_OUT_OF_RANGE, p.expert, 0, "route expert out of range");
        if (!seen.insert(((uint64_t)p.token << 32) | p.rank).second)
            return fail(MFB_ERR_GROUP_DUPLICATE_TOKEN_RANK, p.token, p.rank, "duplicate route pair");
    }
    std::vector<mfb_pair> v(pairs, pairs + n_pairs);
    std::sort(v.begin(), v.end(), [&](const mfb_pair& l, const mfb_pair& r) {
        if (expert_sort_keys) {
            const uint64_t lk = expert_sort_keys[l.expert], rk = expert_sort_keys[r.expert];
            if (lk != rk) return lk < rk;
        }
        if (l.expert != r.expert) return l.expert < r.expert;
        if (l.token != r.token) return l.token < r.token;
        return l.rank < r.rank;
    });
    for (int64_t e = 0; e < num_experts; ++e) { out_offsets[e] = 0xFFFFFFFFu; out_counts[e] = 0; }
    uint32_t ng = 0;
    for (size_t i = 0; i < v.size();) {
        const uint32_t e = v[i].expert;
        const size_t start = i;
        while (i < v.size() && v[i].expert == e) ++i;
        out_offsets[e] = (uint32_t)start;
        out_counts[e] = (uint32_t)(i - start);
        out_groups[ng++] = mfb_group{e, (uint32_t)start, (uint32_t)(i - start)};
    }
    uint32_t nt = 0;
    for (uint32_t gs = 0; gs < ng;) {
        const uint32_t ge = std::min<uint32_t>(ng, gs + (uint32_t)tile_expert_count);
        if (out_tiles) {
            out_tiles[nt] = mfb_tile{gs, ge - gs, out_groups[gs].pair_start,
                                     out_groups[ge - 1].pair_start + out_groups[ge - 1].pair_count - out_groups[gs].pair_start};
        }
        ++nt;
        gs = ge;
    }
    for (size_t i = 0; i < v.size(); ++i) out_sorted[i] = v[i];
    if (out_n_groups) *out_n_groups = ng;
    if (out_n_tiles) *out_n_tiles = nt;
    return MFB_OK;
}
