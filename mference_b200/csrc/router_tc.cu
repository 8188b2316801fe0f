// Router top-k for large blocks of token rows, with the gate contraction on the tensor cores.
//
// The fp32 summation order of a gate logit is part of the contract (router.cu), which ties the full contraction to the
// fp32 pipe: 4096 rows x 256 experts x 2048 took 124 us, a sixth of a prefill layer.  But only the logits of the experts
// that win have to exist in that order.  So:
//   1. router_gemm_kernel: every logit by tcgen05 with fp32 accumulation.  Activations and gate are exact in the operand
//      type (a bf16 gate turned into fp16 for fp16 activations loses at most 2^-25 per element, see below).
//   2. router_candidates_kernel: a bound on the difference between that value and the ordered fp32 sum turns it into an
//      interval; an expert whose upper end lies below the k-th largest lower end cannot be selected.  The logits of the
//      others - nearly always top_k experts or one more - are formed in the contract's order, and the selection and its
//      weights run on those: the same indices and weights, bit for bit.
// Bound.  With A = sum |w_i x_i| <= |w| |x| (2-norms): the ordered sum is off the true one by at most (d/32 + 5 + 1)
// roundings, below 2^-16 A for d <= 4096; the tensor core adds 16 products at a time to the accumulator, each step
// truncating at worst 17 terms at 2^-24 of the largest magnitude, so below 2^-20 A a step and 2^-12 A over d = 4096,
// 2^-13 A over d = 2048.  How many bits it keeps is not documented: that is an assumption, and measured on products of one sign
// (A = |w| |x|) the sums are off by 2^-16.2 A at d = 2048 and 2^-15.2 A at d = 4096 at most, fp16 or bf16.  2^-11 |w| |x|
// (2^-12 up to d = 2048) covers both and the rounding of the norms.  A norm's squares may vanish in fp32, so 2^-60, more than a
// row's vanished squares can amount to, is added to either norm, and 2^-110 to the bound for sums that vanish.  Rows or gates with
// an infinity or a NaN, and gates beyond the fp16 range where they were converted, make every expert a candidate.
#include "common.cuh"
#include "select.cuh"
#include "tcgen05.cuh"
#include "tmap.cuh"

namespace mfb {

namespace {

// A tile of the contraction: 128 token rows x TN experts, 64 k per stage.  What bounds it is the traffic from L2 into the SMs
// (~40 bytes per cycle and SM): 256 experts per tile where there are tiles for every SM all the same, else 64, and for
// short blocks the contraction cut into up to eight pieces whose sums the next kernel adds.
constexpr uint32_t RG_TM = 128, RG_KC = 64, RG_STAGES = 4, RG_MAX_SPLIT = 8;
constexpr uint32_t RG_A_BYTES = RG_TM * RG_KC * 2;
constexpr uint32_t rg_stage_bytes(uint32_t tn) { return RG_A_BYTES + tn * RG_KC * 2; }
constexpr uint32_t rg_smem(uint32_t tn) { return RG_STAGES * rg_stage_bytes(tn) + 1024; }
constexpr uint32_t RG_THREADS = 192;
constexpr uint32_t RC_KC = 256;                                          // elements per lane-major chunk: eight per lane
constexpr uint32_t RC_WARPS = 4;

__device__ __forceinline__ void rg_tma(void* dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}

// Per expert: the bf16 gate row with every 256-element chunk lane-major (position 8 l + s holds element 32 s + l, the
// order lane l adds them in), its fp16 copy in natural order (fp16 activations only), and a bound on its 2-norm.
__global__ void __launch_bounds__(256) router_gate_prep_kernel(const uint16_t* __restrict__ w, uint32_t d, uint16_t* __restrict__ w_lane,
                                                               uint16_t* __restrict__ w_f16, float* __restrict__ w_norm) {
    __shared__ float red[8];
    __shared__ uint32_t beyond_s;
    const size_t row = (size_t)blockIdx.x * d;
    if (threadIdx.x == 0) beyond_s = 0;
    pdl_wait();
    pdl_release();
    __syncthreads();
    float ss = 0.0f;
    bool beyond = false;
    for (uint32_t i = threadIdx.x; i < d; i += 256) {
        const uint16_t b = w[row + i];
        const float v = __uint_as_float((uint32_t)b << 16);
        ss = fmaf(v, v, ss);
        const uint32_t c = i / RC_KC, e = i % RC_KC;
        w_lane[row + c * RC_KC + (e % 32) * 8 + e / 32] = b;
        if (w_f16) {
            beyond |= !(fabsf(v) <= 65504.0f);
            w_f16[row + i] = __half_as_ushort(__float2half_rn(v));
        }
    }
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    if (beyond) beyond_s = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int i = 0; i < 8; ++i) t += red[i];
        w_norm[blockIdx.x] = beyond_s ? INFINITY : sqrtf(t) + 0x1p-60f;
    }
}

// out[z, t, e] = sum over the z-th part of k of x[t, i] w[e, i].
template <uint32_t RG_TN>
__global__ void __launch_bounds__(RG_THREADS) router_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                 uint32_t n_tokens, uint32_t num_experts, uint32_t chunks_per_part,
                                                                 uint32_t n_chunks_all, uint32_t bf16, float* __restrict__ out,
                                                                 uint32_t* __restrict__ status) {
    constexpr uint32_t RG_STAGE_BYTES = rg_stage_bytes(RG_TN);
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[RG_STAGES], empty[RG_STAGES], done;
    __shared__ uint32_t tmem_base, abort_s;
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t e0 = blockIdx.x * RG_TN, t0 = blockIdx.y * RG_TM, c_first = blockIdx.z * chunks_per_part;
    const uint32_t n_chunks = min(chunks_per_part, n_chunks_all - c_first);
    out += (size_t)blockIdx.z * n_tokens * num_experts;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < RG_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&done, 1);
        abort_s = 0;
        fence_barrier_init();
    }
    __syncthreads();
    pdl_wait();   // in front of the TMEM allocation
    pdl_release();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "n"(RG_TN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    auto fail = [&]() { abort_s = 1; atomicOr(status, STATUS_MBAR_TIMEOUT); };
    if (warp == 0) {
        for (uint32_t c = 0; c < n_chunks; ++c) {
            const uint32_t s = c % RG_STAGES, ph = (c / RG_STAGES) & 1u;
            if (!mbar_wait_warp(&empty[s], ph ^ 1u)) { fail(); break; }
            uint8_t* const st = smem + s * RG_STAGE_BYTES;
            if (elect_one()) {
                mbar_expect_tx(&full[s], RG_STAGE_BYTES);
                rg_tma(st, &map_x, (c_first + c) * RG_KC, t0, &full[s]);
                rg_tma(st + RG_A_BYTES, &map_w, (c_first + c) * RG_KC, e0, &full[s]);
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        // kind::f16: fp16 (0) or bf16 (1) operands, both K-major in the 128-byte swizzle, fp32 D, M = 128, N = RG_TN
        const uint32_t idesc = (1u << 4) | (bf16 << 7) | (bf16 << 10) | ((RG_TN >> 3) << 17) | ((RG_TM >> 4) << 24);
        bool ok = true;
        for (uint32_t c = 0; c < n_chunks; ++c) {
            const uint32_t s = c % RG_STAGES, ph = (c / RG_STAGES) & 1u;
            if (!mbar_wait_warp(&full[s], ph)) { fail(); ok = false; break; }
            tc_fence_after();
            const uint64_t a = smem_desc(smem + s * RG_STAGE_BYTES), b = smem_desc(smem + s * RG_STAGE_BYTES + RG_A_BYTES);
            if (elect_one()) {
#pragma unroll
                for (uint32_t kk = 0; kk < RG_KC / 16; ++kk)
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                        ::"r"(tmem), "l"(a + kk * 2), "l"(b + kk * 2), "r"(idesc), "r"((c | kk) ? 1u : 0u) : "memory");
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&empty[s])) : "memory");
            }
            __syncwarp();
        }
        if (ok && elect_one())
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&done)) : "memory");
        __syncwarp();
    } else {
        const uint32_t q = warp & 3u, t = t0 + 32 * q + lane;
        if (mbar_wait_warp(&done, 0)) {
            tc_fence_after();
#pragma unroll
            for (uint32_t col = 0; col < RG_TN; col += 32) {
                float v[32];
                tmem_ld32(tmem + ((32 * q) << 16) + col, v);
                if (t < n_tokens) {
                    float* dst = out + (size_t)t * num_experts + e0 + col;
#pragma unroll
                    for (uint32_t i = 0; i < 32; ++i)
                        if (e0 + col + i < num_experts) dst[i] = v[i];
                }
            }
        } else {
            fail();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (abort_s) {   // a wait ran out: let the copies that are still in flight land before the CTA gives up its memory
        const long long w0 = clock64();
        while (clock64() - w0 < 400000ll) __nanosleep(1000);
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(RG_TN) : "memory");
}

__device__ __forceinline__ float2 rc_pair(uint32_t v, bool bf16) {
    if (bf16) return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
    return __half22float2(*reinterpret_cast<const __half2*>(&v));
}

// volatile: all loads of a batch stay in front of the first use (left to the compiler they came one L2 round trip at a time)
__device__ __forceinline__ uint4 load_gate(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ float add8(float acc, const uint4& q, const float2 (&v)[4]) {
    const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        acc = fmaf(__uint_as_float(u[j] << 16), v[j].x, acc);
        acc = fmaf(__uint_as_float(u[j] & 0xFFFF0000u), v[j].y, acc);
    }
    return acc;
}

// Four warps for TOK tokens (1 or 4).  A warp brings one token's row into shared memory, forms the intervals and lists the
// candidates; then every warp takes candidates of any token of the block, two at a time, and at the end a warp selects
// for its token.  What the work costs is the candidates' gate rows, 4 KB each at d = 2048 out of L2 (~40 bytes per cycle
// and SM: 255 us for 86,064 rows; measured 531), so the row is kept in 16 bits for the sake of resident blocks (as fp32:
// 664 us).  Short blocks of rows take TOK = 1, which spreads them over more SMs.  PER: most experts per lane.
template <int PER, int TOK>
__global__ void __launch_bounds__(RC_WARPS * 32) router_candidates_kernel(
    const float* __restrict__ approx, uint32_t parts, const uint16_t* __restrict__ x, int x_dtype, uint32_t ldx, uint32_t n_tokens, uint32_t d,
    const uint16_t* __restrict__ w_lane, const float* __restrict__ w_norm, uint32_t num_experts, uint32_t top_k, int mode,
    const float* __restrict__ bias, const __nv_bfloat16* __restrict__ per_expert_scale, const float* __restrict__ correction_bias,
    float route_scale, uint32_t* __restrict__ out_idx, uint16_t* __restrict__ out_w) {
    // [TOK][d] rows, lane-major like w_lane; then per token the logits [num_experts] f32 and the list [num_experts] u16
    extern __shared__ __align__(16) uint16_t x_s[];
    __shared__ uint32_t n_cand_s[TOK], rank_e[TOK][32];
    __shared__ float rank_s[TOK][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t t_block = (size_t)blockIdx.x * TOK, t = t_block + warp;
    const bool bf16 = x_dtype == MFB_DT_BF16, own = warp < TOK && t < n_tokens;
    float* const lg_all = reinterpret_cast<float*>(x_s + (size_t)TOK * d);
    uint16_t* const list_all = reinterpret_cast<uint16_t*>(lg_all + TOK * num_experts);
    float* const lg = lg_all + warp * num_experts;
    uint16_t* const list = list_all + warp * num_experts;
    if (warp < TOK && lane == 0) n_cand_s[warp] = 0;
    pdl_wait();
    pdl_release();
    if (own) {
        // everything the intervals need is requested before anything is used: load by load these were two dozen L2 round
        // trips.  Lane l owns experts l, l + 32, ...; a place past the end repeats the last expert and is dropped below.
        float a[PER], nrm[PER], add[PER];
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint32_t e = min(lane + 32 * j, num_experts - 1);
            a[j] = approx[t * num_experts + e];
            nrm[j] = w_norm[e];
            add[j] = bias ? bias[e] : 0.0f;
        }
        for (uint32_t z = 1; z < parts; ++z) {
            float more[PER];
#pragma unroll
            for (int j = 0; j < PER; ++j) more[j] = approx[((size_t)z * n_tokens + t) * num_experts + min(lane + 32 * j, num_experts - 1)];
#pragma unroll
            for (int j = 0; j < PER; ++j) a[j] += more[j];
        }
        const uint4* src = reinterpret_cast<const uint4*>(x + t * ldx);
        uint16_t* dst = x_s + (size_t)warp * d;
        float ss = 0.0f;
#pragma unroll 4
        for (uint32_t p = lane; p < d / 8; p += 32) {   // elements 8 p ... of the row: lanes 8 (p % 4) + i, place (p / 4) % 8
            const uint4 v = src[p];
            uint16_t* out = dst + (p / 32) * RC_KC + (p & 3u) * 64 + ((p >> 2) & 7u);
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = rc_pair(u[j], bf16);
                ss = fmaf(f.x, f.x, ss);
                ss = fmaf(f.y, f.y, ss);
                out[16 * j] = (uint16_t)(u[j] & 0xFFFFu);
                out[16 * j + 8] = (uint16_t)(u[j] >> 16);
            }
        }
        for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, off);
        const float x_norm = sqrtf(ss) + 0x1p-60f, convert = bf16 ? 0.0f : sqrtf((float)d) * 0x1p-25f;
        float lo[PER], hi[PER];   // interval of every expert's score
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint32_t e = lane + 32 * j;
            lo[j] = hi[j] = -INFINITY;
            if (e < num_experts) {
                float v = a[j] + add[j];
                float eps = fmaf(x_norm, fmaf(nrm[j], d <= 2048 ? 0x1p-12f : 0x1p-11f, convert), fmaf(fabsf(add[j]), 0x1p-22f, 0x1p-110f));
                if (mode == MFB_ROUTER_SQRTSOFTPLUS) {
                    // sqrt(softplus) has slope below 0.33; as evaluated it moves in steps of up to 2^-11.5 near zero
                    v = sqrtsoftplus(v) + (correction_bias ? correction_bias[e] : 0.0f);
                    eps = fmaf(0.34f, eps, 0x1p-11f + fabsf(v) * 0x1p-20f);
                }
                lo[j] = v - eps;
                hi[j] = v + eps;
                if (!(fabsf(lo[j]) <= 3.0e38f)) { lo[j] = -INFINITY; hi[j] = INFINITY; }
                lg[e] = -INFINITY;
            }
        }
        float tau = -INFINITY;   // k-th largest lower end
        uint32_t taken = 0;
        for (uint32_t r = 0; r < top_k; ++r) {
            float bv = -INFINITY;
            int bj = -1;
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (!(taken & (1u << j)) && lo[j] > bv) { bv = lo[j]; bj = j; }
            const uint32_t key = bj < 0 ? 0u : sel_key(bv), best = __reduce_max_sync(0xFFFFFFFFu, key);
            if (best == 0) { tau = -INFINITY; break; }
            const uint32_t who = __ballot_sync(0xFFFFFFFFu, key == best);
            if (lane == (uint32_t)__ffs(who) - 1) taken |= 1u << bj;
            tau = __uint_as_float((best & 0x80000000u) ? (best & 0x7FFFFFFFu) : ~best);
        }
        uint32_t n_cand = 0;     // the candidates, in ascending order of the expert
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint32_t e = lane + 32 * j;
            const bool c = e < num_experts && !(hi[j] < tau);
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, c);
            if (c) list[n_cand + __popc(m & ((1u << lane) - 1u))] = (uint16_t)e;
            n_cand += __popc(m);
        }
        if (lane == 0) n_cand_s[warp] = n_cand;
    }
    __syncthreads();
    // the candidates' logits in the order of router_logits_kernel: lane l adds k = l, l + 32, ... with fma, then the xor
    // butterfly, the bias last
    const uint32_t n_chunks = d / RC_KC;
    uint32_t first = 0;          // candidates of the tokens in front, so that the warps take turns across tokens
#pragma unroll
    for (int k = 0; k < TOK; ++k) {
        const uint32_t n = n_cand_s[k];
        for (uint32_t i = (warp - first) & (RC_WARPS - 1); i < n; i += 2 * RC_WARPS) {   // two at a time
            const bool two = i + RC_WARPS < n;
            const uint32_t e0 = list_all[k * num_experts + i], e1 = list_all[k * num_experts + (two ? i + RC_WARPS : i)];
            const uint4* w0 = reinterpret_cast<const uint4*>(w_lane + (size_t)e0 * d) + lane;
            const uint4* w1 = reinterpret_cast<const uint4*>(w_lane + (size_t)e1 * d) + lane;
            const uint4* xr = reinterpret_cast<const uint4*>(x_s + (size_t)k * d) + lane;
            float acc0 = 0.0f, acc1 = 0.0f;
            for (uint32_t c0 = 0; c0 < n_chunks; c0 += 8) {
                uint4 q0[8], q1[8];
#pragma unroll
                for (uint32_t c = 0; c < 8; ++c) {
                    const uint32_t at = min(c0 + c, n_chunks - 1) * 32;
                    q0[c] = load_gate(w0 + at);
                    q1[c] = load_gate(w1 + at);
                }
#pragma unroll
                for (uint32_t c = 0; c < 8; ++c) {
                    if (c0 + c >= n_chunks) break;
                    const uint4 x8 = xr[(c0 + c) * 32];
                    const float2 v[4] = {rc_pair(x8.x, bf16), rc_pair(x8.y, bf16), rc_pair(x8.z, bf16), rc_pair(x8.w, bf16)};
                    acc0 = add8(acc0, q0[c], v);
                    acc1 = add8(acc1, q1[c], v);
                }
            }
            for (int off = 16; off > 0; off >>= 1) {
                acc0 += __shfl_xor_sync(0xFFFFFFFFu, acc0, off);
                acc1 += __shfl_xor_sync(0xFFFFFFFFu, acc1, off);
            }
            if (lane == 0) {
                lg_all[k * num_experts + e0] = bias ? acc0 + bias[e0] : acc0;
                if (two) lg_all[k * num_experts + e1] = bias ? acc1 + bias[e1] : acc1;
            }
        }
        first += n;
    }
    __syncthreads();
    if (!own) return;
    const uint32_t n_cand = n_cand_s[warp];
    uint32_t e = 0;
    uint16_t wgt = 0;
    // Up to 32 candidates: lane i holds one and counts the ones in front of it (greater score, or the same and a lower index).
    float score = -INFINITY;
    if (lane < n_cand) {
        e = list[lane];
        score = lg[e];
        if (mode == MFB_ROUTER_SQRTSOFTPLUS) score = sqrtsoftplus(score) + (correction_bias ? correction_bias[e] : 0.0f);
    }
    const bool odd = lane < n_cand && !(score > -INFINITY);   // a NaN or -infinity: left to the general form
    if (n_cand <= 32 && n_cand >= top_k && !__any_sync(0xFFFFFFFFu, odd)) {
        uint32_t rank = 0;
        for (uint32_t i = 0; i < n_cand; ++i) {
            const float v = __shfl_sync(0xFFFFFFFFu, score, i);
            rank += (v > score || (v == score && i < lane)) ? 1u : 0u;
        }
        if (lane < n_cand) { rank_e[warp][rank] = e; rank_s[warp][rank] = score; }
        __syncwarp();
        const uint32_t r = lane < n_cand ? lane : 0;
        weight_tail(lg, rank_e[warp][r], rank_s[warp][r], top_k, mode, per_expert_scale, route_scale, lane, e, wgt);
    } else {
        // An expert that is not a candidate reads -infinity: it scores below (softmax) or no higher than (sqrt-softplus: 0 +
        // correction) it would, and it would not be selected.
        select_row(lg, num_experts, top_k, mode, per_expert_scale, correction_bias, route_scale, lane, e, wgt);
    }
    if (lane < top_k) {
        out_idx[t * top_k + lane] = e;
        out_w[t * top_k + lane] = wgt;
    }
}

size_t ws_layout(uint32_t num_experts, uint32_t d, size_t* f16_off, size_t* norm_off) {   // bytes
    const size_t plane = (size_t)num_experts * d * 2;
    *f16_off = plane;
    *norm_off = 2 * plane;
    return 2 * plane + num_experts * sizeof(float);
}

}  // namespace

cudaError_t router_tc_init() {
    cudaError_t e = cudaFuncSetAttribute(router_gemm_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rg_smem(64));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(router_gemm_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rg_smem(256));
    return e;
}

// From the size on where the fp32 kernel's 32 x 32 tiles no longer fit one wave: up to there it takes ~29 us whatever the
// number of rows (d = 2048), the three kernels here ~36.
bool router_tc_usable(const void* x, int x_dtype, uint32_t ldx, uint32_t n_tokens, const void* w, uint32_t num_experts, uint32_t d,
                      size_t workspace_floats, int sm_count) {
    size_t a, b;
    return n_tokens > 64 && ((n_tokens + 31) / 32) * ((num_experts + 31) / 32) > (uint32_t)sm_count && x_dtype != MFB_DT_F32 &&
           d % RC_KC == 0 && d <= 16 * RC_KC && ldx % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0 &&
           workspace_floats * sizeof(float) >= ws_layout(num_experts, d, &a, &b);
}

int32_t router_topk_tc(cudaStream_t s, const void* x, int x_dtype, uint32_t ldx, uint32_t n_tokens, const void* w, uint32_t num_experts,
                       uint32_t d, const float* bias, uint32_t top_k, int mode, const __nv_bfloat16* per_expert_scale,
                       const float* correction_bias, float route_scale, float* logits, float* workspace, size_t workspace_floats, int sm_count,
                       uint32_t* status, uint32_t* out_idx, uint16_t* out_w) {
    size_t f16_off, norm_off;
    const size_t gate_floats = (ws_layout(num_experts, d, &f16_off, &norm_off) + 15) / 16 * 4;
    const uint32_t token_tiles = (n_tokens + RG_TM - 1) / RG_TM, n_chunks = d / RG_KC;
    const bool wide_tile = token_tiles >= (uint32_t)sm_count;
    const uint32_t tn = wide_tile ? 256u : 64u, e_tiles = (num_experts + tn - 1) / tn;
    uint32_t parts = (uint32_t)sm_count / (token_tiles * e_tiles);   // pieces of the contraction, at least four chunks each
    parts = parts > RG_MAX_SPLIT ? RG_MAX_SPLIT : parts;
    if (parts > n_chunks / 4) parts = n_chunks / 4;
    while (parts > 1 && gate_floats + (size_t)parts * n_tokens * num_experts > workspace_floats) --parts;
    if (parts < 1) parts = 1;
    const uint32_t per_part = (n_chunks + parts - 1) / parts;
    parts = (n_chunks + per_part - 1) / per_part;
    if (parts > 1) logits = workspace + gate_floats;
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    uint16_t* w_lane = reinterpret_cast<uint16_t*>(ws);
    uint16_t* w_f16 = x_dtype == MFB_DT_BF16 ? nullptr : reinterpret_cast<uint16_t*>(ws + f16_off);
    float* w_norm = reinterpret_cast<float*>(ws + norm_off);
    CUtensorMap map_x, map_w;
    const CUtensorMapDataType type = x_dtype == MFB_DT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const uint64_t xd[2] = {d, n_tokens}, xs[1] = {(uint64_t)ldx * 2}, wd[2] = {d, num_experts}, wst[1] = {(uint64_t)d * 2};
    const uint32_t xb[2] = {RG_KC, RG_TM}, wb[2] = {RG_KC, tn};
    int32_t rc = encode_tensor_map(&map_x, type, 2, x, xd, xs, xb, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!rc) rc = encode_tensor_map(&map_w, type, 2, w_f16 ? (const void*)w_f16 : w, wd, wst, wb, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    MFB_CUDA(launch_dependent(router_gate_prep_kernel, dim3(num_experts), dim3(256), 0, s, (const uint16_t*)w, d, w_lane, w_f16, w_norm));
    const dim3 grid(e_tiles, token_tiles, parts);
    const uint32_t is_bf16 = x_dtype == MFB_DT_BF16 ? 1u : 0u;
    MFB_CUDA(launch_dependent(wide_tile ? router_gemm_kernel<256> : router_gemm_kernel<64>, grid, dim3(RG_THREADS), rg_smem(tn), s, map_x, map_w,
                              n_tokens, num_experts, per_part, n_chunks, is_bf16, logits, status));
    // four tokens per block where that still gives every SM two blocks
    const uint32_t tok = n_tokens < 8u * (uint32_t)sm_count ? 1u : 4u;
    const auto launch = [&](auto kernel) {
        return launch_dependent(kernel, dim3((n_tokens + tok - 1) / tok), dim3(RC_WARPS * 32), tok * ((size_t)d * 2 + num_experts * 6), s, logits, parts,
                                (const uint16_t*)x, x_dtype, ldx, n_tokens, d, w_lane, w_norm, num_experts, top_k, mode, bias, per_expert_scale,
                                correction_bias, route_scale, out_idx, out_w);
    };
    constexpr int MOST = MFB_MAX_EXPERTS / 32;
    MFB_CUDA(num_experts <= 256 ? launch(tok == 4 ? router_candidates_kernel<8, 4> : router_candidates_kernel<8, 1>)
                                : launch(tok == 4 ? router_candidates_kernel<MOST, 4> : router_candidates_kernel<MOST, 1>));
    count_launches(3);
    return MFB_OK;
}

}  // namespace mfb
