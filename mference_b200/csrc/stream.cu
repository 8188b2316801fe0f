// Decode-time expert FFN, streaming form: every warp fetches its own packed rows into a ring of its own with asynchronous
// copies and multiplies the codes on the tensor cores as they lie there.
//
// What bounds it is the integer unpacking of the codes (a logic operation and up to one shift per two codes, at half rate) with the
// copies: at two bits per code a layer's bytes cross HBM faster than the codes can be masked.  So nothing else may
// stand in the way: a warp owns sixteen matrix rows (gate and up of the same rows, or two sixteen-row tiles of down), no
// barrier and no other warp takes part in its loop, and with sixteen warps per SM some 45-90 KB are in flight.  The SIMT
// kernels it replaces (decode.cu) spent three instructions on every code and row: 2018 us per layer of thirteen rows at
// hidden 4096 / intermediate 2048 with 2-bit codes.
//
// Arithmetic: the reference's factored form (Sources/Mference/Metal/MoE/moe.metal:349-529, 902-1062) per scale group,
// acc += scale * sum(code x) + bias * sum(x), fp32.  sum(code x) comes from mma.m16n8k16 on codes that are fp16 subnormals
// (a code masked in place is code * 2^(bit - 24); the activation that meets it is stored times 2^-bit).  Activations enter
// as fp16 numbers, head + remainder * 2^-11, i.e. with 22 bits.  So that no row leaves the range
// of fp16, it is first multiplied by a power of two that brings its largest element near 2^20 (2^14 and 2^12 after the
// factors 2^-6 and 2^-8 of the codes' places); the sums are multiplied back.  In phase 1 the heads of a 16-bit row are nearly
// always all of it: a tile is eight token rows, the columns of the MMA.  Rows whose heads are not (s_inexact, s_rests) are marked, and a
// tile with one takes a second pass over the weights, with the remainders.  A hidden activation of phase 2 always has both: four
// token rows at a time, columns 0-3 of the MMA carry the heads and columns 4-7 the remainders.  Hidden rows are split by phase 1
// with a fixed factor, and it keeps the maximum of each row: one that the fixed factor does not suit is split again by phase 2,
// from fp32 where the first split could not hold it.
#include "stream.cuh"
#include "unpack.cuh"

namespace mfb {

namespace {

constexpr uint32_t SW = 8, STHREADS = SW * 32;   // warps per CTA; two CTAs per SM
// Most token rows per tile: the eight columns of an MMA in phase 1, half of them beside their remainders in phase 2.
__host__ __device__ constexpr uint32_t s_tok(int phase) { return phase == 1 ? 8 : 4; }
constexpr uint32_t CHUNK = 64;                   // bytes of codes per row and ring stage: 256 codes at 2 bits, 128 at 4
struct StreamParams {
    const uint8_t *pool, *shared_blob;
    uint64_t slot_stride;
    mfb_expert_offsets routed_off, shared_off;
    uint32_t d, f, top_k, shared_bits, activation, gate32;
    float limit;
    const mfb_pair* sorted;
    const WorkTile* tiles;
    const uint32_t* n_tiles;
    const __half *xr, *xs;     // [token][d] rows in the order of the routed / the shared codes
    const float* unit;         // [token] what the sums of a row's products are multiplied with; negative: the row is marked
    __half* split;             // [sorted pair][2][f] hidden rows times HIDDEN_FACTOR as heads and remainders
    float* hidden;             // [sorted pair][f] runs of 32 hidden activations whose maximum is not s_plain; the others are not written
    uint32_t* hidden_max;      // [sorted pair] bits of the row's largest magnitude
    float* partial;            // [token, top_k + 1, d]
    uint32_t mul[2] = {4, 64}; // (see s_unpack4)
    uint32_t shared_tiles, parts;          // tiles of the shared expert, in front; units that each of them is cut into
    uint32_t ks, ntok, stages, slot, blk; // warps that share a contraction; token rows per unit; ring depth; bytes of a scale slot;
                                              // codes per scale slot and row (512, or 256 where the contraction is an odd multiple of 256)
    const __half *xr_rest, *xs_rest;      // [token][d] remainders of the marked rows
    int routed_layout;                    // of the codes of phase 1
};

// One ring stage of a warp: two tiles of [16 rows x 64 bytes] of codes (16-byte pieces swizzled so that a lane group's reads of
// eight rows fall into distinct banks).  Scales and biases come per 512 codes into two slots of their own: 16 bytes per row,
// kind and tile (tile 0 32 bytes with 32-element groups).  Fetched with every stage, 4 or 8 bytes per row, they took two
// thirds of the load unit's line look-ups and came from L2 four to eight times over.
constexpr uint32_t S_STAGE = 2048;

// A warp's share of one tile: rows row[m] .. row[m] + 15 of matrix m, blocks of `blk` codes [b0, b1).  Accumulates into acc.
// between() runs when the first stages have been requested and before the token rows are read.
template <int PHASE, int LAYOUT, int SDT, bool G32, typename Between>   // G32: matrix 0 has a scale per 32 codes
__device__ __forceinline__ void s_stream(const uint8_t* const (&codes)[2], const uint8_t* const (&scales)[2], const uint8_t* const (&biases)[2],
                                         uint32_t row_bytes, uint32_t gpr, uint32_t b0, uint32_t b1, uint32_t blk, uint32_t stages, uint32_t slot_bytes, uint8_t* ring,
                                         const __half* x_row, const float* sums, uint32_t lane, float (&acc)[2][4], const uint32_t (&mul)[2], Between between) {
    constexpr int GPC = LAYOUT == L4 ? 2 : 4;          // 64-code groups per stage
    constexpr uint32_t STOK = s_tok(PHASE);
    const uint32_t cpb = blk / (GPC * 64), cmask = cpb - 1, cshift = 31 - __clz(cpb);   // stages per block; the ring holds at most cpb + 1
    const uint32_t c0 = b0 * cpb, c1 = b1 * cpb;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t ring_a = s_smem(ring), crow = lane >> 2, cpiece = lane & 3u, srow = lane & 15u, which = lane >> 4;
    const uint8_t* csrc[2][2];
    const uint8_t* ssrc[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int h = 0; h < 2; ++h) csrc[m][h] = codes[m] + (size_t)(crow + 8 * h) * row_bytes + cpiece * 16;
        ssrc[m] = (which ? biases[m] : scales[m]) + (size_t)srow * gpr * ((G32 && m == 0) ? 4 : 2);
    }
    const uint32_t cdst = crow * 64 + ((cpiece ^ ((crow >> 1) & 3u)) << 4);
    constexpr uint32_t S0 = G32 ? 512 : 256;           // bytes of tile 0's scales (and of its biases) in a slot
    const uint32_t slots = stages * S_STAGE;
    auto issue = [&](uint32_t c, uint32_t slot) {
        if (c < c1) {
            const uint32_t st = ring_a + slot * S_STAGE;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) s_copy<16>(st + m * 1024 + h * 512 + cdst, csrc[m][h] + (size_t)c * CHUNK);
            if ((c & cmask) == 0) {
                const uint32_t b = c >> cshift, sl = ring_a + slots + (b & 1u) * slot_bytes;
                const uint32_t d0 = sl + which * S0 + srow * (G32 ? 32 : 16), d1 = sl + 2 * S0 + which * 256 + srow * 16;
                if (blk == 512) {
                    s_copy<16>(d0, ssrc[0] + (size_t)b * (G32 ? 32 : 16));
                    if (G32) s_copy<16>(d0 + 16, ssrc[0] + (size_t)b * 32 + 16);
                    s_copy<16>(d1, ssrc[1] + (size_t)b * 16);
                } else {
                    if (G32) s_copy<16>(d0, ssrc[0] + (size_t)b * 16);
                    else s_copy<8>(d0, ssrc[0] + (size_t)b * 8);
                    s_copy<8>(d1, ssrc[1] + (size_t)b * 8);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t i = 0; i + 1 < stages; ++i) issue(c0 + i, i);
    between();
    uint32_t slot = 0, fill = stages - 1;
    const uint32_t rsw = (g >> 1) & 3u;
    for (uint32_t c = c0; c < c1; ++c) {
        if (stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();                    // the stage has landed for every lane, and the one to be filled has been read by every lane
        issue(c + stages - 1, fill);
        const uint8_t* st = ring + slot * S_STAGE;
        const uint8_t* sl = ring + slots + ((c >> cshift) & 1u) * slot_bytes + (c & cmask) * (2 * GPC);
        uint32_t sc[2][2][4], bi[2][2][4];   // [matrix][row half][two scales per word]
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint8_t* p = m == 0 ? sl + (G32 ? (c & cmask) * (2 * GPC) + (g + 8 * h) * 32 : (g + 8 * h) * 16) : sl + 2 * S0 + (g + 8 * h) * 16;
                const uint32_t to_bias = m == 0 ? S0 : 256;
                constexpr int W0 = (G32 ? 2 : 1) * GPC / 2, W1 = GPC / 2;
                const int words = m == 0 ? W0 : W1;
                if (words == 4) {
                    *reinterpret_cast<uint4*>(sc[m][h]) = *reinterpret_cast<const uint4*>(p);
                    *reinterpret_cast<uint4*>(bi[m][h]) = *reinterpret_cast<const uint4*>(p + to_bias);
                } else if (words == 2) {
                    *reinterpret_cast<uint2*>(sc[m][h]) = *reinterpret_cast<const uint2*>(p);
                    *reinterpret_cast<uint2*>(bi[m][h]) = *reinterpret_cast<const uint2*>(p + to_bias);
                } else {
                    sc[m][h][0] = *reinterpret_cast<const uint32_t*>(p);
                    bi[m][h][0] = *reinterpret_cast<const uint32_t*>(p + to_bias);
                }
            }
        const uint32_t k0 = c * (GPC * 64);
        float part[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};   // the stage's share: one long chain of sums loses twice as much
#pragma unroll
        for (int j = 0; j < GPC; ++j) {
            uint32_t bf[8];
            {
                const __half* xp = x_row + k0 + j * 64 + (LAYOUT == L2 ? t * 16 : t * 8);
                *reinterpret_cast<uint4*>(bf) = *reinterpret_cast<const uint4*>(xp);
                *reinterpret_cast<uint4*>(bf + 4) = *reinterpret_cast<const uint4*>(xp + (LAYOUT == L2 ? 8 : 32));
            }
            const uint32_t grp = (k0 >> 6) + j;
            float2 lo, hi, both;         // sums of x over the group's halves (only where they are used) and over all of it
            if (G32 || LAYOUT == L2H) {
                lo = *reinterpret_cast<const float2*>(sums + grp * 2 * STOK);
                hi = *reinterpret_cast<const float2*>(sums + (grp * 2 + 1) * STOK);
                both = make_float2(lo.x + hi.x, lo.y + hi.y);
            } else {
                both = *reinterpret_cast<const float2*>(sums + grp * STOK);
                lo = hi = both;
            }
            if (PHASE == 2 && t >= 2) { lo = hi = both = make_float2(0.0f, 0.0f); }   // the remainders' columns carry no bias
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                uint32_t pl[8], ph[8];
                const uint8_t* rl = st + m * 1024 + g * 64;
                if (LAYOUT == L4) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const uint32_t o = (((2 * j + u) ^ rsw) << 4) + t * 4;
                        s_unpack4(*reinterpret_cast<const uint32_t*>(rl + o), mul, reinterpret_cast<uint32_t (&)[4]>(pl[4 * u]));
                        s_unpack4(*reinterpret_cast<const uint32_t*>(rl + 512 + o), mul, reinterpret_cast<uint32_t (&)[4]>(ph[4 * u]));
                    }
                } else if (LAYOUT == L2) {
                    const uint32_t o = ((j ^ rsw) << 4) + t * 4;
                    s_unpack2(*reinterpret_cast<const uint32_t*>(rl + o), mul, pl);
                    s_unpack2(*reinterpret_cast<const uint32_t*>(rl + 512 + o), mul, ph);
                } else {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const uint32_t o = ((j ^ rsw) << 4) + u * 8 + t * 2;
                        s_unpack2h(*reinterpret_cast<const uint16_t*>(rl + o), reinterpret_cast<uint32_t (&)[4]>(pl[4 * u]));
                        s_unpack2h(*reinterpret_cast<const uint16_t*>(rl + 512 + o), reinterpret_cast<uint32_t (&)[4]>(ph[4 * u]));
                    }
                }
                if (G32 && m == 0) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        float ds[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int q = 2 * u; q < 2 * u + 2; ++q) s_mma(ds, pl[2 * q], ph[2 * q], pl[2 * q + 1], ph[2 * q + 1], bf[2 * q], bf[2 * q + 1]);
                        const float sl = s_widen<SDT>(sc[0][0][j], u), sh = s_widen<SDT>(sc[0][1][j], u);
                        const float bl = s_widen<SDT>(bi[0][0][j], u), bh = s_widen<SDT>(bi[0][1][j], u);
                        const float2 sx = u ? hi : lo;
                        part[0][0] = fmaf(sl, ds[0], part[0][0]); part[0][0] = fmaf(bl, sx.x, part[0][0]);
                        part[0][1] = fmaf(sl, ds[1], part[0][1]); part[0][1] = fmaf(bl, sx.y, part[0][1]);
                        part[0][2] = fmaf(sh, ds[2], part[0][2]); part[0][2] = fmaf(bh, sx.x, part[0][2]);
                        part[0][3] = fmaf(sh, ds[3], part[0][3]); part[0][3] = fmaf(bh, sx.y, part[0][3]);
                    }
                } else {
                    float ds[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int q = 0; q < 4; ++q) s_mma(ds, pl[2 * q], ph[2 * q], pl[2 * q + 1], ph[2 * q + 1], bf[2 * q], bf[2 * q + 1]);
                    const float sl = s_widen<SDT>(sc[m][0][j >> 1], j & 1), sh = s_widen<SDT>(sc[m][1][j >> 1], j & 1);
                    const float bl = s_widen<SDT>(bi[m][0][j >> 1], j & 1), bh = s_widen<SDT>(bi[m][1][j >> 1], j & 1);
                    part[m][0] = fmaf(sl, ds[0], part[m][0]); part[m][0] = fmaf(bl, both.x, part[m][0]);
                    part[m][1] = fmaf(sl, ds[1], part[m][1]); part[m][1] = fmaf(bl, both.y, part[m][1]);
                    part[m][2] = fmaf(sh, ds[2], part[m][2]); part[m][2] = fmaf(bh, both.x, part[m][2]);
                    part[m][3] = fmaf(sh, ds[3], part[m][3]); part[m][3] = fmaf(bh, both.y, part[m][3]);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][i] += part[m][i];
        slot = slot + 1 == stages ? 0 : slot + 1;
        fill = fill + 1 == stages ? 0 : fill + 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Brings the tile's rows (in phase 2 heads, then remainders) into shared memory and forms their sums over the scale groups, times
// 2^-24.  src(n) = row n, in phase 2 its two rows; of_row(n) is read beside them and handed to take(n, .).
template <int PHASE, int LAYOUT, bool HALF, bool PAST_L1, typename T, typename Src, typename OfRow, typename Take>
__device__ __forceinline__ void s_stage_rows(Src src, OfRow of_row, Take take, uint32_t n, uint32_t ntok, uint32_t k, uint32_t stride, __half* rows, float* sums) {
    constexpr bool SPLIT = PHASE == 2;
    constexpr uint32_t STOK = s_tok(PHASE);
    const uint32_t runs = k / 16;
    for (uint32_t i0 = 0; i0 < n * runs; i0 += STHREADS) {   // every lane takes part in the shuffles below
        const bool live = i0 + threadIdx.x < n * runs;
        const uint32_t i = live ? i0 + threadIdx.x : n * runs - 1, r = i / runs, e0 = (i % runs) * 16;
        const __half* p = src(r) + e0;
        T mine;
        uint4 v[4];
        v[0] = PAST_L1 ? __ldcg(reinterpret_cast<const uint4*>(p)) : *reinterpret_cast<const uint4*>(p);
        v[1] = PAST_L1 ? __ldcg(reinterpret_cast<const uint4*>(p + 8)) : *reinterpret_cast<const uint4*>(p + 8);
        if (SPLIT) {
            v[2] = *reinterpret_cast<const uint4*>(p + k);
            v[3] = *reinterpret_cast<const uint4*>(p + k + 8);
        }
        const __half* head = reinterpret_cast<const __half*>(v);
        const __half* rest = reinterpret_cast<const __half*>(v + 2);
        if (live && e0 == 0) mine = of_row(r);
        float s = 0.0f;
#pragma unroll
        for (uint32_t e = 0; e < 16; ++e) {
            const uint32_t at = s_pos(e, LAYOUT);
            s = fmaf(SPLIT ? fmaf(__half2float(rest[at]), REST, __half2float(head[at])) : __half2float(head[at]), 1.0f / s_scale(e, LAYOUT), s);
        }
        __half* dst = rows + (size_t)r * stride + e0;
        *reinterpret_cast<uint4*>(dst) = v[0];
        *reinterpret_cast<uint4*>(dst + 8) = v[1];
        if (SPLIT) {
            dst = rows + (size_t)(ntok + r) * stride + e0;
            *reinterpret_cast<uint4*>(dst) = v[2];
            *reinterpret_cast<uint4*>(dst + 8) = v[3];
        }
        s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);
        if (!HALF) s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
        constexpr uint32_t PER = HALF ? 2 : 4;
        if (live && (threadIdx.x & (PER - 1)) == 0) sums[(e0 / (16 * PER)) * STOK + r] = s * CODE_UNIT;
        if (live && e0 == 0) take(r, mine);
    }
}

// Replaces the staged heads of phase 1 and their sums by the remainders of the marked rows; the other rows become zero.
template <int LAYOUT, bool HALF>
__device__ __forceinline__ void s_stage_rests(const __half* x_rest, const mfb_pair* pairs, uint32_t n, uint32_t k, uint32_t stride, __half* rows, float* sums,
                                              const float* unit) {
    const uint32_t runs = k / 16;
    for (uint32_t i0 = 0; i0 < n * runs; i0 += STHREADS) {   // every lane takes part in the shuffles below
        const bool live = i0 + threadIdx.x < n * runs;
        const uint32_t i = live ? i0 + threadIdx.x : n * runs - 1, r = i / runs, e0 = (i % runs) * 16;
        uint4 v[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
        if (unit[r] < 0.0f) {
            const uint4* p = reinterpret_cast<const uint4*>(x_rest + (size_t)pairs[r].token * k + e0);
            v[0] = __ldcg(p);
            v[1] = __ldcg(p + 1);
        }
        const __half* rest = reinterpret_cast<const __half*>(v);
        float s = 0.0f;
#pragma unroll
        for (uint32_t e = 0; e < 16; ++e) s = fmaf(__half2float(rest[s_pos(e, LAYOUT)]), 1.0f / s_scale(e, LAYOUT), s);
        uint4* dst = reinterpret_cast<uint4*>(rows + (size_t)r * stride + e0);
        dst[0] = v[0];
        dst[1] = v[1];
        s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);
        if (!HALF) s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
        constexpr uint32_t PER = HALF ? 2 : 4;
        if (live && (threadIdx.x & (PER - 1)) == 0) sums[(e0 / (16 * PER)) * s_tok(1) + r] = s * CODE_UNIT;
    }
    __syncthreads();
}

// Splits the staged hidden rows whose maximum is not s_plain once more, with a factor of their own.  Rare, hence out of
// line and looked for only by the threads that read a row's maximum beside its first elements.
template <int LAYOUT>
__device__ __noinline__ void s_split_again(const float* hidden, const uint32_t* max_bits, uint32_t n, uint32_t ntok, uint32_t k, uint32_t stride, __half* rows,
                                           float* sums, float* unit) {
    const uint32_t runs = k / 16;
    for (uint32_t i0 = 0; i0 < n * runs; i0 += STHREADS) {
        const bool live = i0 + threadIdx.x < n * runs;
        const uint32_t i = live ? i0 + threadIdx.x : n * runs - 1, r = i / runs, e0 = (i % runs) * 16, most = __ldcg(max_bits + r);
        const bool again = !s_plain(most) && most != 0u;
        float inverse, s = 0.0f;
        const float f = s_factor(most, inverse);
        __half* const head = rows + (size_t)r * stride + e0;
        __half* const rest = rows + (size_t)(ntok + r) * stride + e0;
        bool stored = (most >> 23) < 114u;   // a small row is stored as fp32 throughout, a large one where the first split overflowed
        for (uint32_t e = 0; e < 16; ++e) stored = stored || !(fabsf(__half2float(head[e])) <= 65504.0f);
        if (live && again) {
#pragma unroll 1
            for (uint32_t e = 0; e < 16; ++e) {
                const uint32_t at = s_pos(e, LAYOUT);
                const float v = stored ? __ldcg(hidden + (size_t)r * k + e0 + e)
                                       : fmaf(__half2float(rest[at]), REST, __half2float(head[at])) * (1.0f / (HIDDEN_FACTOR * s_scale(e, LAYOUT)));
                head_and_rest(v * f * s_scale(e, LAYOUT), head[at], rest[at]);
                s += v * f;
            }
            if (e0 == 0) unit[r] = inverse;
        }
        s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);
        s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
        if (live && again && (threadIdx.x & 3u) == 0) sums[(e0 / 64) * s_tok(2) + r] = s * CODE_UNIT;
    }
    __syncthreads();
}

// What kernels further ahead than the direct predecessor wrote is complete before pdl_wait() (common.cuh); it is read past L1,
// which may still hold what the same addresses held for the previous layer.
template <bool EARLY>
__device__ __forceinline__ bool s_tile(const StreamParams& P, WorkTile& T) {
    const uint32_t y = blockIdx.y, cut = P.shared_tiles * P.parts;
    const uint32_t at = y < cut ? y / P.parts : y - cut + P.shared_tiles, first = y < cut ? y % P.parts * P.ntok : 0u;
    // the tile is requested beside the number of tiles (the list is as long as the grid): one trip to L2 instead of two
    const uint4 v = EARLY ? __ldcg(reinterpret_cast<const uint4*>(P.tiles + at)) : *reinterpret_cast<const uint4*>(P.tiles + at);
    if (at >= (EARLY ? __ldcg(P.n_tiles) : *P.n_tiles)) return false;
    T.pair_start = v.x; T.n = v.y; T.slot = (int32_t)v.z; T.shared = v.w;
    if (first >= T.n) return false;
    T.pair_start += first;
    T.n = min(T.n - first, P.ntok);
    return true;
}

// One tile x one block of matrix rows.  EARLY: phase 2 requests its first weights before it waits for phase 1 (tile list and
// weights are older); phase 1, of a single row only, brings that row into shared memory before it waits for the routing,
// and T is not known yet.  One row, four layer calls of 256 experts, hidden 2048: 116.3 -> 109.5 us; eight layers
// carried: 232 -> 218.5; two layers of the 2-bit family, hidden 4096: 106.3 -> 101.4.
// RESTS: phase 1 of a tile with marked rows, with two passes over the weights.  Out of line, and looked for when the first pass is done,
// which is then thrown away.  What calls without such rows pay for it (layers of 8 and 64 rows, hidden 2048; 64 rows of the 2-bit
// family): 60.3 -> 61.3 us, 149.9 -> 151.8, 556 -> 559; with the choice in front of the first pass 0.3 % more, with the
// second pass in line 2 % in all, with a launch of its own 2.5 us a layer.
template <int SDT>
__device__ __noinline__ void s_unit_rests(const StreamParams& P);
template <int PHASE, int LAYOUT, int SDT, bool G32, bool EARLY, bool RESTS = false>
__device__ __forceinline__ void s_unit(const StreamParams& P, WorkTile T, bool shared, uint32_t rb, const mfb_expert_offsets& off, int out_layout,
                                       uint8_t* smem) {
    constexpr bool HALF = G32 || LAYOUT == L2H;
    constexpr uint32_t BITS = LAYOUT == L4 ? 4 : 2, STOK = s_tok(PHASE);
    const uint32_t k = PHASE == 1 ? P.d : P.f, gpr = k / 64, row_bytes = k * BITS / 8, stride = k + 8;
    __half* const rows = reinterpret_cast<__half*>(smem);
    float* const sums = reinterpret_cast<float*>(rows + PHASE * P.ntok * stride);
    float* const unit = sums + (k / 32) * STOK;   // [STOK] what the rows' sums are multiplied with
    uint8_t* const rings = smem + (reinterpret_cast<uint8_t*>(unit + STOK) - smem + 127) / 128 * 128;   // 16 bytes off, bank conflicts made eight layers of 64 rows 1369 us (1240)
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ks = warp % P.ks, rt = warp / P.ks;
    const __half* const x = shared ? P.xs : P.xr;
    const auto stage = [&]() {
        if constexpr (PHASE == 1) {
            const auto token = [&](uint32_t r) { return EARLY ? 0u : P.sorted[T.pair_start + r].token; };
            s_stage_rows<PHASE, LAYOUT, HALF, EARLY, float>([&](uint32_t r) { return x + (size_t)token(r) * P.d; },
                                                     [&](uint32_t r) { return EARLY ? __ldcg(P.unit) : P.unit[token(r)]; },
                                                     [&](uint32_t r, float u) { unit[r] = u; }, T.n, P.ntok, k, stride, rows, sums);
            __syncthreads();
        } else {
            bool again = false;
            s_stage_rows<PHASE, LAYOUT, HALF, false, uint32_t>([&](uint32_t r) { return (const __half*)P.split + (size_t)(T.pair_start + r) * 2 * P.f; },
                                                        [&](uint32_t r) { return __ldcg(P.hidden_max + T.pair_start + r); },
                                                        [&](uint32_t r, uint32_t most) {
                                                            unit[r] = 1.0f / HIDDEN_FACTOR;
                                                            again = again || (!s_plain(most) && most != 0u);
                                                        }, T.n, P.ntok, k, stride, rows, sums);
            if (__syncthreads_or(again))
                s_split_again<LAYOUT>(P.hidden + (size_t)T.pair_start * P.f, P.hidden_max + T.pair_start, T.n, P.ntok, k, stride, rows, sums, unit);
        }
    };
    if (PHASE == 1 || !EARLY) stage();
    if (PHASE == 1 && EARLY) {
        pdl_wait();
        pdl_release();
        if (!s_tile<EARLY>(P, T) || T.slot < 0) return;
    }
    const uint8_t* const blob = shared ? P.shared_blob : P.pool + (uint64_t)T.slot * P.slot_stride;
    const uint32_t tiles = SW / P.ks, row0 = (rb * tiles + rt) * (PHASE == 1 ? 16u : 32u);
    const uint8_t *codes[2], *scales[2], *biases[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const uint32_t r = PHASE == 1 ? row0 : row0 + 16 * m, sb = (G32 && m == 0 ? 4u : 2u);
        const uint32_t w_off = PHASE == 2 ? off.down_w : m ? off.up_w : off.gate_w, s_off = PHASE == 2 ? off.down_s : m ? off.up_s : off.gate_s,
                       b_off = PHASE == 2 ? off.down_b : m ? off.up_b : off.gate_b;
        codes[m] = blob + w_off + (size_t)r * row_bytes;
        scales[m] = blob + s_off + (size_t)r * gpr * sb;
        biases[m] = blob + b_off + (size_t)r * gpr * sb;
    }
    const uint32_t n_blocks = k / P.blk, b0 = n_blocks * ks / P.ks, b1 = n_blocks * (ks + 1) / P.ks;
    const uint32_t g = lane >> 2, t = lane & 3u, col = g & (STOK - 1);   // columns without a token row repeat row 0: nothing reads them
    const __half* x_row = rows + (size_t)((g >= STOK ? P.ntok : 0u) + (col < T.n ? col : 0u)) * stride;
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    s_stream<PHASE, LAYOUT, SDT, G32>(codes, scales, biases, row_bytes, gpr, b0, b1, P.blk, P.stages, P.slot, rings + warp * (P.stages * S_STAGE + 2 * P.slot), x_row,
                               sums + (2 * t & (STOK - 1)), lane, acc, P.mul, [&]() {
        if (PHASE == 2 && EARLY) {
            pdl_wait();
            pdl_release();
            stage();
        }
    });
    if constexpr (PHASE == 1 && !RESTS)
        if (__any_sync(0xFFFFFFFFu, lane < T.n && unit[lane] < 0.0f)) {
            __syncthreads();
            return s_unit_rests<SDT>(P);
        }
    if constexpr (RESTS) {   // the sums in units of the remainders, whose products come on top, and back
        const auto times = [&](float v) {
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i >> 2][i & 3] *= v;
        };
        times(1.0f / REST);
        __syncthreads();
        s_stage_rests<LAYOUT, HALF>(shared ? P.xs_rest : P.xr_rest, P.sorted + T.pair_start, T.n, k, stride, rows, sums, unit);
        s_stream<PHASE, LAYOUT, SDT, G32>(codes, scales, biases, row_bytes, gpr, b0, b1, P.blk, P.stages, P.slot, rings + warp * (P.stages * S_STAGE + 2 * P.slot),
                                   x_row, sums + (2 * t & (STOK - 1)), lane, acc, P.mul, []() {});
        times(REST);
    }
    // sums of the warps that share a contraction, in their order, and the epilogue
    __syncthreads();
    float* const red = reinterpret_cast<float*>(rings);   // [warp][matrix][lane][4]
#pragma unroll
    for (int m = 0; m < 2; ++m)
        *reinterpret_cast<float4*>(red + ((warp * 2 + m) * 32 + lane) * 4) = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
    __syncthreads();
    const uint32_t unit_rows = tiles * (PHASE == 1 ? 16u : 32u);
    for (uint32_t o = threadIdx.x; o < unit_rows * T.n; o += STHREADS) {
        const uint32_t rl = o % unit_rows, n = o / unit_rows;
        const uint32_t tile = PHASE == 1 ? rl >> 4 : rl >> 5, r16 = rl & 15u;
        const float* p = red + (tile * P.ks * 2 * 32 + (r16 & 7u) * 4 + (n >> 1)) * 4 + (r16 >> 3) * 2 + (n & 1u);   // in phase 2 heads; remainders 8 floats on
        float v[2] = {0.0f, 0.0f};
        for (uint32_t q = 0; q < P.ks; ++q)
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const float* e = p + (q * 2 + m) * 128;
                v[m] += PHASE == 1 ? e[0] : fmaf(e[8], REST, e[0]);
            }
        const uint32_t row = rb * unit_rows + rl;
        if (PHASE == 1) {
            const float back = RESTS ? fabsf(unit[n]) : unit[n];
            float gate = v[0] * 16777216.0f * back, up = v[1] * 16777216.0f * back;
            if (!T.shared && P.limit > 0.0f) {   // moe_swiglu_clamp, moe.metal:27-34 (routed experts only)
                gate = fminf(gate, P.limit);
                up = fminf(fmaxf(up, -P.limit), P.limit);
            }
            const float a = hidden_act(gate, (int)P.activation) * up;
            __half head, rest;
            head_and_rest(a * HIDDEN_FACTOR * s_scale(row & 15u, out_layout), head, rest);
            __half* out = P.split + (size_t)(T.pair_start + n) * 2 * P.f + (row & ~15u) + s_pos(row & 15u, out_layout);
            out[0] = head;
            out[P.f] = rest;
            // a warp's 32 elements belong to one row (unit_rows is a multiple of 32); stream_prep_kernel has cleared the maximum
            const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(a) & 0x7FFFFFFFu);
            if (!s_plain(most)) P.hidden[(size_t)(T.pair_start + n) * P.f + row] = a;
            if (lane == 0) atomicMax(P.hidden_max + T.pair_start + n, most);
        } else {
            const mfb_pair pr = P.sorted[T.pair_start + n];
            P.partial[((size_t)pr.token * (P.top_k + 1) + pr.rank) * P.d + row] = ((rl >> 4) & 1u ? v[1] : v[0]) * 16777216.0f * unit[n];
        }
    }
}

template <int SDT>
__device__ __noinline__ void s_unit_rests(const StreamParams& P) {
    extern __shared__ __align__(128) uint8_t smem[];
    WorkTile T;
    s_tile<false>(P, T);
    const int hidden = P.routed_layout == L4 ? L4 : L2;
    if (T.shared && P.shared_bits == 4) s_unit<1, L4, SDT, false, false, true>(P, T, true, blockIdx.x, P.shared_off, L4, smem);
    else if (T.shared) s_unit<1, L2, SDT, false, false, true>(P, T, true, blockIdx.x, P.shared_off, L2, smem);
    else if (P.routed_layout == L2H) s_unit<1, L2H, SDT, true, false, true>(P, T, false, blockIdx.x, P.routed_off, hidden, smem);
    else if (P.routed_layout == L4 && P.gate32) s_unit<1, L4, SDT, true, false, true>(P, T, false, blockIdx.x, P.routed_off, hidden, smem);
    else if (P.routed_layout == L4) s_unit<1, L4, SDT, false, false, true>(P, T, false, blockIdx.x, P.routed_off, hidden, smem);
    else s_unit<1, L2, SDT, false, false, true>(P, T, false, blockIdx.x, P.routed_off, hidden, smem);
}

template <int PHASE, int LAYOUT, int SDT, bool EARLY>   // LAYOUT of the routed experts in this phase; L2H only in phase 1; EARLY: see s_unit
__global__ void __launch_bounds__(STHREADS, 2) stream_kernel(const __grid_constant__ StreamParams P) {
    extern __shared__ __align__(128) uint8_t smem[];
    WorkTile T = {0, 1, 0, 0};
    bool shared = P.shared_blob && blockIdx.y == 0;   // a single row's tiles: the shared expert's in front
    if (!EARLY) {
        pdl_wait();
        pdl_release();
    }
    if (PHASE == 2 || !EARLY) {
        const bool any = s_tile<EARLY>(P, T);
        if (!any || T.slot < 0) {
            if (PHASE == 2 && EARLY) pdl_wait();   // also with nothing to do: the grid must not end before phase 1 has
            if (PHASE == 2 && any) {      // an expert that is not resident contributes nothing: its rows of the partials are cleared
                const uint32_t unit_rows = 32 * (SW / P.ks);
                for (uint32_t o = threadIdx.x; o < unit_rows * T.n; o += STHREADS) {
                    const mfb_pair pr = P.sorted[T.pair_start + o / unit_rows];
                    P.partial[((size_t)pr.token * (P.top_k + 1) + pr.rank) * P.d + blockIdx.x * unit_rows + o % unit_rows] = 0.0f;
                }
            }
            return;
        }
        shared = T.shared != 0;
    }
    constexpr int HIDDEN = LAYOUT == L4 ? L4 : L2;   // order of the routed experts' hidden activations
    if (shared) {
        if (P.shared_bits == 4) s_unit<PHASE, L4, SDT, false, EARLY>(P, T, true, blockIdx.x, P.shared_off, L4, smem);
        else s_unit<PHASE, L2, SDT, false, EARLY>(P, T, true, blockIdx.x, P.shared_off, L2, smem);
        return;
    }
    if (PHASE == 1 && LAYOUT == L2H) s_unit<PHASE, L2H, SDT, true, EARLY>(P, T, false, blockIdx.x, P.routed_off, HIDDEN, smem);
    else if (PHASE == 1 && LAYOUT == L4 && P.gate32) s_unit<PHASE, L4, SDT, true, EARLY>(P, T, false, blockIdx.x, P.routed_off, HIDDEN, smem);
    else s_unit<PHASE, LAYOUT == L2H ? L2 : LAYOUT, SDT, false, EARLY>(P, T, false, blockIdx.x, P.routed_off, HIDDEN, smem);
}

// Token rows: RMSNorm (arithmetic and order of rmsnorm_rows16_kernel, glue.cu) where asked for, then times a power of two as fp16 in
// the order(s) of the codes, with the remainders where the row is marked.  The row crosses global memory once, in 16-byte pieces; one element at a time a single row took
// 13 us.
// COMBINE: the rows are first made from the previous layer's partial rows (the residual stream of a stack), which saves
// a launch and the way through memory: eight layers, one row, 242 -> 232 us.
template <bool COMBINE>
__global__ void __launch_bounds__(COMBINE ? 512 : 256) stream_prep_kernel(const uint16_t* x, int dtype, uint32_t ldx, uint32_t d,
                                                          const __nv_bfloat16* __restrict__ w, float eps, int norm, uint16_t* __restrict__ xn,
                                                          __half* __restrict__ xr, int layout, __half* __restrict__ xs, int layout_s, float* __restrict__ unit,
                                                          __half* __restrict__ xr_rest, __half* __restrict__ xs_rest,
                                                          uint32_t* __restrict__ hidden_max, uint32_t slots, const PendingCombine pc) {
    extern __shared__ __align__(16) uint16_t row_s[];   // [d] the row, then [d] the gain
    uint16_t* const gain_s = row_s + d;
    __shared__ float red[8];
    __shared__ uint32_t red_x[8], red_n[8];
    const size_t row = blockIdx.x;
    const uint16_t* src = x + row * ldx;
    const bool gain = norm && w;
    pdl_wait();
    pdl_release();
    if (threadIdx.x < slots) hidden_max[row * slots + threadIdx.x] = 0u;
    if (COMBINE) {
        for (uint32_t i = threadIdx.x; i < d; i += blockDim.x)
            if (gain) gain_s[i] = __bfloat16_as_ushort(w[i]);
        for (uint32_t q = threadIdx.x; q < d / 4; q += blockDim.x)
            reinterpret_cast<uint2*>(row_s)[q] = combine_quad(pc.partial, pc.route_w, pc.top_k, pc.slots, d, pc.slot_mask, pc.with_shared, pc.y, pc.y, dtype,
                                                              pc.shared_gate, (uint32_t)row, q * 4);
    } else if ((ldx & 7u) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0) {
        for (uint32_t p = threadIdx.x; p < d / 8; p += blockDim.x) {
            reinterpret_cast<uint4*>(row_s)[p] = reinterpret_cast<const uint4*>(src)[p];
            if (gain) reinterpret_cast<uint4*>(gain_s)[p] = reinterpret_cast<const uint4*>(w)[p];
        }
    } else {
        for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) {
            row_s[i] = src[i];
            if (gain) gain_s[i] = __bfloat16_as_ushort(w[i]);
        }
    }
    __syncthreads();
    float inv = 1.0f, largest, smallest;
    {
        float ss = 0.0f;
        uint32_t mx = 0, mn = 0xFFFFFFFFu;   // mn: bits of the smallest element that is not zero, less one
        if (threadIdx.x < 256) {   // the sum's order is that of 256 threads
            for (uint32_t i = threadIdx.x; i < d; i += 256) {
                const float v = widen16(row_s[i], dtype);
                ss = fmaf(v, v, ss);
                const uint32_t bits = __float_as_uint(gain ? v * __uint_as_float((uint32_t)gain_s[i] << 16) : v) & 0x7FFFFFFFu;
                mx = max(mx, bits);
                mn = min(mn, bits - 1u);
            }
            for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, off);
            mx = __reduce_max_sync(0xFFFFFFFFu, mx);
            mn = __reduce_min_sync(0xFFFFFFFFu, mn);
            if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = ss; red_x[threadIdx.x >> 5] = mx; red_n[threadIdx.x >> 5] = mn; }
        }
        __syncthreads();
        float v = red[threadIdx.x & 7u];
        for (int off = 4; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
        if (norm) inv = rsqrtf(v / (float)d + eps);
        // the largest element of the row as it goes into the products, but for its rounding
        largest = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, red_x[threadIdx.x & 7u])) * inv;
        smallest = __uint_as_float(__reduce_min_sync(0xFFFFFFFFu, red_n[threadIdx.x & 7u]) + 1u) * inv;
    }
    float back;
    const float factor = s_factor(__float_as_uint(largest) & 0x7FFFFFFFu, back);
    if (threadIdx.x == 0) unit[row] = back;
    for (uint32_t p = threadIdx.x; p < d / 16; p += blockDim.x) {   // runs of sixteen elements
        uint16_t in[16];
        *reinterpret_cast<uint4*>(in) = reinterpret_cast<const uint4*>(row_s)[2 * p];
        *reinterpret_cast<uint4*>(in + 8) = reinterpret_cast<const uint4*>(row_s)[2 * p + 1];
        if (norm) {
            uint16_t gn[16];
            if (gain) {
                *reinterpret_cast<uint4*>(gn) = reinterpret_cast<const uint4*>(gain_s)[2 * p];
                *reinterpret_cast<uint4*>(gn + 8) = reinterpret_cast<const uint4*>(gain_s)[2 * p + 1];
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
                in[j] = narrow16(widen16(in[j], dtype) * inv * (gain ? __uint_as_float((uint32_t)gn[j] << 16) : 1.0f), dtype);
            uint4* dst = reinterpret_cast<uint4*>(xn + row * d) + 2 * p;
            dst[0] = *reinterpret_cast<const uint4*>(in);
            dst[1] = *reinterpret_cast<const uint4*>(in + 8);
        }
        auto put = [&](__half* out, auto layout_c) {
            constexpr int L = decltype(layout_c)::value;
            __align__(16) __half head[16];
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) head[s_pos(j, L)] = __float2half_rn(widen16(in[j], dtype) * factor * s_scale(j, L));
            uint4* dst = reinterpret_cast<uint4*>(out + row * d) + 2 * p;
            dst[0] = *reinterpret_cast<const uint4*>(head);
            dst[1] = *reinterpret_cast<const uint4*>(head + 8);
        };
        auto put_any = [&](__half* out, int l) {
            if (l == L4) put(out, std::integral_constant<int, L4>());
            else if (l == L2) put(out, std::integral_constant<int, L2>());
            else put(out, std::integral_constant<int, L2H>());
        };
        put_any(xr, layout);
        if (xs) put_any(xs, layout_s);
    }
    if (s_inexact(smallest, largest, factor, dtype, layout == L4 && (!xs || layout_s == L4)))
        s_rests([&](uint32_t i) {
            const float v = widen16(row_s[i], dtype);
            return norm ? widen16(narrow16(v * inv * (gain ? __uint_as_float((uint32_t)gain_s[i] << 16) : 1.0f), dtype), dtype) : v;
        }, d, factor, back, layout, xr_rest + row * d, layout_s, xs ? xs_rest + row * d : nullptr, unit + row);
}

// Cuts every group into tiles of up to `routed_tile` (`shared_tile`) rows.  The shared expert's tiles come first: at four bits they take twice as
// long as the others, and the last units to start should be short.
__global__ void __launch_bounds__(256) stream_tiles_kernel(const mfb_group* __restrict__ groups, const uint32_t* __restrict__ n_groups,
                                                           uint32_t num_experts, const int16_t* __restrict__ slot_of, int has_shared,
                                                           uint32_t routed_tile, uint32_t shared_tile, WorkTile* __restrict__ tiles, uint32_t* __restrict__ n_tiles) {
    __shared__ uint32_t first_s[MFB_MAX_EXPERTS + 2];
    pdl_wait();
    pdl_release();
    const uint32_t ng = *n_groups;
    if (threadIdx.x < 32) {
        const uint32_t lane = threadIdx.x;
        uint32_t run = 0;
        for (uint32_t base = 0; base < ng; base += 32) {
            const uint32_t g = base + lane, tile = g < ng && groups[g].expert >= num_experts ? shared_tile : routed_tile;
            const uint32_t c = g < ng ? (groups[g].pair_count + tile - 1) / tile : 0u;
            uint32_t incl = c;
            for (uint32_t off = 1; off < 32; off <<= 1) {
                const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, incl, off);
                if (lane >= off) incl += a;
            }
            if (g < ng) first_s[g] = run + incl - c;
            run += __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
        if (lane == 0) { first_s[ng] = run; *n_tiles = run; }
    }
    __syncthreads();
    if (ng == 0) return;
    const uint32_t total = first_s[ng];
    const bool last_shared = groups[ng - 1].expert >= num_experts;
    const uint32_t in_front = last_shared ? total - first_s[ng - 1] : 0u;
    for (uint32_t g = threadIdx.x; g < ng; g += blockDim.x) {
        const mfb_group grp = groups[g];
        const bool shared = grp.expert >= num_experts;
        const uint32_t tile = shared ? shared_tile : routed_tile;
        WorkTile t;
        t.shared = shared ? 1u : 0u;
        t.slot = shared ? (has_shared ? 0 : -1) : slot_of ? (int32_t)slot_of[grp.expert] : (int32_t)grp.expert;
        const uint32_t at = shared ? 0u : first_s[g] + in_front;
        for (uint32_t i = 0; i * tile < grp.pair_count; ++i) {
            t.pair_start = grp.pair_start + i * tile;
            t.n = min(tile, grp.pair_count - i * tile);
            tiles[at + i] = t;
        }
    }
}

int routed_layout(const mfb_moe_config& c, const mfb_layer_weights& w) { return c.bits == 4 ? L4 : w.gate_group_size == 32 ? L2H : L2; }

constexpr uint32_t S_SMEM_LIMIT = 114 * 1024;   // two CTAs per SM

using StreamFn = void (*)(const StreamParams);
template <int PHASE, int SDT, bool EARLY>
StreamFn stream_fn(int layout) {
    if (layout == L4) return stream_kernel<PHASE, L4, SDT, EARLY>;
    if (PHASE == 1 && layout == L2H) return stream_kernel<1, L2H, SDT, EARLY>;
    return stream_kernel<PHASE, L2, SDT, EARLY>;
}
template <int PHASE, int SDT>
StreamFn stream_fn(int layout, bool early) { return early ? stream_fn<PHASE, SDT, true>(layout) : stream_fn<PHASE, SDT, false>(layout); }
StreamFn stream_fn(int phase, int layout, uint32_t sdt, bool early) {
    if (sdt == MFB_DT_BF16) return phase == 1 ? stream_fn<1, MFB_DT_BF16>(layout, early) : stream_fn<2, MFB_DT_BF16>(layout, early);
    return phase == 1 ? stream_fn<1, MFB_DT_F16>(layout, early) : stream_fn<2, MFB_DT_F16>(layout, early);
}

uint32_t stream_fixed_smem(uint32_t phase, uint32_t k, uint32_t ntok) { return (phase * ntok * (k + 8) * 2 + (k / 32 + 1) * s_tok((int)phase) * 4 + 127) / 128 * 128; }

}  // namespace

// Token rows per unit: as many as leave room for two CTAs on an SM, up to 2048 elements with a ring of three stages.  A routed expert's
// tile is a unit of either phase (an expert seldom has more than four rows); the shared expert has all rows, and its tiles are units of
// phase 1, one or several of phase 2.
static uint32_t most_rows(uint32_t phase, uint32_t k) { return k <= 2048 ? s_tok((int)phase) : phase == 1 && k <= 6400 ? 4 : 2; }

static uint32_t ring_bytes(uint32_t stages, uint32_t slot) { return SW * (stages * S_STAGE + 2 * slot); }

bool stream_supported(const mfb_moe_config& c) {
    return c.shared_bits != 8 && c.d % 256 == 0 && c.f % 256 == 0 && c.d <= STREAM_LONGEST && c.f <= STREAM_LONGEST;
}

// Only the forms that the handle can reach: the attribute loads the kernel.
static cudaError_t stream_init(const mfb_moe_config& c) {
    for (int phase = 1; phase <= 2; ++phase)
        for (int layout = c.bits == 4 ? L4 : L2; layout <= (c.bits == 4 ? L4 : L2H); ++layout)
            for (bool early : {false, true}) {
                const cudaError_t e = cudaFuncSetAttribute(stream_fn(phase, layout, c.scale_dtype, early), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S_SMEM_LIMIT);
                if (e != cudaSuccess) return e;
            }
    return cudaSuccess;
}

// One allocation for all of it: each of its own costs the creation of a handle up to a millisecond.
cudaError_t stream_alloc(const mfb_moe_config& c, StreamArena* a) {
    const size_t t = c.max_tokens < STREAM_MAX_TOKENS ? c.max_tokens : STREAM_MAX_TOKENS, rows = t * (c.top_k + 1);
    for (const bool measure : {true, false}) {
        size_t at = 0;
        const auto place = [&](auto*& p, size_t count) {
            if (!measure) p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(a->base + at);
            at += (count * sizeof(*p) + 255) / 256 * 256;
        };
        place(a->xr, 2 * t * c.d);
        place(a->tr, t * (c.d / 32));
        if (c.shared_bits) {
            place(a->xs, 2 * t * c.d);
            place(a->ts, t * (c.d / 64));
        }
        if (!measure) {
            a->xr_rest = a->xr + t * c.d;
            if (c.shared_bits) a->xs_rest = a->xs + t * c.d;
        }
        place(a->split, rows * 2 * c.f);
        place(a->th, rows * (c.f / 32));
        place(a->unit, t);
        place(a->hidden_max, rows);
        place(a->tiles, rows);
        place(a->n_tiles, 1);
        place(a->arrivals, 1);
        if (!measure) break;
        const cudaError_t e = cudaMalloc(&a->base, at);
        if (e != cudaSuccess) return e;
    }
    const cudaError_t e = cudaMemset(a->arrivals, 0, sizeof *a->arrivals);
    if (e != cudaSuccess) return e;
    return stream_init(c);
}

void stream_free(StreamArena* a) {
    cudaFree(a->base);
    *a = StreamArena();
}

cudaError_t stream_prep(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const StreamArena& a, const void* x, uint32_t ldx,
                        uint32_t n_tokens, const __nv_bfloat16* norm_w, float norm_eps, void* xn, const PendingCombine* pending) {
    const int layout = routed_layout(c, w), layout_s = c.shared_bits == 2 ? L2 : L4;
    const bool second = c.shared_bits && layout_s != layout;
    count_launches(1);
    const auto launch = [&](auto kernel, uint32_t threads) {
        return launch_dependent(kernel, dim3(n_tokens), dim3(threads), c.d * 4, s, (const uint16_t*)x, (int)c.x_dtype, ldx, c.d, norm_w, norm_eps,
                                norm_eps >= 0.0f ? 1 : 0, (uint16_t*)xn, a.xr, layout, second ? a.xs : nullptr, layout_s, a.unit, a.xr_rest, a.xs_rest, a.hidden_max,
                                c.top_k + 1, pending ? *pending : PendingCombine());
    };
    return pending ? launch(stream_prep_kernel<true>, 512) : launch(stream_prep_kernel<false>, 256);
}

uint32_t stream_tile_rows(const mfb_moe_config& c, uint32_t n_tokens) {
    const uint32_t one = most_rows(1, c.d), two = most_rows(2, c.f), most = one < two ? one : two;
    return n_tokens < most ? n_tokens : most;
}
uint32_t stream_shared_rows(const mfb_moe_config& c, uint32_t n_tokens) { return n_tokens < most_rows(1, c.d) ? n_tokens : most_rows(1, c.d); }

cudaError_t stream_tiles(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const StreamArena& a, bool shared, uint32_t tile_rows,
                         uint32_t shared_rows, const mfb_group* groups, const uint32_t* n_groups) {
    count_launches(1);
    return launch_dependent(stream_tiles_kernel, dim3(1), dim3(256), 0, s, groups, n_groups, c.num_experts, w.slot_of, shared ? 1 : 0,
                            tile_rows, shared_rows, a.tiles, a.n_tiles);
}

cudaError_t stream_ffn(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const StreamArena& a, uint32_t n_tokens, bool shared,
                       const mfb_pair* sorted, float* acts, float* partial, int sm_count,
                       const std::function<cudaError_t()>& between) {
    const int layout = routed_layout(c, w), layout_s = c.shared_bits == 2 ? L2 : L4;
    const uint32_t tile = stream_tile_rows(c, n_tokens), tile_s = stream_shared_rows(c, n_tokens);
    StreamParams P;
    P.pool = w.pool; P.shared_blob = shared ? w.shared_blob : nullptr; P.slot_stride = w.slot_stride;
    P.routed_off = w.routed_off; P.shared_off = w.shared_off;
    P.d = c.d; P.f = c.f; P.top_k = c.top_k; P.shared_bits = c.shared_bits; P.activation = c.activation;
    P.gate32 = w.gate_group_size == 32 ? 1u : 0u; P.limit = c.swiglu_limit;
    P.sorted = sorted; P.tiles = a.tiles; P.n_tiles = a.n_tiles;
    const bool second = c.shared_bits && layout_s != layout;
    P.xr = a.xr; P.xs = second ? a.xs : a.xr; P.xr_rest = a.xr_rest; P.xs_rest = second ? a.xs_rest : a.xr_rest; P.routed_layout = layout;
    P.unit = a.unit; P.split = a.split; P.hidden = acts; P.hidden_max = a.hidden_max; P.partial = partial;
    // most tiles there can be: a routed pair each, until every expert has one and the rest fill up tiles
    const uint32_t pairs = n_tokens * c.top_k;
    uint32_t tiles = pairs < c.num_experts + pairs / tile ? pairs : c.num_experts + pairs / tile;
    P.shared_tiles = shared ? (n_tokens + tile_s - 1) / tile_s : 0u;
    tiles += P.shared_tiles;
    for (int phase = 1; phase <= 2; ++phase) {
        const uint32_t k = phase == 1 ? c.d : c.f, rows = phase == 1 ? c.f : c.d, per_warp = phase == 1 ? 16u : 32u, most = most_rows((uint32_t)phase, k);
        P.ntok = tile_s < most ? tile_s : most;
        P.parts = (tile_s + P.ntok - 1) / P.ntok;
        const uint32_t units = tiles + P.shared_tiles * (P.parts - 1);
        // warps share a contraction until every SM has a CTA: with few tiles, whole contractions per warp would leave SMs without
        // work (two CTAs per SM as the aim: 3 % slower at 8 rows, four: 20 %)
        P.ks = 1;
        while (P.ks < 4 && units * (rows / (per_warp * (SW / P.ks))) < (uint32_t)sm_count) P.ks *= 2;
        const uint32_t fixed = stream_fixed_smem((uint32_t)phase, k, P.ntok);
        P.slot = phase == 1 && P.gate32 ? 1536u : 1024u;
        P.blk = k % 512 == 0 ? 512u : 256u;
        const uint32_t stage_codes = layout == L4 && (!shared || layout_s == L4) ? 128u : 256u;
        const uint32_t deepest = P.blk / stage_codes + 1 < 3u ? P.blk / stage_codes + 1 : 3u;   // (see s_stream)  deeper rings are slower: up to five stages 525 us against 476 for eight layers of 8 rows, 1404 against 1214 for 64
        P.stages = 2;
        while (P.stages < deepest && fixed + ring_bytes(P.stages + 1, P.slot) <= S_SMEM_LIMIT) ++P.stages;
        const dim3 grid(rows / (per_warp * (SW / P.ks)), units);
        // (see s_unit) phase 1: a single row's place is known before the routing; phase 2: only where all CTAs are resident at
        // once - with more, the first ones' requests compete with what is left of phase 1 (64 rows: +1 %)
        const bool early = phase == 1 ? n_tokens == 1 : grid.x * grid.y <= 2u * (uint32_t)sm_count;
        const cudaError_t e = launch_dependent(stream_fn(phase, layout, c.scale_dtype, early), grid, dim3(STHREADS), fixed + ring_bytes(P.stages, P.slot), s, P);
        if (e != cudaSuccess) return e;
        if (phase == 1 && between) {
            const cudaError_t b = between();
            if (b != cudaSuccess) return b;
        }
    }
    count_launches(2);
    return cudaSuccess;
}

}  // namespace mfb
