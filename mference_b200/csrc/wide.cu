// Expert FFN of a block of rows (a prompt chunk) in fp32 accuracy: the arithmetic of the streaming decode kernels (stream.cu), bit for
// bit where no contraction is shared there, with up to sixteen token rows of an expert per unpacking of its codes.
//
// What bounds it is instruction issue and latency: 86 instructions per 16 matrix rows x 64 codes in phase 1, half of them to unpack
// codes with 32-element gate groups, 104 in phase 2 (up to sixteen token rows as heads and remainders), with the MMA pipe (mma.sync) a third and
// a half busy.
// A CTA of four warps takes a tile of sixteen rows and 64 matrix rows in phase 1 (sixteen MMA columns: the heads of a 16-bit row are nearly
// always all of it; a tile with a marked row takes a second pass, see stream.cu), 128 in phase 2 (32 columns: heads and remainders), so that down is
// unpacked once for all of them and a token row's fragments are read once for 32 matrix rows.  Sums of different columns are
// interleaved: a tile of up to eight rows has a loop of its own instead of a bound inside.  Weights come as in stream.cu, each warp's own; the
// rows' pieces are staged by the whole CTA, one barrier per 256 (128) codes.  Few warps with many registers each: phase 2 needs 168.
// 640 rows of hidden 4096, 2-bit, 32-element gate groups: 2199 us with eight warps, eight rows of down per unpacking and
// one fma at a time; with 32 columns 2090; interleaved 1926; four warps and two blocks of rows each 1771; phase 1 with four CTAs per SM 1744.
#include "stream.cuh"
#include "unpack.cuh"
#include "wide.cuh"

namespace mfb {

namespace {

constexpr uint32_t WW = 4, WTHREADS = WW * 32;
constexpr uint32_t WTOK = 16;            // token rows per tile
constexpr uint32_t W_STAGE = 1024;       // bytes of codes per warp, matrix and stage: 16 rows x 64 bytes
constexpr uint32_t W_SMEM_LIMIT = 75 * 1024, W_SMEM_FOUR = 55 * 1024;   // three and four CTAs per SM

struct WideParams {
    const uint8_t *pool, *shared_blob;
    uint64_t slot_stride;
    mfb_expert_offsets routed_off, shared_off;
    uint32_t d, f, top_k, shared_bits, activation, gate32;
    float limit;
    const mfb_pair* sorted;
    const WorkTile* tiles;
    const uint32_t* n_tiles;
    const __half *xr, *xs;           // [token][d] rows in the order of the routed / the shared codes
    const float *x_sums, *x_unit;    // [token][d / 32] sums of 32 elements, [token] factor; negative: the row is marked
    float* hidden;                   // [pair][f], and the same memory as [pair][2][f] fp16 heads and remainders
    const float *h_sums, *h_unit;    // [pair][f / 32], [pair]
    float* partial;
    uint32_t mul[2] = {4, 64};       // (unpack.cuh)
    uint32_t stages, slot, blk, blocks;   // ring depth; bytes of a scale slot; codes per scale slot and row; row blocks of a tile
    const __half *xr_rest, *xs_rest;      // [token][d] remainders of the marked rows
    int routed_layout;                    // of the codes of phase 1
};

// One tile x one block of matrix rows.  RESTS: phase 1 of a tile with marked rows (see s_unit, stream.cu).
template <int SDT>
__device__ __noinline__ void w_unit_rests(const WideParams& P);
template <int PHASE, int LAYOUT, int SDT, bool G32, int NS, bool RESTS = false>
__device__ __forceinline__ void w_unit(const WideParams& P, const WorkTile& T, uint32_t rb, const mfb_expert_offsets& off, uint8_t* smem) {
    constexpr int GPC = LAYOUT == L4 ? 2 : 4;                 // 64-code groups per stage
    constexpr int M = 2;                      // phase 1: gate and up of the same rows; phase 2: two blocks of sixteen rows
    constexpr uint32_t BITS = LAYOUT == L4 ? 4 : 2, SC = GPC * 64, COLS = NS * 8, TOKENS = WTOK;
    // bytes of a staged column: the fragment loads of two neighbouring columns must not share banks
    constexpr uint32_t B_STRIDE = SC * 2 + (LAYOUT == L2 ? 16 : 64), B_STAGE = COLS * B_STRIDE;
    constexpr uint32_t S0 = G32 ? 512 : 256;                  // bytes of matrix 0's scales (and of its biases) in a slot
    constexpr uint32_t WSTAGE = M * W_STAGE;
    const uint32_t k = PHASE == 1 ? P.d : P.f, gpr = k / 64, row_bytes = k * BITS / 8, n_stages = k / SC;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3u;
    const uint32_t n = T.n;
    const uint32_t warp_bytes = P.stages * WSTAGE + 2 * P.slot;
    const uint32_t ring = s_smem(smem) + warp * warp_bytes;
    uint8_t* const ring_b = smem + WW * warp_bytes;
    float* const sums = reinterpret_cast<float*>(ring_b + P.stages * B_STAGE);   // [k / 32][TOKENS]
    float* const unit = sums + (k / 32) * TOKENS;
    // what the lanes copy
    const uint8_t* const blob = T.shared ? P.shared_blob : P.pool + (uint64_t)T.slot * P.slot_stride;
    const uint32_t row0 = (rb * WW + warp) * (PHASE == 1 ? 16u : 32u);
    const uint32_t crow = lane >> 2, cpiece = lane & 3u, srow = lane & 15u, which = lane >> 4;
    const uint8_t* csrc[M];
    const uint8_t* ssrc[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const uint32_t sb = (G32 && m == 0 ? 4u : 2u);
        const uint32_t w_off = PHASE == 2 ? off.down_w : m ? off.up_w : off.gate_w, s_off = PHASE == 2 ? off.down_s : m ? off.up_s : off.gate_s,
                       b_off = PHASE == 2 ? off.down_b : m ? off.up_b : off.gate_b;
        const uint32_t r = PHASE == 1 ? row0 : row0 + 16 * m;
        csrc[m] = blob + w_off + (size_t)(r + crow) * row_bytes + cpiece * 16;
        ssrc[m] = blob + (which ? b_off : s_off) + (size_t)(r + srow) * gpr * sb;
    }
    const uint32_t cdst = ring + crow * 64 + ((cpiece ^ ((crow >> 1) & 3u)) << 4), slots = ring + P.stages * WSTAGE;
    const uint32_t sdst[2] = {slots + which * S0 + srow * (G32 ? 32 : 16), slots + 2 * S0 + which * 256 + srow * 16};
    constexpr uint32_t PPR = SC / 8, PIECES = (COLS * PPR + WTHREADS - 1) / WTHREADS;   // 16-byte pieces per column; per thread
    const __half* bbase = PHASE == 2 ? reinterpret_cast<const __half*>(P.hidden) : T.shared ? P.xs : P.xr;
    uint32_t bsrc[PIECES];           // in pieces
    bool blive[PIECES];
#pragma unroll
    for (uint32_t i = 0; i < PIECES; ++i) {
        const uint32_t p = threadIdx.x + i * WTHREADS, r = p / PPR, q = p % PPR;
        const uint32_t tok = PHASE == 1 ? r : (r >> 3) * 4 + (r & 3u);
        blive[i] = tok < n && r < COLS;
        const uint32_t pair = T.pair_start + (blive[i] ? tok : 0u);
        bsrc[i] = (PHASE == 1 ? P.sorted[pair].token : pair * 2 + ((r >> 2) & 1u)) * (k / 8) + q;
    }
    // a thread's pieces are whole columns apart: one address, constant distances
    const uint32_t bdst = s_smem(ring_b) + threadIdx.x / PPR * B_STRIDE + threadIdx.x % PPR * 16;
    constexpr uint32_t B_APART = WTHREADS / PPR * B_STRIDE;
    const uint32_t cpb = P.blk / SC, cmask = cpb - 1, cshift = 31 - __clz(cpb);
    auto issue = [&](uint32_t c, uint32_t st) {
        if (c < n_stages) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                s_copy<16>(cdst + st * WSTAGE + m * 1024, csrc[m]);
                s_copy<16>(cdst + st * WSTAGE + m * 1024 + 512, csrc[m] + 8 * row_bytes);
                csrc[m] += 64;
            }
            if ((c & cmask) == 0) {
                const uint32_t sl = ((c >> cshift) & 1u) * P.slot;
                if (P.blk == 512) {
                    s_copy<16>(sdst[0] + sl, ssrc[0]);
                    if (G32) s_copy<16>(sdst[0] + sl + 16, ssrc[0] + 16);
                    if (M == 2) s_copy<16>(sdst[1] + sl, ssrc[M - 1]);
                } else {
                    if (G32) s_copy<16>(sdst[0] + sl, ssrc[0]);
                    else s_copy<8>(sdst[0] + sl, ssrc[0]);
                    if (M == 2) s_copy<8>(sdst[1] + sl, ssrc[M - 1]);
                }
                ssrc[0] += P.blk / (G32 ? 16 : 32);
                if (M == 2) ssrc[M - 1] += P.blk / 32;
            }
#pragma unroll
            for (uint32_t i = 0; i < PIECES; ++i) {
                if (blive[i]) s_copy<16>(bdst + i * B_APART + st * B_STAGE, bbase + (size_t)bsrc[i] * 8);
                bsrc[i] += SC / 8;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint64_t acc[M][NS][2] = {};   // [matrix][eight columns][row half] two columns each
    const uint32_t rsw = (g >> 1) & 3u;
    uint32_t off_c[GPC];           // of this lane's codes of each group in row g
#pragma unroll
    for (int j = 0; j < GPC; ++j) off_c[j] = ring + g * 64 + (LAYOUT == L4 ? ((2 * j) ^ rsw) << 4 : (j ^ rsw) << 4) + (LAYOUT == L2H ? t * 2 : t * 4);
    // 4-bit codes: the second piece of a group is the first one's neighbour
    const uint32_t sum_a = s_smem(sums) + (PHASE == 1 ? 2 * t : (2 * t & 3u)) * 4;
    const uint32_t bias_mask = PHASE == 2 && t >= 2 ? 0u : 0xFFFFFFFFu;   // the remainders' columns carry no bias
    const auto times = [&](float v) {
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int q = 0; q < NS; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) acc[m][q][h] = s_mul2(s_pair(v, v), acc[m][q][h]);
    };
    for (int turn = 0; turn < (RESTS ? 2 : 1); ++turn) {
        if (RESTS && turn == 1) {   // the remainders' products come on top of the sums, in units of theirs
            times(1.0f / REST);
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < P.stages * B_STAGE / 16; i += WTHREADS) reinterpret_cast<uint4*>(ring_b)[i] = make_uint4(0u, 0u, 0u, 0u);
            for (uint32_t i = threadIdx.x; i < (k / 32) * TOKENS; i += WTHREADS) sums[i] = 0.0f;   // the heads' are those of the whole rows
#pragma unroll
            for (uint32_t i = 0; i < PIECES; ++i) {
                const uint32_t p = threadIdx.x + i * WTHREADS, tok = p / PPR;
                blive[i] = blive[i] && unit[tok] < 0.0f;
                bsrc[i] -= k / 8;
            }
            bbase = T.shared ? P.xs_rest : P.xr_rest;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                csrc[m] -= row_bytes;
                ssrc[m] -= k / P.blk * (P.blk / (G32 && m == 0 ? 16 : 32));
            }
            __syncthreads();
        }
        for (uint32_t i = 0; i + 1 < P.stages; ++i) issue(i, i);
        if (turn == 0) {
            for (uint32_t i = threadIdx.x; i < (k / 32) * TOKENS; i += WTHREADS) {   // consecutive threads: consecutive sums of one row
                const uint32_t tok = i / (k / 32), grp = i % (k / 32);
                float v = 0.0f;
                if (tok < n) {
                    const uint32_t pair = T.pair_start + tok;
                    v = PHASE == 1 ? P.x_sums[(size_t)P.sorted[pair].token * (k / 32) + grp] : P.h_sums[(size_t)pair * (k / 32) + grp];
                }
                sums[grp * TOKENS + tok] = v;
            }
            if (threadIdx.x < TOKENS && threadIdx.x < n) {
                const uint32_t pair = T.pair_start + threadIdx.x;
                unit[threadIdx.x] = PHASE == 1 ? P.x_unit[P.sorted[pair].token] : P.h_unit[pair];
            }
        }
        uint32_t st = 0, fill = P.stages - 1, sa = sum_a;
#pragma unroll 1
        for (uint32_t c = 0; c < n_stages; ++c) {
            if (P.stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();                 // the stage has landed for every thread, and the one to be filled has been read by every warp
            issue(c + P.stages - 1, fill);
            const uint32_t wt = st * WSTAGE, sl = slots + ((c >> cshift) & 1u) * P.slot + (c & cmask) * (2 * GPC);
            const uint32_t bt = s_smem(ring_b) + st * B_STAGE + g * B_STRIDE + (LAYOUT == L2 ? t * 32 : t * 16);
            uint32_t sc[M][2][4], bi[M][2][4];   // [matrix][row half][two scales per word]
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t p = m == 0 ? sl + (G32 ? (c & cmask) * (2 * GPC) + (g + 8 * h) * 32 : (g + 8 * h) * 16) : sl + 2 * S0 + (g + 8 * h) * 16;
                    const uint32_t to_bias = m == 0 ? S0 : 256;
                    constexpr int W0 = (G32 ? 2 : 1) * GPC / 2, W1 = GPC / 2;
                    const int words = m == 0 ? W0 : W1;
                    const auto get = [&](uint32_t at, uint32_t (&v)[4]) {
                        if (words == 4) {
                            const uint4 u = s_load128(at);
                            v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
                        } else if (words == 2) {
                            const uint2 u = s_load64(at);
                            v[0] = u.x; v[1] = u.y;
                        } else v[0] = s_load32(at);
                    };
                    get(p, sc[m][h]);
                    get(p + to_bias, bi[m][h]);
                    if (PHASE == 2)
                        for (int i = 0; i < words; ++i) bi[m][h][i] &= bias_mask;
                }
            uint64_t part[M][NS][2] = {};
#pragma unroll
            for (int j = 0; j < GPC; ++j) {
                const uint32_t rl = wt + off_c[j];
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    uint32_t pl[8], ph[8];
                    if (LAYOUT == L4) {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const uint32_t o = (u ? rl ^ 16u : rl) + m * 1024;
                            s_unpack4(s_load32(o), P.mul, reinterpret_cast<uint32_t (&)[4]>(pl[4 * u]));
                            s_unpack4(s_load32(o + 512), P.mul, reinterpret_cast<uint32_t (&)[4]>(ph[4 * u]));
                        }
                    } else if (LAYOUT == L2) {
                        s_unpack2(s_load32(rl + m * 1024), P.mul, pl);
                        s_unpack2(s_load32(rl + m * 1024 + 512), P.mul, ph);
                    } else {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            s_unpack2h(s_load16(rl + m * 1024 + u * 8), reinterpret_cast<uint32_t (&)[4]>(pl[4 * u]));
                            s_unpack2h(s_load16(rl + m * 1024 + 512 + u * 8), reinterpret_cast<uint32_t (&)[4]>(ph[4 * u]));
                        }
                    }
                    const auto wide = [&](const uint32_t (&words)[4], int i) {
                        const float v = s_widen<SDT>(words[i >> 1], i & 1);
                        return s_pair(v, v);
                    };
#pragma unroll
                    for (uint32_t q = 0; q < NS; ++q) {
                        uint32_t bf[8];
                        {
                            const uint32_t xp = bt + q * 8 * B_STRIDE + j * 128;
                            const uint4 u = s_load128(xp), v = s_load128(xp + (LAYOUT == L2 ? 16 : 64));
                            bf[0] = u.x; bf[1] = u.y; bf[2] = u.z; bf[3] = u.w; bf[4] = v.x; bf[5] = v.y; bf[6] = v.z; bf[7] = v.w;
                        }
                        const uint32_t sp = sa + (j * 2 * TOKENS + q * (PHASE == 1 ? 8 : 4)) * 4;
                        const uint2 l2 = s_load64(sp), h2 = s_load64(sp + TOKENS * 4);
                        const uint64_t lo = (uint64_t)l2.y << 32 | l2.x, hi = (uint64_t)h2.y << 32 | h2.x;
                        uint64_t (&pt)[2] = part[m][q];
                        const auto add = [&](const float (&ds)[4], int i, uint64_t sx) {   // scales i of the stage
                            pt[0] = s_fma2(wide(sc[m][0], i), s_pair(ds[0], ds[1]), pt[0]); pt[0] = s_fma2(wide(bi[m][0], i), sx, pt[0]);
                            pt[1] = s_fma2(wide(sc[m][1], i), s_pair(ds[2], ds[3]), pt[1]); pt[1] = s_fma2(wide(bi[m][1], i), sx, pt[1]);
                        };
                        if (G32 && m == 0) {
#pragma unroll
                            for (int u = 0; u < 2; ++u) {
                                float ds[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                                for (int e = 2 * u; e < 2 * u + 2; ++e) s_mma(ds, pl[2 * e], ph[2 * e], pl[2 * e + 1], ph[2 * e + 1], bf[2 * e], bf[2 * e + 1]);
                                add(ds, 2 * j + u, u ? hi : lo);
                            }
                        } else {
                            float ds[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                            for (int e = 0; e < 4; ++e) s_mma(ds, pl[2 * e], ph[2 * e], pl[2 * e + 1], ph[2 * e + 1], bf[2 * e], bf[2 * e + 1]);
                            add(ds, j, s_add2(lo, hi));
                        }
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int q = 0; q < NS; ++q)
#pragma unroll
                    for (int h = 0; h < 2; ++h) acc[m][q][h] = s_add2(acc[m][q][h], part[m][q][h]);
            sa += GPC * 2 * TOKENS * 4;
            st = st + 1 == P.stages ? 0 : st + 1;
            fill = fill + 1 == P.stages ? 0 : fill + 1;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (RESTS && turn == 1) times(REST);
    }
    if constexpr (PHASE == 1 && !RESTS)
        if (__any_sync(0xFFFFFFFFu, lane < n && unit[lane] < 0.0f)) {
            __syncthreads();
            return w_unit_rests<SDT>(P);
        }
    // a lane holds rows g and g + 8 of two columns per eight
#pragma unroll
    for (uint32_t q = 0; q < NS; ++q) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t r = row0 + g + (i >> 1) * 8;
            const auto of = [&](int m) { return __uint_as_float((uint32_t)(acc[m][q][i >> 1] >> (32 * (i & 1)))); };
            if (PHASE == 1) {
                const uint32_t tok = q * 8 + 2 * t + (i & 1);
                if (tok >= n) continue;
                const float back = RESTS ? fabsf(unit[tok]) : unit[tok];
                float gate = of(0) * 16777216.0f * back, up = of(M - 1) * 16777216.0f * back;
                if (!T.shared && P.limit > 0.0f) {   // moe_swiglu_clamp, moe.metal:27-34 (routed experts only)
                    gate = fminf(gate, P.limit);
                    up = fminf(fmaxf(up, -P.limit), P.limit);
                }
                P.hidden[(size_t)(T.pair_start + tok) * P.f + r] = hidden_act(gate, (int)P.activation) * up;
            } else {
                const uint32_t tok = q * 4 + (2 * t & 3u) + (i & 1);
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float rest = __shfl_xor_sync(0xFFFFFFFFu, of(m), 2);
                    if (t >= 2 || tok >= n) continue;
                    const mfb_pair pr = P.sorted[T.pair_start + tok];
                    P.partial[((size_t)pr.token * (P.top_k + 1) + pr.rank) * P.d + r + 16 * m] = fmaf(rest, REST, of(m)) * 16777216.0f * unit[tok];
                }
            }
        }
    }
}

template <int SDT>
__device__ __noinline__ void w_unit_rests(const WideParams& P) {
    extern __shared__ __align__(128) uint8_t smem[];
    const WorkTile T = P.tiles[blockIdx.x / P.blocks];
    const uint32_t rb = blockIdx.x % P.blocks;
    if (T.shared && P.shared_bits == 4) w_unit<1, L4, SDT, false, 2, true>(P, T, rb, P.shared_off, smem);
    else if (T.shared) w_unit<1, L2, SDT, false, 2, true>(P, T, rb, P.shared_off, smem);
    else if (P.routed_layout == L2H) w_unit<1, L2H, SDT, true, 2, true>(P, T, rb, P.routed_off, smem);
    else if (P.routed_layout == L4 && P.gate32) w_unit<1, L4, SDT, true, 2, true>(P, T, rb, P.routed_off, smem);
    else if (P.routed_layout == L4) w_unit<1, L4, SDT, false, 2, true>(P, T, rb, P.routed_off, smem);
    else w_unit<1, L2, SDT, false, 2, true>(P, T, rb, P.routed_off, smem);
}

// NS: sets of eight columns.  A loop over as many as the tile has would keep their sums from being interleaved.
template <int PHASE, int LAYOUT, int SDT, bool G32>
__device__ __forceinline__ void w_unit_any(const WideParams& P, const WorkTile& T, uint32_t rb, const mfb_expert_offsets& off, uint8_t* smem) {
    if (T.n > 8) w_unit<PHASE, LAYOUT, SDT, G32, PHASE == 1 ? 2 : 4>(P, T, rb, off, smem);
    else w_unit<PHASE, LAYOUT, SDT, G32, PHASE == 1 ? 1 : 2>(P, T, rb, off, smem);
}

template <int PHASE, int LAYOUT, int SDT>   // LAYOUT of the routed experts in this phase; L2H only in phase 1
__global__ void __launch_bounds__(WTHREADS, PHASE == 1 ? 4 : 3) wide_kernel(const __grid_constant__ WideParams P) {
    extern __shared__ __align__(128) uint8_t smem[];
    pdl_wait();
    pdl_release();
    const uint32_t rb = blockIdx.x % P.blocks, at = blockIdx.x / P.blocks;   // the row blocks of a tile lie next to each other
    const WorkTile T = P.tiles[at];         // the list is as long as the grid
    if (at >= *P.n_tiles) return;
    if (T.slot < 0) {
        if (PHASE == 2)      // an expert that is not resident contributes nothing: its rows of the partials are cleared
            for (uint32_t o = threadIdx.x; o < 32 * WW * T.n; o += WTHREADS) {
                const mfb_pair pr = P.sorted[T.pair_start + o / (32 * WW)];
                P.partial[((size_t)pr.token * (P.top_k + 1) + pr.rank) * P.d + rb * (32 * WW) + o % (32 * WW)] = 0.0f;
            }
        return;
    }
    if (T.shared) {
        if (P.shared_bits == 4) w_unit_any<PHASE, L4, SDT, false>(P, T, rb, P.shared_off, smem);
        else w_unit_any<PHASE, L2, SDT, false>(P, T, rb, P.shared_off, smem);
        return;
    }
    if (PHASE == 1 && LAYOUT == L2H) w_unit_any<PHASE, L2H, SDT, true>(P, T, rb, P.routed_off, smem);
    else if (PHASE == 1 && LAYOUT == L4 && P.gate32) w_unit_any<PHASE, L4, SDT, true>(P, T, rb, P.routed_off, smem);
    else w_unit_any<PHASE, LAYOUT == L2H ? L2 : LAYOUT, SDT, false>(P, T, rb, P.routed_off, smem);
}

// Rows in the form the kernels multiply: times a power of two, in the order of the codes, with the sums of 32 neighbouring elements.
// HIDDEN: fp32 rows, replaced by their heads and remainders; else 16-bit rows in one or two orders, and the remainders of those that fp16
// does not hold (s_loses), which are marked.
template <bool HIDDEN>
__global__ void __launch_bounds__(256) wide_rows_kernel(const void* x, int dtype, uint32_t ldx, uint32_t k, uint32_t routed_rows, int layout, int layout_s,
                                                        __half* xr, __half* xs, float* __restrict__ sums, float* __restrict__ unit, __half* xr_rest, __half* xs_rest) {
    extern __shared__ __align__(16) float row_f[];
    __shared__ uint32_t red[8], red_n[8];
    const uint32_t r = blockIdx.x;
    pdl_wait();
    pdl_release();
    uint32_t mx = 0, mn = 0xFFFFFFFFu;   // mn: bits of the smallest element that is not zero, less one
    for (uint32_t e = threadIdx.x; e < k; e += 256) {
        const float v = HIDDEN ? reinterpret_cast<const float*>(x)[(size_t)r * k + e] : widen16(reinterpret_cast<const uint16_t*>(x)[(size_t)r * ldx + e], dtype);
        row_f[e] = v;
        const uint32_t bits = __float_as_uint(v) & 0x7FFFFFFFu;
        mx = max(mx, bits);
        if (!HIDDEN) mn = min(mn, bits - 1u);
    }
    mx = __reduce_max_sync(0xFFFFFFFFu, mx);
    if (!HIDDEN) mn = __reduce_min_sync(0xFFFFFFFFu, mn);
    if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = mx; red_n[threadIdx.x >> 5] = mn; }
    __syncthreads();
    mx = __reduce_max_sync(0xFFFFFFFFu, red[threadIdx.x & 7u]);
    float back = 1.0f / HIDDEN_FACTOR, factor = HIDDEN_FACTOR;
    if (!HIDDEN || (!s_plain(mx) && mx != 0u)) factor = s_factor(mx, back);
    if (threadIdx.x == 0) unit[r] = back;
    if (!HIDDEN && s_inexact(__uint_as_float(__reduce_min_sync(0xFFFFFFFFu, red_n[threadIdx.x & 7u]) + 1u), __uint_as_float(mx), factor, dtype,
                             layout == L4 && (!xs || layout_s == L4)))
        s_rests([&](uint32_t i) { return row_f[i]; }, k, factor, back, layout, xr_rest + (size_t)r * k, layout_s, xs ? xs_rest + (size_t)r * k : nullptr, unit + r);
    const uint32_t runs = k / 16;
    const bool shared = r >= routed_rows;
    for (uint32_t p0 = 0; p0 < runs; p0 += 256) {   // runs of sixteen elements; every lane takes part in the shuffle
        const uint32_t p = min(p0 + threadIdx.x, runs - 1);
        const bool live = p0 + threadIdx.x < runs;
        const auto put = [&](__half* head_row, __half* rest_row, auto layout_c) {
            constexpr int L = decltype(layout_c)::value;
            __align__(16) __half head[16], rest[16];
            float s = 0.0f;
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
                const float v = row_f[p * 16 + j] * factor * s_scale(j, L);
                if (HIDDEN) head_and_rest(v, head[s_pos(j, L)], rest[s_pos(j, L)]);
                else head[s_pos(j, L)] = __float2half_rn(v);
                s = fmaf(HIDDEN ? fmaf(__half2float(rest[s_pos(j, L)]), REST, __half2float(head[s_pos(j, L)])) : v, 1.0f / s_scale(j, L), s);
            }
            if (live) {
                reinterpret_cast<uint4*>(head_row)[2 * p] = *reinterpret_cast<const uint4*>(head);
                reinterpret_cast<uint4*>(head_row)[2 * p + 1] = *reinterpret_cast<const uint4*>(head + 8);
                if (HIDDEN) {
                    reinterpret_cast<uint4*>(rest_row)[2 * p] = *reinterpret_cast<const uint4*>(rest);
                    reinterpret_cast<uint4*>(rest_row)[2 * p + 1] = *reinterpret_cast<const uint4*>(rest + 8);
                }
            }
            s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);
            if (live && (p & 1u) == 0) sums[(size_t)r * (k / 32) + p / 2] = s * CODE_UNIT;
        };
        const auto put_any = [&](__half* h, __half* rest_row, int l) {
            if (l == L4) put(h, rest_row, std::integral_constant<int, L4>());
            else if (l == L2) put(h, rest_row, std::integral_constant<int, L2>());
            else put(h, rest_row, std::integral_constant<int, L2H>());
        };
        if (HIDDEN) {
            __half* const h = xr + (size_t)r * 2 * k;
            put_any(h, h + k, shared ? layout_s : layout);
        } else {
            put_any(xr + (size_t)r * k, nullptr, layout);
            if (xs) put_any(xs + (size_t)r * k, nullptr, layout_s);
        }
    }
}

// Tiles of up to sixteen rows of an expert, the shared expert's in front.
__global__ void __launch_bounds__(512) wide_tiles_kernel(const mfb_group* __restrict__ groups, const uint32_t* __restrict__ n_groups, uint32_t num_experts,
                                                         const int16_t* __restrict__ slot_of, WorkTile* __restrict__ tiles, uint32_t* __restrict__ n_tiles) {
    __shared__ uint32_t warp_sum[16];
    pdl_wait();
    pdl_release();
    const uint32_t ng = *n_groups, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool last_shared = ng && groups[ng - 1].expert >= num_experts;
    const uint32_t routed = last_shared ? ng - 1 : ng;
    uint32_t in_front = 0;
    if (last_shared) {
        const mfb_group grp = groups[ng - 1];
        in_front = (grp.pair_count + WTOK - 1) / WTOK;
        for (uint32_t i = threadIdx.x; i < in_front; i += blockDim.x) {
            WorkTile t;
            t.pair_start = grp.pair_start + i * WTOK; t.n = min(WTOK, grp.pair_count - i * WTOK); t.slot = 0; t.shared = 1u;
            tiles[i] = t;
        }
    }
    mfb_group grp = {};
    if (threadIdx.x < routed) grp = groups[threadIdx.x];
    const uint32_t mine = (grp.pair_count + WTOK - 1) / WTOK;   // a thread per group: MFB_MAX_EXPERTS of them
    uint32_t incl = mine;
    for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= off) incl += a;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    uint32_t at = in_front + incl - mine;
    for (uint32_t i = 0; i < warp; ++i) at += warp_sum[i];
    if (threadIdx.x == blockDim.x - 1) *n_tiles = at + mine;
    if (mine == 0) return;
    WorkTile t;
    t.shared = 0u;
    t.slot = slot_of ? (int32_t)slot_of[grp.expert] : (int32_t)grp.expert;
    for (uint32_t i = 0; i < mine; ++i) {
        t.pair_start = grp.pair_start + i * WTOK;
        t.n = min(WTOK, grp.pair_count - i * WTOK);
        tiles[at + i] = t;
    }
}

using WideFn = void (*)(const WideParams);
template <int SDT>
WideFn wide_fn(int phase, int layout) {
    if (phase == 2) return layout == L4 ? wide_kernel<2, L4, SDT> : wide_kernel<2, L2, SDT>;
    return layout == L4 ? wide_kernel<1, L4, SDT> : layout == L2 ? wide_kernel<1, L2, SDT> : wide_kernel<1, L2H, SDT>;
}
WideFn wide_fn(int phase, int layout, uint32_t sdt) { return sdt == MFB_DT_BF16 ? wide_fn<MFB_DT_BF16>(phase, layout) : wide_fn<MFB_DT_F16>(phase, layout); }

// A stage of columns is largest with 2-bit codes (256 codes each).
constexpr uint32_t wide_smem(uint32_t phase, uint32_t k, uint32_t stages, uint32_t slot) {
    return WW * (stages * W_STAGE * 2 + 2 * slot) + stages * (phase == 1 ? 16 : 32) * (256 * 2 + 64) + (k / 32 + 1) * WTOK * 4;
}

}  // namespace

static_assert(MFB_MAX_EXPERTS <= 512, "wide_tiles_kernel has a thread per expert");

static_assert(wide_smem(1, STREAM_LONGEST, 2, 1536) <= W_SMEM_LIMIT && wide_smem(2, STREAM_LONGEST, 2, 1024) <= W_SMEM_LIMIT,
              "every shape of the streaming kernels fits");

cudaError_t wide_init(const mfb_moe_config& c) {
    for (int phase = 1; phase <= 2; ++phase)
        for (int layout = c.bits == 4 ? L4 : L2; layout <= (c.bits == 4 ? L4 : L2H); ++layout) {
            const cudaError_t e = cudaFuncSetAttribute(wide_fn(phase, layout, c.scale_dtype), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W_SMEM_LIMIT);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

cudaError_t wide_ffn(cudaStream_t s, const mfb_moe_config& c, const mfb_layer_weights& w, const Arena& a, const void* x, uint32_t ldx, uint32_t n_tokens,
                     uint32_t max_groups) {
    const bool shared = w.shared_blob != nullptr;
    const int layout = c.bits == 4 ? L4 : w.gate_group_size == 32 ? L2H : L2, layout_s = c.shared_bits == 2 ? L2 : L4, layout_h = layout == L4 ? L4 : L2;
    const bool second = shared && layout_s != layout;
    const uint32_t pairs = n_tokens * c.top_k, rows = pairs + (shared ? n_tokens : 0u);
    // scratch: rows in xs16, what the hidden rows need in acts16; the rows' sums, factors and remainders (n * (d / 32 + 1) floats and up to
    // 2 * n * d fp16 numbers) in the n * (top_k + 1) * d floats of the partial rows, which phase 2 writes
    WideParams P;
    __half* const xr = a.xs16;
    __half* const xs = second ? xr + (size_t)n_tokens * c.d : nullptr;
    float* const x_sums = a.partial;
    float* const x_unit = x_sums + (size_t)n_tokens * (c.d / 32);
    __half* const xr_rest = reinterpret_cast<__half*>(x_sums + ((size_t)n_tokens * (c.d / 32 + 1) + 3) / 4 * 4);   // 16-byte pieces
    __half* const xs_rest = second ? xr_rest + (size_t)n_tokens * c.d : xr_rest;
    uint8_t* at = reinterpret_cast<uint8_t*>(a.acts16);
    const auto take = [&](size_t bytes) { uint8_t* p = at; at += (bytes + 255) / 256 * 256; return p; };
    const uint32_t most_tiles = rows / WTOK + max_groups;
    float* const h_sums = reinterpret_cast<float*>(take((size_t)rows * (c.f / 32) * 4));
    float* const h_unit = reinterpret_cast<float*>(take((size_t)rows * 4));
    WorkTile* const tiles = reinterpret_cast<WorkTile*>(take((size_t)most_tiles * sizeof(WorkTile)));
    uint32_t* const n_tiles = reinterpret_cast<uint32_t*>(take(4));
    P.pool = w.pool; P.shared_blob = w.shared_blob; P.slot_stride = w.slot_stride; P.routed_off = w.routed_off; P.shared_off = w.shared_off;
    P.d = c.d; P.f = c.f; P.top_k = c.top_k; P.shared_bits = c.shared_bits; P.activation = c.activation; P.gate32 = w.gate_group_size == 32 ? 1u : 0u;
    P.limit = c.swiglu_limit; P.sorted = a.sorted; P.tiles = tiles; P.n_tiles = n_tiles; P.xr = xr; P.xs = second ? xs : xr;
    P.xr_rest = xr_rest; P.xs_rest = xs_rest; P.routed_layout = layout;
    P.x_sums = x_sums; P.x_unit = x_unit; P.hidden = a.acts; P.h_sums = h_sums; P.h_unit = h_unit; P.partial = a.partial;
    MFB_TRY(launch_dependent(wide_tiles_kernel, dim3(1), dim3(512), 0, s, a.groups, a.n_groups, c.num_experts, w.slot_of, tiles, n_tiles));
    MFB_TRY(launch_dependent(wide_rows_kernel<false>, dim3(n_tokens), dim3(256), c.d * 4, s, x, (int)c.x_dtype, ldx, c.d, n_tokens, layout, layout_s, xr, xs, x_sums, x_unit, xr_rest, xs_rest));
    for (uint32_t phase = 1; phase <= 2; ++phase) {
        const uint32_t k = phase == 1 ? c.d : c.f;
        P.slot = phase == 1 && P.gate32 ? 1536u : 1024u;
        P.blk = k % 512 == 0 ? 512u : 256u;
        P.blocks = phase == 1 ? c.f / (16 * WW) : c.d / (32 * WW);
        // a scale slot holds at most blk codes: the ring is never ahead of it by more (stream.cu)
        const uint32_t stage_codes = layout == L4 && (!shared || layout_s == L4) ? 128u : 256u;
        P.stages = P.blk / stage_codes >= 2 && wide_smem(phase, k, 3, P.slot) <= (phase == 1 ? W_SMEM_FOUR : W_SMEM_LIMIT) ? 3u : 2u;
        MFB_TRY(launch_dependent(wide_fn((int)phase, phase == 1 ? layout : layout_h, c.scale_dtype), dim3(most_tiles * P.blocks), dim3(WTHREADS),
                                 wide_smem(phase, k, P.stages, P.slot), s, P));
        if (phase == 1)
            MFB_TRY(launch_dependent(wide_rows_kernel<true>, dim3(rows), dim3(256), c.f * 4, s, (const void*)a.acts, 0, c.f, c.f, pairs, layout_h, layout_s,
                                     reinterpret_cast<__half*>(a.acts), (__half*)nullptr, h_sums, h_unit, (__half*)nullptr, (__half*)nullptr));
    }
    count_launches(5);
    return cudaSuccess;
}

}  // namespace mfb
