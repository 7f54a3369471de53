// Prefill attention over the packed spike pools on the fifth-generation tensor cores (tcgen05), 16-bit outputs, head_dim 64 or 128.
//
// CTA = (128 query tokens of one portion, timestep, query head), two CTAs per SM.  Thirteen warps (nine in the form of many short portions, below):
//  * warps 8-11 read the packed K and V rows of 64 keys through the block table and turn their bits into operands: K e4m3 bytes, V halves, each
//    a masked word as it is, in the swizzled operand layouts; a stage ahead of the MMAs, the next stage's words already in registers;
//  * warp 12 issues S = Q K^T (kind::f8f6f4, exact: scores are counts) and O += P V (kind::f16, P read from TMEM).  S of step t + 1 goes out as
//    soon as S of step t has been read, ahead of the wait for the weights of step t;
//  * warps 0-7, two threads per query row (32 keys of a step each), turn scores into weights exp((score - popc(q)) * scale) * 2^14 in halves.
//    popc(q) bounds every score of the row: no running maximum, no rescaling of O, and 2^14 keeps the smallest possible weight a normal half.
//    Their 32-bit sum, also times 2^14, divides the row at the end.  For fp16 outputs, whose rounding is as fine as the weights', the sum takes the
//    weights as they are rounded: keys of one score share their rounding, which then cancels (error against 64 bits, three portions of up to
//    300 tokens behind 200, heads of 64 and 128: 2.32e-4 and 2.30e-4 with the sum of the unrounded ones, 2.15e-4 and 2.14e-4 so, 2.20e-4 and 2.29e-4 by
//    SDPA in fp16); bf16 results, whose rounding is 8 times coarser, sum the unrounded ones.
// Bits expand in an order that is cheapest for the bit tricks (byte b of word j: bit j + 8 b; half h: bit j + 16 h), the same for Q and K;
// V's column order is undone when a row is stored.
//
// What bounds it: no pipe by itself.  At 128 channels and 23 steps a CTA the special-function pipe (one exponential per (query, key) pair) is 50 % busy, the
// load/store path's data pipe (operands written, scores and weights moved to and from TMEM) 46 %, TMEM 44 %, the tensor pipe 38 %, issue 50 %, and the MMAs
// read 40 KB of operands a step from shared memory beside that; two CTAs leave some of their waits uncovered.  For prompts of a few hundred tokens a CTA's
// set-up and drain count: 16 x 512 tokens at 64 channels keep the special-function pipe 34 % busy.  Why 64 keys per step: scores, two buffers of weights and O of up to 128
// channels are 256 TMEM columns, so that two CTAs fit an SM and one's set-up and drain hide behind the other's steps.
// Measured, whole fused_qkv_attention calls: three portions of 766 to 1531 tokens behind 700 cached, 28/4 heads of 128, 338 -> 294 us; four of 875
// to 2000 behind 300, 7/1 heads of 128, 137 -> 118; 16 x 512 tokens, 14/2 heads of 64, 130 -> 123 (with one warpgroup on scores).  What came before: comparisons with the
// diagonal in every step and shifts and products per operand register (190 M instructions, 131 M without them), a warp per 32 rows on
// scores (its waits and its exponentials took turns), S behind the weights' product of two steps before.  With 64 keys per
// warpgroup and step (even and odd steps): 307 us; one warpgroup that reads all 64 scores ahead: 324.
#include <algorithm>
#include <type_traits>

#include "spk_tensor.cuh"

namespace {

using namespace spk_tc;

constexpr int kRows = 128;                  // query tokens per CTA
constexpr int kKeys = 64;                   // keys per step
constexpr int kStages = 3;
constexpr int threads_of(int wgs) { return 128 * wgs + 160; }  // WGS warpgroups on scores, one on operands, one warp on MMAs
constexpr int kQBytes = kRows * 128;        // rows of 128 bytes; 64 channels use the first half
constexpr int kKBytes = kKeys * 128;
constexpr int kVColTile = kKeys * 128;      // 64 channels
constexpr uint32_t kTmemS = 0, kTmemP = kKeys, kTmemO = 128;  // scores, two buffers of weights (32 columns each), weighted sum
constexpr int kMaxPortions = 48, kMaxTiles = 512;
constexpr float kLog2e = 1.4426950408889634f;

struct Launch {
    spk_spike_prefill_args a;
    spk_spike_portion portions[kMaxPortions];
    uint32_t tiles[kMaxTiles];  // portion << 24 | query tile of the portion
    int vec;                    // rows of the output allow 16-byte stores
};

struct Bars {
    uint64_t kv_full[kStages], kv_free[kStages], s_full, s_read, p_full[2], q_full, o_full;
    int abort;
    uint32_t tmem;
};

__device__ __forceinline__ void mma_f8_by(uint32_t who, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1 : 0), "r"(who) : "memory");
}
__device__ __forceinline__ void mma_ts_by(uint32_t who, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc ? 1 : 0), "r"(who) : "memory");
}

__device__ __forceinline__ void st_shared16(uint32_t addr, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

// Operands are the packed bits IN PLACE, one logic operation per register: what a masked bit stands for depends on its position alone, a power of
// two that the other operand, or the store of the result, takes out again.
//
// One word's 32 channels as e4m3 bytes at 16-byte groups 2 w and 2 w + 1 of a 128-byte row; row: shared address of the row plus (row & 7) << 4, the
// swizzle.  Register j holds bits j + 8 b; bit e = j % 4 of a byte reads as 2^(e - 9), so a query's register holds 2^(3 - e) where its bit is set
// and every matching bit adds 2^-6 to a score.
constexpr float kScoreUnit = 64.0f;
template <bool QUERY>
__device__ __forceinline__ void expand_bytes(uint32_t row, int w, uint32_t bits) {
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        const uint32_t from = g == 0 ? bits : bits >> 4;
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = QUERY ? ((from >> e) & 0x01010101u) * ((10u - e) << 3) : from & (0x01010101u << e);
        st_shared16(row ^ ((2 * w + g) << 4), v);
    }
}
// One word's 32 channels as halves, four groups of a 64-channel column tile.  Register j holds bits j and j + 16, moved by 4, 8 or 12 (bit 15: by -1) to
// one of positions 11 to 14 of a half: 2^-13, 2^-11, 2^-7 or 2, a normal number each (in a subnormal one a product would lose bits beside
// larger ones of the sum); channel_unit(j) is what takes that out of a column's sum.
__device__ __forceinline__ void expand_halves(uint32_t row, int w, uint32_t bits) {
    const uint32_t moved[5] = {bits << 12, bits << 8, bits << 4, bits, bits >> 1};
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = 4 * g + i, m = j == 15 ? 4 : (j + 1) / 4;
            v[i] = moved[m] & (0x00010001u << (m == 4 ? 14 : j + 12 - 4 * m));
        }
        st_shared16(row ^ ((4 * (w & 1) + g) << 4), v);
    }
}
__device__ __forceinline__ constexpr float channel_unit(int j) {
    return j == 15 || j % 4 == 2 ? 0.5f : j % 4 == 3 ? 8192.0f : j % 4 == 0 ? 2048.0f : 128.0f;
}

template <typename TO>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float lo, float hi) { return pack_bf16(lo, hi); }
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

template <int W>
constexpr int shared_bytes() { return kQBytes + kStages * (kKBytes + W / 2 * kVColTile) + 1024 + 256; }

// WGS: warpgroups on scores.  Two halve the time of a step; one leaves registers for a third CTA per SM at 64 channels, which sets itself up while it
// waits for the tensor memory of one that ends.
template <int W, typename TO, int WGS>
__global__ void __launch_bounds__(threads_of(WGS), WGS == 1 && W == 2 ? 3 : 2)
spike_prefill_kernel(const __grid_constant__ Launch l) {
    constexpr int kVBytes = W / 2 * kVColTile, kScoreWarps = 4 * WGS, kMmaWarp = kScoreWarps + 4;
    extern __shared__ uint8_t raw[];
    uint8_t* q_s = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    uint8_t* k_s = q_s + kQBytes;
    uint8_t* v_s = k_s + kStages * kKBytes;
    Bars* bars = reinterpret_cast<Bars*>(v_s + kStages * kVBytes);
    const spk_spike_prefill_args& a = l.a;
    const int warp = threadIdx.x >> 5;
    const int h = blockIdx.x % a.num_q_heads, ts = blockIdx.x / a.num_q_heads;
    const int g = h / (a.num_q_heads / a.num_kv_heads);
    const uint32_t tile = l.tiles[blockIdx.y];
    const spk_spike_portion& por = l.portions[tile >> 24];
    const int first = static_cast<int>(tile & 0xffffffu) * kRows;  // query row of the portion
    const int nq = por.tokens - first < kRows ? por.tokens - first : kRows;
    const int pos0 = por.context + first;
    const int keys = pos0 + nq;
    const int steps = (keys + kKeys - 1) / kKeys;

    // what the first copies wait for is on its way before the set-up below: the table entries of the first two steps' keys, the query's words
    const int e = threadIdx.x & 127, key = e & (kKeys - 1), half = e >> 6;
    const int bs_log2 = 31 - __clz(a.block_size), bs_mask = a.block_size - 1;
    auto entry = [&](int t) {
        const int j = t * kKeys + key;
        return j < keys ? por.table[j >> bs_log2] : -1;
    };
    const int64_t token = por.start + first + e;
    int block0 = -1, block = -1;
    uint32_t qw[W];
    if (warp >= kScoreWarps && warp < kMmaWarp) {
        block0 = entry(0);
        block = entry(1);
    } else if (warp < kScoreWarps) {
        const uint32_t* q = static_cast<const uint32_t*>(a.q_packed) + ts * a.sq_t + token * a.sq_tok + h * a.sq_h;
#pragma unroll
        for (int w = 0; w < W; ++w) qw[w] = e < nq ? q[w] : 0u;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(smem_u32(&bars->kv_full[i]), 128);
            mbar_init(smem_u32(&bars->kv_free[i]), 1);
        }
        mbar_init(smem_u32(&bars->s_full), 1);
        mbar_init(smem_u32(&bars->s_read), 32 * kScoreWarps);
        for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&bars->p_full[i]), 32 * kScoreWarps);
        mbar_init(smem_u32(&bars->q_full), 128);
        mbar_init(smem_u32(&bars->o_full), 1);
        bars->abort = 0;
    }
    if (warp == kMmaWarp) tmem_alloc(smem_u32(&bars->tmem), 256);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem;
    volatile int* abort = &bars->abort;

    if (warp >= kScoreWarps && warp < kMmaWarp) {  // ---- K and V bits to operands: thread = (key, half of the words)
        const uint32_t* kp = static_cast<const uint32_t*>(a.k_pool) + ts * a.sk_t + g * a.sk_h + half * (W / 2);
        const uint32_t* vp = static_cast<const uint32_t*>(a.v_pool) + ts * a.sv_t + g * a.sv_h + half * (W / 2);
        uint32_t kw[W / 2], vw[W / 2];
        auto fetch = [&](int t, int block) {
            const int j = t * kKeys + key;
#pragma unroll
            for (int i = 0; i < W / 2; ++i) kw[i] = vw[i] = 0u;
            if (j >= keys) return;
            if (block < 0 || block >= a.num_blocks) {
                spk_flag(a.status, SPK_STATUS_BAD_BLOCK);
                return;
            }
            const int64_t ko = block * a.sk_blk + (j & bs_mask) * a.sk_slot, vo = block * a.sv_blk + (j & bs_mask) * a.sv_slot;
#pragma unroll
            for (int i = 0; i < W / 2; ++i) {
                kw[i] = kp[ko + i];
                vw[i] = vp[vo + i];
            }
        };
        fetch(0, block0);
        for (int t = 0; t < steps; ++t) {
            const int stage = t % kStages;
            uint32_t kb[W / 2], vb[W / 2];
#pragma unroll
            for (int i = 0; i < W / 2; ++i) {
                kb[i] = kw[i];
                vb[i] = vw[i];
            }
            if (t + 1 < steps) {
                fetch(t + 1, block);
                block = entry(t + 2);
            }
            if (t >= kStages && !__all_sync(~0u, mbar_wait(smem_u32(&bars->kv_free[stage]), ((t / kStages) - 1) & 1, abort))) break;
            const uint32_t at = key * 128 + ((key & 7) << 4), kr = smem_u32(k_s) + stage * kKBytes + at, vr = smem_u32(v_s) + stage * kVBytes + at;
#pragma unroll
            for (int i = 0; i < W / 2; ++i) {
                const int w = half * (W / 2) + i;
                expand_bytes<false>(kr, w, kb[i]);
                expand_halves(vr + (w >> 1) * kVColTile, w, vb[i]);
            }
            fence_async_shared();
            mbar_arrive(smem_u32(&bars->kv_full[stage]));
        }
    } else if (warp == kMmaWarp) {  // ---- MMAs
        constexpr uint32_t s_desc = (1u << 4) | (static_cast<uint32_t>(kKeys >> 3) << 17) | (static_cast<uint32_t>(kRows >> 4) << 24);
        constexpr uint32_t o_desc = (1u << 4) | (1u << 16) | (static_cast<uint32_t>(W * 32 >> 3) << 17) | (static_cast<uint32_t>(kRows >> 4) << 24);
        const uint32_t who = elect_one();
        auto scores = [&](int t) {
            const int stage = t % kStages;
            if (!mbar_wait(smem_u32(&bars->kv_full[stage]), (t / kStages) & 1, abort)) return false;
            tc_fence_after();
            const uint64_t qd = desc_sw128(smem_u32(q_s), 16, 1024), kd = desc_sw128(smem_u32(k_s + stage * kKBytes), 16, 1024);
#pragma unroll
            for (int s = 0; s < W; ++s)  // 32 channels (32 bytes of a row) per MMA
                mma_f8_by(who, tmem + kTmemS, qd + 2 * s, kd + 2 * s, s_desc, s > 0);
            if (who) mma_commit(smem_u32(&bars->s_full));
            return true;
        };
        bool ok = __all_sync(~0u, mbar_wait(smem_u32(&bars->q_full), 0, abort)) && __all_sync(~0u, scores(0));
        for (int t = 0; ok && t < steps; ++t) {
            const int stage = t % kStages;
            // S of step t + 1 as soon as that of step t is in registers, ahead of the wait for the weights
            if (t + 1 < steps) ok = __all_sync(~0u, mbar_wait(smem_u32(&bars->s_read), t & 1, abort) && scores(t + 1));
            ok = ok && __all_sync(~0u, mbar_wait(smem_u32(&bars->p_full[t & 1]), (t >> 1) & 1, abort));
            if (!ok) break;
            tc_fence_after();
            const uint64_t vd = desc_sw128(smem_u32(v_s + stage * kVBytes), kVColTile, 1024);
#pragma unroll
            for (int s = 0; s < kKeys / 16; ++s)
                mma_ts_by(who, tmem + kTmemO, tmem + kTmemP + (t & 1) * (kKeys / 2) + s * 8, vd + s * (2048 >> 4), o_desc, t > 0 || s > 0);
            if (who) mma_commit(smem_u32(&bars->kv_free[stage]));
            __syncwarp();
        }
        if (who) mma_commit(smem_u32(&bars->o_full));
        mbar_wait(smem_u32(&bars->o_full), 0);
    } else {  // ---- scores to weights: thread = query row; of two warpgroups the first takes the first 32 keys of a step, the second the others
        const int r = e, wg = warp >> 2;
        uint64_t c1, c0;
        {
            int ones = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                ones += __popc(qw[w]);
                if (wg == 0) expand_bytes<true>(smem_u32(q_s) + r * 128 + ((r & 7) << 4), w, qw[w]);
            }
            if (wg == 0) {
                fence_async_shared();
                mbar_arrive(smem_u32(&bars->q_full));
            }
            const float c = a.scale * kLog2e, b = 14.0f - ones * c;
            c1 = f2_pack(c * kScoreUnit, c * kScoreUnit);
            c0 = f2_pack(b, b);
        }
        const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
        uint64_t sums = f2_pack(0.0f, 0.0f), other = sums;  // of this half of a step's keys, and of the other where one warpgroup takes both
        bool ok = true;
        for (int t = 0; t < steps; ++t) {
            // also says that the product of step t - 2, issued before these scores, is complete: its weights lay where step t's go
            ok = __all_sync(~0u, mbar_wait(smem_u32(&bars->s_full), t & 1, abort));
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = wg; c < (WGS == 2 ? wg + 1 : 2); ++c) {
                uint32_t sc[32], p[16];
                tmem_ld32(tmem + lanes + kTmemS + c * 32, sc);
                tmem_wait_ld(sc);
                if (WGS == 2 || c == 1) {
                    tc_fence_before();
                    mbar_arrive(smem_u32(&bars->s_read));
                }
                const int seen = pos0 + r - t * kKeys - c * 32;  // last visible column of this row
                auto weights = [&](auto masked) {  // the two forms are code of their own: only the steps on the diagonal compare columns
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float x, y;
                        f2_unpack(f2_fma(f2_pack(__uint_as_float(sc[2 * i]), __uint_as_float(sc[2 * i + 1])), c1, c0), x, y);
                        x = ex2(x);
                        y = ex2(y);
                        if (decltype(masked)::value) {
                            x = 2 * i <= seen ? x : 0.0f;
                            y = 2 * i + 1 <= seen ? y : 0.0f;
                        }
                        p[i] = pack_pair<__half>(x, y);
                        if (std::is_same<TO, __half>::value) {  // the weights as they enter the product
                            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&p[i]));
                            x = v.x;
                            y = v.y;
                        }
                        sums = f2_add(sums, f2_pack(x, y));
                    }
                };
                if (__all_sync(~0u, seen >= 31)) {
                    weights(std::false_type{});
                } else if (__all_sync(~0u, seen < 0)) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) p[i] = 0u;
                } else {
                    weights(std::true_type{});
                }
                tmem_st16(tmem + lanes + kTmemP + (t & 1) * (kKeys / 2) + c * 16, p);
                if (WGS == 1) {
                    const uint64_t mine = sums;
                    sums = other;
                    other = mine;
                }
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(smem_u32(&bars->p_full[t & 1]));  // one per parity: a fast warp may be a step ahead of a slow one, not two
        }
        float x, y;
        f2_unpack(sums, x, y);
        ok = __all_sync(~0u, ok && mbar_wait(smem_u32(&bars->o_full), 0, abort) && *abort == 0);
        tc_fence_after();
        float sum = x + y;  // the halves' sums are added up last in either form: the same bits
        if (WGS == 2) {     // through the query's operand (every MMA is complete)
            float* parts = reinterpret_cast<float*>(q_s);
            parts[wg * kRows + r] = sum;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            sum = parts[r] + parts[kRows + r];
        } else {
            f2_unpack(other, x, y);
            sum += x + y;
        }
        const float inv = ok && r < nq ? 1.0f / sum : 0.0f;
        TO* out = static_cast<TO*>(a.out) + ts * a.so_t + token * a.so_tok + h * a.so_h;
#pragma unroll
        for (int i = 0; i < W / WGS; ++i) {  // each warpgroup stores its share of the words
            const int w = wg * (W / WGS) + i;
            uint32_t o[32];
            tmem_ld32(tmem + lanes + kTmemO + w * 32, o);
            tmem_wait_ld(o);
            if (r < nq) {
                // column 2 j is channel j of the word, column 2 j + 1 channel j + 16
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    uint32_t v[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int j = (m & 1) * 8 + 2 * k;
                        const float lo = __uint_as_float(o[2 * j + (m >> 1)]) * (inv * channel_unit(j));
                        const float hi = __uint_as_float(o[2 * j + 2 + (m >> 1)]) * (inv * channel_unit(j + 1));
                        v[k] = ok ? pack_pair<TO>(lo, hi) : 0u;
                    }
                    TO* dst = out + w * 32 + m * 8;
                    if (l.vec) {
                        *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            reinterpret_cast<uint16_t*>(dst)[2 * k] = static_cast<uint16_t>(v[k]);
                            reinterpret_cast<uint16_t*>(dst)[2 * k + 1] = static_cast<uint16_t>(v[k] >> 16);
                        }
                    }
                }
            }
            __syncwarp();
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0 && *abort != 0) spk_flag(a.status, SPK_STATUS_DEVICE_WAIT_EXPIRED);
    if (warp == kMmaWarp) tmem_dealloc(tmem, 256);
}

template <int W, typename TO, int WGS>
int launch(const Launch& l, int tiles, cudaStream_t s) {
    constexpr int bytes = shared_bytes<W>();
    static_assert(sizeof(Bars) <= 256 && 2 * bytes <= 224 * 1024, "shared memory of two CTAs");
    static_assert(sizeof(Launch) <= 4096, "kernel parameters");
    const cudaError_t e = cudaFuncSetAttribute(spike_prefill_kernel<W, TO, WGS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return spk_set_cuda_error(e);
    spike_prefill_kernel<W, TO, WGS><<<dim3(l.a.num_q_heads * l.a.T, tiles), threads_of(WGS), bytes, s>>>(l);
    SPK_CHECK_LAUNCH();
    return SPK_OK;
}

}  // namespace

extern "C" int spk_spike_prefill_form(int head_dim, int out_dtype) {
    return (head_dim == 64 || head_dim == 128) && (out_dtype == SPK_BF16 || out_dtype == SPK_F16);
}

extern "C" int spk_spike_prefill(const spk_spike_prefill_args* args, const spk_spike_portion* portions, int n_portions, void* stream) {
    if (args == nullptr || (n_portions > 0 && portions == nullptr)) return SPK_ERR_NULL_POINTER;
    const spk_spike_prefill_args& a = *args;
    if (!spk_spike_prefill_form(a.head_dim, a.dtype)) return SPK_ERR_UNSUPPORTED;
    if (a.T < 1 || a.num_q_heads < 1 || a.num_kv_heads < 1 || a.num_q_heads % a.num_kv_heads != 0 || a.num_blocks < 1 || a.block_size < 1 ||
        (a.block_size & (a.block_size - 1)) != 0 || n_portions < 0)
        return SPK_ERR_BAD_SHAPE;
    if (!(a.scale > 0.0f) || a.scale * a.head_dim > 16.0f) return SPK_ERR_UNSUPPORTED;  // the smallest weight has to stay a normal half
    if (a.q_packed == nullptr || a.k_pool == nullptr || a.v_pool == nullptr || a.out == nullptr) return SPK_ERR_NULL_POINTER;
    const int64_t heads = static_cast<int64_t>(a.num_q_heads) * a.T;
    if (heads > 0x7fffffff) return SPK_ERR_TOO_LARGE;
    for (int i = 0; i < n_portions; ++i) {
        const spk_spike_portion& p = portions[i];
        if (p.tokens < 0 || p.context < 0 || p.start < 0 || p.start > a.n_tok || p.tokens > a.n_tok - p.start) return SPK_ERR_BAD_SHAPE;
        const int64_t keys = static_cast<int64_t>(p.context) + p.tokens;
        if (p.tokens > 0 && p.table == nullptr) return SPK_ERR_NULL_POINTER;
        if (keys > 0x7fffffff - 2 * kKeys) return SPK_ERR_TOO_LARGE;
        if (p.tokens > 0 && keys > static_cast<int64_t>(p.table_len) * a.block_size) return SPK_ERR_BAD_SHAPE;
    }
    Launch l;
    l.a = a;
    l.vec = reinterpret_cast<uintptr_t>(a.out) % 16 == 0 && a.so_t % 8 == 0 && a.so_tok % 8 == 0 && a.so_h % 8 == 0;
    int held = 0, tiles = 0, keys_of[kMaxTiles] = {}, rc = SPK_OK;
    auto flush = [&]() {
        // the tiles that see the most keys start first
        uint32_t order[kMaxTiles];
        int by[kMaxTiles];
        for (int i = 0; i < tiles; ++i) by[i] = i;
        std::stable_sort(by, by + tiles, [&](int x, int y) { return keys_of[x] > keys_of[y]; });
        for (int i = 0; i < tiles; ++i) order[i] = l.tiles[by[i]];
        std::copy(order, order + tiles, l.tiles);
        const cudaStream_t s = spk_stream(stream);
        if (tiles > 0) {
            // One warpgroup on scores at 64 channels where a launch is many short CTAs: up to eight steps, and a wave of a CTA per SM for each of them.  Two warpgroups / one, us,
            // 14/2 heads: 8 x 64 tokens 9.6 / 8.5, 16 x 64 16.0 / 13.8, 32 x 64 27.8 / 22.9, 16 x 128 21.5 / 20.5, 8 x 256 24.1 / 23.5, 16 x 512 98.6 / 91.4; the other way round 4 x 256
            // 13.7 / 13.9, 4 x 512 28.1 / 29.5, 16 x 64 behind 400 33.8 / 35.0, 1 x 1000 21.1 / 24.6.
            const int steps = (*std::max_element(keys_of, keys_of + tiles) + kKeys - 1) / kKeys;
            const bool brief = steps <= 8 && static_cast<int64_t>(steps) * 148 <= heads * tiles;
            if (a.head_dim == 64 && brief) rc = a.dtype == SPK_BF16 ? launch<2, __nv_bfloat16, 1>(l, tiles, s) : launch<2, __half, 1>(l, tiles, s);
            else if (a.head_dim == 64) rc = a.dtype == SPK_BF16 ? launch<2, __nv_bfloat16, 2>(l, tiles, s) : launch<2, __half, 2>(l, tiles, s);
            else rc = a.dtype == SPK_BF16 ? launch<4, __nv_bfloat16, 2>(l, tiles, s) : launch<4, __half, 2>(l, tiles, s);
        }
        held = tiles = 0;
    };
    for (int i = 0; i < n_portions && rc == SPK_OK; ++i) {
        const int n = (portions[i].tokens + kRows - 1) / kRows;
        for (int t = 0; t < n && rc == SPK_OK; ++t) {
            if (t == 0 || held == 0) l.portions[held++] = portions[i];
            l.tiles[tiles] = static_cast<uint32_t>(held - 1) << 24 | static_cast<uint32_t>(t);
            keys_of[tiles] = portions[i].context + std::min((t + 1) * kRows, portions[i].tokens);
            if (++tiles == kMaxTiles || (held == kMaxPortions && t + 1 == n)) flush();
        }
    }
    if (rc == SPK_OK) flush();
    return rc;
}
