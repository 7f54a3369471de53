// Prefill attention with sigmoid key weights on the fifth-generation tensor cores (tcgen05), bf16, head sizes up to 128.
//
// CTA = (128 query tokens of one portion, query head).  Warps, W of them for the weights (16, or 8 in the paired form):
//  * warps W and W + 3 copy K and V: a page of the pool is stored as the swizzled operand tile it becomes, so a 128-key tile is a
//    handful of plain bulk copies (cp.async.bulk), no tensor map, whatever pages the block table names; one copy per lane, the
//    next tile's block-table entries are read ahead;
//  * warp W + 1 (one thread) issues S = Q K^T into a TMEM buffer, warp W + 2 (one thread) O += P V with P read from TMEM,
//    so that neither kind of MMA waits behind the other's operands;
//  * the others turn scores into weights, one thread per query row and half of the columns.  Sixteen warps take even and odd tiles in two
//    score buffers: 1.4 us per tile of keys.  The paired form, for heads of up to 64 channels (values of 128 leave no room for a second
//    accumulator), has one buffer and eight warps, so that two CTAs fit an SM: a tile takes 2.4 us alone and 2.8 beside another CTA, but one
//    CTA's start and end hide behind the other's tiles.  14 heads of 64, sixteen warps / paired: 16 x 512 tokens 60.8 / 42.9 us, 2048 tokens of
//    one prompt 29.5 / 45.4, 512 tokens behind 4096 56.2 / 91.4.  spk_sigmoid_attn_paired draws the line.  Both give the same bits.
// A weight is sigmoid(score) of its own key: no running maximum, no rescaling of O, no denominator.  Weights are computed in
// 32 bits and enter the product as a bf16 pair (hi + lo: 16 significant bits), so O is a 32-bit sum of them to 2^-17.
// Visible keys are those up to the query's own position; the last tile's rows of V beyond the portion's end are cleared in
// shared memory (a page's unwritten rows may hold anything, and 0 * NaN is NaN).
#include "spk_paged_attn.cuh"
#include "spk_tensor.cuh"

namespace {

using namespace spk_tc;

constexpr int kTile = 128;            // query rows, and keys per step
constexpr int kColTile = kTile * 128; // bytes of a 64-channel column tile
constexpr float kLog2e = 1.4426950408889634f;

// NB: score buffers, and parities of tiles.
template <int CK, int CV, int NB>
struct Shape {
    static constexpr int NS = NB == 2 && CK + CV <= 2 ? 4 : 2;  // stages of K and of V
    static constexpr int kSigmoidWarps = 8 * NB, kSigmoidThreads = 32 * kSigmoidWarps, kThreads = kSigmoidThreads + 128;
    static constexpr uint32_t kTmemS = 0, kTmemLo = NB * 128, kTmemO = NB * 192, kColumns = NB * 256;  // S/P-hi, P-lo, O
    static constexpr int kK = CK * kColTile, kV = CV * kColTile;
    static constexpr int kBytes = kK + NS * (kK + kV) + 1024 + 256;
};

struct Bars {
    uint64_t k_full[4], k_free[4], v_full[4], v_free[4], s_full[2], p_full[2], p_free[2], o_full, q_full, s_done;
    int abort;
    uint32_t tmem;
};

template <int CK, int CV, int NB>
__global__ void __launch_bounds__(Shape<CK, CV, NB>::kThreads, 3 - NB)
sigmoid_prefill_kernel(const spk_sigmoid_attn_args a) {
    using Sh = Shape<CK, CV, NB>;
    constexpr int NS = Sh::NS, W = Sh::kSigmoidWarps, kThreads = Sh::kThreads, kSigmoidThreads = Sh::kSigmoidThreads;
    constexpr uint32_t kTmemS = Sh::kTmemS, kTmemLo = Sh::kTmemLo, kTmemO = Sh::kTmemO;
    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_s = base;
    uint8_t* k_s = q_s + Sh::kK;
    uint8_t* v_s = k_s + NS * Sh::kK;
    Bars* bars = reinterpret_cast<Bars*>(v_s + NS * Sh::kV);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int h = blockIdx.x;
    const int g = h / (a.heads / a.kv_heads);
    const int4 tile = reinterpret_cast<const int4*>(a.tiles)[blockIdx.y];
    const int64_t t0 = tile.x;
    const int nq = tile.y, row = tile.z, pos0 = tile.w;
    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + t0 * a.out_stride + static_cast<int64_t>(h) * a.vdim;
    // uniform over the CTA: nothing has been set up yet
    if (row < 0 || row >= a.table_rows || pos0 < 0 || nq < 1 || nq > kTile ||
        static_cast<int64_t>(pos0) + nq > a.max_blocks * a.block_size) {
        if (threadIdx.x == 0) spk_flag(a.status, SPK_STATUS_BAD_SEQ_LEN);
        for (int i = threadIdx.x; i < nq * a.vdim && nq <= kTile; i += kThreads)
            out[(i / a.vdim) * a.out_stride + i % a.vdim] = __float2bfloat16_rn(0.0f);
        return;
    }
    const int keys = pos0 + nq;
    const int tiles = (keys + kTile - 1) / kTile;

    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(smem_u32(&bars->k_full[i]), 1);
            mbar_init(smem_u32(&bars->k_free[i]), 1);
            mbar_init(smem_u32(&bars->v_full[i]), 1);
            mbar_init(smem_u32(&bars->v_free[i]), 1);
        }
        for (int i = 0; i < NB; ++i) {
            mbar_init(smem_u32(&bars->s_full[i]), 1);
            mbar_init(smem_u32(&bars->p_full[i]), 256);
            mbar_init(smem_u32(&bars->p_free[i]), 1);
        }
        mbar_init(smem_u32(&bars->o_full), 1);
        mbar_init(smem_u32(&bars->s_done), 1);
        mbar_init(smem_u32(&bars->q_full), kSigmoidThreads);
        bars->abort = 0;
    }
    if (warp == 0) tmem_alloc(smem_u32(&bars->tmem), Sh::kColumns);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem;
    volatile int* abort = &bars->abort;

    if (warp == W || warp == W + 3) {  // ---- K or V copies
        const bool is_k = warp == W;
        const int cols = is_k ? CK : CV;
        const int gran = a.block_size < kTile ? a.block_size : kTile;  // rows per copy
        const int per = kTile / gran;                                  // copies per column tile, at most 8
        const int p = lane % per, c = lane / per;                      // this lane's copy
        const int bs_log2 = 31 - __clz(a.block_size);
        const int32_t* table = a.tables + static_cast<int64_t>(row) * a.table_stride;
        const SpkPageLayout lay{a.kv_heads, a.block_size, is_k ? a.k_pad : a.v_pad, 1};
        const __nv_bfloat16* pool = static_cast<const __nv_bfloat16*>(is_k ? a.k_pool : a.v_pool);
        uint8_t* stages = is_k ? k_s : v_s;
        const int stage_bytes = is_k ? Sh::kK : Sh::kV;
        uint64_t* full = is_k ? bars->k_full : bars->v_full;
        uint64_t* free = is_k ? bars->k_free : bars->v_free;
        auto entry = [&](int t) {
            const int j = t * kTile + p * gran;
            return t < tiles && j < keys ? table[j >> bs_log2] : 0;
        };
        int next = entry(0);
        int issued = 0;
        for (int t = 0; t < tiles; ++t) {
            int64_t block = next;
            next = entry(t + 1);
            const int stage = t % NS;
            const int valid = keys - t * kTile < kTile ? keys - t * kTile : kTile;
            const int n = (valid + gran - 1) / gran;
            // waits are made warp-uniform: a vote also brings the lanes back together
            if (t >= NS && !__all_sync(~0u, mbar_wait(smem_u32(free + stage), ((t / NS) - 1) & 1, abort))) break;
            const uint32_t bar = smem_u32(full + stage);
            if (lane == 0) mbar_expect(bar, static_cast<uint32_t>(n * cols * gran * 128));
            __syncwarp();
            if (p < n && c < cols) {
                if (block < 0 || block >= a.num_blocks) {
                    spk_flag(a.status, SPK_STATUS_BAD_BLOCK);
                    block = 0;
                }
                const int j = t * kTile + p * gran;
                const __nv_bfloat16* src = pool + spk_page_base(lay, block, g) + (c << (bs_log2 + 6)) + ((j & (a.block_size - 1)) << 6);
                bulk_load(smem_u32(stages + stage * stage_bytes) + c * kColTile + p * gran * 128, src, gran * 128, bar);
            }
            issued = t + 1;
        }
        if (*abort != 0)  // copies in flight land before the CTA's shared memory is given up
            for (int t = issued > NS ? issued - NS : 0; t < issued; ++t) mbar_wait(smem_u32(full + t % NS), (t / NS) & 1);
    } else if (warp == W + 1) {  // ---- scores
        if (lane == 0) {
            constexpr uint32_t idesc = idesc_bf16(kTile, kTile, false, false);
            bool ok = mbar_wait(smem_u32(&bars->q_full), 0, abort);
            for (int t = 0; ok && t < tiles; ++t) {
                const int stage = t % NS, buf = t % NB;
                // the buffer's previous weights (tile t - NB) have been multiplied
                ok = (t < NB || mbar_wait(smem_u32(&bars->p_free[buf]), ((t / NB) - 1) & 1, abort)) &&
                     mbar_wait(smem_u32(&bars->k_full[stage]), (t / NS) & 1, abort);
                if (!ok) break;
                tc_fence_after();
                const uint32_t qa = smem_u32(q_s), kb = smem_u32(k_s + stage * Sh::kK);
#pragma unroll
                for (int s = 0; s < CK * 4; ++s) {
                    const uint32_t off = (s >> 2) * kColTile + (s & 3) * 32;
                    mma_ss(tmem + kTmemS + buf * 128, desc_sw128(qa + off, 16, 1024), desc_sw128(kb + off, 16, 1024), idesc, s > 0);
                }
                mma_commit(smem_u32(&bars->k_free[stage]));
                mma_commit(smem_u32(&bars->s_full[buf]));
            }
            mma_commit(smem_u32(&bars->s_done));
            mbar_wait(smem_u32(&bars->s_done), 0);  // nothing this thread issued is in the tensor pipe any more
        }
    } else if (warp == W + 2) {  // ---- weighted sums
        if (lane == 0) {
            constexpr uint32_t idesc = idesc_bf16(kTile, CV * 64, false, true);
            for (int t = 0; t < tiles; ++t) {
                const int stage = t % NS, buf = t % NB;
                if (!mbar_wait(smem_u32(&bars->v_full[stage]), (t / NS) & 1, abort) ||
                    !mbar_wait(smem_u32(&bars->p_full[buf]), (t / NB) & 1, abort))
                    break;
                tc_fence_after();
                const uint32_t vb = smem_u32(v_s + stage * Sh::kV);
                const int valid = keys - t * kTile < kTile ? keys - t * kTile : kTile;
                const int steps = (valid + 15) >> 4;
                for (int s = 0; s < steps; ++s) {
                    const uint64_t vd = desc_sw128(vb + s * 2048, kColTile, 1024);
                    // a half's weights lie in its own half of the score buffer
                    mma_ts(tmem + kTmemO, tmem + kTmemS + buf * 128 + (s >> 2) * 64 + (s & 3) * 8, vd, idesc, t > 0 || s > 0);
                    mma_ts(tmem + kTmemO, tmem + kTmemLo + buf * 64 + s * 8, vd, idesc, true);
                }
                mma_commit(smem_u32(&bars->p_free[buf]));
                mma_commit(smem_u32(&bars->v_free[stage]));
            }
            mma_commit(smem_u32(&bars->o_full));
            mbar_wait(smem_u32(&bars->o_full), 0);
        }
    } else {  // ---- scores to weights
        // Q rows into the swizzled operand layout, zeros beyond the portion
        for (int i = threadIdx.x; i < kTile * CK * 8; i += kSigmoidThreads) {
            const int r = i / (CK * 8), c = i % (CK * 8);
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (r < nq)
                v = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.q) + ((t0 + r) * a.heads + h) * a.k_pad + c * 8);
            *reinterpret_cast<uint4*>(q_s + (c >> 3) * kColTile + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = v;
        }
        fence_async_shared();
        mbar_arrive(smem_u32(&bars->q_full));
        const int wg = NB == 2 ? (warp >> 2) & 1 : 0, half = NB == 2 ? warp >> 3 : warp >> 2;  // tile parity, column half
        const int r = (warp & 3) * 32 + lane;
        const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint64_t c1 = f2_pack(-a.scale * kLog2e, -a.scale * kLog2e), c0 = f2_pack(-a.head_bias[h] * kLog2e, -a.head_bias[h] * kLog2e);
        bool ok = true;
        for (int t = wg; t < tiles; t += NB) {
            const int stage = t % NS;
            ok = __all_sync(~0u, mbar_wait(smem_u32(&bars->s_full[wg]), (t / NB) & 1, abort));
            if (!ok) break;
            tc_fence_after();
            const int last = pos0 + r - t * kTile;  // last visible column of this row
            const uint32_t sa = tmem + lanes + kTmemS + wg * 128 + half * 64, la = tmem + lanes + kTmemLo + wg * 64 + half * 32;
            // 32 score columns at a time; the hi parts overlay columns of this half that have been read (16 c + 15 < 32 (c + 1))
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                uint32_t sc[32];
                tmem_ld32(sa + c * 32, sc);
                tmem_wait_ld(sc);
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float p0, p1;
                    sigmoid2(f2_fma(f2_pack(__uint_as_float(sc[2 * i]), __uint_as_float(sc[2 * i + 1])), c1, c0), p0, p1);
                    split_bf16(p0, p1, hi[i], lo[i]);
                }
                const int seen = last - half * 64 - c * 32;
                if (!__all_sync(~0u, seen >= 31)) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint32_t m = (2 * i <= seen ? 0xffffu : 0u) | (2 * i + 1 <= seen ? 0xffff0000u : 0u);
                        hi[i] &= m;
                        lo[i] &= m;
                    }
                }
                tmem_st16(sa + c * 16, hi);
                tmem_st16(la + c * 16, lo);
            }
            tmem_wait_st();
            const int valid = keys - t * kTile;
            if (valid < kTile && (valid & 15) != 0) {  // the last tile: clear the V rows its last MMA step reads beyond the end
                ok = __all_sync(~0u, mbar_wait(smem_u32(&bars->v_full[stage]), (t / NS) & 1, abort));
                if (!ok) break;
                const int end = (valid + 15) & ~15;
                for (int i = half * 128 + r; i < (end - valid) * CV * 8; i += 256) {
                    const int c = i / ((end - valid) * 8), rest = i % ((end - valid) * 8);
                    *reinterpret_cast<uint4*>(v_s + stage * Sh::kV + c * kColTile + (valid + (rest >> 3)) * 128 + ((rest & 7) << 4)) =
                        make_uint4(0u, 0u, 0u, 0u);
                }
                fence_async_shared();
            }
            tc_fence_before();
            mbar_arrive(smem_u32(&bars->p_full[wg]));
        }
        ok = __all_sync(~0u, ok && mbar_wait(smem_u32(&bars->o_full), 0, abort) && *abort == 0);
        tc_fence_after();
        const bool vec = a.vdim % 8 == 0 && a.out_stride % 8 == 0 && reinterpret_cast<uintptr_t>(a.out) % 16 == 0;
        if (const int col = (warp >> 2) * 32; col < CV * 64) {  // a warpgroup writes 32 columns of the output
            uint32_t o[32];
            tmem_ld32(tmem + lanes + kTmemO + col, o);
            tmem_wait_ld(o);
            __nv_bfloat16* dst = out + r * a.out_stride + col;
            if (r < nq && vec) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (col + 8 * i >= a.vdim) break;
                    uint4 v;
                    uint32_t* w = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        w[k] = ok ? pack_bf16(__uint_as_float(o[8 * i + 2 * k]) * a.out_scale, __uint_as_float(o[8 * i + 2 * k + 1]) * a.out_scale) : 0u;
                    *reinterpret_cast<uint4*>(dst + 8 * i) = v;
                }
            } else if (r < nq) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (col + i < a.vdim) dst[i] = __float2bfloat16_rn(ok ? __uint_as_float(o[i]) * a.out_scale : 0.0f);
            }
            __syncwarp();
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0 && *abort != 0) spk_flag(a.status, SPK_STATUS_DEVICE_WAIT_EXPIRED);
    if (warp == 0) tmem_dealloc(tmem, Sh::kColumns);
}

template <int CK, int CV, int NB>
int launch(const spk_sigmoid_attn_args& a, cudaStream_t s) {
    constexpr int bytes = Shape<CK, CV, NB>::kBytes;
    static_assert(sizeof(Bars) <= 256 && (3 - NB) * bytes <= 227 * 1024, "shared memory");
    const cudaError_t e = cudaFuncSetAttribute(sigmoid_prefill_kernel<CK, CV, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return spk_set_cuda_error(e);
    sigmoid_prefill_kernel<CK, CV, NB><<<dim3(a.heads, a.n_tiles), Shape<CK, CV, NB>::kThreads, bytes, s>>>(a);
    SPK_CHECK_LAUNCH();
    return SPK_OK;
}

}  // namespace

// Both forms take about 1.4 us of an SM per tile; the paired one saves most of a CTA's start and end (about 5 us), and loses where an SM has one CTA
// alone or the longest CTA sets the time.  Gain of the paired form, measured over heads of 64 (4, 14 and 28 of them, one prompt of 256 to 8192
// tokens, equal and ragged batches of 2 to 16, 0 to 4096 keys before them):
//  * at most an SM's worth of CTAs: 0.57 to 1.03;
//  * up to 6 key tiles: 1.04 to 1.7 once an SM's share of all tiles is 0.85 of the longest CTA's, 0.72 to 1.04 below;
//  * equal CTAs of 7 to 20 tiles: 1.03 to 1.16 where they make an even number of rounds over the SMs, 0.88 to 0.99 in three (pairs take two, each as
//    long as two), 1.06 and 1.01 in five of 8 and 12 tiles, 0.98 and 0.96 of 16 and 20;
//  * CTAs of a mean length between two thirds and nine tenths of the longest, as behind long contexts: 0.85 to 1.03;
//  * prompts of their own (mean about half of the longest): up to 12 tiles 1.06 to 1.4 from 297 CTAs and a share of 1 on, 0.85 to 0.92 below;
//    up to 48 tiles 1.02 to 1.18 from a share of 1.4 on, 0.8 to 0.98 below; beyond, 0.95 to 1.04.
extern "C" int spk_sigmoid_attn_paired(int k_pad, int v_pad, int heads, int64_t n_tiles, int64_t key_tiles, int64_t most) {
    if (k_pad != 64 || v_pad != 64 || heads < 1 || heads > 65535 || n_tiles < 1 || n_tiles > 65535 || most < 1 || most > (1 << 24) || key_tiles < 1 || key_tiles > n_tiles * most)
        return 0;
    constexpr int64_t sms = 148;
    const int64_t ctas = heads * n_tiles, work = heads * key_tiles;
    if (ctas <= sms) return 0;
    if (most <= 6) return 20 * work >= 17 * sms * most;
    const int64_t rounds = (ctas + sms - 1) / sms;
    if (10 * key_tiles >= 9 * n_tiles * most) return most <= 20 && (rounds % 2 == 0 || (most <= 12 && rounds >= 5));
    if (3 * key_tiles > 2 * n_tiles * most) return 0;
    return most <= 12 ? ctas > 2 * sms && work >= sms * most : most <= 48 && 5 * work >= 7 * sms * most;
}

int spk_sigmoid_prefill_launch(const spk_sigmoid_attn_args& a, cudaStream_t s) {
    if (a.n_tiles > 65535) return SPK_ERR_TOO_LARGE;
    const int ck = a.k_pad / 64, cv = a.v_pad / 64;
    if (ck == 1 && cv == 1) return a.paired ? launch<1, 1, 1>(a, s) : launch<1, 1, 2>(a, s);
    if (ck == 1 && cv == 2) return launch<1, 2, 2>(a, s);
    if (ck == 2 && cv == 1) return launch<2, 1, 2>(a, s);
    return launch<2, 2, 2>(a, s);
}
