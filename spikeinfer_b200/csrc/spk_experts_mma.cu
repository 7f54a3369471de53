// The experts' products on the fifth-generation tensor cores (tcgen05), bf16 operands, 32-bit sums.
//
// CTA = (256 weight rows, run of TN tokens of one expert).  The weights are the M operand (two 128-row tiles, an accumulator each), the
// tokens the N operand: a few decoded tokens cost a narrow MMA instead of a padded tile, and every lane of the accumulators is in use.
// Weights and tokens are stored as the swizzled operand tiles they become, so a stage is two plain bulk copies (cp.async.bulk),
// no tensor map and no gather: the launch that normalises the residual has already put every token's row where its experts read it.
//  * gated: the two tiles are gate and up rows of the same 128 features; the epilogue multiplies silu(gate) by up and writes the operand
//    tiles of the next product.
//  * plain: 256 consecutive output features, 32-bit rows.
//
// Few tokens: the time is that of streaming the weights, beside other launches by experts_stream_kernel.  The plain product's are on their way before the gated one is done.
// Where few blocks are streamed, a cluster of S CTAs shares a block, each over its own part of k; the partial sums meet in shared memory and are
// added in the order of the CTAs, so results don't depend on timing.
// Warp 0 copies, warp 1 issues MMAs, the others write the results.  A tile of 64 tokens and more has eight of them, each with half of the tokens: a
// CTA's results wait for its last MMA, and with four warps they took about as long as the MMAs (7500 tokens, 16 experts of 896 x 1216, two
// per token: 91.8 -> 78.9 us gated, 45.7 -> 41.9 plain; 1200 tokens 36.1 -> 33.3, 22.8 -> 21.4).
#include "spk_experts.cuh"
#include "spk_tensor.cuh"

namespace {

using namespace spk_tc;

constexpr int kTileW = 128 * 128;  // bytes of a 128-row, 64-column weight tile

template <int TN>
struct Shape {
    static constexpr int kStage = 2 * kTileW + TN * 128;
    static constexpr int NS = TN >= 256 ? 3 : TN >= 128 ? 4 : TN >= 64 ? 5 : 3;  // the narrow form leaves room for a second CTA
    static constexpr int kBytes = NS * kStage + 1024 + 256;
    static constexpr int kColumns = 2 * TN < 32 ? 32 : 2 * TN;
    static constexpr int kWriters = TN >= 64 ? 8 : 4;  // warps that write results
    static constexpr int kThreads = 64 + 32 * kWriters;
};

struct Bars {
    uint64_t full[8], free[8], done;
    int abort;
    uint32_t tmem;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// What CTA `rank` of the cluster has where this CTA has `addr`.
__device__ __forceinline__ float cluster_load(uint32_t addr, uint32_t rank) {
    float v;
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.f32 %0, [r];\n\t}\n" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
    return v;
}

// Gated results of a warp's 32 features (this lane's is f) for J tokens from `slot` on, of which n exist.  Pairs of lanes trade a token's
// value, so that a store carries two features.
template <int J>
__device__ __forceinline__ void store_gated(const spk_experts_args& a, int64_t slot, int n, int f, int lane, const float (&p)[J], const float (&q)[J]) {
    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out);
    const bool odd = lane & 1;
    const int fe = f & ~1;
    const bool in = fe < spk_operand_columns(a.out_features);
#pragma unroll
    for (int j = 0; j < J; j += 2) {
        const float y0 = p[j] * rcp(1.0f + ex2(-1.4426950408889634f * p[j])) * q[j];
        const float y1 = p[j + 1] * rcp(1.0f + ex2(-1.4426950408889634f * p[j + 1])) * q[j + 1];
        const float got = __shfl_xor_sync(~0u, odd ? y0 : y1, 1);
        const uint32_t v = odd ? pack_bf16(got, y1) : pack_bf16(y0, got);
        const int jj = j + (odd ? 1 : 0);
        if (in && jj < n) *reinterpret_cast<uint32_t*>(out + spk_operand_at(a.rows, slot + jj, fe)) = v;
    }
}

template <int J>
__device__ __forceinline__ void store_plain(const spk_experts_args& a, int64_t slot, int n, int f, const float (&p)[J], const float (&q)[J]) {
    float* out = static_cast<float*>(a.out) + slot * a.out_features + f;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        if (j < n) {
            if (f < a.out_features) out[static_cast<int64_t>(j) * a.out_features] = p[j];
            if (f + 128 < a.out_features) out[static_cast<int64_t>(j) * a.out_features + 128] = q[j];
        }
    }
}

// S > 1: the CTAs of a cluster are the parts of k of one block.
template <int TN, bool GATED, int S>
__global__ void __launch_bounds__(Shape<TN>::kThreads, TN <= 32 ? 2 : 1)
experts_kernel(const spk_experts_args a, const int blocks, const int ktiles) {
    using Sh = Shape<TN>;
    constexpr int NS = Sh::NS;
    static_assert(S == 1 || (TN == 32 && 2 * TN * 128 * 4 <= NS * Sh::kStage), "partial sums take the stages' place");
    int e, rows;
    int64_t row0;
    // uniform over the cluster: nothing has been set up yet
    if (!spk_find_tile<TN>(a.segs, a.experts, blockIdx.y, e, row0, rows)) {
        spk_grid_wait();
        return;
    }
    if (row0 + TN > a.rows) {
        if (threadIdx.x == 0) spk_flag(a.status, SPK_STATUS_BAD_SLOT);
        spk_grid_wait();
        return;
    }
    const int part = S > 1 ? static_cast<int>(blockIdx.x) % S : 0;
    const int kb = ktiles * part / S, kn = ktiles * (part + 1) / S - kb;  // this CTA's k tiles, at least one
    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    Bars* bars = reinterpret_cast<Bars*>(base + NS * Sh::kStage);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(smem_u32(&bars->full[i]), 1);
            mbar_init(smem_u32(&bars->free[i]), 1);
        }
        mbar_init(smem_u32(&bars->done), 1);
        bars->abort = 0;
    }
    if (warp == 0) tmem_alloc(smem_u32(&bars->tmem), Sh::kColumns);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem;
    volatile int* abort = &bars->abort;
    spk_grid_release();  // this CTA has its columns of TMEM: one of the next launch cannot take them first
    const int b = blockIdx.x / S;
    if (warp == 0) {
        if (lane == 0) {
            const uint8_t* w = static_cast<const uint8_t*>(a.w) + ((static_cast<int64_t>(e) * blocks + b) * ktiles + kb) * (2 * kTileW);
            const uint8_t* x = static_cast<const uint8_t*>(a.x) + row0 * 128 + static_cast<int64_t>(kb) * a.rows * 128;
            auto weights = [&](int k) {
                const int s = k % NS;
                const uint32_t bar = smem_u32(&bars->full[s]);
                mbar_expect(bar, Sh::kStage);
                bulk_load(smem_u32(base + s * Sh::kStage), w + static_cast<int64_t>(k) * (2 * kTileW), 2 * kTileW, bar);
            };
            // launched to overlap: the weights of the first stages don't wait for the launch that writes x.  Else a stage's weights and tokens go
            // together: the first MMA would wait for all stages' weights ahead of the first tokens (both products of 64 experts of 512 x 256, 20 tokens
            // each: 15.4 us, against 16.8; 16 of 896 x 1216: 36.9 against 38.4 with 20 tokens each, 54.4 against 55.8 with 2500 in all).
            const int early = TN > 32 || !a.overlap ? 0 : kn < NS ? kn : NS;
            for (int k = 0; k < early; ++k) weights(k);
            spk_grid_wait();
            int issued = 0;
            for (int k = 0; k < kn; ++k) {
                const int s = k % NS;
                if (k >= NS && !mbar_wait(smem_u32(&bars->free[s]), ((k / NS) - 1) & 1, abort)) break;
                if (k >= early) weights(k);
                bulk_load(smem_u32(base + s * Sh::kStage) + 2 * kTileW, x + static_cast<int64_t>(k) * a.rows * 128, TN * 128, smem_u32(&bars->full[s]));
                issued = k + 1;
            }
            if (*abort != 0)  // copies in flight land before the CTA's shared memory is given up
                for (int k = issued > NS ? issued - NS : 0; k < issued; ++k) mbar_wait(smem_u32(&bars->full[k % NS]), (k / NS) & 1);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = idesc_bf16(128, TN, false, false);
            for (int k = 0; k < kn; ++k) {
                const int s = k % NS;
                if (!mbar_wait(smem_u32(&bars->full[s]), (k / NS) & 1, abort)) break;
                tc_fence_after();
                const uint32_t wa = smem_u32(base + s * Sh::kStage), xa = wa + 2 * kTileW;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t xd = desc_sw128(xa + i * 32, 16, 1024);
                    mma_ss(tmem, desc_sw128(wa + i * 32, 16, 1024), xd, idesc, k > 0 || i > 0);
                    mma_ss(tmem + TN, desc_sw128(wa + kTileW + i * 32, 16, 1024), xd, idesc, k > 0 || i > 0);
                }
                mma_commit(smem_u32(&bars->free[s]));
            }
            mma_commit(smem_u32(&bars->done));
            mbar_wait(smem_u32(&bars->done), 0);  // nothing this thread issued is in the tensor pipe any more
        }
    } else {
        const int quad = warp & 3;
        const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
        const bool ok = __all_sync(~0u, mbar_wait(smem_u32(&bars->done), 0, abort)) && *abort == 0;
        tc_fence_after();
        const int f = b * (GATED ? 128 : 256) + quad * 32 + lane;  // this lane's feature (and f + 128)
#pragma unroll 1
        for (int j0 = (warp - 2) / 4 * 32; j0 < TN && j0 < rows; j0 += 8 * Sh::kWriters) {
            uint32_t p[32], q[32];
            tmem_ld32(tmem + lanes + j0, p);
            tmem_ld32(tmem + lanes + TN + j0, q);
            tmem_wait_ld(p);
            tmem_wait_ld(q);
            float x[32], y[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                x[j] = __uint_as_float(p[j]);
                y[j] = __uint_as_float(q[j]);
            }
            if (S == 1) {
                const int n = ok ? min(32, rows - j0) : 0;
                if (GATED) store_gated<32>(a, row0 + j0, n, f, lane, x, y);
                else store_plain<32>(a, row0 + j0, n, f, x, y);
            } else {  // [gate and up, or the two feature halves][token][128 features]
                float* sums = reinterpret_cast<float*>(base) + quad * 32 + lane;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (j < rows) {
                        sums[j * 128] = ok ? x[j] : 0.0f;
                        sums[(TN + j) * 128] = ok ? y[j] : 0.0f;
                    }
                }
            }
        }
    }
    if (S > 1) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (warp >= 2) {  // every CTA adds and writes its own tokens
            constexpr int J = 32 / S;
            const int quad = warp & 3, j0 = part * J, n = min(J, rows - j0);
            const uint32_t own = smem_u32(base) + 4 * (j0 * 128 + quad * 32 + lane);
            float x[J] = {}, y[J] = {};
            if (n > 0) {
#pragma unroll
                for (int r = 0; r < S; ++r) {
#pragma unroll
                    for (int j = 0; j < J; ++j) {
                        if (j < n) {
                            x[j] += cluster_load(own + j * 512, r);
                            y[j] += cluster_load(own + (TN + j) * 512, r);
                        }
                    }
                }
                const int f = b * (GATED ? 128 : 256) + quad * 32 + lane;
                if (GATED) store_gated<J>(a, row0 + j0, n, f, lane, x, y);
                else store_plain<J>(a, row0 + j0, n, f, x, y);
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();  // no CTA leaves while its sums are being read
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0 && *abort != 0) spk_flag(a.status, SPK_STATUS_DEVICE_WAIT_EXPIRED);
    if (warp == 0) tmem_dealloc(tmem, Sh::kColumns);
}

// Few tokens per expert, beside another stream's launches: the CTAs go over the blocks of all experts, the copies of the next block under way while the last stages of this one are
// multiplied and its results written (two sets of accumulators).  What bounds it is HBM, shared with the mixer's launches beside it, and those
// need whole SMs for their products: so one CTA per SM with six stages, no more of them than kStreamCtas, and the next launch's CTAs are let in
// when the copies are all under way.  16 experts of 896 x 1216, whole decode steps of four, 64 rows: a CTA per block, two per SM (160 blocks) 6285 us;
// 160, 80, 54 CTAs 6640, 6070, 6090; 30 rows 5590 -> 5050, 12 rows 5040 -> 4800, one row 3850 -> 3775 (with the mixer on a stream of higher priority).
struct StreamBars {
    uint64_t full[8], free[8], done[2], drained[2], all;
    int abort;
    uint32_t tmem;
};
constexpr int kStreamTokens = 32;
constexpr int kStreamStages = 6;
constexpr int kStreamStage = 2 * kTileW + kStreamTokens * 128;
constexpr int kStreamBytes = kStreamStages * kStreamStage + 1024 + 256;
constexpr int kStreamThreads = 192;
constexpr int kStreamColumns = 128;
constexpr int kStreamCtas = 96;

template <bool GATED>
__global__ void __launch_bounds__(kStreamThreads, 1)
experts_stream_kernel(const spk_experts_args a, const int blocks, const int ktiles) {
    constexpr int NS = kStreamStages, TN = kStreamTokens;
    extern __shared__ uint8_t raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    StreamBars* bars = reinterpret_cast<StreamBars*>(base + NS * kStreamStage);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    struct Tile {
        int e, rows, b;
        int64_t row0;
    };
    // Block i of this CTA, 1; 0 where there is none, -1 where its rows lie outside the matrix (nothing is done for it).  Called by a whole warp.
    auto find = [&](int i, Tile& t) {
        const int at = static_cast<int>(blockIdx.x) + i * static_cast<int>(gridDim.x);
        t.b = at % blocks;
        if (!spk_find_tile<TN>(a.segs, a.experts, at / blocks, t.e, t.row0, t.rows)) return 0;
        return t.row0 + TN > a.rows ? -1 : 1;
    };
    Tile t;
    int there = find(0, t);
    if (there == 0) {  // uniform over the CTA: nothing has been set up yet
        spk_grid_wait();
        return;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(smem_u32(&bars->full[i]), 1);
            mbar_init(smem_u32(&bars->free[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&bars->done[i]), 1);
            mbar_init(smem_u32(&bars->drained[i]), 128);
        }
        mbar_init(smem_u32(&bars->all), 1);
        bars->abort = 0;
    }
    if (warp == 0) tmem_alloc(smem_u32(&bars->tmem), kStreamColumns);
    fence_async_shared();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem;
    volatile int* abort = &bars->abort;
    if (warp == 0) {
        int copied = 0, issued = 0;  // stages since the first block, the same count in warp 1; those whose copies are under way
        bool go = true;
        for (int i = 0; there != 0 && go; ++i) {
            if (there > 0 && lane == 0) {
                const uint8_t* w = static_cast<const uint8_t*>(a.w) + (static_cast<int64_t>(t.e) * blocks + t.b) * ktiles * (2 * kTileW);
                const uint8_t* x = static_cast<const uint8_t*>(a.x) + t.row0 * 128;
                auto weights = [&](int k, int c) {
                    const uint32_t bar = smem_u32(&bars->full[c % NS]);
                    mbar_expect(bar, kStreamStage);
                    bulk_load(smem_u32(base + (c % NS) * kStreamStage), w + static_cast<int64_t>(k) * (2 * kTileW), 2 * kTileW, bar);
                };
                // launched to overlap: the weights of the first stages don't wait for the launch that writes x
                const int early = copied > 0 || !a.overlap ? 0 : ktiles < NS ? ktiles : NS;
                for (int k = 0; k < early; ++k) weights(k, k);
                if (copied == 0) spk_grid_wait();
                for (int k = 0; k < ktiles; ++k) {
                    const int c = copied + k;
                    if (c >= NS && !mbar_wait(smem_u32(&bars->free[c % NS]), ((c / NS) - 1) & 1, abort)) {
                        go = false;
                        break;
                    }
                    if (k >= early) weights(k, c);
                    bulk_load(smem_u32(base + (c % NS) * kStreamStage) + 2 * kTileW, x + static_cast<int64_t>(k) * a.rows * 128, TN * 128,
                              smem_u32(&bars->full[c % NS]));
                    issued = c + 1;
                }
            }
            go = __shfl_sync(~0u, go, 0);
            if (there > 0) copied += ktiles;
            there = find(i + 1, t);
        }
        spk_grid_release();  // the next launch's CTAs may take SMs from here on: this one's copies are all under way
        if (lane == 0) {
            spk_grid_wait();  // also where no block's rows were good
            if (*abort != 0)  // copies in flight land before the CTA's shared memory is given up
                for (int c = issued > NS ? issued - NS : 0; c < issued; ++c) mbar_wait(smem_u32(&bars->full[c % NS]), (c / NS) & 1);
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = idesc_bf16(128, TN, false, false);
        int used = 0, n = 0;
        bool go = true;
        for (int i = 0; there != 0 && go; ++i) {
            if (there > 0) {
                if (lane == 0) {
                    const uint32_t acc = tmem + (n & 1) * 2 * TN;
                    go = n < 2 || mbar_wait(smem_u32(&bars->drained[n & 1]), ((n / 2) - 1) & 1, abort);
                    tc_fence_after();
                    for (int k = 0; k < ktiles && go; ++k) {
                        const int c = used + k;
                        go = mbar_wait(smem_u32(&bars->full[c % NS]), (c / NS) & 1, abort);
                        if (!go) break;
                        tc_fence_after();
                        const uint32_t wa = smem_u32(base + (c % NS) * kStreamStage), xa = wa + 2 * kTileW;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint64_t xd = desc_sw128(xa + j * 32, 16, 1024);
                            mma_ss(acc, desc_sw128(wa + j * 32, 16, 1024), xd, idesc, k > 0 || j > 0);
                            mma_ss(acc + TN, desc_sw128(wa + kTileW + j * 32, 16, 1024), xd, idesc, k > 0 || j > 0);
                        }
                        mma_commit(smem_u32(&bars->free[c % NS]));
                    }
                    mma_commit(smem_u32(&bars->done[n & 1]));
                }
                go = __shfl_sync(~0u, go, 0);
                used += ktiles;
                ++n;
            }
            there = find(i + 1, t);
        }
        if (lane == 0) {
            mma_commit(smem_u32(&bars->all));
            mbar_wait(smem_u32(&bars->all), 0);  // nothing this thread issued is in the tensor pipe any more
        }
    } else {
        const int quad = warp & 3;
        const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
        int n = 0;
        bool ok = true;
        for (int i = 0; there != 0 && ok; ++i) {
            if (there > 0) {
                ok = __all_sync(~0u, mbar_wait(smem_u32(&bars->done[n & 1]), (n / 2) & 1, abort)) && *abort == 0;
                ok = __all_sync(~0u, ok);
                tc_fence_after();
                uint32_t p[32], q[32];
                const uint32_t acc = tmem + lanes + (n & 1) * 2 * TN;
                tmem_ld32(acc, p);
                tmem_ld32(acc + TN, q);
                tmem_wait_ld(p);
                tmem_wait_ld(q);
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->drained[n & 1]));
                float x[32], y[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    x[j] = __uint_as_float(p[j]);
                    y[j] = __uint_as_float(q[j]);
                }
                const int f = t.b * (GATED ? 128 : 256) + quad * 32 + lane;  // this lane's feature (and f + 128)
                const int live = ok ? t.rows : 0;
                if (GATED) store_gated<32>(a, t.row0, live, f, lane, x, y);
                else store_plain<32>(a, t.row0, live, f, x, y);
                ++n;
            } else if (threadIdx.x == 64) {
                spk_flag(a.status, SPK_STATUS_BAD_SLOT);
            }
            there = find(i + 1, t);
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0 && *abort != 0) spk_flag(a.status, SPK_STATUS_DEVICE_WAIT_EXPIRED);
    if (warp == 0) tmem_dealloc(tmem, kStreamColumns);
}

template <bool GATED>
int launch_stream(const spk_experts_args& a, int blocks, int ktiles, cudaStream_t s) {
    static_assert(sizeof(StreamBars) <= 256 && kStreamBytes <= 227 * 1024, "shared memory");
    const int64_t most = spk_most_tiles(a.pairs, a.experts, kStreamTokens) * blocks;
    if (most > 0x3fffffff) return SPK_ERR_TOO_LARGE;
    // as many CTAs as leave each the same number of blocks if every expert in use has one run of tokens, at most kStreamCtas
    const int64_t expected = static_cast<int64_t>(blocks) * (a.pairs < a.experts ? a.pairs : a.experts);
    const int64_t rounds = (expected + kStreamCtas - 1) / kStreamCtas;
    const int64_t ctas = (expected + rounds - 1) / rounds;
    const cudaError_t e = cudaFuncSetAttribute(experts_stream_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamBytes);
    if (e != cudaSuccess) return spk_set_cuda_error(e);
    return spk_launch(experts_stream_kernel<GATED>, dim3(static_cast<unsigned>(ctas)), kStreamThreads, kStreamBytes, s, a.overlap != 0, a, blocks, ktiles);
}

template <int TN, bool GATED, int S>
int launch(const spk_experts_args& a, int blocks, int ktiles, cudaStream_t s) {
    constexpr int bytes = Shape<TN>::kBytes;
    static_assert(sizeof(Bars) <= 256 && bytes <= 227 * 1024, "shared memory");
    const int64_t tiles = spk_most_tiles(a.pairs, a.experts, TN);
    if (tiles > 65535) return SPK_ERR_TOO_LARGE;
    auto kernel = experts_kernel<TN, GATED, S>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return spk_set_cuda_error(e);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2] = {};
    cfg.gridDim = dim3(blocks * S, static_cast<unsigned>(tiles));
    cfg.blockDim = dim3(Shape<TN>::kThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cfg.attrs = attr;
    if (S > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim = {S, 1, 1};
        ++cfg.numAttrs;
    }
    if (TN == 32 && a.overlap) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        ++cfg.numAttrs;
    }
    e = cudaLaunchKernelEx(&cfg, kernel, a, blocks, ktiles);
    if (e != cudaSuccess) return spk_set_cuda_error(e);
    spk_count_launch();
    return SPK_OK;
}

template <bool GATED>
int dispatch(const spk_experts_args& a, cudaStream_t s) {
    const int per = GATED ? 128 : 256;
    const int blocks = (a.out_features + per - 1) / per, ktiles = (a.k + 63) / 64;
    const int64_t mean = (a.pairs + a.experts - 1) / a.experts;
    if (mean > 96) return launch<256, GATED, 1>(a, blocks, ktiles, s);
    if (mean > 40) return launch<128, GATED, 1>(a, blocks, ktiles, s);
    if (mean > 16) return launch<64, GATED, 1>(a, blocks, ktiles, s);
    // Up to 40 blocks (16 experts of 896 x 1216, two per token: the gated product of one or two users, the second one of up to five) four CTAs share
    // each: a CTA streams 30 to 60 GB/s whatever its ring holds.  Whole steps, the blocks of both whole / two parts / four / eight and four: one user
    // 3310 us (the second product in two parts already), 3195, 3078, 3090; two users 3510, 3370, 3255, 3415; four (the second product alone) 3830, 3675,
    // 3680, 3690.  With library products in the mixer, which want whole SMs, four parts were slower than two (4260 against 4103 us).
    if (blocks * (a.pairs < a.experts ? a.pairs : a.experts) <= 40 && ktiles >= 4) return launch<32, GATED, 4>(a, blocks, ktiles, s);
    // Alone a CTA per block, two to an SM, takes more of HBM's rate than the streaming form, whose fewer CTAs leave SMs to what runs beside it.  Both products of 8 and 64 tokens, us, a CTA
    // per block / streaming: 16 experts of 896 x 1216 21.1 / 29.0, 27.9 / 32.4; 64 of 1024 x 640, four per token 21.3 / 37.6, 49.2 / 66.3; 8 of 2048 x 2048 41.3 / 53.0, 44.1 / 53.8.
    // Whole Gotunex steps of four, the same two: 0.5b (16 of 896 x 1216) four rows 4293 / 3860, 8 rows 4277 / 4500, 16 4646 / 4789, 30 4988 / 4962, 48 5470 / 5221.  Weights of more
    // than 256 MB outlast the mixer beside them (16 of 3584 x 4736, 64 rows: 243 / 291 alone).
    const int64_t expected = static_cast<int64_t>(blocks) * (a.pairs < a.experts ? a.pairs : a.experts);
    if (!a.beside || expected * ktiles * (2 * kTileW) > (256ll << 20)) return launch<32, GATED, 1>(a, blocks, ktiles, s);
    return launch_stream<GATED>(a, blocks, ktiles, s);
}

}  // namespace

int spk_experts_mma(const spk_experts_args& a, cudaStream_t s) {
    if (a.rows % kExpertAlign != 0 || reinterpret_cast<uintptr_t>(a.x) % 16 != 0 || reinterpret_cast<uintptr_t>(a.w) % 16 != 0 ||
        reinterpret_cast<uintptr_t>(a.out) % 16 != 0)
        return SPK_ERR_BAD_STRIDE;
    return a.gated ? dispatch<true>(a, s) : dispatch<false>(a, s);
}
