// Products of a few rows (decode steps of a user or two) with a weight matrix: out[r, f] = sum_k x[r, k] w[f, k], bf16 operands, 32-bit sums.
//
// A warp owns one or two features: their weights are asked for first, 16 bytes per lane and eight lines at a time, and where the launch overlaps the
// one ahead of it before that has written x; the rows come through shared memory as 32-bit numbers, so that a weight costs one multiply-add a
// row.  What bounds it is the chain launch, weights from HBM, sum over the lanes; a tensor-core tile of eight rows would be seven
// eighths of padding for one.  Gotunex steps of one row, us a launch, library / here: 896 x 2832 4.8 / 2.9, 896 x 1568 4.1 / 2.5, 384 x 1344 3.1 / 2.9 and
// 896 x 896 4.6 / 2.0 behind the launch ahead; whole steps of one, two, four and eight rows 3555 -> 3250, 3575 -> 3420, 3820 -> 3835, 4340 -> 4665: from
// three rows on the library's.
#include "spk_dense.cuh"
#include "spk_tensor.cuh"

namespace {

using namespace spk_tc;

constexpr int kWarps = 8, kThreads = 32 * kWarps;
constexpr int kPass = 1024;             // columns at a time: four 16-byte pieces per lane
constexpr int kPieces = kPass / 8 / 32;

// Totals over the warp of N values per lane, N a power of two up to 32: lane l ends up with value `index` of them.  Lanes fold half of their values
// away at each of the first levels, so N totals cost N - 1 + 5 - log2(N) exchanges.
template <int N>
__device__ __forceinline__ float totals(float (&v)[N], int lane, int& index) {
    index = 0;
    int o = 16;
#pragma unroll
    for (int half = N / 2; half >= 1; half >>= 1, o >>= 1) {
        const bool upper = lane & o;
        index += upper ? half : 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float send = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(~0u, send, o);
        }
    }
    float t = v[0];
    for (; o >= 1; o >>= 1) t += __shfl_xor_sync(~0u, t, o);
    return t;
}

template <int NR, int F, typename TO>
__global__ void __launch_bounds__(kThreads)
rows_linear_kernel(const spk_rows_linear_args a) {
    __shared__ __align__(16) float xs[NR][2][kPass / 8][4];  // row, lower or upper half of a piece, piece
    spk_grid_release();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t f0 = (static_cast<int64_t>(blockIdx.x) * kWarps + warp) * F;
    const int k = static_cast<int>(a.k), n = static_cast<int>(a.n);
    const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(a.w) + f0 * k;
    uint4 wv[F][kPieces];
    auto weights = [&](int k0) {
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int j = 0; j < kPieces; ++j) {
                const int c = k0 + (j * 32 + lane) * 8;
                wv[f][j] = f0 + f < a.features && c < k ? __ldg(reinterpret_cast<const uint4*>(w + static_cast<int64_t>(f) * k + c)) : make_uint4(0u, 0u, 0u, 0u);
            }
    };
    weights(0);
    spk_grid_wait();
    uint64_t acc[F][NR];
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[f][r] = f2_pack(0.0f, 0.0f);
    for (int k0 = 0; k0 < k; k0 += kPass) {
        if (k0 > 0) {
            __syncthreads();  // the pass before has read its rows
            weights(k0);
        }
        const int pieces = (k - k0 < kPass ? k - k0 : kPass) / 8;
        for (int i = threadIdx.x; i < NR * (kPass / 8); i += kThreads) {
            const int r = i / (kPass / 8), c = i % (kPass / 8);
            if (c >= pieces) continue;
            uint4 u = make_uint4(0u, 0u, 0u, 0u);
            if (r < n) asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"  // not the read-only path: it may move ahead of the wait
                                    : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                                    : "l"(static_cast<const __nv_bfloat16*>(a.x) + r * a.ld_x + k0 + c * 8) : "memory");
            *reinterpret_cast<float4*>(xs[r][0][c]) = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
            *reinterpret_cast<float4*>(xs[r][1][c]) = make_float4(__uint_as_float(u.z << 16), __uint_as_float(u.z & 0xffff0000u), __uint_as_float(u.w << 16), __uint_as_float(u.w & 0xffff0000u));
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
            const int c = j * 32 + lane;
            if (c < pieces) {
                uint64_t w2[F][4];
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    const uint32_t u[4] = {wv[f][j].x, wv[f][j].y, wv[f][j].z, wv[f][j].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) w2[f][i] = f2_pack(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xffff0000u));
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(xs[r][0][c]), hi = *reinterpret_cast<const ulonglong2*>(xs[r][1][c]);
#pragma unroll
                    for (int f = 0; f < F; ++f)
                        acc[f][r] = f2_fma(w2[f][3], hi.y, f2_fma(w2[f][2], hi.x, f2_fma(w2[f][1], lo.y, f2_fma(w2[f][0], lo.x, acc[f][r]))));
                }
            }
        }
    }
    float v[F * NR];
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            float x, y;
            f2_unpack(acc[f][r], x, y);
            v[f * NR + r] = x + y;
        }
    int index;
    const float t = totals<F * NR>(v, lane, index);
    const int r = index % NR;
    const int64_t f = f0 + index / NR;
    if (lane % (32 / (F * NR)) == 0 && r < n && f < a.features) static_cast<TO*>(a.out)[r * a.ld_out + f] = spk_from_float<TO>(t);
}

template <int NR, typename TO>
int launch(const spk_rows_linear_args& a, cudaStream_t s) {
    // two features a warp where one would be more CTAs than the chip holds at once
    const bool two = a.features > static_cast<int64_t>(2 * 148) * kWarps;
    const int64_t per = kWarps * (two ? 2 : 1), grid = (a.features + per - 1) / per;
    if (grid > 0x7fffffffLL) return SPK_ERR_TOO_LARGE;
    return spk_launch(two ? rows_linear_kernel<NR, 2, TO> : rows_linear_kernel<NR, 1, TO>, dim3(static_cast<unsigned>(grid)), kThreads, 0, s, a.overlap != 0, a);
}

template <typename TO>
int dispatch(const spk_rows_linear_args& a, cudaStream_t s) {
    return a.n == 1 ? launch<1, TO>(a, s) : launch<2, TO>(a, s);
}

}  // namespace

extern "C" int spk_rows_linear(const spk_rows_linear_args* args, void* stream) {
    SpkRange nvtx_range("spk_rows_linear");
    if (args == nullptr) return SPK_ERR_NULL_POINTER;
    const spk_rows_linear_args& a = *args;
    if (a.n < 0 || a.n > 2 || a.k < 8 || a.k > (1 << 20) || a.k % 8 != 0 || a.features < 0) return SPK_ERR_BAD_SHAPE;
    if (a.out_dtype != SPK_F32 && a.out_dtype != SPK_BF16) return SPK_ERR_BAD_DTYPE;
    if (a.n == 0 || a.features == 0) return SPK_OK;
    if (a.x == nullptr || a.w == nullptr || a.out == nullptr) return SPK_ERR_NULL_POINTER;
    if (reinterpret_cast<uintptr_t>(a.x) % 16 != 0 || reinterpret_cast<uintptr_t>(a.w) % 16 != 0 || a.ld_x % 8 != 0) return SPK_ERR_BAD_STRIDE;
    return a.out_dtype == SPK_F32 ? dispatch<float>(a, spk_stream(stream)) : dispatch<__nv_bfloat16>(a, spk_stream(stream));
}
