// inf-dist forward for a handful of input rows (one image at a time, dense layers): a 64-row output tile would be empty but for
// them, and 16 such tiles leave most of the GPU idle.  One warp per output channel: it reads its weight row once, 16 bytes a
// lane, against up to eight input rows, which the eight warps of the CTA share through L1; the lanes' best terms are merged by a
// butterfly (larger |t| first, then the lower index: the tie rule of the scan).
// Bound: at one row the weights' 4 * Din * Dout bytes, in practice the latency of launch and of two loads; every load of a warp
// is issued before the first is used.
// Measured on one B200, us (launch included), tiled kernels -> here: 1 x 1024 x 1024: 38 -> 11; 1 x 5120 x 5120: 142 -> 21;
// 8 x 5120 x 5120: 146 -> 73; 12 x 3072 x 4096: 125 -> 54; 16 x 1024 x 1024: 36 -> 12; 16 x 5120 x 5120: 154 -> 157, so that more than eight
// rows take this path only up to 16 M weights.
#include "common.cuh"

namespace linf {
namespace {

constexpr unsigned FULL = 0xffffffffu;

template <int RB, bool VEC>
__global__ void __launch_bounds__(256)
inf_forward_few_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, Dims d,
                            float* __restrict__ y, int* __restrict__ pos, Post post) {
    const int lane = threadIdx.x & 31;
    const int c = blockIdx.x * 8 + (threadIdx.x >> 5), r0 = blockIdx.y * RB;
    if (c >= d.CO) return;
    const int g = c / d.COg, K = d.CIg;
    const float* wr = w + (size_t)c * K;
    const float* xr = x + (size_t)r0 * d.CI + (size_t)g * K;
    const int rows = min(RB, d.R - r0);
    float t[RB]; int at[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) { t[r] = 0.f; at[r] = 0; }
    auto take = [&](int r, float v, int k) { if (fabsf(v) > fabsf(t[r])) { t[r] = v; at[r] = k; } };
    if (VEC) {
#pragma unroll (RB == 1 ? 8 : RB == 2 ? 4 : 2)
        for (int k = 4 * lane; k < K; k += 128) {
            const float4 wv = __ldg(reinterpret_cast<const float4*>(wr + k));
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const float4 xv = __ldg(reinterpret_cast<const float4*>(xr + (size_t)min(r, rows - 1) * d.CI + k));
                take(r, xv.x - wv.x, k); take(r, xv.y - wv.y, k + 1); take(r, xv.z - wv.z, k + 2); take(r, xv.w - wv.w, k + 3);
            }
        }
    } else {
#pragma unroll (RB == 1 ? 8 : 4)
        for (int k = lane; k < K; k += 32) {
            const float wv = __ldg(wr + k);
#pragma unroll
            for (int r = 0; r < RB; ++r) take(r, __ldg(xr + (size_t)min(r, rows - 1) * d.CI + k) - wv, k);
        }
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
#pragma unroll
        for (int s = 16; s; s >>= 1) {
            const float ot = __shfl_xor_sync(FULL, t[r], s); const int oa = __shfl_xor_sync(FULL, at[r], s);
            if (fabsf(ot) > fabsf(t[r]) || (fabsf(ot) == fabsf(t[r]) && oa < at[r])) { t[r] = ot; at[r] = oa; }
        }
        if (lane == 0 && r < rows) {
            const size_t e = (size_t)(r0 + r) * d.CO + c;
            y[e] = post_apply(post, fabsf(t[r]), c);
            if (pos) pos[e] = at[r] | (t[r] < 0.f ? (int)0x80000000 : 0);
        }
    }
}

template <int RB>
int launch_few(const float* x, const float* w, const Dims& d, float* y, int* pos, cudaStream_t st, const Post& post) {
    const dim3 grid((d.CO + 7) / 8, (d.R + RB - 1) / RB);
    const bool vec = (d.CIg & 3) == 0 && aligned16(x) && aligned16(w);
    if (vec) inf_forward_few_rows_kernel<RB, true><<<grid, 256, 0, st>>>(x, w, d, y, pos, post);
    else inf_forward_few_rows_kernel<RB, false><<<grid, 256, 0, st>>>(x, w, d, y, pos, post);
    return launch_status();
}

}  // namespace

// tiled: the alternative is the tiled kernel (else the generic one, which is 6 - 40 times slower).  That one is faster for rows so long that the warps of a CTA,
// each at its own place, do not find them in L1 any more, unless there are few weights (then it has few CTAs).  us, tiled / here, rows x Din x Dout:
// 8 x 16384 x 2048 199 / 183, 8 x 24576 x 1024 189 / 287, 8 x 24576 x 512 > 170 / 145, 5 x 24576 x 1024 186 / 165, 3 x 49152 x 512 249 / 200, 4 x 49152 x 512 248 / 280, 8 x 49152 x 128
// 452 / 247, 4 x 65536 x 512 285 / 375; 2 x 98304 x 512 391 / 327, 2 x 150528 x 256 450 / 508; 8 x 150528 x 64 848 / 747, 8 x 196608 x 64 866 / 972; 1 x 196608 x 512 590 / 513.
bool inf_few_rows_ok(const Dims& d, bool tiled) {
    const double weights = (double)d.CO * d.CIg;
    if (!(d.HW == 1 && d.COg >= 32 && (d.R <= 8 || (d.R <= 16 && weights <= 16e6)))) return false;
    const int rows = d.R < 8 ? d.R : 8;
    const double staged = (double)rows * d.CIg;
    if (!tiled || rows == 1) return true;
    return staged <= 1.3e6 && !(rows == 2 ? staged > 2.5e5 && weights > 32e6 : staged > 1.6e5 && weights > 16e6);
}

int inf_forward_few_rows(const float* x, const float* w, const Dims& d, float* y, int* pos, cudaStream_t st, const Post& post) {
    if (d.R == 1) return launch_few<1>(x, w, d, y, pos, st, post);
    if (d.R == 2) return launch_few<2>(x, w, d, y, pos, st, post);
    if (d.R <= 4) return launch_few<4>(x, w, d, y, pos, st, post);
    return launch_few<8>(x, w, d, y, pos, st, post);
}

}  // namespace linf
