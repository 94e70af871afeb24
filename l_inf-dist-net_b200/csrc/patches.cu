// The patches of a convolution-shaped distance layer as rows of a dense layer, and back.
//
//   unfold   rows[(b, l), c * k * k + ki * k + kj] = x[b, c, ho * stride - pad + ki * dil, wo * stride - pad + kj * dil]   (0 outside)
//   fold     gx[b, c, h, w] = sum of the rows' entries that came from (h, w), over ho, then wo, ascending
//
// Bound: L2 / HBM (unfold writes k * k times the input once).  torch's unfold runs one launch per image and leaves [B, C k k, L], which
// a permuting copy then turned into rows; its adjoint took the reverse way.  B = 64, 64 channels of 16 x 16, k = 3 (38 MB of rows):
// 378 + 27 us before, 18 us here; back 27 + 123 us before, 30 us here.
#include "common.cuh"

namespace linf {
namespace {

struct Patch { int B, C, H, W, k, dil, pad, stride, Ho, Wo; };

constexpr int kRows = 16;       // patches per CTA

// A thread keeps its columns (c, ki, kj) for all patches of the CTA: the divisions are paid once, stores are coalesced.
__global__ void __launch_bounds__(256)
unfold_rows_kernel(const float* __restrict__ x, Patch q, float* __restrict__ rows) {
    const int kk = q.k * q.k, cols = q.C * kk, L = q.Ho * q.Wo;
    const long long first = (long long)blockIdx.x * kRows, total = (long long)q.B * L;
    __shared__ int s_h[kRows], s_w[kRows];
    __shared__ size_t s_base[kRows];
    if (threadIdx.x < kRows && first + threadIdx.x < total) {
        const long long p = first + threadIdx.x;
        const int b = (int)(p / L), l = (int)(p - (long long)b * L), ho = l / q.Wo, wo = l - ho * q.Wo;
        s_h[threadIdx.x] = ho * q.stride - q.pad;
        s_w[threadIdx.x] = wo * q.stride - q.pad;
        s_base[threadIdx.x] = (size_t)b * q.C * q.H * q.W;
    }
    __syncthreads();
    const int n = (int)min((long long)kRows, total - first);
    for (int e = threadIdx.x; e < cols; e += 256) {
        const int c = e / kk, t = e - c * kk, ki = t / q.k, kj = t - ki * q.k;
        const float* xc = x + (size_t)c * q.H * q.W;
#pragma unroll 8
        for (int r = 0; r < n; ++r) {
            const int h = s_h[r] + ki * q.dil, w = s_w[r] + kj * q.dil;
            const bool in = (unsigned)h < (unsigned)q.H && (unsigned)w < (unsigned)q.W;
            rows[(size_t)(first + r) * cols + e] = in ? __ldg(xc + s_base[r] + (size_t)h * q.W + w) : 0.f;
        }
    }
}

// One CTA per (b, h): channels run fastest, so that the k * k entries of a patch and channel are read by neighbouring loads of the same
// CTA and come from L1 but for the first time.
__global__ void __launch_bounds__(256)
fold_rows_kernel(const float* __restrict__ rows, Patch q, float* __restrict__ gx) {
    const int kk = q.k * q.k, cols = q.C * kk, L = q.Ho * q.Wo;
    const int b = blockIdx.x / q.H, h = blockIdx.x - b * q.H;
    const float* rb = rows + (size_t)b * L * cols;
    const int reach = (q.k - 1) * q.dil;
    const int hp = h + q.pad, h0 = hp <= reach ? 0 : (hp - reach + q.stride - 1) / q.stride, h1 = min(hp / q.stride, q.Ho - 1);
    for (int e = threadIdx.x; e < q.W * q.C; e += 256) {
        const int w = e / q.C, c = e - w * q.C;
        const int wp = w + q.pad, w0 = wp <= reach ? 0 : (wp - reach + q.stride - 1) / q.stride, w1 = min(wp / q.stride, q.Wo - 1);
        float s = 0.f;
        for (int ho = h0; ho <= h1; ++ho) {
            const int dh = hp - ho * q.stride, ki = dh / q.dil;
            if (ki * q.dil != dh) continue;
            for (int wo = w0; wo <= w1; ++wo) {
                const int dw = wp - wo * q.stride, kj = dw / q.dil;
                if (kj * q.dil != dw) continue;
                s += __ldg(rb + (size_t)(ho * q.Wo + wo) * cols + c * kk + ki * q.k + kj);
            }
        }
        gx[(((size_t)b * q.C + c) * q.H + h) * q.W + w] = s;
    }
}

int make_patch(int B, int C, int H, int W, int k, int dil, int pad, int stride, Patch* q) {
    if (B <= 0 || C <= 0 || H <= 0 || W <= 0 || k <= 0 || dil <= 0 || pad < 0 || stride <= 0) return LINF_ERR_DIMS;
    const long long hs = (long long)H + 2LL * pad - (long long)dil * (k - 1) - 1, ws = (long long)W + 2LL * pad - (long long)dil * (k - 1) - 1;
    if (hs < 0 || ws < 0) return LINF_ERR_DIMS;
    const long long Ho = hs / stride + 1, Wo = ws / stride + 1, lim = 0x7fffffffLL;
    if ((long long)C * k * k > lim || Ho * Wo > lim || (long long)B * Ho * Wo > lim || (double)B * Ho * Wo * C * k * k > (double)lim ||
        (double)B * C * H * W > (double)lim)
        return LINF_ERR_DIMS;
    *q = Patch{B, C, H, W, k, dil, pad, stride, (int)Ho, (int)Wo};
    return LINF_OK;
}

}  // namespace

int unfold_rows(const float* x, int B, int C, int H, int W, int k, int dil, int pad, int stride, float* rows, cudaStream_t st) {
    Patch q;
    const int rc = make_patch(B, C, H, W, k, dil, pad, stride, &q);
    if (rc) return rc;
    const long long n = (long long)B * q.Ho * q.Wo;
    unfold_rows_kernel<<<(unsigned)((n + kRows - 1) / kRows), 256, 0, st>>>(x, q, rows);
    return launch_status();
}

int fold_rows(const float* rows, int B, int C, int H, int W, int k, int dil, int pad, int stride, float* gx, cudaStream_t st) {
    Patch q;
    const int rc = make_patch(B, C, H, W, k, dil, pad, stride, &q);
    if (rc) return rc;
    if ((long long)B * H > 0x7fffffffLL) return LINF_ERR_DIMS;
    fold_rows_kernel<<<(unsigned)(B * H), 256, 0, st>>>(rows, q, gx);
    return launch_status();
}

}  // namespace linf
