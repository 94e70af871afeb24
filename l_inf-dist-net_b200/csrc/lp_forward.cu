// Forward of the finite-p distance neuron on dense layers (HW == 1, at least 32 outputs and 32 inputs per group; no
// alignment or divisibility is asked for):   y[b,o] = M * (sum_i (|x[b,i] - w[o,i]| / M)^p)^(1/p),  M = max_i |x - w|, which `y` holds on entry.
//
// Bound: FP32 issue for integer p (p = 8: subtraction, scale, two squarings, one multiply-add = 5 lane operations a term), the special-function
// unit (one log2 and one exp2 per term: 16 cycles per term and scheduler) otherwise.
// 64 x 64 (or 64 x 48) output tile per CTA of 128 threads, 8 x 4 (8 x 3) outputs per thread, operand tiles through a ring of
// three cp.async stages; two neighbouring terms of an output sit in one register pair, so subtraction,
// scale and squarings are packed (f32x2).  The sums run over i in ascending order, whatever the tile: the same bits for every width.
//
// Without the scale (p = 8, 16: sums checked against the range of a float afterwards) and the maximum pass this takes 1.87 ms instead of
// 2.72 ms at B = 512, Din = Dout = 5120, p = 8, and the result is as exact.  It is not used: a training run at finite p amplifies the last
// bit of a distance within two steps (hinge loss, Adam with eps = 1e-10), and the nets, whose layers are all aligned, give the same bits from version to version.
// Measured on one B200, us, with the maximum pass (dense value-only kernel before, lists of large entries now), scale and squarings packed:
// B = 512, Din = Dout = 5120: p = 8 3066 -> 2719, 16 3460 -> 3077, 64 4222 -> 3831, 23.7 7118 -> 6726; ragged layers (the generic kernel before): B = 203, Din = 1027,
// Dout = 1333, p = 8 677 -> 221, 23.7 897 -> 377; B = 500, Din = 2050, Dout = 3001, p = 8: 6260 -> 938, 23.7 8050 -> 2030.
#include <math.h>

#include "common.cuh"

namespace linf {
namespace {

typedef unsigned long long u64;

__device__ __forceinline__ u64 mul2(u64 a, u64 b) { u64 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ u64 pack2(float a, float b) { u64 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float lg2_approx(float a) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a)); return r; }
__device__ __forceinline__ float ex2_approx(float a) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a)); return r; }

// a^E of a pair, E a power of two
template <int E>
__device__ __forceinline__ u64 pow2_ct(u64 a) {
    if constexpr (E == 1) return a;
    else { const u64 h = pow2_ct<E / 2>(a); return mul2(h, h); }
}
constexpr int TM = 64, NT = 128, BK = 16, LDK = BK + 4, STAGES = 3;

struct FwdParams {
    const float* x; const float* w; float* y;
    int B, COg, CIg, G, CI, CO;
    float p, inv_p;
};

template <int ROWS, bool AL>
__device__ __forceinline__ void load_rows(float* dst, const float* __restrict__ src, size_t ld, int row0, int rows, int k0, int cols, int tid) {
    if (AL) {
#pragma unroll
        for (int q = tid; q < ROWS * (BK / 4); q += NT) {
            const int r = q / (BK / 4), c = (q % (BK / 4)) * 4;
            const bool in = row0 + r < rows && k0 + c < cols;
            cp_async16(dst + r * LDK + c, src + (in ? (size_t)(row0 + r) * ld + k0 + c : 0), in ? 16 : 0);
        }
    } else {
#pragma unroll 2                      // unrolled fully, the copies' addresses alone exhaust the registers
        for (int q = tid; q < ROWS * BK; q += NT) {
            const int r = q / BK, c = q % BK;
            const bool in = row0 + r < rows && k0 + c < cols;
            cp_async4(dst + r * LDK + c, src + (in ? (size_t)(row0 + r) * ld + k0 + c : 0), in ? 4 : 0);
        }
    }
}

// One output by the rule of the generic kernel: a term counts min(|t| / M, 1)^p with min(NaN, 1) = 1, where M is the largest |t| that is a number.
__device__ __noinline__ float clamped_output(const float* xr, const float* wr, int K, float M, float p, float inv_p) {
    const float rM = M > 0.f ? 1.f / M : 0.f;
    float S = 0.f;
#pragma unroll 8
    for (int k = 0; k < K; ++k) S += ex2_approx(p * lg2_approx(fminf(fabsf(__ldg(xr + k) - __ldg(wr + k)) * rM, 1.f)));
    return M > 0.f ? powf(S, inv_p) * M : 0.f;
}

// IP: 8, 16, 64 at compile time, 0: p at run time.  TJ: output columns per thread.  AL: rows of x and w can be read 16 bytes at a time.
// CLAMP: calls that the generic kernel served before this one.  An infinite or NaN difference, or an M so small that 1 / M is infinite, leaves a sum
// that is not finite, and nothing else does: such outputs are worked out again by that kernel's rule, one thread each.
template <int IP, int TJ, bool AL, bool CLAMP>
__global__ void __launch_bounds__(NT, 3)
lp_forward_kernel(const FwdParams p) {
    extern __shared__ __align__(16) float smem[];
    constexpr int TN = 16 * TJ, NO = 8 * TJ, STAGE = (TM + TN) * LDK;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp & 1, wn = warp >> 1, lm = lane >> 3, ln = lane & 7;
    const int row_off = wm * 32 + lm, col_off = wn * (8 * TJ) + ln;       // + 4i rows, + 8j columns
    const int tiles_m = (p.B + TM - 1) / TM, tiles_n = (p.COg + TN - 1) / TN;
    const int g = blockIdx.x / (tiles_m * tiles_n), tg = blockIdx.x % (tiles_m * tiles_n);
    const int n0 = (tg / tiles_m) * TN, m0 = (tg % tiles_m) * TM;
    const float* xg = p.x + (size_t)g * p.CIg;
    const float* wg = p.w + (size_t)g * p.COg * p.CIg;
    const int KT = (p.CIg + BK - 1) / BK;

    // runs body(e, t01, t23) over the differences of the first n_tiles k-tiles, four terms of an output at a time
    auto sweep = [&](int n_tiles, auto&& body) {
        auto load = [&](int s, int kt) {
            float* st = smem + s * STAGE;
            load_rows<TM, AL>(st, xg, p.CI, m0, p.B, kt * BK, p.CIg, tid);
            load_rows<TN, AL>(st + TM * LDK, wg, p.CIg, n0, p.COg, kt * BK, p.CIg, tid);
        };
        __syncthreads();
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) { if (s < n_tiles) load(s, s); cp_async_commit(); }
        int rd = 0, wr = STAGES - 1;
        for (int kt = 0; kt < n_tiles; ++kt) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();
            if (kt + STAGES - 1 < n_tiles) load(wr, kt + STAGES - 1);
            cp_async_commit();
            const float* As = smem + rd * STAGE + row_off * LDK;
            const float* Bs = smem + rd * STAGE + (TM + col_off) * LDK;
            // two of the four k4 steps per trip: the fully unrolled body runs into instruction fetch stalls
#pragma unroll 2
            for (int k4 = 0; k4 < BK / 4; ++k4) {
                ulonglong2 bf[TJ];
#pragma unroll
                for (int j = 0; j < TJ; ++j) bf[j] = *reinterpret_cast<const ulonglong2*>(Bs + (8 * j) * LDK + k4 * 4);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const ulonglong2 af = *reinterpret_cast<const ulonglong2*>(As + (4 * i) * LDK + k4 * 4);
#pragma unroll
                    for (int j = 0; j < TJ; ++j) body(i * TJ + j, sub_f32x2(af.x, bf[j].x), sub_f32x2(af.y, bf[j].y));
                }
            }
            rd = (rd + 1 == STAGES) ? 0 : rd + 1;
            wr = (wr + 1 == STAGES) ? 0 : wr + 1;
        }
        cp_async_wait<0>();
    };
    auto out = [&](int e) { return p.y + (size_t)(m0 + row_off + 4 * (e / TJ)) * p.CO + (size_t)g * p.COg + n0 + col_off + 8 * (e % TJ); };
    auto inside = [&](int e) { return m0 + row_off + 4 * (e / TJ) < p.B && n0 + col_off + 8 * (e % TJ) < p.COg; };

    float S[NO];
    float rM[NO];
#pragma unroll
    for (int e = 0; e < NO; ++e) {
        const float M = inside(e) ? *out(e) : 0.f;
        rM[e] = M > 0.f ? 1.f / M : 0.f;
        S[e] = 0.f;
    }
    sweep(KT, [&](int e, u64 t01, u64 t23) {
        if constexpr (IP > 0) {
            const u64 rr = pack2(rM[e], rM[e]);
            const u64 u01 = mul2(t01, rr), u23 = mul2(t23, rr);
            float a, b;
            unpack_f32x2(pow2_ct<IP / 2>(u01), a, b);
            S[e] = fmaf(a, a, S[e]); S[e] = fmaf(b, b, S[e]);
            unpack_f32x2(pow2_ct<IP / 2>(u23), a, b);
            S[e] = fmaf(a, a, S[e]); S[e] = fmaf(b, b, S[e]);
        } else {
            // (scalar: packed multiplications around the special-function unit only add moves, 388 -> 409 us at B = 200, 1024 x 2048)
            float t[4];
            unpack_f32x2(t01, t[0], t[1]); unpack_f32x2(t23, t[2], t[3]);
#pragma unroll
            for (int q = 0; q < 4; ++q) S[e] += ex2_approx(p.p * lg2_approx(fabsf(t[q]) * rM[e]));
        }
    });
#pragma unroll
    for (int e = 0; e < NO; ++e)
        if (inside(e)) {
            float* yo = out(e);
            const float M = *yo;
            float y = M > 0.f ? powf(S[e], p.inv_p) * M : 0.f;
            if (CLAMP && !(S[e] < __int_as_float(0x7f800000)))
                y = clamped_output(xg + (size_t)(m0 + row_off + 4 * (e / TJ)) * p.CI, wg + (size_t)(n0 + col_off + 8 * (e % TJ)) * p.CIg, p.CIg, M, p.p, p.inv_p);
            *yo = y;
        }
}

template <int IP, int TJ, bool AL, bool CLAMP>
int launch_fwd(const FwdParams& P, int grid, cudaStream_t st) {
    constexpr int bytes = STAGES * (TM + 16 * TJ) * LDK * 4;
    auto kern = lp_forward_kernel<IP, TJ, AL, CLAMP>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return LINF_ERR_LAUNCH;
    kern<<<grid, NT, bytes, st>>>(P);
    return launch_status();
}
template <int IP, int TJ>
int launch_fwd_tj(const FwdParams& P, int grid, bool al, bool clamp, cudaStream_t st) {
    if (!al) return launch_fwd<IP, TJ, false, true>(P, grid, st);
    return clamp ? launch_fwd<IP, TJ, true, true>(P, grid, st) : launch_fwd<IP, TJ, true, false>(P, grid, st);
}
template <int IP>
int launch_fwd_ip(const FwdParams& P, int grid, bool narrow, bool al, bool clamp, cudaStream_t st) {
    return narrow ? launch_fwd_tj<IP, 3>(P, grid, al, clamp, st) : launch_fwd_tj<IP, 4>(P, grid, al, clamp, st);
}

}  // namespace

// Dense layers with at least 32 channels per group on both sides.  `aligned`: channel counts are multiples of four and x, w and y lie on 16-byte
// boundaries (lp_tiled_ok).  Other calls only at 8 <= p <= 100: below and above, the generic kernels, whose whole powers are products and
// not exp2(p * log2), are up to 1.4 times more exact (y at p = 2 and 3; the gradients behind y at p = 300 and 1000), and they have always served
// these calls.
bool lp_forward_dense_ok(const Dims& d, float p, bool aligned) {
    return d.HW == 1 && d.COg >= 32 && d.CIg >= 32 && (aligned || (p >= 8.f && p <= 100.f));
}

int lp_forward_width = 0;   // 0: tile width by shape; 1: 64 columns; 2: 48 columns (benchmarking knob)

int lp_forward_dense(const float* x, const float* w, const Dims& d, float* y, float p, cudaStream_t st) {
    // The kernel is bound by throughput: an SM of the last, partial wave takes a third of a full wave per CTA it
    // holds.  48-wide tiles cost 3/4 of 64-wide ones and are taken when that buys a shorter launch
    // (B = 512, Dout = 5120: 640 tiles on 444 slots = 1 + 2/3 waves, against 856 tiles = 2 x 3/4).
    const int tiles_m = (d.R + TM - 1) / TM, slots = 3 * sm_count(), sms = sm_count();
    auto count = [&](int tn) { return (long long)tiles_m * ((d.COg + tn - 1) / tn) * d.G; };
    auto cost = [&](int tn) {
        const long long tiles = count(tn), rest = tiles % slots;
        return (tn / 64.0) * ((tiles / slots) + ((rest + sms - 1) / sms) / 3.0);
    };
    const bool narrow = lp_forward_width == 2 || (lp_forward_width == 0 && d.COg >= 48 && cost(48) < 0.97 * cost(64));
    const long long grid = count(narrow ? 48 : 64);
    if (grid > 0x7fffffffLL) return LINF_ERR_DIMS;
    FwdParams P;
    P.x = x; P.w = w; P.y = y;
    P.B = d.R; P.COg = d.COg; P.CIg = d.CIg; P.G = d.G; P.CI = d.CI; P.CO = d.CO;
    P.p = p; P.inv_p = 1.f / p;
    const bool al = (d.CIg & 3) == 0 && aligned16(x) && aligned16(w), clamp = !lp_tiled_ok(d, x, w, y, nullptr, nullptr);
    if (p == 8.f) return launch_fwd_ip<8>(P, (int)grid, narrow, al, clamp, st);
    if (p == 16.f) return launch_fwd_ip<16>(P, (int)grid, narrow, al, clamp, st);
    if (p == 64.f) return launch_fwd_ip<64>(P, (int)grid, narrow, al, clamp, st);
    return launch_fwd_ip<0>(P, (int)grid, narrow, al, clamp, st);
}

}  // namespace linf
