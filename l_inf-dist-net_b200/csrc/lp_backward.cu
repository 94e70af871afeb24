// Both gradients of the finite-p distance neuron in one pass over the (b, o, i) terms, for dense layers
// (HW == 1, at least 32 channels per group on either side; no alignment or divisibility is asked for).
//
//   T[b,o,i]  = g[b,o] * s * |s|^(p-2),   s = (x[b,i] - w[o,i]) / y[b,o]
//   gx[b,i]   =  sum_o T        gw[o,i] = -sum_b T
//
// Bound: FP32 issue (p with a fraction: the special-function unit, one log2 / exp2 pair per term).  What a term costs is
// its power, and the two gradients want the same power, so a thread
// that owns (b, i) pairs walks over the outputs o, adds every term to its gx register and to a running sum
// over its own rows for gw.  The rows of a thread are 16 of the batch and its columns two neighbours of the input, lanes
// run along i: nothing is exchanged between lanes, the warps' gw sums meet in shared memory once per
// eight outputs.  All arithmetic is packed two rows at a time (f32x2).
//
// p = 8 and 16 run without the division by y: T = h * t^(p-1) with h = g / y^(p-1) worked out once per (b, o)
// by the preparation kernel, which also looks whether every y lies where t^(p-1) cannot leave the range of
// a float and whether every h is 0 for g = 0 or else a normal number; if not, the kernel takes the scaled form instead (`flag`).  Per term of both gradients:
// 7 lane operations at p = 8 (subtraction, four products, two multiply-adds) against 2 x 7 of two separate passes.
//
// Work split.  A CTA owns 64 input columns, a range of outputs and a range of batch tiles (16 rows per warp).
// It takes its batch tiles one after the other; the gw sums of the first are stored, the later ones added by
// the same thread with `red` (program order, so the result is the same in every run).  Ranges
// of outputs leave partial gx, ranges of batch tiles partial gw in the workspace, added up in ascending
// order by a last kernel.  `plan_both` chooses the number of ranges.
//
// Measured on one B200, both gradients, us, separate kernels -> here:
//   tiled kernels (lp_tiled.cu):  16384 x 576 x 128: p = 8 1920 -> 380, 23.7 9400 -> 818, 64 3047 -> 546;  2048 x 1024 x 1024: 1178 -> 636, 4000 -> 1464, 1948 -> 951
//   generic kernels (lp.cu):      203 x 1027 x 1333: p = 8 1045 -> 126, 23.7 1700 -> 269, 64 1628 -> 185;  500 x 2050 x 3001: 8970 -> 895, 14220 -> 2096, 14440 -> 1390
#include <math.h>

#include "common.cuh"

namespace linf {
namespace {

typedef unsigned long long u64;

__device__ __forceinline__ u64 mul2(u64 a, u64 b) { u64 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) { u64 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ u64 pack2(float a, float b) { u64 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ u64 abs2(u64 a) { return a & 0x7fffffff7fffffffULL; }
__device__ __forceinline__ float lg2_approx(float a) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a)); return r; }
__device__ __forceinline__ float ex2_approx(float a) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a)); return r; }

struct PowQ { int m; float f; };       // p - 2 = m + f

// s <- s * |s|^(p-2) for N pairs.  IP > 0: p is that even integer (the sign comes with the odd power p - 1: 7 and 15 as
// (a^n * a) * a^n, 63 along the chain 2 3 6 12 15 30 60 63).  IP = 0: p - 2 = q.m + q.f at run time, q.m < 1024; the bit tests are
// uniform over the grid and end with the highest set bit, and one test serves all N pairs: a branch per pair kept the pairs' chains from overlapping
// (p = 23.7, 512 x 5120 x 5120, a size that takes this path in measurements only: 10965 -> 8524 us).
template <int IP, int N>
__device__ __forceinline__ void factors(u64 (&s)[N], const PowQ q) {
    if constexpr (IP == 8 || IP == 16) {
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const u64 a = s[e], a3 = mul2(mul2(a, a), a), a7 = mul2(mul2(a3, a), a3);
            if constexpr (IP == 8) s[e] = a7;
            else s[e] = mul2(mul2(a7, a), a7);
        }
    } else if constexpr (IP == 64) {
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const u64 a = s[e], a3 = mul2(mul2(a, a), a), a6 = mul2(a3, a3), a15 = mul2(mul2(a6, a6), a3), a30 = mul2(a15, a15);
            s[e] = mul2(mul2(a30, a30), a3);
        }
    } else {
        constexpr int NB = 10;
        // the fractional part first: the special-function unit works on it while the FP32 pipe squares
        u64 b[N], v[N], r[N];
        if (q.f != 0.f) {
            const u64 ff = pack2(q.f, q.f);
#pragma unroll
            for (int e = 0; e < N; ++e) {
                float a0, a1;
                unpack_f32x2(s[e], a0, a1);
                unpack_f32x2(mul2(pack2(lg2_approx(fabsf(a0)), lg2_approx(fabsf(a1))), ff), a0, a1);
                r[e] = pack2(ex2_approx(a0), ex2_approx(a1));       // s = 0: exp2(-inf) = 0
            }
        }
#pragma unroll
        for (int e = 0; e < N; ++e) { b[e] = s[e]; v[e] = s[e]; }
        if (q.m & 1) {
#pragma unroll
            for (int e = 0; e < N; ++e) v[e] = mul2(v[e], abs2(s[e]));
        }
#pragma unroll
        for (int k = 1; k < NB; ++k) {
            if ((q.m >> k) == 0) break;
#pragma unroll
            for (int e = 0; e < N; ++e) b[e] = mul2(b[e], b[e]);
            if ((q.m >> k) & 1) {
#pragma unroll
                for (int e = 0; e < N; ++e) v[e] = mul2(v[e], b[e]);
            }
        }
        if (q.f != 0.f) {
#pragma unroll
            for (int e = 0; e < N; ++e) v[e] = mul2(v[e], r[e]);
        }
#pragma unroll
        for (int e = 0; e < N; ++e) s[e] = v[e];
    }
}

constexpr int KO = 8;            // outputs per stage
constexpr int TI = 64;           // input columns per CTA (two per lane)
constexpr int RW = 16;           // batch rows per warp
constexpr int STAGES = 3;

struct BothParams {
    const float* x; const float* w;
    const float* h; const float* g; const float* r;      // [CO][Bp]: g / y^(p-1) (p = 8, 16 only), g, 1 / y
    const int* flag;                                     // [1]: some y needs the scaled form (p = 8, 16 only)
    float* gx; float* gw;                                // results, or the partial results of range 0
    size_t gx_step, gw_step;                             // floats between the partial results of consecutive ranges
    int B, Bp, COg, CIg, G, CI;
    int tiles_i, n_o, n_b;                               // 64-column tiles per group, ranges of outputs / of batch tiles
    PowQ q;
};

// What `clamped_results` needs.  (A struct of its own: with these fields in the one above, or that one as a __grid_constant__, the compiler spills
// twice as much in the kernels that never call the function: p = 64, 2048 x 1024 x 1024 952 -> 1003 us.)
struct ClampParams {
    const float* x; const float* w; const float* y; const float* g;      // y, g: [B][CO]
    int COg, CIg, CI, CO;
    PowQ q;
};

template <int WARPS, bool SCALED>
__host__ __device__ constexpr int stage_floats() { return KO * TI + (SCALED ? 2 : 1) * KO * WARPS * RW; }

// Of what a CTA owns, columns i0 .. i0 + TI - 1 of its rows b0 .. b1 - 1 of gx and of its outputs o0 .. o1 - 1 of gw, the results that are not finite, by the rule
// of the generic kernels: a term counts min(|t| / y, 1)^(p-1) with min(NaN, 1) = 1 and the sign of x - w (gx) or w - x (gw), minus for 0 and NaN.  `gx` and
// `gw` (null: not wanted): this CTA's partial results, of row 0 and output 0 of the group.  A thread each; for calls that the generic kernels served before.
__device__ __noinline__ void clamped_results(const ClampParams& p, int g, int i0, int b0, int b1, int o0, int o1, float* gx, float* gw) {
    const float* wg = p.w + (size_t)g * p.COg * p.CIg;
    const float* xg = p.x + (size_t)g * p.CIg;
    auto term = [&](int b, int o, float t) {
        const size_t at = (size_t)b * p.CO + (size_t)g * p.COg + o;
        const float yv = __ldg(p.y + at), u = fminf(fabsf(t) * (yv > 0.f ? 1.f / yv : 0.f), 1.f);
        float r = u, v = u;                                             // u^(p-1) = u * u^m * u^f
        for (int m = p.q.m; m != 0; m >>= 1) { if (m & 1) r *= v; v *= v; }
        if (p.q.f != 0.f) r *= ex2_approx(p.q.f * lg2_approx(u));
        r *= __ldg(p.g + at);
        return t > 0.f ? r : -r;
    };
    auto finite = [](const float* a) { return fabsf(__ldcg(a)) < __int_as_float(0x7f800000); };     // (L2: other threads have added to it there)
    const int cols = min(TI, p.CIg - i0);
    if (gx != nullptr)
        for (int e = threadIdx.x; e < (b1 - b0) * cols; e += blockDim.x) {
            const int b = b0 + e / cols, i = i0 + e % cols;
            float* dst = gx + (size_t)b * p.CI + i;
            if (finite(dst)) continue;
            const float xv = __ldg(xg + (size_t)b * p.CI + i);
            float a = 0.f;
#pragma unroll 4
            for (int o = o0; o < o1; ++o) a += term(b, o, xv - __ldg(wg + (size_t)o * p.CIg + i));
            *dst = a;
        }
    if (gw != nullptr)
        for (int e = threadIdx.x; e < (o1 - o0) * cols; e += blockDim.x) {
            const int o = o0 + e / cols, i = i0 + e % cols;
            float* dst = gw + (size_t)o * p.CIg + i;
            if (finite(dst)) continue;
            const float wv = __ldg(wg + (size_t)o * p.CIg + i);
            float a = 0.f;
#pragma unroll 4
            for (int b = b0; b < b1; ++b) a += term(b, o, wv - __ldg(xg + (size_t)b * p.CI + i));
            *dst = a;
        }
}

template <int IP, int WARPS, bool DOX, bool DOW, bool AL, bool SCALED>
__device__ __forceinline__ void both_body(const BothParams& p, const ClampParams& rule, float* smem) {
    constexpr int NT = WARPS * 32, BT = WARPS * RW;
    constexpr int STAGE = stage_floats<WARPS, SCALED>();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* part = smem + STAGES * STAGE;                 // [2][WARPS][KO][TI]
    int id = blockIdx.x;
    const int ti = id % p.tiles_i; id /= p.tiles_i;
    const int g = id % p.G; id /= p.G;
    const int ro = id % p.n_o, rb = id / p.n_o;
    const int KT_all = (p.COg + KO - 1) / KO, BT_all = p.Bp / BT;
    const int kt0 = (int)((long long)KT_all * ro / p.n_o), kt1 = (int)((long long)KT_all * (ro + 1) / p.n_o);
    const int bt0 = (int)((long long)BT_all * rb / p.n_b), bt1 = (int)((long long)BT_all * (rb + 1) / p.n_b);
    const int i0 = ti * TI, ic = i0 + 2 * lane;          // first of this thread's two columns
    const float* wg = p.w + (size_t)g * p.COg * p.CIg;
    const float* sa = (SCALED ? p.g : p.h) + (size_t)g * p.COg * p.Bp;
    const float* sr = p.r + (size_t)g * p.COg * p.Bp;
    float* gw = p.gw + (DOW ? (size_t)rb * p.gw_step : 0) + (size_t)g * p.COg * p.CIg;
    // an infinity or a NaN among the sums (a term enters both: one of the two is looked at); in shared memory, a register through the loops costs 2 %
    __shared__ int s_odd;
    const float inf = __int_as_float(0x7f800000);
    if (!AL && tid == 0) s_odd = 0;

    for (int bt = bt0; bt < bt1; ++bt) {
        const int b_first = bt * BT;
        // Outputs past the group and rows past the batch read the last valid row of w and x instead of zeros: their h and g are
        // zero, but t^(p-1) has to stay finite, as it is for every pair that has a y.
        auto load = [&](int s, int kt) {
            float* st = smem + s * STAGE;
            const int o0 = kt * KO;
            if (AL) {
#pragma unroll
                for (int q = tid; q < KO * TI / 4; q += NT) {
                    const int r = q / (TI / 4), c = (q % (TI / 4)) * 4;
                    const bool in = i0 + c < p.CIg;
                    cp_async16(st + r * TI + c, wg + (in ? (size_t)min(o0 + r, p.COg - 1) * p.CIg + i0 + c : 0), in ? 16 : 0);
                }
            } else {
#pragma unroll
                for (int q = tid; q < KO * TI; q += NT) {
                    const int r = q / TI, c = q % TI;
                    const bool in = i0 + c < p.CIg;
                    cp_async4(st + r * TI + c, wg + (in ? (size_t)min(o0 + r, p.COg - 1) * p.CIg + i0 + c : 0), in ? 4 : 0);
                }
            }
#pragma unroll
            for (int q = tid; q < KO * BT / 4; q += NT) {
                const int r = q / (BT / 4), c = (q % (BT / 4)) * 4;
                const bool in = o0 + r < p.COg;
                const size_t off = in ? (size_t)(o0 + r) * p.Bp + b_first + c : 0;
                cp_async16(st + KO * TI + r * BT + c, sa + off, in ? 16 : 0);
                if (SCALED) cp_async16(st + KO * TI + KO * BT + r * BT + c, sr + off, in ? 16 : 0);
            }
        };
        // the warps' sums of one stage, added in warp order and stored (first batch tile of the range) or added to memory
        auto flush = [&](int kt) {
            const float* src = part + (kt & 1) * (WARPS * KO * TI);
#pragma unroll
            for (int q = tid; q < KO * TI / 2; q += NT) {
                const int r = q / (TI / 2), c = (q % (TI / 2)) * 2;
                float2 v = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < WARPS; ++k) {
                    const float2 t = *reinterpret_cast<const float2*>(src + k * (KO * TI) + r * TI + c);
                    v.x -= t.x; v.y -= t.y;
                }
                const int o = kt * KO + r, i = i0 + c;
                if (o < p.COg && i < p.CIg) {
                    if (!AL && !DOX && (!(fabsf(v.x) < inf) || (i + 1 < p.CIg && !(fabsf(v.y) < inf)))) s_odd = 1;
                    float* dst = gw + (size_t)o * p.CIg + i;
                    if (AL) {                            // CIg is a multiple of four: both columns exist and the pair is aligned
                        if (bt == bt0) *reinterpret_cast<float2*>(dst) = v;
                        else asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(dst), "f"(v.x), "f"(v.y) : "memory");
                    } else {
                        const bool two = i + 1 < p.CIg;
                        if (bt == bt0) { dst[0] = v.x; if (two) dst[1] = v.y; }
                        else {
                            asm volatile("red.global.add.f32 [%0], %1;" ::"l"(dst), "f"(v.x) : "memory");
                            if (two) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(dst + 1), "f"(v.y) : "memory");
                        }
                    }
                }
            }
        };
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) { if (kt0 + s < kt1) load(s, kt0 + s); cp_async_commit(); }

        u64 xp[RW / 2][2], acc[DOX ? RW / 2 : 1][2];     // rows 2k, 2k + 1 of the warp's rows, two columns
#pragma unroll
        for (int k = 0; k < RW / 2; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int b = b_first + warp * RW + 2 * k;
                const float* xs = p.x + (size_t)g * p.CIg + min(ic + c, p.CIg - 1);
                xp[k][c] = pack2(__ldg(xs + (size_t)min(b, p.B - 1) * p.CI), __ldg(xs + (size_t)min(b + 1, p.B - 1) * p.CI));
                if (DOX) acc[k][c] = 0;
            }
        int rd = 0, wr = STAGES - 1;
        for (int kt = kt0; kt < kt1; ++kt) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();
            if (kt + STAGES - 1 < kt1) load(wr, kt + STAGES - 1);
            cp_async_commit();
            if (DOW && kt > kt0) flush(kt - 1);
            const float* ws = smem + rd * STAGE + 2 * lane;
            const float* hs = smem + rd * STAGE + KO * TI + warp * RW;
            const float* rs = hs + KO * BT;
            float* pt = part + ((kt & 1) * WARPS + warp) * (KO * TI) + 2 * lane;
#pragma unroll (IP == 8 ? 2 : 1)
            for (int o = 0; o < KO; ++o) {
                const float2 wv = *reinterpret_cast<const float2*>(ws + o * TI);
                const u64 w2[2] = {pack2(wv.x, wv.x), pack2(wv.y, wv.y)};
                u64 sum[2] = {0, 0};
#pragma unroll
                for (int k = 0; k < RW / 2; k += 2) {
                    const ulonglong2 hv = *reinterpret_cast<const ulonglong2*>(hs + o * BT + 2 * k);
                    ulonglong2 rv;
                    if (SCALED) rv = *reinterpret_cast<const ulonglong2*>(rs + o * BT + 2 * k);
                    if constexpr (IP > 0) {
#pragma unroll
                        for (int e = 0; e < 2; ++e)
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                u64 f[1] = {sub_f32x2(xp[k + e][c], w2[c])};
                                if (SCALED) f[0] = mul2(f[0], e ? rv.y : rv.x);
                                factors<IP>(f, p.q);
                                if (DOX) acc[k + e][c] = fma2(e ? hv.y : hv.x, f[0], acc[k + e][c]);
                                if (DOW) sum[c] = fma2(e ? hv.y : hv.x, f[0], sum[c]);
                            }
                    } else {
                        u64 f[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) f[e] = mul2(sub_f32x2(xp[k + (e >> 1)][e & 1], w2[e & 1]), e >> 1 ? rv.y : rv.x);
                        factors<IP>(f, p.q);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const u64 h2 = e >> 1 ? hv.y : hv.x;
                            if (DOX) acc[k + (e >> 1)][e & 1] = fma2(h2, f[e], acc[k + (e >> 1)][e & 1]);
                            if (DOW) sum[e & 1] = fma2(h2, f[e], sum[e & 1]);
                        }
                    }
                }
                if (DOW) {
                    float a0, a1, b0, b1;
                    unpack_f32x2(sum[0], a0, a1);
                    unpack_f32x2(sum[1], b0, b1);
                    *reinterpret_cast<float2*>(pt + o * TI) = make_float2(a0 + a1, b0 + b1);
                }
            }
            rd = (rd + 1 == STAGES) ? 0 : rd + 1;
            wr = (wr + 1 == STAGES) ? 0 : wr + 1;
        }
        cp_async_wait<0>();
        __syncthreads();
        if (DOW && kt1 > kt0) flush(kt1 - 1);
        if (DOX) {
            float* gx = p.gx + (size_t)ro * p.gx_step + (size_t)g * p.CIg + ic;
            bool odd = false;
#pragma unroll
            for (int k = 0; k < RW / 2; ++k) {
                const int b = b_first + warp * RW + 2 * k;
                float a0, a1, b0, b1;
                unpack_f32x2(acc[k][0], a0, a1);
                unpack_f32x2(acc[k][1], b0, b1);
                float* dst = gx + (size_t)b * p.CI;
                if (AL) {
                    if (ic < p.CIg && b < p.B) *reinterpret_cast<float2*>(dst) = make_float2(a0, b0);
                    if (ic < p.CIg && b + 1 < p.B) *reinterpret_cast<float2*>(dst + p.CI) = make_float2(a1, b1);
                } else {
                    // (rows past the batch are 0, columns past the edge anything)
                    odd |= (ic < p.CIg && !(fabsf(a0) < inf && fabsf(a1) < inf)) || (ic + 1 < p.CIg && !(fabsf(b0) < inf && fabsf(b1) < inf));
                    if (ic < p.CIg && b < p.B) dst[0] = a0;
                    if (ic + 1 < p.CIg && b < p.B) dst[1] = b0;
                    if (ic < p.CIg && b + 1 < p.B) dst[p.CI] = a1;
                    if (ic + 1 < p.CIg && b + 1 < p.B) dst[p.CI + 1] = b1;
                }
            }
            if (!AL && odd) s_odd = 1;
        }
    }
    if constexpr (!AL) {
        __syncthreads();
        if (s_odd)
            clamped_results(rule, g, i0, bt0 * BT, min(bt1 * BT, p.B), kt0 * KO, min(kt1 * KO, p.COg),
                            DOX ? p.gx + (size_t)ro * p.gx_step + (size_t)g * p.CIg : nullptr, DOW ? gw : nullptr);
    }
}

// 16 warps per SM whatever the CTA's width: 128 registers a thread
template <int IP, int WARPS, bool DOX, bool DOW, bool AL>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
lp_backward_both_kernel(const BothParams p, const __grid_constant__ ClampParams rule) {
    extern __shared__ __align__(16) float smem[];
    if constexpr (IP == 8 || IP == 16) {
        if (*p.flag == 0) { both_body<IP, WARPS, DOX, DOW, AL, false>(p, rule, smem); return; }
    }
    both_body<IP, WARPS, DOX, DOW, AL, true>(p, rule, smem);
}

// 1 / y (0 where y is not positive) and grad_output, less the rounding of 1 / y, transposed to [CO][Bp] (rows past the batch: zero), and for
// p = 8 / 16 the factor h = g / y^(p-1) with the look at the range of y and h.  With y in [2^-8, 2^8] (p = 8) or [2^-3, 2^4] (p = 16)
// y^(p-1) and its reciprocal stay within 2^+-60, and a difference whose power underflows is below 2^-70 of its row's y^(p-1).
template <int IP>
__global__ void __launch_bounds__(256)
lp_backward_prepare_kernel(const float* __restrict__ g, const float* __restrict__ y, int B, int Bp, int CO,
                           float* __restrict__ gt, float* __restrict__ rt, float* __restrict__ ht, int* __restrict__ flag, float pm1) {
    __shared__ float gs[32][33], ys[32][33];
    const int o0 = blockIdx.x * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    constexpr float LO = IP == 8 ? 0x1p-8f : 0x1p-3f, HI = IP == 8 ? 0x1p8f : 0x1p4f;
    bool bad = false;
    for (int b0 = blockIdx.y * 32; b0 < Bp; b0 += gridDim.y * 32) {
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
            const int b = b0 + ty + k, o = o0 + tx;
            const bool in = b < B && o < CO;
            gs[ty + k][tx] = in ? __ldg(g + (size_t)b * CO + o) : 0.f;
            ys[ty + k][tx] = in ? __ldg(y + (size_t)b * CO + o) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
            const int o = o0 + ty + k, b = b0 + tx;
            if (o < CO) {
                const float gv = gs[tx][ty + k], yv = ys[tx][ty + k];
                const size_t a = (size_t)o * Bp + b;
                // r = fl(1 / y) enters every term as r^(p-1): its rounding, r * y - 1 (exact as one fma), is taken back out of g
                const float rv = yv > 0.f ? 1.f / yv : 0.f;
                const float off = pm1 * fmaf(rv, yv, -1.f);
                rt[a] = rv;
                gt[a] = fabsf(off) < 0.01f && fabsf(gv) < __int_as_float(0x7f800000) ? fmaf(gv, -off, gv) : gv;     // (inf - inf is NaN)
                if (IP == 8 || IP == 16) {
                    bad |= b < B && !(yv >= LO && yv <= HI);
                    float pw = yv, sq = yv;                   // y^(2^k - 1): 7 or 15
#pragma unroll
                    for (int n = 2; n < IP; n *= 2) { sq *= sq; pw *= sq; }
                    const float hv = b < B ? gv / pw : 0.f;
                    bad |= gv != 0.f && !(fabsf(hv) >= 0x1p-126f && fabsf(hv) < __int_as_float(0x7f800000));
                    ht[a] = hv;
                }
            }
        }
        __syncthreads();
    }
    if ((IP == 8 || IP == 16) && __syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

// out = part[0] + part[1] + ... in that order
__global__ void __launch_bounds__(256)
lp_backward_sum_kernel(const float* __restrict__ part, size_t n, int parts, size_t step, float* __restrict__ out, int vec) {
    const size_t t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    size_t done = 0;
    if (vec) {
        const size_t n4 = n / 4;
        for (size_t e = t0; e < n4; e += stride) {
            float4 s = __ldcs(reinterpret_cast<const float4*>(part) + e);
            for (int k = 1; k < parts; ++k) {
                const float4 v = __ldcs(reinterpret_cast<const float4*>(part + k * step) + e);
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            reinterpret_cast<float4*>(out)[e] = s;
        }
        done = n4 * 4;
    }
    for (size_t e = done + t0; e < n; e += stride) {
        float s = __ldcs(part + e);
        for (int k = 1; k < parts; ++k) s += __ldcs(part + k * step + e);
        out[e] = s;
    }
}

size_t up64(size_t n) { return (n + 63) & ~(size_t)63; }

struct BothPlan {
    int warps, Bp, tiles_i, n_o, n_b;
    size_t gx_step, gw_step;          // floats of one partial result
    size_t words;                     // floats of workspace in all
};

// Rows per CTA: 128 where that pads the batch little more than the narrower tiles do (a wider CTA reads every weight fewer
// times and adds to gw in memory fewer times).  Ranges: the pair (n_o, n_b) with the smallest estimate of waves of CTAs
// times the work of one, plus the traffic of the partial results (at most 1.5 GB of it).
BothPlan plan_both(const Dims& d, float p, bool dox, bool dow) {
    BothPlan pl{};
    auto pad = [&](int t) { return (d.R + t - 1) / t * t; };
    pl.warps = d.R <= 32 ? 2 : (long long)pad(128) * 10 <= (long long)pad(64) * 11 ? 8 : 4;
    const int bt = pl.warps * RW;
    pl.Bp = pad(bt);
    pl.tiles_i = (d.CIg + TI - 1) / TI;
    const int KT = (d.COg + KO - 1) / KO, BTs = pl.Bp / bt;
    const int per_sm = 16 / pl.warps, sms = sm_count();
    const double base = (double)pl.tiles_i * d.G;
    // microseconds of one stage of one batch tile on an SM that holds per_sm CTAs
    const double stage_us = (double)KO * bt * TI * per_sm * ((p == 8.f ? 7.0 : 9.0) + 2.0) / 128.0 / 1900.0;
    double best = 1e300;
    pl.n_o = pl.n_b = 1;
    for (int n_b = 1; n_b <= BTs && n_b <= 32; ++n_b)
        for (int n_o = 1; n_o <= KT && n_o <= 64; ++n_o) {
            if (n_b > 1 && n_o * 8 < KT && n_o < 8) continue;      // partial gw is the larger tensor: split the outputs first
            const double units = base * n_o * n_b;
            const double slots = (double)per_sm * sms;
            const double full = floor(units / slots), rest = units - full * slots;
            const double waves = full + (rest > 0 ? 0.3 + 0.7 * ceil(rest / sms) / per_sm : 0.0);
            const double work = (double)((KT + n_o - 1) / n_o) * ((BTs + n_b - 1) / n_b) + 2.0;
            double bytes = 0;
            if (dox && n_o > 1) bytes += 4.0 * (2 * n_o + 1) * d.R * d.CI;
            if (dow && n_b > 1) bytes += 4.0 * (2 * n_b + 1) * d.CO * d.CIg;
            if (bytes > 1.5e9) continue;
            const double us = waves * work * stage_us + bytes / 4e6 + (dox && n_o > 1 ? 3.0 : 0.0) + (dow && n_b > 1 ? 3.0 : 0.0);
            if (us < best) { best = us; pl.n_o = n_o; pl.n_b = n_b; }
        }
    pl.gx_step = up64((size_t)d.R * d.CI);
    pl.gw_step = up64((size_t)d.CO * d.CIg);
    pl.words = 64 + 3 * up64((size_t)d.CO * pl.Bp) + (dox && pl.n_o > 1 ? pl.n_o * pl.gx_step : 0) +
               (dow && pl.n_b > 1 ? pl.n_b * pl.gw_step : 0);
    return pl;
}

template <int IP, int WARPS, bool DOX, bool DOW, bool AL>
int launch_both(const BothParams& P, const ClampParams& C, int grid, cudaStream_t st) {
    constexpr int bytes = (STAGES * stage_floats<WARPS, true>() + (DOW ? 2 * WARPS * KO * TI : 0)) * 4;
    auto kern = lp_backward_both_kernel<IP, WARPS, DOX, DOW, AL>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return LINF_ERR_LAUNCH;
    kern<<<grid, WARPS * 32, bytes, st>>>(P, C);
    return launch_status();
}

template <int IP, int WARPS, bool AL>
int launch_which(const BothParams& P, const ClampParams& C, int grid, bool dox, bool dow, cudaStream_t st) {
    if (dox && dow) return launch_both<IP, WARPS, true, true, AL>(P, C, grid, st);
    if (dox) return launch_both<IP, WARPS, true, false, AL>(P, C, grid, st);
    return launch_both<IP, WARPS, false, true, AL>(P, C, grid, st);
}

// The wide loads are for calls of 2048 rows and more (`both_ok`), which always take 8 warps.
template <int IP>
int launch_ip(const BothParams& P, const ClampParams& C, int grid, int warps, bool al, bool dox, bool dow, cudaStream_t st) {
    if (warps == 8) return al ? launch_which<IP, 8, true>(P, C, grid, dox, dow, st) : launch_which<IP, 8, false>(P, C, grid, dox, dow, st);
    return warps == 4 ? launch_which<IP, 4, false>(P, C, grid, dox, dow, st) : launch_which<IP, 2, false>(P, C, grid, dox, dow, st);
}

}  // namespace

// Which calls take this path: dense layers with at least 32 channels per group on both sides, 2 <= p < 1026 (below 2 the power
// s * |s|^(p-2) has no integer part to start from), and
//   * channel counts that are no multiples of four and 8 <= p <= 100, where the alternative is the generic kernels (figures above; larger p: `separate_better`), or
//   * 2048 rows and more (the pixels of a convolution), where the tiled weight kernel has few CTAs and long sums.
// Aligned layers of fewer rows keep the two tiled kernels, although this one would take half their time at B = 512 as well (5120 x 5120, p = 8: 6585 -> 3333 us): a training run at
// finite p amplifies a changed order of summation within two steps, and the nets, whose layers are of this kind, give the same bits from version to version.
static bool both_ok(const Dims& d, float p) {
    const bool ragged = ((d.CIg | d.COg) & 3) != 0;
    return d.HW == 1 && d.COg >= 32 && d.CIg >= 32 && p >= 2.f && p < 1026.f &&
           (ragged ? p >= 8.f && p <= 100.f : d.R >= 2048);
}

// Calls among them that the two kernels of the separate entry points do better after all.  `tiled`: those would be the tiled ones (lp_tiled_ok).
// The generic kernels clamp |t| / y to 1, which keeps the error of large powers down: against the same sums in 64 bits, error here / there with p = 150, 300,
// 1000 (unaligned tensors, 2100 rows, 64 x 64): 1.26, 1.67, 3.0; with p = 64 and 33, 42, 50, 66, 130 inputs: 1.05, 1.03, 1.01, 0.99, 0.96; elsewhere in 8 <= p <= 100, behind
// the distances as they are now, 0.81 - 0.95.  Against the tiled kernels 0.2 - 0.98 everywhere.
// One gradient alone: the power is not shared, and small calls are a matter of launches (this path has two or three).  us, there / here, rows x Din x Dout: grad_input against the
// tiled kernel, p = 8: 2048 x 64 x 64 18 / 26, 16384 x 144 x 64 64 / 80, 4096 x 128 x 64 18 / 30, 2048 x 128 x 128 32 / 30, 3000 x 300 x 300 104 / 98; p = 23.7: 2048 x 64 x 64 71 / 26,
// 16384 x 64 x 64 73 / 88.  Against the generic kernels, p = 8: grad_weight 8 x 514 x 514 12 / 21, 16 x 300 x 130 13 / 19, 32 x 65 x 65 17 / 19, 16 x 1027 x 1333 41 / 28; grad_input
// 64 x 99 x 37 20 / 22, 64 x 300 x 130 55 / 22.
static bool separate_better(const Dims& d, float p, bool tiled, bool dox, bool dow) {
    if (!tiled && (p > 100.f || (p == 64.f && d.CIg < 64))) return true;
    if (dox && dow) return false;
    if (tiled) return dox && d.COg < 128 && (p == 8.f || p == 16.f || p == 64.f || (d.R >= 8192 && p < 64.f));
    return (double)d.R * d.CO * d.CIg < 4e6 && (dow ? d.R <= 16 : d.COg < 48 && p <= 16.f);
}

size_t lp_backward_both_workspace(const Dims& d, float p, bool dox, bool dow) {
    if (!both_ok(d, p) || !(dox || dow)) return 0;
    return plan_both(d, p, dox, dow).words * sizeof(float);
}

int lp_backward_both(const float* g, const float* x, const float* w, const float* y, const Dims& d,
                     float* gx, float* gw, float p, void* ws, size_t ws_bytes, cudaStream_t st) {
    const bool dox = gx != nullptr, dow = gw != nullptr;
    const bool tiled = lp_tiled_ok(d, x, w, y, g, dox ? gx : gw) && (!dow || aligned16(gw)) && p < 1025.f;
    const size_t need = lp_backward_both_workspace(d, p, dox, dow);
    if (need == 0 || ws == nullptr || separate_better(d, p, tiled, dox, dow)) {        // one gradient at a time
        if (dox) { const int rc = lp_backward_input(g, x, w, y, d, gx, p, st); if (rc) return rc; }
        return dow ? lp_backward_weight(g, x, w, y, d, gw, p, st) : LINF_OK;
    }
    if (ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 255u)) return LINF_ERR_WORKSPACE;
    const BothPlan pl = plan_both(d, p, dox, dow);
    const size_t act = up64((size_t)d.CO * pl.Bp);
    float* base = reinterpret_cast<float*>(ws);
    int* flag = reinterpret_cast<int*>(base);
    float* gt = base + 64; float* rt = gt + act; float* ht = rt + act;
    float* next = ht + act;
    BothParams P{};
    P.x = x; P.w = w; P.h = ht; P.g = gt; P.r = rt; P.flag = flag;
    P.B = d.R; P.Bp = pl.Bp; P.COg = d.COg; P.CIg = d.CIg; P.G = d.G; P.CI = d.CI;
    P.tiles_i = pl.tiles_i; P.n_o = pl.n_o; P.n_b = pl.n_b;
    P.gx = gx; P.gw = gw;
    if (dox && pl.n_o > 1) { P.gx = next; P.gx_step = pl.gx_step; next += pl.n_o * pl.gx_step; }
    if (dow && pl.n_b > 1) { P.gw = next; P.gw_step = pl.gw_step; }
    const float e = p - 2.f, fl = floorf(e);
    P.q.m = (int)fl; P.q.f = e - fl;
    const ClampParams C{x, w, y, g, d.COg, d.CIg, d.CI, d.CO, P.q};
    const long long grid = (long long)pl.tiles_i * d.G * pl.n_o * pl.n_b;
    if (grid > 0x7fffffffLL) return LINF_ERR_DIMS;
    // Wide loads.  (Calls whose CO / G alone is no multiple of four could take them as well, but need the rule of `clamped_results`; the narrow loads cost
    // them up to 4 %: 500 x 2052 x 3001, p = 23.7: 2060 -> 2130 us.)
    const bool al = tiled && pl.warps == 8;

    const dim3 pg((d.CO + 31) / 32, (unsigned)min((pl.Bp + 31) / 32, 64));
    const bool plain = p == 8.f || p == 16.f;
    if (plain && cudaMemsetAsync(flag, 0, sizeof(int), st) != cudaSuccess) return LINF_ERR_LAUNCH;
    if (p == 8.f) lp_backward_prepare_kernel<8><<<pg, 256, 0, st>>>(g, y, d.R, pl.Bp, d.CO, gt, rt, ht, flag, p - 1.f);
    else if (p == 16.f) lp_backward_prepare_kernel<16><<<pg, 256, 0, st>>>(g, y, d.R, pl.Bp, d.CO, gt, rt, ht, flag, p - 1.f);
    else lp_backward_prepare_kernel<0><<<pg, 256, 0, st>>>(g, y, d.R, pl.Bp, d.CO, gt, rt, ht, flag, p - 1.f);
    int rc = launch_status();
    if (rc) return rc;
    if (p == 8.f) rc = launch_ip<8>(P, C, (int)grid, pl.warps, al, dox, dow, st);
    else if (p == 16.f) rc = launch_ip<16>(P, C, (int)grid, pl.warps, al, dox, dow, st);
    else if (p == 64.f) rc = launch_ip<64>(P, C, (int)grid, pl.warps, al, dox, dow, st);
    else rc = launch_ip<0>(P, C, (int)grid, pl.warps, al, dox, dow, st);
    if (rc) return rc;
    auto add_up = [&](const float* part, size_t n, int parts, size_t step, float* out) {
        const int blocks = (int)min((size_t)(8 * sm_count()), (n / 4 + 255) / 256 + 1);
        lp_backward_sum_kernel<<<blocks, 256, 0, st>>>(part, n, parts, step, out, aligned16(out) ? 1 : 0);
        return launch_status();
    };
    if (dox && pl.n_o > 1) { rc = add_up(P.gx, (size_t)d.R * d.CI, pl.n_o, pl.gx_step, gx); if (rc) return rc; }
    if (dow && pl.n_b > 1) { rc = add_up(P.gw, (size_t)d.CO * d.CIg, pl.n_b, pl.gw_step, gw); if (rc) return rc; }
    return LINF_OK;
}

}  // namespace linf
