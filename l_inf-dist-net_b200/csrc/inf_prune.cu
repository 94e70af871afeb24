// inf-dist forward and interval bounds through lists of large entries, for dense layers (HW == 1).
//
// A maximum of |x_i - w_i| over thousands of i is large, and |x_i - w_i| <= |x_i| + |w_i|: with two thresholds tx, tw and
// every entry |x_i| >= tx or |w_i| >= tw looked at, no other i can reach more than tx + tw.  So an output whose
// maximum over the listed entries is GREATER than fl(tx + tw) is final, exactly as the full scan gives it: rounding is
// monotonic, |fl(x - w)| <= fl(|x| + |w|) <= fl(tx + tw), so no unlisted term equals the maximum either and the lowest index
// among equal terms is among the listed ones.  Outputs that do not pass this test are computed by a full scan
// (`fail_kernel`); if there are too many of them, or the lists would be long, the dense kernel does the layer.
//
//   sample_kernel   looks at 128 rows of either side (counts of entries by magnitude) and 1024 outputs; the last CTA takes
//                   tx + tw = the smallest sampled output and divides it so that the lists are shortest, or decides for the dense kernel
//   list_kernel     one warp per row of x and of w writes the row's entries (value, index) of at least its threshold,
//                   ascending, slot by slot across the rows ([slot][row]: a warp that works on 32 rows reads whole lines)
//   gather_kernel   four rows of one side interleaved in shared memory (one 16-byte load gives an entry's four partners), the
//                   lanes of a warp are rows of the other side and walk over their own lists.  Once for the lists of x (skipped when
//                   they are all empty), once for the lists of w, which also merges, tests and stores.
//   fail_kernel     four warps per output that did not pass
// All decisions are taken on the device; the dense kernel is launched behind and returns at once unless it is wanted.
//
// Bound: shared-memory gathers (a random 16-byte load of a warp takes about 10 cycles for 4 x 32 terms) and the 8-byte list entries
// from L2.  How many entries there are depends on the data.  Dout = Din = 5120, B = 512: x uniform in [0,1) or activations of a
// distance net, w ~ N(0,1): 20-45 of 5120; x and w ~ N(0,1): 240.  A gathered term costs as much as eight terms of the
// dense kernel (bounds: five), which sets `budget`.  Measured on one B200, us, full scan -> here, B = 512, Dout = 5120: Din = 784, x uniform 175 -> 100;
// Din = 3072, uniform 560 -> 130; Din = 5120, normal 908 -> 400, 0.25 * normal 902 -> 223; bounds Din = 3072, uniform 1404 -> 190, Din = 5120, normal
// 2325 -> 590.  At Din = 5120, normal: sample 25, lists 28, gathers 2 x 160 (73-81 % of the shared-memory data path), failed outputs 8-30.
#include "common.cuh"

namespace linf {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kBins = 4096, kBinShift = 19;     // bins of |v|: exponent and four bits of the mantissa
constexpr int kSampleCtas = 128;
constexpr int kMaxList = 512;                   // slots per row at most (the thresholds aim at 0.6 of them)
constexpr int kMaxK = 14000;                    // 16 bytes each in shared memory

struct Head {                                   // zeroed before every call
    int ymin_inv;                               // 0x7fffffff - bits of the smallest sampled output
    int ticket;
    int dense;                                  // the dense kernel is wanted
    int any_x;                                  // some list of x is not empty
    int n_fail;
    float tx, tw, bound;
    int pad[56];
};

struct PruneParams {
    const float* xl; const float* xu;           // x (twice), or lower and upper
    const float* w;
    float* y0; int* pos; float* y1;             // forward: y, pos (or null); bounds: lower, -, upper
    int R, G, K, N, CI, CO;                     // K inputs and N outputs per group
    Head* head;
    int* hist;                                  // [2][kBins]
    int* cnt_x; int* cnt_w;                     // [G * R], [CO]
    void* list_x; int2* list_w;                 // [slots][G * R] int2 or int4, [slots][CO]
    int* fail; int fail_cap;
    int slots;
    int vec;                                    // y and pos take 16-byte stores at multiples of four outputs
    float budget;                               // entries per output at which the dense kernel is as fast
    float x_pass;                               // what a pass with lists of x costs, in entries per output
    int* tickets; int n_tickets;                // words that the dense kernel of the bounds wants cleared
    Post post;
};

__device__ __forceinline__ float pinf() { return __int_as_float(0x7f800000); }
__device__ __forceinline__ int signed_at(float t, int at) { return at | (t < 0.f ? (int)0x80000000 : 0); }

__device__ __forceinline__ float4 ld4(const float* a) { return __ldg(reinterpret_cast<const float4*>(a)); }

// one term of an interval bound: U = max of the far ends, m = min (the lower bound is -m, at least 0)
__device__ __forceinline__ void bound_term(float lo, float up, float w, float& m, float& U) {
    const float a = w - lo, b = up - w;
    U = max3(U, a, b);
    m = fminf(m, fminf(a, b));
}

template <bool BOUND, bool VEC>
__global__ void __launch_bounds__(256)
sample_kernel(const PruneParams p) {
    __shared__ __align__(16) int hx[kBins], hw[kBins];
    __shared__ int s_last, s_out[8][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kBins; i += 256) { hx[i] = 0; hw[i] = 0; }
    __syncthreads();
    const int rows = p.R * p.G;
    const int rx = (int)((long long)rows * blockIdx.x / kSampleCtas);         // row of x: r * G + g in memory
    const int r = rx / p.G, g = rx - r * p.G;
    const size_t xa = (size_t)r * p.CI + (size_t)g * p.K;
    // eight outputs of this row of x, every thread on all eight: 9 loads in flight per step
    const float* wr[8];
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int o = (int)((long long)p.N * ((blockIdx.x * 8 + q) * 37 % 1024) / 1024);
        wr[q] = p.w + ((size_t)g * p.N + o) * p.K;
        v[q] = 0.f;
    }
    auto look = [&](float a, float b, const float (&wv)[8]) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = BOUND ? max3(v[q], a - wv[q], wv[q] - b) : fmaxf(v[q], fabsf(a - wv[q]));
        atomicAdd(&hx[__float_as_int(BOUND ? fmaxf(fabsf(a), fabsf(b)) : fabsf(a)) >> kBinShift], 1);
        atomicAdd(&hw[__float_as_int(fabsf(wv[0])) >> kBinShift], 1);
    };
    if (VEC) {
        for (int k = 4 * tid; k < p.K; k += 1024) {
            const float4 a = ld4(p.xl + xa + k), b = BOUND ? ld4(p.xu + xa + k) : a;
            float4 f[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) f[q] = ld4(wr[q] + k);
            float wv[8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#pragma unroll
                for (int q = 0; q < 8; ++q) wv[q] = c == 0 ? f[q].x : c == 1 ? f[q].y : c == 2 ? f[q].z : f[q].w;
                look(c == 0 ? a.x : c == 1 ? a.y : c == 2 ? a.z : a.w, c == 0 ? b.x : c == 1 ? b.y : c == 2 ? b.z : b.w, wv);
            }
        }
    } else {
#pragma unroll 2
        for (int k = tid; k < p.K; k += 256) {
            const float a = __ldg(p.xl + xa + k), b = BOUND ? __ldg(p.xu + xa + k) : a;
            float wv[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) wv[q] = __ldg(wr[q] + k);
            look(a, b, wv);
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int bits = __reduce_min_sync(FULL, 0x7fffffff - __float_as_int(v[q]));    // the largest v of the lanes
        if (lane == 0) s_out[q][warp] = bits;
    }
    __syncthreads();
    if (tid < 8) {
        int bits = s_out[tid][0];
#pragma unroll
        for (int k = 1; k < 8; ++k) bits = min(bits, s_out[tid][k]);
        atomicMax(&p.head->ymin_inv, bits);
    }
    __syncthreads();
    for (int i = tid; i < kBins; i += 256) {
        if (hx[i]) atomicAdd(&p.hist[i], hx[i]);
        if (hw[i]) atomicAdd(&p.hist[kBins + i], hw[i]);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&p.head->ticket, 1) == kSampleCtas - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();

    // ---- the last CTA: entries at or above every bin edge, then the division of the smallest sampled output ----
    constexpr int PER = kBins / 256;                // 16: four 16-byte loads
    __shared__ int tot[2][8];
    __shared__ float s_cost[8]; __shared__ int s_bin[8];
    int above[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int c[PER], sum = 0;
#pragma unroll
        for (int j = 0; j < PER; j += 4) {
            const int4 q = __ldcg(reinterpret_cast<const int4*>(p.hist + h * kBins + tid * PER + j));
            c[j] = q.x; c[j + 1] = q.y; c[j + 2] = q.z; c[j + 3] = q.w;
        }
        int* dst = h ? hw : hx;
#pragma unroll
        for (int j = PER - 1; j >= 0; --j) { sum += c[j]; dst[tid * PER + j] = sum; }
        int incl = sum;                             // of this lane and the lanes above
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const int t = __shfl_down_sync(FULL, incl, s);
            if (lane + s < 32) incl += t;
        }
        if (lane == 0) tot[h][warp] = incl;
        above[h] = incl - sum;
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        for (int k = warp + 1; k < 8; ++k) above[h] += tot[h][k];
        int* dst = h ? hw : hx;
#pragma unroll
        for (int j = 0; j < PER; ++j) dst[tid * PER + j] += above[h];
    }
    __syncthreads();
    const float yref = __int_as_float(0x7fffffff - __ldcg(&p.head->ymin_inv));
    float cost = 3e38f; int bin = 0;
    for (int j = tid * PER; j < tid * PER + PER; ++j) {
        const float tx = __int_as_float(j << kBinShift);
        const float tw = (yref - tx) * 0.999999f;
        if (j == 0 || !(tw > 0.f) || !(yref < 3e38f)) continue;
        const float nx = hx[j] * (1.f / kSampleCtas), nw = hw[__float_as_int(tw) >> kBinShift] * (1.f / kSampleCtas);
        // Lists of x that are (with a bin to spare) empty spare a pass over the weights and the outputs, about a dozen entries' worth, and the building and reading of
        // those lists, a fixed time per row of x.  Measured on bounds, entries' worth per output: 58 with 64 outputs per group, 32 - 36 with 128, 23 with 256, 12 with 1000, 2 - 5 with
        // 3000 and more (100000 x 256 x 64, x = 0.2 * normal, where a constant 12 chose the lists: 300 us by the full scan, 700 by the lists, 357 now).
        const float c = nx + nw + (hx[j - 1] == 0 ? 0.f : p.x_pass);
        if (nx <= 0.6f * p.slots && nw <= 0.6f * p.slots && c < cost) { cost = c; bin = j; }
    }
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        const float oc = __shfl_xor_sync(FULL, cost, s); const int ob = __shfl_xor_sync(FULL, bin, s);
        if (oc < cost || (oc == cost && ob < bin)) { cost = oc; bin = ob; }
    }
    if (lane == 0) { s_cost[warp] = cost; s_bin[warp] = bin; }
    __syncthreads();
    if (tid == 0) {
        for (int k = 1; k < 8; ++k) if (s_cost[k] < cost) { cost = s_cost[k]; bin = s_bin[k]; }
        const float tx = __int_as_float(bin << kBinShift), tw = (yref - tx) * 0.999999f;
        p.head->tx = tx; p.head->tw = tw;
        p.head->bound = __fadd_ru(tx, tw);
        if (!(cost < p.budget)) p.head->dense = 1;
    }
}

// One row's entries of at least `thr`, ascending, written by a warp: (value, index), or (lower, upper, index, -) for PAIR.  Returns how
// many there are; `odd`: an interval that is empty or not finite.  VEC: K is a multiple of four and the row 16-byte aligned.
template <bool PAIR, bool VEC>
__device__ __forceinline__ int list_row(const float* __restrict__ lo, const float* __restrict__ up, int K, float thr, int slots,
                                        void* list, int stride, int row, int lane, bool& odd) {
    constexpr int W = VEC ? 4 : 1, U = VEC ? (PAIR ? 2 : 4) : 8;
    const unsigned below = (1u << lane) - 1u;
    int n = 0;
    for (int k0 = 0; k0 < K; k0 += 32 * U * W) {
        float a[U][W], b[U][W];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + (32 * u + lane) * W;
            if (VEC) {
                const float4 q = k < K ? __ldg(reinterpret_cast<const float4*>(lo + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
                a[u][0] = q.x; a[u][W > 1] = q.y; a[u][W > 1 ? 2 : 0] = q.z; a[u][W > 1 ? 3 : 0] = q.w;
                if (PAIR) {
                    const float4 t = k < K ? __ldg(reinterpret_cast<const float4*>(up + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    b[u][0] = t.x; b[u][W > 1] = t.y; b[u][W > 1 ? 2 : 0] = t.z; b[u][W > 1 ? 3 : 0] = t.w;
                }
            } else {
                a[u][0] = k < K ? __ldg(lo + k) : 0.f;
                if (PAIR) b[u][0] = k < K ? __ldg(up + k) : 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + (32 * u + lane) * W;
            bool hit[W];
            bool any = false;
#pragma unroll
            for (int c = 0; c < W; ++c) {
                if (PAIR) odd |= !(a[u][c] <= b[u][c] && a[u][c] > -pinf() && b[u][c] < pinf());
                hit[c] = k < K && (fabsf(a[u][c]) >= thr || (PAIR && fabsf(b[u][c]) >= thr));
                any |= hit[c];
            }
            if (__ballot_sync(FULL, any) == 0) continue;
            int s = n;
#pragma unroll
            for (int c = 0; c < W; ++c) {
                const unsigned m = __ballot_sync(FULL, hit[c]);
                s += __popc(m & below);
                n += __popc(m);
            }
#pragma unroll
            for (int c = 0; c < W; ++c)
                if (hit[c]) {
                    if (s < slots) {
                        const size_t e = (size_t)s * stride + row;
                        if (PAIR) reinterpret_cast<int4*>(list)[e] = make_int4(__float_as_int(a[u][c]), __float_as_int(b[u][c]), k + c, 0);
                        else reinterpret_cast<int2*>(list)[e] = make_int2(__float_as_int(a[u][c]), k + c);
                    }
                    ++s;
                }
        }
    }
    return n;
}

// Rows 0 .. R * G - 1 are rows of x, in the order g * R + r; the others rows of w.
template <bool BOUND, bool VEC>
__global__ void __launch_bounds__(256)
list_kernel(const PruneParams p) {
    if (p.head->dense) return;
    const int lane = threadIdx.x & 31;
    const int nx = p.R * p.G;
    int row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= nx + p.CO) return;
    bool odd = false;
    if (row < nx) {
        const int g = row / p.R;
        const size_t at = (size_t)(row - g * p.R) * p.CI + (size_t)g * p.K;
        const int n = list_row<BOUND, VEC>(p.xl + at, p.xu + at, p.K, p.head->tx, p.slots, p.list_x, nx, row, lane, odd);
        odd = __any_sync(FULL, odd);
        if (lane == 0) {
            p.cnt_x[row] = min(n, p.slots);
            if (n > p.slots || odd) p.head->dense = 1;
            if (n > 0) p.head->any_x = 1;
        }
    } else {
        row -= nx;
        const float* w = p.w + (size_t)row * p.K;
        const int n = list_row<false, VEC>(w, w, p.K, p.head->tw, p.slots, p.list_w, p.CO, row, lane, odd);
        if (lane == 0) {
            p.cnt_w[row] = min(n, p.slots);
            if (n > p.slots) p.head->dense = 1;
        }
    }
}

// Shared rows, 4 * LG of them as [K][4 * LG] floats.  W_LISTS: rows of x (bounds: lower and upper of half as many rows), lanes = outputs.
// Otherwise: rows of w, lanes = rows of x.  LG neighbouring lanes walk the list of one row together, each with its own four of the shared
// rows: a gather then reads 16 * LG contiguous bytes per entry, which meets fewer bank conflicts, and the warp's
// lists differ less in length; against that, a CTA fills more shared memory and every lane does its list's bookkeeping (`launch_gather`).
template <bool BOUND, bool W_LISTS, bool TRACK, int LG>
__global__ void __launch_bounds__(1024, 1)
gather_kernel(const PruneParams p, int blocks_a, int splits) {
    extern __shared__ __align__(16) float4 rows4[];
    const int any_x = p.head->any_x;
    if (p.head->dense || (!W_LISTS && !any_x)) return;
    constexpr bool PAIRS = BOUND && W_LISTS;
    constexpr int NA = PAIRS ? 2 : 4;                   // outputs of a lane per list row
    constexpr int RW = 32 / LG;                         // list rows of a warp
    const int tid = threadIdx.x, lane = tid & 31, nt = blockDim.x, quad = tid % LG;
    int id = blockIdx.x;
    const int split = id % splits; id /= splits;
    const int blk = id % blocks_a, g = id / blocks_a;
    const int a0 = blk * (NA * LG) + NA * quad;         // first of this lane's shared rows
    {
        const int last = (W_LISTS ? p.R : p.N) - 1;
        const float* src[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            if (PAIRS) src[a] = (a & 1 ? p.xu : p.xl) + (size_t)min(a0 + (a >> 1), last) * p.CI + (size_t)g * p.K;
            else if (W_LISTS) src[a] = p.xl + (size_t)min(a0 + a, last) * p.CI + (size_t)g * p.K;
            else src[a] = p.w + ((size_t)g * p.N + min(a0 + a, last)) * p.K;
        }
#pragma unroll 4
        for (int k = tid / LG; k < p.K; k += nt / LG)
            rows4[k * LG + quad] = make_float4(__ldg(src[0] + k), __ldg(src[1] + k), __ldg(src[2] + k), __ldg(src[3] + k));
    }
    __syncthreads();
    const int NL = W_LISTS ? p.N : p.R;
    const int stride = W_LISTS ? p.CO : p.G * p.R;
    const int* cnt = (W_LISTS ? p.cnt_w : p.cnt_x) + g * NL;
    const int per = ((NL + splits - 1) / splits + RW - 1) / RW * RW;
    const int l_end = min(NL, (split + 1) * per);
    const float bound = p.head->bound;
    [[maybe_unused]] bool lost = false;
    for (int l0 = split * per + (tid >> 5) * RW; l0 < l_end; l0 += (nt >> 5) * RW) {
        if (W_LISTS && __any_sync(FULL, lost)) return;      // more outputs failed than fail_kernel takes: the dense kernel does the layer
        const int l = l0 + lane / LG;
        const int n = l < l_end ? __ldg(cnt + l) : 0;
        const int most = __reduce_max_sync(FULL, n);
        float t[NA];                                    // forward: signed difference of the largest term; bounds: U
        [[maybe_unused]] float m[BOUND ? NA : 1];
        [[maybe_unused]] int at[TRACK ? NA : 1];
#pragma unroll
        for (int a = 0; a < NA; ++a) { t[a] = 0.f; if (BOUND) m[a] = 0.f; if (TRACK) at[a] = 0; }
        constexpr int U = 4;
        float v[U], v2[U]; int k[U];
        // past the end of a list: a NaN, which no comparison takes
        auto fetch = [&](int s) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                v[u] = v2[u] = __int_as_float(0x7fffffff); k[u] = 0;
                if (s + u < n) {
                    const size_t e = (size_t)(s + u) * stride + (size_t)g * NL + l;
                    if (!W_LISTS && BOUND) {
                        const int4 q = __ldg(reinterpret_cast<const int4*>(p.list_x) + e);
                        v[u] = __int_as_float(q.x); v2[u] = __int_as_float(q.y); k[u] = q.z;
                    } else {
                        const int2 q = __ldg((W_LISTS ? p.list_w : reinterpret_cast<const int2*>(p.list_x)) + e);
                        v[u] = __int_as_float(q.x); k[u] = q.y;
                    }
                }
            }
        };
        fetch(0);
        for (int s = 0; s < most; s += U) {
            float c[U], c2[U]; int kk[U];
#pragma unroll
            for (int u = 0; u < U; ++u) { c[u] = v[u]; c2[u] = v2[u]; kk[u] = k[u]; }
            fetch(s + U);                               // the next entries are on their way while these are looked up
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float4 f = rows4[kk[u] * LG + quad];
                const float r[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    if constexpr (PAIRS) bound_term(r[2 * a], r[2 * a + 1], c[u], m[a], t[a]);
                    else if constexpr (BOUND) bound_term(c[u], c2[u], r[a], m[a], t[a]);
                    else {
                        const float d = W_LISTS ? r[a] - c[u] : c[u] - r[a];
                        if (fabsf(d) > fabsf(t[a])) { t[a] = d; if constexpr (TRACK) at[a] = kk[u]; }
                    }
                }
            }
        }
        if (l >= l_end) continue;
        if constexpr (!W_LISTS && !BOUND) {
            if (p.vec && a0 + 3 < p.N) {                // four neighbouring outputs of one row
                const size_t e = (size_t)l * p.CO + g * p.N + a0;
                *reinterpret_cast<float4*>(p.y0 + e) = make_float4(fabsf(t[0]), fabsf(t[1]), fabsf(t[2]), fabsf(t[3]));
                if constexpr (TRACK)
                    *reinterpret_cast<int4*>(p.pos + e) = make_int4(signed_at(t[0], at[0]), signed_at(t[1], at[1]), signed_at(t[2], at[2]), signed_at(t[3], at[3]));
                continue;
            }
        }
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const int r = W_LISTS ? a0 + a : l, o = W_LISTS ? l : a0 + a;
            if (W_LISTS ? r >= p.R : o >= p.N) continue;
            const int c = g * p.N + o;
            const size_t e = (size_t)r * p.CO + c;
            if constexpr (BOUND) {
                float L = 0.f - m[a], U2 = t[a];
                if (W_LISTS) {
                    if (any_x) { L = fmaxf(L, p.y0[e]); U2 = fmaxf(U2, p.y1[e]); }
                    if (L > bound && U2 > bound) {
                        const float lo = post_apply(p.post, L, c), up = post_apply(p.post, U2, c);
                        L = p.post.negate ? up : lo; U2 = p.post.negate ? lo : up;
                    } else {
                        const int s = atomicAdd(&p.head->n_fail, 1);
                        if (s < p.fail_cap) p.fail[s] = (int)e; else lost = true;
                    }
                }
                p.y0[e] = L; p.y1[e] = U2;
            } else {
                float best = fabsf(t[a]); int where = TRACK ? at[TRACK ? a : 0] : 0;
                bool neg = t[a] < 0.f;
                if (W_LISTS) {
                    if (any_x) {
                        const float y = p.y0[e];
                        const int q = TRACK ? p.pos[e] : 0;
                        if (y > best || (TRACK && y == best && (q & 0x7fffffff) < where)) { best = y; where = q & 0x7fffffff; neg = q < 0; }
                    }
                    if (!(best > bound)) {
                        const int s = atomicAdd(&p.head->n_fail, 1);
                        if (s < p.fail_cap) p.fail[s] = (int)e; else lost = true;
                    }
                    best = post_apply(p.post, best, c);
                }
                p.y0[e] = best;
                if (TRACK) p.pos[e] = where | (neg ? (int)0x80000000 : 0);
            }
        }
    }
}

// The outputs that did not pass: a full scan by a CTA of four warps each (by one warp, the 160 dependent loads of a row of 5120 made
// this the longest kernel of a layer with a few hundred such outputs: 40 us).
template <bool BOUND, bool TRACK, bool VEC>
__global__ void __launch_bounds__(128)
fail_kernel(const PruneParams p) {
    __shared__ float s_t[4], s_u[4];
    __shared__ int s_i[4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = p.head->n_fail;
    if (n > p.fail_cap || p.head->dense) {
        // too many, or lists that do not serve: the dense kernel behind this one does the layer.  That of the bounds may combine partial
        // results in memory: the outputs are cleared for it.
        if (blockIdx.x == 0 && tid == 0) p.head->dense = 1;
        if (BOUND) {
            const size_t outs = (size_t)p.R * p.CO;
            for (size_t e = (size_t)blockIdx.x * 128 + tid; e < outs; e += (size_t)gridDim.x * 128) { p.y0[e] = 0.f; p.y1[e] = 0.f; }
            for (int e = blockIdx.x * 128 + tid; e < p.n_tickets; e += gridDim.x * 128) p.tickets[e] = 0;
        }
        return;
    }
    for (int q = blockIdx.x; q < n; q += gridDim.x) {
        const int e = p.fail[q], r = e / p.CO, c = e - r * p.CO, g = c / p.N;
        const size_t xa = (size_t)r * p.CI + (size_t)g * p.K;
        const float* wr = p.w + (size_t)c * p.K;
        float t = 0.f, u = 0.f; int at = 0;             // forward: signed difference, index; bounds: -lower, upper
        auto take = [&](float lo, float up, float w, int k) {
            if (BOUND) {
                bound_term(lo, up, w, t, u);
            } else {
                const float d = lo - w;
                if (fabsf(d) > fabsf(t)) { t = d; at = k; }
            }
        };
        if (VEC) {
#pragma unroll 4
            for (int k = 4 * tid; k < p.K; k += 512) {
                const float4 a = ld4(p.xl + xa + k), b = BOUND ? ld4(p.xu + xa + k) : a, w = ld4(wr + k);
                take(a.x, b.x, w.x, k); take(a.y, b.y, w.y, k + 1); take(a.z, b.z, w.z, k + 2); take(a.w, b.w, w.w, k + 3);
            }
        } else {
#pragma unroll 8
            for (int k = tid; k < p.K; k += 128) {
                const float a = __ldg(p.xl + xa + k);
                take(a, BOUND ? __ldg(p.xu + xa + k) : a, __ldg(wr + k), k);
            }
        }
        // larger |t| first, then the lower index
        auto merge = [&](float ot, float ou, int oa) {
            if (BOUND) { t = fminf(t, ot); u = fmaxf(u, ou); }
            else if (fabsf(ot) > fabsf(t) || (fabsf(ot) == fabsf(t) && oa < at)) { t = ot; at = oa; }
        };
#pragma unroll
        for (int s = 16; s; s >>= 1) {
            const float ot = __shfl_xor_sync(FULL, t, s), ou = __shfl_xor_sync(FULL, u, s);
            const int oa = __shfl_xor_sync(FULL, at, s);
            merge(ot, ou, oa);
        }
        __syncthreads();                                // the previous output's values have been read
        if (lane == 0) { s_t[warp] = t; s_u[warp] = u; s_i[warp] = at; }
        __syncthreads();
        if (tid == 0) {
            for (int k = 1; k < 4; ++k) merge(s_t[k], s_u[k], s_i[k]);
            if (BOUND) {
                const float lo = post_apply(p.post, 0.f - t, c), up = post_apply(p.post, u, c);
                p.y0[e] = p.post.negate ? up : lo;
                p.y1[e] = p.post.negate ? lo : up;
            } else {
                p.y0[e] = post_apply(p.post, fabsf(t), c);
                if (TRACK) p.pos[e] = signed_at(t, at);
            }
        }
    }
}

size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

struct PruneSizes { size_t head, cnt_x, cnt_w, list_x, list_w, fail, total; int slots, fail_cap; };

PruneSizes prune_sizes(const Dims& d, bool bound) {
    PruneSizes s;
    const size_t nx = (size_t)d.R * d.G, outs = (size_t)d.R * d.CO;
    // The lists take 64 MB or, where that is more, half of the call's own tensors: the rows of a large convolution would ask for more than those
    // (131072 rows: 0.5 GB, bounds 1 GB).  20 to 250 entries are what rows have; longer lists than the slots hold send the layer to the dense kernel.
    const size_t own = sizeof(float) * ((bound ? 2 : 1) * (size_t)d.R * d.CI + (size_t)d.CO * d.CIg + 2 * outs);
    const size_t slots = max((size_t)64 << 20, own / 2) / (nx * (bound ? 16 : 8) + (size_t)d.CO * 8);
    s.slots = (int)min(slots, (size_t)min(kMaxList, d.CIg));
    s.fail_cap = (int)(outs / 128 + 1024);
    size_t at = 0;
    s.head = at; at += up256(sizeof(Head) + 2 * kBins * sizeof(int));
    s.cnt_x = at; at += up256(nx * sizeof(int));
    s.cnt_w = at; at += up256((size_t)d.CO * sizeof(int));
    s.list_x = at; at += up256(nx * s.slots * (bound ? 16 : 8));
    s.list_w = at; at += up256((size_t)d.CO * s.slots * 8);
    s.fail = at; at += up256((size_t)s.fail_cap * sizeof(int));
    s.total = at;
    return s;
}

template <bool BOUND, bool W_LISTS, bool TRACK, int LG>
int launch_gather_as(const PruneParams& p, cudaStream_t st) {
    constexpr int NA = (BOUND && W_LISTS ? 2 : 4) * LG;
    const int na = W_LISTS ? p.R : p.N, nl = W_LISTS ? p.N : p.R;
    const int blocks = (na + NA - 1) / NA;
    const size_t smem = (size_t)p.K * 16 * LG;
    int per_sm = (int)(220 * 1024 / (smem + 1024));
    if (per_sm > 4) per_sm = 4;
    if (per_sm < 1) per_sm = 1;
    // 32 warps on an SM (64 registers a thread); no more threads than lanes of work, but enough to fill the shared rows
    int threads = 1024 / per_sm / 32 * 32;           // whole warps
    const int lanes = (nl * LG + 31) / 32 * 32;
    if (threads > lanes) threads = lanes < 256 ? 256 : lanes;
    // enough CTAs for two waves, as long as every warp of a CTA has a list to walk
    const long long want = 2LL * per_sm * sm_count();
    long long splits = (want + (long long)blocks * p.G - 1) / ((long long)blocks * p.G);
    const int most = (int)(((long long)nl * LG + threads - 1) / threads);
    if (splits > most) splits = most;
    if (splits < 1) splits = 1;
    auto kern = gather_kernel<BOUND, W_LISTS, TRACK, LG>;
    if (smem > 40 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return LINF_ERR_LAUNCH;
    kern<<<(unsigned)((long long)blocks * p.G * splits), threads, smem, st>>>(p, blocks, (int)splits);
    return launch_status();
}

// LG = 2 pays for the lists of w under bounds (B = 512, Din = 3072, Dout = 5120: 182 -> 168 us; Din = Dout = 5120, normal: 308 -> 285), as long as
// there are enough rows for twice the rows a CTA; elsewhere one lane per list row is faster (forward, same shapes: 90 / 93, 152 / 174).
template <bool BOUND, bool W_LISTS, bool TRACK>
int launch_gather(const PruneParams& p, cudaStream_t st) {
    if constexpr (BOUND && W_LISTS) {
        if (p.K <= kMaxK / 2 && p.R > 128) return launch_gather_as<BOUND, W_LISTS, TRACK, 2>(p, st);
    }
    return launch_gather_as<BOUND, W_LISTS, TRACK, 1>(p, st);
}

template <bool BOUND, bool TRACK>
int run_pruned(const PruneParams& p, bool vec, cudaStream_t st) {
    if (cudaMemsetAsync(p.head, 0, sizeof(Head) + 2 * kBins * sizeof(int), st) != cudaSuccess) return LINF_ERR_LAUNCH;
    const int blocks = (p.R * p.G + p.CO + 7) / 8;
    if (vec) {
        sample_kernel<BOUND, true><<<kSampleCtas, 256, 0, st>>>(p);
        list_kernel<BOUND, true><<<blocks, 256, 0, st>>>(p);
    } else {
        sample_kernel<BOUND, false><<<kSampleCtas, 256, 0, st>>>(p);
        list_kernel<BOUND, false><<<blocks, 256, 0, st>>>(p);
    }
    int rc = launch_status(2);
    if (rc) return rc;
    rc = launch_gather<BOUND, false, TRACK>(p, st);
    if (rc) return rc;
    rc = launch_gather<BOUND, true, TRACK>(p, st);
    if (rc) return rc;
    if (vec) fail_kernel<BOUND, TRACK, true><<<8 * sm_count(), 128, 0, st>>>(p);
    else fail_kernel<BOUND, TRACK, false><<<8 * sm_count(), 128, 0, st>>>(p);
    return launch_status();
}

}  // namespace

// Which calls are worth the attempt: dense layers with long rows, and enough work that the sample, the lists and five launches (about
// 30 us) are small against the full scan.  Measured, us, full scan / lists, B = 512, x = 0.25 * normal: 1024 x 1024 forward 63 / 60, bounds 122 / 77;
// 784 x 5120 (x uniform) forward 175 / 100.  The kernels for rows that are no multiple of four floats are three times slower, so that the line lies lower
// there (203 x 1027 x 1333, normal: 153 / 67).  Data that do not suit cost, full scan alone / behind the lists, Dout = 5120: found by the sample 176 / 208 (Din = 784), 563 / 603 (3072), 910 / 956
// (5120), bounds 409 / 443, 1405 / 1437, 2326 / 2364; found when half of the outputs have failed 173 / 245, 557 / 649, 899 / 1020, bounds 409 / 504, 1404 / 1521, 2326 / 2483.
bool inf_prune_ok(const Dims& d, bool bound) {
    const double least = (d.CIg & 3) != 0 ? 1.5e8 : bound ? 5e8 : 1.5e9;
    return d.HW == 1 && d.CIg >= 256 && d.CIg <= kMaxK && d.COg >= 64 && d.R >= 64 &&
           (double)d.R * d.CO * d.CIg >= least && (long long)d.R * d.G + d.CO <= 131072;
}

size_t inf_prune_workspace(const Dims& d, bool bound) { return inf_prune_ok(d, bound) ? prune_sizes(d, bound).total : 0; }

// The list pass over a workspace of inf_prune_workspace bytes.  *only_if receives the device flag under which the dense kernel must
// run behind it.  dense_speed: terms per second of the kernel behind, relative to the tiled ones.  tickets: words to clear for that kernel (bounds).
int inf_prune(const float* xl, const float* xu, const float* w, const Dims& d, float* y0, int* pos, float* y1, bool bound,
              void* ws, cudaStream_t st, const Post& post, float dense_speed, const int** only_if, int* tickets, int n_tickets) {
    const PruneSizes s = prune_sizes(d, bound);
    char* base = reinterpret_cast<char*>(ws);
    PruneParams p;
    p.xl = xl; p.xu = xu; p.w = w; p.y0 = y0; p.pos = pos; p.y1 = y1;
    p.R = d.R; p.G = d.G; p.K = d.CIg; p.N = d.COg; p.CI = d.CI; p.CO = d.CO;
    p.head = reinterpret_cast<Head*>(base + s.head);
    p.hist = reinterpret_cast<int*>(base + s.head + sizeof(Head));
    p.cnt_x = reinterpret_cast<int*>(base + s.cnt_x); p.cnt_w = reinterpret_cast<int*>(base + s.cnt_w);
    p.list_x = base + s.list_x; p.list_w = reinterpret_cast<int2*>(base + s.list_w);
    p.fail = reinterpret_cast<int*>(base + s.fail); p.fail_cap = s.fail_cap;
    p.slots = s.slots;
    p.vec = (d.COg & 3) == 0 && aligned16(y0) && (pos == nullptr || aligned16(pos));
    // time of a gathered term against one of the tiled kernels (B = 512, Din = Dout = 5120: 1.6 / 0.18 us per entry and input, bounds 2.2 / 0.45)
    const float gather_cost = bound ? 5.f : 8.5f;
    p.budget = 0.9f * d.CIg / (gather_cost * dense_speed);
    p.post = post;
    p.x_pass = 12.f + 3000.f / d.COg;
    p.tickets = tickets; p.n_tickets = n_tickets;
    *only_if = &p.head->dense;
    const bool vec = (d.CIg & 3) == 0 && aligned16(xl) && aligned16(xu) && aligned16(w);
    if (bound) return run_pruned<true, false>(p, vec, st);
    return pos != nullptr ? run_pruned<false, true>(p, vec, st) : run_pruned<false, false>(p, vec, st);
}

}  // namespace linf
