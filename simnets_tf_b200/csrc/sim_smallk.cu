// Similarity forward for short patches (K = C * bh * bw <= 32: a first layer over a few image channels).
//
// As a generalized GEMM this shape is all prologue and epilogue for the tile kernel of sim_tiled.cu.  Two kernels instead,
// both preparing the parameters of their templates for themselves (no launch in front):
//
//  * sim_fwd_resident, for enough positions to fill the GPU: a persistent CTA keeps the parameters of 32 or 64 templates in
//    shared memory and streams tiles of 128 patches past them, the next tile being gathered while the current one is
//    multiplied; 4 x 8 outputs per thread, packed arithmetic.
//  * sim_fwd_smallk, for few positions: a thread owns one position with its patch in registers and walks the templates four at
//    a time; the templates are split over CTAs as well.
//
// Bound: the FP32 pipe, 3 lane operations per term (difference, scale, fused multiply-add; a fourth for missing data), the
// same operations as everywhere else, so results equal the tile kernel's up to summation order.  Patches in registers with 2
// or 4 positions per thread had left that pipe half idle whichever way the packed instructions were paired: 8 to 12 chains per
// warp at 12 to 16 warps per SM do not cover the latency of difference -> product -> sum (2048 x 3 x 32 x 32 input, 64
// templates of 3x3: 610 to 636 us).  What the resident kernel spends beside the arithmetic adds to its time: 612 us there with two
// range tests per gathered value, 493 with one test of two bits (332 from registers and shared memory alone).  All five modes of the
// forward functor (include/utils/similarity_utils.hpp:17-60 of the reference) are covered.
#include "kernels.cuh"
#include "tile.cuh"

namespace simnets {

namespace {

constexpr int kSkThreads = 128;
constexpr int kSkSmemBytes = 48 * 1024;
constexpr double kSkLog2Pi = 1.8378770664093454835606594728112;

__device__ __forceinline__ float2 sk_abs2(float2 v) { return make_float2(fabsf(v.x), fabsf(v.y)); }

struct SkColumn { long long base; int n, h0, w0; };

__device__ __forceinline__ SkColumn sk_column(const SimGeo& g, long long j, long long P) {
    SkColumn c;
    c.base = -1; c.n = 0; c.h0 = c.w0 = 0;
    if (j >= P) return c;
    const int n = P <= 0x7fffffffLL ? int(uint32_t(j) / uint32_t(g.N)) : int(j / g.N), pos = int(j - (long long)n * g.N);
    c.n = n;
    c.h0 = (pos / g.ow) * g.sh - g.ph;
    c.w0 = (pos % g.ow) * g.sw - g.pw;
    c.base = (long long)n * g.M * g.N + pos;
    return c;
}

struct SkParams {                               // how the parameters of one (template, tap) enter the arithmetic
    float t, scale, constant;
};
template <int MODE>
__device__ __forceinline__ SkParams sk_params(const SimGeo& g, const float* __restrict__ tm, const float* __restrict__ wt, int m, int k) {
    SkParams p = {0.f, 0.f, 0.f};
    if (m < g.M && k < g.K) {
        const size_t src = (size_t)m * g.K + k;
        const float w = g.absw ? fabsf(wt[src]) : wt[src];
        p.t = tm[src];
        p.scale = MODE == SIM_L2N || MODE == SIM_L2N_NAN ? -0.5f * w : -w;
        if (MODE == SIM_L2N_NAN) p.constant = float(0.5 * (double(logf(w + float(g.fudge))) - kSkLog2Pi));
    }
    return p;
}
// the constant the plain normalised L2 adds once per output of template m
__device__ __forceinline__ float sk_row_constant(const SimGeo& g, const float* __restrict__ wt, int m) {
    float c = 0.f;
    if (m < g.M)
        for (int k = 0; k < g.K; ++k) {
            const float w = wt[(size_t)m * g.K + k];
            c += 0.5f * logf((g.absw ? fabsf(w) : w) + float(g.fudge));
        }
    return c + float(-0.5 * double(g.K) * kSkLog2Pi);
}
__device__ __forceinline__ int2 sk_tap(const SimGeo& g, int k) {        // {offset inside a sample, (kh << 16) | kw}
    const int kw = k % g.bw, kh = (k / g.bw) % g.bh, c = k / (g.bw * g.bh);
    return k < g.K ? make_int2((c * g.H + kh) * g.W + kw, (kh << 16) | kw) : make_int2(0, 0);
}
__device__ __forceinline__ float sk_load(const SimGeo& g, const float* __restrict__ xs, const SkColumn& c, int2 tap, float oob) {
    const bool in = uint32_t(c.h0 + (tap.y >> 16)) < uint32_t(g.H) && uint32_t(c.w0 + (tap.y & 0xffff)) < uint32_t(g.W);
    return in ? __ldg(xs + tap.x) : oob;
}

// KT >= K: the patch length at compile time (the tap loops are fully unrolled, the patch is a register array); taps past K have
// zero parameters.  A CTA works on templates [blockIdx.y * slice, ...): all of them unless the parameters would not fit shared
// memory or the positions alone would not fill the GPU.
template <int MODE, int KT>
__global__ void __launch_bounds__(kSkThreads, 4) sim_fwd_smallk(SimGeo g, int slice, const float* __restrict__ x, const float* __restrict__ tm,
                                                                const float* __restrict__ wt, float* __restrict__ y, float* __restrict__ ch_max,
                                                                float* __restrict__ ch_min, int* __restrict__ flag) {
    stream_order();
    constexpr bool MASKED = MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP;
    constexpr bool L1 = MODE == SIM_L1 || MODE == SIM_L1_SKIP;
    extern __shared__ __align__(16) float sm[];
    const int first = blockIdx.y * slice, M = min(slice, g.M - first), Mq = (M + 3) & ~3;
    float* s_t = sm;                            // [KT][Mq] templates, [KT][Mq] scales, then for the NaN-aware L2 [KT][Mq] constants
    float* s_s = s_t + KT * Mq;
    float* s_c = s_s + KT * Mq;                 // (for the plain normalised L2: [Mq] constants added once per output)
    __shared__ int2 tp[KT];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) flag[threadIdx.x] = 0;          // the workspace's status words
    for (int i = threadIdx.x; i < KT * Mq; i += kSkThreads) {
        const int k = i / Mq, m = i - k * Mq;
        const SkParams p = sk_params<MODE>(g, tm, wt, m < M ? first + m : g.M, k);
        s_t[i] = p.t; s_s[i] = p.scale;
        if (MODE == SIM_L2N_NAN) s_c[i] = p.constant;
    }
    if (MODE == SIM_L2N) for (int m = threadIdx.x; m < Mq; m += kSkThreads) s_c[m] = sk_row_constant(g, wt, first + m);
    for (int k = threadIdx.x; k < KT; k += kSkThreads) tp[k] = sk_tap(g, k);
    __syncthreads();

    const long long P = (long long)g.B * g.N;
    const float oob = float(g.oob);
    const float quirk_c = float(-0.5 * double(g.K) * kSkLog2Pi);
    for (long long j = blockIdx.x * (long long)kSkThreads + threadIdx.x; j < P; j += (long long)gridDim.x * kSkThreads) {
        const SkColumn c = sk_column(g, j, P);
        const float* xs = x + (size_t)c.n * g.C * g.H * g.W + c.h0 * g.W + c.w0;
        float2 nx[KT];                          // the patch, NEGATED (d = t + (-x)), each value in both halves of a pair
        uint32_t mask = 0u;
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            float a = k < g.K ? sk_load(g, xs, c, tp[k], oob) : 0.f;
            if (MASKED) { if (a == a) mask |= 1u << k; else a = 0.f; }
            nx[k] = make_float2(-a, -a);
        }
        // per-pixel extrema over the instances, for a consumer that stabilises a log-sum-exp over them (NaN ignored)
        float vmax = -CUDART_INF_F, vmin = CUDART_INF_F;
        float* dst = y + c.base + (long long)first * g.N;
#pragma unroll 1
        for (int m0 = 0; m0 < Mq; m0 += 4) {
            float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int k = 0; k < KT; ++k) {
                const float4 t4 = *reinterpret_cast<const float4*>(s_t + k * Mq + m0), s4 = *reinterpret_cast<const float4*>(s_s + k * Mq + m0);
                float4 c4 = make_float4(0.f, 0.f, 0.f, 0.f);
                if (MODE == SIM_L2N_NAN) c4 = *reinterpret_cast<const float4*>(s_c + k * Mq + m0);
                const float2 k0 = splat2(MASKED ? ((mask >> k) & 1u ? 1.f : 0.f) : 1.f);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 d = add2(h ? make_float2(t4.z, t4.w) : make_float2(t4.x, t4.y), nx[k]);
                    const float2 sc = h ? make_float2(s4.z, s4.w) : make_float2(s4.x, s4.y);
                    if (!MASKED) acc[h] = L1 ? fma2(sc, sk_abs2(d), acc[h]) : fma2(mul2(sc, d), d, acc[h]);
                    else if (L1) acc[h] = fma2(sc, mul2(sk_abs2(d), k0), acc[h]);
                    else acc[h] = fma2(k0, fma2(mul2(sc, d), d, h ? make_float2(c4.z, c4.w) : make_float2(c4.x, c4.y)), acc[h]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q, dst += g.N) {
                if (m0 + q >= M) break;
                float v = q & 1 ? acc[q >> 1].y : acc[q >> 1].x;
                if (MODE == SIM_L2N) {
                    v += s_c[m0 + q];
                    if (g.batch_quirk) v += quirk_c * float(g.B - 1 - c.n);
                }
                vmax = fmaxf(vmax, v);
                vmin = fminf(vmin, v);
                __stcs(dst, v);
            }
        }
        if (ch_max) ch_max[j] = vmax;
        if (ch_min) ch_min[j] = vmin;
    }
}

// Parameters resident in shared memory, tiles of 128 positions streamed past them: rows = templates (TM per CTA, blockIdx.y
// picks them), columns = positions.
template <int MODE> struct ResidentPlanes {
    static constexpr int NA = MODE == SIM_L2N_NAN ? 3 : 2, NB = (MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP) ? 2 : 1;
};
constexpr int kResMaxK = 32, kResTN = 128;
template <int MODE, int TM>
__host__ __device__ constexpr int resident_smem_floats(int K) { return (ResidentPlanes<MODE>::NA * TM + 2 * ResidentPlanes<MODE>::NB * kResTN) * K; }

template <int MODE, int TM>
__global__ void __launch_bounds__(TM * 4, TM == 64 ? 2 : 4) sim_fwd_resident(SimGeo g, const float* __restrict__ x, const float* __restrict__ tm,
                                                                             const float* __restrict__ wt, float* __restrict__ y,
                                                                             float* __restrict__ ch_max, float* __restrict__ ch_min, int* __restrict__ flag) {
    stream_order();
    constexpr int NA = ResidentPlanes<MODE>::NA, NB = ResidentPlanes<MODE>::NB, T = TM * 4, QSTEP = T / kResTN, PER = kResMaxK / QSTEP, TI = TM / 4;
    constexpr bool L1 = MODE == SIM_L1 || MODE == SIM_L1_SKIP;
    using Cfg = TileCfg<TM, kResTN, 8, 4, 8, 1, 1>;
    static_assert(Cfg::THREADS == T, "4 x 8 outputs per thread");
    extern __shared__ __align__(16) float sm[];
    __shared__ long long col_base[2][kResTN];
    __shared__ float row_const[TM];
    __shared__ int2 tp[kResMaxK];                                  // {byte offset inside a sample, bit kh | bit 16 + kw}, or as sk_tap has it
    __shared__ __align__(16) float red[2][TI][kResTN];             // the extrema of each thread row, two tiles' worth
    const int K = g.K, i0 = blockIdx.y * TM;
    float* As = sm;
    float* Bs = sm + NA * TM * K;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) flag[threadIdx.x] = 0;          // the workspace's status words
    for (int i = threadIdx.x; i < K * TM; i += T) {
        const int k = i / TM, m = i % TM;
        const SkParams p = sk_params<MODE>(g, tm, wt, i0 + m, k);
        As[i] = p.t; As[K * TM + i] = p.scale;
        if (NA == 3) As[2 * K * TM + i] = p.constant;
    }
    if (threadIdx.x < TM) row_const[threadIdx.x] = MODE == SIM_L2N ? sk_row_constant(g, wt, i0 + threadIdx.x) : 0.f;
    // one test of two bits per tap, and an offset that is added as it is (2 % less time than one that is scaled): blocks of up to
    // 16 x 16 and offsets whose bytes 32 bits count.  Else two range tests and offsets in elements.
    const bool bits = g.bh <= 16 && g.bw <= 16 && sim_offsets_below(g, 1LL << 29);
    for (int k = threadIdx.x; k < kResMaxK; k += T) {
        const int2 at = sk_tap(g, k);
        tp[k] = bits ? make_int2(4 * at.x, (1 << (at.y >> 16)) | (0x10000 << (at.y & 0xffff))) : at;
    }
    __syncthreads();

    const TileThread<Cfg> t;
    const long long P = (long long)g.B * g.N, tiles = (P + kResTN - 1) / kResTN;
    const float oob = float(g.oob), quirk_c = float(-0.5 * double(K) * kSkLog2Pi);
    // four consecutive positions of a thread are four consecutive floats of one row of y
    const bool vec = (g.N & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
    const int s_lane = threadIdx.x % kResTN, s_k = threadIdx.x / kResTN;
    float rb[PER];
    long long rbase = -1;
    auto fetch = [&](long long tile) {
        const SkColumn c = sk_column(g, tile * kResTN + s_lane, P);
        const float* xs = x + (size_t)c.n * g.C * g.H * g.W + c.h0 * g.W + c.w0;
        rbase = c.base;
        const float outside = c.base >= 0 ? oob : 0.f;
        if (bits) {
            const int missing = c.base >= 0 ? int(missing_taps(c.h0, g.H) | (missing_taps(c.w0, g.W) << 16)) : -1;
#pragma unroll
            for (int s = 0; s < PER; ++s) {
                const int k = s_k + s * QSTEP;
                if (k >= K) break;
                const int2 t = tp[k];
                rb[s] = outside;
                if ((t.y & missing) == 0) rb[s] = __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(xs) + t.x));
            }
        } else {
#pragma unroll
            for (int s = 0; s < PER; ++s) {
                const int k = s_k + s * QSTEP;
                if (k >= K) break;
                const int2 t = tp[k];
                rb[s] = outside;
                if (c.base >= 0 && uint32_t(c.h0 + (t.y >> 16)) < uint32_t(g.H) && uint32_t(c.w0 + (t.y & 0xffff)) < uint32_t(g.W))
                    rb[s] = __ldg(xs + t.x);
            }
        }
    };
    auto commit = [&](int buf) {
        float* B = Bs + buf * NB * K * kResTN;
        if (s_k == 0) col_base[buf][s_lane] = rbase;
#pragma unroll
        for (int s = 0; s < PER; ++s) {
            const int k = s_k + s * QSTEP;
            if (k >= K) break;
            if (NB == 2) {
                const bool nan = rb[s] != rb[s];
                B[k * kResTN + s_lane] = nan ? 0.f : rb[s];
                B[(K + k) * kResTN + s_lane] = nan ? 0.f : 1.f;
            } else {
                B[k * kResTN + s_lane] = rb[s];
            }
        }
    };
    // per-pixel extrema over the instances, for a consumer that stabilises a log-sum-exp over them (NaN ignored); a tile's are
    // reduced over the thread rows and stored one iteration later, behind the barrier that is there anyway
    const bool extrema = ch_max != nullptr || ch_min != nullptr, up = ch_max != nullptr;       // (only when one tile of rows holds all templates)
    auto store_extrema = [&](long long of_tile, int from) {
        const long long j = of_tile * kResTN + threadIdx.x;
        if (threadIdx.x >= kResTN || j >= P) return;
        float v = red[from][0][threadIdx.x];
#pragma unroll
        for (int i = 1; i < TI; ++i) v = up ? fmaxf(v, red[from][i][threadIdx.x]) : fminf(v, red[from][i][threadIdx.x]);
        (up ? ch_max : ch_min)[j] = v;
    };
    long long tile = blockIdx.x;
    int buf = 0;
    if (tile < tiles) { fetch(tile); commit(0); }
    __syncthreads();
    for (; tile < tiles; tile += gridDim.x, buf ^= 1) {
        const bool more = tile + gridDim.x < tiles;
        if (more) fetch(tile + gridDim.x);
        if (extrema && tile >= gridDim.x) store_extrema(tile - gridDim.x, buf ^ 1);
        float2 acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = make_float2(0.f, 0.f);
        const float* B = Bs + buf * NB * K * kResTN + t.tj * 4;
        const float* A = As + t.ti * 4;
#pragma unroll 9
        for (int q = 0; q < K; ++q) {
            float a[NA][4];
            float2 b[NB][4];
#pragma unroll
            for (int p = 0; p < NA; ++p) {
                const float4 v = *reinterpret_cast<const float4*>(A + (p * K + q) * TM);
                a[p][0] = v.x; a[p][1] = v.y; a[p][2] = v.z; a[p][3] = v.w;
            }
#pragma unroll
            for (int p = 0; p < NB; ++p)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 v = *reinterpret_cast<const float4*>(B + (p * K + q) * kResTN + h * (kResTN / 2));
                    b[p][2 * h] = make_float2(v.x, v.y); b[p][2 * h + 1] = make_float2(v.z, v.w);
                }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float2 d = add2(splat2(a[0][r]), neg2(b[0][c])), s2 = splat2(a[1][r]);
                    if (MODE == SIM_L2N_NAN) acc[r][c] = fma2(b[NB - 1][c], fma2(mul2(s2, d), d, splat2(a[NA - 1][r])), acc[r][c]);
                    else if (MODE == SIM_L1_SKIP) acc[r][c] = fma2(s2, mul2(sk_abs2(d), b[NB - 1][c]), acc[r][c]);
                    else if (L1) acc[r][c] = fma2(s2, sk_abs2(d), acc[r][c]);
                    else acc[r][c] = fma2(mul2(s2, d), d, acc[r][c]);
                }
        }
        // results; rows = templates
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            long long cb[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) cb[u] = col_base[buf][h * (kResTN / 2) + t.tj * 4 + u];
            float ext[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) ext[u] = up ? -CUDART_INF_F : CUDART_INF_F;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int m = i0 + t.row(r);
                if (m >= g.M) break;
                float v[4] = {acc[r][2 * h].x, acc[r][2 * h].y, acc[r][2 * h + 1].x, acc[r][2 * h + 1].y};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (MODE == SIM_L2N) {
                        v[u] += row_const[m - i0];
                        if (g.batch_quirk) v[u] += quirk_c * float(g.B - 1 - int(cb[u] / ((long long)g.M * g.N)));
                    }
                }
                if (extrema) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) ext[u] = up ? fmaxf(ext[u], v[u]) : fminf(ext[u], v[u]);
                }
                float* row = y + (long long)m * g.N;
                if (vec && cb[0] >= 0) {
                    __stcs(reinterpret_cast<float4*>(row + cb[0]), make_float4(v[0], v[1], v[2], v[3]));
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) if (cb[u] >= 0) __stcs(row + cb[u], v[u]);
                }
            }
            if (extrema) *reinterpret_cast<float4*>(&red[buf][t.ti][h * (kResTN / 2) + t.tj * 4]) = make_float4(ext[0], ext[1], ext[2], ext[3]);
        }
        if (more) commit(buf ^ 1);
        __syncthreads();
    }
    if (extrema && tile > blockIdx.x) store_extrema(tile - gridDim.x, buf ^ 1);
}

// The same extrema from a finished output tensor, for the forward kernels that do not produce them on the way
__global__ void __launch_bounds__(256) sim_extrema(long long P, int M, int N, const float* __restrict__ y, float* __restrict__ ch_max, float* __restrict__ ch_min) {
    stream_order();
    for (long long q = blockIdx.x * 256LL + threadIdx.x; q < P; q += (long long)gridDim.x * 256) {
        const long long n = q / N;
        const float* p = y + n * (long long)M * N + (q - n * N);
        float hi = -CUDART_INF_F, lo = CUDART_INF_F;
        for (int m = 0; m < M; ++m) { const float v = __ldg(p + (long long)m * N); hi = fmaxf(hi, v); lo = fminf(lo, v); }
        if (ch_max) ch_max[q] = hi;
        if (ch_min) ch_min[q] = lo;
    }
}

template <int KT>
cudaError_t launch_sk(const SimGeo& g, int slice, const float* x, const float* t, const float* w, float* y, float* ch_max, float* ch_min, int* flag, cudaStream_t s) {
    const long long P = (long long)g.B * g.N, want = (P + kSkThreads - 1) / kSkThreads;
    const int slices = (g.M + slice - 1) / slice;
    const dim3 grid(unsigned(std::min<long long>(want, std::max(1, device_sm_count() * 4 / slices))), unsigned(slices));
    const int rows = (slice + 3) & ~3;
    const size_t smem = sizeof(float) * (KT * rows * (g.mode == SIM_L2N_NAN ? 3 : 2) + (g.mode == SIM_L2N ? rows : 0));
#define SK(MODE) in_stream_order(sim_fwd_smallk<MODE, KT>, grid, kSkThreads, smem, s)(g, slice, x, t, w, y, ch_max, ch_min, flag)
    switch (g.mode) {
    case SIM_L1: SK(SIM_L1); break;
    case SIM_L1_SKIP: SK(SIM_L1_SKIP); break;
    case SIM_L2: SK(SIM_L2); break;
    case SIM_L2N: SK(SIM_L2N); break;
    default: SK(SIM_L2N_NAN); break;
    }
#undef SK
    count_launch();
    return cudaGetLastError();
}

template <int MODE, int TM>
cudaError_t launch_resident(const SimGeo& g, const float* x, const float* t, const float* w, float* y, float* ch_max, float* ch_min, int* flag, cudaStream_t s) {
    static SmemLimit limit;
    const int smem = int(sizeof(float)) * resident_smem_floats<MODE, TM>(g.K);
    const cudaError_t e = limit.raise(sim_fwd_resident<MODE, TM>, int(sizeof(float)) * resident_smem_floats<MODE, TM>(kResMaxK));
    if (e != cudaSuccess) return e;
    const long long tiles = ((long long)g.B * g.N + kResTN - 1) / kResTN;
    const int mtiles = (g.M + TM - 1) / TM, per_sm = std::min(TM == 64 ? 2 : 4, 220 * 1024 / (smem + 2 * (TM / 4) * kResTN * int(sizeof(float)) + 4096));
    const int resident = std::max(1, device_sm_count() * per_sm / mtiles);
    const long long rounds = (tiles + resident - 1) / resident;          // equal rounds: as few CTAs as finish in the same number
    const dim3 grid(unsigned((tiles + rounds - 1) / rounds), unsigned(mtiles));
    in_stream_order(sim_fwd_resident<MODE, TM>, grid, TM * 4, smem, s)(g, x, t, w, y, ch_max, ch_min, flag);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

bool sim_smallk_shape(const SimGeo& g) { return g.K <= kResMaxK; }

cudaError_t launch_sim_fwd_smallk(const SimGeo& g, const float* x, const float* t, const float* w, float* y, float* ch_max, float* ch_min,
                                  bool* extrema_done, int* flag, cudaStream_t s) {
    const long long P = (long long)g.B * g.N;
    const int sms = device_sm_count();
    // rows of 32 or 64 templates, whichever pads less; the streaming kernel wherever its tiles give every SM two CTAs' worth
    const int tm = (g.M + 63) / 64 * 64 <= (g.M + 31) / 32 * 32 ? 64 : 32, mtiles = (g.M + tm - 1) / tm;
    if ((P / kResTN) * mtiles * (tm / 32) >= 4LL * sms) {
        *extrema_done = mtiles == 1 && (ch_max == nullptr || ch_min == nullptr);
        if (!*extrema_done) ch_max = ch_min = nullptr;
#define RES(MODE) return tm == 64 ? launch_resident<MODE, 64>(g, x, t, w, y, ch_max, ch_min, flag, s) : launch_resident<MODE, 32>(g, x, t, w, y, ch_max, ch_min, flag, s)
        switch (g.mode) {
        case SIM_L1: RES(SIM_L1);
        case SIM_L1_SKIP: RES(SIM_L1_SKIP);
        case SIM_L2: RES(SIM_L2);
        case SIM_L2N: RES(SIM_L2N);
        default: RES(SIM_L2N_NAN);
        }
#undef RES
    }
    const int kt = g.K <= 4 ? 4 : g.K <= 9 ? 9 : g.K <= 12 ? 12 : g.K <= 16 ? 16 : g.K <= 20 ? 20 : g.K <= 27 ? 27 : 32;
    // templates per CTA: as many as the parameters leave room for, in equal slices; more slices while positions alone give
    // fewer than two CTAs per SM (the extrema need all templates in one CTA)
    const int per = (g.mode == SIM_L2N_NAN ? 3 : 2) * kt * int(sizeof(float)), most = (kSkSmemBytes / (per + int(sizeof(float)))) & ~3;
    int slices = (g.M + most - 1) / most;
    if (ch_max == nullptr && ch_min == nullptr) {
        const long long ctas = (P + kSkThreads - 1) / kSkThreads;
        if (ctas < 2 * sms) slices = std::max<int>(slices, int(std::min<long long>((2 * sms + ctas - 1) / ctas, (g.M + 7) / 8)));
    }
    const int slice = ((g.M + slices - 1) / slices + 3) & ~3;
    *extrema_done = slice >= g.M;
    if (!*extrema_done) ch_max = ch_min = nullptr;
    switch (kt) {
    case 4: return launch_sk<4>(g, slice, x, t, w, y, ch_max, ch_min, flag, s);
    case 9: return launch_sk<9>(g, slice, x, t, w, y, ch_max, ch_min, flag, s);
    case 12: return launch_sk<12>(g, slice, x, t, w, y, ch_max, ch_min, flag, s);
    case 16: return launch_sk<16>(g, slice, x, t, w, y, ch_max, ch_min, flag, s);
    case 20: return launch_sk<20>(g, slice, x, t, w, y, ch_max, ch_min, flag, s);
    case 27: return launch_sk<27>(g, slice, x, t, w, y, ch_max, ch_min, flag, s);
    default: return launch_sk<32>(g, slice, x, t, w, y, ch_max, ch_min, flag, s);
    }
}

cudaError_t launch_sim_extrema(const SimGeo& g, const float* y, float* ch_max, float* ch_min, cudaStream_t s) {
    const long long P = (long long)g.B * g.N;
    if (P == 0 || (ch_max == nullptr && ch_min == nullptr)) return cudaSuccess;
    in_stream_order(sim_extrema, int(std::min<long long>((P + 255) / 256, (long long)device_sm_count() * 16)), 256, 0, s)(P, g.M, g.N, y, ch_max, ch_min);
    count_launch();
    return cudaGetLastError();
}

}  // namespace simnets
