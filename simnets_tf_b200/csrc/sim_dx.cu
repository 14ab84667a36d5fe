// Similarity input gradient (float32).
//
//     dx[n, c, h, w] = sum over the taps (kh, kw) whose patch covers the pixel and over m of  s w dy (t - x)    (L1: sign(t - x))
//
// with s = 2 for plain L2: a generalized GEMM with rows c, columns = pixels and q = (kh, kw, m) as the reduction index.  The
// reference's column gradient followed by col2im (HUJI-Deep/simnets-tf src/kernels/similarity_grad_kernel_cpu.cpp:205-268)
// becomes one gather, nothing is scattered.
//
// With strides a pixel only meets the taps of its own phase, (h + pad) mod stride = kh mod stride: the grid's y index is the
// phase, and a CTA walks the taps of that phase only (a 5x3 block at stride 2x1 would otherwise spend half its terms on dy
// values that are zero by construction).  The (tap, m) cursor of every staging thread advances by additions; dividing the
// reduction index by M for each staged value had taken as many instructions as the terms themselves (256 x 64 x 32 x 32 input,
// 256 templates of 3x3: 10.2 ms).
//
// NaN pixels give 0 in the ignore_nan_input modes, and so does a pixel that no patch covers in every mode.  A tap that the
// padding cuts off, or a step past the last one, contributes 0 * (t - x), which is NaN for an infinite x (or an infinite
// parameter): a sum that came out NaN over a number is added up again over the taps that are there (dx_redo; the test costs 1.5 %
// where 64 rows of channels share a tile: 128 x 64 x 32 x 32 input, 128 templates of 3x3, 1231 -> 1243 us, with kDxFold).
#include "kernels.cuh"
#include "sim_exact.cuh"
#include "tile.cuh"

namespace simnets {
namespace {

__host__ __device__ inline int dx_pad4(int v) { return (v + 3) & ~3; }
// sign of d, 0 for 0 and NaN as in the reference
__device__ __forceinline__ float dx_sign(float d) { return fabsf(d) > 0.f ? __uint_as_float(0x3f800000u | (__float_as_uint(d) & 0x80000000u)) : 0.f; }

// The pixels and taps of one phase along one axis: pixels first, first + stride, ... (n of them), taps r, r + stride, ... (taps
// of them); pixel i meets tap a at output i + shift - a.
struct Axis { int first, n, taps, shift; };
__host__ __device__ inline Axis dx_axis(int size, int block, int stride, int pad, int r) {
    Axis x;
    x.first = ((r - pad) % stride + stride) % stride;
    x.n = x.first < size ? (size - x.first + stride - 1) / stride : 0;
    x.taps = r < block ? (block - r + stride - 1) / stride : 0;
    x.shift = (x.first + pad - r) / stride;
    return x;
}

struct DxPhase {
    int rh, rw;
    Axis h, w;
    __device__ DxPhase(const SimGeo& g, int phase) {
        rh = phase / g.sw; rw = phase - rh * g.sw;
        h = dx_axis(g.H, g.bh, g.sh, g.ph, rh);
        w = dx_axis(g.W, g.bw, g.sw, g.pw, rw);
    }
};

// One pixel: where it lies, and where its output positions lie for tap (0, 0) of the phase.
struct DxPixel {
    long long base;          // offset of x[n, 0, h, w], or -1 past the end
    int n, ho, wo;
    __device__ DxPixel() {}
    __device__ DxPixel(const SimGeo& g, const DxPhase& ph, long long j) : base(-1), n(0), ho(0), wo(0) {
        const int hw = ph.h.n * ph.w.n;
        if (j >= (long long)g.B * hw) return;
        n = j <= 0x7fffffffLL ? int(uint32_t(j) / uint32_t(hw)) : int(j / hw);
        const int p = int(j - (long long)n * hw), i = p / ph.w.n, k = p - i * ph.w.n;
        ho = i + ph.h.shift; wo = k + ph.w.shift;
        base = (long long)n * g.C * g.H * g.W + (ph.h.first + i * g.sh) * g.W + ph.w.first + k * g.sw;
    }
    // offset of dy[n, 0, position met by tap (a, b)], or -1
    __device__ long long at(const SimGeo& g, int a, int b) const {
        const int h = ho - a, w = wo - b;
        return (base >= 0 && uint32_t(h) < uint32_t(g.oh) && uint32_t(w) < uint32_t(g.ow)) ? (long long)n * g.M * g.N + h * g.ow + w : -1;
    }
    __device__ bool covered(const SimGeo& g, const DxPhase& ph) const {
        return max(0, ho - g.oh + 1) <= min(ph.h.taps - 1, ho) && max(0, wo - g.ow + 1) <= min(ph.w.taps - 1, wo);
    }
};

// The value at dx[at] again, term by term, if it is NaN and x[at] is not.
__device__ __noinline__ void dx_redo(const SimGeo& g, const float* __restrict__ x, const float* __restrict__ tm, const float* __restrict__ wt,
                                     const float* __restrict__ dy, float* dx, long long at) {
    if (is_nan(dx[at]) && !is_nan(x[at])) dx[at] = sim_exact_dx(g, x, tm, wt, dy, at);
}

// (t, s w)[tap][m][Cp], channel-contiguous, for the tile kernel
__global__ void __launch_bounds__(256) sim_dx_prep(SimGeo g, const float* __restrict__ tm, const float* __restrict__ wt, float* __restrict__ dxp) {
    stream_order();
    const int taps = g.bh * g.bw, cp = dx_pad4(g.C);
    const long long total = (long long)taps * g.M * cp;
    const float s = g.mode == SIM_L2 ? 2.f : 1.f;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const int c = int(i % cp);
        const long long q = i / cp;
        const int m = int(q % g.M), tap = int(q / g.M);
        const size_t src = ((size_t)m * g.C + c) * taps + tap;
        const float w = c < g.C ? wt[src] : 0.f;
        dxp[i] = c < g.C ? tm[src] : 0.f;
        dxp[total + i] = s * (g.absw ? fabsf(w) : w);
    }
}

// Steps after which a sum is set aside (a private slot in shared memory) and begins again: a sum of M bh bw terms in one register
// is several times farther from the exact one than the reference's, which adds the taps' sums over m (256 templates of 5x5: 1.4e-6
// of the gradient's norm against 3e-7).
constexpr int kDxFold = 256;

template <int TM> struct DxCfg {
    static constexpr int RM = TM == 128 ? 8 : 4, TN = TM == 16 ? 256 : 128;
    using Cfg = TileCfg<TM, TN, 8, RM, 8, 2, 1>;
    static constexpr int SLOT_BYTES = 4 * RM * 8 * Cfg::THREADS;
};

template <int TM, int MODE>
__global__ void __launch_bounds__(DxCfg<TM>::Cfg::THREADS, DxCfg<TM>::Cfg::THREADS == 256 ? (TM == 128 ? 1 : 2) : 3)
sim_dx_tiled(const __grid_constant__ SimGeo g, const float* __restrict__ x, const float* __restrict__ dxp, const float* __restrict__ tm, const float* __restrict__ wt,
             const float* __restrict__ dy, float* __restrict__ dx) {
    stream_order();
    constexpr bool L1 = MODE == SIM_L1 || MODE == SIM_L1_SKIP;
    constexpr bool SKIP_NAN = MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP;
    using Cfg = typename DxCfg<TM>::Cfg;
    constexpr int T = Cfg::THREADS, COLS = Cfg::TN > T ? Cfg::TN / T : 1, QSTEP = T > Cfg::TN ? T / Cfg::TN : 1, QPER = Cfg::KC / QSTEP;
    constexpr int VEC = TM / 4, APER = (2 * Cfg::KC * VEC + T - 1) / T;
    __shared__ __align__(16) float smem[Cfg::SMEM_FLOATS];
    extern __shared__ __align__(16) float2 slots[];                     // [RM x RN / 2][THREADS], if the launch has sums of more than kDxFold steps
    __shared__ long long col_base[Cfg::TN];
    __shared__ unsigned char col_covered[Cfg::TN];
    const DxPhase ph(g, blockIdx.y);
    const int ctiles = (g.C + TM - 1) / TM;
    const int ct = blockIdx.x % ctiles;
    const long long j0 = (long long)(blockIdx.x / ctiles) * Cfg::TN;
    if (j0 >= (long long)g.B * ph.h.n * ph.w.n) return;
    const int i0 = ct * TM;
    const int Q = ph.h.taps * ph.w.taps * g.M, ldc = dx_pad4(g.C);
    const size_t plane = (size_t)g.bh * g.bw * g.M * ldc;
    const TileThread<Cfg> t;

    // dy staging: columns s_lane (+ T), steps s_k, s_k + QSTEP, ... of every chunk; the cursor (tap a, b and m) moves along
    const int s_lane = threadIdx.x % Cfg::TN, s_k = threadIdx.x / Cfg::TN;
    DxPixel px[COLS];
    long long at[COLS];
    int ca = 0, cb_ = 0, cm = s_k;
    float rb[COLS][QPER];
#pragma unroll
    for (int u = 0; u < COLS; ++u) {
        px[u] = DxPixel(g, ph, j0 + s_lane + u * T);
        col_base[s_lane + u * T] = px[u].base;
        col_covered[s_lane + u * T] = px[u].covered(g, ph);
    }
    auto locate = [&]() {
        while (cm >= g.M) { cm -= g.M; if (++cb_ == ph.w.taps) { cb_ = 0; ++ca; } }
#pragma unroll
        for (int u = 0; u < COLS; ++u) {
            const long long o = ca < ph.h.taps ? px[u].at(g, ca, cb_) : -1;
            at[u] = o < 0 ? -1 : o + (long long)cm * g.N;
        }
    };
    if (Q > 0) locate();
    const size_t step = (size_t)QSTEP * g.N;
    auto fetchB = [&](int, float*) {
#pragma unroll
        for (int s = 0; s < QPER; ++s) {
#pragma unroll
            for (int u = 0; u < COLS; ++u) {
                rb[u][s] = 0.f;
                if (at[u] >= 0) { rb[u][s] = __ldg(dy + at[u]); at[u] += step; }
            }
            cm += QSTEP;
            if (cm >= g.M) locate();
        }
    };
    auto commitB = [&](float* Bs) {
#pragma unroll
        for (int s = 0; s < QPER; ++s)
#pragma unroll
            for (int u = 0; u < COLS; ++u) Bs[(s_k + s * QSTEP) * Cfg::TN + s_lane + u * T] = rb[u][s];
    };
    // parameter staging: APER 16-byte copies per thread and chunk, each with a cursor of its own
    int aa[APER], ab[APER], am[APER];
#pragma unroll
    for (int v = 0; v < APER; ++v) { aa[v] = ab[v] = 0; am[v] = ((threadIdx.x + v * T) % (Cfg::KC * VEC)) / VEC; }
    auto fetchA = [&](int, float* As) {
#pragma unroll
        for (int v = 0; v < APER; ++v) {
            const int idx = threadIdx.x + v * T;
            if (idx < 2 * Cfg::KC * VEC) {
                const int p = idx / (Cfg::KC * VEC), row = (idx % (Cfg::KC * VEC)) / VEC, e = (idx % VEC) * 4;
                while (am[v] >= g.M) { am[v] -= g.M; if (++ab[v] == ph.w.taps) { ab[v] = 0; ++aa[v]; } }
                const int left = aa[v] < ph.h.taps ? g.C - (i0 + e) : 0;          // (rows of dxp are padded to a multiple of four channels)
                const int tap = (ph.rh + aa[v] * g.sh) * g.bw + ph.rw + ab[v] * g.sw;
                cp_async16(As + (p * Cfg::KC + row) * TM + e, left > 0 ? dxp + p * plane + ((size_t)tap * g.M + am[v]) * ldc + i0 + e : dxp, left > 0 ? 16 : 0);
                am[v] += Cfg::KC;
            }
        }
    };
    auto commitA = [&](float*) { cp_async_wait_all(); };

    // this thread's own x values (one per output)
    __syncthreads();
    float2 xx[Cfg::RM][Cfg::RN / 2], acc[Cfg::RM][Cfg::RN / 2];
    const size_t chw = (size_t)g.H * g.W;
#pragma unroll
    for (int r_ = 0; r_ < Cfg::RM; ++r_) {
        const int c = i0 + t.row(r_);
#pragma unroll
        for (int c_ = 0; c_ < Cfg::RN; ++c_) {
            const long long cb = col_base[t.col(c_)];
            const float v = (c < g.C && cb >= 0) ? __ldg(x + cb + (size_t)c * chw) : 0.f;
            if (c_ & 1) xx[r_][c_ >> 1].y = -v; else xx[r_][c_ >> 1].x = -v;
            acc[r_][c_ >> 1] = make_float2(0.f, 0.f);
        }
    }
    auto comb = [&](int r_, int cp, const float2 (&a)[2], const float2 (&b)[1]) {
        const float2 d = add2(a[0], xx[r_][cp]);
        const float2 e = mul2(a[1], b[0]);
        acc[r_][cp] = fma2(e, L1 ? make_float2(dx_sign(d.x), dx_sign(d.y)) : d, acc[r_][cp]);
    };
    const int chunks = (Q + Cfg::KC - 1) / Cfg::KC;
    auto fold = [&](int c) {
        const bool first = c == kDxFold / Cfg::KC;
#pragma unroll
        for (int i = 0; i < Cfg::RM * Cfg::RN / 2; ++i) {
            float2& a = acc[i / (Cfg::RN / 2)][i % (Cfg::RN / 2)];
            slots[i * T + threadIdx.x] = first ? a : add2(slots[i * T + threadIdx.x], a);
            a = make_float2(0.f, 0.f);
        }
    };
    tile_mainloop<Cfg, false, false, kDxFold / Cfg::KC>(smem, chunks, t, fetchA, fetchB, commitA, commitB, comb, fold);
    if (Q > kDxFold)
#pragma unroll
        for (int i = 0; i < Cfg::RM * Cfg::RN / 2; ++i) {
            float2& a = acc[i / (Cfg::RN / 2)][i % (Cfg::RN / 2)];
            a = add2(slots[i * T + threadIdx.x], a);
        }

    bool redo = false;
#pragma unroll
    for (int c_ = 0; c_ < Cfg::RN; ++c_) {
        const long long cb = col_base[t.col(c_)];
        if (cb < 0) continue;
        const bool covered = col_covered[t.col(c_)];
#pragma unroll
        for (int r_ = 0; r_ < Cfg::RM; ++r_) {
            const int c = i0 + t.row(r_);
            if (c >= g.C) continue;
            float v = (c_ & 1) ? acc[r_][c_ >> 1].y : acc[r_][c_ >> 1].x;
            const float xv = (c_ & 1) ? xx[r_][c_ >> 1].y : xx[r_][c_ >> 1].x;
            if (!covered || (SKIP_NAN && xv != xv)) v = 0.f;
            redo |= is_nan(v);
            dx[cb + (size_t)c * chw] = v;
        }
    }
    if (redo)
#pragma unroll 1
        for (int i = 0; i < Cfg::RM * Cfg::RN; ++i) {
            const int c = i0 + t.row(i / Cfg::RN);
            const long long cb = col_base[t.col(i % Cfg::RN)];
            if (c < g.C && cb >= 0) dx_redo(g, x, tm, wt, dy, dx, cb + (long long)(c * chw));
        }
}

// Few channels (an image's): a thread owns PP pixels with all CT >= C channels of each, so that a dy value is read once per
// (tap, m) and serves every channel; the parameters of 64 (tap, m) pairs at a time sit in shared memory, where a warp reads
// one address.  A tile kernel would multiply mostly padding rows here (3 of 16).
constexpr int kNarrowThreads = 128, kNarrowQ = 64;

template <int CT, int PP, int MODE>
__global__ void __launch_bounds__(kNarrowThreads) sim_dx_narrow(const __grid_constant__ SimGeo g, const float* __restrict__ x, const float* __restrict__ tm,
                                                                const float* __restrict__ wt, const float* __restrict__ dy, float* __restrict__ dx) {
    stream_order();
    constexpr bool L1 = MODE == SIM_L1 || MODE == SIM_L1_SKIP;
    constexpr bool SKIP_NAN = MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP;
    __shared__ __align__(16) float s_t[kNarrowQ * CT], s_w[kNarrowQ * CT];
    __shared__ float slots[PP * CT][kNarrowThreads];                    // sums set aside, see kDxFold
    const DxPhase ph(g, blockIdx.y);
    const long long j0 = (long long)blockIdx.x * (kNarrowThreads * PP);
    if (j0 >= (long long)g.B * ph.h.n * ph.w.n) return;
    const int taps = g.bh * g.bw;
    const size_t chw = (size_t)g.H * g.W;
    const float scale = MODE == SIM_L2 ? 2.f : 1.f;
    float xv[PP][CT], acc[PP][CT];
    DxPixel px[PP];
#pragma unroll
    for (int p = 0; p < PP; ++p) {
        px[p] = DxPixel(g, ph, j0 + threadIdx.x + p * kNarrowThreads);
#pragma unroll
        for (int c = 0; c < CT; ++c) { xv[p][c] = (px[p].base >= 0 && c < g.C) ? __ldg(x + px[p].base + c * chw) : 0.f; acc[p][c] = 0.f; }
    }
    int steps = 0;
    bool aside = false;
    for (int a = 0; a < ph.h.taps; ++a)
        for (int b = 0; b < ph.w.taps; ++b) {
            const int tap = (ph.rh + a * g.sh) * g.bw + ph.rw + b * g.sw;
            long long at[PP];
#pragma unroll
            for (int p = 0; p < PP; ++p) at[p] = px[p].at(g, a, b);
            for (int m0 = 0; m0 < g.M; m0 += kNarrowQ) {
                const int nm = min(kNarrowQ, g.M - m0);
                if ((steps += nm) > kDxFold) {
#pragma unroll
                    for (int p = 0; p < PP; ++p)
#pragma unroll
                        for (int c = 0; c < CT; ++c) {
                            float& s = slots[p * CT + c][threadIdx.x];
                            s = aside ? s + acc[p][c] : acc[p][c];
                            acc[p][c] = 0.f;
                        }
                    steps = nm;
                    aside = true;
                }
                __syncthreads();
                for (int i = threadIdx.x; i < nm * CT; i += kNarrowThreads) {
                    const int c = i % CT, m = m0 + i / CT;
                    const size_t src = ((size_t)m * g.C + c) * taps + tap;
                    const float w = c < g.C ? __ldg(wt + src) : 0.f;
                    s_t[i] = c < g.C ? __ldg(tm + src) : 0.f;
                    s_w[i] = scale * (g.absw ? fabsf(w) : w);
                }
                __syncthreads();
#pragma unroll 4
                for (int m = 0; m < nm; ++m) {
                    float v[PP];
#pragma unroll
                    for (int p = 0; p < PP; ++p) v[p] = at[p] >= 0 ? __ldg(dy + at[p] + (size_t)(m0 + m) * g.N) : 0.f;
#pragma unroll
                    for (int c = 0; c < CT; ++c) {
                        const float tc = s_t[m * CT + c], wc = s_w[m * CT + c];
#pragma unroll
                        for (int p = 0; p < PP; ++p) {
                            const float d = tc - xv[p][c];
                            acc[p][c] = fmaf(wc * v[p], L1 ? dx_sign(d) : d, acc[p][c]);
                        }
                    }
                }
            }
        }
    if (aside)
#pragma unroll
        for (int p = 0; p < PP; ++p)
#pragma unroll
            for (int c = 0; c < CT; ++c) acc[p][c] += slots[p * CT + c][threadIdx.x];
#pragma unroll
    for (int p = 0; p < PP; ++p) {
        if (px[p].base < 0) continue;
        const bool covered = px[p].covered(g, ph);
        bool redo = false;
#pragma unroll
        for (int c = 0; c < CT; ++c)
            if (c < g.C) {
                const float v = (!covered || (SKIP_NAN && is_nan(xv[p][c]))) ? 0.f : acc[p][c];
                redo |= is_nan(v);
                dx[px[p].base + c * chw] = v;
            }
        if (redo)
#pragma unroll 1
            for (int c = 0; c < g.C; ++c) dx_redo(g, x, tm, wt, dy, dx, px[p].base + (long long)(c * chw));
    }
}

}  // namespace

size_t sim_dx_scratch_floats(const SimGeo& g) { return g.C <= 8 ? 0 : 2 * (size_t)g.bh * g.bw * g.M * dx_pad4(g.C); }

cudaError_t launch_sim_dx(const SimGeo& g, const float* x, const float* t, const float* w, const float* dy, float* dx, float* dxp, cudaStream_t s) {
    const int phases = g.sh * g.sw;
    const Axis h = dx_axis(g.H, g.bh, g.sh, g.ph, g.ph % g.sh), v = dx_axis(g.W, g.bw, g.sw, g.pw, g.pw % g.sw);      // the phase of pixel 0 has the most pixels
    const long long pixels = (long long)g.B * h.n * v.n;
#define DX_MODES(RUN)                            \
    switch (g.mode) {                            \
    case SIM_L1: RUN(SIM_L1); break;             \
    case SIM_L1_SKIP: RUN(SIM_L1_SKIP); break;   \
    case SIM_L2: RUN(SIM_L2); break;             \
    case SIM_L2N: RUN(SIM_L2N); break;           \
    default: RUN(SIM_L2N_NAN); break;            \
    }
    if (phases > 65535) return launch_sim_dx_direct(g, false, x, t, w, dy, dx, s);
    if (g.C <= 8) {
        // four pixels per thread where that still fills the GPU twice over, else one
        const bool many = pixels >= (long long)device_sm_count() * 4096;
        const long long per = kNarrowThreads * (many ? 4 : 1), blocks = (pixels + per - 1) / per;
        if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
        const dim3 grid{unsigned(blocks), unsigned(phases)};
#define NARROW(CT, MODE)                                                                                          \
    do {                                                                                                          \
        if (many) in_stream_order(sim_dx_narrow<CT, 4, MODE>, grid, kNarrowThreads, 0, s)(g, x, t, w, dy, dx);                  \
        else in_stream_order(sim_dx_narrow<CT, 1, MODE>, grid, kNarrowThreads, 0, s)(g, x, t, w, dy, dx);                       \
    } while (0)
#define NARROW_1(MODE) NARROW(1, MODE)
#define NARROW_2(MODE) NARROW(2, MODE)
#define NARROW_4(MODE) NARROW(4, MODE)
#define NARROW_8(MODE) NARROW(8, MODE)
        if (g.C == 1) { DX_MODES(NARROW_1) } else if (g.C == 2) { DX_MODES(NARROW_2) } else if (g.C <= 4) { DX_MODES(NARROW_4) } else { DX_MODES(NARROW_8) }
        count_launch();
        return cudaGetLastError();
    }
    const long long total = (long long)g.bh * g.bw * g.M * dx_pad4(g.C);
    in_stream_order(sim_dx_prep, int(std::min<long long>((total + 255) / 256, (long long)device_sm_count() * 8)), 256, 0, s)(g, t, w, dxp);
    // the tile height that pads the channels least; of two equal ones the taller (its dy values serve more rows)
    const auto padded = [&](int tm) { return (g.C + tm - 1) / tm * tm; };
    int tm = 128;
    for (int c : {64, 32, 16}) if (padded(c) < padded(tm)) tm = c;
    if (tm == 128 && g.C <= 64) tm = 64;
    const int tn = tm == 16 ? 256 : 128;
    const long long blocks = ((pixels + tn - 1) / tn) * ((g.C + tm - 1) / tm);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const dim3 grid{unsigned(blocks), unsigned(phases)};
    const bool folds = (long long)((g.bh + g.sh - 1) / g.sh) * ((g.bw + g.sw - 1) / g.sw) * g.M > kDxFold;         // (the most taps of a phase)
#define DX(TM, MODE)                                                                                                                          \
    do {                                                                                                                                      \
        static SmemLimit limit;                                                                                                               \
        const cudaError_t e = limit.raise(sim_dx_tiled<TM, MODE>, DxCfg<TM>::SLOT_BYTES);                                                     \
        if (e != cudaSuccess) return e;                                                                                                       \
        in_stream_order(sim_dx_tiled<TM, MODE>, grid, DxCfg<TM>::Cfg::THREADS, folds ? DxCfg<TM>::SLOT_BYTES : 0, s)(g, x, dxp, t, w, dy, dx); \
    } while (0)
#define DX_16(MODE) DX(16, MODE)
#define DX_32(MODE) DX(32, MODE)
#define DX_64(MODE) DX(64, MODE)
#define DX_128(MODE) DX(128, MODE)
    if (tm == 16) { DX_MODES(DX_16) } else if (tm == 32) { DX_MODES(DX_32) } else if (tm == 64) { DX_MODES(DX_64) } else { DX_MODES(DX_128) }
    count_launch(2);
    return cudaGetLastError();
#undef DX
#undef DX_MODES
}

}  // namespace simnets
