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
// values that are zero by construction).
//
// Bound: the FP32 pipe, 3 packed operations per term, which every other instruction holds up.  A thread of 4, 5 or 6 channels x 8
// pixels takes 10 T terms/s from registers and shared memory, so the tile's rows follow the channels (16, 20, 24, 32, 40, 48 or 64 of
// them; 19 channels in 32 rows had spent 41 % on padding), and a chunk is instances of ONE tap: its operands advance by one addition
// each, where a cursor per staged value had cost several instructions.  256 x 64 x 32 x 32 input, 256 templates of 3x3: 4981 -> 4237 us
// (62 -> 74 % of the pipe); 37 x 19 x 45 x 37, 100 of 5x3 at stride 2 and 1, L1:
// 490 -> 276; 64 x 24 x 30 x 31, 90 of 3x3: 308 -> 203.  L1 adds e with the sign of d put on it, and 0 e (NaN for an e that is no finite
// number) where d is 0 or NaN: 256 templates of 3x3 over 256 x 64 x 32 x 32 6366 us, 8011 when a sign is multiplied by e.
//
// NaN pixels give 0 in the ignore_nan_input modes, and so does a pixel that no patch covers in every mode.  A tap that the
// padding cuts off, or a step past the last one, contributes 0 * (t - x), which is NaN for an infinite x (or an infinite
// parameter): a sum that came out NaN over a number is added up again over the taps that are there (dx_redo; the test costs 1.5 %
// where 64 rows of channels share a tile: 128 x 64 x 32 x 32 input, 128 templates of 3x3, 1231 -> 1243 us, with kDxFold).
#include <cmath>
#include "kernels.cuh"
#include "sim_exact.cuh"
#include "tile.cuh"

namespace simnets {
namespace {

// sign of d, 0 for 0 and NaN as in the reference
__device__ __forceinline__ float dx_sign(float d) { return fabsf(d) > 0.f ? __uint_as_float(0x3f800000u | (__float_as_uint(d) & 0x80000000u)) : 0.f; }

// e sign(d); e0 = 0 e, which is NaN where e is no finite number
__device__ __forceinline__ float dx_signed(float e, float e0, float d) { return fabsf(d) > 0.f ? __uint_as_float(__float_as_uint(e) ^ (__float_as_uint(d) & 0x80000000u)) : e0; }

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

// The tile: 4 WI x 16 threads of RM channels x 8 pixels each, KC steps per chunk.  A thread's channels are one or two 16-byte vectors
// of a row of parameters, so rows of five or six channels per thread are stored in slots of eight.  Sixteen steps per chunk where a
// thread then stages eight values of dy; the narrower tiles would hold sixteen or thirty-two (96 channels of 48-row tiles: 15 % slower).
template <int RM, int WI> struct DxTile {
    static constexpr int SLOT = RM == 4 ? 4 : 8, TM = 4 * WI * RM, ROW = 4 * WI * SLOT, TN = 128, T = 64 * WI, KC = WI == 4 ? 16 : 8;
    static constexpr int COLS = T < TN ? TN / T : 1, QSTEP = T > TN ? T / TN : 1, QPER = KC / QSTEP, A_COPIES = 2 * KC * ROW / 4;
    static constexpr int STAGE = 2 * KC * ROW + KC * TN, SLOT_BYTES = 4 * RM * 8 * T, PER_SM = WI == 4 ? 2 : (WI == 2 ? (RM == 4 ? 4 : 3) : (RM == 6 ? 5 : 6));
};

// (t, s w)[tap][m][channel tile][slots], for the tile kernel
__global__ void __launch_bounds__(256) sim_dx_prep(SimGeo g, int rm, int slot, int rows, int tiles, const float* __restrict__ tm, const float* __restrict__ wt,
                                                   float* __restrict__ dxp) {
    stream_order();
    const int taps = g.bh * g.bw, row = tiles * rows * slot;             // (rows: of threads per tile)
    const long long total = (long long)taps * g.M * row;
    const float s = g.mode == SIM_L2 ? 2.f : 1.f;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const long long q = i / row;
        const int e = int(i - q * row), r = e % slot, c = r < rm ? e / slot * rm + r : g.C;
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

// FEW: of a few templates, whose chunks of one tap would be mostly padding, a chunk is KC steps (tap, m) of whichever taps they belong to, each
// staged with a cursor of its own.
template <int RM, int WI, int MODE, bool FEW>
__global__ void __launch_bounds__(DxTile<RM, WI>::T, DxTile<RM, WI>::PER_SM)
sim_dx_tiled(const __grid_constant__ SimGeo g, const float* __restrict__ x, const float* __restrict__ dxp, const float* __restrict__ tm, const float* __restrict__ wt,
             const float* __restrict__ dy, float* __restrict__ dx) {
    stream_order();
    constexpr bool L1 = MODE == SIM_L1 || MODE == SIM_L1_SKIP;
    constexpr bool SKIP_NAN = MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP;
    using Tile = DxTile<RM, WI>;
    constexpr int T = Tile::T, TN = Tile::TN, TM = Tile::TM, ROW = Tile::ROW, SLOT = Tile::SLOT, KC = Tile::KC, COLS = Tile::COLS, QSTEP = Tile::QSTEP, QPER = Tile::QPER;
    constexpr int PLANE = KC * ROW, A_PER = (Tile::A_COPIES + T - 1) / T;
    __shared__ __align__(16) float smem[2 * Tile::STAGE];
    extern __shared__ __align__(16) float2 slots[];                     // [4 RM][T], if the launch has sums of more than kDxFold steps
    __shared__ long long col_base[TN];
    __shared__ unsigned char col_covered[TN];
    const DxPhase ph(g, blockIdx.y);
    const int ctiles = (g.C + TM - 1) / TM;
    const int ct = blockIdx.x % ctiles;
    const long long j0 = (long long)(blockIdx.x / ctiles) * TN;
    if (j0 >= (long long)g.B * ph.h.n * ph.w.n) return;
    const int i0 = ct * TM;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // 4 x 8 threads per warp, rows interleaved in pairs as in tile.cuh; columns tj * 4 .. + 3 of either half of the tile
    const int ti = (warp % WI) * 4 + (((lane >> 4) << 1) | (lane & 1)), tj = (warp / WI) * 8 + ((lane & 15) >> 1);
    const auto col = [&](int c) { return (c >> 2) * (TN / 2) + tj * 4 + (c & 3); };

    // A chunk is KC instances of one tap (fewer at the end of a tap).  The next chunk to be staged: tap (a, b) of the phase, instances
    // from m_next on.  This thread brings dy of columns s_lane (+ T), instances s_k, s_k + QSTEP, ...
    const int s_lane = threadIdx.x % TN, s_k = threadIdx.x / TN, chunks_per_tap = (g.M + KC - 1) / KC;
    const int Q = ph.h.taps * ph.w.taps * g.M, chunks = FEW ? (Q + KC - 1) / KC : ph.h.taps * ph.w.taps * chunks_per_tap;
    int a = 0, b = 0, m_next = FEW ? s_k : 0, row_next = 0;              // row_next: first row of the chunk in dxp; FEW: first step, and m_next this thread's
    DxPixel px[COLS];
    const float* at[COLS];
    bool ok[COLS];
#pragma unroll
    for (int u = 0; u < COLS; ++u) {
        px[u] = DxPixel(g, ph, j0 + s_lane + u * T);
        col_base[s_lane + u * T] = px[u].base;
        col_covered[s_lane + u * T] = px[u].covered(g, ph);
    }
    auto locate = [&]() {
        if (FEW)
            while (m_next >= g.M) { m_next -= g.M; if (++b == ph.w.taps) { b = 0; ++a; } }
#pragma unroll
        for (int u = 0; u < COLS; ++u) {
            const long long o = a < ph.h.taps ? px[u].at(g, a, b) : -1;
            ok[u] = o >= 0;
            at[u] = dy + (ok[u] ? o + (long long)(FEW ? m_next : s_k) * g.N : 0);
        }
        if (!FEW) row_next = ((ph.rh + a * g.sh) * g.bw + ph.rw + b * g.sw) * g.M;
    };
    if (chunks > 0) locate();
    // parameter staging: A_PER copies of 16 bytes per thread; their places inside a chunk do not change
    const size_t row_floats = (size_t)ctiles * ROW, plane = (size_t)g.bh * g.bw * g.M * row_floats;
    float rb[COLS][QPER];
    auto fetch = [&](float* stage) {
#pragma unroll
        for (int v = 0; v < A_PER; ++v) {
            const int i = threadIdx.x + v * T, p = i / (PLANE / 4), r = i % (PLANE / 4) / (ROW / 4), e = i % (ROW / 4) * 4;
            bool there = m_next + r < g.M;
            size_t row = row_next + r;
            if (FEW) {
                const int q = row_next + r, tap = q / g.M, ta = tap / ph.w.taps, tb = tap - ta * ph.w.taps;
                there = q < Q;
                row = ((ph.rh + ta * g.sh) * g.bw + ph.rw + tb * g.sw) * g.M + q - tap * g.M;
            }
            if (Tile::A_COPIES % T == 0 || i < Tile::A_COPIES)
                cp_async16(stage + p * PLANE + r * ROW + e, there ? dxp + p * plane + row * row_floats + ct * ROW + e : dxp, there ? 16 : 0);
        }
        if (FEW) {
#pragma unroll
            for (int s = 0; s < QPER; ++s) {
#pragma unroll
                for (int u = 0; u < COLS; ++u) {
                    rb[u][s] = 0.f;
                    if (ok[u]) { rb[u][s] = __ldg(at[u]); at[u] += (size_t)QSTEP * g.N; }
                }
                m_next += QSTEP;
                if (m_next >= g.M) locate();
            }
            row_next += KC;
            return;
        }
        const bool whole = m_next + KC <= g.M;
#pragma unroll
        for (int u = 0; u < COLS; ++u)
#pragma unroll
            for (int s = 0; s < QPER; ++s) {
                rb[u][s] = 0.f;
                if (ok[u] && (whole || m_next + s_k + s * QSTEP < g.M)) rb[u][s] = __ldg(at[u] + (size_t)(s * QSTEP) * g.N);
            }
        m_next += KC; row_next += KC;
#pragma unroll
        for (int u = 0; u < COLS; ++u) at[u] += (size_t)KC * g.N;
        if (m_next >= g.M) {
            m_next = 0;
            if (++b == ph.w.taps) { b = 0; ++a; }
            locate();
        }
    };
    auto commit = [&](float* stage) {
        float* B = stage + 2 * PLANE + s_k * TN + s_lane;
#pragma unroll
        for (int s = 0; s < QPER; ++s)
#pragma unroll
            for (int u = 0; u < COLS; ++u) B[s * QSTEP * TN + u * T] = rb[u][s];
        cp_async_wait_all();
    };

    // this thread's own x values (one per output)
    __syncthreads();
    float2 xx[RM][4], acc[RM][4];
    const size_t chw = (size_t)g.H * g.W;
#pragma unroll
    for (int r_ = 0; r_ < RM; ++r_) {
        const int c = i0 + ti * RM + r_;
#pragma unroll
        for (int c_ = 0; c_ < 8; ++c_) {
            const long long cb = col_base[col(c_)];
            const float v = (c < g.C && cb >= 0) ? __ldg(x + cb + (size_t)c * chw) : 0.f;
            if (c_ & 1) xx[r_][c_ >> 1].y = -v; else xx[r_][c_ >> 1].x = -v;
            acc[r_][c_ >> 1] = make_float2(0.f, 0.f);
        }
    }
    auto step = [&](const float* stage, int q) {
        float t[SLOT], w[SLOT];
        const float* A = stage + q * ROW + ti * SLOT;
        const float4 t4 = *reinterpret_cast<const float4*>(A), w4 = *reinterpret_cast<const float4*>(A + PLANE);
        t[0] = t4.x; t[1] = t4.y; t[2] = t4.z; t[3] = t4.w;
        w[0] = w4.x; w[1] = w4.y; w[2] = w4.z; w[3] = w4.w;
        if (RM == 5) { t[SLOT > 4 ? 4 : 0] = A[4]; w[SLOT > 4 ? 4 : 0] = A[PLANE + 4]; }
        if (RM == 6) {
            const float2 t2 = *reinterpret_cast<const float2*>(A + 4), w2 = *reinterpret_cast<const float2*>(A + PLANE + 4);
            t[SLOT > 4 ? 4 : 0] = t2.x; t[SLOT > 4 ? 5 : 0] = t2.y;
            w[SLOT > 4 ? 4 : 0] = w2.x; w[SLOT > 4 ? 5 : 0] = w2.y;
        }
        float2 g2[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 v = *reinterpret_cast<const float4*>(stage + 2 * PLANE + q * TN + h * (TN / 2) + tj * 4);
            g2[2 * h] = make_float2(v.x, v.y); g2[2 * h + 1] = make_float2(v.z, v.w);
        }
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 d = add2(splat2(t[r]), xx[r][c]), e = mul2(splat2(w[r]), g2[c]);
                if (L1) {
                    const float2 e0 = mul2(e, make_float2(0.f, 0.f));
                    acc[r][c] = add2(acc[r][c], make_float2(dx_signed(e.x, e0.x, d.x), dx_signed(e.y, e0.y, d.y)));
                } else acc[r][c] = fma2(e, d, acc[r][c]);
            }
    };
    auto compute = [&](const float* stage, int steps) {
        // (one branch in the middle and no more: a branch every four steps costs 15 %, and a second copy of the steps for partial
        // chunks as much again where the code grows with it, L1 above all)
#pragma unroll
        for (int q = 0; q < KC; ++q) {
            if (q == KC / 2 && steps <= KC / 2) break;
            step(stage, q);
        }
    };
    if (chunks > 0) {
        fetch(smem);
        commit(smem);
        __syncthreads();
        int m_now = 0, since = 0;
        bool aside = false;
        for (int i = 0; i < chunks; ++i) {
            float* now = smem + (i & 1) * Tile::STAGE;
            float* next = smem + ((i + 1) & 1) * Tile::STAGE;
            const bool more = i + 1 < chunks;
            const int steps = FEW ? min(KC, Q - i * KC) : min(KC, g.M - m_now);
            if ((since += steps) > kDxFold) {
#pragma unroll
                for (int k = 0; k < RM * 4; ++k) {
                    float2& v = acc[k >> 2][k & 3];
                    slots[k * T + threadIdx.x] = aside ? add2(slots[k * T + threadIdx.x], v) : v;
                    v = make_float2(0.f, 0.f);
                }
                aside = true;
                since = steps;
            }
            if (more) fetch(next);
            compute(now, steps);
            if (more) commit(next);
            __syncthreads();
            if ((m_now += KC) >= g.M) m_now = 0;
        }
        if (aside)
#pragma unroll
            for (int k = 0; k < RM * 4; ++k) acc[k >> 2][k & 3] = add2(slots[k * T + threadIdx.x], acc[k >> 2][k & 3]);
    }

    bool redo = false;
#pragma unroll
    for (int c_ = 0; c_ < 8; ++c_) {
        const long long cb = col_base[col(c_)];
        if (cb < 0) continue;
        const bool covered = col_covered[col(c_)];
#pragma unroll
        for (int r_ = 0; r_ < RM; ++r_) {
            const int c = i0 + ti * RM + r_;
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
        for (int i = 0; i < RM * 8; ++i) {
            const int c = i0 + ti * RM + i / 8;
            const long long cb = col_base[col(i % 8)];
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

// The pixels of the phase of pixel 0, which has the most.
static long long dx_pixels(const SimGeo& g) {
    const Axis h = dx_axis(g.H, g.bh, g.sh, g.ph, g.ph % g.sh), w = dx_axis(g.W, g.bw, g.sw, g.pw, g.pw % g.sw);
    return (long long)g.B * h.n * w.n;
}

// The tile of a shape: the least padding of channels by rows and of a tap's templates by the halves of a chunk; a row of a tile costs less the
// more of them share the staged dy values, the start of a tile is paid too (most in the long chunks of the largest), an SM of few tiles takes
// as long as one of its warps, and up to five tiles the busiest SM counts.  `few`: chunks that run through the taps, whose cursors take as long as
// 13 or 42 rows more.  The weights are those that lose least against the best tile over 477 shapes timed in every tile (8 to 200 samples of 12 to
// 200 x 32 x 32, 1 to 64 templates of 3x3 and 1x1): 1.4 % in the mean, a tenth less time than the least padding.
// 64 x 64 x 32 x 32 input, 3x3, in tiles of 64 rows / as picked: 1 template 58.8 / 25.1 us (few), 3 templates 58.9 / 34.4 (two tiles of 32 rows,
// as the next two), 9 91.5 / 70.8, 17 133 / 107; 8 x 24 x 32 x 32 under 17, L1: 62 in 64 CTAs of 24 rows, 36 in 128 of 16.
static const struct { int rm, wi; } kDxTiles[] = {{4, 4}, {6, 2}, {5, 2}, {4, 2}, {6, 1}, {5, 1}, {4, 1}};
struct DxPick { int rm, wi, slot, tiles; bool few; };
static DxPick dx_pick(const SimGeo& g) {
    const double columns = double((dx_pixels(g) + 127) / 128) * g.sh * g.sw / device_sm_count();
    DxPick best = {4, 4, 4, 1, false};
    double least = 0;
    for (const auto& t : kDxTiles)
        for (const bool few : {false, true}) {
            if (few && (t.rm != 4 || t.wi == 4 || g.M > 2 || g.bh * g.bw == 1)) continue;
            const int rows = 4 * t.rm * t.wi, tiles = (g.C + rows - 1) / rows, half = t.wi == 4 ? 8 : 4;
            const double steps = few ? double(g.M) * (rows + (t.wi == 1 ? 13 : 42)) : double((g.M + half - 1) / half * half) * (rows + 6.7) * (t.rm > 4 ? 1.03 : 1);
            const double start = t.wi == 4 ? 245 : (t.wi == 2 ? 27 : 37), alone = t.wi == 4 ? 1 : (t.wi == 2 ? 1.1 : 1.9);
            const double here = columns * tiles, per_sm = here < 5 ? std::ceil(here) : here;
            const double cost = (steps + start) * (std::max(per_sm, alone) + 0.08 * per_sm);
            if (least == 0 || cost < least) { least = cost; best = {t.rm, t.wi, t.rm == 4 ? 4 : 8, tiles, few}; }
        }
    return best;
}
// Room for the parameters in any of the tiles: the pick follows the batch, and a workspace sized for one batch serves every smaller one.
size_t sim_dx_scratch_floats(const SimGeo& g) {
    if (g.C <= 8) return 0;
    size_t row = 0;
    for (const auto& t : kDxTiles) row = std::max(row, size_t((g.C + 4 * t.rm * t.wi - 1) / (4 * t.rm * t.wi)) * 4 * t.wi * (t.rm == 4 ? 4 : 8));
    return 2 * (size_t)g.bh * g.bw * g.M * row;
}

cudaError_t launch_sim_dx(const SimGeo& g, const float* x, const float* t, const float* w, const float* dy, float* dx, float* dxp, cudaStream_t s) {
    const int phases = g.sh * g.sw;
    const long long pixels = dx_pixels(g);
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
    const DxPick pick = dx_pick(g);
    const long long total = (long long)g.bh * g.bw * g.M * pick.tiles * 4 * pick.wi * pick.slot;
    in_stream_order(sim_dx_prep, int(std::min<long long>((total + 255) / 256, (long long)device_sm_count() * 8)), 256, 0, s)(g, pick.rm, pick.slot, 4 * pick.wi, pick.tiles, t, w, dxp);
    const long long blocks = (pixels + 127) / 128 * pick.tiles;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const dim3 grid{unsigned(blocks), unsigned(phases)};
    const bool folds = (long long)((g.bh + g.sh - 1) / g.sh) * ((g.bw + g.sw - 1) / g.sw) * g.M > kDxFold;         // (the most taps of a phase)
#define DX_TILE(RM, WI, MODE, FEW)                                                                                                                   \
    do {                                                                                                                                      \
        using Tile = DxTile<RM, WI>;                                                                                                          \
        static SmemLimit limit;                                                                                                               \
        const cudaError_t e = limit.raise(sim_dx_tiled<RM, WI, MODE, FEW>, Tile::SLOT_BYTES);                                                      \
        if (e != cudaSuccess) return e;                                                                                                       \
        in_stream_order(sim_dx_tiled<RM, WI, MODE, FEW>, grid, Tile::T, folds ? Tile::SLOT_BYTES : 0, s)(g, x, dxp, t, w, dy, dx);                 \
    } while (0)
#define DX_41(MODE) DX_TILE(4, 1, MODE, false)
#define DX_51(MODE) DX_TILE(5, 1, MODE, false)
#define DX_61(MODE) DX_TILE(6, 1, MODE, false)
#define DX_42(MODE) DX_TILE(4, 2, MODE, false)
#define DX_52(MODE) DX_TILE(5, 2, MODE, false)
#define DX_62(MODE) DX_TILE(6, 2, MODE, false)
#define DX_44(MODE) DX_TILE(4, 4, MODE, false)
#define DX_FEW_1(MODE) DX_TILE(4, 1, MODE, true)
#define DX_FEW_2(MODE) DX_TILE(4, 2, MODE, true)
    if (pick.few) {
        if (pick.wi == 1) { DX_MODES(DX_FEW_1) } else { DX_MODES(DX_FEW_2) }
    } else
    switch (pick.wi * 8 + pick.rm) {
    case 12: DX_MODES(DX_41) break;
    case 13: DX_MODES(DX_51) break;
    case 14: DX_MODES(DX_61) break;
    case 20: DX_MODES(DX_42) break;
    case 21: DX_MODES(DX_52) break;
    case 22: DX_MODES(DX_62) break;
    default: DX_MODES(DX_44) break;
    }
    count_launch(2);
    return cudaGetLastError();
#undef DX_TILE
#undef DX_MODES
}

}  // namespace simnets
