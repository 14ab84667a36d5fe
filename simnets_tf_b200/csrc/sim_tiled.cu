// Similarity forward as an implicit-im2col generalized GEMM (float32), and the entry points of the whole float32 family.
//
//   forward   y[n, m, pos]   = sum_k f(t[m,k], w[m,k], patch[k, (n,pos)])              i = m, j = position, q = tap
//
// with the reference's element functors (HUJI-Deep/simnets-tf include/utils/similarity_utils.hpp:17-119).
// The patch matrix of the reference (src/utils/im2col.cpp:247-280) is never built: a tap table gives, for
// each k = (c, kh, kw), its offset inside a sample and its (kh, kw); a position gives its patch corner.
// NaN handling costs no branch in the inner loop: while an input value is staged into shared memory a NaN
// becomes (value 0, mask 0) and the mask multiplies the term (ignore_nan_input modes); in the other modes
// the NaN itself is staged and propagates through the arithmetic exactly as in the reference.
// Per-(m,k) constants (0.5*log(w + fudge) - 0.5*log(2*pi), -w, -0.5*w) are computed once by a prepass,
// which also lays the parameters out tap-major so that the forward kernel's loads are contiguous.
#include <cmath>
#include "kernels.cuh"
#include "tile.cuh"

namespace simnets {

namespace {

constexpr double kLog2Pi = 1.8378770664093454835606594728112;

struct SimWs {
    int* flag;       // [2]: word 1 = a bounded wait of the tensor-core forward kernel ran out (its output is redone)
    float* planes;   // [3][K][Mp]: t, scale (-w or -0.5w), per-term constant; Mp = M rounded up to 4 floats
    float* cm;       // [M] per-instance constant added once per output
    int2* taps;      // [K]: {offset of tap inside a sample, (kh << 16) | kw}
    int2* tests;     // [K]: {byte offset, bit kh | bit 16 + kw}, blocks of up to 16 x 16
    float* part;     // [S][3][M][K] split partial sums of the parameter gradients
    float* dxp;      // [2][bh*bw*M][Cp]: t and s*w (s = 2 for plain L2, else 1), channel-contiguous, for the input gradient
    float* tc_tiles; // pre-split parameter tiles of the tensor-core forward kernel
    float* tc_bias;  // [M] its per-instance constant
    size_t bytes;
};

__host__ inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }
__host__ __device__ inline int pad4(int v) { return (v + 3) & ~3; }

__host__ SimWs carve(const SimGeo& g, void* base) {
    SimWs w;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t bytes) { char* r = p ? p + off : nullptr; off += align256(bytes); return r; };
    w.flag = reinterpret_cast<int*>(take(sizeof(int) * 2));
    w.planes = reinterpret_cast<float*>(take(sizeof(float) * 3 * (size_t)g.K * pad4(g.M)));
    w.cm = reinterpret_cast<float*>(take(sizeof(float) * g.M));
    w.taps = reinterpret_cast<int2*>(take(sizeof(int2) * g.K));
    w.tests = reinterpret_cast<int2*>(take(sizeof(int2) * g.K));
    w.part = reinterpret_cast<float*>(take(sizeof(float) * 3 * (size_t)sim_dparams_splits(g) * g.M * g.K));
    w.dxp = reinterpret_cast<float*>(take(sizeof(float) * sim_dx_scratch_floats(g)));
    w.tc_tiles = reinterpret_cast<float*>(take(sizeof(float) * sim_tc_tile_floats(g)));
    w.tc_bias = reinterpret_cast<float*>(take(sizeof(float) * g.M));
    w.bytes = off;
    return w;
}

// The test of a tap against the image as one AND of two bits with what the position's patch misses: blocks of up to 16 x 16, 32-bit byte
// offsets.  (Two range tests per gathered value, although a patch inside the image skipped them: 256 x 64 x 32 x 32 input, 256 templates
// of 3x3 4134 -> 3913 us, with masks 6046 -> 5557, L1 3119 -> 2838.)
__host__ __device__ inline bool sim_tap_bits(const SimGeo& g) { return g.bh <= 16 && g.bw <= 16 && sim_offsets_below(g, 1LL << 29); }

// One block per instance m: tap-major parameter planes, the per-instance constant, and (block 0) the tap table.
__global__ void __launch_bounds__(128) sim_prep(SimGeo g, const float* __restrict__ tm, const float* __restrict__ wt,
                                                float* __restrict__ planes, float* __restrict__ cm, int2* __restrict__ taps,
                                                int2* __restrict__ tests, int* __restrict__ flag) {
    stream_order();
    __shared__ float red[128];
    const int m = blockIdx.x;
    if (m == 0 && threadIdx.x < 2) flag[threadIdx.x] = 0;
    const float fudge = float(g.fudge);
    const int ldm = pad4(g.M);
    const size_t plane = (size_t)g.K * ldm;
    float csum = 0.f;
    for (int k = threadIdx.x; k < g.K; k += 128) {
        const float t = tm[(size_t)m * g.K + k], w = g.absw ? fabsf(wt[(size_t)m * g.K + k]) : wt[(size_t)m * g.K + k];
        float scale = -w, c = 0.f;
        if (g.mode == SIM_L2N) { scale = -0.5f * w; csum += 0.5f * logf(w + fudge); }
        if (g.mode == SIM_L2N_NAN) { scale = -0.5f * w; c = float(0.5 * (double(logf(w + fudge)) - kLog2Pi)); }
        planes[(size_t)k * ldm + m] = t;
        planes[plane + (size_t)k * ldm + m] = scale;
        planes[2 * plane + (size_t)k * ldm + m] = c;
        const int kw = k % g.bw, kh = (k / g.bw) % g.bh, c_ = k / (g.bw * g.bh);
        if (m == 0) {
            taps[k] = make_int2((c_ * g.H + kh) * g.W + kw, (kh << 16) | kw);
            if (sim_tap_bits(g)) tests[k] = make_int2(4 * ((c_ * g.H + kh) * g.W + kw), (1 << kh) | (0x10000 << kw));
        }
    }
    red[threadIdx.x] = csum;
    __syncthreads();
    for (int s = 64; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) cm[m] = g.mode == SIM_L2N ? red[0] + float(-0.5 * double(g.K) * kLog2Pi) : 0.f;
}

struct SimColumn {
    long long base;     // n*M*N + pos, or -1 past the end
    int n, h0, w0;      // sample, patch corner
};

__device__ __forceinline__ SimColumn sim_column(const SimGeo& g, long long j, long long P) {
    SimColumn c;
    c.base = -1; c.n = 0; c.h0 = c.w0 = 0;
    if (j >= P) return c;
    const int n = int(j / g.N), pos = int(j % g.N);
    c.n = n;
    c.h0 = (pos / g.ow) * g.sh - g.ph;
    c.w0 = (pos % g.ow) * g.sw - g.pw;
    c.base = (long long)n * g.M * g.N + pos;
    return c;
}

__device__ __forceinline__ float sim_tap_value(const SimGeo& g, const float* __restrict__ xs, const SimColumn& col, int2 tap, float oob) {
    const int hh = col.h0 + (tap.y >> 16), ww = col.w0 + (tap.y & 0xffff);
    if (hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) return __ldg(xs + tap.x + col.h0 * g.W + col.w0);
    return oob;
}

// ------------------------------------------------------------------- forward
// MODE is a SimMode; NA = parameter planes used, NB = input planes (value [, mask]).
template <int MODE> struct FwdPlanes {
    static constexpr int NA = MODE == SIM_L2N_NAN ? 3 : 2;
    static constexpr int NB = (MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP) ? 2 : 1;
};

__device__ __forceinline__ float2 abs2(float2 v) { return make_float2(fabsf(v.x), fabsf(v.y)); }

// Tile TM x TN, 8 x 8, 4 x 8 or 4 x 4 outputs per thread; small tiles walk 16 taps per chunk (their chunks are short, and every
// chunk costs a round trip to L2).
template <int TM, int TN> struct FwdTile {
    static constexpr int RM = TM == 128 ? 8 : 4, RN = TN == 128 ? 8 : 4, KC = TM * TN <= 2048 ? 16 : 8, THREADS = (TM / RM) * (TN / RN);
    static constexpr int PER_SM = TN == 128 ? 2 : 512 / THREADS;
};

template <int TM, int TN, int MODE>
__global__ void __launch_bounds__(FwdTile<TM, TN>::THREADS, FwdTile<TM, TN>::PER_SM) sim_fwd_tiled(SimGeo g, const float* __restrict__ x, const float* __restrict__ planes,
                                                     const float* __restrict__ cm, const int2* __restrict__ taps, int bits, float* __restrict__ y) {
    stream_order();
    constexpr int NA = FwdPlanes<MODE>::NA, NB = FwdPlanes<MODE>::NB;
    using Cfg = TileCfg<TM, TN, FwdTile<TM, TN>::KC, FwdTile<TM, TN>::RM, FwdTile<TM, TN>::RN, NA, NB>;
    constexpr int QSTEP = Cfg::THREADS / TN;                     // threads along the taps when a chunk is staged
    static_assert(QSTEP >= 1 && Cfg::THREADS % TN == 0, "a thread stages one column");
    __shared__ __align__(16) float smem[Cfg::SMEM_FLOATS];
    __shared__ long long col_base[Cfg::TN];
    const long long P = (long long)g.B * g.N;
    const int mtiles = (g.M + TM - 1) / TM;
    const int mt = blockIdx.x % mtiles;
    const long long jt = blockIdx.x / mtiles;
    const int i0 = mt * TM;
    const long long j0 = jt * Cfg::TN;

    const TileThread<Cfg> t;
    const float oob = float(g.oob);
    const int ldm = pad4(g.M);
    const size_t plane = (size_t)g.K * ldm;
    const int s_lane = threadIdx.x % TN, s_k = threadIdx.x / TN;
    const SimColumn sc = sim_column(g, j0 + s_lane, P);
    if (s_k == 0) col_base[s_lane] = sc.base;
    const bool live = sc.base >= 0;
    const int missing = live ? int(missing_taps(sc.h0, g.H) | (missing_taps(sc.w0, g.W) << 16)) : -1;
    const float outside = live ? oob : 0.f;
    const float* xs = x + (size_t)sc.n * g.C * g.H * g.W;
    const char* xc = reinterpret_cast<const char*>(xs + sc.h0 * g.W + sc.w0);
    float rb[Cfg::B_PER];

    float2 acc[Cfg::RM][Cfg::RN / 2];
#pragma unroll
    for (int r_ = 0; r_ < Cfg::RM; ++r_)
#pragma unroll
        for (int c_ = 0; c_ < Cfg::RN / 2; ++c_) acc[r_][c_] = make_float2(0.f, 0.f);

    auto fetchA = [&](int chunk, float* As) {
#pragma unroll
        for (int p = 0; p < NA; ++p)
            stage_copy_async<Cfg, TM>(As + p * Cfg::KC * TM, planes + p * plane, ldm, chunk * Cfg::KC, g.K, i0, g.M);
    };
    // A gathered value hangs on its tap's entry: the entries of the next chunk are read while this one is multiplied, so that a
    // chunk waits for one read and not for two in a row (8 x 16 x 20 x 20 input, 48 templates of 3x3: 24.1 -> 19.0 us; 128 x 16 x
    // 24 x 24, 33 of 5x5 with stride 2: 98.7 -> 78.6).  8 x 8 blocking, or 4 x 8 with masks, has no registers left for them
    // (256 x 64 x 32 x 32, 256 of 3x3: 4134 -> 4245).
    constexpr bool AHEAD = Cfg::RM * Cfg::RN <= (NB == 2 ? 16 : 32);
    int2 tap[AHEAD ? Cfg::B_PER : 1];
    if (AHEAD) {
#pragma unroll
        for (int s = 0; s < Cfg::B_PER; ++s) tap[AHEAD ? s : 0] = __ldg(taps + min(s_k + s * QSTEP, g.K - 1));
    }
    // (rows past K pair a zero scale / zero constant with a finite value: the term is exactly 0)
    auto fetchB = [&](int chunk, float*) {
        if (bits) {
#pragma unroll
            for (int s = 0; s < Cfg::B_PER; ++s) {
                const int k = chunk * Cfg::KC + s_k + s * QSTEP;
                rb[s] = 0.f;
                if (k < g.K) {
                    const int2 t = AHEAD ? tap[AHEAD ? s : 0] : __ldg(taps + k);
                    rb[s] = outside;
                    if ((t.y & missing) == 0) rb[s] = __ldg(reinterpret_cast<const float*>(xc + t.x));
                }
                if (AHEAD) tap[AHEAD ? s : 0] = __ldg(taps + min(k + Cfg::KC, g.K - 1));
            }
        } else {
#pragma unroll
            for (int s = 0; s < Cfg::B_PER; ++s) {
                const int k = chunk * Cfg::KC + s_k + s * QSTEP;
                rb[s] = k < g.K && live ? sim_tap_value(g, xs, sc, __ldg(taps + k), oob) : 0.f;
            }
        }
    };
    auto commitA = [&](float*) { cp_async_wait_all(); };
    auto commitB = [&](float* Bs) {
#pragma unroll
        for (int s = 0; s < Cfg::B_PER; ++s) {
            const int o = (s_k + s * QSTEP) * Cfg::TN + s_lane;
            if (NB == 2) {
                const bool nan = rb[s] != rb[s];
                Bs[o] = nan ? 0.f : rb[s];
                Bs[Cfg::KC * Cfg::TN + o] = nan ? 0.f : 1.f;
            } else {
                Bs[o] = rb[s];
            }
        }
    };
    auto comb = [&](int r_, int cp, const float2 (&a)[NA], const float2 (&b)[NB]) {
        const float2 d = add2(a[0], neg2(b[0]));
        if (MODE == SIM_L1) acc[r_][cp] = fma2(a[1], abs2(d), acc[r_][cp]);
        else if (MODE == SIM_L1_SKIP) acc[r_][cp] = fma2(a[1], mul2(abs2(d), b[NB - 1]), acc[r_][cp]);
        else if (MODE == SIM_L2N_NAN) acc[r_][cp] = fma2(b[NB - 1], fma2(mul2(a[1], d), d, a[NA - 1]), acc[r_][cp]);
        else acc[r_][cp] = fma2(mul2(a[1], d), d, acc[r_][cp]);
    };
    tile_mainloop<Cfg, false, false>(smem, (g.K + Cfg::KC - 1) / Cfg::KC, t, fetchA, fetchB, commitA, commitB, comb);

    long long cb[Cfg::RN];
#pragma unroll
    for (int c_ = 0; c_ < Cfg::RN; ++c_) cb[c_] = col_base[t.col(c_)];
    const float quirk_c = float(-0.5 * double(g.K) * kLog2Pi);
#pragma unroll
    for (int r_ = 0; r_ < Cfg::RM; ++r_) {
        const int m = i0 + t.row(r_);
        if (m >= g.M) continue;
        const float cmm = cm[m];
        float* yrow = y + (long long)m * g.N;
#pragma unroll
        for (int c_ = 0; c_ < Cfg::RN; ++c_) {
            if (cb[c_] < 0) continue;
            float v = (c_ & 1) ? acc[r_][c_ >> 1].y : acc[r_][c_ >> 1].x;
            if (MODE == SIM_L2N) {
                v += cmm;
                if (g.batch_quirk) v += quirk_c * float(g.B - 1 - int(cb[c_] / ((long long)g.M * g.N)));
            }
            __stcs(yrow + cb[c_], v);
        }
    }
}

void launch_prep(const SimGeo& g, const SimWs& w, const float* t, const float* wt, cudaStream_t s) {
    in_stream_order(sim_prep, g.M, 128, 0, s)(g, t, wt, w.planes, w.cm, w.taps, w.tests, w.flag);
    count_launch();
}

}  // namespace

bool sim_use_tiled(const SimGeo& g, bool f64, uint32_t flags) {
    if (f64 || g.B == 0) return false;
    if (flags & SIMNETS_FLAG_FORCE_DIRECT) return false;
    if (g.bh >= 32768 || g.bw >= 32768) return false;
    return true;
}

size_t sim_workspace_bytes(const SimGeo& g, bool f64, uint32_t flags) {
    if (!sim_use_tiled(g, f64, flags)) return 256;
    return carve(g, nullptr).bytes;
}

static cudaError_t sim_fwd_tiled_body(const SimGeo& g, const float* x, const float* t, const float* w, float* y, void* ws, uint32_t flags,
                                      cudaStream_t s, float* ch_max, float* ch_min, bool* extrema_done);

cudaError_t launch_sim_fwd_tiled(const SimGeo& g, const float* x, const float* t, const float* w, float* y, void* ws, uint32_t flags,
                                 cudaStream_t s, float* ch_max, float* ch_min) {
    bool done = false;
    const cudaError_t e = sim_fwd_tiled_body(g, x, t, w, y, ws, flags, s, ch_max, ch_min, &done);
    if (e != cudaSuccess || done) return e;
    return launch_sim_extrema(g, y, ch_max, ch_min, s);
}

static cudaError_t sim_fwd_tiled_body(const SimGeo& g, const float* x, const float* t, const float* w, float* y, void* ws, uint32_t flags,
                                      cudaStream_t s, float* ch_max, float* ch_min, bool* extrema_done) {
    const SimWs W = carve(g, ws);
    if (!sim_offsets_below(g, 1LL << 31)) {                 // (the tap tables hold 32 bits)
        const cudaError_t e = launch_zero_words(W.flag, 2, s);
        return e != cudaSuccess ? e : launch_sim_fwd_direct(g, false, x, t, w, y, s);
    }
    if (!sim_tc_shape(g, flags) && sim_smallk_shape(g)) return launch_sim_fwd_smallk(g, x, t, w, y, ch_max, ch_min, extrema_done, W.flag, s);
    launch_prep(g, W, t, w, s);
    if (sim_tc_shape(g, flags)) {
        // opt-in: the expanded square on the tensor cores; behind it the term-by-term kernel, which runs only if a
        // bounded wait of the tensor-core kernel ran out (word 1 of the flags)
        const cudaError_t e = launch_sim_fwd_tc(g, x, W.planes, W.cm, W.taps, W.tc_tiles, W.tc_bias, W.flag, y, s);
        if (e != cudaSuccess) return e;
        return launch_sim_fwd_direct(g, false, x, t, w, y, s, W.flag);
    }
    const long long P = (long long)g.B * g.N;
    // The tile with the least estimated time: tiles per SM (rounded up) x outputs per tile x the relative cost of a term at
    // that tile's register blocking, stretched where too few warps are resident to keep the FP32 pipe fed (the larger tiles on
    // small inputs: 16 x 20 x 20 inputs under 48 templates fill 56 tiles of 64 x 128 on 148 SMs).
    // With masks the 8 x 8 blocking spills at 128 registers, 4 x 8 does not (terms from registers and shared memory alone: 6.5
    // and 7.7 T/s).  Under 16 warps per SM, one CTA of the large tiles, nothing covers a CTA's barriers (16 x 64 x 32 x 32 input,
    // 128 templates of 3x3: 206 us in 128 tiles of 128 x 128, 191 in 256 of 64 x 128; with masks 309 and 239, before both staged less).
    struct { int tm, tn, threads; double cost; } const tiles[] = {{128, 128, 256, 1.0}, {64, 128, 256, g.mode == SIM_L2N_NAN ? 0.98 : 1.05}, {32, 64, 128, 1.6}, {16, 32, 32, 2.0}};
    int pick = 0;
    double best = 0;
    for (int i = 0; i < 4; ++i) {
        const double ctas = double((P + tiles[i].tn - 1) / tiles[i].tn) * ((g.M + tiles[i].tm - 1) / tiles[i].tm);
        const double per_sm = std::ceil(ctas / device_sm_count()), warps = per_sm * tiles[i].threads / 32;
        const double t = per_sm * tiles[i].tm * tiles[i].tn * tiles[i].cost * (warps < 8 ? 8 / warps : 1.0) * (warps < 16 ? 1.15 : 1.0);
        if (i == 0 || t < best) { best = t; pick = i; }
    }
    const long long blocks = ((P + tiles[pick].tn - 1) / tiles[pick].tn) * ((g.M + tiles[pick].tm - 1) / tiles[pick].tm);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const int bits = sim_tap_bits(g);
    const int2* taps = bits ? W.tests : W.taps;
#define FWD(TM, TN, MODE) in_stream_order(sim_fwd_tiled<TM, TN, MODE>, int(blocks), FwdTile<TM, TN>::THREADS, 0, s)(g, x, W.planes, W.cm, taps, bits, y)
#define FWD_MODES(TM, TN)                                        \
    switch (g.mode) {                                            \
    case SIM_L1: FWD(TM, TN, SIM_L1); break;                     \
    case SIM_L1_SKIP: FWD(TM, TN, SIM_L1_SKIP); break;           \
    case SIM_L2: FWD(TM, TN, SIM_L2); break;                     \
    case SIM_L2N: FWD(TM, TN, SIM_L2N); break;                   \
    default: FWD(TM, TN, SIM_L2N_NAN); break;                    \
    }
    if (pick == 0) { FWD_MODES(128, 128) } else if (pick == 1) { FWD_MODES(64, 128) } else if (pick == 2) { FWD_MODES(32, 64) } else { FWD_MODES(16, 32) }
#undef FWD_MODES
#undef FWD
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_sim_dx_tiled(const SimGeo& g, const float* x, const float* t, const float* w, const float* dy, float* dx, void* ws, cudaStream_t s) {
    return launch_sim_dx(g, x, t, w, dy, dx, carve(g, ws).dxp, s);
}

cudaError_t launch_sim_dparams_tiled(const SimGeo& g, const float* x, const float* t, const float* w, const float* dy,
                                     float* dt, float* dw, bool accumulate, void* ws, cudaStream_t s) {
    return launch_sim_dparams(g, x, t, w, dy, dt, dw, accumulate, carve(g, ws).part, s);
}

}  // namespace simnets
