// Shape-agnostic kernels: one thread per output element (or one block per reduced parameter).
// They accept every geometry and both dtypes, serve float64, unusual shapes and the
// SIMNETS_FLAG_FORCE_DIRECT switch, and give the tiled kernels a second GPU implementation to be
// compared with.  Tap addresses come from the geometry structs; no patch matrix is built.
//
// Arithmetic follows the reference's element functors (HUJI-Deep/simnets-tf,
// include/utils/similarity_utils.hpp:17-150 and include/utils/mex_utils.hpp:10-56), accumulation
// order follows its CPU kernels where a thread owns the whole sum.
#include "kernels.cuh"
#include "mex_exact.cuh"
#include "sim_exact.cuh"

namespace simnets {

namespace {

constexpr int kThreads = 256;

constexpr double kLog2Pi = 1.8378770664093454835606594728112;

// Gated launches follow a factorised kernel and work only if that one raised its flag: two CTAs per SM, since what the usual case pays is
// their coming up (eight CTAs of 256 threads for the seven launches of a step: 16.3 us, two 12.8), of more threads, since what the other
// case pays is how few they are.
constexpr int kGatedThreads = 640, kGatedBwdThreads = 2 * kThreads;

// Deterministic sum over kThreads threads (fixed tree), `lane` of a block of as many or of one of several such groups, which all take part;
// the result is valid in lane 0.
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* smem, int lane) {
    smem[lane] = v;
    __syncthreads();
    if (lane < 32) {
        const auto four = [&](int i) { return (smem[i] + smem[i + 128]) + (smem[i + 64] + smem[i + 192]); };
        v = four(lane) + four(lane + 32);
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) v += __shfl_down_sync(0xffffffffu, v, s);
    }
    __syncthreads();
    return v;
}
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* smem) { return block_sum(v, smem, int(threadIdx.x)); }

// ------------------------------------------------------------------ Similarity
template <typename T>
__global__ void __launch_bounds__(kThreads) sim_fwd_direct(SimGeo g, const T* __restrict__ x, const T* __restrict__ tm,
                                                           const T* __restrict__ wt, T* __restrict__ y, const int* __restrict__ gate,
                                                           FastDiv f_N, FastDiv f_M, FastDiv f_ow) {
    stream_order();
    if (gate && gate[1] == 0) return;
    const long long total = (long long)g.B * g.M * g.N;
    const T oob = T(g.oob), fudge = T(g.fudge);
    for (long long idx = blockIdx.x * (long long)kThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kThreads) {
        const long long q = total <= 0x7fffffffLL ? (long long)fast_div(uint32_t(idx), f_N) : idx / g.N;
        const int n = total <= 0x7fffffffLL ? int(fast_div(uint32_t(q), f_M)) : int(q / g.M);
        const int j = int(idx - q * g.N), m = int(q - (long long)n * g.M);
        const int ho = int(fast_div(uint32_t(j), f_ow)), wo = j - ho * g.ow;
        const T* xs = x + (size_t)n * g.C * g.H * g.W;
        const T* tp = tm + (size_t)m * g.K;
        const T* wp = wt + (size_t)m * g.K;
        T sum = T(0);
        int k = 0;
        for (int c = 0; c < g.C; ++c)
            for (int kh = 0; kh < g.bh; ++kh)
                for (int kw = 0; kw < g.bw; ++kw, ++k) {
                    const int hh = ho * g.sh - g.ph + kh, ww = wo * g.sw - g.pw + kw;
                    const T v = (hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) ? xs[((size_t)c * g.H + hh) * g.W + ww] : oob;
                    const T t = tp[k], w = g.absw ? dev_abs(wp[k]) : wp[k], d = t - v;
                    switch (g.mode) {
                    case SIM_L1: sum += -w * dev_abs(d); break;
                    case SIM_L1_SKIP: if (!is_nan(v)) sum += -w * dev_abs(d); break;
                    case SIM_L2: sum += -w * d * d; break;
                    case SIM_L2N: sum += T(0.5) * (-w * d * d + dev_log(w + fudge)); break;
                    default: if (!is_nan(v)) sum += T(0.5) * (-w * d * d - T(kLog2Pi) + dev_log(w + fudge)); break;
                    }
                }
        if (g.mode == SIM_L2N) {
            const T c = T(-0.5 * double(g.K) * kLog2Pi);
            const int reps = g.batch_quirk ? g.B - n : 1;
            for (int i = 0; i < reps; ++i) sum += c;
        }
        y[idx] = sum;
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) sim_dx_direct(SimGeo g, const T* __restrict__ x, const T* __restrict__ tm,
                                                          const T* __restrict__ wt, const T* __restrict__ dy, T* __restrict__ dx) {
    stream_order();
    const long long total = (long long)g.B * g.C * g.H * g.W;
    for (long long idx = blockIdx.x * (long long)kThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kThreads) {
        dx[idx] = sim_exact_dx(g, x, tm, wt, dy, idx);
    }
}

// The forward pass with four instances per thread: their parameters lie in shared memory (the normalisation's logarithm among them, taken
// once per tap instead of once per term), a patch value and its bounds test serve all four.  64 templates of 3x3 over 12 x 3 x 32 x 32 in
// float64: 30 us with an output per thread, 15.7 so.
constexpr int kDirectRows = 4, kDirectTaps = 256;
template <typename T>
__global__ void __launch_bounds__(kThreads) sim_fwd_direct_rows(SimGeo g, const T* __restrict__ x, const T* __restrict__ tm, const T* __restrict__ wt, T* __restrict__ y,
                                                                FastDiv f_N, FastDiv f_ow) {
    stream_order();
    __shared__ T st[kDirectRows * kDirectTaps], sw[kDirectRows * kDirectTaps], sc[kDirectRows * kDirectTaps];          // [tap][instance]
    const int m0 = blockIdx.y * kDirectRows;
    const T fudge = T(g.fudge), oob = T(g.oob);
    for (int i = threadIdx.x; i < g.K * kDirectRows; i += kThreads) {
        const int k = i / kDirectRows, m = min(m0 + i % kDirectRows, g.M - 1);
        const T w = g.absw ? dev_abs(wt[(size_t)m * g.K + k]) : wt[(size_t)m * g.K + k];
        st[i] = tm[(size_t)m * g.K + k];
        sw[i] = w;
        sc[i] = g.mode == SIM_L2N ? dev_log(w + fudge) : g.mode == SIM_L2N_NAN ? dev_log(w + fudge) - T(kLog2Pi) : T(0);
    }
    __syncthreads();
    const long long P = (long long)g.B * g.N;
    const bool l1 = g.mode == SIM_L1 || g.mode == SIM_L1_SKIP, skips = g.mode == SIM_L1_SKIP || g.mode == SIM_L2N_NAN;
    const T half = g.mode == SIM_L2N || g.mode == SIM_L2N_NAN ? T(0.5) : T(1);
    for (long long i = blockIdx.x * (long long)kThreads + threadIdx.x; i < P; i += (long long)gridDim.x * kThreads) {
        const int n = P <= 0x7fffffffLL ? int(fast_div(uint32_t(i), f_N)) : int(i / g.N), j = int(i - (long long)n * g.N);
        const int ho = int(fast_div(uint32_t(j), f_ow)), h0 = ho * g.sh - g.ph, w0 = (j - ho * g.ow) * g.sw - g.pw;
        const T* xs = x + (size_t)n * g.C * g.H * g.W;
        T sum[kDirectRows] = {};
        const T *pt = st, *pw = sw, *pc = sc;
        for (int c = 0; c < g.C; ++c)
            for (int kh = 0; kh < g.bh; ++kh)
                for (int kw = 0; kw < g.bw; ++kw, pt += kDirectRows, pw += kDirectRows, pc += kDirectRows) {
                    const int hh = h0 + kh, ww = w0 + kw;
                    const T v = (hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) ? xs[((size_t)c * g.H + hh) * g.W + ww] : oob;
                    if (skips && is_nan(v)) continue;
#pragma unroll
                    for (int u = 0; u < kDirectRows; ++u) {
                        const T d = pt[u] - v;
                        sum[u] += l1 ? -pw[u] * dev_abs(d) : half * (pc[u] - pw[u] * d * d);
                    }
                }
        const T add = T(-0.5 * double(g.K) * kLog2Pi);
        for (int u = 0; u < kDirectRows && m0 + u < g.M; ++u) {
            if (g.mode == SIM_L2N)
                for (int q = g.batch_quirk ? g.B - n : 1; q > 0; --q) sum[u] += add;
            y[((long long)n * g.M + m0 + u) * g.N + j] = sum[u];
        }
    }
}

// One block per (instance m, TK taps): reduces over batch and output positions, a position decoded and its dy read once for all of them.
// Positions are decoded by multiply and shift (f_N, f_ow; totals of 2^31 and more by division).  The sums are those of the other kernels
// (sim_dparams.cu), the factors of an instance and tap applied at the end.  64 templates of 3x3 over 12 x 3 x 32 x 32 in float64: 92 us
// with one tap per block, 42 so.
template <typename T, int TK, typename Offset>
__global__ void __launch_bounds__(kThreads) sim_dparams_direct(SimGeo g, const T* __restrict__ x, const T* __restrict__ tm,
                                                               const T* __restrict__ wt, const T* __restrict__ dy,
                                                               T* __restrict__ dt, T* __restrict__ dw, int accumulate, FastDiv f_N, FastDiv f_ow) {
    stream_order();
    __shared__ T smem[kThreads];
    const int groups = (g.K + TK - 1) / TK, m = blockIdx.x / groups, k0 = (blockIdx.x - m * groups) * TK;
    const T oob = T(g.oob);
    const bool l1 = g.mode == SIM_L1 || g.mode == SIM_L1_SKIP, skips = g.mode == SIM_L1_SKIP || g.mode == SIM_L2N_NAN;
    T t[TK], sT[TK], sW[TK], sN[TK];
    Offset at[TK];                                       // a tap's offset inside a sample
    int hk[TK], wk[TK];
#pragma unroll
    for (int u = 0; u < TK; ++u) {
        const int k = min(k0 + u, g.K - 1), c = k / (g.bw * g.bh);
        wk[u] = k % g.bw; hk[u] = k / g.bw % g.bh;
        at[u] = (Offset(c) * g.H + hk[u]) * g.W + wk[u];
        t[u] = tm[(size_t)m * g.K + k];
        sT[u] = sW[u] = sN[u] = T(0);
    }
    const long long total = (long long)g.B * g.N;
    for (long long i = threadIdx.x; i < total; i += kThreads) {
        const int n = total <= 0x7fffffffLL ? int(fast_div(uint32_t(i), f_N)) : int(i / g.N), j = int(i - (long long)n * g.N);
        const int ho = int(fast_div(uint32_t(j), f_ow)), h0 = ho * g.sh - g.ph, w0 = (j - ho * g.ow) * g.sw - g.pw;
        const T* xs = x + (long long)n * g.C * g.H * g.W + (long long)h0 * g.W + w0;
        const T err = dy[((size_t)n * g.M + m) * g.N + j];
        T v[TK];
#pragma unroll
        for (int u = 0; u < TK; ++u) v[u] = uint32_t(h0 + hk[u]) < uint32_t(g.H) && uint32_t(w0 + wk[u]) < uint32_t(g.W) ? xs[at[u]] : oob;
#pragma unroll
        for (int u = 0; u < TK; ++u) {
            if (skips && is_nan(v[u])) continue;
            const T d = v[u] - t[u];
            if (l1) {
                sT[u] += err * sign_of(d);
                sW[u] += err * dev_abs(d);
            } else {
                const T p = err * d;
                sT[u] += p;
                sW[u] += p * d;
                sN[u] += err;
            }
        }
    }
#pragma unroll 1
    for (int u = 0; u < TK; ++u) {
        if (k0 + u >= g.K) break;
        T a = T(0), b = T(0), c = T(0);
#pragma unroll
        for (int q = 0; q < TK; ++q) if (q == u) { a = sT[q]; b = sW[q]; c = sN[q]; }
        a = block_sum(a, smem);
        b = block_sum(b, smem);
        if (!l1 && g.mode != SIM_L2) c = block_sum(c, smem);
        if (threadIdx.x != 0) continue;
        const size_t mk = (size_t)m * g.K + k0 + u;
        const T wraw = wt[mk], w = g.absw ? dev_abs(wraw) : wraw;
        T gt = w * a, gw = -b;
        if (g.mode == SIM_L2) gt = T(2) * w * a;
        else if (!l1) gw = T(0.5) * (c / (w + T(g.fudge)) - b);
        if (g.absw) gw *= sign_of(wraw);                   // d|w|/dw, 0 at w = 0
        dt[mk] = accumulate ? dt[mk] + gt : gt;
        dw[mk] = accumulate ? dw[mk] + gw : gw;
    }
}

// ------------------------------------------------------------------------- MEX
template <typename T>
__global__ void __launch_bounds__(kGatedThreads, 2) mex_fwd_direct(MexGeo g, const T* __restrict__ x, const T* __restrict__ off, T* __restrict__ y, const int* __restrict__ gate) {
    stream_order();
    if (gate && (gate[0] | gate[1]) == 0) return;
    const long long total = (long long)g.B * g.M * g.N;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x)
        y[idx] = mex_exact_y(g, x, off, idx);
}

template <typename T>
__global__ void __launch_bounds__(kGatedThreads, sizeof(T) == 4 ? 2 : 1) mex_dx_direct(MexGeo g, const T* __restrict__ x, const T* __restrict__ off,
                                                          const T* __restrict__ y, const T* __restrict__ dy, T* __restrict__ dx, const int* __restrict__ gate) {
    stream_order();
    if (gate && (gate[0] | gate[1]) == 0) return;
    const long long total = (long long)g.B * g.C * g.H * g.W;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x)
        dx[idx] = mex_exact_dx(g, x, off, y, dy, idx);
}

// One block at a time per (region r, instance m, tap k): reduces over batch and the region's positions.
// The grid is capped and strides over the (r, m, k) triples, so that a gated-off launch costs a few
// hundred blocks, not one per parameter.
template <typename T>
__global__ void __launch_bounds__(kThreads) mex_doff_direct(MexGeo g, const T* __restrict__ x, const T* __restrict__ off,
                                                            const T* __restrict__ y, const T* __restrict__ dy,
                                                            T* __restrict__ doff, int accumulate, const int* __restrict__ gate) {
    stream_order();
    __shared__ T smem[kThreads];
    if (gate && (gate[0] | gate[1]) == 0) return;
    const long long triples = (long long)g.R * g.M * g.K;
    for (long long rmk = blockIdx.x; rmk < triples; rmk += gridDim.x) {
        const int k = int(rmk % g.K), m = int((rmk / g.K) % g.M), r = int(rmk / ((long long)g.K * g.M));
        const T o = off[rmk];
        T sum = T(0);
        const long long total = (long long)g.B * g.rs;
        for (long long i = threadIdx.x; i < total; i += kThreads) {
            sum += mex_exact_doff_term(g, x, o, y, dy, r, m, k, i);
        }
        const T rsum = block_sum(sum, smem);
        if (threadIdx.x == 0) doff[rmk] = accumulate ? doff[rmk] + rsum : rsum;
    }
}

// The term-by-term redo behind a factorised forward pass whose 2x2 sum pooling was produced with it: a thread redoes the four
// outputs of one pooling window and their sum (added in window order).
__global__ void __launch_bounds__(kGatedThreads, 2) mex_redo_fwd_pool(MexGeo g, const float* __restrict__ x, const float* __restrict__ off, float* __restrict__ y,
                                                              float* __restrict__ pooled, const int* __restrict__ gate) {
    stream_order();
    if ((gate[0] | gate[1]) == 0) return;
    const int Hp = g.Ho / 2, Wp = g.Wo / 2;
    const long long total = (long long)g.B * g.M * g.Co * Hp * Wp;
    for (long long i = blockIdx.x * (long long)kGatedThreads + threadIdx.x; i < total; i += (long long)gridDim.x * kGatedThreads) {
        const int w = int(i % Wp);
        const long long ph = i / Wp, at = (ph / Hp * g.Ho + 2 * (ph % Hp)) * g.Wo + 2 * w;
        float s = 0.f;
#pragma unroll 1
        for (int u = 0; u < 4; ++u) {
            const long long idx = at + (u >> 1) * g.Wo + (u & 1);
            const float v = mex_exact_y(g, x, off, idx);
            y[idx] = v;
            s = u == 0 ? v : s + v;
        }
        pooled[i] = s;
    }
}

// The same behind both gradients of a layer: one launch redoes dx and doff, kThreads threads a sum.
__global__ void __launch_bounds__(kGatedBwdThreads, 2) mex_redo_bwd(MexGeo g, const float* __restrict__ x, const float* __restrict__ off, const float* __restrict__ y,
                                                         const float* __restrict__ dy, float* __restrict__ dx, float* __restrict__ doff, int accumulate,
                                                         const int* __restrict__ gate) {
    stream_order();
    constexpr int kGroups = kGatedBwdThreads / kThreads;
    __shared__ float smem[kGatedBwdThreads];
    if ((gate[0] | gate[1]) == 0) return;
    const long long total = (long long)g.B * g.C * g.H * g.W;
    for (long long idx = blockIdx.x * (long long)kGatedBwdThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kGatedBwdThreads)
        dx[idx] = mex_exact_dx(g, x, off, y, dy, idx);
    const long long triples = (long long)g.R * g.M * g.K, positions = (long long)g.B * g.rs;
    const int group = threadIdx.x / kThreads, lane = threadIdx.x % kThreads;
    for (long long first = (long long)blockIdx.x * kGroups; first < triples; first += (long long)gridDim.x * kGroups) {
        const long long rmk = first + group;
        const int k = int(rmk % g.K), m = int((rmk / g.K) % g.M), r = int(rmk / ((long long)g.K * g.M));
        float sum = 0.f;
        if (rmk < triples)
            for (long long i = lane; i < positions; i += kThreads) sum += mex_exact_doff_term(g, x, off[rmk], y, dy, r, m, k, i);
        const float rsum = block_sum(sum, smem + group * kThreads, lane);
        if (lane == 0 && rmk < triples) doff[rmk] = accumulate ? doff[rmk] + rsum : rsum;
    }
}

inline int grid_for(long long total, bool gated = false) {
    const int threads = gated ? kGatedThreads : kThreads;
    const long long blocks = (total + threads - 1) / threads, cap = (long long)device_sm_count() * (gated ? 2 : 32);
    return int(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace

#define SIMNETS_DTYPE_SWITCH(is_f64, CALL32, CALL64) do { if (is_f64) { CALL64; } else { CALL32; } } while (0)

cudaError_t launch_sim_fwd_direct(const SimGeo& g, bool f64, const void* x, const void* t, const void* w, void* y, cudaStream_t s,
                                  const int* gate) {
    const long long total = (long long)g.B * g.M * g.N;
    if (total == 0) return cudaSuccess;
    // four instances per thread where that still leaves a thread per place of the GPU, and their parameters fit
    const long long P = (long long)g.B * g.N, rows = (g.M + kDirectRows - 1) / kDirectRows;
    if (gate == nullptr && g.K <= kDirectTaps && rows <= 65535 && P * rows >= 1024LL * device_sm_count()) {
        const dim3 grid(unsigned(std::min<long long>((P + kThreads - 1) / kThreads, std::max<long long>(1, 16LL * device_sm_count() / rows))), unsigned(rows));
        SIMNETS_DTYPE_SWITCH(f64,
            (in_stream_order(sim_fwd_direct_rows<float>, grid, kThreads, 0, s)(g, (const float*)x, (const float*)t, (const float*)w, (float*)y, make_fastdiv(g.N), make_fastdiv(g.ow))),
            (in_stream_order(sim_fwd_direct_rows<double>, grid, kThreads, 0, s)(g, (const double*)x, (const double*)t, (const double*)w, (double*)y, make_fastdiv(g.N), make_fastdiv(g.ow))));
        count_launch();
        return cudaGetLastError();
    }
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(sim_fwd_direct<float>, grid_for(total), kThreads, 0, s)(g, (const float*)x, (const float*)t, (const float*)w, (float*)y, gate, make_fastdiv(g.N), make_fastdiv(g.M), make_fastdiv(g.ow))),
        (in_stream_order(sim_fwd_direct<double>, grid_for(total), kThreads, 0, s)(g, (const double*)x, (const double*)t, (const double*)w, (double*)y, gate, make_fastdiv(g.N), make_fastdiv(g.M), make_fastdiv(g.ow))));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_sim_dx_direct(const SimGeo& g, bool f64, const void* x, const void* t, const void* w, const void* dy, void* dx, cudaStream_t s) {
    const long long total = (long long)g.B * g.C * g.H * g.W;
    if (total == 0) return cudaSuccess;
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(sim_dx_direct<float>, grid_for(total), kThreads, 0, s)(g, (const float*)x, (const float*)t, (const float*)w, (const float*)dy, (float*)dx)),
        (in_stream_order(sim_dx_direct<double>, grid_for(total), kThreads, 0, s)(g, (const double*)x, (const double*)t, (const double*)w, (const double*)dy, (double*)dx)));
    count_launch();
    return cudaGetLastError();
}

namespace {
__global__ void __launch_bounds__(kThreads) zero_words(int* __restrict__ p, int n) {
    stream_order();
    for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) p[i] = 0;
}
}  // namespace

cudaError_t launch_zero_words(int* p, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    in_stream_order(zero_words, std::min((n + kThreads - 1) / kThreads, 64), kThreads, 0, s)(p, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_sim_dparams_direct(const SimGeo& g, bool f64, const void* x, const void* t, const void* w, const void* dy,
                                      void* dt, void* dw, bool accumulate, cudaStream_t s) {
    // as many taps per block as leave every SM one; one where their offsets need 64 bits
#define DP(TK, Offset)                                                                                                                                  \
    SIMNETS_DTYPE_SWITCH(f64,                                                                                                                           \
        (in_stream_order(sim_dparams_direct<float, TK, Offset>, g.M * ((g.K + TK - 1) / TK), kThreads, 0, s)(g, (const float*)x, (const float*)t, (const float*)w, (const float*)dy, (float*)dt, (float*)dw, accumulate, make_fastdiv(g.N), make_fastdiv(g.ow))), \
        (in_stream_order(sim_dparams_direct<double, TK, Offset>, g.M * ((g.K + TK - 1) / TK), kThreads, 0, s)(g, (const double*)x, (const double*)t, (const double*)w, (const double*)dy, (double*)dt, (double*)dw, accumulate, make_fastdiv(g.N), make_fastdiv(g.ow))))
    const bool near = sim_offsets_below(g, 1LL << 31);
    const auto fills = [&](int taps) { return near && (long long)g.M * ((g.K + taps - 1) / taps) >= device_sm_count(); };
    if (fills(8)) { DP(8, int); } else if (fills(4)) { DP(4, int); } else if (fills(2)) { DP(2, int); } else { DP(1, long long); }
#undef DP
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_fwd_direct(const MexGeo& g, bool f64, const void* x, const void* off, void* y, cudaStream_t s, const int* gate) {
    const long long total = (long long)g.B * g.M * g.N;
    if (total == 0) return cudaSuccess;
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(mex_fwd_direct<float>, grid_for(total, gate != nullptr), gate != nullptr ? kGatedThreads : kThreads, 0, s)(g, (const float*)x, (const float*)off, (float*)y, gate)),
        (in_stream_order(mex_fwd_direct<double>, grid_for(total), kThreads, 0, s)(g, (const double*)x, (const double*)off, (double*)y, gate)));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_redo_fwd_pool(const MexGeo& g, const float* x, const float* off, float* y, float* pooled, cudaStream_t s, const int* gate) {
    in_stream_order(mex_redo_fwd_pool, grid_for((long long)g.B * g.M * g.N / 4, true), kGatedThreads, 0, s)(g, x, off, y, pooled, gate);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_redo_bwd(const MexGeo& g, const float* x, const float* off, const float* y, const float* dy, float* dx, float* doff, bool accumulate,
                                cudaStream_t s, const int* gate) {
    in_stream_order(mex_redo_bwd, device_sm_count() * 2, kGatedBwdThreads, 0, s)(g, x, off, y, dy, dx, doff, int(accumulate), gate);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_dx_direct(const MexGeo& g, bool f64, const void* x, const void* off, const void* y, const void* dy, void* dx, cudaStream_t s, const int* gate) {
    const long long total = (long long)g.B * g.C * g.H * g.W;
    if (total == 0) return cudaSuccess;
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(mex_dx_direct<float>, grid_for(total, gate != nullptr), gate != nullptr ? kGatedThreads : kThreads, 0, s)(g, (const float*)x, (const float*)off, (const float*)y, (const float*)dy, (float*)dx, gate)),
        (in_stream_order(mex_dx_direct<double>, grid_for(total), kThreads, 0, s)(g, (const double*)x, (const double*)off, (const double*)y, (const double*)dy, (double*)dx, gate)));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_doff_direct(const MexGeo& g, bool f64, const void* x, const void* off, const void* y, const void* dy,
                                   void* doff, bool accumulate, cudaStream_t s, const int* gate) {
    const long long triples = (long long)g.R * g.M * g.K;
    const long long cap = (long long)device_sm_count() * 16;
    const int blocks = int(triples < cap ? triples : cap);
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(mex_doff_direct<float>, blocks, kThreads, 0, s)(g, (const float*)x, (const float*)off, (const float*)y, (const float*)dy, (float*)doff, accumulate, gate)),
        (in_stream_order(mex_doff_direct<double>, blocks, kThreads, 0, s)(g, (const double*)x, (const double*)off, (const double*)y, (const double*)dy, (double*)doff, accumulate, gate)));
    count_launch();
    return cudaGetLastError();
}

}  // namespace simnets
