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

// Deterministic block-wide sum (fixed tree), result valid in thread 0.
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* smem) {
    smem[threadIdx.x] = v;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) smem[threadIdx.x] += smem[threadIdx.x + s];
        __syncthreads();
    }
    const T r = smem[0];
    __syncthreads();
    return r;
}

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

// One block per (instance m, tap k): reduces over batch and output positions.  Positions are decoded by multiply and shift
// (f_N, f_ow; totals of 2^31 and more by division): a 64-bit division and modulo per term had been most of the instructions.
template <typename T>
__global__ void __launch_bounds__(kThreads) sim_dparams_direct(SimGeo g, const T* __restrict__ x, const T* __restrict__ tm,
                                                               const T* __restrict__ wt, const T* __restrict__ dy,
                                                               T* __restrict__ dt, T* __restrict__ dw, int accumulate, FastDiv f_N, FastDiv f_ow) {
    stream_order();
    __shared__ T smem[kThreads];
    const int mk = blockIdx.x;
    const int m = mk / g.K, k = mk % g.K;
    const int kw = k % g.bw, kh = (k / g.bw) % g.bh, c = k / (g.bw * g.bh);
    const T wraw = wt[mk];
    const T t = tm[mk], w = g.absw ? dev_abs(wraw) : wraw, oob = T(g.oob), fudge = T(g.fudge);
    T st = T(0), sw_ = T(0);
    const long long total = (long long)g.B * g.N;
    for (long long i = threadIdx.x; i < total; i += kThreads) {
        const int n = total <= 0x7fffffffLL ? int(fast_div(uint32_t(i), f_N)) : int(i / g.N), j = int(i - (long long)n * g.N);
        const int ho = int(fast_div(uint32_t(j), f_ow)), wo = j - ho * g.ow;
        const int hh = ho * g.sh - g.ph + kh, ww = wo * g.sw - g.pw + kw;
        const T v = (hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) ? x[(((size_t)n * g.C + c) * g.H + hh) * g.W + ww] : oob;
        const T err = dy[((size_t)n * g.M + m) * g.N + j];
        const T d = v - t;
        switch (g.mode) {
        case SIM_L1: st += err * w * sign_of(d); sw_ += -err * dev_abs(d); break;
        case SIM_L1_SKIP: if (!is_nan(v)) { st += err * w * sign_of(d); sw_ += -err * dev_abs(d); } break;
        case SIM_L2: st += T(2) * err * w * d; sw_ += -err * d * d; break;
        case SIM_L2N: st += err * w * d; sw_ += T(0.5) * (-err * d * d + err / (w + fudge)); break;
        default: if (!is_nan(v)) { st += err * w * d; sw_ += T(0.5) * (-err * d * d + err / (w + fudge)); } break;
        }
    }
    const T rt = block_sum(st, smem);
    T rw = block_sum(sw_, smem);
    if (g.absw) rw *= sign_of(wraw);                   // d|w|/dw, 0 at w = 0
    if (threadIdx.x == 0) {
        dt[mk] = accumulate ? dt[mk] + rt : rt;
        dw[mk] = accumulate ? dw[mk] + rw : rw;
    }
}

// ------------------------------------------------------------------------- MEX
template <typename T>
__global__ void __launch_bounds__(kThreads) mex_fwd_direct(MexGeo g, const T* __restrict__ x, const T* __restrict__ off, T* __restrict__ y, const int* __restrict__ gate) {
    stream_order();
    if (gate && (gate[0] | gate[1]) == 0) return;
    const long long total = (long long)g.B * g.M * g.N;
    for (long long idx = blockIdx.x * (long long)kThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kThreads)
        y[idx] = mex_exact_y(g, x, off, idx);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) mex_dx_direct(MexGeo g, const T* __restrict__ x, const T* __restrict__ off,
                                                          const T* __restrict__ y, const T* __restrict__ dy, T* __restrict__ dx, const int* __restrict__ gate) {
    stream_order();
    if (gate && (gate[0] | gate[1]) == 0) return;
    const long long total = (long long)g.B * g.C * g.H * g.W;
    for (long long idx = blockIdx.x * (long long)kThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kThreads)
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
__global__ void __launch_bounds__(kThreads) mex_redo_fwd_pool(MexGeo g, const float* __restrict__ x, const float* __restrict__ off, float* __restrict__ y,
                                                              float* __restrict__ pooled, const int* __restrict__ gate) {
    stream_order();
    if ((gate[0] | gate[1]) == 0) return;
    const int Hp = g.Ho / 2, Wp = g.Wo / 2;
    const long long total = (long long)g.B * g.M * g.Co * Hp * Wp;
    for (long long i = blockIdx.x * (long long)kThreads + threadIdx.x; i < total; i += (long long)gridDim.x * kThreads) {
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

// The same behind both gradients of a layer: one launch redoes dx and doff.
__global__ void __launch_bounds__(kThreads) mex_redo_bwd(MexGeo g, const float* __restrict__ x, const float* __restrict__ off, const float* __restrict__ y,
                                                         const float* __restrict__ dy, float* __restrict__ dx, float* __restrict__ doff, int accumulate,
                                                         const int* __restrict__ gate) {
    stream_order();
    __shared__ float smem[kThreads];
    if ((gate[0] | gate[1]) == 0) return;
    const long long total = (long long)g.B * g.C * g.H * g.W;
    for (long long idx = blockIdx.x * (long long)kThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kThreads)
        dx[idx] = mex_exact_dx(g, x, off, y, dy, idx);
    const long long triples = (long long)g.R * g.M * g.K;
    for (long long rmk = blockIdx.x; rmk < triples; rmk += gridDim.x) {
        const int k = int(rmk % g.K), m = int((rmk / g.K) % g.M), r = int(rmk / ((long long)g.K * g.M));
        float sum = 0.f;
        for (long long i = threadIdx.x; i < (long long)g.B * g.rs; i += kThreads) sum += mex_exact_doff_term(g, x, off[rmk], y, dy, r, m, k, i);
        const float rsum = block_sum(sum, smem);
        if (threadIdx.x == 0) doff[rmk] = accumulate ? doff[rmk] + rsum : rsum;
    }
}

// gated: the launch follows a factorised kernel and does work only if that one raised the safety flag; a grid that
// just fills the GPU keeps the usual case (every CTA reads the flag and returns) at a few microseconds
inline int grid_for(long long total, bool gated = false) {
    const long long blocks = (total + kThreads - 1) / kThreads;
    const long long cap = (long long)device_sm_count() * (gated ? 8 : 32);
    return int(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace

#define SIMNETS_DTYPE_SWITCH(is_f64, CALL32, CALL64) do { if (is_f64) { CALL64; } else { CALL32; } } while (0)

cudaError_t launch_sim_fwd_direct(const SimGeo& g, bool f64, const void* x, const void* t, const void* w, void* y, cudaStream_t s,
                                  const int* gate) {
    const long long total = (long long)g.B * g.M * g.N;
    if (total == 0) return cudaSuccess;
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
    const int blocks = g.M * g.K;
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(sim_dparams_direct<float>, blocks, kThreads, 0, s)(g, (const float*)x, (const float*)t, (const float*)w, (const float*)dy, (float*)dt, (float*)dw, accumulate, make_fastdiv(g.N), make_fastdiv(g.ow))),
        (in_stream_order(sim_dparams_direct<double>, blocks, kThreads, 0, s)(g, (const double*)x, (const double*)t, (const double*)w, (const double*)dy, (double*)dt, (double*)dw, accumulate, make_fastdiv(g.N), make_fastdiv(g.ow))));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_fwd_direct(const MexGeo& g, bool f64, const void* x, const void* off, void* y, cudaStream_t s, const int* gate) {
    const long long total = (long long)g.B * g.M * g.N;
    if (total == 0) return cudaSuccess;
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(mex_fwd_direct<float>, grid_for(total, gate != nullptr), kThreads, 0, s)(g, (const float*)x, (const float*)off, (float*)y, gate)),
        (in_stream_order(mex_fwd_direct<double>, grid_for(total), kThreads, 0, s)(g, (const double*)x, (const double*)off, (double*)y, gate)));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_redo_fwd_pool(const MexGeo& g, const float* x, const float* off, float* y, float* pooled, cudaStream_t s, const int* gate) {
    in_stream_order(mex_redo_fwd_pool, grid_for((long long)g.B * g.M * g.N / 4, true), kThreads, 0, s)(g, x, off, y, pooled, gate);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_redo_bwd(const MexGeo& g, const float* x, const float* off, const float* y, const float* dy, float* dx, float* doff, bool accumulate,
                                cudaStream_t s, const int* gate) {
    in_stream_order(mex_redo_bwd, device_sm_count() * 8, kThreads, 0, s)(g, x, off, y, dy, dx, doff, int(accumulate), gate);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mex_dx_direct(const MexGeo& g, bool f64, const void* x, const void* off, const void* y, const void* dy, void* dx, cudaStream_t s, const int* gate) {
    const long long total = (long long)g.B * g.C * g.H * g.W;
    if (total == 0) return cudaSuccess;
    SIMNETS_DTYPE_SWITCH(f64,
        (in_stream_order(mex_dx_direct<float>, grid_for(total, gate != nullptr), kThreads, 0, s)(g, (const float*)x, (const float*)off, (const float*)y, (const float*)dy, (float*)dx, gate)),
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
