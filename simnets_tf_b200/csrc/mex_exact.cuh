// The MEX operators term by term, one value at a time: what the reference's element functors compute
// (HUJI-Deep/simnets-tf include/utils/mex_utils.hpp:10-56), in its summation order.  Used by the shape-agnostic kernels and by
// the factorised kernels of mex_gemm.cu for offsets they cannot take.
#pragma once
#include "kernels.cuh"

namespace simnets {
namespace {

__device__ __forceinline__ float dev_exp(float v) { return expf(v); }
__device__ __forceinline__ double dev_exp(double v) { return exp(v); }
__device__ __forceinline__ float dev_log(float v) { return logf(v); }
__device__ __forceinline__ double dev_log(double v) { return log(v); }
template <typename T> __device__ __forceinline__ T pos_inf() { return T(CUDART_INF); }

template <typename T>
__device__ __forceinline__ T mex_tap(const MexGeo& g, const T* __restrict__ xs, int c, int h, int w, int k, T oob) {
    const int kw = k % g.bw, kh = (k / g.bw) % g.bh, kc = k / (g.bw * g.bh);
    const int cc = c * g.sc - g.pc + kc, hh = h * g.sh - g.ph + kh, ww = w * g.sw - g.pw + kw;
    return (cc >= 0 && cc < g.C && hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) ? xs[((size_t)cc * g.H + hh) * g.W + ww] : oob;
}

// y[idx]
template <typename T>
__device__ __forceinline__ T mex_exact_y(const MexGeo& g, const T* __restrict__ x, const T* __restrict__ off, long long idx) {
    const T oob = T(g.oob), eps = T(g.eps), cst = T(g.cst);
    const int j = int(idx % g.N);
    const long long q = idx / g.N;
    const int m = int(q % g.M), n = int(q / g.M);
    const int w = j % g.Wo, h = (j / g.Wo) % g.Ho, c = j / (g.Wo * g.Ho);
    const T* xs = x + (size_t)n * g.C * g.H * g.W;
    const T* o = off + ((size_t)mex_region_of(g, c, h, w) * g.M + m) * g.K;
    T mx = eps > T(0) ? -pos_inf<T>() : pos_inf<T>();
    for (int k = 0; k < g.K; ++k) {
        const T v = o[k] + mex_tap(g, xs, c, h, w, k, oob);
        // comparisons written as the host library's max/min: a NaN operand never replaces mx
        if (eps > T(0)) { if (mx < v) mx = v; } else { if (v < mx) mx = v; }
    }
    if (!g.finite) return mx;
    T sum = T(0);
    for (int k = 0; k < g.K; ++k) sum += dev_exp(eps * (mex_tap(g, xs, c, h, w, k, oob) + o[k] - mx) + cst);
    return mx + dev_log(sum) / eps;
}

template <typename T>
__device__ __forceinline__ T mex_weight(const MexGeo& g, T eps, T cst, T data, T offset, T top, T top_diff) {
    if (g.finite) return top_diff * dev_exp(eps * (data + offset - top) + cst);
    return top_diff * T((data + offset) == top);
}

// dx[idx]
template <typename T>
__device__ __forceinline__ T mex_exact_dx(const MexGeo& g, const T* __restrict__ x, const T* __restrict__ off, const T* __restrict__ y,
                                          const T* __restrict__ dy, long long idx) {
    const T eps = T(g.eps), cst = T(g.cst);
    const int w0 = int(idx % g.W);
    long long q = idx / g.W;
    const int h0 = int(q % g.H); q /= g.H;
    const int c0 = int(q % g.C), n = int(q / g.C);
    const T v = x[idx];
    const T* y_n = y + (size_t)n * g.M * g.N;
    T total_sum = T(0);
    for (int kc = 0; kc < g.bc; ++kc) {
        const int cp = c0 + g.pc - kc;
        if (cp < 0 || cp % g.sc != 0 || cp / g.sc >= g.Co) continue;
        for (int kh = 0; kh < g.bh; ++kh) {
            const int hp = h0 + g.ph - kh;
            if (hp < 0 || hp % g.sh != 0 || hp / g.sh >= g.Ho) continue;
            for (int kw = 0; kw < g.bw; ++kw) {
                const int wp_ = w0 + g.pw - kw;
                if (wp_ < 0 || wp_ % g.sw != 0 || wp_ / g.sw >= g.Wo) continue;
                const int c = cp / g.sc, h = hp / g.sh, w = wp_ / g.sw;
                const int k = (kc * g.bh + kh) * g.bw + kw;
                const int j = (c * g.Ho + h) * g.Wo + w;
                const T* o = off + (size_t)mex_region_of(g, c, h, w) * g.M * g.K + k;
                const T* g_j = dy + mex_dy_base(g, n, j);
                T sum = T(0);
                for (int m = 0; m < g.M; ++m)
                    sum += mex_weight(g, eps, cst, v, o[(size_t)m * g.K], y_n[(size_t)m * g.N + j], g_j[(size_t)m * g.Ng]);
                total_sum += sum;
            }
        }
    }
    return total_sum;
}

// term of position i (0 <= i < B * region_size) in doff[r, m, k]
template <typename T>
__device__ __forceinline__ T mex_exact_doff_term(const MexGeo& g, const T* __restrict__ x, T o, const T* __restrict__ y, const T* __restrict__ dy,
                                                 int r, int m, int k, long long i) {
    const int l = int(i % g.rs), n = int(i / g.rs);
    const int j = mex_region_position(g, r, l);
    if (j < 0) return T(0);
    const int w = j % g.Wo, h = (j / g.Wo) % g.Ho, c = j / (g.Wo * g.Ho);
    const T v = mex_tap(g, x + (size_t)n * g.C * g.H * g.W, c, h, w, k, T(g.oob));
    return mex_weight(g, T(g.eps), T(g.cst), v, o, y[((size_t)n * g.M + m) * g.N + j], dy[mex_dy_base(g, n, j) + (long long)m * g.Ng]);
}

}  // namespace
}  // namespace simnets
