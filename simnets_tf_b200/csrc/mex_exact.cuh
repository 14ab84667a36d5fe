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

// every tap of the patch at output (c, h, w) in order: visit(value, offset).  (Loops instead of two divisions and remainders a tap: a
// forward pass of 128 instances over 64 taps, 16 x 32 x 32 positions, 743 -> 266 us.)  AHEAD: blocks of one pixel are read eight taps at a
// time, for grids of few warps (64 x 8 x 8 positions in 128 CTAs 308 -> 208 us; full grids lose by its registers, 266 -> 420).
template <bool AHEAD, typename T, class Visit>
__device__ __forceinline__ void mex_taps(const MexGeo& g, const T* __restrict__ xs, const T* __restrict__ o, int c, int h, int w, T oob, const Visit& visit) {
    const int c0 = c * g.sc - g.pc, h0 = h * g.sh - g.ph, w0 = w * g.sw - g.pw;
    if (g.bh * g.bw == 1) {
        const bool in = h0 >= 0 && h0 < g.H && w0 >= 0 && w0 < g.W;
        const long long hw = (long long)g.H * g.W;
        const T* p = xs + (long long)c0 * hw + (long long)h0 * g.W + w0;
        if (!AHEAD) {
#pragma unroll 8
            for (int k = 0; k < g.bc; ++k) visit(in && c0 + k >= 0 && c0 + k < g.C ? p[k * hw] : oob, o[k]);
            return;
        }
        for (int k0 = 0; k0 < g.bc; k0 += 8) {
            T v[8], q[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int k = k0 + u, cc = c0 + k;
                v[u] = oob;
                q[u] = T(0);
                if (k < g.bc) q[u] = o[k];
                if (k < g.bc && in && cc >= 0 && cc < g.C) v[u] = p[k * hw];
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (k0 + u < g.bc) visit(v[u], q[u]);
        }
        return;
    }
    for (int cc = c0; cc < c0 + g.bc; ++cc)
        for (int hh = h0; hh < h0 + g.bh; ++hh, o += g.bw) {
            const bool row = cc >= 0 && cc < g.C && hh >= 0 && hh < g.H;
            const T* p = xs + ((long long)cc * g.H + hh) * g.W + w0;
#pragma unroll 2
            for (int k = 0; k < g.bw; ++k) visit(row && w0 + k >= 0 && w0 + k < g.W ? p[k] : oob, o[k]);
        }
}

// y[idx]
template <typename T, bool AHEAD = false>
__device__ __forceinline__ T mex_exact_y(const MexGeo& g, const T* __restrict__ x, const T* __restrict__ off, long long idx) {
    const T oob = T(g.oob), eps = T(g.eps), cst = T(g.cst);
    const int j = int(idx % g.N);
    const long long q = idx / g.N;
    const int m = int(q % g.M), n = int(q / g.M);
    const int w = j % g.Wo, h = (j / g.Wo) % g.Ho, c = j / (g.Wo * g.Ho);
    const T* xs = x + (size_t)n * g.C * g.H * g.W;
    const T* o = off + ((size_t)mex_region_of(g, c, h, w) * g.M + m) * g.K;
    T mx = eps > T(0) ? -pos_inf<T>() : pos_inf<T>();
    mex_taps<AHEAD>(g, xs, o, c, h, w, oob, [&](T t, T q) {
        const T v = q + t;
        // comparisons written as the host library's max/min: a NaN operand never replaces mx
        if (eps > T(0)) { if (mx < v) mx = v; } else { if (v < mx) mx = v; }
    });
    if (!g.finite) return mx;
    T sum = T(0);
    mex_taps<AHEAD>(g, xs, o, c, h, w, oob, [&](T t, T q) { sum += dev_exp(eps * (t + q - mx) + cst); });
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
    // the taps of each axis that meet this value, in order: one residue of the stride, outputs descending
    const int cp = c0 + g.pc, hp = h0 + g.ph, wp = w0 + g.pw;
    for (int kc = cp % g.sc, c = cp / g.sc; kc < g.bc && c >= 0; kc += g.sc, --c) {
        if (c >= g.Co) continue;
        for (int kh = hp % g.sh, h = hp / g.sh; kh < g.bh && h >= 0; kh += g.sh, --h) {
            if (h >= g.Ho) continue;
            for (int kw = wp % g.sw, w = wp / g.sw; kw < g.bw && w >= 0; kw += g.sw, --w) {
                if (w >= g.Wo) continue;
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
    const int n = i <= 0x7fffffffLL ? int(fast_div(uint32_t(i), g.f_rs)) : int(i / g.rs), l = int(i - (long long)n * g.rs);
    int c, h, w;
    if (!mex_region_chw(g, r, l, c, h, w)) return T(0);
    const int j = (c * g.Ho + h) * g.Wo + w;
    const T v = mex_tap(g, x + (size_t)n * g.C * g.H * g.W, c, h, w, k, T(g.oob));
    return mex_weight(g, T(g.eps), T(g.cst), v, o, y[((size_t)n * g.M + m) * g.N + j], dy[mex_dy_base(g, n, j) + (long long)m * g.Ng]);
}

}  // namespace
}  // namespace simnets
