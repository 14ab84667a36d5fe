// The Similarity input gradient term by term, one value at a time: what the reference's element functors compute
// (HUJI-Deep/simnets-tf include/utils/similarity_utils.hpp:17-150), in its summation order.  Used by the shape-agnostic kernels
// and by the gather kernels of sim_dx.cu for values that their padding cannot take.
#pragma once
#include "kernels.cuh"

namespace simnets {
namespace {

template <typename T> __device__ __forceinline__ bool is_nan(T v) { return v != v; }
template <typename T> __device__ __forceinline__ T sign_of(T v) { return T((T(0) < v) - (v < T(0))); }

__device__ __forceinline__ float dev_abs(float v) { return fabsf(v); }
__device__ __forceinline__ double dev_abs(double v) { return fabs(v); }

// dx[idx]
template <typename T>
__device__ __forceinline__ T sim_exact_dx(const SimGeo& g, const T* __restrict__ x, const T* __restrict__ tm, const T* __restrict__ wt,
                                          const T* __restrict__ dy, long long idx) {
    const int w0 = int(idx % g.W);
    long long q = idx / g.W;
    const int h0 = int(q % g.H); q /= g.H;
    const int c = int(q % g.C), n = int(q / g.C);
    const T v = x[idx];
    const T* g_n = dy + (size_t)n * g.M * g.N;
    T total_sum = T(0);
    for (int kh = 0; kh < g.bh; ++kh) {
        const int hp = h0 + g.ph - kh;
        if (hp < 0 || hp % g.sh != 0) continue;
        const int ho = hp / g.sh;
        if (ho >= g.oh) continue;
        for (int kw = 0; kw < g.bw; ++kw) {
            const int wp_ = w0 + g.pw - kw;
            if (wp_ < 0 || wp_ % g.sw != 0) continue;
            const int wo = wp_ / g.sw;
            if (wo >= g.ow) continue;
            const int k = (c * g.bh + kh) * g.bw + kw;
            const int j = ho * g.ow + wo;
            T sum = T(0);
            for (int m = 0; m < g.M; ++m) {
                const T wr = wt[(size_t)m * g.K + k];
                const T t = tm[(size_t)m * g.K + k], w = g.absw ? dev_abs(wr) : wr, err = g_n[(size_t)m * g.N + j];
                switch (g.mode) {
                case SIM_L1: sum += err * w * sign_of(t - v); break;
                case SIM_L1_SKIP: if (!is_nan(v)) sum += err * w * sign_of(t - v); break;
                case SIM_L2: sum += T(2) * err * w * (t - v); break;
                case SIM_L2N: sum += T(0.5) * (T(2) * err * w * (t - v)); break;
                default: if (!is_nan(v)) sum += T(0.5) * (T(2) * err * w * (t - v)); break;
                }
            }
            total_sum += sum;
        }
    }
    return total_sum;
}

}  // namespace
}  // namespace simnets
