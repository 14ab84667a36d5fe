// One EM step of a diagonal Gaussian mixture over the patches of a batch (float32): the statistics of every component from the
// current means and covariances, and the new parameters from them.  The distances are the L2 Similarity forward kernel and the
// moments its parameter-gradient kernel; what lies between and around them is here.
//
// Bound: HBM, 36 us for the log-likelihoods of 64 components over 512 x 30 x 30 patches (118 MB read and written in place).  G lanes share
// a position, each with every G-th component in registers: a maximum and a sum over G lanes, and since a lane always has the same
// components, their masses stay in its registers over all positions.  A thread with all 64 components of a position (251 registers,
// eight warps per SM, masses in shared memory) took 101 us; this takes 57 (24 warps per SM; with 126 registers, 16 warps, 67).
#include "kernels.cuh"

namespace simnets {
namespace {

constexpr int kMixThreads = 128, kMixMost = 198;          // (198: what the first form of this had room for)

// 1 / covariance and log-determinant of every component
__global__ void __launch_bounds__(128) mixture_prep(int taps, const float* __restrict__ covs, float* __restrict__ scales, float* __restrict__ logdet) {
    stream_order();
    __shared__ float red[128];
    const size_t row = (size_t)blockIdx.x * taps;
    float s = 0.f;
    for (int i = threadIdx.x; i < taps; i += 128) {
        const float v = covs[row + i];
        scales[row + i] = 1.f / v;
        s += logf(v);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int d = 64; d > 0; d >>= 1) {
        if (threadIdx.x < d) red[threadIdx.x] += red[threadIdx.x + d];
        __syncthreads();
    }
    if (threadIdx.x == 0) logdet[blockIdx.x] = red[0];
}

// score[b][c][p] = -sum scale (patch - mean)^2 becomes the responsibility softmax_c(score / 2 - logdet / 2); part[cta][c] = sum
// over the CTA's positions.  Lane l of a warp: position l mod (32 / G) of its run, components l / (32 / G) + G i, KT of them.
template <int G, int KT>
__global__ void __launch_bounds__(kMixThreads, 6) mixture_responsibilities(long long P, int k, FastDiv f_N, float* __restrict__ score, const float* __restrict__ logdet,
                                                                        float* __restrict__ part) {
    stream_order();
    constexpr int RUN = 32 / G, WARPS = kMixThreads / 32;
    __shared__ float red[WARPS][G * KT], ld[G * KT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, first = lane / RUN;
    const long long N = f_N.d, step = G * N;
    for (int i = threadIdx.x; i < G * KT; i += kMixThreads) ld[i] = i < k ? logdet[i] : 0.f;
    __syncthreads();
    float mass[KT];
#pragma unroll
    for (int i = 0; i < KT; ++i) mass[i] = 0.f;
    for (long long j0 = ((long long)blockIdx.x * WARPS + warp) * RUN; j0 < P; j0 += (long long)gridDim.x * WARPS * RUN) {
        const long long j = j0 + lane % RUN;
        const bool live = j < P;
        const long long n = !live ? 0 : P <= 0x7fffffffLL ? (long long)fast_div(uint32_t(j), f_N) : j / N;
        float* p = score + n * k * N + (live ? j - n * N : 0) + first * N;
        const float* q = p;
        float v[KT], hi = -CUDART_INF_F, sum = 0.f;
#pragma unroll
        for (int i = 0; i < KT; ++i, q += step) v[i] = live && first + G * i < k ? *q : -CUDART_INF_F;
#pragma unroll
        for (int i = 0; i < KT; ++i) { v[i] = 0.5f * (v[i] - ld[first + G * i]); hi = fmaxf(hi, v[i]); }
#pragma unroll
        for (int d = RUN; d < 32; d <<= 1) hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
#pragma unroll
        for (int i = 0; i < KT; ++i) { v[i] = first + G * i < k ? expf(v[i] - hi) : 0.f; sum += v[i]; }
#pragma unroll
        for (int d = RUN; d < 32; d <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        if (!live) continue;
        const float inv = 1.f / sum;
        asm volatile("" : "+l"(p));                     // (sixteen addresses kept from the reads: 126 registers instead of 80)
#pragma unroll
        for (int i = 0; i < KT; ++i, p += step)
            if (first + G * i < k) {
                const float r = v[i] * inv;
                *p = r;
                mass[i] += r;
            }
    }
#pragma unroll
    for (int i = 0; i < KT; ++i) {
        float s = mass[i];
#pragma unroll
        for (int d = RUN / 2; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane % RUN == 0) red[warp][first + G * i] = s;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < k; c += kMixThreads) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) s += red[w][c];
        part[(size_t)blockIdx.x * k + c] = s;
    }
}

__global__ void __launch_bounds__(128) mixture_mass(int ctas, int k, const float* __restrict__ part, float* __restrict__ mass) {
    stream_order();
    __shared__ float red[128];
    float s = 0.f;
    for (int i = threadIdx.x; i < ctas; i += 128) s += part[(size_t)i * k + blockIdx.x];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int d = 64; d > 0; d >>= 1) {
        if (threadIdx.x < d) red[threadIdx.x] += red[threadIdx.x + d];
        __syncthreads();
    }
    if (threadIdx.x == 0) mass[blockIdx.x] = red[0];
}

// mean + shift / mass; second moment about the NEW mean plus the floor
__global__ void __launch_bounds__(256) mixture_parameters(int n, int taps, float min_var, const float* __restrict__ stats, const float* __restrict__ means,
                                                          float* __restrict__ new_means, float* __restrict__ new_covs) {
    stream_order();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const float mass = fmaxf(stats[2 * n + i / taps], 1.17549435e-38f), step = stats[i] / mass;
    new_covs[i] = stats[n + i] / mass - step * step + min_var;
    new_means[i] = means[i] + step;
}

// lanes per position: at most sixteen components each
int mix_lanes(int k) { return k <= 64 ? 4 : (k <= 128 ? 8 : 16); }
int mix_ctas(const SimGeo& g) {
    const long long P = (long long)g.B * g.N, per = kMixThreads / mix_lanes(g.M), tiles = (P + per - 1) / per, resident = (long long)device_sm_count() * 6;
    const long long rounds = (tiles + resident - 1) / resident;
    return int((tiles + rounds - 1) / rounds);
}

struct MixWs { float *score, *scales, *logdet, *part; void* sim; size_t bytes; };
MixWs mix_carve(const SimGeo& g, void* base) {
    MixWs w;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t bytes) { char* r = p ? p + off : nullptr; off += (bytes + 255) & ~size_t(255); return r; };
    w.score = reinterpret_cast<float*>(take(sizeof(float) * (size_t)g.B * g.M * g.N));
    w.scales = reinterpret_cast<float*>(take(sizeof(float) * (size_t)g.M * g.K));
    w.logdet = reinterpret_cast<float*>(take(sizeof(float) * g.M));
    w.part = reinterpret_cast<float*>(take(sizeof(float) * (size_t)mix_ctas(g) * g.M));
    w.sim = take(sim_workspace_bytes(g, false, 0));
    w.bytes = off;
    return w;
}

}  // namespace

bool mixture_shape(const SimGeo& g, bool f64, uint32_t flags) {
    return sim_use_tiled(g, f64, flags) && flags == 0 && g.mode == SIM_L2 && sim_offsets_below(g, 1LL << 29) && g.M <= kMixMost;
}
size_t mixture_workspace_bytes(const SimGeo& g) { return mix_carve(g, nullptr).bytes; }

cudaError_t launch_mixture_statistics(const SimGeo& g, const float* x, const float* means, const float* covs, float* stats, void* ws, cudaStream_t s) {
    const MixWs w = mix_carve(g, ws);
    const int n = g.M * g.K;
    in_stream_order(mixture_prep, g.M, 128, 0, s)(g.K, covs, w.scales, w.logdet);
    cudaError_t e = launch_sim_fwd_tiled(g, x, means, w.scales, w.score, w.sim, 0, s);
    if (e != cudaSuccess) return e;
    const int ctas = mix_ctas(g);
    const FastDiv f_N = make_fastdiv(g.N);
#define MIX(G, KT) in_stream_order(mixture_responsibilities<G, KT>, ctas, kMixThreads, 0, s)((long long)g.B * g.N, g.M, f_N, w.score, w.logdet, w.part)
    if (g.M <= 16) MIX(4, 4); else if (g.M <= 32) MIX(4, 8); else if (g.M <= 48) MIX(4, 12); else if (g.M <= 64) MIX(4, 16);
    else if (g.M <= 96) MIX(8, 12); else if (g.M <= 128) MIX(8, 16); else MIX(16, 13);
#undef MIX
    in_stream_order(mixture_mass, g.M, 128, 0, s)(ctas, g.M, w.part, stats + 2 * n);
    count_launch(3);
    return launch_sim_dparams_tiled(g, x, means, nullptr, w.score, stats, stats + n, false, w.sim, s);      // (no weights: the plain sums)
}

cudaError_t launch_mixture_parameters(int k, int taps, float min_var, const float* stats, const float* means, float* new_means, float* new_covs, cudaStream_t s) {
    const int n = k * taps;
    in_stream_order(mixture_parameters, (n + 255) / 256, 256, 0, s)(n, taps, min_var, stats, means, new_means, new_covs);
    count_launch();
    return cudaGetLastError();
}

}  // namespace simnets
