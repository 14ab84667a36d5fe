// One EM step of a diagonal Gaussian mixture over the patches of a batch (float32): the statistics of every component from the
// current means and covariances, and the new parameters from them.  The distances are the L2 Similarity forward kernel and the
// moments its parameter-gradient kernel; what lies between and around them is here.
//
// Bound: HBM.  The log-likelihoods of 64 components over 512 x 30 x 30 patches are 118 MB; the element-wise passes, the softmax
// over a strided axis and the sum over positions as separate tensor operations took 435 us of a 935 us step.  Here a thread owns
// a position with its k values in registers (up to 64 components: one read, one exponential each, one write in place; more are
// read twice) and adds each responsibility to a sum of its own in shared memory.  The whole step: 935 -> 423 us.
#include "kernels.cuh"

namespace simnets {
namespace {

constexpr int kMixThreads = 128;
constexpr size_t kMixSmem = 100 * 1024;

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
// over the CTA's positions.
template <int KT>
__global__ void __launch_bounds__(kMixThreads) mixture_responsibilities(long long P, int k, int N, float* __restrict__ score, const float* __restrict__ logdet,
                                                                        float* __restrict__ part) {
    stream_order();
    extern __shared__ float sm[];                       // [k][128] sums, [k] log-determinants
    float* ld = sm + k * kMixThreads;
    for (int i = threadIdx.x; i < k * kMixThreads; i += kMixThreads) sm[i] = 0.f;
    for (int c = threadIdx.x; c < k; c += kMixThreads) ld[c] = logdet[c];
    __syncthreads();
    for (long long j = (long long)blockIdx.x * kMixThreads + threadIdx.x; j < P; j += (long long)gridDim.x * kMixThreads) {
        const long long n = j / N;
        float* p = score + n * k * N + (j - n * N);
        float hi = -CUDART_INF_F, sum = 0.f;
        if (KT > 0) {                                   // KT >= k
            float v[KT > 0 ? KT : 1];
#pragma unroll
            for (int c = 0; c < KT; ++c) v[c] = c < k ? p[(long long)c * N] : -CUDART_INF_F;
#pragma unroll
            for (int c = 0; c < KT; ++c) {
                if (c < k) v[c] = 0.5f * (v[c] - ld[c]);
                hi = fmaxf(hi, v[c]);
            }
#pragma unroll
            for (int c = 0; c < KT; ++c) { v[c] = c < k ? expf(v[c] - hi) : 0.f; sum += v[c]; }
            const float inv = 1.f / sum;
#pragma unroll
            for (int c = 0; c < KT; ++c) {
                if (c >= k) break;
                const float r = v[c] * inv;
                p[(long long)c * N] = r;
                sm[c * kMixThreads + threadIdx.x] += r;
            }
            continue;
        }
        // (the running maximum may still be -inf, components so far away that their distance overflowed: exp(-inf - 0) adds nothing)
        const auto above = [](float top) { return top > -CUDART_INF_F ? top : 0.f; };
        int c = 0;
        for (; c + 8 <= k; c += 8) {
            float v[8], top = hi;
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = 0.5f * (p[(long long)(c + u) * N] - ld[c + u]);
#pragma unroll
            for (int u = 0; u < 8; ++u) top = fmaxf(top, v[u]);
            const float ref = above(top);
            float add = 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) add += expf(v[u] - ref);
            sum = sum * expf(hi - ref) + add;
            hi = top;
        }
        for (; c < k; ++c) {
            const float v = 0.5f * (p[(long long)c * N] - ld[c]), top = fmaxf(hi, v), ref = above(top);
            sum = sum * expf(hi - ref) + expf(v - ref);
            hi = top;
        }
        const float inv = 1.f / sum;
#pragma unroll 8
        for (c = 0; c < k; ++c) {
            const float r = expf(0.5f * (p[(long long)c * N] - ld[c]) - hi) * inv;
            p[(long long)c * N] = r;
            sm[c * kMixThreads + threadIdx.x] += r;
        }
    }
    __syncthreads();
    // one warp per component, a quarter of them each
    for (int c = threadIdx.x >> 5; c < k; c += kMixThreads / 32) {
        float s = 0.f;
        for (int i = threadIdx.x & 31; i < kMixThreads; i += 32) s += sm[c * kMixThreads + i];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if ((threadIdx.x & 31) == 0) part[(size_t)blockIdx.x * k + c] = s;
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

size_t mix_smem(int k) { return sizeof(float) * (size_t)k * (kMixThreads + 1); }
int mix_ctas(const SimGeo& g) {
    const long long P = (long long)g.B * g.N, tiles = (P + kMixThreads - 1) / kMixThreads;
    const long long resident = (long long)device_sm_count() * std::max<long long>(1, std::min<long long>(12, (200 * 1024) / (long long)(mix_smem(g.M) + 1024)));
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
    return sim_use_tiled(g, f64, flags) && flags == 0 && g.mode == SIM_L2 && (long long)g.C * g.H * g.W < (1LL << 29) && mix_smem(g.M) <= kMixSmem;
}
size_t mixture_workspace_bytes(const SimGeo& g) { return mix_carve(g, nullptr).bytes; }

cudaError_t launch_mixture_statistics(const SimGeo& g, const float* x, const float* means, const float* covs, float* stats, void* ws, cudaStream_t s) {
    const MixWs w = mix_carve(g, ws);
    const int n = g.M * g.K;
    in_stream_order(mixture_prep, g.M, 128, 0, s)(g.K, covs, w.scales, w.logdet);
    cudaError_t e = launch_sim_fwd_tiled(g, x, means, w.scales, w.score, w.sim, 0, s);
    if (e != cudaSuccess) return e;
    const int ctas = mix_ctas(g);
#define MIX(KT) in_stream_order(mixture_responsibilities<KT>, ctas, kMixThreads, mix_smem(g.M), s)((long long)g.B * g.N, g.M, g.N, w.score, w.logdet, w.part)
    if (g.M <= 16) MIX(16); else if (g.M <= 32) MIX(32); else if (g.M <= 48) MIX(48); else if (g.M <= 64) MIX(64);
    else {
        e = cudaFuncSetAttribute(mixture_responsibilities<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kMixSmem));
        if (e != cudaSuccess) return e;
        MIX(0);
    }
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
