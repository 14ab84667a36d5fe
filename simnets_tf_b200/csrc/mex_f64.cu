// MEX forward, input gradient and offsets gradient in double precision, factorised like the float32 kernels of mex_tiled.cu:
//
//     S[m,j] = sum_k Eo[m,k] Ex[k,j],      y = mx + mo + (log S + c) / eps
//     dx[tap k of j] = Ex[k,j] sum_m Eo[m,k] Q[m,j],      doff[m,k] = Eo[m,k] sum_j Q[m,j] Ex[k,j]
//
// with Ex = exp(eps (x - mx)), Eo = exp(eps (o - mo)), Q = dy exp(eps (mx + mo - y) + c): M K + K N exponentials instead of one
// per (m, k, j) term.  An exponential costs a few dozen double-precision operations, so the term-by-term kernels of
// direct_kernels.cu were bound by it (layer of 128 instances over 64 channels of 32x32 pixels, batch 12: forward 874 us,
// offsets gradient 1461 us; here 54 and 44).  The factorised form is safe while |eps| * spread(offsets) stays below kSafeSpread64; a status word
// says so otherwise (or when an offset is not finite), and the term-by-term kernels behind these, gated on it, do the work.
//
// One tile kernel serves the three contractions: 64 x 64 outputs, 4 x 4 per thread, 16 steps of the reduction per chunk, double
// buffered.  Small layers (a classifier head has 12 x 10 outputs and 8192 taps) split the reduction over CTAs; the partial sums
// are added in split order by the finishing kernels.
#include "kernels.cuh"

namespace simnets {
namespace {

constexpr double kSafeSpread64 = 300.0;              // exp(-300) is far from the smallest double, and so are products of two
constexpr int kT = 64, kQ = 16, kThreads64 = 256, kLd = kT + 2;

struct Ws64 {
    int* flag;           // [2]
    double *mo, *lse;    // [R][M]
    double *eo;          // [R][M][K]
    double *offn;        // [R][M][K] offsets minus their row's log-sum-exp, when they come raw
    double *mx;          // [B][N]
    double *part;        // split partial sums
    size_t bytes;
};
enum Op64 { kFwd, kDx, kDoff };

struct Split64 { long long it, jt; int steps, splits; };         // tiles along the two output axes (per region), reduction length
__host__ Split64 split_of(const MexGeo& g, Op64 op) {
    const long long P = (long long)g.B * g.rs;
    const long long rows = op == kDx ? g.K : g.M, cols = op == kDoff ? g.K : P, steps = op == kFwd ? g.K : (op == kDx ? g.M : P);
    Split64 s;
    s.it = (rows + kT - 1) / kT; s.jt = (cols + kT - 1) / kT;
    const long long tiles = s.it * s.jt * g.R, chunks = (steps + kQ - 1) / kQ;
    // two CTAs per SM, each with at least four chunks
    long long n = tiles >= 2LL * device_sm_count() ? 1 : (2LL * device_sm_count()) / tiles;
    n = std::max<long long>(1, std::min(n, (chunks + 3) / 4));
    s.steps = int(std::min<long long>(steps, 0x7fffffff));
    s.splits = int(n);
    return s;
}
__host__ size_t part_doubles(const MexGeo& g, Op64 op) {
    const Split64 s = split_of(g, op);
    const size_t n = op == kDoff ? (size_t)g.M * g.K : (size_t)(op == kDx ? g.K : g.M) * ((size_t)g.B * g.rs);
    return op == kDoff || s.splits > 1 ? n * g.R * s.splits : 0;
}
__host__ Ws64 carve64(const MexGeo& g, void* base) {
    Ws64 w;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t doubles) { char* r = p ? p + off : nullptr; off += (doubles * 8 + 255) & ~size_t(255); return reinterpret_cast<double*>(r); };
    w.flag = reinterpret_cast<int*>(take(2));
    w.mo = take((size_t)g.R * g.M);
    w.lse = take((size_t)g.R * g.M);
    w.eo = take((size_t)g.R * g.M * g.K);
    w.offn = take((size_t)g.R * g.M * g.K);
    w.mx = take((size_t)g.B * g.N);
    w.part = take(std::max(part_doubles(g, kFwd), std::max(part_doubles(g, kDx), part_doubles(g, kDoff))));
    w.bytes = off;
    return w;
}

__device__ __forceinline__ double block_reduce(double v, double* red, bool sum) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] = sum ? red[threadIdx.x] + red[threadIdx.x + s] : fmax(red[threadIdx.x], red[threadIdx.x + s]);
        __syncthreads();
    }
    v = red[0];
    __syncthreads();
    return v;
}

// One CTA per (region, instance): reference value, Eo, log-sum-exp and normalised row of raw offsets, the safety verdict.
__global__ void __launch_bounds__(256) mex_prep64(MexGeo g, const double* __restrict__ off, double* __restrict__ mo, double* __restrict__ eo,
                                                  double* __restrict__ offn, double* __restrict__ lse_out, int* __restrict__ flag, int normalize) {
    stream_order();
    __shared__ double red[256];
    const size_t row = (size_t)blockIdx.x * g.K;
    double hi = -CUDART_INF, lo = -CUDART_INF;            // (lo: maximum of the negated values)
    int bad = 0;
    for (int k = threadIdx.x; k < g.K; k += 256) {
        const double v = off[row + k];
        if (!isfinite(v)) bad = 1;
        hi = fmax(hi, v); lo = fmax(lo, -v);
    }
    bad = __syncthreads_or(bad);
    hi = block_reduce(hi, red, false);
    lo = -block_reduce(lo, red, false);
    const double ref = g.eps > 0 ? hi : lo;
    double lse = 0;
    if (normalize) {
        const double base = isfinite(hi) ? hi : 0.0;      // as a stable log-sum-exp treats infinite maxima
        double sum = 0;
        for (int k = threadIdx.x; k < g.K; k += 256) sum += exp(off[row + k] - base);
        lse = base + log(block_reduce(sum, red, true));
        for (int k = threadIdx.x; k < g.K; k += 256) offn[row + k] = off[row + k] - lse;
    }
    if (threadIdx.x == 0) {
        mo[blockIdx.x] = ref - lse;
        lse_out[blockIdx.x] = lse;
        if (bad || !(fabs(g.eps) * (hi - lo) <= kSafeSpread64)) atomicOr(flag, 1);
    }
    for (int k = threadIdx.x; k < g.K; k += 256) eo[row + k] = exp(g.eps * (off[row + k] - ref));
}

struct Col64 { long long base, gbase; int n, c0, h0, w0; double mx; };
__device__ __forceinline__ Col64 col64(const MexGeo& g, int r, long long jl, long long P, const double* __restrict__ mx) {
    Col64 c = {-1, 0, 0, 0, 0, 0, 0.0};
    if (jl >= P) return c;
    const int n = int(jl / g.rs), l = int(jl - (long long)n * g.rs);
    int cc, h, w;
    if (!mex_region_chw(g, r, l, cc, h, w)) return c;
    const int pos = (cc * g.Ho + h) * g.Wo + w;
    c.n = n; c.c0 = cc * g.sc - g.pc; c.h0 = h * g.sh - g.ph; c.w0 = w * g.sw - g.pw;
    c.base = (long long)n * g.M * g.N + pos;
    c.gbase = mex_dy_base(g, n, pos);
    c.mx = mx[(long long)n * g.N + pos];
    return c;
}
__device__ __forceinline__ long long tap_address(const MexGeo& g, const Col64& c, int k) {       // offset of tap k in x, or -1 outside
    const int kw = k % g.bw, q = k / g.bw, cc = c.c0 + q / g.bh, hh = c.h0 + q % g.bh, ww = c.w0 + kw;
    if (cc < 0 || cc >= g.C || hh < 0 || hh >= g.H || ww < 0 || ww >= g.W) return -1;
    return (((long long)c.n * g.C + cc) * g.H + hh) * g.W + ww;
}

// Largest (eps > 0) or smallest tap of every patch, NaN ignored; `lanes` positions per CTA of 256 threads, 256 / lanes slices of the taps.
__global__ void __launch_bounds__(256) mex_colmax64(MexGeo g, const double* __restrict__ x, double* __restrict__ mx, int lanes) {
    stream_order();
    __shared__ double red[256];
    const int slices = 256 / lanes, lane = threadIdx.x % lanes, slice = threadIdx.x / lanes;
    const long long total = (long long)g.B * g.N;
    const bool up = g.eps > 0;
    for (long long first = (long long)blockIdx.x * lanes; first < total; first += (long long)gridDim.x * lanes) {
        const long long idx = first + lane;
        double v = -CUDART_INF;                            // maximum of x or of -x
        if (idx < total) {
            const int pos = int(idx % g.N);
            Col64 c;
            c.n = int(idx / g.N);
            c.w0 = pos % g.Wo * g.sw - g.pw; c.h0 = pos / g.Wo % g.Ho * g.sh - g.ph; c.c0 = pos / (g.Wo * g.Ho) * g.sc - g.pc;
            for (int k = slice; k < g.K; k += slices) {
                const long long a = tap_address(g, c, k);
                const double t = a >= 0 ? x[a] : g.oob;
                v = fmax(v, up ? t : -t);
            }
        }
        red[threadIdx.x] = v;
        __syncthreads();
        for (int s = slices / 2; s > 0; s >>= 1) {
            if (slice < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s * lanes]);
            __syncthreads();
        }
        if (slice == 0 && idx < total) mx[idx] = up ? red[lane] : -red[lane];
        __syncthreads();
    }
}

// The three contractions.  Rows i: instances (forward, offsets gradient) or taps (input gradient); columns j: positions of one
// region (taps for the offsets gradient); reduction q: taps, instances, positions.
template <int OP>
__global__ void __launch_bounds__(kThreads64) mex_gemm64(MexGeo g, Split64 sp, const double* __restrict__ x, const double* __restrict__ eo,
                                                         const double* __restrict__ mo, const double* __restrict__ mx, const double* __restrict__ y,
                                                         const double* __restrict__ dy, double* __restrict__ out, double* __restrict__ part,
                                                         const int* __restrict__ flag) {
    stream_order();
    if (*flag) return;
    __shared__ __align__(16) double As[2][kQ][kLd], Bs[2][kQ][kLd];
    const long long P = (long long)g.B * g.rs;
    const int r = int(blockIdx.x % unsigned(g.R)), split = blockIdx.y;
    const long long tile = blockIdx.x / unsigned(g.R), it = tile % sp.it, jt = tile / sp.it;
    const long long i0 = it * kT, j0 = jt * kT;
    const int chunks = (sp.steps + kQ - 1) / kQ, c_begin = int((long long)chunks * split / sp.splits), c_end = int((long long)chunks * (split + 1) / sp.splits);
    const double* eor = eo + (size_t)r * g.M * g.K;
    const double* mor = mo + (size_t)r * g.M;
    // staging: four elements of each operand per thread, along the axis that is contiguous in memory
    const int e_f = threadIdx.x % kT, q_f = threadIdx.x / kT;         // element fastest: element e_f, steps q_f + 4 s
    const int q_s = threadIdx.x % kQ, e_s = threadIdx.x / kQ;         // step fastest: step q_s, elements e_s + 16 s
    const Col64 jc = OP != kDoff ? col64(g, r, j0 + e_f, P, mx) : Col64{-1, 0, 0, 0, 0, 0, 0.0};
    double ra[4], rb[4];
    auto weight = [&](const Col64& c, int m) {                        // Q[m, position]
        if (c.base < 0 || m >= g.M) return 0.0;
        return dy[c.gbase + (long long)m * g.Ng] * exp(g.eps * (c.mx + mor[m] - y[c.base + (long long)m * g.N]) + g.cst);
    };
    auto ex = [&](const Col64& c, int k) {                            // Ex[k, position]
        if (c.base < 0 || k >= g.K) return 0.0;
        const long long a = tap_address(g, c, k);
        return exp(g.eps * ((a >= 0 ? x[a] : g.oob) - c.mx));
    };
    auto fetch = [&](int chunk) {
        const int q0 = chunk * kQ;
        if (OP == kDoff) {
            const Col64 c = col64(g, r, q0 + q_s, P, mx);
#pragma unroll
            for (int s = 0; s < 4; ++s) { ra[s] = weight(c, int(i0) + e_s + 16 * s); rb[s] = ex(c, int(j0) + e_s + 16 * s); }
            return;
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (OP == kFwd) {
                const int m = int(i0) + e_s + 16 * s, k = q0 + q_s;
                ra[s] = m < g.M && k < g.K ? eor[(size_t)m * g.K + k] : 0.0;
                rb[s] = ex(jc, q0 + q_f + 4 * s);
            } else {
                const int k = int(i0) + e_f, m = q0 + q_f + 4 * s;
                ra[s] = m < g.M && k < g.K ? eor[(size_t)m * g.K + k] : 0.0;
                rb[s] = weight(jc, m);
            }
        }
    };
    auto commit = [&](int buf) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (OP == kDx) As[buf][q_f + 4 * s][e_f] = ra[s]; else As[buf][q_s][e_s + 16 * s] = ra[s];
            if (OP == kDoff) Bs[buf][q_s][e_s + 16 * s] = rb[s]; else Bs[buf][q_f + 4 * s][e_f] = rb[s];
        }
    };
    const int ti = threadIdx.x / 16, tj = threadIdx.x % 16;           // rows ti + 16 a, columns tj + 16 b
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
    if (c_begin < c_end) { fetch(c_begin); commit(0); }
    __syncthreads();
    for (int c = c_begin; c < c_end; ++c) {
        const int buf = (c - c_begin) & 1;
        if (c + 1 < c_end) fetch(c + 1);
#pragma unroll 4
        for (int q = 0; q < kQ; ++q) {
            double a[4], b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) { a[u] = As[buf][q][ti + 16 * u]; b[u] = Bs[buf][q][tj + 16 * u]; }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
        }
        if (c + 1 < c_end) commit(buf ^ 1);
        __syncthreads();
    }
    const long long rows = OP == kDx ? g.K : g.M, cols = OP == kDoff ? g.K : P;
    if (OP == kDoff || sp.splits > 1) {
        double* dst = part + ((size_t)split * g.R + r) * rows * cols;
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const long long i = i0 + ti + 16 * u, j = j0 + tj + 16 * v;
                if (i < rows && j < cols) dst[i * cols + j] = acc[u][v];
            }
        return;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const Col64 c = col64(g, r, j0 + tj + 16 * v, P, mx);
        if (c.base < 0) continue;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long i = i0 + ti + 16 * u;
            if (i >= rows) continue;
            if (OP == kFwd) out[c.base + i * g.N] = c.mx + mor[i] + (log(acc[u][v]) + g.cst) / g.eps;
            else {
                const long long a = tap_address(g, c, int(i));
                if (a >= 0) out[a] = exp(g.eps * (x[a] - c.mx)) * acc[u][v];
            }
        }
    }
}

// Adds the splits of a forward pass or input gradient and finishes the values.
template <int OP>
__global__ void __launch_bounds__(256) mex_finish64(MexGeo g, int splits, const double* __restrict__ x, const double* __restrict__ mo,
                                                    const double* __restrict__ mx, const double* __restrict__ part, double* __restrict__ out,
                                                    const int* __restrict__ flag) {
    stream_order();
    if (*flag) return;
    const long long P = (long long)g.B * g.rs, rows = OP == kDx ? g.K : g.M, per = (long long)g.R * rows * P;
    for (long long idx = blockIdx.x * 256LL + threadIdx.x; idx < per; idx += (long long)gridDim.x * 256) {
        double s = 0;
#pragma unroll 8
        for (int q = 0; q < splits; ++q) s += part[q * per + idx];
        const long long j = idx % P;
        const int i = int(idx / P % rows), r = int(idx / P / rows);
        const Col64 c = col64(g, r, j, P, mx);
        if (c.base < 0) continue;
        if (OP == kFwd) out[c.base + (long long)i * g.N] = c.mx + mo[(size_t)r * g.M + i] + (log(s) + g.cst) / g.eps;
        else {
            const long long a = tap_address(g, c, i);
            if (a >= 0) out[a] = exp(g.eps * (x[a] - c.mx)) * s;
        }
    }
}

// One CTA per (region, instance): adds the splits of the offsets gradient, times Eo, and takes the gradient back through the
// normalisation when the offsets came raw (v - softmax(row) sum(v)).  When the status word is set, the term-by-term kernel has
// left the finished rows in `part`.
__global__ void __launch_bounds__(256) mex_doff_finish64(MexGeo g, int splits, double* __restrict__ part, const double* __restrict__ eo,
                                                         const double* __restrict__ raw, const double* __restrict__ lse, double* __restrict__ doff,
                                                         int normalize, int accumulate, const int* __restrict__ flag) {
    stream_order();
    __shared__ double red[256];
    const bool exact = *flag != 0;
    const size_t n = (size_t)g.R * g.M * g.K, row = (size_t)blockIdx.x * g.K;
    double sum = 0;
    for (int k = threadIdx.x; k < g.K; k += 256) {
        double v = part[row + k];
        if (!exact) {
            for (int q = 1; q < splits; ++q) v += part[q * n + row + k];
            v *= eo[row + k];
        }
        part[row + k] = v;
        sum += v;
    }
    if (normalize) sum = block_reduce(sum, red, true);
    for (int k = threadIdx.x; k < g.K; k += 256) {
        const double v = part[row + k] - (normalize ? exp(raw[row + k] - lse[blockIdx.x]) * sum : 0.0);
        doff[row + k] = accumulate ? doff[row + k] + v : v;
    }
}

bool norm64(uint32_t flags) { return (flags & SIMNETS_FLAG_MEX_NORMALIZED_OFFSETS) != 0; }

cudaError_t prepare64(const MexGeo& g, const Ws64& w, const double* x, const double* off, uint32_t flags, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(w.flag, 0, 2 * sizeof(int), s);
    if (e != cudaSuccess) return e;
    in_stream_order(mex_prep64, g.R * g.M, 256, 0, s)(g, off, w.mo, w.eo, w.offn, w.lse, w.flag, norm64(flags));
    const long long total = (long long)g.B * g.N;
    const int lanes = g.K >= 512 ? 1 : (g.K >= 32 ? 32 : 256);
    in_stream_order(mex_colmax64, int(std::min<long long>((total + lanes - 1) / lanes, 16LL * device_sm_count())), 256, 0, s)(g, x, w.mx, lanes);
    count_launch(2);
    return cudaGetLastError();
}

template <int OP>
cudaError_t gemm64(const MexGeo& g, const Ws64& w, const double* x, const double* y, const double* dy, double* out, int* splits, cudaStream_t s) {
    const Split64 sp = split_of(g, Op64(OP));
    if (sp.it * sp.jt * g.R > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    in_stream_order(mex_gemm64<OP>, dim3(unsigned(sp.it * sp.jt * g.R), unsigned(sp.splits)), kThreads64, 0, s)(g, sp, x, w.eo, w.mo, w.mx, y, dy, out, w.part, w.flag);
    count_launch();
    *splits = sp.splits;
    if (OP != kDoff && sp.splits > 1) {
        const long long per = (long long)g.R * (OP == kDx ? g.K : g.M) * ((long long)g.B * g.rs);
        in_stream_order(mex_finish64<OP>, int(std::min<long long>((per + 255) / 256, 16LL * device_sm_count())), 256, 0, s)(g, sp.splits, x, w.mo, w.mx, w.part, out, w.flag);
        count_launch();
    }
    return cudaGetLastError();
}

}  // namespace

// Finite epsilon, and positions that 32 bits count.
bool mex_use_f64(const MexGeo& g, uint32_t flags) {
    return g.finite && g.B > 0 && !(flags & (SIMNETS_FLAG_FORCE_DIRECT | SIMNETS_FLAG_MEX_EXACT)) && (long long)g.B * g.rs < 0x7fffffffLL;
}
size_t mex_f64_workspace_bytes(const MexGeo& g) { return carve64(g, nullptr).bytes; }

cudaError_t launch_mex_fwd_f64(const MexGeo& g, const double* x, const double* off, double* y, void* ws, uint32_t flags, cudaStream_t s) {
    const Ws64 w = carve64(g, ws);
    cudaError_t e = prepare64(g, w, x, off, flags, s);
    if (e != cudaSuccess) return e;
    int splits;
    e = gemm64<kFwd>(g, w, x, nullptr, nullptr, y, &splits, s);
    if (e != cudaSuccess) return e;
    return launch_mex_fwd_direct(g, true, x, norm64(flags) ? w.offn : off, y, s, w.flag);
}

cudaError_t launch_mex_bwd_f64(const MexGeo& g, const double* x, const double* off, const double* y, const double* dy, double* dx, double* doff,
                               bool accumulate, void* ws, uint32_t flags, cudaStream_t s) {
    const Ws64 w = carve64(g, ws);
    // (a primed workspace holds what the forward pass prepared for the same input and offsets)
    cudaError_t e = flags & SIMNETS_FLAG_MEX_WORKSPACE_PRIMED ? cudaSuccess : prepare64(g, w, x, off, flags, s);
    if (e != cudaSuccess) return e;
    const double* rows = norm64(flags) ? w.offn : off;
    int splits;
    if (dx != nullptr) {
        if (!(g.sc >= g.bc && g.sh >= g.bh && g.sw >= g.bw)) {       // overlapping blocks: several positions add to one input value
            e = launch_mex_dx_direct(g, true, x, rows, y, dy, dx, s, nullptr);
            if (e != cudaSuccess) return e;
        } else {
            e = cudaMemsetAsync(dx, 0, sizeof(double) * (size_t)g.B * g.C * g.H * g.W, s);
            if (e != cudaSuccess) return e;
            e = gemm64<kDx>(g, w, x, y, dy, dx, &splits, s);
            if (e != cudaSuccess) return e;
            e = launch_mex_dx_direct(g, true, x, rows, y, dy, dx, s, w.flag);
            if (e != cudaSuccess) return e;
        }
    }
    if (doff == nullptr) return cudaSuccess;
    e = gemm64<kDoff>(g, w, x, y, dy, nullptr, &splits, s);
    if (e != cudaSuccess) return e;
    e = launch_mex_doff_direct(g, true, x, rows, y, dy, w.part, false, s, w.flag);
    if (e != cudaSuccess) return e;
    in_stream_order(mex_doff_finish64, g.R * g.M, 256, 0, s)(g, splits, w.part, w.eo, off, w.lse, doff, norm64(flags), accumulate, w.flag);
    count_launch();
    return cudaGetLastError();
}

}  // namespace simnets
