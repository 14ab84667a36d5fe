// MEX forward, input gradient and offsets gradient on the FP32 / FP64 pipes as three small contractions, for float64 layers of
// any size, for float32 layers that are too small for the tensor-core kernels, and for input gradients of overlapping blocks.
//
//     S[m,j] = sum_k Eo[m,k] Ex[k,j],      y = mx + mo + (log S + c) / eps
//     T[k,j] = sum_m Eo[m,k] Q[m,j],       dx[pixel] = sum over the taps k and positions j that meet in it of Ex[k,j] T[k,j]
//     doff[m,k] = Eo[m,k] sum_j Q[m,j] Ex[k,j]
//
// with Ex = exp(eps (x - mx)), Eo = exp(eps (o - mo)), Q = dy exp(eps (mx + mo - y) + c): M K + K N exponentials instead of one
// per (m, k, j) term.  The factorised form is safe while |eps| * spread(offsets) stays bounded; the prepass leaves a verdict per
// group of offset rows, and where one of them says no the kernels evaluate term by term instead (mex_exact.cuh).
//
// Why a family of its own for small layers: a forward call is two or three launches (parameters and maxima, contraction, a
// finishing step when the reduction is split), both gradients are three to five, and a CTA's tile is small enough that a few
// hundred positions fill the GPU.  The tensor-core kernels take four and six and walk the chunks of one tile after another on few
// SMs: 512 instances over 256 channels of 2x2 pixels at batch 128, forward and both gradients: 90 us here, 236 there.
//
// Tile: TM rows (16, 32 or 64) x 64 columns, 32 (float64: 16) steps of the reduction per chunk, double buffered; GemmTile says who
// multiplies what.  The reduction is split over CTAs until the GPU is full.  What the pieces cost in cycles (one CTA of 64 x 32 taps on 8 x
// 8 pixels, float32): the positions 1400, the first operands 2100, 32 steps 2100, the results 4600 when a thread decoded and finished
// values of four positions; float64 in 16 outputs per thread 6400 a chunk, 3700 by tensor-core products (their rate allows 2050, the
// exponentials beside them 1300).  Both gradients and the forward pass, before / after: float64 network of four layers at batch 12 702 /
// 493 us a step; 24 instances over 12 x 3 x 3 taps of 24 x 12 x 41 x 40 221 / 123; 512 over 256 of 2 x 2 pixels at batch 256 131 / 82; 64
// over 32 of 16 x 16 pixels at batch 4 45 / 33.
#include <cmath>
#include <cooperative_groups.h>
#include "kernels.cuh"
#include "mex_exact.cuh"
#include "tile.cuh"

namespace simnets {
namespace {

constexpr int kTN = 64, kGemmThreads = 256, kCluster = 8;          // kCluster: CTAs of the largest portable cluster
constexpr int kGemmMap = 2048;                            // pixels of the prepass's map of extremes
constexpr size_t kOverlapBytes = size_t(256) << 20;       // T of overlapping blocks: at most this much at a time

template <typename T> struct Numeric;
template <> struct Numeric<float> {
    static constexpr int kQ = 32;                         // steps of the reduction per chunk
    static constexpr double kSafe = 60.0;                 // exp(-60) squared stays a normal float times any sum of 1s
    static __device__ __forceinline__ float exp_(float v) { return __expf(v); }
    static __device__ __forceinline__ float log_(float v) { return __logf(v); }
};
template <> struct Numeric<double> {
    static constexpr int kQ = 16;
    static constexpr double kSafe = 300.0;
    static __device__ __forceinline__ double exp_(double v) { return exp(v); }
    static __device__ __forceinline__ double log_(double v) { return log(v); }
};

template <typename T> struct Vec16;
template <> struct Vec16<float> { using type = float4; };
template <> struct Vec16<double> { using type = double2; };

// d[8 x 8] += a[8 x 4] b[4 x 8] in float64.  lane = 4 q + t: a = (q, t), b = (t, q), d = (q, 2 t), (q, 2 t + 1).
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

template <typename T>
struct GemmWs {
    int* flag;           // [2] the workspace's status words, written by the contractions of a call that ran the prepass (null in others)
    int* verdict;        // one per CTA of the parameter prepass: offsets that the factorised form cannot take
    T *mo, *lse;         // [R][M]
    T *eo;               // [R][M][K]
    T *offn;             // [R][M][K] offsets minus their row's log-sum-exp, when they come raw
    T *mx;               // [B][N]
    T *part;             // split partial sums
    size_t bytes;
};
enum GemmOp { kFwd, kDx, kDoff };

struct GemmPlan { int it, tm, steps, splits, together; long long jt; };        // row tiles and their height, reduction length, splits (as clusters), column tiles (per region)
__host__ GemmPlan plan_of(const MexGeo& g, GemmOp op, int kQ) {
    const long long P = (long long)g.B * g.rs;
    const int rows = op == kDx ? g.K : g.M;
    GemmPlan s;
    // least rows, a tile counting for 64 more: every row tile stages (and takes the exponentials of) its columns' operand again (24
    // instances over 12 x 3 x 3 taps: products of 108 rows in seven tiles of 16 46 us, in two of 64 26 us)
    s.tm = 64;
    const auto cost = [&](int tm) { return (rows + tm - 1) / tm * (tm + 64); };
    for (int c : {32, 16}) if (cost(c) < cost(s.tm)) s.tm = c;
    s.it = (rows + s.tm - 1) / s.tm;
    s.jt = ((op == kDoff ? g.K : P) + kTN - 1) / kTN;
    const long long steps = op == kFwd ? g.K : (op == kDx ? g.M : P), tiles = s.it * s.jt * g.R, chunks = (steps + kQ - 1) / kQ;
    // as many CTAs as are resident at once
    const long long places = (long long)device_sm_count() * (op == kDoff && kQ == Numeric<float>::kQ && s.tm < 64 ? 3 : 2);
    long long n = tiles >= places ? 1 : places / tiles;
    n = std::max<long long>(1, std::min(n, (chunks * kQ + 63) / 64));       // at least 64 steps each
    s.steps = int(steps);
    s.splits = int(n);
    // The splits of a forward pass or an input gradient are a cluster where all clusters find room at once: beyond that they wait for
    // whole clusters to leave (12 samples of 512 x 256 on 8 x 8 pixels, float64, 288 CTAs: 38 us; apart and added up by another launch 25).
    s.together = op != kDoff && n > 1 && n <= kCluster && tiles * n <= 7LL * device_sm_count() / 4;
    return s;
}
__host__ bool overlapping(const MexGeo& g) { return g.sc < g.bc || g.sh < g.bh || g.sw < g.bw; }
// samples whose T fits at a time, when blocks overlap
__host__ int overlap_samples(const MexGeo& g, size_t size) {
    const size_t per = (size_t)g.K * g.rs * g.R * size;
    return int(std::max<size_t>(1, std::min<size_t>(g.B, kOverlapBytes / per)));
}
__host__ MexGeo with_samples(MexGeo g, int b) { g.B = b; return g; }
__host__ size_t part_elements(const MexGeo& g_in, GemmOp op, size_t size) {
    const MexGeo g = op == kDx && overlapping(g_in) ? with_samples(g_in, overlap_samples(g_in, size)) : g_in;
    const GemmPlan s = plan_of(g, op, size == 8 ? Numeric<double>::kQ : Numeric<float>::kQ);
    const size_t n = op == kDoff ? (size_t)g.M * g.K : (size_t)(op == kDx ? g.K : g.M) * ((size_t)g.B * g.rs);
    return op == kDoff || (s.splits > 1 && !s.together) || (op == kDx && overlapping(g)) ? n * g.R * s.splits : 0;
}
// threads that share a row of offsets in the prepass, and rows per CTA
__host__ __device__ inline int prep_rows(int K) { return K <= 1024 ? kGemmThreads / 32 : 1; }

template <typename T>
__host__ GemmWs<T> carve_gemm(const MexGeo& g, void* base) {
    GemmWs<T> w;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t bytes) { char* r = p ? p + off : nullptr; off += (bytes + 255) & ~size_t(255); return r; };
    auto vals = [&](size_t n) { return reinterpret_cast<T*>(take(n * sizeof(T))); };
    w.flag = reinterpret_cast<int*>(take(16));
    w.verdict = reinterpret_cast<int*>(take(sizeof(int) * (size_t)g.R * g.M));
    w.mo = vals((size_t)g.R * g.M);
    w.lse = vals((size_t)g.R * g.M);
    w.eo = vals((size_t)g.R * g.M * g.K);
    w.offn = vals((size_t)g.R * g.M * g.K);
    w.mx = vals((size_t)g.B * g.N);
    // (the products of overlapping blocks are scratch of the input gradient alone: mex_gemm_products_bytes)
    w.part = vals(std::max(part_elements(g, kFwd, sizeof(T)), std::max(overlapping(g) ? 0 : part_elements(g, kDx, sizeof(T)), part_elements(g, kDoff, sizeof(T)))));
    w.bytes = off;
    return w;
}

template <typename T> __device__ __forceinline__ T t_max(T a, T b) { return a < b || a != a ? b : a; }          // NaN loses

// Reduction over the threads of one offsets row: a warp, or the CTA through shared memory.
template <typename T, bool SUM>
__device__ __forceinline__ T row_reduce(T v, T* red, bool warp) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) { const T o = __shfl_xor_sync(0xffffffffu, v, s); v = SUM ? v + o : t_max(v, o); }
    if (warp) return v;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
#pragma unroll
    for (int i = 1; i < kGemmThreads / 32; ++i) v = SUM ? v + red[i] : t_max(v, red[i]);
    return v;
}

// xb: offset of the patch corner in x; inside: the whole patch lies in the input
struct GemmCol { long long base, gbase, xb; int n, c0, h0, w0; bool inside; };
__device__ __forceinline__ void place_patch(const MexGeo& g, GemmCol& c) {
    c.xb = (((long long)c.n * g.C + c.c0) * g.H + c.h0) * g.W + c.w0;
    c.inside = c.c0 >= 0 && c.c0 + g.bc <= g.C && c.h0 >= 0 && c.h0 + g.bh <= g.H && c.w0 >= 0 && c.w0 + g.bw <= g.W;
}
__device__ __forceinline__ GemmCol gemm_col(const MexGeo& g, int r, long long jl, long long P) {
    GemmCol c = {-1, 0, 0, 0, 0, 0, 0, false};
    if (jl >= P) return c;
    const int n = int(fast_div(uint32_t(jl), g.f_rs)), l = int(jl) - n * g.rs;        // (P < 2^31)
    int cc, h, w;
    if (!mex_region_chw(g, r, l, cc, h, w)) return c;
    const int pos = (cc * g.Ho + h) * g.Wo + w;
    c.n = n; c.c0 = cc * g.sc - g.pc; c.h0 = h * g.sh - g.ph; c.w0 = w * g.sw - g.pw;
    c.base = (long long)n * g.M * g.N + pos;
    c.gbase = mex_dy_base(g, n, pos);
    place_patch(g, c);
    return c;
}
// Decoded taps of a block in shared memory: {offset from the patch corner, (c << 16) | (h << 8) | w}.  Decoding a tap costs two
// divisions and two modulos, which had been most of the instructions around a gathered value (blocks of 12 x 3 x 3).
constexpr int kGemmTaps = 1024;
__device__ __forceinline__ bool taps_tabled(const MexGeo& g) { return g.K <= kGemmTaps && g.bh <= 256 && g.bw <= 256; }
__device__ __forceinline__ void table_taps(const MexGeo& g, int2* __restrict__ tab) {
    if (taps_tabled(g))
        for (int k = threadIdx.x; k < g.K; k += kGemmThreads) {
            const int w = k % g.bw, q = k / g.bw, h = q % g.bh, c = q / g.bh;
            tab[k] = make_int2((c * g.H + h) * g.W + w, (c << 16) | (h << 8) | w);
        }
}
// index of the position's maximum
__device__ __forceinline__ long long col_mx(const MexGeo& g, const GemmCol& c) { return c.base - (long long)c.n * (g.M - 1) * g.N; }
// offset of tap k in x, or -1 outside the input; tab: the table, or null
__device__ __forceinline__ long long tap_address(const MexGeo& g, const GemmCol& c, int k, const int2* __restrict__ tab) {
    if (g.bh * g.bw == 1 && c.inside) return c.xb + (long long)k * (g.H * g.W);
    if (g.bh == g.H && g.bw == g.W && c.inside) return c.xb + k;          // (blocks of whole planes: a run of memory)
    if (tab) {
        const int2 t = tab[k];
        if (c.inside) return c.xb + t.x;
        const int cc = c.c0 + (t.y >> 16), hh = c.h0 + ((t.y >> 8) & 255), ww = c.w0 + (t.y & 255);
        return uint32_t(cc) < uint32_t(g.C) && uint32_t(hh) < uint32_t(g.H) && uint32_t(ww) < uint32_t(g.W) ? c.xb + t.x : -1;
    }
    int kc = k, kh = 0, kw = 0;
    if (g.bh * g.bw > 1) { kw = k % g.bw; const int q = k / g.bw; kh = q % g.bh; kc = q / g.bh; }
    const int cc = c.c0 + kc, hh = c.h0 + kh, ww = c.w0 + kw;
    if (cc < 0 || cc >= g.C || hh < 0 || hh >= g.H || ww < 0 || ww >= g.W) return -1;
    return (((long long)c.n * g.C + cc) * g.H + hh) * g.W + ww;
}

// CTAs [0, prep_ctas): offsets rows -- reference value, Eo, log-sum-exp and normalised row of raw offsets, the safety verdict.
// The others: largest (eps > 0) or smallest tap of every patch, NaN ignored; `lanes` positions per CTA, 256 / lanes slices of
// the taps.
template <typename T>
__global__ void __launch_bounds__(kGemmThreads) mex_gemm_prep(MexGeo g, const T* __restrict__ x, const T* __restrict__ off, T* __restrict__ mo, T* __restrict__ eo,
                                                              T* __restrict__ offn, T* __restrict__ lse_out, int* __restrict__ verdict, T* __restrict__ mx,
                                                              int prep_ctas, int normalize, int lanes, int band) {
    stream_order();
    __shared__ T red[kGemmThreads];
    __shared__ int2 tap_tab[kGemmTaps];
    const T eps = T(g.eps);
    if (int(blockIdx.x) < prep_ctas) {
        const bool warp = prep_rows(g.K) > 1;
        const int threads = warp ? 32 : kGemmThreads, lane = threadIdx.x % threads;
        const int row_id = blockIdx.x * prep_rows(g.K) + threadIdx.x / threads;
        const bool live = row_id < g.R * g.M;
        const size_t row = (size_t)row_id * g.K;
        T hi = -pos_inf<T>(), lo = -pos_inf<T>();             // (lo: maximum of the negated values)
        int bad = 0;
        if (live)
#pragma unroll 4
            for (int k = lane; k < g.K; k += threads) {
                const T v = off[row + k];
                bad |= !isfinite(v);
                hi = t_max(hi, v); lo = t_max(lo, -v);
            }
        hi = row_reduce<T, false>(hi, red, warp);
        lo = -row_reduce<T, false>(lo, red, warp);
        const T ref = eps > T(0) ? hi : lo;
        const T base = isfinite(hi) ? hi : T(0);              // as a stable log-sum-exp treats infinite maxima
        const bool one = normalize && eps == T(1) && sizeof(T) == 8;          // (then Eo are the terms of that sum; float32 takes another exponential for them)
        T lse = T(0);
        if (normalize) {
            T sum = T(0);
            if (live)
#pragma unroll 4
                for (int k = lane; k < g.K; k += threads) {
                    const T e = dev_exp(off[row + k] - base);
                    if (one) eo[row + k] = e;
                    sum += e;
                }
            lse = base + dev_log(row_reduce<T, true>(sum, red, warp));
        }
        if (live) {
            if (lane == 0) { mo[row_id] = ref - lse; lse_out[row_id] = lse; }
            bad |= !(fabs(g.eps) * double(hi - lo) <= Numeric<T>::kSafe);
            if (normalize)
#pragma unroll 4
                for (int k = lane; k < g.K; k += threads) offn[row + k] = off[row + k] - lse;
            if (!one)
#pragma unroll 4
                for (int k = lane; k < g.K; k += threads) eo[row + k] = Numeric<T>::exp_(eps * (off[row + k] - ref));
        }
        bad = __syncthreads_or(bad);
        if (threadIdx.x == 0) verdict[blockIdx.x] = bad;
        return;
    }
    if (band > 0) {
        // blocks that overlap along rows or columns: the extremes over a block's channels of every pixel under `band` output rows, then over
        // every window of those (24 x 12 x 41 x 40, 12 x 3 x 3 blocks: 16.6 us tap by tap, 3.9 so)
        __shared__ T map[kGemmMap];
        const int bands = (g.Ho + band - 1) / band;
        long long id = blockIdx.x - prep_ctas;
        const int h_first = int(id % bands) * band, hs = min(band, g.Ho - h_first); id /= bands;
        const int cb = int(id % g.Co), n = int(id / g.Co);
        const int rows = (hs - 1) * g.sh + g.bh, width = (g.Wo - 1) * g.sw + g.bw, c0 = cb * g.sc - g.pc;
        const bool up = g.eps > 0, cut = c0 < 0 || c0 + g.bc > g.C;
        const T oob = T(g.oob);
        const int cl = max(c0, 0), ch = min(c0 + g.bc, g.C);
        for (int i = threadIdx.x; i < rows * width; i += kGemmThreads) {
            const int hh = h_first * g.sh - g.ph + i / width, ww = i % width - g.pw;
            T v = -pos_inf<T>();
            if (hh >= 0 && hh < g.H && ww >= 0 && ww < g.W) {
                const size_t hw = (size_t)g.H * g.W;
                const T* p = x + ((size_t)n * g.C + cl) * hw + hh * g.W + ww;
#pragma unroll 4
                for (int c = cl; c < ch; ++c, p += hw) { const T t = *p; v = t_max(v, up ? t : -t); }
                if (cut) v = t_max(v, up ? oob : -oob);
            } else v = t_max(v, up ? oob : -oob);
            map[i] = v;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < hs * g.Wo; i += kGemmThreads) {
            const int h = i / g.Wo, w = i - h * g.Wo;
            const T* p = map + h * g.sh * width + w * g.sw;
            T v = -pos_inf<T>();
            for (int a = 0; a < g.bh; ++a, p += width)
#pragma unroll 3
                for (int b = 0; b < g.bw; ++b) v = t_max(v, p[b]);
            mx[((long long)n * g.Co + cb) * g.Ho * g.Wo + (h_first + h) * g.Wo + w] = up ? v : -v;
        }
        return;
    }
    const int slices = kGemmThreads / lanes, lane = threadIdx.x % lanes, slice = threadIdx.x / lanes;
    const long long total = (long long)g.B * g.N, idx = (long long)(blockIdx.x - prep_ctas) * lanes + lane;
    const bool up = g.eps > 0;
    const T oob = T(g.oob);
    const bool pixel = g.bh * g.bw == 1;
    const int2* tab = !pixel && taps_tabled(g) ? tap_tab : nullptr;
    if (!pixel) { table_taps(g, tap_tab); __syncthreads(); }
    T v = -pos_inf<T>();                                      // maximum of x or of -x
    if (idx < total) {
        const int pos = int(idx % g.N);
        GemmCol c;
        c.n = int(idx / g.N);
        c.w0 = pos % g.Wo * g.sw - g.pw; c.h0 = pos / g.Wo % g.Ho * g.sh - g.ph; c.c0 = pos / (g.Wo * g.Ho) * g.sc - g.pc;
        place_patch(g, c);
        if (c.inside && pixel) {
            const T* p = x + c.xb;
            const size_t hw = (size_t)g.H * g.W;
#pragma unroll 8
            for (int k = slice; k < g.K; k += slices) { const T t = p[k * hw]; v = t_max(v, up ? t : -t); }
        } else {
#pragma unroll 4
            for (int k = slice; k < g.K; k += slices) {
                const long long a = tap_address(g, c, k, tab);
                const T t = a >= 0 ? x[a] : oob;
                v = t_max(v, up ? t : -t);
            }
        }
    }
    red[threadIdx.x] = v;
    __syncthreads();
    for (int s = slices / 2; s > 0; s >>= 1) {
        if (slice < s) red[threadIdx.x] = t_max(red[threadIdx.x], red[threadIdx.x + s * lanes]);
        __syncthreads();
    }
    if (slice == 0 && idx < total) mx[idx] = up ? red[lane] : -red[lane];
}

__device__ __forceinline__ bool gemm_unsafe(const int* __restrict__ verdict, int n) {
    int bad = 0;
    for (int i = threadIdx.x; i < n; i += kGemmThreads) bad |= verdict[i];
    return __syncthreads_or(bad) != 0;
}
template <typename T>
__device__ __noinline__ void exact_forward(const MexGeo& g, const T* x, const T* off, T* y) {
    const long long total = (long long)g.B * g.M * g.N, step = (long long)gridDim.x * gridDim.y * kGemmThreads;
    for (long long i = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kGemmThreads + threadIdx.x; i < total; i += step) y[i] = mex_exact_y<T, true>(g, x, off, i);
}
template <typename T>
__device__ __noinline__ void exact_dx(const MexGeo& g, const T* x, const T* off, const T* y, const T* dy, T* dx) {
    const long long total = (long long)g.B * g.C * g.H * g.W, step = (long long)gridDim.x * gridDim.y * kGemmThreads;
    for (long long i = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kGemmThreads + threadIdx.x; i < total; i += step) dx[i] = mex_exact_dx(g, x, off, y, dy, i);
}

// The sums of the offsets gradient term by term, into sums[r][m][k]: `threads` of a CTA (all or a warp) share the positions of TAPS of one
// (r, m) at a time.
template <typename T, int TAPS>
__device__ __forceinline__ void exact_doff_of(const MexGeo& g, const T* x, const T* off, const T* y, const T* dy, T* sums, T* red, int threads) {
    const long long P = (long long)g.B * g.rs, ctas = (long long)gridDim.x * gridDim.y;
    const int groups = (g.K + TAPS - 1) / TAPS, per = kGemmThreads / threads, lane = threadIdx.x % threads;
    const T eps = T(g.eps), cst = T(g.cst), oob = T(g.oob);
    for (long long i = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * per + threadIdx.x / threads; i < (long long)g.R * g.M * groups; i += ctas * per) {
        const long long row = i / groups;
        const int k0 = int(i - row * groups) * TAPS, m = int(row % g.M), r = int(row / g.M);
        int kc[TAPS], kh[TAPS], kw[TAPS];
        long long tap[TAPS];
        T o[TAPS], v[TAPS];
#pragma unroll
        for (int u = 0; u < TAPS; ++u) {
            const int k = min(k0 + u, g.K - 1);
            kw[u] = k % g.bw; kh[u] = k / g.bw % g.bh; kc[u] = k / (g.bw * g.bh);
            tap[u] = ((long long)kc[u] * g.H + kh[u]) * g.W + kw[u];
            o[u] = off[row * g.K + k];
            v[u] = T(0);
        }
#pragma unroll 2
        for (long long j = lane; j < P; j += threads) {
            const GemmCol c = gemm_col(g, r, j, P);
            if (c.base < 0) continue;
            const T top = y[c.base + (long long)m * g.N], d = dy[c.gbase + (long long)m * g.Ng];
#pragma unroll
            for (int u = 0; u < TAPS; ++u) {
                const int cc = c.c0 + kc[u], h = c.h0 + kh[u], w = c.w0 + kw[u];
                const bool in = c.inside || (cc >= 0 && cc < g.C && h >= 0 && h < g.H && w >= 0 && w < g.W);
                v[u] += mex_weight(g, eps, cst, in ? x[c.xb + tap[u]] : oob, o[u], top, d);
            }
        }
#pragma unroll
        for (int u = 0; u < TAPS; ++u) {
            const T sum = row_reduce<T, true>(v[u], red, threads == 32);
            if (lane == 0 && k0 + u < g.K) sums[row * g.K + k0 + u] = sum;
        }
    }
}

// A register adds up 1 / 256 of a sum's B rs terms, up to 1024 of them 1 / 32.  One thread per sum, 459 K positions under 8 instances of
// 4x2x2 taps: 306 ms and 1e-5 of the gradient's norm from float64; so 1.6 ms and 6e-7.  A position is looked up, and its y and dy read, for
// four taps where that leaves every CTA some (128 instances over 64 taps, 2 x 2 regions of 1024 positions: a tap per CTA 824 us, a tap per
// warp 654, four 358).
template <typename T>
__device__ __noinline__ void exact_doff(const MexGeo& g, const T* x, const T* off, const T* y, const T* dy, T* sums, T* red) {
    const int threads = (long long)g.B * g.rs <= 1024 ? 32 : kGemmThreads;
    const long long units = (long long)gridDim.x * gridDim.y * (kGemmThreads / threads);
    if ((long long)g.R * g.M * ((g.K + 3) / 4) >= units) exact_doff_of<T, 4>(g, x, off, y, dy, sums, red, threads);
    else exact_doff_of<T, 1>(g, x, off, y, dy, sums, red, threads);
}

// What a CTA multiplies, in shared memory: As[2][kQ][LDA], Bs[2][kQ][LDB], step by step.  A thread's reads of them are the bound (32
// lanes x 16 bytes take four cycles however few different addresses they have):
//  * float32: TM/8 x 4 outputs per thread in packed arithmetic, half of the threads cover the tile and the two halves share the steps
//    of a chunk: a quarter to a half fewer reads per multiply-add than TM/16 x 4 on all of them.  (8 x 8 outputs and four or eight
//    copies read less still, but adding the copies up and 128 registers cost more than that in layers of a few chunks.)
//  * float64: tensor-core products of 8 x 8 x 4, whose fragments are a value per lane; 16 outputs per thread had read 64 bytes for 16
//    multiply-adds, 16 cycles for 8.
template <typename T, int TM> struct GemmTile;
template <int TM> struct GemmTile<float, TM> {
    static constexpr int kQ = Numeric<float>::kQ, LDA = TM + 4, LDB = kTN + 4, LDT = kTN + 4, RM = TM / 8;
    static constexpr int STAGES = 2 * kQ * (LDA + LDB), FLOATS = STAGES > TM * LDT ? STAGES : TM * LDT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = warp >> 2;
    // 4 x 8 threads per warp (pairs of rows interleaved, as in tile.cuh), 2 x 2 warps
    const int ti = (warp & 1) * 4 + (((lane >> 4) << 1) | (lane & 1)), tj = ((warp >> 1) & 1) * 8 + ((lane & 15) >> 1);
    float2 acc[RM][2];
    __device__ __forceinline__ GemmTile() {
#pragma unroll
        for (int u = 0; u < RM; ++u) acc[u][0] = acc[u][1] = make_float2(0.f, 0.f);
    }
    __device__ __forceinline__ int row(int u) const { return RM == 8 ? (u >> 2) * (TM / 2) + ti * 4 + (u & 3) : ti * RM + u; }
    __device__ __forceinline__ void chunk(const float* __restrict__ As, const float* __restrict__ Bs) {
        As += half * (kQ / 2) * LDA + ti * (RM == 2 ? 2 : 4);
        Bs += half * (kQ / 2) * LDB + tj * 4;
#pragma unroll 8
        for (int q = 0; q < kQ / 2; ++q) {
            float a[RM];
            if (RM == 2) {
                const float2 v = *reinterpret_cast<const float2*>(As + q * LDA);
                a[0] = v.x; a[1] = v.y;
            } else {
#pragma unroll
                for (int h = 0; h < RM / 4; ++h) {
                    const float4 v = *reinterpret_cast<const float4*>(As + q * LDA + h * (TM / 2));
                    a[RM > 2 ? 4 * h : 0] = v.x; a[RM > 2 ? 4 * h + 1 : 0] = v.y; a[RM > 2 ? 4 * h + 2 : 0] = v.z; a[RM > 2 ? 4 * h + 3 : 0] = v.w;
                }
            }
            const float4 b = *reinterpret_cast<const float4*>(Bs + q * LDB);
#pragma unroll
            for (int u = 0; u < RM; ++u) {
                acc[u][0] = fma2(splat2(a[u]), make_float2(b.x, b.y), acc[u][0]);
                acc[u][1] = fma2(splat2(a[u]), make_float2(b.z, b.w), acc[u][1]);
            }
        }
    }
    // the tile's sums as rows of LDT; the stages are free by now
    __device__ __forceinline__ void store(float* __restrict__ tile) {
        tile += tj * 4;
        if (half == 1)
#pragma unroll
            for (int u = 0; u < RM; ++u) *reinterpret_cast<float4*>(tile + row(u) * LDT) = make_float4(acc[u][0].x, acc[u][0].y, acc[u][1].x, acc[u][1].y);
        __syncthreads();
        if (half == 0)
#pragma unroll
            for (int u = 0; u < RM; ++u) {
                float4* p = reinterpret_cast<float4*>(tile + row(u) * LDT);
                const float4 v = *p;
                *p = make_float4(acc[u][0].x + v.x, acc[u][0].y + v.y, acc[u][1].x + v.z, acc[u][1].y + v.w);
            }
        __syncthreads();
    }
};
template <int TM> struct GemmTile<double, TM> {
    // (rows of 64 + 4 values: 4 steps x 4 rows of a fragment's half hit 16 different pairs of banks)
    static constexpr int kQ = Numeric<double>::kQ, LDA = TM + 4, LDB = kTN + 4, LDT = kTN + 2, WI = TM / 16, WJ = 8 / WI, NC = kTN / 8 / WJ;
    static constexpr int STAGES = 2 * kQ * (LDA + LDB), FLOATS = STAGES > TM * LDT ? STAGES : TM * LDT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane >> 2, t = lane & 3;
    const int i0 = (warp % WI) * 16, j0 = (warp / WI) * 8 * NC;
    double acc[2][NC][2];
    __device__ __forceinline__ GemmTile() {
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < NC; ++v) acc[u][v][0] = acc[u][v][1] = 0.0;
    }
    __device__ __forceinline__ void chunk(const double* __restrict__ As, const double* __restrict__ Bs) {
        As += t * LDA + i0 + q;
        Bs += t * LDB + j0 + q;
#pragma unroll
        for (int s = 0; s < kQ; s += 4) {
            double a[2], b[NC];
#pragma unroll
            for (int u = 0; u < 2; ++u) a[u] = As[s * LDA + 8 * u];
#pragma unroll
            for (int v = 0; v < NC; ++v) b[v] = Bs[s * LDB + 8 * v];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int v = 0; v < NC; ++v) mma_f64(acc[u][v], a[u], b[v]);
        }
    }
    __device__ __forceinline__ void store(double* __restrict__ tile) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < NC; ++v)
                *reinterpret_cast<double2*>(tile + (i0 + 8 * u + q) * LDT + j0 + 8 * v + 2 * t) = make_double2(acc[u][v][0], acc[u][v][1]);
        __syncthreads();
    }
};

// The three contractions.  Rows i: instances (forward, offsets gradient) or taps (input gradient); columns j: positions of one
// region (taps for the offsets gradient); reduction q: taps, instances, positions.
template <typename T, int OP, int TM>
__host__ __device__ constexpr int gemm_ctas() { return sizeof(T) == 8 || TM == 64 ? 2 : (OP == kDx && TM == 16 ? 4 : 3); }

// Which way the lanes of a warp go through y, dy and x: along positions, which are neighbours in memory where a region has many of
// them in a sample, or along instances (taps), N (H W) values apart, on maps of a few pixels: of 512 instances over 256 channels of 2 x 2
// pixels a warp along positions touches 32 cache lines per read, along instances four (forward / offsets gradient at batch 256: 21 / 41
// us, 22 / 22).
__host__ inline bool gemm_along_positions(const MexGeo& g, size_t size) {
    const long long sample = std::max<long long>(1, (long long)g.N * size / 128), reach = std::min(32, g.rs);
    const long long positions = (32 + reach - 1) / reach * std::min<long long>(reach, sample), instances = std::min<long long>(32, std::max<long long>(1, 32 * (long long)g.N * size / 128));
    return positions <= instances;
}

// POS: lanes along positions.  The splits of a tile are one cluster (unless their sums go to `part`): each CTA finishes some rows, reading
// the others' sums of them from their shared memory.
template <typename T, int OP, int TM, bool POS>
__global__ void __launch_bounds__(kGemmThreads, gemm_ctas<T, OP, TM>()) mex_gemm(const __grid_constant__ MexGeo g, GemmPlan sp, const T* __restrict__ x, const T* __restrict__ off,
                                                         const T* __restrict__ eo, const T* __restrict__ mo, const T* __restrict__ mx, const T* __restrict__ y,
                                                         const T* __restrict__ dy, T* __restrict__ out, T* __restrict__ part, const int* __restrict__ verdict,
                                                         int verdicts, int to_part, int* __restrict__ flag) {
    stream_order();
    using Tile = GemmTile<T, TM>;
    constexpr int kQ = Tile::kQ, EPQ = kGemmThreads / kQ, LDA = Tile::LDA, LDB = Tile::LDB, LDT = Tile::LDT;       // (step fastest: EPQ elements at a time)
    constexpr int NA = TM * kQ / kGemmThreads, NB = kTN * kQ / kGemmThreads, RPT = kGemmThreads / TM, CPT = kGemmThreads / kTN;
    __shared__ __align__(16) T smem[Tile::FLOATS];
    __shared__ T mos[OP == kFwd ? TM : 1];
    __shared__ int2 tap_tab[OP == kDx ? 1 : kGemmTaps];
    // lanes along instances: the tile's positions, or those of two chunks
    __shared__ GemmCol cols_s[POS ? 1 : (OP == kDoff ? 2 * kQ : kTN)];
    __shared__ T mx_s[POS ? 1 : (OP == kDoff ? 2 * kQ : kTN)];
    const bool pixel = g.bh * g.bw == 1;
    const int2* tab = OP != kDx && !pixel && taps_tabled(g) ? tap_tab : nullptr;
    const long long P = (long long)g.B * g.rs;
    const int r = int(blockIdx.x % unsigned(g.R)), split = blockIdx.y;
    const long long tile = blockIdx.x / unsigned(g.R);
    const int i0 = int(tile % sp.it) * TM;
    const long long j0 = tile / sp.it * kTN;
    const int chunks = (sp.steps + kQ - 1) / kQ, c_begin = int((long long)chunks * split / sp.splits), c_end = int((long long)chunks * (split + 1) / sp.splits);
    const T* eor = eo + (size_t)r * g.M * g.K;
    const T* mor = mo + (size_t)r * g.M;
    const T eps = T(g.eps), cst = T(g.cst), oob = T(g.oob);
    if (OP == kFwd && threadIdx.x < TM && i0 + threadIdx.x < g.M) mos[threadIdx.x] = mor[i0 + threadIdx.x];
    if (tab) table_taps(g, tap_tab);
    // this thread's position: of the tile, or (offsets gradient) of the chunk
    GemmCol col = {-1, 0, 0, 0, 0, 0, 0, false};
    T cmx = T(0);
    auto place = [&](long long j) { col = gemm_col(g, r, j, P); cmx = col.base >= 0 ? mx[col_mx(g, col)] : T(0); };
    auto place_chunk = [&](int chunk) {                               // (offsets gradient, lanes along instances)
        if (threadIdx.x >= kQ || chunk >= c_end) return;
        place((long long)chunk * kQ + threadIdx.x);
        cols_s[POS ? 0 : (chunk & 1) * kQ + threadIdx.x] = col;
    };
    auto place_maxima = [&](int chunk) { if (threadIdx.x < kQ && chunk < c_end) mx_s[POS ? 0 : (chunk & 1) * kQ + threadIdx.x] = cmx; };
    // staging of Eo and, along positions, of what has two positions of the fast axis in a row: element fastest or step fastest
    const int ea_f = threadIdx.x % TM, qa_f = threadIdx.x / TM, eb_f = threadIdx.x % kTN, qb_f = threadIdx.x / kTN;
    const int q_s = threadIdx.x % kQ, e_s = threadIdx.x / kQ;
    if (OP != kDoff) {
        if (POS) place(j0 + eb_f);
        else if (threadIdx.x < kTN) { place(j0 + threadIdx.x); cols_s[POS ? 0 : threadIdx.x] = col; }
    } else if (!POS) place_chunk(c_begin);
    if (tab || !POS) __syncthreads();
    // What a thread stages is requested as it lies in memory while the chunk in front is multiplied, and made an operand (exponentials)
    // when that is done.  v: x, y or Eo; w: dy.
    constexpr bool QA = OP == kDoff, QB = OP == kDx;                  // which operand is Q
    T va[NA], wa[QA ? NA : 1], vb[NB], wb[QB ? NB : 1];
    auto ask_q = [&](const GemmCol& c, int m, T& v, T& w) {
        v = w = T(0);
        if (c.base >= 0 && m < g.M) { v = y[c.base + (long long)m * g.N]; w = dy[c.gbase + (long long)m * g.Ng]; }
    };
    auto ask_x = [&](const GemmCol& c, int k, T& v) {
        v = oob;
        if (c.base < 0 || k >= g.K) return;
        const long long a = tap_address(g, c, k, tab);
        if (a >= 0) v = x[a];
    };
    auto fetch = [&](int chunk) {
        const int q0 = chunk * kQ;
        if (QA) {
            if (POS) {
                place(q0 + q_s);
#pragma unroll
                for (int s = 0; s < NA; ++s) ask_q(col, i0 + e_s + EPQ * s, va[s], wa[QA ? s : 0]);
            } else {
#pragma unroll
                for (int s = 0; s < NA; ++s) ask_q(cols_s[POS ? 0 : (chunk & 1) * kQ + qa_f + RPT * s], i0 + ea_f, va[s], wa[QA ? s : 0]);
            }
        } else {
            const int m = OP == kFwd ? i0 + e_s : q0 + qa_f, k = OP == kFwd ? q0 + q_s : i0 + ea_f, step = OP == kFwd ? EPQ : RPT;
            const T* p = eor + (long long)m * g.K + k;
#pragma unroll
            for (int s = 0; s < NA; ++s, p += (long long)step * g.K) {
                va[s] = T(0);
                if (m + step * s < g.M && k < g.K) va[s] = *p;
            }
        }
        if (QB) {
#pragma unroll
            for (int s = 0; s < NB; ++s) {
                if (POS) ask_q(col, q0 + qb_f + CPT * s, vb[s], wb[QB ? s : 0]);
                else ask_q(cols_s[POS ? 0 : e_s + EPQ * s], q0 + q_s, vb[s], wb[QB ? s : 0]);
            }
        } else if (!POS) {
#pragma unroll
            for (int s = 0; s < NB; ++s) {
                if (OP == kFwd) ask_x(cols_s[POS ? 0 : e_s + EPQ * s], q0 + q_s, vb[s]);
                else ask_x(cols_s[POS ? 0 : (chunk & 1) * kQ + qb_f + CPT * s], int(j0) + eb_f, vb[s]);
            }
        } else {
            const int k = OP == kFwd ? q0 + qb_f : int(j0) + e_s, step = OP == kFwd ? CPT : EPQ;
            if (pixel && col.inside) {
                const long long hw = (long long)g.H * g.W;
                const T* p = x + col.xb + k * hw;
#pragma unroll
                for (int s = 0; s < NB; ++s, p += step * hw) {
                    vb[s] = T(0);
                    if (k + step * s < g.K) vb[s] = *p;
                }
            } else {
#pragma unroll
                for (int s = 0; s < NB; ++s) ask_x(col, k + step * s, vb[s]);
            }
        }
    };
    const auto as_q = [&](bool live, T v, T w, int m, T top) { return live && m < g.M ? w * Numeric<T>::exp_(eps * (top + mor[m] - v) + cst) : T(0); };
    const auto as_ex = [&](bool live, T v, int k, T top) { return live && k < g.K ? Numeric<T>::exp_(eps * (v - top)) : T(0); };
    auto commit = [&](T* As, T* Bs, int chunk) {
        const int q0 = chunk * kQ;
#pragma unroll
        for (int s = 0; s < NA; ++s) {
            const int at = POS ? 0 : (chunk & 1) * kQ + qa_f + RPT * s;
            if (OP == kDx) As[(qa_f + RPT * s) * LDA + ea_f] = va[s];
            else if (OP == kFwd) As[q_s * LDA + e_s + EPQ * s] = va[s];
            else if (POS) As[q_s * LDA + e_s + EPQ * s] = as_q(col.base >= 0, va[s], wa[QA ? s : 0], i0 + e_s + EPQ * s, cmx);
            else As[(qa_f + RPT * s) * LDA + ea_f] = as_q(cols_s[at].base >= 0, va[s], wa[QA ? s : 0], i0 + ea_f, mx_s[at]);
        }
#pragma unroll
        for (int s = 0; s < NB; ++s) {
            const int at = POS ? 0 : (OP == kDoff ? (chunk & 1) * kQ + qb_f + CPT * s : e_s + EPQ * s);
            const bool live = POS ? col.base >= 0 : cols_s[at].base >= 0;
            const T top = POS ? cmx : mx_s[at];
            if (OP == kDoff) {
                if (POS) Bs[q_s * LDB + e_s + EPQ * s] = as_ex(live, vb[s], int(j0) + e_s + EPQ * s, top);
                else Bs[(qb_f + CPT * s) * LDB + eb_f] = as_ex(live, vb[s], int(j0) + eb_f, top);
            } else {
                const int q = POS ? qb_f + CPT * s : q_s, e = POS ? eb_f : e_s + EPQ * s;
                Bs[q * LDB + e] = QB ? as_q(live, vb[s], wb[QB ? s : 0], q0 + q, top) : as_ex(live, vb[s], q0 + q, top);
            }
        }
    };
    Tile sums;
    // (one copy of the staging code, the first round without a chunk to multiply: a kernel that runs for a few microseconds pays for every
    // line of it that has to come from L2)
#pragma unroll 1
    for (int c = c_begin - 1; c < c_end; ++c) {
        T* now = smem + ((c - c_begin) & 1) * kQ * (LDA + LDB);
        T* next = smem + ((c + 1 - c_begin) & 1) * kQ * (LDA + LDB);
        if (c + 1 < c_end) fetch(c + 1);
        if (c >= c_begin) sums.chunk(now, now + kQ * LDA);
        else {
            // (the first operands are on their way while this is looked up; it publishes the maxima too)
            if (!POS && OP != kDoff && threadIdx.x < kTN) mx_s[POS ? 0 : threadIdx.x] = cmx;
            if (!POS && OP == kDoff) place_maxima(c_begin);
            const bool unsafe = gemm_unsafe(verdict, verdicts);
            if (flag != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) flag[threadIdx.x] = threadIdx.x == 0 && unsafe;
            if (unsafe) {
                if (OP == kFwd) exact_forward(g, x, off, out);
                if (OP == kDx) exact_dx(g, x, off, y, dy, out);
                if (OP == kDoff) exact_doff(g, x, off, y, dy, part, smem);
                return;
            }
        }
        if (c + 1 < c_end) commit(next, next + kQ * LDA, c + 1);
        if (OP == kDoff && !POS) { place_chunk(c + 2); place_maxima(c + 2); }
        __syncthreads();
    }
    sums.store(smem);
    const long long rows = OP == kDx ? g.K : g.M, cols = OP == kDoff ? g.K : P;
    if (OP == kDoff || to_part) {
        T* dst = part + ((size_t)split * g.R + r) * rows * cols + i0 * cols + j0 + eb_f;
        if (j0 + eb_f < cols)
#pragma unroll 4
            for (int u = qb_f; u < TM; u += CPT)
                if (i0 + u < rows) dst[u * cols] = smem[u * LDT + eb_f];
        return;
    }
    // this CTA's rows of the tile: all of them, or its share of the cluster's, the others' sums of them added in a fixed order
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int u0 = TM * split / sp.splits, us = TM * (split + 1) / sp.splits - u0;
    if (sp.splits > 1) {
        cluster.sync();
        using Vec = typename Vec16<T>::type;
        constexpr int W = 16 / int(sizeof(T));
        for (int i = threadIdx.x; i < us * (kTN / W); i += kGemmThreads) {
            const int at = (u0 + i / (kTN / W)) * LDT + i % (kTN / W) * W;
            T v[W];
#pragma unroll
            for (int w = 0; w < W; ++w) v[w] = T(0);
            for (int q = 0; q < sp.splits; ++q) {
                const Vec o = *reinterpret_cast<const Vec*>(cluster.map_shared_rank(smem, q) + at);
                const T* ov = reinterpret_cast<const T*>(&o);
#pragma unroll
                for (int w = 0; w < W; ++w) v[w] += ov[w];
            }
            // (no other CTA reads these rows here)
#pragma unroll
            for (int w = 0; w < W; ++w) smem[at + w] = v[w];
        }
        cluster.sync();                                               // (nobody leaves while its sums are being read)
    }
    const auto finish_forward = [&](const GemmCol& c, T top, int u, T v) {
        const T l = Numeric<T>::log_(v) + cst;
        out[c.base + (long long)(i0 + u) * g.N] = top + mos[OP == kFwd ? u : 0] + (eps == T(1) ? l : l / eps);
    };
    if (POS) {
        if (col.base < 0) return;
        if (OP == kFwd) {
#pragma unroll 4
            for (int u = u0 + qb_f; u < u0 + us; u += CPT)
                if (i0 + u < rows) finish_forward(col, cmx, u, smem[u * LDT + eb_f]);
        } else {
            // (all input values of a thread are asked for before the first is used)
            constexpr int PER = TM / CPT < 8 ? TM / CPT : 8;
            for (int first = u0 + qb_f; first < u0 + us; first += CPT * PER) {
                long long a[PER];
                T v[PER];
#pragma unroll
                for (int n = 0; n < PER; ++n) {
                    const int u = first + CPT * n;
                    a[n] = u < u0 + us && i0 + u < rows ? tap_address(g, col, i0 + u, nullptr) : -1;
                    v[n] = a[n] >= 0 ? x[a[n]] : T(0);
                }
#pragma unroll
                for (int n = 0; n < PER; ++n)
                    if (a[n] >= 0) out[a[n]] = Numeric<T>::exp_(eps * (v[n] - cmx)) * smem[(first + CPT * n) * LDT + eb_f];
            }
        }
    } else {
#pragma unroll 4
        for (int i = threadIdx.x; i < us * kTN; i += kGemmThreads) {
            const int e = i / us, u = u0 + i - e * us;
            const GemmCol& c = cols_s[POS ? 0 : e];
            if (c.base < 0 || i0 + u >= rows) continue;
            const T v = smem[u * LDT + e], top = mx_s[POS ? 0 : e];
            if (OP == kFwd) finish_forward(c, top, u, v);
            else {
                const long long a = tap_address(g, c, i0 + u, nullptr);
                if (a >= 0) out[a] = Numeric<T>::exp_(eps * (x[a] - top)) * v;
            }
        }
    }
}

// Adds the splits of a forward pass and finishes the values; `lanes` threads share a value's splits.
template <typename T>
__global__ void __launch_bounds__(256) mex_gemm_finish_fwd(MexGeo g, int splits, int lanes, const T* __restrict__ mo, const T* __restrict__ mx, const T* __restrict__ part,
                                                           T* __restrict__ y, const int* __restrict__ verdict, int verdicts) {
    stream_order();
    if (gemm_unsafe(verdict, verdicts)) return;
    const long long P = (long long)g.B * g.rs, per = (long long)g.R * g.M * P;
    const int lane = threadIdx.x % lanes;
    for (long long first = (long long)blockIdx.x * (256 / lanes); first < per; first += (long long)gridDim.x * (256 / lanes)) {
        const long long idx = first + threadIdx.x / lanes;
        T s = T(0);
        if (idx < per) {
#pragma unroll 8
            for (int q = lane; q < splits; q += lanes) s += part[q * per + idx];
        }
        for (int d = lanes / 2; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane != 0 || idx >= per) continue;
        const long long j = idx % P;
        const int i = int(idx / P % g.M), r = int(idx / P / g.M);
        const GemmCol c = gemm_col(g, r, j, P);
        if (c.base >= 0) y[c.base + (long long)i * g.N] = mx[col_mx(g, c)] + mo[(size_t)r * g.M + i] + (Numeric<T>::log_(s) + T(g.cst)) / T(g.eps);
    }
}

// Input gradient from T[split][r][k][j]: every input value gathers the (tap, position) pairs that meet in it (one pair when
// blocks do not overlap), in tap order.
template <typename T>
__global__ void __launch_bounds__(256) mex_gemm_gather_dx(MexGeo g, FastDiv f_W, FastDiv f_H, FastDiv f_C, int splits, const T* __restrict__ x, const T* __restrict__ mx,
                                                          const T* __restrict__ part, T* __restrict__ dx, const int* __restrict__ verdict, int verdicts) {
    stream_order();
    if (gemm_unsafe(verdict, verdicts)) return;
    const long long P = (long long)g.B * g.rs, total = (long long)g.B * g.C * g.H * g.W;
    const size_t per = (size_t)g.R * g.K * P;
    const T eps = T(g.eps);
    for (long long idx = blockIdx.x * 256LL + threadIdx.x; idx < total; idx += (long long)gridDim.x * 256) {
        int w0, h0, c0, n;
        if (total < 0x7fffffffLL) {                           // (divisions by what the host knows: half of this kernel's time was the others)
            const int a = int(fast_div(uint32_t(idx), f_W)), b = int(fast_div(uint32_t(a), f_H));
            n = int(fast_div(uint32_t(b), f_C));
            w0 = int(idx) - a * g.W; h0 = a - b * g.H; c0 = b - n * g.C;
        } else {
            w0 = int(idx % g.W);
            const long long a = idx / g.W, b = a / g.H;
            h0 = int(a % g.H); c0 = int(b % g.C); n = int(b / g.C);
        }
        const T v = x[idx];
        T sum = T(0);
        // output rows / columns / channels whose block covers this value
        const int cl = max(0, (c0 + g.pc - g.bc) / g.sc + (c0 + g.pc >= g.bc)), ch = min(g.Co - 1, (c0 + g.pc) / g.sc);
        const int hl = max(0, (h0 + g.ph - g.bh) / g.sh + (h0 + g.ph >= g.bh)), hh = min(g.Ho - 1, (h0 + g.ph) / g.sh);
        const int wl = max(0, (w0 + g.pw - g.bw) / g.sw + (w0 + g.pw >= g.bw)), wh = min(g.Wo - 1, (w0 + g.pw) / g.sw);
        // region and place in it along one axis: unshared regions alternate, shared ones are runs
        const auto along = [&](int i, const FastDiv& regions, const FastDiv& run, int& r, int& l) {
            const int q = int(fast_div(uint32_t(i), g.unshared ? regions : run)), m = i - q * int(g.unshared ? regions.d : run.d);
            r = g.unshared ? m : q;
            l = g.unshared ? q : m;
        };
        for (int c = ch; c >= cl; --c) {
            const int rc = g.unshared ? c % g.oc : c / g.rc, lc = g.unshared ? c / g.oc : c % g.rc;
            for (int h = hh; h >= hl; --h) {
                int rh, lh;
                along(h, g.f_oh, g.f_rh, rh, lh);
                const int k0 = ((c0 + g.pc - c * g.sc) * g.bh + h0 + g.ph - h * g.sh) * g.bw + w0 + g.pw;
                const long long j0 = (long long)n * g.rs + (lc * g.rh + lh) * g.rw;
                const T* tops = mx + (long long)n * g.N + (c * g.Ho + h) * g.Wo;
#pragma unroll(sizeof(T) == 4 ? 3 : 1)
                for (int w = wh; w >= wl; --w) {
                    int rw, lw;
                    along(w, g.f_ow, g.f_rw, rw, lw);
                    const T* p = part + ((size_t)((rc * g.oh + rh) * g.ow + rw) * g.K + k0 - w * g.sw) * P + j0 + lw;
                    T t = p[0];
                    for (int q = 1; q < splits; ++q) t += p[q * per];
                    sum += Numeric<T>::exp_(eps * (v - tops[w])) * t;
                }
            }
        }
        dx[idx] = sum;
    }
}

// One CTA per (region, instance): adds the splits of the offsets gradient, times Eo, and takes the gradient back through the
// normalisation when the offsets came raw (v - softmax(row) sum(v)).  Short rows: `groups` threads share a tap's splits.  1024 threads on
// rows of 8192 taps (ten of them in float64: 27 us with 256, 10 so).
template <typename T>
__global__ void __launch_bounds__(1024) mex_gemm_finish_doff(const __grid_constant__ MexGeo g, int splits, int groups, const T* __restrict__ x, const T* __restrict__ off,
                                                             const T* __restrict__ y, const T* __restrict__ dy, T* __restrict__ part, const T* __restrict__ eo,
                                                             const T* __restrict__ raw, const T* __restrict__ lse, T* __restrict__ doff, const int* __restrict__ verdict,
                                                             int verdicts, int normalize, int accumulate) {
    stream_order();
    __shared__ T red[kGemmThreads];
    int bad = 0;
    for (int i = threadIdx.x; i < verdicts; i += blockDim.x) bad |= verdict[i];
    const bool unsafe = __syncthreads_or(bad) != 0;
    const size_t n = (size_t)g.R * g.M * g.K, row = (size_t)blockIdx.x * g.K;
    T sum = T(0);
    const auto keep = [&](int k, T v) {
        if (normalize) part[row + k] = v;
        else doff[row + k] = accumulate ? doff[row + k] + v : v;
        sum += v;
    };
    if (unsafe) {
        for (int k = threadIdx.x; k < g.K; k += blockDim.x) keep(k, part[row + k]);          // (whole sums: exact_doff)
    } else if (groups > 1) {                                  // (K <= 256 / groups, 256 threads)
        const int width = kGemmThreads / groups, k = threadIdx.x % width;
        T v = T(0);
        if (k < g.K)
#pragma unroll 4
            for (int q = threadIdx.x / width; q < splits; q += groups) v += part[q * n + row + k];
        red[threadIdx.x] = v;
        __syncthreads();
        if (threadIdx.x < g.K) {
            for (int q = 1; q < groups; ++q) v += red[q * width + threadIdx.x];
            keep(threadIdx.x, v * eo[row + threadIdx.x]);
        }
        __syncthreads();
    } else {
        for (int k = threadIdx.x; k < g.K; k += blockDim.x) {
            T v = T(0);
#pragma unroll 8
            for (int q = 0; q < splits; ++q) v += part[q * n + row + k];
            keep(k, v * eo[row + k]);
        }
    }
    if (!normalize) return;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = sum;
    __syncthreads();
    sum = T(0);
    for (int w = 0; w < int(blockDim.x / 32); ++w) sum += red[w];
    const T top = lse[blockIdx.x];
    for (int k = threadIdx.x; k < g.K; k += blockDim.x) {     // (a thread reads back what it wrote)
        const T v = part[row + k] - dev_exp(raw[row + k] - top) * sum;
        doff[row + k] = accumulate ? doff[row + k] + v : v;
    }
}

bool gemm_norm(uint32_t flags) { return (flags & SIMNETS_FLAG_MEX_NORMALIZED_OFFSETS) != 0; }
int gemm_verdicts(const MexGeo& g) { return (g.R * g.M + prep_rows(g.K) - 1) / prep_rows(g.K); }
inline int capped_grid(long long n) { return int(std::min<long long>((n + 255) / 256, 16LL * device_sm_count())); }

template <typename T>
cudaError_t gemm_prepare(const MexGeo& g, const GemmWs<T>& w, const T* x, const T* off, uint32_t flags, cudaStream_t s) {
    const long long total = flags & SIMNETS_FLAG_MEX_MAXIMA_GIVEN ? 0 : (long long)g.B * g.N;
    const int prep = gemm_verdicts(g);
    // enough slices of long patches over few positions to fill the GPU
    int lanes = 256;
    while (lanes > 1 && total / lanes < 2LL * device_sm_count() && kGemmThreads / lanes * 4 <= g.K) lanes /= 2;
    // windows that overlap share their pixels' extremes: bands of output rows, as many as give two CTAs per SM and fit the map
    int band = 0;
    long long windows = 0;
    if (total > 0 && (g.sh < g.bh || g.sw < g.bw) && g.bh * g.bw > 1) {
        const long long width = (long long)(g.Wo - 1) * g.sw + g.bw, maps = (long long)g.B * g.Co;
        band = int(std::max<long long>(1, std::min<long long>(g.Ho, maps * g.Ho / (2LL * device_sm_count()))));
        while (band > 1 && ((band - 1LL) * g.sh + g.bh) * width > kGemmMap) --band;
        if (g.bh * width > kGemmMap) band = 0;
        else windows = maps * ((g.Ho + band - 1) / band);
    }
    const long long blocks = prep + (band > 0 ? windows : (total + lanes - 1) / lanes);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    in_stream_order(mex_gemm_prep<T>, unsigned(blocks), kGemmThreads, 0, s)(g, x, off, w.mo, w.eo, w.offn, w.lse, w.verdict, w.mx, prep, int(gemm_norm(flags)), lanes, band);
    count_launch();
    return cudaGetLastError();
}

template <typename T, int OP>
cudaError_t gemm_run(const MexGeo& g, const GemmWs<T>& w, const T* x, const T* off, const T* mx, const T* y, const T* dy, T* out, const GemmPlan& sp, int to_part,
                     cudaStream_t s) {
    const long long blocks = sp.it * sp.jt * g.R;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const dim3 grid(unsigned(blocks), unsigned(sp.splits));
    const int cluster = OP == kDoff || to_part ? 1 : sp.splits;
    const bool along = gemm_along_positions(g, sizeof(T));
#define GEMM_POS(TM, POS) in_stream_order(mex_gemm<T, OP, TM, POS>, grid, kGemmThreads, 0, s, cluster)(g, sp, x, off, w.eo, w.mo, mx, y, dy, out, w.part, w.verdict, gemm_verdicts(g), to_part, w.flag)
#define GEMM(TM) do { if (along) GEMM_POS(TM, true); else GEMM_POS(TM, false); } while (0)
    if (sp.tm == 64) GEMM(64); else if (sp.tm == 32) GEMM(32); else GEMM(16);
#undef GEMM
#undef GEMM_POS
    count_launch();
    return cudaGetLastError();
}

template <typename T>
cudaError_t gemm_dx(const MexGeo& g, GemmWs<T> w, T* products, const T* x, const T* off, const T* y, const T* dy, T* dx, cudaStream_t s) {
    if (overlapping(g)) {
        w.part = products;
    } else {
        const GemmPlan sp = plan_of(g, kDx, Numeric<T>::kQ);
        if (sp.splits == 1 || sp.together) {
            const bool covers = g.pc == 0 && g.ph == 0 && g.pw == 0 && g.sc == g.bc && g.sh == g.bh && g.sw == g.bw && g.C % g.bc == 0 && g.H % g.bh == 0 && g.W % g.bw == 0;
            if (!covers) {
                const cudaError_t e = cudaMemsetAsync(dx, 0, sizeof(T) * (size_t)g.B * g.C * g.H * g.W, s);
                if (e != cudaSuccess) return e;
            }
            return gemm_run<T, kDx>(g, w, x, off, w.mx, y, dy, dx, sp, 0, s);
        }
    }
    // T goes through scratch, as many samples at a time as that has room for
    const int step = overlapping(g) ? overlap_samples(g, sizeof(T)) : g.B;
    for (int n = 0; n < g.B; n += step) {
        const MexGeo q = with_samples(g, std::min(step, g.B - n));
        GemmPlan sp = plan_of(q, kDx, Numeric<T>::kQ);
        const size_t chw = (size_t)g.C * g.H * g.W;
        const T *xn = x + n * chw, *yn = y + (size_t)n * g.M * g.N, *dyn = dy + (size_t)n * g.M * g.Ng, *mxn = w.mx + (size_t)n * g.N;
        if (n > 0 && overlapping(g)) sp.splits = std::min(sp.splits, plan_of(with_samples(g, step), kDx, Numeric<T>::kQ).splits);       // (a short last part must not outgrow the room)
        cudaError_t e = gemm_run<T, kDx>(q, w, xn, off, mxn, yn, dyn, dx + n * chw, sp, 1, s);
        if (e != cudaSuccess) return e;
        in_stream_order(mex_gemm_gather_dx<T>, capped_grid(q.B * (long long)chw), 256, 0, s)(q, make_fastdiv(g.W), make_fastdiv(g.H), make_fastdiv(g.C), sp.splits, xn, mxn, (const T*)w.part, dx + n * chw, (const int*)w.verdict, gemm_verdicts(g));
        count_launch();
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <typename T>
cudaError_t gemm_forward(const MexGeo& g, const T* x, const T* off, T* y, void* ws, uint32_t flags, cudaStream_t s) {
    const GemmWs<T> w = carve_gemm<T>(g, ws);
    cudaError_t e = gemm_prepare(g, w, x, off, flags, s);
    if (e != cudaSuccess) return e;
    const GemmPlan sp = plan_of(g, kFwd, Numeric<T>::kQ);
    e = gemm_run<T, kFwd>(g, w, x, gemm_norm(flags) ? w.offn : off, w.mx, nullptr, nullptr, y, sp, sp.splits > 1 && !sp.together, s);
    if (e != cudaSuccess || sp.splits == 1 || sp.together) return e;
    // (a head's few values over many splits: 32 lanes each, 120 of them over 128 splits in float64 16 -> 4.4 us)
    const long long values = (long long)g.R * g.M * g.B * g.rs;
    const int lanes = sp.splits >= 32 ? 32 : (sp.splits >= 8 ? 8 : 1);
    in_stream_order(mex_gemm_finish_fwd<T>, capped_grid(values * lanes), 256, 0, s)(g, sp.splits, lanes, (const T*)w.mo, (const T*)w.mx, (const T*)w.part, y,
                                                                                    (const int*)w.verdict, gemm_verdicts(g));
    count_launch();
    return cudaGetLastError();
}

template <typename T>
cudaError_t gemm_backward(const MexGeo& g, const T* x, const T* off, const T* y, const T* dy, T* dx, T* doff, bool accumulate, void* ws, void* products, uint32_t flags,
                          cudaStream_t s) {
    GemmWs<T> w = carve_gemm<T>(g, ws);
    // (a primed workspace holds what the forward pass prepared for the same input and offsets, and its status)
    const bool primed = (flags & SIMNETS_FLAG_MEX_WORKSPACE_PRIMED) != 0;
    cudaError_t e = primed ? cudaSuccess : gemm_prepare(g, w, x, off, flags & ~uint32_t(SIMNETS_FLAG_MEX_MAXIMA_GIVEN), s);
    if (primed) w.flag = nullptr;
    if (e != cudaSuccess) return e;
    const T* rows = gemm_norm(flags) ? w.offn : off;
    if (dx != nullptr) {
        e = gemm_dx(g, w, static_cast<T*>(products), x, rows, y, dy, dx, s);
        if (e != cudaSuccess) return e;
    }
    if (doff == nullptr) return cudaSuccess;
    const GemmPlan sp = plan_of(g, kDoff, Numeric<T>::kQ);
    e = gemm_run<T, kDoff>(g, w, x, rows, w.mx, y, dy, doff, sp, 1, s);
    if (e != cudaSuccess) return e;
    int groups = 1;
    while (groups < 32 && g.K * groups * 2 <= kGemmThreads && groups * 4 <= sp.splits) groups *= 2;
    in_stream_order(mex_gemm_finish_doff<T>, g.R * g.M, g.K >= 2048 ? 1024 : kGemmThreads, 0, s)(g, sp.splits, groups, x, rows, y, dy, w.part, (const T*)w.eo, off, (const T*)w.lse, doff,
                                                                            (const int*)w.verdict, gemm_verdicts(g), int(gemm_norm(flags)), int(accumulate));
    count_launch();
    return cudaGetLastError();
}

}  // namespace

// float32 layers small enough for this family.  Forward with pooling + both gradients on the kept workspace, captured, us, here /
// there (pixel layers with 2 x 2 regions; "there" = the tensor-core kernels), around where the two meet:
//     64 over 32, 16x16 pixels    17 M multiply-adds per pass 35 / 39,   34 M  43 / 43,   50 M  51 / 45
//     128 over 64, 8x8            50 M  47 / 49,   67 M  47 / 49,  100 M  62 / 51
//     256 over 128, 8x8          101 M  69 / 70,  134 M  68 / 68,  199 M  92 / 72
//     512 over 256, 4x4          199 M 109 / 117,  268 M 119 / 120,  401 M 171 / 125;   2x2   536 M 219 / 260
//     1024 over 512, 4x4         403 M 189 / 216,  537 M 217 / 219;                     2x2   799 M 351 / 470
// The line grows with the root of the layer's M K, whose chunks the tensor-core kernels walk serially, and lies twice as high on maps of
// up to four pixels, which those read a sector at a time.  Sums are FP32 here, truncated after every eight taps there (distance of y
// from float64, here / there: 64 over 32 4e-8 / 9e-7, 512 over 256 4e-8 / 6e-7 of normal data).
// Overlapping blocks, 24 instances over 12x3x3 taps: 105 M 124 / 192, 837 M 785 / 1121; 64 over 32x3x3: 472 M 246 / 317, 944 M 454 / 527;
// 128 over 32x3x3: 944 M 403 / 409.
// Classifier heads (M <= 16) up to 1024 taps are slower here by 4 to 10 us (512 taps, 0.3 M: 37 / 31) and take half of the launches, which
// is what such a layer costs a host.  Longer patches are read better by their own kernels.
static bool mex_small_layer(const MexGeo& g) {
    const double macs = double(g.R) * g.M * g.K * (double(g.B) * g.rs);
    if (g.M <= 16 && g.K >= 256) return g.K <= 1024 && macs <= 8e6;
    if (overlapping(g)) return g.M < 48 || macs <= 900e6 * 64 / g.M;
    return macs <= 68e6 * std::sqrt(double(g.M) * g.K / 8192.0) * (g.N <= 4 ? 2 : 1);
}
// what every float32 call of this family needs: finite epsilon, positions that 31 bits count, no flag that asks for other kernels
static bool gemm_serves(const MexGeo& g, uint32_t flags) {
    return g.finite && g.B > 0 && (long long)g.B * g.rs < 0x7fffffffLL &&
           !(flags & (SIMNETS_FLAG_FORCE_DIRECT | SIMNETS_FLAG_MEX_EXACT | SIMNETS_FLAG_MEX_NO_TENSORCORE | SIMNETS_FLAG_MEX_TC_ONE_TILE | SIMNETS_FLAG_MEX_NO_PAIR_TILES |
                      SIMNETS_FLAG_MEX_TEST_EXPIRE_WAIT | SIMNETS_FLAG_MEX_NO_SMALL_TILES));
}

bool mex_use_gemm(const MexGeo& g, bool f64, uint32_t flags) {
    if (f64) return g.finite && g.B > 0 && !(flags & (SIMNETS_FLAG_FORCE_DIRECT | SIMNETS_FLAG_MEX_EXACT)) && (long long)g.B * g.rs < 0x7fffffffLL;
    return gemm_serves(g, flags) && mex_small_layer(g);
}
// Gradients of larger layers with too few instances for the tensor cores, whose forward pass other kernels do as well: both gradients, us,
// here / there: 16 instances over 32 taps, 60 M multiply-adds 58 / 221; 8 over 4x2x2, 60 M 193 / 495; 30 over 8x2x2, 601 M 400 / 1586;
// 40 over 64, 600 M 228 / 275; 47 over 200, 600 M 244 / 381.  They prepare their own workspace, in place of the forward pass's.
bool mex_gradients_by_gemm(const MexGeo& g, bool f64, uint32_t flags) {
    return !f64 && g.M < 48 && !(g.M <= 16 && g.K >= 256) && !overlapping(g) && gemm_serves(g, flags) && !mex_small_layer(g);
}
size_t mex_gemm_workspace_bytes(const MexGeo& g, bool f64) { return f64 ? carve_gemm<double>(g, nullptr).bytes : carve_gemm<float>(g, nullptr).bytes; }
size_t mex_gemm_products_bytes(const MexGeo& g, bool f64) {
    const size_t size = f64 ? sizeof(double) : sizeof(float);
    return overlapping(g) ? (part_elements(g, kDx, size) * size + 255) & ~size_t(255) : 0;
}
void* mex_gemm_maxima(const MexGeo& g, bool f64, void* ws) { return f64 ? static_cast<void*>(carve_gemm<double>(g, ws).mx) : carve_gemm<float>(g, ws).mx; }

cudaError_t launch_mex_fwd_gemm(const MexGeo& g, bool f64, const void* x, const void* off, void* y, void* ws, uint32_t flags, cudaStream_t s) {
    return f64 ? gemm_forward<double>(g, (const double*)x, (const double*)off, (double*)y, ws, flags, s) : gemm_forward<float>(g, (const float*)x, (const float*)off, (float*)y, ws, flags, s);
}
cudaError_t launch_mex_bwd_gemm(const MexGeo& g, bool f64, const void* x, const void* off, const void* y, const void* dy, void* dx, void* doff, bool accumulate,
                                void* ws, void* products, uint32_t flags, cudaStream_t s) {
    return f64 ? gemm_backward<double>(g, (const double*)x, (const double*)off, (const double*)y, (const double*)dy, (double*)dx, (double*)doff, accumulate, ws, products, flags, s)
               : gemm_backward<float>(g, (const float*)x, (const float*)off, (const float*)y, (const float*)dy, (float*)dx, (float*)doff, accumulate, ws, products, flags, s);
}

}  // namespace simnets
