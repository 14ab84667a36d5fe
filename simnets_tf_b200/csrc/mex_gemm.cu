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
// Tile: TM rows (16, 32 or 64, whichever pads least) x 64 columns, TM/16 x 4 outputs per thread, 32 (float64: 16) steps of the
// reduction per chunk, double buffered.  The reduction is split over CTAs until two per SM are busy; partial sums are added in split order.
#include <cmath>
#include "kernels.cuh"
#include "mex_exact.cuh"

namespace simnets {
namespace {

constexpr int kTN = 64, kGemmThreads = 256;
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
template <typename T> struct Vec4;
template <> struct Vec4<float> { using type = float4; };
struct __align__(16) Double4 { double x, y, z, w; };
template <> struct Vec4<double> { using type = Double4; };

template <typename T>
struct GemmWs {
    int* flag;           // [2] the workspace's status words
    int* verdict;        // one per CTA of the parameter prepass: offsets that the factorised form cannot take
    T *mo, *lse;         // [R][M]
    T *eo;               // [R][M][K]
    T *offn;             // [R][M][K] offsets minus their row's log-sum-exp, when they come raw
    T *mx;               // [B][N]
    T *part;             // split partial sums
    size_t bytes;
};
enum GemmOp { kFwd, kDx, kDoff };

struct GemmPlan { int it, tm, steps, splits; long long jt; };        // row tiles and their height, reduction length, column tiles (per region)
__host__ GemmPlan plan_of(const MexGeo& g, GemmOp op, int kQ) {
    const long long P = (long long)g.B * g.rs;
    const int rows = op == kDx ? g.K : g.M;
    GemmPlan s;
    s.tm = 64;
    for (int c : {32, 16}) if ((rows + c - 1) / c * c < (rows + s.tm - 1) / s.tm * s.tm) s.tm = c;
    s.it = (rows + s.tm - 1) / s.tm;
    s.jt = ((op == kDoff ? g.K : P) + kTN - 1) / kTN;
    const long long steps = op == kFwd ? g.K : (op == kDx ? g.M : P), tiles = s.it * s.jt * g.R, chunks = (steps + kQ - 1) / kQ;
    long long n = tiles >= 2LL * device_sm_count() ? 1 : (2LL * device_sm_count()) / tiles;
    n = std::max<long long>(1, std::min(n, (chunks * kQ + 63) / 64));       // at least 64 steps each
    s.steps = int(steps);
    s.splits = int(n);
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
    return op == kDoff || s.splits > 1 || (op == kDx && overlapping(g)) ? n * g.R * s.splits : 0;
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
                                                              int prep_ctas, int normalize, int lanes) {
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
        T lse = T(0);
        if (normalize) {
            const T base = isfinite(hi) ? hi : T(0);          // as a stable log-sum-exp treats infinite maxima
            T sum = T(0);
            if (live)
#pragma unroll 4
                for (int k = lane; k < g.K; k += threads) sum += dev_exp(off[row + k] - base);
            lse = base + dev_log(row_reduce<T, true>(sum, red, warp));
        }
        if (live) {
            if (lane == 0) { mo[row_id] = ref - lse; lse_out[row_id] = lse; }
            bad |= !(fabs(g.eps) * double(hi - lo) <= Numeric<T>::kSafe);
#pragma unroll 4
            for (int k = lane; k < g.K; k += threads) {
                const T v = off[row + k];
                if (normalize) offn[row + k] = v - lse;
                eo[row + k] = Numeric<T>::exp_(eps * (v - ref));
            }
        }
        bad = __syncthreads_or(bad);
        if (threadIdx.x == 0) verdict[blockIdx.x] = bad;
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
    for (long long i = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kGemmThreads + threadIdx.x; i < total; i += step) y[i] = mex_exact_y(g, x, off, i);
}
template <typename T>
__device__ __noinline__ void exact_dx(const MexGeo& g, const T* x, const T* off, const T* y, const T* dy, T* dx) {
    const long long total = (long long)g.B * g.C * g.H * g.W, step = (long long)gridDim.x * gridDim.y * kGemmThreads;
    for (long long i = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kGemmThreads + threadIdx.x; i < total; i += step) dx[i] = mex_exact_dx(g, x, off, y, dy, i);
}

// The three contractions.  Rows i: instances (forward, offsets gradient) or taps (input gradient); columns j: positions of one
// region (taps for the offsets gradient); reduction q: taps, instances, positions.
// CTAs per SM that the registers are cut for (24 instances over 12 x 3 x 3 taps, 39 K positions: input gradient 82 us at four, 91
// at three; offsets gradient 52 at three, 56 at four; forward 60 uncut, 63 at three or four)
template <typename T, int OP, int TM>
__host__ __device__ constexpr int gemm_ctas() { return sizeof(T) == 8 || TM == 64 ? 2 : (OP == kDx ? 4 : (OP == kDoff ? 3 : 1)); }

template <typename T, int OP, int TM>
__global__ void __launch_bounds__(kGemmThreads, gemm_ctas<T, OP, TM>()) mex_gemm(const __grid_constant__ MexGeo g, GemmPlan sp, const T* __restrict__ x, const T* __restrict__ off,
                                                         const T* __restrict__ eo, const T* __restrict__ mo, const T* __restrict__ mx, const T* __restrict__ y,
                                                         const T* __restrict__ dy, T* __restrict__ out, T* __restrict__ part, const int* __restrict__ verdict,
                                                         int verdicts, int to_part, int* __restrict__ flag) {
    stream_order();
    constexpr int kQ = Numeric<T>::kQ, EPQ = kGemmThreads / kQ;       // (step fastest: EPQ elements at a time)
    constexpr int NA = TM * kQ / kGemmThreads, NB = kTN * kQ / kGemmThreads;
    constexpr int RM = TM / 16, LDA = TM + 16 / int(sizeof(T)), LDB = kTN + 16 / int(sizeof(T));
    __shared__ __align__(16) T As[2][kQ][LDA], Bs[2][kQ][LDB];
    __shared__ int2 tap_tab[OP == kDx ? 1 : kGemmTaps];
    const int2* tab = OP != kDx && g.bh * g.bw > 1 && taps_tabled(g) ? tap_tab : nullptr;
    if (tab) table_taps(g, tap_tab);                    // (published by the barrier of the next call)
    const bool unsafe = gemm_unsafe(verdict, verdicts);
    if (OP == kFwd && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) flag[threadIdx.x] = threadIdx.x == 0 && unsafe;
    if (unsafe) {
        if (OP == kFwd) exact_forward(g, x, off, out);
        if (OP == kDx) exact_dx(g, x, off, y, dy, out);
        return;                                               // (the offsets gradient's finishing kernel evaluates its rows itself)
    }
    const long long P = (long long)g.B * g.rs;
    const int r = int(blockIdx.x % unsigned(g.R)), split = blockIdx.y;
    const long long tile = blockIdx.x / unsigned(g.R);
    const int i0 = int(tile % sp.it) * TM;
    const long long j0 = tile / sp.it * kTN;
    const int chunks = (sp.steps + kQ - 1) / kQ, c_begin = int((long long)chunks * split / sp.splits), c_end = int((long long)chunks * (split + 1) / sp.splits);
    const T* eor = eo + (size_t)r * g.M * g.K;
    const T* mor = mo + (size_t)r * g.M;
    const T eps = T(g.eps), cst = T(g.cst), oob = T(g.oob);
    // staging, along whichever axis is contiguous in memory: element fastest or reduction step fastest
    const int ea_f = threadIdx.x % TM, qa_f = threadIdx.x / TM, eb_f = threadIdx.x % kTN, qb_f = threadIdx.x / kTN;
    const int q_s = threadIdx.x % kQ, e_s = threadIdx.x / kQ;
    GemmCol jc = {-1, 0, 0, 0, 0, 0, 0, false};
    T jmx = T(0);
    if (OP != kDoff) { jc = gemm_col(g, r, j0 + eb_f, P); if (jc.base >= 0) jmx = mx[col_mx(g, jc)]; }
    T ra[NA], rb[NB];
    auto weight = [&](const GemmCol& c, T cmx, int m) {               // Q[m, position]
        if (c.base < 0 || m >= g.M) return T(0);
        return dy[c.gbase + (long long)m * g.Ng] * Numeric<T>::exp_(eps * (cmx + mor[m] - y[c.base + (long long)m * g.N]) + cst);
    };
    auto ex = [&](const GemmCol& c, T cmx, int k) {                   // Ex[k, position]
        if (c.base < 0 || k >= g.K) return T(0);
        const long long a = tap_address(g, c, k, tab);
        return Numeric<T>::exp_(eps * ((a >= 0 ? x[a] : oob) - cmx));
    };
    auto fetch = [&](int chunk) {
        const int q0 = chunk * kQ;
        if (OP == kDoff) {
            const GemmCol c = gemm_col(g, r, q0 + q_s, P);
            const T cmx = c.base >= 0 ? mx[col_mx(g, c)] : T(0);
#pragma unroll
            for (int s = 0; s < NA; ++s) ra[s] = weight(c, cmx, i0 + e_s + EPQ * s);
#pragma unroll
            for (int s = 0; s < NB; ++s) rb[s] = ex(c, cmx, int(j0) + e_s + EPQ * s);
            return;
        }
#pragma unroll
        for (int s = 0; s < NA; ++s) {
            const int m = OP == kFwd ? i0 + e_s + EPQ * s : q0 + qa_f + kGemmThreads / TM * s, k = OP == kFwd ? q0 + q_s : i0 + ea_f;
            ra[s] = m < g.M && k < g.K ? eor[(size_t)m * g.K + k] : T(0);
        }
#pragma unroll
        for (int s = 0; s < NB; ++s) rb[s] = OP == kFwd ? ex(jc, jmx, q0 + qb_f + 4 * s) : weight(jc, jmx, q0 + qb_f + 4 * s);
    };
    auto commit = [&](int buf) {
#pragma unroll
        for (int s = 0; s < NA; ++s) {
            if (OP == kDx) As[buf][qa_f + kGemmThreads / TM * s][ea_f] = ra[s]; else As[buf][q_s][e_s + EPQ * s] = ra[s];
        }
#pragma unroll
        for (int s = 0; s < NB; ++s) {
            if (OP == kDoff) Bs[buf][q_s][e_s + EPQ * s] = rb[s]; else Bs[buf][qb_f + 4 * s][eb_f] = rb[s];
        }
    };
    const int ti = threadIdx.x / 16, tj = threadIdx.x % 16;           // rows ti RM + a, columns tj 4 + b
    T acc[RM][4];
#pragma unroll
    for (int a = 0; a < RM; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = T(0);
    if (c_begin < c_end) { fetch(c_begin); commit(0); }
    __syncthreads();
    for (int c = c_begin; c < c_end; ++c) {
        const int buf = (c - c_begin) & 1;
        if (c + 1 < c_end) fetch(c + 1);
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            T a[RM], b[4];
            const typename Vec4<T>::type bv = *reinterpret_cast<const typename Vec4<T>::type*>(&Bs[buf][q][tj * 4]);
            b[0] = bv.x; b[1] = bv.y; b[2] = bv.z; b[3] = bv.w;
            if (RM == 2 && sizeof(T) == 4) {
                const float2 av = *reinterpret_cast<const float2*>(&As[buf][q][ti * 2]);
                a[0] = av.x; a[RM > 1 ? 1 : 0] = av.y;
            } else if (RM == 4) {
                const typename Vec4<T>::type av = *reinterpret_cast<const typename Vec4<T>::type*>(&As[buf][q][ti * 4]);
                a[0] = av.x; a[RM > 1 ? 1 : 0] = av.y; a[RM > 2 ? 2 : 0] = av.z; a[RM > 3 ? 3 : 0] = av.w;
            } else {
#pragma unroll
                for (int u = 0; u < RM; ++u) a[u] = As[buf][q][ti * RM + u];
            }
#pragma unroll
            for (int u = 0; u < RM; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
        }
        if (c + 1 < c_end) commit(buf ^ 1);
        __syncthreads();
    }
    const long long rows = OP == kDx ? g.K : g.M, cols = OP == kDoff ? g.K : P;
    if (OP == kDoff || to_part) {
        T* dst = part + ((size_t)split * g.R + r) * rows * cols;
#pragma unroll
        for (int u = 0; u < RM; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const long long i = i0 + ti * RM + u, j = j0 + tj * 4 + v;
                if (i < rows && j < cols) dst[i * cols + j] = acc[u][v];
            }
        return;
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const GemmCol c = gemm_col(g, r, j0 + tj * 4 + v, P);
        if (c.base < 0) continue;
        const T cmx = mx[col_mx(g, c)];
#pragma unroll
        for (int u = 0; u < RM; ++u) {
            const int i = i0 + ti * RM + u;
            if (i >= rows) continue;
            if (OP == kFwd) out[c.base + (long long)i * g.N] = cmx + mor[i] + (Numeric<T>::log_(acc[u][v]) + cst) / eps;
            else {
                const long long a = tap_address(g, c, i, nullptr);
                if (a >= 0) out[a] = Numeric<T>::exp_(eps * (x[a] - cmx)) * acc[u][v];
            }
        }
    }
}

// Adds the splits of a forward pass and finishes the values.
template <typename T>
__global__ void __launch_bounds__(256) mex_gemm_finish_fwd(MexGeo g, int splits, const T* __restrict__ mo, const T* __restrict__ mx, const T* __restrict__ part,
                                                           T* __restrict__ y, const int* __restrict__ verdict, int verdicts) {
    stream_order();
    if (gemm_unsafe(verdict, verdicts)) return;
    const long long P = (long long)g.B * g.rs, per = (long long)g.R * g.M * P;
    for (long long idx = blockIdx.x * 256LL + threadIdx.x; idx < per; idx += (long long)gridDim.x * 256) {
        T s = T(0);
#pragma unroll 8
        for (int q = 0; q < splits; ++q) s += part[q * per + idx];
        const long long j = idx % P;
        const int i = int(idx / P % g.M), r = int(idx / P / g.M);
        const GemmCol c = gemm_col(g, r, j, P);
        if (c.base >= 0) y[c.base + (long long)i * g.N] = mx[col_mx(g, c)] + mo[(size_t)r * g.M + i] + (Numeric<T>::log_(s) + T(g.cst)) / T(g.eps);
    }
}

// Input gradient from T[split][r][k][j]: every input value gathers the (tap, position) pairs that meet in it (one pair when
// blocks do not overlap), in tap order.
template <typename T>
__global__ void __launch_bounds__(256) mex_gemm_gather_dx(MexGeo g, int splits, const T* __restrict__ x, const T* __restrict__ mx, const T* __restrict__ part,
                                                          T* __restrict__ dx, const int* __restrict__ verdict, int verdicts) {
    stream_order();
    if (gemm_unsafe(verdict, verdicts)) return;
    const long long P = (long long)g.B * g.rs, total = (long long)g.B * g.C * g.H * g.W;
    const size_t per = (size_t)g.R * g.K * P;
    const T eps = T(g.eps);
    for (long long idx = blockIdx.x * 256LL + threadIdx.x; idx < total; idx += (long long)gridDim.x * 256) {
        const int w0 = int(idx % g.W);
        long long rest = idx / g.W;
        const int h0 = int(rest % g.H); rest /= g.H;
        const int c0 = int(rest % g.C), n = int(rest / g.C);
        const T v = x[idx];
        T sum = T(0);
        // output rows / columns / channels whose block covers this value
        const int cl = max(0, (c0 + g.pc - g.bc) / g.sc + (c0 + g.pc >= g.bc)), ch = min(g.Co - 1, (c0 + g.pc) / g.sc);
        const int hl = max(0, (h0 + g.ph - g.bh) / g.sh + (h0 + g.ph >= g.bh)), hh = min(g.Ho - 1, (h0 + g.ph) / g.sh);
        const int wl = max(0, (w0 + g.pw - g.bw) / g.sw + (w0 + g.pw >= g.bw)), wh = min(g.Wo - 1, (w0 + g.pw) / g.sw);
        for (int c = ch; c >= cl; --c)
            for (int h = hh; h >= hl; --h)
                for (int w = wh; w >= wl; --w) {
                    const int k = ((c0 + g.pc - c * g.sc) * g.bh + h0 + g.ph - h * g.sh) * g.bw + w0 + g.pw - w * g.sw;
                    const int r = mex_region_of(g, c, h, w);
                    const int lc = g.unshared ? c / g.oc : c % g.rc, lh = g.unshared ? h / g.oh : h % g.rh, lw = g.unshared ? w / g.ow : w % g.rw;
                    const long long j = (long long)n * g.rs + (lc * g.rh + lh) * g.rw + lw;
                    const T* p = part + ((size_t)r * g.K + k) * P + j;
                    T t = p[0];
                    for (int q = 1; q < splits; ++q) t += p[q * per];
                    sum += Numeric<T>::exp_(eps * (v - mx[(long long)n * g.N + (c * g.Ho + h) * g.Wo + w])) * t;
                }
        dx[idx] = sum;
    }
}

// One CTA per (region, instance): adds the splits of the offsets gradient, times Eo, and takes the gradient back through the
// normalisation when the offsets came raw (v - softmax(row) sum(v)).
template <typename T>
__global__ void __launch_bounds__(kGemmThreads) mex_gemm_finish_doff(const __grid_constant__ MexGeo g, int splits, const T* __restrict__ x, const T* __restrict__ off, const T* __restrict__ y,
                                                                     const T* __restrict__ dy, T* __restrict__ part, const T* __restrict__ eo, const T* __restrict__ raw,
                                                                     const T* __restrict__ lse, T* __restrict__ doff, const int* __restrict__ verdict, int verdicts,
                                                                     int normalize, int accumulate) {
    stream_order();
    __shared__ T red[kGemmThreads];
    const bool unsafe = gemm_unsafe(verdict, verdicts);
    const size_t n = (size_t)g.R * g.M * g.K, row = (size_t)blockIdx.x * g.K;
    const int r = blockIdx.x / g.M, m = blockIdx.x - r * g.M;
    T sum = T(0);
    for (int k = threadIdx.x; k < g.K; k += kGemmThreads) {
        T v = T(0);
        if (unsafe) {
            for (long long i = 0; i < (long long)g.B * g.rs; ++i) v += mex_exact_doff_term(g, x, off[row + k], y, dy, r, m, k, i);
        } else {
#pragma unroll 8
            for (int q = 0; q < splits; ++q) v += part[q * n + row + k];
            v *= eo[row + k];
        }
        if (normalize) part[row + k] = v;
        else doff[row + k] = accumulate ? doff[row + k] + v : v;
        sum += v;
    }
    if (!normalize) return;
    sum = row_reduce<T, true>(sum, red, false);
    for (int k = threadIdx.x; k < g.K; k += kGemmThreads) {          // (a thread reads back what it wrote)
        const T v = part[row + k] - dev_exp(raw[row + k] - lse[blockIdx.x]) * sum;
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
    const long long blocks = prep + (total + lanes - 1) / lanes;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    in_stream_order(mex_gemm_prep<T>, unsigned(blocks), kGemmThreads, 0, s)(g, x, off, w.mo, w.eo, w.offn, w.lse, w.verdict, w.mx, prep, int(gemm_norm(flags)), lanes);
    count_launch();
    return cudaGetLastError();
}

template <typename T, int OP>
cudaError_t gemm_run(const MexGeo& g, const GemmWs<T>& w, const T* x, const T* off, const T* mx, const T* y, const T* dy, T* out, const GemmPlan& sp, int to_part,
                     cudaStream_t s) {
    const long long blocks = sp.it * sp.jt * g.R;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const dim3 grid(unsigned(blocks), unsigned(sp.splits));
#define GEMM(TM) in_stream_order(mex_gemm<T, OP, TM>, grid, kGemmThreads, 0, s)(g, sp, x, off, w.eo, w.mo, mx, y, dy, out, w.part, w.verdict, gemm_verdicts(g), to_part, w.flag)
    if (sp.tm == 64) GEMM(64); else if (sp.tm == 32) GEMM(32); else GEMM(16);
#undef GEMM
    count_launch();
    return cudaGetLastError();
}

template <typename T>
cudaError_t gemm_dx(const MexGeo& g, GemmWs<T> w, T* products, const T* x, const T* off, const T* y, const T* dy, T* dx, cudaStream_t s) {
    if (overlapping(g)) {
        w.part = products;
    } else {
        const GemmPlan sp = plan_of(g, kDx, Numeric<T>::kQ);
        if (sp.splits == 1) {
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
        in_stream_order(mex_gemm_gather_dx<T>, capped_grid(q.B * (long long)chw), 256, 0, s)(q, sp.splits, xn, mxn, (const T*)w.part, dx + n * chw, (const int*)w.verdict, gemm_verdicts(g));
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
    e = gemm_run<T, kFwd>(g, w, x, gemm_norm(flags) ? w.offn : off, w.mx, nullptr, nullptr, y, sp, sp.splits > 1, s);
    if (e != cudaSuccess || sp.splits == 1) return e;
    in_stream_order(mex_gemm_finish_fwd<T>, capped_grid((long long)g.R * g.M * g.B * g.rs), 256, 0, s)(g, sp.splits, (const T*)w.mo, (const T*)w.mx, (const T*)w.part, y,
                                                                                                       (const int*)w.verdict, gemm_verdicts(g));
    count_launch();
    return cudaGetLastError();
}

template <typename T>
cudaError_t gemm_backward(const MexGeo& g, const T* x, const T* off, const T* y, const T* dy, T* dx, T* doff, bool accumulate, void* ws, void* products, uint32_t flags,
                          cudaStream_t s) {
    const GemmWs<T> w = carve_gemm<T>(g, ws);
    // (a primed workspace holds what the forward pass prepared for the same input and offsets)
    cudaError_t e = flags & SIMNETS_FLAG_MEX_WORKSPACE_PRIMED ? cudaSuccess : gemm_prepare(g, w, x, off, flags & ~uint32_t(SIMNETS_FLAG_MEX_MAXIMA_GIVEN), s);
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
    in_stream_order(mex_gemm_finish_doff<T>, g.R * g.M, kGemmThreads, 0, s)(g, sp.splits, x, rows, y, dy, w.part, (const T*)w.eo, off, (const T*)w.lse, doff,
                                                                            (const int*)w.verdict, gemm_verdicts(g), int(gemm_norm(flags)), int(accumulate));
    count_launch();
    return cudaGetLastError();
}

}  // namespace

// float32 layers small enough for this family.  Forward with pooling + both gradients on the kept workspace, captured, us, here /
// there (pixel layers with 2 x 2 regions; "there" = the tensor-core kernels):
//     64 over 32, 16x16 pixels     4 M multiply-adds per pass 48 / 37,   17 M  51 / 42,   67 M  88 / 49
//     128 over 64, 8x8             4 M  53 / 45,   17 M  60 / 47,   67 M  78 / 51
//     256 over 128, 8x8            4 M  49 / 62,   25 M  62 / 64,   67 M  74 / 68,  101 M  92 / 70
//     512 over 256, 4x4           17 M  57 / 99,   67 M  78 / 114, 134 M 111 / 119, 200 M 151 / 119
//     1024 over 512, 2x2         200 M 210 / 328
// The line grows with the layer's M K, whose chunks the tensor-core kernels walk serially.  Below M K = 10^4 it lies higher than
// these times alone would have it, by 10 us a layer: sums are FP32 here, truncated after every eight taps there (distance of y from
// float64, here / there: 64 over 32 3e-7 / 9e-7, 128 over 64 4e-7 / 2e-6, 512 over 256 4e-7 / 8e-6), and a forward call with its
// gradients is 6 or 7 launches here and 10 there, which is what such a layer costs a host.
// Overlapping blocks: 24 instances over 12x3x3 taps at 105 M 210 / 248, at 209 M 384 / 428; 8 over 8x5x5 at 41 M 236 / 302.
// Classifier heads (M <= 16) up to 1024 taps: the same reasons; 512 taps at 0.3 M 39 / 31, 1024 at 5 M 59 / 41.  Longer patches
// are read better by their own kernels.
static bool mex_small_layer(const MexGeo& g) {
    const double macs = double(g.R) * g.M * g.K * (double(g.B) * g.rs);
    if (g.M <= 16 && g.K >= 256) return g.K <= 1024 && macs <= 8e6;
    if (overlapping(g)) return macs <= 200e6;
    return macs <= std::min(200e6, std::max(12e6, 25e6 * std::pow(double(g.M) * g.K / 8192.0, 0.75)));
}

// Finite epsilon, and positions that 31 bits count.
bool mex_use_gemm(const MexGeo& g, bool f64, uint32_t flags) {
    if (!g.finite || g.B == 0 || (flags & (SIMNETS_FLAG_FORCE_DIRECT | SIMNETS_FLAG_MEX_EXACT)) || (long long)g.B * g.rs >= 0x7fffffffLL) return false;
    if (f64) return true;
    if (flags & (SIMNETS_FLAG_MEX_NO_TENSORCORE | SIMNETS_FLAG_MEX_TC_ONE_TILE | SIMNETS_FLAG_MEX_NO_PAIR_TILES | SIMNETS_FLAG_MEX_TEST_EXPIRE_WAIT | SIMNETS_FLAG_MEX_NO_SMALL_TILES)) return false;
    return mex_small_layer(g);
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
