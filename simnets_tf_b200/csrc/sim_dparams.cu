// Similarity parameter gradients (float32): per template m and tap k, over all output positions of the batch,
//
//     sT = sum a d,   sW = sum a d^2   (L1: sum a sign(d), sum a |d|),   sN = sum a [x is a number],   a = dy, d = x - t
//
// as a generalized GEMM with rows m, columns k and positions as the reduction index (the reference's element functors:
// HUJI-Deep/simnets-tf include/utils/similarity_utils.hpp:64-119; no patch matrix).
//
// Bound: the FP32 pipe, 4 lane operations per term (5 with missing data).  More than 32 templates over more than 16 taps, blocks of up to 16 x
// 16: sim_dparams_wide, below.  The others (up to 32 templates, up to 16 taps, taller blocks): a CTA of 256 threads owns 32 or 64 templates x
// up to 64 taps, a thread 4 x 2 of them with all its sums in registers: few enough registers for 16 warps per SM, which the chain
// difference -> product -> sums needs (4 x 4 per thread at 12 warps stalled on that chain: FP32 pipe 53 % busy).
// There both operands are contiguous along positions in memory and stay that way in shared memory ([row][position], rows padded by
// four floats so that eight rows of one 16-byte read hit 32 different banks): nothing is transposed, and the packed FP32
// instructions pair two positions, so that no operand needs to be duplicated into both halves.  When the patch is short, the
// threads cover the tile several times over and the copies split the positions of a chunk among themselves (K = 4: sixteen
// ways).  Partial sums of the splits are added in split order.
#include "kernels.cuh"
#include "mma.cuh"
#include "tile.cuh"

namespace simnets {
namespace {

constexpr int kDpThreads = 256, kDpMaxK2 = 32, kDpCtasPerSm = 2;

// Positions after which a thread sets its sums aside (private slots in shared memory) and begins again: one wave of splits leaves a
// split up to all positions, and a sum of that many terms in one register is farther from the exact one the longer it is
// (256 x 64 x 32 x 32 input, 256 templates of 3x3, 65536 positions a split: 2.9e-6 of the gradient's norm; set aside: 5.3e-7).  It costs 1-2 % (L1, the least work per term: 4 %);
// shorter splits instead would write and read their partial sums.
constexpr int kDpFold = 2048;
__host__ __device__ constexpr int dp_slots(int mode) { return mode == SIM_L1 || mode == SIM_L1_SKIP || mode == SIM_L2 ? 16 : 24; }

struct DpTile { int k2, groups, tm, kc; };       // tap columns / 2, copies of the tile per CTA, templates per tile, positions per chunk

// Tile of a patch of K taps: the patch in n equal tiles of at most 64 taps, n the smallest that keeps nearly as many threads
// busy as the best does (K = 36: one tile would leave 112 of 256 threads idle, three of 12 none).  Up to 32 taps a tile takes
// 64 templates, so that a thread still stages few values per term (64 templates of 27 taps over 2048 x 3 x 32 x 32, as this kernel took them: 906
// us in tiles of 32, 760 of 64).  The chunk is long enough that every copy of the tile gets a quad of positions.
__host__ inline DpTile dp_tile(const SimGeo& g) {
    DpTile best = {1, 1, 32, 64};
    double best_busy = 0;
    const int first = (g.K + 2 * kDpMaxK2 - 1) / (2 * kDpMaxK2), last = std::max(first, std::min(first + 3, (g.K + 11) / 12));
    for (int n = first; n <= last; ++n) {
        DpTile t;
        t.k2 = ((g.K + n - 1) / n + 1) / 2;
        t.tm = g.M > 32 && t.k2 >= 2 && t.k2 <= 16 ? 64 : 32;
        t.kc = t.tm == 32 && t.k2 <= 8 ? 64 : 32;
        const int one = t.tm / 4 * t.k2;
        t.groups = std::min(kDpThreads / one, t.kc / 4);
        const int quads = t.kc / 4, rounds = (quads + t.groups - 1) / t.groups;
        const double busy = double(g.K) / (2.0 * t.k2 * n) * (double(one) * quads) / (double(rounds) * kDpThreads);
        if (busy > 1.05 * best_busy) { best_busy = busy; best = t; }
    }
    return best;
}
__host__ inline int dp_tiles(const SimGeo& g, const DpTile& t) { return ((g.M + t.tm - 1) / t.tm) * ((g.K + 2 * t.k2 - 1) / (2 * t.k2)); }

__device__ __forceinline__ float2 dp_abs2(float2 v) { return make_float2(fabsf(v.x), fabsf(v.y)); }
// sign of d, 0 for 0 and NaN as in the reference: 1.0 with d's sign bit, or 0 (two conversions of comparisons cost twice this)
__device__ __forceinline__ float dp_sign(float d) { return fabsf(d) > 0.f ? __uint_as_float(0x3f800000u | (__float_as_uint(d) & 0x80000000u)) : 0.f; }

template <int MODE, int KC, int MAXK, int TM>
__global__ void __launch_bounds__(kDpThreads, kDpCtasPerSm) sim_dparams(SimGeo g, FastDiv f_N, FastDiv f_ow, DpTile tile, const float* __restrict__ x,
                                                             const float* __restrict__ tm, const float* __restrict__ dy,
                                                             float* __restrict__ part, int splits) {
    stream_order();
    constexpr bool MASKED = MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP;
    constexpr bool L1 = MODE == SIM_L1 || MODE == SIM_L1_SKIP;
    // With missing data sN is a contraction that does not involve the templates, dy times a mask of ones and zeros: on tiles of
    // 64 taps the tensor cores take it (dy split in two TF32 parts, the mask exact, one chunk per accumulator), which leaves the
    // FP32 pipe four operations per term instead of five.
    constexpr bool TENSOR_N = MODE == SIM_L2N_NAN && MAXK == 64;
    constexpr bool SUM_N = MASKED && !L1 && !TENSOR_N;
    constexpr int LD = KC + 4, TI = TM / 4;                                           // row stride, floats
    constexpr int A_PER = TM * KC / kDpThreads, B_PER = MAXK * KC / kDpThreads, ROWS = kDpThreads / KC;
    constexpr int A_FLOATS = TM * LD, B_FLOATS = MAXK * LD, STAGE = A_FLOATS + (MASKED ? 2 : 1) * B_FLOATS;
    static_assert(2 * STAGE >= 3 * TM * MAXK || MAXK == 64, "the copies' sums are added up in the stages");
    __shared__ __align__(16) float smem[2 * STAGE];
    extern __shared__ float slots[];                                     // [dp_slots][threads], if a split has more than kDpFold positions
    __shared__ int2 taps[MAXK];                                          // {byte offset inside a sample, kh << 16 | kw}

    const long long P = (long long)g.B * g.N;
    const int TK = 2 * tile.k2, ktiles = (g.K + TK - 1) / TK, mtiles = (g.M + TM - 1) / TM;
    int bid = blockIdx.x;
    const int kt = bid % ktiles; bid /= ktiles;
    const int mt = bid % mtiles, split = bid / mtiles;
    const int m0 = mt * TM, k0 = kt * TK;
    const long long chunks = (P + KC - 1) / KC;
    const long long c_begin = chunks * split / splits, c_end = chunks * (split + 1) / splits;

    for (int i = threadIdx.x; i < MAXK; i += kDpThreads) {
        const int k = k0 + i;
        const int kw = k % g.bw, kh = (k / g.bw) % g.bh, c = k / (g.bw * g.bh);
        taps[i] = k < g.K ? make_int2(4 * ((c * g.H + kh) * g.W + kw), (kh << 16) | kw) : make_int2(0, 0);     // (columns past K: any tap)
    }

    const int G = TI * tile.k2, group = threadIdx.x / G, lid = threadIdx.x - group * G;
    const bool worker = group < tile.groups;
    const int ti = lid & (TI - 1), tj = lid / TI;                        // rows ti + TI r, columns tj + k2 c
    float2 tt[4][2], sT[4][2], sW[4][2], sN[4][SUM_N ? 2 : 1];
    float tN[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};       // 16 templates x 2 x 8 taps per warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, tq = lane & 3, n_row = (warp & 1) * 16, n_col = (warp >> 1) * 16;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int m = m0 + ti + TI * r, k = k0 + tj + tile.k2 * c;
            tt[r][c] = splat2((worker && m < g.M && k < g.K) ? -tm[(size_t)m * g.K + k] : 0.f);
            sT[r][c] = sW[r][c] = make_float2(0.f, 0.f);
            sN[r][SUM_N ? c : 0] = make_float2(0.f, 0.f);
        }

    // staging: this thread brings position q of every chunk, rows e, e + ROWS, ...
    const int q = threadIdx.x % KC, e = threadIdx.x / KC;
    const float oob = float(g.oob);
    float ra[A_PER], rb[B_PER];
    // rows of dy this thread brings (bit s: row e + ROWS s exists) and the first of them
    uint32_t a_rows = 0;
#pragma unroll
    for (int s = 0; s < A_PER; ++s) a_rows |= uint32_t(m0 + e + ROWS * s < g.M) << s;
    const char* dy0 = reinterpret_cast<const char*>(dy) + 4 * (long long)(m0 + e) * g.N;
    const size_t a_step = 4 * (size_t)ROWS * g.N;
    auto fetch = [&](long long chunk) {
        const long long j = chunk * KC + q;
        const bool live = j < P;
        int n = 0, pos = 0;
        if (live) {
            if (P <= 0x7fffffffLL) { n = int(fast_div(uint32_t(j), f_N)); pos = int(j) - n * g.N; }
            else { n = int(j / g.N); pos = int(j - (long long)n * g.N); }
        }
        const int ho = int(fast_div(uint32_t(pos), f_ow)), wo = pos - ho * g.ow;
        const char* a = dy0 + 4 * ((long long)n * g.M * g.N + pos);
        const uint32_t rows = live ? a_rows : 0u;
#pragma unroll
        for (int s = 0; s < A_PER; ++s, a += a_step) {
            ra[s] = 0.f;
            if ((rows >> s) & 1u) ra[s] = __ldg(reinterpret_cast<const float*>(a));
        }
        // dead positions (dy = 0) and columns past K (sums nobody reads) pair with any finite value: they look outside the image
        const int h0 = ho * g.sh - g.ph, w0 = wo * g.sw - g.pw, h_seen = live ? h0 : -0x10000;
        const char* xc = reinterpret_cast<const char*>(x + (size_t)n * g.C * g.H * g.W + h0 * g.W + w0);
        const float outside = live ? oob : 0.f;
#pragma unroll
        for (int s = 0; s < B_PER; ++s) {
            if (MAXK > 4 && ROWS * s >= TK) { rb[s] = 0.f; continue; }
            const int2 t = taps[e + ROWS * s];
            rb[s] = outside;
            if (uint32_t(h_seen + (t.y >> 16)) < uint32_t(g.H) && uint32_t(w0 + (t.y & 0xffff)) < uint32_t(g.W))
                rb[s] = __ldg(reinterpret_cast<const float*>(xc + t.x));
        }
    };
    auto commit = [&](float* stage) {
#pragma unroll
        for (int s = 0; s < A_PER; ++s) stage[(e + ROWS * s) * LD + q] = ra[s];
        float* B = stage + A_FLOATS;
#pragma unroll
        for (int s = 0; s < B_PER; ++s) {
            const int o = (e + ROWS * s) * LD + q;
            if (MASKED) {
                const bool nan = rb[s] != rb[s];
                B[o] = nan ? 0.f : rb[s];
                B[B_FLOATS + o] = nan ? 0.f : 1.f;
            } else {
                B[o] = rb[s];
            }
        }
    };
    auto compute = [&](const float* stage) {
        const float* A = stage + ti * LD;
        const float* B = stage + A_FLOATS + tj * LD;
#pragma unroll 1
        for (int qd = group; qd < KC / 4; qd += tile.groups) {
            float4 a[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4*>(A + TI * r * LD + qd * 4);
            if (MODE == SIM_L2N) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    // (sum of dy per template: the normalisation term's, the same for every tap)
                    sN[r][0] = add2(sN[r][0], add2(make_float2(a[r].x, a[r].y), make_float2(a[r].z, a[r].w)));
                }
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float4 b = *reinterpret_cast<const float4*>(B + c * tile.k2 * LD + qd * 4);
                float4 k4v;
                if (MASKED) k4v = *reinterpret_cast<const float4*>(B + B_FLOATS + c * tile.k2 * LD + qd * 4);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float2 b2 = half ? make_float2(b.z, b.w) : make_float2(b.x, b.y);
                    float2 k2;
                    if (MASKED) k2 = half ? make_float2(k4v.z, k4v.w) : make_float2(k4v.x, k4v.y);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float2 a2 = half ? make_float2(a[r].z, a[r].w) : make_float2(a[r].x, a[r].y);
                        const float2 d = MASKED ? fma2(tt[r][c], k2, b2) : add2(b2, tt[r][c]);
                        if (L1) {
                            sT[r][c] = fma2(a2, make_float2(dp_sign(d.x), dp_sign(d.y)), sT[r][c]);
                            sW[r][c] = fma2(a2, dp_abs2(d), sW[r][c]);
                        } else {
                            const float2 u = mul2(a2, d);
                            sT[r][c] = add2(sT[r][c], u);
                            sW[r][c] = fma2(u, d, sW[r][c]);
                            if (SUM_N) sN[r][SUM_N ? c : 0] = fma2(a2, k2, sN[r][SUM_N ? c : 0]);
                        }
                    }
                }
            }
        }
    };

    auto compute_n = [&](const float* stage) {
        const float* A = stage + (n_row + gq) * LD + tq;
        const float* K = stage + A_FLOATS + B_FLOATS + (n_col + gq) * LD + tq;
        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int p = 0; p < KC; p += 8) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float2 v = split_tf32(A[(u & 1) * 8 * LD + p + (u >> 1) * 4]);
                hi[u] = __float_as_uint(v.x); lo[u] = __float_as_uint(v.y);
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t b0 = __float_as_uint(K[c * 8 * LD + p]), b1 = __float_as_uint(K[c * 8 * LD + p + 4]);
                mma_tf32(s[c], lo, b0, b1);
                mma_tf32(s[c], hi, b0, b1);
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u) tN[c][u] += s[c][u];
    };

    __syncthreads();                                                     // the tap table
    const int n_chunks = int(c_end - c_begin);
    if (n_chunks > 0) {
        fetch(c_begin);
        commit(smem);
        __syncthreads();
        for (int i = 0;;) {
            const int stop = min(n_chunks, i + kDpFold / KC);
            for (; i < stop; ++i) {
                float* now = smem + (i & 1) * STAGE;
                float* next = smem + ((i + 1) & 1) * STAGE;
                const bool more = i + 1 < n_chunks;
                if (more) fetch(c_begin + i + 1);
                if (TENSOR_N) compute_n(now);
                if (worker) compute(now);
                if (more) commit(next);
                __syncthreads();
            }
            if (i == n_chunks) break;
            const bool first = i == kDpFold / KC;
            float* s = slots + threadIdx.x;
            auto aside = [&](float2& v) {
                const float now = v.x + v.y;
                *s = first ? now : *s + now;
                s += kDpThreads;
                v = make_float2(0.f, 0.f);
            };
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    aside(sT[r][c]);
                    aside(sW[r][c]);
                    if (SUM_N || (c == 0 && MODE == SIM_L2N)) aside(sN[r][SUM_N ? c : 0]);
                }
        }
        if (n_chunks > kDpFold / KC) {
            const float* s = slots + threadIdx.x;
            auto join = [&](float2& v) { v.x += *s; s += kDpThreads; };
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    join(sT[r][c]);
                    join(sW[r][c]);
                    if (SUM_N || (c == 0 && MODE == SIM_L2N)) join(sN[r][SUM_N ? c : 0]);
                }
        }
    }

    // the copies' sums, one after the other; then this split's partial sums
    const size_t mk = (size_t)g.M * g.K;
    float* dst = part + (size_t)split * 3 * mk;
    const int last = tile.groups - 1;
    for (int grp = 0; grp <= last; ++grp) {
        if (group == grp) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    float v[3] = {sT[r][c].x + sT[r][c].y, sW[r][c].x + sW[r][c].y, 0.f};
                    if (SUM_N) v[2] = sN[r][SUM_N ? c : 0].x + sN[r][SUM_N ? c : 0].y;
                    else if (!L1) v[2] = sN[r][0].x + sN[r][0].y;
                    const int row = ti + TI * r, col = tj + tile.k2 * c, m = m0 + row, k = k0 + col;
#pragma unroll
                    for (int p = 0; p < (TENSOR_N ? 2 : 3); ++p) {
                        float* s = smem + (p * TM + row) * TK + col;
                        if (grp > 0) v[p] += *s;
                        if (grp < last) *s = v[p];
                        else if (m < g.M && k < g.K) dst[p * mk + (size_t)m * g.K + k] = v[p];
                    }
                }
        }
        if (grp < last) __syncthreads();
    }
    if (TENSOR_N)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int m = m0 + n_row + gq + 8 * (u >> 1), col = n_col + 8 * c + 2 * tq + (u & 1), k = k0 + col;
                if (m < g.M && col < TK && k < g.K) dst[2 * mk + (size_t)m * g.K + k] = tN[c][u];
            }
}

// ---------------------------------------------------------------------------------------------------------- 64 templates
// Tiles of 64 templates x 64 taps (x 32 where the patch has no more, two copies of the tile splitting a chunk's positions).
//
// On this pipe every instruction beside the packed arithmetic costs about two cycles that no other warp fills (parts of the kernel
// above switched off one at a time, 256 x 64 x 32 x 32 input, 256 templates of 3x3, 20 % missing: 9363 us whole, 8330 without sN,
// 7396 without loads, 6181 with neither; interleaving the loads with the products changed nothing).  So the tile is as large as the
// registers allow: a position brings 128 values for 4096 terms instead of 96 for 2048, and the bounds of a tap are one test of two
// bits against what the position's patch misses.  That case: 7.6 ms (5.2 without sN and staging); 64 templates of 3x3 over 2048 x 3 x
// 32 x 32: 760 -> 675 us (552 without staging, its 27 taps in 32 columns).  sN as a fifth packed operation takes what fragments on the
// tensor cores took (7.5 ms): a warp-sized TF32 product holds this pipe up for some twenty cycles.
//
// Operands lie [position][row], so that the packed instructions pair two TAPS: a thread owns 4 templates x 2 pairs of taps with one
// register per sum, half of what pairing positions takes, and reads 12 values (with masks) per position for 16 terms.  A staging
// thread brings two neighbouring rows of one position and stores them as one pair at slot pair ^ ((position >> 2) & 3) of a row of
// 64 + 8 (32 + 8) floats: the stores of 16 positions and the 16-byte reads of eight column groups each hit 32 different banks, and the reading loop knows position & 15 at compile time.
constexpr int kDwTM = 64, kDwKC = 32;
// As kDpFold; one chain per sum here, two or more there, so the chains are shorter: chunks after which a thread sets its sums aside
__host__ inline int dw_fold(long long positions) { return positions <= 512 ? 2 : positions <= 1024 ? 4 : positions <= 4096 ? 8 : 16; }
template <int MODE, int WJ> struct DwTile {
    static constexpr bool MASKED = MODE == SIM_L2N_NAN || MODE == SIM_L1_SKIP;
    static constexpr int TK = 32 * WJ, LDA = kDwTM + 8, LDB = TK + 8, A_FLOATS = kDwKC * LDA, B_FLOATS = kDwKC * LDB;
    static constexpr int STAGE = A_FLOATS + (MASKED ? 2 : 1) * B_FLOATS;
    static constexpr int SMEM = 8 * STAGE, SLOT_BYTES = 4 * (MODE == SIM_L2N_NAN ? 48 : 32) * kDpThreads;        // bytes: two stages; sums set aside
};

// a sign(d); a0 = 0 a where d is 0 or NaN, which is NaN for an a that is no finite number
__device__ __forceinline__ float dw_signed(float a, float a0, float d) { return fabsf(d) > 0.f ? __uint_as_float(__float_as_uint(a) ^ (__float_as_uint(d) & 0x80000000u)) : a0; }

template <int MODE, int WJ>
__global__ void __launch_bounds__(kDpThreads, kDpCtasPerSm) sim_dparams_wide(const __grid_constant__ SimGeo g, FastDiv f_N, FastDiv f_ow, int TK, const float* __restrict__ x,
                                                                             const float* __restrict__ tm, const float* __restrict__ dy,
                                                                             float* __restrict__ part, int splits, int fold) {
    stream_order();
    using Tile = DwTile<MODE, WJ>;
    constexpr bool MASKED = Tile::MASKED, L1 = MODE == SIM_L1 || MODE == SIM_L1_SKIP, SUM_N = MODE == SIM_L2N_NAN, ROW_N = MODE == SIM_L2N;
    constexpr int KC = kDwKC, LDA = Tile::LDA, LDB = Tile::LDB, A_FLOATS = Tile::A_FLOATS, B_FLOATS = Tile::B_FLOATS, STAGE = Tile::STAGE;
    constexpr int A_PAIRS = 4, B_PAIRS = 2 * WJ;                          // pairs staged per thread
    extern __shared__ __align__(16) float smem[];
    float* slots = smem + 2 * STAGE;                                     // [sums][threads], if a split has more than `fold` chunks
    __shared__ int4 taps[16 * WJ];                                       // pairs of {byte offset inside a sample, bit kh | bit 16 + kw}

    const long long P = (long long)g.B * g.N;
    const int ktiles = (g.K + TK - 1) / TK, mtiles = (g.M + kDwTM - 1) / kDwTM;
    int bid = blockIdx.x;
    const int kt = bid % ktiles; bid /= ktiles;
    const int mt = bid % mtiles, split = bid / mtiles;
    const int m0 = mt * kDwTM, k0 = kt * TK, k_end = min(g.K, k0 + TK);
    const long long chunks = (P + KC - 1) / KC;
    const long long c_begin = chunks * split / splits, c_end = chunks * (split + 1) / splits;

    if (threadIdx.x < 32 * WJ) {
        const int k = k0 + threadIdx.x;
        const int kw = k % g.bw, kh = (k / g.bw) % g.bh, c = k / (g.bw * g.bh);
        // (columns past the tile: out of every image)
        reinterpret_cast<int2*>(taps)[threadIdx.x] = k < k_end ? make_int2(4 * ((c * g.H + kh) * g.W + kw), (1 << kh) | (0x10000 << kw)) : make_int2(0, -1);
    }

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // 4 x 8 threads per warp (pairs of rows interleaved, as in tile.cuh), 4 x WJ warps per copy of the tile
    const int ti = (warp & 3) * 4 + (((lane >> 4) << 1) | (lane & 1)), tj = (WJ == 2 ? (warp >> 2) * 8 : 0) + ((lane & 15) >> 1), copy = WJ == 2 ? 0 : warp >> 2;
    float2 tt[4][2], sT[4][2], sW[4][2], sN[SUM_N ? 4 : 1][SUM_N ? 2 : 1];
    bool odd_t = false;                                                  // an infinite or NaN template (L1)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int m = m0 + ti * 4 + r, k = k0 + tj * 4 + 2 * c;
            // (rows and columns past the tile, whose sums nobody reads: never a difference of 0)
            tt[r][c].x = m < g.M && k < k_end ? -tm[(size_t)m * g.K + k] : -1e30f;
            tt[r][c].y = m < g.M && k + 1 < k_end ? -tm[(size_t)m * g.K + k + 1] : -1e30f;
            odd_t |= !(fabsf(tt[r][c].x) < CUDART_INF_F) || !(fabsf(tt[r][c].y) < CUDART_INF_F);
            sT[r][c] = sW[r][c] = sN[SUM_N ? r : 0][SUM_N ? c : 0] = make_float2(0.f, 0.f);
        }
    float rowN[ROW_N ? 2 * A_PAIRS : 1];                                 // the sums of dy of the rows this thread stages
#pragma unroll
    for (int i = 0; i < (ROW_N ? 2 * A_PAIRS : 1); ++i) rowN[i] = 0.f;

    // staging: position `lane` of every chunk, rows 2 (warp + 8 s) and the one behind it
    const float oob = float(g.oob);
    float2 ra[A_PAIRS], rb[B_PAIRS];
    uint32_t a_rows = 0;
#pragma unroll
    for (int s = 0; s < 2 * A_PAIRS; ++s) a_rows |= uint32_t(m0 + 2 * (warp + 8 * (s >> 1)) + (s & 1) < g.M) << s;
    const char* dy0 = reinterpret_cast<const char*>(dy) + 4 * (long long)(m0 + 2 * warp) * g.N;
    const size_t a_step = 4 * (size_t)g.N;
    auto fetch = [&](long long chunk) {
        const long long j = chunk * KC + lane;
        const bool live = j < P;
        int n = 0, pos = 0;
        if (live) {
            if (P <= 0x7fffffffLL) { n = int(fast_div(uint32_t(j), f_N)); pos = int(j) - n * g.N; }
            else { n = int(j / g.N); pos = int(j - (long long)n * g.N); }
        }
        const int ho = int(fast_div(uint32_t(pos), f_ow)), wo = pos - ho * g.ow;
        const char* a = dy0 + 4 * ((long long)n * g.M * g.N + pos);
        const uint32_t rows = live ? a_rows : 0u;
#pragma unroll
        for (int s = 0; s < A_PAIRS; ++s) {
            ra[s] = make_float2(0.f, 0.f);
            if ((rows >> (2 * s)) & 1u) ra[s].x = __ldg(reinterpret_cast<const float*>(a + 16 * s * a_step));
            if ((rows >> (2 * s + 1)) & 1u) ra[s].y = __ldg(reinterpret_cast<const float*>(a + (16 * s + 1) * a_step));
        }
        // dead positions pair dy = 0 with a finite value
        const int h0 = ho * g.sh - g.ph, w0 = wo * g.sw - g.pw;
        const int missing = live ? int(missing_taps(h0, g.H) | (missing_taps(w0, g.W) << 16)) : -1;
        const char* xc = reinterpret_cast<const char*>(x + (size_t)n * g.C * g.H * g.W + h0 * g.W + w0);
        const float outside = live ? oob : 0.f;
#pragma unroll
        for (int s = 0; s < B_PAIRS; ++s) {
            const int4 t = taps[warp + 8 * s];
            rb[s] = make_float2(outside, outside);
            if ((t.y & missing) == 0) rb[s].x = __ldg(reinterpret_cast<const float*>(xc + t.x));
            if ((t.w & missing) == 0) rb[s].y = __ldg(reinterpret_cast<const float*>(xc + t.z));
        }
    };
    const int st_a = lane * LDA + 2 * (warp ^ ((lane >> 2) & 3)), st_b = lane * LDB + 2 * (warp ^ ((lane >> 2) & 3));
    auto commit = [&](float* stage) {                                    // returns whether a value is infinite or NaN (L1)
        bool odd = false;
#pragma unroll
        for (int s = 0; s < A_PAIRS; ++s) {
            *reinterpret_cast<float2*>(stage + st_a + 16 * s) = ra[s];
            if (ROW_N) { rowN[ROW_N ? 2 * s : 0] += ra[s].x; rowN[ROW_N ? 2 * s + 1 : 0] += ra[s].y; }
        }
        float* B = stage + A_FLOATS;
#pragma unroll
        for (int s = 0; s < B_PAIRS; ++s) {
            float2 v = rb[s];
            if (MASKED) {
                const bool nx = v.x != v.x, ny = v.y != v.y;
                v = make_float2(nx ? 0.f : v.x, ny ? 0.f : v.y);
                *reinterpret_cast<float2*>(B + B_FLOATS + st_b + 16 * s) = make_float2(nx ? 0.f : 1.f, ny ? 0.f : 1.f);
            }
            if (MODE == SIM_L1) odd |= !(fabsf(v.x) < CUDART_INF_F) || !(fabsf(v.y) < CUDART_INF_F);
            *reinterpret_cast<float2*>(B + st_b + 16 * s) = v;
        }
        return odd;
    };

    // sixteen positions, from the stage's row 16 half; plain: no infinity or NaN among the operands (L1)
    auto compute = [&](const float* stage, int half, bool plain) {
        const float* A0 = stage + 16 * half * LDA + ti * 4;
        const float* A1 = stage + 16 * half * LDA + (ti ^ 1) * 4;
        const float* B0 = stage + A_FLOATS + 16 * half * LDB + tj * 4;
        const float* B1 = stage + A_FLOATS + 16 * half * LDB + (tj ^ 1) * 4;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int sw = q >> 2;                                        // 16-byte groups swapped by its bit 1, pairs inside one by its bit 0
            const float4 av = *reinterpret_cast<const float4*>((sw & 2 ? A1 : A0) + q * LDA), bv = *reinterpret_cast<const float4*>((sw & 2 ? B1 : B0) + q * LDB);
            const float a[4] = {sw & 1 ? av.z : av.x, sw & 1 ? av.w : av.y, sw & 1 ? av.x : av.z, sw & 1 ? av.y : av.w};
            const float2 b[2] = {sw & 1 ? make_float2(bv.z, bv.w) : make_float2(bv.x, bv.y), sw & 1 ? make_float2(bv.x, bv.y) : make_float2(bv.z, bv.w)};
            float2 k[2];
            if (MASKED) {
                const float4 kv = *reinterpret_cast<const float4*>((sw & 2 ? B1 : B0) + B_FLOATS + q * LDB);
                k[0] = sw & 1 ? make_float2(kv.z, kv.w) : make_float2(kv.x, kv.y);
                k[1] = sw & 1 ? make_float2(kv.x, kv.y) : make_float2(kv.z, kv.w);
            }
            if (L1) {
                float2 d[4][2];
                float least = CUDART_INF_F;
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        d[r][c] = MASKED ? fma2(tt[r][c], k[c], b[c]) : add2(b[c], tt[r][c]);
                        if (!MASKED) least = fminf(fminf(least, fabsf(d[r][c].x)), fabsf(d[r][c].y));
                    }
                // a sign(d) is a with d's sign bit added while no d is 0 or NaN: one instruction per term instead of three
                if (!MASKED && plain && least > 0.f) {
#pragma unroll
                    for (int r = 0; r < 4; ++r)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const float2 u = make_float2(__uint_as_float(__float_as_uint(a[r]) ^ (__float_as_uint(d[r][c].x) & 0x80000000u)),
                                                         __uint_as_float(__float_as_uint(a[r]) ^ (__float_as_uint(d[r][c].y) & 0x80000000u)));
                            sT[r][c] = add2(sT[r][c], u);
                            sW[r][c] = fma2(u, d[r][c], sW[r][c]);
                        }
                } else {
                    const float a0[4] = {a[0] * 0.f, a[1] * 0.f, a[2] * 0.f, a[3] * 0.f};
#pragma unroll
                    for (int r = 0; r < 4; ++r)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            sT[r][c] = add2(sT[r][c], make_float2(dw_signed(a[r], a0[r], d[r][c].x), dw_signed(a[r], a0[r], d[r][c].y)));
                            sW[r][c] = fma2(splat2(a[r]), dp_abs2(d[r][c]), sW[r][c]);
                        }
                }
                continue;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float2 d = MASKED ? fma2(tt[r][c], k[c], b[c]) : add2(b[c], tt[r][c]);
                    const float2 u = mul2(splat2(a[r]), d);
                    sT[r][c] = add2(sT[r][c], u);
                    sW[r][c] = fma2(u, d, sW[r][c]);
                    if (SUM_N) sN[SUM_N ? r : 0][SUM_N ? c : 0] = fma2(splat2(a[r]), k[c], sN[SUM_N ? r : 0][SUM_N ? c : 0]);
                }
        }
    };
    __syncthreads();                                                     // the tap table
    const int n_chunks = int(c_end - c_begin);
    if (n_chunks > 0) {
        fetch(c_begin);
        bool odd = commit(smem);
        odd = MODE == SIM_L1 ? __syncthreads_or(odd) != 0 : (__syncthreads(), false);
        for (int i = 0;;) {
            const int stop = min(n_chunks, i + fold);
            for (; i < stop; ++i) {
                float* now = smem + (i & 1) * STAGE;
                float* next = smem + ((i + 1) & 1) * STAGE;
                const bool more = i + 1 < n_chunks, plain = !odd && !odd_t;
                if (more) fetch(c_begin + i + 1);
                if (WJ == 2) {
#pragma unroll 1
                    for (int half = 0; half < 2; ++half) compute(now, half, plain);
                } else compute(now, copy, plain);
                odd = false;
                if (more) odd = commit(next);
                odd = MODE == SIM_L1 ? __syncthreads_or(odd) != 0 : (__syncthreads(), false);
            }
            if (i == n_chunks) break;
            const bool first = i == fold;
            float* s = slots + threadIdx.x;
            auto aside = [&](float& v) { *s = first ? v : *s + v; s += kDpThreads; v = 0.f; };
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    aside(sT[r][c].x); aside(sT[r][c].y); aside(sW[r][c].x); aside(sW[r][c].y);
                    if (SUM_N) { aside(sN[SUM_N ? r : 0][SUM_N ? c : 0].x); aside(sN[SUM_N ? r : 0][SUM_N ? c : 0].y); }
                }
        }
        if (n_chunks > fold) {
            const float* s = slots + threadIdx.x;
            auto join = [&](float& v) { v += *s; s += kDpThreads; };
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    join(sT[r][c].x); join(sT[r][c].y); join(sW[r][c].x); join(sW[r][c].y);
                    if (SUM_N) { join(sN[SUM_N ? r : 0][SUM_N ? c : 0].x); join(sN[SUM_N ? r : 0][SUM_N ? c : 0].y); }
                }
        }
    }

    const size_t mk = (size_t)g.M * g.K;
    float* dst = part + (size_t)split * 3 * mk;
    float* row_sum = smem;                                               // [64] sums of dy (ROW_N), behind them the second copy's sums
    float2* other = reinterpret_cast<float2*>(smem + kDwTM) + (threadIdx.x & 127);
    constexpr int SUMS = SUM_N ? 3 : 2;
    if (WJ == 1 && copy == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            other[(i * SUMS) * 128] = sT[i >> 1][i & 1];
            other[(i * SUMS + 1) * 128] = sW[i >> 1][i & 1];
            if (SUM_N) other[(i * SUMS + 2) * 128] = sN[SUM_N ? i >> 1 : 0][SUM_N ? i & 1 : 0];
        }
    }
    if (ROW_N) {
#pragma unroll
        for (int i = 0; i < 2 * A_PAIRS; ++i) {
            float v = rowN[ROW_N ? i : 0];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if (lane == 0) row_sum[2 * (warp + 8 * (i >> 1)) + (i & 1)] = v;
        }
    }
    __syncthreads();
    if (copy != 0) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = i >> 1, c = i & 1, m = m0 + ti * 4 + r, k = k0 + tj * 4 + 2 * c;
        float2 v[3] = {sT[r][c], sW[r][c], SUM_N ? sN[SUM_N ? r : 0][SUM_N ? c : 0] : make_float2(0.f, 0.f)};
        if (WJ == 1) {
#pragma unroll
            for (int u = 0; u < SUMS; ++u) v[u] = add2(v[u], other[(i * SUMS + u) * 128]);
        }
        if (ROW_N) v[2] = splat2(row_sum[ti * 4 + r]);
#pragma unroll
        for (int u = 0; u < (L1 || MODE == SIM_L2 ? 2 : 3); ++u) {
            float* p = dst + u * mk + (size_t)m * g.K + k;
            if (m < g.M && k < k_end) p[0] = v[u].x;
            if (m < g.M && k + 1 < k_end) p[1] = v[u].y;
        }
    }
}

// Sums the splits' partial sums in split order and applies the per-parameter factors of the backward functors.  512 threads =
// `slices` slices of the splits x 512 / slices consecutive outputs; the slices are added in a fixed order (same sums on every
// run).  Many splits (short patches: K = 27, 222 splits): 64 slices, so that the few outputs still spread over a couple of
// hundred CTAs; few splits (K = 576: 6): 8 slices, 64 outputs per CTA.
__global__ void __launch_bounds__(512) sim_dparams_reduce(SimGeo g, int splits, int slices, const float* __restrict__ part,
                                                          const float* __restrict__ wt, float* __restrict__ dt, float* __restrict__ dw,
                                                          int accumulate) {
    stream_order();
    __shared__ float red[3][512];
    const int mk = g.M * g.K, lanes = 512 / slices;
    const float fudge = float(g.fudge);
    const bool third = g.mode == SIM_L2N || g.mode == SIM_L2N_NAN;
    const int lane = threadIdx.x & (lanes - 1), slice = threadIdx.x / lanes;
    for (int first = blockIdx.x * lanes; first < mk; first += gridDim.x * lanes) {
        const int i = first + lane;
        float a = 0.f, b = 0.f, c = 0.f;
        if (i < mk) {
#pragma unroll 4
            for (int s = slice; s < splits; s += slices) {
                const float* p = part + (size_t)s * 3 * mk;
                a += p[i]; b += p[mk + i];
                if (third) c += p[2 * mk + i];
            }
        }
        red[0][threadIdx.x] = a; red[1][threadIdx.x] = b; red[2][threadIdx.x] = c;
        __syncthreads();
        if (slice == 0 && i < mk) {
#pragma unroll 8
            for (int q = 1; q < slices; ++q) { a += red[0][q * lanes + lane]; b += red[1][q * lanes + lane]; c += red[2][q * lanes + lane]; }
            const float wraw = wt ? wt[i] : 1.f, w = g.absw ? fabsf(wraw) : wraw;
            float gt, gw;
            if (wt == nullptr) { gt = a; gw = b; }           // no weights: the plain sums (the statistics of mixture.cu)
            else if (g.mode == SIM_L1 || g.mode == SIM_L1_SKIP) { gt = w * a; gw = -b; }
            else if (g.mode == SIM_L2) { gt = 2.f * w * a; gw = -b; }
            else { gt = w * a; gw = 0.5f * (c / (w + fudge) - b); }
            if (g.absw) gw *= wraw > 0.f ? 1.f : (wraw < 0.f ? -1.f : 0.f);          // d|w|/dw, 0 at w = 0
            dt[i] = accumulate ? dt[i] + gt : gt;
            dw[i] = accumulate ? dw[i] + gw : gw;
        }
        __syncthreads();
    }
}

}  // namespace

// Whether tiles of 64 templates x 64 (32) taps serve a shape, and how many taps such a tile takes (the patch in equal parts).  Filled alike,
// they are 1.01 to 1.33 times as fast as the smaller ones (275 shapes of 33 to 192 templates and 17 to 144 taps, 96 x C x 32 x 32; least with
// missing data, most in L1).  Where they are filled 0.75 times as well (17 to 20 and 33 to 48 taps; 65 to 96 templates over 64 columns) both take the
// same within 7 %, with missing data up to 12 % more here (96 templates of 13x2x2 taps 144 -> 163 us, 64 of 4x3x3 L2 63 -> 68, L1 1.00 to 1.10
// faster).  They stay there too: the sums are shorter and in FP32 throughout (templates gradients 2.0e-7 to 3.3e-7 of their norm from
// float64 over 96 samples, 2.3e-7 to 5.6e-7 there).
static int dw_taps(const SimGeo& g) {
    if (g.M <= 32 || g.K <= 16 || g.bh > 16 || g.bw > 16) return 0;
    // (a term of the narrower tile costs some 15 % more staging)
    const int n32 = (g.K + 31) / 32, n64 = (g.K + 63) / 64, n = 1.15 * 32 * n32 < 64 * n64 ? n32 : n64;
    return (g.K + n - 1) / n;
}
static int dw_tiles(const SimGeo& g, int tk) { return ((g.M + kDwTM - 1) / kDwTM) * ((g.K + tk - 1) / tk); }

// How many ways the positions are split: one wave of the CTAs that fit the GPU at once, fewer where a split would hold under 256
// positions (its partial sums are 3 M K floats written and read again).
int sim_dparams_splits(const SimGeo& g) {
    const DpTile t = dp_tile(g);
    const int wide = dw_taps(g), kc = wide > 0 ? kDwKC : t.kc;
    const long long P = (long long)g.B * g.N, chunks = (P + kc - 1) / kc, tiles = wide > 0 ? dw_tiles(g, wide) : dp_tiles(g, t);
    long long s = (device_sm_count() * kDpCtasPerSm) / tiles;
    s = std::min(s, std::max<long long>(1, P / 256));
    return int(std::max<long long>(1, std::min(s, chunks)));
}

cudaError_t launch_sim_dparams(const SimGeo& g, const float* x, const float* t, const float* w, const float* dy, float* dt, float* dw,
                               bool accumulate, float* part, cudaStream_t s) {
    if (!sim_offsets_below(g, 1LL << 29)) return launch_sim_dparams_direct(g, false, x, t, w, dy, dt, dw, accumulate, s);    // (32-bit byte offsets)
    const DpTile tile = dp_tile(g);
    const int splits = sim_dparams_splits(g), wide = dw_taps(g);
    const long long blocks = (long long)(wide > 0 ? dw_tiles(g, wide) : dp_tiles(g, tile)) * splits;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const FastDiv f_N = make_fastdiv(g.N), f_ow = make_fastdiv(g.ow);
    const bool folds = ((long long)g.B * g.N + splits - 1) / splits > kDpFold - tile.kc;          // (a split may have one chunk more than another)
#define DP_TILE(MODE, KC, MAXK, TM)                                                                                                                  \
    do {                                                                                                                                             \
        constexpr int bytes = 4 * kDpThreads * dp_slots(MODE);                                                                                       \
        static SmemLimit limit;                                                                                                                      \
        const cudaError_t e = limit.raise(sim_dparams<MODE, KC, MAXK, TM>, bytes);                                                                   \
        if (e != cudaSuccess) return e;                                                                                                              \
        in_stream_order(sim_dparams<MODE, KC, MAXK, TM>, int(blocks), kDpThreads, folds ? bytes : 0, s)(g, f_N, f_ow, tile, x, t, dy, part, splits); \
    } while (0)
#define DP(MODE)                                            \
    do {                                                    \
        if (tile.tm == 64) DP_TILE(MODE, 32, 32, 64);       \
        else if (tile.kc == 64) DP_TILE(MODE, 64, 16, 32);  \
        else if (tile.k2 <= 16) DP_TILE(MODE, 32, 32, 32);  \
        else DP_TILE(MODE, 32, 64, 32);                     \
    } while (0)
#define DW_TILE(MODE, WJ)                                                                                                                   \
    do {                                                                                                                                    \
        using Tile = DwTile<MODE, WJ>;                                                                                                      \
        static SmemLimit limit;                                                                                                             \
        const cudaError_t e = limit.raise(sim_dparams_wide<MODE, WJ>, Tile::SMEM + Tile::SLOT_BYTES);                                       \
        if (e != cudaSuccess) return e;                                                                                                     \
        const long long each = ((long long)g.B * g.N + splits - 1) / splits;                                                                \
        const int fold = dw_fold(each);                                                                                                     \
        in_stream_order(sim_dparams_wide<MODE, WJ>, int(blocks), kDpThreads, Tile::SMEM + (each > (fold - 1) * kDwKC ? Tile::SLOT_BYTES : 0), s)(g, f_N, f_ow, wide, x, t, dy, part, splits, fold); \
    } while (0)
#define DW(MODE) do { if (wide <= 32) DW_TILE(MODE, 1); else DW_TILE(MODE, 2); } while (0)
    if (wide > 0) {
        switch (g.mode) {
        case SIM_L1: DW(SIM_L1); break;
        case SIM_L1_SKIP: DW(SIM_L1_SKIP); break;
        case SIM_L2: DW(SIM_L2); break;
        case SIM_L2N: DW(SIM_L2N); break;
        default: DW(SIM_L2N_NAN); break;
        }
    } else
    switch (g.mode) {
    case SIM_L1: DP(SIM_L1); break;
    case SIM_L1_SKIP: DP(SIM_L1_SKIP); break;
    case SIM_L2: DP(SIM_L2); break;
    case SIM_L2N: DP(SIM_L2N); break;
    default: DP(SIM_L2N_NAN); break;
    }
#undef DP
#undef DP_TILE
#undef DW
#undef DW_TILE
    const int mk = g.M * g.K, slices = splits >= 64 ? 64 : 8, lanes = 512 / slices;
    in_stream_order(sim_dparams_reduce, std::min((mk + lanes - 1) / lanes, device_sm_count() * 8), 512, 0, s)(g, splits, slices, part, w, dt, dw, accumulate);
    count_launch(2);
    return cudaGetLastError();
}

}  // namespace simnets
