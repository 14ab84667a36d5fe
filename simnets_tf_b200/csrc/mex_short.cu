// Gradients of MEX layers with short patches (K <= 32) under many instances, both from one read of y and dy (float32).
//
//     Q[m,j] = dy exp(eps (mx + mo - y) + c),    dx[tap k of j] = Ex[k,j] sum_m Eo[m,k] Q[m,j],    doff[m,k] = Eo[m,k] sum_j Q[m,j] Ex[k,j]
//
// Bound: HBM.  Such a layer has few taps per output, so y and dy are nearly all of its memory traffic (256 instances over
// 4x2x2 blocks of a 256 x 256 x 32 x 32 input: 4.3 GB each); two kernels that each read both, at 40 to 60 % of the copy rate
// because a tile was staged, multiplied and stored in turn, took 2.31 + 3.12 ms of it.
//
// A persistent CTA walks tiles of 64 positions of one region.  Per 64 instances: y and dy of the next 64 x 64 values are
// requested, Q of the current ones (requested a step earlier) goes to shared memory once, and the eight warps multiply it there
// both ways with tensor-core instructions of warp size (m16n8k8): four warps 16 instances each against Ex over the positions,
// four warps 16 positions each against Eo over the instances.  The products are slivers of K columns, which is why these are
// warp instructions: a tcgen05 tile would be 16 columns wide and its operand staging would cost more than the product.
// Operands are split into two TF32 parts, three products each, as everywhere in this library; Ex and Eo lie split in shared
// memory, Q is split once per row tile.  The values' own loads run one step ahead, as far as registers go, and leave the kernel waiting
// for memory (3.1 TB/s with the products switched off): their lines are prefetched into L2 three steps ahead, one line per thread and
// step (256 instances over 4x2x2 blocks, batch 256: 3833 -> 3554 us; two or six steps 3578, 3662, twelve 3969).  The offsets sums of the CTA live in shared memory, each value private to one thread; a
// CTA's partial sums are written once and added in a fixed order by the reduction.
#include <climits>
#include "mex_common.cuh"
#include "mma.cuh"

namespace simnets {
namespace {

constexpr int kShThreads = 256, kShPos = 64, kShM = 64, kShAhead = 3;

struct ShCol { long long sample; int c0, h0, w0, corner; };         // offset of the sample in x, patch corner; corner = its offset inside the sample

// row length, in (hi, lo) pairs, of the split operands: four rows x eight columns of one fragment read hit all banks
__host__ __device__ constexpr int sh_ld(int kt) { return kt + 4; }
__host__ __device__ inline int sh_smem_bytes(int M, int kt) {
    const int mp = (M + kShM - 1) / kShM * kShM;
    return 4 * (2 * kShM * kShPos + 2 * kShPos * sh_ld(kt) + 2 * mp * sh_ld(kt) + mp + mp * kt + 2 * kt) + kShPos * int(sizeof(ShCol));
}

// Q[m][pos] at m * 64 + (pos ^ sh_swizzle(m)): rows of four consecutive positions stay 16-byte vectors, and both fragment reads
// (8 rows x 4 positions, 4 rows x 8 positions) hit 32 different banks.
__device__ __forceinline__ int sh_swizzle(int m) { return ((m & 3) << 3) | (m & 4); }

__device__ __forceinline__ float sh_exp2(float v) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v)); return r; }

// A fragment of four Q values and NT fragments of a split operand: d[nt] += Q * operand, hi lo products first
template <int NT>
__device__ __forceinline__ void sh_step(float (&d)[NT][4], float q0, float q1, float q2, float q3, const float2* __restrict__ b, int row4) {
    uint32_t ah[4], al[4];
    const float q[4] = {q0, q1, q2, q3};
#pragma unroll
    for (int u = 0; u < 4; ++u) { const float2 s = split_tf32(q[u]); ah[u] = __float_as_uint(s.x); al[u] = __float_as_uint(s.y); }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const float2 b0 = b[nt * 8], b1 = b[row4 + nt * 8];
        mma_tf32(d[nt], al, __float_as_uint(b0.x), __float_as_uint(b1.x));
        mma_tf32(d[nt], ah, __float_as_uint(b0.y), __float_as_uint(b1.y));
        mma_tf32(d[nt], ah, __float_as_uint(b0.x), __float_as_uint(b1.x));
    }
}

// NT: taps / 8 (1, 2 or 4).  VEC: one region and rows of y and dy whose length is a multiple of four floats: four consecutive
// positions are one aligned vector of each.
template <int NT, bool DX, bool DOFF, bool VEC>
__global__ void __launch_bounds__(kShThreads, 2) mex_bwd_short(MexGeo g, int inside, const float* __restrict__ x, const float* __restrict__ eo,
                                                               const float* __restrict__ mo, const float* __restrict__ mx, const float* __restrict__ y,
                                                               const float* __restrict__ dy, float* __restrict__ dx, float* __restrict__ part,
                                                               int fold, const int* __restrict__ flag) {
    stream_order();
    if (*flag) return;
    constexpr int KT = NT * 8, LD = sh_ld(KT);
    extern __shared__ __align__(16) float sm[];
    const int MC = (g.M + kShM - 1) / kShM, MP = MC * kShM, r = blockIdx.y;
    float* Qs = sm;                                                     // [2][64 instances][64 positions], swizzled
    float2* E = reinterpret_cast<float2*>(Qs + 2 * kShM * kShPos);      // [64 positions][LD]
    float2* Eos = E + kShPos * LD;                                      // [MP][LD]
    float* Ds = reinterpret_cast<float*>(Eos + MP * LD);                // [MC][NT][128 threads][4]: the offsets sums
    float* mos = Ds + MP * KT;                                          // [MP]
    int* toff = reinterpret_cast<int*>(mos + MP);                       // [KT] offset of a tap from its patch corner
    int* tchw = toff + KT;                                              // [KT] (c << 16) | (h << 8) | w, for the bounds test
    ShCol* cols = reinterpret_cast<ShCol*>(tchw + KT);                  // [64]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
    const int Kp = pad4(g.K);
    for (int i = tid; i < MP * LD; i += kShThreads) {
        const int m = i / LD, k = i % LD;
        Eos[i] = split_tf32(m < g.M && k < g.K ? eo[((size_t)r * g.M + m) * Kp + k] : 0.f);
    }
    for (int m = tid; m < MP; m += kShThreads) mos[m] = m < g.M ? mo[r * g.M + m] : 0.f;
    if (DOFF) for (int i = tid; i < MP * KT; i += kShThreads) Ds[i] = 0.f;
    if (tid < KT) {
        const Tap t = tap_of<false>(g, tid < g.K ? tid : 0);
        toff[tid] = (t.c * g.H + t.h) * g.W + t.w;
        tchw[tid] = (t.c << 16) | (t.h << 8) | t.w;
    }
    __syncthreads();

    // this CTA's share of the region's positions: whole runs of 32
    const long long runs = ((long long)g.B * g.rs + 31) / 32;
    const long long p_begin = runs * blockIdx.x / gridDim.x * 32, P = min((long long)g.B * g.rs, runs * (blockIdx.x + 1) / gridDim.x * 32);
    const float eps = float(g.eps), oob = float(g.oob), a2 = eps * 1.4426950408889634f, c2 = float(g.cst) * 1.4426950408889634f;
    constexpr int ROWS = VEC ? 16 : 4, PER = kShM / ROWS, W = VEC ? 4 : 1;      // staging: W positions, instances row0, row0 + ROWS, ...
    const int pos = VEC ? (tid & 15) * 4 : tid & (kShPos - 1), row0 = VEC ? tid >> 4 : tid >> 6;
    const int e_pos = tid & (kShPos - 1), e_row = tid >> 6;                     // Ex: one position, taps e_row, e_row + 4, ...
    float ry[PER][W], rg[PER][W], rmx[W], rx[KT / 4];
    Column col = {}, e_col = {};
    long long tile = p_begin;
    auto fetch = [&](int mc) {
        const bool live = col.base >= 0;
        const float* py = y + (live ? col.base : 0) + (long long)(mc * kShM + row0) * g.N;
        const float* pg = dy + (live ? col.gbase : 0) + (long long)(mc * kShM + row0) * g.Ng;
#pragma unroll
        for (int i = 0; i < PER; ++i, py += (long long)ROWS * g.N, pg += (long long)ROWS * g.Ng) {
            const bool ok = live && mc * kShM + row0 + ROWS * i < g.M;
            if (VEC) {
                const float4 a = ok ? __ldcs(reinterpret_cast<const float4*>(py)) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 b = ok ? __ldcs(reinterpret_cast<const float4*>(pg)) : make_float4(0.f, 0.f, 0.f, 0.f);
                ry[i][0] = a.x; ry[i][W > 1 ? 1 : 0] = a.y; ry[i][W > 2 ? 2 : 0] = a.z; ry[i][W > 3 ? 3 : 0] = a.w;
                rg[i][0] = b.x; rg[i][W > 1 ? 1 : 0] = b.y; rg[i][W > 2 ? 2 : 0] = b.z; rg[i][W > 3 ? 3 : 0] = b.w;
            } else {
                ry[i][0] = ok ? __ldcs(py) : 0.f;
                rg[i][0] = ok ? __ldcs(pg) : 0.f;
            }
        }
    };
    auto open_tile = [&](long long t) {                                         // positions, their maxima and their patches
        col = column_of(g, r, t + pos, P, mx);
#pragma unroll
        for (int u = 0; u < W; ++u) rmx[u] = col.mx;                            // (a dead quad: zeros, so that 0 * 2^... stays 0)
        if (VEC) {
            e_col = column_of(g, r, t + e_pos, P, mx);
            if (col.base >= 0) {
                const float4 m4 = *reinterpret_cast<const float4*>(mx + col.base - (long long)col.n * (g.M - 1) * g.N);
                rmx[0] = m4.x; rmx[W > 1 ? 1 : 0] = m4.y; rmx[W > 2 ? 2 : 0] = m4.z; rmx[W > 3 ? 3 : 0] = m4.w;
            }
        } else e_col = col;
        const float* xs = x + (long long)e_col.n * g.C * g.H * g.W;
        const int corner = (e_col.c0 * g.H + e_col.h0) * g.W + e_col.w0;
#pragma unroll
        for (int i = 0; i < KT / 4; ++i) {
            const int k = e_row + 4 * i;
            rx[i] = oob;
            if (e_col.base >= 0 && k < g.K) {
                const int t = tchw[k], cc = e_col.c0 + (t >> 16), hh = e_col.h0 + ((t >> 8) & 255), ww = e_col.w0 + (t & 255);
                if (inside || (cc >= 0 && cc < g.C && hh >= 0 && hh < g.H && ww >= 0 && ww < g.W)) rx[i] = __ldg(xs + corner + toff[k]);
            }
        }
        fetch(0);
    };
    // the L2 lines of a later step: one per thread, 64 rows x 2 lines of y and of dy (positions and instances that exist only)
    const float* const pf_of = (tid >> 7 ? dy : y);
    const int pf_row = (tid >> 1) & (kShM - 1), pf_half = (tid & 1) * 32;
    long long pf_tile = p_begin, pf_base = -1;
    int pf_mc = 0;
    auto pf_place = [&]() {
        const Column c = column_of(g, r, pf_tile + pf_half, P, nullptr);
        pf_base = c.base;
    };
    auto prefetch = [&]() {
        if (!VEC) return;
        if (pf_base >= 0 && pf_mc * kShM + pf_row < g.M) asm volatile("prefetch.global.L2 [%0];" ::"l"(pf_of + pf_base + (long long)(pf_mc * kShM + pf_row) * g.N));
        if (++pf_mc == MC) { pf_mc = 0; pf_tile += kShPos; pf_place(); }
    };
    if (VEC) { pf_place(); for (int i = 0; i < kShAhead; ++i) prefetch(); }
    // who multiplies what: both products, four warps each; one product alone, two warps per row tile
    const int rt = warp & 3;
    const bool does_dx = DX && (!DOFF || warp < 4);
    constexpr int MT = DX && DOFF ? NT : (NT + 1) / 2;                          // column tiles per warp
    const int nt0 = DX && DOFF ? 0 : (warp >> 2) * MT;
    const bool idle = nt0 >= NT;
    if (tile < P) open_tile(tile);
    int qb = 0;
    float acc[MT][4];                                                           // input gradient: 16 positions x 8 taps
    for (; tile < P; tile += kShPos) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[i][u] = 0.f;
        __syncthreads();                                                        // the last tile's Ex and positions are no longer needed
#pragma unroll
        for (int i = 0; i < KT / 4; ++i) {
            const int k = e_row + 4 * i;
            E[e_pos * LD + k] = split_tf32(e_col.base >= 0 && k < g.K ? fast_exp(eps * (rx[i] - e_col.mx)) : 0.f);
        }
        if (tid < kShPos)
            cols[tid] = ShCol{(long long)e_col.n * g.C * g.H * g.W, e_col.c0, e_col.h0, e_col.w0, e_col.base >= 0 ? (e_col.c0 * g.H + e_col.h0) * g.W + e_col.w0 : INT_MIN};
        for (int mc = 0; mc < MC; ++mc, qb ^= 1) {
            float* Q = Qs + qb * kShM * kShPos;
            prefetch();
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int m = row0 + ROWS * i;
                const float mom = mos[mc * kShM + m];
                float q[W];
#pragma unroll
                for (int u = 0; u < W; ++u) q[u] = rg[i][u] * sh_exp2(fmaf(a2, rmx[u] + mom - ry[i][u], c2));       // (dy = 0 for dead rows and positions)
                float* dst = Q + m * kShPos + (pos ^ sh_swizzle(m));
                if (VEC) *reinterpret_cast<float4*>(dst) = make_float4(q[0], q[W > 1 ? 1 : 0], q[W > 2 ? 2 : 0], q[W > 3 ? 3 : 0]);
                else *dst = q[0];
            }
            // request the next values before this step's products
            if (mc + 1 < MC) fetch(mc + 1);
            else if (tile + kShPos < P) open_tile(tile + kShPos);
            __syncthreads();
            if (idle) continue;
            if (does_dx) {
                // rows = positions 16 rt.., columns = taps, reduction = instances
                const int p0 = (rt * 16 + gq) ^ (tq << 3);
                const float* q0 = Q + tq * kShPos;
                const float2* b = Eos + (mc * kShM + tq) * LD + nt0 * 8 + gq;
                float s[MT][4];                                                 // (64 instances on the tensor cores, these sums in FP32)
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int u = 0; u < 4; ++u) s[i][u] = 0.f;
#pragma unroll
                for (int m = 0; m < kShM; m += 8) {
                    const float *lo = q0 + m * kShPos, *hi = lo + 4 * kShPos;
                    sh_step<MT>(s, lo[p0], lo[p0 ^ 8], hi[p0 ^ 4], hi[p0 ^ 12], b + m * LD, 4 * LD);
                }
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[i][u] += s[i][u];
            } else if (DOFF) {
                // rows = instances 16 rt.., columns = taps, reduction = positions
                float4* own = reinterpret_cast<float4*>(Ds) + (mc * NT + nt0) * 128 + (warp & 3) * 32 + lane;
                float s[MT][4];
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    const float4 v = fold ? make_float4(0.f, 0.f, 0.f, 0.f) : own[i * 128];
                    s[i][0] = v.x; s[i][1] = v.y; s[i][2] = v.z; s[i][3] = v.w;
                }
                const float* q0 = Q + (rt * 16 + gq) * kShPos;
                const int sw = sh_swizzle(gq);
                const float2* b = E + tq * LD + nt0 * 8 + gq;
#pragma unroll
                for (int p = 0; p < kShPos; p += 8) {
                    const int c0 = (p + tq) ^ sw, c1 = c0 ^ 4;
                    sh_step<MT>(s, q0[c0], q0[8 * kShPos + c0], q0[c1], q0[8 * kShPos + c1], b + p * LD, 4 * LD);
                }
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    const float4 v = fold ? own[i * 128] : make_float4(0.f, 0.f, 0.f, 0.f);
                    own[i * 128] = make_float4(v.x + s[i][0], v.y + s[i][1], v.z + s[i][2], v.w + s[i][3]);
                }
            }
        }
        if (does_dx && !idle) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int p = rt * 16 + gq + 8 * half;
                const ShCol cl = cols[p];
                if (cl.corner == INT_MIN) continue;
                float* out = dx + cl.sample + cl.corner;
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int k = (nt0 + i) * 8 + 2 * tq + u;
                        if (k >= g.K) continue;
                        const int t = tchw[k], cc = cl.c0 + (t >> 16), hh = cl.h0 + ((t >> 8) & 255), ww = cl.w0 + (t & 255);
                        const float2 e = E[p * LD + k];
                        if (inside || (cc >= 0 && cc < g.C && hh >= 0 && hh < g.H && ww >= 0 && ww < g.W)) out[toff[k]] = (e.x + e.y) * acc[i][half * 2 + u];
                    }
            }
        }
    }
    if (DOFF && !does_dx && !idle) {
        float* dst = part + ((size_t)blockIdx.x * g.R + r) * g.M * g.K;
        for (int mc = 0; mc < MC; ++mc)
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const float4 v = reinterpret_cast<const float4*>(Ds)[(mc * NT + nt0 + i) * 128 + (warp & 3) * 32 + lane];
                const float s[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int m = mc * kShM + rt * 16 + gq + 8 * (u >> 1), k = (nt0 + i) * 8 + 2 * tq + (u & 1);
                    if (m < g.M && k < g.K) dst[(size_t)m * g.K + k] = s[u];
                }
            }
    }
}

int sh_taps(const MexGeo& g) { return g.K <= 8 ? 8 : (g.K <= 16 ? 16 : 32); }
int sh_ctas_per_sm(const MexGeo& g) { return sh_smem_bytes(g.M, sh_taps(g)) <= 112 * 1024 ? 2 : 1; }

}  // namespace

// Short patches under at least 32 instances whose blocks do not overlap, with room for the parameters in shared memory.
bool mex_short_shape(const MexGeo& g) {
    return g.K <= 32 && g.M >= 32 && g.sc >= g.bc && g.sh >= g.bh && g.sw >= g.bw && g.bh <= 256 && g.bw <= 256 && g.R <= 65535 &&
           (long long)g.C * g.H * g.W < (1LL << 31) && sh_smem_bytes(g.M, sh_taps(g)) <= 220 * 1024;
}
// Positions that the one-tile kernels of mex_tc.cu sum in one accumulator.  The tensor cores truncate what they add, so a long
// sum depends on where it is cut (18.9 K positions: 1.4e-4 of the offsets gradient's norm from the exact sum, growing with the
// length): from 1500 positions on (1e-5) this kernel cuts where that one does and accumulates as that one does; below it takes
// shares that fill the GPU and adds the products of 64 positions in FP32 (64 instances over 2x2x2 blocks, 885 positions a share:
// 6.4e-6 of the norm otherwise, the one-tile kernel 4.5e-6; 7.4e-7 so).
static bool sh_long_sums(const MexGeo& g) { return (long long)g.B * g.rs / mex_tc_doff_splits(g) > 1500; }
int mex_short_splits(const MexGeo& g) {
    if (sh_long_sums(g)) return mex_tc_doff_splits(g);
    const long long runs = ((long long)g.B * g.rs + 31) / 32, tiles = (runs + 1) / 2;
    const long long ctas = std::max<long long>(1, (long long)device_sm_count() * sh_ctas_per_sm(g) / g.R);
    const long long each = (tiles + ctas - 1) / ctas;
    return int(std::max<long long>(1, (tiles + each - 1) / each));
}
// Whether the offsets gradient of this layer is worth it: with one CTA per SM the shares of long sums leave SMs idle (200
// instances over 8x2x2 blocks, 0.5 M positions: both gradients 827 us, 755 in two kernels).
bool mex_short_doff(const MexGeo& g) { return !sh_long_sums(g) || sh_ctas_per_sm(g) == 2; }

cudaError_t launch_mex_bwd_short(const MexGeo& g, bool inside, const float* x, const float* eo, const float* mo, const float* mx, const float* y,
                                 const float* dy, float* dx, float* part, const int* flag, cudaStream_t s) {
    const int kt = sh_taps(g), smem = sh_smem_bytes(g.M, kt);
    const int fold = !sh_long_sums(g);
    const dim3 grid(unsigned(mex_short_splits(g)), unsigned(g.R));
    const bool vec = g.R == 1 && g.gp == 1 && g.N % 4 == 0 && ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(dy)) & 15) == 0;
#define SH(NT, DX, DOFF, VEC)                                                                                                                     \
    do {                                                                                                                                          \
        const cudaError_t e = cudaFuncSetAttribute(mex_bwd_short<NT, DX, DOFF, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);    \
        if (e != cudaSuccess) return e;                                                                                                           \
        in_stream_order(mex_bwd_short<NT, DX, DOFF, VEC>, grid, kShThreads, smem, s)(g, int(inside), x, eo, mo, mx, y, dy, dx, part, fold, flag); \
    } while (0)
#define SH_VEC(NT, DX, DOFF) do { if (vec) SH(NT, DX, DOFF, true); else SH(NT, DX, DOFF, false); } while (0)
#define SH_WANTS(NT)                                                                                     \
    do {                                                                                                 \
        if (dx != nullptr && part != nullptr) SH_VEC(NT, true, true);                                    \
        else if (dx != nullptr) SH_VEC(NT, true, false);                                                 \
        else SH_VEC(NT, false, true);                                                                    \
    } while (0)
    if (kt == 8) SH_WANTS(1); else if (kt == 16) SH_WANTS(2); else SH_WANTS(4);
#undef SH_WANTS
#undef SH_VEC
#undef SH
    count_launch();
    return cudaGetLastError();
}

}  // namespace simnets
