// Sequence-parallel form of the gated linear recurrence for prompt portions:
//     St <- diag(a_t) St + k_t (sc_t u_t)^T ,  y_t = St^T (cs c_t) + skip * u_t          (St: N x P per head, fp32)
// The rows of a call are cut into blocks of CL = 64 tokens (counted from row 0 of the call; the carried state enters
// block 0). With b_t = sum of log a over the rows of the block up to and including t:
//     y_t   = sum_n cs c_t[n] exp(b_t[n]) S_in[n, :]  +  sum_{s <= t} M[t, s] u_s  + skip u_t
//     M[t,s]= cs sc_s sum_n c_t[n] k_s[n] exp(b_t[n] - b_s[n])                       (every exponent is <= 0)
//     S_out = diag(exp(b_last)) S_in + sum_s (k_s * exp(b_last - b_s)) (sc_s u_s)^T
// Five launches: block-local cumulative log decays, M, the blocks' own state contributions, a short sequential pass
// over blocks that turns them into the state entering each block, and the outputs. All arithmetic is fp32 (the recurrence's operands are
// fp32 by the models' precision rules); the three products are 64 x 64 tiles whose operands are formed (decay factors applied) while
// they are staged: on the CUDA cores, or, over aligned bf16 rows, on the tensor cores by values cut in three (all three for a decay per head,
// the blocks' own states for a decay per key channel, whose outputs have two fp32 operands).
#include <type_traits>
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "mma.cuh"
#include "launch.h"
#include "seqmix.h"

namespace lcc {
namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16* p) { return __bfloat162float(*p); }

__device__ __forceinline__ bool seq_done(const SeqPos& p) { return p.finished && *p.finished; }

constexpr int CL = 64;          // tokens per block
constexpr int TS = 64;          // output tile edge
constexpr int KS = 16;          // depth of a staged operand slice
constexpr int PAD = TS + 4;

struct Tile {
    float a[KS][PAD];
    float b[KS][PAD];
};

// Stage one KS-deep slice of both operands: fa(r, kk) / fb(r, kk) give element (tile row or column r, depth kk) or 0
// outside the problem. KC: consecutive threads walk the depth index (operands contiguous along it), else the row index.
template <bool KC_A, bool KC_B, typename FA, typename FB>
__device__ __forceinline__ void stage(Tile& sh, FA fa, FB fb) {
#pragma unroll
    for (int i = 0; i < TS * KS / 256; ++i) {
        const int e = threadIdx.x + i * 256;
        { const int r = KC_A ? e / KS : e % TS, kk = KC_A ? e % KS : e / TS; sh.a[kk][r] = fa(r, kk); }
        { const int r = KC_B ? e / KS : e % TS, kk = KC_B ? e % KS : e / TS; sh.b[kk][r] = fb(r, kk); }
    }
}

__device__ __forceinline__ void fma_slice(const Tile& sh, int tm, int tn, float (&acc)[4][4]) {
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
        const float4 av = *reinterpret_cast<const float4*>(&sh.a[kk][tm]);
        const float4 bv = *reinterpret_cast<const float4*>(&sh.b[kk][tn]);
        const float a[4] = {av.x, av.y, av.z, av.w}, b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
}

struct ChunkArgs {
    const void* k; int ld_k;
    const void* c; int ld_c;
    const void* u; int ld_u;
    float* la;                 // [S, heads * NV] log decays, replaced by their block-local cumulative sums
    const float* sc;           // [S, heads] or null
    const float* skip;         // [heads] or null
    float cs;
    float* state;              // [heads, P, N]
    float* y; int ld_y;
    float* ws_m;               // [blocks, heads, CL, CL]
    float* ws_s;               // [blocks, heads, P, N]
    int row0;                  // first row of this pass
    int S;                     // rows of this pass
    int heads, heads_per_group, N, P, NV;   // NV = N (a decay per key channel) or 1 (a decay per head)
};

// ---- 1: block-local cumulative sums of the log decays ---------------------------------------------------------------
__global__ void chunk_cumsum_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    const int col = blockIdx.y * blockDim.x + threadIdx.x, ncol = a.heads * a.NV;
    if (col >= ncol) return;
    const int t0 = blockIdx.x * CL, len = min(CL, a.S - t0);
    float* p = a.la + (size_t)(a.row0 + t0) * ncol + col;
    float acc = 0.f;
    for (int tb = 0; tb < len; tb += 16) {     // 16 independent loads in flight, then the running sum in row order
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = tb + i < len ? p[(size_t)(tb + i) * ncol] : 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            acc += v[i];
            if (tb + i < len) p[(size_t)(tb + i) * ncol] = acc;
        }
    }
}

// ---- 2: M[t, s] -------------------------------------------------------------------------------------------------------
// A decay per head: the product c k^T is the same for every head of a group, so a CTA forms it once per group and writes one decayed copy per head.
template <typename T>
__global__ void __launch_bounds__(256) chunk_weights_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ float sc_[KS][PAD], sk_[KS][PAD];
    const int blk = blockIdx.x, g = blockIdx.y;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int N = a.N, ncol = a.heads;
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16, tm = ty * 4, tn = tx * 4;
    const T* gc = (const T*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * N;
    const T* gk = (const T*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * N;
    const bool live = tn <= tm + 3;            // tiles wholly above the diagonal stay zero
    float acc[4][4] = {};
    for (int n0 = 0; n0 < N; n0 += KS) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < CL * KS / 256; ++i) {
            const int e = threadIdx.x + i * 256, r = e / KS, kk = e % KS, n = n0 + kk;
            const bool ok = r < len && n < N;
            sc_[kk][r] = ok ? ldf(gc + (size_t)r * a.ld_c + n) : 0.f;
            sk_[kk][r] = ok ? ldf(gk + (size_t)r * a.ld_k + n) : 0.f;
        }
        __syncthreads();
        if (!live) continue;
#pragma unroll 4
        for (int kk = 0; kk < KS; ++kk) {
            float cv[4], kv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { cv[i] = sc_[kk][tm + i]; kv[i] = sk_[kk][tn + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(cv[i], kv[j], acc[i][j]);
        }
    }
    for (int hh = g * a.heads_per_group; hh < (g + 1) * a.heads_per_group; ++hh) {
        float* out = a.ws_m + ((size_t)blk * a.heads + hh) * CL * CL;
        const float* hb = a.la + (size_t)(a.row0 + t0) * ncol + hh;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = tm + i;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int s = tn + j;
                float v = 0.f;
                if (s <= t && t < len) {
                    v = acc[i][j] * a.cs * (a.sc ? a.sc[(size_t)(a.row0 + t0 + s) * a.heads + hh] : 1.f);
                    v *= expf(fminf(hb[(size_t)t * ncol] - hb[(size_t)s * ncol], 0.f));
                }
                out[t * CL + s] = v;
            }
        }
    }
}

// A decay per key channel, a CTA per head and block. An exponential per (t, s, n) costs 2080 a channel (145 us for 2048 rows, 8 heads, 128 channels, bound by
// their instructions; warps on the diagonal ran the half above it too). But exp(b_t - b_s) = exp(b_t - b_m) exp(b_m - b_s) for any m between s and t, and neither
// exponent is positive: halves of 64, 32, 16 and 8 rows meet in plain products of rows decayed to the first row of the upper half (64 exponentials per level and
// channel, 1920 of the 2080 weights), and only the tiles of 4 rows on the diagonal keep one per weight (160). Where a factor leaves fp32's normal range the weight
// is below 2^-126 of its c k. Each 128 threads take a quarter of a slab's 16 channels, and the four sums are added at the end. 26 us (41 with 256 threads and
// diagonal tiles of 8 rows, 28 with the latter): latency of a slab's loads, exponentials and products behind three barriers.
template <typename T>
__global__ void __launch_bounds__(512, 2) chunk_weights_vec_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    constexpr int LEVELS = 4;
    __shared__ __align__(16) float sh[3 + LEVELS][KS][PAD];   // c, k, cumulative decays; rows decayed per level (upper half: c, lower: k). At the end: the weights
    auto& sc_ = sh[0]; auto& sk_ = sh[1]; auto& sb_ = sh[2];
    const int blk = blockIdx.x, h = blockIdx.y, g = h / a.heads_per_group;
    const int t0 = blk * CL, len = min(CL, a.S - t0), N = a.N, ncol = a.heads * N;
    const T* gc = (const T*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * N;
    const T* gk = (const T*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * N;
    const float* gb = a.la + (size_t)(a.row0 + t0) * ncol + (size_t)h * N;
    const int part = threadIdx.x >> 7, q = (threadIdx.x ^ (part & 1 ? 127 : 0)) & 127;   // (mirrored, so that no scheduler has all the diagonals)
    int lv = 0, tm = 0, tn = 0;                               // a thread's 4 x 4 weights below the diagonal tiles (120 of 128 threads)
    if (q < 64) { lv = 0; tm = 32 + (q >> 3) * 4; tn = (q & 7) * 4; }
    else if (q < 96) { lv = 1; tm = ((q >> 4) & 1) * 32 + 16 + ((q >> 2) & 3) * 4; tn = ((q >> 4) & 1) * 32 + (q & 3) * 4; }
    else if (q < 112) { lv = 2; tm = ((q >> 2) & 3) * 16 + 8 + ((q >> 1) & 1) * 4; tn = ((q >> 2) & 3) * 16 + (q & 1) * 4; }
    else if (q < 120) { lv = 3; tm = (q & 7) * 8 + 4; tn = (q & 7) * 8; }
    const int dq = (127 - q) / 3, dr = (127 - q) % 3, dt = q >= 80 ? dq * 4 + (dr ? 2 : 0) : 0, ds = q >= 80 ? dq * 4 + (dr == 2 ? 2 : 0) : CL;   // (CL: none)   // and its 2 x 2 on the diagonal
    float2 acc[2][4] = {};                                    // rows (2 i, 2 i + 1) x column j
    float diag[2][2] = {};
    float pc[2], pk[2], pb[2];
    auto fetch = [&](int n0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int e = threadIdx.x + i * 512, r = e / KS, n = n0 + e % KS;
            const bool ok = r < len && n < N;
            pc[i] = ok ? ldf(gc + (size_t)r * a.ld_c + n) : 0.f;
            pk[i] = ok ? ldf(gk + (size_t)r * a.ld_k + n) : 0.f;
            pb[i] = ok ? gb[(size_t)r * ncol + n] : 0.f;
        }
    };
    fetch(0);
    for (int n0 = 0; n0 < N; n0 += KS) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int e = threadIdx.x + i * 512, r = e / KS, kk = e % KS;
            sc_[kk][r] = pc[i]; sk_[kk][r] = pk[i]; sb_[kk][r] = pb[i];
        }
        __syncthreads();
        if (n0 + KS < N) fetch(n0 + KS);
#pragma unroll
        for (int l = 0; l < LEVELS; ++l) {
            const int L = 32 >> l, r = threadIdx.x & 63, m = (r & ~(2 * L - 1)) + L;
            const bool up = r & L;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int kk = (threadIdx.x >> 6) + i * 8;
                const float d = sb_[kk][r] - sb_[kk][m];
                sh[3 + l][kk][r] = (up ? sc_[kk][r] : sk_[kk][r]) * expf(fminf(up ? d : -d, 0.f));
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int i8 = 0; i8 < KS / 4; ++i8) {
            const int kk = part * (KS / 4) + i8;
            if (q < 120) {
                const float4 x = *reinterpret_cast<const float4*>(&sh[3 + lv][kk][tm]), y = *reinterpret_cast<const float4*>(&sh[3 + lv][kk][tn]);
                const float yj[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[0][j] = __ffma2_rn(make_float2(x.x, x.y), make_float2(yj[j], yj[j]), acc[0][j]);
                    acc[1][j] = __ffma2_rn(make_float2(x.z, x.w), make_float2(yj[j], yj[j]), acc[1][j]);
                }
            }
            if (ds <= dt) {
                const float2 c2 = *reinterpret_cast<const float2*>(&sc_[kk][dt]), bt = *reinterpret_cast<const float2*>(&sb_[kk][dt]);
                const float2 k2 = *reinterpret_cast<const float2*>(&sk_[kk][ds]), bs = *reinterpret_cast<const float2*>(&sb_[kk][ds]);
                diag[0][0] = fmaf(c2.x * k2.x, expf(fminf(bt.x - bs.x, 0.f)), diag[0][0]);
                diag[0][1] = fmaf(c2.x * k2.y, expf(fminf(bt.x - bs.y, 0.f)), diag[0][1]);
                diag[1][0] = fmaf(c2.y * k2.x, expf(fminf(bt.y - bs.x, 0.f)), diag[1][0]);
                diag[1][1] = fmaf(c2.y * k2.y, expf(fminf(bt.y - bs.y, 0.f)), diag[1][1]);
            }
        }
    }
    float (*w)[PAD] = reinterpret_cast<float (*)[PAD]>(&sh[0][0][0]);   // [t][s], what lies above the diagonal is not read
    static_assert((3 + LEVELS) * KS >= CL, "the weights fit");
    auto each = [&](auto put) {
        if (q < 120)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) put(w[tm + i][tn + j], (i & 1) ? acc[i >> 1][j].y : acc[i >> 1][j].x);
        if (ds <= dt)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) put(w[dt + i][ds + j], diag[i][j]);
    };
    __syncthreads();
    for (int p = 0; p < 4; ++p) {
        if (part == p) each([p](float& x, float v) { x = p ? x + v : v; });
        __syncthreads();
    }
    float* out = a.ws_m + ((size_t)blk * a.heads + h) * CL * CL;
    const float* gsc = a.sc ? a.sc + (size_t)(a.row0 + t0) * a.heads + h : nullptr;
    for (int e = threadIdx.x; e < CL * CL; e += 512) {
        const int t = e / CL, s = e % CL;
        out[e] = s <= t && t < len ? w[t][s] * a.cs * (gsc ? gsc[(size_t)s * a.heads] : 1.f) : 0.f;
    }
}

// ---- 3: a block's own contribution to the state, stored [p][n] ----------------------------------------------------------
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) chunk_state_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ Tile sh;
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int p0 = blockIdx.y * TS, n0 = blockIdx.z * TS;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int N = a.N, P = a.P, ncol = a.heads * a.NV;
    const T* gu = (const T*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * P;
    const T* gk = (const T*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * N;
    const float* gb = a.la + (size_t)(a.row0 + t0) * ncol + (size_t)h * a.NV;
    const float* gsc = a.sc ? a.sc + (size_t)(a.row0 + t0) * a.heads + h : nullptr;
    const float* blast = gb + (size_t)(len - 1) * ncol;
    const int tm = (threadIdx.x / 16) * 4, tn = (threadIdx.x % 16) * 4;
    __shared__ float rowf[CL];     // per row: the step scale, and in the per-head case the decay from the row to the block's end
    if (threadIdx.x < CL) {
        const int s = threadIdx.x;
        float f = 0.f;
        if (s < len) {
            f = gsc ? gsc[(size_t)s * a.heads] : 1.f;
            if (!VEC) f *= expf(fminf(blast[0] - gb[(size_t)s * ncol], 0.f));
        }
        rowf[s] = f;
    }
    float acc[4][4] = {};
    for (int s0 = 0; s0 < len; s0 += KS) {
        __syncthreads();
        stage<false, false>(sh,
            [&](int r, int kk) { const int s = s0 + kk, p = p0 + r;
                                 return (s < len && p < P) ? ldf(gu + (size_t)s * a.ld_u + p) * rowf[s] : 0.f; },
            [&](int r, int kk) { const int s = s0 + kk, n = n0 + r;
                                 if (s >= len || n >= N) return 0.f;
                                 const float kv = ldf(gk + (size_t)s * a.ld_k + n);
                                 return VEC ? kv * expf(fminf(blast[n] - gb[(size_t)s * ncol + n], 0.f)) : kv; });
        __syncthreads();
        fma_slice(sh, tm, tn, acc);
    }
    float* out = a.ws_s + ((size_t)blk * a.heads + h) * P * N;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int p = p0 + tm + i;
        if (p >= P) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tn + j;
            if (n < N) out[(size_t)p * N + n] = acc[i][j];
        }
    }
}

// ---- 4: contributions -> the state that enters each block; the state after the last block goes back to the slot -----
template <bool VEC>
__global__ void chunk_prefix_kernel(ChunkArgs a, int nblocks, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    const size_t per = (size_t)a.heads * a.P * a.N;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= per) return;
    const int n = (int)(idx % a.N), h = (int)(idx / ((size_t)a.P * a.N));
    const int ncol = a.heads * a.NV;
    float st = a.state[idx];
    for (int b0 = 0; b0 < nblocks; b0 += 8) {  // 8 blocks' loads in flight together; the chain over blocks runs in registers
        float d[8], e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int b = b0 + i;
            if (b < nblocks) {
                const int tlast = min((b + 1) * CL, a.S) - 1;
                d[i] = a.ws_s[(size_t)b * per + idx];
                e[i] = a.la[(size_t)(a.row0 + tlast) * ncol + (size_t)h * a.NV + (VEC ? n : 0)];
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int b = b0 + i;
            if (b < nblocks) {
                a.ws_s[(size_t)b * per + idx] = st;
                st = fmaf(expf(e[i]), st, d[i]);
            }
        }
    }
    a.state[idx] = st;
}

// ---- 5: outputs ---------------------------------------------------------------------------------------------------------
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) chunk_output_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ Tile sh;
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int p0 = blockIdx.y * TS;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int N = a.N, P = a.P, ncol = a.heads * a.NV;
    const T* gu = (const T*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * P;
    const T* gc = (const T*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * N;
    const float* gb = a.la + (size_t)(a.row0 + t0) * ncol + (size_t)h * a.NV;
    const float* sin = a.ws_s + ((size_t)blk * a.heads + h) * P * N;
    const float* gm = a.ws_m + ((size_t)blk * a.heads + h) * CL * CL;
    const int tm = (threadIdx.x / 16) * 4, tn = (threadIdx.x % 16) * 4;
    float acc[4][4] = {};
    for (int n0 = 0; n0 < N; n0 += KS) {       // the entering state, seen through the decayed queries
        __syncthreads();
        stage<true, true>(sh,
            [&](int r, int kk) { const int n = n0 + kk;
                                 if (r >= len || n >= N) return 0.f;
                                 return a.cs * ldf(gc + (size_t)r * a.ld_c + n) * expf(gb[(size_t)r * ncol + (VEC ? n : 0)]); },
            [&](int r, int kk) { const int n = n0 + kk, p = p0 + r;
                                 return (n < N && p < P) ? sin[(size_t)p * N + n] : 0.f; });
        __syncthreads();
        fma_slice(sh, tm, tn, acc);
    }
    for (int s0 = 0; s0 < len; s0 += KS) {     // the block's own rows
        __syncthreads();
        stage<true, false>(sh,
            [&](int r, int kk) { const int s = s0 + kk; return s < len ? gm[r * CL + s] : 0.f; },
            [&](int r, int kk) { const int s = s0 + kk, p = p0 + r;
                                 return (s < len && p < P) ? ldf(gu + (size_t)s * a.ld_u + p) : 0.f; });
        __syncthreads();
        fma_slice(sh, tm, tn, acc);
    }
    const float skip = a.skip ? a.skip[h] : 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = tm + i;
        if (t >= len) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = p0 + tn + j;
            if (p < P) a.y[(size_t)(a.row0 + t0 + t) * a.ld_y + (size_t)h * P + p] = acc[i][j] + skip * ldf(gu + (size_t)t * a.ld_u + p);
        }
    }
}

// ---- the same three products for a decay per head and 16-byte aligned rows ----------------------------------------------
// The forms above stage 16-deep slices element by element, an exponential per staged element, and a decayed copy of c k^T per head
// (2048 rows, 64 heads of 64 x 128: 54 + 92 + 157 us). Here a CTA of 128 threads stages 64-deep slabs with 16-byte loads and an 8 x 4 tile
// per thread multiplies them in packed fp32 pairs (fma.rn.f32x2: each half rounds as a scalar fma does); c k^T is left undecayed once
// per group of heads, and the decays enter where a head's output tile is staged: 15 + 59 + 112 us, bound by
// fp32 multiplies (2.1 and 3.2 GFLOP) and the shared-memory reads that feed them. The prefix over blocks: 30 -> 25 us.
constexpr int SP = 64 + 4;      // pitch of a slab row
struct Slab {
    float a[64][SP], b[64][SP]; // [depth][tile row], [depth][tile column]
};
struct Acc84 {
    float2 v[4][4];             // rows (2 i, 2 i + 1) x column j
};
__device__ __forceinline__ void slab_fma(const Slab& sh, int depth, int tm, int tn, Acc84& acc) {
#pragma unroll 8
    for (int k = 0; k < depth; ++k) {
        const float4 a0 = *reinterpret_cast<const float4*>(&sh.a[k][tm]), a1 = *reinterpret_cast<const float4*>(&sh.a[k][tm + 4]);
        const float4 b4 = *reinterpret_cast<const float4*>(&sh.b[k][tn]);
        const float2 ar[4] = {make_float2(a0.x, a0.y), make_float2(a0.z, a0.w), make_float2(a1.x, a1.y), make_float2(a1.z, a1.w)};
        const float bj[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 bb = make_float2(bj[j], bj[j]);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc.v[i][j] = __ffma2_rn(ar[i], bb, acc.v[i][j]);
        }
    }
}
// 16 bytes of a row -> floats
template <typename T> struct Row16;
template <> struct Row16<bf16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const bf16* p, float (&v)[8]) {
        const uint4 u = *reinterpret_cast<const uint4*>(p);
        const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
    }
};
template <> struct Row16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
        const float4 u = *reinterpret_cast<const float4*>(p);
        v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
    }
};
__device__ __forceinline__ void ld4f(const float* p, float* v) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
// dst[k][r] = src[r][k0 + k] * f(r) for 64 tile rows (zero from `rows` on) and k < 64 (zero from `cols` on): rows contiguous along k
template <typename T, typename F>
__device__ __forceinline__ void slab_across(float (*dst)[SP], const T* src, int ld, int rows, int k0, int cols, F f) {
    constexpr int V = Row16<T>::N;
    for (int e = threadIdx.x; e < 64 * (64 / V); e += 128) {
        const int r = e & 63, k = (e >> 6) * V;
        float v[V] = {};
        if (r < rows && k0 + k < cols) {
            Row16<T>::load(src + (size_t)r * ld + k0 + k, v);
            const float m = f(r);
#pragma unroll
            for (int i = 0; i < V; ++i) v[i] *= m;
        }
#pragma unroll
        for (int i = 0; i < V; ++i) dst[k + i][r] = v[i];
    }
}
// dst[k][c] = src[k][c0 + c] * f(k) for k < 64 (zero from `rows` on) and 64 tile columns (zero from `cols` on): rows contiguous along the tile
template <typename T, typename F>
__device__ __forceinline__ void slab_along(float (*dst)[SP], const T* src, int ld, int rows, int c0, int cols, F f) {
    constexpr int V = Row16<T>::N;
    for (int e = threadIdx.x; e < 64 * (64 / V); e += 128) {
        const int k = e / (64 / V), c = (e % (64 / V)) * V;
        float v[V] = {};
        if (k < rows && c0 + c < cols) {
            Row16<T>::load(src + (size_t)k * ld + c0 + c, v);
            const float m = f(k);
#pragma unroll
            for (int i = 0; i < V; ++i) v[i] *= m;
        }
#pragma unroll
        for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(&dst[k][c + i]) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
}
__device__ __forceinline__ float row_of(const Acc84& acc, int i, int j) { return (i & 1) ? acc.v[i >> 1][j].y : acc.v[i >> 1][j].x; }

// ws_m[blk][group][t][s] = c_t . k_s
template <typename T>
__global__ void __launch_bounds__(128) chunk_products_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ Slab sh;
    const int blk = blockIdx.x, g = blockIdx.y, groups = gridDim.y;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const T* gc = (const T*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * a.N;
    const T* gk = (const T*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * a.N;
    const int tm = (threadIdx.x / 16) * 8, tn = (threadIdx.x % 16) * 4;
    Acc84 acc{};
    for (int n0 = 0; n0 < a.N; n0 += 64) {
        __syncthreads();
        slab_across(sh.a, gc, a.ld_c, len, n0, a.N, [](int) { return 1.f; });
        slab_across(sh.b, gk, a.ld_k, len, n0, a.N, [](int) { return 1.f; });
        __syncthreads();
        slab_fma(sh, min(64, a.N - n0), tm, tn, acc);
    }
    float* out = a.ws_m + ((size_t)blk * groups + g) * CL * CL;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(out + (tm + i) * CL + tn) = make_float4(row_of(acc, i, 0), row_of(acc, i, 1), row_of(acc, i, 2), row_of(acc, i, 3));
}

// a block's own contribution to the state, stored [p][n]
template <typename T>
__global__ void __launch_bounds__(128) chunk_state_head_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ Slab sh;
    __shared__ float rowf[CL];   // per row: the step scale times the decay from the row to the block's end
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int p0 = blockIdx.y * TS;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const T* gu = (const T*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * a.P;
    const T* gk = (const T*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * a.N;
    const float* gb = a.la + (size_t)(a.row0 + t0) * a.heads + h;
    const int tm = (threadIdx.x / 16) * 8, tn = (threadIdx.x % 16) * 4;
    if (threadIdx.x < CL) {
        const int s = threadIdx.x;
        rowf[s] = s < len ? (a.sc ? a.sc[(size_t)(a.row0 + t0 + s) * a.heads + h] : 1.f) *
                                expf(fminf(gb[(size_t)(len - 1) * a.heads] - gb[(size_t)s * a.heads], 0.f))
                          : 0.f;
    }
    __syncthreads();
    slab_along(sh.a, gu, a.ld_u, len, p0, a.P, [&](int s) { return rowf[s]; });
    float* out = a.ws_s + ((size_t)blk * a.heads + h) * a.P * a.N;
    for (int n0 = 0; n0 < a.N; n0 += TS) {
        if (n0) __syncthreads();
        slab_along(sh.b, gk, a.ld_k, len, n0, a.N, [](int) { return 1.f; });
        __syncthreads();
        Acc84 acc{};
        slab_fma(sh, len, tm, tn, acc);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (p0 + tm + i < a.P && n0 + tn < a.N)
                *reinterpret_cast<float4*>(out + (size_t)(p0 + tm + i) * a.N + n0 + tn) = make_float4(row_of(acc, i, 0), row_of(acc, i, 1), row_of(acc, i, 2), row_of(acc, i, 3));
    }
}

// contributions -> the state that enters each block (chunk_prefix_kernel, four neighbouring entries per thread)
__global__ void __launch_bounds__(256) chunk_prefix4_kernel(ChunkArgs a, int nblocks, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    const size_t per = (size_t)a.heads * a.P * a.N;
    const size_t idx = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (idx >= per) return;
    const int h = (int)(idx / ((size_t)a.P * a.N));
    float4 st = *reinterpret_cast<const float4*>(a.state + idx);
    for (int b0 = 0; b0 < nblocks; b0 += 8) {
        float4 d[8];
        float e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int b = b0 + i;
            if (b < nblocks) {
                d[i] = *reinterpret_cast<const float4*>(a.ws_s + (size_t)b * per + idx);
                e[i] = a.la[(size_t)(a.row0 + min((b + 1) * CL, a.S) - 1) * a.heads + h];
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int b = b0 + i;
            if (b < nblocks) {
                *reinterpret_cast<float4*>(a.ws_s + (size_t)b * per + idx) = st;
                const float f = expf(e[i]);
                st = make_float4(fmaf(f, st.x, d[i].x), fmaf(f, st.y, d[i].y), fmaf(f, st.z, d[i].z), fmaf(f, st.w, d[i].w));
            }
        }
    }
    *reinterpret_cast<float4*>(a.state + idx) = st;
}

template <typename T>
__global__ void __launch_bounds__(128) chunk_output_head_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ Slab sh;
    __shared__ float bt[CL], into[CL], scs[CL];   // per row: cumulative log decay, cs x decay from the block's start, cs x step scale
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int p0 = blockIdx.y * TS;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int N = a.N, P = a.P;
    const T* gu = (const T*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * P;
    const T* gc = (const T*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * N;
    const float* sin = a.ws_s + ((size_t)blk * a.heads + h) * P * N;
    const float* gm = a.ws_m + ((size_t)blk * (a.heads / a.heads_per_group) + g) * CL * CL;
    const int tm = (threadIdx.x / 16) * 8, tn = (threadIdx.x % 16) * 4;
    if (threadIdx.x < CL) {
        const int t = threadIdx.x;
        const float b = t < len ? a.la[(size_t)(a.row0 + t0 + t) * a.heads + h] : 0.f;
        bt[t] = b;
        into[t] = t < len ? a.cs * expf(b) : 0.f;
        scs[t] = t < len ? a.cs * (a.sc ? a.sc[(size_t)(a.row0 + t0 + t) * a.heads + h] : 1.f) : 0.f;
    }
    Acc84 acc{};
    for (int n0 = 0; n0 < N; n0 += 64) {       // the entering state, seen through the decayed queries
        __syncthreads();
        slab_across(sh.a, gc, a.ld_c, len, n0, N, [&](int t) { return into[t]; });
        slab_across(sh.b, sin + (size_t)p0 * N, N, min(TS, P - p0), n0, N, [](int) { return 1.f; });
        __syncthreads();
        slab_fma(sh, min(64, N - n0), tm, tn, acc);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < CL * CL / 4; e += 128) {   // the block's own rows: M[t, s], s <= t
        const int t = e & 63, s = (e >> 6) * 4;
        const float4 q = s <= t ? *reinterpret_cast<const float4*>(gm + t * CL + s) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) sh.a[s + i][t] = s + i <= t && t < len ? v[i] * scs[s + i] * expf(fminf(bt[t] - bt[s + i], 0.f)) : 0.f;
    }
    slab_along(sh.b, gu, a.ld_u, len, p0, P, [](int) { return 1.f; });
    __syncthreads();
    slab_fma(sh, len, tm, tn, acc);
    const float skip = a.skip ? a.skip[h] : 0.f;
    if (p0 + tn >= P) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = tm + i;
        if (t >= len) continue;
        const float4 u = *reinterpret_cast<const float4*>(&sh.b[t][tn]);   // the rows' own values are still staged
        *reinterpret_cast<float4*>(a.y + (size_t)(a.row0 + t0 + t) * a.ld_y + (size_t)h * P + p0 + tn) =
            make_float4(row_of(acc, i, 0) + skip * u.x, row_of(acc, i, 1) + skip * u.y, row_of(acc, i, 2) + skip * u.z, row_of(acc, i, 3) + skip * u.w);
    }
}

// ---- the three products of bf16 rows on the tensor cores -------------------------------------------------------------------
// Rows of c, k and u are bf16, so one operand of every product is exact; the other is fp32 (a state, decayed weights) and is cut into
// three bf16 values that hold all its 24 bits (truncated, so that none overflows): the products of mma.sync are then exact too. Its sums are not rounded
// like fp32 adds, and a running sum kept in its accumulators drifts (2.1e-6 of the summed magnitudes over 136 terms of one sign, where
// fp32 adds are 1.8e-7 off): 16 terms are summed there, three parts of them one after another, and added to the sum by the CUDA cores (9e-8; random
// signs 3.0e-9 for 4.5e-9).
// Decays and scales stay fp32. Bound by each warp's chain of cuts, three products and adds (16 to 20 warps per SM; outputs issue in 43 % of the slots and read at 16 % of HBM's rate;
// loads a step ahead, the first while the weights are formed, 73 -> 74): 2048 rows, 64 heads of
// 64 x 128, 7.8 + 33 + 73 us for 16 + 66 + 119 of the fp32 kernels (6.9 + 31 + 71 with running sums in the accumulators).
__device__ __forceinline__ float low_part(float x) {   // x minus its leading 8 bits; nothing behind an infinity or NaN
    return fabsf(x) < INFINITY ? x - __uint_as_float(__float_as_uint(x) & 0xffff0000u) : 0.f;
}
__device__ __forceinline__ void cut3(float x0, float x1, uint32_t (&c)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        c[i] = __byte_perm(__float_as_uint(x0), __float_as_uint(x1), 0x7632);
        if (i < 2) { x0 = low_part(x0); x1 = low_part(x1); }
    }
}
// acc += the three parts' products, the smallest first
__device__ __forceinline__ void add_products(float (&acc)[4], const uint32_t (&a)[3][4], uint32_t b0, uint32_t b1) {
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 2; k >= 0; --k) mma_bf16_16816(d, a[k], b0, b1);
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] += d[i];
}
constexpr int UP = 64 + 8;      // pitch of a staged bf16 tile row: ldmatrix rows fall into different banks
// four consecutive k of rows r and r + 8 as an A fragment: which of a product's 16 places a k takes does not matter, as long as B agrees
__device__ __forceinline__ void rows_a(uint32_t (&a)[4], const bf16* src, int ld, int r, int rows, int k, int cols) {
    const uint2 z = make_uint2(0u, 0u);
    const uint2 lo = r < rows && k < cols ? *reinterpret_cast<const uint2*>(src + (size_t)r * ld + k) : z;
    const uint2 hi = r + 8 < rows && k < cols ? *reinterpret_cast<const uint2*>(src + (size_t)(r + 8) * ld + k) : z;
    a[0] = lo.x; a[1] = hi.x; a[2] = lo.y; a[3] = hi.y;
}

// What an infinite or NaN entry of the uncut rows touches is summed again in plain fp32: the lower parts of most values are zero, and infinity
// times zero is not what the product is. A block's state is when its k hold one; an output when it came out non-finite (as it always
// does then). Not inlined and behind the rest, so that the others' registers and code stay as they are.
__device__ __forceinline__ void absmax8(__nv_bfloat162& most, const uint4& q) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) most = __hmax2_nan(most, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[j])));
}
__device__ __noinline__ void state_plain(const bf16* u, int ld_u, const bf16* k, int ld_k, const float* rowf, float* out, int len, int P, int N) {
    for (int e = threadIdx.x; e < P * N; e += blockDim.x) {
        const int p = e / N, n = e % N;
        float acc = 0.f;
        for (int s = 0; s < len; ++s) acc = fmaf(rowf[s] * bf2f(u[(size_t)s * ld_u + p]), bf2f(k[(size_t)s * ld_k + n]), acc);
        out[e] = acc;
    }
}
// the 32 outputs of a thread of chunk_output_tc_kernel, those that are not finite
__device__ __noinline__ void output_plain(const ChunkArgs& a) {
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int row = a.row0 + blk * CL, len = min(CL, a.S - blk * CL), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* m = a.ws_m + ((size_t)blk * (a.heads / a.heads_per_group) + g) * CL * CL;
    const float* la = a.la + (size_t)row * a.heads + h;
    for (int e = 0; e < 32; ++e) {
        const int t = (e >> 3) * 16 + (lane >> 2) + 8 * ((e >> 1) & 1), p = blockIdx.y * TS + warp * 16 + ((e >> 2) & 1) * 8 + 2 * (lane & 3) + (e & 1);
        if (t >= len || p >= a.P) continue;
        float* y = a.y + (size_t)(row + t) * a.ld_y + (size_t)h * a.P + p;
        if (isfinite(*y)) continue;
        const bf16* c = (const bf16*)a.c + (size_t)(row + t) * a.ld_c + (size_t)g * a.N;
        const bf16* u = (const bf16*)a.u + (size_t)row * a.ld_u + (size_t)h * a.P + p;
        const float* sin = a.ws_s + (((size_t)blk * a.heads + h) * a.P + p) * a.N;
        const float bt = la[(size_t)t * a.heads], into = a.cs * expf(bt);
        float acc = 0.f;
        for (int n = 0; n < a.N; ++n) acc = fmaf(into * bf2f(c[n]), sin[n], acc);
        for (int s = 0; s <= t; ++s) {
            const float sc = a.cs * (a.sc ? a.sc[(size_t)(row + s) * a.heads + h] : 1.f);
            acc = fmaf(m[t * CL + s] * sc * expf(fminf(bt - la[(size_t)s * a.heads], 0.f)), bf2f(u[(size_t)s * a.ld_u]), acc);
        }
        *y = acc + (a.skip ? a.skip[h] : 0.f) * bf2f(u[(size_t)t * a.ld_u]);
    }
}

__global__ void __launch_bounds__(128) chunk_products_tc_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    const int blk = blockIdx.x, g = blockIdx.y, groups = gridDim.y;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const bf16* gc = (const bf16*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * a.N;
    const bf16* gk = (const bf16*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * a.N;
    float acc[4][2][4] = {};
#pragma unroll 2
    for (int n0 = 0; n0 < a.N; n0 += 16) {
        uint32_t kb[4], ca[4][4];   // rows s of this warp's two tiles of 8
        rows_a(kb, gk, a.ld_k, warp * 16 + gq, len, n0 + 4 * tq, a.N);
#pragma unroll
        for (int i = 0; i < 4; ++i) rows_a(ca[i], gc, a.ld_c, i * 16 + gq, len, n0 + 4 * tq, a.N);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float d[2][4] = {};
            mma_bf16_16816(d[0], ca[i], kb[0], kb[2]);
            mma_bf16_16816(d[1], ca[i], kb[1], kb[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) { acc[i][0][e] += d[0][e]; acc[i][1][e] += d[1][e]; }
        }
    }
    float* out = a.ws_m + ((size_t)blk * groups + g) * CL * CL + warp * 16 + 2 * tq;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            *reinterpret_cast<float2*>(out + (i * 16 + gq) * CL + j * 8) = make_float2(acc[i][j][0], acc[i][j][1]);
            *reinterpret_cast<float2*>(out + (i * 16 + gq + 8) * CL + j * 8) = make_float2(acc[i][j][2], acc[i][j][3]);
        }
}

// a warp: 16 of the tile's 64 channels p, 64 key channels n at a time
// (five CTAs per SM: with six, whose 78 registers the compiler takes otherwise, a chained pass of three layers took 50 us more)
__global__ void __launch_bounds__(128, 5) chunk_state_tc_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ __align__(16) bf16 su[3][CL][UP], sk[CL][UP];   // [row s][p], cut in three; [row s][n]
    __shared__ float rowf[CL];   // per row: the step scale times the decay from the row to the block's end
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int p0 = blockIdx.y * TS;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const bf16* gu = (const bf16*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * a.P + p0;
    const bf16* gk = (const bf16*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * a.N;
    const float* gb = a.la + (size_t)(a.row0 + t0) * a.heads + h;
    float* out = a.ws_s + ((size_t)blk * a.heads + h) * a.P * a.N;
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    uint4 ur[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = threadIdx.x + i * 128, r = e >> 3, c = (e & 7) * 8;
        ur[i] = r < len && p0 + c < a.P ? *reinterpret_cast<const uint4*>(gu + (size_t)r * a.ld_u + c) : z;
    }
    if (threadIdx.x < CL) {
        const int s = threadIdx.x;
        rowf[s] = s < len ? (a.sc ? a.sc[(size_t)(a.row0 + t0 + s) * a.heads + h] : 1.f) *
                                expf(fminf(gb[(size_t)(len - 1) * a.heads] - gb[(size_t)s * a.heads], 0.f))
                          : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = threadIdx.x + i * 128, r = e >> 3, c = (e & 7) * 8;
        const uint32_t w[4] = {ur[i].x, ur[i].y, ur[i].z, ur[i].w};
        uint32_t q[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(w[j]);
            uint32_t t[3];
            cut3(f.x * rowf[r], f.y * rowf[r], t);
            q[0][j] = t[0]; q[1][j] = t[1]; q[2][j] = t[2];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4*>(&su[k][r][c]) = make_uint4(q[k][0], q[k][1], q[k][2], q[k][3]);
    }
    const int p = p0 + warp * 16 + gq;
    for (int n0 = 0; n0 < a.N; n0 += 64) {
        uint4 kr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 128, r = e >> 3, c = (e & 7) * 8;
            kr[i] = r < len && n0 + c < a.N ? *reinterpret_cast<const uint4*>(gk + (size_t)r * a.ld_k + n0 + c) : z;
        }
        if (n0) __syncthreads();
        __nv_bfloat162 most = __float2bfloat162_rn(0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 128;
            *reinterpret_cast<uint4*>(&sk[e >> 3][(e & 7) * 8]) = kr[i];
            absmax8(most, kr[i]);
        }
        if (__syncthreads_or(!isfinite(__low2float(most)) || !isfinite(__high2float(most)))) {
            state_plain(gu, a.ld_u, gk, a.ld_k, rowf, out + (size_t)p0 * a.N, len, min(TS, a.P - p0), a.N);
            return;
        }
        float acc[8][4] = {};
#pragma unroll
        for (int ks = 0; ks < CL; ks += 16) {
            uint32_t b[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                ldmatrix_x4_trans(b[j][0], b[j][1], b[j][2], b[j][3], &sk[ks + (lane & 7) + ((lane >> 3) & 1) * 8][j * 16 + (lane >> 4) * 8]);
            uint32_t w[3][4];
#pragma unroll
            for (int k = 0; k < 3; ++k)
                ldmatrix_x4_trans(w[k][0], w[k][1], w[k][2], w[k][3], &su[k][ks + (lane & 7) + (lane >> 4) * 8][warp * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                add_products(acc[2 * j], w, b[j][0], b[j][1]);
                add_products(acc[2 * j + 1], w, b[j][2], b[j][3]);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + j * 8 + 2 * tq;
            if (n >= a.N) continue;
            if (p < a.P) *reinterpret_cast<float2*>(out + (size_t)p * a.N + n) = make_float2(acc[j][0], acc[j][1]);
            if (p + 8 < a.P) *reinterpret_cast<float2*>(out + (size_t)(p + 8) * a.N + n) = make_float2(acc[j][2], acc[j][3]);
        }
    }
}

// The same for a decay per key channel: the decayed k is the operand that is cut, once per 64 key channels and for all value channels (u as it is).
// 2048 rows, 8 heads of 256 x 128: 25 us for 55 of chunk_state_kernel, which formed every decayed k once per 64 value channels.
__device__ __noinline__ void state_vec_plain(const ChunkArgs& a, const bf16* u, const bf16* k, const float* b, const float* sc, float* out, int len, int P, int cols) {
    const int ncol = a.heads * a.N;
    for (int e = threadIdx.x; e < P * cols; e += blockDim.x) {
        const int p = e / cols, n = e % cols;
        float acc = 0.f;
        for (int s = 0; s < len; ++s) {
            const float f = expf(fminf(b[(size_t)(len - 1) * ncol + n] - b[(size_t)s * ncol + n], 0.f)) * (sc ? sc[(size_t)s * a.heads] : 1.f);
            acc = fmaf(bf2f(u[(size_t)s * a.ld_u + p]), bf2f(k[(size_t)s * a.ld_k + n]) * f, acc);
        }
        out[(size_t)p * a.N + n] = acc;
    }
}
__global__ void __launch_bounds__(128, 5) chunk_state_vec_tc_kernel(const __grid_constant__ ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ __align__(16) bf16 sk[3][CL][UP], su[CL][UP];   // [row s][n], cut in three; [row s][p]
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int n0 = blockIdx.y * TS, N = a.N, P = a.P, ncol = a.heads * N;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const bf16* gu = (const bf16*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * P;
    const bf16* gk = (const bf16*)a.k + (size_t)(a.row0 + t0) * a.ld_k + (size_t)g * N + n0;
    const float* gb = a.la + (size_t)(a.row0 + t0) * ncol + (size_t)h * N + n0;
    const float* gsc = a.sc ? a.sc + (size_t)(a.row0 + t0) * a.heads + h : nullptr;
    float* out = a.ws_s + ((size_t)blk * a.heads + h) * P * N + n0;
    {
        const int c = (threadIdx.x & 7) * 8;                    // a thread's 8 key channels, of every 16th row
        const bool in = n0 + c < N;
        float last[8] = {};
        if (in) { ld4f(gb + (size_t)(len - 1) * ncol + c, last); ld4f(gb + (size_t)(len - 1) * ncol + c + 4, last + 4); }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = (threadIdx.x >> 3) + i * 16;
            uint32_t q[3][4] = {};
            if (r < len && in) {
                float kv[8], b[8];
                Row16<bf16>::load(gk + (size_t)r * a.ld_k + c, kv);
                ld4f(gb + (size_t)r * ncol + c, b); ld4f(gb + (size_t)r * ncol + c + 4, b + 4);
                const float f = gsc ? gsc[(size_t)r * a.heads] : 1.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t t[3];
                    cut3(kv[2 * j] * (expf(fminf(last[2 * j] - b[2 * j], 0.f)) * f), kv[2 * j + 1] * (expf(fminf(last[2 * j + 1] - b[2 * j + 1], 0.f)) * f), t);
                    q[0][j] = t[0]; q[1][j] = t[1]; q[2][j] = t[2];
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4*>(&sk[k][r][c]) = make_uint4(q[k][0], q[k][1], q[k][2], q[k][3]);
        }
    }
    for (int p0 = 0; p0 < P; p0 += TS) {
        uint4 ur[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 128, r = e >> 3, c = (e & 7) * 8;
            ur[i] = r < len && p0 + c < P ? *reinterpret_cast<const uint4*>(gu + (size_t)r * a.ld_u + p0 + c) : make_uint4(0u, 0u, 0u, 0u);
        }
        if (p0) __syncthreads();
        __nv_bfloat162 most = __float2bfloat162_rn(0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = threadIdx.x + i * 128;
            *reinterpret_cast<uint4*>(&su[e >> 3][(e & 7) * 8]) = ur[i];
            absmax8(most, ur[i]);
        }
        if (__syncthreads_or(!isfinite(__low2float(most)) || !isfinite(__high2float(most)))) {
            state_vec_plain(a, gu + p0, gk, gb, gsc, out + (size_t)p0 * N, len, min(TS, P - p0), min(TS, N - n0));
            continue;
        }
        float acc[8][4] = {};
#pragma unroll
        for (int ks = 0; ks < CL; ks += 16) {
            uint32_t w[4];
            ldmatrix_x4_trans(w[0], w[1], w[2], w[3], &su[ks + (lane & 7) + (lane >> 4) * 8][warp * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float d[2][4] = {};
#pragma unroll
                for (int k = 2; k >= 0; --k) {
                    uint32_t b[4];
                    ldmatrix_x4_trans(b[0], b[1], b[2], b[3], &sk[k][ks + (lane & 7) + ((lane >> 3) & 1) * 8][j * 16 + (lane >> 4) * 8]);
                    mma_bf16_16816(d[0], w, b[0], b[1]);
                    mma_bf16_16816(d[1], w, b[2], b[3]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) { acc[2 * j][e] += d[0][e]; acc[2 * j + 1][e] += d[1][e]; }
            }
        }
        const int p = p0 + warp * 16 + gq;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = j * 8 + 2 * tq;
            if (n0 + n >= N) continue;
            if (p < P) *reinterpret_cast<float2*>(out + (size_t)p * N + n) = make_float2(acc[j][0], acc[j][1]);
            if (p + 8 < P) *reinterpret_cast<float2*>(out + (size_t)(p + 8) * N + n) = make_float2(acc[j][2], acc[j][3]);
        }
    }
}

// Outputs for a decay per key channel: both operands of the product with the state are fp32 (the decays differ along n), so it stays on the CUDA cores:
// packed fp32 pairs, 8 x (4 NJ) of a tile of 64 rows x 64 NJ channels per thread, so that 16 bytes read from shared memory feed 8 NJ / (2 + NJ) packed products.
// Slabs of 32: rows of 16-byte pieces are swizzled, so that neither the transposing stores nor the reads meet in a bank.
// 2048 rows, 8 heads of 256 x 128: 49 us for 79 of chunk_output_kernel (50 in tiles of 64 channels, 54 with three CTAs per SM and no spill).
template <typename T, int NJ>
__global__ void __launch_bounds__(128, 4) chunk_output_vec_kernel(ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    constexpr int D = 32, TP = 64 * NJ, V = Row16<T>::N;
    __shared__ __align__(16) float sa[D][CL], sb[D][TP];       // [depth][row t], [depth][channel p], swizzled
    auto at = [](int k, int x) { return x ^ (((k >> 2) & 7) << 2); };
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int p0 = blockIdx.y * TP, t0 = blk * CL, len = min(CL, a.S - t0), N = a.N, P = a.P, ncol = a.heads * N;
    const T* gu = (const T*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * P + p0;
    const T* gc = (const T*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * N;
    const float* gb = a.la + (size_t)(a.row0 + t0) * ncol + (size_t)h * N;
    const float* sin = a.ws_s + (((size_t)blk * a.heads + h) * P + p0) * N;
    const float* gm = a.ws_m + ((size_t)blk * a.heads + h) * CL * CL;
    const int tm = (threadIdx.x >> 4) * 8, tn = (threadIdx.x & 15) * 4;
    float2 acc[4][4 * NJ] = {};                                // rows (2 i, 2 i + 1) x column j
    auto product = [&] {
#pragma unroll 4
        for (int k = 0; k < D; ++k) {
            const float4 a0 = *reinterpret_cast<const float4*>(&sa[k][at(k, tm)]), a1 = *reinterpret_cast<const float4*>(&sa[k][at(k, tm + 4)]);
            const float2 ar[4] = {make_float2(a0.x, a0.y), make_float2(a0.z, a0.w), make_float2(a1.x, a1.y), make_float2(a1.z, a1.w)};
#pragma unroll
            for (int m = 0; m < NJ; ++m) {
                const float4 b4 = *reinterpret_cast<const float4*>(&sb[k][at(k, tn) + 64 * m]);
                const float bj[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][4 * m + j] = __ffma2_rn(ar[i], make_float2(bj[j], bj[j]), acc[i][4 * m + j]);
            }
        }
    };
    for (int n0 = 0; n0 < N; n0 += D) {        // the entering state, seen through the decayed queries
        __syncthreads();
#pragma unroll
        for (int e = threadIdx.x; e < CL * (D / V); e += 128) {
            const int r = e / (D / V), k = (e % (D / V)) * V;
            float v[V] = {};
            if (r < len && n0 + k < N) {
                float b[V];
                Row16<T>::load(gc + (size_t)r * a.ld_c + n0 + k, v);
#pragma unroll
                for (int i = 0; i < V; i += 4) ld4f(gb + (size_t)r * ncol + n0 + k + i, b + i);
#pragma unroll
                for (int i = 0; i < V; ++i) v[i] = a.cs * v[i] * expf(b[i]);
            }
#pragma unroll
            for (int i = 0; i < V; ++i) sa[k + i][at(k + i, r)] = v[i];
        }
#pragma unroll
        for (int e = threadIdx.x; e < TP * (D / 4); e += 128) {
            const int r = e / (D / 4), k = (e % (D / 4)) * 4;
            float v[4] = {};
            if (p0 + r < P && n0 + k < N) ld4f(sin + (size_t)r * N + n0 + k, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) sb[k + i][at(k + i, r)] = v[i];
        }
        __syncthreads();
        product();
    }
    for (int s0 = 0; s0 < len; s0 += D) {      // the block's own rows (their weights hold cs, the step scales and the decays)
        __syncthreads();
#pragma unroll
        for (int e = threadIdx.x; e < CL * (D / 4); e += 128) {
            const int r = e / (D / 4), k = (e % (D / 4)) * 4;
            float v[4];
            ld4f(gm + r * CL + s0 + k, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) sa[k + i][at(k + i, r)] = v[i];
        }
#pragma unroll
        for (int e = threadIdx.x; e < D * (TP / V); e += 128) {
            const int k = e / (TP / V), c = (e % (TP / V)) * V;
            float v[V] = {};
            if (s0 + k < len && p0 + c < P) Row16<T>::load(gu + (size_t)(s0 + k) * a.ld_u + c, v);
#pragma unroll
            for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(&sb[k][at(k, c + i)]) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        __syncthreads();
        product();
    }
    const float skip = a.skip ? a.skip[h] : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = tm + i;
        if (t >= len) continue;
#pragma unroll
        for (int m = 0; m < NJ; ++m) {
            const int p = tn + 64 * m;
            if (p0 + p >= P) continue;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[j] = (i & 1) ? acc[i >> 1][4 * m + j].y : acc[i >> 1][4 * m + j].x;
                if (a.skip) v[j] += skip * ldf(gu + (size_t)t * a.ld_u + p + j);
            }
            *reinterpret_cast<float4*>(a.y + (size_t)(a.row0 + t0 + t) * a.ld_y + (size_t)h * P + p0 + p) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}

// a warp: all 64 rows of 16 of the tile's channels, so that every state is cut once
__global__ void __launch_bounds__(128, 4) chunk_output_tc_kernel(const __grid_constant__ ChunkArgs a, SeqPos pos) {
    chain_begin();
    if (seq_done(pos)) return;
    __shared__ __align__(16) bf16 sm[3][CL][UP], su[CL][UP];   // the block's own weights [t][s], cut in three; [row s][p]
    __shared__ float bt[CL], into[CL], scs[CL];   // per row: cumulative log decay, cs x decay from the block's start, cs x step scale
    const int blk = blockIdx.x / a.heads, h = blockIdx.x % a.heads, g = h / a.heads_per_group;
    const int p0 = blockIdx.y * TS;
    const int t0 = blk * CL, len = min(CL, a.S - t0);
    const int N = a.N, P = a.P;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
    const bf16* gu = (const bf16*)a.u + (size_t)(a.row0 + t0) * a.ld_u + (size_t)h * P + p0;
    const bf16* gc = (const bf16*)a.c + (size_t)(a.row0 + t0) * a.ld_c + (size_t)g * N;
    const float* sin = a.ws_s + ((size_t)blk * a.heads + h) * P * N;
    const float* gm = a.ws_m + ((size_t)blk * (a.heads / a.heads_per_group) + g) * CL * CL;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = threadIdx.x + i * 128, r = e >> 3, c = (e & 7) * 8;
        *reinterpret_cast<uint4*>(&su[r][c]) = r < len && p0 + c < P ? *reinterpret_cast<const uint4*>(gu + (size_t)r * a.ld_u + c) : make_uint4(0u, 0u, 0u, 0u);
    }
    if (threadIdx.x < CL) {
        const int t = threadIdx.x;
        const float b = t < len ? a.la[(size_t)(a.row0 + t0 + t) * a.heads + h] : 0.f;
        bt[t] = b;
        into[t] = t < len ? a.cs * expf(b) : 0.f;
        scs[t] = t < len ? a.cs * (a.sc ? a.sc[(size_t)(a.row0 + t0 + t) * a.heads + h] : 1.f) : 0.f;
    }
    __syncthreads();
    // the block's own rows: M[t, s], s <= t. Of a row's pieces of four only those up to the end of its 16 x 16 tile on the diagonal: 77 us became 74
    for (int e = threadIdx.x; e < CL * CL / 4 * 5 / 8; e += 128) {
        const int tile = e < 64 ? 0 : e < 192 ? 1 : e < 384 ? 2 : 3, x = e - 32 * tile * (tile + 1);   // 64 (tile + 1) pieces per 16 rows
        const int t = tile * 16 + x / (4 * tile + 4), s = x % (4 * tile + 4) * 4;
        const float4 q = s <= t ? *reinterpret_cast<const float4*>(gm + t * CL + s) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float v[4] = {q.x, q.y, q.z, q.w};
        float m[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = s + i <= t && t < len ? v[i] * scs[s + i] * expf(fminf(bt[t] - bt[s + i], 0.f)) : 0.f;
        uint32_t c0[3], c1[3];
        cut3(m[0], m[1], c0);
        cut3(m[2], m[3], c1);
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(&sm[k][t][s]) = make_uint2(c0[k], c1[k]);
    }
    float acc[4][2][4] = {};
#pragma unroll 2
    for (int n0 = 0; n0 < N; n0 += 16) {       // the entering state, seen through the queries
        const int n = n0 + 4 * tq;
        float4 st[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int p = p0 + warp * 16 + j * 8 + gq;
            st[j] = p < P && n < N ? *reinterpret_cast<const float4*>(sin + (size_t)p * N + n) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        uint32_t ca[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) rows_a(ca[i], gc, a.ld_c, i * 16 + gq, len, n, N);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint32_t b0[3], b1[3];
            cut3(st[j].x, st[j].y, b0);
            cut3(st[j].z, st[j].w, b1);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 2; k >= 0; --k) mma_bf16_16816(d, ca[i], b0[k], b1[k]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][j][e] += d[e];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float f0 = into[i * 16 + gq], f1 = into[i * 16 + gq + 8];
            acc[i][j][0] *= f0; acc[i][j][1] *= f0;
            acc[i][j][2] *= f1; acc[i][j][3] *= f1;
        }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        uint32_t b[4];
        ldmatrix_x4_trans(b[0], b[1], b[2], b[3], &su[ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][warp * 16 + (lane >> 4) * 8]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i < ks) continue;   // rows above these keys
            uint32_t w[3][4];
#pragma unroll
            for (int k = 0; k < 3; ++k) ldmatrix_x4(w[k][0], w[k][1], w[k][2], w[k][3], &sm[k][i * 16 + (lane & 15)][ks * 16 + (lane >> 4) * 8]);
            add_products(acc[i][0], w, b[0], b[1]);
            add_products(acc[i][1], w, b[2], b[3]);
        }
    }
    const float skip = a.skip ? a.skip[h] : 0.f;
    float odd = 0.f;   // NaN once a value is not finite
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = i * 16 + gq + 8 * r, c = warp * 16 + j * 8 + 2 * tq;
                if (t >= len || p0 + c >= P) continue;
                const float2 u = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(&su[t][c]));
                const float2 v = make_float2(acc[i][j][2 * r] + skip * u.x, acc[i][j][2 * r + 1] + skip * u.y);
                *reinterpret_cast<float2*>(a.y + (size_t)(a.row0 + t0 + t) * a.ld_y + (size_t)h * P + p0 + c) = v;
                odd = fmaf(0.f, v.x, fmaf(0.f, v.y, odd));
            }
    if (odd != 0.f) output_plain(a);
}

template <typename T, bool VEC>
int run_chunked(const ScanArgs& s, SeqPos pos, cudaStream_t st) {
    const size_t per_block = (size_t)s.heads * ((size_t)CL * CL + (size_t)s.P * s.N);
    const int max_blocks = (int)std::min<size_t>(s.ws_floats / per_block, 1 << 20);
    if (max_blocks < 1) return -3;
    ChunkArgs a{};
    a.k = s.k; a.ld_k = s.ld_k; a.c = s.c; a.ld_c = s.ld_c; a.u = s.u; a.ld_u = s.ld_u;
    a.la = s.a; a.sc = s.sc; a.skip = s.skip; a.cs = s.cs; a.state = s.state; a.y = s.y; a.ld_y = s.ld_y;
    a.heads = s.heads; a.heads_per_group = s.heads_per_group; a.N = s.N; a.P = s.P; a.NV = VEC ? s.N : 1;
    const size_t per_state = (size_t)s.heads * s.P * s.N;
    for (int row0 = 0; row0 < s.S; row0 += max_blocks * CL) {
        const int rows = std::min(s.S - row0, max_blocks * CL), nb = (rows + CL - 1) / CL;
        a.row0 = row0; a.S = rows;
        a.ws_m = s.ws; a.ws_s = s.ws + (size_t)nb * s.heads * CL * CL;
        const int ncol = a.heads * a.NV;
        count_launch();
        chained(chunk_cumsum_kernel, dim3(nb, (ncol + 127) / 128), 128, 0, st)(a, pos);
        constexpr int V = Row16<T>::N;
        const bool rows16 = ((s.N | s.P | s.ld_k | s.ld_c | s.ld_u) % V) == 0 && ((s.N | s.P | s.ld_y) % 4) == 0 &&
                            (((uintptr_t)s.k | (uintptr_t)s.c | (uintptr_t)s.u | (uintptr_t)s.y | (uintptr_t)s.state | (uintptr_t)a.ws_m | (uintptr_t)a.ws_s) % 16) == 0 &&
                            (!VEC || ((uintptr_t)s.a % 16) == 0);
        if constexpr (!VEC) {
            if (rows16) {
                const dim3 tiles(nb * s.heads, (s.P + TS - 1) / TS), pairs(nb, s.heads / s.heads_per_group);
                const unsigned prefix = (unsigned)((per_state / 4 + 255) / 256);
                for (int i = 0; i < 4; ++i) count_launch();
                if constexpr (std::is_same_v<T, bf16>) {
                    chained(chunk_products_tc_kernel, pairs, 128, 0, st)(a, pos);
                    chained(chunk_state_tc_kernel, tiles, 128, 0, st)(a, pos);
                    chained(chunk_prefix4_kernel, prefix, 256, 0, st)(a, nb, pos);
                    chained(chunk_output_tc_kernel, tiles, 128, 0, st)(a, pos);
                } else {
                    chained(chunk_products_kernel<T>, pairs, 128, 0, st)(a, pos);
                    chained(chunk_state_head_kernel<T>, tiles, 128, 0, st)(a, pos);
                    chained(chunk_prefix4_kernel, prefix, 256, 0, st)(a, nb, pos);
                    chained(chunk_output_head_kernel<T>, tiles, 128, 0, st)(a, pos);
                }
                continue;
            }
        }
        for (int i = 0; i < 4; ++i) count_launch();
        if constexpr (VEC) chained(chunk_weights_vec_kernel<T>, dim3(nb, s.heads), 512, 0, st)(a, pos);
        else chained(chunk_weights_kernel<T>, dim3(nb, s.heads / s.heads_per_group), 256, 0, st)(a, pos);
        bool state_done = false;
        if constexpr (VEC && std::is_same_v<T, bf16>) {
            if (rows16) {
                chained(chunk_state_vec_tc_kernel, dim3(nb * s.heads, (s.N + TS - 1) / TS), 128, 0, st)(a, pos);
                state_done = true;
            }
        }
        if (!state_done) chained(chunk_state_kernel<T, VEC>, dim3(nb * s.heads, (s.P + TS - 1) / TS, (s.N + TS - 1) / TS), 256, 0, st)(a, pos);
        chained(chunk_prefix_kernel<VEC>, (unsigned)((per_state + 255) / 256), 256, 0, st)(a, nb, pos);
        if constexpr (VEC) {
            if (rows16) {   // channels in tiles of 128 where a head has more than 64
                if (s.P > 64) chained(chunk_output_vec_kernel<T, 2>, dim3(nb * s.heads, (s.P + 127) / 128), 128, 0, st)(a, pos);
                else chained(chunk_output_vec_kernel<T, 1>, dim3(nb * s.heads, 1), 128, 0, st)(a, pos);
                continue;
            }
        }
        chained(chunk_output_kernel<T, VEC>, dim3(nb * s.heads, (s.P + TS - 1) / TS), 256, 0, st)(a, pos);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -100;
}

}  // namespace

size_t gated_scan_ws_floats(int S, int heads, int N, int P) {
    const size_t nb = std::min<size_t>(((size_t)(S > 0 ? S : 1) + CL - 1) / CL, kScanMaxBlocks);
    return nb * (size_t)heads * ((size_t)CL * CL + (size_t)P * N);
}

int gated_scan_chunked(const ScanArgs& a, SeqPos pos, cudaStream_t s) {
    if (!a.ws) return -2;
    if (a.dt == DT_F32) return a.vec_decay ? run_chunked<float, true>(a, pos, s) : run_chunked<float, false>(a, pos, s);
    return a.vec_decay ? run_chunked<bf16, true>(a, pos, s) : run_chunked<bf16, false>(a, pos, s);
}

}  // namespace lcc
