// Attention kernels of the LiveCC path, mma.sync.m16n8k16 bf16 flash-style with cp.async-staged K/V tiles.
// The ViT and prefill kernels here were the round's first implementation and are now the fallback / cross-check of
// the tcgen05 + TMEM kernels (attention_tc.cu, attention_prefill_tc.cu), which the launchers below dispatch to by
// default; the one-token decode attention (HBM-bound) lives only here.
//
//  * flash_fwd_kernel<D, CAUSAL, PAGED>: multi-row attention.
//      - ViT (D=80, non-causal, K/V read from the fused qkv buffer, one cu_seqlens segment per
//        blockIdx.z):  VisionAttention, mq2vl.py:392-454.
//      - decoder prefill (D=128, causal over past+new, K/V read from the paged cache, the G query
//        heads of a KV group packed into the row dimension so a K/V tile is loaded once per group):
//        Qwen2VLAttention, mq2vl.py:572-594 + eager_attention_forward :353-375.
//  * attn_decode_kernel: one new token, split-KV over the paged cache; the 7 query heads of a KV
//    group form one 16-row MMA tile; fuses the 1-D RoPE of q, the RoPE + append of the new k/v.
//    The last CTA of a KV group to finish merges the split-KV partials (no separate combine launch).
// Softmax statistics are fp32; P is rounded to bf16 before P·V (as the reference does, :370).
#include <stdlib.h>

#include "../../include/livecc_b200.h"
#include "common.cuh"
#include "launch.h"
#include "mma.cuh"
#include "ops.h"

namespace lcc {

// One warp: S[16 x 16*NT16] = Q_frag (16 x D) * K_tile^T.  K_tile rows (tokens) start at `ks`
// (row stride LDS elements); NT16 groups of 16 tokens.
template <int D, int LDS, int NT16>
__device__ __forceinline__ void warp_qk(const uint32_t (&qf)[D / 16][4], const bf16* ks, int lane,
                                        float (&s)[NT16 * 2][4]) {
#pragma unroll
    for (int n = 0; n < NT16 * 2; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[n][j] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
        for (int nt = 0; nt < NT16; ++nt) {
            // x4: matrices (tok 0-7,k 0-7) (tok 0-7,k 8-15) (tok 8-15,k 0-7) (tok 8-15,k 8-15)
            const int mat = lane >> 3, r = lane & 7;
            const bf16* p = ks + (size_t)(nt * 16 + (mat >> 1) * 8 + r) * LDS + kk * 16 + (mat & 1) * 8;
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4(b0, b1, b2, b3, p);
            mma_bf16_16816(s[nt * 2], qf[kk], b0, b1);
            mma_bf16_16816(s[nt * 2 + 1], qf[kk], b2, b3);
        }
    }
}

// One warp: O[16 x D] += P (16 x 16*NT16, bf16 A fragments) * V_tile (tokens x D).
template <int D, int LDS, int NT16>
__device__ __forceinline__ void warp_pv(const uint32_t (&pf)[NT16][4], const bf16* vs, int lane,
                                        float (&o)[D / 8][4]) {
#pragma unroll
    for (int kt = 0; kt < NT16; ++kt) {
#pragma unroll
        for (int dn = 0; dn < D / 16; ++dn) {
            // trans x4: matrices (tok 0-7,d 0-7) (tok 8-15,d 0-7) (tok 0-7,d 8-15) (tok 8-15,d 8-15)
            const int mat = lane >> 3, r = lane & 7;
            const bf16* p = vs + (size_t)(kt * 16 + (mat & 1) * 8 + r) * LDS + dn * 16 + (mat >> 1) * 8;
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4_trans(b0, b1, b2, b3, p);
            mma_bf16_16816(o[dn * 2], pf[kt], b0, b1);
            mma_bf16_16816(o[dn * 2 + 1], pf[kt], b2, b3);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Multi-row flash attention. CTA = 4 warps = 64 packed rows; KV tiles of 64 tokens.
// Packed row r of KV group g maps to (query position r / G, query head g*G + r % G).
// ---------------------------------------------------------------------------------------------
struct FlashParams {
    const bf16* q;      // [S, *] row stride q_ld; head h at column h*D
    int q_ld;
    const bf16* k;      // contiguous mode: row stride kv_ld, head g at column g*D
    const bf16* v;
    int kv_ld;
    const bf16* kc;     // paged mode: [pages, Hkv, P=64, D]
    const bf16* vc;
    const int* page_table;
    int Hkv;
    bf16* out;          // [S, *] row stride o_ld; head h at column h*D
    int o_ld;
    const int* cu_seqlens;  // contiguous mode: segment boundaries (blockIdx.z); null => one segment [0,S)
    int S;              // number of query positions (paged mode / single segment)
    int past;           // paged+causal: number of cached tokens before the S new ones
    int G;              // query heads per KV head
    float scale_log2;   // softmax scale * log2(e)
    // split-KV (paged mode only): blockIdx.z = split; partials are merged by flash_merge_kernel
    int nsplit;
    float* part_o;      // [nsplit, Hkv, S*G, D] unnormalised fp32
    float* part_ml;     // [nsplit, Hkv, S*G, 2]
};

template <int D, bool CAUSAL, bool PAGED>
__global__ void __launch_bounds__(128) flash_fwd_kernel(const FlashParams p) {
    constexpr int LDS = D + 8;
    constexpr int BM = 64, BN = 64;
    extern __shared__ __align__(16) uint8_t smem_attn[];
    bf16* sq = reinterpret_cast<bf16*>(smem_attn);           // [64][LDS]
    bf16* sk = sq + BM * LDS;                                 // [2][64][LDS]
    bf16* sv = sk + 2 * BN * LDS;                             // [2][64][LDS]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = blockIdx.y;  // KV head / group
    int seg_start = 0, seg_len = p.S;
    if (!PAGED && p.cu_seqlens) {
        seg_start = p.cu_seqlens[blockIdx.z];
        seg_len = p.cu_seqlens[blockIdx.z + 1] - seg_start;
    }
    const int rows_total = seg_len * p.G;
    const int row0 = blockIdx.x * BM;
    if (row0 >= rows_total) return;

    // ---- stage Q tile (zero-filled beyond rows_total) ----
    for (int i = threadIdx.x; i < BM * (D / 8); i += 128) {
        const int r = i / (D / 8), c = i % (D / 8);
        const int rr = row0 + r;
        const bool ok = rr < rows_total;
        const int pos = ok ? rr / p.G : 0, hq = g * p.G + (ok ? rr % p.G : 0);
        cp_async16(sq + r * LDS + c * 8, p.q + (size_t)(seg_start + pos) * p.q_ld + (size_t)hq * D + c * 8, ok);
    }
    cp_async_commit();

    // KV range for this CTA
    int kv_len = PAGED ? (p.past + p.S) : seg_len;
    if (CAUSAL) {
        const int last_row = min(row0 + BM, rows_total) - 1;
        kv_len = min(kv_len, p.past + last_row / p.G + 1);
    }
    const int n_tiles = (kv_len + BN - 1) / BN;
    int tile_lo = 0, tile_hi = n_tiles;
    const bool split = PAGED && p.nsplit > 1;
    if (split) {
        const int tiles_total = (p.past + p.S + BN - 1) / BN;
        const int tps = (tiles_total + p.nsplit - 1) / p.nsplit;
        tile_lo = blockIdx.z * tps;
        tile_hi = min(n_tiles, tile_lo + tps);
        if (tile_lo >= tile_hi) {  // nothing to do for this split: neutral partial (m = -inf, l = 0)
            cp_async_commit();
            cp_async_wait<0>();
            float* ml = p.part_ml + (((size_t)blockIdx.z * p.Hkv + g) * rows_total + row0) * 2;
            for (int i = threadIdx.x; i < min(BM, rows_total - row0); i += 128) { ml[i * 2] = -INFINITY; ml[i * 2 + 1] = 0.f; }
            return;
        }
    }

    auto load_kv = [&](int tile, int buf) {
        bf16* dk = sk + buf * BN * LDS;
        bf16* dv = sv + buf * BN * LDS;
        const int t0 = tile * BN;
        const bf16 *gk, *gv;
        size_t stride;
        if (PAGED) {
            const int page = p.page_table[tile];
            gk = p.kc + ((size_t)page * p.Hkv + g) * BN * D;
            gv = p.vc + ((size_t)page * p.Hkv + g) * BN * D;
            stride = D;
        } else {
            gk = p.k + (size_t)(seg_start + t0) * p.kv_ld + (size_t)g * D;
            gv = p.v + (size_t)(seg_start + t0) * p.kv_ld + (size_t)g * D;
            stride = p.kv_ld;
        }
        for (int i = threadIdx.x; i < BN * (D / 8); i += 128) {
            const int r = i / (D / 8), c = i % (D / 8);
            const bool ok = (t0 + r) < kv_len;
            cp_async16(dk + r * LDS + c * 8, gk + (size_t)r * stride + c * 8, ok);
            cp_async16(dv + r * LDS + c * 8, gv + (size_t)r * stride + c * 8, ok);
        }
    };

    if (tile_lo < tile_hi) load_kv(tile_lo, 0);
    cp_async_commit();

    cp_async_wait<1>();  // Q landed
    __syncthreads();
    uint32_t qf[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
        const int mat = lane >> 3, r = lane & 7;
        const bf16* ptr = sq + (size_t)(warp * 16 + (mat & 1) * 8 + r) * LDS + kk * 16 + (mat >> 1) * 8;
        ldmatrix_x4(qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], ptr);
    }

    float o[D / 8][4];
#pragma unroll
    for (int d = 0; d < D / 8; ++d)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[d][j] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

    // causal limit (inclusive key index) of this thread's two rows
    int lim[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int rr = row0 + warp * 16 + (lane >> 2) + r * 8;
        lim[r] = CAUSAL ? (p.past + rr / p.G) : (kv_len - 1);
    }

    for (int t = tile_lo; t < tile_hi; ++t) {
        const int buf = (t - tile_lo) & 1;
        if (t + 1 < tile_hi) load_kv(t + 1, buf ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const bf16* ks = sk + buf * BN * LDS;
        const bf16* vs = sv + buf * BN * LDS;
        float s[8][4];
        warp_qk<D, LDS, 4>(qf, ks, lane, s);
        // mask: key index beyond the causal limit or beyond kv_len
        const int kbase = t * BN + 2 * (lane & 3);
        const bool need_mask = CAUSAL ? true : ((t + 1) * BN > kv_len);
        if (need_mask) {
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int kidx = kbase + n * 8;
                if (kidx > lim[0] || kidx >= kv_len) s[n][0] = -INFINITY;
                if (kidx + 1 > lim[0] || kidx + 1 >= kv_len) s[n][1] = -INFINITY;
                if (kidx > lim[1] || kidx >= kv_len) s[n][2] = -INFINITY;
                if (kidx + 1 > lim[1] || kidx + 1 >= kv_len) s[n][3] = -INFINITY;
            }
        }
        uint32_t pf[4][4];
        softmax_step<D, 4>(s, p.scale_log2, m, l, o, pf);
        warp_pv<D, LDS, 4>(pf, vs, lane, o);
        __syncthreads();  // all warps done with this buffer before it is refilled
    }

    // finalize: full row sums across the quad, normalise, store bf16
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
    if (split) {  // unnormalised partial + (m, l) for the merge kernel
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int rr = row0 + warp * 16 + (lane >> 2) + r * 8;
            if (rr >= rows_total) continue;
            const size_t prow = ((size_t)blockIdx.z * p.Hkv + g) * rows_total + rr;
            float* dst = p.part_o + prow * D + 2 * (lane & 3);
#pragma unroll
            for (int d = 0; d < D / 8; ++d)
                *reinterpret_cast<float2*>(dst + d * 8) = make_float2(o[d][2 * r], o[d][2 * r + 1]);
            if ((lane & 3) == 0) { p.part_ml[prow * 2] = m[r]; p.part_ml[prow * 2 + 1] = l[r]; }
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int rr = row0 + warp * 16 + (lane >> 2) + r * 8;
        if (rr >= rows_total) continue;
        const float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
        const int pos = rr / p.G, hq = g * p.G + rr % p.G;
        bf16* dst = p.out + (size_t)(seg_start + pos) * p.o_ld + (size_t)hq * D + 2 * (lane & 3);
#pragma unroll
        for (int d = 0; d < D / 8; ++d) {
            *reinterpret_cast<uint32_t*>(dst + d * 8) = pack_bf16x2(o[d][2 * r] * inv, o[d][2 * r + 1] * inv);
        }
    }
}

// Merge of the split-KV partials of the prefill attention (up to 32 of them): a warp per packed row, four dims per lane. A lane weighs one
// split; the partials are then read four at a time, 16 bytes per lane. (281 rows x 28 heads, 4 splits: 8.8 us; a CTA per
// row with a dim per thread took 15.9.)
constexpr int kMergeRows = 8;   // rows per CTA
__global__ void __launch_bounds__(32 * kMergeRows) flash_merge_kernel(const float* __restrict__ part_o,
                                                                      const float* __restrict__ part_ml, const __grid_constant__ PrefillStreams ps,
                                                                      int Hkv, int G, float scale_log2, bf16* __restrict__ out, int o_ld) {
    chain_begin(part_o, part_ml);
    const PrefillStream& st = ps.st[blockIdx.z];
    const int rr = blockIdx.x * kMergeRows + (threadIdx.x >> 5), g = blockIdx.y, lane = threadIdx.x & 31;
    const int rows_total = st.S * G, nsplit = st.nsplit;
    if (nsplit < 2 || rr >= rows_total) return;
    part_o += st.part_row * 128;
    part_ml += st.part_row * 2;
    out += (size_t)st.row0 * o_ld;
    const size_t row = (size_t)g * rows_total + rr, step = (size_t)Hkv * rows_total;
    float m = -INFINITY, l = 0.f;
    if (lane < nsplit) {
        const float2 ml = *reinterpret_cast<const float2*>(part_ml + (lane * step + row) * 2);
        m = ml.x;
        l = ml.y;
    }
    const float M = warp_max(m);
    const float f = m == -INFINITY ? 0.f : exp2f((m - M) * scale_log2);
    const float L = warp_sum(f * l);
    const unsigned has = __ballot_sync(0xffffffffu, m != -INFINITY);   // a split without keys wrote no partial
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s0 = 0; s0 < nsplit; s0 += 4) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = has >> (s0 + i) & 1 ? *reinterpret_cast<const float4*>(part_o + ((s0 + i) * step + row) * 128 + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float fi = __shfl_sync(0xffffffffu, f, s0 + i);
            acc[0] = fmaf(fi, v[i].x, acc[0]);
            acc[1] = fmaf(fi, v[i].y, acc[1]);
            acc[2] = fmaf(fi, v[i].z, acc[2]);
            acc[3] = fmaf(fi, v[i].w, acc[3]);
        }
    }
    const int pos = rr / G, hq = g * G + rr % G;
    const bool any = L > 0.f;
    *reinterpret_cast<uint2*>(out + (size_t)pos * o_ld + (size_t)hq * 128 + lane * 4) =
        make_uint2(pack_bf16x2(any ? acc[0] / L : 0.f, any ? acc[1] / L : 0.f), pack_bf16x2(any ? acc[2] / L : 0.f, any ? acc[3] / L : 0.f));
}

template <int D, bool CAUSAL, bool PAGED>
static int launch_flash(const FlashParams& p, dim3 grid, cudaStream_t s) {
    constexpr int LDS = D + 8;
    constexpr int smem = (64 + 4 * 64) * LDS * 2;
    auto kern = flash_fwd_kernel<D, CAUSAL, PAGED>;
    static SmemAttrOnce once;  // per instantiation
    if (ensure_dyn_smem(once, kern, smem)) return -1;
    { lcc::count_launch(); kern<<<grid, 128, smem, s>>>(p); }
    return 0;
}

// ---------------------------------------------------------------------------------------------
// ViT attention with MT (= 2) row tiles per warp: CTA = 4 warps = 128 query rows. Every K/V fragment loaded
// with ldmatrix feeds MT MMAs, which halves the shared-memory traffic per FLOP of the 64-row kernel above
// (the limiter of the mma.sync path at head_dim 80). Non-causal, K/V read from the fused qkv buffer, one
// cu_seqlens segment per blockIdx.z (VisionAttention, mq2vl.py:392-454).
// ---------------------------------------------------------------------------------------------
template <int MT>
__global__ void __launch_bounds__(128) vit_flash_kernel(const FlashParams p) {
    constexpr int D = 80, LDS = D + 8, BN = 64, BM = 64 * MT;
    extern __shared__ __align__(16) uint8_t smem_attn[];
    bf16* sq = reinterpret_cast<bf16*>(smem_attn);  // [BM][LDS]
    bf16* sk = sq + BM * LDS;                        // [2][64][LDS]
    bf16* sv = sk + 2 * BN * LDS;                    // [2][64][LDS]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int head = blockIdx.y;
    const int seg_start = p.cu_seqlens[blockIdx.z];
    const int seg_len = p.cu_seqlens[blockIdx.z + 1] - seg_start;
    const int row0 = blockIdx.x * BM;
    if (row0 >= seg_len) return;

    for (int i = threadIdx.x; i < BM * (D / 8); i += 128) {
        const int r = i / (D / 8), c = i % (D / 8);
        const bool ok = (row0 + r) < seg_len;
        cp_async16(sq + r * LDS + c * 8, p.q + (size_t)(seg_start + (ok ? row0 + r : 0)) * p.q_ld + (size_t)head * D + c * 8, ok);
    }
    cp_async_commit();
    const int n_tiles = (seg_len + BN - 1) / BN;
    auto load_kv = [&](int tile, int buf) {
        bf16* dk = sk + buf * BN * LDS;
        bf16* dv = sv + buf * BN * LDS;
        const int t0 = tile * BN;
        const bf16* gk = p.k + (size_t)(seg_start + t0) * p.kv_ld + (size_t)head * D;
        const bf16* gv = p.v + (size_t)(seg_start + t0) * p.kv_ld + (size_t)head * D;
        for (int i = threadIdx.x; i < BN * (D / 8); i += 128) {
            const int r = i / (D / 8), c = i % (D / 8);
            const bool ok = (t0 + r) < seg_len;
            cp_async16(dk + r * LDS + c * 8, gk + (size_t)(ok ? r : 0) * p.kv_ld + c * 8, ok);
            cp_async16(dv + r * LDS + c * 8, gv + (size_t)(ok ? r : 0) * p.kv_ld + c * 8, ok);
        }
    };
    load_kv(0, 0);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();

    uint32_t qf[MT][D / 16][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            const int mat = lane >> 3, r = lane & 7;
            const bf16* ptr = sq + (size_t)((warp * MT + mt) * 16 + (mat & 1) * 8 + r) * LDS + kk * 16 + (mat >> 1) * 8;
            ldmatrix_x4(qf[mt][kk][0], qf[mt][kk][1], qf[mt][kk][2], qf[mt][kk][3], ptr);
        }
    float o[MT][D / 8][4];
    float m[MT][2], l[MT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        m[mt][0] = m[mt][1] = -INFINITY;
        l[mt][0] = l[mt][1] = 0.f;
#pragma unroll
        for (int d = 0; d < D / 8; ++d)
#pragma unroll
            for (int j = 0; j < 4; ++j) o[mt][d][j] = 0.f;
    }

    for (int t = 0; t < n_tiles; ++t) {
        const int buf = t & 1;
        if (t + 1 < n_tiles) load_kv(t + 1, buf ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const bf16* ks = sk + buf * BN * LDS;
        const bf16* vs = sv + buf * BN * LDS;
        float s[MT][8][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[mt][n][j] = 0.f;
        // S = Q K^T : each K fragment feeds MT row tiles
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int mat = lane >> 3, r = lane & 7;
                const bf16* ptr = ks + (size_t)(nt * 16 + (mat >> 1) * 8 + r) * LDS + kk * 16 + (mat & 1) * 8;
                uint32_t b0, b1, b2, b3;
                ldmatrix_x4(b0, b1, b2, b3, ptr);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    mma_bf16_16816(s[mt][nt * 2], qf[mt][kk], b0, b1);
                    mma_bf16_16816(s[mt][nt * 2 + 1], qf[mt][kk], b2, b3);
                }
            }
        }
        if ((t + 1) * BN > seg_len) {  // ragged last tile
            const int kbase = t * BN + 2 * (lane & 3);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    const int kidx = kbase + n * 8;
                    if (kidx >= seg_len) { s[mt][n][0] = -INFINITY; s[mt][n][2] = -INFINITY; }
                    if (kidx + 1 >= seg_len) { s[mt][n][1] = -INFINITY; s[mt][n][3] = -INFINITY; }
                }
        }
        uint32_t pf[MT][4][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) softmax_step<D, 4>(s[mt], p.scale_log2, m[mt], l[mt], o[mt], pf[mt]);
        // O += P V : each V fragment feeds MT row tiles
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
#pragma unroll
            for (int dn = 0; dn < D / 16; ++dn) {
                const int mat = lane >> 3, r = lane & 7;
                const bf16* ptr = vs + (size_t)(kt * 16 + (mat & 1) * 8 + r) * LDS + dn * 16 + (mat >> 1) * 8;
                uint32_t b0, b1, b2, b3;
                ldmatrix_x4_trans(b0, b1, b2, b3, ptr);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    mma_bf16_16816(o[mt][dn * 2], pf[mt][kt], b0, b1);
                    mma_bf16_16816(o[mt][dn * 2 + 1], pf[mt][kt], b2, b3);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float lr = l[mt][r];
            lr += __shfl_xor_sync(0xffffffffu, lr, 1);
            lr += __shfl_xor_sync(0xffffffffu, lr, 2);
            const int rr = row0 + (warp * MT + mt) * 16 + (lane >> 2) + r * 8;
            if (rr >= seg_len) continue;
            const float inv = lr > 0.f ? 1.f / lr : 0.f;
            bf16* dst = p.out + (size_t)(seg_start + rr) * p.o_ld + (size_t)head * D + 2 * (lane & 3);
#pragma unroll
            for (int d = 0; d < D / 8; ++d)
                *reinterpret_cast<uint32_t*>(dst + d * 8) = pack_bf16x2(o[mt][d][2 * r] * inv, o[mt][d][2 * r + 1] * inv);
        }
}

// ViT: qkv [N, 3*heads*80]; segments from cu_seqlens (device int32, nseg+1 entries); max_seg_len bounds the grid.
int vit_attention(const bf16* qkv, int ld, int64_t n_rows, bf16* out, int o_ld, const int* cu_seqlens, int nseg,
                  int max_seg_len, int heads, int head_dim, int impl, cudaStream_t s, bool alike) {
    if (head_dim != 80) return -1;
    if (nseg <= 0 || max_seg_len <= 0) return 0;
    if (impl == 0) {
        const char* e = getenv("LIVECC_B200_VIT_ATTN");  // "mma" forces the mma.sync kernels
        impl = (e && e[0] == 'm') ? 1 : 2;
    }
    if (impl == 2 && cu_seqlens) return vit_attention_tc(qkv, ld, n_rows, out, o_ld, cu_seqlens, nseg, max_seg_len, heads, alike, s);
    FlashParams p{};
    p.q = qkv; p.q_ld = ld;
    p.k = qkv + (size_t)heads * head_dim; p.v = qkv + (size_t)2 * heads * head_dim; p.kv_ld = ld;
    p.out = out; p.o_ld = o_ld; p.cu_seqlens = cu_seqlens; p.S = max_seg_len; p.past = 0; p.G = 1;
    p.Hkv = heads;
    p.scale_log2 = 1.4426950408889634f / sqrtf((float)head_dim);
    // 128-row CTAs (two row tiles per warp) once they still give every SM >= 2 CTAs; else the 64-row kernel
    int dev_sms = 148;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, dev);
    const int ctas128 = ((max_seg_len + 127) / 128) * heads * nseg;
    if (cu_seqlens && ctas128 >= 2 * dev_sms) {
        constexpr int smem = (128 + 4 * 64) * 88 * 2;
        static SmemAttrOnce once;
        if (ensure_dyn_smem(once, vit_flash_kernel<2>, smem)) return -2;
        { lcc::count_launch(); vit_flash_kernel<2><<<dim3((max_seg_len + 127) / 128, heads, nseg), 128, smem, s>>>(p); }
        return 0;
    }
    dim3 grid((max_seg_len + 63) / 64, heads, nseg);
    return launch_flash<80, false, false>(p, grid, s);
}

int attn_prefill_streams(const bf16* q, int q_ld, const bf16* kc, const bf16* vc, const PrefillStreams& ps, int page_size, int Hq, int Hkv, bf16* out,
                         int o_ld, float* part_o, float* part_ml, size_t part_capacity_rows, int num_sms, int impl, cudaStream_t s) {
    if (page_size != 64) return -1;
    if (impl == 0) {
        const char* e = getenv("LIVECC_B200_PREFILL_ATTN");  // "mma" forces the mma.sync kernel
        impl = (e && e[0] == 'm') ? 1 : 2;
    }
    if (impl == 1) {
        for (int b = 0; b < ps.n; ++b) {
            const PrefillStream& st = ps.st[b];
            if (int r = attn_prefill_paged(q + (size_t)st.row0 * q_ld, q_ld, kc, vc, st.page_table, page_size, Hq, Hkv, st.S, st.past,
                                           out + (size_t)st.row0 * o_ld, o_ld, part_o, part_ml, part_capacity_rows, num_sms, 1, s))
                return r;
        }
        return 0;
    }
    const int G = Hq / Hkv;
    if (G < 1 || G > 128 || Hq % Hkv || (q_ld % 8) || (o_ld % 8)) return -1;
    if (!part_o || !part_ml || ((uintptr_t)part_o % 16) || ((uintptr_t)part_ml % 8)) part_capacity_rows = 0;
    for (int b = 0; b < ps.n;) {   // streams whose partials fit together
        PrefillStreams some{};
        some.rows = ps.rows;
        size_t used = 0;
        int longest = 0;   // of those with partials
        for (; b < ps.n; ++b) {
            PrefillStream& st = some.st[some.n];
            st = ps.st[b];
            st.nsplit = attn_prefill_tc_splits(st.S, st.past, Hq, Hkv, part_capacity_rows, num_sms);
            const size_t need = st.nsplit > 1 ? (size_t)st.nsplit * Hq * st.S : 0;
            if (used + need > part_capacity_rows) break;
            st.part_row = used;
            used += need;
            if (need) longest = std::max(longest, st.S);
            ++some.n;
        }
        if (int r = attn_prefill_tc(q, q_ld, kc, vc, some, Hq, Hkv, out, o_ld, part_o, part_ml, s)) return r;
        if (longest) {
            lcc::count_launch();
            chained(flash_merge_kernel, dim3((longest * G + kMergeRows - 1) / kMergeRows, Hkv, some.n), 32 * kMergeRows, 0, s)(
                part_o, part_ml, some, Hkv, G, 1.4426950408889634f / sqrtf(128.f), out, o_ld);
        }
    }
    return 0;
}

// Decoder prefill: q rows of the fused qkv buffer (already rotated), K/V in the paged cache
// (already containing the S new tokens at positions past..past+S-1).
int attn_prefill_paged(const bf16* q, int q_ld, const bf16* kc, const bf16* vc, const int* page_table,
                       int page_size, int Hq, int Hkv, int S, int past, bf16* out, int o_ld, float* part_o,
                       float* part_ml, size_t part_capacity_rows, int num_sms, int impl, cudaStream_t s) {
    if (page_size != 64) return -1;
    if (S <= 0) return 0;
    if (impl == 0) {
        const char* e = getenv("LIVECC_B200_PREFILL_ATTN");  // "mma" forces the mma.sync kernel
        impl = (e && e[0] == 'm') ? 1 : 2;
    }
    if (impl == 2) {
        PrefillStreams ps{};
        ps.n = 1; ps.rows = S;
        ps.st[0].page_table = page_table; ps.st[0].S = S; ps.st[0].past = past;
        return attn_prefill_streams(q, q_ld, kc, vc, ps, page_size, Hq, Hkv, out, o_ld, part_o, part_ml, part_capacity_rows, num_sms, impl, s);
    }
    FlashParams p{};
    p.q = q; p.q_ld = q_ld; p.kc = kc; p.vc = vc; p.page_table = page_table; p.Hkv = Hkv;
    p.out = out; p.o_ld = o_ld; p.cu_seqlens = nullptr; p.S = S; p.past = past; p.G = Hq / Hkv;
    p.scale_log2 = 1.4426950408889634f / sqrtf(128.f);
    const int q_tiles = (S * p.G + 63) / 64;
    const int ctas = q_tiles * Hkv;
    const int kv_tiles = (past + S + 63) / 64;
    // split the KV range when a chunk-sized prefill over a long cache cannot fill two CTAs per SM
    int nsplit = 1;
    const bool merge_ok = (o_ld % 4) == 0 && ((uintptr_t)out % 8) == 0 && ((uintptr_t)part_o % 16) == 0 && ((uintptr_t)part_ml % 8) == 0;
    if (part_o && part_ml && merge_ok && ctas < 2 * num_sms) {
        nsplit = (2 * num_sms + ctas - 1) / ctas;
        if (nsplit > 8) nsplit = 8;
        while (nsplit > 1 && kv_tiles < 8 * nsplit) --nsplit;  // keep >= 8 tiles of work per split
        if ((size_t)nsplit * Hkv * S * p.G > part_capacity_rows) nsplit = 1;
    }
    p.nsplit = nsplit; p.part_o = part_o; p.part_ml = part_ml;
    dim3 grid(q_tiles, Hkv, nsplit);
    if (int r = launch_flash<128, true, true>(p, grid, s)) return r;
    if (nsplit > 1) {
        PrefillStreams ps{};
        ps.n = 1; ps.rows = S;
        ps.st[0].S = S; ps.st[0].nsplit = nsplit;
        lcc::count_launch();
        chained(flash_merge_kernel, dim3((S * p.G + kMergeRows - 1) / kMergeRows, Hkv), 32 * kMergeRows, 0, s)(part_o, part_ml, ps, Hkv, p.G, p.scale_log2, out, o_ld);
    }
    return 0;
}

// ---------------------------------------------------------------------------------------------
// Decode attention (one token). grid = (Hkv, nsplit); CTA = 4 warps; each warp owns 16 of the 64
// tokens of a page-tile; rows of the MMA tile = the G (<=16) query heads of the KV group.
// Device-side scalars (graph-replay friendly): kv_len = tokens already in the cache; the new token
// is appended at slot kv_len by the CTA whose range contains it.
// ---------------------------------------------------------------------------------------------
struct DecodeAttnParams {
    bf16* qkv;          // [ (Hq + 2Hkv) * 128 ] raw projections (+bias) of the new token
    bf16* kc;           // layer K cache [pages, Hkv, 64, 128]
    bf16* vc;
    const int* page_table;
    const int* kv_len;      // device scalar
    const int* rope_pos;    // device scalar: position id of the new token (kv_len + rope_delta)
    const int* finished;    // device flag: non-zero => no-op
    const float* inv_freq;  // [64]
    int Hq, Hkv, nsplit;
    float* part_o;      // [nsplit, Hq, 128]
    float* part_ml;     // [nsplit, Hq, 2]  (running max (unscaled), l)
    int* counters;      // [Hkv] arrival counters, zero between launches (last CTA of a group merges the splits)
    bf16* out;          // [Hq * 128]
    float scale_log2;
    int* done_groups;   // optional: incremented once per KV group when its merged output is in `out`
};

// o_proj role of the fused attention + o_proj kernel (see attn_oproj_kernel)
struct OprojParams {
    const bf16* W;      // [N, K] o_proj weight
    int ldw, N, K;
    bf16* h;            // residual stream, updated in place
    int* sync;          // [0] = KV groups done (producer flag), [1] = o_proj CTAs finished (for the reset)
    int n_cta;          // number of o_proj CTAs
};

__device__ __forceinline__ void rope1d_row(const bf16* src, bf16* dst, int lane_dim /*0..63*/, float pos,
                                           const float* inv_freq) {
    // one (j, j+64) pair; torch bf16 semantics (each product and the sum rounded to bf16)
    const float ang = __fmul_rn(pos, inv_freq[lane_dim]);
    const float c = rbf(cosf(ang)), s = rbf(sinf(ang));
    const float x1 = bf2f(src[lane_dim]), x2 = bf2f(src[lane_dim + 64]);
    dst[lane_dim] = f2bf(rbf(rbf(x1 * c) + rbf(-x2 * s)));
    dst[lane_dim + 64] = f2bf(rbf(rbf(x2 * c) + rbf(x1 * s)));
}

// The decode kernel's K/V tiles go through kDecBuf shared-memory buffers: while one tile is computed the next two are in flight.
constexpr int kDecBuf = 3, kDecLds = 136, kDecSmem = (16 + kDecBuf * 2 * 64) * kDecLds * 2;

// CL = 1: `split` of p.nsplit key ranges, the last CTA of a KV group to arrive merges all splits from global memory. CL = 8: the eight
// CTAs of a cluster hold eight consecutive splits and merge them through their shared memory, one query head each; one partial
// per cluster goes to global memory, and the last cluster to arrive merges p.nsplit / 8 of them (again one head per CTA). What bounds a
// step over a short cache is the chain launch -> page -> tile -> merge, over a long one the bytes in flight: with 64 splits of two CTAs per
// SM and three buffers both get shorter. A merge of 32 partials by one CTA per KV group was the longest link of the chain.
// 16 tokens of four layers: over 8k tokens 11.20 -> 10.93 ms (4.5 us per launch), over 65k 12.31 -> 11.90 ms (6.8 us).
template <int CL>
__device__ __forceinline__ void attn_decode_role(const DecodeAttnParams& p, const int g, const int split,
                                                 uint8_t* smem_attn) {
    constexpr int D = 128, LDS = kDecLds, BN = 64;
    pdl_wait();  // qkv of this token comes from the previous kernel
    if (p.finished && *p.finished) return;
    bf16* sq = reinterpret_cast<bf16*>(smem_attn);  // [16][LDS]
    bf16* sk = sq + 16 * LDS;                        // [kDecBuf][64][LDS]
    bf16* sv = sk + kDecBuf * BN * LDS;              // [kDecBuf][64][LDS]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.Hq / p.Hkv;
    const int kv_old = *p.kv_len;
    const int T = kv_old + 1;
    const float pos = (float)(*p.rope_pos);

    const int n_tiles_total = (T + BN - 1) / BN;
    const int tiles_per_split = (n_tiles_total + p.nsplit - 1) / p.nsplit;
    const int tile_begin = split * tiles_per_split;
    const int tile_end = min(n_tiles_total, tile_begin + tiles_per_split);

    const bool empty = tile_begin >= tile_end;
    // this CTA's merged partial of its split: with a cluster it lies in shared memory behind the warps' partials
    float* po = p.part_o + ((size_t)split * p.Hq + (size_t)g * G) * D;
    float* pml = p.part_ml + ((size_t)split * p.Hq + (size_t)g * G) * 2;
    if (CL > 1) {
        po = reinterpret_cast<float*>(sv);           // [8][128]
        pml = po + 8 * D;                            // [8][2]
    }
    if (empty) {  // empty split: neutral partial
        if (threadIdx.x < G) { pml[threadIdx.x * 2] = -INFINITY; pml[threadIdx.x * 2 + 1] = 0.f; }
    } else {

    // ---- append the new token's k (rotated) and v to the cache (the CTA owning the last tile) ----
    if (tile_end == n_tiles_total) {
        const int page = p.page_table[kv_old / BN], slot = kv_old % BN;
        bf16* dk = p.kc + (((size_t)page * p.Hkv + g) * BN + slot) * D;
        bf16* dv = p.vc + (((size_t)page * p.Hkv + g) * BN + slot) * D;
        const bf16* ksrc = p.qkv + (size_t)(p.Hq + g) * D;
        const bf16* vsrc = p.qkv + (size_t)(p.Hq + p.Hkv + g) * D;
        if (threadIdx.x < 64) rope1d_row(ksrc, dk, threadIdx.x, pos, p.inv_freq);
        else if (threadIdx.x < 80) {
            const int c = threadIdx.x - 64;
            *reinterpret_cast<uint4*>(dv + c * 8) = *reinterpret_cast<const uint4*>(vsrc + c * 8);
        }
        __threadfence();
        __syncthreads();   // the row is written before any thread of this CTA copies the last tile
    }

    auto load_kv = [&](int tile) {
        if (tile < tile_end) {
            const int buf = (tile - tile_begin) % kDecBuf;
            bf16* dk = sk + buf * BN * LDS;
            bf16* dv = sv + buf * BN * LDS;
            const int page = p.page_table[tile];
            const bf16* gk = p.kc + ((size_t)page * p.Hkv + g) * BN * D;
            const bf16* gv = p.vc + ((size_t)page * p.Hkv + g) * BN * D;
            const int t0 = tile * BN;
            for (int i = threadIdx.x; i < BN * (D / 8); i += 128) {
                const int r = i >> 4, c = i & 15;
                const bool ok = (t0 + r) < T;
                cp_async16(dk + r * LDS + c * 8, gk + (size_t)r * D + c * 8, ok);
                cp_async16(dv + r * LDS + c * 8, gv + (size_t)r * D + c * 8, ok);
            }
        }
        cp_async_commit();   // (a group per tile slot, empty past the end, so that the waits count alike)
    };
#pragma unroll
    for (int i = 0; i < kDecBuf - 1; ++i) load_kv(tile_begin + i);

    // ---- q: rotate the G heads of this group into smem (rows >= G zero) while the first tiles arrive ----
    for (int i = threadIdx.x; i < 16 * 64; i += 128) {
        const int r = i >> 6, j = i & 63;
        if (r < G) rope1d_row(p.qkv + (size_t)(g * G + r) * D, sq + r * LDS, j, pos, p.inv_freq);
        else { sq[r * LDS + j] = f2bf(0.f); sq[r * LDS + j + 64] = f2bf(0.f); }
    }
    __syncthreads();

    uint32_t qf[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
        const int mat = lane >> 3, r = lane & 7;
        const bf16* ptr = sq + (size_t)((mat & 1) * 8 + r) * LDS + kk * 16 + (mat >> 1) * 8;
        ldmatrix_x4(qf[kk][0], qf[kk][1], qf[kk][2], qf[kk][3], ptr);
    }
    float o[D / 8][4];
#pragma unroll
    for (int d = 0; d < D / 8; ++d)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[d][j] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

    for (int t = tile_begin; t < tile_end; ++t) {
        const int buf = (t - tile_begin) % kDecBuf;
        cp_async_wait<kDecBuf - 2>();
        __syncthreads();   // tile t has landed for everybody, and everybody is done with the buffer of tile t - 1
        load_kv(t + kDecBuf - 1);
        const bf16* ks = sk + buf * BN * LDS + warp * 16 * LDS;
        const bf16* vs = sv + buf * BN * LDS + warp * 16 * LDS;
        float s[2][4];
        warp_qk<D, LDS, 1>(qf, ks, lane, s);
        const int kbase = t * BN + warp * 16 + 2 * (lane & 3);
        if ((t + 1) * BN > T) {
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int kidx = kbase + n * 8;
                if (kidx >= T) { s[n][0] = -INFINITY; s[n][2] = -INFINITY; }
                if (kidx + 1 >= T) { s[n][1] = -INFINITY; s[n][3] = -INFINITY; }
            }
        }
        uint32_t pf[1][4];
        softmax_step<D, 1>(s, p.scale_log2, m, l, o, pf);
        warp_pv<D, LDS, 1>(pf, vs, lane, o);
    }
    cp_async_wait<0>();   // (empty groups)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }

    // ---- merge the 4 warps (each saw a disjoint token subset) through shared memory ----
    float* so = reinterpret_cast<float*>(sk);  // [4][8][128] fp32 = 16 KB   (only rows < 8 are kept: G <= 8)
    float* sml = so + 4 * 8 * D;               // [4][8][2]
    __syncthreads();
    if ((lane >> 2) < 8) {
        const int r = lane >> 2;  // row (thread's first row); second row r+8 is padding when G <= 8
        float* dst = so + ((size_t)warp * 8 + r) * D + 2 * (lane & 3);
#pragma unroll
        for (int d = 0; d < D / 8; ++d) { dst[d * 8] = o[d][0]; dst[d * 8 + 1] = o[d][1]; }
        if ((lane & 3) == 0) { sml[(warp * 8 + r) * 2] = m[0]; sml[(warp * 8 + r) * 2 + 1] = l[0]; }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < G * D; i += 128) {
        const int r = i / D, d = i % D;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < 4; ++w) M = fmaxf(M, sml[(w * 8 + r) * 2]);
        float acc = 0.f, L = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float mw = sml[(w * 8 + r) * 2];
            const float f = (mw == -INFINITY) ? 0.f : exp2f((mw - M) * p.scale_log2);
            acc += f * so[((size_t)w * 8 + r) * D + d];
            L += f * sml[(w * 8 + r) * 2 + 1];
        }
        po[(size_t)r * D + d] = acc;
        if (d == 0) { pml[r * 2] = M; pml[r * 2 + 1] = L; }
    }
    }  // !empty

    if (CL > 1) {
        // ---- cluster: CTA r merges query head r of the cluster's splits, then of all clusters if it arrives last ----
        pdl_launch_dependents();
        const int rank = (int)cluster_ctarank(), ncl = p.nsplit / CL;
        __syncwarp();
        cluster_sync_all();        // every CTA's partial is in its shared memory
        float M = -INFINITY, acc = 0.f, L = 0.f;
        const int d = threadIdx.x;
        if (rank < G) {
            float mw[CL], lw[CL], ow[CL];
#pragma unroll
            for (int c = 0; c < CL; ++c) {
                mw[c] = ld_cluster_f32(pml + rank * 2, c);
                lw[c] = ld_cluster_f32(pml + rank * 2 + 1, c);
                ow[c] = ld_cluster_f32(po + rank * D + d, c);
                M = fmaxf(M, mw[c]);
            }
#pragma unroll
            for (int c = 0; c < CL; ++c) {
                if (mw[c] != -INFINITY) {   // (an empty split left no output)
                    const float f = exp2f((mw[c] - M) * p.scale_log2);
                    acc = fmaf(f, ow[c], acc);
                    L = fmaf(f, lw[c], L);
                }
            }
        }
        __syncwarp();
        cluster_arrive();          // this CTA has read its peers; it leaves only when they have read it
        if (rank < G && ncl == 1) p.out[(size_t)(g * G + rank) * D + d] = f2bf(L > 0.f ? acc / L : 0.f);
        if (rank < G && ncl > 1) {
            __shared__ int s_last_row;
            const size_t row = (size_t)(split / CL) * p.Hq + (size_t)g * G + rank;
            p.part_o[row * D + d] = acc;
            if (d == 0) { p.part_ml[row * 2] = M; p.part_ml[row * 2 + 1] = L; }
            __threadfence();
            __syncthreads();
            // the KV group's counter holds one 4-bit arrival count per head (at most 8 clusters)
            if (d == 0) {
                const unsigned prev = atomicAdd(reinterpret_cast<unsigned*>(&p.counters[g]), 1u << (4 * rank));
                s_last_row = ((prev >> (4 * rank)) & 15u) == (unsigned)(ncl - 1);
                if (s_last_row) atomicSub(reinterpret_cast<unsigned*>(&p.counters[g]), (unsigned)ncl << (4 * rank));   // ready for the next launch
            }
            __syncthreads();
            if (s_last_row) {
                __threadfence();
                float mw[CL], lw[CL], ow[CL];
                M = -INFINITY; acc = 0.f; L = 0.f;
#pragma unroll
                for (int c = 0; c < CL; ++c) {
                    const size_t r = (size_t)min(c, ncl - 1) * p.Hq + (size_t)g * G + rank;
                    mw[c] = c < ncl ? __ldcg(p.part_ml + r * 2) : -INFINITY;
                    lw[c] = __ldcg(p.part_ml + r * 2 + 1);
                    ow[c] = __ldcg(p.part_o + r * D + d);
                    M = fmaxf(M, mw[c]);
                }
#pragma unroll
                for (int c = 0; c < CL; ++c) {
                    if (mw[c] != -INFINITY) {
                        const float f = exp2f((mw[c] - M) * p.scale_log2);
                        acc = fmaf(f, ow[c], acc);
                        L = fmaf(f, lw[c], L);
                    }
                }
                p.out[(size_t)(g * G + rank) * D + d] = f2bf(L > 0.f ? acc / L : 0.f);
            }
        }
        __syncwarp();
        cluster_wait();
        return;
    }

    // ---- the last CTA of this KV group to arrive merges all splits (replaces a separate combine launch) ----
    pdl_launch_dependents();
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const int prev = atomicAdd(&p.counters[g], 1);
        s_last = (prev == p.nsplit - 1) ? 1 : 0;
    }
    __syncthreads();
    if (!s_last) return;
    if (threadIdx.x == 0) p.counters[g] = 0;  // ready for the next launch
    __threadfence();
    float* sm_m = reinterpret_cast<float*>(smem_attn);  // [8][64]
    float* sm_l = sm_m + 8 * 64;                         // [8][64]
    for (int i = threadIdx.x; i < G * p.nsplit; i += 128) {
        const int r = i / p.nsplit, sp = i % p.nsplit;
        const float* ml = p.part_ml + ((size_t)sp * p.Hq + (size_t)g * G + r) * 2;
        sm_m[r * 64 + sp] = __ldcg(ml);
        sm_l[r * 64 + sp] = __ldcg(ml + 1);
    }
    __syncthreads();
    // warp w merges rows w, w+4; a lane owns 4 consecutive dims (float4 loads, all splits independent)
    for (int r = warp; r < G; r += 4) {
        float M = -INFINITY;
        for (int sp = 0; sp < p.nsplit; ++sp) M = fmaxf(M, sm_m[r * 64 + sp]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float L = 0.f;
        const float* base = p.part_o + ((size_t)g * G + r) * D + lane * 4;
        const size_t sp_stride = (size_t)p.Hq * D;
#pragma unroll 8
        for (int sp = 0; sp < p.nsplit; ++sp) {
            const float ms = sm_m[r * 64 + sp];
            const bool live = ms != -INFINITY;
            const float f = live ? exp2f((ms - M) * p.scale_log2) : 0.f;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live) v = __ldcg(reinterpret_cast<const float4*>(base + sp * sp_stride));
            acc.x += f * v.x; acc.y += f * v.y; acc.z += f * v.z; acc.w += f * v.w;
            L += f * sm_l[r * 64 + sp];
        }
        const float inv = L > 0.f ? 1.f / L : 0.f;
        uint2 o;
        o.x = pack_bf16x2(acc.x * inv, acc.y * inv);
        o.y = pack_bf16x2(acc.z * inv, acc.w * inv);
        *reinterpret_cast<uint2*>(p.out + (size_t)(g * G + r) * D + lane * 4) = o;
    }
    if (p.done_groups) {  // publish this group's slice of `out` to the o_proj CTAs of the fused kernel
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(p.done_groups, 1);
    }
}

__global__ void __launch_bounds__(128) attn_decode_kernel(const DecodeAttnParams p) {
    extern __shared__ __align__(16) uint8_t smem_attn[];
    attn_decode_role<1>(p, blockIdx.x, blockIdx.y, smem_attn);
}
__global__ void __cluster_dims__(1, 8, 1) __launch_bounds__(128) attn_decode_cluster_kernel(const DecodeAttnParams p) {
    extern __shared__ __align__(16) uint8_t smem_attn[];
    attn_decode_role<8>(p, blockIdx.x, blockIdx.y, smem_attn);
}

// Slices of the grid (z) per stream of a batched step. A stream's keys are split by its own length alone, so that its bits do not depend on its
// neighbours: eight splits, sixteen past kBatchLong tokens (the second cluster of a shorter stream, behind all others in the grid, leaves at once).
// Eight splits of eight streams are one wave of CTAs, and more cost their fixed part again (us, 8 | 16 | 32 splits: 8 streams of 200, 2000, 8000,
// 16384 tokens 10.2 | 20.7 | 25.2, 14.8 | 26.6 | 43.8, 30.8 | 41.2 | 59.3, 52.8 | 64.3 | 82.5); few streams of long caches leave SMs idle with
// eight (4 x 8000 27.3 | 21.5 | 31.4, 2 x 8000 19.8 | 19.1 | 16.5, 2 x 30000 54 | 38 | 31). Chosen by the number of streams before, as low as each row has.
constexpr int kBatchLong = 16384;
struct DecodeAttnBatchParams {
    DecodeAttnParams one;
    AttnStream st[kBatchStreams];
    int qkv_ld, out_ld, B;
};
__global__ void __cluster_dims__(1, 8, 1) __launch_bounds__(128) attn_decode_batch_kernel(const __grid_constant__ DecodeAttnBatchParams bp) {
    extern __shared__ __align__(16) uint8_t smem_attn[];
    const int b = blockIdx.z % bp.B, cluster = blockIdx.z / bp.B;
    DecodeAttnParams p = bp.one;
    p.nsplit = bp.st[b].scalars[LCC_SC_KV_LEN] >= kBatchLong ? 16 : 8;
    if (cluster * 8 >= p.nsplit) return;
    p.qkv += (size_t)b * bp.qkv_ld;
    p.out += (size_t)b * bp.out_ld;
    p.page_table = bp.st[b].page_table;
    p.kv_len = bp.st[b].scalars + LCC_SC_KV_LEN;
    p.rope_pos = bp.st[b].scalars + LCC_SC_ROPE_POS;
    p.finished = bp.st[b].scalars + LCC_SC_FINISHED;
    p.part_o += (size_t)b * 8 * p.Hq * 128;
    p.part_ml += (size_t)b * 8 * p.Hq * 2;
    p.counters += b * p.Hkv;
    attn_decode_role<8>(p, blockIdx.x, cluster * 8 + blockIdx.y, smem_attn);
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// ---------------------------------------------------------------------------------------------
// Fused decode attention + o_proj (+ residual). One launch, two CTA roles:
//   CTAs [0, Hkv*nsplit)        : attention (as above); the last CTA of each KV group bumps sync[0]
//   CTAs [Hkv*nsplit, +n_cta)   : o_proj rows. They are resident from the start, issue the first 16
//                                 weight loads per lane, then wait (bounded spin) until sync[0] == Hkv,
//                                 stage the attention output and finish their dot products.
// This removes one kernel boundary per layer and hides o_proj's launch + first-load latency behind the
// attention. Attention CTAs have the lower block indices, so they are always dispatched first and never
// wait on anything: the o_proj CTAs cannot starve them.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float dot8_attn(const uint4& w, const uint4& x) {
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
    const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 a = unpack_bf16x2(ww[j]), b = unpack_bf16x2(xw[j]);
        acc = fmaf(a.x, b.x, acc);
        acc = fmaf(a.y, b.y, acc);
    }
    return acc;
}

__device__ __forceinline__ void oproj_role(const DecodeAttnParams& p, const OprojParams& o, const int cta,
                                           uint8_t* smem) {
    constexpr int ROWS = 4, UNROLL = 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = cta * 16 + warp * ROWS;
    const int K = o.K;
    int rows[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) rows[r] = min(row0 + r, o.N - 1);
    uint4 w[ROWS][UNROLL];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int cc = lane * 8 + u * 256;
            w[r][u] = (cc < K) ? ld_stream16(o.W + (size_t)rows[r] * o.ldw + cc) : make_uint4(0, 0, 0, 0);
        }
    if (p.finished && *p.finished) return;
    // ---- wait for the merged attention output (bounded: a lost signal degrades the result, never hangs) ----
    if (threadIdx.x == 0) {
        int spins = 0;
        while (ld_acquire_gpu(o.sync) < p.Hkv && ++spins < (1 << 20)) __nanosleep(400);
    }
    __syncthreads();
    bf16* xs = reinterpret_cast<bf16*>(smem);
    for (int c = threadIdx.x * 8; c < K; c += blockDim.x * 8)
        *reinterpret_cast<uint4*>(xs + c) = __ldcg(reinterpret_cast<const uint4*>(p.out + c));
    __syncthreads();
    float acc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r] = 0.f;
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
        const int cc = min(lane * 8 + u * 256, K - 8);
        const uint4 xv = *reinterpret_cast<const uint4*>(xs + cc);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] += dot8_attn(w[r][u], xv);
    }
    for (int c = lane * 8 + UNROLL * 256; (c - lane * 8) < K; c += UNROLL * 256) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const int cc = c + u * 256;
                w[r][u] = (cc < K) ? ld_stream16(o.W + (size_t)rows[r] * o.ldw + cc) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int cc = min(c + u * 256, K - 8);
            const uint4 xv = *reinterpret_cast<const uint4*>(xs + cc);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r] += dot8_attn(w[r][u], xv);
        }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r] = warp_sum(acc[r]);
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const int n = row0 + r;
            if (n < o.N) o.h[n] = f2bf(rbf(acc[r]) + bf2f(o.h[n]));  // o_proj + residual (mq2vl.py:593,645)
        }
    }
    // ---- the last o_proj CTA re-arms the flags for the next launch ----
    __syncthreads();
    if (threadIdx.x == 0) {
        const int c = atomicAdd(o.sync + 1, 1);
        if (c == o.n_cta - 1) {
            o.sync[0] = 0;
            o.sync[1] = 0;
            __threadfence();
        }
    }
}

__global__ void __launch_bounds__(128) attn_oproj_kernel(const DecodeAttnParams p, const OprojParams o) {
    extern __shared__ __align__(16) uint8_t smem_attn[];
    const int n_attn = p.Hkv * p.nsplit;
    if ((int)blockIdx.x < n_attn) attn_decode_role<1>(p, blockIdx.x % p.Hkv, blockIdx.x / p.Hkv, smem_attn);
    else oproj_role(p, o, blockIdx.x - n_attn, smem_attn);
}

int attn_decode(bf16* qkv, bf16* kc, bf16* vc, const int* page_table, int page_size, const int* kv_len,
                const int* rope_pos, const int* finished, const float* inv_freq, int Hq, int Hkv, int nsplit,
                float* part_o, float* part_ml, int* counters, bf16* out, bool pdl, cudaStream_t s) {
    if (page_size != 64 || Hq % Hkv || Hq / Hkv > 8) return -1;
    const bool cluster = nsplit % 8 == 0;
    static SmemAttrOnce once, once_cl;
    if (cluster ? ensure_dyn_smem(once_cl, attn_decode_cluster_kernel, kDecSmem) : ensure_dyn_smem(once, attn_decode_kernel, kDecSmem)) return -2;
    DecodeAttnParams p{};
    p.qkv = qkv; p.kc = kc; p.vc = vc; p.page_table = page_table; p.kv_len = kv_len; p.rope_pos = rope_pos;
    p.finished = finished; p.inv_freq = inv_freq; p.Hq = Hq; p.Hkv = Hkv; p.nsplit = nsplit;
    p.part_o = part_o; p.part_ml = part_ml; p.counters = counters; p.out = out;
    p.scale_log2 = 1.4426950408889634f / sqrtf(128.f);
    count_launch();
    if (launch_kernel(cluster ? attn_decode_cluster_kernel : attn_decode_kernel, dim3(Hkv, nsplit), dim3(128), (size_t)kDecSmem, s, pdl, p) != cudaSuccess) return -3;
    return 0;
}

int attn_decode_batch(bf16* qkv, int qkv_ld, bf16* kc, bf16* vc, const AttnStream* streams, int B, int page_size, const float* inv_freq,
                      int Hq, int Hkv, float* part_o, float* part_ml, int* counters, bf16* out, int out_ld, cudaStream_t s) {
    if (page_size != 64 || Hq % Hkv || Hq / Hkv > 8 || B < 1 || B > kBatchStreams) return -1;
    static SmemAttrOnce once;
    if (ensure_dyn_smem(once, attn_decode_batch_kernel, kDecSmem)) return -2;
    DecodeAttnBatchParams bp{};
    DecodeAttnParams& p = bp.one;
    p.qkv = qkv; p.kc = kc; p.vc = vc; p.inv_freq = inv_freq; p.Hq = Hq; p.Hkv = Hkv;
    p.part_o = part_o; p.part_ml = part_ml; p.counters = counters; p.out = out;
    p.scale_log2 = 1.4426950408889634f / sqrtf(128.f);
    for (int b = 0; b < B; ++b) bp.st[b] = streams[b];
    bp.qkv_ld = qkv_ld; bp.out_ld = out_ld; bp.B = B;
    count_launch();
    return launch_kernel(attn_decode_batch_kernel, dim3(Hkv, 8, 2 * B), dim3(128), (size_t)kDecSmem, s, false, bp) == cudaSuccess ? 0 : -3;
}

// Fused attention + o_proj launch (see attn_oproj_kernel). sync: device int[2], zero-initialised once.
int attn_oproj_decode(bf16* qkv, bf16* kc, bf16* vc, const int* page_table, int page_size, const int* kv_len,
                      const int* rope_pos, const int* finished, const float* inv_freq, int Hq, int Hkv, int nsplit,
                      float* part_o, float* part_ml, int* counters, bf16* attn_out, const bf16* o_w, int o_ldw,
                      int o_N, bf16* h, int* sync, cudaStream_t s) {
    if (page_size != 64 || Hq % Hkv || Hq / Hkv > 8) return -1;
    constexpr int smem = kDecSmem;
    if (Hq * 128 * 2 > smem) return -4;
    static SmemAttrOnce once;
    if (ensure_dyn_smem(once, attn_oproj_kernel, smem)) return -2;
    DecodeAttnParams p{};
    p.qkv = qkv; p.kc = kc; p.vc = vc; p.page_table = page_table; p.kv_len = kv_len; p.rope_pos = rope_pos;
    p.finished = finished; p.inv_freq = inv_freq; p.Hq = Hq; p.Hkv = Hkv; p.nsplit = nsplit;
    p.part_o = part_o; p.part_ml = part_ml; p.counters = counters; p.out = attn_out;
    p.scale_log2 = 1.4426950408889634f / sqrtf(128.f);
    p.done_groups = sync;
    OprojParams o{};
    o.W = o_w; o.ldw = o_ldw; o.N = o_N; o.K = Hq * 128; o.h = h; o.sync = sync; o.n_cta = (o_N + 15) / 16;
    lcc::count_launch();
    attn_oproj_kernel<<<Hkv * nsplit + o.n_cta, 128, smem, s>>>(p, o);
    return 0;
}

}  // namespace lcc
