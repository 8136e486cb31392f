// Decoder prefill attention on tcgen05 + TMEM: causal GQA attention of S new tokens over past+S tokens of the
// paged cache, head_dim 128.  Qwen2VLAttention core, mq2vl.py:572-594 + eager_attention_forward :353-375.
//
// Same structure as the ViT kernel (attention_tc.cu): one CTA = 128 TMEM lanes = 128 packed query rows of one KV
// head, warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 softmax (thread = row).  Differences:
//   * rows are (position, query head of the group) pairs: row r of a tile = position pos0 + r/G, head kvh*G + r%G,
//     so a K/V tile is read once for the G heads that share it.  PT = 128/G positions per tile (G=7: 126 rows used).
//     Q is fetched by ONE 3-D TMA box (64 dims, G heads, PT positions) per 64-dim half, which lands in exactly this
//     row order in the SWIZZLE_128B K-major layout.
//   * a K/V tile = one 64-token page of the cache = two TMA boxes [64 tokens][64 dims] (SWIZZLE_128B): K is a K-major
//     B operand, V an MN-major B operand (N = 128 dims = 2 atoms, K = tokens) - no transposes anywhere.
//   * causal mask per row (key index <= past + position), applied only on tiles that reach the diagonal.
//   * split-KV (blockIdx.z): partial (unnormalised O, m, l) in the format of flash_merge_kernel (attention.cu).
// The tail of the last page beyond past+S is never unmasked; V there must be finite (mrope_kv_write zeroes it).
// TMEM (256 columns): S0 @0, S1 @64, O @128 (128 columns); a tile's P overwrites the first half of its S and is the A operand of P.V.
//
// A thread owns a row, so one CTA has four softmax warps, one per scheduler, and a tile is a serial chain (TMEM load, maximum, 64
// exponentials, TMEM store, MMA): 1.8 us per 64 keys with one CTA per SM. Two CTAs fill each other's gaps: 98 KB of shared memory (two
// slots each for K and V, released apart) and half of the TMEM each: 281 rows over 17 k keys 119 -> 89 us (42 us at the
// tensor rate). Four layers of 24 rows over 64 k keys: 245 us less, of 4 x 115 with 8 splits at most (the keys and values alone: 21 us each).
#include <algorithm>

#include "common.cuh"
#include "gemm.h"
#include "launch.h"
#include "ops.h"
#include "seqmix.h"

namespace lcc {
namespace ptc {
constexpr int D = 128, BM = 128, BN = 64, STAGES = 2;
constexpr int Q_ATOM_BYTES = BM * 128;       // [128 rows][64 bf16]
constexpr int Q_BYTES = 2 * Q_ATOM_BYTES;
constexpr int KV_ATOM_BYTES = BN * 128;      // [64 tokens][64 bf16]
constexpr int KV_BYTES = 2 * KV_ATOM_BYTES;  // one K or V tile
constexpr int OFF_Q = 0;
constexpr int OFF_K = OFF_Q + Q_BYTES;
constexpr int OFF_V = OFF_K + STAGES * KV_BYTES;
constexpr int OFF_BAR = OFF_V + STAGES * KV_BYTES;
constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;
constexpr int COL_S = 0, COL_O = 2 * BN, TMEM_COLS = 256;
constexpr int MAX_SPLIT = 32;
constexpr float RESCALE_THRESHOLD = 8.f;
}  // namespace ptc

struct PrefillTcParams {
    bf16* out;
    int o_ld;
    int Hkv, G, PT;
    float scale_log2;
    float* part_o;   // per stream, from its part_row on: [nsplit, Hkv, S*G, 128] unnormalised fp32
    float* part_ml;  // the same: [nsplit, Hkv, S*G, 2]    (raw max, sum)
    PrefillStreams ps;
};

__device__ __forceinline__ float ex2_ftz_p(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// LOCAL: the attention of the hybrid models (plain masks): fp32 queries, rounded to bf16 as they are staged, a window and / or chunks, a sink
// in the softmax, gated output. Their pages are not cleared behind the newest token, and a tile may begin before the first visible
// key: what P = 0 would meet there is zeroed in the staged V tile. (1024 rows of 16 heads on 2, window 1024: 24 us; mma.sync tiles of one
// head and 64 rows, eight of which staged the same keys, took 80. 2048 rows in chunks of 1024: 24 for 102.) A prompt has few tiles per
// CTA, so most of this kernel's code runs once, and fetching it is what it costs: with the staging of Q and the gated output unrolled
// and whole divisions in it, one tile took 36 us for 11.
struct PrefillLocal {
    const float* q;       // [S, Hq, 128]
    SeqPos pos;
    const bf16* gate;
    int ld_gate, chunk, window;
    bool no_sink, gate_channel;
    __device__ __forceinline__ int first_key(int p) const {
        const int lo = chunk > 0 ? p / chunk * chunk : 0;
        return window > 0 ? max(lo, p - window + 1) : lo;
    }
};

template <bool LOCAL>
__global__ void __launch_bounds__(192, 2)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ PrefillTcParams p, const PrefillLocal lp) {
    using namespace ptc;
    if (LOCAL && lp.pos.finished && *lp.pos.finished) return;
    int b = 0, split = LOCAL ? 0 : blockIdx.z;
    if (!LOCAL)
        while (split >= p.ps.st[b].nsplit) split -= p.ps.st[b++].nsplit;
    const PrefillStream& st = p.ps.st[b];
    const int kvh = blockIdx.y;
    const bool parts = !LOCAL && st.nsplit > 1;
    // (with a window or chunks the last rows see the most keys: they start first)
    const int pos0 = (LOCAL ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * p.PT, S = st.S;
    const int past = LOCAL && lp.pos.kv_len ? *lp.pos.kv_len : st.past;
    if (pos0 >= S) return;
    const int npos = min(p.PT, S - pos0);
    const int rows_used = npos * p.G;
    const int rows_total = S * p.G;
    const int row_base = pos0 * p.G;  // packed row index of this tile's row 0
    // KV tiles this CTA needs: keys 0 .. past + last position (causal), restricted to its split
    const int n_tiles = (past + pos0 + npos + BN - 1) / BN;
    int tile_lo = 0, tile_hi = n_tiles;
    const int key0 = LOCAL ? lp.first_key(past + pos0) : 0, key1 = past + pos0 + npos;   // no row of this CTA sees a key outside [key0, key1)
    if (LOCAL) tile_lo = key0 / BN;
    if (parts) {
        const int tiles_total = (past + S + BN - 1) / BN;
        const int tps = (tiles_total + st.nsplit - 1) / st.nsplit;
        tile_lo = split * tps;
        tile_hi = min(n_tiles, tile_lo + tps);
        if (tile_lo >= tile_hi) {  // nothing for this split: neutral partial
            chain_wait();          // (the kernel in front may be the merge of other streams' partials, in the same scratch)
            float* ml = p.part_ml + (st.part_row + ((size_t)split * p.Hkv + kvh) * rows_total + row_base) * 2;
            for (int i = threadIdx.x; i < rows_used; i += blockDim.x) {
                ml[i * 2] = -INFINITY;
                ml[i * 2 + 1] = 0.f;
            }
            return;
        }
    }
    const int T = tile_hi - tile_lo;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;
    uint64_t* k_empty = k_full + STAGES;
    uint64_t* v_full = k_empty + STAGES;
    uint64_t* v_empty = v_full + STAGES;
    uint64_t* s_full = v_empty + STAGES;
    uint64_t* p_full = s_full + 2;
    uint64_t* pv_done = p_full + 1;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(pv_done + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == 0 && lane == 0) {
        if (!LOCAL) prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
        mbar_init(q_full, LOCAL ? 4 : 1);
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) mbar_init(&s_full[i], 1);
        mbar_init(p_full, 4);
        mbar_init(pv_done, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_holder, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    chain_begin();

    if (warp == 0) {
        // ===================== TMA producer =====================
        if (lane == 0) {
            // the box is always (64, G, PT): rows beyond the stream's are the next one's, or zero-filled but still counted; nothing of them is kept
            if (!LOCAL) {
                mbar_arrive_expect_tx(q_full, 2u * 64u * (uint32_t)p.G * (uint32_t)p.PT * 2u);
                tma_load_3d(smem + OFF_Q, &tmap_q, q_full, 0, kvh * p.G, st.row0 + pos0);
                tma_load_3d(smem + OFF_Q + Q_ATOM_BYTES, &tmap_q, q_full, 64, kvh * p.G, st.row0 + pos0);
            }
            const int* page_table = st.page_table;
            for (int i = 0; i < T; ++i) {
                const int st = i % STAGES;
                const uint32_t free = ((i / STAGES) & 1) ^ 1;
                const int page = page_table[tile_lo + i];
                const int row = (page * p.Hkv + kvh) * BN;
                uint8_t* sk = smem + OFF_K + st * KV_BYTES;
                uint8_t* sv = smem + OFF_V + st * KV_BYTES;
                mbar_wait(&k_empty[st], free);
                mbar_arrive_expect_tx(&k_full[st], KV_BYTES);
                tma_load_2d(sk, &tmap_k, &k_full[st], 0, row);
                tma_load_2d(sk + KV_ATOM_BYTES, &tmap_k, &k_full[st], 64, row);
                mbar_wait(&v_empty[st], free);
                mbar_arrive_expect_tx(&v_full[st], KV_BYTES);
                tma_load_2d(sv, &tmap_v, &v_full[st], 0, row);
                tma_load_2d(sv + KV_ATOM_BYTES, &tmap_v, &v_full[st], 64, row);
            }
        }
    } else if (warp == 1) {
        // ===================== MMA issuer =====================
        constexpr uint32_t idesc_qk = make_idesc_bf16(BM, BN);
        constexpr uint32_t idesc_pv = make_idesc_bf16(BM, D) | (1u << 16);  // B (= V) is MN-major
        const uint32_t q_addr = smem_u32(smem + OFF_Q);
        auto issue_qk = [&](int i) {
            const int st = i % STAGES, b = i & 1;
            mbar_wait(&k_full[st], (i / STAGES) & 1);
            if (i >= 2) mbar_wait(pv_done, i & 1);   // P of tile i - 2 lies where S of tile i goes (the MMA of tile i - 1 is yet to be issued)
            tc_fence_after();
            if (lane == 0) {
                const uint32_t k_addr = smem_u32(smem + OFF_K + st * KV_BYTES);
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const uint64_t dq = make_sw128_kmajor_desc(q_addr + a * Q_ATOM_BYTES);
                    const uint64_t dk = make_sw128_kmajor_desc(k_addr + a * KV_ATOM_BYTES);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16_ss(tmem_base + COL_S + b * BN, dq + (uint64_t)(2 * k), dk + (uint64_t)(2 * k), idesc_qk,
                                     (a | k) ? 1u : 0u);
                }
                umma_commit(&k_empty[st]);
                umma_commit(&s_full[b]);
            }
            __syncwarp();
        };
        mbar_wait(q_full, 0);
        issue_qk(0);
        for (int i = 0; i < T; ++i) {
            if (i + 1 < T) issue_qk(i + 1);
            mbar_wait(&v_full[i % STAGES], (i / STAGES) & 1);
            if (LOCAL) {
                const int k0 = (tile_lo + i) * BN, cut_lo = max(key0 - k0, 0), cut_hi = min(key1 - k0, BN);   // the tile's rows in [cut_lo, cut_hi) count
                if (cut_lo > 0 || cut_hi < BN) {
                    uint8_t* sv = smem + OFF_V + (i % STAGES) * KV_BYTES;
                    for (int u = lane; u < BN * 16; u += 32) {
                        const int r = u >> 4, c = u & 15;   // 16 bytes of token row r: eight in each 64-channel half
                        if (r < cut_lo || r >= cut_hi)
                            *reinterpret_cast<uint4*>(sv + (c >> 3) * KV_ATOM_BYTES + r * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                }
            }
            mbar_wait(p_full, i & 1);
            tc_fence_after();
            if (lane == 0) {
                const int st = i % STAGES;
                const uint32_t v_addr = smem_u32(smem + OFF_V + st * KV_BYTES);
#pragma unroll
                for (int ks = 0; ks < BN / 16; ++ks) {  // 16 tokens per MMA: +32 B in P rows, +16 token rows in V
                    const uint64_t dv = make_sw128_mnmajor_desc(v_addr + ks * (16 * 128), KV_ATOM_BYTES);
                    umma_bf16_ts(tmem_base + COL_O, tmem_base + COL_S + (i & 1) * BN + ks * 8, dv, idesc_pv, (i | ks) ? 1u : 0u);
                }
                umma_commit(&v_empty[st]);
                umma_commit(pv_done);
            }
            __syncwarp();
        }
    } else {
        // ===================== softmax / correction / epilogue =====================
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const bool row_ok = row < rows_used;
        const int rpos = row / p.G, rg = row - rpos * p.G;
        const int lim = row_ok ? past + pos0 + rpos : -1;  // last visible key index; invalid rows see nothing
        const int first = LOCAL && row_ok ? lp.first_key(lim) : 0;
        float m_used = -INFINITY, l = 0.f;
        if (LOCAL) {
            if (!lp.no_sink && row_ok) { m_used = 0.f; l = 1.f; }   // the sink (a score of 0 without a value) starts the sum
            // queries: a warp takes its 32 rows one by one, four channels per lane, into the K-major 128-byte-swizzled tile
            const int Hq = p.Hkv * p.G, c = lane & 15;   // lanes 0..15: channels 0..63 in 8-byte pieces
            uint8_t* sq = smem + OFF_Q + (lane >> 4) * Q_ATOM_BYTES;
            int qg = quarter * 32 % p.G;
            const float* src = lp.q + ((size_t)(pos0 + quarter * 32 / p.G) * Hq + kvh * p.G + qg) * D + lane * 4;
            for (int r0 = quarter * 32; r0 < quarter * 32 + 32; r0 += 8) {
                float4 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[j] = r0 + j < rows_used ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const bool next = ++qg == p.G;   // the next position's first head of this group
                    src += next ? (Hq - p.G + 1) * D : D;
                    qg = next ? 0 : qg;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<uint2*>(sq + (r0 + j) * 128 + (((c >> 1) ^ j) << 4) + (c & 1) * 8) =
                        make_uint2(pack_bf16x2(v[j].x, v[j].y), pack_bf16x2(v[j].z, v[j].w));
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(q_full);
        }
        for (int i = 0; i < T; ++i) {
            const int b = i & 1;
            mbar_wait(&s_full[b], (i >> 1) & 1);
            tc_fence_after();
            uint32_t v[2][32];
            tmem_ld_32x32b_x32(tmem_base + COL_S + b * BN + lane_off, v[0]);
            tmem_ld_32x32b_x32(tmem_base + COL_S + b * BN + 32 + lane_off, v[1]);
            tmem_ld_wait();

            const int kbase = (tile_lo + i) * BN;
            if (__any_sync(0xffffffffu, kbase + BN - 1 > lim || (LOCAL && kbase < first))) {  // tile reaches the diagonal (or the first key) of some row of this warp
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (kbase + c * 32 + j > lim || (LOCAL && kbase + c * 32 + j < first)) v[c][j] = __float_as_uint(-INFINITY);
            }
            float mx[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) mx[j] = __uint_as_float(v[0][j]);
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (c > 0 || j >= 8) mx[j & 7] = fmaxf(mx[j & 7], __uint_as_float(v[c][j]));
            float mt = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])));
            mt *= p.scale_log2;
            const bool need = mt > m_used + RESCALE_THRESHOLD;  // false while the row has seen no key (mt = -inf)
            const bool any_need = __any_sync(0xffffffffu, need);
            float alpha = 1.f;
            if (need) {
                alpha = ex2_ftz_p(m_used - mt);  // 0 the first time
                m_used = mt;
                l *= alpha;
            }
            const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;  // all-masked so far: p = ex2(-inf) = 0, not NaN
            uint32_t pk[BN / 2];
            float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    const float p0 = ex2_ftz_p(fmaf(__uint_as_float(v[c][j]), p.scale_log2, -m_sub));
                    const float p1 = ex2_ftz_p(fmaf(__uint_as_float(v[c][j + 1]), p.scale_log2, -m_sub));
                    ls[(j >> 1) & 3] += p0 + p1;
                    pk[c * 16 + (j >> 1)] = pack_bf16x2(p0, p1);
                }
            l += (ls[0] + ls[1]) + (ls[2] + ls[3]);

            if (i > 0) {
                mbar_wait(pv_done, (i - 1) & 1);  // P_{i-1} V_{i-1} retired: O up to date
                tc_fence_after();
                if (any_need) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t o32[32];
                        tmem_ld_32x32b_x32(tmem_base + COL_O + c * 32 + lane_off, o32);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) o32[j] = __float_as_uint(__uint_as_float(o32[j]) * alpha);
                        tmem_st_32x32b_x32(tmem_base + COL_O + c * 32 + lane_off, o32);
                    }
                    tmem_st_wait();
                }
            }
            // P row -> TMEM, over the S it came from: word j = keys (2j, 2j+1), lane = row (the A-operand layout of kind::f16)
            tmem_st_32x32b_x32(tmem_base + COL_S + b * BN + lane_off, pk);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        const bf16* gate = LOCAL && lp.gate && row_ok
                               ? lp.gate + (size_t)(pos0 + rpos) * lp.ld_gate + (lp.gate_channel ? (size_t)(kvh * p.G + rg) * D : (size_t)(kvh * p.G + rg)) : nullptr;
        // (a denominator of 1 to 2 whatever x is, so that the short reciprocal has its range; one Newton step makes up for its error)
        auto sigmoid = [](float x) {
            const float t = expf(-fabsf(x)), d = 1.f + t, r = __fdividef(1.f, d);
            return (x < 0.f ? t : 1.f) * fmaf(r, fmaf(-d, r, 1.f), r);
        };
        mbar_wait(pv_done, (T - 1) & 1);
        tc_fence_after();
        if (parts) {
            const size_t prow = st.part_row + ((size_t)split * p.Hkv + kvh) * rows_total + row_base + row;
            float* dst = p.part_o + prow * D;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t o32[32];
                tmem_ld_32x32b_x32(tmem_base + COL_O + c * 32 + lane_off, o32);
                tmem_ld_wait();
                if (row_ok) {
#pragma unroll
                    for (int g4 = 0; g4 < 8; ++g4)
                        *reinterpret_cast<uint4*>(dst + c * 32 + g4 * 4) =
                            make_uint4(o32[g4 * 4], o32[g4 * 4 + 1], o32[g4 * 4 + 2], o32[g4 * 4 + 3]);
                }
            }
            if (row_ok) {
                p.part_ml[prow * 2] = (m_used == -INFINITY) ? -INFINITY : m_used / p.scale_log2;
                p.part_ml[prow * 2 + 1] = l;
            }
        } else {
            float inv = l > 0.f ? 1.f / l : 0.f;
            const bool wide_gate = LOCAL && gate && lp.gate_channel;
            if (LOCAL && gate && !wide_gate) inv *= sigmoid(bf2f(*gate));
            bf16* dst = p.out + (size_t)(st.row0 + pos0 + rpos) * p.o_ld + (size_t)(kvh * p.G + rg) * D;
#pragma unroll LOCAL ? 1 : 4
            for (int c = 0; c < 4; ++c) {
                uint32_t o32[32];
                tmem_ld_32x32b_x32(tmem_base + COL_O + c * 32 + lane_off, o32);
                uint4 z[4];
                if (wide_gate) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) z[j] = *reinterpret_cast<const uint4*>(gate + c * 32 + j * 8);
                }
                tmem_ld_wait();
                if (wide_gate) {
#pragma unroll
                    for (int g8 = 0; g8 < 4; ++g8) {
                        const uint32_t zw[4] = {z[g8].x, z[g8].y, z[g8].z, z[g8].w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float2 f = unpack_bf16x2(zw[j]);
                            o32[g8 * 8 + 2 * j] = __float_as_uint(__uint_as_float(o32[g8 * 8 + 2 * j]) * sigmoid(f.x));
                            o32[g8 * 8 + 2 * j + 1] = __float_as_uint(__uint_as_float(o32[g8 * 8 + 2 * j + 1]) * sigmoid(f.y));
                        }
                    }
                }
                if (row_ok) {
#pragma unroll
                    for (int g8 = 0; g8 < 4; ++g8) {
                        uint4 o;
                        o.x = pack_bf16x2(__uint_as_float(o32[g8 * 8 + 0]) * inv, __uint_as_float(o32[g8 * 8 + 1]) * inv);
                        o.y = pack_bf16x2(__uint_as_float(o32[g8 * 8 + 2]) * inv, __uint_as_float(o32[g8 * 8 + 3]) * inv);
                        o.z = pack_bf16x2(__uint_as_float(o32[g8 * 8 + 4]) * inv, __uint_as_float(o32[g8 * 8 + 5]) * inv);
                        o.w = pack_bf16x2(__uint_as_float(o32[g8 * 8 + 6]) * inv, __uint_as_float(o32[g8 * 8 + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + c * 32 + g8 * 8) = o;
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// Key ranges of one stream's attention, up to two CTAs per SM, with at least 8 tiles per range and partials that fit into the caller's scratch. A tile
// takes 0.8 us with one CTA per SM and 1.15 with two; the partials cost a launch of 3.5 us and are written and read once. (281 rows over 4 k keys: 4
// splits; 24 rows over 64 k: 32.) Filling the places whatever the range is cost 400 to 640 rows behind 600 to 1500 tokens up to a quarter:
// 400 and 600 rows behind 600 | 1000 | 3000 tokens 17.4 | 22.3 | 47.5 and 20.1 | 24.6 | 50.3 us unsplit, 21.7 | 25.4 | 34.4 and 25.6 | 28.6 |
// 45.8 with every place taken. Other streams of the launch do not count: a stream has the same bits whoever its neighbours are.
int attn_prefill_tc_splits(int S, int past, int Hq, int Hkv, size_t part_capacity_rows, int num_sms) {
    using namespace ptc;
    const int PT = BM / (Hq / Hkv), ctas = (S + PT - 1) / PT * Hkv, kv_tiles = (past + S + BN - 1) / BN;
    const size_t rows = (size_t)Hq * S;
    const int most = (int)std::min((size_t)std::min({2 * num_sms / ctas, MAX_SPLIT, kv_tiles / 8}), part_capacity_rows / rows);
    int nsplit = 1;
    double best = 0.8 * kv_tiles;   // (more CTAs than SMs are never split)
    for (int n = 2; n <= most; ++n) {
        const double us = (double)kv_tiles / n * (ctas * n > num_sms ? 1.15 : 0.8) + 3.5 + (double)rows * n * 1024 / 6.5e6;
        if (us < best) { best = us; nsplit = n; }
    }
    return nsplit;
}

// q: rotated rows of the fused qkv buffer [ps.rows, >= Hq*128] (row stride q_ld); kc/vc: one layer of the page pool
// [pages, Hkv, 64, 128]. Streams with nsplit > 1 leave partials, which the caller merges.
int attn_prefill_tc(const bf16* q, int q_ld, const bf16* kc, const bf16* vc, const PrefillStreams& ps, int Hq, int Hkv, bf16* out, int o_ld,
                    float* part_o, float* part_ml, cudaStream_t s) {
    using namespace ptc;
    const int G = Hq / Hkv, PT = BM / G;
    int q_tiles = 0, slices = 0;
    for (int b = 0; b < ps.n; ++b) {
        q_tiles = std::max(q_tiles, (ps.st[b].S + PT - 1) / PT);
        slices += ps.st[b].nsplit;
    }
    CUtensorMap tq, tk, tv;
    if (make_tmap_bf16_3d_sw128(&tq, q, D, Hq, ps.rows, D, q_ld, G, PT)) return -10;
    const int64_t pool_rows = (int64_t)1 << 31;  // page ids come from the page table; no meaningful row bound here
    if (make_tmap_bf16_2d_box(&tk, kc, pool_rows, D, D, 64, BN, false)) return -11;
    if (make_tmap_bf16_2d_box(&tv, vc, pool_rows, D, D, 64, BN, false)) return -11;
    static SmemAttrOnce once;
    if (ensure_dyn_smem(once, attn_prefill_tc_kernel<false>, SMEM_BYTES)) return -12;
    const PrefillTcParams p{out, o_ld, Hkv, G, PT, 1.4426950408889634f / sqrtf((float)D), part_o, part_ml, ps};
    lcc::count_launch();
    chained(attn_prefill_tc_kernel<false>, dim3(q_tiles, Hkv, slices), 192, SMEM_BYTES, s)(tq, tk, tv, p, PrefillLocal{});
    return 0;
}

bool attn_local_tc_takes(const float* q, const void* k_pages, const void* v_pages, int page_size, const void* gate, int ld_gate, const void* out,
                         int ld_out, int Hq, int G, int D, int DV, int ld_v, const float* sink, const AttnOpts& opt) {
    const bool plain = !sink && opt.softcap <= 0.f && opt.keep_first <= 0 && opt.maps == 1 && !opt.raw && !opt.bias;
    const bool wide_gate = gate && opt.gate_channel;
    return plain && D == ptc::D && DV == ptc::D && ld_v == ptc::D && page_size == ptc::BN && Hq / G <= ptc::BM && ld_out % 8 == 0 && (!wide_gate || ld_gate % 8 == 0) &&
           (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out | (wide_gate ? (uintptr_t)gate : 0)) & 15) == 0;
}

int attn_local_tc(const float* q, const void* k_pages, const void* v_pages, const int* page_table, const void* gate, int ld_gate, void* out,
                  int ld_out, int S, int Hq, int G, int chunk, float scale, SeqPos pos, cudaStream_t s, const AttnOpts& opt) {
    using namespace ptc;
    PrefillTcParams p{};
    p.out = (bf16*)out; p.o_ld = ld_out; p.Hkv = G; p.G = Hq / G; p.PT = BM / p.G;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.ps.n = 1; p.ps.rows = S;
    p.ps.st[0].nsplit = 1;
    p.ps.st[0].page_table = page_table; p.ps.st[0].S = S; p.ps.st[0].past = pos.past;
    const PrefillLocal lp{q, pos, (const bf16*)gate, ld_gate, chunk > 0 ? chunk : 0, opt.window > 0 ? opt.window : 0, opt.no_sink, opt.gate_channel};
    CUtensorMap tk, tv;
    const int64_t pool_rows = (int64_t)1 << 31;  // (as above)
    if (make_tmap_bf16_2d_box(&tk, k_pages, pool_rows, D, D, 64, BN, false) || make_tmap_bf16_2d_box(&tv, v_pages, pool_rows, D, D, 64, BN, false)) return -100;
    static SmemAttrOnce once;
    if (ensure_dyn_smem(once, attn_prefill_tc_kernel<true>, SMEM_BYTES)) return -100;
    count_launch();
    attn_prefill_tc_kernel<true><<<dim3((S + p.PT - 1) / p.PT, G), 192, SMEM_BYTES, s>>>(tk, tk, tv, p, lp);
    return cudaGetLastError() == cudaSuccess ? 0 : -100;
}

}  // namespace lcc
