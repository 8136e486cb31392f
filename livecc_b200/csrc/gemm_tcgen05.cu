// Persistent, warp-specialised tcgen05 GEMM for sm_100a:
//     C[M,N] (bf16) = epilogue( A[M,K] (bf16, K-major) x B[N,K]^T (bf16, K-major, nn.Linear layout) )
//
// Used for every M >= 16 contraction of the LiveCC hot path: ViT patch-embed / qkv / proj /
// fc1 / fc2 / merger (mq2vl.py:304-337,385-458) and the decoder prefill projections
// (mq2vl.py:491-504,539-594, lm_head :1437).
//
// Structure (one CTA per SM, 384 threads):
//   warp 0      : TMA producer  (cp.async.bulk.tensor, SWIZZLE_128B tiles, mbarrier complete_tx)
//   warp 1      : MMA issuer    (one elected lane issues tcgen05.mma, fp32 accumulators in TMEM)
//   warp 2      : TMEM allocator
//   warps 4..11 : epilogue      (tcgen05.ld 32x32b -> registers -> fused epilogue -> bf16 stores);
//                 warp w reads TMEM lane quarter w%4 and the column half (w-4)/4 of the tile
// Pipelines: smem ring (full/empty mbarriers, STAGES deep) between TMA and MMA; a 2-deep TMEM
// accumulator ring (tmem_full/tmem_empty) between MMA and epilogue so the epilogue of tile i
// overlaps the main loop of tile i+1.
//
// The fused epilogues reproduce the reference's bf16 rounding points (one torch op = one rounding).
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "gemm.h"
#include "launch.h"

namespace lcc {

static constexpr int BLOCK_M = 128;
static constexpr int BLOCK_K = 64;   // 64 bf16 = 128 B = one SWIZZLE_128B row
static constexpr int UMMA_K = 16;

// The N tile is a RUN-TIME value (multiple of 16, 32..256): the 148 SMs are filled by choosing the tile width per
// shape (e.g. ViT qkv (1024 x 3840): 224 -> 8 x 18 = 144 tiles = one full wave; 256 or 128 leave a mostly empty
// second wave). Everything that depended on BLOCK_N (stage size, ring depth, TMEM columns, instruction descriptor,
// epilogue chunking) is derived from it on the host and passed in.
static constexpr int MAX_STAGES = 8;
static constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2;
struct GemmTile {
    int bn;          // N tile
    int stages;      // smem ring depth
    int tmem_cols;   // power of two >= two accumulators (+16 when the last 32-column epilogue chunk is half used)
    uint32_t idesc;  // tcgen05 instruction descriptor (M = 128, N = bn)
    int smem_bytes;
};
static GemmTile make_tile(int bn, bool pair = false) {
    GemmTile t;
    t.bn = bn;
    const int stage_bytes = A_BYTES + (pair ? bn / 2 : bn) * BLOCK_K * 2;
    t.stages = (227 * 1024 - 1024 - 256) / stage_bytes;
    if (t.stages > MAX_STAGES) t.stages = MAX_STAGES;
    int cols = 2 * bn + ((bn & 31) ? 16 : 0);
    t.tmem_cols = 32;
    while (t.tmem_cols < cols) t.tmem_cols <<= 1;
    t.idesc = make_idesc_bf16(pair ? 2 * BLOCK_M : BLOCK_M, bn);
    t.smem_bytes = t.stages * stage_bytes + 1024 /*align slack*/ + 256 /*barriers*/;
    return t;
}

__device__ __forceinline__ float quick_gelu_bf16(float x) {
    // ACT2FN["quick_gelu"]: input * sigmoid(1.702 * input), every op rounded to bf16
    // (SP/transformers/activations.py:117-123).
    float t1 = rbf(1.702f * x);
    float t2 = rbf(__fdividef(1.0f, 1.0f + __expf(-t1)));
    return rbf(x * t2);
}
__device__ __forceinline__ float gelu_erf_bf16(float x) {
    return rbf(0.5f * x * (1.0f + erff(x * 0.70710678118654752440f)));
}
__device__ __forceinline__ float silu_bf16(float x) { return rbf(__fdividef(x, 1.0f + __expf(-x))); }

// Fused epilogue of a warp's 32 x 32 chunk of accumulators. Tensor memory gives a thread one row: v = the fp32 bits of columns [col0, col0 + 32) of
// row row0 + lane. Bias, activation and rounding happen there; four lanes then exchange their rows' 16-byte pieces, so that a store (and
// a load of the residual) covers 64 bytes of 8 rows instead of 16 of 32, half a sector each. Bias and residual are fetched while the accumulators
// arrive. Columns >= tile_end belong to the next tile (or are padding) and are dropped. Where K is short this is what a product costs: with a
// row's pieces stored by its own thread 8192 x 5120 x 1280 took 111 us, now 96, and 1024 x 1280 x 1280 14.7, now 11.3.
template <int EPI> struct RowEpi {
    static constexpr bool kBias = EPI == EPI_BIAS || EPI == EPI_BIAS_QUICKGELU || EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_RESIDUAL;
    static constexpr bool kResidual = EPI == EPI_RESIDUAL || EPI == EPI_BIAS_RESIDUAL;
};
struct EpiFetch { uint4 bias[4], res[4]; };

template <int EPI>
__device__ __forceinline__ void epilogue_fetch(EpiFetch& f, int M, int row0, int lane, int col0, int tile_end, const bf16* __restrict__ bias,
                                               const bf16* residual, int ldr) {
    if (RowEpi<EPI>::kBias) {
#pragma unroll
        for (int g = 0; g < 4; ++g) f.bias[g] = col0 + g * 8 < tile_end ? *reinterpret_cast<const uint4*>(bias + col0 + g * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
    if (RowEpi<EPI>::kResidual) {
        const int col = col0 + (lane & 3) * 8;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int row = row0 + (lane & ~3) + k;
            f.res[k] = row < M && col < tile_end ? *reinterpret_cast<const uint4*>(residual + (size_t)row * ldr + col) : make_uint4(0u, 0u, 0u, 0u);
        }
    }
}

// lanes l and l ^ bit exchange: the lane with the bit clear gives b for the other's a
__device__ __forceinline__ void swap_pieces(uint4& a, uint4& b, int bit, int lane) {
    const bool up = lane & bit;
    auto word = [&](uint32_t& x, uint32_t& y) {
        const uint32_t r = __shfl_xor_sync(0xffffffffu, up ? x : y, bit);
        if (up) x = r; else y = r;
    };
    word(a.x, b.x); word(a.y, b.y); word(a.z, b.z); word(a.w, b.w);
}
// p[i] of lane 4 m + k becomes p[k] of lane 4 m + i
__device__ __forceinline__ void quad_transpose(uint4 (&p)[4], int lane) {
    swap_pieces(p[0], p[1], 1, lane); swap_pieces(p[2], p[3], 1, lane);
    swap_pieces(p[0], p[2], 2, lane); swap_pieces(p[1], p[3], 2, lane);
}

// the logits' cap, its inverse and the scale ride in the slots of the residual's stride and the bias, which they have not (set_logit_slots)
struct LogitSlots { float cap, inv_cap, scale; };
__device__ __forceinline__ LogitSlots logit_slots(const bf16* bias, int ldr) {
    const uint64_t b = reinterpret_cast<uint64_t>(bias);
    return {__int_as_float(ldr), __uint_as_float((uint32_t)b), __uint_as_float((uint32_t)(b >> 32))};
}

template <int EPI>
__device__ __forceinline__ void epilogue_chunk(const uint32_t (&v)[32], const EpiFetch& f, bf16* C, int ldc, int M, int row0, int lane, int col0,
                                               int tile_end, int ks, const bf16* __restrict__ bias, const bf16* residual,
                                               int ldr) {
    if (EPI == EPI_PARTIAL_F32 || EPI == EPI_LOGITS_F32) {
        // fp32 partial tile of split ks: P[ks][row][col] (C is the partial buffer, ldc == N)
        float* base = reinterpret_cast<float*>(C) + (size_t)ks * M * (size_t)ldc;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint4 p[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) p[g] = make_uint4(v[h * 16 + g * 4], v[h * 16 + g * 4 + 1], v[h * 16 + g * 4 + 2], v[h * 16 + g * 4 + 3]);
            quad_transpose(p, lane);
            const int col = col0 + h * 16 + (lane & 3) * 4;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int row = row0 + (lane & ~3) + k;
                if (row < M && col < tile_end) {
                    if (EPI == EPI_LOGITS_F32) {
                        const LogitSlots l = logit_slots(bias, ldr);
                        auto store = [&](uint32_t x) {
                            const float y = __uint_as_float(x);
                            return __float_as_uint((l.cap > 0.f ? l.cap * tanhf(y * l.inv_cap) : y) * l.scale);
                        };
                        p[k] = make_uint4(store(p[k].x), store(p[k].y), store(p[k].z), store(p[k].w));
                    }
                    *reinterpret_cast<uint4*>(base + (size_t)row * ldc + col) = p[k];
                }
            }
        }
    } else if (EPI == EPI_SWIGLU || EPI == EPI_CLAMP_GLU) {
        // Weight rows are interleaved in 32-row groups: 16 gate rows then the 16
        // matching up rows. EPI_SWIGLU: out[j] = bf16(silu_bf16(bf16 gate) * bf16 up)  (mq2vl.py:503). EPI_CLAMP_GLU: the activation runs
        // in fp32 on the accumulators and is rounded once; the clamp rides in the (otherwise unused) residual stride as float bits, the
        // sigmoid's slope and the offset of the up half in the (otherwise unused) bias pointer's bits.
        const float limit = __int_as_float(ldr);
        const unsigned long long pb = (unsigned long long)bias;
        const float alpha = __uint_as_float((unsigned)(pb & 0xffffffffull)), up_bias = __uint_as_float((unsigned)(pb >> 32));
        uint32_t o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float y[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float g0 = __uint_as_float(v[2 * j + e]), u0 = __uint_as_float(v[16 + 2 * j + e]);
                if (EPI == EPI_SWIGLU) {
                    y[e] = silu_bf16(rbf(g0)) * rbf(u0);
                } else {
                    const float g = fminf(g0, limit), u = fminf(fmaxf(u0, -limit), limit);
                    y[e] = g / (1.f + __expf(-alpha * g)) * (u + up_bias);
                }
            }
            o[j] = pack_bf16x2(y[0], y[1]);
        }
        uint4 p0 = make_uint4(o[0], o[1], o[2], o[3]), p1 = make_uint4(o[4], o[5], o[6], o[7]);
        swap_pieces(p0, p1, 1, lane);   // two lanes: 32 bytes of one row, then of the other
        const int row = row0 + (lane & ~1), col = ((col0 >> 5) << 4) + (lane & 1) * 8;
        if (col0 < tile_end) {  // BLOCK_N % 32 == 0 for these epilogues: whole chunks only
            if (row < M) *reinterpret_cast<uint4*>(C + (size_t)row * ldc + col) = p0;
            if (row + 1 < M) *reinterpret_cast<uint4*>(C + (size_t)(row + 1) * ldc + col) = p1;
        }
    } else {
        uint4 p[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {  // 4 groups of 8 columns (16 B of bf16 each)
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(v[g * 8 + j]);
            if (RowEpi<EPI>::kBias) {
                const uint32_t bw[4] = {f.bias[g].x, f.bias[g].y, f.bias[g].z, f.bias[g].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 b = unpack_bf16x2(bw[j]);
                    x[2 * j] += b.x;
                    x[2 * j + 1] += b.y;
                }
            }
            if (EPI == EPI_RELU2) {
#pragma unroll
                for (int j = 0; j < 8; ++j) { x[j] = fmaxf(x[j], 0.f); x[j] *= x[j]; }
            }
            if (EPI == EPI_SIGMOID_GATE) {
                const int row = row0 + lane, col = col0 + g * 8;
                const uint4 gg = row < M && col < tile_end ? *reinterpret_cast<const uint4*>(residual + (size_t)row * ldr + col) : make_uint4(0u, 0u, 0u, 0u);
                const uint32_t gw[4] = {gg.x, gg.y, gg.z, gg.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 s = unpack_bf16x2(gw[j]);
                    x[2 * j] = __fdividef(x[2 * j], 1.f + __expf(-s.x));
                    x[2 * j + 1] = __fdividef(x[2 * j + 1], 1.f + __expf(-s.y));
                }
            }
            if (EPI == EPI_GELU_ERF) {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = 0.5f * x[j] * (1.f + erff(x[j] * 0.7071067811865476f));
            }
            if (EPI == EPI_GELU_TANH) {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = 0.5f * x[j] * (1.f + tanhf(0.7978845608028654f * (x[j] + 0.044715f * x[j] * x[j] * x[j])));
            }
            if (EPI == EPI_BIAS_QUICKGELU) {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = quick_gelu_bf16(rbf(x[j]));
            }
            if (EPI == EPI_BIAS_GELU) {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = gelu_erf_bf16(rbf(x[j]));
            }
            p[g] = make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
        }
        quad_transpose(p, lane);
        const int col = col0 + (lane & 3) * 8;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int row = row0 + (lane & ~3) + k;
            if (RowEpi<EPI>::kResidual) {
                const uint32_t aw[4] = {p[k].x, p[k].y, p[k].z, p[k].w}, rw[4] = {f.res[k].x, f.res[k].y, f.res[k].z, f.res[k].w};
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 a = unpack_bf16x2(aw[j]), r = unpack_bf16x2(rw[j]);
                    o[j] = pack_bf16x2(a.x + r.x, a.y + r.y);
                }
                p[k] = make_uint4(o[0], o[1], o[2], o[3]);
            }
            if (row < M && col < tile_end) *reinterpret_cast<uint4*>(C + (size_t)row * ldc + col) = p[k];
        }
    }
}

template <int EPI>
__global__ void __launch_bounds__(384, 1)
gemm_bf16_tn_kernel(const __grid_constant__ CUtensorMap tmap_a,
                    const __grid_constant__ CUtensorMap tmap_b, bf16* C, int M, int N,
                    int K, int ldc, const bf16* __restrict__ bias,
                    const bf16* residual /* may alias C */, int ldr, int splits_arg /* >= 1 */, const GemmTile cfg,
                    const int* __restrict__ tile_groups /* null: one weight matrix */, int batch, int a_col_stride, int c_col_stride) {
    const int BLOCK_N = cfg.bn;
    const int STAGE_BYTES = A_BYTES + BLOCK_N * BLOCK_K * 2;
    // split-K exists only in the EPI_PARTIAL_F32 instantiations; everywhere else splits is the constant 1 and the
    // unit arithmetic below folds back to the plain (m tile, n tile) loop.
    const int splits = (EPI == EPI_PARTIAL_F32) ? splits_arg : 1;
    const int STAGES = cfg.stages;
    extern __shared__ uint8_t smem_raw[];
    // SWIZZLE_128B tiles need 1024-byte alignment.
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    uint64_t* empty_bar = full_bar + MAX_STAGES;
    uint64_t* tmem_full = empty_bar + MAX_STAGES;
    uint64_t* tmem_empty = tmem_full + 2;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty + 2);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    const int m_tiles = (M + BLOCK_M - 1) / BLOCK_M;
    const int n_tiles = (N + BLOCK_N - 1) / BLOCK_N;
    const int num_k_blocks = (K + BLOCK_K - 1) / BLOCK_K;
    // Work unit = (m tile, k split, n tile), m fastest so that the CTAs that share a weight tile run together.
    // splits == 1: a unit is a whole output tile. splits > 1 (EPI_PARTIAL_F32): a unit covers kbps k-blocks and
    // writes an fp32 partial tile; splitk_reduce_kernel sums the partials and applies the epilogue.
    // batched: the products of all batch entries are one list of tiles; entry z = tile / per_z (splits == 1 there)
    const int per_z = m_tiles * n_tiles * splits;
    const int num_tiles = per_z * batch;
    const int kbps = (num_k_blocks + splits - 1) / splits;

    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&tmap_a);
        prefetch_tensormap(&tmap_b);
    }
    if (warp == 1 && lane == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&full_bar[i], 1);
            mbar_init(&empty_bar[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&tmem_full[i], 1);
            mbar_init(&tmem_empty[i], 8);  // one arrive per epilogue warp
        }
        fence_barrier_init();
    }
    if (warp == 2) {
        tmem_alloc(tmem_holder, cfg.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    const int* tile_group = tile_groups;
    chain_begin(tile_group);   // (barriers, tensor maps and TMEM are ready; only now may the next kernel's CTAs ask for TMEM)

    if (warp == 0) {
        // ===================== TMA producer =====================
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            for (int tile_all = blockIdx.x; tile_all < num_tiles; tile_all += gridDim.x) {
                const int z = tile_all / per_z, tile = tile_all - z * per_z;
                const int m_blk = tile % m_tiles, ks = (tile / m_tiles) % splits, n_blk = tile / (m_tiles * splits);
                // grouped: the m tile's weight matrix starts at row grp * N of the stacked B; all three roles skip empty tiles
                const int grp = tile_group ? tile_group[m_blk] : z;
                if (grp < 0) continue;
                const int kb0 = ks * kbps, kb1 = min(kb0 + kbps, num_k_blocks);
                for (int kb = kb0; kb < kb1; ++kb) {
                    mbar_wait(&empty_bar[stage], phase ^ 1);
                    uint8_t* sa = smem + stage * STAGE_BYTES;
                    uint8_t* sb = sa + A_BYTES;
                    mbar_arrive_expect_tx(&full_bar[stage], STAGE_BYTES);
                    tma_load_2d(sa, &tmap_a, &full_bar[stage], z * a_col_stride + kb * BLOCK_K, m_blk * BLOCK_M);
                    tma_load_2d(sb, &tmap_b, &full_bar[stage], kb * BLOCK_K, grp * N + n_blk * BLOCK_N);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ===================== MMA issuer =====================
        const uint32_t idesc = cfg.idesc;
        int stage = 0;
        uint32_t phase = 0;
        int acc = 0;
        uint32_t acc_phase = 0;
        for (int tile_all = blockIdx.x; tile_all < num_tiles; tile_all += gridDim.x) {
            const int tile = tile_all % per_z;
            if (tile_group && tile_group[tile % m_tiles] < 0) continue;
            mbar_wait(&tmem_empty[acc], acc_phase ^ 1);
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + acc * BLOCK_N;
            const int ks = (tile / m_tiles) % splits;
            const int kb0 = ks * kbps, kb1 = min(kb0 + kbps, num_k_blocks);
            for (int kb = kb0; kb < kb1; ++kb) {
                mbar_wait(&full_bar[stage], phase);
                tc_fence_after();
                if (lane == 0) {
                    const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
                    const uint32_t sb = sa + A_BYTES;
                    const uint64_t da = make_sw128_kmajor_desc(sa);
                    const uint64_t db = make_sw128_kmajor_desc(sb);
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
                        // advance start address by k*32 bytes (>>4 => +2k) inside the swizzle atom
                        umma_bf16_ss(tmem_d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc,
                                     ((kb - kb0) | k) != 0 ? 1u : 0u);
                    }
                    umma_commit(&empty_bar[stage]);  // frees the smem slot when the MMAs retire
                    if (kb == kb1 - 1) umma_commit(&tmem_full[acc]);
                }
                __syncwarp();
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
    } else if (warp >= 4) {
        // ===================== Epilogue =====================
        const int q = warp & 3;          // TMEM lane quarter this warp may access (warp id mod 4)
        const int half = (warp - 4) >> 2;  // which half of the tile's columns this warp converts
        const int chunks = (BLOCK_N + 31) >> 5;  // 32-column epilogue chunks; the last one may be half used (BLOCK_N % 32 == 16)
        const int chunks_h0 = (chunks + 1) >> 1;
        const int c_begin = half ? chunks_h0 : 0, c_end = half ? chunks : chunks_h0;
        int acc = 0;
        uint32_t acc_phase = 0;
        for (int tile_all = blockIdx.x; tile_all < num_tiles; tile_all += gridDim.x) {
            const int z = tile_all / per_z, tile = tile_all - z * per_z;
            const int m_blk = tile % m_tiles, ks = (tile / m_tiles) % splits, n_blk = tile / (m_tiles * splits);
            if (tile_group && tile_group[m_blk] < 0) continue;
            mbar_wait(&tmem_full[acc], acc_phase);
            tc_fence_after();
            const int row0 = m_blk * BLOCK_M + q * 32;
            const int tile_end = min(N, (n_blk + 1) * BLOCK_N);  // columns past it belong to the next tile (or are padding)
#pragma unroll 1
            for (int c = c_begin; c < c_end; ++c) {
                uint32_t v[32];
                const uint32_t taddr =
                    tmem_base + (uint32_t)(acc * BLOCK_N + c * 32) + ((uint32_t)(q * 32) << 16);
                tmem_ld_32x32b_x32(taddr, v);
                const int col0 = n_blk * BLOCK_N + c * 32;
                EpiFetch f;
                epilogue_fetch<EPI>(f, M, row0, lane, col0, tile_end, bias, residual, ldr);
                tmem_ld_wait();
                // batched: entry z's columns start at z * c_col_stride (floats when the output is fp32)
                bf16* Cz = (EPI == EPI_PARTIAL_F32) ? reinterpret_cast<bf16*>(reinterpret_cast<float*>(C) + (size_t)z * c_col_stride)
                                                    : C + (size_t)z * c_col_stride;
                epilogue_chunk<EPI>(v, f, Cz, ldc, M, row0, lane, col0, tile_end, ks, bias,
                                    EPI == EPI_SIGMOID_GATE ? residual + (size_t)z * c_col_stride : residual, ldr);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[acc]);
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem_base, cfg.tmem_cols);
    }
}

// ----------------------------------------------------------------------------
// CTA-pair variant (cta_group::2): one 256 x BLOCK_N output tile per pair of CTAs on a TPC.
// Each CTA stages ITS 128 rows of A and HALF of the B tile (BLOCK_N/2 rows) per k-block: shared-memory traffic per CTA and
// k-block drops from 2*(16 KB + 128*bn) to 2*(16 KB + 64*bn) bytes, which lifts the shared-memory bound of the one-CTA
// kernel (bn = 256: 768 -> 512 clocks per k-block = the tensor floor). The leader CTA (cluster rank 0) issues the MMAs for
// both; accumulators live in both CTAs' TMEM (rows 0-127 in the leader, 128-255 in the peer), each CTA runs the epilogue of
// its own rows. Barriers: `full` lives in the leader and is credited by both CTAs' TMA loads; `empty` and `tmem_full` exist
// in both CTAs and are signalled by the leader's multicast commits; `tmem_empty` lives in the leader and counts the epilogue
// warps of both CTAs.
// ----------------------------------------------------------------------------
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
gemm2_bf16_tn_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, bf16* C, int M,
                     int N, int K, int ldc, const bf16* __restrict__ bias, const bf16* residual /* may alias C */, int ldr,
                     int splits_arg /* >= 1 */, const GemmTile cfg) {
    const int splits = (EPI == EPI_PARTIAL_F32) ? splits_arg : 1;
    const int BLOCK_N = cfg.bn;
    const int HALF_N = BLOCK_N >> 1;
    const int STAGE_BYTES = A_BYTES + HALF_N * BLOCK_K * 2;
    const int STAGES = cfg.stages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    uint64_t* empty_bar = full_bar + MAX_STAGES;
    uint64_t* tmem_full = empty_bar + MAX_STAGES;
    uint64_t* tmem_empty = tmem_full + 2;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty + 2);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

    const int m_pairs = (M + 2 * BLOCK_M - 1) / (2 * BLOCK_M);
    const int n_tiles = (N + BLOCK_N - 1) / BLOCK_N;
    const int num_k_blocks = (K + BLOCK_K - 1) / BLOCK_K;
    const int num_units = m_pairs * n_tiles * splits;  // (m pair, k split, n tile), m fastest
    const int kbps = (num_k_blocks + splits - 1) / splits;

    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&tmap_a);
        prefetch_tensormap(&tmap_b);
    }
    if (warp == 1 && lane == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&full_bar[i], 1);   // used in the leader: its producer's arrive.expect_tx (bytes of both CTAs)
            mbar_init(&empty_bar[i], 1);  // one multicast commit of the leader's MMA warp
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&tmem_full[i], 1);    // one multicast commit
            mbar_init(&tmem_empty[i], 16);  // used in the leader: 8 epilogue warps of each CTA
        }
        fence_barrier_init();
    }
    if (warp == 2) {
        tmem_alloc_cg2(tmem_holder, cfg.tmem_cols);
        tmem_relinquish_cg2();
    }
    tc_fence_before();
    __syncwarp();        // barrier.cluster is .aligned: the warp must be converged
    cluster_sync_all();  // barriers of BOTH CTAs are initialised before any remote arrive / TMA credit
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    chain_begin();

    if (warp == 0) {
        // ===================== TMA producer (both CTAs) =====================
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            for (int unit = pair; unit < num_units; unit += num_pairs) {
                const int m_pair = unit % m_pairs, ks = (unit / m_pairs) % splits, n_blk = unit / (m_pairs * splits);
                const int kb0 = ks * kbps, kb1 = min(kb0 + kbps, num_k_blocks);
                for (int kb = kb0; kb < kb1; ++kb) {
                    mbar_wait(&empty_bar[stage], phase ^ 1);
                    uint8_t* sa = smem + stage * STAGE_BYTES;
                    uint8_t* sb = sa + A_BYTES;
                    if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
                    const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), 0);
                    tma_load_2d_cg2(sa, &tmap_a, bar, kb * BLOCK_K, m_pair * 2 * BLOCK_M + (int)rank * BLOCK_M);
                    tma_load_2d_cg2(sb, &tmap_b, bar, kb * BLOCK_K, n_blk * BLOCK_N + (int)rank * HALF_N);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ===================== MMA issuer (leader CTA only) =====================
        if (leader) {
            const uint32_t idesc = cfg.idesc;  // M = 256, N = BLOCK_N
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            for (int unit = pair; unit < num_units; unit += num_pairs) {
                mbar_wait(&tmem_empty[acc], acc_phase ^ 1);
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + acc * BLOCK_N;
                const int ks = (unit / m_pairs) % splits;
                const int kb0 = ks * kbps, kb1 = min(kb0 + kbps, num_k_blocks);
                for (int kb = kb0; kb < kb1; ++kb) {
                    mbar_wait(&full_bar[stage], phase);
                    tc_fence_after();
                    if (lane == 0) {
                        const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
                        const uint32_t sb = sa + A_BYTES;
                        const uint64_t da = make_sw128_kmajor_desc(sa);
                        const uint64_t db = make_sw128_kmajor_desc(sb);
#pragma unroll
                        for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
                            umma_bf16_ss_cg2(tmem_d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc,
                                             ((kb - kb0) | k) != 0 ? 1u : 0u);
                        umma_commit_cg2(&empty_bar[stage], 3);  // frees the slot in both CTAs when the MMAs retire
                        if (kb == kb1 - 1) umma_commit_cg2(&tmem_full[acc], 3);
                    }
                    __syncwarp();
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (++acc == 2) { acc = 0; acc_phase ^= 1; }
            }
        }
    } else if (warp >= 4) {
        // ===================== Epilogue (both CTAs, own 128 rows) =====================
        const int q = warp & 3;
        const int half = (warp - 4) >> 2;
        const int chunks = (BLOCK_N + 31) >> 5;
        const int chunks_h0 = (chunks + 1) >> 1;
        const int c_begin = half ? chunks_h0 : 0, c_end = half ? chunks : chunks_h0;
        int acc = 0;
        uint32_t acc_phase = 0;
        for (int unit = pair; unit < num_units; unit += num_pairs) {
            const int m_pair = unit % m_pairs, ks = (unit / m_pairs) % splits, n_blk = unit / (m_pairs * splits);
            mbar_wait(&tmem_full[acc], acc_phase);
            tc_fence_after();
            const int row0 = m_pair * 2 * BLOCK_M + (int)rank * BLOCK_M + q * 32;
            const int tile_end = min(N, (n_blk + 1) * BLOCK_N);
#pragma unroll 1
            for (int c = c_begin; c < c_end; ++c) {
                uint32_t v[32];
                const uint32_t taddr = tmem_base + (uint32_t)(acc * BLOCK_N + c * 32) + ((uint32_t)(q * 32) << 16);
                tmem_ld_32x32b_x32(taddr, v);
                const int col0 = n_blk * BLOCK_N + c * 32;
                EpiFetch f;
                epilogue_fetch<EPI>(f, M, row0, lane, col0, tile_end, bias, residual, ldr);
                tmem_ld_wait();
                epilogue_chunk<EPI>(v, f, C, ldc, M, row0, lane, col0, tile_end, ks, bias, residual, ldr);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tmem_empty[acc]), 0));
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
    }

    tc_fence_before();
    __syncwarp();        // lanes that skipped a single-lane role loop wait here for their lane 0
    cluster_sync_all();  // neither CTA may exit (or free TMEM) while the pair's MMAs / remote arrives can still touch it
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc_cg2(tmem_base, cfg.tmem_cols);
    }
}

// ----------------------------------------------------------------------------
// CTA pair with the operands swapped, for few rows: the WEIGHTS are the 256-row operand, the activations the columns.
//
// Products of a few hundred rows have too few tiles for the SMs and take every weight tile in once per 128 rows. Here a pair multiplies 256
// weight rows by up to 512 activation rows (two MMAs of up to 256 columns per k-step, each CTA staging its 128 weight rows and half of the
// activation rows): M = 281 is ONE tile of 288 columns, and a weight element reaches exactly one SM. The width is a run-time value, a
// multiple of 32; where the tiles are too few, the pairs of a cluster split K and add their accumulators through distributed shared memory
// (no partials in global memory, no second launch, fixed order). Which products gain: see choose_swap.
//
// Structure (per CTA 384 threads): as the pair kernel above. TMEM lane = weight row = output column, TMEM column = activation row = output
// row: a thread owns one output column, so its bias is one register; two shuffle rounds turn four threads' columns into 8-byte pieces of
// an output row, stored (and the residual read) as 64-byte runs. That is dearer than the row-wise store of the other kernels, so many
// rows stay with those.
// ----------------------------------------------------------------------------
struct SwapTile {
    int bm, n1, n2;      // activation rows per tile = columns of the first and (0: none) second MMA, multiples of 32
    int stages;          // ring depth
    int tmem_cols;
    int splits;          // pairs of a cluster that share a tile's K range
    uint32_t idesc1, idesc2;
    int stage_bytes, smem_bytes;
};
static constexpr int kSwapMax = 512, kSwapSplits = 4;
static SwapTile make_swap(int bm, int splits) {
    SwapTile t;
    t.bm = bm;
    t.n1 = bm <= 256 ? bm : (bm / 2 + 31) / 32 * 32;
    t.n2 = bm - t.n1;
    t.stage_bytes = A_BYTES + bm / 2 * BLOCK_K * 2;
    t.stages = (227 * 1024 - 1024 - 256) / t.stage_bytes;
    if (t.stages > MAX_STAGES) t.stages = MAX_STAGES;
    t.tmem_cols = 32;
    while (t.tmem_cols < bm) t.tmem_cols <<= 1;
    t.splits = splits;
    t.idesc1 = make_idesc_bf16(2 * BLOCK_M, t.n1);
    t.idesc2 = t.n2 ? make_idesc_bf16(2 * BLOCK_M, t.n2) : 0u;
    t.smem_bytes = t.stages * t.stage_bytes + 1024 /*align slack*/ + 256 /*barriers*/;
    return t;
}

// Bounded waits. When a signal of the swapped kernel does not come in time, the thread that waits raises the flag of every CTA of its
// cluster and the library's fault word. Every wait that has to wait sees the flag and gives up too; nothing more is loaded or multiplied; the
// epilogue writes NaN over every value that it did not see completed (with a split K: of every value of the cluster, whose shares are
// all in it); copies and products under way get a limited time to end; then tensor memory is freed and the kernel returns.
constexpr unsigned long long kWaitNs = 2000000000ull, kDrainNs = 20000000ull;
struct GiveUp {
    volatile int* flag;           // in this CTA's shared memory
    int ctas;                     // of the cluster
    unsigned long long ns;        // limit of a wait
    int* fault;                   // host-visible word, or null
};
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, P1;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_for(uint64_t* bar, uint32_t parity, const GiveUp& g) {
    // (without the hint a try may sleep for longer than a whole product; products of 24 to 1024 rows take 3 to 6 % less time with it and
    // one lane issuing the products: 281 x 3584 x 18944 50.7 -> 47.5 us)
    if (mbar_try(bar, parity, 1000u)) return true;
    unsigned long long t0, now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (;;) {
        if (mbar_try(bar, parity, 1000u)) return true;
        if (*g.flag) return false;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (now - t0 <= g.ns) continue;
        for (int c = 0; c < g.ctas; ++c)
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_shared(smem_u32(const_cast<const int*>(g.flag)), c)), "r"(1) : "memory");
        if (g.fault) {
            *reinterpret_cast<volatile int*>(g.fault) = 1;
            __threadfence_system();
        }
        return false;
    }
}
// the same for a whole warp: all lanes or none
__device__ __forceinline__ bool warp_wait_for(uint64_t* bar, uint32_t parity, const GiveUp& g) {
    return __all_sync(0xffffffffu, mbar_wait_for(bar, parity, g));
}
// what is under way ends, or its time does; the flag does not cut it short
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
    unsigned long long t0, now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    do {
        if (mbar_try(bar, parity, 1000u)) return;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    } while (now - t0 <= kDrainNs);
}

__device__ __forceinline__ float ld_cluster_addr_f32(uint32_t cluster_addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
    return v;
}

// what an accumulator becomes before it is rounded to bf16 (the activations of EPI_BIAS_QUICKGELU / EPI_BIAS_GELU follow the rounding)
template <int EPI>
__device__ __forceinline__ float swap_unary(float x, float bias) {
    if (EPI == EPI_BIAS || EPI == EPI_BIAS_QUICKGELU || EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_RESIDUAL) x += bias;
    if (EPI == EPI_RELU2) { x = fmaxf(x, 0.f); x *= x; }
    if (EPI == EPI_GELU_ERF) x = 0.5f * x * (1.f + erff(x * 0.7071067811865476f));
    if (EPI == EPI_GELU_TANH) x = 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    if (EPI == EPI_BIAS_QUICKGELU) x = quick_gelu_bf16(rbf(x));
    if (EPI == EPI_BIAS_GELU) x = gelu_erf_bf16(rbf(x));
    return x;
}
template <int EPI> struct SwapEpi {
    static constexpr bool kGlu = EPI == EPI_SWIGLU || EPI == EPI_CLAMP_GLU;
    static constexpr bool kResidual = EPI == EPI_RESIDUAL || EPI == EPI_BIAS_RESIDUAL;
};

// A warp's chunk: v[j] = accumulator of output row m0 + j, output column n (one per lane). res: the residual's 8-byte pieces at the
// places this lane will store (rows m0 + 4 k + (lane & 3), columns (n & ~3) ..), EPI_*RESIDUAL only.
template <int EPI>
__device__ __forceinline__ void swap_store(const float (&v)[32], bf16* C, int ldc, int M, int N, int m0, int n, int lane, float bias,
                                           const uint2 (&res)[8], float limit, float alpha, float up_bias) {
    if (SwapEpi<EPI>::kGlu) {
        // lanes 0..15 hold gate rows, 16..31 the matching up rows: of rows j, j + 1 the lower half makes row j, the upper half row j + 1
        const bool hi = lane & 16;
        uint32_t o[8];   // rows j + hi (low half) and j + 2 + hi (high half), j = 0, 4, ...
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float y[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int j = 4 * k + 2 * e;
                const float r = __shfl_xor_sync(0xffffffffu, hi ? v[j] : v[j + 1], 16);
                const float g = hi ? r : v[j], u = hi ? v[j + 1] : r;
                if (EPI == EPI_SWIGLU) y[e] = silu_bf16(rbf(g)) * rbf(u);
                else {
                    const float gc = fminf(g, limit), uc = fminf(fmaxf(u, -limit), limit);
                    y[e] = gc / (1.f + __expf(-alpha * gc)) * (uc + up_bias);
                }
            }
            o[k] = pack_bf16x2(y[0], y[1]);
        }
        const int col = ((n >> 5) << 4) + (lane & 12);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t w[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {   // even lane: row 4 k' + hi of two columns, odd lane: row 4 k' + 2 + hi
                const uint32_t own = o[2 * k + e], other = __shfl_xor_sync(0xffffffffu, own, 1);
                w[e] = (lane & 1) ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
            }
            const uint32_t recv = __shfl_xor_sync(0xffffffffu, (lane & 2) ? w[0] : w[1], 2);
            const uint2 q = (lane & 2) ? make_uint2(recv, w[1]) : make_uint2(w[0], recv);
            const int row = m0 + 4 * (2 * k + ((lane >> 1) & 1)) + 2 * (lane & 1) + (hi ? 1 : 0);
            if (row < M && n < N) *reinterpret_cast<uint2*>(C + (size_t)row * ldc + col) = q;
        }
        return;
    }
    const int col = n & ~3;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        uint32_t w[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {   // rows j, j + 1: the even lane keeps row j of two columns, the odd lane row j + 1
            const int j = 4 * k + 2 * e;
            const uint32_t own = pack_bf16x2(swap_unary<EPI>(v[j], bias), swap_unary<EPI>(v[j + 1], bias));
            const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
            w[e] = (lane & 1) ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
        }
        const uint32_t recv = __shfl_xor_sync(0xffffffffu, (lane & 2) ? w[0] : w[1], 2);
        uint2 q = (lane & 2) ? make_uint2(recv, w[1]) : make_uint2(w[0], recv);
        const int row = m0 + 4 * k + (lane & 3);
        if (SwapEpi<EPI>::kResidual) {
            const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), ra = unpack_bf16x2(res[k].x), rb = unpack_bf16x2(res[k].y);
            q = make_uint2(pack_bf16x2(a.x + ra.x, a.y + ra.y), pack_bf16x2(b.x + rb.x, b.y + rb.y));
        }
        if (row < M && n < N) *reinterpret_cast<uint2*>(C + (size_t)row * ldc + col) = q;
    }
}

template <int EPI>
__global__ void __launch_bounds__(384, 1)
gemm_swap_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x1,
                 const __grid_constant__ CUtensorMap tmap_x2, bf16* C, int M, int N, int K, int ldc, const bf16* __restrict__ bias,
                 const bf16* residual /* may alias C */, int ldr, const SwapTile cfg, float limit, float alpha, float up_bias,
                 unsigned long long wait_ns, int* fault) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int STAGES = cfg.stages, STAGE_BYTES = cfg.stage_bytes, S = cfg.splits;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    uint64_t* empty_bar = full_bar + MAX_STAGES;
    uint64_t* tmem_full = empty_bar + MAX_STAGES;
    uint64_t* tmem_empty = tmem_full + 1;
    uint64_t* drained = tmem_empty + 1;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(drained + 1);
    const GiveUp g{reinterpret_cast<volatile int*>(tmem_holder + 1), 2 * S, wait_ns, fault};

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t crank = cluster_ctarank();
    const int rank = crank & 1, split = crank >> 1;        // CTA of the pair; pair of the cluster
    const uint32_t lead = crank & ~1u;
    const bool leader = rank == 0;
    const int cluster = blockIdx.x / (2 * S), num_clusters = gridDim.x / (2 * S);

    const int m_tiles = (M + cfg.bm - 1) / cfg.bm, n_tiles = (N + 2 * BLOCK_M - 1) / (2 * BLOCK_M);
    const int nkb = (K + BLOCK_K - 1) / BLOCK_K;
    const int kb0 = (int)((long long)nkb * split / S), kb1 = (int)((long long)nkb * (split + 1) / S);
    const int units = m_tiles * n_tiles;   // m fastest: the tiles that share weight rows run together. S > 1: one unit per cluster

    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&tmap_w);
        prefetch_tensormap(&tmap_x1);
        if (cfg.n2) prefetch_tensormap(&tmap_x2);
    }
    if (warp == 1 && lane == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&full_bar[i], 1);   // used in the leader: its producer's arrive.expect_tx (bytes of both CTAs)
            mbar_init(&empty_bar[i], 1);  // one multicast commit of the leader's MMA warp
        }
        mbar_init(tmem_full, 1);    // one multicast commit
        mbar_init(tmem_empty, 16);  // used in the leader: 8 epilogue warps of each CTA
        mbar_init(drained, 1);      // the leader's last commit
        *g.flag = 0;
        fence_barrier_init();
    }
    if (warp == 2) {
        tmem_alloc_cg2(tmem_holder, cfg.tmem_cols);
        tmem_relinquish_cg2();
    }
    tc_fence_before();
    __syncwarp();        // barrier.cluster is .aligned: the warp must be converged
    cluster_sync_all();  // barriers of all CTAs are initialised before any remote arrive / TMA credit
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    chain_begin();

    if (warp == 0) {
        // ===================== TMA producer (both CTAs) =====================
        if (lane == 0) {
            int stage = 0, issued = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int unit = cluster; ok && unit < units; unit += num_clusters) {
                const int m0 = (unit % m_tiles) * cfg.bm, n0 = (unit / m_tiles) * 2 * BLOCK_M;
                for (int kb = kb0; kb < kb1; ++kb) {
                    ok = mbar_wait_for(&empty_bar[stage], phase ^ 1, g);
                    if (!ok) break;
                    uint8_t* sw = smem + stage * STAGE_BYTES;
                    uint8_t* sx = sw + A_BYTES;
                    if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
                    const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), lead);
                    tma_load_2d_cg2(sw, &tmap_w, bar, kb * BLOCK_K, n0 + rank * BLOCK_M);
                    tma_load_2d_cg2(sx, &tmap_x1, bar, kb * BLOCK_K, m0 + rank * (cfg.n1 / 2));
                    if (cfg.n2)
                        tma_load_2d_cg2(sx + cfg.n1 / 2 * BLOCK_K * 2, &tmap_x2, bar, kb * BLOCK_K, m0 + cfg.n1 + rank * (cfg.n2 / 2));
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                    ++issued;
                }
            }
            // no CTA leaves while copies into it are under way: the leader's barriers count those of both CTAs
            for (int i = max(0, issued - STAGES); leader && i < issued; ++i) {
                const uint32_t p = (i / STAGES) & 1;
                if (!mbar_wait_for(&full_bar[i % STAGES], p, g)) mbar_drain(&full_bar[i % STAGES], p);
            }
            if (!ok) __nanosleep(1000000);   // (one CTA may have issued a few more than the other)
        }
    } else if (warp == 1) {
        // ===================== MMA issuer (one lane of the leader CTA) =====================
        if (leader && lane == 0) {
            int stage = 0;
            uint32_t phase = 0, acc_phase = 0;
            const uint16_t both = (uint16_t)(3u << lead);
            bool ok = true;
            for (int unit = cluster; unit < units; unit += num_clusters) {
                ok = mbar_wait_for(tmem_empty, acc_phase ^ 1, g);
                if (!ok) break;
                tc_fence_after();
                for (int kb = kb0; kb < kb1; ++kb) {
                    ok = mbar_wait_for(&full_bar[stage], phase, g);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sw = smem_u32(smem + stage * STAGE_BYTES);
                    const uint64_t dw = make_sw128_kmajor_desc(sw);
                    const uint64_t dx = make_sw128_kmajor_desc(sw + A_BYTES);
                    const uint64_t dx2 = make_sw128_kmajor_desc(sw + A_BYTES + cfg.n1 / 2 * BLOCK_K * 2);
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
                        const uint32_t add = ((kb - kb0) | k) != 0 ? 1u : 0u;
                        umma_bf16_ss_cg2(tmem_base, dw + (uint64_t)(k * 2), dx + (uint64_t)(k * 2), cfg.idesc1, add);
                        if (cfg.n2) umma_bf16_ss_cg2(tmem_base + cfg.n1, dw + (uint64_t)(k * 2), dx2 + (uint64_t)(k * 2), cfg.idesc2, add);
                    }
                    umma_commit_cg2(&empty_bar[stage], both);  // frees the slot in both CTAs when the MMAs retire
                    if (kb == kb1 - 1) umma_commit_cg2(tmem_full, both);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                acc_phase ^= 1;
            }
            // the products read both CTAs' shared memory and write both halves of tensor memory: they end before either CTA leaves
            umma_commit_cg2(drained, (uint16_t)(1u << lead));
            if (!mbar_wait_for(drained, 0, g)) mbar_drain(drained, 0);
        }
    } else if (warp >= 4) {
        // ===================== Epilogue (both CTAs, own 128 weight rows) =====================
        const int q = warp & 3, half = (warp - 4) >> 2;   // TMEM lane quarter; every other chunk of 32 activation rows
        const int chunks = cfg.bm >> 5;
        bool lost = false;
        uint32_t acc_phase = 0;
        for (int unit = cluster; unit < units; unit += num_clusters) {
            const int m0 = (unit % m_tiles) * cfg.bm;
            const int n = (unit / m_tiles) * 2 * BLOCK_M + rank * BLOCK_M + q * 32 + lane;
            float b = 0.f;
            if (EPI == EPI_BIAS || EPI == EPI_BIAS_QUICKGELU || EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_RESIDUAL) b = n < N ? bf2f(bias[n]) : 0.f;
            // the chunks this warp finishes: all of its half, or with a split K range those this pair owns
            auto owner = [&](int c) { return S == 1 ? 0 : c * S / chunks; };
            auto mine = [&](int c) { return S == 1 ? (c & 1) == half : owner(c) == split && ((c - (split * chunks + S - 1) / S) & 1) == half; };
            uint2 res[8];
            auto fetch = [&](int c) {   // the residual of chunk c, in flight while the accumulators are awaited
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int row = m0 + c * 32 + 4 * k + (lane & 3);
                    res[k] = row < M && n < N ? *reinterpret_cast<const uint2*>(residual + (size_t)row * ldr + (n & ~3)) : make_uint2(0u, 0u);
                }
            };
            int c = 0;
            while (c < chunks && !mine(c)) ++c;
            if (SwapEpi<EPI>::kResidual && c < chunks) fetch(c);
            lost = !warp_wait_for(tmem_full, acc_phase, g) || lost;   // (behind a phase that never ended the next one's parity reads as past)
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
            float* red = reinterpret_cast<float*>(smem) + q * 32 + lane;   // [chunk][32 columns][128 weight rows]: over the drained ring
            if (S > 1) {
                for (int d = half; d < chunks; d += 2) {
                    if (owner(d) == split) continue;
                    uint32_t v[32];
                    tmem_ld_32x32b_x32(taddr + d * 32, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) red[(size_t)(d * 32 + j) * BLOCK_M] = __uint_as_float(v[j]);
                }
                __syncwarp();
                cluster_sync_all();
                lost = __any_sync(0xffffffffu, lost || *g.flag);   // a share of any pair of the cluster is missing
            }
            while (c < chunks) {
                int next = c + 1;
                while (next < chunks && !mine(next)) ++next;
                uint32_t v[32];
                tmem_ld_32x32b_x32(taddr + c * 32, v);
                tmem_ld_wait();
                float x[32];
                if (S > 1) {
                    const uint32_t at = smem_u32(red + (size_t)c * 32 * BLOCK_M);
#pragma unroll
                    for (int j = 0; j < 32; ++j) x[j] = 0.f;
                    for (int sp = 0; sp < S; ++sp) {   // in split order, whoever adds
                        const uint32_t from = mapa_shared(at, 2 * sp + rank);
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            x[j] += sp == split ? __uint_as_float(v[j]) : ld_cluster_addr_f32(from + j * BLOCK_M * 4);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(v[j]);
                }
                uint2 now[8];
                if (SwapEpi<EPI>::kResidual) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) now[k] = res[k];
                    if (next < chunks) fetch(next);
                }
                swap_store<EPI>(x, C, ldc, M, N, m0 + c * 32, n, lane, b, now, limit, alpha, up_bias);
                c = next;
            }
            if (lost) {   // (behind the stores: a test per value inside them costs 3 to 5 % of a product)
                __syncwarp();
                const int col = SwapEpi<EPI>::kGlu ? ((n >> 5) << 4) + (lane & 15) : n;
                for (int d = 0; d < chunks; ++d)
                    for (int j = 0; mine(d) && j < 32; ++j)
                        if (m0 + d * 32 + j < M && n < N) C[(size_t)(m0 + d * 32 + j) * ldc + col] = __ushort_as_bfloat16(0x7fff);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(tmem_empty), lead));
            acc_phase ^= 1;
        }
    }

    if (S > 1 && warp < 4) {
        __syncwarp();
        cluster_sync_all();   // the epilogue warps' barrier of the split reduction counts every thread of the cluster
    }
    tc_fence_before();
    __syncwarp();        // lanes that skipped a single-lane role loop wait here for their lane 0
    cluster_sync_all();  // no CTA may exit (or free TMEM) while the pair's MMAs / remote reads and arrives can still touch it
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc_cg2(tmem_base, cfg.tmem_cols);
    }
}


// ----------------------------------------------------------------------------
// Host side
// ----------------------------------------------------------------------------
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                    const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode_fn() {
    static PFN_encodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) !=
                cudaSuccess ||
            qres != cudaDriverEntryPointSuccess)
            return nullptr;
        fn = reinterpret_cast<PFN_encodeTiled>(p);
    }
    return fn;
}

int make_tmap_bf16_2d_box(CUtensorMap* tm, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_cols,
                          int box_rows, bool swizzle32) {
    PFN_encodeTiled fn = get_encode_fn();
    if (!fn) return -1;
    cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstride,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -2;
}

int make_tmap_bf16_3d_sw128(CUtensorMap* tm, const void* ptr, int64_t d0, int64_t d1, int64_t d2, int64_t stride1,
                            int64_t stride2, int box1, int box2) {
    PFN_encodeTiled fn = get_encode_fn();
    if (!fn) return -1;
    cuuint64_t gdim[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
    cuuint64_t gstride[2] = {(cuuint64_t)stride1 * 2, (cuuint64_t)stride2 * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)box1, (cuuint32_t)box2};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), gdim, gstride, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -2;
}

// 2-D bf16 row-major [rows, cols] with row stride ld (elements); box = [box_rows, 64 cols], SW128.
int make_tmap_bf16_2d(CUtensorMap* tm, const void* ptr, int64_t rows, int64_t cols, int64_t ld,
                      int box_rows) {
    return make_tmap_bf16_2d_box(tm, ptr, rows, cols, ld, BLOCK_K, box_rows, false);
}

// The clamped GLU has no residual and no bias: those slots carry the clamp, the slope and the offset.
static void glu_slots(const GemmArgs& a, int& ldr, const bf16*& bias) {
    memcpy(&ldr, &a.epi_param, sizeof(int));
    const float ab[2] = {a.epi_alpha, a.epi_up_bias};
    static_assert(sizeof(bias) == sizeof(ab), "two floats ride in a pointer");
    memcpy(&bias, ab, sizeof(ab));
}

static void set_logit_slots(const GemmArgs& a, int& ldr, const bf16*& bias) {
    const float cap = a.logit_cap > 0.f ? a.logit_cap : 0.f, is[2] = {cap > 0.f ? 1.f / cap : 0.f, a.logit_scale};
    memcpy(&ldr, &cap, sizeof(int));
    memcpy(&bias, is, sizeof(is));
}

template <int EPI>
static int launch_cfg(const GemmArgs& a, int bn, int num_sms, cudaStream_t stream) {
    const GemmTile cfg = make_tile(bn);
    CUtensorMap ta, tb;
    const int batch = a.batch > 1 ? a.batch : 1;
    // batched: A's map spans every entry's columns (a k-block that runs past an entry's K meets zero columns of B)
    if (make_tmap_bf16_2d(&ta, a.A, a.M, batch > 1 ? (int64_t)(batch - 1) * a.a_col_stride + a.K : a.K, a.lda, BLOCK_M)) return -10;
    if (make_tmap_bf16_2d(&tb, a.B, (int64_t)a.N * (a.tile_group ? a.groups : batch), a.K, a.ldb, bn)) return -11;
    auto kern = gemm_bf16_tn_kernel<EPI>;
    static SmemAttrOnce once;  // per template instantiation
    if (ensure_dyn_smem(once, kern, 227 * 1024)) return -12;
    const int m_tiles = (a.M + BLOCK_M - 1) / BLOCK_M, n_tiles = (a.N + bn - 1) / bn;
    const int splits = (EPI == EPI_PARTIAL_F32 && a.splits > 1) ? a.splits : 1;
    const int tiles = m_tiles * n_tiles * splits * batch;
    const int grid = tiles < num_sms ? tiles : num_sms;
    lcc::count_launch();
    int ldr = a.ldr;
    const bf16* bias = (const bf16*)a.bias;
    if (EPI == EPI_CLAMP_GLU) glu_slots(a, ldr, bias);
    if (EPI == EPI_LOGITS_F32) set_logit_slots(a, ldr, bias);
    chained(kern, grid, 384, cfg.smem_bytes, stream)(ta, tb, (bf16*)a.C, a.M, a.N, a.K, a.ldc, bias, (const bf16*)a.residual, ldr, splits, cfg,
                                                     a.tile_group, batch, a.a_col_stride, a.c_col_stride);
    return cudaGetLastError() == cudaSuccess ? 0 : -13;
}

template <int EPI>
static int launch_cfg2(const GemmArgs& a, int bn, int num_sms, cudaStream_t stream) {
    const GemmTile cfg = make_tile(bn, true);
    CUtensorMap ta, tb;
    if (make_tmap_bf16_2d(&ta, a.A, a.M, a.K, a.lda, BLOCK_M)) return -10;
    if (make_tmap_bf16_2d(&tb, a.B, a.N, a.K, a.ldb, bn / 2)) return -11;
    auto kern = gemm2_bf16_tn_kernel<EPI>;
    static SmemAttrOnce once;
    if (ensure_dyn_smem(once, kern, 227 * 1024)) return -12;
    const int m_pairs = (a.M + 2 * BLOCK_M - 1) / (2 * BLOCK_M), n_tiles = (a.N + bn - 1) / bn;
    const int splits = (EPI == EPI_PARTIAL_F32 && a.splits > 1) ? a.splits : 1;
    const int units = m_pairs * n_tiles * splits;
    const int pairs = units < num_sms / 2 ? units : num_sms / 2;
    lcc::count_launch();
    int ldr = a.ldr;
    const bf16* bias = (const bf16*)a.bias;
    if (EPI == EPI_CLAMP_GLU) glu_slots(a, ldr, bias);
    chained(kern, 2 * pairs, 384, cfg.smem_bytes, stream)(ta, tb, (bf16*)a.C, a.M, a.N, a.K, a.ldc, bias, (const bf16*)a.residual, ldr, splits, cfg);
    return cudaGetLastError() == cudaSuccess ? 0 : -13;
}

static int launch_epi2(const GemmArgs& a, int bn, int num_sms, cudaStream_t stream) {
    switch (a.epi) {
        case EPI_NONE: return launch_cfg2<EPI_NONE>(a, bn, num_sms, stream);
        case EPI_BIAS: return launch_cfg2<EPI_BIAS>(a, bn, num_sms, stream);
        case EPI_BIAS_QUICKGELU: return launch_cfg2<EPI_BIAS_QUICKGELU>(a, bn, num_sms, stream);
        case EPI_BIAS_GELU: return launch_cfg2<EPI_BIAS_GELU>(a, bn, num_sms, stream);
        case EPI_RESIDUAL: return launch_cfg2<EPI_RESIDUAL>(a, bn, num_sms, stream);
        case EPI_BIAS_RESIDUAL: return launch_cfg2<EPI_BIAS_RESIDUAL>(a, bn, num_sms, stream);
        case EPI_SWIGLU: return launch_cfg2<EPI_SWIGLU>(a, bn, num_sms, stream);
        case EPI_RELU2: return launch_cfg2<EPI_RELU2>(a, bn, num_sms, stream);
        case EPI_GELU_TANH: return launch_cfg2<EPI_GELU_TANH>(a, bn, num_sms, stream);
        case EPI_GELU_ERF: return launch_cfg2<EPI_GELU_ERF>(a, bn, num_sms, stream);
        case EPI_CLAMP_GLU: return launch_cfg2<EPI_CLAMP_GLU>(a, bn, num_sms, stream);
    }
    return -14;
}

// Clusters of 2 * splits CTAs (one per SM) that the device holds at once, 0 when that cannot be asked; a hardware fact, kept per device and
// size once it is known.
static int max_clusters(int dev, int splits, int num_sms) {
    static std::atomic<int> known[64][kSwapSplits + 1];
    if (dev < 0) return 0;
    int n = dev < 64 ? known[dev][splits].load(std::memory_order_relaxed) : 0;
    if (n) return n;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(num_sms / (2 * splits) * 2 * splits);
    cfg.blockDim = dim3(384);
    cfg.dynamicSmemBytes = 227 * 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(gemm_swap_kernel<EPI_NONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_swap_kernel<EPI_NONE>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();   // the question's error is not the caller's
        return 0;
    }
    if (dev < 64) known[dev][splits].store(n, std::memory_order_relaxed);
    return n;
}
static int current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) == cudaSuccess) return dev;
    cudaGetLastError();
    return -1;
}

template <int EPI>
static int launch_swap(const GemmArgs& a, int bm, int splits, int num_sms, cudaStream_t stream) {
    const int units = (a.M + bm - 1) / bm * ((a.N + 2 * BLOCK_M - 1) / (2 * BLOCK_M));
    const int clusters = std::min(units, max_clusters(current_device(), splits, num_sms));
    if (clusters < 1) return -15;
    const SwapTile cfg = make_swap(bm, splits);
    // a shared K range: every unit has its cluster, every pair a k-block, and the partial accumulators fit over the ring
    if (splits > 1 && (clusters < units || (a.K + BLOCK_K - 1) / BLOCK_K < splits || bm * BLOCK_M * 4 > cfg.stages * cfg.stage_bytes)) return -15;
    CUtensorMap tw, t1, t2;
    if (make_tmap_bf16_2d(&tw, a.B, a.N, a.K, a.ldb, BLOCK_M)) return -10;
    if (make_tmap_bf16_2d(&t1, a.A, a.M, a.K, a.lda, cfg.n1 / 2)) return -11;
    if (make_tmap_bf16_2d(&t2, a.A, a.M, a.K, a.lda, (cfg.n2 ? cfg.n2 : cfg.n1) / 2)) return -11;
    auto kern = gemm_swap_kernel<EPI>;
    static SmemAttrOnce once;
    if (ensure_dyn_smem(once, kern, 227 * 1024)) return -12;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(clusters * 2 * splits);
    lc.blockDim = dim3(384);
    lc.dynamicSmemBytes = cfg.smem_bytes;
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = chain_next() ? 2 : 1;
    lcc::count_launch();
    return cudaLaunchKernelEx(&lc, kern, tw, t1, t2, (bf16*)a.C, a.M, a.N, a.K, a.ldc, (const bf16*)a.bias, (const bf16*)a.residual, a.ldr, cfg,
                              a.epi_param, a.epi_alpha, a.epi_up_bias, a.wait_ns ? (unsigned long long)a.wait_ns : kWaitNs, a.fault) == cudaSuccess ? 0 : -13;
}

static int launch_epi_swap(const GemmArgs& a, int bm, int splits, int num_sms, cudaStream_t stream) {
    switch (a.epi) {
        case EPI_NONE: return launch_swap<EPI_NONE>(a, bm, splits, num_sms, stream);
        case EPI_BIAS: return launch_swap<EPI_BIAS>(a, bm, splits, num_sms, stream);
        case EPI_BIAS_QUICKGELU: return launch_swap<EPI_BIAS_QUICKGELU>(a, bm, splits, num_sms, stream);
        case EPI_BIAS_GELU: return launch_swap<EPI_BIAS_GELU>(a, bm, splits, num_sms, stream);
        case EPI_RESIDUAL: return launch_swap<EPI_RESIDUAL>(a, bm, splits, num_sms, stream);
        case EPI_BIAS_RESIDUAL: return launch_swap<EPI_BIAS_RESIDUAL>(a, bm, splits, num_sms, stream);
        case EPI_SWIGLU: return launch_swap<EPI_SWIGLU>(a, bm, splits, num_sms, stream);
        case EPI_RELU2: return launch_swap<EPI_RELU2>(a, bm, splits, num_sms, stream);
        case EPI_GELU_TANH: return launch_swap<EPI_GELU_TANH>(a, bm, splits, num_sms, stream);
        case EPI_GELU_ERF: return launch_swap<EPI_GELU_ERF>(a, bm, splits, num_sms, stream);
        case EPI_CLAMP_GLU: return launch_swap<EPI_CLAMP_GLU>(a, bm, splits, num_sms, stream);
    }
    return -14;
}

static int launch_epi(const GemmArgs& a, int bn, int num_sms, cudaStream_t stream) {
    switch (a.epi) {
        case EPI_NONE: return launch_cfg<EPI_NONE>(a, bn, num_sms, stream);
        case EPI_BIAS: return launch_cfg<EPI_BIAS>(a, bn, num_sms, stream);
        case EPI_BIAS_QUICKGELU: return launch_cfg<EPI_BIAS_QUICKGELU>(a, bn, num_sms, stream);
        case EPI_BIAS_GELU: return launch_cfg<EPI_BIAS_GELU>(a, bn, num_sms, stream);
        case EPI_RESIDUAL: return launch_cfg<EPI_RESIDUAL>(a, bn, num_sms, stream);
        case EPI_BIAS_RESIDUAL: return launch_cfg<EPI_BIAS_RESIDUAL>(a, bn, num_sms, stream);
        case EPI_SWIGLU: return launch_cfg<EPI_SWIGLU>(a, bn, num_sms, stream);
        case EPI_RELU2: return launch_cfg<EPI_RELU2>(a, bn, num_sms, stream);
        case EPI_GELU_TANH: return launch_cfg<EPI_GELU_TANH>(a, bn, num_sms, stream);
        case EPI_GELU_ERF: return launch_cfg<EPI_GELU_ERF>(a, bn, num_sms, stream);
        case EPI_CLAMP_GLU: return launch_cfg<EPI_CLAMP_GLU>(a, bn, num_sms, stream);
        case EPI_SIGMOID_GATE: return launch_cfg<EPI_SIGMOID_GATE>(a, bn, num_sms, stream);
    }
    return -14;
}

// Tile-width choice. What the B200 measurements say:
//  * with one CTA per SM the main loop is bound by SHARED-MEMORY bandwidth, not by the tensor pipe: per 64-deep k-block the
//    TMA writes 16 KB (A) + bn*128 B (B) into shared memory and the four MMAs read the same bytes back: 2*(16384 + 128*bn) B
//    at 128 B/clk = 256 + 2*bn clocks against the tensor floor of 2*bn (bn = 256: 67 %, 128: 50 %, 64: 33 % — the measured
//    per-k-block times of every shape in the sweep fit this at the ~1.4 GHz the SMs run under tensor load);
//  * every launch carries ~8 us that does not depend on the tile (launch gap, barrier/TMEM set-up, first TMA round trip,
//    the un-overlapped epilogue of the last tile), which is 30-60 % of the M = 281 / 1024 GEMMs of the streaming path;
// For grouped and batched products, those with a gate and those with fp32 output: 64-wide tiles never win; between 128 and 256 columns the cost is
// (waves over the SMs) x (128 + bn), ties to the narrower tile. (Widths in between, which fill a last wave, are weighed for plain products only.)
static int choose_bn(int M, int N, int num_sms) {
    if (N <= 64) return 64;
    const long long m_tiles = (M + BLOCK_M - 1) / BLOCK_M;
    auto cost = [&](int bn) {
        const long long tiles = m_tiles * ((N + bn - 1) / bn);
        return ((tiles + num_sms - 1) / num_sms) * (long long)(128 + bn);
    };
    return cost(128) <= cost(256) ? 128 : 256;
}

// Plain products: one CTA per tile, or a CTA pair, and how wide a tile. Waves of tiles x 64-deep k-blocks x the time of one, plus a launch: 6.5 us and
// 0.26, 0.275, 0.285, 0.30, 0.345, 0.385 us for 96 to 256 columns of a CTA, 8 us and 0.31, 0.31, 0.325, 0.345, 0.335 for 128 to 256 of a pair,
// which brings in half the bytes per multiplication and has 74 units of 256 rows for 148 of 128. What gains by a width in between is a
// last wave that is filled. Measured (us, back to back; one CTA of 128 or 256 columns | its best width | pair | taken):
// 1024 x 5120 x 1280 25 | 160: 21.6 | 23.2 | 21.6, 2048 x 1280 x 5120 31.3 | 192: 27.9 | 31.2 | 160: 29.3, 2090 x 4608 x 3584 66 | 192: 58 | 61 | 58,
// 2090 x 3584 x 3584 47.7 | 224: 44.2 | 46 | 44.2, 8192 x 1280 x 5120 107 | 224: 95 | 98 | 95, 512 x 10304 x 2048 29 | 160: 24 | 26 | 24,
// 8192 x 3840 x 1280 66 | 256: 66 | 62.4 | pair, 2090 x 37888 x 3584 432 | 224: 424 | 389 | pair, 600 x 37888 x 3584 128 | 256: 128 | 139 | 128.
// Both forms add over k in the same order at every width.
static double tile_us(int M, int N, int K, int rows, int bn, int at_once, double per_kb) {
    const long long units = (long long)((M + rows - 1) / rows) * ((N + bn - 1) / bn), nkb = (K + BLOCK_K - 1) / BLOCK_K;
    return (double)((units + at_once - 1) / at_once * nkb) * per_kb;
}
// width of one CTA's tile, and its estimate
static int choose_alone(int M, int N, int K, int num_sms, double* us) {
    static constexpr double per_kb[6] = {0.26, 0.275, 0.285, 0.30, 0.345, 0.385};
    int width = 64;
    if (N <= 64) { *us = 0.; return width; }
    *us = 1e300;
    for (int i = 0; i < 6; ++i) {
        const double t = 6.5 + tile_us(M, N, K, BLOCK_M, 96 + 32 * i, num_sms, per_kb[i]);
        if (t < *us) { *us = t; width = 96 + 32 * i; }
    }
    return width;
}
// width of a pair's tile, 0 where one CTA (estimate `alone`) is not slower
static int choose_pair(int M, int N, int K, int num_sms, double alone, double* us) {
    static constexpr double per_kb[5] = {0.31, 0.31, 0.325, 0.345, 0.335};
    *us = alone;
    if (N <= 64 || num_sms < 2) return 0;
    double best = alone;
    int width = 0;
    for (int i = 0; i < 5; ++i) {
        const double t = 8.0 + tile_us(M, N, K, 2 * BLOCK_M, 128 + 32 * i, num_sms / 2, per_kb[i]);
        if (t < best) { best = t; width = 128 + 32 * i; }
    }
    if (width) *us = best;
    return width;
}

// estimates: the swapped form (waves of tiles of bm rows, nkb k-blocks a share), and K split through the scratch (two launches, the partials written and read once)
static double swap_us(int bm, int waves, int nkb, int splits) {
    return 6.5 + waves * nkb * std::max(0.42, bm / 700.0) + 0.5 * bm / 64 + (splits > 1 ? 2.5 + 0.8 * bm / 64 : 0.0);
}
static int splitk_width(const GemmArgs& a) { return a.block_n ? a.block_n : (a.N >= 256 ? 256 : (a.N >= 128 ? 128 : 64)); }
static double scratch_us(const GemmArgs& a, int ranges, int num_sms) {
    const int w = splitk_width(a), tiles = (a.M + BLOCK_M - 1) / BLOCK_M * ((a.N + w - 1) / w), nkb = (a.K + BLOCK_K - 1) / BLOCK_K;
    return 14.0 + (tiles * ranges + num_sms - 1) / num_sms * ((nkb + ranges - 1) / ranges) * 0.41 + (double)a.M * a.N * ranges * 4 / 6.5e6;
}

// Few rows: is the swapped kernel the better one? `other`: the estimate of the best other form (0: none, narrow products). One wave of
// clusters of 2 s CTAs (two waves where all rows are one tile), max(0.42, rows / 700) us per k-block of a pair's share, 6.5 us for the launch,
// 2.5 and 0.8 per 64 rows for the exchange of a split, 0.5 per 64 rows for the store. Measured (us, best of the other forms | this, back to back):
// 281 rows x 3584 x 18944 52 | 48, x 37888 x 3584 81 | 72, 24 x 4608 x 3584 19.3 | 15.9, 256 x 5120 x 5120 28.5 | 27.1; others stay for 328 x 3584 x 3584
// 20.3 | 23.9 (taken while the exchange was held to cost 3.5 whatever the rows), 1288 x 1280 x 5120 27.0 | 28.1, 24 x 3584 x 18944 31 | 40. Over 208
// products (8 to 2048 rows of the models' shapes) the choice of all forms takes 0.7 % more than the best form of each, at most 11 %.
// The unsplit forms have the same bits; a split of K changes the order of the sum.
static bool choose_swap(int M, int N, int K, int num_sms, double other, int* bm_out, int* splits_out) {
    const int n_tiles = (N + 2 * BLOCK_M - 1) / (2 * BLOCK_M), nkb = (K + BLOCK_K - 1) / BLOCK_K;
    const int t0 = (M + kSwapMax - 1) / kSwapMax;
    // (the fewest tiles there can be, against the most clusters and waves: most products of thousands of rows end here)
    if ((long long)t0 * n_tiles > (long long)num_sms / 2 * (t0 == 1 ? 2 : 1)) return false;
    const int dev = current_device();
    int fit[kSwapSplits + 1];
    for (int sp = 1; sp <= kSwapSplits; ++sp) fit[sp] = max_clusters(dev, sp, num_sms);
    double best = other;
    bool found = false;
    for (int tiles = t0; tiles <= 2 * t0 + 2; ++tiles) {
        const int bm = ((M + tiles - 1) / tiles + 31) / 32 * 32, m_tiles = (M + bm - 1) / bm, units = m_tiles * n_tiles;
        for (int sp = 1; sp <= kSwapSplits; ++sp) {
            if (fit[sp] < 1) continue;
            const int waves = (units + fit[sp] - 1) / fit[sp];
            if (waves > (sp == 1 && m_tiles == 1 ? 2 : 1) || nkb < 4 * sp) continue;
            const SwapTile t = make_swap(bm, sp);
            if (sp > 1 && bm * BLOCK_M * 4 > t.stages * t.stage_bytes) continue;
            const double us = swap_us(bm, waves, (nkb + sp - 1) / sp, sp);
            if (us < best) { best = us; *bm_out = bm; *splits_out = sp; found = true; }
        }
    }
    return found;
}

// Sum of the split-K partials + the fused epilogue (same rounding points as the in-kernel epilogues):
// C = bf16(sum [+ bias]) [then bf16(. + residual)].  One thread per 8 columns; residual may alias C.
__global__ void splitk_reduce_kernel(const float* __restrict__ part, int splits, int M, int N,
                                     const bf16* __restrict__ bias, const bf16* residual, int ldr, bf16* C, int ldc,
                                     int epi) {
    chain_begin(part);
    const int groups = N / 8;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)M * groups) return;
    const int row = (int)(idx / groups), col = (int)(idx % groups) * 8;
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int ks = 0; ks < splits; ++ks) {
        const float4* src = reinterpret_cast<const float4*>(part + ((size_t)ks * M + row) * (size_t)N + col);
        const float4 a = src[0], b = src[1];
        x[0] += a.x; x[1] += a.y; x[2] += a.z; x[3] += a.w;
        x[4] += b.x; x[5] += b.y; x[6] += b.z; x[7] += b.w;
    }
    if (epi == EPI_BIAS || epi == EPI_BIAS_RESIDUAL) {
        const uint4 bb = *reinterpret_cast<const uint4*>(bias + col);
        const uint32_t bw[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(bw[j]);
            x[2 * j] += f.x;
            x[2 * j + 1] += f.y;
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = rbf(x[j]);
    if (epi == EPI_RESIDUAL || epi == EPI_BIAS_RESIDUAL) {
        const uint4 rr = *reinterpret_cast<const uint4*>(residual + (size_t)row * ldr + col);
        const uint32_t rw[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = unpack_bf16x2(rw[j]);
            x[2 * j] += f.x;
            x[2 * j + 1] += f.y;
        }
    }
    uint4 o;
    o.x = pack_bf16x2(x[0], x[1]);
    o.y = pack_bf16x2(x[2], x[3]);
    o.z = pack_bf16x2(x[4], x[5]);
    o.w = pack_bf16x2(x[6], x[7]);
    *reinterpret_cast<uint4*>(C + (size_t)row * ldc + col) = o;
}

// Split-K for small-M GEMMs whose tile count cannot occupy the SMs (prefill down_proj at M ~ 281: 84 tiles on 148 SMs).
// Bit-exact on integer operands (test_gemm_splitk_exact_integer_operands), whole-model parity with it forced on. Measured on B200: it pays only for long K — down_proj (K = 18944) 86.7 -> 60.9 us,
// while qkv / o_proj (K = 3584) get slower (23 -> 34 us) — so the default applies it for K >= 8192 only.
// LIVECC_B200_GEMM_SPLITK=1 forces it for every eligible shape, =0 disables it.
static int splitk_mode() {
    static const int mode = [] {   // 0 off, 1 forced, 2 default (long K only)
        const char* e = getenv("LIVECC_B200_GEMM_SPLITK");
        return !e ? 2 : (e[0] == '1' ? 1 : (e[0] == '0' ? 0 : 2));
    }();
    return mode;
}
// Into how many ranges (0: not at all)?
static int splitk_ranges(const GemmArgs& a, int num_sms) {
    const int mode = splitk_mode();
    if (!mode || !a.splitk_ws || a.M > 384) return 0;
    if (mode == 2 && a.K < 8192) return 0;
    if (a.epi != EPI_NONE && a.epi != EPI_BIAS && a.epi != EPI_RESIDUAL && a.epi != EPI_BIAS_RESIDUAL) return 0;
    const int block_n = splitk_width(a), m_tiles = (a.M + BLOCK_M - 1) / BLOCK_M, n_tiles = (a.N + block_n - 1) / block_n;
    const int tiles = m_tiles * n_tiles;
    const int nkb = (a.K + BLOCK_K - 1) / BLOCK_K;
    if (tiles * 2 > num_sms) return 0;
    int splits = (2 * num_sms + tiles / 2) / tiles;  // about two work units per CTA
    if (splits > 8) splits = 8;
    if (splits > nkb / 4) splits = nkb / 4;  // >= 4 k-blocks per unit
    while (splits > 1 && (splits - 1) * ((nkb + splits - 1) / splits) >= nkb) --splits;  // no empty split
    while (splits > 1 && (size_t)splits * a.M * a.N * 4 > a.splitk_ws_bytes) --splits;
    return splits < 2 ? 0 : splits;
}
static int run_splitk(const GemmArgs& a, int splits, int num_sms, cudaStream_t stream) {
    GemmArgs p = a;
    p.C = a.splitk_ws;
    p.ldc = a.N;
    p.epi = EPI_PARTIAL_F32;
    p.splits = splits;
    p.bias = nullptr;
    p.residual = nullptr;
    if (int r = launch_cfg<EPI_PARTIAL_F32>(p, splitk_width(a), num_sms, stream)) return r;
    const int64_t threads = (int64_t)a.M * (a.N / 8);
    lcc::count_launch();
    chained(splitk_reduce_kernel, (int)((threads + 255) / 256), 256, 0, stream)(
        (const float*)a.splitk_ws, splits, a.M, a.N, (const bf16*)a.bias, (const bf16*)a.residual, a.ldr, (bf16*)a.C,
        a.ldc, a.epi);
    return cudaGetLastError() == cudaSuccess ? 0 : -13;
}

// The form that a plain product of block_n = 0 takes (a split K in global memory counts as FORM_ONE; splitk_ranges decides on it).
GemmPlan gemm_plan(const GemmArgs& a, int num_sms) {
    GemmPlan p;
    double us = 0.;
    p.width = choose_alone(a.M, a.N, a.K, num_sms, &us);
    const int width = choose_pair(a.M, a.N, a.K, num_sms, us, &us);
    if (width) p.width = width;
    if (width) p.form = FORM_PAIR;
    if (const int ranges = splitk_ranges(a, num_sms)) {
        us = scratch_us(a, ranges, num_sms);
        p.form = FORM_ONE;
    }
    int bm = 0, splits = 0;
    if (splitk_mode() != 1 && a.epi != EPI_PARTIAL_F32 && choose_swap(a.M, a.N, a.K, num_sms, us, &bm, &splits)) p = GemmPlan{FORM_SWAP, bm, splits};
    return p;
}

static int check_args(const GemmArgs& a) {
    if (a.M <= 0 || a.N <= 0 || a.K <= 0) return -1;
    if ((a.K % 8) || (a.lda % 8) || (a.ldb % 8) || (a.N % 8) || (a.ldc % (a.c_f32 ? 4 : 8))) return -2;
    if ((a.epi == EPI_SWIGLU || a.epi == EPI_CLAMP_GLU) && (a.N % 32)) return -3;
    if ((a.epi == EPI_RESIDUAL || a.epi == EPI_BIAS_RESIDUAL || a.epi == EPI_SIGMOID_GATE) && (!a.residual || (a.ldr % 8))) return -4;
    if (a.epi == EPI_SIGMOID_GATE && (((uintptr_t)a.residual % 16) || a.tile_group)) return -4;
    if ((a.epi == EPI_BIAS || a.epi == EPI_BIAS_QUICKGELU || a.epi == EPI_BIAS_GELU ||
         a.epi == EPI_BIAS_RESIDUAL) && !a.bias) return -5;
    if (a.tile_group && a.groups < 1) return -1;
    if (a.batch > 1 && (a.tile_group || (a.K % BLOCK_K) || (a.a_col_stride % 8) || (a.c_col_stride % 8) || a.a_col_stride < 0 || a.c_col_stride < 0)) return -7;
    if (a.c_f32 && (a.epi != EPI_NONE || (a.ldc % 4))) return -8;
    return 0;
}

int gemm_bf16_tn_form(const GemmArgs& a, GemmForm form, int width, int splits, int num_sms, cudaStream_t stream) {
    if (int r = check_args(a)) return r;
    if (a.tile_group || a.batch > 1 || a.c_f32 || a.epi == EPI_SIGMOID_GATE || a.epi == EPI_PARTIAL_F32 || width < 32 || (width % 32)) return -6;
    if (form == FORM_SWAP) {
        if (width > kSwapMax || splits < 1 || splits > kSwapSplits) return -6;
        return launch_epi_swap(a, width, splits, num_sms, stream);
    }
    if (width > 256) return -6;
    return form == FORM_PAIR ? launch_epi2(a, width, num_sms, stream) : launch_epi(a, width, num_sms, stream);
}

static int forced_width() {   // tuning hook (0/unset = model)
    static const int forced = [] { const char* e = getenv("LIVECC_B200_GEMM_BN"); return e ? atoi(e) : 0; }();
    return forced;
}

SumOrder gemm_sum_order(const GemmArgs& a, int num_sms) {
    if (forced_width() <= 0) {
        const GemmPlan p = gemm_plan(a, num_sms);
        if (p.form == FORM_SWAP) return SumOrder{p.splits, false};
    }
    const int ranges = splitk_ranges(a, num_sms);
    return ranges ? SumOrder{ranges, true} : SumOrder{};
}

int gemm_bf16_tn_order(const GemmArgs& a, const SumOrder& order, int num_sms, cudaStream_t stream) {
    if (int r = check_args(a)) return r;
    if (a.tile_group || a.batch > 1 || a.c_f32 || a.block_n || a.epi == EPI_SIGMOID_GATE) return -6;
    if (gemm_sum_order(a, num_sms) == order) return gemm_bf16_tn(a, num_sms, stream);
    if (order.ranges == 1) {
        double us = 0.;
        const int alone = choose_alone(a.M, a.N, a.K, num_sms, &us), pair = choose_pair(a.M, a.N, a.K, num_sms, us, &us);
        return pair ? launch_epi2(a, pair, num_sms, stream) : launch_epi(a, alone, num_sms, stream);
    }
    // as many rows at a time as the scratch, or one wave of clusters, holds. Ranges of equal length may go either way with the same bits (ascending sums
    // of the same parts, the same roundings behind them); rows that take several waves of clusters are faster through the scratch: two
    // sequences of 281 rows, x 3584 x 3584 and x 3584 x 18944 together 146 us by clusters, 104 by the scratch.
    const int nkb = (a.K + BLOCK_K - 1) / BLOCK_K, n_tiles = (a.N + 2 * BLOCK_M - 1) / (2 * BLOCK_M);
    const bool can_scratch = order.scratch || (a.splitk_ws && nkb % order.ranges == 0 && (a.epi == EPI_NONE || a.epi == EPI_BIAS || a.epi == EPI_RESIDUAL || a.epi == EPI_BIAS_RESIDUAL));
    const int scratch_rows = can_scratch ? (int)std::min<size_t>(a.splitk_ws_bytes / ((size_t)order.ranges * a.N * 4), 1 << 20) / BLOCK_M * BLOCK_M : 0;
    bool scratch = order.scratch;
    int rows = scratch_rows, bm = kSwapMax;
    if (!scratch) {
        auto fits = [&](int h) { const SwapTile t = make_swap(h, order.ranges); return h * BLOCK_M * 4 <= t.stages * t.stage_bytes; };
        while (bm > 32 && !fits(bm)) bm -= 32;
        rows = max_clusters(current_device(), order.ranges, num_sms) / n_tiles * bm;
        if (rows > 0 && scratch_rows > 0) {
            const int launches = (a.M + rows - 1) / rows, h = std::min(bm, (std::min(rows, a.M) + 31) / 32 * 32);
            const double clusters_us = launches * swap_us(h, 1, (nkb + order.ranges - 1) / order.ranges, order.ranges);
            if (a.M > rows && scratch_us(a, order.ranges, num_sms) < clusters_us) { scratch = true; rows = scratch_rows; }
        }
    }
    if (rows < 1) return -15;
    for (int m0 = 0; m0 < a.M; m0 += rows) {
        GemmArgs p = a;
        p.M = std::min(rows, a.M - m0);
        p.A = (const bf16*)a.A + (size_t)m0 * a.lda;
        p.C = (bf16*)a.C + (size_t)m0 * a.ldc;
        if (a.residual) p.residual = (const bf16*)a.residual + (size_t)m0 * a.ldr;
        const int tiles = (p.M + bm - 1) / bm;
        if (int r = scratch ? run_splitk(p, order.ranges, num_sms, stream)
                            : launch_epi_swap(p, ((p.M + tiles - 1) / tiles + 31) / 32 * 32, order.ranges, num_sms, stream))
            return r;
    }
    return 0;
}

int gemm_bf16_tn(const GemmArgs& a, int num_sms, cudaStream_t stream) {
    if (int r = check_args(a)) return r;
    const bool plain = !a.tile_group && a.batch <= 1 && !a.c_f32;
    const int forced = forced_width();
    const bool choose = plain && a.block_n == 0 && forced <= 0 && a.epi != EPI_SIGMOID_GATE;
    int width = 0;
    if (choose) {
        const GemmPlan p = gemm_plan(a, num_sms);
        if (p.form == FORM_SWAP) return launch_epi_swap(a, p.width, p.splits, num_sms, stream);
        width = p.form == FORM_PAIR ? -p.width : p.width;
    }
    if (plain)
        if (const int ranges = splitk_ranges(a, num_sms)) return run_splitk(a, ranges, num_sms, stream);
    int block_n = a.block_n;
    if (block_n == 0) block_n = forced > 0 ? forced : (width ? width : choose_bn(a.M, a.N, num_sms));
    // block_n < 0: the CTA pair's kernel with tile width -block_n
    const bool pair = block_n < 0 && plain && a.epi != EPI_SIGMOID_GATE && (a.epi <= EPI_SWIGLU || block_n % 32 == 0);
    if (block_n < 0) block_n = -block_n;
    if (block_n < 32 || block_n > 256 || (block_n % 16) || ((a.epi == EPI_SWIGLU || a.epi == EPI_CLAMP_GLU) && (block_n % 32))) return -6;
    if (pair) return (block_n % 32) ? -6 : launch_epi2(a, block_n, num_sms, stream);
    if (a.c_f32) {   // the fp32 tile store of the split-K instantiation, as one split
        GemmArgs p = a;
        p.splits = 1;
        return a.logits ? launch_cfg<EPI_LOGITS_F32>(p, block_n, num_sms, stream) : launch_cfg<EPI_PARTIAL_F32>(p, block_n, num_sms, stream);
    }
    return launch_epi(a, block_n, num_sms, stream);
}

}  // namespace lcc
