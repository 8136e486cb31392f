// General-shape linear layers: C[M,N] = A[M,K] x W[N,K]^T (+ bias), fp32 accumulation, bf16 or fp32 storage.
// Two CUDA-core kernels cover every shape the tensor-core GEMM (gemm_tcgen05.cu) does not take: ragged N or K, fp32
// storage (true fp32 FMAs, no reduced-precision matrix mode), and the few-row case of a decode step, where the
// weight matrix is streamed once and every row of A is multiplied against it (HBM-bound).
#include <type_traits>
#include "common.cuh"
#include "launch.h"
#include "seqmix.h"

namespace lcc {
namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<bf16>(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

constexpr int BM = 64, BN = 64, BK = 16;

// One of several independent problems per blockIdx.z (plain calls: one group, no lists). With row_off the group's rows are
// row_off[z] .. row_off[z+1]-1 of C and of the row list a_rows (or of A itself).
struct Grp {
    int64_t a_stride, w_stride, c_stride;
    const int* row_off;
    const int* a_rows;
    int act;
    int compact;   // few-row kernel with lists: blockIdx.y counts the non-empty lists of `compact` groups (0: blockIdx.y is the group)
    int glu_F;     // few-row kernel, GLU form: a warp owns output column n = the gate row and the up row of that column
    int glu_il16;
    float glu_limit;
    float glu_alpha, glu_up_bias;   // g * sigmoid(alpha g) * (u + up_bias)
    const void* gate = nullptr;     // the store multiplies by sigmoid(gate[row, z * gate_stride + column]) (no lists)
    int ld_gate = 0;
    int64_t gate_stride = 0;
    float cap = 0.f, inv_cap = 0.f, scale = 0.f;   // logits (few-row kernel, LOGITS): the store holds cap * tanh(v / cap) * scale (no cap: v * scale)
    float* copy = nullptr;                         // ... and a second time here, rows as in C
};
template <typename T>
__device__ __forceinline__ float gated(float v, const Grp& g, int z, int row, int col) {
    if (!g.gate) return v;
    return v / (1.f + expf(-ldf((const T*)g.gate + (size_t)row * g.ld_gate + z * g.gate_stride + col)));
}
__device__ __forceinline__ float act_of(float v, int act) {
    if (act == ACT_RELU2) { v = fmaxf(v, 0.f); v *= v; }
    else if (act == ACT_GELU_ERF) v = 0.5f * v * (1.f + erff(v * 0.7071067811865476f));
    else if (act == ACT_GELU_TANH) v = 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
    return v;
}

// 64 x 64 output tile per CTA, 256 threads x (4 x 4) accumulators, k-slices of 16 staged in shared memory as fp32.
template <typename T, typename TC>
__global__ void __launch_bounds__(256) linear_tile_kernel(const T* __restrict__ A, int lda, const T* __restrict__ W, int ldw,
                                                          const float* __restrict__ bias, TC* __restrict__ C, int ldc, int M,
                                                          int N, int K, Grp g) {
    chain_begin(A);
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    int row0 = 0;
    if (g.row_off) {
        row0 = g.row_off[blockIdx.z];
        M = g.row_off[blockIdx.z + 1] - row0;
        if (m0 >= M) return;
    }
    A += blockIdx.z * g.a_stride; W += blockIdx.z * g.w_stride; C += blockIdx.z * g.c_stride + (size_t)row0 * ldc;
    const int* arow = g.a_rows ? g.a_rows + row0 : nullptr;
    if (!arow) A += (size_t)row0 * lda;
    const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 rows x 16 k per operand = 1024 elements, 4 per thread; consecutive threads read consecutive k (coalesced)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + i * 256, r = e / BK, k = e % BK;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + k;
            As[k][r] = (gm < M && gk < K) ? ldf(A + (size_t)(arow ? arow[gm] : gm) * lda + gk) : 0.f;
            Ws[k][r] = (gn < N && gk < K) ? ldf(W + (size_t)gn * ldw + gk) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { a[i] = As[k][tm + i]; w[i] = Ws[k][tn + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + tm + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tn + j;
            if (gn < N) stf(C + (size_t)gm * ldc + gn, gated<T>(act_of(acc[i][j] + (bias ? bias[gn] : 0.f), g.act), g, blockIdx.z, gm, gn));
        }
    }
}

// Few rows (M <= 8), the shape of a decode step: the weight matrix is streamed once (HBM-bound; small matrices are bound by the latency
// of one memory round trip). A warp owns WR output columns and keeps WR x WU independent 16-byte non-allocating loads of their weight
// rows in flight per lane before it touches the activations (which stay in L1); lanes stride over k and keep one accumulator per
// (column, row of A), so the order of a column's sum does not depend on WR, WU or M. MM is the number of rows the accumulators hold: with
// accumulators and addresses for eight rows a one-row step had the registers for four loads per weight row only: 32 tokens of four
// recurrent layers of width 2048 took 10.93 ms and take 8.68 ms, of two routed layers 6.34 and 5.06 ms.
// KS: warps that share a group of columns, each with every KS-th piece of k; their sums meet in shared memory in a fixed order. A warp of one column reads
// as much of A from L1 as of W from memory and unpacks both; two columns and half of k halve that with the same loads in flight.
// LOGITS: the store caps, scales and copies (a form of its own: tanh in every fp32 store cost the others registers, two rows of 16 x 8448 26 us for 12).
// Scalar loads when K or a row start is not 16-byte aligned.
constexpr int kRowsMax = kLogitRows;
template <typename T> struct Vec16;
template <> struct Vec16<bf16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4& u, float (&v)[8]) {
        const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
    }
};
template <> struct Vec16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(const uint4& u, float (&v)[4]) {
        v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
    }
};

template <typename T, typename TC, bool VEC, int MM, int WR, int WU, bool GLU = false, int KS = 1, bool LOGITS = false>
__global__ void __launch_bounds__(256) linear_rows_kernel(const T* __restrict__ A, int lda, const T* __restrict__ W, int ldw,
                                                          const float* __restrict__ bias, TC* __restrict__ C, int ldc, int M_all,
                                                          int N, int K, Grp g) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = warp % KS;
    const int n0 = (blockIdx.x * ((blockDim.x >> 5) / KS) + warp / KS) * (GLU ? 1 : WR);
    if (KS == 1 && n0 >= N) return;     // (with KS > 1 all warps meet below; columns past the end read the last one and store nothing)
    int row0 = 0, z = blockIdx.y;
    constexpr int V = Vec16<T>::N;
    // the weight row behind accumulator r: output columns n0, n0 + 1, ...; in the GLU form (WR = 2) the gate row (r = 0) and
    // the up row (r = 1) of output column n0
    auto wrow = [&](int r) -> int {
        if (GLU) return g.glu_il16 ? ((n0 >> 4) << 5) + (n0 & 15) + 16 * r : n0 + r * g.glu_F;
        return min(n0 + r, N - 1);
    };
    uint4 wq[WR][WU];
    auto load_weights = [&](int kb) {
#pragma unroll
        for (int r = 0; r < WR; ++r)
#pragma unroll
            for (int u = 0; u < WU; ++u) {
                const int k = kb + u * 32 * V * KS;
                wq[r][u] = k < K ? ld_stream16(W + (size_t)wrow(r) * ldw + k) : make_uint4(0, 0, 0, 0);
            }
    };
    // Which weights it reads is known before the kernel in front has finished: their first loads don't wait for it. (Up to two rows: with
    // eight, the loads held across the row addresses cost 18 registers and 5 to 10 % of the routed products of 8 to 24 rows.)
    constexpr bool EARLY = VEC && MM <= 2;
    bool loaded = false;
    if (EARLY && !g.row_off) {
        W += z * g.w_stride;
        load_weights((part * 32 + lane) * V);
        loaded = true;
    }
    chain_begin(A);
    if (g.row_off) {
        if (g.compact) {
            // a decode step routes a handful of rows to a handful of lists: the grid has one y per possible non-empty list
            int seen = -1;
            for (z = 0; z < g.compact; ++z)
                if (g.row_off[z + 1] > g.row_off[z] && ++seen == (int)blockIdx.y) break;
            if (z == g.compact) return;
        }
        row0 = g.row_off[z];
        M_all = g.row_off[z + 1] - row0;
    }
    const T* A0 = A + z * g.a_stride;
    if (!EARLY || !loaded) W += z * g.w_stride;
    TC* C0 = C + z * g.c_stride + (size_t)row0 * ldc;
    const int* arow = g.a_rows ? g.a_rows + row0 : nullptr;
    if (!arow) A0 += (size_t)row0 * lda;
    // a group with more than MM rows walks them in blocks (the weights come from L2 after the first block); a row's
    // sum is the same whatever block it falls into
    for (int mb = 0; mb < M_all; mb += MM) {
    const int M = min(MM, M_all - mb);
    const T* arp[MM];
#pragma unroll
    for (int m = 0; m < MM; ++m) arp[m] = A0 + (size_t)(m < M ? (arow ? arow[mb + m] : mb + m) : 0) * lda;
    C = C0 + (size_t)mb * ldc;
    float acc[WR][MM];
#pragma unroll
    for (int r = 0; r < WR; ++r)
#pragma unroll
        for (int m = 0; m < MM; ++m) acc[r][m] = 0.f;
    if (VEC) {
        for (int kb = (part * 32 + lane) * V; kb < K; kb += 32 * V * WU * KS) {
            if (!EARLY || !loaded) load_weights(kb);
            loaded = false;
#pragma unroll
            for (int u = 0; u < WU; ++u) {
                const int k = min(kb + u * 32 * V * KS, K - V);      // past the end the weights are zero; keep the address valid
                float wv[WR][V];
#pragma unroll
                for (int r = 0; r < WR; ++r) Vec16<T>::unpack(wq[r][u], wv[r]);
#pragma unroll
                for (int m = 0; m < MM; ++m) {
                    if (m < M) {
                        float av[V];
                        Vec16<T>::unpack(*reinterpret_cast<const uint4*>(arp[m] + k), av);
#pragma unroll
                        for (int r = 0; r < WR; ++r)
#pragma unroll
                            for (int i = 0; i < V; ++i) acc[r][m] = fmaf(av[i], wv[r][i], acc[r][m]);
                    }
                }
            }
        }
    } else {
        for (int k = part * 32 + lane; k < K; k += 32 * KS) {
#pragma unroll
            for (int r = 0; r < WR; ++r) {
                const float wv = ldf(W + (size_t)wrow(r) * ldw + k);
#pragma unroll
                for (int m = 0; m < MM; ++m)
                    if (m < M) acc[r][m] = fmaf(ldf(arp[m] + k), wv, acc[r][m]);
            }
        }
    }
    if (GLU) {
#pragma unroll
        for (int m = 0; m < MM; ++m) {
            if (m < M) {
                const float gt = fminf(warp_sum(acc[0][m]), g.glu_limit);
                const float up = fminf(fmaxf(warp_sum(acc[WR - 1][m]), -g.glu_limit), g.glu_limit);
                if (lane == 0) stf(C + (size_t)m * ldc + n0, gt / (1.f + expf(-g.glu_alpha * gt)) * (up + g.glu_up_bias));
            }
        }
        continue;
    }
    __shared__ float sums[KS > 1 ? 8 : 1][WR * MM];
    if (KS > 1) {
#pragma unroll
        for (int r = 0; r < WR; ++r)
#pragma unroll
            for (int m = 0; m < MM; ++m) {
                const float v = m < M ? warp_sum(acc[r][m]) : 0.f;
                if (lane == 0) sums[warp][r * MM + m] = v;
            }
        __syncthreads();
        if (part != 0) return;          // (one block of rows: KS > 1 is not for lists)
    }
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const int n = n0 + r;
#pragma unroll
        for (int m = 0; m < MM; ++m) {
            if (m < M) {
                float v = KS > 1 ? sums[warp][r * MM + m] : warp_sum(acc[r][m]);
#pragma unroll
                for (int i = 1; i < KS; ++i) v += sums[KS > 1 ? warp + i : 0][r * MM + m];
                if (lane != 0 || n >= N) continue;
                if constexpr (LOGITS) {
                    const float lg = (g.cap > 0.f ? g.cap * tanhf(v * g.inv_cap) : v) * g.scale;
                    C[(size_t)m * ldc + n] = lg;
                    if (g.copy) g.copy[(size_t)(mb + m) * ldc + n] = lg;
                } else stf(C + (size_t)m * ldc + n, gated<T>(act_of(v + (bias ? bias[n] : 0.f), g.act), g, z, mb + m, n));
            }
        }
    }
    }
}

template <typename T, typename TC, bool LOGITS = false>
int launch_linear(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N, int K,
                  cudaStream_t s, int groups = 1, Grp g = Grp{0, 0, 0, nullptr, nullptr, ACT_NONE, 0, 0, 0, 0.f}, int M_total = 0,
                  void* glu_tmp = nullptr, int ld_tmp = 0) {
    // GLU form: N = glu_F output columns from 2 * glu_F weight rows
    // lists: the row kernel while all groups together have few rows (a decode step routes `top` rows per sequence)
    if (g.row_off ? M_total <= 8 * kRowsMax : M <= kRowsMax) {
        constexpr int V = Vec16<T>::N;
        const bool vec = (K % V) == 0 && (lda % V) == 0 && (ldw % V) == 0 && ((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0 &&
                         (g.a_stride % V) == 0 && (g.w_stride % V) == 0;
        int grid_y = groups;
        if (g.row_off && M_total < groups) { g.compact = groups; grid_y = M_total; }
        count_launch();
        // rows of A that share a weight row: M, or, with lists, at most M of a list's rows (longer lists walk blocks of MM)
        const int mm = M;
#define LCC_ROWS_KS(MMN, WRN, WUN, WARPS, GLUB, KSN)                                                                           \
    do {                                                                                                                       \
        constexpr int per = (WARPS) / (KSN) * (GLUB ? 1 : WRN);                                                                \
        const dim3 grid((N + per - 1) / per, grid_y);                                                                          \
        if (vec) chained(linear_rows_kernel<T, TC, true, MMN, WRN, WUN, GLUB, KSN, LOGITS && !(GLUB)>, grid, WARPS * 32, 0, s)((const T*)A, lda, (const T*)W, ldw, bias, (TC*)C, ldc, M, N, K, g); \
        else chained(linear_rows_kernel<T, TC, false, MMN, WRN, WUN, GLUB, KSN, LOGITS && !(GLUB)>, grid, WARPS * 32, 0, s)((const T*)A, lda, (const T*)W, ldw, bias, (TC*)C, ldc, M, N, K, g);    \
    } while (0)
#define LCC_ROWS(MMN, WRN, WUN, WARPS, GLUB) LCC_ROWS_KS(MMN, WRN, WUN, WARPS, GLUB, 1)
        if (g.glu_F > 0) {
            if constexpr (std::is_same<T, TC>::value) {
                if (mm == 1) LCC_ROWS(1, 2, 8, 2, true);
                else if (mm <= 2) LCC_ROWS(2, 2, 8, 2, true);
                else LCC_ROWS(8, 2, 4, 2, true);
                return cudaGetLastError() == cudaSuccess ? 0 : -100;
            } else {
                return -2;
            }
        }
        // Wide matrices: for one row a column per warp and CTAs of 4 warps, which leave and arrive in small portions; two columns and 8 warps for
        // more rows. Narrower ones: warps share columns, four by four or two by two, so that the whole matrix is in flight at once. How many share
        // depends on the matrix alone, never on M: so do a row's bits. Sharing pays where k is long against what it costs (sums that meet in shared
        // memory) and the columns do not fill the chip by themselves. One | two | four | eight rows in bf16, each warp its own columns -> so, us, products
        // chained as in a step: by four 64 x 2048 2.8 -> 1.8 | 4.7 -> 2.2 | 9.4 -> 4.1 | 16.1 -> 6.2, 2048 x 4096 6.2 -> 4.1 | 10.5 -> 5.8 | 19.6 -> 16.9 |
        // 34.0 -> 26.2, 4096 x 4096 12.4 -> 7.5 | 12.1 -> 11.8 | 38.3 -> 26.6 | 64.4 -> 39.7; by two 2048 x 1024 2.7 -> 2.5 | 4.3 -> 4.0 | 6.8 -> 6.2 | 11.1 -> 9.0,
        // 6208 x 2048 8.4 -> 6.9 | 11.4 -> 10.2 | 21.6 -> 21.9 | 36.3 -> 33.4. It is not free everywhere inside the lines: 4096 x 2048 by two
        // 4.4 -> 4.2 | 6.2 -> 7.5 | 20.5 -> 16.5 | 34.7 -> 25.1, 3000 x 2048 4.3 -> 3.8 | 6.2 -> 4.7 | 11.8 -> 13.5 | 19.3 -> 21.4. Beyond the lines: by four
        // 2048 x 1024 2.8 | 3.4 | 10.0 | 14.4, 4096 x 2048 5.1 | 6.9 | 18.0 | 26.4; by two 6208 x 1024 5.2 | 6.5 | 15.9 | 22.7 for 5.6 | 8.3 | 13.0 | 21.0. In fp32,
        // which costs half as much to unpack, by four 2048 x 2048 3.7 -> 3.5 | 5.8 -> 4.7 | 18.6 -> 15.1 | 28.6 -> 19.7, 2560 x 1024 3.0 -> 2.8 | 3.6 -> 4.3.
        // Longer k in bf16, 2048 x 8448, filled the SMs in front of the attention that runs beside it: a routed step of four sequences 435 us for 404.
        // U: what a warp reads of a row of W at once.
        constexpr int U = 32 * V;
        constexpr bool F32 = sizeof(T) == 4;
        const bool shared_k = !g.row_off && (F32 || K <= 24 * U);
        const bool by4 = shared_k && ((N <= 1024 && K >= 4 * U) || (N <= (F32 ? 2048 : 18 * kSms) && K >= 8 * U) || (!F32 && N <= 4608 && K >= 16 * U));
        const bool by2 = shared_k && K >= (N <= 2048 ? 4 : 6) * U;
        // waves of CTAs in a form that has room for so many columns per SM (by its registers). Eight rows: one of 16 columns costs 4/3 of one of 12
        auto waves = [&](int per_sm) { return (N + per_sm * kSms - 1) / (per_sm * kSms); };
        if (N >= 8192) {
            if (mm == 1) LCC_ROWS(1, 1, 8, 4, false);
            else if (mm <= 2) LCC_ROWS(2, 2, 8, 8, false);
            else LCC_ROWS(8, 2, 4, 8, false);
        } else if (by4) {
            if (mm == 1 && K <= 8 * U) LCC_ROWS_KS(1, 2, 2, 4, false, 4);
            else if (mm == 1) LCC_ROWS_KS(1, 2, 4, 4, false, 4);
            else if (mm <= 2 && N > 1024 && N <= 2048) LCC_ROWS_KS(2, 2, 2, 4, false, 4);
            else if (mm <= 2 && N <= 1024 && K > 8 * U && (!F32 || N > 256)) LCC_ROWS_KS(2, 1, 4, 4, false, 4);
            else if (mm <= 2) LCC_ROWS_KS(2, 1, 2, 4, false, 4);
            else if (N > 6 * kSms && N <= 8 * kSms) LCC_ROWS_KS(8, 2, 2, 4, false, 4);     // one wave of two columns in place of two of one: 1024 x 2048 8.5 -> 6.2 us
            else LCC_ROWS_KS(8, 1, 2, 4, false, 4);
        } else if (by2) {
            if (mm == 1) LCC_ROWS_KS(1, 2, 4, 4, false, 2);
            else if (mm <= 2 && (F32 ? waves(24) <= waves(32) : waves(24) == 1)) LCC_ROWS_KS(2, 2, 4, 4, false, 2);
            else if (mm <= 2) LCC_ROWS_KS(2, F32 ? 2 : 1, F32 ? 2 : 4, 4, false, 2);
            else if (F32 || 4 * waves(16) < 3 * waves(12)) LCC_ROWS_KS(8, 2, 2, 4, false, 2);
            else LCC_ROWS_KS(8, 1, 4, 4, false, 2);
        } else if (mm == 1 && K > 8 * U && N <= 2048) {
            LCC_ROWS(1, 1, 16, 2, false);
        } else if (mm == 1) {
            LCC_ROWS(1, 1, 8, 2, false);          // (16 loads a lane above 2048 columns: 4096 x 3072 11.1 us for 6.9)
        } else if (mm <= 2) {
            LCC_ROWS(2, 1, 8, 2, false);
        } else {
            LCC_ROWS(8, 1, 4, 2, false);
        }
#undef LCC_ROWS_KS
#undef LCC_ROWS
    } else if (g.glu_F > 0) {
        // raw gate and up columns into the caller's scratch, then the activation as a row kernel
        if (!glu_tmp || ld_tmp < 2 * N || !std::is_same<T, TC>::value) return -2;
        Grp raw = g;
        raw.glu_F = 0;
        raw.c_stride = 0;
        dim3 grid((2 * N + BN - 1) / BN, (M + BM - 1) / BM, groups);
        count_launch();
        chained(linear_tile_kernel<T, T>, grid, 256, 0, s)((const T*)A, lda, (const T*)W, ldw, bias, (T*)glu_tmp, ld_tmp, M, 2 * N, K, raw);
        if (cudaGetLastError() != cudaSuccess) return -100;
        const int rows = g.row_off ? M_total : M;
        return glu_clamp_swish(sizeof(T) == 4 ? DT_F32 : DT_BF16, glu_tmp, ld_tmp, C, ldc, rows, N, g.glu_limit, s, g.glu_il16 != 0, g.glu_alpha, g.glu_up_bias);
    } else {
        dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, groups);
        count_launch();
        chained(linear_tile_kernel<T, TC>, grid, 256, 0, s)((const T*)A, lda, (const T*)W, ldw, bias, (TC*)C, ldc, M, N, K, g);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -100;
}

}  // namespace

int linear_any(int dt, const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, bool c_f32,
               int M, int N, int K, cudaStream_t s) {
    if (!A || !W || !C || M < 1 || N < 1 || K < 1 || lda < K || ldw < K || ldc < N) return -2;
    if (dt == DT_F32) return launch_linear<float, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, s);
    if (c_f32) return launch_linear<bf16, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, s);
    return launch_linear<bf16, bf16>(A, lda, W, ldw, bias, C, ldc, M, N, K, s);
}

int linear_logits(int dt, const void* A, int lda, const void* W, int ldw, float* C, float* copy, int ldc, int M, int N, int K, float cap, float scale,
                  cudaStream_t s) {
    if (!A || !W || !C || M < 1 || M > kRowsMax || N < 1 || K < 1 || lda < K || ldw < K || ldc < N || scale == 0.f) return -2;
    Grp g{0, 0, 0, nullptr, nullptr, ACT_NONE, 0, 0, 0, 0.f};
    g.cap = cap > 0.f ? cap : 0.f; g.inv_cap = cap > 0.f ? 1.f / cap : 0.f; g.scale = scale; g.copy = copy;
    if (dt == DT_F32) return launch_linear<float, float, true>(A, lda, W, ldw, nullptr, C, ldc, M, N, K, s, 1, g);
    return launch_linear<bf16, float, true>(A, lda, W, ldw, nullptr, C, ldc, M, N, K, s, 1, g);
}

int linear_grouped(const GroupedLinear& q, cudaStream_t s) {
    if (!q.A || !q.W || !q.C || q.groups < 1 || q.groups > 65535 || q.M < 1 || q.N < 1 || q.K < 1 || q.lda < q.K || q.ldw < q.K ||
        q.ldc < q.N || (q.a_rows && !q.row_off))
        return -2;
    if (q.glu_F > 0 && (q.N != q.glu_F || q.act != ACT_NONE || q.c_f32 || (q.glu_il16 && (q.glu_F % 16)) || q.c_stride != 0 ||
                        (q.groups > 1 && !q.row_off)))
        return -2;
    if (q.gate && (q.row_off || q.glu_F > 0)) return -2;
    const Grp g{q.a_stride, q.w_stride, q.c_stride, q.row_off, q.a_rows, q.act, 0, q.glu_F, q.glu_il16 ? 1 : 0, q.glu_limit, q.glu_alpha, q.glu_up_bias,
                q.gate, q.ld_gate, q.gate_stride};
    const int mt = q.row_off ? (q.M_total > 0 ? q.M_total : q.M * q.groups) : 0;
    if (q.dt == DT_F32) return launch_linear<float, float>(q.A, q.lda, q.W, q.ldw, nullptr, q.C, q.ldc, q.M, q.N, q.K, s, q.groups, g, mt, q.glu_tmp, q.ld_tmp);
    if (q.c_f32) return launch_linear<bf16, float>(q.A, q.lda, q.W, q.ldw, nullptr, q.C, q.ldc, q.M, q.N, q.K, s, q.groups, g, mt);
    return launch_linear<bf16, bf16>(q.A, q.lda, q.W, q.ldw, nullptr, q.C, q.ldc, q.M, q.N, q.K, s, q.groups, g, mt, q.glu_tmp, q.ld_tmp);
}

}  // namespace lcc
