// Projections of a decode step shared by up to 8 streams: y[b] = W x[b], every weight byte read once for all of them. The streams are the
// 8 columns of mma.sync m16n8k16, the weights its 16 rows, straight from global memory into the fragments: a lane's 16-byte load
// is 8 consecutive k of one weight row, and because the same k are loaded of x, which 4 of a product's 16 places they take does not matter.
//
// HBM-bound: 7 TB/s of weights are 24 bytes per clock and SM, two products (512 bytes of weights each) per 43 clocks; eight columns on the CUDA cores would be 96
// multiply-adds per clock and SM beside the unpacking. What a CTA needs is loads in flight: its 8 warps share the K of 16 or 32 rows
// (a round of them reads 1 KB of each row), 8 to 16 loads of 16 bytes per lane, and add their partials through shared memory. x is read through L1.
#include "common.cuh"
#include "launch.h"
#include "mma.cuh"
#include "ops.h"

namespace lcc {

enum { GB_BIAS = 0, GB_RESIDUAL = 1, GB_SWIGLU = 2, GB_LOGITS = 3 };

struct GemvBatchParams {
    const bf16* W;
    const bf16* x;     // [B][ldx]
    int N, K, ldx, B;
    const bf16* bias;  // GB_BIAS
    bf16* out;         // [B][ldo]; GB_RESIDUAL: the residual stream, in and out
    int ldo;
    float *out_f32, *out_f32_b;  // GB_LOGITS [B][ldo], twice
    const int* finished[kBatchStreams];
    const uint8_t* pf_ptr;  // L2 prefetch of the next kernel's weights by this grid's last CTAs (see gemv.cu)
    unsigned pf_bytes;
};

constexpr int kGbWarps = 8;

// Measured with 8 streams (hidden 3584; for comparison one stream's CUDA-core kernels): lm_head 168 us (172), gate/up 43.8 (43), down 25.3 (25),
// qkv 9.0 (11.1, RMSNorm included), o 10.1 (9.6).
// MT: 16-row tiles per CTA (GB_SWIGLU: 16 gate rows and their 16 up rows). UN: units of 64 k in flight.
// CTAs per SM are fixed, or a change of a few registers moves these times by a tenth (the head at 68 registers 170 us).
template <int MT, int UN, int EPI>
__global__ void __launch_bounds__(kGbWarps * 32, EPI == GB_SWIGLU ? 3 : UN > 1 ? 2 : 4) gemv_batch_kernel(const GemvBatchParams p) {
    __shared__ float part[kGbWarps][MT * 128];   // [row][stream] per warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int tile = blockIdx.x, n0 = tile * MT * 16, units = p.K >> 6;
    const bf16* w0 = p.W + (size_t)(n0 + g) * p.K + t * 8;
    const bf16* x0 = p.x + (size_t)(g < p.B ? g : 0) * p.ldx + t * 8;
    float acc[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][i] = 0.f;
    uint4 w[UN][MT][2][2];
    auto load = [&](int u, uint4 (&d)[MT][2][2]) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int r = 0; r < 2; ++r) d[m][r][h] = ld_stream16(w0 + (size_t)(m * 16 + r * 8) * p.K + u * 64 + h * 32);
    };
    auto compute = [&](int u, const uint4 (&d)[MT][2][2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 x = __ldg(reinterpret_cast<const uint4*>(x0 + u * 64 + h * 32));   // (columns past B repeat stream 0 and are not stored)
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const uint32_t a0[4] = {d[m][0][h].x, d[m][1][h].x, d[m][0][h].y, d[m][1][h].y};
                const uint32_t a1[4] = {d[m][0][h].z, d[m][1][h].z, d[m][0][h].w, d[m][1][h].w};
                mma_bf16_16816(acc[m], a0, x.x, x.y);
                mma_bf16_16816(acc[m], a1, x.z, x.w);
            }
        }
    };
    int u = warp;
    const int done = lane < p.B ? *p.finished[lane] : 1;
    bool open = false;
    auto ended = [&] {   // every stream has ended (a replayed graph): nothing to do, seen while the first weights arrive
        if (open || !__all_sync(0xffffffffu, done)) { open = true; return false; }
        return true;
    };
    if constexpr (UN == 1) {   // (the loop turned like this: gate/up 43.8 us, 48.4 as below)
        if (u < units) load(u, w[0]);
        if (ended()) return;
        while (u < units) {
            compute(u, w[0]);
            u += kGbWarps;
            if (u < units) load(u, w[0]);
        }
    } else {
        for (; u + (UN - 1) * kGbWarps < units; u += UN * kGbWarps) {
#pragma unroll
            for (int i = 0; i < UN; ++i) load(u + i * kGbWarps, w[i]);
            if (ended()) return;
#pragma unroll
            for (int i = 0; i < UN; ++i) compute(u + i * kGbWarps, w[i]);
        }
        if (ended()) return;
    }
    if (UN > 1) {
#pragma unroll
        for (int i = 0; i < UN - 1; ++i)
            if (u + i * kGbWarps < units) load(u + i * kGbWarps, w[i]);
#pragma unroll
        for (int i = 0; i < UN - 1; ++i)
            if (u + i * kGbWarps < units) compute(u + i * kGbWarps, w[i]);
    }
    // ---- partials: warps in order ----
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        float* d = part[warp] + m * 128 + g * 8 + t * 2;
        *reinterpret_cast<float2*>(d) = make_float2(acc[m][0], acc[m][1]);
        *reinterpret_cast<float2*>(d + 64) = make_float2(acc[m][2], acc[m][3]);
    }
    __syncthreads();
    if (EPI != GB_LOGITS && p.pf_bytes) {   // (nothing follows the head)
        const unsigned ntail = min(gridDim.x, 296u);
        if (blockIdx.x + ntail >= gridDim.x) {
            const unsigned lines = (p.pf_bytes + 127u) >> 7, per = (lines + ntail - 1) / ntail;
            const unsigned l0 = (blockIdx.x - (gridDim.x - ntail)) * per, l1 = min(lines, l0 + per);
            for (unsigned l = l0 + threadIdx.x; l < l1; l += kGbWarps * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pf_ptr + (size_t)l * 128));
        }
    }
    const int i = threadIdx.x;   // one (row, stream) per thread; MT = 2 uses all 256
    float sum = 0.f;
    if (i < MT * 128) {
#pragma unroll
        for (int k = 0; k < kGbWarps; ++k) sum += part[k][i];
    }
    if (EPI == GB_SWIGLU) {   // rows 0..15 gate, 16..31 up
        __syncthreads();
        part[0][i] = sum;
        __syncthreads();
        if (i >= 128) return;
    }
    if (i >= MT * 128) return;
    const int b = i & 7, r = i >> 3;
    if (b >= p.B || *p.finished[b]) return;
    if (EPI == GB_SWIGLU) {
        const float gt = rbf(sum), up = rbf(part[0][i + 128]);
        const float sl = rbf(gt / (1.0f + expf(-gt)));
        p.out[(size_t)b * p.ldo + tile * 16 + r] = f2bf(sl * up);
        return;
    }
    const int n = n0 + r;
    const size_t o = (size_t)b * p.ldo + n;
    if (EPI == GB_BIAS) p.out[o] = f2bf(sum + bf2f(p.bias[n]));
    else if (EPI == GB_RESIDUAL) p.out[o] = f2bf(rbf(sum) + bf2f(p.out[o]));
    else { const float v = rbf(sum); p.out_f32[o] = v; p.out_f32_b[o] = v; }
}

template <int MT, int UN, int EPI>
static int launch_batch(const GemvBatchParams& p, cudaStream_t s) {
    if (p.B < 1 || p.B > kBatchStreams || p.N % (MT * 16) || p.K % 64 || p.ldx % 8) return -1;
    count_launch();
    gemv_batch_kernel<MT, UN, EPI><<<p.N / (MT * 16), kGbWarps * 32, 0, s>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

static GemvBatchParams params_of(const GemvBatch& a) {
    GemvBatchParams p{};
    p.W = a.W; p.x = a.x; p.N = a.N; p.K = a.K; p.ldx = a.ldx; p.B = a.B;
    for (int b = 0; b < a.B && b < kBatchStreams; ++b) p.finished[b] = a.finished[b];
    p.pf_ptr = (const uint8_t*)a.pf_ptr; p.pf_bytes = (unsigned)a.pf_bytes;
    return p;
}

int gemv_batch_bias(const GemvBatch& a, const bf16* bias, bf16* out, int ldo, cudaStream_t s) {
    GemvBatchParams p = params_of(a);
    p.bias = bias; p.out = out; p.ldo = ldo;
    return launch_batch<1, 4, GB_BIAS>(p, s);
}
int gemv_batch_residual(const GemvBatch& a, bf16* h_inout, int ldo, cudaStream_t s) {
    GemvBatchParams p = params_of(a);
    p.out = h_inout; p.ldo = ldo;
    // (Two CTAs per tile, sharing K through a cluster, was taken for K > 8192: at two CTAs per SM it never pays, N x K = 1536 to 8192 x 1536 to 27648,
    // 8 streams: 3584 x 18944 26.4 us either way, 25.3 for 27.0 in a step, 2560 x 18944 22.2 | 21.8, 7168 x 18944 49.6 | 52.2, 1536 x 18944 17.0 | 19.2.)
    return launch_batch<1, 4, GB_RESIDUAL>(p, s);
}
int gemv_batch_swiglu(const GemvBatch& a, bf16* act, int ldo, cudaStream_t s) {
    GemvBatchParams p = params_of(a);
    p.out = act; p.ldo = ldo;
    return launch_batch<2, 1, GB_SWIGLU>(p, s);   // (2 units in flight were slower: registers)
}
int gemv_batch_logits(const GemvBatch& a, float* logits, float* logits_copy, int ldo, cudaStream_t s) {
    GemvBatchParams p = params_of(a);
    p.out_f32 = logits; p.out_f32_b = logits_copy; p.ldo = ldo;
    return launch_batch<2, 1, GB_LOGITS>(p, s);
}

}  // namespace lcc
