// HBM-bound row kernels of the LiveCC path: casts, LayerNorm, RMSNorm, ViT 2-D rotary, M-RoPE +
// paged-KV append, embedding gather/scatter. Coalesced, mostly 16-byte accesses; grids sized from the row count.
#include <algorithm>

#include "common.cuh"
#include "launch.h"
#include "ops.h"

namespace lcc {

// ------------------------------------------------------------------------------------------
// f32 -> bf16 (pixel_values_videos.to(bf16), mq2vl.py:309)
// ------------------------------------------------------------------------------------------
__global__ void cast_f32_bf16_kernel(const float* __restrict__ in, bf16* __restrict__ out, int64_t n) {
    int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x * 8;
    for (; i + 8 <= n; i += stride) {
        float4 a = *reinterpret_cast<const float4*>(in + i);
        float4 b = *reinterpret_cast<const float4*>(in + i + 4);
        uint4 o;
        o.x = pack_bf16x2(a.x, a.y); o.y = pack_bf16x2(a.z, a.w);
        o.z = pack_bf16x2(b.x, b.y); o.w = pack_bf16x2(b.z, b.w);
        *reinterpret_cast<uint4*>(out + i) = o;
    }
    // tail (n % 8): handled by the first threads
    if (blockIdx.x == 0 && threadIdx.x < (n & 7)) {
        int64_t j = (n & ~int64_t(7)) + threadIdx.x;
        out[j] = f2bf(in[j]);
    }
}

// Ids, positions and scalars of the turns of one call (blockIdx.y: the stream). As separate copies (one of them from pageable host memory, which waits)
// and small launches they kept the device idle for some 50 us in front of every stream's turn (a turn that reads 281 tokens 1.47 ms, 1.42 so; eight streams 12.26 and 11.92).
constexpr int kTurns = 8;
struct TurnBatch { lcc_turn t[kTurns]; };
__global__ void turn_setup_kernel(const __grid_constant__ TurnBatch b) {
    const lcc_turn& t = b.t[blockIdx.y];
    const int at = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (int i = at; i < t.L; i += step) t.seq[i] = t.ids[i];
    if (t.pos3)
        for (int i = at; i < t.S; i += step) t.pos3[i] = t.pos3[t.S + i] = t.pos3[2 * t.S + i] = t.pos_base + i;
    if (at < 8) t.scalars[at] = t.values[at];
}
int turn_setup(const lcc_turn* turns, int n, cudaStream_t s) {
    if (!turns || n < 1 || n > kTurns) return -2;
    TurnBatch b{};
    int longest = 1;
    for (int i = 0; i < n; ++i) {
        const lcc_turn& t = b.t[i] = turns[i];
        if (!t.ids || !t.seq || t.L < 1 || (t.pos3 && t.S < 1) || !t.scalars) return -2;
        longest = std::max(longest, t.L);
    }
    lcc::count_launch();
    turn_setup_kernel<<<dim3(std::min((longest + 255) / 256, 2 * kSms), n), 256, 0, s>>>(b);
    return 0;
}

int cast_f32_bf16(const float* in, bf16* out, int64_t n, int num_sms, cudaStream_t s) {
    if (n <= 0) return 0;
    int64_t blocks = (n / 8 + 255) / 256;
    if (blocks < 1) blocks = 1;
    if (blocks > (int64_t)num_sms * 16) blocks = (int64_t)num_sms * 16;
    { lcc::count_launch(); cast_f32_bf16_kernel<<<(int)blocks, 256, 0, s>>>(in, out, n); }
    return 0;
}

// ------------------------------------------------------------------------------------------
// GPU frame ingest: uint8 frames [T,3,H,W] -> bf16 patch rows [N, 3*2*14*14] in one pass,
// replacing the host-side rescale/normalize/patchify of Qwen2VLVideoProcessor._preprocess
// (video_processing_qwen2_vl.py:240-272; fused mean/std: image_processing_backends.py:301-304,327) plus the
// f32 H2D copy and the bf16 cast (mq2vl.py:309). Bit-identical to cast_bf16(host patchify): the value is
// bf16( (float(u8) - mean255[c]) / std255[c] ) with IEEE fp32 subtract and divide; odd T repeats the last frame.
// Row order (t, h/2, w/2, 2, 2), column order (c, tp, 14, 14).
// ------------------------------------------------------------------------------------------
// A value depends on its byte and its channel only, so a CTA computes the 3 x 256 values once (the divisions are what a thread per pixel
// pair spent its time on, beside 64-bit index divisions and 4-byte stores: 8.7 us for 1024 patches and 44 for 8192, now 6.9 and 21) and looks them up; a thread takes a 14-pixel
// row of a patch, and a group of patch rows leaves through shared memory as 16-byte stores.
constexpr int kPatchRows = 8;   // patch rows per CTA
template <bool PAIRS>           // two bytes per load: frames at an even address (W and the patch size are even)
__global__ void __launch_bounds__(256) patchify_u8_kernel(const uint8_t* __restrict__ frames, int T, int H, int W, int rows,
                                                          bf16* __restrict__ out, float m0, float m1, float m2, float s0, float s1,
                                                          float s2) {
    constexpr int P = 14, TP = 2, MS = 2, COLS = 3 * TP * P * P, LINES = 3 * TP * P;
    __shared__ uint16_t value[3][256];
    __shared__ __align__(16) uint32_t tile[kPatchRows][COLS / 2];
    const int gw = W / P, wbn = gw / MS, hbn = H / (P * MS);
    const int row0 = blockIdx.x * kPatchRows, n = min(kPatchRows, rows - row0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float mean = c == 0 ? m0 : (c == 1 ? m1 : m2), sd = c == 0 ? s0 : (c == 1 ? s1 : s2);
        value[c][threadIdx.x] = __bfloat16_as_ushort(f2bf(__fdiv_rn(__fsub_rn((float)threadIdx.x, mean), sd)));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * LINES; i += 256) {
        const int r = i / LINES, line = i % LINES, row = row0 + r;
        // row -> (t, hb, wb, hi, wi); line -> (c, tp, py)
        const int in_win = row % (MS * MS), win = row / (MS * MS);
        const int wb = win % wbn, hb = (win / wbn) % hbn, t = win / (wbn * hbn);
        const int ph = hb * MS + in_win / MS, pw = wb * MS + in_win % MS;
        const int py = line % P, tp = (line / P) % TP, c = line / (P * TP);
        const int tf = min(t * TP + tp, T - 1);
        const uint8_t* src = frames + (((size_t)tf * 3 + c) * H + (size_t)ph * P + py) * W + (size_t)pw * P;
        uint32_t px[P / 2];
#pragma unroll
        for (int k = 0; k < P / 2; ++k)
            px[k] = PAIRS ? (uint32_t)reinterpret_cast<const uint16_t*>(src)[k] : (uint32_t)src[2 * k] | ((uint32_t)src[2 * k + 1] << 8);
#pragma unroll
        for (int k = 0; k < P / 2; ++k)
            tile[r][line * (P / 2) + k] = (uint32_t)value[c][px[k] & 255u] | ((uint32_t)value[c][px[k] >> 8] << 16);
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)row0 * COLS);
    const uint4* st = reinterpret_cast<const uint4*>(&tile[0][0]);
    for (int i = threadIdx.x; i < n * (COLS / 8); i += 256) dst[i] = st[i];
}

int patchify_u8(const uint8_t* frames, int T, int H, int W, bf16* out, const float* mean255, const float* std255,
                cudaStream_t s) {
    if (T <= 0 || H % 28 || W % 28) return -1;
    const int rows = (T + 1) / 2 * (H / 14) * (W / 14), blocks = (rows + kPatchRows - 1) / kPatchRows;
    lcc::count_launch();
    if ((uintptr_t)frames % 2 == 0)
        patchify_u8_kernel<true><<<blocks, 256, 0, s>>>(frames, T, H, W, rows, out, mean255[0], mean255[1], mean255[2], std255[0], std255[1], std255[2]);
    else
        patchify_u8_kernel<false><<<blocks, 256, 0, s>>>(frames, T, H, W, rows, out, mean255[0], mean255[1], mean255[2], std255[0], std255[1], std255[2]);
    return 0;
}

// ------------------------------------------------------------------------------------------
// LayerNorm over rows (nn.LayerNorm eps=1e-6, mq2vl.py:464-465,317): fp32 two-pass statistics, y = bf16((x - mean) * rstd * w + b).
// RMSNorm over rows (Qwen2VLRMSNorm, mq2vl.py:126-131): y = w * bf16(x * rsqrt(mean(x^2) + eps)).
// dim % 8 == 0. The rows of a step are few and short, so latency bounds them: a row is read once, all of its 16-byte loads (and those of
// the weights) in flight together, and stays in registers through the passes. The team depends on the width alone, so a row's sums do
// not depend on how many rows there are. With a warp per row and three passes over memory, an RMSNorm of 24 rows of 3584 took 5.3 us
// back to back, of 281 rows 5.7 and of 2090 rows 8.1; now 1.9, 2.6 and 7.7.
// Columns beyond what the registers hold (TEAM x 8 x KEEP) are read again in each pass.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float sum8(const uint4& u) {
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
    return ((a.x + a.y) + (b.x + b.y)) + ((c.x + c.y) + (d.x + d.y));
}
__device__ __forceinline__ float dev8(const uint4& u, float mean) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(w[j]);
        const float d0 = f.x - mean, d1 = f.y - mean;
        s = fmaf(d0, d0, fmaf(d1, d1, s));
    }
    return s;
}
template <bool RMS>
__device__ __forceinline__ uint4 norm8(const uint4& u, const uint4& wv, const uint4& bv, float mean, float r) {
    const uint32_t uw[4] = {u.x, u.y, u.z, u.w}, ww[4] = {wv.x, wv.y, wv.z, wv.w}, bw[4] = {bv.x, bv.y, bv.z, bv.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(uw[j]), g = unpack_bf16x2(ww[j]);
        if (RMS) {
            o[j] = pack_bf16x2(g.x * rbf(f.x * r), g.y * rbf(f.y * r));
        } else {
            const float2 h = unpack_bf16x2(bw[j]);
            o[j] = pack_bf16x2((f.x - mean) * r * g.x + h.x, (f.y - mean) * r * g.y + h.y);
        }
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// Sum over the CTA, the same in all threads: per lane over the warps, then over the lanes. Buffers alternate, so one barrier is enough.
template <int TEAM>
__device__ __forceinline__ float team_sum(float v, float (&red)[2][TEAM / 32][32], int& flip) {
    const int lane = threadIdx.x & 31;
    red[flip][threadIdx.x >> 5][lane] = v;
    __syncthreads();
    float t = red[flip][0][lane];
#pragma unroll
    for (int i = 1; i < TEAM / 32; ++i) t += red[flip][i][lane];
    flip ^= 1;
    return warp_sum(t);
}

template <bool RMS, int TEAM, int KEEP>   // KEEP: 16-byte pieces of a row per thread
__global__ void __launch_bounds__(TEAM) norm_rows_kernel(const bf16* __restrict__ x, int ldx, const bf16* __restrict__ w,
                                                         const bf16* __restrict__ b, bf16* __restrict__ y, int ldy, int rows, int dim,
                                                         float eps) {
    chain_begin(x);
    __shared__ float red[2][TEAM / 32][32];
    int flip = 0;
    constexpr int STEP = TEAM * 8;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 next[KEEP], wv[KEEP], bv[KEEP];
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
        const int c = threadIdx.x * 8 + i * STEP;
        next[i] = wv[i] = bv[i] = zero;
        if (c >= dim) continue;
        next[i] = *reinterpret_cast<const uint4*>(x + (size_t)blockIdx.x * ldx + c);
        wv[i] = *reinterpret_cast<const uint4*>(w + c);
        if (!RMS) bv[i] = *reinterpret_cast<const uint4*>(b + c);
    }
    const int rest = threadIdx.x * 8 + KEEP * STEP;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const bf16* xr = x + (size_t)row * ldx;
        bf16* yr = y + (size_t)row * ldy;
        uint4 u[KEEP];
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const int c = threadIdx.x * 8 + i * STEP;
            u[i] = next[i];
            if (c < dim && row + (int)gridDim.x < rows) next[i] = *reinterpret_cast<const uint4*>(xr + (size_t)gridDim.x * ldx + c);
        }
        float mean = 0.f;
        if (!RMS) {
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < KEEP; ++i) sum += sum8(u[i]);
            for (int c = rest; c < dim; c += STEP) sum += sum8(*reinterpret_cast<const uint4*>(xr + c));
            mean = team_sum<TEAM>(sum, red, flip) / (float)dim;
        }
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if ((int)threadIdx.x * 8 + i * STEP < dim) sq += dev8(u[i], mean);
        for (int c = rest; c < dim; c += STEP) sq += dev8(*reinterpret_cast<const uint4*>(xr + c), mean);
        const float r = rsqrtf(team_sum<TEAM>(sq, red, flip) / (float)dim + eps);
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const int c = threadIdx.x * 8 + i * STEP;
            if (c < dim) *reinterpret_cast<uint4*>(yr + c) = norm8<RMS>(u[i], wv[i], bv[i], mean, r);
        }
        for (int c = rest; c < dim; c += STEP)
            *reinterpret_cast<uint4*>(yr + c) = norm8<RMS>(*reinterpret_cast<const uint4*>(xr + c), *reinterpret_cast<const uint4*>(w + c),
                                                           RMS ? zero : *reinterpret_cast<const uint4*>(b + c), mean, r);
    }
}

// Many rows of up to 1536 columns: a warp per row needs no barrier. Its sums run as a team's above do, so a row's result does not depend on
// the form. 8192 rows of 1280: 14.3 us, 18.4 as teams of 192; 1024 rows: 6.3 us (profiled), 4.7 as teams. Four CTAs per SM: without the bound the layer
// norm takes 80 registers, room for three (repeated 8.1 and 9.1 us, 4096 rows 5.2 and 6.7).
template <bool RMS>
__global__ void __launch_bounds__(256, 4) norm_rows_warp_kernel(const bf16* __restrict__ x, int ldx, const bf16* __restrict__ w,
                                                             const bf16* __restrict__ b, bf16* __restrict__ y, int ldy, int rows, int dim,
                                                             float eps) {
    chain_begin(x);
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const bf16* xr = x + (size_t)row * ldx;
    bf16* yr = y + (size_t)row * ldy;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 u[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const int c = lane * 8 + i * 256;
        u[i] = c < dim ? *reinterpret_cast<const uint4*>(xr + c) : zero;
    }
    float mean = 0.f;
    if (!RMS) {
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 6; ++i) sum += sum8(u[i]);
        mean = warp_sum(sum) / (float)dim;
    }
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < 6; ++i) sq += lane * 8 + i * 256 < dim ? dev8(u[i], mean) : 0.f;
    const float r = rsqrtf(warp_sum(sq) / (float)dim + eps);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const int c = lane * 8 + i * 256;
        if (c < dim)
            *reinterpret_cast<uint4*>(yr + c) = norm8<RMS>(u[i], *reinterpret_cast<const uint4*>(w + c), RMS ? zero : *reinterpret_cast<const uint4*>(b + c), mean, r);
    }
}

template <bool RMS>
static int norm_rows(const bf16* x, int ldx, const bf16* w, const bf16* b, bf16* y, int ldy, int rows, int dim, float eps, cudaStream_t s) {
    if (rows <= 0) return 0;
    if (dim % 8 || ldx % 8 || ldy % 8) return -1;
    lcc::count_launch();
    // (one wave: a CTA walks over further rows with the weights it has, the next row's loads in flight)
    const int sms = kSms;
    if (dim <= 1536 && rows >= 16 * sms) chained(norm_rows_warp_kernel<RMS>, (rows + 7) / 8, 256, 0, s)(x, ldx, w, b, y, ldy, rows, dim, eps);
    else if (dim <= 512) chained(norm_rows_kernel<RMS, 64, 1>, min(rows, 16 * sms), 64, 0, s)(x, ldx, w, b, y, ldy, rows, dim, eps);
    else if (dim <= 1536) chained(norm_rows_kernel<RMS, 192, 1>, min(rows, 5 * sms), 192, 0, s)(x, ldx, w, b, y, ldy, rows, dim, eps);
    else chained(norm_rows_kernel<RMS, 256, 2>, min(rows, 3 * sms), 256, 0, s)(x, ldx, w, b, y, ldy, rows, dim, eps);
    return 0;
}

int layernorm(const bf16* x, int ldx, const bf16* w, const bf16* b, bf16* y, int ldy, int rows, int dim,
              float eps, cudaStream_t s) {
    return norm_rows<false>(x, ldx, w, b, y, ldy, rows, dim, eps, s);
}

int rmsnorm(const bf16* x, int ldx, const bf16* w, bf16* y, int ldy, int rows, int dim, float eps,
            cudaStream_t s) {
    return norm_rows<true>(x, ldx, w, nullptr, y, ldy, rows, dim, eps, s);
}

// ------------------------------------------------------------------------------------------
// ViT 2-D rotary (mq2vl.py:725-752 table, :257-268 application).
// Table: cos/sin [N, head_dim/2] fp32 where column j < hd/4 uses the patch's h id and
// hd/4 <= j < hd/2 its w id, angle = id * inv_freq[j mod hd/4]; (h,w) ids follow the merge-window
// patch order of the processor. Built once per grid shape.
// ------------------------------------------------------------------------------------------
__global__ void vit_rope_table_kernel(float* __restrict__ cos_t, float* __restrict__ sin_t, int t, int h,
                                      int w, int merge, int half /* = head_dim/2 */,
                                      const float* __restrict__ inv_freq /* [half/2] */) {
    chain_begin();
    const int per_frame = h * w;
    const int n = t * per_frame;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n * half) return;
    const int p = idx / half, j = idx % half;
    int r = p % per_frame;
    // merge-window order: (h/m, w/m, m, m)
    const int wm = w / merge;
    const int win = r / (merge * merge), in = r % (merge * merge);
    const int hy = (win / wm) * merge + in / merge;
    const int wx = (win % wm) * merge + in % merge;
    const int q = half / 2;
    const float pos = (float)(j < q ? hy : wx);
    const float ang = __fmul_rn(pos, inv_freq[j % q]);
    cos_t[idx] = cosf(ang);
    sin_t[idx] = sinf(ang);
}

int vit_rope_table(float* cos_t, float* sin_t, int t, int h, int w, int merge, int head_dim,
                   const float* inv_freq, cudaStream_t s) {
    const int half = head_dim / 2;
    const int total = t * h * w * half;
    if (total <= 0) return 0;
    { lcc::count_launch(); chained(vit_rope_table_kernel, (total + 255) / 256, 256, 0, s)(cos_t, sin_t, t, h, w, merge, half, inv_freq); }
    return 0;
}

// In-place rotation of the q and k thirds of qkv [N, 3*heads*hd] (fp32 math, one rounding to bf16).
// out[i] = x[i]*cos[i] + rot(x)[i]*sin[i], rot(x) = cat(-x[hd/2:], x[:hd/2]); cos[i] = table[i mod hd/2].
__global__ void vit_rope_apply_kernel(bf16* __restrict__ qkv, int ld, const float* __restrict__ cos_t,
                                      const float* __restrict__ sin_t, int N, int heads, int hd) {
    chain_begin(qkv, cos_t, sin_t);
    // one thread = 8 consecutive rotation pairs (x[j..j+8), x[j+half..j+half+8)): two 16-byte loads/stores of
    // bf16 and four float4 loads of cos/sin; requires half % 8 == 0 (hd = 80 -> half = 40)
    const int half = hd / 2;
    const int chunks = half / 8;
    const int per_row = 2 * heads * chunks;  // q and k
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)N * per_row) return;
    const int row = (int)(idx / per_row);
    const int r = (int)(idx % per_row);
    const int which = r / (heads * chunks);  // 0 = q, 1 = k
    const int hh = (r / chunks) % heads;
    const int j0 = (r % chunks) * 8;
    bf16* base = qkv + (size_t)row * ld + (size_t)which * heads * hd + (size_t)hh * hd + j0;
    const uint4 u1 = *reinterpret_cast<const uint4*>(base);
    const uint4 u2 = *reinterpret_cast<const uint4*>(base + half);
    const float4* cp = reinterpret_cast<const float4*>(cos_t + (size_t)row * half + j0);
    const float4* sp = reinterpret_cast<const float4*>(sin_t + (size_t)row * half + j0);
    const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    const uint32_t w1[4] = {u1.x, u1.y, u1.z, u1.w}, w2[4] = {u2.x, u2.y, u2.z, u2.w};
    uint32_t o1[4], o2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 a = unpack_bf16x2(w1[k]), b = unpack_bf16x2(w2[k]);
        // (q * cos) + (rotate_half(q) * sin) with separately rounded products (no FMA contraction)
        const float p0 = __fadd_rn(__fmul_rn(a.x, c[2 * k]), __fmul_rn(-b.x, sn[2 * k]));
        const float p1 = __fadd_rn(__fmul_rn(a.y, c[2 * k + 1]), __fmul_rn(-b.y, sn[2 * k + 1]));
        const float q0 = __fadd_rn(__fmul_rn(b.x, c[2 * k]), __fmul_rn(a.x, sn[2 * k]));
        const float q1 = __fadd_rn(__fmul_rn(b.y, c[2 * k + 1]), __fmul_rn(a.y, sn[2 * k + 1]));
        o1[k] = pack_bf16x2(p0, p1);
        o2[k] = pack_bf16x2(q0, q1);
    }
    *reinterpret_cast<uint4*>(base) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
    *reinterpret_cast<uint4*>(base + half) = make_uint4(o2[0], o2[1], o2[2], o2[3]);
}

int vit_rope_apply(bf16* qkv, int ld, const float* cos_t, const float* sin_t, int N, int heads, int hd,
                   cudaStream_t s) {
    if ((hd / 2) % 8 || ld % 8) return -1;
    const int64_t total = (int64_t)N * 2 * heads * (hd / 16);
    if (total <= 0) return 0;
    { lcc::count_launch(); chained(vit_rope_apply_kernel, (int)((total + 255) / 256), 256, 0, s)(qkv, ld, cos_t, sin_t, N, heads, hd); }
    return 0;
}

// ------------------------------------------------------------------------------------------
// Embedding gather + scatter of video features (mq2vl.py:1255-1272).
// out[s] = is_video(ids[s]) ? video_embeds[rank of s among video tokens] : table[ids[s]].
// Kernel 1 (single CTA) computes the exclusive rank by a block scan; kernel 2 copies rows.
// ------------------------------------------------------------------------------------------
__global__ void video_rank_kernel(const __grid_constant__ PrefillStreams ps, int64_t video_id, int* __restrict__ rank) {
    chain_begin();
    const PrefillStream& st = ps.st[blockIdx.x];
    const int64_t* __restrict__ ids = st.ids;
    const int S = st.S;
    if (!st.video) video_id = -1;
    rank += st.row0;
    __shared__ int warp_tot[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < S; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int flag = (i < S && ids[i] == video_id) ? 1 : 0;
        int v = flag;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int n = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += n;
        }
        if (lane == 31) warp_tot[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int t = (lane < (int)(blockDim.x >> 5)) ? warp_tot[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int n = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += n;
            }
            warp_tot[lane] = t;  // inclusive scan of warp totals
        }
        __syncthreads();
        const int prefix = carry + (warp > 0 ? warp_tot[warp - 1] : 0) + v - flag;
        if (i < S) rank[i] = flag ? prefix : -1;
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_tot[(blockDim.x >> 5) - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0 && st.total_video) *st.total_video = carry;
}

__global__ void embed_gather_kernel(const __grid_constant__ PrefillStreams ps, const int* __restrict__ rank, const bf16* __restrict__ table,
                                    bf16* __restrict__ out, int H, int64_t vocab) {
    chain_begin(rank);
    const int row = blockIdx.x;
    const PrefillStream& st = ps.st[ps.of_row(row)];
    const bf16* __restrict__ video = st.video;
    const int n_video_rows = video ? st.n_video : 0;
    const int rk = rank[row];
    int64_t id = st.ids[row - st.row0];
    if (id < 0) id = 0;
    if (id >= vocab) id = vocab - 1;
    // A placeholder beyond the last feature row (more <|video_pad|> ids than ViT rows) keeps its text embedding:
    // nothing is read past the end of `video`; the host raises on the count mismatch (mq2vl.py:1169-1175).
    const bf16* src = (rk >= 0 && rk < n_video_rows) ? video + (size_t)rk * H : table + (size_t)id * H;
    bf16* dst = out + (size_t)row * H;
    for (int c = threadIdx.x * 8; c < H; c += blockDim.x * 8)
        *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(src + c);
}

int embed_gather(const int64_t* ids, const bf16* table, const bf16* video, int n_video_rows, int64_t video_id, bf16* out,
                 int* rank_ws, int* total_video, int S, int H, int64_t vocab, cudaStream_t s) {
    if (S <= 0) return 0;
    PrefillStreams ps{};
    ps.n = 1; ps.rows = S;
    ps.st[0].ids = ids; ps.st[0].video = video; ps.st[0].n_video = n_video_rows; ps.st[0].total_video = total_video; ps.st[0].S = S;
    return embed_gather_streams(ps, table, video_id, out, rank_ws, H, vocab, s);
}

int embed_gather_streams(const PrefillStreams& ps, const bf16* table, int64_t video_id, bf16* out, int* rank_ws, int H, int64_t vocab, cudaStream_t s) {
    if (H % 8) return -1;
    lcc::count_launch();
    chained(video_rank_kernel, ps.n, 1024, 0, s)(ps, video_id, rank_ws);
    lcc::count_launch();
    chained(embed_gather_kernel, ps.rows, 128, 0, s)(ps, rank_ws, table, out, H, vocab);
    return 0;
}

// ------------------------------------------------------------------------------------------
// M-RoPE on q,k of the fused qkv rows + append of (rotated k, v) to the paged KV cache
// (mq2vl.py:188-201 cos/sin in fp32 rounded to bf16, :244-254 section select + rotate-half,
// cache_utils.py:102-121 append). Prefill form: S rows.
//   qkv  [S, (Hq + 2*Hkv) * 128] : q is rotated in place, k/v are read.
//   pos3 [3, S] int32            : temporal / height / width position of every new token.
//   cache layer base: K at kc, V at vc, each [num_pages, Hkv, P, 128]; token (kv_start + s) lives in
//   page page_table[(kv_start+s)/P], slot (kv_start+s)%P.
// q*cos + rotate_half(q)*sin is evaluated the way torch does on bf16 tensors: each product and the
// sum are rounded to bf16.
// ------------------------------------------------------------------------------------------
struct MropeSections { int s0, s1; };  // boundaries in [0, 64): j < s0 -> T, j < s0+s1 -> H, else W

__device__ __forceinline__ void mrope_cos_sin(int j /*0..63*/, int pt, int ph, int pw, MropeSections sec,
                                              const float* inv_freq, float& c, float& s) {
    const int p = j < sec.s0 ? pt : (j < sec.s0 + sec.s1 ? ph : pw);
    const float ang = __fmul_rn((float)p, inv_freq[j]);
    c = rbf(cosf(ang));
    s = rbf(sinf(ang));
}

// One warp per (token, slice of kMropeHeads heads): the token's 64 angles are the same for every head, so a lane forms its two once and
// walks the slice with them. (A warp per head formed them 36 times per token: 4.5 us for 281 tokens and 23.4 for 2090, back to back; now 3.7 and 13.0.)
constexpr int kMropeHeads = 9;
__global__ void __launch_bounds__(256) mrope_kv_write_kernel(bf16* __restrict__ qkv, int ld, const __grid_constant__ PrefillStreams ps,
                                      const float* __restrict__ inv_freq, MropeSections sec, int Hq, int Hkv,
                                      bf16* __restrict__ kc, bf16* __restrict__ vc, int page_size) {
    chain_begin(qkv);
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int heads_total = Hq + 2 * Hkv, slices = (heads_total + kMropeHeads - 1) / kMropeHeads;
    if (gw >= ps.rows * slices) return;
    const int h0 = gw % slices * kMropeHeads, h1 = min(heads_total, h0 + kMropeHeads);
    bf16* row = qkv + (size_t)(gw / slices) * ld;
    const PrefillStream& st = ps.st[ps.of_row(gw / slices)];
    const int s_idx = gw / slices - st.row0, S = st.S;
    const int* __restrict__ pos3 = st.pos3;
    const int* __restrict__ page_table = st.page_table;
    const int tok = st.past + s_idx;
    const int page = page_table[tok / page_size], slot = tok % page_size;
    // lane owns rotation pairs j = 2*lane, 2*lane+1  (x[j], x[j+64])
    uint32_t lo[kMropeHeads], hi[kMropeHeads];
#pragma unroll
    for (int i = 0; i < kMropeHeads; ++i)
        if (h0 + i < h1) {
            lo[i] = *reinterpret_cast<const uint32_t*>(row + (h0 + i) * 128 + 2 * lane);
            hi[i] = *reinterpret_cast<const uint32_t*>(row + (h0 + i) * 128 + 64 + 2 * lane);
        }
    const int pt = pos3[s_idx], ph = pos3[S + s_idx], pw = pos3[2 * S + s_idx];
    float c0, s0, c1, s1;
    mrope_cos_sin(2 * lane, pt, ph, pw, sec, inv_freq, c0, s0);
    mrope_cos_sin(2 * lane + 1, pt, ph, pw, sec, inv_freq, c1, s1);
#pragma unroll
    for (int i = 0; i < kMropeHeads; ++i) {
        const int hh = h0 + i;
        if (hh >= h1) break;
        if (hh >= Hq + Hkv) {  // V: plain copy into the cache
            const int kvh = hh - Hq - Hkv;
            bf16* dst = vc + (((size_t)page * Hkv + kvh) * page_size + slot) * 128;
            *reinterpret_cast<uint32_t*>(dst + 2 * lane) = lo[i];
            *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = hi[i];
            // The V slots of the last page behind the newest token are zeroed: the tensor-core prefill kernel multiplies
            // them by P = 0 (masked keys), which must not meet NaN/Inf bit patterns of a recycled page.
            if (s_idx == S - 1)
                for (int k = lane; k < (page_size - 1 - slot) * 16; k += 32)
                    *reinterpret_cast<uint4*>(dst + 128 + k * 8) = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        const float2 x1 = unpack_bf16x2(lo[i]), x2 = unpack_bf16x2(hi[i]);
        const float o1a = rbf(rbf(x1.x * c0) + rbf(-x2.x * s0));
        const float o1b = rbf(rbf(x1.y * c1) + rbf(-x2.y * s1));
        const float o2a = rbf(rbf(x2.x * c0) + rbf(x1.x * s0));
        const float o2b = rbf(rbf(x2.y * c1) + rbf(x1.y * s1));
        bf16* dst = hh < Hq ? row + hh * 128 : kc + (((size_t)page * Hkv + (hh - Hq)) * page_size + slot) * 128;
        *reinterpret_cast<uint32_t*>(dst + 2 * lane) = pack_bf16x2(o1a, o1b);
        *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = pack_bf16x2(o2a, o2b);
    }
}

int mrope_kv_write(bf16* qkv, int ld, const int* pos3, int S, const float* inv_freq, int sec_t, int sec_h,
                   int Hq, int Hkv, bf16* kc, bf16* vc, const int* page_table, int page_size, int kv_start,
                   cudaStream_t s) {
    if (S <= 0) return 0;
    PrefillStreams ps{};
    ps.n = 1; ps.rows = S;
    ps.st[0].pos3 = pos3; ps.st[0].page_table = page_table; ps.st[0].S = S; ps.st[0].past = kv_start;
    return mrope_kv_write_streams(qkv, ld, ps, inv_freq, sec_t, sec_h, Hq, Hkv, kc, vc, page_size, s);
}

int mrope_kv_write_streams(bf16* qkv, int ld, const PrefillStreams& ps, const float* inv_freq, int sec_t, int sec_h, int Hq, int Hkv, bf16* kc,
                           bf16* vc, int page_size, cudaStream_t s) {
    const int64_t warps = (int64_t)ps.rows * ((Hq + 2 * Hkv + kMropeHeads - 1) / kMropeHeads);
    const int wpb = 8;
    MropeSections sec{sec_t, sec_h};
    lcc::count_launch();
    chained(mrope_kv_write_kernel, (int)((warps + wpb - 1) / wpb), wpb * 32, 0, s)(
        qkv, ld, ps, inv_freq, sec, Hq, Hkv, kc, vc, page_size);
    return 0;
}

}  // namespace lcc
