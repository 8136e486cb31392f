// GPU frame ingest: the antialiased bicubic resize of
//   REF/livecc-utils/src/livecc_utils/video_process_patch.py:101-106,150-155
//   transforms.functional.resize(clip_u8_TCHW, [H, W], BICUBIC, antialias=True)
// reproduced bit for bit: torchvision casts uint8 -> float32, ATen's CPU upsample_bicubic2d_aa runs a width pass then a
// height pass with a float32 intermediate, torchvision clamps to [0,255], rounds half to even and casts to uint8.
// The window/weight tables are built on the host with the same mixed float/double arithmetic as ATen
// (_compute_indices_min_size_weights_aa<float>, aa_filter with a = -0.5); the rounding order of the compiled wheel
// (FMA-contracted polynomial; tap sums with 4-wide unfused groups and a fused remainder) is stated in
// oracle/resize_aa.py and pinned by tests/test_resize_cpu.py / tests/golden/resize_aa_golden.json.
//
// One kernel, both passes. The bytes are decided by sums that are within a proven bound of the stated ones, and by the stated order where the bound does
// not settle the rounding (see "device" below): HBM traffic = source + output, the width pass on the tensor cores.
#include <cuda_fp16.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "launch.h"
#include "mma.cuh"
#include "resize.h"

namespace lcc {

// ---- host: ATen's window / weight table ----------------------------------------------------------------------------
// x86-64 baseline has no FMA instruction, so the compiler cannot contract the float expressions below; every fused
// operation is written as fmaf (correctly rounded in glibc with or without hardware FMA).
static inline float cubic_weight(float x) {
    x = fabsf(x);
    if (x < 1.0f) {
        const float t1 = fmaf(1.5f, x, -2.5f);  // (a + 2) x - (a + 3), a = -0.5
        return fmaf(t1 * x, x, 1.0f);
    }
    if (x < 2.0f) {
        const float u1 = fmaf(-0.5f, x, 2.5f);  // a x - 5 a
        const float u2 = fmaf(u1, x, -4.0f);    // (...) x + 8 a
        return fmaf(u2, x, 2.0f);               // (...) x - 4 a
    }
    return 0.0f;
}

static inline void aa_scale(int in_size, int out_size, float& scale, float& support, float& invscale) {
    scale = (float)in_size / (float)out_size;  // area_pixel_compute_scale<float>(align_corners=false, no scale factor)
    support = scale >= 1.0f ? (float)(2.0 * (double)scale) : 2.0f;
    invscale = scale >= 1.0f ? (float)(1.0 / (double)scale) : 1.0f;
}

int resize_aa_taps(int in_size, int out_size) {
    if (in_size <= 0 || out_size <= 0) return -1;
    float scale, support, invscale;
    aa_scale(in_size, out_size, scale, support, invscale);
    return (int)ceilf(support) * 2 + 1;
}

// Windows and weights, [out_size][taps].
static void aa_columns(int in_size, int out_size, int taps, int32_t* xmin_out, int32_t* xsize_out, float* weights) {
    float scale, support, invscale;
    aa_scale(in_size, out_size, scale, support, invscale);
    for (int i = 0; i < out_size; ++i) {
        const float center = (float)((double)scale * ((double)i + 0.5));
        const float lo = center - support, hi = center + support;
        int64_t xmin = (int64_t)((double)lo + 0.5);
        if (xmin < 0) xmin = 0;
        int64_t xmax = (int64_t)((double)hi + 0.5);
        if (xmax > in_size) xmax = in_size;
        int64_t xsize = xmax - xmin;
        if (xsize < 0) xsize = 0;
        if (xsize > taps) xsize = taps;
        float total = 0.0f;
        float* col = weights + (size_t)i * taps;
        for (int j = (int)xsize; j < taps; ++j) col[j] = 0.0f;
        for (int j = 0; j < (int)xsize; ++j) {
            const float d = (float)(j + xmin) - center;
            const float w = cubic_weight((float)(((double)d + 0.5) * (double)invscale));
            col[j] = w;
            total += w;
        }
        if (total != 0.0f)
            for (int j = 0; j < (int)xsize; ++j) col[j] /= total;
        xmin_out[i] = (int32_t)xmin;
        xsize_out[i] = (int32_t)xsize;
    }
}

int resize_aa_table(int in_size, int out_size, int32_t* xmin_out, int32_t* xsize_out, float* weights) {
    const int taps = resize_aa_taps(in_size, out_size);
    if (taps < 0) return -1;
    std::vector<float> cols((size_t)out_size * taps);
    aa_columns(in_size, out_size, taps, xmin_out, xsize_out, cols.data());
    for (int x0 = 0; x0 < out_size; x0 += 16)      // tap-major, in squares that stay in the cache
        for (int j = 0; j < taps; ++j)
            for (int x = x0; x < std::min(x0 + 16, out_size); ++x) weights[(size_t)j * out_size + x] = cols[(size_t)x * taps + j];
    return 0;
}

// ---- device ----------------------------------------------------------------------------------------------------------
// A CTA owns th output rows x tw output columns of one plane and stages the source window that its taps cover (nr rows). What the stated order of
// roundings costs is instructions: a byte is converted, multiplied and added, each rounded, for every tap that it enters, 22 times at 1080p -> 448x796
// (18 to 22 M warp instructions, 32.8 us for two frames). So the sums are formed in a cheaper way first:
//   width:  8 output columns are a [16 rows x 16 k] x [16 k x 8] product per 16 source columns of their common window (banded weights, zero outside a
//           column's taps). Bytes minus 128 are exact in fp16; a weight is the sum of two fp16 values, 22 bits (mma.sync: k is a few dozen, a tcgen05
//           tile would be mostly zeros). One LDS.32 holds four neighbouring bytes of a row: k is permuted so that they are one thread's operands.
//   height: fused multiply-adds down a column of the float tile, two columns per instruction.
// The result r differs from the stated one by at most `bound` (plan: rounding errors of both, from the very tables). Where r is further than that from
// every rounding boundary its byte is the stated one's. The other pixels (0.1 to 0.3 % of noise) are summed again in the stated order by the whole
// warp, a lane per source row; where they are many (pictures that sit on a boundary) the whole tile is.
// Two frames of 1080p -> 448x796 replayed from a graph: 17.7 us (20 as a call of its own; with the filter on the CUDA cores 31.4), one 10.7 (17.7), six 43 (86),
// 16 110 (222); two of 2160p 47 (139), of 1080p -> 140x140 24.5 (124), six of 360p -> 448x796 22.4 (30.5). A checkerboard of single pixels, where every
// byte is in doubt and every tile is summed twice, 50 (32), at half size 35 (24); edges of 12 x 20 pixels 20.6. What is left is latency (issue slots 55 % used): CTAs start (6 us), a lone
// warp's doubtful pixel holds its CTA (4 us). No gain: CTAs that go through planes with two row buffers (21 us, less of them fit), 128 threads (21), those pixels without
// loops (19: code that runs once is fetched).
struct ResizeParams {
    const uint8_t* src;
    uint8_t* dst;
    size_t src_bytes;
    int h, w, H, W;
    const int2* tap_w; const float* wt_w;     // [W] {first tap, taps}, [W][taps_w]
    const int2* tap_h; const float2* wt_h;    // [H], [H][taps_h], each weight twice
    const int32_t* col_c0; const int32_t* col_len;                 // per column tile: first staged source column (multiple of 4), columns staged
    const int32_t* row_r0; const int32_t* row_nr;                  // per row tile: first source row, window rows
    const int32_t* win;    // per 8 output columns: first source column of their window (multiple of 4)
    const uint4* frag;     // [8 columns][ks][lane]: weights as operand B, {high 0..1, high 2..3, low 0..1, low 2..3}
    float frag_scale;      // a power of two: what the sums are multiplied by
    float bound;
    int ks;                // k-steps of a window
    int taps_w, taps_h, th, tw_log2;    // output rows per CTA, log2 of its columns (8 to 128)
    int rows16;            // staged rows, multiple of 16
    int stride;            // bytes between staged rows (odd multiple of 16: eight rows' words fall into 32 banks)
    int dense;             // pixels of a warp's 256 up to which the warp sums them one by one (negative: the stated order throughout)
};

// float(u8) without the quarter-rate I2F: 0x4B000000 | u is the float 2^23 + u (exact), minus 2^23.
__device__ __forceinline__ float u8_to_float(uint32_t u) { return __fsub_rn(__uint_as_float(0x4B000000u | u), 8388608.0f); }

__device__ __forceinline__ uint32_t to_u8(float v) {  // clamp(0, 255), round half to even (torch.round), cast
    return (uint32_t)__float2int_rn(fminf(fmaxf(v, 0.f), 255.f));
}

// __byte_perm selector that puts the second word's byte 0 into byte c of the first
__device__ __forceinline__ uint32_t byte_into(int c) { return c & 2 ? (c & 1 ? 0x4210 : 0x3410) : (c & 1 ? 0x3240 : 0x3214); }

constexpr int RS_THREADS = 256, RS_WARPS = RS_THREADS / 32;

// Staged rows keep the 16-byte phase that they have in memory: column c of a tile's row r is byte (phase0 + r * w) % 16 + c - c0.
__device__ __forceinline__ int row_phase(const ResizeParams& p, int phase0, int r) { return (phase0 + r * p.w) & 15; }

// bytes 0,1 (or 2,3) of w minus 128 as two fp16: 0x6400 | u is the fp16 1024 + u
template <int SEL>
__device__ __forceinline__ uint32_t bytes_to_half2(uint32_t w) {
    const uint32_t x = __byte_perm(w, 0x64646464u, SEL);
    const __half2 y = __hsub2(*reinterpret_cast<const __half2*>(&x), __floats2half2_rn(1152.f, 1152.f));
    return *reinterpret_cast<const uint32_t*>(&y);
}
__device__ __forceinline__ void mma_f16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c0, float c1, float c2, float c3) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
// Steps j0 .. j1 - 1 of a stated sum of n terms; value(j) and weight(j) are asked for in that order (j0 is a multiple of 32).
template <typename V, typename Wt>
__device__ __forceinline__ float stated_steps(float acc, int j0, int j1, int n, V value, Wt weight) {
    const int unfused = (((n - 1) >> 2) << 2) + 1;   // the first term, whole groups of 4 with a rounding each for product and sum; then up to 3 fused steps
    int j = j0;
    if (j == 0 && j1 > 0) { acc = __fmul_rn(value(0), weight(0)); j = 1; }
#pragma unroll 4
    for (; j < min(j1, unfused); ++j) acc = __fadd_rn(acc, __fmul_rn(value(j), weight(j)));
    for (; j < j1; ++j) acc = __fmaf_rn(value(j), weight(j), acc);
    return acc;
}

// What a CTA keeps in shared memory.
struct Staged {
    const uint8_t* rows;    // [rows16][stride] source bytes
    const float2* wt_h;     // [th][taps_h]
    const float* wt_w;      // [tw][taps_w]
    const int2* tap_h;      // [th] {first row of the window, rows}
    const int2* tap_w;      // [tw] {first column of the window, columns}
    int phase0;
};

// One pixel in the stated order, by a warp: lane = source row, then down the rows.
__device__ __forceinline__ float stated_pixel(const ResizeParams& p, const Staged& s, int xl, int yl) {
    const int lane = threadIdx.x & 31;
    const int2 tw = s.tap_w[xl], th = s.tap_h[yl];
    const float* ww = s.wt_w + xl * p.taps_w;
    const float2* wh = s.wt_h + yl * p.taps_h;
    float acc = 0.f;
    for (int rb = 0; rb < th.y; rb += 32) {
        const int r = th.x + min(rb + lane, th.y - 1);
        const uint8_t* row = s.rows + r * p.stride + row_phase(p, s.phase0, r) + tw.x;
        const float v = stated_steps(0.f, 0, tw.y, tw.y, [&](int j) { return u8_to_float(row[j]); }, [&](int j) { return ww[j]; });
        acc = stated_steps(acc, rb, min(rb + 32, th.y), th.y, [&](int j) { return __shfl_sync(0xffffffffu, v, j - rb); }, [&](int j) { return wh[j].x; });
    }
    return acc;
}

// A whole tile in the stated order: thread = one column, four rows side by side, then four columns of an output row.
__device__ __noinline__ void stated_tile(const ResizeParams& p, const Staged& s, float* tile, uint8_t* out, int X0, int X1, int y0, int y1, int nr) {
    const int TW = 1 << p.tw_log2, TWP = TW + 8;
    {
        const int xl = threadIdx.x & (TW - 1), step = (RS_THREADS >> p.tw_log2) * 4;
        const int2 tw = s.tap_w[xl];
        const float* ww = s.wt_w + xl * p.taps_w;
        const int unfused = ((tw.y - 1) >> 2) << 2;
        for (int rb = (threadIdx.x >> p.tw_log2) * 4; rb < nr; rb += step) {
            const uint8_t* row[4];
            float acc[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = min(rb + q, nr - 1);
                row[q] = s.rows + r * p.stride + row_phase(p, s.phase0, r) + tw.x;
                acc[q] = tw.y > 0 ? __fmul_rn(u8_to_float(row[q][0]), ww[0]) : 0.f;
            }
            int j = 1;
#pragma unroll 4
            for (; j <= unfused; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[q] = __fadd_rn(acc[q], __fmul_rn(u8_to_float(row[q][j]), ww[j]));
            for (; j < tw.y; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[q] = __fmaf_rn(u8_to_float(row[q][j]), ww[j], acc[q]);
#pragma unroll
            for (int q = 0; q < 4; ++q) tile[min(rb + q, nr - 1) * TWP + xl] = acc[q];
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < (y1 - y0) << (p.tw_log2 - 2); idx += RS_THREADS) {
        const int yl = idx >> (p.tw_log2 - 2), xl = (idx & ((TW >> 2) - 1)) << 2;
        const int2 th = s.tap_h[yl];
        const float* t = tile + th.x * TWP + xl;
        const float2* wh = s.wt_h + yl * p.taps_h;
        const int unfused = ((th.y - 1) >> 2) << 2;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < th.y; ++j, t += TWP) {
            const float4 v = *reinterpret_cast<const float4*>(t);
            const float w = wh[j].x;
            if (j == 0) a = make_float4(__fmul_rn(v.x, w), __fmul_rn(v.y, w), __fmul_rn(v.z, w), __fmul_rn(v.w, w));
            else if (j <= unfused)
                a = make_float4(__fadd_rn(a.x, __fmul_rn(v.x, w)), __fadd_rn(a.y, __fmul_rn(v.y, w)), __fadd_rn(a.z, __fmul_rn(v.z, w)), __fadd_rn(a.w, __fmul_rn(v.w, w)));
            else a = make_float4(__fmaf_rn(v.x, w, a.x), __fmaf_rn(v.y, w, a.y), __fmaf_rn(v.z, w, a.z), __fmaf_rn(v.w, w, a.w));
        }
        uint8_t* o = out + (size_t)(y0 + yl) * p.W + X0 + xl;
        if (X0 + xl < X1) o[0] = (uint8_t)to_u8(a.x);
        if (X0 + xl + 1 < X1) o[1] = (uint8_t)to_u8(a.y);
        if (X0 + xl + 2 < X1) o[2] = (uint8_t)to_u8(a.z);
        if (X0 + xl + 3 < X1) o[3] = (uint8_t)to_u8(a.w);
    }
}

// Width pass of 8 output columns over 16-row tiles m = m0, m0 + step, ..: KS k-steps with the weights in registers, or (KS = 0) p.ks of them from L1.
// Each k-step starts from its products with the low parts and is added in fp32: an accumulator as large as a pixel would cost the products their last
// bits. The sums keep the weights' power of two.
template <int KS, bool W4>
__device__ __forceinline__ void width_products(const ResizeParams& p, const uint8_t* rows, float* tile, int nt, int xl, int c0, int phase0, int m0, int step) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int ks_n = KS ? KS : p.ks, TWP = (1 << p.tw_log2) + 8, mts = p.rows16 >> 4;
    const uint4* fr = p.frag + (size_t)nt * ks_n * 32 + lane;
    uint4 b[KS ? KS : 1];
    if (KS) {
#pragma unroll
        for (int k = 0; k < KS; ++k) b[k] = __ldg(fr + k * 32);
    }
    const int mrow = step * 16 * p.stride, mtile = step * 16 * TWP;
    // 16 rows further on a row has the same phase. W4: words lie on word boundaries; otherwise one is cut from two.
    const int at = (__ldg(p.win + nt) - c0) + 4 * tig, at0 = at + row_phase(p, phase0, g), at1 = at + row_phase(p, phase0, g + 8);
    const int sh0 = (at0 & 3) * 8, sh1 = (at1 & 3) * 8;
    const uint32_t* ar = reinterpret_cast<const uint32_t*>(rows + (m0 * 16 + g) * p.stride + (at0 & ~3));
    const int half = (8 * p.stride + (at1 & ~3) - (at0 & ~3)) >> 2;
    float* t = tile + (m0 * 16 + g) * TWP + xl + 2 * tig;
#pragma unroll 2
    for (int m = m0; m < mts; m += step, ar += mrow >> 2, t += mtile) {
        float v[4], lo[4];
        auto kstep = [&](int k, const uint4& w) {
            const uint32_t u0 = W4 ? ar[4 * k] : __funnelshift_r(ar[4 * k], ar[4 * k + 1], sh0);
            const uint32_t u1 = W4 ? ar[half + 4 * k] : __funnelshift_r(ar[half + 4 * k], ar[half + 4 * k + 1], sh1);
            const uint32_t a[4] = {bytes_to_half2<0x4140>(u0), bytes_to_half2<0x4140>(u1), bytes_to_half2<0x4342>(u0), bytes_to_half2<0x4342>(u1)};
            float d[4];
            mma_f16_16816(lo, a, w.z, w.w, 0.f, 0.f, 0.f, 0.f);
            mma_f16_16816(d, a, w.x, w.y, lo[0], lo[1], lo[2], lo[3]);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = k == 0 ? d[i] : v[i] + d[i];
        };
        if (KS) {
#pragma unroll
            for (int k = 0; k < KS; ++k) kstep(k, b[KS ? k : 0]);
        } else {
            kstep(0, __ldg(fr));
#pragma unroll 2
            for (int k = 1; k < ks_n; ++k) kstep(k, __ldg(fr + (size_t)k * 32));
        }
        *reinterpret_cast<float2*>(t) = make_float2(v[0], v[1]);
        *reinterpret_cast<float2*>(t + 8 * TWP) = make_float2(v[2], v[3]);
    }
}

__device__ __forceinline__ void rs_fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// Source window of a plane to shared memory in chunks of 16 bytes; rows keep their phase. win: its first byte.
__device__ __forceinline__ void stage_rows(const ResizeParams& p, uint8_t* rows, const uint8_t* win, int nr, int cols) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(p.src), hi = lo + p.src_bytes, at = reinterpret_cast<uintptr_t>(win);
    const int phase0 = (int)(at & 15), r = warp * 2 + (lane >> 4);
    const uint8_t* chunk0 = win - phase0;
    const bool inside = at - phase0 >= lo && at + (size_t)(nr - 1) * p.w + cols + 15 <= hi;   // every chunk lies in the clip
    for (int b = (lane & 15) * 16; b < cols + 15; b += 256) {
        if (inside) {
            uint32_t d = smem_u32(rows) + r * p.stride + b;
            int o = phase0 + r * p.w;      // (a window that fits in shared memory spans less than 2^31 bytes of a plane)
#pragma unroll 1
            for (int k = r; k < nr; k += RS_WARPS * 2, o += RS_WARPS * 2 * p.w, d += RS_WARPS * 2 * p.stride)
                if (b < (o & 15) + cols) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(chunk0 + b + (o & ~15)) : "memory");
        } else {
            for (int k = r; k < nr; k += RS_WARPS * 2) {
                const uintptr_t g = at + (size_t)k * p.w, a = (g & ~uintptr_t(15)) + b;
                uint8_t* d = rows + k * p.stride + b;
                if (b >= (int)(g & 15) + cols) continue;
                if (a >= lo && a + 16 <= hi) {
                    cp_async16(d, reinterpret_cast<const void*>(a), true);
                } else {  // the ends of a clip that lies at an odd address
                    for (int i = 0; i < 16; ++i)
                        if (a + i >= lo && a + i < hi) d[i] = *reinterpret_cast<const uint8_t*>(a + i);
                }
            }
        }
    }
    cp_async_commit();
}

template <int KS, bool W4>
__global__ void __launch_bounds__(RS_THREADS, 4) resize_bicubic_aa_u8_kernel(const __grid_constant__ ResizeParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int plane = blockIdx.z, rt = blockIdx.y, ct = blockIdx.x;
    const int TW = 1 << p.tw_log2, TWP = TW + 8;
    const int y0 = rt * p.th, y1 = min(y0 + p.th, p.H);
    const int X0 = ct * TW, X1 = min(X0 + TW, p.W);
    const int r0 = p.row_r0[rt], nr = p.row_nr[rt];
    const int c0 = p.col_c0[ct], seg = p.col_len[ct];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // shared memory carve-up (no integer round trips on the pointers: the compiler must keep them in the shared window)
    uint8_t* rows = smem;
    float* tile = reinterpret_cast<float*>(smem + p.rows16 * p.stride);
    float* wt_w = tile + p.rows16 * TWP;
    float2* wt_h = reinterpret_cast<float2*>(wt_w + p.taps_w * TW);
    int2* tap_w = reinterpret_cast<int2*>(wt_h + p.taps_h * p.th);
    int2* tap_h = tap_w + TW;
    int* dense = reinterpret_cast<int*>(tap_h + p.th);

    const uint8_t* win = p.src + ((size_t)plane * p.h + r0) * p.w + c0;
    const int phase0 = (int)(reinterpret_cast<uintptr_t>(win) & 15);
    stage_rows(p, rows, win, nr, min(seg, p.w - c0));
#pragma unroll 1
    for (int i = threadIdx.x; i < p.taps_h * (y1 - y0); i += RS_THREADS) wt_h[i] = __ldg(p.wt_h + (size_t)y0 * p.taps_h + i);
#pragma unroll 1
    for (int i = threadIdx.x; i * 4 < p.taps_w * TW; i += RS_THREADS)   // (the table is padded to whole tiles)
        reinterpret_cast<float4*>(wt_w)[i] = __ldg(reinterpret_cast<const float4*>(p.wt_w + (size_t)X0 * p.taps_w) + i);
#pragma unroll 1
    for (int i = threadIdx.x; i < TW + p.th; i += RS_THREADS) {
        if (i < TW) { const int2 v = __ldg(p.tap_w + min(X0 + i, p.W - 1)); tap_w[i] = make_int2(v.x - c0, v.y); }
        else { const int2 v = __ldg(p.tap_h + min(y0 + i - TW, p.H - 1)); tap_h[i - TW] = make_int2(v.x - r0, v.y); }
    }
    if (threadIdx.x == 0) *dense = 0;
    cp_async_wait<0>();
    __syncthreads();

    uint8_t* out = p.dst + (size_t)plane * p.H * p.W;
    const Staged st{rows, wt_h, wt_w, tap_h, tap_w, phase0};
    if (p.dense < 0) {
        stated_tile(p, st, tile, out, X0, X1, y0, y1, nr);
        return;
    }
    // ---- width pass: a warp takes 8 output columns and 16-row tiles
    {
        const int nts = 1 << (p.tw_log2 - 3), have = (X1 - X0 + 7) >> 3;
        if (nts >= RS_WARPS) {
            for (int nt = warp; nt < have; nt += RS_WARPS) width_products<KS, W4>(p, rows, tile, (X0 >> 3) + nt, nt * 8, c0, phase0, 0, 1);
        } else if ((warp & (nts - 1)) < have) {
            const int nt = warp & (nts - 1);
            width_products<KS, W4>(p, rows, tile, (X0 >> 3) + nt, nt * 8, c0, phase0, warp >> (p.tw_log2 - 3), RS_WARPS >> (p.tw_log2 - 3));
        }
    }
    __syncthreads();

    // ---- height pass + round/clamp/cast: thread = 4 adjacent columns in either half of the tile, one output row
    const bool vec = (p.W & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 3) == 0;
    const int t8 = p.tw_log2 - 3;
    const float sure = 0.5f - p.bound;
#pragma unroll 1
    for (int i0 = warp * 32; i0 < (y1 - y0) << t8; i0 += RS_THREADS) {
        const int idx = min(i0 + lane, ((y1 - y0) << t8) - 1);
        const int yl = idx >> t8, xl = (idx & ((1 << t8) - 1)) << 2, y = y0 + yl;
        const int2 tap = tap_h[yl];
        const float* t = tile + tap.x * TWP + xl;
        const unsigned long long* wc = reinterpret_cast<const unsigned long long*>(wt_h + yl * p.taps_h);
        unsigned long long s[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 4
        for (int j = 0; j < tap.y; ++j, t += TWP) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(t), v = *reinterpret_cast<const ulonglong2*>(t + (TW >> 1));
            const unsigned long long w = wc[j];
            rs_fma2(s[0], u.x, w); rs_fma2(s[1], u.y, w);
            rs_fma2(s[2], v.x, w); rs_fma2(s[3], v.y, w);
        }
        uint32_t o4[2], doubt = 0;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            float a[4], d[4];
            int q[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a[0]), "=f"(a[1]) : "l"(s[2 * hf]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a[2]), "=f"(a[3]) : "l"(s[2 * hf + 1]));
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float k = __fmaf_rn(a[c], p.frag_scale, 12582912.f);      // 1.5 * 2^23: round half to even, the integer in the low bits
                q[c] = __float_as_int(k) - 0x4B400000 + 128;
                d[c] = fabsf(__fmaf_rn(a[c], p.frag_scale, -__fsub_rn(k, 12582912.f)));
            }
            // four integers, each clamped to 0 .. 255
            asm("{\n.reg .b32 h;\ncvt.pack.sat.u8.s32.b32 h, %4, %3, 0;\ncvt.pack.sat.u8.s32.b32 %0, %2, %1, h;\n}" : "=r"(o4[hf]) : "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]));
            if (fmaxf(fmaxf(d[0], d[1]), fmaxf(d[2], d[3])) > sure)
                for (int c = 0; c < 4; ++c) doubt |= (d[c] > sure && X0 + xl + hf * (TW >> 1) + c < X1 ? 1u : 0u) << (4 * hf + c);
        }
        if (i0 + lane >= (y1 - y0) << t8) doubt = 0;
        unsigned who = __ballot_sync(0xffffffffu, doubt != 0);
        if (who && (int)__reduce_add_sync(0xffffffffu, __popc(doubt)) > p.dense) {
            if (lane == 0) *dense = 1;
            who = 0;
        }
        for (; who; who &= who - 1) {
            const int src = __ffs(who) - 1, yy = __shfl_sync(0xffffffffu, yl, src), xx = __shfl_sync(0xffffffffu, xl, src);
            for (uint32_t bits = __shfl_sync(0xffffffffu, doubt, src); bits; bits &= bits - 1) {
                const int c = __ffs(bits) - 1;
                const uint32_t v = to_u8(stated_pixel(p, st, xx + (c >> 2) * (TW >> 1) + (c & 3), yy));
                const uint32_t sel = byte_into(c & 3);
                if (lane == src && c < 4) o4[0] = __byte_perm(o4[0], v, sel);
                if (lane == src && c >= 4) o4[1] = __byte_perm(o4[1], v, sel);
            }
        }
        if (i0 + lane >= (y1 - y0) << t8) continue;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int X = X0 + xl + hf * (TW >> 1);
            uint8_t* o = out + (size_t)y * p.W + X;
            if (vec && X + 4 <= X1) {
                *reinterpret_cast<uint32_t*>(o) = o4[hf];
            } else {
                for (int c = 0; c < 4 && X + c < X1; ++c) o[c] = (uint8_t)(o4[hf] >> (8 * c));
            }
        }
    }
    __syncthreads();
    if (*dense) stated_tile(p, st, tile, out, X0, X1, y0, y1, nr);
}

// ---- plan ------------------------------------------------------------------------------------------------------------
struct ResizePlan {
    int h, w, H, W;
    int taps_w, taps_h, ks;
    int th, tw_log2, max_rows, rows16, stride, row_tiles, col_tiles, dense;
    float frag_scale, bound;
    size_t smem;
    void* dev = nullptr;  // one allocation: operands, all int tables, both weight tables
    const uint4* frag;
    const float *wt_w, *wt_h;
    const int32_t *tap_w, *tap_h, *col_c0, *col_len, *row_r0, *row_nr, *win;
};

static SmemAttrOnce g_resize_smem[5][2];

// Largest error of rounding (2: of cutting) a number of magnitude up to m to 24 bits: half (one) unit in the last place of m.
// (By the exponent's bits: a plan asks some 100,000 times. m is 0 or far from double's limits.)
static double half_ulp(double m) {
    uint64_t u;
    memcpy(&u, &m, 8);
    u &= 0x7ff0000000000000ull;
    memcpy(&m, &u, 8);
    return m * 0x1p-24;
}

// A float as fp16, rounded to nearest even, by its bits; `back` is its value. 0 stands for what would be subnormal; magnitudes are below 2^15.
static uint16_t to_half(float v, float* back) {
    uint32_t u;
    if (fabsf(v) < 0x1p-14f) v = 0.f;
    memcpy(&u, &v, 4);
    const uint32_t r = (u & 0x7fffffffu) + 0xfffu + (u >> 13 & 1), kept = r & ~0x1fffu;
    const uint32_t whole = v == 0.f ? 0u : kept | (u & 0x80000000u);
    memcpy(back, &whole, 4);
    return v == 0.f ? 0 : (uint16_t)((kept >> 13) - (112 << 10) | (u >> 16 & 0x8000u));
}

// |stated sum - sum without rounding| of an axis, over values in lo .. hi: every product and every sum rounds (the fused steps round once for both).
static double order_error(const float* wt, int n, double lo, double hi) {
    double e = 0, top = 0, low = 0;      // range of the partial sum
    for (int j = 0; j < n; ++j) {
        const double w = wt[j], a = w * lo, b = w * hi;
        top += std::max(a, b); low += std::min(a, b);
        if (j < ((n - 1) >> 2 << 2) + 1) e += half_ulp(std::max(fabs(a), fabs(b)));
        if (j > 0) e += half_ulp(1.001 * std::max(top, -low));      // (with the errors up to here: fewer than 1000 terms)
    }
    return e;
}


ResizePlan* resize_plan_create(int h, int w, int H, int W, int th_override) {
    if (h <= 0 || w <= 0 || H <= 0 || W <= 0 || w > (1 << 15) || h > (1 << 15) || W > (1 << 14) || H > (1 << 14)) return nullptr;
    // Output width 1 together with a height change: the reference's dependency (ATen) gives a result that is NOT the separable
    // filter (its [h, 1] intermediate is stride-ambiguous; found by the randomized oracle check). Unreachable from the path
    // (sizes are multiples of 28): refuse rather than differ silently.
    if (W == 1 && h != H) return nullptr;
    const int tw_taps = resize_aa_taps(w, W), th_taps = resize_aa_taps(h, H);
    std::vector<int32_t> xw(W), nw(W), xh(H), nh(H);
    std::vector<float> cw((size_t)((W + 127) & ~127) * tw_taps, 0.f), rw((size_t)H * th_taps);    // weights column by column (padded to whole tiles) and row by row
    aa_columns(w, W, tw_taps, xw.data(), nw.data(), cw.data());
    aa_columns(h, H, th_taps, xh.data(), nh.data(), rw.data());
    auto row_windows = [&](int th, std::vector<int32_t>& r0s, std::vector<int32_t>& nrs) {
        int m = 1;
        r0s.clear(); nrs.clear();
        for (int y0 = 0; y0 < H; y0 += th) {
            int lo = xh[y0], hi = lo;
            for (int y = y0; y < std::min(y0 + th, H); ++y) { lo = std::min(lo, xh[y]); hi = std::max(hi, xh[y] + nh[y]); }
            r0s.push_back(lo); nrs.push_back(std::max(hi - lo, 1));
            m = std::max(m, hi - lo);
        }
        return m;
    };
    const size_t kSmem = 227 * 1024;
    std::vector<int32_t> rr0, rnr;
    {   // Sizes that are refused: one output row's window (or th_override rows') of 64 or 128 columns with its weights does not fit in shared memory.
        const int TW = W <= 64 ? 64 : 128;
        int seg = 1;
        for (int X0 = 0; X0 < W; X0 += TW) {
            int lo = xw[X0], hi = lo;
            for (int X = X0; X < std::min(X0 + TW, W); ++X) { lo = std::min(lo, xw[X]); hi = std::max(hi, xw[X] + nw[X]); }
            seg = std::max(seg, hi - lo);
        }
        const int th = th_override > 0 ? th_override : 1;
        const size_t rows = row_windows(th, rr0, rnr);
        if ((rows * TW + (size_t)tw_taps * TW + (size_t)th_taps * th + rows) * 4 + 16 + rows * (((seg + 30) >> 4) << 4) > kSmem) return nullptr;
    }
    // ---- operands of the width pass: windows of 8 output columns
    const int nts = (W + 7) / 8;
    std::vector<int32_t> win(nts), wend(nts);
    int ks = 1;
    for (int nt = 0; nt < nts; ++nt) {
        int lo = xw[nt * 8], hi = lo + 1;
        for (int X = nt * 8; X < std::min(nt * 8 + 8, W); ++X) { lo = std::min(lo, xw[X]); hi = std::max(hi, xw[X] + nw[X]); }
        win[nt] = lo & ~3;
        ks = std::max(ks, (hi - win[nt] + 15) / 16);
    }
    float wmax = 0.f;
    for (float v : cw) wmax = std::max(wmax, fabsf(v));
    int up = 14;                                             // weights times 2^up stay below half of fp16's range
    while (up > -14 && ldexpf(wmax, up) > 32768.f) --up;
    std::vector<uint16_t> frag((size_t)nts * ks * 32 * 8, 0);
    // The width pass off its true sums. PTX promises of an mma step products and sums of at least single precision, in an order and with a rounding of the
    // hardware's choice, so no one form is taken for granted: a step of n products that are not zero, whose magnitudes add up to S with the addend's, is at most
    // (n + 4) units in the last of S's 24 bits off. That covers fp32 adds one by one in any order (n), however they round or cut, addends aligned to the
    // largest and cut behind 24 bits, all at once (n + 1, and 1 for the sum) or half by half (n + 2, and 2). The products are exact (11 x 8 bits). What the
    // hardware does with subnormal operands is left open too: there are none.
    const double scale = ldexp(1.0, -up);
    const float raise = ldexpf(1.f, up);
    double f_w = 0, sum_lo = 1e9, sum_hi = -1e9;
    for (int X = 0; X < W; ++X) {
        const int nt = X >> 3, g = X & 7;
        double off = 0, so_far = 0, sum = 0, hs = 0, ls = 0;    // of this k-step: magnitudes of the high and of the low parts
        int n = 0;
        for (int j = 0; j < nw[X]; ++j) {
            const float v = cw[(size_t)X * tw_taps + j], sv = v * raise;
            const int col = xw[X] + j - win[nt], k = col >> 4, tig = (col & 15) >> 2, b = col & 3;
            uint16_t* f = &frag[(((size_t)nt * ks + k) * 32 + g * 4 + tig) * 8];
            float hi, lo;
            f[b] = to_half(sv, &hi);
            f[4 + b] = to_half(sv - hi, &lo);
            const double h = hi, l = lo;
            off += 128 * scale * fabs((double)sv - h - l);      // bytes minus 128 are -128 .. 127
            hs += scale * fabs(h); ls += scale * fabs(l); sum += v;
            ++n;
            if (j + 1 == nw[X] || ((col + 1) & 15) == 0) {      // (128.1: with the errors up to here)
                off += (n + 4) * 2 * (half_ulp(128.1 * (hs + ls)) + half_ulp(128.1 * ls));
                so_far += hs + ls;
                if (so_far > hs + ls) off += half_ulp(128.1 * so_far);      // the fp32 add of the steps before
                hs = ls = 0; n = 0;
            }
        }
        f_w = std::max(f_w, off);
        sum_lo = std::min(sum_lo, sum); sum_hi = std::max(sum_hi, sum);
    }
    // ---- bound: stated sums off the true ones, the kernel's sums off the true ones, and 128 standing for 128 times the sums of the weights
    double e_w = 0, ah = 0, hs_lo = 1e9, hs_hi = -1e9, e_h = 0, f_h = 0;
    double v_lo = 1e9, v_hi = -1e9;      // range of the width pass over bytes
    for (int X = 0; X < W; ++X) {
        double lo = 0, hi = 0;
        const float* c = &cw[(size_t)X * tw_taps];
        for (int j = 0; j < nw[X]; ++j) { const double v = 255.0 * c[j]; (v < 0 ? lo : hi) += v; }
        v_lo = std::min(v_lo, lo); v_hi = std::max(v_hi, hi);
        e_w = std::max(e_w, order_error(c, nw[X], 0.0, 255.0));
    }
    for (int y = 0; y < H; ++y) {
        double a = 0, s = 0;
        const float* r = &rw[(size_t)y * th_taps];
        for (int j = 0; j < nh[y]; ++j) { a += fabs((double)r[j]); s += r[j]; }
        ah = std::max(ah, a); hs_lo = std::min(hs_lo, s); hs_hi = std::max(hs_hi, s);
        e_h = std::max(e_h, order_error(r, nh[y], v_lo - e_w, v_hi + e_w));
        f_h = std::max(f_h, order_error(r, nh[y], v_lo - 128.01, v_hi - 127.99));
    }
    const double off = 128.0 * std::max(std::max(fabs(sum_lo * hs_lo - 1), fabs(sum_hi * hs_hi - 1)), std::max(fabs(sum_lo * hs_hi - 1), fabs(sum_hi * hs_lo - 1)));
    const double bound = 1.02 * (e_w * ah + e_h + f_w * ah + f_h + off) + 1e-6;

    // ---- tile: of those that fit, the one with the least estimated time for two frames (of 20 tiles timed at eight sizes it is within 5 % of the best for two frames but
    // for 1080p -> 140x140, 24.4 us for 22.1; one frame up to 1.2 times the best, 1.5 at 140x140; 16 frames up to 1.27 and 1.36). A CTA's instructions are counted, and some 2500 cycles of its
    // life (loads, two barriers) are no issue slots; at most 8 CTAs of an SM share its four schedulers.
    struct Tile { int tw, th, rows, rows16, stride; size_t smem; } best{};
    double best_t = 1e30;
    std::vector<int32_t> cc0, clen;
    auto columns = [&](int TW) {
        cc0.clear(); clen.clear();
        int m = 16;
        for (int n0 = 0; n0 < nts; n0 += TW / 8) {
            int lo = win[n0], hi = lo;
            for (int nt = n0; nt < std::min(n0 + TW / 8, nts); ++nt) { lo = std::min(lo, win[nt]); hi = std::max(hi, win[nt] + 16 * ks); }
            cc0.push_back(lo); clen.push_back(hi - lo);
            m = std::max(m, clen.back());
        }
        m = (m + 15 + 3 + 15) >> 4;    // behind a phase of up to 15, and the word that a last word may be cut from
        return (m | 1) << 4;
    };
    std::vector<std::pair<int, int>> heights;      // rows per CTA, the source rows they cover
    for (int th : {32, 16, 8, 4, 2, 1}) {
        const int t = th_override > 0 ? th_override : th;
        heights.push_back({t, row_windows(t, rr0, rnr)});
        if (th_override > 0) break;
    }
    for (int TW : {128, 64, 32, 16, 8}) {
        const int stride = columns(TW);
        for (auto [t, rows] : heights) {
            const int rows16 = (rows + 15) & ~15;
            const size_t sm = (size_t)rows16 * (stride + (TW + 8) * 4) + ((size_t)tw_taps * TW + ((size_t)th_taps + 1) * t * 2 + 2 * TW + 1) * 4;
            if (sm > kSmem) continue;
            const double ctas = 6.0 * ((W + TW - 1) / TW) * ((H + t - 1) / t), occ = std::min<double>(4, floor(228.0 * 1024 / (sm + 1024)));
            const double instr = 700 + 5.0 * rows * ((stride + 255) / 256) + (rows16 / 16) * (TW / 8) * (17.0 * ks + 14) + t * TW / 256.0 * (8.0 * th_taps + 90) + 0.3 * t * TW;
            const double est = std::max(1.0, ctas / (148 * occ)) * (2500 + occ * instr / 4);
            if (est < best_t) { best_t = est; best = {TW, t, rows, rows16, stride, sm}; }
        }
    }
    if (!best.tw) return nullptr;
    columns(best.tw);
    row_windows(best.th, rr0, rnr);
    ResizePlan* pl = new ResizePlan();
    pl->h = h; pl->w = w; pl->H = H; pl->W = W;
    pl->taps_w = tw_taps; pl->taps_h = th_taps; pl->ks = ks;
    pl->frag_scale = ldexpf(1.f, -up); pl->bound = (float)bound;
    // warp instructions: a pixel one by one against a warp's share of the tile
    pl->dense = bound < 0.125 ? (int)((best.rows16 * best.tw * tw_taps * 5.5 + best.th * best.tw * th_taps * 4.0) / (RS_THREADS * (6.0 * tw_taps * ((th_taps + 31) / 32) + 5.0 * th_taps + 80))) : -1;
    pl->th = best.th; pl->tw_log2 = best.tw == 8 ? 3 : best.tw == 16 ? 4 : best.tw == 32 ? 5 : best.tw == 64 ? 6 : 7; pl->stride = best.stride;
    pl->max_rows = best.rows; pl->rows16 = best.rows16;
    pl->row_tiles = (int)rr0.size(); pl->col_tiles = (int)cc0.size();
    pl->smem = best.smem;
    // tables: weights column by column (padded to whole tiles) and row by row (each twice), {first tap, taps} pairs
    const size_t o_wh = (size_t)pl->col_tiles * best.tw * tw_taps;
    std::vector<float> flt(o_wh + (size_t)H * th_taps * 2);
    memcpy(flt.data(), cw.data(), o_wh * 4);
    for (size_t i = 0; i < rw.size(); ++i) flt[o_wh + 2 * i] = flt[o_wh + 2 * i + 1] = rw[i];
    std::vector<int32_t> ints;
    auto put = [&](const std::vector<int32_t>& v) { size_t o = ints.size(); ints.insert(ints.end(), v.begin(), v.end()); return o; };
    auto pairs = [&](const std::vector<int32_t>& a, const std::vector<int32_t>& b) {
        const size_t o = ints.size();
        for (size_t i = 0; i < a.size(); ++i) { ints.push_back(a[i]); ints.push_back(b[i]); }
        return o;
    };
    const size_t o_tw = pairs(xw, nw), o_th = pairs(xh, nh), o_c0 = put(cc0), o_cl = put(clen), o_r0 = put(rr0), o_rn = put(rnr), o_wi = put(win);
    const size_t fb = frag.size() * 2, wb = flt.size() * 4, bytes = fb + wb + ints.size() * 4;   // (operands and weights: 16-byte, pairs: 8-byte boundaries)
    if (cudaMalloc(&pl->dev, bytes) != cudaSuccess) { delete pl; return nullptr; }
    std::vector<uint8_t> host(bytes);
    memcpy(host.data(), frag.data(), fb);
    memcpy(host.data() + fb, flt.data(), wb);
    memcpy(host.data() + fb + wb, ints.data(), ints.size() * 4);
    if (cudaMemcpy(pl->dev, host.data(), bytes, cudaMemcpyHostToDevice) != cudaSuccess) { cudaFree(pl->dev); delete pl; return nullptr; }
    const uint8_t* dev = reinterpret_cast<const uint8_t*>(pl->dev);
    pl->frag = reinterpret_cast<const uint4*>(dev);
    pl->wt_w = reinterpret_cast<const float*>(dev + fb); pl->wt_h = pl->wt_w + o_wh;
    const int32_t* dip = reinterpret_cast<const int32_t*>(dev + fb + wb);
    pl->tap_w = dip + o_tw; pl->tap_h = dip + o_th;
    pl->col_c0 = dip + o_c0; pl->col_len = dip + o_cl; pl->row_r0 = dip + o_r0; pl->row_nr = dip + o_rn; pl->win = dip + o_wi;
    return pl;
}

void resize_plan_destroy(ResizePlan* pl) {
    if (!pl) return;
    if (pl->dev) cudaFree(pl->dev);
    delete pl;
}

void resize_plan_info(const ResizePlan* pl, int* th, int* max_rows, int64_t* smem) {
    if (th) *th = pl->th;
    if (max_rows) *max_rows = pl->max_rows;
    if (smem) *smem = (int64_t)pl->smem;
}

template <int KS, bool W4>
static int resize_launch(const ResizeParams& p, dim3 grid, size_t smem, cudaStream_t s) {
    if (ensure_dyn_smem(g_resize_smem[KS][W4], resize_bicubic_aa_u8_kernel<KS, W4>, 227 * 1024)) return -2;
    count_launch();
    resize_bicubic_aa_u8_kernel<KS, W4><<<grid, RS_THREADS, smem, s>>>(p);
    return 0;
}

int resize_bicubic_aa_u8(const ResizePlan* pl, const uint8_t* src, int planes, uint8_t* dst, cudaStream_t s) {
    if (!pl || planes <= 0 || planes > 65535 || pl->row_tiles > 65535) return -1;
    ResizeParams p;
    p.src = src; p.dst = dst;
    p.src_bytes = (size_t)planes * pl->h * pl->w;
    p.h = pl->h; p.w = pl->w; p.H = pl->H; p.W = pl->W;
    p.tap_w = reinterpret_cast<const int2*>(pl->tap_w); p.wt_w = pl->wt_w;
    p.tap_h = reinterpret_cast<const int2*>(pl->tap_h); p.wt_h = reinterpret_cast<const float2*>(pl->wt_h);
    p.col_c0 = pl->col_c0; p.col_len = pl->col_len; p.row_r0 = pl->row_r0; p.row_nr = pl->row_nr;
    p.win = pl->win; p.frag = pl->frag; p.frag_scale = pl->frag_scale; p.bound = pl->bound; p.ks = pl->ks;
    p.taps_w = pl->taps_w; p.taps_h = pl->taps_h; p.th = pl->th; p.tw_log2 = pl->tw_log2; p.rows16 = pl->rows16; p.stride = pl->stride; p.dense = pl->dense;
    const dim3 grid(pl->col_tiles, pl->row_tiles, planes);
    // Both axes enlarged (5 taps) and CTAs of one wave (4 per SM): the stated order throughout has fewer steps behind one another than products, test and doubtful
    // pixels. One frame, products | stated: 360x640 -> 448x796 7.8 | 6.8 us, 300x400 -> 560x784 8.3 | 7.7; two 10.7 | 10.3 and 13.0 | 12.0; three (more
    // than a wave) 13.8 | 14.2 and 15.9 | 16.1. With an axis made smaller: 480x640 -> 280x784 7.5 | 8.0, 480x854 -> 448x796 8.2 | 8.9.
    if (pl->taps_w <= 5 && pl->taps_h <= 5 && (size_t)grid.x * grid.y * grid.z <= 4 * kSms) p.dense = -1;
    const bool w4 = ((p.w | (int)reinterpret_cast<uintptr_t>(src)) & 3) == 0;   // every row starts on a word boundary
    switch (pl->ks) {
        case 1: return w4 ? resize_launch<1, true>(p, grid, pl->smem, s) : resize_launch<1, false>(p, grid, pl->smem, s);
        case 2: return w4 ? resize_launch<2, true>(p, grid, pl->smem, s) : resize_launch<2, false>(p, grid, pl->smem, s);
        case 3: return w4 ? resize_launch<3, true>(p, grid, pl->smem, s) : resize_launch<3, false>(p, grid, pl->smem, s);
        case 4: return w4 ? resize_launch<4, true>(p, grid, pl->smem, s) : resize_launch<4, false>(p, grid, pl->smem, s);
        default: return w4 ? resize_launch<0, true>(p, grid, pl->smem, s) : resize_launch<0, false>(p, grid, pl->smem, s);
    }
}

}  // namespace lcc
