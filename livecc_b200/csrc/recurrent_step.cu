// One token of a gated linear recurrence with everything around it in one kernel: a decode step of a state-space layer (short causal convolution and
// silu, step sizes and decays, recurrence, skip, gate, group norm) or of gated linear attention (decays, recurrence, head norm, gate). As kernels
// of their own (recurrent.cu, rowops.cu) these are four and three links of a step's chain, each waiting for the one before it to leave the chip:
// 1.2 + 2.8 + 7.6 + 3.3 us and 1.1 + 4.2 + 2.6 us of a step of 239 (width 2048, 64 heads of 64 x 128 | 8 heads of 256 x 128). Here 5.3 and 4.1, and the
// step takes 205; a prompt of 128 tokens and 31 steps 7.21 ms for 8.18.
//
// A cluster of 8 CTAs owns the channels of one norm group, a CTA an eighth of them: value channels of one head, whose states are one contiguous block.
// The state (32 KB a CTA), what the convolution carries, its weights and the norm's were written before the kernel in front started: they are
// loaded before the wait, all in flight together. What the group has in common (its sum of squares) goes through the cluster's shared memory.
#include <math.h>

#include "../../include/livecc_b200.h"
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
template <typename T> __device__ __forceinline__ float stored(float v);      // as the storage type holds it
template <> __device__ __forceinline__ float stored<float>(float v) { return v; }
template <> __device__ __forceinline__ float stored<bf16>(float v) { return rbf(v); }

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }

constexpr int kStepCtas = 8, kStepThreads = 256, kStepTaps = 4, kStepChannels = 128, kStepState = 128;

// E: float4 pieces of state per thread. A piece's lanes: N / 4 neighbouring ones hold a channel.
template <typename T, bool CONV, int E>
__global__ void __cluster_dims__(kStepCtas, 1, 1) __launch_bounds__(kStepThreads) scan_step_kernel(const __grid_constant__ ScanStep a, SeqPos pos) {
    __shared__ __align__(16) float sk[kStepState], sc[kStepState], sd[kStepState];
    __shared__ float su[kStepChannels], sy[kStepChannels], part[kStepCtas], red[32], dt_s, decay_s;
    const int tid = threadIdx.x, N = a.N, N4 = N >> 2, PC = a.group / kStepCtas;
    const int c0 = blockIdx.x * PC, h = c0 / a.P, g = h / a.heads_per_group;      // (a cluster's CTAs are neighbours, so are its channels)
    const int HP = a.heads * a.P, GN = a.heads / a.heads_per_group * N;
    cluster_arrive();
    // ---- written before the kernel in front started
    float4* gs = reinterpret_cast<float4*>(a.state + (size_t)c0 * N);
    float4 st[E];
#pragma unroll
    for (int i = 0; i < E; ++i) st[i] = gs[tid + kStepThreads * i];
    // the convolution's channels of this CTA: its own value channels, then the key and read-out channels of its group
    constexpr int SLOTS = CONV ? 2 : 1;
    int chan[SLOTS];
    float cw[SLOTS][kStepTaps], cx[SLOTS][kStepTaps], cb[SLOTS];
    if (CONV) {
#pragma unroll
        for (int i = 0; i < SLOTS; ++i) {
            const int s = tid + kStepThreads * i;
            chan[i] = s < PC ? c0 + s : s < PC + N ? HP + g * N + s - PC : s < PC + 2 * N ? HP + GN + g * N + s - PC - N : -1;
            cb[i] = chan[i] >= 0 ? a.conv_b[chan[i]] : 0.f;
#pragma unroll
            for (int j = 0; j < kStepTaps; ++j) {
                cw[i][j] = chan[i] >= 0 && j < a.taps ? a.conv_w[(size_t)chan[i] * a.taps + j] : 0.f;
                cx[i][j] = chan[i] >= 0 && j < a.taps - 1 ? a.carry[(size_t)chan[i] * (a.taps - 1) + j] : 0.f;
            }
        }
    }
    const float bias = CONV ? a.dt_bias[h] : 0.f, rate = CONV ? -expf(a.a_log[h]) : a.inv_tau, skip = a.skip ? a.skip[h] : 0.f;
    const float wn = tid < PC ? a.norm_w[(c0 + tid) % a.w_len] : 0.f;
    chain_begin();
    cluster_wait();
    if (pos.finished && *pos.finished) return;
    // ---- the token's rows
    const float gate = tid < PC ? ldf((const T*)a.gate + c0 + tid) : 0.f;
    if (CONV) {
        const T* in = (const T*)a.u;
        if (tid == kStepThreads - 1) {
            const float dt = softplus_f(ldf((const T*)a.dec + h) + bias);
            dt_s = dt;
            decay_s = expf(rate * dt);
        }
#pragma unroll
        for (int i = 0; i < SLOTS; ++i) {
            const int s = tid + kStepThreads * i;
            if (chan[i] < 0) continue;
            const float x = ldf(in + chan[i]);
            float acc = cb[i];
#pragma unroll
            for (int j = 0; j < kStepTaps; ++j) {
                if (j == a.taps - 1) cx[i][j] = x;
                if (j < a.taps) acc = fmaf(cw[i][j], cx[i][j], acc);
            }
            const float v = stored<T>(silu_f(acc));
            if (s < PC) su[s] = v;
            else if (s < PC + N) sk[s - PC] = v;
            else sc[s - PC - N] = v * a.cs;
        }
    } else {
        for (int n = tid; n < N; n += kStepThreads) {
            sk[n] = ldf((const T*)a.k + g * N + n);
            sc[n] = ldf((const T*)a.c + g * N + n) * a.cs;
            const float z = ldf((const T*)a.dec + h * N + n);
            sd[n] = expf((fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * rate);    // log(sigmoid(z)) = min(z, 0) - log1p(exp(-|z|))
        }
        if (tid < PC) su[tid] = ldf((const T*)a.u + c0 + tid);
    }
    __syncthreads();
    // ---- recurrence
    const int n = (tid & (N4 - 1)) * 4;
    const float4 k4 = *reinterpret_cast<const float4*>(sk + n), c4 = *reinterpret_cast<const float4*>(sc + n);
    const float4 d4 = CONV ? make_float4(decay_s, decay_s, decay_s, decay_s) : *reinterpret_cast<const float4*>(sd + n);
    const float step = CONV ? dt_s : 1.f;
    float y[E];
#pragma unroll
    for (int i = 0; i < E; ++i) {
        const float u = su[(tid + kStepThreads * i) / N4] * step;
        st[i].x = fmaf(d4.x, st[i].x, k4.x * u); st[i].y = fmaf(d4.y, st[i].y, k4.y * u);
        st[i].z = fmaf(d4.z, st[i].z, k4.z * u); st[i].w = fmaf(d4.w, st[i].w, k4.w * u);
        y[i] = fmaf(st[i].w, c4.w, fmaf(st[i].z, c4.z, fmaf(st[i].y, c4.y, st[i].x * c4.x)));
    }
#pragma unroll
    for (int i = 0; i < E; ++i) gs[tid + kStepThreads * i] = st[i];
    for (int o = N4 >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < E; ++i) y[i] += __shfl_xor_sync(0xffffffffu, y[i], o);
    if ((tid & (N4 - 1)) == 0) {
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const int c = (tid + kStepThreads * i) / N4;
            sy[c] = fmaf(skip, su[c], y[i]);
        }
    }
    __syncthreads();
    // ---- norm over the group
    const float act = a.gate_first == 2 ? sigmoid_f(gate) : silu_f(gate);
    float v = tid < PC ? sy[tid] : 0.f;
    if (a.gate_first == 1) v *= act;
    const float ss = block_sum(tid < PC ? v * v : 0.f, red);
    if (tid < kStepCtas) {
        const uint32_t at = mapa_shared(smem_u32(part + cluster_ctarank()), tid);
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(ss) : "memory");
    }
    cluster_sync_all();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < kStepCtas; ++i) total += part[i];
    const float rn = 1.f / sqrtf(total / (float)a.group + a.eps);
    if (tid < PC) stf((T*)a.out + c0 + tid, a.gate_first == 1 ? v * rn * wn : v * rn * wn * act);
    if (CONV) {   // what the next token's convolution reads: own channels, and the group's by its first CTA, now that all of its CTAs have read them
        const bool first = c0 % (a.heads_per_group * a.P) == 0;
#pragma unroll
        for (int i = 0; i < SLOTS; ++i) {
            if (chan[i] < 0 || (!first && tid + kStepThreads * i >= PC)) continue;
#pragma unroll
            for (int j = 1; j < kStepTaps; ++j)
                if (j < a.taps) a.carry[(size_t)chan[i] * (a.taps - 1) + j - 1] = cx[i][j];
        }
    }
}

template <typename T, bool CONV>
int launch_step(const ScanStep& a, SeqPos pos, cudaStream_t s) {
    const dim3 grid(a.heads * a.P / a.group * kStepCtas);
    count_launch();
    switch (a.group / kStepCtas * a.N / 4 / kStepThreads) {
        case 1: chained(scan_step_kernel<T, CONV, 1>, grid, kStepThreads, 0, s)(a, pos); break;
        case 2: chained(scan_step_kernel<T, CONV, 2>, grid, kStepThreads, 0, s)(a, pos); break;
        case 4: chained(scan_step_kernel<T, CONV, 4>, grid, kStepThreads, 0, s)(a, pos); break;
        case 8: chained(scan_step_kernel<T, CONV, 8>, grid, kStepThreads, 0, s)(a, pos); break;
        default: return -2;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -100;
}

}  // namespace

bool scan_step_takes(const ScanStep& a) {
    const int HP = a.heads * a.P, PC = a.group / kStepCtas;
    if (!(a.N == 32 || a.N == 64 || a.N == 128) || a.group < 1 || a.group % kStepCtas || HP % a.group || PC > kStepChannels || a.P % PC) return false;
    const int pieces = PC * a.N / 4, e = pieces / kStepThreads;
    if (pieces % kStepThreads || !(e == 1 || e == 2 || e == 4 || e == 8) || (uintptr_t)a.state % 16) return false;
    if (!a.conv_w) return true;
    // a key group's channels are carried on by one CTA, behind a barrier of the cluster: the group lies inside it
    return a.taps >= 2 && a.taps <= kStepTaps && PC + 2 * a.N <= 2 * kStepThreads && a.group % (a.heads_per_group * a.P) == 0;
}

int scan_step(const ScanStep& a, SeqPos pos, cudaStream_t s) {
    if (!scan_step_takes(a)) return -2;
    if (a.dt == LCC_DT_F32) return a.conv_w ? launch_step<float, true>(a, pos, s) : launch_step<float, false>(a, pos, s);
    return a.conv_w ? launch_step<bf16, true>(a, pos, s) : launch_step<bf16, false>(a, pos, s);
}

}  // namespace lcc
