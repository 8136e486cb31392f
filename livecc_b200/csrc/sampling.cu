// Token selection for one stream, fused into one launch per step (the reference spends ~10
// tiny launches and a host sync per token here: gen/utils.py:2762-2805):
//   RepetitionPenaltyLogitsProcessor (logits_process.py:407-410) over the whole id history,
//   optional ThresholdLogitsProcessor (REF/demo/infer.py:10-23),
//   argmax (greedy; gen/utils.py:2793), EOS / max_new_tokens stop, append to the sequence buffer,
//   advance of the device-side stream scalars, and the embedding row of the chosen token for the
//   next decode step (mq2vl.py:1256).
// Everything the next step needs stays on the device, so a whole generate() call runs without a host sync.
//
// What bounds it is latency: one SM has too few loads in flight for 152k logits and a long history. A stream is served by one
// cluster of kCl CTAs (8, the portable size): each takes 1/8 of the history and of the vocabulary, the partial results meet in
// the CTAs' shared memory, and no scratch in global memory is needed. One CTA per
// stream took 33 us with 8k ids of history and 94 us with 65k; a 16-token turn of four layers over 65k tokens went from 13.41 to 12.31 ms
// with the cluster, over 8k tokens from 11.45 to 11.20 ms.
#include "../../include/livecc_b200.h"
#include "common.cuh"
#include "launch.h"
#include "ops.h"

namespace lcc {

constexpr int kCl = 8, kThreads = 1024;

// Stores a 32-bit value at `dst`'s place in the shared memory of cluster CTA `rank`.
__device__ __forceinline__ void st_cluster(const void* dst, uint32_t v, uint32_t rank) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_shared(smem_u32(dst), rank)), "r"(v) : "memory");
}

// Warp 0 of every CTA hands its value to all CTAs of the cluster (slot = the sender's rank); after the barrier each of them reads all
// kCl slots. A slot array is used once per launch.
__device__ __forceinline__ void cluster_share(float (&slots)[kCl], float v, uint32_t rank) {
    if (threadIdx.x < kCl) st_cluster(&slots[rank], __float_as_uint(v), threadIdx.x);
    __syncwarp();
    cluster_sync_all();
}

__device__ __forceinline__ void sample_greedy_body(const SampleArgs& a) {
    int* sc = a.scalars;
    // (every CTA reads the scalars before the first cluster barrier; rank 0 changes them after the last one)
    if (sc[LCC_SC_FINISHED]) return;
    __shared__ float red_v[32];
    __shared__ int red_i[32];
    __shared__ float cl_max[kCl], cl_sum[kCl], cl_best[kCl];
    __shared__ int cl_idx[kCl];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = cluster_ctarank();
    const int first = (int)rank * kThreads + tid, step = kCl * kThreads;
    const int hist = sc[LCC_SC_SEQ_LEN];
    const bool threshold = a.thr_token >= 0 && a.thr_token < a.V;

    // 1. repetition penalty: gather from raw, scatter to proc (idempotent under duplicate ids)
    if (a.repetition_penalty != 1.0f) {
        // torch's CUDA `scores / penalty` multiplies by fp32(1.0 / (double)penalty); the host passes that value
        const float inv_pen = a.inv_repetition_penalty != 0.f ? a.inv_repetition_penalty : 1.0f / a.repetition_penalty;
#pragma unroll 4
        for (int i = first; i < hist; i += step) {
            const int64_t id = a.seq[i];
            if (id >= 0 && id < a.V) {
                const float v = a.logits_raw[id];
                a.logits_proc[id] = v < 0.f ? v * a.repetition_penalty : v * inv_pen;
            }
        }
    }
    __syncwarp();
    cluster_sync_all();   // the penalised logits are visible to the whole cluster (read below past L1); all CTAs have read the scalars

    // 2. optional streaming-EOS threshold: if softmax(scores)[tok] <= thr then scores[tok] = -inf
    if (threshold) {
        float mx = -INFINITY;
        for (int i = first; i < a.V; i += step) mx = fmaxf(mx, __ldcg(a.logits_proc + i));
        mx = warp_max(mx);
        if (lane == 0) red_v[warp] = mx;
        __syncthreads();
        if (warp == 0) mx = warp_max(red_v[lane]);
        cluster_share(cl_max, mx, rank);
        mx = cl_max[0];
#pragma unroll
        for (int r = 1; r < kCl; ++r) mx = fmaxf(mx, cl_max[r]);
        float se = 0.f;
        for (int i = first; i < a.V; i += step) se += expf(__ldcg(a.logits_proc + i) - mx);
        se = warp_sum(se);
        if (lane == 0) red_v[warp] = se;   // (the cluster barrier above also ordered the reads of red_v)
        __syncthreads();
        if (warp == 0) se = warp_sum(red_v[lane]);
        cluster_share(cl_sum, se, rank);
        if (rank == 0 && tid == 0) {
            float tot = 0.f;
#pragma unroll
            for (int r = 0; r < kCl; ++r) tot += cl_sum[r];
            const float thr = a.thr_base + a.thr_step * (float)sc[LCC_SC_N_GENERATED];
            const float pr = expf(__ldcg(a.logits_proc + a.thr_token) - mx) / tot;
            if (pr <= thr) a.logits_proc[a.thr_token] = -INFINITY;
        }
        __syncwarp();
        cluster_sync_all();
    }

    // 3. argmax, lowest index on ties. float4 loads, up to 5 independent loads in flight per thread (152k logits).
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    const int V4 = a.V >> 2;
    const float4* lp4 = reinterpret_cast<const float4*>(a.logits_proc);
#pragma unroll 5
    for (int i = first; i < V4; i += step) {
        const float4 v = __ldcg(lp4 + i);
        const int b = i << 2;
        if (v.x > bv) { bv = v.x; bi = b; }  // indices increase per thread => first max kept
        if (v.y > bv) { bv = v.y; bi = b + 1; }
        if (v.z > bv) { bv = v.z; bi = b + 2; }
        if (v.w > bv) { bv = v.w; bi = b + 3; }
    }
    for (int i = (V4 << 2) + first; i < a.V; i += step) {
        const float v = __ldcg(a.logits_proc + i);
        if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { red_v[warp] = bv; red_i[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        bv = red_v[lane];
        bi = red_i[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) {
            st_cluster(&cl_best[rank], __float_as_uint(bv), 0);
            st_cluster(&cl_idx[rank], (uint32_t)bi, 0);
        }
    }
    __syncwarp();
    cluster_sync_all();
    if (rank != 0) return;
    bv = cl_best[0];
    bi = cl_idx[0];
#pragma unroll
    for (int r = 1; r < kCl; ++r)
        if (cl_best[r] > bv || (cl_best[r] == bv && cl_idx[r] < bi)) { bv = cl_best[r]; bi = cl_idx[r]; }
    const int tok = bi == 0x7fffffff ? 0 : bi;

    // 4. bookkeeping (single thread) + 5. embedding row for the next step (all threads of CTA 0)
    if (tid == 0) {
        a.seq[hist] = tok;
        sc[LCC_SC_SEQ_LEN] = hist + 1;
        const int n = sc[LCC_SC_N_GENERATED] + 1;
        sc[LCC_SC_N_GENERATED] = n;
        sc[LCC_SC_LAST_TOKEN] = tok;
        if (a.advance_kv) {
            sc[LCC_SC_KV_LEN] += 1;
            sc[LCC_SC_ROPE_POS] += 1;
        }
        if (tok == a.eos_token_id || tok == a.eos_token_id2 || n >= a.max_new_tokens) sc[LCC_SC_FINISHED] = 1;
    }
    if (!a.embed || !a.h) return;  // models whose step embeds the token itself (it reads the id from the sequence buffer)
    const bf16* src = a.embed + (size_t)tok * a.H;
    for (int c = tid * 8; c < a.H; c += kThreads * 8)
        *reinterpret_cast<uint4*>(a.h + c) = *reinterpret_cast<const uint4*>(src + c);
}

__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kThreads) sample_greedy_kernel(const SampleArgs a) { sample_greedy_body(a); }

// One cluster per stream of a batched decode step: stream b uses row b of the logits / hidden buffers and its own id
// buffer and scalars. Also publishes the decode kernel's sticky error flag in scalars[LCC_SC_NATIVE_ERROR].
__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kThreads) sample_greedy_batch_kernel(const SampleArgs base, const SampleBatch sb) {
    const int b = blockIdx.x / kCl;
    SampleArgs a = base;
    a.logits_raw = base.logits_raw + (size_t)b * base.V;
    a.logits_proc = base.logits_proc + (size_t)b * base.V;
    a.h = base.h + (size_t)b * base.H;
    a.seq = sb.seq[b];
    a.scalars = sb.scalars[b];
    if (sb.err && blockIdx.x % kCl == 0 && threadIdx.x == 0) {
        const int e = *sb.err;
        if (e) a.scalars[LCC_SC_NATIVE_ERROR] = e;
    }
    __syncwarp();
    sample_greedy_body(a);
}

int sample_greedy(const SampleArgs& a, cudaStream_t s) {
    if (a.V <= 0 || (a.embed && a.H % 8)) return -1;
    lcc::count_launch();
    sample_greedy_kernel<<<kCl, kThreads, 0, s>>>(a);
    return 0;
}

int sample_greedy_batch(const SampleArgs& base, const SampleBatch& sb, cudaStream_t s) {
    if (base.V <= 0 || base.H % 8 || sb.B < 1 || sb.B > 8) return -1;
    lcc::count_launch();
    sample_greedy_batch_kernel<<<sb.B * kCl, kThreads, 0, s>>>(base, sb);
    return 0;
}

}  // namespace lcc
