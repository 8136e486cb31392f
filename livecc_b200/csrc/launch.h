// Launch helper: ordinary launch or programmatic dependent launch (PDL) of a kernel.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <stdint.h>

namespace lcc {

// Process-wide count of kernel launches issued by this library (every launch site calls count_launch()). Launches
// recorded into a CUDA graph are counted once at capture; the host adds (nodes x replays) itself. Read through
// lcc_launch_count() (bench.py's `gpu_launches` is this counter, not arithmetic).
inline std::atomic<uint64_t> g_launches{0};
inline void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// SMs of a B200, for the sizes of grids whose kernels run whatever the number is (the entry points take the device's own count).
constexpr int kSms = 148;

// cudaFuncAttributeMaxDynamicSharedMemorySize is a per-device attribute of a kernel: remember per (kernel
// instantiation, device) that it was raised, so a second engine on another device of the same process works.
struct SmemAttrOnce {
    bool set[64] = {};
};
template <typename Kern>
inline int ensure_dyn_smem(SmemAttrOnce& once, Kern kern, int bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
    if (!once.set[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return -1;
        once.set[dev] = true;
    }
    return 0;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                 bool pdl, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// A chain of short kernels: inside a ChainScope each may be set up while the one before it in the stream still runs (programmatic dependent
// launch), and chain_begin() in common.cuh, by which it begins, waits for that one. A step of the hybrid models is 30 (recurrent design, four layers) and 22
// kernels of 2 to 10 us on one row; as ordinary graph nodes, kernels that return at once cost 2.7 to 4 us each. Chained, and with the first
// weights of a linear layer loaded before the wait, a prompt of 128 tokens and 31 replayed steps took 8.29 ms for 8.48 (recurrent design, then
// 45 kernels a step) and 4.86 for 5.14 (routed, two layers), one step launched by the host 0.32 ms for 0.38 and 0.33 for 0.36 (four layers each).
// Matrix products, row kernels and attention of the vision tower and of a prefill are chained too: what they set up (barriers, tensor memory, tensor
// maps) and their launch lie beside the kernel in front. A turn that reads 281 tokens behind 17 k 1.45 -> 1.39 ms, eight streams' turn 11.99 -> 11.93,
// 1024 and 8192 patches 453 -> 440 and 1132 -> 1105 us, prompts of the hybrid models 1.72 -> 1.67 and 0.56 -> 0.525 ms.
// A kernel that takes tensor memory takes it before it opens the door to the next one: that one could otherwise hold what this one waits for.
// (The first stages' weights asked for before the wait changed little, turn by turn -1 to +0.6 %.) Prompt attention of the hybrid models (few and large
// CTAs) stays outside: chained, its CTAs go where there is room while the kernel in front still holds the other SMs, and stay there two to an SM.
// 281 rows behind 4000 tokens of four layers with distance tables took 2.59 ms unchained, 2.76 with every kernel chained, 2.52 now. So do the decoder's
// decode kernels: each of their thousands of CTAs would pay for the wait with its cached activations (gate/up 44 -> 50 us, lm_head 170 -> 202).
// (An ordinary kernel of a scope lets the one behind it in when it is complete.)
// The first launch of a scope and the one after chain_break() (behind a copy, a fork or a join with another stream) are ordinary: whatever
// was enqueued before is complete when they start. Outside a scope every launch is.
enum class Chain { off, broken, on };
inline thread_local Chain t_chain = Chain::off;   // of the launching thread
inline void chain_break() { if (t_chain == Chain::on) t_chain = Chain::broken; }
struct ChainScope {
    ChainScope() { t_chain = Chain::broken; }
    ~ChainScope() { t_chain = Chain::off; }
    ChainScope(const ChainScope&) = delete;
    ChainScope& operator=(const ChainScope&) = delete;
};

// Is the launch that comes next chained? (Asked once for each launch of a scope.)
inline bool chain_next() {
    const bool chain = t_chain == Chain::on;
    if (t_chain == Chain::broken) t_chain = Chain::on;
    return chain;
}

template <typename... KArgs>
struct ChainLaunch {
    void (*kern)(KArgs...);
    dim3 grid, block;
    size_t smem;
    cudaStream_t s;
    template <typename... Args>
    void operator()(Args... args) const {
        launch_kernel(kern, grid, block, smem, s, chain_next(), args...);   // (an error stays in cudaGetLastError, as with <<<>>>)
    }
};
template <typename... KArgs>
inline ChainLaunch<KArgs...> chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    return {kern, grid, block, smem, s};
}

}  // namespace lcc
