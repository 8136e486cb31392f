// C-ABI entry points every model family needs: context, launch counter, the tensor-core GEMM and token selection.
// Kept apart from cabi.cu so that a library holding only one model family's kernels can be linked.
#include "../../include/livecc_b200.h"
#include "cabi_common.h"
#include "gemm.h"
#include "launch.h"
#include "ops.h"
#include "seqmix.h"

#include <deque>
#include <mutex>

using lcc::bf16;

namespace {

// Fault words of the contexts, in mapped host memory that every device sees. Allocating such memory waits for whatever the GPU is doing (a
// context beside running work took 340 ms for 3), so a page is taken once and its words go round: the one given back last is handed out last,
// 1024 contexts later, when no kernel of its former owner can be under way. Pages stay for the life of the process (one per 1024 live contexts).
std::mutex g_words_mu;
std::deque<int*>& words() {
    static auto* w = new std::deque<int*>;
    return *w;
}
int* take_fault_word() {
    std::lock_guard<std::mutex> lock(g_words_mu);
    if (words().empty()) {
        int* page = nullptr;
        constexpr int n = 1024;
        if (cudaHostAlloc((void**)&page, n * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;   // (no pinned memory to be had: a lost signal then shows as NaN only)
        }
        for (int i = 0; i < n; ++i) words().push_back(page + i);
    }
    int* w = words().front();
    words().pop_front();
    *w = 0;
    return w;
}
void give_fault_word(int* w) {
    if (!w) return;
    std::lock_guard<std::mutex> lock(g_words_mu);
    words().push_back(w);
}

}  // namespace

extern "C" {

int lcc_abi_version(void) { return LCC_ABI_VERSION; }

lcc_ctx* lcc_create(int device) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return nullptr;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return nullptr;
    if (prop.major != 10) return nullptr;  // sm_100a only: there is no fallback path
    if (cudaSetDevice(device) != cudaSuccess) return nullptr;
    lcc_ctx* c = new lcc_ctx();
    c->device = device;
    c->num_sms = prop.multiProcessorCount;
    c->err[0] = 0;
    c->fault = take_fault_word();
    return c;
}

void lcc_destroy(lcc_ctx* ctx) {
    if (!ctx) return;
    give_fault_word(ctx->fault);
    delete ctx;
}

int lcc_check_fault(lcc_ctx* ctx) {
    if (!ctx) return -1;
    LCC_CHECK_FAULT(ctx, "lcc_check_fault");
    return 0;
}

const char* lcc_last_error(lcc_ctx* ctx) { return ctx ? ctx->err : "null ctx"; }

int lcc_num_sms(lcc_ctx* ctx) { return ctx ? ctx->num_sms : -1; }

uint64_t lcc_launch_count(void) { return lcc::g_launches.load(std::memory_order_relaxed); }

int lcc_gemm_bf16(lcc_ctx* ctx, const void* A, int lda, const void* B, int ldb, void* C, int ldc,
                  int M, int N, int K, const void* bias, const void* residual, int ldr, int epilogue,
                  int block_n, void* splitk_ws, int64_t splitk_ws_bytes, lcc_stream_t stream) {
    if (!ctx) return -1;
    lcc::GemmArgs a;
    a.splitk_ws = splitk_ws;
    a.splitk_ws_bytes = splitk_ws_bytes > 0 ? (size_t)splitk_ws_bytes : 0;
    a.A = A; a.B = B; a.C = C;
    a.M = M; a.N = N; a.K = K;
    a.lda = lda; a.ldb = ldb; a.ldc = ldc;
    a.bias = bias; a.residual = residual; a.ldr = ldr;
    a.epi = epilogue; a.block_n = block_n; a.fault = ctx->fault;
    int r = lcc::gemm_bf16_tn(a, ctx->num_sms, (cudaStream_t)stream);
    if (r) LCC_FAIL(ctx, r, "lcc_gemm_bf16 failed (code %d; M=%d N=%d K=%d epi=%d)", r, M, N, K, epilogue);
    LCC_CHECK_FAULT(ctx, "lcc_gemm_bf16");
    return 0;
}

int lcc_gemm_plan(int num_sms, int M, int N, int K, int32_t* plan) {
    if (!plan || num_sms < 2 || M < 1 || N < 1 || K < 1) return -1;
    lcc::GemmArgs a{};
    a.M = M; a.N = N; a.K = K;
    a.epi = lcc::EPI_NONE;
    const lcc::GemmPlan p = lcc::gemm_plan(a, num_sms);
    plan[0] = p.form; plan[1] = p.width; plan[2] = p.splits;
    return 0;
}

int lcc_gemm_form(lcc_ctx* ctx, const void* A, int lda, const void* B, int ldb, void* C, int ldc, int M, int N, int K, const void* bias,
                  const void* residual, int ldr, int epilogue, int form, int width, int splits, float limit, float alpha, float up_bias,
                  int64_t wait_ns, lcc_stream_t stream) {
    if (!ctx || wait_ns < 0) return -1;
    lcc::GemmArgs a{};
    a.fault = ctx->fault; a.wait_ns = (uint64_t)wait_ns;
    a.A = A; a.B = B; a.C = C;
    a.M = M; a.N = N; a.K = K;
    a.lda = lda; a.ldb = ldb; a.ldc = ldc;
    a.bias = bias; a.residual = residual; a.ldr = ldr;
    a.epi = epilogue; a.epi_param = limit; a.epi_alpha = alpha; a.epi_up_bias = up_bias;
    int r = form < lcc::FORM_ONE || form > lcc::FORM_SWAP ? -6 : lcc::gemm_bf16_tn_form(a, (lcc::GemmForm)form, width, splits, ctx->num_sms, (cudaStream_t)stream);
    if (r) LCC_FAIL(ctx, r, "lcc_gemm_form failed (code %d; M=%d N=%d K=%d epi=%d form=%d width=%d splits=%d)", r, M, N, K, epilogue, form, width, splits);
    LCC_CHECK_FAULT(ctx, "lcc_gemm_form");
    return 0;
}

#define OP_RET(ctx, expr, name)                                              \
    do {                                                                     \
        if (!(ctx)) return -1;                                               \
        int rc__ = (expr);                                                   \
        if (rc__) LCC_FAIL(ctx, rc__, name " failed (code %d)", rc__);       \
        LCC_CHECK_LAUNCH(ctx, name);                                         \
        return 0;                                                            \
    } while (0)

int lcc_gated_scan(lcc_ctx* ctx, int dt, const void* k, int ld_k, const void* c, int ld_c, const void* u, int ld_u, float* log_decay, int vec_decay,
                   const float* sc, const float* skip, float cs, float* state, float* y, int ld_y, int S, int heads, int heads_per_group, int N, int P,
                   float* ws, int64_t ws_floats, lcc_stream_t stream) {
    lcc::ScanArgs a{};
    a.dt = dt; a.k = k; a.ld_k = ld_k; a.c = c; a.ld_c = ld_c; a.u = u; a.ld_u = ld_u;
    a.a = log_decay; a.vec_decay = vec_decay; a.sc = sc; a.skip = skip; a.cs = cs; a.state = state; a.y = y; a.ld_y = ld_y;
    a.S = S; a.heads = heads; a.heads_per_group = heads_per_group; a.N = N; a.P = P;
    a.ws = ws; a.ws_floats = ws_floats > 0 ? (size_t)ws_floats : 0;
    if (dt != lcc::DT_F32 && dt != lcc::DT_BF16) return -1;
    OP_RET(ctx, lcc::gated_scan(a, lcc::SeqPos{}, (cudaStream_t)stream), "lcc_gated_scan");
}

int lcc_attn_masked(lcc_ctx* ctx, int dt, const float* q, const void* k_pages, const void* v_pages, const int32_t* page_table, int page_size, const void* gate,
                    int ld_gate, int gate_channel, void* out, int ld_out, int S, int past, int Hq, int G, int D, int DV, int chunk, int window, int sink,
                    float scale, lcc_stream_t stream) {
    if (dt != lcc::DT_F32 && dt != lcc::DT_BF16) return -1;
    lcc::AttnOpts o;
    o.window = window; o.no_sink = !sink; o.gate_channel = gate_channel != 0;
    OP_RET(ctx, lcc::attn_masked(dt, q, k_pages, v_pages, page_table, page_size, gate, ld_gate, out, ld_out, S, Hq, G, D, DV, chunk, scale, true,
                                 lcc::SeqPos{past, nullptr, nullptr}, (cudaStream_t)stream, o), "lcc_attn_masked");
}

int64_t lcc_gated_scan_ws_floats(int S, int heads, int N, int P) { return (int64_t)lcc::gated_scan_ws_floats(S, heads, N, P); }

int lcc_sample_greedy(lcc_ctx* ctx, const float* logits_raw, float* logits_proc, int V, int64_t* seq,
                      int32_t* scalars, const lcc_sampling* sp, int advance_kv, const void* embed, void* h,
                      int H, lcc_stream_t stream) {
    if (!sp) return -1;
    lcc::SampleArgs a{};
    a.logits_raw = logits_raw; a.logits_proc = logits_proc; a.V = V; a.seq = seq; a.scalars = scalars;
    a.repetition_penalty = sp->repetition_penalty; a.inv_repetition_penalty = sp->inv_repetition_penalty; a.thr_token = sp->thr_token; a.thr_base = sp->thr_base;
    a.thr_step = sp->thr_step; a.eos_token_id = sp->eos_token_id; a.eos_token_id2 = sp->eos_token_id2;
    a.max_new_tokens = sp->max_new_tokens;
    a.advance_kv = advance_kv; a.embed = (const bf16*)embed; a.h = (bf16*)h; a.H = H;
    OP_RET(ctx, lcc::sample_greedy(a, (cudaStream_t)stream), "lcc_sample_greedy");
}

}  // extern "C"
