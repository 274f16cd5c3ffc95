// batch_decoder.cu — B independent request streams decoded in lockstep (all at the same position), one token each
// per step: the second workload of the whole-decoder benchmark (64 concurrent streams).
//
// Per layer the B hidden vectors go through the reference's BATCHED kernels: RMSNorm over rows, K-quant GEMMs with
// N = B tokens (gemm_quant_batched, src/kernels/gemv_q4.cu:2478-2495 — the prefill arithmetic, which is what the
// reference uses whenever more than one token is in flight), per-head q/k norm + RoPE + INT8 KV store for every stream,
// ragged-batch decode attention over the B caches, SwiGLU, residual adds; then the final norm, fp16 logits for the B
// rows and a greedy argmax per row on the device.  Weights are read once per step for all streams.
#include "../../include/jllm_b200.h"
#include "../../include/jllm_b200_api.hpp"
#include "common.cuh"
#include "elementwise.cuh"
#include "attention.cuh"
#include "mmq.cuh"
#include "gemv.cuh"
#include "mmq_few.cuh"
#include <cmath>
#include <new>
#include <vector>

namespace jb {

// greedy argmax of every row of fp16 logits [B][V] (lowest index among equal maxima, non-finite skipped); CTA (slice, row).
// One CTA per row left most of the machine idle (8 rows of 151936: 12.7 us, all of it the latency of a CTA's loads), so a row is cut into
// slices; the last CTA of a row to finish settles it, the last of all moves the step on: state[0] = position, state[2] = steps recorded,
// seq_lens[b] = position + 1 for the attention of the next step, tokens[b] = its prompt token while there are some.
constexpr int AR_SLICES = 16;
struct ArArgs {
    const __half* logits; int V, B; int* tokens; int* state; int* out; int out_cap; int* seq_lens; const int* prompt; int n_prompt;
    float* best; int* index; unsigned int* tickets;       // [B][AR_SLICES], [B][AR_SLICES], [1 + B], zero between steps
};
__device__ __forceinline__ void ar_take(float& best, int& bi, float v, int i) { if (v > best || (v == best && i < bi)) { best = v; bi = i; } }
__device__ __forceinline__ void ar_warp(float& best, int& bi) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o); const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
        ar_take(best, bi, ov, oi);
    }
}
__global__ void __launch_bounds__(1024) argmax_rows_kernel(const ArArgs a) {
    pdl_launch();
    pdl_wait();
    __shared__ float sv[32]; __shared__ int si[32]; __shared__ bool last_row, last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = blockIdx.y, S = gridDim.x, threads = S * blockDim.x, t0 = blockIdx.x * blockDim.x + tid;
    const __half* row = a.logits + (size_t)b * a.V;
    float best = -INFINITY; int bi = 0x7FFFFFFF;
    auto take = [&](float v, int i) { if (isfinite(v)) ar_take(best, bi, v, i); };
    if (a.V % 8 == 0 && ((uintptr_t)row & 15) == 0) {
        #pragma unroll 4
        for (int i = t0; i < a.V / 8; i += threads) {
            const uint4 w = reinterpret_cast<const uint4*>(row)[i];
            const uint32_t u[4] = {w.x, w.y, w.z, w.w};
            #pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[e]));
                take(f.x, 8 * i + 2 * e); take(f.y, 8 * i + 2 * e + 1);
            }
        }
    } else {
        for (int i = t0; i < a.V; i += threads) take(__half2float(row[i]), i);
    }
    ar_warp(best, bi);
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        best = lane < (int)(blockDim.x >> 5) ? sv[lane] : -INFINITY; bi = lane < (int)(blockDim.x >> 5) ? si[lane] : 0x7FFFFFFF;
        ar_warp(best, bi);
        if (lane == 0) {
            a.best[b * AR_SLICES + blockIdx.x] = best; a.index[b * AR_SLICES + blockIdx.x] = bi;
            __threadfence();
            last_row = atomicAdd(&a.tickets[1 + b], 1u) == (unsigned)S - 1;
        }
        __syncwarp();
        if (last_row) {
            __threadfence();
            best = lane < S ? __ldcg(&a.best[b * AR_SLICES + lane]) : -INFINITY; bi = lane < S ? __ldcg(&a.index[b * AR_SLICES + lane]) : 0x7FFFFFFF;
            ar_warp(best, bi);
            if (lane == 0) {
                if (bi == 0x7FFFFFFF) bi = 0;
                a.tickets[1 + b] = 0u;
                a.tokens[b] = bi;
                const int k = a.state[2];                 // every row reads it before the last of them moves it on
                if (a.out && k < a.out_cap) a.out[(size_t)k * a.B + b] = bi;
                __threadfence();
            }
        }
        if (lane == 0) last = last_row && atomicAdd(&a.tickets[0], 1u) == (unsigned)a.B - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int p = a.state[0] + 1;
    __syncthreads();
    if (tid == 0) { a.tickets[0] = 0u; a.state[0] = p; a.state[2] = a.state[2] + 1; }
    for (int i = tid; i < a.B; i += blockDim.x) {
        a.seq_lens[i] = p + 1;
        if (a.prompt && p < a.n_prompt) a.tokens[i] = a.prompt[(size_t)i * a.n_prompt + p];
    }
}
// the first step of a request: position 0
__global__ void batch_begin_kernel(int* state, int* seq_lens, int* tokens, const int* prompt, int n_prompt, int B) {
    pdl_wait();
    const int p = state[0];
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
        seq_lens[b] = p + 1;
        if (prompt && p < n_prompt) tokens[b] = prompt[(size_t)b * n_prompt + p];
    }
}

}  // namespace jb

using namespace jb;

struct jllm_b200_batch_decoder {
    jllm_b200_model_desc m;
    std::vector<jllm_b200_layer_desc> layers;
    std::vector<jllm::KVCachePool> kv;
    int B = 0;
    __half *x = nullptr, *x2 = nullptr, *normed = nullptr, *q = nullptr, *k = nullptr, *v = nullptr, *att = nullptr, *gate = nullptr,
           *up = nullptr, *sw = nullptr, *y = nullptr, *logits = nullptr;
    float* best = nullptr; int* best_at = nullptr; unsigned int* tickets = nullptr;      // argmax_rows_kernel
    int *state = nullptr, *tokens = nullptr, *seq_lens = nullptr, *out_tokens = nullptr, *prompt_dev = nullptr;
    int out_cap = 0, prompt_cap = 0;
    void** lists = nullptr;            // device: [layer][4 (k, v, k scales, v scales)][B] pointers
    std::vector<unsigned char> maps;   // host: [layer][B][K, V] TMA tensor maps of the caches (128 bytes each), passed to the kernel as parameters
    void* slab = nullptr;
    MfModel few;                       // the products of up to MF_MAX_TOKENS streams; its scratch is in the slab too
    MmqWork mmq;                       // in the slab: the captured step holds its addresses, all of it is there from the start
    int kernels_per_step = 0;
    cudaGraphExec_t graph_exec = nullptr;   // one decode step from the device-side state
    int host_pos = -1;                      // host mirror of the device-side position (-1 until generate has run): the bound of step_device
};

#define BCHK(call) do { const int rc__ = (call); if (rc__) return rc__; } while (0)

static int bdec_enqueue_step(jllm_b200_batch_decoder* d, const int* prompt, int n_prompt, cudaStream_t st) {
    const jllm_b200_model_desc& m = d->m;
    const int B = d->B, H = m.hidden_dim, QD = m.n_heads * m.head_dim, KVD = m.n_kv_heads * m.head_dim, I = m.intermediate_dim, V = m.vocab_size;
    const float scale = 1.0f / sqrtf((float)m.head_dim);
    const long long l0 = jllm_b200_launch_count();
    BCHK(launch_embed_rows(d->x, m.tok_embd, m.embd_type, d->tokens, B, H, st));
    MfModel& f = d->few;
    const bool few = !f.layers.empty();
    if (few) BCHK(launch_mf_norm(nullptr, nullptr, d->x, nullptr, d->layers[0].rms_attn, m.rms_eps, H, mf_operand(f.layers[0].qkv, f.xh4, f.xh6), B, st));
    for (int l = 0; l < m.n_layers; ++l) {
        const jllm_b200_layer_desc& w = d->layers[l];
        void** L = d->lists + (size_t)l * 4 * B;
        if (few) {
            const MfPrep pr = { d->q, w.q_norm, w.k_norm, m.rms_eps, (int8_t* const*)L, (int8_t* const*)(L + B), (float* const*)(L + 2 * B), (float* const*)(L + 3 * B),
                                nullptr, nullptr, nullptr, nullptr, d->state, 0, 0, m.n_heads, m.n_kv_heads, m.rope_neox != 0 };
            const MfProduct& qkv = f.layers[l].qkv;
            BCHK(launch_mf_sums(qkv, mf_operand(qkv, f.xh4, f.xh6), f.part, B, st));
            BCHK(launch_mf_prep(qkv, f.part, pr, m.rope_theta, B, st));
        } else {
            BCHK(launch_rmsnorm(d->normed, d->x, nullptr, w.rms_attn, true, B, H, m.rms_eps, st));
            BCHK(launch_mmq(d->q, resolve_weight(w.wq), w.type_wq, d->normed, QD, B, H, nullptr, st, &d->mmq));
            BCHK(launch_mmq_ex(d->k, resolve_weight(w.wk), w.type_wk, d->normed, KVD, B, H, nullptr, true, st, &d->mmq));      // same activations as Q
            BCHK(launch_mmq_ex(d->v, resolve_weight(w.wv), w.type_wv, d->normed, KVD, B, H, nullptr, true, st, &d->mmq));
            BCHK(launch_qkv_prep_batched(d->q, d->k, d->v, w.q_norm, w.k_norm, m.rms_eps, (int8_t* const*)L, (int8_t* const*)(L + B),
                                         (float* const*)(L + 2 * B), (float* const*)(L + 3 * B), B, m.n_heads, m.n_kv_heads, m.head_dim,
                                         d->state, m.rope_theta, m.rope_neox != 0, st));
        }
        AttnCall c;
        c.out = d->att; c.q = d->q; c.k_list = (const void* const*)L; c.v_list = (const void* const*)(L + B);
        c.ks_list = (const float* const*)(L + 2 * B); c.vs_list = (const float* const*)(L + 3 * B); c.seq_lens = d->seq_lens;
        c.tma_maps = d->maps.empty() ? nullptr : d->maps.data() + (size_t)l * B * 2 * 128;
        c.batch = B; c.max_seq = m.max_context; c.n_heads = m.n_heads; c.n_kv = m.n_kv_heads; c.hd = m.head_dim; c.chd = m.head_dim;
        c.scale = scale; c.kv_int8 = 1;
        c.n_splits = 1;      // the step is one captured graph for every position: no slices (the streams of a step are short or many)
        BCHK(launch_attention(c, st));
        if (few) {
            const MfLayer& p = f.layers[l];
            BCHK(launch_mf_quantise(d->att, mf_operand(p.wo, f.xa, f.xa), QD, B, st));
            BCHK(launch_mf_sums(p.wo, mf_operand(p.wo, f.xa, f.xa), f.part, B, st));
            BCHK(launch_mf_norm(&p.wo, f.part, d->x, d->x2, w.rms_ffn, m.rms_eps, H, mf_operand(p.gate_up, f.xh4, f.xh6), B, st));
            BCHK(launch_mf_sums(p.gate_up, mf_operand(p.gate_up, f.xh4, f.xh6), f.part, B, st));
            BCHK(launch_mf_glu(p.gate_up, f.part, mf_operand(p.down, f.xi, f.xi), B, st));
            BCHK(launch_mf_sums(p.down, mf_operand(p.down, f.xi, f.xi), f.part, B, st));
            const bool more = l + 1 < m.n_layers;
            const MfOperand next = mf_operand(more ? f.layers[l + 1].qkv : f.out, f.xh4, f.xh6);
            BCHK(launch_mf_norm(&p.down, f.part, d->x2, d->x, more ? d->layers[l + 1].rms_attn : m.output_norm, m.rms_eps, H, next, B, st));
            continue;
        }
        BCHK(launch_mmq_ex(d->x2, resolve_weight(w.wo), w.type_wo, d->att, H, B, QD, d->x, false, st, &d->mmq));           // + residual
        BCHK(launch_rmsnorm(d->normed, d->x2, nullptr, w.rms_ffn, true, B, H, m.rms_eps, st));
        BCHK(launch_mmq_pair(d->gate, d->up, resolve_weight(w.w_gate), w.type_w_gate, resolve_weight(w.w_up), w.type_w_up, d->normed, I, I, B, H, st, &d->mmq));   // one launch where the tensor-core kernel serves both
        BCHK(launch_glu(d->sw, d->gate, d->up, B, I, false, st));
        BCHK(launch_mmq_ex(d->x, resolve_weight(w.w_down), w.type_w_down, d->sw, H, B, I, d->x2, false, st, &d->mmq));     // + residual
    }
    if (few) {
        BCHK(launch_mf_out(f.out, mf_operand(f.out, f.xh4, f.xh6), d->logits, f.part, B, st));
    } else {
        BCHK(launch_rmsnorm(d->normed, d->x, nullptr, m.output_norm, true, B, H, m.rms_eps, st));
        BCHK(launch_mmq(d->logits, resolve_weight(m.output), m.output_type, d->normed, V, B, H, nullptr, st, &d->mmq));
    }
    const ArArgs ar = { d->logits, V, B, d->tokens, d->state, d->out_tokens, d->out_cap, d->seq_lens, prompt, n_prompt, d->best, d->best_at, d->tickets };
    const DeviceCtx* cx = ctx();
    if (!cx) return JB_ERR_CUDA;
    const int slices = B >= 2 * AR_SLICES ? (B >= cx->sm_count ? 1 : 4) : AR_SLICES;      // one to two CTAs of 1024 threads per SM
    JB_CUDA(launch_k(argmax_rows_kernel, dim3(slices, B), dim3(1024), 0, st, pdl_enabled(), ar));
    count_launch();
    d->kernels_per_step = (int)(jllm_b200_launch_count() - l0);
    return JB_OK;
}

extern "C" {

jllm_b200_batch_decoder* jllm_b200_batch_decoder_create(const jllm_b200_model_desc* model, int n_streams) {
    if (!model || !model->layers || model->n_layers <= 0 || n_streams < 2 || n_streams > 1024) { set_error(JB_ERR_ARG, "batch decoder: bad model description or stream count"); return nullptr; }
    if (model->hidden_dim % QK_K || model->intermediate_dim % QK_K || (model->n_heads * model->head_dim) % QK_K) {
        set_error(JB_ERR_ARG, "batch decoder: hidden/intermediate/q dims must be multiples of 256"); return nullptr;
    }
    if (!ctx()) return nullptr;
    jllm_b200_batch_decoder* d = new (std::nothrow) jllm_b200_batch_decoder();
    if (!d) return nullptr;
    d->m = *model; d->B = n_streams;
    d->layers.assign(model->layers, model->layers + model->n_layers);
    d->m.layers = d->layers.data();
    const int B = n_streams;
    const size_t H = model->hidden_dim, QD = (size_t)model->n_heads * model->head_dim, KVD = (size_t)model->n_kv_heads * model->head_dim,
                 I = model->intermediate_dim, V = model->vocab_size;
    d->kv.resize(B);
    jllm::KVCachePool::Config c = { model->n_layers, model->n_kv_heads, model->head_dim, model->max_context, 0, 1 };
    for (int b = 0; b < B; ++b)
        if (!d->kv[b].init(c) || !d->kv[b].kv_scale_ptr(0, 0, false)) { set_error(JB_ERR_NOMEM, "batch decoder: KV pool %d", b); jllm_b200_batch_decoder_destroy(d); return nullptr; }
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    d->out_cap = model->max_context + 8; d->prompt_cap = model->max_context + 8;
    const size_t total = 4 * al(B * H * 2) + 2 * al(B * QD * 2) + 2 * al(B * KVD * 2) + 3 * al(B * I * 2) + al(B * V * 2) + al(64) + 2 * al((size_t)B * 4) + 2 * al((size_t)B * AR_SLICES * 4) + al((size_t)(1 + B) * 4) +
                         al((size_t)d->out_cap * B * 4) + al((size_t)d->prompt_cap * B * 4) + al((size_t)model->n_layers * 4 * B * sizeof(void*));
    // product scratch of every step: nothing of it may move once a step is captured
    const struct { size_t M, M2, K; } products[6] = { { QD, 0, H }, { KVD, 0, H }, { H, 0, QD }, { I, I, H }, { H, 0, I }, { V, 0, H } };
    size_t need = 0;
    bool wide = false;
    for (const auto& g : products) {
        const int M = (int)g.M, M2 = (int)g.M2, K = (int)g.K;
        for (int t : { T_Q4K, T_Q6K })
            for (size_t b : { mmq_tc_scratch_bytes(t, M, B, K), mmq_tc_scratch_bytes_pair(t, M, M2, B, K), mmq_stream_scratch_bytes(t, M, B, K), mmq_scratch_bytes(B, K) })
                if (b > need) need = b;
        wide = wide || mmq_wide_applies(M, M2, B, K);
    }
    if (B <= MF_MAX_TOKENS && d->few.plan(d->m, true)) { need = al(d->few.bytes(B)); wide = false; }
    if (cudaMalloc(&d->slab, total + need) != cudaSuccess) { cudaGetLastError(); d->slab = nullptr; set_error(JB_ERR_NOMEM, "batch decoder: %zu B of activations and product scratch", total + need); jllm_b200_batch_decoder_destroy(d); return nullptr; }
    if (d->few.layers.empty()) { d->mmq.act = (char*)d->slab + total; d->mmq.act_bytes = need; d->mmq.held = true; }
    else d->few.place((char*)d->slab + total, B);
    cudaMemset(d->slab, 0, total);
    char* p = (char*)d->slab;
    auto take = [&](size_t b) { char* r = p; p += al(b); return r; };
    d->x = (__half*)take(B * H * 2); d->x2 = (__half*)take(B * H * 2); d->normed = (__half*)take(B * H * 2); d->y = (__half*)take(B * H * 2);
    d->q = (__half*)take(B * QD * 2); d->att = (__half*)take(B * QD * 2);
    d->k = (__half*)take(B * KVD * 2); d->v = (__half*)take(B * KVD * 2);
    d->gate = (__half*)take(B * I * 2); d->up = (__half*)take(B * I * 2); d->sw = (__half*)take(B * I * 2);
    d->logits = (__half*)take(B * V * 2);
    d->state = (int*)take(64); d->tokens = (int*)take((size_t)B * 4); d->seq_lens = (int*)take((size_t)B * 4);
    d->out_tokens = (int*)take((size_t)d->out_cap * B * 4); d->prompt_dev = (int*)take((size_t)d->prompt_cap * B * 4);
    d->best = (float*)take((size_t)B * AR_SLICES * 4); d->best_at = (int*)take((size_t)B * AR_SLICES * 4); d->tickets = (unsigned int*)take((size_t)(1 + B) * 4);
    d->lists = (void**)take((size_t)model->n_layers * 4 * B * sizeof(void*));
    std::vector<void*> host((size_t)model->n_layers * 4 * B);
    for (int l = 0; l < model->n_layers; ++l)
        for (int b = 0; b < B; ++b) {
            host[((size_t)l * 4 + 0) * B + b] = d->kv[b].key_ptr(l, 0);
            host[((size_t)l * 4 + 1) * B + b] = d->kv[b].val_ptr(l, 0);
            host[((size_t)l * 4 + 2) * B + b] = d->kv[b].kv_scale_ptr(l, 0, false);
            host[((size_t)l * 4 + 3) * B + b] = d->kv[b].kv_scale_ptr(l, 0, true);
        }
    cudaMemcpy(d->lists, host.data(), host.size() * sizeof(void*), cudaMemcpyHostToDevice);
    if (model->head_dim == 128) {       // tensor maps of every (layer, stream) cache for the TMA attention path
        std::vector<unsigned char> maps((size_t)model->n_layers * B * 2 * 128);
        bool ok = true;
        for (int l = 0; l < model->n_layers && ok; ++l)
            for (int b = 0; b < B && ok; ++b)
                ok = attn_tma_encode(&maps[(((size_t)l * B + b) * 2 + 0) * 128], d->kv[b].key_ptr(l, 0), model->max_context, model->n_kv_heads) &&
                     attn_tma_encode(&maps[(((size_t)l * B + b) * 2 + 1) * 128], d->kv[b].val_ptr(l, 0), model->max_context, model->n_kv_heads);
        if (ok) d->maps.swap(maps);       // else: the general attention kernel serves the pointer lists
    }
    if (wide) d->mmq.wide_scratch(MMQ_WEIGHT_BYTES, false);
    splitk_buffer((size_t)B * model->n_heads * 64 * (model->head_dim + 4), true);
    return d;
}
void jllm_b200_batch_decoder_destroy(jllm_b200_batch_decoder* d) {
    if (!d) return;
    if (d->graph_exec) cudaGraphExecDestroy(d->graph_exec);
    if (d->slab) cudaFree(d->slab);
    if (d->mmq.wide) cudaFree(d->mmq.wide);
    for (auto& p : d->kv) p.destroy();
    delete d;
}
int jllm_b200_batch_decoder_generate(jllm_b200_batch_decoder* d, const int* host_prompts, int n_prompt, int n_new, int* host_out, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const int B = d->B;
    if (n_prompt <= 0 || n_new < 0 || !host_prompts) return set_error(JB_ERR_ARG, "batch decoder: n_prompt=%d n_new=%d", n_prompt, n_new);
    if (n_prompt + n_new > d->m.max_context || n_prompt > d->prompt_cap) return set_error(JB_ERR_LIMIT, "batch decoder: %d tokens exceed the context of %d", n_prompt + n_new, d->m.max_context);
    for (long long i = 0; i < (long long)B * n_prompt; ++i)
        if (host_prompts[i] < 0 || host_prompts[i] >= d->m.vocab_size) return set_error(JB_ERR_ARG, "batch decoder: prompt token %d outside the vocabulary", host_prompts[i]);
    JB_CUDA(cudaMemcpyAsync(d->prompt_dev, host_prompts, (size_t)B * n_prompt * sizeof(int), cudaMemcpyHostToDevice, st));
    JB_CUDA(cudaMemsetAsync(d->state, 0, 64, st));
    for (auto& p : d->kv) p.clear();
    const int total_steps = n_prompt + (n_new > 0 ? n_new - 1 : 0);
    d->host_pos = -1;
    JB_CUDA(launch_k(batch_begin_kernel, dim3(1), dim3(128), 0, st, pdl_enabled(), d->state, d->seq_lens, d->tokens, (const int*)d->prompt_dev, n_prompt, B));
    count_launch();
    for (int s = 0; s < total_steps; ++s) BCHK(bdec_enqueue_step(d, d->prompt_dev, n_prompt, st));
    d->host_pos = total_steps;              // every step advances the device-side position by one
    if (n_new > 0 && host_out)
        JB_CUDA(cudaMemcpyAsync(host_out, d->out_tokens + (size_t)(n_prompt - 1) * B, (size_t)n_new * B * sizeof(int), cudaMemcpyDeviceToHost, st));
    JB_CUDA(cudaStreamSynchronize(st));
    return jllm_b200_device_status(stream);
}
/* one more step from the device-side state (after generate): no host copy, no wait */
int jllm_b200_batch_decoder_step_device(jllm_b200_batch_decoder* d, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    // The position lives on the device; the host mirror keeps a step from writing K/V rows past the per-stream pools.
    if (d->host_pos < 0) return set_error(JB_ERR_STATE, "batch decoder: step_device before generate");
    if (d->host_pos >= d->m.max_context) return set_error(JB_ERR_LIMIT, "batch decoder: position %d is outside the context of %d", d->host_pos, d->m.max_context);
    ++d->host_pos;
    if (st == nullptr || st == cudaStreamLegacy) return bdec_enqueue_step(d, nullptr, 0, st);   // the default stream cannot be captured
    if (!d->graph_exec) {
        cudaGraph_t g = nullptr;
        JB_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        const int rc = bdec_enqueue_step(d, nullptr, 0, st);
        const cudaError_t e = cudaStreamEndCapture(st, &g);
        if (rc) { if (g) cudaGraphDestroy(g); return rc; }
        if (e != cudaSuccess) return cuda_error(e, "cudaStreamEndCapture");
        const cudaError_t ie = cudaGraphInstantiate(&d->graph_exec, g, 0);
        cudaGraphDestroy(g);
        if (ie != cudaSuccess) { d->graph_exec = nullptr; return cuda_error(ie, "cudaGraphInstantiate"); }
    }
    JB_CUDA(cudaGraphLaunch(d->graph_exec, st));
    count_launch(d->kernels_per_step);
    return JB_OK;
}
const void* jllm_b200_batch_decoder_logits(jllm_b200_batch_decoder* d) { return d->logits; }
int jllm_b200_batch_decoder_kernels_per_step(jllm_b200_batch_decoder* d) { return d->kernels_per_step; }

}  // extern "C"
