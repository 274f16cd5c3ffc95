// decoder.cu — the decoder session: sequencing of decode steps, prompt chunks and greedy generation over a model family's
// step (decoder.cuh), with the token and the position kept in device memory so that a single captured CUDA graph serves
// every step.  Stands where the reference's Engine::decode_step loop sits (src/engine/decode.cu:2101-2194).
#include "decoder.cuh"
#include <cfloat>
#include <cmath>
#include <vector>

namespace jb {

// greedy argmax over fp32 logits; also advances the device-side step state:
// state[0] = position, state[1] = current token, state[2] = number of tokens written to `out`.
// Several CTAs scan slices of the vocabulary; each leaves its best (value, index) in scratch, and the last one to
// finish (atomic ticket, no waiting) reduces them and advances the state.  scratch: [0] ticket, [32..32+G) values,
// [32+G..32+2G) indices, G = gridDim.x <= 64.
__global__ void __launch_bounds__(1024) argmax_advance_kernel(const float* logits, int n, int* state, int* out, int out_cap, unsigned int* scratch) {
    pdl_wait();
    __shared__ float sv[32]; __shared__ int si[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x;
    float best = -INFINITY; int bi = 0x7FFFFFFF;
    auto take = [&](float v, int i) { if (isfinite(v) && (v > best || (v == best && i < bi))) { best = v; bi = i; } };
    const int n4 = ((uintptr_t)logits & 15) == 0 ? n / 4 : 0;
    for (int i = blockIdx.x * blockDim.x + tid; i < n4; i += G * blockDim.x) {
        const float4 v = reinterpret_cast<const float4*>(logits)[i];
        take(v.x, 4 * i); take(v.y, 4 * i + 1); take(v.z, 4 * i + 2); take(v.w, 4 * i + 3);
    }
    for (int i = 4 * n4 + blockIdx.x * blockDim.x + tid; i < n; i += G * blockDim.x) take(logits[i], i);
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o); const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) { sv[warp] = best; si[warp] = bi; }
    __syncthreads();
    // the warps', then the CTAs' candidates by one warp (by one thread, a load after the other, this end took half of the kernel's 10.4 us)
    if (warp != 0) return;
    auto reduce = [&]() {
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o); const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
    };
    const bool have = lane < (int)(blockDim.x >> 5);
    best = have ? sv[lane] : -INFINITY; bi = have ? si[lane] : 0x7FFFFFFF;
    reduce();
    int last = 0;
    if (lane == 0) {
        reinterpret_cast<float*>(scratch)[32 + blockIdx.x] = best;
        reinterpret_cast<int*>(scratch)[32 + G + blockIdx.x] = bi;
        __threadfence();
        last = atomicAdd(scratch, 1u) == (unsigned)G - 1;
    }
    if (!__shfl_sync(0xFFFFFFFFu, last, 0)) return;
    __threadfence();
    best = -INFINITY; bi = 0x7FFFFFFF;
    for (int g = lane; g < G; g += 32) {
        const float v = __ldcg(reinterpret_cast<const float*>(scratch) + 32 + g); const int i = __ldcg(reinterpret_cast<const int*>(scratch) + 32 + G + g);
        if (i != 0x7FFFFFFF && (v > best || (v == best && i < bi))) { best = v; bi = i; }
    }
    reduce();
    if (lane != 0) return;
    scratch[0] = 0u;
    if (bi == 0x7FFFFFFF) bi = 0;
    const int k = state[2];
    if (out && k < out_cap) out[k] = bi;
    state[2] = k + 1;
    state[1] = bi;
    state[0] = state[0] + 1;
}

__global__ void set_state_kernel(int* state, int pos, int token) {
    pdl_wait();
    if (threadIdx.x == 0) { state[0] = pos; state[1] = token; }
}
// prompt feeding inside a graph: token for this step comes from a device list
__global__ void next_prompt_kernel(int* state, const int* prompt, int idx_base) {
    pdl_wait();
    if (threadIdx.x == 0) { const int p = state[0]; state[1] = prompt[p - idx_base]; }
}

int launch_argmax_advance(jllm_b200_decoder* d, cudaStream_t st) {
    const int ag = d->vocab >= 64 * 1024 ? 64 : (d->vocab + 1023) / 1024;
    JB_CUDA(launch_k(argmax_advance_kernel, dim3(ag), dim3(1024), 0, st, pdl_enabled(), (const float*)d->logits, d->vocab, d->state,
                     d->out_tokens, d->out_cap, (unsigned int*)(d->state + 32)));
    count_launch();
    return JB_OK;
}

}  // namespace jb

using namespace jb;

int jllm_b200_decoder::session_alloc() {
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    out_cap = prompt_cap = max_context + 8;
    const size_t total = al((size_t)vocab * 4) + al(1024) + 2 * al((size_t)out_cap * 4);
    if (cudaMalloc(&session_slab, total) != cudaSuccess) { cudaGetLastError(); session_slab = nullptr; return set_error(JB_ERR_NOMEM, "decoder: %zu B of session state", total); }
    cudaMemset(session_slab, 0, total);
    char* p = (char*)session_slab;
    auto take = [&](size_t b) { char* r = p; p += al(b); return r; };
    logits = (float*)take((size_t)vocab * 4);
    state = (int*)take(1024);
    out_tokens = (int*)take((size_t)out_cap * 4);
    prompt_dev = (int*)take((size_t)prompt_cap * 4);
    pf_tokens = prompt_dev;
    JB_CUDA(cudaStreamSynchronize(cudaStreamLegacy));      // this slab and the family's are zeroed before a stream that does not wait for the default one uses them
    return JB_OK;
}
void jllm_b200_decoder::session_free() {
    if (graph_exec) cudaGraphExecDestroy(graph_exec);
    if (own_stream) cudaStreamDestroy(own_stream);
    if (session_slab) cudaFree(session_slab);
    if (row_logits) cudaFree(row_logits);
    graph_exec = nullptr; own_stream = nullptr; session_slab = nullptr; row_logits = nullptr;
}

static int splits_for_ctx(const jllm_b200_decoder* d, int upto_pos) { return d->attn_splits(upto_pos + 1); }

// graph of one step; re-captured when the split count of the attention changes
static int dec_graph_for(jllm_b200_decoder* d, int n_splits, cudaStream_t st) {
    if (d->graph_exec && d->graph_splits == n_splits) return JB_OK;
    if (d->graph_exec) { cudaGraphExecDestroy(d->graph_exec); d->graph_exec = nullptr; }
    cudaGraph_t g = nullptr;
    JB_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    const int rc = d->enqueue_step(n_splits, st);
    const cudaError_t e = cudaStreamEndCapture(st, &g);
    if (rc) { if (g) cudaGraphDestroy(g); return rc; }
    if (e != cudaSuccess) return cuda_error(e, "cudaStreamEndCapture");
    const cudaError_t ie = cudaGraphInstantiate(&d->graph_exec, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) { d->graph_exec = nullptr; return cuda_error(ie, "cudaGraphInstantiate"); }
    d->graph_splits = n_splits;
    return JB_OK;
}
// one step from the device-side state: the captured graph of its slice count, or the launches themselves
static int run_step(jllm_b200_decoder* d, int pos, cudaStream_t st) {
    const int ns = splits_for_ctx(d, pos);
    if (!d->use_graph) return d->enqueue_step(ns, st);
    DCHK(dec_graph_for(d, ns, st));
    JB_CUDA(cudaGraphLaunch(d->graph_exec, st));
    count_launch(d->kernels_per_step);
    return JB_OK;
}
// the default stream cannot be captured: graph sessions run on their own, ordered after what the caller queued
static int usable_stream(jllm_b200_decoder* d, cudaStream_t& st) {
    if (!d->use_graph || (st != nullptr && st != cudaStreamLegacy)) return JB_OK;
    if (!d->own_stream) JB_CUDA(cudaStreamCreateWithFlags(&d->own_stream, cudaStreamNonBlocking));
    JB_CUDA(cudaStreamSynchronize(st));
    st = d->own_stream;
    return JB_OK;
}
static int check_tokens(const jllm_b200_decoder* d, const int* tokens, int n, int start) {
    if (start < 0 || start + n > d->max_context) return set_error(JB_ERR_LIMIT, "decoder: positions %d..%d exceed the context of %d", start, start + n - 1, d->max_context);
    for (int i = 0; i < n; ++i)
        if (tokens[i] < 0 || tokens[i] >= d->vocab_full) return set_error(JB_ERR_ARG, "decoder: token %d outside the vocabulary", tokens[i]);
    return JB_OK;
}
// tokens at positions start .. start + n - 1 are about to run: a recurrent state takes them only where it stands, or from 0
static int advance_state(jllm_b200_decoder* d, int start, int n) {
    if (d->keeps_state() && start != 0 && start != d->held) return set_error(JB_ERR_STATE, "decoder: position %d, but the recurrent state stands at %d", start, d->held);
    d->held = start + n;
    return JB_OK;
}
// n >= 2 tokens through the chunk path; logits [n_want][vocab] of the (rising) wanted positions
static int feed_chunks(jllm_b200_decoder* d, const int* tokens, int n, int start, const int* want, int n_want, float* out, cudaStream_t st) {
    DCHK(check_tokens(d, tokens, n, start));
    DCHK(advance_state(d, start, n));
    const int chunk = d->pf_chunk < 2 ? 2 : d->pf_chunk;
    DCHK(d->reserve_chunk(n < chunk ? n : chunk, st));
    std::vector<int> rows;
    int done = 0, w = 0;
    while (done < n) {
        int c = n - done < chunk ? n - done : chunk;
        if (n - done - c == 1 && c > 2) --c;                // avoid a chunk of one token: the batched products of the K-quant family need two
        JB_CUDA(cudaMemcpyAsync(d->pf_tokens, tokens + done, (size_t)c * sizeof(int), cudaMemcpyHostToDevice, st));
        DCHK(d->enqueue_chunk(d->pf_tokens, c, start + done, st));
        rows.clear();
        while (w < n_want && want[w] < done + c) rows.push_back(want[w++] - done);
        if (!rows.empty()) DCHK(d->enqueue_rows(rows.data(), (int)rows.size(), out + (size_t)(w - (int)rows.size()) * d->vocab, st));
        done += c;
    }
    return JB_OK;
}

extern "C" {

void jllm_b200_decoder_destroy(jllm_b200_decoder* d) {
    if (!d) return;
    d->session_free();
    delete d;
}
int jllm_b200_decoder_reset(jllm_b200_decoder* d) {
    JB_CUDA(cudaMemset(d->state, 0, 64));
    JB_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    d->held = 0;
    d->clear_cache();
    return JB_OK;
}
int jllm_b200_decoder_step(jllm_b200_decoder* d, int token, int position, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (position < 0 || position >= d->max_context) return set_error(JB_ERR_ARG, "decoder: position %d outside the context of %d", position, d->max_context);
    if (token < 0 || token >= d->vocab_full) return set_error(JB_ERR_ARG, "decoder: token %d outside the vocabulary", token);
    DCHK(advance_state(d, position, 1));
    JB_CUDA(launch_k(set_state_kernel, dim3(1), dim3(32), 0, st, false, d->state, position, token));
    count_launch();
    return d->enqueue_step(splits_for_ctx(d, position), st);
}

int jllm_b200_decoder_feed(jllm_b200_decoder* d, const int* host_tokens, int n_tokens, int start_pos, const int* want, int n_want,
                           float* host_logits, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (!host_tokens || n_tokens < 1 || n_want < 0 || (n_want > 0 && (!want || !host_logits))) return set_error(JB_ERR_ARG, "decoder: feed of %d tokens, %d positions wanted", n_tokens, n_want);
    for (int i = 0; i < n_want; ++i)
        if (want[i] < 0 || want[i] >= n_tokens || (i && want[i] <= want[i - 1])) return set_error(JB_ERR_ARG, "decoder: wanted positions must rise within the %d tokens fed", n_tokens);
    DCHK(usable_stream(d, st));
    stream = (void*)st;
    const size_t V = d->vocab;
    if (n_tokens == 1 || !d->has_chunks()) {
        int w = 0;
        for (int i = 0; i < n_tokens; ++i) {
            const int pos_tok[2] = { start_pos + i, host_tokens[i] };
            DCHK(check_tokens(d, &host_tokens[i], 1, start_pos + i));
            DCHK(advance_state(d, start_pos + i, 1));
            JB_CUDA(launch_k(set_state_kernel, dim3(1), dim3(32), 0, st, false, d->state, pos_tok[0], pos_tok[1]));
            count_launch();
            DCHK(run_step(d, pos_tok[0], st));
            if (w < n_want && want[w] == i) {
                JB_CUDA(cudaMemcpyAsync(host_logits + (size_t)w * V, d->logits, V * sizeof(float), cudaMemcpyDeviceToHost, st));
                ++w;
            }
        }
    } else {
        if ((size_t)n_want * V > d->row_logits_cap) {
            if (d->row_logits) cudaFree(d->row_logits);
            d->row_logits = nullptr; d->row_logits_cap = 0;
            if (cudaMalloc(&d->row_logits, (size_t)n_want * V * sizeof(float)) != cudaSuccess) { cudaGetLastError(); return set_error(JB_ERR_NOMEM, "decoder: logits of %d positions", n_want); }
            d->row_logits_cap = (size_t)n_want * V;
        }
        DCHK(feed_chunks(d, host_tokens, n_tokens, start_pos, want, n_want, d->row_logits, st));
        if (n_want) JB_CUDA(cudaMemcpyAsync(host_logits, d->row_logits, (size_t)n_want * V * sizeof(float), cudaMemcpyDeviceToHost, st));
    }
    d->host_pos = start_pos + n_tokens;
    JB_CUDA(cudaStreamSynchronize(st));
    return jllm_b200_device_status(stream);
}
int jllm_b200_decoder_prefill(jllm_b200_decoder* d, const int* host_tokens, int n_tokens, int start_pos, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (!d->has_chunks()) return set_error(JB_ERR_STATE, "decoder: batched prefill is not available in a tensor-parallel session");
    if (!host_tokens || n_tokens < 2) return set_error(JB_ERR_ARG, "decoder: batched prefill needs at least two tokens (got %d)", n_tokens);
    // logits of the last prompt token only (src/engine/decode.cu:2019-2050), greedy token on the device; the step state
    // moves to the position after the prompt, so jllm_b200_decoder_step_device continues from there
    const int last = n_tokens - 1;
    DCHK(feed_chunks(d, host_tokens, n_tokens, start_pos, &last, 1, d->logits, st));
    JB_CUDA(launch_k(set_state_kernel, dim3(1), dim3(32), 0, st, false, d->state, start_pos + last, host_tokens[last]));
    count_launch();
    DCHK(launch_argmax_advance(d, st));
    d->host_pos = start_pos + n_tokens;
    return JB_OK;
}
int jllm_b200_decoder_set_prefill_chunk(jllm_b200_decoder* d, int tokens) {
    if (tokens < 2) return set_error(JB_ERR_ARG, "decoder: prefill chunk of %d tokens", tokens);
    d->pf_chunk = tokens;
    return JB_OK;
}

int jllm_b200_decoder_generate(jllm_b200_decoder* d, const int* host_prompt, int n_prompt, int n_new, int* host_out, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    DCHK(usable_stream(d, st));
    stream = (void*)st;
    if (n_prompt <= 0 || n_new < 0 || !host_prompt) return set_error(JB_ERR_ARG, "decoder: n_prompt=%d n_new=%d", n_prompt, n_new);
    if (n_prompt + n_new > d->max_context) return set_error(JB_ERR_LIMIT, "decoder: %d tokens exceed the context of %d", n_prompt + n_new, d->max_context);
    for (int i = 0; i < n_prompt; ++i)
        if (host_prompt[i] < 0 || host_prompt[i] >= d->vocab_full) return set_error(JB_ERR_ARG, "decoder: prompt token %d outside the vocabulary", host_prompt[i]);
    if (d->batched_prefill && d->has_chunks() && n_prompt >= 2) {
        // the prompt in one batched pass (the first generated token comes out of it), then n_new - 1 self-feeding decode steps
        JB_CUDA(cudaMemsetAsync(d->state, 0, 64, st));
        d->clear_cache();
        DCHK(jllm_b200_decoder_prefill(d, host_prompt, n_prompt, 0, stream));
        for (int s = 1; s < n_new; ++s) DCHK(jllm_b200_decoder_step_device(d, stream));
        if (n_new > 0 && host_out) JB_CUDA(cudaMemcpyAsync(host_out, d->out_tokens, (size_t)n_new * sizeof(int), cudaMemcpyDeviceToHost, st));
        JB_CUDA(cudaStreamSynchronize(st));
        return jllm_b200_device_status(stream);
    }
    JB_CUDA(cudaMemcpyAsync(d->prompt_dev, host_prompt, (size_t)n_prompt * sizeof(int), cudaMemcpyHostToDevice, st));
    JB_CUDA(cudaMemsetAsync(d->state, 0, 64, st));
    d->clear_cache();
    // steps 0 .. n_prompt-1 consume prompt tokens; every step's argmax is recorded, the first n_prompt-1 are discarded below
    const int total_steps = n_prompt + (n_new > 0 ? n_new - 1 : 0);
    for (int s = 0; s < total_steps; ++s) {
        DCHK(advance_state(d, s, 1));
        if (s < n_prompt) {
            JB_CUDA(launch_k(next_prompt_kernel, dim3(1), dim3(32), 0, st, false, d->state, (const int*)d->prompt_dev, 0));
            count_launch();
        }
        DCHK(run_step(d, s, st));
    }
    if (n_new > 0 && host_out)
        JB_CUDA(cudaMemcpyAsync(host_out, d->out_tokens + (n_prompt - 1), (size_t)n_new * sizeof(int), cudaMemcpyDeviceToHost, st));
    JB_CUDA(cudaStreamSynchronize(st));
    return jllm_b200_device_status(stream);
}
// One user-facing step: token and position come from (pinned) host memory, the sampled token goes back to
// host memory, and the call returns when it is there — the per-token host/device boundary of the reference
// engine (src/engine/decode.cu:2170-2175), minus the 600 KB logits copy (sampling runs on the device).
int jllm_b200_decoder_step_sync(jllm_b200_decoder* d, const int* host_pos_token, int* host_next, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (!host_pos_token || !host_next) return set_error(JB_ERR_PTR, "decoder: null host pointer");
    if (d->use_graph && (st == nullptr || st == cudaStreamLegacy)) {
        if (!d->own_stream) JB_CUDA(cudaStreamCreateWithFlags(&d->own_stream, cudaStreamNonBlocking));
        st = d->own_stream;
    }
    const int pos = host_pos_token[0], tok = host_pos_token[1];
    if (pos < 0 || pos >= d->max_context) return set_error(JB_ERR_ARG, "decoder: position %d outside the context of %d", pos, d->max_context);
    if (tok < 0 || tok >= d->vocab_full) return set_error(JB_ERR_ARG, "decoder: token %d outside the vocabulary", tok);
    DCHK(advance_state(d, pos, 1));
    JB_CUDA(cudaMemcpyAsync(d->state, host_pos_token, 2 * sizeof(int), cudaMemcpyHostToDevice, st));
    DCHK(run_step(d, pos, st));
    JB_CUDA(cudaMemcpyAsync(host_next, d->state + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    JB_CUDA(cudaStreamSynchronize(st));
    d->host_pos = pos + 1;
    return JB_OK;
}
// Enqueues the next step entirely from device-side state (position and token left by the previous step's argmax);
// nothing crosses the host boundary and the call does not wait.
int jllm_b200_decoder_step_device(jllm_b200_decoder* d, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (d->use_graph && (st == nullptr || st == cudaStreamLegacy)) return set_error(JB_ERR_ARG, "decoder: graph replay needs a non-default stream");
    if (d->host_pos >= d->max_context) return set_error(JB_ERR_LIMIT, "decoder: context of %d exhausted", d->max_context);
    DCHK(advance_state(d, d->host_pos, 1));
    DCHK(run_step(d, d->host_pos, st));
    d->host_pos += 1;
    return JB_OK;
}
const float* jllm_b200_decoder_logits(jllm_b200_decoder* d) { return d->logits; }
int jllm_b200_decoder_last_token(jllm_b200_decoder* d, void* stream) {
    int h[3] = { 0, 0, 0 };
    if (cudaMemcpyAsync(h, d->state, sizeof h, cudaMemcpyDeviceToHost, (cudaStream_t)stream) != cudaSuccess) return -1;
    cudaStreamSynchronize((cudaStream_t)stream);
    return h[1];
}
int jllm_b200_decoder_kernels_per_step(jllm_b200_decoder* d) { return d->kernels_per_step; }
int jllm_b200_decoder_recorded_tokens(jllm_b200_decoder* d, int first, int n, int* host_out, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    int h[3] = { 0, 0, 0 };
    if (cudaMemcpyAsync(h, d->state, sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    const int have = h[2] < d->out_cap ? h[2] : d->out_cap;
    if (host_out && n > 0 && first >= 0 && first < have) {
        const int m = first + n <= have ? n : have - first;
        if (cudaMemcpyAsync(host_out, d->out_tokens + first, (size_t)m * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return -1;
        cudaStreamSynchronize(st);
    }
    return h[2];
}
const void* jllm_b200_decoder_buffer(jllm_b200_decoder* d, int which) { return d->buffer(which); }

}  // extern "C"
