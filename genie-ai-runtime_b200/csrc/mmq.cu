// mmq.cu — batched K-quant GEMM (prefill), first CUDA-core version.
//
// Arithmetic mirrors the reference's default prefill path: activations are quantised
// per 32 without clamping; Q4_K keeps (half d, half sum-of-x) per group and folds the
// weight sub-scales as half products, Q6_K keeps fp32 d (mmq_q4k_llama.cu:383-404,
// :159-163, :321-322; mmq_q6k_llama.cu:424-438, :208, :361).
#include "mmq.cuh"
#include "dense.cuh"
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace jb {

struct ActQ { int8_t* q; float* d; float* s; };   // [N][K] codes, [N][K/32] scale, [N][K/32] sum

size_t mmq_scratch_bytes(int N, int K) { return (size_t)N * K + 2 * (size_t)N * (K / 32) * sizeof(float) + 256; }

// While it lives, this thread's allocations, waits and event queries neither fail under its own capture nor invalidate the capture of
// another thread (which they do in the default mode).
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
cudaError_t mmq_alloc(void** p, size_t bytes) {
    const RelaxedCapture relaxed;
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) { cudaGetLastError(); *p = nullptr; }
    return e;
}
void* MmqWork::scratch(size_t bytes, bool capturing) {
    if (bytes > act_bytes) {
        if (capturing && bytes > capture_limit) return nullptr;
        few = many = MmqOperand();               // the operands that lay there are gone, also when the new buffer gets the old address
        const bool keep = held || capturing;     // the old buffer stays: all of them together take less than the newest
        size_t want = keep && bytes < 2 * act_bytes ? 2 * act_bytes : bytes;
        if (act && !keep) { const RelaxedCapture relaxed; cudaFree(act); }
        act = nullptr; act_bytes = 0; held = false;
        if (mmq_alloc(&act, want) != cudaSuccess && mmq_alloc(&act, want = bytes) != cudaSuccess) return nullptr;
        act_bytes = want;
    }
    held = held || capturing;
    return act;
}
// An object whose request was refused does not ask for as much again: it stays with the fused kernel, whose results differ in their last bits.  A captured
// call asks too, so that it takes the way an uncaptured one takes; what it was given stays.
void* MmqWork::wide_scratch(size_t weights, bool capturing) {
    const size_t need = weights + gemm_pair_part_floats() * sizeof(float);
    if (need <= wide_bytes) return wide;
    if (need >= wide_refused || (capturing && (!capture_limit || wide))) return nullptr;
    void* p = nullptr;
    if (mmq_alloc(&p, need) != cudaSuccess) { wide_refused = need; return nullptr; }
    if (wide) { const RelaxedCapture relaxed; cudaFree(wide); }
    wide = p; wide_bytes = need;
    return wide;
}
// one warp per 32-element group of one token
__global__ void mmq_quantize_kernel(const __half* x, ActQ a, int N, int K, int ds4) {
    pdl_wait();
    const long long g = (long long)blockIdx.x * blockDim.y + threadIdx.y;
    const int lane = threadIdx.x, G = K / 32;
    if (g >= (long long)N * G) return;
    const float v = __half2float(x[g * 32 + lane]);
    const float amax = warp_max(fabsf(v));
    float sum = v;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    const float d = __fdiv_rn(amax, 127.0f), dinv = d > 0.f ? __fdiv_rn(1.0f, d) : 0.f;
    a.q[g * 32 + lane] = (int8_t)__float2int_rn(__fmul_rn(v, dinv));
    if (lane == 0) {
        a.d[g] = ds4 ? __half2float(__float2half_rn(d)) : d;
        a.s[g] = ds4 ? __half2float(__float2half_rn(sum)) : 0.f;
    }
}

// one warp per (row, token); lanes stride over 32-groups (Q4_K) / 16-groups (Q6_K)
__global__ void mmq_simple_kernel(__half* y, const uint8_t* W, int type, ActQ a, int M, int N, int K, int32_t* dbg) {
    pdl_wait();
    const int row = blockIdx.x * blockDim.y + threadIdx.y, tok = blockIdx.y, lane = threadIdx.x;
    if (row >= M) return;
    const int nb = K / QK_K;
    const int8_t* q8 = a.q + (size_t)tok * K;
    const float* d8 = a.d + (size_t)tok * (K / 32);
    const float* s8 = a.s + (size_t)tok * (K / 32);
    float acc = 0.f;
    if (type == T_Q4K) {
        for (int g = lane; g < nb * 8; g += 32) {
            const uint8_t* blk = W + ((size_t)row * nb + (g >> 3)) * Q4K_BYTES;
            const int j = g & 7;
            const uint32_t* s = reinterpret_cast<const uint32_t*>(blk + 4);
            int sc, mn; scale_min_k4(j, s[0], s[1], s[2], sc, mn);
            const uint32_t* qs = reinterpret_cast<const uint32_t*>(blk + 16 + 32 * (j >> 1));
            const int* xq = reinterpret_cast<const int*>(q8 + g * 32);
            int dot = 0;
            #pragma unroll
            for (int w = 0; w < 8; ++w) dot = dp4a_us((j & 1) ? (qs[w] >> 4) & 0x0F0F0F0Fu : qs[w] & 0x0F0F0F0Fu, xq[w], dot);
            if (dbg) dbg[((size_t)tok * M + row) * (nb * 8) + g] = dot;
            const __half dh = __ushort_as_half(*reinterpret_cast<const unsigned short*>(blk));
            const __half mh = __hneg(__ushort_as_half(*reinterpret_cast<const unsigned short*>(blk + 2)));
            const float ax = __half2float(__hmul(dh, __float2half_rn((float)sc)));
            const float ay = __half2float(__hmul(mh, __float2half_rn((float)mn)));
            acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(ax, d8[g]), (float)dot));
            acc = __fadd_rn(acc, __fmul_rn(ay, s8[g]));
        }
    } else {
        for (int g = lane; g < nb * 16; g += 32) {
            const uint8_t* blk = W + ((size_t)row * nb + (g >> 4)) * Q6K_BYTES;
            const int e0 = (g & 15) * 16;
            int dot = 0;
            for (int i = 0; i < 16; ++i) {
                const int e = e0 + i, n = e >> 7, r = e & 127, quarter = r >> 5, l = r & 31;
                int lo = (quarter & 1) ? blk[64 * n + 32 + l] : blk[64 * n + l];
                lo = (quarter & 2) ? (lo >> 4) : (lo & 0xF);
                const int qv = (lo | (((blk[128 + 32 * n + l] >> (2 * quarter)) & 3) << 4)) - 32;
                dot += qv * (int)q8[(g >> 4) * 256 + e];
            }
            if (dbg) dbg[((size_t)tok * M + row) * (nb * 16) + g] = dot;
            const float d = h2f_bits(blk[208] | (blk[209] << 8));
            acc += __fmul_rn(__fmul_rn(__fmul_rn((float)dot, (float)(int8_t)blk[192 + (g & 15)]), d8[g >> 1]), d);
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) y[(size_t)tok * M + row] = __float2half_rn(acc);
}

static bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) { cudaGetLastError(); return false; }
    return cs != cudaStreamCaptureStatusNone;
}

int launch_add_half(__half* out, const __half* a, const __half* b, long long n, cudaStream_t st);      // elementwise.cu

static int launch_mmq_impl(__half* y, const void* W, int type, const __half* x, int M, int N, int K, int32_t* dbg, const __half* residual,
                           bool same_x, cudaStream_t st, MmqWork* w, bool cap);

// The library's scratch: an object per stream, so that calls on different streams do not meet.  A call holds its object while it enqueues
// its launches (quantiser, product, sum; a session those of a whole chunk), so that threads that share a stream do not mix theirs; the lock on all of them is
// held for the look-up alone.  A stream that has none takes one
// whose last work is known to be over (sessions record an event at the end of a prompt: mmq_mark), else a new one; when there are
// MMQ_STREAMS, the one that was not used for the longest time, behind its event (every call records one from half of them on).  Nothing
// here waits on the host: a wait for the device would invalidate any capture in the process.
// Captured calls have objects apart from these, which their graphs keep: one per stream handle (a stream's id cannot be asked for under
// capture); a handle beyond MMQ_GRAPHS shares the one that was captured into least recently.
constexpr int MMQ_STREAMS = 32, MMQ_GRAPHS = 32;
struct MmqEntry {
    unsigned long long id = 0, used = 0;
    cudaEvent_t done = nullptr; bool marked = false;      // all work so far lies before the event: no one is using it (users) since
    int users = 0;                                        // leases that hold it or wait for it
    std::recursive_mutex mu;                              // a session's products take theirs inside the chunk's
    MmqWork work;
};
struct MmqPool {
    typedef MmqEntry Entry;
    std::mutex mu;                               // everything but the entries' work
    Entry streams[MMQ_STREAMS], graphs[MMQ_GRAPHS];
    int n_streams = 0, n_graphs = 0;
    unsigned long long clock = 0;
    size_t asked = 0;                            // most scratch that a call has asked for outside of captures

    static Entry* oldest(Entry* e, int n, bool marked) {
        Entry* o = nullptr;
        for (int i = 0; i < n; ++i) if ((e[i].marked || !marked) && (!o || e[i].used < o->used)) o = &e[i];
        return o;
    }
    static bool id_of(cudaStream_t st, unsigned long long& id) {
        id = 0;                                  // the default stream, which has two handles
        if (!st || st == cudaStreamLegacy || cudaStreamGetId(st, &id) == cudaSuccess) return true;
        cudaGetLastError();
        return false;
    }
    Entry* find(unsigned long long id) {
        for (int i = 0; i < n_streams; ++i) if (streams[i].id == id) return &streams[i];
        return nullptr;
    }
    Entry* of_graph(cudaStream_t st) {
        const unsigned long long id = (unsigned long long)(uintptr_t)st;
        Entry* e = nullptr;
        for (int i = 0; i < n_graphs; ++i) if (graphs[i].id == id) e = &graphs[i];
        if (!e) e = n_graphs < MMQ_GRAPHS ? &graphs[n_graphs++] : oldest(graphs, n_graphs, false);
        e->id = id; e->used = ++clock;
        return e;
    }
    Entry* of_stream(cudaStream_t st) {
        const RelaxedCapture relaxed;
        unsigned long long id;
        if (!id_of(st, id)) return nullptr;
        Entry* e = find(id);
        if (!e) {
            for (int i = 0; i < n_streams && !e; ++i) if (streams[i].marked && cudaEventQuery(streams[i].done) == cudaSuccess) e = &streams[i];
            cudaGetLastError();                  // "not ready" is an answer
            if (!e && n_streams < MMQ_STREAMS) e = &streams[n_streams++];
            if (!e) {
                e = oldest(streams, n_streams, true);
                if (!e || cudaStreamWaitEvent(st, e->done, 0) != cudaSuccess) { cudaGetLastError(); return nullptr; }
            }
            e->work.few = e->work.many = MmqOperand();
        }
        e->id = id; e->used = ++clock; e->marked = false;
        return e;
    }
    void mark(cudaStream_t st) {
        const RelaxedCapture relaxed;
        unsigned long long id;
        Entry* e = id_of(st, id) ? find(id) : nullptr;
        if (!e || e->users || (!e->done && cudaEventCreateWithFlags(&e->done, cudaEventDisableTiming) != cudaSuccess)) { cudaGetLastError(); return; }
        e->marked = cudaEventRecord(e->done, st) == cudaSuccess;
        if (!e->marked) cudaGetLastError();
    }
};
static MmqPool g_mmq_pool[16];                   // per device
MmqLease::MmqLease(MmqWork* own, cudaStream_t stream) : w(own), st(stream), cap(capturing(stream)) {
    DeviceCtx* c = own ? nullptr : ctx();
    if (!c) return;
    pool = &g_mmq_pool[c->device];
    size_t asked;
    {
        std::lock_guard<std::mutex> lock(pool->mu);
        e = cap ? pool->of_graph(st) : pool->of_stream(st);
        if (!e) return;
        ++e->users;
        asked = pool->asked;
    }
    e->mu.lock();
    w = &e->work;
    if (cap) w->capture_limit = asked;
}
MmqLease::~MmqLease() {
    if (!e) return;
    const size_t bytes = w->act_bytes;
    e->mu.unlock();
    std::lock_guard<std::mutex> lock(pool->mu);
    --e->users;
    if (cap) return;
    if (bytes > pool->asked) pool->asked = bytes;
    if (pool->n_streams > MMQ_STREAMS / 2) pool->mark(st);
}

void mmq_mark(cudaStream_t st) {
    DeviceCtx* c = ctx();
    if (!c || capturing(st)) return;
    std::lock_guard<std::mutex> lock(g_mmq_pool[c->device].mu);
    g_mmq_pool[c->device].mark(st);
}

int launch_mmq(__half* y, const void* W, int type, const __half* x, int M, int N, int K, int32_t* dbg, cudaStream_t st, MmqWork* own) {
    const MmqLease l(own, st);
    return launch_mmq_impl(y, W, type, x, M, N, K, dbg, nullptr, false, st, l.w, l.cap);
}
int launch_mmq_ex(__half* y, const void* W, int type, const __half* x, int M, int N, int K, const __half* residual, bool same_x, cudaStream_t st, MmqWork* own) {
    const MmqLease l(own, st);
    return launch_mmq_impl(y, W, type, x, M, N, K, nullptr, residual, same_x, st, l.w, l.cap);
}

// Two products over the same activations (gate and up): one launch of the tensor-core kernel when both matrices are of one
// type and that kernel is the one each would get on its own; else one product after the other, the second reusing the
// quantised operand of the first.
int launch_mmq_pair(__half* y1, __half* y2, const void* W1, int type1, const void* W2, int type2, const __half* x, int M1, int M2, int N, int K,
                    cudaStream_t st, MmqWork* own) {
    const MmqLease l(own, st);
    MmqWork* w = l.w;
    static const bool tc_off = [] { const char* e = getenv("JLLM_B200_MMQ"); return e && !strcmp(e, "cuda"); }();
    static const bool pair_off = [] { const char* e = getenv("JLLM_B200_MMQ_PAIR"); return e && e[0] == '0'; }();
    const bool ok = !tc_off && !pair_off && type1 == type2 && M1 > 0 && M2 > 0 && N > 0 && K > 0 && K % QK_K == 0 && y1 && y2 && W1 && W2 && x &&
                    (type1 == T_Q4K || type1 == T_Q6K) && !mmq_stream_applies(W1, type1, M1, N, K) && !mmq_stream_applies(W2, type2, M2, N, K) &&
                    mmq_tc_applies(W1, type1, M1, N, K) && mmq_tc_applies(W2, type2, M2, N, K);
    if (!ok) {
        const int rc = launch_mmq_impl(y1, W1, type1, x, M1, N, K, nullptr, nullptr, false, st, w, l.cap);
        return rc ? rc : launch_mmq_impl(y2, W2, type2, x, M2, N, K, nullptr, nullptr, true, st, w, l.cap);
    }
    const size_t need = mmq_tc_scratch_bytes_pair(type1, M1, M2, N, K);
    __half* xq = w ? (__half*)w->scratch(need, l.cap) : nullptr;
    if (!xq) return set_error(JB_ERR_NOMEM, "batched gemm: %zu B of activation scratch unavailable", need);
    return launch_mmq_tc_pair(y1, y2, W1, W2, type1, x, xq, M1, M2, N, K, false, st, *w, mmq_wide_applies(M1, M2, N, K) ? w->wide_scratch(MMQ_WEIGHT_BYTES, l.cap) : nullptr);
}

int launch_mmq_ready(__half* y1, __half* y2, const void* W1, const void* W2, int type, const __half* xq, int M1, int M2, int N, int K, cudaStream_t st, MmqWork* own) {
    const MmqLease l(own, st);
    if (!mmq_tc_applies(W1, type, M1, N, K) || (W2 && !mmq_tc_applies(W2, type, M2, N, K))) return set_error(JB_ERR_ARG, "batched gemm: %d x %d over %d tokens is not for the tensor-core path", M1, K, N);
    const size_t need = mmq_tc_scratch_bytes_pair(type, M1, M2, N, K);
    __half* scratch = l.w ? (__half*)l.w->scratch(need, l.cap) : nullptr;
    if (!scratch) return set_error(JB_ERR_NOMEM, "batched gemm: %zu B of scratch unavailable", need);
    l.w->few = l.w->many = MmqOperand();         // sums of K ranges may lie where another call left its operand
    return launch_mmq_tc_pair(y1, y2, W1, W2, type, nullptr, scratch, M1, M2, N, K, false, st, *l.w, mmq_wide_applies(M1, M2, N, K) ? l.w->wide_scratch(MMQ_WEIGHT_BYTES, l.cap) : nullptr, xq);
}

static int launch_mmq_impl(__half* y, const void* W, int type, const __half* x, int M, int N, int K, int32_t* dbg, const __half* residual,
                           bool same_x, cudaStream_t st, MmqWork* w, bool cap) {
    if (M <= 0 || N <= 0) return JB_OK;
    if (K <= 0 || K % QK_K) return set_error(JB_ERR_ARG, "batched gemm: K=%d is not a positive multiple of 256", K);
    if (type != T_Q4K && type != T_Q6K) return set_error(JB_ERR_TYPE, "batched gemm: ggml type %d", type);
    if (!y || !W || !x) return set_error(JB_ERR_PTR, "batched gemm: null pointer");
    if (type == T_Q4K && ((uintptr_t)W & 3)) return set_error(JB_ERR_PTR, "batched gemm: Q4_K weights must be 4-byte aligned");
    // JLLM_B200_MMQ=cuda keeps the CUDA-core kernel (the one that can also export the integer accumulators)
    static const bool tc_off = [] { const char* e = getenv("JLLM_B200_MMQ"); return e && !strcmp(e, "cuda"); }();
    if (!dbg && !tc_off && mmq_stream_applies(W, type, M, N, K)) {
        const size_t need_s = mmq_stream_scratch_bytes(type, M, N, K);
        void* sc = w ? w->scratch(need_s, cap) : nullptr;
        if (!sc) return set_error(JB_ERR_NOMEM, "batched gemm: %zu B of activation scratch unavailable", need_s);
        return launch_mmq_stream(y, W, type, x, sc, M, N, K, residual, same_x, st, *w);
    }
    if (residual) {          // the other kernels have no fused exit: product, then the add (in place)
        const int rc = launch_mmq_impl(y, W, type, x, M, N, K, dbg, nullptr, false, st, w, cap);
        return rc ? rc : launch_add_half(y, residual, y, (long long)N * M, st);
    }
    if (!dbg && !tc_off && mmq_tc_applies(W, type, M, N, K)) {
        const size_t need_tc = mmq_tc_scratch_bytes(type, M, N, K);
        __half* xq = w ? (__half*)w->scratch(need_tc, cap) : nullptr;
        if (!xq) return set_error(JB_ERR_NOMEM, "batched gemm: %zu B of activation scratch unavailable", need_tc);
        return launch_mmq_tc_pair(y, nullptr, W, nullptr, type, x, xq, M, 0, N, K, same_x, st, *w, mmq_wide_applies(M, 0, N, K) ? w->wide_scratch(MMQ_WEIGHT_BYTES, cap) : nullptr);
    }
    const size_t need = mmq_scratch_bytes(N, K);
    uint8_t* base = w ? (uint8_t*)w->scratch(need, cap) : nullptr;
    if (!base) return set_error(JB_ERR_NOMEM, "batched gemm: %zu B of activation scratch unavailable", need);
    w->few = w->many = MmqOperand();
    ActQ a;
    a.q = (int8_t*)base;
    a.d = (float*)(base + (((size_t)N * K + 255) & ~(size_t)255));
    a.s = a.d + (size_t)N * (K / 32);
    const long long groups = (long long)N * (K / 32);
    JB_CUDA(launch_k(mmq_quantize_kernel, dim3((unsigned)((groups + 3) / 4)), dim3(32, 4), 0, st, pdl_enabled(), x, a, N, K, (int)(type == T_Q4K)));
    count_launch();
    JB_CUDA(launch_k(mmq_simple_kernel, dim3((M + 3) / 4, N), dim3(32, 4), 0, st, pdl_enabled(), y, (const uint8_t*)W, type, a, M, N, K, dbg));
    count_launch();
    return JB_OK;
}

}  // namespace jb
