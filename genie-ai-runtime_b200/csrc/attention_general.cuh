// attention_general.cuh — the general attention slice: one query head against keys [kv0, kv1) of an FP16, INT8, BF16 or
// FP32 cache of any head size up to 512 (values may have their own), optional sliding window, cache slot stride >= head
// size, optional softmax sink (a logit that joins the denominator only).
//
// Same mathematics as the reference's decode / split-K / prefill kernels (src/kernels/attention.cu:244-375, :382-514,
// :837-941: s_j = scale * q . k_j with k = k8 * ks for INT8, online softmax, o = Σ p_j v_j with v = v8 * vs), arranged
// differently: the 32 lanes of a warp split the head dimension (dims lane, lane + 32, ...), every warp walks its own
// strided run of keys and keeps its running maximum, sum and output accumulators in REGISTERS — no shared score tile,
// no CTA-wide barrier per tile — and the warps' states are merged once through shared memory at the end.
// Used by the general kernels of attention.cu and by the allocation-free entry point.
#pragma once
#include "layernorm.cuh"
#include <cfloat>
#include <type_traits>

namespace jb {

constexpr int AG_WARPS = 4;
constexpr int AG_THREADS = AG_WARPS * 32;
constexpr int AG_MAXD = 16;                 // dims per lane: head sizes up to 512
constexpr int AG_WIDE = 40;                 // the wide instances: up to 1280

// kv_kind: EK_F16, EK_INT8 (with scales ks / vs), EK_BF16 or EK_F32.  vhd: value head size (slots of the value cache are
// vhd wide; 0 = the keys' size and slot stride).  ldk, ldv: row strides in elements (0: n_kv slots).
struct AgCache { const void* k; const void* v; const float* ks; const float* vs; int n_kv, chd, kv_kind, window, vhd = 0, ldk = 0, ldv = 0; };

inline size_t ag_smem_bytes(int hd) { return (size_t)AG_WARPS * (hd + 2) * sizeof(float); }

__device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
// element d of a cache row of type CT (INT8 rows carry a scale)
template <typename CT> __device__ __forceinline__ float ag_elem(const char* row, int d, float) { return to_f32(reinterpret_cast<const CT*>(row)[d]); }
template <> __device__ __forceinline__ float ag_elem<int8_t>(const char* row, int d, float sc) { return (float)reinterpret_cast<const int8_t*>(row)[d] * sc; }
// Factor on the scores of the query at position p: 1 + coef * ln(floor((p + 1) / every) + 1); every <= 0: none.
__device__ __forceinline__ float q_temp_factor(int p, float coef, double every) {
    return every > 0.0 ? 1.0f + coef * logf((float)(floor((double)(p + 1) / every) + 1.0)) : 1.0f;
}
// Weight of the accumulated outputs when the softmax has running maximum M, running sum L and an optional sink logit.
__device__ __forceinline__ float sink_norm(float M, float L, const float* sink) {
    if (!sink) return L > 0.f ? 1.0f / L : 0.f;
    if (!(L > 0.f)) return 0.f;
    const float top = fmaxf(M, *sink), e = expf(M - top);
    return e / (L * e + expf(*sink - top));
}

// sigmoid of a head's gate logit; 1 without gates
__device__ __forceinline__ float head_gate(const float* gate, int ldg, int row, int head) { return gate ? 1.0f / (1.0f + expf(-gate[(size_t)row * ldg + head])) : 1.0f; }

template <typename CT, int MAXD, typename QT, class Emit>
__device__ __forceinline__ void ag_slice_typed(const QT* q, const AgCache& c, int kvh, int hd, int seq, int kv0, int kv1, float scale,
                                         float* sm, float& M, float& L, Emit emit) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int vhd = c.vhd > 0 ? c.vhd : hd, vslot = c.vhd > 0 ? c.vhd : c.chd;
    constexpr size_t es = sizeof(CT);
    const bool scaled = es == 1;
    const size_t krow = (c.ldk > 0 ? (size_t)c.ldk : (size_t)c.n_kv * c.chd) * es, koff = (size_t)kvh * c.chd * es;
    const size_t vrow = (c.ldv > 0 ? (size_t)c.ldv : (size_t)c.n_kv * vslot) * es, voff = (size_t)kvh * vslot * es;
    float qr[MAXD], acc[MAXD];
    #pragma unroll
    for (int i = 0; i < MAXD; ++i) { const int d = lane + 32 * i; qr[i] = d < hd ? to_f32(q[d]) : 0.f; acc[i] = 0.f; }
    float m = -FLT_MAX, l = 0.f;
    const int first = c.window > 0 ? max(kv0, seq - c.window) : kv0;      // keys before the window contribute nothing
    // Small heads: the rows of BATCH keys are requested together and the keys taken in the same order as one by one (a key at a time, each with its
    // trip to memory, 134 FP32 keys of 128 took 41 us; so 8).
    constexpr int BATCH = MAXD <= 4 ? 8 : MAXD <= 8 ? 4 : 1;
    for (int p0 = first + warp; p0 < kv1; p0 += BATCH * AG_WARPS) {
        float kd[BATCH][MAXD], vd[BATCH][MAXD], s[BATCH];
        #pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            const int p = min(p0 + j * AG_WARPS, kv1 - 1);
            const char* kr = reinterpret_cast<const char*>(c.k) + (size_t)p * krow + koff;
            const float ksc = scaled && c.ks ? c.ks[(size_t)p * c.n_kv + kvh] : 1.0f;
            #pragma unroll
            for (int i = 0; i < MAXD; ++i) { const int d = lane + 32 * i; kd[j][i] = d < hd ? ag_elem<CT>(kr, d, ksc) : 0.f; }
        }
        if (BATCH > 1) {
            #pragma unroll
            for (int j = 0; j < BATCH; ++j) {
                const int p = min(p0 + j * AG_WARPS, kv1 - 1);
                const char* vr = reinterpret_cast<const char*>(c.v) + (size_t)p * vrow + voff;
                const float vsc = scaled && c.vs ? c.vs[(size_t)p * c.n_kv + kvh] : 1.0f;
                #pragma unroll
                for (int i = 0; i < MAXD; ++i) { const int d = lane + 32 * i; vd[j][i] = d < vhd ? ag_elem<CT>(vr, d, vsc) : 0.f; }
            }
        }
        #pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            float dot = 0.f;
            #pragma unroll
            for (int i = 0; i < MAXD; ++i) dot += qr[i] * kd[j][i];
            s[j] = warp_sum(dot) * scale;
        }
        #pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            const int p = p0 + j * AG_WARPS;
            if (p >= kv1) break;
            const float m_new = fmaxf(m, s[j]), corr = expf(m - m_new), pw = expf(s[j] - m_new);
            m = m_new;
            l = l * corr + pw;
            if (BATCH > 1) {
                #pragma unroll
                for (int i = 0; i < MAXD; ++i) { const int d = lane + 32 * i; if (d < vhd) acc[i] = acc[i] * corr + pw * vd[j][i]; }
            } else {
                const char* vr = reinterpret_cast<const char*>(c.v) + (size_t)p * vrow + voff;
                const float vsc = scaled && c.vs ? c.vs[(size_t)p * c.n_kv + kvh] : 1.0f;
                #pragma unroll
                for (int i = 0; i < MAXD; ++i) { const int d = lane + 32 * i; if (d < vhd) acc[i] = acc[i] * corr + pw * ag_elem<CT>(vr, d, vsc); }
            }
        }
    }
    // merge the warps' states
    float* sm_m = sm; float* sm_l = sm + AG_WARPS; float* sm_o = sm + 2 * AG_WARPS;     // [warp][vhd]
    if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
    #pragma unroll
    for (int i = 0; i < MAXD; ++i) { const int d = lane + 32 * i; if (d < vhd) sm_o[warp * vhd + d] = acc[i]; }
    __syncthreads();
    M = -FLT_MAX;
    #pragma unroll
    for (int w = 0; w < AG_WARPS; ++w) M = fmaxf(M, sm_m[w]);
    float e[AG_WARPS];
    L = 0.f;
    #pragma unroll
    for (int w = 0; w < AG_WARPS; ++w) { e[w] = sm_l[w] > 0.f ? expf(sm_m[w] - M) : 0.f; L += sm_l[w] * e[w]; }
    for (int d = tid; d < vhd; d += AG_THREADS) {
        float o = 0.f;
        #pragma unroll
        for (int w = 0; w < AG_WARPS; ++w) o += sm_o[w * vhd + d] * e[w];
        emit(d, o);
    }
}

// Runs on all AG_THREADS threads of the CTA.  On return M and L hold the slice's running maximum and sum (the same
// on every thread; M = -FLT_MAX for an empty slice) and emit(d, acc_d) has been called once per dimension d with the
// unnormalised output, each d by exactly one thread.  `sm` = ag_smem_bytes(hd) of shared memory.
template <int MAXD = AG_MAXD, typename QT, class Emit>
__device__ __forceinline__ void ag_slice(const QT* q, const AgCache& c, int kvh, int hd, int seq, int kv0, int kv1, float scale,
                                         float* sm, float& M, float& L, Emit emit) {
    // fp16 queries go with an FP16 or INT8 cache, BF16 and FP32 queries with a cache of their own type
    if constexpr (sizeof(QT) == 2 && !std::is_same<QT, __nv_bfloat16>::value) {
        if (c.kv_kind == EK_INT8) { ag_slice_typed<int8_t, MAXD>(q, c, kvh, hd, seq, kv0, kv1, scale, sm, M, L, emit); return; }
    }
    ag_slice_typed<QT, MAXD>(q, c, kvh, hd, seq, kv0, kv1, scale, sm, M, L, emit);
}

// out = Σ_s acc_s e^{m_s-M} / (Σ_s l_s e^{m_s-M} [+ e^{sink-M}]) over the partial records (m, l, acc[hd]) of one head (reference :944-969)
template <typename OT>
__device__ __forceinline__ void ag_merge_slices(OT* out, const float* pb, int hd, int n_splits, const float* sink = nullptr, float gate = 1.f) {
    float M = -FLT_MAX;
    for (int s = 0; s < n_splits; ++s) M = fmaxf(M, pb[(size_t)s * (hd + 2)]);
    float L = 0.f;
    for (int s = 0; s < n_splits; ++s) L += pb[(size_t)s * (hd + 2) + 1] * expf(pb[(size_t)s * (hd + 2)] - M);
    const float inv = sink_norm(M, L, sink) * gate;
    for (int d = threadIdx.x; d < hd; d += blockDim.x) {
        float acc = 0.f;
        for (int s = 0; s < n_splits; ++s) acc += pb[(size_t)s * (hd + 2) + 2 + d] * expf(pb[(size_t)s * (hd + 2)] - M);
        out[d] = from_f32<OT>(acc * inv);
    }
}

}  // namespace jb
