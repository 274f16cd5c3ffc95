// mmq_few.cuh — the K-quant products of a few tokens (2..128) and the kernels between them: see mmq_few.cu.
#pragma once
#include "../../include/jllm_b200.h"
#include "common.cuh"
#include "elementwise.cuh"
#include <cuda.h>
#include <vector>

namespace jb {

constexpr int MF_MAX_TOKENS = 128;
constexpr int MF_MAX_SEG = 3;

// One matrix of a product.  Its 128-row tiles times its super-blocks are its units of work, dealt evenly to the `ctas` CTAs from cta0 on:
// CTA i takes units [i * units / ctas, (i + 1) * units / ctas), so a tile has the sums of one or several consecutive CTAs.
// perm: weight rows r, r + 1, ... of a tile lie `128 / perm` positions apart (mf_position), 1: in order.
struct MfSeg { int cta0, ctas, tiles, units, M, m0, q6, perm; };
struct MfProduct {                       // fixed by the weights; a session keeps one per product
    CUtensorMap map[MF_MAX_SEG];
    MfSeg seg[MF_MAX_SEG];
    int nseg = 0, K = 0, rows = 0;       // rows: 128 x tiles of all segments, the width of a token's partial sums
    int slots = 0;                       // sums of a tile, at most
};
struct MfWeight { const void* W; int type; int M; };
// false: these weights stay with the other kernels
bool mf_plan(MfProduct& p, const MfWeight* w, int n, int K);

inline int mf_padded(int N) { return (N + 15) & ~15; }
inline size_t mf_x_bytes(int K, int N) { return (size_t)(K / QK_K) * 34 * 16 * mf_padded(N); }       // quantised activations, either flavour
inline size_t mf_part_bytes(const MfProduct& p, int N) { return (size_t)p.slots * N * p.rows * sizeof(float); }
size_t mf_edge_bytes(int N);                                                                         // partial sums of a product with outputs of its own

// Quantised activations of a product: x4 for Q4_K matrices, x6 for Q6_K ones (null where the product has none).
struct MfOperand { __half* x4 = nullptr; __half* x6 = nullptr; };
inline MfOperand mf_operand(const MfProduct& p, void* x4, void* x6) {
    MfOperand o;
    for (int i = 0; i < p.nseg; ++i) (p.seg[i].q6 ? o.x6 : o.x4) = (__half*)(p.seg[i].q6 ? x6 : x4);
    return o;
}

// Sums [slot][token][rows] into part.
int launch_mf_sums(const MfProduct& p, const MfOperand& x, float* part, int N, cudaStream_t st);
// y[token][M] in fp16 of a product of one matrix; edge: mf_edge_bytes of scratch.
int launch_mf_out(const MfProduct& p, const MfOperand& x, __half* y, float* edge, int N, cudaStream_t st);

// The kernels between the products.
// x (+ the sums of the product in front, when p is given: x_out) -> RMSNorm with weights w, quantised into q (w null: the sum alone)
int launch_mf_norm(const MfProduct* p, const float* part, const __half* x, __half* x_out, const float* w, float eps, int H, const MfOperand& q, int N, cudaStream_t st);
// sums of Q, K, V -> head norms, rotation, q in fp16, K and V rows into the caches: lists (streams at one position) or one cache (tokens of a prompt)
struct MfPrep {
    __half* q; const float* q_norm; const float* k_norm; float eps;
    int8_t* const* k_list; int8_t* const* v_list; float* const* ks_list; float* const* vs_list;
    int8_t* k; int8_t* v; float* ks; float* vs;
    const int* d_pos; int pos, pos_step;
    int n_heads, n_kv, neox;
};
int launch_mf_prep(const MfProduct& p, const float* part, const MfPrep& a, float theta, int N, cudaStream_t st);
// silu(gate) * up of the sums of a gate and up product, quantised
int launch_mf_glu(const MfProduct& p, const float* part, const MfOperand& q, int N, cudaStream_t st);
// fp16 vectors [N][K], quantised
int launch_mf_quantise(const __half* x, const MfOperand& q, int K, int N, cudaStream_t st);

// ── the kernels between the products of many tokens (mmq_rows.cu): fp16 results in, rows of mmq_tc.cu's operand out (x4 as for Q4_K, x6 as for
// Q6_K matrices, null where not asked for) ──
inline int mr_width(int K) { return K + (K / 16 + 63) / 64 * 64; }       // columns of a Q4_K operand: sums and centring sums of K / 32 groups, in whole K tiles; Q6_K: K
// x + add (add null: x alone; else x_out) -> RMSNorm with weights w, quantised (w null: the sum alone)
int launch_mr_norm(const __half* x, const __half* add, __half* x_out, const float* w, float eps, int H, const MfOperand& q, int N, cudaStream_t st);
// head norms and rotation of q in place, K and V rows of tokens pos .. pos + N - 1 into one cache
struct MrPrep {
    __half* q; const __half* k_in; const __half* v_in; const float* q_norm; const float* k_norm; float eps;
    int8_t* k; int8_t* v; float* ks; float* vs;
    int pos, n_heads, n_kv, neox;
};
int launch_mr_prep(const MrPrep& a, float theta, int N, cudaStream_t st);
int launch_mr_glu(const __half* gate, const __half* up, const MfOperand& q, int K, int N, cudaStream_t st);
int launch_mr_quantise(const __half* x, const MfOperand& q, int K, int N, cudaStream_t st);

// ── the layers of a Llama / Qwen3 model over a few tokens ──
struct MfLayer { MfProduct qkv, wo, gate_up, down; };
struct MfModel {
    std::vector<MfLayer> layers;         // empty: the model stays with the other kernels
    MfProduct out;                       // nseg 0: logits are not asked for
    int hidden = 0, q_dim = 0, ffn = 0;
    // scratch: operands of the hidden width in both flavours, of the heads' outputs and of the MLP's; partial sums
    void *xh4 = nullptr, *xh6 = nullptr, *xa = nullptr, *xi = nullptr;
    float* part = nullptr;
    bool plan(const jllm_b200_model_desc& m, bool with_out);
    size_t bytes(int N) const;
    void place(void* scratch, int N);
    // the same operands as rows of many tokens (mmq_rows.cu)
    size_t row_bytes(int N) const;
    void place_rows(void* scratch, int N);
};

}  // namespace jb
