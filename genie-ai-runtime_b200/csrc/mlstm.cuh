// mlstm.cuh — the matrix memory of xLSTM: per head a state S [dim][vdim], a normaliser n [dim] and a running maximum m, all fp32,
//     m' = max(f + m, i),  S' = e^(f + m - m') S + e^(i - m') k v^T,  n' likewise with k alone,
//     o = S'^T q / (max(|n' . q|, e^(-m')) + 1e-6)
// with log gates i = cap tanh((zi + bi) / cap) and f = logsigmoid(cap tanh((zf + bf) / cap)); then o over its root mean square,
// times a weight, times sigmoid(g).  Everything but the projections (q, k, v, g, zi, zf) is computed in fp32.
#pragma once
#include "layernorm.cuh"

namespace jb {

struct MlstmCall {
    int kind = EK_BF16, heads = 0, dim = 0, vdim = 0;
    // projections of the tokens, activation type, row stride ld: q [heads * dim], k, v [heads * vdim], g at these columns
    const void* proj = nullptr; int ld = 0, off_q = 0, off_k = 0, off_v = 0, off_g = 0;
    const float* gates = nullptr; int ldgates = 0;       // raw i [heads] then f [heads] of each token, fp32
    const float* bias = nullptr;                         // the same order
    float cap = 0.f, eps = 0.f;
    const float* norm_w = nullptr;                       // [heads * vdim]
    float* state = nullptr;                              // mlstm_state_floats: S [head][dim][pad8(vdim)], n [head][dim], m [head], and room for the next n and m
    float* raw = nullptr;                                // [tokens][heads * vdim] fp32, scratch of prompts
    void* out = nullptr; int ldo = 0;                    // activation type
};
size_t mlstm_state_floats(int heads, int dim, int vdim);
// Tokens start .. start + n - 1 of one sequence (a state older than position 0 is not read).  d_pos: one token at *d_pos instead.
int launch_mlstm(const MlstmCall& a, int n, int start, const int* d_pos, cudaStream_t st);
bool mlstm_chunks_apply(const MlstmCall& a, int n);                       // tensor-core kernels for prompts: bf16, sizes they hold
int launch_mlstm_chunks(const MlstmCall& a, int n, int start, cudaStream_t st);   // leaves `raw`, S, and the next n and m

// Up to how many tokens one chunk of mlstm_short.cu serves.  us with the norm that follows, there / in mlstm_chunk.cu, 16 and 64 tokens: 8 heads of 256 x 512
// 12.1 and 13.5 / 16.4 and 17.4, 4 heads of 128 x 256 8.7 and 9.5 / 12.3 and 12.4.
constexpr int MLSTM_SHORT = 64;
int launch_mlstm_short(const MlstmCall& a, int n, int start, cudaStream_t st);

// floats from n (or m) to its next value
__host__ __device__ inline size_t mlstm_next(const MlstmCall& a) { return (size_t)a.heads * a.dim + pad8(a.heads); }

#ifdef __CUDACC__
__device__ __forceinline__ float mlstm_log_i(const MlstmCall& a, int t, int h) { return a.cap * tanhf((a.gates[(size_t)t * a.ldgates + h] + a.bias[h]) / a.cap); }
__device__ __forceinline__ float mlstm_log_f(const MlstmCall& a, int t, int h) {
    const float x = a.cap * tanhf((a.gates[(size_t)t * a.ldgates + a.heads + h] + a.bias[a.heads + h]) / a.cap);
    return fminf(x, 0.f) - log1pf(expf(-fabsf(x)));
}
#endif

}  // namespace jb
