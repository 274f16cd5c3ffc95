// attention.cuh — host-side call block of the attention kernels.
#pragma once
#include "layernorm.cuh"

namespace jb {

struct AttnCall {
    void* out = nullptr; const void* q = nullptr;      // fp16, or the cache's type when that is BF16 / FP32
    const void* k = nullptr; const void* v = nullptr; const float* ks = nullptr; const float* vs = nullptr;
    // ragged batch: device arrays of per-sequence pointers / lengths (batch entries)
    const void* const* k_list = nullptr; const void* const* v_list = nullptr;
    const float* const* ks_list = nullptr; const float* const* vs_list = nullptr; const int* seq_lens = nullptr;
    // ragged batch on the TMA path: HOST array of [batch][K, V] tensor maps (built from the caches' addresses, see
    // jllm_b200_attn_plan_create; they travel to the kernel as parameters); the K/V pointer lists are then not needed
    const void* tma_maps = nullptr;
    int batch = 1, max_seq = 0;      // max_seq: rows every cache holds (bounds the slices of a ragged batch and the tensor maps)
    int n_heads = 0, n_kv = 0, hd = 0, chd = 0, seq_len = 0;
    const int* d_pos = nullptr;       // device position: seq_len = *d_pos + 1
    float scale = 1.f; int kv_int8 = 0, window = 0, n_splits = 0;
    int causal_start = -1;            // >= 0: prefill, `batch` = number of query tokens
    // BF16 / FP32 caches (kv_kind overrides kv_int8): own value head size, row strides of q and out, softmax sink per query
    // head, query temperature 1 + qt_coef * ln(floor((p + 1) / qt_every) + 1) at position p
    int kv_kind = -1, vhd = 0, ldq = 0, ldo = 0;
    const float* sink = nullptr;
    float qt_coef = 0.f; double qt_every = 0.0;
    // BF16 / FP32 caches: row strides of k and v in elements (0: n_kv slots); gate: a logit per (row, query head), row stride ldg,
    // whose sigmoid multiplies the head's output; records: leave the slices' (m, l, acc[vhd]) at [row][head][slice], unmerged and
    // without gate; k2: the last hd2 of the hd key elements lie there (row stride ldk2), the same for every head
    int ldk = 0, ldv = 0;
    const float* gate = nullptr; int ldg = 0;
    float* records = nullptr;
    bool early = false;               // latent decode: the cache rows and *d_pos were complete before the kernel in front of this one started
    float* scratch = nullptr;                                          // latent caches: where merged slices go in between (null: the library's)
    const void* k2 = nullptr; int hd2 = 0, ldk2 = 0;
    int kind() const { return kv_kind >= 0 ? kv_kind : kv_int8 ? EK_INT8 : EK_F16; }
};

int    attn_splits_for(int seq_len);
float* splitk_buffer(size_t floats, bool may_alloc);
int    launch_attention_general(const AttnCall& c, cudaStream_t st);
int    launch_attention_merge(const AttnCall& c, const float* part, int n_splits, int ldo, cudaStream_t st);   // records [batch][head][slice] -> out
int    launch_attention(const AttnCall& c, cudaStream_t st);      // picks the fast path when it applies
bool   attention_tma_applies(const AttnCall& c);                  // INT8 KV, head_dim 128, GQA 1/2/4, no window, cache extent known
int    launch_attention_tma(const AttnCall& c, cudaStream_t st);
bool   attn_tma_encode(void* map_out128, const void* cache_base, int rows, int n_kv);
bool   attention_prefill_fast_applies(const AttnCall& c);          // causal prefill (causal_start >= 0), INT8 KV, head_dim 128, GQA 1/2/4
int    launch_attention_prefill_fast(const AttnCall& c, cudaStream_t st);
// causal prefill on tcgen05 (attention_tc.cu): BF16 caches, and INT8 caches with a workspace (c.scratch, attention_tc_scratch bytes)
constexpr int AT_MIN_TOKENS = 64;
int    attention_tc_min_tokens(int n_heads, int n_kv);            // INT8 caches
bool   attention_tc_applies(const AttnCall& c);
int    launch_attention_tc(const AttnCall& c, cudaStream_t st);
size_t attention_tc_scratch(int n_kv, int positions);
bool   attention_bf16_applies(const AttnCall& c);                  // BF16 cache, head sizes multiples of 8 up to 256: decode and causal prefill
int    launch_attention_bf16(const AttnCall& c, cudaStream_t st);
int    launch_attention_float(const AttnCall& c, cudaStream_t st);    // BF16 and FP32 caches: the tensor-core kernels where they apply
int    attn_bf16_splits(int seq_len, int n_heads, int n_kv);       // KV slices of a decode call at this length
// Latent caches (one key row of c.hd elements that all heads share, its first c.vhd also the value; c.n_kv = 1, c.v = c.k):
// the tensor-core kernel where it applies, else the general one.
bool   attention_latent_applies(const AttnCall& c);
int    attn_latent_splits(int seq_len, int rows);                  // KV slices for `rows` (token, head) pairs
size_t attn_latent_records(int n_heads, int vhd);                  // floats of the records of any call with these heads, decoding (both number formats) or a chunk
int    launch_attention_latent(const AttnCall& c, cudaStream_t st);
bool   attention_keys2_applies(const AttnCall& c);                 // causal prefill with keys in two parts (k2)

}  // namespace jb
