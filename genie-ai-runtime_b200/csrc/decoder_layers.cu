// decoder_layers.cu — models described layer by layer (jllm_b200_layered_desc) behind the decoder session.
//
// One decode step is six launches per layer, each product taking the work around it along:
//   [residual step + norm1 + Q/K/V product, K / V rows straight into the cache]  ->  attention  ->  W_o
//   [residual step + norm2 + router product]  ->  [routing + gate / up + SwiGLU of the chosen experts]  ->  [W_down, weighted sum]
// and the residual step of the last sublayer rides in the logits product.  A prompt chunk runs the same steps over all its
// tokens: residual step (layernorm.cu), tensor-core products (dense_tc.cu; fp32: dense_simt.cu), query-tiled attention, and
// experts over expert-major copies of the tokens (moe.cu).
//
// Parallel layers (one norm, both sublayers read it) put every product of the normed vector into one matrix, and both outputs
// into one.  A decode step is three launches around an mLSTM mixer,
//   [residual step + norm + q, k, v, gates, gate / up with gelu]  ->  recurrence  ->  [ls1 * (W_o att) + ls2 * (W_down act)]
// and six around latent attention, whose middle is
//   [latent norm + queries with rotation; one CTA stores the latent row]  ->  W_k^T per head  ->  attention over the latents
//   ->  [slice merge + gate + W_v per head].
// A prompt chunk expands the latents to keys and values when that costs less arithmetic than scoring against the latents
// themselves (long chunks), and otherwise works like a decode step.
#include "../../include/jllm_b200_api.hpp"
#include "decoder.cuh"
#include "attention.cuh"
#include "dense.cuh"
#include "mlstm.cuh"
#include <new>
#include <vector>

using namespace jb;

namespace {

// Activations of `rows` tokens; x ping-pongs between two buffers because the product that applies the residual step reads
// the old row in every CTA while one of them stores the new one.
struct Acts {
    void* slab = nullptr;
    float *x[2] = {nullptr, nullptr}, *y = nullptr, *z = nullptr, *wts = nullptr;
    void *h = nullptr, *q = nullptr, *att = nullptr, *hp = nullptr, *a = nullptr, *ye = nullptr;
    int *ids = nullptr, *rank = nullptr, *slots = nullptr, *counts = nullptr, *off = nullptr, *rows = nullptr;
    // parallel layers: second sublayer's output, raw mLSTM outputs; projections of h, normed query latents, unrotated queries, attention
    // outputs over latents (q: latent queries; z: what of the projections stays fp32)
    float *y2 = nullptr, *raw = nullptr, *records = nullptr, *part = nullptr;      // part: K ranges of a prompt's products
    void *proj = nullptr, *qn = nullptr, *qu = nullptr, *lat = nullptr;
};
struct Rotation { int half, dims; double base; float2* table; };

constexpr int DT_HEADS = MOE_MAX_EXPERTS;       // most heads of a product with a matrix per head
enum { MIX_ATTENTION = 0, MIX_LATENT = 1, MIX_MLSTM = 2 };
// sizes and places of a parallel layer's rows and buffers
struct LatentDims {
    int H, dim, rot, vdim, q_rank, r, r8, kd, off_c, off_r, off_g, ldz;       // kd: elements of a cache row
    explicit LatentDims(const jllm_b200_layer_spec& w) : H(w.n_heads), dim(w.head_dim), rot(w.rot_dim), vdim(w.v_dim), q_rank(w.q_rank), r(w.kv_rank), r8(pad8(w.kv_rank)),
        kd(pad8(w.kv_rank) + pad8(w.rot_dim)), off_c(pad8(w.q_rank)), off_r(pad8(w.q_rank) + pad8(w.kv_rank)), off_g(off_r + pad8(w.rot_dim)), ldz(off_g + pad8(w.n_heads)) {}
};
struct MlstmDims {
    int H, dim, vdim, off_k, off_v, off_g, ld, ldz;
    explicit MlstmDims(const jllm_b200_layer_spec& w) : H(w.n_heads), dim(w.head_dim), vdim(w.v_dim), off_k(pad8(H * dim)), off_v(2 * off_k), off_g(off_v + pad8(H * vdim)),
        ld(off_g + pad8(H * vdim)), ldz(pad8(2 * H)) {}
};

struct LayerDecoder : jllm_b200_decoder {
    jllm_b200_layered_desc m;
    std::vector<jllm_b200_layer_spec> layers;
    std::vector<int> source;                    // layer whose cache rows a layer reads
    jllm::LayeredKVCache kv;
    int kind = EK_BF16;
    int max_q = 0, max_v = 0, max_e = 0, max_top = 0, max_ff = 0, max_heads = 0;
    int max_z = 0, max_proj = 0, max_qn = 0, max_qu = 0, max_lat = 0, max_raw = 0;       // parallel layers
    size_t max_rec = 0;
    bool recurrent = false;
    std::vector<Rotation> rotations;
    std::vector<int> rotation_of;               // per layer, -1: none
    void *kexp = nullptr, *vexp = nullptr;      // keys and values expanded from latents, max_context rows
    Acts one, many;                             // decode step, prompt chunk
    int last_x = 0;                             // which x buffer the chunk's residual ended in
    NormStep pending;                           // the last sublayer's exit of the chunk, still to be applied

    ~LayerDecoder() override { if (one.slab) cudaFree(one.slab); if (many.slab) cudaFree(many.slab); if (kexp) cudaFree(kexp); if (vexp) cudaFree(vexp); for (auto& r : rotations) cudaFree(r.table); kv.destroy(); }
    int alloc_acts(Acts& a, size_t rows, bool chunk, cudaStream_t st);
    NormStep entry(const Acts& a, const float* w, const float* b) const;
    MoeRoute route(const jllm_b200_layer_spec& w) const;
    DenseGemm product(const Acts& a) const { DenseGemm g; g.kind = kind; g.early = true; g.part = a.part; g.part_floats = a.part ? gemm_pair_part_floats() : 0; return g; }
    AttnCall attention_call(int l, const Acts& a) const;
    // parallel layers
    int in_segments(OutSeg* seg, const jllm_b200_layer_spec& w, const Acts& a, int& M) const;
    LatentRows latent_rows_call(int l, const Acts& a) const;
    AttnCall latent_call(int l, const Acts& a) const;
    MlstmCall mlstm_call(int l, const Acts& a) const;
    bool expands(int l, int n) const;
    int add_rotation(int half, int dims, double base);
    int latent_step(int l, const Acts& a, int n_splits, cudaStream_t st);
    int latent_chunk(int l, const Acts& a, int n, int start, cudaStream_t st);
    bool keeps_state() const override { return recurrent; }
    int enqueue_step(int n_splits, cudaStream_t st) override;
    int reserve_chunk(int tokens, cudaStream_t st) override;
    int enqueue_chunk(const int* dev_tokens, int n, int start, cudaStream_t st) override;
    int enqueue_rows(const int* host_rows, int n, float* out, cudaStream_t st) override;
    int attn_splits(int seq_len) const override {
        if (kind == EK_F32) return attn_splits_for(seq_len);
        int s = 1;
        for (const auto& w : layers) {
            const int n = w.mixer == MIX_LATENT ? attn_latent_splits(seq_len, w.n_heads) : w.mixer == MIX_MLSTM ? 1 : attn_bf16_splits(seq_len, w.n_heads, w.n_kv_heads);
            s = n > s ? n : s;
        }
        return s;
    }
    void clear_cache() override {}              // rows beyond the position are never read
    const void* buffer(int which) override { return which == 0 ? one.x[0] : which == 7 ? kv.key_ptr(0, 0) : nullptr; }
};

int LayerDecoder::alloc_acts(Acts& a, size_t R, bool chunk, cudaStream_t st) {
    const size_t es = elem_bytes(kind), W = pad8(m.width), T = max_top;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    bool ranges = chunk && kind == EK_BF16;
    for (int pass = 0; pass < 2; ++pass) {
        size_t at = 0;
        auto take = [&](size_t b) { void* r = (char*)a.slab + at; at += al(b); return r; };
        float* x0 = (float*)take(R * W * 4); float* x1 = (float*)take(R * W * 4); float* y = (float*)take(R * W * 4);
        void* h = take(R * W * es); void* q = take(R * pad8(max_q) * es); void* att = take(R * pad8(max_v) * es);
        float* z = (float*)take(R * (max_e > max_z ? max_e : max_z) * 4); float* wts = (float*)take(R * T * 4);
        int* ids = (int*)take(R * T * 4); void* ga = take(R * T * pad8(max_ff) * es);
        float *y2 = nullptr, *raw = nullptr, *rec = nullptr; void *proj = nullptr, *qn = nullptr, *qu = nullptr, *lat = nullptr;
        if (m.parallel) {
            proj = take(R * max_proj * es); qu = take(R * max_qu * es); rec = (float*)take(max_rec * 4);
            if (chunk) { y2 = (float*)take(R * W * 4); raw = (float*)take(R * max_raw * 4); qn = take(R * max_qn * es); lat = take(R * max_lat * es); }
        }
        int *rank = nullptr, *slots = nullptr, *counts = nullptr, *off = nullptr, *rows = nullptr; void *hp = nullptr, *ye = nullptr; float* part = nullptr;
        if (chunk) {
            rank = (int*)take(R * T * 4); slots = (int*)take(R * T * 4); counts = (int*)take((size_t)(max_e + 1) * 4); off = (int*)take((size_t)(max_e + 1) * 4);
            rows = (int*)take(R * 4);
            if (!m.parallel) { hp = take(R * T * W * es); ye = take(R * T * W * es); }
        }
        const size_t acts = at;
        if (ranges) part = (float*)take(gemm_pair_part_floats() * 4);
        if (pass == 0) {
            if (ranges && cudaMalloc(&a.slab, at) != cudaSuccess) { cudaGetLastError(); a.slab = nullptr; ranges = false; }      // the products do without
            if (!a.slab && cudaMalloc(&a.slab, acts) != cudaSuccess) { cudaGetLastError(); a.slab = nullptr; return set_error(JB_ERR_NOMEM, "decoder: %zu B of activations", acts); }
            JB_CUDA(cudaMemsetAsync(a.slab, 0, acts, st));         // the padding of every row stays zero; on the stream of the kernels that follow
            continue;
        }
        a.x[0] = x0; a.x[1] = x1; a.y = y; a.h = h; a.q = q; a.att = att; a.z = z; a.wts = wts; a.ids = ids; a.a = ga;
        a.rank = rank; a.slots = slots; a.counts = counts; a.off = off; a.rows = rows; a.hp = hp; a.ye = ye;
        a.y2 = y2; a.raw = raw; a.proj = proj; a.qn = qn; a.qu = qu; a.lat = lat; a.records = rec; a.part = part;
    }
    return JB_OK;
}

NormStep LayerDecoder::entry(const Acts& a, const float* w, const float* b) const {
    NormStep n;
    n.W = m.width; n.eps = m.eps; n.mult = m.residual_mult; n.next_w = w; n.next_b = b; n.h = a.h; n.rms = m.rms_norm; n.embed_scale = m.embed_scale;
    return n;
}
MoeRoute LayerDecoder::route(const jllm_b200_layer_spec& w) const {
    MoeRoute r;
    r.n_experts = w.n_experts; r.top = w.top; r.n_groups = w.n_groups > 0 ? w.n_groups : 1; r.keep_groups = w.n_groups > 1 ? w.keep_groups : 1; r.correction = w.correction;
    return r;
}
AttnCall LayerDecoder::attention_call(int l, const Acts& a) const {
    const jllm_b200_layer_spec& w = layers[l];
    AttnCall c;
    c.out = a.att; c.q = a.q; c.k = kv.key_ptr(source[l], 0); c.v = kv.val_ptr(source[l], 0); c.kv_kind = kind;
    c.n_heads = w.n_heads; c.n_kv = w.n_kv_heads; c.hd = c.chd = w.head_dim; c.vhd = w.v_dim; c.ldq = pad8(w.n_heads * w.head_dim); c.ldo = pad8(w.n_heads * w.v_dim);
    c.scale = w.scale; c.sink = w.sink; c.qt_coef = w.q_temp_coef; c.qt_every = w.q_temp_every; c.max_seq = m.max_context;
    return c;
}
// output places of the Q/K/V product: q rows to the activations, k and v rows to the cache at row 0 of `pos`
template <class Args>
void qkv_segments(Args& g, const jllm_b200_layer_spec& w, void* q, void* k, void* v, int at_pos) {
    const int Q = w.n_heads * w.head_dim, K = w.n_kv_heads * w.head_dim, V = w.n_kv_heads * w.v_dim;
    g.seg[0] = OutSeg{q, pad8(Q), Q, 0, 0};
    g.nseg = 1; g.M = Q;
    if (w.kv_from < 0) {
        g.seg[1] = OutSeg{k, K, K, 0, at_pos};
        g.seg[2] = OutSeg{v, V, V, 0, at_pos};
        g.nseg = 3; g.M = Q + K + V;
    }
}

// output places of the products of h: what stays fp32 or goes on as projections, then the MLP's activation
int LayerDecoder::in_segments(OutSeg* seg, const jllm_b200_layer_spec& w, const Acts& a, int& M) const {
    int n = 0;
    if (w.mixer == MIX_LATENT) {
        const LatentDims d(w);
        seg[n++] = OutSeg{a.z, d.ldz, d.ldz, 1, 0};
    } else {
        const MlstmDims d(w);
        seg[n++] = OutSeg{a.proj, d.ld, d.ld, 0, 0};
        seg[n++] = OutSeg{a.z, d.ldz, d.ldz, 1, 0};
    }
    if (w.mlp_dim > 0) { seg[n] = OutSeg{a.a, pad8(w.mlp_dim), 2 * w.mlp_dim, 0, 0}; seg[n++].pair = PAIR_GELU; }
    M = 0;
    for (int i = 0; i < n; ++i) M += seg[i].rows;
    return n;
}
LatentRows LayerDecoder::latent_rows_call(int l, const Acts& a) const {
    const jllm_b200_layer_spec& w = layers[l];
    const LatentDims d(w);
    LatentRows r;
    r.z = a.z; r.ldz = d.ldz; r.off_q = 0; r.off_c = d.off_c; r.off_r = d.off_r; r.q_rank = d.q_rank; r.kv_rank = d.r; r.rot_dim = d.rot;
    r.q_w = w.dq_norm; r.c_w = w.dkv_norm; r.eps = m.eps; r.rot = rotations[rotation_of[l]].table; r.qn = a.qn; r.ldqn = pad8(d.q_rank);
    r.cache = kv.key_ptr(l, 0); r.ld = d.kd;
    return r;
}
// attention of latent queries (a.q, [token][head][kd]) over the latent rows
AttnCall LayerDecoder::latent_call(int l, const Acts& a) const {
    const LatentDims d(layers[l]);
    AttnCall c;
    c.out = a.lat; c.q = a.q; c.k = c.v = kv.key_ptr(l, 0); c.kv_kind = kind; c.n_heads = d.H; c.n_kv = 1; c.hd = c.chd = d.kd; c.vhd = d.r8;
    c.ldk = c.ldv = d.kd; c.ldq = d.H * d.kd; c.ldo = d.H * d.r8; c.scale = layers[l].scale; c.max_seq = m.max_context;
    return c;
}
MlstmCall LayerDecoder::mlstm_call(int l, const Acts& a) const {
    const jllm_b200_layer_spec& w = layers[l];
    const MlstmDims d(w);
    MlstmCall c;
    c.kind = kind; c.heads = d.H; c.dim = d.dim; c.vdim = d.vdim; c.proj = a.proj; c.ld = d.ld; c.off_k = d.off_k; c.off_v = d.off_v; c.off_g = d.off_g;
    c.gates = a.z; c.ldgates = d.ldz; c.bias = w.gate_bias; c.cap = w.gate_cap; c.eps = m.eps; c.norm_w = w.head_norm; c.state = kv.state_ptr(l); c.raw = a.raw;
    c.out = a.att; c.ldo = pad8(d.H * d.vdim);
    return c;
}
// Whether a chunk of n tokens expands the latents: per position it costs the two expansion products, and saves, per query, the
// difference between scores and sums over the latent and over the expanded heads.  Counted half: the expansion is a plain product
// at several times the rate of the attention kernels.
bool LayerDecoder::expands(int l, int n) const {
    const LatentDims d(layers[l]);
    if (kind != EK_BF16 || d.dim % 8 || d.rot % 8 || d.vdim % 8 || d.dim + d.rot > 256 || d.vdim > 256) return false;
    return 2ll * n * (d.kd + d.r8 - d.dim - d.rot - d.vdim) > (long long)(d.dim + d.vdim) * d.r;
}
int LayerDecoder::add_rotation(int half, int dims, double base) {
    for (size_t i = 0; i < rotations.size(); ++i) if (rotations[i].half == half && rotations[i].dims == dims && rotations[i].base == base) return (int)i;
    Rotation r = {half, dims, base, nullptr};
    if (cudaMalloc(&r.table, (size_t)m.max_context * half * sizeof(float2)) != cudaSuccess) { cudaGetLastError(); set_error(JB_ERR_NOMEM, "decoder: rotation table"); return -1; }
    rotations.push_back(r);
    return launch_rotation_table(r.table, m.max_context, half, dims, base, nullptr) ? -1 : (int)rotations.size() - 1;
}

int LayerDecoder::latent_step(int l, const Acts& a, int n_splits, cudaStream_t st) {
    const jllm_b200_layer_spec& w = layers[l];
    const LatentDims d(w);
    const int es = elem_bytes(kind), rec = d.r8 + 2;
    const Rotation& rot = rotations[rotation_of[l]];
    float* part = a.records;
    if ((size_t)d.H * n_splits * rec > max_rec) return set_error(JB_ERR_LIMIT, "decoder: records of %d slices", n_splits);
    DenseGemv u;
    u.mode = GEMV_PAIR; u.kind = kind; u.W = w.w_uq; u.M = d.H * (d.rot + d.dim); u.K = d.q_rank; u.d_pos = state;
    u.norm.x = a.z; u.norm.next_w = w.dq_norm; u.norm.W = d.q_rank; u.norm.eps = m.eps; u.norm.rms = 1;
    u.seg[0] = OutSeg{(char*)a.q + (size_t)d.r8 * es, d.H * d.kd, d.H * d.rot, 0, 0, PAIR_ROT, rot.table, rot.half, d.rot, d.kd};
    u.seg[1] = OutSeg{a.qu, d.H * pad8(d.dim), d.H * d.dim, 0, 0, PAIR_NONE, nullptr, 0, d.dim, pad8(d.dim)};
    u.nseg = 2;
    u.side = latent_rows_call(l, a); u.side.d_pos = state;
    DCHK(launch_dense_gemv(u, st));
    HeadProduct k;
    k.kind = kind; k.heads = d.H; k.M = d.r; k.K = d.dim; k.W = w.w_uk_t; k.x = a.qu; k.ldx = pad8(d.dim); k.y = a.q; k.ldy = d.kd;
    DCHK(launch_head_product(k, st));
    AttnCall c = latent_call(l, a);
    c.out = a.att; c.d_pos = state; c.n_splits = n_splits; c.records = part; c.early = true;      // the product in front of it runs behind the one that stored the row
    DCHK(launch_attention_latent(c, st));
    HeadProduct v;
    v.kind = kind; v.heads = d.H; v.M = d.vdim; v.K = d.r; v.W = (const char*)w.w_ukv + (size_t)d.H * d.dim * d.r8 * es; v.y = a.att; v.ldy = d.vdim;
    v.records = part; v.n_splits = n_splits; v.rec = rec; v.gate = a.z + d.off_g;
    return launch_head_product(v, st);
}

int LayerDecoder::latent_chunk(int l, const Acts& a, int N, int start, cudaStream_t st) {
    const jllm_b200_layer_spec& w = layers[l];
    const LatentDims d(w);
    const int es = elem_bytes(kind), d8 = pad8(d.dim);
    const Rotation& rot = rotations[rotation_of[l]];
    DCHK(launch_latent_rows(latent_rows_call(l, a), kind, N, start, st));
    const bool wide = expands(l, N);
    DenseGemm u = product(a);
    u.kind = kind; u.W = w.w_uq; u.M = d.H * (d.rot + d.dim); u.K = d.q_rank; u.N = N; u.x = a.qn; u.start = start; u.nseg = 2;
    const int qd = d.dim + d.rot;
    if (wide) {
        u.seg[0] = OutSeg{(char*)a.q + (size_t)d.dim * es, d.H * qd, d.H * d.rot, 0, 0, PAIR_ROT, rot.table, rot.half, d.rot, qd};
        u.seg[1] = OutSeg{a.q, d.H * qd, d.H * d.dim, 0, 0, PAIR_NONE, nullptr, 0, d.dim, qd};
    } else {
        u.seg[0] = OutSeg{(char*)a.q + (size_t)d.r8 * es, d.H * d.kd, d.H * d.rot, 0, 0, PAIR_ROT, rot.table, rot.half, d.rot, d.kd};
        u.seg[1] = OutSeg{a.qu, d.H * d8, d.H * d.dim, 0, 0, PAIR_NONE, nullptr, 0, d.dim, d8};
    }
    DCHK(launch_dense_gemm(u, st));
    if (wide) {
        if (!kexp) {
            size_t k = 0, v = 0;
            for (size_t i = 0; i < layers.size(); ++i)
                if (layers[i].mixer == MIX_LATENT) {
                    const LatentDims e(layers[i]);
                    if ((size_t)e.H * e.dim > k) k = (size_t)e.H * e.dim;
                    if ((size_t)e.H * e.vdim > v) v = (size_t)e.H * e.vdim;
                }
            if (cudaMalloc(&kexp, k * es * m.max_context) != cudaSuccess || cudaMalloc(&vexp, v * es * m.max_context) != cudaSuccess) {
                cudaGetLastError();
                if (kexp) cudaFree(kexp);
                kexp = vexp = nullptr;
                return set_error(JB_ERR_NOMEM, "decoder: expanded keys and values of %d positions", m.max_context);
            }
        }
        DenseGemm e = product(a);
        e.kind = kind; e.W = w.w_ukv; e.M = d.H * (d.dim + d.vdim); e.K = d.r; e.N = start + N; e.x = kv.key_ptr(l, 0); e.ldx = d.kd; e.nseg = 2;
        e.seg[0] = OutSeg{kexp, d.H * d.dim, d.H * d.dim, 0, 0};
        e.seg[1] = OutSeg{vexp, d.H * d.vdim, d.H * d.vdim, 0, 0};
        DCHK(launch_dense_gemm(e, st));
        AttnCall c;
        c.out = a.att; c.q = a.q; c.k = kexp; c.v = vexp; c.kv_kind = kind; c.n_heads = c.n_kv = d.H; c.hd = c.chd = qd; c.vhd = d.vdim;
        c.ldq = d.H * qd; c.ldo = pad8(d.H * d.vdim); c.ldk = d.H * d.dim; c.ldv = d.H * d.vdim; c.scale = w.scale; c.max_seq = m.max_context;
        c.k2 = (const char*)kv.key_ptr(l, 0) + (size_t)d.r8 * es; c.hd2 = d.rot; c.ldk2 = d.kd; c.gate = a.z + d.off_g; c.ldg = d.ldz;
        c.causal_start = start; c.batch = N; c.n_splits = 1;
        return launch_attention_bf16(c, st);
    }
    DenseGemm k;
    k.kind = kind; k.W = w.w_uk_t; k.M = d.r; k.K = d.dim; k.N = N; k.x = a.qu; k.ldx = d.H * d8; k.n_groups = d.H; k.x_step = d8; k.y_step = d.kd;
    k.seg[0] = OutSeg{a.q, d.H * d.kd, d.r, 0, 0};
    DCHK(launch_dense_gemm(k, st));
    AttnCall c = latent_call(l, a);
    c.gate = a.z + d.off_g; c.ldg = d.ldz; c.causal_start = start; c.batch = N; c.scratch = a.records; c.n_splits = attention_latent_applies(c) ? 0 : 1;
    DCHK(launch_attention_latent(c, st));
    DenseGemm v;
    v.kind = kind; v.W = (const char*)w.w_ukv + (size_t)d.H * d.dim * d.r8 * es; v.M = d.vdim; v.K = d.r; v.N = N; v.x = a.lat; v.ldx = d.H * d.r8; v.n_groups = d.H; v.x_step = d.r8;
    v.y_step = d.vdim; v.seg[0] = OutSeg{a.att, pad8(d.H * d.vdim), d.vdim, 0, 0};
    return launch_dense_gemm(v, st);
}

int LayerDecoder::enqueue_step(int n_splits, cudaStream_t st) {
    const long long l0 = jllm_b200_launch_count();
    const Acts& a = one;
    const int* d_pos = state;
    int cur = 0;                                  // x[cur]: residual before the pending exit
    const float *post_w = nullptr, *post_b = nullptr, *ls = nullptr;
    bool first = true;
    auto norm = [&](const float* w, const float* b) {
        NormStep n = entry(a, w, b);
        if (first) { first = false; n.tokens = state + 1; n.embed = m.embed; n.x_out = a.x[cur]; }
        else { n.x = a.x[cur]; n.y = a.y; n.post_w = post_w; n.post_b = post_b; n.ls = ls; n.x_out = a.x[cur ^ 1]; cur ^= 1; }
        return n;
    };
    for (int l = 0; l < m.n_layers; ++l) {
        const jllm_b200_layer_spec& w = layers[l];
        if (m.parallel) {
            DenseGemv g;
            g.mode = GEMV_PAIR; g.kind = kind; g.W = w.w_in; g.K = m.width; g.norm = norm(w.norm1_w, w.norm1_b); g.norm.h = nullptr;
            g.nseg = in_segments(g.seg, w, a, g.M);
            DCHK(launch_dense_gemv(g, st));
            if (w.mixer == MIX_LATENT) DCHK(latent_step(l, a, n_splits, st));
            else                       DCHK(launch_mlstm(mlstm_call(l, a), 1, 0, d_pos, st));
            DenseGemv o;
            o.mode = w.mlp_dim > 0 ? GEMV_TWO : GEMV_PLAIN; o.kind = kind; o.W = w.w_out; o.M = m.width; o.K = w.n_heads * w.v_dim; o.x = a.att; o.x2 = a.a; o.K2 = w.mlp_dim;
            o.ls = w.ls1; o.ls2 = w.ls2; o.seg[0] = OutSeg{a.y, pad8(m.width), m.width, 1, 0};
            DCHK(launch_dense_gemv(o, st));
            ls = w.mlp_dim > 0 ? nullptr : w.ls1;        // the plain product leaves the factor to the residual step
            continue;
        }
        DenseGemv g;
        g.mode = GEMV_NORM; g.kind = kind; g.W = w.w_qkv; g.K = m.width; g.d_pos = d_pos;
        g.norm = norm(w.norm1_w, w.norm1_b); g.norm.h = nullptr;
        qkv_segments(g, w, a.q, kv.key_ptr(l, 0), kv.val_ptr(l, 0), 1);
        DCHK(launch_dense_gemv(g, st));
        AttnCall c = attention_call(l, a);
        c.d_pos = d_pos; c.n_splits = n_splits;
        DCHK(launch_attention_float(c, st));
        DenseGemv o;
        o.kind = kind; o.W = w.w_o; o.M = m.width; o.K = w.n_heads * w.v_dim; o.x = a.att; o.seg[0] = OutSeg{a.y, pad8(m.width), m.width, 1, 0};
        DCHK(launch_dense_gemv(o, st));
        post_w = w.norm1b_w; post_b = w.norm1b_b;
        if (w.n_experts <= 0) continue;
        DenseGemv r;
        r.mode = GEMV_NORM; r.kind = kind; r.W = w.w_router; r.M = w.n_experts; r.K = m.width; r.norm = norm(w.norm2_w, w.norm2_b);
        r.seg[0] = OutSeg{a.z, w.n_experts, w.n_experts, 1, 0};
        DCHK(launch_dense_gemv(r, st));
        DenseGemv u;
        u.mode = GEMV_MOE_UP; u.kind = kind; u.W = w.w_gate; u.W_up = w.w_up; u.M = w.expert_dim; u.K = m.width; u.x = a.h; u.route = route(w); u.z = a.z;
        u.ids = a.ids; u.wts = a.wts; u.seg[0] = OutSeg{a.a, pad8(w.expert_dim), w.expert_dim, 0, 0};
        DCHK(launch_dense_gemv(u, st));
        DenseGemv d;
        d.mode = GEMV_MOE_DOWN; d.kind = kind; d.W = w.w_down; d.M = m.width; d.K = w.expert_dim; d.x = a.a; d.route = route(w); d.ids = a.ids; d.wts = a.wts;
        d.seg[0] = OutSeg{a.y, pad8(m.width), m.width, 1, 0};
        DCHK(launch_dense_gemv(d, st));
        post_w = w.norm2b_w; post_b = w.norm2b_b;
    }
    DenseGemv f;
    f.mode = GEMV_NORM; f.kind = kind; f.W = m.head ? m.head : m.embed; f.M = m.vocab_size; f.K = m.width; f.norm = norm(m.final_w, m.final_b); f.norm.h = nullptr;
    f.softcap = m.logit_softcap; f.seg[0] = OutSeg{logits, m.vocab_size, m.vocab_size, 1, 0};
    DCHK(launch_dense_gemv(f, st));
    DCHK(launch_argmax_advance(this, st));
    kernels_per_step = (int)(jllm_b200_launch_count() - l0);
    return JB_OK;
}

int LayerDecoder::reserve_chunk(int tokens, cudaStream_t st) {
    if (tokens <= pf_cap) return JB_OK;
    if (many.slab) { JB_CUDA(cudaDeviceSynchronize()); cudaFree(many.slab); many = Acts(); pf_cap = 0; }
    DCHK(alloc_acts(many, tokens, true, st));
    pf_cap = tokens;
    return JB_OK;
}

int LayerDecoder::enqueue_chunk(const int* dev_tokens, int N, int start, cudaStream_t st) {
    const Acts& a = many;
    int cur = 0;
    NormStep exit;                                // exit of the sublayer before: y (or expert outputs) and its norm
    bool first = true;
    auto norm = [&](const float* w, const float* b) {
        NormStep n = exit;
        const NormStep e = entry(a, w, b);
        n.W = e.W; n.eps = e.eps; n.mult = e.mult; n.rms = e.rms; n.next_w = w; n.next_b = b; n.h = a.h;
        if (first) { n = e; n.tokens = dev_tokens; n.embed = m.embed; n.x_out = a.x[cur]; first = false; }
        else { n.x = a.x[cur]; n.x_out = a.x[cur ^ 1]; cur ^= 1; }
        return n;
    };
    for (int l = 0; l < m.n_layers; ++l) {
        const jllm_b200_layer_spec& w = layers[l];
        DCHK(launch_norm_rows(norm(w.norm1_w, w.norm1_b), kind, N, st));
        if (m.parallel) {
            DenseGemm g = product(a);
            g.kind = kind; g.W = w.w_in; g.K = m.width; g.N = N; g.x = a.h;
            g.nseg = in_segments(g.seg, w, a, g.M);
            DCHK(launch_dense_gemm(g, st));
            if (w.mixer == MIX_LATENT) DCHK(latent_chunk(l, a, N, start, st));
            else                       DCHK(launch_mlstm(mlstm_call(l, a), N, start, nullptr, st));
            DenseGemm o = product(a);
            o.kind = kind; o.W = w.w_out; o.M = m.width; o.K = w.n_heads * w.v_dim; o.N = N; o.x = a.att; o.ldw = pad8(o.K) + pad8(w.mlp_dim);
            o.seg[0] = OutSeg{a.y, pad8(m.width), m.width, 1, 0};
            DCHK(launch_dense_gemm(o, st));
            exit = NormStep(); exit.y = a.y; exit.ls = w.ls1;
            if (w.mlp_dim > 0) {
                o.W = (const char*)w.w_out + (size_t)pad8(o.K) * elem_bytes(kind); o.K = w.mlp_dim; o.x = a.a; o.seg[0].y = a.y2;
                DCHK(launch_dense_gemm(o, st));
                exit.y2 = a.y2; exit.ls2 = w.ls2;
            }
            continue;
        }
        DenseGemm g = product(a);
        g.kind = kind; g.W = w.w_qkv; g.K = m.width; g.N = N; g.x = a.h;
        qkv_segments(g, w, a.q, kv.key_ptr(l, start), kv.val_ptr(l, start), 0);
        DCHK(launch_dense_gemm(g, st));
        AttnCall c = attention_call(l, a);
        c.causal_start = start; c.batch = N; c.n_splits = 1;
        DCHK(launch_attention_float(c, st));
        DenseGemm o = product(a);
        o.kind = kind; o.W = w.w_o; o.M = m.width; o.K = w.n_heads * w.v_dim; o.N = N; o.x = a.att; o.seg[0] = OutSeg{a.y, pad8(m.width), m.width, 1, 0};
        DCHK(launch_dense_gemm(o, st));
        exit = NormStep(); exit.y = a.y; exit.post_w = w.norm1b_w; exit.post_b = w.norm1b_b;
        if (w.n_experts <= 0) continue;
        DCHK(launch_norm_rows(norm(w.norm2_w, w.norm2_b), kind, N, st));
        const MoeRoute r = route(w);
        JB_CUDA(cudaMemsetAsync(a.counts, 0, (size_t)w.n_experts * sizeof(int), st));
        DenseGemm z = product(a);
        z.kind = kind; z.W = w.w_router; z.M = w.n_experts; z.K = m.width; z.N = N; z.x = a.h; z.seg[0] = OutSeg{a.z, w.n_experts, w.n_experts, 1, 0};
        DCHK(launch_dense_gemm(z, st));
        DCHK(launch_moe_topk(a.z, r, N, a.ids, a.wts, a.counts, a.rank, st));
        DCHK(launch_moe_permute(a.h, a.hp, kind, m.width, r, N, a.ids, a.rank, a.counts, a.slots, a.off, st));
        DenseGemm u;
        u.kind = kind; u.W = w.w_gate; u.W_up = w.w_up; u.swiglu = 1; u.M = w.expert_dim; u.K = m.width; u.N = N * w.top; u.x = a.hp; u.off = a.off; u.n_groups = w.n_experts;
        u.seg[0] = OutSeg{a.a, pad8(w.expert_dim), w.expert_dim, 0, 0};
        DCHK(launch_dense_gemm(u, st));
        DenseGemm d;
        d.kind = kind; d.W = w.w_down; d.M = m.width; d.K = w.expert_dim; d.N = N * w.top; d.x = a.a; d.off = a.off; d.n_groups = w.n_experts;
        d.seg[0] = OutSeg{a.ye, pad8(m.width), m.width, 0, 0};
        DCHK(launch_dense_gemm(d, st));
        exit = NormStep(); exit.y_exp = a.ye; exit.slots = a.slots; exit.wts = a.wts; exit.top = w.top; exit.post_w = w.norm2b_w; exit.post_b = w.norm2b_b;
    }
    pending = exit; last_x = cur;
    return JB_OK;
}

int LayerDecoder::enqueue_rows(const int* rows, int n, float* out, cudaStream_t st) {
    const Acts& a = many;
    JB_CUDA(cudaMemcpyAsync(a.rows, rows, (size_t)n * sizeof(int), cudaMemcpyHostToDevice, st));
    NormStep f = pending;
    f.W = m.width; f.eps = m.eps; f.mult = m.residual_mult; f.rms = m.rms_norm; f.next_w = m.final_w; f.next_b = m.final_b; f.h = a.h; f.x = a.x[last_x]; f.row_index = a.rows;
    DCHK(launch_norm_rows(f, kind, n, st));
    DenseGemm g;
    g.kind = kind; g.early = true; g.W = m.head ? m.head : m.embed; g.M = m.vocab_size; g.K = m.width; g.N = n; g.x = a.h; g.softcap = m.logit_softcap;
    g.seg[0] = OutSeg{out, m.vocab_size, m.vocab_size, 1, 0};
    return launch_dense_gemm(g, st);
}

int check_parallel_layer(const jllm_b200_layered_desc& m, int l) {
    const jllm_b200_layer_spec& w = m.layers[l];
    if (w.n_heads <= 0 || w.head_dim <= 0 || w.v_dim <= 0 || w.mlp_dim < 0) return set_error(JB_ERR_ARG, "decoder: layer %d has %d heads of %d / %d", l, w.n_heads, w.head_dim, w.v_dim);
    if (!w.w_in || !w.w_out || !w.norm1_w) return set_error(JB_ERR_PTR, "decoder: layer %d lacks a tensor", l);
    if (w.mixer == MIX_LATENT) {
        if (w.q_rank <= 0 || w.kv_rank <= 0 || w.rot_dim <= 0 || w.rot_dim % 2 || w.rot_dims <= 0 || w.rot_dims % 2 || w.rot_dims > w.rot_dim || !(w.rot_base > 0.0))
            return set_error(JB_ERR_ARG, "decoder: layer %d has latents of %d and %d, %d of %d rotated", l, w.q_rank, w.kv_rank, w.rot_dims, w.rot_dim);
        if (pad8(w.kv_rank) + pad8(w.rot_dim) > 1280) return set_error(JB_ERR_LIMIT, "decoder: layer %d has latent rows of %d elements", l, pad8(w.kv_rank) + pad8(w.rot_dim));
        if (w.n_heads > DT_HEADS) return set_error(JB_ERR_LIMIT, "decoder: layer %d has %d heads", l, w.n_heads);
        if (!w.w_uq || !w.w_ukv || !w.w_uk_t || !w.dq_norm || !w.dkv_norm) return set_error(JB_ERR_PTR, "decoder: layer %d lacks a latent tensor", l);
    } else if (w.mixer == MIX_MLSTM) {
        if (!(w.gate_cap > 0.f) || w.head_dim > 2048 || w.v_dim > 2048) return set_error(JB_ERR_ARG, "decoder: layer %d: memory of %d x %d, gate cap %g", l, w.head_dim, w.v_dim, w.gate_cap);
        if (!w.gate_bias || !w.head_norm) return set_error(JB_ERR_PTR, "decoder: layer %d lacks a memory tensor", l);
    } else {
        return set_error(JB_ERR_ARG, "decoder: layer %d: mixer %d in a parallel model", l, w.mixer);
    }
    return JB_OK;
}
int check_layer(const jllm_b200_layered_desc& m, int l) {
    const jllm_b200_layer_spec& w = m.layers[l];
    if (m.parallel) return check_parallel_layer(m, l);
    if (w.mixer != MIX_ATTENTION) return set_error(JB_ERR_ARG, "decoder: layer %d: mixer %d in a sequential model", l, w.mixer);
    if (w.n_heads <= 0 || w.n_kv_heads <= 0 || w.n_heads % w.n_kv_heads || w.head_dim <= 0 || w.head_dim > 512 || w.v_dim <= 0 || w.v_dim > 512)
        return set_error(JB_ERR_ARG, "decoder: layer %d has %d query and %d KV heads of %d / %d", l, w.n_heads, w.n_kv_heads, w.head_dim, w.v_dim);
    if (w.kv_from >= 0) {
        if (w.kv_from >= l) return set_error(JB_ERR_ARG, "decoder: layer %d takes its keys from layer %d", l, w.kv_from);
        const jllm_b200_layer_spec& s = m.layers[w.kv_from];
        if (s.kv_from >= 0 || s.n_kv_heads != w.n_kv_heads || s.head_dim != w.head_dim || s.v_dim != w.v_dim)
            return set_error(JB_ERR_ARG, "decoder: layer %d cannot use the keys of layer %d", l, w.kv_from);
    }
    if (!w.w_qkv || !w.w_o || !w.norm1_w || !w.norm1_b || !w.norm1b_w || !w.norm1b_b) return set_error(JB_ERR_PTR, "decoder: layer %d lacks a mixer tensor", l);
    if (w.n_experts > 0) {
        const int groups = w.n_groups > 1 ? w.n_groups : 1, keep = groups > 1 ? w.keep_groups : 1;
        if (w.n_experts > MOE_MAX_EXPERTS || w.n_experts % groups || keep < 1 || keep > groups || w.top < 1 || w.top > MOE_MAX_TOP || w.top > keep * (w.n_experts / groups) || w.expert_dim <= 0)
            return set_error(JB_ERR_LIMIT, "decoder: layer %d routes to %d of %d experts (%d of %d groups)", l, w.top, w.n_experts, keep, groups);
        if (!w.w_router || !w.w_gate || !w.w_up || !w.w_down || !w.norm2_w || !w.norm2_b || !w.norm2b_w || !w.norm2b_b)
            return set_error(JB_ERR_PTR, "decoder: layer %d lacks an expert tensor", l);
    }
    return JB_OK;
}

}  // namespace

extern "C" jllm_b200_decoder* jllm_b200_decoder_create_layered(const jllm_b200_layered_desc* model, int flags) {
    if (!model || !model->layers || model->n_layers <= 0 || model->width <= 0 || model->vocab_size <= 0 || model->max_context <= 0) { set_error(JB_ERR_ARG, "decoder: empty model description"); return nullptr; }
    if (model->dtype != EK_BF16 && model->dtype != EK_F32) { set_error(JB_ERR_TYPE, "decoder: element kind %d", model->dtype); return nullptr; }
    if (!model->embed || !model->final_w || (!model->rms_norm && !model->final_b)) { set_error(JB_ERR_PTR, "decoder: null embedding or final norm"); return nullptr; }
    for (int l = 0; l < model->n_layers; ++l) if (check_layer(*model, l)) return nullptr;
    if (!ctx()) return nullptr;
    LayerDecoder* d = new (std::nothrow) LayerDecoder();
    if (!d) return nullptr;
    d->m = *model;
    d->layers.assign(model->layers, model->layers + model->n_layers);
    d->m.layers = d->layers.data();
    d->kind = model->dtype;
    if (!(d->m.embed_scale > 0.f)) d->m.embed_scale = 1.f;
    d->use_graph = (flags & 2) != 0; d->batched_prefill = (flags & 16) != 0;
    std::vector<int> kw, vw;
    std::vector<int64_t> states;
    int vmax = 0;
    auto grow = [](int& a, int b) { if (b > a) a = b; };
    d->max_e = d->max_top = d->max_ff = 1;
    for (int l = 0; l < model->n_layers; ++l) {
        const jllm_b200_layer_spec& w = d->layers[l];
        d->rotation_of.push_back(-1);
        states.push_back(0);
        if (model->parallel) {
            d->source.push_back(l);
            vw.push_back(0);
            grow(d->max_v, w.n_heads * w.v_dim); grow(d->max_heads, w.n_heads); grow(d->max_ff, w.mlp_dim);
            if (w.mixer == MIX_LATENT) {
                const LatentDims n(w);
                kw.push_back(n.kd);
                grow(d->max_q, n.H * n.kd); grow(d->max_q, n.H * (n.dim + n.rot)); grow(d->max_z, n.ldz); grow(d->max_qn, pad8(n.q_rank)); grow(d->max_qu, n.H * pad8(n.dim)); grow(d->max_lat, n.H * n.r8);
                if (attn_latent_records(n.H, n.r8) > d->max_rec) d->max_rec = attn_latent_records(n.H, n.r8);
                if ((d->rotation_of[l] = d->add_rotation(w.rot_dim / 2, w.rot_dims, w.rot_base)) < 0) { jllm_b200_decoder_destroy(d); return nullptr; }
            } else {
                const MlstmDims n(w);
                kw.push_back(0);
                states.back() = (int64_t)mlstm_state_floats(n.H, n.dim, n.vdim);
                d->recurrent = true;
                grow(d->max_z, n.ldz); grow(d->max_proj, n.ld); grow(d->max_raw, n.H * n.vdim);
            }
            continue;
        }
        d->source.push_back(w.kv_from >= 0 ? w.kv_from : l);
        kw.push_back(w.n_kv_heads * w.head_dim); vw.push_back(w.n_kv_heads * w.v_dim);
        grow(d->max_q, w.n_heads * w.head_dim); grow(d->max_v, w.n_heads * w.v_dim); grow(d->max_heads, w.n_heads);
        if (w.n_experts > 0) { grow(d->max_e, w.n_experts); grow(d->max_top, w.top); grow(d->max_ff, w.expert_dim); }
    }
    d->vocab = d->vocab_full = model->vocab_size; d->max_context = model->max_context;
    if (!d->kv.init(model->n_layers, kw.data(), vw.data(), d->source.data(), model->max_context, elem_bytes(d->kind), states.data())) {
        set_error(JB_ERR_NOMEM, "decoder: KV cache of %d positions", model->max_context); jllm_b200_decoder_destroy(d); return nullptr;
    }
    // scratch that must exist before any graph capture
    for (const auto& w : d->layers) grow(vmax, w.v_dim);
    if (d->alloc_acts(d->one, 1, false, cudaStreamLegacy) || d->session_alloc() || !splitk_buffer((size_t)d->max_heads * 64 * (vmax + 2), true)) { jllm_b200_decoder_destroy(d); return nullptr; }
    return d;
}
