// dense.cuh — products with dense weights (bf16 or fp32, row-major [out][in], rows padded to a multiple of 8 elements,
// zero-filled): the decode family for one token (dense_gemv.cu), the tensor-core product for many (dense_tc.cu, bf16) and a
// CUDA-core product in true fp32 (dense_simt.cu).
#pragma once
#include "latent.cuh"
#include <functional>
#include "moe.cuh"

namespace jb {

// Consecutive output rows of a product that go to one place: y[token * ld + row], fp32 or the activation type.
// pair: what becomes of two adjacent rows (2 j, 2 j + 1).  PAIR_SILU / PAIR_GELU: gate and up rows interleaved, the output row j
// is act(gate) * up.  PAIR_ROT: the two parts of a rotated pair, turned by the angle of the token's position and of pair
// j mod half (rot: (cos, sin) tables [position][half]); they stay at their rows.  Pair segments start at an even row.
// blk > 0: output row r lies at (r / blk) * blk_ld + r % blk (heads that sit apart).
enum PairKind { PAIR_NONE = 0, PAIR_SILU = 1, PAIR_GELU = 2, PAIR_ROT = 3 };
struct OutSeg {
    void* y = nullptr; long long ld = 0; int rows = 0; int f32 = 0; int at_pos = 0;   // at_pos: decode only, y += *d_pos * ld
    int pair = PAIR_NONE; const float2* rot = nullptr; int half = 0;
    int blk = 0, blk_ld = 0;
};
constexpr int MAX_SEG = 3;

// ── decode: one token ──
enum GemvMode {
    GEMV_NORM = 0,       // input: the residual step of layernorm.cuh (its h); CTA 0 stores x' and, when norm.h is set, h
    GEMV_PLAIN = 1,      // input: vector x of the activation type, pad8(K) elements
    GEMV_MOE_UP = 2,     // input x; routes the token from z, then out[k][f] = silu(gate row) * up row of expert ids[k], k < top, f < M; CTA 0 stores ids and wts
    GEMV_MOE_DOWN = 3,   // input x = [top][pad8(K)]; y[row] = sum_k wts[k] * (W[ids[k]][row] . x[k])
    GEMV_TWO = 4,        // inputs x (K) and x2 (K2), rows of W = [pad8(K) | pad8(K2)]; y[row] = ls[row] * (W[row] . x) + ls2[row] * (W[row] . x2)
    GEMV_PAIR = 5,       // GEMV_NORM whose work items are pairs of adjacent rows: the mode of products with pair segments
};
struct DenseGemv {
    int mode = GEMV_PLAIN, kind = EK_BF16;
    const void* W = nullptr; const void* W_up = nullptr;
    int M = 0, K = 0;
    OutSeg seg[MAX_SEG]; int nseg = 1;
    float softcap = 0.f;                     // y := softcap * tanh(y / softcap), fp32 outputs
    const int* d_pos = nullptr;
    const void* x = nullptr;
    const void* x2 = nullptr; int K2 = 0;
    const float* ls = nullptr; const float* ls2 = nullptr;      // GEMV_TWO: per output row; null: 1
    bool late = false;                       // GEMV_PLAIN: the kernel in front may still be writing W (the other modes, and a model's weights, do not wait for it)
    LatentRows side;                         // side.z set (GEMV_PAIR): one more CTA stores the token's latent row
    NormStep norm;
    MoeRoute route; const float* z = nullptr; int* ids = nullptr; float* wts = nullptr;
};
int launch_dense_gemv(const DenseGemv& a, cudaStream_t st);

// ── many tokens ──
// y[t][r] = sum_k W[r][k] * x[t][k].  With groups (experts): W holds n_groups matrices of M rows one after the other and
// group g multiplies token rows [off[g], off[g + 1]) (off on the device).  swiglu: W is the gate, W_up the up matrix, and
// the output is silu(gate) * up.  Without off, n_groups > 1 are blocks of the inner and outer dimensions (heads): group g
// multiplies columns g * x_step .. of every token row and its output goes to y + g * y_step.
struct DenseGemm {
    int kind = EK_BF16;
    const void* W = nullptr; const void* W_up = nullptr;
    int M = 0, K = 0, N = 0;                 // rows (per group), inner size, token rows in all
    const void* x = nullptr;                 // [N][ldx]
    int ldw = 0, ldx = 0;                    // row strides, multiples of 8; 0: pad8(K)
    int start = 0;                           // position of token row 0 (rotated segments)
    int x_step = 0, y_step = 0;              // bf16: x_step is a multiple of 8
    OutSeg seg[MAX_SEG]; int nseg = 1;
    float softcap = 0.f; int swiglu = 0;
    const int* off = nullptr; int n_groups = 1;
    bool early = false;                      // W was complete before the kernel in front of this one started (a model's weights)
    float* part = nullptr; size_t part_floats = 0;      // optional workspace of K ranges (gemm_pair_part_floats), one per stream
};
constexpr int GP_MIN_TOKENS = 128;
bool gemm_pair_applies(const DenseGemm& a);
bool gemm_pair_one_round(const DenseGemm& a);
size_t gemm_pair_part_floats();
int launch_gemm_pair(const DenseGemm& a, cudaStream_t st, const std::function<int()>& behind = nullptr);       // fp16 (EK_F16) or bf16 operands, pairs of CTAs (gemm_pair.cu)
int launch_dense_gemm(const DenseGemm& a, cudaStream_t st);      // bf16: tensor cores; fp32: CUDA cores; one token: the decode product
int launch_dense_gemm_tc(const DenseGemm& a, cudaStream_t st);
int launch_dense_gemm_simt(const DenseGemm& a, cudaStream_t st);

#ifdef __CUDACC__
// 16 bytes of weights times 16 bytes of input
__device__ __forceinline__ float dot16(uint4 w, uint4 h, float acc, float) {
    acc = fmaf(__uint_as_float(w.x), __uint_as_float(h.x), acc); acc = fmaf(__uint_as_float(w.y), __uint_as_float(h.y), acc);
    acc = fmaf(__uint_as_float(w.z), __uint_as_float(h.z), acc); return fmaf(__uint_as_float(w.w), __uint_as_float(h.w), acc);
}
__device__ __forceinline__ float dot16(uint4 w, uint4 h, float acc, __nv_bfloat16) {
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w}, hh[4] = {h.x, h.y, h.z, h.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        acc = fmaf(__uint_as_float(ww[i] << 16), __uint_as_float(hh[i] << 16), acc);
        acc = fmaf(__uint_as_float(ww[i] & 0xFFFF0000u), __uint_as_float(hh[i] & 0xFFFF0000u), acc);
    }
    return acc;
}
__device__ __forceinline__ float silu_f(float g) { return g / (1.0f + expf(-g)); }
// 0.5 z (1 + tanh u) = z / (1 + e^(-2 u)) with u = sqrt(2 / pi) (z + 0.044715 z^3)
__device__ __forceinline__ float gelu_tanh_f(float z) { return __fdividef(z, 1.0f + expf(-1.5957691216057308f * fmaf(0.044715f * z * z, z, z))); }
__device__ __forceinline__ float pair_act(int kind, float g) { return kind == PAIR_SILU ? silu_f(g) : gelu_tanh_f(g); }
// (u, v) turned by the angle whose cosine and sine are cs
__device__ __forceinline__ float2 rotate_pair(float u, float v, float2 cs) { return make_float2(u * cs.x - v * cs.y, v * cs.x + u * cs.y); }
__device__ __forceinline__ int seg_place(const OutSeg& g, int r) { return g.blk > 0 ? (r / g.blk) * g.blk_ld + r % g.blk : r; }
template <typename T>
__device__ __forceinline__ void store_as(void* y, long long o, int f32, float v) {
    if (f32) reinterpret_cast<float*>(y)[o] = v;
    else     reinterpret_cast<T*>(y)[o] = from_f32<T>(v);
}
// y_off: elements added to the place (the output of a group of heads)
template <typename T>
__device__ __forceinline__ void store_seg(const OutSeg* seg, int nseg, float softcap, const int* d_pos, long long token, int row, float v, long long y_off = 0) {
    int s = 0;
    while (s + 1 < nseg && row >= seg[s].rows) { row -= seg[s].rows; ++s; }
    if (softcap > 0.f) v = softcap * tanhf(v / softcap);
    store_as<T>(seg[s].y, y_off + (token + (seg[s].at_pos ? *d_pos : 0)) * seg[s].ld + seg_place(seg[s], row), seg[s].f32, v);
}
// rows `row` (even) and row + 1 of `M`; pos: position of the token
template <typename T>
__device__ __forceinline__ void store_rows2(const OutSeg* seg, int nseg, float softcap, const int* d_pos, long long token, int pos, int row, int M, float v, float v2,
                                            long long y_off = 0) {
    int s = 0, r = row;
    while (s + 1 < nseg && r >= seg[s].rows) { r -= seg[s].rows; ++s; }
    const OutSeg& g = seg[s];
    if (g.pair == PAIR_NONE) {
        store_seg<T>(seg, nseg, softcap, d_pos, token, row, v, y_off);
        if (row + 1 < M) store_seg<T>(seg, nseg, softcap, d_pos, token, row + 1, v2, y_off);
        return;
    }
    const long long at = y_off + (token + (g.at_pos ? *d_pos : 0)) * g.ld;
    if (g.pair == PAIR_ROT) {
        const float2 o = rotate_pair(v, v2, g.rot[(size_t)pos * g.half + (r >> 1) % g.half]);
        store_as<T>(g.y, at + seg_place(g, r), g.f32, o.x);
        store_as<T>(g.y, at + seg_place(g, r + 1), g.f32, o.y);
    } else {
        store_as<T>(g.y, at + seg_place(g, r >> 1), g.f32, pair_act(g.pair, v) * v2);
    }
}
// The drain of a tensor-core tile: lanes of tensor memory are rows, so 32 tokens of a warp's 32 rows go through 4 KB of shared memory
// ([token][row], written and read without bank conflicts) and come back as four adjacent rows of one token per lane, stored together.
// (Stored from the accumulator's lanes, a value at a time with segment, bounds and pair cases around each, a column took 25
// instructions and a tile of 256 tokens 26 us, as long as its K loop at K = 6000.)
template <typename T>
__device__ __forceinline__ void store4_16(T* p, float4 v);
template <> __device__ __forceinline__ void store4_16<__nv_bfloat16>(__nv_bfloat16* p, float4 v) { store4(p, v); }
template <> __device__ __forceinline__ void store4_16<__half>(__half* p, float4 v) {
    const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
// The place of rows row .. row + 3 (row a multiple of four), found once per tile; for outputs that are rows4_aligned.  Lanes of a warp may
// lie in different segments, so neither finding a place nor storing leaves the warp converged: __syncwarp before the next tcgen05.ld.
template <typename T>
struct Rows4 {
    char* y; long long ld; const float2* rot; int kind, f32, half, pair0, row;      // kind: of the pair, -1: no such rows
    __device__ __forceinline__ Rows4(const OutSeg* seg, int nseg, int M, int r, long long y_off) : row(r) {
        const bool second = nseg > 1 && r >= seg[0].rows;
        r -= second ? seg[0].rows : 0;
        const bool third = second && nseg > 2 && r >= seg[1].rows;
        r -= third ? seg[1].rows : 0;
        const int s = (int)second + (int)third;
        kind = row < M ? seg[s].pair : -1;
        f32 = seg[s].f32; half = seg[s].half; rot = seg[s].rot; ld = seg[s].ld; pair0 = r >> 1;
        const long long at = y_off + seg_place(seg[s], kind == PAIR_SILU || kind == PAIR_GELU ? r >> 1 : r);
        y = reinterpret_cast<char*>(seg[s].y) + at * (f32 ? 4 : (int)sizeof(T));
    }
    // v[k]: tokens token + 4 k, the first n of which (k < n) exist; one case per call, so that the eight stores leave together
    __device__ __forceinline__ void store8(long long token, int pos, int n, float softcap, float4 (&v)[8]) const {
        if (kind < 0) return;
        const long long step = 4 * ld * (f32 ? 4 : (int)sizeof(T));
        char* p = y + token * ld * (f32 ? 4 : (int)sizeof(T));
        if (kind == PAIR_SILU || kind == PAIR_GELU) {
            #pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float a = pair_act(kind, v[k].x) * v[k].y, b = pair_act(kind, v[k].z) * v[k].w;
                const T t[2] = {from_f32<T>(a), from_f32<T>(b)};
                if (k < n) {
                    if (f32) *reinterpret_cast<float2*>(p + k * step) = make_float2(a, b);
                    else     *reinterpret_cast<uint32_t*>(p + k * step) = (uint32_t)*reinterpret_cast<const unsigned short*>(&t[0]) | (uint32_t)*reinterpret_cast<const unsigned short*>(&t[1]) << 16;
                }
            }
            return;
        }
        if (kind == PAIR_ROT) {
            const float2* c = rot + (size_t)pos * half;
            const int i = pair0 % half, j = (pair0 + 1) % half;
            #pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (k < n) {
                    const float2 a = rotate_pair(v[k].x, v[k].y, __ldg(c + i + 4 * k * half)), b = rotate_pair(v[k].z, v[k].w, __ldg(c + j + 4 * k * half));
                    v[k] = make_float4(a.x, a.y, b.x, b.y);
                }
            }
        } else if (softcap > 0.f) {
            #pragma unroll
            for (int k = 0; k < 8; ++k) {
                v[k].x = softcap * tanhf(v[k].x / softcap); v[k].y = softcap * tanhf(v[k].y / softcap);
                v[k].z = softcap * tanhf(v[k].z / softcap); v[k].w = softcap * tanhf(v[k].w / softcap);
            }
        }
        if (f32) {
            #pragma unroll
            for (int k = 0; k < 8; ++k) if (k < n) store4(reinterpret_cast<float*>(p + k * step), v[k]);
        } else {
            #pragma unroll
            for (int k = 0; k < 8; ++k) if (k < n) store4_16<T>(reinterpret_cast<T*>(p + k * step), v[k]);
        }
    }
};
// the same for outputs that are not
template <typename T>
__device__ __noinline__ void store_four(const OutSeg* seg, int nseg, float softcap, long long token, int pos, int row, int M, float4 v, long long y_off) {
    if (row < M) store_rows2<T>(seg, nseg, softcap, nullptr, token, pos, row, M, v.x, v.y, y_off);
    if (row + 2 < M) store_rows2<T>(seg, nseg, softcap, nullptr, token, pos, row + 2, M, v.z, v.w, y_off);
}
#endif
// Whether every group of four rows that starts at a multiple of four lies in one segment, whole and aligned for one store.
inline bool rows4_aligned(const OutSeg* seg, int nseg, int M, int y_step) {
    int rows = 0;
    for (int i = 0; i < nseg; ++i) {
        const OutSeg& g = seg[i];
        if (g.rows % 4 || g.ld % 4 || ((uintptr_t)g.y & 15) || (g.blk > 0 && (g.blk % 4 || g.blk_ld % 4)) || y_step % 4) return false;
        rows += g.rows;
    }
    return M % 4 == 0 && rows >= M;
}

}  // namespace jb
