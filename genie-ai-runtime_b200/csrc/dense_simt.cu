// dense_simt.cu — dense products over many tokens on the CUDA cores, in true fp32 (FFMA, no reduced-precision matrix mode): the 32-bit
// path of layer-list models.  64 (rows) x 32 (tokens) output tiles, 4 x 2 per thread, K tiles of 32; groups (experts) on grid.z.
//
// At the sizes of prompts in this format a launch has few CTAs, so a tile's chain of K tiles sets the time: the next K tile is
// requested as 16-byte loads before the present one is multiplied and stored into the other half of shared memory after it, one
// barrier per K tile.  A value is summed over k in ascending order.
#include "dense.cuh"

namespace jb {

constexpr int DS_M = 64, DS_N = 32, DS_K = 32, DS_THREADS = 256;

struct DsTile { float w[DS_K][DS_M + 4], x[DS_K][DS_N + 4]; };
template <bool GLU> struct DsUp { float u[DS_K][DS_M + 4]; };
template <> struct DsUp<false> {};

// four elements at k of a row, zero beyond K; vec: 16-byte aligned rows
__device__ __forceinline__ float4 ds_load(const float* row, bool in, int k, int K, bool vec) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!in || k >= K) return v;
    if (vec && k + 4 <= K) return load4(row + k);
    v.x = row[k];
    if (k + 1 < K) v.y = row[k + 1];
    if (k + 2 < K) v.z = row[k + 2];
    if (k + 3 < K) v.w = row[k + 3];
    return v;
}
template <int LD>
__device__ __forceinline__ void ds_put(float (*t)[LD], int k, int j, float4 v) { t[k][j] = v.x; t[k + 1][j] = v.y; t[k + 2][j] = v.z; t[k + 3][j] = v.w; }

template <bool GLU>
__global__ void __launch_bounds__(DS_THREADS) dense_simt_kernel(const __grid_constant__ DenseGemm a, bool vec) {
    pdl_wait();
    __shared__ __align__(16) DsTile tile[2];
    __shared__ __align__(16) DsUp<GLU> up[2];
    const int grp = blockIdx.z, t_lo = a.off ? a.off[grp] : 0, t_hi = a.off ? a.off[grp + 1] : a.N;
    const int r0 = blockIdx.x * DS_M, ldw = a.ldw > 0 ? a.ldw : pad8(a.K), ldx = a.ldx > 0 ? a.ldx : pad8(a.K);
    const float* W = reinterpret_cast<const float*>(a.W) + (size_t)grp * a.M * ldw;
    const float* V = GLU ? reinterpret_cast<const float*>(a.W_up) + (size_t)grp * a.M * ldw : nullptr;
    const float* x = reinterpret_cast<const float*>(a.x) + (size_t)grp * a.x_step;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;                      // thread: rows 4 tx .., tokens 2 ty ..
    const int lk = 4 * (threadIdx.x & 7), lj = threadIdx.x >> 3;                 // loads: row (or token) lj and row lj + 32, elements lk ..
    const bool in0 = r0 + lj < a.M, in1 = r0 + lj + 32 < a.M;
    const float *w0 = W + (size_t)(r0 + lj) * ldw, *w1 = w0 + (size_t)32 * ldw, *v0 = GLU ? V + (size_t)(r0 + lj) * ldw : nullptr, *v1 = GLU ? v0 + (size_t)32 * ldw : nullptr;
    for (int t0 = t_lo + blockIdx.y * DS_N; t0 < t_hi; t0 += gridDim.y * DS_N) {
    const bool inx = t0 + lj < t_hi;
    const float* xr = x + (size_t)(t0 + lj) * ldx;
    float4 f[3], h[2];
    auto fetch = [&](int k) {
        f[0] = ds_load(w0, in0, k + lk, a.K, vec); f[1] = ds_load(w1, in1, k + lk, a.K, vec); f[2] = ds_load(xr, inx, k + lk, a.K, vec);
        if (GLU) { h[0] = ds_load(v0, in0, k + lk, a.K, vec); h[1] = ds_load(v1, in1, k + lk, a.K, vec); }
    };
    auto put = [&](int b) {
        ds_put(tile[b].w, lk, lj, f[0]); ds_put(tile[b].w, lk, lj + 32, f[1]); ds_put(tile[b].x, lk, lj, f[2]);
        if constexpr (GLU) { ds_put(up[b].u, lk, lj, h[0]); ds_put(up[b].u, lk, lj + 32, h[1]); }
    };
    float acc[4][2] = {}, acu[4][2] = {};
    fetch(0);
    put(0);
    __syncthreads();
    for (int k0 = 0, b = 0; k0 < a.K; k0 += DS_K, b ^= 1) {
        const bool more = k0 + DS_K < a.K;
        if (more) fetch(k0 + DS_K);
        #pragma unroll
        for (int k = 0; k < DS_K; ++k) {
            const float4 w = load4(&tile[b].w[k][4 * tx]);
            const float2 v = *reinterpret_cast<const float2*>(&tile[b].x[k][2 * ty]);
            acc[0][0] = fmaf(w.x, v.x, acc[0][0]); acc[0][1] = fmaf(w.x, v.y, acc[0][1]); acc[1][0] = fmaf(w.y, v.x, acc[1][0]); acc[1][1] = fmaf(w.y, v.y, acc[1][1]);
            acc[2][0] = fmaf(w.z, v.x, acc[2][0]); acc[2][1] = fmaf(w.z, v.y, acc[2][1]); acc[3][0] = fmaf(w.w, v.x, acc[3][0]); acc[3][1] = fmaf(w.w, v.y, acc[3][1]);
            if constexpr (GLU) {
                const float4 u = load4(&up[b].u[k][4 * tx]);
                acu[0][0] = fmaf(u.x, v.x, acu[0][0]); acu[0][1] = fmaf(u.x, v.y, acu[0][1]); acu[1][0] = fmaf(u.y, v.x, acu[1][0]); acu[1][1] = fmaf(u.y, v.y, acu[1][1]);
                acu[2][0] = fmaf(u.z, v.x, acu[2][0]); acu[2][1] = fmaf(u.z, v.y, acu[2][1]); acu[3][0] = fmaf(u.w, v.x, acu[3][0]); acu[3][1] = fmaf(u.w, v.y, acu[3][1]);
            }
        }
        if (more) put(b ^ 1);
        __syncthreads();
    }
    #pragma unroll
    for (int j = 0; j < 2; ++j)
        #pragma unroll
        for (int i = 0; i < 4; i += 2) {
            const int r = r0 + 4 * tx + i, t = t0 + 2 * ty + j;
            if (r < a.M && t < t_hi)
                store_rows2<float>(a.seg, a.nseg, a.softcap, nullptr, t, a.start + t, r, a.M, GLU ? silu_f(acc[i][j]) * acu[i][j] : acc[i][j],
                                   GLU ? silu_f(acc[i + 1][j]) * acu[i + 1][j] : acc[i + 1][j], (long long)grp * a.y_step);
        }
    }
}

int launch_dense_gemm_simt(const DenseGemm& a, cudaStream_t st) {
    if (a.N <= 0 || a.M <= 0) return JB_OK;
    if (a.kind != EK_F32) return set_error(JB_ERR_TYPE, "dense fp32 gemm: element kind %d", a.kind);
    if (!a.W || !a.x || (a.swiglu && !a.W_up) || (a.n_groups > 1 && !a.off && !a.x_step)) return set_error(JB_ERR_PTR, "dense fp32 gemm: null pointer");
    const int tiles = (a.N + DS_N - 1) / DS_N;
    const dim3 grid((a.M + DS_M - 1) / DS_M, tiles < 65535 ? tiles : 65535, a.n_groups);
    const int ldw = a.ldw > 0 ? a.ldw : pad8(a.K), ldx = a.ldx > 0 ? a.ldx : pad8(a.K);
    const bool vec = !(((uintptr_t)a.W | (uintptr_t)a.x | (a.swiglu ? (uintptr_t)a.W_up : 0)) & 15) && ldw % 4 == 0 && ldx % 4 == 0 && a.x_step % 4 == 0;
    if ((a.N + 63) / 64 > 65535) return set_error(JB_ERR_LIMIT, "dense fp32 gemm: %d tokens", a.N);
    if (a.swiglu) JB_CUDA(launch_k(dense_simt_kernel<true>, grid, dim3(DS_THREADS), 0, st, pdl_enabled(), a, vec));
    else          JB_CUDA(launch_k(dense_simt_kernel<false>, grid, dim3(DS_THREADS), 0, st, pdl_enabled(), a, vec));
    count_launch();
    return JB_OK;
}
// One token (the logits after a prompt) is a product of the decode family: 151936 x 2560 in bf16 take 122 us there, the weights at the
// rate of memory, and 145 us in tiles of 16 tokens; the smallest tile of this file is 32 tokens wide.
static bool ds_one_token(const DenseGemm& a) {
    if (a.N != 1 || a.n_groups != 1 || a.off || a.swiglu || a.M <= 0 || a.K <= 0 || a.K % 8 || a.K > 8192 || (a.ldw > 0 && a.ldw != a.K) || (((uintptr_t)a.W | (uintptr_t)a.x) & 15)) return false;
    for (int i = 0; i < a.nseg; ++i) if (a.seg[i].pair != PAIR_NONE) return false;
    return a.W && a.x;
}
int launch_dense_gemm(const DenseGemm& a, cudaStream_t st) {
    if (ds_one_token(a)) {
        DenseGemv g;
        g.kind = a.kind; g.W = a.W; g.M = a.M; g.K = a.K; g.x = a.x; g.softcap = a.softcap; g.nseg = a.nseg; g.late = !a.early;
        for (int i = 0; i < a.nseg; ++i) g.seg[i] = a.seg[i];
        return launch_dense_gemv(g, st);
    }
    return a.kind == EK_F32 ? launch_dense_gemm_simt(a, st) : launch_dense_gemm_tc(a, st);
}

}  // namespace jb
