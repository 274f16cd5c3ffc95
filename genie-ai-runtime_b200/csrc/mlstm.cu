// mlstm.cu — the mLSTM recurrence token by token (decoding; prompts in fp32 and of sizes the chunk kernel does not hold), and the
// head norm and output gate of prompts.
//
// A cluster of CTAs per head, each with a slice of the value columns: all of them keep n, each its columns of S.  One token works
// on the state in global memory, several on a copy in shared memory.  For one token the cluster also exchanges the sums of
// squares, so the normed and gated output leaves the same kernel.
#include "mlstm.cuh"
#include <cooperative_groups.h>

namespace jb {

namespace cg = cooperative_groups;
constexpr int ML_THREADS = 256, ML_MAX_CLUSTER = 8, ML_MAX_DIM = 2048, ML_BATCH = 16, ML_EARLY = 16;

struct MlArgs { MlstmCall c; int n, start; const int* d_pos; int vs, in_smem, early; };      // vs: value columns per CTA

size_t mlstm_state_floats(int heads, int dim, int vdim) { return (size_t)heads * dim * pad8(vdim) + 2 * ((size_t)heads * dim + pad8(heads)); }

template <typename T, bool ONE>
__global__ void __launch_bounds__(ML_THREADS) mlstm_kernel(const MlArgs p) {
    extern __shared__ __align__(16) float ml_sm[];
    __shared__ float red[2 * ML_THREADS / 32], csum[ML_MAX_CLUSTER];
    const MlstmCall& c = p.c;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, h = blockIdx.y, rank = blockIdx.x, D = c.dim, vld = pad8(c.vdim);
    const int c0 = min(rank * p.vs, vld), vs = min(p.vs, vld - c0), cols4 = vs / 4;
    float* qs = ml_sm; float* ks = qs + pad8(D); float* ns = ks + pad8(D); float* po = ns + pad8(D);      // po: partial outputs [group][vs]
    float* Sg = c.state + ((size_t)h * D) * vld + c0;
    float* ng = c.state + (size_t)c.heads * D * vld + (size_t)h * D;
    float* mg = c.state + (size_t)c.heads * D * vld + (size_t)c.heads * D + h;
    const int groups = cols4 > 0 ? ML_THREADS / cols4 : 0, cg4 = cols4 > 0 ? tid % cols4 : 0, rg = cols4 > 0 ? tid / cols4 : 0;
    const bool mine = cols4 > 0 && rg < groups;
    // Inside a decode step the kernel in front of this one began after the state and the position were last written (p.early): both
    // are read while it still runs.
    if (!(ONE && p.early)) pdl_wait();
    const int start = p.d_pos ? *p.d_pos : p.start;
    const bool fresh = start == 0;
    float4 early[ONE ? ML_EARLY : 1];
    if (ONE) {
        #pragma unroll
        for (int u = 0; u < ML_EARLY; ++u) {
            const int d = rg + u * groups;
            early[ONE ? u : 0] = mine && !fresh && d < D ? load4(Sg + (size_t)d * vld + 4 * cg4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    for (int d = tid; d < D; d += ML_THREADS) ns[d] = fresh ? 0.f : ng[d];
    float m = fresh ? 0.f : *mg;
    if (ONE && p.early) pdl_wait();
    pdl_launch();
    float* S = Sg;
    int lds = vld;
    if (!ONE && p.in_smem) {
        S = po + 4 * ML_THREADS; lds = p.vs;
        if (mine) for (int d = rg; d < D; d += groups) store4(S + (size_t)d * lds + 4 * cg4, fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : load4(Sg + (size_t)d * vld + 4 * cg4));
    }
    cluster.sync();                                        // everyone runs and has read n and m
    for (int t = 0; t < p.n; ++t) {
        const T* row = reinterpret_cast<const T*>(c.proj) + (size_t)t * c.ld;
        const float li = mlstm_log_i(c, t, h), lf = mlstm_log_f(c, t, h);
        const float mn = fmaxf(lf + m, li), keep = expf(lf + m - mn), add = expf(li - mn);
        const bool blank = fresh && t == 0 && (ONE || !p.in_smem);       // the state in memory is an earlier sequence's
        m = mn;
        if (!ONE) __syncthreads();                         // the token before is done with shared memory
        const float qscale = 1.0f / sqrtf((float)D);
        float part = 0.f;
        for (int d = tid; d < D; d += ML_THREADS) {
            const float q = to_f32(row[c.off_q + h * D + d]) * qscale, k = add * to_f32(row[c.off_k + h * D + d]);
            const float n = fmaf(keep, ns[d], k);
            qs[d] = q; ks[d] = k; ns[d] = n;
            part = fmaf(n, q, part);
        }
        const float nq = block_sum<ML_THREADS>(part, red);
        if (mine) {
            float v[4];
            #pragma unroll
            for (int e = 0; e < 4; ++e) { const int d = c0 + 4 * cg4 + e; v[e] = d < c.vdim ? to_f32(row[c.off_v + h * c.vdim + d]) : 0.f; }
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int d0 = rg; d0 < D; d0 += ML_BATCH * groups) {         // a batch of rows is read before the first is written
                float4 s[ML_BATCH];
                #pragma unroll
                for (int u = 0; u < ML_BATCH; ++u) {
                    const int d = d0 + u * groups;
                    if (ONE && u < ML_EARLY && d0 == rg) s[u] = early[u];
                    else if (d < D && !blank) s[u] = load4(S + (size_t)d * lds + 4 * cg4);
                    else s[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                #pragma unroll
                for (int u = 0; u < ML_BATCH; ++u) {
                    const int d = d0 + u * groups;
                    if (d < D) {
                        const float k = ks[d], q = qs[d];
                        s[u].x = fmaf(keep, s[u].x, k * v[0]); s[u].y = fmaf(keep, s[u].y, k * v[1]); s[u].z = fmaf(keep, s[u].z, k * v[2]); s[u].w = fmaf(keep, s[u].w, k * v[3]);
                        store4(S + (size_t)d * lds + 4 * cg4, s[u]);
                        acc.x = fmaf(s[u].x, q, acc.x); acc.y = fmaf(s[u].y, q, acc.y); acc.z = fmaf(s[u].z, q, acc.z); acc.w = fmaf(s[u].w, q, acc.w);
                    }
                }
            }
            store4(po + (size_t)rg * vs + 4 * cg4, acc);
        }
        __syncthreads();
        const float inv = 1.0f / (fmaxf(fabsf(nq), expf(-m)) + 1e-6f);
        if (ONE) {
            float o[ML_MAX_DIM / ML_THREADS], sq = 0.f;
            #pragma unroll
            for (int u = 0; u < ML_MAX_DIM / ML_THREADS; ++u) {
                const int j = tid + u * ML_THREADS;
                o[u] = 0.f;
                if (j < vs) { for (int g = 0; g < groups; ++g) o[u] += po[(size_t)g * vs + j]; o[u] *= inv; sq = fmaf(o[u], o[u], sq); }
            }
            sq = block_sum<ML_THREADS>(sq, red + ML_THREADS / 32);
            if (tid < (int)cluster.num_blocks()) *cluster.map_shared_rank(&csum[rank], tid) = sq;
            cluster.sync();
            sq = 0.f;
            for (int r = 0; r < (int)cluster.num_blocks(); ++r) sq += csum[r];
            const float rs = 1.0f / sqrtf(sq / (float)c.vdim + c.eps);
            #pragma unroll
            for (int u = 0; u < ML_MAX_DIM / ML_THREADS; ++u) {
                const int j = tid + u * ML_THREADS, d = h * c.vdim + c0 + j;
                if (j < vs && c0 + j < c.vdim)
                    reinterpret_cast<T*>(c.out)[d] = from_f32<T>(o[u] * rs * c.norm_w[d] * (1.0f / (1.0f + expf(-to_f32(row[c.off_g + d])))));
            }
        } else {
            for (int j = tid; j < vs; j += ML_THREADS) {
                float o = 0.f;
                for (int g = 0; g < groups; ++g) o += po[(size_t)g * vs + j];
                if (c0 + j < c.vdim) c.raw[(size_t)t * c.heads * c.vdim + h * c.vdim + c0 + j] = o * inv;
            }
        }
    }
    if (!ONE && p.in_smem && mine)
        for (int d = rg; d < D; d += groups) store4(Sg + (size_t)d * vld + 4 * cg4, load4(S + (size_t)d * lds + 4 * cg4));
    if (rank == 0) {
        for (int d = tid; d < D; d += ML_THREADS) ng[d] = ns[d];
        if (tid == 0) *mg = m;
    }
}

// raw outputs -> over each head's root mean square, times the weight, times sigmoid(g): a warp per (token, head)
template <typename T>
__global__ void __launch_bounds__(256) mlstm_out_kernel(const MlstmCall c, int n, bool take_next, bool vec) {
    pdl_wait();
    pdl_launch();
    if (take_next) {                                       // the chunk kernel left the next n and m beside the old ones
        float* ns = c.state + (size_t)c.heads * c.dim * pad8(c.vdim);
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)c.heads * c.dim + c.heads; i += (size_t)gridDim.x * blockDim.x) ns[i] = ns[i + mlstm_next(c)];
    }
    const int lane = threadIdx.x & 31, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, t = w / c.heads, h = w - t * c.heads;
    if (t >= n) return;
    const float* o = c.raw + ((size_t)t * c.heads + h) * c.vdim;
    const T* g = reinterpret_cast<const T*>(c.proj) + (size_t)t * c.ld + c.off_g + h * c.vdim;
    T* out = reinterpret_cast<T*>(c.out) + (size_t)t * c.ldo + h * c.vdim;
    float sq = 0.f;
    if (vec) {                                             // fours of everything from whole boundaries
        const float* w4 = c.norm_w + h * c.vdim;
        for (int d = 4 * lane; d < c.vdim; d += 128) { const float4 v = load4(o + d); sq = fmaf(v.x, v.x, sq); sq = fmaf(v.y, v.y, sq); sq = fmaf(v.z, v.z, sq); sq = fmaf(v.w, v.w, sq); }
        const float rs = 1.0f / sqrtf(warp_sum(sq) / (float)c.vdim + c.eps);
        auto gated = [&](float v, float w, float z) { return __fdividef(v * rs * w, 1.0f + expf(-z)); };
        for (int d = 4 * lane; d < c.vdim; d += 128) {
            const float4 v = load4(o + d), w = load4(w4 + d), z = load4(g + d);
            store4(out + d, make_float4(gated(v.x, w.x, z.x), gated(v.y, w.y, z.y), gated(v.z, w.z, z.z), gated(v.w, w.w, z.w)));
        }
        return;
    }
    for (int d = lane; d < c.vdim; d += 32) sq = fmaf(o[d], o[d], sq);
    const float rs = 1.0f / sqrtf(warp_sum(sq) / (float)c.vdim + c.eps);
    for (int d = lane; d < c.vdim; d += 32) out[d] = from_f32<T>(o[d] * rs * c.norm_w[h * c.vdim + d] * (1.0f / (1.0f + expf(-to_f32(g[d])))));
}

template <typename T>
static int ml_go(MlArgs p, dim3 grid, size_t fixed, size_t slab, cudaStream_t st) {
    const bool one = p.n == 1;
    p.in_smem = !one && fixed + slab <= 160 * 1024;
    const size_t smem = fixed + (p.in_smem ? slab : 0);
    if (!one) JB_CUDA(cudaFuncSetAttribute(mlstm_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
    if (one) JB_CUDA(launch_cluster_k(mlstm_kernel<T, true>, grid, dim3(ML_THREADS), dim3(grid.x), smem, st, pdl_enabled(), p));
    else     JB_CUDA(launch_cluster_k(mlstm_kernel<T, false>, grid, dim3(ML_THREADS), dim3(grid.x), smem, st, pdl_enabled(), p));
    count_launch();
    return JB_OK;
}

int launch_mlstm(const MlstmCall& a, int n, int start, const int* d_pos, cudaStream_t st) {
    if (n <= 0) return JB_OK;
    DeviceCtx* x = ctx();
    if (!x) return set_error(JB_ERR_STATE, "mlstm: library not initialised");
    if (a.heads <= 0 || a.heads > 65535 || a.dim <= 0 || a.dim > ML_MAX_DIM || a.vdim <= 0 || a.vdim > ML_MAX_DIM || !(a.cap > 0.f) || (d_pos && n != 1) || (!d_pos && start < 0))
        return set_error(JB_ERR_ARG, "mlstm: %d heads of %d x %d, gate cap %g", a.heads, a.dim, a.vdim, a.cap);
    if (!a.proj || !a.gates || !a.bias || !a.norm_w || !a.state || !a.out || (n > 1 && !a.raw)) return set_error(JB_ERR_PTR, "mlstm: null pointer");
    const bool chunks = n > 1 && mlstm_chunks_apply(a, n);
    if (chunks) {
        const int rc = launch_mlstm_chunks(a, n, start, st);
        if (rc) return rc;
    } else {
        MlArgs p = {};
        p.c = a; p.n = n; p.start = start; p.d_pos = d_pos; p.early = d_pos != nullptr;
        const int vld = pad8(a.vdim);
        unsigned cl = 1;
        while (cl < ML_MAX_CLUSTER && ((a.heads * cl < (unsigned)x->sm_count && vld / (int)(2 * cl) >= 16) || vld / (int)cl > 1024)) cl *= 2;
        p.vs = ((vld + (int)cl - 1) / (int)cl + 3) & ~3;
        const size_t fixed = ((size_t)3 * pad8(a.dim) + 4 * ML_THREADS) * sizeof(float), slab = (size_t)a.dim * p.vs * sizeof(float);
        const dim3 grid(cl, a.heads);
        const int rc = a.kind == EK_F32 ? ml_go<float>(p, grid, fixed, slab, st) : ml_go<__nv_bfloat16>(p, grid, fixed, slab, st);
        if (rc || n == 1) return rc;
    }
    const dim3 og((unsigned)(((long long)n * a.heads * 32 + 255) / 256));
    const uintptr_t four = a.kind == EK_F32 ? 15 : 7;
    const bool vec = a.vdim % 4 == 0 && a.ld % 4 == 0 && a.off_g % 4 == 0 && a.ldo % 4 == 0 && !(((uintptr_t)a.raw | (uintptr_t)a.norm_w) & 15) && !(((uintptr_t)a.proj | (uintptr_t)a.out) & four);
    if (a.kind == EK_F32) JB_CUDA(launch_k(mlstm_out_kernel<float>, og, dim3(256), 0, st, pdl_enabled(), a, n, chunks, vec));
    else                  JB_CUDA(launch_k(mlstm_out_kernel<__nv_bfloat16>, og, dim3(256), 0, st, pdl_enabled(), a, n, chunks, vec));
    count_launch();
    return JB_OK;
}

}  // namespace jb
