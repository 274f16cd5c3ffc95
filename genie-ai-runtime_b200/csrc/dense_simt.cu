// dense_simt.cu — dense products over many tokens on the CUDA cores, in true fp32 (FFMA, no reduced-precision matrix mode): the 32-bit
// path of layer-list models; groups (experts) on grid.z.
//
// A launch has few tokens per weight matrix here (an expert of a 130-token prompt: 16), so it is bound by the weights' way from memory and by the
// tokens that pad a tile.  A WARP holds a tile of 64 rows x 16 tokens, 8 x 4 values per lane, and the warps of a CTA take
// four k of a K tile in turn; a CTA is 16, 32 or 64 tokens wide (the other warps' tiles) and its warps' sums meet in shared memory in a fixed order.  Operands come by
// cp.async in three stages (gate and up: four), K contiguous as in memory: a lane reads four k of a row at a time, 12 (gate and up: 20) 16-byte reads of shared memory,
// free of conflicts, for 128 (256) multiply-adds.
//
// 130 tokens, width 1024, 32 experts of 768, top 4, us before (64 x 32 tiles, 4 x 2 values a thread, tiles transposed through registers) / here:
// gate and up 169 / 89 (their weights at the rate of memory: 31), down 108 / 57; 3072 x 1024 and 1024 x 2048 67 and 71 / 47 and 30.  The reads of
// shared memory, four passes for each of 16 bytes a lane, now take 1.5 times the multiply-adds.  Error against 64 bits of the whole request 5.5e-7 / 3.4e-7.
#include "dense.cuh"

namespace jb {

constexpr int DS_M = 64, DS_T = 16, DS_WARPS = 8, DS_THREADS = DS_WARPS * 32;
// K tile and stages: two CTAs per SM; rows K + 4 words apart, so that eight rows' reads lie in different banks
template <bool GLU> constexpr int DS_K = GLU ? 32 : 64;
template <bool GLU> constexpr int DS_STAGES = GLU ? 4 : 3;

template <bool GLU, int WT> constexpr int ds_stage() { return (DS_M * (GLU ? 2 : 1) + DS_T * WT) * (DS_K<GLU> + 4); }      // floats
template <bool GLU, int WT> constexpr size_t ds_smem() {
    const size_t stages = (size_t)DS_STAGES<GLU> * ds_stage<GLU, WT>(), sums = (size_t)DS_WARPS * DS_M * DS_T * (GLU ? 2 : 1);
    return (stages > sums ? stages : sums) * sizeof(float);
}

// Groups of unlike sizes, known on the device alone: the tiles of group g start at item off[g] / width + g, which leaves room for as many as the tokens
// before it can fill, with a part of a tile in every group.  False: no tile there.
template <int WIDTH>
__device__ __forceinline__ bool ds_find(const int* off, int n_groups, int item, int& grp, int& t0, int& t_hi) {
    const int lane = threadIdx.x & 31;
    for (int base = 0;; base += 32) {
        const int g = min(base + lane, n_groups - 1), lo = off[g], hi = off[g + 1], first = lo / WIDTH + g;
        const unsigned begun = __ballot_sync(0xFFFFFFFFu, base + lane < n_groups && first <= item);
        if (begun == 0xFFFFFFFFu && base + 32 < n_groups && off[base + 32] / WIDTH + base + 32 <= item) continue;
        const int at = 31 - __clz(begun);
        grp = base + at;
        t0 = __shfl_sync(0xFFFFFFFFu, lo + (item - first) * WIDTH, at);
        t_hi = __shfl_sync(0xFFFFFFFFu, hi, at);
        return t0 < t_hi;
    }
}

// WT: 16-token tiles of a CTA; its 8 / WT warps on a tile share K
template <bool GLU, int WT>
__global__ void __launch_bounds__(DS_THREADS, 2) dense_simt_kernel(const __grid_constant__ DenseGemm a, int tiles, bool vec) {
    pdl_wait();
    pdl_launch();
    extern __shared__ __align__(16) float ds_sm[];
    constexpr int KG = DS_WARPS / WT, ROWS = DS_M * (GLU ? 2 : 1) + DS_T * WT, STAGE = ds_stage<GLU, WT>(), KT = DS_K<GLU>, LD = KT + 4, STAGES = DS_STAGES<GLU>, QUADS = KT / 4, PER = DS_THREADS / QUADS;
    const int r0 = blockIdx.x * DS_M, ldw = a.ldw > 0 ? a.ldw : pad8(a.K), ldx = a.ldx > 0 ? a.ldx : pad8(a.K);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tx = lane & 7, ty = lane >> 3, wt = warp % WT, kg = warp / WT;
    const int k_tiles = (a.K + KT - 1) / KT;
    for (int item = blockIdx.y; item < tiles; item += gridDim.y) {
        int grp = blockIdx.z, t0 = item * DS_T * WT, t_hi = a.N;
        if (a.off && !ds_find<DS_T * WT>(a.off, a.n_groups, item, grp, t0, t_hi)) continue;
        const float* W = reinterpret_cast<const float*>(a.W) + (size_t)grp * a.M * ldw;
        const float* V = GLU ? reinterpret_cast<const float*>(a.W_up) + (size_t)grp * a.M * ldw : nullptr;
        const float* x = reinterpret_cast<const float*>(a.x) + (size_t)grp * a.x_step;
        // QUADS pieces of 16 bytes a row: thread's piece of every PER-th row
        auto fetch = [&](int kt) {
            float* st = ds_sm + (kt % STAGES) * STAGE;
            const int k = kt * KT + 4 * (threadIdx.x % QUADS);
            #pragma unroll
            for (int j = 0; j < ROWS; j += PER) {
                const int r = j + threadIdx.x / QUADS;
                if (r >= ROWS) break;
                const float* src; bool in;
                if (j < DS_M) { src = W + (size_t)(r0 + r) * ldw; in = r0 + r < a.M; }
                else if (GLU && j < 2 * DS_M) { src = V + (size_t)(r0 + r - DS_M) * ldw; in = r0 + r - DS_M < a.M; }
                else { const int t = t0 + r - DS_M * (GLU ? 2 : 1); src = x + (size_t)t * ldx; in = t < t_hi; }
                float* dst = st + r * LD + 4 * (threadIdx.x % QUADS);
                const int left = in ? max(0, min(4, a.K - k)) : 0;               // elements of the piece; the rest is zero
                if (vec) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(left ? src + k : x), "r"(4 * left) : "memory");
                } else {
                    #pragma unroll
                    for (int e = 0; e < 4; ++e) dst[e] = e < left ? src[k + e] : 0.f;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        float acc[8][4] = {}, acu[GLU ? 8 : 1][4] = {};
        #pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) { if (s < k_tiles) fetch(s); else asm volatile("cp.async.commit_group;" ::: "memory"); }
        for (int kt = 0; kt < k_tiles; ++kt) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();                             // the tile has landed, and the one before it is read
            if (kt + STAGES - 1 < k_tiles) fetch(kt + STAGES - 1); else asm volatile("cp.async.commit_group;" ::: "memory");
            const float* st = ds_sm + (kt % STAGES) * STAGE;
            #pragma unroll 1
            for (int q = kg; q < QUADS; q += KG) {
                float4 xv[4];
                #pragma unroll
                for (int j = 0; j < 4; ++j) xv[j] = load4(st + (DS_M * (GLU ? 2 : 1) + DS_T * wt + ty + 4 * j) * LD + 4 * q);
                #pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 w = load4(st + (tx + 8 * i) * LD + 4 * q);
                    #pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(w.w, xv[j].w, fmaf(w.z, xv[j].z, fmaf(w.y, xv[j].y, fmaf(w.x, xv[j].x, acc[i][j]))));
                    if constexpr (GLU) {
                        const float4 u = load4(st + (DS_M + tx + 8 * i) * LD + 4 * q);
                        #pragma unroll
                        for (int j = 0; j < 4; ++j) acu[i][j] = fmaf(u.w, xv[j].w, fmaf(u.z, xv[j].z, fmaf(u.y, xv[j].y, fmaf(u.x, xv[j].x, acu[i][j]))));
                    }
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // [kg][wt][token 16][row 64] (then the same of `up`): the sums of a value's K groups, in their order
        constexpr int PART = DS_WARPS * DS_T * DS_M;
        float* mine = ds_sm + (kg * WT + wt) * DS_T * DS_M;
        #pragma unroll
        for (int i = 0; i < 8; ++i)
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                mine[(ty + 4 * j) * DS_M + tx + 8 * i] = acc[i][j];
                if constexpr (GLU) mine[PART + (ty + 4 * j) * DS_M + tx + 8 * i] = acu[i][j];
            }
        __syncthreads();
        for (int e = threadIdx.x; e < WT * DS_T * DS_M / 2; e += DS_THREADS) {
            const int r = 2 * (e % (DS_M / 2)), tl = e / (DS_M / 2), t = t0 + tl, at = tl * DS_M + r;
            if (t >= t_hi || r0 + r >= a.M) continue;
            float2 s = *reinterpret_cast<const float2*>(ds_sm + at), u = make_float2(0.f, 0.f);
            if (GLU) u = *reinterpret_cast<const float2*>(ds_sm + PART + at);
            #pragma unroll
            for (int g = 1; g < KG; ++g) {
                const float2 v = *reinterpret_cast<const float2*>(ds_sm + g * WT * DS_T * DS_M + at);
                s.x += v.x; s.y += v.y;
                if (GLU) { const float2 w = *reinterpret_cast<const float2*>(ds_sm + PART + g * WT * DS_T * DS_M + at); u.x += w.x; u.y += w.y; }
            }
            store_rows2<float>(a.seg, a.nseg, a.softcap, nullptr, t, a.start + t, r0 + r, a.M, GLU ? silu_f(s.x) * u.x : s.x, GLU ? silu_f(s.y) * u.y : s.y, (long long)grp * a.y_step);
        }
        __syncthreads();                                 // before the next tokens' tiles take the place of the sums
    }
}

template <bool GLU, int WT>
static int ds_go(const DenseGemm& a, bool vec, cudaStream_t st) {
    static bool set[16] = {};
    DeviceCtx* c = ctx();
    if (!c) return JB_ERR_CUDA;
    if (!set[c->device]) { JB_CUDA(cudaFuncSetAttribute(dense_simt_kernel<GLU, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ds_smem<GLU, WT>())); set[c->device] = true; }
    // Groups of unlike sizes have no more tiles than this (see ds_find), wherever their tokens are (a few CTAs for each group, walking its tiles, took twice as long as
    // before where all tokens went to one expert of many: 2048 tokens, gate and up of 768 x 1024, 316 -> 673 us; so 203).
    const int width = DS_T * WT, tiles = a.off ? a.N / width + a.n_groups : (a.N + width - 1) / width;
    JB_CUDA(launch_k(dense_simt_kernel<GLU, WT>, dim3((a.M + DS_M - 1) / DS_M, tiles < 65535 ? tiles : 65535, a.off ? 1 : a.n_groups), dim3(DS_THREADS), ds_smem<GLU, WT>(), st, pdl_enabled(), a, tiles, vec));
    count_launch();
    return JB_OK;
}
int launch_dense_gemm_simt(const DenseGemm& a, cudaStream_t st) {
    if (a.N <= 0 || a.M <= 0) return JB_OK;
    if (a.kind != EK_F32) return set_error(JB_ERR_TYPE, "dense fp32 gemm: element kind %d", a.kind);
    if (!a.W || !a.x || (a.swiglu && !a.W_up) || (a.n_groups > 1 && !a.off && !a.x_step)) return set_error(JB_ERR_PTR, "dense fp32 gemm: null pointer");
    const int ldw = a.ldw > 0 ? a.ldw : pad8(a.K), ldx = a.ldx > 0 ? a.ldx : pad8(a.K);
    const bool vec = !(((uintptr_t)a.W | (uintptr_t)a.x | (a.swiglu ? (uintptr_t)a.W_up : 0)) & 15) && ldw % 4 == 0 && ldx % 4 == 0 && a.x_step % 4 == 0;
    if ((a.N + 63) / 64 > 65535) return set_error(JB_ERR_LIMIT, "dense fp32 gemm: %d tokens", a.N);
    DeviceCtx* c = ctx();
    if (!c) return JB_ERR_CUDA;
    // Wider tiles read the weights less often, narrower ones make more CTAs and pad less: as wide as still leaves two CTAs per SM, and no
    // wider than a group's tokens are on average.
    const long long per_group = a.off ? a.N / a.n_groups : a.N, row_tiles = (long long)((a.M + DS_M - 1) / DS_M) * a.n_groups;
    int wt = 1;
    while (wt < 4 && per_group >= 2 * wt * DS_T && row_tiles * ((per_group + 2 * wt * DS_T - 1) / (2 * wt * DS_T)) >= 2 * c->sm_count) wt *= 2;
    if (a.swiglu) return wt == 1 ? ds_go<true, 1>(a, vec, st) : wt == 2 ? ds_go<true, 2>(a, vec, st) : ds_go<true, 4>(a, vec, st);
    return wt == 1 ? ds_go<false, 1>(a, vec, st) : wt == 2 ? ds_go<false, 2>(a, vec, st) : ds_go<false, 4>(a, vec, st);
}
// One token (the logits after a prompt) is a product of the decode family: 151936 x 2560 in bf16 take 122 us there, the weights at the
// rate of memory, and 145 us in tiles of 16 tokens, the narrowest of this file.
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
