// dense_gemv.cu — one token against dense weights: the decode products of layer-list models, HBM-bound.
//
// Two CTAs of eight warps per SM; the output rows (or gate / up row pairs) are dealt to the CTAs in contiguous runs and
// within a CTA to groups of 1, 2, 4 or 8 warps that share a row (as many as make the warps' work most even).  A warp walks R
// rows at a time and keeps eight 16-byte weight loads per lane in flight, one batch ahead of the arithmetic.
// Where the rows do not depend on the previous kernel (all modes but the expert ones, and not where the caller says `late`) the first
// batch is requested before griddepcontrol.wait, so the weights stream in while the input vector is still being produced and normed.  The input
// vector is held in shared memory in the activation type (what the prompt path multiplies), sums are fp32.
#include "dense.cuh"

namespace jb {

constexpr int DG_THREADS = 256, DG_WARPS = DG_THREADS / 32, DG_LOADS = 8, DG_AHEAD = 64 << 10;

struct DgArgs {
    DenseGemv g;
    int nchunk;          // 16-byte chunks of the input vector (of one expert's input for GEMV_MOE_DOWN, of both inputs for GEMV_TWO)
    int n1;              // GEMV_TWO: chunks of the first input
    uint32_t magic;      // ceil(2^32 / nchunk): chunk / nchunk by one multiply
    int split;           // warps that share a row (1, 2, 4 or 8), each with its range of chunks
    int off_part;        // shared memory: start of the partial sums
};

template <typename T, int MODE, int R>
__global__ void __launch_bounds__(DG_THREADS, 2) dense_gemv_kernel(const DgArgs p) {
    constexpr int U = DG_LOADS / R;              // chunks per row in a batch
    constexpr bool DUO = MODE == GEMV_MOE_UP || MODE == GEMV_PAIR;     // an item is two rows: gate and up of an expert, or adjacent ones
    constexpr bool NORM = MODE == GEMV_NORM || MODE == GEMV_PAIR;
    constexpr int STEP = DUO ? R / 2 : R;                             // items per group of rows
    extern __shared__ __align__(16) unsigned char dg_sm[];
    __shared__ float red[NORM_RED * DG_WARPS];
    __shared__ int s_ids[MOE_MAX_TOP];
    __shared__ float s_wts[MOE_MAX_TOP];
    const DenseGemv& g = p.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int items = MODE == GEMV_MOE_UP ? g.route.top * g.M : MODE == GEMV_PAIR ? (g.M + 1) / 2 : g.M;
    // this CTA's items [i0, i1); warp (grp, part) takes items i0 + grp, + groups, ... and chunks [c0, c1) of each
    const int n_cta = MODE == GEMV_PAIR && g.side.z ? gridDim.x - 1 : gridDim.x;
    if (MODE == GEMV_PAIR && blockIdx.x == n_cta) {
        pdl_wait();
        pdl_launch();
        latent_row<T, DG_THREADS>(g.side, 0, *g.side.d_pos, false, red);
        return;
    }
    const int i0 = (int)((long long)items * blockIdx.x / n_cta), i1 = (int)((long long)items * (blockIdx.x + 1) / n_cta);
    const int groups = DG_WARPS / p.split, grp = warp / p.split, part = warp - grp * p.split;
    const int mine = i1 - i0 > grp ? (i1 - i0 - grp + groups - 1) / groups : 0;
    const int nchunk = MODE == GEMV_MOE_DOWN ? p.nchunk * g.route.top : p.nchunk;
    const int c0 = (int)((long long)nchunk * part / p.split), c1 = (int)((long long)nchunk * (part + 1) / p.split);
    const int nb = (c1 - c0 + 32 * U - 1) / (32 * U);
    const int n_batches = ((mine + STEP - 1) / STEP) * nb;
    uint4* hs = reinterpret_cast<uint4*>(dg_sm);
    float* partial = reinterpret_cast<float*>(dg_sm + p.off_part);

    auto item_at = [&](int j) { return i0 + grp + min(j, mine - 1) * groups; };
    auto load = [&](int j, int b, uint4 (&w)[DG_LOADS]) {             // batch b of the rows of the warp's items j .. j + STEP - 1
        #pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint4* row = nullptr;
            int item = 0;
            if (MODE == GEMV_MOE_UP) {
                item = item_at(j);
                const int k = item / g.M, f = item - k * g.M;
                row = reinterpret_cast<const uint4*>(r == 0 ? g.W : g.W_up) + ((size_t)s_ids[k] * g.M + f) * p.nchunk;
            } else {
                item = MODE == GEMV_PAIR ? min(2 * item_at(j + r / 2) + (r & 1), g.M - 1) : item_at(j + r);
                row = reinterpret_cast<const uint4*>(g.W) + (size_t)item * p.nchunk;
            }
            #pragma unroll
            for (int u = 0; u < U; ++u) {
                const int c = c0 + (b * U + u) * 32 + lane;
                w[r * U + u] = make_uint4(0, 0, 0, 0);
                if (c < c1) {
                    if (MODE == GEMV_MOE_DOWN) {
                        const int k = p.nchunk == 1 ? c : (int)__umulhi((uint32_t)c, p.magic);
                        w[r * U + u] = __ldg(row + (size_t)s_ids[k] * g.M * p.nchunk + (c - k * p.nchunk));
                    } else {
                        w[r * U + u] = __ldg(row + c);
                    }
                }
            }
        }
    };
    auto finish = [&](int item, float v, float v2) {
        if (MODE == GEMV_MOE_UP) {
            const int k = item / g.M, f = item - k * g.M;
            reinterpret_cast<T*>(g.seg[0].y)[(long long)k * g.seg[0].ld + f] = from_f32<T>(silu_f(v) * v2);
        } else if (MODE == GEMV_PAIR) {
            store_rows2<T>(g.seg, g.nseg, g.softcap, g.d_pos, 0, g.d_pos ? *g.d_pos : 0, 2 * item, g.M, v, v2);
        } else {
            store_seg<T>(g.seg, g.nseg, g.softcap, g.d_pos, 0, item, v);
        }
    };

    uint4 cur[DG_LOADS], nxt[DG_LOADS];
    if (MODE == GEMV_PLAIN && g.late) pdl_wait();
    if (MODE != GEMV_MOE_UP && MODE != GEMV_MOE_DOWN) { if (n_batches > 0) load(0, 0, cur); }
    // The rest of the CTA's first rows on their way into L2 while the input vector is being produced and normed; more than DG_AHEAD delays the loads
    // behind them (a request of a model with parallel layers, 512 + 16 tokens, us at 0 / 32 / 64 / 128 / 256 KB: 7932 / 7788 / 7778 / 7907 / 8118).  Not
    // where a CTA has no more than that, half of it in its first loads: width 1024, 8 + 32 tokens, without / always / so: 8696 / 8721 / 8687 (parallel
    // layers), 10575 / 10711 / 10663 (the same in fp32), 12995 / 13082 / 13024 (sequential, fp32); width 2560 13960 / 13793 / 13810, 15505 / 15457 / 15448.
    if (MODE != GEMV_MOE_UP && MODE != GEMV_MOE_DOWN && !g.late) {
        const long long row = (long long)p.nchunk * 16;
        const int r0 = MODE == GEMV_PAIR ? 2 * i0 : i0, r1 = MODE == GEMV_PAIR ? min(2 * i1, g.M) : i1;
        const char* at = reinterpret_cast<const char*>(g.W) + r0 * row;
        const long long bytes = min((long long)DG_AHEAD, (r1 - r0) * row);
        for (long long o = (r1 - r0) * row > DG_AHEAD ? (long long)threadIdx.x * 2048 : bytes; o < bytes; o += DG_THREADS * 2048)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at + o), "r"((uint32_t)min(2048ll, bytes - o)) : "memory");
    }
    if (NORM) norm_prefetch<DG_THREADS>(g.norm);
    pdl_wait();
    pdl_launch();
    // ── the input vector ──
    if (NORM) {
        float* buf = reinterpret_cast<float*>(dg_sm + (size_t)p.nchunk * 16);
        T* h = reinterpret_cast<T*>(hs);
        norm_step_row<T, DG_THREADS>(g.norm, 0, buf, red, blockIdx.x == 0 && g.norm.x_out, h);
        __syncthreads();
        if (blockIdx.x == 0 && g.norm.h)
            for (int i = threadIdx.x; i < p.nchunk; i += DG_THREADS) reinterpret_cast<uint4*>(g.norm.h)[i] = hs[i];
    } else {
        for (int i = threadIdx.x; i < nchunk; i += DG_THREADS)
            hs[i] = MODE == GEMV_TWO && i >= p.n1 ? reinterpret_cast<const uint4*>(g.x2)[i - p.n1] : reinterpret_cast<const uint4*>(g.x)[i];
        if (MODE == GEMV_MOE_UP) {
            if (warp == 0) {
                float* c = reinterpret_cast<float*>(dg_sm + (size_t)nchunk * 16);
                moe_route_warp(g.z, g.route, c, c + g.route.n_experts, c + 2 * g.route.n_experts, [&](int k, int id, float w) {
                    s_ids[k] = id; s_wts[k] = w;
                    if (blockIdx.x == 0) { g.ids[k] = id; g.wts[k] = w; }
                });
            }
        } else if (MODE == GEMV_MOE_DOWN) {
            for (int k = threadIdx.x; k < g.route.top; k += DG_THREADS) { s_ids[k] = g.ids[k]; s_wts[k] = g.wts[k]; }
        }
        __syncthreads();
        if ((MODE == GEMV_MOE_UP || MODE == GEMV_MOE_DOWN) && n_batches > 0) load(0, 0, cur);
    }
    // ── the products ──
    float acc[R], f1[MODE == GEMV_TWO ? R : 1], f2[MODE == GEMV_TWO ? R : 1];
    #pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
    int j = 0, b = 0;
    for (int it = 0; it < n_batches; ++it) {
        int j_n = j, b_n = b + 1;
        if (b_n == nb) { b_n = 0; j_n += STEP; }
        if (it + 1 < n_batches) load(j_n, b_n, nxt);
        if constexpr (MODE == GEMV_TWO) {
            if (b == 0) {
                #pragma unroll
                for (int r = 0; r < R; ++r) { const int row = item_at(j + r); f1[r] = g.ls ? __ldg(g.ls + row) : 1.f; f2[r] = g.ls2 ? __ldg(g.ls2 + row) : 1.f; }
            }
        }
        #pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + (b * U + u) * 32 + lane;
            if (c < c1) {
                const uint4 h = hs[c];
                if (MODE == GEMV_MOE_DOWN) {
                    const float w = s_wts[p.nchunk == 1 ? c : (int)__umulhi((uint32_t)c, p.magic)];
                    #pragma unroll
                    for (int r = 0; r < R; ++r) acc[r] = fmaf(w, dot16(cur[r * U + u], h, 0.f, T()), acc[r]);
                } else if constexpr (MODE == GEMV_TWO) {
                    #pragma unroll
                    for (int r = 0; r < R; ++r) acc[r] = fmaf(c < p.n1 ? f1[r] : f2[r], dot16(cur[r * U + u], h, 0.f, T()), acc[r]);
                } else {
                    #pragma unroll
                    for (int r = 0; r < R; ++r) acc[r] = dot16(cur[r * U + u], h, acc[r], T());
                }
            }
        }
        if (b_n == 0) {
            #pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = warp_sum(acc[r]);
            if (p.split > 1) {
                #pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int jj = j + (DUO ? r / 2 : r);
                    if (lane == r && jj < mine) partial[((item_at(jj) - i0) * p.split + part) * (DUO ? 2 : 1) + (DUO ? r & 1 : 0)] = acc[r];
                }
            } else if (DUO) {
                #pragma unroll
                for (int r = 0; r < R; r += 2) if (lane == r && j + r / 2 < mine) finish(item_at(j + r / 2), acc[r], acc[R > 1 ? r + 1 : 0]);
            } else {
                #pragma unroll
                for (int r = 0; r < R; ++r) if (lane == r && j + r < mine) finish(item_at(j + r), acc[r], 0.f);
            }
            #pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = 0.f;
        }
        #pragma unroll
        for (int i = 0; i < DG_LOADS; ++i) cur[i] = nxt[i];
        j = j_n; b = b_n;
    }
    if (p.split > 1) {                           // partial sums of a row in the order of its chunks
        __syncthreads();
        for (int i = threadIdx.x; i < i1 - i0; i += DG_THREADS) {
            float v = 0.f, v2 = 0.f;
            for (int q = 0; q < p.split; ++q) {
                if (DUO) { v += partial[(i * p.split + q) * 2]; v2 += partial[(i * p.split + q) * 2 + 1]; }
                else v += partial[i * p.split + q];
            }
            finish(i0 + i, v, v2);
        }
    }
}

template <typename T, int MODE, int R>
static int dg_go(const DgArgs& p, int grid, size_t smem, cudaStream_t st) {
    static size_t set = 48 * 1024;
    if (smem > set) {
        JB_CUDA(cudaFuncSetAttribute(dense_gemv_kernel<T, MODE, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        set = smem;
    }
    JB_CUDA(launch_k(dense_gemv_kernel<T, MODE, R>, dim3(grid), dim3(DG_THREADS), smem, st, pdl_enabled(), p));
    count_launch();
    return JB_OK;
}
template <typename T, int MODE>
static int dg_rows(const DgArgs& p, int R, int grid, size_t smem, cudaStream_t st) {
    if constexpr (MODE == GEMV_MOE_UP) return dg_go<T, MODE, 2>(p, grid, smem, st);
    else if constexpr (MODE == GEMV_PAIR) return R == 4 ? dg_go<T, MODE, 4>(p, grid, smem, st) : dg_go<T, MODE, 2>(p, grid, smem, st);
    else return R == 4 ? dg_go<T, MODE, 4>(p, grid, smem, st) : R == 2 ? dg_go<T, MODE, 2>(p, grid, smem, st) : dg_go<T, MODE, 1>(p, grid, smem, st);
}
template <typename T>
static int dg_mode(const DgArgs& p, int R, int grid, size_t smem, cudaStream_t st) {
    switch (p.g.mode) {
        case GEMV_NORM:   return dg_rows<T, GEMV_NORM>(p, R, grid, smem, st);
        case GEMV_PLAIN:  return dg_rows<T, GEMV_PLAIN>(p, R, grid, smem, st);
        case GEMV_TWO:    return dg_rows<T, GEMV_TWO>(p, R, grid, smem, st);
        case GEMV_PAIR:   return dg_rows<T, GEMV_PAIR>(p, R, grid, smem, st);
        case GEMV_MOE_UP: return dg_rows<T, GEMV_MOE_UP>(p, R, grid, smem, st);
        default:          return dg_rows<T, GEMV_MOE_DOWN>(p, R, grid, smem, st);
    }
}

int launch_dense_gemv(const DenseGemv& a, cudaStream_t st) {
    DeviceCtx* c = ctx();
    if (!c) return set_error(JB_ERR_STATE, "dense gemv: library not initialised");
    if (a.M <= 0 || a.K <= 0) return set_error(JB_ERR_ARG, "dense gemv: M=%d K=%d", a.M, a.K);
    const bool norm = a.mode == GEMV_NORM || a.mode == GEMV_PAIR, moe = a.mode == GEMV_MOE_UP || a.mode == GEMV_MOE_DOWN, duo = a.mode == GEMV_MOE_UP || a.mode == GEMV_PAIR;
    if (!a.W || (!norm && !a.x) || (a.mode == GEMV_TWO && (!a.x2 || a.K2 <= 0)) || (a.mode == GEMV_MOE_UP && (!a.W_up || !a.z)) || (moe && (!a.ids || !a.wts)))
        return set_error(JB_ERR_PTR, "dense gemv: null pointer");
    if (moe && (a.route.top <= 0 || a.route.top > MOE_MAX_TOP || a.route.n_experts > MOE_MAX_EXPERTS)) return set_error(JB_ERR_LIMIT, "dense gemv: top %d of %d experts", a.route.top, a.route.n_experts);
    DgArgs p;
    p.g = a;
    const int es = a.kind == EK_F32 ? 4 : 2;
    p.n1 = pad8(a.K) * es / 16;
    p.nchunk = p.n1 + (a.mode == GEMV_TWO ? pad8(a.K2) * es / 16 : 0);
    p.magic = p.nchunk > 1 ? (uint32_t)((0x100000000ull + p.nchunk - 1) / p.nchunk) : 0;
    const int chunks = a.mode == GEMV_MOE_DOWN ? p.nchunk * a.route.top : p.nchunk;
    const int items = a.mode == GEMV_MOE_UP ? a.route.top * a.M : a.mode == GEMV_PAIR ? (a.M + 1) / 2 : a.M;
    const int side = a.mode == GEMV_PAIR && a.side.z ? 1 : 0, slots = 2 * c->sm_count - side;
    const int grid = items < slots ? items : slots, per_cta = (items + grid - 1) / grid;
    // warps per row and rows at a time: the fewest loads of the busiest warp (slots of a batch that a row does not fill count a
    // little: they cost no traffic, but leave less in flight; so do the reduction at the end of a row and a split)
    int R = 1;
    double best = 1e30;
    for (int S = 1; S <= DG_WARPS; S *= 2) {
        const int rows = (per_cta + DG_WARPS / S - 1) / (DG_WARPS / S), lanes = ((chunks + S - 1) / S + 31) / 32;
        for (int r = duo ? 2 : 1; r <= (a.mode == GEMV_MOE_UP ? 2 : 4); r *= 2) {
            const int u = DG_LOADS / r, step = duo ? r / 2 : r, trips = (rows + step - 1) / step, nb = (lanes + u - 1) / u;
            const double used = (double)trips * r * lanes, room = (double)trips * r * nb * u;
            const double cost = used + 0.5 * (room - used) + 1.0 * trips + (S > 1 ? 2.0 : 0.0);
            if (cost < best - 1e-9) { best = cost; R = r; p.split = S; }
        }
    }
    size_t smem = (size_t)chunks * 16;
    if (norm) smem += (size_t)pad8(a.K) * 4;
    if (a.mode == GEMV_MOE_UP) smem += ((size_t)(2 * a.route.n_experts + a.route.n_groups) * 4 + 15) & ~(size_t)15;
    p.off_part = (int)smem;
    if (p.split > 1) smem += (size_t)per_cta * p.split * (duo ? 8 : 4);
    if (smem > (size_t)c->max_smem_optin - 2048) return set_error(JB_ERR_LIMIT, "dense gemv: input of %d elements", a.K);
    return a.kind == EK_F32 ? dg_mode<float>(p, R, grid + side, smem, st) : dg_mode<__nv_bfloat16>(p, R, grid + side, smem, st);
}

}  // namespace jb
