// gemm_pair.cu — products of 16-bit operands over many tokens by PAIRS of CTAs: tcgen05.mma with cta_group::2, both operands
// brought by TMA, the accumulator in the tensor memory of both CTAs.
//
// What bounds it: shared memory.  One CTA alone (dense_tc.cu: 128 x 256 tiles) writes 48 KB of operands per K tile of 64 and the
// tensor pipe reads 48 KB, 192 B per clock against the 128 that shared memory serves.  A pair works on 256 (weight rows) x 256
// (tokens): each CTA keeps 128 rows of the weights and HALF of the tokens' tile, 32 KB in and 32 KB out per K tile, which is just
// what the 512 clocks of its four MMAs allow.
//
// One persistent pair per two SMs walks the output tiles, token tile fastest; six stages of 32 KB per CTA; two accumulators of 256
// columns so that the drain of a tile overlaps the K loop of the next.  Tiles left over after the last full round of pairs would
// keep a few pairs busy for a whole tile time (2560 x 9728 over 2048 tokens: 80 tiles for 74 pairs); with a workspace they are cut
// into K ranges that fill one short round, and a second kernel adds the fp32 partial sums in a fixed order.
// Warps: 0 TMA producer (both CTAs), 1 MMA issuer (the even CTA; the odd one only holds its tensor memory), 2-3 idle, 4-7 drain.
// Weight rows are the M side: the drain's lanes are rows, as in dense_tc.cu.  Every mbarrier wait is bounded.
#include "dense.cuh"
#include "tc.cuh"
#include <type_traits>

namespace jb {

constexpr int GP_M = 128, GP_K = 64, GP_STAGES = 6, GP_THREADS = 256, GP_TOKENS = 256;
constexpr int GP_A_BYTES = GP_M * GP_K * 2, GP_STAGE_BYTES = GP_A_BYTES + GP_TOKENS / 2 * GP_K * 2;
constexpr int GP_SMEM = GP_STAGES * GP_STAGE_BYTES + 16 * 1024 + 1024;          // operands, the drain's transposes, alignment

struct GpArgs {
    OutSeg seg[MAX_SEG]; int nseg, vec, start;       // vec: rows4_aligned
    int M, N, n_tile, k_tiles;                       // n_tile: token box, a multiple of 16
    int tiles_n, width, n_full, n_items, ksplit;     // tokens are dealt evenly: token tile i holds [i * width, (i + 1) * width)
    float softcap;
    float* part;                                     // [K range][tail tile][token of the tile][256 rows]
    int* status;
};

__device__ __forceinline__ uint32_t gp_leader(uint32_t addr) {       // the same shared address in the even CTA of the pair
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// a load into this CTA's memory whose bytes are counted on the even CTA's barrier
__device__ __forceinline__ void gp_load(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void gp_commit(uint64_t* bar) {           // arrives on the barrier at this address in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void gp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                                                                                           const __grid_constant__ GpArgs a) {
    extern __shared__ uint8_t gp_smem_raw[];
    __shared__ uint64_t full[GP_STAGES], empty[GP_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int fail;
    uint8_t* smem = gp_smem_raw + ((1024u - (smem_u32(gp_smem_raw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = blockIdx.x & 1, n_pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < GP_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        fence_mbar_init();
        fail = 0;
    }
    // Both CTAs run before either asks for the pair's tensor memory: an allocation that began before the peer was there never returned
    // (seen once in some hundred launches that follow one another, where the CTAs of a pair start as the SMs fall free).
    __syncwarp();
    gp_cluster_sync();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    pdl_launch();
    __syncwarp();
    tc_fence_before();
    gp_cluster_sync();                               // barriers and tensor memory of both CTAs are there
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int n_tail = a.ksplit > 1 ? (a.n_items - a.n_full) / a.ksplit : 0;
    // work item w -> weight rows mt * 256 .., tokens [n0, n_end), K tiles [t0, t1)
    auto locate = [&](int w, int& tile, int& sp, int& mt, int& n0, int& n_end, int& t0, int& t1) {
        tile = w; sp = 0; t0 = 0; t1 = a.k_tiles;
        if (w >= a.n_full && a.ksplit > 1) {
            const int i = w - a.n_full;
            tile = a.n_full + i / a.ksplit; sp = i % a.ksplit;
            t0 = (int)((long long)sp * a.k_tiles / a.ksplit); t1 = (int)((long long)(sp + 1) * a.k_tiles / a.ksplit);
        }
        mt = tile / a.tiles_n;
        n0 = min((tile - mt * a.tiles_n) * a.width, a.N);
        n_end = min(n0 + a.width, a.N);
    };

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            const uint32_t bytes = 2u * (GP_A_BYTES + (uint32_t)a.n_tile / 2 * GP_K * 2);
            for (int w = blockIdx.x >> 1; w < a.n_items && !fail; w += n_pairs) {
                int tile, sp, mt, n0, n_end, t0, t1;
                locate(w, tile, sp, mt, n0, n_end, t0, t1);
                const int wrow = (2 * mt + rank) * GP_M, half = max(16, (n_end - n0 + 15) & ~15) / 2;
                for (int t = t0; t < t1; ++t, ++it) {
                    const int s = it % GP_STAGES;
                    if (!tc_wait(&empty[s], ((it / GP_STAGES) & 1) ^ 1) || fail) { tc_fail(&fail, a.status); break; }
                    uint8_t* st = smem + s * GP_STAGE_BYTES;
                    const uint32_t bar = gp_leader(smem_u32(&full[s]));
                    if (rank == 0) mbar_expect_tx(&full[s], bytes);
                    gp_load(st, &wmap, t * GP_K, wrow, bar);
                    gp_load(st + GP_A_BYTES, &xmap, t * GP_K, n0 + rank * half, bar);
                }
            }
            // nothing may still arrive at this CTA's barriers, or be on its way into its memory, when it leaves
            for (uint32_t i = 0; i < GP_STAGES && i < it; ++i) {
                const uint32_t last = it - 1 - i;
                if (!tc_wait(&empty[last % GP_STAGES], (last / GP_STAGES) & 1)) { tc_fail(&fail, a.status); break; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && lane == 0) {
            // 16-bit x 16-bit -> fp32, both operands K-major, M = 256 over the pair, N = the tile's tokens rounded up to 16
            const uint32_t kind = std::is_same<T, __half>::value ? 0u : (1u << 7) | (1u << 10);
            const uint32_t idesc0 = (1u << 4) | kind | ((uint32_t)(2 * GP_M >> 4) << 24);
            const uint64_t ad0 = tc_smem_desc(smem_u32(smem)), bd0 = tc_smem_desc(smem_u32(smem + GP_A_BYTES));
            uint32_t it = 0, j = 0;
            bool ok = true;
            for (int w = blockIdx.x >> 1; w < a.n_items && ok; w += n_pairs, ++j) {
                int tile, sp, mt, n0, n_end, t0, t1;
                locate(w, tile, sp, mt, n0, n_end, t0, t1);
                const uint32_t d = tmem + (j & 1) * 256u, idesc = idesc0 | ((uint32_t)(max(16, (n_end - n0 + 15) & ~15) >> 3) << 17);
                if (!tc_wait(&acc_empty[j & 1], ((j >> 1) & 1) ^ 1)) { ok = false; break; }
                tc_fence_after();
                for (int t = t0; t < t1; ++t, ++it) {
                    const uint32_t s = it % GP_STAGES;
                    if (!tc_wait(&full[s], (it / GP_STAGES) & 1)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t ad = ad0 + (uint64_t)(s * (GP_STAGE_BYTES >> 4)), bd = bd0 + (uint64_t)(s * (GP_STAGE_BYTES >> 4));
                    #pragma unroll
                    for (int k = 0; k < 4; ++k) gp_mma(d, ad + 2 * k, bd + 2 * k, idesc, (uint32_t)(t != t0 || k != 0));
                    gp_commit(&empty[s]);
                }
                gp_commit(&acc_full[j & 1]);
            }
            if (!ok) tc_fail(&fail, a.status);
        }
    } else if (warp >= 4) {
        const int q = warp & 3, r4 = q * 32 + 4 * (lane & 7);
        float* stage = reinterpret_cast<float*>(smem + GP_STAGES * GP_STAGE_BYTES) + q * 1024;
        uint32_t j = 0;
        for (int w = blockIdx.x >> 1; w < a.n_items; w += n_pairs, ++j) {
            const uint32_t acc = j & 1;
            int tile, sp, mt, n0, n_end, t0, t1;
            locate(w, tile, sp, mt, n0, n_end, t0, t1);
            bool good = true;
            if (lane == 0) good = tc_wait(&acc_full[acc], (j >> 1) & 1) && !fail;
            good = __shfl_sync(0xFFFFFFFFu, (int)good, 0) != 0;
            if (!good) { if (lane == 0) tc_fail(&fail, a.status); break; }
            tc_fence_after();
            const int cols = n_end - n0;
            const uint32_t t_acc = tmem + ((uint32_t)(q * 32) << 16) + acc * 256u;
            // a K range of a tail tile leaves its partial sums, rows side by side
            float* part = n_tail > 0 && w >= a.n_full ? a.part + (((size_t)sp * n_tail + (tile - a.n_full)) * a.n_tile) * 256 + rank * GP_M + r4 : nullptr;
            const Rows4<T> rows(a.seg, a.nseg, a.M, (2 * mt + rank) * GP_M + r4, 0);
            for (int cb = 0; cb < cols; cb += 32) {
                uint32_t r[32];
                __syncwarp();                            // the load needs the whole warp, and the buffer's readers are done
                tc_ld32(t_acc + (uint32_t)cb, r);
                #pragma unroll
                for (int c = 0; c < 32; ++c) stage[c * 32 + lane] = __uint_as_float(r[c]);
                __syncwarp();
                float4 v[8];
                #pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = load4(stage + k * 128 + 4 * lane);
                const int i = cb + (lane >> 3), live = (cols - i + 3) >> 2;                     // this lane's tokens: i, i + 4, .. below cols
                if (part) {
                    #pragma unroll
                    for (int k = 0; k < 8; ++k) if (k < live) store4(part + (size_t)(i + 4 * k) * 256, v[k]);
                } else if (a.vec) {
                    rows.store8(n0 + i, a.start + n0 + i, live, a.softcap, v);
                } else {
                    for (int k = 0; k < 8 && k < live; ++k) {
                        const float4 u = load4(stage + k * 128 + 4 * lane);
                        store_four<T>(a.seg, a.nseg, a.softcap, n0 + i + 4 * k, a.start + n0 + i + 4 * k, rows.row, a.M, u, 0);
                    }
                }
            }
            __syncwarp();
            tc_fence_before();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(gp_leader(smem_u32(&acc_empty[acc]))) : "memory");
        }
    }
    __syncwarp();
    tc_fence_before();
    gp_cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
    // a CTA that left while its peer still frees the pair's tensor memory would make room for another kernel's allocation on its SM
    __syncwarp();
    gp_cluster_sync();
}

// Sum of the tail tiles' K ranges in their order; a thread takes two adjacent rows of one token, CTA (x: tokens of a tile, y: tail tile).
template <typename T>
__global__ void __launch_bounds__(256) gemm_pair_sum_kernel(const GpArgs a) {
    pdl_wait();
    pdl_launch();
    const int n_tail = (a.n_items - a.n_full) / a.ksplit, tile = a.n_full + blockIdx.y, mt = tile / a.tiles_n, n0 = (tile - mt * a.tiles_n) * a.width;
    const int c = blockIdx.x * 2 + (threadIdx.x >> 7), rl = 2 * (threadIdx.x & 127), row = mt * 256 + rl, tok = n0 + c;
    if (c >= a.width || tok >= a.N || row >= a.M) return;
    const float* p = a.part + ((size_t)blockIdx.y * a.n_tile + c) * 256 + rl;
    const size_t step = (size_t)n_tail * a.n_tile * 256;
    float2 s = __ldcg(reinterpret_cast<const float2*>(p));
    for (int k = 1; k < a.ksplit; ++k) { const float2 v = __ldcg(reinterpret_cast<const float2*>(p + k * step)); s.x += v.x; s.y += v.y; }
    store_rows2<T>(a.seg, a.nseg, a.softcap, nullptr, tok, a.start + tok, row, a.M, s.x, s.y);
}

// The cost of a choice: full rounds, then the tail in one round of shorter items, each with its partial sums.  A tile costs the operand
// rows it fetches, 128 of weights and width / 2 of tokens per CTA: at width 256 fetching them from L2 and multiplying take about the same
// time (9472 x 2560 over 2048 tokens: 74.0 us, 70.9 without the weight loads, 1342 TFLOP/s; counted by width alone, 21632 x 2560 went to
// tiles of 160 tokens and took 241 us).
static void gp_pick(int tiles_m, int N, int k_tiles, int n_pairs, bool may_split, GpArgs& p) {
    double best = 1e30;
    for (int c = GP_TOKENS; c >= 16; c -= 16) {
        const int tn = (N + c - 1) / c, width = ((N + tn - 1) / tn + 15) & ~15, tiles = tiles_m * tn, rounds = tiles / n_pairs, tail = tiles - rounds * n_pairs;
        int ks = 1;
        if (tail > 0 && may_split) {
            ks = n_pairs / tail;
            if (ks > k_tiles / 8) ks = k_tiles / 8;
            if (ks > 16) ks = 16;
            if (ks < 1) ks = 1;
        }
        const double fixed = 8.0 / k_tiles, cost = (rounds + (tail == 0 ? 0.0 : 1.0 / ks + (ks > 1 ? fixed + 0.02 * ks : 0.0)) + fixed) * (128 + width / 2);
        if (cost < best - 1e-9) {
            best = cost;
            p.n_tile = p.width = width; p.tiles_n = (N + width - 1) / width; p.ksplit = ks;
            const int all = tiles_m * p.tiles_n;
            p.n_full = ks > 1 ? all / n_pairs * n_pairs : all;
            p.n_items = p.n_full + (all - p.n_full) * ks;
        }
    }
}

size_t gemm_pair_part_floats() { DeviceCtx* c = ctx(); return c ? (size_t)(c->sm_count / 2) * 256 * GP_TOKENS : 0; }

// 16-bit operands, one matrix, no gate / up maps: everything else stays with dense_tc.cu.
bool gemm_pair_applies(const DenseGemm& a) {
    return (a.kind == EK_BF16 || a.kind == EK_F16) && !a.swiglu && !a.off && a.n_groups == 1 && a.N >= GP_MIN_TOKENS && a.M >= 256;
}

// One round of pairs without K ranges: the one-CTA kernel spreads the same rows over twice as many, narrower tiles and starts faster
// (2560 x 9728 over 256 / 1024 tokens 49 / 54 us there, 58 / 61 here; 6144 x 2560 over 512: 19.3 and 22.2).  From a second round on, or where its
// tiles would be wider than 192 tokens, the pairs gain (21632 x 2560 over 160 tokens 38.0 against 44.2, 12288 x 2560 over 256: 23.5 and 30.2).
bool gemm_pair_one_round(const DenseGemm& a) {
    DeviceCtx* c = ctx();
    if (!c) return false;
    GpArgs p = {};
    gp_pick((a.M + 255) / 256, a.N, (a.K + GP_K - 1) / GP_K, c->sm_count / 2, a.part != nullptr && a.part_floats >= gemm_pair_part_floats(), p);
    return p.ksplit == 1 && p.n_items <= c->sm_count / 2;
}

int launch_gemm_pair(const DenseGemm& a, cudaStream_t st, const std::function<int()>& behind) {
    DeviceCtx* c = ctx();
    if (!c) return set_error(JB_ERR_STATE, "paired gemm: library not initialised");
    if (!a.W || !a.x) return set_error(JB_ERR_PTR, "paired gemm: null pointer");
    if (a.K <= 0) return set_error(JB_ERR_LIMIT, "paired gemm: K=%d", a.K);
    GpArgs p = {};
    p.start = a.start; p.nseg = a.nseg; p.M = a.M; p.N = a.N; p.softcap = a.softcap; p.status = c->d_status; p.part = a.part;
    for (int i = 0; i < MAX_SEG; ++i) p.seg[i] = a.seg[i];
    p.vec = rows4_aligned(a.seg, a.nseg, a.M, 0);
    p.k_tiles = (a.K + GP_K - 1) / GP_K;
    const int n_pairs = c->sm_count / 2;
    gp_pick((a.M + 255) / 256, a.N, p.k_tiles, n_pairs, a.part != nullptr && a.part_floats >= gemm_pair_part_floats(), p);
    CUtensorMap wm, xm;
    const CUtensorMapDataType dt = a.kind == EK_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const long long ldw = a.ldw > 0 ? a.ldw : pad8(a.K), ldx = a.ldx > 0 ? a.ldx : pad8(a.K);
    if (!encode_tile_map(&wm, dt, a.W, a.M, a.K, ldw, GP_M) || !encode_tile_map(&xm, dt, a.x, a.N, a.K, ldx, p.n_tile / 2))
        return set_error(JB_ERR_CUDA, "paired gemm: tensor map refused (M=%d N=%d K=%d)", a.M, a.N, a.K);
    const bool half = a.kind == EK_F16;
    void (*kern)(CUtensorMap, CUtensorMap, GpArgs) = half ? gemm_pair_kernel<__half> : gemm_pair_kernel<__nv_bfloat16>;
    if (!c->gemm_pair_attr[half]) {
        JB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM));
        c->gemm_pair_attr[half] = true;
    }
    const dim3 grid(2u * (unsigned)(p.n_items < n_pairs ? p.n_items : n_pairs));
    JB_CUDA(launch_k(kern, grid, dim3(GP_THREADS), GP_SMEM, st, pdl_enabled(), wm, xm, p));
    count_launch();
    if (behind) { const int rc = behind(); if (rc) return rc; }
    if (p.ksplit > 1) {
        const dim3 g((p.width + 1) / 2, (p.n_items - p.n_full) / p.ksplit);
        if (half) JB_CUDA(launch_k(gemm_pair_sum_kernel<__half>, g, dim3(256), 0, st, pdl_enabled(), p));
        else      JB_CUDA(launch_k(gemm_pair_sum_kernel<__nv_bfloat16>, g, dim3(256), 0, st, pdl_enabled(), p));
        count_launch();
    }
    return JB_OK;
}

}  // namespace jb
