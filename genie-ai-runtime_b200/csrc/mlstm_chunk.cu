// mlstm_chunk.cu — the mLSTM recurrence of a prompt in chunks of 128 tokens on the 5th-generation tensor cores.
//
// Within a chunk, with F the running sum of the log forget gates, A_s = i_s - F_s, M_t = max(m_0, max of A_s for s <= t) and m_0
// the maximum carried in, the recurrence unrolls to
//     m_t = F_t + M_t
//     o_t ~ e^(m_0 - M_t) S_0^T q_t + sum_{s <= t} e^(A_s - M_t) (q_t . k_s) v_s        (its denominator alike, with n and ones)
//     S_L = e^(m_0 - M_L) S_0 + sum_s e^(A_s - M_L) k_s v_s^T
// A CTA owns one head and 32 value columns and walks the chunks in order.  Only S passes from chunk to chunk: everything else of a chunk is done
// by warps that run ahead of it or behind it,
//     warp 0 TMA, 1 MMA issuer, 2 and 3 the gates of every second chunk (F, A and M in fp64, handed on as two floats each);
//     4-11 the scores' weights: a thread reads half of its token's scores from tensor memory and puts the weighted ones back in their place;
//     12-19 the state: a thread holds 32 columns of a row of S in registers, adds the chunk's part and lays the row out for the next product; n . q;
//     20-23 n, and the outputs, a thread per token; 24 issues the products of the weights and the values.
// q, k and v are bf16 as the projections left them; every fp32 operand of a product (the weighted scores, the weighted values, the state) goes in as
// two bf16 parts, its rounding and the remainder, so the products keep about 16 bits of mantissa and nothing fp32 is cut to bf16.
// q and k lie as TMA brings them, [token][dim]: K-major for the scores and q S, MN-major as the A operand of k^T v.  Every mbarrier wait is bounded.
#include "mlstm.cuh"
#include "mma.cuh"
#include "tc.cuh"

namespace jb {

constexpr int MC_L = 128, MC_V = 32, MC_THREADS = 800, MC_MAX_DIM = 256;
constexpr uint32_t MC_TILE = MC_L * 128;                               // bytes of 64 columns of a chunk's rows
// tensor memory: two buffers of scores, 128 columns, over which their weights are written (16 tokens: 8 columns of first parts, 8 of second);
// q S, the chunk's own part of the outputs, k^T v of 128 dimensions each (first parts | second parts, 64 columns)
constexpr uint32_t MC_TM_SC = 0, MC_TM_QS = 256, MC_TM_PV = 320, MC_TM_U = 384;

// A, M: as two floats, in units of log2 (M less the logarithm of the scores' scale over MC_LOW); a = e^(m_0 - M_t), w = e^(A_s - M_L), em = e^(-m_t)
struct alignas(16) McGates { float2 A[MC_L], M[MC_L]; float a[MC_L], w[MC_L], em[MC_L], decay; };
struct McArgs { MlstmCall c; int n, start; int* status; };

__device__ __forceinline__ float2 mc_two(double x) { const float hi = (float)x; return make_float2(hi, (float)(x - (double)hi)); }
// e^(A - M) times the scores' scale, times 1 / MC_LOW, by which the score it weighs is multiplied first: their product may be a subnormal number, which the
// exponential alone (2^x to 2^-22, zero below 2^-126; its other form takes four instructions in place of one) would leave out
constexpr float MC_LOW = 1.0f / (1 << 24);
__device__ __forceinline__ float mc_weight(float Ax, float Ay, float2 M) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((Ax - M.x) + (Ay - M.y))); return y; }
__device__ __forceinline__ void mc_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    hi = fa_pack(x, y);
    lo = fa_pack(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xFFFF0000u));
}
__device__ __forceinline__ void mc_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}
// 16 columns each, without waiting
__device__ __forceinline__ void mc_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
__device__ __forceinline__ void mc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mc_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
// tc_wait with polls that may be suspended for a microsecond: two dozen warps that poll as often as they can take a third of the issue slots
__device__ __forceinline__ bool mc_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    unsigned long long t0 = 0;
    for (uint32_t i = 0; i < TC_WAIT_LIMIT; ++i) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(addr), "r"(parity), "r"(1000u) : "memory");
        if (ok) return true;
        if ((i & 63u) == 63u) {
            const unsigned long long t = global_ns();
            if (!t0) t0 = t; else if (t - t0 > 2000000000ull) return false;
        }
    }
    return false;
}
// whether the phase is over: one poll
__device__ __forceinline__ bool mc_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(50u) : "memory");
    return ok != 0;
}
// 16 bytes of row r of a swizzled tile of 128-byte rows
__device__ __forceinline__ uint32_t mc_at(uint32_t base, int r, int c) { return base + (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }
__device__ __forceinline__ uint4 mc_lds(uint32_t addr) {
    uint4 x;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(addr));
    return x;
}
__device__ __forceinline__ void mc_sts(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Gates of the chunk's `valid` tokens from t0 on, four to a lane of one warp; scale: log2 of the scores' scale; take(m): the maximum carried in, give(m): the one carried on, and g is free
template <class Take, class Give>
__device__ __forceinline__ bool mc_gates(const MlstmCall& c, int h, int t0, int valid, double scale, McGates* g, Take take, Give give) {
    constexpr double LOG2E = 1.4426950408889634074;
    const int lane = threadIdx.x & 31;
    double F[4], a[4];
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int t = 4 * lane + e, at = t0 + min(t, valid - 1);
        const float f = mlstm_log_f(c, at, h), i = mlstm_log_i(c, at, h);
        F[e] = t < valid ? (double)f : 0.0;
        a[e] = t < valid ? (double)i : -1e30;
    }
    #pragma unroll
    for (int e = 1; e < 4; ++e) F[e] += F[e - 1];
    double sum = F[3];                                              // inclusive sums over lanes
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(0xFFFFFFFFu, sum, o); if (lane >= o) sum += u; }
    const double FL = __shfl_sync(0xFFFFFFFFu, sum, 31);
    sum = __shfl_up_sync(0xFFFFFFFFu, sum, 1);
    if (lane == 0) sum = 0.0;
    double M = -1e30;
    #pragma unroll
    for (int e = 0; e < 4; ++e) { F[e] += sum; a[e] -= F[e]; M = fmax(M, a[e]); }
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(0xFFFFFFFFu, M, o); if (lane >= o) M = fmax(M, u); }
    const double top = __shfl_sync(0xFFFFFFFFu, M, 31);
    M = __shfl_up_sync(0xFFFFFFFFu, M, 1);
    double m;
    if (!take(m)) return false;
    const double ML = fmax(m, top);
    if (!give(FL + ML)) return false;
    double Mt = lane == 0 ? m : fmax(m, M);
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int t = 4 * lane + e;
        Mt = fmax(Mt, a[e]);
        g->A[t] = mc_two(a[e] * LOG2E); g->M[t] = mc_two(fma(Mt, LOG2E, -scale - 24.0));
        g->a[t] = expf((float)(m - Mt));
        g->w[t] = t < valid ? expf((float)(a[e] - ML)) : 0.f;
        g->em[t] = expf((float)(-(F[e] + Mt)));
    }
    if (lane == 0) g->decay = expf((float)(m - ML));
    return true;
}

// KC: chunks of 64 dimensions, 2 or 4
template <int KC> struct McLayout {
    static constexpr uint32_t q = 0, k = q + KC * MC_TILE, v = k + KC * MC_TILE, vw = v + 2 * MC_TILE, s = vw + MC_TILE, g = s + KC * 64 * 128,
                              n = g + ((2 * (uint32_t)sizeof(McGates) + 127) & ~127u), sum = n + 2 * KC * 64 * 4, nq = sum + 4 * MC_L * 4, bytes = nq + 4 * MC_L * 4;
};

// WHOLE: outputs lie at 16-byte boundaries, else at 8-byte ones
template <int KC, bool WHOLE>
__global__ void __launch_bounds__(MC_THREADS, 1) mlstm_chunk_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                                                                    const __grid_constant__ CUtensorMap vmap, const __grid_constant__ McArgs p) {
    extern __shared__ uint8_t mc_raw[];
    // One phase per chunk, those in pairs one per two chunks: no phase completes before all who wait for the one before have seen that one.
    __shared__ uint64_t q_full, k_full, v_full[2], q_free, k_free, v_free[2], g_full[2], g_free[2], sc_full[2], p_full[2], r_full[2], vw_full, u_done, s_full, qs_done, o_done, o_free, m_full, n_full[2], nq_done[2], drain[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int fail;
    __shared__ volatile double m_next;                               // the maximum carried into the next chunk
    __shared__ volatile int odd[2];                                  // last chunk + 1 whose values hold an infinity or NaN
    using L = McLayout<KC>;
    const MlstmCall& c = p.c;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y, v0 = blockIdx.x * MC_V;
    uint8_t* base = mc_raw + ((1024u - (smem_u32(mc_raw) & 1023u)) & 1023u);
    const uint32_t sm = smem_u32(base);
    McGates* gates = reinterpret_cast<McGates*>(base + L::g);
    float* ns = reinterpret_cast<float*>(base + L::n);                  // [buffer][dimension]
    float* rsum = reinterpret_cast<float*>(base + L::sum);              // [buffer][half][token]: sums of the weights, n . q
    float* nq = reinterpret_cast<float*>(base + L::nq);
    const int D = c.dim, vld = pad8(c.vdim), chunks = (p.n + MC_L - 1) / MC_L;
    float* Sg = c.state + (size_t)h * D * vld;
    float* ng = c.state + (size_t)c.heads * D * vld + (size_t)h * D;
    float* mg = c.state + (size_t)c.heads * D * vld + (size_t)c.heads * D + h;
    const bool fresh = p.start == 0;
    const float qscale = 1.0f / sqrtf((float)D);
    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1); mbar_init(&k_full, 1); mbar_init(&q_free, 9); mbar_init(&k_free, 5);
        for (int b = 0; b < 2; ++b) { mbar_init(&v_full[b], 1); mbar_init(&v_free[b], 13); mbar_init(&g_full[b], 1); mbar_init(&g_free[b], 20); mbar_init(&sc_full[b], 1); mbar_init(&p_full[b], 8); mbar_init(&r_full[b], 16); odd[b] = 0; }
        mbar_init(&vw_full, 8); mbar_init(&u_done, 1); mbar_init(&s_full, 8);
        mbar_init(&qs_done, 1); mbar_init(&o_done, 1); mbar_init(&o_free, 4); mbar_init(&m_full, 1); for (int b = 0; b < 2; ++b) { mbar_init(&n_full[b], 4); mbar_init(&nq_done[b], 8); } mbar_init(&drain[0], 1); mbar_init(&drain[1], 1);
        fence_mbar_init();
        fail = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();
    pdl_launch();
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    constexpr uint32_t kind = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 4) << 24), amn = 1u << 15, bmn = 1u << 16, n64 = (uint32_t)(64 >> 3) << 17, n128 = (uint32_t)(128 >> 3) << 17;
    // a warp's wait: false on all lanes when it ran out or another role gave up
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
        const bool ok = __all_sync(0xFFFFFFFFu, mc_wait(bar, parity) && !fail);
        __syncwarp();
        if (!ok && lane == 0) tc_fail(&fail, p.status);
        return ok;
    };
    auto arrive = [&](uint64_t* bar) { __syncwarp(); if (lane == 0) mbar_arrive(bar); __syncwarp(); };

    if (warp == 0) {
        if (lane == 0) {
            int ch[3] = {0, 0, 0};                                   // chunks of q, k and v requested: each as soon as its place is free
            unsigned long long since = global_ns();
            for (uint32_t i = 1; ch[0] + ch[1] + ch[2] < 3 * chunks && !fail; ++i) {
                bool got = false;
                if (ch[2] < chunks && mc_test(&v_free[ch[2] & 1], ((ch[2] >> 1) & 1) ^ 1)) {
                    const int b = ch[2] & 1;
                    mbar_expect_tx(&v_full[b], MC_TILE);
                    mc_load_3d(sm + L::v + b * MC_TILE, &vmap, v0, ch[2]++ * MC_L, h, &v_full[b]);
                    got = true;
                }
                if (ch[0] < chunks && mc_test(&q_free, (ch[0] & 1) ^ 1)) {
                    mbar_expect_tx(&q_full, KC * MC_TILE);
                    for (int k = 0; k < KC; ++k) mc_load_3d(sm + L::q + k * MC_TILE, &qmap, 64 * k, ch[0] * MC_L, h, &q_full);
                    ++ch[0];
                    got = true;
                }
                if (ch[1] < chunks && mc_test(&k_free, (ch[1] & 1) ^ 1)) {
                    mbar_expect_tx(&k_full, KC * MC_TILE);
                    for (int k = 0; k < KC; ++k) mc_load_3d(sm + L::k + k * MC_TILE, &kmap, 64 * k, ch[1] * MC_L, h, &k_full);
                    ++ch[1];
                    got = true;
                }
                if (got) since = global_ns();
                else if ((i & 63u) == 0 && global_ns() - since > 2000000000ull) break;
            }
            if (ch[0] + ch[1] + ch[2] < 3 * chunks) tc_fail(&fail, p.status);
            // its own copies are not in flight when it leaves
            if (ch[0] > 0) tc_wait(&q_full, (ch[0] - 1) & 1);
            if (ch[1] > 0) tc_wait(&k_full, (ch[1] - 1) & 1);
            for (int i = max(0, ch[2] - 2); i < ch[2]; ++i) tc_wait(&v_full[i & 1], (i >> 1) & 1);
        }
    } else if (warp == 1) {
        // The whole warp runs the loop (its values are then uniform), one lane waits and issues; a wait that ran out leaves it idle for the rest.
        const bool leader = tc_elect();
        const uint32_t qd = tc_desc_lo(sm + L::q), kd = tc_desc_lo(sm + L::k), wd = tc_desc_lo(sm + L::vw), sd = tc_desc_lo(sm + L::s);
        const uint32_t kt = ((sm + L::k) >> 4 & 0x3FFFu) | (MC_TILE >> 4) << 16;      // MN-major: 64 dimensions a tile, the next ones in the tile behind
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            if (leader && ok && !tc_wait(bar, parity)) { ok = false; tc_fail(&fail, p.status); }
            __syncwarp();
        };
        for (int ch = -1; ch < chunks; ++ch) {
            const uint32_t par = ch & 1;
            if (ch >= 0) {
                wait(&vw_full, par);
                if (leader && ok) {
                    tc_fence_after();
                    #pragma unroll 1
                    for (int k = 0; k < MC_L / 16; ++k)
                        #pragma unroll
                        for (int m = 0; m < KC / 2; ++m)
                            tc_mma_ss(tmem + MC_TM_U + 64 * m, kt + (uint32_t)(2 * m * (MC_TILE >> 4) + k * (2048 >> 4)), TC_DESC_HI, wd + (uint32_t)(k * (2048 >> 4)), TC_DESC_HI, kind | amn | bmn | n64, (uint32_t)(k != 0));
                    tc_commit(&u_done);
                    tc_commit(&k_free);
                }
                __syncwarp();
                if (ch > 0) wait(&o_free, par ^ 1);                  // the outputs of the chunk before have been read, and so its weights used
                wait(&s_full, par);
                if (leader && ok) {
                    tc_fence_after();
                    #pragma unroll 1
                    for (int k = 0; k < 4 * KC; ++k)
                        tc_mma_ss(tmem + MC_TM_QS, qd + (uint32_t)((k >> 2) * (MC_TILE >> 4) + 2 * (k & 3)), TC_DESC_HI, sd + (uint32_t)(k * (2048 >> 4)), TC_DESC_HI, kind | bmn | n64, (uint32_t)(k != 0));
                    tc_commit(&qs_done);
                    tc_commit(&q_free);
                }
                __syncwarp();
            }
            if (ch + 1 < chunks) {
                wait(&q_full, par ^ 1);
                wait(&k_full, par ^ 1);
                if (leader && ok) {
                    tc_fence_after();
                    #pragma unroll 1
                    for (int k = 0; k < 4 * KC; ++k) {
                        const uint32_t o = (uint32_t)((k >> 2) * (MC_TILE >> 4) + 2 * (k & 3));
                        tc_mma_ss(tmem + MC_TM_SC + ((ch + 1) & 1) * 128u, qd + o, TC_DESC_HI, kd + o, TC_DESC_HI, kind | n128, (uint32_t)(k != 0));
                    }
                    tc_commit(&sc_full[(ch + 1) & 1]);
                }
                __syncwarp();
            }
        }
        // nothing of this CTA may still be running on the tensor pipe when the columns are freed
        if (leader) { tc_commit(&drain[0]); tc_wait(&drain[0], 0); }
    } else if (warp < 4) {
        const double scale = -0.5 * log2((double)D);                 // of the scores, dim^-1/2
        for (int ch = warp - 2; ch < chunks; ch += 2) {
            const int b = ch & 1;
            const bool ok = mc_gates(c, h, ch * MC_L, min(MC_L, p.n - ch * MC_L), scale, &gates[b],
                [&](double& m) {
                    if (ch > 0 && !wait_all(&m_full, (ch & 1) ^ 1)) return false;
                    m = ch > 0 ? m_next : fresh ? 0.0 : (double)*mg;
                    return true;
                },
                [&](double m) {
                    __syncwarp();
                    if (lane == 0) {
                        m_next = m;
                        // other slices may still have to read n and m: the new ones wait beside them for the launch that follows
                        if (ch + 1 == chunks && blockIdx.x == 0) mg[mlstm_next(c)] = (float)m;
                    }
                    arrive(&m_full);
                    return wait_all(&g_free[b], ((ch >> 1) & 1) ^ 1);
                });
            if (!ok) break;
            arrive(&g_full[b]);
        }
    } else if (warp >= 4 && warp < 12) {
        const int q = warp & 3, t = q * 32 + lane, part = (warp - 4) >> 2;       // two warps a quarter of the tokens, every other 16 columns each
        for (int ch = 0; ch < chunks; ++ch) {
            const int b = ch & 1;
            const McGates& g = gates[b];
            if (!wait_all(&g_full[b], (ch >> 1) & 1) || !wait_all(&sc_full[b], (ch >> 1) & 1)) break;
            tc_fence_after();
            const float2 Mt = g.M[t];
            const uint32_t sc = tmem + MC_TM_SC + b * 128u + ((uint32_t)(q * 32) << 16);
            float sum[2] = {0.f, 0.f};
            #pragma unroll 1
            for (int j = part; j < 8; j += 2) {                      // columns 16 j ..; rolled, as everything here: unrolled, the roles' code is fetched more slowly than it runs
                uint32_t x[16];                                      // scores; then first and second parts of the weighted ones
                __syncwarp();
                if (j <= 2 * q + 1) {
                    mc_ld16(sc + 16u * j, x);
                    mc_ld_wait();
                    float v[16];
                    #pragma unroll
                    for (int i = 0; i < 16; i += 2) {                // those of later tokens too: a branch around each would leave them one behind another
                        const float4 A = *reinterpret_cast<const float4*>(&g.A[16 * j + i]);
                        v[i] = (__uint_as_float(x[i]) * MC_LOW) * mc_weight(A.x, A.y, Mt);
                        v[i + 1] = (__uint_as_float(x[i + 1]) * MC_LOW) * mc_weight(A.z, A.w, Mt);
                    }
                    if (j >= 2 * q) {                                // later tokens weigh nothing
                        #pragma unroll
                        for (int i = 0; i < 16; ++i) if (16 * j + i > t) v[i] = 0.f;
                    }
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        sum[0] += v[2 * i]; sum[1] += v[2 * i + 1];
                        mc_split(v[2 * i], v[2 * i + 1], x[i], x[8 + i]);
                    }
                } else {
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) x[i] = 0u;
                }
                __syncwarp();
                mc_st16(sc + 16u * j, x);
            }
            __syncwarp();
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            rsum[(2 * b + part) * MC_L + t] = sum[0] + sum[1];
            tc_fence_before();
            arrive(&g_free[b]);
            arrive(&r_full[b]);
            arrive(&p_full[b]);
        }
    } else if (warp >= 12 && warp < 20) {
        const int m = (warp - 12) >> 2, q = warp & 3, d = m * 128 + q * 32 + lane, id = threadIdx.x - 384, r = (warp - 12) * 16 + (lane >> 1), half = lane & 1;
        const bool mine = m < KC / 2;                                // the warp's dimensions exist
        float S[MC_V];
        #pragma unroll
        for (int i = 0; i < MC_V / 4; ++i) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!fresh && mine && d < D && v0 + 4 * i < vld) x = *reinterpret_cast<const float4*>(Sg + (size_t)d * vld + v0 + 4 * i);
            S[4 * i] = x.x; S[4 * i + 1] = x.y; S[4 * i + 2] = x.z; S[4 * i + 3] = x.w;
        }
        auto put_state = [&]() {                                     // the state as two bf16 parts for the next product
            if (mine) {
                #pragma unroll
                for (int i = 0; i < MC_V / 8; ++i) {
                    uint32_t hi[4], lo[4];
                    #pragma unroll
                    for (int e = 0; e < 4; ++e) mc_split(S[8 * i + 2 * e], S[8 * i + 2 * e + 1], hi[e], lo[e]);
                    mc_sts(mc_at(sm + L::s, d, i), hi[0], hi[1], hi[2], hi[3]);
                    mc_sts(mc_at(sm + L::s, d, 4 + i), lo[0], lo[1], lo[2], lo[3]);
                }
            }
            fence_proxy_async();
            arrive(&s_full);
        };
        put_state();
        int ch = 0;
        for (; ch < chunks; ++ch) {
            const int b = ch & 1;
            const McGates& g = gates[b];
            if (!wait_all(&g_full[b], (ch >> 1) & 1) || !wait_all(&v_full[b], (ch >> 1) & 1)) break;
            const float w = g.w[r], decay = g.decay;
            bool finite = true;
            #pragma unroll
            for (int i = 0; i < 2; ++i) {                            // values weighted for the state; those of the chunk before have been used
                const int cc = 2 * half + i;
                const uint4 x4 = mc_lds(mc_at(sm + L::v + b * MC_TILE, r, cc));
                const uint32_t x[4] = {x4.x, x4.y, x4.z, x4.w};
                uint32_t hi[4], lo[4];
                #pragma unroll
                for (int e = 0; e < 4; ++e) {
                    finite = finite && (x[e] & 0x7F80u) != 0x7F80u && (x[e] & 0x7F800000u) != 0x7F800000u;
                    mc_split(w * __uint_as_float(x[e] << 16), w * __uint_as_float(x[e] & 0xFFFF0000u), hi[e], lo[e]);
                }
                mc_sts(mc_at(sm + L::vw, r, cc), hi[0], hi[1], hi[2], hi[3]);
                mc_sts(mc_at(sm + L::vw, r, 4 + cc), lo[0], lo[1], lo[2], lo[3]);
            }
            if (!finite) odd[b] = ch + 1;
            fence_proxy_async();
            arrive(&v_free[b]);
            arrive(&vw_full);
            arrive(&g_free[b]);
            if (!wait_all(&q_full, ch & 1) || !wait_all(&n_full[b], (ch >> 1) & 1)) break;
            {                                                        // n . q of the carried normaliser: a token and half of the dimensions a thread
                const int t = id & 127, part = id >> 7;
                const float* n = ns + b * KC * 64;
                float dot[2] = {0.f, 0.f};
                #pragma unroll 2
                for (int i = 4 * KC * part; i < 4 * KC * (part + 1); ++i) {
                    const uint4 x = mc_lds(mc_at(sm + L::q + (i >> 3) * MC_TILE, t, i & 7));
                    const float4 n0 = load4(n + 8 * i), n1 = load4(n + 8 * i + 4);
                    dot[0] = fmaf(n0.x, __uint_as_float(x.x << 16), dot[0]); dot[1] = fmaf(n0.y, __uint_as_float(x.x & 0xFFFF0000u), dot[1]);
                    dot[0] = fmaf(n0.z, __uint_as_float(x.y << 16), dot[0]); dot[1] = fmaf(n0.w, __uint_as_float(x.y & 0xFFFF0000u), dot[1]);
                    dot[0] = fmaf(n1.x, __uint_as_float(x.z << 16), dot[0]); dot[1] = fmaf(n1.y, __uint_as_float(x.z & 0xFFFF0000u), dot[1]);
                    dot[0] = fmaf(n1.z, __uint_as_float(x.w << 16), dot[0]); dot[1] = fmaf(n1.w, __uint_as_float(x.w & 0xFFFF0000u), dot[1]);
                }
                nq[(2 * b + part) * MC_L + t] = dot[0] + dot[1];
                arrive(&q_free);
                arrive(&nq_done[b]);
                arrive(&r_full[b]);
            }
            if (!wait_all(&u_done, ch & 1)) break;
            tc_fence_after();
            if (mine) {
                const uint32_t u = tmem + MC_TM_U + 64u * m + ((uint32_t)(q * 32) << 16);
                #pragma unroll
                for (int k = 0; k < MC_V; k += 16) {
                    uint32_t x[16], y[16];
                    __syncwarp();
                    mc_ld16(u + k, x);
                    mc_ld16(u + 32u + k, y);
                    mc_ld_wait();
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) S[k + i] = fmaf(S[k + i], decay, __uint_as_float(x[i]) + __uint_as_float(y[i]));
                }
            }
            tc_fence_before();
            if (ch + 1 < chunks) {
                if (!wait_all(&qs_done, ch & 1)) break;
                put_state();
            }
        }
        if (ch == chunks && mine && d < D) {
            #pragma unroll
            for (int i = 0; i < MC_V / 4; ++i)
                if (v0 + 4 * i < vld) *reinterpret_cast<float4*>(Sg + (size_t)d * vld + v0 + 4 * i) = make_float4(S[4 * i], S[4 * i + 1], S[4 * i + 2], S[4 * i + 3]);
        }
    } else if (warp >= 20 && warp < 24) {
        const int q = warp & 3, t = q * 32 + lane;
        auto all = [&](bool ok) {
            int x;
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n" : "=r"(x) : "r"((int)ok) : "memory");
            return x != 0;
        };
        const int id = threadIdx.x - 640;
        for (int i = id; i < KC * 64; i += 128) ns[i] = !fresh && i < D ? ng[i] : 0.f;
        arrive(&n_full[0]);
        int ch = 0;
        for (; ch < chunks; ++ch) {
            const int b = ch & 1, t0 = ch * MC_L;
            const McGates& g = gates[b];
            if (!all(wait_all(&g_full[b], (ch >> 1) & 1) && wait_all(&k_full, ch & 1) && (ch == 0 || wait_all(&nq_done[b ^ 1], ((ch - 1) >> 1) & 1)))) break;
            __syncwarp();
            if (id < 32 * KC) {                                      // n, two dimensions a thread: into the buffer whose n . q is done
                const uint32_t col = sm + L::k + (uint32_t)(id >> 5) * MC_TILE + (uint32_t)(id & 3) * 4;
                uint32_t at[8];                                      // of the rows of an eight
                #pragma unroll
                for (int e = 0; e < 8; ++e) at[e] = mc_at(col, e, (id & 31) >> 2);
                float n0[2] = {0.f, 0.f}, n1[2] = {0.f, 0.f};
                #pragma unroll 1
                for (int s = 0; s < MC_L; s += 8) {
                    const float4 wa = load4(&g.w[s]), wb = load4(&g.w[s + 4]);
                    const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
                    #pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        uint32_t x;
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x) : "r"(at[e] + s * 128));
                        n0[e & 1] = fmaf(w[e], __uint_as_float(x << 16), n0[e & 1]);
                        n1[e & 1] = fmaf(w[e], __uint_as_float(x & 0xFFFF0000u), n1[e & 1]);
                    }
                }
                const float2 old = reinterpret_cast<const float2*>(ns + b * KC * 64)[id];
                reinterpret_cast<float2*>(ns + (b ^ 1) * KC * 64)[id] = make_float2(fmaf(old.x, g.decay, n0[0] + n0[1]), fmaf(old.y, g.decay, n1[0] + n1[1]));
            }
            arrive(&n_full[b ^ 1]);
            arrive(&k_free);
            if (!all(wait_all(&qs_done, ch & 1) && wait_all(&r_full[b], (ch >> 1) & 1) && wait_all(&o_done, ch & 1))) break;
            tc_fence_after();
            __syncwarp();
            const uint32_t row = tmem + ((uint32_t)(q * 32) << 16);
            const float a = g.a[t], f = qscale * a;
            const bool by_product = odd[b] != ch + 1;
            float o[MC_V];
            #pragma unroll
            for (int k = 0; k < MC_V; k += 16) {
                uint32_t x[16], y[16];
                __syncwarp();
                mc_ld16(row + MC_TM_QS + k, x);
                mc_ld16(row + MC_TM_QS + 32u + k, y);
                mc_ld_wait();
                #pragma unroll
                for (int i = 0; i < 16; ++i) o[k + i] = (__uint_as_float(x[i]) + __uint_as_float(y[i])) * f;
                if (by_product) {
                    __syncwarp();
                    mc_ld16(row + MC_TM_PV + k, x);
                    mc_ld_wait();
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) o[k + i] += __uint_as_float(x[i]);
                }
            }
            if (!by_product) {                                       // a weight of zero times an infinity or NaN of a later token: not by the product
                #pragma unroll 1
                for (int j = 0; j < 8; ++j) {
                    uint32_t x[16];
                    __syncwarp();
                    mc_ld16(row + MC_TM_SC + b * 128u + 16u * j, x);
                    mc_ld_wait();
                    #pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const int s = 16 * j + e;
                        const uint32_t hi = x[e >> 1], lo = x[8 + (e >> 1)];
                        const float wt = e & 1 ? __uint_as_float(hi & 0xFFFF0000u) + __uint_as_float(lo & 0xFFFF0000u) : __uint_as_float(hi << 16) + __uint_as_float(lo << 16);
                        if (s <= t) {
                            #pragma unroll
                            for (int i = 0; i < MC_V / 8; ++i) {
                                const uint4 v = mc_lds(mc_at(sm + L::v + b * MC_TILE, s, i));
                                const uint32_t y[4] = {v.x, v.y, v.z, v.w};
                                #pragma unroll
                                for (int k = 0; k < 4; ++k) { o[8 * i + 2 * k] = fmaf(wt, __uint_as_float(y[k] << 16), o[8 * i + 2 * k]); o[8 * i + 2 * k + 1] = fmaf(wt, __uint_as_float(y[k] & 0xFFFF0000u), o[8 * i + 2 * k + 1]); }
                            }
                        }
                    }
                }
            }
            const int at = 2 * b * MC_L + t;
            const float z = a * ((nq[at] + nq[at + MC_L]) * qscale) + (rsum[at] + rsum[at + MC_L]), inv = 1.0f / (fmaxf(fabsf(z), g.em[t]) + 1e-6f);
            tc_fence_before();
            arrive(&o_free);
            arrive(&g_free[b]);
            if (!by_product) all(true);                              // other warps read the values too; for all of them it is one way or the other
            // turned through the values' place, where they have been used by now: rows of 128 bytes, each warp its own
            const uint32_t st = sm + L::v + b * MC_TILE;
            __syncwarp();
            #pragma unroll
            for (int i = 0; i < MC_V / 4; ++i)
                mc_sts(mc_at(st, t, i), __float_as_uint(o[4 * i] * inv), __float_as_uint(o[4 * i + 1] * inv), __float_as_uint(o[4 * i + 2] * inv), __float_as_uint(o[4 * i + 3] * inv));
            __syncwarp();
            uint4 y[8];
            #pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = mc_lds(mc_at(st, q * 32 + 4 * i + (lane >> 3), lane & 7));
            fence_proxy_async();
            arrive(&v_free[b]);
            const int r = t0 + q * 32 + (lane >> 3), col = v0 + 4 * (lane & 7);
            float* out = c.raw + ((size_t)r * c.heads + h) * c.vdim + col;
            #pragma unroll
            for (int i = 0; i < 8; ++i)
                if (r + 4 * i < p.n && col < c.vdim) {
                    float* o4 = out + (size_t)(4 * i) * c.heads * c.vdim;
                    if (WHOLE) *reinterpret_cast<uint4*>(o4) = y[i];
                    else { *reinterpret_cast<uint2*>(o4) = make_uint2(y[i].x, y[i].y); *reinterpret_cast<uint2*>(o4 + 2) = make_uint2(y[i].z, y[i].w); }
                }
            __syncwarp();
        }
        if (ch == chunks && blockIdx.x == 0 && id < 32 * KC)         // what the thread itself wrote
            for (int i = 2 * id; i < min(2 * id + 2, D); ++i) ng[mlstm_next(c) + i] = ns[(chunks & 1) * KC * 64 + i];
    } else if (warp == 24) {
        // the chunk's own part of the outputs, beside the other products' issuer: neither then waits for what the other's need
        const bool leader = tc_elect();
        const uint32_t vd = tc_desc_lo(sm + L::v);
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            if (leader && ok && !tc_wait(bar, parity)) { ok = false; tc_fail(&fail, p.status); }
            __syncwarp();
        };
        for (int ch = 0; ch < chunks; ++ch) {
            const uint32_t par = ch & 1;
            if (ch > 0) wait(&o_free, par ^ 1);
            wait(&v_full[par], (ch >> 1) & 1);
            wait(&p_full[par], (ch >> 1) & 1);
            if (leader && ok) {
                tc_fence_after();
                #pragma unroll 1
                for (int k = 0; k < MC_L / 16; ++k)
                    #pragma unroll
                    for (int part = 0; part < 2; ++part)
                        tc_mma_ts(tmem + MC_TM_PV, tmem + MC_TM_SC + par * 128u + (uint32_t)(k * 16 + part * 8), vd + par * (MC_TILE >> 4) + (uint32_t)(k * (2048 >> 4)), TC_DESC_HI, kind | bmn | n64, (uint32_t)(part != 0 || k != 0));
                tc_commit(&o_done);
                tc_commit(&v_free[par]);
            }
            __syncwarp();
        }
        if (leader) { tc_commit(&drain[1]); tc_wait(&drain[1], 0); }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

bool mlstm_chunks_apply(const MlstmCall& a, int n) {
    return a.kind == EK_BF16 && n >= 16 && a.dim % 8 == 0 && a.dim <= MC_MAX_DIM && a.vdim % 8 == 0 && a.ld % 8 == 0 && a.off_q % 8 == 0 && a.off_k % 8 == 0 && a.off_v % 8 == 0 &&
           !((uintptr_t)a.proj & 15) && !((uintptr_t)a.raw & 7) && !((uintptr_t)a.state & 15) && (n <= MLSTM_SHORT || encode_tiled_fn());
}
// [head][token][column] of a part of the projections, boxes of 64 columns x a chunk, zero outside a head's columns and behind the last token
static bool mc_map(CUtensorMap* map, const MlstmCall& a, int off, int cols, int n) {
    const cuuint64_t gdim[3] = {(cuuint64_t)cols, (cuuint64_t)n, (cuuint64_t)a.heads}, gstr[2] = {(cuuint64_t)a.ld * 2, (cuuint64_t)cols * 2};
    const cuuint32_t box[3] = {64, MC_L, 1}, estr[3] = {1, 1, 1};
    return encode_tiled_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(reinterpret_cast<const __nv_bfloat16*>(a.proj)) + off, gdim, gstr, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
template <int KC, bool WHOLE>
static int mc_go(const MlstmCall& a, int n, int start, int* status, cudaStream_t st) {
    constexpr int smem = (int)McLayout<KC>::bytes + 1024;
    static bool attr = false;
    if (!attr) { JB_CUDA(cudaFuncSetAttribute(mlstm_chunk_kernel<KC, WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); attr = true; }
    CUtensorMap qm, km, vm;
    if (!mc_map(&qm, a, a.off_q, a.dim, n) || !mc_map(&km, a, a.off_k, a.dim, n) || !mc_map(&vm, a, a.off_v, a.vdim, n))
        return set_error(JB_ERR_CUDA, "mlstm chunks: tensor map refused (%d tokens, heads of %d x %d)", n, a.dim, a.vdim);
    const McArgs p = {a, n, start, status};
    JB_CUDA(launch_k(mlstm_chunk_kernel<KC, WHOLE>, dim3((a.vdim + MC_V - 1) / MC_V, a.heads), dim3(MC_THREADS), (size_t)smem, st, pdl_enabled(), qm, km, vm, p));
    count_launch();
    return JB_OK;
}
int launch_mlstm_chunks(const MlstmCall& a, int n, int start, cudaStream_t st) {
    DeviceCtx* x = ctx();
    if (!x) return set_error(JB_ERR_STATE, "mlstm chunks: library not initialised");
    if (!mlstm_chunks_apply(a, n)) return set_error(JB_ERR_ARG, "mlstm chunks: %d tokens, heads of %d x %d", n, a.dim, a.vdim);
    if (n <= MLSTM_SHORT) return launch_mlstm_short(a, n, start, st);
    if ((uintptr_t)a.raw & 15) return a.dim <= 128 ? mc_go<2, false>(a, n, start, x->d_status, st) : mc_go<4, false>(a, n, start, x->d_status, st);
    return a.dim <= 128 ? mc_go<2, true>(a, n, start, x->d_status, st) : mc_go<4, true>(a, n, start, x->d_status, st);
}

}  // namespace jb
