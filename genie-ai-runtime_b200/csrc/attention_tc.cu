// attention_tc.cu — causal prefill attention on the 5th-generation tensor cores: tcgen05.mma with scores, softmax weights and outputs
// in tensor memory.  BF16 caches (keys in one or two parts, values of their own size), and INT8 caches whose codes were widened to
// 16 bits first (exactly: a code has 7 bits), with the scale of a key applied to its scores and the scale of a value to its weights.
//
// What bounds it: the instructions and the latency of the softmax.  Per tile of 128 rows x 64 keys the products take 512 clocks (heads of
// 128; 640 at 192 / 128; 768 for int8, whose weights are two planes) and the exponentials 512 (16 per clock and SM), and neither pipe is
// half busy: 1024 tokens behind 1024 others, 32 heads of 128: 52.4 us (bf16, 32 key heads) and 77 to 80 (int8, 8 key heads, widening not
// included).  With 64-bit descriptors formed by one lane, which issues an MMA every 60 to 100 clocks, where a whole warp's uniform values let one
// go every 25, and with the scales of int8 caches fetched by every softmax thread from global memory, they took 63.3 and 88.0.
//   * a CTA owns two tiles of 128 query rows, (token, head of the group) pairs, so that one tile's products run under the other's
//     softmax and both read the same tile of 64 keys;
//   * S = Q K^T, 128 x 64 in fp32, goes to tensor memory; a thread reads its row, frees S for the next tile at once, and writes the
//     weights as the A operand of O += P V back to tensor memory: bf16 for bf16 caches, as the older kernel has it; two bf16 planes
//     (rounding and remainder, 16 bits of mantissa) for int8 caches, whose older kernel held them in 15 bits;
//   * O stays in tensor memory; it is rescaled only when a row's maximum has risen by more than 2^8 since the last time (the conditional
//     rescaling that FlashAttention-4 describes), which leaves weights and sums in range and the result unchanged up to rounding;
//   * V is read as it lies, [key][dim]: the B operand of the second product is MN-major.
// Warps: 0 TMA (int8: the scales too), 1 MMA issuer (bf16: 1 and 2, a tile each), 3 idle, 4-7 and 8-11 the softmax of the two tiles (a warp's
// index modulo 4 is its quarter of tensor memory).  Every mbarrier wait is bounded.
#include "attention.cuh"
#include "attention_general.cuh"
#include "mma.cuh"
#include "tc.cuh"

namespace jb {

constexpr int AT_ROWS = 128, AT_KEYS = 64, AT_THREADS = 384;
constexpr int AT_QCHUNK = AT_ROWS * 128, AT_KCHUNK = AT_KEYS * 128;      // bytes of 64 elements of a tile's rows
constexpr float AT_LAZY = 8.0f;
// INT8: the tile's 64 key and 64 value scales lie behind the ring
constexpr int AT_SCALES = 2 * AT_KEYS * 4;
constexpr int at_stages(int qc, int vc, bool int8) { const int s = (224 * 1024 - 2 * qc * AT_QCHUNK) / ((qc + vc) * AT_KCHUNK + (int8 ? AT_SCALES : 0)); return s > 6 ? 6 : s; }

struct AtArgs {
    void* out; int R, dim1, vdim, ldo, n_tokens, start;
    float scale; const float* sink; float qt_coef; double qt_every; const float* gate; int ldg;
    const float* ks; const float* vs; int lds;       // INT8: scales [kv head][lds]
    const __nv_bfloat16 *q, *k, *k2, *v; long long ldq, ldk, ldk2, ldv; int dim;      // BF16: what the maps describe, for at_row
    int* status;
};

__device__ __forceinline__ void at_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void at_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
                   "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
                   "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// the bits of exp2f wherever the result is at least 2^-126 (compared for every float in [-150, 16]); zero below
__device__ __forceinline__ float at_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// lower half of the descriptor of an MN-major operand tile: rows of 64 elements (128 bytes, swizzled), eight rows 1024 bytes apart, the next 64
// elements one chunk further
__device__ __forceinline__ uint32_t at_desc_mn(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | ((uint32_t)(AT_KCHUNK >> 4) << 16); }
// the warp's wait: false on every lane when it ran out or another role gave up
__device__ __forceinline__ bool at_wait(uint64_t* bar, uint32_t parity, volatile int* fail, int* status) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) { ok = tc_wait(bar, parity) && !*fail; if (!ok) tc_fail(fail, status); }
    return __shfl_sync(0xFFFFFFFFu, ok, 0) != 0;
}

__device__ __forceinline__ float at_dot8(uint4 x, uint4 y, float s) {
    const uint32_t a[4] = {x.x, x.y, x.z, x.w}, b[4] = {y.x, y.y, y.z, y.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        s = fmaf(__uint_as_float(a[i] << 16), __uint_as_float(b[i] << 16), s);
        s = fmaf(__uint_as_float(a[i] & 0xFFFF0000u), __uint_as_float(b[i] & 0xFFFF0000u), s);
    }
    return s;
}
// One output row by one warp, over the keys that the row sees and no others: for rows whose tile holds an infinite or NaN value of a
// LATER token, which the products above multiply with a weight of zero.  fsc, m: score factor and maximum in base 2; inv: 1 / sum.
__device__ __noinline__ void at_row(const AtArgs& a, int g, int tok, int head, float fsc, float m, float inv) {
    const int lane = threadIdx.x & 31, pos = a.start + tok, d0 = 4 * lane;
    const __nv_bfloat16* q = a.q + tok * a.ldq + (long long)head * a.dim;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int base = 0; base <= pos; base += 32) {
        const int key = min(base + lane, pos);
        float s = 0.f;
        for (int d = 0; d < a.dim; d += 8) {
            const __nv_bfloat16* k = d < a.dim1 ? a.k + key * a.ldk + (long long)g * a.dim1 + d : a.k2 + key * a.ldk2 + d - a.dim1;
            s = at_dot8(*reinterpret_cast<const uint4*>(q + d), *reinterpret_cast<const uint4*>(k), s);
        }
        const float p = __bfloat162float(__float2bfloat16_rn(at_exp2(s * fsc - m)));
        for (int j = 0; j < 32 && base + j <= pos; ++j) {
            const float w = __shfl_sync(0xFFFFFFFFu, p, j);
            if (d0 < a.vdim) {
                const uint2 v = *reinterpret_cast<const uint2*>(a.v + (base + j) * a.ldv + (long long)g * a.vdim + d0);
                acc[0] = fmaf(w, __uint_as_float(v.x << 16), acc[0]); acc[1] = fmaf(w, __uint_as_float(v.x & 0xFFFF0000u), acc[1]);
                acc[2] = fmaf(w, __uint_as_float(v.y << 16), acc[2]); acc[3] = fmaf(w, __uint_as_float(v.y & 0xFFFF0000u), acc[3]);
            }
        }
    }
    if (d0 < a.vdim)
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)tok * a.ldo + (size_t)head * a.vdim + d0) =
            make_uint2(fa_pack(acc[0] * inv, acc[1] * inv), fa_pack(acc[2] * inv, acc[3] * inv));
}

// QC: 64-element chunks of a query (and key) row, VC of a value row
template <int QC, int VC, bool INT8>
__global__ void __launch_bounds__(AT_THREADS, 1) attn_tc_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                                                                const __grid_constant__ CUtensorMap k2map, const __grid_constant__ CUtensorMap vmap,
                                                                const __grid_constant__ AtArgs a) {
    extern __shared__ uint8_t at_smem_raw[];
    // Waits, 12 to 20 MMAs and commits of a turn take about 1400 clocks of an issuing warp: a warp per tile where the softmax takes less (heads of
    // 128, bf16: 63 us with one, 52 with two); int8 tiles, whose softmax takes more, run better out of step behind one (77 us; 84 with two).
    constexpr int ST = at_stages(QC, VC, INT8), STAGE = (QC + VC) * AT_KCHUNK, ISSUERS = INT8 ? 1 : 2;
    __shared__ uint64_t q_full, full[ST], empty[ST], s_full[2], s_free[2], p_full[2], o_done[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = blockIdx.y;
    const uint32_t qs = (smem_u32(at_smem_raw) + 1023u) & ~1023u, ring = qs + 2 * QC * AT_QCHUNK;
    float* scales = reinterpret_cast<float*>(at_smem_raw + (ring - smem_u32(at_smem_raw)) + ST * STAGE);       // [stage][keys 64 | values 64]
    const int total = a.n_tokens * a.R, row0 = (gridDim.x - 1 - blockIdx.x) * 2 * AT_ROWS;        // longest tiles first
    const int n_keys = a.start + (min(row0 + 2 * AT_ROWS, total) - 1) / a.R + 1, tiles = (n_keys + AT_KEYS - 1) / AT_KEYS;

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1);
        for (int s = 0; s < ST; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], ISSUERS); }
        for (int x = 0; x < 2; ++x) { mbar_init(&s_full[x], 1); mbar_init(&s_free[x], 4); mbar_init(&p_full[x], 4); mbar_init(&o_done[x], 1); }
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
    const uint32_t tmem = tmem_slot;                  // tile x, columns 256 x ..: S 64, P 32 + 32, O 128

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(&q_full, 2 * QC * AT_QCHUNK);
            for (int x = 0; x < 2; ++x)
                for (int c = 0; c < QC; ++c) at_load_3d(qs + (x * QC + c) * AT_QCHUNK, &qmap, c * 64, g * a.R, (row0 + x * AT_ROWS) / a.R, &q_full);
            for (int t = 0; t < tiles; ++t) {
                const int s = t % ST;
                if (!tc_wait(&empty[s], ((t / ST) & 1) ^ 1) || fail) { tc_fail(&fail, a.status); break; }
                const uint32_t st = ring + s * STAGE;
                mbar_expect_tx(&full[s], STAGE + (INT8 ? AT_SCALES : 0));
                if (INT8) {
                    bulk_g2s(scales + s * 2 * AT_KEYS, a.ks + (size_t)g * a.lds + t * AT_KEYS, AT_SCALES / 2, &full[s]);
                    bulk_g2s(scales + s * 2 * AT_KEYS + AT_KEYS, a.vs + (size_t)g * a.lds + t * AT_KEYS, AT_SCALES / 2, &full[s]);
                }
                for (int c = 0; c < QC; ++c) {
                    if (c * 64 < a.dim1) at_load_3d(st + c * AT_KCHUNK, &kmap, c * 64, g, t * AT_KEYS, &full[s]);
                    else                 at_load_3d(st + c * AT_KCHUNK, &k2map, c * 64 - a.dim1, 0, t * AT_KEYS, &full[s]);
                }
                for (int c = 0; c < VC; ++c) at_load_3d(st + (QC + c) * AT_KCHUNK, &vmap, c * 64, g, t * AT_KEYS, &full[s]);
            }
            tc_wait(&q_full, 0);                      // its own copies are not in flight when it leaves
            for (int t = max(0, tiles - ST); t < tiles && !fail; ++t) if (!tc_wait(&full[t % ST], (t / ST) & 1)) break;
        }
    } else if (warp <= ISSUERS) {
        // The whole warp runs the loop (its values are then uniform), one lane waits and issues; a wait that ran out leaves it idle for the rest.
        const bool leader = tc_elect();
        const uint32_t kind = INT8 ? 0u : (1u << 7) | (1u << 10), m128 = (uint32_t)(AT_ROWS >> 4) << 24;
        const uint32_t i_qk = (1u << 4) | kind | ((uint32_t)(AT_KEYS >> 3) << 17) | m128;
        const uint32_t i_pv = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(VC * 64 >> 3) << 17) | m128;
        const uint32_t q_lo = tc_desc_lo(qs), k_lo = tc_desc_lo(ring), v_lo = at_desc_mn(ring + QC * AT_KCHUNK);
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            if (leader && ok && !tc_wait(bar, parity)) { ok = false; tc_fail(&fail, a.status); }
            __syncwarp();
        };
        wait(&q_full, 0);
        uint32_t s = 0, sn = 0, pn = 0;               // stage of key tile t; stage and parity of the one whose scores come next
        for (int t = -1; t < tiles; ++t) {
            #pragma unroll
            for (int i = 0; i < 2 / ISSUERS; ++i) {
                const int x = ISSUERS == 2 ? warp - 1 : i;
                const uint32_t d = tmem + x * 256u, p = d + 64u, o = d + 128u;
                if (t + 1 < tiles) {                  // scores over the next keys, as soon as the present ones are read
                    if (i == 0) wait(&full[sn], pn);
                    wait(&s_free[x], (t + 1) & 1 ^ 1);
                    if (leader && ok) {
                        tc_fence_after();
                        const uint32_t qd = q_lo + x * QC * (AT_QCHUNK >> 4), kd = k_lo + sn * (STAGE >> 4);
                        #pragma unroll
                        for (int c = 0; c < QC; ++c)
                            #pragma unroll
                            for (int k = 0; k < 4; ++k)
                                tc_mma_ss(d, qd + (uint32_t)(c * (AT_QCHUNK >> 4) + 2 * k), TC_DESC_HI, kd + (uint32_t)(c * (AT_KCHUNK >> 4) + 2 * k), TC_DESC_HI, i_qk, (uint32_t)(c != 0 || k != 0));
                        tc_commit(&s_full[x]);
                    }
                    __syncwarp();
                }
                if (t < 0) continue;
                wait(&p_full[x], t & 1);
                if (leader && ok) {
                    tc_fence_after();
                    const uint32_t vd = v_lo + s * (STAGE >> 4);
                    #pragma unroll
                    for (int k = 0; k < 4; ++k) tc_mma_ts(o, p + 8 * k, vd + (uint32_t)(k * (2048 >> 4)), TC_DESC_HI, i_pv, (uint32_t)(t != 0 || k != 0));
                    if (INT8) {
                        #pragma unroll
                        for (int k = 0; k < 4; ++k) tc_mma_ts(o, p + 32 + 8 * k, vd + (uint32_t)(k * (2048 >> 4)), TC_DESC_HI, i_pv, 1u);
                    }
                    tc_commit(&o_done[x]);
                    if (i == 2 / ISSUERS - 1) tc_commit(&empty[s]);
                }
                __syncwarp();
            }
            if (++sn == ST) { sn = 0; pn ^= 1; }
            if (t >= 0 && ++s == ST) s = 0;
        }
    } else if (warp >= 4) {
        const int x = (warp - 4) >> 2, q = warp & 3, fr = row0 + x * AT_ROWS + q * 32 + lane, frc = min(fr, total - 1);
        const int tok = frc / a.R, head = g * a.R + frc - tok * a.R, pos = a.start + tok;
        const int first_pos = a.start + min(row0 + x * AT_ROWS + q * 32, total - 1) / a.R;        // least position among the warp's rows
        // Scores in units of log2 are raw scores (times their key's scale) times fsc.  Where that is positive it waits for the exponent's subtraction,
        // a multiply-add; else scores are multiplied by it first and the factor left is 1.
        const float fsc = a.scale * q_temp_factor(pos, a.qt_coef, a.qt_every) * FA_LOG2E;
        const bool late = __all_sync(0xFFFFFFFFu, fsc > 0.f && fsc < INFINITY);
        const float early = late ? 1.f : fsc, f2 = late ? fsc : 1.f;
        const uint32_t tm = tmem + x * 256u + ((uint32_t)(q * 32) << 16);
        float m = -INFINITY, l = 0.f;                 // m: in units of the scores before f2
        bool good = true;
        uint32_t stage = 0, stage_parity = 0;
        for (int t = 0; t < tiles; ++t) {
            if (INT8 && !at_wait(&full[stage], stage_parity, &fail, a.status)) { good = false; break; }       // the scales are there to see
            if (!at_wait(&s_full[x], t & 1, &fail, a.status)) { good = false; break; }
            tc_fence_after();
            uint32_t s0[32], s1[32];
            __syncwarp();
            tc_ld32(tm, s0);
            tc_ld32(tm + 32u, s1);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[x]);
            __syncwarp();
            float v[64];
            #pragma unroll
            for (int i = 0; i < 32; ++i) { v[i] = __uint_as_float(s0[i]); v[32 + i] = __uint_as_float(s1[i]); }
            const int k0 = t * AT_KEYS;
            const float* tile_scales = scales + stage * 2 * AT_KEYS;
            if (INT8) {
                #pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float4 f = *reinterpret_cast<const float4*>(tile_scales + 4 * i);
                    v[4 * i] *= f.x; v[4 * i + 1] *= f.y; v[4 * i + 2] *= f.z; v[4 * i + 3] *= f.w;
                }
            }
            if (!late) {
                #pragma unroll
                for (int i = 0; i < 64; ++i) v[i] *= early;
            }
            const bool diagonal = k0 + AT_KEYS - 1 > first_pos;
            if (diagonal) {
                #pragma unroll
                for (int i = 0; i < 64; ++i) if (k0 + i > pos) v[i] = -INFINITY;
            }
            float mx[4] = {v[0], v[1], v[2], v[3]};
            #pragma unroll
            for (int i = 4; i < 64; ++i) mx[i & 3] = fmaxf(mx[i & 3], v[i]);
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            float corr = 1.f;
            if ((top - m) * f2 > AT_LAZY) { corr = at_exp2((m - top) * f2); m = top; }          // the first tile: every row sees key 0
            const float base = m == -INFINITY ? 0.f : -m * f2;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            #pragma unroll
            for (int i = 0; i < 64; ++i) { v[i] = at_exp2(fmaf(v[i], f2, base)); sum[i & 3] += v[i]; }
            l = l * corr + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
            uint32_t hi[32], lo[32];
            if (INT8) {
                const float4* vs = reinterpret_cast<const float4*>(tile_scales + AT_KEYS);
                // `seen`: a masked weight is zero whatever the scale of its value; asked where some scale of a diagonal tile is not finite
                auto planes = [&](auto seen) {
                    #pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float4 f = vs[i];
                        const float w[4] = {seen(4 * i) ? v[4 * i] * f.x : 0.f, seen(4 * i + 1) ? v[4 * i + 1] * f.y : 0.f,
                                            seen(4 * i + 2) ? v[4 * i + 2] * f.z : 0.f, seen(4 * i + 3) ? v[4 * i + 3] * f.w : 0.f};
                        #pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const uint32_t h = fa_pack(w[2 * e], w[2 * e + 1]);
                            hi[2 * i + e] = h;
                            lo[2 * i + e] = fa_pack(w[2 * e] - __uint_as_float(h << 16), w[2 * e + 1] - __uint_as_float(h & 0xFFFF0000u));
                        }
                    }
                };
                const float* sc = reinterpret_cast<const float*>(vs);
                if (diagonal && __any_sync(0xFFFFFFFFu, !(isfinite(sc[lane]) && isfinite(sc[lane + 32])))) planes([&](int i) { return k0 + i <= pos; });
                else planes([](int) { return true; });
            } else {
                #pragma unroll
                for (int i = 0; i < 32; ++i) hi[i] = fa_pack(v[2 * i], v[2 * i + 1]);
            }
            if (t > 0) {                              // the product before has read P and left O
                if (!at_wait(&o_done[x], (t - 1) & 1, &fail, a.status)) { good = false; break; }
                tc_fence_after();
                if (__any_sync(0xFFFFFFFFu, corr != 1.f)) {
                    #pragma unroll 1
                    for (int c = 0; c < VC * 64; c += 32) {
                        uint32_t o[32];
                        __syncwarp();
                        tc_ld32(tm + 128u + (uint32_t)c, o);
                        #pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                        at_st32(tm + 128u + (uint32_t)c, o);
                    }
                }
            }
            __syncwarp();
            at_st32(tm + 64u, hi);
            if (INT8) at_st32(tm + 96u, lo);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[x]);
            if (INT8 && ++stage == ST) { stage = 0; stage_parity ^= 1; }
        }
        m *= f2;
        if (good) good = at_wait(&o_done[x], (tiles - 1) & 1, &fail, a.status);
        if (good) {
            tc_fence_after();
            const float inv = sink_norm(m / FA_LOG2E, l, a.sink ? a.sink + head : nullptr) * head_gate(a.gate, a.ldg, tok, head);
            __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)tok * a.ldo + (size_t)head * a.vdim;
            __half* oh = reinterpret_cast<__half*>(a.out) + (size_t)tok * a.ldo + (size_t)head * a.vdim;
            bool finite = true;
            #pragma unroll 1
            for (int c = 0; c < VC * 64; c += 32) {
                uint32_t o[32];
                __syncwarp();
                tc_ld32(tm + 128u + (uint32_t)c, o);
                if (!INT8) {
                    #pragma unroll
                    for (int i = 0; i < 32; ++i) finite = finite && (o[i] & 0x7F800000u) != 0x7F800000u;
                }
                if (fr < total) {
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t w[4];
                        #pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float u = __uint_as_float(o[8 * i + 2 * e]) * inv, z = __uint_as_float(o[8 * i + 2 * e + 1]) * inv;
                            if (INT8) { const __half2 h = __floats2half2_rn(u, z); w[e] = *reinterpret_cast<const uint32_t*>(&h); }
                            else      w[e] = fa_pack(u, z);
                        }
                        if (c + 8 * i < a.vdim) {
                            if (INT8) *reinterpret_cast<uint4*>(oh + c + 8 * i) = make_uint4(w[0], w[1], w[2], w[3]);
                            else      *reinterpret_cast<uint4*>(ob + c + 8 * i) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
            }
            // sums of scores that are finite over outputs that are not: some value is infinite or NaN, and it may be one that the row does not see
            if (!INT8) {
                __syncwarp();
                for (unsigned rows = __ballot_sync(0xFFFFFFFFu, fr < total && !finite && isfinite(l)); rows; rows &= rows - 1) {
                    const int r = __ffs(rows) - 1;
                    at_row(a, g, __shfl_sync(0xFFFFFFFFu, tok, r), __shfl_sync(0xFFFFFFFFu, head, r), __shfl_sync(0xFFFFFFFFu, fsc, r), __shfl_sync(0xFFFFFFFFu, m == -INFINITY ? 0.f : m, r),
                           __shfl_sync(0xFFFFFFFFu, inv, r));
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Codes of rows [0, rows) of an INT8 cache as 16-bit numbers (keys fp16, values bf16: both exact), their scales head by head, zero in
// the rest of the last 64 positions.  A thread takes 16 codes of a key and of a value.
__global__ void __launch_bounds__(256) attn_widen_kernel(const uint4* k, const uint4* v, const float* ks, const float* vs, uint4* k16, uint4* v16, float* kso, float* vso,
                                                         int rows, int padded, int n_kv, int lds) {
    pdl_wait();
    pdl_launch();
    const int per = n_kv * 8;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int r = (int)(i / per), e = (int)(i - (long long)r * per);
    if (r >= padded) return;
    if ((e & 7) == 0) {
        const int h = e >> 3;
        kso[(size_t)h * lds + r] = r < rows ? ks[(size_t)r * n_kv + h] : 0.f;
        vso[(size_t)h * lds + r] = r < rows ? vs[(size_t)r * n_kv + h] : 0.f;
    }
    if (r >= rows) return;
    const uint4 kc = __ldcg(k + i), vc = __ldcg(v + i);
    const uint32_t kw[4] = {kc.x, kc.y, kc.z, kc.w}, vw[4] = {vc.x, vc.y, vc.z, vc.w};
    uint32_t ko[8], vo[8];
    #pragma unroll
    for (int j = 0; j < 4; ++j)
        #pragma unroll
        for (int p = 0; p < 2; ++p) {
            const float a = (float)(int8_t)(kw[j] >> (16 * p)), b = (float)(int8_t)(kw[j] >> (16 * p + 8));
            const __half2 h = __floats2half2_rn(a, b);
            ko[2 * j + p] = *reinterpret_cast<const uint32_t*>(&h);
            vo[2 * j + p] = fa_pack((float)(int8_t)(vw[j] >> (16 * p)), (float)(int8_t)(vw[j] >> (16 * p + 8)));
        }
    k16[2 * i] = make_uint4(ko[0], ko[1], ko[2], ko[3]); k16[2 * i + 1] = make_uint4(ko[4], ko[5], ko[6], ko[7]);
    v16[2 * i] = make_uint4(vo[0], vo[1], vo[2], vo[3]); v16[2 * i + 1] = make_uint4(vo[4], vo[5], vo[6], vo[7]);
}

// ── host side ──
// [outer][middle][inner] elements of 16 bits, boxes of 64 x box_mid x box_out, 128-byte swizzle, zero outside
static bool at_map(CUtensorMap* map, bool half, const void* base, long long inner, long long mid, long long mid_ld, long long outer, long long outer_ld, int box_mid, int box_out) {
    const cuuint64_t gdim[3] = {(cuuint64_t)inner, (cuuint64_t)mid, (cuuint64_t)outer};
    const cuuint64_t gstr[2] = {(cuuint64_t)mid_ld * 2, (cuuint64_t)outer_ld * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_mid, (cuuint32_t)box_out}, estr[3] = {1, 1, 1};
    return encode_tiled_fn() && encode_tiled_fn()(map, half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), gdim, gstr, box, estr,
                                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static bool al16(const void* p) { return ((uintptr_t)p & 15) == 0; }

size_t attention_tc_scratch(int n_kv, int positions) {
    const size_t rows = (size_t)((positions + AT_KEYS - 1) / AT_KEYS) * AT_KEYS;
    return rows * n_kv * (2 * 128 * 2 + 2 * sizeof(float));
}

// From how many tokens on a chunk over an INT8 cache gains.  Here a CTA walks all keys of 256 rows alone, 2.3 us per 64 keys, and 64 tokens
// in groups of four are one CTA per KV head; the kernel of attention_prefill.cu deals two tokens to a CTA and is the faster one until
// tokens x KV heads fill the machine with them.  32 / 8 heads after 2000 positions, 64 / 192 /
// 256 tokens: 41 / 84 / 110 us there, 85 / 88 / 89 here; 8 / 2 heads, 512 / 1024 tokens: 76 / 130 and 95 / 112; 32 / 32 heads, 64 tokens:
// 121 and 95.  Groups it does not take go to the general kernel without this one (32 / 2 heads, 64 tokens: 2250 us, 78 here).
int attention_tc_min_tokens(int n_heads, int n_kv) {
    const int R = n_kv > 0 ? n_heads / n_kv : 0;
    if (R > 4) return AT_MIN_TOKENS;
    const int n = (2048 + n_kv - 1) / (n_kv > 0 ? n_kv : 1);
    return n > AT_MIN_TOKENS ? n : AT_MIN_TOKENS;
}
// Query rows in groups that divide a tile, head sizes in whole 16-byte rows that fill their 64-element chunks but for the last, more keys
// than one tile.  INT8: a workspace for the widened codes.
bool attention_tc_applies(const AttnCall& c) {
    const int kind = c.kind(), R = c.n_kv > 0 ? c.n_heads / c.n_kv : 0;
    if ((kind != EK_BF16 && kind != EK_INT8) || c.causal_start < 0 || c.batch < AT_MIN_TOKENS || c.window || c.records || c.k_list || R < 1 || R > 128 || (R & (R - 1)) || c.n_heads != R * c.n_kv) return false;
    if (!c.out || !c.q || !c.k || !c.v || !al16(c.out) || !al16(c.q) || !al16(c.k) || !al16(c.v) || c.n_kv > 65535) return false;
    if (kind == EK_INT8) return c.batch >= attention_tc_min_tokens(c.n_heads, c.n_kv) && c.hd == 128 && c.chd == 128 && c.ks && c.vs && c.scratch && !c.sink && !c.gate && c.qt_coef == 0.f;
    const int vd = c.vhd > 0 ? c.vhd : c.hd, d1 = c.hd - c.hd2;
    if (c.hd % 8 || vd % 8 || c.hd > 192 || vd > 128 || c.chd != c.hd || (c.k2 ? d1 % 64 || c.hd2 <= 0 || c.hd2 > 64 || !al16(c.k2) || c.ldk2 % 8 : c.hd2 != 0)) return false;
    // heads of 64 have a kernel of their own size on mma.sync, whose CTAs are shorter: this one needs the rows to fill the machine (32 / 8 heads,
    // 256 / 512 / 1024 tokens: 8.1 / 15.8 / 36.1 us there, 9.7 / 15.6 / 27.5 here; 8 / 2 heads, 1024 / 2048: 21.5 / 51.5 and 26.9 / 50.0)
    if (c.hd == 64 && vd == 64 && (long long)c.batch * c.n_heads < 16384) return false;
    // so have heads of 128; over one tile of keys it is the faster one (64 tokens: 6.1 us there, 7.0 here; 80: 8.0 and 7.0)
    if (c.hd == 128 && vd == 128 && c.causal_start + c.batch <= AT_KEYS) return false;
    return c.ldq % 8 == 0 && c.ldo % 8 == 0 && c.ldk % 8 == 0 && c.ldv % 8 == 0;
}

template <int QC, int VC, bool INT8>
static int at_go(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& k2, const CUtensorMap& v, const AtArgs& a, int n_kv, cudaStream_t st) {
    const size_t smem = (size_t)2 * QC * AT_QCHUNK + (size_t)at_stages(QC, VC, INT8) * ((QC + VC) * AT_KCHUNK + (INT8 ? AT_SCALES : 0)) + 1024;
    bool& attr = ctx()->attn_tc_attr[INT8 ? 6 : 2 * (QC - 1) + VC - 1];
    if (!attr) {
        JB_CUDA(cudaFuncSetAttribute(attn_tc_kernel<QC, VC, INT8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr = true;
    }
    const long long rows = (long long)a.n_tokens * a.R;
    JB_CUDA(launch_k(attn_tc_kernel<QC, VC, INT8>, dim3((unsigned)((rows + 2 * AT_ROWS - 1) / (2 * AT_ROWS)), n_kv), dim3(AT_THREADS), smem, st, pdl_enabled(), q, k, k2, v, a));
    count_launch();
    return JB_OK;
}

int launch_attention_tc(const AttnCall& c, cudaStream_t st) {
    DeviceCtx* cx = ctx();
    if (!cx) return JB_ERR_CUDA;
    const bool int8 = c.kind() == EK_INT8;
    const int R = c.n_heads / c.n_kv, vd = c.vhd > 0 ? c.vhd : c.hd, d1 = c.hd - (c.k2 ? c.hd2 : 0), keys = c.causal_start + c.batch;
    const long long ldq = c.ldq > 0 ? c.ldq : (long long)c.n_heads * c.hd, ldk = c.ldk > 0 ? c.ldk : (long long)c.n_kv * d1, ldv = c.ldv > 0 ? c.ldv : (long long)c.n_kv * vd;
    AtArgs a = {};
    a.out = c.out; a.R = R; a.dim1 = d1; a.vdim = vd; a.ldo = c.ldo > 0 ? c.ldo : c.n_heads * vd; a.n_tokens = c.batch; a.start = c.causal_start;
    a.scale = c.scale; a.sink = c.sink; a.qt_coef = c.qt_coef; a.qt_every = c.qt_every; a.gate = c.gate; a.ldg = c.ldg; a.status = cx->d_status;
    const void *kp = c.k, *vp = c.v;
    if (!int8) {
        a.q = (const __nv_bfloat16*)c.q; a.k = (const __nv_bfloat16*)c.k; a.k2 = (const __nv_bfloat16*)c.k2; a.v = (const __nv_bfloat16*)c.v;
        a.ldq = ldq; a.ldk = ldk; a.ldk2 = c.ldk2; a.ldv = ldv; a.dim = c.hd;
    } else {
        const int padded = (keys + AT_KEYS - 1) / AT_KEYS * AT_KEYS;
        char* s = reinterpret_cast<char*>(c.scratch);
        const size_t plane = (size_t)padded * c.n_kv * 128 * 2, sc = (size_t)padded * c.n_kv * sizeof(float);
        a.ks = reinterpret_cast<const float*>(s + 2 * plane); a.vs = reinterpret_cast<const float*>(s + 2 * plane + sc); a.lds = padded;
        kp = s; vp = s + plane;
        const long long n = (long long)padded * c.n_kv * 8;
        JB_CUDA(launch_k(attn_widen_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, pdl_enabled(), (const uint4*)c.k, (const uint4*)c.v, c.ks, c.vs, (uint4*)kp, (uint4*)vp,
                         const_cast<float*>(a.ks), const_cast<float*>(a.vs), keys, padded, c.n_kv, padded));
        count_launch();
    }
    CUtensorMap qm, km, k2m, vm;
    if (!at_map(&qm, int8, c.q, c.hd, c.n_heads, c.hd, c.batch, ldq, R, AT_ROWS / R) || !at_map(&km, int8, kp, d1, c.n_kv, d1, keys, ldk, 1, AT_KEYS) ||
        !at_map(&vm, false, vp, vd, c.n_kv, vd, keys, ldv, 1, AT_KEYS) || !(c.k2 ? at_map(&k2m, false, c.k2, c.hd2, 1, c.ldk2, keys, c.ldk2, 1, AT_KEYS) : (k2m = km, true)))
        return set_error(JB_ERR_CUDA, "prefill attention: tensor map refused (%d heads of %d / %d)", c.n_heads, c.hd, vd);
    if (int8) return at_go<2, 2, true>(qm, km, k2m, vm, a, c.n_kv, st);
    const int qc = (c.hd + 63) / 64, vc = (vd + 63) / 64;
    if (qc == 1) return vc == 1 ? at_go<1, 1, false>(qm, km, k2m, vm, a, c.n_kv, st) : at_go<1, 2, false>(qm, km, k2m, vm, a, c.n_kv, st);
    if (qc == 2) return vc == 1 ? at_go<2, 1, false>(qm, km, k2m, vm, a, c.n_kv, st) : at_go<2, 2, false>(qm, km, k2m, vm, a, c.n_kv, st);
    return vc == 1 ? at_go<3, 1, false>(qm, km, k2m, vm, a, c.n_kv, st) : at_go<3, 2, false>(qm, km, k2m, vm, a, c.n_kv, st);
}

}  // namespace jb
