// mmq_stream.cu — batched K-quant GEMM for FEW tokens (2..64): the weights are streamed once, as in the GEMV.
//
// y[N x M] = x[N x K] . W^T with the arithmetic of the tensor-core prefill kernel (mmq_tc.cu: fp16 operands built from
// the reference's quantised values — half(d*sc)*(q-8) and half(d8*q8), min term and centring constant as 16 extra K
// columns per super-block, mmq_q4k_llama.cu:159-163, :383-404; mmq_q6k_llama.cu:424-438), so the two kernels give the
// same numbers up to the order of the fp32 accumulation and the existing oracle is the checker.
//
// With N <= 64 the product is bound by HBM (every weight byte is used N times, against ~300 needed to fill the tensor pipe), and the
// 128 x 256 tiles of the prefill kernel leave most of the machine idle.  What then costs time is the chain of a launch (latency of the
// first weights, a few super-blocks per warp, the sum of the K ranges) and the conversion of codes to fp16 fragments, so here:
//   * every WARP streams on its own: 16 weight rows (one MMA tile) and a run of super-blocks, the next one requested before the
//     present one is multiplied, no barrier of the CTA in the loop (a CTA-wide ring of stages, filled by all threads and with a
//     barrier per super-block, ran at 5 % of HBM: 21.9 us for 9728 x 2560 at 8 tokens);
//   * the warps of a CTA share row tiles between K ranges, whose sums meet in shared memory in a fixed order: no second kernel;
//   * a warp dequantises its weights straight into mma.sync.m16n8k16 A fragments in registers and multiplies them against the 8-token
//     B fragments of all token tiles, one 16-byte load per (sub-block, token tile) from the operand that the quantise pre-kernel writes
//     block-major; lane c of a quad takes weights 8c..8c+7 of every 32-weight sub-block on both operands, which is a permutation of
//     K inside an MMA and leaves the sums unchanged.
#include "mmq.cuh"
#include <cstdio>
#include <cstdlib>

namespace jb {

constexpr int MS_XROW   = 288;                    // halves per (token, super-block): 256 products, 8 group sums, 8 centring sums, pad
constexpr int MS_XROWB  = MS_XROW * 2;            // bytes of a row
constexpr int MS_W6SLOT = 240;                    // Q6_K block slot: 210 B at any even offset below 16, rounded to 16
constexpr int MS_WARPS = 8;                        // per CTA, at most

struct MsArgs {
    __half* y; const __half* res;                 // output; optional residual [N][M]: y = half(float(res) + float(half(product)))
    const uint8_t* W; const __half* xb;           // weights; activation operand, block-major
    int M, N, NP, nb;                             // NP = tokens padded to a multiple of 8
    int rt, ks;                                   // row tiles of a CTA, K ranges of a row tile (a warp each)
};

__device__ __forceinline__ void ms_mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t ms_lds32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }

// four codes (one per byte, already masked) -> (q - bias) * s as two half2 words; 0x6400 | q is the half 1024 + q
__device__ __forceinline__ void ms_codes4(uint32_t q4, __half2 kbias, __half2 s, uint32_t& lo, uint32_t& hi) {
    const uint32_t a = __byte_perm(q4, 0x64646464u, 0x4140), b = __byte_perm(q4, 0x64646464u, 0x4342);
    const __half2 ha = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&a), kbias), s);
    const __half2 hb = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&b), kbias), s);
    lo = *reinterpret_cast<const uint32_t*>(&ha); hi = *reinterpret_cast<const uint32_t*>(&hb);
}
// the same with the scale given as an fp16 (hi, lo) split of an fp32 product, so each weight is rounded to fp16 once
__device__ __forceinline__ void ms_codes4_split(uint32_t q4, __half2 kbias, __half2 shi, __half2 slo, uint32_t& lo, uint32_t& hi) {
    const uint32_t a = __byte_perm(q4, 0x64646464u, 0x4140), b = __byte_perm(q4, 0x64646464u, 0x4342);
    const __half2 qa = __hsub2(*reinterpret_cast<const __half2*>(&a), kbias), qb = __hsub2(*reinterpret_cast<const __half2*>(&b), kbias);
    const __half2 ra = __hfma2(qa, shi, __hmul2(qa, slo)), rb = __hfma2(qb, shi, __hmul2(qb, slo));
    lo = *reinterpret_cast<const uint32_t*>(&ra); hi = *reinterpret_cast<const uint32_t*>(&rb);
}

// ── activation operand ────────────────────────────────────────────────────
// One warp per 32-element group of one token (the quantiser of mmq_tc_quantize_kernel, mmq_q4k_llama.cu:383-404 /
// mmq_q6k_llama.cu:424-438), written block-major: xb[(kb * NP + token) * 288 + ...]: 256 products half(d*q) in K order,
// then for Q4_K the 8 group sums half(Σx) and the 8 centring sums half(d*Σq); zero elsewhere and for padded tokens.
__global__ void mms_quantize_kernel(const __half* x, __half* xb, int N, int NP, int K, int ds4) {
    pdl_wait();
    const long long g = (long long)blockIdx.x * blockDim.y + threadIdx.y;
    const int lane = threadIdx.x, G = K / 32;
    if (g >= (long long)NP * G) return;
    const int t = (int)(g / G), gi = (int)(g - (long long)t * G), kb = gi >> 3, j = gi & 7;
    __half* row = xb + ((size_t)kb * NP + t) * MS_XROW;
    if (t >= N) {                                      // padded token: zeros
        row[32 * j + lane] = __float2half_rn(0.f);
        if (lane < 4) row[256 + 4 * j + lane] = __float2half_rn(0.f);
        return;
    }
    const float v = __half2float(x[(size_t)t * K + (size_t)gi * 32 + lane]);
    const float amax = warp_max(fabsf(v));
    float sum = v;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    float d = __fdiv_rn(amax, 127.0f);
    const float dinv = d > 0.f ? __fdiv_rn(1.0f, d) : 0.f;
    const int q = __float2int_rn(__fmul_rn(v, dinv));
    int qsum = q;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) qsum += __shfl_xor_sync(0xFFFFFFFFu, qsum, o);
    if (ds4) d = __half2float(__float2half_rn(d));
    row[32 * j + lane] = __float2half_rn(__fmul_rn(d, (float)q));
    if (lane == 0) {
        row[256 + j] = __float2half_rn(ds4 ? sum : 0.f);
        row[264 + j] = __float2half_rn(ds4 ? __fmul_rn(d, (float)qsum) : 0.f);
    }
    if (lane >= 16 && j < 4) row[272 + 4 * j + (lane - 16) % 4] = __float2half_rn(0.f);      // pad halves 272..287
}

// ── the product ───────────────────────────────────────────────────────────
// A warp owns 16 weight rows and a run of super-blocks.  Q4_K blocks are 16-byte aligned and go straight to registers, a super-block
// ahead of the one that is multiplied; Q6_K blocks (2-byte aligned) come as the enclosing 16-byte pieces by cp.async into two private
// slots of the warp.  The activation operand is read from L2 through L1 as whole fragments.
template <int NT>
__device__ __forceinline__ void ms_tokens(uint4 (&b)[NT], const uint8_t* xq) {
    #pragma unroll
    for (int t = 0; t < NT; ++t) b[t] = *reinterpret_cast<const uint4*>(xq + (size_t)t * 8 * MS_XROWB);       // not the read-only path: the kernel in front wrote it
}
template <int NT>
__device__ __forceinline__ void ms_step(float (&acc)[NT][4], const uint32_t (&k0)[4], const uint32_t (&k1)[4], const uint4 (&b)[NT]) {
    #pragma unroll
    for (int t = 0; t < NT; ++t) ms_mma_f16(acc[t], k0, b[t].x, b[t].y);      // NT independent accumulators between two
    #pragma unroll
    for (int t = 0; t < NT; ++t) ms_mma_f16(acc[t], k1, b[t].z, b[t].w);      // MMAs into the same one
}
struct MsQ4 { uint4 hA, hB; uint2 qA[4], qB[4]; };
__device__ __forceinline__ void ms_load4(MsQ4& w, const uint8_t* pA, const uint8_t* pB, int c) {
    w.hA = __ldg(reinterpret_cast<const uint4*>(pA)); w.hB = __ldg(reinterpret_cast<const uint4*>(pB));
    #pragma unroll
    for (int il = 0; il < 4; ++il) {
        w.qA[il] = __ldg(reinterpret_cast<const uint2*>(pA + 16 + 32 * il + 8 * c));
        w.qB[il] = __ldg(reinterpret_cast<const uint2*>(pB + 16 + 32 * il + 8 * c));
    }
}
// xb: this lane's 8 halves of sub-block 0, token g of token tile 0
template <int NT>
__device__ __forceinline__ void ms_block4(float (&acc)[NT][4], const MsQ4& w, const uint8_t* xb, int c) {
    const __half dhA = __ushort_as_half((unsigned short)(w.hA.x & 0xFFFFu)), dhB = __ushort_as_half((unsigned short)(w.hB.x & 0xFFFFu));
    const __half2 k1032 = __half2half2(__ushort_as_half((unsigned short)0x6408));      // 1024 + 8
    #pragma unroll
    for (int il = 0; il < 4; ++il)
        #pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
            const int j = 2 * il + sub;
            uint4 b[NT];
            ms_tokens<NT>(b, xb + j * 64);
            int scA, mnA, scB, mnB;
            scale_min_k4(j, w.hA.y, w.hA.z, w.hA.w, scA, mnA);
            scale_min_k4(j, w.hB.y, w.hB.z, w.hB.w, scB, mnB);
            const __half2 sA = __half2half2(__hmul(dhA, __int2half_rn(scA))), sB = __half2half2(__hmul(dhB, __int2half_rn(scB)));
            uint32_t k0[4], k1[4];                   // A fragments of the sub-block's two k-steps
            ms_codes4((w.qA[il].x >> (4 * sub)) & 0x0F0F0F0Fu, k1032, sA, k0[0], k0[2]);
            ms_codes4((w.qA[il].y >> (4 * sub)) & 0x0F0F0F0Fu, k1032, sA, k1[0], k1[2]);
            ms_codes4((w.qB[il].x >> (4 * sub)) & 0x0F0F0F0Fu, k1032, sB, k0[1], k0[3]);
            ms_codes4((w.qB[il].y >> (4 * sub)) & 0x0F0F0F0Fu, k1032, sB, k1[1], k1[3]);
            ms_step<NT>(acc, k0, k1, b);
        }
    // the extra k-step: columns 0..7 = half(-dmin) * half(m_j) against the group sums, 8..15 = 8 * half(d*sc_j) against the centring
    // sums; this lane holds columns 2c, 2c+1 (a0/a1) and 8+2c, 9+2c (a2/a3)
    const __half mhA = __hneg(__ushort_as_half((unsigned short)(w.hA.x >> 16))), mhB = __hneg(__ushort_as_half((unsigned short)(w.hB.x >> 16)));
    const __half eight = __ushort_as_half((unsigned short)0x4800);
    uint32_t e[4];
    int s0, m0, s1, m1;
    scale_min_k4(2 * c, w.hA.y, w.hA.z, w.hA.w, s0, m0); scale_min_k4(2 * c + 1, w.hA.y, w.hA.z, w.hA.w, s1, m1);
    { const __half2 mn = __halves2half2(__hmul(mhA, __int2half_rn(m0)), __hmul(mhA, __int2half_rn(m1)));
      const __half2 ce = __halves2half2(__hmul(eight, __hmul(dhA, __int2half_rn(s0))), __hmul(eight, __hmul(dhA, __int2half_rn(s1))));
      e[0] = *reinterpret_cast<const uint32_t*>(&mn); e[2] = *reinterpret_cast<const uint32_t*>(&ce); }
    scale_min_k4(2 * c, w.hB.y, w.hB.z, w.hB.w, s0, m0); scale_min_k4(2 * c + 1, w.hB.y, w.hB.z, w.hB.w, s1, m1);
    { const __half2 mn = __halves2half2(__hmul(mhB, __int2half_rn(m0)), __hmul(mhB, __int2half_rn(m1)));
      const __half2 ce = __halves2half2(__hmul(eight, __hmul(dhB, __int2half_rn(s0))), __hmul(eight, __hmul(dhB, __int2half_rn(s1))));
      e[1] = *reinterpret_cast<const uint32_t*>(&mn); e[3] = *reinterpret_cast<const uint32_t*>(&ce); }
    const uint8_t* xe = xb + 512 - 12 * c;           // 16 c on, 4 c wanted
    #pragma unroll
    for (int t = 0; t < NT; ++t) {
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(xe + (size_t)t * 8 * MS_XROWB), b1 = *reinterpret_cast<const uint32_t*>(xe + (size_t)t * 8 * MS_XROWB + 16);
        ms_mma_f16(acc[t], e, b0, b1);
    }
}
// pA, pB: shared addresses of this lane's two blocks, at any even offset of their slots
template <int NT>
__device__ __forceinline__ void ms_block6(float (&acc)[NT][4], uint32_t pA, uint32_t pB, const uint8_t* xb, int c) {
    const __half2 k1056 = __half2half2(__ushort_as_half((unsigned short)0x6420));      // 1024 + 32
    #pragma unroll
    for (int n = 0; n < 2; ++n) {
        uint32_t frag[4][2][4];                      // [quarter][k-step][a0..a3]
        #pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            const uint32_t p = rs ? pB : pA;
            const uint32_t al = p & ~3u, sh = (p & 2u) * 8u;
            auto field8 = [&](uint32_t off, uint32_t& w0, uint32_t& w1) {     // 8 bytes at block offset `off`
                const uint32_t x0 = ms_lds32(al + off), x1 = ms_lds32(al + off + 4), x2 = ms_lds32(al + off + 8);
                w0 = __funnelshift_r(x0, x1, sh); w1 = __funnelshift_r(x1, x2, sh);
            };
            uint32_t la[2], lb[2], h[2], sc[2];
            field8(64 * n + 8 * c, la[0], la[1]);            // ql[64n + l]:      quarters 0 (low nibble) and 2 (high)
            field8(64 * n + 32 + 8 * c, lb[0], lb[1]);       // ql[64n + 32 + l]: quarters 1 and 3
            field8(128 + 32 * n + 8 * c, h[0], h[1]);        // qh[32n + l]: bit pairs of the four quarters
            field8(192 + 8 * n, sc[0], sc[1]);               // scales 8n + 2*quarter + (l >= 16): one int8 per quarter for this lane
            const float d = h2f_bits(ms_lds32((p + 208) & ~3u) >> (((p + 208) & 2u) * 8u));
            #pragma unroll
            for (int qt = 0; qt < 4; ++qt) {
                const float ds = __fmul_rn(d, (float)(int)(int8_t)((sc[qt >> 1] >> (8 * (2 * (qt & 1) + (c >> 1)))) & 0xFFu));
                const __half hs = __float2half_rn(ds);
                const __half2 shi = __half2half2(hs), slo = __half2half2(__float2half_rn(ds - __half2float(hs)));
                #pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const uint32_t q = ((((qt & 1) ? lb[x] : la[x]) >> (4 * (qt >> 1))) & 0x0F0F0F0Fu) | (((h[x] >> (2 * qt)) & 0x03030303u) << 4);
                    ms_codes4_split(q, k1056, shi, slo, frag[qt][x][rs], frag[qt][x][2 + rs]);
                }
            }
        }
        #pragma unroll
        for (int qt = 0; qt < 4; ++qt) {
            uint4 b[NT];
            ms_tokens<NT>(b, xb + (4 * n + qt) * 64);
            ms_step<NT>(acc, frag[qt][0], frag[qt][1], b);
        }
    }
}

// NT: 8-token tiles of a CTA.  Two CTAs share an SM up to 128 registers.  At four and six tiles that has to be asked for: Q4_K 9728 x 2560 over
// 48 tokens 36.4 -> 28.9 us, Q6_K 2560 x 9728 over 32 tokens 32.5 -> 24.6; elsewhere the compiler's own choice is the faster one.
template <int TYPE, int NT>
__global__ void __launch_bounds__(MS_WARPS * 32, NT == 4 || NT == 6 ? 2 : 0) mms_kernel(const MsArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int BB = TYPE == T_Q4K ? Q4K_BYTES : Q6K_BYTES;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int rt = warp / a.ks, ks = warp - rt * a.ks;                       // row tile of the CTA, K range
    const int row0 = (blockIdx.x * a.rt + rt) * 16;
    const int tok0 = NT <= 4 ? blockIdx.y * NT * 8 : 0;                      // more than four token tiles a CTA: they are not dealt
    const bool live = row0 < a.M;
    const int kb0 = (int)((long long)ks * a.nb / a.ks), kb1 = (int)((long long)(ks + 1) * a.nb / a.ks);
    const size_t rb = (size_t)a.nb * BB;
    float acc[NT][4];
    #pragma unroll
    for (int t = 0; t < NT; ++t) { acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f; }
    const uint8_t* xb = reinterpret_cast<const uint8_t*>(a.xb) + (size_t)(tok0 + g) * MS_XROWB + c * 16;
    const size_t x_block = (size_t)a.NP * MS_XROWB;
    // a row past M multiplies the last row's weights and is never stored
    const uint8_t *wA = a.W + (size_t)min(row0 + g, a.M - 1) * rb, *wB = a.W + (size_t)min(row0 + g + 8, a.M - 1) * rb;
    if (TYPE == T_Q4K) {
        MsQ4 cur, nxt;
        if (live) ms_load4(cur, wA + (size_t)kb0 * BB, wB + (size_t)kb0 * BB, c);        // weights do not depend on the kernel in front
        pdl_wait();
        pdl_launch();
        if (live)
            for (int kb = kb0; kb < kb1; ++kb) {
                if (kb + 1 < kb1) ms_load4(nxt, wA + (size_t)(kb + 1) * BB, wB + (size_t)(kb + 1) * BB, c);
                ms_block4<NT>(acc, cur, xb + (size_t)kb * x_block, c);
                cur = nxt;
            }
    } else {
        uint8_t* ring = smem + (size_t)warp * 2 * 16 * MS_W6SLOT;
        const uintptr_t wend = (uintptr_t)a.W + (size_t)a.M * rb;            // no copy reads past the tensor
        auto fetch = [&](int kb) {                   // the 16 blocks of super-block kb: 15 pieces of 16 bytes each
            uint8_t* slot = ring + (size_t)((kb - kb0) & 1) * 16 * MS_W6SLOT;
            #pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int idx = lane + 32 * i, r = idx / 15, pc = idx - r * 15;
                const uintptr_t src = (uintptr_t)a.W + (size_t)min(row0 + r, a.M - 1) * rb + (size_t)kb * BB;
                const uintptr_t p16 = (src & ~(uintptr_t)15) + 16u * (uintptr_t)pc;
                if (idx >= 240 || p16 >= src + BB) continue;
                uint8_t* dst = slot + r * MS_W6SLOT + 16 * pc;
                if (p16 + 16 <= wend) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"((const void*)p16) : "memory");
                else for (uintptr_t q = p16; q < wend; ++q) dst[q - p16] = *reinterpret_cast<const uint8_t*>(q);      // the tensor's last bytes
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (live) fetch(kb0);
        pdl_wait();
        pdl_launch();
        if (live)
            for (int kb = kb0; kb < kb1; ++kb) {
                if (kb + 1 < kb1) { fetch(kb + 1); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncwarp();
                const uint32_t slot = smem_u32(ring) + (uint32_t)((kb - kb0) & 1) * 16u * MS_W6SLOT;
                ms_block6<NT>(acc, slot + g * MS_W6SLOT + (uint32_t)((uintptr_t)(wA + (size_t)kb * BB) & 15), slot + (g + 8) * MS_W6SLOT + (uint32_t)((uintptr_t)(wB + (size_t)kb * BB) & 15),
                              xb + (size_t)kb * x_block, c);
                __syncwarp();                        // the slot is read before it is filled again
            }
        __syncthreads();                             // the sums below reuse the slots
    }
    // partial sums of the K ranges: ranges 1.. leave theirs in shared memory, range 0 adds them in order and stores
    float* red = reinterpret_cast<float*>(smem);             // [row tile][range - 1][NT * 4][32 lanes]
    if (ks > 0 && live) {
        float* dst = red + ((size_t)(rt * (a.ks - 1) + ks - 1) * NT * 4) * 32 + lane;
        #pragma unroll
        for (int t = 0; t < NT; ++t)
            #pragma unroll
            for (int e = 0; e < 4; ++e) dst[(t * 4 + e) * 32] = acc[t][e];
    }
    __syncthreads();
    if (ks > 0 || !live) return;
    for (int k = 0; k + 1 < a.ks; ++k) {
        const float* src = red + ((size_t)(rt * (a.ks - 1) + k) * NT * 4) * 32 + lane;
        #pragma unroll
        for (int t = 0; t < NT; ++t)
            #pragma unroll
            for (int e = 0; e < 4; ++e) acc[t][e] += src[(t * 4 + e) * 32];
    }
    // D fragment: rows g / g+8 of the tile, tokens 8t + 2c and 8t + 2c + 1
    #pragma unroll
    for (int t = 0; t < NT; ++t) {
        #pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = row0 + g + 8 * (e >> 1), tok = tok0 + 8 * t + 2 * c + (e & 1);
            if (row < a.M && tok < a.N) {
                const size_t o = (size_t)tok * a.M + row;
                const __half pr = __float2half_rn(acc[t][e]);
                a.y[o] = a.res ? __float2half_rn(__fadd_rn(__half2float(a.res[o]), __half2float(pr))) : pr;
            }
        }
    }
}

// ── host side ─────────────────────────────────────────────────────────────
bool mmq_stream_applies(const void* W, int type, int M, int N, int K) {
    static const bool off = [] { const char* e = getenv("JLLM_B200_MMQ_STREAM"); return e && e[0] == '0'; }();
    if (off || N < 2 || N > 64 || M < 16 || K % QK_K) return false;
    // the largest matrices at more than 40 tokens: the tensor-core kernel is as fast or faster (here / there, us: Q4_K 9728 x 2560, 40 tokens
    // 24.9 / 28.5, 48: 28.9 / 28.6, 64: 36.8 / 28.8; Q6_K 2560 x 9728 28.9 / 27.9, 34.9 / 27.9, 44.6 / 28.2; Q6_K 151936 x 2560 274 / 279, 283 / 279,
    // 304 / 280); the smaller ones stay faster here (Q4_K 2560 x 4096, 64 tokens: 17.0 / 20.5)
    if (N > 40 && (long long)M * K >= (1ll << 24) && mmq_tc_applies(W, type, M, N, K)) return false;
    if (type == T_Q4K) return ((uintptr_t)W & 15) == 0;
    return type == T_Q6K && ((uintptr_t)W & 1) == 0;
}

// K ranges of a row tile: enough warps to keep about sixteen on every SM, at least two super-blocks each; row tiles fill the CTA up.
static void ms_shape(int M, int nb, int sm_count, int& rt, int& ks) {
    const int tiles = (M + 15) / 16;
    ks = (16 * sm_count + tiles - 1) / tiles;
    if (ks > (nb + 1) / 2) ks = (nb + 1) / 2;
    if (ks > MS_WARPS) ks = MS_WARPS;
    if (ks < 1) ks = 1;
    rt = MS_WARPS / ks;
}

static int ms_tiles(int N) { return N <= 48 ? (N + 7) / 8 : 8; }       // 8-token MMA tiles the kernel is built for
// Few rows leave SMs idle (1024 rows: 64 CTAs): the token tiles are then dealt evenly to as many CTAs as it takes, each with the weights to
// itself.  1024 x 2560 over 16 / 32 / 48 / 64 tokens: Q4_K 9.3 / 9.3 / 12.0 / 15.1 us with one, 6.8 / 7.9 / 8.7 / 8.6 dealt; Q6_K 8.1 / 11.2 /
// 13.4 / 12.8 and 7.5 / 9.1 / 9.3 / 9.7.
static int ms_split(int N, int ctas, int sm_count) {
    const int t = ms_tiles(N);
    int ty = 1;
    for (int d = 2; d <= t && ctas * ty < sm_count; ++d)
        if (t % d == 0) ty = d;
    return ty;
}

size_t mmq_stream_scratch_bytes(int type, int M, int N, int K) {
    (void)type; (void)M;
    return (((size_t)(K / QK_K) * 8 * ms_tiles(N) * MS_XROWB + 255) & ~(size_t)255) + 256;
}

// `residual` (optional, [N][M]): the residual exit of a layer fused in (add_half arithmetic: the product is rounded to fp16
// first).  `reuse_operand`: the caller multiplies the SAME activations by another matrix of the same weight type right after
// the previous call on this stream (Q and K, gate and up): the quantised operand in `scratch` is still valid and the quantise
// launch is skipped; the library checks pointer, shape, flavour and scratch address and quantises again if anything differs.
int launch_mmq_stream(__half* y, const void* W, int type, const __half* x, void* scratch, int M, int N, int K, const __half* residual,
                      bool reuse_operand, cudaStream_t st, MmqWork& work) {
    DeviceCtx* cx = ctx();
    if (!cx) return JB_ERR_CUDA;
    const int nb = K / QK_K, NPk = ms_tiles(N) * 8;      // tokens of the operand (padded ones are zero columns)
    __half* xb = reinterpret_cast<__half*>(scratch);
    const long long groups = (long long)NPk * (K / 32);
    const int ds4 = type == T_Q4K;
    const MmqOperand op = {x, scratch, (void*)st, N, K, ds4};
    if (!reuse_operand || !work.few.is(op)) {
        JB_CUDA(launch_k(mms_quantize_kernel, dim3((unsigned)((groups + 3) / 4)), dim3(32, 4), 0, st, pdl_enabled(), x, xb, N, NPk, K, ds4));
        count_launch();
        work.few = op;
        work.many = MmqOperand();                        // the scratch is shared: the other layout's operand is gone
    }
    MsArgs a = {};
    a.y = y; a.res = residual; a.W = (const uint8_t*)W; a.xb = xb; a.M = M; a.N = N; a.NP = NPk; a.nb = nb;
    ms_shape(M, nb, cx->sm_count, a.rt, a.ks);
    const int tiles = (M + 15) / 16, ctas = (tiles + a.rt - 1) / a.rt, ty = ms_split(N, ctas, cx->sm_count);
    const int NT = ms_tiles(N) / ty;
    typedef void (*Kern)(MsArgs);
    static const Kern k4[8] = { mms_kernel<T_Q4K, 1>, mms_kernel<T_Q4K, 2>, mms_kernel<T_Q4K, 3>, mms_kernel<T_Q4K, 4>, mms_kernel<T_Q4K, 5>, mms_kernel<T_Q4K, 6>, nullptr, mms_kernel<T_Q4K, 8> };
    static const Kern k6[8] = { mms_kernel<T_Q6K, 1>, mms_kernel<T_Q6K, 2>, mms_kernel<T_Q6K, 3>, mms_kernel<T_Q6K, 4>, mms_kernel<T_Q6K, 5>, mms_kernel<T_Q6K, 6>, nullptr, mms_kernel<T_Q6K, 8> };
    const Kern kern = ds4 ? k4[NT - 1] : k6[NT - 1];
    const int ki = (ds4 ? 0 : 8) + NT - 1, warps = a.rt * a.ks;
    const size_t red = (size_t)a.rt * (a.ks - 1) * NT * 4 * 32 * sizeof(float), slots = ds4 ? 0 : (size_t)warps * 2 * 16 * MS_W6SLOT, smem = red > slots ? red : slots;
    if (!cx->mms_attr[ki]) {
        JB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_WARPS * 2 * 16 * MS_W6SLOT));
        cx->mms_attr[ki] = true;
    }
    static const bool verbose = getenv("JLLM_B200_MMQ_DEBUG") != nullptr;
    if (verbose) fprintf(stderr, "[mmq_stream] type %d M=%d N=%d K=%d: %d x %d CTAs of %d row tiles x %d K ranges, smem %zu\n", type, M, N, K, ctas, ty, a.rt, a.ks, smem);
    JB_CUDA(launch_k(kern, dim3(ctas, ty), dim3(warps * 32), smem, st, pdl_enabled(), a));
    count_launch();
    return JB_OK;
}

}  // namespace jb
