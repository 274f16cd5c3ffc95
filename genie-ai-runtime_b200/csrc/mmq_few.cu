// mmq_few.cu — K-quant products of a few tokens (2..128) on tcgen05, and the kernels between them.
//
// y[N x M] = x[N x K] . W^T with the arithmetic of mmq_tc.cu: fp16 operands built from the reference's quantised values
// (half(d*sc)*(q-8) and half(d8*q8), min term and centring constant as 16 extra K columns per super-block, mmq_q4k_llama.cu:159-163,
// :383-404; mmq_q6k_llama.cu:424-438), summed in fp32.
//
// With so few tokens a product is bound by its weights' way from memory and by turning codes into fp16, not by the tensor cores:
//   * one CTA per SM, each with an equal run of (128-row tile, super-block) units whatever the matrix' shape: 9728 x 2560 twice is
//     1520 units, 10.3 per CTA.  A tile that several CTAs share has several partial sums; the kernel that uses the product adds them
//     in order of K, so there is no second launch for them;
//   * weights come by TMA, a super-block of 128 rows at a time, four ahead, requested before the kernel in front is done (they do not
//     depend on it).  Q6_K rows are no multiple of 16 bytes; 2, 4 or 8 of them are, so a tensor map takes that many rows as one and a
//     copy brings every 2nd, 4th or 8th row from the 16-byte boundary in front of its block;
//   * 16 warps turn codes into fp16, a row and 64 weights per thread, and store them to TENSOR memory, where the A operand of an MMA
//     may lie: half the shared-memory traffic of an operand tile there, and no bank conflicts.  The order of K within a super-block is
//     the one that costs least to unpack (two codes of a word 16 bits apart); the activations are laid out in it (mf_pos4, mf_pos6);
//   * activations are written once by the kernel in front as the image that an MMA without swizzle reads: [chunk of 8][token][8],
//     a bulk copy per half super-block;
//   * four more warps take the finished sums out while the next tile is multiplied.
// The kernels between two products (norms, rotation, SwiGLU) add the sums up, work and quantise in one launch: nine launches a layer in place of
// seventeen.
//
// Measured with cold weights, us at 8 / 64 / 128 tokens, in brackets what served before (warps streaming rows into mma.sync up to 40 tokens, the
// 128 x 256 tiles of mmq_tc.cu): gate and up, Q4_K 9728 x 2560 twice, 12.8 / 16.9 / 22.4 (27.2 / 35.4 / -); W_down, Q6_K 2560 x 9728,
// 11.2 / 13.4 / 18.3 (16.8 / 27.1 / -); Wo, Q4_K 2560 x 4096, 6.7 / 8.9 / 12.4 (7.5 / 20.3 / -); logits, Q6_K 151936 x 2560, 91 / 99 / 123
// (125 / 280 / -), of which 62 / 75 / 103 are left without the arithmetic on the codes (at 64 tokens ALU 61 % and issue slots 71 % busy), and memory needs 49.
// A prompt chunk of 8 layers: 33 tokens 696 us (1283); above 128 tokens an accumulator and two
// super-blocks of weights no longer fit into tensor memory.
#include "mmq_few.cuh"
#include "mmq.cuh"
#include "tc.cuh"
#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace jb {

constexpr int MF_ROWS = 128, MF_WSTAGES = 4, MF_ASTAGES = 3, MF_XSTAGES = 8;     // super-blocks in flight, at most
constexpr int MF_PITCH4 = 144, MF_PITCH6 = 240;           // bytes of a row's super-block in shared memory
constexpr int MF_WBYTES4 = MF_ROWS * MF_PITCH4, MF_WBYTES6 = MF_ROWS * MF_PITCH6;
constexpr int MF_ACOLS = 136;                             // tensor-memory columns of a super-block: 256 weights and the 16 extra ones
constexpr int MF_PRODUCERS = 16, MF_DRAINS = 4;           // warps
constexpr int MF_THREADS = 32 * (3 + MF_PRODUCERS + MF_DRAINS);
constexpr int MF_OUT_TOK = 16;                            // tokens of an output tile on its way through shared memory
constexpr int MF_OUT_BYTES = MF_OUT_TOK * MF_ROWS * 2;
constexpr int MF_SMEM = 227 * 1024 - 1024;                // dynamic: alignment, weights, activations, output tile

struct MfArgs {
    MfSeg seg[MF_MAX_SEG];
    int nseg, nb, N, NP, rows;
    const __half* x4; const __half* x6;
    float* part;                          // sums [slot][token][rows], or of the tiles that CTAs share [CTA][2][token][128]
    __half* y;                            // outputs of the product itself
    int* status;
};

__host__ __device__ __forceinline__ int mf_first(const MfSeg& s, int cta) { return (int)((uint32_t)cta * (uint32_t)s.units / (uint32_t)s.ctas); }
__host__ __device__ __forceinline__ int mf_owner(const MfSeg& s, int unit) { return (int)(((uint32_t)(unit + 1) * (uint32_t)s.ctas - 1u) / (uint32_t)s.units); }

// where K lies: element e of 32-weight group j of a super-block (codes two by two, 16 bits apart in their word), for Q4_K and Q6_K
__device__ __forceinline__ int mf_swap(int e) { return (e & ~3) | ((e & 1) << 1) | ((e >> 1) & 1); }
__device__ __forceinline__ int mf_pos4(int j, int e) { return 32 * j + mf_swap(e); }
__device__ __forceinline__ int mf_pos6(int j, int e) { return 128 * (j >> 2) + 64 * (e >> 4) + 16 * (j & 3) + mf_swap(e & 15); }

__device__ __forceinline__ uint32_t mf_pack(__half lo, __half hi) { return (uint32_t)__half_as_ushort(lo) | ((uint32_t)__half_as_ushort(hi) << 16); }
__device__ __forceinline__ uint4 mf_lds128(uint32_t a) { uint4 v; asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v; }
__device__ __forceinline__ uint2 mf_lds64(uint32_t a) { uint2 v; asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t mf_lds16(uint32_t a) { unsigned short v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a)); return v; }
__device__ __forceinline__ void mf_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
                   "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
                   "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void mf_st4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0,%1,%2,%3};" ::"r"(a), "r"(b), "r"(c), "r"(d), "r"(taddr) : "memory");
}
__device__ __forceinline__ void mf_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mf_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// whether all four drain warps say so: they meet at barriers, so they leave together or not at all
__device__ __forceinline__ bool mf_drains_all(bool ok) {
    int x;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n" : "=r"(x) : "r"((int)ok) : "memory");
    return x != 0;
}

__device__ __forceinline__ __half2 mf_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
__device__ __forceinline__ uint32_t mf_u32(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
// bytes 0 and 2 of a word as two halves
__device__ __forceinline__ __half2 mf_bytes(uint32_t w) { return __hsub2(mf_h2((w & 0x00FF00FFu) | 0x64006400u), mf_h2(0x64006400u)); }

// Two codes of a word (bits 0-3 and 16-19; `high`: bits 4-7 and 20-23) -> (q - 8) * s, both roundings as in mmq_tc.cu: 0x6400 | q is the
// half 1024 + q, 0x6400 | 16 q is 1024 + 16 q, and (1024 + 16 q) / 16 - 72 = q - 8 is exact (numbers put into a half's mantissa: the conversion of
// Kim et al., "Who Says Elephants Can't Run", 2022).
__device__ __forceinline__ uint32_t mf_low(uint32_t w, __half2 s) { return mf_u32(__hmul2(__hsub2(mf_h2((w & 0x000F000Fu) | 0x64006400u), mf_h2(0x64086408u)), s)); }
__device__ __forceinline__ uint32_t mf_high(uint32_t w, __half2 s) { return mf_u32(__hmul2(__hfma2(mf_h2((w & 0x00F000F0u) | 0x64006400u), mf_h2(0x2C002C00u), mf_h2(0xD480D480u)), s)); }

// The scales of half f of a Q4_K super-block, four groups at a time (scale_min_k4 for j = 4 f .. 4 f + 3): half(d * sc) and half(-dmin * m) of
// groups 0 and 2, 1 and 3 of them.
struct MfS4 { __half2 d02, d13, m02, m13; };
__device__ __forceinline__ MfS4 mf_scales4(const uint4& hd, int f) {
    const uint32_t sc = f ? (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u) : hd.y & 0x3F3F3F3Fu;
    const uint32_t mn = f ? ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u) : hd.z & 0x3F3F3F3Fu;
    const __half2 dm = mf_h2(hd.x), d = __low2half2(dm), m = __hneg2(__high2half2(dm));
    MfS4 r;
    r.d02 = __hmul2(d, mf_bytes(sc)); r.d13 = __hmul2(d, mf_bytes(sc >> 8));
    r.m02 = __hmul2(m, mf_bytes(mn)); r.m13 = __hmul2(m, mf_bytes(mn >> 8));
    return r;
}
// 64 weights of a Q4_K super-block, 32 bytes of packed codes -> 32 columns of two halves each
__device__ __forceinline__ void mf_codes4(uint32_t (&o)[32], const uint4& q0, const uint4& q1, __half2 a, __half2 b) {
    const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    #pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t v = w[i] >> 8;
        o[2 * i] = mf_low(w[i], a); o[2 * i + 1] = mf_low(v, a);
        o[16 + 2 * i] = mf_high(w[i], b); o[16 + 2 * i + 1] = mf_high(v, b);
    }
}
// Two 6-bit codes: nibbles of `low`, upper bits of `high` -> (q - 32) * scale, the scale an fp16 (hi, lo) split of an fp32 product.  Low nibbles
// make 1024 + q (upper bits at 4, 5), high ones 1024 + 16 q (at 8, 9), so that no nibble is shifted and one shifted word of upper bits serves both.
__device__ __forceinline__ uint32_t mf_six_low(uint32_t low, uint32_t high, __half2 shi, __half2 slo) {
    const __half2 q = __hsub2(mf_h2((low & 0x000F000Fu) | ((high & 0x00300030u) | 0x64006400u)), mf_h2(0x64206420u));      // 1024 + 32
    return mf_u32(__hfma2(q, shi, __hmul2(q, slo)));
}
__device__ __forceinline__ uint32_t mf_six_high(uint32_t low, uint32_t high, __half2 shi, __half2 slo) {
    const __half2 q = __hfma2(mf_h2((low & 0x00F000F0u) | ((high & 0x03000300u) | 0x64006400u)), mf_h2(0x2C002C00u), mf_h2(0xD600D600u));      // / 16 - 64 - 32
    return mf_u32(__hfma2(q, shi, __hmul2(q, slo)));
}
struct MfQ6 { uint32_t la[4], lb[4], h[4], sc[2], d; };
// Sixteen bytes from byte 4 W + sh / 8 of 32 aligned ones.  The offset of a block from a 16-byte boundary is the same for all rows of a warp
// (unless a row is an odd number of blocks long), so which words these are is a branch and not a selection.
template <int W>
__device__ __forceinline__ void mf_field16(uint32_t (&w)[4], uint32_t al, uint32_t sh) {
    const uint4 x = mf_lds128(al), y = mf_lds128(al + 16);
    const uint32_t v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(v[W + i], v[W + i + 1], sh);
}
template <int W>
__device__ __forceinline__ void mf_fields6(MfQ6& r, uint32_t al, uint32_t sh, int n, int lh) {
    mf_field16<W>(r.la, al + 64 * n + 16 * lh, sh);
    mf_field16<W>(r.lb, al + 64 * n + 32 + 16 * lh, sh);
    mf_field16<W>(r.h, al + 128 + 32 * n + 16 * lh, sh);
}
__device__ __forceinline__ void mf_load6(MfQ6& r, uint32_t at, int n, int lh) {
    const uint32_t al16 = at & ~15u, sh16 = (at & 2u) * 8u;
    switch ((at >> 2) & 3u) {
        case 0: mf_fields6<0>(r, al16, sh16, n, lh); break;
        case 1: mf_fields6<1>(r, al16, sh16, n, lh); break;
        case 2: mf_fields6<2>(r, al16, sh16, n, lh); break;
        default: mf_fields6<3>(r, al16, sh16, n, lh); break;
    }
}
__device__ __forceinline__ void mf_scales6(MfQ6& r, uint32_t at, int n) {
    const uint32_t s = at + 192 + 8 * n, al = s & ~7u, sh = (s & 2u) * 8u;
    const bool odd = (s & 4u) != 0;
    const uint2 x = mf_lds64(al), y = mf_lds64(al + 8);
    const uint32_t v0 = odd ? x.y : x.x, v1 = odd ? y.x : x.y, v2 = odd ? y.y : y.x;
    r.sc[0] = __funnelshift_r(v0, v1, sh); r.sc[1] = __funnelshift_r(v1, v2, sh);
    r.d = mf_lds16(at + 208);
}
// 64 weights of a Q6_K super-block, of half n the run lh of 16 in each quarter.  hi = half(d * sc) and lo = half(d * sc - hi), exact products of
// two halves rounded once: what the fp32 product's split is in mmq_tc.cu.
__device__ __forceinline__ void mf_codes6(uint32_t (&o)[32], const MfQ6& r, int lh) {
    const __half2 d = __half2half2(__ushort_as_half((unsigned short)r.d)), bias = mf_h2(0x64806480u);      // signed bytes: 1024 + 128 + sc
    const __half2 s01 = __hsub2(mf_h2(((r.sc[0] >> (8 * lh)) & 0x00FF00FFu) ^ 0x64806480u), bias), s23 = __hsub2(mf_h2(((r.sc[1] >> (8 * lh)) & 0x00FF00FFu) ^ 0x64806480u), bias);
    const __half2 h01 = __hmul2(d, s01), h23 = __hmul2(d, s23), l01 = __hfma2(d, s01, __hneg2(h01)), l23 = __hfma2(d, s23, __hneg2(h23));
    const __half2 shi[4] = {__low2half2(h01), __high2half2(h01), __low2half2(h23), __high2half2(h23)};
    const __half2 slo[4] = {__low2half2(l01), __high2half2(l01), __low2half2(l23), __high2half2(l23)};
    #pragma unroll
    for (int i = 0; i < 4; ++i)
        #pragma unroll
        for (int x = 0; x < 2; ++x) {                     // bytes 0 and 2 of the words, then 1 and 3
            const uint32_t a = x ? r.la[i] >> 8 : r.la[i], b = x ? r.lb[i] >> 8 : r.lb[i], h = x ? r.h[i] >> 8 : r.h[i], h4 = h << 4, h2 = h << 2;
            o[2 * i + x] = mf_six_low(a, h4, shi[0], slo[0]);
            o[8 + 2 * i + x] = mf_six_low(b, h2, shi[1], slo[1]);
            o[16 + 2 * i + x] = mf_six_high(a, h4, shi[2], slo[2]);
            o[24 + 2 * i + x] = mf_six_high(b, h2, shi[3], slo[3]);
        }
}

// OUT: the product stores its own fp16 outputs; else all sums go to a.part
template <bool OUT>
__global__ void __launch_bounds__(MF_THREADS, 1) mf_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1,
                                                           const __grid_constant__ CUtensorMap map2, const __grid_constant__ MfArgs a) {
    extern __shared__ uint8_t mf_smem_raw[];
    __shared__ uint64_t w_full[MF_WSTAGES], w_empty[MF_WSTAGES], x_full[MF_XSTAGES], x_empty[MF_XSTAGES], a_full[MF_ASTAGES], a_empty[MF_ASTAGES], acc_full[2], acc_empty[2], drain_bar;
    __shared__ uint32_t tmem_slot;
    uint8_t* smem = mf_smem_raw + ((128u - (smem_u32(mf_smem_raw) & 127u)) & 127u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int si = 0;
    while (si + 1 < a.nseg && (int)blockIdx.x >= a.seg[si + 1].cta0) ++si;
    const MfSeg sg = a.seg[si];
    const int cta = blockIdx.x - sg.cta0, u0 = mf_first(sg, cta), u1 = mf_first(sg, cta + 1), nb = a.nb;
    const bool q6 = sg.q6 != 0;
    const int NP = a.NP, chunk = NP * 16;                                  // bytes of an activation chunk
    const int w_bytes = q6 ? MF_WBYTES6 : MF_WBYTES4, last_chunks = q6 ? 16 : 18;
    // a stage of activations: a super-block, half of one above 96 tokens; tensor memory holds three super-blocks of weights and two accumulators of 48 tokens
    const int parts = NP > 96 ? 2 : 1, x_bytes = (last_chunks + (parts == 1 ? 16 : 0)) * chunk;
    const int nx = min(MF_XSTAGES, (MF_SMEM - 128 - MF_OUT_BYTES - MF_WSTAGES * w_bytes) / x_bytes);
    const int na = NP <= 96 ? 3 : 2, acc_n = 512 - na * MF_ACOLS >= 2 * NP ? 2 : 1;
    uint8_t* xring = smem + MF_WSTAGES * w_bytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < MF_WSTAGES; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], MF_PRODUCERS / 2); }
        for (int s = 0; s < MF_XSTAGES; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 1); }
        for (int s = 0; s < MF_ASTAGES; ++s) { mbar_init(&a_full[s], MF_PRODUCERS / 2); mbar_init(&a_empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], MF_DRAINS); }
        mbar_init(&drain_bar, 1);
        fence_mbar_init();
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch();
    const uint32_t tmem = tmem_slot, acc0 = tmem + na * MF_ACOLS;

    if (warp == 0) {
        // weights: independent of the kernel in front
        if (lane == 0) {
            const CUtensorMap* map = si == 0 ? &map0 : si == 1 ? &map1 : &map2;
            const int p = q6 ? sg.perm : 1, rb = nb * Q6K_BYTES, rows = MF_ROWS / p;
            int n = 0, s = 0, tile = u0 / nb, kb = u0 - tile * nb;
            uint32_t parity = 1;
            for (int u = u0; u < u1; ++u, ++n) {
                if (!tc_wait(&w_empty[s], parity)) break;
                mbar_expect_tx(&w_full[s], w_bytes);
                uint8_t* dst = smem + s * w_bytes;
                if (!q6) tma_load_2d(dst, map, kb * Q4K_BYTES, tile * MF_ROWS, &w_full[s]);
                else for (int i = 0; i < p; ++i) tma_load_2d(dst + i * rows * MF_PITCH6, map, (i * rb + kb * Q6K_BYTES) & ~15, tile * rows, &w_full[s]);
                if (++kb == nb) { kb = 0; ++tile; }
                if (++s == MF_WSTAGES) { s = 0; parity ^= 1; }
            }
            if (n < u1 - u0) {
                atomicExch(a.status, JB_ERR_TIMEOUT);
                for (int i = n > MF_WSTAGES ? n - MF_WSTAGES : 0; i < n; ++i) tc_wait(&w_full[i % MF_WSTAGES], (i / MF_WSTAGES) & 1);      // own copies land before the CTA ends
            }
        }
    } else if (warp == 1) {
        // activations: written by the kernel in front
        pdl_wait();
        if (lane == 0) {
            const uint8_t* x = reinterpret_cast<const uint8_t*>(q6 ? a.x6 : a.x4);
            const size_t block = (size_t)(16 + last_chunks) * chunk;
            int n = 0, s = 0, kb = u0 % nb, part = 0;
            const int all = (u1 - u0) * parts;
            uint32_t parity = 1;
            for (; n < all; ++n) {
                if (!tc_wait(&x_empty[s], parity)) break;
                const uint32_t bytes = parts == 1 ? x_bytes : part ? last_chunks * chunk : 16 * chunk;
                mbar_expect_tx(&x_full[s], bytes);
                bulk_g2s(xring + (size_t)s * x_bytes, x + kb * block + part * 16 * chunk, bytes, &x_full[s]);
                if (++part == parts) { part = 0; if (++kb == nb) kb = 0; }
                if (++s == nx) { s = 0; parity ^= 1; }
            }
            if (n < all) {
                atomicExch(a.status, JB_ERR_TIMEOUT);
                for (int i = n > nx ? n - nx : 0; i < n; ++i) tc_wait(&x_full[i % nx], (i / nx) & 1);
            }
        }
    } else if (warp == 2) {
        // fp16 x fp16 -> fp32, A in tensor memory, B without swizzle: chunks of K NP * 16 bytes apart, groups of eight tokens 128.
        // The issue of the MMAs is the longest chain here (17 of them a super-block, each faster than its operands' set-up), so the whole warp
        // runs the loop (its values are then uniform), without divisions, and one lane issues.
        const bool leader = tc_elect();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(NP >> 3) << 17) | ((uint32_t)(MF_ROWS >> 4) << 24);
        const uint32_t bd_hi = 8u | (1u << 14), bd_lo0 = ((smem_u32(xring) >> 4) & 0x3FFFu) | ((uint32_t)NP << 16);
        const uint32_t step = 2u * NP, x16 = (uint32_t)x_bytes >> 4;       // 16-byte units from one K step, one stage to the next
        bool ok = true;
        uint32_t sa = 0, pa = 0, sx = 0, px = 0, acc = 0, pacc = 1, d = acc0;
        int kb = u0 % nb;
        bool first = true;
        for (int u = u0; u < u1; ++u) {
            if (first && !tc_wait_all(&acc_empty[acc], pacc)) { ok = false; break; }
            if (!tc_wait_all(&x_full[sx], px) || !tc_wait_all(&a_full[sa], pa)) { ok = false; break; }
            tc_fence_after();
            uint32_t ta = tmem + sa * MF_ACOLS, bd_lo = bd_lo0 + sx * x16;
            if (++kb == nb) kb = 0;
            const bool last = kb == 0 || u + 1 == u1;
            if (leader) {
                #pragma unroll
                for (int k = 0; k < 8; ++k) tc_mma_ts(d, ta + 8 * k, bd_lo + k * step, bd_hi, idesc, (uint32_t)(!first || k));
            }
            ta += 64; bd_lo += 8 * step;
            if (parts == 2) {
                if (leader) tc_commit(&x_empty[sx]);
                __syncwarp();
                if (++sx == (uint32_t)nx) { sx = 0; px ^= 1; }
                if (!tc_wait_all(&x_full[sx], px)) { ok = false; break; }
                tc_fence_after();
                bd_lo = bd_lo0 + sx * x16;
            }
            if (leader) {
                #pragma unroll
                for (int k = 0; k < 8; ++k) tc_mma_ts(d, ta + 8 * k, bd_lo + k * step, bd_hi, idesc, 1u);
                if (!q6) tc_mma_ts(d, ta + 64, bd_lo + 8 * step, bd_hi, idesc, 1u);
                tc_commit(&a_empty[sa]);
                tc_commit(&x_empty[sx]);
                if (last) tc_commit(&acc_full[acc]);
            }
            __syncwarp();
            first = last;
            if (++sa == (uint32_t)na) { sa = 0; pa ^= 1; }
            if (++sx == (uint32_t)nx) { sx = 0; px ^= 1; }
            if (last) {
                d += NP;
                if (++acc == (uint32_t)acc_n) { acc = 0; pacc ^= 1; d = acc0; }
            }
        }
        if (leader) {
            if (!ok) atomicExch(a.status, JB_ERR_TIMEOUT);
            tc_commit(&drain_bar);                                         // nothing may run on the tensor pipe when the columns are freed
            tc_wait(&drain_bar, 0);
        }
        __syncwarp();
    } else if (warp < 3 + MF_PRODUCERS) {
        // codes -> fp16 in tensor memory: two sets of eight warps take the super-blocks in turn, so that one set's waits and copies lie behind
        // the other's arithmetic; a thread has half a row of 128 weights
        const int pw = warp - 3, quarter = warp & 3, f = (pw >> 2) & 1, set = pw >> 3;
        const int row = 32 * quarter + lane;                               // lane of tensor memory; which row of the tile it is: see the drain
        const uint32_t lane_base = tmem + ((uint32_t)(32 * quarter) << 16);
        const int p = sg.perm, per = MF_ROWS / p, rb = nb * Q6K_BYTES;
        const uint32_t mis0 = q6 ? (uint32_t)((row / per) * rb) : 0u;      // byte of the row in its group of p
        const uint32_t w0 = smem_u32(smem) + row * (q6 ? MF_PITCH6 : MF_PITCH4);
        uint32_t s = set, pw_ = 0, sa = set, pa = 1;                       // MF_WSTAGES is even: a set has stages of weights of its own (a stage that changed hands could be a round further than its parity tells)
        int kb = (u0 + set) % nb;
        bool ok = true;
        for (int u = u0 + set; u < u1; u += 2) {
            if (!tc_wait_all(&w_full[s], pw_)) { ok = false; break; }
            const uint32_t col = lane_base + sa * MF_ACOLS + 64 * f;
            uint32_t o[32];
            if (!q6) {
                const uint32_t at = w0 + s * MF_WBYTES4;
                const uint4 hd = mf_lds128(at), q0 = mf_lds128(at + 16 + 64 * f), q1 = mf_lds128(at + 32 + 64 * f), q2 = mf_lds128(at + 48 + 64 * f), q3 = mf_lds128(at + 64 + 64 * f);
                const MfS4 sc = mf_scales4(hd, f);
                const __half2 c02 = __hmul2(mf_h2(0x48004800u), sc.d02), c13 = __hmul2(mf_h2(0x48004800u), sc.d13);      // centring constants: 8 half(d * sc)
                mf_codes4(o, q0, q1, __low2half2(sc.d02), __low2half2(sc.d13));
                if (!tc_wait_all(&a_empty[sa], pa)) { ok = false; break; }
                tc_fence_after();
                __syncwarp();
                mf_st32(col, o);
                mf_st4(lane_base + sa * MF_ACOLS + 128 + 4 * f, mf_u32(__lows2half2(sc.m02, sc.m13)), mf_u32(__lows2half2(c02, c13)), mf_u32(__highs2half2(sc.m02, sc.m13)), mf_u32(__highs2half2(c02, c13)));
                mf_codes4(o, q2, q3, __high2half2(sc.d02), __high2half2(sc.d13));
                __syncwarp();
                mf_st32(col + 32, o);
            } else {
                const uint32_t at = w0 + s * MF_WBYTES6 + ((mis0 + (uint32_t)(kb * Q6K_BYTES)) & 15u);
                MfQ6 r;
                mf_scales6(r, at, f);
                mf_load6(r, at, f, 0);
                mf_codes6(o, r, 0);
                if (!tc_wait_all(&a_empty[sa], pa)) { ok = false; break; }
                tc_fence_after();
                __syncwarp();
                mf_st32(col, o);
                mf_load6(r, at, f, 1);
                mf_codes6(o, r, 1);
                __syncwarp();
                mf_st32(col + 32, o);
                kb += 2;
                while (kb >= nb) kb -= nb;
            }
            mf_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&w_empty[s]); mbar_arrive(&a_full[sa]); }
            s += 2;
            if (s >= MF_WSTAGES) { s -= MF_WSTAGES; pw_ ^= 1; }
            sa += 2; if (sa >= (uint32_t)na) { sa -= na; pa ^= 1; }
        }
        if (!ok && lane == 0) atomicExch(a.status, JB_ERR_TIMEOUT);
    } else {
        // finished sums: fp32 to a.part, or fp16 outputs through shared memory (rows of a tile lie `perm` apart)
        pdl_wait();
        const int dw = warp - 3 - MF_PRODUCERS, quarter = warp & 3, pos = 32 * quarter + lane;
        __half* stage = reinterpret_cast<__half*>(xring + nx * x_bytes);
        const int p = sg.perm, per = MF_ROWS / p, row = (pos % per) * p + pos / per;      // row of the tile at this position
        uint32_t piece = 0;
        for (int u = u0; u < u1; ++piece) {
            const int tile = u / nb, kb0 = u - tile * nb, len = min(nb - kb0, u1 - u);
            const uint32_t acc = piece % acc_n;
            const bool full = tc_wait_all(&acc_full[acc], (piece / acc_n) & 1);
            if (OUT ? !mf_drains_all(full) : !full) { if (lane == 0) atomicExch(a.status, JB_ERR_TIMEOUT); break; }
            tc_fence_after();
            const bool whole = OUT && len == nb;
            float* dst = OUT ? a.part + ((size_t)(2 * blockIdx.x + (kb0 == 0)) * a.N) * MF_ROWS + pos
                             : a.part + (size_t)(cta - mf_owner(sg, tile * nb)) * a.N * a.rows + sg.m0 + tile * MF_ROWS + pos;
            const size_t ld = OUT ? MF_ROWS : a.rows;
            for (int t0 = 0; t0 < a.N; t0 += MF_OUT_TOK) {
                uint32_t r[16];
                __syncwarp();
                mf_ld16(acc0 + acc * NP + t0 + ((uint32_t)(32 * quarter) << 16), r);
                if (!whole) {
                    #pragma unroll
                    for (int t = 0; t < 16; ++t) if (t0 + t < a.N) dst[(size_t)(t0 + t) * ld] = __uint_as_float(r[t]);
                } else {
                    #pragma unroll
                    for (int t = 0; t < 16; ++t) stage[t * MF_ROWS + row] = __float2half_rn(__uint_as_float(r[t]));
                    asm volatile("bar.sync 2, 128;" ::: "memory");
                    // a token's 128 rows are 16 pieces of 16 bytes; eight tokens at a time
                    const int dt = dw * 32 + lane;
                    #pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int t = (dt >> 4) + 8 * i, r8 = 8 * (dt & 15), row8 = tile * MF_ROWS + r8;
                        if (t0 + t < a.N && row8 < sg.M)
                            *reinterpret_cast<uint4*>(a.y + (size_t)(t0 + t) * sg.M + row8) = *reinterpret_cast<const uint4*>(stage + t * MF_ROWS + r8);
                    }
                    asm volatile("bar.sync 2, 128;" ::: "memory");
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
            u += len;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Outputs of the tiles that several CTAs share: block (boundary between two CTAs, group of tokens); the first boundary inside a tile stands for it.
__global__ void __launch_bounds__(256) mf_edge_kernel(const __grid_constant__ MfArgs a) {
    pdl_wait();
    pdl_launch();
    const MfSeg& s = a.seg[0];
    const int u = mf_first(s, blockIdx.x + 1), tile = u / a.nb, kb = u - tile * a.nb, first = mf_owner(s, tile * a.nb);
    if (kb == 0 || u >= s.units || first != (int)blockIdx.x) return;
    const int last = mf_owner(s, (tile + 1) * a.nb - 1), lane = threadIdx.x & 31, t = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (t >= a.N) return;
    const int per = MF_ROWS / s.perm;
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int pos = 32 * i + lane, row = tile * MF_ROWS + (pos % per) * s.perm + pos / per;
        float v = a.part[((size_t)(2 * first + 1) * a.N + t) * MF_ROWS + pos];
        for (int c = first + 1; c <= last; ++c) v += a.part[((size_t)(2 * c) * a.N + t) * MF_ROWS + pos];
        if (row < s.M) a.y[(size_t)t * s.M + row] = __float2half_rn(v);
    }
}

// ── the kernels between the products ──────────────────────────────────────
// What they read: sums of rows 4 lane .. 4 lane + 3 of a tile, in order of K.
struct MfSums { const float* part; MfSeg seg[MF_MAX_SEG]; int nb, N, rows; };
// What a kernel can know before the product in front is done (where its sums lie, angles, weights of a norm) it forms ahead of its wait: rotation and
// SwiGLU kernels of eight streams 6.1 and 5.1 -> 3.3 us after their product's end.
struct MfPlace { const float* p; int count, perm; size_t slot; int at[4]; };
__device__ __forceinline__ MfPlace mf_place(const MfSums& a, const MfSeg& s, int tile, int tok, int lane) {
    const int first = mf_owner(s, tile * a.nb), per = MF_ROWS / s.perm, shift = __ffs(s.perm) - 1;
    MfPlace r;
    r.count = mf_owner(s, (tile + 1) * a.nb - 1) - first + 1;
    r.p = a.part + (size_t)tok * a.rows + s.m0 + tile * MF_ROWS;
    r.slot = (size_t)a.N * a.rows;
    r.perm = s.perm;
    #pragma unroll
    for (int e = 0; e < 4; ++e) r.at[e] = s.perm == 1 ? 4 * lane + e : ((4 * lane + e) & (s.perm - 1)) * per + ((4 * lane + e) >> shift);
    return r;
}
template <int BATCH>
__device__ __forceinline__ void mf_sum4(float (&v)[4], const MfPlace& s) {
    // every sum of a batch is requested before the first is added: one trip to L2 for all (added as they came, nine sums of W_down took 13 us)
    v[0] = v[1] = v[2] = v[3] = 0.f;
    for (int c0 = 0; c0 < s.count; c0 += BATCH) {
        float w[BATCH][4];
        #pragma unroll
        for (int c = 0; c < BATCH; ++c) {
            const float* q = s.p + (c0 + c) * s.slot;
            if (c0 + c >= s.count) w[c][0] = w[c][1] = w[c][2] = w[c][3] = 0.f;
            else if (s.perm == 1) {
                const float4 x = *reinterpret_cast<const float4*>(q + s.at[0]);
                w[c][0] = x.x; w[c][1] = x.y; w[c][2] = x.z; w[c][3] = x.w;
            } else {
                #pragma unroll
                for (int e = 0; e < 4; ++e) w[c][e] = q[s.at[e]];
            }
        }
        #pragma unroll
        for (int c = 0; c < BATCH; ++c)
            if (c0 + c < s.count) { v[0] += w[c][0]; v[1] += w[c][1]; v[2] += w[c][2]; v[3] += w[c][3]; }
    }
}
struct MfQuant { __half* x4; __half* x6; int N, NP; };
// Elements 4 lane .. 4 lane + 3 of 128 consecutive ones (fp16 values), group 4 kq + lane / 8 of super-block kb, quantised as in mmq_tc.cu;
// the sum of x in the order of that kernel's 32-lane tree (partners 16, 8, 4, 2, 1 apart).
__device__ __forceinline__ void mf_quantise4(const MfQuant& a, const float (&v)[4], int kb, int kq, int tok, int lane) {
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    #pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    const float d = __fdiv_rn(amax, 127.0f), dinv = d > 0.f ? __fdiv_rn(1.0f, d) : 0.f;
    const int j = 4 * kq + (lane >> 3), e0 = 4 * (lane & 7);
    float q[4];
    int qsum = 0;
    #pragma unroll
    for (int i = 0; i < 4; ++i) { const int c = __float2int_rn(__fmul_rn(v[i], dinv)); qsum += c; q[i] = (float)c; }
    if (a.x4) {
        float s[4];
        #pragma unroll
        for (int i = 0; i < 4; ++i) { s[i] = v[i] + __shfl_xor_sync(0xFFFFFFFFu, v[i], 4); }
        #pragma unroll
        for (int i = 0; i < 4; ++i) { s[i] = s[i] + __shfl_xor_sync(0xFFFFFFFFu, s[i], 2); }
        #pragma unroll
        for (int i = 0; i < 4; ++i) { s[i] = s[i] + __shfl_xor_sync(0xFFFFFFFFu, s[i], 1); }
        const float sum = __fadd_rn(__fadd_rn(s[0], s[2]), __fadd_rn(s[1], s[3]));
        #pragma unroll
        for (int o = 4; o > 0; o >>= 1) qsum += __shfl_xor_sync(0xFFFFFFFFu, qsum, o);
        const float dh = __half2float(__float2half_rn(d));
        __half* x = a.x4 + (size_t)kb * 34 * a.NP * 8;
        const int at = mf_pos4(j, e0);
        *reinterpret_cast<uint2*>(x + ((size_t)(at >> 3) * a.NP + tok) * 8 + (at & 7)) =
            make_uint2(mf_pack(__float2half_rn(__fmul_rn(dh, q[0])), __float2half_rn(__fmul_rn(dh, q[2]))),
                       mf_pack(__float2half_rn(__fmul_rn(dh, q[1])), __float2half_rn(__fmul_rn(dh, q[3]))));
        if ((lane & 7) == 0) {                            // columns 256 + 4 il ..: sums of the two groups of run il, then their centring sums
            const int ex = 4 * (j >> 1) + (j & 1);
            __half* o = x + ((size_t)(32 + (ex >> 3)) * a.NP + tok) * 8 + (ex & 7);
            o[0] = __float2half_rn(sum);
            o[2] = __float2half_rn(__fmul_rn(dh, (float)qsum));
        }
    }
    if (a.x6) {
        __half* x = a.x6 + (size_t)kb * 32 * a.NP * 8;
        const int at = mf_pos6(j, e0);
        *reinterpret_cast<uint2*>(x + ((size_t)(at >> 3) * a.NP + tok) * 8 + (at & 7)) =
            make_uint2(mf_pack(__float2half_rn(__fmul_rn(d, q[0])), __float2half_rn(__fmul_rn(d, q[2]))),
                       mf_pack(__float2half_rn(__fmul_rn(d, q[1])), __float2half_rn(__fmul_rn(d, q[3]))));
    }
}
__device__ __forceinline__ void mf_load4(float (&v)[4], const __half* p) {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void mf_store4(__half* p, const float (&v)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(mf_pack(__float2half_rn(v[0]), __float2half_rn(v[1])), mf_pack(__float2half_rn(v[2]), __float2half_rn(v[3])));
}
__device__ __forceinline__ float mf_half(float v) { return __half2float(__float2half_rn(v)); }

// One CTA per token, a warp per 128 elements (MF_NORM_TILES per warp at most).  Bound by its launch and one trip to L2: the sums, x and
// the weights are requested together.
constexpr int MF_NORM_TILES = 4;
template <int TILES, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) mf_norm_kernel(const __grid_constant__ MfSums sums, const __half* x, __half* x_out, const float* w, float eps, int H, MfQuant q) {
    __shared__ float red[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, tok = blockIdx.x, tiles = H / MF_ROWS;
    pdl_launch();
    MfPlace at = {};
    float4 wn = make_float4(0.f, 0.f, 0.f, 0.f);
    if (TILES == 1) {                                     // a warp per tile
        if (sums.part) at = mf_place(sums, sums.seg[0], warp, tok, lane);
        if (w) wn = *reinterpret_cast<const float4*>(w + warp * MF_ROWS + 4 * lane);
    }
    pdl_wait();
    float v[TILES][4], ss = 0.f;
    #pragma unroll
    for (int i = 0; i < TILES; ++i) {
        const int tile = warp + i * warps;
        if (tile >= tiles) break;
        mf_load4(v[i], x + (size_t)tok * H + tile * MF_ROWS + 4 * lane);
        if (sums.part) {
            float y[4];
            if (TILES > 1) at = mf_place(sums, sums.seg[0], tile, tok, lane);
            mf_sum4<THREADS < 1024 ? 5 : 3>(y, at);
            #pragma unroll
            for (int e = 0; e < 4; ++e) v[i][e] = mf_half(__fadd_rn(v[i][e], mf_half(y[e])));
            mf_store4(x_out + (size_t)tok * H + tile * MF_ROWS + 4 * lane, v[i]);
        }
        #pragma unroll
        for (int e = 0; e < 4; ++e) ss += v[i][e] * v[i][e];
    }
    if (!w) return;
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    ss = 0.f;
    for (int i = 0; i < warps; ++i) ss += red[i];
    const float rrms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)H), eps)));
    #pragma unroll
    for (int i = 0; i < TILES; ++i) {
        const int tile = warp + i * warps;
        if (tile >= tiles) break;
        if (TILES > 1) wn = *reinterpret_cast<const float4*>(w + tile * MF_ROWS + 4 * lane);
        const float wv[4] = {wn.x, wn.y, wn.z, wn.w};
        #pragma unroll
        for (int e = 0; e < 4; ++e) v[i][e] = mf_half(__fmul_rn(__fmul_rn(v[i][e], rrms), wv[e]));
        mf_quantise4(q, v[i], tile >> 1, tile & 1, tok, lane);
    }
}

// A warp per head of 128 and token: the arithmetic of qkv_prep_kernel (elementwise.cu) on the fp16 results of the products.
__global__ void __launch_bounds__(256, 3) mf_prep_kernel(const __grid_constant__ MfSums sums, const __grid_constant__ MfPrep a, const __grid_constant__ RopeFreq fr) {
    const int lane = threadIdx.x & 31, head = blockIdx.x * 8 + (threadIdx.x >> 5), tok = blockIdx.y;
    pdl_launch();
    if (head >= a.n_heads + 2 * a.n_kv) { pdl_wait(); return; }
    const bool is_q = head < a.n_heads, is_k = !is_q && head < a.n_heads + a.n_kv;
    const int hh = is_q ? head : is_k ? head - a.n_heads : head - a.n_heads - a.n_kv;
    const int pos = (a.d_pos ? *a.d_pos : a.pos) + tok * a.pos_step;
    // Ahead of the wait for the product: the position, which was settled before the kernels of this step (the first of them starts no kernel early),
    // its angles, and where the sums lie.
    float c[4], s[4];
    if (is_q || is_k) {
        #pragma unroll
        for (int e = 0; e < 4; ++e) sincosf(__fmul_rn((float)pos, fr.f[a.neox ? 4 * (lane & 15) + e : 2 * lane + e / 2]), &s[e], &c[e]);
    }
    const MfPlace at_ = mf_place(sums, sums.seg[is_q ? 0 : is_k ? 1 : 2], hh, tok, lane);
    pdl_wait();
    float v[4];
    mf_sum4<4>(v, at_);
    #pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = mf_half(v[e]);
    if (is_q || is_k) {
        const float* nw = is_q ? a.q_norm : a.k_norm;
        if (nw) {
            const float ss = warp_sum((v[0] * v[0] + v[1] * v[1]) + (v[2] * v[2] + v[3] * v[3]));
            const float rrms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, 128.0f), a.eps)));
            const float4 wn = *reinterpret_cast<const float4*>(nw + 4 * lane);
            const float wv[4] = {wn.x, wn.y, wn.z, wn.w};
            #pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = mf_half(__fmul_rn(__fmul_rn(v[e], rrms), wv[e]));
        }
        if (a.neox) {                                     // pairs (i, i + 64): the partner is 16 lanes away
            #pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float o = __shfl_xor_sync(0xFFFFFFFFu, v[e], 16);
                v[e] = mf_half(lane < 16 ? __fsub_rn(__fmul_rn(v[e], c[e]), __fmul_rn(o, s[e])) : __fadd_rn(__fmul_rn(o, s[e]), __fmul_rn(v[e], c[e])));
            }
        } else {
            #pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const float v0 = v[e], v1 = v[e + 1];
                v[e] = mf_half(__fsub_rn(__fmul_rn(v0, c[e]), __fmul_rn(v1, s[e])));
                v[e + 1] = mf_half(__fadd_rn(__fmul_rn(v0, s[e]), __fmul_rn(v1, c[e])));
            }
        }
        if (is_q) { mf_store4(a.q + ((size_t)tok * a.n_heads + hh) * 128 + 4 * lane, v); return; }
    }
    const float mx = warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
    const float scale = __fdiv_rn(mx, 127.0f), inv = scale > 0.f ? __fdiv_rn(127.0f, mx) : 0.f;
    int8_t* cache = a.k_list ? (is_k ? a.k_list : a.v_list)[tok] : is_k ? a.k : a.v;
    float* scales = a.k_list ? (is_k ? a.ks_list : a.vs_list)[tok] : is_k ? a.ks : a.vs;
    const size_t at = (size_t)pos * a.n_kv + hh;
    uint32_t codes = 0;
    #pragma unroll
    for (int e = 0; e < 4; ++e) codes |= (uint32_t)(max(-127, min(127, __float2int_rn(__fmul_rn(v[e], inv)))) & 0xFF) << (8 * e);
    *reinterpret_cast<uint32_t*>(cache + at * 128 + 4 * lane) = codes;
    if (lane == 0) scales[at] = scale;
}

// A warp per 128 elements and token: silu(gate) * up of the sums (glu_kernel's arithmetic), or fp16 vectors as they are.
template <bool GLU>
__global__ void __launch_bounds__(256) mf_vec_kernel(const __grid_constant__ MfSums sums, const __half* x, int K, MfQuant q) {
    const int lane = threadIdx.x & 31, tile = blockIdx.x * 8 + (threadIdx.x >> 5), tok = blockIdx.y;
    pdl_launch();
    if (tile >= K / MF_ROWS) { pdl_wait(); return; }
    MfPlace g_at, u_at;
    if (GLU) { g_at = mf_place(sums, sums.seg[0], tile, tok, lane); u_at = mf_place(sums, sums.seg[1], tile, tok, lane); }
    pdl_wait();
    float v[4];
    if (GLU) {
        float u[4];
        mf_sum4<2>(v, g_at);
        mf_sum4<2>(u, u_at);
        #pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float g = mf_half(v[e]);
            v[e] = mf_half(__fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), mf_half(u[e])));
        }
    } else {
        mf_load4(v, x + (size_t)tok * K + tile * MF_ROWS + 4 * lane);
    }
    mf_quantise4(q, v, tile >> 1, tile & 1, tok, lane);
}

// ── host side ─────────────────────────────────────────────────────────────
bool mf_plan(MfProduct& p, const MfWeight* w, int n, int K) {
    DeviceCtx* c = ctx();
    if (!c || n < 1 || n > MF_MAX_SEG || K <= 0 || K % QK_K || !encode_tiled_fn()) return false;
    const int nb = K / QK_K;
    p = MfProduct();
    p.nseg = n; p.K = K;
    double cost[MF_MAX_SEG], all = 0;
    for (int i = 0; i < n; ++i) {
        MfSeg& s = p.seg[i];
        s.q6 = w[i].type == T_Q6K;
        // tensor maps: rows from 16-byte boundaries, `perm` of them a multiple of 16 bytes, none left over; 16-byte stores of eight outputs
        if ((!s.q6 && w[i].type != T_Q4K) || !w[i].W || ((uintptr_t)w[i].W & 15) || w[i].M < 8 || w[i].M % 8) return false;
        s.perm = 1;
        while (s.q6 && (long long)s.perm * nb % 8) s.perm *= 2;
        s.M = w[i].M; s.tiles = (s.M + MF_ROWS - 1) / MF_ROWS; s.units = s.tiles * nb; s.m0 = p.rows;
        if ((long long)s.tiles * nb > (1 << 22)) return false;     // mf_first and mf_owner multiply in 32 bits
        p.rows += s.tiles * MF_ROWS;
        all += cost[i] = s.units * (s.q6 ? 1.45 : 1.0);            // bytes of a super-block, and the work of unpacking it
        const int rb = nb * block_bytes(w[i].type), pitch = s.q6 ? MF_PITCH6 : MF_PITCH4;
        const cuuint64_t gdim[2] = {(cuuint64_t)s.perm * rb, (cuuint64_t)(s.M / s.perm)};
        const cuuint64_t gstr[1] = {(cuuint64_t)s.perm * rb};
        const cuuint32_t box[2] = {(cuuint32_t)pitch, (cuuint32_t)(MF_ROWS / s.perm)}, estr[2] = {1, 1};
        if (encode_tiled_fn()(&p.map[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(w[i].W), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return false;
    }
    // SMs in proportion to the work
    int left = c->sm_count, cta0 = 0;
    for (int i = 0; i < n; ++i) {
        MfSeg& s = p.seg[i];
        int g = i + 1 == n ? left : (int)(left * cost[i] / all + 0.5);
        if (g > left - (n - 1 - i)) g = left - (n - 1 - i);
        if (g < 1) g = 1;
        all -= cost[i]; left -= g;
        s.cta0 = cta0; s.ctas = g < s.units ? g : s.units;
        cta0 += s.ctas;
        for (int t = 0; t < s.tiles; ++t) {
            const int k = mf_owner(s, (t + 1) * nb - 1) - mf_owner(s, t * nb) + 1;
            if (k > p.slots) p.slots = k;
        }
    }
    return true;
}
size_t mf_edge_bytes(int N) { DeviceCtx* c = ctx(); return (size_t)(c ? c->sm_count : 148) * 2 * N * MF_ROWS * sizeof(float); }

static int mf_launch(const MfProduct& p, const MfOperand& x, float* part, __half* y, int N, cudaStream_t st) {
    DeviceCtx* c = ctx();
    if (!c) return JB_ERR_CUDA;
    MfArgs a = {};
    int grid = 0;
    for (int i = 0; i < p.nseg; ++i) { a.seg[i] = p.seg[i]; grid = p.seg[i].cta0 + p.seg[i].ctas; }
    a.nseg = p.nseg; a.nb = p.K / QK_K; a.N = N; a.NP = mf_padded(N); a.rows = p.rows; a.x4 = x.x4; a.x6 = x.x6; a.part = part; a.y = y;
    a.status = c->d_status;
    auto kern = y ? mf_kernel<true> : mf_kernel<false>;
    if (!c->mf_attr[y ? 1 : 0]) {
        JB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MF_SMEM));
        c->mf_attr[y ? 1 : 0] = true;
    }
    static const bool verbose = getenv("JLLM_B200_MMQ_DEBUG") != nullptr;
    for (int i = 0; verbose && i < p.nseg; ++i)
        fprintf(stderr, "[mmq_few] type %d M=%d N=%d K=%d: %d of %d CTAs, %d tiles of %d super-blocks\n", p.seg[i].q6 ? T_Q6K : T_Q4K, p.seg[i].M, N, p.K, p.seg[i].ctas, grid, p.seg[i].tiles, a.nb);
    JB_CUDA(launch_k(kern, dim3(grid), dim3(MF_THREADS), MF_SMEM, st, pdl_enabled(), p.map[0], p.map[p.nseg > 1 ? 1 : 0], p.map[p.nseg > 2 ? 2 : 0], a));
    count_launch();
    if (y && grid > 1) {
        JB_CUDA(launch_k(mf_edge_kernel, dim3(grid - 1, (N + 7) / 8), dim3(256), 0, st, pdl_enabled(), a));
        count_launch();
    }
    return JB_OK;
}
int launch_mf_sums(const MfProduct& p, const MfOperand& x, float* part, int N, cudaStream_t st) { return mf_launch(p, x, part, nullptr, N, st); }
int launch_mf_out(const MfProduct& p, const MfOperand& x, __half* y, float* edge, int N, cudaStream_t st) { return mf_launch(p, x, edge, y, N, st); }

static MfSums mf_sums(const MfProduct* p, const float* part, int N) {
    MfSums s = {};
    if (!p) return s;
    s.part = part; s.nb = p->K / QK_K; s.N = N; s.rows = p->rows;
    for (int i = 0; i < p->nseg; ++i) s.seg[i] = p->seg[i];
    return s;
}
int launch_mf_norm(const MfProduct* p, const float* part, const __half* x, __half* x_out, const float* w, float eps, int H, const MfOperand& q, int N, cudaStream_t st) {
    const int tiles = H / MF_ROWS, warps = tiles < 32 ? tiles : 32;
    if (H % MF_ROWS || tiles > 32 * MF_NORM_TILES) return set_error(JB_ERR_ARG, "few-token norm: width %d", H);
    auto kern = tiles <= 20 ? mf_norm_kernel<1, 640> : tiles <= 32 ? mf_norm_kernel<1, 1024> : tiles <= 64 ? mf_norm_kernel<2, 1024> : mf_norm_kernel<4, 1024>;      // by registers
    JB_CUDA(launch_k(kern, dim3(N), dim3(32 * warps), 0, st, pdl_enabled(), mf_sums(p, part, N), x, x_out, w, eps, H, MfQuant{q.x4, q.x6, N, mf_padded(N)}));
    count_launch();
    return JB_OK;
}
int launch_mf_prep(const MfProduct& p, const float* part, const MfPrep& a, float theta, int N, cudaStream_t st) {
    JB_CUDA(launch_k(mf_prep_kernel, dim3((a.n_heads + 2 * a.n_kv + 7) / 8, N), dim3(256), 0, st, pdl_enabled(), mf_sums(&p, part, N), a, make_rope_freq(128, theta)));
    count_launch();
    return JB_OK;
}
int launch_mf_glu(const MfProduct& p, const float* part, const MfOperand& q, int N, cudaStream_t st) {
    const int I = p.seg[0].M;
    JB_CUDA(launch_k(mf_vec_kernel<true>, dim3((I / MF_ROWS + 7) / 8, N), dim3(256), 0, st, pdl_enabled(), mf_sums(&p, part, N), (const __half*)nullptr, I, MfQuant{q.x4, q.x6, N, mf_padded(N)}));
    count_launch();
    return JB_OK;
}
int launch_mf_quantise(const __half* x, const MfOperand& q, int K, int N, cudaStream_t st) {
    JB_CUDA(launch_k(mf_vec_kernel<false>, dim3((K / MF_ROWS + 7) / 8, N), dim3(256), 0, st, pdl_enabled(), MfSums(), x, K, MfQuant{q.x4, q.x6, N, mf_padded(N)}));
    count_launch();
    return JB_OK;
}

// The scratch of a model over N tokens.
static size_t mf_align(size_t b) { return (b + 255) & ~(size_t)255; }
bool MfModel::plan(const jllm_b200_model_desc& m, bool with_out) {
    layers.clear();
    // the switches that choose among the general kernels are theirs: a session under one of them runs these
    static const bool off = [] {
        const char *mmq = getenv("JLLM_B200_MMQ"), *stream = getenv("JLLM_B200_MMQ_STREAM"), *pair = getenv("JLLM_B200_MMQ_PAIR");
        return (mmq && !strcmp(mmq, "cuda")) || (stream && stream[0] == '0') || (pair && pair[0] == '0');
    }();
    if (off) return false;
    hidden = m.hidden_dim; q_dim = m.n_heads * m.head_dim; ffn = m.intermediate_dim;
    const int kv_dim = m.n_kv_heads * m.head_dim;
    // a head is a 128-row tile; norms keep a token in one CTA's registers
    if (m.head_dim != MF_ROWS || hidden % QK_K || q_dim % QK_K || ffn % QK_K || hidden > 32 * MF_NORM_TILES * MF_ROWS) return false;
    auto own = [](const void* W) { return resolve_weight(W) == W ? W : nullptr; };       // weights in host memory are read by the other kernels
    // norm vectors are read as float4; others (from inside a file, say) are read element by element by the other kernels, which also refuse null ones
    auto norm = [](const float* w) { return w && !((uintptr_t)w & 15); };
    if (with_out && !norm(m.output_norm)) return false;
    std::vector<MfLayer> all(m.n_layers);
    for (int l = 0; l < m.n_layers; ++l) {
        const jllm_b200_layer_desc& w = m.layers[l];
        if (!norm(w.rms_attn) || !norm(w.rms_ffn) || (w.q_norm && !norm(w.q_norm)) || (w.k_norm && !norm(w.k_norm))) return false;
        const MfWeight qkv[3] = {{own(w.wq), w.type_wq, q_dim}, {own(w.wk), w.type_wk, kv_dim}, {own(w.wv), w.type_wv, kv_dim}};
        const MfWeight wo = {own(w.wo), w.type_wo, hidden}, gu[2] = {{own(w.w_gate), w.type_w_gate, ffn}, {own(w.w_up), w.type_w_up, ffn}}, down = {own(w.w_down), w.type_w_down, hidden};
        if (!mf_plan(all[l].qkv, qkv, 3, hidden) || !mf_plan(all[l].wo, &wo, 1, q_dim) || !mf_plan(all[l].gate_up, gu, 2, hidden) || !mf_plan(all[l].down, &down, 1, ffn)) return false;
    }
    if (with_out) {
        const MfWeight o = {own(m.output), m.output_type, m.vocab_size};
        if (!mf_plan(out, &o, 1, hidden)) return false;
    }
    layers.swap(all);
    return true;
}
size_t MfModel::bytes(int N) const {
    size_t p = out.nseg ? mf_edge_bytes(N) : 0;
    for (const MfLayer& l : layers)
        for (const MfProduct* q : {&l.qkv, &l.wo, &l.gate_up, &l.down})
            if (mf_part_bytes(*q, N) > p) p = mf_part_bytes(*q, N);
    return 2 * mf_align(mf_x_bytes(hidden, N)) + mf_align(mf_x_bytes(q_dim, N)) + mf_align(mf_x_bytes(ffn, N)) + mf_align(p);
}
void MfModel::place(void* scratch, int N) {
    char* p = (char*)scratch;
    auto take = [&](size_t b) { char* r = p; p += mf_align(b); return (void*)r; };
    xh4 = take(mf_x_bytes(hidden, N)); xh6 = take(mf_x_bytes(hidden, N)); xa = take(mf_x_bytes(q_dim, N)); xi = take(mf_x_bytes(ffn, N));
    part = (float*)p;
}

static size_t mr_bytes(int K, int N) { return mf_align((size_t)N * mr_width(K) * sizeof(__half)); }
size_t MfModel::row_bytes(int N) const { return 2 * mr_bytes(hidden, N) + mr_bytes(q_dim, N) + mr_bytes(ffn, N); }
void MfModel::place_rows(void* scratch, int N) {
    char* p = (char*)scratch;
    auto take = [&](int K) { char* r = p; p += mr_bytes(K, N); return (void*)r; };
    xh4 = take(hidden); xh6 = take(hidden); xa = take(q_dim); xi = take(ffn);
}

}  // namespace jb
