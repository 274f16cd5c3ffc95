// mmq_rows.cu — what lies between the K-quant products of many tokens: residual and RMSNorm, head norms with rotation and the cache rows, SwiGLU;
// each writes the operand of the product that follows.
//
// At a few hundred tokens their launches and trips to memory set the time, beyond that the arithmetic on an element (the quantiser's
// conversions, expf and the division of SwiGLU): eight elements a lane, 16-byte accesses, angles once per token.  512 tokens, hidden 2560, MLP 9728,
// 32 / 8 heads, as separate kernels with a quantiser each / here, us: residual, norm and quantiser (for Q4_K and for Q6_K matrices) 14.4 / 5.1;
// head norms, rotation and cache rows 16.6 / 9.6; SwiGLU and quantiser 12.8 / 9.9.
#include "mmq_few.cuh"
#include "mmq_quant.cuh"

namespace jb {

struct MrOut { __half* x4; __half* x6; int K, Kp; };
__device__ __forceinline__ void mr_store(const MrOut& o, const float (&v)[8], int tok, int sb, int lane) {
    mq_rows8(v, o.x4 ? o.x4 + (size_t)tok * o.Kp : nullptr, o.x6 ? o.x6 + (size_t)tok * o.K : nullptr, sb, o.K, o.Kp, lane);
}
__device__ __forceinline__ float mr_half(float v) { return __half2float(__float2half_rn(v)); }

// One CTA per token, a warp per super-block (BLOCKS of them at most).
template <int BLOCKS>
__global__ void __launch_bounds__(1024) mr_norm_kernel(const __half* x, const __half* add, __half* x_out, const float* w, float eps, int H, MrOut out) {
    __shared__ float red[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, tok = blockIdx.x, nsb = H / QK_K;
    pdl_launch();
    pdl_wait();
    float v[BLOCKS][8], ss = 0.f;
    #pragma unroll
    for (int i = 0; i < BLOCKS; ++i) {
        const int sb = warp + i * warps;
        if (sb >= nsb) break;
        const size_t at = (size_t)tok * H + sb * QK_K + 8 * lane;
        mq_load8(v[i], x + at);
        if (add) {
            float y[8];
            mq_load8(y, add + at);
            #pragma unroll
            for (int e = 0; e < 8; ++e) v[i][e] = mr_half(__fadd_rn(v[i][e], y[e]));
            mq_store8(x_out + at, v[i]);
        }
        #pragma unroll
        for (int e = 0; e < 8; ++e) ss += v[i][e] * v[i][e];
    }
    if (!w) return;
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    ss = 0.f;
    for (int i = 0; i < warps; ++i) ss += red[i];
    const float rrms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)H), eps)));
    #pragma unroll
    for (int i = 0; i < BLOCKS; ++i) {
        const int sb = warp + i * warps;
        if (sb >= nsb) break;
        #pragma unroll
        for (int e = 0; e < 8; e += 4) {
            const float4 n = *reinterpret_cast<const float4*>(w + sb * QK_K + 8 * lane + e);
            v[i][e] = mr_half(__fmul_rn(__fmul_rn(v[i][e], rrms), n.x)); v[i][e + 1] = mr_half(__fmul_rn(__fmul_rn(v[i][e + 1], rrms), n.y));
            v[i][e + 2] = mr_half(__fmul_rn(__fmul_rn(v[i][e + 2], rrms), n.z)); v[i][e + 3] = mr_half(__fmul_rn(__fmul_rn(v[i][e + 3], rrms), n.w));
        }
        mr_store(out, v[i], tok, sb, lane);
    }
}

// One CTA per token: the angles of its position are formed once for all its heads (64 sincosf; one per head and pair was most of the time), then
// a warp per head of 128: the arithmetic of qkv_prep_kernel (elementwise.cu).
__global__ void __launch_bounds__(256) mr_prep_kernel(const __grid_constant__ MrPrep a, const __grid_constant__ RopeFreq fr) {
    __shared__ float2 turn[64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tok = blockIdx.x, pos = a.pos + tok;
    if (threadIdx.x < 64) {
        float c, s;
        sincosf(__fmul_rn((float)pos, fr.f[threadIdx.x]), &s, &c);
        turn[threadIdx.x] = make_float2(c, s);
    }
    __syncthreads();
    pdl_launch();
    pdl_wait();
    float2 t[4];
    #pragma unroll
    for (int e = 0; e < 4; ++e) t[e] = a.neox ? turn[4 * (lane & 15) + e] : turn[2 * lane + e / 2];
    for (int head = warp; head < a.n_heads + 2 * a.n_kv; head += 8) {
        const bool is_q = head < a.n_heads, is_k = !is_q && head < a.n_heads + a.n_kv;
        const int hh = is_q ? head : is_k ? head - a.n_heads : head - a.n_heads - a.n_kv;
        const __half* src = (is_q ? a.q + (size_t)tok * a.n_heads * 128 : (is_k ? a.k_in : a.v_in) + (size_t)tok * a.n_kv * 128) + hh * 128 + 4 * lane;
        const uint2 raw = *reinterpret_cast<const uint2*>(src);
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        float v[4] = {lo.x, lo.y, hi.x, hi.y};
        if (is_q || is_k) {
            const float* nw = is_q ? a.q_norm : a.k_norm;
            if (nw) {
                const float ss = warp_sum((v[0] * v[0] + v[1] * v[1]) + (v[2] * v[2] + v[3] * v[3]));
                const float rrms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, 128.0f), a.eps)));
                const float4 wn = *reinterpret_cast<const float4*>(nw + 4 * lane);
                const float wv[4] = {wn.x, wn.y, wn.z, wn.w};
                #pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = mr_half(__fmul_rn(__fmul_rn(v[e], rrms), wv[e]));
            }
            if (a.neox) {                                 // pairs (i, i + 64): the partner is 16 lanes away
                #pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float o = __shfl_xor_sync(0xFFFFFFFFu, v[e], 16);
                    v[e] = mr_half(lane < 16 ? __fsub_rn(__fmul_rn(v[e], t[e].x), __fmul_rn(o, t[e].y)) : __fadd_rn(__fmul_rn(o, t[e].y), __fmul_rn(v[e], t[e].x)));
                }
            } else {
                #pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const float v0 = v[e], v1 = v[e + 1];
                    v[e] = mr_half(__fsub_rn(__fmul_rn(v0, t[e].x), __fmul_rn(v1, t[e].y)));
                    v[e + 1] = mr_half(__fadd_rn(__fmul_rn(v0, t[e].y), __fmul_rn(v1, t[e].x)));
                }
            }
            if (is_q) {
                const __half2 o0 = __halves2half2(__float2half_rn(v[0]), __float2half_rn(v[1])), o1 = __halves2half2(__float2half_rn(v[2]), __float2half_rn(v[3]));
                *reinterpret_cast<uint2*>(a.q + ((size_t)tok * a.n_heads + hh) * 128 + 4 * lane) = make_uint2(*reinterpret_cast<const uint32_t*>(&o0), *reinterpret_cast<const uint32_t*>(&o1));
                continue;
            }
        }
        const float mx = warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
        const float scale = __fdiv_rn(mx, 127.0f), inv = scale > 0.f ? __fdiv_rn(127.0f, mx) : 0.f;
        const size_t at = (size_t)pos * a.n_kv + hh;
        uint32_t codes = 0;
        #pragma unroll
        for (int e = 0; e < 4; ++e) codes |= (uint32_t)(max(-127, min(127, __float2int_rn(__fmul_rn(v[e], inv)))) & 0xFF) << (8 * e);
        *reinterpret_cast<uint32_t*>((is_k ? a.k : a.v) + at * 128 + 4 * lane) = codes;
        if (lane == 0) (is_k ? a.ks : a.vs)[at] = scale;
    }
}

// A warp per super-block and token: silu(gate) * up (glu_kernel's arithmetic), or x as it is.
template <bool GLU>
__global__ void __launch_bounds__(256) mr_vec_kernel(const __half* x, const __half* up, int N, MrOut out) {
    const int lane = threadIdx.x & 31, nsb = out.K / QK_K;
    const long long item = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    pdl_launch();
    pdl_wait();
    if (item >= (long long)N * nsb) return;
    const int tok = (int)(item / nsb), sb = (int)(item - (long long)tok * nsb);
    const size_t at = (size_t)tok * out.K + sb * QK_K + 8 * lane;
    float v[8];
    mq_load8(v, x + at);
    if (GLU) {
        float u[8];
        mq_load8(u, up + at);
        #pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = mr_half(__fmul_rn(__fdiv_rn(v[e], __fadd_rn(1.0f, expf(-v[e]))), u[e]));
    }
    mr_store(out, v, tok, sb, lane);
}

static MrOut mr_out(const MfOperand& q, int K) { return MrOut{q.x4, q.x6, K, mr_width(K)}; }
int launch_mr_norm(const __half* x, const __half* add, __half* x_out, const float* w, float eps, int H, const MfOperand& q, int N, cudaStream_t st) {
    const int nsb = H / QK_K, warps = nsb < 32 ? nsb : 32;
    if (H % QK_K || nsb > 64) return set_error(JB_ERR_ARG, "norm over rows: width %d", H);
    JB_CUDA(launch_k(nsb <= 32 ? mr_norm_kernel<1> : mr_norm_kernel<2>, dim3(N), dim3(32 * warps), 0, st, pdl_enabled(), x, add, x_out, w, eps, H, mr_out(q, H)));
    count_launch();
    return JB_OK;
}
int launch_mr_prep(const MrPrep& a, float theta, int N, cudaStream_t st) {
    JB_CUDA(launch_k(mr_prep_kernel, dim3(N), dim3(256), 0, st, pdl_enabled(), a, make_rope_freq(128, theta)));
    count_launch();
    return JB_OK;
}
template <bool GLU>
static int mr_vec(const __half* x, const __half* up, const MfOperand& q, int K, int N, cudaStream_t st) {
    const long long items = (long long)N * (K / QK_K);
    JB_CUDA(launch_k(mr_vec_kernel<GLU>, dim3((unsigned)((items + 7) / 8)), dim3(256), 0, st, pdl_enabled(), x, up, N, mr_out(q, K)));
    count_launch();
    return JB_OK;
}
int launch_mr_glu(const __half* gate, const __half* up, const MfOperand& q, int K, int N, cudaStream_t st) { return mr_vec<true>(gate, up, q, K, N, st); }
int launch_mr_quantise(const __half* x, const MfOperand& q, int K, int N, cudaStream_t st) { return mr_vec<false>(x, nullptr, q, K, N, st); }

}  // namespace jb
