// mmq_quant.cuh — rows of the tensor-core products' activation operand (mmq_tc.cu): X'[t][0..K) = half(d * q) (codes x scale of the reference's
// quantiser, mmq_q4k_llama.cu:383-404, mmq_q6k_llama.cu:424-438); for Q4_K matrices also X'[t][K + g] = half(sum of x over group g) (the
// reference's DS4 sum) and X'[t][K + K/32 + g] = half(d * sum of codes of group g), zero up to the padded width Kp; for Q6_K ones d stays fp32.
#pragma once
#include "common.cuh"

namespace jb {

__device__ __forceinline__ void mq_load8(float (&v)[8], const __half* p) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i])); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void mq_store8(__half* p, const float (&v)[8]) {
    uint32_t w[4];
    #pragma unroll
    for (int i = 0; i < 4; ++i) { const __half2 h = __halves2half2(__float2half_rn(v[2 * i]), __float2half_rn(v[2 * i + 1])); w[i] = *reinterpret_cast<const uint32_t*>(&h); }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
// A warp's super-block sb of one token: lane 4j + c holds elements 8c..8c+7 of group j.  row4, row6: the token's rows (null: not wanted).
// The sum of x is taken in the order of a 32-lane xor-shuffle tree over single elements (partners 16, 8, 4, 2, 1 apart), so that it has the bits
// of the reference's quantiser and of its CPU restatement.
__device__ __forceinline__ void mq_rows8(const float (&v)[8], __half* row4, __half* row6, int sb, int K, int Kp, int lane) {
    const int G = K / 32, gi = sb * 8 + (lane >> 2);
    float amax = 0.f;
    #pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    const float d = __fdiv_rn(amax, 127.0f), dinv = d > 0.f ? __fdiv_rn(1.0f, d) : 0.f;
    float q[8];
    int qsum = 0;
    #pragma unroll
    for (int i = 0; i < 8; ++i) { const int c = __float2int_rn(__fmul_rn(v[i], dinv)); qsum += c; q[i] = (float)c; }
    auto products = [&](__half* row, float s) {
        float o[8];
        #pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = __fmul_rn(s, q[i]);
        mq_store8(row + (size_t)sb * QK_K + 8 * lane, o);
    };
    if (row4) {
        float s[8];
        #pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = v[i] + __shfl_xor_sync(0xFFFFFFFFu, v[i], 2);       // elements 16 apart
        #pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = s[i] + __shfl_xor_sync(0xFFFFFFFFu, s[i], 1);       // 8 apart
        const float sum = __fadd_rn(__fadd_rn(__fadd_rn(s[0], s[4]), __fadd_rn(s[2], s[6])), __fadd_rn(__fadd_rn(s[1], s[5]), __fadd_rn(s[3], s[7])));   // 4, 2, 1 apart
        qsum += __shfl_xor_sync(0xFFFFFFFFu, qsum, 1);
        qsum += __shfl_xor_sync(0xFFFFFFFFu, qsum, 2);
        const float dh = __half2float(__float2half_rn(d));
        products(row4, dh);
        if ((lane & 3) == 0) {
            row4[K + gi] = __float2half_rn(sum);
            row4[K + G + gi] = __float2half_rn(__fmul_rn(dh, (float)qsum));
        }
        if (sb == 0) for (int z = K + 2 * G + lane; z < Kp; z += 32) row4[z] = __float2half_rn(0.f);
    }
    if (row6) products(row6, d);
}

}  // namespace jb
