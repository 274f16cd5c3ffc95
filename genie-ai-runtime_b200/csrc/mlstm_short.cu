// mlstm_short.cu — the mLSTM recurrence of a prompt (or the end of one) of 16 to 64 tokens: one chunk, on mma.sync (m16n8k16, fp32 accumulation).
//
// The formulas are those of mlstm_chunk.cu, whose warps hand a chunk of 128 tokens on to one another through a dozen barriers: right where
// chunk follows chunk, but with a single one every hand-over is waited for.  Here a CTA (one head, 32 value columns) takes its chunk in three steps
// between barriers: rows and gates, weighted scores, outputs and state.  8 heads of 256 x 512, 16 / 64 tokens, with the norm that
// follows: 12.1 / 13.5 us, in mlstm_chunk.cu 16.4 / 17.4; 65 tokens as two chunks of 64 took 19.5, in one of mlstm_chunk.cu 17.4.
//
// Warps 0-15 compute; warp 16 forms the gates (F, A and M in fp64, handed on as two floats each), warps 17-19 fetch rows by cp.async, 17 and 18
// form n . q.  n is one more column of the state product, its values ones.  fp32 operands go in as two bf16 parts, as there.
#include "mlstm.cuh"
#include "mma.cuh"

namespace jb {

constexpr int MH_L = MLSTM_SHORT, MH_V = 32, MH_WARPS = 16, MH_COMPUTE = 32 * MH_WARPS, MH_THREADS = MH_COMPUTE + 128;

struct MhGates { float2 A[MH_L], M[MH_L]; float a[MH_L], w[MH_L], em[MH_L], decay; };      // a = e^(m_0 - M_t), w = e^(A_s - M_L), em = e^(-m_t)
struct MhArgs { MlstmCall c; int n, start; };

__device__ __forceinline__ float2 mh_two(double x) { const float hi = (float)x; return make_float2(hi, (float)(x - (double)hi)); }
__device__ __forceinline__ float mh_weight(float2 A, float2 M) { return expf((A.x - M.x) + (A.y - M.y)); }
// 64-byte rows (32 columns), conflict-free for ldmatrix
__device__ __forceinline__ uint32_t mh_off(int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); }
__device__ __forceinline__ void mh_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    hi = fa_pack(x, y);
    lo = fa_pack(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xFFFF0000u));
}
__device__ __forceinline__ void mh_st32(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t mh_ld32(uint32_t addr) { uint32_t v; asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr)); return v; }

// RB: bytes of a row of q or k in shared memory (dim rounded up to 64 elements)
template <int RB> struct MhLayout {
    static constexpr uint32_t up(uint32_t b) { return (b + 127) & ~127u; }
    static constexpr uint32_t q = 0, k = q + MH_L * RB, v = k + MH_L * RB, vw = v + MH_L * 64, p = vw + 2 * MH_L * 64, s = p + 2 * MH_L * 128, g = s + 2 * (RB / 2) * 64,
                              n = g + up(sizeof(MhGates)), nq = n + (RB / 2) * 4, sum = nq + MH_L * 4, bytes = sum + 4 * MH_L * 4;
};

// one warp; m: the maximum carried in, then the one to carry on
__device__ __forceinline__ void mh_gates(const MlstmCall& c, int h, int n, double& m, MhGates* g) {
    const int lane = threadIdx.x & 31;
    double f[2], a[2];
    #pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        f[e] = t < n ? (double)mlstm_log_f(c, t, h) : 0.0;
        a[e] = t < n ? (double)mlstm_log_i(c, t, h) : -1e30;
    }
    double F = f[0] + f[1];                                         // inclusive sums over lane pairs
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(0xFFFFFFFFu, F, o); if (lane >= o) F += u; }
    const double F0 = F - f[1], F1 = F;
    a[0] -= F0; a[1] -= F1;
    double M = fmax(a[0], a[1]);
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(0xFFFFFFFFu, M, o); if (lane >= o) M = fmax(M, u); }
    double before = __shfl_up_sync(0xFFFFFFFFu, M, 1);
    if (lane == 0) before = -1e30;
    const double M0 = fmax(m, fmax(before, a[0])), M1 = fmax(m, M);
    const double ML = __shfl_sync(0xFFFFFFFFu, M1, 31), FL = __shfl_sync(0xFFFFFFFFu, F1, 31);
    #pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        const double Mt = e ? M1 : M0;
        g->A[t] = mh_two(a[e]); g->M[t] = mh_two(Mt);
        g->a[t] = expf((float)(m - Mt));
        g->w[t] = t < n ? expf((float)(a[e] - ML)) : 0.f;
        g->em[t] = expf((float)(-((e ? F1 : F0) + Mt)));
    }
    if (lane == 0) g->decay = expf((float)(m - ML));
    m = FL + ML;
}

template <int RB>
__global__ void __launch_bounds__(MH_THREADS, 1) mlstm_short_kernel(const MhArgs p) {
    extern __shared__ __align__(128) unsigned char mh_sm[];
    __shared__ volatile int odd;                                     // some value is an infinity or NaN
    const MlstmCall& c = p.c;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane & 7, lm = lane >> 3, h = blockIdx.y, v0 = blockIdx.x * MH_V;
    constexpr int KT = RB / 32, QC = RB / 16;                        // 16-row tiles of the dimension (at most one per warp), 16-byte chunks of a row
    using L = MhLayout<RB>;
    const int D = c.dim, vld = pad8(c.vdim), steps = (p.n + 15) >> 4;       // tokens in sixteens
    const uint32_t sm = smem_u32(mh_sm), qa = sm + L::q, ka = sm + L::k, va = sm + L::v;
    MhGates& g = *reinterpret_cast<MhGates*>(mh_sm + L::g);
    float* ns = reinterpret_cast<float*>(mh_sm + L::n);
    float* nq = reinterpret_cast<float*>(mh_sm + L::nq);
    float* rsum = reinterpret_cast<float*>(mh_sm + L::sum);           // [quarter of the tokens scored][token]
    float* Sg = c.state + (size_t)h * D * vld;
    float* ng = c.state + (size_t)c.heads * D * vld + (size_t)h * D;
    float* mg = c.state + (size_t)c.heads * D * vld + (size_t)c.heads * D + h;
    const __nv_bfloat16* proj = reinterpret_cast<const __nv_bfloat16*>(c.proj);
    const bool fresh = p.start == 0;
    const float qscale = 1.0f / sqrtf((float)D);
    if (tid == 0) odd = 0;
    pdl_wait();
    pdl_launch();
    float S[4][4];                                                   // rows 16 warp .., columns 8 nt ..
    if (warp < MH_WARPS) {
        #pragma unroll
        for (int nt = 0; nt < 4; ++nt)
            #pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = warp * 16 + (lane >> 2) + 8 * (e >> 1), v = v0 + nt * 8 + (lane & 3) * 2 + (e & 1);
                S[nt][e] = !fresh && d < D && v < vld ? Sg[(size_t)d * vld + v] : 0.f;
            }
        if (warp < KT) {                                             // the state as two bf16 parts for the product with q
            #pragma unroll
            for (int nt = 0; nt < 4; ++nt)
                #pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    uint32_t hi, lo;
                    mh_split(S[nt][2 * hf], S[nt][2 * hf + 1], hi, lo);
                    const uint32_t o = mh_off(warp * 16 + (lane >> 2) + 8 * hf, nt) + (lane & 3) * 4;
                    mh_st32(sm + L::s + o, hi);
                    mh_st32(sm + L::s + (RB / 2) * 64 + o, lo);
                }
        }
        for (int d = tid; d < RB / 2; d += MH_COMPUTE) ns[d] = !fresh && d < D ? ng[d] : 0.f;
    } else if (warp == MH_WARPS) {
        double m = fresh ? 0.0 : (double)*mg;
        mh_gates(c, h, p.n, m, &g);
        // other slices may still have to read n and m: the new ones wait beside them for the launch that follows
        if (blockIdx.x == 0 && lane == 0) mg[mlstm_next(c)] = (float)m;
    } else {
        for (int i = tid - MH_COMPUTE - 32; i < 16 * steps * QC; i += 96) {
            const int r = i / QC, cc = i - r * QC;
            const bool in = r < p.n && cc * 8 < D;
            const __nv_bfloat16* row = proj + (size_t)r * c.ld + h * D + cc * 8;
            fa_cp16(qa + fa_off<RB / 2>(r, cc), in ? row + c.off_q : proj, in);
            fa_cp16(ka + fa_off<RB / 2>(r, cc), in ? row + c.off_k : proj, in);
        }
        for (int i = tid - MH_COMPUTE - 32; i < 4 * MH_L; i += 96) {  // all 64: weights of zero meet those behind the last
            const int r = i >> 2, cc = i & 3;
            const bool in = r < p.n && v0 + cc * 8 < c.vdim;
            fa_cp16(va + mh_off(r, cc), in ? proj + (size_t)r * c.ld + c.off_v + h * c.vdim + v0 + cc * 8 : proj, in);
        }
        fa_commit();
        fa_wait<0>();
    }
    __syncthreads();                                                 // rows, gates and state are there
    if (warp == MH_WARPS) return;
    if (warp > MH_WARPS) {
        if (warp < MH_WARPS + 3) {                                   // n . q of the carried normaliser, a token per lane
            const int r = tid - MH_COMPUTE - 32;
            float dot = 0.f;
            #pragma unroll 8
            for (int k = 0; k < QC; ++k) {
                uint32_t x[4];
                asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(qa + fa_off<RB / 2>(r, k)));
                const float4 n0 = load4(ns + 8 * k), n1 = load4(ns + 8 * k + 4);
                dot = fmaf(n0.x, __uint_as_float(x[0] << 16), dot); dot = fmaf(n0.y, __uint_as_float(x[0] & 0xFFFF0000u), dot);
                dot = fmaf(n0.z, __uint_as_float(x[1] << 16), dot); dot = fmaf(n0.w, __uint_as_float(x[1] & 0xFFFF0000u), dot);
                dot = fmaf(n1.x, __uint_as_float(x[2] << 16), dot); dot = fmaf(n1.y, __uint_as_float(x[2] & 0xFFFF0000u), dot);
                dot = fmaf(n1.z, __uint_as_float(x[3] << 16), dot); dot = fmaf(n1.w, __uint_as_float(x[3] & 0xFFFF0000u), dot);
            }
            nq[r] = dot * qscale;
        }
        asm volatile("bar.arrive 1, %0;" ::"n"(MH_THREADS - 32) : "memory");
        return;
    }
    const int wm = warp & 3, wn = warp >> 2;
    if (wm < steps) {
        // scores of 16 tokens against 16, weighted by the gates
        float s[2][2][4];                                            // even and odd steps
        #pragma unroll
        for (int i = 0; i < 4; ++i) { s[i >> 1][i & 1][0] = s[i >> 1][i & 1][1] = s[i >> 1][i & 1][2] = s[i >> 1][i & 1][3] = 0.f; }
        const bool any = wn <= wm;                                   // some of the one are not later than some of the other
        if (any) {
            #pragma unroll 4
            for (int k = 0; k < KT; ++k) {
                uint32_t a[4], kb[4];
                fa_ldsm(a, qa + fa_off<RB / 2>(wm * 16 + (lane & 15), k * 2 + (lane >> 4)));
                fa_ldsm(kb, ka + fa_off<RB / 2>(wn * 16 + (lm >> 1) * 8 + lr, k * 2 + (lm & 1)));
                fa_mma(s[k & 1][0], a, kb[0], kb[1]);
                fa_mma(s[k & 1][1], a, kb[2], kb[3]);
            }
        }
        #pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int t = wm * 16 + (lane >> 2) + 8 * hf;
            const float2 Mt = g.M[t];
            float sum = 0.f;
            #pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int s0 = wn * 16 + i * 8 + (lane & 3) * 2;
                const float x = any && s0 <= t ? (s[0][i][2 * hf] + s[1][i][2 * hf]) * qscale * mh_weight(g.A[s0], Mt) : 0.f;
                const float y = any && s0 + 1 <= t ? (s[0][i][2 * hf + 1] + s[1][i][2 * hf + 1]) * qscale * mh_weight(g.A[s0 + 1], Mt) : 0.f;
                sum += x + y;
                uint32_t hi, lo;
                mh_split(x, y, hi, lo);
                const uint32_t o = fa_off<64>(t, s0 >> 3) + (lane & 3) * 4;
                mh_st32(sm + L::p + o, hi);
                mh_st32(sm + L::p + MH_L * 128 + o, lo);
            }
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
            if ((lane & 3) == 0) rsum[wn * MH_L + t] = sum;
        }
    }
    if (tid < 4 * MH_L) {                                            // values weighted for the state
        const int r = tid >> 2, cc = tid & 3;
        uint32_t x[4], hi[4], lo[4];
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(va + mh_off(r, cc)));
        const float w = g.w[r];
        bool finite = true;
        #pragma unroll
        for (int e = 0; e < 4; ++e) {
            finite = finite && (x[e] & 0x7F80u) != 0x7F80u && (x[e] & 0x7F800000u) != 0x7F800000u;
            mh_split(w * __uint_as_float(x[e] << 16), w * __uint_as_float(x[e] & 0xFFFF0000u), hi[e], lo[e]);
        }
        if (!finite) odd = 1;
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(sm + L::vw + mh_off(r, cc)), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(sm + L::vw + MH_L * 64 + mh_off(r, cc)), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
    }
    asm volatile("bar.sync 1, %0;" ::"n"(MH_THREADS - 32) : "memory");      // the scores, the weighted values and n . q are there
    if (wm < steps) {
        // outputs of 16 tokens x 8 columns: the carried state, then the chunk's own tokens
        float o[4] = {0.f, 0.f, 0.f, 0.f}, o2[4] = {0.f, 0.f, 0.f, 0.f};        // of the two parts
        #pragma unroll 4
        for (int k = 0; k < KT; ++k) {
            uint32_t a[4], sb[4];
            fa_ldsm(a, qa + fa_off<RB / 2>(wm * 16 + (lane & 15), k * 2 + (lane >> 4)));
            fa_ldsm_t(sb, sm + L::s + (uint32_t)(lm >> 1) * (RB / 2) * 64 + mh_off(k * 16 + (lm & 1) * 8 + lr, wn));
            fa_mma(o, a, sb[0], sb[1]);
            fa_mma(o2, a, sb[2], sb[3]);
        }
        #pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float f = qscale * g.a[wm * 16 + (lane >> 2) + 8 * (e >> 1)];
            o[e] *= f; o2[e] *= f;
        }
        if (!odd) {
            #pragma unroll
            for (int kk = 0; kk < 4; kk += 2) {
                if (kk <= wm) {                                      // later tokens weigh nothing
                    uint32_t vb[4];
                    fa_ldsm_t(vb, va + mh_off(kk * 16 + lm * 8 + lr, wn));
                    #pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        uint32_t a[4], a1[4];
                        fa_ldsm(a, sm + L::p + part * MH_L * 128 + fa_off<64>(wm * 16 + (lane & 15), kk * 2 + (lane >> 4)));
                        fa_ldsm(a1, sm + L::p + part * MH_L * 128 + fa_off<64>(wm * 16 + (lane & 15), kk * 2 + 2 + (lane >> 4)));
                        fa_mma(part ? o2 : o, a, vb[0], vb[1]);
                        fa_mma(part ? o2 : o, a1, vb[2], vb[3]);
                    }
                }
            }
        } else {                                                     // a weight of zero times an infinity or NaN of a later token: not by the product
            #pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int t = wm * 16 + (lane >> 2) + 8 * hf;
                for (int s = 0; s <= t; ++s) {
                    const uint32_t at = sm + L::p + fa_off<64>(t, s >> 3) + (s & 6) * 2, hi = mh_ld32(at), lo = mh_ld32(at + MH_L * 128), x = mh_ld32(va + mh_off(s, wn) + (lane & 3) * 4);
                    const float w = s & 1 ? __uint_as_float(hi & 0xFFFF0000u) + __uint_as_float(lo & 0xFFFF0000u) : __uint_as_float(hi << 16) + __uint_as_float(lo << 16);
                    o[2 * hf] = fmaf(w, __uint_as_float(x << 16), o[2 * hf]); o[2 * hf + 1] = fmaf(w, __uint_as_float(x & 0xFFFF0000u), o[2 * hf + 1]);
                }
            }
        }
        #pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int t = wm * 16 + (lane >> 2) + 8 * hf, v = v0 + wn * 8 + (lane & 3) * 2;
            if (t < p.n && v < c.vdim) {
                const float z = g.a[t] * nq[t] + ((rsum[t] + rsum[MH_L + t]) + (rsum[2 * MH_L + t] + rsum[3 * MH_L + t]));
                const float inv = 1.0f / (fmaxf(fabsf(z), g.em[t]) + 1e-6f);
                *reinterpret_cast<float2*>(c.raw + ((size_t)t * c.heads + h) * c.vdim + v) = make_float2((o[2 * hf] + o2[2 * hf]) * inv, (o[2 * hf + 1] + o2[2 * hf + 1]) * inv);
            }
        }
    }
    // the state after the chunk
    if (warp >= KT) return;
    const float decay = g.decay;
    #pragma unroll
    for (int nt = 0; nt < 4; ++nt) { S[nt][0] *= decay; S[nt][1] *= decay; S[nt][2] *= decay; S[nt][3] *= decay; }
    float N[4] = {0.f, 0.f, 0.f, 0.f};                               // column 0: sum of w_s k_s by the weights' first parts, column 1 by their second
    #pragma unroll
    for (int kk = 0; kk < MH_L / 16; ++kk) {
        if (kk >= steps) break;
        uint32_t wb[2];
        #pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float2 w = *reinterpret_cast<const float2*>(&g.w[kk * 16 + e * 8 + (lane & 3) * 2]);
            uint32_t hi, lo;
            mh_split(w.x, w.y, hi, lo);
            wb[e] = lane < 4 ? hi : lane < 8 ? lo : 0u;
        }
        uint32_t a[4];
        fa_ldsm_t(a, ka + fa_off<RB / 2>(kk * 16 + (lm >> 1) * 8 + lr, warp * 2 + (lm & 1)));
        #pragma unroll
        for (int part = 0; part < 2; ++part)
            #pragma unroll
            for (int n2 = 0; n2 < 2; ++n2) {
                uint32_t vb[4];
                fa_ldsm_t(vb, sm + L::vw + part * MH_L * 64 + mh_off(kk * 16 + (lm & 1) * 8 + lr, n2 * 2 + (lm >> 1)));
                fa_mma(S[2 * n2], a, vb[0], vb[1]);
                fa_mma(S[2 * n2 + 1], a, vb[2], vb[3]);
            }
        fa_mma(N, a, wb[0], wb[1]);
    }
    #pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
        const int d = warp * 16 + (lane >> 2) + 8 * hf;
        if (d >= D) continue;
        if (blockIdx.x == 0 && (lane & 3) == 0) ng[mlstm_next(c) + d] = fmaf(ns[d], decay, N[2 * hf] + N[2 * hf + 1]);
        #pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const int v = v0 + nt * 8 + (lane & 3) * 2;
            if (v < vld) *reinterpret_cast<float2*>(Sg + (size_t)d * vld + v) = make_float2(S[nt][2 * hf], S[nt][2 * hf + 1]);
        }
    }
}

template <int RB>
static int mh_go(const MlstmCall& a, int n, int start, bool& attr, cudaStream_t st) {
    if (!attr) { JB_CUDA(cudaFuncSetAttribute(mlstm_short_kernel<RB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MhLayout<RB>::bytes)); attr = true; }
    const MhArgs p = {a, n, start};
    JB_CUDA(launch_k(mlstm_short_kernel<RB>, dim3((a.vdim + MH_V - 1) / MH_V, a.heads), dim3(MH_THREADS), (size_t)MhLayout<RB>::bytes, st, pdl_enabled(), p));
    count_launch();
    return JB_OK;
}
int launch_mlstm_short(const MlstmCall& a, int n, int start, cudaStream_t st) {
    DeviceCtx* x = ctx();
    if (!x) return set_error(JB_ERR_STATE, "mlstm short: library not initialised");
    if (n > MLSTM_SHORT) return set_error(JB_ERR_ARG, "mlstm short: %d tokens", n);
    bool (&attr)[3] = x->mlstm_short_attr;
    return a.dim <= 64 ? mh_go<128>(a, n, start, attr[0], st) : a.dim <= 128 ? mh_go<256>(a, n, start, attr[1], st) : mh_go<512>(a, n, start, attr[2], st);
}

}  // namespace jb
