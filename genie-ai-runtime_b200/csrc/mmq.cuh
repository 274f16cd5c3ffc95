// mmq.cuh — prefill / batched K-quant GEMM launchers.
#pragma once
#include "common.cuh"
#include <functional>
#include <vector>

namespace jb {

// y[N x M] half (token-major) = x[N x K] half . W^T, W in Q4_K / Q6_K blocks, with the
// arithmetic of the reference's default prefill path (gemm_quant_batched,
// src/kernels/gemv_q4.cu:2478-2495 -> mmq_q4k_llama.cu / mmq_q6k_llama.cu).
// own: the scratch of a session that has one; else the library's for this stream.
// dbg_dots (optional): integer accumulators [N][M][K/32] (Q4_K) or [N][M][K/16] (Q6_K).
int launch_mmq(__half* y, const void* W, int type, const __half* x, int M, int N, int K, int32_t* dbg_dots, cudaStream_t st, MmqWork* own = nullptr);
// the same with a residual added on the way out (y = half(float(residual) + float(half(product))), residual [N][M] or null)
// and, for a second matrix multiplied by the SAME activations right after the first on this stream, `same_x_as_last`
int launch_mmq_ex(__half* y, const void* W, int type, const __half* x, int M, int N, int K, const __half* residual, bool same_x_as_last,
                  cudaStream_t st, MmqWork* own = nullptr);
int launch_mmq_pair(__half* y1, __half* y2, const void* W1, int type1, const void* W2, int type2, const __half* x, int M1, int M2, int N, int K,
                    cudaStream_t st, MmqWork* own = nullptr);
// The tensor-core path over activations that are quantised already: xq [N][columns of mmq_tc.cu's operand for `type`]
int launch_mmq_ready(__half* y1, __half* y2, const void* W1, const void* W2, int type, const __half* xq, int M1, int M2, int N, int K, cudaStream_t st, MmqWork* own = nullptr);
size_t mmq_scratch_bytes(int N, int K);
// The library's scratch for a stream (own: a session's), kept from other threads while it lives; w null: there is none to be had
struct MmqPool; struct MmqEntry;
struct MmqLease {
    MmqWork* w; cudaStream_t st; bool cap;       // cap: the stream is being captured
    MmqLease(MmqWork* own, cudaStream_t stream);
    ~MmqLease();
    MmqLease(const MmqLease&) = delete;
    MmqLease& operator=(const MmqLease&) = delete;
private:
    MmqPool* pool = nullptr; MmqEntry* e = nullptr;
};
void mmq_mark(cudaStream_t st);       // all products on st so far may be taken for over once the stream has come here
cudaError_t mmq_alloc(void** p, size_t bytes);      // cudaMalloc, whether this thread or another one captures
// tensor-core path (mmq_tc.cu): tcgen05.mma over fp16 operands built from the same quantised values
bool   mmq_tc_applies(const void* W, int type, int M, int N, int K);
size_t mmq_tc_scratch_bytes(int type, int M, int N, int K);
int    launch_mmq_tc_pair(__half* y, __half* y2, const void* W, const void* W2, int type, const __half* x, __half* xq, int M, int M2, int N, int K,
                          bool same_x_as_last, cudaStream_t st, MmqWork& work, void* wide = nullptr, const __half* ready = nullptr);
size_t mmq_tc_scratch_bytes_pair(int type, int M, int M2, int N, int K);
// many tokens: the weights are expanded to the fp16 operand once, then multiplied by gemm_pair.cu
bool   mmq_wide_applies(int M, int M2, int N, int K);
constexpr size_t MMQ_WEIGHT_BYTES = (size_t)64 << 20;      // expanded weights of a piece, at most
struct MmqPiece { const void* W; const void* W2; int type, M, M2, K, r0, rows; };      // rows r0 .. of W's and W2's (null: none) rows in a row
size_t mmq_piece_bytes(const MmqPiece& p);                 // of its expanded weights
void   mmq_pieces(std::vector<MmqPiece>& out, const void* W1, const void* W2, int type, int M1, int M2, int K);
int    launch_mmq_expand(const MmqPiece& p, void* wq, bool ahead, cudaStream_t st);
// behind: launches to go right behind the product, before the sum of its K ranges; part: gemm_pair_part_floats
int    launch_mmq_piece(const MmqPiece& p, const void* wq, const __half* xq, __half* y1, __half* y2, int N, float* part, cudaStream_t st, const std::function<int()>& behind = nullptr);
// few tokens (2..64): weights streamed once, mma.sync on fp16 operands with the tensor-core path's arithmetic (mmq_stream.cu)
bool   mmq_stream_applies(const void* W, int type, int M, int N, int K);
size_t mmq_stream_scratch_bytes(int type, int M, int N, int K);
int    launch_mmq_stream(__half* y, const void* W, int type, const __half* x, void* scratch, int M, int N, int K, const __half* residual,
                         bool reuse_operand, cudaStream_t st, MmqWork& work);

}  // namespace jb
