// Internal launcher interfaces shared by the translation units of the library.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

#include <cudaTypedefs.h>

#include <atomic>

namespace race {

// launch with programmatic dependence on the kernel before (common.cuh); for kernels in which every thread calls chain_wait
// before its first access to global memory, so that the launch means the same as a plain one
// Only for calls of up to 2^17 stream-tokens of 64 buckets, whose kernels take microseconds: in longer ones a successor
// with 200 KB of shared memory that is resident early takes the L1 from the streaming kernel still running.  Plain over
// chained time of whole calls, eight heads, at 2^13 / 2^15 / 2^17 / 2^19: fp32 forward 1.25 / 1.12 / 1.03 / 1.01, training
// 1.06 / 1.10 / 0.99 / 0.93; bf16 with S = 64 forward 1.10 / 1.16 / 1.01 / 0.93, training 1.03 / 1.03 / 0.93 / 0.90; bf16 with
// S = 512 forward 1.24 / 1.12 / 1.06 / 1.04, training 1.04 / 1.04 / 1.06 / 0.97.
inline bool chain_launches(int64_t stream_tokens, int buckets) { return stream_tokens * buckets <= (64ll << 17); }
inline bool chain_launches(const Dims& dm) { return chain_launches(dm.N * dm.T, dm.S); }
template <typename... P, typename... A>
cudaError_t launch_chain(bool chained, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                         A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<A&&>(args)...);
}

// SMs of the current device (148 where there is none); asked for several times in a call, so the answer is kept per device
inline int device_sm_count() {
    static std::atomic<int> known[64];
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev < 64 && (sms = known[dev].load(std::memory_order_relaxed)) > 0) return sms;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
    if (dev < 64) known[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

// the driver's tensor-map encoder (causal_tc.cu); null if it cannot be looked up
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();

// ---- CUDA-core causal path (causal_simt.cu) -------------------------------------------------
int simt_groups(int S);
bool simt_supported(const Dims& dm);
int simt_default_tile_tokens(const Dims& dm, int sm_count);
// tile totals -> scan -> outputs; totals_only stops after the scan and writes only state_out;
// skip_output stops after the scan but leaves the exclusive tile prefixes in ws; global_norm selects
// the global-normalisation estimator (one denominator per token) in the output pass.
cudaError_t causal_fwd_simt(const void* pq, const void* pk, const void* v, void* out,
                            const float* carry_in, float* state_out, float* ws, const Dims& dm,
                            int dtype, int tile_tokens, bool totals_only, cudaStream_t stream,
                            bool skip_output = false, bool skip_totals = false, bool global_norm = false);

// in-place exclusive scan over the per-tile totals in ws (+ carry_in), inclusive total to state_out
// (reverse: exclusive SUFFIX sums, last tile first -- the scans of the backward)
cudaError_t causal_scan_tiles(float* ws, const float* carry_in, float* state_out, const Dims& dm,
                              int tile_tokens, cudaStream_t stream, bool write_prefix = true, bool reverse = false);

// which passes of a causal forward to run: totals (per-tile sums into ws) and/or scan + outputs.  kPhasePrefixOnly, with
// kPhaseTotals alone: the caller uses the totals for the prefixes of the tiles only, so the last tile's are not formed
// (with kPhaseAll that follows from state_out == null).
constexpr int kPhaseTotals = 1, kPhaseOutput = 2, kPhaseAll = 3, kPhasePrefixOnly = 4;

// Whether the output kernel forms the state before each tile itself (CarryFold) instead of a tile_scan launch between
// the two.  A launch costs 2 to 5 us in the chain of a small call; folding reads every tile's predecessors again, about
// tiles^2 / 2 states per stream, from lines of L2 that many CTAs ask for at once.  Scan over fold time of 64-token tiles:
// 1.10 wherever N tiles^2 is at most 2048 (1 to 64 streams, 2 to 32 tiles; at least 1.06 with d_k = 128, whose states are twice
// as large); from 4096 on 0.99 to 1.02 with d_k = 64 and 0.94 to 0.97 with d_k = 128; at 8192 down to 0.96 and 0.78.  Hence
// the line at N tiles^2 = 14 per SM.  One or two tiles: always less than the scan reads and writes (bf16, 48 streams of three
// tiles: 100 -> 93 us).
// A state written over the carry it came from would be read by other tiles' CTAs after the write: scan then.
inline bool fold_carry(int64_t N, int64_t tiles, int64_t state_floats, const float* carry_in, const float* state_out) {
    if (tiles > 1 && carry_in && state_out && carry_in < state_out + N * state_floats &&
        state_out < carry_in + N * state_floats)
        return false;
    return tiles <= 2 || (tiles <= 32 && N * tiles * tiles <= 14 * (int64_t)device_sm_count());
}

// ---- causal backward (causal_bwd_simt.cu): S <= 64, d_k <= 128 ---------------------------------
bool causal_bwd_supported(const Dims& dm, int dtype);
// grad_carry: with the gradient of a carried-in state
int causal_bwd_tile_tokens(const Dims& dm, int dtype, int sm_count, bool grad_carry);
size_t causal_bwd_workspace_bytes(const Dims& dm, int dtype, int tile_tokens, bool grad_carry);
// carry_in: state before the first token (nullable); d_state: gradient reaching the state after the last token
// (nullable); d_carry: receives the gradient of carry_in (nullable)
cudaError_t causal_bwd_simt(const void* pq, const void* pk, const void* v, const void* dout, const float* carry_in,
                            const float* d_state, void* dpq, void* dpk, void* dv, float* d_carry, void* ws,
                            const Dims& dm, int dtype, int tile_tokens, cudaStream_t stream, int* status = nullptr);

// ---- non-causal path (noncausal_simt.cu) ------------------------------------------------------
cudaError_t noncausal_query(const void* pq, const float* totals, void* out, const Dims& dm, int dtype,
                            int sm_count, cudaStream_t stream);
cudaError_t noncausal_state_grads(const float* totals, const float* dE_state, float* grads,
                                  const Dims& dm, cudaStream_t stream);
cudaError_t noncausal_token_grads(const void* pk, const void* v, const void* dout, const float* totals,
                                  const float* grads, void* dpq, void* dpk, void* dv, const Dims& dm,
                                  int dtype, int sm_count, cudaStream_t stream);

// tensor-core token kernels of the non-causal path (noncausal_tc.cu): S = 64, d_k = 64
bool noncausal_tensor_supported(const Dims& dm, int dtype);
cudaError_t noncausal_query_tensor(const void* pq, const float* totals, void* out, const Dims& dm, int dtype,
                                   int sm_count, cudaStream_t stream);
// de_state: the totals pass over (pQ, dO) in state layout
cudaError_t noncausal_token_grads_tensor(const void* pk, const void* v, const void* dout, const float* totals,
                                         const float* de_state, void* dpq, void* dpk, void* dv, const Dims& dm,
                                         int dtype, int sm_count, cudaStream_t stream);

// ---- bucket-probability producer (bucket_probs.cu) --------------------------------------------
// exact: fp32 accuracy of the projections (training) at the tensor-core geometries
// x [outer, T, heads, d] -> probs [outer*heads, T, L, 2^K]; rows = outer*heads*T (heads = 1: plain rows)
// x1, probs1: null, or a second tensor of the same shape, in the same launch where the geometry's kernel takes two
cudaError_t bucket_probs(const void* x, const void* x1, const float* planes, void* probs, void* probs1, int64_t rows,
                         int64_t T, int heads, int d, int L, int K, int dtype_x, int dtype_probs, cudaStream_t stream, bool exact = false);

// dx of the same (bucket_probs_bwd.cu): dprobs [outer*heads, T, L, 2^K] and x, dx [outer, T, heads, d], one type
bool bucket_probs_bwd_supported(int d, int L, int K, int dtype);
cudaError_t bucket_probs_bwd(const void* x, const void* x1, const float* planes, const void* dprobs, const void* dprobs1,
                             void* dx, void* dx1, int64_t rows, int64_t T, int heads, int d, int L, int K, int dtype,
                             cudaStream_t stream);

// ---- incremental step (decode.cu) -------------------------------------------------------------
// a few new tokens per stream (dm.T <= decode_max_tokens()) against a running state; state_in may be
// null (zeros) or equal state_out (in place)
int decode_max_tokens();
cudaError_t decode_step_launch(const void* pq, const void* pk, const void* v, void* out, const float* state_in,
                               float* state_out, const Dims& dm, int dtype, cudaStream_t stream);

// the same from K, V, Q [N/heads, T, heads, d] and the hyperplanes (decode_qkv.cu): d = 64, L = 4, K = 4 and d = 128,
// L = 8, K = 6
bool decode_qkv_supported(int64_t N, int64_t T, int d, int L, int K, int dtype);
cudaError_t decode_step_qkv_launch(const void* k, const void* v, const void* q, const float* planes, void* out,
                                   const float* state_in, float* state_out, int64_t N, int T, int heads, int d,
                                   int dtype, float eps, cudaStream_t stream);

// ---- tcgen05 tensor-core causal path (causal_tc.cu) ------------------------------------------
bool tensor_supported(const Dims& dm, int dtype);
int tensor_chunk_tokens();
int tensor_default_tile_tokens(const Dims& dm, int sm_count);
int tensor_bf16_tile_tokens(const Dims& dm, int sm_count);   // bf16 without a state to return: at least as long
size_t tensor_workspace_bytes(const Dims& dm, int dtype, int tile_tokens);
// the single-pass form of the fp32 forward (one persistent kernel): its tile length and its workspace
int tensor_single_pass_tile_tokens(const Dims& dm, int sm_count);
size_t tensor_single_pass_workspace_bytes(const Dims& dm, int tile_tokens);
// single_pass: the fp32 forward as one persistent kernel (needs phases == kPhaseAll and its larger workspace)
cudaError_t causal_fwd_tensor(const void* pq, const void* pk, const void* v, void* out,
                              const float* carry_in, float* state_out, void* ws, bool single_pass, const Dims& dm,
                              int dtype, int tile_tokens, cudaStream_t stream, int* status,
                              int phases = kPhaseAll, bool global_norm = false, long long wait_cycles = 0,
                              int withhold_chunk = -1);

// out_t = sum_{j <= t} (q_t . k_j) v_j + q_t . carry (reverse: j >= t, carry = state of the tokens after the call)
// on fp32 [N, T, 64] tensors with the three launches of the fp32 tensor forward, no normalisation; hq, hk, hv, ho > 1:
// that tensor is laid out [N / h, T, h, 64]
// The causal forward from Q, K, V and the hyperplanes [16][64] on the fp32 tensor kernels (d_k = 64, L = 4, R = 16);
// Q, K, V, out in the layout [N/heads, T, heads, 64]; workspace as for the three-launch form.
bool tensor_qkv_supported(const Dims& dm, int dtype, int L, int R);
cudaError_t causal_fwd_qkv_tensor(const void* q, const void* k, const void* v, const float* planes, void* out,
                                  const float* carry_in, float* state_out, void* ws, const Dims& dm, int tile_tokens,
                                  cudaStream_t stream, int* status, int phases, bool global_norm);
// Epilogue of the first backward pass, run by the forward-direction plain product X = raw(dO, V, pK) where it stores
// its result: with A_t = ablock[block of t] + achunk[chunk of t] + the running sum of pK inside the chunk (the V
// operand of that pass; taken with the triangular product the forward uses for its running sum), inv = 1/(A_t + eps):
//     out <- dPQ = X inv,   w_out <- W = pq_true inv,   g_out <- g = -dPQ W
struct BwdX {
    const float* pq_true;   // [N, T, 64] the query probabilities
    const float* ablock;    // [N, nblk, 64]  sums of pK over the tokens before each block (carry included)
    const float* achunk;    // [N, nchunk, 64] sums of pK from the start of the block to the start of each chunk
    float* w_out;           // [N, T, 64]
    float* g_out;           // [N, T, 64]
    int64_t nblk, nchunk;
    int block_tokens;       // tokens per block (a multiple of the 64-token chunk)
    float eps;
};
cudaError_t causal_raw_tensor(const void* q, const void* k, const void* v, void* out, const float* carry_in,
                              float* state_out, void* ws, const Dims& dm, int tile_tokens, bool reverse,
                              cudaStream_t stream, int* status, int phases = kPhaseAll, const BwdX* bwdx = nullptr,
                              int hq = 1, int hk = 1, int hv = 1, int ho = 1);

// ---- causal backward on the tensor kernels (causal_bwd_tc.cu): fp32, S = 64, d_k = 64 ----------
bool causal_bwd_tensor_supported(const Dims& dm, int dtype);
int causal_bwd_tensor_tile_tokens(const Dims& dm, int sm_count);
size_t causal_bwd_tensor_workspace_bytes(const Dims& dm, int tile_tokens);
cudaError_t causal_bwd_tensor(const void* pq, const void* pk, const void* v, const void* dout, const float* carry_in,
                              const float* d_state, void* dpq, void* dpk, void* dv, float* d_carry, void* ws,
                              const Dims& dm, int tile_tokens, cudaStream_t stream, int* status);

// bf16, S = 64, 128, 256 or 512, d_k 64 or 128 (causal_bwd_bf16_tc.cu); v, dout, dv with dm.H heads
bool causal_bwd_bf16_supported(const Dims& dm);
int causal_bwd_bf16_tile_tokens(const Dims& dm, int sm_count);
size_t causal_bwd_bf16_workspace_bytes(const Dims& dm, int tile_tokens);
cudaError_t causal_bwd_bf16(const void* pq, const void* pk, const void* v, const void* dout, const float* carry_in,
                            const float* d_state, void* dpq, void* dpk, void* dv, float* d_carry, void* ws,
                            const Dims& dm, int tile_tokens, cudaStream_t stream, int* status);

// bf16 tensor path (causal_tc_bf16.cu): S a multiple of 64 (1, 2, 4 or 8 bucket groups), d_k 64 or 128
bool tensor_bf16_supported(const Dims& dm);
// ... with V / out in the layout [N/H, T, H, D] also for one bucket group (race_b200_causal_fwd_heads)
bool tensor_bf16_heads_supported(const Dims& dm);
cudaError_t causal_fwd_tensor_bf16(const void* pq, const void* pk, const void* v, void* out,
                                   const float* carry_in, float* state_out, void* ws, const Dims& dm,
                                   int tile_tokens, cudaStream_t stream, int* status, int phases,
                                   bool global_norm = false);

}  // namespace race
