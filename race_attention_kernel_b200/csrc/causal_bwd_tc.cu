// Causal backward on the tcgen05 kernels (fp32, S = 64, d_k = 64): gradients of
//     out_t = sum_s pQ_t[s] B_t[s,:] / (A_t[s] + eps),   A_t, B_t inclusive prefixes of pK and pK (x) V
// (src/race_baseline.py:45-51; the reference has no causal backward, its design note only outlines one for
// the other estimator, docs/causal_v2_design.md:689-741).  With inv_t = 1/(A_t + eps), W_t = pQ_t inv_t:
//     X_t   = B_t dO_t                         dPQ_t = X_t inv_t          g_t = -X_t W_t inv_t
//     dV_j  = sum_{t >= j} (pK_j . W_t) dO_t
//     dPK_j = sum_{t >= j} g_t + sum_{t >= j} (V_j . dO_t) W_t
// Each sum over tokens with an inner product in it is a plain causal (or anti-causal) product
//     raw(q, k, v)_t = sum_{j <= t} (q_t . k_j) v_j          (reverse: j >= t)
// which is what the forward's tensor kernels compute when they skip the normalisation: same TMA / TMEM /
// tcgen05 pipeline, same bf16 hi/lo limbs, the tile totals / scan / output launches with other tensors in the
// roles of pQ, pK, V.  So the backward is three such passes and a few streaming kernels:
//     1. block sums of pK (with the running sum at every 64-token chunk start) and their scan
//     2. X  = raw(dO, V, pK)                   state of the pass = B^T, so carry_in enters transposed.  X is not
//        stored: the pass takes A_t = block prefix + chunk prefix + running sum inside the chunk (one more
//        triangular product over its V operand, which is pK) and writes dPQ = X inv, W = pQ inv and g = -dPQ W
//        from its epilogue; then the block sums of g
//     3. dV = raw_reverse(pK, W, dO)           state = sum W^T dO: its carry is the gradient of the final B, its
//                                              total the gradient of the carried-in B
//     4. P  = raw_reverse(V, dO, W)            state = the transpose of pass 3's
//     5. reverse scan of the chunk sums of g (carry: gradient of the final A), then dPK = P + running suffix sum
// V, dO and dV may be in the layout [N / heads, T, heads, 64] (dm.H > 1).
// P is written into the dPK buffer (same shape and type), so the scratch memory is W and g ([N, T, 64] fp32 each)
// plus the block / chunk sums and the tile states of the passes.
#include <algorithm>

#include "common.cuh"
#include "launch.h"

namespace race {
namespace {

constexpr int S = 64, D = 64;
constexpr int kSF = S * (D + 1);
constexpr int kBlk = 512;          // tokens per block of the streaming kernels
constexpr int kPwThreads = 256;    // one CTA per block

inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// sums[n][b][c] = sum over the tokens of block b of x[n][t][c]; kChunks: also chunk[n][j][c] = the sum of x over the
// tokens of chunk j's block that precede chunk j (64-token chunks; a block is kBlk / 64 of them).
// Bound by the read of x.  A CTA per block, 16-byte loads: 16 threads per row, 16 rows at a time, eight loads of a thread
// in flight, partial sums added through shared memory.  (One thread per block and column read 4 bytes at a time along
// a chain of 512 tokens: 32 streams of 16384 tokens, 134 MB, took 39 us.)
template <bool kChunks>
__global__ void __launch_bounds__(kPwThreads)
bwd_block_sums(const float* x, float* __restrict__ sums, float* __restrict__ chunk, int64_t T, int64_t nblk,
               int64_t nchunk) {
    constexpr int kCh = kBlk / 64, kSums = kChunks ? kCh : 1, kWarps = kPwThreads / 32;
    __shared__ __align__(16) float red[kWarps][kSums][64];
    __shared__ float tot[kSums][64];
    chain_release();
    chain_wait();
    const int64_t gb = blockIdx.x, n = gb / nblk, b = gb - n * nblk;
    const int64_t t0 = b * kBlk;
    const int len = (int)min(T - t0, (int64_t)kBlk);
    const int tid = threadIdx.x, c4 = tid & 15, slot = tid >> 4;
    const float4* p = reinterpret_cast<const float4*>(x + (n * T + t0) * 64) + c4;
    float4 acc[kSums];
#pragma unroll
    for (int j = 0; j < kSums; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kCh; j += 2) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int t = 64 * j + 16 * u + slot;
            v[u] = t < len ? ld_chain(p + t * 16) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            float4& s = acc[kChunks ? j + u / 4 : 0];
            s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w;
        }
    }
#pragma unroll
    for (int j = 0; j < kSums; ++j) {
        acc[j].x += __shfl_xor_sync(0xffffffffu, acc[j].x, 16);
        acc[j].y += __shfl_xor_sync(0xffffffffu, acc[j].y, 16);
        acc[j].z += __shfl_xor_sync(0xffffffffu, acc[j].z, 16);
        acc[j].w += __shfl_xor_sync(0xffffffffu, acc[j].w, 16);
        if ((tid & 31) < 16) *reinterpret_cast<float4*>(&red[tid >> 5][j][4 * c4]) = acc[j];
    }
    __syncthreads();
    for (int i = tid; i < kSums * 64; i += kPwThreads) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) s += red[w][i >> 6][i & 63];
        tot[i >> 6][i & 63] = s;
    }
    __syncthreads();
    if (tid < 64) {
        float run = 0.f;
#pragma unroll
        for (int j = 0; j < kSums; ++j) {
            if (kChunks && 64 * j < len) chunk[(n * nchunk + t0 / 64 + j) * 64 + tid] = run;
            run += tot[j][tid];
        }
        sums[gb * 64 + tid] = run;
    }
}

// in-place exclusive scan over the blocks of a stream (reverse: suffix sums, last block first); carry is the A part
// ([64] floats at offset S*D) of a packed state per stream or null; total (nullable) receives carry + everything
__global__ void __launch_bounds__(64)
bwd_block_scan(float* __restrict__ sums, const float* carry_state, float* __restrict__ total_state,
               int64_t nblk, int reverse) {
    chain_release();
    chain_wait();
    const int c = threadIdx.x;
    const int64_t n = blockIdx.x;
    float run = carry_state ? carry_state[n * kSF + S * D + c] : 0.f;
    float* p = sums + n * nblk * 64 + c;
    auto at = [&](int64_t b) { return (reverse ? nblk - 1 - b : b) * 64; };
    int64_t b = 0;
    for (; b + 16 <= nblk; b += 16) {
        float v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = p[at(b + u)];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            p[at(b + u)] = run;
            run += v[u];
        }
    }
    for (; b < nblk; ++b) {
        const float v = p[at(b)];
        p[at(b)] = run;
        run += v;
    }
    if (total_state) total_state[n * kSF + S * D + c] = run;
}

// reverse streaming kernel: dPK_j = P_j + suffix[block] + sum_{t >= j, t in block} g_t (P in pdpk on entry).
// Bound by two reads and a write of [N, T, 64].  A CTA per block walks it from its end in pieces of 128 tokens: 16 threads
// (4 columns each) per token, eight consecutive tokens per thread, so that sixteen 16-byte loads of a thread are in
// flight; the sums of the threads behind it come through shared memory.  (One thread per block and column, 4 bytes and
// four tokens at a time: 32 streams of 16384 tokens, 403 MB, took 103 us.)
__global__ void __launch_bounds__(kPwThreads)
bwd_pointwise_rev(const float* g, float* __restrict__ pdpk, const float* gsuffix, int64_t T,
                  int64_t nblk) {
    constexpr int kOwn = 8, kSlots = kPwThreads / 16, kPiece = kOwn * kSlots;
    __shared__ float4 part[2][kSlots][16];
    chain_release();
    chain_wait();
    const int64_t gb = blockIdx.x, n = gb / nblk, b = gb - n * nblk;
    const int64_t t0 = b * kBlk;
    const int len = (int)min(T - t0, (int64_t)kBlk);
    const int c4 = threadIdx.x & 15, slot = threadIdx.x >> 4;
    const int64_t row0 = (n * T + t0) * 16 + c4;
    const float4* gp = reinterpret_cast<const float4*>(g) + row0;
    float4* pp = reinterpret_cast<float4*>(pdpk) + row0;
    auto add = [](float4& a, const float4& x) { a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w; };
    float4 carry = reinterpret_cast<const float4*>(gsuffix)[gb * 16 + c4];
    for (int s = (len - 1) / kPiece; s >= 0; --s) {
        const int t = s * kPiece + slot * kOwn;
        float4 gv[kOwn], pv[kOwn];
#pragma unroll
        for (int u = 0; u < kOwn; ++u) {
            const bool live = t + u < len;
            gv[u] = live ? ld_chain<kLdOnce>(gp + (t + u) * 16) : make_float4(0.f, 0.f, 0.f, 0.f);
            pv[u] = live ? pp[(t + u) * 16] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float4 own = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = kOwn - 1; u >= 0; --u) add(own, gv[u]);
        part[s & 1][slot][c4] = own;
        __syncthreads();   // (the buffer of the piece before last was read before everyone came here)
        float4 run = carry;
#pragma unroll
        for (int k = kSlots - 1; k >= 0; --k) {
            const float4 x = part[s & 1][k][c4];
            if (k > slot) add(run, x);
            add(carry, x);
        }
#pragma unroll
        for (int u = kOwn - 1; u >= 0; --u) {
            add(run, gv[u]);
            add(pv[u], run);
            if (t + u < len) pp[(t + u) * 16] = pv[u];
        }
    }
}

// dst[n] = the state src[n] with its B part ([64][64]) transposed and its A part zeroed
__global__ void __launch_bounds__(256)
bwd_transpose_state(const float* src, float* __restrict__ dst) {
    __shared__ float tile[64][65];
    chain_release();
    chain_wait();
    const int64_t n = blockIdx.x;
    const float* s = src + n * kSF;
    float* d = dst + n * kSF;
    for (int i = threadIdx.x; i < S * D; i += 256) tile[i >> 6][i & 63] = s[i];
    __syncthreads();
    for (int i = threadIdx.x; i < S * D; i += 256) d[i] = tile[i & 63][i >> 6];
    if (threadIdx.x < S) d[S * D + threadIdx.x] = 0.f;
}

struct BwdLayout {
    size_t tiles, tiles2, w, g, asum, gsum, achunk, st0, total;
};
BwdLayout bwd_layout(const Dims& dm, int tile_tokens) {
    const int64_t tiles = (dm.T + tile_tokens - 1) / tile_tokens;
    const int64_t nblk = (dm.T + kBlk - 1) / kBlk;
    const size_t tok = align256((size_t)dm.N * dm.T * 64 * sizeof(float));
    const size_t blk = align256((size_t)dm.N * nblk * 64 * sizeof(float));
    const size_t st = align256((size_t)dm.N * kSF * sizeof(float));
    BwdLayout l;
    const size_t tl = align256((size_t)dm.N * tiles * kSF * sizeof(float));
    l.tiles = 0;
    l.tiles2 = tl;
    l.w = 2 * tl;
    l.g = l.w + tok;
    l.asum = l.g + tok;
    l.gsum = l.asum + blk;
    l.achunk = l.gsum + blk;
    l.st0 = l.achunk + align256((size_t)dm.N * ((dm.T + 63) / 64) * 64 * sizeof(float));
    l.total = l.st0 + st;
    return l;
}

#define RACE_CK(expr)                                  \
    do {                                               \
        cudaError_t e_ = (expr);                       \
        if (e_ != cudaSuccess) return e_;              \
    } while (0)

}  // namespace

bool causal_bwd_tensor_supported(const Dims& dm, int dtype) {
    return dtype == RACE_DTYPE_F32 && tensor_supported(dm, dtype);
}

int causal_bwd_tensor_tile_tokens(const Dims& dm, int sm_count) {
    return tensor_default_tile_tokens(dm, sm_count);
}

size_t causal_bwd_tensor_workspace_bytes(const Dims& dm, int tile_tokens) {
    if (dm.N == 0 || dm.T == 0) return 0;
    return bwd_layout(dm, tile_tokens).total;
}

cudaError_t causal_bwd_tensor(const void* pq, const void* pk, const void* v, const void* dout, const float* carry_in,
                              const float* d_state, void* dpq, void* dpk, void* dv, float* d_carry, void* ws,
                              const Dims& dm, int tile_tokens, cudaStream_t stream, int* status) {
    const BwdLayout l = bwd_layout(dm, tile_tokens);
    char* base = (char*)ws;
    float* ws_tiles = (float*)(base + l.tiles);
    float* w = (float*)(base + l.w);
    float* g = (float*)(base + l.g);
    float* asum = (float*)(base + l.asum);
    float* gsum = (float*)(base + l.gsum);
    float* ws_tiles2 = (float*)(base + l.tiles2);
    float* st_t = (float*)(base + l.st0);      // a transposed carry
    const int64_t tiles = (dm.T + tile_tokens - 1) / tile_tokens;
    const int64_t nblk = (dm.T + kBlk - 1) / kBlk;
    const unsigned pw_grid = (unsigned)(dm.N * nblk);

    // 1. sums of pK: per block (then scanned, carry included) and inside the block up to every chunk start
    float* achunk = (float*)(base + l.achunk);
    const int64_t nchunk = (dm.T + 63) / 64;
    RACE_CK(launch_chain(chain_launches(dm), bwd_block_sums<true>, pw_grid, kPwThreads, 0, stream, (const float*)pk, asum, achunk, dm.T, nblk,
                         nchunk));
    RACE_CK(launch_chain(chain_launches(dm), bwd_block_scan, (unsigned)dm.N, 64, 0, stream, asum, carry_in, nullptr, nblk, 0));
    // 2. X = raw(dO, V, pK), the state of the pass is B^T; its epilogue writes dPQ, W and g.  Then the block sums of g.
    if (carry_in) RACE_CK(launch_chain(chain_launches(dm), bwd_transpose_state, (unsigned)dm.N, 256, 0, stream, carry_in, st_t));
    BwdX bx;
    bx.pq_true = (const float*)pq;
    bx.ablock = asum;
    bx.achunk = achunk;
    bx.w_out = w;
    bx.g_out = g;
    bx.nblk = nblk;
    bx.nchunk = nchunk;
    bx.block_tokens = kBlk;
    bx.eps = dm.eps;
    RACE_CK(causal_raw_tensor(dout, v, pk, dpq, carry_in ? st_t : nullptr, nullptr, ws_tiles, dm, tile_tokens,
                              /*reverse=*/false, stream, status, kPhaseAll, &bx, dm.H, dm.H, 1, 1));
    RACE_CK(launch_chain(chain_launches(dm), bwd_block_sums<false>, pw_grid, kPwThreads, 0, stream, (const float*)g, gsum, nullptr, dm.T, nblk, nchunk));
    // 3. dV = raw_reverse(pK, W, dO); state sum W^T dO: carry = gradient of the final B, total = gradient of carry_in's B.
    //    Pass 4 below has the roles of W and dO swapped, so its tile totals are the transposes of this pass's:
    //    the totals launch runs once and the second tile buffer gets the transposed states.
    RACE_CK(causal_raw_tensor(nullptr, w, dout, nullptr, nullptr, nullptr, ws_tiles, dm, tile_tokens, true, stream, status,
                              d_carry ? kPhaseTotals : kPhaseTotals | kPhasePrefixOnly, nullptr, 1, 1, dm.H, 1));
    RACE_CK(launch_chain(chain_launches(dm), bwd_transpose_state, (unsigned)(dm.N * tiles), 256, 0, stream, (const float*)ws_tiles, ws_tiles2));
    RACE_CK(causal_raw_tensor(pk, w, dout, dv, d_state, d_carry, ws_tiles, dm, tile_tokens,
                              /*reverse=*/true, stream, status, kPhaseOutput, nullptr, 1, 1, dm.H, dm.H));
    // 4. P = raw_reverse(V, dO, W) into the dPK buffer; state = the transpose of pass 3's
    if (d_state) RACE_CK(launch_chain(chain_launches(dm), bwd_transpose_state, (unsigned)dm.N, 256, 0, stream, d_state, st_t));
    RACE_CK(causal_raw_tensor(v, dout, w, dpk, d_state ? st_t : nullptr, nullptr, ws_tiles2, dm, tile_tokens,
                              /*reverse=*/true, stream, status, kPhaseOutput, nullptr, dm.H, dm.H, 1, 1));
    // 5. dPK = P + suffix sums of g (carry: gradient of the final A; total: gradient of carry_in's A, which
    //    overwrites the A part that pass 3 left in d_carry)
    RACE_CK(launch_chain(chain_launches(dm), bwd_block_scan, (unsigned)dm.N, 64, 0, stream, gsum, d_state, d_carry, nblk, 1));
    return launch_chain(chain_launches(dm), bwd_pointwise_rev, pw_grid, kPwThreads, 0, stream, (const float*)g, (float*)dpk, (const float*)gsum,
                        dm.T, nblk);
}

}  // namespace race
