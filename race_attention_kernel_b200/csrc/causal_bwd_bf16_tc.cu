// Causal backward for bf16 tensors on tcgen05 (S = 64 or a multiple of 128 up to 512, d_k in {64, 128}): gradients of
//     out_t = sum_s pQ_t[s] B_t[s,:] / (A_t[s] + eps)          (src/race_baseline.py:45-51; no causal backward there)
// with inv_t = 1/(A_t + eps), W_t = pQ_t inv_t, and the sums of causal_bwd_simt.cu:
//     X_t = B_t dO_t      dPQ_t = X_t inv_t      g_t = -dPQ_t W_t
//     dPK_j = sum_{t >= j} g_t + sum_{t >= j} (V_j . dO_t) W_t        dV_j = sum_{t >= j} (pK_j . W_t) dO_t
// Launches over state tiles of a multiple of 128 tokens:
//     totals of (pK, V) and their exclusive scan               the forward's kernels: state before every tile
//     bwd_prefix_rows    tile walked forwards in chunks of 128 tokens, B on chip:
//                          X = dO B^T + tril(dO V^T) pK;  dPQ, the suffix sums of g inside the chunk (GS), the running
//                          A at every chunk start;  B += pK^T V;  tile totals of (W (x) dO, g)
//     reverse scan of those totals
//     bwd_suffix_rows    tile walked backwards, SB = sum W (x) dO of everything later on chip:
//                          dPK = V SB^T + triu(V dO^T) W + GS + later g;  dV = pK SB + triu(pK W^T) dO;  SB += W^T dO
// Tables are independent, so a CTA owns SB (64 or 128) buckets; only dV sums over buckets: with several bucket blocks
// they leave fp32 shares which bwd_dv_sum adds in block order.
//
// Precision: inputs are exact one-limb operands, accumulators are fp32, everything computed (W, the masked products, the
// states, g) is split into hi + lo bf16 limbs (split2t: 2^-16 of a value); in the one product of two computed factors,
// triu(V dO^T) . W, the product of the low limbs (up to 2^-14 of a term) is left out.  Enough for the results, which are
// rounded to bf16 (2^-9): dK, dV and dQ of a training step are as far from the 64-bit ones as with fp32 products on the CUDA
// cores (4.6e-3 to 5.6e-3; ratio of the errors 0.9999 +- 0.0007 for dK and 1.0012 +- 0.0005 for dQ over 30 draws at S = 64).
// It is not enough for the fp32 gradient of a carried-in state, which causal_bwd_simt.cu forms (but for heads > 1).
//
// Why this shape of kernel.  On CUDA cores the two passes took 1.31 of the 1.73 ms of a training step at S = 64 (96
// streams of 4096 tokens) and 9.05 of 9.79 ms at S = 512, d_k = 128 (32 streams of 4096).  Chunks of 128 tokens and blocks of 128 buckets make every product 128 x 128 x 128 (full M, N of
// the tensor core; M = 64 runs at half rate), an accumulator row is a thread's token, and TMA writes the operand tiles
// as the tensor core reads them (128-byte swizzle, both majors), so the only data the warps move are the computed
// limbs.  Shared memory (224 KB at 128 x 128) holds one chunk: a chunk's chain of products is serial, and what bounds
// the kernels is that chain; the products themselves take about half of it.
#include <cudaTypedefs.h>

#include <algorithm>

#include "common.cuh"
#include "launch.h"
#include "tc_rows.cuh"

namespace race {
namespace {

constexpr int C = 128;              // tokens per chunk
// 8 warps on the bucket side (W, dPQ / dPK), 8 on the token x token products (masks, sums of g, dV), 4 on the state, and
// one group with the TMA and MMA warps
constexpr int kThreads = 24 * 32;
constexpr int kStateWarp = 16, kTmaWarp = 20, kMmaWarp = 21;
constexpr int kRegsP = 104, kRegsG = 72, kRegsS = 64, kRegsM = 64;   // 8, 8, 4, 4 warps: exactly the 768 x 80 of the launch
constexpr uint32_t tG = 256;        // tensor-memory columns of the token x token products

__device__ __forceinline__ float2 unpack2(uint32_t u) {
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

// Shared memory: per stage dO | V | pK | pQ; the operand tiles of the state; kSuffix has a slot of its own for W's low
// limb (the prefix pass puts it where V was, which no product reads by then).
template <int SB, int D, bool kSuffix>
struct Lay {
    static constexpr int kDO = C * D * 2, kP = C * SB * 2;
    static constexpr int kV = kSuffix ? kDO : (kDO > kP ? kDO : kP);
    static constexpr int kStage = kDO + kV + 2 * kP;
    static constexpr int oDO = 0, oV = kDO, oK = kDO + kV, oQ = oK + kP;     // inside a stage
    static constexpr int kStages = (SB == 64 && D == 64) ? 2 : 1;
    static constexpr int oWlo = kStages * kStage;
    static constexpr int oB = oWlo + (kSuffix ? kP : 0);                     // [hi | lo][SB rows][D]
    static constexpr int kB = SB * D * 2;
    static constexpr int oCar = oB + 2 * kB;                                 // [2][SB] fp32 running A / later g
    static constexpr int oTot = oCar + 2 * SB * 4;                           // [SB] prefix: totals of g; suffix: A before the chunk
    static constexpr int oBars = oTot + SB * 4;
    static constexpr int kNumBars = 24;
    static constexpr int oMisc = oBars + kNumBars * 8;
    static constexpr int kSmem = oMisc + 16 + 1024;
    static_assert(kSmem <= 227 * 1024, "shared memory of the backward");
};
// A wait on a barrier never lags it by two phases: every party that waits on one also has to arrive somewhere before the
// next phase of that barrier can complete.
enum Bar {
    bFull = 0,      // [2] dO, V, pK of the stage have landed
    bFullQ = 2,     // [2] pQ
    bTri = 4,       // triangular matrix of the chunk in the G columns; prefix: the sums of g of the chunk before are read (8)
    bA = 5,         // running sums of pK inside the chunk
    bG = 6,         // first token x token product
    bSt = 7,        // state updated with the chunk
    bXb = 8,        // operand tiles of the state no longer read
    bBt = 9,        // operand tiles of the state before the chunk written, accumulator read (4)
    bW = 10,        // W limbs written, running sums read (8)
    bGm = 11,       // masked first product written (8)
    bX = 12,        // bucket-side result (X / P) complete
    bXg = 13,       // prefix: X read, g limbs written, upper triangle written (16)
    bH = 14,        // suffix: second token x token product.  prefix: totals updated, W no longer read
    bHm = 15,       // suffix: masked second product written (8)
    bPf = 16,       // suffix: P read (8)
    bVf = 17,       // suffix: dV read (8)
    bEnd = 18,      // every product of the chunk has run
    bEmpty = 19,    // [2] ... of the chunk in the stage
    bDrain = 21
};

struct Args {
    const float* ws;         // state tiles: exclusive prefixes (suffixes)
    float* ws_out;           // prefix: totals of (W (x) dO, g)
    __nv_bfloat16* dp;       // dPQ / dPK [N, T, S]
    float* gs;               // [N, T, S] sums of g from the token to the end of its chunk
    float* achunk;           // [N, chunks, S] running A before each chunk
    void* dv;                // bf16 [N/H, T, H, D], or with several bucket blocks their fp32 shares [block][N, T, D]
    int64_t T;
    int S, heads, tile_tokens;
    float eps;
    bool sectors;            // dp and a bf16 dv begin on a 32-byte boundary
    int* status;
};

struct Setup {
    Ctx cx;
    uint32_t tmem;
    int64_t tile, tiles, n, t_begin, t_end;
    int g0, block, nch;      // first bucket of the CTA, its block, chunks of the tile
};

template <typename Ly, int SB>
__device__ __forceinline__ Setup begin(const Args& a) {
    extern __shared__ uint8_t smem_raw[];
    Setup s;
    s.cx.sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    s.cx.sm_u32 = smem_u32(s.cx.sm);
    s.cx.bars = Ly::oBars;
    s.cx.abort_flag = reinterpret_cast<volatile int*>(s.cx.sm + Ly::oMisc + 4);
    s.cx.status = a.status;
    const int blocks = a.S / SB;
    s.block = (int)(blockIdx.x % (unsigned)blocks);
    s.g0 = s.block * SB;
    s.tiles = gridDim.x / blocks;
    s.tile = blockIdx.x / blocks;
    s.n = blockIdx.y;
    s.t_begin = s.tile * a.tile_tokens;
    s.t_end = min(a.T, s.t_begin + (int64_t)a.tile_tokens);
    s.nch = (int)((s.t_end - s.t_begin + C - 1) / C);
    chain_release();
    if (threadIdx.x == 0) {
        *s.cx.abort_flag = 0;
        for (int i = 0; i < Ly::kNumBars; ++i) {
            constexpr uint32_t kEight = (1u << bTri) | (1u << bW) | (1u << bGm) | (1u << bHm) | (1u << bPf) | (1u << bVf);
            mbar_init(s.cx.bar(i), (kEight >> i) & 1u ? 8u : i == bXg ? 16u : i == bBt ? 4u : 1u);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if ((threadIdx.x >> 5) == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(s.cx.sm_u32 + Ly::oMisc), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    s.tmem = *reinterpret_cast<volatile uint32_t*>(s.cx.sm + Ly::oMisc);
    chain_wait();
    return s;
}
__device__ __forceinline__ void finish(uint32_t tmem) {
    tc_fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}
// the lanes of a warp have written operands or read accumulators: one arrival
__device__ __forceinline__ void arrive_warp(const Ctx& cx, int bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(cx.bar(bar));
}

// TMA producer (one lane): dO, V, pK, pQ of the c-th chunk that is processed
template <typename Ly>
__device__ __forceinline__ void produce(const Setup& s, const Args& a, const CUtensorMap* map_do, const CUtensorMap* map_v,
                                        const CUtensorMap* map_k, const CUtensorMap* map_q, bool reverse) {
    const Ctx& cx = s.cx;
    const int h = (int)(s.n % a.heads), mb = (int)(s.n / a.heads);
    int issued = 0;
    for (int c = 0; c < s.nch; ++c) {
        const int st = c % Ly::kStages;
        if (c >= Ly::kStages && !wait_bar(cx, bEmpty + st, (uint32_t)((c / Ly::kStages - 1) & 1), 301)) break;
        const uint32_t dst = cx.sm_u32 + st * Ly::kStage;
        const int tok = (int)(s.t_begin + (int64_t)(reverse ? s.nch - 1 - c : c) * C);
        mbar_arrive_expect_tx(cx.bar(bFull + st), 2 * Ly::kDO + Ly::kP);
        tma_load_4d(dst + Ly::oK, map_k, cx.bar(bFull + st), 0, tok, s.g0 / 64, (int)s.n);
        tma_load_5d(dst + Ly::oDO, map_do, cx.bar(bFull + st), 0, tok, 0, h, mb);
        tma_load_5d(dst + Ly::oV, map_v, cx.bar(bFull + st), 0, tok, 0, h, mb);
        mbar_arrive_expect_tx(cx.bar(bFullQ + st), Ly::kP);
        tma_load_4d(dst + Ly::oQ, map_q, cx.bar(bFullQ + st), 0, tok, s.g0 / 64, (int)s.n);
        issued = c + 1;
    }
    if (*cx.abort_flag)   // copies in flight land before the CTA may exit
        for (int c = max(0, issued - Ly::kStages); c < issued; ++c)
            for (int b = 0; b < 2; ++b) {
                const long long t0 = clock64();
                while (!mbar_try_wait(cx.bar((b ? bFullQ : bFull) + c % Ly::kStages), (uint32_t)((c / Ly::kStages) & 1)) &&
                       clock64() - t0 < (1ll << 24)) {}
            }
}

// State accumulator <-> operand tiles: a thread owns one row (bucket) of D values.  With 64 rows the accumulator's row r
// is on lane (r % 16) + 32 (r / 16), so half of a warp's lanes own one.
template <int SB>
struct StateRow {
    int row;
    bool live;
    __device__ __forceinline__ StateRow(int w, int lane)
        : row(SB == 128 ? 32 * w + lane : 16 * w + (lane & 15)), live(SB == 128 || lane < 16) {}
};
template <int SB>
__device__ __forceinline__ void store_state_limbs(uint8_t* hi_tile, int lo_off, const StateRow<SB>& r, int col,
                                                  const float (&v)[16]) {
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split2t(v[2 * i], v[2 * i + 1], hi[i], lo[i]);
    if (r.live) {
        sw_store_row<SB, 8>(hi_tile, r.row, col, hi);
        sw_store_row<SB, 8>(hi_tile + lo_off, r.row, col, lo);
    }
}

// Carry into the tile: B -> accumulator and operand tiles (state warps)
template <int SB, int D, typename Ly>
__device__ __forceinline__ void load_state(const Setup& s, const Args& a, int w, int lane) {
    const StateRow<SB> r(w, lane);
    const float* src = a.ws + (s.n * s.tiles + s.tile) * (int64_t)(a.S * (D + 1)) + (int64_t)(s.g0 + r.row) * D;
#pragma unroll 1
    for (int cb = 0; cb < D; cb += 16) {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            const float4 x = r.live ? ld_chain(reinterpret_cast<const float4*>(src + cb + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
        }
        tmem_st_words16(((uint32_t)(32 * w) << 16) + s.tmem + cb, reinterpret_cast<const uint32_t(&)[16]>(v));
        store_state_limbs<SB>(s.cx.sm + Ly::oB, Ly::kB, r, cb, v);
    }
    tmem_wait_st();
    fence_proxy_async();
    tc_fence_before();
    arrive_warp(s.cx, bBt);
}
// after every chunk but the last: updated accumulator -> operand tiles
template <int SB, int D, typename Ly>
__device__ __forceinline__ void carry_state(const Setup& s, int w, int lane) {
    StateRow<SB> r(w, lane);
    bool ok = true;
    for (int c = 1; c < s.nch && ok; ++c) {
        asm volatile("" : "+r"(r.row));   // (addresses per chunk, not kept in registers this group does not have)
        RACE_TRACE(2, c, 0);
        if (!(ok = wait_bar_warp(s.cx, bSt, (uint32_t)((c - 1) & 1), 201))) break;
        if (!(ok = wait_bar_warp(s.cx, bXb, (uint32_t)((c - 1) & 1), 202))) break;
        RACE_TRACE(2, c, 1);
        tc_fence_after();
#pragma unroll
        for (int cb = 0; cb < D; cb += 16) {
            float v[16];
            tmem_ld_rows16(((uint32_t)(32 * w) << 16) + s.tmem + cb, v);
            store_state_limbs<SB>(s.cx.sm + Ly::oB, Ly::kB, r, cb, v);
        }
        fence_proxy_async();
        tc_fence_before();
        arrive_warp(s.cx, bBt);
        RACE_TRACE(2, c, 2);
    }
}

// the 64 columns [64 wg, +64) of a token x token product: mask (kUpper: column >= row stays), split, and write the limbs
// over the 32 columns they came from (16 words of hi, 16 of lo).  32-column blocks outside the triangle are only zeroed.
template <bool kUpper>
__device__ __forceinline__ void mask_product(uint32_t tm_lane, int row, int wg) {
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {
        const int col0 = 64 * wg + 32 * hb;
        uint32_t hi[16], lo[16];
        if (kUpper ? col0 + 31 < (row & ~31) : col0 > (row | 31)) {
#pragma unroll
            for (int i = 0; i < 16; ++i) hi[i] = lo[i] = 0u;
        } else {
            float v[32];
            tmem_ld_rows32(tm_lane + tG + col0, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int col = col0 + 2 * i;
                const float x = (kUpper ? col >= row : col <= row) ? v[2 * i] : 0.f;
                const float y = (kUpper ? col + 1 >= row : col + 1 <= row) ? v[2 * i + 1] : 0.f;
                split2t(x, y, hi[i], lo[i]);
            }
        }
        tmem_st_words16(tm_lane + tG + col0, hi);
        tmem_st_words16(tm_lane + tG + col0 + 16, lo);
    }
    tmem_wait_st();
    tc_fence_before();
}
template <bool kUpper>
__device__ __forceinline__ void write_tri(uint32_t tm_lane, int row, int wg) {
    uint32_t tr[32];
    tri_words<kUpper>(row, wg, tr);
    tmem_st_words32(tm_lane + tG + 32 * wg, tr);
    tc_fence_before();
}
// fp32 rows lie in the workspace (256-byte aligned): 32-byte stores.  bf16 rows lie in the caller's tensors, which only
// promise 16 bytes: a sector at a time where they happen to begin on one (sectors), else in two halves (96 streams of 4096
// tokens, S = 64, d_k = 64, a training step: 508 us against 520).
__device__ __forceinline__ void store_row16(float* dst, const float (&v)[16]) {
    st_global_32b(dst, reinterpret_cast<const uint32_t(&)[8]>(v[0]));
    st_global_32b(dst + 8, reinterpret_cast<const uint32_t(&)[8]>(v[8]));
}
__device__ __forceinline__ void store_row16(__nv_bfloat16* dst, const float (&v)[16], bool sectors) {
    uint32_t d[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) d[i] = pack2(v[2 * i], v[2 * i + 1]);
    if (sectors) {
        st_global_32b(dst, d);
    } else {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(d[0], d[1], d[2], d[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(d[4], d[5], d[6], d[7]);
    }
}

// ------------------------------------------------------------------------------------------------
template <int SB, int D>
__global__ void __launch_bounds__(kThreads, 1)
bwd_prefix_rows(const __grid_constant__ CUtensorMap map_do, const __grid_constant__ CUtensorMap map_v,
                const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q, const Args a) {
    using Ly = Lay<SB, D, false>;
    constexpr int HC = SB / 2;                       // bucket columns of a worker group
    constexpr uint32_t tTot = 128, tX = 384;
    const Setup s = begin<Ly, SB>(a);
    const Ctx& cx = s.cx;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* car = reinterpret_cast<float*>(cx.sm + Ly::oCar);
    float* tot = reinterpret_cast<float*>(cx.sm + Ly::oTot);
    const int64_t sf = (int64_t)a.S * (D + 1);
    const int wg = (warp >> 2) & 1, w = warp & 3, row = 32 * w + lane;
    const uint32_t tm_lane = s.tmem + ((uint32_t)(32 * w) << 16);
    const int col0 = HC * wg;                        // first bucket column of this thread inside the block

    if (warp < 8) {
        regs_inc<kRegsP>();
        const float* slice_a = a.ws + (s.n * s.tiles + s.tile) * sf + (int64_t)a.S * D + s.g0;
        if (row < HC) car[col0 + row] = slice_a[col0 + row];
        asm volatile("bar.sync 5, 256;" ::: "memory");
        const int64_t nchunk = (a.T + C - 1) / C;
        bool ok = true;
        for (int c = 0; c < s.nch && ok; ++c) {
            const uint32_t ph = (uint32_t)(c & 1);
            const int st = c % Ly::kStages;
            uint8_t* stage = cx.sm + st * Ly::kStage;
            const int64_t tok = s.t_begin + (int64_t)c * C + row;
            const bool live = tok < s.t_end;
            // ---- running A, W = pQ / (A + eps) -> limbs over pQ and over V ---------------------------------
            // every warp of the group has published / read the running A of the chunk before
            if (c > 0 && !(ok = wait_bar_warp(cx, bXg, ph ^ 1, 101))) break;
            if (row < HC)
                a.achunk[(s.n * nchunk + s.t_begin / C + c) * a.S + s.g0 + col0 + row] = car[(c & 1) * SB + col0 + row];
            if (!(ok = wait_bar_warp(cx, bFullQ + st, (uint32_t)((c / Ly::kStages) & 1), 102))) break;
            RACE_TRACE(wg, c, 0);
            if (!(ok = wait_bar_warp(cx, bA, ph, 103))) break;
            RACE_TRACE(wg, c, 1);
            tc_fence_after();
            float inv[HC];
#pragma unroll
            for (int cb = 0; cb < HC; cb += 16) {
                float v[16];
                tmem_ld_rows16(tm_lane + tX + col0 + cb, v);
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 c4 = *reinterpret_cast<const float4*>(car + (c & 1) * SB + col0 + cb + i);
                    v[i] += c4.x; v[i + 1] += c4.y; v[i + 2] += c4.z; v[i + 3] += c4.w;
                    if (row == C - 1)
                        *reinterpret_cast<float4*>(car + ((c + 1) & 1) * SB + col0 + cb + i) =
                            make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) inv[cb + i] = __fdividef(1.f, v[i] + a.eps);
            }
            if (!(ok = wait_bar_warp(cx, bSt, ph, 104))) break;   // V has been read: its slot takes the low limbs
#pragma unroll
            for (int p = 0; p < HC / 8; ++p) {
                const uint32_t off = sw_piece<C>(row, col0 + 8 * p);
                const uint4 q4 = *reinterpret_cast<const uint4*>(stage + Ly::oQ + off);
                const uint32_t qq[4] = {q4.x, q4.y, q4.z, q4.w};
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 q2 = unpack2(qq[i]);
                    split2t(q2.x * inv[8 * p + 2 * i], q2.y * inv[8 * p + 2 * i + 1], hi[i], lo[i]);
                }
                *reinterpret_cast<uint4*>(stage + Ly::oQ + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(stage + Ly::oV + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            fence_proxy_async();
            tc_fence_before();
            arrive_warp(cx, bW);
            RACE_TRACE(wg, c, 2);
            // ---- X -> dPQ, g = -dPQ W -> limbs over W ----------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bX, ph, 106))) break;
            RACE_TRACE(wg, c, 3);
            tc_fence_after();
            __nv_bfloat16* dst = a.dp + (s.n * a.T + tok) * a.S + s.g0 + col0;
#pragma unroll
            for (int cb = 0; cb < HC; cb += 16) {     // inv <- dPQ
                float v[16];
                tmem_ld_rows16(tm_lane + tX + col0 + cb, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) inv[cb + i] = v[i] *= inv[cb + i];
                if (live) store_row16(dst + cb, v, a.sectors);
            }
            if (!(ok = wait_bar_warp(cx, bH, ph, 107))) break;    // the totals have read W
            RACE_TRACE(wg, c, 4);
#pragma unroll
            for (int p = 0; p < HC / 8; ++p) {
                const uint32_t off = sw_piece<C>(row, col0 + 8 * p);
                const uint4 h4 = *reinterpret_cast<const uint4*>(stage + Ly::oQ + off);
                const uint4 l4 = *reinterpret_cast<const uint4*>(stage + Ly::oV + off);
                const uint32_t hh[4] = {h4.x, h4.y, h4.z, h4.w}, ll[4] = {l4.x, l4.y, l4.z, l4.w};
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 wh = unpack2(hh[i]), wl = unpack2(ll[i]);
                    split2t(-inv[8 * p + 2 * i] * (wh.x + wl.x), -inv[8 * p + 2 * i + 1] * (wh.y + wl.y), hi[i], lo[i]);
                }
                *reinterpret_cast<uint4*>(stage + Ly::oQ + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(stage + Ly::oV + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            fence_proxy_async();
            tc_fence_before();
            arrive_warp(cx, bXg);
            RACE_TRACE(wg, c, 5);
        }
    } else if (warp < kStateWarp) {
        regs_dec<kRegsG>();
        if (row < HC) tot[col0 + row] = 0.f;
        asm volatile("bar.sync 6, 256;" ::: "memory");
        write_tri<false>(tm_lane, row, wg);
        arrive_warp(cx, bTri);
        bool ok = true;
        for (int c = 0; c < s.nch && ok; ++c) {
            const uint32_t ph = (uint32_t)(c & 1);
            const int64_t tok = s.t_begin + (int64_t)c * C + row;
            const bool live = tok < s.t_end;
            // ---- causal mask of dO V^T --------------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bG, ph, 105))) break;
            RACE_TRACE(3, c, 0);
            tc_fence_after();
            mask_product<false>(tm_lane, row, wg);
            arrive_warp(cx, bGm);
            RACE_TRACE(3, c, 1);
            if (!(ok = wait_bar_warp(cx, bX, ph, 106))) break;
            tc_fence_after();
            write_tri<true>(tm_lane, row, wg);
            arrive_warp(cx, bXg);
            // ---- suffix sums of g inside the chunk ------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bEnd, ph, 107))) break;
            RACE_TRACE(3, c, 2);
            tc_fence_after();
            write_tri<false>(tm_lane, row, wg);
            float* gdst = a.gs + (s.n * a.T + tok) * a.S + s.g0 + col0;
#pragma unroll
            for (int cb = 0; cb < HC; cb += 16) {
                float v[16];
                tmem_ld_rows16(tm_lane + tX + col0 + cb, v);
                if (live) store_row16(gdst + cb, v);
                if (row == 0) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        float4* t4 = reinterpret_cast<float4*>(tot + col0 + cb + i);
                        const float4 x = *t4;
                        *t4 = make_float4(x.x + v[i], x.y + v[i + 1], x.z + v[i + 2], x.w + v[i + 3]);
                    }
                }
            }
            tc_fence_before();
            arrive_warp(cx, bTri);
            RACE_TRACE(3, c, 3);
        }
    } else if (warp < kTmaWarp) {
        regs_dec<kRegsS>();
        load_state<SB, D, Ly>(s, a, w, lane);
        carry_state<SB, D, Ly>(s, w, lane);
    } else {
        regs_dec<kRegsM>();
        if (warp == kTmaWarp && lane == 0) produce<Ly>(s, a, &map_do, &map_v, &map_k, &map_q, false);
        if (warp == kMmaWarp) {
            const uint32_t tm0 = __shfl_sync(0xffffffffu, s.tmem, 0), smb0 = __shfl_sync(0xffffffffu, cx.sm_u32, 0);
            constexpr uint32_t iTS = idesc_mn(C, SB), iTT = idesc_mn(C, C), iSD = idesc_mn(SB, D);
            if (elect_one()) {
                bool ok = true;
                for (int c = 0; c < s.nch && ok; ++c) {
                    const uint32_t ph = (uint32_t)(c & 1);
                    const int st = c % Ly::kStages;
                    // opaque per chunk: the descriptors are one addition each; kept across chunks they would be spilled
                    uint32_t tm = tm0, smb = smb0;
                    asm volatile("" : "+r"(tm), "+r"(smb));
                    const uint32_t base = smb + st * Ly::kStage;
                    const uint32_t sDO = base + Ly::oDO, sV = base + Ly::oV, sK = base + Ly::oK, sQ = base + Ly::oQ;
                    if (!(ok = wait_bar(cx, bTri, ph, 401))) break;
                    if (!(ok = wait_bar(cx, bFull + st, (uint32_t)((c / Ly::kStages) & 1), 402))) break;
                    tc_fence_after();
                    mma_sw_ta<true, 8, true, C>(tm + tX, tm + tG, sK, iTS);                      // A_loc = tril . pK
                    mma_commit(cx.bar(bA));
                    mma_sw<true, D / 16, false, C, false, C>(tm + tG, sDO, sV, iTT);             // G = dO . V^T (over tril)
                    mma_commit(cx.bar(bG));
                    if (!(ok = wait_bar(cx, bBt, ph, 403))) break;
                    tc_fence_after();
                    mma_sw<false, 8, true, C, true, C>(tm, sK, sV, iSD);                         // B += pK^T . V
                    mma_commit(cx.bar(bSt));
                    if (!(ok = wait_bar(cx, bW, ph, 404))) break;
                    tc_fence_after();
                    mma_sw<true, D / 16, false, C, false, SB>(tm + tX, sDO, smb + Ly::oB, iTS);  // X = dO . B^T
                    mma_sw<false, D / 16, false, C, false, SB>(tm + tX, sDO, smb + Ly::oB + Ly::kB, iTS);
                    mma_commit(cx.bar(bXb));
                    if (!(ok = wait_bar(cx, bGm, ph, 405))) break;
                    tc_fence_after();
                    mma_sw_ta<false, 8, true, C, true>(tm + tX, tm + tG, sK, iTS);               // X += tril(G) . pK
                    mma_sw_ta<false, 8, true, C, true>(tm + tX, tm + tG + 16, sK, iTS);
                    mma_commit(cx.bar(bX));
                    if (c == 0) mma_sw<true, 8, true, C, true, C>(tm + tTot, sQ, sDO, iSD);      // totals += W^T . dO
                    else mma_sw<false, 8, true, C, true, C>(tm + tTot, sQ, sDO, iSD);
                    mma_sw<false, 8, true, C, true, C>(tm + tTot, sV, sDO, iSD);
                    mma_commit(cx.bar(bH));
                    if (!(ok = wait_bar(cx, bXg, ph, 406))) break;
                    tc_fence_after();
                    mma_sw_ta<true, 8, true, C>(tm + tX, tm + tG, sQ, iTS);                      // GS = triu . g
                    mma_sw_ta<false, 8, true, C>(tm + tX, tm + tG, sV, iTS);
                    mma_commit(cx.bar(bEnd));
                    mma_commit(cx.bar(bEmpty + st));
                }
                mma_commit(cx.bar(bDrain));
                const long long t0 = clock64();
                while (!mbar_try_wait(cx.bar(bDrain), 0) && clock64() - t0 < cx.limit) {}
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // totals of the tile
    float* slice = a.ws_out + (s.n * s.tiles + s.tile) * sf;
    if (warp < 4) {
        const StateRow<SB> r(w, lane);
        float* dst = slice + (int64_t)(s.g0 + r.row) * D;
#pragma unroll
        for (int cb = 0; cb < D; cb += 16) {
            float v[16];
            tmem_ld_rows16(tm_lane + tTot + cb, v);
            if (r.live) store_row16(dst + cb, v);
        }
    } else if (tid >= 256 && tid < 256 + SB) {
        slice[(int64_t)a.S * D + s.g0 + tid - 256] = tot[tid - 256];
    }
    finish(s.tmem);
}

// ------------------------------------------------------------------------------------------------
template <int SB, int D>
__global__ void __launch_bounds__(kThreads, 1)
bwd_suffix_rows(const __grid_constant__ CUtensorMap map_do, const __grid_constant__ CUtensorMap map_v,
                const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q, const Args a) {
    using Ly = Lay<SB, D, true>;
    constexpr int HC = SB / 2, HD = D / 2;
    constexpr uint32_t tP = 128, tV = 384;
    const Setup s = begin<Ly, SB>(a);
    const Ctx& cx = s.cx;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* car = reinterpret_cast<float*>(cx.sm + Ly::oCar);
    float* sac = reinterpret_cast<float*>(cx.sm + Ly::oTot);
    const int64_t sf = (int64_t)a.S * (D + 1);
    const int wg = (warp >> 2) & 1, w = warp & 3, row = 32 * w + lane;
    const uint32_t tm_lane = s.tmem + ((uint32_t)(32 * w) << 16);
    const int col0 = HC * wg;

    if (warp < 8) {
        regs_inc<kRegsP>();
        const float* slice_a = a.ws + (s.n * s.tiles + s.tile) * sf + (int64_t)a.S * D + s.g0;
        const int64_t nchunk = (a.T + C - 1) / C;
        // running A before chunk cc, read a chunk ahead by the thread of column col0 + row
        const float* ac = a.achunk + (s.n * nchunk + s.t_begin / C) * a.S + s.g0 + col0 + row;
        if (row < HC) {
            car[col0 + row] = slice_a[col0 + row];
            sac[col0 + row] = ac[(int64_t)(s.nch - 1) * a.S];
        }
        asm volatile("bar.sync 5, 256;" ::: "memory");
        arrive_warp(cx, bPf);
        bool ok = true;
        for (int c = 0; c < s.nch && ok; ++c) {
            const uint32_t ph = (uint32_t)(c & 1);
            const int st = c % Ly::kStages, cc = s.nch - 1 - c;
            uint8_t* stage = cx.sm + st * Ly::kStage;
            const int64_t tok = s.t_begin + (int64_t)cc * C + row;
            const bool live = tok < s.t_end;
            // ---- W limbs over pQ and in a slot of its own ----------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bPf, ph, 101))) break;   // the group has finished the chunk before
            const float next_a = (row < HC && cc > 0) ? ac[(int64_t)(cc - 1) * a.S] : 0.f;
            if (!(ok = wait_bar_warp(cx, bFullQ + st, (uint32_t)((c / Ly::kStages) & 1), 102))) break;
            RACE_TRACE(wg, c, 0);
            if (!(ok = wait_bar_warp(cx, bA, ph, 103))) break;
            RACE_TRACE(wg, c, 1);
            tc_fence_after();
#pragma unroll
            for (int cb = 0; cb < HC; cb += 16) {
                float v[16];
                tmem_ld_rows16(tm_lane + tP + col0 + cb, v);
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 c4 = *reinterpret_cast<const float4*>(sac + col0 + cb + i);
                    v[i] = __fdividef(1.f, v[i] + c4.x + a.eps); v[i + 1] = __fdividef(1.f, v[i + 1] + c4.y + a.eps);
                    v[i + 2] = __fdividef(1.f, v[i + 2] + c4.z + a.eps); v[i + 3] = __fdividef(1.f, v[i + 3] + c4.w + a.eps);
                }
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const uint32_t off = sw_piece<C>(row, col0 + cb + 8 * p);
                    const uint4 q4 = *reinterpret_cast<const uint4*>(stage + Ly::oQ + off);
                    const uint32_t qq[4] = {q4.x, q4.y, q4.z, q4.w};
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 q2 = unpack2(qq[i]);
                        split2t(q2.x * v[8 * p + 2 * i], q2.y * v[8 * p + 2 * i + 1], hi[i], lo[i]);
                    }
                    *reinterpret_cast<uint4*>(stage + Ly::oQ + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4*>(cx.sm + Ly::oWlo + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
            }
            fence_proxy_async();
            tc_fence_before();
            arrive_warp(cx, bW);
            RACE_TRACE(wg, c, 2);
            // ---- dPK = P + sums of g (requested while the products run) -------------------------------------------
            const float* gsrc = a.gs + (s.n * a.T + tok) * a.S + s.g0 + col0;
            float gsv[HC];
#pragma unroll
            for (int i = 0; i < HC; i += 4) {
                const float4 x = live ? ld_chain<kLdOnce>(reinterpret_cast<const float4*>(gsrc + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
                gsv[i] = x.x; gsv[i + 1] = x.y; gsv[i + 2] = x.z; gsv[i + 3] = x.w;
            }
            if (!(ok = wait_bar_warp(cx, bX, ph, 106))) break;
            RACE_TRACE(wg, c, 3);
            tc_fence_after();
            __nv_bfloat16* dst = a.dp + (s.n * a.T + tok) * a.S + s.g0 + col0;
#pragma unroll
            for (int cb = 0; cb < HC; cb += 16) {
                float v[16];
                tmem_ld_rows16(tm_lane + tP + col0 + cb, v);
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 c4 = *reinterpret_cast<const float4*>(car + (c & 1) * SB + col0 + cb + i);
                    const float4 g4 = make_float4(gsv[cb + i] + c4.x, gsv[cb + i + 1] + c4.y, gsv[cb + i + 2] + c4.z,
                                                  gsv[cb + i + 3] + c4.w);
                    if (row == 0) *reinterpret_cast<float4*>(car + ((c + 1) & 1) * SB + col0 + cb + i) = g4;
                    v[i] += g4.x; v[i + 1] += g4.y; v[i + 2] += g4.z; v[i + 3] += g4.w;
                }
                if (live) store_row16(dst + cb, v, a.sectors);
            }
            if (row < HC) sac[col0 + row] = next_a;   // every warp has formed its W: the products are done
            tc_fence_before();
            arrive_warp(cx, bPf);
            RACE_TRACE(wg, c, 4);
        }
    } else if (warp < kStateWarp) {
        regs_dec<kRegsG>();
        write_tri<false>(tm_lane, row, wg);
        arrive_warp(cx, bTri);
        arrive_warp(cx, bVf);
        const bool shares = a.S > SB;
        bool ok = true;
        for (int c = 0; c < s.nch && ok; ++c) {
            const uint32_t ph = (uint32_t)(c & 1);
            const int64_t tok = s.t_begin + (int64_t)(s.nch - 1 - c) * C + row;
            const bool live = tok < s.t_end;
            // ---- masks of V dO^T and of pK W^T ---------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bG, ph, 105))) break;
            RACE_TRACE(3, c, 0);
            tc_fence_after();
            mask_product<true>(tm_lane, row, wg);
            arrive_warp(cx, bGm);
            RACE_TRACE(3, c, 1);
            if (!(ok = wait_bar_warp(cx, bH, ph, 108))) break;
            RACE_TRACE(3, c, 2);
            tc_fence_after();
            mask_product<true>(tm_lane, row, wg);
            arrive_warp(cx, bHm);
            RACE_TRACE(3, c, 3);
            // ---- dV ---------------------------------------------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bEnd, ph, 107))) break;
            RACE_TRACE(3, c, 4);
            tc_fence_after();
            write_tri<false>(tm_lane, row, wg);
            arrive_warp(cx, bTri);
            const int64_t srow = ((int64_t)s.block * gridDim.y + s.n) * a.T + tok;
            const int64_t orow = ((s.n / a.heads) * a.T + tok) * a.heads + s.n % a.heads;
#pragma unroll
            for (int cb = 0; cb < HD; cb += 16) {
                float v[16];
                tmem_ld_rows16(tm_lane + tV + HD * wg + cb, v);
                if (!live) continue;
                if (shares) store_row16((float*)a.dv + srow * D + HD * wg + cb, v);
                else store_row16((__nv_bfloat16*)a.dv + orow * D + HD * wg + cb, v, a.sectors);
            }
            tc_fence_before();
            arrive_warp(cx, bVf);
            RACE_TRACE(3, c, 5);
        }
    } else if (warp < kTmaWarp) {
        regs_dec<kRegsS>();
        load_state<SB, D, Ly>(s, a, w, lane);
        carry_state<SB, D, Ly>(s, w, lane);
    } else {
        regs_dec<kRegsM>();
        if (warp == kTmaWarp && lane == 0) produce<Ly>(s, a, &map_do, &map_v, &map_k, &map_q, true);
        if (warp == kMmaWarp) {
            const uint32_t tm0 = __shfl_sync(0xffffffffu, s.tmem, 0), smb0 = __shfl_sync(0xffffffffu, cx.sm_u32, 0);
            constexpr uint32_t iTS = idesc_mn(C, SB), iTT = idesc_mn(C, C), iTD = idesc_mn(C, D), iSD = idesc_mn(SB, D);
            if (elect_one()) {
                bool ok = true;
                for (int c = 0; c < s.nch && ok; ++c) {
                    const uint32_t ph = (uint32_t)(c & 1);
                    const int st = c % Ly::kStages;
                    // opaque per chunk: the descriptors are one addition each; kept across chunks they would be spilled
                    uint32_t tm = tm0, smb = smb0;
                    asm volatile("" : "+r"(tm), "+r"(smb));
                    const uint32_t base = smb + st * Ly::kStage;
                    const uint32_t sDO = base + Ly::oDO, sV = base + Ly::oV, sK = base + Ly::oK, sWh = base + Ly::oQ;
                    const uint32_t sBh = smb + Ly::oB, sBl = sBh + Ly::kB, sWl = smb + Ly::oWlo;
                    if (!(ok = wait_bar(cx, bTri, ph, 401))) break;
                    if (!(ok = wait_bar(cx, bPf, ph, 407))) break;
                    if (!(ok = wait_bar(cx, bFull + st, (uint32_t)((c / Ly::kStages) & 1), 402))) break;
                    tc_fence_after();
                    mma_sw_ta<true, 8, true, C>(tm + tP, tm + tG, sK, iTS);                  // A_loc = tril . pK
                    mma_commit(cx.bar(bA));
                    mma_sw<true, D / 16, false, C, false, C>(tm + tG, sV, sDO, iTT);         // V . dO^T (over tril)
                    mma_commit(cx.bar(bG));
                    if (!(ok = wait_bar(cx, bBt, ph, 403))) break;
                    if (!(ok = wait_bar(cx, bVf, ph, 408))) break;
                    tc_fence_after();
                    mma_sw<true, SB / 16, false, C, true, SB>(tm + tV, sK, sBh, iTD);        // dV = pK . SB
                    mma_sw<false, SB / 16, false, C, true, SB>(tm + tV, sK, sBl, iTD);
                    if (!(ok = wait_bar(cx, bW, ph, 404))) break;
                    tc_fence_after();
                    mma_sw<true, D / 16, false, C, false, SB>(tm + tP, sV, sBh, iTS);        // P = V . SB^T
                    mma_sw<false, D / 16, false, C, false, SB>(tm + tP, sV, sBl, iTS);
                    mma_commit(cx.bar(bXb));
                    if (!(ok = wait_bar(cx, bGm, ph, 405))) break;
                    tc_fence_after();
                    mma_sw_ta<false, 8, true, C, true>(tm + tP, tm + tG, sWh, iTS);          // P += triu(V dO^T) . W
                    mma_sw_ta<false, 8, true, C, true>(tm + tP, tm + tG, sWl, iTS);
                    mma_sw_ta<false, 8, true, C, true>(tm + tP, tm + tG + 16, sWh, iTS);
                    mma_commit(cx.bar(bX));
                    mma_sw<true, SB / 16, false, C, false, C>(tm + tG, sK, sWh, iTT);        // pK . W^T
                    mma_sw<false, SB / 16, false, C, false, C>(tm + tG, sK, sWl, iTT);
                    mma_commit(cx.bar(bH));
                    mma_sw<false, 8, true, C, true, C>(tm, sWh, sDO, iSD);                   // SB += W^T . dO
                    mma_sw<false, 8, true, C, true, C>(tm, sWl, sDO, iSD);
                    mma_commit(cx.bar(bSt));
                    if (!(ok = wait_bar(cx, bHm, ph, 406))) break;
                    tc_fence_after();
                    mma_sw_ta<false, 8, true, C, true>(tm + tV, tm + tG, sDO, iTD);          // dV += triu(pK W^T) . dO
                    mma_sw_ta<false, 8, true, C, true>(tm + tV, tm + tG + 16, sDO, iTD);
                    mma_commit(cx.bar(bEnd));
                    mma_commit(cx.bar(bEmpty + st));
                }
                mma_commit(cx.bar(bDrain));
                const long long t0 = clock64();
                while (!mbar_try_wait(cx.bar(bDrain), 0) && clock64() - t0 < cx.limit) {}
            }
        }
    }
    finish(s.tmem);
}

// dV [N/H, T, H, D] = sum over the bucket blocks of their shares [block][N, T, D], in block order; 8 values per thread
__global__ void __launch_bounds__(256)
bwd_dv_sum(const float* shares, __nv_bfloat16* __restrict__ dv, int64_t rows, int64_t T, int heads, int D,
           int blocks) {
    chain_release();
    chain_wait();
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int per = D / 8;
    if (i >= rows * per) return;
    const int64_t r = i / per;
    const int c = (int)(i % per) * 8;
    float acc[8] = {};
    for (int b = 0; b < blocks; ++b) {
        const float4* p = reinterpret_cast<const float4*>(shares + (b * rows + r) * D + c);
        const float4 x = ld_chain<kLdOnce>(p), y = ld_chain<kLdOnce>(p + 1);
        acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
        acc[4] += y.x; acc[5] += y.y; acc[6] += y.z; acc[7] += y.w;
    }
    const int64_t n = r / T, t = r - n * T;
    *reinterpret_cast<uint4*>(dv + (((n / heads) * T + t) * heads + n % heads) * D + c) =
        make_uint4(pack2(acc[0], acc[1]), pack2(acc[2], acc[3]), pack2(acc[4], acc[5]), pack2(acc[6], acc[7]));
}

// ---- host side ---------------------------------------------------------------------------------
inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

struct WsLayout {
    size_t prefix, suffix, gs, achunk, shares, total;
};
WsLayout ws_layout(const Dims& dm, int tile) {
    const int64_t tiles = (dm.T + tile - 1) / tile, nchunk = (dm.T + C - 1) / C;
    const size_t st = align256((size_t)dm.N * tiles * state_floats_per_stream(dm.S, dm.D) * 4);
    WsLayout l;
    l.prefix = 0;
    l.suffix = st;
    l.gs = 2 * st;
    l.achunk = l.gs + align256((size_t)dm.N * dm.T * dm.S * 4);
    l.shares = l.achunk + align256((size_t)dm.N * nchunk * dm.S * 4);
    l.total = l.shares + (dm.S > 128 ? align256((size_t)(dm.S / 128) * dm.N * dm.T * dm.D * 4) : 0);
    return l;
}

// [N/heads][T][heads][width] as (64 values, T tokens, column blocks, heads, outer), boxes of `blocks` x 128 tokens
bool map_rows(CUtensorMap* map, const void* base, int64_t N, int64_t T, int width, int blocks, int heads, int dims_n) {
    auto fn = tensor_map_encoder();
    if (!fn) return false;
    cuuint64_t dims[5] = {64, (cuuint64_t)T, (cuuint64_t)(width / 64), (cuuint64_t)(dims_n == 5 ? heads : N),
                          (cuuint64_t)(N / heads)};
    cuuint64_t strides[4] = {(cuuint64_t)heads * width * 2, 128, (cuuint64_t)(dims_n == 5 ? width : T * width) * 2,
                             (cuuint64_t)T * heads * width * 2};
    cuuint32_t box[5] = {64, (cuuint32_t)C, (cuuint32_t)blocks, 1, 1};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)dims_n, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int SB, int D>
cudaError_t launch(const void* pq, const void* pk, const void* v, const void* dout, const float* carry_in,
                   const float* d_state, void* dpq, void* dpk, void* dv, float* d_carry, void* ws, const Dims& dm,
                   int tile, cudaStream_t stream, int* status) {
    const WsLayout l = ws_layout(dm, tile);
    char* base = (char*)ws;
    float* wp = (float*)(base + l.prefix);
    float* wsf = (float*)(base + l.suffix);
    const int64_t tiles = (dm.T + tile - 1) / tile;
    const int blocks = dm.S / SB;
    auto k1 = bwd_prefix_rows<SB, D>;
    auto k2 = bwd_suffix_rows<SB, D>;
    constexpr int smem1 = Lay<SB, D, false>::kSmem, smem2 = Lay<SB, D, true>::kSmem;
    cudaError_t err = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1);
    if (err == cudaSuccess) err = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2);
    if (err != cudaSuccess) return err;
    // state before every tile: the forward's totals and scan
    err = causal_fwd_tensor(nullptr, pk, v, nullptr, nullptr, nullptr, wp, false, dm, RACE_DTYPE_BF16, tile, stream, status,
                            kPhaseTotals | kPhasePrefixOnly);
    if (err == cudaSuccess) err = causal_scan_tiles(wp, carry_in, nullptr, dm, tile, stream, true);
    if (err != cudaSuccess) return err;
    CUtensorMap mdo, mv, mk, mq;
    if (!map_rows(&mdo, dout, dm.N, dm.T, D, D / 64, dm.H, 5) || !map_rows(&mv, v, dm.N, dm.T, D, D / 64, dm.H, 5) ||
        !map_rows(&mk, pk, dm.N, dm.T, dm.S, SB / 64, 1, 4) || !map_rows(&mq, pq, dm.N, dm.T, dm.S, SB / 64, 1, 4))
        return cudaErrorInvalidValue;
    Args a;
    a.ws = wp;
    a.ws_out = wsf;
    a.dp = (__nv_bfloat16*)dpq;
    a.gs = (float*)(base + l.gs);
    a.achunk = (float*)(base + l.achunk);
    a.dv = nullptr;
    a.T = dm.T;
    a.S = dm.S;
    a.heads = dm.H;
    a.tile_tokens = tile;
    a.eps = dm.eps;
    a.status = status;
    auto on_sector = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; };
    a.sectors = on_sector(dpq);
    const dim3 grid((unsigned)(tiles * blocks), (unsigned)dm.N);
    err = launch_chain(chain_launches(dm), k1, grid, kThreads, smem1, stream, mdo, mv, mk, mq, a);
    if (err == cudaSuccess) err = causal_scan_tiles(wsf, d_state, d_carry, dm, tile, stream, true, /*reverse=*/true);
    if (err != cudaSuccess) return err;
    a.ws = wsf;
    a.dp = (__nv_bfloat16*)dpk;
    a.dv = blocks > 1 ? (void*)(base + l.shares) : dv;
    a.sectors = on_sector(dpk) && on_sector(a.dv);
    err = launch_chain(chain_launches(dm), k2, grid, kThreads, smem2, stream, mdo, mv, mk, mq, a);
    if (err != cudaSuccess || blocks == 1) return err;
    const int64_t rows = dm.N * dm.T;
    return launch_chain(chain_launches(dm), bwd_dv_sum, (unsigned)((rows * (D / 8) + 255) / 256), 256, 0, stream, (const float*)(base + l.shares),
                        (__nv_bfloat16*)dv, rows, dm.T, dm.H, D, blocks);
}

}  // namespace

bool causal_bwd_bf16_supported(const Dims& dm) {
    return (dm.S == 64 || dm.S == 128 || dm.S == 256 || dm.S == 512) && (dm.D == 64 || dm.D == 128) && dm.N <= 65535 &&
           dm.T < (1ll << 31) - 4096;
}

// One CTA per SM: tiles that fill the last wave of (stream, tile, bucket block) items; a CTA's set-up and its share of
// the totals and scans cost about two chunks
int causal_bwd_bf16_tile_tokens(const Dims& dm, int sm_count) {
    const int64_t sms = sm_count > 0 ? sm_count : 148, blocks = dm.S == 64 ? 1 : dm.S / 128;
    int best = 2048;
    double best_cost = 1e300;
    for (int tile = 4096; tile >= C; tile -= C) {
        const int64_t ctas = dm.N * blocks * ((dm.T + tile - 1) / tile), waves = (ctas + sms - 1) / sms;
        const double cost = (double)waves * (std::min<int64_t>(tile, (dm.T + C - 1) / C * C) + 256.0);
        if (cost < best_cost * 0.999) { best_cost = cost; best = tile; }
        if (ctas > 64 * sms) break;
    }
    return best;
}

size_t causal_bwd_bf16_workspace_bytes(const Dims& dm, int tile) {
    return dm.N == 0 || dm.T == 0 ? 0 : ws_layout(dm, tile).total;
}

cudaError_t causal_bwd_bf16(const void* pq, const void* pk, const void* v, const void* dout, const float* carry_in,
                            const float* d_state, void* dpq, void* dpk, void* dv, float* d_carry, void* ws, const Dims& dm,
                            int tile, cudaStream_t stream, int* status) {
#define RACE_CASE(SB_, D_)                                                                                            \
    if ((dm.S == 64) == (SB_ == 64) && dm.D == D_)                                                                     \
        return launch<SB_, D_>(pq, pk, v, dout, carry_in, d_state, dpq, dpk, dv, d_carry, ws, dm, tile, stream, status);
    RACE_CASE(64, 64) RACE_CASE(64, 128) RACE_CASE(128, 64) RACE_CASE(128, 128)
#undef RACE_CASE
    return cudaErrorInvalidValue;
}

}  // namespace race
