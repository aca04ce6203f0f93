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
// Precision is that of fp32 arithmetic on the bf16 inputs up to 2^-17: inputs are exact one-limb operands, everything
// computed (W, the masked products, the states, g) is split into hi + lo bf16 limbs, accumulators are fp32.
//
// Why this shape of kernel.  On CUDA cores the two passes took 3.3 of 3.4 ms of ... (S = 64) and 9.0 of 9.8 ms (S = 512)
// of a training step.  Chunks of 128 tokens and blocks of 128 buckets make every product 128 x 128 x 128 (full M, N of
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
constexpr int kThreads = 16 * 32;   // 8 worker warps, 4 state warps, one group with the TMA and MMA warps
constexpr int kTmaWarp = 12, kMmaWarp = 13;
constexpr uint32_t tG = 256;        // tensor-memory columns: states [0, 256), masked products [256, 384), results [384, 512)

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
    static constexpr int oTot = oCar + 2 * SB * 4;                           // [SB] fp32 totals of g (prefix pass)
    static constexpr int oBars = oTot + SB * 4;
    static constexpr int kNumBars = 20;
    static constexpr int oMisc = oBars + kNumBars * 8;
    static constexpr int kSmem = oMisc + 16 + 1024;
    static_assert(kSmem <= 227 * 1024, "shared memory of the backward");
};
enum Bar {
    bFull = 0,      // [2] dO, V, pK of the stage have landed
    bFullQ = 2,     // [2] pQ
    bTri = 4,       // the triangular matrix of the chunk is in the G columns, every result of the chunk before is read (8)
    bA = 5,         // running sums of pK inside the chunk
    bG = 6,         // first token x token product
    bSt = 7,        // state updated with the chunk
    bXb = 8,        // operand tiles of the state no longer read
    bBt = 9,        // operand tiles of the state before the chunk written, accumulator read (4)
    bW = 10,        // W limbs written, running sums read (8)
    bGm = 11,       // masked first product written (8)
    bX = 12,        // prefix: X complete.  suffix: second token x token product complete
    bXg = 13,       // prefix: X read, g limbs written (8).  suffix: masked second product written (8)
    bEnd = 14,      // every product of the chunk has run
    bEmpty = 15,    // [2] ... of the chunk in the stage
    bDrain = 17
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
    if (threadIdx.x == 0) {
        *s.cx.abort_flag = 0;
        for (int i = 0; i < Ly::kNumBars; ++i) {
            const uint32_t cnt = (i == bTri || i == bW || i == bGm || i == bXg) ? 8u : i == bBt ? 4u : 1u;
            mbar_init(s.cx.bar(i), cnt);
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
                                                  const float (&v)[32]) {
    uint32_t hi[16], lo[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) split2(v[2 * i], v[2 * i + 1], hi[i], lo[i]);
    if (r.live) {
        sw_store_row<SB, 16>(hi_tile, r.row, col, hi);
        sw_store_row<SB, 16>(hi_tile + lo_off, r.row, col, lo);
    }
}

// Carry into the tile: B -> accumulator and operand tiles (state warps)
template <int SB, int D, typename Ly>
__device__ __forceinline__ void load_state(const Setup& s, const Args& a, int w, int lane) {
    const StateRow<SB> r(w, lane);
    const float* src = a.ws + (s.n * s.tiles + s.tile) * (int64_t)(a.S * (D + 1)) + (int64_t)(s.g0 + r.row) * D;
#pragma unroll
    for (int cb = 0; cb < D; cb += 32) {
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            const float4 x = r.live ? __ldg(reinterpret_cast<const float4*>(src + cb + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
        }
        tmem_st_rows32(((uint32_t)(32 * w) << 16) + s.tmem + cb, v);
        store_state_limbs<SB>(s.cx.sm + Ly::oB, Ly::kB, r, cb, v);
    }
    fence_proxy_async();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(s.cx.bar(bBt));
}
// after every chunk but the last: updated accumulator -> operand tiles
template <int SB, int D, typename Ly>
__device__ __forceinline__ void carry_state(const Setup& s, int w, int lane) {
    const StateRow<SB> r(w, lane);
    bool ok = true;
    for (int c = 1; c < s.nch && ok; ++c) {
        if (!(ok = wait_bar_warp(s.cx, bSt, (uint32_t)((c - 1) & 1), 201))) break;
        if (!(ok = wait_bar_warp(s.cx, bXb, (uint32_t)((c - 1) & 1), 202))) break;
        tc_fence_after();
#pragma unroll
        for (int cb = 0; cb < D; cb += 32) {
            float v[32];
            tmem_ld_rows32(((uint32_t)(32 * w) << 16) + s.tmem + cb, v);
            store_state_limbs<SB>(s.cx.sm + Ly::oB, Ly::kB, r, cb, v);
        }
        fence_proxy_async();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s.cx.bar(bBt));
    }
}

// the 64 columns [64 wg, +64) of a token x token product: mask (kUpper: column >= row stays), split, and write the limbs
// over the columns just read (hi in the first 32, lo in the second)
template <bool kUpper>
__device__ __forceinline__ void mask_product(uint32_t tm_lane, int row, int wg) {
    uint32_t hi[32], lo[32];
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {
        float v[32];
        tmem_ld_rows32(tm_lane + tG + 64 * wg + 32 * hb, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int col = 64 * wg + 32 * hb + 2 * i;
            const float x = (kUpper ? col >= row : col <= row) ? v[2 * i] : 0.f;
            const float y = (kUpper ? col + 1 >= row : col + 1 <= row) ? v[2 * i + 1] : 0.f;
            split2(x, y, hi[16 * hb + i], lo[16 * hb + i]);
        }
    }
    tmem_st_words32(tm_lane + tG + 64 * wg, hi);
    tmem_st_words32(tm_lane + tG + 64 * wg + 32, lo);
    tc_fence_before();
}
template <bool kUpper>
__device__ __forceinline__ void write_tri(uint32_t tm_lane, int row, int wg) {
    uint32_t tr[32];
    tri_words<kUpper>(row, wg, tr);
    tmem_st_words32(tm_lane + tG + 32 * wg, tr);
    tc_fence_before();
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

    if (warp >= 12) regs_dec<72>();
    if (warp < 8) {
        regs_inc<168>();
        const int wg = warp >> 2, w = warp & 3, row = 32 * w + lane;
        const uint32_t tm_lane = s.tmem + ((uint32_t)(32 * w) << 16);
        const int col0 = HC * wg;                    // first bucket column of this thread inside the block
        const float* slice_a = a.ws + (s.n * s.tiles + s.tile) * sf + (int64_t)a.S * D + s.g0;
        if (row < HC) {
            car[col0 + row] = slice_a[col0 + row];
            tot[col0 + row] = 0.f;
        }
        asm volatile("bar.sync 5, 256;" ::: "memory");
        write_tri<false>(tm_lane, row, wg);
        __syncwarp();
        if (lane == 0) mbar_arrive(cx.bar(bTri));
        const int64_t nchunk = (a.T + C - 1) / C;
        bool ok = true;
        for (int c = 0; c < s.nch && ok; ++c) {
            const uint32_t ph = (uint32_t)(c & 1);
            const int st = c % Ly::kStages;
            uint8_t* stage = cx.sm + st * Ly::kStage;
            const int64_t tok = s.t_begin + (int64_t)c * C + row;
            const bool live = tok < s.t_end;
            // ---- running A, W = pQ / (A + eps) -> limbs over pQ and over V ---------------------------------
            if (!(ok = wait_bar_warp(cx, bTri, ph, 101))) break;   // every worker has finished the chunk before
            if (row < HC)
                a.achunk[(s.n * nchunk + s.t_begin / C + c) * a.S + s.g0 + col0 + row] = car[(c & 1) * SB + col0 + row];
            if (!(ok = wait_bar_warp(cx, bFullQ + st, (uint32_t)((c / Ly::kStages) & 1), 102))) break;
            if (!(ok = wait_bar_warp(cx, bA, ph, 103))) break;
            tc_fence_after();
            float inv[HC];
            uint32_t pq[HC / 2];
#pragma unroll
            for (int cb = 0; cb < HC; cb += 32) {
                float v[32];
                tmem_ld_rows32(tm_lane + tX + col0 + cb, v);
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 c4 = *reinterpret_cast<const float4*>(car + (c & 1) * SB + col0 + cb + i);
                    v[i] += c4.x; v[i + 1] += c4.y; v[i + 2] += c4.z; v[i + 3] += c4.w;
                }
                if (row == C - 1) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4*>(car + ((c + 1) & 1) * SB + col0 + cb + i) =
                            make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) inv[cb + i] = __fdividef(1.f, v[i] + a.eps);
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
                    pq[4 * p + i] = qq[i];
                    const float2 q2 = unpack2(qq[i]);
                    split2(q2.x * inv[8 * p + 2 * i], q2.y * inv[8 * p + 2 * i + 1], hi[i], lo[i]);
                }
                *reinterpret_cast<uint4*>(stage + Ly::oQ + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(stage + Ly::oV + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bW));
            // ---- causal mask of dO V^T --------------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bG, ph, 105))) break;
            tc_fence_after();
            mask_product<false>(tm_lane, row, wg);
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bGm));
            // ---- X -> dPQ, g limbs over W ---------------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bX, ph, 106))) break;
            tc_fence_after();
            __nv_bfloat16* dst = a.dp + (s.n * a.T + tok) * a.S + s.g0 + col0;
#pragma unroll
            for (int cb = 0; cb < HC; cb += 32) {
                float v[32];
                tmem_ld_rows32(tm_lane + tX + col0 + cb, v);
                uint32_t hi[16], lo[16], d[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float i0 = inv[cb + 2 * i], i1 = inv[cb + 2 * i + 1];
                    const float2 q2 = unpack2(pq[cb / 2 + i]);
                    const float d0 = v[2 * i] * i0, d1 = v[2 * i + 1] * i1;
                    d[i] = pack2(d0, d1);
                    split2(-d0 * (q2.x * i0), -d1 * (q2.y * i1), hi[i], lo[i]);
                }
                sw_store_row<C, 16>(stage + Ly::oQ, row, col0 + cb, hi);
                sw_store_row<C, 16>(stage + Ly::oV, row, col0 + cb, lo);
                if (live) {
                    st_global_32b(dst + cb, reinterpret_cast<const uint32_t(&)[8]>(d[0]));
                    st_global_32b(dst + cb + 16, reinterpret_cast<const uint32_t(&)[8]>(d[8]));
                }
            }
            write_tri<true>(tm_lane, row, wg);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bXg));
            // ---- suffix sums of g inside the chunk ------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bEnd, ph, 107))) break;
            tc_fence_after();
            float* gdst = a.gs + (s.n * a.T + tok) * a.S + s.g0 + col0;
#pragma unroll
            for (int cb = 0; cb < HC; cb += 32) {
                float v[32];
                tmem_ld_rows32(tm_lane + tX + col0 + cb, v);
                if (live) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8)
                        st_global_32b(gdst + cb + i, reinterpret_cast<const uint32_t(&)[8]>(v[i]));
                }
                if (row == 0) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        float4* t4 = reinterpret_cast<float4*>(tot + col0 + cb + i);
                        const float4 x = *t4;
                        *t4 = make_float4(x.x + v[i], x.y + v[i + 1], x.z + v[i + 2], x.w + v[i + 3]);
                    }
                }
            }
            write_tri<false>(tm_lane, row, wg);
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bTri));
        }
    } else if (warp < 12) {
        regs_dec<96>();
        load_state<SB, D, Ly>(s, a, warp & 3, lane);
        carry_state<SB, D, Ly>(s, warp & 3, lane);
    } else if (warp == kTmaWarp) {
        if (lane == 0) produce<Ly>(s, a, &map_do, &map_v, &map_k, &map_q, false);
    } else if (warp == kMmaWarp) {
        const uint32_t tm = __shfl_sync(0xffffffffu, s.tmem, 0), smb = __shfl_sync(0xffffffffu, cx.sm_u32, 0);
        constexpr uint32_t iTS = idesc_mn(C, SB), iTT = idesc_mn(C, C), iSD = idesc_mn(SB, D);
        if (elect_one()) {
            bool ok = true;
            for (int c = 0; c < s.nch && ok; ++c) {
                const uint32_t ph = (uint32_t)(c & 1);
                const int st = c % Ly::kStages;
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
                if (c == 0) mma_sw<true, 8, true, C, true, C>(tm + tTot, sQ, sDO, iSD);      // totals += W^T . dO
                else mma_sw<false, 8, true, C, true, C>(tm + tTot, sQ, sDO, iSD);
                mma_sw<false, 8, true, C, true, C>(tm + tTot, sV, sDO, iSD);
                if (!(ok = wait_bar(cx, bGm, ph, 405))) break;
                tc_fence_after();
                mma_sw_ta<false, 8, true, C, true>(tm + tX, tm + tG, sK, iTS);               // X += tril(G) . pK
                mma_sw_ta<false, 8, true, C, true>(tm + tX, tm + tG + 32, sK, iTS);
                mma_commit(cx.bar(bX));
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
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // totals of the tile
    float* slice = a.ws_out + (s.n * s.tiles + s.tile) * sf;
    if (warp >= 8 && warp < 12) {
        const int w = warp & 3;
        const StateRow<SB> r(w, lane);
        float* dst = slice + (int64_t)(s.g0 + r.row) * D;
#pragma unroll
        for (int cb = 0; cb < D; cb += 32) {
            float v[32];
            tmem_ld_rows32(((uint32_t)(32 * w) << 16) + s.tmem + tTot + cb, v);
            if (r.live) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) st_global_32b(dst + cb + i, reinterpret_cast<const uint32_t(&)[8]>(v[i]));
            }
        }
    } else if (tid < SB) {
        slice[(int64_t)a.S * D + s.g0 + tid] = tot[tid];
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
    const int64_t sf = (int64_t)a.S * (D + 1);

    if (warp >= 12) regs_dec<72>();
    if (warp < 8) {
        regs_inc<168>();
        const int wg = warp >> 2, w = warp & 3, row = 32 * w + lane;
        const uint32_t tm_lane = s.tmem + ((uint32_t)(32 * w) << 16);
        const int col0 = HC * wg;
        const float* slice_a = a.ws + (s.n * s.tiles + s.tile) * sf + (int64_t)a.S * D + s.g0;
        if (row < HC) car[col0 + row] = slice_a[col0 + row];
        asm volatile("bar.sync 5, 256;" ::: "memory");
        write_tri<false>(tm_lane, row, wg);
        __syncwarp();
        if (lane == 0) mbar_arrive(cx.bar(bTri));
        const int64_t nchunk = (a.T + C - 1) / C;
        const bool shares = a.S > SB;
        bool ok = true;
        for (int c = 0; c < s.nch && ok; ++c) {
            const uint32_t ph = (uint32_t)(c & 1);
            const int st = c % Ly::kStages, cc = s.nch - 1 - c;
            uint8_t* stage = cx.sm + st * Ly::kStage;
            const int64_t tok = s.t_begin + (int64_t)cc * C + row;
            const bool live = tok < s.t_end;
            // ---- W limbs over pQ and in a slot of its own ----------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bTri, ph, 101))) break;   // every worker has finished the chunk before
            const float* ac = a.achunk + (s.n * nchunk + s.t_begin / C + cc) * a.S + s.g0 + col0;
            if (!(ok = wait_bar_warp(cx, bFullQ + st, (uint32_t)((c / Ly::kStages) & 1), 102))) break;
            if (!(ok = wait_bar_warp(cx, bA, ph, 103))) break;
            tc_fence_after();
#pragma unroll
            for (int cb = 0; cb < HC; cb += 32) {
                float v[32];
                tmem_ld_rows32(tm_lane + tP + col0 + cb, v);
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 c4 = __ldg(reinterpret_cast<const float4*>(ac + cb + i));
                    v[i] = __fdividef(1.f, v[i] + c4.x + a.eps); v[i + 1] = __fdividef(1.f, v[i + 1] + c4.y + a.eps);
                    v[i + 2] = __fdividef(1.f, v[i + 2] + c4.z + a.eps); v[i + 3] = __fdividef(1.f, v[i + 3] + c4.w + a.eps);
                }
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const uint32_t off = sw_piece<C>(row, col0 + cb + 8 * p);
                    const uint4 q4 = *reinterpret_cast<const uint4*>(stage + Ly::oQ + off);
                    const uint32_t qq[4] = {q4.x, q4.y, q4.z, q4.w};
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 q2 = unpack2(qq[i]);
                        split2(q2.x * v[8 * p + 2 * i], q2.y * v[8 * p + 2 * i + 1], hi[i], lo[i]);
                    }
                    *reinterpret_cast<uint4*>(stage + Ly::oQ + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4*>(cx.sm + Ly::oWlo + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
            }
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bW));
            // ---- mask of V dO^T, then of pK W^T -------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bG, ph, 105))) break;
            tc_fence_after();
            mask_product<true>(tm_lane, row, wg);
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bGm));
            // sums of g of this chunk, requested while the products run
            float gsv[HC];
            const float* gsrc = a.gs + (s.n * a.T + tok) * a.S + s.g0 + col0;
#pragma unroll
            for (int i = 0; i < HC; i += 4) {
                const float4 x = live ? __ldcs(reinterpret_cast<const float4*>(gsrc + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
                gsv[i] = x.x; gsv[i + 1] = x.y; gsv[i + 2] = x.z; gsv[i + 3] = x.w;
            }
            if (!(ok = wait_bar_warp(cx, bX, ph, 106))) break;
            tc_fence_after();
            mask_product<true>(tm_lane, row, wg);
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bXg));
            // ---- dPK = P + sums of g ------------------------------------------------------------------------------
            __nv_bfloat16* dst = a.dp + (s.n * a.T + tok) * a.S + s.g0 + col0;
#pragma unroll
            for (int cb = 0; cb < HC; cb += 32) {
                float v[32];
                tmem_ld_rows32(tm_lane + tP + col0 + cb, v);
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 c4 = *reinterpret_cast<const float4*>(car + (c & 1) * SB + col0 + cb + i);
                    const float4 g4 = make_float4(gsv[cb + i] + c4.x, gsv[cb + i + 1] + c4.y, gsv[cb + i + 2] + c4.z,
                                                  gsv[cb + i + 3] + c4.w);
                    if (row == 0) *reinterpret_cast<float4*>(car + ((c + 1) & 1) * SB + col0 + cb + i) = g4;
                    v[i] += g4.x; v[i + 1] += g4.y; v[i + 2] += g4.z; v[i + 3] += g4.w;
                }
                uint32_t d[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) d[i] = pack2(v[2 * i], v[2 * i + 1]);
                if (live) {
                    st_global_32b(dst + cb, reinterpret_cast<const uint32_t(&)[8]>(d[0]));
                    st_global_32b(dst + cb + 16, reinterpret_cast<const uint32_t(&)[8]>(d[8]));
                }
            }
            // ---- dV ---------------------------------------------------------------------------------------------------
            if (!(ok = wait_bar_warp(cx, bEnd, ph, 107))) break;
            tc_fence_after();
#pragma unroll
            for (int cb = 0; cb < HD; cb += 32) {
                float v[32];
                tmem_ld_rows32(tm_lane + tV + HD * wg + cb, v);
                if (!live) continue;
                if (shares) {
                    float* o = (float*)a.dv + (((int64_t)s.block * gridDim.y + s.n) * a.T + tok) * D + HD * wg + cb;
#pragma unroll
                    for (int i = 0; i < 32; i += 8) st_global_32b(o + i, reinterpret_cast<const uint32_t(&)[8]>(v[i]));
                } else {
                    __nv_bfloat16* o = (__nv_bfloat16*)a.dv +
                                       (((s.n / a.heads) * a.T + tok) * a.heads + s.n % a.heads) * D + HD * wg + cb;
                    uint32_t d[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) d[i] = pack2(v[2 * i], v[2 * i + 1]);
                    st_global_32b(o, reinterpret_cast<const uint32_t(&)[8]>(d[0]));
                    st_global_32b(o + 16, reinterpret_cast<const uint32_t(&)[8]>(d[8]));
                }
            }
            write_tri<false>(tm_lane, row, wg);
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(bTri));
        }
    } else if (warp < 12) {
        regs_dec<96>();
        load_state<SB, D, Ly>(s, a, warp & 3, lane);
        carry_state<SB, D, Ly>(s, warp & 3, lane);
    } else if (warp == kTmaWarp) {
        if (lane == 0) produce<Ly>(s, a, &map_do, &map_v, &map_k, &map_q, true);
    } else if (warp == kMmaWarp) {
        const uint32_t tm = __shfl_sync(0xffffffffu, s.tmem, 0), smb = __shfl_sync(0xffffffffu, cx.sm_u32, 0);
        constexpr uint32_t iTS = idesc_mn(C, SB), iTT = idesc_mn(C, C), iTD = idesc_mn(C, D), iSD = idesc_mn(SB, D);
        const uint32_t sBh = smb + Ly::oB, sBl = sBh + Ly::kB, sWl = smb + Ly::oWlo;
        if (elect_one()) {
            bool ok = true;
            for (int c = 0; c < s.nch && ok; ++c) {
                const uint32_t ph = (uint32_t)(c & 1);
                const int st = c % Ly::kStages;
                const uint32_t base = smb + st * Ly::kStage;
                const uint32_t sDO = base + Ly::oDO, sV = base + Ly::oV, sK = base + Ly::oK, sWh = base + Ly::oQ;
                if (!(ok = wait_bar(cx, bTri, ph, 401))) break;
                if (!(ok = wait_bar(cx, bFull + st, (uint32_t)((c / Ly::kStages) & 1), 402))) break;
                tc_fence_after();
                mma_sw_ta<true, 8, true, C>(tm + tP, tm + tG, sK, iTS);                  // A_loc = tril . pK
                mma_commit(cx.bar(bA));
                mma_sw<true, D / 16, false, C, false, C>(tm + tG, sV, sDO, iTT);         // V . dO^T (over tril)
                mma_commit(cx.bar(bG));
                if (!(ok = wait_bar(cx, bBt, ph, 403))) break;
                tc_fence_after();
                mma_sw<true, SB / 16, false, C, true, SB>(tm + tV, sK, sBh, iTD);        // dV = pK . SB
                mma_sw<false, SB / 16, false, C, true, SB>(tm + tV, sK, sBl, iTD);
                if (!(ok = wait_bar(cx, bW, ph, 404))) break;
                tc_fence_after();
                mma_sw<true, D / 16, false, C, false, SB>(tm + tP, sV, sBh, iTS);        // P = V . SB^T
                mma_sw<false, D / 16, false, C, false, SB>(tm + tP, sV, sBl, iTS);
                mma_commit(cx.bar(bXb));
                mma_sw<false, 8, true, C, true, C>(tm, sWh, sDO, iSD);                   // SB += W^T . dO
                mma_sw<false, 8, true, C, true, C>(tm, sWl, sDO, iSD);
                mma_commit(cx.bar(bSt));
                if (!(ok = wait_bar(cx, bGm, ph, 405))) break;
                tc_fence_after();
                mma_sw_ta<false, 8, true, C, true>(tm + tP, tm + tG, sWh, iTS);          // P += triu(V dO^T) . W
                mma_sw_ta<false, 8, true, C, true>(tm + tP, tm + tG, sWl, iTS);
                mma_sw_ta<false, 8, true, C, true>(tm + tP, tm + tG + 32, sWh, iTS);
                mma_sw<true, SB / 16, false, C, false, C>(tm + tG, sK, sWh, iTT);        // pK . W^T
                mma_sw<false, SB / 16, false, C, false, C>(tm + tG, sK, sWl, iTT);
                mma_commit(cx.bar(bX));
                if (!(ok = wait_bar(cx, bXg, ph, 406))) break;
                tc_fence_after();
                mma_sw_ta<false, 8, true, C, true>(tm + tV, tm + tG, sDO, iTD);          // dV += triu(pK W^T) . dO
                mma_sw_ta<false, 8, true, C, true>(tm + tV, tm + tG + 32, sDO, iTD);
                mma_commit(cx.bar(bEnd));
                mma_commit(cx.bar(bEmpty + st));
            }
            mma_commit(cx.bar(bDrain));
            const long long t0 = clock64();
            while (!mbar_try_wait(cx.bar(bDrain), 0) && clock64() - t0 < cx.limit) {}
        }
    }
    finish(s.tmem);
}

// dV [N/H, T, H, D] = sum over the bucket blocks of their shares [block][N, T, D], in block order; 8 values per thread
__global__ void __launch_bounds__(256)
bwd_dv_sum(const float* __restrict__ shares, __nv_bfloat16* __restrict__ dv, int64_t rows, int64_t T, int heads, int D,
           int blocks) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int per = D / 8;
    if (i >= rows * per) return;
    const int64_t r = i / per;
    const int c = (int)(i % per) * 8;
    float acc[8] = {};
    for (int b = 0; b < blocks; ++b) {
        const float4* p = reinterpret_cast<const float4*>(shares + (b * rows + r) * D + c);
        const float4 x = __ldcs(p), y = __ldcs(p + 1);
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
                            kPhaseTotals);
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
    const dim3 grid((unsigned)(tiles * blocks), (unsigned)dm.N);
    k1<<<grid, kThreads, smem1, stream>>>(mdo, mv, mk, mq, a);
    err = cudaGetLastError();
    if (err == cudaSuccess) err = causal_scan_tiles(wsf, d_state, d_carry, dm, tile, stream, true, /*reverse=*/true);
    if (err != cudaSuccess) return err;
    a.ws = wsf;
    a.dp = (__nv_bfloat16*)dpk;
    a.dv = blocks > 1 ? (void*)(base + l.shares) : dv;
    k2<<<grid, kThreads, smem2, stream>>>(mdo, mv, mk, mq, a);
    err = cudaGetLastError();
    if (err != cudaSuccess || blocks == 1) return err;
    const int64_t rows = dm.N * dm.T;
    bwd_dv_sum<<<(unsigned)((rows * (D / 8) + 255) / 256), 256, 0, stream>>>((const float*)(base + l.shares),
                                                                             (__nv_bfloat16*)dv, rows, dm.T, dm.H, D, blocks);
    return cudaGetLastError();
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
