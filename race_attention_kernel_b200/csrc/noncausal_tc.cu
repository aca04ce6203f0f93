// Non-causal per-bucket token kernels on the tensor cores (tcgen05 / TMEM / TMA), S = 64 buckets, d_k = 64.
//
// Every token-side product of the non-causal path is "rows of a [T, 64] input times one constant
// 64 x 64 matrix of the stream":
//   forward :  out = pQ . E                         (E = Bs / (A + eps))
//   backward:  dPQ = dO . E^T;  dPK = V . dBs^T + dA;  dV = pK . dBs
//              (dBs = dE / (A + eps), dA[s] = - dE[s] . Bs[s] / (A + eps)^2, dE = pQ^T dO from the totals kernel)
// (the forward is the second half of the four lines the reference quotes from upstream,
// analysis/hot-path.md:157-162; the gradients are its closed form).
//
// A streaming kernel: it reads and writes every token row once, so memory is the bound and everything else has to stay
// out of the way of it.  One persistent CTA per SM owns an equal share of all 128-token chunks (a share may begin and
// end inside a stream); per chunk it runs one item (forward) or three (backward).  An item lives in one slot of a ring:
//   * TMA brings the 128 rows (128-byte swizzle: a thread reads its row 16 bytes at a time without bank conflicts);
//   * fp32: the four warps of a worker group split their rows into bf16 hi + lo limbs and put them into tensor memory as
//     the A operand (hi.hi + hi.lo + lo.hi); bf16: the slot is the A operand as it is (exact in one limb);
//   * M = 128 products against limb tiles of the stream's matrix in shared memory (one image serves as X and X^T);
//   * the group writes the result rows over the slot and TMA stores them.
// So global memory only sees whole-row TMA transfers.  (Before, the fragment layout went straight to global memory:
// 8-byte accesses to eight rows per instruction, eight cache lines for 256 bytes, 4.3 TB/s of the copy's 6.5.)
// A preparation group splits the matrices of the next stream meanwhile (two buffers).  Every wait on a barrier is
// bounded; a wait that runs out raises the CTA's abort flag and a device status word, and the CTA leaves.
#include <algorithm>

#include "common.cuh"
#include "launch.h"
#include "tc_rows.cuh"

namespace race {
namespace {

constexpr int C = 128;                      // tokens per chunk
constexpr int kGroups = 4;                  // worker groups of four warps; group g takes the items g (mod 4)
constexpr int kPrepWarp = 16, kLoadWarp = 20, kMmaWarp = 21, kStoreWarp = 22;
constexpr int kNcThreads = 24 * 32;
constexpr int kTile = 64 * 64 * 2;          // one bf16 limb tile of a 64 x 64 matrix

template <typename Tin, bool kBwd>
struct NcLay {
    static constexpr int kSlot = C * 64 * (int)sizeof(Tin);
    static constexpr int kMat = (kBwd ? 4 : 2) * kTile;          // E hi | lo (| dBs hi | lo)
    static constexpr int kSlots = (sizeof(Tin) == 4 ? (kBwd ? 5 : 6) : (kBwd ? 9 : 12));
    static constexpr int oSlot = 0, oMat = kSlots * kSlot;       // [2] matrices
    static constexpr int oDa = oMat + 2 * kMat;                  // [4][64] dA: read by the workers after the products
    static constexpr int oBars = oDa + (kBwd ? 4 * 64 * 4 : 0);
    static constexpr int bFull = 0, bOut = kSlots, bEmpty = 2 * kSlots, bA = 3 * kSlots, bO = bA + kGroups,
                         bMat = bO + kGroups, bMatFree = bMat + 2, bDrain = bMatFree + 2, kNumBars = bDrain + 1;
    static constexpr int oMisc = oBars + kNumBars * 8;
    static constexpr int kSmem = oMisc + 16 + 1024;
    static_assert(kSmem <= 227 * 1024, "shared memory of the non-causal token kernel");
};

__device__ int g_nc_status = 0;   // first bounded wait that ran out (0: none)

struct NcMaps {
    CUtensorMap in[3], out[3];
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// offset of the 16-byte piece p of row r in a slot: [row][128 bytes] blocks of 128 rows, swizzled
__device__ __forceinline__ uint32_t slot_piece(int r, int p) {
    return (uint32_t)((p >> 3) * (C * 128) + r * 128 + (((p & 7) ^ (r & 7)) << 4));
}

// steps: forward {E}; backward {dO . E^T, V . dBs^T + dA, pK . dBs}
template <typename Tin, bool kBwd>
__global__ void __launch_bounds__(kNcThreads, 1)
nc_stream_tc(const __grid_constant__ NcMaps maps, const float* __restrict__ totals, const float* __restrict__ de_state,
             int64_t total_chunks, int64_t chunks_per_stream, float eps) {
    using Ly = NcLay<Tin, kBwd>;
    constexpr bool kF32 = sizeof(Tin) == 4;
    constexpr int kSteps = kBwd ? 3 : 1, NS = Ly::kSlots;
    extern __shared__ uint8_t smem_raw[];
    Ctx cx;
    cx.sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    cx.sm_u32 = smem_u32(cx.sm);
    cx.bars = Ly::oBars;
    cx.abort_flag = reinterpret_cast<volatile int*>(cx.sm + Ly::oMisc + 4);
    cx.status = &g_nc_status;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // this CTA's chunks and items
    const int64_t first = total_chunks * blockIdx.x / gridDim.x, last = total_chunks * (blockIdx.x + 1) / gridDim.x;
    const int nitems = (int)(last - first) * kSteps;
    const int64_t n0 = first / chunks_per_stream;

    if (tid == 0) {
        *cx.abort_flag = 0;
        for (int i = 0; i < Ly::kNumBars; ++i)
            mbar_init(cx.bar(i), ((i >= Ly::bOut && i < Ly::bEmpty) || (i >= Ly::bA && i < Ly::bO) ||
                                  (i >= Ly::bMat && i < Ly::bMatFree)) ? 4u : 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(cx.sm_u32 + Ly::oMisc), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(cx.sm + Ly::oMisc);
    // columns of group g: A hi (32) | A lo (32) | result (64)

    if (warp < 4 * kGroups) {
        const int g = warp >> 2, row = 32 * (warp & 3) + lane;
        const uint32_t tm = tmem + 128 * g + ((uint32_t)(32 * (warp & 3)) << 16);
        bool ok = true;
        for (int item = g; item < nitems && ok; item += kGroups) {
            const uint32_t ph = (uint32_t)((item / kGroups) & 1);
            const int slot = item % NS, step = item % kSteps;
            uint8_t* sm = cx.sm + Ly::oSlot + slot * Ly::kSlot;
            if (kF32) {
                if (!(ok = wait_bar_warp(cx, Ly::bFull + slot, (uint32_t)((item / NS) & 1), 101))) break;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        const float4 x = *reinterpret_cast<const float4*>(sm + slot_piece(row, 8 * h + p));
                        split2(x.x, x.y, hi[2 * p], lo[2 * p]);
                        split2(x.z, x.w, hi[2 * p + 1], lo[2 * p + 1]);
                    }
                    tmem_st_words16(tm + 16 * h, hi);
                    tmem_st_words16(tm + 32 + 16 * h, lo);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(cx.bar(Ly::bA + g));
            }
            if (!(ok = wait_bar_warp(cx, Ly::bO + g, ph, 102))) break;
            tc_fence_after();
            const int64_t n = (first + item / kSteps) / chunks_per_stream;
            const float* da = reinterpret_cast<const float*>(cx.sm + Ly::oDa) + ((n - n0) & 3) * 64;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v[32];
                tmem_ld_rows32(tm + 64 + 32 * h, v);
                if (kBwd && step == 1) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float4 b = *reinterpret_cast<const float4*>(da + 32 * h + i);
                        v[i] += b.x; v[i + 1] += b.y; v[i + 2] += b.z; v[i + 3] += b.w;
                    }
                }
                if (kF32) {
#pragma unroll
                    for (int p = 0; p < 8; ++p)
                        *reinterpret_cast<float4*>(sm + slot_piece(row, 8 * h + p)) =
                            make_float4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
                } else {
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            __nv_bfloat162 b2 = __floats2bfloat162_rn(v[8 * p + 2 * i], v[8 * p + 2 * i + 1]);
                            w[i] = *reinterpret_cast<uint32_t*>(&b2);
                        }
                        *reinterpret_cast<uint4*>(sm + slot_piece(row, 4 * h + p)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(Ly::bOut + slot));
        }
    } else if (warp < kLoadWarp) {
        // matrices of the streams of this CTA, one after the other: thread = (bucket row, half of the columns)
        const int s = (tid - 32 * kPrepWarp) >> 1, c0 = 32 * (tid & 1);
        const int64_t n_end = last > first ? (last - 1) / chunks_per_stream : n0 - 1;
        bool ok = true;
        for (int64_t n = n0; n <= n_end && ok; ++n) {
            const int k = (int)(n - n0);
            const float* st = totals + n * (64 * 65);
            const float* de = de_state + n * (64 * 65);
            float4 b[8], d[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                b[i] = __ldg(reinterpret_cast<const float4*>(st + s * 64 + c0) + i);
                if (kBwd) d[i] = __ldg(reinterpret_cast<const float4*>(de + s * 64 + c0) + i);
            }
            const float inv = 1.f / (st[64 * 64 + s] + eps);
            if (k >= 2 && !(ok = wait_bar_warp(cx, Ly::bMatFree + (k & 1), (uint32_t)(((k >> 1) - 1) & 1), 201))) break;
            uint8_t* mat = cx.sm + Ly::oMat + (k & 1) * Ly::kMat;
            auto put = [&](const float4 (&m)[8], int off) {
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    uint4 h, l;
                    split2(m[i].x * inv, m[i].y * inv, h.x, l.x);
                    split2(m[i].z * inv, m[i].w * inv, h.y, l.y);
                    split2(m[i + 1].x * inv, m[i + 1].y * inv, h.z, l.z);
                    split2(m[i + 1].z * inv, m[i + 1].w * inv, h.w, l.w);
                    *reinterpret_cast<uint4*>(mat + off + op_off(s, c0 + 4 * i)) = h;
                    *reinterpret_cast<uint4*>(mat + off + kTile + op_off(s, c0 + 4 * i)) = l;
                }
            };
            put(b, 0);
            if (kBwd) {
                put(d, 2 * kTile);
                float acc = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    acc = fmaf(d[i].x, b[i].x, acc); acc = fmaf(d[i].y, b[i].y, acc);
                    acc = fmaf(d[i].z, b[i].z, acc); acc = fmaf(d[i].w, b[i].w, acc);
                }
                acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                if (c0 == 0) reinterpret_cast<float*>(cx.sm + Ly::oDa)[(k & 3) * 64 + s] = -acc * inv * inv;
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(cx.bar(Ly::bMat + (k & 1)));
        }
    } else if (warp == kLoadWarp) {
        if (lane == 0) {
            int issued = 0;
            int64_t n = n0, ch = first - n0 * chunks_per_stream;
            for (int item = 0, step = 0; item < nitems; ++item) {
                const int slot = item % NS;
                if (item >= NS && !wait_bar(cx, Ly::bEmpty + slot, (uint32_t)((item / NS - 1) & 1), 301)) break;
                mbar_arrive_expect_tx(cx.bar(Ly::bFull + slot), Ly::kSlot);
                tma_load_4d(cx.sm_u32 + Ly::oSlot + slot * Ly::kSlot, &maps.in[step], cx.bar(Ly::bFull + slot), 0, (int)(ch * C), 0,
                            (int)n);
                issued = item + 1;
                if (++step == kSteps) {
                    step = 0;
                    if (++ch == chunks_per_stream) { ch = 0; ++n; }
                }
            }
            if (*cx.abort_flag)   // copies in flight land before the CTA may exit
                for (int item = max(0, issued - NS); item < issued; ++item) {
                    const long long t0 = clock64();
                    while (!mbar_try_wait(cx.bar(Ly::bFull + item % NS), (uint32_t)((item / NS) & 1)) &&
                           clock64() - t0 < (1ll << 24)) {}
                }
        }
    } else if (warp == kMmaWarp) {
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), smb = __shfl_sync(0xffffffffu, cx.sm_u32, 0);
        constexpr uint32_t kId = idesc_mn(C, 64), kLimb = kTile >> 4;
        if (elect_one()) {
            bool ok = true;
            int64_t ch = first - n0 * chunks_per_stream;
            int k = 0, step = 0;      // stream of this CTA
            bool fresh = true;
            for (int item = 0; item < nitems && ok; ++item) {
                const int g = item % kGroups, slot = item % NS;
                if (fresh) {
                    if (!(ok = wait_bar(cx, Ly::bMat + (k & 1), (uint32_t)((k >> 1) & 1), 401))) break;
                    fresh = false;
                }
                if (kF32) {
                    if (!(ok = wait_bar(cx, Ly::bA + g, (uint32_t)((item / kGroups) & 1), 402))) break;
                } else {
                    // the slot is the operand; the group's accumulator has been read once its previous item is stored
                    if (!(ok = wait_bar(cx, Ly::bFull + slot, (uint32_t)((item / NS) & 1), 403))) break;
                    if (item >= kGroups &&
                        !(ok = wait_bar(cx, Ly::bOut + (item - kGroups) % NS, (uint32_t)(((item - kGroups) / NS) & 1), 404))) break;
                }
                tc_fence_after();
                const uint32_t d = tm + 128 * g + 64, mat = smb + Ly::oMat + (k & 1) * Ly::kMat + ((kBwd && step > 0) ? 2 * kTile : 0);
                const bool transposed = kBwd && step < 2;
                auto product = [&](auto tr) {
                    constexpr bool kT = decltype(tr)::value;    // X^T: rows of X are the N index (K-major); X: N-major
                    constexpr uint32_t kHi = kT ? kHiK : kHiMN, kStep = kT ? 16u : 128u, id = kT ? kId : kId | kBmn;
                    const uint32_t b = kT ? lo_k(mat) : lo_mn(mat);
                    if constexpr (kF32) {
                        const uint32_t a = tm + 128 * g;
                        mma_k64_ta<true, kHi, kStep>(d, a, b, id);
                        mma_k64_ta<false, kHi, kStep>(d, a, b + kLimb, id);
                        mma_k64_ta<false, kHi, kStep>(d, a + 32, b, id);
                    } else {
                        const uint32_t a = sw_lo<false, C>(smb + Ly::oSlot + slot * Ly::kSlot);
#pragma unroll
                        for (int l = 0; l < 2; ++l)
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                const uint64_t ad = desc64(kHiSw, a + 2 * kk), bd = desc64(kHi, b + l * kLimb + kk * kStep);
                                if (l == 0 && kk == 0) mma_issue<false>(d, ad, bd, id);
                                else mma_issue<true>(d, ad, bd, id);
                            }
                    }
                };
                if (transposed) product(std::true_type{});
                else product(std::false_type{});
                mma_commit(cx.bar(Ly::bO + g));
                if (++step == kSteps) {
                    step = 0;
                    if (++ch == chunks_per_stream) {
                        ch = 0;
                        mma_commit(cx.bar(Ly::bMatFree + (k & 1)));
                        ++k;
                        fresh = true;
                    }
                }
            }
            mma_commit(cx.bar(Ly::bDrain));
            const long long t0 = clock64();
            while (!mbar_try_wait(cx.bar(Ly::bDrain), 0) && clock64() - t0 < cx.limit) {}
        }
    } else if (warp == kStoreWarp) {
        if (lane == 0) {
            int64_t n = n0, ch = first - n0 * chunks_per_stream;
            for (int item = 0, step = 0; item < nitems; ++item) {
                const int slot = item % NS;
                if (!wait_bar(cx, Ly::bOut + slot, (uint32_t)((item / NS) & 1), 501)) break;
                tma_store_4d(&maps.out[step], cx.sm_u32 + Ly::oSlot + slot * Ly::kSlot, 0, (int)(ch * C), 0, (int)n);
                if (item >= 1) {   // all but the newest store have read their slot
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    mbar_arrive(cx.bar(Ly::bEmpty + (item - 1) % NS));
                }
                if (++step == kSteps) {
                    step = 0;
                    if (++ch == chunks_per_stream) { ch = 0; ++n; }
                }
            }
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// [N][T][64] as (one 128-byte row block of values, T tokens, blocks, N streams); a box is 128 tokens of whole rows
bool nc_map(CUtensorMap* map, const void* base, const Dims& dm, int dtype) {
    auto fn = tensor_map_encoder();
    if (!fn) return false;
    const bool f32 = dtype == RACE_DTYPE_F32;
    const cuuint64_t eb = f32 ? 4 : 2, per = 128 / eb;
    cuuint64_t dims[4] = {per, (cuuint64_t)dm.T, 64 / per, (cuuint64_t)dm.N};
    cuuint64_t strides[3] = {64 * eb, 128, (cuuint64_t)dm.T * 64 * eb};
    cuuint32_t box[4] = {(cuuint32_t)per, (cuuint32_t)C, (cuuint32_t)(64 / per), 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename Tin, bool kBwd>
cudaError_t launch_nc(const NcMaps& maps, const float* totals, const float* de_state, const Dims& dm, int sm_count,
                      cudaStream_t stream) {
    auto kern = nc_stream_tc<Tin, kBwd>;
    constexpr int smem = NcLay<Tin, kBwd>::kSmem;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    const int64_t per_stream = (dm.T + C - 1) / C, total = dm.N * per_stream;
    const unsigned grid = (unsigned)std::min<int64_t>(total, sm_count > 0 ? sm_count : 148);
    kern<<<grid, kNcThreads, smem, stream>>>(maps, totals, de_state, total, per_stream, dm.eps);
    return cudaGetLastError();
}

}  // namespace

bool noncausal_tensor_supported(const Dims& dm, int dtype) {
    return (dtype == RACE_DTYPE_F32 || dtype == RACE_DTYPE_BF16) && dm.S == 64 && dm.D == 64 && dm.N <= 65535 &&
           dm.T < (1ll << 31) - C;
}

cudaError_t noncausal_query_tensor(const void* pq, const float* totals, void* out, const Dims& dm, int dtype,
                                   int sm_count, cudaStream_t stream) {
    NcMaps m{};
    if (!nc_map(&m.in[0], pq, dm, dtype) || !nc_map(&m.out[0], out, dm, dtype)) return cudaErrorInvalidValue;
    return dtype == RACE_DTYPE_F32 ? launch_nc<float, false>(m, totals, totals, dm, sm_count, stream)
                                   : launch_nc<__nv_bfloat16, false>(m, totals, totals, dm, sm_count, stream);
}

cudaError_t noncausal_token_grads_tensor(const void* pk, const void* v, const void* dout, const float* totals,
                                         const float* de_state, void* dpq, void* dpk, void* dv, const Dims& dm,
                                         int dtype, int sm_count, cudaStream_t stream) {
    NcMaps m{};
    const void* in[3] = {dout, v, pk};      // dPQ = dO . E^T;  dPK = V . dBs^T + dA;  dV = pK . dBs
    void* out[3] = {dpq, dpk, dv};
    for (int i = 0; i < 3; ++i)
        if (!nc_map(&m.in[i], in[i], dm, dtype) || !nc_map(&m.out[i], out[i], dm, dtype)) return cudaErrorInvalidValue;
    return dtype == RACE_DTYPE_F32 ? launch_nc<float, true>(m, totals, de_state, dm, sm_count, stream)
                                   : launch_nc<__nv_bfloat16, true>(m, totals, de_state, dm, sm_count, stream);
}

}  // namespace race
