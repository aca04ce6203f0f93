// Shared device/host helpers of the RACE prefix-path kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/race_b200.h"

namespace race {

// Problem sizes every kernel receives by value.
struct Dims {
    int64_t N;  // streams
    int64_t T;  // tokens per stream
    int S;      // L*R bucket features per token
    int D;      // head dim
    float eps;
    int H = 1;  // heads of the V / out layout: [N/H, T, H, D] (1: the plain [N, T, D])
};

constexpr int kSimtThreads = 256;
constexpr int kSimtChunk = 32;    // tokens per chunk of the CUDA-core kernels
constexpr int kGroupBuckets = 64; // buckets one CTA owns; wider S is split over a cluster

__host__ __device__ inline int state_floats_per_stream(int S, int D) { return S * (D + 1); }

// Launches of one call are chained (programmatic dependent launch, launch_chain in launch.h): a kernel lets its
// successor start while it still runs (chain_release, at its start), and the successor sets itself up and waits, in
// every thread, for everything before it (chain_wait) ahead of its first access to global memory.  For calls of a few microseconds the
// gaps between launches are a third of the time.
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads of a chained kernel.  What it reads may have been written while it was already resident, so it must not go through
// the read-only path (__ldg, or a plain load of a const __restrict__ parameter: both promise that the data does not change
// while the grid lives), and the compiler must not move it ahead of chain_wait.
enum LdPolicy { kLdCached, kLdL2, kLdOnce };   // ld.global, .cg (L2 only), .cs (streamed)
#define RACE_LD_CHAIN(T, SUFFIX, OUT, ...)                                                                             \
    template <LdPolicy kPolicy = kLdCached>                                                                            \
    __device__ __forceinline__ T ld_chain(const T* p) {                                                                \
        T v;                                                                                                           \
        if (kPolicy == kLdOnce) asm volatile("ld.global.cs." SUFFIX " " OUT ";" : __VA_ARGS__ : "l"(p) : "memory");    \
        else if (kPolicy == kLdL2) asm volatile("ld.global.cg." SUFFIX " " OUT ";" : __VA_ARGS__ : "l"(p) : "memory"); \
        else asm volatile("ld.global." SUFFIX " " OUT ";" : __VA_ARGS__ : "l"(p) : "memory");                          \
        return v;                                                                                                      \
    }
RACE_LD_CHAIN(float, "f32", "%0, [%1]", "=f"(v))
RACE_LD_CHAIN(float2, "v2.f32", "{%0, %1}, [%2]", "=f"(v.x), "=f"(v.y))
RACE_LD_CHAIN(float4, "v4.f32", "{%0, %1, %2, %3}, [%4]", "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w))
RACE_LD_CHAIN(uint4, "v4.u32", "{%0, %1, %2, %3}, [%4]", "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w))
#undef RACE_LD_CHAIN

// The state a tile starts from, formed by the output kernel itself (fold): carry_in + the totals of the tiles before it,
// added tile by tile in the order tile_scan adds them, so both routes give the same bits.  Not folded: the slot of the
// tile already holds that prefix (tile_scan).  The CTA of the last tile also writes the state after the sequence.
struct CarryFold {
    const float* carry_in;    // [N][state] or null (zeros)
    float* state_out;         // [N][state] or null
    int fold;
};

// Threads 0 .. NT-1 of the CTA: prefix of `cnt` tiles at p, p + step, ... (4 floats per thread and column, up to three
// columns and six tiles in flight: the loads are L2 latencies, a column at a time they were a chain of them).
// b_floats: floats of the B part, which goes to sb; the A part goes to sa.
template <int NT>
__device__ __forceinline__ void fold_prefix(const float* p, int64_t step, int cnt, const float* carry, float* state_out,
                                            float* sb, float* sa, int b_floats, int state_floats, int tid) {
    constexpr int kCols = 3, kTiles = 6;
    for (int base = 4 * tid; base < state_floats; base += 4 * NT * kCols) {
        float4 run[kCols];
#pragma unroll
        for (int u = 0; u < kCols; ++u) {
            const int i = base + 4 * NT * u;
            run[u] = carry && i < state_floats ? ld_chain<kLdL2>(reinterpret_cast<const float4*>(carry + i))
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int t = 0; t < cnt; t += kTiles) {
            float4 x[kTiles][kCols];
#pragma unroll
            for (int j = 0; j < kTiles; ++j)
#pragma unroll
                for (int u = 0; u < kCols; ++u) {
                    const int i = base + 4 * NT * u;
                    x[j][u] = t + j < cnt && i < state_floats
                                  ? ld_chain<kLdL2>(reinterpret_cast<const float4*>(p + (t + j) * step + i))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
            for (int j = 0; j < kTiles; ++j)
                if (t + j < cnt)
#pragma unroll
                    for (int u = 0; u < kCols; ++u) {
                        run[u].x += x[j][u].x; run[u].y += x[j][u].y; run[u].z += x[j][u].z; run[u].w += x[j][u].w;
                    }
        }
#pragma unroll
        for (int u = 0; u < kCols; ++u) {
            const int i = base + 4 * NT * u;
            if (i >= state_floats) continue;
            *reinterpret_cast<float4*>(i < b_floats ? sb + i : sa + (i - b_floats)) = run[u];
            if (state_out) {
                const float4 x = ld_chain<kLdL2>(reinterpret_cast<const float4*>(p + cnt * step + i));
                *reinterpret_cast<float4*>(state_out + i) =
                    make_float4(run[u].x + x.x, run[u].y + x.y, run[u].z + x.z, run[u].w + x.w);
            }
        }
    }
}

// ---- element access: 4 consecutive elements as float4 -------------------------------------
__device__ __forceinline__ float4 load4(const float* p) {
    return *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    uint2 raw = *reinterpret_cast<const uint2*>(p);
    __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&raw.x);
    __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&raw.y);
    float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
}
// streaming (read-once) variants
__device__ __forceinline__ float4 load4_stream(const float* p) {
    return __ldcs(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ float4 load4_stream(const __nv_bfloat16* p) {
    uint2 raw = __ldcs(reinterpret_cast<const uint2*>(p));
    __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&raw.x);
    __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&raw.y);
    float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
}
__device__ __forceinline__ void store4_stream(float* p, float4 x) {
    __stcs(reinterpret_cast<float4*>(p), x);
}
__device__ __forceinline__ void store4_stream(__nv_bfloat16* p, float4 x) {
    __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y);
    __nv_bfloat162 b = __floats2bfloat162_rn(x.z, x.w);
    uint2 raw;
    raw.x = *reinterpret_cast<uint32_t*>(&a);
    raw.y = *reinterpret_cast<uint32_t*>(&b);
    __stcs(reinterpret_cast<uint2*>(p), raw);
}

// Copy a [rows x cols_pad] block into shared memory (row stride ld floats) from a row-major
// global matrix of row length `width`: rows [row0, row0+rows_valid) and columns
// [col0, col0+cols_valid); everything else is zero-filled (padded tokens must read as pK = 0
// and a finite V so that they add nothing to the running sums).  cols_* are multiples of 4.
template <typename Tin>
__device__ __forceinline__ void stage_block(float* dst, int ld, const Tin* src, int64_t row0,
                                            int rows, int rows_valid, int width, int col0,
                                            int cols_pad, int cols_valid, int tid, int nthreads) {
    const int vec_per_row = cols_pad >> 2;
    const int total = rows * vec_per_row;
    for (int i = tid; i < total; i += nthreads) {
        const int r = i / vec_per_row;
        const int c = (i - r * vec_per_row) << 2;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows_valid && c < cols_valid)
            x = load4_stream(src + (row0 + r) * (int64_t)width + col0 + c);
        *reinterpret_cast<float4*>(dst + r * ld + c) = x;
    }
}

}  // namespace race
