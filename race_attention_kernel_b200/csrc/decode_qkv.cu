// Incremental step of the operator from K, V, Q and the hyperplanes: the bucket probabilities of the new tokens
// (src/race_baseline.py:41-44) and the state update of the chunked evaluation (src/race_chunked.py:54-63) in one
// launch, with K, V, Q and out in the operator's layout [outer, T, heads, d_k].
//
// The work is one read and one write of the state (4 S (d_k + 1) bytes each per stream), everything else is small, so
// what counts is (a) one launch instead of three with the probabilities and a flattened V between them in memory, and
// (b) that the state is requested before anything else: a thread holds its whole share of B in registers (SC / 4 ..
// rows of a column quad) while the projections, probabilities and W of the token are formed.
// A CTA owns SC buckets of one stream: all 64 of the small geometry; 128 of the 512 (two tables) of the wide one, whose
// four CTAs form a thread-block cluster and add their shares of the output through distributed shared memory.
// Projections: eight threads per (row, plane), fp32 FMAs.
#include <cooperative_groups.h>

#include "common.cuh"
#include "launch.h"
#include "probs_frag.cuh"

namespace cg = cooperative_groups;

namespace race {
namespace {

constexpr int kThreads = 256;

template <int D_, int L_, int K_, int SC_>
struct StepGeo {
    static constexpr int D = D_, L = L_, K = K_, SC = SC_, R = 1 << K, S = L * R, G = S / SC;   // G: CTAs per stream
    static constexpr int TPC = SC / R, PPC = TPC * K;        // tables, planes per CTA
    static constexpr int QUADS = D / 4, RPP = kThreads / QUADS, NP = SC / RPP;   // rows per pass, passes
    static constexpr int EPT = D / 8;                        // elements of a dot product per thread
    static_assert(2 * PPC * 8 <= kThreads && 2 * SC <= kThreads && 32 % QUADS == 0, "thread roles of the step");
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
}

// grid (G, N), clusters of G.  state_in may be null (zeros) and may equal state_out: every float is read and written by
// the same thread, A by the CTA that owns its buckets.
template <typename Geo, typename Tin>
__global__ void __launch_bounds__(kThreads, Geo::NP <= 4 ? 5 : 2)
decode_step_qkv(const Tin* __restrict__ k, const Tin* __restrict__ v, const Tin* __restrict__ q,
                const float* __restrict__ planes, Tin* __restrict__ out, const float* state_in, float* state_out, int T,
                int heads, float eps) {
    constexpr int D = Geo::D, K = Geo::K, SC = Geo::SC, R = Geo::R, S = Geo::S, G = Geo::G;
    extern __shared__ __align__(16) float sm[];
    __shared__ float sp1[2][Geo::PPC];          // p1 of every plane: row 0 = K, row 1 = Q
    __shared__ float spk[SC], spq[SC], sw[SC];
    __shared__ __align__(16) float red[kThreads / 32][D];
    float* part = sm;                           // [G][T][D] (rank 0): the CTAs' shares of the outputs, G > 1
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x;
    const int64_t n = blockIdx.y;
    const int64_t row_step = (int64_t)heads * D;                                    // one token further
    const int64_t tok0 = ((n / heads) * T * heads + n % heads) * D;                 // token 0 of the stream
    const int64_t sbase = n * (int64_t)(S * (D + 1));
    const int col = (tid % Geo::QUADS) * 4, row = tid / Geo::QUADS;
    if constexpr (G > 1) cg::this_cluster().barrier_arrive();   // every CTA of the cluster runs before the first remote write
    const int64_t boff = sbase + (int64_t)(rank * SC + row) * D + col;

    float4 b[Geo::NP];
#pragma unroll
    for (int i = 0; i < Geo::NP; ++i)
        b[i] = state_in ? __ldcs(reinterpret_cast<const float4*>(state_in + boff + (int64_t)i * Geo::RPP * D))
                        : make_float4(0.f, 0.f, 0.f, 0.f);
    float a = (tid < SC && state_in) ? state_in[sbase + (int64_t)S * D + rank * SC + tid] : 0.f;

    // dot product of this thread's group of eight: (row of K or Q, plane of the CTA)
    const int grp = tid >> 3, e0 = (tid & 7) * 4;
    const bool dot = grp < 2 * Geo::PPC;
    const Tin* xrow = ((grp & 1) ? q : k) + tok0 + e0;
    float4 pl[Geo::EPT / 4];
    if (dot) {
        const float* prow = planes + (int64_t)(rank * Geo::PPC + (grp >> 1)) * D + e0;
#pragma unroll
        for (int i = 0; i < Geo::EPT / 4; ++i) pl[i] = ld4(prow + 32 * i);
    }
    for (int t = 0; t < T; ++t) {
        const float4 vv = ld4(v + tok0 + t * row_step + col);
        if (dot) {
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < Geo::EPT / 4; ++i) {
                const float4 x = ld4(xrow + t * row_step + 32 * i);
                s = fmaf(x.x, pl[i].x, s); s = fmaf(x.y, pl[i].y, s); s = fmaf(x.z, pl[i].z, s); s = fmaf(x.w, pl[i].w, s);
            }
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            if ((tid & 7) == 0) {
                const float th = fast_tanh(s) * rsqrtf((float)D), sq = th * th;   // |th| <= 1/8, as soft_bits8
                sp1[grp & 1][grp >> 1] =
                    0.5f + 0.5f * th * fmaf(sq, fmaf(sq, fmaf(sq, -17.f / 315.f, 2.f / 15.f), -1.f / 3.f), 1.f);
            }
        }
        __syncthreads();
        if (tid < 2 * SC) {
            const int which = tid / SC, s = tid % SC, table = s / R, r = s % R;
            float p = 1.f;
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const float p1 = sp1[which][table * K + j];
                p *= ((r >> (K - 1 - j)) & 1) ? p1 : 1.f - p1;
            }
            (which ? spq : spk)[s] = p;
        }
        __syncthreads();
        if (tid < SC) {
            a += spk[tid];
            sw[tid] = spq[tid] / (a + eps);
        }
        __syncthreads();
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < Geo::NP; ++i) {
            const float pk = spk[row + i * Geo::RPP], w = sw[row + i * Geo::RPP];
            b[i].x = fmaf(pk, vv.x, b[i].x); b[i].y = fmaf(pk, vv.y, b[i].y);
            b[i].z = fmaf(pk, vv.z, b[i].z); b[i].w = fmaf(pk, vv.w, b[i].w);
            acc.x = fmaf(w, b[i].x, acc.x); acc.y = fmaf(w, b[i].y, acc.y);
            acc.z = fmaf(w, b[i].z, acc.z); acc.w = fmaf(w, b[i].w, acc.w);
        }
        if (t == T - 1) {
#pragma unroll
            for (int i = 0; i < Geo::NP; ++i)
                __stcs(reinterpret_cast<float4*>(state_out + boff + (int64_t)i * Geo::RPP * D), b[i]);
            if (tid < SC) state_out[sbase + (int64_t)S * D + rank * SC + tid] = a;
        }
        // lanes with the same column quad, then the warps (and, with G > 1, the CTAs of the stream)
#pragma unroll
        for (int off = Geo::QUADS; off < 32; off <<= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
            acc.z += __shfl_xor_sync(0xffffffffu, acc.z, off);
            acc.w += __shfl_xor_sync(0xffffffffu, acc.w, off);
        }
        if (lane < Geo::QUADS) *reinterpret_cast<float4*>(&red[warp][col]) = acc;
        if (G > 1 && t == 0) cg::this_cluster().barrier_wait();
        __syncthreads();
        if (tid < D) {
            float o = 0.f;
#pragma unroll
            for (int i = 0; i < kThreads / 32; ++i) o += red[i][tid];
            if constexpr (G == 1) {
                out[tok0 + t * row_step + tid] = (Tin)o;
            } else {
                float* dst = cg::this_cluster().map_shared_rank(part, 0);
                dst[(rank * T + t) * D + tid] = o;
            }
        }
    }
    if constexpr (G > 1) {
        cg::this_cluster().sync();
        if (rank == 0)
            for (int i = tid; i < T * D; i += kThreads) {
                float o = 0.f;
#pragma unroll
                for (int g = 0; g < G; ++g) o += part[g * T * D + i];
                out[tok0 + (i / D) * row_step + i % D] = (Tin)o;
            }
    }
}

template <typename Geo, typename Tin>
cudaError_t launch_step(const void* k, const void* v, const void* q, const float* planes, void* out,
                        const float* state_in, float* state_out, int64_t N, int T, int heads, float eps,
                        cudaStream_t stream) {
    const size_t smem = Geo::G > 1 ? (size_t)Geo::G * T * Geo::D * sizeof(float) : 0;
    auto kern = decode_step_qkv<Geo, Tin>;
    if (Geo::G > 1) {
        // the attribute belongs to the process: always the most any call needs, or two threads with steps of different
        // lengths take it from each other between setting it and launching
        cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               Geo::G * decode_max_tokens() * Geo::D * (int)sizeof(float));
        if (err != cudaSuccess) return err;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(Geo::G, (unsigned)N);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = Geo::G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = Geo::G > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, (const Tin*)k, (const Tin*)v, (const Tin*)q, planes, (Tin*)out, state_in,
                              state_out, T, heads, eps);
}

}  // namespace

bool decode_qkv_supported(int64_t N, int64_t T, int d, int L, int K, int dtype) {
    return N >= 0 && N <= 65535 && T >= 0 && T <= decode_max_tokens() &&
           (dtype == RACE_DTYPE_F32 || dtype == RACE_DTYPE_BF16) &&
           ((d == 64 && L == 4 && K == 4) || (d == 128 && L == 8 && K == 6));
}

cudaError_t decode_step_qkv_launch(const void* k, const void* v, const void* q, const float* planes, void* out,
                                   const float* state_in, float* state_out, int64_t N, int T, int heads, int d,
                                   int dtype, float eps, cudaStream_t stream) {
    using Small = StepGeo<64, 4, 4, 64>;
    using Wide = StepGeo<128, 8, 6, 128>;
    if (d == 64)
        return dtype == RACE_DTYPE_F32
                   ? launch_step<Small, float>(k, v, q, planes, out, state_in, state_out, N, T, heads, eps, stream)
                   : launch_step<Small, __nv_bfloat16>(k, v, q, planes, out, state_in, state_out, N, T, heads, eps, stream);
    return dtype == RACE_DTYPE_F32
               ? launch_step<Wide, float>(k, v, q, planes, out, state_in, state_out, N, T, heads, eps, stream)
               : launch_step<Wide, __nv_bfloat16>(k, v, q, planes, out, state_in, state_out, N, T, heads, eps, stream);
}

}  // namespace race
