// Backward of the bucket-probability producer (the derivative of src/race_baseline.py:41-44): from the rows x, the
// hyperplanes and the gradient of the probabilities, the gradient of x.
//   proj = x . planes^T;  th = tanh(proj);  p1 = sigmoid(2 th / sqrt(d)) per plane, p0 = 1 - p1
//   probs[l][r] = product over the K planes of p_{bit}(l, k)
//   D[l,k]   = d L / d p1[l,k] = sum over the other planes' bits of their probability x (dP[bit k = 1] - dP[bit k = 0])
//   dproj    = D . 2 p0 p1 . (1 - th^2) / sqrt(d);      dx = dproj . planes
// D is evaluated from the last plane to the first: the 2^(k+1) values left are paired, their differences are contracted
// with the probabilities of the planes before k to D[k], and the pairs are replaced by their expectation.  Differences
// are taken first, so the common part of dP, which the softmax cancels, does not cost precision.
//
// A warp takes 16 rows at a time and nothing but x, dP and dx crosses memory.  Both contractions ([16 x D] . [D x L K]
// and [16 x L K] . [L K x D]) run on mma.sync m16n8k16 with bf16 limbs and fp32 accumulation: bf16 rows of x are exact in
// one limb, against hi/lo limbs of the planes and of dproj; fp32 rows, their planes and dproj take three limbs and every
// k-step an accumulator of its own (six_products), since nothing rounds the result afterwards and the factor 1 - th^2 =
// 4 e^(-2 |proj|) / .. turns an absolute error of proj (3e-5 with two limbs) into twice that relative error of dx.  The
// index permutations of the forward kernel (bucket_probs_mma_wide) put the K planes of whole tables into one lane of a quad,
// and the accumulators of the first product are, lane by lane, the A fragments of the second; its columns are permuted so
// that a lane ends up with eight consecutive features of its two rows.
// Bound by memory (x, dP in, dx out) at d_k = 64, by the 240 mma.sync per 16 rows at d_k = 128, L = 8, K = 6.
#include <algorithm>

#include "common.cuh"
#include "launch.h"
#include "probs_frag.cuh"

namespace race {
namespace {

constexpr int kBwdThreads = 128;

template <int D, int L, int K>
struct BwdProbs {
    static constexpr int NT = L * K / 8, NJ = D / 16, R = 1 << K, TPL = L / 4, NS = 2 * NT;   // NS plane slots per lane
    static constexpr int KS = NS / 4, NB = D / 8;                                            // second product
    static constexpr int kTab1 = NT * NJ * 32, kTab2 = NB * KS * 32;                         // 16-byte items
    static constexpr int smem_bytes(bool x32) { return (kTab1 + kTab2) * (16 + (x32 ? 8 : 0)); }
    static constexpr int kCtas = D == 64 ? 5 : 3;   // resident CTAs per SM (registers)
    static_assert(D % 32 == 0 && L % 4 == 0 && (L * K) % 16 == 0, "geometry of the tensor-core producer");
    // plane of slot s of lane t of a quad
    static __device__ __forceinline__ int plane(int t, int s) { return (TPL * t + s / K) * K + s % K; }
};

// gradient of the probabilities of one (row, table): R consecutive values
template <int R>
__device__ __forceinline__ void load_dp(const float* p, float (&v)[R]) {
#pragma unroll
    for (int i = 0; i < R; i += 4) {
        const float4 x = ld_chain(reinterpret_cast<const float4*>(p + i));
        v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
    }
}
template <int R>
__device__ __forceinline__ void load_dp(const __nv_bfloat16* p, float (&v)[R]) {
#pragma unroll
    for (int i = 0; i < R; i += 8) {
        const uint4 x = ld_chain(reinterpret_cast<const uint4*>(p + i));
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[i + 2 * j] = __uint_as_float(w[j] << 16);
            v[i + 2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
        }
    }
}

// c += a . b over one k-step with three limbs of both (b = {b0 hi, b1 hi, b0 lo, b1 lo}, r = the third limbs): an accumulator of
// its own, small products first, added to c with rounding.  The tensor core rounds its additions down, and in one chain over
// all k-steps that is a bias of the size of the projections (d_k = 128: 11): dK and dQ 4.3e-6 off the 64-bit result, where
// fp32 FMAs are 1.3e-6 off.
__device__ __forceinline__ void six_products(float (&c)[4], const uint32_t (&hi)[4], const uint32_t (&lo)[4],
                                             const uint32_t (&rest)[4], const uint4& b, const uint2& r) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16_16816(s, rest, b.x, b.y);
    mma_bf16_16816(s, lo, b.z, b.w);
    mma_bf16_16816(s, hi, r.x, r.y);
    mma_bf16_16816(s, lo, b.x, b.y);
    mma_bf16_16816(s, hi, b.z, b.w);
    mma_bf16_16816(s, hi, b.x, b.y);
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += s[i];
}

template <int D, int L, int K, typename Tx, typename Tp>
__global__ void __launch_bounds__(kBwdThreads, BwdProbs<D, L, K>::kCtas)
bucket_probs_bwd_mma(const Tx* x0, const Tx* x1, const float* planes,
                     const Tp* dprobs0, const Tp* dprobs1, Tx* __restrict__ dx0,
                     Tx* __restrict__ dx1, int64_t rows, int64_t T, int heads) {
    const Tx* x = blockIdx.y ? x1 : x0;   // two tensors (K and Q): one launch, the halves of its grid
    const Tp* dprobs = blockIdx.y ? dprobs1 : dprobs0;
    Tx* __restrict__ dx = blockIdx.y ? dx1 : dx0;
    using W = BwdProbs<D, L, K>;
    constexpr int NT = W::NT, NJ = W::NJ, R = W::R, TPL = W::TPL, KS = W::KS;
    constexpr bool kX32 = sizeof(Tx) == 4;
    extern __shared__ __align__(16) uint8_t bwd_smem[];
    uint4* tab1 = reinterpret_cast<uint4*>(bwd_smem);          // [(nt NJ + j) 32 + lane] = {b0 hi, b1 hi, b0 lo, b1 lo}
    uint4* tab2 = tab1 + W::kTab1;                             // [(nb KS + j) 32 + lane]
    uint2* tab1r = reinterpret_cast<uint2*>(tab2 + W::kTab2);   // fp32 rows: third limbs {b0, b1} of tab1 ...
    uint2* tab2r = tab1r + W::kTab1;                            // ... and of tab2
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    chain_release();
    chain_wait();
    for (int i = threadIdx.x; i < W::kTab1; i += kBwdThreads) {
        const int ln = i & 31, f = i >> 5, j = f % NJ, nt = f / NJ;
        const int fg = ln >> 2, ft = ln & 3;
        const float* src = planes + (int64_t)W::plane(fg >> 1, 2 * nt + (fg & 1)) * D + 32 * (j >> 1) + 8 * ft + 4 * (j & 1);
        const float4 v = ld_chain(reinterpret_cast<const float4*>(src));
        uint4 w;
        split_pair(v.x, v.y, w.x, w.z);
        split_pair(v.z, v.w, w.y, w.w);
        tab1[i] = w;
        if (kX32) tab1r[i] = make_uint2(rest_pair(v.x, v.y, w.x, w.z), rest_pair(v.z, v.w, w.y, w.w));
    }
    for (int i = threadIdx.x; i < W::kTab2; i += kBwdThreads) {
        const int ln = i & 31, f = i >> 5, j = f % KS, nb = f / KS;
        const int fg = ln >> 2, ft = ln & 3;
        const int feat = 32 * (nb >> 2) + 8 * (fg >> 1) + 2 * (nb & 3) + (fg & 1);   // column fg of block nb
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = ld_chain(planes + (int64_t)W::plane(ft, 4 * j + e) * D + feat);
        uint4 w;
        split_pair(v[0], v[1], w.x, w.z);
        split_pair(v[2], v[3], w.y, w.w);
        tab2[i] = w;
        if (kX32) tab2r[i] = make_uint2(rest_pair(v[0], v[1], w.x, w.z), rest_pair(v[2], v[3], w.y, w.w));
    }
    __syncthreads();
    const float inv_scale = rsqrtf((float)D);
    const int64_t blocks = (rows + 15) / 16;
    const int64_t warp_global = (int64_t)blockIdx.x * (kBwdThreads / 32) + (threadIdx.x >> 5);
    const int64_t warps_total = (int64_t)gridDim.x * (kBwdThreads / 32);
    for (int64_t blk = warp_global; blk < blocks; blk += warps_total) {
        const int64_t r0 = blk * 16;
        bool live[2];
        int64_t off[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t row = r0 + g + 8 * h;
            live[h] = row < rows;
            const int64_t rr = live[h] ? row : 0;
            const int64_t n = rr / T, tok = rr - n * T;
            const int64_t mb = n / heads, hd = n - mb * heads;
            off[h] = ((mb * T + tok) * heads + hd) * D + 8 * t;
        }
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
#pragma unroll
        for (int m = 0; m < D / 32; ++m) {
            uint32_t hi[2][4], lo[2][4], rest[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if constexpr (kX32) {
                    float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
                    if (live[h]) {
                        v0 = ld_chain<kLdOnce>(reinterpret_cast<const float4*>(x + off[h] + 32 * m));
                        v1 = ld_chain<kLdOnce>(reinterpret_cast<const float4*>(x + off[h] + 32 * m) + 1);
                    }
                    split_pair(v0.x, v0.y, hi[h][0], lo[h][0]);
                    split_pair(v0.z, v0.w, hi[h][1], lo[h][1]);
                    split_pair(v1.x, v1.y, hi[h][2], lo[h][2]);
                    split_pair(v1.z, v1.w, hi[h][3], lo[h][3]);
                    rest[h][0] = rest_pair(v0.x, v0.y, hi[h][0], lo[h][0]);
                    rest[h][1] = rest_pair(v0.z, v0.w, hi[h][1], lo[h][1]);
                    rest[h][2] = rest_pair(v1.x, v1.y, hi[h][2], lo[h][2]);
                    rest[h][3] = rest_pair(v1.z, v1.w, hi[h][3], lo[h][3]);
                } else {
                    uint4 v = make_uint4(0u, 0u, 0u, 0u);
                    if (live[h]) v = ld_chain<kLdOnce>(reinterpret_cast<const uint4*>(x + off[h] + 32 * m));
                    hi[h][0] = v.x; hi[h][1] = v.y; hi[h][2] = v.z; hi[h][3] = v.w;
                }
            }
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
                const int j = 2 * m + jj;
                const uint32_t ahi[4] = {hi[0][2 * jj], hi[1][2 * jj], hi[0][2 * jj + 1], hi[1][2 * jj + 1]};
                uint32_t alo[4], ar[4];
                if constexpr (kX32) {
                    alo[0] = lo[0][2 * jj]; alo[1] = lo[1][2 * jj]; alo[2] = lo[0][2 * jj + 1]; alo[3] = lo[1][2 * jj + 1];
                    ar[0] = rest[0][2 * jj]; ar[1] = rest[1][2 * jj]; ar[2] = rest[0][2 * jj + 1]; ar[3] = rest[1][2 * jj + 1];
                }
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint4 b = tab1[(nt * NJ + j) * 32 + lane];
                    if constexpr (kX32) {
                        const uint2 r = tab1r[(nt * NJ + j) * 32 + lane];
                        six_products(acc[nt], ahi, alo, ar, b, r);
                    } else {
                        mma_bf16_16816(acc[nt], ahi, b.z, b.w);
                        mma_bf16_16816(acc[nt], ahi, b.x, b.y);
                    }
                }
            }
        }
        // gradient of the projections of the lane's (row, table) pairs, in place of the projections
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int tb = 0; tb < TPL; ++tb) {
                float v[R];
                if (live[h]) {
                    load_dp<R>(dprobs + ((r0 + g + 8 * h) * L + TPL * t + tb) * R, v);
                } else {
#pragma unroll
                    for (int i = 0; i < R; ++i) v[i] = 0.f;
                }
                float p1[K], scale[K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const int s = tb * K + k;
                    const float pr = acc[s >> 1][2 * h + (s & 1)];
                    const float e = __expf(-2.f * fabsf(pr));
                    const float r1 = __fdividef(1.f, 1.f + e);
                    const float th = copysignf((1.f - e) * r1, pr) * inv_scale;
                    const float sq = th * th;    // |th| <= 1/sqrt(d_k): the odd polynomial of tanh to th^7
                    const float half = 0.5f * th * fmaf(sq, fmaf(sq, fmaf(sq, -17.f / 315.f, 2.f / 15.f), -1.f / 3.f), 1.f);
                    p1[k] = 0.5f + half;
                    // 2 p0 p1 (1 - tanh^2) / sqrt(d); 1 - tanh^2 = 4 e / (1 + e)^2
                    scale[k] = 2.f * (0.25f - half * half) * (4.f * e * r1 * r1) * inv_scale;
                }
#pragma unroll
                for (int k = K - 1; k >= 0; --k) {
                    float d[R / 2];
#pragma unroll
                    for (int i = 0; i < R / 2; ++i)
                        if (i < (1 << k)) {
                            d[i] = v[2 * i + 1] - v[2 * i];
                            v[i] = fmaf(p1[k], d[i], v[2 * i]);
                        }
#pragma unroll
                    for (int kk = K - 2; kk >= 0; --kk)
                        if (kk < k) {
#pragma unroll
                            for (int i = 0; i < R / 4; ++i)
                                if (i < (1 << kk)) d[i] = fmaf(p1[kk], d[2 * i + 1] - d[2 * i], d[2 * i]);
                        }
                    const int s = tb * K + k;
                    acc[s >> 1][2 * h + (s & 1)] = d[0] * scale[k];
                }
            }
        }
        // A fragments of the second product: slots 4 j .. 4 j + 3 of both rows
        uint32_t ahi[KS][4], alo[KS][4], ar[KS][4];
#pragma unroll
        for (int j = 0; j < KS; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int nt = 2 * j + (i >> 1), h = i & 1;
                split_pair(acc[nt][2 * h], acc[nt][2 * h + 1], ahi[j][i], alo[j][i]);
                if (kX32) ar[j][i] = rest_pair(acc[nt][2 * h], acc[nt][2 * h + 1], ahi[j][i], alo[j][i]);
            }
#pragma unroll
        for (int m = 0; m < D / 32; ++m) {
            float o[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
#pragma unroll
                for (int j = 0; j < KS; ++j) {
                    const uint4 b = tab2[((4 * m + i) * KS + j) * 32 + lane];
                    if constexpr (kX32) {
                        const uint2 r = tab2r[((4 * m + i) * KS + j) * 32 + lane];
                        six_products(o[i], ahi[j], alo[j], ar[j], b, r);
                    } else {
                        mma_bf16_16816(o[i], ahi[j], b.z, b.w);
                        mma_bf16_16816(o[i], alo[j], b.x, b.y);
                        mma_bf16_16816(o[i], ahi[j], b.x, b.y);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!live[h]) continue;
                Tx* dst = dx + off[h] + 32 * m;
                if constexpr (kX32) {
                    __stcs(reinterpret_cast<float4*>(dst), make_float4(o[0][2 * h], o[0][2 * h + 1], o[1][2 * h], o[1][2 * h + 1]));
                    __stcs(reinterpret_cast<float4*>(dst) + 1, make_float4(o[2][2 * h], o[2][2 * h + 1], o[3][2 * h], o[3][2 * h + 1]));
                } else {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        __nv_bfloat162 b2 = __floats2bfloat162_rn(o[i][2 * h], o[i][2 * h + 1]);
                        w[i] = *reinterpret_cast<uint32_t*>(&b2);
                    }
                    __stcs(reinterpret_cast<uint4*>(dst), make_uint4(w[0], w[1], w[2], w[3]));
                }
            }
        }
    }
}

template <int D, int L, int K, typename Tx, typename Tp>
cudaError_t launch_probs_bwd(const void* x, const void* x1, const float* planes, const void* dprobs, const void* dprobs1,
                             void* dx, void* dx1, int64_t rows, int64_t T, int heads, cudaStream_t stream) {
    auto kern = bucket_probs_bwd_mma<D, L, K, Tx, Tp>;
    constexpr int smem = BwdProbs<D, L, K>::smem_bytes(sizeof(Tx) == 4);
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // the plane tables are built once per CTA: the resident CTAs walk the rows
    const int64_t resident = (int64_t)(sms > 0 ? sms : 148) * BwdProbs<D, L, K>::kCtas / (x1 ? 2 : 1);
    const dim3 grid((unsigned)std::min<int64_t>((rows + 63) / 64, std::max<int64_t>(resident, 1)), x1 ? 2 : 1);
    return launch_chain(chain_launches(rows, L << K), kern, grid, kBwdThreads, smem, stream, (const Tx*)x, (const Tx*)x1, planes,
                        (const Tp*)dprobs, (const Tp*)dprobs1, (Tx*)dx, (Tx*)dx1, rows, T, heads);
}

}  // namespace

bool bucket_probs_bwd_supported(int d, int L, int K, int dtype) {
    return (dtype == RACE_DTYPE_F32 || dtype == RACE_DTYPE_BF16) &&
           ((d == 64 && L == 4 && K == 4) || (d == 128 && L == 8 && K == 6));
}

cudaError_t bucket_probs_bwd(const void* x, const void* x1, const float* planes, const void* dprobs, const void* dprobs1,
                             void* dx, void* dx1, int64_t rows, int64_t T, int heads, int d, int L, int K, int dtype,
                             cudaStream_t stream) {
    if (!bucket_probs_bwd_supported(d, L, K, dtype)) return cudaErrorInvalidValue;
    using b16 = __nv_bfloat16;
    if (d == 64)
        return dtype == RACE_DTYPE_F32
                   ? launch_probs_bwd<64, 4, 4, float, float>(x, x1, planes, dprobs, dprobs1, dx, dx1, rows, T, heads, stream)
                   : launch_probs_bwd<64, 4, 4, b16, b16>(x, x1, planes, dprobs, dprobs1, dx, dx1, rows, T, heads, stream);
    return dtype == RACE_DTYPE_F32
               ? launch_probs_bwd<128, 8, 6, float, float>(x, x1, planes, dprobs, dprobs1, dx, dx1, rows, T, heads, stream)
               : launch_probs_bwd<128, 8, 6, b16, b16>(x, x1, planes, dprobs, dprobs1, dx, dx1, rows, T, heads, stream);
}

}  // namespace race
