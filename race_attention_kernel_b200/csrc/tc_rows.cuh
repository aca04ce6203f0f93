// Pieces of the tcgen05 kernels that work on chunks of 128 tokens (one accumulator row per tensor-memory lane, one token
// row per worker thread) with operand tiles in the 128-byte-swizzled layout that TMA writes, so that no warp moves an
// operand from one layout to another.
//
// An operand tile is [rows][64-value blocks of 128 bytes], block b at b * rows * 128 bytes, 16-byte piece j of row r of
// a block at r * 128 + ((j ^ (r & 7)) << 4).  The same image is read in two ways:
//   * K-major (the contraction runs along the row): 8-row groups every 1024 bytes; 16 values further = +32 bytes inside
//     a block, 64 values = the next block;
//   * MN-major (the contraction runs over the rows): 64-value blocks every rows * 128 bytes along M or N, 8-row groups
//     every 1024 bytes along K; 16 rows further = +2048 bytes.
#pragma once

#include "tc_common.cuh"

namespace race {
namespace {

constexpr uint32_t kHiSw = (1024u >> 4) | (1u << 14) | (2u << 29);   // stride 1024, descriptor version 1, 128-byte swizzle

template <bool kMn, int kRows>
__device__ __forceinline__ uint32_t sw_lo(uint32_t addr) {
    return ((addr >> 4) & 0x3FFF) | (kMn ? (uint32_t)(kRows * 128 / 16) << 16 : 1u << 16);
}
template <bool kMn, int kRows>
__device__ __forceinline__ constexpr uint32_t sw_step(int k) {   // k-step (16 values of the contraction) in lo-word units
    return kMn ? (uint32_t)k * 128u : (uint32_t)((k >> 2) * (kRows * 128 / 16) + (k & 3) * 2);
}
// D (+)= A . B over 16 * kSteps values, both operands in shared memory; kARows / kBRows: rows of the operand's tile
template <bool kZero, int kSteps, bool kAMn, int kARows, bool kBMn, int kBRows>
__device__ __forceinline__ void mma_sw(uint32_t d, uint32_t a_addr, uint32_t b_addr, uint32_t idesc) {
    const uint32_t a = sw_lo<kAMn, kARows>(a_addr), b = sw_lo<kBMn, kBRows>(b_addr);
    const uint32_t id = idesc | (kAMn ? kAmn : 0u) | (kBMn ? kBmn : 0u);
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
        const uint64_t ad = desc64(kHiSw, a + sw_step<kAMn, kARows>(k)), bd = desc64(kHiSw, b + sw_step<kBMn, kBRows>(k));
        if (kZero && k == 0) mma_issue<false>(d, ad, bd, id);
        else mma_issue<true>(d, ad, bd, id);
    }
}
// the same with A in tensor memory (packed bf16 pairs, 8 columns per k-step).  kLimbs: A is one limb of a 128 x 128
// matrix that was written over the fp32 columns it came from, 32 columns at a time: [16 words of hi | 16 words of lo]
template <bool kZero, int kSteps, bool kBMn, int kBRows, bool kLimbs = false>
__device__ __forceinline__ void mma_sw_ta(uint32_t d, uint32_t a_tmem, uint32_t b_addr, uint32_t idesc) {
    const uint32_t b = sw_lo<kBMn, kBRows>(b_addr);
    const uint32_t id = idesc | (kBMn ? kBmn : 0u);
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
        const uint64_t bd = desc64(kHiSw, b + sw_step<kBMn, kBRows>(k));
        const uint32_t at = a_tmem + (kLimbs ? 32 * (k >> 1) + 8 * (k & 1) : 8 * k);
        if (kZero && k == 0) mma_issue_ta<false>(d, at, bd, id);
        else mma_issue_ta<true>(d, at, bd, id);
    }
}

// byte offset of the 16-byte piece that holds columns [col, col + 8) of row `row` in a tile of kRows rows
template <int kRows>
__device__ __forceinline__ uint32_t sw_piece(int row, int col) {
    return (uint32_t)((col >> 6) * (kRows * 128) + row * 128 + ((((col >> 3) & 7) ^ (row & 7)) << 4));
}

// Register budgets of the roles (all four warps of a group): the shares stay below the 512 x 128 of the launch
template <int kRegs>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs)); }
template <int kRegs>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs)); }

// hi + lo limbs of a pair: hi is the upper half of the fp32 word (exact remainder), lo its remainder rounded to bf16;
// |error| <= 2^-16 |x|.  One conversion instead of two per pair: that instruction runs at a quarter of the ALU rate and
// is what a stage of limb splitting is bound by.
__device__ __forceinline__ void split2t(float a, float b, uint32_t& hi, uint32_t& lo) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    hi = __byte_perm(ua, ub, 0x7632);
    const float2 r = __fadd2_rn(make_float2(a, b), make_float2(-__uint_as_float(ua & 0xffff0000u), -__uint_as_float(ub & 0xffff0000u)));
    __nv_bfloat162 l = __floats2bfloat162_rn(r.x, r.y);
    lo = *reinterpret_cast<uint32_t*>(&l);
}

// 32 lanes x 16 columns
__device__ __forceinline__ void tmem_ld_rows16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// ... and words; no wait inside (tmem_wait_st)
__device__ __forceinline__ void tmem_st_words16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(taddr) : "memory");
}

// 32 packed words of the warp's lanes <-> 32 columns; waits for completion
__device__ __forceinline__ void tmem_st_words32(uint32_t taddr, const uint32_t (&r)[32]) {
    tmem_st_rows32(taddr, reinterpret_cast<const float(&)[32]>(r));
}

// one 32-byte store (a full sector of the row this thread owns)
__device__ __forceinline__ void st_global_32b(void* p, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}

// Rows [kRows][64-value blocks] of packed bf16 words -> a block's pieces: words w[0 .. 4 n) = columns [col, col + 8 n)
template <int kRows, int kWords>
__device__ __forceinline__ void sw_store_row(uint8_t* tile, int row, int col, const uint32_t (&w)[kWords]) {
#pragma unroll
    for (int p = 0; p < kWords / 4; ++p)
        *reinterpret_cast<uint4*>(tile + sw_piece<kRows>(row, col + 8 * p)) =
            make_uint4(w[4 * p], w[4 * p + 1], w[4 * p + 2], w[4 * p + 3]);
}

// words 32 half .. 32 half + 31 of row `row` of the 128 x 128 triangular ones matrix as a tensor-memory A operand:
// ones where the column is <= row (kUpper: >= row)
template <bool kUpper>
__device__ __forceinline__ void tri_words(int row, int half, uint32_t (&w)[32]) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const int k0 = 64 * half + 2 * i;
        const bool a = kUpper ? k0 >= row : k0 <= row, b = kUpper ? k0 + 1 >= row : k0 + 1 <= row;
        w[i] = (a ? 0x3F80u : 0u) | (b ? 0x3F800000u : 0u);
    }
}

}  // namespace
}  // namespace race
