// Float32 products on the bfloat16 tensor cores without giving up 32 bits: what the kernels that do so share.
//
// A float is the sum of three bfloat16 (24 bits in three times 8, each piece the rounded rest of the ones before), and a
// product of two bfloat16 is exact in the tensor core's float sums.  Of the nine products of pieces six are formed,
//   a0 w0 + (a0 w1 + a1 w0) + (a0 w2 + a1 w1 + a2 w0);
// the other three lie below 2^-24 of the product together, which is what a float product is itself rounded by.  (The method is that of
// G. Henry, P. T. P. Tang and A. Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations",
// 2019.)  The tensor core's own additions
// round towards zero, which over a long k would shrink a sum by more than float additions in order miss it by, so an
// accumulator takes CHUNK k only: first the small products, then the large ones (four roundings of the sum's own size), and is
// then added into registers with ordinary float additions.  What is left of it: sums whose products all have one sign are 0.6 * 2^-23 of
// their size too small on average.
//
// A bfloat16 ends where a float does, so the pieces of small floats would lose their low bits: both operands are split at
// SCALE times their size, which keeps every bit of the smallest float, and the sums are scaled back (both exact).  What is large enough
// to overflow for that, infinities and NaN come out as infinity or NaN; write-backs form every sum that is not finite again,
// with float arithmetic from the operands (plain_sums), so they end as they would there.
#pragma once

#include "tcgen05.cuh"

namespace {

constexpr int CHUNK = BK;           // k of one accumulator: a row of 64 bfloat16 is the 128 bytes of the swizzle
constexpr int N_PIECES = 3;
// the products in the order in which an accumulator takes them, small ones first
constexpr int N_PRODUCTS = 6;
__device__ constexpr int PIECE_OF_A[N_PRODUCTS] = {0, 1, 2, 0, 1, 0};
__device__ constexpr int PIECE_OF_W[N_PRODUCTS] = {2, 1, 0, 1, 0, 0};

constexpr float SCALE = 0x1p20f, UNSCALE = 0x1p-40f;        // of an operand, of a sum of products

// Two floats into their three pieces, each a pair of bfloat16 (x0 in the low half).
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t (&piece)[N_PIECES]) {
    float2 v = __fmul2_rn(make_float2(x0, x1), make_float2(SCALE, SCALE));
#pragma unroll
    for (int i = 0; i < N_PIECES; i++) {
        const __nv_bfloat162 h = __float22bfloat162_rn(v);
        piece[i] = *reinterpret_cast<const uint32_t*>(&h);
        if (i + 1 < N_PIECES)       // the rest, exactly
            v = __ffma2_rn(make_float2(__uint_as_float(piece[i] << 16), __uint_as_float(piece[i] & 0xffff0000u)), make_float2(-1.0f, -1.0f), v);
    }
}

// Eight floats that follow one another along k: sixteen bytes of each piece.
__device__ __forceinline__ void split_eight(const float4& x, const float4& y, uint4 (&piece)[N_PIECES]) {
    uint32_t p0[N_PIECES], p1[N_PIECES], p2[N_PIECES], p3[N_PIECES];
    split_pair(x.x, x.y, p0);
    split_pair(x.z, x.w, p1);
    split_pair(y.x, y.y, p2);
    split_pair(y.z, y.w, p3);
#pragma unroll
    for (int i = 0; i < N_PIECES; i++) piece[i] = make_uint4(p0[i], p1[i], p2[i], p3[i]);
}

__device__ __forceinline__ bool is_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// The sums of a row of a with up to four rows of w in float arithmetic, by a whole warp; K is a multiple of 4 and all rows start on 16
// bytes.  Returns whether the row of a holds a NaN: then its sum with any row is one.
__device__ __forceinline__ bool plain_sums(const float* a, const float* w, int ldw, int rows, int K, float (&sum)[4]) {
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    bool nan = false;
#pragma unroll 1
    for (int k = (threadIdx.x & 31) * 4; k < K; k += 128) {
        const float4 x = *reinterpret_cast<const float4*>(a + k);
        nan |= x.x != x.x || x.y != x.y || x.z != x.z || x.w != x.w;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 y = *reinterpret_cast<const float4*>(w + (size_t)min(i, rows - 1) * ldw + k);
            s[i] = fmaf(x.x, y.x, s[i]);
            s[i] = fmaf(x.y, y.y, s[i]);
            s[i] = fmaf(x.z, y.z, s[i]);
            s[i] = fmaf(x.w, y.w, s[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) sum[i] = warp_sum(s[i]);
    return __any_sync(0xffffffffu, nan);
}

// tensor-core product with the A operand in tensor memory
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint4& x, const uint4& y) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w), "r"(y.x), "r"(y.y), "r"(y.z), "r"(y.w)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The instructions of one chunk into the accumulator at tmem_d, which they overwrite.  a: tensor-memory address of the first
// piece's columns (two k a column, the pieces one behind the other); w: shared-memory address of the first piece's tile, the
// pieces w_piece bytes apart.
__device__ __forceinline__ void issue_chunk(uint32_t tmem_d, uint32_t a, uint32_t w, uint32_t w_piece, uint32_t idesc) {
#pragma unroll
    for (int p = 0; p < N_PRODUCTS; p++) {
        const uint64_t dw = make_smem_desc(w + PIECE_OF_W[p] * w_piece);
#pragma unroll
        for (int k = 0; k < CHUNK / UMMA_K; k++)
            umma_bf16_ta(tmem_d, a + PIECE_OF_A[p] * (CHUNK / 2) + 8 * k, dw + (uint64_t)(2 * k), idesc, p > 0 || k > 0 ? 1u : 0u);
    }
}

}  // namespace
