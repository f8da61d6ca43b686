// Building blocks of the fp32 attention kernels on warp-level tensor-core instructions (flash.cu): tiles of rows in
// shared memory that are read without bank conflicts both along the head dimension and along the rows, and fp32
// products as three TF32 products.
//
// x = hi + lo, hi the nearest TF32 value, lo = x - hi (exact; the instruction reads its upper 11 bits).  a b is
// hi hi + hi lo + lo hi up to 2^-23 of |a b|.  The instruction cuts its running sums off instead of rounding them, so
// a chain is short (two instructions, 16 columns; with single ones, or with lo rounded, the errors are the same to 3 % and
// the kernels 5 to 10 % slower) and chains are added in fp32; the small terms have one chain of their own, added at the
// end.  What is cut off has a mean, half a unit of the last place per instruction: CUT of the sum is added with the small terms,
// in scores (forward and backward alike: a probability is the exponential of a difference of the two) and in the output;
// 1.5 and 2 times that gave larger errors, and sums of gradients, which change sign more often, smaller ones without.
// 2-norm errors against 64 bits at T = 256, head sizes 32 / 64 / 128, without it and with it: output 1.75 / 1.63 / 1.80e-7 ->
// 1.45 / 1.49 / 1.54e-7, lse 4.6 / 4.3 / 4.6e-8 -> 3.8 / 3.7 / 3.9e-8, dqkv at T = 2048, 128 columns, 3.43 -> 3.38e-7.
// Elements below 2^-108 lose bits of lo (the instruction's operands end at 2^-136).
//
// FINE, for short sequences, where there are few sums to round and what a product leaves out is what counts: three pieces
// of 8 bits and six products, so that no bit of x is left out and the products of the first pieces (16 bits) are added
// up without being cut off.
//
// Why these instructions and not tcgen05 (flash_x2.cu) where sequences are short or a head's elements differ too much: the operands stay
// plain fp32 in shared memory, of any size, there is no pass over them first, and probabilities go from accumulator to operand
// without leaving registers.  Three TF32 products a multiply-add leave 170 of them per cycle and SM, against 128 on the FMA
// pipe, which the kernels these replaced used to 19 %.
#pragma once
#include "common.cuh"

namespace bmb {
namespace fm {

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A tile is rows of HS floats; the 16-byte unit u of row r lies at unit u ^ f(r).  f makes both ways of reading hit
// eight different 16-byte bank groups per quarter warp: two neighbouring rows x four neighbouring units (operands
// read along the head dimension) and four rows of one parity x two neighbouring units (operands read along rows).
__device__ __forceinline__ int unit_of(int r, int u) { return u ^ ((((r >> 1) & 3) << 1) ^ ((r & 1) << 2)); }
template <int HS>
__device__ __forceinline__ float4 tile_ld(const float *t, int r, int u) {
    return *reinterpret_cast<const float4 *>(t + r * HS + (unit_of(r, u) << 2));
}
// Start copying rows [0, ROWS) from src (row pitch ld floats); rows from `valid` on are filled with zeros.
template <int HS, int ROWS, int NT>
__device__ __forceinline__ void tile_copy(float *t, const float *src, long long ld, int valid) {
    constexpr int V4 = HS / 4;
#pragma unroll
    for (int i = 0; i < ROWS * V4 / NT; ++i) {
        const int lin = i * NT + (int)threadIdx.x, r = lin / V4, u = lin % V4;
        const bool ok = r < valid;
        cp_async16(t + r * HS + (unit_of(r, u) << 2), src + (ok ? (long long)r * ld : 0LL) + u * 4, ok);
    }
}

constexpr float CUT = 5.9604644775390625e-8f;      // 2^-24
enum Form { COARSE, COARSE_CUT, FINE };             // three products, with CUT, six products
struct HiLo { uint32_t hi, mid, lo; };              // (mid: FINE only)
template <Form FORM>
__device__ __forceinline__ HiLo split(float x) {
    HiLo s;
    if (FORM == FINE) {
        s.hi = (__float_as_uint(x) + 0x8000u) & 0xffff0000u;
        const float r = x - __uint_as_float(s.hi);
        s.mid = (__float_as_uint(r) + 0x8000u) & 0xffff0000u;
        s.lo = __float_as_uint(r - __uint_as_float(s.mid));
    } else {
        s.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
        s.mid = 0;
        s.lo = __float_as_uint(x - __uint_as_float(s.hi));
    }
    return s;
}
template <bool FIRST>
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(FIRST ? 0.0f : d[0]), "f"(FIRST ? 0.0f : d[1]),
                   "f"(FIRST ? 0.0f : d[2]), "f"(FIRST ? 0.0f : d[3]));
}
// Four neighbouring groups of 8 columns: big[j] (+)= a_hi b_hi, small[j] (+)= the smaller products; FIRST and FIRST_SMALL
// start the sums.  Issued so that an instruction never waits for the one before it.
template <bool FIRST, bool FIRST_SMALL, Form FORM>
__device__ __forceinline__ void mma3x4(float (&big)[4][4], float (&small)[4][4], const HiLo (&a)[4], const HiLo (&b0)[4], const HiLo (&b1)[4]) {
    if (FORM == FINE) {
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<FIRST_SMALL>(small[j], a[0].lo, a[1].lo, a[2].lo, a[3].lo, b0[j].hi, b1[j].hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<false>(small[j], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b0[j].lo, b1[j].lo);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<false>(small[j], a[0].mid, a[1].mid, a[2].mid, a[3].mid, b0[j].mid, b1[j].mid);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<false>(small[j], a[0].mid, a[1].mid, a[2].mid, a[3].mid, b0[j].hi, b1[j].hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<FIRST>(big[j], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b0[j].hi, b1[j].hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<false>(small[j], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b0[j].mid, b1[j].mid);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<FIRST_SMALL>(small[j], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b0[j].lo, b1[j].lo);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<FIRST>(big[j], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b0[j].hi, b1[j].hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) mma<false>(small[j], a[0].lo, a[1].lo, a[2].lo, a[3].lo, b0[j].hi, b1[j].hi);
    }
}
// Chains added up, and what was left out of them, times f: rounded once.
template <Form FORM>
__device__ __forceinline__ float whole(float sum, float small, float f) { return fmaf(sum, f, (FORM == COARSE_CUT ? fmaf(sum, CUT, small) : small) * f); }

// s = f times 16 rows of A (a_row + lane/4, + 8) times 32 rows of B (b_row ..), along the head dimension.  s[j] is the
// instruction's accumulator for rows 8j .. 8j+7 of B: [0], [1] = A row lane/4, B rows 2(lane%4), + 1; [2], [3] = A
// row + 8.  The order of the head's columns inside an instruction is free as long as A and B agree: a thread's four
// neighbouring columns serve two instructions.
template <int HS, Form FORM>
__device__ __forceinline__ void scores(float (&s)[4][4], float f, const float *A, int a_row, const float *B, int b_row) {
    constexpr int FOLD = 2;                        // instructions' worth of 8 columns that the tensor core adds up by itself
    const int g = (threadIdx.x >> 2) & 7, t = threadIdx.x & 3;
    float big[4][4], small[4][4];
#pragma unroll
    for (int kk = 0; kk < HS / 16; ++kk) {
        const float4 x = tile_ld<HS>(A, a_row + g, 4 * kk + t), y = tile_ld<HS>(A, a_row + g + 8, 4 * kk + t);
        float4 b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = tile_ld<HS>(B, b_row + 8 * j + g, 4 * kk + t);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const HiLo a[4] = {split<FORM>(h ? x.z : x.x), split<FORM>(h ? y.z : y.x), split<FORM>(h ? x.w : x.y), split<FORM>(h ? y.w : y.y)};
            HiLo b0[4], b1[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { b0[j] = split<FORM>(h ? b[j].z : b[j].x); b1[j] = split<FORM>(h ? b[j].w : b[j].y); }
            if (kk == 0 && h == 0) mma3x4<true, true, FORM>(big, small, a, b0, b1);
            else if ((2 * kk + h) % FOLD == 0) mma3x4<true, false, FORM>(big, small, a, b0, b1);
            else mma3x4<false, false, FORM>(big, small, a, b0, b1);
            if ((2 * kk + h) % FOLD == FOLD - 1) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[j][i] = 2 * kk + h < FOLD ? big[j][i] : s[j][i] + big[j][i];
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[j][i] = whole<FORM>(s[j][i], small[j][i], f);
}

// o = o * (f0 | f1) + p (16 x 32, laid out as scores() leaves it) times 32 rows of B.  Columns of o: accumulator
// 4J + j of this thread holds, for A row lane/4 ([0], [1]) and + 8 ([2], [3]), head columns 32J + 8(lane%4) + j and
// + 4.  (The thread's four neighbouring columns serve four instructions, so its results are eight neighbours.)
template <int HS, Form FORM, bool RESCALE>
__device__ __forceinline__ void contract(float (&o)[HS / 8][4], float f0, float f1, const float (&p)[4][4], const float *B, int b_row) {
    constexpr int FOLD = 2;
    const int g = (threadIdx.x >> 2) & 7, t = threadIdx.x & 3;
    HiLo a[4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int i = 0; i < 4; ++i) a[ks][i] = split<FORM>(p[ks][i == 1 ? 2 : i == 2 ? 1 : i]);
#pragma unroll
    for (int J = 0; J < HS / 32; ++J) {
        float small[4][4], sum[4][4];
#pragma unroll
        for (int k0 = 0; k0 < 4; k0 += FOLD) {
            float big[4][4];
#pragma unroll
            for (int ks = k0; ks < k0 + FOLD; ++ks) {
                const int r = b_row + 8 * ks + 2 * t;
                const float4 u = tile_ld<HS>(B, r, 8 * J + g), v = tile_ld<HS>(B, r + 1, 8 * J + g);
                const HiLo b0[4] = {split<FORM>(u.x), split<FORM>(u.y), split<FORM>(u.z), split<FORM>(u.w)}, b1[4] = {split<FORM>(v.x), split<FORM>(v.y), split<FORM>(v.z), split<FORM>(v.w)};
                if (ks == 0) mma3x4<true, true, FORM>(big, small, a[ks], b0, b1);
                else if (ks == k0) mma3x4<true, false, FORM>(big, small, a[ks], b0, b1);
                else mma3x4<false, false, FORM>(big, small, a[ks], b0, b1);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) sum[j][i] = k0 == 0 ? big[j][i] : sum[j][i] + big[j][i];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float (&q)[4] = o[4 * J + j];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float x = whole<FORM>(sum[j][i], small[j][i], 1.0f);
                q[i] = RESCALE ? fmaf(q[i], i < 2 ? f0 : f1, x) : q[i] + x;
            }
        }
    }
}

// Store this thread's part of 16 rows of results (row r0 and r0 + 8, those below `valid`), times f0 / f1; true if
// a value is not finite.
template <int HS>
__device__ __forceinline__ bool store_rows(float *dst, long long ld, int r0, int valid, const float (&o)[HS / 8][4], float f0, float f1) {
    const int t = threadIdx.x & 3;
    bool bad = false;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = r0 + 8 * h;
        if (r >= valid) continue;
        const float f = h ? f1 : f0;
#pragma unroll
        for (int J = 0; J < HS / 32; ++J) {
            float4 *d = reinterpret_cast<float4 *>(dst + (long long)r * ld + 32 * J + 8 * t);
            const float4 x = make_float4(o[4 * J][2 * h] * f, o[4 * J + 1][2 * h] * f, o[4 * J + 2][2 * h] * f, o[4 * J + 3][2 * h] * f);
            const float4 y = make_float4(o[4 * J][2 * h + 1] * f, o[4 * J + 1][2 * h + 1] * f, o[4 * J + 2][2 * h + 1] * f,
                                         o[4 * J + 3][2 * h + 1] * f);
            d[0] = x;
            d[1] = y;
            const float sum = fabsf(x.x) + fabsf(x.y) + fabsf(x.z) + fabsf(x.w) + fabsf(y.x) + fabsf(y.y) + fabsf(y.z) + fabsf(y.w);
            bad = bad || !(sum <= 3.402823466e38f);               // (NaN fails the comparison)
        }
    }
    return bad;
}

}  // namespace fm
}  // namespace bmb
