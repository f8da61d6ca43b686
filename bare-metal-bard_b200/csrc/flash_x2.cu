// Fused causal attention at fp32 accuracy on the tensor cores (src/flash.h:36-62, src/flash.cu): every fp32 operand as two
// fp16 pieces, three fp16 products for one fp32 product.  Head sizes 32, 64 and 128.
//
//   x 2^k = hi + lo 2^-11,  hi = fp16(x 2^k),  lo = fp16((x 2^k - hi) 2^11),   k from the largest element of 64 rows
//
// hi and lo hold 22 to 23 bits of x; a b is hi hi + 2^-11 (hi lo + lo hi) up to 2^-22 of |a b|.  The products of the small
// pieces come first and are scaled by 2^-11 by the first instruction that adds products of the large ones (scale-input-d), so
// one accumulator serves all.  Elements down to 2^-28 of the largest of their 64 rows keep all bits that hi and lo have, smaller
// ones are held to 2^-51 of it, which is 2^-31 of the largest in their row or column (see below).  Probabilities and dS are split in
// registers, scaled by the most that they can be, and so are held to 2^-45 (forward) or 2^-50 (backward) of a weight of 1.
// Why fp16 and not bf16 or TF32: at the same accuracy bf16 takes six products, TF32 three at half the rate and twice the
// bytes in shared memory, which is what bounds the 64-column products below (69 cycles with both operands there, 40 with
// one in tensor memory, 32 by the pipe's rate).
//
// The tensor core cuts its running sums off, on average 2.2e-8 of the sum an instruction of 16 columns (measured); the mean is put
// back with the factor that unscales the sums (CUT), and sums over positions leave tensor memory every 64 positions for
// fp32 registers.
//
// What two pieces cannot serve is left to the kernels of flash.cu, which run behind these for the heads that have any of it: 64 rows
// whose largest element is not in 2^-45 .. 2^30 (nor zero) or not finite, a row or column whose largest element is below 2^-20 of that
// (and not zero; of V in the backward, a row below 2^-12), D beyond 2^70, lse beyond 2^19, a row's largest score beyond 2^22
// (MOST_SCORE), a probability beyond sqrt(2) (of an lse that is not the scores').  Inside these limits no sum can overflow.
//
// Bound by what a step of 64 columns waits for in turn (products, exponentials and splits, sums) and by the FMA pipe, on which
// the splits and exponentials of 128 x 64 elements are 1000 to 1400 cycles; products 2600 (64 columns, keys' side).  Four
// warpgroups compute: with two, as with longer pieces of a row in registers, the step was no faster (12.5 KB of code a loop instead
// of 35 and 16 columns at a time count for more).  us, the kernels of flash.cu -> these, split pass included: B8 T1024 12 heads of
// 64 forward 253 -> 123, backward 958 -> 283; B4 T2048 8 x 128 664 -> 211, 2490 -> 649; B2 T777 12 x 32 41 -> 31, 105 -> 47.
// 2-norm errors against 64 bits there: 8 x 160 x 4 heads of 64 and up, output 0.95 to 1.0 of those kernels', lse 0.7, dqkv 0.82 to 1.0.
#include "tc_common.cuh"
#include <cuda_fp16.h>
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>

namespace bmb {
// flash.cu: the kernels on warp-level instructions, for the heads left out here.
int flash_fwd_left(int hs, float *out, float *lse, const float *qkv, int T, int NH, float scale, LeftOut left, cudaStream_t st);
int flash_bwd_left(int hs, float *dqkv, const float *dsum, const float *dout, const float *qkv, const float *lse, int T, int NH, float scale,
                   LeftOut left, cudaStream_t st);
namespace {

using namespace tc;

constexpr int XB = 64;                             // positions of a block: one step, one ring slot, one scale
constexpr int ROWS_BYTES = 3 * XB * 4;             // what the backward knows of the queries of a block, beside their images
// Four warpgroups that compute, one of copying and issuing warps.
constexpr int COMPUTE = 512, THREADS = COMPUTE + 128, W_COPY = COMPUTE / 32, W_ISSUE = W_COPY + 1;
constexpr int REGS_COMPUTE = 104, REGS_OTHER = 64; // 512 x 104 + 128 x 64 = 640 x 96, the launch's registers
constexpr float LEAST = 2.8421709430404007e-14f, MOST = 1073741824.0f;       // 2^-45, 2^30: the largest element of a block
constexpr double CUT = 2.17e-8;                    // of a sum, cut off by an instruction, on average
// Of a row's largest score, times log2(e): the reference of its exponentials is that score rounded to fp32, and what the rounding
// leaves (at most 1/4 here; 8 at 2^27) is part of the exponents, which have room for 1/2.
constexpr float MOST_SCORE = 4194304.0f - 8.0f;     // (of the reference, which the score may pass by 6)
constexpr float TINY = 7.5231638e-37f;             // 2^-120: dS is scaled by no more than its inverse
constexpr float WINDOW = 113.0f;                   // exponents of probabilities are followed to 2^-113
// What scores and lse are both multiplied with: a row whose weight lies on one key has lse = its score, bit for bit, and that
// key the probability 1, although neither may be rounded little at its size.
constexpr float LOG2E = 1.4426950408889634f, INV_LOG2E = 0.693147182f, INV_LOG2E_REST = 7.348693210e-09f;

template <int HS> struct Geo {
    static constexpr int ROWB = HS >= 64 ? 128 : 64;       // bytes of an image row: 128- or 64-byte swizzle
    static constexpr int CE = ROWB / 2, NCH = HS / CE;     // elements of a row, rows side by side for the head size
    static constexpr int KPC = CE / 16;                    // instructions along a row
    static constexpr uint32_t LT = ROWB == 128 ? 2 : 4;    // the descriptor's layout type
    static constexpr int PIECE = XB * HS * 2, BLK = 2 * PIECE;
    static constexpr int TPIECE = 128 * HS * 2, TILE = 2 * TPIECE;
};

// q is multiplied with scale before it is split (q + q_rest: with more bits than fp32 has), so that scores need no factor but a
// power of two; the other factors undo that and put the mean of what is cut off back.
struct Factors { float q, q_rest, dp, sums, dk, dq, dv; };

// ---- operands as images ----------------------------------------------------------------------------------------------
// Image of 64 positions of one head: [hi, lo][NCH][64 rows of ROWB bytes, swizzled], one contiguous bulk copy.  Both readings
// that the tensor core makes of it (along the head dimension; along the positions) have the same layout.
struct Images {
    uint8_t *img;                  // [which: q, k, v, dO][BH][nblk][BLK]
    float *unscale;                // [which][BH][nblk]: what an image's values are multiplied with
    uint8_t *flags;                // [BH][which][nblk]: a block that two pieces cannot serve
    LeftOut left;                  // heads that these kernels leave to those of flash.cu
    // Backward, [BH][nblk][3][64]: of every query minus the rest of lse log2(e) (past the end: - infinity), its whole part - WINDOW, and D
    float *rows;
    // Backward, powers of two (or zero), no less than any element of what they stand for:
    float4 *tops;                  // [BH][nblk]: V, dO, and D of the block
    uint8_t *ptops;                // [BH][nblk][3][64], as codes: of a row of V, of a row of dO, of its D
};

// x + xe, y + ye (xe, ye: what fp32 does not hold of them)
__device__ __forceinline__ void split2(float x, float xe, float y, float ye, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const __half2 l = __floats2half2_rn(((x - __low2float(h)) + xe) * 2048.0f, ((y - __high2float(h)) + ye) * 2048.0f);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }      // -126 <= e <= 127
__device__ __forceinline__ int exponent(float x) { return (int)(__float_as_uint(x) >> 23 & 255) - 127; }
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// The least power of two above |x| (at most 2^127), or zero, and its code: the exponent's bits.
__device__ __forceinline__ uint32_t top_code(float x) { return x == 0.0f ? 0u : min((__float_as_uint(x) >> 23 & 255) + 1, 254u); }
__device__ __forceinline__ float top_of(uint32_t code) { return __uint_as_float(code << 23); }

// One block: 64 positions of one head of q, k, v or dO; bound by memory (4 bytes read and 4 written an element).  With dO also
// D = rowsum(dO O).
template <int HS>
__global__ void __launch_bounds__(256, HS == 32 ? 5 : HS == 64 ? 4 : 2) split_x2_k(const Images im, float *__restrict__ dsum, const float *__restrict__ qkv,
                                                  const float *__restrict__ dout, const float *__restrict__ out,
                                                  const float *__restrict__ lse, int T, int NH, int BH, int nblk, int nw, Factors fac) {
    using G = Geo<HS>;
    constexpr int UPR = HS / 8, ITEMS = XB * UPR / 256;
    __shared__ float red[8];
    __shared__ __align__(16) __half2 columns[8][4 * UPR];
    __shared__ int dred;
    if (threadIdx.x == 0) dred = 0;
    const int blk = (int)(blockIdx.x % (unsigned)nblk), which = (int)(blockIdx.x / (unsigned)nblk % (unsigned)nw);
    const int bh = (int)(blockIdx.x / (unsigned)nblk / (unsigned)nw), b = bh / NH, h = bh % NH, C = NH * HS;
    const long long ld = which < 3 ? 3LL * C : C;
    const float *src = (which < 3 ? qkv + which * C : dout) + ((long long)b * T + blk * XB) * ld + h * HS;
    float v[ITEMS][8], rest[ITEMS][8], rowmax[ITEMS], most = 0.0f, dmax = 0.0f;      // rest: of q only
    uint8_t *ptops = im.ptops + ((long long)bh * nblk + blk) * (3 * XB);
    bool lost = false;                                       // D or lse out of range
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int u = i * 256 + (int)threadIdx.x, r = u / UPR, c = u % UPR * 8, pos = blk * XB + r;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
        if (pos < T) {
            x = __ldg(reinterpret_cast<const float4 *>(src + r * ld + c));
            y = __ldg(reinterpret_cast<const float4 *>(src + r * ld + c) + 1);
        }
        v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w; v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
        if (which == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float q = v[i][j];
                v[i][j] = q * fac.q;
                rest[i][j] = fmaf(q, fac.q, -v[i][j]) + q * fac.q_rest;
            }
        }
        float m = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j += 2) asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(v[i][j]), "f"(v[i][j + 1]));
        if (which == 3) {
            float a = 0.0f;
            if (pos < T) {
                const float *o = out + ((long long)b * T + pos) * C + h * HS + c;
                const float4 p = __ldg(reinterpret_cast<const float4 *>(o)), q = __ldg(reinterpret_cast<const float4 *>(o) + 1);
                a = (x.x * p.x + x.y * p.y + x.z * p.z + x.w * p.w) + (y.x * q.x + y.y * q.y + y.z * q.z + y.w * q.w);
            }
#pragma unroll
            for (int o = UPR / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (c == 0) {
                const long long at = (long long)bh * T + pos, to = ((long long)bh * nblk + blk) * (3 * XB) + r;
                const float L = pos < T ? lse[at] : INFINITY;
                if (pos < T) {
                    dsum[at] = a;
                    lost = lost || !(fabsf(a) <= 1.1805916e21f) || !(fabsf(L) <= 524288.0f);
                }
                dmax = fmaxf(dmax, fabsf(a));
                ptops[2 * XB + r] = (uint8_t)top_code(a);
                im.rows[to + 2 * XB] = fmaf(a, -fac.dp, a);
                const float w = rintf(L * LOG2E);
                im.rows[to + XB] = (pos < T ? w : 0.0f) - WINDOW;
                im.rows[to] = pos < T ? -fmaf(L, LOG2E, -w) : -INFINITY;
            }
        }
#pragma unroll
        for (int o = UPR / 2; o > 0; o >>= 1) asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(__shfl_xor_sync(0xffffffffu, m, o)));
        rowmax[i] = m;
        if (nw == 4 && which >= 2 && c == 0) ptops[(which - 2) * XB + r] = (uint8_t)top_code(m);
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(most) : "f"(m));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) asm("max.NaN.f32 %0, %0, %1;" : "+f"(most) : "f"(__shfl_xor_sync(0xffffffffu, most, o)));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = most;
    __syncthreads();
    if (dmax > 0.0f) atomicMax(&dred, __float_as_int(dmax));             // (not negative: ordered as whole numbers are)
#pragma unroll
    for (int i = 0; i < 8; ++i) asm("max.NaN.f32 %0, %0, %1;" : "+f"(most) : "f"(red[i]));
    const bool usable = most >= LEAST && most < MOST;
    bool bad = lost || (most != 0.0f && !usable);
    // Rows and columns of the block against its largest element: products sum along both, and hold 2^-31 of a row's or column's largest
    // element where that is 2^-20 of the block's.
    // (In V of a backward rows from 2^-12 on: dS of a row has one scale for a block's 64 keys, so what belongs to small rows of V loses bits
    // where the large ones have hardly any weight.  The same of dO would be a rule for its time alone: gradients of single positions fall
    // below 2^-12 of their neighbours' as soon as a model is sure of some of them, and with that rule 10 % and more of a character model's
    // step went to the kernels behind; a key that only such positions look at has its dK to 2^-42 of what a large one could give.)
    const float low_end = 9.5367432e-7f * most, low_row = nw == 4 && which == 2 ? 2.44140625e-4f * most : low_end;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) bad = bad || (rowmax[i] != 0.0f && rowmax[i] < low_row);
    const int e = usable ? exponent(most) : 14;
    const float f = usable ? pow2(14 - e) : 0.0f;
    uint8_t *img = im.img + (((long long)which * BH + bh) * nblk + blk) * G::BLK;
    __half2 colmax[4];                                       // the largest elements of this thread's columns, by their large pieces
#pragma unroll
    for (int j = 0; j < 4; ++j) colmax[j] = __half2(0.0f, 0.0f);
    auto put = [&](bool q) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int u = i * 256 + (int)threadIdx.x, r = u / UPR, c = u % UPR;
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                split2(v[i][2 * j] * f, q ? rest[i][2 * j] * f : 0.0f, v[i][2 * j + 1] * f, q ? rest[i][2 * j + 1] * f : 0.0f, hi[j], lo[j]);
                colmax[j] = __hmax2(colmax[j], __habs2(*reinterpret_cast<const __half2 *>(&hi[j])));
            }
            const int ch = c / (G::CE / 8), uc = c % (G::CE / 8), x = G::ROWB == 128 ? (r & 7) : (r >> 1 & 3);
            uint8_t *d = img + ch * (XB * G::ROWB) + r * G::ROWB + ((uc ^ x) << 4);
            *reinterpret_cast<uint4 *>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4 *>(d + G::PIECE) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    };
    if (which == 0) put(true);
    else put(false);
#pragma unroll
    for (int o = 16; o >= UPR; o >>= 1)
#pragma unroll
        for (int j = 0; j < 4; ++j) colmax[j] = __hmax2(colmax[j], __shfl_xor_sync(0xffffffffu, colmax[j], o));
    if ((threadIdx.x & 31) < UPR) *reinterpret_cast<uint4 *>(&columns[threadIdx.x >> 5][4 * (threadIdx.x & 31)]) = *reinterpret_cast<const uint4 *>(colmax);
    __syncthreads();
    if (threadIdx.x < 4 * UPR) {
        __half2 m = columns[0][threadIdx.x];
#pragma unroll
        for (int i = 1; i < 8; ++i) m = __hmax2(m, columns[i][threadIdx.x]);
        columns[0][threadIdx.x] = m;
        bad = bad || fminf(__low2float(m), __high2float(m)) < low_end * f;
    }
    bad = __syncthreads_or(bad);
    if (bad && usable) {                                     // something is small, or a column is zero, which is no harm
        bool small = false;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            small = small || (rowmax[i] != 0.0f && rowmax[i] < low_row);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const __half2 m = columns[0][4 * ((int)threadIdx.x % UPR) + j / 2];
                small = small || (v[i][j] != 0.0f && (j & 1 ? __high2float(m) : __low2float(m)) < low_end * f);
            }
        }
        bad = __syncthreads_or(small || lost);
    }
    if (threadIdx.x == 0) {
        // A block of zeros in V or dO has no size of its own: what dS is scaled by (bwd_x2's bound) is then D's.
        im.unscale[((long long)which * BH + bh) * nblk + blk] = which >= 2 && most == 0.0f ? 0.0f : pow2(e - 14);
        im.flags[((long long)bh * nw + which) * nblk + blk] = bad;
        if (which == 0 && blk == 0) im.left.flagged[bh] = 0;
        if (blockIdx.x == 0) *im.left.taken = 0;
        if (nw == 4 && which >= 2) reinterpret_cast<float *>(im.tops + (long long)bh * nblk + blk)[which - 2] = top_of(top_code(most));
        if (which == 3) im.tops[(long long)bh * nblk + blk].z = fmaxf(top_of(top_code(__int_as_float(dred))), TINY);
    }
    let_successor_start();
}

// ---- shared pieces of the attention kernels --------------------------------------------------------------------------
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// D (+)= A B; SCALED: D = A B + D 2^-11.  A from shared memory (descriptor) or from tensor memory (address).
__device__ __forceinline__ void mma_scaled(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 11;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void mma_ts_scaled(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, 11;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc) : "memory");
}
// 128 rows of a tile x 64 rows of a block, along the columns 16 K0 .. 16 K1 - 1 of the head: small terms first.
template <int HS, int K0 = 0, int K1 = HS / 16>
__device__ __forceinline__ void issue_scores(uint32_t d, uint32_t tile, uint32_t blk) {
    using G = Geo<HS>;
    constexpr uint32_t idesc = make_idesc(0, 0, 0, XB, 128);
    auto a = [&](int piece, int ks) { return smem_desc(tile + piece * G::TPIECE + ks / G::KPC * (128 * G::ROWB) + ks % G::KPC * 32, 16, 8 * G::ROWB, G::LT); };
    auto b = [&](int piece, int ks) { return smem_desc(blk + piece * G::PIECE + ks / G::KPC * (XB * G::ROWB) + ks % G::KPC * 32, 16, 8 * G::ROWB, G::LT); };
#pragma unroll
    for (int ks = K0; ks < K1; ++ks) mma_f16(d, a(1, ks), b(0, ks), idesc, ks > K0 ? 1u : 0u);
#pragma unroll
    for (int ks = K0; ks < K1; ++ks) mma_f16(d, a(0, ks), b(1, ks), idesc, 1u);
#pragma unroll
    for (int ks = K0; ks < K1; ++ks) {
        if (ks == K0) mma_scaled(d, a(0, ks), b(0, ks), idesc);
        else mma_f16(d, a(0, ks), b(0, ks), idesc, 1u);
    }
}
// 128 x 64 weights in tensor memory (in the 16 columns of 16 weights: hi, lo) x the block's 64 rows.
template <int HS>
__device__ __forceinline__ void issue_sum(uint32_t d, uint32_t w, uint32_t blk) {
    using G = Geo<HS>;
    constexpr uint32_t idesc = make_idesc(0, 0, 1, HS, 128);
    auto b = [&](int piece, int ks) { return smem_desc(blk + piece * G::PIECE + ks * (16 * G::ROWB), XB * G::ROWB, 8 * G::ROWB, G::LT); };
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_ts(d, w + ks * 16 + 8, b(0, ks), idesc, ks ? 1u : 0u);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) mma_ts(d, w + ks * 16, b(1, ks), idesc, 1u);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        if (ks == 0) mma_ts_scaled(d, w + ks * 16, b(0, ks), idesc);
        else mma_ts(d, w + ks * 16, b(0, ks), idesc, 1u);
    }
}
// A tile of 128 positions from block `blk` on (the second half only where there is one): bytes copied.
template <int HS>
__device__ __forceinline__ uint32_t tile_bytes(int blk, int nblk) { return blk + 1 < nblk ? Geo<HS>::TILE : Geo<HS>::TILE / 2; }
template <int HS>
__device__ __forceinline__ void copy_tile(uint32_t dst, const uint8_t *blocks, int blk, int nblk, uint32_t bar) {
    using G = Geo<HS>;
    for (int half = 0; half < 2 && blk + half < nblk; ++half)
#pragma unroll
        for (int p = 0; p < 2 * G::NCH; ++p)
            bulk_copy(dst + p * (128 * G::ROWB) + half * (XB * G::ROWB), blocks + (long long)(blk + half) * G::BLK + p * (XB * G::ROWB), XB * G::ROWB, bar);
}
// Every lane waits; true if none gave up (what follows is for whole warps).
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *giveup) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, giveup));
}
// The 256 threads of a tile (named barrier 1 + t): whether all of them are still on course, so that they leave together.
__device__ __forceinline__ bool pair_all(int t, bool ok) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %2, 0;\n\tbar.red.and.pred p, %1, 256, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r) : "r"(1 + t), "r"((uint32_t)ok) : "memory");
    return r != 0;
}
__device__ __forceinline__ bool any_flag(const uint8_t *flags, int n) {
    bool f = false;
    for (int i = threadIdx.x; i < n; i += THREADS) f = f || flags[i];
    return __syncthreads_or(f);
}
// Two floats in one register pair (FFMA2 and its like do two in one issue slot).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f2 both(float x) { return pack(x, x); }
__device__ __forceinline__ void unpack(f2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ float low(f2 v) { float a, b; unpack(v, a, b); return a; }
__device__ __forceinline__ float high(f2 v) { float a, b; unpack(v, a, b); return b; }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 max2(f2 a, f2 b) { return pack(fmaxf(low(a), low(b)), fmaxf(high(a), high(b))); }

// 2^(v - b - 99) for v >= b, b whole numbers, v - b < 200, given m = MAGIC - b: v rounded to a whole number leaves a rest of at
// most 1/2, whose power is a polynomial of degree 6 (fitted for the smallest largest relative error, 3e-9; with the roundings
// 2.6e-8 root mean square, 6.6e-8 at most: ex2.approx errs by three times that, which was half of the error of a gradient);
// the whole number goes to the exponent as it is.
constexpr float MAGIC = 12582912.0f;               // 1.5 2^23
__device__ __forceinline__ f2 exp2_from(f2 v, f2 m) {
    constexpr float S = 1.5777218104420236e-30f;   // 2^-99
    const f2 r = add2(v, m), f = add2(v, fma2(r, both(-1.0f), m));
    f2 h = fma2(both(0x1.416b50p-13f * S), f, both(0x1.5f082ep-10f * S));
    h = fma2(h, f, both(0x1.3b2de0p-7f * S));
    h = fma2(h, f, both(0x1.c6af7cp-5f * S));
    h = fma2(h, f, both(0x1.ebfbdcp-3f * S));
    h = fma2(h, f, both(0x1.62e430p-1f * S));
    h = fma2(h, f, both(S));
    return pack(__int_as_float(__float_as_int(low(h)) + (__float_as_int(low(r)) << 23)),
                __int_as_float(__float_as_int(high(h)) + (__float_as_int(high(r)) << 23)));
}
// The same with the special-function unit for the rest, given m = MAGIC - 99 - b: 12 cycles less of the FMA pipe a pair, and an
// error of 5e-8, which gradients have room for (3 % faster; the forward 5 %, but with errors above those of the kernels before).
__device__ __forceinline__ f2 exp2_unit(f2 v, f2 m) {
    const f2 r = add2(v, m), f = add2(v, fma2(r, both(-1.0f), m));
    float a, b;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(low(f)));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(high(f)));
    return pack(__int_as_float(__float_as_int(a) + (__float_as_int(low(r)) << 23)), __int_as_float(__float_as_int(b) + (__float_as_int(high(r)) << 23)));
}
// N columns of this thread's row, pairs.
template <int N>
__device__ __forceinline__ void ld_cols(uint32_t addr, f2 (&v)[N / 2]) {
    if constexpr (N == 64) {
        float x[64];
        tmem_ld64(addr, x);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = pack(x[2 * i], x[2 * i + 1]);
    } else if constexpr (N == 32) {
        float x[32];
        tmem_ld32(addr, x);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = pack(x[2 * i], x[2 * i + 1]);
    } else if constexpr (N == 8) {
        uint32_t r[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr) : "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = pack(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
    } else {
        float x[16];
        tmem_ld16(addr, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = pack(x[2 * i], x[2 * i + 1]);
    }
}
#define BMB_R16(r) "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), \
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
__device__ __forceinline__ void pairs16(f2 (&v)[8], const uint32_t (&r)[16]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = pack(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
// 16 columns from each of two places, one wait.
__device__ __forceinline__ void ld_cols16x2(uint32_t a, uint32_t b, f2 (&x)[8], f2 (&y)[8]) {
    uint32_t r[16], q[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : BMB_R16(r), BMB_R16(q) : "r"(a), "r"(b) : "memory");
    pairs16(x, r);
    pairs16(y, q);
}
// 16 columns of scores; HALVES: the sum of the head's two halves, 64 columns apart.
template <bool HALVES>
__device__ __forceinline__ void ld_scores(uint32_t addr, f2 (&v)[8]) {
    if constexpr (HALVES) {
        f2 x[8];
        ld_cols16x2(addr, addr + 64, v, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = add2(v[i], x[i]);
    } else {
        ld_cols<16>(addr, v);
    }
}
// The larger of m and 16 values.
__device__ __forceinline__ float max16(float m, const f2 (&v)[8]) {
    float b = m;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        m = fmax3(m, low(v[i]), high(v[i]));
        b = fmax3(b, low(v[i + 1]), high(v[i + 1]));
    }
    return fmaxf(m, b);
}
__device__ __forceinline__ void st8(uint32_t addr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// 16 weights of this thread's row, below 2^16, as pieces over the 16 columns at `addr`.  (Complete after tmem_wait_st().)
__device__ __forceinline__ void put_weights(uint32_t addr, const f2 *p) {
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const __half2 h = __floats2half2_rn(low(p[i]), high(p[i]));
        const f2 rest = mul2(fma2(pack(__low2float(h), __high2float(h)), both(-1.0f), p[i]), both(2048.0f));
        const __half2 l = __floats2half2_rn(low(rest), high(rest));
        hi[i] = *reinterpret_cast<const uint32_t *>(&h);
        lo[i] = *reinterpret_cast<const uint32_t *>(&l);
    }
    st8(addr, hi);
    st8(addr + 8, lo);
}
// acc += g * the N columns at `addr`.
template <int N>
__device__ __forceinline__ void drain(uint32_t addr, f2 (&acc)[N / 2], float g) {
    constexpr int W = N >= 32 ? 32 : N;
#pragma unroll
    for (int c = 0; c < N; c += W) {
        f2 v[W / 2];
        ld_cols<W>(addr + c, v);
#pragma unroll
        for (int i = 0; i < W / 2; ++i) acc[c / 2 + i] = fma2(v[i], both(g), acc[c / 2 + i]);
    }
}
// A warp's 32 rows x N columns, f each, from registers (a row a thread) through `stage` (32 x N floats) to rows of pitch ld;
// rows from `valid` on are left out.
template <int N>
__device__ __forceinline__ void store_tile(uint8_t *stage, float *dst, long long ld, int valid, const f2 (&v)[N / 2], float f) {
    const int lane = threadIdx.x & 31;
    constexpr int U = N / 4, RPI = 32 / U;                  // 16-byte units of a row; rows an instruction of the warp stores
    constexpr int MASK = U < 8 ? U - 1 : 7;
#pragma unroll
    for (int u = 0; u < U; ++u)
        *reinterpret_cast<float4 *>(stage + (lane * U + (u ^ (lane & MASK))) * 16) = make_float4(low(v[2 * u]) * f, high(v[2 * u]) * f, low(v[2 * u + 1]) * f, high(v[2 * u + 1]) * f);
    __syncwarp();
#pragma unroll 4
    for (int i = 0; i < U; ++i) {
        const int r = i * RPI + lane / U, u = lane % U;
        if (r < valid) *reinterpret_cast<float4 *>(dst + r * ld + u * 4) = *reinterpret_cast<const float4 *>(stage + (r * U + (u ^ (r & MASK))) * 16);
    }
    __syncwarp();
}

// ---- forward ---------------------------------------------------------------------------------------------------------
// A CTA has 256 queries of one head, two tiles of 128; keys come 64 at a time.
//   warps 0-7, 8-15  a tile's softmax: half of a query's 64 scores a thread, from tensor memory, weights back over them as pieces,
//                    half of the columns of the sums of the step before added to fp32 registers;
//   warp 16          copies the tiles and, in the order of their use (S 0, S 1, P V 0, S 2, P V 1, ..), blocks of K and V;
//   warps 17, 18     issue a tile's products.
template <int HS> struct Fwd {
    using G = Geo<HS>;
    static constexpr int STAGES = HS == 128 ? 3 : 6;
    // Tensor memory, 256 columns a tile: two buffers of 64 scores and two of sums.  At 128 columns one buffer of each: the scores'
    // two halves of the head are summed apart (eight products in a row err too much), and the sums take 128 columns.
    static constexpr bool HALVES = HS == 128;
    static constexpr int BUFS = HALVES ? 1 : 2;
    static constexpr int OFF_RING = 2 * G::TILE, OFF_TOP = OFF_RING + STAGES * G::BLK;
    static constexpr int OFF_BAR = OFF_TOP + BUFS * 2048, SMEM = OFF_BAR + 256;          // (tops: [buffer][tile][half][row])
};

template <int HS>
__global__ void __launch_bounds__(THREADS, 1)
flash_fwd_x2_k(float *__restrict__ out, float *__restrict__ lse, const Images im, int T, int NH, int BH, int nblk, int span, Factors fac, int *__restrict__ status) {
    using G = Geo<HS>;
    using F = Fwd<HS>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t base = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + F::OFF_BAR);
    enum { Q_FULL = 0, FULL = 2, EMPTY = FULL + F::STAGES, S_FULL = EMPTY + F::STAGES, P_FULL = S_FULL + 4, PV_DONE = P_FULL + 4, O_FREE = PV_DONE + 4,
           NBARS = O_FREE + 4 };
    static_assert(NBARS * 8 + 8 <= 256, "barriers");
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + NBARS);
    volatile int *giveup = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [bar0](int i) { return bar0 + 8u * (uint32_t)i; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bh = blockIdx.x, q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * span;       // longest first
    if (threadIdx.x == 0) {
        for (int t = 0; t < 2; ++t) mbar_init(bar(Q_FULL + t), 1);
        for (int s = 0; s < F::STAGES; ++s) { mbar_init(bar(FULL + s), 1); mbar_init(bar(EMPTY + s), 2); }
        for (int i = 0; i < 4; ++i) { mbar_init(bar(S_FULL + i), 1); mbar_init(bar(P_FULL + i), 8); mbar_init(bar(PV_DONE + i), 1); mbar_init(bar(O_FREE + i), 8); }
        *giveup = 0;
        mbar_init_fence();
    }
    if (warp == W_COPY) tmem_alloc(smem_u32(tmem_slot), 512);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    wait_for_predecessor();                                  // the images are there
    const bool left = any_flag(im.flags + (long long)bh * 3 * nblk, 3 * nblk);            // this head is flash.cu's

    int steps[2];                                            // blocks of keys that a tile sees
#pragma unroll
    for (int t = 0; t < 2; ++t) steps[t] = 128 * t < span && q0 + 128 * t < T ? (min(T, q0 + 128 * t + 128) + XB - 1) / XB : 0;
    const int nsteps = max(steps[0], steps[1]);

    if (left) {
        if (threadIdx.x == 0) im.left.flagged[bh] = 1;
    } else if (warp >= W_COPY) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_OTHER));
        if (warp == W_COPY && elect_one()) {
            const uint8_t *q = im.img + (long long)bh * nblk * G::BLK, *k = q + (long long)BH * nblk * G::BLK, *v = k + (long long)BH * nblk * G::BLK;
            bool ok = true;
            int item = 0, armed_to = 0;
            auto copy = [&](const uint8_t *blocks, int blk) {
                const int s = item % F::STAGES;
                if (!ok || !mbar_wait(bar(EMPTY + s), (uint32_t)(item / F::STAGES & 1) ^ 1u, giveup)) { ok = false; return; }
                mbar_arrive_expect_tx(bar(FULL + s), G::BLK);
                bulk_copy(base + F::OFF_RING + s * G::BLK, blocks + (long long)blk * G::BLK, G::BLK, bar(FULL + s));
                armed_to = ++item;
            };
            for (int t = 0; t < 2; ++t) {
                if (!steps[t]) continue;
                mbar_arrive_expect_tx(bar(Q_FULL + t), tile_bytes<HS>(q0 / XB + 2 * t, nblk));
                copy_tile<HS>(base + t * G::TILE, q, q0 / XB + 2 * t, nblk, bar(Q_FULL + t));
                if (t == 0) copy(k, 0);
            }
            for (int e = 0; ok && e < nsteps; ++e) {
                if (e + 1 < nsteps) copy(k, e + 1);
                copy(v, e);
            }
            if (!ok) {
                for (int t = 0; t < 2; ++t) if (steps[t]) mbar_drain(bar(Q_FULL + t), 0);
                for (int i = max(0, armed_to - F::STAGES); i < armed_to; ++i) mbar_drain(bar(FULL + i % F::STAGES), (uint32_t)(i / F::STAGES & 1));
            }
        } else if ((warp == W_ISSUE || warp == W_ISSUE + 1) && elect_one()) {
            const int t = warp - W_ISSUE, mine = t ? steps[1] : steps[0];
            const uint32_t q = base + t * G::TILE, s_tmem = tmem + (uint32_t)(256 * t), o_tmem = s_tmem + 128;
            bool ok = mine == 0 || mbar_wait(bar(Q_FULL + t), 0, giveup);
            int item = 0;
            auto slot = [&]() { return base + F::OFF_RING + (uint32_t)(item % F::STAGES * G::BLK); };
            auto arrived = [&]() { return ok = ok && mbar_wait(bar(FULL + item % F::STAGES), (uint32_t)(item / F::STAGES & 1), giveup); };
            auto release = [&]() { commit(bar(EMPTY + item % F::STAGES)); ++item; };
            // blocks past this tile's diagonal are waited for and released, so that both issuers' releases stay in one phase
            auto scores = [&](int e) {
                if (!arrived()) return;
                fence_after();
                if (e < mine) {
                    const uint32_t d = s_tmem + (uint32_t)(e % F::BUFS * 64);
                    if constexpr (F::HALVES) { issue_scores<HS, 4, 8>(d + 64, q, slot()); issue_scores<HS, 0, 4>(d, q, slot()); }
                    else issue_scores<HS>(d, q, slot());
                    commit(bar(S_FULL + 2 * t + (e & 1)));
                }
                release();
            };
            // P of step e is there, and the sums that its product overwrites have been taken
            auto weights = [&](int e) {
                const int f = e - F::BUFS;
                ok = ok && mbar_wait(bar(P_FULL + 2 * t + (e & 1)), (uint32_t)(e >> 1 & 1), giveup) &&
                     (f < 0 || mbar_wait(bar(O_FREE + 2 * t + (f & 1)), (uint32_t)(f >> 1 & 1), giveup));
                fence_after();
                return ok;
            };
            auto sums = [&](int e, uint32_t v) {
                issue_sum<HS>(o_tmem + (uint32_t)(e % F::BUFS * HS), s_tmem + (uint32_t)(e % F::BUFS * 64), v);
                commit(bar(PV_DONE + 2 * t + (e & 1)));
            };
            if (nsteps > 0) scores(0);
            for (int e = 0; ok && e < nsteps; ++e) {
                if constexpr (F::HALVES) {
                    // The scores' second half goes to columns that P has been read from, the first over P itself, behind P V.
                    const bool more = e + 1 < nsteps;
                    const uint32_t k = slot();
                    const int kslot = item % F::STAGES;
                    if (more && !arrived()) break;
                    if (e < mine) {
                        if (!(ok = mbar_wait(bar(P_FULL + 2 * t + (e & 1)), (uint32_t)(e >> 1 & 1), giveup))) break;
                        fence_after();
                        if (e + 1 < mine) issue_scores<HS, 4, 8>(s_tmem + 64, q, k);
                    }
                    if (more) ++item;
                    if (!arrived()) break;
                    if (e < mine) {
                        if (e > 0 && !(ok = mbar_wait(bar(O_FREE + 2 * t + ((e - 1) & 1)), (uint32_t)((e - 1) >> 1 & 1), giveup))) break;
                        fence_after();
                        sums(e, slot());
                    }
                    release();
                    if (more) {
                        if (e + 1 < mine) {
                            issue_scores<HS, 0, 4>(s_tmem, q, k);
                            commit(bar(S_FULL + 2 * t + ((e + 1) & 1)));
                        }
                        commit(bar(EMPTY + kslot));
                    }
                } else {
                    if (e + 1 < nsteps) scores(e + 1);
                    if (!arrived()) break;
                    if (e < mine) {
                        if (!weights(e)) break;
                        sums(e, slot());
                    }
                    release();
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_COMPUTE));
        const int t = warp >> 3, half = warp >> 2 & 1, quad = warp & 3, row = quad * 32 + lane;
        const int mine = t ? steps[1] : steps[0], first = q0 + 128 * t, qi = first + row;
        constexpr int H = HS / 2;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16, s_addr = tmem + (uint32_t)(256 * t + 32 * half) + lanes;
        const uint32_t o_addr = tmem + (uint32_t)(256 * t + 128 + H * half) + lanes;
        float *tops = reinterpret_cast<float *>(smem + F::OFF_TOP) + t * 256 + row;
        const float *uk = im.unscale + ((long long)BH + bh) * nblk, *uv = uk + (long long)BH * nblk;
        const float cq = im.unscale[(long long)bh * nblk + min(q0 / XB + 2 * t + (row >> 6), nblk - 1)] * LOG2E;
        f2 o[H / 2];
        float m = 0.0f, l = 0.0f;
#pragma unroll
        for (int i = 0; i < H / 2; ++i) o[i] = 0ull;
        bool ok = true;
        auto take = [&](int e) {                             // the sums of step e
            const float g = __ldg(uv + e);
            if (!ok || !warp_wait(bar(PV_DONE + 2 * t + (e & 1)), (uint32_t)(e >> 1 & 1), giveup)) { ok = false; return; }
            fence_after();
            drain<H>(o_addr + (uint32_t)(e % F::BUFS * HS), o, g);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(O_FREE + 2 * t + (e & 1)));
        };
        for (int e = 0; e < mine; ++e) {
            const float c = __ldg(uk + e) * cq;
            ok = ok && warp_wait(bar(S_FULL + 2 * t + (e & 1)), (uint32_t)(e >> 1 & 1), giveup);
            fence_after();
            const uint32_t sa = s_addr + (uint32_t)(e % F::BUFS * 64);
            // 32 of the 64 columns, 16 at a time
            const int k0 = e * XB + 32 * half;
            const bool edge = k0 + 31 > first;
            auto scores = [&](int j, f2 (&s)[8]) {
                ld_scores<F::HALVES>(sa + 16 * j, s);
                if (edge) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int k = k0 + 16 * j + 2 * i;
                        s[i] = pack(k > qi ? -INFINITY : low(s[i]), k + 1 > qi ? -INFINITY : high(s[i]));
                    }
                }
            };
            f2 s[2][8];
            float top = -INFINITY;
            if (ok) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    scores(j, s[j]);
                    top = max16(top, s[j]);
                }
            }
            // the row's other half: one buffer is enough where the next scores wait for these weights
            float *at = tops + e % F::BUFS * 512;
            at[half * 128] = top;
            ok = pair_all(t, ok);
            if (!ok) break;
            top = fmaxf(top, at[(half ^ 1) * 128]) * c;      // key 0 is visible to every row: finite in step 0
            // The reference of the exponentials, a whole number two below the maximum (where most of a row's weight is, exponents
            // are small and rounded little), follows it in jumps of more than 2^4, so most steps rescale nothing.  Weights are
            // 2^9 times their exponentials: at most 2^15, and a quarter more where scores are large (MOST_SCORE).
            float alpha = 1.0f;
            if (e == 0) {
                m = ceilf(top) - 2.0f;
                if (m < -MOST_SCORE) l = NAN;                // (told at the end)
            } else if (top > m + 6.0f) { const float to = ceilf(top) - 2.0f; alpha = exp2f(m - to); m = to; }
            f2 sum = 0ull;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (F::HALVES) scores(j, s[j]);              // (again: there are no registers to keep them in)
#pragma unroll
                for (int i = 0; i < 8; ++i) s[j][i] = exp2_from(max2(fma2(s[j][i], both(c), both(-m)), both(-108.0f)), both(MAGIC + 108.0f));
                put_weights(sa + 16 * j, s[j]);
                sum = add2(sum, add2(add2(add2(s[j][0], s[j][1]), add2(s[j][2], s[j][3])), add2(add2(s[j][4], s[j][5]), add2(s[j][6], s[j][7]))));
            }
            l = fmaf(l, alpha, low(sum) + high(sum));
            tmem_wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(P_FULL + 2 * t + (e & 1)));
            if (e > 0) take(e - 1);
            if (__any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll
                for (int i = 0; i < H / 2; ++i) o[i] = mul2(o[i], both(alpha));
            }
        }
        if (mine > 0) {                                      // (also who has given up: the barrier is the whole tile's)
            take(mine - 1);
            float *at = tops + mine % F::BUFS * 512;
            at[half * 128] = l;
            ok = pair_all(t, ok);
            l += at[(half ^ 1) * 128];
        }
        if (ok && mine > 0) {
            // (every product that reads this tile's queries has retired)
            const int b = bh / NH, h = bh % NH, C = NH * HS;
            const float inv = 1.0f / l;
#pragma unroll
            for (int i = 0; i < H / 2; ++i) {                // o (1 + sums) / l, rounded once
                const f2 y = mul2(o[i], both(inv));
                o[i] = fma2(fma2(y, both(-l), o[i]), both(inv), mul2(y, both(fac.sums)));
                o[i] = add2(y, o[i]);
            }
            store_tile<H>(smem + warp * (32 * H * 4), out + ((long long)b * T + first + quad * 32) * C + h * HS + half * H, C, T - first - quad * 32, o, 1.0f);
            if ((m > MOST_SCORE || l != l) && qi < T) im.left.flagged[bh] = 1;          // (m never falls)
            if (half == 0 && qi < T) lse[(long long)bh * T + qi] = fmaf(m, INV_LOG2E, fmaf(m, INV_LOG2E_REST, logf(l * 1.953125e-3f)));
        }
    }

    fence_before();
    __syncthreads();
    if (warp == W_COPY) {
        fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && *giveup) {
        *reinterpret_cast<volatile int *>(status) = 4;
        __threadfence_system();
    }
}

// ---- backward --------------------------------------------------------------------------------------------------------
// A CTA has 128 rows of one head, of keys (KV: dV = P^T dO, dK = dS^T Q) or of queries (dQ = dS K), and walks the other side
// 64 columns at a time:
//   S = A1 B1^T, dP = A2 B2^T; KV: sum2 = P B2; sum1 = dS B1       (A1, A2, B1, B2: K, V, Q, dO or Q, dO, K, V)
template <int HS> struct Bwd {
    using G = Geo<HS>;
    static constexpr int N1 = HS == 128 ? 2 : 4, N2 = HS == 128 ? 1 : 3;     // ring slots of B1 and of B2
    // Tensor memory: S and dP, two buffers of 64 columns each or, at 128 columns, one with the two halves of the head apart.
    static constexpr bool HALVES = HS == 128;
    static constexpr int BUFS = HALVES ? 1 : 2;
    static constexpr int OFF_B1 = 2 * G::TILE, OFF_B2 = OFF_B1 + N1 * G::BLK, OFF_ROWS = OFF_B2 + N2 * G::BLK, OFF_OWN = OFF_ROWS + N2 * ROWS_BYTES;
    static constexpr int OFF_BAR = OFF_OWN + 128 * 4;      // (OFF_OWN: what a row's dS is scaled by in its own block)
    static constexpr int SMEM = OFF_BAR + 256;
    static_assert(N1 >= BUFS && N2 >= BUFS, "a step's blocks stay until its sums are done");
};

template <int HS, bool KV>
__device__ __forceinline__ void bwd_x2(uint8_t *smem, float *__restrict__ dqkv, const Images &im, int T, int NH, int BH, int nblk, int bh, int r0,
                                       Factors fac, int *__restrict__ status) {
    using G = Geo<HS>;
    using F = Bwd<HS>;
    const uint32_t base = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + F::OFF_BAR);
    enum { A_FULL = 0, FULL1 = 2, EMPTY1 = FULL1 + F::N1, FULL2 = EMPTY1 + F::N1, EMPTY2 = FULL2 + F::N2, S_FULL = EMPTY2 + F::N2, DP_FULL = S_FULL + 2,
           W_FULL = DP_FULL + 2, DONE1 = W_FULL + 2, DONE2 = DONE1 + 2, FREE1 = DONE2 + 2, FREE2 = FREE1 + 2, NBARS = FREE2 + 2 };
    static_assert(NBARS * 8 + 8 <= 256, "barriers");
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + NBARS);
    volatile int *giveup = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [bar0](int i) { return bar0 + 8u * (uint32_t)i; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int t = 0; t < 2; ++t) mbar_init(bar(A_FULL + t), 1);
        for (int s = 0; s < F::N1; ++s) { mbar_init(bar(FULL1 + s), 1); mbar_init(bar(EMPTY1 + s), 1); }
        for (int s = 0; s < F::N2; ++s) { mbar_init(bar(FULL2 + s), 1); mbar_init(bar(EMPTY2 + s), 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar(S_FULL + i), 1); mbar_init(bar(DP_FULL + i), 1);
            mbar_init(bar(W_FULL + i), 8);
            mbar_init(bar(DONE1 + i), 1); mbar_init(bar(DONE2 + i), 1);
            mbar_init(bar(FREE1 + i), 16); mbar_init(bar(FREE2 + i), 16);
        }
        *giveup = 0;
        mbar_init_fence();
    }
    if (warp == W_COPY) tmem_alloc(smem_u32(tmem_slot), 512);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    wait_for_predecessor();                                  // the images are there
    const bool left = any_flag(im.flags + (long long)bh * 4 * nblk, 4 * nblk);            // this head is flash.cu's
    constexpr uint32_t COL_DP = 128, COL_1 = 256, COL_2 = 256 + HS;          // S 2 x 64, dP 2 x 64, sum1, sum2

    // column blocks: KV: queries from this tile's first key on; else keys up to this tile's last query
    const int c0 = KV ? r0 / XB : 0, n = (KV ? nblk : min(nblk, r0 / XB + 2)) - c0;
    const long long side = (long long)BH * nblk, head = (long long)bh * nblk;
    constexpr int WA1 = KV ? 1 : 0, WA2 = KV ? 2 : 3, WB1 = KV ? 0 : 1, WB2 = KV ? 3 : 2;

    if (left) {
        if (threadIdx.x == 0) im.left.flagged[bh] = 1;
    } else if (warp >= W_COPY) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_OTHER));
        if (warp == W_COPY && elect_one()) {
            auto blocks = [&](int which) { return im.img + (which * side + head) * G::BLK; };
            bool ok = true;
            int i1 = 0, i2 = 0;
            auto copy1 = [&]() {
                const int s = i1 % F::N1;
                if (!ok || !mbar_wait(bar(EMPTY1 + s), (uint32_t)(i1 / F::N1 & 1) ^ 1u, giveup)) { ok = false; return; }
                mbar_arrive_expect_tx(bar(FULL1 + s), G::BLK);
                bulk_copy(base + F::OFF_B1 + s * G::BLK, blocks(WB1) + (long long)(c0 + i1) * G::BLK, G::BLK, bar(FULL1 + s));
                ++i1;
            };
            auto copy2 = [&]() {
                const int s = i2 % F::N2;
                if (!ok || !mbar_wait(bar(EMPTY2 + s), (uint32_t)(i2 / F::N2 & 1) ^ 1u, giveup)) { ok = false; return; }
                mbar_arrive_expect_tx(bar(FULL2 + s), G::BLK + (KV ? ROWS_BYTES : 0));
                if (KV) bulk_copy(base + F::OFF_ROWS + s * ROWS_BYTES, im.rows + (head + c0 + i2) * (3 * XB), ROWS_BYTES, bar(FULL2 + s));
                bulk_copy(base + F::OFF_B2 + s * G::BLK, blocks(WB2) + (long long)(c0 + i2) * G::BLK, G::BLK, bar(FULL2 + s));
                ++i2;
            };
            const uint32_t tb = tile_bytes<HS>(r0 / XB, nblk);
            mbar_arrive_expect_tx(bar(A_FULL), tb);
            copy_tile<HS>(base, blocks(WA1), r0 / XB, nblk, bar(A_FULL));
            copy1();
            mbar_arrive_expect_tx(bar(A_FULL + 1), tb);
            copy_tile<HS>(base + G::TILE, blocks(WA2), r0 / XB, nblk, bar(A_FULL + 1));
            for (int e = 0; ok && e < n; ++e) {
                copy2();
                if (e + 1 < n) copy1();
            }
            if (!ok) {
                for (int t = 0; t < 2; ++t) mbar_drain(bar(A_FULL + t), 0);
                for (int i = max(0, i1 - F::N1); i < i1; ++i) mbar_drain(bar(FULL1 + i % F::N1), (uint32_t)(i / F::N1 & 1));
                for (int i = max(0, i2 - F::N2); i < i2; ++i) mbar_drain(bar(FULL2 + i % F::N2), (uint32_t)(i / F::N2 & 1));
            }
        } else if (warp == W_ISSUE && elect_one()) {
            bool ok = mbar_wait(bar(A_FULL), 0, giveup);
            bool second = false;                              // the second tile has been waited for
            auto slot1 = [&](int e) { return base + F::OFF_B1 + (uint32_t)(e % F::N1 * G::BLK); };
            auto slot2 = [&](int e) { return base + F::OFF_B2 + (uint32_t)(e % F::N2 * G::BLK); };
            auto scores = [&](uint32_t d, int e, uint32_t tile, uint32_t blk) {
                if constexpr (F::HALVES) { issue_scores<HS, 0, 4>(d, tile, blk); issue_scores<HS, 4, 8>(d + 64, tile, blk); }
                else issue_scores<HS>(d + (uint32_t)(e % F::BUFS * 64), tile, blk);
            };
            auto S = [&](int e) {
                if (!ok || e >= n) return;
                if (!mbar_wait(bar(FULL1 + e % F::N1), (uint32_t)(e / F::N1 & 1), giveup)) { ok = false; return; }
                fence_after();
                scores(tmem, e, base, slot1(e));
                commit(bar(S_FULL + (e & 1)));
            };
            auto dP = [&](int e) {
                if (!ok || e >= n) return;
                if (!second && !mbar_wait(bar(A_FULL + 1), 0, giveup)) { ok = false; return; }
                second = true;
                if (!mbar_wait(bar(FULL2 + e % F::N2), (uint32_t)(e / F::N2 & 1), giveup)) { ok = false; return; }
                fence_after();
                scores(tmem + COL_DP, e, base + G::TILE, slot2(e));
                commit(bar(DP_FULL + (e & 1)));
                if (!KV) commit(bar(EMPTY2 + e % F::N2));
            };
            auto sum2 = [&](int e) {
                if (!KV || !ok) return;
                if (e > 0 && !mbar_wait(bar(FREE2 + ((e - 1) & 1)), (uint32_t)((e - 1) >> 1 & 1), giveup)) { ok = false; return; }
                fence_after();
                issue_sum<HS>(tmem + COL_2, tmem + (uint32_t)(e % F::BUFS * 64), slot2(e));
                commit(bar(DONE2 + (e & 1)));
                commit(bar(EMPTY2 + e % F::N2));
            };
            auto sum1 = [&](int e) {
                if (!ok) return;
                if (e > 0 && !mbar_wait(bar(FREE1 + ((e - 1) & 1)), (uint32_t)((e - 1) >> 1 & 1), giveup)) { ok = false; return; }
                fence_after();
                issue_sum<HS>(tmem + COL_1, tmem + COL_DP + (uint32_t)(e % F::BUFS * 64), slot1(e));
                commit(bar(DONE1 + (e & 1)));
                commit(bar(EMPTY1 + e % F::N1));
            };
            // Products of one thread retire in order, so a buffer's next product needs no barrier for the one that read it.
            for (int e = 0; e < F::BUFS; ++e) { S(e); dP(e); }
            for (int e = 0; ok && e < n; ++e) {
                if (!mbar_wait(bar(W_FULL + (e & 1)), (uint32_t)(e >> 1 & 1), giveup)) break;
                sum2(e);
                sum1(e);
                S(e + F::BUFS);
                dP(e + F::BUFS);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_COMPUTE));
        // Two pairs of warpgroups take the steps in turn, a warpgroup half of its columns; each adds a quarter of the columns of
        // every step's sums to registers.
        const int w = warp >> 3, half = warp >> 2 & 1, quad = warp & 3, row = quad * 32 + lane, ri = r0 + row;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16;
        constexpr int H = HS / 4;
        f2 acc1[H / 2], acc2[KV ? H / 2 : 1];
#pragma unroll
        for (int i = 0; i < H / 2; ++i) acc1[i] = 0ull;
#pragma unroll
        for (int i = 0; i < (KV ? H / 2 : 1); ++i) acc2[i] = 0ull;
        const float *u1 = im.unscale + WB1 * side + head + c0, *u2 = im.unscale + WB2 * side + head + c0;
        const int rb = min(r0 / XB + (row >> 6), nblk - 1);
        const float ca1 = im.unscale[WA1 * side + head + rb] * LOG2E;
        const float ca2 = im.unscale[WA2 * side + head + rb];
        const float *mine = im.rows + (head + rb) * (3 * XB) + (row & 63);
        const float lr = KV ? 0.0f : mine[0], lb = KV ? 0.0f : mine[XB], drow = KV ? 0.0f : mine[2 * XB], vmost = lb + (WINDOW + 0.5f);
        // late: a probability beyond sqrt(2), of an lse that is not these scores'.  The queries' side looks, before exponents so far above 0
        // run over; the keys' side has the same pairs, and the head is computed again for both.
        bool ok = true, late = false;
        // dS of a row and a step is scaled so that it is at most 2^15.5 whatever the data: by 1 / (the largest that dP and D can be there, of
        // the row itself and of the columns that it sees; not below 2^-60 of all columns', so that the others stay finite).
        const float4 *tops = im.tops + head + c0;
        const float dtop = KV ? 0.0f : fmaxf(top_of(top_code(drow)), TINY);
        float own, *own_block = reinterpret_cast<float *>(smem + F::OFF_OWN) + row;
        {
            // largest of what a row sees in its own block: a queries' row V up to it, a keys' row dO and D from it on
            const uint8_t *pt = im.ptops + (head + rb) * (3 * XB) + (KV ? XB : 0);
            auto code = [&](int r) { return KV ? pt[r] | (uint32_t)pt[XB + r] << 16 : (uint32_t)pt[r]; };
            const int hb = quad & 1;                         // the row's half of the block
            uint32_t sees = code(hb * 32 + lane), other = hb != KV ? code((hb ^ 1) * 32 + lane) : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t next = KV ? __shfl_down_sync(0xffffffffu, sees, o) : __shfl_up_sync(0xffffffffu, sees, o);
                if (KV ? lane + o < 32 : lane >= o) sees = max_u16x2(sees, next);
                other = max_u16x2(other, __shfl_xor_sync(0xffffffffu, other, o));
            }
            sees = max_u16x2(sees, other);
            const float4 b = im.tops[head + rb];
            own = top_of(KV ? pt[(row & 63) - XB] : pt[(row & 63) + XB]) * HS;
            const float of_row = KV ? TINY : dtop, all = KV ? fmaxf(own * b.y, b.z) : own * b.x;
            // (four threads write what each of them reads)
            *own_block = fmaxf(fmaxf(own * top_of(sees & 255u), KV ? top_of(sees >> 16) : 0.0f), fmaxf(of_row, all * 8.6736174e-19f));
        }
        auto bound = [&](int e) {
            const float4 b = __ldg(tops + e);
            return e == rb - c0 ? *own_block : KV ? fmaxf(own * b.y, b.z) : fmaxf(own * b.x, dtop);
        };
        constexpr float DOWN = 6.103515625e-5f;              // 2^-14
        float carried = 0.0f;
        auto take1 = [&](int e, float bnd) {
            if (!ok || e < 0) return;
            const float g = __ldg(u1 + e) * (DOWN * bnd);
            if (!warp_wait(bar(DONE1 + (e & 1)), (uint32_t)(e >> 1 & 1), giveup)) { ok = false; return; }
            fence_after();
            drain<H>(tmem + COL_1 + lanes + (uint32_t)((warp >> 2) * H), acc1, g);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(FREE1 + (e & 1)));
        };
        auto take2 = [&](int e) {
            if constexpr (KV) {
                if (!ok || e < 0) return;
                const float g = __ldg(u2 + e) * DOWN;
                if (!warp_wait(bar(DONE2 + (e & 1)), (uint32_t)(e >> 1 & 1), giveup)) { ok = false; return; }
                fence_after();
                drain<H>(tmem + COL_2 + lanes + (uint32_t)((warp >> 2) * H), acc2, g);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(FREE2 + (e & 1)));
            }
        };
        for (int e = w; e < n; e += 2) {
            // the sums of this warpgroup's last step, in order
            take2(e - 2);
            take1(e - 2, carried);
            if (!ok) break;
            carried = bound(e);
            const float g = __uint_as_float(0x7f000000u - __float_as_uint(carried)), cs = __ldg(u1 + e) * ca1, cp = __ldg(u2 + e) * ca2 * g;
            const int col0 = (c0 + e) * XB + 32 * half;
            if (!warp_wait(bar(S_FULL + w), (uint32_t)(e >> 1 & 1), giveup) || !warp_wait(bar(DP_FULL + w), (uint32_t)(e >> 1 & 1), giveup)) { ok = false; break; }
            fence_after();
            const uint32_t sa = tmem + lanes + (uint32_t)(e % F::BUFS * 64 + 32 * half), da = sa + COL_DP;
            const float4 *cols = reinterpret_cast<const float4 *>(smem + F::OFF_ROWS + e % F::N2 * ROWS_BYTES) + 8 * half;
            const bool edge = KV ? col0 < r0 + 127 : col0 + 31 > r0;
            auto mask = [&](int j, f2 (&p)[8], float with) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int k = col0 + j + 2 * i;
                    p[i] = pack((KV ? k < ri : k > ri) ? with : low(p[i]), (KV ? k + 1 < ri : k + 1 > ri) ? with : high(p[i]));
                }
            };
            // 16 columns at a time, so that the loop stays in the instruction cache and its registers are few
            auto weights = [&](int j, f2 (&p)[8], const f2 (&d)[8]) {
                // p = 2^14 2^(S - lse): lse's whole part goes to the exponent (exp2_from), so nothing is rounded at its size.
                float vtop = -INFINITY;
                if (!KV && edge) mask(j, p, -INFINITY);
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    float4 r = make_float4(lr, lr, lr, lr), b = make_float4(lb, lb, lb, lb);
                    if (KV) { r = cols[(j + 2 * i) / 4]; b = cols[16 + (j + 2 * i) / 4]; }
                    const f2 b0 = pack(b.x, b.y), b1 = pack(b.z, b.w);
                    p[i] = max2(fma2(p[i], both(cs), pack(r.x, r.y)), b0);
                    p[i + 1] = max2(fma2(p[i + 1], both(cs), pack(r.z, r.w)), b1);
                    if (!KV) vtop = fmax3(fmax3(vtop, low(p[i]), high(p[i])), low(p[i + 1]), high(p[i + 1]));
                    p[i] = exp2_unit(p[i], fma2(b0, both(-1.0f), both(MAGIC - 99.0f)));
                    p[i + 1] = exp2_unit(p[i + 1], fma2(b1, both(-1.0f), both(MAGIC - 99.0f)));
                }
                if (!KV) late = late || vtop > vmost;
                if (KV && edge) mask(j, p, 0.0f);
                if (KV) put_weights(sa + j, p);
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    float4 D = make_float4(drow, drow, drow, drow);
                    if (KV) D = cols[32 + (j + 2 * i) / 4];
                    p[i] = mul2(p[i], fma2(d[i], both(cp), mul2(pack(D.x, D.y), both(-g))));
                    p[i + 1] = mul2(p[i + 1], fma2(d[i + 1], both(cp), mul2(pack(D.z, D.w), both(-g))));
                }
                put_weights(da + j, p);
            };
#pragma unroll 1
            for (int j = 0; j < 32; j += 16) {
                f2 p[8], d[8];
                ld_scores<F::HALVES>(sa + j, p);
                ld_scores<F::HALVES>(da + j, d);
                weights(j, p, d);
            }
            tmem_wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(W_FULL + w));
            take2(e - 1);
            take1(e - 1, e > 0 ? bound(e - 1) : 0.0f);
        }
        // steps n - 2 and n - 1, as far as this warpgroup has not taken their sums
        const bool last = ((n - 1) & 1) == w;                // this warpgroup's own last step is n - 1 (and took n - 2)
        if (!last) { take2(n - 2); if (n > 1) take1(n - 2, bound(n - 2)); }
        take2(n - 1);
        take1(n - 1, bound(n - 1));
        if (!KV && late && ri < T) im.left.flagged[bh] = 1;
        if (ok) {
            // every product has retired: the tiles' memory is free
            const int b = bh / NH, h = bh % NH, C = NH * HS, valid = T - r0 - quad * 32;
            const long long ld = 3LL * C;
            uint8_t *stage = smem + warp * (32 * H * 4);
            float *dst = dqkv + ((long long)b * T + r0 + quad * 32) * ld + (KV ? C : 0) + h * HS + (warp >> 2) * H;
            store_tile<H>(stage, dst, ld, valid, acc1, KV ? fac.dk : fac.dq);
            if constexpr (KV) store_tile<H>(stage, dst + C, ld, valid, acc2, fac.dv);
        }
    }

    fence_before();
    __syncthreads();
    if (warp == W_COPY) {
        fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && *giveup) {
        *reinterpret_cast<volatile int *>(status) = 4;
        __threadfence_system();
    }
}

template <int HS>
__global__ void __launch_bounds__(THREADS, 1)
flash_bwd_x2_k(float *__restrict__ dqkv, const Images im, int T, int NH, int BH, int nblk, Factors fac, int *__restrict__ status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int bh = blockIdx.x, rank = blockIdx.y >> 1, tiles = gridDim.y >> 1;
    if (blockIdx.y & 1) bwd_x2<HS, false>(smem, dqkv, im, T, NH, BH, nblk, bh, (tiles - 1 - rank) * 128, fac, status);
    else bwd_x2<HS, true>(smem, dqkv, im, T, NH, BH, nblk, bh, rank * 128, fac, status);
}

// Once per kernel and device: shared memory above 48 KB, and whether the registers that a block is launched with cover what its
// warpgroups ask for (setmaxnreg would wait for them for good).
int prepare(const void *kernel, int bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, int> done;
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(kernel, current_device());
    const auto it = done.find(key);
    if (it != done.end()) return it->second;
    cudaFuncAttributes at;
    BMB_CUDA(cudaFuncGetAttributes(&at, kernel));
    BMB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    return done[key] = at.numRegs * THREADS >= REGS_COMPUTE * COMPUTE + REGS_OTHER * 128 ? BMB_OK : BMB_E_UNSUPPORTED;
}

struct Layout { size_t images, unscale, flags, left_out, rows, tops, ptops, total; };
Layout layout(long long BH, int nblk, int HS, int nw) {
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    const size_t blocks = (size_t)BH * nblk;
    Layout L;
    L.images = up(blocks * nw * XB * HS * 4);
    L.unscale = up(blocks * nw * 4);
    L.flags = up(blocks * nw);
    L.left_out = up((size_t)BH + 4);
    L.rows = nw == 4 ? up(blocks * ROWS_BYTES) : 0;
    L.tops = nw == 4 ? up(blocks * sizeof(float4)) : 0;
    L.ptops = nw == 4 ? up(blocks * 3 * XB) : 0;
    L.total = L.images + L.unscale + L.flags + L.left_out + L.rows + L.tops + L.ptops;
    return L;
}
constexpr size_t KEPT = CALL_SCRATCH_KEPT;          // bytes of images at a time (or one head's)

struct Call {
    float *out, *lse, *dqkv, *dsum;
    const float *qkv, *dout;
    int B, T, NH;
    float scale;
};

// Heads whose images lie in `scr`: the head `a` points at and those behind it.
template <int HS, bool BACKWARD>
int launch_x2(const Call &a, int BH, int span, uint8_t *scr, int *status_dev, cudaStream_t st) {
    const int nblk = ceil_div(a.T, XB), nw = BACKWARD ? 4 : 3, smem = BACKWARD ? Bwd<HS>::SMEM : Fwd<HS>::SMEM;
    const Layout L = layout(BH, nblk, HS, nw);
    Images im;
    im.img = scr;
    im.unscale = (float *)(scr + L.images);
    im.flags = scr + L.images + L.unscale;
    im.left = LeftOut{im.flags + L.flags + 4, (int *)(im.flags + L.flags), BH};
    im.rows = (float *)(im.flags + L.flags + L.left_out);
    im.tops = (float4 *)(im.flags + L.flags + L.left_out + L.rows);
    im.ptops = im.flags + L.flags + L.left_out + L.rows + L.tops;
    const double cut = (HS == 32 ? 2 : 4) * CUT, sums = 4 * CUT, q = a.scale * (1.0 + cut);      // products in a row
    Factors fac;
    fac.q = (float)q;
    fac.q_rest = (float)(q - fac.q);
    fac.dp = (float)cut;
    fac.sums = (float)sums;
    fac.dk = (float)(a.scale / q * (1.0 + cut) * (1.0 + sums));
    fac.dq = (float)(a.scale * (1.0 + cut) * (1.0 + sums));
    fac.dv = (float)(1.0 + sums);
    split_x2_k<HS><<<(unsigned)((long long)BH * nblk * nw), 256, 0, st>>>(im, a.dsum, a.qkv, a.dout, a.out, a.lse, a.T, a.NH, BH, nblk, nw, fac);
    count_launch();
    BMB_LAUNCH_CHECK();
    const dim3 grid((unsigned)BH, BACKWARD ? 2 * ceil_div(a.T, 128) : ceil_div(a.T, span));
    if (BACKWARD) {
        BMB_TRY(launch_in_chain(flash_bwd_x2_k<HS>, grid, THREADS, smem, st, a.dqkv, im, a.T, a.NH, BH, nblk, fac, status_dev));
        return flash_bwd_left(HS, a.dqkv, a.dsum, a.dout, a.qkv, a.lse, a.T, a.NH, a.scale, im.left, st);
    }
    BMB_TRY(launch_in_chain(flash_fwd_x2_k<HS>, grid, THREADS, smem, st, a.out, a.lse, im, a.T, a.NH, BH, nblk, span, fac, status_dev));
    return flash_fwd_left(HS, a.out, a.lse, a.qkv, a.T, a.NH, a.scale, im.left, st);
}

template <int HS, bool BACKWARD>
int run_x2(const Call &a, bool in_trainer, cudaStream_t st) {
    const int nblk = ceil_div(a.T, XB), nw = BACKWARD ? 4 : 3;
    // Images of more than KEPT bytes are made and used one after the other: of some of the sequences, or of some of a sequence's heads.
    const size_t head = layout(1, nblk, HS, nw).total, fit = std::max<size_t>(1, KEPT / head);
    int nb = (int)std::min<size_t>(a.B, fit / a.NH), nh = a.NH;
    if (nb) nb = ceil_div(a.B, ceil_div(a.B, nb));           // (parts of one size)
    else { nb = 1; nh = ceil_div(a.NH, ceil_div(a.NH, (long long)fit)); }
    // A CTA's two tiles of queries share its keys and hide each other's latency, but one is faster alone where SMs are free.
    const long long BH = (long long)nb * nh;
    const int span = BH * ceil_div(a.T, 256) <= sm_count() * 9 / 10 ? 128 : 256;
    if ((BACKWARD ? 2 * ceil_div(a.T, 128) : ceil_div(a.T, span)) > 65535 || BH * nblk * nw >= (1LL << 31)) return BMB_E_UNSUPPORTED;
    // A captured launch would carry the scratch's address.
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (!in_trainer && (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)) {
        cudaGetLastError();
        return BMB_E_UNSUPPORTED;
    }
    BMB_TRY(prepare(BACKWARD ? (const void *)flash_bwd_x2_k<HS> : (const void *)flash_fwd_x2_k<HS>, BACKWARD ? Bwd<HS>::SMEM : Fwd<HS>::SMEM));
    const size_t bytes = layout(BH, nblk, HS, nw).total;
    if (bytes > (16ull << 30)) return BMB_E_UNSUPPORTED;
    int *status_dev = nullptr;
    volatile int *status_host = nullptr;
    BMB_TRY(status_word(&status_dev, &status_host));
    if (*status_host != 0) return fail(BMB_E_TIMEOUT, "an earlier kernel on this device gave up waiting on a barrier");
    // A trainer's launches use the block that its captured steps hold, other calls one of their own.
    std::unique_lock<std::mutex> turn(split_mutex(), std::defer_lock);
    if (in_trainer) turn.lock();
    uint8_t *scr = (uint8_t *)(in_trainer ? split_scratch(bytes, st) : call_scratch(bytes, st));
    if (!scr) return BMB_E_UNSUPPORTED;
    struct Done {
        uint8_t *scr;
        cudaStream_t st;
        bool in_trainer;
        ~Done() { if (in_trainer) scratch_release(SCR_SPLIT, st); else call_scratch_done(scr, st); }
    };
    const Done done{scr, st, in_trainer};
    if (in_trainer) BMB_TRY(scratch_acquire(SCR_SPLIT, st));
    for (int b = 0; b < a.B; b += nb)
        for (int h = 0; h < a.NH; h += nh) {
            const long long C = (long long)a.NH * HS, x = b * (C * a.T) + (long long)h * HS, x3 = b * (3 * C * a.T) + (long long)h * HS;
            const long long row = ((long long)b * a.NH + h) * a.T;
            const Call part{a.out + x, a.lse + row, BACKWARD ? a.dqkv + x3 : nullptr, BACKWARD ? a.dsum + row : nullptr, a.qkv + x3,
                            BACKWARD ? a.dout + x : nullptr, a.B, a.T, a.NH, a.scale};
            BMB_TRY((launch_x2<HS, BACKWARD>(part, std::min(nb, a.B - b) * std::min(nh, a.NH - h), span, scr, status_dev, st)));
        }
    return BMB_OK;
}

}  // namespace

// BMB_E_UNSUPPORTED: nothing was launched.
int flash_forward_x2(float *out, float *lse, const float *qkv, int B, int T, int NH, int hs, float scale, bool in_trainer, cudaStream_t st) {
    const Call a{out, lse, nullptr, nullptr, qkv, nullptr, B, T, NH, scale};
    return hs == 32 ? run_x2<32, false>(a, in_trainer, st) : hs == 64 ? run_x2<64, false>(a, in_trainer, st) : run_x2<128, false>(a, in_trainer, st);
}
int flash_backward_x2(float *dqkv, float *dsum, const float *dout, const float *qkv, const float *out, const float *lse, int B, int T, int NH, int hs,
                      float scale, bool in_trainer, cudaStream_t st) {
    const Call a{const_cast<float *>(out), const_cast<float *>(lse), dqkv, dsum, qkv, dout, B, T, NH, scale};
    return hs == 32 ? run_x2<32, true>(a, in_trainer, st) : hs == 64 ? run_x2<64, true>(a, in_trainer, st) : run_x2<128, true>(a, in_trainer, st);
}

}  // namespace bmb
