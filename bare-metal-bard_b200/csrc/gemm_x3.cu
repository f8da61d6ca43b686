// fp32 products on the tensor cores: every fp32 operand as three bf16 pieces, x = b1 + b2 + b3.
//
//   b1 = bf16(x), b2 = bf16(x - b1), b3 = bf16(x - b1 - b2)      (each difference is exact)
//
// Three pieces hold all 24 bits of x, so  a b = sum over i + j <= 4 of a_i b_j  up to 2^-26 of |a b|: six bf16
// products (kind::f16, fp32 accumulators) stand for one fp32 product.  The tensor core does not round its running
// sums but cuts them off, which over a long K costs far more than the pieces do (1.6e-8 of the sum per instruction:
// 1e-4 at K = 50 000).  So a sum stays in tensor memory for one slice of 32 K only -- small terms first, the two
// instructions of b1 b1 last, so that only those meet a sum of full size -- and is then added, rounded, to
// accumulators in the epilogue warps' registers, while the next slice is multiplied into the other buffer.
// Against a 64-bit product this is closer than the sequential multiply-adds of the SIMT kernels at every size it
// takes (uniform operands, 2-norm: K = 16 4.9e-8 against 7.4e-8, 1024 1.2e-7 against 5.7e-7, 8192 2.2e-7 against 1.6e-6).
//
// Measured on B200, split pass included, SIMT kernels -> this: 4096^3 2445 -> 585 us (235 TFLOP/s of fp32 products),
// 8192x3072x768 (NT) 747 -> 178, 768x768x8192 (TN) 658 -> 76, 8192x50304x768 (NT) 11.5 -> 2.6 ms.
//
// Two or three launches: split_x3_k writes both operands as images of the slices the product reads, gemm_x3_k
// multiplies, and where K is shared among CTAs reduce_x3_k adds the parts in a fixed order (no atomics: two calls
// give the same bits).
//
// Image of an operand of R rows (whatever its transposition, the split pass turns it): [K/32][3 pieces][Rp rows]
// of 64-byte rows (32 bf16 of K) in the 64-byte swizzle that the matrix descriptor names, so that one piece of
// one slice of a tile is one contiguous bulk copy and needs no tensor map.  K and the rows of the
// last tile are filled up with zeros.
//
// What the pieces cannot serve is not stored but computed again by the sequential fp32 chain from the original operands:
// behind the last product of a CTA, when no barrier is waited for any more, in blocks by all its threads, or in the pass that
// adds the parts.
//   Sums that are not finite: a_i b_j of the pieces of an infinite operand gives NaN where the fp32 product is infinite,
//   and a sum may overflow in another order.
//   Panels of 64 rows (or columns) with an element that has bits below 2^-133, the smallest bf16 number (elements below
//   about 2^-109): the split pass notes where three pieces do not add up to the element.
//   Sums below 2^-100.
// 4096^3: 575 us; with one infinity in A 1.8 ms, with one in every row 5.5 (SIMT kernels 2.4).
// 2-norm errors at K = 512, this against the SIMT kernels: 0.95e-7 and 4.1e-7 with A and B of ordinary size and with A 2^-108
// and B 2^108 times that; the same bits from 2^-110 on.
#include "tc_common.cuh"
#include <cuda_bf16.h>
#include <mutex>
#include <type_traits>

namespace bmb {
using namespace tc;
namespace {

constexpr int XK = 32;                      // K per slice
constexpr int ROWB = XK * 2;                // bytes per image row
constexpr int XM = 128;                     // rows of a tile
constexpr int XA_BYTES = 3 * XM * ROWB;     // 24 KB per slice
constexpr int X_THREADS = 320;              // producer warp, issuer warp, 8 epilogue warps
__host__ __device__ constexpr int x_stage_bytes(int bn) { return XA_BYTES + 3 * bn * ROWB; }
__host__ __device__ constexpr int x_stages(int bn) { return bn >= 192 ? 3 : bn == 128 ? 4 : 5; }
__host__ __device__ constexpr int x_smem_bytes(int bn) { return x_stages(bn) * x_stage_bytes(bn) + 1024 + 256; }

__host__ __device__ inline long long round_up(long long a, long long b) { return (a + b - 1) / b * b; }

struct Operand {
    const float *src;
    uint8_t *img;
    int rows, rows_pad;           // R and the image's rows
    int k_contig;                 // 1: element (r, k) at r * K + k; 0: at k * R + r
    int panels, kgroups;          // work split: panels of 64 rows, groups of KG slices
    uint8_t *lost;                // [panels][kgroups, filled up to words]: an element of the block has bits that its pieces do not hold
};
constexpr int KG = 4;             // slices a block of the split pass takes one after the other

// `lost` gets bits where the pieces do not add up: a bit of x or y lies below bf16's smallest number (or it is not finite).
__device__ __forceinline__ void split3(float x, float y, uint32_t &p1, uint32_t &p2, uint32_t &p3, uint32_t &lost) {
    constexpr float BMAX = 3.3895313892515355e38f;      // largest bf16: above it the first piece must not become infinite
    const __nv_bfloat162 a = __floats2bfloat162_rn(fminf(fmaxf(x, -BMAX), BMAX), fminf(fmaxf(y, -BMAX), BMAX));
    const float rx = x - __low2float(a), ry = y - __high2float(a);
    const __nv_bfloat162 b = __floats2bfloat162_rn(rx, ry);
    const float sx = rx - __low2float(b), sy = ry - __high2float(b);
    const __nv_bfloat162 c = __floats2bfloat162_rn(sx, sy);
    lost |= __float_as_uint(sx - __low2float(c)) | __float_as_uint(sy - __high2float(c));
    p1 = *reinterpret_cast<const uint32_t *>(&a);
    p2 = *reinterpret_cast<const uint32_t *>(&b);
    p3 = *reinterpret_cast<const uint32_t *>(&c);
}

// Bound by memory: 4 bytes read and 6 written per element.  A thread turns 8 K-neighbours of one row into one
// 16-byte unit of each piece; a warp's stores are 512 contiguous bytes per piece.  Operands with K contiguous are
// read where they lie, the others go through shared memory (64 rows x 32 K at a time).
__global__ void __launch_bounds__(256) split_x3_k(const Operand a, const Operand b, long long blocks_a, int K, int vec_a, int vec_b) {
    __shared__ float tile[XK][65];
    const bool first = (long long)blockIdx.x < blocks_a;
    const Operand &o = first ? a : b;
    const int vec = first ? vec_a : vec_b;
    const long long id = (long long)blockIdx.x - (first ? 0 : blocks_a);
    const int panel = (int)(id % o.panels), kgroup = (int)(id / o.panels);
    const float *src = o.src;
    uint8_t *img = o.img;
    const int row_in = threadIdx.x >> 2, unit = threadIdx.x & 3;
    const int r = panel * 64 + row_in;
    const int nslices = (K + XK - 1) / XK;
    uint32_t lost = 0;
    for (int ks = kgroup * KG; ks < nslices && ks < (kgroup + 1) * KG; ++ks) {
        float v[8];
        const int k0 = ks * XK + unit * 8;
        if (o.k_contig) {
            const float *p = src + (long long)r * K + k0;
            if (r < o.rows && vec && k0 + 8 <= K) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(p)), y = __ldg(reinterpret_cast<const float4 *>(p) + 1);
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = (r < o.rows && k0 + i < K) ? __ldg(p + i) : 0.0f;
            }
        } else {
            __syncthreads();                       // the previous slice has been read
            const int c = (threadIdx.x & 15) * 4, rr = panel * 64 + c;
#pragma unroll
            for (int j = 0; j < XK; j += 16) {
                const int k = ks * XK + j + (threadIdx.x >> 4);
                const float *p = src + (long long)k * o.rows + rr;
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k < K) {
                    if (vec && rr + 4 <= o.rows) x = __ldg(reinterpret_cast<const float4 *>(p));
                    else {
                        if (rr < o.rows) x.x = __ldg(p);
                        if (rr + 1 < o.rows) x.y = __ldg(p + 1);
                        if (rr + 2 < o.rows) x.z = __ldg(p + 2);
                        if (rr + 3 < o.rows) x.w = __ldg(p + 3);
                    }
                }
                float *t = &tile[j + (threadIdx.x >> 4)][c];
                t[0] = x.x; t[1] = x.y; t[2] = x.z; t[3] = x.w;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = tile[unit * 8 + i][row_in];
        }
        uint32_t p1[4], p2[4], p3[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split3(v[2 * i], v[2 * i + 1], p1[i], p2[i], p3[i], lost);
        const long long piece = (long long)o.rows_pad * ROWB;
        uint8_t *d = img + (long long)ks * 3 * piece + (long long)r * ROWB + ((unit ^ ((r >> 1) & 3)) << 4);
        *reinterpret_cast<uint4 *>(d) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
        *reinterpret_cast<uint4 *>(d + piece) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
        *reinterpret_cast<uint4 *>(d + 2 * piece) = make_uint4(p3[0], p3[1], p3[2], p3[3]);
    }
    lost = __syncthreads_or(lost != 0);
    const int words = (o.kgroups + 3) / 4, i = kgroup + (int)threadIdx.x;     // the last block clears the rest of its word
    if (threadIdx.x == 0 || (kgroup == o.kgroups - 1 && i < 4 * words)) o.lost[(long long)panel * words * 4 + i] = threadIdx.x == 0 && lost;
}

// What a product needs besides the images: where the operands lie (for elements computed again) and the result.
struct Result {
    const float *A, *B;
    int ta, tb, M, N, K;
    float alpha, beta;
    float *C;
    const float *bias;             // added to every row, or null
    const uint32_t *lostA, *lostB; // Operand::lost, `words` a panel
    int words;
};
// Word i of what says whether panel a of A, and panels b, b + 1, .. of B, lost bits.
__device__ __forceinline__ const uint32_t *lost_word(const Result &p, int a, int b, int i) {
    return i < p.words ? p.lostA + (long long)a * p.words + i : p.lostB + (long long)b * p.words + (i - p.words);
}
__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) <= 3.402823466e38f); }
// A sum that is not taken: not finite, or so small that what the tensor core cuts off below the smallest fp32 number,
// up to 2^-149 an instruction, is more than a rounding of it.
constexpr float TOO_SMALL = 7.8886090522101181e-31f;     // 2^-100
__device__ __forceinline__ bool doubtful(float x) { return not_finite(x) || (fabsf(x) < TOO_SMALL && x != 0.0f); }
__device__ __forceinline__ void store_element(const Result &p, int m, int n, float s) {
    float *c = p.C + (size_t)m * p.N + n;
    float o = p.alpha * s;
    if (p.beta != 0.0f) o = fmaf(p.beta, *c, o);
    *c = p.bias ? o + p.bias[n] : o;
}
// Out of line: a call in the middle of the 128 sums of an epilogue thread would cost registers that there are not.
__device__ __noinline__ void put_element(const Result &p, int m, int n, float s) { store_element(p, m, n, s); }

// 128 x 64 elements by the sequential chain over k, as the SIMT kernels have it.  Thread 16 y + x of the first 256 has rows
// m0 + 8 y .. and columns n0 + 4 x ..; every thread of the block calls it.
constexpr int TM = 8, CN = 64, CK = 32, C_THREADS = 256;
struct ChainTile { float a[CK][16 * TM + 4], b[CK][CN + 4]; };
// X rows (or columns) x 32 k of an operand, on the way from global to shared memory: 8 neighbours in memory a thread and trip.
template <int X>
struct ChainSlice {
    static constexpr int TRIPS = X * CK / 8 / C_THREADS;
    float v[TRIPS][8];
    static __device__ __forceinline__ void place(int trip, bool kc, int &x, int &k) {
        const int lin = trip * C_THREADS + (int)threadIdx.x;
        x = kc ? lin % X : lin % (X / 8) * 8;
        k = kc ? lin / X * 8 : lin / (X / 8);
    }
    __device__ __forceinline__ void read(const float *src, bool kc, bool vec, int x0, int xe, int k0, int ke) {
#pragma unroll
        for (int r = 0; r < TRIPS; ++r) {
            int x, k;
            place(r, kc, x, k);
            x += x0; k += k0;
            const float *s = src + (kc ? (long long)x * ke + k : (long long)k * xe + x);
            if (vec && x + (kc ? 1 : 8) <= xe && k + (kc ? 8 : 1) <= ke) {
                const float4 lo = __ldg(reinterpret_cast<const float4 *>(s)), hi = __ldg(reinterpret_cast<const float4 *>(s) + 1);
                v[r][0] = lo.x; v[r][1] = lo.y; v[r][2] = lo.z; v[r][3] = lo.w;
                v[r][4] = hi.x; v[r][5] = hi.y; v[r][6] = hi.z; v[r][7] = hi.w;
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[r][i] = x + (kc ? 0 : i) < xe && k + (kc ? i : 0) < ke ? __ldg(s + i) : 0.0f;
            }
        }
    }
    __device__ __forceinline__ void put(float (*d)[X + 4], bool kc) const {
#pragma unroll
        for (int r = 0; r < TRIPS; ++r) {
            int x, k;
            place(r, kc, x, k);
            if (kc) {
#pragma unroll
                for (int i = 0; i < 8; ++i) d[k + i][x] = v[r][i];
            } else {
                *reinterpret_cast<float4 *>(&d[k][x]) = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
                *reinterpret_cast<float4 *>(&d[k][x + 4]) = make_float4(v[r][4], v[r][5], v[r][6], v[r][7]);
            }
        }
    }
};
__device__ __forceinline__ void chain_block(float (&acc)[TM][4], const Result &from, int m0, int n0, ChainTile &t) {
    const Result p = from;                          // in registers (behind the reference it is read again after each barrier)
    const int tid = threadIdx.x;
    const bool works = tid < C_THREADS, kca = !p.ta, kcb = p.tb != 0;
    const bool veca = ((uintptr_t)p.A & 15) == 0 && (kca ? p.K : p.M) % 4 == 0, vecb = ((uintptr_t)p.B & 15) == 0 && (kcb ? p.K : p.N) % 4 == 0;
    ChainSlice<16 * TM> a;
    ChainSlice<CN> b;
    unsigned long long sum[TM][2];                  // two columns each: an instruction follows two chains
#pragma unroll
    for (int i = 0; i < TM; ++i) sum[i][0] = sum[i][1] = 0ull;
    if (works) { a.read(p.A, kca, veca, m0, p.M, 0, p.K); b.read(p.B, kcb, vecb, n0, p.N, 0, p.K); }
    for (int k0 = 0; k0 < p.K; k0 += CK) {
        __syncthreads();                            // the slice before has been read
        if (works) { a.put(t.a, kca); b.put(t.b, kcb); }
        __syncthreads();
        if (!works) continue;
        if (k0 + CK < p.K) { a.read(p.A, kca, veca, m0, p.M, k0 + CK, p.K); b.read(p.B, kcb, vecb, n0, p.N, k0 + CK, p.K); }
#pragma unroll 8
        for (int k = 0; k < CK; ++k) {
            float x[TM];
#pragma unroll
            for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4 *>(x + i) = *reinterpret_cast<const float4 *>(&t.a[k][tid / 16 * TM + i]);
            const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(&t.b[k][tid % 16 * 4]);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                unsigned long long xx;
                asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(x[i]));
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[i][0]) : "l"(xx), "l"(y.x));
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[i][1]) : "l"(xx), "l"(y.y));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; j += 2) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i][j]), "=f"(acc[i][j + 1]) : "l"(sum[i][j / 2]));
}
// The parts of a tile (128 rows, two halves of half_cols columns) that its epilogue warps left out: byte 4 * half + quarter
// of `left` stands for 32 rows of one half.  (The tile lies in dynamic shared memory, 16 bytes aligned at `at`; named here
// and not handed over, so that it is read as such.)
__device__ __noinline__ void tile_again(const Result &p, int m0, int n0, int half_cols, unsigned long long left, int at) {
    extern __shared__ uint8_t smem_raw[];
    ChainTile &t = *reinterpret_cast<ChainTile *>(smem_raw + at);
    auto missing = [&](int row, int col) { return (left >> (8 * (4 * (col / half_cols) + row / 32)) & 1) != 0; };
    for (int c = 0; c < 2 * half_cols; c += CN) {
        const int last = c + CN - 1;
        bool any = false;
        for (int r = 0; r < XM; r += 32) any = any || missing(r, c) || missing(r, last);
        if (!any) continue;
        float acc[TM][4];
        chain_block(acc, p, m0, n0 + c, t);
        if (threadIdx.x >= C_THREADS) continue;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = (int)threadIdx.x / 16 * TM + i, col = c + (int)threadIdx.x % 16 * 4 + j;
                if (m0 + row < p.M && n0 + col < p.N && missing(row, col)) store_element(p, m0 + row, n0 + col, acc[i][j]);
            }
    }
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Items (tile, part of K), part-major, dealt round-robin: CTAs work at about the same depth of K.
struct XIter {
    int tiles_m, tiles_n, tiles, total, parts, kblocks, grid, i;
    __device__ __forceinline__ void init(int tm_, int tn_, int parts_, int kblocks_) {
        tiles_m = tm_; tiles_n = tn_; tiles = tm_ * tn_; parts = parts_; kblocks = kblocks_;
        total = tiles * parts_; grid = (int)gridDim.x; i = (int)blockIdx.x;
    }
    __device__ __forceinline__ bool next(int &tm, int &tn, int &part, int &kb0, int &kb1) {
        if (i >= total) return false;
        part = i / tiles;
        const int t = i - part * tiles;
        constexpr int GM = 8;                       // tiles of neighbouring rows share a panel of B in L2
        const int per_group = GM * tiles_n, g = t / per_group, first = g * GM;
        const int gsz = tiles_m - first < GM ? tiles_m - first : GM;
        const int r = t - g * per_group;
        tm = first + r % gsz;
        tn = r / gsz;
        kb0 = (int)((long long)part * kblocks / parts);
        kb1 = (int)((long long)(part + 1) * kblocks / parts);
        i += grid;
        return true;
    }
    __device__ __forceinline__ int item() const { return i - grid; }     // the last one that next() gave
};

// One persistent CTA per SM.  Bound by shared memory and the tensor pipe together: a slice of a 128 x 256 tile
// lands 72 KB and has 144 KB read by its 12 instructions of 128 cycles, 1690 cycles at 128 bytes a cycle against
// 1536 of the pipe.
//   warp 0     one lane copies slices into the ring (six contiguous copies per slice);
//   warp 1     one lane issues the 12 instructions of a slice into one of two accumulator buffers;
//   warps 2-9  add each finished buffer to their register accumulators (a lane quadrant and half of the columns
//              each) and store the tile; in the 16x256b shape four lanes hold 32 contiguous bytes of a row, so
//              the registers go to global memory in whole sectors.
template <int BN>
__global__ void __launch_bounds__(X_THREADS, 1)
gemm_x3_k(const uint8_t *__restrict__ imgA, int rowsA, const uint8_t *__restrict__ imgB, int rowsB, const Result p, int kblocks, int parts, float *__restrict__ ws, int vec, uint8_t *left, int *__restrict__ status) {
    constexpr int STAGES = x_stages(BN), STAGE = x_stage_bytes(BN), PA = XM * ROWB, PB = BN * ROWB;
    constexpr uint32_t ACC = BN == 192 ? 256 : BN, TCOLS = 2 * ACC;      // (allocations are powers of two)
    constexpr int NC = BN / 64;                     // 32-column chunks per epilogue warp (half of the columns)
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *gen = smem_raw + (base - smem_u32(smem_raw));
    uint64_t *bars = reinterpret_cast<uint64_t *>(gen + STAGES * STAGE);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 4);
    volatile int *giveup = reinterpret_cast<volatile int *>(tmem_slot + 1), *again = giveup + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * STAGES;
    const uint32_t tfull0 = empty0 + 8 * STAGES, tempty0 = tfull0 + 16;

    XIter it;
    it.init((p.M + XM - 1) / XM, (p.N + BN - 1) / BN, parts, kblocks);
    int tm, tn, part, kb0, kb1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(tfull0 + 8 * a, 1); mbar_init(tempty0 + 8 * a, 8); }
        *giveup = 0;
        *again = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), TCOLS);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            int armed[STAGES];
#pragma unroll
            for (int i = 0; i < STAGES; ++i) armed[i] = -1;
            const long long pieceA = (long long)rowsA * ROWB, pieceB = (long long)rowsB * ROWB;
            while (ok && it.next(tm, tn, part, kb0, kb1)) {
                const uint8_t *ga = imgA + (long long)tm * PA, *gb = imgB + (long long)tn * PB;
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(empty0 + 8 * s, ph ^ 1, giveup)) { ok = false; break; }
                    const uint32_t fb = full0 + 8 * s, sa = base + s * STAGE, sb = sa + XA_BYTES;
                    mbar_arrive_expect_tx(fb, STAGE);
#pragma unroll
                    for (int i = 0; i < STAGES; ++i) if (i == s) armed[i] = (int)ph;
                    // b1 last in use, first to arrive makes no difference: the slice is waited for as a whole
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        bulk_copy(sa + q * PA, ga + ((long long)kb * 3 + q) * pieceA, PA, fb);
                        bulk_copy(sb + q * PB, gb + ((long long)kb * 3 + q) * pieceB, PB, fb);
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
            if (!ok) {
#pragma unroll
                for (int i = 0; i < STAGES; ++i)
                    if (armed[i] >= 0) mbar_drain(full0 + 8 * i, (uint32_t)armed[i]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = make_idesc(1u, 0u, 0u, BN, XM);
            int s = 0, acc = 0;
            uint32_t ph = 0, acc_ph = 0;
            bool ok = true;
            while (ok && it.next(tm, tn, part, kb0, kb1)) {
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(tempty0 + 8 * acc, acc_ph ^ 1, giveup) || !mbar_wait(full0 + 8 * s, ph, giveup)) { ok = false; break; }
                    fence_after();
                    const uint32_t d = tmem_base + (uint32_t)acc * ACC;
                    const uint32_t sa = base + s * STAGE, sb = sa + XA_BYTES;
                    // pieces of A and B, smallest terms first
                    constexpr int TA[6] = {2, 0, 1, 1, 0, 0}, TB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
                    for (int t = 0; t < 6; ++t)
#pragma unroll
                        for (int k = 0; k < 2; ++k)
                            mma_f16(d, smem_desc(sa + TA[t] * PA + 32 * k, 16, 8 * ROWB, 4), smem_desc(sb + TB[t] * PB + 32 * k, 16, 8 * ROWB, 4),
                                    idesc, (t | k) ? 1u : 0u);
                    commit(empty0 + 8 * s);
                    commit(tfull0 + 8 * acc);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                    if (++acc == 2) { acc = 0; acc_ph ^= 1; }
                }
            }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2;
        int acc = 0;
        uint32_t acc_ph = 0;
        bool ok = true;
        while (ok && it.next(tm, tn, part, kb0, kb1)) {
            // this lane's share of the words on whether this warp's panels lost bits; asked for here (volatile), beside the first
            // products, and wanted at the end: at K up to 5000 a word a lane
            uint32_t lost = 0;
            {
                const int pa = (tm * XM + q * 32) / 64, pb = (tn * BN + half * (BN / 2)) / 64, nb = (tn * BN + half * (BN / 2) + BN / 2 - 1) / 64 - pb + 1;
                if (lane < (1 + nb) * p.words) asm volatile("ld.global.b32 %0, [%1];" : "=r"(lost) : "l"(lost_word(p, pa, pb, lane)));
                for (int i = lane + 32; i < (1 + nb) * p.words; i += 32) lost |= __ldg(lost_word(p, pa, pb, i));
            }
            float sum[NC][32];
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int i = 0; i < 32; ++i) sum[c][i] = 0.0f;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(tfull0 + 8 * acc, acc_ph, giveup)) { ok = false; break; }
                fence_after();
                const uint32_t trow = tmem_base + acc * ACC + half * (BN / 2) + ((uint32_t)(q * 32) << 16);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    float v[16];
                    tmem_ld_16x256b_x4_nowait(trow + (uint32_t)(c * 32), v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum[c][i] += v[i];
                    tmem_ld_16x256b_x4_nowait(trow + (uint32_t)(c * 32) + (16u << 16), v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum[c][16 + i] += v[i];
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
                if (++acc == 2) { acc = 0; acc_ph ^= 1; }
            }
            if (!ok) break;
            const int m0 = tm * XM + q * 32 + (lane >> 2), nb = tn * BN + half * (BN / 2) + 2 * (lane & 3);
            float *D = parts > 1 ? ws + (long long)part * p.M * p.N : p.C;
            const float alpha = parts > 1 ? 1.0f : p.alpha, beta = parts > 1 ? 0.0f : p.beta;
            const float *bias = parts > 1 ? nullptr : p.bias;
            // sum[c] of row m0 + 8k and columns nb + 32c + 8j, + 1
            auto value = [&](int c, int j, int k) { return make_float2(sum[c][(k >> 1) * 16 + 4 * j + 2 * (k & 1)], sum[c][(k >> 1) * 16 + 4 * j + 2 * (k & 1) + 1]); };
            // Nothing hides this end (the next tile's sums need these registers), so the common case is a multiply and a
            // store per pair: a whole tile, aligned, of whole operands, all sums finite and none too small.
            if (parts == 1) {
                float least = 1.0f, most = 0.0f;
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        asm("min.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(least) : "f"(sum[c][i]), "f"(sum[c][i + 1]));
                        asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(most) : "f"(sum[c][i]), "f"(sum[c][i + 1]));
                    }
                bool leave = lost != 0 || not_finite(most);
                if (least < TOO_SMALL) {                // (or there are zeros)
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i) leave = leave || doubtful(sum[c][i]);
                }
                leave = __any_sync(0xffffffffu, leave);
                if (lane == 0) {
                    left[(size_t)it.item() * 8 + 4 * half + q] = leave;
                    if (leave) *again = 1;
                }
                if (leave) continue;
            } else if (__any_sync(0xffffffffu, lost != 0)) {         // the pass that adds the parts computes these
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) sum[c][i] = __int_as_float(0x7fffffff);
            }
            if (vec && (tm + 1) * XM <= p.M && (tn + 1) * BN <= p.N) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float *row = D + (size_t)(m0 + 8 * k) * p.N + nb;
                    if (beta == 0.0f && !bias) {
#pragma unroll
                        for (int c = 0; c < NC; ++c)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 x = value(c, j, k);
                                *reinterpret_cast<float2 *>(row + c * 32 + 8 * j) = make_float2(alpha * x.x, alpha * x.y);
                            }
                    } else {
#pragma unroll
                        for (int c = 0; c < NC; ++c)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float2 x = value(c, j, k);
                                float2 *d = reinterpret_cast<float2 *>(row + c * 32 + 8 * j), o = make_float2(alpha * x.x, alpha * x.y);
                                if (beta != 0.0f) {
                                    const float2 old = *d;
                                    o.x = fmaf(beta, old.x, o.x);
                                    o.y = fmaf(beta, old.y, o.y);
                                }
                                if (bias) { o.x += __ldg(bias + nb + c * 32 + 8 * j); o.y += __ldg(bias + nb + c * 32 + 8 * j + 1); }
                                *d = o;
                            }
                    }
                }
            } else {
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int n = nb + c * 32 + 8 * j;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int m = m0 + 8 * k;
                            const float2 x = value(c, j, k);
                            if (m >= p.M || n >= p.N) continue;
                            const bool second = n + 1 < p.N;
                            float *d = D + (size_t)m * p.N + n;
                            if (parts > 1) {
                                d[0] = x.x;
                                if (second) d[1] = x.y;
                                continue;
                            }
                            // (256 columns: one sum more in registers than there are, so edges take the call, which is slow)
                            if (BN == 256) {
                                put_element(p, m, n, x.x);
                                if (second) put_element(p, m, n + 1, x.y);
                                continue;
                            }
                            float2 o = make_float2(alpha * x.x, alpha * x.y);
                            if (beta != 0.0f) {
                                o.x = fmaf(beta, d[0], o.x);
                                if (second) o.y = fmaf(beta, d[1], o.y);
                            }
                            if (bias) {
                                o.x += __ldg(bias + n);
                                if (second) o.y += __ldg(bias + n + 1);
                            }
                            if (vec) *reinterpret_cast<float2 *>(d) = o;        // (N is even: there is a second)
                            else { d[0] = o.x; if (second) d[1] = o.y; }
                        }
                    }
            }
        }
    }

    fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        fence_after();
        tmem_dealloc(tmem_base, TCOLS);
    }
    if (threadIdx.x == 0 && *giveup) {
        *reinterpret_cast<volatile int *>(status) = 1;
        __threadfence_system();
    }
    // (all products and copies are done: the ring is free)
    if (*again && !*giveup) {
        it.init((p.M + XM - 1) / XM, (p.N + BN - 1) / BN, parts, kblocks);
        while (it.next(tm, tn, part, kb0, kb1)) {
            const unsigned long long l = *reinterpret_cast<const volatile unsigned long long *>(left + (size_t)it.item() * 8);
            if (l) tile_again(p, tm * XM, tn * BN, BN / 2, l, (int)(gen - smem_raw));
        }
    }
}

// Those of four neighbouring elements of a row that `again` names, by the sequential chain.  16 neighbouring threads read the
// same values of A and neighbouring ones of B, four steps of k at a time.
__device__ __noinline__ void four_again(const Result &from, int m, int n, uint32_t again) {
    const Result p = from;
    const long long as = p.ta ? p.M : 1, bk = p.tb ? 1 : p.N, bn = p.tb ? p.K : 1;
    const float *a = p.A + (p.ta ? (long long)m : (long long)m * p.K), *b = p.B + n * bn;
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    auto steps = [&](int k, auto count) {
        constexpr int N = decltype(count)::value;
        float x[N], y[N][4];
#pragma unroll
        for (int q = 0; q < N; ++q) {
            x[q] = __ldg(a + (k + q) * as);
#pragma unroll
            for (int j = 0; j < 4; ++j) y[q][j] = n + j < p.N ? __ldg(b + (k + q) * bk + j * bn) : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < N; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[j] = fmaf(x[q], y[q][j], s[j]);
    };
    int k = 0;
    for (; k + 4 <= p.K; k += 4) steps(k, std::integral_constant<int, 4>());
    for (; k < p.K; ++k) steps(k, std::integral_constant<int, 1>());
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if ((again >> j & 1) && n + j < p.N) store_element(p, m, n + j, s[j]);
}
// The parts of a K shared among CTAs, added in order.
__global__ void __launch_bounds__(256) reduce_x3_k(const Result p, int parts, const float *__restrict__ ws, int vec4) {
    const long long n = (long long)p.M * p.N, step = (long long)gridDim.x * blockDim.x;
    if (vec4) {
        for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n / 4; e += step) {
            float4 s = __ldg(reinterpret_cast<const float4 *>(ws) + e);
            for (int q = 1; q < parts; ++q) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(ws + q * n) + e);
                s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
            }
            if (doubtful(s.x) || doubtful(s.y) || doubtful(s.z) || doubtful(s.w)) {
                const int row = (int)(4 * e / p.N), col = (int)(4 * e % p.N);
                const float v[4] = {s.x, s.y, s.z, s.w};
                uint32_t again = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    again |= (doubtful(v[i]) ? 1u : 0u) << i;
                    if (!(again >> i & 1)) put_element(p, row, col + i, v[i]);
                }
                four_again(p, row, col, again);
                continue;
            }
            float4 o = make_float4(p.alpha * s.x, p.alpha * s.y, p.alpha * s.z, p.alpha * s.w);
            float4 *cp = reinterpret_cast<float4 *>(p.C + 4 * e);
            if (p.beta != 0.0f) {
                const float4 old = *cp;
                o.x = fmaf(p.beta, old.x, o.x); o.y = fmaf(p.beta, old.y, o.y);
                o.z = fmaf(p.beta, old.z, o.z); o.w = fmaf(p.beta, old.w, o.w);
            }
            if (p.bias) {                           // N is a multiple of 4 here: the four are of one row
                const float *b = p.bias + (int)(4 * e % p.N);
                o.x += __ldg(b); o.y += __ldg(b + 1); o.z += __ldg(b + 2); o.w += __ldg(b + 3);
            }
            *cp = o;
        }
    } else {
        for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += step) {
            float s = ws[e];
            for (int q = 1; q < parts; ++q) s += ws[q * n + e];
            if (doubtful(s)) four_again(p, (int)(e / p.N), (int)(e % p.N), 1u);
            else put_element(p, (int)(e / p.N), (int)(e % p.N), s);
        }
    }
}

template <int BN>
int launch_x3(int grid, const uint8_t *imgA, int rowsA, const uint8_t *imgB, int rowsB, const Result &p, int kblocks, int parts, float *ws, int vec, uint8_t *left, int *status, cudaStream_t st) {
    static std::mutex mu;
    static bool set[64];
    const int d = current_device();
    if (d < 0 || d >= 64) return BMB_E_UNSUPPORTED;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!set[d]) {
            BMB_CUDA(cudaFuncSetAttribute(gemm_x3_k<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, x_smem_bytes(BN)));
            set[d] = true;
        }
    }
    gemm_x3_k<BN><<<grid, X_THREADS, x_smem_bytes(BN), st>>>(imgA, rowsA, imgB, rowsB, p, kblocks, parts, ws,
                                                             vec, left, status);
    return BMB_OK;
}

// A larger block is given back by the product that took it (unless a trainer keeps it): (M + N) K above 1.8e8, products of
// milliseconds.
constexpr size_t SPLIT_KEPT = 1ull << 30;

struct XPlan { int bn, parts; };
// Widths (us, 256 / 192 / 128 / 64 columns): 8192x768x768 70 / 62 / 75 / 118, 8192x2304x768 132 / 151 / 175 / 284,
// 4096x1536x384 42 / 37 / 44 / 64, 4096x1152x384 60 / 37 / 33 / 48, 512^3 23 / 22 / 21 / 19.
// Cycles of a plan: rounds of items over the SMs, each its slices plus the end that the next item's products do
// not hide, and the pass that adds the parts (its traffic stays in L2: about 3 KB a cycle, and a launch).
XPlan choose_x3(int units, int M, int N, int kblocks) {
    const int widths[4] = {256, 192, 128, 64};
    const double slice[4] = {1750, 1450, 1180, 880}, tail[4] = {1300, 1050, 800, 600};
    XPlan best{128, 1};
    double best_t = 1e300;
    for (int w = 0; w < 4; ++w) {
        const long long tiles = (long long)ceil_div(M, XM) * ceil_div(N, widths[w]);
        const bool ragged = M % XM || N % widths[w];
        for (int s = 1; s <= 16; ++s) {
            if (s > 1 && kblocks / s < 4) break;
            const double rounds = (double)ceil_div(tiles * s, units);
            double t = rounds * (ceil_div(kblocks, s) * slice[w] + tail[w]) + 3000;
            // the tile with an edge ends last, whatever their number (one size: 2000 x 2000 x 500 58 us, 42 with 128 columns)
            if (s == 1 && ragged && widths[w] == 256) t += 40000;
            if (s > 1) t += 4000 + (double)M * N * 4 * (2 * s + 1) / 3000;
            if (t < best_t) { best_t = t; best = {widths[w], s}; }
        }
    }
    return best;
}

}  // namespace

std::mutex &split_mutex() {
    static std::mutex mu[64];
    const int d = current_device();
    return mu[d >= 0 && d < 64 ? d : 0];
}

// Takes products of 2^18 results and more with K from 192, and of 2^31 multiply-adds and more with K from 128 (measured,
// SIMT against this: 1024x384x384 43 / 19 us, 4096x128x384 43 / 21, 4096x4096x128 89 / 76, but 2048x2048x128 29 / 33,
// 4096x384x128 17 / 19, 4096x4096x64 50 / 70; two launches and a pass over the operands cost about 13 us whatever the
// size).  Fewer results are left to the SIMT kernels although a long K would gain (256x256x1024 about 25 / 18 us): they are
// the products that callers compare, element by element, with the sequential fp32 chain, which the SIMT kernels follow bit
// for bit and this one does not.  A caller that says it does not (GEMM_ANY_ORDER: the trainer) has them from 2^14 results on.
// BMB_E_UNSUPPORTED: nothing launched, the product is the SIMT kernels' (also where there is no memory for the images).
int gemm_x3(int transA, int transB, int M, int N, int K, float alpha, const float *A, const float *B, float beta, float *C,
            const float *bias, int flags, cudaStream_t st) {
    if (M < 32 || N < 32) return BMB_E_UNSUPPORTED;
    if (!(K >= 128 && (double)M * N * K >= 2147483648.0) &&
        !(K >= 192 && (double)M * N >= ((flags & GEMM_ANY_ORDER) ? 16384.0 : 262144.0))) return BMB_E_UNSUPPORTED;
    // A captured launch would carry the scratch's address, and two captured branches would share it unordered.
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (!(flags & GEMM_SCRATCH_IN_CAPTURE) && (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)) {
        cudaGetLastError();
        return BMB_E_UNSUPPORTED;
    }
    if (M >= (1 << 29) || N >= (1 << 29)) return BMB_E_UNSUPPORTED;
    const int kblocks = ceil_div(K, XK);
    const XPlan plan = choose_x3(sm_count(), M, N, kblocks);
    const long long rowsA = round_up(M, XM), rowsB = round_up(N, plan.bn);
    const long long imgA = (long long)kblocks * 3 * rowsA * ROWB, imgB = (long long)kblocks * 3 * rowsB * ROWB;
    const long long ws = plan.parts > 1 ? (long long)plan.parts * M * N * 4 : 0;
    const long long tiles = (long long)ceil_div(M, XM) * ceil_div(N, plan.bn) * plan.parts;
    Operand oa{A, nullptr, M, (int)rowsA, transA ? 0 : 1, (int)(rowsA / 64), ceil_div(kblocks, KG), nullptr};
    Operand ob{B, nullptr, N, (int)rowsB, transB ? 1 : 0, (int)(rowsB / 64), ceil_div(kblocks, KG), nullptr};
    const long long na = (long long)oa.panels * oa.kgroups, nb = (long long)ob.panels * ob.kgroups;
    const int words = ceil_div(oa.kgroups, 4);
    const long long flagsA = 4LL * words * oa.panels, flagsB = 4LL * words * ob.panels;
    const long long marks = plan.parts > 1 ? 0 : 8 * tiles;
    const long long need = imgA + imgB + ws + marks + flagsA + flagsB;      // the images: multiples of 256 bytes (without parts there is no ws)
    if (tiles >= (1LL << 30) || na + nb >= (1LL << 31) || need > (16LL << 30)) return BMB_E_UNSUPPORTED;
    int *status_dev = nullptr;
    volatile int *status_host = nullptr;
    BMB_TRY(status_word(&status_dev, &status_host));
    if (*status_host != 0) return fail(BMB_E_TIMEOUT, "an earlier kernel on this device gave up waiting on a barrier");
    std::lock_guard<std::mutex> turn(split_mutex());
    uint8_t *scr = (uint8_t *)split_scratch((size_t)need, st);
    if (!scr) return BMB_E_UNSUPPORTED;
    oa.img = scr;
    ob.img = scr + imgA;
    float *w = (float *)(scr + imgA + imgB);
    uint8_t *left = scr + imgA + imgB;                    // 8 bytes a tile, where there are no parts
    oa.lost = scr + imgA + imgB + ws + marks;
    ob.lost = oa.lost + flagsA;

    auto vec_of = [](const float *p, int inner) { return ((uintptr_t)p & 15) == 0 && inner % 4 == 0; };
    const Result p{A, B, transA, transB, M, N, K, alpha, beta, C, bias, (const uint32_t *)oa.lost, (const uint32_t *)ob.lost, words};
    const bool even = N % 2 == 0 && (plan.parts > 1 || ((uintptr_t)C & 7) == 0);
    const int grid = (int)(tiles < sm_count() ? tiles : sm_count());
    BMB_TRY(scratch_acquire(SCR_SPLIT, st));
    split_x3_k<<<(unsigned)(na + nb), 256, 0, st>>>(oa, ob, na, K, vec_of(A, transA ? M : K), vec_of(B, transB ? K : N));
    int rc = BMB_OK;
    if (plan.bn == 256) rc = launch_x3<256>(grid, oa.img, (int)rowsA, ob.img, (int)rowsB, p, kblocks, plan.parts, w, even, left, status_dev, st);
    else if (plan.bn == 192) rc = launch_x3<192>(grid, oa.img, (int)rowsA, ob.img, (int)rowsB, p, kblocks, plan.parts, w, even, left, status_dev, st);
    else if (plan.bn == 128) rc = launch_x3<128>(grid, oa.img, (int)rowsA, ob.img, (int)rowsB, p, kblocks, plan.parts, w, even, left, status_dev, st);
    else rc = launch_x3<64>(grid, oa.img, (int)rowsA, ob.img, (int)rowsB, p, kblocks, plan.parts, w, even, left, status_dev, st);
    if (rc != BMB_OK) return rc;
    count_launch(2);
    if (plan.parts > 1) {
        const int vec4 = N % 4 == 0 && ((uintptr_t)C & 15) == 0;
        const long long blocks = ceil_div((long long)M * N, vec4 ? 1024 : 256);
        reduce_x3_k<<<(unsigned)(blocks < 8 * sm_count() ? blocks : 8 * sm_count()), 256, 0, st>>>(p, plan.parts, w, vec4);
        count_launch();
    }
    BMB_LAUNCH_CHECK();
    BMB_TRY(scratch_release(SCR_SPLIT, st));
    if (cs == cudaStreamCaptureStatusNone && !(flags & GEMM_SCRATCH_IN_CAPTURE)) split_scratch_give_back(SPLIT_KEPT);
    return BMB_OK;
}

}  // namespace bmb
