// Fused causal attention in fp32 (src/flash.h:36-62, src/flash.cu): split products, and the row-group SIMT code behind them.
//
// The score matrix never reaches global memory: the forward walks key tiles
// with a running row max / row sum and writes out (B,T,C) plus
// lse = max + log(sum) (src/flash.cu:292-310); the backward rebuilds
// P = exp(S - lse) and uses  dS = P * (dP - D),  D = rowsum(dO * O)
// (src/flash.cu:447-453), in two kernels so that dQ (reduced over keys) and
// dK/dV (reduced over queries) each stay in registers and are written with
// plain stores -- dqkv is overwritten, not accumulated.
//
// Long sequences go to the kernels of flash_x2.cu (wants_x2).  Short ones, captures outside a trainer, and heads with something that
// two fp16 pieces cannot serve run here, on warp-level tensor-core instructions, every fp32 product as three TF32 ones
// (flash_mma.cuh).  Behind them stand the row-group kernels (configuration 1): a query row (or, for dK/dV, a key
// row) belongs to G = HS/32 adjacent lanes, each holding a 32-float slice of the head dimension in registers; key /
// value (or query / dO) rows are staged in shared memory and read as warp-wide broadcasts; dot products finish with
// log2(G) shuffles.  A block whose result is not finite everywhere is computed again by them: split products of
// infinite operands give NaN where the fp32 chain gives an infinity, or a probability of zero.
// q, k and v are read straight out of the fused (B,T,3C) projection.
#include "flash_mma.cuh"
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <map>
#include <mutex>

namespace bmb {
int launch_flash_dsum(float *dsum, const float *dout, const float *out, int B, int T, int NH, int HS, cudaStream_t st);
bool flash_tc_supported(int T, int C, int NH, const float *qkv, const float *out);
int flash_forward_tc(float *out, float *lse, const float *qkv, int B, int T, int C, int NH, bool qkv_rounded,
                     cudaStream_t st);
int flash_backward_tc(float *dqkv, float *dsum, const float *dout, const float *qkv, const float *out,
                      const float *lse, int B, int T, int C, int NH, bool rounded, cudaStream_t st, float *dbias_qkv = nullptr);
int flash_forward_x2(float *out, float *lse, const float *qkv, int B, int T, int NH, int hs, float scale, bool in_trainer, cudaStream_t st);
int flash_backward_x2(float *dqkv, float *dsum, const float *dout, const float *qkv, const float *out, const float *lse, int B, int T, int NH, int hs,
                      float scale, bool in_trainer, cudaStream_t st);
namespace {

#define LD4(p) (*reinterpret_cast<const float4 *>(p))
#define ST4(p) (*reinterpret_cast<float4 *>(p))

constexpr int FT = 128;    // threads per block
// Rows staged per tile: 64, or 32 at head size 128 (static shared memory stays under 48 KB).
template <int HS> struct tile_rows { static constexpr int value = (HS >= 128) ? 32 : 64; };

template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Copy TILE rows of HS floats (row r at src + r*ld) into dense smem [TILE][HS];
// rows at or beyond `valid` are zero filled.
template <int HS, int TILE, int NT>
__device__ __forceinline__ void stage_rows(float *__restrict__ dst, const float *__restrict__ src,
                                           long long ld, int valid, int tid) {
    constexpr int V4 = HS / 4;
    for (int lin = tid; lin < TILE * V4; lin += NT) {
        const int r = lin / V4, c = (lin % V4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < valid) v = LD4(src + (long long)r * ld + c);
        ST4(dst + r * HS + c) = v;
    }
}

// ------------------------------------------------------------------ forward
// Rows [i0, min(i0 + nrows, T)) of one head, by NT threads (NT / G rows at a time).  smem: 2 * tile_rows * HS floats.
template <int HS, int KC, int NT>
__device__ __forceinline__ void fwd_rows(float *__restrict__ smem, float *__restrict__ out, float *__restrict__ lse,
                                         const float *__restrict__ qkv, int T, int NH, float scale, int bh, int i0, int nrows) {
    constexpr int G = HS / 32, TILE = tile_rows<HS>::value;
    float *Ks = smem, *Vs = smem + TILE * HS;
    const int tid = threadIdx.x, sub = tid % G;
    const int b = bh / NH, h = bh % NH;
    const int C = NH * HS;
    const int end = min(i0 + nrows, T);           // rows from here on are not ours
    const int row = i0 + tid / G;                 // this thread's query
    const long long ld = 3LL * C;
    const float *base = qkv + (long long)b * T * ld + h * HS;

    float q[32], o[32];
    if (row < end) {
#pragma unroll
        for (int d = 0; d < 32; d += 4) {
            const float4 v = LD4(base + (long long)row * ld + sub * 32 + d);
            q[d] = v.x * scale; q[d + 1] = v.y * scale; q[d + 2] = v.z * scale; q[d + 3] = v.w * scale;
        }
    } else {
#pragma unroll
        for (int d = 0; d < 32; ++d) q[d] = 0.0f;
    }
#pragma unroll
    for (int d = 0; d < 32; ++d) o[d] = 0.0f;
    float m = -INFINITY, l = 0.0f;

    // Last query row any lane of this warp owns: chunks past it are skipped.
    const int warp_last = min(end - 1, i0 + ((tid | 31) / G));

    for (int j0 = 0; j0 < end; j0 += TILE) {
        __syncthreads();
        stage_rows<HS, TILE, NT>(Ks, base + (long long)j0 * ld + C, ld, T - j0, tid);
        stage_rows<HS, TILE, NT>(Vs, base + (long long)j0 * ld + 2 * C, ld, T - j0, tid);
        __syncthreads();

        for (int c0 = 0; c0 < TILE; c0 += KC) {
            if (j0 + c0 > warp_last) break;       // warp-uniform
            float s[KC];
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                const float *kr = Ks + (c0 + c) * HS + sub * 32;
                float a = 0.0f;
#pragma unroll
                for (int d = 0; d < 32; d += 4) {
                    const float4 kv = LD4(kr + d);
                    a = fmaf(q[d], kv.x, a); a = fmaf(q[d + 1], kv.y, a);
                    a = fmaf(q[d + 2], kv.z, a); a = fmaf(q[d + 3], kv.w, a);
                }
                a = group_sum<G>(a);
                const int kg = j0 + c0 + c;
                s[c] = (kg > row || kg >= T) ? -INFINITY : a;
            }
            float cmax = s[0];
#pragma unroll
            for (int c = 1; c < KC; ++c) cmax = fmaxf(cmax, s[c]);
            const float mnew = fmaxf(m, cmax);
            const bool live = mnew > -INFINITY;
            const float resc = live ? __expf(m - mnew) : 1.0f;
            float csum = 0.0f;
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                s[c] = live ? __expf(s[c] - mnew) : 0.0f;
                csum += s[c];
            }
            m = mnew;
            l = l * resc + csum;
#pragma unroll
            for (int d = 0; d < 32; ++d) o[d] *= resc;
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                const float *vr = Vs + (c0 + c) * HS + sub * 32;
#pragma unroll
                for (int d = 0; d < 32; d += 4) {
                    const float4 vv = LD4(vr + d);
                    o[d] = fmaf(s[c], vv.x, o[d]); o[d + 1] = fmaf(s[c], vv.y, o[d + 1]);
                    o[d + 2] = fmaf(s[c], vv.z, o[d + 2]); o[d + 3] = fmaf(s[c], vv.w, o[d + 3]);
                }
            }
        }
    }

    if (row < end) {
        const float inv = (l > 0.0f) ? 1.0f / l : 0.0f;
        float *dst = out + ((long long)b * T + row) * C + h * HS + sub * 32;
#pragma unroll
        for (int d = 0; d < 32; d += 4)
            ST4(dst + d) = make_float4(o[d] * inv, o[d + 1] * inv, o[d + 2] * inv, o[d + 3] * inv);
        if (sub == 0) lse[(long long)bh * T + row] = m + __logf(l);
    }
}

template <int HS, int KC>
__global__ void __launch_bounds__(FT)
flash_fwd_simt_k(float *__restrict__ out, float *__restrict__ lse, const float *__restrict__ qkv,
                 int T, int NH, float scale) {
    __shared__ __align__(16) float smem[2 * tile_rows<HS>::value * HS];
    constexpr int R = FT / (HS / 32);
    fwd_rows<HS, KC, FT>(smem, out, lse, qkv, T, NH, scale, blockIdx.y, blockIdx.x * R, R);
}

// Rows [i0, i0 + nrows) again by the row-group code, inside a kernel that found its own result not finite.
template <int HS, int NT>
__device__ __noinline__ void fwd_rows_again(float *smem, float *out, float *lse, const float *qkv, int T, int NH, float scale,
                                            int bh, int i0, int nrows) {
    constexpr int R = NT / (HS / 32);
    for (int r = 0; r < nrows; r += R) fwd_rows<HS, 16, NT>(smem, out, lse, qkv, T, NH, scale, bh, i0 + r, min(R, nrows - r));
}

// The items (`each` a head) of the heads that flash_x2.cu leaves to these kernels (none as a rule, or one, or all): body(head, item), its
// shared memory free.  Blocks take them as they come free, the first item of every head before any second one (1024 heads at a time).
template <typename Body>
__device__ __forceinline__ void for_left_out(const LeftOut &left, int each, Body body) {
    __shared__ uint16_t list[1024];
    __shared__ int count;
    __shared__ long long next;
    bool any = false;
    for (int i = threadIdx.x; i < left.heads; i += blockDim.x) any = any || left.flagged[i];
    if (!__syncthreads_or(any)) return;
    long long item = blockIdx.x, first = 0;                        // this block's; the first of these heads
    for (int h0 = 0; h0 < left.heads; h0 += 1024) {
        __syncthreads();
        if (threadIdx.x < 32) {
            int n = 0;
            for (int i = threadIdx.x; i < 1024 && h0 + i - (int)threadIdx.x < left.heads; i += 32) {
                const bool f = h0 + i < left.heads && left.flagged[h0 + i];
                const uint32_t word = __ballot_sync(0xffffffffu, f);
                if (f) list[n + __popc(word & ((1u << threadIdx.x) - 1u))] = (uint16_t)i;
                n += __popc(word);
            }
            if (threadIdx.x == 0) count = n;
        }
        __syncthreads();
        const int heads = count;
        for (; item < first + (long long)heads * each; item = next) {
            const int i = (int)(item - first);                     // (at most 1024 heads of 65535 items)
            body(h0 + list[i % heads], i / heads);
            if (threadIdx.x == 0) next = (long long)gridDim.x + atomicAdd(left.taken, 1);
            __syncthreads();
        }
        first += (long long)heads * each;
    }
}

// How the products are split (flash_mma.cuh): scores and output, and sums of gradients.
__host__ __device__ constexpr fm::Form scores_form(bool fine) { return fine ? fm::FINE : fm::COARSE_CUT; }
__host__ __device__ constexpr fm::Form gradient_form(bool fine) { return fine ? fm::FINE : fm::COARSE; }

// Forward on warp-level tensor-core instructions.  A block owns 64 queries of one head, a warp 16 of them; keys come 32
// at a time, two buffers, the next 32 copied while these are multiplied.  Scores, probabilities and output stay in
// registers; the running maximum moves once per 32 keys.  Bound by the tensor pipe: 3 instructions of 8 cycles for 8
// keys x 8 columns x 16 rows in either product, beside which the splits take about half of the issue slots.
// (the tensor pipe is about half busy: two to three warps a scheduler do not cover the latency of splits and products; more
// registers a thread, for more of them under way, are worth more than a third block: 1 x 2048 x 4 x 64 124 -> 105 us.)
// Measured, the kernel before (4 rows x 16 columns a thread on the FMA pipe) -> this: B8 T1024 12 heads of 64 936 -> 253 us,
// B4 T2048 8 x 128 3608 -> 670, B2 T777 12 x 32 191 -> 42, B1 T64 2 x 32 18.9 -> 7.1.  2-norm errors against 64 bits there:
// 2.7e-7 -> 1.7e-7, 3.5e-7 -> 1.8e-7, 2.5e-7 -> 1.6e-7, 1.2e-7 -> 0.9e-7.
template <int HS, bool FINE>
__device__ __forceinline__ void fwd_mma(float *__restrict__ smem, float *__restrict__ out, float *__restrict__ lse, const float *__restrict__ qkv,
                                        int T, int NH, float scale, int bh, int i0) {
    float *Qs = smem, *Ks = Qs + 64 * HS, *Vs = Ks + 2 * 32 * HS;      // Ks, Vs: two buffers each
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int b = bh / NH, h = bh % NH;
    const int C = NH * HS;
    const long long ld = 3LL * C;
    const float *base = qkv + (long long)b * T * ld + h * HS;

    auto copy_keys = [&](int j0, int buf) {
        fm::tile_copy<HS, 32, 128>(Ks + buf * 32 * HS, base + (long long)j0 * ld + C, ld, T - j0);
        fm::tile_copy<HS, 32, 128>(Vs + buf * 32 * HS, base + (long long)j0 * ld + 2 * C, ld, T - j0);
        fm::cp_commit();
    };
    fm::tile_copy<HS, 64, 128>(Qs, base + (long long)i0 * ld, ld, T - i0);
    copy_keys(0, 0);

    float o[HS / 8][4];
#pragma unroll
    for (int c = 0; c < HS / 8; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[c][i] = 0.0f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
    const int row0 = i0 + warp * 16, jmax = min(T, i0 + 64);

    int buf = 0;
    for (int j0 = 0; j0 < jmax; j0 += 32, buf ^= 1) {
        fm::cp_wait_all();
        __syncthreads();               // everyone's part of these 32 keys is here, and the other buffer has been read
        if (j0 + 32 < jmax) copy_keys(j0 + 32, buf ^ 1);
        if (j0 > row0 + 15) continue;  // (per warp) all of these keys lie after all of its queries
        float s[4][4];
        fm::scores<HS, scores_form(FINE)>(s, scale, Qs, warp * 16, Ks + buf * 32 * HS, 0);
        const bool edge = j0 + 31 > row0 || j0 + 32 > T;               // some pair is masked
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (edge) {
                    const int key = j0 + 8 * j + 2 * t + (i & 1), row = row0 + g + 8 * (i >> 1);
                    if (key > row || key >= T) s[j][i] = -INFINITY;
                }
            }
        float resc[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float cmax = s[0][2 * r];
#pragma unroll
            for (int j = 0; j < 4; ++j) cmax = fmaxf(cmax, fmaxf(s[j][2 * r], s[j][2 * r + 1]));
            cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, 1));
            cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, 2));
            const float mnew = fmaxf(m[r], cmax);
            const bool seen = mnew > -INFINITY;
            resc[r] = seen ? __expf(m[r] - mnew) : 1.0f;
            float csum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 2 * r; i < 2 * r + 2; ++i) {
                    s[j][i] = seen ? __expf(s[j][i] - mnew) : 0.0f;
                    csum += s[j][i];
                }
            m[r] = mnew;
            l[r] = l[r] * resc[r] + csum;             // this thread's keys; the row's four lanes are added at the end
        }
        fm::contract<HS, scores_form(FINE), true>(o, resc[0], resc[1], s, Vs + buf * 32 * HS, 0);
    }

    bool bad = false;
    float inv[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        inv[r] = (l[r] > 0.0f) ? 1.0f / l[r] : 0.0f;
        const int row = row0 + g + 8 * r;
        if (row < T) {
            const float v = m[r] + __logf(l[r]);
            if (t == 0) lse[(long long)bh * T + row] = v;
            bad = bad || !(fabsf(v) <= 3.402823466e38f);
        }
    }
    bad = fm::store_rows<HS>(out + ((long long)b * T + row0) * C + h * HS, C, g, T - row0, o, inv[0], inv[1]) || bad;
    if (__syncthreads_or(bad)) fwd_rows_again<HS, 128>(smem, out, lse, qkv, T, NH, scale, bh, i0, 64);
}
// Blocks of 64 rows, a head's longest first: of every head (grid: heads x blocks) ...
template <int HS, bool FINE>
__global__ void __launch_bounds__(128, HS == 32 ? 3 : 2)
flash_fwd_mma_k(float *__restrict__ out, float *__restrict__ lse, const float *__restrict__ qkv, int T, int NH, float scale) {
    extern __shared__ __align__(16) float smem[];
    fwd_mma<HS, FINE>(smem, out, lse, qkv, T, NH, scale, blockIdx.x, ((int)gridDim.y - 1 - (int)blockIdx.y) * 64);
}
// ... or of those left out.
template <int HS>
__global__ void __launch_bounds__(128, HS == 32 ? 3 : 2)
flash_fwd_left_k(float *__restrict__ out, float *__restrict__ lse, const float *__restrict__ qkv, int T, int NH, float scale, LeftOut left) {
    extern __shared__ __align__(16) float smem[];
    wait_for_predecessor();
    const int blocks = (T + 63) / 64;
    for_left_out(left, blocks, [&](int bh, int y) { fwd_mma<HS, false>(smem, out, lse, qkv, T, NH, scale, bh, (blocks - 1 - y) * 64); });
}

// ----------------------------------------------------------------- backward
// D[b,h,t] = sum_d dO[b,t,h,d] * O[b,t,h,d]; one warp per row (src/flash.cu:471-489).
__global__ void flash_dsum_k(float *__restrict__ dsum, const float *__restrict__ dout,
                             const float *__restrict__ out, int T, int NH, int HS, long long rows) {
    const int lane = threadIdx.x & 31;
    const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    if (w >= rows) return;
    const int t = (int)(w % T);
    const int h = (int)((w / T) % NH);
    const long long b = w / ((long long)T * NH);
    const long long off = (b * T + t) * (long long)(NH * HS) + (long long)h * HS;
    float a = 0.0f;
    for (int d = lane; d < HS; d += 32) a += dout[off + d] * out[off + d];
    a = warp_sum(a);
    if (lane == 0) dsum[w] = a;
}

// The same sums with 128-bit loads over the (B*T, C) arrays in storage order: GL = HS/4 consecutive
// lanes hold one head of one token and add up with shuffles.  Needs 16-byte aligned rows.
template <int GL>
__global__ void __launch_bounds__(256) flash_dsum_vec_k(float *__restrict__ dsum, const float *__restrict__ dout,
                                                        const float *__restrict__ out, int T, int NH, long long n4) {
    const int c4 = NH * GL;                                // 128-bit words per token
    const long long stride = (long long)gridDim.x * blockDim.x;
    // whole warps stay in the loop for the shuffles
    const long long n4_up = (n4 + 31) & ~31LL;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n4_up; e += stride) {
        float a = 0.0f;
        if (e < n4) {
            const float4 x = __ldg(reinterpret_cast<const float4 *>(dout) + e);
            const float4 y = __ldg(reinterpret_cast<const float4 *>(out) + e);
            a = x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
        }
#pragma unroll
        for (int o = GL / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (e < n4 && (threadIdx.x & (GL - 1)) == 0) {
            const long long bt = e / c4;
            const int h = (int)(e - bt * c4) / GL;
            const long long b = bt / T;
            const int t = (int)(bt - b * T);
            dsum[(b * NH + h) * T + t] = a;
        }
    }
}

// dQ: a row group owns a query row; keys stream through shared memory.  Rows and threads as in fwd_rows.
template <int HS, int KC, int NT>
__device__ __forceinline__ void bwd_q_rows(float *__restrict__ smem, float *__restrict__ dqkv, const float *__restrict__ qkv,
                                           const float *__restrict__ dout, const float *__restrict__ lse,
                                           const float *__restrict__ dsum, int T, int NH, float scale, int bh, int i0, int nrows) {
    constexpr int G = HS / 32, TILE = tile_rows<HS>::value;
    float *Ks = smem, *Vs = smem + TILE * HS;
    const int tid = threadIdx.x, sub = tid % G;
    const int b = bh / NH, h = bh % NH;
    const int C = NH * HS;
    const int end = min(i0 + nrows, T);
    const int row = i0 + tid / G;
    const long long ld = 3LL * C;
    const float *base = qkv + (long long)b * T * ld + h * HS;

    float q[32], go[32], dq[32];
    float lrow = 0.0f, drow = 0.0f;
    if (row < end) {
        const float *dor = dout + ((long long)b * T + row) * C + h * HS + sub * 32;
#pragma unroll
        for (int d = 0; d < 32; d += 4) {
            const float4 v = LD4(base + (long long)row * ld + sub * 32 + d);
            q[d] = v.x * scale; q[d + 1] = v.y * scale; q[d + 2] = v.z * scale; q[d + 3] = v.w * scale;
            const float4 g = LD4(dor + d);
            go[d] = g.x; go[d + 1] = g.y; go[d + 2] = g.z; go[d + 3] = g.w;
        }
        lrow = lse[(long long)bh * T + row];
        drow = dsum[(long long)bh * T + row];
    } else {
#pragma unroll
        for (int d = 0; d < 32; ++d) { q[d] = 0.0f; go[d] = 0.0f; }
    }
#pragma unroll
    for (int d = 0; d < 32; ++d) dq[d] = 0.0f;

    const int warp_last = min(end - 1, i0 + ((tid | 31) / G));
    for (int j0 = 0; j0 < end; j0 += TILE) {
        __syncthreads();
        stage_rows<HS, TILE, NT>(Ks, base + (long long)j0 * ld + C, ld, T - j0, tid);
        stage_rows<HS, TILE, NT>(Vs, base + (long long)j0 * ld + 2 * C, ld, T - j0, tid);
        __syncthreads();
        for (int c0 = 0; c0 < TILE; c0 += KC) {
            if (j0 + c0 > warp_last) break;
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                const float *kr = Ks + (c0 + c) * HS + sub * 32;
                const float *vr = Vs + (c0 + c) * HS + sub * 32;
                float s = 0.0f, dp = 0.0f;
                float kreg[32];
#pragma unroll
                for (int d = 0; d < 32; d += 4) {
                    const float4 kv = LD4(kr + d), vv = LD4(vr + d);
                    kreg[d] = kv.x; kreg[d + 1] = kv.y; kreg[d + 2] = kv.z; kreg[d + 3] = kv.w;
                    s = fmaf(q[d], kv.x, s); s = fmaf(q[d + 1], kv.y, s);
                    s = fmaf(q[d + 2], kv.z, s); s = fmaf(q[d + 3], kv.w, s);
                    dp = fmaf(go[d], vv.x, dp); dp = fmaf(go[d + 1], vv.y, dp);
                    dp = fmaf(go[d + 2], vv.z, dp); dp = fmaf(go[d + 3], vv.w, dp);
                }
                s = group_sum<G>(s);
                dp = group_sum<G>(dp);
                const int kg = j0 + c0 + c;
                const bool on = (kg <= row) && (kg < T) && (row < end);
                const float p = on ? __expf(s - lrow) : 0.0f;
                const float ds = p * (dp - drow);
#pragma unroll
                for (int d = 0; d < 32; ++d) dq[d] = fmaf(ds, kreg[d], dq[d]);
            }
        }
    }
    if (row < end) {
        float *dst = dqkv + ((long long)b * T + row) * ld + h * HS + sub * 32;
#pragma unroll
        for (int d = 0; d < 32; d += 4)
            ST4(dst + d) = make_float4(dq[d] * scale, dq[d + 1] * scale, dq[d + 2] * scale, dq[d + 3] * scale);
    }
}

template <int HS, int KC>
__global__ void __launch_bounds__(FT)
flash_bwd_q_simt_k(float *__restrict__ dqkv, const float *__restrict__ qkv,
                   const float *__restrict__ dout, const float *__restrict__ lse,
                   const float *__restrict__ dsum, int T, int NH, float scale) {
    __shared__ __align__(16) float smem[2 * tile_rows<HS>::value * HS];
    constexpr int R = FT / (HS / 32);
    bwd_q_rows<HS, KC, FT>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, blockIdx.y, blockIdx.x * R, R);
}

// dK, dV: a row group owns a key row; queries at or after it stream through
// shared memory together with dO, lse and D.  smem: 2 * QT * (HS + 1) floats.
constexpr int QT = 32;   // queries staged per tile
template <int HS, int KC, int NT>
__device__ __forceinline__ void bwd_kv_rows(float *__restrict__ smem, float *__restrict__ dqkv, const float *__restrict__ qkv,
                                            const float *__restrict__ dout, const float *__restrict__ lse,
                                            const float *__restrict__ dsum, int T, int NH, float scale, int bh, int j0, int nrows) {
    constexpr int G = HS / 32;
    float *Qs = smem, *Os = Qs + QT * HS, *Ls = Os + QT * HS, *Ds = Ls + QT;
    const int tid = threadIdx.x, sub = tid % G;
    const int b = bh / NH, h = bh % NH;
    const int C = NH * HS;
    const int end = min(j0 + nrows, T);
    const int key = j0 + tid / G;
    const long long ld = 3LL * C;
    const float *base = qkv + (long long)b * T * ld + h * HS;

    float k[32], v[32], dk[32], dv[32];
    if (key < end) {
#pragma unroll
        for (int d = 0; d < 32; d += 4) {
            const float4 a = LD4(base + (long long)key * ld + C + sub * 32 + d);
            const float4 c = LD4(base + (long long)key * ld + 2 * C + sub * 32 + d);
            k[d] = a.x; k[d + 1] = a.y; k[d + 2] = a.z; k[d + 3] = a.w;
            v[d] = c.x; v[d + 1] = c.y; v[d + 2] = c.z; v[d + 3] = c.w;
        }
    } else {
#pragma unroll
        for (int d = 0; d < 32; ++d) { k[d] = 0.0f; v[d] = 0.0f; }
    }
#pragma unroll
    for (int d = 0; d < 32; ++d) { dk[d] = 0.0f; dv[d] = 0.0f; }

    // First key row of this warp: queries before it contribute nothing.
    const int warp_first = j0 + ((tid & ~31) / G);
    constexpr int V4 = HS / 4;
    for (int i0 = (j0 / QT) * QT; i0 < T; i0 += QT) {
        __syncthreads();
        for (int lin = tid; lin < QT * V4; lin += NT) {
            const int r = lin / V4, c = (lin % V4) * 4;
            float4 qv = make_float4(0.f, 0.f, 0.f, 0.f), gv = qv;
            if (i0 + r < T) {
                qv = LD4(base + (long long)(i0 + r) * ld + c);
                gv = LD4(dout + ((long long)b * T + i0 + r) * C + h * HS + c);
            }
            ST4(Qs + r * HS + c) = qv;
            ST4(Os + r * HS + c) = gv;
        }
        if (tid < QT) {
            const bool ok = i0 + tid < T;
            Ls[tid] = ok ? lse[(long long)bh * T + i0 + tid] : 0.0f;
            Ds[tid] = ok ? dsum[(long long)bh * T + i0 + tid] : 0.0f;
        }
        __syncthreads();
        if (i0 + QT - 1 < warp_first) continue;   // warp-uniform; barriers are outside
#pragma unroll 2
        for (int r = 0; r < QT; ++r) {
            const int qg = i0 + r;
            const float *qr = Qs + r * HS + sub * 32;
            const float *gr = Os + r * HS + sub * 32;
            float s = 0.0f, dp = 0.0f;
            float qreg[32], greg[32];
#pragma unroll
            for (int d = 0; d < 32; d += 4) {
                const float4 qv = LD4(qr + d), gv = LD4(gr + d);
                qreg[d] = qv.x; qreg[d + 1] = qv.y; qreg[d + 2] = qv.z; qreg[d + 3] = qv.w;
                greg[d] = gv.x; greg[d + 1] = gv.y; greg[d + 2] = gv.z; greg[d + 3] = gv.w;
                s = fmaf(qv.x, k[d], s); s = fmaf(qv.y, k[d + 1], s);
                s = fmaf(qv.z, k[d + 2], s); s = fmaf(qv.w, k[d + 3], s);
                dp = fmaf(gv.x, v[d], dp); dp = fmaf(gv.y, v[d + 1], dp);
                dp = fmaf(gv.z, v[d + 2], dp); dp = fmaf(gv.w, v[d + 3], dp);
            }
            s = group_sum<G>(s) * scale;
            dp = group_sum<G>(dp);
            const bool on = (qg >= key) && (qg < T) && (key < end);
            const float p = on ? __expf(s - Ls[r]) : 0.0f;
            const float ds = p * (dp - Ds[r]);
#pragma unroll
            for (int d = 0; d < 32; ++d) {
                dv[d] = fmaf(p, greg[d], dv[d]);
                dk[d] = fmaf(ds, qreg[d], dk[d]);
            }
        }
    }
    if (key < end) {
        float *dkp = dqkv + ((long long)b * T + key) * ld + C + h * HS + sub * 32;
        float *dvp = dkp + C;
#pragma unroll
        for (int d = 0; d < 32; d += 4) {
            ST4(dkp + d) = make_float4(dk[d] * scale, dk[d + 1] * scale, dk[d + 2] * scale, dk[d + 3] * scale);
            ST4(dvp + d) = make_float4(dv[d], dv[d + 1], dv[d + 2], dv[d + 3]);
        }
    }
}

template <int HS, int KC>
__global__ void __launch_bounds__(FT)
flash_bwd_kv_simt_k(float *__restrict__ dqkv, const float *__restrict__ qkv,
                    const float *__restrict__ dout, const float *__restrict__ lse,
                    const float *__restrict__ dsum, int T, int NH, float scale) {
    __shared__ __align__(16) float smem[2 * QT * (HS + 1)];
    constexpr int R = FT / (HS / 32);
    bwd_kv_rows<HS, KC, FT>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, blockIdx.y, blockIdx.x * R, R);
}

template <int HS, int NT>
__device__ __noinline__ void bwd_q_rows_again(float *smem, float *dqkv, const float *qkv, const float *dout, const float *lse,
                                              const float *dsum, int T, int NH, float scale, int bh, int i0, int nrows) {
    constexpr int R = NT / (HS / 32);
    for (int r = 0; r < nrows; r += R) bwd_q_rows<HS, 8, NT>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, bh, i0 + r, min(R, nrows - r));
}
template <int HS, int NT>
__device__ __noinline__ void bwd_kv_rows_again(float *smem, float *dqkv, const float *qkv, const float *dout, const float *lse,
                                               const float *dsum, int T, int NH, float scale, int bh, int j0, int nrows) {
    constexpr int R = NT / (HS / 32);
    for (int r = 0; r < nrows; r += R) bwd_kv_rows<HS, 8, NT>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, bh, j0 + r, min(R, nrows - r));
}

// Backward on warp-level tensor-core instructions: blocks of 16 rows a warp (4 warps; 8 at head size 128, where two
// tiles of 64 rows would leave one block of 4 warps to an SM), 32 rows of the other side at a time in two buffers.
template <int HS> struct bwd_warps { static constexpr int value = HS == 128 ? 8 : 4; };
template <int HS> constexpr int fwd_smem() { return (64 + 4 * 32) * HS * 4; }
template <int HS> constexpr int bwd_smem() { return (2 * bwd_warps<HS>::value * 16 * HS + 4 * 32 * HS + 4 * 32) * 4; }

// dQ = scale * sum over keys of dS K, dS = P (dO V^T - D), P = exp(scale Q K^T - lse).
template <int HS, bool FINE>
__device__ __forceinline__ void bwd_q_mma(float *__restrict__ smem, float *__restrict__ dqkv, const float *__restrict__ qkv,
                                          const float *__restrict__ dout, const float *__restrict__ lse,
                                          const float *__restrict__ dsum, int T, int NH, float scale, int bh, int i0) {
    constexpr int NW = bwd_warps<HS>::value, NT = NW * 32, ROWS = NW * 16;
    float *Qs = smem, *Os = Qs + ROWS * HS, *Ks = Os + ROWS * HS, *Vs = Ks + 2 * 32 * HS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int b = bh / NH, h = bh % NH;
    const int C = NH * HS;
    const long long ld = 3LL * C;
    const float *base = qkv + (long long)b * T * ld + h * HS;
    auto copy_keys = [&](int j0, int buf) {
        fm::tile_copy<HS, 32, NT>(Ks + buf * 32 * HS, base + (long long)j0 * ld + C, ld, T - j0);
        fm::tile_copy<HS, 32, NT>(Vs + buf * 32 * HS, base + (long long)j0 * ld + 2 * C, ld, T - j0);
        fm::cp_commit();
    };
    fm::tile_copy<HS, ROWS, NT>(Qs, base + (long long)i0 * ld, ld, T - i0);
    fm::tile_copy<HS, ROWS, NT>(Os, dout + ((long long)b * T + i0) * C + h * HS, C, T - i0);
    copy_keys(0, 0);

    const int row0 = i0 + warp * 16, jmax = min(T, i0 + ROWS);
    float lrow[2] = {0.0f, 0.0f}, drow[2] = {0.0f, 0.0f};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = row0 + g + 8 * r;
        if (row < T) { lrow[r] = lse[(long long)bh * T + row]; drow[r] = dsum[(long long)bh * T + row]; }
    }
    float dq[HS / 8][4];
#pragma unroll
    for (int c = 0; c < HS / 8; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) dq[c][i] = 0.0f;

    float most = 0.0f;                 // a score may overflow before it is scaled (the row-group code scales q first)
    int buf = 0;
    for (int j0 = 0; j0 < jmax; j0 += 32, buf ^= 1) {
        fm::cp_wait_all();
        __syncthreads();
        if (j0 + 32 < jmax) copy_keys(j0 + 32, buf ^ 1);
        if (j0 > row0 + 15) continue;
        float s[4][4], dp[4][4];
        fm::scores<HS, scores_form(FINE)>(s, scale, Qs, warp * 16, Ks + buf * 32 * HS, 0);
        fm::scores<HS, scores_form(FINE)>(dp, 1.0f, Os, warp * 16, Vs + buf * 32 * HS, 0);
        const bool edge = j0 + 31 > row0 || j0 + 32 > T || row0 + 16 > T;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; i += 2) asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(most) : "f"(s[j][i]), "f"(s[j][i + 1]));
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int key = j0 + 8 * j + 2 * t + (i & 1), row = row0 + g + 8 * (i >> 1);
                const bool on = !edge || (key <= row && key < T && row < T);
                const float p = on ? __expf(s[j][i] - lrow[i >> 1]) : 0.0f;
                s[j][i] = p * (dp[j][i] - drow[i >> 1]);
            }
        fm::contract<HS, gradient_form(FINE), false>(dq, 1.0f, 1.0f, s, Ks + buf * 32 * HS, 0);
    }
    const bool bad = fm::store_rows<HS>(dqkv + ((long long)b * T + row0) * ld + h * HS, ld, g, T - row0, dq, scale, scale) || most > 3.402823466e38f;
    if (__syncthreads_or(bad)) bwd_q_rows_again<HS, NT>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, bh, i0, ROWS);
}

// dV = sum over queries of P^T dO, dK = scale * sum of dS^T Q: the transposed scores, keys as rows.
template <int HS, bool FINE>
__device__ __forceinline__ void bwd_kv_mma(float *__restrict__ smem, float *__restrict__ dqkv, const float *__restrict__ qkv,
                                           const float *__restrict__ dout, const float *__restrict__ lse,
                                           const float *__restrict__ dsum, int T, int NH, float scale, int bh, int j0) {
    constexpr int NW = bwd_warps<HS>::value, NT = NW * 32, ROWS = NW * 16;
    float *Ks = smem, *Vs = Ks + ROWS * HS, *Qs = Vs + ROWS * HS, *Os = Qs + 2 * 32 * HS, *Ls = Os + 2 * 32 * HS, *Ds = Ls + 2 * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int b = bh / NH, h = bh % NH;
    const int C = NH * HS;
    const long long ld = 3LL * C;
    const float *base = qkv + (long long)b * T * ld + h * HS;
    auto copy_queries = [&](int i0, int buf) {
        fm::tile_copy<HS, 32, NT>(Qs + buf * 32 * HS, base + (long long)i0 * ld, ld, T - i0);
        fm::tile_copy<HS, 32, NT>(Os + buf * 32 * HS, dout + ((long long)b * T + i0) * C + h * HS, C, T - i0);
        if (threadIdx.x < 64) {
            const int r = threadIdx.x & 31;
            const bool ok = i0 + r < T;
            const float *src = (threadIdx.x < 32 ? lse : dsum) + (long long)bh * T + (ok ? i0 + r : 0);
            fm::cp_async4((threadIdx.x < 32 ? Ls : Ds) + buf * 32 + r, src, ok);
        }
        fm::cp_commit();
    };
    fm::tile_copy<HS, ROWS, NT>(Ks, base + (long long)j0 * ld + C, ld, T - j0);
    fm::tile_copy<HS, ROWS, NT>(Vs, base + (long long)j0 * ld + 2 * C, ld, T - j0);
    copy_queries(j0, 0);                   // j0 is a multiple of 32: queries before it see none of these keys

    const int key0 = j0 + warp * 16;
    float dk[HS / 8][4], dv[HS / 8][4];
#pragma unroll
    for (int c = 0; c < HS / 8; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i) dk[c][i] = dv[c][i] = 0.0f;

    int buf = 0;
    for (int i0 = j0; i0 < T; i0 += 32, buf ^= 1) {
        fm::cp_wait_all();
        __syncthreads();
        if (i0 + 32 < T) copy_queries(i0 + 32, buf ^ 1);
        if (i0 + 31 < key0) continue;      // (per warp) all of these queries come before all of its keys
        const float *q = Qs + buf * 32 * HS, *go = Os + buf * 32 * HS, *Lb = Ls + buf * 32, *Db = Ds + buf * 32;
        const bool edge = i0 < key0 + 15 || i0 + 32 > T || key0 + 16 > T;
        float p[4][4], ds[4][4];
        fm::scores<HS, scores_form(FINE)>(p, scale, Ks, warp * 16, q, 0);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = 8 * j + 2 * t + (i & 1), key = key0 + g + 8 * (i >> 1);
                const bool on = !edge || (i0 + c >= key && i0 + c < T && key < T);
                p[j][i] = on ? __expf(p[j][i] - Lb[c]) : 0.0f;
            }
        fm::contract<HS, gradient_form(FINE), false>(dv, 1.0f, 1.0f, p, go, 0);
        fm::scores<HS, scores_form(FINE)>(ds, 1.0f, Vs, warp * 16, go, 0);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) ds[j][i] = p[j][i] * (ds[j][i] - Db[8 * j + 2 * t + (i & 1)]);
        fm::contract<HS, gradient_form(FINE), false>(dk, 1.0f, 1.0f, ds, q, 0);
    }
    float *dkp = dqkv + ((long long)b * T + key0) * ld + C + h * HS;
    bool bad = fm::store_rows<HS>(dkp, ld, g, T - key0, dk, scale, scale);
    bad = fm::store_rows<HS>(dkp + C, ld, g, T - key0, dv, 1.0f, 1.0f) || bad;
    if (__syncthreads_or(bad)) bwd_kv_rows_again<HS, NT>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, bh, j0, ROWS);
}

// Both in one grid (one partly filled last wave instead of two), the longest blocks first: the first key block has all
// queries, the last query block all keys.
// Measured with D, row-group kernels -> this: B8 T1024 12 heads of 64 2436 -> 960 us, B4 T2048 8 x 128 18754 -> 2501,
// B2 T777 12 x 32 445 -> 105.  2-norm errors of dq / dk / dv against 64 bits at 8 x 128: 4.9 / 10.8 / 10.8e-7 -> 3.2 / 3.7 / 3.3e-7.
template <int HS, bool FINE>
__device__ __forceinline__ void bwd_mma(float *__restrict__ smem, float *__restrict__ dqkv, const float *__restrict__ qkv, const float *__restrict__ dout,
                                        const float *__restrict__ lse, const float *__restrict__ dsum, int T, int NH, float scale, int bh, int y, int blocks) {
    constexpr int ROWS = bwd_warps<HS>::value * 16;
    if (y & 1) bwd_q_mma<HS, FINE>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, bh, (blocks - 1 - (y >> 1)) * ROWS);
    else bwd_kv_mma<HS, FINE>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, bh, (y >> 1) * ROWS);
}
template <int HS, bool FINE>
__global__ void __launch_bounds__(bwd_warps<HS>::value * 32, HS == 128 ? 1 : HS == 64 ? 2 : 3)
flash_bwd_mma_k(float *__restrict__ dqkv, const float *__restrict__ qkv, const float *__restrict__ dout,
                const float *__restrict__ lse, const float *__restrict__ dsum, int T, int NH, float scale) {
    extern __shared__ __align__(16) float smem[];
    bwd_mma<HS, FINE>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, blockIdx.x, blockIdx.y, gridDim.y >> 1);
}
template <int HS>
__global__ void __launch_bounds__(bwd_warps<HS>::value * 32, HS == 128 ? 1 : HS == 64 ? 2 : 3)
flash_bwd_left_k(float *__restrict__ dqkv, const float *__restrict__ qkv, const float *__restrict__ dout,
                 const float *__restrict__ lse, const float *__restrict__ dsum, int T, int NH, float scale, LeftOut left) {
    extern __shared__ __align__(16) float smem[];
    wait_for_predecessor();
    constexpr int ROWS = bwd_warps<HS>::value * 16;
    const int blocks = (T + ROWS - 1) / ROWS;
    for_left_out(left, 2 * blocks, [&](int bh, int y) { bwd_mma<HS, false>(smem, dqkv, qkv, dout, lse, dsum, T, NH, scale, bh, y, blocks); });
}

struct FwdCfg { int kc; const char *name; };
struct BwdCfg { int kc; const char *name; };
// Forward config 2 is the tensor-core kernel (flash_tc.cu), head size 64 only.
// Config 0 of both tables: warp-level tensor-core instructions, fp32 products in three TF32 ones; 1: the row-group code.
const FwdCfg FWD[] = {{32, "mma-3xtf32 q64 k32"}, {16, "simt-fp32 rowgroup keys16"},
                      {0, "tcgen05-tf32 q2x128 k64 (head size 64 only)"}};
// Backward config 2 is the tensor-core kernel pair (flash_tc_bwd.cu), head size 64 only.
const BwdCfg BWD[] = {{32, "mma-3xtf32 rows16 per warp, 32 at a time"}, {8, "simt-fp32 rowgroup keys8"},
                      {0, "tcgen05-tf32 dq128x128 dkv128x128 (head size 64 only)"}};
constexpr int NFWD = 3, NBWD = 3, FWD_TC = 2, BWD_TC = 2;

// Sequences up to here take six products for one instead of three: against kernels on the FMA pipe in chains of 8, the error of
// the output at T = 128 is 0.69 (three products: 1.00 to 1.04), at T = 8 0.84 (1.5), and from 129 on three are no worse than
// those.  128 x 128 positions, 4 heads of 64: forward 22 -> 37 us, backward 76 -> 123 (the FMA pipe: 54 and 184).
constexpr int FINE_T = 128;

// Whether flash_x2.cu takes a call: where its three launches and its tiles of 128 rows pay.  The backward goes the way that the
// forward of its sizes went, although it gains from T = 192 on wherever that is: its scores then err as those that lse was made of
// (errors of dqkv 4 to 9 % smaller).  A trainer runs both, so there the two together count.  us, these kernels / flash_x2.cu, heads x T,
// forward | backward.  32 columns: 48 x 400 25 / 25 | 60 / 40, 16 x 400 17 / 21 | 50 / 24, 96 x 256 19 / 22 | 50 / 37, 2 x 512 21 / 21 | 54 / 23;
// 64: 48 x 256 19 / 19 | 56 / 29, 96 x 256 25 / 27 | 88 / 51, 96 x 400 58 / 43 | 199 / 99, 48 x 200 18 / 19 | 50 / 29;
// 128: 48 x 200 35 / 31 | 101 / 50, 96 x 256 46 / 57 | 208 / 115, 96 x 400 115 / 93 | 462 / 207, 48 x 136 25 / 27 | 74 / 39.
bool wants_x2(int hs, long long heads, int T, bool trains) {
    if (trains && T >= 192) return true;
    if (hs == 32) return T >= 512 || (T >= 384 && heads >= 40);
    return T >= 384 || (T >= (hs == 64 ? 240 : 192) && heads <= 64);
}

bool shape_ok(const float *a, const float *b, int C, int NH) {
    return NH > 0 && C % NH == 0 && (((uintptr_t)a | (uintptr_t)b) & 15) == 0;
}

// Dynamic shared memory above 48 KB is opted into once per kernel and device.
int allow_smem(const void *kernel, int bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, bool> done;
    std::lock_guard<std::mutex> lk(mu);
    bool &d = done[{kernel, current_device()}];
    if (!d) BMB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    d = true;
    return BMB_OK;
}

template <int HS>
int launch_fwd_mma(float *out, float *lse, const float *qkv, int B, int T, int NH, float scale, cudaStream_t st) {
    const auto kernel = T <= FINE_T ? flash_fwd_mma_k<HS, true> : flash_fwd_mma_k<HS, false>;
    BMB_TRY(allow_smem((const void *)kernel, fwd_smem<HS>()));
    kernel<<<dim3(B * NH, ceil_div(T, 64)), 128, fwd_smem<HS>(), st>>>(out, lse, qkv, T, NH, scale);
    count_launch();
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}
template <int HS>
int launch_bwd_mma(float *dqkv, const float *dsum, const float *dout, const float *qkv, const float *lse, int B, int T, int NH, float scale,
                   cudaStream_t st) {
    constexpr int ROWS = bwd_warps<HS>::value * 16;
    const auto kernel = T <= FINE_T ? flash_bwd_mma_k<HS, true> : flash_bwd_mma_k<HS, false>;
    BMB_TRY(allow_smem((const void *)kernel, bwd_smem<HS>()));
    kernel<<<dim3(B * NH, 2 * ceil_div(T, ROWS)), bwd_warps<HS>::value * 32, bwd_smem<HS>(), st>>>(dqkv, qkv, dout, lse, dsum, T, NH, scale);
    count_launch();
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}
// Two blocks an SM, which is what runs side by side of most of these kernels.
int left_grid(long long items) { return (int)std::min<long long>(items, 2 * sm_count()); }
template <int HS>
int launch_fwd_left(float *out, float *lse, const float *qkv, int T, int NH, float scale, LeftOut left, cudaStream_t st) {
    BMB_TRY(allow_smem((const void *)flash_fwd_left_k<HS>, fwd_smem<HS>()));
    return launch_in_chain(flash_fwd_left_k<HS>, left_grid((long long)left.heads * ceil_div(T, 64)), 128, fwd_smem<HS>(), st, out, lse, qkv, T, NH, scale,
                           left);
}
template <int HS>
int launch_bwd_left(float *dqkv, const float *dsum, const float *dout, const float *qkv, const float *lse, int T, int NH, float scale,
                    LeftOut left, cudaStream_t st) {
    constexpr int ROWS = bwd_warps<HS>::value * 16;
    BMB_TRY(allow_smem((const void *)flash_bwd_left_k<HS>, bwd_smem<HS>()));
    return launch_in_chain(flash_bwd_left_k<HS>, left_grid(2LL * left.heads * ceil_div(T, ROWS)), bwd_warps<HS>::value * 32, bwd_smem<HS>(), st,
                           dqkv, qkv, dout, lse, dsum, T, NH, scale, left);
}

template <int HS>
int run_fwd(int cfg, float *out, float *lse, const float *qkv, int B, int T, int NH, float scale,
            bool in_trainer, cudaStream_t st) {
    if (cfg == 0 && ceil_div(T, 64) > 65535) cfg = 1;              // (blocks of rows on grid y)
    if (cfg == 0) {
        if (wants_x2(HS, (long long)B * NH, T, in_trainer)) {
            const int rc = flash_forward_x2(out, lse, qkv, B, T, NH, HS, scale, in_trainer, st);
            if (rc != BMB_E_UNSUPPORTED) return rc;
        }
        return launch_fwd_mma<HS>(out, lse, qkv, B, T, NH, scale, st);
    } else {
        constexpr int R = FT / (HS / 32);
        dim3 grid(ceil_div(T, R), B * NH);
        flash_fwd_simt_k<HS, 16><<<grid, FT, 0, st>>>(out, lse, qkv, T, NH, scale);
    }
    count_launch();
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}

template <int HS>
int run_bwd(int cfg, float *dqkv, float *dsum, const float *dout, const float *qkv, const float *out,
            const float *lse, int B, int T, int NH, float scale, bool in_trainer, cudaStream_t st) {
    constexpr int ROWS = bwd_warps<HS>::value * 16;
    if (cfg == 0 && ceil_div(T, ROWS) > 32767) cfg = 1;
    // Short rows of 128 columns and more heads than SMs: a block's 128 rows are padding for the most part (64 x 4 heads, T = 8 92 us
    // against 60 by row groups, 32 96 / 81, but 64 164 / 294; 2 x 4 heads, T = 8 33 / 38).
    const long long heads = (long long)B * NH;
    if (cfg == 0 && HS == 128 && T <= 32 && heads > sm_count() && heads <= 65535) cfg = 1;
    if (cfg == 0) {
        if (wants_x2(HS, (long long)B * NH, T, in_trainer)) {
            const int rc = flash_backward_x2(dqkv, dsum, dout, qkv, out, lse, B, T, NH, HS, scale, in_trainer, st);
            if (rc != BMB_E_UNSUPPORTED) return rc;
        }
        BMB_TRY(launch_flash_dsum(dsum, dout, out, B, T, NH, HS, st));
        return launch_bwd_mma<HS>(dqkv, dsum, dout, qkv, lse, B, T, NH, scale, st);
    }
    constexpr int R = FT / (HS / 32);
    const long long rows = (long long)B * NH * T;
    flash_dsum_k<<<ceil_div(rows * 32, 256), 256, 0, st>>>(dsum, dout, out, T, NH, HS, rows);
    dim3 grid(ceil_div(T, R), B * NH);
    flash_bwd_kv_simt_k<HS, 8><<<grid, FT, 0, st>>>(dqkv, qkv, dout, lse, dsum, T, NH, scale);
    flash_bwd_q_simt_k<HS, 8><<<grid, FT, 0, st>>>(dqkv, qkv, dout, lse, dsum, T, NH, scale);
    count_launch(3);
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}

}  // namespace

// Behind flash_x2.cu (T > FINE_T), for the heads that it leaves out.
int flash_fwd_left(int hs, float *out, float *lse, const float *qkv, int T, int NH, float scale, LeftOut left, cudaStream_t st) {
    const auto run = hs == 32 ? launch_fwd_left<32> : hs == 64 ? launch_fwd_left<64> : launch_fwd_left<128>;
    return run(out, lse, qkv, T, NH, scale, left, st);
}
int flash_bwd_left(int hs, float *dqkv, const float *dsum, const float *dout, const float *qkv, const float *lse, int T, int NH, float scale,
                   LeftOut left, cudaStream_t st) {
    const auto run = hs == 32 ? launch_bwd_left<32> : hs == 64 ? launch_bwd_left<64> : launch_bwd_left<128>;
    return run(dqkv, dsum, dout, qkv, lse, T, NH, scale, left, st);
}

int launch_flash_dsum(float *dsum, const float *dout, const float *out, int B, int T, int NH, int HS, cudaStream_t st) {
    const long long rows = (long long)B * NH * T;
    const bool vec = (HS == 32 || HS == 64 || HS == 128) && (((uintptr_t)dout | (uintptr_t)out) & 15) == 0;
    if (vec) {
        const long long n4 = rows * (HS / 4);
        long long blocks = (n4 + 255) / 256;
        const long long cap = 16LL * sm_count();
        if (blocks > cap) blocks = cap;
        if (HS == 32) flash_dsum_vec_k<8><<<(int)blocks, 256, 0, st>>>(dsum, dout, out, T, NH, n4);
        else if (HS == 64) flash_dsum_vec_k<16><<<(int)blocks, 256, 0, st>>>(dsum, dout, out, T, NH, n4);
        else flash_dsum_vec_k<32><<<(int)blocks, 256, 0, st>>>(dsum, dout, out, T, NH, n4);
    } else {
        flash_dsum_k<<<ceil_div(rows * 32, 256), 256, 0, st>>>(dsum, dout, out, T, NH, HS, rows);
    }
    count_launch();
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}
}  // namespace bmb

using namespace bmb;

extern "C" {

int bmb_flash_num_configs(void) { return NFWD; }
const char *bmb_flash_config_name(int cfg) { return (cfg >= 0 && cfg < NFWD) ? FWD[cfg].name : "?"; }
// fp32 arithmetic: split products (config 0); TF32/BF16 math modes: the tensor-core kernel.
int bmb_flash_default_config(void) { return bmb_get_math_mode() == BMB_MATH_FP32 ? 0 : FWD_TC; }

int bmb_flash_attention_forward_cfg(int cfg, float *out, float *lse, const float *qkv, int B, int T,
                                    int C, int NH) {
    return bmb_flash_attention_forward_ex(cfg, 0, out, lse, qkv, B, T, C, NH);
}

int bmb_flash_attention_forward_ex(int cfg, int flags, float *out, float *lse, const float *qkv, int B, int T,
                                   int C, int NH) {
    return flash_forward(cfg, flags, out, lse, qkv, B, T, C, NH, false);
}

}  // extern "C"
namespace bmb {
int flash_forward(int cfg, int flags, float *out, float *lse, const float *qkv, int B, int T, int C, int NH, bool in_trainer) {
    if (cfg < 0 || cfg >= NFWD) return fail(BMB_E_UNSUPPORTED, "flash: no forward config %d", cfg);
    if (B <= 0 || T <= 0) return BMB_OK;
    if (!shape_ok(out, qkv, C, NH)) return fail(BMB_E_ARG, "flash: bad shape or alignment (C=%d NH=%d)", C, NH);
    const int hs = C / NH;
    const float scale = 1.0f / sqrtf((float)hs);
    cudaStream_t st = cur_stream();
    if (cfg == FWD_TC) {
        if (!flash_tc_supported(T, C, NH, qkv, out))
            return fail(BMB_E_UNSUPPORTED, "flash: the tensor-core config needs head size 64 (got %d)", hs);
        return flash_forward_tc(out, lse, qkv, B, T, C, NH, (flags & BMB_FLASH_OPERANDS_ROUNDED) != 0, st);
    }
    switch (hs) {
    case 32:  return run_fwd<32>(cfg, out, lse, qkv, B, T, NH, scale, in_trainer, st);
    case 64:  return run_fwd<64>(cfg, out, lse, qkv, B, T, NH, scale, in_trainer, st);
    case 128: return run_fwd<128>(cfg, out, lse, qkv, B, T, NH, scale, in_trainer, st);
    default:  return fail(BMB_E_UNSUPPORTED, "flash: no tile config for head size %d", hs);
    }
}
}  // namespace bmb
extern "C" {

int bmb_flash_attention_forward(float *out, float *lse, const float *qkv, int B, int T, int C,
                                int NH) {
    int cfg = bmb_flash_default_config();
    // The preferred config may not serve this head size: fall back through the table (src/flash.cu:419-432).
    if (cfg == FWD_TC && !(NH > 0 && C % NH == 0 && flash_tc_supported(T, C, NH, qkv, out))) cfg = 0;
    return bmb_flash_attention_forward_cfg(cfg, out, lse, qkv, B, T, C, NH);
}

int bmb_flash_num_bwd_configs(void) { return NBWD; }
const char *bmb_flash_bwd_config_name(int cfg) { return (cfg >= 0 && cfg < NBWD) ? BWD[cfg].name : "?"; }
int bmb_flash_default_bwd_config(void) { return bmb_get_math_mode() == BMB_MATH_FP32 ? 0 : BWD_TC; }

int bmb_flash_attention_backward_cfg(int cfg, float *dqkv, float *dsum, const float *dout,
                                     const float *qkv, const float *out, const float *lse, int B,
                                     int T, int C, int NH) {
    return bmb_flash_attention_backward_ex(cfg, 0, dqkv, dsum, dout, qkv, out, lse, B, T, C, NH);
}

int bmb_flash_attention_backward_ex(int cfg, int flags, float *dqkv, float *dsum, const float *dout,
                                    const float *qkv, const float *out, const float *lse, int B,
                                    int T, int C, int NH) {
    return flash_backward(cfg, flags, dqkv, dsum, dout, qkv, out, lse, B, T, C, NH, false);
}

}  // extern "C"
namespace bmb {
int flash_backward(int cfg, int flags, float *dqkv, float *dsum, const float *dout, const float *qkv, const float *out, const float *lse,
                   int B, int T, int C, int NH, bool in_trainer) {
    if (cfg < 0 || cfg >= NBWD) return fail(BMB_E_UNSUPPORTED, "flash: no backward config %d", cfg);
    if (B <= 0 || T <= 0) return BMB_OK;
    if (!shape_ok(dqkv, qkv, C, NH) || !shape_ok(dout, out, C, NH))
        return fail(BMB_E_ARG, "flash: bad shape or alignment (C=%d NH=%d)", C, NH);
    const int hs = C / NH;
    const float scale = 1.0f / sqrtf((float)hs);
    cudaStream_t st = cur_stream();
    if (cfg == BWD_TC) {
        if (!flash_tc_supported(T, C, NH, qkv, dqkv))
            return fail(BMB_E_UNSUPPORTED, "flash: the tensor-core config needs head size 64 (got %d)", hs);
        return flash_backward_tc(dqkv, dsum, dout, qkv, out, lse, B, T, C, NH, (flags & BMB_FLASH_OPERANDS_ROUNDED) != 0, st);
    }
    switch (hs) {
    case 32:  return run_bwd<32>(cfg, dqkv, dsum, dout, qkv, out, lse, B, T, NH, scale, in_trainer, st);
    case 64:  return run_bwd<64>(cfg, dqkv, dsum, dout, qkv, out, lse, B, T, NH, scale, in_trainer, st);
    case 128: return run_bwd<128>(cfg, dqkv, dsum, dout, qkv, out, lse, B, T, NH, scale, in_trainer, st);
    default:  return fail(BMB_E_UNSUPPORTED, "flash: no backward tile config for head size %d", hs);
    }
}
}  // namespace bmb
extern "C" {

int bmb_flash_attention_backward(float *dqkv, float *dsum, const float *dout, const float *qkv,
                                 const float *out, const float *lse, int B, int T, int C, int NH) {
    int cfg = bmb_flash_default_bwd_config();
    if (cfg == BWD_TC && !(NH > 0 && C % NH == 0 && flash_tc_supported(T, C, NH, qkv, dqkv))) cfg = 0;
    return bmb_flash_attention_backward_cfg(cfg, dqkv, dsum, dout, qkv, out, lse, B, T, C, NH);
}

}  // extern "C"
