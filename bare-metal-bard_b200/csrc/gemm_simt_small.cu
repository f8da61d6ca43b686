// fp32 SIMT GEMM in small tiles, for products that leave most SMs without a 128 x 128 tile of their own.
//
// Each element is the same sequential chain of fused multiply-adds over k as in the other SIMT kernels, so the results
// are theirs bit for bit; only the number of SMs at work changes.  A chain cannot be cut along K without changing its
// roundings, so a product of few elements is bound by what a thread reads for its chains: shared memory gives a warp 128 bytes a
// cycle, also of words that several lanes share.  Tiles of 64 x 64 with 8 x 4 elements a thread (48 cycles of reads a step of k and
// 32 of multiply-adds; measured 53 to 70), 64 x 32 with 4 x 4 (32 and 16; 31 to 42), or 32 x 32 with 2 x 4 (24 and 8; 23 to 30).
// More elements a thread read less, but one warp a scheduler then waits for its own multiply-adds (64 x 64 with 8 x 8: 100).
//
// Operands lie in shared memory as they lie in global memory -- rows of 32 k (36 floats apart: eight rows' 16-byte words
// are in different banks) or rows of m / n -- and are copied asynchronously three slices ahead, in 16-byte words where
// they are aligned, so no layout needs a transposing pass; the next four k are read while these are multiplied.  The 128 x 128
// kernels reuse an operand twice as often and stay ahead where every SM has a tile.
// Measured, 128 x 128 tiles -> these: 1024^3 (NN) 96 -> 62 us, 512^3 49 -> 14.5, 256x384x1536 140 -> 30, 64x64x4096 446 -> 74,
// batch 12 of 256x64x256 34 -> 8.9, batch 100 of 200x64x200 48 -> 24.  (Read where they are used, without 64 x 32 tiles: 64.7, 18.6,
// 36.5, 88, 10.4, 24.7.)
#include "common.cuh"
#include <mutex>

namespace bmb {
namespace {

constexpr int BK = 32, STAGES = 4;

// Floats of one operand's slice: X rows of BK + 4 (k contiguous), or BK rows of X + 4.
template <int X, bool KC> __host__ __device__ constexpr int slice_floats() { return KC ? X * (BK + 4) : BK * (X + 4); }

// Start copying one slice: element (x, k), x in [x0, x0 + X), k in [k0, k0 + BK); what lies outside is zero.
template <int X, bool KC, bool VEC, int NT>
__device__ __forceinline__ void copy_slice(float *s, const float *__restrict__ src, long long ld, int x0, int k0, int xe, int ke) {
    constexpr int INNER = KC ? BK : X, OUTER = KC ? X : BK, PITCH = INNER + 4, W = VEC ? 4 : 1;
    const int inner0 = KC ? k0 : x0, outer0 = KC ? x0 : k0, inner_end = KC ? ke : xe, outer_end = KC ? xe : ke;
#pragma unroll
    for (int i = 0; i < INNER * OUTER / W / NT; ++i) {
        const int lin = i * NT + (int)threadIdx.x, o = lin / (INNER / W), in = lin % (INNER / W) * W;
        const int left = (outer0 + o < outer_end) ? inner_end - (inner0 + in) : 0;      // elements from here to the row's end
        const int bytes = left >= W ? 4 * W : left > 0 ? 4 * left : 0;
        const float *p = src + (bytes ? (long long)(outer0 + o) * ld + inner0 + in : 0LL);
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(s + o * PITCH + in);
        if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(p), "r"(bytes) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(p), "r"(bytes) : "memory");
    }
}

// Four k of a thread's T rows (or columns): rows N apart where k is contiguous, else neighbours in groups of four, N groups apart.
template <int X, int T, int N, bool KC>
__device__ __forceinline__ void read4(float (&v)[T][4], const float *s, int t, int k) {
    if (KC) {
#pragma unroll
        for (int i = 0; i < T; ++i) {
            const float4 r = *reinterpret_cast<const float4 *>(s + (t + N * i) * (BK + 4) + k);
            v[i][0] = r.x; v[i][1] = r.y; v[i][2] = r.z; v[i][3] = r.w;
        }
    } else if (T % 4 == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < T; i += 4) {
                const float4 r = *reinterpret_cast<const float4 *>(s + (k + q) * (X + 4) + (t + N * (i / 4)) * 4);
                v[i][q] = r.x; v[i + 1][q] = r.y; v[i + 2][q] = r.z; v[i + 3][q] = r.w;
            }
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < T; i += 2) {
                const float2 r = *reinterpret_cast<const float2 *>(s + (k + q) * (X + 4) + t * T + i);
                v[i][q] = r.x; v[i + 1][q] = r.y;
            }
    }
}
template <int T, int N, bool KC>
__device__ __forceinline__ int place(int t, int i) { return KC ? t + N * i : T % 4 == 0 ? (t + N * (i / 4)) * 4 + i % 4 : t * T + i; }

// Behind the product, where FUSED: + bias (a row), and GELU of the result as a second output.
struct Behind { const float *bias; float *gelu; };

template <int BM, int BN, int TM, int TN, bool TA, bool TB, bool VEC, bool FUSED>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_small_k(int M, int N, int K, float alpha, const float *__restrict__ A, long long sA, const float *__restrict__ B,
                  long long sB, float beta, float *__restrict__ C, long long sC, Behind behind) {
    constexpr bool AKC = !TA, BKC = TB;
    constexpr int NX = BN / TN, NY = BM / TM, NT = NY * NX;
    constexpr int SA = slice_floats<BM, AKC>(), SB = slice_floats<BN, BKC>();
    extern __shared__ __align__(16) float smem[];
    // a warp is 8 threads of columns x 4 of rows: its reads of either operand are one pass of shared memory
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tx = warp % (NX / 8) * 8 + (lane & 7), ty = warp / (NX / 8) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    A += (long long)blockIdx.z * sA;
    B += (long long)blockIdx.z * sB;
    C += (long long)blockIdx.z * sC;
    const long long lda = TA ? M : K, ldb = TB ? K : N;

    float acc[TM][TN];
    unsigned long long acc2[TM][TN / 2];        // two columns each
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) { acc[i][j] = 0.0f; acc2[i][j / 2] = 0ull; }

    const int nk = (K + BK - 1) / BK;
    auto fetch = [&](int kt) {
        if (kt < nk) {
            float *s = smem + (kt % STAGES) * (SA + SB);
            copy_slice<BM, AKC, VEC, NT>(s, A, lda, m0, kt * BK, M, K);
            copy_slice<BN, BKC, VEC, NT>(s + SA, B, ldb, n0, kt * BK, N, K);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) fetch(i);
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                    // the slice is here for everyone, and the one before it has been read
        const float *as = smem + (kt % STAGES) * (SA + SB), *bs = as + SA;
        float a[2][TM][4], b[2][TN][4];     // the next four k are read beside the products of these
        read4<BM, TM, NY, AKC>(a[0], as, ty, 0);
        read4<BN, TN, NX, BKC>(b[0], bs, tx, 0);
        fetch(kt + STAGES - 1);
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            const int h = (k / 4) & 1;
            if (k + 4 < BK) {
                read4<BM, TM, NY, AKC>(a[h ^ 1], as, ty, k + 4);
                read4<BN, TN, NX, BKC>(b[h ^ 1], bs, tx, k + 4);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; j += 2) {
                        if (BKC) {
                            acc[i][j] = fmaf(a[h][i][q], b[h][j][q], acc[i][j]);
                            acc[i][j + 1] = fmaf(a[h][i][q], b[h][j + 1][q], acc[i][j + 1]);
                        } else {            // neighbouring columns came in one word: two chains in one instruction
                            unsigned long long aa, bb;
                            asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[h][i][q]));
                            asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b[h][j][q]), "f"(b[h][j + 1][q]));
                            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2[i][j / 2]) : "l"(aa), "l"(bb));
                        }
                    }
        }
    }
    if (!BKC) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; j += 2) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i][j]), "=f"(acc[i][j + 1]) : "l"(acc2[i][j / 2]));
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + place<TM, NY, AKC>(ty, i);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + place<TN, NX, BKC>(tx, j);
            if (n >= N) continue;
            float *c = C + (size_t)m * N + n;
            float o = alpha * acc[i][j];
            if (beta != 0.0f) o = fmaf(beta, *c, o);
            if (FUSED && behind.bias) o = __fadd_rn(o, __ldg(behind.bias + n));
            *c = o;
            if (FUSED && behind.gelu) behind.gelu[(size_t)m * N + n] = gelu_tanh(o);
        }
    }
}

template <int BM, int BN, int TM, int TN, bool TA, bool TB, bool VEC, bool FUSED>
int launch_small(int batch, int M, int N, int K, float alpha, const float *A, long long sA, const float *B, long long sB, float beta,
                 float *C, long long sC, const Behind &behind, cudaStream_t st) {
    constexpr int SMEM = STAGES * (slice_floats<BM, !TA>() + slice_floats<BN, TB>()) * 4;
    if (SMEM > 48 * 1024) {
        static std::mutex mu;
        static bool set[64];
        const int d = current_device();
        if (d < 0 || d >= 64) return BMB_E_UNSUPPORTED;
        std::lock_guard<std::mutex> lk(mu);
        if (!set[d]) {
            BMB_CUDA(cudaFuncSetAttribute(gemm_simt_small_k<BM, BN, TM, TN, TA, TB, VEC, FUSED>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
            set[d] = true;
        }
    }
    gemm_simt_small_k<BM, BN, TM, TN, TA, TB, VEC, FUSED><<<dim3(ceil_div(N, BN), ceil_div(M, BM), batch), (BM / TM) * (BN / TN), SMEM, st>>>(
        M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind);
    count_launch();
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}

template <bool TA, bool TB, bool VEC, bool FUSED = false>
int pick_small(int bm, int bn, int batch, int M, int N, int K, float alpha, const float *A, long long sA, const float *B, long long sB, float beta,
               float *C, long long sC, const Behind &behind, cudaStream_t st) {
    if (bn == 64) return launch_small<64, 64, 8, 4, TA, TB, VEC, FUSED>(batch, M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind, st);
    if (bm == 64) return launch_small<64, 32, 4, 4, TA, TB, VEC, FUSED>(batch, M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind, st);
    return launch_small<32, 32, 2, 4, TA, TB, VEC, FUSED>(batch, M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind, st);
}

}  // namespace

// BMB_E_UNSUPPORTED: the product has tiles enough for the 128 x 128 kernels. bias, gelu (may be null; op(A) = A, op(B) = B^T only):
// as bmb_bias_forward and bmb_gelu_forward behind it, to the bit, where those do not round (emit_rounded).
int gemm_simt_small(int transA, int transB, int batch, int M, int N, int K, float alpha, const float *A, long long sA, const float *B,
                    long long sB, float beta, float *C, long long sC, const float *bias, float *gelu, cudaStream_t st) {
    // Cycles per k of the SM with the most tiles: what one tile takes by itself, and each where there are several (measured, B with
    // k contiguous and not; 128 x 128 178 and 165).  One or two slices of K are over before the larger of the small
    // tiles has its copies under way (batch 128 of 64x64x32: 10.0 us against 6.7).
    const int sms = sm_count();
    auto cycles = [&](int x, int y, double alone, double each) {
        const long long per_sm = ceil_div((long long)ceil_div(M, x) * ceil_div(N, y) * batch, sms);
        return per_sm <= 1 ? alone : each * per_sm;
    };
    const double c128 = cycles(128, 128, 178, 165), c64 = K < 96 ? 1e300 : transB ? cycles(64, 64, 70, 56) : cycles(64, 64, 59, 53);
    const double c6432 = K < 96 ? 1e300 : transB ? cycles(64, 32, 42, 33) : cycles(64, 32, 41, 31), c32 = cycles(32, 32, 30, 23);
    if (c128 <= c64 && c128 <= c6432 && c128 <= c32) return BMB_E_UNSUPPORTED;
    const int bn = c64 <= c6432 && c64 <= c32 ? 64 : 32, bm = bn == 64 || c6432 <= c32 ? 64 : 32;
    if (ceil_div(M, bm) > 65535 || batch > 65535) return BMB_E_UNSUPPORTED;
    const bool vec = (((uintptr_t)A | (uintptr_t)B) & 15) == 0 && (transA ? M : K) % 4 == 0 && (transB ? K : N) % 4 == 0 &&
                     sA % 4 == 0 && sB % 4 == 0;
    const Behind behind{bias, gelu};
    if (bias || gelu) {
        if (transA || !transB || batch != 1) return BMB_E_UNSUPPORTED;
        return vec ? pick_small<false, true, true, true>(bm, bn, batch, M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind, st)
                   : pick_small<false, true, false, true>(bm, bn, batch, M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind, st);
    }
#define BMB_SMALL(TA, TB)                                                                                                       \
    return vec ? pick_small<TA, TB, true>(bm, bn, batch, M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind, st)                 \
               : pick_small<TA, TB, false>(bm, bn, batch, M, N, K, alpha, A, sA, B, sB, beta, C, sC, behind, st)
    if (!transA && !transB) BMB_SMALL(false, false);
    if (!transA) BMB_SMALL(false, true);
    if (!transB) BMB_SMALL(true, false);
    BMB_SMALL(true, true);
#undef BMB_SMALL
}

}  // namespace bmb
