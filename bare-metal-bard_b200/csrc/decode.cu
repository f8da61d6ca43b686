// Sampling in fp32 (src/train_gpt.cu:46-102): the forward pass of one position with the keys and values of the
// positions before it already in place, and the attention of one sequence's window.
//
// A distribution over tokens is an exponential of sums that every layer before it amplifies: two fp32 implementations
// of a model of 7 layers can differ by 1e-4 of it, and a text is only the same where every draw is. So everything here
// follows, operation by operation, the order that the pass over a whole batch has: products are the sequential chain of
// multiply-adds over k (as in the SIMT kernels), layernorm is the one-warp form, attention takes 8 keys at a time.
//
// One position: every product is a matrix times one vector, bound by launches, by one trip to L2 (where the weights of a
// model that samples in a loop stay) and by the chain, 4 cycles a step. So 32 outputs a block, one lane each, rows of
// weights copied to shared memory ahead of it, and what stands before or after the product (layernorm, residual, GELU)
// rides in the same launch: five launches a layer. Measured at 6 layers of 6 heads x 64,
// 256 positions: a text of 300 tokens, 45 of them past the context, 1075 -> 82 ms (the whole batch of 16 x 256 rows each token before).
#include "common.cuh"
#include <cmath>
#include <mutex>

namespace bmb {
namespace {

// The launches of one position form a chain in which each kernel may start while the one before it still runs: it lets its
// successor start at once, copies what does not depend on its predecessor (weights, earlier positions' values), and then
// waits for the predecessor's end -- so every kernel has waited for all before it when it ends.
// a warp that follows the chains and four that copy weights ahead of it; rows 4 banks apart
constexpr int GV_OUT = 32, GV_NT = 160, GV_CP = 128, GV_K = 128, GV_PITCH = GV_K + 4, GV_STAGES = 8;
constexpr int GV_MAX_IN = 4096, GV_MAX_LN = 1024;
constexpr int GV_SMEM = (GV_STAGES * GV_OUT * GV_PITCH + GV_MAX_IN) * 4;

// y[o] = f(W[o] . v + bias[o]) (+ add[o]), v = layernorm(x) when ln_w is given (each block for itself: a few hundred
// values against 32 rows of them), f = GELU when `gelu`. in % 4 == 0.
__global__ void __launch_bounds__(GV_NT) decode_gemv_k(float *__restrict__ y, const float *__restrict__ x, const float *__restrict__ W,
                                                       const float *__restrict__ bias, const float *__restrict__ ln_w,
                                                       const float *__restrict__ ln_b, const float *__restrict__ add, int in, int out, int gelu) {
    extern __shared__ __align__(16) float smem[];
    float *v = smem + GV_STAGES * GV_OUT * GV_PITCH;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, o0 = blockIdx.x * GV_OUT;
    const int nk = (in + GV_K - 1) / GV_K;
    auto fetch = [&](int kt) {
        if (kt < nk && warp > 0) {
            float *s = smem + (kt % GV_STAGES) * GV_OUT * GV_PITCH;
#pragma unroll
            for (int i = 0; i < GV_OUT * GV_K / 4 / GV_CP; ++i) {
                const int lin = i * GV_CP + (int)threadIdx.x - 32, r = lin / (GV_K / 4), c = lin % (GV_K / 4) * 4, k = kt * GV_K + c;
                const bool ok = o0 + r < out && k < in;
                const float *p = W + (ok ? (size_t)(o0 + r) * in + k : 0);
                const uint32_t d = (uint32_t)__cvta_generic_to_shared(s + r * GV_PITCH + c);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(p), "r"(ok ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    let_successor_start();
#pragma unroll
    for (int i = 0; i < GV_STAGES - 1; ++i) fetch(i);
    wait_for_predecessor();
    if (!ln_w) {
        for (int i = threadIdx.x * 4; i < in; i += GV_NT * 4) *reinterpret_cast<float4 *>(v + i) = *reinterpret_cast<const float4 *>(x + i);
    } else if (warp == 0) {
        // the sums of the one-warp layernorm, in its order
        const int n4 = in >> 2;
        float4 r[GV_MAX_LN / 128];
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < GV_MAX_LN / 128; ++i) {
            const int c4 = lane + 32 * i;
            r[i] = c4 < n4 ? *reinterpret_cast<const float4 *>(x + c4 * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            sum += (r[i].x + r[i].y) + (r[i].z + r[i].w);
        }
        const float mu = warp_sum(sum) / in;
        float sq = 0.0f;
#pragma unroll
        for (int i = 0; i < GV_MAX_LN / 128; ++i) {
            if (lane + 32 * i < n4) {
                const float a = r[i].x - mu, b = r[i].y - mu, c = r[i].z - mu, d = r[i].w - mu;
                sq += (a * a + b * b) + (c * c + d * d);
            }
        }
        const float var = warp_sum(sq) / in;
        const float rs = rsqrtf(var + 1e-5f);
#pragma unroll
        for (int i = 0; i < GV_MAX_LN / 128; ++i) {
            const int c4 = lane + 32 * i;
            if (c4 < n4) {
                const float4 w = *reinterpret_cast<const float4 *>(ln_w + c4 * 4), b = *reinterpret_cast<const float4 *>(ln_b + c4 * 4);
                float4 o;
                o.x = ((r[i].x - mu) * rs) * w.x + b.x;
                o.y = ((r[i].y - mu) * rs) * w.y + b.y;
                o.z = ((r[i].z - mu) * rs) * w.z + b.z;
                o.w = ((r[i].w - mu) * rs) * w.w + b.w;
                *reinterpret_cast<float4 *>(v + c4 * 4) = o;
            }
        }
    }
    float s = 0.0f;
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GV_STAGES - 2) : "memory");
        __syncthreads();
        fetch(kt + GV_STAGES - 1);
        if (warp != 0) continue;
        const float *w = smem + (kt % GV_STAGES) * GV_OUT * GV_PITCH + lane * GV_PITCH, *a = v + kt * GV_K;
        const int left = min(GV_K, in - kt * GV_K);
        auto step = [&](const float4 &p, const float4 &q) {
            s = fmaf(p.x, q.x, s); s = fmaf(p.y, q.y, s); s = fmaf(p.z, q.z, s); s = fmaf(p.w, q.w, s);
        };
        if (left == GV_K) {
            // the next 16 values are read while these 16 are added (the chain alone is 64 cycles)
            float4 p[2][4], q[2][4];
            auto read = [&](int k, int h) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    p[h][i] = *reinterpret_cast<const float4 *>(a + k + 4 * i);
                    q[h][i] = *reinterpret_cast<const float4 *>(w + k + 4 * i);
                }
            };
            read(0, 0);
#pragma unroll
            for (int k = 0; k < GV_K; k += 16) {
                const int h = (k / 16) & 1;
                if (k + 16 < GV_K) read(k + 16, h ^ 1);
#pragma unroll
                for (int i = 0; i < 4; ++i) step(p[h][i], q[h][i]);
            }
        } else {
            for (int k = 0; k < left; k += 4) step(*reinterpret_cast<const float4 *>(a + k), *reinterpret_cast<const float4 *>(w + k));
        }
    }
    const int o = o0 + lane;
    if (warp == 0 && o < out) {
        if (bias) s += bias[o];
        if (gelu) s = gelu_tanh(s);
        y[o] = add ? add[o] + s : s;
    }
}

// x = wte[token] + wpe[pos]
__global__ void decode_embed_k(float *__restrict__ x, const float *__restrict__ wte, const float *__restrict__ wpe, int token, int pos, int C) {
    for (int i = threadIdx.x; i < C; i += blockDim.x) x[i] = wte[(size_t)token * C + i] + wpe[(size_t)pos * C + i];
}

// ---- attention, 8 keys at a time -------------------------------------------------------------------------------------
constexpr int KC = 8;

// A score: HS/16 neighbouring lanes with 16 columns each, even and odd columns summed apart.
__device__ __forceinline__ unsigned long long pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void load_query(unsigned long long (&q2)[8], const float *q, float scale) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float4 v = *reinterpret_cast<const float4 *>(q + 2 * i);
        q2[i] = pack(v.x * scale, v.y * scale);
        q2[i + 1] = pack(v.z * scale, v.w * scale);
    }
}
template <int GL>
__device__ __forceinline__ float score(const unsigned long long (&q2)[8], const float *k) {
    unsigned long long acc = 0ull;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float4 v = *reinterpret_cast<const float4 *>(k + 2 * i);
        fma2(acc, q2[i], pack(v.x, v.y));
        fma2(acc, q2[i + 1], pack(v.z, v.w));
    }
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc));
    float s = lo + hi;
#pragma unroll
    for (int o = 1; o < GL; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// One head of the newest row against keys 0 .. pos; qkv: rows of 3C, the newest at `pos`. The running maximum before and
// after each 8 keys is a prefix maximum, so scores and exponentials are computed side by side and only the row sum and
// the output column of each thread follow the keys one after the other.
// smem: pos + 1 scores in whole groups of 8, two values a group, and, where they fit, the values of all keys, on their way
// while the scores are computed.
constexpr int DA_NT = 512, DA_MAX_V = 160 * 1024;
template <int HS>
__global__ void __launch_bounds__(DA_NT) decode_attention_k(float *__restrict__ y, const float *__restrict__ qkv, int pos, int C, float scale, int stage_v) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float total;
    constexpr int GL = HS / 16, KEYS = DA_NT / GL;
    const int n = pos + 1, groups = (n + KC - 1) / KC, tid = threadIdx.x, lane = tid & 31;
    float *vs = smem, *p = smem + (stage_v ? groups * KC * HS : 0);
    float *gmax = p + groups * KC, *gsum = gmax + groups;        // running maximum, then rescaling factor; sum of a group
    const long long ld = 3LL * C;
    const float *base = qkv + blockIdx.x * HS;
    const int sub = tid % GL;
    let_successor_start();
    if (stage_v) {
        bool waited = false;                                     // the newest position's row comes from the predecessor
        for (int i = tid; i < groups * KC * HS / 4; i += DA_NT) {
            const int j = i / (HS / 4), c = i % (HS / 4) * 4;
            if (j >= pos && !waited) { wait_for_predecessor(); waited = true; }
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(vs + j * HS + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(base + (long long)min(j, pos) * ld + 2 * C + c),
                         "r"(j < n ? 16 : 0) : "memory");
        }
    }
    wait_for_predecessor();
    unsigned long long q2[8];
    load_query(q2, base + (long long)pos * ld + sub * 16, scale);
#pragma unroll 2
    for (int j0 = 0; j0 < groups * KC; j0 += KEYS) {             // whole warps stay in the loop for the shuffles
        const int j = j0 + tid / GL;
        const float s = score<GL>(q2, base + (long long)min(j, pos) * ld + C + sub * 16);
        if (sub == 0 && j < groups * KC) p[j] = j < n ? s : -INFINITY;
    }
    __syncthreads();
    if (tid < 32) {
        float before = -INFINITY;
        for (int g0 = 0; g0 < groups; g0 += 32) {
            const int g = g0 + lane;
            float m = -INFINITY;
            if (g < groups) {
#pragma unroll
                for (int c = 0; c < KC; ++c) m = fmaxf(m, p[g * KC + c]);
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, m, o);
                if (lane >= o) m = fmaxf(m, up);
            }
            m = fmaxf(m, before);
            if (g < groups) gmax[g] = m;
            before = __shfl_sync(0xffffffffu, m, 31);
        }
    }
    __syncthreads();
    const float m = tid > 0 && tid < groups ? gmax[tid - 1] : -INFINITY, mnew = tid < groups ? gmax[tid] : -INFINITY;
    __syncthreads();                                             // maxima are read before factors take their place
    if (tid < groups) {                                          // (at most one group a thread)
        const bool live = mnew > -INFINITY;
        float csum = 0.0f;
#pragma unroll
        for (int c = 0; c < KC; ++c) {
            const float e = live ? __expf(p[tid * KC + c] - mnew) : 0.0f;
            p[tid * KC + c] = e;
            csum += e;
        }
        gmax[tid] = live ? __expf(m - mnew) : 1.0f;
        gsum[tid] = csum;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float o = 0.0f;
    if (tid < HS && stage_v) {
#pragma unroll 2
        for (int g = 0; g < groups; ++g) {                       // (a masked key's probability is zero, its value too)
            float x[KC], e[KC];
#pragma unroll
            for (int c = 0; c < KC; ++c) { x[c] = vs[(g * KC + c) * HS + tid]; e[c] = p[g * KC + c]; }
            o = fmaf(o, gmax[g], 0.0f);
#pragma unroll
            for (int c = 0; c < KC; ++c) o = fmaf(e[c], x[c], o);
        }
    } else if (tid < HS) {
        const float *v = base + 2 * C + tid;
        for (int j0 = 0; j0 < n; j0 += 4 * KC) {                 // 32 values under way at a time
            float x[4 * KC];
#pragma unroll
            for (int c = 0; c < 4 * KC; ++c) x[c] = j0 + c < n ? v[(long long)(j0 + c) * ld] : 0.0f;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (j0 + h * KC >= n) break;
                o = fmaf(o, gmax[j0 / KC + h], 0.0f);
#pragma unroll
                for (int c = 0; c < KC; ++c) o = fmaf(p[j0 + h * KC + c], x[h * KC + c], o);
            }
        }
    } else if (tid == HS) {
        float l = 0.0f;
        for (int g = 0; g < groups; ++g) l = l * gmax[g] + gsum[g];
        total = l;
    }
    __syncthreads();
    if (tid < HS) y[blockIdx.x * HS + tid] = o * ((total > 0.0f) ? 1.0f / total : 0.0f);
}

// All rows of one sequence's window: as decode_attention_k, WR neighbouring rows of a head a block, so that what is read of a key
// or value serves all of them.  Scores and exponentials are computed side by side and only a row's sum and its output follow the
// keys one after the other, a thread a column: at 256 positions of 6 heads x 64 10 us, against 38 for a walk over the keys in which
// every 8 of them waited for the 8 before.
// smem: the rows' queries, their scores in whole groups of 8, a factor and a sum a group, and, where they fit, the values.
constexpr int WR = 8, WA_NT = 256, WA_MAX_V = 96 * 1024;
template <int HS>
__global__ void __launch_bounds__(WA_NT) window_attention_k(float *__restrict__ out, const float *__restrict__ qkv, int T, int C, float scale, int stage_v) {
    extern __shared__ __align__(16) float smem[];
    constexpr int GL = HS / 16, KEYS = WA_NT / GL, SETS = WA_NT / HS, RT = WR / SETS;      // RT rows a thread in the output
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * WR, n = min(T, i0 + WR);      // longest blocks first
    const int groups = (n + KC - 1) / KC, keys = groups * KC;
    float *qs = smem, *p = qs + WR * HS, *factor = p + WR * keys, *gsum = factor + WR * groups, *vs = gsum + WR * groups;
    const long long ld = 3LL * C;
    const float *base = qkv + blockIdx.y * HS;
    if (stage_v) {
        for (int i = tid; i < keys * HS / 4; i += WA_NT) {
            const int j = i / (HS / 4), c = i % (HS / 4) * 4;
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(vs + j * HS + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(base + (long long)min(j, T - 1) * ld + 2 * C + c),
                         "r"(j < T ? 16 : 0) : "memory");
        }
    }
    for (int i = tid; i < WR * HS; i += WA_NT) qs[i] = base[(long long)min(i0 + i / HS, T - 1) * ld + i % HS] * scale;
    __syncthreads();
    const int sub = tid % GL;
    for (int j0 = 0; j0 < keys; j0 += KEYS) {                    // whole warps stay in the loop for the shuffles
        const int j = j0 + tid / GL;
        const float *k = base + (long long)min(j, T - 1) * ld + C + sub * 16;
        unsigned long long k2[8];
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            const float4 v = *reinterpret_cast<const float4 *>(k + 2 * i);
            k2[i] = pack(v.x, v.y);
            k2[i + 1] = pack(v.z, v.w);
        }
#pragma unroll
        for (int r = 0; r < WR; ++r) {
            unsigned long long acc = 0ull;
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                const float4 q = *reinterpret_cast<const float4 *>(qs + r * HS + sub * 16 + 2 * i);
                fma2(acc, pack(q.x, q.y), k2[i]);
                fma2(acc, pack(q.z, q.w), k2[i + 1]);
            }
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc));
            float s = lo + hi;
#pragma unroll
            for (int o = 1; o < GL; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (sub == 0 && j < keys) p[r * keys + j] = (j > i0 + r || j >= T) ? -INFINITY : s;
        }
    }
    __syncthreads();
    {
        // a warp a row: prefix maxima, 8 keys a lane, and with them the exponentials
        float *pr = p + warp * keys, before = -INFINITY;
        for (int g0 = 0; g0 < groups; g0 += 32) {
            const int g = g0 + lane;
            float x[KC], m = -INFINITY;
#pragma unroll
            for (int c = 0; c < KC; ++c) { x[c] = g < groups ? pr[g * KC + c] : -INFINITY; m = fmaxf(m, x[c]); }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, m, o);
                if (lane >= o) m = fmaxf(m, up);
            }
            const float mnew = fmaxf(m, before), up = __shfl_up_sync(0xffffffffu, mnew, 1), mold = lane ? up : before;
            before = __shfl_sync(0xffffffffu, mnew, 31);
            if (g < groups) {
                const bool live = mnew > -INFINITY;
                float csum = 0.0f;
#pragma unroll
                for (int c = 0; c < KC; ++c) {
                    const float e = live ? __expf(x[c] - mnew) : 0.0f;
                    pr[g * KC + c] = e;
                    csum += e;
                }
                factor[warp * groups + g] = live ? __expf(mold - mnew) : 1.0f;
                gsum[warp * groups + g] = csum;
            }
        }
    }
    if (stage_v) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int d = tid % HS, r0 = tid / HS * RT;
    float o[RT], l[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) o[r] = l[r] = 0.0f;
#pragma unroll 2
    for (int g = 0; g < groups; ++g) {
        float x[KC];
#pragma unroll
        for (int c = 0; c < KC; ++c) {
            const int j = g * KC + c;
            x[c] = stage_v ? vs[j * HS + d] : (j < T ? base[(long long)j * ld + 2 * C + d] : 0.0f);
        }
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            const float *e = p + (r0 + r) * keys + g * KC, f = factor[(r0 + r) * groups + g];
            l[r] = l[r] * f + gsum[(r0 + r) * groups + g];
            o[r] = fmaf(o[r], f, 0.0f);
#pragma unroll
            for (int c = 0; c < KC; ++c) o[r] = fmaf(e[c], x[c], o[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
        if (i0 + r0 + r < T) out[(long long)(i0 + r0 + r) * C + blockIdx.y * HS + d] = o[r] * ((l[r] > 0.0f) ? 1.0f / l[r] : 0.0f);
}

}  // namespace

// Sizes these kernels take: the attention's head sizes, a layernorm of one warp, and a context of at most 512 groups of
// 8 keys (one a thread in decode_attention_k).
bool decode_accepts(int T, int C, int NH) {
    const int hs = (NH > 0 && C % NH == 0) ? C / NH : 0;
    return (hs == 32 || hs == 64 || hs == 128) && C <= GV_MAX_LN && T <= DA_NT * KC;
}

int decode_embed(float *x, const float *wte, const float *wpe, int token, int pos, int C, cudaStream_t st) {
    decode_embed_k<<<1, 256, 0, st>>>(x, wte, wpe, token, pos, C);
    count_launch();
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}

int decode_gemv(float *y, const float *x, const float *W, const float *bias, const float *ln_w, const float *ln_b, const float *add,
                int in, int out, bool gelu, cudaStream_t st) {
    static std::mutex mu;
    static bool set[64];
    const int d = current_device();
    if (d < 0 || d >= 64 || in > GV_MAX_IN || (ln_w && in > GV_MAX_LN) || in % 4) return fail(BMB_E_UNSUPPORTED, "decode_gemv: %d inputs", in);
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!set[d]) BMB_CUDA(cudaFuncSetAttribute(decode_gemv_k, cudaFuncAttributeMaxDynamicSharedMemorySize, GV_SMEM));
        set[d] = true;
    }
    return launch_in_chain(decode_gemv_k, dim3(ceil_div(out, GV_OUT)), GV_NT, GV_SMEM, st, y, x, W, bias, ln_w, ln_b, add, in, out, gelu ? 1 : 0);
}

int decode_attention(float *y, const float *qkv, int pos, int C, int NH, cudaStream_t st) {
    const int hs = C / NH;
    const float scale = 1.0f / sqrtf((float)hs);
    const size_t groups = ceil_div(pos + 1, KC), v_bytes = groups * KC * hs * sizeof(float);
    const int stage_v = v_bytes <= DA_MAX_V;
    const size_t smem = (stage_v ? v_bytes : 0) + groups * (KC + 2) * sizeof(float);
    static std::mutex mu;
    static bool set[64];
    const int d = current_device();
    if (d < 0 || d >= 64) return fail(BMB_E_ARG, "device index %d out of range", d);
    {
        std::lock_guard<std::mutex> lk(mu);
        const int most = DA_MAX_V + DA_NT * (KC + 2) * (int)sizeof(float);
        if (!set[d]) {
            BMB_CUDA(cudaFuncSetAttribute(decode_attention_k<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
            BMB_CUDA(cudaFuncSetAttribute(decode_attention_k<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
            BMB_CUDA(cudaFuncSetAttribute(decode_attention_k<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        }
        set[d] = true;
    }
    if (hs == 32) return launch_in_chain(decode_attention_k<32>, dim3(NH), DA_NT, smem, st, y, qkv, pos, C, scale, stage_v);
    if (hs == 64) return launch_in_chain(decode_attention_k<64>, dim3(NH), DA_NT, smem, st, y, qkv, pos, C, scale, stage_v);
    return launch_in_chain(decode_attention_k<128>, dim3(NH), DA_NT, smem, st, y, qkv, pos, C, scale, stage_v);
}

template <int HS>
static int run_window(float *out, const float *qkv, int T, int C, int NH, cudaStream_t st) {
    static_assert(WA_NT / 32 == WR && WA_NT % HS == 0, "a warp a row, whole rows of columns");
    const size_t keys = (size_t)ceil_div(T, KC) * KC, v_bytes = keys * HS * sizeof(float);
    const int stage_v = v_bytes <= WA_MAX_V;
    const size_t smem = (WR * HS + WR * keys + 2 * WR * (keys / KC)) * sizeof(float) + (stage_v ? v_bytes : 0);
    static std::mutex mu;
    static bool set[64];
    const int d = current_device();
    if (d < 0 || d >= 64) return fail(BMB_E_ARG, "device index %d out of range", d);
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!set[d]) BMB_CUDA(cudaFuncSetAttribute(window_attention_k<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        set[d] = true;
    }
    window_attention_k<HS><<<dim3(ceil_div(T, WR), NH), WA_NT, smem, st>>>(out, qkv, T, C, 1.0f / sqrtf((float)HS), stage_v);
    count_launch();
    BMB_LAUNCH_CHECK();
    return BMB_OK;
}
int window_attention(float *out, const float *qkv, int T, int C, int NH, cudaStream_t st) {
    const int hs = C / NH;
    return hs == 32 ? run_window<32>(out, qkv, T, C, NH, st) : hs == 64 ? run_window<64>(out, qkv, T, C, NH, st) : run_window<128>(out, qkv, T, C, NH, st);
}

}  // namespace bmb
