// Sampling in fp32 (src/train_gpt.cu:46-102): the forward pass of one position with the keys and values of the
// positions before it already in place, and the attention of one sequence's window.
//
// A distribution over tokens is an exponential of sums that every layer before it amplifies: two fp32 implementations
// of a model of 7 layers can differ by 1e-4 of it, and a text is only the same where every draw is. So everything here
// follows, operation by operation, the order that the pass over a whole batch has: products are the sequential chain of
// multiply-adds over k (as in the SIMT kernels), layernorm is the one-warp form, attention takes 8 keys at a time.
//
// One position: every product is a matrix times one vector, bound by the trips to L2 that hand vectors on (where the weights of
// a model that samples in a loop stay) and by the chain, 4 cycles a step. So 32 outputs a warp, one lane each, rows of weights
// copied to shared memory ahead of it, what stands before or after the product (layernorm, residual, GELU) beside it, and all
// layers in one launch whose blocks wait for one another's results (decode_position_k).
#include "tc_common.cuh"
#include <cmath>
#include <mutex>

namespace bmb {
namespace {

// slices of 32 rows of weights and 128 inputs, rows 4 banks apart
constexpr int GV_OUT = 32, GV_K = 128, GV_PITCH = GV_K + 4, GV_STAGES = 8;
constexpr int GV_MAX_IN = 4096, GV_MAX_LN = 1024;

// s + w[0] a[0] + w[1] a[1] + .. in that order, `left` (a multiple of 4, at most GV_K) steps.
__device__ __forceinline__ float follow_chain(float s, const float *w, const float *a, int left) {
    auto step = [&](int k) {
        const float4 p = *reinterpret_cast<const float4 *>(a + k), q = *reinterpret_cast<const float4 *>(w + k);
        s = fmaf(p.x, q.x, s); s = fmaf(p.y, q.y, s); s = fmaf(p.z, q.z, s); s = fmaf(p.w, q.w, s);
    };
    if (left == GV_K) {
#pragma unroll
        for (int k = 0; k < GV_K; k += 4) step(k);
    } else {
        for (int k = 0; k < left; k += 4) step(k);
    }
    return s;
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
template <int GL, typename Part>
__device__ __forceinline__ float score(const unsigned long long (&q2)[8], Part part) {
    unsigned long long acc = 0ull;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float4 v = part(i / 2);
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

template <int GL>
__device__ __forceinline__ float score(const unsigned long long (&q2)[8], const float *k) {
    return score<GL>(q2, [&](int c) { return *reinterpret_cast<const float4 *>(k + 4 * c); });
}

// One head of the newest row against keys 0 .. pos; qkv: rows of 3C, the newest at `pos`. The running maximum before and
// after each 8 keys is a prefix maximum, so scores and exponentials are computed side by side and only the row sum and
// the output column of each thread follow the keys one after the other.
// smem: pos + 1 scores in whole groups of 8, two values a group, and, where they fit, the values or both the values and the keys
// before the newest, copied while the newest is waited for (stage: 0, 1, 2 of the two).
constexpr int DA_NT = 512, DA_MAX_V = 160 * 1024;
// `newest` puts the newest position's query, key and value (HS each) where its argument points and returns, for all threads
// alike, whether it could; `put` takes output column d.
template <int HS, typename Newest, typename Put>
__device__ __forceinline__ bool decode_head(float *smem, const float *qkv, int pos, int C, int head, float scale, int stage, Newest newest, Put put) {
    __shared__ float total;
    __shared__ __align__(16) float last[3 * HS];
    constexpr int GL = HS / 16, KEYS = DA_NT / GL;
    const int n = pos + 1, groups = (n + KC - 1) / KC, tid = threadIdx.x, lane = tid & 31;
    float *vs = smem, *ks = smem + groups * KC * HS, *p = smem + stage * groups * KC * HS;
    // (a key's 16-byte parts, so that the 8 lanes of a phase of a 16-byte read find 8 bank groups)
    auto place = [&](int j, int c) { return ks + j * HS + 4 * (c ^ (((c >> 3) + j * (HS / 32)) & 3)); };
    float *gmax = p + groups * KC, *gsum = gmax + groups;        // running maximum, then rescaling factor; sum of a group
    const long long ld = 3LL * C;
    const float *base = qkv + head * HS;
    const int sub = tid % GL;
    auto copy = [&](float *to, const float *from) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from) : "memory");
    };
    if (stage == 2)                                              // the rows before the newest
        for (int i = tid; i < pos * (HS / 4); i += DA_NT) copy(place(i / (HS / 4), i % (HS / 4)), base + (long long)(i / (HS / 4)) * ld + C + i % (HS / 4) * 4);
    if (stage)
        for (int i = tid; i < pos * (HS / 4); i += DA_NT) copy(vs + 4 * i, base + (long long)(i / (HS / 4)) * ld + 2 * C + i % (HS / 4) * 4);
    if (stage == 2) asm volatile("cp.async.wait_all;" ::: "memory");
    if (!newest(last)) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        return false;
    }
    if (stage)
        for (int i = tid; i < (groups * KC - pos) * HS; i += DA_NT) vs[pos * HS + i] = i < HS ? last[2 * HS + i] : 0.0f;
    unsigned long long q2[8];
    load_query(q2, last + sub * 16, scale);
#pragma unroll 2
    for (int j0 = 0; j0 < groups * KC; j0 += KEYS) {             // whole warps stay in the loop for the shuffles
        const int j = j0 + tid / GL;
        const float s = stage == 2 ? score<GL>(q2, [&](int c) { return *reinterpret_cast<const float4 *>(j < pos ? place(j, sub * 4 + c) : last + HS + sub * 16 + 4 * c); })
                                   : score<GL>(q2, j < pos ? base + (long long)j * ld + C + sub * 16 : last + HS + sub * 16);
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
    if (tid < HS && stage) {
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
            for (int c = 0; c < 4 * KC; ++c) x[c] = j0 + c < pos ? v[(long long)(j0 + c) * ld] : j0 + c == pos ? last[2 * HS + tid] : 0.0f;
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
    if (tid < HS) put(tid, o * ((total > 0.0f) ? 1.0f / total : 0.0f));
    __syncthreads();                                             // shared memory may be overwritten
    return true;
}

// ---- one position through all layers ------------------------------------------------------------------------------------
// A launch for a position: blocks of 32 outputs of every product, one or more a block, and a block a head. A block knows its
// tiles of all layers beforehand: one warp copies their weights ahead into a ring, eight read the vector of the next product as it
// comes, and one normalises it, follows the chains and hands the results on. Every value is handed on as a pair with a tag (launch
// and layer), written and read as one 8-byte word: who reads a vector reads until all tags are right, 0.5 us after the last was
// written. (A count behind a fence, which the reader polls before it reads, took 2.5 us; one warp reading 1536 pairs in turns 3.2.)
// A value is written again a layer later only when everyone has read it, since each product reads all of what comes before it.
// All blocks have to be there: a cooperative launch.
// Bound by what follows one on the other: 9 C steps of the chains a layer (6.3 cycles a step; 4 is the instruction's latency), five
// hand-overs and the attention. At 6 heads x 64 and 150 positions a layer takes 16 us; as five launches, each started beside the
// end of the one before, it took 33.
constexpr int DP_NT = DA_NT, DP_LOAD = 8;                        // warps that read vectors
constexpr int DP_SMEM = (GV_STAGES * GV_OUT * GV_PITCH + GV_MAX_IN + 3 * GV_MAX_LN) * 4;         // weights, a vector as read, layernorm
enum { DP_QKV = 0, DP_PROJ, DP_FC, DP_FCPROJ, DP_HEAD };
constexpr long long DP_WAIT = 4000000000LL;                       // about two seconds
struct DecodeJob { const float *W; int in, rows, step, layer, o0; };       // 32 (or fewer) rows of a product's weights
// the vectors handed on, in pairs
__host__ __device__ constexpr int ex_x(int) { return 0; }
__host__ __device__ constexpr int ex_x2(int C) { return C; }
__host__ __device__ constexpr int ex_y(int C) { return 2 * C; }
__host__ __device__ constexpr int ex_qkv(int C) { return 3 * C; }
__host__ __device__ constexpr int ex_h(int C) { return 6 * C; }
__host__ __device__ constexpr int ex_size(int C) { return 10 * C; }

// (One 64-bit access a pair: the halves of a vector access are accesses of their own, in no order.)
__device__ __forceinline__ void put_pair(uint2 *p, float v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)tag << 32 | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ bool get_pair(const uint2 *p, unsigned tag, float &v) {
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    v = __uint_as_float((uint32_t)a);
    return (uint32_t)(a >> 32) == tag;
}
__device__ __forceinline__ bool get_pairs4(const uint2 *p, unsigned tag, float4 &v) {
    unsigned long long a[4];
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a[0]), "=l"(a[1]) : "l"(p) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a[2]), "=l"(a[3]) : "l"(p + 2) : "memory");
    v = make_float4(__uint_as_float((uint32_t)a[0]), __uint_as_float((uint32_t)a[1]), __uint_as_float((uint32_t)a[2]), __uint_as_float((uint32_t)a[3]));
    return (uint32_t)(a[0] >> 32) == tag && (uint32_t)(a[1] >> 32) == tag && (uint32_t)(a[2] >> 32) == tag && (uint32_t)(a[3] >> 32) == tag;
}
// Calls `look` until it is true for this thread; false when the limit ran out.
template <typename Look>
__device__ __forceinline__ bool look_until(Look look, int *status) {
    if (look()) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (look()) return true;
        if (clock64() - t0 > DP_WAIT) {
            *reinterpret_cast<volatile int *>(status) = 10;
            __threadfence_system();
            return false;
        }
    }
}

template <int HS>
__global__ void __launch_bounds__(DP_NT) decode_position_k(const DecodeModel m, const float *__restrict__ x0, const float *__restrict__ x1, int first, int pos, int stage, unsigned tag0, int *__restrict__ status) {
    extern __shared__ __align__(16) float smem[];
    __shared__ uint64_t bars[2 * GV_STAGES + 2];
    __shared__ int giveup;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, C = m.C;
    const int gemv_blocks = (int)gridDim.x - m.NH;

    if ((int)blockIdx.x >= gemv_blocks) {
        const int head = (int)blockIdx.x - gemv_blocks;
        for (int l = first; l < m.L; ++l) {
            const unsigned tag = tag0 + l;
            const bool ok = decode_head<HS>(smem, m.qkv + l * m.layer, pos, C, head, m.scale, stage, [&](float *last) {
                bool here = true;
                if (threadIdx.x < 3 * HS) {
                    const int part = threadIdx.x / HS, d = threadIdx.x % HS;
                    const uint2 *p = m.exchange + ex_qkv(C) + part * C + head * HS + d;
                    float v;
                    here = look_until([&]() { return get_pair(p, tag, v); }, status);
                    last[threadIdx.x] = v;
                }
                return __syncthreads_and(here) != 0;
            }, [&](int d, float o) { put_pair(m.exchange + ex_y(C) + head * HS + d, o, tag); });
            if (!ok) return;
        }
        return;
    }

    const uint32_t full0 = tc::smem_u32(bars), empty0 = full0 + 8 * GV_STAGES, loaded = empty0 + 8 * GV_STAGES, wanted = loaded + 8;
    if (threadIdx.x == 0) {
        for (int i = 0; i < GV_STAGES; ++i) { tc::mbar_init(full0 + 8 * i, 1); tc::mbar_init(empty0 + 8 * i, 1); }
        tc::mbar_init(loaded, DP_LOAD);
        tc::mbar_init(wanted, 1);
        giveup = 0;
        tc::mbar_init_fence();
    }
    __syncthreads();
    if (warp >= 2 + DP_LOAD) return;
    // This block's tiles, in the order of their use: those of a layer are counted through, then those of the head.
    const int tc_ = C / GV_OUT, per_layer = 9 * tc_;
    auto jobs = [&](auto use) {
        for (int l = first; l < m.L; ++l)
            for (int i = blockIdx.x; i < per_layer; i += gemv_blocks) {
                DecodeJob j{nullptr, C, GV_OUT, DP_QKV, l, 0};
                const size_t lC = (size_t)l * C;
                if (i < 3 * tc_) { j.o0 = i * GV_OUT; j.W = m.qkvw + 3 * lC * C; }
                else if (i < 4 * tc_) { j.step = DP_PROJ; j.o0 = (i - 3 * tc_) * GV_OUT; j.W = m.apw + lC * C; }
                else if (i < 8 * tc_) { j.step = DP_FC; j.o0 = (i - 4 * tc_) * GV_OUT; j.W = m.fcw + 4 * lC * C; }
                else { j.step = DP_FCPROJ; j.o0 = (i - 8 * tc_) * GV_OUT; j.W = m.fpw + 4 * lC * C; j.in = 4 * C; }
                if (!use(j)) return;
            }
        for (int o = blockIdx.x * GV_OUT; o < m.Vp; o += gemv_blocks * GV_OUT)
            if (!use(DecodeJob{m.wte, C, min(GV_OUT, m.Vp - o), DP_HEAD, m.L, o})) return;
    };
    int s = 0;
    uint32_t ph = 0;
    if (warp == 1) {
        int armed = 0, first = 0;                                // stages copied to; the one of the oldest copy that may be under way
        jobs([&](const DecodeJob &j) {
            for (int k = 0; k < j.in; k += GV_K) {
                if (!__all_sync(0xffffffffu, tc::mbar_wait(empty0 + 8 * s, ph ^ 1, &giveup))) return false;
                const uint32_t bytes = (uint32_t)min(GV_K, j.in - k) * 4;
                if (lane == 0) tc::mbar_arrive_expect_tx(full0 + 8 * s, bytes * j.rows);
                __syncwarp();
                if (lane < j.rows)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(tc::smem_u32(smem + (s * GV_OUT + lane) * GV_PITCH)), "l"(j.W + (size_t)(j.o0 + lane) * j.in + k), "r"(bytes),
                                 "r"(full0 + 8 * s) : "memory");
                ++armed;
                if (++s == GV_STAGES) { s = 0; ph ^= 1; }
            }
            return true;
        });
        first = max(0, armed - GV_STAGES);                       // nothing is left in flight, however this ends
        for (int i = first; i < armed; ++i) tc::mbar_drain(full0 + 8 * (i % GV_STAGES), (uint32_t)(i / GV_STAGES & 1));
        return;
    }
    constexpr int RAW = GV_STAGES * GV_OUT * GV_PITCH, NORMED = RAW + GV_MAX_IN;      // a vector as read, and after the layernorm
    int vectors = 0, step = -1, layer = -1;                       // how many so far; of the product and layer that the last one was for
    if (warp >= 2) {
        jobs([&](const DecodeJob &j) {
            if (j.step == step && j.layer == layer) return true;  // (several tiles of one product)
            step = j.step; layer = j.layer;
            const unsigned tag = tag0 + j.layer, want = j.step == DP_QKV || j.step == DP_HEAD ? tag - 1 : tag;
            const uint2 *x = m.exchange + (j.step == DP_PROJ ? ex_y(C) : j.step == DP_FC ? ex_x2(C) : j.step == DP_FCPROJ ? ex_h(C) : ex_x(C));
            bool ok = tc::mbar_wait(wanted, (uint32_t)(vectors & 1), &giveup);      // (the one before is no longer read; and looks beside a chain slow it down)
            ++vectors;
            for (int i = ((int)threadIdx.x - 64) * 4; ok && i < j.in; i += DP_LOAD * 128) {
                float4 v;
                if (j.layer == first && (j.step == DP_QKV || j.step == DP_HEAD)) {
                    v = __ldg(reinterpret_cast<const float4 *>(x0 + i));
                    if (x1) {
                        const float4 a = __ldg(reinterpret_cast<const float4 *>(x1 + i));
                        v = make_float4(v.x + a.x, v.y + a.y, v.z + a.z, v.w + a.w);
                    }
                } else {
                    ok = look_until([&]() { return get_pairs4(x + i, want, v); }, status);
                }
                *reinterpret_cast<float4 *>(smem + RAW + i) = v;
            }
            if (!ok) giveup = 1;
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(loaded);
            return *reinterpret_cast<volatile int *>(&giveup) == 0;
        });
        return;
    }
    int v = 0;                                                    // where the vector of a product lies in `smem`
    jobs([&](const DecodeJob &j) {
        const int l = j.layer, o = j.o0 + lane;
        const unsigned tag = tag0 + l;
        bool ok = true;
        // what is added to this lane's output
        float bias = 0.0f, add = 0.0f;
        if (j.step != DP_HEAD)
            bias = __ldg((j.step == DP_QKV ? m.qkvb + (size_t)l * 3 * C : j.step == DP_PROJ ? m.apb + (size_t)l * C : j.step == DP_FC ? m.fcb + (size_t)l * 4 * C
                                                                                                          : m.fpb + (size_t)l * C) + o);
        if (j.step == DP_PROJ && l == first) add = x1 ? x0[o] + x1[o] : x0[o];     // (complete before the product's own vector is)
        if (j.step == DP_PROJ && l > first) ok = look_until([&]() { return get_pair(m.exchange + ex_x(C) + o, tag - 1, add); }, status);
        if (j.step == DP_FCPROJ) ok = look_until([&]() { return get_pair(m.exchange + ex_x2(C) + o, tag, add); }, status);
        const int stages = (j.in + GV_K - 1) / GV_K;
        for (int i = 0, s1 = s, ph1 = ph; i < min(stages, GV_STAGES); ++i) {       // the weights are there long before the vector
            ok = ok && tc::mbar_wait(full0 + 8 * s1, ph1, &giveup);
            if (++s1 == GV_STAGES) { s1 = 0; ph1 ^= 1; }
        }
        if (j.step != step || l != layer) {
            step = j.step; layer = l;
            if (lane == 0) tc::mbar_arrive(wanted);
            const bool norm = j.step == DP_QKV || j.step == DP_FC || j.step == DP_HEAD;
            const int n4 = C >> 2;
            float4 *gain = reinterpret_cast<float4 *>(smem + NORMED + GV_MAX_LN), *shift = gain + GV_MAX_LN / 4;
            if (norm) {                                           // (read before the vector is waited for)
                const float *w = (j.step == DP_QKV ? m.ln1w : j.step == DP_FC ? m.ln2w : m.lnfw) + (j.step == DP_HEAD ? 0 : (size_t)l * C);
                const float *b = (j.step == DP_QKV ? m.ln1b : j.step == DP_FC ? m.ln2b : m.lnfb) + (j.step == DP_HEAD ? 0 : (size_t)l * C);
                for (int i = lane; i < n4; i += 32) {
                    const float4 a = __ldg(reinterpret_cast<const float4 *>(w) + i), c = __ldg(reinterpret_cast<const float4 *>(b) + i);
                    gain[i] = a;
                    shift[i] = c;
                }
            }
            ok = __all_sync(0xffffffffu, ok && tc::mbar_wait(loaded, (uint32_t)(vectors & 1), &giveup) && *reinterpret_cast<volatile int *>(&giveup) == 0);
            if (!ok) {
                if (lane == 0) giveup = 1;
                return false;
            }
            ++vectors;
            v = RAW;
            if (norm) {
                // the sums of the one-warp layernorm, in its order
                constexpr int N4 = GV_MAX_LN / 128;
                float4 r[N4];
                float sum = 0.0f;
#pragma unroll
                for (int i = 0; i < N4; ++i) {
                    if (32 * i >= n4) break;
                    r[i] = lane + 32 * i < n4 ? *reinterpret_cast<const float4 *>(smem + v + (lane + 32 * i) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
                    sum += (r[i].x + r[i].y) + (r[i].z + r[i].w);
                }
                const float mu = warp_sum(sum) / C;
                float sq = 0.0f;
#pragma unroll
                for (int i = 0; i < N4; ++i) {
                    if (32 * i >= n4) break;
                    if (lane + 32 * i < n4) {
                        const float a = r[i].x - mu, c = r[i].y - mu, d = r[i].z - mu, e = r[i].w - mu;
                        sq += (a * a + c * c) + (d * d + e * e);
                    }
                }
                const float var = warp_sum(sq) / C;
                const float rs = rsqrtf(var + 1e-5f);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < N4; ++i) {
                    if (32 * i >= n4) break;
                    if (lane + 32 * i < n4) {
                        const float4 g = gain[lane + 32 * i], a = shift[lane + 32 * i];
                        float4 y;
                        y.x = ((r[i].x - mu) * rs) * g.x + a.x;
                        y.y = ((r[i].y - mu) * rs) * g.y + a.y;
                        y.z = ((r[i].z - mu) * rs) * g.z + a.z;
                        y.w = ((r[i].w - mu) * rs) * g.w + a.w;
                        *reinterpret_cast<float4 *>(smem + NORMED + (lane + 32 * i) * 4) = y;
                    }
                }
                __syncwarp();
                v = NORMED;
            }
        }
        float sum = 0.0f;
        for (int i = 0; i < stages; ++i) {
            if (i >= GV_STAGES) ok = tc::mbar_wait(full0 + 8 * s, ph, &giveup) && ok;
            sum = follow_chain(sum, smem + (s * GV_OUT + lane) * GV_PITCH, smem + v + i * GV_K, min(GV_K, j.in - i * GV_K));
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(empty0 + 8 * s);
            if (++s == GV_STAGES) { s = 0; ph ^= 1; }
        }
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0) giveup = 1;
            return false;
        }
        if (lane < j.rows) {
            if (j.step == DP_QKV) {
                put_pair(m.exchange + ex_qkv(C) + o, sum + bias, tag);
                m.qkv[l * m.layer + (size_t)pos * 3 * C + o] = sum + bias;       // for the positions to come
            } else if (j.step == DP_PROJ) {
                sum += bias;
                put_pair(m.exchange + ex_x2(C) + o, add + sum, tag);
            } else if (j.step == DP_FC) {
                put_pair(m.exchange + ex_h(C) + o, gelu_tanh(sum + bias), tag);
            } else if (j.step == DP_FCPROJ) {
                sum += bias;
                put_pair(m.exchange + ex_x(C) + o, add + sum, tag);
            } else {
                m.logits[o] = sum;
            }
        }
        return true;
    });
}

// All rows of one sequence's window: as decode_head, WR neighbouring rows of a head a block, so that what is read of a key
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
// 8 keys (one a thread in decode_head).
bool decode_accepts(int T, int C, int NH) {
    const int hs = (NH > 0 && C % NH == 0) ? C / NH : 0;
    return (hs == 32 || hs == 64 || hs == 128) && C <= GV_MAX_LN && T <= DA_NT * KC;
}

// Pairs of 8 bytes that the launches of decode_position hand vectors on in; zero before the first.
size_t decode_exchange(int C) { return (size_t)ex_size(C); }

template <int HS>
static int run_position(const DecodeModel &m, const float *x0, const float *x1, int first, int pos, unsigned launch, cudaStream_t st) {
    const size_t groups = ceil_div(pos + 1, KC), v_bytes = groups * KC * HS * sizeof(float);
    int stage = 2 * v_bytes <= DA_MAX_V ? 2 : v_bytes <= DA_MAX_V ? 1 : 0;
    const size_t att = stage * v_bytes + groups * (KC + 2) * sizeof(float), smem = att > DP_SMEM ? att : DP_SMEM;
    static std::mutex mu;
    static bool set[64];
    const int d = current_device();
    if (d < 0 || d >= 64) return fail(BMB_E_ARG, "device index %d out of range", d);
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!set[d])
            BMB_CUDA(cudaFuncSetAttribute(decode_position_k<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, DA_MAX_V + DA_NT * (KC + 2) * (int)sizeof(float)));
        set[d] = true;
    }
    int *status_dev = nullptr;
    volatile int *status_host = nullptr;
    BMB_TRY(tc::status_word(&status_dev, &status_host));
    if (*status_host != 0) return fail(BMB_E_TIMEOUT, "an earlier kernel on this device gave up waiting");
    const int tiles = 9 * m.C / GV_OUT, room = sm_count() - m.NH, blocks = (tiles < room ? tiles : room) + m.NH;
    unsigned tag0 = launch * (unsigned)m.L + 1;
    DecodeModel model = m;
    void *args[] = {&model, &x0, &x1, &first, &pos, &stage, &tag0, &status_dev};
    BMB_CUDA(cudaLaunchCooperativeKernel((const void *)decode_position_k<HS>, dim3(blocks), dim3(DP_NT), args, smem, st));
    count_launch();
    return BMB_OK;
}
int decode_position(const DecodeModel &m, const float *x0, const float *x1, int first, int pos, unsigned launch, cudaStream_t st) {
    const int hs = m.C / m.NH;
    return hs == 32 ? run_position<32>(m, x0, x1, first, pos, launch, st)
                    : hs == 64 ? run_position<64>(m, x0, x1, first, pos, launch, st) : run_position<128>(m, x0, x1, first, pos, launch, st);
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
