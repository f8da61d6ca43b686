// Shared host/device helpers for libbmb: status plumbing, the per-thread
// stream, per-device scratch, and small device utilities.
#pragma once
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdarg>
#include <cstdint>
#include <mutex>
#include "../../include/bmb.h"

namespace bmb {

// ---- status -------------------------------------------------------------
int fail(int code, const char *fmt, ...);

#define BMB_CUDA(x)                                                           \
    do {                                                                      \
        cudaError_t e__ = (x);                                                \
        if (e__ != cudaSuccess)                                               \
            return ::bmb::fail(BMB_E_CUDA, "%s -> %s (%s:%d)", #x,            \
                               cudaGetErrorString(e__), __FILE__, __LINE__);  \
    } while (0)

// After a kernel launch: report a launch-configuration error, never sync.
#define BMB_LAUNCH_CHECK()                                                    \
    do {                                                                      \
        cudaError_t e__ = cudaGetLastError();                                 \
        if (e__ != cudaSuccess)                                               \
            return ::bmb::fail(BMB_E_CUDA, "launch -> %s (%s:%d)",            \
                               cudaGetErrorString(e__), __FILE__, __LINE__);  \
    } while (0)

#define BMB_TRY(x)                                                            \
    do {                                                                      \
        int s__ = (x);                                                        \
        if (s__ != BMB_OK) return s__;                                        \
    } while (0)

// ---- per-thread stream ----------------------------------------------------
cudaStream_t cur_stream();

// Per-thread switch read by the kernels that produce GEMM / attention operands
// (layernorm, GELU, bias add, cross-entropy backward, attention): when on, they
// store TF32-rounded values so that the tensor-core kernels can read them in
// place.  The training step turns it on in TF32 mode; the C ABI leaves it off.
bool emit_rounded();
void set_emit_rounded(bool on);

// ---- deferred column sums --------------------------------------------------
// The parameter-gradient sums of the backward kernels are two-stage: a kernel leaves G partial rows, a small
// launch adds them up in a fixed order.  While a collector is installed for the calling thread, those kernels take
// their partial rows from the collector's arena (instead of the shared per-device scratch, which the next call
// would overwrite) and only note the final sum as a job; one batched launch at the end of the backward pass then
// does all of them -- the same sums in the same order, a few dozen launches fewer.
struct ColumnAddJob {
    float *dst, *dst2, *dst3;     // as launch_column_add: columns [ncols_first, ..) go to dst2, from 2 * ncols_first on to dst3
    const float *partial;
    int ncols_first, G, ncols;
};
struct ColumnAddCollector {
    float *arena = nullptr;       // device memory for the partial rows of one backward pass
    size_t cap = 0, used = 0;     // floats
    ColumnAddJob *jobs = nullptr; // host array, filled while `record` is set (the job list is the same every pass)
    int max_jobs = 0, njobs = 0, max_cols = 0;
    bool record = false;
};
void set_column_add_collector(ColumnAddCollector *c);      // nullptr: sums are finished by their own launches again
int launch_column_add_jobs(const ColumnAddJob *jobs_dev, int njobs, int max_cols, cudaStream_t st);

// ---- data-parallel exchange: a list of ranges of a flat float buffer ------
// (offsets and lengths in floats, each a multiple of 4)
constexpr int DP_MAX_RANGES = 16;
struct DpRangeList {
    unsigned long long off[DP_MAX_RANGES], len[DP_MAX_RANGES];
    int n;
};

// ---- per-device scratch ---------------------------------------------------
// The reference keeps process-wide static device scratch (src/nn.cu:347, 362)
// that every rank thread shares regardless of device.  Here each device owns
// its own block, grown on demand and kept until process exit.
// Returns nullptr (and records an error) on failure.
enum ScratchSlot { SCR_REDUCE = 0, SCR_GEMM_A = 1, SCR_GEMM_B = 2, SCR_MISC = 3, SCR_SPLIT = 4, SCR_SLOTS = 5 };
void *device_scratch(ScratchSlot slot, size_t bytes);
// Order the users of a scratch slot across streams of one device: acquire before the first launch that writes
// the slot, release after the last launch that reads it (both on the stream those launches go to).
int scratch_acquire(ScratchSlot slot, cudaStream_t st);
int scratch_release(ScratchSlot slot, cudaStream_t st);
// The release of a block that a call has acquired, at the call's end (its last launch reads the block).
struct ScratchRelease {
    ScratchSlot slot;
    cudaStream_t st;
    bool on;
    ~ScratchRelease() { if (on) scratch_release(slot, st); }
};
// The slots (bit 1 << slot) that this thread's calls have taken blocks of since the last call of this function: what a
// captured graph holds, so that its replays can take their turn at them.
unsigned scratch_slots_taken();
// Counts the times any scratch block of the current device but SCR_SPLIT was (re)allocated.  A caller that keeps
// scratch addresses beyond one call (the trainer's captured graph) compares it before reusing them.
unsigned long long scratch_generation();
int current_device();
int sm_count();

// Launch counter (all kernels launched by this library in this process).
void count_launch(int n = 1);
long long launches_total();

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// Internal flag of gemm_any_bias: the launches of a captured stream may use the per-device scratch, because the caller
// has sized it by an eager pass, keeps its products in one line and watches scratch_generation().  Without it, products
// that need scratch stay out of captures.
constexpr int GEMM_SCRATCH_IN_CAPTURE = 1 << 20;
// Internal flag: nobody compares this product's elements with the sequential fp32 chain, so a split product may serve
// small ones too.
constexpr int GEMM_ANY_ORDER = 1 << 21;
// Internal flag: an fp32 product must be the sequential chain over k.
constexpr int GEMM_CHAIN = 1 << 22;
// SCR_SPLIT (the images of split fp32 products) is sized, handed over and used under this lock of the current device, held
// from the scratch's address to the last launch that reads it: products of several threads and streams take turns, and the
// block is not moved under one of them.  These functions are called with the lock held.
std::mutex &split_mutex();
// The block, at least `bytes` long, to be acquired for `st`; nullptr where there is no memory, or `st` is being captured and
// the block would have to grow.  Growing waits for the block's last use.
void *split_scratch(size_t bytes, cudaStream_t st);
// Waits for the block's last use and frees it if it is larger than `above` bytes and nobody keeps it (trainers do, one count
// each: their captured steps hold its address).
void split_scratch_give_back(size_t above);
void split_scratch_keep(int change);
unsigned long long split_scratch_generation();      // counts the block's moves, as scratch_generation() those of the others
// A block for one call's launches on `st` (not captured), until call_scratch_done: calls on several streams have blocks of their own, up to
// CALL_SCRATCH_KEPT bytes of a device in all (a larger one is given back by the call that took it); beyond that they take turns.
// nullptr: there is no memory.
constexpr size_t CALL_SCRATCH_KEPT = 1ull << 30;
void *call_scratch(size_t bytes, cudaStream_t st);
int call_scratch_done(void *p, cudaStream_t st);
// Internal GEMM dispatch shared by attention and the trainer: math is a
// BMB_MATH_* value, flags the BMB_GEMM_* bits, strides in elements.
int gemm_any(int math, int flags, int ta, int tb, int batch, int M, int N, int K, float alpha,
             const float *A, long long sA, const float *B, long long sB, float beta, float *C,
             long long sC, cudaStream_t st);
// Same with a bias row added to every output row (null = none).
int gemm_any_bias(int math, int flags, int ta, int tb, int batch, int M, int N, int K, float alpha,
                  const float *A, long long sA, const float *B, long long sB, float beta, float *C,
                  long long sC, const float *bias, cudaStream_t st, float *aux_gelu = nullptr);
// (aux_gelu: a second output of the same shape, GELU of the result -- in the product's epilogue where the
//  tensor-core kernel can, by a pass of its own otherwise)

// bmb_flash_attention_*_ex; in_trainer: forward and backward both run, and, as with GEMM_SCRATCH_IN_CAPTURE, a captured stream's
// launches may use SCR_SPLIT, because the caller has sized it and takes care of its moves.
int flash_forward(int cfg, int flags, float *out, float *lse, const float *qkv, int B, int T, int C, int NH, bool in_trainer);
int flash_backward(int cfg, int flags, float *dqkv, float *dsum, const float *dout, const float *qkv, const float *out, const float *lse,
                   int B, int T, int C, int NH, bool in_trainer);

// Heads that the attention of flash_x2.cu leaves to the kernels behind it: a byte each of `heads`, and how many pieces of their work are taken
// (zero before the launch).
struct LeftOut { uint8_t *flagged; int *taken, heads; };

// A model as decode_position reads it: its tensors (layer-stacked, as the trainer keeps them), the keys and values so far (rows
// of 3C), the pairs that activations are handed on in, and the logits.
struct DecodeModel {
    const float *wte, *ln1w, *ln1b, *qkvw, *qkvb, *apw, *apb, *ln2w, *ln2b, *fcw, *fcb, *fpw, *fpb, *lnfw, *lnfb;
    float *qkv, *logits;
    uint2 *exchange;
    size_t layer;                 // floats from a layer's rows in qkv to the next one's
    int C, NH, L, Vp;
    float scale;
};
size_t decode_exchange(int C);
// The position's row before layer `first` (which may be L: the head alone) is x0, or x0 + x1 where that is given. `launch` counts the launches with one
// exchange: another one each time.
int decode_position(const DecodeModel &m, const float *x0, const float *x1, int first, int pos, unsigned launch, cudaStream_t st);

}  // namespace bmb

// ---- device helpers ---------------------------------------------------------
#ifdef __CUDACC__
namespace bmb {
// A launch that may start when the blocks of the one before it in the stream have all said so (let_successor_start) or ended; it
// waits for that one's end itself (wait_for_predecessor) before it reads what that wrote.  Its set-up and its launch then lie
// beside the end of the one before.
__device__ __forceinline__ void let_successor_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P, typename... A>
int launch(bool in_chain, void (*kernel)(P...), dim3 grid, dim3 threads, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = in_chain ? 1 : 0;
    BMB_CUDA(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
    count_launch();
    return BMB_OK;
}
template <typename... P, typename... A>
int launch_in_chain(void (*kernel)(P...), dim3 grid, dim3 threads, size_t smem, cudaStream_t st, A... args) {
    return launch(true, kernel, grid, threads, smem, st, args...);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Block-wide sum / max with the result in every thread.  `red` is a shared
// array of at least 32 floats; two barriers per call, safe to call repeatedly
// with the same array.
template <bool IS_MAX>
__device__ __forceinline__ float block_reduce(float v, float *red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    v = IS_MAX ? warp_max(v) : warp_sum(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    v = (lane < nw) ? red[lane] : (IS_MAX ? -3.402823466e38f : 0.0f);
    v = IS_MAX ? warp_max(v) : warp_sum(v);
    return v;
}
// tanh-approximation GELU with the accurate tanhf (src/nn.cu:118-127).
__device__ __forceinline__ float gelu_tanh(float x) {
    const float s = 0.7978845608028654f;
    return 0.5f * x * (1.0f + tanhf(s * (x + 0.044715f * x * x * x)));
}
// The same form with the hardware's approximate tanh (one special-function instruction; absolute error of tanh about
// 2^-11, i.e. of the order of a TF32 rounding of the result): for an activation that is rounded to TF32 anyway.
__device__ __forceinline__ float gelu_tanh_fast(float x) {
    const float u = 0.7978845608028654f * fmaf(0.044715f * x * x, x, x);
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
    const float hx = 0.5f * x;
    return fmaf(hx, t, hx);
}
// Round to nearest TF32 (ties away), result as an fp32 bit pattern whose low
// 13 mantissa bits are zero.
__device__ __forceinline__ float round_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}
// The same rounding with two integer instructions instead of a conversion (which shares the
// special-function unit with exp): add half a TF32 ulp to the magnitude, clear the low 13 bits.
// For finite values and infinities the result equals cvt.rna.tf32.f32.
__device__ __forceinline__ float round_tf32_alu(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}
// For a value that only the tensor core will read: kind::tf32 ignores the low 13 bits of an operand,
// so adding half a TF32 ulp is all it takes to turn that truncation into rounding to nearest.
__device__ __forceinline__ float round_tf32_for_mma(float x) { return __uint_as_float(__float_as_uint(x) + 0x1000u); }
}  // namespace bmb
#endif
