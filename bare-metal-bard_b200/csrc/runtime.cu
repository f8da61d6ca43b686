// Library-wide state: last-error text, per-thread stream, per-device scratch,
// the math-mode switch and the launch counter.
#include "common.cuh"
#include <atomic>
#include <mutex>
#include <cstring>
#include <cstdlib>

namespace bmb {

static thread_local char g_err[512] = "";
static thread_local cudaStream_t g_stream = 0;
static std::atomic<long long> g_launches{0};
static std::atomic<int> g_math{-1};

int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    if (getenv("BMB_VERBOSE")) fprintf(stderr, "bmb: error %d: %s\n", code, g_err);
    return code;
}

cudaStream_t cur_stream() { return g_stream; }

static thread_local bool g_emit_rounded = false;
bool emit_rounded() { return g_emit_rounded; }
void set_emit_rounded(bool on) { g_emit_rounded = on; }

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launches_total() { return g_launches.load(std::memory_order_relaxed); }

int current_device() {
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

int sm_count() {
    static int cache[64];
    static std::once_flag once;
    std::call_once(once, [] { for (int &c : cache) c = 0; });
    const int d = current_device();
    if (d < 0 || d >= 64) return 148;
    if (cache[d] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || n <= 0) n = 148;
        cache[d] = n;
    }
    return cache[d];
}

struct Scratch { void *p = nullptr; size_t cap = 0; };
static Scratch g_scratch[64][SCR_SLOTS];
static std::mutex g_scratch_mu;
static std::atomic<unsigned long long> g_scratch_gen[64];

unsigned long long scratch_generation() {
    const int d = current_device();
    return (d < 0 || d >= 64) ? 0ULL : g_scratch_gen[d].load(std::memory_order_relaxed);
}

static thread_local unsigned g_slots_taken = 0;
unsigned scratch_slots_taken() {
    const unsigned was = g_slots_taken;
    g_slots_taken = 0;
    return was;
}

void *device_scratch(ScratchSlot slot, size_t bytes) {
    const int d = current_device();
    if (d < 0 || d >= 64) { fail(BMB_E_ARG, "device index %d out of range", d); return nullptr; }
    g_slots_taken |= 1u << slot;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    Scratch &s = g_scratch[d][slot];
    if (s.cap >= bytes && s.p) return s.p;
    // Growing: earlier work on this device may still read the old block.  Anything that has
    // remembered the old address (a captured CUDA graph) learns of the move from the generation count.
    if (s.p) { cudaDeviceSynchronize(); cudaFree(s.p); s.p = nullptr; s.cap = 0; }
    g_scratch_gen[d].fetch_add(1, std::memory_order_relaxed);
    size_t want = bytes < (1u << 20) ? (1u << 20) : bytes;
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, want);
    if (e != cudaSuccess) { fail(BMB_E_CUDA, "scratch cudaMalloc(%zu) -> %s", want, cudaGetErrorString(e)); return nullptr; }
    s.p = p; s.cap = want;
    return p;
}

// The end of a scratch slot's last use.  A caller about to overwrite a slot first makes its stream wait for that use, so
// that two streams of one device take turns instead of racing.  Always, whatever the stream's handle: cudaStreamPerThread
// is one handle for a stream of each thread, and a destroyed stream's handle may come back for another (behind the same
// stream's own work the wait costs the device nothing).
// (Not while a stream is being captured: the captured launches carry their own order, and an event recorded inside a
// capture cannot be waited for outside it.)
struct SlotUse { cudaEvent_t done = nullptr; bool valid = false; };
static SlotUse g_slot_use[64][SCR_SLOTS];

static bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) { cudaGetLastError(); return false; }
    return cs != cudaStreamCaptureStatusNone;
}

int scratch_acquire(ScratchSlot slot, cudaStream_t st) {
    const int d = current_device();
    if (d < 0 || d >= 64 || capturing(st)) return BMB_OK;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    SlotUse &u = g_slot_use[d][slot];
    if (u.valid) BMB_CUDA(cudaStreamWaitEvent(st, u.done, 0));
    return BMB_OK;
}

int scratch_release(ScratchSlot slot, cudaStream_t st) {
    const int d = current_device();
    if (d < 0 || d >= 64 || capturing(st)) return BMB_OK;
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    SlotUse &u = g_slot_use[d][slot];
    if (!u.done) BMB_CUDA(cudaEventCreateWithFlags(&u.done, cudaEventDisableTiming));
    BMB_CUDA(cudaEventRecord(u.done, st));
    u.valid = true;
    return BMB_OK;
}

// ---- the block of split fp32 products ----
static int g_split_keepers[64];
static unsigned long long g_split_gen[64];

// While another stream is being captured in the global mode, this thread's allocations would be refused and end that capture.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

static bool split_scratch_drop(int d) {
    Scratch &s = g_scratch[d][SCR_SPLIT];
    if (!s.p) return true;
    RelaxedCapture relaxed;
    const SlotUse &u = g_slot_use[d][SCR_SPLIT];             // (written under split_mutex(), as everything here)
    if ((u.valid && cudaEventSynchronize(u.done) != cudaSuccess) || cudaFree(s.p) != cudaSuccess) { cudaGetLastError(); return false; }
    s = Scratch();
    ++g_split_gen[d];
    return true;
}

void *split_scratch(size_t bytes, cudaStream_t st) {
    const int d = current_device();
    if (d < 0 || d >= 64) return nullptr;
    g_slots_taken |= 1u << SCR_SPLIT;
    Scratch &s = g_scratch[d][SCR_SPLIT];
    if (s.p && s.cap >= bytes) return s.p;
    if (capturing(st) || !split_scratch_drop(d)) return nullptr;
    RelaxedCapture relaxed;
    const size_t want = bytes < (1u << 20) ? (1u << 20) : bytes;
    void *p = nullptr;
    if (cudaMalloc(&p, want) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    s.p = p; s.cap = want;
    ++g_split_gen[d];
    return p;
}

void split_scratch_give_back(size_t above) {
    const int d = current_device();
    if (d < 0 || d >= 64 || g_split_keepers[d] > 0 || g_scratch[d][SCR_SPLIT].cap <= above) return;
    (void)split_scratch_drop(d);
}

unsigned long long split_scratch_generation() {
    const int d = current_device();
    return (d < 0 || d >= 64) ? 0ULL : g_split_gen[d];
}

// ---- blocks for the length of a call ----
namespace {
struct CallBlock {
    void *p = nullptr;
    size_t cap = 0;
    cudaEvent_t done = nullptr;      // behind its last use, which `user`'s stream had
    const void *user = nullptr;
    bool taken = false;              // a call is making its launches
    unsigned long long when = 0;
};
struct CallBlocks {
    CallBlock of[8];
    size_t total = 0;
    unsigned long long uses = 0;
};
std::mutex g_call_mu;
CallBlocks g_call_blocks[64];

bool drop_block(CallBlocks &all, CallBlock &b) {
    if (b.p && (cudaEventSynchronize(b.done) != cudaSuccess || cudaFree(b.p) != cudaSuccess)) { cudaGetLastError(); return false; }
    all.total -= b.cap;
    b.p = nullptr;
    b.cap = 0;
    return true;
}
}  // namespace

void *call_scratch(size_t bytes, cudaStream_t st) {
    const int d = current_device();
    if (d < 0 || d >= 64) return nullptr;
    static thread_local char thread;         // (cudaStreamPerThread is one handle for a stream of each thread)
    const void *user = st == cudaStreamPerThread ? (const void *)&thread : (const void *)st;
    RelaxedCapture relaxed;
    std::lock_guard<std::mutex> lk(g_call_mu);
    CallBlocks &all = g_call_blocks[d];
    // this stream's last block, or one that nobody uses any more, or a new one, or the one that has been in use for longest
    CallBlock *mine = nullptr, *idle = nullptr, *oldest = nullptr, *empty = nullptr;
    for (CallBlock &b : all.of) {
        if (b.taken) continue;
        if (!b.p) { empty = &b; continue; }
        if (b.cap < bytes) continue;
        if (b.user == user) { if (!mine || b.cap < mine->cap) mine = &b; }
        else if (!oldest || b.when < oldest->when) oldest = &b;
    }
    if (!mine && oldest) {
        if (cudaEventQuery(oldest->done) == cudaSuccess) idle = oldest;
        else cudaGetLastError();
    }
    CallBlock *use = mine ? mine : idle;
    if (!use && !(oldest && (!empty || all.total + bytes > CALL_SCRATCH_KEPT))) {
        for (CallBlock &b : all.of) {                        // (none is large enough: smaller ones make room)
            if (empty && all.total + bytes <= CALL_SCRATCH_KEPT) break;
            if (b.p && !b.taken && drop_block(all, b)) empty = &b;
        }
        if (!empty) return nullptr;
        if (!empty->done && cudaEventCreateWithFlags(&empty->done, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        const size_t want = bytes < (1u << 20) ? (1u << 20) : bytes;
        if (cudaMalloc(&empty->p, want) != cudaSuccess) { cudaGetLastError(); empty->p = nullptr; return nullptr; }
        empty->cap = want;
        all.total += want;
        use = empty;
    } else {
        if (!use) use = oldest;
        // (also behind the same stream's work: a handle may have come back for another stream)
        if (cudaStreamWaitEvent(st, use->done, 0) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    }
    use->taken = true;
    use->user = user;
    use->when = ++all.uses;
    return use->p;
}

int call_scratch_done(void *p, cudaStream_t st) {
    const int d = current_device();
    RelaxedCapture relaxed;
    std::lock_guard<std::mutex> lk(g_call_mu);
    CallBlocks &all = g_call_blocks[d];
    for (CallBlock &b : all.of)
        if (b.p == p) {
            BMB_CUDA(cudaEventRecord(b.done, st));
            b.taken = false;
            if (all.total > CALL_SCRATCH_KEPT) drop_block(all, b);
            break;
        }
    return BMB_OK;
}

void split_scratch_keep(int change) {
    const int d = current_device();
    if (d >= 0 && d < 64) g_split_keepers[d] += change;
}

}  // namespace bmb

extern "C" {

const char *bmb_last_error(void) { return bmb::g_err; }
long long bmb_launch_count(void) { return bmb::launches_total(); }
const char *bmb_version(void) { return "bmb-b200 0.1 (sm_100a)"; }

int bmb_set_stream(void *s) { bmb::g_stream = (cudaStream_t)s; return BMB_OK; }
void *bmb_get_stream(void) { return (void *)bmb::g_stream; }

int bmb_set_math_mode(int mode) {
    if (mode < BMB_MATH_FP32 || mode > BMB_MATH_BF16)
        return bmb::fail(BMB_E_ARG, "math mode %d unknown", mode);
    bmb::g_math.store(mode);
    return BMB_OK;
}

int bmb_get_math_mode(void) {
    int m = bmb::g_math.load();
    if (m < 0) {
        // Default: fp32, the reference's arithmetic; BMB_MATH=tf32|bf16 opts in.
        m = BMB_MATH_FP32;
        const char *e = getenv("BMB_MATH");
        if (e && !strcmp(e, "tf32")) m = BMB_MATH_TF32;
        if (e && !strcmp(e, "bf16")) m = BMB_MATH_BF16;
        bmb::g_math.store(m);
    }
    return m;
}

}  // extern "C"
