// api.cu -- C host layer behind the C ABI (include/mela.h).
//
// Host entry points mirror the reference MEX gateways' semantics (input
// validation order, logical/double reading, MATLAB column-major layout) and
// run every computation on the GPU: host arrays are copied in, packed,
// processed and unpacked by kernels, and copied out.  Device entry points
// are stream-ordered and never synchronise.
#include <chrono>
#include <condition_variable>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include "mela_common.cuh"
#include "mela_internal.h"
#include "mela_host.h"

namespace mela {

// ---------------------------------------------------------------- errors
static thread_local char t_err[512] = "";

void set_error(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(t_err, sizeof t_err, fmt, ap);
    va_end(ap);
}

mela_status cuda_status(cudaError_t e, const char *what)
{
    set_error("%s: %s", what, cudaGetErrorString(e));
    if (e == cudaErrorMemoryAllocation) return MELA_ERR_NOMEM;
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return MELA_ERR_NO_DEVICE;
    return MELA_ERR_CUDA;
}

__device__ u32 g_device_error;

static constexpr int kMaxDevices = 64;
static std::mutex g_dev_mu;
static u32 *g_err_addr[kMaxDevices];
static int g_sms[kMaxDevices];

static int current_device()
{
    int d = 0;
    cudaGetDevice(&d);
    return (d >= 0 && d < kMaxDevices) ? d : 0;
}

u32 *device_error_word()
{
    int d = current_device();
    std::lock_guard<std::mutex> g(g_dev_mu);
    if (!g_err_addr[d]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_device_error) == cudaSuccess) g_err_addr[d] = (u32 *)p;
    }
    return g_err_addr[d];
}

int sm_count()
{
    int d = current_device();
    std::lock_guard<std::mutex> g(g_dev_mu);
    if (!g_sms[d]) {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d);
        g_sms[d] = v > 0 ? v : 1;
    }
    return g_sms[d];
}

// ---------------------------------------------------------------- per-thread context
// One non-blocking stream per host thread and device for the host entry
// points; device buffers come from the stream-ordered pool (cached between
// calls, so repeated gateway calls do not pay cudaMalloc).
struct HostCtx {
    cudaStream_t stream[kMaxDevices] = {};
    cudaStream_t copy_in[kMaxDevices] = {};   // pipelined host products: uploads
    cudaStream_t copy_out[kMaxDevices] = {};  //   and downloads
    cudaStream_t side[kMaxDevices] = {};      // work forked off a caller's stream
    cudaStream_t capture[kMaxDevices] = {};   // origin of graph captures
};
static thread_local HostCtx t_ctx;

mela_status host_stream(cudaStream_t *s)
{
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        set_error("no CUDA device visible");
        return MELA_ERR_NO_DEVICE;
    }
    int d = current_device();
    if (!t_ctx.stream[d]) {
        MELA_CUDA_TRY(cudaStreamCreateWithFlags(&t_ctx.stream[d], cudaStreamNonBlocking));
        cudaMemPool_t pool;
        if (cudaDeviceGetDefaultMemPool(&pool, d) == cudaSuccess) {
            unsigned long long thr = ~0ull;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
        }
    }
    *s = t_ctx.stream[d];
    return MELA_OK;
}

// The calling thread's upload and download streams (created on first use).
static mela_status copy_streams(cudaStream_t *in, cudaStream_t *out)
{
    const int d = current_device();
    if (!t_ctx.copy_in[d]) MELA_CUDA_TRY(cudaStreamCreateWithFlags(&t_ctx.copy_in[d], cudaStreamNonBlocking));
    if (!t_ctx.copy_out[d]) MELA_CUDA_TRY(cudaStreamCreateWithFlags(&t_ctx.copy_out[d], cudaStreamNonBlocking));
    *in = t_ctx.copy_in[d];
    *out = t_ctx.copy_out[d];
    return MELA_OK;
}

mela_status side_stream(cudaStream_t *s)
{
    const int d = current_device();
    if (!t_ctx.side[d]) MELA_CUDA_TRY(cudaStreamCreateWithFlags(&t_ctx.side[d], cudaStreamNonBlocking));
    *s = t_ctx.side[d];
    return MELA_OK;
}

mela_status capture_stream(cudaStream_t *s)
{
    const int d = current_device();
    if (!t_ctx.capture[d]) MELA_CUDA_TRY(cudaStreamCreateWithFlags(&t_ctx.capture[d], cudaStreamNonBlocking));
    *s = t_ctx.capture[d];
    return MELA_OK;
}

DevBuf::~DevBuf()
{
    if (p) cudaFreeAsync(p, s);
}

mela_status DevBuf::alloc(size_t bytes, cudaStream_t st)
{
    s = st;
    if (bytes == 0) bytes = 16;
    cudaError_t e = cudaMallocAsync(&p, bytes, st);
    if (e != cudaSuccess) {
        p = nullptr;
        return cuda_status(e, "cudaMallocAsync");
    }
    return MELA_OK;
}

// The calling thread's page-locked words per device: what a call reads back
// lands here, so that the read is stream-ordered and one synchronisation ends
// the call.
namespace {
constexpr size_t kSmallBytes = (size_t)256 << 10;
struct Readback {
    u32 err;
    long long value;
    alignas(64) unsigned char small[kSmallBytes];
    alignas(64) unsigned char in[24 << 10];
};
// Sets not in use, kept for other threads: short-lived threads then neither
// allocate (page-locking 280 KB takes 0.1 ms) nor free (which may wait for the
// device).  At most kSpareReadbacks.
constexpr size_t kSpareReadbacks = 32;
std::mutex g_readback_mu;
std::vector<Readback *> *g_readback_spare = nullptr;
Readback *readback_new()
{
    {
        std::lock_guard<std::mutex> g(g_readback_mu);
        if (g_readback_spare && !g_readback_spare->empty()) {
            Readback *r = g_readback_spare->back();
            g_readback_spare->pop_back();
            return r;
        }
    }
    Readback *r = nullptr;
    if (cudaHostAlloc((void **)&r, sizeof(Readback), cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return r;
}
void readback_spare(Readback *r)
{
    if (!r) return;
    {
        std::lock_guard<std::mutex> g(g_readback_mu);
        if (!g_readback_spare) g_readback_spare = new std::vector<Readback *>();
        if (g_readback_spare->size() < kSpareReadbacks) {
            g_readback_spare->push_back(r);
            return;
        }
    }
    cudaFreeHost(r);
}
struct Readbacks {
    Readback *dev[kMaxDevices] = {};
    ~Readbacks()  // given back when the thread ends
    {
        for (Readback *r : dev) readback_spare(r);
    }
};
thread_local Readbacks t_readback;
Readback *readback()
{
    Readback *&r = t_readback.dev[current_device()];
    if (!r) r = readback_new();
    return r;
}
}  // namespace

// Waits for s; r holds the device error word by then (null: ask for it).
static mela_status finish_words(cudaStream_t s, const Readback *r)
{
    MELA_CUDA_TRY(cudaStreamSynchronize(s));
    if (r && r->err == 0) return MELA_OK;
    u32 flags = 0;
    if (mela_device_error_flags(&flags, 1) == MELA_OK && (flags & kErrWaitTimeout)) {
        set_error("a bounded device-side wait timed out");
        return MELA_ERR_TIMEOUT;
    }
    return MELA_OK;
}

mela_status finish(cudaStream_t s)
{
    Readback *r = readback();
    const u32 *word = device_error_word();
    const bool queued = r && word && cudaMemcpyAsync(&r->err, word, sizeof r->err, cudaMemcpyDeviceToHost, s) == cudaSuccess;
    if (!queued) cudaGetLastError();
    return finish_words(s, queued ? r : nullptr);
}

bool posted(Posted *to)
{
    Readback *r = readback();
    const u32 *word = device_error_word();
    if (!r || !word) return false;
    *to = Posted{&r->value, &r->err, word, r->small, r->in, kSmallBytes};
    return true;
}

mela_status finish_posted(cudaStream_t s) { return finish_words(s, readback()); }

void *posted_take()
{
    Readback *&slot = t_readback.dev[current_device()], *r = slot;
    slot = nullptr;
    return r;
}

void posted_give(void *words)
{
    Readback *&slot = t_readback.dev[current_device()];
    readback_spare(slot);
    slot = (Readback *)words;
}

mela_status read_value(long long *value, const long long *d, cudaStream_t s, bool last)
{
    Readback *r = readback();
    MELA_CUDA_TRY(cudaMemcpyAsync(r ? &r->value : value, d, sizeof *value, cudaMemcpyDeviceToHost, s));
    if (last) {
        mela_status st = finish(s);
        if (st != MELA_OK) return st;
    } else {
        MELA_CUDA_TRY(cudaStreamSynchronize(s));
    }
    if (r) *value = r->value;
    return MELA_OK;
}

// ---------------------------------------------------------------- products
i64 even_words(i64 bits)
{
    i64 w = words_of(bits);
    return (w + 1) & ~1LL;
}

static i64 round_up(i64 x, i64 a) { return (x + a - 1) / a * a; }

// workspace layout for each variant
struct GemmPlan {
    int variant;          // base variant
    int tc_tile;          // tile choice: tensor cores 1 single CTAs / 2 CTA pairs; M4RI 1 = 8 warps
    i64 ldbt;             // packed Bt row pitch (words)
    size_t bt_bytes;      // packed Bt
    i64 mp, np, kp;       // padded byte-operand shape (tensor cores)
    size_t a8_bytes, b8_bytes;
    size_t total;
};

// Workspace layout of a concrete variant argument (AUTO already resolved).
static GemmPlan plan_gemm(int32_t variant, i64 m, i64 k, i64 n)
{
    GemmPlan p{};
    Tuning t{};
    if (!decode_gemm_variant(variant, &t) || t.base == MELA_GEMM_AUTO) t.base = MELA_GEMM_PLAIN;
    p.variant = t.base;
    p.tc_tile = t.tc_tile;
    p.ldbt = even_words(k);
    if (p.variant == MELA_GEMM_PLAIN) p.bt_bytes = (size_t)n * p.ldbt * 8;
    if (p.variant == MELA_GEMM_TC) {
        p.mp = round_up(m, 256);  // 256-row tiles for CTA pairs
        p.np = round_up(n, 256);
        p.kp = round_up(k, 128);  // bytes = values
        p.a8_bytes = (size_t)p.mp * p.kp;
        p.b8_bytes = (size_t)p.np * p.kp;
    }
    if (p.variant == MELA_GEMM_TC_FP4) {
        p.mp = round_up(m, 256);
        p.np = round_up(n, 256);
        p.kp = round_up(k, 256) / 2;  // bytes, two values each
        p.a8_bytes = (size_t)p.mp * p.kp;
        p.b8_bytes = (size_t)p.np * p.kp;
    }
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    p.total = al(p.bt_bytes) + al(p.a8_bytes) + al(p.b8_bytes);
    return p;
}

struct GemmBufs {
    u64 *Bt;
    unsigned char *A8, *B8;
};

static GemmBufs carve(const GemmPlan &p, void *ws)
{
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    unsigned char *w = (unsigned char *)ws;
    GemmBufs b;
    b.Bt = (u64 *)w;
    b.A8 = w + al(p.bt_bytes);
    b.B8 = b.A8 + al(p.a8_bytes);
    return b;
}

static mela_status check_ws(const GemmPlan &p, void *ws, size_t ws_bytes)
{
    if (ws_bytes < p.total || (p.total && !ws)) {
        set_error("mela_dev_matmul: workspace of %zu bytes needed, %zu given", p.total, ws_bytes);
        return MELA_ERR_INVALID;
    }
    return MELA_OK;
}

// A product's form.  AUTO only takes one that the call's buffers allow: the
// tensor-core forms read their expanded operands with 16-byte accesses, the
// Four-Russians form needs no workspace at all.
static int32_t form_of(int32_t variant, const u64 *A, i64 lda, i64 m, i64 k, i64 n, const void *ws, cudaStream_t s)
{
    const int32_t v = resolve_gemm_variant(variant, A, lda, m, k, n, s);
    if (v == variant || ((uintptr_t)ws & 15) == 0) return v;
    double density;
    mela_dispatch_last(&density);
    return remember_variant(MELA_GEMM_M4RI, density);
}

// Operand preparation: B transposed (plain and tensor-core forms) and the
// 0/1 byte expansion of A and Bt (tensor-core form).
mela_status gemm_prepare(int variant, const u64 *A, i64 lda, const u64 *B, i64 ldb, i64 m, i64 k,
                         i64 n, void *ws, size_t ws_bytes, cudaStream_t s)
{
    if (m == 0 || n == 0 || k == 0) return MELA_OK;
    variant = form_of(variant, A, lda, m, k, n, ws, s);
    GemmPlan p = plan_gemm(variant, m, k, n);
    mela_status st = check_ws(p, ws, ws_bytes);
    if (st != MELA_OK) return st;
    GemmBufs b = carve(p, ws);
    if (p.variant == MELA_GEMM_TC_FP4 && k >= (1LL << 23)) {
        set_error("fp4 tensor-core product needs k < 2^23 (exact f32 sums)");
        return MELA_ERR_UNSUPPORTED;
    }
    if (p.variant == MELA_GEMM_PLAIN) {
        if ((st = launch_transpose(B, ldb, k, n, b.Bt, p.ldbt, s)) != MELA_OK) return st;
        if (p.ldbt > words_of(k)) {
            // the pad word of each Bt row must read as zero
            MELA_CUDA_TRY(cudaMemset2DAsync(b.Bt + words_of(k), (size_t)p.ldbt * 8, 0, 8, (size_t)n, s));
        }
    }
    if ((p.variant == MELA_GEMM_TC || p.variant == MELA_GEMM_TC_FP4) && ((uintptr_t)ws & 15)) {
        set_error("mela_dev_matmul: the tensor-core forms need a 16-byte aligned workspace");
        return MELA_ERR_INVALID;
    }
    if (p.variant == MELA_GEMM_TC || p.variant == MELA_GEMM_TC_FP4)
        return launch_expand(A, lda, m, p.mp, b.A8, B, ldb, n, p.np, b.B8, k, p.kp, p.variant == MELA_GEMM_TC_FP4, s);
    return MELA_OK;
}

// The product kernel itself on prepared operands.
mela_status gemm_run(int variant, const u64 *A, i64 lda, const u64 *B, i64 ldb, u64 *C, i64 ldc,
                     i64 m, i64 k, i64 n, void *ws, size_t ws_bytes, cudaStream_t s)
{
    if (m == 0 || n == 0) return MELA_OK;
    if (k == 0) {
        MELA_CUDA_TRY(cudaMemset2DAsync(C, (size_t)ldc * 8, 0, (size_t)words_of(n) * 8, (size_t)m, s));
        return MELA_OK;
    }
    variant = form_of(variant, A, lda, m, k, n, ws, s);
    GemmPlan p = plan_gemm(variant, m, k, n);
    mela_status st = check_ws(p, ws, ws_bytes);
    if (st != MELA_OK) return st;
    GemmBufs b = carve(p, ws);
    switch (p.variant) {
    case MELA_GEMM_PLAIN: return launch_gemm_plain(A, lda, b.Bt, p.ldbt, C, ldc, m, k, n, s);
    case MELA_GEMM_TC: return launch_gemm_tc(b.A8, b.B8, p.mp, p.np, p.kp, C, ldc, m, n, s, false, p.tc_tile);
    case MELA_GEMM_TC_FP4:
        if (k >= (1LL << 23)) {
            set_error("fp4 tensor-core product needs k < 2^23 (exact f32 sums)");
            return MELA_ERR_UNSUPPORTED;
        }
        return launch_gemm_tc(b.A8, b.B8, p.mp, p.np, p.kp, C, ldc, m, n, s, true, p.tc_tile);
    case MELA_GEMM_M4RI: return launch_gemm_m4ri(A, lda, B, ldb, C, ldc, m, k, n, s, p.tc_tile);
    default:
        set_error("unknown product variant %d", p.variant);
        return MELA_ERR_INVALID;
    }
}

mela_status gemm_device(int variant, const u64 *A, i64 lda, const u64 *B, i64 ldb, u64 *C, i64 ldc,
                        i64 m, i64 k, i64 n, void *ws, size_t ws_bytes, cudaStream_t s)
{
    if (m > 0 && n > 0 && k > 0) {
        const bool chosen = MELA_VARIANT_BASE(variant) == MELA_GEMM_AUTO;
        variant = form_of(variant, A, lda, m, k, n, ws, s);
        if (chosen && ((uintptr_t)ws & 15) == 0 &&
            !(packed_apart(A, lda, m, k, C, ldc, m, n) && packed_apart(B, ldb, k, n, C, ldc, m, n))) {
            // a result over an operand: the forms that expand both operands
            // before they write are right at every size
            double density;
            mela_dispatch_last(&density);
            variant = remember_variant(k < (1LL << 23) ? MELA_GEMM_TC_FP4 : MELA_GEMM_TC, density);
        }
        const GemmPlan p = plan_gemm(variant, m, k, n);
        const bool fp4 = p.variant == MELA_GEMM_TC_FP4;
        if ((fp4 || p.variant == MELA_GEMM_TC) && k < (1LL << 23) &&
            gemm_strassen_fits(A, lda, B, ldb, C, ldc, m, k, n, fp4, p.tc_tile)) {
            if (mela_status st = check_ws(p, ws, ws_bytes); st != MELA_OK) return st;
            return launch_gemm_strassen(A, lda, B, ldb, C, ldc, m, k, n, ws, ws_bytes, fp4, s);
        }
    }
    mela_status st = gemm_prepare(variant, A, lda, B, ldb, m, k, n, ws, ws_bytes, s);
    if (st != MELA_OK) return st;
    return gemm_run(variant, A, lda, B, ldb, C, ldc, m, k, n, ws, ws_bytes, s);
}

size_t gemm_workspace(int variant, i64 m, i64 k, i64 n)
{
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    if (MELA_VARIANT_BASE(variant) != MELA_GEMM_AUTO) return plan_gemm(variant, m, k, n).total;
    // AUTO decides on the data: room for any configuration it may pick
    size_t most = plan_gemm(fixed_gemm_variant(m, k, n), m, k, n).total;
    for (int c = 0; c < config_count(MELA_OP_MATMUL); ++c) {
        const size_t t = plan_gemm(config_variant(MELA_OP_MATMUL, c), m, k, n).total;
        if (t > most) most = t;
    }
    return most;
}

// ---------------------------------------------------------------- host-matrix helpers
namespace {
// Host threads that copy a caller's (pageable) array into page-locked
// staging memory in parallel: one copy thread saturates neither the host's
// memory system nor the PCIe link.  Created on first use, never torn down.
class CopyPool {
public:
    static CopyPool &get()
    {
        static CopyPool *p = new CopyPool();
        return *p;
    }
    // dst[0, bytes) = src[0, bytes), split over the pool and the caller;
    // to_device: dst is about to be read by a DMA.
    void copy(void *dst, const void *src, size_t bytes, bool to_device)
    {
        const int parts = (int)workers_.size() + 1;
        if (bytes < ((size_t)1 << 18) || parts == 1) {
            copy_part((char *)dst, (const char *)src, bytes, to_device);
            return;
        }
        std::lock_guard<std::mutex> one_job(call_mu_);  // callers on other threads queue here
        std::unique_lock<std::mutex> lk(mu_);
        job_dst_ = (char *)dst;
        job_src_ = (const char *)src;
        job_bytes_ = bytes;
        job_parts_ = parts;
        job_stream_ = to_device;
        pending_ = parts - 1;
        ++gen_;
        lk.unlock();
        cv_.notify_all();
        run_part(0);
        lk.lock();
        done_.wait(lk, [&] { return pending_ == 0; });
    }

private:
    CopyPool()
    {
        unsigned hw = std::thread::hardware_concurrency();
        int n = hw >= 4 ? (int)(hw / 2) : 1;
        if (n > 8) n = 8;
        for (int i = 1; i < n; ++i) workers_.emplace_back([this, i] { loop(i); });
        for (auto &t : workers_) t.detach();
    }
    void run_part(int i)
    {
        const size_t per = (job_bytes_ / job_parts_ + 63) & ~(size_t)63;
        const size_t a = per * (size_t)i, b = a + per < job_bytes_ ? a + per : job_bytes_;
        if (a < b) copy_part(job_dst_ + a, job_src_ + a, b - a, job_stream_);
    }
    // A page-locked slot is filled with streaming stores: a DMA that finds the
    // slot's lines modified in the cores' caches runs at 7 GB/s for 8 MB instead
    // of 52 GB/s, and the fill itself takes 154 us instead of 262.
    static void copy_part(char *dst, const char *src, size_t bytes, bool stream)
    {
#if defined(__x86_64__)
        if (stream && ((uintptr_t)dst & 15) == 0) {
            size_t i = 0;
            for (; i + 64 <= bytes; i += 64) {
                const __m128i a = _mm_loadu_si128((const __m128i *)(src + i));
                const __m128i b = _mm_loadu_si128((const __m128i *)(src + i + 16));
                const __m128i c = _mm_loadu_si128((const __m128i *)(src + i + 32));
                const __m128i d = _mm_loadu_si128((const __m128i *)(src + i + 48));
                _mm_stream_si128((__m128i *)(dst + i), a);
                _mm_stream_si128((__m128i *)(dst + i + 16), b);
                _mm_stream_si128((__m128i *)(dst + i + 32), c);
                _mm_stream_si128((__m128i *)(dst + i + 48), d);
            }
            std::memcpy(dst + i, src + i, bytes - i);
            _mm_sfence();
            return;
        }
#endif
        (void)stream;
        std::memcpy(dst, src, bytes);
    }
    void loop(int i)
    {
        unsigned long long seen = 0;
        for (;;) {
            std::unique_lock<std::mutex> lk(mu_);
            cv_.wait(lk, [&] { return gen_ != seen; });
            seen = gen_;
            lk.unlock();
            run_part(i);
            lk.lock();
            if (--pending_ == 0) done_.notify_one();
        }
    }
    std::vector<std::thread> workers_;
    std::mutex call_mu_, mu_;
    std::condition_variable cv_, done_;
    unsigned long long gen_ = 0;
    int pending_ = 0, job_parts_ = 1;
    bool job_stream_ = false;
    char *job_dst_ = nullptr;
    const char *job_src_ = nullptr;
    size_t job_bytes_ = 0;
};

// Page-locked staging slots, taken in turn across calls, uploads and
// downloads: a slot is refilled once the copy that used it has completed
// (its event, which any thread can wait for).
constexpr int kStageSlots = 3;
constexpr size_t kStageSmall = (size_t)1 << 20, kStageBytes = (size_t)8 << 20;  // the two sizes of a slot
struct Staging {
    void *slot[kStageSlots] = {};
    cudaEvent_t read[kStageSlots] = {};  // the copy from or into the slot is done
    cudaEvent_t fence = nullptr;         // the device staging buffer is allocated
    int next = 0;                        // the next slot
    size_t cap = 0;                      // bytes of a slot
};
// The sets of a device (events belong to it), shared by the host threads: a
// call takes one for an upload or a download, so there are no more of them than
// calls have ever been copying at once, at most kStageSets (384 MB); a copy
// that finds none left goes by the driver.  The set used last is taken first.
constexpr int kStageSets = 16;
struct StagePool {
    std::vector<Staging *> spare;
    int made = 0;
    bool asked[2] = {};   // a download has asked for slots of that size
    bool failed = false;  // page-locked memory has run out
};
std::mutex g_stage_mu;
StagePool *g_stage[kMaxDevices];

// Slots of at least `bytes` for S, whose copies have ended.
bool staging_grow(Staging &S, size_t bytes)
{
    for (int i = 0; i < kStageSlots; ++i) {
        if (S.read[i]) cudaEventSynchronize(S.read[i]);
        if (S.slot[i]) cudaFreeHost(S.slot[i]);
        S.slot[i] = nullptr;
    }
    S.cap = 0;
    bool ok = S.fence || cudaEventCreateWithFlags(&S.fence, cudaEventDisableTiming) == cudaSuccess;
    for (int i = 0; ok && i < kStageSlots; ++i)
        ok = (S.read[i] || cudaEventCreateWithFlags(&S.read[i], cudaEventDisableTiming) == cudaSuccess) &&
             cudaHostAlloc(&S.slot[i], bytes, cudaHostAllocPortable) == cudaSuccess;
    if (ok) {
        S.cap = bytes;
        return true;
    }
    cudaGetLastError();
    for (int i = 0; i < kStageSlots; ++i) {
        if (S.slot[i]) cudaFreeHost(S.slot[i]);
        S.slot[i] = nullptr;
    }
    return false;
}

// A set for the life of this object; S is null where there is none.
class StagingLease {
public:
    // Pieces of up to `want` bytes.  An upload always gets them; a download,
    // which can also go by the driver or in smaller pieces, does not make the
    // first call of a process pay for new slots (page-locking takes 0.5 ms a
    // MB): they are made when it asks for the second time.
    StagingLease(size_t want, bool download) : dev_(current_device())
    {
        const int size = want > kStageSmall;
        const size_t bytes = size ? kStageBytes : kStageSmall;
        bool grow = true;
        {
            std::lock_guard<std::mutex> g(g_stage_mu);
            StagePool *&P = g_stage[dev_];
            if (!P) P = new StagePool();
            if (download) {
                grow = P->asked[size];
                P->asked[size] = true;
            }
            if (P->failed) grow = false;
            if (!P->spare.empty()) {
                size_t i = P->spare.size() - 1;
                for (size_t j = i + 1; j-- > 0;)
                    if (P->spare[j]->cap >= bytes) {
                        i = j;
                        break;
                    }
                S = P->spare[i];
                P->spare.erase(P->spare.begin() + (long)i);
            } else if (grow && P->made < kStageSets) {
                S = new Staging();
                ++P->made;
            }
        }
        if (!S || S->cap >= bytes) return;
        if (!grow && (S->cap == 0 || !download)) {
            give_back();
            return;
        }
        if (grow && !staging_grow(*S, bytes)) {
            {
                std::lock_guard<std::mutex> g(g_stage_mu);
                g_stage[dev_]->failed = true;
            }
            give_back();
        }
    }
    ~StagingLease() { give_back(); }
    StagingLease(const StagingLease &) = delete;
    StagingLease &operator=(const StagingLease &) = delete;
    Staging *S = nullptr;

private:
    void give_back()
    {
        if (!S) return;
        std::lock_guard<std::mutex> g(g_stage_mu);
        g_stage[dev_]->spare.push_back(S);
        S = nullptr;
    }
    int dev_;
};
thread_local mela_upload_stats t_upload_stats;

double now_us()
{
    return std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

}  // namespace

// Column blocks of the MATLAB array go through the page-locked slots: the
// host copy of block b+1 (parallel memcpy) overlaps the upload of block b on
// the upload stream, and each block is packed on s as soon as it has landed
// (blocks are whole packed words: multiples of 64 columns).
static mela_status upload_and_pack_blocks(const mela_host_matrix *M, u64 *dP, i64 ld, cudaStream_t s,
                                          DevBuf &staging, i64 cols_per_block, Staging &S)
{
    const i64 m = M->rows, n = M->cols;
    const size_t esz = M->kind == MELA_KIND_DOUBLE ? 8 : 1;
    mela_status st = staging.alloc((size_t)m * (size_t)n * esz, s);
    if (st != MELA_OK) return st;
    cudaStream_t sin = nullptr, sout = nullptr;
    if ((st = copy_streams(&sin, &sout)) != MELA_OK) return st;
    // the device staging buffer comes from s's pool: uploads wait for it
    MELA_CUDA_TRY(cudaEventRecord(S.fence, s));
    MELA_CUDA_TRY(cudaStreamWaitEvent(sin, S.fence, 0));
    const char *src = (const char *)M->data;
    char *dst = (char *)staging.p;
    for (i64 j0 = 0; j0 < n; j0 += cols_per_block) {
        const int slot = S.next;
        S.next = (slot + 1) % kStageSlots;
        const i64 nc = n - j0 < cols_per_block ? n - j0 : cols_per_block;
        const size_t off = (size_t)j0 * (size_t)m * esz, bytes = (size_t)nc * (size_t)m * esz;
        const double t0 = now_us();
        MELA_CUDA_TRY(cudaEventSynchronize(S.read[slot]));  // the slot's previous upload is done
        const double t1 = now_us();
        CopyPool::get().copy(S.slot[slot], src + off, bytes, true);
        t_upload_stats.slot_wait_us += t1 - t0;
        t_upload_stats.host_copy_us += now_us() - t1;
        t_upload_stats.blocked_bytes += (int64_t)bytes;
        t_upload_stats.blocks += 1;
        MELA_CUDA_TRY(cudaMemcpyAsync(dst + off, S.slot[slot], bytes, cudaMemcpyHostToDevice, sin));
        MELA_CUDA_TRY(cudaEventRecord(S.read[slot], sin));
        MELA_CUDA_TRY(cudaStreamWaitEvent(s, S.read[slot], 0));
        // the last block also writes the row padding words
        const i64 words = j0 + nc >= n ? ld - j0 / 64 : words_of(nc);
        if ((st = launch_pack_words(M->kind, m, nc, dst + off, dP + j0 / 64, ld, words, s)) != MELA_OK)
            return st;
    }
    return MELA_OK;
}

// Device bytes into the caller's (pageable) array, ending the call on s.
// Results come down through the staging slots, the host copy of one piece
// (which also takes the array's first-touch page faults) overlapping the
// download of the next two: 9.4 MB into a fresh array took the driver's own
// pageable copy 1.2-3 ms, 0.5 MB 60 us more than this (700 x 300 x 700 149 us
// the whole call, 212).  Below 8 MiB the calling thread copies by itself: in a
// fresh array the page faults of several threads get in one another's way (whole
// calls, result of 2.2 MB: 0.37 ms, 0.78 with the copy threads, 0.51 by the
// driver; 4.5 MB 0.62, 1.24, 0.88; in an array in use 0.43 and 0.45 at 4.5 MB, at
// 16 MB 1.2 and 0.6).  Small ones land in the thread's page-locked words, so that
// the result and the error word need one wait.
mela_status download_finish(void *dst, const void *src, size_t bytes, cudaStream_t s)
{
    Readback *rb = readback();
    if (bytes <= kSmallBytes && rb) {
        MELA_CUDA_TRY(cudaMemcpyAsync(rb->small, src, bytes, cudaMemcpyDeviceToHost, s));
        const mela_status st = finish(s);
        if (st == MELA_OK) std::memcpy(dst, rb->small, bytes);
        return st;
    }
    const bool alone = bytes < ((size_t)8 << 20);
    const size_t least = (size_t)(alone ? 128 : 512) << 10, most = alone ? kStageSmall : kStageBytes;
    size_t piece = (bytes / 4 + 0xffff) & ~(size_t)0xffff;
    if (piece < least) piece = least;
    if (piece > most) piece = most;
    StagingLease lease(piece, true);
    if (!lease.S) {
        MELA_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
        return finish(s);
    }
    Staging &S = *lease.S;
    if (piece > S.cap) piece = S.cap;
    const size_t pieces = (bytes + piece - 1) / piece;
    const int first = S.next;
    size_t issued = 0;
    for (size_t c = 0; c < pieces; ++c) {
        for (; issued < pieces && issued < c + kStageSlots; ++issued) {
            const int slot = (int)((first + issued) % kStageSlots);
            const size_t off = issued * piece, len = bytes - off < piece ? bytes - off : piece;
            MELA_CUDA_TRY(cudaEventSynchronize(S.read[slot]));
            MELA_CUDA_TRY(cudaMemcpyAsync(S.slot[slot], (const char *)src + off, len, cudaMemcpyDeviceToHost, s));
            MELA_CUDA_TRY(cudaEventRecord(S.read[slot], s));
            S.next = (slot + 1) % kStageSlots;
        }
        const int slot = (int)((first + c) % kStageSlots);
        const size_t off = c * piece, len = bytes - off < piece ? bytes - off : piece;
        MELA_CUDA_TRY(cudaEventSynchronize(S.read[slot]));
        if (alone)
            std::memcpy((char *)dst + off, S.slot[slot], len);
        else
            CopyPool::get().copy((char *)dst + off, S.slot[slot], len, false);
    }
    return finish(s);
}

mela_status upload_and_pack(const mela_host_matrix *M, u64 *dP, i64 ld, cudaStream_t s,
                            DevBuf &staging)
{
    const i64 m = M->rows, n = M->cols;
    if (m == 0 || n == 0) {
        if (m > 0) MELA_CUDA_TRY(cudaMemsetAsync(dP, 0, (size_t)m * ld * 8, s));
        return MELA_OK;
    }
    const size_t esz = M->kind == MELA_KIND_DOUBLE ? 8 : 1;
    const size_t bytes = (size_t)m * (size_t)n * esz;
    // blocks of whole packed words: a quarter of the array, so that the host
    // copies overlap the uploads, but at least 1 MiB and at most a staging slot
    const size_t col_bytes = (size_t)m * esz;
    i64 cols_per_block = (i64)(kStageBytes / col_bytes) / 64 * 64;
    const size_t quarter = bytes / 4 > ((size_t)1 << 20) ? bytes / 4 : (size_t)1 << 20;
    const i64 want = ((i64)(quarter / col_bytes) + 63) / 64 * 64;
    if (want >= 64 && want < cols_per_block) cols_per_block = want;
    if (bytes >= ((size_t)2 << 20) && cols_per_block >= 64) {
        const StagingLease lease((size_t)cols_per_block * col_bytes, false);
        if (lease.S) return upload_and_pack_blocks(M, dP, ld, s, staging, cols_per_block, *lease.S);
    }
    mela_status st = staging.alloc(bytes, s);
    if (st != MELA_OK) return st;
    MELA_CUDA_TRY(cudaMemcpyAsync(staging.p, M->data, bytes, cudaMemcpyHostToDevice, s));
    t_upload_stats.direct_bytes += (int64_t)bytes;
    return launch_pack(M->kind, m, n, staging.p, dP, ld, s);
}

}  // namespace mela

// ---------------------------------------------------------------- C ABI
using namespace mela;

extern "C" int mela_version(void) { return 10000; }

extern "C" void mela_upload_stats_get(mela_upload_stats *out, int reset)
{
    if (out) *out = t_upload_stats;
    if (reset) t_upload_stats = mela_upload_stats{};
}

extern "C" const char *mela_status_string(mela_status s)
{
    switch (s) {
    case MELA_OK: return "ok";
    case MELA_ERR_INVALID: return "invalid argument";
    case MELA_ERR_SPARSE: return "sparse input not supported";
    case MELA_ERR_DIM: return "inner dimensions must agree";
    case MELA_ERR_TYPE: return "input must be logical or double";
    case MELA_ERR_NOMEM: return "out of memory";
    case MELA_ERR_CUDA: return "CUDA error";
    case MELA_ERR_TIMEOUT: return "device wait timed out";
    case MELA_ERR_UNSUPPORTED: return "unsupported";
    case MELA_ERR_NO_DEVICE: return "no CUDA device";
    }
    return "unknown status";
}

extern "C" const char *mela_last_error(void) { return t_err; }

extern "C" mela_status mela_device_error_flags(uint32_t *flags, int clear)
{
    u32 *p = device_error_word();
    if (!p) {
        set_error("device error word unavailable");
        return MELA_ERR_CUDA;
    }
    u32 v = 0;
    MELA_CUDA_TRY(cudaMemcpy(&v, p, 4, cudaMemcpyDeviceToHost));
    if (clear && v) MELA_CUDA_TRY(cudaMemset(p, 0, 4));
    if (flags) *flags = v;
    return MELA_OK;
}

extern "C" size_t mela_matmul_workspace_size(int32_t variant, int64_t m, int64_t k, int64_t n)
{
    Tuning t;
    if (!decode_gemm_variant(variant, &t)) return 0;
    return gemm_workspace(variant, m, k, n);
}

extern "C" mela_status mela_dev_matmul(int32_t variant, const uint64_t *dA, int64_t lda,
                                       const uint64_t *dB, int64_t ldb, uint64_t *dC, int64_t ldc,
                                       int64_t m, int64_t k, int64_t n, void *workspace,
                                       size_t workspace_bytes, void *stream)
{
    Tuning tn;
    if (m < 0 || k < 0 || n < 0 || !decode_gemm_variant(variant, &tn) ||
        lda < words_of(k) || ldb < words_of(n) || ldc < words_of(n)) {
        set_error("mela_dev_matmul: bad shape, leading dimension or variant");
        return MELA_ERR_INVALID;
    }
    if (m > 0 && n > 0 && (!dC || (k > 0 && (!dA || !dB)))) {
        set_error("mela_dev_matmul: null operand");
        return MELA_ERR_INVALID;
    }
    return gemm_device(variant, (const u64 *)dA, lda, (const u64 *)dB, ldb, (u64 *)dC, ldc, m, k,
                       n, workspace, workspace_bytes, (cudaStream_t)stream);
}

static mela_status check_dev_matmul_args(int32_t variant, const uint64_t *dA, int64_t lda,
                                         const uint64_t *dB, int64_t ldb, int64_t ldc, int64_t m,
                                         int64_t k, int64_t n)
{
    Tuning tn;
    if (m < 0 || k < 0 || n < 0 || !decode_gemm_variant(variant, &tn) ||
        lda < words_of(k) || ldb < words_of(n) || ldc < words_of(n)) {
        set_error("bad shape, leading dimension or variant");
        return MELA_ERR_INVALID;
    }
    if (m > 0 && n > 0 && k > 0 && (!dA || !dB)) {
        set_error("null operand");
        return MELA_ERR_INVALID;
    }
    return MELA_OK;
}

extern "C" mela_status mela_dev_matmul_prepare(int32_t variant, const uint64_t *dA, int64_t lda,
                                               const uint64_t *dB, int64_t ldb, int64_t m,
                                               int64_t k, int64_t n, void *workspace,
                                               size_t workspace_bytes, void *stream)
{
    mela_status st = check_dev_matmul_args(variant, dA, lda, dB, ldb, words_of(n), m, k, n);
    if (st != MELA_OK) return st;
    return gemm_prepare(variant, (const u64 *)dA, lda, (const u64 *)dB, ldb, m, k, n, workspace,
                        workspace_bytes, (cudaStream_t)stream);
}

extern "C" mela_status mela_dev_matmul_run(int32_t variant, const uint64_t *dA, int64_t lda,
                                           const uint64_t *dB, int64_t ldb, uint64_t *dC,
                                           int64_t ldc, int64_t m, int64_t k, int64_t n,
                                           void *workspace, size_t workspace_bytes, void *stream)
{
    mela_status st = check_dev_matmul_args(variant, dA, lda, dB, ldb, ldc, m, k, n);
    if (st != MELA_OK) return st;
    if (m > 0 && n > 0 && !dC) {
        set_error("null output");
        return MELA_ERR_INVALID;
    }
    return gemm_run(variant, (const u64 *)dA, lda, (const u64 *)dB, ldb, (u64 *)dC, ldc, m, k, n,
                    workspace, workspace_bytes, (cudaStream_t)stream);
}

// Tensor-core product of host matrices with the transfers overlapped.  A is
// cut into row blocks A_i and B into column blocks B_j (up to 4 x 4); the
// upload stream sends A_0, B_0, A_1, B_1, ...; the compute stream prepares
// each block as it lands (A_i expanded; B_j transposed and expanded) and runs
// the product C_ij = A_i B_j as soon as both of its blocks are in, in the
// order (i, j <= i) after A_i and (i <= j, j) after B_j; the download stream
// sends each C_ij back while the next one is computed.  The first product thus
// starts after two blocks have landed rather than after all of B.  (With
// page-locked host buffers the three streams run concurrently; pageable
// buffers still give the right result, with less overlap.)
static constexpr i64 kPipeMin = 8192;  // pipelined when m and n both reach this

static mela_status matmul_packed_host_pipelined(const uint64_t *A, int64_t lda, const uint64_t *B, int64_t ldb,
                                                uint64_t *C, int64_t ldc, i64 m, i64 k, i64 n, int variant,
                                                cudaStream_t s)
{
    cudaStream_t sin = nullptr, sout = nullptr;
    mela_status st = copy_streams(&sin, &sout);
    if (st != MELA_OK) return st;
    const bool fp4 = MELA_VARIANT_BASE(variant) == MELA_GEMM_TC_FP4;
    if (fp4 && k >= (1LL << 23)) {
        set_error("fp4 tensor-core product needs k < 2^23 (exact f32 sums)");
        return MELA_ERR_UNSUPPORTED;
    }
    const GemmPlan p = plan_gemm(variant, m, k, n);
    const i64 wk = words_of(k), wn = words_of(n);
    // blocks: a multiple of 256 rows (columns), at most 4 per operand
    const i64 mb = round_up((m + 3) / 4, 256), nb = round_up((n + 3) / 4, 256);
    const int bm = (int)((m + mb - 1) / mb), bn = (int)((n + nb - 1) / nb);
    DevBuf dA, dB, dC, ws;
    if ((st = dA.alloc((size_t)m * wk * 8, s)) != MELA_OK) return st;
    if ((st = dB.alloc((size_t)k * wn * 8, s)) != MELA_OK) return st;
    if ((st = dC.alloc((size_t)m * wn * 8, s)) != MELA_OK) return st;
    if ((st = ws.alloc(p.total, s)) != MELA_OK) return st;
    const GemmBufs b = carve(p, ws.p);
    u64 *a = (u64 *)dA.p, *bb = (u64 *)dB.p, *c = (u64 *)dC.p;

    // events: buffers allocated; A_i uploaded; B_j uploaded; C_ij computed; copy streams done
    constexpr int kMaxEv = 1 + 4 + 4 + 16 + 2;
    cudaEvent_t evs[kMaxEv];
    const int nev = 1 + bm + bn + bm * bn + 2;
    int made = 0;
    auto cleanup = [&]() {
        for (int i = 0; i < made; ++i) cudaEventDestroy(evs[i]);
    };
    for (; made < nev; ++made) {
        if (cudaEventCreateWithFlags(&evs[made], cudaEventDisableTiming) != cudaSuccess) {
            cleanup();
            set_error("cudaEventCreate failed");
            return MELA_ERR_CUDA;
        }
    }
    cudaEvent_t ev_alloc = evs[0], ev_done_in = evs[nev - 2], ev_done_out = evs[nev - 1];
    auto ev_a = [&](int i) { return evs[1 + i]; };
    auto ev_b = [&](int j) { return evs[1 + bm + j]; };
    auto ev_c = [&](int i, int j) { return evs[1 + bm + bn + i * bn + j]; };
    auto rows_of = [&](int i) { return (m - i * mb) < mb ? (m - i * mb) : mb; };
    auto cols_of = [&](int j) { return (n - j * nb) < nb ? (n - j * nb) : nb; };

    auto product = [&](int i, int j) -> mela_status {
        const i64 r0 = i * mb, c0 = j * nb, rows = rows_of(i), cols = cols_of(j);
        mela_status e = launch_gemm_tc(b.A8 + (size_t)r0 * p.kp, b.B8 + (size_t)c0 * p.kp, round_up(rows, 256),
                                       round_up(cols, 256), p.kp, c + r0 * wn + c0 / 64, wn, rows, cols, s, fp4,
                                       p.tc_tile);
        if (e != MELA_OK) return e;
        MELA_CUDA_TRY(cudaEventRecord(ev_c(i, j), s));
        MELA_CUDA_TRY(cudaStreamWaitEvent(sout, ev_c(i, j), 0));
        MELA_CUDA_TRY(cudaMemcpy2DAsync(C + r0 * ldc + c0 / 64, (size_t)ldc * 8, c + r0 * wn + c0 / 64,
                                        (size_t)wn * 8, (size_t)words_of(cols) * 8, (size_t)rows,
                                        cudaMemcpyDeviceToHost, sout));
        return MELA_OK;
    };
    auto run = [&]() -> mela_status {
        MELA_CUDA_TRY(cudaEventRecord(ev_alloc, s));
        MELA_CUDA_TRY(cudaStreamWaitEvent(sin, ev_alloc, 0));
        MELA_CUDA_TRY(cudaStreamWaitEvent(sout, ev_alloc, 0));
        for (int r = 0; r < (bm > bn ? bm : bn); ++r) {
            if (r < bm) {
                const i64 r0 = r * mb;
                MELA_CUDA_TRY(cudaMemcpy2DAsync(a + r0 * wk, (size_t)wk * 8, A + r0 * lda, (size_t)lda * 8,
                                                (size_t)wk * 8, (size_t)rows_of(r), cudaMemcpyHostToDevice, sin));
                MELA_CUDA_TRY(cudaEventRecord(ev_a(r), sin));
            }
            if (r < bn) {
                const i64 w0 = r * nb / 64;
                MELA_CUDA_TRY(cudaMemcpy2DAsync(bb + w0, (size_t)wn * 8, B + w0, (size_t)ldb * 8,
                                                (size_t)words_of(cols_of(r)) * 8, (size_t)k,
                                                cudaMemcpyHostToDevice, sin));
                MELA_CUDA_TRY(cudaEventRecord(ev_b(r), sin));
            }
        }
        mela_status e;
        for (int r = 0; r < (bm > bn ? bm : bn); ++r) {
            if (r < bm) {
                const i64 r0 = r * mb, rows = rows_of(r);
                MELA_CUDA_TRY(cudaStreamWaitEvent(s, ev_a(r), 0));
                e = launch_expand(a + r0 * wk, wk, rows, round_up(rows, 256), b.A8 + (size_t)r0 * p.kp, nullptr, 0, 0, 0,
                                  nullptr, k, p.kp, fp4, s);
                if (e != MELA_OK) return e;
                for (int j = 0; j < r && j < bn; ++j)
                    if ((e = product(r, j)) != MELA_OK) return e;
            }
            if (r < bn) {
                const i64 c0 = r * nb, cols = cols_of(r);
                MELA_CUDA_TRY(cudaStreamWaitEvent(s, ev_b(r), 0));
                e = launch_expand(nullptr, 0, 0, 0, nullptr, bb + c0 / 64, wn, cols, round_up(cols, 256),
                                  b.B8 + (size_t)c0 * p.kp, k, p.kp, fp4, s);
                if (e != MELA_OK) return e;
                for (int i = 0; i <= r && i < bm; ++i)
                    if ((e = product(i, r)) != MELA_OK) return e;
            }
        }
        return MELA_OK;
    };
    st = run();
    // the buffers are released on s: it waits for both copy streams first
    if (cudaEventRecord(ev_done_in, sin) == cudaSuccess) cudaStreamWaitEvent(s, ev_done_in, 0);
    if (cudaEventRecord(ev_done_out, sout) == cudaSuccess) cudaStreamWaitEvent(s, ev_done_out, 0);
    const mela_status fin = finish(s);
    cleanup();
    return st != MELA_OK ? st : fin;
}

extern "C" mela_status mela_matmul_packed_host(const uint64_t *A, int64_t lda, const uint64_t *B,
                                               int64_t ldb, uint64_t *C, int64_t ldc, int64_t m,
                                               int64_t k, int64_t n, int32_t variant)
{
    Tuning tn;
    if (m < 0 || k < 0 || n < 0 || lda < words_of(k) || ldb < words_of(n) || ldc < words_of(n) ||
        !decode_gemm_variant(variant, &tn)) {
        set_error("mela_matmul_packed_host: bad shape or variant");
        return MELA_ERR_INVALID;
    }
    if (m == 0 || n == 0) return MELA_OK;
    cudaStream_t s;
    mela_status st = host_stream(&s);
    if (st != MELA_OK) return st;
    {
        // The transfers are pipelined for an explicit tensor-core variant, and
        // for AUTO under the fixed rule; AUTO with a cost model installed
        // uploads first, since the model's choice depends on the data.
        int32_t v = variant;
        if (tn.base == MELA_GEMM_AUTO && !costmodel_loaded()) v = fixed_gemm_variant(m, k, n);
        const int b = MELA_VARIANT_BASE(v);
        if ((b == MELA_GEMM_TC || b == MELA_GEMM_TC_FP4) && k > 0 && m >= kPipeMin && n >= kPipeMin)
            return matmul_packed_host_pipelined(A, lda, B, ldb, C, ldc, m, k, n, v, s);
    }
    const i64 wk = words_of(k), wn = words_of(n);
    DevBuf dA, dB, dC, ws;
    if ((st = dA.alloc((size_t)m * (wk ? wk : 1) * 8, s)) != MELA_OK) return st;
    if ((st = dB.alloc((size_t)(k ? k : 1) * wn * 8, s)) != MELA_OK) return st;
    if ((st = dC.alloc((size_t)m * wn * 8, s)) != MELA_OK) return st;
    size_t wsb = gemm_workspace(variant, m, k, n);
    if ((st = ws.alloc(wsb, s)) != MELA_OK) return st;
    if (k > 0) {
        MELA_CUDA_TRY(cudaMemcpy2DAsync(dA.p, (size_t)wk * 8, A, (size_t)lda * 8, (size_t)wk * 8,
                                        (size_t)m, cudaMemcpyHostToDevice, s));
        MELA_CUDA_TRY(cudaMemcpy2DAsync(dB.p, (size_t)wn * 8, B, (size_t)ldb * 8, (size_t)wn * 8,
                                        (size_t)k, cudaMemcpyHostToDevice, s));
    }
    st = gemm_device(variant, (const u64 *)dA.p, wk, (const u64 *)dB.p, wn, (u64 *)dC.p, wn, m, k, n,
                     ws.p, wsb, s);
    if (st != MELA_OK) return st;
    MELA_CUDA_TRY(cudaMemcpy2DAsync(C, (size_t)ldc * 8, dC.p, (size_t)wn * 8, (size_t)wn * 8,
                                    (size_t)m, cudaMemcpyDeviceToHost, s));
    return finish(s);
}

// Shared body of the two product gateways (reference validation order:
// src/mela_matmul_gf2.c:75-88).
static mela_status matmul_host(const mela_host_matrix *A, const mela_host_matrix *B, uint8_t *C,
                               int variant)
{
    if (!A || !B) {
        set_error("null argument");
        return MELA_ERR_INVALID;
    }
    if (A->sparse || B->sparse) return MELA_ERR_SPARSE;
    if (A->cols != B->rows) return MELA_ERR_DIM;
    auto ok_kind = [](int k) { return k == MELA_KIND_LOGICAL || k == MELA_KIND_DOUBLE; };
    if (!ok_kind(A->kind) || !ok_kind(B->kind)) return MELA_ERR_TYPE;
    const i64 m = A->rows, k = A->cols, n = B->cols;
    if (m < 0 || k < 0 || n < 0) return MELA_ERR_INVALID;
    if (m == 0 || n == 0) return MELA_OK;
    if (!C || (k > 0 && (!A->data || !B->data))) {
        set_error("null data pointer");
        return MELA_ERR_INVALID;
    }
    cudaStream_t s;
    mela_status st = host_stream(&s);
    if (st != MELA_OK) return st;
    const size_t ea = A->kind == MELA_KIND_DOUBLE ? 8 : 1, eb = B->kind == MELA_KIND_DOUBLE ? 8 : 1;
    if (k > 0 && gemm_small_fits(m, k, n, ea, eb)) {
        if (variant == MELA_GEMM_AUTO) remember_variant(MELA_GEMM_PLAIN, -1.0);  // AND and parity, untabled
        const size_t ab = ((size_t)m * k * ea + 255) & ~(size_t)255, bb = ((size_t)k * n * eb + 255) & ~(size_t)255;
        // The kernel writes up to 64 KB of result into the thread's page-locked
        // words itself, where two copies and their start cost more than one
        // GPU's scattered writes over the bus (64^3 43 -> 32 us a call, 200^3 52
        // -> 47; 300 x 64 x 300, 90 KB, 51 -> 59).  Up to 24 KB of operands go
        // up from there in one copy (100 x 120 x 80 34 -> 33 us, 16^3 38 -> 28;
        // 64 x 200 x 64, 26 KB, 37 -> 41: the driver's own staging overlaps).
        Posted to;
        const bool post = (size_t)m * n <= ((size_t)64 << 10) && posted(&to);
        DevBuf all;
        if ((st = all.alloc(ab + bb + (post ? 0 : (size_t)m * n), s)) != MELA_OK) return st;
        unsigned char *dA = (unsigned char *)all.p, *dB = dA + ab;
        if (post && ab + bb <= ((size_t)24 << 10)) {
            std::memcpy(to.in, A->data, (size_t)m * k * ea);
            std::memcpy(to.in + ab, B->data, (size_t)k * n * eb);
            MELA_CUDA_TRY(cudaMemcpyAsync(dA, to.in, ab + (size_t)k * n * eb, cudaMemcpyHostToDevice, s));
        } else {
            MELA_CUDA_TRY(cudaMemcpyAsync(dA, A->data, (size_t)m * k * ea, cudaMemcpyHostToDevice, s));
            MELA_CUDA_TRY(cudaMemcpyAsync(dB, B->data, (size_t)k * n * eb, cudaMemcpyHostToDevice, s));
        }
        t_upload_stats.direct_bytes += (int64_t)((size_t)m * k * ea + (size_t)k * n * eb);
        if (post) {
            st = launch_gemm_small(A->kind, dA, B->kind, dB, to.bytes, m, k, n, to.err_word, to.err, s);
            if (st == MELA_OK) st = finish_posted(s);
            if (st == MELA_OK) std::memcpy(C, to.bytes, (size_t)m * n);
            return st;
        }
        unsigned char *dC = dB + bb;
        st = launch_gemm_small(A->kind, dA, B->kind, dB, dC, m, k, n, nullptr, nullptr, s);
        if (st != MELA_OK) return st;
        return download_finish(C, dC, (size_t)m * n, s);
    }
    const i64 lda = even_words(k), ldb = even_words(n), ldc = even_words(n);
    DevBuf pA, pB, pC, sA, sB, ws, outb;
    if ((st = pA.alloc((size_t)m * lda * 8, s)) != MELA_OK) return st;
    if ((st = pB.alloc((size_t)(k ? k : 1) * ldb * 8, s)) != MELA_OK) return st;
    if ((st = pC.alloc((size_t)m * ldc * 8, s)) != MELA_OK) return st;
    if ((st = upload_and_pack(A, (u64 *)pA.p, lda, s, sA)) != MELA_OK) return st;
    if ((st = upload_and_pack(B, (u64 *)pB.p, ldb, s, sB)) != MELA_OK) return st;
    size_t wsb = gemm_workspace(variant, m, k, n);
    if ((st = ws.alloc(wsb, s)) != MELA_OK) return st;
    st = gemm_device(variant, (const u64 *)pA.p, lda, (const u64 *)pB.p, ldb, (u64 *)pC.p, ldc, m,
                     k, n, ws.p, wsb, s);
    if (st != MELA_OK) return st;
    if ((st = outb.alloc((size_t)m * n, s)) != MELA_OK) return st;
    if ((st = launch_unpack((const u64 *)pC.p, ldc, m, n, (unsigned char *)outb.p, s)) != MELA_OK)
        return st;
    return download_finish(C, outb.p, (size_t)m * n, s);
}

extern "C" mela_status mela_matmul_gf2(const mela_host_matrix *A, const mela_host_matrix *B,
                                       uint8_t *C)
{
    return matmul_host(A, B, C, MELA_GEMM_AUTO);
}

extern "C" mela_status mela_matmul_m4ri(const mela_host_matrix *A, const mela_host_matrix *B,
                                        uint8_t *C)
{
    return matmul_host(A, B, C, MELA_GEMM_M4RI);
}
