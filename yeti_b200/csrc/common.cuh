// Shared definitions of the yeti_b200 library (host + device).
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/yeti_b200.h"

#define YETI_API extern "C" __attribute__((visibility("default")))

namespace yeti {

// Thread-local error text returned by yeti_last_error().
void set_error(const char *fmt, ...);

// Raise from a cudaError_t: records the text and returns YETI_ECUDA.
int cuda_fail(cudaError_t e, const char *what, const char *file, int line);

#define YETI_CUDA(expr)                                                     \
    do {                                                                    \
        cudaError_t _e = (expr);                                            \
        if (_e != cudaSuccess)                                              \
            return ::yeti::cuda_fail(_e, #expr, __FILE__, __LINE__);        \
    } while (0)

#define YETI_CHECK(cond, code, ...)                                         \
    do {                                                                    \
        if (!(cond)) {                                                      \
            ::yeti::set_error(__VA_ARGS__);                                 \
            return (code);                                                  \
        }                                                                   \
    } while (0)

// Propagate a non-zero status.
#define YETI_TRY(expr)                                                      \
    do {                                                                    \
        int _rc = (expr);                                                   \
        if (_rc != YETI_OK) return _rc;                                     \
    } while (0)

}  // namespace yeti

// Context: device, stream and device-memory accounting.
struct yeti_ctx {
    // the caller (until yeti_ctx_destroy) and every operator: whoever lets go
    // last deletes the context, in whatever order they are destroyed (a
    // garbage collector does not keep one)
    std::atomic<int> holders{1};
    std::atomic<bool> closed{false};    // yeti_ctx_destroy was called
    int device = 0;
    cudaStream_t stream = nullptr;      // stream all work goes to
    unsigned long long stream_id = 0;   // its id (ctx.cu), taken when it was set
    cudaStream_t own_stream = nullptr;  // stream created by the context
    size_t hbm_budget = 0;              // 0: unbounded
    std::atomic<size_t> bytes_in_use{0};
    // allocate with cudaMallocAsync / cudaFreeAsync on `stream` (no implicit
    // device synchronisation; for contexts driven by the serving loop)
    bool stream_ordered = false;
    // Freed blocks kept for the next allocations (dev_alloc): a call's
    // scratch costs a list lookup instead of cudaMalloc and cudaFree, which
    // took 2 to 4 ms of a Gauss call or an operator setup.  An allocation
    // takes the smallest kept block that holds it and is at most an eighth
    // larger (no larger under an HBM budget, which therefore bounds what the
    // device gives); a new block has the size asked for.  Each kept block
    // carries an event recorded on the context's stream when it was freed, which
    // another stream waits for before it takes the block.  At most kPoolBytes
    // are kept, the blocks freed last; they are given back with the context, and
    // earlier by yeti_ctx_trim, when an allocation of any context on the device
    // fails, or when the HBM budget needs the room.  (When
    // a full pool kept the oldest instead, a 32x24x28 p=3 setup after calls of
    // other sizes paid for cudaMalloc and cudaFree of its 80 MB blocks every
    // time: up to 11 ms against 1.4 ms.)
    struct PoolBlock {
        void *ptr;
        cudaEvent_t freed;
        unsigned long long stream;   // id of the stream it was recorded on
        uint64_t age;          // count of blocks kept before it
    };
    std::mutex pool_mu;
    std::multimap<size_t, PoolBlock> pool;     // by size
    std::unordered_map<void *, size_t> larger; // sizes of blocks in use that exceed what was asked for
    size_t pool_bytes = 0;
    uint64_t pool_age = 0;
    // device-time accounting of the element kernels (yeti_ctx_set_timing)
    bool timing = false;
    std::mutex timing_mu;
    std::map<std::string, double> kernel_ms;
};

namespace yeti {

constexpr size_t kPoolBytes = size_t(512) << 20;   // most a context keeps of freed blocks
constexpr size_t kPoolBlock = size_t(128) << 20;   // largest block it keeps

// Device allocation charged against the context budget.  A block may come
// from the context's pool: its last user's work has been enqueued on the
// context's stream of that time (or is done), so all work on a buffer must
// be enqueued on the context's stream before the buffer is freed.
int dev_alloc(yeti_ctx *ctx, void **ptr, size_t bytes);
void dev_free(yeti_ctx *ctx, void *ptr, size_t bytes);
// Give the pool's blocks back to the device.
void pool_release(yeti_ctx *ctx);
// One holder less; the last one deletes the context.
void ctx_let_go(yeti_ctx *ctx);

// A holder of a context.
struct CtxHold {
    yeti_ctx *ctx = nullptr;
    CtxHold() = default;
    CtxHold(const CtxHold &) = delete;
    CtxHold &operator=(const CtxHold &) = delete;
    ~CtxHold() {
        if (ctx) ctx_let_go(ctx);
    }
    void take(yeti_ctx *c) {
        c->holders.fetch_add(1);
        ctx = c;
    }
};

// RAII device buffer owned by a context, or a view of a part of another one
// (owned == false).
struct DevBuf {
    yeti_ctx *ctx = nullptr;
    void *ptr = nullptr;
    size_t bytes = 0;
    bool owned = true;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    DevBuf(DevBuf &&o) noexcept : ctx(o.ctx), ptr(o.ptr), bytes(o.bytes), owned(o.owned) {
        o.ptr = nullptr;
        o.bytes = 0;
    }
    DevBuf &operator=(DevBuf &&o) noexcept {
        if (this != &o) {
            release();
            ctx = o.ctx;
            ptr = o.ptr;
            bytes = o.bytes;
            owned = o.owned;
            o.ptr = nullptr;
            o.bytes = 0;
        }
        return *this;
    }
    ~DevBuf() { release(); }
    int alloc(yeti_ctx *c, size_t n) {
        release();
        ctx = c;
        int rc = dev_alloc(c, &ptr, n);
        if (rc == YETI_OK) bytes = n;
        return rc;
    }
    void view(void *p, size_t n) {
        release();
        ptr = p;
        bytes = n;
        owned = false;
    }
    void release() {
        if (ptr && owned) dev_free(ctx, ptr, bytes);
        ptr = nullptr;
        bytes = 0;
        owned = true;
    }
    template <class T> T *as() const { return static_cast<T *>(ptr); }
};

// Upload a host array into a fresh DevBuf.
template <class T>
int upload(yeti_ctx *ctx, DevBuf &buf, const T *host, size_t n) {
    YETI_TRY(buf.alloc(ctx, n * sizeof(T) + 16));
    if (n)
        YETI_CUDA(cudaMemcpyAsync(buf.ptr, host, n * sizeof(T),
                                  cudaMemcpyHostToDevice, ctx->stream));
    return YETI_OK;
}

// Host arrays uploaded together: add() copies them into one host buffer,
// commit() allocates `arena`, makes one copy and turns the arrays' buffers into
// views of it (arena must outlive them).
class UploadPack {
    struct Item {
        DevBuf *buf;
        size_t off, bytes;
    };
    std::vector<Item> items;
    std::vector<char> host;

public:
    template <class T>
    void add(DevBuf &buf, const T *data, size_t n) {
        const size_t off = (host.size() + 255) & ~size_t(255), bytes = n * sizeof(T);
        host.resize(off + bytes + 16);
        if (bytes) memcpy(host.data() + off, data, bytes);
        items.push_back({&buf, off, bytes});
    }
    template <class T>
    void add(DevBuf &buf, const std::vector<T> &v) {
        add(buf, v.data(), v.size());
    }
    int commit(yeti_ctx *ctx, DevBuf &arena) {
        YETI_TRY(upload(ctx, arena, host.data(), host.size()));
        for (const Item &it : items) it.buf->view(arena.as<char>() + it.off, it.bytes);
        items.clear();
        host.clear();
        return YETI_OK;
    }
};

// Guard that makes ctx->device current for the scope.
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

// Is `p` device-accessible memory (device or managed)?
bool is_device_pointer(const void *p);

// Let `func` (a kernel) use the device's whole opt-in shared memory: the
// same value on every call, so host threads that launch the kernel
// concurrently cannot lower the limit under each other's launch.  Fails with
// YETI_EUNSUPPORTED when `need` dynamic bytes exceed it.
int set_smem_optin(const void *func, int device, size_t need, const char *what);

// With the context's timing on, the device time of the work enqueued on
// ctx->stream during the object's lifetime (CUDA events on that stream,
// waited for on destruction) is added to ctx->kernel_ms[name]; with timing
// off it does nothing.
struct KernelTimer {
    yeti_ctx *ctx;
    const char *name;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    KernelTimer(yeti_ctx *c, const char *n);
    ~KernelTimer();
};

// Process-wide count of kernel launches issued by the library (reported by
// yeti_kernel_launches(); lets callers verify the device path ran).
void count_launches(uint64_t n);

}  // namespace yeti
