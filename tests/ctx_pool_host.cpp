// The context's allocations (yeti_b200/csrc/ctx.cu) on a CUDA runtime that is
// a few lists: what is asked of the device, in which sizes, and which stream
// waits for what.  Run with the name of a scenario; exits 0 if it holds.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "common.cuh"

namespace fake {
size_t capacity = size_t(1) << 40, used = 0, next = 4096;
std::map<void *, size_t> blocks;                       // device memory in use
std::vector<size_t> mallocs;                           // sizes asked for, in order
uintptr_t next_event = 1, next_stream = 0x1000;
std::set<uintptr_t> events;
std::map<uintptr_t, cudaStream_t> recorded;            // event -> stream
std::vector<std::pair<cudaStream_t, cudaStream_t>> waits;   // (waiting stream, stream of the event)
std::map<cudaStream_t, unsigned long long> ids;         // handle -> the stream it names now
unsigned long long next_id = 1;
}  // namespace fake
using namespace fake;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    mallocs.push_back(n);
    if (n > capacity - used) return cudaErrorMemoryAllocation;
    used += n;
    *p = reinterpret_cast<void *>(next);
    next += (n + 511) / 512 * 512;
    blocks[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    auto it = blocks.find(p);
    if (it == blocks.end()) return cudaErrorInvalidValue;
    used -= it->second;
    blocks.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    events.insert(next_event);
    *e = reinterpret_cast<cudaEvent_t>(next_event++);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    return events.erase(reinterpret_cast<uintptr_t>(e)) ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    recorded[reinterpret_cast<uintptr_t>(e)] = s;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    waits.push_back({s, recorded.at(reinterpret_cast<uintptr_t>(e))});
    return cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long *id) {
    if (!ids.count(s)) ids[s] = next_id++;
    return *id = ids[s], cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(next_stream += 16);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "out of memory"; }
const char *cudaGetErrorName(cudaError_t) { return "cudaErrorMemoryAllocation"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 0, cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) { return cudaErrorInvalidValue; }
}

#define HOLDS(c)                                                        \
    do {                                                                \
        if (!(c)) {                                                     \
            std::printf("%s:%d: not so: %s\n", __FILE__, __LINE__, #c); \
            std::exit(1);                                               \
        }                                                               \
    } while (0)

static const size_t MiB = size_t(1) << 20;

static yeti_ctx *context(size_t budget = 0) {
    yeti_ctx *c = nullptr;
    HOLDS(yeti_ctx_create(0, budget, &c) == YETI_OK);
    return c;
}
static void *take(yeti_ctx *c, size_t n) {
    void *p = nullptr;
    return yeti::dev_alloc(c, &p, n) == YETI_OK ? p : nullptr;
}

// A new block has the size asked for, whether the pool would keep it or not.
static void sizes() {
    yeti_ctx *c = context();
    for (size_t n : {16 * MiB + 512, 127 * MiB, 130 * MiB, size_t(6400) * MiB + 512}) {
        void *p = take(c, n);
        HOLDS(p && mallocs.back() == n && yeti_ctx_bytes_in_use(c) == n);
        yeti::dev_free(c, p, n);
        HOLDS(yeti_ctx_bytes_in_use(c) == 0);
    }
    HOLDS(used == 16 * MiB + 512 + 127 * MiB);      // the larger ones went straight back
    void *huge = take(c, SIZE_MAX - 100);
    HOLDS(!huge && mallocs.back() > SIZE_MAX / 2);
    yeti_ctx_destroy(c);
    HOLDS(used == 0 && events.empty());
}

// Memory that holds a set of blocks exactly holds them through a context.
static void device_just_large_enough() {
    const std::vector<size_t> want = {100 * MiB, 90 * MiB, 17 * MiB, 300 * MiB};
    for (size_t n : want) capacity = n + (capacity == size_t(1) << 40 ? 0 : capacity);
    yeti_ctx *c = context();
    for (int round = 0; round < 3; round++) {
        std::vector<void *> p;
        for (size_t n : want) HOLDS((p.push_back(take(c, n)), p.back()));
        HOLDS(used == capacity && !take(c, 512));
        for (size_t k = 0; k < p.size(); k++) yeti::dev_free(c, p[k], want[k]);
        void *other = take(c, 450 * MiB);            // what is kept gives way
        HOLDS(other);
        yeti::dev_free(c, other, 450 * MiB);
    }
    yeti_ctx_destroy(c);
    HOLDS(used == 0 && events.empty());
}

// The budget bounds what the device has given, kept blocks included, and takes
// every set of blocks that adds up to it.
static void budget() {
    yeti_ctx *c = context(400 * MiB);
    for (int round = 0; round < 3; round++) {
        std::vector<std::pair<void *, size_t>> p;
        for (size_t n : {101 * MiB, 99 * MiB, 33 * MiB, 67 * MiB, 90 * MiB, 10 * MiB}) {
            p.push_back({take(c, n - round * 512), n - round * 512});
            HOLDS(p.back().first && used <= 400 * MiB);
        }
        HOLDS(!take(c, 1 * MiB) && used <= 400 * MiB);
        for (auto &b : p) yeti::dev_free(c, b.first, b.second);
        HOLDS(used <= 400 * MiB && yeti_ctx_bytes_in_use(c) == 0);
    }
    yeti_ctx_destroy(c);
    HOLDS(used == 0);
}

// A repeated sequence of calls asks nothing more of the device; a block serves
// requests up to an eighth smaller, and goes back at its own size.
static void reuse() {
    yeti_ctx *c = context();
    const std::vector<size_t> want = {80 * MiB, 76 * MiB, 40 * MiB, 3000, 1000};
    size_t asked = 0;
    for (int round = 0; round < 4; round++) {
        std::vector<void *> p;
        for (size_t n : want) p.push_back(take(c, n));
        for (size_t k = 0; k < p.size(); k++) yeti::dev_free(c, p[k], want[k]);
        if (round == 0) asked = mallocs.size();
        HOLDS(mallocs.size() == asked);
    }
    void *p = take(c, 72 * MiB);                     // in the block of 76 MiB
    HOLDS(mallocs.size() == asked && blocks.at(p) == 76 * MiB && yeti_ctx_bytes_in_use(c) == 72 * MiB);
    yeti::dev_free(c, p, 72 * MiB);
    void *q = take(c, 76 * MiB);
    HOLDS(mallocs.size() == asked && q == p);
    void *r = take(c, 60 * MiB);                     // not in the one of 80 MiB
    HOLDS(mallocs.size() == asked + 1 && blocks.at(r) == 60 * MiB);
    yeti::dev_free(c, q, 76 * MiB);
    yeti::dev_free(c, r, 60 * MiB);
    HOLDS(c->pool_bytes == used && c->larger.empty());
    yeti_ctx_destroy(c);
    HOLDS(used == 0 && events.empty());
}

// What a context keeps goes back on request, and when another one, serving or
// not, finds the device full.
static void given_back() {
    capacity = 400 * MiB;
    yeti_ctx *a = context(), *b = context();
    auto keep = [&] {
        void *p = take(a, 120 * MiB), *q = take(a, 110 * MiB);
        HOLDS(p && q);
        yeti::dev_free(a, p, 120 * MiB);
        yeti::dev_free(a, q, 110 * MiB);
        HOLDS(used == 230 * MiB && yeti_ctx_bytes_in_use(a) == 0);
    };
    keep();
    HOLDS(yeti_ctx_trim(a) == YETI_OK && used == 0 && events.empty());
    for (bool serving : {false, true}) {
        b->stream_ordered = serving;
        keep();
        void *p = take(b, 300 * MiB);
        HOLDS(p && used == 300 * MiB);
        yeti::dev_free(b, p, 300 * MiB);
        HOLDS(used == 0);
    }
    HOLDS(yeti_ctx_trim(nullptr) == YETI_EINVAL);
    yeti_ctx_destroy(a);
    void *p = take(b, 401 * MiB);                    // past the context that is gone
    HOLDS(!p);
    yeti_ctx_destroy(b);
}

// A stream that takes a block waits for the one that freed it, unless it is
// the same; a handle that names a stream created since is not.
static void order() {
    yeti_ctx *c = context();
    cudaStream_t s[] = {reinterpret_cast<cudaStream_t>(0x11), reinterpret_cast<cudaStream_t>(0x22)};
    size_t n = 0;
    for (int from : {0, 1})
        for (int to : {0, 1})
            for (bool again : {false, true}) {
                HOLDS(yeti_ctx_set_stream(c, s[from]) == YETI_OK);
                void *p = take(c, 3 * MiB);
                HOLDS(p && waits.size() == n);
                yeti::dev_free(c, p, 3 * MiB);
                if (again) ids[s[to]] = next_id++;       // destroyed, and created at the same place
                HOLDS(yeti_ctx_set_stream(c, s[to]) == YETI_OK);
                HOLDS(take(c, 3 * MiB) == p);
                if (from != to || again) HOLDS(waits.size() == ++n && waits.back() == std::make_pair(s[to], s[from]));
                HOLDS(waits.size() == n);
                yeti::dev_free(c, p, 3 * MiB);
                HOLDS(yeti_ctx_trim(c) == YETI_OK);
            }
    // the handle of each thread's own stream says nothing about which
    HOLDS(yeti_ctx_set_stream(c, cudaStreamPerThread) == YETI_OK);
    for (int k = 0; k < 2; k++) {
        void *p = take(c, 3 * MiB);
        HOLDS(p && waits.size() == n + k);
        yeti::dev_free(c, p, 3 * MiB);
    }
    yeti_ctx_destroy(c);
    HOLDS(used == 0 && events.empty());
}

int main(int, char **argv) {
    const std::map<std::string, void (*)()> all = {{"sizes", sizes},
                                                   {"device_just_large_enough", device_just_large_enough},
                                                   {"budget", budget},
                                                   {"reuse", reuse},
                                                   {"given_back", given_back},
                                                   {"order", order}};
    all.at(argv[1])();
}
