// A CUDA runtime without a GPU, for LD_PRELOAD before libgravcuda.so: device
// memory is host memory, launches do nothing but the few listed in `emulate`,
// and an allocation can be made to fail.  It counts what a host path does
// with its memory: live buffers, buffers freed twice, and work left on the
// default stream.  With the emulated kernels a build sees two bodies in one
// leaf cell, one sink group, and lists of every kind whose queue claims 8192
// items.
#include <stddef.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <mutex>
#include <set>
#include <string>

namespace {
constexpr int kOutOfMemory = 2, kInvalidValue = 1;
std::recursive_mutex mu;
std::map<const void *, std::string> names;     // host stub -> kernel name
std::map<const void *, int> smem_limit;        // kernel -> its dynamic shared memory attribute
std::map<std::string, unsigned> grids;         // kernel -> blocks of its last launch (x)
std::map<std::string, long> first_at;          // kernel -> allocations made before its first launch
std::map<void *, size_t> live;
std::set<void *> host_live;
size_t live_bytes = 0, peak_bytes = 0;
long long cells = 1;  // what a tree needs room for
int last_error = 0;
long nalloc = 0, fail_at = 0, double_frees = 0, trims = 0, pending = 0, device_waits = 0;
long elsewhere = 0, freed_early = 0;  // launches on other streams, and pool buffers freed under them
bool once = false;  // the failing allocation succeeds once the pool has been trimmed

int ret(int e) {
    if (e)
        last_error = e;
    return e;
}
int get(void **p, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    *p = nullptr;
    nalloc++;
    if (fail_at && nalloc >= fail_at && !(once && trims))
        return ret(kOutOfMemory);
    *p = calloc(1, n + 256);
    live[*p] = n;
    live_bytes += n;
    if (live_bytes > peak_bytes)
        peak_bytes = live_bytes;
    return 0;
}
int put(void *p) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (!p)
        return 0;
    const auto it = live.find(p);
    if (it == live.end()) {
        double_frees++;
        return ret(kInvalidValue);
    }
    live_bytes -= it->second;
    live.erase(it);
    free(p);
    return 0;
}
// work on the default stream, which other streams do not wait for
void on(void *stream) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (!stream)
        pending++;
    else
        elsewhere++;
}
void waited(void *stream) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (!stream)
        pending = 0;
}

template <typename T>
T arg(void **args, int k) {
    return *static_cast<T *>(args[k]);
}
void emulate(const std::string &f, void **a) {
    auto is = [&](const char *s) { return f.find(s) != std::string::npos; };
    if (is("k_split_root")) {  // the root alone, on level 0
        arg<int64_t *>(a, 6)[0] = 0;
        arg<int64_t *>(a, 6)[1] = 1;
    } else if (is("k_split_write")) {
        if (arg<int64_t>(a, 5) < cells)
            *arg<unsigned *>(a, 6) = 1;
    } else if (is("k_runs_compact") || is("k_runs_k1")) {
    } else if (is("k_runs")) {
        arg<int64_t *>(a, 3)[0] = 1;
    } else if (is("k_piece_count")) {
        arg<int64_t *>(a, 3)[0] = 1;
    } else if (is("k_groups")) {  // nln_group: centre (3 doubles), first, count, radius
        unsigned char *g = arg<unsigned char *>(a, 5);
        const int32_t two = 2;
        memcpy(g + 32, &two, 4);
    } else if (is("k_walkILb0")) {  // counting pass: points, quadrupoles, order 4, correction
        int64_t *c = arg<int64_t *>(a, 8);
        const int64_t v[6] = {2, 1, 1, 2, 2, arg<int64_t>(a, 2)};
        if (c)
            memcpy(c, v, sizeof(v));
    } else if (is("k_queue_count")) {
        int64_t *all = arg<int64_t *>(a, 5);
        all[0] = 3;
    } else if (is("k_queue_nrem")) {
        for (int k = 0; k < 3; k++) arg<int64_t *>(a, 2)[k] = 8192;
    } else if (is("DeviceScanKernel")) {  // exclusive sums of the int64 counts
        const int64_t *in = arg<const int64_t *>(a, 0);
        int64_t *out = arg<int64_t *>(a, 1), s = 0;
        for (int i = 0; i < 2; i++) {
            const int64_t v = in[i];
            out[i] = s;
            s += v;
        }
    }
}
void launched(const void *f, void **args) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    first_at.emplace(names[f], nalloc);
    emulate(names[f], args);
}
struct dim3_ {
    unsigned x, y, z;
};
}  // namespace

extern "C" {
void fake_reset(long fail, int until_trimmed) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    nalloc = double_frees = trims = pending = elsewhere = freed_early = device_waits = 0;
    fail_at = fail;
    once = until_trimmed != 0;
    first_at.clear();
    peak_bytes = live_bytes;
    cells = 1;
}
// allocations asked for, buffers live, buffers freed twice, trims, default-stream work not
// waited for, last error
void fake_counts(long *out) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    const long v[6] = {nalloc, (long)live.size(), double_frees, trims, pending, last_error};
    memcpy(out, v, sizeof(v));
}
// allocations made before the kernel's first launch since the reset; -1: not launched
long fake_allocs_before(const char *kernel) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    for (auto &k : first_at)
        if (k.first.find(kernel) != std::string::npos)
            return k.second;
    return -1;
}
// device bytes in use, and the most since the reset
void fake_bytes(long *out) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    out[0] = (long)live_bytes;
    out[1] = (long)peak_bytes;
}
long fake_freed_early() { return freed_early; }
long fake_device_waits() { return device_waits; }
void fake_cells(long long need) { cells = need; }
unsigned fake_grid(const char *kernel) {
    for (auto &k : grids)
        if (k.first.find(kernel) != std::string::npos)
            return k.second;
    return 0;
}
int fake_smem_limit(const char *kernel) {
    for (auto &k : smem_limit)
        if (names[k.first].find(kernel) != std::string::npos)
            return k.second;
    return -1;
}

void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *,
                            void *, void *, int *) {
    names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
static thread_local struct {
    dim3_ g, b;
    size_t s;
    void *st;
} cfg;
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t s, void *st) {
    cfg = {g, b, s, st};
    return 0;
}
int __cudaPopCallConfiguration(dim3_ *g, dim3_ *b, size_t *s, void *st) {
    *g = cfg.g;
    *b = cfg.b;
    *s = cfg.s;
    *(void **)st = cfg.st;
    return 0;
}
int cudaLaunchKernel(const void *f, dim3_, dim3_, void **args, size_t, void *st) {
    launched(f, args);
    on(st);
    return 0;
}
struct launch_ {  // cudaLaunchConfig_t's first members
    dim3_ grid, block;
    size_t smem;
    void *stream;
};
int cudaLaunchKernelExC(const launch_ *cfg, const void *f, void **args) {
    launched(f, args);
    on(cfg->stream);
    grids[names[f]] = cfg->grid.x;
    return 0;
}

int cudaMalloc(void **p, size_t n) { return get(p, n); }
int cudaMallocFromPoolAsync(void **p, size_t n, void *, void *st) {
    if (!n)
        return ret(kInvalidValue);
    on(st);
    return get(p, n);
}
int cudaFree(void *p) {
    waited(nullptr);
    return put(p);
}
int cudaFreeAsync(void *p, void *) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    freed_early += elsewhere > 0;
    return p ? put(p) : ret(kInvalidValue);
}
int cudaMallocHost(void **p, size_t n) {
    *p = aligned_alloc(4096, (n + 4095) / 4096 * 4096);
    std::lock_guard<std::recursive_mutex> lk(mu);
    host_live.insert(*p);
    return 0;
}
int cudaFreeHost(void *p) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    host_live.erase(p);
    free(p);
    return 0;
}
int cudaMemPoolCreate(void **p, const void *) {
    *p = (void *)0x1000;
    return 0;
}
int cudaMemPoolSetAttribute(void *, int, void *) { return 0; }
int cudaMemPoolTrimTo(void *, size_t) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    trims++;
    return 0;
}
// kind 1, host to device: begins when the default stream is done, and may return while the copy
// is still under way; 2, device to host: ends before it returns; 3, on the device: does not wait
int cudaMemcpy(void *d, const void *s, size_t n, int kind) {
    memcpy(d, s, n);
    if (kind != 3)
        waited(nullptr);
    if (kind != 2)
        on(nullptr);
    return 0;
}
int cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *st) {
    memcpy(d, s, n);
    on(st);
    return 0;
}
int cudaMemset(void *p, int v, size_t n) {
    memset(p, v, n);
    on(nullptr);
    return 0;
}
int cudaMemsetAsync(void *p, int v, size_t n, void *st) {
    memset(p, v, n);
    on(st);
    return 0;
}

int cudaGetLastError() {
    const int e = last_error;
    last_error = 0;
    return e;
}
int cudaPeekAtLastError() { return last_error; }
const char *cudaGetErrorString(int) { return "fake"; }
int cudaGetDevice(int *d) {
    *d = 0;
    return 0;
}
int cudaSetDevice(int) { return 0; }
int cudaGetDeviceCount(int *n) {
    *n = 1;
    return 0;
}
int cudaGetDeviceProperties_v2(void *, int) { return ret(kInvalidValue); }
int cudaDeviceGetAttribute(int *v, int a, int) {
    *v = a == 16 ? 148 : a == 75 ? 10 : a == 76 ? 0 : a == 8 ? 49152 : a == 10 ? 32 : a == 5 ? 0x7fffffff : 1024;
    return 0;
}
int cudaDeviceSynchronize() {
    std::lock_guard<std::recursive_mutex> lk(mu);
    waited(nullptr);
    elsewhere = 0;
    device_waits++;
    return 0;
}
int cudaFuncGetAttributes(void *a, const void *) {  // cudaFuncAttributes: versions after 3 sizes, 2 ints
    memset(a, 0, 3 * sizeof(size_t) + 4 * sizeof(int));
    int *i = (int *)((size_t *)a + 3);
    i[0] = 1024;
    i[1] = 32;
    i[2] = i[3] = 100;
    return 0;
}
int cudaFuncSetAttribute(const void *f, int, int v) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    smem_limit[f] = v;
    return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
    *n = 3;
    return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 3;
    return 0;
}
int cudaGetSymbolAddress(void **p, const void *) {
    static char scratch[64 << 20];
    *p = scratch;
    return 0;
}
int cudaPointerGetAttributes(void *a, const void *p) {  // page-locked host memory, mapped
    memset(a, 0, 24);
    *(int *)a = 1;
    ((const void **)a)[1] = p;
    ((const void **)a)[2] = p;
    return 0;
}
static int encode(...) { return 0; }
int cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long, int *q) {
    *fn = (void *)encode;
    *q = 0;
    return 0;
}

int cudaStreamCreateWithFlags(void **s, unsigned) {
    *s = (void *)0x2000;
    return 0;
}
int cudaStreamDestroy(void *) { return 0; }
int cudaStreamSynchronize(void *s) {
    waited(s);
    return 0;
}
int cudaStreamQuery(void *) { return 0; }
int cudaStreamWaitEvent(void *, void *, unsigned) { return 0; }
int cudaStreamIsCapturing(void *, int *s) {
    *s = 0;
    return 0;
}
int cudaStreamBeginCapture(void *, int) { return 0; }
int cudaStreamEndCapture(void *, void **g) {
    *g = nullptr;
    return 0;
}
int cudaEventCreate(void **e) {
    *e = (void *)0x3000;
    return 0;
}
int cudaEventCreateWithFlags(void **e, unsigned) { return cudaEventCreate(e); }
int cudaEventDestroy(void *) { return 0; }
int cudaEventRecord(void *, void *) { return 0; }
int cudaEventQuery(void *) { return 0; }
int cudaEventSynchronize(void *) { return 0; }
int cudaEventElapsedTime(float *ms, void *, void *) {
    *ms = 0;
    return 0;
}
int cudaGraphDestroy(void *) { return 0; }
int cudaGraphExecDestroy(void *) { return 0; }
int cudaGraphInstantiate(void **g, void *, unsigned long long) {
    *g = nullptr;
    return 0;
}
int cudaGraphLaunch(void *, void *) { return 0; }
}
