// The kept device arrays of csrc/device_pool.cu over a stand-in for the CUDA
// calls it makes: allocations with addresses that come back after a free and
// ids that do not, a device reset, work in flight, captures, a host out of
// memory. argv[1] names one check; the exit code is the number of failures.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <string>
#include <vector>

static int fail_new = -1;   // allocations of the host until one fails, -1: none does
void* operator new(size_t n)
{
    if (fail_new >= 0 && fail_new-- == 0) throw std::bad_alloc();
    if (void* p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
struct Unfailing {   // the stand-in's own allocations
    int was = fail_new;
    Unfailing() { fail_new = -1; }
    ~Unfailing() { fail_new = was; }
};

namespace fake {
struct Block {
    size_t bytes;
    unsigned long long id;
};
std::map<char*, Block>& blocks() { static auto* m = new std::map<char*, Block>; return *m; }
std::multimap<size_t, char*>& holes() { static auto* m = new std::multimap<size_t, char*>; return *m; }
char* top = reinterpret_cast<char*>(0x700000000000ULL);
unsigned long long next_id = 0;
size_t total = 64ULL << 30, used = 0;
bool working = false;       // work in flight on the device
bool capturing = false;     // a stream of another thread is being captured
bool forbidden = false;     // ... in the mode that forbids allocating to every thread
bool invalidated = false;   // the capture was spoilt
int bad_frees = 0;

void vanish()   // a device reset
{
    for (auto& b : blocks()) holes().emplace(b.second.bytes, b.first);
    blocks().clear();
    used = 0;
    working = false;
}
bool live(void* p) { return blocks().count(static_cast<char*>(p)) != 0; }
}  // namespace fake

extern "C" {
cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t CUDARTAPI cudaSetDevice(int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemGetInfo(size_t* f, size_t* t) { *f = fake::total - fake::used; *t = fake::total; return cudaSuccess; }
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n)
{
    Unfailing u;
    if (fake::forbidden) { fake::invalidated = true; return cudaErrorStreamCaptureUnsupported; }
    if (fake::used + n > fake::total) return cudaErrorMemoryAllocation;
    auto hole = fake::holes().find(n);
    char* at = fake::top;
    if (hole != fake::holes().end()) {
        at = hole->second;
        fake::holes().erase(hole);
    } else {
        fake::top += n;
    }
    fake::blocks()[at] = {n, ++fake::next_id};
    fake::used += n;
    *p = at;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFree(void* p)
{
    Unfailing u;
    if (fake::forbidden) { fake::invalidated = true; return cudaErrorStreamCaptureUnsupported; }
    if (!p) return cudaSuccess;
    auto it = fake::blocks().find(static_cast<char*>(p));
    if (it == fake::blocks().end()) { fake::bad_frees++; return cudaErrorInvalidValue; }
    fake::used -= it->second.bytes;
    fake::holes().emplace(it->second.bytes, it->first);
    fake::blocks().erase(it);
    fake::working = false;   // freeing waits
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaDeviceSynchronize(void)
{
    if (fake::capturing) { fake::invalidated = true; return cudaErrorStreamCaptureUnsupported; }
    fake::working = false;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    memset(a, 0, sizeof(*a));
    a->type = fake::live(const_cast<void*>(p)) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
static CUresult fake_range(CUdeviceptr* base, size_t* n, CUdeviceptr p)
{
    auto it = fake::blocks().find(reinterpret_cast<char*>(p));
    if (it == fake::blocks().end()) return CUDA_ERROR_NOT_FOUND;
    *base = p;
    *n = it->second.bytes;
    return CUDA_SUCCESS;
}
static CUresult fake_attribute(void* out, CUpointer_attribute what, CUdeviceptr p)
{
    auto it = fake::blocks().find(reinterpret_cast<char*>(p));
    if (it == fake::blocks().end() || what != CU_POINTER_ATTRIBUTE_BUFFER_ID) return CUDA_ERROR_INVALID_VALUE;
    *static_cast<unsigned long long*>(out) = it->second.id;
    return CUDA_SUCCESS;
}
cudaError_t CUDARTAPI cudaGetDriverEntryPoint(const char* name, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q)
{
    *fn = !strcmp(name, "cuMemGetAddressRange") ? reinterpret_cast<void*>(fake_range)
          : !strcmp(name, "cuPointerGetAttribute") ? reinterpret_cast<void*>(fake_attribute) : nullptr;
    if (q) *q = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
}

namespace clspmv { int device_release(void* p, int idle_on); }
static struct AtExit {   // made before, so destroyed after, whatever the included file makes
    void* array = nullptr;
    ~AtExit()
    {
        if (!array) return;
        clspmv::device_release(array, -1);
        if (!fake::live(array)) _Exit(1);   // kept, as at any other time
    }
} at_exit;

#include "device_pool.cu"

using clspmv::device_alloc;
using clspmv::device_release;

static int failures = 0;
#define CHECK(c) \
    do { if (!(c)) { failures++; printf("line %d: %s\n", __LINE__, #c); } } while (0)

static void* make(size_t n)
{
    void* p = nullptr;
    CHECK(device_alloc(&p, n) == CLSPMV_OK && fake::live(p));
    return p;
}
static constexpr size_t MB = 1 << 20;

static void reuse()   // kept for the next request that it fits, given back by trim
{
    void* a = make(MB);
    device_release(a, clspmv::kIdleAll);
    CHECK(fake::live(a) && make(MB) == a);
    device_release(a, clspmv::kIdleAll);
    device_release(a, clspmv::kIdleAll);   // a second release of the same array
    void *b = make(MB), *c = make(MB);
    CHECK(b != c);
    device_release(b, clspmv::kIdleAll);
    CHECK(make(2 * MB) != b);
    clspmv_device_trim();
    CHECK(!fake::live(b) && fake::live(c));
}

static void bounds()   // 1/64 of the device and 256 arrays, the oldest leave first
{
    std::vector<void*> p;
    for (int i = 0; i < 12; i++) p.push_back(make(100 * MB));
    for (void* q : p) device_release(q, clspmv::kIdleAll);
    size_t held = 0;
    for (void* q : p) held += fake::live(q) ? 100 * MB : 0;
    CHECK(held <= fake::total / 64 && held + 100 * MB > fake::total / 64 && !fake::live(p[0]) && fake::live(p[11]));
    clspmv_device_trim();
    p.clear();
    for (int i = 0; i < 300; i++) p.push_back(make(4096));
    for (void* q : p) device_release(q, clspmv::kIdleAll);
    int n = 0;
    for (void* q : p) n += fake::live(q);
    CHECK(n <= 256 && n >= 250 && fake::live(p[299]));
    clspmv_device_trim();
    void* big = make(fake::total / 32);   // more than the list may hold
    device_release(big, clspmv::kIdleAll);
    CHECK(!fake::live(big));
}

static void low_memory()   // given back for an allocation that fails, and when little is left after a large one
{
    void* a = make(500 * MB);
    device_release(a, clspmv::kIdleAll);
    void* rest = nullptr;
    CHECK(device_alloc(&rest, fake::total - 200 * MB) == CLSPMV_OK && !fake::live(a));
    cudaFree(rest);
    a = make(500 * MB);
    device_release(a, clspmv::kIdleAll);
    rest = make(fake::total - fake::total / 8);
    CHECK(!fake::live(a));
    cudaFree(rest);
    a = make(500 * MB);   // little is left after allocations that are not this library's
    CHECK(cudaMalloc(&rest, fake::total - fake::total / 8) == cudaSuccess);
    device_release(a, clspmv::kIdleAll);
    CHECK(!fake::live(a));
    cudaFree(rest);
    a = make(500 * MB);
    device_release(a, clspmv::kIdleAll);
    CHECK(fake::live(a));
}

static void reset()   // kept arrays that a device reset took away
{
    void *a = make(MB), *b = make(3 * MB);
    device_release(a, clspmv::kIdleAll);
    device_release(b, clspmv::kIdleAll);
    fake::vanish();
    void* mine = nullptr;
    CHECK(cudaMalloc(&mine, MB) == cudaSuccess && mine == a);   // the address belongs to the caller now
    void *c = make(MB), *d = make(3 * MB);
    CHECK(c != mine && fake::live(d));
    device_release(c, clspmv::kIdleAll);
    CHECK(make(MB) == c);
    clspmv_device_trim();
    CHECK(fake::live(mine) && fake::live(c) && fake::live(d) && fake::bad_frees == 0);
}

static void freed_by_the_caller()   // an array the caller freed, whose address a later one of the caller's got
{
    void* a = make(MB);
    cudaFree(a);
    void* mine = nullptr;
    CHECK(cudaMalloc(&mine, MB) == cudaSuccess && mine == a);
    device_release(mine, clspmv::kIdleAll);   // no array of device_alloc: freed
    CHECK(!fake::live(mine));
    a = make(MB);
    device_release(a, clspmv::kIdleAll);
    cudaFree(a);
    CHECK(cudaMalloc(&mine, MB) == cudaSuccess && mine == a);
    CHECK(make(MB) != mine);
    clspmv_device_trim();
    CHECK(fake::live(mine));
}

static void waits()   // nothing is kept with work in flight; one wait for arrays released together
{
    void *a = make(MB), *b = make(MB);
    fake::working = true;
    const int idle_on = device_release(a, clspmv::kIdleNone);
    CHECK(!fake::working && fake::live(a) && idle_on == 0);
    fake::working = true;
    CHECK(device_release(b, idle_on) == 0 && fake::working && fake::live(b));
    void* c = make(MB);
    fake::vanish();   // and with it what the wait keeps
    void* mine = nullptr;
    CHECK(cudaMalloc(&mine, 512) == cudaSuccess);
    c = make(MB);
    fake::working = true;
    device_release(c, clspmv::kIdleNone);
    CHECK(!fake::working && fake::live(mine) && fake::bad_frees == 0);
    clspmv_device_trim();
    CHECK(fake::blocks().size() == 1 && fake::live(mine));
}

static void capture()   // a release while another thread captures a stream
{
    void *a = make(MB), *b = make(MB);
    fake::working = fake::capturing = true;
    device_release(a, clspmv::kIdleNone);
    CHECK(!fake::invalidated && !fake::working);
    fake::working = fake::forbidden = true;   // as cudaFree: refused, and not handed out
    device_release(b, clspmv::kIdleNone);
    fake::capturing = fake::forbidden = false;
    CHECK(make(MB) == a && make(MB) != b);
}

static void host_memory()   // no exception leaves a call, and no array is lost
{
    for (int n = 0; n < 12; n++) {
        void *a = nullptr, *b = make(3 * MB), *c = nullptr;
        bool threw = false;
        fail_new = n;
        try {
            device_alloc(&a, MB);
            device_release(b, clspmv::kIdleNone);
            device_release(a, clspmv::kIdleNone);
            device_alloc(&c, 2 * MB);
            device_release(c, clspmv::kIdleAll);
            clspmv_device_trim();
        } catch (...) {
            threw = true;
        }
        fail_new = -1;
        CHECK(!threw);
        clspmv_device_trim();
        CHECK(fake::blocks().empty());
        fake::vanish();
    }
}

static void at_exit_check() { at_exit.array = make(MB); }

int main(int argc, char** argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "reuse") reuse();
    else if (what == "bounds") bounds();
    else if (what == "low_memory") low_memory();
    else if (what == "reset") reset();
    else if (what == "freed_by_the_caller") freed_by_the_caller();
    else if (what == "waits") waits();
    else if (what == "capture") capture();
    else if (what == "host_memory") host_memory();
    else if (what == "at_exit") at_exit_check();
    else return 99;
    return failures;
}
