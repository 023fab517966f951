// device_pool.cu — device arrays of the converters and uploads, with a
// bounded list of freed ones kept for the next call.
//
// Mapping and unmapping device memory costs far more than converting into
// it: on B200, cudaMalloc / cudaFree of an array that needs pages of its own
// take 350 / 300 us up to 64 MB and 0.7 / 1.1 ms at 1 GB, and a conversion
// makes three arrays and drops the last result's three. A freed array is
// therefore kept, and handed to the next request that it fits: the 4x4 SBELL
// of 64M entries (0.43 ms of kernels) converts in 0.52 instead of 5.5 ms, the
// SELL-32 of the power-law matrix of 700k rows in 0.41 instead of 4.0 ms.
//
// A kept array has no work pending on it: device_release waits for the
// device first, by what cudaFree waits with (wait_as_free_does), so it may be
// used on any stream by any thread. The list holds at most 1/64 of a device's
// memory (2.9 GB of 183 GB) in kKeptMost arrays, the oldest leaving first. It
// is given back when an allocation fails, when less than 1/8 of the device is
// left after a large new one or once the list has grown by kLarge since the
// last look (asking the driver takes 0.1 to 0.3 ms), and by clspmv_device_trim.
//
// Only arrays that device_alloc made are kept; any other pointer goes to
// cudaFree. An array is known by the driver's id of its allocation, which no
// other one of the process gets: one that the caller freed, or that a device
// reset took away, is neither handed out nor freed again, whoever owns its
// address by then.
#include <cuda.h>
#include <algorithm>
#include <list>
#include <mutex>
#include <unordered_map>
#include "api_internal.h"
#include "clspmv_b200.h"

namespace clspmv {
namespace {

struct Kept {
    void* p;
    size_t bytes;
    int device;
    unsigned long long id;
};
struct Made {
    size_t bytes;
    unsigned long long id;
};

// Never destroyed: a matrix may be released by a destructor that runs after this file's would have.
std::mutex& g_mu = *new std::mutex;
std::list<Kept>& g_kept = *new std::list<Kept>;      // oldest first
std::list<Kept>& g_marker = *new std::list<Kept>;    // wait_as_free_does, one per device
auto& g_kept_bytes = *new std::unordered_map<int, size_t>;   // per device
auto& g_made = *new std::unordered_map<void*, Made>;         // arrays made by device_alloc and not yet cudaFree'd
auto& g_seen = *new std::unordered_map<int, size_t>;         // bytes kept when the device's free memory was last looked at
auto& g_limit = *new std::unordered_map<int, size_t>;        // limit_of, per device

constexpr size_t kGrain = 512;
constexpr size_t kLarge = 64u << 20;
constexpr size_t kKeptMost = 256;   // arrays on the list, so that a search stays short

size_t limit_of(int device)
{
    std::lock_guard<std::mutex> lock(g_mu);
    auto it = g_limit.find(device);
    if (it != g_limit.end()) return it->second;
    size_t fr = 0, total = 0;
    int cur = -1;
    cudaGetDevice(&cur);
    if (cur != device) cudaSetDevice(device);
    if (cudaMemGetInfo(&fr, &total) != cudaSuccess) {
        cudaGetLastError();
        total = 0;
    }
    if (cur >= 0 && cur != device) cudaSetDevice(cur);
    return g_limit[device] = total / 64;
}

// The driver's id of the allocation at p, 0 if there is none (0.14 us).
unsigned long long allocation_id(void* p)
{
    typedef CUresult (*Attribute)(void*, CUpointer_attribute, CUdeviceptr);
    static const Attribute attribute = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            fn = nullptr;
        }
        return reinterpret_cast<Attribute>(fn);
    }();
    unsigned long long id = 0;
    if (!attribute || attribute(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS) return 0;
    return id;
}

bool alive(const Kept& k) { return allocation_id(k.p) == k.id; }

// Moves an entry from the list to `out` (g_mu held); returns the next one. Allocates nothing.
std::list<Kept>::iterator unlist(std::list<Kept>::iterator it, std::list<Kept>& out)
{
    auto held = g_kept_bytes.find(it->device);
    if (held != g_kept_bytes.end()) held->second -= it->bytes;
    auto next = std::next(it);
    out.splice(out.end(), g_kept, it);
    return next;
}
// ... and off the arrays made.
std::list<Kept>::iterator forget(std::list<Kept>::iterator it, std::list<Kept>& out)
{
    auto made = g_made.find(it->p);
    if (made != g_made.end() && made->second.id == it->id) g_made.erase(made);
    return unlist(it, out);
}

// Takes the kept arrays of `device` (all devices: -1) off the list.
std::list<Kept> take_kept(int device)
{
    std::list<Kept> out;
    std::lock_guard<std::mutex> lock(g_mu);
    for (auto it = g_kept.begin(); it != g_kept.end();)
        it = device < 0 || it->device == device ? forget(it, out) : std::next(it);
    for (auto it = g_marker.begin(); it != g_marker.end();) {
        auto next = std::next(it);
        if (device < 0 || it->device == device) out.splice(out.end(), g_marker, it);
        it = next;
    }
    for (auto& seen : g_seen)
        if (device < 0 || seen.first == device) seen.second = 0;
    return out;
}

void free_all(const std::list<Kept>& l)
{
    for (const Kept& k : l)
        if (k.p && alive(k) && cudaFree(k.p) != cudaSuccess) cudaGetLastError();
}

// Waits for all work of the current device by freeing a small allocation:
// cudaFree waits for it, and is allowed where another thread captures a
// stream in its own (thread-local) mode, or any thread in relaxed mode.
// cudaDeviceSynchronize, the cheaper wait (1.8 against 4 us on B200), fails
// there and spoils the capture. Another small allocation is made first, so
// that their page of the device stays mapped.
bool wait_as_free_does(int device)
{
    auto marker_of = [&]() -> Kept& {   // g_mu held
        for (Kept& k : g_marker)
            if (k.device == device) return k;
        g_marker.push_back(Kept{nullptr, kGrain, device, 0});
        return g_marker.back();
    };
    {
        std::lock_guard<std::mutex> lock(g_mu);
        marker_of();
    }
    Kept last, next{nullptr, kGrain, device, 0};
    if (cudaMalloc(&next.p, kGrain) != cudaSuccess) return false;
    next.id = allocation_id(next.p);
    {
        std::lock_guard<std::mutex> lock(g_mu);
        Kept& m = marker_of();
        last = m;
        m = next;
    }
    if ((!last.p || !alive(last)) && cudaMalloc(&last.p, kGrain) != cudaSuccess) return false;
    return cudaFree(last.p) == cudaSuccess;
}

// Gives the kept arrays of the current device back when less than 1/8 of it is left.
void give_back_if_short(int device)
{
    size_t fr = 0, total = 0;
    if (cudaMemGetInfo(&fr, &total) == cudaSuccess && fr < total / 8) free_all(take_kept(device));
}

// Puts an array on the list; false where it has to be freed instead.
bool keep_array(void* p, int* idle_on)
{
    const unsigned long long id = allocation_id(p);
    size_t bytes = 0;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        for (const Kept& k : g_kept)
            if (k.p == p && k.id == id) return true;   // released already
        auto it = g_made.find(p);
        if (id && it != g_made.end() && it->second.id == id) bytes = it->second.bytes;
    }
    cudaPointerAttributes at{};
    if (!bytes || cudaPointerGetAttributes(&at, p) != cudaSuccess || at.type != cudaMemoryTypeDevice) return false;
    const size_t limit = limit_of(at.device);
    if (bytes > limit) return false;
    if (*idle_on != kIdleAll && *idle_on != at.device) {
        int cur = -1;
        cudaGetDevice(&cur);
        if (cur != at.device) cudaSetDevice(at.device);
        const bool idle = wait_as_free_does(at.device);
        if (cur >= 0 && cur != at.device) cudaSetDevice(cur);
        if (!idle) return false;
        *idle_on = at.device;
    }
    std::list<Kept> drop, gone;
    bool look = false;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        size_t& seen = g_seen[at.device];
        for (auto it = g_kept.begin(); it != g_kept.end();) {
            if (it->p == p && it->id == id) return true;
            it = it->p == p ? forget(it, gone) : std::next(it);   // gone: its address is this one's
        }
        size_t& held = g_kept_bytes[at.device];
        g_kept.push_back(Kept{p, bytes, at.device, id});
        held += bytes;
        for (auto it = g_kept.begin(); (held > limit || g_kept.size() > kKeptMost) && it != g_kept.end();)
            it = it->device == at.device ? forget(it, drop) : std::next(it);
        look = held >= seen + kLarge;
        if (look) seen = held;
    }
    free_all(drop);
    if (look) {
        int cur = -1;
        cudaGetDevice(&cur);
        if (cur != at.device) cudaSetDevice(at.device);
        give_back_if_short(at.device);
        if (cur >= 0 && cur != at.device) cudaSetDevice(cur);
    }
    return true;
}

}  // namespace

int device_alloc(void** out, size_t bytes)
{
    *out = nullptr;
    bytes = (std::max<size_t>(bytes, 1) + kGrain - 1) / kGrain * kGrain;
    int device = 0;
    cudaGetDevice(&device);
    {
        // the smallest kept array that holds the request and is at most 1/8 larger
        std::list<Kept> gone;
        std::lock_guard<std::mutex> lock(g_mu);
        const size_t most = bytes + bytes / 8 + kGrain;
        while (true) {
            auto best = g_kept.end();
            for (auto it = g_kept.begin(); it != g_kept.end(); ++it)
                if (it->device == device && it->bytes >= bytes && it->bytes <= most && (best == g_kept.end() || it->bytes < best->bytes))
                    best = it;
            if (best == g_kept.end()) break;
            if (alive(*best)) {
                *out = best->p;
                unlist(best, gone);
                return CLSPMV_OK;
            }
            forget(best, gone);
        }
    }
    void* p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        free_all(take_kept(device));
        if (cudaMalloc(&p, bytes) != cudaSuccess) {
            cudaGetLastError();
            return CLSPMV_ERR_ALLOC;
        }
    }
    try {
        const Made made{bytes, allocation_id(p)};
        std::lock_guard<std::mutex> lock(g_mu);
        g_made[p] = made;
    } catch (...) {   // the host is out of memory
        if (cudaFree(p) != cudaSuccess) cudaGetLastError();
        return CLSPMV_ERR_ALLOC;
    }
    if (bytes >= kLarge) give_back_if_short(device);
    *out = p;
    return CLSPMV_OK;
}

int device_release(void* p, int idle_on)
{
    if (!p) return idle_on;
    try {
        if (keep_array(p, &idle_on)) return idle_on;
    } catch (...) {   // the host is out of memory
    }
    cudaGetLastError();
    {
        std::lock_guard<std::mutex> lock(g_mu);
        g_made.erase(p);
    }
    if (cudaFree(p) != cudaSuccess) cudaGetLastError();
    return idle_on;
}

}  // namespace clspmv

extern "C" int clspmv_device_trim(void)
{
    clspmv::free_all(clspmv::take_kept(-1));
    return CLSPMV_OK;
}
