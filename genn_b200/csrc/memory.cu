// See memory.h.
#include "memory.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <map>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <unordered_set>
#include <vector>

namespace b200
{
namespace
{
std::mutex g_poolMutex;
std::unordered_map<int, cudaMemPool_t> g_pools;
std::unordered_set<void*> g_direct;                 // allocations that did not come from a pool

std::mutex g_hostMutex;
std::multimap<size_t, void*> g_hostIdle;            // capacity -> block
std::unordered_map<void*, size_t> g_hostAll;        // every block and its capacity
size_t g_hostIdleBytes = 0;

size_t hostClass(size_t bytes)
{
    size_t c = 4096;
    while(c < bytes) c <<= 1;
    return c;
}

// Page-locked chunks through which a large pull passes.
constexpr size_t CHUNK = 256 * 1024;
// (40 + 20 MB into fresh pageable memory, whose page faults bound it, on 16 cores: 9.3 ms of a whole load and pull with 6
// threads, 8.3 with 8, 7.4 with 12, 7.0 with 16; populating the pages ahead with one call per chunk made it slower)
constexpr unsigned int MOST_THREADS = 16;

void store(void *host, const void *chunk, size_t count, unsigned int elemBytes, bool widen)
{
    if(!widen || elemBytes == 4u) {
        memcpy(host, chunk, count * elemBytes);
        return;
    }
    uint32_t *out = static_cast<uint32_t*>(host);
    if(elemBytes == 2u) {
        const uint16_t *in = static_cast<const uint16_t*>(chunk);
        for(size_t i = 0; i < count; i++) out[i] = in[i];
    }
    else {
        const uint8_t *in = static_cast<const uint8_t*>(chunk);
        for(size_t i = 0; i < count; i++) out[i] = in[i];
    }
}
}   // anonymous namespace

cudaError_t poolAllocBytes(void **p, size_t bytes, cudaStream_t stream)
{
    if(bytes >= POOL_MOST) {
        const cudaError_t e = cudaMalloc(p, bytes);
        if(e == cudaSuccess) {
            std::lock_guard<std::mutex> lock(g_poolMutex);
            g_direct.insert(*p);
        }
        return e;
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if(e != cudaSuccess) return e;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_poolMutex);
        cudaMemPool_t &mine = g_pools[device];
        if(!mine) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = device;
            e = cudaMemPoolCreate(&mine, &props);
            if(e != cudaSuccess) return e;
            uint64_t keep = POOL_KEEP;
            e = cudaMemPoolSetAttribute(mine, cudaMemPoolAttrReleaseThreshold, &keep);
            if(e != cudaSuccess) return e;
        }
        pool = mine;
    }
    return cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 16), pool, stream);
}

cudaError_t poolFree(void *p, cudaStream_t stream)
{
    if(!p) return cudaSuccess;
    {
        std::lock_guard<std::mutex> lock(g_poolMutex);
        if(g_direct.erase(p)) return cudaFree(p);
    }
    return cudaFreeAsync(p, stream);
}

cudaError_t hostAcquire(void **p, size_t bytes)
{
    const size_t c = hostClass(bytes);
    {
        std::lock_guard<std::mutex> lock(g_hostMutex);
        auto it = g_hostIdle.find(c);
        if(it != g_hostIdle.end()) {
            *p = it->second;
            g_hostIdle.erase(it);
            g_hostIdleBytes -= c;
            return cudaSuccess;
        }
    }
    const cudaError_t e = cudaHostAlloc(p, c, cudaHostAllocPortable);
    if(e == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_hostMutex);
        g_hostAll[*p] = c;
    }
    return e;
}

void hostRelease(void *p)
{
    if(!p) return;
    // what was used last is likeliest to be used next: it stays, and other idle blocks, the largest first, make room for it
    std::vector<void*> out;
    {
        std::lock_guard<std::mutex> lock(g_hostMutex);
        auto it = g_hostAll.find(p);
        if(it == g_hostAll.end()) return;
        const size_t c = it->second;
        while(!g_hostIdle.empty() && g_hostIdleBytes + c > HOST_KEEP) {
            auto largest = std::prev(g_hostIdle.end());
            out.push_back(largest->second);
            g_hostIdleBytes -= largest->first;
            g_hostIdle.erase(largest);
        }
        if(c <= HOST_KEEP) {
            g_hostIdle.emplace(c, p);
            g_hostIdleBytes += c;
        }
        else out.push_back(p);
        for(void *q : out) g_hostAll.erase(q);
    }
    for(void *q : out) cudaFreeHost(q);
}

cudaError_t pullLarge(void *host, const void *device, size_t count, unsigned int elemBytes, bool widen, int deviceIndex, cudaStream_t stream)
{
    const size_t perChunk = CHUNK / elemBytes, chunks = (count + perChunk - 1) / perChunk;
    // a second pull meanwhile (another model, another thread) gets chunks of its own
    const unsigned int threads = (unsigned int)std::min<size_t>(std::min(MOST_THREADS, std::max(1u, std::thread::hardware_concurrency())), (chunks + 1) / 2);
    void *staged = nullptr;
    cudaError_t e = hostAcquire(&staged, (size_t)threads * 2u * CHUNK);
    if(e != cudaSuccess) return e;
    std::atomic<int> failed{cudaSuccess};
    // every thread takes every threads-th chunk, two of them on their way
    auto work = [&](unsigned int t) {
        cudaSetDevice(deviceIndex);
        unsigned char *const buffer = static_cast<unsigned char*>(staged) + (size_t)t * 2u * CHUNK;
        cudaEvent_t arrived[2] = {nullptr, nullptr};
        auto check = [&](cudaError_t err) { if(err != cudaSuccess) failed = (int)err; };
        for(auto &ev : arrived) check(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        auto begin = [&](size_t c, unsigned int slot) {
            if(c >= chunks || failed != cudaSuccess) return;
            check(cudaMemcpyAsync(buffer + slot * CHUNK, static_cast<const unsigned char*>(device) + c * perChunk * elemBytes,
                                  std::min(perChunk, count - c * perChunk) * elemBytes, cudaMemcpyDeviceToHost, stream));
            check(cudaEventRecord(arrived[slot], stream));
        };
        begin(t, 0);
        unsigned int slot = 0;
        for(size_t c = t; c < chunks && failed == cudaSuccess; c += threads, slot ^= 1u) {
            begin(c + threads, slot ^ 1u);
            unsigned char *const to = static_cast<unsigned char*>(host) + c * perChunk * (widen ? 4u : elemBytes);
            const size_t n = std::min(perChunk, count - c * perChunk);
            check(cudaEventSynchronize(arrived[slot]));
            store(to, buffer + slot * CHUNK, n, elemBytes, widen);
        }
        for(auto ev : arrived) {
            if(ev) {
                cudaEventSynchronize(ev);
                cudaEventDestroy(ev);
            }
        }
    };
    std::vector<std::thread> helpers;
    unsigned int started = 1;
    try {
        helpers.reserve(threads);
        for(; started < threads; started++) helpers.emplace_back(work, started);
    }
    catch(const std::exception&) {}         // (no more threads to be had: this one does their part)
    work(0);
    for(unsigned int t = started; t < threads; t++) work(t);
    for(auto &h : helpers) h.join();
    hostRelease(staged);
    return (cudaError_t)failed.load();
}
}   // namespace b200
