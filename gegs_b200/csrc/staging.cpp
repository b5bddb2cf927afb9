// Pageable host memory goes through pinned buffers, a chunk at a time, by a few
// threads: each copies its chunk on the CPU while the DMA engine works on its
// previous one. The driver's own path for pageable memory is one thread's memcpy,
// and writes to memory that is touched for the first time (a result array that
// the caller has just allocated) at the speed of page faults. 31 MB, host with
// 16 threads: to the device 2.9 to 1.6 ms -> 0.96, from it 1.5 -> 0.8, from it
// into a new array 5.9 -> 1.5 (1 MB chunks, 4 threads; 8 threads and 0.5 or 2 MB
// chunks are no faster).
#include "staging.h"
#include "../../include/gegs_post.h"
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

namespace {

constexpr size_t kChunk = (size_t)1 << 20;
constexpr int kThreads = 4;
constexpr size_t kSetBytes = kChunk * 2 * kThreads;
constexpr size_t kSmall = (size_t)2 << 20;     // below, the threads cost more than they save
constexpr int kSets = 4;                       // copies that can be under way at once; a further one takes the driver's path
constexpr int kMaxDevices = 64;

// Pinned buffers kept for the next copy: at most kSets of 8 MB.
std::mutex g_mu;
char *g_free[kSets];
int g_nfree = 0, g_total = 0;

char *take_set()
{
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (g_nfree) return g_free[--g_nfree];
        if (g_total == kSets) return nullptr;
        g_total++;
    }
    void *p = nullptr;
    if (cudaHostAlloc(&p, kSetBytes, cudaHostAllocPortable) == cudaSuccess) return (char *)p;
    cudaGetLastError();
    std::lock_guard<std::mutex> lock(g_mu);
    g_total--;
    return nullptr;
}

void give_set(char *p)
{
    std::lock_guard<std::mutex> lock(g_mu);
    g_free[g_nfree++] = p;
}

bool pinned(const void *p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type != cudaMemoryTypeUnregistered;
}

struct Copy {
    char *dev, *host, *set;
    size_t bytes;
    bool in;                        // to the device
    int device;
    cudaStream_t stream;
    std::atomic<size_t> next{0};
    std::atomic<int> error{0};

    // One thread's share: chunks as they come, in two buffers by turns.
    void work(int id)
    {
        cudaError_t c = cudaSetDevice(device);
        cudaEvent_t ev[2] = {};
        for (int k = 0; k < 2 && c == cudaSuccess; k++) c = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
        char *buf[2] = {set + (size_t)(2 * id) * kChunk, set + (size_t)(2 * id + 1) * kChunk};
        size_t at[2], len[2] = {0, 0};
        for (int k = 0; c == cudaSuccess && error.load() == 0; k ^= 1) {
            if (len[k]) {           // this buffer's previous chunk
                c = cudaEventSynchronize(ev[k]);
                if (c != cudaSuccess) break;
                if (!in) memcpy(host + at[k], buf[k], len[k]);
                len[k] = 0;
            }
            const size_t o = next.fetch_add(kChunk);
            if (o >= bytes) {
                if (!len[k ^ 1]) break;
                continue;           // the other buffer's last chunk
            }
            at[k] = o;
            len[k] = bytes - o < kChunk ? bytes - o : kChunk;
            if (in) memcpy(buf[k], host + o, len[k]);
            c = in ? cudaMemcpyAsync(dev + o, buf[k], len[k], cudaMemcpyHostToDevice, stream)
                   : cudaMemcpyAsync(buf[k], dev + o, len[k], cudaMemcpyDeviceToHost, stream);
            if (c == cudaSuccess) c = cudaEventRecord(ev[k], stream);
        }
        if (c != cudaSuccess || len[0] || len[1]) cudaStreamSynchronize(stream);   // after an error: nothing in flight on the buffers
        for (int k = 0; k < 2; k++)
            if (ev[k]) cudaEventDestroy(ev[k]);
        if (c != cudaSuccess) error.store((int)c);
    }
};

cudaError_t staged(char *dev, char *host, size_t bytes, bool in, cudaStream_t s)
{
    char *set = bytes < kSmall || pinned(host) ? nullptr : take_set();
    if (!set) {
        cudaError_t c = in ? cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s)
                           : cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s);
        return c == cudaSuccess ? cudaStreamSynchronize(s) : c;
    }
    Copy c;
    c.dev = dev; c.host = host; c.set = set; c.bytes = bytes; c.in = in; c.stream = s;
    cudaGetDevice(&c.device);
    std::thread t[kThreads - 1];
    int n = 0;
    try {
        for (; n < kThreads - 1; n++) t[n] = std::thread([&c, n] { c.work(n + 1); });
    } catch (const std::exception &) {
        // fewer threads, then
    }
    c.work(0);
    for (int k = 0; k < n; k++) t[k].join();
    give_set(set);
    return (cudaError_t)c.error.load();
}

cudaMemPool_t g_pool[kMaxDevices];

}  // namespace

cudaError_t staged_to_device(void *dst, const void *src, size_t bytes, cudaStream_t s)
{
    return staged((char *)dst, (char *)const_cast<void *>(src), bytes, true, s);
}

cudaError_t staged_to_host(void *dst, const void *src, size_t bytes, cudaStream_t s)
{
    return staged((char *)const_cast<void *>(src), (char *)dst, bytes, false, s);
}

cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s)
{
    int device = 0;
    cudaError_t c = cudaGetDevice(&device);
    if (c != cudaSuccess) return c;
    if (device < 0 || device >= kMaxDevices) return cudaMallocAsync(p, bytes, s);
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (!g_pool[device]) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = device;
            c = cudaMemPoolCreate(&g_pool[device], &props);
            if (c != cudaSuccess) { g_pool[device] = nullptr; return c; }
            uint64_t keep = kScratchKept;
            cudaMemPoolSetAttribute(g_pool[device], cudaMemPoolAttrReleaseThreshold, &keep);
        }
        pool = g_pool[device];
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

extern "C" void gegs_trim(void)
{
    std::lock_guard<std::mutex> lock(g_mu);
    while (g_nfree) {
        cudaFreeHost(g_free[--g_nfree]);
        g_total--;
    }
    for (int d = 0; d < kMaxDevices; d++)
        if (g_pool[d]) cudaMemPoolTrimTo(g_pool[d], 0);
}
