// call_scratch.cu -- see call_scratch.hpp.
#include "call_scratch.hpp"

#include <cstdint>
#include <cstring>
#include <mutex>

namespace vsmc_b200 {

namespace {

constexpr int kEntries = 16; // (device, context) pairs served
constexpr int kSlots = 64;   // calls in flight per pair

struct Entry {
    int dev;
    unsigned long long id; // its context
    char *host;
    uint64_t used;
    cudaMemPool_t pool;
    bool has_pool;
};

std::mutex g_mutex;
Entry g_entries[kEntries];
int g_n = 0;

template <typename F>
F driver_function(const char *name)
{
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
        p = nullptr;
    return reinterpret_cast<F>(p);
}

// The entry of the current device and context, or -1.  Called with the
// mutex held.  A stream that is being captured gets none (creating it would
// end the capture, and its work runs when the call is over).
int find_entry(cudaStream_t s, unsigned long long id)
{
    int dev = 0;
    if (id == 0 || cudaGetDevice(&dev) != cudaSuccess)
        return -1;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    if (st != cudaStreamCaptureStatusNone)
        return -1;
    for (int k = 0; k < g_n; ++k)
        if (g_entries[k].dev == dev && g_entries[k].id == id)
            return k;
    if (g_n == kEntries)
        return -1;
    Entry e;
    std::memset(&e, 0, sizeof(e));
    e.dev = dev;
    e.id = id;
    void *h = nullptr;
    if (cudaHostAlloc(&h, kSlots * kSlotBytes,
                      cudaHostAllocPortable | cudaHostAllocMapped) !=
        cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    e.host = static_cast<char *>(h);
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    if (cudaMemPoolCreate(&e.pool, &props) == cudaSuccess) {
        uint64_t keep = kPoolKeep;
        cudaMemPoolSetAttribute(e.pool, cudaMemPoolAttrReleaseThreshold,
                                &keep);
        e.has_pool = true;
    } else {
        cudaGetLastError();
    }
    g_entries[g_n] = e;
    return g_n++;
}

} // namespace

unsigned long long context_id()
{
    typedef int (*GetCurrent)(void **);
    typedef int (*GetId)(void *, unsigned long long *);
    static const GetCurrent current =
        driver_function<GetCurrent>("cuCtxGetCurrent");
    static const GetId id_of = driver_function<GetId>("cuCtxGetId");
    void *ctx = nullptr;
    unsigned long long id = 0;
    if (current == nullptr || id_of == nullptr || current(&ctx) != 0 ||
        ctx == nullptr || id_of(ctx, &id) != 0)
        return 0;
    return id;
}

CallScratch::CallScratch(cudaStream_t s)
    : s_(s), entry_(-1), index_(-1), waited_(false), slot_(nullptr),
      mem_(nullptr)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    entry_ = find_entry(s, context_id());
    if (entry_ < 0)
        return;
    Entry &e = g_entries[entry_];
    for (int k = 0; k < kSlots; ++k)
        if (!((e.used >> k) & 1u)) {
            e.used |= uint64_t(1) << k;
            index_ = k;
            slot_ = e.host + k * kSlotBytes;
            break;
        }
}

CallScratch::~CallScratch()
{
    if (mem_ != nullptr)
        cudaFreeAsync(mem_, s_);
    if (index_ >= 0) {
        // (a call that failed after its launches; a stream that cannot be
        // waited for keeps the slot)
        if (!waited_ && cudaStreamSynchronize(s_) != cudaSuccess)
            return;
        std::lock_guard<std::mutex> lock(g_mutex);
        g_entries[entry_].used &= ~(uint64_t(1) << index_);
    }
}

cudaError_t CallScratch::alloc(size_t bytes, void **p)
{
    cudaError_t e =
        entry_ >= 0 && g_entries[entry_].has_pool
            ? cudaMallocFromPoolAsync(&mem_, bytes, g_entries[entry_].pool, s_)
            : cudaMallocAsync(&mem_, bytes, s_);
    if (e != cudaSuccess)
        mem_ = nullptr;
    *p = mem_;
    return e;
}

} // namespace vsmc_b200
