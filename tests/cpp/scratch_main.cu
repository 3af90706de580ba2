// scratch_main.cu -- the generic calls' pinned slots and pool
// (vsmc_b200/csrc/call_scratch.cu) over device resets: each context of the
// process gets memory of its own.
#include "../../vsmc_b200/csrc/call_scratch.hpp"

#include <cstdio>

using vsmc_b200::CallScratch;

namespace {

__global__ void k_put(int *slot, int *mem, int v)
{
    *mem = v;
    *slot = *mem + 1;
}

bool ok(cudaError_t e, const char *what)
{
    if (e != cudaSuccess)
        std::printf("%s: %s\n", what, cudaGetErrorString(e));
    return e == cudaSuccess;
}

bool call(int v)
{
    cudaStream_t s;
    if (!ok(cudaStreamCreate(&s), "stream"))
        return false;
    bool good = false;
    {
        CallScratch a(s), b(s);
        void *p = nullptr;
        if (a.slot() == nullptr || b.slot() == nullptr ||
            a.slot() == b.slot()) {
            std::printf("no slots of their own\n");
        } else if (ok(a.alloc(1 << 20, &p), "alloc")) {
            k_put<<<1, 1, 0, s>>>(static_cast<int *>(a.slot()),
                                  static_cast<int *>(p), v);
            good = ok(cudaGetLastError(), "launch") &&
                   ok(cudaStreamSynchronize(s), "synchronize") &&
                   *static_cast<int *>(a.slot()) == v + 1;
        }
    }
    return ok(cudaStreamDestroy(s), "destroy") && good;
}

} // namespace

int main()
{
    unsigned long long last = 0;
    for (int k = 0; k < 5; ++k) {
        cudaFree(nullptr);
        const unsigned long long id = vsmc_b200::context_id();
        if (id == 0 || id == last || !call(100 + k) || !call(200 + k) ||
            vsmc_b200::context_id() != id) {
            std::printf("failed after %d resets\n", k);
            return 1;
        }
        last = id;
        if (!ok(cudaDeviceReset(), "reset"))
            return 1;
    }
    std::printf("ok\n");
    return 0;
}
