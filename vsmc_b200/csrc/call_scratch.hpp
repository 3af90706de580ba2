// call_scratch.hpp -- memory for the generic entry points' calls: a small
// pinned host slot a kernel or copy puts the call's result in, and scratch
// device memory ordered on the caller's stream.
//
// cudaMallocAsync on the device's default pool gives freed memory back to
// the system at every synchronisation (its release threshold is 0), so a
// call that allocates, runs and waits paid for mapping and unmapping pages
// each time: 0.5 to 3 ms a call.  The library's own pool keeps up to
// kPoolKeep bytes.  Both are held per device and context (a handful),
// created at the first call; every call works without them too.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace vsmc_b200 {

// The current context's id, which no other context of the process ever has
// (a handle may come back: cudaDeviceReset ends a context and its memory, and
// the device's next one can stand at the same address); 0: none is current.
unsigned long long context_id();

constexpr size_t kSlotBytes = 256;
constexpr size_t kPoolKeep = 32u << 20;

// A call's resources; released by the destructor (the scratch on `s`).  The
// slot goes to another call then, so the destructor first waits for what the
// stream may still write there, unless the call has waited itself.
class CallScratch {
  public:
    explicit CallScratch(cudaStream_t s);
    ~CallScratch();
    CallScratch(const CallScratch &) = delete;
    CallScratch &operator=(const CallScratch &) = delete;

    // Pinned host memory of kSlotBytes that device code can write, or
    // nullptr (none free, or `s` is being captured): then results go through
    // device memory.
    void *slot() const { return slot_; }
    // The stream has been waited for since the slot's last use.
    void waited() { waited_ = true; }
    // `bytes` of device memory (once per call).
    cudaError_t alloc(size_t bytes, void **p);

  private:
    cudaStream_t s_;
    int entry_;
    int index_;
    bool waited_;
    void *slot_;
    void *mem_;
};

} // namespace vsmc_b200
