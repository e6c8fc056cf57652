// Launches that run ahead of the host (the hierarchy builders' rounds and levels): each
// launch writes three ints and then its number to a slot of mapped pinned memory
// (ring_publish), and the host polls for the number up to kAhead launches later instead of
// waiting after every launch.  The launches overlap their start with the end of the one
// before (programmatic dependent launch): a kernel calls ring_wait before it reads what the
// one before wrote.  No events lie between them, which would end that overlap.
#pragma once
#include <atomic>

#include "eos_internal.cuh"

namespace eos {

// Waits for the launch before this one, then lets the next one start its blocks.
__device__ __forceinline__ void ring_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void ring_publish(int* slot, int a, int b, int c, int number) {
  volatile int* s = slot;
  s[0] = a;
  s[1] = b;
  s[2] = c;
  __threadfence_system();
  s[3] = number;
}

struct RoundRing {
  // Two launches in flight keep the device busy; more run on past the last round or level
  // (builds of 20k and 1.06M triangles 530 and 1,118 us with four, 516 and 1,087 with two).
  static constexpr int kAhead = eos_ctx::kRingSlots;
  eos_ctx* ctx;
  long long issued = 0, done = 0;
  explicit RoundRing(eos_ctx* c) : ctx(c) {}
  eos_status init() {
    EOS_TRY(host_words(ctx));
    // launch numbers go on from sequence to sequence: a late write of an earlier sequence's
    // launch past its end is never taken for one of this
    base = ctx->ring_next;
    return EOS_OK;
  }
  bool full() const { return issued - done == kAhead; }
  bool empty() const { return issued == done; }
  int* next_slot() const { return ctx->ring_dev + 4 * (int)((base + issued) % kAhead); }
  int next_number() const { return (int)((base + issued) & 0x7fffffff); }
  // The next launch of `kernel`, whose arguments take next_slot() and next_number().
  template <class... P, class... A>
  eos_status launch(void (*kernel)(P...), int grid, int block, A... args) {
    cudaLaunchAttribute overlap;
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = ctx->stream;
    cfg.attrs = &overlap;
    cfg.numAttrs = 1;
    EOS_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
    ++issued;
    ctx->ring_next = base + issued;
    return EOS_OK;
  }
  // The oldest unread launch's three ints.  When it does not publish (it gave up and set its
  // error bit, or the device failed) the stream runs empty, which ends the wait.
  eos_status read(int* out) {
    const volatile int* s = ctx->ring_host + 4 * (int)((base + done) % kAhead);
    const int number = (int)((base + done) & 0x7fffffff);
    for (int polls = 1; s[3] != number; ++polls) {
      if (polls % 4096) continue;
      const cudaError_t e = cudaStreamQuery(ctx->stream);
      if (e == cudaErrorNotReady) continue;
      EOS_CUDA(e);
      if (s[3] != number) return EOS_ERR_TIMEOUT;
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    for (int k = 0; k < 3; ++k) out[k] = s[k];
    ++done;
    return EOS_OK;
  }

 private:
  long long base = 0;
};

}  // namespace eos
