// Read-back of launches that run ahead of the host: each launch writes four ints to a slot
// of mapped pinned memory (the last one its number), and the host reads slot k once the
// event behind that launch has passed, up to kAhead launches later, instead of waiting
// after every launch.
#pragma once
#include "eos_internal.cuh"

namespace eos {

struct RoundRing {
  static constexpr int kAhead = 4;
  eos_ctx* ctx;
  int ahead;
  long long issued = 0, done = 0;
  explicit RoundRing(eos_ctx* c, int n = kAhead) : ctx(c), ahead(n) {}
  eos_status init() {
    static_assert(kAhead <= (int)(sizeof(ctx->ring_ev) / sizeof(ctx->ring_ev[0])), "one event per slot");
    if (!ctx->ring_host) {
      if (cudaHostAlloc(&ctx->ring_host, 16 * kAhead, cudaHostAllocMapped) != cudaSuccess ||
          cudaHostGetDevicePointer(&ctx->ring_dev, ctx->ring_host, 0) != cudaSuccess) {
        cudaGetLastError();
        if (ctx->ring_host) cudaFreeHost(ctx->ring_host);
        ctx->ring_host = ctx->ring_dev = nullptr;
        return EOS_ERR_OOM;
      }
    }
    for (int k = 0; k < 4 * kAhead; ++k) ctx->ring_host[k] = -1;
    for (cudaEvent_t& e : ctx->ring_ev)
      if (!e) EOS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return EOS_OK;
  }
  int* next_slot() const { return ctx->ring_dev + 4 * (int)(issued % kAhead); }
  bool full() const { return issued - done == ahead; }
  bool empty() const { return issued == done; }
  // After a launch that writes next_slot().
  eos_status launched() {
    EOS_CUDA(cudaGetLastError());
    EOS_CUDA(cudaEventRecord(ctx->ring_ev[issued % kAhead], ctx->stream));
    ++issued;
    return EOS_OK;
  }
  // The oldest unread launch's first three ints.
  eos_status read(int* out) {
    const int slot = (int)(done % kAhead);
    EOS_CUDA(cudaEventSynchronize(ctx->ring_ev[slot]));
    const volatile int* s = ctx->ring_host + 4 * slot;
    if (s[3] != (int)done) return EOS_ERR_TIMEOUT;  // the launch gave up (its error bit is set)
    for (int k = 0; k < 3; ++k) out[k] = s[k];
    ++done;
    return EOS_OK;
  }
};

}  // namespace eos
