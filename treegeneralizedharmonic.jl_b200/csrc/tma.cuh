// Tiled tensor copies into shared memory and the mbarriers they complete on, with bounded waits.
#pragma once
#include <cuda.h>

namespace tgh {

// The tensor maps of one working array, viewed as 4-d (x, y, z, block x 20 + variable): the boxes of h and Pi
// of the TMA Pi kernel's two tile shapes, or of the tile Pi kernel's (whole).
struct PiMaps {
  CUtensorMap h, pi;
};
struct TmaMaps {
  PiMaps whole, inner;
};

struct WaitStatus {
  int* err;         // in the host's memory: TGH_ERR_TIMEOUT is stored here by a wait that gives up
  long long limit;  // polls a wait may make; for tests, negative: give up at once, -2: at a component's second box only
  __device__ __forceinline__ long long first_limit() const { return limit == -2 ? 1ll << 26 : limit; }
  __device__ __forceinline__ void gave_up() const {
    *(volatile int*)err = TGH_ERR_TIMEOUT;
    __threadfence_system();
  }
};

// a launch of one of the staged Pi kernels over the blocks [b0, b0 + nb) on a device of `sms` SMs; first: the problem's
// first launch of its form, which tells the device how much shared memory the kernel may ask for (the attribute is the
// device's, and a problem stays on one)
struct PiLaunch {
  int b0, nb, sms;
  bool first;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait on one phase of an mbarrier: false when it gave up
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, long long limit) {
  for (long long it = 0; it <= limit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load_4d(unsigned dst, const CUtensorMap* map, int x, int y, int z, int c,
                                            unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(c), "r"(bar)
      : "memory");
}

}  // namespace tgh
