// Loads of what a kernel before may have written, in kernels started by launch_chained (runtime.hpp).
#pragma once

namespace mpsg {

// An ordinary load (not the read-only path), after the wait for the kernel before: volatile, so it stays
// behind that wait, and without a memory clobber, so it may pass the kernel's own stores, which never
// go to its operands (a plain C++ load waits for every earlier store to shared memory: with it, the packing
// of a chi = 517 two-site H_eff makes the whole 3 us slower, 92.7 instead of 89.6).
__device__ __forceinline__ double load_dep(const double* p) {
  double x;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(x) : "l"(p));
  return x;
}

}  // namespace mpsg
