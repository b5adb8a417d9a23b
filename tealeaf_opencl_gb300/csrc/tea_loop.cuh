// Primitives of the kernels that run a whole solver loop in one cooperative
// launch (tea_cg_loop.cu, tea_mixed.cu): every block forms the reduced values
// itself from the supertile partials, so a pass costs one grid barrier.
#pragma once

#include "tea_device.cuh"

namespace tea {

// t + 0.0 without the FP64 pipe: only -0 changes (a signalling NaN, which no
// arithmetic makes, would be quieted)
__device__ __forceinline__ double plus_zero(double t) {
  const long long b = __double_as_longlong(t);
  return __longlong_as_double(b == (long long)0x8000000000000000ull ? 0 : b);
}

// Grid barrier on a counter that only grows during the launch.  Bounded: a
// block that polls spin_limit times, or sees another's error flag, sets the
// flag and returns false, and the kernel must return.
__device__ __forceinline__ bool loop_barrier(unsigned int* bar, int* err, int* timed_out,
                                             unsigned int target, long long spin_limit,
                                             int* go) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    for (long long spins = 0;;) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - target) >= 0) break;
      if (++spins > spin_limit || ((spins & 255) == 0 && *(volatile int*)err)) {
        atomicExch(err, 1);
        *timed_out = 1;
        ok = 0;
        break;
      }
    }
    *go = ok;
  }
  __syncthreads();
  return *go != 0;
}

// The reduced value (step 4 of the summation order) in lane 0 of warps 0 and
// 1 of every block.  lanes: shared memory for 256 doubles, tiles: for 8; go:
// one shared word.
__device__ __forceinline__ double loop_total(const double* partials, int ns, double* lanes,
                                             double* tiles) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kBlock) {
    double a = 0.0;
#pragma unroll 4
    for (int k = threadIdx.x; k < ns; k += kBlock) a = a + __ldcg(partials + k);
    lanes[threadIdx.x] = a;
  }
  __syncthreads();
  if (warp < 2) {
    const double* a = lanes + warp * 128 + lane;
    const double t = bfly4(a[0], a[32], a[64], a[96]);
    if ((lane & 7) == 0) tiles[warp * 4 + bfly4_slot(lane)] = t;
  }
  __syncthreads();
  double t = 0.0;
  if (warp < 2) {
    t = lane < 8 ? plus_zero(tiles[lane]) : 0.0;
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) t = t + __shfl_xor_sync(0xffffffffu, t, off);
  }
  return t;
}

}  // namespace tea
