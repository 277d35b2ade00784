// mkf_common.cuh - shared host/device helpers of libMKF.so (sm_100a).
#pragma once
#include <atomic>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include "mkf_types.h"
#include "mkf_b200.h"

#define MKF_API extern "C" __attribute__((visibility("default")))

namespace mkf {

// Thread-local last error text (mkfLastError).
void setError(const char *fmt, ...);
// Record a CUDA error as the last error; returns MKF_ERR_CUDA when e != cudaSuccess.
int cudaFail(cudaError_t e, const char *what);
int smCount();

// Allow `kern` maxSmem bytes of dynamic shared memory on the current device; called before every launch
// that needs more than 48 KB. The limit belongs to the kernel on one device and goes with a reset of that
// device, so nothing here remembers that it was set (0.13 us a call).
template <typename K>
void allowSmem(K kern, size_t maxSmem)
{
   cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)maxSmem);
}
// Resident CTAs per SM of `kern` for a block size and dynamic shared-memory size (allowSmem beforehand
// above 48 KB), computed on the first call for a cache slot and kept there (a relaxed atomic: host
// threads that race compute the same value).
template <typename K>
int cachedOccupancy(std::atomic<int> &slot, K kern, int threads, size_t smem)
{
   int v = slot.load(std::memory_order_relaxed);
   if (v > 0) { return v; }
   int n = 0;
   cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem);
   v = n > 0 ? n : 1;
   slot.store(v, std::memory_order_relaxed);
   return v;
}
// Log a message on stderr the way the original library reports CUDA failures (ctuErr).
void logError(const char *fmt, ...);

static constexpr unsigned FULL = 0xFFFFFFFFu;

// Relation index of f to t as the original computes it (binMapCUDA.cuh:141-145):
// 0 below, 1 equal or unordered, 2 above.
template <typename T>
__device__ __forceinline__ unsigned relIdx(T f, T t) { return 1u - (f < t) + (f > t); }

// Bits [0, r) set, r in [0, 32]: the upper word of (0 : 0xFFFFFFFF) << min(r, 32).
__device__ __forceinline__ uint32_t thermo(uint32_t r) { return __funnelshift_lc(0xFFFFFFFFu, 0u, r); }

}  // namespace mkf
