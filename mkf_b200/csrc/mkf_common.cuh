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

// Resident CTAs per SM of `kern` for a block size and dynamic shared-memory size, computed on the
// first call for a cache slot and kept there (a relaxed atomic: host threads that race compute the
// same value). maxSmem > 48 KB is first allowed with cudaFuncSetAttribute.
template <typename K>
int cachedOccupancy(std::atomic<int> &slot, K kern, int threads, size_t smem, size_t maxSmem = 0)
{
   int v = slot.load(std::memory_order_relaxed);
   if (v > 0) { return v; }
   if (maxSmem > 48 * 1024) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)maxSmem); }
   int n = 0;
   cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem);
   v = n > 0 ? n : 1;
   slot.store(v, std::memory_order_relaxed);
   return v;
}
// Allow `kern` maxSmem bytes of dynamic shared memory on the current device (once per device: `done`
// has a bit for each).
template <typename K>
void allowSmem(std::atomic<uint64_t> &done, K kern, size_t maxSmem)
{
   int dev = 0;
   if (cudaGetDevice(&dev) != cudaSuccess) { return; }
   const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;
   if (done.load(std::memory_order_relaxed) & bit) { return; }
   if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)maxSmem) == cudaSuccess) {
      done.fetch_or(bit, std::memory_order_relaxed);
   }
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
