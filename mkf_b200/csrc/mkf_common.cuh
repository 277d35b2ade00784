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

// Number of the calling thread's current CUDA context (no two contexts of a process share one, and a
// device has a new one after a reset); 0 when it is not known. What belongs to a context is kept by this.
unsigned long long contextId();

// Contexts in which a kernel's shared-memory limit was raised.
struct SmemAllowed
{
   std::atomic<unsigned long long> ctx[8] = {};
};
// Allow `kern` maxSmem bytes of dynamic shared memory in the current context; called before every launch
// that needs more than 48 KB. (Raised before each launch, not once per context, a call costs 0.5 us more:
// 64^3 FP32, one threshold 28.3 -> 28.8 us.)
template <typename K>
void allowSmem(SmemAllowed &done, K kern, size_t maxSmem)
{
   const unsigned long long id = contextId();
   std::atomic<unsigned long long> &slot = done.ctx[id % 8];
   if (id != 0 && slot.load(std::memory_order_relaxed) == id) { return; }
   if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)maxSmem) == cudaSuccess) {
      slot.store(id, std::memory_order_relaxed);
   }
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
