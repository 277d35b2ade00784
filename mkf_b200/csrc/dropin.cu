// dropin.cu - the original MKF GPU entry points, re-implemented for sm_100a.
//
//   binMapCUDA            replaces binMapCUDA.cu:144-264 (kernels binMapCUDA.cuh:282-338)
//   binMapCUDACleanup     replaces binMapCUDA.cu:266-270
//   mkfCUDAGetBPFD        replaces mkfCUDA.cu:12-61 (kernels bpfdCUDA.cuh:92-206)
//   mkfCUDAGetBPFDH       replaces mkfCUDA.cu:72-91
//   mkfCUDACleanup        replaces mkfCUDA.cu:93-99 (never resets the device)
//   mkfCUDAGetBPFDautoCtx replaces mkfCUDA.cu:101-167
//
// Behaviour kept from the original: argument meaning, the packed-map layout, unit dimensions
// dropped before the layout is set (copyNonZeroDef), several enabled fields summed element-wise
// in the field's own precision, FP32 fields compared with the threshold rounded to float, the
// counts accumulating into the caller's array, NULL returns on error, synchronous calls.
// Behaviour that differs (each is undefined or wrong in the original):
//   * FP64 fields are compared in FP64 on every path (the original reads them as float when the
//     row length is not a multiple of 32, when strided, or when several fields are summed);
//   * any row length works (the original's strided kernel shuffles across exited lanes);
//   * padding bits past the row end are written as 0;
//   * rows shorter than 32 elements contribute X-1 cells (the original counts 2X-1).
#include <cstdio>
#include <cstring>
#include <mutex>
#include "mkf_common.cuh"
#include "binMapCUDA.h"
#include "mkfCUDA.h"

namespace mkf {

struct PackArgs
{
   const void *f[BMCU_FIELD_MAX];
   int nF;
   int64_t sx, sy, sz;
   int X, Y, Z;            // region mapped
   uint32_t rowWS, planeWS;
   double t;
   uint32_t m;
   uint32_t *w;
   long long nWords;       // rowWS * Y * Z
};

// One warp per row (y, z) of the map: lane j thresholds element x = 32 w + j (the sum of the
// fields) of word w, U words per step with all their loads issued before the first ballot (U = 8:
// a 256-element row in one step, 1-2 KB in flight per warp), and a ballot assembles each word;
// lanes 0..U-1 store the step's words. Loads are coalesced along x for planar fields; elements
// past the row end are not read (their bits are 0).
template <typename T, int U>
__global__ void __launch_bounds__(256) packMap(const __grid_constant__ PackArgs a)
{
   const int lane = threadIdx.x & 31;
   const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
   const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
   const long long nRows = (long long)a.Y * a.Z;
   const T t = (T)a.t;
   const T *f0 = (const T *)a.f[0];
   for (long long row = gw; row < nRows; row += nw) {
      const uint32_t r32 = (uint32_t)row;  // rows fit 32 bits (checked at launch)
      const int z = (int)(r32 / (uint32_t)a.Y);
      const int y = (int)(r32 - (uint32_t)z * (uint32_t)a.Y);
      const long long base = (long long)y * a.sy + (long long)z * a.sz;
      uint32_t *wrow = a.w + (size_t)z * a.planeWS + (size_t)y * a.rowWS;
      for (int w0 = 0; w0 < (int)a.rowWS; w0 += U) {
         T v[U];
         bool in[U];
#pragma unroll
         for (int u = 0; u < U; u++) {
            const int x = 32 * (w0 + u) + lane;
            in[u] = x < a.X;
            v[u] = in[u] ? __ldg(f0 + base + (long long)x * a.sx) : T(0);
         }
         for (int k = 1; k < a.nF; k++) {
#pragma unroll
            for (int u = 0; u < U; u++) {
               const int x = 32 * (w0 + u) + lane;
               if (in[u]) { v[u] += __ldg((const T *)a.f[k] + base + (long long)x * a.sx); }
            }
         }
         uint32_t mine = 0;
#pragma unroll
         for (int u = 0; u < U; u++) {
            const uint32_t word = __ballot_sync(FULL, in[u] ? (a.m >> relIdx(v[u], t)) & 1u : 0u);
            mine = (lane == u) ? word : mine;
         }
         if (lane < U && w0 + lane < (int)a.rowWS) { wrow[w0 + lane] = mine; }
      }
   }
}

// One planar field whose rows are whole words (X a multiple of 32): map word i is elements
// 32 i .. 32 i + 31 of the field, so the map is a flat pass with no row arithmetic. A warp takes
// kPackWords consecutive words per step: lane j loads element j of each (coalesced loads in
// flight), one ballot per word, and lane i stores word i of the step. The grid is the resident
// CTAs only, each warp looping over steps (measured on the 256^3 FP32 ball, events around the
// call: 16 words per step on a resident grid 21.0-21.2 us, 32 words per step on 8 CTAs per SM
// 23.0 us).
static constexpr int kPackWords = 16;
template <typename T, int U = kPackWords>
__global__ void __launch_bounds__(256) packFlat(const __grid_constant__ PackArgs a)
{
   const int lane = threadIdx.x & 31;
   const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
   const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
   const T t = (T)a.t;
   const T *__restrict__ f0 = (const T *)a.f[0];
   for (long long w0 = gw * U; w0 < a.nWords; w0 += nw * U) {
      const int n = (int)min((long long)U, a.nWords - w0);
      const T *p = f0 + w0 * 32 + lane;
      T v[U];
#pragma unroll
      for (int u = 0; u < U; u++) { v[u] = u < n ? __ldg(p + 32 * u) : T(0); }
      uint32_t mine = 0;
#pragma unroll
      for (int u = 0; u < U; u++) {
         const uint32_t word = __ballot_sync(FULL, (a.m >> relIdx(v[u], t)) & 1u);
         mine = (lane == u) ? word : mine;
      }
      if (lane < n) { a.w[w0 + lane] = mine; }
   }
}

template <typename T>
static void launchPack(const PackArgs &a, long long grid)
{
   if (a.nF == 1 && a.sx == 1 && a.sy == a.X && a.sz == (int64_t)a.X * a.Y && (int64_t)a.rowWS * 32 == a.X &&
       (int64_t)a.planeWS == (int64_t)a.rowWS * a.Y) {
      long long g = (a.nWords + kPackWords * 8 - 1) / (kPackWords * 8);  // 8 warps of kPackWords words per CTA
      static std::atomic<int> occ{0};
      const long long cap = (long long)smCount() * cachedOccupancy(occ, packFlat<T>, 256, 0);
      if (g > cap) { g = cap; }
      packFlat<T><<<(unsigned)(g < 1 ? 1 : g), 256>>>(a);
      return;
   }
   // words per step: as many as a row has, up to 8
   if (a.rowWS >= 8) { packMap<T, 8><<<(unsigned)grid, 256>>>(a); }
   else if (a.rowWS >= 4) { packMap<T, 4><<<(unsigned)grid, 256>>>(a); }
   else if (a.rowWS >= 2) { packMap<T, 2><<<(unsigned)grid, 256>>>(a); }
   else { packMap<T, 1><<<(unsigned)grid, 256>>>(a); }
}

struct CountArgs
{
   const uint32_t *w;
   int X;                  // elements per row
   int rows, planes;       // row pairs + 1, plane pairs + 1
   uint32_t rowWS, planeWS;
   long long nItems;       // rowWS * (rows-1) * runs of kCountZ plane pairs
   unsigned long long *out;
};

// Packed map -> 256 counts. Each thread takes 32 cells of one row pair in kCountZ plane pairs, all of
// its map words loaded before the first is used (the kernel is bound by the latency of these loads:
// one plane pair at a time, four in turn per thread, took 11.9 us for the 256^3 map under ncu, this
// 9.5). A cell's corners are bits b and b + 1 of four words; uniform cells (all corners equal) are
// counted by popcount; only mixed cells form their 8-bit code, counted in a per-warp shared histogram.
static constexpr int kCountZ = 4;
template <typename I>
__global__ void __launch_bounds__(256) countMap(const __grid_constant__ CountArgs a)
{
   __shared__ uint32_t sh[8][256];
   __shared__ unsigned long long sEnds[2];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) { (&sh[0][0])[i] = 0; }
   if (threadIdx.x < 2) { sEnds[threadIdx.x] = 0; }
   __syncthreads();
   uint32_t *h = sh[warp];
   unsigned long long n0 = 0, n255 = 0;
   // (I: 32-bit index arithmetic when every item index fits, else 64-bit)
   const I stride = (I)gridDim.x * blockDim.x, rowWS = (I)a.rowWS, rowPairs = (I)(a.rows - 1);
   for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < (I)a.nItems; i += stride) {
      const I rp = i / rowWS;
      const int wi = (int)(i - rp * rowWS);
      const I zq = rp / rowPairs;
      const int y = (int)(rp - zq * rowPairs);
      const int z = (int)zq * kCountZ, nZ = min(kCountZ, a.planes - 1 - z);
      const int nValid = min(32, a.X - 1 - 32 * wi);
      if (nValid <= 0) { continue; }
      const uint32_t vmask = (nValid >= 32) ? 0xFFFFFFFFu : ((1u << nValid) - 1u);
      const bool nx = (wi + 1) < (int)a.rowWS;
      // per plane: the two rows' words and the words after them (bit 0 is used)
      uint32_t w[kCountZ + 1][4];
#pragma unroll
      for (int p = 0; p <= kCountZ; p++) {
         const uint32_t *q = a.w + (size_t)(z + min(p, nZ)) * a.planeWS + (size_t)y * a.rowWS + wi;
         w[p][0] = q[0];
         w[p][1] = q[a.rowWS];
         w[p][2] = nx ? q[1] : 0u;
         w[p][3] = nx ? q[a.rowWS + 1] : 0u;
      }
#pragma unroll
      for (int p = 0; p < kCountZ; p++) {
         const uint32_t v0 = w[p][0], v2 = w[p][1], v4 = w[p + 1][0], v6 = w[p + 1][1];
         const uint32_t v1 = __funnelshift_r(v0, w[p][2], 1), v3 = __funnelshift_r(v2, w[p][3], 1);
         const uint32_t v5 = __funnelshift_r(v4, w[p + 1][2], 1), v7 = __funnelshift_r(v6, w[p + 1][3], 1);
         const uint32_t vm = p < nZ ? vmask : 0u;
         const uint32_t all = v0 & v1 & v2 & v3 & v4 & v5 & v6 & v7 & vm;
         const uint32_t none = ~(v0 | v1 | v2 | v3 | v4 | v5 | v6 | v7) & vm;
         uint32_t mixed = vm & ~(all | none);
         n255 += __popc(all);
         n0 += __popc(none);
         // word j's bits b, b + 1 go to code bits 2j, 2j + 1: shifted left by 2j as a (hi:lo) pair, the
         // top bit from the x + 1 word, one funnel shift by b brings them into place
         const uint32_t l1 = v2 << 2, h1 = v3 >> 29, l2 = v4 << 4, h2 = v5 >> 27, l3 = v6 << 6, h3 = v7 >> 25;
         while (mixed) {
            const int j = 31 - __clz(mixed);
            mixed ^= 1u << j;
            uint32_t c = (__funnelshift_r(l1, h1, j) & ~3u) | (__funnelshift_r(v0, v1 >> 31, j) & 3u);
            c = (__funnelshift_r(l2, h2, j) & ~15u) | (c & 15u);
            c = (__funnelshift_r(l3, h3, j) & ~63u) | (c & 63u);
            atomicAdd(h + (c & 255u), 1u);
         }
      }
   }
   n0 = __reduce_add_sync(FULL, (unsigned)n0) ;
   n255 = __reduce_add_sync(FULL, (unsigned)n255);
   if (lane == 0) {
      if (n0) { atomicAdd(&sEnds[0], n0); }
      if (n255) { atomicAdd(&sEnds[1], n255); }
   }
   __syncthreads();
   for (int c = threadIdx.x; c < 256; c += blockDim.x) {
      unsigned long long s = 0;
      for (int k = 0; k < 8; k++) { s += sh[k][c]; }
      if (c == 0) { s += sEnds[0]; }
      if (c == 255) { s += sEnds[1]; }
      if (s) { atomicAdd(a.out + c, s); }
   }
}

static int launchCount(unsigned long long *out, const BMOrg *pO, const uint32_t *w, cudaStream_t s)
{
   CountArgs a;
   a.w = w;
   a.X = (int)pO->rowElem;
   a.rows = (int)pO->rowPairs + 1;
   a.planes = (int)pO->planePairs + 1;
   a.rowWS = pO->rowWS;
   a.planeWS = pO->planeWS;
   a.out = out;
   if (pO->rowPairs == 0 || pO->planePairs == 0 || pO->rowElem < 2 || pO->rowWS == 0) { return MKF_OK; }
   a.nItems = (long long)a.rowWS * pO->rowPairs * ((pO->planePairs + kCountZ - 1) / kCountZ);
   // one item per thread up to 4 CTAs per SM: every CTA ends with up to 256 global atomics on the same
   // 256 counters, so fewer, busier CTAs finish sooner
   long long grid = (a.nItems + 255) / 256;
   const long long cap = (long long)smCount() * 4;
   if (grid > cap) { grid = cap; }
   if (grid < 1) { grid = 1; }
   if (a.nItems + grid * 256 < (1LL << 31)) { countMap<uint32_t><<<(unsigned)grid, 256, 0, s>>>(a); }
   else { countMap<unsigned long long><<<(unsigned)grid, 256, 0, s>>>(a); }
   return cudaFail(cudaGetLastError(), "countMap launch");
}

// Library-owned buffers of the original's lazy-allocation convention.
static uint32_t *gMap = nullptr;
static size_t gMapWords = 0;
static size_t *gBPFDDev = nullptr;
static size_t *gBPFDHost = nullptr;

static size_t *gBPFDStage = nullptr;  // pinned: counts on their way to the caller's array

// Pairs of timing events that no call is using. A pair belongs to the context that it was made in (a
// reset of the device ends that context and its events) and is used in it only. At most kEventPairs are
// kept, and the clean-up functions give the current context's back.
struct EventPair
{
   unsigned long long ctx;
   cudaEvent_t e0, e1;
};
static constexpr int kEventPairs = 16;
static std::mutex gEventMu;
static EventPair gEvents[kEventPairs];
static int gNumEvents = 0;

static void destroyEvents(const EventPair &p)
{
   if (p.e0) { cudaEventDestroy(p.e0); }
   if (p.e1) { cudaEventDestroy(p.e1); }
}

static EventPair takeEvents()
{
   const unsigned long long ctx = contextId();
   {
      std::lock_guard<std::mutex> lk(gEventMu);
      for (int i = 0; i < gNumEvents && ctx != 0; i++) {
         if (gEvents[i].ctx == ctx) {
            const EventPair p = gEvents[i];
            gEvents[i] = gEvents[--gNumEvents];
            return p;
         }
      }
   }
   EventPair p = {ctx, nullptr, nullptr};
   cudaEventCreate(&p.e0);
   cudaEventCreate(&p.e1);
   return p;
}

static void giveEvents(const EventPair &p)
{
   if (p.ctx != 0 && p.e0 && p.e1) {
      std::lock_guard<std::mutex> lk(gEventMu);
      if (gNumEvents < kEventPairs) {
         gEvents[gNumEvents++] = p;
         return;
      }
   }
   destroyEvents(p);
}

static void dropEvents()
{
   const unsigned long long ctx = contextId();
   std::lock_guard<std::mutex> lk(gEventMu);
   int n = 0;
   for (int i = 0; i < gNumEvents; i++) {
      if (gEvents[i].ctx == ctx) { destroyEvents(gEvents[i]); }
      else { gEvents[n++] = gEvents[i]; }
   }
   gNumEvents = n;
}

// Stage timer of the original's interface (events made and destroyed by each call instead of kept:
// 68.0 -> 69.5 us for the pair of calls on a 256^3 map).
class EventTimer
{
 public:
   EventTimer() : ev_(takeEvents()) { cudaEventRecord(ev_.e0, 0); }
   ~EventTimer() { giveEvents(ev_); }
   EventTimer(const EventTimer &) = delete;
   EventTimer &operator=(const EventTimer &) = delete;
   void mark() { cudaEventRecord(ev_.e1, 0); }
   // wait for the mark (or for work issued after it on the stream: one wait for both) and read the time
   float stop(bool stream = false)
   {
      float ms = 0;
      if (stream) { cudaStreamSynchronize(0); }
      else { cudaEventSynchronize(ev_.e1); }
      cudaEventElapsedTime(&ms, ev_.e0, ev_.e1);
      return ms;
   }

 private:
   EventPair ev_;
};

}  // namespace mkf

using namespace mkf;

MKF_API BMPackWord *binMapCUDA(KernInfo *pK, BMPackWord *pW, BMOrg *pO, const BMFieldInfo *pF, const BinMapF64 *pM)
{
   if (!pF || !pM) { return nullptr; }
   int nField = 0;
   if (pF->pFieldDevPtrTable) { nField = countValidPtrByMask(pF->pFieldDevPtrTable, pF->fieldTableMask); }
   FieldDef d[3];
   const int nDim = copyNonZeroDef(d, pF->pD, 3);
   if (nDim <= 0 || nField <= 0) { return nullptr; }
   if (pF->elemID != ENC_F32 && pF->elemID != ENC_F64) {
      logError("binMapCUDA() - element encoding 0x%02X not supported\n", pF->elemID);
      return nullptr;
   }
   BMOrg org;
   const size_t words = setBMO(&org, d, (char)pF->profID);
   if (pO) { *pO = org; }
   if (words == 0) { return nullptr; }
   if (!pW) {
      if (gMapWords < words) {
         if (gMap) { cudaFree(gMap); gMap = nullptr; gMapWords = 0; }
         if (cudaMalloc(&gMap, words * sizeof(uint32_t)) != cudaSuccess) {
            cudaGetLastError();
            logError("binMapCUDA() - cudaMalloc(%zu) failed\n", words * sizeof(uint32_t));
            return nullptr;
         }
         gMapWords = words;
      }
      pW = gMap;
   }
   PackArgs a;
   memset(&a, 0, sizeof(a));
   ConstFieldPtr fp[BMCU_FIELD_MAX];
   a.nF = copyValidPtrByMask(fp, BMCU_FIELD_MAX, pF->pFieldDevPtrTable, pF->fieldTableMask);
   for (int i = 0; i < a.nF; i++) { a.f[i] = fp[i].p; }
   // element strides of the dimensions that copyNonZeroDef kept
   if (pF->pS) {
      int k = 0;
      int64_t st[3] = {0, 0, 0};
      for (int i = 0; i < 3 && k < nDim; i++) {
         if (pF->pD[i] > 1) { st[k++] = pF->pS[i]; }
      }
      a.sx = st[0];
      a.sy = st[1];
      a.sz = st[2];
   } else {
      a.sx = 1;
      a.sy = d[0];
      a.sz = (int64_t)d[0] * d[1];
   }
   a.X = d[0];
   a.Y = (int)org.rowPairs + 1;
   a.Z = (int)org.planePairs + 1;
   a.rowWS = org.rowWS;
   a.planeWS = org.planeWS;
   a.t = (pF->elemID == ENC_F32) ? (double)(float)pM->t[0] : pM->t[0];
   a.m = pM->m;
   a.w = pW;
   a.nWords = (long long)org.rowWS * a.Y * a.Z;
   if ((long long)a.Y * a.Z >= (1LL << 32)) {
      logError("binMapCUDA() - %d x %d rows exceed 2^32\n", a.Y, a.Z);
      return nullptr;
   }
   EventTimer tm;
   long long grid = ((long long)a.Y * a.Z + 7) / 8;  // a warp per row
   const long long cap = (long long)smCount() * 8;      // one wave of 8 CTAs (64 warps) per SM
   if (grid > cap) { grid = cap; }
   if (pF->elemID == ENC_F32) { launchPack<float>(a, grid); }
   else { launchPack<double>(a, grid); }
   cudaError_t e = cudaGetLastError();
   tm.mark();
   const float ms = tm.stop();
   if (e == cudaSuccess) { e = cudaGetLastError(); }
   if (e != cudaSuccess) {
      logError("binMapCUDA() - r=%d -> %s\n", (int)e, cudaGetErrorName(e));
      return nullptr;
   }
   if (pK) { pK->dtms[0] = ms; }
   return pW;
}

MKF_API void binMapCUDACleanup(void)
{
   if (gMap) { cudaFree(gMap); gMap = nullptr; gMapWords = 0; }
   dropEvents();
}

MKF_API size_t *mkfCUDAGetBPFD(KernInfo *pK, size_t *pBPFD, const BMOrg *pO, const BMPackWord *pW, const int profile)
{
   (void)profile;  // every profile of the original yields the same counts
   if (!pBPFD) { return nullptr; }
   if (!pO || !pW) { return pBPFD; }
   EventTimer tm;
   const int rc = launchCount((unsigned long long *)pBPFD, pO, pW, 0);
   tm.mark();
   const float ms = tm.stop();
   if (rc != MKF_OK) { logError("mkfCUDAGetBPFD() - %s\n", mkfLastError()); }
   if (pK) { pK->dtms[1] = ms; }
   return pBPFD;
}

MKF_API size_t *mkfCUDAGetBPFDH(KernInfo *pK, size_t *pBPFDH, const BMOrg *pO, const BMPackWord *pW, const int profile)
{
   (void)profile;
   const size_t bytes = sizeof(size_t) * MKF_BINS;
   if (!pBPFDH) {
      if (!gBPFDHost && cudaMallocHost(&gBPFDHost, bytes) != cudaSuccess) { cudaGetLastError(); gBPFDHost = nullptr; }
      pBPFDH = gBPFDHost;
   }
   if (!gBPFDDev && cudaMalloc(&gBPFDDev, bytes) != cudaSuccess) { cudaGetLastError(); gBPFDDev = nullptr; }
   if (!gBPFDStage && cudaMallocHost(&gBPFDStage, bytes) != cudaSuccess) { cudaGetLastError(); gBPFDStage = nullptr; }
   if (!pBPFDH || !gBPFDDev || !gBPFDStage) { return nullptr; }
   cudaMemsetAsync(gBPFDDev, 0, bytes, 0);
   cudaGetLastError();  // clear any error left by earlier calls before checking ours
   // the count and the copy of its result in one go, with one wait at the end
   EventTimer tm;
   const int rc = (pO && pW) ? launchCount((unsigned long long *)gBPFDDev, pO, pW, 0) : MKF_OK;
   tm.mark();
   cudaError_t e = cudaMemcpyAsync(gBPFDStage, gBPFDDev, bytes, cudaMemcpyDeviceToHost, 0);
   const float ms = tm.stop(true);
   if (rc != MKF_OK) { logError("mkfCUDAGetBPFD() - %s\n", mkfLastError()); }
   if (pK && pO && pW) { pK->dtms[1] = ms; }
   if (e == cudaSuccess) { e = cudaGetLastError(); }
   if (e != cudaSuccess) { logError("mkfCUDAGetBPFDH() - r=%d -> %s\n", (int)e, cudaGetErrorName(e)); return nullptr; }
   memcpy(pBPFDH, gBPFDStage, bytes);
   return pBPFDH;
}

MKF_API void mkfCUDACleanup(int lvl)
{
   (void)lvl;  // the original resets the device when lvl > 0; a shared device is never reset here
   if (gBPFDHost) { cudaFreeHost(gBPFDHost); gBPFDHost = nullptr; }
   if (gBPFDDev) { cudaFree(gBPFDDev); gBPFDDev = nullptr; }
   if (gBPFDStage) { cudaFreeHost(gBPFDStage); gBPFDStage = nullptr; }
   dropEvents();
}

MKF_API int mkfCUDAGetBPFDautoCtx(Context *pC, const FieldDef def[3], const BinMapF64 *pM, const int profile)
{
   cudaError_t r;
   if (!pC) { return 0; }
   if (pC->pHF) {
      if (!pC->pDF) {
         r = cudaMalloc(&pC->pDF, pC->bytesF);
         if (r != cudaSuccess) { logError("cudaMalloc() - r=%d\n", (int)r); pC->pDF = nullptr; }
      }
      if (pC->pDF) {
         r = cudaMemcpy(pC->pDF, pC->pHF, pC->bytesF, cudaMemcpyHostToDevice);
         if (r != cudaSuccess) { logError("cudaMemcpy() - r=%d\n", (int)r); }
      }
      if (!pC->pDU) {
         r = cudaMalloc(&pC->pDU, pC->bytesU);
         if (r != cudaSuccess) { logError("cudaMalloc() - r=%d\n", (int)r); pC->pDU = nullptr; }
      }
      if (pC->pDF && pC->pDU) {
         ConstFieldPtr fieldPtr[BMCU_FIELD_MAX];
         BMFieldInfo fi;
         setupFields(&fi, autoFieldPtr(fieldPtr, pC), pC->nField, def, pC->bytesElem, profile);
         if (!binMapCUDA(&pC->ki, pC->pDU, &pC->bmo, &fi, pM)) { return 0; }
         if (pC->pHU) {
            r = cudaMemcpy(pC->pHU, pC->pDU, pC->bytesU, cudaMemcpyDeviceToHost);
            if (r != cudaSuccess) { logError("cudaMemcpy() - r=%d\n", (int)r); }
         }
      }
   } else if (pC->pHU) {
      r = cudaMemcpy(pC->pDU, pC->pHU, pC->bytesU, cudaMemcpyHostToDevice);
      if (r != cudaSuccess) { logError("cudaMemcpy() - r=%d\n", (int)r); }
      if (!pC->pDZ) {
         r = cudaMalloc(&pC->pDZ, pC->bytesZ);
         if (r != cudaSuccess) { logError("cudaMalloc() - r=%d\n", (int)r); pC->pDZ = nullptr; }
      }
   }
   if (pC->pDU && pC->pDZ) {
      cudaMemset(pC->pDZ, 0, pC->bytesZ);
      mkfCUDAGetBPFD(&pC->ki, (size_t *)pC->pDZ, &pC->bmo, pC->pDU, MKFCU_PROFILE_FAST);
      if (pC->pHZ) {
         r = cudaMemcpy(pC->pHZ, pC->pDZ, pC->bytesZ, cudaMemcpyDeviceToHost);
         if (r != cudaSuccess) { logError("cudaMemcpy() - r=%d\n", (int)r); }
      }
   }
   return 1;
}
