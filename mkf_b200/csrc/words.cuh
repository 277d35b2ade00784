// words.cuh - the word-parallel counting kernel: one to kWordMaxK thresholds of any relations
// counted in one read (words.cu has the single-field launches, words_batch.cu the batched ones).
//
// A warp item is a strip of W tiles in x, 31 row pairs (32 rows, lane = row) and D planes, walked
// plane by plane and from right to left within a plane. A tile is 32 rows of 128 bytes: 32 elements
// of a FP32 field, 16 of a FP64 field.
//  * copy: cp.async fills the warp's ring of tiles in shared memory ahead of the tile it counts, 16
//    bytes per lane where rows lie on 16-byte boundaries (8 instructions per tile) and, as the nine
//    blocks that a row touches, where they lie elsewhere (MIS, 9 instructions); with strided x one
//    element per lane. No registers hold data in flight, and the ring runs on over the end of an item into
//    the next;
//  * map: a lane reads its own row (the 16-byte skew of the row pitch spreads the lanes' 128-bit
//    reads over all banks) and forms the row's map bits itself, one nibble per element: FP32 as the
//    sign of a fused multiply-add (two elements per instruction) shifted into the word, FP64 as a
//    compare and a predicated OR;
//  * codes: the nibbles of this row and the next lane's, in this plane and the previous one (whose
//    words wait in shared memory), merge into one nibble per x position, and a cell's 8-bit code is
//    two neighbouring nibbles: a byte of the word for even cells, a byte of the word shifted by one
//    nibble for odd ones. About 60 instructions form the codes of 32 x 32 cells;
//  * count: groups of 8 cells that are all zeros or all ones only add to a counter; the others (8
//    codes in two words) go to the lane's queue in shared memory, drained into the CTA's histogram
//    when some lane's fills up.
// A tile's last cells need the first nibble of the tile to its right, which is the one just
// counted; only a strip's last tile loads that element from memory. Single elements cost a DRAM burst
// each: with strips of one tile a 2048 x 2048 x 256 FP32 field of 4.3 GB read 8.0 GB.
// What bounds it: the integer ALU pipe (63 % busy) and issue (65 %) from three thresholds on, about 250
// instructions per threshold and 32 x 32 cells; with one threshold the field's bytes and the halos
// (32 rows per 31, D + 1 planes per D). Measured against the vote-per-row kernel that it replaced
// for two and more thresholds (B200, us): 128 x 2048 x 2048 FP32 plane waves, 3 thresholds 748 -> 604,
// 2 647 -> 417; 512^3 FP32 GRF 3 302 -> 220, 2 193 -> 151; 128 x 1024 x 1024 FP64 plane waves 3 270 -> 221;
// 96 uneven FP32 fields, one threshold, one batch 1550 -> 1112; 288 x 320 x 384 FP32, 5 thresholds of 5
// relations (before: a binary search per element and a loop per map bit) 656 -> 120; moments of
// 400^3 FP64, 2 thresholds 747 -> 154.
#pragma once
#include "blocks.cuh"

namespace mkf {

// MIS: rows start anywhere in a 16-byte block; a tile row is then the 9 whole blocks it touches.
template <typename T, bool MIS>
struct RowGeom
{
   static constexpr int EL = 128 / (int)sizeof(T);  // elements of a tile row
   static constexpr int NR = EL / 8;                // words of 8 nibbles per tile row
   static constexpr int EX = MIS ? 16 / (int)sizeof(T) : 0;  // elements of the ninth block
   // 128 bytes, the element after the strip, skew: 16-byte reads by 8 lanes fall in all 32 banks
   static constexpr int PITCH = MIS ? 176 : 144;
   static constexpr int STAGE = 32 * PITCH;         // one tile
};

// CTA: up to 16 warps (one CTA per SM); the rings, queues and state words share 227 KB of shared
// memory with the histograms.
constexpr int kWdWarps = 16;
constexpr int kWdQueue = 9;   // queue entries per lane (a tile row adds up to NR)

// Shared memory of a warp: the ring, the queue (8 bytes of codes and one of threshold per entry) and
// per threshold and lane the state words: previous plane (NR / 2 per tile), the element after
// the strip, the word to the right, the all-ones groups.
__host__ __device__ constexpr int wordState(int nr, int K, int W) { return K * (W * (nr / 2) + 3); }
// Ring stages. A third one in place of a quarter of the warps measured 4-14 % slower (one threshold,
// 256^3 to 512^3).
constexpr int kWdStages = 2;
__host__ __device__ constexpr int wordWarpBytes(int nr, int K, int W, bool mis)
{
   return kWdStages * 32 * (mis ? 176 : 144) + kWdQueue * 288 + wordState(nr, K, W) * 128;
}

// Dynamic shared memory of a CTA: 227 KB less the static part (histograms, a batch's task).
constexpr int kWdDynBytes = 232448 - 1024 * (kWordMaxK + 1) - 2048;

// Warps of a batch CTA that the memory holds for a field (its form for fields with unit x stride has larger
// tiles: 14 of FP32, one threshold, 11 with eight).
__host__ __device__ constexpr int wordBatchWarps(int nr, int K, int W, bool mis)
{
   return kWdDynBytes / wordWarpBytes(nr, K, W, mis) < kWdWarps ? kWdDynBytes / wordWarpBytes(nr, K, W, mis) : kWdWarps;
}

// A threshold as the map step uses it.
struct alignas(16) RowThresh
{
   float s0, s1, c0, c1;  // FP32: first test (sign of s * f + c)
   float u0, u1, d0, d1;  // FP32: second test (relations with both)
   double g, l;           // FP64: f > g, f < l
   int mode, pad_;        // bit 0: "f > t" is tested, bit 1: "f < t"
};
static_assert(sizeof(RowThresh) == 64 && offsetof(RowThresh, u0) == 16 && offsetof(RowThresh, g) == 32, "read as 16-byte vectors");

struct RowShared
{
   alignas(1024) uint32_t hist[kWordMaxK * 256];  // bin: a code as it lies in the nibbles (rowCode)
   RowThresh th[kWordMaxK];
   unsigned long long ones[kWordMaxK], cells;
   unsigned next;  // next work item to hand out
   double mom[2][2][2];
};

__device__ __forceinline__ void rowSetup(const WordTask &a, RowShared &S)
{
   for (int i = threadIdx.x; i < a.K * 256; i += blockDim.x) { S.hist[i] = 0; }
   if (threadIdx.x < a.K) {
      const int k = threadIdx.x;
      S.ones[k] = 0;
      RowThresh &t = S.th[k];
      const int mode = a.mode[k];
      // "f > t": the sign of t - f; "f < t": the sign of f - t. c is never -0 (-0 - 0 would have its
      // sign set), and a NaN result has sign 0: neither test holds, the relation "equal".
      const float cg = (float)a.tlo[k] + 0.0f, cl = 0.0f - (float)a.thi[k];
      t.s0 = t.s1 = mode == 0 ? 0.0f : (mode & 1) ? -1.0f : 1.0f;  // (no test: 0 * f + 0, sign 0)
      t.c0 = t.c1 = mode == 0 ? 0.0f : (mode & 1) ? cg : cl;
      t.u0 = t.u1 = 1.0f;
      t.d0 = t.d1 = cl;
      t.g = a.tlo[k];
      t.l = a.thi[k];
      t.mode = mode;
   }
   if (threadIdx.x == 0) {
      S.cells = 0;
      S.next = 0;
      for (int q = 0; q < 8; q++) { (&S.mom[0][0][0])[q] = 0.0; }
   }
   __syncthreads();
}

// The pattern of a code as it lies in two nibbles (low: x, high: x + 1): bit 3 this row and bit 2
// the next one in the current plane, bits 1 and 0 the same in the previous plane.
__device__ __forceinline__ int rowCode(int c)
{
   return ((c >> 1) & 1) | ((c >> 4) & 2) | ((c << 2) & 4) | ((c >> 1) & 8) | ((c << 1) & 16) | ((c >> 2) & 32) | ((c << 4) & 64) |
          ((c << 1) & 128);
}

// Add the CTA's counts of one field to its output rows (whole CTA): mixed codes as counted, 255
// with the all-ones groups, 0 the cells that remain. A threshold whose map was counted negated
// (WordTask::inv) has code c in bin 255 - c.
__device__ inline void rowFlush(const WordTask &a, RowShared &S)
{
   __syncthreads();
   const int lane = threadIdx.x & 31, nWarps = blockDim.x >> 5;
   for (int k = threadIdx.x >> 5; k < a.K; k += nWarps) {
      unsigned long long *o = (unsigned long long *)(a.out + (size_t)a.outRow[k] * 256);
      const int flip = (a.inv >> k) & 1 ? 255 : 0;
      const unsigned long long groups = S.ones[k];
      uint32_t sum = 0;
      for (int c = lane; c < 256; c += 32) {
         const uint32_t v = c ? S.hist[k * 256 + c] : 0u;  // (bin 0 holds the drain's idle lanes)
         const unsigned long long n = v + (c == 255 ? 8 * groups : 0ull);
         sum += v;
         if (n) { atomicAdd(o + (rowCode(c) ^ flip), n); }
      }
      sum = __reduce_add_sync(FULL, sum);
      if (lane == 0) {
         const unsigned long long n0 = S.cells - 8 * groups - sum;
         if (n0) { atomicAdd(o + flip, n0); }
      }
   }
}

__device__ __forceinline__ void cpCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpWait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t ldShared(uint32_t at)
{
   uint32_t v;
   asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
   return v;
}
__device__ __forceinline__ void stShared(uint32_t at, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }

// Geometry of one work item.
struct RowItem
{
   int x0, y0, z0, nPln;  // first element, row and plane of the tile, planes of cells
   int ys, ye;            // row pairs counted: y in [ys, ye)
   int nT;                // tiles of the strip
};

template <int EL>
__host__ __device__ __forceinline__ RowItem rowItemOf(const WordTask &a, long long it)
{
   RowItem m;
   int ix, iy, iz;
   if (a.nItems < 0x7FFFFFFFLL) {
      const uint32_t i = (uint32_t)it, q = i / (uint32_t)a.nStripX;
      ix = (int)(i - q * (uint32_t)a.nStripX);
      iz = (int)(q / (uint32_t)a.nTileY);
      iy = (int)(q - (uint32_t)iz * (uint32_t)a.nTileY);
   } else {
      const long long q = it / a.nStripX;
      ix = (int)(it - q * a.nStripX);
      iz = (int)(q / a.nTileY);
      iy = (int)(q - (long long)iz * a.nTileY);
   }
   m.x0 = EL * a.W * ix;
   m.nT = min(a.W, (a.X - 1 - m.x0 + EL - 1) / EL);
   m.ys = 31 * iy;
   m.ye = min(m.ys + 31, a.Y - 1);
   m.y0 = max(0, min(m.ys, a.Y - 32));  // the last tile is shifted back inside the field
   m.z0 = a.D * iz;
   m.nPln = min(a.D, a.Z - 1 - m.z0);
   return m;
}

// Copies an item's tiles one after another into the warp's ring: 32 rows of EL elements, with the
// last tile of a strip also the element after each row; rows past the field's last repeat it, elements
// past the row end are zero.
template <typename T, bool MIS, typename CP = AsyncCopy>
struct RowCopier
{
   using G = RowGeom<T, MIS>;
   static constexpr int B = (int)sizeof(T);
   const char *p;         // this lane's first element of the tile (vec, MIS: of the row lane / 8, 16 (lane % 8) bytes on)
   const char *after;     // the element after the tile, row = lane
   int64_t sy, sz, tile;  // byte steps: row, plane, tile
   int64_t step0;         // (not vec) from the address used past the row end to the lane's column
   int last;              // the field's last row, counted from the tile's first
   int nx;                // elements from the strip's last tile to the row end (>= 2)
   int nEnd, adj;         // (vec) the strip's last tile: bytes to copy, and the way back to a valid address where none are
   int nAfter;            // bytes of the element after the strip (0: past the row end)
   int nT, tiles, planes; // tiles of a plane; left in the plane, planes left
   bool vec, wide;        // wide: all 32 rows inside, byte offsets below 2^32

   __host__ __device__ __forceinline__ void begin(const WordTask &a, const RowItem &m, int lane)
   {
      vec = MIS || a.vec;
      sy = a.sy * B;
      sz = a.sz * B;
      tile = (int64_t)G::EL * a.sx * B;
      nT = tiles = m.nT;
      planes = m.nPln + 1;
      last = a.Y - 1 - m.y0;
      wide = last >= 31 && sy >= 0 && sy < (1 << 26);
      nx = a.X - m.x0 - G::EL * (nT - 1);
      const char *c = (const char *)a.f + ((int64_t)m.x0 * a.sx + (int64_t)m.y0 * a.sy + (int64_t)m.z0 * a.sz) * B + tile * (nT - 1);
      nAfter = nx > G::EL ? B : 0;
      after = c + (MIS || nAfter ? tile : 0) + (int64_t)min(lane, last) * sy;
      step0 = 0;
      adj = 0;
      if (vec) {
         nEnd = max(0, min(16, nx * B - 16 * (lane & 7)));
         p = c + 16 * (lane & 7) + (int64_t)min(lane >> 3, last) * sy;
         if (!MIS && nEnd == 0) { adj = -16 * (lane & 7); }
      } else {
         const int col = lane & (G::EL - 1);  // (FP64: 16 elements, two rows at once)
         nEnd = col < nx ? B : 0;
         p = c + (int64_t)(nEnd > 0 ? col : 0) * a.sx * B + (int64_t)min(lane / G::EL, last) * sy;
         if (nEnd == 0) { step0 = (int64_t)col * a.sx * B; }
      }
   }
   __host__ __device__ __forceinline__ bool left() const { return planes > 0; }
   // The 16-byte block of a row whose first byte would be at q (off bytes from the tile's first
   // element), cut at the row end.
   __host__ __device__ __forceinline__ void block(uint32_t d, const char *q, int off, bool end)
   {
      const uint32_t sh = (uint32_t)(uintptr_t)q & 15u;
      q -= sh;
      if (end) {
         const int n = max(0, min(16, nx * B - off + (int)sh));
         CP::template copy<16>(d, n > 0 ? q : q - off, n);
      } else {
         CP::template copy<16>(d, q, 16);
      }
   }
   __host__ __device__ __forceinline__ void copy(uint32_t dst, int lane)
   {
      const bool end = tiles == nT;
      if constexpr (MIS) {
         const uint32_t d = dst + (uint32_t)((lane >> 3) * G::PITCH + (lane & 7) * 16);
         if (wide && !end) {
            const uint32_t step = 4u * (uint32_t)sy;
#pragma unroll
            for (int i = 0; i < 8; i++) { block(d + (uint32_t)(i * 4 * G::PITCH), p + (uint64_t)(step * (uint32_t)i), 16 * (lane & 7), false); }
         } else {
            const int r0 = lane >> 3;
#pragma unroll 1
            for (int i = 0; i < 8; i++) {
               block(d + (uint32_t)(i * 4 * G::PITCH), p + (int64_t)(min(r0 + 4 * i, last) - min(r0, last)) * sy, 16 * (lane & 7), end);
            }
         }
         // the ninth block, lane = row (the row may end in it also left of the strip's last tile)
         const uint32_t sh = (uint32_t)(uintptr_t)after & 15u;
         const int n = max(0, min(16, (nx + (end ? 0 : G::EL)) * B - 128 + (int)sh));
         CP::template copy<16>(dst + (uint32_t)(lane * G::PITCH + 128), after - sh - (n > 0 ? 0 : 128), n);
         after -= tile;
      } else if (vec) {
         const char *q = p + (end ? adj : 0);
         const int n = end ? nEnd : 16;
         const uint32_t d = dst + (uint32_t)((lane >> 3) * G::PITCH + (lane & 7) * 16);
         if (wide) {
            const uint32_t step = 4u * (uint32_t)sy;
#pragma unroll
            for (int i = 0; i < 8; i++) { CP::template copy<16>(d + (uint32_t)(i * 4 * G::PITCH), q + (uint64_t)(step * (uint32_t)i), n); }
         } else {
            const int r0 = lane >> 3;
#pragma unroll 1
            for (int i = 0; i < 8; i++) {
               CP::template copy<16>(d + (uint32_t)(i * 4 * G::PITCH), q + (int64_t)(min(r0 + 4 * i, last) - min(r0, last)) * sy, n);
            }
         }
      } else {
         const int n = end ? nEnd : B;
         constexpr int R = 32 / G::EL;  // rows per copy
         const int r0 = lane / G::EL;
         const uint32_t d = dst + (uint32_t)(r0 * G::PITCH + (lane & (G::EL - 1)) * B);
         if (wide) {
            const uint32_t step = (uint32_t)R * (uint32_t)sy;
#pragma unroll 8
            for (int i = 0; i < G::EL; i++) { CP::template copy<B>(d + (uint32_t)(i * R * G::PITCH), p + (uint64_t)(step * (uint32_t)i), n); }
         } else {
#pragma unroll 1
            for (int i = 0; i < G::EL; i++) {
               CP::template copy<B>(d + (uint32_t)(i * R * G::PITCH), p + (int64_t)(min(r0 + R * i, last) - min(r0, last)) * sy, n);
            }
         }
      }
      if (end) {
         if (!MIS) { CP::template copy<B>(dst + (uint32_t)(lane * G::PITCH + 128), after, nAfter); }
         p += step0;
      }
      p -= tile;
      if (--tiles == 0) {
         tiles = nT;
         p += tile * nT + sz - step0;
         after += sz + (MIS ? tile * nT : 0);
         --planes;
      }
   }
};

// A threshold's test in registers. FP32: {s, s}, {c, c} of the first sign test; FP64: both values.
struct RowTestF32
{
   unsigned long long s, c;
   __device__ __forceinline__ void load(const RowThresh &t)
   {
      asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(s), "=l"(c) : "r"((uint32_t)__cvta_generic_to_shared(&t.s0)) : "memory");
   }
};
struct RowTestF64
{
   double g, l;
   __device__ __forceinline__ void load(const RowThresh &t)
   {
      asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(g), "=d"(l) : "r"((uint32_t)__cvta_generic_to_shared(&t.g)) : "memory");
   }
};

// A lane's tile row (EL elements at addr in shared memory).
template <int EX>
struct RowF32
{
   using Test = RowTestF32;
   unsigned long long v[16 + EX / 2];  // two elements each
   __device__ __forceinline__ void load(uint32_t addr)
   {
#pragma unroll
      for (int i = 0; i < 8 + EX / 4; i++) {
         asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v[2 * i]), "=l"(v[2 * i + 1]) : "r"(addr + 16u * (uint32_t)i) : "memory");
      }
   }
   // Map bits of the row for one threshold: bit 3 of nibble j of s[i] is element 8 i + j (s[4]: the
   // EX elements of the ninth block).
   __device__ __forceinline__ void bits(uint32_t (&s)[4 + (EX ? 1 : 0)], const RowTestF32 &th, const RowThresh &both, bool two) const
   {
      if (!two) {
#pragma unroll
         for (int i = 0; i < 4 + (EX ? 1 : 0); i++) {
            uint32_t w = 0;
#pragma unroll
            for (int j = (i < 4 ? 4 : EX / 2) - 1; j >= 0; j--) {
               unsigned long long d;
               uint32_t lo, hi;
               asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(v[4 * i + j]), "l"(th.s), "l"(th.c));
               asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(d));
               w = __funnelshift_l(hi, w, 4);
               w = __funnelshift_l(lo, w, 4);
            }
            s[i] = w;
         }
      } else {
         unsigned long long u2, d2;
         asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(u2), "=l"(d2) : "r"((uint32_t)__cvta_generic_to_shared(&both.u0)) : "memory");
#pragma unroll
         for (int i = 0; i < 4 + (EX ? 1 : 0); i++) {
            uint32_t w = 0;
#pragma unroll
            for (int j = (i < 4 ? 4 : EX / 2) - 1; j >= 0; j--) {
               unsigned long long d, e;
               uint32_t lo, hi;
               asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(v[4 * i + j]), "l"(th.s), "l"(th.c));
               asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(e) : "l"(v[4 * i + j]), "l"(u2), "l"(d2));
               d |= e;
               asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(d));
               w = __funnelshift_l(hi, w, 4);
               w = __funnelshift_l(lo, w, 4);
            }
            s[i] = w;
         }
      }
   }
   __device__ __forceinline__ float at(int i) const { return __uint_as_float((uint32_t)(v[i >> 1] >> (32 * (i & 1)))); }
};
template <int EX>
struct RowF64
{
   using Test = RowTestF64;
   double v[16 + EX];
   __device__ __forceinline__ void load(uint32_t addr)
   {
#pragma unroll
      for (int i = 0; i < 8 + EX / 2; i++) {
         asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[2 * i]), "=d"(v[2 * i + 1]) : "r"(addr + 16u * (uint32_t)i) : "memory");
      }
   }
   __device__ __forceinline__ void bits(uint32_t (&s)[2 + (EX ? 1 : 0)], const RowTestF64 &th, bool greater, bool less) const
   {
      s[0] = s[1] = 0;
      if (EX) { s[EX ? 2 : 0] = 0; }
      if (greater) {
#pragma unroll
         for (int i = 0; i < 16 + EX; i++) {
            if (v[i] > th.g) { s[i >> 3] |= 8u << (4 * (i & 7)); }
         }
      }
      if (less) {
#pragma unroll
         for (int i = 0; i < 16 + EX; i++) {
            if (v[i] < th.l) { s[i >> 3] |= 8u << (4 * (i & 7)); }
         }
      }
   }
   __device__ __forceinline__ double at(int i) const { return v[i]; }
};
template <typename T, int EX> struct RowOf;
template <int EX> struct RowOf<float, EX> { using type = RowF32<EX>; };
template <int EX> struct RowOf<double, EX> { using type = RowF64<EX>; };

// The map bit of one element.
__device__ __forceinline__ uint32_t rowBit(float x, const RowTestF32 &t, const RowThresh &th, bool greater, bool less)
{
   uint32_t q = __float_as_uint(fmaf(x, __uint_as_float((uint32_t)t.s), __uint_as_float((uint32_t)t.c))) >> 31;
   if (greater && less) { q |= __float_as_uint(fmaf(x, th.u0, th.d0)) >> 31; }
   return q;
}
__device__ __forceinline__ uint32_t rowBit(double x, const RowTestF64 &t, const RowThresh &, bool greater, bool less)
{
   return (greater && x > t.g) || (less && x < t.l);
}

// Count the queued groups of 8 cells: every lane its own entries, all lanes together (a lane without
// one adds to bin 0, which the flush leaves out; sharing the entries out evenly, found by a search
// over the lanes' counts, measured slower). q: this lane's first entry, qk its first entry's
// threshold, n its entries.
static __device__ __noinline__ void rowDrain(uint32_t q, uint32_t qk, int n, uint32_t hist)
{
   for (int i = 0; __any_sync(FULL, i < n); i++) {
      uint32_t E = 0, O = 0, k = 0;
      if (i < n) {
         asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(E), "=r"(O) : "r"(q + 256u * (uint32_t)i) : "memory");
         asm volatile("ld.shared.u8 %0, [%1];" : "=r"(k) : "r"(qk + 32u * (uint32_t)i) : "memory");
      }
      const uint32_t h = hist + k * 1024u;  // (1024-byte aligned: offsets are ORed in)
#pragma unroll
      for (int b = 0; b < 4; b++) {
         const uint32_t e = b == 0 ? E << 2 : E >> (8 * b - 2), o = b == 0 ? O << 2 : O >> (8 * b - 2);
         asm volatile("red.shared.add.u32 [%0], 1;" ::"r"((e & 0x3FCu) | h) : "memory");
         asm volatile("red.shared.add.u32 [%0], 1;" ::"r"((o & 0x3FCu) | h) : "memory");
      }
   }
}

// A warp's share of the CTA's work items item(0), item(1), .. below end of field `a`, handed out one
// at a time, counted into the CTA's histogram and totals. KT: the number of thresholds when it is
// known (their tests, all-ones groups and words to the right then stay in registers), 0 any number.
// mem: shared address of the warp's memory (wordWarpBytes).
template <typename T, bool MOM, int KT, bool MIS, typename ITEM>
__device__ __forceinline__ void rowItems(const WordTask &a, ITEM item, long long end, uint32_t mem, RowShared &S)
{
   using G = RowGeom<T, MIS>;
   using Row = typename RowOf<T, G::EX>::type;
   constexpr int NR = G::NR, STAGES = kWdStages, KR = KT > 0 ? KT : 1;
   const int lane = threadIdx.x & 31, K = KT > 0 ? KT : a.K;
   const uint32_t q0 = mem + (uint32_t)(STAGES * G::STAGE + lane * 8), qk0 = mem + (uint32_t)(STAGES * G::STAGE + kWdQueue * 256 + lane);
   const uint32_t qMax = q0 + (kWdQueue - NR) * 256u;
   // state words (rows of 32): per threshold the element after the strip, the word to the right and
   // the all-ones groups; then per tile and threshold the previous plane's
   const uint32_t misc0 = mem + (uint32_t)(STAGES * G::STAGE + kWdQueue * 288 + lane * 4), prev0 = misc0 + (uint32_t)K * 384u;
   uint32_t greater = 0, less = 0;  // thresholds with a test "f > t", with "f < t"
   for (int k = 0; k < K; k++) {
      greater |= (uint32_t)(a.mode[k] & 1) << k;
      less |= (uint32_t)((a.mode[k] >> 1) & 1) << k;
   }
   // copy cursor: the item whose tiles are copied (end: none left). It is at most one item ahead of
   // the one being counted, whose successor it holds by the time that one is done.
   RowCopier<T, MIS> cp;
   cp.planes = 0;
   long long pIt = -1;
   int pS = 0;
   auto copy = [&]() {
      if (!cp.left() && pIt < end) {
         int j = 0;
         if (lane == 0) { j = (int)atomicAdd(&S.next, 1u); }
         pIt = item(__shfl_sync(FULL, j, 0));
         if (pIt < end) { cp.begin(a, rowItemOf<G::EL>(a, pIt), lane); }
      }
      if (cp.left()) { cp.copy(mem + (uint32_t)(pS * G::STAGE), lane); }
      pS = pS + 1 == STAGES ? 0 : pS + 1;
      cpCommit();
   };
   copy();
   long long it = pIt;
#pragma unroll
   for (int s = 0; s + 2 < STAGES; s++) { copy(); }

   const uint32_t hist = (uint32_t)__cvta_generic_to_shared(S.hist);
   typename Row::Test test[KR];
   uint32_t ones[KR], right[KR];
   if constexpr (KT > 0) {
#pragma unroll
      for (int k = 0; k < KT; k++) {
         test[k].load(S.th[k]);
         ones[k] = right[k] = 0;
      }
   } else {
      for (int k = 0; k < K; k++) { stShared(misc0 + (uint32_t)k * 384u + 256u, 0u); }
   }
   unsigned long long cells = 0;
   uint32_t qa = q0, qk = qk0;
   double mom[MOM ? 2 : 1][2][2] = {};
   int cS = 0;
   for (; it < end; it = pIt) {
      const RowItem m = rowItemOf<G::EL>(a, it);
      const int nx = a.X - 1 - m.x0;  // cells from the strip's first to the row end
      const bool rowIn = m.y0 + lane >= m.ys && m.y0 + lane < m.ye;
      // masks of this row's bits and the next row's (a lane without a row pair has all-zeros cells)
      const uint32_t lm8 = rowIn ? 0x88888888u : 0u, lm4 = lm8 >> 1;
      cells += (unsigned long long)(unsigned)min(G::EL * m.nT, nx) * (unsigned)(m.ye - m.ys) * (unsigned)m.nPln;
      uint32_t rowLow = 0;
      if (MIS) {
         rowLow = (uint32_t)(uintptr_t)a.f + (uint32_t)(((int64_t)m.x0 + (int64_t)min(m.y0 + lane, a.Y - 1) * a.sy + (int64_t)m.z0 * a.sz) * (int64_t)sizeof(T));
      }
      for (int p = 0; p <= m.nPln; p++) {
         double sum[MOM ? 2 : 1][2][2] = {};
         // MIS: where this lane's row starts in its first 16-byte block
         const uint32_t off = MIS ? (rowLow + (uint32_t)p * (uint32_t)(a.sz * (int64_t)sizeof(T))) & 15u : 0u;
         for (int t = m.nT - 1; t >= 0; t--) {
            // the next tile: wait for it, then start the copy into the stage of the one before, which
            // every lane has read
            cpWait<STAGES - 2>();
            __syncwarp();
            copy();
            const uint32_t row = mem + (uint32_t)(cS * G::STAGE + lane * G::PITCH);
            cS = cS + 1 == STAGES ? 0 : cS + 1;
            Row v;
            v.load(row);
            const bool atEnd = t == m.nT - 1;
            T x = T(0);  // the element after the strip
            if (atEnd) { x = *reinterpret_cast<const T *>(__cvta_shared_to_generic(row + 128u + (MIS ? off : 0u))); }
            const int nc = nx - G::EL * t;  // the tile's cells
            const uint32_t prevT = prev0 + (uint32_t)(t * K) * (NR / 2 * 128u);
            // one threshold: tst, its tests in registers; o, r its all-ones groups and word to the right
            auto count = [&](int k, const typename Row::Test &tst, uint32_t &o, uint32_t &r, uint32_t misc, uint32_t prev) {
               uint32_t s[NR + (MIS ? 1 : 0)], F[NR], P[NR / 2], after = 0;
               // the previous plane's nibbles, two words in one (bits 3, 2 of the even word, 1, 0 of the
               // odd one), read ahead of their use
#pragma unroll
               for (int i = 0; i < NR / 2; i++) { P[i] = ldShared(prev + 128u * (uint32_t)i); }
               if (atEnd) { after = ldShared(misc); }
               const bool G1 = (greater >> k) & 1u, L1 = (less >> k) & 1u;
               if constexpr (sizeof(T) == 4) { v.bits(s, tst, S.th[k], G1 && L1); }
               else { v.bits(s, tst, G1, L1); }
               if constexpr (MIS) {  // to the row's first element
                  const uint32_t by = sizeof(T) == 4 ? off : off >> 1;
#pragma unroll
                  for (int i = 0; i < NR; i++) { s[i] = __funnelshift_r(s[i], s[i + 1], by); }
               }
               if constexpr (MOM) {
                  double s1 = 0.0, q1 = 0.0, s0 = 0.0, q2 = 0.0;
#pragma unroll
                  for (int i = 0; i < G::EL; i++) {
                     const double d = (double)v.at(i);
                     if (s[i >> 3] & (8u << (4 * (i & 7)))) { s1 += d; q1 += d * d; }
                     else { s0 += d; q2 += d * d; }
                  }
                  if (atEnd && nx == G::EL * m.nT) {  // the element after the strip is the row's last
                     const double d = (double)x;
                     if (rowBit(x, tst, S.th[k], G1, L1)) { s1 += d; q1 += d * d; }
                     else { s0 += d; q2 += d * d; }
                  }
                  double (&to)[2][2] = sum[k];
                  to[0][0] += s0;
                  to[0][1] += q2;
                  to[1][0] += s1;
                  to[1][1] += q1;
               }
               if (atEnd) {
                  const uint32_t b = rowBit(x, tst, S.th[k], G1, L1);
                  const uint32_t f = ((b << 3) & lm8) | ((__shfl_down_sync(FULL, b, 1) << 2) & lm4);
                  r = f | (after >> 2);
                  stShared(misc, f);
               }
               // this row (bit 3) and the next (bit 2)
#pragma unroll
               for (int i = 0; i < NR; i++) { F[i] = (s[i] & lm8) | ((__shfl_down_sync(FULL, s[i], 1) >> 1) & lm4); }
#pragma unroll
               for (int i = 0; i < NR / 2; i++) { stShared(prev + 128u * (uint32_t)i, F[2 * i] | (F[2 * i + 1] >> 2)); }
               if (p == 0) { return; }
               uint32_t E[NR], O[NR];
#pragma unroll
               for (int i = 0; i < NR / 2; i++) {
                  E[2 * i] = F[2 * i] | ((P[i] >> 2) & 0x33333333u);
                  E[2 * i + 1] = F[2 * i + 1] | (P[i] & 0x33333333u);
               }
#pragma unroll
               for (int i = 0; i < NR; i++) { O[i] = __funnelshift_r(E[i], i + 1 < NR ? E[i + 1 < NR ? i + 1 : 0] : r, 4); }
               r = E[0];
               if (__any_sync(FULL, nc < G::EL)) {  // cells past the row end: all zeros
#pragma unroll
                  for (int i = 0; i < NR; i++) {
                     const int e = max(0, min(4, (nc - 8 * i + 1) >> 1)), q = max(0, min(4, (nc - 8 * i) >> 1));
                     E[i] &= (uint32_t)((1ull << (8 * e)) - 1ull);
                     O[i] &= (uint32_t)((1ull << (8 * q)) - 1ull);
                  }
               }
#pragma unroll
               for (int i = 0; i < NR; i++) {
                  // uniform (E and O both 0 or both ~0): o counts -E; else queued
                  asm volatile(
                     "{\n\t.reg .pred p;\n\t"
                     "setp.ne.u32 p, %5, 0;\n\t"
                     "@p st.shared.v2.u32 [%0], {%3, %4};\n\t"
                     "@p st.shared.u8 [%1], %6;\n\t"
                     "@p add.u32 %0, %0, 256;\n\t"
                     "@p add.u32 %1, %1, 32;\n\t"
                     "@!p sub.u32 %2, %2, %3;\n\t}"
                     : "+r"(qa), "+r"(qk), "+r"(o)
                     : "r"(E[i]), "r"(O[i]), "r"((E[i] ^ O[i]) | (E[i] ^ (uint32_t)((int32_t)E[i] >> 31))), "r"(k)
                     : "memory");
               }
               if (__any_sync(FULL, qa > qMax)) {
                  rowDrain(q0, qk0, (int)((qa - q0) >> 8), hist);
                  qa = q0;
                  qk = qk0;
               }
            };
            if constexpr (KT > 0) {
#pragma unroll
               for (int k = 0; k < KT; k++) {
                  count(k, test[k], ones[k], right[k], misc0 + (uint32_t)k * 384u, prevT + (uint32_t)k * (NR / 2 * 128u));
               }
            } else {
#pragma unroll 1
               for (int k = 0; k < K; k++) {
                  const uint32_t misc = misc0 + (uint32_t)k * 384u;
                  typename Row::Test tst;
                  tst.load(S.th[k]);
                  uint32_t r = ldShared(misc + 128u), o = ldShared(misc + 256u);
                  count(k, tst, o, r, misc, prevT + (uint32_t)k * (NR / 2 * 128u));
                  stShared(misc + 128u, r);
                  stShared(misc + 256u, o);
               }
            }
         }
         if constexpr (MOM) {
            const int y = m.y0 + lane;
            if ((rowIn || (m.ye == a.Y - 1 && y == a.Y - 1)) && (p < m.nPln || m.z0 + p == a.Z - 1)) {
#pragma unroll
               for (int q = 0; q < 8; q++) { (&mom[0][0][0])[q] += (&sum[0][0][0])[q]; }
            }
         }
      }
   }
   cpWait<0>();
   __syncwarp();
   rowDrain(q0, qk0, (int)((qa - q0) >> 8), hist);
   auto total = [&](int k, uint32_t o) {
      // (per lane below 2^32 groups: a warp's share of a field of 2^40 cells or fewer)
      unsigned long long n = o;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) { n += __shfl_xor_sync(FULL, n, d); }
      if (lane == 0 && n) { atomicAdd(&S.ones[k], n); }
   };
   if constexpr (KT > 0) {
#pragma unroll
      for (int k = 0; k < KT; k++) { total(k, ones[k]); }
   } else {
      for (int k = 0; k < K; k++) { total(k, ldShared(misc0 + (uint32_t)k * 384u + 256u)); }
   }
   if (lane == 0 && cells) { atomicAdd(&S.cells, cells); }
   if constexpr (MOM) {
#pragma unroll
      for (int q = 0; q < 8; q++) {
         double x = (&mom[0][0][0])[q];
#pragma unroll
         for (int o = 16; o > 0; o >>= 1) { x += __shfl_xor_sync(FULL, x, o); }
         if (lane == 0 && x != 0.0) { atomicAdd(&S.mom[0][0][0] + q, x); }
      }
   }
   __syncwarp();
}

}  // namespace mkf
