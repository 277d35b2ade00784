// blocks.cuh - asynchronous copies into shared memory of rows that start anywhere in a 16-byte block, as
// the whole blocks they touch. The address arithmetic is host code too, so that it can be checked without a
// GPU (the copy itself is a parameter).
//
// A block holds bytes outside the row. Those before the field's first element are read and not used: a
// field that does not start on a 16-byte boundary starts inside an allocation, whose start is on one. No
// byte after the field's last element is read: allocations end anywhere.
#pragma once
#include "fused.cuh"

namespace mkf {

// cp.async of BYTES bytes, of which the first n are read and the rest are zeros.
struct AsyncCopy
{
   template <int BYTES>
   static __device__ __forceinline__ void copy(uint32_t dst, const void *src, int n)
   {
      if (BYTES == 16) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory"); }
      else if (BYTES == 8) { asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory"); }
      else { asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory"); }
   }
};

// Whether the last block of the last row in memory is the only one that reaches past the field: unit x
// stride, rows and planes a block or more apart (RingBlocks; other fields are copied by elements).
template <typename A>
__host__ __device__ __forceinline__ bool blockRows(const A &a, int bytes)
{
   return a.sx == 1 && a.sy * bytes >= 16 && a.sz * bytes >= 16;
}

// ---- the staged rank-table kernel's tiles (thermo_tma.cu)

// Geometry of one work item: 31 x positions of cells, 8 row pairs, up to D planes of cells.
struct TmItem
{
   int xa, xoff;     // tile x (a multiple of ALIGN) and this item's first lane column in it
   int y0, z0, nPln; // tile rows y0 .. y0 + 8, planes z0 .. z0 + nPln
   uint32_t rowsOK;  // bit j: this lane counts row pair j
   unsigned cells;   // cells the item counts (warp total)
};

template <int ALIGN>
__host__ __device__ __forceinline__ TmItem itemOf(const FusedArgs &a, long long it, int lane)
{
   TmItem m;
   const int ix = (int)(it % a.nSegX);
   const long long rest = it / a.nSegX;
   const int iy = (int)(rest % a.nTileY);
   const int iz = (int)(rest / a.nTileY);
   const int xs = 31 * ix, ys = 8 * iy;
   const int xe = min(xs + 31, a.X - 1), ye = min(ys + 8, a.Y - 1);
   const int x0 = min(xs, a.X - 32);  // lanes at x0 + lane, all inside the field
   m.xa = x0 & ~(ALIGN - 1);
   m.xoff = x0 - m.xa;
   m.y0 = min(ys, a.Y - 9);
   m.z0 = a.D * iz;
   m.nPln = min(a.D, a.Z - 1 - m.z0);
   const int jlo = ys - m.y0, jhi = ye - m.y0;
   const bool laneIn = x0 + lane >= xs && x0 + lane < xe;
   m.rowsOK = laneIn ? (((1u << jhi) - 1u) & ~((1u << jlo) - 1u)) : 0u;
   m.cells = (unsigned)(xe - xs) * (unsigned)(jhi - jlo) * (unsigned)m.nPln;
   return m;
}

constexpr int kTmRows = 9;  // rows of a plane tile: 8 row pairs

// Copies the tiles of an item plane by plane: 9 rows of 32 elements, each as the NB + 1 blocks it touches.
template <typename T, typename CP = AsyncCopy>
struct RingBlocks
{
   static constexpr int B = (int)sizeof(T);
   static constexpr int NB = 2 * B;             // blocks of a row of 32 elements
   static constexpr int NR = 32 / NB;           // rows per copy of blocks
   static constexpr int ROWB = 16 * (NB + 1);   // bytes of a tile row
   static_assert(8 % NR == 0 && NB + kTmRows <= 32, "rows of NB + 1 blocks");
   const char *col;  // this lane's block of its row among the first NR, plus the row's offset in a block

   __host__ __device__ __forceinline__ void begin(const FusedArgs &a, const TmItem &m, int lane)
   {
      col = (const char *)a.f + ((int64_t)(m.xa + m.xoff) + (int64_t)(m.y0 + lane / NB) * a.sy + (int64_t)m.z0 * a.sz) * (int64_t)B + 16 * (lane % NB);
   }
   // Whether a block of the item's last plane ends after the field.
   static __host__ __device__ __forceinline__ bool atLast(const FusedArgs &a, const TmItem &m)
   {
      return (a.X - 32 - m.xa - m.xoff) * B < 16 && m.y0 + 9 == a.Y && m.z0 + m.nPln + 1 == a.Z;
   }
   // Copy a plane: NB blocks of NR rows at a time; then the ninth row's and, by the next nine lanes, each
   // row's last block, which it touches only where it does not start on a boundary.
   __host__ __device__ __forceinline__ void copy(const FusedArgs &a, uint32_t tile, int lane)
   {
      plane<false>(tile, lane, col, a.sy * (int64_t)B, nullptr);
      col += a.sz * (int64_t)B;
   }
   // The last plane of an item that atLast holds for: cut at the field's end.
   __host__ __device__ __forceinline__ void copyLast(const FusedArgs &a, uint32_t tile, int lane)
   {
      cutPlane(tile, lane, col, a.sy * (int64_t)B, (const char *)a.f + (a.X + (int64_t)(a.Y - 1) * a.sy + (int64_t)(a.Z - 1) * a.sz) * (int64_t)B);
   }

 private:
   // Out of line: a warp comes here once at most, and a check in every plane made the kernel 2 to 15 % slower.
   static __host__ __device__ __noinline__ void cutPlane(uint32_t tile, int lane, const char *col, int64_t sy, const char *end)
   {
      plane<true>(tile, lane, col, sy, end);
   }
   template <bool CUT>
   static __host__ __device__ __forceinline__ void plane(uint32_t tile, int lane, const char *col, int64_t sy, const char *end)
   {
      const uint32_t dst = tile + (uint32_t)((lane / NB) * ROWB + (lane % NB) * 16);
      const char *q = col;
#pragma unroll
      for (int k = 0; k < 8 / NR; ++k) {
         CP::template copy<16>(dst + (uint32_t)(k * NR * ROWB), (const void *)((uintptr_t)q & ~(uintptr_t)15), 16);
         q += sy * NR;
      }
      const int row = lane < NB ? 8 : lane - NB, blk = lane < NB ? lane : NB;
      q = col + sy * (row - lane / NB) + 16 * (blk - lane % NB);
      if (lane < NB || (lane < NB + kTmRows && ((uintptr_t)q & 15) != 0)) {
         const char *b = (const char *)((uintptr_t)q & ~(uintptr_t)15);
         CP::template copy<16>(tile + (uint32_t)(row * ROWB + blk * 16), b, CUT && end - b < 16 ? (int)(end - b) : 16);
      }
   }
};

}  // namespace mkf
