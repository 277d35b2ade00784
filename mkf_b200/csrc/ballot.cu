// ballot.cu - fused counting kernel for one threshold on fields of middle size, and for a few of one test
// (two of any) on strided, flat or narrow fields and part of those off 16-byte boundaries (useBallots): map
// words packed by warp votes from registers.
//
// The other kernel for few thresholds (words.cuh) lets each lane pack its own row from a copy of the
// tile in shared memory. That costs fewer instructions per threshold, but a FP64 tile row holds only
// 16 elements there, and its larger CTAs start more slowly; the rule at useBallots has the figures.
// A warp item is a tile of 32 x positions (31 cells), 32 rows (31 row pairs) and D planes, walked plane
// by plane:
//  * load: lane = x; the warp issues the 32 rows' coalesced loads at once;
//  * pack: one ballot per row and threshold gives that row's 32-bit map word; lane r keeps row r's;
//  * count: lane = row pair. A cell's eight corners are bits b and b+1 of four words (this lane's
//    row and the next lane's row, previous and current plane), so all-ones and all-zeros cells
//    are popcounts of ANDs and ORs of the words and their one-bit shifts; only mixed cells form
//    their 8-bit code, counted in a per-CTA shared histogram.
#include <cmath>
#include <cstring>
#include "fused.cuh"

namespace mkf {

// FP32 fields whose items lie inside the field and are at least kBlPfDepth planes deep load the next
// plane while counting the current one (two plane buffers in registers at 2 CTAs per SM, 128
// registers): 1.55 x faster with one threshold on a 1024^3 FP32 GRF (0.70 vs 1.09 ms; fields of that size
// come here if their rows lie off 16-byte boundaries), slower for shallow items, which keep the single
// buffer at 4 CTAs per SM.
static constexpr int kBlPfDepth = 16;
static constexpr int kBlWarps = 8;
static constexpr int kBlD = 32;  // default planes of cells per work item
// Untuned fields get at least this many work items per SM (the slab depth is halved until they
// do): measured on 256^3 to 512^3 fields, fewer items than ~0.6 of the resident warps leave SMs
// idle while deeper items win nothing.
static constexpr int kBlItemsPerSM = 20;

// The map bit of the tests in MODE (WordTask::mode): 1 f > tlo, 2 f < thi, 3 either.
template <int MODE, typename T>
__device__ __forceinline__ bool ballotBit(T v, T tlo, T thi)
{
   return (MODE == 1 && v > tlo) || (MODE == 2 && v < thi) || (MODE == 3 && (v > tlo || v < thi));
}

// State of one warp item between planes: the previous plane's map words and the cell counts.
template <int K>
struct BallotCarry
{
   uint32_t pw[K], pn[K];  // previous plane: this lane's row word and the next row's
   uint32_t n0[K], n1[K];  // all-zeros and all-ones cells counted by this lane
};

// Load one plane's 32 x 32 tile (lane = x). INNER: every row of the tile lies inside the field
// and the row stride in bytes `syb` times 31 fits 32 bits, so each row address is one multiply-add
// on the plane pointer; otherwise rows past the field end repeat its last row (their cells are
// masked out when counted) and addresses are formed in 64 bits.
template <typename T, bool INNER>
__device__ __forceinline__ void loadPlane(T (&v)[32], const T *__restrict__ p, int64_t sy, uint32_t syb, int nRow)
{
#pragma unroll
   for (int r = 0; r < 32; r++) {
      if (INNER) {
         v[r] = __ldg((const T *)((const char *)p + (uint64_t)(syb * (uint32_t)r)));
      } else {
         v[r] = __ldg(p + (int64_t)min(r, nRow - 1) * sy);
      }
   }
}

// Map, pack and count one plane (see the file comment). `first`: no previous plane yet.
// `sRow` is the warp's 32-word transposition buffer per threshold.
template <int MODE, int K, typename T>
__device__ __forceinline__ void countPlane(const T (&v)[32], BallotCarry<K> &c, const T (&tlo)[K], const T (&thi)[K], bool xin, int lane,
                                           uint32_t vm, bool first, uint32_t (*sRow)[32], uint32_t *sHist)
{
#pragma unroll
   for (int r = 0; r < 32; r++) {
#pragma unroll
      for (int k = 0; k < K; k++) {
         // every lane stores the same (warp-uniform) word
         sRow[k][r] = __ballot_sync(FULL, xin && ballotBit<MODE>(v[r], tlo[k], thi[k]));
      }
   }
   __syncwarp();
   uint32_t cw[K];
#pragma unroll
   for (int k = 0; k < K; k++) { cw[k] = sRow[k][lane]; }
   __syncwarp();
#pragma unroll
   for (int k = 0; k < K; k++) {
      const uint32_t cn = __shfl_down_sync(FULL, cw[k], 1);
      if (!first) {
         const uint32_t a0 = c.pw[k], a1 = c.pn[k], a2 = cw[k], a3 = cn;
         const uint32_t all = a0 & (a0 >> 1) & a1 & (a1 >> 1) & a2 & (a2 >> 1) & a3 & (a3 >> 1) & vm;
         const uint32_t any = a0 | (a0 >> 1) | a1 | (a1 >> 1) | a2 | (a2 >> 1) | a3 | (a3 >> 1);
         c.n1[k] += __popc(all);
         c.n0[k] += __popc(vm & ~any);
         uint32_t mixed = vm & any & ~all;
         if (mixed) {
            // word j's bits b, b+1 go to code bits 2j, 2j+1: pre-shift j's word left by 2j as a
            // 64-bit (hi:lo) pair, so one funnel shift by b brings them into place
            const uint32_t l1 = a1 << 2, h1 = a1 >> 30, l2 = a2 << 4, h2 = a2 >> 28, l3 = a3 << 6, h3 = a3 >> 26;
            do {
               const int b = 31 - __clz(mixed);
               mixed ^= 1u << b;
               uint32_t code = (__funnelshift_r(l1, h1, b) & ~3u) | ((a0 >> b) & 3u);
               code = (__funnelshift_r(l2, h2, b) & ~15u) | (code & 15u);
               code = (__funnelshift_r(l3, h3, b) & ~63u) | (code & 63u);
               atomicAdd(sHist + k * 256 + (code & 255u), 1u);
            } while (mixed);
         }
      }
      c.pw[k] = cw[k];
      c.pn[k] = cn;
   }
}

// One warp counts work item `it` (31 x 31 cells, D planes) of field `a` into the CTA's histogram
// and all-zeros / all-ones totals. INNER: the field is at least 32 x 32 in x and y with a positive
// row stride below 2^32 / 31 bytes; edge tiles are then shifted back inside the field (their cells
// already counted by the neighbouring tile are masked out), so no load needs clamping.
// PF: the next plane's loads are issued before the current plane is counted (two plane buffers
// in registers, alternating; INNER fields only).
template <typename T, int MODE, int K, bool INNER, bool PF>
__device__ __forceinline__ void ballotItem(const WordTask &a, long long it, const T (&tlo)[K], const T (&thi)[K], uint32_t (*sRow)[32],
                                           uint32_t *sHist, unsigned long long (*sEnds)[2])
{
   const int lane = threadIdx.x & 31;
   const T *__restrict__ F = (const T *)a.f;
   const uint32_t syb = (uint32_t)(a.sy * (int64_t)sizeof(T));
   const int ix = (int)(it % a.nStripX);
   const long long rest = it / a.nStripX;
   const int iy = (int)(rest % a.nTileY);
   const int iz = (int)(rest / a.nTileY);
   // this item's cells: x in [xs, xe), y in [ys, ye), z in [z0, z0 + nPln)
   const int xs = 31 * ix, ys = 31 * iy, z0 = a.D * iz;
   const int xe = min(xs + 31, a.X - 1), ye = min(ys + 31, a.Y - 1);
   const int nPln = min(a.D, a.Z - 1 - z0);
   // tile origin: bit b of a word is x0 + b, lane l counts the row pair y0 + l
   const int x0 = INNER ? min(xs, a.X - 32) : xs;
   const int y0 = INNER ? min(ys, a.Y - 32) : ys;
   const int nRow = INNER ? 32 : min(32, a.Y - y0);
   const bool xin = INNER || x0 + lane < a.X;
   const T *base = F + (long long)(INNER ? x0 + lane : min(x0 + lane, a.X - 1)) * a.sx + (long long)y0 * a.sy +
                   (long long)z0 * a.sz;
   const uint32_t vm = (y0 + lane >= ys && y0 + lane < ye)
                          ? ((0xFFFFFFFFu >> (32 - (xe - x0))) & (0xFFFFFFFFu << (xs - x0)))
                          : 0u;
   BallotCarry<K> c;
#pragma unroll
   for (int k = 0; k < K; k++) { c.pw[k] = c.pn[k] = c.n0[k] = c.n1[k] = 0; }
   if (PF && INNER) {
      T va[32], vb[32];
      loadPlane<T, INNER>(va, base, a.sy, syb, nRow);
      for (int p = 0; p <= nPln; p += 2) {
         if (p + 1 <= nPln) { loadPlane<T, INNER>(vb, base + (long long)(p + 1) * a.sz, a.sy, syb, nRow); }
         countPlane<MODE, K>(va, c, tlo, thi, xin, lane, vm, p == 0, sRow, sHist);
         if (p + 1 > nPln) { break; }
         if (p + 2 <= nPln) { loadPlane<T, INNER>(va, base + (long long)(p + 2) * a.sz, a.sy, syb, nRow); }
         countPlane<MODE, K>(vb, c, tlo, thi, xin, lane, vm, false, sRow, sHist);
      }
   } else {
      for (int p = 0; p <= nPln; ++p) {
         T v[32];
         loadPlane<T, INNER>(v, base + (long long)p * a.sz, a.sy, syb, nRow);
         countPlane<MODE, K>(v, c, tlo, thi, xin, lane, vm, p == 0, sRow, sHist);
      }
   }
#pragma unroll
   for (int k = 0; k < K; k++) {
      const unsigned long long s0 = __reduce_add_sync(FULL, c.n0[k]);
      const unsigned long long s1 = __reduce_add_sync(FULL, c.n1[k]);
      if (lane == 0) {
         if (s0) { atomicAdd(&sEnds[k][0], s0); }
         if (s1) { atomicAdd(&sEnds[k][1], s1); }
      }
   }
}

template <typename T, int MODE, int K, bool INNER, int MINB, bool PF>
__global__ void __launch_bounds__(kBlWarps * 32, MINB) ballotBPFD(const __grid_constant__ WordTask a)
{
   __shared__ uint32_t sHist[K * 256];
   __shared__ unsigned long long sEnds[K][2];  // all-zeros, all-ones cells
   __shared__ uint32_t sRows[kBlWarps][K][32];
   for (int i = threadIdx.x; i < K * 256; i += blockDim.x) { sHist[i] = 0; }
   if (threadIdx.x < K * 2) { (&sEnds[0][0])[threadIdx.x] = 0; }
   __syncthreads();
   T tlo[K], thi[K];
#pragma unroll
   for (int k = 0; k < K; k++) {
      tlo[k] = (T)a.tlo[k];
      thi[k] = (T)a.thi[k];
   }
   const long long gw = (long long)blockIdx.x * kBlWarps + (threadIdx.x >> 5);
   const long long nw = (long long)gridDim.x * kBlWarps;
   for (long long it = gw; it < a.nItems; it += nw) {
      ballotItem<T, MODE, K, INNER, PF>(a, it, tlo, thi, sRows[threadIdx.x >> 5], sHist, sEnds);
   }
   __syncthreads();
   // mixed codes as counted, 0 / 255 from the totals; counted negated, code c belongs in bin 255 - c
   for (int i = threadIdx.x; i < K * 256; i += blockDim.x) {
      const int k = i >> 8, c = i & 255;
      unsigned long long v = sHist[i];
      if (c == 0) { v += sEnds[k][0]; }
      if (c == 255) { v += sEnds[k][1]; }
      if (v) { atomicAdd((unsigned long long *)(a.out + (size_t)a.outRow[k] * 256 + ((a.inv >> k) & 1u ? 255 - c : c)), v); }
   }
}

template <typename T, int MODE, int K, bool INNER, int MINB, bool PF>
static int launchBallotT(const WordTask &a, cudaStream_t s)
{
   static std::atomic<int> occ{0};
   auto kern = ballotBPFD<T, MODE, K, INNER, MINB, PF>;
   const int blocksPerSM = cachedOccupancy(occ, kern, kBlWarps * 32, 0);
   long long grid = (a.nItems + kBlWarps - 1) / kBlWarps;
   const long long cap = (long long)smCount() * blocksPerSM;
   if (grid > cap) { grid = cap; }
   if (grid < 1) { grid = 1; }
   kern<<<(unsigned)grid, kBlWarps * 32, 0, s>>>(a);
   return cudaFail(cudaGetLastError(), "ballotBPFD launch");
}

static bool innerTiles(const WordTask &a, int enc)
{
   const int64_t syb = a.sy * (enc == ENC_F32 ? 4 : 8);
   return a.X >= 32 && a.Y >= 32 && syb > 0 && syb * 31 < (int64_t)1 << 32;
}

template <typename T, int MODE, int K>
static int launchBallotK(const WordTask &a, int enc, cudaStream_t s)
{
   constexpr bool F32 = sizeof(T) == 4;
   if (!innerTiles(a, enc)) { return launchBallotT<T, MODE, K, false, 2, false>(a, s); }
   if constexpr (F32 && K <= 2) {
      if (a.D >= kBlPfDepth) { return launchBallotT<T, MODE, K, true, 2, true>(a, s); }
      return launchBallotT<T, MODE, K, true, 4, false>(a, s);
   }
   return launchBallotT<T, MODE, K, true, F32 ? 3 : 2, false>(a, s);
}

template <typename T, int MODE>
static int launchBallotM(const WordTask &a, int enc, cudaStream_t s)
{
   if (a.K == 1) { return launchBallotK<T, MODE, 1>(a, enc, s); }
   if (a.K == 2) { return launchBallotK<T, MODE, 2>(a, enc, s); }
   if constexpr (MODE < 3) {
      if (a.K == 3) { return launchBallotK<T, MODE, 3>(a, enc, s); }
      if (a.K == 4) { return launchBallotK<T, MODE, 4>(a, enc, s); }
      if (a.K == 5) { return launchBallotK<T, MODE, 5>(a, enc, s); }
      if constexpr (sizeof(T) == 8) {
         if (a.K == 6) { return launchBallotK<T, MODE, 6>(a, enc, s); }
      }
   }
   setError("vote kernel: %d thresholds", a.K);
   return MKF_ERR_UNSUPPORTED;
}

template <typename T>
static int dispatchBallot(const WordTask &a, int enc, cudaStream_t s)
{
   switch (a.K == 2 && a.mode[1] != a.mode[0] ? 3 : a.mode[0]) {
      case 1: return launchBallotM<T, 1>(a, enc, s);
      case 2: return launchBallotM<T, 2>(a, enc, s);
      default: return launchBallotM<T, 3>(a, enc, s);
   }
}

// Where this kernel counts a field. Its cost follows the content (uniform cells cost nothing), the others'
// hardly does, and the content is not known here. So a line stands where this kernel is the faster one on
// Gaussian fields (GRF), plane waves and balls with noise alike, or by more on some than slower on others.
// B200, time of a call with the other kernel over that with this one, on GRF / waves / balls:
//  one threshold, word kernel: FP32 64^3 0.87, 128^3 1.07, 256^3 1.07; aligned rows 512^3 0.95, 128 x 2048 x 2048
//   0.90; other rows 500^3 1.04 / 1.02 / 1.17, 291 x 361 x 823 GRF 0.92, 17 x 2048 x 2048 1.32 / 1.24 / 1.40, strided 500^3 1.9; FP64 64^3 0.76,
//   128^3 1.04, 256 x 512 x 512 1.13, 333 x 401 x 487 1.31
//  two to four, word kernel: 100^3 0.7, 128^3 0.9;
//   strided x: FP32 128^3 0.9, 200 x 210 x 190 0.85 to 1.0, 256^3 1.1 to 1.3, 500^3 1.26 to 1.7; FP64 160 x 150 x 170 0.9
//   to 1.07, 200 x 210 x 190 1.2 to 1.7; 512 x 6 x 512 FP32 1.3 to 1.5, 512 x 40 x 512 1.05 to 1.16, 512 x 512 x 20 1.1, FP64 1.25;
//   few planes: 2 x 2048 x 2048 FP32 other rows 1.3, FP64 aligned 1.05 to 1.2, other rows 1.6 to 1.9; 9 x 1024 x 1024
//   1.0 to 1.25, 1.0 to 1.25, 1.3 to 1.6; 5 x 1024 x 1024 FP64 aligned 2 thresholds 1.08 / 0.97 / 1.12, 4 0.98 / 0.93 / 0.85;
//   33 x 1024 x 1024 FP32 other rows 1.1 / 0.95 / 1.2; 17 x 512 x 512 1.0 / 0.88 / 1.05, FP64 1.2 / 1.05 / 1.2;
//   few columns: 512 x 512 x 20 other rows FP32 1.1 (2000 x 1000 x 17 0.9 / 0.93 / 1.08), FP64 1.2, aligned FP64 1.15; where the word kernel's tiles fit the row
//   and the votes' 31 cells do not, FP64 512 x 512 x 8 4 thresholds 0.75, 2000 x 1000 x 17 0.6 to 0.8, FP32 512 x 512 x 33 0.7;
//   few rows: 512 x 6 x 512 FP32 1.1, FP64 1.25 to 1.5; 512 x 40 x 512 FP64 1.03 to 1.15, other rows 1.1 to 1.3;
//   2000 x 20 x 1000 FP64 aligned 4 thresholds 0.86 / 0.91 / 1.07;
//   thick fields: FP32 other rows 400^3 2 and 3 thresholds 0.84 / 0.8 / 1.04, 4 1.0 / 1.12 / 1.22, 278 x 222 x 614
//   GRF 0.89, 500^3 0.80 / 1.0 / 1.05 (from 2^27 voxels on 599 x 611 x 515 balls 3 thresholds 1.22, 4 1.27, 861 x 841 x 512 5 1.36);
//   FP64 aligned 0.9 to 1.07 but 4 thresholds from 2^24 voxels on 0.97 / 1.06 / 1.07; other rows 2 thresholds
//   200 x 210 x 190 0.99 / 1.09 / 1.18, 4 0.93 / 1.15 / 1.11, from 2^24 voxels on 1.07 to 1.2
//  five and six, rank table: strided x FP32 300 x 333 x 277 0.94 / 1.07 / 1.10, 500^3 0.95 / 1.28 / 1.27, FP64 300 x 333 x
//   277 1.15, 500^3 1.35, few rows (512 x 9 x 1024) 0.55; 2 x 2048 x 2048 1.2 to 1.3, 5 x 1024 x 1024 0.9 to 1.0, 9 x 4096
//   x 4096 0.9 / 1.05 / 1.26; rows of less than 32 elements 1.4 to 2 (the staged kernel does not take them).
bool useBallots(const WordTask &a, int enc)
{
   const bool f64 = enc == ENC_F64, aligned = wordRowsAligned(a, enc), strided = a.sx != 1;
   const double voxels = (double)a.X * a.Y * a.Z;
   if (a.K == 1) {
      return voxels >= (double)(1 << 20) &&
             (f64 || strided || voxels < (double)(1 << 26) || (!aligned && (a.Z < 34 || voxels >= (double)(1 << 27))));
   }
   if (a.K > (f64 ? 6 : 5) || voxels < (double)(a.Y < 9 ? 1 << 20 : 1 << 21)) { return false; }
   for (int k = 0; k < a.K && a.K > 2; k++) {  // (two thresholds may differ in their tests)
      if (a.mode[k] != a.mode[0] || a.mode[k] == 3) { return false; }
   }
   // cells that either kernel's tiles cover in a row
   const int el = f64 ? 16 : 32, word = (a.X - 1 + el - 1) / el * el, vote = (a.X - 1 + 30) / 31 * 31;
   const bool narrow = a.X < 64 && (f64 || voxels < (double)(1 << 24));
   if (a.X < 64 && 10 * vote > 13 * word && !(f64 && strided && a.X >= 32)) { return false; }
   if (a.K >= 5) {
      if (a.X < 32) { return true; }
      if (a.Y < 64) { return false; }
      if (strided) { return voxels >= (double)(f64 ? 3 << 23 : 1 << 25) || (a.Z < 10 && voxels >= (double)(1 << 23)); }
      if (a.Z < 8 && voxels >= (double)(1 << 23)) { return a.K == 5 ? f64 || !aligned : !aligned && a.Z < 5; }
      return a.K == 5 && !f64 && !aligned && voxels >= (double)(1 << 27);
   }
   if (strided) { return narrow || a.Y < 64 || (a.Z < 10 && voxels >= (double)(1 << 23)) || voxels >= (double)(f64 ? 3 << 21 : 3 << 22); }
   if (f64 && aligned) {
      const bool large = voxels >= (double)(1 << 24);
      return (a.X < 32 && a.K < 4) || (a.Y < 64 && (a.K < 4 || !large)) || (a.Z < 10 && voxels >= (double)(a.K == 2 ? 1 << 22 : 1 << 23)) ||
             (a.K == 4 && large && innerTiles(a, enc));
   }
   if (f64) { return narrow || a.Y < 64 || a.Z < 34 || voxels >= (double)(a.K == 3 ? 1 << 24 : 1 << 22); }
   if (aligned) { return a.Y < 9; }
   return narrow || a.Y < (a.K == 4 ? 64 : 16) || a.Z < (voxels < (double)(1 << 23) ? 10 : 34) || voxels >= (double)(1 << 27);
}

int launchBallots(WordTask &a, int enc, cudaStream_t s)
{
   a.nStripX = (a.X - 1 + 30) / 31;
   a.nTileY = (a.Y - 1 + 30) / 31;
   a.D = tunedDepth(kFamBallot, enc, a.K, a.X, a.Y, a.Z,
                    sizeDepth(kBlD, (long long)a.nStripX * a.nTileY, a.Z, (long long)smCount() * kBlItemsPerSM));
   a.nSlabZ = (a.Z - 1 + a.D - 1) / a.D;
   a.nItems = (long long)a.nStripX * a.nTileY * a.nSlabZ;
   if (a.K == 2 && a.mode[1] != a.mode[0]) {  // both made "f > tlo or f < thi", the test not wanted never true
      for (int k = 0; k < 2; k++) {
         if (!(a.mode[k] & 1)) { a.tlo[k] = INFINITY; }
         if (!(a.mode[k] & 2)) { a.thi[k] = -INFINITY; }
      }
   }
   return enc == ENC_F32 ? dispatchBallot<float>(a, enc, s) : dispatchBallot<double>(a, enc, s);
}

}  // namespace mkf
