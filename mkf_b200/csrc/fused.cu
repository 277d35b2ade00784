// fused.cu - one read of a scalar field -> K binary pattern frequency distributions: thresholds are
// classified and routed to the counting kernels.
//
// Replaces the original two-pass path binMapCUDA (binMapCUDA.cu:144-264, threshold + pack) followed
// by mkfCUDAGetBPFD (mkfCUDA.cu:12-61, pack -> 256-bin counts), which makes one full pass per
// threshold and materialises the packed map in device memory. Here the packed map never exists:
//
//  * thresholds whose map is constant (an empty or full relation mask, a NaN threshold) are counted
//    without reading the field;
//  * a few thresholds, of any relations, go to the word-parallel kernel (words.cuh), in passes of up
//    to kWordMaxK;
//  * more thresholds that share one relation (<, <=, > or >=) go to the rank-table kernels
//    (thermo_tma.cu, thermo.cu), whose cost hardly grows with their number.
//
// Pattern bit order is the original's (bpfdCUDA.cuh:45-61): bit i <-> corner
// (x + (i&1), y + ((i>>1)&1), z + ((i>>2)&1)). Every row of X elements yields X-1 cells.
#include <algorithm>
#include <cmath>
#include <cstring>
#include "fused.cuh"

namespace mkf {

// Add `cells` to bin `bin` of output row `row` (a threshold whose map is constant).
__global__ void addConstBin(uint64_t *out, int row, int bin, unsigned long long cells)
{
   out[(size_t)row * 256 + bin] += cells;
}

int launchConstBin(uint64_t *out, int row, int bin, unsigned long long cells, cudaStream_t s)
{
   addConstBin<<<1, 1, 0, s>>>(out, row, bin, cells);
   return cudaFail(cudaGetLastError(), "addConstBin launch");
}

// Threshold pair (tlo, thi) that makes a FP32 comparison give the exact result of comparing the
// element promoted to double with t: f > t <=> f > tlo and f >= t <=> f >= thi.
void floatBoundsPlain(double t, double &tlo, double &thi)
{
   const float fl = (float)t;
   if ((double)fl == t) { tlo = thi = fl; return; }
   float a, b;
   if ((double)fl > t) { b = fl; a = std::nextafter(fl, -INFINITY); }
   else { a = fl; b = std::nextafter(fl, INFINITY); }
   tlo = a;
   thi = b;
}

void splitThresholds(const MKFThreshSet *pT, ThreshSplit &q)
{
   q.n = q.nConst = 0;
   q.cls = -2;
   for (int i = 0; i < pT->nT; i++) {
      const double t = pT->t[i];
      const uint32_t m = (pT->m ? pT->m[i] : pT->mAll) & BMC_AL;
      if (m == 0 || m == BMC_AL || std::isnan(t)) {
         const bool one = (m == BMC_AL) || (std::isnan(t) && (m & BMC_EQ));
         q.constIdx[q.nConst] = i;
         q.constBin[q.nConst++] = one ? 255 : 0;
         continue;
      }
      int cls = -1;
      if (m == BMC_GT) { cls = 0; }
      else if (m == (BMC_GT | BMC_EQ)) { cls = 1; }
      else if (m == BMC_LT) { cls = 2; }
      else if (m == (BMC_LT | BMC_EQ)) { cls = 3; }
      if (q.n == 0) { q.cls = cls; }
      else if (cls != q.cls) { q.cls = -1; }
      // insertion keeps the thresholds sorted ascending, equal ones in the caller's order
      int b = q.n++;
      while (b > 0 && pT->t[q.idx[b - 1]] > t) { q.idx[b] = q.idx[b - 1]; b--; }
      q.idx[b] = i;
   }
}

// Thresholds of one relation that the word kernels count rather than a rank-table kernel, whose cost
// hardly grows with their number (B200, us, word kernel / rank table): 512^3 FP32 GRF 4 thresholds
// 244 / 302, 5 325 / 304; 128 x 2048 x 2048 FP32 plane waves 4 739 / 734, 5 947 / 1145; 256 x 512 x 512
// FP64 GRF 4 158 / 165, 5 221 / 166; rows off 16-byte boundaries: 401 x 403 x 405 FP32 GRF 3 130 / 144,
// 4 150 / 143, plane waves 4 137 / 143; 333 x 401 x 487 FP64 GRF 4 161 / 144, 5 193 / 144, plane waves
// 4 138 / 144, 5 165 / 145; 100 x 101 x 99 FP64 4 12.2 / 13.0.
static constexpr int kWordThresholds = 4;

void fillRankArgs(FusedArgs &a, const MKFFieldDesc *pF, const MKFThreshSet *pT, const ThreshSplit &q, int row0)
{
   memset(&a, 0, sizeof(a));
   const int X = pF->def[0], Y = pF->def[1], Z = pF->def[2];
   const bool planar = !(pF->stride[0] | pF->stride[1] | pF->stride[2]);
   a.f = pF->p;
   a.sx = planar ? 1 : pF->stride[0];
   a.sy = planar ? (int64_t)X : pF->stride[1];
   a.sz = planar ? (int64_t)X * Y : pF->stride[2];
   a.X = X; a.Y = Y; a.Z = Z;
   a.K = q.n;
   for (int i = 0; i < 64; i++) { a.tlo[i] = a.thi[i] = INFINITY; }
   for (int k = 0; k < q.n; k++) {
      const double t = pT->t[q.idx[k]];
      if (pF->enc == ENC_F32) { floatBoundsPlain(t, a.tlo[k], a.thi[k]); }
      else { a.tlo[k] = a.thi[k] = t; }
      a.outRow[k] = row0 + q.idx[k];
   }
   a.rankHi = (q.cls == 1 || q.cls == 2);
   a.complement = (q.cls >= 2);
   const bool eqBit = (q.cls == 1 || q.cls == 3);
   a.nanRank = (eqBit != (a.complement != 0)) ? (uint32_t)q.n : 0u;
}

void fillWordTask(WordTask &w, const MKFFieldDesc *pF, const MKFThreshSet *pT, const ThreshSplit &q, int k0, int n, int row0)
{
   memset(&w, 0, sizeof(w));
   const int X = pF->def[0], Y = pF->def[1];
   const bool planar = !(pF->stride[0] | pF->stride[1] | pF->stride[2]);
   w.f = pF->p;
   w.sx = planar ? 1 : pF->stride[0];
   w.sy = planar ? (int64_t)X : pF->stride[1];
   w.sz = planar ? (int64_t)X * Y : pF->stride[2];
   w.X = X; w.Y = Y; w.Z = pF->def[2];
   w.K = n;
   for (int k = 0; k < n; k++) {
      const int i = q.idx[k0 + k];
      fillWordThresh(w, k, pF->enc, pT->t[i], pT->m ? pT->m[i] : pT->mAll, row0 + i);
   }
}

// Fields of kSoloVoxels or more with more than two thresholds fill the GPU on their own, and the
// single-field kernels (specialised on the number of thresholds; the TMA-staged rank table on aligned rows)
// count them faster than the batched ones. A served burst of 64 fields of 32^3 to 320^3 with 1-8 thresholds:
// the cut at 2^23 voxels 1750 us, at 2^24 1800, at 2^26 2015.
static constexpr double kSoloVoxels = (double)(1 << 23);

void BatchMix::add(const MKFFieldDesc *pF, const MKFThreshSet *pT)
{
   const int e = pF->enc == ENC_F32 ? 0 : 1;
   const double vox = (double)pF->def[0] * (double)pF->def[1] * (double)pF->def[2];
   ThreshSplit q;
   splitThresholds(pT, q);
   if (q.n == 0 || (q.n > 2 && (vox >= kSoloVoxels || q.n > kWordMaxK))) { return; }
   if (q.n <= 2 || q.cls < 0) { words[e] = true; }
   else {
      fields[e]++;
      voxels[e] += vox;
      thresholds[e] += vox * q.n;
   }
}

// A batch whose fields differ goes to the batched word kernel in one launch (fields of 1 to 8 thresholds,
// 64 fields served: up to 2 thresholds in the word kernel and the rest in the rank table's 1869 us, all
// 1537; plans of 40 to 70 fields 535 / 453, 774 / 607, 669 / 599). Where no field needs the word kernel the
// rank table alone counts it, whose cost hardly grows with the thresholds. Word kernel over rank table, plans
// (GRF / waves / balls): 400 fields of 12^3 to 20^3 3 thresholds 1.8, 8 2.9; 100 of 40^3 to 80^3 FP32 3 1.15, 5 1.25,
// 8 1.65; 64 of 60^3 to 120^3 FP32 3 1.02 / 0.86 / 0.86, 4 1.1 / 1.0 / 1.04, 5 1.26 / 1.14 / 1.25, FP64 3 1.14 / 1.03 / 1.08;
// 24 of 150^3 to 200^3 FP32 3 1.0 / 0.76 / 0.71, 4 1.05 / 0.9 / 0.87, 5 1.16 / 1.0 / 0.97, FP64 3 1.08 / 0.94 / 0.87, 4 1.13 /
// 1.05 / 1.0; in one-shot batches (shallow items, time with the host's) 0.9 to 0.95 up to 5 thresholds, from 100^3 on 6
// 1.0 to 1.2, 8 1.1 to 1.4.
int BatchMix::wordMax(int enc, int depth) const
{
   const int e = enc == ENC_F32 ? 0 : 1;
   if (words[e] || fields[e] == 0) { return kWordMaxK; }
   const double vox = voxels[e] / fields[e], k = thresholds[e] / voxels[e];
   const bool rank = depth < 0 ? vox >= (double)(1 << 20) && k >= 5.5 : vox < (double)(e ? 1 << 20 : 1 << 19) || k >= (e ? 3.5 : 4.5);
   return rank ? 2 : kWordMaxK;
}

// Split one field of a batch (rows from row0): up to kWordMaxK thresholds of any relations, but of one
// relation up to wordMax (BatchMix), fill `w` for the batched word kernel (returns kPlanWords); more
// thresholds that share one thermometer relation and fit the rank table fill `t` for the batched thermometer
// kernel (kPlanThermo); the rest takes the single-field path (kPlanSingle). Constant maps are added to `consts`.
int planBatchField(const MKFFieldDesc *pF, const MKFThreshSet *pT, int row0, FieldTask &t, WordTask &w,
                   std::vector<ConstEntry> &consts, bool &anyVarying, int wordMax, int depth)
{
   memset(&t, 0, sizeof(t));
   memset(&w, 0, sizeof(w));
   const double vox = (double)pF->def[0] * (double)pF->def[1] * (double)pF->def[2];
   if (depth < 0) {
      // by size: shallow work items for small fields, so that a launch over many of them has
      // items enough for every SM (measured best for batches of fields up to ~400^3)
      depth = vox <= (double)(1 << 25) ? 8 : 0;
   }
   ThreshSplit q;
   splitThresholds(pT, q);
   for (int c = 0; c < q.nConst; c++) { consts.push_back({row0 + q.constIdx[c], q.constBin[c]}); }
   anyVarying = q.n > 0;
   if (q.n == 0) { return kPlanSingle; }
   const bool word = q.n <= 2 || (q.n <= kWordMaxK && vox < kSoloVoxels);
   auto words = [&]() {
      fillWordTask(w, pF, pT, q, 0, q.n, row0);
      fillWordGrid(w, pF->enc, depth > 0 ? depth : 32, q.n <= 4 ? 2 : 1);
      return kPlanWords;
   };
   if (word && (q.cls < 0 || q.n <= wordMax)) { return words(); }
   if (q.cls < 0 || vox >= kSoloVoxels) { return kPlanSingle; }
   FusedArgs a;
   fillRankArgs(a, pF, pT, q, row0);
   t.f = a.f;
   t.sx = a.sx; t.sy = a.sy; t.sz = a.sz;
   t.X = a.X; t.Y = a.Y; t.Z = a.Z;
   t.K = a.K;
   memcpy(t.tlo, a.tlo, sizeof(t.tlo));
   memcpy(t.thi, a.thi, sizeof(t.thi));
   memcpy(t.outRow, a.outRow, sizeof(t.outRow));
   t.rankHi = a.rankHi;
   t.complement = a.complement;
   t.nanRank = a.nanRank;
   if (prepareThermoTask(t, pF->enc, depth)) { return kPlanThermo; }
   return word ? words() : kPlanSingle;
}

int countVarying(uint64_t *out, const MKFFieldDesc *pF, const MKFThreshSet *pT, const ThreshSplit &q, cudaStream_t s)
{
   bool words = q.cls < 0 || q.n <= kWordThresholds;
   if (!words && q.n <= (pF->enc == ENC_F32 ? 5 : 6)) {
      // votes (useBallots), or a field of too few columns or rows for the staged rank-table kernel (5 thresholds,
      // word kernel / rank table read from global memory, us: 64 x 64 x 20 FP32 17 / 24, FP64 14 / 24, 2000 x 1000 x 17
      // FP64 78 / 200, 64 x 6 x 64 FP32 14 / 20; but 512 x 6 x 512 FP64 1.5 x)
      WordTask w;
      fillWordTask(w, pF, pT, q, 0, q.n, 0);
      words = useBallots(w, pF->enc) || w.X < 32 || (w.Y < 9 && (double)w.X * w.Y * w.Z < (double)(1 << 19));
   }
   if (!words) {
      FusedArgs a;
      fillRankArgs(a, pF, pT, q, 0);
      a.out = out;
      const int rc = launchThermo(a, pF->enc, s);
      if (rc != MKF_ERR_UNSUPPORTED) { return rc; }
   }
   const int passes = (q.n + kWordMaxK - 1) / kWordMaxK;
   for (int p = 0; p < passes; p++) {
      const int k0 = (int)((long long)q.n * p / passes), k1 = (int)((long long)q.n * (p + 1) / passes);
      WordTask w;
      fillWordTask(w, pF, pT, q, k0, k1 - k0, 0);
      w.out = out;
      const int rc = useBallots(w, pF->enc) ? launchBallots(w, pF->enc, s) : launchWords(w, pF->enc, s);
      if (rc != MKF_OK) { return rc; }
   }
   return MKF_OK;
}

int fieldBPFD(uint64_t *out, const MKFFieldDesc *pF, const MKFThreshSet *pT, int flags, cudaStream_t s)
{
   if (!out || !pF || !pT || !pF->p) { setError("mkfFieldBPFD: NULL argument"); return MKF_ERR_ARG; }
   const int K = pT->nT;
   if (K < 1 || K > MKF_MAX_THRESH || !pT->t) { setError("mkfFieldBPFD: nT=%d out of range 1..%d", K, MKF_MAX_THRESH); return MKF_ERR_ARG; }
   if (pF->enc != ENC_F32 && pF->enc != ENC_F64) { setError("mkfFieldBPFD: encoding 0x%02X not supported", pF->enc); return MKF_ERR_UNSUPPORTED; }
   const int X = pF->def[0], Y = pF->def[1], Z = pF->def[2];
   if (X < 1 || Y < 1 || Z < 1) { setError("mkfFieldBPFD: bad dimensions %d %d %d", X, Y, Z); return MKF_ERR_ARG; }
   if (!(flags & MKF_F_ACCUMULATE)) {
      const cudaError_t e = cudaMemsetAsync(out, 0, (size_t)K * 256 * sizeof(uint64_t), s);
      if (e != cudaSuccess) { return cudaFail(e, "cudaMemsetAsync"); }
   }
   const unsigned long long cells = (unsigned long long)(X - 1) * (unsigned long long)(Y - 1) * (unsigned long long)(Z - 1);
   if (cells == 0) { return MKF_OK; }
   ThreshSplit q;
   splitThresholds(pT, q);
   int rc = q.n > 0 ? countVarying(out, pF, pT, q, s) : MKF_OK;
   for (int c = 0; c < q.nConst && rc == MKF_OK; c++) { rc = launchConstBin(out, q.constIdx[c], q.constBin[c], cells, s); }
   return rc;
}

}  // namespace mkf
