// fused.cuh - arguments shared by the counting kernels (words.cuh, thermo.cu, thermo_tma.cu) and
// their routing (fused.cu).
#pragma once
#include <algorithm>
#include <utility>
#include <vector>
#include "mkf_common.cuh"

namespace mkf {

struct FusedArgs
{
   const void *f;
   int64_t sx, sy, sz;   // element strides
   int X, Y, Z;
   int K;                // thresholds in this pass (sorted ascending)
   int D;                // planes of cells per slab
   int nSegX, nTileY, nSlabZ;
   long long nItems;     // nSegX * nTileY * nSlabZ warp work items
   uint32_t nanRank;     // rank of a NaN element
   int rankHi;           // the rank counts thresholds <= f (else < f)
   int complement;       // stored codes are the bitwise complement of the true codes
   uint64_t *out;        // [.][256] distributions
   int outRow[MKF_MAX_THRESH];  // output row of sorted threshold k
   double tlo[64];       // sorted thresholds for the "f > t" test, +inf padded
   double thi[64];       // sorted thresholds for the "f >= t" test, +inf padded
   // thermometer kernel: order-preserving 32-bit keys of the thresholds it compares against
   // (the high word for FP64 fields), sorted, and the most thresholds sharing one bucket of the
   // 2^14-bucket rank table
   uint32_t tkey[MKF_MAX_THRESH];
   int lutC;
};


// One field of a batch, as the batched thermometer kernel reads it from device memory.
struct FieldTask
{
   const void *f;
   int64_t sx, sy, sz;
   int X, Y, Z, K, D, nSegX, nTileY, nSlabZ;
   long long nItems;
   uint32_t nanRank;
   int rankHi, complement, variant;  // variant: bit 0 ">=", bit 1 FP64, bit 2 shifted edge items, bit 3 lutC > 1
   int lutC, pad_;
   uint64_t *out;
   int outRow[MKF_MAX_THRESH];
   uint32_t tkey[MKF_MAX_THRESH];
   double tlo[64], thi[64];
};

// Most thresholds the word-parallel kernels take in one read (any relations).
#ifndef WORDS_MAX_K
#define WORDS_MAX_K 8
#endif
constexpr int kWordMaxK = WORDS_MAX_K;
constexpr int kWordMaxDepth = 64;  // planes of cells per work item (untuned)

// One field for the word-parallel kernels.
struct WordTask
{
   const void *f;
   int64_t sx, sy, sz;    // element strides
   int X, Y, Z;
   int K;                 // 1 .. kWordMaxK
   int mode[kWordMaxK];   // tests of the map: bit 0 "f > tlo", bit 1 "f < thi"
   int outRow[kWordMaxK];
   double tlo[kWordMaxK], thi[kWordMaxK];  // exact-equivalent thresholds of the two tests
   uint32_t inv;          // bit k: threshold k is counted negated, code c is stored in bin 255 - c
   int vec;               // rows and planes on 16-byte boundaries, unit x stride
   uint64_t *out;
   double *mom;           // moments kernel: [K][2 map values][sum f, sum f^2]
   int D, W;              // planes of cells and tiles in x (words.cuh) per work item
   int nStripX, nTileY, nSlabZ, pad_;
   long long nItems;
};

// Consecutive work items [begin, end) of one field.
struct BatchChunk
{
   int field, pad_;
   long long begin, end;
};

// Cut a batch's fields (tasks of one kernel) into chunks. A CTA waits for its slowest warp at the end
// of a chunk and fills its copy pipeline anew at the start, so chunks are as long as leaves every one
// of `ctas` CTAs about four of them, in multiples of the warps that count it, and the costliest come first:
// with chunks of 64 items, 64 served fields gave 29 and 65 chunks to 148 SMs (733 and 638 us). cost: of an
// item of a task; warps: of a CTA that count items of a task; at most maxRounds items each.
template <typename TASK, typename COST, typename WARPS>
std::vector<BatchChunk> cutChunks(const std::vector<TASK> &tasks, int ctas, int maxRounds, COST cost, WARPS warpsOf)
{
   double total = 0.0;
   for (const TASK &t : tasks) { total += (double)t.nItems * cost(t); }
   std::vector<std::pair<double, int>> order;
   for (size_t f = 0; f < tasks.size(); f++) { order.push_back({-cost(tasks[f]), (int)f}); }
   std::stable_sort(order.begin(), order.end());
   std::vector<BatchChunk> chunks;
   for (const auto &o : order) {
      const TASK &t = tasks[o.second];
      const int warps = warpsOf(t);
      long long n = (long long)(total / (4.0 * ctas) / -o.first / warps + 0.5);
      n = (n < 1 ? 1 : n > maxRounds ? maxRounds : n) * warps;
      for (long long b = 0; b < t.nItems; b += n) { chunks.push_back({o.second, 0, b, b + n < t.nItems ? b + n : t.nItems}); }
   }
   return chunks;
}

struct BatchArgs
{
   const FieldTask *tasks;
   const BatchChunk *chunks;
   int nChunks;
   unsigned *counter;  // next chunk to hand out; zero at launch
};

struct WordBatchArgs
{
   const WordTask *tasks;
   const BatchChunk *chunks;
   int nChunks;
   unsigned *counter;  // next chunk to hand out; zero at launch
};

struct ConstEntry { int row, bin; };

// A threshold set split into constant maps and varying thresholds (indices into the set, sorted by
// value). cls: the relation all varying ones share (0 >, 1 >=, 2 <, 3 <=), negative when they differ
// or it is = or !=.
struct ThreshSplit
{
   int n, nConst, cls;
   int idx[MKF_MAX_THRESH], constIdx[MKF_MAX_THRESH], constBin[MKF_MAX_THRESH];
};
void splitThresholds(const MKFThreshSet *pT, ThreshSplit &q);
// Count the varying thresholds of a split, adding to out (no allocation, no clearing).
int countVarying(uint64_t *out, const MKFFieldDesc *pF, const MKFThreshSet *pT, const ThreshSplit &q, cudaStream_t s);
// Add `cells` to bin `bin` of output row `row`.
int launchConstBin(uint64_t *out, int row, int bin, unsigned long long cells, cudaStream_t s);
void floatBoundsPlain(double t, double &tlo, double &thi);
// Count one field for any thresholds (fused.cu).
int fieldBPFD(uint64_t *out, const MKFFieldDesc *pF, const MKFThreshSet *pT, int flags, cudaStream_t s);

enum { kPlanSingle = 0, kPlanThermo = 1, kPlanWords = 2 };
// The fields of a batch that either batched kernel could count, by element type, and which of them does.
struct BatchMix
{
   bool words[2] = {false, false};  // some field needs the word kernel: 1 or 2 thresholds, or relations that differ
   int fields[2] = {0, 0};          // the others of up to kWordMaxK thresholds: their number,
   double voxels[2] = {0.0, 0.0}, thresholds[2] = {0.0, 0.0};  // voxels, and thresholds times voxels
   void add(const MKFFieldDesc *pF, const MKFThreshSet *pT);
   int wordMax(int enc, int depth) const;  // most thresholds of one relation for the word kernel
};
// depth: planes of cells per work item; 0 = each kernel's default, -1 = chosen by field size.
int planBatchField(const MKFFieldDesc *pF, const MKFThreshSet *pT, int row0, FieldTask &t, WordTask &w,
                   std::vector<ConstEntry> &consts, bool &anyVarying, int wordMax, int depth);

// Slab depth (planes of cells per work item) of a single-field launch of kernel family `family`
// (tune.cu): the depth mkfTune measured best for this kind of field, else `def`. A family is one kernel
// with one way of reading the field, so that what was measured on it is used by it only: the word kernel
// on aligned rows, on others and with strided x; the vote kernel; the rank table read from global memory;
// the staged rank table filled by TMA (also with thresholds sharing buckets), by blocks and by elements.
enum { kFamWords, kFamWordsBlocks, kFamWordsElems, kFamBallot, kFamThermo, kFamThermoTma, kFamThermoTmaShared,
       kFamThermoBlocks, kFamThermoElems, kNumFamilies };
static constexpr int kTmNumVariants = 4;  // variants of the TMA rank-table kernel (thermo_tma.cu)
int tunedDepth(int family, int enc, int K, int X, int Y, int Z, int def);
// Kernel variant (CTA shape, histogram copies) of such a launch: the one mkfTune measured best for
// this kind of field, else `def`. Families without variants use 0.
int tunedVariant(int family, int enc, int K, int X, int Y, int Z, int def);
// The untuned slab depth: def halved (down to 4) until a field of itemsPerPlane work items per
// plane and Z planes has at least minItems items.
int sizeDepth(int def, long long itemsPerPlane, int Z, long long minItems);
// Whether mkfBatchPlanCreate measures the slab depth of each new plan (tune.cu).
bool batchTuning();

// Fill a task's key table and item grid; false if its thresholds share a rank-table bucket.
bool prepareThermoTask(FieldTask &t, int enc, int depth = 0);
// Launch the batched thermometer kernel over tasks of one element type (enc) whose largest
// threshold count is maxK.
// Chunks of one kernel variant of the batched rank-table kernel: [c0, c1) of the sorted chunk list.
struct ThermoGroup
{
   int variant, c0, c1, maxK;
};
static constexpr int kThVariants = 16;  // variant indices 0..15 (FieldTask::variant & 13 is used)
// Sort a batch's chunks by their field's variant (stable within a variant) and return the groups.
std::vector<ThermoGroup> groupThermoChunks(std::vector<BatchChunk> &chunks, const std::vector<FieldTask> &tasks);
// One launch per group; counters[v] (zeroed beforehand) hands out the chunks of variant v.
int launchThermoGroups(const FieldTask *dTasks, const BatchChunk *dChunks, const std::vector<ThermoGroup> &groups,
                       unsigned *counters, int enc, cudaStream_t s);

// Fill a word task's field and its thresholds k0 .. k0 + n of a split (rows from row0).
void fillWordTask(WordTask &w, const MKFFieldDesc *pF, const MKFThreshSet *pT, const ThreshSplit &q, int k0, int n, int row0);
// Word tasks (words.cu): threshold t with relation mask m as the k-th of a task (inv zeroed
// beforehand) whose counts go to output row `row`; the item grid for a slab depth and strip width.
void fillWordThresh(WordTask &a, int k, int enc, double t, uint32_t m, int row);
bool wordRowsAligned(const WordTask &a, int enc);  // unit x stride, rows and planes on 16-byte boundaries
void fillWordGrid(WordTask &a, int enc, int depth, int strip);

// Count one field for a task's thresholds, 1 .. kWordMaxK of any relations (words.cu; fills the
// task's item grid).
int launchWords(WordTask &a, int enc, cudaStream_t s);

// The same by warp votes, for one threshold or a few of one test; whether it is the faster one
// (ballot.cu).
int launchBallots(WordTask &a, int enc, cudaStream_t s);
bool useBallots(const WordTask &a, int enc);

// Counts and descriptive moments of one or two thresholds (any relations) in one read (words.cu):
// a.mom is device double[K][2][2], per threshold and map value the sum of f and of f^2.
int launchWordsMoments(WordTask &a, int enc, cudaStream_t s);

// Chunks of the batched kernels' tasks (words_batch.cu, thermo.cu).
std::vector<BatchChunk> wordChunks(const std::vector<WordTask> &tasks, int enc);
std::vector<BatchChunk> thermoChunks(const std::vector<FieldTask> &tasks);
// The batched word kernel over the chunks of tasks of one element type (words_batch.cu).
int launchWordsBatch(const WordBatchArgs &b, int enc, cudaStream_t s);

// Whether a pass's field and threshold count suit the TMA-staged rank-table kernel (thermo_tma.cu):
// 3..16 thresholds, unit x stride, rows and planes on 16-byte boundaries, X >= 32, Y >= 9.
bool tmaRowsAligned(const FusedArgs &a, int enc);

// Launch the thermometer kernel for a pass whose thresholds all share one relation
// (< <= > >=); fills the key table of `a` first.
int launchThermo(FusedArgs &a, int enc, cudaStream_t s);

}  // namespace mkf
