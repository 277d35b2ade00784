// words_batch.cu - many fields in one launch of the word-parallel counting kernel (words.cuh).
#include <algorithm>
#include "words.cuh"

namespace mkf {

// A CTA takes chunks of consecutive work items from a global counter; chunks never span fields.
// When the next chunk belongs to another field, the CTA adds its counts of the previous field to
// that field's output rows first.
template <typename T>
__global__ void __launch_bounds__(kWdWarps * 32, 1) wordBatch(const __grid_constant__ WordBatchArgs b)
{
   __shared__ RowShared S;
   __shared__ WordTask F;
   __shared__ int sChunk;
   extern __shared__ __align__(16) unsigned char dyn[];
   const int warp = __shfl_sync(FULL, threadIdx.x >> 5, 0);
   int cur = -1;
   for (;;) {
      if (threadIdx.x == 0) { sChunk = (int)atomicAdd(b.counter, 1u); }
      __syncthreads();
      const int c = sChunk;
      if (threadIdx.x == 0) { S.next = 0; }  // (every warp is past the last chunk's items)
      __syncthreads();
      if (c >= b.nChunks) { break; }
      const BatchChunk ch = b.chunks[c];
      if (ch.field != cur) {
         if (cur >= 0) {
            rowFlush(F, S);
            __syncthreads();
         }
         const uint32_t *src = reinterpret_cast<const uint32_t *>(b.tasks + ch.field);
         for (int i = threadIdx.x; i < (int)(sizeof(WordTask) / 4); i += blockDim.x) {
            reinterpret_cast<uint32_t *>(&F)[i] = src[i];
         }
         __syncthreads();
         rowSetup(F, S);
         cur = ch.field;
      }
      // fields with unit x stride are read as if no row were aligned (aligned ones too: most fields of
      // a batch are not, and one form keeps the kernel small)
      const uint32_t mem = (uint32_t)__cvta_generic_to_shared(dyn);
      const bool mis = F.sx == 1;
      const int bytes = wordWarpBytes(RowGeom<T, true>::NR, F.K, F.W, mis);
      const auto item = [&](int j) { return ch.begin + j; };
      if (warp < wordBatchWarps(RowGeom<T, true>::NR, F.K, F.W, mis)) {
         if (!mis) { rowItems<T, false, 0, false>(F, item, ch.end, mem + (uint32_t)(warp * bytes), S); }
         else if (F.K == 1) { rowItems<T, false, 1, true>(F, item, ch.end, mem + (uint32_t)(warp * bytes), S); }
         else { rowItems<T, false, 0, true>(F, item, ch.end, mem + (uint32_t)(warp * bytes), S); }
      }
   }
   if (cur >= 0) { rowFlush(F, S); }
}

std::vector<BatchChunk> wordChunks(const std::vector<WordTask> &tasks, int enc)
{
   // tiles of an item, each about half a threshold's work before the thresholds'
   return cutChunks(tasks, smCount(), 16, [](const WordTask &t) { return (t.D + 1.0) * t.W * (t.K + 0.5); },
                    [enc](const WordTask &t) { return wordBatchWarps(enc == ENC_F32 ? 4 : 2, t.K, t.W, t.sx == 1); });
}

template <typename T>
static int launchBatchT(const WordBatchArgs &b, cudaStream_t s)
{
   static SmemAllowed allowed;
   auto kern = wordBatch<T>;
   allowSmem(allowed, kern, kWdDynBytes);
   long long grid = smCount();
   if (grid > b.nChunks) { grid = b.nChunks; }
   if (grid < 1) { grid = 1; }
   kern<<<(unsigned)grid, kWdWarps * 32, kWdDynBytes, s>>>(b);
   return cudaFail(cudaGetLastError(), "wordBatch launch");
}

int launchWordsBatch(const WordBatchArgs &b, int enc, cudaStream_t s)
{
   return enc == ENC_F32 ? launchBatchT<float>(b, s) : launchBatchT<double>(b, s);
}

}  // namespace mkf
