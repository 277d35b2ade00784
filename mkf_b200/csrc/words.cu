// words.cu - single-field launches of the word-parallel counting kernel (words.cuh), for one to
// kWordMaxK thresholds of any relations, optionally with the field's moments per map value
// from the same read.
#include <algorithm>
#include <cmath>
#include "words.cuh"

namespace mkf {

template <typename T, bool MOM, int KT, bool MIS>
__global__ void __launch_bounds__(kWdWarps * 32, 1) wordBPFD(const __grid_constant__ WordTask a)
{
   __shared__ RowShared S;
   extern __shared__ __align__(16) unsigned char dyn[];
   rowSetup(a, S);
   const int warp = __shfl_sync(FULL, threadIdx.x >> 5, 0), warps = blockDim.x >> 5;
   // in round r the CTA's items are (r gridDim + blockIdx) warps .., so the whole grid works on
   // neighbouring strips
   rowItems<T, MOM, KT, MIS>(a, [&](int j) { return ((long long)(j / warps) * gridDim.x + blockIdx.x) * warps + j % warps; }, a.nItems,
                            (uint32_t)__cvta_generic_to_shared(dyn) + (uint32_t)(warp * wordWarpBytes(RowGeom<T, MIS>::NR, a.K, a.W, MIS)), S);
   rowFlush(a, S);
   if (MOM && threadIdx.x < a.K * 4) {
      const int k = threadIdx.x >> 2, b = (threadIdx.x >> 1) & 1, q = threadIdx.x & 1;
      const double x = S.mom[k][b][q];
      if (x != 0.0) { atomicAdd(a.mom + k * 4 + (b ^ ((a.inv >> k) & 1)) * 2 + q, x); }
   }
}

void fillWordThresh(WordTask &a, int k, int enc, double t, uint32_t m, int row)
{
   m &= BMC_AL;
   if (enc == ENC_F32) { floatBoundsPlain(t, a.tlo[k], a.thi[k]); }
   else { a.tlo[k] = a.thi[k] = t; }
   // tests f > t (G) and f < t (L); the map is a test, both, or the complement (counted negated,
   // which also maps NaN as "equal")
   switch (m) {
      case 0: a.mode[k] = 0; break;  // (constant maps: the moments kernel only)
      case BMC_AL: a.mode[k] = 0; a.inv |= 1u << k; break;
      case BMC_GT: a.mode[k] = 1; break;
      case BMC_LT | BMC_EQ: a.mode[k] = 1; a.inv |= 1u << k; break;
      case BMC_LT: a.mode[k] = 2; break;
      case BMC_GT | BMC_EQ: a.mode[k] = 2; a.inv |= 1u << k; break;
      case BMC_EQ: a.mode[k] = 3; a.inv |= 1u << k; break;
      default: a.mode[k] = 3; break;  // < or >
   }
   a.outRow[k] = row;
}

bool wordRowsAligned(const WordTask &a, int enc)
{
   const int64_t b = enc == ENC_F32 ? 4 : 8;
   return a.sx == 1 && ((uintptr_t)a.f % 16) == 0 && (a.sy * b) % 16 == 0 && (a.sz * b) % 16 == 0;
}

void fillWordGrid(WordTask &a, int enc, int depth, int strip)
{
   const int el = enc == ENC_F32 ? 32 : 16;
   a.vec = wordRowsAligned(a, enc);
   const int tiles = (a.X - 1 + el - 1) / el;
   a.W = strip;
   a.nStripX = (tiles + strip - 1) / strip;
   a.nTileY = (a.Y - 1 + 30) / 31;
   a.D = depth < 1 ? 1 : depth;
   a.nSlabZ = (a.Z - 1 + a.D - 1) / a.D;
   a.nItems = (long long)a.nStripX * a.nTileY * a.nSlabZ;
}

// Warps per CTA whose shared memory fits strips of W tiles.
static int wordWarps(int enc, int K, int W, bool mis)
{
   return std::min(kWdWarps, kWdDynBytes / wordWarpBytes(enc == ENC_F32 ? 4 : 2, K, W, mis));
}

// Planes per work item and tiles per strip; tuned: the planes are given (0: chosen too).
static void wordGrid(const WordTask &a, int enc, bool mis, int ctas, int tuned, int &depth, int &strip)
{
   // Cost of a grid, fitted to sweeps of depth and strip over 256^3 to 128 x 2048^2 fields with one
   // and three thresholds (the choice is within 5 % of the best swept). The busiest warp's tiles:
   // rounds of items of (D + 1) planes (one is the halo) of W tiles, and about one tile's time to start
   // each. The element after each strip's rows costs a memory burst where the field does not stay in L2
   // (512^3 FP32, one threshold: W = 1 143 us, 2 122, 4 107, 8 106; three thresholds, bound by their
   // arithmetic: 239, 219), and wide strips leave room for fewer warps.
   const int el = enc == ENC_F32 ? 32 : 16;
   const int chunks = (a.X - 1 + el - 1) / el, cellsZ = a.Z - 1;
   const long long tiles = (a.Y - 1 + 30) / 31;
   const double burst = 128.0 * chunks * a.Y * a.Z > 32e6 ? 0.7 / a.K : 0.0;
   double best = 0.0;
   depth = strip = 1;
   const int maxW = std::min(chunks, 8);
   for (int w = maxW;; w = (w + 1) / 2) {
      const int strips = (chunks + w - 1) / w, W = (chunks + strips - 1) / strips;
      const int perCta = wordWarps(enc, a.K, W, mis);
      const long long warps = (long long)ctas * perCta;
      auto consider = [&](long long r, int d) {
         const double cost = (double)r * ((d + 1) * W + 1) * (1.0 + burst / W) * std::sqrt((double)perCta / kWdWarps);
         if (best == 0.0 || cost < best) {
            best = cost;
            depth = d;
            strip = W;
         }
      };
      if (tuned > 0) {
         consider((strips * tiles * ((cellsZ + tuned - 1) / tuned) + warps - 1) / warps, tuned);
      }
      for (int r = 1; r <= 16 && tuned == 0; r++) {
         // the shallowest slabs that r rounds take
         const long long slabs = std::min<long long>(cellsZ, r * warps / (strips * tiles));
         if (slabs < 1) { continue; }
         const int d = (int)((cellsZ + slabs - 1) / slabs);
         if (d <= kWordMaxDepth) { consider(r, d); }
      }
      if (w == 1) { break; }
   }
   if (best == 0.0) {  // more than 16 rounds of the deepest items
      depth = kWordMaxDepth;
      strip = std::min(chunks, 4);
   }
}

template <typename T, bool MOM, int KT, bool MIS>
static int launchWordsT(WordTask &a, int enc, cudaStream_t s)
{
   static SmemAllowed allowed;
   auto kern = wordBPFD<T, MOM, KT, MIS>;
   allowSmem(allowed, kern, kWdDynBytes);
   int depth, strip;
   const int family = MIS ? kFamWordsBlocks : a.vec ? kFamWords : kFamWordsElems;
   wordGrid(a, enc, MIS, smCount(), MOM ? 0 : tunedDepth(family, enc, a.K, a.X, a.Y, a.Z, 0), depth, strip);
   fillWordGrid(a, enc, depth, strip);
   const int warps = wordWarps(enc, a.K, a.W, MIS);
   const long long grid = std::min<long long>((a.nItems + warps - 1) / warps, smCount());
   kern<<<(unsigned)grid, warps * 32, warps * wordWarpBytes(RowGeom<T, MIS>::NR, a.K, a.W, MIS), s>>>(a);
   return cudaFail(cudaGetLastError(), "wordBPFD launch");
}

template <typename T, bool MIS>
static int dispatchWords(WordTask &a, int enc, cudaStream_t s)
{
   switch (a.K) {
      case 1: return launchWordsT<T, false, 1, MIS>(a, enc, s);
      case 2: return launchWordsT<T, false, 2, MIS>(a, enc, s);
      case 3: return launchWordsT<T, false, 3, MIS>(a, enc, s);
      case 4: return launchWordsT<T, false, 4, MIS>(a, enc, s);
      default: return launchWordsT<T, false, 0, MIS>(a, enc, s);
   }
}

int launchWords(WordTask &a, int enc, cudaStream_t s)
{
   if (a.K < 1 || a.K > kWordMaxK) { setError("word kernel: %d thresholds", a.K); return MKF_ERR_UNSUPPORTED; }
   fillWordGrid(a, enc, 1, 1);
   const bool mis = a.sx == 1 && !a.vec;
   if (enc == ENC_F32) { return mis ? dispatchWords<float, true>(a, enc, s) : dispatchWords<float, false>(a, enc, s); }
   return mis ? dispatchWords<double, true>(a, enc, s) : dispatchWords<double, false>(a, enc, s);
}

template <typename T>
static int dispatchMoments(WordTask &a, int enc, cudaStream_t s)
{
   return a.K == 1 ? launchWordsT<T, true, 1, false>(a, enc, s) : launchWordsT<T, true, 2, false>(a, enc, s);
}

int launchWordsMoments(WordTask &a, int enc, cudaStream_t s)
{
   if (a.K < 1 || a.K > 2 || a.X < 2 || a.Y < 2 || a.Z < 2) { return MKF_ERR_UNSUPPORTED; }
   return enc == ENC_F32 ? dispatchMoments<float>(a, enc, s) : dispatchMoments<double>(a, enc, s);
}

}  // namespace mkf
