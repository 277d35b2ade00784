// copy_check.cu - the address arithmetic of the counting kernels' asynchronous copies, run on the host:
// every work item, tile, plane and lane of fields of many shapes, strides and offsets copies into a model
// of the shared-memory stage. No byte after the field may be read and none before the 16-byte block that it starts
// in, and every element must lie where the kernels read it. Prints "copy check ok".
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "words.cuh"

using namespace mkf;

static unsigned char stage[32 * 176];
static uintptr_t fieldLo, fieldHi;
static long long reads = 0;
static char what[256];

#define FAIL(...) do { printf("%s: ", what); printf(__VA_ARGS__); printf("\n"); exit(1); } while (0)

struct ModelCopy
{
   template <int BYTES>
   static __host__ __device__ void copy(uint32_t dst, const void *src, int n)
   {
#ifndef __CUDA_ARCH__
      const uintptr_t s = (uintptr_t)src;
      if (dst % BYTES || s % BYTES) { FAIL("misaligned copy of %d bytes", BYTES); }
      if (n < 0 || n > BYTES || dst + BYTES > sizeof(stage)) { FAIL("copy of %d of %d bytes to %u", n, BYTES, dst); }
      if (n > 0 && (s < (fieldLo & ~(uintptr_t)15) || s + n > fieldHi)) {
         FAIL("read of [%lld, %lld) of a field of %lld bytes", (long long)(s - fieldLo), (long long)(s + n - fieldLo), (long long)(fieldHi - fieldLo));
      }
      memcpy(stage + dst, src, n);
      memset(stage + dst + n, 0, BYTES - n);
      reads++;
#endif
   }
};

template <typename T>
struct Field
{
   std::vector<T> mem;
   const T *p;
   int64_t sx, sy, sz;
   int X, Y, Z;
   Field(int X_, int Y_, int Z_, int64_t sx_, int64_t sy_, int64_t sz_, int offset) : sx(sx_), sy(sy_), sz(sz_), X(X_), Y(Y_), Z(Z_)
   {
      const int64_t d[3] = {(X - 1) * sx, (Y - 1) * sy, (Z - 1) * sz};
      int64_t lo = 0, hi = 0;
      for (int64_t v : d) { (v < 0 ? lo : hi) += v; }
      mem.resize((size_t)(hi - lo + 1) + 64);
      for (size_t i = 0; i < mem.size(); i++) { mem[i] = (T)(i + 1); }
      const T *first = mem.data() + 16;
      while ((uintptr_t)first % 16) { first++; }
      first += offset;
      p = first - lo;
      fieldLo = (uintptr_t)first;
      fieldHi = (uintptr_t)(first + (hi - lo + 1));
   }
   T at(int x, int y, int z) const { return p[x * sx + y * sy + z * sz]; }
};

template <typename T, bool MIS>
static void checkWords(const Field<T> &f, bool vec, int D, int W)
{
   using G = RowGeom<T, MIS>;
   using Copier = RowCopier<T, MIS, ModelCopy>;
   WordTask a;
   memset(&a, 0, sizeof(a));
   a.f = f.p;
   a.sx = f.sx; a.sy = f.sy; a.sz = f.sz;
   a.X = f.X; a.Y = f.Y; a.Z = f.Z;
   a.K = 1;
   a.D = D;
   a.W = W;
   a.vec = vec;
   const int tiles = (f.X - 1 + G::EL - 1) / G::EL;
   a.nStripX = (tiles + W - 1) / W;
   a.nTileY = (f.Y - 1 + 30) / 31;
   a.nSlabZ = (f.Z - 1 + D - 1) / D;
   a.nItems = (long long)a.nStripX * a.nTileY * a.nSlabZ;
   std::vector<Copier> c(32);
   for (long long it = 0; it < a.nItems; it++) {
      const RowItem m = rowItemOf<G::EL>(a, it);
      for (int l = 0; l < 32; l++) { c[l].begin(a, m, l); }
      for (int p = 0; p <= m.nPln; p++) {
         for (int t = m.nT - 1; t >= 0; t--) {
            memset(stage, 0xAB, sizeof(stage));
            for (int l = 0; l < 32; l++) {
               if (!c[l].left()) { FAIL("no copies left at plane %d, tile %d", p, t); }
               c[l].copy(0, l);
            }
            for (int l = 0; l < 32; l++) {
               const int y = m.y0 + l < f.Y ? m.y0 + l : f.Y - 1, z = m.z0 + p, x0 = m.x0 + G::EL * t;
               const T *start = &f.p[x0 * f.sx + y * f.sy + z * f.sz];
               const int off = MIS ? (int)((uintptr_t)start & 15) : 0;
               const int n = G::EL + (t == m.nT - 1);  // with the element after the strip
               for (int i = 0; i < n; i++) {
                  T v;
                  memcpy(&v, stage + l * G::PITCH + off + i * (int)sizeof(T), sizeof(T));
                  const T want = x0 + i < f.X ? f.at(x0 + i, y, z) : T(0);
                  if (v != want) { FAIL("words item %lld plane %d tile %d row %d element %d", it, p, t, l, i); }
               }
            }
         }
      }
      if (c[0].left()) { FAIL("copies left over"); }
   }
}

template <typename T>
static void checkRing(const Field<T> &f, int D)
{
   using R = RingBlocks<T, ModelCopy>;
   FusedArgs a;
   memset(&a, 0, sizeof(a));
   a.f = f.p;
   a.sx = f.sx; a.sy = f.sy; a.sz = f.sz;
   a.X = f.X; a.Y = f.Y; a.Z = f.Z;
   a.D = D;
   a.nSegX = (f.X - 1 + 30) / 31;
   a.nTileY = (f.Y - 1 + 7) / 8;
   a.nSlabZ = (f.Z - 1 + D - 1) / D;
   a.nItems = (long long)a.nSegX * a.nTileY * a.nSlabZ;
   std::vector<R> r(32);
   for (long long it = 0; it < a.nItems; it++) {
      TmItem m;
      for (int l = 0; l < 32; l++) {
         m = itemOf<16 / (int)sizeof(T)>(a, it, l);
         r[l].begin(a, m, l);
      }
      for (int p = 0; p <= m.nPln; p++) {
         memset(stage, 0xAB, sizeof(stage));
         for (int l = 0; l < 32; l++) {
            if (p == m.nPln && R::atLast(a, m)) { r[l].copyLast(a, 0, l); }
            else { r[l].copy(a, 0, l); }
         }
         for (int j = 0; j < kTmRows; j++) {
            const T *start = &f.p[m.xa + m.xoff + (m.y0 + j) * f.sy + (m.z0 + p) * f.sz];
            for (int l = 0; l < 32; l++) {
               T v;
               memcpy(&v, stage + j * R::ROWB + ((uintptr_t)start & 15) + l * sizeof(T), sizeof(T));
               if (v != start[l]) { FAIL("ring item %lld plane %d row %d lane %d", it, p, j, l); }
            }
         }
      }
   }
}

template <typename T>
static void checkAll(const char *type)
{
   const int shapes[][3] = {{2, 2, 2}, {3, 3, 2}, {17, 5, 3}, {33, 32, 3}, {34, 33, 4}, {35, 40, 3}, {64, 31, 5}, {65, 63, 2}, {130, 9, 3}, {32, 9, 2}};
   for (const auto &s : shapes) {
      const int X = s[0], Y = s[1], Z = s[2];
      const int64_t views[][2] = {{X, (int64_t)X * Y}, {X + 1, (int64_t)(X + 1) * Y}, {X + 3, (int64_t)(X + 3) * (Y + 2) + 1}, {-(X + 2), (int64_t)(X + 2) * Y},
                                  {X, -(int64_t)X * Y - 1}, {-X, -(int64_t)X * Y}, {0, X}, {X, 0}, {1, X + Y}, {(int64_t)X * Z + 1, X}};
      for (const auto &v : views) {
         for (int offset = 0; offset < 4; offset++) {
            const Field<T> f(X, Y, Z, 1, v[0], v[1], offset);
            snprintf(what, sizeof(what), "%s %dx%dx%d strides 1 %lld %lld offset %d", type, X, Y, Z, (long long)v[0], (long long)v[1], offset);
            const bool blocks = blockRows(f, (int)sizeof(T));
            for (int W : {1, 3}) {
               for (int D : {1, 2, 64}) {
                  checkWords<T, true>(f, false, D, W);
                  checkWords<T, false>(f, false, D, W);
               }
            }
            if (X >= 32 && Y >= 9 && blocks) {
               for (int D : {1, 2, 64}) { checkRing<T>(f, D); }
            }
            const int64_t b = (int64_t)sizeof(T);
            if ((uintptr_t)f.p % 16 == 0 && v[0] * b % 16 == 0 && v[1] * b % 16 == 0) { checkWords<T, false>(f, true, 2, 2); }
            const Field<T> g(X, Y, Z, 2, 2 * v[0], 2 * v[1] + 1, offset);
            checkWords<T, false>(g, false, 2, 2);
            const Field<T> h(X, Y, Z, -1, v[0], v[1], offset);
            checkWords<T, false>(h, false, 2, 1);
         }
      }
   }
}

int main()
{
   checkAll<float>("FP32");
   checkAll<double>("FP64");
   printf("copy check ok: %lld copies\n", reads);
   return 0;
}
