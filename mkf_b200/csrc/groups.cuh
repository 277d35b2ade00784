// groups.cuh - the symmetry groups of the 256 cell patterns and their weights in the four measures.
#pragma once
#include <stdint.h>

namespace mkf {

// Symmetry group of each 2x2x2 pattern under the 48 symmetries of the cube, numbered as the
// original numbers them (mkfUtil.c:40-58, generated by c8sGetMap cell8Sym.c:341-363).
constexpr uint8_t kGroupOf[256] = {
   0,  1,  1,  2,  1,  2,  3,  5,  1,  3,  2,  5,  2,  5,  5,  8,
   1,  2,  3,  5,  3,  5,  7,  9,  4,  6,  6,  10, 6,  10, 13, 16,
   1,  3,  2,  5,  4,  6,  6,  10, 3,  7,  5,  9,  6,  13, 10, 16,
   2,  5,  5,  8,  6,  10, 13, 16, 6,  13, 10, 16, 11, 15, 15, 19,
   1,  3,  4,  6,  2,  5,  6,  10, 3,  7,  6,  13, 5,  9,  10, 16,
   2,  5,  6,  10, 5,  8,  13, 16, 6,  13, 11, 15, 10, 16, 15, 19,
   3,  7,  6,  13, 6,  13, 11, 15, 7,  12, 13, 14, 13, 14, 15, 18,
   5,  9,  10, 16, 10, 16, 15, 19, 13, 14, 15, 18, 15, 18, 17, 20,
   1,  4,  3,  6,  3,  6,  7,  13, 2,  6,  5,  10, 5,  10, 9,  16,
   3,  6,  7,  13, 7,  13, 12, 14, 6,  11, 13, 15, 13, 15, 14, 18,
   2,  6,  5,  10, 6,  11, 13, 15, 5,  13, 8,  16, 10, 15, 16, 19,
   5,  10, 9,  16, 13, 15, 14, 18, 10, 15, 16, 19, 15, 17, 18, 20,
   2,  6,  6,  11, 5,  10, 13, 15, 5,  13, 10, 15, 8,  16, 16, 19,
   5,  10, 13, 15, 9,  16, 14, 18, 10, 15, 15, 17, 16, 19, 18, 20,
   5,  13, 10, 15, 10, 15, 15, 17, 9,  14, 16, 18, 16, 18, 19, 20,
   8,  16, 16, 19, 16, 19, 18, 20, 16, 18, 19, 20, 19, 20, 20, 21 };

// Per-group weights of the original: Euler gWK (mkfUtil.c:33-38), surface gWS and mean
// curvature gWM (mkfHacks.c:9-20).
constexpr int kWK[22] = { 0, 3, 0, 6, 6, -3, 3, 9, 0, -6, -6, 0, 12, 0, -3, -8, -3, -12, -6, 0, 3, 0 };
constexpr double kWS[22] = {
   0, 0.944412, 1.05178, 0.921095, 0.496906, 0.949947, 0.865898, 0.793181, 0.926631, 0.638921, 0.764068,
   0.784616, 0.874463, 0.868666, 0.557639, 0.682786, 0.923863, 0.496906, 0.737983, 0.65947, 0.0812817, 0 };
constexpr double kWM[22] = {
   0, 0.763019, 0.642656, 0.616236, 0.686801, 0.187756, 0.167269, 0.161335, 0, -0.431447, -0.287632,
   0, 0, -0.143816, -0.592783, -0.540019, -0.475387, -0.686801, -0.616236, -0.727774, -0.331571, 0 };

// The same for the device: the patterns sorted by group (group q holds member[first[q]] ..
// member[first[q + 1] - 1]) and the weights. Constant data of the module, so that it is there in every
// context, also in one made after a device reset.
struct GroupTables
{
   uint8_t member[256];
   int first[23];
   int wK[22];
   double wS[22], wM[22];
};
constexpr GroupTables groupTables()
{
   GroupTables t = {};
   int n = 0;
   for (int q = 0; q < 22; q++) {
      t.first[q] = n;
      for (int c = 0; c < 256; c++) {
         if (kGroupOf[c] == q) { t.member[n++] = (uint8_t)c; }
      }
      t.wK[q] = kWK[q];
      t.wS[q] = kWS[q];
      t.wM[q] = kWM[q];
   }
   t.first[22] = n;
   return t;
}

}  // namespace mkf
