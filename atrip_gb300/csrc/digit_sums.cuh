// Whether sums of digit products are exact in FP32 accumulators, in whatever
// order they are formed.  Plain C++.
#pragma once

#include <cmath>

namespace atrip_gb300 {

constexpr int kNormSlices = 7;  // digits 0..6

// The largest sum of q_s^2 over a row (or column) of an operand, per digit s.
struct DigitNorms {
  double q2[kNormSlices];
};

// An accumulator of level L adds up q_s q'_(L-s), s <= L, along `terms`
// particle contractions (norms nT, nV) and as many hole contractions (nH, nU).
// By Cauchy and Schwarz the magnitudes of what it adds come to at most
//     B = terms sum_s (sqrt(nT_s nV_(L-s)) + sqrt(nH_s nU_(L-s))).
// A partial sum P of a whole sum S has |P| <= (B + |S|) / 2, as |P| + |S - P|
// <= B; it is exact below 2^24.  Levels above 0 are checked to end at |S| <
// 2^22 and are exact for B < 2^25 - 2^22; the limit leaves 2^16 for what
// roundings could have done to the S that is checked.  Level 0 is not checked
// and needs B < 2^24.
//
// loose: level 6 may have B < 2^26 - 2^22 - 2^16.  Its partial sums then stay
// below 2^25, where each of its 7 K additions is rounded by at most 2: 14 K
// units of 2^-62 of the grids' largest product, below half of K 2^-53 of one
// that is within 2^4 of it.
inline bool level_sums_exact(int terms, const DigitNorms &nT, const DigitNorms &nV,
                             const DigitNorms &nH, const DigitNorms &nU, bool loose = false) {
  for (int L = 0; L < kNormSlices; ++L) {
    double b = 0;
    for (int s = 0; s <= L; ++s)
      b += std::sqrt(nT.q2[s] * nV.q2[L - s]) + std::sqrt(nH.q2[s] * nU.q2[L - s]);
    const double end = 0x1p22 + 0x1p16;
    const double most = L == 0 ? 0x1p24 : (loose && L == 6 ? 0x1p26 : 0x1p25) - end;
    if (!(terms * b < most)) return false;
  }
  return true;
}

}  // namespace atrip_gb300
