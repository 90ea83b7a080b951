// hw_slices.hpp -- grid points per CTA (the slice) of every member of a context, where
// the caller names none.
#pragma once

#include <algorithm>
#include <vector>

namespace hw {

// 2048 points fill the GPU best when there are members for every SM.  When there are
// not, a member's time is its CTA's, and smaller slices put more SMs on it, as long as few
// SMs are given two CTAs: 512 points up to eight CTAs, 1024 up to sixteen.  Grids of up to
// 1024 points stay in one CTA, where no step crosses the cluster.  One member, us an RHS in
// slices of 2048, 1024, 512 and 256 points: flat HS2 of 2048 points 27 27 24 24, of 4096
// 37 28 24 30, of 8192 39 28 30, of 16384 41 36; HS3 on a slope (sixteen reference depths)
// of 4096 367 275 253 302, of 8192 395 303 302, of 16384 430 359; flat of 1024 in one CTA
// 20, in two 24.  Slices of 512 points may use every SM once, of 1024 points put a second
// CTA on a quarter of them (148 and 185 CTAs of B200's 148 SMs).  Runs in slices of 1024 and
// of 2048 points, by the CTAs of 1024, ms: random bathymetries with sixteen references 164
// 62 71, 172 67 72, 188 68 74, 196 70 75, 212 74 76, 216 75 76, 224 82 77; flat tanks 156
// 10.3 11.8, 180 10.6 11.8, 188 11.4 11.8, 210 11.6 11.8, 226 11.8 11.9.  The line is short of
// where the two meet (216 to 224) by what one more large member moves the count.
//
// nx: the members' grids; named: their slices where the caller gave them (0: not); sms:
// the device's SMs; sixteen(M): whether a cluster of sixteen CTAs of M points can be
// resident (more than eight are beyond what every device of the architecture promises).
template <class Sixteen>
std::vector<int> choose_slices(const std::vector<int>& nx, const std::vector<int>& named, int sms,
                               const Sixteen& sixteen) {
  const size_t n = nx.size();
  std::vector<int> m(n);
  for (int least = 512; least <= 2048; least *= 2) {
    long long ctas = 0;
    for (size_t i = 0; i < n; ++i) {
      const int N = nx[i];
      m[i] = named[i] > 0 ? named[i]
                          : (N <= 1024 ? N : std::min(2048, std::max({least, N / 16, std::min(N / 8, 1024)})));
      if (named[i] <= 0 && N / m[i] > 8 && m[i] < 2048 && !sixteen(m[i])) m[i] = std::min(2048, N / 8);
      ctas += std::max(1, N / m[i]);
    }
    if (ctas <= (least == 512 ? sms : sms + sms / 4)) break;
  }
  return m;
}

}  // namespace hw
