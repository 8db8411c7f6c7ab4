// Launch size classes of the autotuner and the choices kept for them. Plain C++.
#pragma once
#include <initializer_list>

namespace cgb {

// A tuned choice holds for the launches of one class: work items (32-instance tiles, times
// directions in the derivative sweeps) per SM up to 1, 2, 4, ... 64 and more for `few` tiles (at most
// 16 per SM, which the cooperative sweeps are for), up to 64 and more for more tiles. No class holds
// launches of both few and more tiles, whose candidates differ. Below one item per SM and above 64 the
// choice no longer depends on the size; in between each doubling changes how many warps or teams an SM
// holds (with one class from 16 up, the rollout's Jacobian of 65536 instances ran the variant that 4096
// had chosen, 8.2 ms in place of 5.8). The first call of a class times every candidate (the Jacobian:
// 15 ms where calls take 0.5 ms, 210 where they take 11), so there are no more of them: with a class
// for every power of two, first calls of 32, 64, ... 131072 instances took 0.72 s, now 0.44 s.
constexpr int kSizeClasses = 10;
inline int size_class(long long items, bool few, int sms) {
  int c = 0;
  while (c < 7 && items > static_cast<long long>(sms) << c) ++c;
  return few ? c : items <= 64ll * sms ? 8 : 9;
}

// The kept choice (-1: none) of class c, or of the nearest class with one, among those that `usable`
// accepts; -1: none.
template <class Choice, class F>
int kept_choice(const Choice (&row)[kSizeClasses], int c, F usable) {
  for (int d = 0; d < kSizeClasses; ++d)
    for (int k : {c - d, c + d})
      if (k >= 0 && k < kSizeClasses) {
        const int v = row[k];
        if (v >= 0 && usable(v)) return v;
      }
  return -1;
}

}  // namespace cgb
