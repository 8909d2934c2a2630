// strips.h -- how launches are cut into strips.
#pragma once

#include "kernels.cuh"

namespace fapk {

// Numbers the strips of a launch and chooses their length (in units of its
// numbering).
// CTAs of an SM share its issue slots, so the launch ends with the SM that got
// the most strips: their number rounded up, times a strip's cost (`unit` a unit
// and `start` for the staging of A), is made least over the lengths that
// give nearly every slot of the GPU (`per_sm` CTAs an SM) a strip; the shortest
// where none does.  Against the longest power of two with three strips an SM:
// 877 x 114,599 x 19 FP32 475 -> 439 us, 2,000 x 20,000 x 19 FP32 204 -> 181 us;
// counting turns of the slots instead takes 384 strips for 4,000 x 9,000 x 36
// packed, 203 us instead of 189 (576 strips).
// `strips` gives a job's strips of a length.
template <typename Job, typename Strips>
inline int number_strips(Job *segs, int nseg, int sm_count, int per_sm, int longest, int unit, int start, int *per,
                         Strips strips) {
  auto count = [&](int units) {
    long long n = 0;
    for (int i = 0; i < nseg; i++) n += strips(segs[i], units);
    return n;
  };
  long long best = -1;
  *per = 1;
  for (int units = 1; units <= longest; units++) {
    const long long n = count(units), cost = (n + sm_count - 1) / sm_count * (unit * units + start);
    if (n * 20 >= 17LL * per_sm * sm_count && (best < 0 || cost <= best)) best = cost, *per = units;
  }
  int n = 0;
  for (int i = 0; i < nseg; i++) {
    segs[i].strip_begin = n;
    n += strips(segs[i], *per);
  }
  return n;
}

}  // namespace fapk
