// How the executors that march (band_march.cu, line_march.cu) cut their way into segments.
#pragma once
#include <algorithm>

namespace tf {

// n steps of each of `columns` independent columns, on `resident` workers: a segment of `len` steps costs len + lead, and
// columns * ceil(n / len) of them run in rounds of `resident`.  Returns the len with the least rounds * (len + lead), the
// longest of several; none below min_len but where n is.  Called in front of every launch, so it looks at one len per number of
// rounds, the least that needs no more of them, and stops where another round cannot pay: rounds * len is at least
// n * columns / resident.  (All len in turn took 14 us at n = 3 126, 1.2 ms at 262 144.)
inline int segment_length(int n, long long columns, long long resident, int lead, int min_len) {
  const long long most = min_len > 1 ? std::max(1, (n - 1) / (min_len - 1)) : n;  // segments
  const long long work = (n * columns + resident - 1) / resident;
  long long best = -1;
  int best_len = n;
  for (long long r = (columns + resident - 1) / resident; best < 0 || r * lead + work < best; ++r) {
    const long long segs = std::min(most, r * resident / columns);
    const int len = (int)((n + segs - 1) / segs);
    const long long rounds = (columns * ((n + len - 1) / len) + resident - 1) / resident, t = rounds * (len + lead);
    if (best < 0 || t < best) { best = t; best_len = len; }
    if (segs == most) break;
  }
  return best_len;
}

}  // namespace tf
