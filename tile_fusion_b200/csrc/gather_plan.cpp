// Host side of the balanced gather (gather.cu): cutting the nonzeros of an operator into units of about equal work.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "gather.h"
#include "tf_internal.h"

namespace tf {

void build_gather_plan(int m, const int *ap, int groups, bool ticket_sums, GatherPlan &out) {
  out = GatherPlan();
  const long long nnz = ap[m];
  const long long cost = nnz + 2LL * m;
  // As many units as make whole rounds of the resident groups, of at most about 256 nonzeros: units take about equally long,
  // so a round that only some groups have a unit in costs a whole one.  Shorter units spend their time on the three dependent
  // reads in front of the first product (R-MAT n = 200 000, degree 20, 64 columns, both products: 192 us with 128, 183 with
  // 256, 253 with 512, before the rounds were whole), so at least 32.  A unit is closed by the row that does not fit any more:
  // half a row's cost, and three hundredths for luck, keep the last round from spilling over.
  const double share = (double)cost / std::max(1, groups), rounds = std::max(1.0, std::ceil(share / 256));
  const int target = (int)std::max(32.0, std::ceil(share / rounds * 1.03 + 0.5 * cost / std::max(1, m)));
  // A row at least this long is cut.  (Cutting only from twice that on: the same on large graphs, 25.4 instead of 22.7 us
  // at n = 20 000, where one long row is what the launch waits for.)
  const int long_row = ticket_sums ? kHeavyRowNnz : target;
  using Range = GatherPlan::Range;
  std::vector<Range> plain, &pieces = out.ranges;
  int pos = 0, open_cost = 0;
  Range open{0, 0, 0, -1};
  auto close = [&] {
    if (open_cost > 0) plain.push_back(open);
    open_cost = 0;
  };
  for (int r = 0; r < m; ++r)
    if (ap[r + 1] == ap[r]) out.empty_rows.push_back(r);
  const bool listed = !out.empty_rows.empty();
  for (int r = 0; r < m; ++r) {
    const int len = ap[r + 1] - ap[r];
    if (len == 0) continue;
    if (listed) out.rows.push_back(r);
    if (len >= long_row) {
      close();
      const int first_slot = out.n_slots;
      auto piece_of = [&](int j0, int j1) { pieces.push_back(Range{out.n_slots++, j0, j1, (int)out.heavy.size()}); };
      if (ticket_sums) {
        // the ticket executor gives such a row to the 16 warps of a CTA in runs of whole 32 nonzeros, one beyond kSegmentNnz
        // to several CTAs, each its segment
        const int n_seg = (len + kSegmentNnz - 1) / kSegmentNnz, seg = (len + n_seg - 1) / n_seg;
        for (int s0 = ap[r]; s0 < ap[r + 1]; s0 += seg) {
          const int s1 = std::min(ap[r + 1], s0 + seg), per = ((s1 - s0 + 15) / 16 + 31) / 32 * 32;
          for (int j = s0; j < s1; j += per) piece_of(j, std::min(s1, j + per));
        }
      } else {
        // pieces of about sqrt(len): the group that adds them up last reads as many partial rows as a piece has gathers
        const int piece = std::max(target, std::min(512, (int)std::sqrt((double)len)));
        const int n = (len + piece - 1) / piece;
        for (int k = 0; k < n; ++k) piece_of(ap[r] + (int)((long long)len * k / n), ap[r] + (int)((long long)len * (k + 1) / n));
      }
      out.heavy.push_back(GatherHeavy{r, first_slot, out.n_slots - first_slot, 0});
    } else {
      if (open_cost > 0 && open_cost + len + 2 > target) close();
      if (open_cost == 0) open = Range{pos, ap[r], ap[r], -1};
      open.j1 = ap[r + 1];
      open_cost += len + 2;
    }
    ++pos;
  }
  close();
  // long rows in order of length, longest first, so that their additions at the end are not what the launch waits for
  std::stable_sort(pieces.begin(), pieces.end(),
                   [&](const Range &a, const Range &b) { return out.heavy[a.heavy].n_slots > out.heavy[b.heavy].n_slots; });
  pieces.insert(pieces.end(), plain.begin(), plain.end());

  out.units.resize(pieces.size());
  size_t n = 0;
  for (size_t i = 0; i < pieces.size(); ++i) {
    const int batches = (pieces[i].j1 - pieces[i].j0 + kGatherBatch - 1) / kGatherBatch;
    out.units[i] = GatherUnit{pieces[i].pos, (int)n, batches, pieces[i].heavy};
    n += (size_t)batches * kGatherBatch;
  }
  out.n_entries = n + kGatherBatch;
}

size_t fill_gather_entries(const GatherPlan &g, int m, const int *ap, const int *ai, const float *ax, size_t u0, size_t u1,
                           uint32_t *cols, float *vals) {
  size_t w = 0;
  int row = -1;  // plain units come in row order: the row ends inside them are found by walking ap
  for (size_t i = u0; i < u1; ++i) {
    const GatherPlan::Range &u = g.ranges[i];
    const int len = u.j1 - u.j0;
    std::memcpy(cols + w, ai + u.j0, sizeof(int) * (size_t)len);
    std::memcpy(vals + w, ax + u.j0, sizeof(float) * (size_t)len);
    if (u.heavy < 0) {
      if (row < 0) row = (int)(std::upper_bound(ap, ap + m + 1, u.j0) - ap) - 1;  // the first row that ends behind j0
      while (ap[row + 1] <= u.j0) ++row;
      for (; row < m && ap[row + 1] <= u.j1; ++row)
        if (ap[row + 1] > ap[row]) cols[w + (ap[row + 1] - 1 - u.j0)] |= kGatherEnd;
    } else {
      cols[w + len - 1] |= kGatherEnd;
    }
    w += len;
    for (; w % kGatherBatch != 0; ++w) { cols[w] = (uint32_t)ai[u.j1 - 1]; vals[w] = 0.f; }
  }
  if (u1 == g.ranges.size())
    for (int k = 0; k < kGatherBatch; ++k, ++w) { cols[w] = 0; vals[w] = 0.f; }
  return w;
}

}  // namespace tf
