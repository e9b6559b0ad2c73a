// Balanced gather: out = A * X for a CSR operator whose rows share too few columns for gather tiles (graphs).
// Host plan and launcher; the kernel is in gather.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>
#include <vector>

namespace tf {

// A unit is what one group of lanes works through: whole consecutive non-empty rows, or one piece of a row that is
// too long for a group.  {first row (its position in `rows`) or slot of the partial sum, first entry, batches, index
// into `heavy` or -1}.
struct GatherUnit {
  int pos, p0, batches, heavy;
};
struct GatherHeavy {
  int row, first_slot, n_slots, pad;
};
constexpr int kGatherBatch = 8;             // entries a group works on together
constexpr uint32_t kGatherEnd = 0x80000000u;  // on the column id: last entry of a row or of a piece

struct GatherPlan {
  std::vector<GatherUnit> units;      // pieces of long rows first: they take longest
  std::vector<GatherHeavy> heavy;
  std::vector<int> rows;              // non-empty rows in order; left empty when every row has a nonzero
  std::vector<int> empty_rows;
  struct Range { int pos, j0, j1, heavy; };
  std::vector<Range> ranges;          // the nonzeros of every unit
  size_t n_entries = 0;               // see fill_gather_entries
  int n_slots = 0;
};
// `groups`: lane groups resident on the device, which sets how finely the work is cut.  ticket_sums: rows are cut where the
// warps of the ticket executor's CTA cut them and nowhere else, so that the sums are added in its order.
void build_gather_plan(int m, const int *ap, int groups, bool ticket_sums, GatherPlan &out);
// The entries of the units [u0, u1), those of u0 first: column | kGatherEnd and value of every nonzero, unit after unit, each
// unit filled up to whole batches with entries of value 0 that name its last column again (they follow the unit's last row end,
// so their sums go nowhere).  Behind the last unit there is one batch more, of zeros, because a group reads one batch ahead.
// Returns their number.
size_t fill_gather_entries(const GatherPlan &g, int m, const int *ap, const int *ai, const float *ax, size_t u0, size_t u1,
                           uint32_t *cols, float *vals);

}  // namespace tf

namespace tfk {

constexpr int kGatherResident = 768;  // threads of the gather kernel resident per SM

struct GatherParams {
  const int *cols;      // column | end bit
  const float *vals;
  const int4 *units;
  const int *rows;      // null: row = position
  const int4 *heavy;
  int *heavy_cnt;       // per (long row, panel): pieces that have delivered; zero between launches
  float *partial;       // n_slots x partial_ld
  const float *dense;
  float *out;
  int ld_in, ld_out, partial_ld;
  int n_cols;           // columns computed
  int n_units;
  int panel_w, panels, unit_blocks;  // (filled in by the launcher) columns per pass over the units, ...
  int relu;
};

// Lanes per group for a dense width: each lane owns four columns.
int gather_group(int n_cols);
// vec_in / vec_out: rows of X / of the result start on 16-byte boundaries.
cudaError_t launch_gather(bool vec_in, bool vec_out, const GatherParams &p, cudaStream_t s);
// D = (A .* (Q K^T)) V over the same units (sddmm_gather.cu): V is p.dense, D p.out, both of n_cols columns; m rows of Q.
bool sddmm_gather_supported(int kq, int nv);  // both up to 128
int sddmm_group(int kq, int nv);              // lanes that work on a unit
int sddmm_resident(int kq, int nv);           // threads of the kernel resident per SM
cudaError_t launch_sddmm_gather(const GatherParams &p, const float *Q, const float *K, int kq, int m, cudaStream_t s);
// dst[r][0:ld] = src[r][0:n_cols], the rest zero: rows of a width that is no multiple of four made readable as float4.
// (dst on a 16-byte boundary, ld the next multiple of four)
cudaError_t launch_pad_rows(const float *src, long long rows, int n_cols, int ld, float *dst, cudaStream_t s);

}  // namespace tfk
