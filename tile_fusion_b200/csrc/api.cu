// C ABI of libtilefusion_b200: plans (device-resident operators + item lists) and executors.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <climits>
#include <cstring>
#include <condition_variable>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <string>
#include <vector>

#include "band_march.h"
#include "gather.h"
#include "gemm_tc_host.h"
#include "host_stage.h"
#include "kernels.cuh"
#include "lattice_march.h"
#include "launch.h"
#include "line_march.h"
#include "row_gemm.h"
#include "spmm_gemm.h"
#include "tf_internal.h"

namespace {

using tf::fail;

#define TF_CUDA(call)                                                                         \
  do {                                                                                        \
    cudaError_t e__ = (call);                                                                 \
    if (e__ != cudaSuccess)                                                                   \
      return fail(TF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e__));          \
  } while (0)

#define TF_TRY(call)              \
  do {                            \
    const int rc__ = (call);      \
    if (rc__ != TF_OK) return rc__; \
  } while (0)

template <class T>
struct DevBuf {
  T *p = nullptr;
  size_t n = 0;
  ~DevBuf() { if (p) cudaFree(p); }
  int alloc(size_t count) {
    if (p) { cudaFree(p); p = nullptr; }
    n = count;
    if (count == 0) return TF_OK;
    cudaError_t e = cudaMalloc(&p, count * sizeof(T));
    if (e != cudaSuccess) { p = nullptr; return fail(TF_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e)); }
    return TF_OK;
  }
  int upload(const T *h, size_t count) {
    int rc = alloc(count);
    if (rc != TF_OK || count == 0) return rc;
    TF_CUDA(cudaMemcpy(p, h, count * sizeof(T), cudaMemcpyHostToDevice));
    return TF_OK;
  }
  int upload(const std::vector<T> &v) { return upload(v.data(), v.size()); }
};

struct DevCsr {
  int m = 0, n = 0;
  DevBuf<int> ap, ai;
  DevBuf<float> ax;
  int upload(const tf_csr &h) {
    m = h.m; n = h.n;
    int rc = ap.upload(h.ap, (size_t)h.m + 1);
    if (rc == TF_OK) rc = ai.upload(h.ai, (size_t)h.ap[h.m]);
    if (rc == TF_OK) rc = ax.upload(h.ax, (size_t)h.ap[h.m]);
    return rc;
  }
};

// Operator of the balanced gather (gather.cu).
struct DevGather {
  bool on = false;
  int n_units = 0, n_empty = 0, partial_ld = 0, n_slots = 0;
  DevBuf<int> cols;
  DevBuf<float> vals;
  DevBuf<int4> units, heavy;
  DevBuf<int> rows, empty, cnt;
  DevBuf<float> partial;
  // For the host-pointer calls, where no row is cut and units are in row order: units [0, u] read rows < in_rows[u] of the
  // operand, and with them every row < out_rows[u] of the result is final.
  std::vector<long long> in_rows, out_rows;
  void follow_units(const tf::GatherPlan &g, int m, const int *ai) {
    const int n = (int)g.units.size();
    if (!g.heavy.empty()) return;
    in_rows.resize(n);
    out_rows.resize(n);
    long long need = 0;
    for (int u = 0; u < n; ++u) {
      for (int j = g.ranges[u].j0; j < g.ranges[u].j1; ++j) need = std::max<long long>(need, ai[j] + 1LL);
      const int pos = u + 1 < n ? g.units[u + 1].pos : 0;
      in_rows[u] = need;
      out_rows[u] = u + 1 == n ? m : (g.rows.empty() ? pos : g.rows[pos]);
    }
  }
  // The entries are made in pieces of 4 MB by up to four threads, each of which copies its pieces to the device.  (Arrays of all
  // of them cost more in first touches than the copies take: an SDDMM plan of 8.4 M nonzeros 25.4 ms, like this 19.8.)
  int upload_entries(const tf::GatherPlan &g, const tf_csr &A) {
    int rc = cols.alloc(g.n_entries), dev = 0;
    if (rc == TF_OK) rc = vals.alloc(g.n_entries);
    if (rc != TF_OK) return rc;
    TF_CUDA(cudaGetDevice(&dev));
    constexpr size_t kPiece = (size_t)1 << 19;  // entries
    const size_t n = g.units.size();
    if (n == 0) {  // the batch behind the last unit
      TF_CUDA(cudaMemset(cols.p, 0, cols.n * sizeof(int)));
      TF_CUDA(cudaMemset(vals.p, 0, vals.n * sizeof(float)));
      return TF_OK;
    }
    const size_t parts = g.n_entries < 2 * kPiece ? 1 : std::min<size_t>(4, std::max(1u, std::thread::hardware_concurrency() / 2));
    auto at = [&](size_t u) { return u < n ? (size_t)g.units[u].p0 : g.n_entries; };  // where unit u begins, or all end
    std::vector<cudaError_t> errors(parts, cudaSuccess);
    auto part = [&](size_t k) {
      cudaError_t &e = errors[k];
      try {
        std::unique_ptr<uint32_t[]> c;
        std::unique_ptr<float[]> v;
        size_t room = 0;
        e = cudaSetDevice(dev);
        size_t u = n * k / parts;
        const size_t end = n * (k + 1) / parts;
        while (u < end && e == cudaSuccess) {
          size_t to = u + 1;
          while (to < end && at(to + 1) - at(u) <= kPiece) ++to;
          const size_t count = at(to) - at(u);
          if (count > room) {
            room = std::max(count, std::min(kPiece, g.n_entries));
            c.reset(new uint32_t[room]);
            v.reset(new float[room]);
          }
          tf::fill_gather_entries(g, A.m, A.ap, A.ai, A.ax, u, to, c.get(), v.get());
          e = cudaMemcpy(cols.p + at(u), c.get(), count * sizeof(int), cudaMemcpyHostToDevice);
          if (e == cudaSuccess) e = cudaMemcpy(vals.p + at(u), v.get(), count * sizeof(float), cudaMemcpyHostToDevice);
          u = to;
        }
      } catch (const std::bad_alloc &) {
        e = cudaErrorMemoryAllocation;
      }
    };
    std::vector<std::thread> pool;
    size_t started = 1;
    try {
      pool.reserve(parts);
      for (; started < parts; ++started) pool.emplace_back(part, started);
    } catch (const std::exception &) {  // no thread to be had: the rest is done here
    }
    part(0);
    for (size_t k = started; k < parts; ++k) part(k);
    for (std::thread &th : pool) th.join();
    for (cudaError_t e : errors) TF_CUDA(e);
    return TF_OK;
  }
  // n_cols: width of the dense operand the units are cut for; max_cols: widest one the operator will meet; follow: see above
  int build(const tf_csr &A, int n_cols, int max_cols, int sm_count, bool follow = false, int resident = tfk::kGatherResident,
            bool ticket_sums = false) {
    tf::GatherPlan g;
    tf::build_gather_plan(A.m, A.ap, sm_count * (resident / tfk::gather_group(n_cols)), ticket_sums, g);
    n_units = (int)g.units.size();
    n_empty = (int)g.empty_rows.size();
    n_slots = g.n_slots;
    partial_ld = (std::max(n_cols, max_cols) + 3) / 4 * 4;
    const int panels = (partial_ld + 127) / 128;  // the most any width up to that is read in
    if (follow) follow_units(g, A.m, A.ai);
    if (!g.rows.empty()) g.rows.resize(g.rows.size() + 2, 0);  // a group looks one row ahead (with the row of Q, two)
    int rc = upload_entries(g, A);
    if (rc == TF_OK) rc = units.upload(reinterpret_cast<const int4 *>(g.units.data()), g.units.size());
    if (rc == TF_OK) rc = heavy.upload(reinterpret_cast<const int4 *>(g.heavy.data()), g.heavy.size());
    if (rc == TF_OK) rc = rows.upload(g.rows);
    if (rc == TF_OK) rc = empty.upload(g.empty_rows);
    if (rc == TF_OK) rc = cnt.alloc(g.heavy.size() * (size_t)panels);
    if (rc == TF_OK) rc = partial.alloc((size_t)g.n_slots * partial_ld);
    if (rc != TF_OK) return rc;
    if (cnt.n) TF_CUDA(cudaMemset(cnt.p, 0, cnt.n * sizeof(int)));
    on = true;
    return TF_OK;
  }
  // What a product keeps between its groups, for a caller's buffer in the place of the plan's own: the counters of the cut rows,
  // then their partial sums.
  size_t scratch_counters() const { return (cnt.n * sizeof(int) + 255) / 256 * 256; }
  size_t scratch_bytes() const { return heavy.n ? scratch_counters() + (size_t)n_slots * partial_ld * sizeof(float) : 0; }
};

}  // namespace

struct tf_plan {
  int chain = 0;  // 0 SpMM-SpMM, 1 GeMM-SpMM, 2 SDDMM-SpMM
  int mode = TF_MODE_STREAM;
  int m = 0, n_cols = 0, k_dim = 0, halo_rows = 0;
  int first_cols = 0;  // columns of the first operator (rows of C)
  DevCsr first, second;
  bool first_is_second = false;
  tf::HostPlan hp;
  DevBuf<int4> items;
  DevBuf<int> seg_t, seg_out;  // rows of T / D that are accumulated atomically from segments of a heavy row
  DevBuf<int> prod_done, cons_done;
  DevBuf<tfk::ExecState> state;
  DevBuf<float> inter, sendbuf;
  // gather tiles (stream / unfused mode)
  struct DevTiling {
    DevBuf<int> row_ptr, rows, halo_ptr, halo;
    DevBuf<unsigned short> slot;
    DevBuf<int2> meta;
    std::vector<int> meta_off;  // per tile: offset of its row table, in 16-byte units
    bool on = false;
    // ap, ax: host CSR of the operator the tiling belongs to; with_meta: build the pipeline's row tables
    int upload(const tf::Tiling &t, const int *ap, const float *ax, bool with_meta) {
      on = t.tiled;
      if (!on) return TF_OK;
      int rc = TF_OK;
      if (with_meta) {
        const int nt = t.tiles();
        meta_off.assign(nt + 1, 0);
        size_t pairs = 0;
        for (int k = 0; k < nt; ++k) {
          meta_off[k] = (int)(pairs / 2);
          pairs += (size_t)tfk::kTileMetaPlanes * ((t.tile_row_ptr[k + 1] - t.tile_row_ptr[k] + 7) / 8 * 8);
        }
        std::vector<int2> m(pairs, make_int2(0, 0));
        for (int k = 0; k < nt; ++k) {
          const int rp = t.tile_row_ptr[k], nR = t.tile_row_ptr[k + 1] - rp, R = (nR + 7) / 8 * 8;
          int2 *blk = m.data() + 2 * (size_t)meta_off[k];
          for (int i = 0; i < R; ++i) blk[tfk::kTileMetaNnz * R + i] = make_int2(-1, 0);
          for (int i = 0; i < nR; ++i) {
            const int r = t.rows[rp + i], cnt = ap[r + 1] - ap[r];
            blk[tfk::kTileMetaNnz * R + i] = make_int2(r, cnt);
            for (int q = 0; q < std::min(cnt, tfk::kTileMetaNnz); ++q) {
              int2 e;
              e.x = (int)t.slot[ap[r] + q] * 128;
              std::memcpy(&e.y, &ax[ap[r] + q], 4);
              blk[q * R + i] = e;
            }
          }
        }
        rc = meta.upload(m);
      }
      if (rc == TF_OK) rc = row_ptr.upload(t.tile_row_ptr);
      if (rc == TF_OK) rc = rows.upload(t.rows);
      if (rc == TF_OK) rc = halo_ptr.upload(t.tile_halo_ptr);
      if (rc == TF_OK) rc = halo.upload(t.halo);
      if (rc == TF_OK) rc = slot.upload(t.slot);
      return rc;
    }
    tfk::TileArrays view() const {
      tfk::TileArrays a{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
      if (on) a = tfk::TileArrays{row_ptr.p, rows.p, halo_ptr.p, halo.p, slot.p, meta.p};
      return a;
    }
  } ptile, ctile;
  // balanced gather: operators without row reuse (graphs); `second` serves both products when B == A
  DevGather g_first, g_second;
  int ld_t = 0;              // floats per row of the intermediate: n_cols rounded up to whole float4
  DevBuf<float> g_pad;       // rows of C of a width that is no multiple of four, padded to ld_t
  struct Piece { int f_begin, f_end, begin, end; long long in_rows, out_rows; };  // units of the first and second operator
  std::vector<Piece> pieces;  // see make_gather_pieces
  bool keep_t = false;       // the caller asked for the intermediate: every call leaves it in `inter`
  bool spmm_first = false;   // GeMM-SpMM on the balanced gather: D = (A B) C instead of A (B C)
  bool ticket_sums = false;  // every sum in the order of the ticket executor (tensor_cores > 0)
  bool one_sums = false;     // (with spmm_first) those of the one launch, in two
  tfk::RowGemmSums sums() const { return ticket_sums ? tfk::kSumsTicket : one_sums && spmm_first ? tfk::kSumsSpmmGemm : tfk::kSumsFree; }
  size_t dyn_smem = 0;
  int tile_slots = 0;
  bool pipe = false;  // every item of phases 1 and 2 is a gather tile: run them on the tile pipeline
  int pipe_grid = 0, pipe_rows = 0;
  // tensor-core dense producer
  bool use_tc = false;
  int sm_count = 0;
  DevBuf<float> w_hi, w_lo;  // split, transposed weight [n_cols][k] (ticket executor), [row_gemm_pad_n][row_gemm_pad_k] otherwise
  CUtensorMap tm_whi, tm_wlo;
  int tile_info[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // producer bx,by,bz,tiles ; consumer bx,by,bz,tiles
  // plane-marching executor (both operators are star stencils on one grid)
  struct March {
    bool on = false, same = false;  // same: one operator on both sides (B == A)
    bool ragged = false;            // a width off the multiples of four: C is padded to rows of ld_t in g_pad (see build_march)
    bool halves = false;            // planes from the half maps: nx is odd, or ragged
    bool identity_first = false;    // GeMM-SpMM: the first operator is the identity, the operand is the producer's T
    bool halo_lo = false, halo_hi = false;  // a neighbour rank below / above supplies plane -1 / nz of T
    int nx = 0, ny = 0, nz = 0, ncls_f = 0, ncls_a = 0, z_shift = 0, grid = 0, n_items = 0, n_phase1 = 0;
    long long planes_c = 0;
    DevBuf<unsigned> pcls_f, pcls_a;
    std::vector<float> dict_f, dict_a;   // host copies: the dictionaries travel as kernel parameters
    DevBuf<int4> items;
    DevBuf<int4> star_items;         // GeMM-SpMM in two launches: the items of the one-product kernel
    int n_star = 0;
    int first_idle_sm = INT_MAX;
    int n_boundary = 0;              // rows of the neighbours' halo that this rank produces (phase 0)
    DevBuf<int> b_ap, b_ai;
    DevBuf<float> b_ax;
    DevBuf<tfk::MarchState> st;   // [0]: tickets of phase 1 (or of the whole grid), [1]: of phase 2 -- the two may run side by side
    std::vector<tf::MarchItem> host_items;
    // host-pointer path (single GPU): the grid again, cut into slabs of planes that run one launch each while the
    // planes of C for the next slab arrive and the planes of D of the one before leave
    struct Slab { int item_begin, item_end, z_begin, z_end; };
    std::vector<Slab> slabs;
  } march;
  // line-marching executor (both operators are five-point operators on one 2-D grid)
  struct Lines {
    bool on = false, same = false;
    bool any_align = false;  // rows off the 16-byte grid are taken (value by value) instead of refused
    int nx = 0, ny = 0, tiles = 0;
    DevBuf<unsigned> words_f, words_a;
    tfk::LineParams par;
  } lines;
  // band-marching executor (both operators are banded)
  struct Band {
    int block = 0;  // rows per block; 0: not taken
    DevBuf<int> quads_f, quads_a;
    tfk::BandParams par;
  } band;
  // GeMM-SpMM in one launch
  struct OneLaunch {
    bool on = false;
    tfk::SpmmGemmParams par = {};
    DevBuf<float> coef;
    std::vector<Piece> pieces;  // of a host-pointer call: bricks [begin, end)
  } one;
  // schedule mode
  DevBuf<int> s_ptr2, s_id, s_type, s_ker;
  int s_n1 = 0;
  std::vector<int> s_ptr1;
  bool s_has_ker = false;
  // host-pointer path: staging buffers, streams and the segments of the copy/compute pipeline
  struct Seg { int item_begin, item_end; long long in_rows, out_rows; };
  std::vector<Seg> segs;
  cudaStream_t s_h2d = nullptr, s_run = nullptr, s_d2h = nullptr;
  std::vector<cudaEvent_t> ev_in, ev_run;
  std::unique_ptr<tf::HostPipe> host_pipe;   // copies of the host-pointer calls; pinned slots for pageable arrays (host_stage.h)
  ~tf_plan() {
    for (cudaEvent_t e : ev_in) cudaEventDestroy(e);
    for (cudaEvent_t e : ev_run) cudaEventDestroy(e);
    if (s_h2d) cudaStreamDestroy(s_h2d);
    if (s_run) cudaStreamDestroy(s_run);
    if (s_d2h) cudaStreamDestroy(s_d2h);
  }
  DevBuf<float> h_in0, h_in1, h_in2, h_out;
  int grid = 0, vec = 1, ch = 1;
  int epoch = 1;  // flags start at 0, so no pass may use 0
  int spin_limit = 1 << 22;
  long long launches = 0;
  int device = 0;
};

namespace {

int device_ready(int *sm_count) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(TF_ERR_CUDA, std::string("no usable CUDA device: ") + cudaGetErrorString(e));
  cudaDeviceProp prop;
  TF_CUDA(cudaGetDeviceProperties(&prop, dev));
  if (prop.major < 10) return fail(TF_ERR_CUDA, "this library is built for sm_100a (B200) only");
  *sm_count = prop.multiProcessorCount;
  return TF_OK;
}

int default_rows_per_block(int n_cols, bool gemm) {
  if (gemm) return 64;
  return n_cols >= 128 ? 64 : 128;
}

// pt, ct: the gather tiles of a plan the tile pipeline runs; its tile items carry the extents of the
// tile ({kind, flag, tile, rows rounded up to 8} {need, staged rows, offset of the staged rows, offset
// of the row table}), so that the kernel needs no further lookup before it can start on a tile.
int upload_items(tf_plan &p, const tf::Tiling *pt = nullptr, const tf::Tiling *ct = nullptr) {
  std::vector<int4> raw(2 * p.hp.items.size());
  for (size_t i = 0; i < p.hp.items.size(); ++i) {
    const tf::Item &it = p.hp.items[i];
    raw[2 * i] = make_int4(it.kind, it.block, it.row_begin, it.row_end);
    raw[2 * i + 1] = make_int4(it.need, it.base, it.aux0, it.aux1);
    if (p.pipe && (it.kind == tf::ITEM_PRODUCE_TILED || it.kind == tf::ITEM_CONSUME_TILED)) {
      const tf::Tiling &t = it.kind == tf::ITEM_PRODUCE_TILED ? *pt : *ct;
      const int k = it.row_begin;
      const tf_plan::DevTiling &dt = it.kind == tf::ITEM_PRODUCE_TILED ? p.ptile : p.ctile;
      raw[2 * i].w = (t.tile_row_ptr[k + 1] - t.tile_row_ptr[k] + 7) / 8 * 8;
      raw[2 * i + 1] = make_int4(it.need, t.tile_halo_ptr[k + 1] - t.tile_halo_ptr[k], t.tile_halo_ptr[k], dt.meta_off[k]);
    }
  }
  int rc = p.items.upload(raw);
  if (rc == TF_OK && !p.hp.seg_t_rows.empty()) rc = p.seg_t.upload(p.hp.seg_t_rows);
  if (rc == TF_OK && !p.hp.seg_out_rows.empty()) rc = p.seg_out.upload(p.hp.seg_out_rows);
  return rc;
}

// Rows that segments of a heavy row add into start a pass at zero; a final ReLU is applied to them after it.
int segments_begin(tf_plan &p, const tfk::Params &P, cudaStream_t s) {
  TF_CUDA(tfk::launch_rows_fix(p.seg_t.p, (int)p.hp.seg_t_rows.size(), p.n_cols, p.inter.p, false, s));
  TF_CUDA(tfk::launch_rows_fix(p.seg_out.p, (int)p.hp.seg_out_rows.size(), p.n_cols, P.out, false, s));
  return TF_OK;
}
int segments_end(tf_plan &p, const tfk::Params &P, cudaStream_t s) {
  if (P.relu) TF_CUDA(tfk::launch_rows_fix(p.seg_out.p, (int)p.hp.seg_out_rows.size(), p.n_cols, P.out, true, s));
  return TF_OK;
}

int finish_plan(tf_plan &p, const tf_plan_opts &o, int sm_count, bool ring) {
  const bool a16 = true;  // buffers owned by the plan are 256-byte aligned; callers' pointers are checked per call
  tfk::choose_shape(p.n_cols, a16, &p.vec, &p.ch);
  if (p.dyn_smem > 0) { p.vec = 4; p.ch = 1; }
  int occ = tfk::stream_occupancy(p.chain, p.vec, p.ch, ring, p.dyn_smem);
  if (occ <= 0) return fail(TF_ERR_CUDA, "occupancy query failed for the executor kernel");
  // The resident-CTA query answers 1 for any kernel that allocates tensor memory.  Two CTAs of this
  // kernel fit an SM (256 of 512 tensor-memory columns each, half the shared memory, 64 registers), and
  // the executor does not depend on the answer for progress: only running CTAs hold tickets.
  if (p.use_tc && occ == 1 && p.dyn_smem <= 106 * 1024) occ = 2;
  if (o.ctas_per_sm > 0) occ = std::min(occ, o.ctas_per_sm);
  p.grid = sm_count * occ;
  return TF_OK;
}

int zero_state(tf_plan &p) {
  int rc = p.state.alloc(1);
  if (rc != TF_OK) return rc;
  TF_CUDA(cudaMemset(p.state.p, 0, sizeof(tfk::ExecState)));
  const size_t np = (size_t)p.hp.n_prod, nc = (size_t)p.hp.n_cons;
  rc = p.prod_done.alloc(std::max<size_t>(np, 1));
  if (rc == TF_OK) rc = p.cons_done.alloc(std::max<size_t>(nc, 1));
  if (rc != TF_OK) return rc;
  TF_CUDA(cudaMemset(p.prod_done.p, 0, p.prod_done.n * sizeof(int)));
  TF_CUDA(cudaMemset(p.cons_done.p, 0, p.cons_done.n * sizeof(int)));
  return TF_OK;
}

int check_opts(const tf_plan_opts *o, tf_plan_opts &out) {
  std::memset(&out, 0, sizeof(out));
  out.slack_blocks = -1;
  if (o) out = *o;
  if (out.mode < TF_MODE_STREAM || out.mode > TF_MODE_UNFUSED) return fail(TF_ERR_ARG, "plan: unknown mode");
  if (out.rows_per_block < 0 || out.halo_rows < 0 || out.n_boundary < 0) return fail(TF_ERR_ARG, "plan: negative option");
  if (out.tile_slots > tfk::kTileMaxSlots) return fail(TF_ERR_ARG, "plan: tile_slots above the shared-memory capacity");
  if (out.n_boundary > 0 && !out.boundary_rows) return fail(TF_ERR_ARG, "plan: boundary_rows is null");
  return TF_OK;
}

int load_schedule(tf_plan &p, const tf_schedule *s, bool need_ker) {
  if (!s) return fail(TF_ERR_ARG, "plan: TF_MODE_SCHEDULE needs a schedule");
  if (need_ker && !s->has_ker) return fail(TF_ERR_ARG, "plan: GeMM-SpMM needs a schedule with ker_begin (separated packing)");
  for (size_t k = 0; k < s->id.size(); ++k)
    if (s->id[k] < 0 || s->id[k] >= p.m || (s->type[k] != 0 && s->type[k] != 1))
      return fail(TF_ERR_ARG, "plan: schedule row id or type out of range");
  if (need_ker) {
    const int np = s->ptr1[s->n1];
    for (int w = 0; w < np; ++w) {
      const int kb = s->ptr2[w], ke1 = s->ker[2 * w];
      for (int k = kb; k < ke1; ++k)
        if (s->type[k] != 0 || s->id[k] != s->id[kb] + (k - kb))
          return fail(TF_ERR_ARG, "plan: GeMM-SpMM tiles must list consecutive first-loop rows");
      for (int k = ke1; k < s->ptr2[w + 1]; ++k)
        if (s->type[k] != 1) return fail(TF_ERR_ARG, "plan: ker_begin does not separate the two loops");
    }
  }
  p.s_n1 = s->n1;
  p.s_ptr1 = s->ptr1;
  p.s_has_ker = s->has_ker;
  int rc = p.s_ptr2.upload(s->ptr2);
  if (rc == TF_OK) rc = p.s_id.upload(s->id);
  if (rc == TF_OK) rc = p.s_type.upload(s->type);
  if (rc == TF_OK && s->has_ker) rc = p.s_ker.upload(s->ker);
  return rc;
}

void build_segments(tf_plan &p, int n_seg);

static_assert(tf::kMarchMaxClasses == tfk::kMarchMaxClassesDev, "host and device class limits differ");

std::vector<int4> march_items_raw(const std::vector<tf::MarchItem> &items) {
  std::vector<int4> raw(2 * items.size());
  for (size_t i = 0; i < items.size(); ++i) {
    raw[2 * i] = make_int4(items[i].x0, items[i].y0, items[i].zs, items[i].ze);
    raw[2 * i + 1] = make_int4(items[i].c0, items[i].flags, 0, 0);
  }
  return raw;
}

// The narrowest width off the multiples of four that marches plane by plane: 16 columns are computed whatever the width, so one to three stay with
// the gather, whose reads of four columns are a quarter of that (5 columns at 100 x 90 x 110: 187 us there, 71 here).
constexpr int kMarchMinRagged = 5;

// Whether a width off the multiples of four marches on such a grid.  A tile of 16 x 8 points is marched through whatever the grid
// has of it, and 16 columns whatever the width: from two chunks of columns on, what exists must be more than half of the points and two
// fifths of points and columns together; one chunk, whose rows cost the gather a line each for a few columns, is ahead from 45 % of the
// points on.  March and gather, us: 2 x 2 x 30 000, 33 columns (3 % of the points) 576 and 40; 10 x 10 x 1500 (39 %), 33 86 and 59, 5 40
// and 36; 20 x 12 x 500 (47 %), 47 64 and 54, 5 32 and 34; 12 x 6 x 2000 (56 %), 18 (32 % with the columns) 49 and 40, 99 (50 %) 102 and
// 110; 36 x 36 x 100 (68 %), 33 (46 %) 52 and 52; 24 x 24 x 300 (75 %), 18 (42 %) 47 and 46, 47 66 and 75.  Up to 16 384 rows the chain of
// steps counts for more (20 x 20 x 20 (52 %), 99 25 and 20; 12 x 12 x 50 (56 %), 47 22 and 20; 12 x 16 x 20 (75 %), 33 19 and 20), except
// on few planes, where launches are all that either takes (33 x 17 x 9 (49 %), 33 19 and 20; 18 x 11 x 4 (39 %) 19 and 20).
bool ragged_march_pays(int nx, int ny, int nz, int n_cols) {
  const long long chunks = (n_cols + tfk::kMarchCols - 1) / tfk::kMarchCols, rows = (long long)nx * ny * nz;
  const long long tiles = (long long)((nx + tfk::kMarchW - 1) / tfk::kMarchW) * ((ny + tfk::kMarchH - 1) / tfk::kMarchH);
  const double points = (double)nx * ny / ((double)tiles * tfk::kMarchW * tfk::kMarchH);
  const double columns = (double)n_cols / ((double)chunks * tfk::kMarchCols);
  if (nz <= 16 && rows * chunks <= 16384) return points > 1. / 3;
  return chunks == 1 ? points >= 0.45 : points > (rows <= 16384 ? 0.6 : 0.5) && points * columns >= 0.4;
}

// Plane-marching executor: taken when both operators of an SpMM-SpMM chain are star stencils on the same
// grid (lattice.cpp).  The general plan is built as well and serves calls whose operands are not 16-byte
// aligned.
// Fp == null: the first operator is the identity (GeMM-SpMM: the dense producer has written T, and the marching
// kernel computes D = A * (I * T); the products with the identity's zeros and its one are exact, so D is what the
// CSR consumer gives).
// star: behind the dense product on the one-product march.  Taken only where every row names all of its neighbours: the march
// multiplies a neighbour that is not named by zero, and an infinity there would not stay where it belongs.
int build_march(tf_plan &p, const tf_csr *Fp, const tf_csr &A, int halo_rows, int sm_count, const std::vector<int> &boundary_rows,
                bool star = false) {
  tf::LatticeOp lf, la;
  int rc = TF_OK;
  if (Fp) {
    rc = tf::analyse_lattice_operator(Fp->m, Fp->n, Fp->ap, Fp->ai, Fp->ax, 0, lf, halo_rows == 0);
    if (rc != TF_OK || !lf.ok) return rc;
  }
  if (Fp == &A && halo_rows == 0) la = lf;
  else {
    rc = tf::analyse_lattice_operator(A.m, A.n, A.ap, A.ai, A.ax, halo_rows, la, true);
    if (rc != TF_OK || !la.ok || (star && !la.full)) return rc;
  }
  if (!Fp) {
    lf.ok = true; lf.nx = la.nx; lf.ny = la.ny; lf.nz = la.nz; lf.n_classes = 1;
    lf.dict.assign(16, 0.f);
    lf.dict[3] = 1.f;                    // class 0: centre coefficient 1; class 1: all zero
    lf.patch_cls = la.patch_cls;         // same rows exist: zero class where A has none
    for (uint32_t &w : lf.patch_cls) {
      uint32_t v = 0;
      for (int b = 0; b < 4; ++b) v |= (uint32_t)(((w >> (8 * b)) & 255u) == (uint32_t)la.n_classes ? 1u : 0u) << (8 * b);
      w = v;
    }
  }
  const tf_csr &F = Fp ? *Fp : A;
  if (la.nx != lf.nx || la.ny != lf.ny || la.nz != lf.nz) return TF_OK;
  // Widths off the multiples of four march from a padded copy of C: the copy is a pass more, but the gather took two with seven row
  // reads each (and the same copy).  Infinities stay where the gather leaves them: full stencils and half maps only.
  // Gather and march, us: 100 x 90 x 110, 9 columns 202 and 77, 33 406 and 212, 47 454 and 235, 99 798 and 460; 31 x 40 x 50, 33 columns
  // 40 and 28; 12 x 16 x 20 19.5 and 17.4.  (48 columns of the first take 142: the copy is 60 of the difference.  Marching to a padded D
  // that another launch crops: 318 at 47 columns.)
  const bool ragged = p.n_cols % 4 != 0;
  if (ragged && (p.n_cols < kMarchMinRagged || halo_rows > 0 || !lf.full || !la.full || !ragged_march_pays(lf.nx, lf.ny, lf.nz, p.n_cols))) return TF_OK;
  if (halo_rows == 0 && (la.ghost_lo || la.ghost_hi)) return TF_OK;
  // with a neighbour rank below (above), the first operator must reach one plane of C below (above) the rank's
  // own: the boundary planes of T that the rank computes itself need them
  if (lf.ghost_lo > 1 || lf.ghost_hi > 1) return TF_OK;
  const int occ = tfk::march_ctas_per_sm();
  if (occ <= 0) return TF_OK;  // the kernel does not fit this device: general path
  tf_plan::March &M = p.march;
  M.nx = lf.nx; M.ny = lf.ny; M.nz = lf.nz;
  M.ragged = ragged;
  M.halves = ragged || M.nx % 2 != 0;
  M.ncls_f = lf.n_classes; M.ncls_a = la.n_classes;
  M.z_shift = lf.ghost_lo;
  M.planes_c = (long long)lf.nz + lf.ghost_lo + lf.ghost_hi;
  M.halo_lo = halo_rows > 0 && la.ghost_lo; M.halo_hi = halo_rows > 0 && la.ghost_hi;
  // With a halo exchange in flight a few SMs are left to the NCCL send / receive kernels: the persistent CTAs of
  // phase 1 would otherwise hold every SM until they finish, and the exchange would only start then.
  // With neighbour ranks the last SMs stay free while phase 1 runs: the kernels of the halo exchange and phase 2
  // start there, beside the persistent CTAs.
  M.grid = sm_count * occ;
  M.first_idle_sm = halo_rows > 0 ? std::max(1, sm_count - 6) : INT_MAX;
  const int working = std::min(sm_count, M.first_idle_sm) * occ;
  // phase 1: the planes of D that need no plane of T from a neighbour rank; phase 2: the first and / or last plane
  const int z1 = M.halo_lo ? 1 : 0, z2 = M.nz - (M.halo_hi ? 1 : 0);
  tf::build_march_items(M.nx, M.ny, z1, z2, p.n_cols, tfk::kMarchW, tfk::kMarchH, tfk::kMarchCols, working, 1, M.host_items);
  M.n_phase1 = (int)M.host_items.size();
  if (M.halo_lo) tf::build_march_items(M.nx, M.ny, 0, 1, p.n_cols, tfk::kMarchW, tfk::kMarchH, tfk::kMarchCols, M.grid, 1, M.host_items);
  if (M.halo_hi && M.nz > 1)
    tf::build_march_items(M.nx, M.ny, M.nz - 1, M.nz, p.n_cols, tfk::kMarchW, tfk::kMarchH, tfk::kMarchCols, M.grid, 1, M.host_items);
  M.n_items = (int)M.host_items.size();
  if (halo_rows == 0 && M.nz >= 8 && !ragged) {  // (host calls of ragged widths go through the gather's pieces)
    const int n_slabs = std::min(32, M.nz / 4);
    for (int sl = 0; sl < n_slabs; ++sl) {
      const int za = (int)((long long)M.nz * sl / n_slabs), zb = (int)((long long)M.nz * (sl + 1) / n_slabs);
      const int b = (int)M.host_items.size();
      tf::build_march_items(M.nx, M.ny, za, zb, p.n_cols, tfk::kMarchW, tfk::kMarchH, tfk::kMarchCols, M.grid, 1, M.host_items);
      M.slabs.push_back(tf_plan::March::Slab{b, (int)M.host_items.size(), za, zb});
    }
  }
  rc = M.items.upload(march_items_raw(M.host_items));
  if (rc == TF_OK) rc = M.pcls_f.upload(lf.patch_cls);
  M.dict_f = lf.dict;
  M.same = Fp == &A && halo_rows == 0;
  M.identity_first = Fp == nullptr;
  if (rc == TF_OK && !M.same) rc = M.pcls_a.upload(la.patch_cls);
  M.dict_a = M.same ? lf.dict : la.dict;
  if (rc == TF_OK) rc = M.st.alloc(2);
  if (rc == TF_OK && Fp && !boundary_rows.empty()) {
    // phase 0 of such a plan: the boundary rows of the first operator as a CSR of their own, in send-buffer order
    std::vector<int> bp(1, 0), bi;
    std::vector<float> bx;
    for (int r : boundary_rows) {
      bi.insert(bi.end(), F.ai + F.ap[r], F.ai + F.ap[r + 1]);
      bx.insert(bx.end(), F.ax + F.ap[r], F.ax + F.ap[r + 1]);
      bp.push_back((int)bi.size());
    }
    M.n_boundary = (int)boundary_rows.size();
    rc = M.b_ap.upload(bp);
    if (rc == TF_OK) rc = M.b_ai.upload(bi);
    if (rc == TF_OK) rc = M.b_ax.upload(bx);
  }
  if (rc != TF_OK) return rc;
  TF_CUDA(cudaMemset(M.st.p, 0, 2 * sizeof(tfk::MarchState)));
  M.on = true;
  return TF_OK;
}

bool aligned(const void *q, size_t a);

// One launch over the march items [item_begin, item_end).
int run_march(tf_plan &p, const float *C, float *D, int item_begin, int item_end, bool with_halo, cudaStream_t s) {
  tf_plan::March &M = p.march;
  if (item_end <= item_begin) { p.launches = 0; return TF_OK; }
  CUtensorMap tm, tm_odd;
  const int ld = M.ragged ? p.ld_t : p.n_cols;
  const float *src = M.ragged ? p.g_pad.p : C;
  int mr = M.halves ? tfk::march_make_half_map(&tm, src, ld, M.nx, M.ny, M.planes_c, 0)
                    : tfk::march_make_map(&tm, src, ld, M.nx, M.ny, M.ny, M.planes_c);
  tm_odd = tm;
  if (M.halves && mr == 0) mr = tfk::march_make_half_map(&tm_odd, src, ld, M.nx, M.ny, M.planes_c, 1);
  if (mr != 0) return fail(TF_ERR_CUDA, "cuTensorMapEncodeTiled failed for the dense operand (code " + std::to_string(mr) + ")");
  tfk::MarchParams Q;
  std::memset(&Q, 0, sizeof(Q));
  Q.pcls_f = M.pcls_f.p; Q.pcls_a = M.same ? M.pcls_f.p : M.pcls_a.p;
  std::memcpy(Q.dict_f, M.dict_f.data(), std::min(sizeof(Q.dict_f), M.dict_f.size() * sizeof(float)));
  std::memcpy(Q.dict_a, M.dict_a.data(), std::min(sizeof(Q.dict_a), M.dict_a.size() * sizeof(float)));
  Q.ncls_f = M.ncls_f; Q.ncls_a = M.ncls_a;
  Q.out = D;
  Q.items = M.items.p;
  Q.item_begin = item_begin; Q.item_end = item_end;
  Q.st = M.st.p + (with_halo ? 1 : 0);
  Q.nx = M.nx; Q.ny = M.ny; Q.nz = M.nz;
  Q.pnx = (M.nx + 1) / 2; Q.pny = (M.ny + 1) / 2;
  Q.n_cols = p.n_cols;
  Q.z_shift = M.z_shift;
  if (with_halo) {  // the received planes sit after the local rows of the intermediate: the lower neighbour's first
    const size_t plane = (size_t)M.nx * M.ny * p.n_cols;
    const float *halo = p.inter.p + (size_t)(p.hp.inter_rows - p.halo_rows) * p.n_cols;
    if (M.halo_lo) Q.t_lo = halo;
    if (M.halo_hi) Q.t_hi = halo + (M.halo_lo ? plane : 0);
  }
  Q.wait_limit = p.spin_limit;
  // phase 1 of a plan with neighbour ranks keeps the last SMs free; every other launch uses what it finds
  const bool keep_free = !with_halo && p.halo_rows > 0;
  Q.first_idle_sm = keep_free ? M.first_idle_sm : INT_MAX;
  if (M.ragged) TF_CUDA(tfk::launch_pad_rows(C, p.first_cols, p.n_cols, ld, p.g_pad.p, s));
  TF_CUDA(tfk::launch_lattice_march(keep_free ? M.grid : std::min(M.grid, std::max(1, item_end - item_begin)), tm, tm_odd, Q, M.halves, M.ragged, s));
  p.launches = M.ragged ? 2 : 1;
  return TF_OK;
}

// D = A * T with the one-product march, T in the plan's intermediate (with a row to spare behind it).
int run_star(tf_plan &p, float *D, bool relu, cudaStream_t s) {
  tf_plan::March &M = p.march;
  CUtensorMap tm;
  const int mr = tfk::march_make_map(&tm, p.inter.p, p.n_cols, M.nx, M.ny, M.ny, M.nz, tfk::kMarchH + 2);
  if (mr != 0) return fail(TF_ERR_CUDA, "cuTensorMapEncodeTiled failed for the intermediate (code " + std::to_string(mr) + ")");
  tfk::MarchParams Q;
  std::memset(&Q, 0, sizeof(Q));
  Q.pcls_a = M.pcls_a.p;
  std::memcpy(Q.dict_a, M.dict_a.data(), std::min(sizeof(Q.dict_a), M.dict_a.size() * sizeof(float)));
  Q.ncls_a = M.ncls_a;
  Q.out = D;
  Q.items = M.star_items.p;
  Q.item_end = M.n_star;
  Q.st = M.st.p;
  Q.nx = M.nx; Q.ny = M.ny; Q.nz = M.nz;
  Q.pnx = (M.nx + 1) / 2; Q.pny = (M.ny + 1) / 2;
  Q.n_cols = p.n_cols;
  Q.wait_limit = p.spin_limit;
  TF_CUDA(tfk::launch_star_march(std::min(M.n_star, p.sm_count * tfk::star_ctas_per_sm()), tm, Q, relu, s));
  p.launches = 1;
  return TF_OK;
}

// Pieces of a host-pointer call on operators that name rows near their own (grids, bands): the rows of the input that a piece
// needs arrive while the one before is computed, and finished rows leave while the next one is.  None where a row is cut or
// where the first piece already needs more than half of the input (graphs).
void make_gather_pieces(tf_plan &p, int n) {
  const DevGather &g = p.g_second, &f = p.first_is_second ? p.g_second : p.g_first;
  const bool two = p.chain == 0;  // the rows of T are made by units of the first operator
  const int units = (int)g.in_rows.size();
  if (units < 2 * n || (two && f.in_rows.empty())) return;
  tf_plan::Piece q{0, 0, 0, 0, 0, 0};
  for (int s = 0; s < n; ++s) {
    q.begin = q.end;
    q.f_begin = q.f_end;
    q.end = (int)((long long)units * (s + 1) / n);
    q.in_rows = g.in_rows[q.end - 1];
    q.out_rows = g.out_rows[q.end - 1];
    if (two) {
      while (q.f_end < (int)f.out_rows.size() && (q.f_end == 0 || f.out_rows[q.f_end - 1] < q.in_rows)) ++q.f_end;
      q.in_rows = f.in_rows[q.f_end - 1];
    }
    p.pieces.push_back(q);
  }
  if (2 * p.pieces[0].in_rows > (two ? p.first_cols : p.m)) p.pieces.clear();
}

// The rest of a SpMM-SpMM plan that runs on the balanced gather.
int make_gather_plan(std::unique_ptr<tf_plan> &p, const tf_csr &F, const tf_csr &A, const tf_plan_opts &o, int sm_count,
                     tf_plan **out) {
  p->ld_t = (p->n_cols + 3) / 4 * 4;
  int rc = p->g_second.build(A, p->n_cols, p->n_cols, sm_count, true);
  if (rc == TF_OK && !p->first_is_second) rc = p->g_first.build(F, p->n_cols, p->n_cols, sm_count, true);
  if (rc == TF_OK) rc = p->inter.alloc((size_t)p->m * p->ld_t);
  if (rc == TF_OK && p->ld_t != p->n_cols) rc = p->g_pad.alloc((size_t)p->first_cols * p->ld_t);
  if (rc == TF_OK) rc = zero_state(*p);
  if (rc != TF_OK) return rc;
  make_gather_pieces(*p, 16);
  p->hp.inter_rows = p->m;
  p->hp.n_prod = (p->first_is_second ? p->g_second : p->g_first).n_units;
  p->hp.n_cons = p->g_second.n_units;
  if (o.lattice_march >= 0) {
    rc = build_march(*p, &F, A, 0, sm_count, {});
    if (rc != TF_OK) return rc;
  }
  p->sm_count = sm_count;
  *out = p.release();
  return TF_OK;
}

// Line-marching executor: taken when both operators of an SpMM-SpMM chain are five-point operators on one 2-D grid.
int build_lines(tf_plan &p, const tf_csr &F, const tf_csr &A, bool same, int sm_count) {
  tf::LineOp f, a;
  tf::analyse_line_operator(A.m, A.n, A.ap, A.ai, A.ax, a);
  if (!a.ok) return TF_OK;
  if (!same) {
    tf::analyse_line_operator(F.m, F.n, F.ap, F.ai, F.ax, f);
    if (!f.ok || f.nx != a.nx) return TF_OK;
  }
  const tf::LineOp &first = same ? a : f;
  tf_plan::Lines &L = p.lines;
  L.same = same;
  L.nx = a.nx; L.ny = a.ny; L.tiles = a.tiles;
  if (a.ny == 2) {  // two long lines: gather tiles decline them, and the executor behind those reads rows that lie anywhere
    tf::Tiling t;
    tf::build_tiling(A.m, A.ap, A.ai, tf::kPipeTileSlots, tf::kDefaultTileMaxBz, tf::kPipeTileRows, t);
    if (!t.tiled) tf::build_tiling(A.m, A.ap, A.ai, tf::kDefaultTileSlotsSmall, tf::kDefaultTileMaxBz, tfk::tiled_threads(0), t);
    L.any_align = !t.tiled;
  }
  int rc = L.words_a.upload(a.words);
  if (rc == TF_OK && !same) rc = L.words_f.upload(f.words);
  if (rc == TF_OK) rc = zero_state(p);
  if (rc != TF_OK) return rc;
  std::memset(&L.par, 0, sizeof(L.par));
  std::memcpy(L.par.dict_f, first.dict.data(), first.dict.size() * sizeof(float));
  std::memcpy(L.par.dict_a, a.dict.data(), a.dict.size() * sizeof(float));
  L.par.none_f = 0x01010101u * (unsigned)first.n_classes;
  L.par.none_a = 0x01010101u * (unsigned)a.n_classes;
  L.par.words_a = L.words_a.p;
  L.par.words_f = same ? L.words_a.p : L.words_f.p;
  L.par.nx = L.nx; L.par.ny = L.ny; L.par.tiles = L.tiles; L.par.n_cols = p.n_cols;
  p.sm_count = sm_count;
  L.on = true;
  return TF_OK;
}

// The lines [y_begin, y_end) of D.
int run_lines(tf_plan &p, const float *C, float *D, int y_begin, int y_end, cudaStream_t s) {
  const bool on16 = aligned(C, 16) && aligned(D, 16), vec = p.n_cols % 4 == 0 && (on16 || !p.lines.any_align);
  if (vec && !on16)
    return fail(TF_ERR_ARG, "this plan reads rows as 16-byte vectors and needs 16-byte aligned dense operands "
                            "(build the plan with tile_slots < 0 otherwise)");
  tfk::LineParams P = p.lines.par;
  P.in = C; P.out = D;
  P.y_begin = y_begin; P.y_end = y_end;
  TF_CUDA(tfk::launch_line_march(P, vec, p.lines.same, p.sm_count, s));
  p.launches = 1;
  return TF_OK;
}

// Band-marching executor: taken when both operators of an SpMM-SpMM chain are banded and no grid was recognised.
int build_band(tf_plan &p, const tf_csr &F, const tf_csr &A, bool same, int sm_count) {
  int reach_a = 0, pairs_a = 0, reach_f = 0, pairs_f = 0;
  if (!tf::band_shape(A.m, A.n, A.ap, A.ai, &reach_a, &pairs_a)) return TF_OK;
  reach_f = reach_a; pairs_f = pairs_a;
  if (!same && !tf::band_shape(F.m, F.n, F.ap, F.ai, &reach_f, &pairs_f)) return TF_OK;
  const int block = std::max(reach_a, reach_f) <= 64 ? 64 : 128;
  if (tfk::band_smem(block, pairs_f, pairs_a, same) > tfk::kBandSmemMax) return TF_OK;
  tf_plan::Band &K = p.band;
  tf::BandOp op;
  tf::build_band_operator(F.m, F.ap, F.ai, F.ax, block, pairs_f, op);
  int rc = K.quads_f.upload(op.quads);
  if (rc == TF_OK && !same) {
    tf::build_band_operator(A.m, A.ap, A.ai, A.ax, block, pairs_a, op);
    rc = K.quads_a.upload(op.quads);
  }
  if (rc == TF_OK) rc = zero_state(p);
  if (rc != TF_OK) return rc;
  std::memset(&K.par, 0, sizeof(K.par));
  K.par.quads_f = reinterpret_cast<const int4 *>(K.quads_f.p);
  K.par.quads_a = same ? K.par.quads_f : reinterpret_cast<const int4 *>(K.quads_a.p);
  K.par.pairs_f = pairs_f; K.par.pairs_a = pairs_a;
  K.par.same = same;
  K.par.m = A.m; K.par.n_cols = p.n_cols;
  K.block = block;
  p.sm_count = sm_count;
  return TF_OK;
}

// The blocks [block_begin, block_end) of rows of D.
int run_band(tf_plan &p, const float *C, float *D, int block_begin, int block_end, cudaStream_t s) {
  if (!(aligned(C, 16) && aligned(D, 16)))
    return fail(TF_ERR_ARG, "this plan reads rows as 16-byte vectors and needs 16-byte aligned dense operands "
                            "(build the plan with tile_slots < 0 otherwise)");
  CUtensorMap tm, tm_d;
  TF_TRY(tfk::band_make_map(&tm, C, p.m, p.n_cols, p.band.block));
  TF_TRY(tfk::band_make_map(&tm_d, D, p.m, p.n_cols, 32));
  tfk::BandParams P = p.band.par;
  P.out = D;
  P.error = &p.state.p->error;
  P.wait_limit = p.spin_limit;
  P.block_begin = block_begin; P.block_end = block_end;
  TF_CUDA(tfk::launch_band_march(tm, tm_d, p.band.block, P, p.sm_count, s));
  p.launches = 1;
  return TF_OK;
}
int band_blocks(const tf_plan &p) { return (p.m + p.band.block - 1) / p.band.block; }

// The CSR arrays of an operator that a plan holds as line words or band quads only, for the calls that need them after all.
int restore_csr(tf_plan &p, bool second) {
  DevCsr &out = second || p.first_is_second ? p.second : p.first;
  if (out.ap.n) return TF_OK;
  std::vector<int> ap(1, 0), ai;
  std::vector<float> ax;
  auto fetch = [](auto &host, const auto &dev) {
    host.resize(dev.n);
    return cudaMemcpy(host.data(), dev.p, dev.n * sizeof(*dev.p), cudaMemcpyDeviceToHost);
  };
  if (p.lines.on) {
    const tf_plan::Lines &L = p.lines;
    std::vector<unsigned> words;
    TF_CUDA(fetch(words, second || L.same ? L.words_a : L.words_f));
    const float *dict = reinterpret_cast<const float *>(second || L.same ? L.par.dict_a : L.par.dict_f);
    for (int y = 0; y < L.ny; ++y)
      for (int x = 0; x < L.nx; ++x) {
        const int t = x / tf::kLineOut, i = x - t * tf::kLineOut + 2, r = y * L.nx + x;
        const unsigned cls = words[((size_t)y * L.tiles + t) * 8 + i / 4] >> (8 * (i & 3)) & 255u;
        const int off[5] = {-L.nx, -1, 0, 1, L.nx};
        const bool in[5] = {y > 0, x > 0, true, x < L.nx - 1, y < L.ny - 1};
        for (int q = 0; q < 5; ++q)
          if (in[q]) { ai.push_back(r + off[q]); ax.push_back(dict[8 * (size_t)cls + q]); }
        ap.push_back((int)ai.size());
      }
  } else {
    const tf_plan::Band &K = p.band;
    const bool a = second || K.par.same;
    const int pairs = a && !K.par.same ? K.par.pairs_a : K.par.pairs_f;
    std::vector<int> quads;
    TF_CUDA(fetch(quads, a && !K.par.same ? K.quads_a : K.quads_f));
    for (int r = 0; r < p.m; ++r) {
      for (int k = 0; k < 2 * pairs; ++k) {
        const int *q = &quads[4 * (((size_t)(r / K.block) * pairs + k / 2) * K.block + r % K.block) + 2 * (k & 1)];
        if (q[0] & 1) continue;  // no nonzero
        ai.push_back(r + q[0] / 128);
        float v;
        std::memcpy(&v, &q[1], 4);
        ax.push_back(v);
      }
      ap.push_back((int)ai.size());
    }
  }
  tf_csr h;
  std::memset(&h, 0, sizeof(h));
  h.m = p.m; h.n = p.m;
  h.ap = ap.data(); h.ai = ai.data(); h.ax = ax.data();
  return out.upload(h);
}

// T of a march that leaves none behind, where the caller asked for it.
int leave_intermediate(tf_plan &p, const float *C, cudaStream_t s) {
  if (!p.keep_t) return TF_OK;
  const DevCsr &f = p.first_is_second ? p.second : p.first;
  return tf_spmm_dev(f.ap.p, f.ai.p, f.ax.p, p.m, C, p.n_cols, p.inter.p, s);
}

// GeMM-SpMM in one launch (spmm_gemm.cu): star stencils with every neighbour stored, shapes of the tensor-core tile.  It adds up
// rows of B, so B should not be much wider than the result: on flat grids it is ahead up to K = 8 N (700 000 points, 128 -> 16:
// 126 us and 131, 256 -> 16: 216 and 210), on 3-D grids up to 1.5 N (1 M points, 128 -> 128: 290 and 382, 100 -> 64: 271 and 253,
// 128 -> 64: 258 and 251, 64 -> 16: 124 and 106).  Small grids keep the executors they had, although a launch or two could be gained
// there too (4 913 points in 3-D, 64 -> 64: 9.0 us and 15.3): the march and the gather behind the dense product give the same bits, which
// (A B) W does not, and on such grids they are compared.
// Where coefficients differ from row to row and bricks are cut off by a thin grid, the gather behind the dense product is ahead earlier: it
// has no brick to fill, and reads the coefficients with the columns.  With e of the bricks' points in the grid (former and one launch, us):
// flat, 5 x 100 000 (e = 0.63), K = 2 N 64 -> 32 105 and 103, 3 N 126 and 133, 8 N 256 -> 32 235 and 262; 9 x 50 000 (0.75), 8 N 210 and 198.
// 3-D, 5 x 2 x 30 000, 256 -> 256 (e = 0.31) 308 and 480; 5 x 6 x 10 000 (0.47) 314 and 343; 17 x 5 x 4000 (0.53), 256 -> 256 359 and 341,
// 320 -> 256 394 and 412; 5 x 6 x 10 000 (0.63), 160 -> 128 175 and 175, 192 -> 128 189 and 200; 9 x 9 x 4000 (0.68), 192 -> 128 208 and 202.
// What launches cost counts for less on larger grids (5 x 20 000, 4 N 128 -> 32 44 and 40).  At 16 columns the dense product in front
// computes as many for nothing: 5 x 6 x 10 000, 24 -> 16 56 and 47.
double one_launch_depth(const tf::StarOp &op, const tf::BrickGrid &g, long long rows, int n_cols) {  // largest K / N
  const bool flat = op.nz == 1;
  const double e = (double)rows / ((double)g.bricks() * tf::kStarRows);
  if (flat) return op.uniform || e > 0.7 ? 8. : std::min(8., 2. + (1 << 18) / (double)rows);
  return op.uniform || n_cols <= 16 ? 1.5 : std::min(1.5, 4. * e - 1.1 + (1 << 14) / (double)rows);
}

bool one_launch_pays(const tf_plan &p, const tf_csr &A, tf::StarOp &op, tf::BrickGrid &grid) {
  if (p.ticket_sums || !tfk::tc_supported(p.k_dim, p.n_cols) || A.m < (1 << 12)) return false;
  tf::analyse_star_operator(A.m, A.n, A.ap, A.ai, A.ax, op);
  return op.nx && (op.nz == 1 || A.m >= (1 << 15)) && tf::choose_bricks(op, tfk::spmm_gemm_points(p.k_dim, p.n_cols), grid) &&
         p.k_dim <= one_launch_depth(op, grid, A.m, p.n_cols) * p.n_cols;
}

int build_one_launch(tf_plan &p, const tf_csr &A) {
  tf::StarOp op;
  tf_plan::OneLaunch &O = p.one;
  if (!one_launch_pays(p, A, op, O.par.grid)) return TF_OK;
  if (p.mode == TF_MODE_UNFUSED) {  // what runs in one launch otherwise, in two: only the order of the sums
    p.one_sums = true;
    return TF_OK;
  }
  if (op.uniform) std::copy(op.coef.begin(), op.coef.end(), O.par.uniform);
  else TF_TRY(O.coef.upload(op.coef));
  O.par.coef = O.coef.p;
  // a host-pointer call goes layer by layer (on a flat grid row of bricks by row of bricks), up to 16 at a time
  const tf::BrickGrid &g = O.par.grid;
  const bool deep = g.nz > 1;
  const int layers = deep ? g.bz() : g.by(), per = g.bricks() / layers, n = std::min(16, layers);
  const long long points = (long long)g.nx * (deep ? g.ny : 1), thick = 1LL << (deep ? g.lz : g.ly);
  for (int i = 0; i < n; ++i) {
    const int a = (int)((long long)layers * i / n), b = (int)((long long)layers * (i + 1) / n);
    O.pieces.push_back(tf_plan::Piece{0, 0, a * per, b * per, std::min<long long>(p.m, (b * thick + 1) * points), std::min<long long>(p.m, b * thick * points)});
  }
  O.on = true;
  return TF_OK;
}

// GeMM-SpMM on the balanced gather.  The two products may be taken in either order, D = A (B C) = (A B) C: the sparse
// product reads one row of its operand per nonzero, so it is given the narrower one -- B where k < n_cols, else B C.
// (Rows of B that do not start on 16-byte boundaries would be gathered value by value; then B C comes first.  So it does
// on grids and bands: with a handful of nonzeros a row there is little to choose, and every consumer gives the same bits.)
int make_gemm_gather_plan(std::unique_ptr<tf_plan> &p, const tf_csr &A, const tf_plan_opts &o, bool tiled, int sm_count, tf_plan **out) {
  p->spmm_first = p->one_sums || (!tiled && !p->ticket_sums && p->k_dim % 4 == 0 && p->k_dim < p->n_cols);
  const int width = p->spmm_first ? p->k_dim : p->n_cols;
  p->ld_t = (width + 3) / 4 * 4;
  const size_t wn = (size_t)tfk::row_gemm_pad_n(p->n_cols) * tfk::row_gemm_pad_k(p->k_dim);
  int rc = p->g_second.build(A, width, std::max(p->k_dim, p->n_cols), sm_count, tiled && !p->one_sums, tfk::kGatherResident, p->ticket_sums);
  if (rc == TF_OK && !p->one.on) rc = p->inter.alloc((size_t)(p->m + 1) * p->ld_t);  // (the one-product march may read one row more)
  if (rc == TF_OK) rc = p->w_hi.alloc(wn);
  if (rc == TF_OK) rc = p->w_lo.alloc(wn);
  if (rc == TF_OK) rc = zero_state(*p);
  if (rc != TF_OK) return rc;
  make_gather_pieces(*p, 16);
  p->hp.inter_rows = p->one.on ? 0 : p->m;
  p->hp.n_cons = p->g_second.n_units;
  if (tiled && o.lattice_march >= 0 && p->n_cols % 4 == 0 && !p->one.on && !p->one_sums) {
    rc = build_march(*p, nullptr, A, 0, sm_count, {}, true);
    if (rc != TF_OK) return rc;
    tf_plan::March &M = p->march;
    if (M.on) {
      std::vector<tf::MarchItem> items;
      tf::build_march_items(M.nx, M.ny, 0, M.nz, p->n_cols, tfk::kMarchW, tfk::kMarchH, tfk::kMarchCols,
                            sm_count * tfk::star_ctas_per_sm(), 1, items);
      rc = M.star_items.upload(march_items_raw(items));
      if (rc != TF_OK) return rc;
      M.n_star = (int)items.size();
    }
  }
  p->sm_count = sm_count;
  *out = p.release();
  return TF_OK;
}

// Common plan construction for the two-operator chains.
int make_chain_plan(int chain, const tf_csr *A, const tf_csr *B, int k_dim, int n_cols, const tf_plan_opts *opts,
                    const tf_schedule *sched, tf_plan **out) {
  if (!A || !out) return fail(TF_ERR_ARG, "plan: null argument");
  if (n_cols <= 0) return fail(TF_ERR_ARG, "plan: dense width must be positive");
  tf_plan_opts o;
  int rc = check_opts(opts, o);
  if (rc != TF_OK) return rc;
  if (A->m <= 0) return fail(TF_ERR_ARG, "plan: matrix must have rows");
  if ((long long)A->m + o.halo_rows != A->n)
    return fail(TF_ERR_ARG, "plan: A must be m x (m + halo_rows): its columns index rows of the intermediate");
  rc = tf::check_csr(A->m, A->n, A->ap, A->ai, false);
  if (rc != TF_OK) return rc;
  if (!A->ax) return fail(TF_ERR_ARG, "plan: null value array");
  const tf_csr *F = chain == 0 ? (B ? B : A) : nullptr;
  if (F) {
    if (F->m != A->m) return fail(TF_ERR_ARG, "plan: B must have as many rows as A");
    if (F != A) {
      rc = tf::check_csr(F->m, F->n, F->ap, F->ai, false);
      if (rc != TF_OK) return rc;
      if (!F->ax) return fail(TF_ERR_ARG, "plan: null value array");
    }
    if (o.mode == TF_MODE_SCHEDULE && o.halo_rows) return fail(TF_ERR_UNSUPPORTED, "plan: schedule mode is single-GPU");
  }
  if (o.mode != TF_MODE_STREAM && (o.halo_rows || o.n_boundary))
    return fail(TF_ERR_UNSUPPORTED, "plan: halo exchange is available in stream mode only");
  int sm_count = 0;
  rc = device_ready(&sm_count);
  if (rc != TF_OK) return rc;

  std::unique_ptr<tf_plan> p(new tf_plan());
  cudaGetDevice(&p->device);
  p->chain = chain; p->mode = o.mode;
  p->m = A->m; p->n_cols = n_cols; p->k_dim = k_dim; p->halo_rows = o.halo_rows;
  p->ticket_sums = chain == 1 && o.tensor_cores > 0;
  if (F) {
    p->first_cols = F->n;
    p->first_is_second = F == A;
  }

  tf::PlanParams pp;
  pp.m = A->m; pp.n_cols = n_cols;
  pp.producer_is_gemm = chain == 1;
  pp.rows_per_block = o.rows_per_block > 0 ? o.rows_per_block : default_rows_per_block(n_cols, chain == 1);
  pp.max_block_nnz = pp.rows_per_block * 32;
  pp.halo_rows = o.halo_rows;
  pp.boundary_rows.assign(o.boundary_rows, o.boundary_rows + o.n_boundary);
  for (int i = 0; i < o.n_boundary; ++i)
    if (pp.boundary_rows[i] < 0 || pp.boundary_rows[i] >= A->m || (i && pp.boundary_rows[i] <= pp.boundary_rows[i - 1]))
      return fail(TF_ERR_ARG, "plan: boundary_rows must be sorted local row ids");
  pp.ring_bytes = o.mode == TF_MODE_STREAM ? (o.ring_bytes == 0 ? (48LL << 20) : (long long)o.ring_bytes) : -1;

  // grid size first (the default slack depends on how many CTAs are resident); ring-ness does not
  // change the resource use enough to matter for this estimate
  rc = finish_plan(*p, o, sm_count, false);
  if (rc != TF_OK) return rc;
  pp.max_ctas = p->grid;
  pp.slack_blocks = o.mode == TF_MODE_UNFUSED ? (1 << 30) : o.slack_blocks;
  if (chain == 0 && F && o.mode == TF_MODE_STREAM && o.lattice_march >= 0 && o.ring_bytes <= 0 && o.halo_rows == 0 && o.n_boundary == 0 &&
      o.rows_per_block == 0 && o.slack_blocks < 0 && o.ctas_per_sm == 0 && o.tile_slots == 0 && o.tile_max_bz == 0 &&
      o.tile_double_buffer == 0 && o.tile_pipeline == 0) {
    rc = build_lines(*p, *F, *A, F == A, sm_count);
    if (rc != TF_OK) return rc;
    if (p->lines.on) {
      *out = p.release();
      return TF_OK;
    }
  }
  // gather tiles: 16-byte staging copies need rows that are multiples of 4 floats
  tf::Tiling pt, ct;
  // a tile holds one row per 4 lanes... of the CTA that runs it: 256 rows (sparse chains) or 512 (GeMM-SpMM)
  const int tile_rows = tfk::tiled_threads(chain);
  const int slots = o.tile_slots == 0 ? (chain == 1 ? tf::kDefaultTileSlots : tf::kDefaultTileSlotsSmall) : o.tile_slots;
  // SpMM-SpMM with both operators tiled runs on the tile pipeline (one CTA per SM, about four tiles in
  // flight each).  Its tiles are a little smaller: two chunk buffers and two row tables share the SM's
  // shared memory.  It has no ring addressing, so a ring is only kept when the caller asked for one.
  bool want_pipe = false;
  {
    const int ps = o.tile_slots == 0 ? tf::kPipeTileSlots : o.tile_slots;
    const size_t need = tfk::tile_pipeline_smem(ps, tf::kPipeTileRows);
    if (chain == 0 && F && o.mode != TF_MODE_SCHEDULE && o.tile_pipeline >= 0 && o.ring_bytes <= 0 &&
        o.tile_double_buffer <= 0 && n_cols % 4 == 0 && need > 0 && need <= 226 * 1024) {
      const int max_bz = o.tile_max_bz > 0 ? o.tile_max_bz : tf::kDefaultTileMaxBz;
      tf::build_tiling(F->m, F->ap, F->ai, ps, max_bz, tf::kPipeTileRows, pt);
      if (pt.tiled && F != A) tf::build_tiling(A->m, A->ap, A->ai, ps, max_bz, tf::kPipeTileRows, ct);
      else if (pt.tiled) ct = pt;
      if (pt.tiled && ct.tiled) {
        want_pipe = true;
        p->tile_slots = ps;
        p->pipe_rows = tf::kPipeTileRows;
        p->dyn_smem = (size_t)ps * 132;  // for the launches of phase 0, which run on the two-CTA kernel
        rc = finish_plan(*p, o, sm_count, false);
        if (rc != TF_OK) return rc;
        pp.ring_bytes = -1;
        pp.max_ctas = 4 * sm_count;
      } else {
        pt = tf::Tiling();
        ct = tf::Tiling();
      }
    }
  }
  if (!want_pipe && o.mode != TF_MODE_SCHEDULE && slots > 0 && n_cols % 4 == 0) {
    const int max_bz = o.tile_max_bz > 0 ? o.tile_max_bz : tf::kDefaultTileMaxBz;
    const bool dbl = o.tile_double_buffer > 0 || (o.tile_double_buffer == 0 && tf::kDefaultTileDoubleBuffer);
    const int cap = dbl ? slots / 2 : slots;  // half-size tiles leave room for the next chunk's copies
    if (F) tf::build_tiling(F->m, F->ap, F->ai, cap, max_bz, tile_rows, pt);
    if (F == A) ct = pt;
    else tf::build_tiling(A->m, A->ap, A->ai, cap, max_bz, tile_rows, ct);
    if (pt.tiled || ct.tiled) {
      p->dyn_smem = (size_t)slots * 132;  // 128 B of staging + one source row id per slot
      p->tile_slots = slots;
      rc = finish_plan(*p, o, sm_count, false);  // the staging buffer lowers the resident CTA count
      if (rc != TF_OK) return rc;
      pp.max_ctas = p->grid;
    }
  }
  if (want_pipe && F && o.mode == TF_MODE_STREAM && o.lattice_march >= 0 && o.halo_rows == 0 && o.n_boundary == 0 && o.rows_per_block == 0 &&
      o.slack_blocks < 0 && o.ctas_per_sm == 0 && o.tile_slots == 0 && o.tile_max_bz == 0 && o.tile_pipeline == 0) {
    tf::LatticeOp grid;  // (star stencils on a 3-D grid march plane by plane; looked for only where there is a band at all)
    int reach = 0, pairs = 0;
    const bool band = tf::band_shape(A->m, A->n, A->ap, A->ai, &reach, &pairs);
    if (band) rc = tf::analyse_lattice_operator(A->m, A->n, A->ap, A->ai, A->ax, 0, grid, true);
    if (rc == TF_OK && band && !grid.ok) rc = build_band(*p, *F, *A, F == A, sm_count);
    if (rc != TF_OK) return rc;
    if (p->band.block) {
      p->tile_info[0] = pt.bx; p->tile_info[1] = pt.by; p->tile_info[2] = pt.bz; p->tile_info[3] = pt.tiles();
      p->tile_info[4] = ct.bx; p->tile_info[5] = ct.by; p->tile_info[6] = ct.bz; p->tile_info[7] = ct.tiles();
      *out = p.release();
      return TF_OK;
    }
  }
  // dense producer on the tensor cores: 128-row tiles, its K slices live in the same dynamic buffer
  const bool want_tc = chain == 1 && o.mode != TF_MODE_SCHEDULE && o.tensor_cores >= 0 && tfk::tc_supported(k_dim, n_cols);
  if (want_tc) {
    p->use_tc = true;
    p->dyn_smem = std::max(p->dyn_smem, (size_t)tfk::tc_smem_bytes_host(n_cols));
    if (o.rows_per_block == 0) pp.rows_per_block = tfk::kTcRowsHost;
    pp.max_block_nnz = pp.rows_per_block * 32;
    rc = p->w_hi.alloc((size_t)k_dim * tfk::row_gemm_pad_n(n_cols));  // either producer's form (k_dim is a multiple of four)
    if (rc == TF_OK) rc = p->w_lo.alloc((size_t)k_dim * tfk::row_gemm_pad_n(n_cols));
    if (rc == TF_OK) rc = tfk::tc_make_map(&p->tm_whi, p->w_hi.p, n_cols, k_dim, n_cols);
    if (rc == TF_OK) rc = tfk::tc_make_map(&p->tm_wlo, p->w_lo.p, n_cols, k_dim, n_cols);
    if (rc == TF_OK) rc = finish_plan(*p, o, sm_count, false);
    if (rc != TF_OK) return rc;
    pp.max_ctas = p->grid;
  }
  // The launches of their own keep all of T (and where rows are padded, of C: `bytes` in all).  Where the ticket executor would
  // keep a ring of at most 48 MB, that is memory a program may count on (its operands may fill the device), so more than a 48th
  // of it (4 GB) is not taken.  (48 MB hold the ring of a grid up to about 100 columns: this is for some 10 M rows and more.)
  auto keeps_whole = [&](size_t bytes, bool &whole) -> int {
    size_t mem_free = 0, mem = 0;
    TF_CUDA(cudaMemGetInfo(&mem_free, &mem));
    whole = bytes <= mem / 48;
    if (whole) return TF_OK;
    TF_TRY(tf::build_stream_plan(pp, F ? F->ap : nullptr, F ? F->ai : nullptr, A->ap, A->ai, &pt, &ct, p->hp));
    whole = p->hp.ring_rows == 0;  // (it would keep all of T as well)
    if (whole) p->hp = tf::HostPlan();
    return TF_OK;
  };
  // No operator is tiled and nothing asks for the ticket executor's own knobs: the balanced gather runs the chain.
  if (chain == 0 && F && o.mode == TF_MODE_STREAM && !pt.tiled && !ct.tiled && o.ring_bytes <= 0 && o.halo_rows == 0 &&
      o.n_boundary == 0 && o.rows_per_block == 0 && o.slack_blocks < 0 && o.ctas_per_sm == 0) {
    const size_t ld = (n_cols + 3) / 4 * 4 * sizeof(float);
    bool whole = false;
    TF_TRY(keeps_whole(A->m * ld + (n_cols % 4 ? F->n * ld : 0), whole));
    if (whole) return make_gather_plan(p, *F, *A, o, sm_count, out);
  }
  p->tile_info[0] = pt.bx; p->tile_info[1] = pt.by; p->tile_info[2] = pt.bz; p->tile_info[3] = pt.tiles();
  p->tile_info[4] = ct.bx; p->tile_info[5] = ct.by; p->tile_info[6] = ct.bz; p->tile_info[7] = ct.tiles();
  // (The unfused mode takes the two products one after the other in the order in which the one launch takes them where that has
  // one accumulator, so that it gives the same bits there.)
  if (chain == 1 && (o.mode == TF_MODE_STREAM || (o.mode == TF_MODE_UNFUSED && n_cols > 128)) && o.tensor_cores >= 0 &&
      tfk::row_gemm_supported(n_cols) && o.ring_bytes <= 0 && o.halo_rows == 0 && o.n_boundary == 0 && o.rows_per_block == 0 &&
      o.slack_blocks < 0 && o.ctas_per_sm == 0) {
    bool whole = o.mode == TF_MODE_UNFUSED;
    if (!whole) TF_TRY(keeps_whole((size_t)A->m * n_cols * sizeof(float), whole));
    if (whole && ct.tiled && o.lattice_march >= 0) TF_TRY(build_one_launch(*p, *A));
    if (whole && (o.mode == TF_MODE_STREAM || p->one_sums)) return make_gemm_gather_plan(p, *A, o, ct.tiled, sm_count, out);
  }
  rc = p->second.upload(*A);
  if (rc == TF_OK && F && F != A) rc = p->first.upload(*F);
  if (rc != TF_OK) return rc;
  rc = tf::build_stream_plan(pp, F ? F->ap : nullptr, F ? F->ai : nullptr, A->ap, A->ai, &pt, &ct, p->hp);
  if (rc != TF_OK) return rc;
  rc = p->ptile.upload(pt, F ? F->ap : nullptr, F ? F->ax : nullptr, want_pipe);
  if (rc == TF_OK) rc = p->ctile.upload(ct, A->ap, A->ax, want_pipe);
  if (rc != TF_OK) return rc;
  p->pipe = want_pipe && p->hp.ring_rows == 0;
  for (int i = p->hp.phase_begin[1]; p->pipe && i < p->hp.phase_begin[3]; ++i)
    p->pipe = p->hp.items[i].kind == tf::ITEM_PRODUCE_TILED || p->hp.items[i].kind == tf::ITEM_CONSUME_TILED;
  p->pipe_grid = (o.halo_rows > 0 || o.n_boundary > 0) ? std::max(1, sm_count - 8) : sm_count;
  rc = finish_plan(*p, o, sm_count, p->hp.ring_rows > 0);
  if (rc != TF_OK) return rc;

  // with a halo exchange in flight, leave a few SMs half empty so that the NCCL send/recv kernels can
  // start while the persistent executor occupies the GPU (they would otherwise wait for it to drain)
  if ((o.halo_rows > 0 || o.n_boundary > 0) && p->grid > sm_count) p->grid = std::max(sm_count, p->grid - 16);
  // phase 0 items: boundary rows -> send buffer, in runs of consecutive rows
  if (!pp.boundary_rows.empty()) {
    std::vector<tf::Item> pre;
    size_t i = 0;
    while (i < pp.boundary_rows.size()) {
      size_t j = i + 1;
      while (j < pp.boundary_rows.size() && pp.boundary_rows[j] == pp.boundary_rows[j - 1] + 1 &&
             (int)(j - i) < pp.rows_per_block)
        ++j;
      tf::Item it{};
      it.kind = 3; it.row_begin = pp.boundary_rows[i]; it.row_end = pp.boundary_rows[i] + (int)(j - i);
      it.aux0 = (int)i;
      pre.push_back(it);
      i = j;
    }
    const int shift = (int)pre.size();
    p->hp.items.insert(p->hp.items.begin(), pre.begin(), pre.end());
    p->hp.phase_begin[1] += shift; p->hp.phase_begin[2] += shift; p->hp.phase_begin[3] += shift;
    rc = p->sendbuf.alloc(pp.boundary_rows.size() * (size_t)n_cols);
    if (rc != TF_OK) return rc;
  }
  if (o.mode == TF_MODE_STREAM && !o.halo_rows && !o.n_boundary) build_segments(*p, 16);
  rc = upload_items(*p, &pt, &ct);
  if (rc == TF_OK) rc = zero_state(*p);
  if (rc == TF_OK) rc = p->inter.alloc((size_t)p->hp.inter_rows * n_cols);
  if (rc != TF_OK) return rc;
  TF_CUDA(cudaMemset(p->inter.p, 0, p->inter.n * sizeof(float)));
  if (o.mode == TF_MODE_SCHEDULE) {
    rc = load_schedule(*p, sched, chain == 1);
    if (rc != TF_OK) return rc;
  }
  if (chain == 0 && F && o.mode == TF_MODE_STREAM && o.lattice_march >= 0 && o.ring_bytes <= 0 && n_cols % 4 == 0) {
    rc = build_march(*p, F, *A, o.halo_rows, sm_count, pp.boundary_rows);
    if (rc != TF_OK) return rc;
  }
  // GeMM-SpMM with a grid operator, the tensor-core producer and the whole intermediate in memory: the consumer is
  // the marching kernel
  if (chain == 1 && o.mode == TF_MODE_STREAM && o.lattice_march >= 0 && p->use_tc && p->hp.ring_rows == 0 && n_cols % 4 == 0) {
    rc = build_march(*p, nullptr, *A, o.halo_rows, sm_count, pp.boundary_rows);
    if (rc != TF_OK) return rc;
  }
  p->sm_count = sm_count;
  *out = p.release();
  return TF_OK;
}

tfk::Params base_params(tf_plan &p) {
  tfk::Params P;
  std::memset(&P, 0, sizeof(P));
  const DevCsr &f = p.first_is_second ? p.second : p.first;
  P.f_ap = f.ap.p; P.f_ai = f.ai.p; P.f_ax = f.ax.p;
  P.s_ap = p.second.ap.p; P.s_ai = p.second.ai.p; P.s_ax = p.second.ax.p;
  P.inter = p.inter.p;
  P.items = p.items.p;
  P.prod_done = p.prod_done.p; P.cons_done = p.cons_done.p;
  P.st = p.state.p;
  P.n_cols = p.n_cols; P.k_dim = p.k_dim; P.m_local = p.m;
  P.ring_rows = (int)p.hp.ring_rows;
  P.n_prod = p.hp.n_prod;
  P.n_cons = p.hp.n_cons;
  P.tile_rows = p.pipe_rows;
  P.pt = p.ptile.view();
  P.ct = p.ctile.view();
  P.tile_slots = p.tile_slots;
  P.spin_limit = p.spin_limit;
  return P;
}

bool aligned(const void *q, size_t a) { return (reinterpret_cast<uintptr_t>(q) % a) == 0; }
bool march_usable(const tf_plan &p, const float *C, const float *D) {
  return p.march.on && !(p.keep_t && p.march.halves) && (p.march.ragged || (aligned(C, 16) && aligned(D, 16)));
}

// vector width usable with the caller's pointers (plan-owned buffers are always aligned)
void call_shape(const tf_plan &p, std::initializer_list<const void *> ptrs, int *vec, int *ch) {
  bool a16 = true;
  for (const void *q : ptrs) a16 = a16 && (!q || aligned(q, 16));
  tfk::choose_shape(p.n_cols, a16, vec, ch);
}

// Plans that run the staged kernel variant -- gather tiles or the tensor-core producer -- use 16-byte vector
// accesses on the dense operands whatever their width: refuse operands that are not aligned before any launch.
int check_tiled_alignment(const tf_plan &p, const tfk::Params &P) {
  if (p.dyn_smem > 0 && !(aligned(P.in0, 16) && (!P.out || aligned(P.out, 16))))
    return fail(TF_ERR_ARG, "this plan (gather tiles or tensor-core producer) needs 16-byte aligned dense operands "
                            "(build the plan with tile_slots < 0 and tensor_cores < 0 otherwise)");
  return TF_OK;
}

// Tensor-core producer: split the weight for this call and describe B to the TMA unit.
int prepare_tc(tf_plan &p, tfk::Params &P, cudaStream_t s) {
  P.use_tc = 0;
  if (!p.use_tc) return TF_OK;
  TF_CUDA(tfk::tc_split_weight(P.in1, P.w_transposed, p.k_dim, p.n_cols, p.w_hi.p, p.w_lo.p, s));
  int rc = tfk::tc_make_map(&P.tm_a, P.in0, p.m, p.k_dim, tfk::kTcRowsHost);
  if (rc != TF_OK) return rc;
  P.tm_whi = p.tm_whi;
  P.tm_wlo = p.tm_wlo;
  P.use_tc = 1;
  return TF_OK;
}

// One launch over the items [Q.item_begin, Q.item_end) of phases 1 and 2.
cudaError_t launch_items(tf_plan &p, int vec, int ch, bool ring, const tfk::Params &Q, cudaStream_t s) {
  if (p.pipe) return tfk::launch_tile_pipeline(p.pipe_grid, Q, s);
  return tfk::launch_stream(p.chain, vec, ch, ring, p.grid, p.dyn_smem, Q, s);
}

int run_phases(tf_plan &p, tfk::Params &P, int first_phase, int last_phase, cudaStream_t s) {
  int vec, ch;
  call_shape(p, {P.in0, P.in1, P.in2, P.out}, &vec, &ch);
  int rca = check_tiled_alignment(p, P);
  if (rca != TF_OK) return rca;
  if (p.dyn_smem > 0) { vec = 4; ch = 1; }  // the tiled kernel variant; its direct items loop over panels
  rca = prepare_tc(p, P, s);
  if (rca != TF_OK) return rca;
  const bool ring = p.hp.ring_rows > 0;
  if (first_phase <= 1 && last_phase >= 1) ++p.epoch;  // a new pass over the producer blocks
  P.epoch = p.epoch;
  p.launches = 0;
  if (first_phase <= 1 && last_phase >= 1) {
    rca = segments_begin(p, P, s);
    if (rca != TF_OK) return rca;
  }
  for (int ph = first_phase; ph <= last_phase; ++ph) {
    P.item_begin = p.hp.phase_begin[ph];
    P.item_end = p.hp.phase_begin[ph + 1];
    if (P.item_end <= P.item_begin) continue;
    tfk::Params Q = P;
    if (ph == 0) Q.inter = p.sendbuf.p;
    Q.reset_wm = (ph == 2) || (ph == 1 && p.hp.phase_begin[3] == p.hp.phase_begin[2] && last_phase >= 1);
    if (ph == 0) TF_CUDA(tfk::launch_stream(p.chain, vec, ch, ring, p.grid, p.dyn_smem, Q, s));
    else TF_CUDA(launch_items(p, vec, ch, ring, Q, s));
    ++p.launches;
  }
  if (last_phase == 2) return segments_end(p, P, s);
  return TF_OK;
}

// Segments of the item list for the host pipeline: after segment j, the producers listed so far have
// read input rows < in_rows, and every output row < out_rows is final.
void build_segments(tf_plan &p, int n_seg) {
  p.segs.clear();
  const int b = p.hp.phase_begin[1], e = p.hp.phase_begin[2];
  const int n = e - b;
  if (n <= 0 || p.hp.phase_begin[3] != e) return;
  n_seg = std::max(1, std::min(n_seg, n / std::max(1, p.grid)));
  if (!p.hp.seg_t_rows.empty() || !p.hp.seg_out_rows.empty()) n_seg = 1;  // rows finished by atomic adds: no early copies
  std::vector<int> suffix_min(n + 1, p.m);
  for (int i = n - 1; i >= 0; --i) {
    const tf::Item &it = p.hp.items[b + i];
    const bool cons = it.kind == tf::ITEM_CONSUME || it.kind == tf::ITEM_CONSUME_TILED;
    suffix_min[i] = std::min(suffix_min[i + 1], cons ? it.aux1 : p.m);
  }
  long long in_rows = 0;
  for (int s = 0; s < n_seg; ++s) {
    const int i0 = (int)((long long)n * s / n_seg), i1 = (int)((long long)n * (s + 1) / n_seg);
    for (int i = i0; i < i1; ++i) {
      const tf::Item &it = p.hp.items[b + i];
      if (it.kind == tf::ITEM_PRODUCE || it.kind == tf::ITEM_PRODUCE_TILED) in_rows = std::max<long long>(in_rows, it.aux0 + 1LL);
    }
    p.segs.push_back(tf_plan::Seg{b + i0, b + i1, in_rows, (long long)suffix_min[i1]});
  }
}

// Copies of one host-pointer call: plain for pinned arrays, through the pinned rings for pageable ones.
int begin_host_pipe(tf_plan &p, const void *h_in, const void *h_out) {
  if (!p.host_pipe) {
    const int t = (int)std::min(8u, std::max(2u, std::thread::hardware_concurrency() / 2));
    p.host_pipe.reset(new tf::HostPipe(t));
  }
  TF_CUDA(p.host_pipe->begin(p.device, tf::is_pageable(h_in), tf::is_pageable(h_out), (size_t)8 << 20, 16));
  return TF_OK;
}

int ensure_streams(tf_plan &p) {
  if (!p.s_h2d) {
    TF_CUDA(cudaStreamCreateWithFlags(&p.s_h2d, cudaStreamNonBlocking));
    TF_CUDA(cudaStreamCreateWithFlags(&p.s_run, cudaStreamNonBlocking));
    TF_CUDA(cudaStreamCreateWithFlags(&p.s_d2h, cudaStreamNonBlocking));
  }
  return TF_OK;
}

// Host pipeline: the dense input is copied in row chunks on one stream, the item list runs in segments
// on a second as soon as the rows a segment reads have arrived, and finished output rows leave on a
// third.  in_rows x in_cols floats come from h_in; D is m x n_cols.
int run_host_pipeline(tf_plan &p, tfk::Params &P, const float *h_in, long long in_rows, int in_cols, float *d_in,
                      float *h_out, float *d_out) {
  TF_TRY(ensure_streams(p));
  const int ns = (int)p.segs.size();
  while ((int)p.ev_in.size() < ns) {
    cudaEvent_t a, b;
    TF_CUDA(cudaEventCreateWithFlags(&a, cudaEventDisableTiming));
    TF_CUDA(cudaEventCreateWithFlags(&b, cudaEventDisableTiming));
    p.ev_in.push_back(a); p.ev_run.push_back(b);
  }
  int vec, ch;
  call_shape(p, {P.in0, P.in1, P.in2, P.out}, &vec, &ch);
  if (p.dyn_smem > 0) { vec = 4; ch = 1; }
  int rc = prepare_tc(p, P, p.s_run);
  if (rc != TF_OK) return rc;
  rc = begin_host_pipe(p, h_in, h_out);
  if (rc != TF_OK) return rc;
  const bool ring = p.hp.ring_rows > 0;
  ++p.epoch;
  P.epoch = p.epoch;
  p.launches = 0;
  long long in_done = 0, out_done = 0;
  rc = segments_begin(p, P, p.s_run);
  if (rc != TF_OK) return rc;
  for (int s = 0; s < ns; ++s) {
    const tf_plan::Seg &g = p.segs[s];
    const long long in_to = s == ns - 1 ? in_rows : std::min(in_rows, g.in_rows);
    if (in_to > in_done)
      TF_CUDA(p.host_pipe->upload(d_in + in_done * in_cols, h_in + in_done * in_cols, (size_t)(in_to - in_done) * in_cols * 4, p.s_h2d));
    in_done = std::max(in_done, in_to);
    TF_CUDA(cudaEventRecord(p.ev_in[s], p.s_h2d));
    TF_CUDA(cudaStreamWaitEvent(p.s_run, p.ev_in[s], 0));
    tfk::Params Q = P;
    Q.item_begin = g.item_begin; Q.item_end = g.item_end;
    Q.reset_wm = s == ns - 1;
    TF_CUDA(launch_items(p, vec, ch, ring, Q, p.s_run));
    ++p.launches;
    if (s == ns - 1) {
      rc = segments_end(p, P, p.s_run);
      if (rc != TF_OK) return rc;
    }
    TF_CUDA(cudaEventRecord(p.ev_run[s], p.s_run));
    const long long out_to = s == ns - 1 ? p.m : g.out_rows;
    if (out_to > out_done) {
      TF_CUDA(cudaStreamWaitEvent(p.s_d2h, p.ev_run[s], 0));
      TF_CUDA(p.host_pipe->download(h_out + out_done * p.n_cols, d_out + out_done * p.n_cols,
                               (size_t)(out_to - out_done) * p.n_cols * 4, p.s_d2h));
      out_done = out_to;
    }
  }
  TF_CUDA(p.host_pipe->finish());
  TF_CUDA(cudaStreamSynchronize(p.s_d2h));
  TF_CUDA(cudaStreamSynchronize(p.s_run));
  return TF_OK;
}

// The same pipeline for plans that march: one launch per slab of planes (of lines on a 2-D grid, of blocks of rows down a
// band).  A slab [za, zb) reads the planes za - 2 .. zb + 1 of C and completes the planes [za, zb) of D, so the copies run
// two planes ahead of the kernel and the output leaves slab by slab.  Pageable arrays go piece by piece through rings of
// pinned slots (host_stage.h).
int run_host_march(tf_plan &p, const float *h_in, float *d_in, float *h_out, float *d_out) {
  tf_plan::March &M = p.march;
  TF_TRY(ensure_streams(p));
  const bool lines = p.lines.on, band = p.band.block != 0;
  const int nz = lines ? p.lines.ny : (band ? band_blocks(p) : M.nz);
  const long long plane_rows = lines ? p.lines.nx : (band ? p.band.block : (long long)M.nx * M.ny);
  // (lines and blocks: slabs of 2 MB, at most 32 -- smaller copies cost more than what they overlap)
  const int ns = lines || band ? (int)std::max<long long>(1, std::min<long long>({32, nz / 8, (long long)p.m * p.n_cols * 4 >> 21}))
                               : (int)M.slabs.size();
  auto at = [&](int z) { return (size_t)std::min<long long>(p.m, z * plane_rows) * p.n_cols; };  // first float of plane z
  while ((int)p.ev_in.size() < ns) {
    cudaEvent_t a, b;
    TF_CUDA(cudaEventCreateWithFlags(&a, cudaEventDisableTiming));
    TF_CUDA(cudaEventCreateWithFlags(&b, cudaEventDisableTiming));
    p.ev_in.push_back(a); p.ev_run.push_back(b);
  }
  int rc = begin_host_pipe(p, h_in, h_out);
  if (rc != TF_OK) return rc;
  int planes_in = 0;
  long long launches = 0;
  for (int sl = 0; sl < ns; ++sl) {
    const int z_begin = lines || band ? (int)((long long)nz * sl / ns) : M.slabs[sl].z_begin;
    const int z_end = lines || band ? (int)((long long)nz * (sl + 1) / ns) : M.slabs[sl].z_end;
    const int need = std::min(nz, z_end + 2);
    if (need > planes_in)
      TF_CUDA(p.host_pipe->upload(d_in + at(planes_in), h_in + at(planes_in), (at(need) - at(planes_in)) * sizeof(float), p.s_h2d));
    planes_in = std::max(planes_in, need);
    TF_CUDA(cudaEventRecord(p.ev_in[sl], p.s_h2d));
    TF_CUDA(cudaStreamWaitEvent(p.s_run, p.ev_in[sl], 0));
    rc = lines ? run_lines(p, d_in, d_out, z_begin, z_end, p.s_run)
               : (band ? run_band(p, d_in, d_out, z_begin, z_end, p.s_run)
                       : run_march(p, d_in, d_out, M.slabs[sl].item_begin, M.slabs[sl].item_end, false, p.s_run));
    if (rc != TF_OK) return rc;
    launches += p.launches;
    TF_CUDA(cudaEventRecord(p.ev_run[sl], p.s_run));
    TF_CUDA(cudaStreamWaitEvent(p.s_d2h, p.ev_run[sl], 0));
    TF_CUDA(p.host_pipe->download(h_out + at(z_begin), d_out + at(z_begin), (at(z_end) - at(z_begin)) * sizeof(float), p.s_d2h));
  }
  p.launches = launches;
  if (lines || band) TF_TRY(leave_intermediate(p, d_in, p.s_run));
  TF_CUDA(p.host_pipe->finish());
  TF_CUDA(cudaStreamSynchronize(p.s_d2h));
  TF_CUDA(cudaStreamSynchronize(p.s_run));
  return TF_OK;
}

int run_unfused(tf_plan &p, tfk::Params &P, cudaStream_t s) {
  // all producers are listed before all consumers: one launch per half, T through HBM
  int vec, ch;
  call_shape(p, {P.in0, P.in1, P.in2, P.out}, &vec, &ch);
  int rca = check_tiled_alignment(p, P);
  if (rca != TF_OK) return rca;
  if (p.dyn_smem > 0) { vec = 4; ch = 1; }
  rca = prepare_tc(p, P, s);
  if (rca != TF_OK) return rca;
  ++p.epoch;
  P.epoch = p.epoch;
  const int np = P.n_prod;
  p.launches = 0;
  rca = segments_begin(p, P, s);
  if (rca != TF_OK) return rca;
  tfk::Params Q = P;
  Q.item_begin = 0; Q.item_end = np; Q.reset_wm = 0;
  TF_CUDA(launch_items(p, vec, ch, false, Q, s));
  Q.item_begin = np; Q.item_end = (int)p.hp.items.size(); Q.reset_wm = 1;
  TF_CUDA(launch_items(p, vec, ch, false, Q, s));
  p.launches = 2;
  return segments_end(p, P, s);
}

int run_schedule(tf_plan &p, tfk::Params &P, cudaStream_t s) {
  int vec, ch;
  call_shape(p, {P.in0, P.in1, P.in2, P.out}, &vec, &ch);
  p.launches = 0;
  for (int l = 0; l < p.s_n1; ++l) {
    const int nparts = p.s_ptr1[l + 1] - p.s_ptr1[l];
    if (nparts <= 0) continue;
    const int grid = std::min(nparts, p.grid);
    TF_CUDA(tfk::launch_schedule_level(p.chain, vec, ch, grid, P, p.s_ptr2.p, p.s_id.p, p.s_type.p,
                                       p.s_has_ker ? p.s_ker.p : nullptr, p.s_ptr1[l], p.s_ptr1[l + 1], s));
    ++p.launches;
  }
  return TF_OK;
}

int run_chain(tf_plan &p, tfk::Params &P, cudaStream_t s) {
  if (p.mode == TF_MODE_SCHEDULE) return run_schedule(p, P, s);
  if (p.mode == TF_MODE_UNFUSED) return run_unfused(p, P, s);
  return run_phases(p, P, 1, 2, s);
}

// Y = op * X, both row-major with their own row lengths; vec_in / vec_out: rows start on 16-byte boundaries.
tfk::GatherParams gather_params(const DevGather &g, const float *X, int ld_in, float *Y, int ld_out, int n_cols) {
  tfk::GatherParams P;
  std::memset(&P, 0, sizeof(P));
  P.cols = g.cols.p; P.vals = g.vals.p; P.units = g.units.p; P.rows = g.rows.p; P.heavy = g.heavy.p;
  P.heavy_cnt = g.cnt.p; P.partial = g.partial.p; P.partial_ld = g.partial_ld;
  P.dense = X; P.ld_in = ld_in;
  P.out = Y; P.ld_out = ld_out;
  P.n_cols = n_cols;
  P.n_units = g.n_units;
  return P;
}
// (a run of units: the caller has seen to the empty rows)
int run_gather(const DevGather &g, const float *X, int ld_in, bool vec_in, float *Y, int ld_out, bool vec_out, int n_cols,
               bool relu, cudaStream_t s, int unit_begin = 0, int unit_end = -1, void *scratch = nullptr) {
  tfk::GatherParams P = gather_params(g, X, ld_in, Y, ld_out, n_cols);
  if (scratch && g.heavy.n) {
    P.heavy_cnt = (int *)scratch;
    P.partial = (float *)((char *)scratch + g.scratch_counters());
    TF_CUDA(cudaMemsetAsync(scratch, 0, g.cnt.n * sizeof(int), s));
  }
  P.relu = relu ? 1 : 0;
  if (unit_end >= 0) { P.units += unit_begin; P.n_units = unit_end - unit_begin; }
  else TF_CUDA(tfk::launch_rows_fix(g.empty.p, g.n_empty, ld_out, Y, false, s));
  TF_CUDA(tfk::launch_gather(vec_in, vec_out, P, s));
  return TF_OK;
}

int run_gather_spmm_spmm(tf_plan &p, const float *C, float *D, cudaStream_t s) {
  const DevGather &f = p.first_is_second ? p.g_second : p.g_first;
  const float *src = C;
  int ld = p.n_cols;
  bool vec = ld % 4 == 0 && aligned(C, 16);
  if (p.g_pad.n) {
    TF_CUDA(tfk::launch_pad_rows(C, p.first_cols, p.n_cols, p.ld_t, p.g_pad.p, s));
    src = p.g_pad.p; ld = p.ld_t; vec = true;
  }
  int rc = run_gather(f, src, ld, vec, p.inter.p, p.ld_t, true, vec ? p.ld_t : p.n_cols, false, s);
  if (rc != TF_OK) return rc;
  p.launches = p.g_pad.n ? 3 : 2;
  return run_gather(p.g_second, p.inter.p, p.ld_t, true, D, p.n_cols, p.n_cols % 4 == 0 && aligned(D, 16), p.n_cols, false, s);
}

// GeMM-SpMM in one launch; split: the weight may have changed since the launch before.
int run_one_launch(tf_plan &p, const float *B, const float *W, int w_transposed, bool relu, float *D, int brick_begin, int brick_end, bool split,
                   cudaStream_t s) {
  p.launches = 1;
  if (split && !tfk::spmm_gemm_resident(p.k_dim, p.n_cols)) {
    TF_CUDA(tfk::row_gemm_split(W, w_transposed, p.k_dim, p.n_cols, tfk::kSumsFree, p.w_hi.p, p.w_lo.p, s));
    p.launches = 2;
  }
  tfk::SpmmGemmParams P = p.one.par;
  P.b = B; P.w = W; P.out = D;
  P.k = p.k_dim; P.n = p.n_cols; P.w_transposed = w_transposed;
  P.brick_begin = brick_begin; P.brick_end = brick_end;
  P.relu = relu ? 1 : 0;
  P.error = &p.state.p->error; P.wait_limit = p.spin_limit;
  return tfk::spmm_gemm(P, p.w_hi.p, p.w_lo.p, p.sm_count, s);
}

// The two products in launches of their own, T in between (`t`, rows of p.ld_t floats).
int run_two_products(tf_plan &p, const float *B, const float *W, int w_transposed, bool relu, float *D, float *t, cudaStream_t s) {
  const int n = p.n_cols, k = p.k_dim;
  TF_CUDA(tfk::row_gemm_split(W, w_transposed, k, n, p.sums(), p.w_hi.p, p.w_lo.p, s));
  p.launches = tfk::row_gemm_form(k, n) == tfk::kRowFma ? 2 : 3;
  if (p.spmm_first) {
    TF_TRY(run_gather(p.g_second, B, k, aligned(B, 16), t, p.ld_t, true, k, false, s));
    return tfk::row_gemm(t, p.m, k, p.ld_t, W, w_transposed, p.w_hi.p, p.w_lo.p, n, D, n, relu, p.sums(), &p.state.p->error,
                         p.spin_limit, p.sm_count, s);
  }
  TF_TRY(tfk::row_gemm(B, p.m, k, k, W, w_transposed, p.w_hi.p, p.w_lo.p, n, t, p.ld_t, false, p.sums(),
                       &p.state.p->error, p.spin_limit, p.sm_count, s));
  return run_gather(p.g_second, t, p.ld_t, true, D, n, n % 4 == 0 && aligned(D, 16), n, relu, s);
}

bool overlap(const float *a, size_t na, const float *b, size_t nb) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return x < y + nb * sizeof(float) && y < x + na * sizeof(float);
}

int run_gather_gemm_spmm(tf_plan &p, const float *B, const float *W, int w_transposed, bool relu, float *D, cudaStream_t s) {
  const size_t rows = (size_t)p.m, n = (size_t)p.n_cols, k = (size_t)p.k_dim;
  if (p.dyn_smem > 0 && !(aligned(B, 16) && aligned(D, 16)))
    return fail(TF_ERR_ARG, "this plan (gather tiles or tensor-core producer) needs 16-byte aligned dense operands "
                            "(build the plan with tile_slots < 0 and tensor_cores < 0 otherwise)");
  if (!p.one.on || p.keep_t) return run_two_products(p, B, W, w_transposed, relu, D, p.inter.p, s);
  if (!overlap(D, rows * n, B, rows * k) && !overlap(D, rows * n, W, k * n))
    return run_one_launch(p, B, W, w_transposed, relu, D, 0, p.one.par.grid.bricks(), true, s);
  // The one launch reads B and W while it writes D.  Where D lies over either, T is formed first; it comes from the stream's pool
  // for the call, so that such a call can be captured as any other.
  float *t = nullptr;
  TF_CUDA(cudaMallocAsync(&t, rows * p.ld_t * sizeof(float), s));
  const int rc = run_two_products(p, B, W, w_transposed, relu, D, t, s);
  const cudaError_t e = cudaFreeAsync(t, s);
  if (rc == TF_OK) TF_CUDA(e);
  return rc;
}

int set_device(const tf_plan &p) {
  TF_CUDA(cudaSetDevice(p.device));
  return TF_OK;
}

}  // namespace

extern "C" {

int tf_plan_spmm_spmm(const tf_csr *A, const tf_csr *B, int n_cols, const tf_plan_opts *o,
                      const tf_schedule *sched, tf_plan **out) {
  return make_chain_plan(0, A, B, 0, n_cols, o, sched, out);
}

int tf_plan_gemm_spmm(const tf_csr *A, int k, int n_cols, const tf_plan_opts *o, const tf_schedule *sched,
                      tf_plan **out) {
  if (k <= 0) return fail(TF_ERR_ARG, "plan: inner dimension must be positive");
  return make_chain_plan(1, A, nullptr, k, n_cols, o, sched, out);
}

int tf_plan_sddmm_spmm(const tf_csr *A, int kq, int nv, const tf_plan_opts *opts, tf_plan **out) {
  if (!A || !out) return fail(TF_ERR_ARG, "plan: null argument");
  if (kq <= 0 || nv <= 0) return fail(TF_ERR_ARG, "plan: dense widths must be positive");
  tf_plan_opts o;
  int rc = check_opts(opts, o);
  if (rc != TF_OK) return rc;
  if (A->m <= 0 || A->n <= 0) return fail(TF_ERR_ARG, "plan: matrix must have rows and columns");
  rc = tf::check_csr(A->m, A->n, A->ap, A->ai, false);
  if (rc != TF_OK) return rc;
  if (!A->ax) return fail(TF_ERR_ARG, "plan: null value array");
  int sm_count = 0;
  rc = device_ready(&sm_count);
  if (rc != TF_OK) return rc;
  std::unique_ptr<tf_plan> p(new tf_plan());
  cudaGetDevice(&p->device);
  p->chain = 2; p->mode = TF_MODE_STREAM;
  p->m = A->m; p->n_cols = nv; p->k_dim = kq;
  if (tfk::sddmm_gather_supported(kq, nv) && o.rows_per_block == 0 && o.ctas_per_sm == 0) {
    p->second.m = A->m; p->second.n = A->n;
    rc = p->g_second.build(*A, 4 * tfk::sddmm_group(kq, nv), nv, sm_count, false, tfk::sddmm_resident(kq, nv));  // (units for groups of that size)
    if (rc == TF_OK) rc = zero_state(*p);
    if (rc != TF_OK) return rc;
    *out = p.release();
    return TF_OK;
  }
  rc = p->second.upload(*A);
  if (rc != TF_OK) return rc;
  p->first_is_second = true;
  tf::PlanParams pp;
  pp.m = A->m; pp.n_cols = nv;
  pp.rows_per_block = o.rows_per_block > 0 ? o.rows_per_block : 32;
  pp.max_block_nnz = pp.rows_per_block * 32;
  rc = tf::build_single_pass_plan(pp, A->ap, p->hp);
  if (rc == TF_OK) rc = finish_plan(*p, o, sm_count, false);
  if (rc == TF_OK) rc = upload_items(*p);
  if (rc == TF_OK) rc = zero_state(*p);
  if (rc != TF_OK) return rc;
  *out = p.release();
  return TF_OK;
}

void tf_plan_free(tf_plan *p) { delete p; }

int tf_plan_info(const tf_plan *p, long long info[8]) {
  if (!p || !info) return fail(TF_ERR_ARG, "tf_plan_info: null argument");
  info[0] = (long long)p->hp.items.size();
  info[1] = p->hp.n_prod;
  info[2] = p->hp.n_cons;
  info[3] = p->hp.ring_rows;
  info[4] = p->march.on ? p->march.grid : (p->pipe ? p->pipe_grid : p->grid);
  info[5] = p->march.on         ? tfk::kMarchThreads
            : p->lines.on       ? 32 * tfk::kLineWarps
            : p->band.block     ? tfk::band_threads(p->band.block, p->band.par, p->sm_count)
            : p->one.on && !p->keep_t ? tfk::kSpmmGemmThreads
            : p->pipe           ? 672
            : p->g_second.on    ? tfk::kThreads
            : p->dyn_smem > 0   ? tfk::tiled_threads(p->chain)
                                : tfk::kThreads;
  info[6] = p->launches;
  info[7] = p->hp.inter_rows;
  return TF_OK;
}

int tf_plan_tile_info(const tf_plan *p, int info[8]) {
  if (!p || !info) return fail(TF_ERR_ARG, "tf_plan_tile_info: null argument");
  for (int i = 0; i < 8; ++i) info[i] = p->tile_info[i];
  return TF_OK;
}

int tf_plan_set_wait_limit(tf_plan *p, int polls) {
  if (!p || polls <= 0) return fail(TF_ERR_ARG, "tf_plan_set_wait_limit: bad argument");
  p->spin_limit = polls;
  return TF_OK;
}

int tf_plan_status(tf_plan *p, void *stream) {
  if (!p) return fail(TF_ERR_ARG, "tf_plan_status: null plan");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  TF_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  if (p->march.on) {
    tfk::MarchState ms[2];
    TF_CUDA(cudaMemcpy(ms, p->march.st.p, sizeof(ms), cudaMemcpyDeviceToHost));
    if (ms[0].error || ms[1].error) {
      cudaMemset(p->march.st.p, 0, sizeof(ms));
      return fail(TF_ERR_TIMEOUT, "a bounded in-kernel wait ran out; the output of the last call is not valid");
    }
  }
  tfk::ExecState st;
  TF_CUDA(cudaMemcpy(&st, p->state.p, sizeof(st), cudaMemcpyDeviceToHost));
  if (st.error) {
    // leave the plan usable: clear the executor state
    cudaMemset(p->state.p, 0, sizeof(st));
    return fail(TF_ERR_TIMEOUT, "a bounded in-kernel wait ran out; the output of the last call is not valid");
  }
  return TF_OK;
}

int tf_exec_spmm_spmm(tf_plan *p, const float *C, float *D, void *stream) {
  if (!p || !C || !D) return fail(TF_ERR_ARG, "tf_exec_spmm_spmm: null argument");
  if (p->chain != 0) return fail(TF_ERR_ARG, "tf_exec_spmm_spmm: plan was built for another chain");
  if (p->halo_rows || p->sendbuf.n) return fail(TF_ERR_ARG, "tf_exec_spmm_spmm: plan has halo rows, drive it with tf_exec_phase");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  if (p->lines.on || p->band.block) {
    TF_TRY(p->lines.on ? run_lines(*p, C, D, 0, p->lines.ny, (cudaStream_t)stream) : run_band(*p, C, D, 0, band_blocks(*p), (cudaStream_t)stream));
    return leave_intermediate(*p, C, (cudaStream_t)stream);
  }
  if (march_usable(*p, C, D)) return run_march(*p, C, D, 0, p->march.n_items, false, (cudaStream_t)stream);
  if (p->g_second.on) return run_gather_spmm_spmm(*p, C, D, (cudaStream_t)stream);
  tfk::Params P = base_params(*p);
  P.in0 = C; P.out = D;
  return run_chain(*p, P, (cudaStream_t)stream);
}

// GeMM-SpMM on a grid operator: the dense producer writes all rows of T (one launch of the tensor-core kernel), the
// marching kernel consumes them (items [item_begin, item_end)).
int run_gemm_march(tf_plan &p, const float *B, const float *W, int w_transposed, bool relu, float *D, bool produce, int item_begin,
                   int item_end, bool with_halo, cudaStream_t s) {
  long long launches = 0;
  if (produce) {
    TF_CUDA(tfk::row_gemm_split(W, w_transposed, p.k_dim, p.n_cols, p.sums(), p.w_hi.p, p.w_lo.p, s));
    int rc = tfk::row_gemm(B, p.m, p.k_dim, p.k_dim, W, w_transposed, p.w_hi.p, p.w_lo.p, p.n_cols, p.inter.p, p.n_cols, false,
                           p.sums(), &p.march.st.p[0].error, p.spin_limit, p.sm_count, s);
    if (rc != TF_OK) return rc;
    launches = tfk::row_gemm_form(p.k_dim, p.n_cols) == tfk::kRowFma ? 1 : 2;   // (weight split and) dense product
  }
  if (p.march.n_star > 0) {
    int rc = run_star(p, D, relu, s);
    p.launches += launches;
    return rc;
  }
  int rc = run_march(p, p.inter.p, D, item_begin, item_end, with_halo, s);
  p.launches += launches;
  return rc;
}

bool gemm_march_usable(const tf_plan &p, const float *B, const float *D, int relu) {
  return p.chain == 1 && p.march.on && p.march.identity_first && (!relu || p.march.n_star > 0) && aligned(B, 16) && aligned(D, 16);
}

int tf_exec_gemm_spmm(tf_plan *p, const float *B, const float *W, int w_transposed, int relu, float *D,
                      void *stream) {
  if (!p || !B || !W || !D) return fail(TF_ERR_ARG, "tf_exec_gemm_spmm: null argument");
  if (p->chain != 1) return fail(TF_ERR_ARG, "tf_exec_gemm_spmm: plan was built for another chain");
  if (p->halo_rows || p->sendbuf.n) return fail(TF_ERR_ARG, "tf_exec_gemm_spmm: plan has halo rows, drive it with tf_exec_phase");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  if (gemm_march_usable(*p, B, D, relu))
    return run_gemm_march(*p, B, W, w_transposed, relu != 0, D, true, 0, p->march.n_items, false, (cudaStream_t)stream);
  if (p->g_second.on) return run_gather_gemm_spmm(*p, B, W, w_transposed, relu != 0, D, (cudaStream_t)stream);
  tfk::Params P = base_params(*p);
  P.in0 = B; P.in1 = W; P.out = D; P.w_transposed = w_transposed; P.relu = relu;
  return run_chain(*p, P, (cudaStream_t)stream);
}

int tf_exec_sddmm_spmm(tf_plan *p, const float *Q, const float *K, const float *V, float *D, void *stream) {
  if (!p || !Q || !K || !V || !D) return fail(TF_ERR_ARG, "tf_exec_sddmm_spmm: null argument");
  if (p->chain != 2) return fail(TF_ERR_ARG, "tf_exec_sddmm_spmm: plan was built for another chain");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  if (p->g_second.on) {
    const DevGather &g = p->g_second;
    const tfk::GatherParams G = gather_params(g, V, p->n_cols, D, p->n_cols, p->n_cols);
    TF_CUDA(tfk::launch_rows_fix(g.empty.p, g.n_empty, p->n_cols, D, false, (cudaStream_t)stream));
    TF_CUDA(tfk::launch_sddmm_gather(G, Q, K, p->k_dim, p->m, (cudaStream_t)stream));
    p->launches = 1;
    return TF_OK;
  }
  tfk::Params P = base_params(*p);
  P.in0 = Q; P.in1 = K; P.in2 = V; P.out = D;
  return run_phases(*p, P, 1, 1, (cudaStream_t)stream);
}

size_t tf_exec_spmm_work_bytes(const tf_plan *p) { return p && p->g_second.on ? p->g_second.scratch_bytes() : 0; }

int tf_exec_spmm(tf_plan *p, const float *X, int n_cols, float *out, void *stream) {
  return tf_exec_spmm_work(p, X, n_cols, out, nullptr, 0, stream);
}

int tf_exec_spmm_work(tf_plan *p, const float *X, int n_cols, float *out, void *work, size_t work_bytes, void *stream) {
  if (!p || !X || !out) return fail(TF_ERR_ARG, "tf_exec_spmm: null argument");
  if (work && (work_bytes < tf_exec_spmm_work_bytes(p) || !aligned(work, 16)))
    return fail(TF_ERR_ARG, "tf_exec_spmm_work: work space too small or not on a 16-byte boundary");
  if (n_cols <= 0) return fail(TF_ERR_ARG, "tf_exec_spmm: bad width");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  const cudaStream_t s = (cudaStream_t)stream;
  if (p->g_second.on) {
    const DevGather &g = p->g_second;
    const bool in16 = n_cols % 4 == 0 && aligned(X, 16), out16 = n_cols % 4 == 0 && aligned(out, 16);
    // (as many columns at a time as the partial sums of cut rows have room for; the first pass sees to the rows without nonzeros)
    for (int c = 0; c < n_cols; c += g.partial_ld)
      TF_TRY(run_gather(g, X + c, n_cols, in16, out + c, n_cols, out16, std::min(g.partial_ld, n_cols - c), false, s, 0,
                        c ? g.n_units : -1, work));
    return TF_OK;
  }
  if (!p->second.ap.n) TF_TRY(restore_csr(*p, true));
  return tf_spmm_dev(p->second.ap.p, p->second.ai.p, p->second.ax.p, p->m, X, n_cols, out, stream);
}

int tf_exec_phase(tf_plan *p, int phase, const float *in0, const float *in1, int w_transposed, int relu,
                  float *D, void *stream) {
  if (!p || !in0) return fail(TF_ERR_ARG, "tf_exec_phase: null argument");
  if (phase < 0 || phase > 2) return fail(TF_ERR_ARG, "tf_exec_phase: phase must be 0, 1 or 2");
  if (p->chain > 1 || p->mode != TF_MODE_STREAM) return fail(TF_ERR_ARG, "tf_exec_phase: stream-mode chain plans only");
  if (p->chain == 1 && !in1) return fail(TF_ERR_ARG, "tf_exec_phase: GeMM-SpMM needs the weight");
  if (phase > 0 && !D) return fail(TF_ERR_ARG, "tf_exec_phase: null output");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  // plane-marching plans: phase 0 (boundary rows of T for the neighbours: two planes at most) is a plain CSR product
  // of those rows into the send buffer -- a fraction of the time the general executor's launch takes for so little
  // work --, phases 1 and 2 run on the marching kernel, the second with the received planes of T
  if (phase == 0 && p->chain == 0 && p->march.on && p->march.n_boundary > 0 && aligned(in0, 16)) {
    const tf_plan::March &M = p->march;
    int vec, ch;
    tfk::choose_shape(p->n_cols, aligned(in0, 16) && aligned(p->sendbuf.p, 16), &vec, &ch);
    const int grid = std::max(1, std::min((M.n_boundary + tfk::kWarps - 1) / tfk::kWarps, 148 * 8));
    TF_CUDA(tfk::launch_spmm(vec, ch, grid, M.b_ap.p, M.b_ai.p, M.b_ax.p, M.n_boundary, in0, p->n_cols, p->sendbuf.p,
                             (cudaStream_t)stream));
    p->launches = 1;
    return TF_OK;
  }
  if (phase == 2 && p->march.n_star > 0) {  // no exchange: phase 1 was the whole chain
    p->launches = 0;
    return TF_OK;
  }
  if (phase > 0 && gemm_march_usable(*p, in0, D, relu))
    return phase == 1 ? run_gemm_march(*p, in0, in1, w_transposed, relu != 0, D, true, 0, p->march.n_phase1, false, (cudaStream_t)stream)
                      : run_gemm_march(*p, in0, in1, w_transposed, relu != 0, D, false, p->march.n_phase1, p->march.n_items, true,
                                       (cudaStream_t)stream);
  if (phase > 0 && p->chain == 0 && march_usable(*p, in0, D))
    return phase == 1 ? run_march(*p, in0, D, 0, p->march.n_phase1, false, (cudaStream_t)stream)
                      : run_march(*p, in0, D, p->march.n_phase1, p->march.n_items, true, (cudaStream_t)stream);
  if (p->lines.on || p->band.block) {  // no exchange: phase 1 is the whole chain
    p->launches = 0;
    return phase == 1 ? tf_exec_spmm_spmm(p, in0, D, stream) : TF_OK;
  }
  if (p->g_second.on) {  // no exchange: phase 1 is the whole chain
    p->launches = 0;
    if (phase != 1) return TF_OK;
    return p->chain == 0 ? run_gather_spmm_spmm(*p, in0, D, (cudaStream_t)stream)
                         : run_gather_gemm_spmm(*p, in0, in1, w_transposed, relu != 0, D, (cudaStream_t)stream);
  }
  tfk::Params P = base_params(*p);
  P.in0 = in0; P.in1 = in1; P.out = D; P.w_transposed = w_transposed; P.relu = relu;
  return run_phases(*p, P, phase, phase, (cudaStream_t)stream);
}

int tf_plan_intermediate(tf_plan *p, float **dev_ptr, long long *rows, int *cols) {
  if (!p) return fail(TF_ERR_ARG, "tf_plan_intermediate: null plan");
  if (!p->keep_t) {  // executors that leave no T = F C (T = B W) in memory do so from now on
    TF_TRY(set_device(*p));
    if (p->spmm_first) {
      p->ld_t = (p->n_cols + 3) / 4 * 4;
      TF_TRY(p->inter.alloc((size_t)(p->m + 1) * p->ld_t));
      p->spmm_first = false;
    } else if (p->lines.on || p->band.block) {
      TF_TRY(restore_csr(*p, false));
      TF_TRY(p->inter.alloc((size_t)p->m * p->n_cols));
      p->hp.inter_rows = p->m;
    } else if (p->one.on) {
      TF_TRY(p->inter.alloc((size_t)(p->m + 1) * p->ld_t));
      p->hp.inter_rows = p->m;
    }
    p->keep_t = true;
  }
  if (dev_ptr) *dev_ptr = p->inter.p;
  if (rows) *rows = p->hp.inter_rows;
  if (cols) *cols = p->ld_t ? p->ld_t : p->n_cols;
  return TF_OK;
}

int tf_plan_exchange_buffers(tf_plan *p, float **send, long long *send_rows, float **halo, long long *halo_rows) {
  if (!p) return fail(TF_ERR_ARG, "tf_plan_exchange_buffers: null plan");
  if (send) *send = p->sendbuf.p;
  if (send_rows) *send_rows = p->n_cols ? (long long)(p->sendbuf.n / p->n_cols) : 0;
  if (halo) *halo = p->halo_rows ? p->inter.p + (size_t)(p->hp.inter_rows - p->halo_rows) * p->n_cols : nullptr;
  if (halo_rows) *halo_rows = p->halo_rows;
  return TF_OK;
}

// ---- host-pointer executors -------------------------------------------------
static int stage_in(DevBuf<float> &buf, const float *h, size_t count, cudaStream_t s) {
  if (buf.n < count) { int rc = buf.alloc(count); if (rc != TF_OK) return rc; }
  TF_CUDA(cudaMemcpyAsync(buf.p, h, count * sizeof(float), cudaMemcpyHostToDevice, s));
  return TF_OK;
}

static int finish_host(tf_plan *p, float *D, size_t count) {
  if (p->h_out.n < count) return fail(TF_ERR_ARG, "internal: output staging missing");
  TF_CUDA(cudaMemcpyAsync(D, p->h_out.p, count * sizeof(float), cudaMemcpyDeviceToHost, 0));
  return tf_plan_status(p, nullptr);
}

// Graph operators: any row of D may need any row of C, so the call is upload, both products, download; pageable arrays
// still go through the pinned rings.
static int run_host_whole(tf_plan &p, const float *C, size_t nin, float *D, size_t nout, const std::function<int()> &run) {
  int rc = ensure_streams(p);
  if (rc == TF_OK) rc = begin_host_pipe(p, C, D);
  if (rc != TF_OK) return rc;
  TF_CUDA(p.host_pipe->upload(p.h_in0.p, C, nin * sizeof(float), p.s_run));
  rc = run();
  if (rc != TF_OK) return rc;
  TF_CUDA(p.host_pipe->download(D, p.h_out.p, nout * sizeof(float), p.s_run));
  TF_CUDA(p.host_pipe->finish());
  TF_CUDA(cudaStreamSynchronize(p.s_run));
  return TF_OK;
}

// Both chains on the pieces of a plan (make_gather_pieces): rows of the input (B or C) arrive in pieces, the rows of T that a
// piece can make follow, then the rows of D that have all they need, which leave while the next piece arrives.
static int run_host_pieces(tf_plan &p, const float *in, int w_transposed, bool relu, float *D) {
  const DevGather &g = p.g_second, &f = p.first_is_second ? p.g_second : p.g_first;
  const bool gemm = p.chain == 1;
  const bool one = p.one.on && !p.keep_t;
  const std::vector<tf_plan::Piece> &pieces = one ? p.one.pieces : p.pieces;
  const int ns = (int)pieces.size(), n = p.n_cols, k = gemm ? p.k_dim : p.n_cols;  // k: width of the input
  while ((int)p.ev_in.size() < ns) {
    cudaEvent_t a, b;
    TF_CUDA(cudaEventCreateWithFlags(&a, cudaEventDisableTiming));
    TF_CUDA(cudaEventCreateWithFlags(&b, cudaEventDisableTiming));
    p.ev_in.push_back(a); p.ev_run.push_back(b);
  }
  TF_TRY(begin_host_pipe(p, in, D));
  if (one) {}
  else if (gemm) TF_CUDA(tfk::row_gemm_split(p.h_in1.p, w_transposed, k, n, p.sums(), p.w_hi.p, p.w_lo.p, p.s_run));
  else TF_CUDA(tfk::launch_rows_fix(f.empty.p, f.n_empty, p.ld_t, p.inter.p, false, p.s_run));
  TF_CUDA(tfk::launch_rows_fix(g.empty.p, g.n_empty, n, p.h_out.p, false, p.s_run));
  const bool pad = p.g_pad.n != 0, vec = pad || n % 4 == 0;  // (the buffers of the call start on 16-byte boundaries)
  long long in_done = 0, out_done = 0;
  p.launches = 1;
  for (int s = 0; s < ns; ++s) {
    const tf_plan::Piece &sg = pieces[s];
    const long long in_to = gemm && s == ns - 1 ? p.m : std::max(in_done, sg.in_rows);
    if (in_to > in_done) {
      float *src = p.h_in0.p + in_done * k;
      TF_CUDA(p.host_pipe->upload(src, in + in_done * k, (size_t)(in_to - in_done) * k * 4, p.s_h2d));
      TF_CUDA(cudaEventRecord(p.ev_in[s], p.s_h2d));
      TF_CUDA(cudaStreamWaitEvent(p.s_run, p.ev_in[s], 0));
      if (one) {
      } else if (gemm) {
        TF_TRY(tfk::row_gemm(src, (int)(in_to - in_done), k, k, p.h_in1.p, w_transposed, p.w_hi.p, p.w_lo.p, n,
                             p.inter.p + in_done * p.ld_t, p.ld_t, false, p.sums(), &p.state.p->error, p.spin_limit, p.sm_count, p.s_run));
        ++p.launches;
      } else if (pad) {
        TF_CUDA(tfk::launch_pad_rows(src, in_to - in_done, n, p.ld_t, p.g_pad.p + in_done * p.ld_t, p.s_run));
        ++p.launches;
      }
      in_done = in_to;
    }
    if (!gemm && sg.f_end > sg.f_begin) {
      TF_TRY(run_gather(f, pad ? p.g_pad.p : p.h_in0.p, pad ? p.ld_t : n, vec, p.inter.p, p.ld_t, true, vec ? p.ld_t : n, false, p.s_run,
                        sg.f_begin, sg.f_end));
      ++p.launches;
    }
    const long long before = p.launches;
    if (one) TF_TRY(run_one_launch(p, p.h_in0.p, p.h_in1.p, w_transposed, relu, p.h_out.p, sg.begin, sg.end, s == 0, p.s_run));
    else TF_TRY(run_gather(g, p.inter.p, p.ld_t, true, p.h_out.p, n, n % 4 == 0, n, relu, p.s_run, sg.begin, sg.end));
    p.launches = before + 1;
    if (sg.out_rows > out_done) {
      TF_CUDA(cudaEventRecord(p.ev_run[s], p.s_run));
      TF_CUDA(cudaStreamWaitEvent(p.s_d2h, p.ev_run[s], 0));
      TF_CUDA(p.host_pipe->download(D + out_done * n, p.h_out.p + out_done * n, (size_t)(sg.out_rows - out_done) * n * 4, p.s_d2h));
      out_done = sg.out_rows;
    }
  }
  TF_CUDA(p.host_pipe->finish());
  TF_CUDA(cudaStreamSynchronize(p.s_d2h));
  TF_CUDA(cudaStreamSynchronize(p.s_run));
  return TF_OK;
}

int tf_spmm_spmm_host(tf_plan *p, const float *C, float *D) {
  if (!p || !C || !D) return fail(TF_ERR_ARG, "tf_spmm_spmm_host: null argument");
  if (p->chain != 0) return fail(TF_ERR_ARG, "tf_spmm_spmm_host: plan was built for another chain");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  const size_t nd = (size_t)p->m * p->n_cols;
  if (!p->march.slabs.empty() || ((p->lines.on || p->band.block) && nd * sizeof(float) >= ((size_t)1 << 20))) {
    const size_t nin = (size_t)p->first_cols * p->n_cols;
    if (p->h_in0.n < nin) rc = p->h_in0.alloc(nin);
    if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
    if (rc != TF_OK) return rc;
    if (p->lines.on || p->band.block || march_usable(*p, p->h_in0.p, p->h_out.p)) {
      rc = run_host_march(*p, C, p->h_in0.p, D, p->h_out.p);
      if (rc != TF_OK) return rc;
      return tf_plan_status(p, nullptr);
    }
  }
  if (p->segs.size() > 1) {
    const size_t nin = (size_t)p->first_cols * p->n_cols;
    if (p->h_in0.n < nin) rc = p->h_in0.alloc(nin);
    if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
    if (rc != TF_OK) return rc;
    tfk::Params P = base_params(*p);
    P.in0 = p->h_in0.p; P.out = p->h_out.p;
    rc = run_host_pipeline(*p, P, C, p->first_cols, p->n_cols, p->h_in0.p, D, p->h_out.p);
    if (rc != TF_OK) return rc;
    return tf_plan_status(p, nullptr);
  }
  if (p->g_second.on && nd * sizeof(float) >= ((size_t)1 << 20)) {
    const size_t nin = (size_t)p->first_cols * p->n_cols;
    if (p->h_in0.n < nin) rc = p->h_in0.alloc(nin);
    if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
    if (rc == TF_OK) rc = ensure_streams(*p);
    if (rc == TF_OK)
      rc = !p->pieces.empty() ? run_host_pieces(*p, C, 0, false, D)
                              : run_host_whole(*p, C, nin, D, nd, [&] { return run_gather_spmm_spmm(*p, p->h_in0.p, p->h_out.p, p->s_run); });
    if (rc != TF_OK) return rc;
    return tf_plan_status(p, nullptr);
  }
  rc = stage_in(p->h_in0, C, (size_t)p->first_cols * p->n_cols, 0);
  if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
  if (rc == TF_OK) rc = tf_exec_spmm_spmm(p, p->h_in0.p, p->h_out.p, nullptr);
  if (rc != TF_OK) return rc;
  return finish_host(p, D, nd);
}

int tf_gemm_spmm_host(tf_plan *p, const float *B, const float *W, int w_transposed, int relu, float *D) {
  if (!p || !B || !W || !D) return fail(TF_ERR_ARG, "tf_gemm_spmm_host: null argument");
  if (p->chain != 1) return fail(TF_ERR_ARG, "tf_gemm_spmm_host: plan was built for another chain");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  const size_t nd = (size_t)p->m * p->n_cols;
  if (p->segs.size() > 1) {
    const size_t nin = (size_t)p->m * p->k_dim;
    if (p->h_in0.n < nin) rc = p->h_in0.alloc(nin);
    if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
    if (rc != TF_OK) return rc;
    TF_TRY(ensure_streams(*p));
    rc = stage_in(p->h_in1, W, (size_t)p->k_dim * p->n_cols, p->s_run);  // the weight first, on the stream that uses it
    if (rc != TF_OK) return rc;
    tfk::Params P = base_params(*p);
    P.in0 = p->h_in0.p; P.in1 = p->h_in1.p; P.out = p->h_out.p; P.w_transposed = w_transposed; P.relu = relu;
    rc = run_host_pipeline(*p, P, B, p->m, p->k_dim, p->h_in0.p, D, p->h_out.p);
    if (rc != TF_OK) return rc;
    return tf_plan_status(p, nullptr);
  }
  if (p->g_second.on && nd * sizeof(float) >= ((size_t)1 << 20)) {
    const size_t nin = (size_t)p->m * p->k_dim;
    if (p->h_in0.n < nin) rc = p->h_in0.alloc(nin);
    if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
    if (rc != TF_OK) return rc;
    TF_TRY(ensure_streams(*p));
    TF_TRY(stage_in(p->h_in1, W, (size_t)p->k_dim * p->n_cols, p->s_run));  // the weight first, on the stream that uses it
    if (!p->pieces.empty() || (p->one.on && !p->keep_t)) rc = run_host_pieces(*p, B, w_transposed, relu != 0, D);
    else
      rc = run_host_whole(*p, B, nin, D, nd, [&] {
        return run_gather_gemm_spmm(*p, p->h_in0.p, p->h_in1.p, w_transposed, relu != 0, p->h_out.p, p->s_run);
      });
    if (rc != TF_OK) return rc;
    return tf_plan_status(p, nullptr);
  }
  rc = stage_in(p->h_in0, B, (size_t)p->m * p->k_dim, 0);
  if (rc == TF_OK) rc = stage_in(p->h_in1, W, (size_t)p->k_dim * p->n_cols, 0);
  if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
  if (rc == TF_OK) rc = tf_exec_gemm_spmm(p, p->h_in0.p, p->h_in1.p, w_transposed, relu, p->h_out.p, nullptr);
  if (rc != TF_OK) return rc;
  return finish_host(p, D, nd);
}

int tf_sddmm_spmm_host(tf_plan *p, const float *Q, const float *K, const float *V, float *D) {
  if (!p || !Q || !K || !V || !D) return fail(TF_ERR_ARG, "tf_sddmm_spmm_host: null argument");
  if (p->chain != 2) return fail(TF_ERR_ARG, "tf_sddmm_spmm_host: plan was built for another chain");
  int rc = set_device(*p);
  if (rc != TF_OK) return rc;
  const size_t nd = (size_t)p->m * p->n_cols;
  rc = stage_in(p->h_in0, Q, (size_t)p->m * p->k_dim, 0);
  if (rc == TF_OK) rc = stage_in(p->h_in1, K, (size_t)p->second.n * p->k_dim, 0);
  if (rc == TF_OK) rc = stage_in(p->h_in2, V, (size_t)p->second.n * p->n_cols, 0);
  if (rc == TF_OK && p->h_out.n < nd) rc = p->h_out.alloc(nd);
  if (rc == TF_OK) rc = tf_exec_sddmm_spmm(p, p->h_in0.p, p->h_in1.p, p->h_in2.p, p->h_out.p, nullptr);
  if (rc != TF_OK) return rc;
  return finish_host(p, D, nd);
}

int tf_spmm_dev(const int *Ap, const int *Ai, const float *Ax, int m, const float *X, int n_cols, float *out,
                void *stream) {
  if (!Ap || !Ai || !Ax || !X || !out) return fail(TF_ERR_ARG, "tf_spmm_dev: null argument");
  if (m < 0 || n_cols <= 0) return fail(TF_ERR_ARG, "tf_spmm_dev: bad size");
  int vec, ch;
  tfk::choose_shape(n_cols, aligned(X, 16) && aligned(out, 16), &vec, &ch);
  const int grid = std::max(1, std::min((m + tfk::kWarps - 1) / tfk::kWarps, 148 * 8));
  TF_CUDA(tfk::launch_spmm(vec, ch, grid, Ap, Ai, Ax, m, X, n_cols, out, (cudaStream_t)stream));
  return TF_OK;
}

int tf_fill_uniform(float *dev, long long count, unsigned long long seed, long long offset, void *stream) {
  if (!dev || count < 0) return fail(TF_ERR_ARG, "tf_fill_uniform: bad argument");
  TF_CUDA(tfk::launch_fill(false, dev, count, seed, offset, 1.f, (cudaStream_t)stream));
  return TF_OK;
}

int tf_fill_normal(float *dev, long long count, unsigned long long seed, long long offset, float sigma,
                   void *stream) {
  if (!dev || count < 0) return fail(TF_ERR_ARG, "tf_fill_normal: bad argument");
  TF_CUDA(tfk::launch_fill(true, dev, count, seed, offset, sigma, (cudaStream_t)stream));
  return TF_OK;
}

}  // extern "C"
