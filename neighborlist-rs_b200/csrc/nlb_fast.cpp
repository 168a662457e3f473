// nlb_fast.cpp -- single-system, single-cutoff cell-list builds without a
// host round trip in the middle, replayed as a CUDA graph.
//
// The pipeline (bin histogram memset, atom prep, bin scan, scatter, placement,
// group count, group emit) is issued back to back on the caller's stream.
// The emit pass reads the edge total from device memory and writes into a
// capacity-bounded arena (the previous total x 1.25, or a density estimate);
// the host learns the total from the count pass, and only if the arena or
// the count's records were too small does it grow them and run the missing
// passes again.
//
// Mode 1 (nlb_single_pipeline), and narrow cells of a few atoms, take the
// pair-task kernels of the multi-cutoff path instead: count per (atom, stencil
// cell), scan, emit.
//
// The first call with a given set of launch parameters runs the work
// directly; a repeated call with identical parameters (same positions
// buffer, cell, cutoff, sizes and workspace) captures the sequence into a
// CUDA graph and replays it from then on.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "nlb_internal.h"

namespace nlb {

namespace {

// Everything the issued work depends on; compared bytewise.
struct FastKey {
  const double* d_pos;
  int64_t n;
  GridParams grid;
  GuardBand band;
  cudaStream_t stream;
  void* bufs[kSlotCount];
  int64_t capacity;
  int64_t mask_cap;
  int32_t need_rank;
  int32_t prof;
  int32_t split;  // segments per group (0: pair tasks)
  int32_t bucket;
  int32_t ex_flags;
  // The output options' cell: the grid does not tell an auto-box, whose
  // vectors have no H S term, from a cell with the same matrix.
  int32_t ex_has_cell;
  double ex_h[9];
};

struct FastState {
  FastKey key;
  bool have_key = false;
  cudaGraphExec_t exec = nullptr;
  int launches = 0;  // kernels per replay
  int64_t last_m = 0;
  int64_t last_mask_words = 0;
  int64_t last_records = 0;  // records the last group search asked for
};

thread_local FastState tl_states[16];

FastState& state_for(Ctx& c) { return tl_states[c.device & 15]; }

int64_t stencil_cells_of(const GridParams& g) {
  return (int64_t)(2 * g.ns[0] + 1) * (2 * g.ns[1] + 1) * (2 * g.ns[2] + 1);
}

// 64-bit words of the group search's zeroed state.
int64_t group_state_words(int64_t max_groups) {
  return 16 + 16 * kGroupRegions + group_blocks(max_groups) + (max_groups + 1) / 2;
}

// Expected edges for sizing the first arena: half the pairs within rc at the
// system's mean density, plus one list entry per atom of slack.
int64_t estimate_edges(const SystemPlan& sp, double rc) {
  const double* h = sp.cell.h;
  const double det = h[0] * (h[4] * h[8] - h[7] * h[5]) - h[1] * (h[3] * h[8] - h[6] * h[5]) +
                     h[2] * (h[3] * h[7] - h[6] * h[4]);
  const double vol = std::fabs(det);
  const double rho = vol > 0 ? (double)sp.n / vol : 0.0;
  const double per_atom = 0.5 * rho * (4.0 / 3.0) * 3.141592653589793 * rc * rc * rc;
  const double est = (double)sp.n * (per_atom + 1.0);
  return (int64_t)std::min(est, 4.0e12);
}

std::atomic<int32_t> g_pipeline_mode{0};

}  // namespace

namespace {
thread_local int32_t tl_last_pipeline = -1;  // pipeline of this thread's last fast-path build
}  // namespace

int32_t single_pipeline_mode() { return g_pipeline_mode.load(); }
int32_t last_single_pipeline() { return tl_last_pipeline; }
int32_t set_single_pipeline_mode(int32_t mode) { return g_pipeline_mode.exchange(mode); }

void release_fast_states() {
  for (FastState& fs : tl_states) {
    if (fs.exec) cudaGraphExecDestroy(fs.exec);
    fs = FastState();
  }
}

// The result arrays for `capacity` half edges.
bool out_arrays(Ctx& c, SystemPlan& sp, int64_t capacity) {
  const size_t edges = (size_t)capacity * (sp.ex_flags & NLB_DIRECTED ? 2 : 1);
  sp.out_src = slot<int64_t>(c, kSlotOutEi, 2 * edges);
  sp.out_sh = slot<int32_t>(c, kSlotOutSh, 3 * edges);
  const bool vec = sp.ex_flags & NLB_VECTORS, dist = sp.ex_flags & NLB_DISTANCES;
  sp.out_vec = vec ? slot<double>(c, kSlotOutVec, 3 * edges) : nullptr;
  sp.out_dist = dist ? slot<double>(c, kSlotOutDist, edges) : nullptr;
  return sp.out_src && sp.out_sh && (!vec || sp.out_vec) && (!dist || sp.out_dist);
}

// Sizes every workspace buffer of the fast pipeline (may allocate; never
// inside a capture).
Status prepare_fast(Ctx& c, SystemPlan& sp, int64_t capacity, int64_t mask_cap) {
  const int64_t n = sp.n;
  const int64_t nb = sp.grid.total_bins;
  const int64_t cells = stencil_cells_of(sp.grid);
  const int64_t row = n * cells + 1;
  sp.row = row;
  GridBuffers& b = sp.gb;
  const void* tab_before = c.bufs[kSlotRankTab].p;
  const size_t tab_cap = c.bufs[kSlotRankTab].cap;
  b.rank_of_bin = slot<int32_t>(c, kSlotRankTab, nb);
  sp.rank_cached = b.rank_of_bin == tab_before && tab_cap > 0 && c.rank_nb[0] == sp.grid.nb[0] &&
                   c.rank_nb[1] == sp.grid.nb[1] && c.rank_nb[2] == sp.grid.nb[2];
  // Zeroed block, so that a single memset at the start clears everything and
  // the kernels follow each other directly: bin histogram, scatter cursors, 2
  // task counters, 64-bit mask cursor (8-byte aligned: 2 nb + 2 is even),
  // build completion count, emit task counter, loose flag, a word unused, then
  // (8-byte aligned) the offsets scan's state, or the group search's ticket,
  // error word, total, completion count, record cursor, block sums and segment
  // counts and the bin scan's state.
  const int64_t max_groups = n / 32 + std::min<int64_t>(n, nb) + 1;
  const bool bin_scan = sp.grouped && nb > kPrepBinScanMax;
  const int64_t group_words = group_state_words(max_groups);
  const int64_t words64 = sp.grouped ? group_words + (bin_scan ? bin_scan_words(nb) : 0)
                                     : scan_tmp_elems(row);
  sp.zeroed_words = 2 * (size_t)nb + 8 + 2 * (size_t)words64;
  int32_t* zeroed = slot<int32_t>(c, kSlotBinCount, sp.zeroed_words);
  if (!zeroed) return fail(NLB_ERR_NOMEM, "device allocation failed");
  b.bin_count = zeroed;
  b.bin_fill = zeroed + nb;
  b.counters = zeroed + 2 * nb;
  b.mask_top = reinterpret_cast<unsigned long long*>(zeroed + 2 * nb + 2);
  b.build_done = zeroed + 2 * nb + 4;
  b.emit_queue = reinterpret_cast<uint32_t*>(zeroed + 2 * nb + 5);
  b.loose = zeroed + 2 * nb + 6;
  int64_t* state = reinterpret_cast<int64_t*>(zeroed + 2 * nb + 8);
  sp.scan_state = state;
  b.bin_scan = bin_scan ? reinterpret_cast<uint64_t*>(state + group_words) : nullptr;
  b.group_start = sp.grouped ? slot<int32_t>(c, kSlotGroupStart, nb) : nullptr;
  b.fill = slot<int32_t>(c, kSlotFill, n);
  const int64_t max_tasks = max_groups * cells;
  // (The group search needs no task headers, masks, counts or offsets.)
  b.task_hdr = slot<int4>(c, kSlotTaskHdr, sp.grouped ? 1 : max_tasks);
  if (sp.grouped) {
    GroupSearch& o = sp.search;
    const int32_t split = o.split;
    std::memset(&o, 0, sizeof(o));
    o.split = split;
    o.state = reinterpret_cast<uint64_t*>(state);
    o.total = state + 2;
    o.done = reinterpret_cast<int32_t*>(state + 3);
    o.records = state + 4;
    o.chunk_top = reinterpret_cast<unsigned long long*>(state + 16);
    o.block_sum = reinterpret_cast<uint64_t*>(state + 16 + 16 * kGroupRegions);
    o.group_done =
        reinterpret_cast<int32_t*>(state + 16 + 16 * kGroupRegions + group_blocks(max_groups));
    o.chunk_cap = mask_cap / 32;
    o.masks = slot<uint32_t>(c, kSlotMasks, mask_cap);
    o.cand = slot<uint32_t>(c, kSlotCand, mask_cap);
    o.cshift = slot<uint32_t>(c, kSlotCshift, mask_cap);
    o.block_base = slot<int64_t>(c, kSlotGroupBase, group_blocks(max_groups));
    o.group_total = slot<int64_t>(c, kSlotGroupTotal, max_groups);
    o.atom_base = slot<int64_t>(c, kSlotAtomBase, 32 * (size_t)max_groups);
    o.seg_cnt = slot<uint32_t>(c, kSlotSegCnt, (size_t)max_groups * split * 32);
    o.seg_rec = slot<longlong2>(c, kSlotSegRec, (size_t)max_groups * split);
    o.max_groups = max_groups;
    o.withhold = -1;
    o.spin_limit = kGroupSpinLimit;
    o.report = c.prof ? nullptr : c.d_report;
    if (!o.masks || !o.cand || !o.cshift || !o.block_base || !o.group_total || !o.atom_base || !o.seg_cnt || !o.seg_rec ||
        !b.group_start)
      return fail(NLB_ERR_NOMEM, "device allocation failed");
    b.masks = nullptr;
    b.mask_cap = 0;
  } else {
    b.masks = slot<uint32_t>(c, kSlotMasks, mask_cap);
    b.mask_cap = mask_cap;
    if (!b.masks) return fail(NLB_ERR_NOMEM, "device allocation failed");
  }
  const bool chunk_boxes = !sp.grouped && nb > 0 && (double)n / (double)nb >= kChunkPruneMinPerBin;
  b.cbox = chunk_boxes ? slot<float4>(c, kSlotCbox, 2 * (size_t)n) : nullptr;
  b.bin_start = slot<int64_t>(c, kSlotBinStart, nb + 1);
  b.key = slot<uint64_t>(c, kSlotKey, n);
  b.rank = slot<int32_t>(c, kSlotRank, n);
  const int64_t entries = b.bucket > 0 ? nb * b.bucket : n;
  b.skey = slot<uint64_t>(c, kSlotSkey, entries);
  b.sidx = slot<int32_t>(c, kSlotSidx, entries);
  b.skey2 = slot<uint64_t>(c, kSlotSkey2, n);
  b.sidx2 = slot<int32_t>(c, kSlotSidx2, n);
  b.px = slot<double>(c, kSlotPx, n);
  b.py = slot<double>(c, kSlotPy, n);
  b.pz = slot<double>(c, kSlotPz, n);
  b.meta = slot<SlotMeta>(c, kSlotMeta, n);
  b.p32 = slot<float4>(c, kSlotP32, n);
  b.sbin = slot<int32_t>(c, kSlotSbin, n);
  b.groups = slot<GroupRec>(c, kSlotGroups, n / 32 + std::min<int64_t>(n, nb) + 1);
  b.irr_list = slot<int32_t>(c, kSlotIrrList, n);
  b.irr = slot<uint8_t>(c, kSlotIrr, n);
  b.scan_tmp = slot<int64_t>(c, kSlotScanTmp, scan_tmp_elems(sp.grouped ? nb : std::max<int64_t>(row, nb)));
  sp.counts = slot<uint32_t>(c, kSlotCounts, sp.grouped ? 1 : row);
  sp.offs = slot<int64_t>(c, kSlotOffs, sp.grouped ? 1 : row + 1);
  if (!out_arrays(c, sp, capacity))
    return fail(NLB_ERR_NOMEM, "device allocation for the edge lists failed");
  if (!b.rank_of_bin || !b.bin_start || !b.key || !b.rank || !b.skey || !b.sidx || !b.skey2 ||
      !b.sidx2 || !b.px || !b.py || !b.pz || !b.meta || !b.p32 || !b.sbin || !b.groups ||
      !b.irr_list || !b.irr || !b.scan_tmp || !sp.counts || !sp.offs ||
      !b.task_hdr || (chunk_boxes && !b.cbox) || !b.fill)
    return fail(NLB_ERR_NOMEM, "device allocation failed");
  return Status{NLB_OK};
}

// Segments per group: slices of the row of its candidates (stencils of up to
// 32 cells), or runs of stencil cells.
//   * As many as give the chip one round of warps (28 per SM): fewer leave
//     warps idle (10,008 atoms at rc 6: 90 us with two per group, 75 with six
//     to nine), more describe the cells again (81 us with twelve); slices of
//     at least 24 candidates (1000 isolated atoms: 70 us with 16 to 24, 78
//     with 64; a cell of 60 atoms: 58 with 16, 57 with 24 to 32).
//   * Runs of cells (more than 32 of them: narrow cells) of at least 96
//     candidates: a segment per cell, of one to ten candidates in a cell of a
//     few atoms, leaves the group's last warp up to 729 segments to add up (1
//     atom in a skewed cell at rc 7: 69 us, 51 with 48 candidates, 53 with 96;
//     16 atoms at rc 20: 74, 60, 58, and 66 with 24; 60 at rc 25: 78, 76, 76,
//     and 83 with a limit of 64 runs; all without the pair tasks that narrow
//     cells take unless output options are wanted).
//   * Large bins (above kSplitDense atoms): slices of about 192 candidates, up
//     to 18,000 segments.  A slice near the group is all hits, and a warp with
//     a whole cell of them was the last to end by far (10,008 atoms at rc 14:
//     198 us with one segment per cell, 190 with slices of 192, 202 with 96;
//     30,000 atoms at rc 14: 508 us per cell, 450 with slices of 192, 426 with
//     384).
constexpr double kSplitDense = 64.0;
constexpr int64_t kSplitTarget = 5000, kSplitDenseTarget = 18000;
constexpr int64_t kSplitLeast = 24, kSplitCells = 96, kSplitSlice = 192;
int32_t group_split(int64_t n, int64_t nb, int64_t cells) {
  const int64_t groups = n / 32 + std::min<int64_t>(n, nb) + 1;  // (at most)
  const int64_t row = (int64_t)((double)cells * (double)n / (double)nb);  // candidates of a group
  int64_t want = kSplitTarget / groups;
  if ((double)n > kSplitDense * (double)nb)
    want = std::max(want, std::min(row / kSplitSlice, kSplitDenseTarget / groups));
  want = std::min({want, cells <= 32 ? row / kSplitLeast : std::min(cells, row / kSplitCells),
                   ((int64_t)1 << 30) / groups});
  return (int32_t)std::max<int64_t>(want, 1);
}

// Records the group search asks room for: one per 32 candidates of a segment,
// with the groups and candidates of a uniform density.
int64_t group_records(int64_t n, int64_t nb, int64_t cells, int32_t split) {
  const double per_bin = (double)n / (double)nb;
  const double filled = (double)nb * (1.0 - std::exp(-per_bin));
  const double groups = std::max(filled, (double)n / 32.0 + 0.5 * filled) + 1.0;
  const double records = groups * ((double)cells * per_bin / 32.0 + split);
  return (int64_t)std::min(1.25 * records, 1e12) + 64 * kGroupRegions;
}

double group_search_bytes(int64_t n, double volume, double rc) {
  // (bins at least rc wide, 27 stencil cells)
  const double bins = volume / (rc * rc * rc);
  const int64_t nb = bins > 1.0 ? (int64_t)std::min(bins, 1e9) : 1;
  const int32_t split = group_split(n, nb, 27);
  const double groups = (double)n / 32.0 + (double)std::min<int64_t>(n, nb) + 1.0;
  double bytes = 384.0 * (double)group_records(n, nb, 27, split) +  // masks, candidates, shifts
                 groups * (280.0 + 144.0 * split);                  // offsets, segment counts
  if (bucket_build(n, nb)) bytes += 12.0 * (double)nb * bucket_entries(n, nb);
  return 1.25 * bytes;
}

// Hits the emit pass stages at a time.  A segment whose records hold more is
// written in several windows, each with its own loads and scan; a larger stage
// leaves fewer warps on an SM (25 with 1536 hits, 16 with 4096).  By the most a
// segment can be expected to hold: all pairs of its slice, or all hits of its
// group.  The small stage (us a call, small / large stage):
//   * groups in several segments, up to 2560 hits: 10,008 atoms at rc 6 59.4 /
//     61.4, 10,000 at rc 5 54.0 / 56.5, at rc 7 65.3 / 67.1, 15,000 at rc 6 63.9 /
//     66.8, 20,001 with vectors at rc 5 87.2 / 88.9, 2,000 at rc 8 56.0 / 57.2;
//   * groups in one segment, up to 1024 hits: 40,000 atoms at rc 5 83 / 87,
//     80,000 107 / 112; at rc 6, with 1,480, some gain and some lose (40,000 97 /
//     95, 60,000 115 / 119, 100,000 153 / 149);
//   * long launches of groups whose hits mostly fit it: a million atoms at rc 6
//     763 / 836, 300,000 276 / 293.
// The large one for the rest: 400,000 atoms at rc 8 895 / 774, 78,000 at rc 14
// 891 / 760 (712 with 6144, but 100,000 at rc 6 137 -> 146), 10,008 at rc 14 158
// / 145, 30,000 at rc 8 113 / 108.
constexpr int32_t kStageSmall = 1536, kStageLarge = 4096;
constexpr double kStageSplit = 2560.0, kStageWhole = 1024.0, kStageLong = 2048.0;  // hits
constexpr int64_t kStageFew = 20000;  // segments
int32_t group_stage(const SystemPlan& sp) {
  const double hits = 32.0 * (double)estimate_edges(sp, std::sqrt(sp.rc_sq[0])) / (double)sp.n;
  const int64_t items = sp.search.max_groups * sp.search.split;
  const double slice = (double)stencil_cells_of(sp.grid) * (double)sp.n /
                       ((double)sp.grid.total_bins * (double)sp.search.split);
  const double most = std::min(32.0 * slice, hits);
  if (most <= (sp.search.split > 1 ? kStageSplit : kStageWhole)) return kStageSmall;
  return items > kStageFew && hits <= kStageLong ? kStageSmall : kStageLarge;
}

// The group search's two launches.
void issue_search(Ctx& c, SystemPlan& sp, const double* d_pos, int64_t capacity, bool count) {
  const GroupBand band = group_band(sp.band);
  const int32_t cells = (int32_t)stencil_cells_of(sp.grid);
  if (count) {
    GroupSearch o = sp.search;
    int32_t tile = 0, spins = 0;
    if (take_scan_stall(&tile, &spins)) {  // failure-detection hook
      o.withhold = tile;
      o.spin_limit = spins;
    }
    launch_group_count(sp.grid, sp.gb, cells, band, o, c.stream);
    c.mark(2);
    c.mark(3);
    c.mark(4);
  }
  GroupOut out;
  std::memset(&out, 0, sizeof(out));
  out.ei = sp.out_src;
  out.sh = sp.out_sh;
  out.vec = sp.out_vec;
  out.dist = sp.out_dist;
  out.pos = d_pos;
  out.cell = sp.ex_cell;
  out.capacity = capacity;
  out.directed = sp.ex_flags & NLB_DIRECTED ? 1 : 0;
  out.stage = group_stage(sp);
  out.orig_bits = 2;
  while (((int64_t)1 << out.orig_bits) < sp.n) ++out.orig_bits;
  launch_group_emit(sp.grid, sp.gb, cells, band, sp.search, out, c.stream);
}

EmitTargets fast_targets(const SystemPlan& sp, int64_t capacity, int64_t* report = nullptr) {
  EmitTargets t;
  std::memset(&t, 0, sizeof(t));
  t.src[0] = sp.out_src;
  t.sh[0] = sp.out_sh;
  t.total_dev = sp.offs + sp.row;
  t.capacity = capacity;
  t.scan_error = sp.scan_state + 1;
  t.report = report;
  t.mask_top = sp.gb.mask_top;
  t.grid_scan_error = bin_scan_error(sp.grid, sp.gb);
  return t;
}

// Issues the whole pipeline on c.stream (no host synchronisation).
void issue_fast(Ctx& c, SystemPlan& sp, const double* d_pos, int64_t capacity) {
  cudaStream_t s = c.stream;
  const int64_t n = sp.n;
  c.mark(0);
  cudaMemsetAsync(sp.gb.bin_count, 0, sizeof(int32_t) * sp.zeroed_words, s);
  launch_grid_build(sp.grid, d_pos, n, sp.gb, s, !sp.rank_cached);
  c.mark(1);
  if (sp.grouped) {
    // (Phases: the offsets are part of the count pass.)
    issue_search(c, sp, d_pos, capacity, true);
    c.mark(5);
    return;
  }
  launch_pair_count(sp.grid, sp.gb, n, sp.band, sp.counts, s);
  c.mark(2);
  exclusive_scan_u32_zeroed(sp.counts, sp.row, sp.offs, sp.scan_state, s);
  c.mark(3);
  c.mark(4);
  launch_pair_emit(sp.grid, sp.gb, n, sp.band, sp.offs,
                   fast_targets(sp, capacity, c.prof ? nullptr : c.d_report), s);
  c.mark(5);
}

Status wait_report(Ctx& c) {
  volatile int64_t* r = c.h_report;
  for (uint32_t k = 1; r[0] == 0; ++k) {
    if ((k & 127) != 0) continue;
    const cudaError_t q = cudaStreamQuery(c.stream);
    if (q == cudaErrorNotReady) continue;
    if (q != cudaSuccess) return cuda_fail(q, "neighbour-list pipeline");
    if (r[0] == 0) {
      // (a launch that failed to start leaves its error with the runtime)
      const cudaError_t le = cudaGetLastError();
      if (le != cudaSuccess) return cuda_fail(le, "neighbour-list pipeline launch");
      return fail(NLB_ERR_CUDA, "the search ended without its report");
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return Status{NLB_OK};
}

// Runs the fast pipeline for a planned single-cutoff cell-list system and
// leaves M edges in sp.out_src ([src | dst]) / sp.out_sh.
//
// (The group search counts a row of candidates -- at most 32 images of all
// atoms -- in 32 bits.)
// Narrow cells, whose stencils have hundreds of cells, keep the pair tasks up to
// 128 atoms: one to four groups leave the group search with long runs of nearly
// empty cells and one warp that adds them up, while a warp per (group, cell)
// spreads them over the chip.  Device time of a repeated build, pair tasks / group
// search, us: 1 atom, 729 cells 39 / 41, 16 atoms, 729 cells 39 / 46, 32 atoms,
// 343 cells 39 / 46, 60 atoms, 567 cells 48 / 55, 100 atoms, 343 cells 56 / 58;
// 200 atoms, 245 cells 73 / 64, 100 atoms, 125 cells 54 / 47.  With output
// options the group search's one pass wins (66 / 62 to 75 / 80 us a call).
constexpr int64_t kNarrowCells = 125, kNarrowAtoms = 128;
bool takes_group_search(const SystemPlan& sp, int ex_flags) {
  if (!fast_eligible(sp) || single_pipeline_mode() != 0 || sp.n >= ((int64_t)1 << 26)) return false;
  return ex_flags || sp.n > kNarrowAtoms || stencil_cells_of(sp.grid) <= kNarrowCells;
}

// The build without the memory that the searches above ask for: the group
// search's records, or result arrays by the density's estimate.  FP64 per-atom
// passes with 12 bytes an atom besides the cell list, and result arrays of
// exactly M edges; the output options are left to the caller (sp.ex_flags 0).
Status run_lean(Ctx& c, SystemPlan& sp, const double* d_pos, int64_t* m_out,
                bool stream_ordered) {
  FastState& fs = state_for(c);
  fs.have_key = false;
  for (int s : {kSlotMasks, kSlotCand, kSlotCshift, kSlotAtomBase, kSlotSegCnt, kSlotSegRec,
                kSlotTaskHdr, kSlotCounts, kSlotOffs, kSlotSkey, kSlotOutEi, kSlotOutSh,
                kSlotOutVec, kSlotOutDist})
    c.drop(s);
  sp.gb = GridBuffers{};
  sp.fp32 = false;
  sp.grouped = false;
  sp.ex_flags = 0;
  Status st = count_system(c, sp, d_pos);
  if (!st.ok()) return st;
  DevLists L;
  st = device_outputs(c, sp.m, L);
  if (!st.ok()) return st;
  const int64_t zero = 0;
  st = emit_system(c, sp, d_pos, L, &zero, 0);
  if (!st.ok()) return st;
  sp.out_src = L.src[0];
  sp.out_sh = L.sh[0];
  if (c.stream == c.own_stream) {
    const cudaError_t e = stream_ordered ? cudaSuccess : cudaStreamSynchronize(c.stream);
    if (e != cudaSuccess) return cuda_fail(e, "neighbour-list pipeline");
  } else {
    const cudaError_t e = cudaEventRecord(c.early_ev, c.stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
    c.early_stream = c.stream;
  }
  *m_out = sp.m[0];
  return Status{NLB_OK};
}

// M reaches the host through host-mapped memory as soon as it is known: when
// the count pass ends (mode 1: when its emit pass starts).  On a caller's
// stream the call then returns at once: the emit is queued on that stream
// ahead of anything the caller queues there.  On the library's own stream it
// also waits for that work.
Status run_fast(Ctx& c, SystemPlan& sp, const double* d_pos, int64_t* m_out,
                bool stream_ordered) {
  FastState& fs = state_for(c);
  const int64_t cells = stencil_cells_of(sp.grid);
  sp.grouped = takes_group_search(sp, sp.ex_flags);
  sp.search.split = sp.grouped ? group_split(sp.n, sp.grid.total_bins, cells) : 0;
  tl_last_pipeline = sp.grouped ? 0 : 1;
  sp.gb.bucket = 0;
  if (sp.grouped && bucket_build(sp.n, sp.grid.total_bins))
    sp.gb.bucket = bucket_entries(sp.n, sp.grid.total_bins);
  const double rc = std::sqrt(sp.rc_sq[0]);
  int64_t capacity = std::max<int64_t>(
      {4096, (int64_t)(1.25 * (double)fs.last_m), (int64_t)(1.5 * (double)estimate_edges(sp, rc))});
  // Keep the arena's current size if it is already large enough.
  const size_t per = sp.ex_flags & NLB_DIRECTED ? 2 : 1;
  size_t have = std::min(c.bufs[kSlotOutSh].cap / (3 * sizeof(int32_t)),
                         c.bufs[kSlotOutEi].cap / (2 * sizeof(int64_t)));
  if (sp.ex_flags & NLB_VECTORS)
    have = std::min(have, c.bufs[kSlotOutVec].cap / (3 * sizeof(double)));
  if (sp.ex_flags & NLB_DISTANCES) have = std::min(have, c.bufs[kSlotOutDist].cap / sizeof(double));
  if ((int64_t)(have / per) > capacity) capacity = (int64_t)(have / per);
  // Hit-mask arena: the last run's need x 1.25, at least 64 words per atom;
  // the group search's records (32 words each) by the density, or the last
  // run's need.
  int64_t mask_cap = std::max<int64_t>(64 * sp.n + 4096, fs.last_mask_words + fs.last_mask_words / 4);
  if (sp.grouped)
    mask_cap = 32 * std::max<int64_t>(
                        group_records(sp.n, sp.grid.total_bins, cells, sp.search.split),
                        fs.last_records + fs.last_records / 8);
  int64_t mask_have = (int64_t)(c.bufs[kSlotMasks].cap / sizeof(uint32_t));
  if (sp.grouped)
    mask_have = std::min({mask_have, (int64_t)(c.bufs[kSlotCand].cap / sizeof(uint32_t)),
                          (int64_t)(c.bufs[kSlotCshift].cap / sizeof(uint32_t))});
  if (mask_have > mask_cap) mask_cap = mask_have;
  Status st = prepare_fast(c, sp, capacity, mask_cap);
  if (st.code == NLB_ERR_NOMEM) return run_lean(c, sp, d_pos, m_out, stream_ordered);
  if (!st.ok()) return st;

  FastKey key;
  std::memset(&key, 0, sizeof(key));
  key.d_pos = d_pos;
  key.n = sp.n;
  key.grid = sp.grid;
  key.band = sp.band;
  key.stream = c.stream;
  for (int i = 0; i < kSlotCount; ++i) key.bufs[i] = c.bufs[i].p;
  key.capacity = capacity;
  key.mask_cap = mask_cap;
  key.need_rank = sp.rank_cached ? 0 : 1;
  key.prof = c.prof ? 1 : 0;
  key.split = sp.search.split;
  key.bucket = sp.gb.bucket;
  key.ex_flags = sp.ex_flags;
  key.ex_has_cell = sp.ex_cell.has_cell;
  std::memcpy(key.ex_h, sp.ex_cell.h, sizeof(key.ex_h));

  const bool report = !c.prof;
  if (report) c.h_report[0] = 0;

  // (An armed failure-detection hook must reach a directly launched scan,
  // never a captured or replayed one.)
  const bool same = !scan_stall_armed() && fs.have_key &&
                    std::memcmp(&key, &fs.key, sizeof(key)) == 0;
  bool launched = false;
  if (same && fs.exec) {
    if (cudaGraphLaunch(fs.exec, c.stream) == cudaSuccess) {
      note_launches(fs.launches);
      note_graph_replay();
      launched = true;
    } else {
      cudaGetLastError();
    }
  } else if (same && c.stream != nullptr && c.stream != cudaStreamLegacy && !c.prof) {
    // (Profiling runs stay outside graphs: its per-phase events are timed on
    // directly launched kernels.)
    // Second identical call: capture the sequence once and replay it.
    if (fs.exec) {
      cudaGraphExecDestroy(fs.exec);
      fs.exec = nullptr;
    }
    cudaGraph_t graph = nullptr;
    const int64_t l0 = nlb_kernel_launches();
    if (cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      issue_fast(c, sp, d_pos, capacity);
      if (cudaStreamEndCapture(c.stream, &graph) == cudaSuccess && graph) {
        if (cudaGraphInstantiate(&fs.exec, graph, 0) != cudaSuccess) fs.exec = nullptr;
        cudaGraphDestroy(graph);
      }
    }
    cudaGetLastError();
    fs.launches = (int)(nlb_kernel_launches() - l0);
    if (fs.exec && cudaGraphLaunch(fs.exec, c.stream) == cudaSuccess) {
      note_graph_replay();
      launched = true;
    }
    cudaGetLastError();
  }
  if (!launched) {
    if (!same && fs.exec) {
      cudaGraphExecDestroy(fs.exec);
      fs.exec = nullptr;
    }
    issue_fast(c, sp, d_pos, capacity);
  }
  fs.key = key;
  fs.have_key = true;
  for (int a = 0; a < 3; ++a) c.rank_nb[a] = sp.grid.nb[a];

  if (report) {
    Status rs = wait_report(c);
    if (!rs.ok()) return rs;
    const volatile int64_t* r = c.h_report;
    const int64_t m = r[1];
    if (r[2] != 0) return fail(NLB_ERR_CUDA, "prefix scan gave up waiting for a tile");
    if (sp.grouped) fs.last_records = r[3];
    if (m <= capacity && (!sp.grouped || r[3] <= sp.search.chunk_cap)) {
      if (c.stream == c.own_stream) {
        if (!stream_ordered) {
          const cudaError_t e = cudaStreamSynchronize(c.stream);
          if (e != cudaSuccess) return cuda_fail(e, "neighbour-list pipeline");
        }
      } else {
        const cudaError_t e = cudaEventRecord(c.early_ev, c.stream);
        if (e != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
        c.early_stream = c.stream;
      }
      fs.last_m = m;
      if (!sp.grouped) fs.last_mask_words = r[3];
      *m_out = m;
      return Status{NLB_OK};
    }
    // (Too little room: the synchronous path below grows the arrays.)
  }

  // Without the report (phase profiling, or too little room): one
  // synchronisation reads the total edges and the scan's wait-error word.
  cudaError_t e = cudaMemcpyAsync(c.h_small, sp.grouped ? sp.search.total : sp.offs + sp.row,
                                  sizeof(int64_t), cudaMemcpyDeviceToHost, c.stream);
  if (e == cudaSuccess)  // the scan's (or the group search's) wait-error word
    e = cudaMemcpyAsync(c.h_small + 1, sp.scan_state + 1, sizeof(int64_t),
                        cudaMemcpyDeviceToHost, c.stream);
  c.h_small[2] = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c.h_small + 2, sp.grouped ? (const void*)sp.search.records : sp.gb.mask_top,
                        sizeof(int64_t), cudaMemcpyDeviceToHost, c.stream);
  // Grids too large for k_prep's own bin scan use a separate scan (state in
  // gb.scan_tmp): its error word too.
  c.h_small[3] = 0;
  if (const int64_t* bad = bin_scan_error(sp.grid, sp.gb); e == cudaSuccess && bad)
    e = cudaMemcpyAsync(c.h_small + 3, bad, sizeof(int64_t), cudaMemcpyDeviceToHost, c.stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
  if (e != cudaSuccess) return cuda_fail(e, "neighbour-list pipeline");
  if (c.h_small[1] != 0 || c.h_small[3] != 0)
    return fail(NLB_ERR_CUDA, "prefix scan gave up waiting for a tile");
  const int64_t m = c.h_small[0];
  if (c.prof) {
    c.prof_pending_count = true;
    c.prof_pending_emit = true;
    c.harvest();
  }
  const int64_t records = c.h_small[2];
  const bool recount = sp.grouped && records > sp.search.chunk_cap;
  if (m > capacity || recount) {
    // Too little room: grow it (outside any capture) and run what is missing
    // again.  The records: the count pass once more, its state cleared first.
    const int64_t cap2 = m > capacity ? m + m / 8 + 1024 : capacity;
    if (!out_arrays(c, sp, cap2)) return run_lean(c, sp, d_pos, m_out, stream_ordered);
    if (recount) {
      GroupSearch& o = sp.search;
      o.masks = slot<uint32_t>(c, kSlotMasks, 32 * (size_t)records);
      o.cand = slot<uint32_t>(c, kSlotCand, 32 * (size_t)records);
      o.cshift = slot<uint32_t>(c, kSlotCshift, 32 * (size_t)records);
      if (!o.masks || !o.cand || !o.cshift) return run_lean(c, sp, d_pos, m_out, stream_ordered);
      o.chunk_cap = records;
      cudaMemsetAsync(o.state, 0, sizeof(uint64_t) * (size_t)group_state_words(o.max_groups), c.stream);
    }
    if (sp.grouped)
      issue_search(c, sp, d_pos, cap2, recount);
    else
      launch_pair_emit(sp.grid, sp.gb, sp.n, sp.band, sp.offs, fast_targets(sp, cap2), c.stream);
    c.h_small[1] = 0;
    e = cudaSuccess;
    if (recount)
      e = cudaMemcpyAsync(c.h_small + 1, sp.search.state + 1, sizeof(int64_t),
                          cudaMemcpyDeviceToHost, c.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
    if (e != cudaSuccess) return cuda_fail(e, "emit pass");
    if (c.h_small[1] != 0) return fail(NLB_ERR_CUDA, "prefix scan gave up waiting for a tile");
    fs.have_key = false;  // workspace pointers changed
  }
  fs.last_m = m;
  if (sp.grouped)
    fs.last_records = records;
  else
    fs.last_mask_words = records;
  *m_out = m;
  return Status{NLB_OK};
}

Status run_brute_rows(Ctx& c, SystemPlan& sp, const double* d_pos, int64_t* m_out,
                      bool stream_ordered) {
  FastState& fs = state_for(c);
  const int64_t n = sp.n;
  int32_t tile = 0, spins = 0;
  take_scan_stall(&tile, &spins);  // (no launch here waits for another)
  int64_t capacity = std::max<int64_t>(
      {4096, (int64_t)(1.25 * (double)fs.last_m),
       (int64_t)(1.5 * (double)estimate_edges(sp, std::sqrt(sp.rc_sq[0])))});
  capacity = std::min(capacity, n * (n - 1) / 2 + 1);
  BruteRows rows;
  rows.masks = slot<uint32_t>(c, kSlotBruteMasks, 32 * (size_t)kBruteRowAtoms);
  // (offsets, counts and the completion count, which every launch leaves at
  // zero)
  const bool fresh = c.bufs[kSlotBruteRows].p == nullptr;
  rows.offs = slot<int64_t>(c, kSlotBruteRows, 2 * (size_t)kBruteRowAtoms + 2);
  rows.counts = reinterpret_cast<int32_t*>(rows.offs + kBruteRowAtoms + 1);
  rows.done = rows.counts + kBruteRowAtoms;
  // (before anything can fail: the next call finds the block there)
  if (fresh && rows.offs) cudaMemsetAsync(rows.done, 0, sizeof(int32_t), c.stream);
  if (!rows.masks || !rows.offs || !out_arrays(c, sp, capacity))
    return fail(NLB_ERR_NOMEM, "device allocation failed");
  c.h_report[0] = 0;
  c.mark(0);
  c.mark(1);
  launch_brute_masks(sp.brute, d_pos, (int32_t)n, sp.rc_sq[0], rows, c.d_report, c.stream);
  c.mark(2);
  c.mark(3);
  c.mark(4);
  launch_brute_write(sp.brute, d_pos, (int32_t)n, rows, sp.out_src, sp.out_sh, capacity, c.stream);
  c.mark(5);
  Status st = wait_report(c);
  if (!st.ok()) return st;
  const int64_t m = const_cast<volatile int64_t*>(c.h_report)[1];
  fs.have_key = false;  // (the result arrays are not the ones of the last search)
  if (m > capacity) {
    if (!out_arrays(c, sp, m))
      return fail(NLB_ERR_NOMEM, "device allocation for the edge lists failed");
    launch_brute_write(sp.brute, d_pos, (int32_t)n, rows, sp.out_src, sp.out_sh, m, c.stream);
  }
  if (c.stream == c.own_stream || c.prof) {
    if (!stream_ordered || c.prof) {
      const cudaError_t e = cudaStreamSynchronize(c.stream);
      if (e != cudaSuccess) return cuda_fail(e, "brute force");
    }
  } else {
    const cudaError_t e = cudaEventRecord(c.early_ev, c.stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
    c.early_stream = c.stream;
  }
  if (c.prof) {
    c.prof_pending_count = true;
    c.prof_pending_emit = true;
    c.harvest();
  }
  fs.last_m = m;
  *m_out = m;
  return Status{NLB_OK};
}

Status device_bounds(Ctx& c, const double* d_pos, int64_t n, double bounds6[6]) {
  const bool fresh = c.bufs[kSlotBounds].p == nullptr;
  void* tmp = c.raw(kSlotBounds, bounds_tmp_bytes());
  if (!tmp) return fail(NLB_ERR_NOMEM, "device allocation failed");
  if (fresh) cudaMemsetAsync(tmp, 0, bounds_tmp_bytes(), c.stream);
  c.h_report[0] = 0;
  launch_bounds_report(d_pos, n, tmp, c.d_report, c.stream);
  Status st = wait_report(c);
  if (!st.ok()) return st;
  for (int a = 0; a < 6; ++a) {
    const int64_t bits = const_cast<volatile int64_t*>(c.h_report)[1 + a];
    std::memcpy(&bounds6[a], &bits, sizeof(double));
  }
  return Status{NLB_OK};
}

}  // namespace nlb
