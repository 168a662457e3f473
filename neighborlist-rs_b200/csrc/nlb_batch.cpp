// nlb_batch.cpp -- batched systems (src/batch.rs:10-290).
//
// Splits the concatenated positions into systems wherever the batch id
// changes.  Consecutive systems of at most kBatchMaxAtoms atoms form a run
// that is planned, counted and emitted on the device by the batched kernels
// (k_batch.cu): four launches and one synchronisation per run, whatever the
// number of systems.  Larger systems take the single-system pipeline.  Lists
// are concatenated in system order with atom indices offset by each system's
// first atom, and each system is planned exactly like a single call (auto-box
// margin and mic_safe from the largest cutoff).
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "nlb_internal.h"

namespace nlb {

extern std::atomic<uint64_t> g_bf_threshold;

namespace {
double wall_ms() {
  return std::chrono::duration<double, std::milli>(
             std::chrono::steady_clock::now().time_since_epoch())
      .count();
}
}  // namespace

namespace {

// Grows a context buffer to `need` bytes, keeping its first `used` bytes
// (a device-to-device copy and a free of the old block, only on growth).
bool grow_keep(Ctx::Buf& b, size_t need, size_t used, cudaStream_t s) {
  if (need <= b.cap) return true;
  const size_t cap = std::max<size_t>(need + need / 2, 1 << 16);
  void* q = nullptr;
  if (cudaMalloc(&q, cap) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (b.p) {
    if (used) cudaMemcpyAsync(q, b.p, used, cudaMemcpyDeviceToDevice, s);
    cudaStreamSynchronize(s);
    cudaFree(b.p);
  }
  b.p = q;
  b.cap = cap;
  return true;
}

// The k output lists of one batched call, in the context's persistent
// buffers (allocation only when a call needs more than any before it).
struct Outputs {
  Ctx& c;
  std::vector<int64_t> total;
  Outputs(Ctx& ctx, int32_t k) : c(ctx), total(k, 0) {
    if (c.batch_out.size() < 3 * (size_t)k) c.batch_out.resize(3 * (size_t)k);
  }
  void* src(int32_t q) const { return c.batch_out[3 * q].p; }
  void* dst(int32_t q) const { return c.batch_out[3 * q + 1].p; }
  void* shf(int32_t q) const { return c.batch_out[3 * q + 2].p; }
  bool reserve(const std::vector<int64_t>& add, cudaStream_t s) {
    for (size_t q = 0; q < total.size(); ++q) {
      const size_t used = (size_t)total[q], need = (size_t)(total[q] + add[q]);
      if (!grow_keep(c.batch_out[3 * q], 8 * need, 8 * used, s) ||
          !grow_keep(c.batch_out[3 * q + 1], 8 * need, 8 * used, s) ||
          !grow_keep(c.batch_out[3 * q + 2], 12 * need, 12 * used, s))
        return false;
    }
    return true;
  }
};

CutoffSet make_pass(const std::vector<double>& rc_sq, int32_t g0, bool disjoint) {
  CutoffSet cs;
  std::memset(&cs, 0, sizeof(cs));
  const int32_t k = (int32_t)rc_sq.size();
  cs.k = std::min<int32_t>(kMaxCutoffsPerPass, k - g0);
  for (int32_t q = 0; q < cs.k; ++q) cs.rc_sq[q] = rc_sq[g0 + q];
  cs.disjoint = disjoint ? 1 : 0;
  cs.lower_sq = g0 > 0 ? rc_sq[g0 - 1] : -1.0;
  cs.max_sq = rc_sq.back();
  return cs;
}

// One run [a, b) of small systems through the batched kernels.
// With sys_off (k rows of n_systems + 1, sorted cutoff order), also writes
// the first edge of each of systems [a, b) in every list.
Status run_small(Ctx& c, const double* d_pos, const std::vector<int64_t>& starts,
                 const int64_t* d_starts, const double* d_cells, const uint8_t* d_pbcs,
                 const uint8_t* d_has, int32_t a, int32_t b, double rc_max,
                 const std::vector<double>& rc_sq, bool disjoint, bool multi, Outputs& out,
                 std::vector<int64_t>* sys_off) {
  cudaStream_t s = c.stream;
  const int32_t ns = b - a;
  const int32_t k = (int32_t)rc_sq.size();
  if (k + 3 > kSmallHost) return fail(NLB_ERR_VALUE, "too many cutoffs");
  const int64_t run_start = starts[a];
  const int64_t run_atoms = starts[b] - run_start;
  const int64_t row = run_atoms + 1;

  // Work items, largest systems first for load balance across the
  // persistent CTAs (larger systems split into chunks of atoms).
  std::vector<int64_t> sizes(ns);
  for (int32_t i = 0; i < ns; ++i) sizes[i] = starts[a + i + 1] - starts[a + i];
  // (every candidate launch shape when this kind of batch is new)
  ShapeTrials trials;
  Status st = trials.prepare(c, make_tune_key(c.device, k, sizes.data(), ns, rc_max),
                             sizes.data(), ns, kSlotBatch0 + 1);
  if (!st.ok()) return st;

  SysPlan* plans = slot<SysPlan>(c, kSlotBatch0 + 0, ns);
  int32_t* flags = slot<int32_t>(c, kSlotBatch0 + 2, 3);  // [0] plan error, [1..2] work counters
  uint32_t* counts = slot<uint32_t>(c, kSlotBatch0 + 3, (size_t)k * row);
  int64_t* offs = slot<int64_t>(c, kSlotBatch0 + 4, (size_t)k * row + 1);
  int64_t* scan_tmp = slot<int64_t>(c, kSlotBatch0 + 5, scan_tmp_elems((int64_t)k * row));
  if (!plans || !flags || !counts || !offs || !scan_tmp)
    return fail(NLB_ERR_NOMEM, "device allocation failed");

  cudaMemsetAsync(flags, 0, sizeof(int32_t) * 3, s);
  cudaMemsetAsync(counts, 0, sizeof(uint32_t) * (size_t)k * row, s);
  c.mark(0);
  launch_plan(d_pos, d_starts, a, b, d_cells, d_pbcs, d_has, rc_max, g_bf_threshold.load(),
              multi ? 1 : 0, run_start, plans, flags, s);
  c.mark(1);
  // (The counts are the same in every shape: each trial writes all of them.)
  for (size_t t = 0; t < trials.w.size(); ++t) {
    trials.mark(c, t);
    for (int32_t g0 = 0; g0 < k; g0 += kMaxCutoffsPerPass) {
      const CutoffSet cs = make_pass(rc_sq, g0, disjoint);
      cudaMemsetAsync(flags + 1, 0, sizeof(int32_t) * 2, s);
      launch_batch_count(plans, trials.w[t], d_pos, cs, counts + (size_t)g0 * row, row,
                         flags + 1, s);
    }
  }
  trials.mark(c, trials.w.size());
  c.mark(2);
  exclusive_scan_u32(counts, (int64_t)k * row, offs, scan_tmp, s);
  c.mark(3);
  // Per-system edge offsets within this run, one row of ns + 1 per cutoff.
  std::vector<int64_t> run_bounds;
  if (sys_off) {
    int64_t* d_bounds = slot<int64_t>(c, kSlotBatch0 + 11, (size_t)k * (ns + 1));
    if (!d_bounds) return fail(NLB_ERR_NOMEM, "device allocation failed");
    for (int32_t q = 0; q < k; ++q)
      launch_sys_bounds(plans, ns, offs + (size_t)q * row, row, d_bounds + (size_t)q * (ns + 1), s);
    run_bounds.resize((size_t)k * (ns + 1));
    cudaMemcpyAsync(run_bounds.data(), d_bounds, sizeof(int64_t) * run_bounds.size(),
                    cudaMemcpyDeviceToHost, s);
  }
  cudaError_t e = cudaMemcpy2DAsync(c.h_small, sizeof(int64_t), offs, sizeof(int64_t) * row,
                                    sizeof(int64_t), (size_t)k + 1, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c.h_small + k + 1, flags, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)  // the scan's bounded-wait error word
    e = cudaMemcpyAsync(c.h_small + k + 2, scan_tmp + 1, sizeof(int64_t), cudaMemcpyDeviceToHost,
                        s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "batched count pass");
  if (c.h_small[k + 2] != 0) return fail(NLB_ERR_CUDA, "prefix scan gave up waiting for a tile");
  if (c.prof) {
    c.harvest();
    c.prof_pending_count = true;
    c.harvest();
  }
  const int32_t plan_err = (int32_t)(c.h_small[k + 1] & 0xffffffff);
  if (plan_err == 1) return fail(NLB_ERR_VALUE, "Cell matrix is not invertible");
  if (plan_err == 2) return fail(NLB_ERR_VALUE, "stencil too large for this cutoff and cell");
  std::vector<int64_t> m(k);
  for (int32_t q = 0; q < k; ++q) m[q] = c.h_small[q + 1] - c.h_small[q];
  if (sys_off) {
    const size_t stride = starts.size();  // n_systems + 1
    for (int32_t q = 0; q < k; ++q)
      for (int32_t i = 0; i < ns; ++i)
        (*sys_off)[(size_t)q * stride + a + i] = out.total[q] + run_bounds[(size_t)q * (ns + 1) + i];
  }
  if (!out.reserve(m, s)) return fail(NLB_ERR_NOMEM, "device allocation for the edge lists failed");

  const BatchItems& bw = trials.pick(c);
  c.mark(4);
  for (int32_t g0 = 0; g0 < k; g0 += kMaxCutoffsPerPass) {
    const CutoffSet cs = make_pass(rc_sq, g0, disjoint);
    EmitTargets t;
    std::memset(&t, 0, sizeof(t));
    for (int32_t q = 0; q < cs.k; ++q) {
      t.src[q] = static_cast<int64_t*>(out.src(g0 + q));
      t.dst[q] = static_cast<int64_t*>(out.dst(g0 + q));
      t.sh[q] = static_cast<int32_t*>(out.shf(g0 + q));
      t.base[q] = out.total[g0 + q];
    }
    cudaMemsetAsync(flags + 1, 0, sizeof(int32_t) * 2, s);
    launch_batch_emit(plans, bw, d_pos, cs, offs + (size_t)g0 * row, row, t, flags + 1, s);
  }
  c.mark(5);
  if (c.prof) c.prof_pending_emit = true;
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "batched emit launch");
  for (int32_t q = 0; q < k; ++q) out.total[q] += m[q];
  return Status{NLB_OK};
}

// ---------------------------------------------------------------- device-sized batches
//
// A batch whose systems all take the batched kernels, of a kind whose launch
// shape is decided, runs plan -> count -> scan -> emit with no host round
// trip in between: the emit pass reads each list's total from the device and
// writes into grow-only arenas (capacity: the last batch's largest list x
// 1.25, at least 16 edges per atom), writing nothing if a list does not fit
// (the host then grows the arenas and emits again).  The second identical
// call (same sizes, shape, cutoffs, buffers and stream) captures the
// sequence as a CUDA graph and later calls replay it; the inputs are
// uploaded before the graph runs, so new positions and cells of the same
// shapes reuse it.

struct BatchGraph {
  std::vector<unsigned char> key;
  cudaGraphExec_t exec = nullptr;
  int launches = 0;
  int64_t last_m = 0;  // largest list of the last device-sized batch
};

thread_local BatchGraph tl_bgraph[16];

template <class T>
void put(std::vector<unsigned char>& k, const T& v) {
  const unsigned char* b = reinterpret_cast<const unsigned char*>(&v);
  k.insert(k.end(), b, b + sizeof(T));
}

struct FastBatchArgs {
  const double* d_pos;
  const int64_t* d_starts;
  const double* d_cells;
  const uint8_t* d_pbcs;
  const uint8_t* d_has;
  int32_t n_sys;
  int64_t row;
  double rc_max;
  bool disjoint, multi;
  SysPlan* plans;
  int32_t* flags;
  uint32_t* counts;
  int64_t* offs;
  int64_t* scan_tmp;
  int64_t* d_bounds;  // nullptr: no per-system offsets
  BatchItems bw;
  int64_t cap;
  bool use_rec;          // records_pay: count pass records hits, expansion writes the lists
  BatchRecords rec;
  int32_t* rec_flags;    // rec.seg_top / overflow / need_recompute (zeroed per batch)
};

void issue_emit_fast(Ctx& c, const FastBatchArgs& a, const std::vector<double>& rc_sq,
                     cudaStream_t s, bool recompute = false) {
  const int32_t k = (int32_t)rc_sq.size();
  if (a.use_rec && !recompute) {
    EmitTargets t;
    std::memset(&t, 0, sizeof(t));
    for (int32_t q = 0; q < k; ++q) {
      t.src[q] = static_cast<int64_t*>(c.batch_out[3 * q].p);
      t.dst[q] = static_cast<int64_t*>(c.batch_out[3 * q + 1].p);
      t.sh[q] = static_cast<int32_t*>(c.batch_out[3 * q + 2].p);
    }
    t.capacity = a.cap;
    t.scan_error = a.scan_tmp + 1;
    launch_batch_expand(a.rec, a.plans, a.d_pos, a.offs, a.row, k, t, s);
    return;
  }
  for (int32_t g0 = 0; g0 < k; g0 += kMaxCutoffsPerPass) {
    const CutoffSet cs = make_pass(rc_sq, g0, a.disjoint);
    EmitTargets t;
    std::memset(&t, 0, sizeof(t));
    for (int32_t q = 0; q < cs.k; ++q) {
      t.src[q] = static_cast<int64_t*>(c.batch_out[3 * (g0 + q)].p);
      t.dst[q] = static_cast<int64_t*>(c.batch_out[3 * (g0 + q) + 1].p);
      t.sh[q] = static_cast<int32_t*>(c.batch_out[3 * (g0 + q) + 2].p);
    }
    t.capacity = a.cap;
    t.scan_error = a.scan_tmp + 1;
    cudaMemsetAsync(a.flags + 1, 0, sizeof(int32_t) * 2, s);
    launch_batch_emit(a.plans, a.bw, a.d_pos, cs, a.offs + (size_t)g0 * a.row, a.row, t,
                      a.flags + 1, s);
  }
}

void issue_batch_fast(Ctx& c, const FastBatchArgs& a, const std::vector<double>& rc_sq) {
  cudaStream_t s = c.stream;
  const int32_t k = (int32_t)rc_sq.size();
  cudaMemsetAsync(a.flags, 0, sizeof(int32_t) * 3, s);
  cudaMemsetAsync(a.counts, 0, sizeof(uint32_t) * (size_t)k * a.row, s);
  if (a.use_rec) cudaMemsetAsync(a.rec_flags, 0, sizeof(int32_t) * 3, s);
  c.mark(0);
  launch_plan(a.d_pos, a.d_starts, 0, a.n_sys, a.d_cells, a.d_pbcs, a.d_has, a.rc_max,
              g_bf_threshold.load(), a.multi ? 1 : 0, 0, a.plans, a.flags, s);
  c.mark(1);
  for (int32_t g0 = 0; g0 < k; g0 += kMaxCutoffsPerPass) {
    const CutoffSet cs = make_pass(rc_sq, g0, a.disjoint);
    cudaMemsetAsync(a.flags + 1, 0, sizeof(int32_t) * 2, s);
    launch_batch_count(a.plans, a.bw, a.d_pos, cs, a.counts + (size_t)g0 * a.row, a.row,
                       a.flags + 1, s, a.use_rec ? &a.rec : nullptr);
  }
  c.mark(2);
  exclusive_scan_u32(a.counts, (int64_t)k * a.row, a.offs, a.scan_tmp, s);
  if (a.d_bounds)
    for (int32_t q = 0; q < k; ++q)
      launch_sys_bounds(a.plans, a.n_sys, a.offs + (size_t)q * a.row, a.row,
                        a.d_bounds + (size_t)q * (a.n_sys + 1), s);
  c.mark(3);
  c.mark(4);
  issue_emit_fast(c, a, rc_sq, s);
  c.mark(5);
}

// Grows the k arenas (src, dst, shift per list) to `cap` edges each.
bool arenas_for(Ctx& c, int32_t k, int64_t cap, cudaStream_t s) {
  if (c.batch_out.size() < 3 * (size_t)k) c.batch_out.resize(3 * (size_t)k);
  for (int32_t q = 0; q < k; ++q)
    if (!grow_keep(c.batch_out[3 * q], 8 * (size_t)cap, 0, s) ||
        !grow_keep(c.batch_out[3 * q + 1], 8 * (size_t)cap, 0, s) ||
        !grow_keep(c.batch_out[3 * q + 2], 12 * (size_t)cap, 0, s))
      return false;
  return true;
}

int64_t arena_capacity(const Ctx& c, int32_t k) {
  if (c.batch_out.size() < 3 * (size_t)k) return 0;
  int64_t cap = INT64_MAX;
  for (int32_t q = 0; q < k; ++q)
    cap = std::min<int64_t>({cap, (int64_t)(c.batch_out[3 * q].cap / 8),
                             (int64_t)(c.batch_out[3 * q + 1].cap / 8),
                             (int64_t)(c.batch_out[3 * q + 2].cap / 12)});
  return cap;
}

// Whether a batch with several lists expands records instead of testing again.
// Tests without a cell are cheap, and among few atoms cheaper than records of
// them: two lists of systems without a cell, recomputed / expanded, us a call:
// 300 of 64 atoms 319 / 329, 300 of 100 480 / 488, 64 of 128 222 / 218, 500 of
// 128 929 / 941, 64 of 200 314 / 303, 20 of 900 617 / 483, 300 of 8 to 256
// (an atom has 176 in its system) 658 / 644.  With cells records always won
// (185 of 16 atoms 230 / 212, 20 of 900 724 / 602).
constexpr int64_t kRecordMates = 112;  // atoms in an atom's system, on average
bool records_pay(int32_t k, bool any_cell, const std::vector<int64_t>& sizes) {
  if (k == 1 || any_cell) return k <= kBatchRecordLists;
  int64_t atoms = 0, mates = 0;
  for (int64_t n : sizes) {
    atoms += n;
    mates += n * n;
  }
  return k <= kBatchRecordLists && mates > kRecordMates * atoms;
}

// The device-sized path for a batch of small systems only (one run).
// *handled = false (nothing issued) when the batch's kind still has launch
// shapes to time or phases are being profiled: the caller runs the counted
// path instead.
Status run_small_fast(Ctx& c, const double* d_pos, const std::vector<int64_t>& starts,
                      const int64_t* d_starts, const double* d_cells, const uint8_t* d_pbcs,
                      const uint8_t* d_has, bool any_cell, double rc_max,
                      const std::vector<double>& rc_sq, const std::vector<int32_t>& order,
                      bool disjoint, bool multi, nlb_result* outs, int64_t* sys_offsets,
                      bool* handled) {
  *handled = false;
  cudaStream_t s = c.stream;
  const int32_t ns = (int32_t)starts.size() - 1;
  const int32_t k = (int32_t)rc_sq.size();
  if (k + 4 > kSmallHost) return fail(NLB_ERR_VALUE, "too many cutoffs");
  const int64_t run_atoms = starts[ns];
  std::vector<int64_t> sizes(ns);
  for (int32_t i = 0; i < ns; ++i) sizes[i] = starts[i + 1] - starts[i];
  ShapeTrials trials;
  Status st = trials.prepare(c, make_tune_key(c.device, k, sizes.data(), ns, rc_max),
                             sizes.data(), ns, kSlotBatch0 + 1);
  if (!st.ok()) return st;
  if (trials.timed) return Status{NLB_OK};
  *handled = true;

  FastBatchArgs a;
  std::memset(&a, 0, sizeof(a));
  a.d_pos = d_pos;
  a.d_starts = d_starts;
  a.d_cells = d_cells;
  a.d_pbcs = d_pbcs;
  a.d_has = d_has;
  a.n_sys = ns;
  a.row = run_atoms + 1;
  a.rc_max = rc_max;
  a.disjoint = disjoint;
  a.multi = multi;
  a.plans = slot<SysPlan>(c, kSlotBatch0 + 0, ns);
  a.flags = slot<int32_t>(c, kSlotBatch0 + 2, 3);
  a.counts = slot<uint32_t>(c, kSlotBatch0 + 3, (size_t)k * a.row);
  a.offs = slot<int64_t>(c, kSlotBatch0 + 4, (size_t)k * a.row + 1);
  a.scan_tmp = slot<int64_t>(c, kSlotBatch0 + 5, scan_tmp_elems((int64_t)k * a.row));
  if (sys_offsets) a.d_bounds = slot<int64_t>(c, kSlotBatch0 + 11, (size_t)k * (ns + 1));
  if (!a.plans || !a.flags || !a.counts || !a.offs || !a.scan_tmp ||
      (sys_offsets && !a.d_bounds))
    return fail(NLB_ERR_NOMEM, "device allocation failed");
  a.bw = trials.w[0];

  BatchGraph& bg = tl_bgraph[c.device & 15];
  int64_t cap = std::max<int64_t>({4096, bg.last_m + bg.last_m / 4, 16 * run_atoms});
  const int64_t have = arena_capacity(c, k);
  if (have > cap) cap = have;
  if (!arenas_for(c, k, cap, s)) return fail(NLB_ERR_NOMEM, "device allocation for the edge lists failed");
  // The arenas' actual capacity (so that repeated calls see the same value
  // once the arenas stop growing).
  a.cap = arena_capacity(c, k);
  // Hit records: at most one segment per atom plus one per 32 records, and a
  // record holds at least one of a list's <= cap edges.  Without the memory
  // for them the emit pass recomputes.
  const int64_t segs = run_atoms + k * (cap / 32 + 1) + 1024;
  a.use_rec = records_pay(k, any_cell, sizes) && segs <= INT32_MAX / 2;
  if (a.use_rec) {
    a.rec.seg_cap = (int)segs;
    a.rec.seg_hdr = slot<int4>(c, kSlotBatch0 + 13, (size_t)segs * (k > 1 ? 2 : 1));
    a.rec.rec = slot<uint32_t>(c, kSlotBatch0 + 14, (size_t)segs * 96);
    a.rec.meta = slot<SlotMeta>(c, kSlotBatch0 + 15, (size_t)run_atoms);
    a.rec_flags = slot<int32_t>(c, kSlotBatch0 + 12, 3);
    a.rec.seg_top = a.rec_flags;
    a.rec.overflow = a.rec_flags + 1;
    a.rec.need_recompute = a.rec_flags + 2;
    a.use_rec = a.rec.seg_hdr && a.rec.rec && a.rec.meta && a.rec_flags;
    if (!a.use_rec) std::memset(&a.rec, 0, sizeof(a.rec));
  }

  // Everything the issued work depends on.
  std::vector<unsigned char> key;
  key.reserve(512 + 8 * (size_t)k);
  put(key, a);
  put(key, s);
  put(key, g_bf_threshold.load());
  for (int32_t q = 0; q < k; ++q) {
    put(key, rc_sq[q]);
    put(key, c.batch_out[3 * q].p);
    put(key, c.batch_out[3 * q + 1].p);
    put(key, c.batch_out[3 * q + 2].p);
  }
  // (Phase profiling times directly launched kernels: no graph then.)
  const bool same = !scan_stall_armed() && !c.prof && key == bg.key;
  bool launched = false;
  if (same && bg.exec) {
    if (cudaGraphLaunch(bg.exec, s) == cudaSuccess) {
      note_launches(bg.launches);
      note_graph_replay();
      launched = true;
    } else {
      cudaGetLastError();
    }
  } else if (same && s != nullptr) {
    // Second identical call: capture once, replay from now on.
    if (bg.exec) {
      cudaGraphExecDestroy(bg.exec);
      bg.exec = nullptr;
    }
    cudaGraph_t graph = nullptr;
    const int64_t l0 = nlb_kernel_launches();
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      issue_batch_fast(c, a, rc_sq);
      if (cudaStreamEndCapture(s, &graph) == cudaSuccess && graph) {
        if (cudaGraphInstantiate(&bg.exec, graph, 0) != cudaSuccess) bg.exec = nullptr;
        cudaGraphDestroy(graph);
      }
    }
    cudaGetLastError();
    bg.launches = (int)(nlb_kernel_launches() - l0);
    if (bg.exec && cudaGraphLaunch(bg.exec, s) == cudaSuccess) {
      note_graph_replay();
      launched = true;
    }
    cudaGetLastError();
  }
  if (!launched) {
    if (!same && bg.exec) {
      cudaGraphExecDestroy(bg.exec);
      bg.exec = nullptr;
    }
    issue_batch_fast(c, a, rc_sq);
  }
  bg.key.swap(key);

  const double t_issue = wall_ms();
  // One synchronisation: list totals, plan errors, the scan's error word,
  // per-system offsets.
  cudaError_t e = cudaMemcpy2DAsync(c.h_small, sizeof(int64_t), a.offs, sizeof(int64_t) * a.row,
                                    sizeof(int64_t), (size_t)k + 1, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c.h_small + k + 1, a.flags, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c.h_small + k + 2, a.scan_tmp + 1, sizeof(int64_t),
                        cudaMemcpyDeviceToHost, s);
  c.h_small[k + 3] = 0;
  if (e == cudaSuccess && a.use_rec)  // the expansion found incomplete records
    e = cudaMemcpyAsync(c.h_small + k + 3, a.rec.need_recompute, sizeof(int32_t),
                        cudaMemcpyDeviceToHost, s);
  std::vector<int64_t> bounds;
  if (e == cudaSuccess && sys_offsets) {
    bounds.resize((size_t)k * (ns + 1));
    e = cudaMemcpyAsync(bounds.data(), a.d_bounds, sizeof(int64_t) * bounds.size(),
                        cudaMemcpyDeviceToHost, s);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "batched build");
  const double t_synced = wall_ms();
  if (c.prof) {
    c.prof_pending_count = true;
    c.prof_pending_emit = true;
    c.harvest();
    c.prof_host_ms[1] += t_synced - t_issue;
  }
  if (c.h_small[k + 2] != 0) return fail(NLB_ERR_CUDA, "prefix scan gave up waiting for a tile");
  const int32_t plan_err = (int32_t)(c.h_small[k + 1] & 0xffffffff);
  if (plan_err == 1) return fail(NLB_ERR_VALUE, "Cell matrix is not invertible");
  if (plan_err == 2) return fail(NLB_ERR_VALUE, "stencil too large for this cutoff and cell");
  std::vector<int64_t> m(k);
  int64_t m_max = 0;
  for (int32_t q = 0; q < k; ++q) {
    m[q] = c.h_small[q + 1] - c.h_small[q];
    m_max = std::max(m_max, m[q]);
  }
  if (m_max > cap) {
    // An arena was too small (nothing was written): grow and emit again
    // (recomputing: the records were sized for the smaller arena).
    a.cap = m_max + m_max / 8 + 1024;
    if (!arenas_for(c, k, a.cap, s))
      return fail(NLB_ERR_NOMEM, "device allocation for the edge lists failed");
    issue_emit_fast(c, a, rc_sq, s, true);
    bg.key.clear();  // arena pointers changed
  } else if ((c.h_small[k + 3] & 0xffffffff) != 0) {
    // The records were incomplete (a segment or an image shift did not fit):
    // the expansion wrote nothing; recompute the list.
    issue_emit_fast(c, a, rc_sq, s, true);
  }
  bg.last_m = m_max;

  // Exact-sized pinned results, in input cutoff order.
  for (int32_t q = 0; q < k; ++q) {
    nlb_result& r = outs[order[q]];
    st = alloc_result(m[q], &r);
    if (!st.ok()) return st;
    if (m[q] == 0) continue;
    cudaMemcpyAsync(r.edge_index, c.batch_out[3 * q].p, 8 * m[q], cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(r.edge_index + m[q], c.batch_out[3 * q + 1].p, 8 * m[q],
                    cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(r.shift, c.batch_out[3 * q + 2].p, 12 * m[q], cudaMemcpyDeviceToHost, s);
  }
  if (sys_offsets) {
    const size_t stride = (size_t)ns + 1;
    for (int32_t q = 0; q < k; ++q) {
      int64_t* row = sys_offsets + (size_t)order[q] * stride;
      std::memcpy(row, bounds.data() + (size_t)q * stride, sizeof(int64_t) * stride);
      row[ns] = m[q];
    }
  }
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    for (int32_t q = 0; q < k; ++q) nlb_result_free(&outs[order[q]]);
    return cuda_fail(e, "batched emit");
  }
  if (c.prof) c.prof_host_ms[2] += wall_ms() - t_synced;
  return Status{NLB_OK};
}

}  // namespace

void release_batch_graphs() {
  for (BatchGraph& bg : tl_bgraph) {
    if (bg.exec) cudaGraphExecDestroy(bg.exec);
    bg = BatchGraph();
  }
}

// First atom of every system (a new system wherever the id changes) and n
// at the end; false when an id decreases.  Four ids per step with SSE2:
// most steps hold no change.
bool batch_starts(const int32_t* batch, int64_t n, std::vector<int64_t>& starts) {
  starts.clear();
  starts.push_back(0);
  int64_t i = 1;
#if defined(__SSE2__)
  for (; i + 4 <= n; i += 4) {
    const __m128i cur = _mm_loadu_si128(reinterpret_cast<const __m128i*>(batch + i));
    const __m128i prv = _mm_loadu_si128(reinterpret_cast<const __m128i*>(batch + i - 1));
    const int changed = _mm_movemask_ps(_mm_castsi128_ps(_mm_cmpeq_epi32(cur, prv))) ^ 0xF;
    if (!changed) continue;
    if (_mm_movemask_ps(_mm_castsi128_ps(_mm_cmpgt_epi32(prv, cur))) != 0) return false;
    for (int k = 0; k < 4; ++k)
      if ((changed >> k) & 1) starts.push_back(i + k);
  }
#endif
  for (; i < n; ++i) {
    if (batch[i] == batch[i - 1]) continue;
    if (batch[i] < batch[i - 1]) return false;
    starts.push_back(i);
  }
  starts.push_back(n);
  return true;
}

Status run_batch(const double* pos, int64_t n, const int32_t* batch, int64_t n_batch,
                 const double* cutoffs, int32_t k, const double* cells, const uint8_t* pbcs,
                 const uint8_t* has_cell, int64_t n_cells, bool disjoint, bool multi,
                 nlb_result* outs, int64_t* sys_offsets) {
  zero_results(outs, k);
  if (n_batch != n) return fail(NLB_ERR_VALUE, "positions and batch must have the same length");
  if (k <= 0) return Status{NLB_OK};
  if (!cutoffs_valid(cutoffs, k))
    return fail(NLB_ERR_VALUE, multi ? "All cutoffs must be positive and finite"
                                     : "Cutoff must be positive and finite");
  if (n == 0) {
    if (sys_offsets) std::memset(sys_offsets, 0, sizeof(int64_t) * (size_t)k);  // no systems
    return empty_results(outs, k);
  }
  if (!pos || !batch) return fail(NLB_ERR_VALUE, "positions or batch is NULL");

  std::vector<int64_t> starts;
  if (!batch_starts(batch, n, starts))
    return fail(NLB_ERR_VALUE, "Batch IDs must be monotonic (non-decreasing)");
  const int32_t n_sys = (int32_t)starts.size() - 1;
  const int64_t have = cells ? n_cells : (int64_t)n_sys;
  if (have < (int64_t)n_sys)
    return fail(NLB_ERR_VALUE, "Expected at least " + std::to_string(n_sys) +
                                   " cells, but got " + std::to_string(have));

  std::vector<double> cs(cutoffs, cutoffs + k);
  double rc_max = NAN;
  for (double r : cs) rc_max = fmax_nan_ignoring(rc_max, r);
  const std::vector<int32_t> order = cutoff_order(cutoffs, k);
  std::vector<double> rc_sq(k);
  for (int32_t q = 0; q < k; ++q) rc_sq[q] = cutoffs[order[q]] * cutoffs[order[q]];

  Ctx* c = nullptr;
  Status st = get_ctx(&c);
  if (!st.ok()) return st;
  const double t_call = wall_ms();
  cudaStream_t s = c->stream;
  double* d_pos = nullptr;
  st = upload_positions(*c, pos, n, &d_pos);
  if (!st.ok()) return st;
  int64_t* d_starts = slot<int64_t>(*c, kSlotBatch0 + 6, starts.size());
  double* d_cells = nullptr;
  uint8_t* d_pbcs = nullptr;
  uint8_t* d_has = nullptr;
  if (!d_starts) return fail(NLB_ERR_NOMEM, "device allocation failed");
  cudaMemcpyAsync(d_starts, starts.data(), sizeof(int64_t) * starts.size(),
                  cudaMemcpyHostToDevice, s);
  if (cells && n_sys > 0) {
    d_cells = slot<double>(*c, kSlotBatch0 + 7, 9 * (size_t)n_sys);
    d_pbcs = slot<uint8_t>(*c, kSlotBatch0 + 8, 3 * (size_t)n_sys);
    d_has = slot<uint8_t>(*c, kSlotBatch0 + 9, (size_t)n_sys);
    if (!d_cells || !d_pbcs || !d_has) return fail(NLB_ERR_NOMEM, "device allocation failed");
    cudaMemcpyAsync(d_cells, cells, sizeof(double) * 9 * n_sys, cudaMemcpyHostToDevice, s);
    if (pbcs)
      cudaMemcpyAsync(d_pbcs, pbcs, 3 * (size_t)n_sys, cudaMemcpyHostToDevice, s);
    else
      cudaMemsetAsync(d_pbcs, 1, 3 * (size_t)n_sys, s);
    if (has_cell)
      cudaMemcpyAsync(d_has, has_cell, (size_t)n_sys, cudaMemcpyHostToDevice, s);
    else
      cudaMemsetAsync(d_has, 1, (size_t)n_sys, s);
  }

  bool all_small = true;
  for (int32_t i = 0; i < n_sys && all_small; ++i)
    all_small = starts[i + 1] - starts[i] <= kBatchMaxAtoms;
  if (all_small) {
    const double t_up = wall_ms();
    bool handled = false;
    const bool any_cell =
        cells && (!has_cell || std::any_of(has_cell, has_cell + n_sys, [](uint8_t h) { return h; }));
    st = run_small_fast(*c, d_pos, starts, d_starts, d_cells, d_pbcs, d_has, any_cell, rc_max, rc_sq,
                        order, disjoint, multi, outs, sys_offsets, &handled);
    if (c->prof && handled) {
      c->prof_host_ms[0] += t_up - t_call;
      c->prof_host_ms[3] += wall_ms() - t_call;
    }
    if (!st.ok() || handled) return st;
  }

  Outputs out(*c, k);
  // Per-system offsets in sorted cutoff order while the runs go by.
  std::vector<int64_t> sys_off;
  if (sys_offsets) sys_off.assign((size_t)k * starts.size(), 0);
  int32_t i = 0;
  while (i < n_sys) {
    const int64_t ni = starts[i + 1] - starts[i];
    if (ni <= kBatchMaxAtoms) {
      int32_t j = i;
      while (j < n_sys && starts[j + 1] - starts[j] <= kBatchMaxAtoms) ++j;
      st = run_small(*c, d_pos, starts, d_starts, d_cells, d_pbcs, d_has, i, j, rc_max, rc_sq,
                     disjoint, multi, out, sys_offsets ? &sys_off : nullptr);
      if (!st.ok()) return st;
      i = j;
      continue;
    }
    // A large system: the single-system pipeline.
    const double* h9 = nullptr;
    bool pb[3] = {false, false, false};
    if (cells && (!has_cell || has_cell[i])) {
      h9 = cells + 9 * (size_t)i;
      for (int a = 0; a < 3; ++a) pb[a] = pbcs ? pbcs[3 * (size_t)i + a] != 0 : true;
    }
    SystemPlan sp;
    st = plan_system(pos + 3 * starts[i], ni, h9, pb, cs, disjoint, multi, sp);
    if (!st.ok()) return st;
    st = count_system(*c, sp, d_pos + 3 * starts[i]);
    if (!st.ok()) return st;
    if (!out.reserve(sp.m, s)) return fail(NLB_ERR_NOMEM, "device allocation for the edge lists failed");
    DevLists L;
    L.src.resize(k);
    L.dst.resize(k);
    L.sh.resize(k);
    for (int32_t q = 0; q < k; ++q) {
      L.src[q] = static_cast<int64_t*>(out.src(q));
      L.dst[q] = static_cast<int64_t*>(out.dst(q));
      L.sh[q] = static_cast<int32_t*>(out.shf(q));
    }
    st = emit_system(*c, sp, d_pos + 3 * starts[i], L, out.total.data(), starts[i]);
    if (!st.ok()) return st;
    for (int32_t q = 0; q < k; ++q) {
      if (sys_offsets) sys_off[(size_t)q * starts.size() + i] = out.total[q];
      out.total[q] += sp.m[q];
    }
    ++i;
  }

  for (int32_t q = 0; q < k; ++q) {
    nlb_result& r = outs[order[q]];
    st = alloc_result(out.total[q], &r);
    if (!st.ok()) return st;
    const int64_t m = out.total[q];
    if (m == 0) continue;
    cudaMemcpyAsync(r.edge_index, out.src(q), 8 * m, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(r.edge_index + m, out.dst(q), 8 * m, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(r.shift, out.shf(q), 12 * m, cudaMemcpyDeviceToHost, s);
  }
  if (sys_offsets) {
    const size_t stride = starts.size();
    for (int32_t q = 0; q < k; ++q) {
      sys_off[(size_t)q * stride + n_sys] = out.total[q];
      std::memcpy(sys_offsets + (size_t)order[q] * stride, sys_off.data() + (size_t)q * stride,
                  sizeof(int64_t) * stride);
    }
  }
  cudaError_t e = cudaStreamSynchronize(s);
  if (c->prof) c->harvest();
  if (e != cudaSuccess) {
    for (int32_t q = 0; q < k; ++q) nlb_result_free(&outs[q]);
    return cuda_fail(e, "batched emit");
  }
  return Status{NLB_OK};
}

}  // namespace nlb
