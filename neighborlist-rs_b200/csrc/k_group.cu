// k_group.cu -- single-cutoff cell-list search in two launches: a count pass
// that keeps every pair test's outcome as bit masks, and an emit pass that
// writes the list from them.
//
// A group is a run of at most 32 atoms of one bin (canonical order: bins in
// rank order, runs in slot order); the row of its candidates -- its stencil
// cells' atoms, cell after cell -- is split into segments (slices of the row,
// or runs of cells when there are more than 32).  A segment is one warp's work
// in both passes; warps share nothing, so the slowest segment holds up nobody.
//
// k_group_count, per segment:
//   1. one lane per stencil cell describes it (candidates, image shift, FP32
//      translation into the group's bin frame);
//   2. the cells' candidates, end to end, stream through the warp 32 at a
//      time: moved into the group's frame, dropped when farther from the group's FP32 box than
//      the guard band allows (then no atom of the group can reach them), and
//      appended to a ring across cells, so that the test below runs on 32
//      live candidates whatever the bins' occupancy;
//   3. 32 candidates (lane = candidate) against the group's atoms, four atoms
//      at a time on the packed FP32 units: t = dx^2 - rc^2 + dy^2 + dz^2, the
//      half-list predicate, one ballot per atom.  A pair with |t| within the
//      guard band (make_guard_band) is decided by the reference's FP64
//      expressions, prune test included (src/search.rs:500-505, 540-553);
//   4. the hit masks of a chunk with any hit are stored with its candidates'
//      slots (one record of 32 mask words -- one per atom -- and 32 slots, and
//      32 packed image shifts when the chunk has any).
// The warp that completes a group's last segment turns the segments' counts
// per atom into offsets within the group, stores the group's total and adds
// it to the total of its block of 64 groups; the last CTA scans the blocks'
// totals (bounded waits for each block's groups), which gives M.  No warp
// waits for another one's group: a look-back over the groups in this kernel
// cost half of its time (each warp waited for every group before its own).
//
// k_group_emit, per segment: the group's first output slot is its block's
// plus the totals of the block's earlier groups; the records' masks are
// expanded into a shared stage in output order (atom by atom) and written
// with consecutive threads on consecutive slots; M is known, so the
// destinations go straight behind the sources.
//
// Measured (B200, ncu, warm): 250,000 atoms at rc 6 (11,300 groups, 11 M
// edges): count 123 us, 65 % of issue slots, 7,500 instructions per group of
// which 4,400 the pair tests; emit 112 us against 55 us for writing the same
// bytes from registers.  A million atoms: 2,110 -> 874 us per call, against
// one launch that counted, waited for its offsets and moved the destinations
// (761 with the later changes to loads, segments, stage and recheck: count 346,
// emit 319; the output alone takes 173 us to fill).  The emit is bound by latency
// and issue (49 % of slots, 20 warps an SM by shared memory: 352 us; with the
// candidates packed to four bytes 25 warps and 319) rather than by its stores:
// shifts written as whole sectors, three words a lane exchanged by shuffles
// (36 -> 12 sector writes per 32 edges), cost 372 us, and masks kept in
// registers for more warps 375.
//
// Candidates on the lanes rather than atoms: bins hold 20-25 atoms at the
// usual densities, so a third of atom lanes would idle, while the ring keeps
// candidate lanes full.
//
// Atoms whose home stencil differs from their stored bin ("irregular",
// within rounding of a bin face) are counted and written by one warp each in
// FP64 over their own stencil, exactly like the pair-task kernels.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "k_traverse.cuh"

namespace nlb {

namespace {

// One warp per CTA: segments differ in size, and a CTA's slot is free as soon
// as its segment is done (a million atoms, rc 6: 928 us with four warps per
// CTA, 903 with two, 874 with one).
constexpr int kGThreads = 32;
constexpr int kGRing = 64;     // candidates waiting per warp
constexpr int kGWindow = 16;   // records expanded per emit window

// A block's word: the sum of its groups' totals, and above it their number.
constexpr int kGCountShift = 48;
constexpr uint64_t kGSumMask = (1ull << kGCountShift) - 1;

__device__ __forceinline__ uint64_t g_load(const uint64_t* p) {
  return *reinterpret_cast<const volatile uint64_t*>(p);
}

// Candidates waiting for their test, one ring per warp.
struct GRing {
  float4 at[kGRing];  // position in the group's frame; .w: original index, + 1 in an image
                      // cell (bits): the half-list test is io < .w
  int2 id[kGRing];    // sorted slot, image shift
};

__device__ __forceinline__ int32_t unpack_shift(uint32_t w, int a) {
  return (int32_t)(w << (22 - 10 * a)) >> 22;
}

// Euclidean division with the common in-range cases first.
__device__ __forceinline__ void g_div_mod(int32_t v, int32_t m, int32_t& rem, int32_t& quot) {
  if (v >= 0 && v < m) {
    rem = v;
    quot = 0;
  } else if (v < 0 && v >= -m) {
    rem = v + m;
    quot = -1;
  } else if (v >= m && v < 2 * m) {
    rem = v - m;
    quot = 1;
  } else {
    div_mod(v, m, rem, quot);
  }
}

// Offset of stencil cell c from the home bin, in bins per axis (x outer).
__device__ __forceinline__ int3 cell_offset(const GridParams& g, int32_t n_cells, int32_t c) {
  int32_t ix, iy, iz;
  if (n_cells == 27 && g.ns[1] == 1 && g.ns[2] == 1) {  // (one bin each way: the usual grid)
    ix = c / 9;
    iy = c / 3 - 3 * ix;
    iz = c - 3 * (c / 3);
  } else {
    const int32_t ny = 2 * g.ns[1] + 1, nz = 2 * g.ns[2] + 1;
    ix = c / (ny * nz);
    const int32_t rem = c - ix * (ny * nz);
    iy = rem / nz;
    iz = rem - iy * nz;
  }
  return make_int3(ix - g.ns[0], iy - g.ns[1], iz - g.ns[2]);
}

// Cell c of the stencil centred on bin (hx, hy, hz): its bin, image shift
// (three signed 10-bit fields; at most 1024 cells, so |shift| <= 511) and
// candidate slots.
__device__ __forceinline__ int2 g_describe(const GridParams& g, const GridBuffers& b, int32_t hx,
                                           int32_t hy, int32_t hz, int32_t n_cells, int32_t c,
                                           int32_t bin[3], uint32_t& shift) {
  const int3 d = cell_offset(g, n_cells, c);
  int32_t sh[3];
  g_div_mod(hx + d.x, g.nb[0], bin[0], sh[0]);
  g_div_mod(hy + d.y, g.nb[1], bin[1], sh[1]);
  g_div_mod(hz + d.z, g.nb[2], bin[2], sh[2]);
  shift = ((uint32_t)sh[0] & 1023u) | ((uint32_t)sh[1] & 1023u) << 10 |
          ((uint32_t)sh[2] & 1023u) << 20;
  const int32_t r = b.rank_of_bin[bin[0] + g.nb[0] * (bin[1] + g.nb[1] * bin[2])];
  return make_int2((int32_t)b.bin_start[r], (int32_t)b.bin_start[r + 1]);
}

// The cell's FP64 image offset and prune target (bin centre + offset), in
// the reference's order (src/search.rs:493-505).
__device__ __forceinline__ void g_place_cell(const GridParams& g, const int32_t bin[3],
                                             uint32_t sh, double off[3], double cs[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    off[k] = dadd(dadd(dmul(g.h[3 * k], (double)unpack_shift(sh, 0)),
                       dmul(g.h[3 * k + 1], (double)unpack_shift(sh, 1))),
                  dmul(g.h[3 * k + 2], (double)unpack_shift(sh, 2)));
    double v = dadd(g.origin[k], dmul(g.basis[0][k], (double)bin[0]));
    v = dadd(v, dmul(g.basis[1][k], (double)bin[1]));
    v = dadd(v, dmul(g.basis[2][k], (double)bin[2]));
    cs[k] = dadd(v, off[k]);
  }
}

// Writes edge e (atoms i, j, shift s): sources and destinations in ei, shifts
// in sh.  EX: the output options too -- the directed list's reverse edge (j,
// i, -s) at M + e, the displacement d = (r_j - r_i) + H s (-d for the reverse)
// and its length -- with the expressions of k_extras.cu.  d_ei: entries
// between the sources and the destinations.
template <bool EX>
__device__ __forceinline__ void write_edge(const GroupOut& o, int64_t d_ei, int64_t M, int64_t e,
                                           int32_t i, int32_t j, int32_t s0, int32_t s1,
                                           int32_t s2) {
  o.ei[e] = (int64_t)i;
  o.ei[d_ei + e] = (int64_t)j;
  int32_t* sp = o.sh + 3 * e;
  sp[0] = s0;
  sp[1] = s1;
  sp[2] = s2;
  if (!EX) return;
  if (o.directed) {
    o.ei[M + e] = (int64_t)j;
    o.ei[d_ei + M + e] = (int64_t)i;
    sp += 3 * M;
    sp[0] = -s0;
    sp[1] = -s1;
    sp[2] = -s2;
  }
  if (!o.vec && !o.dist) return;
  double d[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d[k] = dsub(__ldg(&o.pos[3 * (int64_t)j + k]), __ldg(&o.pos[3 * (int64_t)i + k]));
    if (o.cell.has_cell)
      d[k] = dadd(d[k], dadd(dadd(dmul(o.cell.h[3 * k], (double)s0),
                                  dmul(o.cell.h[3 * k + 1], (double)s1)),
                             dmul(o.cell.h[3 * k + 2], (double)s2)));
  }
  if (o.vec) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      o.vec[3 * e + k] = d[k];
      if (o.directed) o.vec[3 * (M + e) + k] = -d[k];
    }
  }
  if (o.dist) {
    const double r = __dsqrt_rn(norm2(d[0], d[1], d[2]));
    o.dist[e] = r;
    if (o.directed) o.dist[M + e] = r;
  }
}

// Irregular atom p (its home stencil is not its stored bin): one warp walks
// its own stencil in FP64 exactly like pair_irregular in k_search2.cu.
// Returns its edge count; EMIT: its edges go to slots [e0, ...) in canonical
// order.
template <bool EMIT, bool EX>
__device__ uint32_t g_irregular(const GridParams& g, const GridBuffers& b, int32_t n_cells,
                                double rc_sq, int32_t p, int64_t e0, const GroupOut* out,
                                int64_t d_ei, int64_t M) {
  const int lane = threadIdx.x & 31;
  const double xi = b.px[p], yi = b.py[p], zi = b.pz[p];
  const SlotMeta mi = b.meta[p];
  double fi[3];
  matvec(g.hinv, xi, yi, zi, fi);
  int32_t home[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int32_t v = sat_i32(dmul(fi[a], (double)g.nb[a]));
    home[a] = v < g.nb[a] - 1 ? v : g.nb[a] - 1;
  }
  uint32_t count = 0;
  for (int32_t c = 0; c < n_cells; ++c) {
    int32_t bin[3];
    uint32_t csh;
    const int2 range = g_describe(g, b, home[0], home[1], home[2], n_cells, c, bin, csh);
    double off[3], cs[3];
    g_place_cell(g, bin, csh, off, cs);
    if (norm2(dsub(cs[0], xi), dsub(cs[1], yi), dsub(cs[2], zi)) > g.prune_sq) continue;
    for (int32_t jb = range.x; jb < range.y; jb += 32) {
      const int32_t j = jb + lane;
      bool hit = false;
      SlotMeta mj{};
      if (j < range.y) {
        const double ex = dadd(dsub(b.px[j], xi), off[0]);
        const double ey = dadd(dsub(b.py[j], yi), off[1]);
        const double ez = dadd(dsub(b.pz[j], zi), off[2]);
        mj = b.meta[j];
        hit = norm2(ex, ey, ez) < rc_sq && (mi.orig < mj.orig || (mi.orig == mj.orig && csh != 0));
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (EMIT && hit) {
        const int64_t e = e0 + count + __popc(m & lanemask_lt());
        write_edge<EX>(*out, d_ei, M, e, mi.orig, mj.orig, (mj.sx - mi.sx) + unpack_shift(csh, 0),
                       (mj.sy - mi.sy) + unpack_shift(csh, 1),
                       (mj.sz - mi.sz) + unpack_shift(csh, 2));
      }
      count += __popc(m);
    }
  }
  return count;
}

// The reference's FP64 test of candidate slot j, image shift sh, for the atom
// at slot q: distance and prune (src/search.rs:500-505, 540-553).
__device__ __forceinline__ bool exact_hit(const GridParams& g, const GridBuffers& b, double rc_sq,
                                          int32_t q, int32_t j, uint32_t sh) {
  const int32_t lin = b.sbin[j];
  const int32_t bin[3] = {lin % g.nb[0], lin / g.nb[0] % g.nb[1], lin / (g.nb[0] * g.nb[1])};
  double off[3], cs[3];
  g_place_cell(g, bin, sh, off, cs);
  const double xi = b.px[q], yi = b.py[q], zi = b.pz[q];
  const double ex = dadd(dsub(b.px[j], xi), off[0]);
  const double ey = dadd(dsub(b.py[j], yi), off[1]);
  const double ez = dadd(dsub(b.pz[j], zi), off[2]);
  return norm2(ex, ey, ez) < rc_sq &&
         !(norm2(dsub(cs[0], xi), dsub(cs[1], yi), dsub(cs[2], zi)) > g.prune_sq);
}

// Warp minimum (redux.sync of one FP32 value; NaN operands ignored).
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// Adds v to *p with release and acquire ordering at device scope (lighter
// than the full fences of __threadfence around a relaxed atomic).
__device__ __forceinline__ int32_t add_acq_rel(int32_t* p, int32_t v) {
  int32_t r;
  asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], %2;"
               : "=r"(r)
               : "l"(p), "r"(v)
               : "memory");
  return r;
}

// Shared memory of one warp of the count pass.
struct GCountWarp {
  float4 xy[16];  // atom pairs, negated: {-x, -x', -y, -y'}
  float4 zi[16];  // {-z, -z', original indices}
  uint4 mask[8];  // a chunk's hit masks, one word per atom
  GRing ring;
  float4 cell[32];   // the cells with candidates: translation, first slot minus place in the row
  uint32_t shift[32];
};
static_assert(sizeof(GCountWarp) % 16 == 0, "vector accesses");

// Takes room for the records of `candidates` candidates (at most one per 32)
// from a region.
// Lane 0 gets the first record, or -1 without room; the others 0 (so that
// nothing waits for the atomic before the first record is stored).
__device__ __forceinline__ int64_t take_records(const GroupSearch& o, int region,
                                                int64_t candidates) {
  const int64_t room = (candidates + 31) >> 5;
  if (threadIdx.x != 0) return 0;
  const int64_t cap = o.chunk_cap / kGroupRegions;
  const int64_t at =
      room > 0 ? (int64_t)atomicAdd(&o.chunk_top[16 * region], (unsigned long long)room) : 0;
  return at + room <= cap ? region * cap + at : -1;
}

// Candidates of the cells [c0, c0 + nc) of a group (segments of more than 32
// cells).
__device__ __noinline__ int64_t row_candidates(const GridParams& g, const GridBuffers& b,
                                               const GroupRec& grp, int32_t n_cells, int32_t c0,
                                               int32_t nc) {
  const int lane = threadIdx.x & 31;
  int64_t sum = 0;
  for (int32_t c = lane; c < nc; c += 32) {
    int32_t bin[3];
    uint32_t sh;
    const int2 r = g_describe(g, b, grp.bx, grp.by, grp.bz, n_cells, c0 + c, bin, sh);
    sum += r.y - r.x;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
  return sum;
}

// The offsets of group t, once all its segments are counted: each segment's
// counts become each atom's hits in the segments before it, atom_base the
// atoms' first slots within the group; the group's total goes to its block.
__device__ __forceinline__ void finish_group(const GridParams& g, const GridBuffers& b,
                                             int32_t n_cells, const GroupBand& band,
                                             const GroupSearch& o, int32_t t,
                                             const GroupRec& grp, unsigned irr_mask,
                                             uint32_t own) {
  const int lane = threadIdx.x & 31;
  uint32_t run = own;
  if (o.split > 1) {
    run = 0;
    uint32_t* row = o.seg_cnt + (int64_t)t * o.split * 32 + lane;
    for (int s0 = 0; s0 < o.split; s0 += 16) {  // (16 loads in flight)
      uint32_t v[16];
#pragma unroll
      for (int s = 0; s < 16; ++s) v[s] = s0 + s < o.split ? __ldcg(&row[32 * (s0 + s)]) : 0u;
#pragma unroll
      for (int s = 0; s < 16; ++s) {
        if (s0 + s < o.split) row[32 * (s0 + s)] = run;
        run += v[s];
      }
    }
  }
  for (unsigned m = irr_mask; m; m &= m - 1) {
    const int l = __ffs(m) - 1;
    const uint32_t v = g_irregular<false, false>(g, b, n_cells, band.rc_sq, grp.first + l, 0,
                                                 nullptr, 0, 0);
    if (lane == l) run = v;
  }
  int64_t x = run;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, s);
    if (lane >= s) x += y;
  }
  o.atom_base[(int64_t)t * 32 + lane] = x - (int64_t)run;
  if (lane == 31) {
    o.group_total[t] = x;
    if (t != o.withhold)  // false only under the test hook
      atomicAdd(reinterpret_cast<unsigned long long*>(&o.block_sum[t / kGroupBlock]),
                (unsigned long long)x + (1ull << kGCountShift));
  }
}

// The last CTA: exclusive scan of the blocks' sums into block_base, M, and
// the report to the host.  Every group's CTA has ended, so a block whose
// groups are not all there (the test hook) is waited for in vain: the wait is
// bounded, and the error word set.
__device__ void finish_list(const GridBuffers& b, const GroupSearch& o, int32_t n_groups) {
  const int lane = threadIdx.x;
  const int32_t n_blocks = (n_groups + kGroupBlock - 1) / kGroupBlock;
  const int32_t per = (n_blocks + 31) / 32;
  const int32_t b0 = lane * per < n_blocks ? lane * per : n_blocks;
  const int32_t b1 = b0 + per < n_blocks ? b0 + per : n_blocks;
  int64_t sum = 0;
  bool failed = false;
#pragma unroll 4
  for (int32_t k = b0; k < b1; ++k) {
    const uint64_t want =
        (uint64_t)(n_groups - k * kGroupBlock < kGroupBlock ? n_groups - k * kGroupBlock
                                                            : kGroupBlock);
    uint64_t v = g_load(&o.block_sum[k]);
    for (int spins = 0; (v >> kGCountShift) != want && spins < o.spin_limit; ++spins) {
      __nanosleep(32);
      v = g_load(&o.block_sum[k]);
    }
    failed = failed || (v >> kGCountShift) != want;
    sum += (int64_t)(v & kGSumMask);
  }
  int64_t x = sum;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, s);
    if (lane >= s) x += y;
  }
  const int64_t M = __shfl_sync(0xffffffffu, x, 31);
  int64_t run = x - sum;
  for (int32_t k = b0; k < b1; ++k) {
    o.block_base[k] = run;
    run += (int64_t)(g_load(&o.block_sum[k]) & kGSumMask);
  }
  // (records asked for, as room for kGroupRegions equal regions)
  static_assert(kGroupRegions == 32, "one region per lane");
  int64_t records = (int64_t)g_load(reinterpret_cast<uint64_t*>(&o.chunk_top[16 * lane]));
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const int64_t y = __shfl_xor_sync(0xffffffffu, records, s);
    records = y > records ? y : records;
  }
  records *= kGroupRegions;
  const bool any_failed = __any_sync(0xffffffffu, failed);
  if (lane == 0) {
    const int64_t err = (any_failed ? 1 : 0) | (b.bin_scan ? (int64_t)b.bin_scan[1] : 0);
    o.state[1] = (uint64_t)err;
    *o.total = M;
    *o.records = records;
    if (o.report) {
      volatile int64_t* r = o.report;
      r[1] = M;
      r[2] = err;
      r[3] = records;
      __threadfence_system();
      r[0] = 1;
    }
  }
}

__global__ void __launch_bounds__(kGThreads, 28)
    k_group_count(const __grid_constant__ GridParams g, const __grid_constant__ GridBuffers b,
                  int32_t n_cells, const __grid_constant__ GroupBand band,
                  const __grid_constant__ GroupSearch o) {
  extern __shared__ __align__(16) unsigned char gsm[];
  const int lane = threadIdx.x;
  GCountWarp& w_sm = *reinterpret_cast<GCountWarp*>(gsm);
  float4* const shift_of = reinterpret_cast<float4*>(gsm + sizeof(GCountWarp));
  GRing& ring = w_sm.ring;
  uint32_t* const mbuf = reinterpret_cast<uint32_t*>(w_sm.mask);
  const float2 nrc2 = make_float2(-band.rc2, -band.rc2);
  // Each stencil cell's translation into the home bin's frame (the same for
  // every group; FP64, rounded once).
  for (int32_t c = lane; c < n_cells; c += 32) {
    const int3 d = cell_offset(g, n_cells, c);
    float t[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      t[k] = __double2float_rn(dadd(dadd(dmul(g.basis[0][k], (double)d.x),
                                         dmul(g.basis[1][k], (double)d.y)),
                                    dmul(g.basis[2][k], (double)d.z)));
    shift_of[c] = make_float4(t[0], t[1], t[2], 0.f);
  }
  __syncwarp();
  pdl_wait();
  const int32_t split = o.split;
  const int64_t item = blockIdx.x;
  const int32_t t = (int32_t)((uint32_t)item / (uint32_t)split);
  const int32_t seg = (int32_t)(item - (int64_t)t * split);
  // (up to 32 cells: a segment is a slice of the row of all their candidates)
  const bool slices = n_cells <= 32;
  const int32_t c0 = slices ? 0 : n_cells * seg / split;
  const int32_t nc = slices ? n_cells : n_cells * (seg + 1) / split - c0;
  // (loaded together; the record of a group past the last is not used)
  const int32_t n_groups = b.counters[0], loose = *b.loose;
  const GroupRec grp = b.groups[t];
  const int64_t n_items = (int64_t)n_groups * split;
  // (an atom outside its stored bin by more than rounding: certain hits are
  // rechecked too, since the reference may prune their cell)
  const float near_lo = loose != 0 ? -INFINITY : -band.width;
  if (item < n_items) {
    const int32_t len = grp.end - grp.first < 32 ? grp.end - grp.first : 32;
    const int32_t p = grp.first + (lane < len ? lane : 0);
    const float4 a = b.p32[p];
    const bool irregular = lane < len && b.irr[p] != 0;
    const unsigned irr_mask = __ballot_sync(0xffffffffu, irregular);

    // The group's atoms (pairs, negated; irregular and missing ones far away
    // and after every candidate) and box.
    {
      const bool on = lane < len && !irregular;
      float* xy = reinterpret_cast<float*>(w_sm.xy) + 4 * (lane >> 1) + (lane & 1);
      float* zi = reinterpret_cast<float*>(w_sm.zi) + 4 * (lane >> 1) + (lane & 1);
      xy[0] = on ? -a.x : -1e30f;
      xy[2] = on ? -a.y : -1e30f;
      zi[0] = on ? -a.z : -1e30f;
      zi[2] = on ? a.w : __int_as_float(0x7fffffff);
    }
    const float3 glo = make_float3(warp_min(a.x), warp_min(a.y), warp_min(a.z));
    const float3 ghi = make_float3(-warp_min(-a.x), -warp_min(-a.y), -warp_min(-a.z));
    // (the halves rounded up: the box test's slack, a band width, is far above
    // the middle's rounding)
    const float3 mid = make_float3(0.5f * (glo.x + ghi.x), 0.5f * (glo.y + ghi.y),
                                   0.5f * (glo.z + ghi.z));
    const float3 half = make_float3(0.5f * (ghi.x - glo.x) * 1.000001f,
                                    0.5f * (ghi.y - glo.y) * 1.000001f,
                                    0.5f * (ghi.z - glo.z) * 1.000001f);
    __syncwarp();
    // Room for records is taken for each run of up to 32 cells, from one of
    // kGroupRegions regions (a single cursor would hand out one place every
    // 2 ns).
    const int region = (int)(item % kGroupRegions);
    int64_t taken = 0;  // lane 0: the segment's first record (-1: no room)

    uint32_t cnt = 0;  // lane: this atom's hits in the segment
    int32_t fill = 0, head = 0, n_rec = 0;
    const int n_quads = (len + 3) >> 2;

    // 3. the oldest v candidates of the ring against the group's atoms
    auto test = [&](int v) {
      const int k = (head + lane) & (kGRing - 1);
      const bool valid = lane < v;
      const float4 cj = ring.at[k];
      const float cx = cj.x, cy = cj.y, cz = cj.z;
      const int32_t jj = valid ? __float_as_int(cj.w) : 0;
      const float2 cx2 = make_float2(cx, cx), cy2 = make_float2(cy, cy),
                   cz2 = make_float2(cz, cz);
      float closest = INFINITY;  // smallest |t|
#pragma unroll 2
      for (int q = 0; q < n_quads; ++q) {
        unsigned m[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 xy = w_sm.xy[2 * q + h], zi = w_sm.zi[2 * q + h];
          const float2 dx = __fadd2_rn(cx2, make_float2(xy.x, xy.y));
          const float2 dy = __fadd2_rn(cy2, make_float2(xy.z, xy.w));
          const float2 dz = __fadd2_rn(cz2, make_float2(zi.x, zi.y));
          const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, nrc2)));
          m[2 * h] = __ballot_sync(0xffffffffu, d2.x < 0.f && __float_as_int(zi.z) < jj);
          m[2 * h + 1] = __ballot_sync(0xffffffffu, d2.y < 0.f && __float_as_int(zi.w) < jj);
          closest = fminf(fminf(closest, fabsf(d2.x)), fabsf(d2.y));
        }
        w_sm.mask[q] = make_uint4(m[0], m[1], m[2], m[3]);
      }
      if (__any_sync(0xffffffffu, closest <= band.width) || near_lo == -INFINITY) {
        // Some pair lies within the guard band: the reference's FP64 test.  Each
        // lane takes its candidate's pairs one after the other, the lanes side
        // by side: on a lattice whose cutoff is one of its distances, or in a
        // cell as wide as the cutoff, a chunk has a pair or more per atom in
        // the band (a crystal of 32,000 atoms with the cutoff on a shell: 180
        // -> 106 us against one atom of the group after the other, 108,000 333
        // -> 193; 100 atoms in a cell as wide as the cutoff 78 -> 57).
        uint32_t open = 0;  // the group's atoms whose pair with the lane's candidate is undecided
        for (int i = 0; i < len; ++i) {
          const float* xy = reinterpret_cast<const float*>(&w_sm.xy[i >> 1]) + (i & 1);
          const float* zi = reinterpret_cast<const float*>(&w_sm.zi[i >> 1]) + (i & 1);
          const float dx = __fadd_rn(cx, xy[0]), dy = __fadd_rn(cy, xy[2]),
                      dz = __fadd_rn(cz, zi[0]);
          const float d2 =
              __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, -band.rc2)));
          if (__float_as_int(zi[2]) < jj && d2 >= near_lo && d2 <= band.width) open |= 1u << i;
        }
        __syncwarp();
        for (; open; open &= open - 1) {
          const int i = __ffs(open) - 1;
          if (exact_hit(g, b, band.rc_sq, grp.first + i, ring.id[k].x, (uint32_t)ring.id[k].y))
            atomicOr(&mbuf[i], 1u << lane);
          else
            atomicAnd(&mbuf[i], ~(1u << lane));
        }
      }
      __syncwarp();
      const uint32_t h = lane < 4 * n_quads ? mbuf[lane] : 0u;
      if (__any_sync(0xffffffffu, h != 0)) {
        cnt += __popc(h);
        const int64_t base = __shfl_sync(0xffffffffu, taken, 0);
        if (base >= 0) {
          const int2 id = valid ? ring.id[k] : make_int2(0, 0);
          const uint32_t sh = (uint32_t)id.y;
          const bool shifted = __any_sync(0xffffffffu, sh != 0);
          const int64_t at = (base + n_rec) * 32 + lane;
          o.masks[at] = h;
          o.cand[at] = (uint32_t)id.x | (shifted ? 0x80000000u : 0u);
          if (shifted) o.cshift[at] = sh;
        }
        ++n_rec;
      }
      __syncwarp();  // (the masks and the ring slots are free again)
      head = (head + v) & (kGRing - 1);
      fill -= v;
    };

    const float reach = band.reach_sq;
    for (int32_t cb = 0; cb < nc; cb += 32) {
      // 1. up to 32 cells: lane = cell; the cells with candidates, in order,
      // and where each one's candidates start in the row of all of them
      int32_t k = 0, first = 0;
      uint32_t sh = 0;
      if (cb + lane < nc) {
        int32_t bin[3];
        const int2 r = g_describe(g, b, grp.bx, grp.by, grp.bz, n_cells, c0 + cb + lane, bin, sh);
        first = r.x;
        k = r.y - r.x;
      }
      int32_t start = k;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, start, s);
        if (lane >= s) start += y;
      }
      int32_t tot = __shfl_sync(0xffffffffu, start, 31);
      start -= k;
      int32_t f_begin = 0;
      if (slices && split > 1) {  // (about equal slices; the last one to the end)
        const int32_t per = tot / split, more = tot - per * split;
        f_begin = per * seg + min(seg, more);
        tot = f_begin + per + (seg < more ? 1 : 0);
      }
      const unsigned some = __ballot_sync(0xffffffffu, k > 0);
      if (k > 0) {
        const int at = __popc(some & lanemask_lt());
        const float4 tc = shift_of[c0 + cb + lane];
        w_sm.cell[at] = make_float4(tc.x, tc.y, tc.z, __int_as_float(first - start));
        w_sm.shift[at] = sh;
      } else {
        start = 0x7fffffff;
      }
      if (cb == 0) {
        taken = take_records(
            o, region, nc > 32 ? row_candidates(g, b, grp, n_cells, c0, nc) : tot - f_begin);
      }
      __syncwarp();

      // 2. the row's candidates, 32 at a time, through the ring (the next 32
      // are loaded before these are tested)
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f), tc = q;
      int32_t j = 0;
      // (cells that start before the slice)
      int32_t before = __popc(__ballot_sync(0xffffffffu, start < f_begin)) - 1;
      uint32_t csh = 0;
      auto fetch = [&](int32_t f0) {
        // cells that start in this window, at their place in it
        const uint32_t d = (uint32_t)(start - f0);
        const unsigned starts = __reduce_or_sync(0xffffffffu, d < 32u ? 1u << d : 0u);
        const int c = before + __popc(starts & (lanemask_lt() << 1 | 1u));
        before += __popc(starts);
        if (f0 + lane < tot) {
          tc = w_sm.cell[c];
          csh = w_sm.shift[c];
          j = f0 + lane + __float_as_int(tc.w);
          q = b.p32[j];
        }
      };
      if (f_begin < tot) fetch(f_begin);
      const bool last = cb + 32 >= nc;
      for (int32_t f0 = f_begin;; f0 += 32) {
        const float cx = q.x + tc.x, cy = q.y + tc.y, cz = q.z + tc.z;
        const int32_t jo = __float_as_int(q.w) + (csh != 0 ? 1 : 0);
        const int2 id = make_int2(j, (int32_t)csh);
        const bool on = f0 + lane < tot;
        if (f0 + 32 < tot) fetch(f0 + 32);
        const float gx = fmaxf(fabsf(cx - mid.x) - half.x, 0.f);
        const float gy = fmaxf(fabsf(cy - mid.y) - half.y, 0.f);
        const float gz = fmaxf(fabsf(cz - mid.z) - half.z, 0.f);
        const bool keep = on && !(__fmaf_rn(gx, gx, __fmaf_rn(gy, gy, gz * gz)) > reach);
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int at = (head + fill + __popc(km & lanemask_lt())) & (kGRing - 1);
          ring.at[at] = make_float4(cx, cy, cz, __int_as_float(jo));
          ring.id[at] = id;
        }
        fill += __popc(km);
        __syncwarp();
        // (a full chunk, or what is left after the last candidates)
        const bool end = f0 + 32 >= tot;
        while (fill >= 32 || (fill > 0 && end && last)) test(fill < 32 ? fill : 32);
        if (end) break;
      }
      __syncwarp();  // (the cells' records are free again)
    }

    if (lane == 0) o.seg_rec[item] = make_longlong2(taken, n_rec);
    int32_t before = split - 1;
    if (split > 1) {
      // The last segment of the group to be counted finishes it.
      o.seg_cnt[item * 32 + lane] = cnt;
      __syncwarp();
      if (lane == 0) before = add_acq_rel(&o.group_done[t], 1);
      before = __shfl_sync(0xffffffffu, before, 0);
      __syncwarp();
    }
    if (before == split - 1) finish_group(g, b, n_cells, band, o, t, grp, irr_mask, cnt);
  }
  // The last CTA to end scans the blocks.
  __syncwarp();
  int32_t last = 0;
  if (lane == 0) last = add_acq_rel(o.done, 1) == (int32_t)gridDim.x - 1;
  if (__shfl_sync(0xffffffffu, last, 0)) {
    __syncwarp();
    finish_list(b, o, n_groups);
  }
}

// Shared memory of one warp of the emit pass.
struct GEmitWarp {
  uint32_t mask[32 * kGWindow];  // the window's records: hit masks
  // and candidates: original index, and wrap + image shift in the bits above
  uint32_t cand[32 * kGWindow];
  SlotMeta meta[32];             // the group's atoms
  int64_t slot[32];              // atom's next output slot minus its place in the stage
};
// (behind it: uint16_t hits[GroupOut::stage], atom << 10 | candidate, in output
// order)
static_assert(sizeof(GEmitWarp) % 16 == 0 && 32 * kGWindow <= 1024, "vector accesses, 10-bit entries");

__device__ __forceinline__ void copy16(void* smem, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(smem)),
               "l"(global)
               : "memory");
}

// Emit pass (the file comment).  Writes nothing when a wait gave up, the list
// does not fit, or the records did not (the host then grows the arrays and
// runs what is missing again).
template <bool EX>
__global__ void __launch_bounds__(kGThreads, 28)
    k_group_emit(const __grid_constant__ GridParams g, const __grid_constant__ GridBuffers b,
                 int32_t n_cells, double rc_sq, const __grid_constant__ GroupSearch o,
                 const __grid_constant__ GroupOut out) {
  extern __shared__ __align__(16) unsigned char gsm[];
  const int lane = threadIdx.x;
  GEmitWarp& w_sm = *reinterpret_cast<GEmitWarp*>(gsm);
  uint16_t* const hits = reinterpret_cast<uint16_t*>(&w_sm + 1);
  pdl_wait();
  const int32_t split = o.split;
  const int64_t item = blockIdx.x;
  const int32_t t = (int32_t)((uint32_t)item / (uint32_t)split);
  const int32_t seg = (int32_t)(item - (int64_t)t * split);
  // (loaded together; what belongs to a group past the last is not used)
  const int64_t M = *o.total, records = *o.records;
  const uint64_t err = o.state[1];
  const int32_t n_groups = b.counters[0];
  const longlong2 rec = o.seg_rec[item];
  const GroupRec grp = b.groups[t];
  int64_t slot = o.block_base[t / kGroupBlock] + o.atom_base[(int64_t)t * 32 + lane];
  if (split > 1) slot += o.seg_cnt[item * 32 + lane];  // (the atom's hits in earlier segments)
  // The group's first slot: its block's and the block's groups before it.
  int64_t base = 0;
#pragma unroll
  for (int k = 0; k < kGroupBlock / 32; ++k) {
    const int32_t u = t / kGroupBlock * kGroupBlock + 32 * k + lane;
    if (u < t) base += o.group_total[u];
  }
  if (err != 0 || M > out.capacity || records > o.chunk_cap || t >= n_groups) return;
  const int64_t d_ei = EX && out.directed ? 2 * M : M;
  const int64_t first_rec = rec.x;
  const int n_rec = (int)rec.y;
  const int32_t len = grp.end - grp.first < 32 ? grp.end - grp.first : 32;
  const int32_t p = grp.first + (lane < len ? lane : 0);
  w_sm.meta[lane] = b.meta[p];
  const bool irregular = seg == 0 && lane < len && b.irr[p] != 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) base += __shfl_xor_sync(0xffffffffu, base, s);
  slot += base;

  // A candidate's original index takes orig_bits, each component of its shift a
  // third of the rest (2 bits at the most atoms, 6 at 10,000).
  const int s_bits = (32 - out.orig_bits) / 3;
  const int32_t s_half = 1 << (s_bits - 1);
  const uint32_t s_mask = (1u << s_bits) - 1u, orig_mask = (1u << out.orig_bits) - 1u;
  const int down = 32 - s_bits;
  const int up[3] = {down - out.orig_bits, down - out.orig_bits - s_bits,
                     down - out.orig_bits - 2 * s_bits};

  for (int r0 = 0; r0 < n_rec;) {
    // A window of up to kGWindow records whose hits fit the stage.
    const int n_load = n_rec - r0 < kGWindow ? n_rec - r0 : kGWindow;
    const int64_t at = (first_rec + r0) * 32;
    for (int k = lane; k < 8 * n_load; k += 32) copy16(&w_sm.mask[4 * k], &o.masks[at + 4 * k]);
    // (the shifts of the window's candidates, packed when all fit)
    bool wide = false;
#pragma unroll 4
    for (int c = 0; c < n_load; ++c) {
      const uint32_t w = o.cand[at + 32 * c + lane];
      const uint32_t csh = w >> 31 ? o.cshift[at + 32 * c + lane] : 0u;
      const SlotMeta mj = b.meta[w & 0x7fffffffu];
      const int32_t s0 = mj.sx + unpack_shift(csh, 0), s1 = mj.sy + unpack_shift(csh, 1),
                    s2 = mj.sz + unpack_shift(csh, 2);
      wide = wide || (uint32_t)(s0 + s_half) > s_mask || (uint32_t)(s1 + s_half) > s_mask ||
             (uint32_t)(s2 + s_half) > s_mask;
      w_sm.cand[32 * c + lane] =
          (uint32_t)mj.orig | (((uint32_t)s0 & s_mask) | ((uint32_t)s1 & s_mask) << s_bits |
                               ((uint32_t)s2 & s_mask) << (2 * s_bits))
                                  << out.orig_bits;
    }
    wide = __any_sync(0xffffffffu, wide);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    int n_win = 0, total = 0, mine = 0;
    for (; n_win < n_load; ++n_win) {
      const int k = __popc(w_sm.mask[32 * n_win + lane]);
      const int sum = __reduce_add_sync(0xffffffffu, k);
      if (total + sum > out.stage) break;
      total += sum;
      mine += k;
    }
    int pre = mine;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, pre, s);
      if (lane >= s) pre += y;
    }
    pre -= mine;
    w_sm.slot[lane] = slot - pre;
    slot += mine;
    for (int c = 0; c < n_win; ++c) {
      uint32_t h = w_sm.mask[32 * c + lane];
      const uint32_t entry = (uint32_t)lane << 10 | (uint32_t)c << 5;
      while (h) {
        hits[pre++] = (uint16_t)(entry | (uint32_t)(__ffs(h) - 1));
        h &= h - 1;
      }
    }
    __syncwarp();
#pragma unroll 2
    for (int k = lane; k < total; k += 32) {
      const uint32_t v = hits[k];
      const uint32_t cj = w_sm.cand[v & 1023u];
      const SlotMeta ml = w_sm.meta[v >> 10];
      const int64_t e = w_sm.slot[v >> 10] + k;
      int32_t s0 = (int32_t)(cj << up[0]) >> down, s1 = (int32_t)(cj << up[1]) >> down,
              s2 = (int32_t)(cj << up[2]) >> down;
      if (wide) {
        const uint32_t w = o.cand[at + (v & 1023u)];
        const uint32_t csh = w >> 31 ? o.cshift[at + (v & 1023u)] : 0u;
        const SlotMeta mj = b.meta[w & 0x7fffffffu];
        s0 = mj.sx + unpack_shift(csh, 0);
        s1 = mj.sy + unpack_shift(csh, 1);
        s2 = mj.sz + unpack_shift(csh, 2);
      }
      write_edge<EX>(out, d_ei, M, e, ml.orig, (int32_t)(cj & orig_mask), s0 - ml.sx, s1 - ml.sy,
                     s2 - ml.sz);
    }
    __syncwarp();
    r0 += n_win;
  }
  for (unsigned im = __ballot_sync(0xffffffffu, irregular); im; im &= im - 1) {
    const int l = __ffs(im) - 1;
    const int64_t e0 =
        o.block_base[t / kGroupBlock] + base + o.atom_base[(int64_t)t * 32 + l];
    g_irregular<true, EX>(g, b, n_cells, rc_sq, grp.first + l, e0, &out, d_ei, M);
  }
}

}  // namespace

GroupBand group_band(const GuardBand& band) {
  GroupBand gb;
  gb.rc_sq = band.rc_sq;
  gb.rc2 = (float)band.rc_sq;
  // (half-width from the rounded rc^2 to the farther edge of the band)
  const float up = std::nextafter(band.hi - gb.rc2, INFINITY);
  const float down = std::nextafter(gb.rc2 - band.lo, INFINITY);
  gb.width = std::max(up, down);
  gb.reach_sq = band.hi + (band.hi - band.lo);
  return gb;
}

void launch_group_count(const GridParams& g, const GridBuffers& b, int32_t n_cells,
                        const GroupBand& band, const GroupSearch& o, cudaStream_t s) {
  const size_t smem = sizeof(GCountWarp) + sizeof(float4) * (size_t)n_cells;
  ensure_smem_attr((const void*)k_group_count, (int)smem);
  launch_pdl(k_group_count, dim3((unsigned)(o.max_groups * o.split)),
             dim3(kGThreads), smem, s, g, b, n_cells, band, o);
  note_launches(1);
}

void launch_group_emit(const GridParams& g, const GridBuffers& b, int32_t n_cells,
                       const GroupBand& band, const GroupSearch& o, const GroupOut& out,
                       cudaStream_t s) {
  const auto k = out.directed || out.vec || out.dist ? &k_group_emit<true> : &k_group_emit<false>;
  launch_pdl(k, dim3((unsigned)(o.max_groups * o.split)), dim3(kGThreads),
             sizeof(GEmitWarp) + 2 * (size_t)out.stage, s, g, b, n_cells, band.rc_sq, o, out);
  note_launches(1);
}

}  // namespace nlb
