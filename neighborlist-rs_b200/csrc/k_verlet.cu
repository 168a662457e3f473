// k_verlet.cu -- kernels of the Verlet (skin) list manager.
//
//   k_verlet_pack     a rebuilt list into the manager's form: atoms as int32
//                   pairs, shifts packed into three signed 10-bit fields (and
//                   unpacked ones beside them, read only when some shift does
//                   not fit)
//   k_max_disp      max_i |r_i - r_i,ref|^2 over the atoms (FP64, exact
//                   squares and sums; the max of non-negative doubles is
//                   taken on their bit patterns, which order the same way)
//   k_verlet_compact  one launch per update: that maximum, and one pass over
//                   the stored edges (i, j, S): kept when |(r_j - r_i) +
//                   H.S|^2 < rc^2 with the current positions (the
//                   displacement expression of k_extras.cu), compacted in
//                   stored order by a decoupled look-back over tiles ([src |
//                   dst], shifts); M and the maximum go to the host through
//                   host-mapped memory
// A streaming kernel: 12 B + two position gathers per stored edge, 28 B (+ 8
// for the destinations' move, int32 in between) per kept edge.  With 28-byte
// stored edges, read again for the kept ones, int64 destinations in between,
// a launch of its own for the maximum and copies and a synchronisation for
// the results, an update of the 10,008-atom liquid (rc 6, skin 1) took 74 us.
#include <algorithm>
#include <atomic>

#include "nlb_kernels.h"

namespace nlb {

namespace {

__device__ __forceinline__ void edge_disp(const double* __restrict__ pos,
                                          const EdgeExtrasCell& cell, int64_t i, int64_t j,
                                          int32_t s0, int32_t s1, int32_t s2, double* d) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double rel = dsub(pos[3 * j + k], pos[3 * i + k]);
    if (cell.has_cell) {
      const double hs = dadd(dadd(dmul(cell.h[3 * k], (double)s0),
                                  dmul(cell.h[3 * k + 1], (double)s1)),
                             dmul(cell.h[3 * k + 2], (double)s2));
      d[k] = dadd(rel, hs);
    } else {
      d[k] = rel;
    }
  }
}

// Image shift of stored edge e.
__device__ __forceinline__ void edge_shift(const VerletEdges& list, bool wide, int64_t e,
                                           uint32_t packed, int32_t s[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k)
    s[k] = wide ? list.plain[3 * e + k] : (int32_t)(packed << (22 - 10 * k)) >> 22;
}

// Largest squared displacement over the calling grid's share of the atoms,
// reduced over the warp.
__device__ __forceinline__ double max_disp_share(const double* __restrict__ pos,
                                                 const double* __restrict__ ref, int64_t n) {
  double best = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double d = norm2(dsub(pos[3 * i], ref[3 * i]), dsub(pos[3 * i + 1], ref[3 * i + 1]),
                           dsub(pos[3 * i + 2], ref[3 * i + 2]));
    // NaN (a broken trajectory) must force a rebuild: map it to +inf.
    const double v = d != d ? INFINITY : d;
    best = v > best ? v : best;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  return best;
}

__global__ void k_max_disp(const double* __restrict__ pos, const double* __restrict__ ref,
                           int64_t n, unsigned long long* __restrict__ out) {
  const double best = max_disp_share(pos, ref, n);
  if ((threadIdx.x & 31) == 0)
    atomicMax(out, (unsigned long long)__double_as_longlong(best));
}

constexpr int kVcThreads = 256;
constexpr int kVcPer = 8;                          // stored edges per thread
constexpr int kVcTile = kVcThreads * kVcPer;       // stored edges per tile
constexpr uint64_t kVcShift = 62;
constexpr uint64_t kVcAggregate = 1ull << kVcShift;
constexpr uint64_t kVcInclusive = 2ull << kVcShift;
constexpr uint64_t kVcValue = (1ull << kVcShift) - 1;

__global__ void k_verlet_pack(const int64_t* __restrict__ ei, const int32_t* __restrict__ sh,
                              int64_t m, int2* __restrict__ ij, uint32_t* __restrict__ packed,
                              int32_t* __restrict__ plain, int32_t* __restrict__ wide) {
  bool far = false;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < m;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int32_t s0 = sh[3 * e], s1 = sh[3 * e + 1], s2 = sh[3 * e + 2];
    ij[e] = make_int2((int32_t)ei[e], (int32_t)ei[m + e]);
    packed[e] = ((uint32_t)s0 & 1023u) | ((uint32_t)s1 & 1023u) << 10 | ((uint32_t)s2 & 1023u) << 20;
    plain[3 * e] = s0;
    plain[3 * e + 1] = s1;
    plain[3 * e + 2] = s2;
    far = far || (uint32_t)(s0 + 512) > 1023u || (uint32_t)(s1 + 512) > 1023u ||
          (uint32_t)(s2 + 512) > 1023u;
  }
  if (far) atomicExch(wide, 1);
}

// CTAs first take their share of the largest displacement, then tiles of
// kVcTile stored edges in order (tickets): tested at rc with the current
// positions (each warp a run of 256 edges, lane-striped so that loads are
// coalesced), the tile's first output slot found by a decoupled look-back over
// the tiles before it (bounded polls; a wait that runs out sets state[1] and
// the tile writes nothing), the kept edges written in stored order: sources
// and shifts in place, destinations to dst_tmp.  Once every tile is written
// (all tickets are held by running CTAs, so the wait ends; bounded all the
// same), the CTAs move the destinations behind the M sources.  The last CTA
// to end clears the state for the next launch and reports {M, error word,
// displacement bits}.  state (zero on entry): [0] ticket, [1] error, [2] tiles
// done, [3] M, [4] CTAs done, [5] displacement, [6 + t] tile t's look-back
// word.
__global__ void __launch_bounds__(kVcThreads)
    k_verlet_compact(const double* __restrict__ pos, const double* __restrict__ ref, int64_t n,
                     EdgeExtrasCell cell, VerletEdges list, double rc_sq,
                     int64_t* __restrict__ out_ei, int32_t* __restrict__ out_sh,
                     int32_t* __restrict__ dst_tmp, uint64_t* __restrict__ state,
                     int32_t spin_limit, int64_t* report) {
  __shared__ int64_t s_tile, s_base;
  __shared__ int32_t warp_cnt[kVcThreads / 32];
  __shared__ int32_t s_skip;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t m = list.m;
  const int64_t n_tiles = (m + kVcTile - 1) / kVcTile;
  uint64_t* const tiles = state + 6;
  const bool wide = *list.wide != 0;
  if ((int64_t)blockIdx.x * kVcThreads < n) {
    const double far = max_disp_share(pos, ref, n);
    if (lane == 0)
      atomicMax(reinterpret_cast<unsigned long long*>(&state[5]),
                (unsigned long long)__double_as_longlong(far));
  }
  for (;;) {
    if (tid == 0) s_tile = (int64_t)atomicAdd(reinterpret_cast<unsigned long long*>(state), 1ull);
    __syncthreads();
    const int64_t t = s_tile;
    if (t >= n_tiles) break;
    const int64_t wbase = t * kVcTile + (int64_t)warp * 32 * kVcPer;
    int2 ij[kVcPer];
    uint32_t psh[kVcPer], kmask[kVcPer];
    int32_t wtot = 0;
#pragma unroll
    for (int k = 0; k < kVcPer; ++k) {
      const int64_t e = wbase + 32 * k + lane;
      ij[k] = e < m ? list.ij[e] : make_int2(0, 0);
      psh[k] = e < m ? list.packed[e] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kVcPer; ++k) {
      const int64_t e = wbase + 32 * k + lane;
      bool keep = false;
      if (e < m) {
        int32_t s[3];
        edge_shift(list, wide, e, psh[k], s);
        double d[3];
        edge_disp(pos, cell, ij[k].x, ij[k].y, s[0], s[1], s[2], d);
        keep = norm2(d[0], d[1], d[2]) < rc_sq;
      }
      kmask[k] = __ballot_sync(0xffffffffu, keep);
      wtot += __popc(kmask[k]);
    }
    if (lane == 0) warp_cnt[warp] = wtot;
    __syncthreads();
    int32_t woff = 0, tile_tot = 0;
#pragma unroll
    for (int w = 0; w < kVcThreads / 32; ++w) {
      const int32_t v = warp_cnt[w];
      woff += w < warp ? v : 0;
      tile_tot += v;
    }
    if (warp == 0) {
      // Publish the tile's count at once, then walk back over the tiles
      // before it (32 at a time) to its first output slot.
      if (lane == 0) {
        __threadfence();
        *reinterpret_cast<volatile uint64_t*>(&tiles[t]) =
            (t == 0 ? kVcInclusive : kVcAggregate) | (uint64_t)tile_tot;
      }
      int64_t prefix = 0;
      bool failed_any = false;
      if (t > 0) {
        int64_t tt = t - 1;
        for (;;) {
          const int64_t pred = tt - lane;
          uint64_t v = kVcInclusive;
          bool failed = false;
          if (pred >= 0) {
            int spins = 0;
            v = *reinterpret_cast<const volatile uint64_t*>(&tiles[pred]);
            while ((v >> kVcShift) == 0 && spins < spin_limit) {
              __nanosleep(32);
              v = *reinterpret_cast<const volatile uint64_t*>(&tiles[pred]);
              ++spins;
            }
            failed = (v >> kVcShift) == 0;
          }
          if (__any_sync(0xffffffffu, failed)) {
            if (lane == 0) atomicExch(reinterpret_cast<unsigned long long*>(&state[1]), 1ull);
            failed_any = true;
            break;
          }
          const unsigned inc = __ballot_sync(0xffffffffu, (v >> kVcShift) == 2);
          const int stop = __ffs(inc) - 1;
          int64_t val = (pred >= 0 && lane <= (stop < 0 ? 31 : stop)) ? (int64_t)(v & kVcValue) : 0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
          prefix += val;
          if (stop >= 0) break;
          tt -= 32;
        }
        if (lane == 0 && !failed_any) {
          __threadfence();
          *reinterpret_cast<volatile uint64_t*>(&tiles[t]) =
              kVcInclusive | (uint64_t)(prefix + tile_tot);
        }
      }
      if (lane == 0) {
        s_base = prefix;
        s_skip = failed_any ? 1 : 0;
        if (t == n_tiles - 1) state[3] = failed_any ? 0 : (uint64_t)(prefix + tile_tot);
      }
    }
    __syncthreads();
    if (!s_skip) {
      const int64_t g = s_base + woff;
      int32_t acc = 0;
#pragma unroll
      for (int k = 0; k < kVcPer; ++k) {
        if ((kmask[k] >> lane) & 1u) {
          const int64_t o = g + acc + __popc(kmask[k] & ((1u << lane) - 1u));
          int32_t s[3];
          edge_shift(list, wide, wbase + 32 * k + lane, psh[k], s);
          out_ei[o] = (int64_t)ij[k].x;
          dst_tmp[o] = ij[k].y;
          out_sh[3 * o] = s[0];
          out_sh[3 * o + 1] = s[1];
          out_sh[3 * o + 2] = s[2];
        }
        acc += __popc(kmask[k]);
      }
    }
    // One thread releases the tile's writes (ordered before it by the
    // barrier) with the completion count.
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(reinterpret_cast<unsigned long long*>(&state[2]), 1ull);
    }
  }
  if (tid == 0) {
    int spins = 0;
    unsigned long long d = *reinterpret_cast<volatile unsigned long long*>(&state[2]);
    while (d < (unsigned long long)n_tiles && spins < spin_limit) {
      __nanosleep(64);
      d = *reinterpret_cast<volatile unsigned long long*>(&state[2]);
      ++spins;
    }
    s_skip = d >= (unsigned long long)n_tiles ? 0 : 1;
    if (s_skip) atomicExch(reinterpret_cast<unsigned long long*>(&state[1]), 1ull);
    __threadfence();
  }
  __syncthreads();
  if (!s_skip) {
    const int64_t total = (int64_t)*reinterpret_cast<volatile uint64_t*>(&state[3]);
    for (int64_t k = (int64_t)blockIdx.x * kVcThreads + tid; k < total;
         k += (int64_t)gridDim.x * kVcThreads)
      out_ei[total + k] = (int64_t)__ldcg(&dst_tmp[k]);
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    s_skip = atomicAdd(reinterpret_cast<unsigned long long*>(&state[4]), 1ull) ==
             (unsigned long long)gridDim.x - 1ull;
    __threadfence();
  }
  __syncthreads();
  if (!s_skip) return;
  // The last CTA: every other one has ended.
  volatile uint64_t* st = state;
  const uint64_t kept = st[3], err = st[1], far = st[5];
  __syncthreads();
  for (int64_t k = tid; k < 6 + n_tiles; k += kVcThreads) state[k] = 0;
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    volatile int64_t* r = report;
    r[1] = (int64_t)kept;
    r[2] = (int64_t)err;
    r[3] = (int64_t)far;
    __threadfence_system();
    r[0] = 1;
  }
}

int stream_grid(int64_t items) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t want = (items + 255) / 256;
  const int64_t cap = (int64_t)sms * 8;
  return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

}  // namespace

void launch_max_disp(const double* pos, const double* ref, int64_t n, unsigned long long* out,
                     cudaStream_t s) {
  cudaMemsetAsync(out, 0, sizeof(unsigned long long), s);
  if (n <= 0) return;
  k_max_disp<<<stream_grid(n), 256, 0, s>>>(pos, ref, n, out);
  note_launches(1);
}

void launch_verlet_pack(const int64_t* ei, const int32_t* sh, int64_t m, int2* ij,
                        uint32_t* packed, int32_t* plain, int32_t* wide, cudaStream_t s) {
  cudaMemsetAsync(wide, 0, sizeof(int32_t), s);
  if (m <= 0) return;
  k_verlet_pack<<<stream_grid(m), 256, 0, s>>>(ei, sh, m, ij, packed, plain, wide);
  note_launches(1);
}

int64_t verlet_compact_state_words(int64_t m) { return 6 + (m + kVcTile - 1) / kVcTile; }

void launch_verlet_compact(const double* pos, const double* ref, int64_t n,
                           const EdgeExtrasCell& cell, const VerletEdges& list, double rc_sq,
                           int64_t* out_ei, int32_t* out_sh, int32_t* dst_tmp, uint64_t* state,
                           int32_t spin_limit, int64_t* report, cudaStream_t s) {
  // (SMs and resident CTAs per SM of each device, looked up once)
  static std::atomic<int> cached[64][2];
  int dev = 0;
  cudaGetDevice(&dev);
  const bool known = dev >= 0 && dev < 64;
  int sms = known ? cached[dev][0].load() : 0, per_sm = known ? cached[dev][1].load() : 0;
  if (sms <= 0 || per_sm <= 0) {
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_verlet_compact, kVcThreads, 0);
    sms = std::max(sms, 1);
    per_sm = std::max(per_sm, 1);
    if (known) {
      cached[dev][0].store(sms);
      cached[dev][1].store(per_sm);
    }
  }
  const int64_t n_tiles = (list.m + kVcTile - 1) / kVcTile;
  const int64_t grid = std::min<int64_t>((int64_t)sms * per_sm, std::max<int64_t>(n_tiles, sms));
  k_verlet_compact<<<(unsigned)grid, kVcThreads, 0, s>>>(pos, ref, n, cell, list, rc_sq, out_ei,
                                                         out_sh, dst_tmp, state, spin_limit,
                                                         report);
  note_launches(1);
}

}  // namespace nlb
