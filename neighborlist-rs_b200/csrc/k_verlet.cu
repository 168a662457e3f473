// k_verlet.cu -- kernels of the Verlet (skin) list manager.
//
//   k_verlet_pack     a rebuilt list into the manager's form: atoms as int32
//                   pairs, shifts packed into three signed 10-bit fields (and
//                   unpacked ones beside them, read only when some shift does
//                   not fit)
//   k_max_disp      max_i |r_i - r_i,ref|^2 over the atoms (FP64, exact
//                   squares and sums; the max of non-negative doubles is
//                   taken on their bit patterns, which order the same way)
//   k_verlet_count  that maximum, and one pass over the stored edges (i, j, S):
//                   kept when |(r_j - r_i) + H.S|^2 < rc^2 with the current
//                   positions (the displacement expression of k_extras.cu), as
//                   a bit per edge and counts; M and the maximum go to the
//                   host through host-mapped memory as soon as they are known
//   k_verlet_write  the kept edges in stored order ([src | dst], shifts), while
//                   the caller goes on
// Streaming kernels: 12 B + two position gathers per stored edge, 12 + 28 B per
// kept edge.  An update of the 10,008-atom liquid (rc 6, skin 1, 0.7 M stored
// edges) has a floor of 5 us and is a chain of latencies: 16 us for the count,
// 7.6 for the write; the call took 74 us in three launches with copies and a
// synchronisation, 45 in one launch that found the slots by a look-back and
// moved the destinations behind the sources at its end, and takes 32.
#include <algorithm>

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
constexpr int kVcPer = 8;                     // stored edges per thread
constexpr int kVcTile = kVcThreads * kVcPer;  // stored edges per CTA
constexpr int kVcWords = kVcTile / 32;        // its mask words

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

// An update's first launch: the CTA's share of the largest displacement, and
// one tile of kVcTile stored edges tested at rc with the current positions
// (each warp a run of 256 edges, lane-striped so that loads are coalesced): a
// mask word per 32 edges and the tile's count. The last CTA to end turns the
// counts into the tiles' first slots, reports {M, displacement bits} and
// leaves done and disp zero for the next launch.
__global__ void __launch_bounds__(kVcThreads)
    k_verlet_count(const double* __restrict__ pos, const double* __restrict__ ref, int64_t n,
                   const __grid_constant__ EdgeExtrasCell cell,
                   const __grid_constant__ VerletEdges list, double rc_sq,
                   const __grid_constant__ VerletWork work, int64_t* report) {
  __shared__ int64_t warp_sum[kVcThreads / 32];
  __shared__ double warp_far[kVcThreads / 32];
  __shared__ bool s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t m = list.m;
  const int64_t n_tiles = (m + kVcTile - 1) / kVcTile;
  pdl_wait();
  const int64_t t = blockIdx.x;
  const int64_t wbase = t * kVcTile + (int64_t)warp * 32 * kVcPer;
  const bool wide = *list.wide != 0;
  int2 ij[kVcPer];
  uint32_t psh[kVcPer];
#pragma unroll
  for (int k = 0; k < kVcPer; ++k) {
    const int64_t e = wbase + 32 * k + lane;
    ij[k] = e < m ? list.ij[e] : make_int2(0, 0);
    psh[k] = e < m ? list.packed[e] : 0u;
  }
  const bool moved = t * kVcThreads < n;
  if (moved) {
    const double far = max_disp_share(pos, ref, n);
    if (lane == 0) warp_far[warp] = far;
  }
  uint32_t word = 0;  // lane k: the run's mask word k
  int32_t kept = 0;
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
    const uint32_t mask = __ballot_sync(0xffffffffu, keep);
    if (lane == k) word = mask;
    kept += __popc(mask);
  }
  if (t < n_tiles && lane < kVcPer) work.masks[t * kVcWords + warp * kVcPer + lane] = word;
  if (lane == 0) warp_sum[warp] = kept;
  __syncthreads();
  if (tid == 0) {
    int64_t sum = 0;
    double far = 0.0;
    for (int w = 0; w < kVcThreads / 32; ++w) {
      sum += warp_sum[w];
      if (moved && warp_far[w] > far) far = warp_far[w];
    }
    if (moved)
      atomicMax(reinterpret_cast<unsigned long long*>(work.disp),
                (unsigned long long)__double_as_longlong(far));
    if (t < n_tiles) work.base[t] = sum;
    // (the CTA's writes, ordered before this by the barrier, are released
    // with it)
    __threadfence();
    s_last = atomicAdd(reinterpret_cast<unsigned long long*>(work.done), 1ull) ==
             (unsigned long long)gridDim.x - 1ull;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  // Thread k takes the k-th run of tiles: its sum, the sums before it, and the
  // tiles' first slots.
  const int64_t per = (n_tiles + kVcThreads - 1) / kVcThreads;
  const int64_t b0 = tid * per < n_tiles ? tid * per : n_tiles;
  const int64_t b1 = b0 + per < n_tiles ? b0 + per : n_tiles;
  int64_t mine = 0;
#pragma unroll 4
  for (int64_t k = b0; k < b1; ++k) mine += __ldcg(&work.base[k]);
  int64_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int64_t slot = incl - mine, total = 0;
#pragma unroll
  for (int w = 0; w < kVcThreads / 32; ++w) {
    slot += w < warp ? warp_sum[w] : 0;
    total += warp_sum[w];
  }
#pragma unroll 4
  for (int64_t k = b0; k < b1; ++k) {
    const int64_t c = __ldcg(&work.base[k]);
    work.base[k] = slot;
    slot += c;
  }
  if (tid == 0) {
    *work.total = total;
    volatile int64_t* r = report;
    r[1] = total;
    r[2] = 0;
    r[3] = (int64_t) * reinterpret_cast<volatile uint64_t*>(work.disp);
    *work.done = 0;
    *work.disp = 0;
    __threadfence_system();
    r[0] = 1;
  }
}

// Its second launch: the kept edges, in stored order, a CTA per tile.
__global__ void __launch_bounds__(kVcThreads)
    k_verlet_write(const __grid_constant__ VerletEdges list,
                   const __grid_constant__ VerletWork work, int64_t* __restrict__ out_ei,
                   int32_t* __restrict__ out_sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_wait();
  const int64_t t = blockIdx.x;
  const bool wide = *list.wide != 0;
  const int64_t M = *work.total;
  int64_t o0 = work.base[t];
  // the run's mask words, and the kept edges of the runs before it
  static_assert(kVcWords == 64, "two words a lane");
  const uint32_t w0 = work.masks[t * kVcWords + lane], w1 = work.masks[t * kVcWords + 32 + lane];
  const int first = warp * kVcPer;
  o0 += __reduce_add_sync(0xffffffffu, (lane < first ? __popc(w0) : 0) +
                                           (lane + 32 < first ? __popc(w1) : 0));
  const int64_t wbase = t * kVcTile + (int64_t)first * 32;
  uint32_t mask[kVcPer];
  int2 ij[kVcPer];
  uint32_t psh[kVcPer];
#pragma unroll
  for (int k = 0; k < kVcPer; ++k) {
    mask[k] = __shfl_sync(0xffffffffu, first < 32 ? w0 : w1, (first + k) & 31);
    if ((mask[k] >> lane) & 1u) {
      ij[k] = list.ij[wbase + 32 * k + lane];
      psh[k] = list.packed[wbase + 32 * k + lane];
    }
  }
#pragma unroll
  for (int k = 0; k < kVcPer; ++k) {
    if ((mask[k] >> lane) & 1u) {
      const int64_t o = o0 + __popc(mask[k] & ((1u << lane) - 1u));
      int32_t s[3];
      edge_shift(list, wide, wbase + 32 * k + lane, psh[k], s);
      out_ei[o] = (int64_t)ij[k].x;
      out_ei[M + o] = (int64_t)ij[k].y;
      out_sh[3 * o] = s[0];
      out_sh[3 * o + 1] = s[1];
      out_sh[3 * o + 2] = s[2];
    }
    o0 += __popc(mask[k]);
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

int64_t verlet_tiles(int64_t m) { return (m + kVcTile - 1) / kVcTile; }
int64_t verlet_mask_words(int64_t m) { return verlet_tiles(m) * kVcWords; }

void launch_verlet_update(const double* pos, const double* ref, int64_t n,
                          const EdgeExtrasCell& cell, const VerletEdges& list, double rc_sq,
                          const VerletWork& work, int64_t* out_ei, int32_t* out_sh,
                          int64_t* report, cudaStream_t s) {
  const int64_t n_tiles = verlet_tiles(list.m);
  // (with few stored edges, a CTA per SM at most for the displacements)
  const int64_t moves = std::min<int64_t>((n + kVcThreads - 1) / kVcThreads, 148);
  const int64_t grid = std::max<int64_t>({n_tiles, moves, 1});
  launch_pdl(k_verlet_count, dim3((unsigned)grid), dim3(kVcThreads), 0, s, pos, ref, n, cell, list,
             rc_sq, work, report);
  note_launches(1);
  if (n_tiles == 0) return;
  launch_pdl(k_verlet_write, dim3((unsigned)n_tiles), dim3(kVcThreads), 0, s, list, work, out_ei,
             out_sh);
  note_launches(1);
}

}  // namespace nlb
