// particles.cu -- swimmer force spreading and the swimmer / tracer Move kernels.
//
// Spreading (reference SwimmerArray.cu:42-121) adds, for each swimmer, -P n at
// the tail r - l n and +P n at the head r through the 4^3 Peskin stencil.  The
// reference scatters with FP64 atomics in arbitrary order.  Here the result is
// deterministic and uses no floating-point atomics: AddForces records the 2n
// dipole ends (origin, Peskin weights, force) and lists them under every tile
// their stencil touches; each tile then sums its ends, in integers or in end
// order.  The tiles are either force tiles (k_force_fixed and k_force_tile,
// which write the dense force field of an FP64 lattice) or, for FP32/BF16/FP16
// lattices, the slabs of the fused step kernel, which spreads the ends itself so
// the force field never goes through HBM.
//
// The original 4^3-origin-bin kernels below (k_spread_bin ... k_spread_gather)
// serve lbswim_spread_forces_noalloc.
#include <algorithm>
#include <mutex>
#include <string>

#include "fixed_stencil.cuh"
#include "lbswim_device.cuh"
#include "lbswim_internal.h"

namespace lbswim {

constexpr int BIN = 4;  // spread bin edge, in lattice sites

struct Dims {
  int n[3];
  int nb[3];  // bins per axis
  long long N;
};

// Sites along axis a, for a thread's own axis (no local copy of the array).
__device__ __forceinline__ int dim_of(const Dims& D, int a) {
  return a == 0 ? D.n[0] : (a == 1 ? D.n[1] : D.n[2]);
}

// acc + a b: FP64 rounds the product and the sum on their own (the oracle's
// order, bit for bit); FP32 lets the compiler fuse them.
template <class T>
__device__ __forceinline__ T add_prod(T acc, T a, T b) {
  if constexpr (sizeof(T) == 8)
    return __dadd_rn(acc, __dmul_rn(a, b));
  else
    return acc + a * b;
}

template <class T>
__device__ __forceinline__ void stencil_setup(const Dims& D, const double r[3], int o[3],
                                              T phi[3][4]) {
  for (int d = 0; d < 3; ++d) {
    const double x0 = ceil(r[d] - 2.);
    o[d] = wrap_any((int)x0, D.n[d]);
#pragma unroll
    for (int i = 0; i < 4; ++i) phi[d][i] = peskin_delta<T>((T)(r[d] - (x0 + i)));
  }
}

// One record per dipole end: e = 2i is the tail, 2i + 1 the head.
template <class T>
__global__ void k_spread_bin(int nsw, const double* __restrict__ r, const double* __restrict__ nv,
                             double P, double l, Dims D, EndRecord<T>* __restrict__ ends,
                             unsigned* __restrict__ bin_count) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 2 * nsw) return;
  const int i = e >> 1;
  const bool head = e & 1;
  double rr[3], F[3];
  for (int a = 0; a < 3; ++a) {
    const double na = nv[nsw * a + i];
    rr[a] = head ? r[nsw * a + i] : __dsub_rn(r[nsw * a + i], __dmul_rn(na, l));
    F[a] = -P * na;
    if (head) F[a] *= -1.0;
  }
  EndRecord<T> rec;
  stencil_setup<T>(D, rr, rec.o, rec.phi);
  rec.pad = 0;
  for (int a = 0; a < 3; ++a) rec.F[a] = (T)F[a];
  ends[e] = rec;
  const int b = ((rec.o[0] / BIN) * D.nb[1] + rec.o[1] / BIN) * D.nb[2] + rec.o[2] / BIN;
  atomicAdd(bin_count + b, 1u);
}

template <class T>
__global__ void k_spread_scatter(int nends, const EndRecord<T>* __restrict__ ends, Dims D,
                                 unsigned* __restrict__ bin_count,
                                 const unsigned* __restrict__ bin_start, int* __restrict__ order) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nends) return;
  const int* o = ends[e].o;
  const int b = ((o[0] / BIN) * D.nb[1] + o[1] / BIN) * D.nb[2] + o[2] / BIN;
  // Counting back down leaves bin_count at zero for the next call.
  const unsigned slot = atomicSub(bin_count + b, 1u) - 1u;
  order[bin_start[b] + slot] = e;
}

// Put each bin's ends in increasing end order (bins hold a handful of ends).
__global__ void k_spread_sort(int nbins, const unsigned* __restrict__ bin_start,
                              int* __restrict__ order) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbins) return;
  const unsigned s = bin_start[b], t = bin_start[b + 1];
  for (unsigned i = s + 1; i < t; ++i) {
    const int v = order[i];
    unsigned j = i;
    while (j > s && order[j - 1] > v) {
      order[j] = order[j - 1];
      --j;
    }
    order[j] = v;
  }
}

__device__ __forceinline__ int candidate_bins(int x, int n, int out[4]) {
  int nb = 0;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int b = wrap_any(x - s, n) / BIN;
    bool seen = false;
    for (int q = 0; q < nb; ++q) seen |= (out[q] == b);
    if (!seen) out[nb++] = b;
  }
  return nb;
}

// Per-site gather.  accumulate = 0: F = sum (ZeroForce folded in); 1: F += sum.
template <class T>
__global__ void __launch_bounds__(256) k_spread_gather(Dims D, const EndRecord<T>* __restrict__ ends,
                                                       const unsigned* __restrict__ bin_start,
                                                       const int* __restrict__ order,
                                                       T* __restrict__ force, int accumulate) {
  const int z = blockIdx.x * 32 + threadIdx.x;
  const int y = blockIdx.y * 8 + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= D.n[2] || y >= D.n[1]) return;
  int bx[4], by[4], bz[4];
  const int nbx = candidate_bins(x, D.n[0], bx);
  const int nby = candidate_bins(y, D.n[1], by);
  const int nbz = candidate_bins(z, D.n[2], bz);
  T acc0 = T(0), acc1 = T(0), acc2 = T(0);
  bool hit = false;
  for (int i = 0; i < nbx; ++i)
    for (int j = 0; j < nby; ++j)
      for (int k = 0; k < nbz; ++k) {
        const int b = (bx[i] * D.nb[1] + by[j]) * D.nb[2] + bz[k];
        const unsigned s = bin_start[b], t = bin_start[b + 1];
        for (unsigned q = s; q < t; ++q) {
          const EndRecord<T>& e = ends[order[q]];
          const T wx = axis_weight(x, e.o[0], D.n[0], e.phi[0]);
          const T wy = axis_weight(y, e.o[1], D.n[1], e.phi[1]);
          const T wz = axis_weight(z, e.o[2], D.n[2], e.phi[2]);
          bool cover = true;
          if (D.n[0] >= 4) cover &= ((x - e.o[0] + D.n[0]) % D.n[0]) <= 3;
          if (D.n[1] >= 4) cover &= ((y - e.o[1] + D.n[1]) % D.n[1]) <= 3;
          if (D.n[2] >= 4) cover &= ((z - e.o[2] + D.n[2]) % D.n[2]) <= 3;
          if (!cover) continue;
          const T d3 = wx * wy * wz;
          acc0 += d3 * e.F[0];
          acc1 += d3 * e.F[1];
          acc2 += d3 * e.F[2];
          hit = true;
        }
      }
  const long long s = (long long)x * D.n[1] * D.n[2] + (long long)y * D.n[2] + z;
  if (!accumulate) {
    force[s] = acc0;
    force[D.N + s] = acc1;
    force[2 * D.N + s] = acc2;
  } else if (hit) {
    force[s] += acc0;
    force[D.N + s] += acc1;
    force[2 * D.N + s] += acc2;
  }
}

// ---- exclusive scan of bin counts (three passes, 4096 entries per CTA) -------
constexpr int SCAN_THREADS = 512, SCAN_PER_THREAD = 8, SCAN_TILE = SCAN_THREADS * SCAN_PER_THREAD;

__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned* warp_sums,
                                                         unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    unsigned w = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) warp_sums[lane] = w;
  }
  __syncthreads();
  total = warp_sums[(blockDim.x >> 5) - 1];
  const unsigned before = warp ? warp_sums[warp - 1] : 0u;
  __syncthreads();
  return before + x - v;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(const unsigned* __restrict__ in, int n,
                                                             unsigned* __restrict__ tile_sums) {
  __shared__ unsigned ws[32];
  const long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  unsigned s = 0;
  for (int i = 0; i < SCAN_PER_THREAD; ++i)
    if (base + i < n) s += in[base + i];
  unsigned total;
  block_exclusive_scan(s, ws, total);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_top(unsigned* __restrict__ tile_sums, int ntiles) {
  __shared__ unsigned ws[32];
  __shared__ unsigned carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < ntiles; base += 1024) {
    const int i = base + threadIdx.x;
    const unsigned v = i < ntiles ? tile_sums[i] : 0u;
    unsigned total;
    const unsigned ex = block_exclusive_scan(v, ws, total);
    if (i < ntiles) tile_sums[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply(const unsigned* __restrict__ in, int n,
                                                             const unsigned* __restrict__ tile_off,
                                                             unsigned* __restrict__ out,
                                                             unsigned grand_total) {
  __shared__ unsigned ws[32];
  const long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  unsigned v[SCAN_PER_THREAD];
  unsigned s = 0;
  for (int i = 0; i < SCAN_PER_THREAD; ++i) {
    v[i] = base + i < n ? in[base + i] : 0u;
    s += v[i];
  }
  unsigned total;
  unsigned run = block_exclusive_scan(s, ws, total) + tile_off[blockIdx.x];
  for (int i = 0; i < SCAN_PER_THREAD; ++i) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = grand_total;
}

// ---- tile-touch spreading ------------------------------------------------------
// Every dipole end is listed under each force tile its stencil touches; a tile's
// list is then put in end order, and one CTA per tile sums, for each of its
// sites, the covering ends of its list in that order.  The per-site order is a
// fixed function of the input, so the result is deterministic.
struct TileGrid {
  int T[3];   // tile edge per axis
  FastDiv by[3];  // division by it
  int h;      // sites beyond the tile (every side) that also need the force
  int nt[3];  // tiles per axis
};

// Tiles along one axis whose extended region holds one of the nodes o..o+3:
// the sites o-h .. o+3+h form one cyclic interval, so the tiles form the cyclic
// range first, first+1, ... (count of them, at most nt).  An interval that
// wraps past the end covers the tiles from `first` to the last one and from 0
// to the tile of its wrapped end; if those meet, it covers every tile.  o is a
// wrapped node (0 <= o < n, as records hold them) and h < n.
__device__ __forceinline__ void touched_range(int o, int n, FastDiv by, int h, int nt, int& first,
                                              int& count) {
  const int len = 4 + 2 * h;
  if (len >= n) {
    first = 0;
    count = nt;
    return;
  }
  const int a = o - h < 0 ? o - h + n : o - h, b = a + len - 1;
  first = (int)div_by((unsigned)a, by);
  if (b < n) {
    count = (int)div_by((unsigned)b, by) - first + 1;
  } else {
    const int last = (int)div_by((unsigned)(b - n), by);
    count = last >= first ? nt : (nt - first) + last + 1;
  }
}

__device__ __forceinline__ int node_after(int o, int j, int n) {
  int t = o + j;
  while (t >= n) t -= n;
  return t;
}

constexpr int REC_ENDS = 64, REC_THREADS = 3 * REC_ENDS;  // records of a block

// List end e under every tile of grid G whose extended region its stencil
// touches.  At most CAP ends are kept per tile; the count goes on, and `over` takes the
// later ones: (tile, the end's place among the tile's, number of the tile among the end's).
struct DropEnd {
  __device__ void operator()(int, unsigned, int) const {}
};
template <int CAP, class Over = DropEnd>
__device__ __forceinline__ void bucket_end(int e, const int o[3], const Dims& D, const TileGrid& G,
                                           unsigned* __restrict__ count, int* __restrict__ list,
                                           Over over = Over()) {
  int f[3], c[3];
  for (int a = 0; a < 3; ++a) touched_range(o[a], D.n[a], G.by[a], G.h, G.nt[a], f[a], c[a]);
  auto tile = [&](int i, int j, int k) {
    const int kx = f[0] + i < G.nt[0] ? f[0] + i : f[0] + i - G.nt[0];
    const int ky = f[1] + j < G.nt[1] ? f[1] + j : f[1] + j - G.nt[1];
    const int kz = f[2] + k < G.nt[2] ? f[2] + k : f[2] + k - G.nt[2];
    return (kx * G.nt[1] + ky) * G.nt[2] + kz;
  };
  // all of a pair of x tiles' counts in flight before the first is used
  const bool pairs = c[1] <= 2 && c[2] <= 2;
  for (int i0 = 0; i0 < c[0]; i0 += 2) {
    if (pairs) {
      unsigned slot[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (i0 + (q >> 2) < c[0] && ((q >> 1) & 1) < c[1] && (q & 1) < c[2])
          slot[q] = atomicAdd(count + tile(i0 + (q >> 2), (q >> 1) & 1, q & 1), 1u);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (i0 + (q >> 2) < c[0] && ((q >> 1) & 1) < c[1] && (q & 1) < c[2]) {
          const int i = i0 + (q >> 2), j = (q >> 1) & 1, k = q & 1, t = tile(i, j, k);
          if (slot[q] < (unsigned)CAP)
            list[(long long)t * CAP + slot[q]] = e;
          else
            over(t, slot[q], (i * c[1] + j) * c[2] + k);
        }
    } else {
      for (int i = i0; i < min(i0 + 2, c[0]); ++i)
        for (int j = 0; j < c[1]; ++j)
          for (int k = 0; k < c[2]; ++k) {
            const int t = tile(i, j, k);
            const unsigned slot = atomicAdd(count + t, 1u);
            if (slot < (unsigned)CAP)
              list[(long long)t * CAP + slot] = e;
            else
              over(t, slot, (i * c[1] + j) * c[2] + k);
          }
    }
  }
}

// Axis a of the FP32 record of one end (tail or head) of a swimmer at r with
// orientation n; returns |F_a| as float bits.
__device__ __forceinline__ unsigned record_axis32(double r, double n, bool head, double P,
                                                  double l, const Dims& D, int a,
                                                  EndRecord<float>& rec) {
  const double x = head ? r : __dsub_rn(r, __dmul_rn(n, l));
  double F = -P * n;
  if (head) F *= -1.0;
  int x0;
  float dr;
  stencil_axis(x, x0, dr);
  rec.o[a] = wrap_any(x0, dim_of(D, a));
  float w[4];
  peskin_weights4(dr, w);
#pragma unroll
  for (int j = 0; j < 4; ++j) rec.phi[a][j] = w[j];
  rec.F[a] = (float)F;
  if (a == 0) rec.pad = 0;
  return __float_as_uint(fmaxf(0.f, fabsf((float)F)));  // 0 for a NaN
}

// The swimmer arrays of one launch, each with its first block (of MOVE_SWIMMERS
// swimmers, or REC_ENDS ends) and its first end among all of the lattice's.
constexpr int LIST_ARRAYS = 8;
struct SwimmerPart {
  int n, block0, end0;
  double *r, *v, *nv;
  lbswim_common_params common;
  unsigned long long seed, step;
};
struct SwimmerList {
  int count;
  SwimmerPart part[LIST_ARRAYS];
};
__device__ __forceinline__ int part_of_block(const SwimmerList& w) {
  int m = 0;
  while (m + 1 < w.count && (int)blockIdx.x >= w.part[m + 1].block0) ++m;
  return m;
}

// Where the end records of a swimmer array go: the records, the largest |F| (FP32),
// and the buckets of the tiles of G.
template <class T>
struct RecordTarget {
  EndRecord<T>* ends;
  unsigned* max_f;
  TileGrid G;
  unsigned* count;
  int* list;
};

// The rest of a block's records e0, e0 + 1, ... (REC_ENDS of them, thread (q, a) for
// axis a of record q, a <= 2; ids offset by e_base): the largest force, the buckets
// and the copy to global memory.  Every thread of the block calls it; smax is 0
// before.  BUCKETS: the records may be listed in buckets.
template <bool BUCKETS>
__device__ __forceinline__ void finish_records32(int q, int a, int e0, int nends, int e_base,
                                                 unsigned big, EndRecord<float>* srec,
                                                 unsigned& smax, const Dims& D,
                                                 const RecordTarget<float>& to) {
  // non-negative floats order like their bit patterns: a warp's largest, then
  // one shared-memory atomic per warp
  big = __reduce_max_sync(0xffffffffu, big);
  if ((threadIdx.x & 31) == 0 && big) atomicMax(&smax, big);
  __syncthreads();
  if (BUCKETS && a == 0 && e0 + q < nends && to.count)
    bucket_end<SLAB_BUCKET_CAP>(e_base + e0 + q, srec[q].o, D, to.G, to.count, to.list);
  if (threadIdx.x == 0) atomicMax(to.max_f, smax);
  const int words = min(REC_ENDS, nends - e0) * (int)(sizeof(EndRecord<float>) / 4);
  const unsigned* src = reinterpret_cast<const unsigned*>(srec);
  unsigned* dst = reinterpret_cast<unsigned*>(to.ends + e0);
  for (int w = threadIdx.x; w < words; w += blockDim.x) dst[w] = src[w];
}

// One record per dipole end: e = 2i is the tail, 2i + 1 the head; a thread per
// (end, axis).  Records are assembled in shared memory and written out as one
// contiguous block.  The stencil origin comes from the bits of the position
// (stencil_axis) and the four weights from one square root (peskin_weights4),
// like the FP32 interpolation.
__device__ __forceinline__ void end_records_block(int blk, int nsw, const double* __restrict__ r,
                                                  const double* __restrict__ nv, double P,
                                                  double l, const Dims& D, int e_base,
                                                  const RecordTarget<float>& to) {
  __shared__ EndRecord<float> srec[REC_ENDS];
  __shared__ unsigned smax;
  if (threadIdx.x == 0) smax = 0u;
  __syncthreads();
  const int q = threadIdx.x % REC_ENDS, a = threadIdx.x / REC_ENDS;
  const int e0 = blk * REC_ENDS, e = e0 + q, nends = 2 * nsw;
  unsigned big = 0u;
  if (e < nends) {
    const long long at = (long long)nsw * a + (e >> 1);
    big = record_axis32(r[at], nv[at], e & 1, P, l, D, a, srec[q]);
  }
  finish_records32<true>(q, a, e0, nends, e_base, big, srec, smax, D, to);
}

__global__ void __launch_bounds__(REC_THREADS) k_end_records(const __grid_constant__ SwimmerList w,
                                                             Dims D, RecordTarget<float> to) {
  const SwimmerPart& p = w.part[part_of_block(w)];
  to.ends += p.end0;
  end_records_block(blockIdx.x - p.block0, p.n, p.r, p.nv, p.common.P, p.common.l, D, p.end0, to);
}

// Slab buckets of recorded ends (the slab shape changed since they were recorded).
__global__ void k_bucket_ends(int nends, const EndRecord<float>* __restrict__ ends, Dims D,
                              TileGrid G, unsigned* __restrict__ count, int* __restrict__ list) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nends) return;
  const int o[3] = {ends[e].o[0], ends[e].o[1], ends[e].o[2]};
  bucket_end<SLAB_BUCKET_CAP>(e, o, D, G, count, list);
}

template <int PASS>
__global__ void k_touch(int nends, const EndRecord<double>* __restrict__ ends, Dims D, TileGrid G,
                        unsigned* __restrict__ count, const unsigned* __restrict__ start,
                        int* __restrict__ list) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nends) return;
  const int ox = ends[e].o[0], oy = ends[e].o[1], oz = ends[e].o[2];
  int fx, cx, fy, cy, fz, cz;
  touched_range(ox, D.n[0], G.by[0], G.h, G.nt[0], fx, cx);
  touched_range(oy, D.n[1], G.by[1], G.h, G.nt[1], fy, cy);
  touched_range(oz, D.n[2], G.by[2], G.h, G.nt[2], fz, cz);
  for (int i = 0; i < cx; ++i) {
    const int kx = fx + i < G.nt[0] ? fx + i : fx + i - G.nt[0];
    for (int j = 0; j < cy; ++j) {
      const int ky = fy + j < G.nt[1] ? fy + j : fy + j - G.nt[1];
      for (int k = 0; k < cz; ++k) {
        const int kz = fz + k < G.nt[2] ? fz + k : fz + k - G.nt[2];
        const int t = (kx * G.nt[1] + ky) * G.nt[2] + kz;
        if (PASS == 0) {
          atomicAdd(count + t, 1u);
        } else {
          // counting back down leaves the counts at zero for the next call
          const unsigned slot = atomicSub(count + t, 1u) - 1u;
          list[start[t] + slot] = e;
        }
      }
    }
  }
}

// Exclusive-scan finish that also writes the grand total to out[n].
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply_total(
    const unsigned* __restrict__ in, int n, const unsigned* __restrict__ tile_off,
    unsigned* __restrict__ out) {
  __shared__ unsigned ws[32];
  const long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  unsigned v[SCAN_PER_THREAD];
  unsigned s = 0;
  for (int i = 0; i < SCAN_PER_THREAD; ++i) {
    v[i] = base + i < n ? in[base + i] : 0u;
    s += v[i];
  }
  unsigned total;
  unsigned run = block_exclusive_scan(s, ws, total) + tile_off[blockIdx.x];
  for (int i = 0; i < SCAN_PER_THREAD; ++i) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
    if (base + i == n - 1) out[n] = run;
  }
}

// ---- force spreading of FP64 lattices -------------------------------------------
// Force tiles of 4 (x) x 8 (y) x 32 (z) sites.  The end records list every end
// under the tiles its stencil touches, in buckets of FT_CAP and, past those, chains
// (TileChains).  Two kernels sum them:
//  * k_force_fixed (default): the (end, node) contributions are integers of 72 (256 ends)
//    to 84 bits below the tile's largest force, added as three words with shared-memory
//    atomics that return nothing, and converted once.  All 32 lanes work on the nodes of
//    an end.  Integer sums do not depend on their order.
//  * k_force_tile (LBSWIM_COMPAT_EXACT_F64, and suspensions too dense for
//    buckets): every site adds the ends that cover it in end order,
//    ((phi_x phi_y) phi_z) F as the reference does (SwimmerArray.cu:64-73).  A
//    row's 32 lanes have half an end each on average and run as long as the one
//    with most, on the narrow FP64 pipe.
constexpr int FT_X = 4, FT_Y = 8, FT_Z = 32, FT_THREADS = 256, FT_CAP = 256;

// Entries FT_CAP, FT_CAP + 1, ... of a tile hang on its 32 chains in turn, so that the
// lanes of a warp walk them side by side and a tile with many ends (swimmers in a
// cluster) takes its own and no others: 256^3 with 65,536 swimmers in a sixteenth of the
// box, where some tiles hold 500 ends, took 24 ms while such a tile went through all
// 131,072, and 950 us when every tile's ends were listed by a counting sort.  An entry is
// end * touch + the tile's number among the end's; chain c has
// (count - FT_CAP + 31 - c) / 32 of them, so heads left over from before do not matter.
struct TileChains {
  int* head;  // [tiles][32]; null: no tile can have more than FT_CAP ends
  int* next;  // [ends * touch]
  int touch;  // tiles an end can touch
  FastDiv by_touch;
  int* ids;  // exact mode: [2][half] the ends of tiles with more, and in order
  long long half;
  unsigned long long* id_end;  // ids in use
};
struct ChainEnd {
  TileChains ch;
  int e;
  __device__ void operator()(int t, unsigned slot, int i) const {
    const int entry = e * ch.touch + i;
    ch.next[entry] = atomicExch(ch.head + 32 * t + (int)(slot & 31u), entry);
  }
};
static_assert(FT_CAP % 32 == 0, "entry FT_CAP hangs on chain 0");
// The end of the entry after `at` on this lane's chain (at < 0: the first one), which
// becomes `at`.
__device__ __forceinline__ int chain_step(const TileChains& ch, int tile, int& at) {
  at = at < 0 ? ch.head[32 * tile + (threadIdx.x & 31)] : ch.next[at];
  return (int)div_by((unsigned)at, ch.by_touch);
}

// Axis a of the record of an end (tail or head) of a swimmer at r, n.  FIXED: the
// weights are integers in units of 2^-63 (fixed_weights4) in place of doubles, and
// `lost` is set when the coordinate is not a number; otherwise they are the
// reference's delta per node.
template <bool FIXED>
__device__ __forceinline__ void record_axis64(double r, double n, bool head, double P,
                                                  double l, const Dims& D, int a,
                                                  EndRecord<double>& rec, unsigned& lost) {
  const double x = head ? r : __dsub_rn(r, __dmul_rn(n, l));
  double F = -P * n;
  if (head) F *= -1.0;
  const double x0 = ceil(x - 2.);
  rec.o[a] = wrap_any((int)x0, dim_of(D, a));
  rec.F[a] = F;
  if (!FIXED) {
#pragma unroll
    for (int j = 0; j < 4; ++j) rec.phi[a][j] = peskin_delta<double>(x - (x0 + j));
    return;
  }
  long long w[4];
  const double dr = x - x0;
  if (dr >= 1.0 && dr <= 2.0) {
    fixed_weights4(dr, w);
  } else {  // a coordinate beyond 2^52, or not a number
    for (int j = 0; j < 4; ++j) w[j] = (long long)(peskin_delta<double>(x - (x0 + j)) * 0x1p63);
    if (!(dr >= -4.0 && dr <= 4.0)) lost = 1u;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) rec.phi[a][j] = bits_double((unsigned long long)w[j]);
}

// The rest of a block's records e0, e0 + 1, ... (ENDS of them, thread (q, a)
// for axis a of record q, a <= 2): the force of lost ends, the buckets and the copy to
// global memory.  Every thread of the block calls it.
constexpr int REC64_ENDS = 64, REC64_THREADS = 3 * REC64_ENDS;
template <bool FIXED, bool BUCKETS, int ENDS>
__device__ __forceinline__ void finish_records64(int q, int a, int e0, int nends,
                                                 EndRecord<double>* srec, const unsigned* lost,
                                                 const Dims& D, const RecordTarget<double>& to,
                                                 const TileChains& ch) {
  __syncthreads();
  if (a == 0 && e0 + q < nends) {
    if (FIXED && lost[q])  // the force of a lost end is not a number
      for (int c = 0; c < 3; ++c) srec[q].F[c] = bits_double(0x7ff8000000000000ull);
    if (BUCKETS && to.count)
      bucket_end<FT_CAP>(e0 + q, srec[q].o, D, to.G, to.count, to.list, ChainEnd{ch, e0 + q});
  }
  __syncthreads();
  const int words = min(ENDS, nends - e0) * (int)(sizeof(EndRecord<double>) / 8);
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(srec);
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(to.ends + e0);
  for (int w = threadIdx.x; w < words; w += blockDim.x) dst[w] = src[w];
}

// One thread per (end, axis), 64 ends per block: the axes' chains of FP64
// operations run side by side.  e = 2i is the tail, 2i + 1 the head.
template <bool FIXED>
__global__ void __launch_bounds__(REC64_THREADS) k_end_records_f64(
    int nsw, const double* __restrict__ r, const double* __restrict__ nv, double P, double l,
    Dims D, RecordTarget<double> to, TileChains ch) {
  __shared__ EndRecord<double> srec[REC64_ENDS];
  __shared__ unsigned lost[REC64_ENDS];
  if (ch.id_end && blockIdx.x == 0 && threadIdx.x == 0) *ch.id_end = 0ull;
  const int q = threadIdx.x % REC64_ENDS, a = threadIdx.x / REC64_ENDS;
  const int nends = 2 * nsw, e0 = blockIdx.x * REC64_ENDS, e = e0 + q;
  if (a == 0) lost[q] = 0u;
  __syncthreads();
  if (e < nends) {
    const int i = e >> 1;
    const bool head = e & 1;
    const double na = nv[(long long)nsw * a + i], ra = r[(long long)nsw * a + i];
    record_axis64<FIXED>(ra, na, head, P, l, D, a, srec[q], lost[q]);
    if (a == 0) srec[q].pad = 0;
  }
  finish_records64<FIXED, true, REC64_ENDS>(q, a, e0, nends, srec, lost, D, to, ch);
}
static_assert(sizeof(EndRecord<double>) % 8 == 0, "records are copied as 64-bit words");

// The ends rec(0), ..., rec(cnt - 1) added to every site of a tile in that order.
// A warp walks z rows: a ballot picks the ends covering a row, each lane then
// collects those that cover its own site and adds them.
template <bool FIXED, class Rec>
__device__ __forceinline__ void force_gather(const Dims& D, int kx, int ky, int kz, int cnt,
                                             Rec rec, double* __restrict__ force, int accumulate) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto phi = [](const EndRecord<double>& e, int a, int i) {
    return FIXED ? (double)(long long)double_bits(e.phi[a][i]) * 0x1p-63 : e.phi[a][i];
  };
  const int z = kz * FT_Z + lane;
  const bool zval = z < D.n[2];
  // no axis shorter than a stencil: one node of an end lands on a site
  const bool single = D.n[0] >= 4 && D.n[1] >= 4 && D.n[2] >= 4;
  for (int row = warp; row < FT_X * FT_Y; row += blockDim.x / 32) {
    const int x = kx * FT_X + row / FT_Y, y = ky * FT_Y + row % FT_Y;
    if (x >= D.n[0] || y >= D.n[1]) continue;
    const long long s = (long long)x * D.n[1] * D.n[2] + (long long)y * D.n[2] + z;
    // the sums start from the base force and add the ends in end order, as
    // the oracle's serial spreading does
    double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
    if (accumulate && zval) {
      acc0 = force[s];
      acc1 = force[D.N + s];
      acc2 = force[2 * D.N + s];
    }
    bool hit = false;
    for (int base = 0; base < cnt; base += 32) {
      const int q = base + lane;
      bool covers = false;
      if (q < cnt) {
        const EndRecord<double>& e = rec(q);
        covers = covers_axis(x, e.o[0], D.n[0]) && covers_axis(y, e.o[1], D.n[1]);
      }
      const unsigned m = __ballot_sync(0xffffffffu, covers);  // every lane takes part
      unsigned mine = 0u;
      if (zval)
        for (unsigned mm = m; mm; mm &= mm - 1) {
          const int b = __ffs(mm) - 1;
          if (covers_axis(z, rec(base + b).o[2], D.n[2])) mine |= 1u << b;
        }
      hit |= mine != 0u;
      for (; mine; mine &= mine - 1) {
        const EndRecord<double>& e = rec(base + __ffs(mine) - 1);
        if (single) {
          int i = x - e.o[0], j = y - e.o[1], k = z - e.o[2];
          i += i < 0 ? D.n[0] : 0;
          j += j < 0 ? D.n[1] : 0;
          k += k < 0 ? D.n[2] : 0;
          const double px = phi(e, 0, i), py = phi(e, 1, j), pz = phi(e, 2, k);
          acc0 = __dadd_rn(acc0, end_contrib(px, py, pz, e.F[0]));
          acc1 = __dadd_rn(acc1, end_contrib(px, py, pz, e.F[1]));
          acc2 = __dadd_rn(acc2, end_contrib(px, py, pz, e.F[2]));
          continue;
        }
        // node by node in (i, j, k) order, as AccumulateDeltaForce adds them
        // (several nodes land on one site when an axis is shorter than 4)
        for (int i = 0; i < 4; ++i) {
          if (wrap_any(e.o[0] + i, D.n[0]) != x) continue;
          for (int j = 0; j < 4; ++j) {
            if (wrap_any(e.o[1] + j, D.n[1]) != y) continue;
            for (int k = 0; k < 4; ++k) {
              if (wrap_any(e.o[2] + k, D.n[2]) != z) continue;
              const double px = phi(e, 0, i), py = phi(e, 1, j), pz = phi(e, 2, k);
              acc0 = __dadd_rn(acc0, end_contrib(px, py, pz, e.F[0]));
              acc1 = __dadd_rn(acc1, end_contrib(px, py, pz, e.F[1]));
              acc2 = __dadd_rn(acc2, end_contrib(px, py, pz, e.F[2]));
            }
          }
        }
      }
    }
    if (zval && (!accumulate || hit)) {
      force[s] = acc0;
      force[D.N + s] = acc1;
      force[2 * D.N + s] = acc2;
    }
  }
}

// The ends of a tile in end order, by rank, then force_gather.  start: counting-
// sorted lists [start[tile], start[tile + 1]) (with `sorted` as scratch for the
// long ones); null: buckets, whose count is zeroed for the next call, and chains.
__global__ void __launch_bounds__(FT_THREADS) k_force_tile(
    Dims D, TileGrid G, const EndRecord<double>* __restrict__ ends,
    const unsigned* __restrict__ start, unsigned* __restrict__ count,
    const int* __restrict__ list, int* __restrict__ sorted, TileChains ch,
    double* __restrict__ force, int accumulate) {
  __shared__ EndRecord<double> srec[FT_CAP];
  __shared__ int skey[FT_CAP];
  __shared__ unsigned long long place;
  const int tile = blockIdx.x;
  const int kz = tile % G.nt[2], ky = (tile / G.nt[2]) % G.nt[1], kx = tile / (G.nt[1] * G.nt[2]);
  const int tid = threadIdx.x;
  const int cnt = (int)(start ? start[tile + 1] - start[tile] : count[tile]);
  const int* ids = list + (start ? (long long)start[tile] : (long long)tile * FT_CAP);
  int* in_order = start ? sorted + start[tile] : nullptr;
  const bool in_smem = cnt <= FT_CAP;
  if (in_smem) {
    for (int q = tid; q < cnt; q += FT_THREADS) skey[q] = ids[q];
    __syncthreads();
    for (int q = tid; q < cnt; q += FT_THREADS) srec[rank_of(skey[q], skey, cnt)] = ends[skey[q]];
  } else {
    // more ends than fit: order them in global scratch and read records from there
    if (!start) {
      if (tid == 0) place = atomicAdd(ch.id_end, (unsigned long long)cnt);
      __syncthreads();
      int* all = ch.ids + place;
      in_order = all + ch.half;
      for (int q = tid; q < FT_CAP; q += FT_THREADS) all[q] = ids[q];
      if (tid < 32)
        for (int q = FT_CAP + tid, at = -1; q < cnt; q += 32) all[q] = chain_step(ch, tile, at);
      __syncthreads();
      ids = all;
    }
    for (int q = tid; q < cnt; q += FT_THREADS) {
      const int k = ids[q];
      int r = 0;
      for (int j = 0; j < cnt; ++j) r += ids[j] < k;
      in_order[r] = k;
    }
  }
  __syncthreads();
  if (!start && tid == 0) count[tile] = 0u;  // every thread has read it
  auto rec = [&](int q) -> const EndRecord<double>& {
    return in_smem ? srec[q] : ends[in_order[q]];
  };
  force_gather<false>(D, kx, ky, kz, cnt, rec, force, accumulate);
}

// Words of the fixed-point sums of a tile, [3 components][3 words][sites]: rows
// are padded by 4 and planes by 16 words, so that the 32 nodes that a warp adds
// at once (2 planes x 4 rows x 4 columns) fall into 32 banks.
constexpr int FF_ROW = FT_Z + 4, FF_PLANE = FT_Y * FF_ROW + 16, FF_SITES = FT_X * FF_PLANE;
constexpr int FF_CHUNK = 32;  // ends staged at a time, at most
static_assert(FF_ROW % 32 == 4 && FF_PLANE % 32 == 16 && FF_SITES % 4 == 0, "bank layout");

// The sums of a tile are numbers hi 2^(2 low) + mid 2^low + lo, hi signed.  A contribution
// is cut into two unsigned digits of `low` bits and a signed top, small enough that all
// contributions to a site, `most` of them, keep each word within 32 bits: 84 bits in all
// for 16 of them, 81 for 32, 72 for 256.  Past 256 the digits have the 26 bits that
// 32 contributions and a carried rest leave room for, and their carries move up after
// each batch of ends: 73 bits for 2048, 61 for 2^23.  (Stencil nodes of an end can meet on
// a site, 2^log2_fold of them: 64 on a lattice of one site, which has 25 bits.)
struct SumWords {
  int low, bits;
};
__device__ __forceinline__ SumWords sum_words(long long most, int log2_fold) {
  const int n = most > 1 ? 64 - __clzll(most - 1) : 0;  // most <= 2^n
  const int top = max(min(28, 32 - n), 2), low = n <= 8 ? top : (log2_fold == 6 ? 25 : 26);
  return SumWords{low, 2 * low + top};
}
// The digits of v 2^32 / 2^m, |v| < 2^60 and m < 96, toward minus infinity.
__device__ __forceinline__ void cut_words(long long v, int m, int low, unsigned mask, unsigned& lo,
                                          unsigned& mid, int& hi) {
  const unsigned v0 = (unsigned)v, v1 = (unsigned)(v >> 32), sg = (unsigned)((int)v1 >> 31);
  const bool one = m >= 32, two = m >= 64;  // whole words of the shift
  const unsigned a0 = two ? v1 : (one ? v0 : 0u), a1 = two ? sg : (one ? v1 : v0),
                 a2 = one ? sg : v1;
  const unsigned x0 = __funnelshift_r(a0, a1, m), x1 = __funnelshift_r(a1, a2, m),
                 x2 = __funnelshift_r(a2, sg, m);
  lo = x0 & mask;
  mid = __funnelshift_r(x0, x1, low) & mask;
  hi = (int)__funnelshift_r(x1, x2, 2 * low);  // 2 low is 48 to 56
}
// The double nearest to a sum in the units of k (2^(k - 1082), fixed_site.cuh).
__device__ __forceinline__ double words_to_double(unsigned lo, unsigned mid, int hi, int low,
                                                  int k) {
  const unsigned long long l = (unsigned long long)mid * (1u << low) + lo;
  const long long t = (long long)hi * (1 << (2 * low - 32)) + hi_word(l);  // the sum / 2^32
  const unsigned long long sg = (unsigned long long)(t >> 63);
  const unsigned c0 = ((unsigned)l ^ (unsigned)sg) + ((unsigned)sg & 1u);
  const unsigned long long a = ((unsigned long long)t ^ sg) + (c0 == 0u ? sg & 1u : 0u);
  // the top word that is not zero, and the two after it
  const bool b1 = hi_word(a) == 0u, b2 = a == 0ull;
  const unsigned a1 = (unsigned)a;
  const unsigned u2 = b2 ? c0 : (b1 ? a1 : hi_word(a)), u1 = b2 ? 0u : (b1 ? c0 : a1),
                 u0 = b1 ? 0u : c0;
  const int lz = leading_zeros(u2);
  const unsigned h = __funnelshift_l(u1, u2, lz), g = __funnelshift_l(u0, u1, lz);
  const unsigned long long m = (((unsigned long long)h << 32) | g) >> 1;
  const bool below = ((u0 << (lz & 31)) | (g & 1u)) != 0u;
  const double r = round_to_double(m | (below ? 1u : 0u), lz + (b2 ? 32 : (b1 ? 0 : -32)), k);
  return u2 == 0u ? 0.0 : bits_double(double_bits(r) | (sg & 0x8000000000000000ull));
}

// Default FP64 spreading (see above).  A record's weights and force components are
// taken as 62-bit mantissas with exponents of their own, so a contribution keeps its
// digits however small its factors; the unit of a component's sums lies 74 bits below
// the largest such component among a tile's 256 ends, 83 below 32 ends' (sum_words).
// In a unit that all components and tiles shared, 60 bits below the largest force,
// swimmers aligned with an axis lost the digits of the other components.  Tiles with
// forces that are not finite, or below 2^-894, take FP64 arithmetic in end order.
// Bound by the integer pipe where most tiles have ends (16,000 warp instructions a
// tile, a quarter of them in the conversions), so a thread's sites differ in x alone and
// the record loads run under the zeroing: AddForces at 256^3 with 65,536 swimmers 313 us,
// against 840 in FP64 by site; 65x47x90 with 1074 20 against 76.  Up to two tiles
// to an SM, the chain of a block's phases bounds the launch: 512 threads shorten
// each, and the list is read with its count (onto a force 24^3 18.5 -> 14.5 us, 64^3 22.6 ->
// 19.5); with more tiles they cost occupancy (64x64x80, 384 tiles, 23.0 -> 23.4; 80^3 26.7
// -> 28.6; 256^3 316 -> 380 alone), and of a few ends without buckets each tile first
// picks its own (256^3 with 32 swimmers 199 -> 88 us).
template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_force_fixed(
    Dims D, TileGrid G, const EndRecord<double>* __restrict__ ends, int nends,
    unsigned* __restrict__ count, const int* __restrict__ list, TileChains ch,
    double* __restrict__ force, int accumulate) {
  __shared__ __align__(16) unsigned sums[9 * FF_SITES];
  __shared__ Digits dig[15][FF_CHUNK];  // mantissas of 12 weights, 3 force components per end
  __shared__ unsigned char shift[12][FF_CHUNK];       // binades of a weight below 1/2 ...
  __shared__ unsigned short exponent[3][FF_CHUNK];    // ... and the force's biased exponent
  __shared__ int org[3][FF_CHUNK];
  __shared__ unsigned top_f[3];  // largest high word of |F| (1 for what has none)
  constexpr int WARPS = THREADS / 32;
  static_assert(WARPS % FT_Y == 0 && FF_CHUNK == 32, "the mappings below");
  const int tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kz = tile % G.nt[2], ky = (tile / G.nt[2]) % G.nt[1], kx = tile / (G.nt[1] * G.nt[2]);
  // without buckets (DIRECT_ENDS_F64 ends at most) a tile goes through all of them, or,
  // where many tiles have none, picks its own
  constexpr bool PICK = THREADS == FT_THREADS;
  __shared__ int own[DIRECT_ENDS_F64 + 1];
  int cnt = count ? (int)count[tile] : nends;
  const long long s0 = (long long)tile * FT_CAP;
  // entry of a chunk that this lane stages; few tiles read it before the count is
  // known (the bucket has FT_CAP > lane of them), many tiles are mostly empty
  constexpr bool EARLY = THREADS > FT_THREADS;
  int mine = lane;
  if (EARLY && count) mine = list[s0 + lane];
  if (tid < 3) top_f[tid] = 0u;
  if (PICK && !count && warp == 0) {
    int n = 0;
    for (int base = 0; base < DIRECT_ENDS_F64; base += 32) {
      const int e = base + lane;
      bool in = e < nends;
      if (in)
        for (int a = 0; a < 3; ++a) {
          int f, c;
          touched_range(ends[e].o[a], D.n[a], G.by[a], 0, G.nt[a], f, c);
          int k = (a == 0 ? kx : (a == 1 ? ky : kz)) - f;
          in = in && (k < 0 ? k + G.nt[a] : k) < c;
        }
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) own[n + __popc(m & ((1u << lane) - 1u))] = e;
      n += __popc(m);
    }
    if (lane == 0) own[DIRECT_ENDS_F64] = n;
  }
  // contributions an end can make to one site: stencil nodes that fold onto it
  int log2_fold = 0;
  for (int a = 0; a < 3; ++a) log2_fold += D.n[a] >= 4 ? 0 : (D.n[a] == 1 ? 2 : 1);
  const int batch = max(FF_CHUNK >> log2_fold, 1);
  __syncthreads();
  if (tid == 0 && count) count[tile] = 0u;  // every thread has read it
  const bool picked = PICK && !count;
  if (picked) cnt = own[DIRECT_ENDS_F64];
  // the q-th end of the tile; those past the bucket one after another, from `at` = -1 on
  auto entry = [&](int q, int& at) {
    if (q >= FT_CAP) return chain_step(ch, tile, at);
    return count ? list[s0 + q] : (picked ? own[q] : q);
  };
  int at = -1;
  const int z0 = kz * FT_Z, y0 = ky * FT_Y, x0 = kx * FT_X;
  if (cnt == 0) {
    if (!accumulate)
      for (int t = tid; t < FT_X * FT_Y * FT_Z; t += THREADS) {
        const int z = z0 + t % FT_Z, y = y0 + (t / FT_Z) % FT_Y, x = x0 + t / (FT_Z * FT_Y);
        if (x >= D.n[0] || y >= D.n[1] || z >= D.n[2]) continue;
        const long long s = ((long long)x * D.n[1] + y) * D.n[2] + z;
        force[s] = force[D.N + s] = force[2 * D.N + s] = 0.0;
      }
    return;
  }
  auto in_order = [&]() {
    auto rec = [&](int q) -> const EndRecord<double>& { return ends[q]; };
    force_gather<true>(D, kx, ky, kz, nends, rec, force, accumulate);
  };
  auto f_word = [](double F) {
    const unsigned long long b = double_bits(F);
    return (hi_word(b) & 0x7fffffffu) | ((unsigned)b != 0u ? 1u : 0u);
  };
  // the words of a chunk's records: lane q has end q, a warp every WARPS-th word;
  // their way here is covered by the zeroing, or by the chunk before
  constexpr int WORDS = (18 + WARPS - 1) / WARPS;
  unsigned long long word[WORDS];
  auto fetch = [&](int m) {
    if (lane >= m) return;
    const EndRecord<double>& e = ends[mine];
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
      const int w = warp + i * WARPS;
      if (w < 12) word[i] = double_bits(e.phi[w >> 2][w & 3]);
      else if (w < 15) word[i] = double_bits(e.F[w - 12]);
      else if (w < 18) word[i] = (unsigned)e.o[w - 15];
    }
  };
  if (!EARLY && lane < cnt) mine = entry(lane, at);
  fetch(min(FF_CHUNK, cnt));
  // the later chunks' forces; every warp walks the chains
  for (int q = FF_CHUNK + lane, ahead = -1; q < cnt; q += FF_CHUNK) {
    const bool turn = (q / FF_CHUNK) % WARPS == warp;
    if (q < FT_CAP && !turn) continue;
    const EndRecord<double>& e = ends[entry(q, ahead)];
    if (turn)
      for (int c = 0; c < 3; ++c) atomicMax(top_f + c, f_word(e.F[c]));
  }
  for (int i = tid; i < 9 * FF_SITES / 4; i += THREADS)
    reinterpret_cast<uint4*>(sums)[i] = make_uint4(0u, 0u, 0u, 0u);
  const long long most = (long long)cnt << log2_fold;
  const SumWords sw = sum_words(most, log2_fold);
  const unsigned mask = (1u << sw.low) - 1u;
  const int jy = (lane >> 2) & 3, jz = lane & 3;
  int kf[3];  // |F_c| < 2^(kf[c] - 1022)
  for (int base = 0; base < cnt; base += FF_CHUNK) {
    const int m = min(FF_CHUNK, cnt - base);
    const int next = base + FF_CHUNK + lane;
    if (next < cnt) mine = entry(next, at);
    if (base) __syncthreads();  // the chunk before has been added
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
      const int w = warp + i * WARPS;  // uniform in the warp
      const unsigned long long b = lane < m ? word[i] : 0ull;
      if (w < 12) {
        // weights are not negative but for rounding
        const unsigned long long p = (long long)b > 0 ? b : 0ull;
        const int e = p ? max(__clzll((long long)p) - 2, 0) : 0;
        dig[w][lane] = digits((long long)(p << e));
        shift[w][lane] = (unsigned char)e;
      } else if (w < 15) {
        const int e = (int)((hi_word(b) >> 20) & 0x7ffu);
        const long long v =
            e ? (long long)(((b << 11) | 0x8000000000000000ull) >> 2) : 0ll;
        const long long sg = (long long)b >> 63;
        dig[w][lane] = digits((v ^ sg) - sg);
        exponent[w - 12][lane] = (unsigned short)e;
        if (base == 0) {
          const unsigned f = __reduce_max_sync(0xffffffffu, f_word(bits_double(b)));
          if (lane == 0) atomicMax(top_f + (w - 12), f);
        }
      } else if (w < 18) {
        org[w - 15][lane] = (int)b;
      }
    }
    fetch(min(FF_CHUNK, cnt - base - FF_CHUNK));
    __syncthreads();
    if (base == 0) {
      bool range = true;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        kf[c] = (int)(top_f[c] >> 20);
        range = range && (top_f[c] == 0u || (kf[c] >= FIXED_MIN_K && kf[c] <= FIXED_MAX_K));
      }
      if (!range) {  // uniform in the block
        in_order();
        return;
      }
    }
    for (int first = 0; first < m; first += batch) {
      for (int q = first + warp; q < min(m, first + batch); q += WARPS) {
        const int ly = node_after(org[1][q], jy, D.n[1]) - y0;
        const int lz = node_after(org[2][q], jz, D.n[2]) - z0;
        const bool in_yz = (unsigned)ly < (unsigned)FT_Y && (unsigned)lz < (unsigned)FT_Z;
        if (!in_yz) continue;
        const Digits wyz = digits(mul_hi(dig[4 + jy][q], dig[8 + jz][q]) << 2);
        const int eyz = 93 - sw.bits + shift[4 + jy][q] + shift[8 + jz][q];
        Digits F[3];  // (the sums' atomics would have them read again for each node)
        int eF[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          F[c] = dig[12 + c][q];
          eF[c] = kf[c] - exponent[c][q] + eyz;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int ix = (lane >> 4) + 2 * h;
          const int lx = node_after(org[0][q], ix, D.n[0]) - x0;
          if ((unsigned)lx >= (unsigned)FT_X) continue;
          const Digits w = digits(mul_hi(dig[ix][q], wyz) << 2);
          const int ew = shift[ix][q];
          unsigned* sum = sums + lx * FF_PLANE + ly * FF_ROW + lz;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            unsigned lo, mid;
            int hi;
            cut_words(mul_hi(w, F[c]), min(ew + eF[c], 95), sw.low, mask, lo, mid, hi);
            atomicAdd(sum + (3 * c) * FF_SITES, lo);
            atomicAdd(sum + (3 * c + 1) * FF_SITES, mid);
            atomicAdd(reinterpret_cast<int*>(sum + (3 * c + 2) * FF_SITES), hi);
          }
        }
      }
      if (most > 256 && (first + batch < m || base + FF_CHUNK < cnt)) {
        __syncthreads();
        for (int i = tid; i < FF_SITES; i += THREADS)
          for (int c = 0; c < 3; ++c) {
            unsigned* w = sums + 3 * c * FF_SITES + i;
            const unsigned mid = w[FF_SITES] + (w[0] >> sw.low);
            w[0] &= mask;
            w[FF_SITES] = mid & mask;
            w[2 * FF_SITES] += mid >> sw.low;
          }
        if (first + batch < m) __syncthreads();
      }
    }
  }
  __syncthreads();
  // a warp has one row of sites in every (WARPS / FT_Y)-th plane
  const int ly = warp % FT_Y, y = y0 + ly, z = z0 + lane;
  if (y >= D.n[1] || z >= D.n[2]) return;
#pragma unroll
  for (int i = 0; i < FT_X * FT_Y / WARPS; ++i) {
    const int lx = warp / FT_Y + i * (WARPS / FT_Y), x = x0 + lx;
    if (x >= D.n[0]) break;
    const unsigned* sum = sums + lx * FF_PLANE + ly * FF_ROW + lane;
    const long long s = ((long long)x * D.n[1] + y) * D.n[2] + z;
    unsigned w[9], any = 0u;
#pragma unroll
    for (int j = 0; j < 9; ++j) any |= w[j] = sum[j * FF_SITES];
    const bool some = __any_sync(__activemask(), any != 0u);  // else the row is empty
    if (accumulate && !some) continue;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double f = 0.0;
      if (some)
        f = words_to_double(w[3 * c], w[3 * c + 1], (int)w[3 * c + 2], sw.low, kf[c] + 58 - sw.bits);
      if (accumulate && f == 0.0) continue;
      force[c * D.N + s] = accumulate ? force[c * D.N + s] + f : f;
    }
  }
}

// ---- Move kernels -----------------------------------------------------------
// Stencil nodes and Peskin weights of position r (interp.cu:23-30).  FP64: the
// reference's arithmetic (a delta per node), for exact mode and for points
// given by the caller; FP32: one FP64 difference per axis and one square root
// for its four weights (GB300's FP64 pipe is narrow).
template <class T>
__device__ __forceinline__ void interp_setup(const Dims& D, const double r[3], int idx[3][4],
                                             T phi[3][4]) {
  for (int d = 0; d < 3; ++d) {
    const double x0 = ceil(r[d] - 2.);
    const int o = wrap_any((int)x0, D.n[d]);
    T w[4];
    if constexpr (sizeof(T) == 4) peskin_weights4((T)(r[d] - x0), w);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int t = o + i;
      while (t >= D.n[d]) t -= D.n[d];
      idx[d][i] = t;
      if constexpr (sizeof(T) == 8)
        phi[d][i] = peskin_delta<T>(r[d] - (x0 + i));
      else
        phi[d][i] = w[i];
    }
  }
}

// New periodic coordinate of the FP32 path: a compare-and-shift (valid while a
// step moves a particle less than one box length).
__device__ __forceinline__ double wrap_shift(double r, int n) {
  return r >= n ? r - n : (r < 0.0 ? r + n : r);
}
// New periodic coordinate of the FP64 paths, the reference's fmod(x + size, size)
// (SwimmerArray.cu:167, TracerArray.cu:40).  x + n in [0, 2n), as after any
// ordinary move, takes no division: x + n - n is exact in [n, 2n).  A result
// outside [0, n) raises LBSWIM_STATUS_PARTICLE_OUTSIDE.
__device__ __forceinline__ double wrap_position(double x, int n, unsigned* status) {
  const double size = (double)n, t = __dadd_rn(x, size);
  if (t >= 0.0 && t < 2.0 * size) return t >= size ? __dsub_rn(t, size) : t;
  const double out = fmod(t, size);
  if (!in_box(out, n)) raise_status(status, LBSWIM_STATUS_PARTICLE_OUTSIDE);
  return out;
}

// InterpVelocity, interp.cu:8-47: u at r through the 4^3 Peskin stencil, from
// the FP64 SoA field, every operation rounded in the reference's order ...
__device__ __forceinline__ void interp_velocity(const double* __restrict__ u, const Dims& D,
                                                const double r[3], double v[3]) {
  int idx[3][4];
  double phi[3][4];
  interp_setup<double>(D, r, idx, phi);
  v[0] = v[1] = v[2] = 0.0;
  const long long nynz = (long long)D.n[1] * D.n[2];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      const double pij = phi[0][i] * phi[1][j];
      const long long row = idx[0][i] * nynz + (long long)idx[1][j] * D.n[2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double d3 = pij * phi[2][k];
        const long long s = row + idx[2][k];
        v[0] = add_prod(v[0], d3, u[s]);
        v[1] = add_prod(v[1], d3, u[D.N + s]);
        v[2] = add_prod(v[2], d3, u[2 * D.N + s]);
      }
    }
}

// ... or from the packed float4 field of a reduced-precision lattice (one 16-byte
// load per node).
__device__ __forceinline__ void interp_velocity(const float4* __restrict__ h, const Dims& D,
                                                const double r[3], float v[3]) {
  int idx[3][4];
  float phi[3][4];
  interp_setup<float>(D, r, idx, phi);
  v[0] = v[1] = v[2] = 0.f;
  const long long nynz = (long long)D.n[1] * D.n[2];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      const float pij = phi[0][i] * phi[1][j];
      const long long row = idx[0][i] * nynz + (long long)idx[1][j] * D.n[2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float d3 = pij * phi[2][k];
        const float4 q = __ldg(h + row + idx[2][k]);
        v[0] += d3 * q.x;
        v[1] += d3 * q.y;
        v[2] += d3 * q.z;
      }
    }
}

// FP64 moves in exact mode (LBSWIM_COMPAT_EXACT_F64): the reference's operations
// in its order.  DoSwimmerArrayMove, SwimmerArray.cu:123-210: two threads per
// swimmer, one for its own point and one for its rear point, so that the two
// ordered chains of 450 FP64 operations run side by side.  Small blocks spread
// a small array over the SMs (a warp's FP64 instruction takes 64 clocks of its
// scheduler, whatever its active lanes): 1024 swimmers 130 -> 56 us.
constexpr int EXACT_MOVE_BLOCK = 64;
__global__ void __launch_bounds__(EXACT_MOVE_BLOCK) k_swimmers_move_exact(
    int nsw, double* __restrict__ swr, double* __restrict__ swv, double* __restrict__ swn,
    lbswim_common_params c, unsigned long long seed, unsigned long long step, Dims D,
    const double* __restrict__ u, unsigned* status) {
  const int t = blockIdx.x * EXACT_MOVE_BLOCK + threadIdx.x;
  const int i = t >> 1;
  const bool rear = t & 1, valid = i < nsw;
  double r[3] = {0.0, 0.0, 0.0}, n0[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0};
  bool tumble = false;
  if (valid) {
    double p[3];
    for (int d = 0; d < 3; ++d) {
      r[d] = swr[(long long)nsw * d + i];
      n0[d] = swn[(long long)nsw * d + i];
      p[d] = rear ? __dsub_rn(r[d], __dmul_rn(n0[d], c.l)) : r[d];
    }
    tumble = rng_uniform(seed, (uint32_t)i, step) < c.alpha;
    if (!rear || (!tumble && !c.rotational_advection_off)) interp_velocity(u, D, p, v);
  }
  double vm[3];
  for (int d = 0; d < 3; ++d) vm[d] = __shfl_xor_sync(0xffffffffu, v[d], 1);
  if (rear || !valid) return;
  for (int d = 0; d < 3; ++d) {
    double rDot = __dmul_rn(__dmul_rn(c.mobility, c.P), n0[d]);
    if (!c.translational_advection_off) rDot = __dadd_rn(rDot, v[d]);
    swv[(long long)nsw * d + i] = rDot;
    swr[(long long)nsw * d + i] = wrap_position(__dadd_rn(r[d], rDot), D.n[d], status);
  }
  double nn[3];
  if (tumble) {  // a direction uniform on the sphere
    rng_normal3(seed, (uint32_t)i, step, nn);
  } else if (!c.rotational_advection_off) {  // rotate with the local shear
    for (int d = 0; d < 3; ++d) nn[d] = __dadd_rn(n0[d], (v[d] - vm[d]) / c.l);
  } else {
    return;  // orientation unchanged
  }
  const double norm = __dsqrt_rn(
      __dadd_rn(__dadd_rn(__dmul_rn(nn[0], nn[0]), __dmul_rn(nn[1], nn[1])), __dmul_rn(nn[2], nn[2])));
  for (int d = 0; d < 3; ++d) swn[(long long)nsw * d + i] = nn[d] / norm;
}

// DoTracerArrayMove, TracerArray.cu:12-43 (s accumulated per tracer).
__global__ void __launch_bounds__(EXACT_MOVE_BLOCK) k_tracers_move_exact(
    int ntr, double* __restrict__ r, double* __restrict__ s, double* __restrict__ v, Dims D,
    const double* __restrict__ u, unsigned* status) {
  const int i = blockIdx.x * EXACT_MOVE_BLOCK + threadIdx.x;
  if (i >= ntr) return;
  double rr[3], ss[3], vv[3];
  for (int d = 0; d < 3; ++d) {
    rr[d] = r[(long long)ntr * d + i];
    ss[d] = s[(long long)ntr * d + i];
  }
  interp_velocity(u, D, rr, vv);
  for (int d = 0; d < 3; ++d) {
    v[(long long)ntr * d + i] = vv[d];
    r[(long long)ntr * d + i] = wrap_position(__dadd_rn(rr[d], vv[d]), D.n[d], status);
    s[(long long)ntr * d + i] = __dadd_rn(ss[d], vv[d]);
  }
}

// ---- FP64 moves (default) ------------------------------------------------------
// A block interpolates its points, four lanes each (one per z node), from integer
// weights (fixed_weights4), in three phases: a thread per (point, axis) forms the
// weights, a lane sums its 16 nodes a component, a thread per (particle, axis)
// updates it.  A lane's 16 velocities become integers below 2^60 under the
// largest exponent of the point's 64, and are summed over y, x and z with three
// 32-bit multiply-adds a product: within 2^-57 of the largest velocity in all (rms
// 2^-59), where FP64 sums are within 2^-53 of their terms.  Where the largest velocity
// has hardly any weight (a front in a fluid at rest) that is the coarser one: the sum of
// weight times size, in FP32 beside the integers, sends such points to FP64 (7% of the
// time).  The 400 FP64 operations a point took before ran on two lanes per clock and SM.
// 1,048,576 tracers at 256^3: 748 -> 450 us; 65,536 swimmers 204 -> 107 us, one
// swimmer 50 -> 8 us.
//
// A small array's blocks take 16 points and give each component lanes of its own,
// so that their chains run side by side (one swimmer 10.9 -> 7.6 us, 1074 18.3 ->
// 15.2, 4096 tracers 8.6 -> 5.9); a lane of a large one's, of 64 points, takes the
// three in turn and forms the nodes' offsets once (1,048,576 tracers 470 -> 430).  80
// registers a thread keep three of the large blocks to an SM (65,536 swimmers 123 us in
// 102 registers, 109 in 80).
constexpr int MOVE64_FEW = 16, MOVE64_MANY = 64;
constexpr int MOVE64_MANY_FROM = 16384;  // points
constexpr int move64_block(int points) { return points == MOVE64_FEW ? 12 * points : 4 * points; }

template <int POINTS>
struct Stencil64 {
  Digits w[3][4][POINTS];
  int o[3][POINTS];
  bool lost[3][POINTS];  // the coordinate is not a finite number
  double vel[3][POINTS];
};

// Weights and wrapped origin of coordinate x of point p on axis a.
template <int POINTS>
__device__ __forceinline__ void point_axis64(const Dims& D, double x, int a, int p,
                                             Stencil64<POINTS>& st) {
  const double x0 = ceil(x - 2.);
  st.o[a][p] = wrap_any((int)x0, dim_of(D, a));
  const double dr = x - x0;
  st.lost[a][p] = !finite_d(x);
  long long w[4];
  if (dr >= 1.0 && dr <= 2.0) {
    fixed_weights4(dr, w);
  } else {  // a coordinate beyond 2^52, or a lost one
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = (long long)(peskin_delta<double>(x - (x0 + j)) * 0x1p63);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) st.w[a][j][p] = digits(w[j]);
}

// b as digits of an integer below 2^60 in units of 2^(ke - 1082), toward zero, for a
// double of biased exponent ke - drop.
__device__ __forceinline__ Digits velocity_digits(unsigned long long b, int drop) {
  const unsigned long long m =
      ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;  // bit 62
  const long long v = (long long)(m >> min(drop + 3, 63));
  const long long sg = (long long)b >> 63;
  return digits((v ^ sg) - sg);
}
// acc, t += a b by digits (t holds the cross products, in units of 2^32)
__device__ __forceinline__ void mul_add(Digits a, Digits b, long long& acc, long long& t) {
  t += (long long)a.h * b.l;
  t += (long long)a.l * b.h;
  acc += (long long)a.h * b.h;
}
__device__ __forceinline__ long long sum_of(long long acc, long long t) {
  return acc + ((t + 0x80000000ll) >> 32);
}

// Velocity of the block's points; I: the type of the site offsets.
template <int POINTS, class I>
__device__ __forceinline__ void gather64(const double* __restrict__ u, const Dims& D,
                                         Stencil64<POINTS>& st) {
  const int p = (threadIdx.x >> 2) % POINTS, k = threadIdx.x & 3;
  const I nynz = (I)D.n[1] * D.n[2];
  I xo[4];
  int yo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    xo[i] = (I)node_after(st.o[0][p], i, D.n[0]) * nynz;
    yo[i] = node_after(st.o[1][p], i, D.n[1]) * D.n[2];
  }
  const int z = node_after(st.o[2][p], k, D.n[2]);
  float wyz[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    wyz[j] = (float)st.w[1][j][p].h * (float)st.w[2][k][p].h * 0x1p-62f;
  const int c0 = POINTS == MOVE64_FEW ? threadIdx.x / (4 * POINTS) : 0;
#pragma unroll 1
  for (int c = c0; c < (POINTS == MOVE64_FEW ? c0 + 1 : 3); ++c) {
    const double* __restrict__ uc = u + c * D.N + z;
    unsigned long long b[16];
    unsigned top = 0u;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      b[q] = double_bits(__ldg(uc + xo[q >> 2] + yo[q & 3]));
      top = max(top, hi_word(b[q]) & 0x7fffffffu);
    }
    top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = max(top, __shfl_xor_sync(0xffffffffu, top, 2));
    const int ke = (int)(top >> 20);
    long long xa = 0, xt = 0;
    float sizes = 0.f;  // sum of weight times size, the binade below, in units of 2^(ke - 1022)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      long long ya = 0, yt = 0;
      float part = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int drop = ke - (int)((hi_word(b[4 * i + j]) >> 20) & 0x7ffu);
        mul_add(st.w[1][j][p], velocity_digits(b[4 * i + j], drop), ya, yt);
        part = __fmaf_rn(wyz[j], __uint_as_float((unsigned)max(126 - drop, 0) << 23), part);
      }
      sizes = __fmaf_rn(part, (float)st.w[0][i][p].h * 0x1p-31f, sizes);
      // a product with a weight halves; the sums come back below 2^60
      mul_add(st.w[0][i][p], digits(2 * sum_of(ya, yt)), xa, xt);
    }
    long long v = mul_hi(digits(8 * sum_of(xa, xt)), st.w[2][k][p]);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    const bool fits = ke >= FIXED_MIN_K && ke <= FIXED_MAX_K;
    const bool lost = st.lost[0][p] | st.lost[1][p] | st.lost[2][p];
    if (k == 0 && fits) st.vel[c][p] = signed_fixed_to_double(v, ke - 1);
    // in FP64: velocities beyond the integers' range or not finite, and stencils whose
    // largest velocity has so little weight that its units are too coarse for the rest
    sizes += __shfl_xor_sync(0xffffffffu, sizes, 1);
    sizes += __shfl_xor_sync(0xffffffffu, sizes, 2);
    const bool redo = top != 0u && (!fits || sizes < 0x1p-6f);
    if (__any_sync(0xffffffffu, redo)) {
      double s = 0.0;
#pragma unroll 1
      for (int q = 0; q < 16; ++q) {
        const Digits wx = st.w[0][q >> 2][p], wy = st.w[1][q & 3][p], wz = st.w[2][k][p];
        const double w = (((double)wx.h * 0x1p32 + wx.l) * ((double)wy.h * 0x1p32 + wy.l)) *
                         ((double)wz.h * 0x1p32 + wz.l) * 0x1p-189;
        const I site = (I)node_after(st.o[0][p], q >> 2, D.n[0]) * nynz +
                       node_after(st.o[1][p], q & 3, D.n[1]) * D.n[2];
        s = fma(w, uc[site], s);
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (k == 0 && redo) st.vel[c][p] = s;
    }
    if (k == 0 && !fits && !redo) st.vel[c][p] = 0.0;  // a fluid at rest
    // no weights: no velocity
    if (k == 0 && lost) st.vel[c][p] = bits_double(0x7ff8000000000000ull);
  }
}

template <int POINTS, class I>
__global__ void __launch_bounds__(move64_block(POINTS), POINTS == MOVE64_MANY ? 3 : 4) k_tracers_move_f64(
    int ntr, double* __restrict__ r, double* __restrict__ s, double* __restrict__ v, Dims D,
    const double* __restrict__ u, unsigned* status) {
  __shared__ Stencil64<POINTS> st;
  const int p = threadIdx.x % POINTS, a = threadIdx.x / POINTS;
  const int i = blockIdx.x * POINTS + p;
  const long long at = (long long)ntr * a + i;
  const bool mine = a < 3, valid = mine && i < ntr;
  double x = 0.0, sa = 0.0;
  if (valid) {
    x = r[at];
    sa = s[at];
  }
  if (mine) point_axis64(D, x, a, p, st);
  __syncthreads();
  gather64<POINTS, I>(u, D, st);
  __syncthreads();
  if (!valid) return;
  const double w = st.vel[a][p];
  v[at] = w;
  r[at] = wrap_position(x + w, dim_of(D, a), status);
  s[at] = sa + w;
}

// The first half of a block's points are its swimmers, the others their rear points
// r - l n; the threads (p < half, axis) update them.
// RECORD: the block then records the ends of the moved swimmers into `to`, for
// the next step (thread (p, a): axis a of the tail, p < half, or head of its swimmer).
template <bool RECORD, int POINTS, class I>
__global__ void __launch_bounds__(move64_block(POINTS), POINTS == MOVE64_MANY ? 3 : 4) k_swimmers_move_f64(
    int nsw, double* __restrict__ swr, double* __restrict__ swv, double* __restrict__ swn,
    lbswim_common_params c, unsigned long long seed, unsigned long long step, Dims D,
    const double* __restrict__ u, unsigned* status, RecordTarget<double> to) {
  __shared__ Stencil64<POINTS> st;
  constexpr int HALF = POINTS / 2;
  __shared__ double turned[3][HALF], moved[3][HALF];
  const int p = threadIdx.x % POINTS, a = threadIdx.x / POINTS;
  const int q = p % HALF, i = blockIdx.x * HALF + q;
  const long long at = (long long)nsw * a + i;
  const bool rear = p >= HALF, mine = a < 3, valid = mine && i < nsw;
  double x = 0.0, na = 0.0;
  if (valid) {
    x = swr[at];
    na = swn[at];
  }
  if (mine) point_axis64(D, rear ? __dsub_rn(x, __dmul_rn(na, c.l)) : x, a, p, st);
  __syncthreads();
  gather64<POINTS, I>(u, D, st);
  __syncthreads();
  const bool update = valid && !rear;
  bool tumble = false;
  if (update) {
    tumble = rng_uniform(seed, (uint32_t)i, step) < c.alpha;
    const double va = st.vel[a][q];
    double rDot = __dmul_rn(__dmul_rn(c.mobility, c.P), na);
    if (!c.translational_advection_off) rDot = __dadd_rn(rDot, va);
    swv[at] = rDot;
    const double xn = wrap_position(__dadd_rn(x, rDot), dim_of(D, a), status);
    swr[at] = xn;
    moved[a][q] = xn;
    if (tumble) {  // a direction uniform on the sphere
      double g[3];
      rng_normal3(seed, (uint32_t)i, step, g);
      turned[a][q] = a == 0 ? g[0] : (a == 1 ? g[1] : g[2]);
    } else {  // rotate with the local shear
      turned[a][q] = na + (va - st.vel[a][HALF + q]) / c.l;
    }
  }
  __syncthreads();
  double nn = na;
  if (update && (tumble || !c.rotational_advection_off)) {  // else the orientation is unchanged
    const double nx = turned[0][q], ny = turned[1][q], nz = turned[2][q];
    const double norm =
        __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(nx, nx), __dmul_rn(ny, ny)), __dmul_rn(nz, nz)));
    nn = turned[a][q] / norm;
    swn[at] = nn;
  }
  if constexpr (RECORD) {
    __shared__ EndRecord<double> srec[POINTS];
    __shared__ unsigned lost[POINTS];
    if (a == 0) lost[p] = 0u;
    __syncthreads();  // every axis of a swimmer has been normalised
    if (update) turned[a][q] = nn;
    __syncthreads();
    const int e = 2 * q + (rear ? 1 : 0);  // of the block
    if (valid) {
      record_axis64<true>(moved[a][q], turned[a][q], rear, c.P, c.l, D, a, srec[e], lost[e]);
      if (a == 0) srec[e].pad = 0;
    }
    finish_records64<true, false, POINTS>(e, a, blockIdx.x * POINTS, 2 * nsw, srec, lost, D, to,
                                          TileChains{});
  }
}

template <class U, class T>
__global__ void k_interp_points(int np, const double* __restrict__ r, double* __restrict__ v,
                                Dims D, const U* __restrict__ u) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const double rr[3] = {r[i], r[np + i], r[2 * np + i]};
  T vv[3];
  interp_velocity(u, D, rr, vv);
  for (int d = 0; d < 3; ++d) v[np * d + i] = (double)vv[d];
}

__global__ void k_rng_draws(unsigned long long seed, int n, unsigned long long step,
                            float* __restrict__ uni, double* __restrict__ g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uni[i] = rng_uniform(seed, (uint32_t)i, step);
  double nn[3];
  rng_normal3(seed, (uint32_t)i, step, nn);
  for (int d = 0; d < 3; ++d) g[n * d + i] = nn[d];
}

// ---- seeded initial states made on the device ------------------------------------
// Counter streams keyed (seed, index) at steps far above any move step:
// INIT_STEP_SITE for densities, INIT_STEP_PART for particle positions and
// orientations (block 0: position uniforms, blocks 1-2: orientation normals).
constexpr unsigned long long INIT_STEP_SITE = 0xffffffffffff0001ull;
constexpr unsigned long long INIT_STEP_PART = 0xffffffffffff0002ull;

__global__ void k_init_density(long long N, unsigned long long seed, double amp, double rho0,
                               double* __restrict__ rho, double* __restrict__ u,
                               float4* __restrict__ hydro) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N;
       s += (long long)gridDim.x * blockDim.x) {
    uint32_t x[4];
    rng_block(seed, (uint32_t)s, INIT_STEP_SITE, (uint32_t)(s >> 32), x);
    const double r = 1.0 + amp * (u53(x[0], x[1]) - 0x1.0p-53);  // 1 + amp U[0, 1)
    if (hydro) {
      hydro[s] = make_float4(0.f, 0.f, 0.f, (float)(r - rho0));
    } else {
      rho[s] = r;
      u[s] = u[N + s] = u[2 * N + s] = 0.0;
    }
  }
}

// Positions uniform in the box; orientations (when nv is set) uniform on the sphere.
__global__ void k_init_particles(int n, unsigned long long seed, Dims D, double* __restrict__ r,
                                 double* __restrict__ nv, double* __restrict__ zero_a,
                                 double* __restrict__ zero_b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t x[4];
  rng_block(seed, (uint32_t)i, INIT_STEP_PART, 0u, x);
  const double ux = u53(x[0], x[1]) - 0x1.0p-53, uy = u53(x[2], x[3]) - 0x1.0p-53;
  rng_block(seed, (uint32_t)i, INIT_STEP_PART, 3u, x);
  const double uz = u53(x[0], x[1]) - 0x1.0p-53;
  const double uu[3] = {ux, uy, uz};
  for (int d = 0; d < 3; ++d) {
    r[(long long)n * d + i] = uu[d] * D.n[d];
    if (zero_a) zero_a[(long long)n * d + i] = 0.0;
    if (zero_b) zero_b[(long long)n * d + i] = 0.0;
  }
  if (nv) {
    double g[3];
    rng_normal3(seed, (uint32_t)i, INIT_STEP_PART, g);
    const double norm = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(g[0], g[0]), __dmul_rn(g[1], g[1])),
                                             __dmul_rn(g[2], g[2])));
    for (int d = 0; d < 3; ++d) nv[(long long)n * d + i] = g[d] / norm;
  }
}

// ---- FP32-path Move kernels ------------------------------------------------------
// A block interpolates 64 points in three phases.  (1) A thread per (point, axis)
// forms the wrapped origin node and the Peskin weights in shared memory.  (2) Four
// lanes per point, one per z node, gather its 4^3 nodes, and the partial sums are
// added with a fixed shuffle tree, so the result does not depend on scheduling.
// (3) A thread per (particle, axis) updates it.  GB300's FP64 pipe is narrow: the
// stencil origin comes from the bits of the position by integer operations,
// positions advance in Q44 fixed point, and orientations update in FP32.  With a
// thread per particle in phases 1 and 3 a small array waited for one warp's chain
// of three axes (and two points): 54 swimmers 11 -> 7 us, 3809 11.6 -> 7.9,
// 65,536 the same.
constexpr int MOVE_BLOCK = 256, MOVE_POINTS = MOVE_BLOCK / 4;

// Stencils of a block's points, one array per field so that neighbouring threads
// write them without bank conflicts: wrapped origin node, Peskin weights per axis
// and node, whether the point is gathered, and its velocity.
struct StencilSet {
  int o[3][MOVE_POINTS];
  int active[MOVE_POINTS];
  float w[3][4][MOVE_POINTS];
  float vel[3][MOVE_POINTS];
};

// Exact FP64 value of a float, from its bits (no FP64 instruction).
__device__ __forceinline__ double f2d_exact(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned long long sign = (unsigned long long)(u >> 31) << 63;
  const int e = (int)((u >> 23) & 0xffu);
  unsigned m = u & 0x7fffffu;
  if (e == 255)  // inf / nan
    return __longlong_as_double((long long)(sign | (0x7ffull << 52) | ((unsigned long long)m << 29)));
  if (e == 0) {
    if (m == 0) return __longlong_as_double((long long)sign);
    const int msb = 31 - __clz((int)m);  // subnormal: m * 2^-149
    const unsigned long long mant = ((unsigned long long)m << (52 - msb)) & 0xfffffffffffffull;
    return __longlong_as_double((long long)(sign | ((unsigned long long)(msb - 149 + 1023) << 52) | mant));
  }
  return __longlong_as_double(
      (long long)(sign | ((unsigned long long)(e + 896) << 52) | ((unsigned long long)m << 29)));
}

// Periodic coordinates as Q44 fixed point (44 fraction bits), for lattices
// shorter than 2^19 sites per axis.  pos_to_q44 takes 0 <= r < 2^19 (else
// returns false), rounding to nearest; q44_to_pos returns the FP64 nearest to
// q * 2^-44, q >= 0.  Integer operations only.
constexpr int Q44 = 44;
__device__ __forceinline__ bool pos_to_q44(double r, long long& q) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(r);
  const int ex = (int)(b >> 52);  // negative r gives ex >= 2048
  if (ex >= 1023 + 19) return false;
  if (ex < 1023 - Q44 - 2) {  // r < 2^-46 rounds to 0
    q = 0;
    return true;
  }
  const unsigned long long mant = (b & 0xfffffffffffffull) | (1ull << 52);
  const int sh = 1075 - Q44 - ex;  // q = mant * 2^-sh, -10 <= sh <= 55
  if (sh <= 0) {
    q = (long long)(mant << (-sh));
  } else {
    const unsigned long long rem = mant & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    unsigned long long v = mant >> sh;
    v += (rem > half || (rem == half && (v & 1ull))) ? 1ull : 0ull;
    q = (long long)v;
  }
  return true;
}
__device__ __forceinline__ double q44_to_pos(long long q) {
  if (q <= 0) return 0.0;
  const unsigned long long u = (unsigned long long)q;
  const int msb = 63 - __clzll((long long)u);
  int e = msb - Q44;
  unsigned long long m;
  if (msb <= 52) {
    m = u << (52 - msb);
  } else {
    const int sh = msb - 52;
    const unsigned long long rem = u & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    m = u >> sh;
    m += (rem > half || (rem == half && (m & 1ull))) ? 1ull : 0ull;
    if (m >> 53) {
      m >>= 1;
      ++e;
    }
  }
  return __longlong_as_double(
      (long long)(((unsigned long long)(e + 1023) << 52) | (m & 0xfffffffffffffull)));
}

// r + v moved back into [0, n) by one shift, like wrap_shift: in Q44
// when r and r + v allow it (the result then lies in the box by construction),
// else in FP64, where a result outside [0, n) -- a non-finite r or v, or a
// move longer than the box -- raises LBSWIM_STATUS_PARTICLE_OUTSIDE.
__device__ __forceinline__ double advance_position(double r, float v, int n, unsigned* status) {
  long long q;
  if (n < (1 << 19) && fabsf(v) < (float)n && pos_to_q44(r, q)) {
    q += fx_quant(v, 0x1.0p44f);
    const long long nq = (long long)n << Q44;
    q = q >= nq ? q - nq : (q < 0 ? q + nq : q);
    return q44_to_pos(q);
  }
  const double out = wrap_shift(r + f2d_exact(v), n);
  if (!in_box(out, n)) raise_status(status, LBSWIM_STATUS_PARTICLE_OUTSIDE);
  return out;
}

// The 53-bit uniform of rng_normal3 rounded to FP32 (relative error 2^-24 at
// every magnitude, so the logarithm of a small draw stays close to FP64's).
__device__ __forceinline__ float u53f(uint32_t a, uint32_t b) {
  const unsigned long long m = ((unsigned long long)a << 21) | (unsigned long long)(b >> 11);
  return __ull2float_rn(m + 1ull) * 0x1.0p-53f;
}

// -2 log u of that uniform in FP32; for u >= 1/2 through log1p of the exact
// 1 - u, so that draws near 1 keep their small logarithm.
__device__ __forceinline__ float neg2log_u53(uint32_t a, uint32_t b) {
  const unsigned long long m1 =
      (((unsigned long long)a << 21) | (unsigned long long)(b >> 11)) + 1ull;  // 1 .. 2^53
  if (m1 >= (1ull << 52))
    return -2.f * log1pf(-__ull2float_rn((1ull << 53) - m1) * 0x1.0p-53f);
  return -2.f * logf(__ull2float_rn(m1) * 0x1.0p-53f);
}

// Three normal deviates of a tumble in FP32 from the counter blocks and the
// uniforms of rng_normal3 (Box-Muller).
__device__ __forceinline__ void rng_normal3_f(uint64_t seed, uint32_t swimmer, uint64_t step,
                                              float g[3]) {
  uint32_t a[4], b[4];
  rng_block(seed, swimmer, step, 1u, a);
  rng_block(seed, swimmer, step, 2u, b);
  const float r1 = sqrtf(neg2log_u53(a[0], a[1]));
  const float r2 = sqrtf(neg2log_u53(b[0], b[1]));
  float s1, c1, s2, c2;
  sincospif(2.f * u53f(a[2], a[3]), &s1, &c1);
  sincospif(2.f * u53f(b[2], b[3]), &s2, &c2);
  g[0] = r1 * c1;
  g[1] = r1 * s1;
  g[2] = r2 * c2;
}

// Axis a of the stencil of point p at coordinate x.
__device__ __forceinline__ void point_axis(const Dims& D, double x, int a, int p, StencilSet& st) {
  int x0;
  float dr;
  stencil_axis(x, x0, dr);
  st.o[a][p] = wrap_any(x0, dim_of(D, a));
  float w[4];
  peskin_weights4(dr, w);
#pragma unroll
  for (int j = 0; j < 4; ++j) st.w[a][j][p] = w[j];
}

// Lane k of a point's four takes z node k for the four y and x nodes.  I is the type
// of the site offsets: int while N < 2^31.
template <class Set, class I>
__device__ __forceinline__ float3 gather_point(const float4* __restrict__ h, const Dims& D,
                                               const Set& st, int p, int k) {
  float vx = 0.f, vy = 0.f, vz = 0.f;
  if (st.active[p]) {
    const int nz = D.n[2];
    const I nynz = (I)D.n[1] * D.n[2];
    const int z = node_after(st.o[2][p], k, nz);
    const float wz = st.w[2][k][p];
    I xo[4];
    float wx[4];
#pragma unroll
    for (int ix = 0; ix < 4; ++ix) {
      xo[ix] = (I)node_after(st.o[0][p], ix, D.n[0]) * nynz;
      wx[ix] = st.w[0][ix][p];
    }
#pragma unroll
    for (int jy = 0; jy < 4; ++jy) {
      const I yz = (I)node_after(st.o[1][p], jy, D.n[1]) * nz + z;
      const float wyz = st.w[1][jy][p] * wz;
#pragma unroll
      for (int ix = 0; ix < 4; ++ix) {
        const float4 q = __ldg(h + xo[ix] + yz);
        const float w = wx[ix] * wyz;
        vx += w * q.x;
        vy += w * q.y;
        vz += w * q.z;
      }
    }
  }
  return make_float3(vx, vy, vz);
}
// Sum over a point's four lanes (fixed shuffle tree).
__device__ __forceinline__ float3 sum_lanes(float3 v) {
#pragma unroll
  for (int off = 2; off > 0; off >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
    v.z += __shfl_xor_sync(0xffffffffu, v.z, off);
  }
  return v;
}

// Phase 2 for a block's 64 points.
template <class I>
__device__ __forceinline__ void gather_points(const float4* __restrict__ h, const Dims& D,
                                              StencilSet& st) {
  const int p = threadIdx.x >> 2, k = threadIdx.x & 3;
  const float3 v = sum_lanes(gather_point<StencilSet, I>(h, D, st, p, k));
  if (k < 3) st.vel[k][p] = k == 0 ? v.x : (k == 1 ? v.y : v.z);
}

template <class I>
__device__ __forceinline__ void tracers_move_block(int blk, int ntr, double* __restrict__ r,
                                                   double* __restrict__ s,
                                                   double* __restrict__ v, Dims D,
                                                   const float4* __restrict__ h,
                                                   unsigned* status) {
  __shared__ StencilSet st;
  const int p = threadIdx.x % MOVE_POINTS, a = threadIdx.x / MOVE_POINTS;
  const int i = blk * MOVE_POINTS + p;
  const long long at = (long long)ntr * a + i;
  const bool valid = a < 3 && i < ntr;
  // s is read with r, so the update at the end waits on no load of its own
  double x = 0.0, sa = 0.0;
  if (valid) {
    x = r[at];
    sa = s[at];
    point_axis(D, x, a, p, st);
  }
  if (a == 3) st.active[p] = i < ntr;
  __syncthreads();
  gather_points<I>(h, D, st);
  __syncthreads();
  if (!valid) return;
  const float w = st.vel[a][p];
  const double vd = f2d_exact(w);
  v[at] = vd;
  r[at] = advance_position(x, w, dim_of(D, a), status);
  s[at] = sa + vd;
}

// Large tracer arrays: a block takes 256 tracers, a thread forms the stencil of one
// (all axes) and updates it, and four lanes gather two points at a time.  With
// twice the loads in flight per thread 1,048,576 tracers take 118 us against 146 with
// 64 per block; 60,938 take 15.6 us against 13.3, and 864 11 us against 5.4.
constexpr int WIDE_TRACERS = 256;
struct WideStencilSet {
  int o[3][WIDE_TRACERS];
  int active[WIDE_TRACERS];
  float w[3][4][WIDE_TRACERS];
  float3 vel[WIDE_TRACERS];
};
constexpr int TRACERS_WIDE_FROM = 65536;

__device__ __forceinline__ void wide_stencil(const Dims& D, const double r[3],
                                             WideStencilSet& st, int p) {
  float dr[3];
  for (int d = 0; d < 3; ++d) {
    int x0;
    stencil_axis(r[d], x0, dr[d]);
    st.o[d][p] = wrap_any(x0, D.n[d]);
  }
  st.active[p] = 1;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float w[4];
    peskin_weights4(dr[d], w);
#pragma unroll
    for (int j = 0; j < 4; ++j) st.w[d][j][p] = w[j];
  }
}

template <class I = int>
__device__ __forceinline__ void tracers_move_wide_block(int blk, int ntr, double* __restrict__ r,
                                                        double* __restrict__ s,
                                                        double* __restrict__ v, const Dims& D,
                                                        const float4* __restrict__ h,
                                                        unsigned* status) {
  __shared__ WideStencilSet st;
  const int i = blk * WIDE_TRACERS + threadIdx.x;
  const bool valid = i < ntr;
  double rr[3] = {0.0, 0.0, 0.0}, ss[3] = {0.0, 0.0, 0.0};
  if (valid) {
    for (int d = 0; d < 3; ++d) {
      rr[d] = r[(long long)ntr * d + i];
      ss[d] = s[(long long)ntr * d + i];
    }
    wide_stencil(D, rr, st, threadIdx.x);
  } else {
    st.active[threadIdx.x] = 0;
  }
  __syncthreads();
  const int k = threadIdx.x & 3;
  for (int p = threadIdx.x >> 2; p < WIDE_TRACERS; p += 2 * MOVE_POINTS) {
    const float3 a = gather_point<WideStencilSet, I>(h, D, st, p, k);
    const float3 b = gather_point<WideStencilSet, I>(h, D, st, p + MOVE_POINTS, k);
    const float3 sa = sum_lanes(a), sb = sum_lanes(b);
    if (k == 0) {
      st.vel[p] = sa;
      st.vel[p + MOVE_POINTS] = sb;
    }
  }
  __syncthreads();
  if (!valid) return;
  const float3 w = st.vel[threadIdx.x];
  const float vv[3] = {w.x, w.y, w.z};
  for (int d = 0; d < 3; ++d) {
    const double vd = f2d_exact(vv[d]);
    v[(long long)ntr * d + i] = vd;
    r[(long long)ntr * d + i] = advance_position(rr[d], vv[d], D.n[d], status);
    s[(long long)ntr * d + i] = ss[d] + vd;
  }
}

template <bool WIDE, class I>
__global__ void __launch_bounds__(MOVE_BLOCK) k_tracers_move_f32(
    int ntr, double* __restrict__ r, double* __restrict__ s, double* __restrict__ v, Dims D,
    const float4* __restrict__ h, unsigned* status) {
  if constexpr (WIDE)
    tracers_move_wide_block<I>(blockIdx.x, ntr, r, s, v, D, h, status);
  else
    tracers_move_block<I>(blockIdx.x, ntr, r, s, v, D, h, status);
}

// Points [0, 32) of a block are its swimmers, [32, 64) their rear points r - l n; the
// threads (p < 32, axis) update them: SwimmerArray.cu:151-209 with the FP32 path's
// arithmetic (Q44 positions, FP32 turn added to the FP64 orientation, FP32 tumble
// normals).  RECORD: the block also records the ends of the moved swimmers into
// `to`, for the next step (thread (p, a): axis a of the tail, p < 32, or head of
// swimmer p % 32).
constexpr int MOVE_SWIMMERS = MOVE_POINTS / 2;
static_assert(2 * MOVE_SWIMMERS == REC_ENDS, "the ends of a block's swimmers");
template <bool RECORD, class I = int, bool BUCKETS = false>
__device__ __forceinline__ void swimmers_move_block(
    int blk, int nsw, double* __restrict__ swr, double* __restrict__ swv,
    double* __restrict__ swn, const lbswim_common_params& c, unsigned long long seed,
    unsigned long long step, const Dims& D, const float4* __restrict__ h, unsigned* status,
    const RecordTarget<float>& to = RecordTarget<float>{}) {
  __shared__ StencilSet st;
  __shared__ float turned[3][MOVE_SWIMMERS];
  const int p = threadIdx.x % MOVE_POINTS, a = threadIdx.x / MOVE_POINTS;
  const int q = p % MOVE_SWIMMERS, i = blk * MOVE_SWIMMERS + q;
  const long long at = (long long)nsw * a + i;
  const bool rear = p >= MOVE_SWIMMERS, valid = a < 3 && i < nsw, update = valid && !rear;
  double x = 0.0, na = 0.0;
  if (valid) {
    x = swr[at];
    na = swn[at];
  }
  bool tumble = false, rotate = false;
  if (i < nsw) {
    tumble = rng_uniform(seed, (uint32_t)i, step) < c.alpha;
    rotate = !tumble && !c.rotational_advection_off;
  }
  // the rear point as the dipole-end records compute it
  if (valid && (!rear || rotate))
    point_axis(D, rear ? __dsub_rn(x, __dmul_rn(na, c.l)) : x, a, p, st);
  if (a == 3) st.active[p] = i < nsw && (!rear || rotate);
  __syncthreads();
  gather_points<I>(h, D, st);
  __syncthreads();
  double xn = 0.0, nn = na;
  float inv = 0.f;
  if (update) {
    const float va = st.vel[a][q];
    float rDot = (float)(c.mobility * c.P) * (float)na;
    if (!c.translational_advection_off) rDot += va;
    swv[at] = f2d_exact(rDot);
    xn = advance_position(x, rDot, dim_of(D, a), status);
    swr[at] = xn;
    if (tumble) {
      float g[3];
      rng_normal3_f(seed, (uint32_t)i, step, g);
      inv = 1.f / sqrtf(__fmaf_rn(g[2], g[2], __fmaf_rn(g[1], g[1], __fmul_rn(g[0], g[0]))));
      nn = f2d_exact((a == 0 ? g[0] : (a == 1 ? g[1] : g[2])) * inv);
    } else if (rotate) {
      // the small turn (v - v_rear) / l is formed in FP32 and added to the FP64
      // orientation, which keeps its direction; the FP32 norm only rescales it
      const float inv_l = 1.f / (float)c.l;
      nn = __dadd_rn(na, f2d_exact((va - st.vel[a][MOVE_SWIMMERS + q]) * inv_l));
      turned[a][q] = (float)nn;
    }
  }
  __syncthreads();
  if (update && rotate) {
    const float tx = turned[0][q], ty = turned[1][q], tz = turned[2][q];
    // the roundings are spelt out: every instance of this code gives the same bits
    const float sq = __fmaf_rn(tz, tz, __fmaf_rn(ty, ty, __fmul_rn(tx, tx)));
    nn = __dmul_rn(nn, f2d_exact(1.f / sqrtf(sq)));
  }
  if (update && (tumble || rotate)) swn[at] = nn;
  if (RECORD && to.ends) {  // uniform in the block
    __shared__ double moved[2][3][MOVE_SWIMMERS];
    __shared__ EndRecord<float> srec[REC_ENDS];
    __shared__ unsigned smax;
    if (threadIdx.x == 0) smax = 0u;
    if (update) {
      moved[0][a][q] = xn;
      moved[1][a][q] = nn;
    }
    __syncthreads();
    const int e = 2 * q + (rear ? 1 : 0);  // of the block
    unsigned big = 0u;
    if (valid)
      big = record_axis32(moved[0][a][q], moved[1][a][q], rear, c.P, c.l, D, a, srec[e]);
    finish_records32<BUCKETS>(e, a, blk * REC_ENDS, 2 * nsw, 0, big, srec, smax, D, to);
  }
}

template <bool RECORD, class I>
__global__ void __launch_bounds__(MOVE_BLOCK) k_swimmers_move_f32(
    const __grid_constant__ SwimmerList w, Dims D, const float4* __restrict__ h, unsigned* status,
    RecordTarget<float> to) {
  const SwimmerPart& p = w.part[part_of_block(w)];
  to.ends += p.end0;
  swimmers_move_block<RECORD, I>(blockIdx.x - p.block0, p.n, p.r, p.v, p.nv, p.common, p.seed,
                                 p.step, D, h, status, to);
}

// ---- batched ensembles: per-step reset, end records, moves --------------------
__device__ __forceinline__ int ens_find(const int* __restrict__ prefix, int nmem, int item) {
  int lo = 0, hi = nmem - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= item)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ Dims ens_dims(const EnsMember& M) {
  Dims D;
  for (int a = 0; a < 3; ++a) {
    D.n[a] = M.size[a];
    D.nb[a] = (M.size[a] + BIN - 1) / BIN;
  }
  D.N = M.n;
  return D;
}

__device__ __forceinline__ TileGrid ens_grid(const EnsMember& M) {
  TileGrid G;
  G.T[0] = M.lx;
  G.T[1] = M.tile == 1 ? 16 : 8;  // as slab_section_of
  G.T[2] = M.tile == 1 ? 16 : 32;
  G.h = 1;
  G.by[0] = FastDiv{M.by_lx[0], M.by_lx[1]};
  for (int a = 0; a < 3; ++a) {
    G.nt[a] = M.nt[a];
    if (a) G.by[a] = FastDiv{1u, (unsigned)__ffs(G.T[a]) - 1u};  // powers of two
  }
  return G;
}

// Before a run: zero the slab counts and largest |F| of every member that steps,
// and the slab counters.
__global__ void k_ens_reset(EnsTable t) {
  const int nmem = *t.nmem;
  if (blockIdx.x == 0 && threadIdx.x < 2) t.counters[threadIdx.x] = 0u;
  for (int m = blockIdx.x; m < nmem; m += gridDim.x) {
    const EnsMember& M = t.mem[m];
    if (M.limit <= 0) continue;
    const int nslabs = M.nt[0] * M.nt[1] * M.nt[2];
    for (int i = threadIdx.x; i < nslabs; i += blockDim.x) M.bucket_count[i] = 0u;
    if (threadIdx.x < 2) M.max_abs_f[threadIdx.x] = 0u;
  }
}

// After a run: the largest |F| of a member's last step to the first word, beside
// its records (a member's last move makes none).
__global__ void k_ens_finish(EnsTable t) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= *t.nmem) return;
  const EnsMember& M = t.mem[m];
  if (M.limit > 0) M.max_abs_f[0] = M.max_abs_f[(M.limit - 1) & 1];
}

// The records of a run's first step; the later ones' are made by the moves.
__global__ void __launch_bounds__(REC_THREADS) k_ens_records(EnsTable t) {
  const int nmem = *t.nmem;
  const int total = t.rec_prefix[nmem];
  for (int vb = blockIdx.x; vb < total; vb += gridDim.x) {
    const int m = ens_find(t.rec_prefix, nmem, vb);
    const EnsMember& M = t.mem[m];
    if (M.limit <= 0) continue;
    end_records_block(vb - t.rec_prefix[m], M.nsw, M.sw_r, M.sw_n, M.common.P, M.common.l,
                      ens_dims(M), 0,
                      RecordTarget<float>{(EndRecord<float>*)M.ends, M.max_abs_f, ens_grid(M),
                                          M.bucket_count, M.bucket_list});
    __syncthreads();
  }
}

static_assert(ENS_ENDS_PER_BLOCK == REC_ENDS && ENS_SWIMMERS_PER_BLOCK == MOVE_SWIMMERS &&
                  ENS_TRACERS_PER_BLOCK == MOVE_POINTS,
              "batched work items per block");

// The moves of a step, and the records of the next one (none by a member's last
// move, so that its records stay those of the forces of its last step).  Tracers in
// blocks of 256, the better form for one large array, took a step of 512 members with
// a million tracers from 2.07 to 2.11 ms.
__global__ void __launch_bounds__(MOVE_BLOCK) k_ens_move(EnsTable t, int parity) {
  const int nmem = *t.nmem;
  const int nsb = t.sw_prefix[nmem], total = nsb + t.tr_prefix[nmem];
  const unsigned long long g = (unsigned long long)t.g_step[parity];
  if (blockIdx.x == 0 && threadIdx.x == 0) t.g_step[parity ^ 1] = (long long)g + 1;
  for (int vb = blockIdx.x; vb < total; vb += gridDim.x) {
    if (vb < nsb) {
      const int m = ens_find(t.sw_prefix, nmem, vb);
      const EnsMember& M = t.mem[m];
      if ((long long)g >= M.limit) continue;  // uniform in the block: no barrier skipped
      const bool more = (long long)g + 1 < M.limit;
      swimmers_move_block<true, int, true>(
          vb - t.sw_prefix[m], M.nsw, M.sw_r, M.sw_v, M.sw_n, M.common, M.seed, M.step0 + g,
          ens_dims(M), (const float4*)M.hyd[parity], M.status,
          RecordTarget<float>{more ? (EndRecord<float>*)M.ends : nullptr,
                              M.max_abs_f + (parity ^ 1), ens_grid(M), M.bucket_count,
                              M.bucket_list});
    } else {
      const int m = ens_find(t.tr_prefix, nmem, vb - nsb);
      const EnsMember& M = t.mem[m];
      if ((long long)g >= M.limit) continue;
      tracers_move_block<int>(vb - nsb - t.tr_prefix[m], M.ntr, M.tr_r, M.tr_s, M.tr_v,
                              ens_dims(M), (const float4*)M.hyd[parity], M.status);
    }
    __syncthreads();
  }
}

void ens_launch_reset(const EnsTable& t, cudaStream_t s) {
  k_ens_reset<<<152, 256, 0, s>>>(t);
  LB_CHECK_LAUNCH(1);
}
void ens_launch_finish(const EnsTable& t, int members, cudaStream_t s) {
  k_ens_finish<<<(members + 255) / 256, 256, 0, s>>>(t);
  LB_CHECK_LAUNCH(1);
}
void ens_launch_records(const EnsTable& t, int grid, cudaStream_t s) {
  k_ens_records<<<grid, REC_THREADS, 0, s>>>(t);
  LB_CHECK_LAUNCH(1);
}
void ens_launch_move(const EnsTable& t, int parity, int grid, cudaStream_t s) {
  k_ens_move<<<grid, MOVE_BLOCK, 0, s>>>(t, parity);
  LB_CHECK_LAUNCH(1);
}

// ---- host side -----------------------------------------------------------------
static Dims make_dims(const Lattice* L) {
  Dims D;
  for (int a = 0; a < 3; ++a) {
    D.n[a] = L->size[a];
    D.nb[a] = (L->size[a] + BIN - 1) / BIN;
  }
  D.N = L->n;
  return D;
}

static int slabs_of(const TileGrid& G) { return G.nt[0] * G.nt[1] * G.nt[2]; }

static TileGrid force_tiles(const Lattice* L) {
  TileGrid G;
  G.T[0] = FT_X;
  G.T[1] = FT_Y;
  G.T[2] = FT_Z;
  G.h = 0;
  for (int a = 0; a < 3; ++a) {
    G.nt[a] = (L->size[a] + G.T[a] - 1) / G.T[a];
    G.by[a] = fast_div((unsigned)G.T[a]);
  }
  return G;
}

// Upper bound on the tile-list entries of one end: 4 + 2h consecutive sites per
// axis meet at most ceil((4 + 2h) / T) + 1 tiles, plus one more when they wrap
// around a partial last tile.
static long long touches_per_end(const TileGrid& G) {
  long long m = 1;
  for (int a = 0; a < 3; ++a)
    m *= std::min<long long>(G.nt[a], (4 + 2 * G.h + G.T[a] - 1) / G.T[a] + 2);
  return m;
}

static void free_chains(SpreadScratch& S) {
  void* ptrs[] = {S.chain_head, S.chain_next, S.chain_ids};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  S.chain_head = S.chain_next = S.chain_ids = nullptr;
  S.chain_room = 0;
}

static void free_lists(TileLists& TL) {
  void* ptrs[] = {TL.count, TL.start, TL.scan_tmp, TL.list, TL.sorted};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  TL = TileLists();
}

void spread_free(SpreadScratch& S) {
  {
    SpreadScratch::Prepared& P = S.prep;
    void* ptrs[] = {P.ends, P.bucket_count, P.bucket_list, P.max_abs_force};
    for (void* p : ptrs)
      if (p) cudaFree(p);
    P = SpreadScratch::Prepared();
  }
  if (S.ends) cudaFree(S.ends);
  if (S.max_abs_force) cudaFree(S.max_abs_force);
  if (S.bucket_count) cudaFree(S.bucket_count);
  if (S.bucket_list) cudaFree(S.bucket_list);
  S.ends = nullptr;
  S.max_abs_force = nullptr;
  S.bucket_count = nullptr;
  S.bucket_list = nullptr;
  S.bucket_slabs = 0;
  S.bucket_tile = -1;
  free_lists(S.ftiles);
  free_chains(S);
}

static size_t record_bytes(const Lattice* L) {
  return L->precision == LBSWIM_F64 ? sizeof(EndRecord<double>) : sizeof(EndRecord<float>);
}

// Room for `total` pending ends, keeping the records already pending.
static void ensure_ends(Lattice* L, int total) {
  SpreadScratch& S = L->spread;
  const size_t rec = record_bytes(L);
  if (S.capacity_ends >= total && S.ends_bytes >= rec * (size_t)total) return;
  const int cap = std::max(total + total / 2, 64);
  void* fresh = nullptr;
  LB_CUDA(cudaMalloc(&fresh, rec * cap));
  if (S.ends && S.pending > 0)
    LB_CUDA(cudaMemcpyAsync(fresh, S.ends, rec * S.pending, cudaMemcpyDeviceToDevice, L->stream));
  LB_CUDA(cudaStreamSynchronize(L->stream));
  if (S.ends) cudaFree(S.ends);
  S.ends = fresh;
  S.capacity_ends = cap;
  S.ends_bytes = rec * cap;
}

static void ensure_lists(Lattice* L, TileLists& TL, const TileGrid& G, int nends) {
  const int ntiles = G.nt[0] * G.nt[1] * G.nt[2];
  if (TL.ntiles != ntiles) {
    LB_CUDA(cudaStreamSynchronize(L->stream));
    const long long keep = TL.capacity;
    int* keep_list = TL.list;
    int* keep_sorted = TL.sorted;
    if (TL.count) cudaFree(TL.count);
    if (TL.start) cudaFree(TL.start);
    if (TL.scan_tmp) cudaFree(TL.scan_tmp);
    TL.count = TL.start = TL.scan_tmp = nullptr;
    LB_CUDA(cudaMalloc(&TL.count, sizeof(unsigned) * ntiles));
    LB_CUDA(cudaMalloc(&TL.start, sizeof(unsigned) * (ntiles + 1)));
    const int nscan = (ntiles + SCAN_TILE - 1) / SCAN_TILE;
    LB_CUDA(cudaMalloc(&TL.scan_tmp, sizeof(unsigned) * std::max(nscan, 1)));
    LB_CUDA(cudaMemsetAsync(TL.count, 0, sizeof(unsigned) * ntiles, L->stream));
    TL.ntiles = ntiles;
    TL.capacity = keep;
    TL.list = keep_list;
    TL.sorted = keep_sorted;
  }
  const long long need = std::max<long long>((long long)nends * touches_per_end(G), 64);
  if (TL.capacity < need) {
    LB_CUDA(cudaStreamSynchronize(L->stream));
    if (TL.list) cudaFree(TL.list);
    if (TL.sorted) cudaFree(TL.sorted);
    TL.list = TL.sorted = nullptr;
    LB_CUDA(cudaMalloc(&TL.list, sizeof(int) * need));
    LB_CUDA(cudaMalloc(&TL.sorted, sizeof(int) * need));
    TL.capacity = need;
  }
}

// Lists of nends recorded ends per tile of G (entries unordered within a tile).
static void bin_ends(Lattice* L, TileLists& TL, const TileGrid& G, int nends) {
  ensure_lists(L, TL, G, nends);
  const Dims D = make_dims(L);
  const EndRecord<double>* ends = (const EndRecord<double>*)L->spread.ends;
  k_touch<0><<<(nends + 255) / 256, 256, 0, L->stream>>>(nends, ends, D, G, TL.count, nullptr,
                                                         nullptr);
  const int nscan = (TL.ntiles + SCAN_TILE - 1) / SCAN_TILE;
  k_scan_tiles<<<nscan, SCAN_THREADS, 0, L->stream>>>(TL.count, TL.ntiles, TL.scan_tmp);
  k_scan_top<<<1, 1024, 0, L->stream>>>(TL.scan_tmp, nscan);
  k_scan_apply_total<<<nscan, SCAN_THREADS, 0, L->stream>>>(TL.count, TL.ntiles, TL.scan_tmp,
                                                            TL.start);
  k_touch<1><<<(nends + 255) / 256, 256, 0, L->stream>>>(nends, ends, D, G, TL.count, TL.start,
                                                         TL.list);
  LB_CHECK_LAUNCH(5);
}

// Buckets of FT_CAP ends per force tile, counts zero between calls.
static void ensure_tile_buckets(Lattice* L, int ntiles) {
  SpreadScratch& S = L->spread;
  if (S.bucket_count) return;  // the tiles of an FP64 lattice never change
  unsigned* count = nullptr;
  LB_CUDA(cudaMalloc(&count, sizeof(unsigned) * ntiles));
  const cudaError_t e = cudaMalloc(&S.bucket_list, sizeof(int) * (size_t)ntiles * FT_CAP);
  if (e != cudaSuccess) {
    cudaFree(count);
    S.bucket_list = nullptr;
    LB_CUDA(e);
  }
  S.bucket_count = count;
  S.bucket_slabs = ntiles;
  LB_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned) * ntiles, L->stream));
}

// Buckets while the average tile lists at most half of one (an end touches 2.6
// tiles of 1024 sites on average).
static bool tiles_take_buckets(const TileGrid& G, long long nends) {
  return nends <= 48ll * G.nt[0] * G.nt[1] * G.nt[2] &&
         nends * touches_per_end(G) <= 0x7fffffffll;  // a chain's entries
}

// Chains for the tiles that may list more of nends ends than a bucket holds.
static TileChains tile_chains(Lattice* L, const TileGrid& G, int nends, bool exact) {
  TileChains ch{};
  if (nends <= FT_CAP) return ch;
  SpreadScratch& S = L->spread;
  ch.touch = (int)touches_per_end(G);
  ch.by_touch = fast_div((unsigned)ch.touch);
  ch.half = (long long)nends * ch.touch;
  if (S.chain_room < ch.half || (exact && !S.chain_ids)) {
    LB_CUDA(cudaStreamSynchronize(L->stream));
    free_chains(S);
    // the ids' counter after the heads
    LB_CUDA(cudaMalloc(&S.chain_head, sizeof(int) * 32 * (size_t)slabs_of(G) + 8));
    LB_CUDA(cudaMalloc(&S.chain_next, sizeof(int) * ch.half));
    if (exact) LB_CUDA(cudaMalloc(&S.chain_ids, sizeof(int) * 2 * ch.half));
    S.chain_room = ch.half;
  }
  ch.head = S.chain_head;
  ch.next = S.chain_next;
  if (exact) {
    ch.ids = S.chain_ids;
    ch.half = S.chain_room;
    ch.id_end = reinterpret_cast<unsigned long long*>(S.chain_head + 32 * (size_t)slabs_of(G));
  }
  return ch;
}

// force = base + the spread of the nends ends recorded (and listed in buckets and chains).
static void spread_fixed(Lattice* L, int nends, const TileChains& ch) {
  SpreadScratch& S = L->spread;
  const TileGrid G = force_tiles(L);
  const int ntiles = slabs_of(G);
  const int threads = ntiles <= 2 * sm_count() ? 2 * FT_THREADS : FT_THREADS;
  auto kernel = threads > FT_THREADS ? k_force_fixed<2 * FT_THREADS> : k_force_fixed<FT_THREADS>;
  kernel<<<ntiles, threads, 0, L->stream>>>(
      make_dims(L), G, (const EndRecord<double>*)S.ends, nends,
      nends > DIRECT_ENDS_F64 ? S.bucket_count : nullptr, S.bucket_list, ch, (double*)L->force,
      L->force_zero_pending ? 0 : 1);
  LB_CHECK_LAUNCH(1);
  L->force_zero_pending = false;
}

// force = base + the spread of W's dipole ends on an FP64 lattice.  With buckets it
// takes two launches in place of eight, which at 16^3 took 36 us of device time
// together and take 13 us.  Denser suspensions list their ends by a counting
// sort (k_force_tile orders long lists in global scratch).
static void add_forces_f64(Swimmers* W, Lattice* L) {
  SpreadScratch& S = L->spread;
  const int nends = 2 * W->n;
  if (nends == 0) {
    if (L->force_zero_pending) lattice_zero_force_now(L);
    return;
  }
  const bool exact = L->compat & LBSWIM_COMPAT_EXACT_F64;
  const Dims D = make_dims(L);
  const TileGrid G = force_tiles(L);
  const int ntiles = G.nt[0] * G.nt[1] * G.nt[2];
  const bool buckets = tiles_take_buckets(G, nends);
  ensure_ends(L, nends);
  if (buckets) ensure_tile_buckets(L, ntiles);
  const TileChains ch = buckets ? tile_chains(L, G, nends, exact) : TileChains{};
  S.prep.valid = false;  // its records share the buffer
  EndRecord<double>* ends = (EndRecord<double>*)S.ends;
  const int grid = (nends + REC64_ENDS - 1) / REC64_ENDS;
  if (buckets && !exact) {
    k_end_records_f64<true><<<grid, REC64_THREADS, 0, L->stream>>>(
        W->n, W->r, W->nv, W->common.P, W->common.l, D,
        RecordTarget<double>{ends, nullptr, G,
                             nends > DIRECT_ENDS_F64 ? S.bucket_count : nullptr, S.bucket_list},
        ch);
    LB_CHECK_LAUNCH(1);
    spread_fixed(L, nends, ch);
    return;
  }
  k_end_records_f64<false><<<grid, REC64_THREADS, 0, L->stream>>>(
      W->n, W->r, W->nv, W->common.P, W->common.l, D,
      RecordTarget<double>{ends, nullptr, G, buckets ? S.bucket_count : nullptr, S.bucket_list},
      ch);
  LB_CHECK_LAUNCH(1);
  if (!buckets) bin_ends(L, S.ftiles, G, nends);
  k_force_tile<<<ntiles, FT_THREADS, 0, L->stream>>>(
      D, G, ends, buckets ? nullptr : S.ftiles.start, S.bucket_count,
      buckets ? S.bucket_list : S.ftiles.list, S.ftiles.sorted, ch, (double*)L->force,
      L->force_zero_pending ? 0 : 1);
  LB_CHECK_LAUNCH(1);
  L->force_zero_pending = false;
}

void spread_materialise(Lattice* L) {
  if (L->spread.pending > 0) {
    lattice_force_from_slabs(L);
    L->spread.pending = 0;
    L->spread.stepped = false;
    L->force_zero_pending = false;
  } else if (L->force_zero_pending) {
    lattice_zero_force_now(L);
  }
}

static TileGrid slab_grid(const Lattice* L, int lx) {
  TileGrid G;
  G.T[0] = lx;
  slab_section_of(L->fused_tile, &G.T[1], &G.T[2]);
  G.h = 1;  // the step kernel collides a one-site ring around its slab
  for (int a = 0; a < 3; ++a) {
    G.nt[a] = (L->size[a] + G.T[a] - 1) / G.T[a];
    G.by[a] = fast_div((unsigned)G.T[a]);
  }
  return G;
}

// Buckets (count and list) for at least nslabs slabs; replacing them waits for
// the lattice's work.
static void grow_buckets(Lattice* L, int nslabs, unsigned*& count, int*& list, int& slabs) {
  if (slabs >= nslabs && count) return;
  LB_CUDA(cudaStreamSynchronize(L->stream));
  if (count) cudaFree(count);
  if (list) cudaFree(list);
  count = nullptr;
  list = nullptr;
  slabs = 0;
  LB_CUDA(cudaMalloc(&count, sizeof(unsigned) * nslabs));
  LB_CUDA(cudaMalloc(&list, sizeof(int) * (size_t)nslabs * SLAB_BUCKET_CAP));
  slabs = nslabs;
}

// Buckets for slabs of lx planes; those of short slabs (4 KB each, twice: a dense lattice in
// slabs of one plane takes a fifth of its own size) while they take a quarter of what is
// free on the device, otherwise of 32 planes.  Returns which.
static int grow_slab_buckets(Lattice* L, int lx, unsigned*& count, int*& list, int& slabs) {
  const int longer = std::min(32, L->size[0]), nslabs = slabs_of(slab_grid(L, lx));
  if (lx < longer && (slabs < nslabs || !count)) {
    size_t free = 0, total = 0;
    LB_CUDA(cudaMemGetInfo(&free, &total));
    if (sizeof(int) * (size_t)nslabs * SLAB_BUCKET_CAP > free / 4) lx = longer;
  }
  grow_buckets(L, slabs_of(slab_grid(L, lx)), count, list, slabs);
  return lx;
}

int spread_reserve(Lattice* L, int nends, int lx) {
  ensure_ends(L, nends);
  SpreadScratch& S = L->spread;
  if (!S.max_abs_force) LB_CUDA(cudaMalloc(&S.max_abs_force, 2 * sizeof(unsigned)));
  S.bucket_tile = -1;
  return grow_slab_buckets(L, lx, S.bucket_count, S.bucket_list, S.bucket_slabs);
}

// Empty buckets for slabs of S.lx planes.
static void clear_buckets(Lattice* L) {
  SpreadScratch& S = L->spread;
  S.lx = grow_slab_buckets(L, S.lx, S.bucket_count, S.bucket_list, S.bucket_slabs);
  const int nslabs = slabs_of(slab_grid(L, S.lx));
  LB_CUDA(cudaMemsetAsync(S.bucket_count, 0, sizeof(unsigned) * nslabs, L->stream));
  S.bucket_tile = L->fused_tile;
}

SlabSpread spread_prepare_slabs(Lattice* L) {
  SpreadScratch& S = L->spread;
  S.last_pending = S.pending;
  const bool direct = S.pending <= DIRECT_ENDS;
  if (direct) {
    S.lx = choose_slab_lx(L, S.pending);
    S.bucket_tile = -1;
  } else if (S.bucket_tile != L->fused_tile) {
    S.lx = choose_slab_lx(L, S.pending);
    clear_buckets(L);
    if (S.pending > 0) {
      k_bucket_ends<<<(S.pending + 255) / 256, 256, 0, L->stream>>>(
          S.pending, (const EndRecord<float>*)S.ends, make_dims(L), slab_grid(L, S.lx),
          S.bucket_count, S.bucket_list);
      LB_CHECK_LAUNCH(1);
    }
  }
  SlabSpread out;
  out.ends = S.ends;
  out.count = direct ? nullptr : S.bucket_count;
  out.list = S.bucket_list;
  out.npending = S.pending;
  out.max_abs_force = S.max_abs_force;
  out.lx = S.lx;
  return out;
}

// The parts of nw arrays, `per` items of 1 / `scale` of a swimmer a block, their ends
// counted from end0; returns the number of blocks.
static int list_parts(Swimmers* const* w, int nw, int per, int scale, int end0, SwimmerList& out) {
  int blocks = 0;
  out.count = nw;
  for (int i = 0; i < nw; ++i) {
    const Swimmers* W = w[i];
    out.part[i] = SwimmerPart{W->n, blocks, end0, W->r, W->v, W->nv, W->common, W->seed, W->step};
    blocks += (int)(((long long)scale * W->n + per - 1) / per);
    end0 += 2 * W->n;
  }
  return blocks;
}

// FP32 records of the arrays' ends, the first of them end0 of the lattice's.
static void launch_end_records(Swimmers* const* w, int nw, Lattice* L, int end0,
                               const RecordTarget<float>& to) {
  SwimmerList list;
  const int blocks = list_parts(w, nw, REC_ENDS, 2, end0, list);
  if (blocks == 0) return;
  k_end_records<<<blocks, REC_THREADS, 0, L->stream>>>(list, make_dims(L), to);
  LB_CHECK_LAUNCH(1);
}

// Records W's ends after the pending ones of a reduced-precision lattice, listed
// under the step kernel's slabs.
static void append_ends(Swimmers* W, Lattice* L) {
  SpreadScratch& S = L->spread;
  const int nends = 2 * W->n;
  ensure_ends(L, S.pending + nends);
  if (!S.max_abs_force) LB_CUDA(cudaMalloc(&S.max_abs_force, 2 * sizeof(unsigned)));
  if (S.pending == 0) {
    S.bucket_tile = -1;
    const int expected = std::max(nends, S.last_pending);
    if (expected > DIRECT_ENDS) {
      S.lx = choose_slab_lx(L, expected);
      clear_buckets(L);
    }
  }
  const bool fill = S.bucket_tile == L->fused_tile;
  if (S.pending == 0) LB_CUDA(cudaMemsetAsync(S.max_abs_force, 0, sizeof(unsigned), L->stream));
  launch_end_records(&W, 1, L, S.pending,
                     RecordTarget<float>{(EndRecord<float>*)S.ends, S.max_abs_force,
                                         fill ? slab_grid(L, S.lx) : TileGrid{},
                                         fill ? S.bucket_count : nullptr, S.bucket_list});
  S.pending += nends;
}

// 64-bit site offsets in the move kernels: when 32-bit ones would
// overflow, or when the lattice asks for them (LBSWIM_COMPAT_WIDE_INDEX).
static bool wide_particle_index(const Lattice* L) {
  return L->n >= (1ll << 31) || (L->compat & LBSWIM_COMPAT_WIDE_INDEX);
}

static void swimmers_mark(Swimmers* W, cudaStream_t stream) {
  if (!W->done) LB_CUDA(cudaEventCreateWithFlags(&W->done, cudaEventDisableTiming));
  LB_CUDA(cudaEventRecord(W->done, stream));
}

// Swimmer fields into page-locked host buffers by the kernel itself: one launch in
// place of three copies, whose starts cost more than the bytes of a small array.
__global__ void k_swimmers_to_host(int n3, const double* __restrict__ r,
                                   const double* __restrict__ v, const double* __restrict__ nv,
                                   double* __restrict__ hr, double* __restrict__ hv,
                                   double* __restrict__ hn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n3) return;
  if (hr) hr[i] = r[i];
  if (hv) hv[i] = v[i];
  if (hn) hn[i] = nv[i];
}

// Swimmers whose fields a kernel writes to the host.  A read-back alone takes 15 us
// up to 4096 swimmers; above, the copies leave the SMs to the next step's records for
// 1.6 us more (8192 swimmers 19.1 us against 17.6, 65,536 40.8 against 39.1).
constexpr int DIRECT_READ_SWIMMERS = 4096;

void swimmers_read(Swimmers* W, double* r, double* v, double* n) {
  if (!W->copy) {
    // ahead of the blocks of queued tracer moves
    int least = 0, greatest = 0;
    LB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    LB_CUDA(cudaStreamCreateWithPriority(&W->copy, cudaStreamNonBlocking, greatest));
  }
  if (W->done) LB_CUDA(cudaStreamWaitEvent(W->copy, W->done, 0));
  double* dst[3] = {r, v, n};
  const double* src[3] = {W->r, W->v, W->nv};
  double* mapped[3] = {nullptr, nullptr, nullptr};
  const size_t bytes = sizeof(double) * 3 * (size_t)W->n;
  bool direct = W->n > 0 && W->n <= DIRECT_READ_SWIMMERS;
  for (int f = 0; f < 3 && direct; ++f)
    if (dst[f]) {
      mapped[f] = (double*)mapped_host(dst[f], bytes);
      direct = mapped[f] != nullptr;
    }
  if (direct) {
    k_swimmers_to_host<<<(3 * W->n + 255) / 256, 256, 0, W->copy>>>(
        3 * W->n, W->r, W->v, W->nv, mapped[0], mapped[1], mapped[2]);
    LB_CHECK_LAUNCH(1);
  } else {
    for (int f = 0; f < 3; ++f)
      if (dst[f] && bytes)
        LB_CUDA(cudaMemcpyAsync(dst[f], src[f], bytes, cudaMemcpyDeviceToHost, W->copy));
  }
  LB_CUDA(cudaStreamSynchronize(W->copy));
}

void swimmers_wait(Swimmers* W) {
  if (W->done) LB_CUDA(cudaEventSynchronize(W->done));
}

// SwimmerArray::AddForces (SwimmerArray.cu:114-121).
void swimmers_add_forces(Swimmers* W, Lattice* L) {
  // ends already spread by a Step belong to the base from now on
  if (L->spread.stepped) spread_materialise(L);
  if (L->precision == LBSWIM_F64)
    add_forces_f64(W, L);
  else
    append_ends(W, L);
  swimmers_mark(W, L->stream);
  L->force_version++;
}

// FP64 move of an array, recording the moved swimmers' ends into `to` when given.
static void launch_move_f64(Swimmers* W, Lattice* L, const RecordTarget<double>* to) {
  const Dims D = make_dims(L);
  const double* u = (const double*)L->u;
  if (L->compat & LBSWIM_COMPAT_EXACT_F64) {
    k_swimmers_move_exact<<<(int)((2ll * W->n + EXACT_MOVE_BLOCK - 1) / EXACT_MOVE_BLOCK),
                            EXACT_MOVE_BLOCK, 0, L->stream>>>(
        W->n, W->r, W->v, W->nv, W->common, W->seed, W->step, D, u, L->status);
  } else {
    const bool wide = wide_particle_index(L), many = 2ll * W->n >= MOVE64_MANY_FROM;
    constexpr int FEW = MOVE64_FEW, MANY = MOVE64_MANY;
    auto k = to     ? (wide ? k_swimmers_move_f64<true, FEW, long long>
                            : k_swimmers_move_f64<true, FEW, int>)
             : many ? (wide ? k_swimmers_move_f64<false, MANY, long long>
                            : k_swimmers_move_f64<false, MANY, int>)
                    : (wide ? k_swimmers_move_f64<false, FEW, long long>
                            : k_swimmers_move_f64<false, FEW, int>);
    const int points = !to && many ? MANY : FEW;
    k<<<(int)((2ll * W->n + points - 1) / points), move64_block(points), 0, L->stream>>>(
        W->n, W->r, W->v, W->nv, W->common, W->seed, W->step, D, u, L->status,
        to ? *to : RecordTarget<double>{});
  }
  LB_CHECK_LAUNCH(1);
  swimmers_mark(W, L->stream);
}

// FP32 move of nw arrays in one launch, recording the moved swimmers' ends into `to`
// when given.
static void launch_move_f32(Swimmers* const* w, int nw, Lattice* L,
                            const RecordTarget<float>* to) {
  SwimmerList list;
  const int blocks = list_parts(w, nw, MOVE_SWIMMERS, 1, 0, list);
  if (blocks == 0) return;
  const bool wide = wide_particle_index(L);
  auto k = to ? (wide ? k_swimmers_move_f32<true, long long> : k_swimmers_move_f32<true, int>)
              : (wide ? k_swimmers_move_f32<false, long long> : k_swimmers_move_f32<false, int>);
  k<<<blocks, MOVE_BLOCK, 0, L->stream>>>(list, make_dims(L), (const float4*)L->hydro, L->status,
                                          to ? *to : RecordTarget<float>{});
  LB_CHECK_LAUNCH(1);
  for (int i = 0; i < nw; ++i) swimmers_mark(w[i], L->stream);
}

void swimmers_move(Swimmers* W, Lattice* L) {
  if (W->n > 0) {
    if (L->precision == LBSWIM_F64)
      launch_move_f64(W, L, nullptr);
    else
      launch_move_f32(&W, 1, L, nullptr);
  }
  W->step++;
}

bool swimmers_move_together(Swimmers* const* w, int nw, const Lattice* L) {
  if (nw < 1 || nw > (L->precision == LBSWIM_F64 ? 1 : LIST_ARRAYS)) return false;
  for (int i = 0; i < nw; ++i) {
    if (w[i]->n <= 0) return false;
    for (int j = 0; j < i; ++j)
      if (w[j] == w[i]) return false;
  }
  return true;
}

static int ends_of(Swimmers* const* w, int nw) {
  long long n = 0;
  for (int i = 0; i < nw; ++i) n += 2ll * w[i]->n;
  if (n > 0x7fffffffll) throw LbswimError{LBSWIM_ENOTSUP, "more than 2^30 swimmers on a lattice"};
  return (int)n;
}

// Before the step of a system step: room for the records that its moves will make
// for the next step (reduced precision: in buffers of their own, whose counts
// the step kernel clears).
void swimmers_prepare_room(Swimmers* const* w, int nw, Lattice* L) {
  SpreadScratch::Prepared& P = L->spread.prep;
  P.valid = false;
  P.clear = 0;
  P.clear_max = false;
  if (L->precision == LBSWIM_F64) return;
  const int nends = ends_of(w, nw);
  if (P.capacity_ends < nends) {
    // the buffers may still be read by earlier work on the stream
    LB_CUDA(cudaStreamSynchronize(L->stream));
    if (P.ends) cudaFree(P.ends);
    P.ends = nullptr;
    P.capacity_ends = 0;
    const int cap = std::max(nends + nends / 2, 64);
    LB_CUDA(cudaMalloc(&P.ends, sizeof(EndRecord<float>) * cap));
    P.capacity_ends = cap;
    P.ends_bytes = sizeof(EndRecord<float>) * cap;
  }
  if (!P.max_abs_force) LB_CUDA(cudaMalloc(&P.max_abs_force, 2 * sizeof(unsigned)));
  P.clear_max = true;
  if (nends > DIRECT_ENDS) {
    P.lx = grow_slab_buckets(L, choose_slab_lx(L, nends), P.bucket_count, P.bucket_list,
                             P.bucket_slabs);
    P.clear = slabs_of(slab_grid(L, P.lx));
  }
}

// The moves of lbswim_system_step (after swimmers_prepare_room and the step): the
// moved swimmers' ends are also recorded, and the next step's AddForces takes them
// if nothing changed in between (swimmers_add_forces_prepared).  Several arrays move
// in one launch and are recorded in one: four of 7,800 in a 192x200x208 lattice
// 50 us a step less.  A small suspension's move records it itself, one launch on the
// critical path less; a larger one's ends are recorded, and listed under their
// slabs, by a kernel after it, so that a read-back of the swimmers waits for the
// move only (an upload for both) and one wave of blocks pays the bucket atomics
// once.
void swimmers_move_preparing(Swimmers* const* w, int nw, Lattice* L, unsigned long long epoch) {
  SpreadScratch& S = L->spread;
  SpreadScratch::Prepared& P = S.prep;
  P.valid = false;
  const int nends = ends_of(w, nw);
  if (L->precision == LBSWIM_F64) {
    // records for the kernel that add_forces_f64 would choose, which has run before
    const TileGrid G = force_tiles(L);
    if ((L->compat & LBSWIM_COMPAT_EXACT_F64) || nends > DIRECT_ENDS_F64 ||
        !tiles_take_buckets(G, nends) || S.capacity_ends < nends) {
      swimmers_move(w[0], L);
      return;
    }
    const RecordTarget<double> to{(EndRecord<double>*)S.ends, nullptr, G, nullptr, nullptr};
    launch_move_f64(w[0], L, &to);
  } else if (nends <= DIRECT_ENDS) {
    const RecordTarget<float> to{(EndRecord<float>*)P.ends, P.max_abs_force, TileGrid{}, nullptr,
                                 nullptr};
    launch_move_f32(w, nw, L, &to);
    P.tile = -1;
  } else {
    launch_move_f32(w, nw, L, nullptr);
    launch_end_records(w, nw, L, 0,
                       RecordTarget<float>{(EndRecord<float>*)P.ends, P.max_abs_force,
                                           slab_grid(L, P.lx), P.bucket_count, P.bucket_list});
    for (int i = 0; i < nw; ++i) {
      if (!w[i]->recorded)
        LB_CUDA(cudaEventCreateWithFlags(&w[i]->recorded, cudaEventDisableTiming));
      LB_CUDA(cudaEventRecord(w[i]->recorded, L->stream));
    }
    P.tile = L->fused_tile;
  }
  P.owners = nw;
  for (int i = 0; i < nw; ++i) {
    w[i]->step++;
    P.owner[i] = w[i];
    P.owner_step[i] = w[i]->step;
  }
  P.valid = true;
  P.epoch = epoch;
  P.nends = nends;
}

// AddForces of the arrays (right after ZeroForce) from the prepared records, when
// the last thing that happened to them and to this lattice was that preparing move.
bool swimmers_add_forces_prepared(Swimmers* const* w, int nw, Lattice* L,
                                  unsigned long long epoch) {
  SpreadScratch& S = L->spread;
  SpreadScratch::Prepared& P = S.prep;
  if (!P.valid || P.owners != nw || P.epoch != epoch || S.pending != 0 || S.stepped ||
      P.nends != ends_of(w, nw))
    return false;
  for (int i = 0; i < nw; ++i)
    if (P.owner[i] != w[i] || P.owner_step[i] != w[i]->step) return false;
  if (L->precision == LBSWIM_F64) {
    spread_fixed(L, P.nends, TileChains{});  // DIRECT_ENDS_F64 at most
  } else {
    if (P.tile >= 0 && P.tile != L->fused_tile) return false;
    std::swap(S.ends, P.ends);
    std::swap(S.ends_bytes, P.ends_bytes);
    std::swap(S.capacity_ends, P.capacity_ends);
    std::swap(S.bucket_count, P.bucket_count);
    std::swap(S.bucket_list, P.bucket_list);
    std::swap(S.bucket_slabs, P.bucket_slabs);
    std::swap(S.max_abs_force, P.max_abs_force);
    S.bucket_tile = P.tile;  // -1: no buckets
    S.lx = P.lx;
    S.pending = P.nends;
  }
  P.valid = false;
  for (int i = 0; i < nw; ++i) swimmers_mark(w[i], L->stream);
  L->force_version++;
  return true;
}

// ---- tracer work order ------------------------------------------------------------
// Tracer cells of 4 x 4 x 8 sites, z fastest: a block's 256 tracers lie in a
// 4 x 4 x 256 run along z, whose stencil rows share more cache lines than a
// cube's (3 us per coupled step less than 8 x 8 x 8 cells at 256^3).
constexpr int TR_BINX = 4, TR_BINY = 4, TR_BINZ = 8;

__global__ void k_tr_bin(int n, const double* __restrict__ r, Dims D, int nb1, int nb2,
                         int* __restrict__ bin_of, unsigned* __restrict__ count) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int c[3];
  for (int d = 0; d < 3; ++d)
    c[d] = wrap_any((int)floor(r[n * d + k]), D.n[d]) / (d == 0 ? TR_BINX : d == 1 ? TR_BINY : TR_BINZ);
  const int b = (c[0] * nb1 + c[1]) * nb2 + c[2];
  bin_of[k] = b;
  atomicAdd(count + b, 1u);
}

__global__ void k_tr_permute(int n, const int* __restrict__ bin_of, unsigned* __restrict__ count,
                             const unsigned* __restrict__ start, const double* __restrict__ r,
                             const double* __restrict__ s, const double* __restrict__ v,
                             const int* __restrict__ perm, double* __restrict__ r2,
                             double* __restrict__ s2, double* __restrict__ v2,
                             int* __restrict__ perm2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int b = bin_of[k];
  const unsigned slot = start[b] + atomicSub(count + b, 1u) - 1u;
  for (int d = 0; d < 3; ++d) {
    r2[(long long)n * d + slot] = r[(long long)n * d + k];
    s2[(long long)n * d + slot] = s[(long long)n * d + k];
    v2[(long long)n * d + slot] = v[(long long)n * d + k];
  }
  perm2[slot] = perm[k];
}

__global__ void k_iota(int n, int* __restrict__ p) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) p[k] = k;
}

// dst[d][k] = src[d][perm[k]] (user order -> work order) or the inverse.
template <bool TO_WORK>
__global__ void k_tr_reorder(int n, const int* __restrict__ perm, const double* __restrict__ src,
                             double* __restrict__ dst) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int u = perm[k];
  for (int d = 0; d < 3; ++d) {
    if (TO_WORK)
      dst[(long long)n * d + k] = src[(long long)n * d + u];
    else
      dst[(long long)n * d + u] = src[(long long)n * d + k];
  }
}

// Any non-finite value among n doubles sets *flag.
__global__ void k_any_nonfinite(const double* __restrict__ a, long long n,
                                unsigned* __restrict__ flag) {
  unsigned bad = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    bad |= !(fabs(a[i]) <= 1.7976931348623157e308);
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1u);
}

// The check runs on the device, on the uploaded copy: a host scan of the
// caller's buffer by one core reads it several times slower than the link
// delivers it (1M tracer positions: ~1.2 ms against 0.12 ms for the copy).
void upload_checked_finite(double* stage, const double* host, long long n, unsigned* flag,
                           const char* what) {
  if (n <= 0) return;
  LB_CUDA(cudaMemcpy(stage, host, sizeof(double) * n, cudaMemcpyHostToDevice));
  LB_CUDA(cudaMemset(flag, 0, sizeof(unsigned)));
  const long long blocks = std::min<long long>((n + 255) / 256, 152LL * 8);
  k_any_nonfinite<<<(int)blocks, 256>>>(stage, n, flag);
  LB_CHECK_LAUNCH(1);
  unsigned bad = 0;
  LB_CUDA(cudaMemcpy(&bad, flag, sizeof(unsigned), cudaMemcpyDeviceToHost));
  if (bad) throw LbswimError{LBSWIM_EINVAL, std::string(what) + " holds a non-finite value"};
}

void tracers_alloc(Tracers* T) {
  const size_t n = (size_t)(T->n > 0 ? T->n : 1);
  double** bufs[] = {&T->r, &T->s, &T->v, &T->r2, &T->s2, &T->v2, &T->staging};
  for (double** b : bufs) {
    LB_CUDA(cudaMalloc(b, sizeof(double) * 3 * n));
    LB_CUDA(cudaMemset(*b, 0, sizeof(double) * 3 * n));
  }
  LB_CUDA(cudaMalloc(&T->perm, sizeof(int) * n));
  LB_CUDA(cudaMalloc(&T->perm2, sizeof(int) * n));
  LB_CUDA(cudaMalloc(&T->bin_of, sizeof(int) * n));
  LB_CUDA(cudaMalloc(&T->flag, 256));
  k_iota<<<(int)((n + 255) / 256), 256>>>((int)n, T->perm);
  LB_CHECK_LAUNCH(1);
  LB_CUDA(cudaDeviceSynchronize());
}

void tracers_free(Tracers* T) {
  if (T->side) {
    cudaStreamSynchronize(T->side);
    cudaStreamDestroy(T->side);
    cudaEventDestroy(T->done);
    T->side = nullptr;
  }
  void* ptrs[] = {T->r,    T->s,      T->v,      T->r2,        T->s2,        T->v2,
                  T->perm, T->perm2,  T->bin_of, T->staging,   T->bin_count, T->bin_start,
                  T->scan_tmp, T->flag};
  for (void* p : ptrs)
    if (p) cudaFree(p);
}

static double* tr_field_ptr(Tracers* T, int field) {
  return field == LBSWIM_TR_R ? T->r : (field == LBSWIM_TR_S ? T->s : T->v);
}

void tracers_h2d(Tracers* T, int field, const double* host) {
  LB_CUDA(cudaDeviceSynchronize());  // particle arrays are not bound to one stream
  if (T->n <= 0) return;
  double* dst = tr_field_ptr(T, field);
  const size_t bytes = sizeof(double) * 3 * T->n;
  // positions must be finite: checked on the staged copy, before the field
  // changes
  const bool check = field == LBSWIM_TR_R;
  if (check)
    upload_checked_finite(T->staging, host, 3LL * T->n, T->flag, "tracer positions");
  if (T->identity) {
    if (check) {
      LB_CUDA(cudaMemcpyAsync(dst, T->staging, bytes, cudaMemcpyDeviceToDevice, 0));
      LB_CUDA(cudaStreamSynchronize(0));
    } else {
      LB_CUDA(cudaMemcpy(dst, host, bytes, cudaMemcpyHostToDevice));
    }
  } else {
    if (!check) LB_CUDA(cudaMemcpy(T->staging, host, bytes, cudaMemcpyHostToDevice));
    k_tr_reorder<true><<<(T->n + 255) / 256, 256>>>(T->n, T->perm, T->staging, dst);
    LB_CHECK_LAUNCH(1);
    LB_CUDA(cudaDeviceSynchronize());
  }
  if (field == LBSWIM_TR_R) T->needs_sort = true;
}

void tracers_d2h(Tracers* T, int field, double* host) {
  LB_CUDA(cudaDeviceSynchronize());
  if (T->n <= 0) return;
  const double* src = tr_field_ptr(T, field);
  if (T->identity) {
    LB_CUDA(cudaMemcpy(host, src, sizeof(double) * 3 * T->n, cudaMemcpyDeviceToHost));
  } else {
    k_tr_reorder<false><<<(T->n + 255) / 256, 256>>>(T->n, T->perm, src, T->staging);
    LB_CHECK_LAUNCH(1);
    LB_CUDA(cudaMemcpy(host, T->staging, sizeof(double) * 3 * T->n, cudaMemcpyDeviceToHost));
  }
}

static void tracers_sort(Tracers* T, Lattice* L, cudaStream_t stream) {
  const Dims D = make_dims(L);
  const int nb0 = (D.n[0] + TR_BINX - 1) / TR_BINX, nb1 = (D.n[1] + TR_BINY - 1) / TR_BINY,
            nb2 = (D.n[2] + TR_BINZ - 1) / TR_BINZ;
  const int nbins = nb0 * nb1 * nb2;
  if (T->nbins != nbins) {
    LB_CUDA(cudaStreamSynchronize(stream));
    if (T->bin_count) cudaFree(T->bin_count);
    if (T->bin_start) cudaFree(T->bin_start);
    if (T->scan_tmp) cudaFree(T->scan_tmp);
    T->bin_count = T->bin_start = T->scan_tmp = nullptr;
    LB_CUDA(cudaMalloc(&T->bin_count, sizeof(unsigned) * nbins));
    LB_CUDA(cudaMalloc(&T->bin_start, sizeof(unsigned) * (nbins + 1)));
    LB_CUDA(cudaMalloc(&T->scan_tmp, sizeof(unsigned) * ((nbins + SCAN_TILE - 1) / SCAN_TILE)));
    LB_CUDA(cudaMemsetAsync(T->bin_count, 0, sizeof(unsigned) * nbins, stream));
    T->nbins = nbins;
  }
  const int g = (T->n + 255) / 256;
  k_tr_bin<<<g, 256, 0, stream>>>(T->n, T->r, D, nb1, nb2, T->bin_of, T->bin_count);
  const int nscan = (nbins + SCAN_TILE - 1) / SCAN_TILE;
  k_scan_tiles<<<nscan, SCAN_THREADS, 0, stream>>>(T->bin_count, nbins, T->scan_tmp);
  k_scan_top<<<1, 1024, 0, stream>>>(T->scan_tmp, nscan);
  k_scan_apply<<<nscan, SCAN_THREADS, 0, stream>>>(T->bin_count, nbins, T->scan_tmp,
                                                      T->bin_start, (unsigned)T->n);
  k_tr_permute<<<g, 256, 0, stream>>>(T->n, T->bin_of, T->bin_count, T->bin_start, T->r,
                                         T->s, T->v, T->perm, T->r2, T->s2, T->v2, T->perm2);
  LB_CHECK_LAUNCH(5);
  std::swap(T->r, T->r2);
  std::swap(T->s, T->s2);
  std::swap(T->v, T->v2);
  std::swap(T->perm, T->perm2);
  T->identity = false;
  T->needs_sort = false;
  T->moves_since_sort = 0;
}

static void tracers_move_on(Tracers* T, Lattice* L, cudaStream_t stream) {
  if (T->needs_sort || T->moves_since_sort >= TRACER_RESORT_MOVES) tracers_sort(T, L, stream);
  T->moves_since_sort++;
  const Dims D = make_dims(L);
  if (L->precision == LBSWIM_F64) {
    const double* u = (const double*)L->u;
    if (L->compat & LBSWIM_COMPAT_EXACT_F64) {
      k_tracers_move_exact<<<(T->n + EXACT_MOVE_BLOCK - 1) / EXACT_MOVE_BLOCK, EXACT_MOVE_BLOCK,
                             0, stream>>>(T->n, T->r, T->s, T->v, D, u, L->status);
    } else {
      const bool far = wide_particle_index(L), many = T->n >= MOVE64_MANY_FROM;
      const int points = many ? MOVE64_MANY : MOVE64_FEW;
      auto k = many ? (far ? k_tracers_move_f64<MOVE64_MANY, long long>
                           : k_tracers_move_f64<MOVE64_MANY, int>)
                    : (far ? k_tracers_move_f64<MOVE64_FEW, long long>
                           : k_tracers_move_f64<MOVE64_FEW, int>);
      k<<<(T->n + points - 1) / points, move64_block(points), 0, stream>>>(T->n, T->r, T->s, T->v,
                                                                           D, u, L->status);
    }
  }
  else {
    const bool far = wide_particle_index(L), wide = T->n >= TRACERS_WIDE_FROM;
    const int per = wide ? WIDE_TRACERS : MOVE_POINTS;
    auto k = wide ? (far ? k_tracers_move_f32<true, long long> : k_tracers_move_f32<true, int>)
                  : (far ? k_tracers_move_f32<false, long long> : k_tracers_move_f32<false, int>);
    k<<<(T->n + per - 1) / per, MOVE_BLOCK, 0, stream>>>(T->n, T->r, T->s, T->v, D, L->hydro,
                                                         L->status);
  }
  LB_CHECK_LAUNCH(1);
}

void tracers_move(Tracers* T, Lattice* L) {
  if (T->n <= 0) return;
  if (T->side_pending) LB_CUDA(cudaStreamWaitEvent(L->stream, T->done, 0));
  tracers_move_on(T, L, L->stream);
}

void tracers_move_async(Tracers* T, Lattice* L) {
  if (T->n <= 0) return;
  if (!T->side) {
    // Least priority: when the lattice's stream has a higher one, the next
    // step's blocks are dispatched ahead of tracer blocks still queued, and the
    // tracer move fills the SMs the step leaves idle.
    int least = 0, greatest = 0;
    LB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    LB_CUDA(cudaStreamCreateWithPriority(&T->side, cudaStreamNonBlocking, least));
    LB_CUDA(cudaEventCreateWithFlags(&T->done, cudaEventDisableTiming));
  }
  LB_CUDA(cudaStreamWaitEvent(T->side, L->hydro_ready, 0));
  tracers_move_on(T, L, T->side);
  LB_CUDA(cudaEventRecord(T->done, T->side));
  T->side_pending = true;
  cudaEvent_t ev;
  if (L->reader_pool.empty()) {
    LB_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  } else {
    ev = L->reader_pool.back();
    L->reader_pool.pop_back();
  }
  LB_CUDA(cudaEventRecord(ev, T->side));
  L->readers.emplace_back(L->precision == LBSWIM_F64 ? (const void*)L->u : (const void*)L->hydro, ev);
}

void lattice_interp_velocity(Lattice* L, int np, const double* r_host, double* v_host) {
  if (np <= 0) return;
  const Dims D = make_dims(L);
  double *r = nullptr, *v = nullptr;
  LB_CUDA(cudaMalloc(&r, sizeof(double) * 3 * np));
  cudaError_t e = cudaMalloc(&v, sizeof(double) * 3 * np);
  if (e != cudaSuccess) {
    cudaFree(r);
    LB_CUDA(e);
  }
  try {
    LB_CUDA(cudaMemcpyAsync(r, r_host, sizeof(double) * 3 * np, cudaMemcpyHostToDevice, L->stream));
    if (L->precision == LBSWIM_F64)
      k_interp_points<double, double><<<(np + 255) / 256, 256, 0, L->stream>>>(np, r, v, D,
                                                                              (const double*)L->u);
    else
      k_interp_points<float4, float><<<(np + 255) / 256, 256, 0, L->stream>>>(np, r, v, D,
                                                                             L->hydro);
    LB_CHECK_LAUNCH(1);
    LB_CUDA(cudaMemcpyAsync(v_host, v, sizeof(double) * 3 * np, cudaMemcpyDeviceToHost, L->stream));
    LB_CUDA(cudaStreamSynchronize(L->stream));
  } catch (...) {
    cudaFree(r);
    cudaFree(v);
    throw;
  }
  cudaFree(r);
  cudaFree(v);
}

// ---- allocation-free spreading ------------------------------------------------
// Scratch of lbswim_spread_forces_noalloc: one file-scope device array that
// every GPU loading the library holds until exit.  Layout (bytes):
//   bin counts [NOALLOC_MAX_BINS] | bin starts [NOALLOC_MAX_BINS + 1] |
//   scan tile sums | end order [NOALLOC_MAX_ENDS] | end records [NOALLOC_MAX_ENDS]
constexpr int NOALLOC_MAX_ENDS = 2 * LBSWIM_NOALLOC_MAX_SWIMMERS;
constexpr int NOALLOC_MAX_BINS = LBSWIM_NOALLOC_MAX_SPREAD_BINS;
constexpr size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t NA_COUNT = 0;
constexpr size_t NA_START = NA_COUNT + align256(sizeof(unsigned) * NOALLOC_MAX_BINS);
constexpr size_t NA_TILES = NA_START + align256(sizeof(unsigned) * (NOALLOC_MAX_BINS + 1));
constexpr size_t NA_ORDER =
    NA_TILES + align256(sizeof(unsigned) * ((NOALLOC_MAX_BINS + SCAN_TILE - 1) / SCAN_TILE));
constexpr size_t NA_ENDS = NA_ORDER + align256(sizeof(int) * NOALLOC_MAX_ENDS);
constexpr size_t NA_BYTES = NA_ENDS + align256(sizeof(EndRecord<double>) * NOALLOC_MAX_ENDS);

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

// Device address of g_noalloc_scratch, looked up once per device with that
// device current (the symbol's name in host code is only a stand-in).
static unsigned char* noalloc_scratch_for_current_device() {
  static std::mutex mu;
  static unsigned char* addr[64] = {nullptr};
  int dev = 0;
  LB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) throw LbswimError{LBSWIM_ENOTSUP, "device index out of range"};
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    LB_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    addr[dev] = (unsigned char*)p;
  }
  return addr[dev];
}

void spread_forces_noalloc(const double* r, const double* nv, int nsw, double P, double l,
                           const int size[3], double* force, int accumulate,
                           cudaStream_t stream) {
  Dims D;
  for (int a = 0; a < 3; ++a) {
    D.n[a] = size[a];
    D.nb[a] = (size[a] + BIN - 1) / BIN;
  }
  D.N = (long long)size[0] * size[1] * size[2];
  const long long nbins = (long long)D.nb[0] * D.nb[1] * D.nb[2];
  // Every limit is checked before anything is enqueued (the swimmer count
  // before it is doubled, so that no count can wrap past the check).
  if (nsw < 0 || nsw > LBSWIM_NOALLOC_MAX_SWIMMERS)
    throw LbswimError{LBSWIM_EINVAL, "swimmer count outside the allocation-free limit of 0.." +
                                         std::to_string(LBSWIM_NOALLOC_MAX_SWIMMERS)};
  if (nbins > NOALLOC_MAX_BINS)
    throw LbswimError{LBSWIM_EINVAL,
                      "lattice larger than the allocation-free limit (" +
                          std::to_string(NOALLOC_MAX_BINS) + " spread bins of 4^3 sites)"};
  // the gather's grid is (ceil(nz / 32), ceil(ny / 8), nx) blocks
  if (D.n[0] > 65535 || (D.n[1] + 7) / 8 > 65535)
    throw LbswimError{LBSWIM_EINVAL, "lattice axes beyond the allocation-free limit "
                                     "(nx <= 65535, ny <= 524280)"};
  const int nends = 2 * nsw;
  unsigned char* base = noalloc_scratch_for_current_device();
  unsigned* bin_count = (unsigned*)(base + NA_COUNT);
  unsigned* bin_start = (unsigned*)(base + NA_START);
  unsigned* tiles = (unsigned*)(base + NA_TILES);
  int* order = (int*)(base + NA_ORDER);
  EndRecord<double>* ends = (EndRecord<double>*)(base + NA_ENDS);
  // The array keeps the previous call's contents: the counts must start at zero.
  LB_CUDA(cudaMemsetAsync(bin_count, 0, sizeof(unsigned) * nbins, stream));
  const int nb = (int)nbins;
  if (nends > 0) {
    k_spread_bin<double><<<(nends + 255) / 256, 256, 0, stream>>>(nsw, r, nv, P, l, D, ends,
                                                                  bin_count);
    LB_CHECK_LAUNCH(1);
  }
  const int ntiles = (nb + SCAN_TILE - 1) / SCAN_TILE;
  k_scan_tiles<<<ntiles, SCAN_THREADS, 0, stream>>>(bin_count, nb, tiles);
  k_scan_top<<<1, 1024, 0, stream>>>(tiles, ntiles);
  k_scan_apply<<<ntiles, SCAN_THREADS, 0, stream>>>(bin_count, nb, tiles, bin_start,
                                                    (unsigned)nends);
  LB_CHECK_LAUNCH(3);
  if (nends > 0) {
    k_spread_scatter<double><<<(nends + 255) / 256, 256, 0, stream>>>(nends, ends, D, bin_count,
                                                                      bin_start, order);
    k_spread_sort<<<(nb + 255) / 256, 256, 0, stream>>>(nb, bin_start, order);
    LB_CHECK_LAUNCH(2);
  }
  dim3 grid((D.n[2] + 31) / 32, (D.n[1] + 7) / 8, D.n[0]);
  k_spread_gather<double><<<grid, dim3(32, 8), 0, stream>>>(D, ends, bin_start, order, force,
                                                            accumulate);
  LB_CHECK_LAUNCH(1);
}

void lattice_init_random(Lattice* L, unsigned long long seed, double amp) {
  const bool packed = L->precision != LBSWIM_F64;
  if (packed) L->rho0 = 1.0;  // as a new lattice: the same stored bits whatever came before
  k_init_density<<<(int)std::min<long long>((L->n + 255) / 256, 152LL * 32), 256, 0, L->stream>>>(
      L->n, seed, amp, L->rho0, packed ? nullptr : (double*)L->rho,
      packed ? nullptr : (double*)L->u, packed ? L->hydro : nullptr);
  LB_CHECK_LAUNCH(1);
  L->shadow_f_version = 0;
  lattice_init_from_hydro(L);
}

void swimmers_init_random(Swimmers* W, const Lattice* L, unsigned long long seed) {
  LB_CUDA(cudaDeviceSynchronize());
  if (W->n > 0) {
    k_init_particles<<<(W->n + 255) / 256, 256>>>(W->n, seed, make_dims(L), W->r, W->nv, W->v,
                                                   nullptr);
    LB_CHECK_LAUNCH(1);
  }
  LB_CUDA(cudaDeviceSynchronize());
}

void tracers_init_random(Tracers* T, const Lattice* L, unsigned long long seed) {
  LB_CUDA(cudaDeviceSynchronize());
  if (T->n > 0) {
    // user order = work order until the next re-binning
    k_iota<<<(T->n + 255) / 256, 256>>>(T->n, T->perm);
    k_init_particles<<<(T->n + 255) / 256, 256>>>(T->n, seed, make_dims(L), T->r, nullptr, T->s,
                                                   T->v);
    LB_CHECK_LAUNCH(2);
    T->identity = true;
    T->needs_sort = true;
    T->moves_since_sort = 0;
  }
  LB_CUDA(cudaDeviceSynchronize());
}

void rng_draws(unsigned long long seed, int n, unsigned long long step, float* u_host,
               double* g_host) {
  if (n <= 0) return;
  float* u = nullptr;
  double* g = nullptr;
  LB_CUDA(cudaMalloc(&u, sizeof(float) * n));
  cudaError_t e = cudaMalloc(&g, sizeof(double) * 3 * n);
  if (e != cudaSuccess) {
    cudaFree(u);
    LB_CUDA(e);
  }
  k_rng_draws<<<(n + 255) / 256, 256>>>(seed, n, step, u, g);
  cudaError_t le = cudaGetLastError();
  if (le == cudaSuccess) le = cudaMemcpy(u_host, u, sizeof(float) * n, cudaMemcpyDeviceToHost);
  if (le == cudaSuccess) le = cudaMemcpy(g_host, g, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost);
  cudaFree(u);
  cudaFree(g);
  LB_CUDA(le);
  count_launches(1);
}

}  // namespace lbswim
