// Spatial sort and dead-particle removal of one species
// (Particles::SortSpatially / RemoveDead,
// src/framework/containers/particles_sort.cpp:103-253).
//
// The reference bins with Kokkos::BinSort (sort_within_bins = false), whose
// order inside a cell is unspecified. This sort produces the stable order
// (ascending original index inside every cell), which is one of the orders
// the reference may produce, and is deterministic:
//   1. key per particle (PositionToTileIndex, src/global/utils/sorting.h:
//      119-135: (i1*n2 + i2)*n3 + i3; dead -> last bin) and a count per bin;
//      the counting atomics (one per group of a warp's lanes with one key)
//      return each particle's place in its bin, in arrival order;
//   2. exclusive scan of the counts -> bin offsets; the dead are counted per
//      block of particles, whose scan places them in order;
//   3. every particle's arrays are packed into one record at its place;
//   4. a pass over the records writes them back into the arrays, each bin in
//      ascending original index: a particle's place in its bin is the number
//      of smaller indices there (bins above kBigBin are sorted first).
// Packed records instead of one gather per array: a random particle order
// touches two 32-byte sectors per particle instead of one per array (11 in
// FP32 3D), and nothing is copied back. 2 x 16.8 M particles in random order
// (128^3 cells, with the injection) went from 9.45 to 2.92 ms.
// Nothing here synchronises with the host; the dead count stays on the
// device until the caller reads it.
#include <climits>
#include <type_traits>

#include <cuda_runtime.h>

#include "sort.cuh"

namespace pic {

namespace {

constexpr int kScanThreads = 512;
constexpr int kScanItems   = 8;
constexpr int kScanTile    = kScanThreads * kScanItems;

template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* sh, T& total) {
  // warp inclusive scan
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  T         x    = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[wid] = x;
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    T         s  = lane < nw ? sh[lane] : (T)0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) sh[lane] = s;
  }
  __syncthreads();
  const T warp_off = wid > 0 ? sh[wid - 1] : (T)0;
  total            = sh[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_off + x - v;
}

// per-tile sums of in[0..n)
template <typename Tin, typename T>
__global__ void k_tile_sums(const Tin* in, int64_t n, T* sums) {
  __shared__ T  sh[32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  T             s    = 0;
#pragma unroll
  for (int it = 0; it < kScanItems; ++it) {
    const int64_t i = base + (int64_t)it * kScanThreads + threadIdx.x;
    if (i < n) s += (T)in[i];
  }
  T total;
  block_exclusive_scan<T>(s, sh, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// exclusive scan of one tile with a carried-in offset per tile
template <typename Tin, typename T>
__global__ void k_tile_scan(const Tin* in, int64_t n, const T* tile_off, T* out) {
  __shared__ T  sh[32];
  __shared__ T  carry;
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  if (threadIdx.x == 0) carry = tile_off ? tile_off[blockIdx.x] : (T)0;
  __syncthreads();
  // each thread owns kScanItems consecutive elements
  T         v[kScanItems];
  T         s  = 0;
  const int t0 = threadIdx.x * kScanItems;
#pragma unroll
  for (int it = 0; it < kScanItems; ++it) {
    const int64_t i = base + t0 + it;
    v[it]           = i < n ? (T)in[i] : (T)0;
    s += v[it];
  }
  T total;
  T pre = block_exclusive_scan<T>(s, sh, total) + carry;
#pragma unroll
  for (int it = 0; it < kScanItems; ++it) {
    const int64_t i = base + t0 + it;
    if (i < n) out[i] = pre;
    pre += v[it];
  }
}

}  // namespace

// exclusive scan (out may alias in only through separate buffers)
template <typename Tin, typename T>
cudaError_t exclusive_scan(const Tin* in, int64_t n, T* out, ScanScratch<T>& scr, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles == 1) {
    PIC_KL(k_tile_scan<Tin, T><<<1, kScanThreads, 0, s>>>(in, n, (const T*)nullptr, out));
    return cudaGetLastError();
  }
  T* sums = scr.get(tiles * 2 + 2, s);
  if (!sums) return cudaErrorMemoryAllocation;
  T* offs = sums + tiles + 1;
  PIC_KL(k_tile_sums<Tin, T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, sums));
  // recursive scan of the tile sums (depth log_4096(n))
  ScanScratch<T> sub;
  cudaError_t    e = exclusive_scan<T, T>(sums, tiles, offs, sub, s);
  if (e != cudaSuccess) {
    sub.release(s);
    return e;
  }
  PIC_KL(k_tile_scan<Tin, T><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, offs, out));
  e = cudaGetLastError();
  sub.release(s);
  return e;
}

template cudaError_t exclusive_scan<int32_t, int64_t>(const int32_t*, int64_t, int64_t*,
                                                      ScanScratch<int64_t>&, cudaStream_t);
template cudaError_t exclusive_scan<int64_t, int64_t>(const int64_t*, int64_t, int64_t*,
                                                      ScanScratch<int64_t>&, cudaStream_t);
template cudaError_t exclusive_scan<int32_t, int32_t>(const int32_t*, int64_t, int32_t*,
                                                      ScanScratch<int32_t>&, cudaStream_t);

namespace {

// Place of the cell lx within its tile row: the even cells first, then the
// odd ones. A warp's lanes then cover cells two apart, whose order-2 support
// boxes never start on the same node, so fewer of their J-window atomics
// fall on one word; the window reads stay in distinct banks.
__device__ __forceinline__ int tile_row_slot(int lx, int tx) {
  return (lx & 1) ? (tx + 1) / 2 + lx / 2 : lx / 2;
}

// the bin of one particle; ok = false for a live particle outside the grid
// (kept with the dead, tag untouched)
__device__ __forceinline__ int32_t sort_key(const SortArgs& a, short tag, int i1, int i2, int i3,
                                            bool& ok) {
  ok = true;
  if (tag != PIC_TAG_ALIVE) return a.dead_bin;
  if (!a.spatial) return 0;
  ok = i1 >= 0 && i1 < a.n[0] && i2 >= 0 && i2 < a.n[1] && (a.dim == 2 || (i3 >= 0 && i3 < a.n[2]));
  if (!ok) return a.dead_bin;
  if (a.tiled) {
    const int tx = i1 >> a.tile_log[0], ty = i2 >> a.tile_log[1], tz = i3 >> a.tile_log[2];
    const int sx = 1 << a.tile_log[0];
    const int lx = i1 & (sx - 1), ly = i2 & ((1 << a.tile_log[1]) - 1),
              lz = i3 & ((1 << a.tile_log[2]) - 1);
    const int t  = (tz * a.ntiles[1] + ty) * a.ntiles[0] + tx;
    return (((((t << a.tile_log[2]) + lz) << a.tile_log[1]) + ly) << a.tile_log[0]) +
           tile_row_slot(lx, sx);
  }
  return a.dim == 2 ? i1 * a.n[1] + i2 : (i1 * a.n[1] + i2) * a.n[2] + i3;
}

__device__ __forceinline__ int32_t sort_key_at(const SortArgs& a, int64_t p, bool& ok) {
  return sort_key(a, a.tag[p], a.i[0][p], a.i[1][p], a.dim == 3 ? a.i[2][p] : 0, ok);
}

// 1. places within the bins and counts; the dead per block
__global__ void __launch_bounds__(256) k_keys(SortArgs a) {
  __shared__ int s_dead;
  const int64_t  p0 = (int64_t)blockIdx.x * kSortBlock;
  const int      lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_dead = 0;
  __syncthreads();
  int dead = 0;
  for (int it = 0; it < kSortBlock / 256; ++it) {
    const int64_t p   = p0 + it * 256 + threadIdx.x;
    int32_t       key = -1;
    bool          ok  = true;
    if (p < a.npart) key = sort_key_at(a, p, ok);
    if (!ok) atomicAdd(a.err + ERR_OUT_OF_GRID, 1ull);
    dead += key == a.dead_bin;
    if (!a.spatial) continue;
    // one atomic for the lanes of a warp that share a bin
    const unsigned peers  = __match_any_sync(0xffffffffu, key);
    const int      leader = __ffs(peers) - 1, cnt = __popc(peers);
    const bool     live   = key >= 0 && key != a.dead_bin;
    int            base   = 0;
    if (lane == leader && live) {
      base = atomicAdd(a.count + key, cnt);
      if (base <= kBigBin && base + cnt > kBigBin) a.big[atomicAdd(a.nbig, 1)] = key;
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    if (live) a.rank[p] = base + __popc(peers & ((1u << lane) - 1u));
  }
  dead = __reduce_add_sync(0xffffffffu, dead);
  if (lane == 0 && dead) atomicAdd(&s_dead, dead);
  __syncthreads();
  if (threadIdx.x == 0) {
    a.dead_cnt[blockIdx.x] = s_dead;
    if (s_dead) atomicAdd(a.count + a.dead_bin, s_dead);
    if (!a.spatial) {  // one bin of the living
      const int64_t here = a.npart - p0 < kSortBlock ? a.npart - p0 : kSortBlock;
      atomicAdd(a.count, (int)here - s_dead);
    }
  }
}

// one particle's arrays as 32-bit words: cells, offsets, [previous ones],
// momenta and weight, tag, original index
template <int D, int RW, bool PREV>
struct SortRec {
  static constexpr int DIM  = D;
  static constexpr int DATA = (PREV ? 4 : 2) * D + 4 * RW + 1;  // words before the index
  static constexpr int Q    = (DATA + 1 + 7) / 8 * 2;           // 16-byte words, whole 32-byte sectors
  unsigned w[4 * Q];
  __device__ __forceinline__ void load(const SortArgs& a, int64_t p) {
    int k = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) w[k++] = (unsigned)a.i[d][p];
#pragma unroll
    for (int d = 0; d < D; ++d) w[k++] = __float_as_uint(a.dx[d][p]);
    if constexpr (PREV) {
#pragma unroll
      for (int d = 0; d < D; ++d) w[k++] = (unsigned)a.ip[d][p];
#pragma unroll
      for (int d = 0; d < D; ++d) w[k++] = __float_as_uint(a.dxp[d][p]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if constexpr (RW == 1) {
        w[k++] = ((const unsigned*)a.u[c])[p];
      } else {
        const uint2 v = ((const uint2*)a.u[c])[p];
        w[k++] = v.x, w[k++] = v.y;
      }
    }
    w[k++] = (unsigned short)a.tag[p];
    w[k++] = (unsigned)p;
#pragma unroll
    for (; k < 4 * Q; ++k) w[k] = 0u;
  }
  __device__ __forceinline__ void store(const SortArgs& a, int64_t p) const {
    int k = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) a.i[d][p] = (int)w[k++];
#pragma unroll
    for (int d = 0; d < D; ++d) a.dx[d][p] = __uint_as_float(w[k++]);
    if constexpr (PREV) {
#pragma unroll
      for (int d = 0; d < D; ++d) a.ip[d][p] = (int)w[k++];
#pragma unroll
      for (int d = 0; d < D; ++d) a.dxp[d][p] = __uint_as_float(w[k++]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if constexpr (RW == 1) {
        ((unsigned*)a.u[c])[p] = w[k++];
      } else {
        ((uint2*)a.u[c])[p] = make_uint2(w[k], w[k + 1]);
        k += 2;
      }
    }
    a.tag[p] = (int16_t)(uint16_t)w[k];
  }
  __device__ __forceinline__ short tag() const { return (short)(uint16_t)w[DATA - 1]; }
  __device__ __forceinline__ int32_t index() const { return (int32_t)w[DATA]; }
};
// perm only (no records)
struct NoRec {
  static constexpr int Q = 1;
};

// 3. the records packed to their places (or, without records, the
// permutation). A warp's records pass through shared memory, so that
// consecutive lanes write one record's consecutive 16-byte words.
template <typename R>
__global__ void __launch_bounds__(256) k_scatter(SortArgs a) {
  constexpr bool PACK = !std::is_same_v<R, NoRec>;
  __shared__ uint4   s_rec[PACK ? 256 * R::Q : 1];
  __shared__ int64_t s_pos[256];
  __shared__ int     s_warp[8];
  const int64_t p0 = (int64_t)blockIdx.x * kSortBlock;
  const int     lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // dead particles before the block's next 256, and whether it holds any
  int64_t    dead0    = a.dead_off[blockIdx.x];
  const bool any_dead = a.dead_cnt[blockIdx.x] != 0;
  for (int it = 0; it < kSortBlock / 256; ++it) {
    const int64_t p = p0 + it * 256 + threadIdx.x;
    if (p0 + it * 256 >= a.npart) break;  // the same for the whole block
    int32_t key = -1;
    bool    ok;
    R       r;
    if (p < a.npart) {
      if constexpr (PACK) {
        r.load(a, p);
        key = sort_key(a, r.tag(), (int)r.w[0], (int)r.w[1], R::DIM == 3 ? (int)r.w[2] : 0, ok);
      } else {
        key = sort_key_at(a, p, ok);
      }
    }
    const bool dead   = key == a.dead_bin;
    int64_t    before = dead0;  // dead particles before p
    if (any_dead) {
      const unsigned ball = __ballot_sync(0xffffffffu, dead);
      if (lane == 0) s_warp[wid] = __popc(ball);
      __syncthreads();
      int total = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        if (w < wid) before += s_warp[w];
        total += s_warp[w];
      }
      before += __popc(ball & ((1u << lane) - 1u));
      dead0 += total;
      __syncthreads();
    }
    int64_t pos = -1;
    if (key >= 0)
      pos = dead ? a.off[key] + before : (a.spatial ? a.off[key] + a.rank[p] : p - before);
    if constexpr (PACK) {
      uint4* mine = s_rec + wid * (32 * R::Q);
#pragma unroll
      for (int q = 0; q < R::Q; ++q)
        mine[lane * R::Q + q] =
            make_uint4(r.w[4 * q], r.w[4 * q + 1], r.w[4 * q + 2], r.w[4 * q + 3]);
      s_pos[threadIdx.x] = pos;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < R::Q; ++q) {
        const int     e = q * 32 + lane, t = e / R::Q;
        const int64_t d = s_pos[wid * 32 + t];
        if (d >= 0) a.rec[d * R::Q + e % R::Q] = mine[e];
      }
      __syncwarp();
    } else if (pos >= 0) {
      a.perm[pos] = (int32_t)p;
    }
  }
}

// the original index of the particle at place p after the scatter
template <typename R>
__device__ __forceinline__ int32_t index_at(const SortArgs& a, int64_t p) {
  if constexpr (std::is_same_v<R, NoRec>) return a.perm[p];
  else return (int32_t)((const unsigned*)a.rec)[p * (4 * R::Q) + R::DATA];
}

// bins above kBigBin: their indices put in order in a.rank (free after the
// scatter) by rank counting (O(m^2 / threads)); blocks stride over the bins
// the counting listed, whose number only the device knows. The indices are counted
// from shared memory, 1024 at a time: read from the records, which lie 64 bytes
// apart, 12^3 bins of 1500 took a sort of 2.86 ms
// (1.08 so; 1.75 with the indices in an array of their own).
template <typename R>
__global__ void __launch_bounds__(256) k_fix_big(SortArgs a) {
  __shared__ int4 s_idx[256];
  const int nbig = *a.nbig, tid = threadIdx.x;
  for (int bi = blockIdx.x; bi < nbig; bi += gridDim.x) {
    const int     b  = a.big[bi];
    const int64_t lo = a.off[b], hi = a.off[b + 1];
    for (int64_t q0 = lo; q0 < hi; q0 += 256) {
      const int64_t q = q0 + tid;
      const int32_t x = q < hi ? index_at<R>(a, q) : 0;
      int64_t       r = lo;
      for (int64_t z0 = lo; z0 < hi; z0 += 1024) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int64_t z = z0 + k * 256 + tid;
          reinterpret_cast<int32_t*>(s_idx)[k * 256 + tid] = z < hi ? index_at<R>(a, z) : INT_MAX;
        }
        __syncthreads();
        int smaller = 0;
#pragma unroll 4
        for (int k = 0; k < 256; ++k) {
          const int4 v = s_idx[k];
          smaller += (v.x < x) + (v.y < x) + (v.z < x) + (v.w < x);
        }
        r += smaller;
      }
      if (q < hi) a.rank[r] = x;
    }
  }
}

// place of index x in a big bin [lo, hi), whose indices are in order in a.rank
__device__ __forceinline__ int64_t big_place(const SortArgs& a, int64_t lo, int64_t hi, int32_t x) {
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (a.rank[mid] < x) lo = mid + 1;
    else                 hi = mid;
  }
  return lo;
}

// 4. records back into the arrays, each at the place that the number of
// smaller indices in its bin gives it (the dead and a plain compaction are in
// order as they are). A block's records are consecutive: they are read 16
// bytes per thread and handed over in shared memory, where most of a bin's
// indices are found too
template <typename R>
__global__ void __launch_bounds__(256) k_unpack(SortArgs a) {
  __shared__ uint4   s_rec[256 * R::Q];
  __shared__ int32_t s_idx[256];
  const int64_t p0 = (int64_t)blockIdx.x * 256;
  const int     n  = (int)(a.npart - p0 < 256 ? a.npart - p0 : 256);
#pragma unroll
  for (int q = 0; q < R::Q; ++q) {
    const int e = q * 256 + (int)threadIdx.x;
    if (e < n * R::Q) s_rec[e] = __ldcs(a.rec + p0 * R::Q + e);
  }
  __syncthreads();
  R r;
#pragma unroll
  for (int q = 0; q < R::Q; ++q) {
    const uint4 v = s_rec[threadIdx.x * R::Q + q];
    r.w[4 * q] = v.x, r.w[4 * q + 1] = v.y, r.w[4 * q + 2] = v.z, r.w[4 * q + 3] = v.w;
  }
  const int32_t x    = r.index();
  s_idx[threadIdx.x] = x;
  __syncthreads();
  if ((int)threadIdx.x >= n) return;
  bool          ok;
  const int32_t key =
    sort_key(a, r.tag(), (int)r.w[0], (int)r.w[1], R::DIM == 3 ? (int)r.w[2] : 0, ok);
  int64_t place = p0 + threadIdx.x;
  if (a.spatial && key != a.dead_bin) {
    const int64_t lo = a.off[key], hi = a.off[key + 1];
    if (hi - lo > kBigBin) {
      place = big_place(a, lo, hi, x);
    } else {
      // the bin's part in this block, then what lies before and after it
      const int b0 = (int)(lo > p0 ? lo - p0 : 0), b1 = (int)(hi < p0 + n ? hi - p0 : n);
      int       smaller = 0;
#pragma unroll 4
      for (int z = b0; z < b1; ++z) smaller += s_idx[z] < x;
      for (int64_t z = lo; z < p0; ++z) smaller += index_at<R>(a, z) < x;
      for (int64_t z = p0 + n; z < hi; ++z) smaller += index_at<R>(a, z) < x;
      place = lo + smaller;
    }
  }
  r.store(a, place);
}

// the permutation (new index -> old index) into a.perm2, from the particle
// arrays as they were
template <typename R>
__global__ void k_final_perm(SortArgs a) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < a.npart; p += stride) {
    const int32_t x = index_at<R>(a, p);
    bool          ok;
    const int32_t key   = sort_key_at(a, x, ok);
    int64_t       place = p;
    if (a.spatial && key != a.dead_bin) {
      const int64_t lo = a.off[key], hi = a.off[key + 1];
      if (hi - lo > kBigBin) {
        place = big_place(a, lo, hi, x);
      } else {
        place = lo;
        for (int64_t z = lo; z < hi; ++z) place += index_at<R>(a, z) < x;
      }
    }
    a.perm2[place] = x;
  }
}

// 5. one gather per array through perm into its staging buffer, then a
// copy back. (A single kernel gathering every array at once ran at half the
// speed on nearly sorted input: its many concurrent scattered streams lose
// the L2 locality each array's gather has on its own.)
template <typename T>
__global__ void k_gather(const T* __restrict__ src, T* __restrict__ dst, const int32_t* perm,
                         int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    dst[i] = src[perm[i]];
  }
}

__global__ void k_set_tags(int16_t* tag, int64_t np, const int32_t* n_dead) {
  const int64_t nalive = np - *n_dead;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += stride) {
    tag[i] = i < nalive ? (int16_t)PIC_TAG_ALIVE : (int16_t)PIC_TAG_DEAD;
  }
}

dim3 grid_n(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > pic::sm_count() * 64) b = pic::sm_count() * 64;
  if (b < 1) b = 1;
  return dim3((unsigned)b);
}

}  // namespace

namespace {
// calls f.operator()<D, RW, PREV>() for the species' layout
template <typename F>
cudaError_t by_layout(int dim, int real_bytes, bool prev, F&& f) {
  const int rw = real_bytes / 4;
#define PIC_SR(DD, RR, PP) \
  if (dim == DD && rw == RR && prev == PP) return f(SortRec<DD, RR, PP>{});
  PIC_SR(2, 1, false)
  PIC_SR(2, 1, true)
  PIC_SR(2, 2, false)
  PIC_SR(2, 2, true)
  PIC_SR(3, 1, false)
  PIC_SR(3, 1, true)
  PIC_SR(3, 2, false)
  PIC_SR(3, 2, true)
#undef PIC_SR
  return cudaErrorInvalidValue;
}
template <typename F>
cudaError_t with_layout(const SortArgs& a, F&& f) {
  return a.rec ? by_layout(a.dim, a.real_bytes, a.prev, f) : f(NoRec{});
}
}  // namespace

int sort_record_words(int dim, int real_bytes, bool prev) {
  int q = 0;
  by_layout(dim, real_bytes, prev, [&](auto r) {
    q = decltype(r)::Q;
    return cudaSuccess;
  });
  return q;
}

cudaError_t sort_scatter(const SortArgs& a, cudaStream_t s) {
  cudaError_t   e;
  const int64_t nbins  = (int64_t)a.dead_bin + 1;
  const int64_t blocks = (a.npart + kSortBlock - 1) / kSortBlock;
  if ((e = cudaMemsetAsync(a.count, 0, sizeof(int32_t) * (nbins + 1), s)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(a.nbig, 0, sizeof(int32_t), s)) != cudaSuccess) return e;
  PIC_KL(k_keys<<<(unsigned)blocks, 256, 0, s>>>(a));
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  ScanScratch<int64_t> scr;
  e = exclusive_scan<int32_t, int64_t>(a.count, nbins + 1, a.off, scr, s);
  scr.release(s);
  if (e != cudaSuccess) return e;
  ScanScratch<int32_t> scr2;
  e = exclusive_scan<int32_t, int32_t>(a.dead_cnt, blocks, a.dead_off, scr2, s);
  scr2.release(s);
  if (e != cudaSuccess) return e;
  return with_layout(a, [&](auto r) {
    using R = decltype(r);
    PIC_KL(k_scatter<R><<<(unsigned)blocks, 256, 0, s>>>(a));
    if (a.spatial && a.npart > kBigBin) PIC_KL(k_fix_big<R><<<pic::sm_count() * 2, 256, 0, s>>>(a));
    return cudaGetLastError();
  });
}

cudaError_t sort_unpack(const SortArgs& a, cudaStream_t s) {
  return by_layout(a.dim, a.real_bytes, a.prev, [&](auto r) {
    PIC_KL(k_unpack<decltype(r)><<<(unsigned)((a.npart + 255) / 256), 256, 0, s>>>(a));
    return cudaGetLastError();
  });
}

cudaError_t sort_final_perm(const SortArgs& a, cudaStream_t s) {
  return with_layout(a, [&](auto r) {
    PIC_KL(k_final_perm<decltype(r)><<<grid_n(a.npart), 256, 0, s>>>(a));
    return cudaGetLastError();
  });
}

namespace {
// arr_k[i] -> dst_k[i] = arr_k[perm[i]] for every listed array: the
// permutation is read once per particle for all arrays of the species
struct MultiGather {
  const void* src[kMaxSortArrays];
  void*       dst[kMaxSortArrays];
  int         esz[kMaxSortArrays];
  int64_t     es[kMaxSortArrays];  // element stride of src
  int         n;
};

// N arrays: every value of a particle is loaded before any is stored, so a
// thread keeps N loads in flight instead of one
template <int N>
__global__ void k_gather_multi(MultiGather g, const int32_t* __restrict__ perm, int64_t np) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += stride) {
    const int64_t j = perm[i];
    uint64_t      v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int64_t jk = j * g.es[k];
      if (g.esz[k] == 4)      v[k] = (uint32_t)((const int32_t*)g.src[k])[jk];
      else if (g.esz[k] == 8) v[k] = (uint64_t)((const int64_t*)g.src[k])[jk];
      else                    v[k] = (uint16_t)((const int16_t*)g.src[k])[jk];
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (g.esz[k] == 4)      ((int32_t*)g.dst[k])[i] = (int32_t)(uint32_t)v[k];
      else if (g.esz[k] == 8) ((int64_t*)g.dst[k])[i] = (int64_t)v[k];
      else                    ((int16_t*)g.dst[k])[i] = (int16_t)(uint16_t)v[k];
    }
  }
}

template <int N>
cudaError_t launch_gather_n(const MultiGather& g, const int32_t* perm, int64_t np, dim3 grid,
                            cudaStream_t s) {
  if constexpr (N > kMaxSortArrays) {
    return cudaErrorInvalidValue;
  } else {
    if (g.n != N) return launch_gather_n<N + 1>(g, perm, np, grid, s);
    PIC_KL(k_gather_multi<N><<<grid, 256, 0, s>>>(g, perm, np));
    return cudaGetLastError();
  }
}

// copies of the packed staging areas back into the caller's arrays: packed
// arrays in 16-byte pieces where both ends allow it (chunk c of array k
// covers bytes [c * 16, c * 16 + 16)), strided ones element by element
// (chunk c is element c)
struct MultiCopy {
  const char* src[kMaxSortArrays];
  char*       dst[kMaxSortArrays];
  int64_t     bytes[kMaxSortArrays];
  int64_t     es[kMaxSortArrays];  // element stride of dst
  int         esz[kMaxSortArrays];
  int64_t     first_chunk[kMaxSortArrays + 1];
  int         vec[kMaxSortArrays];  // packed, both pointers 16-byte aligned
  int         n;
};

__global__ void k_copy_multi(MultiCopy m) {
  const int64_t total  = m.first_chunk[m.n];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int           k      = 0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < total; c += stride) {
    while (c >= m.first_chunk[k + 1]) ++k;
    const int64_t q = c - m.first_chunk[k];
    if (m.es[k] != 1) {
      const int64_t d = q * m.es[k];
      if (m.esz[k] == 4)      ((int32_t*)m.dst[k])[d] = ((const int32_t*)m.src[k])[q];
      else if (m.esz[k] == 8) ((int64_t*)m.dst[k])[d] = ((const int64_t*)m.src[k])[q];
      else                    ((int16_t*)m.dst[k])[d] = ((const int16_t*)m.src[k])[q];
      continue;
    }
    const int64_t off = q * 16;
    const int64_t len = m.bytes[k] - off < 16 ? m.bytes[k] - off : 16;
    if (m.vec[k] && len == 16) {
      *(int4*)(m.dst[k] + off) = *(const int4*)(m.src[k] + off);
    } else {
      for (int64_t b = 0; b < len; ++b) m.dst[k][off + b] = m.src[k][off + b];
    }
  }
}

// one array through a shared staging buffer, any element stride
template <typename T>
__global__ void k_gather_strided(const T* __restrict__ src, T* __restrict__ dst,
                                 const int32_t* perm, int64_t n, int64_t es) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride)
    dst[i] = src[(int64_t)perm[i] * es];
}
template <typename T>
__global__ void k_unpack_strided(const T* __restrict__ src, T* __restrict__ dst, int64_t n,
                                 int64_t es) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride)
    dst[i * es] = src[i];
}
}  // namespace

cudaError_t sort_apply_all(const GatherSet& g, const int32_t* perm, int64_t n, cudaStream_t s) {
  if (n <= 0 || g.n == 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  bool        staged_apart = true;  // every array has its own staging area
  for (int k = 0; k < g.n && staged_apart; ++k)
    for (int q = 0; q < k; ++q) staged_apart = staged_apart && g.tmp[q] != g.tmp[k];
  if (staged_apart) {
    // one gather of all arrays (perm read once), then one copy back
    MultiGather mg{};
    MultiCopy   mc{};
    mg.n = mc.n = g.n;
    mc.first_chunk[0] = 0;
    for (int k = 0; k < g.n; ++k) {
      mg.src[k] = g.arr[k];
      mg.dst[k] = g.tmp[k];
      mg.esz[k] = g.esz[k];
      mg.es[k]  = g.stride[k];
      mc.src[k] = (const char*)g.tmp[k];
      mc.dst[k] = (char*)g.arr[k];
      mc.bytes[k] = n * g.esz[k];
      mc.es[k]    = g.stride[k];
      mc.esz[k]   = g.esz[k];
      mc.vec[k] = g.stride[k] == 1 && ((uintptr_t)g.tmp[k] % 16 == 0) &&
                  ((uintptr_t)g.arr[k] % 16 == 0);
      mc.first_chunk[k + 1] =
        mc.first_chunk[k] + (g.stride[k] == 1 ? (mc.bytes[k] + 15) / 16 : n);
    }
    if ((e = launch_gather_n<1>(mg, perm, n, grid_n(n), s)) != cudaSuccess) return e;
    PIC_KL(k_copy_multi<<<grid_n(mc.first_chunk[g.n]), 256, 0, s>>>(mc));
    return cudaGetLastError();
  }
  // one shared staging buffer: the arrays go in turn
  for (int k = 0; k < g.n; ++k) {
    if (g.stride[k] != 1) {
      if (g.esz[k] == 8) {
        PIC_KL(k_gather_strided<int64_t><<<grid_n(n), 256, 0, s>>>((const int64_t*)g.arr[k], (int64_t*)g.tmp[k], perm, n, g.stride[k]));
        PIC_KL(k_unpack_strided<int64_t><<<grid_n(n), 256, 0, s>>>((const int64_t*)g.tmp[k], (int64_t*)g.arr[k], n, g.stride[k]));
      } else if (g.esz[k] == 4) {
        PIC_KL(k_gather_strided<int32_t><<<grid_n(n), 256, 0, s>>>((const int32_t*)g.arr[k], (int32_t*)g.tmp[k], perm, n, g.stride[k]));
        PIC_KL(k_unpack_strided<int32_t><<<grid_n(n), 256, 0, s>>>((const int32_t*)g.tmp[k], (int32_t*)g.arr[k], n, g.stride[k]));
      } else {
        PIC_KL(k_gather_strided<int16_t><<<grid_n(n), 256, 0, s>>>((const int16_t*)g.arr[k], (int16_t*)g.tmp[k], perm, n, g.stride[k]));
        PIC_KL(k_unpack_strided<int16_t><<<grid_n(n), 256, 0, s>>>((const int16_t*)g.tmp[k], (int16_t*)g.arr[k], n, g.stride[k]));
      }
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      continue;
    }
    if (g.esz[k] == 4)
      PIC_KL(k_gather<int32_t><<<grid_n(n), 256, 0, s>>>((const int32_t*)g.arr[k], (int32_t*)g.tmp[k], perm, n));
    else if (g.esz[k] == 8)
      PIC_KL(k_gather<int64_t><<<grid_n(n), 256, 0, s>>>((const int64_t*)g.arr[k], (int64_t*)g.tmp[k], perm, n));
    else
      PIC_KL(k_gather<int16_t><<<grid_n(n), 256, 0, s>>>((const int16_t*)g.arr[k], (int16_t*)g.tmp[k], perm, n));
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    e = cudaMemcpyAsync(g.arr[k], g.tmp[k], (size_t)n * g.esz[k], cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t set_tags_after_removal(int16_t* tag, int64_t np, const int32_t* n_dead,
                                   cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  PIC_KL(k_set_tags<<<grid_n(np), 256, 0, s>>>(tag, np, n_dead));
  return cudaGetLastError();
}

namespace {
__global__ void k_tile_offsets(const int64_t* off, int64_t tile_cells, int ntiles,
                               int32_t* tile_start) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t <= ntiles) tile_start[t] = (int32_t)off[(int64_t)t * tile_cells];
}
}  // namespace

cudaError_t tile_offsets(const int64_t* off, int64_t tile_cells, int ntiles, int32_t* tile_start,
                         cudaStream_t s) {
  PIC_KL(k_tile_offsets<<<(ntiles + 256) / 256, 256, 0, s>>>(off, tile_cells, ntiles, tile_start));
  return cudaGetLastError();
}

}  // namespace pic
