// Host-side declarations for the sort and scan kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pic_types.h"

namespace pic {

// stream-ordered scratch for the recursive levels of the scan
template <typename T>
struct ScanScratch {
  T*      p   = nullptr;
  int64_t cap = 0;
  T* get(int64_t n, cudaStream_t s) {
    if (n > cap) {
      if (p) cudaFreeAsync(p, s);
      p   = nullptr;
      cap = 0;
      if (cudaMallocAsync((void**)&p, sizeof(T) * n, s) != cudaSuccess) return nullptr;
      cap = n;
    }
    return p;
  }
  void release(cudaStream_t s) {
    if (p) cudaFreeAsync(p, s);
    p   = nullptr;
    cap = 0;
  }
};

template <typename Tin, typename T>
cudaError_t exclusive_scan(const Tin* in, int64_t n, T* out, ScanScratch<T>& scr, cudaStream_t s);

// particles per block of the key and scatter passes, in index order (the dead
// of a block are counted together)
constexpr int kSortBlock = 2048;
// bins above this many particles are ordered by k_fix_big, not by counting
constexpr int kBigBin = 1024;

struct SortArgs {
  // particle arrays; the previous positions only when they move too
  int32_t *i[3], *ip[3];
  float   *dx[3], *dxp[3];
  void    *u[4];      // momenta, weight
  int16_t *tag;
  int      real_bytes;
  bool     prev;
  int64_t  npart;
  int      dim;
  int      n[3];
  int      spatial;   // 1: cell key, 0: alive/dead only
  int      tiled;     // with spatial: tile-major key (tile, then cell in tile)
  int      tile_log[3];  // log2 of the tile shape
  int      ntiles[3]; // tiles per axis
  int32_t  dead_bin;  // index of the last bin
  // scratch
  int32_t*  rank;     // npart: place of a particle among its bin's, in arrival order
  int32_t*  dead_off; // one per block of kSortBlock particles: dead before it
  int32_t*  dead_cnt; // the same, counts
  int32_t*  count;    // dead_bin + 2 entries
  int64_t*  off;      // dead_bin + 2 entries
  int32_t*  perm;     // npart: particle at each place, bins in arrival order (without records)
  int32_t*  perm2;    // npart: new index -> old index (sort_final_perm)
  uint4*    rec;      // npart records (null: perm instead)
  int32_t*  big;      // bins of more than kBigBin particles, at most npart / kBigBin
  int32_t*  nbig;
  unsigned long long* err;
};

// 16-byte words of one particle's record (every array above and the index)
int sort_record_words(int dim, int real_bytes, bool prev);

// counts, offsets and the records (or perm) scattered to their bins, in arrival
// order within a bin, without host synchronisation. The dead count is left in
// count[dead_bin]
cudaError_t sort_scatter(const SortArgs& a, cudaStream_t s);
// the records back into the particle arrays, each bin in index order
cudaError_t sort_unpack(const SortArgs& a, cudaStream_t s);
// the permutation, each bin in index order, into a.perm2; reads the particle
// arrays' keys, so it comes before sort_unpack
cudaError_t sort_final_perm(const SortArgs& a, cudaStream_t s);

// every listed array permuted in place: arr_k[i] <- arr_k[perm[i]], staged
// through tmp_k. With a staging area per array, one kernel gathers all
// arrays (the permutation read once) and one copies them back; when the
// tmp_k share one buffer the arrays go in turn
constexpr int kMaxSortArrays = 32;  // 3D with prev arrays needs 17, phi and payloads more
struct GatherSet {
  void*   arr[kMaxSortArrays];
  void*   tmp[kMaxSortArrays];
  int     esz[kMaxSortArrays];     // element bytes: 2, 4 or 8
  int64_t stride[kMaxSortArrays];  // element stride of arr (payload columns); tmp is packed
  int     n = 0;
};
cudaError_t sort_apply_all(const GatherSet& g, const int32_t* perm, int64_t n, cudaStream_t s);

// tags of [0, np - *n_dead) alive and of the rest dead (RemoveDead)
cudaError_t set_tags_after_removal(int16_t* tag, int64_t np, const int32_t* n_dead,
                                   cudaStream_t s);

// tile_start[t] = off[t * tile_cells] for t in [0, ntiles]
cudaError_t tile_offsets(const int64_t* off, int64_t tile_cells, int ntiles, int32_t* tile_start,
                         cudaStream_t s);

}  // namespace pic
