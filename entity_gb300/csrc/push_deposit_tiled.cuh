// Tiled fused push + deposit: one CTA per tile of cells.
//
// The species' particles are stored tile-major (PIC_SORT_TILED), so the
// particles of a tile are one contiguous range per species and are read and
// written back fully coalesced. The CTA
//   1. stages the E/B window of its tile (tile + interpolation halo + a drift
//      margin of M cells) in shared memory: one TMA box load (all six
//      components) that runs while the CTA clears its J window and scans its
//      particles' weights, or a strided copy loop for a window that wraps
//      across a periodic edge;
//   2. pushes every particle of the tile (all species) gathering E/B from
//      shared memory, and deposits its current into a shared-memory J window
//      (tile + deposit halo + margin); at orders 1-3 from records, after the
//      pushes (DepStage: every particle in 3D, in 2D those whose shape support
//      moved),
//   3. adds the J window to global J once, wrapping periodic images onto
//      their active cells (the fold SynchronizeFields performs in the
//      reference, src/framework/domain/metadomain_comm.cpp:408-562).
//
// Accumulation in the J window: fixed point split over 32-bit words.
// 32-bit integer shared-memory atomics are the fastest this GPU has (a
// microbenchmark measured 9.1 Top/s, against 2.8 for float, 1.6 for 64-bit
// integers and 0.5 for double), and integer sums do not depend on the order
// of the additions. Each tile scales contributions by a power of two 2^s so
// that |v 2^s| < 2^b, rounds them to integers (exact up to the quantisation
// 2^-s) and adds them as 32-bit words: X modulo 2^32 and X >> 12 (float),
// or three 16-bit words and a signed top word (double). With N
// particles in the tile no cell takes more than N additions per component,
// so b = min(30, 43 - log2 N) (float; 29 bits at 16k particles) or
// b = 62 - log2 N (double) overflows neither a word nor the 64-bit total.
// The tile's sum is exact and
// independent of the order of the additions; each cell is rounded to real
// once, at the flush. A tile denser than the words allow (N > 2^20 in float,
// 2^16 in double) accumulates in real_t atomics instead.
//
// A particle that has drifted more than M cells outside its tile since the
// last tiled sort, or whose stencil can reach the ghost layers of a
// non-periodic axis, is not touched here: it is appended to the species'
// overflow list and pushed afterwards by the per-particle kernel (global
// gathers, global atomics, the reference's coordinates), and the hot kernel
// holds only the shared-memory path. The push is the same code as the untiled
// kernel's: a particle's new state does not depend on the binning. The deposit
// is its factored form (pic_common.cuh), rounded elsewhere than the reference's
// form of the per-particle kernels, and a tile's entries are rounded to its own
// unit: J depends on the binning in its last bits.
#pragma once

#include <type_traits>

#include "fixed_acc.cuh"
#include "push_deposit.cuh"
#include "tma.cuh"

namespace pic {

constexpr int kDriftMargin     = 1;

// tile shape per (dimension, precision, order): the shared-memory windows
// must fit one CTA's 227 KB
template <int D, typename real, int O>
struct TileShape {
  // 2D: 16 x 8 cells. The 512^2 pair plasma (2 x 16 ppc) ran push+deposit in
  // 0.578 ms with 32 x 32 tiles (256 CTAs, 0.56 waves), 0.456 ms with
  // 16 x 16, 0.419 ms with 16 x 8 and 0.429 ms with 8 x 8.
  // NT threads per CTA; MINB CTAs per SM asked of the register allocator.
  // The kernel is latency-bound, so warps per SM pay: FP32 at 256 threads ran
  // 0.543 ms with the allocator's 80 registers (3 CTAs/SM), 0.388 ms at 64
  // (4 CTAs), 0.350 ms at 48 (5 CTAs, no spill) and 0.366 ms at 40 (6 CTAs,
  // spilling); 512 threads x 2 gave 0.408 ms
  static constexpr int X = 16, Y = 8, Z = 1, NT = 256,
                       MINB = sizeof(real) == 4 ? (O == 3 ? 4 : 5) : 1,  // order 3 spills at 5
                       CHUNK = 2048;
};
// 3D FP32. One CTA per SM (the shared memory), so the thread count sets the
// warps that hide the kernel's latencies, and the register file what each may
// use. Steps of the 256^3 turbulence plasma (order 2, 2 x 8 ppc) took 26.8 ms
// with 768 threads (80 registers) and 26.7 with 1024 (64); steps of the 96^3
// sweep plasma (order 3, 2 x 32 ppc) 12.5, 12.0 and 11.9 ms with 640, 768 and
// 1024. CHUNK: particles pushed between deposits. More of them fill the
// records' classes more evenly and wait at fewer barriers: 5120, 10240 and
// 20480 (more than a tile of the turbulence plasma holds) gave 28.9, 26.7 and
// 25.6 ms, 20480 and 36864 (a tile of the sweep plasma) 11.9 and 11.6 ms.
template <int O>
struct TileShape<3, float, O> {
  static constexpr int X = (O == 3 ? 8 : 16), Y = 8, Z = 8, NT = 1024, MINB = 1,
                       CHUNK = (O == 3 ? 36 : 20) * 1024;
};
// FP64 (8 x 8 x 4 cells) is bound by the FP64 pipe (two lanes per SM and
// clock): 384 and 512 threads, chunks of 4608 and 5120 particles all gave
// 10.1 to 10.2 ms per step of the 64^3 turbulence box
template <int O>
struct TileShape<3, double, O> {
  static constexpr int X = 8, Y = 8, Z = 4, NT = 384, MINB = 1, CHUNK = 4608;
};

// window halos (cells below / above the tile) of the interpolation and the
// deposit stencils at order O, plus the drift margin
template <int O>
struct Halo {
  static constexpr int E_LO = (O == 3 ? 2 : 1) + kDriftMargin;
  static constexpr int E_HI = (O >= 2 ? 2 : 1) + kDriftMargin;
  static constexpr int J_LO = (O >= 2 ? 2 : 1) + kDriftMargin;
  static constexpr int J_HI = (O >= 2 ? 3 : 2) + kDriftMargin;
};

template <typename real>
struct TiledSpecies {
  SpeciesPtrs    sp;
  const int32_t* tile_start;  // ntiles + 1 offsets into the particle arrays
  real           ndth, charge;
  int            vay;
  int32_t*       ovf;         // particles left to the per-particle kernel
  unsigned*      ovf_count;
};

// Deposit records (orders 1-3). A particle's push appends a 32-byte record
// (48 in FP64: cell offsets from the tile, the offsets before and after the
// move, q w, in 2D the out-of-plane velocity) to a buffer in global memory
// (written and read back by the same CTA), and the CTA deposits the records once
// it has pushed a chunk of its particles. The live records of all SMs are 98 MB at
// order 2 in 3D and 179 MB at order 3, so part of them leaves L2 before it is read:
// 115 bytes of DRAM traffic per particle on the turbulence plasma, 78 of them the
// particle's and its cells' own, at a fifth of the DRAM peak.
//   - The records are queued by bank class, the shared-memory bank (of 32) of
//     the first J-window word of the particle's Esirkepov box. Row r of a
//     buffer holds the r-th record of each class, and a warp takes a row: its
//     32 lanes add to entries at the same offsets from 32 first words in 32
//     different banks, so every atomic of the warp is one wavefront. Deposited
//     in cell order, lanes of one cell serialise on its words (3.6 wavefronts
//     per atomic on the turbulence plasma, the shared pipe at 65 % of its
//     peak).
//   - Most particles end a step with both shape supports starting at the same
//     node on every axis (support_unmoved): their box is (O + 1) wide on each
//     axis, a stencil the compiler unrolls to its exact extent (54 of the 144
//     entries at order 2 in 3D). The others, whose box is O + 2 wide on some
//     axis, have rows of their own, so no warp runs the wide stencil for one
//     lane.
// J does not depend on the records to the bit: the window's integer sums are
// independent of the order of the additions. A full class hands its records
// to the next one, which costs a bank conflict; the rows of a region hold a
// whole chunk, so a record always finds a place. A CTA claims one of nslots
// buffers; there are as many as CTAs that can be resident at once. A buffer
// passes from one CTA to the next by a release and an acquire (take_slot,
// give_slot): the last holder's records and discards come before the next
// one's records.
struct DepStage {
  uint4*    rec    = nullptr;  // nslots buffers of two regions (unmoved, moved)
  unsigned* claim  = nullptr;  // nslots words: 0 free, 1 held
  int       nslots = 0, per_sm = 1;  // buffers, and CTAs resident on one SM
};

// Called by one thread. A buffer's index, or -1 when the limit ran out. The
// search starts with this SM's own buffers, one of which its last CTA has just
// given back. The fence orders the claim before the CTA's records (its other
// warps start them behind a barrier).
__device__ __forceinline__ int take_slot(const DepStage& st) {
  const unsigned n = (unsigned)st.nslots;
  unsigned       sm;
  asm("mov.u32 %0, %%smid;" : "=r"(sm));
  unsigned sl = (sm * (unsigned)st.per_sm) % n;
  for (unsigned k = 0; k < 64u * n; ++k) {
    if (atomicCAS(st.claim + sl, 0u, 1u) == 0u) {
      __threadfence();
      return (int)sl;
    }
    if (++sl == n) sl = 0;
  }
  return -1;
}
// Called by one thread behind a barrier that follows the CTA's last use of the
// buffer: the fence orders every warp's records and discards before the word.
__device__ __forceinline__ void give_slot(const DepStage& st, int slot) {
  __threadfence();
  atomicExch(st.claim + slot, 0u);
}

// drops the 128-byte line at p (128-byte aligned) from L2 without writing it
// back; its contents are undefined until written again
__device__ __forceinline__ void discard_l2_line(const void* p) {
  asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
}

template <typename real>
struct TiledArgs {
  TiledSpecies<real> s[kMaxTiledSpecies];
  int                nsp;
  PushConsts         pc;
  int                periodic[3];
  int                ntiles[3];
  int                tile0, tile1;  // linear tiles [tile0, tile1) of this launch
  FieldView<real>    EB;
  FieldView<real>    J;
  real               dt, dx, inv_dt;
  int                write_prev;
  unsigned long long* err;
  // tiled tensor map of EB (x, y, [z], component) with the E-window box;
  // eb_tma = 0 when the field array does not meet TMA's alignment rules
  alignas(64) CUtensorMap eb_map;
  int                eb_tma;
  // FP32: the exact 64-bit accumulator the tile sums are flushed into (null:
  // float atomics into J)
  FixedJ             fj;
  // where a tile's pushed particles wait for their deposit
  DepStage           st;
  // warps taken lane_stride at a time read their particles interleaved
  // (1, 2 or 4; a divisor of the CTA's warps): a warp of a cell-sorted tile
  // then spans 32 lane_stride / ppc cells (the rule is with the caller)
  int                lane_stride = 1;
};

template <int D, int O, typename real>
struct TiledGeom {
  using TS                = TileShape<D, real, O>;
  static constexpr int TX = TS::X, TY = TS::Y, TZ = (D == 3 ? TS::Z : 1);
  static constexpr int NT = TS::NT;
  using H                 = Halo<O>;
  static constexpr int WE0 = TX + H::E_LO + H::E_HI;
  static constexpr int WE1 = TY + H::E_LO + H::E_HI;
  static constexpr int WE2 = D == 3 ? TZ + H::E_LO + H::E_HI : 1;
  static constexpr int WJ0 = TX + H::J_LO + H::J_HI;
  static constexpr int WJ1 = TY + H::J_LO + H::J_HI;
  static constexpr int WJ2 = D == 3 ? TZ + H::J_LO + H::J_HI : 1;
  static constexpr int NJ  = WJ0 * WJ1 * WJ2;
  // J window: FixedAcc<real>::WORDS planes of 3 * NJ 32-bit words
  static constexpr int    WORDS      = FixedAcc<real>::WORDS;
  static constexpr int    PLANE      = 3 * NJ;
  static constexpr size_t jw_bytes   = 4 * (size_t)(WORDS * PLANE);
  // Deposit records: all particles' (REC_ALL), or those of particles whose
  // support moved, the others depositing at once
  static constexpr bool   REC        = O >= 1;
  static constexpr bool   REC_ALL    = D == 3;
  static constexpr int    RECW       = sizeof(real) == 4 ? 2 : 3;  // 16-byte words per record
  static constexpr int    CHUNK      = TS::CHUNK;                  // particles between deposits
  static constexpr int    ROWS       = CHUNK / 32;                 // rows per region
  static constexpr size_t region     = (size_t)CHUNK * RECW;       // 16-byte words
  static constexpr size_t moved      = REC_ALL ? region : 0;       // start of the moved region
  static constexpr size_t slot_words = moved + region;
  static_assert(CHUNK % 32 == 0 && CHUNK >= NT, "a chunk holds one particle per thread at least");
  // E window rows: a TMA box row is a multiple of 16 bytes and starts on a
  // 16-byte boundary, so the row is widened to WEX elements and the window
  // sits R = (x start mod A) elements into it (A elements per 16 bytes)
  static constexpr int    A          = 16 / (int)sizeof(real);
  static constexpr int    WEX_TMA    = ((WE0 + A - 1 + A - 1) / A) * A;
  static constexpr size_t kSmemMax   = 232448 - 512;  // per-CTA limit less the static words
  static constexpr bool fits(int wx, int wy) {
    return ((sizeof(real) * 6 * (size_t)wx * wy * WE2 + 127) / 128) * 128 + jw_bytes <= kSmemMax;
  }
  // The interpolation's lanes in one cell read x, x + 1, the next row and the
  // next plane of a window row: the row and plane strides must differ in
  // shared-memory bank (mod 32 words) or those reads conflict. The box's y
  // extent is padded (rows beyond the window are loaded and never read)
  // until x, x + 1, + row, + plane and their sums fall in 8 distinct banks.
  static constexpr bool banks_distinct(int wx, int wy) {
    // word offsets of the eight reads; a read of real_t covers w words
    const int w = (int)sizeof(real) / 4, row = wx * w, pl = wx * wy * w;
    const int o[8] = { 0, w, row, row + w, pl, pl + w, row + pl, row + pl + w };
    for (int i = 0; i < 8; ++i)
      for (int j = i + 1; j < 8; ++j) {
        const int d = ((o[i] - o[j]) % 32 + 32) % 32;
        if (d < w || d > 32 - w) return false;
      }
    return true;
  }
  static constexpr int pick_wey() {
    int best = WE1;
    for (int y = WE1 + 3; y >= WE1; --y)
      if (D == 3 && banks_distinct(WEX_TMA, y) && fits(WEX_TMA, y)) best = y;
    return best;
  }
  static constexpr bool   TMA        = fits(WEX_TMA, WE1);
  static constexpr int    WEX        = TMA ? WEX_TMA : WE0;
  static constexpr int    WEY        = TMA ? pick_wey() : WE1;
  static constexpr int    NE         = WEX * WEY * WE2;
  static constexpr size_t eb_bytes   = sizeof(real) * 6 * (size_t)NE;
  static constexpr size_t smem_bytes = ((eb_bytes + 127) / 128) * 128 + jw_bytes;
};

// J-window accumulators: base is the word of ghost-inclusive node (0, 0, 0)
template <typename G, typename FA>
struct JWinFixed : BoxAdd {
  unsigned* w;
  int       base;
  __device__ __forceinline__ JWinFixed(unsigned* w_, int b) : w(w_), base(b) {}
  __device__ __forceinline__ JWinFixed at(int i, int j, int k) const {
    return { w, base + i + j * G::WJ0 + k * (G::WJ0 * G::WJ1) };
  }
  template <typename real>
  __device__ __forceinline__ void operator()(int i, int j, int k, int c, real v) const {
    FA::add(w + base + (i + j * G::WJ0 + k * (G::WJ0 * G::WJ1) + c * G::NJ), G::PLANE, v);
  }
};
template <typename G, typename real>
struct JWinReal : BoxAdd {
  real* w;
  int   base;
  __device__ __forceinline__ JWinReal(real* w_, int b) : w(w_), base(b) {}
  __device__ __forceinline__ JWinReal at(int i, int j, int k) const {
    return { w, base + i + j * G::WJ0 + k * (G::WJ0 * G::WJ1) };
  }
  __device__ __forceinline__ void operator()(int i, int j, int k, int c, real v) const {
    atomicAdd(w + base + (i + j * G::WJ0 + k * (G::WJ0 * G::WJ1) + c * G::NJ), v);
  }
};

// wraps a ghost-free coordinate of a periodic axis into [0, n)
__device__ __forceinline__ int wrap_periodic(int x, int n) {
  x %= n;
  return x < 0 ? x + n : x;
}

// REC: deposits go through records (DepStage); without, every particle
// deposits as it is pushed (order 0, or no buffers)
template <int D, int O, typename real, bool REC>
__global__ void __launch_bounds__(TileShape<D, real, O>::NT, TileShape<D, real, O>::MINB)
    k_push_deposit_tiled(const __grid_constant__ TiledArgs<real> a) {
  using G               = TiledGeom<D, O, real>;
  using H               = Halo<O>;
  using FA              = FixedAcc<real>;
  constexpr int  NT     = G::NT;
  constexpr int  M      = kDriftMargin;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  real*          EBs = reinterpret_cast<real*>(smem_raw);
  unsigned*      Jw  = reinterpret_cast<unsigned*>(smem_raw + ((G::eb_bytes + 127) / 128) * 128);
  real*          Jr  = reinterpret_cast<real*>(Jw);  // real_t accumulation of dense tiles
  __shared__ unsigned int s_qmax;  // bit pattern of the tile's largest |q w| max(1/dt, 1)
  __shared__ __align__(8) unsigned long long s_bar;  // completion of the E-window load
  __shared__ int      s_slot;         // the claimed record buffer, -1 for none
  __shared__ unsigned s_cnt[2][32];   // records per class, unmoved and moved supports

  const int t  = blockIdx.x + a.tile0;
  const int tx = t % a.ntiles[0];
  const int ty = (t / a.ntiles[0]) % a.ntiles[1];
  const int tz = D == 3 ? t / (a.ntiles[0] * a.ntiles[1]) : 0;
  const int T0[3] = { tx * G::TX, ty * G::TY, tz * G::TZ };
  const int ng    = a.pc.ng;

  // 1. E/B window, ghost-inclusive start g0 along each axis; the window's
  //    rows start R elements into the widened shared rows
  const int g0[3] = { ng + T0[0] - H::E_LO, ng + T0[1] - H::E_LO,
                      D == 3 ? ng + T0[2] - H::E_LO : 0 };
  const int R     = G::TMA ? (g0[0] & (G::A - 1)) : 0;
  bool      tma   = false;
  if constexpr (G::TMA) {
    // one box load covers the window when no periodic axis wraps inside it
    // (beyond a non-periodic edge the load's zero fill is what the copy
    // loop writes too)
    const int we[3] = { G::WE0, G::WE1, G::WE2 };
    tma = a.eb_tma != 0 && (smem_addr(EBs) & 127u) == 0u;
#pragma unroll
    for (int d = 0; d < D; ++d)
      if (a.periodic[d] && (g0[d] < 0 || g0[d] + we[d] > a.pc.ext[d])) tma = false;
  }
  const unsigned bar = smem_addr(&s_bar);
  if (tma) {
    if (threadIdx.x == 0) {
      mbar_init(bar, 1);
      mbar_expect_tx(bar, (unsigned)G::eb_bytes);
      if constexpr (D == 3) tma_load_4d(smem_addr(EBs), &a.eb_map, bar, g0[0] - R, g0[1], g0[2], 0);
      else                  tma_load_3d(smem_addr(EBs), &a.eb_map, bar, g0[0] - R, g0[1], 0);
    }
  } else {
    // reads ghost cells where the window overlaps them and the periodic
    // image beyond (zero beyond a non-periodic edge: no valid particle's
    // stencil reaches there)
    for (int idx = threadIdx.x; idx < 6 * G::WE0 * G::WE1 * G::WE2; idx += NT) {
      int       r  = idx;
      const int wi = r % G::WE0;
      r /= G::WE0;
      const int wj = r % G::WE1;
      r /= G::WE1;
      const int wk = r % G::WE2;
      const int c  = r / G::WE2;
      int       gc[3] = { T0[0] - H::E_LO + wi, T0[1] - H::E_LO + wj,
                          D == 3 ? T0[2] - H::E_LO + wk : 0 };
      bool      inside = true;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        if (gc[d] < -ng || gc[d] >= a.pc.n[d] + ng) {
          if (a.periodic[d]) gc[d] = wrap_periodic(gc[d], a.pc.n[d]);
          else inside = false;
        }
      }
      EBs[R + wi + G::WEX * (wj + G::WEY * (wk + G::WE2 * c))] =
          inside ? a.EB.ld(gc[0] + ng, gc[1] + ng, D == 3 ? gc[2] + ng : 0, c) : (real)0;
    }
  }
  for (int idx = threadIdx.x; idx < G::WORDS * G::PLANE; idx += NT)
    Jw[idx] = 0u;
  // largest contribution bound of the tile, |q w| max(1/dt, 1), and its
  // particle count (an upper bound on the additions any cell receives)
  if constexpr (REC) {
    if (threadIdx.x < 64) (&s_cnt[0][0])[threadIdx.x] = 0u;
  }
  if (threadIdx.x == 0) {
    s_qmax = 0u;
    s_slot = REC ? take_slot(a.st) : -1;
  }
  __syncthreads();
  // (with the exact global accumulator the bound is the call's, known already)
  const bool global_unit = sizeof(real) == 4 && a.fj.p != nullptr;
  float      qmax = 0.f;
  int64_t    ntile = 0;
  for (int s = 0; s < a.nsp; ++s) {
    const real*   w  = (const real*)a.s[s].sp.w;
    const float   qs = fabsf((float)a.s[s].charge);
    const int64_t lo = a.s[s].tile_start[t], hi = a.s[s].tile_start[t + 1];
    ntile += hi - lo;
    if (global_unit) continue;
    for (int64_t p = lo + threadIdx.x; p < hi; p += NT) qmax = fmaxf(qmax, fabsf((float)w[p]) * qs);
  }
  qmax *= fmaxf((float)a.inv_dt, 1.f);
  atomicMax(&s_qmax, __float_as_uint(qmax));  // non-negative floats order as their bits
  __syncthreads();
  const bool fixed = ntile <= FA::NMAX;
  real       scale = 1, unscale = 1;
  int        ex = 0, b = FA::bits(ntile);
  if (global_unit) {
    // the call's bound, and no more bits than the global unit has, so that
    // a tile total becomes global units by a left shift
    ex = a.fj.exponent();
    b  = min(b, a.fj.bits);
  } else {
    frexpf(__uint_as_float(s_qmax) * 1.0000002f, &ex);  // |contribution| < 2^ex
  }
  scale   = (real)ldexp(1.0, b - ex);
  unscale = (real)ldexp(1.0, ex - b);

  {
    // every thread waits for the window; a lost wait (the limit ran out on
    // any thread) abandons the tile on all of them and is counted
    bool done = !tma || mbar_wait_bounded(bar, 0u);
    if constexpr (REC) done = done && s_slot >= 0;
    if (__syncthreads_or(!done)) {
      if (threadIdx.x == 0) {
        atomicAdd(a.err + ERR_WAIT_TIMEOUT, 1ull);
        if (REC && s_slot >= 0) give_slot(a.st, s_slot);
      }
      return;
    }
  }
  const SmemView<real> ebv{ EBs, g0[0] - R, g0[1], g0[2], G::WEX, G::WEX * G::WEY, G::NE };
  const int joff[3] = { ng + T0[0] - H::J_LO, ng + T0[1] - H::J_LO,
                        D == 3 ? ng + T0[2] - H::J_LO : 0 };
  const int jb      = -joff[0] - joff[1] * G::WJ0 - joff[2] * (G::WJ0 * G::WJ1);
  // The thread's particle within each NT-particle group. With lane_stride
  // ls, ls consecutive warps share 32 ls consecutive particles, lane l of the
  // group's k-th warp taking particle ls l + k: each warp spans ls times as
  // many cells, so fewer of its lanes add to one J word, and the group
  // still reads whole lines.
  const int ls      = a.lane_stride;
  const int lane    = (int)(threadIdx.x & 31);
  const int wid     = (int)(threadIdx.x >> 5);
  const int local   = (wid / ls) * (32 * ls) + ls * lane + wid % ls;
  uint4*    recs    = REC ? a.st.rec + (size_t)s_slot * G::slot_words : nullptr;
  // cell of a record relative to the tile: 8 bits per axis, offset by 64
  static_assert(G::TX + kDriftMargin + 2 < 64 && G::TY + kDriftMargin + 2 < 64 &&
                    G::TZ + kDriftMargin + 2 < 64,
                "record cells are 8-bit offsets from the tile origin");
  // the two accumulations, chosen once per deposit: a test at every entry
  // cost the order-2 kernel a sixth of its instructions
  const JWinFixed<G, FA>   add_fixed{ Jw, jb };
  const JWinReal<G, real> add_real{ Jr, jb };

  // 2. particles of the tile (this CTA's part of them), species by species;
  //    with records in chunks, each pushed by the whole CTA and then deposited
  auto part = [&](int k, unsigned y) -> int64_t {
    const int32_t* ts = a.s[k].tile_start + t;
    if (gridDim.y == 1) return ts[y - blockIdx.y];
    // whole groups of 128 particles, the largest lane-strided group
    const unsigned n   = (unsigned)(ts[1] - ts[0]);
    const unsigned len = ((n + gridDim.y - 1) / gridDim.y + 127u) & ~127u;
    return ts[0] + (int64_t)min((uint64_t)n, (uint64_t)len * y);
  };
  int     s  = 0;
  int64_t p0 = part(0, blockIdx.y);  // first particle of the CTA's next group
  for (;;) {
    int pend = 0;  // particles since the last deposit, rounded up to groups
    while (s < a.nsp) {
      const TiledSpecies<real>& S = a.s[s];
      real*          ux[3]  = { (real*)S.sp.ux1, (real*)S.sp.ux2, (real*)S.sp.ux3 };
      const real*    w      = (const real*)S.sp.w;
      int32_t*       ia[3]  = { S.sp.i1, S.sp.i2, S.sp.i3 };
      int32_t*       ipa[3] = { S.sp.i1p, S.sp.i2p, S.sp.i3p };
      float*         da[3]  = { S.sp.dx1, S.sp.dx2, S.sp.dx3 };
      float*         dpa[3] = { S.sp.dx1p, S.sp.dx2p, S.sp.dx3p };
      const int64_t  hi = part(s, blockIdx.y + 1);
      for (; p0 < hi && (!REC || pend + NT <= G::CHUNK); p0 += NT, pend += NT) {
        const int64_t p = p0 + local;
        if (p >= hi) continue;
        // the whole state is loaded before the first test of it: one latency
        Prtl<real> q;
        q.tag = S.sp.tag[p];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          q.i[d]  = ia[d][p];
          q.dx[d] = da[d][p];
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) q.u[d] = ux[d][p];
        const real wq = w[p];
        if (q.tag != PIC_TAG_ALIVE) {
          if (q.tag != PIC_TAG_DEAD) atomicAdd(a.err + ERR_BAD_TAG, 1ull);
          continue;
        }
        if (!cells_in_grid<D>(q.i, a.pc.n)) {
          atomicAdd(a.err + ERR_OUT_OF_GRID, 1ull);
          continue;
        }
        bool near = true, edge = false;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const int T = d == 0 ? G::TX : (d == 1 ? G::TY : G::TZ);
          near = near && (q.i[d] >= T0[d] - M) && (q.i[d] < T0[d] + T + M);
          // a stencil that can reach the ghost layers of a non-periodic axis is
          // deposited at the reference's coordinates: there the reference keeps
          // the raw ghost currents, unfolded along the periodic axes
          edge = edge || (!a.periodic[d] &&
                          (q.i[d] < H::J_LO - M + 1 || q.i[d] >= a.pc.n[d] - (H::J_HI - M) - 1));
        }
        {
          // particles that drifted past the margin, or whose stencil can reach
          // the ghost layers of a non-periodic axis, are left to the
          // per-particle kernel (global gathers, reference coordinates)
          const bool     defer = !near || edge;
          const unsigned ball  = __ballot_sync(__activemask(), defer);
          if (defer) {
            const int leader = __ffs(ball) - 1;
            unsigned  base   = 0;
            if (lane == leader) base = atomicAdd(S.ovf_count, (unsigned)__popc(ball));
            base = __shfl_sync(ball, base, leader);
            S.ovf[base + __popc(ball & ((1u << lane) - 1u))] = (int32_t)p;
            continue;
          }
        }
        real e0[3], b0[3];
        int  ic[3] = { q.i[0] + ng, q.i[1] + ng, D == 3 ? q.i[2] + ng : 0 };
        real dc[3] = { (real)q.dx[0], (real)q.dx[1], D == 3 ? (real)q.dx[2] : (real)0 };
        if constexpr (O == 0) interp_zigzag<D, real>(ebv, ic, dc, e0, b0);
        else                  interp_shape<D, O, real>(ebv, ic, dc, e0, b0);
#pragma unroll
        for (int d = 0; d < D; ++d) {
          e0[d] = e0[d] * a.dx;
          b0[d] = b0[d] * a.dx;
        }
        if (S.vay) vay<real>(S.ndth, q.u, e0, b0);
        else       boris<real>(S.ndth, q.u, e0, b0);
        move_and_bound<D, real>(q, true, a.dt, a.dx, a.pc);
#pragma unroll
        for (int d = 0; d < D; ++d) {
          ia[d][p] = q.i[d];
          da[d][p] = q.dx[d];
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) ux[d][p] = q.u[d];
        if (q.tag != PIC_TAG_ALIVE) S.sp.tag[p] = q.tag;
        if (a.write_prev) {
#pragma unroll
          for (int d = 0; d < D; ++d) {
            ipa[d][p] = q.ip[d];
            dpa[d][p] = q.dxp[d];
          }
        }
        if (q.tag == PIC_TAG_DEAD || S.charge == (real)0) continue;
        // deposit at the coordinates before the periodic wrap (a shift of both
        // i and i_prev by n leaves every contribution unchanged up to the image
        // cell, which the flush folds back)
#pragma unroll
        for (int d = 0; d < D; ++d) {
          q.i[d] -= q.wrap[d];
          q.ip[d] -= q.wrap[d];
        }
        // in fixed point the weight carries the power-of-two scale, so every
        // contribution arrives scaled exactly (w 2^s rounds like w)
        const real wp = fixed ? wq * scale : wq;
        if constexpr (REC) {
          // the 2D deposit reads the out-of-plane velocity, the 3D one none
          real vp[3] = { 0, 0, 0 };
          if constexpr (D == 2) deposit_velocity<D, real>(q, a.dx, vp);
          const bool unmoved = support_unmoved<D, O, real>(q);
          if (!G::REC_ALL && unmoved) {
            if (fixed)
              deposit_with_velocity<D, O, real, BOX_UNMOVED>(q, vp, wp, S.charge, a.inv_dt, ng, nullptr,
                                                      add_fixed);
            else
              deposit_with_velocity<D, O, real, BOX_UNMOVED>(q, vp, wp, S.charge, a.inv_dt, ng, nullptr,
                                                      add_real);
            continue;
          }
          // first node of the box, as a J-window word (the move stays within
          // one cell per axis: move_and_bound steps the cell by one at most)
          int      word  = jb;
          unsigned cells = 0;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const int f0 = shape_first_node<O>(q.ip[d], (real)q.dxp[d]);
            const int f1 = shape_first_node<O>(q.i[d], (real)q.dx[d]);
            word += (min(f0, f1) + ng) * (d == 0 ? 1 : (d == 1 ? G::WJ0 : G::WJ0 * G::WJ1));
            cells |= ((unsigned)(q.i[d] - T0[d] + 64) << (8 * d)) |
                     ((unsigned)(q.ip[d] - q.i[d] + 1) << (24 + 2 * d));
          }
          const int region = unmoved ? 0 : 1;
          unsigned  cls = (unsigned)word, row = 0;
          for (int k = 0; k < 32; ++k, ++cls) {
            cls &= 31u;
            row = atomicAdd(&s_cnt[region][cls], 1u);
            if (row < (unsigned)G::ROWS) break;
          }
          uint4*     r     = recs + (unmoved ? 0 : G::moved) + (size_t)(row * 32 + cls) * G::RECW;
          const real coeff = wp * S.charge;
          const unsigned z = D == 3 ? __float_as_uint(q.dx[2]) : 0u;
          const unsigned y = D == 3 ? __float_as_uint(q.dxp[2]) : 0u;
          if constexpr (sizeof(real) == 4) {
            __stcg(r, make_uint4(cells, __float_as_uint(q.dx[0]), __float_as_uint(q.dx[1]),
                                 D == 3 ? z : __float_as_uint((float)vp[2])));
            __stcg(r + 1, make_uint4(__float_as_uint(q.dxp[0]), __float_as_uint(q.dxp[1]), y,
                                     __float_as_uint((float)coeff)));
          } else {
            const long long cb = __double_as_longlong((double)coeff);
            const long long vb = __double_as_longlong((double)vp[2]);
            __stcg(r, make_uint4(cells, __float_as_uint(q.dx[0]), __float_as_uint(q.dx[1]), z));
            __stcg(r + 1, make_uint4(__float_as_uint(q.dxp[0]), __float_as_uint(q.dxp[1]), y, 0u));
            __stcg(r + 2, make_uint4((unsigned)cb, (unsigned)(cb >> 32), (unsigned)vb,
                                     (unsigned)(vb >> 32)));
          }
        } else {
          if (fixed)
            deposit_particle<D, O, real, true>(q, wp, S.charge, a.inv_dt, a.dx, ng, nullptr,
                                               add_fixed);
          else
            deposit_particle<D, O, real, true>(q, wp, S.charge, a.inv_dt, a.dx, ng, nullptr,
                                               add_real);
        }
      }
      if (p0 < hi) break;  // the chunk is full
      if (++s < a.nsp) p0 = part(s, blockIdx.y);
    }
    __syncthreads();
    if constexpr (REC) {
      // a warp per row of records; a record's coefficient is the product
      // weight * charge that the direct deposit forms, times charge 1
      auto drain = [&](auto unmoved, const auto& add) {
        constexpr bool UNMOVED = decltype(unmoved)::value;
        const unsigned mine    = min(s_cnt[UNMOVED ? 0 : 1][lane], (unsigned)G::ROWS);
        const int      rows    = (int)__reduce_max_sync(0xffffffffu, mine);
        uint4*         first   = recs + (UNMOVED ? 0 : G::moved);
        for (int row = wid; row < rows; row += NT / 32) {
          uint4* line = first + (size_t)row * (32 * G::RECW);
          if (row < (int)mine) {
            const uint4* r  = line + lane * G::RECW;
            const uint4  u0 = __ldcg(r), u1 = __ldcg(r + 1);
            Prtl<real>   q;
            const float dx[3]  = { __uint_as_float(u0.y), __uint_as_float(u0.z), __uint_as_float(u0.w) };
            const float dxp[3] = { __uint_as_float(u1.x), __uint_as_float(u1.y), __uint_as_float(u1.z) };
            real        vp[3]  = { 0, 0, 0 }, coeff;
            if constexpr (sizeof(real) == 4) {
              coeff = __uint_as_float(u1.w);
              vp[2] = D == 2 ? dx[2] : 0.f;
            } else {
              const uint4 u2 = __ldcg(r + 2);
              coeff = __hiloint2double((int)u2.y, (int)u2.x);
              vp[2] = __hiloint2double((int)u2.w, (int)u2.z);
            }
#pragma unroll
            for (int d = 0; d < D; ++d) {
              q.i[d]   = (int)((u0.x >> (8 * d)) & 255u) - 64 + T0[d];
              q.ip[d]  = q.i[d] + (int)((u0.x >> (24 + 2 * d)) & 3u) - 1;
              q.dx[d]  = dx[d];
              q.dxp[d] = dxp[d];
            }
            deposit_with_velocity<D, O, real, UNMOVED ? BOX_UNMOVED : BOX_FULL>(q, vp, coeff, (real)1, a.inv_dt, ng, nullptr,
                                                       add);
          }
          // the row has been used: what L2 still holds of it is dropped
          // unwritten (a line is written again before it is read again)
          __syncwarp();
          if (lane < 4 * G::RECW) discard_l2_line((const char*)line + 128 * lane);
        }
      };
      if (fixed) {
        if constexpr (G::REC_ALL) drain(std::true_type{}, add_fixed);
        drain(std::false_type{}, add_fixed);
      } else {
        if constexpr (G::REC_ALL) drain(std::true_type{}, add_real);
        drain(std::false_type{}, add_real);
      }
      __syncthreads();
      if (threadIdx.x < 64) (&s_cnt[0][0])[threadIdx.x] = 0u;
    }
    if (s >= a.nsp) break;
    __syncthreads();
  }
  if constexpr (REC) {
    if (threadIdx.x == 0) give_slot(a.st, s_slot);
  }

  // 3. flush the J window (periodic images folded onto active cells)
  for (int idx = threadIdx.x; idx < 3 * G::NJ; idx += NT) {
    real      v = 0;
    long long units = 0;  // the entry in global units (exact accumulator)
    if (fixed) {
      if (!FA::nonzero(Jw + idx, G::PLANE)) continue;
      const long long t = FA::total(Jw + idx, G::PLANE);
      if (global_unit) units = (long long)((unsigned long long)t << (a.fj.bits - b));
      else             v = FA::to_real(t, unscale);
    } else {
      v = Jr[idx];
      if (v == (real)0) continue;
      if (global_unit) units = __float2ll_rn((float)v * ldexpf(1.f, a.fj.bits - ex));
    }
    int       r  = idx;
    const int wi = r % G::WJ0;
    r /= G::WJ0;
    const int wj = r % G::WJ1;
    r /= G::WJ1;
    const int wk = r % G::WJ2;
    const int c  = r / G::WJ2;
    int       gc[3] = { T0[0] - H::J_LO + wi, T0[1] - H::J_LO + wj,
                        D == 3 ? T0[2] - H::J_LO + wk : 0 };
    bool      inside = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (a.periodic[d]) {
        gc[d] = wrap_periodic(gc[d], a.pc.n[d]);
      } else if (gc[d] < -ng || gc[d] >= a.pc.n[d] + ng) {
        inside = false;
      }
    }
    if (inside) {
      if constexpr (sizeof(real) == 4) {
        if (global_unit) {
          a.fj.add_units(gc[0] + ng, gc[1] + ng, D == 3 ? gc[2] + ng : 0, c, units);
          continue;
        }
      }
      atomicAdd(a.J.p + a.J.idx(gc[0] + ng, gc[1] + ng, D == 3 ? gc[2] + ng : 0, c), v);
    } else {
      atomicAdd(a.err + ERR_STENCIL_OUT, 1ull);
    }
  }
}

template <int D, int O, typename real>
cudaError_t launch_push_deposit_tiled(const TiledArgs<real>& a, cudaStream_t s);

// 16-byte words of one record buffer and the number of buffers (the CTAs that
// can be resident at once); no buffers (0, 0) where none are used
template <int D, int O, typename real>
cudaError_t deposit_record_words(size_t* words, int* slots);

// tile shape of a build, for the host (sort key and tile count)
void tile_shape(int dim, int real_bytes, int order, int out[3]);

}  // namespace pic
