// Particle push and current deposition kernels (SR, Minkowski).
//
// k_push_deposit runs one thread per particle over a grid-stride loop and
// serves three modes: the reference's separate pusher (Pusher_kernel,
// src/kernels/pushers/sr.hpp:117-332), its separate deposit
// (DepositCurrents_kernel, src/kernels/currents_deposit.hpp:108-761), and the
// fused pass that keeps the previous position in registers so the 12
// prev-arrays never round-trip through HBM.
#pragma once

#include <climits>

#include "deposit_fixed.cuh"
#include "fixed_acc.cuh"
#include "pic_common.cuh"

namespace pic {

enum Mode { MODE_PUSH = 0, MODE_DEPOSIT = 1, MODE_FUSED = 2 };

template <typename real>
struct PDArgs {
  SpeciesPtrs     sp;
  PushConsts      pc;
  FieldView<real> EB;
  FieldView<real> J;
  real            dt, dx, ndth, inv_dt, charge;
  int             vay;
  int             write_prev;
  unsigned long long* err;
  // optional: process only the particles listed (indices into the arrays),
  // *list_count of them (a device counter)
  const int32_t*  list       = nullptr;
  const unsigned* list_count = nullptr;
  // optional (FP32): deposit into the exact 64-bit accumulator instead of J
  FixedJ          fj;
  // which of the two kernels takes the particles (BoundArgs::chunked); null: this one
  const unsigned* chunked = nullptr;
  // elements of the EB and J arrays where these can be taken as VecField
  int             eb_count = 0, j_count = 0;
};

// One particle's load and push, stored back; false when nothing is deposited.
// In MODE_DEPOSIT only the loads, of the previous position too.
template <int D, int O, typename real, int MODE, bool PHOTON, typename V>
__device__ __forceinline__ bool push_particle(const PDArgs<real>& a, const V& EB, int64_t p,
                                              Prtl<real>& q) {
  real*    ux[3]  = { (real*)a.sp.ux1, (real*)a.sp.ux2, (real*)a.sp.ux3 };
  int32_t* ia[3]  = { a.sp.i1, a.sp.i2, a.sp.i3 };
  int32_t* ipa[3] = { a.sp.i1p, a.sp.i2p, a.sp.i3p };
  float*   da[3]  = { a.sp.dx1, a.sp.dx2, a.sp.dx3 };
  float*   dpa[3] = { a.sp.dx1p, a.sp.dx2p, a.sp.dx3p };
  q.tag = a.sp.tag[p];
  if constexpr (MODE == MODE_DEPOSIT) {
    if (q.tag == PIC_TAG_DEAD) return false;
  } else {
    if (q.tag != PIC_TAG_ALIVE) {
      if (q.tag != PIC_TAG_DEAD) atomicAdd(a.err + ERR_BAD_TAG, 1ull);
      return false;
    }
  }
#pragma unroll
  for (int d = 0; d < D; ++d) {
    q.i[d]  = ia[d][p];
    q.dx[d] = da[d][p];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) q.u[d] = ux[d][p];
  if (!cells_in_grid<D>(q.i, a.pc.n)) {
    // a cell outside the grid is invalid input; report it, touch nothing
    atomicAdd(a.err + ERR_OUT_OF_GRID, 1ull);
    return false;
  }
  if constexpr (MODE == MODE_DEPOSIT) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      q.ip[d]  = ipa[d][p];
      q.dxp[d] = dpa[d][p];
    }
  } else {
    if constexpr (!PHOTON) {
      real e0[3], b0[3];
      int  ic[3] = { q.i[0] + a.pc.ng, q.i[1] + a.pc.ng, D == 3 ? q.i[2] + a.pc.ng : 0 };
      real dc[3] = { (real)q.dx[0], (real)q.dx[1], D == 3 ? (real)q.dx[2] : (real)0 };
      if constexpr (O == 0) {
        interp_zigzag<D, real>(EB, ic, dc, e0, b0);
      } else {
        interp_shape<D, O, real>(EB, ic, dc, e0, b0);
      }
      // transform_xyz<U, XYZ> (src/metrics/minkowski.h:264-296)
#pragma unroll
      for (int d = 0; d < D; ++d) {
        e0[d] = e0[d] * a.dx;
        b0[d] = b0[d] * a.dx;
      }
      if (a.vay) {
        vay<real>(a.ndth, q.u, e0, b0);
      } else {
        boris<real>(a.ndth, q.u, e0, b0);
      }
    }
    move_and_bound<D, real>(q, !PHOTON, a.dt, a.dx, a.pc);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      ia[d][p] = q.i[d];
      da[d][p] = q.dx[d];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) ux[d][p] = q.u[d];
    if (q.tag != PIC_TAG_ALIVE) a.sp.tag[p] = q.tag;
    if (MODE == MODE_PUSH || a.write_prev) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        ipa[d][p] = q.ip[d];
        dpa[d][p] = q.dxp[d];
      }
    }
  }
  return q.tag != PIC_TAG_DEAD;
}

// scale of the per-particle contributions to the exact accumulator and the
// shift to its unit (see k_push_deposit)
__device__ __forceinline__ void fixed_scale(const FixedJ& fj, float& scale, int& shift) {
  const int b = min(30, fj.bits);
  scale       = ldexpf(1.f, b - fj.exponent());
  shift       = fj.bits - b;
}

// 2D FP32 asks for three CTAs per SM (80 registers instead of the
// allocator's 96, an 8-byte spill): the never-sorted two-stream adjoint
// problem's forward, which runs here, went from 134.1 to 128.8 ms. 3D FP32 at order
// 3 asks for two (128 registers of 255) where it pushes: 3.5 M particles in random
// order 5.20 and 4.54 ms fused, 2.46 and 2.21 ms pushed, in cell order 3.32 and 2.80,
// 1.08 and 0.84 ms.
// VEC (FP32): the fields are read by rows (VecField), and float currents added
// by rows (red_row). Particles in random order are bound by the lines and atomics
// of their stencils in L1 and L2, rows are two thirds fewer: 14.2 M particles at
// order 2 pushed in 5.43 and deposited in 3.92 ms without, 4.11 and 2.25 with
// (three blocks per SM for the deposit: 2.22, two 2.38, one 2.76 ms).
template <int D, int O, typename real, int MODE, bool PHOTON, bool VEC>
__device__ __forceinline__ void push_deposit_all(const PDArgs<real>& a) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t n = a.list ? (int64_t)*a.list_count : a.sp.npart;
  // exact accumulator: each contribution is rounded to a multiple of
  // 2^(ex - b) with b = min(30, bits), an int32 conversion (a 64-bit one
  // runs on the FP64 pipe), then shifted to the call's unit 2^(ex - bits)
  float fj_scale = 0.f;
  int   fj_shift = 0;
  if constexpr (sizeof(real) == 4 && MODE != MODE_PUSH) {
    if (a.fj.p) fixed_scale(a.fj, fj_scale, fj_shift);
  }
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += stride) {
    const int64_t p = a.list ? (int64_t)a.list[t] : t;
    Prtl<real>    q;
    bool          deposits, rows = false;
    if constexpr (VEC && MODE != MODE_DEPOSIT) {
      // (an invalid cell is refused by the push; the support starts at most two
      // nodes below the cell)
      const VecField EB(a.EB, a.eb_count);
      rows = EB.template covers<O + 1>(a.sp.i1[p] + a.pc.ng + 1, a.sp.i2[p] + a.pc.ng + 1,
                                       D == 3 ? a.sp.i3[p] + a.pc.ng + 1 : 0);
      if (rows) deposits = push_particle<D, O, real, MODE, PHOTON>(a, EB, p, q);
    }
    if (!rows) deposits = push_particle<D, O, real, MODE, PHOTON>(a, a.EB, p, q);
    if (!deposits) continue;
    if constexpr (VEC && MODE != MODE_PUSH) {
      if (!a.fj.p && a.j_count > 0) {
        real vp[3];
        deposit_velocity<D, real>(q, a.dx, vp);
        const int s1 = (int)a.J.s1, s2 = (int)a.J.s2, s3 = (int)a.J.s3;
        const bool ok = deposit_rows<D, O>(
          q, vp[2], ((const real*)a.sp.w)[p], a.charge, a.inv_dt, a.pc.ng, a.pc.ext,
          [&](auto n, int i, int j, int k, int c, const float* r) {
            constexpr int M = decltype(n)::value;
            const int     e = i + j * s1 + k * s2 + c * s3;
            if (M <= 4 && (e + M + 3) / 4 * 4 <= a.j_count) {
              red_row<(M <= 4 ? M : 4)>(a.J.p + e, r);
            } else if (M == 5 && (e + M + 3) / 4 * 4 <= a.j_count) {
              red_row<4>(a.J.p + e, r);
              if (r[M - 1] != 0.f) atomicAdd(a.J.p + e + 4, r[M - 1]);
            } else {
#pragma unroll
              for (int m = 0; m < M; ++m)
                if (r[m] != 0.f) atomicAdd(a.J.p + e + m, r[m]);
            }
          });
        if (!ok) atomicAdd(a.err + ERR_STENCIL_OUT, 1ull);
        continue;
      }
    }
    if constexpr (MODE != MODE_PUSH) {
      const real*            w    = (const real*)a.sp.w;
      const FieldView<real>& J    = a.J;
      auto                   to_J = [&](int i, int j, int k, int c, real v) {
        atomicAdd(J.p + J.idx(i, j, k, c), v);
      };
      bool ok;
      if constexpr (sizeof(real) == 4) {
        if (a.fj.p)
          ok = deposit_particle<D, O, real>(q, w[p], a.charge, a.inv_dt, a.dx, a.pc.ng, a.pc.ext,
                                            [&](int i, int j, int k, int c, real v) {
                                              const int x = __float2int_rn(v * fj_scale);
                                              a.fj.add_units(i, j, k, c,
                                                             (long long)((unsigned long long)
                                                                         (long long)x << fj_shift));
                                            });
        else
          ok = deposit_particle<D, O, real>(q, w[p], a.charge, a.inv_dt, a.dx, a.pc.ng, a.pc.ext,
                                            to_J);
      } else {
        ok = deposit_particle<D, O, real>(q, w[p], a.charge, a.inv_dt, a.dx, a.pc.ng, a.pc.ext,
                                          to_J);
      }
      if (!ok) atomicAdd(a.err + ERR_STENCIL_OUT, 1ull);
    }
  }
}

template <int D, int O, typename real, int MODE, bool PHOTON, bool VEC>
__global__ void __launch_bounds__(256, (D == 2 && sizeof(real) == 4)
                                           ? 3
                                           : (VEC ? (MODE == MODE_DEPOSIT ? 3 : 2)
                                                  : (O == 3 && sizeof(real) == 4 && MODE != MODE_DEPOSIT ? 2 : 1)))
    k_push_deposit(const __grid_constant__ PDArgs<real> a) {
  if constexpr (D == 2 && O >= 2 && sizeof(real) == 4 && MODE == MODE_FUSED && !PHOTON)
    if (a.chunked && *a.chunked != 0u) return;
  push_deposit_all<D, O, real, MODE, PHOTON, VEC>(a);
}

// The particles that a tiled launch left to this kernel, every species' list in
// one launch (blockIdx.y). The lists are short and a particle is one long chain
// of latencies, so the lists share the SMs: two of 512^2 pairs took 9.5 us each
// in launches of their own, 14 us together, two of 100 x 75 x 61 turbulence 25
// and 45 us. Order 3 in 3D asks for three blocks per SM: 2 x 2.1 M particles all in
// the lists took 3.64 ms, with four 4.34 ms (order 2 1.42 and 1.45, order 1 0.63 and
// 0.56).
constexpr int kMaxTiledSpecies = 4;
template <typename real>
struct DrainArgs {
  PDArgs<real> s[kMaxTiledSpecies];
  int          n = 0;
};
template <int D, int O, typename real>
__global__ void __launch_bounds__(128, (D == 2 && sizeof(real) == 4) ? 6 : (O == 3 ? 3 : 4))
    k_push_deposit_lists(const __grid_constant__ DrainArgs<real> d) {
  push_deposit_all<D, O, real, MODE_FUSED, false, false>(d.s[blockIdx.y]);
}

// The grid nodes around the cells of a block's n consecutive particles from p0
// on (2D): nodes w0 to w0 + wn - 1 per axis, ghost-free, two below the cells
// and three above, which holds the interpolation's and the deposit's stencils
// at every order with one cell of move. All cells that lie in the grid, or,
// where that is more than max_nodes, those within 8 of the middle particle's, if
// half of the particles are there; none (wn = 0) when neither fits. sh: four shared
// ints.
__device__ __forceinline__ void chunk_window(const SpeciesPtrs& sp, const int* n_grid, int64_t p0,
                                             int n, int max_nodes, int* sh, int* w0, int* wn) {
  const int tid = threadIdx.x;
  int       mid[2];
  if (tid < 2) sh[tid] = INT_MAX, sh[2 + tid] = INT_MIN;
  mid[0] = sp.i1[p0 + n / 2], mid[1] = sp.i2[p0 + n / 2];
  __syncthreads();
  int lo[2] = { INT_MAX, INT_MAX }, hi[2] = { INT_MIN, INT_MIN };
  for (int l = tid; l < n; l += blockDim.x) {
    const int c[2] = { sp.i1[p0 + l], sp.i2[p0 + l] };
    if (!cells_in_grid<2>(c, n_grid)) continue;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      lo[d] = min(lo[d], c[d]), hi[d] = max(hi[d], c[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
    hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
    if ((tid & 31) == 0) atomicMin(&sh[d], lo[d]), atomicMax(&sh[2 + d], hi[d]);
  }
  __syncthreads();
  if (cells_in_grid<2>(mid, n_grid)) {
    for (int t = 0; t < 2; ++t) {
      if (t == 1) {
        int near = 0;
        for (int l = tid; l - tid < n; l += blockDim.x)
          near += __syncthreads_count(l < n && abs(sp.i1[p0 + l] - mid[0]) <= 8 &&
                                      abs(sp.i2[p0 + l] - mid[1]) <= 8);
        if (2 * near < n) break;
      }
      int64_t nodes = 1;
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const int l = t == 0 ? sh[d] : max(sh[d], mid[d] - 8);
        const int h = t == 0 ? sh[2 + d] : min(sh[2 + d], mid[d] + 8);
        w0[d] = l - 2, wn[d] = h - l + 6;
        nodes *= wn[d];
      }
      if (nodes <= max_nodes) return;
    }
  }
  w0[0] = w0[1] = wn[0] = wn[1] = 0;
}

// the window's nodes of the six field components, component-major (zero
// outside the array)
template <typename real>
__device__ __forceinline__ void stage_window(const FieldView<real>& F, const PushConsts& pc,
                                             const int* w0, const int* wn, real* out) {
  const int nodes = wn[0] * wn[1];
  for (int e = threadIdx.x; e < nodes; e += blockDim.x) {
    const int  i = w0[0] + e % wn[0] + pc.ng, j = w0[1] + e / wn[0] + pc.ng;
    const bool ok = i >= 0 && i < pc.ext[0] && j >= 0 && j < pc.ext[1];
#pragma unroll
    for (int c = 0; c < 6; ++c) out[c * nodes + e] = ok ? F.ld(i, j, 0, c) : (real)0;
  }
}

// Fused push + deposit of consecutive particles of a species without a tile
// binning (2D, FP32, the exact accumulator): a block takes `chunk` of them
// and, where they lie together (particles in cell order, or drifted from it
// without spreading far), reads E and B from a shared-memory window and sums
// their currents there as the integers the exact accumulator takes, adding each
// node of the window to it once. J is the same to the bit as with an addition
// per entry. The per-particle kernel is bound by its 21 to 40 64-bit global
// atomics per particle at order 2 and by the 64-bit addresses of its 54 field
// reads: 1.05 M cell-ordered particles, 16 per cell, took 135 us, in windows 79.
// Particles that do not lie with the others go through the grid as before.
template <int O>
__global__ void __launch_bounds__(256, O == 3 ? 3 : 4) k_push_deposit_chunk(const __grid_constant__ PDArgs<float> a, int ls) {
  constexpr int chunk = kChunk;
  using FA = FixedAcc<float>;
  __shared__ float    EBw[6 * kChunkNodes];
  __shared__ unsigned win[6 * kChunkNodes];
  __shared__ int      sh[4];
  if (*a.chunked == 0u) return;
  const int64_t p0  = (int64_t)blockIdx.x * chunk;
  const int     n   = (int)(a.sp.npart - p0 < chunk ? a.sp.npart - p0 : chunk);
  const int     tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  int           w0[2], wn[2];
  chunk_window(a.sp, a.pc.n, p0, n, kChunkNodes, sh, w0, wn);
  const int nodes = wn[0] * wn[1];
  stage_window(a.EB, a.pc, w0, wn, EBw);
  for (int e = tid; e < 6 * nodes; e += 256) win[e] = 0u;
  float scale;
  int   shift;
  fixed_scale(a.fj, scale, shift);
  __syncthreads();
  const int             ng = a.pc.ng;
  const int             org = -(w0[0] + ng) - (w0[1] + ng) * wn[0];
  const SmemView<float> EBv{ EBw, w0[0] + ng, w0[1] + ng, 0, wn[0], 0, nodes };
  // ls warps read their particles interleaved
  const int    local = (wid / ls) * (32 * ls) + ls * lane + wid % ls;
  const float* w     = (const float*)a.sp.w;
  for (int l = local; l < n; l += 256) {
    const int64_t p  = p0 + l;
    const int     c[2] = { a.sp.i1[p], a.sp.i2[p] };
    bool          in   = cells_in_grid<2>(c, a.pc.n);
#pragma unroll
    for (int d = 0; d < 2; ++d) in = in && c[d] - 2 >= w0[d] && c[d] + 3 < w0[d] + wn[d];
    Prtl<float> q;
    bool        ok;
    if (in ? !push_particle<2, O, float, MODE_FUSED, false>(a, EBv, p, q)
           : !push_particle<2, O, float, MODE_FUSED, false>(a, a.EB, p, q))
      continue;
    // a particle that crossed a periodic edge deposits at its new coordinates
    if (in && q.wrap[0] == 0 && q.wrap[1] == 0)
      ok = deposit_particle<2, O, float>(
        q, w[p], a.charge, a.inv_dt, a.dx, ng, a.pc.ext, [&](int i, int j, int, int c, float v) {
          FA::add(win + (org + i + j * wn[0] + c * nodes), 3 * nodes, v * scale);
        });
    else
      ok = deposit_particle<2, O, float>(
        q, w[p], a.charge, a.inv_dt, a.dx, ng, a.pc.ext, [&](int i, int j, int k, int c, float v) {
          const int x = __float2int_rn(v * scale);
          a.fj.add_units(i, j, k, c, (long long)((unsigned long long)(long long)x << shift));
        });
    if (!ok) atomicAdd(a.err + ERR_STENCIL_OUT, 1ull);
  }
  __syncthreads();
  for (int e = tid; e < 3 * nodes; e += 256) {
    if (!FA::nonzero(win + e, 3 * nodes)) continue;
    a.fj.add_units(w0[0] + e % nodes % wn[0] + ng, w0[1] + e % nodes / wn[0] + ng, 0, e / nodes,
                   (long long)((unsigned long long)FA::total(win + e, 3 * nodes) << shift));
  }
}

// host-side launcher, explicitly instantiated per (D, O, real)
template <int D, int O, typename real>
cudaError_t launch_push_deposit(const PDArgs<real>& a, int mode, bool photon, cudaStream_t s);
template <int D, int O, typename real>
cudaError_t launch_push_deposit_lists(const DrainArgs<real>& d, cudaStream_t s);

}  // namespace pic
