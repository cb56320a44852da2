// Output preparation on the device (the compute half of the reference's field
// and particle output; the file format is the caller's):
//   - ComputeMoments (src/framework/domain/metadomain_io.cpp:123-170) with
//     ParticleMoments_kernel<SRPIC, Minkowski, F> (src/kernels/
//     particle_moments.hpp:44-405): Rho, Charge, N, Nppc, T^{ab}, V deposited
//     at cell centres with a spline or constant smoothing window;
//   - SynchronizeFields(Comm::Bckp) for periodic axes (the additive ghost fold);
//   - NormalizeVectorByRho_kernel (particle_moments.hpp:407-478);
//   - ComputeDivergence_kernel (src/kernels/divergences.hpp), Cartesian;
//   - DeepCopyFields + FieldsToPhys_kernel<Minkowski> (src/kernels/
//     fields_to_phys.hpp:33-241) fused with the writer's downsampling
//     (src/output/writer.cpp:199-300): one pass from the staggered field to a
//     packed array of cell-centred tetrad components;
//   - PrtlToPhys_kernel<SRPIC, Minkowski, false> (src/kernels/prtls_to_phys.hpp:
//     28-218) as Particles::OutputWrite launches it
//     (src/framework/containers/particles_io.cpp:93-235): every stride-th
//     particle in physical coordinates.
// The moment deposit ends in global atomics, so its sums run in no fixed order,
// like the reference's ScatterView on CUDA.
#include <climits>
#include <cmath>
#include <type_traits>

#include "ctx_internal.cuh"

using namespace pic_internal;

namespace pic {
namespace {

// prtl_shape::S1..S6 (src/kernels/particle_shapes.hpp:25-166), x >= 0; the
// constants are rounded to real from their double quotients and every
// product and sum is evaluated in the reference's order
template <int ORDER, typename real>
__device__ __forceinline__ real spline(real x) {
  const real ZERO = 0, ONE = 1, TWO = 2, THREE = 3, HALF = 0.5, THREE_HALFS = 1.5;
  const real INV_4 = 0.25, INV_8 = 0.125, THREE_FOURTHS = 0.75;
  const real x2 = x * x, x3 = x * x * x;
  switch (ORDER) {
    case 0: return ONE;
    case 1: return x < ONE ? ONE - x : ZERO;
    case 2:
      if (x < HALF) return (real)0.75 - x2;
      if (x < THREE_HALFS) return HALF * ((THREE_HALFS - x) * (THREE_HALFS - x));
      return ZERO;
    case 3:
      if (x < ONE) return (real)(2.0 / 3.0) - x2 + HALF * x3;
      if (x < TWO) return (real)(4.0 / 3.0) - TWO * x + x2 - (real)(1.0 / 6.0) * x3;
      return ZERO;
    case 4:
      if (x < HALF)
        return (real)(115.0 / 192.0) - (real)(5.0 / 8.0) * x2 + INV_4 * (x2 * x2);
      if (x < THREE_HALFS)
        return (real)(55.0 / 96.0) + (real)(5.0 / 24.0) * x - (real)(5.0 / 4.0) * x2 +
               (real)(5.0 / 6.0) * x3 - (real)(1.0 / 6.0) * (x2 * x2);
      if (x < (real)2.5)
        return (real)(625.0 / 384.0) - (real)(125.0 / 48.0) * x + (real)(25.0 / 16.0) * x2 -
               (real)(5.0 / 12.0) * x3 + (real)(1.0 / 24.0) * (x2 * x2);
      return ZERO;
    case 5:
      if (x <= ONE)
        return (real)(11.0 / 20.0) - HALF * x2 + INV_4 * (x2 * x2) - (real)(1.0 / 12.0) * x3 * x2;
      if (x < TWO)
        return (real)(17.0 / 40.0) + (real)(5.0 / 8.0) * x - (real)(7.0 / 4.0) * x2 +
               (real)(5.0 / 4.0) * x3 - (real)(3.0 / 8.0) * (x2 * x2) +
               (real)(1.0 / 24.0) * x3 * x2;
      if (x < THREE)
        return (real)(81.0 / 40.0) - (real)(27.0 / 8.0) * x + (real)(9.0 / 4.0) * x2 -
               THREE_FOURTHS * x3 + INV_8 * (x2 * x2) - (real)(1.0 / 120.0) * x3 * x2;
      return ZERO;
    case 6:
      if (x <= HALF)
        return (real)(5887.0 / 11520.0) - (real)(77.0 / 192.0) * x2 +
               (real)(7.0 / 48.0) * (x2 * x2) - (real)(1.0 / 36.0) * (x3 * x3);
      if (x < THREE_HALFS)
        return (real)(7861.0 / 15360.0) - (real)(7.0 / 768.0) * x - (real)(91.0 / 256.0) * x2 -
               (real)(35.0 / 288.0) * x3 + (real)(21.0 / 64.0) * (x2 * x2) -
               (real)(7.0 / 48.0) * x3 * x2 + (real)(1.0 / 48.0) * (x3 * x3);
      if (x < (real)2.5)
        return (real)(1379.0 / 7680.0) + (real)(1267.0 / 960.0) * x - (real)(329.0 / 128.0) * x2 +
               (real)(133.0 / 72.0) * x3 - (real)(21.0 / 32.0) * (x2 * x2) +
               (real)(7.0 / 60.0) * x3 * x2 - (real)(1.0 / 120.0) * (x3 * x3);
      if (x < (real)3.5)
        return (real)(117649.0 / 46080.0) - (real)(16807.0 / 3840.0) * x +
               (real)(2401.0 / 768.0) * x2 - (real)(343.0 / 288.0) * x3 +
               (real)(49.0 / 192.0) * (x2 * x2) - (real)(7.0 / 240.0) * x3 * x2 +
               (real)(1.0 / 720.0) * (x3 * x3);
      return ZERO;
  }
  return ZERO;
}

dim3 blocks_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > pic::sm_count() * 32) b = pic::sm_count() * 32;
  return dim3((unsigned)b);
}

template <typename real>
struct MomArgs {
  SpeciesPtrs     sp;
  FieldView<real> buf;
  int             comp, ng, n[3];
  int             id, c1, c2, smoothing, use_weights;
  real            inv_n0, dx;
};

// cell and coefficient of particle p (particle_moments.hpp:291-365,
// Cartesian); false for one that is not deposited
template <int D, typename real>
__device__ __forceinline__ bool moment_of(const MomArgs<real>& a, int64_t p, int* cell, real& coeff,
                                          bool& out_of_grid) {
  const real     ONE   = 1;
  const int32_t* ia[3] = { a.sp.i1, a.sp.i2, a.sp.i3 };
  const real*    ux[3] = { (const real*)a.sp.ux1, (const real*)a.sp.ux2, (const real*)a.sp.ux3 };
  // every load before the first test: one latency
  const bool moving = a.id == PIC_MOM_T || a.id == PIC_MOM_V;
  const short tag   = a.sp.tag[p];
  real        u[3]  = { 0, 0, 0 };
  const real  w     = a.use_weights ? ((const real*)a.sp.w)[p] : ONE;
  if (moving) {
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = ux[c][p];
  }
  out_of_grid = false;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    cell[d] = ia[d][p];
    if (cell[d] < 0 || cell[d] >= a.n[d]) out_of_grid = true;
  }
  out_of_grid = out_of_grid && tag == PIC_TAG_ALIVE;
  if (tag != PIC_TAG_ALIVE || out_of_grid) return false;
  const real mass = (real)a.sp.mass, m_or_1 = a.sp.mass == 0.0f ? ONE : mass;
  if (moving) {
    const real nsq  = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
    const real u0   = a.sp.mass == 0.0f ? sqrt(nsq) : sqrt(ONE + nsq);
    auto       comp = [&](int c) { return c == 1 ? u[0] : (c == 2 ? u[1] : (c == 3 ? u[2] : u0)); };
    if (a.id == PIC_MOM_T) {
      coeff = m_or_1 / u0;
      coeff *= comp(a.c1);
      coeff *= comp(a.c2);
    } else {
      coeff = m_or_1 * comp(a.c1) / u0;
    }
  } else {
    coeff = a.id == PIC_MOM_RHO ? mass : a.id == PIC_MOM_CHARGE ? (real)a.sp.charge : ONE;
  }
  if (a.id != PIC_MOM_NPPC) {
    // sqrt_det_h of Minkowski<D> (src/metrics/minkowski.h:144-152)
    const real h = D == 2 ? a.dx * a.dx : a.dx * a.dx * a.dx;
    coeff *= a.inv_n0 / h;
    if (a.use_weights) coeff *= w;
  }
  return true;
}

// The windowed kernel's block: threads, particles, nodes of its shared window
template <int T, int C, int N>
struct MomBlock {
  static constexpr int THREADS = T, CHUNK = C, NODES = N;
};
using MomDense = MomBlock<512, 4096, 4096>;
using MomLarge = MomBlock<512, 2048, 4352>;
using MomSmall = MomBlock<256, 512, 2560>;
using MomWide  = MomBlock<256, 512, 3840>;  // orders 5 and 6

// Window sums in fixed point. A contribution v, |v| <= 2^18, is split into
// h + l 2^-19 (two words) or h + m 2^-19 + l 2^-38 (three), integers of at most 2^18
// each, all but the last exact, and each is added to a 32-bit word: a chunk's additions
// (2^12 at most) stay within 2^30. The integers come by adding 1.5 * 2^23, whose
// sum's low mantissa bits they are.
constexpr int kMomTop = 18, kMomStep = 19;
template <int WORDS>
__device__ __forceinline__ void moment_add(int* w, int plane, float v) {
  const float MAGIC = 12582912.f, STEP = (float)(1 << kMomStep);
  float       t = v + MAGIC, r = v - (t - MAGIC);
  atomicAdd(w, __float_as_int(t) - 0x4B400000);
#pragma unroll
  for (int k = 1; k < WORDS; ++k) {
    t = __fmaf_rn(r, STEP, MAGIC);
    r = __fmaf_rn(r, STEP, MAGIC - t);
    atomicAdd(w + k * plane, __float_as_int(t) - 0x4B400000);
  }
}
// The sum of a node times 2^e. Two words: one conversion and two exact scalings (2^e
// itself may be no normal float), because FP64 runs at 1/64 of the FP32 rate: in
// double the flush took a twelfth of the kernel.
template <int WORDS>
__device__ __forceinline__ float moment_total(const int* w, int plane, int e) {
  const long long t = (long long)w[0] * (1 << kMomStep) + w[plane];
  if constexpr (WORDS == 2) {
    const int a = (e - kMomStep) / 2;
    return __ll2float_rn(t) * __int_as_float((127 + a) << 23) *
           __int_as_float((127 + e - kMomStep - a) << 23);
  } else {
    return (float)ldexp((double)t + (double)w[2 * plane] * (1.0 / (1 << kMomStep)), e - kMomStep);
  }
}
// the block's largest coefficient over the largest of a cell, at most, for two words
// and for three
constexpr float kMomRange2 = 256.f, kMomRange3 = 67108864.f;

// a chunk's particles waiting for their deposit, queued by the shared-memory
// bank (of 32) of their window's first node: row r holds the r-th of each bank
template <int D, typename B>
struct MomQueue {
  int   word[B::CHUNK];
  float dx[D][B::CHUNK];
  float coeff[B::CHUNK];
};
// shape factors of one particle along each axis, and the products over its nodes
template <int D, int ORDER, typename real>
struct MomShape {
  static constexpr int W = (ORDER + 1) / 2;
  real                 s[D][2 * W + 1];
  __device__ __forceinline__ MomShape(const float* dx, bool spl) {
    const real cst = (real)1 / ((real)2 * (real)W + (real)1);
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
      for (int q = 0; q <= 2 * W; ++q) {
        const real dl = fabs((real)dx[d] - ((real)(q - W) + (real)0.5));
        s[d][q]       = spl ? spline<ORDER, real>(dl) : cst;
      }
  }
  template <typename F>
  __device__ __forceinline__ void each(const F& add) const {
#pragma unroll
    for (int k = 0; k <= (D == 3 ? 2 * W : 0); ++k)
#pragma unroll
      for (int j = 0; j <= 2 * W; ++j)
#pragma unroll
        for (int i = 0; i <= 2 * W; ++i) {
          real sh = s[0][i] * s[1][j];
          if (D == 3) sh = sh * s[D - 1][k];
          add(i, j, k, sh);
        }
  }
};

// one particle's additions straight onto the grid
template <int D, int ORDER, typename real>
__device__ __forceinline__ void moment_on_grid(const MomArgs<real>& a, const int* cell,
                                               const float* dx, real coeff) {
  using Shape = MomShape<D, ORDER, real>;
  const Shape S(dx, a.smoothing == PIC_SMOOTH_SPLINE);
  S.each([&](int i, int j, int k, real sh) {
    atomicAdd(a.buf.p + a.buf.idx(cell[0] + i - Shape::W + a.ng, cell[1] + j - Shape::W + a.ng,
                                  D == 3 ? cell[2] + k - Shape::W + a.ng : 0, a.comp),
              coeff * sh);
  });
}

// ParticleMoments_kernel::operator() (particle_moments.hpp:291-404),
// Cartesian, every particle's additions straight onto the grid
template <int D, int ORDER, typename real>
__global__ void __launch_bounds__(256) k_output_moment_direct(MomArgs<real> a,
                                                              unsigned long long* err) {
  const float*  da[3]  = { a.sp.dx1, a.sp.dx2, a.sp.dx3 };
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < a.sp.npart; p += stride) {
    int   cell[3] = { 0, 0, 0 };
    real  coeff;
    bool  oob;
    const bool ok = moment_of<D, real>(a, p, cell, coeff, oob);
    if (oob) atomicAdd(err + ERR_OUT_OF_GRID, 1ull);
    if (!ok) continue;
    float dx[D];
#pragma unroll
    for (int d = 0; d < D; ++d) dx[d] = da[d][p];
    moment_on_grid<D, ORDER, real>(a, cell, dx, coeff);
  }
}

template <int D, typename B>
constexpr size_t moment_smem() {
  return 8 * B::NODES + sizeof(MomQueue<D, B>);
}

// The same in FP32, a block depositing CHUNK consecutive particles. Where these
// lie together (any spatial order: a box of cells that the window
// holds), it sums them in a shared-memory window in fixed point, scaled by the
// block's largest coefficient, and adds the window's nodes to the grid once;
// particles apart from the others (across a periodic edge, after a drift) add
// to the grid directly, and so does a whole block in random order. The sums
// have two words a node, 37 bits below the scale, where every occupied cell's largest
// coefficient is within kMomRange2 of the block's, and three, 56 bits, where it is
// within kMomRange3 (a cold region beside a hot one): an addition errs by 2^-29
// of its cell's largest coefficient at most, where a float sum errs by 2^-24 of itself.
// A block that neither suits (or whose coefficients are not finite, or too small) adds
// to the grid, like one whose window has no room for the third word.
// A particle makes (2 W + 1)^D additions, which bound the kernel. 16.8 M
// sorted particles at order 2 took 1.64 ms with global atomics, which meet in
// a few L2 lines, 1.05 ms in the window in their own order (the lanes of one
// cell meet in its words, eight wavefronts an atomic), and 0.43 ms queued by
// bank, a warp's 32 lanes adding in 32 banks (with sums of 30 bits; 7.1 M took 191
// us with those, 203 us with these).
template <int D, int ORDER, typename B>
__global__ void __launch_bounds__(B::THREADS) k_output_moment(MomArgs<float> a,
                                                              unsigned long long* err) {
  using real         = float;
  constexpr int W    = (ORDER + 1) / 2;
  constexpr int ROWS = B::CHUNK / 32;
  constexpr int kMomThreads = B::THREADS, kMomChunk = B::CHUNK;
  extern __shared__ __align__(16) int win[];
  MomQueue<D, B>& qu = *reinterpret_cast<MomQueue<D, B>*>(win + 2 * B::NODES);
  __shared__ int      s_lo[3], s_hi[3], s_mid[3], s_bad;
  __shared__ unsigned s_max, s_min, s_cnt[32];
  const int32_t* ia[3] = { a.sp.i1, a.sp.i2, a.sp.i3 };
  const float*   da[3] = { a.sp.dx1, a.sp.dx2, a.sp.dx3 };
  const int64_t  p0    = (int64_t)blockIdx.x * kMomChunk;
  const int      n     = (int)(a.sp.npart - p0 < kMomChunk ? a.sp.npart - p0 : kMomChunk);
  const int      tid = threadIdx.x, lane = tid & 31;
  if (tid < 3) s_lo[tid] = INT_MAX, s_hi[tid] = INT_MIN, s_mid[tid] = 0;
  if (tid < 32) s_cnt[tid] = 0u;
  if (tid == 0) s_bad = 0, s_max = 0u, s_min = ~0u;
  __syncthreads();
  // 1. the block's box of cells (of all that lie in the grid)
  {
    int lo[3] = { INT_MAX, INT_MAX, INT_MAX }, hi[3] = { INT_MIN, INT_MIN, INT_MIN };
#pragma unroll
    for (int k = 0; k < kMomChunk / kMomThreads; ++k) {
      const int l = k * kMomThreads + tid;
      if (l >= n) break;
      int  c[3];
      bool ok = true;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        c[d] = ia[d][p0 + l];
        ok   = ok && c[d] >= 0 && c[d] < a.n[d];
      }
      if (!ok) continue;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        lo[d] = min(lo[d], c[d]), hi[d] = max(hi[d], c[d]);
        if (l == n / 2) s_mid[d] = c[d];
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
      hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
      if (lane == 0) atomicMin(&s_lo[d], lo[d]), atomicMax(&s_hi[d], hi[d]);
    }
  }
  __syncthreads();
  // 2. the window: all cells, or those within 12 of the middle particle's where
  //    these hold half of the particles
  int  w0[3] = { 0, 0, 0 }, wn[3] = { 1, 1, 1 };
  bool windowed = false;
  if (s_lo[0] <= s_hi[0]) {
    for (int t = 0; t < 2 && !windowed; ++t) {
      if (t == 1) {
        int near = 0;
#pragma unroll
        for (int k = 0; k < kMomChunk / kMomThreads; ++k) {
          const int l  = k * kMomThreads + tid;
          bool      in = l < n;
#pragma unroll
          for (int d = 0; d < D; ++d) in = in && abs(ia[d][p0 + l] - s_mid[d]) <= 12;
          near += __syncthreads_count(in);
        }
        if (2 * near < n) break;
      }
      int64_t vol = 1;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const int lo = t == 0 ? s_lo[d] : max(s_lo[d], s_mid[d] - 12);
        const int hi = t == 0 ? s_hi[d] : min(s_hi[d], s_mid[d] + 12);
        w0[d] = lo - W, wn[d] = hi - lo + 1 + 2 * W;
        vol *= max(wn[d], 0);
      }
      windowed = vol > 0 && vol <= B::NODES;
    }
  }
  const int nodes = wn[0] * wn[1] * wn[2];
  if (windowed)
    for (int e = tid; e < min(3 * nodes, 2 * B::NODES); e += kMomThreads) win[e] = 0;
  __syncthreads();
  // 3. the window's particles into the queue, the others onto the grid
  float cmax = 0.f;
  bool  bad  = false;
#pragma unroll 1
  for (int l = tid; l < n; l += kMomThreads) {
    int   cell[3] = { 0, 0, 0 };
    real  coeff;
    bool  oob;
    const bool ok = moment_of<D, real>(a, p0 + l, cell, coeff, oob);
    if (oob) atomicAdd(err + ERR_OUT_OF_GRID, 1ull);
    if (!ok) continue;
    float dx[D];
    bool  in = windowed;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      dx[d] = da[d][p0 + l];
      in    = in && cell[d] - W >= w0[d] && cell[d] + W < w0[d] + wn[d];
    }
    if (!in) {
      moment_on_grid<D, ORDER, real>(a, cell, dx, coeff);
      continue;
    }
    const float m = fabsf(coeff);
    bad  = bad || !(m <= 0x1p126f);
    cmax = fmaxf(cmax, m);
    const int word = (cell[0] - W - w0[0]) +
                     wn[0] * ((cell[1] - W - w0[1]) + (D == 3 ? wn[1] * (cell[2] - W - w0[2]) : 0));
    // the cell's largest coefficient, in the first word of its window's first
    // node (non-negative floats order as their bits)
    atomicMax(win + word, __float_as_int(m));
    // a full bank hands its particles to the next one; the queue holds them all
    unsigned cls = (unsigned)word, row = 0;
    for (int k = 0; k < 32; ++k, ++cls) {
      cls &= 31u;
      row = atomicAdd(&s_cnt[cls], 1u);
      if (row < (unsigned)ROWS) break;
    }
    const int e = (int)(row * 32 + cls);
    qu.word[e]  = word;
    qu.coeff[e] = coeff;
#pragma unroll
    for (int d = 0; d < D; ++d) qu.dx[d][e] = dx[d];
  }
  const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(cmax));
  if (!windowed) return;
  if (lane == 0) atomicMax(&s_max, m);
  if (bad) s_bad = 1;
  __syncthreads();
  // the least of the occupied cells' largest coefficients
  unsigned least = ~0u;
  for (int e = tid; e < nodes; e += kMomThreads) {
    if (win[e] > 0) least = min(least, (unsigned)win[e]);
    win[e] = 0;
  }
  least = __reduce_min_sync(0xffffffffu, least);
  if (lane == 0) atomicMin(&s_min, least);
  __syncthreads();
  const float top = __uint_as_float(s_max), low = __uint_as_float(s_min);
  if (top == 0.f && !s_bad) return;
  const int words = s_bad || top < 0x1p-108f ? 0
                    : top <= kMomRange2 * low ? 2
                    : top <= kMomRange3 * low && 3 * nodes <= 2 * B::NODES ? 3 : 0;
  // 4. the queue into the window; |coefficient| < 2^ex, and its product with
  //    the shape factors stays below
  int ex = 0;
  if (words) frexpf(top * 1.0000002f, &ex);
  const float scale = ldexpf(1.f, kMomTop - ex);
  const int   mine  = (int)min(s_cnt[lane], (unsigned)ROWS);
  auto deposit = [&](auto&& add) {
    for (int row = tid >> 5; row < mine; row += kMomThreads / 32) {
      const int e = row * 32 + lane, word = qu.word[e];
      float     dx[D];
#pragma unroll
      for (int d = 0; d < D; ++d) dx[d] = qu.dx[d][e];
      const MomShape<D, ORDER, real> S(dx, a.smoothing == PIC_SMOOTH_SPLINE);
      const real                     coeff = qu.coeff[e];
      S.each([&](int i, int j, int k, real sh) {
        add(word + i + wn[0] * (j + wn[1] * k), coeff, sh);
      });
    }
  };
  auto on_grid = [&](int e, real v) {
    const int i = e % wn[0], j = (e / wn[0]) % wn[1], k = e / (wn[0] * wn[1]);
    atomicAdd(a.buf.p + a.buf.idx(w0[0] + i + a.ng, w0[1] + j + a.ng, D == 3 ? w0[2] + k + a.ng : 0,
                                  a.comp),
              v);
  };
  if (words == 0) {
    deposit([&](int e, real coeff, real sh) { on_grid(e, coeff * sh); });
    return;
  }
  if (words == 2)
    deposit([&](int e, real coeff, real sh) { moment_add<2>(win + e, nodes, (coeff * scale) * sh); });
  else
    deposit([&](int e, real coeff, real sh) { moment_add<3>(win + e, nodes, (coeff * scale) * sh); });
  __syncthreads();
  for (int e = tid; e < nodes; e += kMomThreads) {
    const real v = words == 2 ? moment_total<2>(win + e, nodes, ex - kMomTop)
                              : moment_total<3>(win + e, nodes, ex - kMomTop);
    if (v != (real)0) on_grid(e, v);
  }
}

template <int D, int ORDER, typename B>
cudaError_t launch_moment_window(const MomArgs<float>& a, unsigned long long* err, cudaStream_t s) {
  constexpr size_t  smem = moment_smem<D, B>();
  const cudaError_t e    = cudaFuncSetAttribute(k_output_moment<D, ORDER, B>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  PIC_KL(k_output_moment<D, ORDER, B>
         <<<(unsigned)((a.sp.npart + B::CHUNK - 1) / B::CHUNK), B::THREADS, smem, s>>>(a, err));
  return cudaGetLastError();
}

template <int D, int ORDER, typename real>
cudaError_t launch_moment(const MomArgs<real>& a, unsigned long long* err, cudaStream_t s) {
  // FP64 adds to the grid: the window's fixed point would be coarser than double.
  // In the windowed kernel, whose 128 KB of shared memory it asked for all the
  // same, a 3D block of 512 threads had an SM to itself: 27,648 particles at order 2
  // took 157 us there, 13 us so, 7.1 M 1.96 and 1.81 ms, 480,000 in 2D 88 and 68 us
  if constexpr (sizeof(real) == 4) {
    // Three large blocks per SM at least, else small ones; the largest in 3D from 8
    // particles per cell on, where their windows still hold most chunks. Small,
    // 2048 and 4096 particles, us at order 2: 27,648 at 2 per cell 9, 19 and 31; 1.0 M at
    // 4 per cell 41, 37 and 45; 7.1 M at 8 per cell 258, 222 and 203 (order 3 746, 607
    // and 583); 6.5 M in 2D 147, 114 and 142.
    // Orders 5 and 6, seldom used and long to compile, have small ones with room for
    // their wider windows at every size.
    if constexpr (ORDER <= 4) {
      if (a.sp.npart / MomLarge::CHUNK >= 3 * pic::sm_count()) {
        if constexpr (D == 3)
          if (a.sp.npart >= 8 * (int64_t)a.n[0] * a.n[1] * a.n[2])
            return launch_moment_window<D, ORDER, MomDense>(a, err, s);
        return launch_moment_window<D, ORDER, MomLarge>(a, err, s);
      }
    }
    return launch_moment_window<D, ORDER, std::conditional_t<ORDER <= 4, MomSmall, MomWide>>(a, err, s);
  } else {
    PIC_KL(k_output_moment_direct<D, ORDER, real><<<blocks_for(a.sp.npart), 256, 0, s>>>(a, err));
    return cudaGetLastError();
  }
}

// NormalizeVectorByRho_kernel (particle_moments.hpp:407-478): cmp::AlmostZero
// with the real type's epsilon (src/global/utils/comparators.h:37-42)
template <typename real>
__global__ void k_normalize_by_rho(GridInfo g, FieldView<real> f, int cr, int v1, int v2, int v3) {
  const real    eps   = sizeof(real) == 4 ? (real)1.1920928955078125e-07 : (real)2.220446049250313e-16;
  const int     n3    = g.dim == 3 ? g.n[2] : 1;
  const int64_t count = (int64_t)g.n[0] * g.n[1] * n3;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t % g.n[0]) + g.ng;
    const int j = (int)((t / g.n[0]) % g.n[1]) + g.ng;
    const int k = g.dim == 3 ? (int)(t / ((int64_t)g.n[0] * g.n[1])) + g.ng : 0;
    const real rho = f.p[f.idx(i, j, k, cr)];
    if (fabs(rho) <= eps) continue;
    f.p[f.idx(i, j, k, v1)] /= rho;
    f.p[f.idx(i, j, k, v2)] /= rho;
    f.p[f.idx(i, j, k, v3)] /= rho;
  }
}

// FieldsToPhys_kernel<Minkowski> (fields_to_phys.hpp:125-236) at the output
// cells (o1, o2, o3) * dwn (writer.cpp:199-300 with first cell 0), written to
// out[c][o3][o2][o1]
template <int D, typename real>
__global__ void k_output_field(GridInfo g, FieldView<real> F, int c0, int ncomp, unsigned flags,
                               real dx, int d1, int d2, int d3, int o1, int o2, int o3,
                               real* out) {
  const real    INV_2 = 0.5, INV_4 = 0.25;
  const int64_t count = (int64_t)o1 * o2 * o3;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)(t % o1), b = (int)((t / o1) % o2), e = (int)(t / ((int64_t)o1 * o2));
    const int i = a * d1 + g.ng, j = b * d2 + g.ng, k = D == 3 ? e * d3 + g.ng : 0;
    auto      at = [&](int ii, int jj, int kk, int c) { return F.p[F.idx(ii, jj, kk, c0 + c)]; };
    real      f[3];
    if (ncomp == 1) {
      out[t] = at(i, j, k, 0);
      continue;
    }
    if (flags & PIC_OUT_INTERP_EDGES) {
      if (D == 2) {
        f[0] = INV_2 * (at(i, j, k, 0) + at(i, j + 1, k, 0));
        f[1] = INV_2 * (at(i, j, k, 1) + at(i + 1, j, k, 1));
        f[2] = INV_4 * (at(i, j, k, 2) + at(i + 1, j, k, 2) + at(i, j + 1, k, 2) +
                        at(i + 1, j + 1, k, 2));
      } else {
        f[0] = INV_4 * (at(i, j, k, 0) + at(i, j + 1, k, 0) + at(i, j, k + 1, 0) +
                        at(i, j + 1, k + 1, 0));
        f[1] = INV_4 * (at(i, j, k, 1) + at(i + 1, j, k, 1) + at(i, j, k + 1, 1) +
                        at(i + 1, j, k + 1, 1));
        f[2] = INV_4 * (at(i, j, k, 2) + at(i + 1, j, k, 2) + at(i, j + 1, k, 2) +
                        at(i + 1, j + 1, k, 2));
      }
    } else if (flags & PIC_OUT_INTERP_FACES) {
      f[0] = INV_2 * (at(i, j, k, 0) + at(i + 1, j, k, 0));
      f[1] = INV_2 * (at(i, j, k, 1) + at(i, j + 1, k, 1));
      f[2] = D == 3 ? INV_2 * (at(i, j, k, 2) + at(i, j, k + 1, 2)) : at(i, j, k, 2);
    } else {
      f[0] = at(i, j, k, 0);
      f[1] = at(i, j, k, 1);
      f[2] = at(i, j, k, 2);
    }
    // transform<Idx::U, Idx::T> of Minkowski (minkowski.h:263-300): times
    // sqrt(h_ii) = dx along the simulated axes
    if (flags & PIC_OUT_TO_HAT) {
      f[0] *= dx;
      f[1] *= dx;
      if (D == 3) f[2] *= dx;
    }
    out[t]             = f[0];
    out[t + count]     = f[1];
    out[t + 2 * count] = f[2];
  }
}

// ComputeDivergence_kernel<Minkowski> (src/kernels/divergences.hpp:23-135),
// Cartesian branch: the backward-difference divergence of E over the active
// cells, summed left to right as written there
template <int D, typename real>
__global__ void k_divergence(GridInfo g, FieldView<real> EB, FieldView<real> out, int comp) {
  const int     n3    = D == 3 ? g.n[2] : 1;
  const int64_t count = (int64_t)g.n[0] * g.n[1] * n3;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t % g.n[0]) + g.ng;
    const int j = (int)((t / g.n[0]) % g.n[1]) + g.ng;
    const int k = D == 3 ? (int)(t / ((int64_t)g.n[0] * g.n[1])) + g.ng : 0;
    real      v = EB.p[EB.idx(i, j, k, 0)] - EB.p[EB.idx(i - 1, j, k, 0)] +
             EB.p[EB.idx(i, j, k, 1)] - EB.p[EB.idx(i, j - 1, k, 1)];
    if (D == 3) v = v + EB.p[EB.idx(i, j, k, 2)] - EB.p[EB.idx(i, j, k - 1, 2)];
    out.p[out.idx(i, j, k, comp)] = v;
  }
}

template <typename real>
struct PrtlOutArgs {
  SpeciesPtrs sp;
  int64_t     stride, nout;
  int         dim;
  real        dx, xmin[3];
  real*       x[3];
  real*       u[3];
  real*       w;
};

// PrtlToPhys_kernel<SRPIC, Minkowski, false>::operator() (prtls_to_phys.hpp:
// 121-200): convert<Crd::Cd, Crd::Ph> is x * dx + x_min (minkowski.h:161-178),
// and transform_xyz<XYZ, T> leaves Cartesian velocities unchanged
template <typename real>
__global__ void k_output_particles(PrtlOutArgs<real> a) {
  const int32_t* ia[3] = { a.sp.i1, a.sp.i2, a.sp.i3 };
  const float*   da[3] = { a.sp.dx1, a.sp.dx2, a.sp.dx3 };
  const real*    ux[3] = { (const real*)a.sp.ux1, (const real*)a.sp.ux2, (const real*)a.sp.ux3 };
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < a.nout;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = p * a.stride;
    for (int d = 0; d < a.dim; ++d) {
      const real xc = (real)ia[d][q] + (real)da[d][q];
      a.x[d][p]     = xc * a.dx + a.xmin[d];
    }
    for (int d = 0; d < 3; ++d) a.u[d][p] = ux[d][q];
    a.w[p] = ((const real*)a.sp.w)[q];
  }
}

template <typename real>
int output_moment(pic_ctx* c, const pic_species* sp, int nsp, const pic_moment_params* prm,
                  void* bckp, int comp, cudaStream_t s) {
  MomArgs<real> a{};
  a.buf  = em_view<real>(c, bckp);
  a.comp = comp;
  a.ng   = c->grid.ng;
  for (int d = 0; d < 3; ++d) a.n[d] = c->grid.n[d];
  a.id          = prm->id;
  a.c1          = prm->c1;
  a.c2          = prm->c2;
  a.smoothing   = prm->smoothing;
  a.use_weights = prm->use_weights;
  a.inv_n0      = (real)prm->inv_n0;
  a.dx          = (real)prm->dx;
  for (int k = 0; k < nsp; ++k) {
    if (sp[k].npart == 0) continue;
    a.sp = sptrs(sp + k);
    cudaError_t e = cudaErrorInvalidValue;
#define PIC_MOM_CASE(DD, OO)                 \
  if (c->grid.dim == DD && prm->order == OO) \
    e = launch_moment<DD, OO, real>(a, c->d_err, s);
#define PIC_MOM_ORDERS(DD) \
  PIC_MOM_CASE(DD, 0) PIC_MOM_CASE(DD, 1) PIC_MOM_CASE(DD, 2) PIC_MOM_CASE(DD, 3) \
  PIC_MOM_CASE(DD, 4) PIC_MOM_CASE(DD, 5) PIC_MOM_CASE(DD, 6)
    PIC_MOM_ORDERS(2)
    PIC_MOM_ORDERS(3)
#undef PIC_MOM_ORDERS
#undef PIC_MOM_CASE
    if (e != cudaSuccess) return PIC_ERR_CUDA;
  }
  return PIC_OK;
}

template <typename real>
int output_field(pic_ctx* c, const void* src, int is_em, int c0, int ncomp, unsigned flags,
                 double dx, const int32_t dwn[3], void* out, cudaStream_t s) {
  const GridInfo  g = ginfo(c);
  FieldView<real> F = is_em ? em_view<real>(c, src) : cur_view<real>(c, src);
  int             o[3] = { 1, 1, 1 }, dd[3] = { 1, 1, 1 };
  for (int d = 0; d < g.dim; ++d) {
    dd[d] = dwn[d];
    o[d]  = (g.n[d] + dwn[d] - 1) / dwn[d];
  }
  const int64_t count = (int64_t)o[0] * o[1] * o[2];
  if (g.dim == 2)
    PIC_KL(k_output_field<2, real><<<blocks_for(count), 256, 0, s>>>(
      g, F, c0, ncomp, flags, (real)dx, dd[0], dd[1], dd[2], o[0], o[1], o[2], (real*)out));
  else
    PIC_KL(k_output_field<3, real><<<blocks_for(count), 256, 0, s>>>(
      g, F, c0, ncomp, flags, (real)dx, dd[0], dd[1], dd[2], o[0], o[1], o[2], (real*)out));
  return cuda_status(cudaGetLastError());
}

template <typename real>
int output_particles(pic_ctx* c, const pic_species* sp, int64_t stride, double dx,
                     const double xmin[3], void* const x[3], void* const u[3], void* w,
                     int64_t nout, cudaStream_t s) {
  PrtlOutArgs<real> a{};
  a.sp     = sptrs(sp);
  a.stride = stride;
  a.nout   = nout;
  a.dim    = c->grid.dim;
  a.dx     = (real)dx;
  for (int d = 0; d < 3; ++d) {
    a.xmin[d] = (real)xmin[d];
    a.x[d]    = d < a.dim ? (real*)x[d] : nullptr;
    a.u[d]    = (real*)u[d];
  }
  a.w = (real*)w;
  PIC_KL(k_output_particles<real><<<blocks_for(nout), 256, 0, s>>>(a));
  return cuda_status(cudaGetLastError());
}

}  // namespace
}  // namespace pic

extern "C" {

int pic_output_moment(pic_ctx* c, const pic_species* sp, int32_t nspecies,
                      const pic_moment_params* prm, void* bckp, int32_t comp, void* stream) {
  if (!c || !prm || !bckp || nspecies < 0 || (nspecies > 0 && !sp)) return PIC_ERR_ARG;
  if (comp < 0 || comp >= 6) return PIC_ERR_ARG;
  if (prm->id < PIC_MOM_RHO || prm->id > PIC_MOM_V) return PIC_ERR_ARG;
  // only the spline and constant windows exist (shapeFunction,
  // particle_moments.hpp:111-144); orders beyond 6 need more than 3 ghosts
  if (prm->smoothing != PIC_SMOOTH_SPLINE && prm->smoothing != PIC_SMOOTH_CONST) return PIC_ERR_ARG;
  if (prm->order < 0) return PIC_ERR_ARG;
  if (prm->order > 6) return PIC_ERR_UNSUPPORTED;
  if ((prm->order + 1) / 2 > c->grid.ng) return PIC_ERR_ARG;  // "Window size too large"
  if (prm->id == PIC_MOM_T && (prm->c1 < 0 || prm->c1 > 3 || prm->c2 < 0 || prm->c2 > 3))
    return PIC_ERR_ARG;
  if (prm->id == PIC_MOM_V && (prm->c1 < 1 || prm->c1 > 3)) return PIC_ERR_ARG;
  if (!(prm->dx > 0.0)) return PIC_ERR_ARG;
  for (int k = 0; k < nspecies; ++k) {
    int st = validate_species(c, sp + k, false);
    if (st != PIC_OK) return st;
    // "Rho & Charge for massless particles not defined"
    if ((prm->id == PIC_MOM_RHO || prm->id == PIC_MOM_CHARGE) && sp[k].mass == 0.0f)
      return PIC_ERR_ARG;
  }
  cudaStream_t s = strm(stream);
  return is_f64(c) ? pic::output_moment<double>(c, sp, nspecies, prm, bckp, comp, s)
                   : pic::output_moment<float>(c, sp, nspecies, prm, bckp, comp, s);
}

int pic_sync_moments(pic_ctx* c, void* bckp, int32_t c0, int32_t c1, void* stream) {
  if (!c || !bckp || c0 < 0 || c1 > 6 || c0 >= c1) return PIC_ERR_ARG;
  if (is_f64(c))
    return cuda_status(pic::launch_adj_fold<double>(ginfo(c), em_view<double>(c, bckp), c0, c1,
                                                    strm(stream)));
  return cuda_status(pic::launch_adj_fold<float>(ginfo(c), em_view<float>(c, bckp), c0, c1,
                                                 strm(stream)));
}

int pic_normalize_by_rho(pic_ctx* c, void* bckp, int32_t c_rho, int32_t c_v1, int32_t c_v2,
                         int32_t c_v3, void* stream) {
  if (!c || !bckp) return PIC_ERR_ARG;
  const int cs[4] = { c_rho, c_v1, c_v2, c_v3 };
  for (int a = 0; a < 4; ++a) {
    if (cs[a] < 0 || cs[a] >= 6) return PIC_ERR_ARG;
    for (int b = 0; b < a; ++b)
      if (cs[a] == cs[b]) return PIC_ERR_ARG;
  }
  const GridInfo g     = ginfo(c);
  const int64_t  cells = (int64_t)g.n[0] * g.n[1] * (g.dim == 3 ? g.n[2] : 1);
  cudaStream_t   s     = strm(stream);
  if (is_f64(c))
    PIC_KL(pic::k_normalize_by_rho<double><<<pic::blocks_for(cells), 256, 0, s>>>(
      g, em_view<double>(c, bckp), c_rho, c_v1, c_v2, c_v3));
  else
    PIC_KL(pic::k_normalize_by_rho<float><<<pic::blocks_for(cells), 256, 0, s>>>(
      g, em_view<float>(c, bckp), c_rho, c_v1, c_v2, c_v3));
  return cuda_status(cudaGetLastError());
}

int pic_output_divergence(pic_ctx* c, const void* EB, void* bckp, int32_t comp, void* stream) {
  if (!c || !EB || !bckp || comp < 0 || comp >= 6) return PIC_ERR_ARG;
  if (c->grid.ng < 1) return PIC_ERR_ARG;
  const GridInfo g     = ginfo(c);
  const int64_t  cells = (int64_t)g.n[0] * g.n[1] * (g.dim == 3 ? g.n[2] : 1);
  cudaStream_t   s     = strm(stream);
  if (is_f64(c)) {
    if (g.dim == 2)
      PIC_KL(pic::k_divergence<2, double><<<pic::blocks_for(cells), 256, 0, s>>>(
        g, em_view<double>(c, EB), em_view<double>(c, bckp), comp));
    else
      PIC_KL(pic::k_divergence<3, double><<<pic::blocks_for(cells), 256, 0, s>>>(
        g, em_view<double>(c, EB), em_view<double>(c, bckp), comp));
  } else {
    if (g.dim == 2)
      PIC_KL(pic::k_divergence<2, float><<<pic::blocks_for(cells), 256, 0, s>>>(
        g, em_view<float>(c, EB), em_view<float>(c, bckp), comp));
    else
      PIC_KL(pic::k_divergence<3, float><<<pic::blocks_for(cells), 256, 0, s>>>(
        g, em_view<float>(c, EB), em_view<float>(c, bckp), comp));
  }
  return cuda_status(cudaGetLastError());
}

int pic_output_field(pic_ctx* c, const void* src, int32_t is_em, int32_t c0, int32_t ncomp,
                     uint32_t flags, double dx, const int32_t dwn[3], void* out, void* stream) {
  if (!c || !src || !dwn || !out) return PIC_ERR_ARG;
  const int nc = is_em ? 6 : 3;
  if (ncomp != 1 && ncomp != 3) return PIC_ERR_ARG;
  if (c0 < 0 || c0 + ncomp > nc) return PIC_ERR_ARG;
  if (flags & ~(PIC_OUT_INTERP_EDGES | PIC_OUT_INTERP_FACES | PIC_OUT_TO_HAT)) return PIC_ERR_ARG;
  if ((flags & PIC_OUT_INTERP_EDGES) && (flags & PIC_OUT_INTERP_FACES)) return PIC_ERR_ARG;
  if (ncomp == 1 && flags != 0) return PIC_ERR_ARG;
  // the interpolation reads one cell beyond the active range
  if ((flags & (PIC_OUT_INTERP_EDGES | PIC_OUT_INTERP_FACES)) && c->grid.ng < 1) return PIC_ERR_ARG;
  if ((flags & PIC_OUT_TO_HAT) && !(dx > 0.0)) return PIC_ERR_ARG;
  for (int d = 0; d < c->grid.dim; ++d)
    if (dwn[d] < 1) return PIC_ERR_ARG;
  cudaStream_t s = strm(stream);
  return is_f64(c) ? pic::output_field<double>(c, src, is_em, c0, ncomp, flags, dx, dwn, out, s)
                   : pic::output_field<float>(c, src, is_em, c0, ncomp, flags, dx, dwn, out, s);
}

int pic_output_particles(pic_ctx* c, const pic_species* sp, int64_t stride, double dx,
                         const double xmin[3], void* const x_out[3], void* const u_out[3],
                         void* w_out, int64_t* nout, void* stream) {
  if (!c || !sp || !xmin || !x_out || !u_out || !w_out || !nout || stride < 1) return PIC_ERR_ARG;
  int st = validate_species(c, sp, false);
  if (st != PIC_OK) return st;
  const int64_t n = sp->npart / stride;
  *nout           = n;
  if (n == 0) return PIC_OK;
  for (int d = 0; d < c->grid.dim; ++d)
    if (!x_out[d]) return PIC_ERR_ARG;
  if (!u_out[0] || !u_out[1] || !u_out[2]) return PIC_ERR_ARG;
  cudaStream_t s = strm(stream);
  return is_f64(c) ? pic::output_particles<double>(c, sp, stride, dx, xmin, x_out, u_out, w_out, n, s)
                   : pic::output_particles<float>(c, sp, stride, dx, xmin, x_out, u_out, w_out, n, s);
}

}  // extern "C"
