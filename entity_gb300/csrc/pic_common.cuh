// Device-side building blocks of the SR particle-in-cell step: shape
// functions, field interpolation, Boris/Vay velocity updates, the Cartesian
// position update with particle boundaries, and the zigzag / Esirkepov current
// deposit. Every routine follows the operation order of the reference kernel
// it cites (paths relative to the entity repository) so that, compiled with
// -fmad=false, a particle's new cell, offset and momentum are bit-identical to
// the reference arithmetic (but for the sign of an exactly zero field). The
// deposit has two forms, the reference's expressions and a factored one.
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "pic_types.h"

namespace pic {

// ---------------------------------------------------------------------------
// constants per precision: src/global/utils/numeric.h:31-67
// ---------------------------------------------------------------------------
template <typename real>
struct K;
template <>
struct K<float> {
  static constexpr float THIRD = 0.333333f;  // numeric.h:41 (not 1/3)
};
template <>
struct K<double> {
  static constexpr double THIRD = 0.3333333333333333;
};

// one term of an interpolation sum, `c += a * b` as the reference writes it
// (src/kernels/pushers/sr.hpp:1118-1369, gr.hpp:594-662): the product and the
// sum round separately (the library is built with -fmad=false)
template <typename real>
__device__ __forceinline__ real iacc(real a, real b, real c) {
  return c + a * b;
}

// staggering of (ex1, ex2, ex3, bx1, bx2, bx3) per axis: 1 = dual
// (src/kernels/pushers/sr.hpp:1210-1366)
__device__ __forceinline__ int stag_of(int c, int a) {
  // bit (c*3 + a) of the 6x3 table {100, 010, 001, 011, 101, 110}
  constexpr unsigned tbl = (1u << 0) | (1u << 4) | (1u << 8) | (1u << 10) | (1u << 11) |
                           (1u << 12) | (1u << 14) | (1u << 15) | (1u << 16);
  return (tbl >> (c * 3 + a)) & 1u;
}

// ---------------------------------------------------------------------------
// shape functions: src/kernels/particle_shapes.hpp:25-63, 544-614
// ---------------------------------------------------------------------------
template <typename real>
__device__ __forceinline__ real S3near(real x) {
  const real HALF = 0.5;
  return (real)(2.0 / 3.0) - x * x + HALF * (x * x * x);
}
template <typename real>
__device__ __forceinline__ real S3far(real x) {
  const real TWO = 2;
  return (real)(4.0 / 3.0) - TWO * x + x * x - (real)(1.0 / 6.0) * (x * x * x);
}
template <typename real>
__device__ __forceinline__ real S3f(real x) {
  const real ONE = 1, TWO = 2;
  return x < ONE ? S3near(x) : (x < TWO ? S3far(x) : (real)0);
}

template <int O, bool STAG, typename real>
__device__ __forceinline__ void shape(int i, real di, int& imin, real* S) {
  const real ONE = 1, HALF = 0.5, THREE_FOURTHS = 0.75, THREE_HALFS = 1.5;
  if constexpr (O == 1) {
    if constexpr (!STAG) {
      imin = i;
      S[0] = ONE - di;
      S[1] = di;
    } else {
      if (di < HALF) {
        imin = i - 1;
        S[0] = HALF - di;
        S[1] = ONE - S[0];
      } else {
        imin = i;
        S[0] = THREE_HALFS - di;
        S[1] = ONE - S[0];
      }
    }
  } else if constexpr (O == 2) {
    if constexpr (!STAG) {
      if (di < HALF) {
        imin = i - 1;
        S[0] = HALF * ((HALF - di) * (HALF - di));
        S[1] = THREE_FOURTHS - di * di;
        S[2] = ONE - S[0] - S[1];
      } else {
        imin = i;
        S[0] = HALF * ((THREE_HALFS - di) * (THREE_HALFS - di));
        S[1] = THREE_FOURTHS - (ONE - di) * (ONE - di);
        S[2] = ONE - S[0] - S[1];
      }
    } else {
      imin = i - 1;
      S[0] = HALF * ((ONE - di) * (ONE - di));
      S[2] = HALF * (di * di);
      S[1] = ONE - S[0] - S[2];
    }
  } else {
    static_assert(O == 3, "shape orders 1..3");
    // |t - n| is the distance to node n; for 1 < t < 2 its pieces are known
    // (t and 3 - t in (1, 2), t - 1 and 2 - t in (0, 1)): one test in place of
    // two per node
    real t = ONE + di;
    imin   = i - 1;
    if constexpr (STAG) {
      t = (di < HALF ? (real)1.5 : HALF) + di;
      if (di < HALF) imin = i - 2;
    }
    if (t > ONE && t < (real)2) {
      S[0] = S3far<real>(t);
      S[1] = S3near<real>(t - ONE);
      S[2] = S3near<real>((real)2 - t);
      S[3] = S3far<real>((real)3 - t);
    } else {
#pragma unroll
      for (int n = 0; n < 4; n++) S[n] = S3f<real>(fabs(t - (real)n));
    }
  }
}

// prtl_shape::for_deposit (particle_shapes.hpp:934-1024)
template <int O, typename real>
__device__ __forceinline__ void for_deposit(int i_init, real di_init, int i_fin, real di_fin,
                                            int& i_min, int& i_max, real* iS, real* fS) {
  int  i_init_min, i_fin_min;
  real iS_[O + 1], fS_[O + 1];
  shape<O, false>(i_init, di_init, i_init_min, iS_);
  shape<O, false>(i_fin, di_fin, i_fin_min, fS_);
  const real ZERO = 0;
  if (i_init_min < i_fin_min) {
    i_min = i_init_min;
    i_max = i_min + O + 1;
#pragma unroll
    for (int j = 0; j < O + 1; j++) iS[j] = iS_[j];
    iS[O + 1] = ZERO;
    fS[0]     = ZERO;
#pragma unroll
    for (int j = 0; j < O + 1; j++) fS[j + 1] = fS_[j];
  } else if (i_init_min > i_fin_min) {
    i_min = i_fin_min;
    i_max = i_min + O + 1;
    iS[0] = ZERO;
#pragma unroll
    for (int j = 0; j < O + 1; j++) iS[j + 1] = iS_[j];
#pragma unroll
    for (int j = 0; j < O + 1; j++) fS[j] = fS_[j];
    fS[O + 1] = ZERO;
  } else {
    i_min = i_init_min;
    i_max = i_min + O;
#pragma unroll
    for (int j = 0; j < O + 1; j++) iS[j] = iS_[j];
    iS[O + 1] = ZERO;
#pragma unroll
    for (int j = 0; j < O + 1; j++) fS[j] = fS_[j];
    fS[O + 1] = ZERO;
  }
}

// The first node of shape<O, false>'s support for the cell i and offset di:
// i at order 1, i - 1 at order 3, and at order 2 the one the offset's half
// of the cell selects (the same comparison shape makes)
template <int O, typename real>
__device__ __forceinline__ int shape_first_node(int i, real di) {
  if constexpr (O == 2) return di < (real)0.5 ? i - 1 : i;
  else                  return O == 3 ? i - 1 : i;
}

// true when for_deposit's initial and final supports start at the same node
// along every simulated axis: the Esirkepov box is then O + 1 nodes wide on
// each axis (for_deposit's third case), never O + 2
template <int D, int O, typename real, typename P>
__device__ __forceinline__ bool support_unmoved(const P& q) {
  bool same = true;
#pragma unroll
  for (int a = 0; a < D; ++a)
    same = same && shape_first_node<O>(q.ip[a], (real)q.dxp[a]) ==
                       shape_first_node<O>(q.i[a], (real)q.dx[a]);
  return same;
}

// for_deposit when both supports start at the same node (support_unmoved):
// its third case, with i_max = i_min + O known to the compiler's caller
template <int O, typename real>
__device__ __forceinline__ void for_deposit_unmoved(int i_init, real di_init, int i_fin,
                                                    real di_fin, int& i_min, real* iS, real* fS) {
  int  i_fin_min;
  real iS_[O + 1], fS_[O + 1];
  shape<O, false>(i_init, di_init, i_min, iS_);
  shape<O, false>(i_fin, di_fin, i_fin_min, fS_);
#pragma unroll
  for (int j = 0; j < O + 1; j++) {
    iS[j] = iS_[j];
    fS[j] = fS_[j];
  }
  iS[O + 1] = (real)0;
  fS[O + 1] = (real)0;
}

// ---------------------------------------------------------------------------
// field access through a small view; ghost-inclusive indices
// ---------------------------------------------------------------------------
template <typename real>
struct FieldView {
  static constexpr bool kRows = false;
  real*   p;
  int64_t s0, s1, s2, s3;
  __device__ __forceinline__ int64_t idx(int i, int j, int k, int c) const {
    return (int64_t)i * s0 + (int64_t)j * s1 + (int64_t)k * s2 + (int64_t)c * s3;
  }
  __device__ __forceinline__ real ld(int i, int j, int k, int c) const {
    return __ldg(p + idx(i, j, k, c));
  }
};

// A float field whose x1 neighbours are adjacent, whose array starts on 16 bytes
// and whose elements 32 bits index: a stencil row is read as one or two 16-byte
// words. Particles in random order are bound by the lines their reads touch in
// L1, one per load and lane: a row of O + 1 values then counts 1.25 to 1.75
// instead of O + 1.
struct VecField {
  static constexpr bool kRows = true;
  const float*          p;
  int                   s1, s2, s3, count;  // count: elements of the array
  __device__ __forceinline__ VecField(const FieldView<float>& f, int n)
      : p(f.p), s1((int)f.s1), s2((int)f.s2), s3((int)f.s3), count(n) {}
  // the 16-byte words that hold the rows of N nodes per axis from (i, j, k) on
  // lie within the array, for every component (row_elements bounds the sum, for a cell
  // of the grid)
  template <int N>
  __device__ __forceinline__ bool covers(int i, int j, int k) const {
    return i + (j + N) * s1 + (k + N) * s2 + 5 * s3 + N + 8 <= count;
  }
  // no branch: the loads of a stencil's rows are in flight together
  template <int N>
  __device__ __forceinline__ void row(int i, int j, int k, int c, float* r) const {
    static_assert(N >= 1 && N <= 4, "at most four floats");
    const int    idx = i + j * s1 + k * s2 + c * s3, a = idx & 3;
    const float* q = p + (idx - a);
    const float4 v = __ldg(reinterpret_cast<const float4*>(q));
    float4       w = make_float4(0.f, 0.f, 0.f, 0.f);
    asm("{\n\t.reg .pred t;\n\tsetp.gt.s32 t, %4, 4;\n\t"
        "@t ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%5];\n\t}"
        : "+f"(w.x), "+f"(w.y), "+f"(w.z), "+f"(w.w)
        : "r"(a + N), "l"(q + 4));
    const float x[7] = { v.x, v.y, v.z, v.w, w.x, w.y, w.z };
    float       t[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) t[n] = a & 2 ? x[n + 2] : x[n];
#pragma unroll
    for (int n = 0; n < N; ++n) r[n] = a & 1 ? t[n + 1] : t[n];
  }
};

// N values along x1 from (i, j, k) on
template <int N, typename real, typename V>
__device__ __forceinline__ void load_row(const V& f, int i, int j, int k, int c, real* r) {
  if constexpr (V::kRows) {
    f.template row<N>(i, j, k, c, r);
  } else {
#pragma unroll
    for (int n = 0; n < N; ++n) r[n] = f.ld(i + n, j, k, c);
  }
}

// a window of a field staged in shared memory: ghost-inclusive index g maps
// to window index g - off along every axis; 32-bit strides
template <typename real>
struct SmemView {
  static constexpr bool kRows = false;
  const real* p;
  int         off0, off1, off2;
  int         s1, s2, s3;
  __device__ __forceinline__ real ld(int i, int j, int k, int c) const {
    return p[(i - off0) + (j - off1) * s1 + (k - off2) * s2 + c * s3];
  }
};

// ---------------------------------------------------------------------------
// interpolation: src/kernels/pushers/sr.hpp:851-1369 (V = FieldView or SmemView)
// ---------------------------------------------------------------------------
template <int D, typename real, typename V>
__device__ __forceinline__ void interp_zigzag(const V& EB, const int* ic,
                                              const real* d_, real* e0, real* b0) {
  const real ONE = 1, HALF = 0.5;
  int        ind[3];
  real       wpm[3], wpp[3], wdm[3], wdp[3];
#pragma unroll
  for (int a = 0; a < D; ++a) {
    ind[a] = (int)(d_[a] + HALF);
    wpm[a] = ONE - d_[a];
    wpp[a] = d_[a];
    wdm[a] = (real)(ind[a] + 1) - (d_[a] + HALF);
    wdp[a] = ONE - wdm[a];
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    int  lo[3] = { 0, 0, 0 };
    real wm[3], wp[3];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      if (stag_of(c, a)) {
        lo[a] = ic[a] - 1 + ind[a];
        wm[a] = wdm[a];
        wp[a] = wdp[a];
      } else {
        lo[a] = ic[a];
        wm[a] = wpm[a];
        wp[a] = wpp[a];
      }
    }
    if (D == 3 && c == 5) {
      // the reference's 3D Bx3 (sr.hpp:1100-1116) reads the dual x2 stencil
      // (j - 1 + indy, j + indy) with the primal weights ponpmy / ponppy
      wm[1] = wpm[1];
      wp[1] = wpp[1];
    }
    real v;
    if constexpr (D == 2) {
      // sr.hpp:905-977
      const real c000 = EB.ld(lo[0], lo[1], 0, c);
      const real c100 = EB.ld(lo[0] + 1, lo[1], 0, c);
      const real c010 = EB.ld(lo[0], lo[1] + 1, 0, c);
      const real c110 = EB.ld(lo[0] + 1, lo[1] + 1, 0, c);
      const real c00  = c000 * wm[0] + c100 * wp[0];
      const real c10  = c010 * wm[0] + c110 * wp[0];
      v               = c00 * wm[1] + c10 * wp[1];
    } else {
      // sr.hpp:978-1117
      const real c000 = EB.ld(lo[0], lo[1], lo[2], c);
      const real c100 = EB.ld(lo[0] + 1, lo[1], lo[2], c);
      const real c010 = EB.ld(lo[0], lo[1] + 1, lo[2], c);
      const real c110 = EB.ld(lo[0] + 1, lo[1] + 1, lo[2], c);
      const real c001 = EB.ld(lo[0], lo[1], lo[2] + 1, c);
      const real c101 = EB.ld(lo[0] + 1, lo[1], lo[2] + 1, c);
      const real c011 = EB.ld(lo[0], lo[1] + 1, lo[2] + 1, c);
      const real c111 = EB.ld(lo[0] + 1, lo[1] + 1, lo[2] + 1, c);
      const real c00  = c000 * wm[0] + c100 * wp[0];
      const real c10  = c010 * wm[0] + c110 * wp[0];
      const real c0   = c00 * wm[1] + c10 * wp[1];
      const real c01  = c001 * wm[0] + c101 * wp[0];
      const real c11  = c011 * wm[0] + c111 * wp[0];
      const real c1   = c01 * wm[1] + c11 * wp[1];
      v               = c0 * wm[2] + c1 * wp[2];
    }
    if (c < 3) e0[c] = v; else b0[c - 3] = v;
  }
}

// Two floats in one 64-bit register: the packed operations round each half
// as the scalar ones do and take one issue slot for both. The assembler
// contracts a packed product and sum into one multiply-add, whatever
// -fmad=false says (it leaves scalar ones alone), so a sum is written as
// x * 1 + y with a one it cannot see through; the parity tests would show a
// contraction as other bits.
static __constant__ float kPackedOne = 1.f;
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r.v)
      : "l"(b.v), "l"(f2(kPackedOne, kPackedOne).v), "l"(a.v));
  return r;
}
__device__ __forceinline__ void unpack(F2 a, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}

// one component's running sums c += S * EB (sr.hpp:1151-1369), products and
// sums rounded separately; a sum starts with its first product (0 + x is x up
// to the sign of a zero). T is real, or F2 for two components at once; row(b,
// c, t) reads the taps t[a] of row (b, c), Sx, Sy and Sz are the taps' weights.
template <int D, int O, typename T, typename Row, typename WX, typename WY, typename WZ>
__device__ __forceinline__ T interp_sum(Row&& row, WX&& Sx, WY&& Sy, WZ&& Sz) {
  T v;
#pragma unroll
  for (int c = 0; c < (D == 3 ? O + 1 : 1); ++c) {
    T c0;
#pragma unroll
    for (int b = 0; b < O + 1; ++b) {
      T c00, tap[O + 1];
      row(b, c, tap);
#pragma unroll
      for (int a = 0; a < O + 1; ++a) {
        const T t = Sx(a) * tap[a];
        c00       = a == 0 ? t : c00 + t;
      }
      const T t = c00 * Sy(b);
      c0        = b == 0 ? t : c0 + t;
    }
    if constexpr (D == 3) {
      const T t = c0 * Sz(c);
      v         = c == 0 ? t : v + t;
    } else {
      v = c0;
    }
  }
  return v;
}

template <int D, int O, typename real, typename V>
__device__ __forceinline__ void interp_shape(const V& EB, const int* ic,
                                             const real* dc, real* e0, real* b0) {
  // first node and weights per axis, [0] primal and [1] dual
  int  mn[2][3] = { { 0, 0, 0 }, { 0, 0, 0 } };
  real S[2][3][O + 1];
#pragma unroll
  for (int a = 0; a < D; ++a) {
    shape<O, false>(ic[a], dc[a], mn[0][a], S[0][a]);
    shape<O, true>(ic[a], dc[a], mn[1][a], S[1][a]);
  }
  real out[6];
  if constexpr (sizeof(real) == 4) {
    // Two components per packed operation, those of like staggering along x1
    // and x2 together: (ex1, bx2), (ex2, bx1) and the odd pair (ex3, bx3). The
    // order-2 3D interpolation is 468 scalar operations, 195 packed ones.
#pragma unroll
    for (int pr = 0; pr < 3; ++pr) {
      const int ca = pr, cb = pr == 0 ? 4 : (pr == 1 ? 3 : 5);
      const int xa = stag_of(ca, 0), ya = stag_of(ca, 1), za = stag_of(ca, 2);
      const int xb = stag_of(cb, 0), yb = stag_of(cb, 1), zb = stag_of(cb, 2);
      F2 X[O + 1], Y[O + 1], Z[O + 1];
#pragma unroll
      for (int k = 0; k < O + 1; ++k) {
        X[k] = f2(S[xa][0][k], S[xb][0][k]);
        Y[k] = f2(S[ya][1][k], S[yb][1][k]);
        if constexpr (D == 3) Z[k] = f2(S[za][2][k], S[zb][2][k]);
      }
      const F2 r = interp_sum<D, O, F2>(
        [&](int b, int c, F2* t) {
          real u[O + 1], w[O + 1];
          load_row<O + 1>(EB, mn[xa][0], mn[ya][1] + b, D == 3 ? mn[za][2] + c : 0, ca, u);
          load_row<O + 1>(EB, mn[xb][0], mn[yb][1] + b, D == 3 ? mn[zb][2] + c : 0, cb, w);
#pragma unroll
          for (int a = 0; a < O + 1; ++a) t[a] = f2(u[a], w[a]);
        },
        [&](int k) { return X[k]; }, [&](int k) { return Y[k]; }, [&](int k) { return Z[k]; });
      unpack(r, out[ca], out[cb]);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const int x = stag_of(c, 0), y = stag_of(c, 1), z = stag_of(c, 2);
      out[c] = interp_sum<D, O, real>(
        [&](int b, int k, real* t) {
          load_row<O + 1>(EB, mn[x][0], mn[y][1] + b, D == 3 ? mn[z][2] + k : 0, c, t);
        },
        [&](int k) { return S[x][0][k]; }, [&](int k) { return S[y][1][k]; },
        [&](int k) { return S[z][2][k]; });
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    e0[c] = out[c];
    b0[c] = out[c + 3];
  }
}

// ---------------------------------------------------------------------------
// velocity updates: sr.hpp:337-437
// ---------------------------------------------------------------------------
template <typename real>
__device__ __forceinline__ void boris(real ndth, real* u, real* e0, real* b0) {
  const real ONE = 1, TWO = 2;
  real       COEFF = ndth;
  e0[0] *= COEFF;
  e0[1] *= COEFF;
  e0[2] *= COEFF;
  real u0[3] = { u[0] + e0[0], u[1] + e0[1], u[2] + e0[2] };
  COEFF *= ONE / sqrt(ONE + (u0[0] * u0[0] + u0[1] * u0[1] + u0[2] * u0[2]));
  b0[0] *= COEFF;
  b0[1] *= COEFF;
  b0[2] *= COEFF;
  COEFF = TWO / (ONE + (b0[0] * b0[0] + b0[1] * b0[1] + b0[2] * b0[2]));
  const real u1[3] = { (u0[0] + (u0[1] * b0[2] - u0[2] * b0[1])) * COEFF,
                       (u0[1] + (u0[2] * b0[0] - u0[0] * b0[2])) * COEFF,
                       (u0[2] + (u0[0] * b0[1] - u0[1] * b0[0])) * COEFF };
  u0[0] += (u1[1] * b0[2] - u1[2] * b0[1]) + e0[0];
  u0[1] += (u1[2] * b0[0] - u1[0] * b0[2]) + e0[1];
  u0[2] += (u1[0] * b0[1] - u1[1] * b0[0]) + e0[2];
  u[0] = u0[0];
  u[1] = u0[1];
  u[2] = u0[2];
}

template <typename real>
__device__ __forceinline__ void vay(real ndth, real* u, real* e0, real* b0) {
  const real ONE = 1, TWO = 2, INV_2 = 0.5;
  real       COEFF = ndth;
  e0[0] *= COEFF;
  e0[1] *= COEFF;
  e0[2] *= COEFF;
  b0[0] *= COEFF;
  b0[1] *= COEFF;
  b0[2] *= COEFF;
  COEFF      = ONE / sqrt(ONE + (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]));
  real u1[3] = { (u[0] + TWO * e0[0] + (u[1] * b0[2] - u[2] * b0[1]) * COEFF),
                 (u[1] + TWO * e0[1] + (u[2] * b0[0] - u[0] * b0[2]) * COEFF),
                 (u[2] + TWO * e0[2] + (u[0] * b0[1] - u[1] * b0[0]) * COEFF) };
  COEFF       = (u1[0] * b0[0] + u1[1] * b0[1] + u1[2] * b0[2]);
  real COEFF2 = ONE + (u1[0] * u1[0] + u1[1] * u1[1] + u1[2] * u1[2]) -
                (b0[0] * b0[0] + b0[1] * b0[1] + b0[2] * b0[2]);
  COEFF = ONE / sqrt(INV_2 * (COEFF2 + sqrt(COEFF2 * COEFF2 +
                                            (real)4 * (b0[0] * b0[0] + b0[1] * b0[1] +
                                                       b0[2] * b0[2] + COEFF * COEFF))));
  COEFF2 = ONE / (ONE + (b0[0] * COEFF) * (b0[0] * COEFF) + (b0[1] * COEFF) * (b0[1] * COEFF) +
                  (b0[2] * COEFF) * (b0[2] * COEFF));
  const real dotub = (u1[0] * b0[0] + u1[1] * b0[1] + u1[2] * b0[2]);
  u[0] = COEFF2 * (u1[0] + COEFF * dotub * (b0[0] * COEFF) + u1[1] * b0[2] * COEFF -
                   u1[2] * b0[1] * COEFF);
  u[1] = COEFF2 * (u1[1] + COEFF * dotub * (b0[1] * COEFF) + u1[2] * b0[0] * COEFF -
                   u1[0] * b0[2] * COEFF);
  u[2] = COEFF2 * (u1[2] + COEFF * dotub * (b0[2] * COEFF) + u1[0] * b0[1] * COEFF -
                   u1[1] * b0[0] * COEFF);
}

// ---------------------------------------------------------------------------
// one particle's state in registers
// ---------------------------------------------------------------------------
template <typename real>
struct Prtl {
  int   i[3];
  float dx[3];
  int   ip[3];
  float dxp[3];
  real  u[3];
  short tag;
  int   wrap[3];  // periodic shift applied to i and ip by the boundary step
};

// positionPush (Cartesian) + boundaryConditions: sr.hpp:526-572, 659-814.
// `ip`, `dxp` receive the pre-move cell/offset (wrapped with the particle on a
// periodic crossing, as the reference does to i*_prev).
template <int D, typename real>
__device__ __forceinline__ void move_and_bound(Prtl<real>& q, bool massive, real dt, real dx,
                                               const PushConsts& pc) {
  const real ONE = 1, ZERO = 0;
  const real dt_inv_energy =
    massive ? (dt / sqrt(ONE + q.u[0] * q.u[0] + q.u[1] * q.u[1] + q.u[2] * q.u[2]))
            : (dt / sqrt(q.u[0] * q.u[0] + q.u[1] * q.u[1] + q.u[2] * q.u[2]));
#pragma unroll
  for (int a = 0; a < D; ++a) {
    q.ip[a]   = q.i[a];
    q.wrap[a] = 0;
    q.dxp[a] = q.dx[a];
    q.dx[a] += (q.u[a] / dx) * dt_inv_energy;
    q.i[a] += (int)(q.dx[a] >= ONE) - (int)(q.dx[a] < ZERO);
    q.dx[a] -= (q.dx[a] >= ONE);
    q.dx[a] += (q.dx[a] < ZERO);
  }
#pragma unroll
  for (int a = 0; a < D; ++a) {
    bool invert = false;
    if (q.i[a] < 0) {
      const int bc = pc.bc[a][0];
      if (bc == PIC_BC_PERIODIC) {
        q.i[a] += pc.n[a];
        q.ip[a] += pc.n[a];
        q.wrap[a] = pc.n[a];
      } else if (bc == PIC_BC_ABSORB) {
        q.tag = PIC_TAG_DEAD;
      } else if (bc == PIC_BC_REFLECT) {
        q.i[a]  = 0;
        q.dx[a] = ONE - q.dx[a];
        invert  = true;
      } else if (bc == PIC_BC_AXIS && a == 1) {
        q.i[a]  = 0;
        q.dx[a] = ONE - q.dx[a];
      }
    } else if (q.i[a] >= pc.n[a]) {
      const int bc = pc.bc[a][1];
      if (bc == PIC_BC_PERIODIC) {
        q.i[a] -= pc.n[a];
        q.ip[a] -= pc.n[a];
        q.wrap[a] = -pc.n[a];
      } else if (bc == PIC_BC_ABSORB) {
        q.tag = PIC_TAG_DEAD;
      } else if (bc == PIC_BC_REFLECT) {
        q.i[a]  = pc.n[a] - 1;
        q.dx[a] = ONE - q.dx[a];
        invert  = true;
      } else if (bc == PIC_BC_AXIS && a == 1) {
        q.i[a]  = pc.n[a] - 1;
        q.dx[a] = ONE - q.dx[a];
      }
    }
    if (invert) q.u[a] = -q.u[a];
  }
}

// ---------------------------------------------------------------------------
// current deposit of one particle: src/kernels/currents_deposit.hpp:108-761
// `add(i, j, k, c, v)` accumulates v into J at ghost-inclusive (i, j, k).
// ---------------------------------------------------------------------------
// An accumulator that can fix the box's first node derives from BoxAdd: its
// at(i, j, k) returns one that takes node offsets, so an entry's address is
// the box's plus a constant.
struct BoxAdd {};
template <typename Add>
struct AtBox {
  Add& add;
  int  i0, j0, k0;
  template <typename real>
  __device__ __forceinline__ void operator()(int i, int j, int k, int c, real v) const {
    add(i0 + i, j0 + j, k0 + k, c, v);
  }
};
template <typename Add>
__device__ __forceinline__ auto at_box(Add& add, int i0, int j0, int k0) {
  if constexpr (std::is_base_of_v<BoxAdd, Add>) return add.at(i0, j0, k0);
  else                                          return AtBox<Add>{ add, i0, j0, k0 };
}
// Extent of the Esirkepov box (orders 1-3): any (each entry's add is
// predicated on the particle's own extent), O + 1 nodes per axis (the caller
// has checked support_unmoved), or all O + 2 nodes per axis added without
// predicates (entries outside the particle's extent are exact zeros; the
// accumulator must hold them).
enum Box { BOX_ANY, BOX_UNMOVED, BOX_FULL };
// FACTORED: the entries as products of two factors (below) instead of the
// reference's expressions, equal but for rounding
// Returns false, touching nothing, when the particle's stencil would reach
// outside the ghost-inclusive extents `ext` (possible only for moves longer
// than the ghost layers allow, i.e. a time step beyond the CFL limit);
// ext == nullptr skips the check (the caller guarantees the window).
template <int D, int O, typename real, int BOX = BOX_ANY, bool FACTORED = BOX != BOX_ANY,
          typename Add>
__device__ __forceinline__ bool deposit_with_velocity(const Prtl<real>& q, const real* vp,
                                                      real weight, real charge, real inv_dt,
                                                      int ng, const int* ext, Add&& add);

// Cartesian velocity of the deposit (currents_deposit.hpp:130-165); only the
// unsimulated direction's component enters a 2D deposit
template <int D, typename real>
__device__ __forceinline__ void deposit_velocity(const Prtl<real>& q, real dx, real* vp) {
  const real ONE = 1, ZERO = 0;
  vp[0] = q.u[0] / dx;
  vp[1] = q.u[1] / dx;
  vp[2] = (D == 3) ? q.u[2] / dx : q.u[2];
  const real inv_energy = ONE / sqrt(ONE + (q.u[0] * q.u[0] + q.u[1] * q.u[1] + q.u[2] * q.u[2]));
  if (isnan(vp[2]) || isinf(vp[2])) vp[2] = ZERO;
  vp[0] *= inv_energy;
  vp[1] *= inv_energy;
  vp[2] *= inv_energy;
}

template <int D, int O, typename real, bool FACTORED = false, int BOX = BOX_ANY, typename Add>
__device__ __forceinline__ bool deposit_particle(const Prtl<real>& q, real weight, real charge,
                                                 real inv_dt, real dx, int ng, const int* ext,
                                                 Add&& add) {
  real vp[3];
  deposit_velocity<D, real>(q, dx, vp);
  return deposit_with_velocity<D, O, real, BOX, FACTORED>(q, vp, weight, charge, inv_dt, ng, ext,
                                                          add);
}

// the deposit proper, given the particle velocity vp (the GR deposit passes
// its metric velocity, currents_deposit.hpp:138-159)
template <int D, int O, typename real, int BOX, bool FACTORED, typename Add>
__device__ __forceinline__ bool deposit_with_velocity(const Prtl<real>& q, const real* vp,
                                                      real weight, real charge, real inv_dt,
                                                      int ng, const int* ext, Add&& add) {
  constexpr bool UNMOVED = BOX == BOX_UNMOVED;
  static_assert(BOX == BOX_ANY || O >= 1, "the zigzag deposit has no support box");
  static_assert(FACTORED || BOX == BOX_ANY, "the reference's form takes any extent");
  const real ONE = 1, HALF = 0.5, INV_2 = 0.5;
  if constexpr (O == 0) {
    if (ext) {
#pragma unroll
      for (int a = 0; a < D; ++a) {
        if (min(q.ip[a], q.i[a]) + ng < 0 || max(q.ip[a], q.i[a]) + ng + 1 >= ext[a]) return false;
      }
    }
  }
  const real coeff = weight * charge;

  if constexpr (O == 0) {
    // zigzag (currents_deposit.hpp:167-405)
    real W_1[3], W_2[3], F_1[3], F_2[3];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      const int   ic = q.i[a], ip = q.ip[a];
      const float dxp_r = (float)(ic == ip) * (q.dx[a] + q.dxp[a]) * (float)INV_2;
      W_1[a] = INV_2 * ((real)(dxp_r + q.dxp[a]) + (real)(ic > ip));
      W_2[a] = INV_2 * ((real)(q.dx[a] + dxp_r) + (real)((int)(ic > ip) + ip - ic));
      F_1[a] = ((real)(ic > ip) + (real)dxp_r - (real)q.dxp[a]) * coeff * inv_dt;
      F_2[a] = ((real)(ic - ip - (int)(ic > ip)) + (real)q.dx[a] - (real)dxp_r) * coeff * inv_dt;
    }
    if constexpr (D == 2) {
      const real Fx3_1 = HALF * vp[2] * coeff;
      const real Fx3_2 = HALF * vp[2] * coeff;
      const int  a = q.ip[0] + ng, b = q.ip[1] + ng, c = q.i[0] + ng, d = q.i[1] + ng;
      add(a, b, 0, 0, F_1[0] * (ONE - W_1[1]));
      add(a, b + 1, 0, 0, F_1[0] * W_1[1]);
      add(c, d, 0, 0, F_2[0] * (ONE - W_2[1]));
      add(c, d + 1, 0, 0, F_2[0] * W_2[1]);
      add(a, b, 0, 1, F_1[1] * (ONE - W_1[0]));
      add(a + 1, b, 0, 1, F_1[1] * W_1[0]);
      add(c, d, 0, 1, F_2[1] * (ONE - W_2[0]));
      add(c + 1, d, 0, 1, F_2[1] * W_2[0]);
      add(a, b, 0, 2, Fx3_1 * (ONE - W_1[0]) * (ONE - W_1[1]));
      add(a + 1, b, 0, 2, Fx3_1 * W_1[0] * (ONE - W_1[1]));
      add(a, b + 1, 0, 2, Fx3_1 * (ONE - W_1[0]) * W_1[1]);
      add(a + 1, b + 1, 0, 2, Fx3_1 * W_1[0] * W_1[1]);
      add(c, d, 0, 2, Fx3_2 * (ONE - W_2[0]) * (ONE - W_2[1]));
      add(c + 1, d, 0, 2, Fx3_2 * W_2[0] * (ONE - W_2[1]));
      add(c, d + 1, 0, 2, Fx3_2 * (ONE - W_2[0]) * W_2[1]);
      add(c + 1, d + 1, 0, 2, Fx3_2 * W_2[0] * W_2[1]);
    } else {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int t1 = a == 0 ? 1 : 0;
        const int t2 = a == 2 ? 1 : 2;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int*  o = h == 0 ? q.ip : q.i;
          const real* W = h == 0 ? W_1 : W_2;
          const real  F = h == 0 ? F_1[a] : F_2[a];
#pragma unroll
          for (int s2 = 0; s2 < 2; ++s2) {
#pragma unroll
            for (int s1 = 0; s1 < 2; ++s1) {
              int idx[3] = { o[0] + ng, o[1] + ng, o[2] + ng };
              idx[t1] += s1;
              idx[t2] += s2;
              const real w1 = s1 ? W[t1] : (ONE - W[t1]);
              const real w2 = s2 ? W[t2] : (ONE - W[t2]);
              add(idx[0], idx[1], idx[2], a, F * w1 * w2);
            }
          }
        }
      }
    }
  } else {
    // Esirkepov (currents_deposit.hpp:406-754); jx arrays are formed on the
    // fly as running prefix sums instead of stored tensors
    constexpr int N = O + 2;
    real          iS[D][N], fS[D][N];
    int           imin[3] = { 0, 0, 0 }, imax[3] = { 0, 0, 0 };
#pragma unroll
    for (int a = 0; a < D; ++a) {
      if constexpr (UNMOVED) {
        for_deposit_unmoved<O>(q.ip[a], (real)q.dxp[a], q.i[a], (real)q.dx[a], imin[a], iS[a], fS[a]);
        imax[a] = imin[a] + O;
      } else {
        for_deposit<O>(q.ip[a], (real)q.dxp[a], q.i[a], (real)q.dx[a], imin[a], imax[a], iS[a], fS[a]);
      }
      if (ext && (imin[a] + ng < 0 || imax[a] + ng >= ext[a])) return false;
    }
    constexpr real THIRD = K<real>::THIRD;
    const real     Q     = coeff * inv_dt;
    if constexpr (!FACTORED) {
      // the add of an entry inside the particle's extent
      auto put = [&](bool in, int i, int j, int k, int c, real v) {
        if (in) add(i, j, k, c, v);
      };
      const int  d1 = imax[0] - imin[0], d2 = imax[1] - imin[1];
      const int  i0 = imin[0] + ng, j0 = imin[1] + ng;
      // Every entry of the (O+2)-wide stencil is computed and only the add is
      // predicated on the stencil extent: the loops carry no divergent
      // branches. Each entry's arithmetic is the reference's expression; the
      // factors that do not depend on the innermost index are formed once.
      if constexpr (D == 2) {
        const real QVx3 = coeff * vp[2];
        real hd0[N], hs0[N];  // HALF * (fS - iS), HALF * (fS + iS) along x1
#pragma unroll
        for (int i = 0; i < N; ++i) {
          hd0[i] = HALF * (fS[0][i] - iS[0][i]);
          hs0[i] = HALF * (fS[0][i] + iS[0][i]);
        }
        // jx1: prefix over i (currents_deposit.hpp:496-518, 547-551)
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const real s1 = fS[1][j] + iS[1][j];
          real       acc = 0;
#pragma unroll
          for (int i = 0; i < N - 1; ++i) {
            const real W = hd0[i] * s1;
            acc          = (i == 0) ? (-Q * W) : (acc - Q * W);
            put(i < d1 && j <= d2, i0 + i, j0 + j, 0, 0, acc);
          }
        }
        // jx2: prefix over j
#pragma unroll
        for (int i = 0; i < N; ++i) {
          real acc = 0;
#pragma unroll
          for (int j = 0; j < N - 1; ++j) {
            const real W = hs0[i] * (fS[1][j] - iS[1][j]);
            acc          = (j == 0) ? (-Q * W) : (acc - Q * W);
            put(i <= d1 && j < d2, i0 + i, j0 + j, 0, 1, acc);
          }
        }
        // jx3
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const real ga = HALF * iS[0][i] + fS[0][i];
          const real gb = HALF * fS[0][i] + iS[0][i];
#pragma unroll
          for (int j = 0; j < N; ++j) {
            const real W = THIRD * (fS[1][j] * ga + iS[1][j] * gb);
            put(i <= d1 && j <= d2, i0 + i, j0 + j, 0, 2, QVx3 * W);
          }
        }
      } else {
        const int d3 = imax[2] - imin[2];
        const int k0 = imin[2] + ng;
        real      t0[N], t1[N], t2[N];  // THIRD * (fS - iS) per axis
#pragma unroll
        for (int i = 0; i < N; ++i) {
          t0[i] = THIRD * (fS[0][i] - iS[0][i]);
          t1[i] = THIRD * (fS[1][i] - iS[1][i]);
          t2[i] = THIRD * (fS[2][i] - iS[2][i]);
        }
        // jx1: prefix over i (currents_deposit.hpp:620-700, 716-724)
#pragma unroll
        for (int j = 0; j < N; ++j) {
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const real P = (iS[1][j] * iS[2][k] + fS[1][j] * fS[2][k]) +
                           HALF * (iS[2][k] * fS[1][j] + iS[1][j] * fS[2][k]);
            const bool ok = (j <= d2) && (k <= d3);
            real       acc = 0;
#pragma unroll
            for (int i = 0; i < N - 1; ++i) {
              const real W = t0[i] * P;
              acc          = (i == 0) ? (-Q * W) : (acc - Q * W);
              put(ok && i < d1, i0 + i, j0 + j, k0 + k, 0, acc);
            }
          }
        }
        // jx2: prefix over j
#pragma unroll
        for (int i = 0; i < N; ++i) {
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const real P = iS[0][i] * iS[2][k] + fS[0][i] * fS[2][k] +
                           HALF * (iS[2][k] * fS[0][i] + iS[0][i] * fS[2][k]);
            const bool ok = (i <= d1) && (k <= d3);
            real       acc = 0;
#pragma unroll
            for (int j = 0; j < N - 1; ++j) {
              const real W = t1[j] * P;
              acc          = (j == 0) ? (-Q * W) : (acc - Q * W);
              put(ok && j < d2, i0 + i, j0 + j, k0 + k, 1, acc);
            }
          }
        }
        // jx3: prefix over k
#pragma unroll
        for (int i = 0; i < N; ++i) {
#pragma unroll
          for (int j = 0; j < N; ++j) {
            const real P = iS[0][i] * iS[1][j] + fS[0][i] * fS[1][j] +
                           HALF * (iS[0][i] * fS[1][j] + iS[1][j] * fS[0][i]);
            const bool ok = (i <= d1) && (j <= d2);
            real       acc = 0;
#pragma unroll
            for (int k = 0; k < N - 1; ++k) {
              const real W = t2[k] * P;
              acc          = (k == 0) ? (-Q * W) : (acc - Q * W);
              put(ok && k < d3, i0 + i, j0 + j, k0 + k, 2, acc);
            }
          }
        }
      }
    } else {
      // The reference's products of initial and final shapes, written in the
      // mean m = (iS + fS) / 2 and the half difference h = (fS - iS) / 2:
      //   iS iS' + fS fS' + (iS' fS + iS fS') / 2 = 3 (m m' + h h' / 3),
      // and the prefix sum along the moving axis taken of 2 h once per axis,
      // not of every entry's product: an entry is one product of its axis'
      // prefix and its transverse factor. That is 2 operations per transverse
      // factor and 1 per entry in place of 8 and 3, with fewer roundings on
      // the way to each entry (the factors are positive sums: no cancellation).
      // THIRD keeps the reference's single-precision value.
      constexpr real ONE_THIRD = (real)(1.0 / 3.0);
      int lim[3] = { 0, 0, 0 };
#pragma unroll
      for (int a = 0; a < D; ++a) lim[a] = UNMOVED ? O : imax[a] - imin[a];
      // nodes an axis' loops visit, and whether node i is inside the extent
      constexpr int NN = UNMOVED ? O + 1 : N;
      auto node = [&](int a, int i) { return BOX != BOX_ANY || i <= lim[a]; };
      auto face = [&](int a, int i) { return BOX != BOX_ANY || i < lim[a]; };
      auto&& to = at_box(add, imin[0] + ng, imin[1] + ng, D == 3 ? imin[2] + ng : 0);
      real m[D][NN], h[D][NN];
#pragma unroll
      for (int a = 0; a < D; ++a)
#pragma unroll
        for (int i = 0; i < NN; ++i) {
          m[a][i] = HALF * (fS[a][i] + iS[a][i]);
          h[a][i] = HALF * (fS[a][i] - iS[a][i]);
        }
      // A[i] = c (h[0] + .. + h[i]) along axis a; past the particle's own extent
      // the sum is zero but for rounding, and BOX_FULL makes it so
      auto prefix = [&](int a, real c, real* A) {
        real pre = 0;
#pragma unroll
        for (int i = 0; i < NN - 1; ++i) {
          pre  = i == 0 ? h[a][0] : pre + h[a][i];
          A[i] = c * pre;
        }
        if constexpr (BOX == BOX_FULL) A[NN - 2] = NN - 2 < lim[a] ? A[NN - 2] : (real)0;
      };
      if constexpr (D == 2) {
        real A[NN - 1];
        // jx1: prefix over i (currents_deposit.hpp:496-518, 547-551):
        // -Q (fS - iS) / 2 (fS' + iS') = (-2 Q) h m'
        prefix(0, (real)-2 * Q, A);
#pragma unroll
        for (int i = 0; i < NN - 1; ++i)
#pragma unroll
          for (int j = 0; j < NN; ++j)
            if (face(0, i) && node(1, j)) to(i, j, 0, 0, A[i] * m[1][j]);
        // jx2: prefix over j
        prefix(1, (real)-2 * Q, A);
#pragma unroll
        for (int j = 0; j < NN - 1; ++j)
#pragma unroll
          for (int i = 0; i < NN; ++i)
            if (node(0, i) && face(1, j)) to(i, j, 0, 1, A[j] * m[0][i]);
        // jx3: Q v3 THIRD (fS1 (iS0 / 2 + fS0) + iS1 (fS0 / 2 + iS0))
        const real q3 = (coeff * vp[2]) * ((real)3 * THIRD);
#pragma unroll
        for (int i = 0; i < NN; ++i) {
          const real qm = q3 * m[0][i], qh = (q3 * ONE_THIRD) * h[0][i];
#pragma unroll
          for (int j = 0; j < NN; ++j)
            if (node(0, i) && node(1, j)) to(i, j, 0, 2, fma(qh, h[1][j], qm * m[1][j]));
        }
      } else {
        const real c6 = (real)-6 * THIRD * Q;
        // component a: prefix along axis a, transverse factor of the axes b < c
        // (currents_deposit.hpp:620-754)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
          real      A[NN - 1];
          prefix(a, c6, A);
#pragma unroll
          for (int k = 0; k < NN; ++k) {
            const real hk = ONE_THIRD * h[c][k], mk = m[c][k];
#pragma unroll
            for (int j = 0; j < NN; ++j) {
              const real P  = fma(hk, h[b][j], mk * m[b][j]);
              const bool ok = node(b, j) && node(c, k);
#pragma unroll
              for (int i = 0; i < NN - 1; ++i)
                if (ok && face(a, i))
                  to(a == 0 ? i : j, a == 1 ? i : (a == 0 ? j : k), a == 2 ? i : k, a, A[i] * P);
            }
          }
        }
      }
    }
  }
  return true;
}

// Adds r[0 .. N - 1] (N <= 4) to N consecutive floats from p on with 16-byte
// vector reductions: one, or two where they straddle a 16-byte boundary, zeros
// filling up. The caller vouches for whole 16-byte words around them.
template <int N>
__device__ __forceinline__ void red_row(float* p, const float* r) {
  static_assert(N >= 1 && N <= 4, "at most four floats");
  const int a = (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 3);
  // the row shifted right by a slots
  float u[5] = { 0.f, 0.f, 0.f, 0.f, 0.f }, t[8];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const float even = k < N ? r[k < N ? k : 0] : 0.f, odd = k > 0 && k <= N ? r[k > 0 && k <= N ? k - 1 : 0] : 0.f;
    u[k] = a & 1 ? odd : even;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float lo = k < 5 ? u[k < 5 ? k : 0] : 0.f, hi = k >= 2 && k < 7 ? u[k >= 2 && k < 7 ? k - 2 : 0] : 0.f;
    t[k] = a & 2 ? hi : lo;
  }
  float* q = p - a;
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(q), "f"(t[0]), "f"(t[1]),
               "f"(t[2]), "f"(t[3])
               : "memory");
  if (a + N > 4)
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(q + 4), "f"(t[4]), "f"(t[5]),
                 "f"(t[6]), "f"(t[7])
                 : "memory");
}

// The deposit's reference form (orders 1-3, FP32) by rows along x1:
// row(n, i, j, k, c, r) adds r[0 .. n - 1] to component c at nodes (i .. i + n - 1,
// j, k), ghost-inclusive, entries outside the particle's extent being zero.
// Every entry is deposit_with_velocity's, to the bit. False when the stencil
// leaves the extents.
template <int D, int O, typename Row>
__device__ __forceinline__ bool deposit_rows(const Prtl<float>& q, float vx3, float weight,
                                             float charge, float inv_dt, int ng, const int* ext,
                                             Row&& row) {
  constexpr int N = O + 2;
  const float   HALF = 0.5f, THIRD = K<float>::THIRD;
  float         iS[D][N], fS[D][N];
  int           lo[3] = { 0, 0, 0 }, d[3] = { 0, 0, 0 };
#pragma unroll
  for (int a = 0; a < D; ++a) {
    int hi;
    for_deposit<O>(q.ip[a], q.dxp[a], q.i[a], q.dx[a], lo[a], hi, iS[a], fS[a]);
    if (lo[a] + ng < 0 || hi + ng >= ext[a]) return false;
    d[a] = hi - lo[a];
    lo[a] += ng;
  }
  const float coeff = weight * charge, Q = coeff * inv_dt;
  auto        next  = [&](int n, float acc, float W) { return n == 0 ? -Q * W : acc - Q * W; };
  if constexpr (D == 2) {
    const float QVx3 = coeff * vx3;
    float       hs0[N], acc[N];
#pragma unroll
    for (int i = 0; i < N; ++i) hs0[i] = HALF * (fS[0][i] + iS[0][i]);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float s1 = fS[1][j] + iS[1][j], ds = fS[1][j] - iS[1][j];
      float       r1[N - 1], r2[N], r3[N], a1 = 0;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (i < N - 1) {
          a1    = next(i, a1, (HALF * (fS[0][i] - iS[0][i])) * s1);
          r1[i] = i < d[0] ? a1 : 0.f;
        }
        if (j < N - 1) {
          acc[i] = next(j, acc[i], hs0[i] * ds);
          r2[i]  = i <= d[0] ? acc[i] : 0.f;
        }
        const float ga = HALF * iS[0][i] + fS[0][i], gb = HALF * fS[0][i] + iS[0][i];
        r3[i]          = i <= d[0] ? QVx3 * (THIRD * (fS[1][j] * ga + iS[1][j] * gb)) : 0.f;
      }
      if (j <= d[1]) {
        row(std::integral_constant<int, N - 1>{}, lo[0], lo[1] + j, 0, 0, r1);
        row(std::integral_constant<int, N>{}, lo[0], lo[1] + j, 0, 2, r3);
      }
      if (j < N - 1 && j < d[1]) row(std::integral_constant<int, N>{}, lo[0], lo[1] + j, 0, 1, r2);
    }
  } else {
    float t[3][N];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int i = 0; i < N; ++i) t[a][i] = THIRD * (fS[a][i] - iS[a][i]);
    // jx1
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const float P = (iS[1][j] * iS[2][k] + fS[1][j] * fS[2][k]) +
                        HALF * (iS[2][k] * fS[1][j] + iS[1][j] * fS[2][k]);
        float r[N - 1], acc = 0;
#pragma unroll
        for (int i = 0; i < N - 1; ++i) {
          acc  = next(i, acc, t[0][i] * P);
          r[i] = i < d[0] ? acc : 0.f;
        }
        if (j <= d[1] && k <= d[2])
          row(std::integral_constant<int, N - 1>{}, lo[0], lo[1] + j, lo[2] + k, 0, r);
      }
    // jx2, prefix along x2, and jx3, along x3: a = the moving axis, b the other
#pragma unroll
    for (int a = 1; a < 3; ++a) {
      const int b = 3 - a;
#pragma unroll
      for (int m = 0; m < N; ++m) {  // along b
        float P[N], acc[N];
#pragma unroll
        for (int i = 0; i < N; ++i)
          P[i] = a == 1 ? iS[0][i] * iS[b][m] + fS[0][i] * fS[b][m] +
                            HALF * (iS[b][m] * fS[0][i] + iS[0][i] * fS[b][m])
                        : iS[0][i] * iS[b][m] + fS[0][i] * fS[b][m] +
                            HALF * (iS[0][i] * fS[b][m] + iS[b][m] * fS[0][i]);
#pragma unroll
        for (int l = 0; l < N - 1; ++l) {  // along a
          float r[N];
#pragma unroll
          for (int i = 0; i < N; ++i) {
            acc[i] = next(l, acc[i], t[a][l] * P[i]);
            r[i]   = i <= d[0] ? acc[i] : 0.f;
          }
          if (l < d[a] && m <= d[b])
            row(std::integral_constant<int, N>{}, lo[0], lo[1] + (a == 1 ? l : m),
                lo[2] + (a == 1 ? m : l), a, r);
        }
      }
    }
  }
  return true;
}

// true when the cell of every simulated axis lies in [0, n)
template <int D>
__device__ __forceinline__ bool cells_in_grid(const int* i, const int* n) {
  bool ok = true;
#pragma unroll
  for (int a = 0; a < D; ++a) ok = ok && (i[a] >= 0) && (i[a] < n[a]);
  return ok;
}

}  // namespace pic
