// Field kernels of the SR step on a Cartesian (Minkowski) grid: Faraday and
// Ampere Yee updates, the J -> E coupling, the periodic current fold, the
// digital current filter and ghost exchange, and the FP64 energy reduction.
//
// The update kernels map one thread to one active cell (i1 fastest; the fold and
// the ghost fill visit the cells near periodic edges only) and, where the
// reference follows the update with a periodic CommunicateFields, write the
// cell's new value straight into its ghost images as well, which removes the
// reference's separate halo pass (src/framework/domain/comm_nompi.hpp:44-63).
#include <algorithm>

#include <cuda_runtime.h>

#include "fields.cuh"
#include "pic_common.cuh"

namespace pic {

namespace {

struct CellIter {
  int     n[3];
  int     ng;
  int     dim;
  int64_t count;
  __device__ __forceinline__ void cell(int64_t t, int& i, int& j, int& k) const {
    i = (int)(t % n[0]);
    t /= n[0];
    j = (int)(t % n[1]);
    k = (int)(t / n[1]);
    i += ng;
    j += ng;
    k = (dim == 3) ? k + ng : 0;
  }
};

// the active cells within ng of an edge of a periodic axis, each once: whole
// planes along x3, then rows along x2 of the other planes, then cells along x1
struct EdgeIter {
  int      n[3], e[3];  // cells, and edge cells (both ends) per axis
  int      ng, dim;
  unsigned c3, c2, count;
  // the k-th edge cell of axis d: the lower ones, then the upper ones
  __device__ __forceinline__ int edge(int d, int k) const { return k < ng ? k : n[d] - 2 * ng + k; }
  // the k-th cell of axis d that is not an edge cell
  __device__ __forceinline__ int inner(int d, int k) const { return e[d] ? ng + k : k; }
  __device__ __forceinline__ void cell(unsigned t, int& i, int& j, int& k) const {
    if (t < c3) {
      const unsigned r = t / (unsigned)n[0];
      i = (int)(t - r * n[0]);
      j = (int)(r % (unsigned)n[1]);
      k = edge(2, (int)(r / (unsigned)n[1]));
    } else if (t < c3 + c2) {
      t -= c3;
      const unsigned r = t / (unsigned)n[0];
      i = (int)(t - r * n[0]);
      j = edge(1, (int)(r % (unsigned)e[1]));
      k = inner(2, (int)(r / (unsigned)e[1]));
    } else {
      t -= c3 + c2;
      const unsigned m1 = (unsigned)(n[1] - e[1]), r = t / (unsigned)e[0];
      i = edge(0, (int)(t - r * e[0]));
      j = inner(1, (int)(r % m1));
      k = inner(2, (int)(r / m1));
    }
    i += ng;
    j += ng;
    k = (dim == 3) ? k + ng : 0;
  }
};

// visits every ghost image of active cell (i, j, k) across periodic
// dimensions (images: i + n when i < 2 ng, i - n when i >= n)
template <int D, typename F>
__device__ __forceinline__ void for_images(const GridInfo& g, int i, int j, int k, F&& f) {
  int sh[3][2];
  int ns[3];
  const int c[3] = { i, j, k };
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    ns[d]    = 1;
    sh[d][0] = 0;
    if (d < D && g.periodic[d]) {
      if (c[d] < 2 * g.ng) sh[d][ns[d]++] = g.n[d];
      else if (c[d] >= g.n[d]) sh[d][ns[d]++] = -g.n[d];
    }
  }
  for (int a = 0; a < ns[0]; ++a)
    for (int b = 0; b < ns[1]; ++b)
      for (int e = 0; e < ns[2]; ++e) {
        if (a == 0 && b == 0 && e == 0) continue;
        f(i + sh[0][a], j + sh[1][b], k + sh[2][e]);
      }
}

CellIter make_iter(const GridInfo& g) {
  CellIter it;
  it.n[0]  = g.n[0];
  it.n[1]  = g.n[1];
  it.n[2]  = g.dim == 3 ? g.n[2] : 1;
  it.ng    = g.ng;
  it.dim   = g.dim;
  it.count = (int64_t)it.n[0] * it.n[1] * it.n[2];
  return it;
}

EdgeIter make_edges(const GridInfo& g) {
  EdgeIter it;
  it.ng  = g.ng;
  it.dim = g.dim;
  for (int d = 0; d < 3; ++d) {
    it.n[d] = d < g.dim ? g.n[d] : 1;
    it.e[d] = d < g.dim && g.periodic[d] ? 2 * g.ng : 0;  // a grid has at least that many cells
  }
  it.c3    = (unsigned)it.e[2] * it.n[0] * it.n[1];
  it.c2    = (unsigned)(it.n[2] - it.e[2]) * it.e[1] * it.n[0];
  it.count = it.c3 + it.c2 + (unsigned)(it.n[2] - it.e[2]) * (it.n[1] - it.e[1]) * it.e[0];
  return it;
}

dim3 grid_for(int64_t count, int threads) {
  int64_t b = (count + threads - 1) / threads;
  if (b > pic::sm_count() * 128) b = pic::sm_count() * 128;
  if (b < 1) b = 1;
  return dim3((unsigned)b);
}

// ---------------------------------------------------------------------------
// Faraday: src/kernels/faraday_mink.hpp:71-166 (+ CommunicateFields(B))
// ---------------------------------------------------------------------------
template <int D, typename real, bool YEE>
__global__ void k_faraday(GridInfo g, CellIter it, FieldView<real> EB, real coeff1, real coeff2,
                          Stencil<real> st) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i1, i2, i3;
    it.cell(t, i1, i2, i3);
#define F(a, b, c, comp) EB.p[EB.idx(a, b, c, comp)]
    real nb[3];
    if constexpr (D == 2) {
      const real alphax = (real)1 - (real)2 * st.betaxy - (real)3 * st.deltax;
      const real alphay = (real)1 - (real)2 * st.betayx - (real)3 * st.deltay;
      if constexpr (YEE) {
        nb[0] = F(i1, i2, 0, 3) + coeff1 * (-alphay * (F(i1, i2 + 1, 0, 2) - F(i1, i2, 0, 2)));
        nb[1] = F(i1, i2, 0, 4) + coeff1 * (+alphax * (F(i1 + 1, i2, 0, 2) - F(i1, i2, 0, 2)));
        nb[2] = F(i1, i2, 0, 5) + coeff2 * (+alphay * (F(i1, i2 + 1, 0, 0) - F(i1, i2, 0, 0)) -
                                            alphax * (F(i1 + 1, i2, 0, 1) - F(i1, i2, 0, 1)));
      } else {
        nb[0] = F(i1, i2, 0, 3) +
                coeff1 * (-alphay * (F(i1, i2 + 1, 0, 2) - F(i1, i2, 0, 2)) -
                          st.deltay * (F(i1, i2 + 2, 0, 2) - F(i1, i2 - 1, 0, 2)) -
                          st.betayx * (F(i1 + 1, i2 + 1, 0, 2) - F(i1 + 1, i2, 0, 2)) -
                          st.betayx * (F(i1 - 1, i2 + 1, 0, 2) - F(i1 - 1, i2, 0, 2)));
        nb[1] = F(i1, i2, 0, 4) +
                coeff1 * (+alphax * (F(i1 + 1, i2, 0, 2) - F(i1, i2, 0, 2)) +
                          st.deltax * (F(i1 + 2, i2, 0, 2) - F(i1 - 1, i2, 0, 2)) +
                          st.betaxy * (F(i1 + 1, i2 + 1, 0, 2) - F(i1, i2 + 1, 0, 2)) +
                          st.betaxy * (F(i1 + 1, i2 - 1, 0, 2) - F(i1, i2 - 1, 0, 2)));
        nb[2] = F(i1, i2, 0, 5) +
                coeff2 * (+alphay * (F(i1, i2 + 1, 0, 0) - F(i1, i2, 0, 0)) +
                          st.deltay * (F(i1, i2 + 2, 0, 0) - F(i1, i2 - 1, 0, 0)) +
                          st.betayx * (F(i1 + 1, i2 + 1, 0, 0) - F(i1 + 1, i2, 0, 0)) +
                          st.betayx * (F(i1 - 1, i2 + 1, 0, 0) - F(i1 - 1, i2, 0, 0)) -
                          alphax * (F(i1 + 1, i2, 0, 1) - F(i1, i2, 0, 1)) -
                          st.deltax * (F(i1 + 2, i2, 0, 1) - F(i1 - 1, i2, 0, 1)) -
                          st.betaxy * (F(i1 + 1, i2 + 1, 0, 1) - F(i1, i2 + 1, 0, 1)) -
                          st.betaxy * (F(i1 + 1, i2 - 1, 0, 1) - F(i1, i2 - 1, 0, 1)));
      }
    } else {
      const real alphax = (real)1 - (real)2 * st.betaxy - (real)2 * st.betaxz - (real)3 * st.deltax;
      const real alphay = (real)1 - (real)2 * st.betayx - (real)2 * st.betayz - (real)3 * st.deltay;
      const real alphaz = (real)1 - (real)2 * st.betazx - (real)2 * st.betazy - (real)3 * st.deltaz;
      if constexpr (YEE) {
        nb[0] = F(i1, i2, i3, 3) +
                coeff1 * (+alphaz * (F(i1, i2, i3 + 1, 1) - F(i1, i2, i3, 1)) -
                          alphay * (F(i1, i2 + 1, i3, 2) - F(i1, i2, i3, 2)));
        nb[1] = F(i1, i2, i3, 4) +
                coeff1 * (+alphax * (F(i1 + 1, i2, i3, 2) - F(i1, i2, i3, 2)) -
                          alphaz * (F(i1, i2, i3 + 1, 0) - F(i1, i2, i3, 0)));
        nb[2] = F(i1, i2, i3, 5) +
                coeff1 * (+alphay * (F(i1, i2 + 1, i3, 0) - F(i1, i2, i3, 0)) -
                          alphax * (F(i1 + 1, i2, i3, 1) - F(i1, i2, i3, 1)));
      } else {
        nb[0] = F(i1, i2, i3, 3) +
                coeff1 * (+alphaz * (F(i1, i2, i3 + 1, 1) - F(i1, i2, i3, 1)) +
                          st.deltaz * (F(i1, i2, i3 + 2, 1) - F(i1, i2, i3 - 1, 1)) +
                          st.betazx * (F(i1 + 1, i2, i3 + 1, 1) - F(i1 + 1, i2, i3, 1)) +
                          st.betazx * (F(i1 - 1, i2, i3 + 1, 1) - F(i1 - 1, i2, i3, 1)) +
                          st.betazy * (F(i1, i2 + 1, i3 + 1, 1) - F(i1, i2 + 1, i3, 1)) +
                          st.betazy * (F(i1, i2 - 1, i3 + 1, 1) - F(i1, i2 - 1, i3, 1)) -
                          alphay * (F(i1, i2 + 1, i3, 2) - F(i1, i2, i3, 2)) -
                          st.deltay * (F(i1, i2 + 2, i3, 2) - F(i1, i2 - 1, i3, 2)) -
                          st.betayx * (F(i1 + 1, i2 + 1, i3, 2) - F(i1 + 1, i2, i3, 2)) -
                          st.betayx * (F(i1 - 1, i2 + 1, i3, 2) - F(i1 - 1, i2, i3, 2)) -
                          st.betayz * (F(i1, i2 + 1, i3 + 1, 2) - F(i1, i2, i3 + 1, 2)) -
                          st.betayz * (F(i1, i2 + 1, i3 - 1, 2) - F(i1, i2, i3 - 1, 2)));
        nb[1] = F(i1, i2, i3, 4) +
                coeff1 * (+alphax * (F(i1 + 1, i2, i3, 2) - F(i1, i2, i3, 2)) +
                          st.deltax * (F(i1 + 2, i2, i3, 2) - F(i1 - 1, i2, i3, 2)) +
                          st.betaxy * (F(i1 + 1, i2 + 1, i3, 2) - F(i1, i2 + 1, i3, 2)) +
                          st.betaxy * (F(i1 + 1, i2 - 1, i3, 2) - F(i1, i2 - 1, i3, 2)) +
                          st.betaxz * (F(i1 + 1, i2, i3 + 1, 2) - F(i1, i2, i3 + 1, 2)) +
                          st.betaxz * (F(i1 + 1, i2, i3 - 1, 2) - F(i1, i2, i3 - 1, 2)) -
                          alphaz * (F(i1, i2, i3 + 1, 0) - F(i1, i2, i3, 0)) -
                          st.deltaz * (F(i1, i2, i3 + 2, 0) - F(i1, i2, i3 - 1, 0)) -
                          st.betazx * (F(i1 + 1, i2, i3 + 1, 0) - F(i1 + 1, i2, i3, 0)) -
                          st.betazx * (F(i1 - 1, i2, i3 + 1, 0) - F(i1 - 1, i2, i3, 0)) -
                          st.betazy * (F(i1, i2 + 1, i3 + 1, 0) - F(i1, i2 + 1, i3, 0)) -
                          st.betazy * (F(i1, i2 - 1, i3 + 1, 0) - F(i1, i2 - 1, i3, 0)));
        nb[2] = F(i1, i2, i3, 5) +
                coeff1 * (+alphay * (F(i1, i2 + 1, i3, 0) - F(i1, i2, i3, 0)) +
                          st.deltay * (F(i1, i2 + 2, i3, 0) - F(i1, i2 - 1, i3, 0)) +
                          st.betayx * (F(i1 + 1, i2 + 1, i3, 0) - F(i1 + 1, i2, i3, 0)) +
                          st.betayx * (F(i1 - 1, i2 + 1, i3, 0) - F(i1 - 1, i2, i3, 0)) +
                          st.betayz * (F(i1, i2 + 1, i3 + 1, 0) - F(i1, i2, i3 + 1, 0)) +
                          st.betayz * (F(i1, i2 + 1, i3 - 1, 0) - F(i1, i2, i3 - 1, 0)) -
                          alphax * (F(i1 + 1, i2, i3, 1) - F(i1, i2, i3, 1)) -
                          st.deltax * (F(i1 + 2, i2, i3, 1) - F(i1 - 1, i2, i3, 1)) -
                          st.betaxy * (F(i1 + 1, i2 + 1, i3, 1) - F(i1, i2 + 1, i3, 1)) -
                          st.betaxy * (F(i1 + 1, i2 - 1, i3, 1) - F(i1, i2 - 1, i3, 1)) -
                          st.betaxz * (F(i1 + 1, i2, i3 + 1, 1) - F(i1, i2, i3 + 1, 1)) -
                          st.betaxz * (F(i1 + 1, i2, i3 - 1, 1) - F(i1, i2, i3 - 1, 1)));
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) F(i1, i2, i3, 3 + c) = nb[c];
    for_images<D>(g, i1, i2, i3, [&](int a, int b, int e) {
#pragma unroll
      for (int c = 0; c < 3; ++c) F(a, b, e, 3 + c) = nb[c];
    });
#undef F
  }
}

// ---------------------------------------------------------------------------
// Ampere (ampere_mink.hpp:48-88) + CurrentsAmpere (ampere_mink.hpp:134-214)
// + CommunicateFields(E | J)
// ---------------------------------------------------------------------------
template <int D, typename real, bool CURL, bool CUR, bool FILL>
__global__ void k_ampere(GridInfo g, CellIter it, FieldView<real> EB, FieldView<real> J,
                         real coeff1, real coeff2, real jcoeff, real ppc0) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i1, i2, i3;
    it.cell(t, i1, i2, i3);
#define F(a, b, c, comp) EB.p[EB.idx(a, b, c, comp)]
    real ne[3] = { F(i1, i2, i3, 0), F(i1, i2, i3, 1), F(i1, i2, i3, 2) };
    if constexpr (CURL) {
      if constexpr (D == 2) {
        ne[0] += coeff1 * (F(i1, i2, 0, 5) - F(i1, i2 - 1, 0, 5));
        ne[1] += coeff1 * (F(i1 - 1, i2, 0, 5) - F(i1, i2, 0, 5));
        ne[2] += coeff2 * (F(i1, i2 - 1, 0, 3) - F(i1, i2, 0, 3) + F(i1, i2, 0, 4) -
                           F(i1 - 1, i2, 0, 4));
      } else {
        ne[0] += coeff1 * (F(i1, i2, i3 - 1, 4) - F(i1, i2, i3, 4) + F(i1, i2, i3, 5) -
                           F(i1, i2 - 1, i3, 5));
        ne[1] += coeff1 * (F(i1 - 1, i2, i3, 5) - F(i1, i2, i3, 5) + F(i1, i2, i3, 3) -
                           F(i1, i2, i3 - 1, 3));
        ne[2] += coeff1 * (F(i1, i2 - 1, i3, 3) - F(i1, i2, i3, 3) + F(i1, i2, i3, 4) -
                           F(i1 - 1, i2, i3, 4));
      }
    }
    real nj[3];
    if constexpr (CUR) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const real jv = J.p[J.idx(i1, i2, i3, c)];
        ne[c] += jv * jcoeff;
        nj[c] = jv / ppc0;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) F(i1, i2, i3, c) = ne[c];
    if constexpr (CUR) {
#pragma unroll
      for (int c = 0; c < 3; ++c) J.p[J.idx(i1, i2, i3, c)] = nj[c];
    }
    if constexpr (FILL) {
      for_images<D>(g, i1, i2, i3, [&](int a, int b, int e) {
#pragma unroll
        for (int c = 0; c < 3; ++c) F(a, b, e, c) = ne[c];
        if constexpr (CUR) {
#pragma unroll
          for (int c = 0; c < 3; ++c) J.p[J.idx(a, b, e, c)] = nj[c];
        }
      });
    }
#undef F
  }
}

// ---------------------------------------------------------------------------
// periodic current fold + ghost fill: SynchronizeFields(J) followed by
// CommunicateFields(J) (metadomain_comm.cpp:408-562, 204-367). The sum runs
// over the images in dir::Directions<D>::all order and is added to the
// active value last, as AddBufferedFields does.
// ---------------------------------------------------------------------------
template <int D, typename real>
__global__ void k_sync_currents(GridInfo g, EdgeIter it, FieldView<real> J) {
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i1, i2, i3;
    it.cell(t, i1, i2, i3);
    const int c[3] = { i1, i2, i3 };
    real      buf[3] = { 0, 0, 0 };
    // directions v in lexicographic order over {-1,0,1}^D \ {0}; the source
    // of v is c + n*v, valid when v_d = +1 -> c_d < 2ng, v_d = -1 -> c_d >= n
    for (int a = -1; a <= 1; ++a)
      for (int b = -1; b <= 1; ++b)
        for (int e = (D == 3 ? -1 : 0); e <= (D == 3 ? 1 : 0); ++e) {
          if (a == 0 && b == 0 && e == 0) continue;
          const int v[3] = { a, b, e };
          int       src[3];
          bool      ok = true;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            src[d] = c[d];
            if (v[d] == 0) continue;
            if (d >= D || !g.periodic[d]) {
              ok = false;
            } else if (v[d] == 1) {
              ok = ok && (c[d] < 2 * g.ng);
              src[d] = c[d] + g.n[d];
            } else {
              ok = ok && (c[d] >= g.n[d]);
              src[d] = c[d] - g.n[d];
            }
          }
          if (!ok) continue;
#pragma unroll
          for (int cc = 0; cc < 3; ++cc) buf[cc] += J.p[J.idx(src[0], src[1], src[2], cc)];
        }
    real nv[3];
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) {
      nv[cc]                          = J.p[J.idx(i1, i2, i3, cc)] + buf[cc];
      J.p[J.idx(i1, i2, i3, cc)] = nv[cc];
    }
    for_images<D>(g, i1, i2, i3, [&](int a, int b, int e) {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) J.p[J.idx(a, b, e, cc)] = nv[cc];
    });
  }
}

// plain ghost fill of components [c0, c1): images of cells near the edges. A
// thread per cell and component: with the components in a loop, each one's load
// waited for the stores before it (256^2, six
// components: 4.2 us, 2.4 us so; the adjoint fold below 14.9 and 5.5 us).
template <int D, typename real>
__global__ void k_fill_ghosts(GridInfo g, EdgeIter it, FieldView<real> f, int c0, int c1) {
  const unsigned stride = gridDim.x * blockDim.x;
  for (int c = c0 + blockIdx.y; c < c1; c += gridDim.y)
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < it.count; t += stride) {
      int i1, i2, i3;
      it.cell(t, i1, i2, i3);
      const real v = f.p[f.idx(i1, i2, i3, c)];
      for_images<D>(g, i1, i2, i3, [&](int a, int b, int e) { f.p[f.idx(a, b, e, c)] = v; });
    }
}

// ---------------------------------------------------------------------------
// digital filter pass in 2D: digital_filter.hpp:183-195; reads
// src, writes dst at the active cells and their periodic ghost images
// ---------------------------------------------------------------------------
template <typename real>
__global__ void k_filter2(GridInfo g, CellIter it, FieldView<real> src, FieldView<real> dst) {
  const real    INV_4 = 0.25, INV_8 = 0.125, INV_16 = 0.0625;
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i1, i2, i3;
    it.cell(t, i1, i2, i3);
    real nv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#define b(x, y, z) src.p[src.idx(x, y, z, c)]
      nv[c] = INV_4 * b(i1, i2, 0) +
              INV_8 * (b(i1 - 1, i2, 0) + b(i1 + 1, i2, 0) + b(i1, i2 - 1, 0) + b(i1, i2 + 1, 0)) +
              INV_16 * (b(i1 - 1, i2 - 1, 0) + b(i1 + 1, i2 + 1, 0) + b(i1 - 1, i2 + 1, 0) +
                        b(i1 + 1, i2 - 1, 0));
#undef b
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) dst.p[dst.idx(i1, i2, i3, c)] = nv[c];
    for_images<2>(g, i1, i2, i3, [&](int a, int bb, int e) {
#pragma unroll
      for (int c = 0; c < 3; ++c) dst.p[dst.idx(a, bb, e, c)] = nv[c];
    });
  }
}

// one component's 27-point sum, the terms in the reference's order
// (digital_filter.hpp:352-379; the (i, j, k +- 1) pair appears twice in the 1/32
// group, as in :365); b[z][y][x] is the cell's neighbourhood
template <typename T>
__device__ __forceinline__ T filter_sum(const T (*b)[3][3], T i8, T i16, T i32, T i64) {
#define B(x, y, z) b[(z) + 1][(y) + 1][(x) + 1]
  return i8 * B(0, 0, 0) +
         i16 * (B(-1, 0, 0) + B(1, 0, 0) + B(0, -1, 0) + B(0, 1, 0) + B(0, 0, -1) + B(0, 0, 1)) +
         i32 * (B(-1, -1, 0) + B(1, 1, 0) + B(-1, 1, 0) + B(1, -1, 0) + B(0, -1, -1) + B(0, 1, 1) +
                B(0, 0, -1) + B(0, 0, 1) + B(-1, 0, -1) + B(1, 0, 1) + B(-1, 0, 1) + B(1, 0, -1)) +
         i64 * (B(-1, -1, -1) + B(1, 1, 1) + B(-1, 1, 1) + B(1, -1, -1) + B(-1, -1, 1) +
                B(1, 1, -1) + B(-1, 1, -1) + B(1, -1, 1));
#undef B
}

// The 3D pass in FP32: a block of 32 x 8 threads marches along x3 over zlen cells, with
// the plane ahead staged in shared memory (double-buffered, one-cell halo) and
// each thread's last three 3 x 3 neighbourhoods of each component in
// registers: a cell reads 9 new values per component, not 27. The first
// two components are summed as one packed operation. The terms and their order
// are the reference's: the same bits. 256^3: 307 us a pass with every cell
// reading its 27 values from a staged block (665 instructions per cell), 220 us;
// 100 x 75 x 61 18.6 and 14.5 us.
constexpr int kFltX = 32, kFltY = 8;
__global__ void __launch_bounds__(256) k_filter3_march(GridInfo g, FieldView<float> src,
                                                       FieldView<float> dst, int zlen) {
  using real = float;
  constexpr int SX = kFltX + 2, SY = kFltY + 2, PLANE = SX * SY, NS = 3 * PLANE,
                TRIPS = (NS + 255) / 256;
  __shared__ real sm[2][NS];
  const int ng = g.ng;
  // first active cell of the block, ghost-inclusive
  const int x0 = ng + blockIdx.x * kFltX, y0 = ng + blockIdx.y * kFltY, z0 = ng + blockIdx.z * zlen;
  const int ex = g.n[0] + 2 * ng, ey = g.n[1] + 2 * ng;
  const int z1 = min(z0 + zlen, g.n[2] + ng);  // past the block's last cell
  const int tx = threadIdx.x % kFltX, ty = threadIdx.x / kFltX;
  // where this thread's staged elements lie in a plane (cells past the array
  // belong to no active cell of this block)
  const real* from[TRIPS];
#pragma unroll
  for (int k = 0; k < TRIPS; ++k) {
    const int t = threadIdx.x + k * 256, c = t / PLANE, y = (t % PLANE) / SX;
    const int gx = x0 - 1 + (t % PLANE) % SX, gy = y0 - 1 + y;
    from[k] = t < NS && gx < ex && gy < ey ? src.p + src.idx(gx, gy, 0, c) : nullptr;
  }
  real v[TRIPS];
  auto fetch = [&](int z) {
#pragma unroll
    for (int k = 0; k < TRIPS; ++k) v[k] = from[k] ? __ldg(from[k] + (int64_t)z * src.s2) : (real)0;
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int k = 0; k < TRIPS; ++k) {
      const int t = threadIdx.x + k * 256;
      if (t < NS) sm[buf][t] = v[k];
    }
  };
  const real  INV_8 = 0.125, INV_16 = 0.0625, INV_32 = 0.03125, INV_64 = 0.015625;
  const int   i1 = x0 + tx, i2 = y0 + ty;
  const bool  mine = i1 < g.n[0] + ng && i2 < g.n[1] + ng;
  F2   bp[3][3][3];  // components 0 and 1
  real b2[3][3][3];
  auto take = [&](int buf, int z) {  // plane z of the neighbourhoods from a buffer
#pragma unroll
    for (int y = 0; y < 3; ++y)
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const real* q = &sm[buf][(ty + y) * SX + tx + x];
        bp[z][y][x]   = f2(q[0], q[PLANE]);
        b2[z][y][x]   = q[2 * PLANE];
      }
  };
  auto shift = [&]() {
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
      for (int y = 0; y < 3; ++y)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          bp[z][y][x] = bp[z + 1][y][x];
          b2[z][y][x] = b2[z + 1][y][x];
        }
  };
  fetch(z0 - 1);
  put(0);
  fetch(z0);
  __syncthreads();
  take(0, 1);
  put(1);
  fetch(z0 + 1);
  __syncthreads();
  take(1, 2);
  for (int i3 = z0, buf = 0; i3 < z1; ++i3, buf ^= 1) {
    // (the buffer's last readers passed the previous barrier)
    put(buf);
    if (i3 + 2 <= z1) fetch(i3 + 2);
    __syncthreads();
    shift();
    take(buf, 2);
    if (mine) {
      real     nv[3];
      const F2 r = filter_sum(bp, f2(INV_8, INV_8), f2(INV_16, INV_16), f2(INV_32, INV_32),
                              f2(INV_64, INV_64));
      unpack(r, nv[0], nv[1]);
      nv[2] = filter_sum(b2, INV_8, INV_16, INV_32, INV_64);
#pragma unroll
      for (int c = 0; c < 3; ++c) dst.p[dst.idx(i1, i2, i3, c)] = nv[c];
      for_images<3>(g, i1, i2, i3, [&](int a, int bb, int e) {
#pragma unroll
        for (int c = 0; c < 3; ++c) dst.p[dst.idx(a, bb, e, c)] = nv[c];
      });
    }
  }
}

// The 3D pass in FP64: a block holds 32 x 8 cells of one plane and a one-cell halo of
// the three components in shared memory, and each cell's sum reads its 27 values there.
// The sums are bound by the FP64 pipe, two lanes per SM and clock, and want many warps:
// marching with the neighbourhoods in registers took 65.6 us a pass at 64^3, 473 at
// 128^3 and 1432 at 192^3, blocks of four planes 59.6, 381 and 1231, of one plane
// 53.3, 367 and 1220 (24^3: 12.4, 34.9 and 12.4).
__global__ void __launch_bounds__(256) k_filter3_staged(GridInfo g, FieldView<double> src,
                                                        FieldView<double> dst) {
  constexpr int SX = kFltX + 2, SY = kFltY + 2, SZ = 3, NS = 3 * SZ * SY * SX,
                TRIPS = (NS + 255) / 256;
  __shared__ double sm[3][SZ][SY][SX];
  const int ng = g.ng;
  // first active cell of the block, ghost-inclusive (a plane per block can be more
  // planes than a grid's y and z hold)
  const int bx = (g.n[0] + kFltX - 1) / kFltX, by = (g.n[1] + kFltY - 1) / kFltY;
  const int x0 = ng + (int)(blockIdx.x % bx) * kFltX, y0 = ng + (int)(blockIdx.x / bx % by) * kFltY,
            i3 = ng + (int)(blockIdx.x / bx / by);
  const int ex = g.n[0] + 2 * ng, ey = g.n[1] + 2 * ng;
  // a fixed trip count, unrolled: every thread's loads are in flight together
  double v[TRIPS];
#pragma unroll
  for (int k = 0; k < TRIPS; ++k) {
    const int t = threadIdx.x + k * 256;
    const int x = t % SX, y = (t / SX) % SY, z = (t / (SX * SY)) % SZ, c = t / (SX * SY * SZ);
    const int gx = x0 - 1 + x, gy = y0 - 1 + y, gz = i3 - 1 + z;
    // cells past the array belong to no active cell of this block
    v[k] = t < NS && gx < ex && gy < ey ? src.p[src.idx(gx, gy, gz, c)] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < TRIPS; ++k) {
    const int t = threadIdx.x + k * 256;
    if (t < NS) (&sm[0][0][0][0])[t] = v[k];
  }
  __syncthreads();
  const int tx = threadIdx.x % kFltX, ty = threadIdx.x / kFltX;
  const int i1 = x0 + tx, i2 = y0 + ty;
  if (i1 >= g.n[0] + ng || i2 >= g.n[1] + ng) return;
  double nv[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double b[3][3][3];
#pragma unroll
    for (int q = 0; q < 27; ++q) b[q / 9][q / 3 % 3][q % 3] = sm[c][q / 9][ty + q / 3 % 3][tx + q % 3];
    nv[c] = filter_sum(b, 0.125, 0.0625, 0.03125, 0.015625);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) dst.p[dst.idx(i1, i2, i3, c)] = nv[c];
  for_images<3>(g, i1, i2, i3, [&](int a, int bb, int e) {
#pragma unroll
    for (int c = 0; c < 3; ++c) dst.p[dst.idx(a, bb, e, c)] = nv[c];
  });
}

void filter3(const GridInfo& g, FieldView<float> a, FieldView<float> b, cudaStream_t s) {
  // x3 cells per block: as many as leave four blocks per SM, 4 to 16 (a block
  // stages two planes more than it has cells; 100 x 75 x 61: 14.5 us, 23.0 with 16)
  const int     bx = (g.n[0] + kFltX - 1) / kFltX, by = (g.n[1] + kFltY - 1) / kFltY;
  const int64_t fit  = (int64_t)bx * by * g.n[2] / (4 * pic::sm_count());
  const int     zlen = (int)std::min<int64_t>(16, std::max<int64_t>(4, fit));
  PIC_KL(k_filter3_march<<<dim3(bx, by, (g.n[2] + zlen - 1) / zlen), 256, 0, s>>>(g, a, b, zlen));
}
void filter3(const GridInfo& g, FieldView<double> a, FieldView<double> b, cudaStream_t s) {
  const unsigned blocks = (unsigned)((g.n[0] + kFltX - 1) / kFltX) * ((g.n[1] + kFltY - 1) / kFltY) * g.n[2];
  PIC_KL(k_filter3_staged<<<blocks, 256, 0, s>>>(g, a, b));
}

// copy all cells (ghost-inclusive) of a 3-component field
template <typename real>
__global__ void k_copy3(GridInfo g, FieldView<real> src, FieldView<real> dst) {
  const int     e0 = g.n[0] + 2 * g.ng, e1 = g.n[1] + 2 * g.ng;
  const int     e2 = g.dim == 3 ? g.n[2] + 2 * g.ng : 1;
  const int64_t count  = (int64_t)e0 * e1 * e2 * 3;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += stride) {
    int64_t r = t;
    const int i = (int)(r % e0);
    r /= e0;
    const int j = (int)(r % e1);
    r /= e1;
    const int k = (int)(r % e2);
    const int c = (int)(r / e2);
    dst.p[dst.idx(i, j, k, c)] = src.p[src.idx(i, j, k, c)];
  }
}

// zero all cells of a 3-component field
template <typename real>
__global__ void k_zero3(GridInfo g, FieldView<real> f) {
  const int     e0 = g.n[0] + 2 * g.ng, e1 = g.n[1] + 2 * g.ng;
  const int     e2 = g.dim == 3 ? g.n[2] + 2 * g.ng : 1;
  const int64_t count  = (int64_t)e0 * e1 * e2 * 3;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += stride) {
    int64_t r = t;
    const int i = (int)(r % e0);
    r /= e0;
    const int j = (int)(r % e1);
    r /= e1;
    const int k = (int)(r % e2);
    const int c = (int)(r / e2);
    f.p[f.idx(i, j, k, c)] = (real)0;
  }
}

// FP64 field energy (reduced_stats.hpp:145-187, Minkowski weights)
template <int D, typename real>
__global__ void k_energy(CellIter it, FieldView<real> EB, double dx, double* out) {
  __shared__ double sh[2][32];
  const double  dV     = D == 3 ? dx * dx * dx : dx * dx;
  double        e2 = 0, b2 = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i1, i2, i3;
    it.cell(t, i1, i2, i3);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double h  = (c < D) ? dx * dx : 1.0;
      const double ev = (double)EB.p[EB.idx(i1, i2, i3, c)];
      const double bv = (double)EB.p[EB.idx(i1, i2, i3, c + 3)];
      e2 += ev * ev * h * dV;
      b2 += bv * bv * h * dV;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    e2 += __shfl_down_sync(0xffffffffu, e2, o);
    b2 += __shfl_down_sync(0xffffffffu, b2, o);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sh[0][wid] = e2;
    sh[1][wid] = b2;
  }
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    e2 = lane < nw ? sh[0][lane] : 0.0;
    b2 = lane < nw ? sh[1][lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) {
      e2 += __shfl_down_sync(0xffffffffu, e2, o);
      b2 += __shfl_down_sync(0xffffffffu, b2, o);
    }
    if (lane == 0) {
      atomicAdd(out, e2);
      atomicAdd(out + 1, b2);
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename real>
cudaError_t launch_faraday(const GridInfo& g, FieldView<real> EB, real c1, real c2,
                           const Stencil<real>& st, bool yee, cudaStream_t s) {
  const CellIter it = make_iter(g);
  const dim3     gr = grid_for(it.count, 256);
  if (g.dim == 2) {
    if (yee) PIC_KL(k_faraday<2, real, true><<<gr, 256, 0, s>>>(g, it, EB, c1, c2, st));
    else     PIC_KL(k_faraday<2, real, false><<<gr, 256, 0, s>>>(g, it, EB, c1, c2, st));
  } else {
    if (yee) PIC_KL(k_faraday<3, real, true><<<gr, 256, 0, s>>>(g, it, EB, c1, c2, st));
    else     PIC_KL(k_faraday<3, real, false><<<gr, 256, 0, s>>>(g, it, EB, c1, c2, st));
  }
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_ampere(const GridInfo& g, FieldView<real> EB, FieldView<real> J, real c1,
                          real c2, real jcoeff, real ppc0, bool curl, bool cur, bool fill,
                          cudaStream_t s) {
  const CellIter it = make_iter(g);
  const dim3     gr = grid_for(it.count, 256);
#define PIC_AMP(DD, A, B, C) PIC_KL(k_ampere<DD, real, A, B, C><<<gr, 256, 0, s>>>(g, it, EB, J, c1, c2, jcoeff, ppc0))
#define PIC_AMP_D(DD)                                                   \
  if (curl && cur && fill) PIC_AMP(DD, true, true, true);              \
  else if (curl && cur) PIC_AMP(DD, true, true, false);                 \
  else if (curl && fill) PIC_AMP(DD, true, false, true);               \
  else if (curl) PIC_AMP(DD, true, false, false);                       \
  else if (cur && fill) PIC_AMP(DD, false, true, true);                 \
  else if (cur) PIC_AMP(DD, false, true, false);
  if (g.dim == 2) {
    PIC_AMP_D(2)
  } else {
    PIC_AMP_D(3)
  }
#undef PIC_AMP_D
#undef PIC_AMP
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_sync_currents(const GridInfo& g, FieldView<real> J, cudaStream_t s) {
  const EdgeIter it = make_edges(g);
  if (it.count == 0) return cudaSuccess;
  const dim3     gr = grid_for(it.count, 256);
  if (g.dim == 2) PIC_KL(k_sync_currents<2, real><<<gr, 256, 0, s>>>(g, it, J));
  else            PIC_KL(k_sync_currents<3, real><<<gr, 256, 0, s>>>(g, it, J));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_fill_ghosts(const GridInfo& g, FieldView<real> f, int c0, int c1, cudaStream_t s) {
  const EdgeIter it = make_edges(g);
  if (it.count == 0 || c1 <= c0) return cudaSuccess;
  dim3 gr = grid_for(it.count, 256);
  gr.y    = (unsigned)(c1 - c0);
  if (g.dim == 2) PIC_KL(k_fill_ghosts<2, real><<<gr, 256, 0, s>>>(g, it, f, c0, c1));
  else            PIC_KL(k_fill_ghosts<3, real><<<gr, 256, 0, s>>>(g, it, f, c0, c1));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_filter(const GridInfo& g, FieldView<real> J, FieldView<real> buff, int npasses,
                          cudaStream_t s) {
  if (npasses <= 0) return cudaSuccess;
  const CellIter it       = make_iter(g);
  const dim3     gr       = grid_for(it.count, 256);
  const bool     all_per  = g.periodic[0] && g.periodic[1] && (g.dim == 2 || g.periodic[2]);
  const int64_t  ncells_g = (int64_t)(g.n[0] + 2 * g.ng) * (g.n[1] + 2 * g.ng) *
                           (g.dim == 3 ? g.n[2] + 2 * g.ng : 1) * 3;
  const dim3     grc      = grid_for(ncells_g, 256);
  if (all_per) {
    // ping-pong: every ghost cell is an image and is rewritten each pass
    FieldView<real> a = J, b = buff;
    for (int p = 0; p < npasses; ++p) {
      if (g.dim == 2) PIC_KL(k_filter2<real><<<gr, 256, 0, s>>>(g, it, a, b));
      else            filter3(g, a, b, s);
      FieldView<real> t = a;
      a                 = b;
      b                 = t;
    }
    if (npasses % 2 == 1) PIC_KL(k_copy3<real><<<grc, 256, 0, s>>>(g, buff, J));
  } else {
    // reference order: buff <- J (incl. non-periodic ghosts), filter, fill
    for (int p = 0; p < npasses; ++p) {
      PIC_KL(k_copy3<real><<<grc, 256, 0, s>>>(g, J, buff));
      if (g.dim == 2) PIC_KL(k_filter2<real><<<gr, 256, 0, s>>>(g, it, buff, J));
      else            filter3(g, buff, J, s);
    }
  }
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_copy3(const GridInfo& g, FieldView<real> src, FieldView<real> dst,
                         cudaStream_t s) {
  const int64_t ncells_g = (int64_t)(g.n[0] + 2 * g.ng) * (g.n[1] + 2 * g.ng) *
                           (g.dim == 3 ? g.n[2] + 2 * g.ng : 1) * 3;
  PIC_KL(k_copy3<real><<<grid_for(ncells_g, 256), 256, 0, s>>>(g, src, dst));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_zero3(const GridInfo& g, FieldView<real> f, cudaStream_t s) {
  // a packed field is one block of memory (1028 x 516 cells: 12.5 us by
  // k_zero3's divisions, 1.6 us by a memset)
  const int64_t e0 = g.n[0] + 2 * g.ng, e1 = g.n[1] + 2 * g.ng;
  const int64_t e2 = g.dim == 3 ? g.n[2] + 2 * g.ng : 1;
  if (f.s0 == 1 && f.s1 == e0 && (g.dim == 2 || f.s2 == e0 * e1) && f.s3 == e0 * e1 * e2)
    return cudaMemsetAsync(f.p, 0, sizeof(real) * (size_t)(3 * e0 * e1 * e2), s);
  const int64_t ncells_g = (int64_t)(g.n[0] + 2 * g.ng) * (g.n[1] + 2 * g.ng) *
                           (g.dim == 3 ? g.n[2] + 2 * g.ng : 1) * 3;
  PIC_KL(k_zero3<real><<<grid_for(ncells_g, 256), 256, 0, s>>>(g, f));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_energy(const GridInfo& g, FieldView<real> EB, double dx, double* out,
                          cudaStream_t s) {
  const CellIter it = make_iter(g);
  int64_t        b  = (it.count + 255) / 256;
  if (b > pic::sm_count() * 8) b = pic::sm_count() * 8;
  if (g.dim == 2) PIC_KL(k_energy<2, real><<<(unsigned)b, 256, 0, s>>>(it, EB, dx, out));
  else            PIC_KL(k_energy<3, real><<<(unsigned)b, 256, 0, s>>>(it, EB, dx, out));
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// adjoint (transposed) field operators. Each forward update of the step is a
// periodic linear map on the active cells (ghosts hold images); its transpose
// is applied in gather form to a ghost-filled adjoint field. Yee stencils only.
// ---------------------------------------------------------------------------

// lam(active, c < 3) = 2 h_c dV E_c: the gradient of the E part of the FP64
// energy of k_energy with respect to E; lam(active, c >= 3) = 0
template <int D, typename real>
__global__ void k_adj_seed(CellIter it, FieldView<real> EB, FieldView<real> lam, double dx) {
  const double  dV     = D == 3 ? dx * dx * dx : dx * dx;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i1, i2, i3;
    it.cell(t, i1, i2, i3);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double h = (c < D) ? dx * dx : 1.0;
      lam.p[lam.idx(i1, i2, i3, c)] = (real)(2.0 * h * dV * (double)EB.p[EB.idx(i1, i2, i3, c)]);
      lam.p[lam.idx(i1, i2, i3, c + 3)] = (real)0;
    }
  }
}

// transpose of CurrentsAmpere's E += jcoeff * J: lamJ = jcoeff * lamE at the
// active cells and their images
template <int D, typename real>
__global__ void k_adj_currents(GridInfo g, CellIter it, FieldView<real> lam, FieldView<real> lamJ,
                               real jcoeff) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i1, i2, i3;
    it.cell(t, i1, i2, i3);
    real v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v[c]                              = jcoeff * lam.p[lam.idx(i1, i2, i3, c)];
      lamJ.p[lamJ.idx(i1, i2, i3, c)] = v[c];
    }
    for_images<D>(g, i1, i2, i3, [&](int a, int b, int e) {
#pragma unroll
      for (int c = 0; c < 3; ++c) lamJ.p[lamJ.idx(a, b, e, c)] = v[c];
    });
  }
}

// transpose of k_ampere's curl: lamB(active) += A^T lamE (lamE ghost-filled)
template <int D, typename real>
__global__ void k_adj_ampere(CellIter it, FieldView<real> lam, real a1, real a2) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i, j, k;
    it.cell(t, i, j, k);
#define L(a, b, c, comp) lam.p[lam.idx(a, b, c, comp)]
    if constexpr (D == 2) {
      L(i, j, 0, 5) += a1 * (L(i, j, 0, 0) - L(i, j + 1, 0, 0)) + a1 * (L(i + 1, j, 0, 1) - L(i, j, 0, 1));
      L(i, j, 0, 3) += a2 * (L(i, j + 1, 0, 2) - L(i, j, 0, 2));
      L(i, j, 0, 4) += a2 * (L(i, j, 0, 2) - L(i + 1, j, 0, 2));
    } else {
      L(i, j, k, 3) += a1 * (L(i, j, k, 1) - L(i, j, k + 1, 1)) + a1 * (L(i, j + 1, k, 2) - L(i, j, k, 2));
      L(i, j, k, 4) += a1 * (L(i, j, k + 1, 0) - L(i, j, k, 0)) + a1 * (L(i, j, k, 2) - L(i + 1, j, k, 2));
      L(i, j, k, 5) += a1 * (L(i, j, k, 0) - L(i, j + 1, k, 0)) + a1 * (L(i + 1, j, k, 1) - L(i, j, k, 1));
    }
#undef L
  }
}

// transpose of k_faraday (Yee): lamE(active) += F^T lamB (lamB ghost-filled)
template <int D, typename real>
__global__ void k_adj_faraday(CellIter it, FieldView<real> lam, real c1, real c2) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < it.count; t += stride) {
    int i, j, k;
    it.cell(t, i, j, k);
#define L(a, b, c, comp) lam.p[lam.idx(a, b, c, comp)]
    if constexpr (D == 2) {
      L(i, j, 0, 2) += c1 * (L(i, j, 0, 3) - L(i, j - 1, 0, 3)) + c1 * (L(i - 1, j, 0, 4) - L(i, j, 0, 4));
      L(i, j, 0, 0) += c2 * (L(i, j - 1, 0, 5) - L(i, j, 0, 5));
      L(i, j, 0, 1) += c2 * (L(i, j, 0, 5) - L(i - 1, j, 0, 5));
    } else {
      L(i, j, k, 0) += c1 * (L(i, j, k, 4) - L(i, j, k - 1, 4)) + c1 * (L(i, j - 1, k, 5) - L(i, j, k, 5));
      L(i, j, k, 1) += c1 * (L(i, j, k - 1, 3) - L(i, j, k, 3)) + c1 * (L(i, j, k, 5) - L(i - 1, j, k, 5));
      L(i, j, k, 2) += c1 * (L(i, j, k, 3) - L(i, j - 1, k, 3)) + c1 * (L(i - 1, j, k, 4) - L(i, j, k, 4));
    }
#undef L
  }
}

// transpose of the ghost fill: every active cell adds the values its ghost
// images accumulated (components [c0, c1)) and clears them
template <int D, typename real>
__global__ void k_adj_fold(GridInfo g, EdgeIter it, FieldView<real> f, int c0, int c1) {
  const unsigned stride = gridDim.x * blockDim.x;
  for (int c = c0 + blockIdx.y; c < c1; c += gridDim.y)
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < it.count; t += stride) {
      int i1, i2, i3;
      it.cell(t, i1, i2, i3);
      // each ghost cell is the image of exactly one active cell, so the
      // thread that folds it may also clear it
      real acc = 0;
      for_images<D>(g, i1, i2, i3, [&](int a, int b, int e) {
        real* q = f.p + f.idx(a, b, e, c);
        acc += *q;
        *q = (real)0;
      });
      f.p[f.idx(i1, i2, i3, c)] += acc;
    }
}

// zero the ghost cells of components [c0, c1)
template <typename real>
__global__ void k_zero_ghosts(GridInfo g, FieldView<real> f, int c0, int c1) {
  const int     e0 = g.n[0] + 2 * g.ng, e1 = g.n[1] + 2 * g.ng;
  const int     e2 = g.dim == 3 ? g.n[2] + 2 * g.ng : 1;
  const int64_t count  = (int64_t)e0 * e1 * e2;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += stride) {
    int64_t   r = t;
    const int i = (int)(r % e0);
    r /= e0;
    const int j = (int)(r % e1);
    const int k = (int)(r / e1);
    const bool ghost = i < g.ng || i >= g.n[0] + g.ng || j < g.ng || j >= g.n[1] + g.ng ||
                       (g.dim == 3 && (k < g.ng || k >= g.n[2] + g.ng));
    if (!ghost) continue;
    for (int c = c0; c < c1; ++c) f.p[f.idx(i, j, k, c)] = (real)0;
  }
}

template <typename real>
cudaError_t launch_adj_seed(const GridInfo& g, FieldView<real> EB, FieldView<real> lam, double dx,
                            cudaStream_t s) {
  const CellIter it = make_iter(g);
  if (g.dim == 2) PIC_KL(k_adj_seed<2, real><<<grid_for(it.count, 256), 256, 0, s>>>(it, EB, lam, dx));
  else            PIC_KL(k_adj_seed<3, real><<<grid_for(it.count, 256), 256, 0, s>>>(it, EB, lam, dx));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_adj_currents(const GridInfo& g, FieldView<real> lam, FieldView<real> lamJ,
                                real jcoeff, cudaStream_t s) {
  const CellIter it = make_iter(g);
  if (g.dim == 2) PIC_KL(k_adj_currents<2, real><<<grid_for(it.count, 256), 256, 0, s>>>(g, it, lam, lamJ, jcoeff));
  else            PIC_KL(k_adj_currents<3, real><<<grid_for(it.count, 256), 256, 0, s>>>(g, it, lam, lamJ, jcoeff));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_adj_ampere(const GridInfo& g, FieldView<real> lam, real a1, real a2,
                              cudaStream_t s) {
  const CellIter it = make_iter(g);
  if (g.dim == 2) PIC_KL(k_adj_ampere<2, real><<<grid_for(it.count, 256), 256, 0, s>>>(it, lam, a1, a2));
  else            PIC_KL(k_adj_ampere<3, real><<<grid_for(it.count, 256), 256, 0, s>>>(it, lam, a1, a2));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_adj_faraday(const GridInfo& g, FieldView<real> lam, real c1, real c2,
                               cudaStream_t s) {
  const CellIter it = make_iter(g);
  if (g.dim == 2) PIC_KL(k_adj_faraday<2, real><<<grid_for(it.count, 256), 256, 0, s>>>(it, lam, c1, c2));
  else            PIC_KL(k_adj_faraday<3, real><<<grid_for(it.count, 256), 256, 0, s>>>(it, lam, c1, c2));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_adj_fold(const GridInfo& g, FieldView<real> f, int c0, int c1, cudaStream_t s) {
  const EdgeIter it = make_edges(g);
  if (it.count == 0 || c1 <= c0) return cudaSuccess;
  dim3 gr = grid_for(it.count, 256);
  gr.y    = (unsigned)(c1 - c0);
  if (g.dim == 2) PIC_KL(k_adj_fold<2, real><<<gr, 256, 0, s>>>(g, it, f, c0, c1));
  else            PIC_KL(k_adj_fold<3, real><<<gr, 256, 0, s>>>(g, it, f, c0, c1));
  return cudaGetLastError();
}

template <typename real>
cudaError_t launch_zero_ghosts(const GridInfo& g, FieldView<real> f, int c0, int c1,
                               cudaStream_t s) {
  const int64_t cells = (int64_t)(g.n[0] + 2 * g.ng) * (g.n[1] + 2 * g.ng) *
                        (g.dim == 3 ? g.n[2] + 2 * g.ng : 1);
  PIC_KL(k_zero_ghosts<real><<<grid_for(cells, 256), 256, 0, s>>>(g, f, c0, c1));
  return cudaGetLastError();
}

#define PIC_INST_ADJ_FIELDS(R)                                                                     \
  template cudaError_t launch_adj_seed<R>(const GridInfo&, FieldView<R>, FieldView<R>, double,     \
                                          cudaStream_t);                                           \
  template cudaError_t launch_adj_currents<R>(const GridInfo&, FieldView<R>, FieldView<R>, R,      \
                                              cudaStream_t);                                       \
  template cudaError_t launch_adj_ampere<R>(const GridInfo&, FieldView<R>, R, R, cudaStream_t);    \
  template cudaError_t launch_adj_faraday<R>(const GridInfo&, FieldView<R>, R, R, cudaStream_t);   \
  template cudaError_t launch_adj_fold<R>(const GridInfo&, FieldView<R>, int, int, cudaStream_t);  \
  template cudaError_t launch_zero_ghosts<R>(const GridInfo&, FieldView<R>, int, int, cudaStream_t);
PIC_INST_ADJ_FIELDS(float)
PIC_INST_ADJ_FIELDS(double)

#define PIC_INST_FIELDS(R)                                                                       \
  template cudaError_t launch_faraday<R>(const GridInfo&, FieldView<R>, R, R, const Stencil<R>&, \
                                         bool, cudaStream_t);                                    \
  template cudaError_t launch_ampere<R>(const GridInfo&, FieldView<R>, FieldView<R>, R, R, R, R, \
                                        bool, bool, bool, cudaStream_t);                         \
  template cudaError_t launch_sync_currents<R>(const GridInfo&, FieldView<R>, cudaStream_t);     \
  template cudaError_t launch_fill_ghosts<R>(const GridInfo&, FieldView<R>, int, int,            \
                                             cudaStream_t);                                      \
  template cudaError_t launch_filter<R>(const GridInfo&, FieldView<R>, FieldView<R>, int,        \
                                        cudaStream_t);                                           \
  template cudaError_t launch_zero3<R>(const GridInfo&, FieldView<R>, cudaStream_t);             \
  template cudaError_t launch_copy3<R>(const GridInfo&, FieldView<R>, FieldView<R>, cudaStream_t); \
  template cudaError_t launch_energy<R>(const GridInfo&, FieldView<R>, double, double*,          \
                                        cudaStream_t);

PIC_INST_FIELDS(float)
PIC_INST_FIELDS(double)

}  // namespace pic
