// Kernels of the exact global current accumulation (deposit_fixed.cuh).
#include <climits>

#include "deposit_fixed.cuh"
#include "pic_types.h"

namespace pic {

// One block of 256 threads looks at every fourth particle of 32 chunks over a species:
// whether the cells of three chunks in four fit a window. All its loads are in flight
// together (one after another they took 25 us).
__device__ __forceinline__ void chunk_order(const BoundArgs& a, int s) {
  constexpr int EACH   = 4;  // chunks of a warp, and particles of a lane in each
  const int     lane   = threadIdx.x & 31;
  const int64_t chunks = (a.n[s] + kChunk - 1) / kChunk, part = chunks / 32 + 1;
  static_assert(kChunk == 32 * EACH * 4, "a fourth of a chunk");
  int c[EACH][EACH][2];
#pragma unroll
  for (int r = 0; r < EACH; ++r) {
    // at another place in each thirty-second: equal steps can meet a row's end each time
    const int     w  = (threadIdx.x >> 5) * EACH + r;
    const int64_t p0 = (chunks * w / 32 + w * 29 % part) % chunks * kChunk;
#pragma unroll
    for (int k = 0; k < EACH; ++k) {
      int64_t p = p0 + (k * 32 + lane) * 4;
      p         = p < a.n[s] ? p : a.n[s] - 1;
#pragma unroll
      for (int d = 0; d < 2; ++d) c[r][k][d] = a.cells[s][d][p];
    }
  }
  int fit = 0;
#pragma unroll
  for (int r = 0; r < EACH; ++r) {
    int64_t nodes = 1;
    bool    some  = true;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      int lo = INT_MAX, hi = INT_MIN;
#pragma unroll
      for (int k = 0; k < EACH; ++k)
        if (cells_in_grid<2>(c[r][k], a.grid)) lo = min(lo, c[r][k][d]), hi = max(hi, c[r][k][d]);
      lo   = __reduce_min_sync(0xffffffffu, lo);
      hi   = __reduce_max_sync(0xffffffffu, hi);
      some = some && lo <= hi;
      nodes *= (int64_t)hi - lo + 6;
    }
    fit += some && nodes <= kChunkNodes;
  }
  __shared__ int s_fit;
  if (threadIdx.x == 0) s_fit = 0;
  __syncthreads();
  if (lane == 0) atomicAdd(&s_fit, fit);
  __syncthreads();
  if (threadIdx.x == 0) *a.chunked[s] = 4 * s_fit >= 3 * 32;
}

// max |w| |q| over the weights of up to kBoundSpecies species (blockIdx.y);
// 16-byte loads where the array allows, one atomic per block. A species whose order is
// asked for has its first block do that besides.
__global__ void k_weight_bound(const __grid_constant__ BoundArgs a) {
  const int     s      = blockIdx.y;
  if (blockIdx.x == 0 && a.chunked[s]) chunk_order(a, s);
  const float*  w      = a.w[s];
  const int64_t n      = a.n[s];
  const int64_t tid    = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t n4     = (reinterpret_cast<uintptr_t>(w) % 16 == 0) ? n / 4 : 0;
  const float4* w4     = reinterpret_cast<const float4*>(w);
  float         m      = 0.f;
  // four loads in flight per thread
  int64_t i = tid;
  for (; i + 3 * stride < n4; i += 4 * stride) {
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = w4[i + k * stride];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      m = fmaxf(m, fmaxf(fmaxf(fabsf(v[k].x), fabsf(v[k].y)), fmaxf(fabsf(v[k].z), fabsf(v[k].w))));
  }
  for (; i < n4; i += stride) {
    const float4 v = w4[i];
    m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
  }
  for (i = 4 * n4 + tid; i < n; i += stride) m = fmaxf(m, fabsf(w[i]));
  // |q| max|w| = max |q||w|: multiplication by |q| >= 0 keeps the order
  m = m * a.q[s];
  // non-negative floats order as their bit patterns
  __shared__ unsigned sm;
  if (threadIdx.x == 0) sm = 0u;
  __syncthreads();
  atomicMax(&sm, __reduce_max_sync(0xffffffffu, __float_as_uint(m)));
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(a.bound, sm);
}

// One total per thread at a time, neighbours along x in neighbouring threads
// (a block per grid row left half of its threads idle on the rows' last few
// cells: 260 us at 256^3, 124 us so). PACKED: J is laid out like the totals.
template <bool PACKED>
__global__ void __launch_bounds__(256) k_fixed_to_real(FixedJ fj, FieldView<float> J, int64_t e0,
                                                       int64_t e1, int64_t e2, int64_t count,
                                                       int overwrite) {
  const int      ex      = fj.exponent();
  const float    unscale = ldexpf(1.f, ex - fj.bits);
  const int64_t  stride  = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += stride) {
    const long long x = __ldcs(fj.p + t);
    float*          o = J.p + t;
    if constexpr (!PACKED) {
      const int64_t r = t / e0, i = t - r * e0, q = r / e1, j = r - q * e1, c = q / e2, k = q - c * e2;
      o = J.p + J.idx((int)i, (int)j, (int)k, (int)c);
    }
    if (overwrite) *o = __ll2float_rn(x) * unscale;
    else if (x != 0) *o = *o + __ll2float_rn(x) * unscale;
  }
}

cudaError_t launch_weight_bound(const BoundArgs& a, cudaStream_t s) {
  int64_t nmax = 0;
  for (int k = 0; k < a.ns; ++k) nmax = a.n[k] > nmax ? a.n[k] : nmax;
  if (a.ns <= 0 || nmax <= 0) return cudaSuccess;
  // enough 256-thread blocks for one 16-byte load per thread, at most 4 per SM
  int64_t blocks = (nmax / 4 + 255) / 256;
  if (blocks > sm_count() * 4) blocks = sm_count() * 4;
  if (blocks < 1) blocks = 1;
  PIC_KL(k_weight_bound<<<dim3((unsigned)blocks, (unsigned)a.ns), 256, 0, s>>>(a));
  return cudaGetLastError();
}

cudaError_t launch_fixed_to_real(const FixedJ& fj, FieldView<float> J, const int* ext,
                                 bool overwrite, cudaStream_t s) {
  const int64_t count = (int64_t)3 * ext[0] * ext[1] * ext[2];
  int64_t blocks = (count + 255) / 256;
  if (blocks > sm_count() * 64) blocks = sm_count() * 64;
  const bool packed = J.s0 == 1 && J.s1 == fj.s1 && (ext[2] == 1 || J.s2 == fj.s2) && J.s3 == fj.s3;
  if (packed)
    PIC_KL(k_fixed_to_real<true><<<(unsigned)blocks, 256, 0, s>>>(fj, J, ext[0], ext[1], ext[2],
                                                                  count, overwrite ? 1 : 0));
  else
    PIC_KL(k_fixed_to_real<false><<<(unsigned)blocks, 256, 0, s>>>(
      fj, J, ext[0], ext[1], ext[2], count, overwrite ? 1 : 0));
  return cudaGetLastError();
}

}  // namespace pic
