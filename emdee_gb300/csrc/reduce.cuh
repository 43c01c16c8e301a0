// reduce.cuh -- deterministic block and grid reductions of FP64 partial sums.
//
// THREADS is the largest block size the kernel is launched with.  Each block reduces
// its per-thread values (warp shuffles, then warps in order) and writes one partial
// per quantity; the last block to finish (ticket counter) sums the partials in a fixed
// order with Neumaier compensation.  The result does not depend on block scheduling.
#pragma once

namespace emdee {

// Per-thread FP64 values -> result[q], also into result2 if set (e.g. pinned host
// memory: no copy back).  partials holds NQ doubles per block.
//
// A small system waits for this reduction's latency, a chain of FP64 additions on a
// pipe that takes 16 clocks per warp instruction, so the chain is kept short: the
// values of a warp are summed and distributed over the lanes together (NQ/2 + NQ/4 +
// ... additions, not 5 NQ), the warps' sums are added by one thread per quantity, and
// the last block's warps take the quantities side by side (5 sums: k_bonded 34 -> 25 us
// at 512 molecules, k_vv_post_free 13 -> 11 us at 16,001 atoms).
template <int NQ, int THREADS>
__device__ __forceinline__ void grid_reduce(const double (&v)[NQ], double* partials, unsigned int* ticket,
                                            double* result, double* result2 = nullptr) {
  static_assert(NQ <= 16, "at most 16 quantities");
  constexpr int P = NQ <= 1 ? 1 : NQ <= 2 ? 2 : NQ <= 4 ? 4 : NQ <= 8 ? 8 : 16;
  __shared__ double red[P][THREADS / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  double w[P];
#pragma unroll
  for (int q = 0; q < P; q++) w[q] = q < NQ ? v[q] : 0.0;
#pragma unroll
  for (int l = 0; l < 5; l++) {
    const int o = 16 >> l, h = P >> (l + 1);   // quantities a lane keeps after this level
    if (h >= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int k = 0; k < h; k++) {
        const double keep = up ? w[k + h] : w[k];
        w[k] = keep + __shfl_xor_sync(0xffffffffu, up ? w[k] : w[k + h], o);
      }
    } else {
      w[0] += __shfl_xor_sync(0xffffffffu, w[0], o);
    }
  }
  // lane q * (32 / P) holds the warp's sum of quantity q
  if (lane % (32 / P) == 0) red[lane / (32 / P)][warp] = w[0];
  __syncthreads();
  if (warp == 0) {
    if (lane < NQ) {
      double x = 0.0;
      for (int k = 0; k < nw; k++) x += red[lane][k];
      partials[(size_t)blockIdx.x * NQ + lane] = x;
      __threadfence();   // the partial is visible before the ticket counts this block
    }
    __syncwarp();
    if (lane == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // last block: a group of warps per quantity sums the partials in a fixed order
  // (Neumaier), which never depends on which block finished last
  const int per = nw / NQ > 0 ? nw / NQ : 1, groups = nw / per;
  for (int q0 = 0; q0 < NQ; q0 += groups) {
    const int q = q0 + warp / per, part = warp % per;
    if (q < NQ && warp / per < groups) {
      double s = 0.0, c = 0.0;
      constexpr int U = 8;   // partials in flight per thread, added in increasing block order
      for (unsigned int b0 = part * 32 + lane; b0 < gridDim.x; b0 += U * per * 32) {
        double xs[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const unsigned int b = b0 + u * per * 32;
          xs[u] = b < gridDim.x ? __ldcg(&partials[(size_t)b * NQ + q]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (b0 + u * per * 32 >= gridDim.x) break;
          const double x = xs[u], t = s + x;
          c += fabs(s) >= fabs(x) ? (s - t) + x : (x - t) + s;
          s = t;
        }
      }
      double x = s + c;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) red[q][part] = x;
    }
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    double x = 0.0;
    for (int k = 0; k < per; k++) x += red[threadIdx.x][k];
    result[threadIdx.x] = x;
    if (result2) result2[threadIdx.x] = x;
  }
  if (threadIdx.x == 0) *ticket = 0;
}

// ---- float-float (FP32 pair) reductions: every level on the FP32 pipe ----------
//
// A value is carried as hi + lo with |lo| << |hi|; additions use Knuth's
// error-free two-sum on the high parts and plain addition of the low parts, so
// the sum keeps about 48 significant bits.  Only the final hi + lo conversion
// per quantity touches FP64.

__device__ __forceinline__ void ff_add(float& hi, float& lo, float bh, float bl) {
  const float s = hi + bh, bp = s - hi, err = (hi - (s - bp)) + (bh - bp);
  hi = s;
  lo = lo + bl + err;
}

// Quantities whose bit is clear in MASK are known to be zero: they skip every
// level and their result is written as 0.
template <int NQ, unsigned MASK = ~0u>
__device__ __forceinline__ void warp_sum_ff(float (&hi)[NQ], float (&lo)[NQ]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      if (!((MASK >> q) & 1u)) continue;
      const float h2 = __shfl_down_sync(0xffffffffu, hi[q], o), l2 = __shfl_down_sync(0xffffffffu, lo[q], o);
      ff_add(hi[q], lo[q], h2, l2);
    }
}

// Per-thread float-float values (hi + lo) -> result[q] (FP64), also into result2 if
// set; partials holds NQ float2 per block.  Every level runs on the FP32 pipe.
template <int NQ, int THREADS>
__device__ __forceinline__ void grid_reduce_ff2(const float (&vh)[NQ], const float (&vl)[NQ], float2* partials,
                                                unsigned int* ticket, double* result, double* result2) {
  __shared__ float2 red2[NQ][THREADS / 32];
  __shared__ bool last2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  float hi[NQ], lo[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    hi[q] = vh[q];
    lo[q] = vl[q];
  }
  warp_sum_ff<NQ>(hi, lo);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; q++) red2[q][warp] = make_float2(hi[q], lo[q]);
  __syncthreads();
  if (threadIdx.x < NQ) {
    const int q = threadIdx.x;
    float h = 0.f, l = 0.f;
    for (int w = 0; w < nw; w++) ff_add(h, l, red2[q][w].x, red2[q][w].y);
    partials[(size_t)blockIdx.x * NQ + q] = make_float2(h, l);
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last2 = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last2) return;
  __threadfence();
#pragma unroll
  for (int q = 0; q < NQ; q++) hi[q] = lo[q] = 0.f;
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x)   // block order per thread
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const float2 x = __ldcg(&partials[(size_t)b * NQ + q]);
      ff_add(hi[q], lo[q], x.x, x.y);
    }
  warp_sum_ff<NQ>(hi, lo);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; q++) red2[q][warp] = make_float2(hi[q], lo[q]);
  __syncthreads();
  if (threadIdx.x < NQ) {
    const int q = threadIdx.x;
    float h = 0.f, l = 0.f;
    for (int w = 0; w < nw; w++) ff_add(h, l, red2[q][w].x, red2[q][w].y);
    result[q] = (double)h + (double)l;
    if (result2) result2[q] = (double)h + (double)l;
  }
  if (threadIdx.x == 0) *ticket = 0;
}

// Per-thread FP32 values -> result[q] (FP64), also into result2 if set.  partials holds
// NQ float2 per block.
// The last block (ticket) sums the partials in block order; the result does not
// depend on block scheduling.  done (pinned host memory), if set, gets the value stamp
// once result2 is in place: the host can read it there before the grid has drained.
template <int NQ, int THREADS, unsigned MASK = ~0u>
__device__ __forceinline__ void grid_reduce_ff(const float (&v)[NQ], float2* partials, unsigned int* ticket,
                                               double* result, double* result2 = nullptr,
                                               unsigned int* done = nullptr, unsigned int stamp = 0) {
  __shared__ float2 red[NQ][THREADS / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  float hi[NQ], lo[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    hi[q] = v[q];
    lo[q] = 0.f;
  }
  warp_sum_ff<NQ, MASK>(hi, lo);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; q++)
      if ((MASK >> q) & 1u) red[q][warp] = make_float2(hi[q], lo[q]);
  __syncthreads();
  if (threadIdx.x < NQ && ((MASK >> threadIdx.x) & 1u)) {
    const int q = threadIdx.x;
    float h = 0.f, l = 0.f;
    for (int w = 0; w < nw; w++) ff_add(h, l, red[q][w].x, red[q][w].y);
    partials[(size_t)blockIdx.x * NQ + q] = make_float2(h, l);
    __threadfence();   // the partial is visible before the ticket counts this block
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    hi[q] = 0.f;
    lo[q] = 0.f;
  }
  // U partials per quantity in flight per thread, added in increasing block order
  constexpr int U = 8;
  for (unsigned int b0 = threadIdx.x; b0 < gridDim.x; b0 += U * blockDim.x) {
    float2 x[U][NQ];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const unsigned int b = b0 + u * blockDim.x;
#pragma unroll
      for (int q = 0; q < NQ; q++)
        if ((MASK >> q) & 1u) x[u][q] = b < gridDim.x ? __ldcg(&partials[(size_t)b * NQ + q]) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (b0 + u * blockDim.x < gridDim.x)
#pragma unroll
        for (int q = 0; q < NQ; q++)
          if ((MASK >> q) & 1u) ff_add(hi[q], lo[q], x[u][q].x, x[u][q].y);
  }
  warp_sum_ff<NQ, MASK>(hi, lo);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NQ; q++)
      if ((MASK >> q) & 1u) red[q][warp] = make_float2(hi[q], lo[q]);
  __syncthreads();
  if (threadIdx.x < NQ) {
    const int q = threadIdx.x;
    float h = 0.f, l = 0.f;
    if ((MASK >> q) & 1u)
      for (int w = 0; w < nw; w++) ff_add(h, l, red[q][w].x, red[q][w].y);
    result[q] = (double)h + (double)l;
    if (result2) result2[q] = (double)h + (double)l;   // e.g. pinned host memory: no copy back
    if (done) __threadfence_system();
  }
  __syncwarp();
  if (threadIdx.x == 0) {
    *ticket = 0;
    if (done) *(volatile unsigned int*)done = stamp;
  }
}

}  // namespace emdee
