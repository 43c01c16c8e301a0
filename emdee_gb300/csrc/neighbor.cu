// neighbor.cu -- skin-displacement check, cell binning into tiles and the
// Verlet neighbor-list build (src/neighbor_lists.f90).
//
// The pair set is the reference's: every pair (i, j) whose minimum-image
// distance, computed from scaled FP64 coordinates exactly as in
// src/neighbor_lists.f90:247-250 (Rs = R/L, d = Rs_i - Rs_j, d -= anint(d),
// r2 = dx^2 + dy^2 + dz^2), is below (rc+skin)^2/L^2, that is not excluded
// (EmDee_ignore_pair), not in the same rigid body and whose types interact.
// An FP32 distance in a tile-local frame decides every candidate that is
// clearly inside or outside; candidates within a relative 4e-5 of the
// threshold are decided by the FP64 test.  This file is compiled with
// -fmad=false so the FP64 test rounds like the reference.
//
// Unlike the reference's half lists, the lists are full (each pair appears in
// the lists of both atoms), so the force kernel owns every atom's force and
// needs no atomics.
#include <algorithm>
#include <cmath>
#include <vector>

#include "chain.cuh"
#include "system.hpp"
#include "tile.cuh"

namespace emdee {

static const int NDIV = 2;   // src/EmDeeData.f90:33
static const double BAND = LIST_BAND;

// ---------------------------------------------------------------------------------
// skin check: maximum_approach_sq (src/neighbor_lists.f90:41-59)
//
// The reference scans atoms in order, refreshing "next" only when a new
// maximum appears.  Its result is max + 2 sqrt(max*next) + next, where
// next = the largest value before the first occurrence of the maximum (or the
// maximum itself when that occurrence is atom 1).  (m, p) pairs over
// contiguous index ranges combine associatively:
//   (mA,pA) . (mB,pB) = mB > mA ? (mB, max(mA, pB)) : (mA, pA)
// ---------------------------------------------------------------------------------

// Values are squared displacements (>= 0), so their IEEE-754 bit patterns order
// like the values: the combine runs on 64-bit integers (-1 = none) instead of
// the slow FP64 pipe.
struct MaxPrev {
  long long m, p;   // bit patterns; p < 0: no element precedes the first maximum
};

__device__ __forceinline__ MaxPrev mp_combine(MaxPrev a, MaxPrev b) {
  if (b.m > a.m) return MaxPrev{b.m, a.m > b.p ? a.m : b.p};
  return a;
}

// Each warp takes `chunks` x 32 consecutive atoms: SKIN_CHUNKS where the grid fills the
// SMs, fewer below (the ordered combine of a chunk waits for its loads, so a small
// system in chunks of 8 pays eight memory latencies in a row; 16,001 atoms: 11.5 -> 6 us
// with the sums written straight to pinned memory).
// The value does not depend on it.
static const int SKIN_THREADS = 256, SKIN_CHUNKS = 8;
static int skin_chunks(int N, int most) {
  const int c = N / (152 * 4 * SKIN_THREADS);
  return c < 1 ? 1 : c < most ? c : most;
}

__device__ __forceinline__ MaxPrev warp_ordered_combine(MaxPrev acc) {
  // after the loop lane 0 holds the combination of lanes 0..31 in lane order
  const int lane = threadIdx.x & 31;
  for (int o = 1; o < 32; o <<= 1) {
    MaxPrev other{(long long)__shfl_down_sync(0xffffffffu, (unsigned long long)acc.m, o),
                  (long long)__shfl_down_sync(0xffffffffu, (unsigned long long)acc.p, o)};
    if ((lane & (2 * o - 1)) == 0) acc = mp_combine(acc, other);
  }
  return acc;
}

__device__ __forceinline__ float4 pack_delta(float4 p0, double dx, double dy, double dz, float scale);

// PACK: also the FP32 positions of k_pack_delta, from the displacements at hand (one pass
// over R and R0 less: 4096 rigid waters, 5 steps, 783 -> 779 us).
template <bool PACK>
__global__ void __launch_bounds__(SKIN_THREADS) k_skin(const double* R, const double* R0,
                                                       int N, int chunks, double skinSq, longlong2* partial,
                                                       unsigned int* ticket, double* result, double* hostResult,
                                                       const int* slotOf,
                                                       const float4* pos0, float scale,
                                                       float4* __restrict__ pos4, unsigned long long* done,
                                                       unsigned int stamp) {
  chain_wait();
  __shared__ MaxPrev wsum[SKIN_THREADS / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int base = (blockIdx.x * (SKIN_THREADS / 32) + warp) * 32 * chunks;
  MaxPrev run{-1, -1};
  for (int c = 0; c < chunks; c++) {
    const int i = base + c * 32 + lane;
    MaxPrev v{-1, -1};
    if (i < N) {
      double d0 = R[3 * i] - R0[3 * i], d1 = R[3 * i + 1] - R0[3 * i + 1], d2 = R[3 * i + 2] - R0[3 * i + 2];
      v.m = __double_as_longlong(d0 * d0 + d1 * d1 + d2 * d2);
      if (PACK) pos4[slotOf[i]] = pack_delta(pos0[i], d0, d1, d2, scale);
    }
    v = warp_ordered_combine(v);
    run = mp_combine(run, v);   // meaningful in lane 0
  }
  if (lane == 0) wsum[warp] = run;
  __syncthreads();
  if (threadIdx.x == 0) {
    MaxPrev b = wsum[0];
    for (int w = 1; w < SKIN_THREADS / 32; w++) b = mp_combine(b, wsum[w]);
    partial[blockIdx.x] = make_longlong2(b.m, b.p);
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // last block: each warp combines a contiguous range of block partials in
  // order, then warp results are combined in order
  const int nb = gridDim.x, per = (nb + SKIN_THREADS - 1) / SKIN_THREADS;
  MaxPrev acc{-1, -1};
  for (int k = 0; k < per; k++) {
    int b = threadIdx.x * per + k;
    if (b < nb) {
      longlong2 v = __ldcg(&partial[b]);
      acc = mp_combine(acc, MaxPrev{v.x, v.y});
    }
  }
  acc = warp_ordered_combine(acc);
  if (lane == 0) wsum[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    MaxPrev b = wsum[0];
    for (int w = 1; w < SKIN_THREADS / 32; w++) b = mp_combine(b, wsum[w]);
    double maximum = __longlong_as_double(b.m), next = __longlong_as_double(b.p < 0 ? b.m : b.p);
    double value = maximum + 2 * sqrt(maximum * next) + next;
    result[8] = hostResult[8] = value;   // pinned host memory: read after the synchronisation
    result[9] = hostResult[9] = value > skinSq ? 1.0 : 0.0;
    *ticket = 0;
    *(volatile unsigned long long*)done = 2ull * stamp + (value > skinSq ? 1 : 0);   // pinned, one store
  }
}

static void ensure_partials(System& s, int n) {
  if (s.partialCap < n) {
    CK(cudaFree(s.dPartials));
    s.partialCap = std::max(n, 1024);
    CK(cudaMalloc(&s.dPartials, sizeof(double) * 5 * s.partialCap));
  }
}

void device_skin_launch(System& s, bool pack) {
  const int N = s.natoms, chunks = skin_chunks(N, SKIN_CHUNKS), per = SKIN_THREADS * chunks;
  const int blocks = (N + per - 1) / per;
  const Grid& g = s.grid;
  ensure_partials(s, blocks);
  prof_begin(s, PK_SKIN);
  launch_chained(pack ? k_skin<true> : k_skin<false>, blocks, SKIN_THREADS, 0, s.stream, s.dR, s.dR0, N, chunks,
                 s.skinSq, (longlong2*)s.dPartials, s.dTicket, s.dResult, s.hResult, g.dSlotOf, g.dPos0,
                 (float)((double)g.M / *s.Lbox), g.dPos4, s.hSkinDone, ++s.skinStamp);
  CK(cudaGetLastError());
  prof_end(s, PK_SKIN);
}

bool device_skin_check(System& s) {
  device_skin_launch(s, false);
  CK(cudaStreamSynchronize(s.stream));
  return s.hResult[9] != 0.0;
}

// ---------------------------------------------------------------------------------
// binning (src/neighbor_lists.f90:122-128) and tile sort
// ---------------------------------------------------------------------------------

// FP32 rounding of a double (nearest even) on the integer pipes when the result
// is a normal float, else the hardware conversion
__device__ __forceinline__ float d2f(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return d2f_normal(b) ? __uint_as_float(d2f_bits(b)) : (float)x;
}

// value of an integer-valued double with |f| < 2^31, from its bits (no FP64 pipe)
__device__ __forceinline__ int dint_exact(double f) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(f);
  const int e = (int)((b >> 52) & 0x7FF) - 1023;
  if (e < 0) return 0;
  const int v = (int)(((b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) >> (52 - e));
  return (b >> 63) ? -v : v;
}

// FP32 copy of a charge, zero below the reference's threshold (|q| > epsilon,
// src/EmDeeCode.f90:879-880), compared and converted on the integer pipes
__device__ __forceinline__ float charge_f32(double q) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(q) & 0x7FFFFFFFFFFFFFFFull;
  return b > 0x3CB0000000000000ull ? d2f(q) : 0.0f;   // 0x3CB0... = 2^-52
}

// Per atom (API order): the image-resolved cell K = floor(M R / L) of each
// coordinate, the cell's rank, the cell-local FP32 position u = M R/L - K with the
// charge (the build-time reference pos0 of the packing), the coordinates R0 of
// this build for the skin check, and the atom's place among its cell's atoms.
// M R/L is one FP64 product per coordinate; its floor and remainder are the only
// other FP64 operations (the remainder is exact), and every later stage of the
// build reads u instead of recomputing it.  A cell index that differs from the
// reference's int(M (R/L - floor(R/L))) by rounding at a cell boundary changes
// only the order of candidates, not the pair set.
__global__ void k_assign(const double* R, const double* __restrict__ charge, int N, double scale,
                         TileGeom g, int4* atomK, int* count, int* inCell, float4* pos0, double* __restrict__ R0,
                         int* dMax, unsigned long long* fail) {
  chain_wait();
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < 4) dMax[a] = 0;   // the maxima of this build and its failure flag
  if (a == 4) *fail = 0ull;
  if (a >= N) return;
  int c[3], K[3];
  float u[3];
  for (int d = 0; d < 3; d++) {
    const double r = R[3 * a + d], t = r * scale, fl = floor(t);
    K[d] = dint_exact(fl);
    int ci = K[d] % g.M;
    c[d] = ci < 0 ? ci + g.M : ci;
    u[d] = d2f(t - fl);
    R0[3 * a + d] = r;
  }
  int rank = cell_rank(g, c[0], c[1], c[2]);
  atomK[a] = make_int4(K[0], K[1], K[2], rank);
  pos0[a] = make_float4(u[0], u[1], u[2], charge_f32(charge[a]));
  // one atomic per distinct cell of the warp (neighbouring atoms often share a
  // cell); each atom keeps its place among the cell's atoms for the scatter
  const unsigned active = __activemask();
  const unsigned peers = __match_any_sync(active, rank);
  const int leader = __ffs(peers) - 1, lane = threadIdx.x & 31;
  int base = 0;
  if (lane == leader) base = atomicAdd(&count[rank], __popc(peers));
  base = __shfl_sync(peers, base, leader);
  inCell[a] = base + __popc(peers & ((1u << lane) - 1u));
}

// device-wide exclusive scan (counts -> starts) in two phases, starts[n] = total: tiles,
// then every block adds the tiles before its own.  The counts are left zero for the next
// build.  (Launches and memsets are what a rebuild of a small system costs.)  Adding the tiles
// up in every block is quadratic in their number: above SCAN_DIRECT a block of its own
// scans the sums in between (7,600 tiles: 37 us without, 41 with it; 61,000: 366 and 320).
static const int SCAN_THREADS = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
static const int SCAN_DIRECT = 8192;

__global__ void k_scan_local(int* in, int* out, int n, int* blockSums) {
  chain_wait();
  __shared__ int buf[SCAN_TILE];
  __shared__ int ws[33];
  int base = blockIdx.x * SCAN_TILE;
  for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_THREADS) buf[k] = base + k < n ? in[base + k] : 0;
  __syncthreads();
  // (after the loads: a store between them keeps each waiting for the one before, 34 us
  // against 7 for the 438,976 cells of 1,048,576 atoms)
  for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_THREADS)
    if (base + k < n) in[base + k] = 0;
  int total = block_exclusive_scan<SCAN_ITEMS>(buf, SCAN_TILE, ws);
  for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_THREADS)
    if (base + k < n) out[base + k] = buf[k];
  if (threadIdx.x == 0) blockSums[blockIdx.x] = total;
}

// exclusive scan of the tiles' totals in place, by one block; the sum to out[n]
__global__ void k_scan_sums(int* blockSums, int nb, int* out, int n) {
  chain_wait();
  __shared__ int buf[SCAN_TILE];
  __shared__ int ws[33];
  int before = 0;
  for (int base = 0; base < nb; base += SCAN_TILE) {
    const int m = min(SCAN_TILE, nb - base);
    for (int k = threadIdx.x; k < m; k += SCAN_THREADS) buf[k] = blockSums[base + k];
    __syncthreads();
    const int total = block_exclusive_scan<SCAN_ITEMS>(buf, m, ws);
    for (int k = threadIdx.x; k < m; k += SCAN_THREADS) blockSums[base + k] = before + buf[k];
    before += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = before;
}

// SCANNED: blockSums holds the tiles' starts, otherwise their totals
template <bool SCANNED>
__global__ void k_scan_add(int* out, int n, const int* blockSums) {
  chain_wait();
  __shared__ int ws[SCAN_THREADS / 32];
  int add = 0;
  if (SCANNED) {
    add = blockSums[blockIdx.x];
  } else {
    int before = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += SCAN_THREADS) before += blockSums[b];
    before = __reduce_add_sync(0xffffffffu, before);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = before;
    __syncthreads();
    for (int w = 0; w < SCAN_THREADS / 32; w++) add += ws[w];
  }
  const int base = blockIdx.x * SCAN_TILE;
  for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_THREADS)
    if (base + k < n) out[base + k] += add;
  if (!SCANNED && threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) out[n] = add + blockSums[blockIdx.x];
}

static void device_scan(System& s, int* in, int* out, int n) {
  int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  launch_chained(k_scan_local, nb, SCAN_THREADS, 0, s.stream, in, out, n, s.grid.dScanTmp);
  if (nb > SCAN_DIRECT) {
    launch_chained(k_scan_sums, 1, SCAN_THREADS, 0, s.stream, s.grid.dScanTmp, nb, out, n);
    s.prof.total++;
  }
  launch_chained(nb > SCAN_DIRECT ? k_scan_add<true> : k_scan_add<false>, nb, SCAN_THREADS, 0, s.stream, out, n,
                 s.grid.dScanTmp);
  CK(cudaGetLastError());
}

__global__ void k_scatter(const int4* atomK, int N, const int* start, const int* inCell, int* orig) {
  chain_wait();
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= N) return;
  orig[start[atomK[a].w] + inCell[a]] = a;
}

// Order inside a cell: ascending cell-local x coordinate u.x (pos0 of k_assign,
// so the build's staged positions are sorted along x within every cell and hence
// along every stencil row), ties by ascending atom index.  Deterministic for
// given coordinates.
__global__ void k_sort_cells(const int* start, int nRanks, int* orig, const float4* pos0, float* key) {
  chain_wait();
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nRanks) return;
  int b = start[r], e = start[r + 1];
  for (int i = b; i < e; i++) key[i] = pos0[orig[i]].x;
  for (int i = b + 1; i < e; i++) {
    int v = orig[i], j = i - 1;
    float kv = key[i];
    while (j >= b && (key[j] > kv || (key[j] == kv && orig[j] > v))) {
      orig[j + 1] = orig[j];
      key[j + 1] = key[j];
      j--;
    }
    orig[j + 1] = v;
    key[j + 1] = kv;
  }
}

// The same order for dense cells: one warp per cell; each atom's place is the
// number of atoms of the cell that precede it in (x key, atom index) order.
// Cells of more than 32 atoms are sorted by lane 0 as above.
__global__ void k_sort_cells_warp(const int* start, int nRanks, int* orig, const float4* pos0) {
  chain_wait();
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= nRanks) return;
  const int b = start[r], n = start[r + 1] - b;
  if (n <= 1) return;
  if (n > 32) {
    if (lane == 0)
      for (int i = b + 1; i < b + n; i++) {
        const int v = orig[i];
        const float kv = pos0[v].x;
        int j = i - 1;
        while (j >= b) {
          const int u = orig[j];
          const float ku = pos0[u].x;
          if (!(ku > kv || (ku == kv && u > v))) break;
          orig[j + 1] = u;
          j--;
        }
        orig[j + 1] = v;
      }
    return;
  }
  const int a = lane < n ? orig[b + lane] : 0;
  const float k = lane < n ? pos0[a].x : 0.0f;
  int place = 0;
  for (int j = 0; j < n; j++) {
    const int aj = __shfl_sync(0xffffffffu, a, j);
    const float kj = __shfl_sync(0xffffffffu, k, j);
    place += (kj < k || (kj == k && aj < a)) ? 1 : 0;
  }
  __syncwarp();
  if (lane < n) orig[b + place] = a;
}

// per slot: image cell, type, slot of the atom, and the FP32 position and charge
// (pos0 of k_assign)
__global__ void k_fill_slots(const int* orig, int N, const int4* atomK, const int* type, int4* K, uint8_t* type8,
                             int* slotOf, const float4* pos0, float4* pos4) {
  chain_wait();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= N) return;
  int a = orig[s];
  K[s] = atomK[a];
  slotOf[a] = s;
  type8[s] = (uint8_t)(type[a] - 1);
  pos4[s] = pos0[a];
}

__global__ void k_halo_table(TileGeom g, int2* tab) {
  const int t = blockIdx.x;
  for (int h = threadIdx.x; h < g.haloCells; h += blockDim.x) tab[(size_t)t * g.haloCells + h] = halo_entry(g, t, h);
}

// per tile: number of atoms and of halo atoms; global maxima in maxOut[0..1]
__global__ void k_tile_info(const int* start, TileGeom g, int* info, int* maxOut) {
  __shared__ int sum;
  int t = blockIdx.x;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  int local = 0, hx, hy, hz;
  for (int h = threadIdx.x; h < g.haloCells; h += blockDim.x) {
    int r = halo_rank(g, t, h, hx, hy, hz);
    local += start[r + 1] - start[r];
  }
  atomicAdd(&sum, local);
  __syncthreads();
  if (threadIdx.x == 0) {
    int cells = g.TB * g.TB * g.TB;
    int n = start[(t + 1) * cells] - start[t * cells];
    info[2 * t] = n;
    info[2 * t + 1] = sum;
    atomicMax(&maxOut[0], n);
    atomicMax(&maxOut[1], sum);
  }
}

// ---------------------------------------------------------------------------------
// per-step packing
// ---------------------------------------------------------------------------------

// cell-local position of each slot in units of the cell edge, u = M R/L - K, and
// the charge, from the coordinates (after a change of the box since the build)
__global__ void k_pack_mixed(const double* R, const double* __restrict__ charge, const int* orig,
                             const int4* K, int N, double scale, float4* pos4) {
  chain_wait();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= N) return;
  int a = orig[s];
  int4 k = K[s];
  float ux = (float)(R[3 * a] * scale - (double)k.x);
  float uy = (float)(R[3 * a + 1] * scale - (double)k.y);
  float uz = (float)(R[3 * a + 2] * scale - (double)k.z);
  double q = charge[a];
  pos4[s] = make_float4(ux, uy, uz, fabs(q) > 2.220446049250313e-16 ? (float)q : 0.0f);
}

// Between builds, with the box of the last build: u = u0 + (R - R0) M/L, the
// displacement since the build rounded to FP32 and scaled in FP32 (one FP64
// subtraction per coordinate instead of the FP64 M R/L - K).  The fused step
// kernel packs with the same arithmetic.
__device__ __forceinline__ float4 pack_delta(float4 p0, double dx, double dy, double dz, float scale) {
  return make_float4(fmaf(d2f(dx), scale, p0.x), fmaf(d2f(dy), scale, p0.y), fmaf(d2f(dz), scale, p0.z), p0.w);
}

__global__ void k_pack_delta(const double* R, const double* R0, const int* orig,
                             const float4* pos0, int N, float scale, float4* pos4) {
  chain_wait();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= N) return;
  int a = orig[s];
  pos4[s] = pack_delta(pos0[a], R[3 * a] - R0[3 * a], R[3 * a + 1] - R0[3 * a + 1], R[3 * a + 2] - R0[3 * a + 2],
                       scale);
}

// scaled FP64 coordinates Rs = R/L (src/EmDeeCode.f90:1228) in slot order, and their box
// fractions (the FP64 mode has no FP32 positions between builds: they take that array)
__global__ void k_pack_fp64(const double* R, const int* orig, int N, double L, double* Rs, int4* frac) {
  chain_wait();
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= N) return;
  int a = orig[s];
  const double x = R[3 * a] / L, y = R[3 * a + 1] / L, z = R[3 * a + 2] / L;
  Rs[3 * s] = x;
  Rs[3 * s + 1] = y;
  Rs[3 * s + 2] = z;
  frac[s] = make_int4(box_fraction(x), box_fraction(y), box_fraction(z), 0);
}

void device_pack(System& s) {
  Grid& g = s.grid;
  int N = s.natoms, th = 256, bl = (N + th - 1) / th;
  prof_begin(s, PK_PACK);
  if (s.precision == 1) {
    launch_chained(k_pack_fp64, bl, th, 0, s.stream, s.dR, g.dOrig, N, *s.Lbox, g.dRs64, (int4*)g.dPos4);
  } else if (*s.Lbox == s.builtL) {
    launch_chained(k_pack_delta, bl, th, 0, s.stream, s.dR, s.dR0, g.dOrig, g.dPos0, N, (float)((double)g.M / *s.Lbox), g.dPos4);
  } else {   // the box changed since the build: from the coordinates
    launch_chained(k_pack_mixed, bl, th, 0, s.stream, s.dR, s.dCharge, g.dOrig, g.dK, N, (double)g.M / *s.Lbox, g.dPos4);
  }
  CK(cudaGetLastError());
  prof_end(s, PK_PACK);
}

// ---------------------------------------------------------------------------------
// list build
// ---------------------------------------------------------------------------------


struct BuildArgs {
  TileGeom g;
  unsigned long long* fail;   // set if a list or a tile outgrew its room: the force kernels queued behind skip
  const int2* tab;
  const float4* pos4;
  const int* start;
  const int* orig;
  const int4* K;
  const uint8_t* type8;
  const int* body;
  int hasBodies;
  const uint8_t* interact;
  int ntypes;
  const int* exFirst;
  const int* exCount;
  const int* exItem;
  int hasEx;
  const double* R;
  double L;
  float lo2, hi2, loIn2, hiIn2;   // FP32 band limits, cell units^2
  double thr, thrIn;              // FP64 thresholds, scaled units^2
  int layered;                    // inner threshold below the outer one
  int minimg;                     // M == 5: a stencil cell may hold a non-minimum image
  float Mf;
  int haloCap;
  uint16_t* nb;
  int* nbCount;
  int* nbInner;
  uint16_t* selfIdx;
  int cap, tileStride;
  float invM;
  int tpa, tpaShift;   // threads per atom of the split build (a power of 2) and its log2
  int allInteract;     // every type pair interacts
  int* layout;         // out: per tile off[0..haloCells] and cst[0..haloCells-1] (stage_frame_saved)
  int* maxCount;
};

__device__ __forceinline__ bool excluded(const BuildArgs& A, int a, int b) {
  int f = A.exFirst[a], n = A.exCount[a];
  for (int k = 0; k < n; k++) {
    int v = A.exItem[f + k] - 1;
    if (v == b) return true;
    if (v > b) break;
  }
  return false;
}

// Blocks of the thread-per-atom build: at most BUILD_THREADS threads, each taking
// the same number of the tile's atoms (tile_threads); without a tuned count, as few
// rounds as blocks of BUILD_THREADS_RULE threads allow.
static const int BUILD_THREADS = 512;
static const int BUILD_THREADS_RULE = 256;
static const int BUILD_THREADS_SPLIT = 1024;  // split build: several threads per tile atom
enum BuildMode : int { BUILD_ONE = 0, BUILD_SPLIT, BUILD_WARP, BUILD_SPARSE };
static const int BUILD_PAD = 4;               // halo entries past the last one, far away

// List layout: for tile t, chunk c (8 entries) and tile-local atom li, the
// entries 8c..8c+7 of atom li are 16 contiguous bytes at
//   nb + ((t * capC + c) * tileStride + li) * 8
// so a warp reads one chunk of 32 consecutive atoms with one 512-byte access.
// Unused entries of the last chunk hold the sentinel halo index haloCap.
__device__ __forceinline__ size_t nb_index(int t, int capC, int tileStride, int li, int n) {
  return (((size_t)t * capC + (n >> 3)) * tileStride + li) * 8 + (n & 7);
}

// Every atom scans the 25 rows of 5 stencil cells around it, each over the run of cells
// that can hold a neighbor at the row's distance.  Candidates go in segments of up to
// 32: four loads at a time, the bits of r^2 minus the bits of the lower band limit, whose
// sign is shifted into the segment's mask (10 instructions a candidate, no branch; the
// unsigned minimum of the differences tells whether any candidate lies in the band and
// the segment needs the FP64 test).  The mask's bits are then taken in order, and a
// thread that owns its atom stores 8 entries at a time.  The kernel is bound by
// instruction issue.  1M Lennard-Jones atoms: 630 -> 535 us against candidates that went
// through their tests and a 2-byte store one by one (L2 sectors 122 -> 26 M).
// The list order is (row, halo index), a function of the coordinates.
// BUILD_SPLIT: A.tpa threads per atom, which take consecutive rows: a first sweep counts,
// the group's prefix sums give each thread its output positions, a second writes (in the
// same order as one thread).
// BUILD_WARP: a warp per atom, its lanes side by side over each row's candidates, the
// accepted ones placed by ballots (the same order again): for dense cells, whose rows
// fill the lanes (4096 water molecules, 17 atoms per cell: 262
// us with 8 threads per atom, 130 us so).
// GENERAL: several atom types, bodies, exclusions or layered lists; MINIMG: M = 5.
// BUILD_SPARSE: BUILD_ONE for boxes with more tiles than atoms, which are bound by their
// blocks of 64 threads in flight: 64 registers (1000 atoms in 244,000 tiles, a rebuild 2475 us
// with 80, 2223 so).
// Register budget: BUILD_ONE BUILD_MAXNREG (1,048,576 atoms: 565 us with 80, 569 with 72, and
// the 72 led the tuner astray more often), the others 64, in blocks of up to 1024 threads.
#ifndef BUILD_MAXNREG
#define BUILD_MAXNREG 80
#endif
template <bool GENERAL, bool MINIMG, int MODE>
__global__ void __maxnreg__(MODE == BUILD_ONE ? BUILD_MAXNREG : 64) k_build(BuildArgs A) {
  chain_wait();
  constexpr bool SPLIT = MODE == BUILD_SPLIT;
  extern __shared__ __align__(16) unsigned char sraw[];
  __shared__ int ws[33];
  const TileGeom g = A.g;
  const int t = blockIdx.x, cells = g.TB * g.TB * g.TB;
  // shared memory: the staged halo (and the entries that a segment of four may read
  // past its end), the halo cell offsets, then for the general variant the halo atoms'
  // keys (their body, or with exclusions the atom), the type filter and their types
  float4* hpos = (float4*)sraw;
  int* off = (int*)(hpos + A.haloCap + BUILD_PAD);
  int* hkey = off + g.haloCells + 1;
  const bool single = !GENERAL || A.allInteract;
  uint8_t* sinter = (uint8_t*)(hkey + (GENERAL ? A.haloCap : 0));
  uint8_t* htype = sinter + A.ntypes * A.ntypes;
  for (int k = threadIdx.x; k < A.ntypes * A.ntypes; k += blockDim.x) sinter[k] = A.interact[k];
  // the layout, saved for the force kernels until the next build: first slots
  // straight to global memory, cell sizes scanned into off
  int* lay = A.layout + (size_t)t * (2 * g.haloCells + 1);
  {
    const int2* tt = A.tab + (size_t)t * g.haloCells;
    for (int h = threadIdx.x; h < g.haloCells; h += blockDim.x) {
      const int r = tt[h].x, b = A.start[r];
      lay[g.haloCells + 1 + h] = b;
      off[h] = A.start[r + 1] - b;
    }
    __syncthreads();
    const int total = block_exclusive_scan<8>(off, g.haloCells, ws);
    if (threadIdx.x == 0) off[g.haloCells] = total;
    __syncthreads();
  }
  const int haloCount = off[g.haloCells];
  const int tb = A.start[t * cells], te = A.start[(t + 1) * cells];
  // sizes taken from the previous build: a tile or halo that outgrew them is
  // reported (the host re-sizes and builds again) before anything is staged
  if (te - tb > A.tileStride || haloCount > A.haloCap) {
    if (threadIdx.x == 0) {
      atomicOr(A.maxCount + 1, 1);
      *A.fail = 1ull;
    }
    return;
  }
  for (int h = threadIdx.x; h <= g.haloCells; h += blockDim.x) lay[h] = off[h];
  if (te == tb) return;   // no lists, but the force kernels stage the tile's halo
  // every thread reads back only the first slots it wrote itself
  for (int h = threadIdx.x; h < g.haloCells; h += blockDim.x)
    mark_halo_cell(hpos, h, off[h], off[h + 1], lay[g.haloCells + 1 + h]);
  __syncthreads();
  const bool filterByAtom = GENERAL && (A.hasBodies || A.hasEx);
  stage_marked(g, haloCount, A.pos4, hpos, filterByAtom ? hkey : nullptr, single ? (uint8_t*)nullptr : htype, A.type8);
  if (threadIdx.x < BUILD_PAD) hpos[haloCount + threadIdx.x] = make_float4(1e9f, 1e9f, 1e9f, 0.f);
  if (filterByAtom)   // every thread reads back only the slots it wrote itself
    for (int k = threadIdx.x; k < haloCount; k += blockDim.x) {
      const int a = A.orig[hkey[k]];
      hkey[k] = A.hasEx ? a : A.body[a];
    }
  __syncthreads();
  // slot of halo index q (for the rare band test): its cell is looked up
  auto slot_of = [&](int q) {
    int lo = 0, hi = g.haloCells - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (off[mid] <= q) lo = mid;
      else hi = mid - 1;
    }
    return lay[g.haloCells + 1 + lo] + (q - off[lo]);
  };
  const bool none = A.ntypes == 1 && !sinter[0];   // the only type pair does not interact: empty lists
  const bool layered = GENERAL && A.layered;
  const int HW = g.HW, capC = A.cap >> 3, chunkStride = A.tileStride * 8;
  const int loBits = __float_as_int(A.lo2);
  const unsigned band = (unsigned)(__float_as_int(A.hi2) - loBits);
  const int tpa = SPLIT ? A.tpa : 1, sub = SPLIT ? (int)(threadIdx.x & (tpa - 1)) : 0;
  const int tshift = SPLIT ? A.tpaShift : 0;
  const unsigned gmask = (0xFFFFFFFFu >> (32 - tpa)) << ((threadIdx.x & 31) & ~(tpa - 1));
  int longest = 0;
  const int li0 = MODE == BUILD_WARP ? threadIdx.x >> 5 : threadIdx.x >> tshift;
  const int liStep = MODE == BUILD_WARP ? blockDim.x >> 5 : blockDim.x >> tshift;
  const bool writer = MODE == BUILD_WARP ? (threadIdx.x & 31) == 0 : sub == 0;
  for (int li = li0; li < te - tb; li += liStep) {
    const int si = tb + li;
    const int rank = A.K[si].w, lr = rank - t * cells;
    const int hcx = lr % g.TB + 2, hcy = (lr / g.TB) % g.TB + 2, hcz = lr / (g.TB * g.TB) + 2;
    const int myq = off[hcx + HW * (hcy + HW * hcz)] + (si - A.start[rank]);
    if (writer) A.selfIdx[si] = (uint16_t)myq;
    const float4 pi = hpos[myq];
    const int ai = A.orig[si], ti = single ? 0 : A.type8[si];
    const int bi = filterByAtom && A.hasBodies ? A.body[ai] : -1;
    // the first exclusions of the atom (lists are ascending; -1: none)
    constexpr int EX = 4;
    int ex[EX], nEx = 0;
    if (GENERAL) {
      nEx = filterByAtom && A.hasEx ? A.exCount[ai] : 0;
#pragma unroll
      for (int k = 0; k < EX; k++) ex[k] = k < nEx ? A.exItem[A.exFirst[ai] + k] - 1 : -1;
    }
    auto allowed = [&](int q) {
      if (!single && !sinter[ti * A.ntypes + htype[q]]) return false;
      if (filterByAtom) {
        const int key = hkey[q];
        if (A.hasBodies && (A.hasEx ? A.body[key] : key) == bi) return false;
        if (nEx > 0) {
#pragma unroll
          for (int k = 0; k < EX; k++)
            if (key == ex[k]) return false;
          if (nEx > EX && excluded(A, ai, key)) return false;
        }
      }
      return true;
    };
    auto dist2 = [&](int q) {
      const float4 pj = hpos[q];
      float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
      if (MINIMG) {
        dx -= A.Mf * rintf(dx * A.invM);
        dy -= A.Mf * rintf(dy * A.invM);
        dz -= A.Mf * rintf(dz * A.invM);
      }
      return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    };
    // window [q0, q1) of halo indices of stencil row (rz, ry) (the 5 cells of a row are
    // consecutive): with rho the distance from atom i to the row's y-z cross-section, only
    // cells that reach |x_j - x_i| < sqrt(hi2 - rho^2) can hold a neighbor; a 1e-3 cell
    // margin covers the FP32 rounding of the frame and the approximate square root (cell
    // hx spans [hx - C, hx - C + 1] in the frame).
    auto window = [&](int rz, int ry, int& q0, int& q1) {
      const int hz = hcz + rz, hy = hcy + ry, h0 = (hcx - 2) + HW * (hy + HW * hz);
      int c0 = 0, c1 = 4;
      if (!MINIMG) {
        const float y0 = (float)(hy - g.C), z0 = (float)(hz - g.C);
        const float dy = fmaxf(fmaxf(y0 - pi.y, pi.y - (y0 + 1.0f)) - 1e-3f, 0.0f);
        const float dz = fmaxf(fmaxf(z0 - pi.z, pi.z - (z0 + 1.0f)) - 1e-3f, 0.0f);
        const float rem = A.hi2 - fmaf(dy, dy, dz * dz);
        if (rem <= 0.0f) {
          q0 = q1 = 0;
          return;
        }
        const float w = fmaf(rem, rsqrtf(rem), 1e-3f);
        const int shift = g.C - (hcx - 2);
        c0 = min(max((int)floorf(pi.x - w) + shift, 0), 4);
        c1 = min(max((int)floorf(pi.x + w) + shift, 0), 4);
      }
      q0 = off[h0 + c0];
      q1 = off[h0 + c1 + 1];
    };
    // accepted candidates of q, q + 1, ... (at most 32, up to q1): bit 31 - j is q + j
    auto segment = [&](int q, int q1) {
      const int len = min(32, q1 - q);
      unsigned m = 0, near = 0xFFFFFFFFu;
      for (int u = 0; u < len; u += 4)
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const int d = __float_as_int(dist2(q + u + v)) - loBits;
          m = __funnelshift_l((unsigned)d, m, 1);
          near = min(near, (unsigned)d);
        }
      m <<= (32 - ((len + 3) & ~3));
      if (near < band)   // some candidate lies within the band: the FP64 test decides it
        for (int j = 0; j < len; j++) {
          const unsigned d = (unsigned)(__float_as_int(dist2(q + j)) - loBits);
          if (d < band && exact_inside(A.R, A.L, ai, A.orig[slot_of(q + j)], A.thr)) m |= 0x80000000u >> j;
        }
      m &= (unsigned)((int)0x80000000 >> (len - 1));                                  // candidates before q1
      if ((unsigned)(myq - q) < 32u) m &= ~(0x80000000u >> (myq - q));                // not the atom itself
      return m;
    };
    // f(q) of every accepted neighbor of a row; inner / outer entries of layered lists
    // in the sweep they belong to
    auto row = [&](int rz, int ry, auto&& f) {
      int q0, q1;
      window(rz, ry, q0, q1);
      for (int q = q0; q < q1; q += 32) {
        unsigned m = segment(q, q1);
        while (m) {
          const int j = __clz(m);
          m &= 0x7FFFFFFFu >> j;
          if (GENERAL && !allowed(q + j)) continue;
          f(q + j);
        }
      }
    };
    auto inside = [&](int q) {
      const float r2 = dist2(q);
      return r2 < A.loIn2 || (r2 < A.hiIn2 && exact_inside(A.R, A.L, ai, A.orig[slot_of(q)], A.thrIn));
    };
    int n = 0, nIn = 0;
    if (MODE == BUILD_WARP) {
      constexpr unsigned FULL = 0xffffffffu;
      const int lane = threadIdx.x & 31;
      int w0 = 0, w1 = 0;   // window of row `lane`
      if (lane < 25 && !none) window(lane / 5 - 2, lane % 5 - 2, w0, w1);
      uint16_t* myList = A.nb + ((size_t)t * capC * A.tileStride + li) * 8;
      for (int pass = 0; pass <= (layered ? 1 : 0); pass++) {
        for (int r = 0; r < 25; r++) {
          const int q1 = __shfl_sync(FULL, w1, r);
          for (int q = __shfl_sync(FULL, w0, r) + lane; q - lane < q1; q += 32) {
            const int d = __float_as_int(dist2(min(q, haloCount - 1))) - loBits;
            bool acc = q < q1 && d < 0 && q != myq;
            const bool near = q < q1 && (unsigned)d < band;
            if (__any_sync(FULL, near) && near) acc = exact_inside(A.R, A.L, ai, A.orig[slot_of(q)], A.thr);
            if (GENERAL && acc) acc = allowed(q) && (!layered || inside(q) == (pass == 0));
            const unsigned m = __ballot_sync(FULL, acc);
            const int at = n + __popc(m & ((1u << lane) - 1u));
            if (acc && at < A.cap) myList[(at >> 3) * chunkStride + (at & 7)] = (uint16_t)q;
            n += __popc(m);
          }
        }
        if (pass == 0) nIn = n;
      }
      // sentinel padding of the last chunk
      if ((n & 7) && lane < 8 - (n & 7) && n + lane < A.cap)
        myList[((n + lane) >> 3) * chunkStride + ((n + lane) & 7)] = (uint16_t)A.haloCap;
    } else if (MODE == BUILD_ONE || MODE == BUILD_SPARSE) {
      // rows in the order dz = -2..2 (outer), dy = -2..2 (inner); layered lists take the
      // inner entries in a first sweep and the outer ones in a second.  The last 8 entries
      // sit in four registers until they are complete.
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      uint4* out = reinterpret_cast<uint4*>(A.nb) + ((size_t)t * capC * A.tileStride + li);
      auto push = [&](int q) {
        w.x = __funnelshift_r(w.x, w.y, 16);
        w.y = __funnelshift_r(w.y, w.z, 16);
        w.z = __funnelshift_r(w.z, w.w, 16);
        w.w = __funnelshift_r(w.w, (unsigned)q, 16);
        n++;
        if ((n & 7) == 0) {
          if (n <= A.cap) *out = w;
          out += A.tileStride;
        }
      };
      for (int pass = 0; pass <= (layered ? 1 : 0) && !none; pass++) {
        for (int rz = -2; rz <= 2; rz++)
          for (int ry = -2; ry <= 2; ry++)
            row(rz, ry, [&](int q) {
              if (layered && inside(q) == (pass == 1)) return;
              push(q);
            });
        if (pass == 0) nIn = n;
      }
      const int count = n;
      while (n & 7) push(A.haloCap);   // sentinel padding of the last chunk
      n = count;
    } else {
      uint16_t* myList = A.nb + ((size_t)t * capC * A.tileStride + li) * 8;
      auto put = [&](int k, int q) {
        if (k < A.cap) myList[(k >> 3) * chunkStride + (k & 7)] = (uint16_t)q;
      };
      const int r0 = 25 * sub >> tshift, r1 = 25 * (sub + 1) >> tshift;
      int cIn = 0, cOut = 0;
      if (!none)
        for (int r = r0; r < r1; r++) {
          if (GENERAL) {
            row(r / 5 - 2, r % 5 - 2, [&](int q) {
              if (!layered || inside(q)) cIn++;
              else cOut++;
            });
          } else {   // nothing to filter: the masks' bits are the count
            int q0, q1;
            window(r / 5 - 2, r % 5 - 2, q0, q1);
            for (int q = q0; q < q1; q += 32) cIn += __popc(segment(q, q1));
          }
        }
      // exclusive prefix sums over the group's threads, in sub order
      int pIn = cIn, pOut = cOut;
      for (int o = 1; o < tpa; o <<= 1) {
        const int yIn = __shfl_up_sync(gmask, pIn, o), yOut = __shfl_up_sync(gmask, pOut, o);
        if (sub >= o) {
          pIn += yIn;
          pOut += yOut;
        }
      }
      const int totIn = __shfl_sync(gmask, pIn, tpa - 1, tpa), totOut = __shfl_sync(gmask, pOut, tpa - 1, tpa);
      int kIn = pIn - cIn, kOut = totIn + pOut - cOut;
      if (!none)
        for (int r = r0; r < r1; r++)
          row(r / 5 - 2, r % 5 - 2, [&](int q) {
            if (!layered || inside(q)) put(kIn++, q);
            else put(kOut++, q);
          });
      n = totIn + totOut;
      nIn = totIn;
      // sentinel padding of the last chunk
      if (sub == 0)
        for (int k = n; (k & 7) && k < A.cap; k++) put(k, A.haloCap);
    }
    if (writer) {
      A.nbCount[si] = n;
      A.nbInner[si] = nIn;
    }
    longest = max(longest, n);
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  if ((threadIdx.x & 31) == 0 && longest > 0) {
    atomicMax(A.maxCount, longest);
    if (longest > A.cap) *A.fail = 1ull;
  }
}

template <typename T>
static void grow(T*& p, size_t& have, size_t need) {
  if (have >= need) return;
  CK(cudaFree(p));
  CK(cudaMalloc(&p, sizeof(T) * need));
  have = need;
}


double expected_entries(const System& s) {
  const double L = *s.Lbox;
  return s.natoms / (L * L * L) * 4.18879020478639 * s.xRcSq * s.xRc;
}

int split_threads(const System& s, double entries, int maxThreads) {
  int tpa = 1;
  while (tpa < 32 && (double)s.natoms * tpa * 2 <= 152.0 * 2048 && s.grid.tileAtoms * tpa * 2 <= maxThreads &&
         entries / (tpa * 2) >= 8.0)
    tpa *= 2;
  return tpa;
}

// threads per atom of the build (its candidates are about twice the entries); 32 is the
// warp-per-atom kernel, the rule's choice where a row of 5 cells fills the lanes
static int build_tpa(const System& s) {
  if (s.buildTpa > 0) return s.buildTpa;
  const Grid& g = s.grid;
  if (s.natoms >= 8.0 * g.M * g.M * g.M) return 32;
  return std::min(16, split_threads(s, 2.0 * expected_entries(s), BUILD_THREADS_SPLIT));
}

int build_block_threads(const System& s) {
  const Grid& g = s.grid;
  const int least = halo_min_threads(make_geom(g.M, g.TB)), tpa = build_tpa(s);
  if (tpa > 1) return std::max(least, std::min(BUILD_THREADS_SPLIT, (g.tileAtoms * tpa + 31) / 32 * 32));
  return std::max(least, s.buildThreads > 0 ? std::min(s.buildThreads, BUILD_THREADS)
                                            : tile_threads(g.tileAtoms, 0, BUILD_THREADS_RULE));
}

// the general build variant: several types, bodies, exclusions or layered lists
static bool build_general(const System& s) {
  return s.ntypes > 1 || s.nbodies > 0 || s.hasExclusions || s.xInRcSq < s.xRcSq;
}

static size_t build_smem(const Grid& g, int ntypes, bool general) {
  return (size_t)(g.maxHalo + BUILD_PAD) * (sizeof(float4) + (general ? sizeof(int) + 1 : 0)) +
         sizeof(int) * (g.haloCells + 1) + (size_t)ntypes * ntypes + 16;
}

// Tile edge: EMDEE_TILE, else the system's tuned edge (tileOverride), else a rule: by the
// atoms per cell, smaller where the tiles would not give every SM two blocks (two-level
// lists, whose launches have one thread per atom, keep the larger tiles).
static int rule_tile(System& s, int M, double perCell) {
  int tb = std::min(perCell <= 4.0 ? 4 : perCell <= 9.0 ? 3 : perCell <= 24.0 ? 2 : 1, M);
  while (tb > 1 && !two_level_active(s)) {
    const int nT = (M + tb - 1) / tb;
    if (nT * nT * nT >= 2 * 152) break;
    tb--;
  }
  return tb;
}

static int choose_tile(System& s, int M, double perCell) {
  if (const char* e = getenv("EMDEE_TILE")) {
    int tb = atoi(e);
    if (tb >= 1 && tb <= 6) return std::min(tb, M);
  }
  if (s.tileOverride > 0) return std::min(s.tileOverride, M);
  return rule_tile(s, M, perCell);
}

// Tile edge, threads per atom and block sizes tuned on the system itself at its first
// build (mixed precision, EMDEE_TILE unset).  For each edge from min(rule - 1, 3)
// (in small systems, where few large tiles leave most SMs idle, from the least that gives a
// tile an atom and no SM more than 64 tiles) to 6 cells (the rule's edge always among them) a first build sizes the
// tiles; then the list build and the pair kernel are timed with CUDA events (the faster of two
// launches, after a warm-up launch of the pair kernel), each after a pass that moves the
// memory traffic of an integration step, at the rule's shape and, on the edges whose cost so
// is within 1.5 of the least, at block sizes from 64 to 512 threads (threads loop over the
// tile's atoms in rounds; the best size balances the rounds of typical tiles against
// residency) and at 2 to 32 threads per atom.  The cost of an
// edge is its fastest pair launch plus a seventh of its fastest build (a rebuild
// every ~7 steps, typical of a liquid with the reference's skin).  The rule's edge
// and block sizes stay unless another choice is more than 5 % cheaper.  The choice
// is kept per (cells per edge, atoms per cell to 1/8, types, model variant) for the
// process, so systems of the same shape use the same tiles and blocks and give
// bit-identical results.
// Reads and rewrites R and P with their own bits and reads F (zero is 0 at run
// time): the memory traffic of an integration step, so that timed tuning launches
// meet the L2 contents a step leaves.
__global__ void k_touch(double* __restrict__ R, double* __restrict__ P, const double* __restrict__ F, long n,
                        long long zero) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const long long f = __double_as_longlong(F[i]) & zero;
    R[i] = __longlong_as_double(__double_as_longlong(R[i]) ^ f);
    P[i] = __longlong_as_double(__double_as_longlong(P[i]) ^ f);
  }
}

struct TileChoice {
  int tb, buildTpa, buildThreads, pairTpa, pairThreads;
};
static std::vector<std::pair<std::vector<long>, TileChoice>> g_tileTuned;

static void use_choice(System& s, const TileChoice& c) {
  s.tileOverride = c.tb;
  s.buildTpa = c.buildTpa;
  s.buildThreads = c.buildThreads;
  s.pairTpa = c.pairTpa;
  s.pairThreads = c.pairThreads;
}

void device_tune_tile(System& s, bool ljOnly, void (*pair)(System&)) {
  if (getenv("EMDEE_TILE") || (getenv("EMDEE_AUTOTUNE") && !strcmp(getenv("EMDEE_AUTOTUNE"), "0"))) return;
  const double L = *s.Lbox;
  const int M = std::max((int)std::floor(NDIV * L / s.xRc), 2 * NDIV + 1);
  const double perCell = (double)s.natoms / ((double)M * M * M);
  const std::vector<long> key = {M, (long)std::lround(perCell * 8.0), s.ntypes, ljOnly ? 1 : 0, s.nbodies > 0,
                                 s.hasExclusions ? 1 : 0};
  for (const auto& e : g_tileTuned)
    if (e.first == key) {
      use_choice(s, e.second);
      return;
    }
  const int rule = rule_tile(s, M, perCell);
  const bool chainReq = s.keChainReq;   // no kinetic pass queued behind the timed pair launches
  s.keChainReq = false;
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  auto timed = [&](auto&& f) {
    double best = 1e30;
    for (int k = 0; k < 2; k++) {
      if (!s.phaseShared) {   // (shared R and P may belong to another system's stream)
        k_touch<<<4 * 152, 256, 0, s.stream>>>(s.dR, s.dP, s.F(), 3L * s.natoms, 0LL);
        CK(cudaGetLastError());
        s.prof.total++;
      }
      CK(cudaEventRecord(e0, s.stream));
      f();
      CK(cudaEventRecord(e1, s.stream));
      CK(cudaEventSynchronize(e1));
      float ms = 0.f;
      CK(cudaEventElapsedTime(&ms, e0, e1));
      best = std::min(best, (double)ms);
    }
    return best;
  };
  const bool log = getenv("EMDEE_TUNE_LOG") != nullptr;
  auto timed_build = [&] {
    const double ms = timed([&] { device_build_lists(s); });
    if (log)
      fprintf(stderr, "  edge %d build, %d per atom, %d threads: %.1f us\n", s.tileOverride, s.buildTpa,
              build_block_threads(s), 1e3 * ms);
    return ms;
  };
  auto timed_pair = [&] {
    pair(s);   // warm-up
    const double ms = timed([&] { pair(s); });
    if (log)
      fprintf(stderr, "  edge %d pair, %d per atom, %d threads: %.1f us\n", s.tileOverride, s.pairTpa,
              pair_block_threads(s), 1e3 * ms);
    return ms;
  };
  // the rule's shape on every edge
  struct Edge {
    int tb, tileAtoms;
    double build, pair;
    double cost() const { return pair + build / 7.0; }
  };
  std::vector<Edge> edges;
  double bestRule = 1e30;
  const bool small = s.natoms < 152 * 1024;   // fewer atoms than half the GPU's threads
  int lowest = std::max(1, std::min(rule - 1, 3));
  if (small) {   // the least edge that gives a tile an atom, and no SM more than 64 tiles
    int tb = 1;
    auto tiles = [&](int e) { return std::pow((M + e - 1) / e, 3.0); };
    while (tb < lowest && (perCell * (tb * tb * tb) < 1.0 || tiles(tb) > 64 * 152)) tb++;
    lowest = tb;
  }
  for (int tb = lowest; tb <= std::min(6, M); tb++) {
    use_choice(s, TileChoice{tb, 0, 0, 0, 0});
    device_build_lists(s);   // sizes the tiles of this edge
    if (s.grid.TB != tb) continue;   // did not fit (halo or shared memory): the build shrank the edge
    edges.push_back(Edge{tb, s.grid.tileAtoms, timed_build(), timed_pair()});
    bestRule = std::min(bestRule, edges.back().cost());
  }
  double best = 1e30, ruleCost = 1e30;
  TileChoice choice = {rule, 0, 0, 0, 0};
  for (const Edge& e : edges) {
    const int tb = e.tb;
    if (tb == rule) ruleCost = e.cost();
    double msBuild = e.build, msPair = e.pair;
    TileChoice here = {tb, 0, 0, 0, 0};
    // other shapes have gained up to 1.3 times on the rule's
    if (e.cost() <= 1.5 * bestRule) {
      use_choice(s, here);
      device_build_lists(s);
      // (threads per atom, threads per block): with one thread per atom 64 to 256 threads
      // in steps of 32 and 320 to 512 in steps of 64, from the least the halo scans need up to the
      // largest tile, and the splits that the GPU has threads and the lists entries for
      const int thMin = halo_min_threads(make_geom(s.grid.M, tb)), thMax = (s.grid.tileAtoms + 31) / 32 * 32;
      const double entries = expected_entries(s);
      std::vector<std::pair<int, int>> shapes;
      for (int th = 64; th <= 512; th += th < 256 ? 32 : 64)
        if (th >= thMin && (th <= thMax || (th == 64 && entries >= 2.0))) shapes.push_back({1, th});
      for (int tpa = 2; tpa <= 32; tpa *= 2)
        if ((double)s.natoms * tpa <= 152.0 * 2048 * 2 && entries >= tpa) shapes.push_back({tpa, 0});
      for (const auto& sh : shapes) {
        s.buildTpa = sh.first;
        s.buildThreads = sh.second;
        const double ms = timed_build();
        if (ms < msBuild) {
          msBuild = ms;
          here.buildTpa = sh.first;
          here.buildThreads = sh.second;
        }
      }
      for (const auto& sh : shapes) {
        s.pairTpa = sh.first;
        s.pairThreads = sh.second;
        const double ms = timed_pair();
        if (ms < msPair) {
          msPair = ms;
          here.pairTpa = sh.first;
          here.pairThreads = sh.second;
        }
      }
    }
    const double cost = msPair + msBuild / 7.0;
    if (log)
      fprintf(stderr, "tile edge %d (at most %d atoms per tile): cost %.1f us, build %d x %d, pair %d x %d\n", tb,
              e.tileAtoms, 1e3 * cost, here.buildTpa, here.buildThreads, here.pairTpa, here.pairThreads);
    if (cost < best) {
      best = cost;
      choice = here;
    }
  }
  if (ruleCost < 1e30 && best > 0.95 * ruleCost) choice = {rule, 0, 0, 0, 0};
  CK(cudaEventDestroy(e0));
  CK(cudaEventDestroy(e1));
  use_choice(s, choice);
  s.r0Valid = false;   // the system's own first build comes next, with the chosen edge
  s.keChainReq = chainReq;
  g_tileTuned.push_back({key, choice});
}

void build_flags(System& s) {
  CK(cudaMemcpyAsync(s.hFlags + 2, s.grid.dTileInfo + 2 * s.grid.nTiles + 2, 2 * sizeof(int), cudaMemcpyDeviceToHost,
                     s.stream));
}

// src/neighbor_lists.f90:175-195 (build part) and 199-300.  reuse: keep the tile
// sizes of the previous build when the cell geometry is unchanged (no per-tile
// count pass and no synchronisation for it); returns false if a tile outgrew them.
// defer: returns without waiting for the build (build_settled).
static bool build_lists(System& s, bool reuse, bool defer) {
  Grid& g = s.grid;
  GridCaps& c = g.caps;
  const int N = s.natoms;
  const double L = *s.Lbox;
  // two-level lists: this build writes the outer lists, of radius rc + skin + delta
  const bool outer = two_level_active(s);
  const double delta = outer ? outer_delta(s) : 0.0;
  const double xRc = s.xRc + delta, xRcSq = xRc * xRc;
  uint16_t*& nbList = outer ? g.dNbOuter : g.dNb;
  size_t& nbCap = outer ? c.nbOuter : c.nb;
  int& cap = outer ? g.capOuter : g.cap;
  int M = (int)std::floor(NDIV * L / xRc);
  M = std::max(M, 2 * NDIV + 1);
  double perCell = (double)N / ((double)M * M * M);
  int TB = choose_tile(s, M, perCell);
  reuse = reuse && g.M == M && g.TB == TB && g.maxHalo > 0 && g.tileStride > 0 && c.atoms >= (size_t)N;
  // the entries past the halo (BUILD_PAD, one of them a sentinel) come on top
  size_t smemLimit = 200 * 1024 + (BUILD_PAD - 1) * (sizeof(float4) + sizeof(int) + 1);
  for (;;) {
    TileGeom geo = make_geom(M, TB);
    g.M = M;
    g.TB = TB;
    g.nT = geo.nT;
    g.nTiles = geo.nT * geo.nT * geo.nT;
    g.nRanks = g.nTiles * TB * TB * TB;
    g.haloCells = geo.haloCells;
    if (c.ranks < (size_t)g.nRanks + 1) {   // zero between builds (k_scan_local)
      grow(g.dCount, c.ranks, (size_t)g.nRanks + 1);
      CK(cudaMemsetAsync(g.dCount, 0, sizeof(int) * c.ranks, s.stream));
    }
    if (!g.dStart || c.scan < (size_t)g.nRanks + 1) {
      CK(cudaFree(g.dStart));
      CK(cudaFree(g.dScanTmp));
      CK(cudaMalloc(&g.dStart, sizeof(int) * (g.nRanks + 1)));
      CK(cudaMalloc(&g.dScanTmp, sizeof(int) * ((g.nRanks + SCAN_TILE) / SCAN_TILE + 1)));
      c.scan = (size_t)g.nRanks + 1;
    }
    if (c.atoms < (size_t)N) {
      CK(cudaFree(g.dOrig)); CK(cudaFree(g.dK)); CK(cudaFree(g.dAtomK)); CK(cudaFree(g.dPos4));
      CK(cudaFree(g.dType8)); CK(cudaFree(g.dRs64)); CK(cudaFree(g.dNbCount)); CK(cudaFree(g.dNbInner));
      CK(cudaFree(g.dSelf));
      CK(cudaFree(g.dSlotOf));
      CK(cudaFree(g.dPos0));
      CK(cudaFree(g.dKeyX));
      CK(cudaMalloc(&g.dKeyX, sizeof(float) * N));
      CK(cudaMalloc(&g.dSlotOf, sizeof(int) * N));
      CK(cudaMalloc(&g.dPos0, sizeof(float4) * N));
      CK(cudaMalloc(&g.dOrig, sizeof(int) * N));
      CK(cudaMalloc(&g.dK, sizeof(int4) * N));
      CK(cudaMalloc(&g.dAtomK, sizeof(int4) * N));
      CK(cudaMalloc(&g.dPos4, sizeof(float4) * N));
      CK(cudaMalloc(&g.dType8, N));
      CK(cudaMalloc(&g.dRs64, sizeof(double) * 3 * N));
      CK(cudaMalloc(&g.dNbCount, sizeof(int) * N));
      CK(cudaMalloc(&g.dNbInner, sizeof(int) * N));
      CK(cudaMalloc(&g.dSelf, sizeof(uint16_t) * N));
      c.atoms = N;
    }
    if (c.tiles < (size_t)g.nTiles) {
      CK(cudaFree(g.dTileInfo));
      CK(cudaMalloc(&g.dTileInfo, sizeof(int) * (2 * g.nTiles + 6)));
      c.tiles = g.nTiles;
    }
    int th = 256, bl = (N + th - 1) / th;
    int* dMax = g.dTileInfo + 2 * g.nTiles;
    s.prof.total += reuse ? 6 : 7;   // assign, 2 scan phases, scatter, sort, fill (, tile info)
    // the slot array holds each atom's place in its cell until k_fill_slots
    launch_chained(k_assign, bl, th, 0, s.stream, s.dR, s.dCharge, N, (double)M / L, geo, g.dAtomK, g.dCount, g.dSlotOf,
                                      g.dPos0, s.dR0, dMax, (unsigned long long*)(s.dResult + BUILD_FAILED));
    CK(cudaGetLastError());
    device_scan(s, g.dCount, g.dStart, g.nRanks);
    launch_chained(k_scatter, bl, th, 0, s.stream, g.dAtomK, N, g.dStart, g.dSlotOf, g.dOrig);
    if (perCell >= 8.0)   // dense cells: a warp per cell
      launch_chained(k_sort_cells_warp, (g.nRanks + 7) / 8, 256, 0, s.stream, g.dStart, g.nRanks, g.dOrig, g.dPos0);
    else
      launch_chained(k_sort_cells, (g.nRanks + 255) / 256, 256, 0, s.stream, g.dStart, g.nRanks, g.dOrig, g.dPos0, g.dKeyX);
    launch_chained(k_fill_slots, bl, th, 0, s.stream, g.dOrig, N, g.dAtomK, s.dType, g.dK, g.dType8, g.dSlotOf, g.dPos0,
                                          g.dPos4);
    if (reuse) break;
    k_tile_info<<<g.nTiles, 128, 0, s.stream>>>(g.dStart, geo, g.dTileInfo, dMax);
    CK(cudaGetLastError());
    int hmax[2];
    CK(cudaMemcpyAsync(hmax, dMax, sizeof(int) * 2, cudaMemcpyDeviceToHost, s.stream));
    CK(cudaStreamSynchronize(s.stream));
    g.tileAtoms = hmax[0];
    g.tileStride = hmax[0] > 24 ? (hmax[0] + 31) / 32 * 32 : std::max(8, (hmax[0] + 7) / 8 * 8);
    g.maxHalo = hmax[1];
    size_t smem = build_smem(g, s.ntypes, build_general(s));
    size_t smem64 = (size_t)(g.maxHalo + 1) * (4 * sizeof(double) + sizeof(int4) + 1) + 64;
    if ((g.maxHalo > 65534 || smem > smemLimit || (s.precision == 1 && smem64 > smemLimit)) && TB > 1) {
      TB--;
      continue;
    }
    if (g.maxHalo > 65534 || smem > smemLimit) fatal("neighbor list build", "too many atoms around a cell");
    break;
  }
  TileGeom geo = make_geom(g.M, g.TB);
  if (g.tabM != g.M || g.tabTB != g.TB) {   // the halo table depends on the geometry only
    size_t need = (size_t)g.nTiles * g.haloCells;
    if (g.haloTabCap < need) {
      CK(cudaFree(g.dHaloTab));
      CK(cudaMalloc(&g.dHaloTab, sizeof(int2) * need));
      g.haloTabCap = need;
    }
    k_halo_table<<<g.nTiles, 128, 0, s.stream>>>(geo, g.dHaloTab);
    CK(cudaGetLastError());
    s.prof.total++;
    g.tabM = g.M;
    g.tabTB = g.TB;
  }
  // neighbor capacity: expected full-list count with margin, grown on overflow
  if (cap == 0) {
    double rho = N / (L * L * L);
    double expected = rho * 4.18879020478639 * xRcSq * xRc;
    cap = (int)std::min(65528.0, expected * 1.35 + 32);
  }
  cap = (cap + 7) / 8 * 8;
  if (outer && c.outerAtoms < (size_t)N) {
    CK(cudaFree(g.dNbCountOuter));
    CK(cudaFree(g.dROuter));
    CK(cudaMalloc(&g.dNbCountOuter, sizeof(int) * N));
    CK(cudaMalloc(&g.dROuter, sizeof(double) * 3 * N));
    c.outerAtoms = N;
  }
  const double invL2 = 1.0 / (L * L);
  BuildArgs A;
  A.g = geo;
  A.tab = g.dHaloTab;
  A.pos4 = g.dPos4;
  A.start = g.dStart;
  A.orig = g.dOrig;
  A.K = g.dK;
  A.type8 = g.dType8;
  A.body = s.dBody;
  A.hasBodies = s.nbodies > 0;
  A.interact = s.models.interact;
  A.ntypes = s.ntypes;
  A.exFirst = s.dExFirst;
  A.exCount = s.dExCount;
  A.exItem = s.dExItem;
  A.hasEx = s.hasExclusions;
  A.R = s.dR;
  A.L = L;
  A.thr = xRcSq * invL2;    // src/neighbor_lists.f90:213-214 (outer lists: rc + skin + delta)
  A.thrIn = s.xInRcSq * invL2;
  double M2 = (double)g.M * g.M;
  A.lo2 = (float)(A.thr * M2 * (1.0 - BAND));
  A.hi2 = (float)(A.thr * M2 * (1.0 + BAND));
  A.loIn2 = (float)(A.thrIn * M2 * (1.0 - BAND));
  A.hiIn2 = (float)(A.thrIn * M2 * (1.0 + BAND));
  A.layered = s.xInRcSq < s.xRcSq ? 1 : 0;
  A.minimg = g.M == 5 ? 1 : 0;
  A.Mf = (float)g.M;
  A.haloCap = g.maxHalo;
  A.nbCount = outer ? g.dNbCountOuter : g.dNbCount;
  A.nbInner = g.dNbInner;
  A.selfIdx = g.dSelf;
  A.tileStride = g.tileStride;
  A.maxCount = g.dTileInfo + 2 * g.nTiles + 2;
  A.fail = (unsigned long long*)(s.dResult + BUILD_FAILED);
  grow(g.dLayout, g.layoutCap, (size_t)g.nTiles * (2 * g.haloCells + 1));
  A.layout = g.dLayout;
  const bool general = build_general(s);
  size_t smem = build_smem(g, s.ntypes, general);
  A.invM = 1.0f / A.Mf;
  A.tpa = build_tpa(s);
  A.tpaShift = 0;
  while (1 << A.tpaShift < A.tpa) A.tpaShift++;
  A.allInteract = 1;
  for (size_t q = 0; q < (size_t)s.ntypes * s.ntypes; q++)
    if (!s.interact[q]) A.allInteract = 0;
  void (*kb)(BuildArgs) = nullptr;
#define BUILD_KERNEL(MODE)                                                             \
  kb = general ? (A.minimg ? k_build<true, true, MODE> : k_build<true, false, MODE>)   \
               : (A.minimg ? k_build<false, true, MODE> : k_build<false, false, MODE>)
  if (A.tpa == 1 && g.nTiles > N) BUILD_KERNEL(BUILD_SPARSE);
  else if (A.tpa == 1) BUILD_KERNEL(BUILD_ONE);
  else if (A.tpa < 32) BUILD_KERNEL(BUILD_SPLIT);
  else BUILD_KERNEL(BUILD_WARP);
#undef BUILD_KERNEL
  const int buildThreads = build_block_threads(s);
  CK(cudaFuncSetAttribute(kb, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
#ifdef EMDEE_MAX_CARVEOUT
  CK(cudaFuncSetAttribute(kb, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
#endif
  for (int attempt = 0; attempt < 3; attempt++) {
    size_t need = (size_t)g.nTiles * cap * g.tileStride;
    grow(nbList, nbCap, need);
    A.nb = nbList;
    A.cap = cap;
    if (attempt > 0) {   // k_assign zeroed them for the first
      CK(cudaMemsetAsync(A.maxCount, 0, sizeof(int), s.stream));
      CK(cudaMemsetAsync(A.fail, 0, sizeof(*A.fail), s.stream));
    }
    if (chain_fits(g.nTiles)) launch_chained(kb, g.nTiles, buildThreads, smem, s.stream, A);
    else kb<<<g.nTiles, buildThreads, smem, s.stream>>>(A);
    s.prof.total++;
    CK(cudaGetLastError());
    if (defer) break;
    const int* mc = s.hFlags + 2;   // pinned: largest list, tile-size overflow
    build_flags(s);
    CK(cudaStreamSynchronize(s.stream));
    if (mc[1]) return false;
    if (mc[0] <= cap) break;
    if (mc[0] > 65528) fatal("neighbor list build", "more than 65528 neighbors for one atom");
    cap = std::min(65528, (mc[0] + mc[0] / 8 + 16 + 7) / 8 * 8);
  }
  s.r0Valid = true;   // R0 was written by k_assign
  s.builtL = L;
  s.listsOuter = outer;
  if (outer) {   // the reference positions of the coverage test
    CK(cudaMemcpyAsync(g.dROuter, s.dR, sizeof(double) * 3 * N, cudaMemcpyDeviceToDevice, s.stream));
    s.outerDelta = delta;
    s.outerL = L;
  }
  return true;
}

void device_build_lists(System& s, bool defer) {
  prof_begin(s, PK_BUILD);
  if (!build_lists(s, true, defer)) build_lists(s, false, false);
  prof_end(s, PK_BUILD);
}

bool build_settled(const System& s) { return !s.hFlags[3] && s.hFlags[2] <= s.grid.cap; }

// ---------------------------------------------------------------------------------
// two-level lists
// ---------------------------------------------------------------------------------
//
// An outer build lists every pair within rc + skin + delta; the force kernel of a
// rebuild step filters those lists into the lists the reference would build (every
// pair within rc + skin, the same FP32 + FP64-band test as k_build), as long as
// the outer lists still hold every such pair: with d1 >= d2 the two largest
// displacements since the outer build, a pair now within rc + skin was within
// rc + skin + d1 + d2 then, so d1 + d2 < delta suffices.  The rebuild schedule and
// the pair sets stay those of the reference; only the work per rebuild changes.

// Off unless requested (EmDee_set_outer_skin, or EMDEE_OUTER_SKIN for systems that
// did not set it).  Measured on the 1M-atom Lennard-Jones bench (skin 0.3, T* 1.5):
// the fastest of a million atoms cross any outer skin up to 0.9 within two rebuild
// periods, so outer builds (1.7x a build at rc + skin + 0.45) come every second
// rebuild, and the filtering launch costs about as much as the build it replaces:
// 387 us per step against 350 with single-level lists.  Slower dynamics (more
// rebuilds per outer build) are where the outer lists pay.
double outer_delta(System& s) {
  if (s.outerSkin >= 0.0) return s.outerSkin;
  static const double env = getenv("EMDEE_OUTER_SKIN") ? atof(getenv("EMDEE_OUTER_SKIN")) : 0.0;
  return env > 0.0 ? env : 0.0;
}

bool two_level_active(System& s) {
  const double d = outer_delta(s);
  if (!(d > 0.0) || s.precision != 0 || s.nlayers != 1 || !(s.skin > 0.0) || s.xInRcSq < s.xRcSq) return false;
  if (!pair_lj_only(s)) return false;
  return (int)std::floor(NDIV * *s.Lbox / (s.xRc + d)) > 2 * NDIV + 1;   // outer cells: M > 5
}

// Coverage test of the outer lists and start of a new rebuild period: the largest
// and second largest squared displacement since the outer build (FP64 differences,
// FP32 squares, compared as non-negative bit patterns, an order-independent pair);
// result[40] = 0 if d1 + d2 < delta (with a relative margin for the FP32 squares),
// else 1, result[41] = d1 + d2.  Also R0 = R and pos0 = the current packed position
// of every atom (the reference positions of the skin check and of the packing).
__global__ void __launch_bounds__(SKIN_THREADS) k_cover(const double* __restrict__ R, const double* __restrict__ RO,
                                                        const int* __restrict__ slotOf,
                                                        const float4* __restrict__ pos4, int N, double delta,
                                                        double* __restrict__ R0, float4* __restrict__ pos0,
                                                        int2* partial, unsigned int* ticket, double* result) {
  __shared__ int2 wsum[SKIN_THREADS / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int a = 0, b = 0;   // bits of the largest and second largest d^2 (FP32, >= 0)
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    float d2 = 0.0f;
    for (int k = 0; k < 3; k++) {
      const double r = R[3 * i + k];
      const float d = d2f(r - RO[3 * i + k]);
      d2 = fmaf(d, d, d2);
      R0[3 * i + k] = r;
    }
    pos0[i] = pos4[slotOf[i]];
    const int v = __float_as_int(d2);
    b = max(b, min(a, v));
    a = max(a, v);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const int oa = __shfl_down_sync(0xffffffffu, a, o), ob = __shfl_down_sync(0xffffffffu, b, o);
    b = max(max(b, ob), min(a, oa));
    a = max(a, oa);
  }
  if (lane == 0) wsum[warp] = make_int2(a, b);
  __syncthreads();
  if (threadIdx.x == 0) {
    int2 t = wsum[0];
    for (int w = 1; w < SKIN_THREADS / 32; w++) {
      t.y = max(max(t.y, wsum[w].y), min(t.x, wsum[w].x));
      t.x = max(t.x, wsum[w].x);
    }
    partial[blockIdx.x] = t;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  int2 t = make_int2(0, 0);
  for (unsigned int k = 0; k < gridDim.x; k++) {
    const int2 p = __ldcg(&partial[k]);
    t.y = max(max(t.y, p.y), min(t.x, p.x));
    t.x = max(t.x, p.x);
  }
  const double sum = sqrt((double)__int_as_float(t.x)) + sqrt((double)__int_as_float(t.y));
  result[41] = sum;
  result[40] = sum * (1.0 + 1e-5) < delta ? 0.0 : 1.0;
  *ticket = 0;
}

// The filtering pair launch on the current outer lists, with the lists regrown
// until the longest filtered list fits; false if skip was set (nothing ran).
static bool refilter(System& s, bool compute, const double* skip) {
  Grid& g = s.grid;
  ensure_partials(s, g.nTiles);
  for (;;) {
    grow(g.dNb, g.caps.nb, (size_t)g.nTiles * g.cap * g.tileStride);
    int* innerMax = g.dTileInfo + 2 * g.nTiles + 4;
    CK(cudaMemsetAsync(innerMax, 0, sizeof(int), s.stream));
    prof_begin(s, PK_PAIR);
    device_pair_refilter(s, compute, skip);
    prof_end(s, PK_PAIR);
    // the kernel's last block wrote the sums into hResult[0..4]
    if (skip) CK(cudaMemcpyAsync(s.hResult + 40, s.dResult + 40, 2 * sizeof(double), cudaMemcpyDeviceToHost, s.stream));
    CK(cudaMemcpyAsync(s.hFlags, innerMax, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    CK(cudaStreamSynchronize(s.stream));
    if (skip && s.hResult[40] != 0.0) {
      prof_drop_last(s);
      return false;
    }
    const int mc = s.hFlags[0];
    if (mc <= g.cap) return true;
    if (mc > 65528) fatal("neighbor list build", "more than 65528 neighbors for one atom");
    g.cap = std::min(65528, (mc + mc / 8 + 16 + 7) / 8 * 8);
    skip = nullptr;   // covered: filter again with room for the longest list
  }
}

void device_rebuild_two_level(System& s, bool compute) {
  Grid& g = s.grid;
  const int N = s.natoms;
  if (s.listsOuter && *s.Lbox == s.outerL && s.outerDelta == outer_delta(s)) {
    if (!s.packReady) device_pack(s);
    const int blocks = std::min((N + SKIN_THREADS - 1) / SKIN_THREADS, 4 * 152);
    ensure_partials(s, blocks);
    prof_begin(s, PK_BUILD);
    k_cover<<<blocks, SKIN_THREADS, 0, s.stream>>>(s.dR, g.dROuter, g.dSlotOf, g.dPos4, N, s.outerDelta, s.dR0,
                                                   g.dPos0, (int2*)s.dPartials, s.dTicket, s.dResult);
    CK(cudaGetLastError());
    prof_end(s, PK_BUILD);
    if (refilter(s, compute, s.dResult + 40)) return;
  }
  device_build_lists(s);
  s.outerBuilds++;
  refilter(s, compute, nullptr);
}

// ---------------------------------------------------------------------------------
// pair-set dump (test support): every full-list entry as (orig_i, orig_j)
// ---------------------------------------------------------------------------------

__global__ void k_dump_pairs(TileGeom g, const int2* tab, const int* start, const int* orig, const uint16_t* nb,
                             const int* nbCount, int cap, int tileStride, const long long* outStart, int2* out) {
  extern __shared__ int hslot[];
  __shared__ int ws[33];
  __shared__ int off[1001], cst[1000];
  const int t = blockIdx.x, cells = g.TB * g.TB * g.TB;
  halo_layout(g, t, tab, start, off, cst, (int*)nullptr, ws);
  for (int h = threadIdx.x; h < g.haloCells; h += blockDim.x)
    for (int k = off[h]; k < off[h + 1]; k++) hslot[k] = cst[h] + (k - off[h]);
  __syncthreads();
  const int tb = start[t * cells], te = start[(t + 1) * cells];
  for (int li = threadIdx.x; li < te - tb; li += blockDim.x) {
    int si = tb + li, ai = orig[si];
    long long o = outStart[si];
    for (int k = 0; k < nbCount[si]; k++) {
      int q = nb[nb_index(t, cap >> 3, tileStride, li, k)];
      out[o + k] = make_int2(ai + 1, orig[hslot[q]] + 1);
    }
  }
}

long device_neighbor_pairs(System& s, int* pairs, long capacity) {
  Grid& g = s.grid;
  int N = s.natoms;
  if (!s.r0Valid) return 0;
  std::vector<int> cnt(N), orig(N);
  CK(cudaStreamSynchronize(s.stream));
  CK(cudaMemcpy(cnt.data(), g.dNbCount, sizeof(int) * N, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(orig.data(), g.dOrig, sizeof(int) * N, cudaMemcpyDeviceToHost));
  std::vector<long long> st(N + 1, 0);
  for (int i = 0; i < N; i++) st[i + 1] = st[i] + cnt[i];
  long long total = st[N];
  long npairs = (long)(total / 2);
  if (npairs > capacity) return -npairs;
  long long* dSt;
  int2* dOut;
  CK(cudaMalloc(&dSt, sizeof(long long) * (N + 1)));
  CK(cudaMalloc(&dOut, sizeof(int2) * (total + 1)));
  CK(cudaMemcpy(dSt, st.data(), sizeof(long long) * (N + 1), cudaMemcpyHostToDevice));
  TileGeom geo = make_geom(g.M, g.TB);
  CK(cudaFuncSetAttribute(k_dump_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(int) * g.maxHalo));
  k_dump_pairs<<<g.nTiles, 128, sizeof(int) * g.maxHalo, s.stream>>>(geo, g.dHaloTab, g.dStart, g.dOrig, g.dNb,
                                                                      g.dNbCount, g.cap, g.tileStride, dSt, dOut);
  CK(cudaGetLastError());
  std::vector<int2> h(total);
  CK(cudaStreamSynchronize(s.stream));
  CK(cudaMemcpy(h.data(), dOut, sizeof(int2) * total, cudaMemcpyDeviceToHost));
  CK(cudaFree(dSt));
  CK(cudaFree(dOut));
  std::vector<std::pair<int, int>> v;
  v.reserve(npairs);
  for (auto& e : h)
    if (e.x < e.y) v.push_back({e.x, e.y});
  std::sort(v.begin(), v.end());
  long n = (long)v.size();
  if (n > capacity) return -n;
  for (long k = 0; k < n; k++) {
    pairs[2 * k] = v[k].first;
    pairs[2 * k + 1] = v[k].second;
  }
  return n;
}

// ---------------------------------------------------------------------------------
// radial distribution histograms over the current lists (src/EmDeeCode.f90:1281-1395)
// ---------------------------------------------------------------------------------

struct RdfArgs {
  TileGeom g;
  const int* layout;
  const int* start;
  const int* orig;
  const uint16_t* self;
  const uint16_t* nb;
  const int* count;   // entries to scan per slot (all, or the inner part)
  const uint8_t* type8;
  const double* R;
  int cap, tileStride, bins, ntp;   // ntp: histogram rows (type pairs, symm1D order)
  double invL, Rc2, binsByRc;
  float limit;   // box_limit(Rc2)
  const uint8_t* hasPair;   // [type] (0-based)
  const uint8_t* pairOn;    // [ti * ntypes + tj]
  int ntypes, haloCap;
  unsigned long long* hist;   // [pair][bin]
  int sharedHist;             // histogram fits in shared memory
};

// Threads per block, as many as the largest tile has atoms up to this: tiles of 4 to 6 cells
// in mixed precision have 140 to 480, and their staged halo leaves room for two to four blocks
// per SM.  100 bins, with at most 128 threads -> so: 32,003 atoms 265 -> 157 us, 300,000 1266 ->
// 898, 1,000,000 6587 -> 2568.
static const int RDF_THREADS = 512;

// A halo atom as the histogram needs it: scaled coordinates, slot, type; box fractions
// and slot
struct __align__(16) RdfAtom {
  double x, y, z;
  int slot, type;
  int4 frac;
};

// The lists hold every pair twice, at the same distance: it is counted from one of its
// atoms, the lower slot if the slots' sum is even and the higher one if it is odd (half of
// every atom's pairs).  The FP64 distance, bound by its pipe, is evaluated for the entries
// that a mask of FP32 tests leaves, on nearly full warps.  32,003
// atoms, 100 bins: 330 us with both directions, FP64 rounding and gathers of R, 140 us so.
// STAGED: the halo atoms are staged as RdfAtom; tiles whose halo does not fit so keep
// the slots only and gather the rest.
template <bool STAGED>
__global__ void __launch_bounds__(RDF_THREADS) k_rdf(RdfArgs A) {
  extern __shared__ __align__(16) unsigned char sraw[];
  const TileGeom g = A.g;
  const int t = blockIdx.x, cells = g.TB * g.TB * g.TB;
  RdfAtom* halo = (RdfAtom*)sraw;
  int* hslot = (int*)sraw;
  unsigned int* sh = STAGED ? (unsigned int*)(halo + A.haloCap) : (unsigned int*)(hslot + A.haloCap);
  auto slot = [&](int q) { return STAGED ? halo[q].slot : hslot[q]; };
  auto load = [&](int sj) {
    const int a = A.orig[sj];
    const double x = A.invL * A.R[3 * a], y = A.invL * A.R[3 * a + 1], z = A.invL * A.R[3 * a + 2];
    return RdfAtom{x, y, z, sj, A.type8[sj], make_int4(box_fraction(x), box_fraction(y), box_fraction(z), sj)};
  };
  const int* lay = A.layout + (size_t)t * (2 * g.haloCells + 1);
  for (int h = threadIdx.x; h < g.haloCells; h += blockDim.x) {
    const int b = lay[h], e = lay[h + 1], s0 = lay[g.haloCells + 1 + h];
    for (int q = b; q < e; q++) (STAGED ? halo[q].slot : hslot[q]) = s0 + q - b;
  }
  const int hn = A.bins * A.ntp;
  if (A.sharedHist)
    for (int k = threadIdx.x; k < hn; k += blockDim.x) sh[k] = 0u;
  __syncthreads();
  if (STAGED) {
    const int nh = lay[g.haloCells];
    for (int q = threadIdx.x; q < nh; q += blockDim.x) halo[q] = load(halo[q].slot);
    __syncthreads();
  }
  const int tb = A.start[t * cells], te = A.start[(t + 1) * cells];
  for (int li = threadIdx.x; li < te - tb; li += blockDim.x) {
    const int si = tb + li;
    const RdfAtom pi = STAGED ? halo[A.self[si]] : load(si);
    if (!A.hasPair[pi.type]) continue;
    const int n = A.count[si];
    const uint4* lp = reinterpret_cast<const uint4*>(A.nb) + ((size_t)t * (A.cap >> 3) * A.tileStride + li);
    masked_entries(
        lp, A.tileStride, n,
        [&](int q) {
          const int sj = slot(q);
          if (((si ^ sj) & 1) ? si < sj : si > sj) return false;
          return !STAGED || box_dist2(pi.frac, halo[q].frac) < A.limit;
        },
        [&](int q) {
          const RdfAtom pj = STAGED ? halo[q] : load(hslot[q]);
          if (!A.pairOn[pi.type * A.ntypes + pj.type]) return;
          const double dx = wrap_half(pi.x - pj.x), dy = wrap_half(pi.y - pj.y), dz = wrap_half(pi.z - pj.z);
          const double r2 = dx * dx + dy * dy + dz * dz;
          if (!(r2 < A.Rc2)) return;
          const int bin = min((int)(sqrt(r2) * A.binsByRc), A.bins - 1);
          const int a = min(pi.type, pj.type), b = max(pi.type, pj.type), p = a + (b + 1) * b / 2;   // symm1D - 1 (0-based types)
          if (A.sharedHist) atomicAdd(&sh[p * A.bins + bin], 1u);
          else atomicAdd(&A.hist[(size_t)p * A.bins + bin], 1ull);
        });
  }
  if (A.sharedHist) {
    __syncthreads();
    for (int k = threadIdx.x; k < hn; k += blockDim.x)
      if (sh[k]) atomicAdd(&A.hist[k], (unsigned long long)sh[k]);
  }
}

// counts[pair][bin] (pairs in symm1D order over types 1..maxtype), each pair once
void device_rdf_counts(System& s, int bins, double Rc, const std::vector<uint8_t>& hasPair,
                       const std::vector<uint8_t>& pairOn, int ntp, std::vector<unsigned long long>& counts) {
  Grid& g = s.grid;
  const int nt = s.ntypes;
  RdfArgs A;
  A.g = make_geom(g.M, g.TB);
  A.layout = g.dLayout;
  A.start = g.dStart;
  A.orig = g.dOrig;
  A.self = g.dSelf;
  A.nb = g.dNb;
  A.count = Rc < 1.0001 * s.InRc ? g.dNbInner : g.dNbCount;
  A.type8 = g.dType8;
  A.R = s.dR;
  A.cap = g.cap;
  A.tileStride = g.tileStride;
  A.bins = bins;
  A.ntp = ntp;
  const double invL = 1.0 / *s.Lbox;
  A.invL = invL;
  A.Rc2 = Rc * Rc * (invL * invL);
  A.limit = box_limit(A.Rc2);
  A.binsByRc = bins / (Rc * invL);
  A.ntypes = nt;
  A.haloCap = g.maxHalo;
  // histogram, then the two type filters: one buffer kept with the system
  const size_t hn = (size_t)bins * ntp, bytes = sizeof(unsigned long long) * hn, filters = (size_t)nt + (size_t)nt * nt;
  if (s.rdfCap < bytes + filters) {
    CK(cudaFree(s.dRdf));
    CK(cudaMalloc(&s.dRdf, bytes + filters));
    s.rdfCap = bytes + filters;
  }
  uint8_t* dHas = s.dRdf + bytes;
  std::vector<uint8_t> host(hasPair);
  host.insert(host.end(), pairOn.begin(), pairOn.end());
  CK(cudaMemsetAsync(s.dRdf, 0, bytes, s.stream));
  CK(cudaMemcpyAsync(dHas, host.data(), filters, cudaMemcpyHostToDevice, s.stream));
  A.hasPair = dHas;
  A.pairOn = dHas + nt;
  A.hist = (unsigned long long*)s.dRdf;
  A.sharedHist = (hn * sizeof(unsigned int) <= 48 * 1024) ? 1 : 0;
  const size_t histBytes = A.sharedHist ? hn * sizeof(unsigned int) : 0;
  const bool staged = sizeof(RdfAtom) * (size_t)g.maxHalo + histBytes <= 200 * 1024;
  const size_t smem = (staged ? sizeof(RdfAtom) : sizeof(int)) * (size_t)g.maxHalo + histBytes;
  auto kern = staged ? k_rdf<true> : k_rdf<false>;
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<g.nTiles, std::min(RDF_THREADS, (g.tileAtoms + 31) / 32 * 32), smem, s.stream>>>(A);
  CK(cudaGetLastError());
  s.prof.total++;
  counts.assign(hn, 0ull);
  CK(cudaMemcpyAsync(counts.data(), s.dRdf, bytes, cudaMemcpyDeviceToHost, s.stream));
  CK(cudaStreamSynchronize(s.stream));
}

// ---------------------------------------------------------------------------------
// fused step: pending boosts, move, skin displacement and FP32 packing in one pass
// ---------------------------------------------------------------------------------

// Contiguous atom ranges combined in index order, as in k_skin, so the skin value
// is the same for any range size.  Each
// statement rounds as the separate kernels do (this file uses -fmad=false).
static const int STEP_CHUNKS = 2;   // at most 64 consecutive atoms per warp (skin_chunks): many warps in flight

// FMA (mixed precision only): the updates use fused multiply-adds, which halves the
// work on the FP64 pipe (the limit of this kernel on GB300); FP64 mode keeps the
// reference's separately rounded statements.
// VV: the opening half of EmDee_verlet_step (src/EmDeeCode.f90:1107-1211), with the shadow
// start values in s0 if it is set; each statement as in k_vv_pre_free.
template <int NK, bool UNITM, bool PACK, bool FMA, bool VV>
__global__ void __launch_bounds__(SKIN_THREADS) k_step_fused(double* __restrict__ R, double* __restrict__ P,
                                                             const double* F,
                                                             const double* __restrict__ invMass,
                                                             const double* R0, int N, int chunks, double cf0,
                                                             double cf1, double CP, double skinSq,
                                                             const int* slotOf,
                                                             const float4* pos0, float scale,
                                                             float4* __restrict__ pos4, longlong2* partial,
                                                             unsigned int* ticket, double* result,
                                                             double* hostResult, double* __restrict__ s0,
                                                             unsigned long long* done, unsigned int stamp) {
  chain_wait();
  __shared__ MaxPrev wsum[SKIN_THREADS / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int base = (blockIdx.x * (SKIN_THREADS / 32) + warp) * 32 * chunks;
  MaxPrev run{-1, -1};
  for (int c = 0; c < chunks; c++) {
    const int i = base + c * 32 + lane;
    MaxPrev v{-1, -1};
    if (i < N) {
      const double im = UNITM ? 1.0 : invMass[i];
      double r[3];
      for (int d = 0; d < 3; d++) {
        double p = P[3 * i + d];
        if (VV && s0 != nullptr) {
          const double f = F[3 * i + d];
          s0[3 * i + d] = 2.5 * R[3 * i + d] + cf0 * im * (p - cf0 * f);
        }
        if (FMA) {
          if (NK >= 1) p = fma(cf0, F[3 * i + d], p);
          if (NK >= 2) p = fma(cf1, F[3 * i + d], p);
        } else {
          if (NK >= 1) p = p + cf0 * F[3 * i + d];
          if (NK >= 2) p = p + cf1 * F[3 * i + d];
        }
        if (NK >= 1) P[3 * i + d] = p;
        if (FMA) r[d] = UNITM || (VV && im == 1.0) ? fma(CP, p, R[3 * i + d]) : fma(CP * p, im, R[3 * i + d]);
        else r[d] = R[3 * i + d] + (UNITM ? CP * p : CP * p * im);
        R[3 * i + d] = r[d];
      }
      const double d0 = r[0] - R0[3 * i], d1 = r[1] - R0[3 * i + 1], d2 = r[2] - R0[3 * i + 2];
      v.m = __double_as_longlong(FMA ? fma(d2, d2, fma(d1, d1, d0 * d0)) : d0 * d0 + d1 * d1 + d2 * d2);
      if (PACK) pos4[slotOf[i]] = pack_delta(pos0[i], d0, d1, d2, scale);
    }
    v = warp_ordered_combine(v);
    run = mp_combine(run, v);
  }
  if (lane == 0) wsum[warp] = run;
  __syncthreads();
  if (threadIdx.x == 0) {
    MaxPrev b = wsum[0];
    for (int w = 1; w < SKIN_THREADS / 32; w++) b = mp_combine(b, wsum[w]);
    partial[blockIdx.x] = make_longlong2(b.m, b.p);
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int nb = gridDim.x, per = (nb + SKIN_THREADS - 1) / SKIN_THREADS;
  MaxPrev acc{-1, -1};
  for (int k = 0; k < per; k++) {
    int b = threadIdx.x * per + k;
    if (b < nb) {
      longlong2 v = __ldcg(&partial[b]);
      acc = mp_combine(acc, MaxPrev{v.x, v.y});
    }
  }
  acc = warp_ordered_combine(acc);
  if (lane == 0) wsum[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    MaxPrev b = wsum[0];
    for (int w = 1; w < SKIN_THREADS / 32; w++) b = mp_combine(b, wsum[w]);
    double maximum = __longlong_as_double(b.m), next = __longlong_as_double(b.p < 0 ? b.m : b.p);
    double value = maximum + 2 * sqrt(maximum * next) + next;
    result[8] = value;
    result[9] = value > skinSq ? 1.0 : 0.0;
    hostResult[8] = value;   // pinned host memory: read after the next synchronisation
    hostResult[9] = result[9];
    *ticket = 0;
    *(volatile unsigned long long*)done = 2ull * stamp + (value > skinSq ? 1 : 0);
  }
}

void device_step_fused(System& s, double CP, bool vv, double* s0) {
  const int N = s.natoms, chunks = skin_chunks(N, STEP_CHUNKS), per = SKIN_THREADS * chunks;
  const int blocks = (N + per - 1) / per;
  ensure_partials(s, blocks);
  const bool pack = s.precision == 0 && s.r0Valid && *s.Lbox == s.builtL;
  const Grid& g = s.grid;
  const float scale = g.M > 0 ? (float)((double)g.M / *s.Lbox) : 0.0f;
  if (vv) {   // no kick is pending: the half-step's own
    s.pendCF[0] = 0.5 * CP;
    s.npend = 1;
  }
  s.skinStamp++;
  prof_begin(s, PK_MOVE);
#define STEP_ARGS s.dR, s.dP, s.F(), s.dInvMass, s.dR0, N, chunks, s.pendCF[0], s.pendCF[1], CP, s.skinSq, g.dSlotOf, \
                  g.dPos0, scale, g.dPos4, (longlong2*)s.dPartials, s.dTicket, s.dResult, s.hResult, s0, s.hSkinDone, s.skinStamp
#define STEP_LAUNCH(NK, UM, PK, FM, VV) launch_chained(k_step_fused<NK, UM, PK, FM, VV>, blocks, SKIN_THREADS, 0, s.stream, STEP_ARGS)
#define STEP_NK(UM, PK, FM)                            \
  if (vv) STEP_LAUNCH(1, UM, PK, FM, true);            \
  else if (s.npend == 0) STEP_LAUNCH(0, UM, PK, FM, false); \
  else if (s.npend == 1) STEP_LAUNCH(1, UM, PK, FM, false); \
  else STEP_LAUNCH(2, UM, PK, FM, false);
  if (pack) {   // mixed precision: fused multiply-adds
    if (s.unitMass) { STEP_NK(true, true, true) } else { STEP_NK(false, true, true) }
  } else if (s.precision == 0) {
    if (s.unitMass) { STEP_NK(true, false, true) } else { STEP_NK(false, false, true) }
  } else {
    if (s.unitMass) { STEP_NK(true, false, false) } else { STEP_NK(false, false, false) }
  }
#undef STEP_NK
#undef STEP_LAUNCH
#undef STEP_ARGS
  CK(cudaGetLastError());
  prof_end(s, PK_MOVE);
  s.npend = 0;
  s.skinReady = s.r0Valid;
  s.packReady = pack;
}

// the skin value left by the fused step (its last block also wrote hResult[8..9])
bool device_skin_from_step(System& s) {
  CK(cudaStreamSynchronize(s.stream));
  return s.hResult[9] != 0.0;
}

}  // namespace emdee
