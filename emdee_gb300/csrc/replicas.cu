// replicas.cu -- many independent systems advanced together by one persistent
// kernel (no reference counterpart: the reference runs one system per call).
//
// One thread block owns one replica for the whole run: every step it performs,
// with block-wide barriers between the phases, the reference's velocity-Verlet
// loop body (test/common/contained.f90:63-72) -- boost(dt/2), displace(dt),
// the skin check of src/neighbor_lists.f90:41-59, a neighbor-list rebuild when
// it fires, the pair forces, boost(dt/2) -- so a whole trajectory of hundreds of
// replicas is one launch (captured once in a CUDA graph and replayed).
//
// Per replica, in shared memory: the positions of its atoms as 32-bit fractions of the
// box (slot order), whose differences are minimum images without image arithmetic and
// finer than FP32 coordinates, and the cell starts.  In global memory: R, P, F, R0 of
// the system (FP64, API order) and the replica's own cell-sorted order and full neighbor
// lists (8 slots of 16 bits per 16-byte chunk, chunk-major).  Blocks are issued largest
// replica first.
//
// Scope: up to 8 atom types (pair models with their modifiers), no charges, no
// rigid bodies, no exclusions, one model layer, FP32 pair arithmetic (the mixed
// mode).  The pair set is the
// reference's: FP32 prefilter, FP64 test of src/neighbor_lists.f90:247-250 for
// candidates within 4e-5 of the threshold (this file uses -fmad=false).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "reduce.cuh"
#include "system.hpp"
#include "tile.cuh"

namespace emdee {

struct RepDesc {
  double *R, *P, *F, *R0;        // the system's arrays (API order)
  const double* invMass;
  int unitMass;
  int N, M, minimg, cap;
  double L, frac, skinSq, thr;   // frac = 2^32 / L; thr = (rc+skin)^2 / L^2
  float lo2, hi2, Mf;            // list band, cell units^2
  float rc2, unit, unit2;        // cut-off^2 in box fractions^2; 2^32 / L and its square
  PairEntry<float> model;          // type pair (1, 1)
  int ntypes;
  int ljAll;                       // every type pair is lj_cut without modifier
  const PairEntry<float>* table;   // the system's layer-1 pair table, [jtype][itype]
  const int* type;                 // atom types (1-based, API order)
  int* orig;        // slot -> atom
  uint16_t* slotOf; // atom -> slot
  int4* frac4;      // per atom: box fractions and cell during a build
  double* Rb;       // coordinates of the build that made the lists below
  uint4* list;      // entries 8c..8c+7 of slot i: list[c * N + i]
  int* count;       // per slot
  double* out;      // [0] Epair [1] Wpair [2..4] 2KE per dim [5] builds [6] overflow [7] steps done
  int computeLast;  // unused by the kernel (host bookkeeping)
};

static const double REP_BAND = 4e-5;
static const int REP_MAXT = 8;   // atom types a replica may have

__device__ __forceinline__ bool rep_exact_inside(const double* R, double L, int a, int b, double thr) {
  double d[3];
  for (int k = 0; k < 3; k++) {
    double x = R[3 * a + k] / L - R[3 * b + k] / L;
    d[k] = x - round(x);
  }
  return d[0] * d[0] + d[1] * d[1] + d[2] * d[2] < thr;
}

// (max, prev) combine of the skin check over contiguous index ranges (see neighbor.cu)
struct RepMP {
  long long m, p;
};
__device__ __forceinline__ RepMP rep_combine(RepMP a, RepMP b) {
  if (b.m > a.m) return RepMP{b.m, a.m > b.p ? a.m : b.p};
  return a;
}
__device__ __forceinline__ RepMP rep_warp_ordered(RepMP acc) {
  const int lane = threadIdx.x & 31;
  for (int o = 1; o < 32; o <<= 1) {
    RepMP other{(long long)__shfl_down_sync(0xffffffffu, (unsigned long long)acc.m, o),
                (long long)__shfl_down_sync(0xffffffffu, (unsigned long long)acc.p, o)};
    if ((lane & (2 * o - 1)) == 0) acc = rep_combine(acc, other);
  }
  return acc;
}

struct RepShared {
  RepDesc d;
  int rebuild, overflow;
  int scan[33];
  RepMP wmp[32];
  float2 wff[2][32];
  double wke[3][32];
};

// box fraction of a coordinate: low word of R 2^32 / L + 1.5 2^52
__device__ __forceinline__ int rep_fraction(double r, const RepDesc& D) {
  const double t = fma(r, D.frac, 6755399441055744.0);
  if ((__double2hiint(t) & 0xFFF00000) == 0x43300000) return __double2loint(t);
  return __double2loint(fma(r / D.L - floor(r / D.L), 4294967296.0, 6755399441055744.0));   // 2^19 boxes away
}

static const int REP_PAD = 4;   // positions a segment of four may read past the last one

// Cells, cell-sorted order and full lists from the coordinates Rb.  The cell of an atom is
// the product of its box fraction and M (a cell index that differs from the reference's
// int(M Rs) by rounding changes only the order of candidates).  Lists as k_build makes
// them: 25 rows of up to 5 cells (one or two runs of slots where a row wraps around the
// box), only cells in reach of the row's distance, candidates tested into a mask four at
// a time, 8 entries stored at once.  (8000 atoms on one SM: 1.35 ms when every atom went
// through all 125 cells one candidate at a time with FP64 cell indices, about
// 0.75 ms so.)
template <int THREADS>
__device__ __noinline__ void rep_build(RepShared& S, const double* Rb, float4* pos, int* cellStart, int* cursor,
                                       bool copyR0) {
  const RepDesc& D = S.d;
  const int N = D.N, M = D.M, cells = M * M * M;
  for (int c = threadIdx.x; c < cells; c += THREADS) cellStart[c] = 0;
  __syncthreads();
  for (int a = threadIdx.x; a < N; a += THREADS) {
    int f[3], cell = 0;
    for (int d = 2; d >= 0; d--) {
      const double r = Rb[3 * a + d];
      f[d] = rep_fraction(r, D);
      cell = (int)__umulhi((unsigned)f[d], (unsigned)M) + M * cell;
      D.Rb[3 * a + d] = r;
      if (copyR0) D.R0[3 * a + d] = r;
    }
    D.frac4[a] = make_int4(f[0], f[1], f[2], cell);
    atomicAdd(&cellStart[cell], 1);
  }
  __syncthreads();
  constexpr int ITEMS = 8192 / THREADS;
  int carry = 0;
  for (int base = 0; base < cells; base += THREADS * ITEMS) {
    const int n = min(THREADS * ITEMS, cells - base);
    const int total = block_exclusive_scan<ITEMS>(cellStart + base, n, S.scan);
    for (int c = threadIdx.x; c < n; c += THREADS) cursor[base + c] = cellStart[base + c] += carry;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) cellStart[cells] = N;
  __syncthreads();
  for (int a = threadIdx.x; a < N; a += THREADS) D.orig[atomicAdd(&cursor[D.frac4[a].w], 1)] = a;
  __syncthreads();
  // deterministic order inside a cell: ascending atom index
  for (int c = threadIdx.x; c < cells; c += THREADS) {
    const int b = cellStart[c], e = cellStart[c + 1];
    for (int i = b + 1; i < e; i++) {
      const int v = D.orig[i];
      int j = i - 1;
      while (j >= b && D.orig[j] > v) {
        D.orig[j + 1] = D.orig[j];
        j--;
      }
      D.orig[j + 1] = v;
    }
  }
  __syncthreads();
  // positions in cell edges (FP32), with the cell
  for (int s = threadIdx.x; s < N; s += THREADS) {
    const int a = D.orig[s];
    const int4 f = D.frac4[a];
    const float u = 2.3283064365386963e-10f;   // 2^-32
    const int cx = f.w % M, cy = f.w / M % M, cz = f.w / (M * M);
    pos[s] = make_float4((float)cx + u * (float)((unsigned)f.x * (unsigned)M), (float)cy + u * (float)((unsigned)f.y * (unsigned)M),
                         (float)cz + u * (float)((unsigned)f.z * (unsigned)M), __int_as_float(f.w));
    D.slotOf[a] = (uint16_t)s;
  }
  if (threadIdx.x < REP_PAD) pos[N + threadIdx.x] = make_float4(1e9f, 1e9f, 1e9f, 0.f);
  __syncthreads();
  const int loBits = __float_as_int(D.lo2);
  const unsigned band = (unsigned)(__float_as_int(D.hi2) - loBits);
  const float Mf = D.Mf, invM = 1.0f / Mf, hi2 = D.hi2;
  const bool minimg = D.minimg;
  const int cap = D.cap;
  for (int i = threadIdx.x; i < N; i += THREADS) {
    const float4 pi = pos[i];
    const int cell = __float_as_int(pi.w), cx = cell % M, cy = cell / M % M, cz = cell / (M * M);
    const int ai = D.orig[i];
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    uint4* out = D.list + i;
    int n = 0;
    auto push = [&](int q) {
      w.x = __funnelshift_r(w.x, w.y, 16);
      w.y = __funnelshift_r(w.y, w.z, 16);
      w.z = __funnelshift_r(w.z, w.w, 16);
      w.w = __funnelshift_r(w.w, (unsigned)q, 16);
      n++;
      if ((n & 7) == 0) {
        if (n <= cap) *out = w;
        out += N;
      }
    };
    for (int r = 0; r < 25; r++) {
      const int sy = r % 5 - 2, sz = r / 5 - 2;
      int ny = cy + sy, nz = cz + sz, c0 = cx - 2, c1 = cx + 2;
      if (!minimg) {
        const float dy = fmaxf(fmaxf((float)ny - pi.y, pi.y - (float)(ny + 1)) - 1e-3f, 0.0f);
        const float dz = fmaxf(fmaxf((float)nz - pi.z, pi.z - (float)(nz + 1)) - 1e-3f, 0.0f);
        const float rem = hi2 - fmaf(dy, dy, dz * dz);
        if (rem <= 0.0f) continue;
        const float reach = fmaf(rem, rsqrtf(rem), 1e-3f);
        c0 = max(c0, (int)floorf(pi.x - reach));
        c1 = min(c1, (int)floorf(pi.x + reach));
      }
      const float py = pi.y - (ny < 0 ? -Mf : ny >= M ? Mf : 0.f), pz = pi.z - (nz < 0 ? -Mf : nz >= M ? Mf : 0.f);
      ny += ny < 0 ? M : ny >= M ? -M : 0;
      nz += nz < 0 ? M : nz >= M ? -M : 0;
      const int* row = cellStart + M * (ny + M * nz);
      // the run of slots inside the box, and the one across its face if the row wraps
      for (int part = 0; part < 2; part++) {
        int a0 = max(c0, 0), a1 = min(c1, M - 1);
        float px = pi.x;
        if (part == 1) {
          if (c0 < 0) {
            a0 = c0 + M;
            a1 = M - 1;
            px += Mf;
          } else if (c1 >= M) {
            a0 = 0;
            a1 = c1 - M;
            px -= Mf;
          } else {
            break;
          }
        }
        const int q1 = row[a1 + 1];
        for (int q = row[a0]; q < q1; q += 32) {
          const int len = min(32, q1 - q);
          unsigned m = 0, near = 0xFFFFFFFFu;
          auto bits = [&](int j) {
            const float4 pj = pos[j];
            float dx = px - pj.x, dy = py - pj.y, dz = pz - pj.z;
            if (minimg) {
              dx -= Mf * rintf(dx * invM);
              dy -= Mf * rintf(dy * invM);
              dz -= Mf * rintf(dz * invM);
            }
            return __float_as_int(fmaf(dz, dz, fmaf(dy, dy, dx * dx))) - loBits;
          };
          for (int u = 0; u < len; u += 4)
#pragma unroll
            for (int v = 0; v < 4; v++) {
              const int d = bits(q + u + v);
              m = __funnelshift_l((unsigned)d, m, 1);
              near = min(near, (unsigned)d);
            }
          m <<= (32 - ((len + 3) & ~3));
          if (near < band)   // some candidate lies within the band: the FP64 test decides it
            for (int j = 0; j < len; j++)
              if ((unsigned)bits(q + j) < band && rep_exact_inside(Rb, D.L, ai, D.orig[q + j], D.thr))
                m |= 0x80000000u >> j;
          m &= (unsigned)((int)0x80000000 >> (len - 1));
          if ((unsigned)(i - q) < 32u) m &= ~(0x80000000u >> (i - q));
          while (m) {
            const int j = __clz(m);
            m &= 0x7FFFFFFFu >> j;
            push(q + j);
          }
        }
      }
    }
    D.count[i] = n;
    if (n > cap) atomicMax(&S.overflow, n);
    while (n & 7) push(i);   // the pair loop masks the entries past the count
  }
  __syncthreads();
}

// slot-order box fractions and types from the coordinates R
template <int THREADS>
__device__ __forceinline__ void rep_pack(const RepDesc& D, int4* pos) {
  for (int s = threadIdx.x; s < D.N; s += THREADS) {
    const int a = D.orig[s];
    pos[s] = make_int4(rep_fraction(D.R[3 * a], D), rep_fraction(D.R[3 * a + 1], D), rep_fraction(D.R[3 * a + 2], D),
                       D.ntypes > 1 ? D.type[a] - 1 : 0);
  }
}

// Pair forces of one replica (full lists, one thread per slot, no atomics) in units of
// the box fractions.  LJ: every type pair lj_cut without modifier (E = 4 eps sr6 (sr6 -
// 1), W = 24 eps sr6 (2 sr6 - 1)); otherwise the general model code.  COMPUTE: energies
// too (the virial is always summed).  TPA threads per atom (1 or 2): with 2, the two
// threads of a pair take alternate chunks of the atom's list and add their partial
// forces at the end.
template <bool LJ, bool COMPUTE, int TPA>
__device__ __forceinline__ void rep_pairs(const RepDesc& D, const int4* pos, const NBParams<float>* ptab, float& Ep,
                                          float& Wp) {
  const NBParams<float> mdl = D.model.model;
  const int nt = D.ntypes, N = D.N;
  const float rc2 = D.rc2, unit2 = D.unit2, unit = D.unit;
  const float sigc = mdl.sigsq * unit2, eps48 = 2.0f * mdl.eps24;
  const int cap = D.cap;
  const uint4* list = D.list;   // rebuilt by this kernel: plain loads
  const int* count = D.count;
  const int* orig = D.orig;
  double* __restrict__ F = D.F;
  const int sub = TPA == 1 ? 0 : (int)(threadIdx.x & (TPA - 1));
  const unsigned pmask = TPA == 1 ? 0xffffffffu : (3u << ((threadIdx.x & 31) & ~1u));
  for (int i = threadIdx.x / TPA; i < N; i += blockDim.x / TPA) {
    const int4 pi = pos[i];
    const int n = min(count[i], cap);
    const NBParams<float>* row = ptab + pi.w * nt;
    float fx = 0.f, fy = 0.f, fz = 0.f;
    const int nch = (n + 7) >> 3;
    // 8 entries per 16-byte load, the next chunk requested before this one is used
    uint4 cur = sub < nch ? list[(size_t)sub * N + i] : make_uint4(0u, 0u, 0u, 0u);
    for (int c = sub; c < nch; c += TPA) {
      const uint4 nxt = c + TPA < nch ? list[(size_t)(c + TPA) * N + i] : cur;
      const unsigned words[4] = {cur.x, cur.y, cur.z, cur.w};
      const int left = n - 8 * c;   // entries of this chunk, if fewer than 8
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int4 pj = pos[(words[u >> 1] >> ((u & 1) * 16)) & 0xFFFF];
        const float dx = (float)box_delta(pi.x, pj.x), dy = (float)box_delta(pi.y, pj.y), dz = (float)box_delta(pi.z, pj.z);
        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        const bool in = r2 < rc2 && u < left;
        const float inv2 = in ? Ops<float>::rcp(r2) : 0.f;   // zeroes every term of the others
        float E = 0.f, W;
        if (LJ) {
          float sg = sigc, e48 = eps48, e24 = mdl.eps24, e4 = mdl.eps4;
          if (nt > 1) {
            const NBParams<float>& m = row[pj.w];
            sg = m.sigsq * unit2;
            e24 = m.eps24;
            e48 = 2.0f * e24;
            e4 = m.eps4;
          }
          const float sr2 = sg * inv2, sr6 = sr2 * sr2 * sr2;
          W = sr6 * fmaf(e48, sr6, -e24);
          if (COMPUTE) E = sr6 * fmaf(e4, sr6, -e4);
        } else {
          const float invR2 = (in ? inv2 : 1.f) * unit2, invR = sqrtf(invR2);
          const NBParams<float>& m = nt == 1 ? mdl : row[pj.w];
          nb_compute(m, E, W, invR, invR2);
          modifier_compute(m, E, W, invR, invR2);
          W = in ? W : 0.f;
          E = in ? E : 0.f;
        }
        if (COMPUTE) Ep += E;
        Wp += W;
        const float sc = W * inv2;
        fx = fmaf(sc, dx, fx);
        fy = fmaf(sc, dy, fy);
        fz = fmaf(sc, dz, fz);
      }
      cur = nxt;
    }
    if (TPA == 2) {
      fx += __shfl_xor_sync(pmask, fx, 1);
      fy += __shfl_xor_sync(pmask, fy, 1);
      fz += __shfl_xor_sync(pmask, fz, 1);
    }
    if (sub == 0) {
      const int a = orig[i];
      F[3 * a] = f2d_exact(fx * unit);
      F[3 * a + 1] = f2d_exact(fy * unit);
      F[3 * a + 2] = f2d_exact(fz * unit);
    }
  }
}

// One pass over the atoms between two force evaluations (the boost(dt/2) that ends a step,
// the boost(dt/2) and displace(dt) that begin the next, FP64 with the fused multiply-adds
// of the single-system mixed path, the skin displacement, and the new positions' box
// fractions at their slots).  Without END the first kick is left out, without BEGIN the
// rest.  Each warp takes a contiguous range of atoms, as the skin check's combine needs.
template <int THREADS, bool END, bool BEGIN>
__device__ __forceinline__ void rep_advance(RepShared& S, int4* pos, double dt, bool kinetic) {
  const RepDesc& D = S.d;
  const int N = D.N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = THREADS / 32;
  const double dt_2 = 0.5 * dt;
  const int per = (N + nw - 1) / nw, a0 = warp * per, a1 = min(N, a0 + per);
  double ke[3] = {0.0, 0.0, 0.0};
  RepMP run{-1, -1};
  for (int base = a0; base < a1; base += 32) {
    const int a = base + lane;
    RepMP v{-1, -1};
    if (a < a1) {
      const double im = D.unitMass ? 1.0 : D.invMass[a];
      double dr[3];
      int x[3];
      for (int d = 0; d < 3; d++) {
        const double f = D.F[3 * a + d];
        double p = D.P[3 * a + d];
        if (END) {
          p = fma(dt_2, f, p);
          if (kinetic) ke[d] += im * (p * p);
        }
        if (BEGIN) {
          p = fma(dt_2, f, p);
          const double r = D.unitMass ? fma(dt, p, D.R[3 * a + d]) : fma(dt * p, im, D.R[3 * a + d]);
          D.R[3 * a + d] = r;
          dr[d] = r - D.R0[3 * a + d];
          x[d] = rep_fraction(r, D);
        }
        D.P[3 * a + d] = p;
      }
      if (BEGIN) {
        v.m = __double_as_longlong(fma(dr[2], dr[2], fma(dr[1], dr[1], dr[0] * dr[0])));
        int4* q = &pos[D.slotOf[a]];
        q->x = x[0];
        q->y = x[1];
        q->z = x[2];
      }
    }
    if (BEGIN) run = rep_combine(run, rep_warp_ordered(v));
  }
  if (END && kinetic) {
    for (int d = 0; d < 3; d++)
      for (int o = 16; o > 0; o >>= 1) ke[d] += __shfl_down_sync(0xffffffffu, ke[d], o);
    if (lane == 0)
      for (int d = 0; d < 3; d++) S.wke[d][warp] = ke[d];
  }
  if (BEGIN && lane == 0) S.wmp[warp] = run;
  __syncthreads();
  if (END && kinetic && threadIdx.x < 3) {
    double x = 0.0;
    for (int w = 0; w < nw; w++) x += S.wke[threadIdx.x][w];
    D.out[2 + threadIdx.x] = x;
  }
  if (BEGIN && threadIdx.x == 32) {
    RepMP b = S.wmp[0];
    for (int w = 1; w < nw; w++) b = rep_combine(b, S.wmp[w]);
    const double mx = __longlong_as_double(b.m), nx = __longlong_as_double(b.p < 0 ? b.m : b.p);
    S.rebuild = mx + 2 * sqrt(mx * nx) + nx > D.skinSq;
  }
  __syncthreads();
}

template <int THREADS, int TPA>
__global__ void __launch_bounds__(THREADS) k_replicas(const RepDesc* __restrict__ descs, const int* __restrict__ order,
                                                      int steps, double dt, int nprop, int Nmax, int cellsMax) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ RepShared S;
  int4* pos = (int4*)smem;   // box fractions and type; during a build cell units and cell
  NBParams<float>* ptab = (NBParams<float>*)(pos + Nmax + REP_PAD);   // [ti * ntypes + tj]
  int* cellStart = (int*)(ptab + REP_MAXT * REP_MAXT);
  int* cursor = cellStart + cellsMax + 1;
  if (threadIdx.x == 0) {
    S.d = descs[order[blockIdx.x]];
    S.overflow = 0;
  }
  __syncthreads();
  {
    const int nt = S.d.ntypes;
    for (int q = threadIdx.x; q < nt * nt; q += THREADS) {
      const int ti = q / nt, tj = q % nt;
      ptab[q] = S.d.table[ti * nt + tj].model;   // pair(jtype, itype) for an atom of type ti
    }
  }
  const RepDesc& D = S.d;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = THREADS / 32;
  int done = (int)D.out[7];
  // Lists as the system's were built, from the positions of the last build (R0): those of
  // an earlier run serve if they were made from the same positions, bit for bit, and had
  // room (lists that outgrew it are built again, which reports them in this launch's out).
  bool same = true;
  for (int i = threadIdx.x; i < D.N; i += THREADS) same = same && D.count[i] <= D.cap;
  for (int q = threadIdx.x; q < 3 * D.N; q += THREADS)
    same = same && __double_as_longlong(D.Rb[q]) == __double_as_longlong(D.R0[q]);
  if (!__syncthreads_and(same)) rep_build<THREADS>(S, D.R0, (float4*)pos, cellStart, cursor, false);
  double builds = D.out[5];
  // steps < 0: forces, energy and virial at the current positions only
  const bool evaluate = steps < 0;
  const int nsteps = evaluate ? 1 : steps;
  rep_pack<THREADS>(D, pos);
  __syncthreads();
  bool compute = false;
  for (int k = 0; k < nsteps; k++) {
    const bool kinetic = compute;   // of the step that the pass below ends
    compute = evaluate || (k + 1) % nprop == 0;   // every nprop-th step of this call
    if (!evaluate) {
      if (k == 0) rep_advance<THREADS, false, true>(S, pos, dt, false);
      else rep_advance<THREADS, true, true>(S, pos, dt, kinetic);
      if (S.rebuild) {
        rep_build<THREADS>(S, D.R, (float4*)pos, cellStart, cursor, true);
        rep_pack<THREADS>(D, pos);
        builds += 1.0;
        __syncthreads();
      }
    }
    // pair forces (full lists, no atomics); energies on compute steps, virial every step
    float Ep = 0.f, Wp = 0.f;
    if (D.ljAll) {
      if (compute) rep_pairs<true, true, TPA>(D, pos, ptab, Ep, Wp);
      else rep_pairs<true, false, TPA>(D, pos, ptab, Ep, Wp);
    } else {
      rep_pairs<false, true, TPA>(D, pos, ptab, Ep, Wp);
    }
    {
      float hi[2] = {0.5f * Ep, 0.5f * Wp}, lo[2] = {0.f, 0.f};
      warp_sum_ff<2>(hi, lo);
      if (lane == 0) {
        S.wff[0][warp] = make_float2(hi[0], lo[0]);
        S.wff[1][warp] = make_float2(hi[1], lo[1]);
      }
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      float h = 0.f, l = 0.f;
      for (int w = 0; w < nw; w++) ff_add(h, l, S.wff[threadIdx.x][w].x, S.wff[threadIdx.x][w].y);
      if (threadIdx.x == 1 || compute) D.out[threadIdx.x] = (double)h + (double)l;
    }
  }
  // the boost that ends the last step
  if (!evaluate && nsteps > 0) rep_advance<THREADS, true, false>(S, pos, dt, compute);
  __syncthreads();
  if (threadIdx.x == 0) {
    D.out[5] = builds;
    D.out[6] = (double)S.overflow;
    D.out[7] = (double)(done + (evaluate ? 0 : steps));
  }
}

// ---- host -----------------------------------------------------------------------

struct Replicas {
  std::vector<tEmDee*> md;
  std::vector<System*> sys;
  std::vector<RepDesc> desc;
  RepDesc* dDesc = nullptr;
  int* dOrder = nullptr;
  double* dOut = nullptr;
  double* hOut = nullptr;
  std::vector<void*> owned;
  int n = 0, Nmax = 0, cellsMax = 0, threads = 0, tpa = 1;
  size_t smem = 0;
  cudaStream_t stream = nullptr;
  cudaGraphExec_t graph = nullptr;
  int gSteps = -1, gNprop = -1;
  double gDt = 0.0;
  int steps = 0;
  std::vector<double*> saved;     // checkpoints: R, F, R0 per replica
  std::vector<tEmDee> savedMd;
};

template <int TPA>
static void rep_launch_tpa(Replicas& B, int steps, double dt, int nprop, cudaStream_t st) {
  switch (B.threads) {
    case 256:
      k_replicas<256, TPA><<<B.n, 256, B.smem, st>>>(B.dDesc, B.dOrder, steps, dt, nprop, B.Nmax, B.cellsMax);
      break;
    case 512:
      k_replicas<512, TPA><<<B.n, 512, B.smem, st>>>(B.dDesc, B.dOrder, steps, dt, nprop, B.Nmax, B.cellsMax);
      break;
    default:
      k_replicas<1024, TPA><<<B.n, 1024, B.smem, st>>>(B.dDesc, B.dOrder, steps, dt, nprop, B.Nmax, B.cellsMax);
      break;
  }
}

static void rep_launch(Replicas& B, int steps, double dt, int nprop, cudaStream_t st) {
  if (B.tpa == 2) rep_launch_tpa<2>(B, steps, dt, nprop, st);
  else rep_launch_tpa<1>(B, steps, dt, nprop, st);
  CK(cudaGetLastError());
}

static void rep_set_smem(Replicas& B) {
  const int b = (int)B.smem;
  CK(cudaFuncSetAttribute(k_replicas<256, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  CK(cudaFuncSetAttribute(k_replicas<512, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  CK(cudaFuncSetAttribute(k_replicas<1024, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  CK(cudaFuncSetAttribute(k_replicas<256, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  CK(cudaFuncSetAttribute(k_replicas<512, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
  CK(cudaFuncSetAttribute(k_replicas<1024, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
}

// Chooses the block size and the pair phase's threads per atom by timing a few steps
// of every candidate on scratch copies of the replicas' state (the systems themselves
// are not touched).  The choice is kept per batch shape (the sorted replica sizes and
// type counts) for the life of the process, so batches of the same shape run the same
// configuration and give bit-identical results.
static std::vector<std::pair<std::vector<int>, std::pair<int, int>>> g_repTuned;

static std::vector<int> rep_shape(const Replicas& B) {
  std::vector<int> key;
  for (const RepDesc& d : B.desc) key.push_back(d.N * 16 + d.ntypes);
  std::sort(key.begin(), key.end());
  return key;
}

static void rep_autotune(Replicas& B, double dt, int nprop) {
  const std::vector<int> key = rep_shape(B);
  for (const auto& e : g_repTuned)
    if (e.first == key) {
      B.threads = e.second.first;
      B.tpa = e.second.second;
      return;
    }
  std::vector<RepDesc> scratch = B.desc;
  std::vector<void*> tmp;
  for (int r = 0; r < B.n; r++) {
    RepDesc& d = scratch[r];
    size_t b3 = sizeof(double) * 3 * d.N;
    double *R, *P, *F, *R0, *out;
    CK(cudaMalloc(&R, b3));
    CK(cudaMalloc(&P, b3));
    CK(cudaMalloc(&F, b3));
    CK(cudaMalloc(&R0, b3));
    CK(cudaMalloc(&out, sizeof(double) * 8));
    CK(cudaMemcpyAsync(R, d.R, b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(P, d.P, b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(F, d.F, b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(R0, d.R0, b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(out, d.out, sizeof(double) * 8, cudaMemcpyDeviceToDevice, B.stream));
    d.R = R;
    d.P = P;
    d.F = F;
    d.R0 = R0;
    d.out = out;
    tmp.insert(tmp.end(), {R, P, F, R0, out});
  }
  RepDesc* dScratch;
  CK(cudaMalloc(&dScratch, sizeof(RepDesc) * B.n));
  CK(cudaMemcpyAsync(dScratch, scratch.data(), sizeof(RepDesc) * B.n, cudaMemcpyHostToDevice, B.stream));
  RepDesc* keep = B.dDesc;
  B.dDesc = dScratch;
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  int best = 1024, bestTpa = 1;
  float bestMs = 1e30f;
  for (int cfg = 0; cfg < 6; cfg++) {
    const int th = 256 << (cfg % 3), tpa = 1 + cfg / 3;
    B.threads = th;
    B.tpa = tpa;
    rep_launch(B, 2, dt, nprop, B.stream);   // warm-up
    CK(cudaEventRecord(e0, B.stream));
    rep_launch(B, 10, dt, nprop, B.stream);
    CK(cudaEventRecord(e1, B.stream));
    CK(cudaEventSynchronize(e1));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    if (ms < bestMs) {
      bestMs = ms;
      best = th;
      bestTpa = tpa;
    }
  }
  CK(cudaEventDestroy(e0));
  CK(cudaEventDestroy(e1));
  B.dDesc = keep;
  CK(cudaFree(dScratch));
  for (void* p : tmp) CK(cudaFree(p));
  B.threads = best;
  B.tpa = bestTpa;
  g_repTuned.push_back({key, {best, bestTpa}});
}

}  // namespace emdee

using namespace emdee;

extern "C" {

void* EmDee_replicas_create(int n, tEmDee** systems) {
  const char* task = "replica batch setup";
  if (n < 1 || !systems) fatal(task, "at least one system is required");
  Replicas* B = new Replicas;
  B->n = n;
  CK(cudaStreamCreateWithFlags(&B->stream, cudaStreamNonBlocking));
  CK(cudaMalloc(&B->dOut, sizeof(double) * 8 * n));
  CK(cudaMallocHost(&B->hOut, sizeof(double) * 8 * n));
  CK(cudaMemset(B->dOut, 0, sizeof(double) * 8 * n));
  std::vector<int> order(n);
  for (int r = 0; r < n; r++) {
    tEmDee* md = systems[r];
    System& s = *sys_of(*md);
    if (!s.initialized) fatal(task, "every system must be initialized (box and coordinates uploaded)");
    if (s.ntypes > REP_MAXT || s.nbodies > 0 || s.hasExclusions || s.nlayers != 1 || s.precision != 0)
      fatal(task, "replicas must have at most 8 atom types, no bodies, no exclusions, one layer and mixed precision");
    for (int a = 0; a < s.natoms; a++)
      if (s.charged[a]) fatal(task, "replicas must carry no charges");
    if (s.natoms > 65535) fatal(task, "replicas are limited to 65535 atoms");
    flush_pending(s);
    s.keSpecValid = false;   // the batch moves P and F
    CK(cudaStreamSynchronize(s.stream));
    RepDesc d;
    memset(&d, 0, sizeof d);
    d.R = s.dR;
    d.P = s.dP;
    d.F = s.F();
    d.R0 = s.dR0;
    d.invMass = s.dInvMass;
    d.unitMass = s.unitMass ? 1 : 0;
    d.N = s.natoms;
    const double L = *s.Lbox;
    d.M = std::max((int)std::floor(2.0 * L / s.xRc), 5);
    // a cell edge of exactly (rc + skin) / 2 leaves no room for the fractions' rounding
    if (d.M > 5 && L / d.M < 0.5 * s.xRc * (1.0 + 1e-8)) d.M--;
    d.minimg = d.M == 5;
    d.L = L;
    d.frac = 4294967296.0 / L;
    d.skinSq = s.skinSq;
    d.thr = s.xRcSq / (L * L);
    const double M2 = (double)d.M * d.M;
    d.lo2 = (float)(d.thr * M2 * (1.0 - REP_BAND));
    d.hi2 = (float)(d.thr * M2 * (1.0 + REP_BAND));
    d.rc2 = (float)(s.RcSq * d.frac * d.frac);
    d.unit2 = (float)(d.frac * d.frac);
    d.unit = (float)d.frac;
    d.Mf = (float)d.M;
    CK(cudaMemcpy(&d.model, s.models.d32, sizeof(PairEntry<float>), cudaMemcpyDeviceToHost));
    d.ntypes = s.ntypes;
    d.table = s.models.d32;
    d.ljAll = 1;
    for (int ti = 0; ti < s.ntypes; ti++)
      for (int tj = 0; tj < s.ntypes; tj++) {
        const NBParams<double>& m = s.P(ti, tj, 0).model.p;
        if (!(m.kind == MK_LJ_CUT && m.modifier == NONE)) d.ljAll = 0;
      }
    d.type = s.dType;
    // list capacity: twice the ideal-gas count within rc+skin, at least 64
    const double expect = 4.0 / 3.0 * 3.14159265358979 * std::pow(s.xRc, 3) * s.natoms / (L * L * L);
    d.cap = std::max(64, ((int)(2.0 * expect) + 7) / 8 * 8);   // a multiple of the 8-entry chunk
    CK(cudaMalloc(&d.orig, sizeof(int) * d.N));
    CK(cudaMalloc(&d.slotOf, sizeof(uint16_t) * d.N));
    CK(cudaMalloc(&d.frac4, sizeof(int4) * d.N));
    CK(cudaMalloc(&d.Rb, sizeof(double) * 3 * d.N));
    CK(cudaMemset(d.Rb, 0xFF, sizeof(double) * 3 * d.N));   // no lists yet (NaN)
    CK(cudaMalloc(&d.list, sizeof(uint16_t) * (size_t)d.cap * d.N));
    CK(cudaMalloc(&d.count, sizeof(int) * d.N));
    B->owned.insert(B->owned.end(), {d.orig, d.slotOf, d.frac4, d.Rb, d.list, d.count});
    d.out = B->dOut + 8 * r;
    B->desc.push_back(d);
    B->md.push_back(md);
    B->sys.push_back(&s);
    B->Nmax = std::max(B->Nmax, d.N);
    B->cellsMax = std::max(B->cellsMax, d.M * d.M * d.M);
    order[r] = r;
  }
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return B->desc[a].N > B->desc[b].N; });
  B->smem = sizeof(int4) * ((size_t)B->Nmax + REP_PAD) + sizeof(NBParams<float>) * REP_MAXT * REP_MAXT +
            sizeof(int) * (2 * (size_t)B->cellsMax + 1);
  // the limit of 125 stencil offsets and a type byte per atom besides is kept
  if (B->smem + sizeof(float4) * (125 - REP_PAD) + (size_t)B->Nmax > 227 * 1024) fatal(task, "the largest replica does not fit in one block's shared memory");
  CK(cudaMalloc(&B->dDesc, sizeof(RepDesc) * n));
  CK(cudaMemcpy(B->dDesc, B->desc.data(), sizeof(RepDesc) * n, cudaMemcpyHostToDevice));
  CK(cudaMalloc(&B->dOrder, sizeof(int) * n));
  CK(cudaMemcpy(B->dOrder, order.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
  rep_set_smem(*B);
  // EMDEE_REPLICA_THREADS=threads[,pair threads per atom] fixes the configuration
  const char* e = getenv("EMDEE_REPLICA_THREADS");
  B->threads = e ? atoi(e) : 0;
  if (B->threads != 256 && B->threads != 512 && B->threads != 1024) B->threads = 0;
  const char* comma = e ? strchr(e, ',') : nullptr;
  B->tpa = comma && atoi(comma + 1) == 2 ? 2 : 1;
  return B;
}

// Advances every replica by `steps` velocity-Verlet steps of dt, energies at every
// nprop-th step of the call, and writes each system's results back.
void EmDee_replicas_run(void* batch, int steps, double dt, int nprop) {
  const char* task = "replica batch run";
  Replicas& B = *(Replicas*)batch;
  if (steps < 0 || nprop < 1) fatal(task, "invalid number of steps");
  for (System* s : B.sys) {
    flush_pending(*s);
    s->keSpecValid = false;
    CK(cudaStreamSynchronize(s->stream));
  }
  if (B.threads == 0) rep_autotune(B, dt, nprop);
  if (steps == 0) return;
  if (!B.graph || B.gSteps != steps || B.gDt != dt || B.gNprop != nprop) {
    if (B.graph) CK(cudaGraphExecDestroy(B.graph));
    cudaGraph_t g;
    CK(cudaStreamBeginCapture(B.stream, cudaStreamCaptureModeThreadLocal));
    rep_launch(B, steps, dt, nprop, B.stream);
    CK(cudaMemcpyAsync(B.hOut, B.dOut, sizeof(double) * 8 * B.n, cudaMemcpyDeviceToHost, B.stream));
    CK(cudaStreamEndCapture(B.stream, &g));
    CK(cudaGraphInstantiate(&B.graph, g, 0));
    CK(cudaGraphDestroy(g));
    B.gSteps = steps;
    B.gDt = dt;
    B.gNprop = nprop;
  }
  CK(cudaGraphLaunch(B.graph, B.stream));
  CK(cudaStreamSynchronize(B.stream));
  B.steps += steps;
  const bool computeLast = steps % nprop == 0;
  for (int r = 0; r < B.n; r++) {
    const double* o = &B.hOut[8 * r];
    if (o[6] > 0) fatal(task, "a neighbor list outgrew its capacity");
    tEmDee* md = B.md[r];
    System& s = *B.sys[r];
    md->Builds += (int)o[5];
    md->Virial.Total = o[1];
    md->Virial.Body = 0.0;
    if (computeLast) {
      md->Energy.Dispersion = o[0];
      md->Energy.Coulomb = 0.0;
      md->Energy.Bond = 0.0;
      md->Energy.Angle = 0.0;
      md->Energy.Potential = o[0];
      md->Energy.ShadowPotential = o[0];
      for (int d = 0; d < 3; d++) {
        md->Kinetic.TransPart[d] = 0.5 * o[2 + d];
        md->Kinetic.RotPart[d] = 0.0;
      }
      md->Kinetic.Rotational = 0.0;
      md->Kinetic.Total = md->Kinetic.TransPart[0] + md->Kinetic.TransPart[1] + md->Kinetic.TransPart[2];
    }
    md->Energy.UpToDate = computeLast;
    md->Kinetic.UpToDate = computeLast;
    // the forces belong to the current positions; the system's own lists are
    // older than R0 now, so its next force computation rebuilds them
    s.forcesUpToDate[0] = 1;
    s.layerEnergy[0] = md->Energy;
    s.layerVirial[0] = md->Virial;
    s.r0Valid = false;
  }
  // device results: counters restart; the device keeps the total step count
  std::vector<double> reset((size_t)8 * B.n, 0.0);
  for (int r = 0; r < B.n; r++) reset[8 * r + 7] = (double)B.steps;
  CK(cudaMemcpy(B.dOut, reset.data(), sizeof(double) * reset.size(), cudaMemcpyHostToDevice));
}

int EmDee_replicas_block_size(void* batch) { return ((Replicas*)batch)->threads; }

int EmDee_replicas_pair_threads(void* batch) { return ((Replicas*)batch)->tpa; }

// Forces, potential energy and virial of every replica at its current positions (lists
// rebuilt from them, which then become the build positions R0); no step is taken and no
// build is counted.  Energy and Virial are written back into each tEmDee.
void EmDee_replicas_evaluate(void* batch) {
  Replicas& B = *(Replicas*)batch;
  for (System* s : B.sys) {
    flush_pending(*s);
    s->keSpecValid = false;
    CK(cudaStreamSynchronize(s->stream));
  }
  if (B.threads == 0) B.threads = 1024;
  for (int r = 0; r < B.n; r++)
    CK(cudaMemcpyAsync(B.desc[r].R0, B.desc[r].R, sizeof(double) * 3 * B.desc[r].N, cudaMemcpyDeviceToDevice,
                       B.stream));
  rep_launch(B, -1, 0.0, 1, B.stream);
  CK(cudaMemcpyAsync(B.hOut, B.dOut, sizeof(double) * 8 * B.n, cudaMemcpyDeviceToHost, B.stream));
  CK(cudaStreamSynchronize(B.stream));
  for (int r = 0; r < B.n; r++) {
    const double* o = &B.hOut[8 * r];
    if (o[6] > 0) fatal("replica batch evaluation", "a neighbor list outgrew its capacity");
    tEmDee* md = B.md[r];
    md->Energy.Dispersion = o[0];
    md->Energy.Coulomb = md->Energy.Bond = md->Energy.Angle = 0.0;
    md->Energy.Potential = md->Energy.ShadowPotential = o[0];
    md->Energy.UpToDate = true;
    md->Virial.Total = o[1];
    md->Virial.Body = 0.0;
    System& s = *B.sys[r];
    s.forcesUpToDate[0] = 1;
    s.layerEnergy[0] = md->Energy;
    s.layerVirial[0] = md->Virial;
    s.r0Valid = false;
  }
  std::vector<double> reset((size_t)8 * B.n, 0.0);
  for (int r = 0; r < B.n; r++) reset[8 * r + 7] = (double)B.steps;
  CK(cudaMemcpy(B.dOut, reset.data(), sizeof(double) * reset.size(), cudaMemcpyHostToDevice));
}

// Copies item ("coordinates", "momenta" or "forces") of every replica into / from one
// contiguous device array [n][N][3] (replicas of equal size), on the batch stream.
static double* rep_item(RepDesc& d, const char* item) {
  if (!strcmp(item, "coordinates")) return d.R;
  if (!strcmp(item, "momenta")) return d.P;
  if (!strcmp(item, "forces")) return d.F;
  fatal("replica batch copy", "unknown item");
}

void EmDee_replicas_gather(void* batch, const char* item, double* dst) {
  Replicas& B = *(Replicas*)batch;
  for (System* sy : B.sys) {
    flush_pending(*sy);
    sy->keSpecValid = false;
  }
  size_t off = 0;
  for (int r = 0; r < B.n; r++) {
    const size_t n = (size_t)3 * B.desc[r].N;
    CK(cudaMemcpyAsync(dst + off, rep_item(B.desc[r], item), sizeof(double) * n, cudaMemcpyDeviceToDevice, B.stream));
    off += n;
  }
  CK(cudaStreamSynchronize(B.stream));
}

void EmDee_replicas_scatter(void* batch, const char* item, const double* src) {
  Replicas& B = *(Replicas*)batch;
  for (System* sy : B.sys) {
    flush_pending(*sy);
    sy->keSpecValid = false;
  }
  size_t off = 0;
  for (int r = 0; r < B.n; r++) {
    const size_t n = (size_t)3 * B.desc[r].N;
    CK(cudaMemcpyAsync(rep_item(B.desc[r], item), src + off, sizeof(double) * n, cudaMemcpyDeviceToDevice, B.stream));
    off += n;
  }
  CK(cudaStreamSynchronize(B.stream));
}

// Saves (R, F, R0, Energy, Virial) of every replica; EmDee_replicas_restore puts them back for
// the replicas whose mask entry is nonzero (Metropolis rejections in hybrid Monte Carlo)
void EmDee_replicas_checkpoint(void* batch) {
  Replicas& B = *(Replicas*)batch;
  for (System* sy : B.sys) {
    flush_pending(*sy);
    sy->keSpecValid = false;
  }
  if (B.saved.empty()) {
    for (int r = 0; r < B.n; r++) {
      double* p;
      CK(cudaMalloc(&p, sizeof(double) * 9 * B.desc[r].N));
      B.saved.push_back(p);
    }
    B.savedMd.resize(B.n);
  }
  for (int r = 0; r < B.n; r++) {
    const size_t b3 = sizeof(double) * 3 * B.desc[r].N;
    CK(cudaMemcpyAsync(B.saved[r], B.desc[r].R, b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(B.saved[r] + 3 * B.desc[r].N, B.desc[r].F, b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(B.saved[r] + 6 * B.desc[r].N, B.desc[r].R0, b3, cudaMemcpyDeviceToDevice, B.stream));
    B.savedMd[r] = *B.md[r];
  }
  CK(cudaStreamSynchronize(B.stream));
}

void EmDee_replicas_restore(void* batch, const int* mask) {
  Replicas& B = *(Replicas*)batch;
  if (B.saved.empty()) fatal("replica batch restore", "no checkpoint has been taken");
  for (int r = 0; r < B.n; r++) {
    if (!mask[r]) continue;
    const size_t b3 = sizeof(double) * 3 * B.desc[r].N;
    CK(cudaMemcpyAsync(B.desc[r].R, B.saved[r], b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(B.desc[r].F, B.saved[r] + 3 * B.desc[r].N, b3, cudaMemcpyDeviceToDevice, B.stream));
    CK(cudaMemcpyAsync(B.desc[r].R0, B.saved[r] + 6 * B.desc[r].N, b3, cudaMemcpyDeviceToDevice, B.stream));
    tEmDee* md = B.md[r];
    const int builds = md->Builds;
    md->Energy = B.savedMd[r].Energy;
    md->Virial = B.savedMd[r].Virial;
    md->Builds = builds;
  }
  CK(cudaStreamSynchronize(B.stream));
}

void EmDee_replicas_destroy(void* batch) {
  Replicas* B = (Replicas*)batch;
  if (!B) return;
  cudaStreamSynchronize(B->stream);
  if (B->graph) cudaGraphExecDestroy(B->graph);
  for (void* p : B->owned) cudaFree(p);
  for (double* p : B->saved) cudaFree(p);
  cudaFree(B->dDesc);
  cudaFree(B->dOrder);
  cudaFree(B->dOut);
  cudaFreeHost(B->hOut);
  cudaStreamDestroy(B->stream);
  delete B;
}

}  // extern "C"
