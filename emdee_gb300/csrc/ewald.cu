// ewald.cu -- Ewald k-space electrostatics for coul_long (src/kspace_ewald.f90,
// src/modelClass_kspace.f90, src/coul_long.f90).
//
// Host: the reference's set-up, statement by statement (alpha and kmax from the
// accuracy, the half k-lattice inside the sphere of radius nmax * 2pi/L, the
// prefactors, the charge list by type, the rigid-pair and self-energy
// discounts, the Coulomb constants per type pair and layer).
// Device, FP64.  Both sums are bound by the FP64 pipe (2 FMA per clock per SM), so
// the kernels are built around the fewest FP64 operations per atom and k-vector and
// an even spread over the SMs.  The k-vectors come in rows (n1, n2) with
// n3 = -z..z; with a = q exp(i(n1 x + n2 y)) computed once per row and g = exp(i m z),
// the products Re a Re g, Im a Im g, Re a Im g, Im a Re g serve both n3 = m and
// n3 = -m: 2 FMAs per k-vector in the structure factors, 4 in the forces (about 16
// and 22 operations when every k-vector is evaluated by itself).
//   k_ewald_tables the powers exp(i 2pi m x_d / L), m = 0..nmax, of every charged
//                  atom, by the reference's complex recursion (charge included in x)
//   k_ewald_sf     one block per group of tasks (row, 4 values of m) and chunk of
//                  charged atoms of one type: the chunk's partial structure factors
//   k_ewald_sigma  per pair of k-vectors (m, -m): S summed over the type's chunks in
//                  order, sigma(k, t) = sum_u S(k, u) lambda(u, t), energy terms
//                  prefac(k) sum_t Re(S conj-free dot sigma), grid reduction; the
//                  four coefficients per (row, m) that the forces need
//   k_ewald_force  a few atoms per block, the rows spread over 32 threads per atom:
//                  F += sum_k vec(k) (Re sigma Im qe - Re qe Im sigma), added to the
//                  pair forces (no atomics: one thread per component)
// Every sum has a fixed order (atoms of a chunk, chunks, rows of a thread, threads),
// so results do not depend on scheduling.
// 3,000 charges, nmax 12 (1000 water molecules, accuracy 1e-6): structure factors 2395
// -> 77 us, forces 3528 -> 97 us (about 46 and 80 us at the pipe's peak).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "reduce.cuh"
#include "system.hpp"

namespace emdee {

static const double EW_PI = 3.14159265358979324;
// structure factors: tasks per block, values of m per task, charged atoms staged at a time
static const int SF_THREADS = 192, SF_M = 4, SF_ATOMS = 16;
// Forces: atoms per block and threads per atom.  Small blocks of equal work: 3,000 atoms
// give 750 blocks, 4.9 per SM, so that the last round of blocks costs little.
static const int FORCE_ATOMS = 4, FORCE_SPLIT = 32;
// Atoms whose power tables a block held when the k-vectors per dimension were limited
// to what fits: the limit is kept.
static const int TABLE_LIMIT_ATOMS = 64;

struct EwArgs {
  const double* R;
  double invL;   // 1 / current box length (theta = 2 pi R / L)
  double unit2;  // 2 * 2 pi / L of the set-up: vec(k) = unit2 prefac(k) n
  int nq, nvecs, nmax, ntypes, ntasks, nrows, npairs, nchunks;
  const int* item;
  const int* qtype;
  const double* value;
  const int4* task;     // n1, n2, first m, row
  const int4* row;      // n1, n2, z, first pair; rows in descending z
  const int2* pair;     // per (row, m = 0..z): k-vectors with n3 = m and n3 = -m (-1: none)
  const int4* chunk;    // first atom, last + 1, type
  const int* typeChunk;  // per type: its chunks [typeChunk[t], typeChunk[t + 1])
  const double* prefac;
  const double* lambda;   // this layer: [t][u]
  double2* table;         // [d][m][atom]
  double2* partial;       // [chunk][v]
  double2* coef;          // [t][pair][2]: (U, V), (X, Y)
  double* F;
  double* epart;
  unsigned int* ticket;
  double* result;
  double* hostResult;
  const double* skip;   // if set and *skip != 0 (a rebuild is due), the launches do nothing
};

__device__ __forceinline__ bool skipped(const EwArgs& A) {
  return A.skip != nullptr && __double_as_longlong(*A.skip) != 0;
}

// powers exp(i 2pi m x / L), m = 0..nm, of every coordinate of the charged atoms
// (src/kspace_ewald.f90:205-243: B = Z; G(j) = B; B = B*Z); those of x times the charge
__global__ void __launch_bounds__(128) k_ewald_tables(EwArgs A) {
  if (skipped(A)) return;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 3 * A.nq) return;
  const int d = k / A.nq, j = k - d * A.nq;
  const double q = d == 0 ? A.value[j] : 1.0;
  const double theta = 6.28318530717958648 * (A.R[3 * A.item[j] + d] * A.invL);
  double zi, zr;
  sincos(theta, &zi, &zr);
  double2* out = A.table + (size_t)d * (A.nmax + 1) * A.nq + j;
  out[0] = make_double2(q, 0.0);
  double br = zr, bi = zi;
  for (int m = 1; m <= A.nmax; m++) {
    out[(size_t)m * A.nq] = make_double2(q * br, q * bi);
    const double nr = br * zr - bi * zi, ni = br * zi + bi * zr;
    br = nr;
    bi = ni;
  }
}

// a = G1 G2 (conjugated for negative n2)
__device__ __forceinline__ double2 row_phase(double2 gx, double2 gy, int n2) {
  const double gyi = n2 < 0 ? -gy.y : gy.y;
  return make_double2(fma(gx.x, gy.x, -(gx.y * gyi)), fma(gx.x, gyi, gx.y * gy.x));
}

__global__ void __launch_bounds__(SF_THREADS) k_ewald_sf(EwArgs A) {
  if (skipped(A)) return;
  extern __shared__ __align__(16) unsigned char smem[];
  double2* T = (double2*)smem;   // [atom][d][m], an odd number of entries per atom
  const int rows = A.nmax + 1, W = 3 * rows, S = W | 1;
  const int ti = blockIdx.x * SF_THREADS + threadIdx.x;
  const bool active = ti < A.ntasks;
  const int4 task = active ? A.task[ti] : make_int4(0, 0, 1, 0);
  const int4 ch = A.chunk[blockIdx.y];
  const int ox = task.x, oy = rows + abs(task.y);
  int oz[SF_M];
#pragma unroll
  for (int u = 0; u < SF_M; u++) oz[u] = 2 * rows + min(task.z + u, A.nmax);
  double s0r = 0.0, s0i = 0.0, rr[SF_M], ii[SF_M], ri[SF_M], ir[SF_M];
#pragma unroll
  for (int u = 0; u < SF_M; u++) rr[u] = ii[u] = ri[u] = ir[u] = 0.0;
  for (int a0 = ch.x; a0 < ch.y; a0 += SF_ATOMS) {
    const int na = min(SF_ATOMS, ch.y - a0);
    __syncthreads();
    for (int k = threadIdx.x; k < W * SF_ATOMS; k += SF_THREADS) {
      const int e = k / SF_ATOMS, a = k % SF_ATOMS;
      if (a < na) T[a * S + e] = A.table[(size_t)e * A.nq + a0 + a];
    }
    __syncthreads();
    if (!active) continue;
    for (int a = 0; a < na; a++) {
      const double2* t = T + a * S;
      const double2 c = row_phase(t[ox], t[oy], task.y);
      if (task.z == 1) {
        s0r += c.x;
        s0i += c.y;
      }
#pragma unroll
      for (int u = 0; u < SF_M; u++) {
        const double2 g = t[oz[u]];
        rr[u] = fma(c.x, g.x, rr[u]);
        ii[u] = fma(c.y, g.y, ii[u]);
        ri[u] = fma(c.x, g.y, ri[u]);
        ir[u] = fma(c.y, g.x, ir[u]);
      }
    }
  }
  if (!active) return;
  const int4 row = A.row[task.w];
  double2* out = A.partial + (size_t)blockIdx.y * A.nvecs;
  if (task.z == 1) {
    const int v = A.pair[row.w].x;
    if (v >= 0) out[v] = make_double2(s0r, s0i);
  }
#pragma unroll
  for (int u = 0; u < SF_M; u++) {
    const int m = task.z + u;
    if (m > row.z) break;
    const int2 v = A.pair[row.w + m];
    if (v.x >= 0) out[v.x] = make_double2(rr[u] - ii[u], ri[u] + ir[u]);
    if (v.y >= 0) out[v.y] = make_double2(rr[u] + ii[u], ir[u] - ri[u]);
  }
}

static const int EW_MAXT = 16;   // charged atom types handled by the k-space kernels
// A block sums the chunks of SIGMA_PAIRS pairs in SIGMA_SLICES slices, then a thread per
// pair and type forms the coefficients.  Latency of loads and of the FP64 unit: 32 pairs in
// 8 slices and one thread for all types of a pair ran on few SMs (23 us at 1000 molecules,
// 8 pairs in 16 slices 17).
static const int SIGMA_PAIRS = 8, SIGMA_SLICES = 16;

__global__ void __launch_bounds__(SIGMA_PAIRS * SIGMA_SLICES) k_ewald_sigma(EwArgs A) {
  if (skipped(A)) return;
  __shared__ double part[SIGMA_SLICES][4][SIGMA_PAIRS];
  __shared__ double Ss[EW_MAXT][4][SIGMA_PAIRS];
  const int x = threadIdx.x % SIGMA_PAIRS, y = threadIdx.x / SIGMA_PAIRS;
  const int p = blockIdx.x * SIGMA_PAIRS + x;
  const int2 v = p < A.npairs ? A.pair[p] : make_int2(-1, -1);
  for (int u = 0; u < A.ntypes; u++) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    const double2 none = make_double2(0.0, 0.0);
    for (int c = A.typeChunk[u] + y; c < A.typeChunk[u + 1]; c += SIGMA_SLICES) {
      const double2* in = A.partial + (size_t)c * A.nvecs;
      const double2 a = v.x >= 0 ? in[v.x] : none, b = v.y >= 0 ? in[v.y] : none;
      s[0] += a.x;
      s[1] += a.y;
      s[2] += b.x;
      s[3] += b.y;
    }
    for (int k = 0; k < 4; k++) part[y][k][x] = s[k];
    __syncthreads();
    if (y < 4) {
      double t = 0.0;
      for (int k = 0; k < SIGMA_SLICES; k++) t += part[k][y][x];
      Ss[u][y][x] = t;
    }
    __syncthreads();
  }
  double e[1] = {0.0};
  if (p < A.npairs) {
    const double pp = v.x >= 0 ? A.prefac[v.x] : 0.0, pm = v.y >= 0 ? A.prefac[v.y] : 0.0;
    const double wp = A.unit2 * pp, wm = A.unit2 * pm;
    for (int t = y; t < A.ntypes; t += SIGMA_SLICES) {
      double s[4] = {0.0, 0.0, 0.0, 0.0};
      for (int u = 0; u < A.ntypes; u++) {
        const double lam = A.lambda[t * A.ntypes + u];
        for (int k = 0; k < 4; k++) s[k] = fma(Ss[u][k][x], lam, s[k]);
      }
      const double dp = fma(Ss[t][0][x], s[0], Ss[t][1][x] * s[1]), dm = fma(Ss[t][2][x], s[2], Ss[t][3][x] * s[3]);
      const double ar = wp * s[0], ai = wp * s[1], br = wm * s[2], bi = wm * s[3];
      double2* out = A.coef + ((size_t)t * A.npairs + p) * 2;
      out[0] = make_double2(ar + br, ai - bi);
      out[1] = make_double2(ar - br, ai + bi);
      e[0] = fma(pp, dp, fma(pm, dm, e[0]));
    }
  }
  grid_reduce<1, SIGMA_PAIRS * SIGMA_SLICES>(e, A.epart, A.ticket, A.result, A.hostResult);
}

// With rho = unit2 prefac sigma, a row adds to (x, y, z) the values n1 Im(a H0),
// n2 Im(a H0) and Im(a H1), H0 = sum conj(rho) g^n3, H1 = sum n3 conj(rho) g^n3.  Of
// n3 = m and n3 = -m together, with g = exp(i m z) and the sums and differences
// U = Re(rho+ + rho-), V = Im(rho+ - rho-), X = Re(rho+ - rho-), Y = Im(rho+ + rho-):
//   H0 += (U gr + V gi, X gi - Y gr),  H1 += m (X gr + Y gi, U gi - V gr).
__global__ void __launch_bounds__(FORCE_ATOMS * FORCE_SPLIT) k_ewald_force(EwArgs A) {
  if (skipped(A)) return;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[3][FORCE_SPLIT][FORCE_ATOMS];
  const int rows = A.nmax + 1;
  double2* T = (double2*)smem;   // [d][m][atom], then m times the powers of z
  double2* Tm = T + 3 * rows * FORCE_ATOMS;
  const int a = threadIdx.x % FORCE_ATOMS, split = threadIdx.x / FORCE_ATOMS, j = blockIdx.x * FORCE_ATOMS + a;
  const bool active = j < A.nq;
  for (int e = split; e < 3 * rows; e += FORCE_SPLIT) {
    const double2 g = active ? A.table[(size_t)e * A.nq + j] : make_double2(0.0, 0.0);
    T[e * FORCE_ATOMS + a] = g;
    if (e >= 2 * rows) {
      const double m = (double)(e - 2 * rows);
      Tm[(e - 2 * rows) * FORCE_ATOMS + a] = make_double2(m * g.x, m * g.y);
    }
  }
  __syncthreads();
  const double2* coef = A.coef + (size_t)(active ? A.qtype[j] : 0) * A.npairs * 2;
  double f0 = 0.0, f1 = 0.0, f2 = 0.0;
  for (int r = split; r < A.nrows; r += FORCE_SPLIT) {
    const int4 row = __ldg(&A.row[r]);
    const double2 c = row_phase(T[row.x * FORCE_ATOMS + a], T[(rows + abs(row.y)) * FORCE_ATOMS + a], row.y);
    const double2* w = coef + 2 * row.w;
    double h0r = __ldg(&w[0]).x, h0i = -__ldg(&w[1]).y, h1r = 0.0, h1i = 0.0;
#pragma unroll 2
    for (int m = 1; m <= row.z; m++) {
      const double2 g = T[(2 * rows + m) * FORCE_ATOMS + a], gm = Tm[m * FORCE_ATOMS + a];
      const double2 uv = __ldg(&w[2 * m]), xy = __ldg(&w[2 * m + 1]);
      h0r = fma(uv.x, g.x, fma(uv.y, g.y, h0r));
      h0i = fma(xy.x, g.y, fma(-xy.y, g.x, h0i));
      h1r = fma(xy.x, gm.x, fma(xy.y, gm.y, h1r));
      h1i = fma(uv.x, gm.y, fma(-uv.y, gm.x, h1i));
    }
    const double x = fma(c.x, h0i, c.y * h0r);
    f0 = fma((double)row.x, x, f0);
    f1 = fma((double)row.y, x, f1);
    f2 = fma(c.x, h1i, fma(c.y, h1r, f2));
  }
  red[0][split][a] = f0;
  red[1][split][a] = f1;
  red[2][split][a] = f2;
  __syncthreads();
  if (threadIdx.x < 3 * FORCE_ATOMS && active) {   // thread d * FORCE_ATOMS + a: component d of atom a
    double f = 0.0;
    for (int k = 0; k < FORCE_SPLIT; k++) f += red[split][k][a];
    A.F[3 * A.item[j] + split] += f;
  }
}

// ---- host -----------------------------------------------------------------------

static int symm1D(int i, int j) {   // src/math.f90:695-702 (1-based)
  int x = std::min(i, j) - 1, y = std::max(i, j) - 1;
  return x + (y + 1) * y / 2 + 1;
}

static double inverse_of_x_plus_ln_x(double y) {   // src/math.f90:642-657
  const double tol = 1.0e-12;
  double x = y > 0.5671432904097839 ? y - std::log(y) : std::exp(y);
  double x0 = x + 1.0;
  while (std::fabs(x - x0) > tol * x0) {
    x0 = x;
    x = x * (y + 1.0 - std::log(x)) / (x + 1.0);
  }
  return x;
}

// src/kspace_ewald.f90:107-170 for a cubic box of edge L
static void ewald_update(Ewald& e, double L) {
  const double unit = 2.0 * EW_PI / L, unitSq = unit * unit;
  const int nmax = (int)std::ceil(e.kmax / unit);
  if (nmax != e.nmax) {
    e.nmax = nmax;
    const long M = 2 * nmax + 1, maxnvecs = M * M * M / 2, M2 = M, M2M3 = M * M;
    const double kmaxSq = unitSq * nmax * nmax;
    e.n.clear();
    for (long i = maxnvecs + 1; i <= 2 * maxnvecs; i++) {
      const long n1 = i / M2M3, j = i - n1 * M2M3, n2 = j / M2, n3 = j - n2 * M2;
      const int k0 = (int)n1 - nmax, k1 = (int)n2 - nmax, k2 = (int)n3 - nmax;
      if (unitSq * k0 * k0 + unitSq * k1 * k1 + unitSq * k2 * k2 <= kmaxSq) {
        e.n.push_back(k0);
        e.n.push_back(k1);
        e.n.push_back(k2);
      }
    }
    e.nvecs = (int)(e.n.size() / 3);
    e.prefac.assign(e.nvecs, 0.0);
    const double B = -0.25 / (e.alpha * e.alpha);
    e.Volume = L * L * L;
    const double fourPiByV = 4.0 * EW_PI / e.Volume;
    for (int v = 0; v < e.nvecs; v++) {
      const double k[3] = {unit * e.n[3 * v], unit * e.n[3 * v + 1], unit * e.n[3 * v + 2]};
      const double ksq = k[0] * k[0] + k[1] * k[1] + k[2] * k[2];
      e.prefac[v] = fourPiByV * std::exp(ksq * B) / ksq;
    }
    e.unit = unit;
  } else {
    const double factor = e.Volume / (L * L * L);
    for (int v = 0; v < e.nvecs; v++) e.prefac[v] = factor * e.prefac[v];
    e.Volume = L * L * L;
  }
  e.L = L;
}

void ewald_free(System& s) {
  Ewald& e = s.ewald;
  cudaFree(e.dItem);
  cudaFree(e.dQType);
  cudaFree(e.dValue);
  cudaFree(e.dTask);
  cudaFree(e.dRow);
  cudaFree(e.dPair);
  cudaFree(e.dChunk);
  cudaFree(e.dTypeChunk);
  cudaFree(e.dPrefac);
  cudaFree(e.dLambda);
  cudaFree(e.dTable);
  cudaFree(e.dPartial);
  cudaFree(e.dCoef);
  cudaFree(e.dEnergyPartial);
  e.dItem = e.dQType = e.dTypeChunk = nullptr;
  e.dValue = e.dPrefac = e.dLambda = e.dEnergyPartial = nullptr;
  e.dTask = e.dRow = e.dChunk = nullptr;
  e.dPair = nullptr;
  e.dTable = e.dPartial = e.dCoef = nullptr;
}

template <typename T>
static T* upload_vec(const std::vector<T>& h) {
  T* d = nullptr;
  CK(cudaMalloc(&d, sizeof(T) * std::max<size_t>(h.size(), 1)));
  if (!h.empty()) CK(cudaMemcpy(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
  return d;
}

// Rows, pairs, tasks and chunks of the k-space sums (see the head of this file).  The
// k-vectors of a row are consecutive in e.n, n3 ascending.
static void ewald_plan(Ewald& e) {
  std::vector<int4> row;
  std::vector<int2> pair;
  for (int v = 0; v < e.nvecs;) {
    int w = v;
    while (w < e.nvecs && e.n[3 * w] == e.n[3 * v] && e.n[3 * w + 1] == e.n[3 * v + 1]) w++;
    row.push_back(make_int4(e.n[3 * v], e.n[3 * v + 1], e.n[3 * (w - 1) + 2], v));
    v = w;
  }
  std::stable_sort(row.begin(), row.end(), [](const int4& a, const int4& b) { return a.z > b.z; });
  int zmax = 0;
  for (int4& r : row) {
    const int v0 = r.w, n0 = e.n[3 * v0 + 2];   // first k-vector of the row and its n3 (-z, or 1 in the row 0, 0)
    r.w = (int)pair.size();
    for (int m = 0; m <= r.z; m++)
      pair.push_back(make_int2(m >= n0 ? v0 + m - n0 : -1, m > 0 && -m >= n0 ? v0 - m - n0 : -1));
    zmax = std::max(zmax, r.z);
  }
  std::vector<int4> task;
  for (int m = 1; m <= std::max(zmax, 1); m += SF_M)
    for (int r = 0; r < (int)row.size(); r++)
      if (row[r].z >= m || m == 1) task.push_back(make_int4(row[r].x, row[r].y, m, r));
  e.nrows = (int)row.size();
  e.npairs = (int)pair.size();
  e.ntasks = (int)task.size();
  // Chunks of atoms of one type: with the task groups about four blocks per SM, at
  // least 8 atoms in a chunk
  const int groups = std::max(1, (e.ntasks + SF_THREADS - 1) / SF_THREADS);
  const int want = std::max(1, std::min(e.nq / 8, 4 * 152 / groups));
  std::vector<int4> chunk;
  std::vector<int> typeChunk;
  for (int t = 0; t < e.ntypes; t++) {
    typeChunk.push_back((int)chunk.size());
    const int n = e.last[t] - e.first[t];
    const int c = std::max(1, std::min(n, (int)((long)want * n / e.nq)));
    for (int k = 0; k < c; k++)
      chunk.push_back(make_int4(e.first[t] + (int)((long)n * k / c), e.first[t] + (int)((long)n * (k + 1) / c), t, 0));
  }
  typeChunk.push_back((int)chunk.size());
  e.nchunks = (int)chunk.size();
  e.dRow = upload_vec(row);
  e.dPair = upload_vec(pair);
  e.dTask = upload_vec(task);
  e.dChunk = upload_vec(chunk);
  e.dTypeChunk = upload_vec(typeChunk);
}

// src/modelClass_kspace.f90:111-243 and src/EmDeeData.f90:403-412
void ewald_initialize(System& s, double kspaceRc) {
  const char* task = "kspace model initialization";
  Ewald& e = s.ewald;
  ewald_free(s);
  e = Ewald();
  const int N = s.natoms;
  const double eps = 2.220446049250313e-16;
  std::vector<char> charged(N);
  int ncharged = 0, maxType = 0;
  for (int i = 0; i < N; i++) {
    charged[i] = std::fabs(s.charge[i]) > eps;
    if (charged[i]) {
      ncharged++;
      maxType = std::max(maxType, s.atomType[i]);
    }
  }
  if (ncharged == 0) fatal(task, "system has no charged atoms");
  std::vector<char> present(maxType + 1, 0);
  for (int i = 0; i < N; i++)
    if (charged[i]) present[s.atomType[i]] = 1;
  std::vector<int> local(maxType + 1, 0);
  for (int t = 1; t <= maxType; t++)
    if (present[t]) {
      e.type.push_back(t);
      local[t] = (int)e.type.size();
    }
  e.ntypes = (int)e.type.size();
  if (e.ntypes > EW_MAXT) fatal(task, "more than 16 types of charged atoms");
  // charge list: every atom of each charged type, type by type
  for (int t = 0; t < e.ntypes; t++) {
    e.first.push_back((int)e.item.size());
    for (int i = 0; i < N; i++)
      if (s.atomType[i] == e.type[t]) {
        e.item.push_back(i);
        e.qtype.push_back(t);
        e.value.push_back(s.charge[i]);
      }
    e.last.push_back((int)e.item.size());
  }
  e.nq = (int)e.item.size();
  // src/kspace_ewald.f90:82-103
  const double acc = s.kspace.accuracy;
  const double sp = std::sqrt(inverse_of_x_plus_ln_x(-std::log(acc)));
  e.alpha = sp / kspaceRc;
  e.kmax = 2.0 * e.alpha * sp;
  printf("KSPACE PARAMETERS: alpha = %10.5f and kmax = %10.5f\n", e.alpha, e.kmax);
  fflush(stdout);
  e.beta = 2.0 * e.alpha / std::sqrt(EW_PI);
  // rigid pairs (positions at initialization) and self energy
  e.nTypePairs = e.ntypes * (e.ntypes - 1) / 2 + e.ntypes;
  e.Erigid.assign(e.nTypePairs, 0.0);
  const double L = *s.Lbox, invL = 1.0 / L;
  std::vector<double> R((size_t)3 * N);
  CK(cudaMemcpy(R.data(), s.dR, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost));
  for (int b = 0; b < s.nbodies; b++) {
    const BodyState& B = s.hBodies[b];
    for (int ii = 0; ii < B.NP - 1; ii++) {
      const int i = s.hBodyAtom[B.first + ii];
      if (!charged[i]) continue;
      for (int jj = ii + 1; jj < B.NP; jj++) {
        const int j = s.hBodyAtom[B.first + jj];
        if (!charged[j]) continue;
        double Rij[3];
        for (int d = 0; d < 3; d++) {
          Rij[d] = R[3 * i + d] - R[3 * j + d];
          Rij[d] = Rij[d] - L * std::round(invL * Rij[d]);
        }
        const double rsq = Rij[0] * Rij[0] + Rij[1] * Rij[1] + Rij[2] * Rij[2];
        // src/modelClass_kspace.f90:318-332
        const double QiQj = s.charge[i] * s.charge[j], r = std::sqrt(rsq), x = e.alpha * r, ex = std::exp(-x * x);
        const double Eij = -QiQj * (1.0 - uerfc<double>(x, ex)) / r;
        e.Erigid[symm1D(local[s.atomType[i]], local[s.atomType[j]]) - 1] += Eij;
      }
    }
  }
  for (int t = 1; t <= e.ntypes; t++) {
    double q2 = 0.0;
    for (int k = e.first[t - 1]; k < e.last[t - 1]; k++) q2 += e.value[k] * e.value[k];
    e.Erigid[symm1D(t, t) - 1] -= e.alpha * q2 / std::sqrt(EW_PI);
  }
  // Coulomb constants per type pair and layer (me%pair%kCoul)
  const int nt = e.ntypes, nl = s.nlayers;
  e.lambda.assign((size_t)nt * nt * nl, 0.0);
  e.lambda1D.assign((size_t)e.nTypePairs * nl, 0.0);
  for (int i = 1; i <= nt; i++)
    for (int j = i; j <= nt; j++)
      for (int l = 0; l < nl; l++) {
        const double lam = s.P(e.type[i - 1] - 1, e.type[j - 1] - 1, l).kCoul;
        e.lambda[((size_t)l * nt + (j - 1)) * nt + (i - 1)] = lam;
        e.lambda[((size_t)l * nt + (i - 1)) * nt + (j - 1)] = lam;
        e.lambda1D[(size_t)l * e.nTypePairs + symm1D(i, j) - 1] = lam;
      }
  ewald_update(e, L);
  // device copies
  e.dItem = upload_vec(e.item);
  e.dQType = upload_vec(e.qtype);
  e.dValue = upload_vec(e.value);
  e.dPrefac = upload_vec(e.prefac);
  e.dLambda = upload_vec(e.lambda);
  ewald_plan(e);
  CK(cudaMalloc(&e.dTable, sizeof(double2) * (size_t)3 * (e.nmax + 1) * e.nq));
  CK(cudaMalloc(&e.dPartial, sizeof(double2) * std::max<size_t>((size_t)e.nchunks * e.nvecs, 1)));
  CK(cudaMalloc(&e.dCoef, sizeof(double2) * std::max<size_t>((size_t)2 * nt * e.npairs, 1)));
  CK(cudaMalloc(&e.dEnergyPartial, sizeof(double) * (e.npairs / SIGMA_PAIRS + 1)));
  // coul_long and other models that need the k-space alpha (src/coul_long.f90:55-64,
  // src/modelClass_coul.f90:101-106)
  for (int l = 0; l < nl; l++) {
    Model& m = s.coul[l];
    if (!m.requires_kspace) continue;
    m.p.alpha = e.alpha;
    if (m.kind == MK_COUL_LONG) m.p.beta = 2.0 * e.alpha / std::sqrt(EW_PI);
  }
  s.modelsUploaded = false;
}

// k-space energy of the current layer (plus the rigid-pair and self discounts);
// forces added to the current layer's force array
static EwArgs ewald_args(System& s, const double* skip) {
  Ewald& e = s.ewald;
  const int l = s.layer - 1;
  EwArgs A;
  A.R = s.dR;
  A.invL = 1.0 / *s.Lbox;
  A.unit2 = 2.0 * e.unit;
  A.nq = e.nq;
  A.nvecs = e.nvecs;
  A.nmax = e.nmax;
  A.ntypes = e.ntypes;
  A.ntasks = e.ntasks;
  A.nrows = e.nrows;
  A.npairs = e.npairs;
  A.nchunks = e.nchunks;
  A.item = e.dItem;
  A.qtype = e.dQType;
  A.value = e.dValue;
  A.task = e.dTask;
  A.row = e.dRow;
  A.pair = e.dPair;
  A.chunk = e.dChunk;
  A.typeChunk = e.dTypeChunk;
  A.prefac = e.dPrefac;
  A.lambda = e.dLambda + (size_t)l * e.ntypes * e.ntypes;
  A.table = e.dTable;
  A.partial = e.dPartial;
  A.coef = e.dCoef;
  A.F = s.F();
  A.epart = e.dEnergyPartial;
  A.ticket = s.dTicket + 4;
  A.result = s.dResult + 22;
  A.hostResult = s.hResult + 22;   // pinned: read after the synchronisation
  A.skip = skip;
  return A;
}

void ewald_launch(System& s, const double* skip, cudaStream_t stream) {
  Ewald& e = s.ewald;
  const EwArgs A = ewald_args(s, skip);
  const int rows = e.nmax + 1;
  if ((size_t)3 * rows * TABLE_LIMIT_ATOMS * sizeof(double2) > 227 * 1024)
    fatal("kspace computation", "too many k-vectors per dimension");
  const size_t smemSF = (size_t)((3 * rows) | 1) * SF_ATOMS * sizeof(double2);
  CK(cudaFuncSetAttribute(k_ewald_sf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemSF));
  k_ewald_tables<<<(3 * e.nq + 127) / 128, 128, 0, stream>>>(A);
  CK(cudaGetLastError());
  const dim3 grid((e.ntasks + SF_THREADS - 1) / SF_THREADS, e.nchunks);
  k_ewald_sf<<<grid, SF_THREADS, smemSF, stream>>>(A);
  CK(cudaGetLastError());
  k_ewald_sigma<<<(e.npairs + SIGMA_PAIRS - 1) / SIGMA_PAIRS, SIGMA_PAIRS * SIGMA_SLICES, 0, stream>>>(A);
  CK(cudaGetLastError());
  s.prof.total += 3;
}

void ewald_add(System& s, const double* skip) {
  Ewald& e = s.ewald;
  const EwArgs A = ewald_args(s, skip);
  const size_t smemF = (size_t)4 * (e.nmax + 1) * FORCE_ATOMS * sizeof(double2);
  CK(cudaFuncSetAttribute(k_ewald_force, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemF));
  k_ewald_force<<<(e.nq + FORCE_ATOMS - 1) / FORCE_ATOMS, FORCE_ATOMS * FORCE_SPLIT, smemF, s.stream>>>(A);
  CK(cudaGetLastError());
  s.prof.total++;
}

double ewald_energy(System& s) {
  const Ewald& e = s.ewald;
  const int l = s.layer - 1;
  const double Ek = s.hResult[22];
  // src/modelClass_kspace.f90:247-314, energy part
  double disc = 0.0;
  for (int k = 0; k < e.nTypePairs; k++) disc += e.lambda1D[(size_t)l * e.nTypePairs + k] * e.Erigid[k];
  return Ek + disc;
}

}  // namespace emdee
