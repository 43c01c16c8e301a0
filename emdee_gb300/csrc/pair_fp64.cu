// pair_fp64.cu -- pair forces, energies and virials in FP64 with the
// reference's per-pair arithmetic (src/compute.f90:20-100).
//
// Same tiling and lists as the FP32 kernel; the halo holds the scaled FP64
// coordinates Rs = R/L and each pair goes through exactly the operations of the
// reference: Rij = Rs_i - Rs_j, Rij -= anint(Rij), r2 = sum(Rij^2),
// invR2 = invL2/r2, invR = sqrt(invR2), model and modifier, Coulomb term,
// Fij = Wsum*invR2*Rij, and finally F = L*F.  Compiled with -fmad=false so every
// operation rounds as written.  Only the order in which the pair forces of an
// atom are summed differs from the reference (full lists instead of
// Newton's-third-law half lists).
#include <algorithm>

#include "chain.cuh"
#include "reduce.cuh"
#include "system.hpp"
#include "tile.cuh"

namespace emdee {

static const int PAIR64_THREADS = 128, PAIR64_MANY = 8192;
static const int PAIR64_STATIC = 512;   // the kernel's static shared memory at most (the sums of grid_reduce)

struct __align__(32) D4 {
  double x, y, z, w;
};

struct PairArgsD {
  TileGeom g;
  const double* Rs;        // slot order, double[N][3]
  const double* charge;    // API order
  const uint8_t* type8;
  const int* start;
  const int* orig;
  const uint16_t* self;
  const uint16_t* nb;
  const int* count;
  int cap, tileStride, haloCap;
  const PairEntry<double>* table;
  const NBParams<double>* coul;
  int ntypes;
  double Rc2, invL2, L;
  double* F;
  double* partials;
  unsigned int* ticket;
  double* result;
  double* hostResult;
  const int* layout;
  const int4* frac;   // box fractions, slot order
  float limit;        // box_limit(Rc2)
};

// The kernel is bound by the FP64 pipe (2 operations per clock per SM).  FP64 round() and
// the models' unused roots and divisions were most of its work; the image shift is
// decided on the integer pipe (wrap_half, tile.cuh) and, for one atom type with
// Lennard-Jones and no charges, MOD compiles in the modifier, so that only what it uses
// is evaluated, in the same operations (MOD < 0: any models).  Half of the lanes were
// idle, since a list holds entries beyond the cut-off (30 %): an FP32 test of the box
// fractions now picks those that can lie within it (masked_entries).  32,003 atoms,
// force-shifted: 650 -> 450 us
// (FP64 lanes 52 -> 66 % in use; tiles of 62 atoms in warps of 32 leave the rest).
// STAGED: the fractions are staged beside the coordinates.  A halo that does not fit so in
// shared memory (beyond 4732 atoms) goes without them: every entry gets the FP64 distance
// (9000 atoms, 5300 in a halo, one type: 6.52 ms, masked by fractions made from the staged
// coordinates on the way 8.49; 5500 in one halo 3.38 and 4.46 ms).
template <bool COMPUTE, int MOD, bool STAGED>
__global__ void __launch_bounds__(PAIR64_THREADS) k_pair_fp64(PairArgsD A) {
  chain_wait();
  extern __shared__ __align__(32) unsigned char sraw[];
  const TileGeom g = A.g;
  const int t = blockIdx.x, cells = g.TB * g.TB * g.TB;
  D4* hpos = (D4*)sraw;   // Rs.xyz, charge
  int4* hfrac = (int4*)(hpos + A.haloCap + 1);
  uint8_t* htype = (uint8_t*)(hfrac + (STAGED ? A.haloCap + 1 : 0));
  const int tb = A.start[t * cells], te = A.start[(t + 1) * cells];
  if (te > tb) {   // (a nearly empty box has hundreds of thousands of tiles without atoms)
    // from the layout saved by the list build: every halo index's slot first (in the
    // position it will hold), then the atoms, one thread each
    const int* lay = A.layout + (size_t)t * (2 * g.haloCells + 1);
    int* mark = (int*)sraw;
    for (int h = threadIdx.x; h < g.haloCells; h += blockDim.x) {
      const int b = lay[h], e = lay[h + 1], s0 = lay[g.haloCells + 1 + h];
      for (int q = b; q < e; q++) mark[q * (sizeof(D4) / sizeof(int))] = s0 + q - b;
    }
    __syncthreads();
    const int halo = lay[g.haloCells];
    for (int q = threadIdx.x; q < halo; q += blockDim.x) {
      const int sj = mark[q * (sizeof(D4) / sizeof(int))];
      hpos[q] = D4{A.Rs[3 * sj], A.Rs[3 * sj + 1], A.Rs[3 * sj + 2], MOD < 0 ? A.charge[A.orig[sj]] : 0.0};
      if (STAGED) hfrac[q] = A.frac[sj];
      if (MOD < 0) htype[q] = A.type8[sj];
    }
    __syncthreads();
  }
  NBParams<double> coul;
  if (MOD < 0) coul = *A.coul;
  NBParams<double> lj = A.table[0].model;
  if (MOD >= 0) {
    lj.kind = MK_LJ_CUT;
    lj.modifier = MOD;
  }
  const int capC = A.cap >> 3;
  double Ep = 0.0, Ec = 0.0, Wp = 0.0, Wc = 0.0;
  int within = 0;
  for (int li = threadIdx.x; li < te - tb; li += blockDim.x) {
    const int si = tb + li, qi = A.self[si];
    const D4 pi = hpos[qi];
    const int ti = MOD < 0 ? htype[qi] : 0;
    const bool ich = MOD < 0 && fabs(pi.w) > 2.220446049250313e-16;
    const int n = min(A.count[si], A.cap);
    const uint4* lp = reinterpret_cast<const uint4*>(A.nb) + ((size_t)t * capC * A.tileStride + li);
    double Fi[3] = {0.0, 0.0, 0.0};
    auto pair = [&](int qj) {
      const D4 pj = hpos[qj];
      const double Rij[3] = {wrap_half(pi.x - pj.x), wrap_half(pi.y - pj.y), wrap_half(pi.z - pj.z)};
      const double r2 = Rij[0] * Rij[0] + Rij[1] * Rij[1] + Rij[2] * Rij[2];
      if (!(r2 < A.Rc2)) return;
      within++;
      const double invR2 = A.invL2 / r2;
      const double invR = sqrt(invR2);   // dropped where the models do not use it
      double Wsum;
      if (MOD >= 0) {
        double E = 0.0;
        if (COMPUTE) {
          nb_compute(lj, E, Wsum, invR, invR2);
          modifier_compute(lj, E, Wsum, invR, invR2);
          Ep += E;
        } else {
          Wsum = nb_virial(lj, invR, invR2);
          modifier_virial(lj, Wsum, invR, invR2);
        }
        Wp += Wsum;
      } else {
        const PairEntry<double>& pe = A.table[ti * A.ntypes + htype[qj]];
        const bool ijch = ich && fabs(pj.w) > 2.220446049250313e-16;
        Wsum = pair_eval<double, COMPUTE>(pe, coul, ijch, pi.w, pj.w, invR, invR2, Ep, Ec, Wp, Wc);
      }
      const double s = Wsum * invR2;
      for (int d = 0; d < 3; d++) Fi[d] += s * Rij[d];
    };
    if (STAGED) {
      const int4 fi = hfrac[qi];
      masked_entries(lp, A.tileStride, n, [&](int qj) { return box_dist2(fi, hfrac[qj]) < A.limit; }, pair);
    } else {
      const uint16_t* entry = reinterpret_cast<const uint16_t*>(lp);
      for (int k = 0; k < n; k++) pair(entry[(size_t)(k >> 3) * A.tileStride * 8 + (k & 7)]);
    }
    double* Fa = A.F + 3 * (size_t)A.orig[si];
    for (int d = 0; d < 3; d++) Fa[d] = A.L * Fi[d];
  }
  const double v[5] = {0.5 * Ep, 0.5 * Ec, 0.5 * Wp, 0.5 * Wc, 0.5 * (double)within};
  grid_reduce<5, PAIR64_THREADS>(v, A.partials, A.ticket, A.result, A.hostResult);
}

template <bool COMPUTE, bool STAGED, int MOD>
static void launch_fp64(System& s, const PairArgsD& A, size_t smem, int nTiles, int threads) {
  auto kern = k_pair_fp64<COMPUTE, MOD, STAGED>;
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (chain_fits(nTiles)) launch_chained(kern, nTiles, threads, smem, s.stream, A);
  else kern<<<nTiles, threads, smem, s.stream>>>(A);
}

template <bool COMPUTE, bool STAGED>
static void launch_fp64_mod(System& s, const PairArgsD& A, size_t smem, int nt, int th, int mod) {
  switch (mod) {
    case NONE: launch_fp64<COMPUTE, STAGED, NONE>(s, A, smem, nt, th); break;
    case SHIFTED: launch_fp64<COMPUTE, STAGED, SHIFTED>(s, A, smem, nt, th); break;
    case SHIFTED_FORCE: launch_fp64<COMPUTE, STAGED, SHIFTED_FORCE>(s, A, smem, nt, th); break;
    case SMOOTHED: launch_fp64<COMPUTE, STAGED, SMOOTHED>(s, A, smem, nt, th); break;
    case SHIFTED_SMOOTHED: launch_fp64<COMPUTE, STAGED, SHIFTED_SMOOTHED>(s, A, smem, nt, th); break;
    case SQUARE_SMOOTHED: launch_fp64<COMPUTE, STAGED, SQUARE_SMOOTHED>(s, A, smem, nt, th); break;
    case SHIFTED_SQUARE_SMOOTHED: launch_fp64<COMPUTE, STAGED, SHIFTED_SQUARE_SMOOTHED>(s, A, smem, nt, th); break;
    default: launch_fp64<COMPUTE, STAGED, -1>(s, A, smem, nt, th); break;
  }
}

void device_pair_forces_fp64(System& s, bool compute, bool useInRc, double rc2scaled) {
  Grid& g = s.grid;
  const double L = *s.Lbox;
  PairArgsD A;
  A.g = make_geom(g.M, g.TB);
  A.Rs = g.dRs64;
  A.charge = s.dCharge;
  A.type8 = g.dType8;
  A.start = g.dStart;
  A.orig = g.dOrig;
  A.self = g.dSelf;
  A.nb = g.dNb;
  A.count = useInRc ? g.dNbInner : g.dNbCount;
  A.cap = g.cap;
  A.tileStride = g.tileStride;
  A.haloCap = g.maxHalo;
  A.table = s.models.d64 + (size_t)(s.layer - 1) * s.ntypes * s.ntypes;
  A.coul = s.models.coul64 + (s.layer - 1);
  A.ntypes = s.ntypes;
  A.invL2 = 1.0 / (L * L);   // src/EmDeeData.f90:658-659
  A.Rc2 = rc2scaled;
  A.L = L;
  A.F = s.F();
  A.partials = s.dPartials;
  A.ticket = s.dTicket;
  A.result = s.dResult;
  A.hostResult = s.hResult;   // pinned: no copy back
  A.layout = g.dLayout;
  A.frac = (const int4*)g.dPos4;
  A.limit = box_limit(A.Rc2);
  const size_t atom = sizeof(D4) + 1, halo = g.maxHalo + 1, limit = 227 * 1024 - PAIR64_STATIC;
  const bool staged = halo * (atom + sizeof(int4)) + 16 <= limit;
  const size_t smem = halo * (staged ? atom + sizeof(int4) : atom) + 16;
  if (smem > limit) fatal("pair forces", "too many atoms around a cell for FP64 arithmetic");
  const int mod = pair_lj_only(s) ? s.P(0, 0, s.layer - 1).model.p.modifier : -1;
  // As many threads as the largest tile has atoms, in whole warps, up to PAIR64_THREADS, and
  // enough for the halo's cells; all of them where the last block has very many tiles' sums to
  // add.  2000 atoms in a box of 60 (1331 tiles), 10 steps: 1155 us with 32 threads, 889 with
  // 64; in a box of 150 (19,683 tiles) 6.27 ms with 64, 4.98 with 128
  const int fit = std::max(halo_min_threads(A.g), (g.tileAtoms + 31) / 32 * 32);
  const int th = g.nTiles >= PAIR64_MANY ? PAIR64_THREADS : std::min(PAIR64_THREADS, fit);
  auto run = staged ? (compute ? launch_fp64_mod<true, true> : launch_fp64_mod<false, true>)
                    : (compute ? launch_fp64_mod<true, false> : launch_fp64_mod<false, false>);
  run(s, A, smem, g.nTiles, th, mod);
  CK(cudaGetLastError());
}

}  // namespace emdee
