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

static const int PAIR64_THREADS = 128;

struct __align__(32) D4 {
  double x, y, z, w;
};

struct PairArgsD {
  TileGeom g;
  const int2* tab;
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
template <bool COMPUTE, int MOD>
__global__ void __launch_bounds__(PAIR64_THREADS) k_pair_fp64(PairArgsD A) {
  chain_wait();
  extern __shared__ __align__(32) unsigned char sraw[];
  const TileGeom g = A.g;
  const int t = blockIdx.x, cells = g.TB * g.TB * g.TB;
  D4* hpos = (D4*)sraw;   // Rs.xyz, charge
  int4* hfrac = (int4*)(hpos + A.haloCap + 1);
  uint8_t* htype = (uint8_t*)(hfrac + A.haloCap + 1);
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
    hfrac[q] = A.frac[sj];
    if (MOD < 0) htype[q] = A.type8[sj];
  }
  __syncthreads();
  NBParams<double> coul;
  if (MOD < 0) coul = *A.coul;
  NBParams<double> lj = A.table[0].model;
  if (MOD >= 0) {
    lj.kind = MK_LJ_CUT;
    lj.modifier = MOD;
  }
  const int tb = A.start[t * cells], te = A.start[(t + 1) * cells];
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
    const int4 fi = hfrac[qi];
    masked_entries(
        lp, A.tileStride, n, [&](int qj) { return box_dist2(fi, hfrac[qj]) < A.limit; },
        [&](int qj) {
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
        });
    double* Fa = A.F + 3 * (size_t)A.orig[si];
    for (int d = 0; d < 3; d++) Fa[d] = A.L * Fi[d];
  }
  const double v[5] = {0.5 * Ep, 0.5 * Ec, 0.5 * Wp, 0.5 * Wc, 0.5 * (double)within};
  grid_reduce<5, PAIR64_THREADS>(v, A.partials, A.ticket, A.result, A.hostResult);
}

template <bool COMPUTE, int MOD>
static void launch_fp64(System& s, const PairArgsD& A, size_t smem, int nTiles, int threads) {
  CK(cudaFuncSetAttribute(k_pair_fp64<COMPUTE, MOD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (chain_fits(nTiles)) launch_chained(k_pair_fp64<COMPUTE, MOD>, nTiles, threads, smem, s.stream, A);
  else k_pair_fp64<COMPUTE, MOD><<<nTiles, threads, smem, s.stream>>>(A);
}

template <bool COMPUTE>
static void launch_fp64_mod(System& s, const PairArgsD& A, size_t smem, int nt, int th, int mod) {
  switch (mod) {
    case NONE: launch_fp64<COMPUTE, NONE>(s, A, smem, nt, th); break;
    case SHIFTED: launch_fp64<COMPUTE, SHIFTED>(s, A, smem, nt, th); break;
    case SHIFTED_FORCE: launch_fp64<COMPUTE, SHIFTED_FORCE>(s, A, smem, nt, th); break;
    case SMOOTHED: launch_fp64<COMPUTE, SMOOTHED>(s, A, smem, nt, th); break;
    case SHIFTED_SMOOTHED: launch_fp64<COMPUTE, SHIFTED_SMOOTHED>(s, A, smem, nt, th); break;
    case SQUARE_SMOOTHED: launch_fp64<COMPUTE, SQUARE_SMOOTHED>(s, A, smem, nt, th); break;
    case SHIFTED_SQUARE_SMOOTHED: launch_fp64<COMPUTE, SHIFTED_SQUARE_SMOOTHED>(s, A, smem, nt, th); break;
    default: launch_fp64<COMPUTE, -1>(s, A, smem, nt, th); break;
  }
}

void device_pair_forces_fp64(System& s, bool compute, bool useInRc, double rc2scaled) {
  Grid& g = s.grid;
  const double L = *s.Lbox;
  PairArgsD A;
  A.g = make_geom(g.M, g.TB);
  A.tab = g.dHaloTab;
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
  const size_t smem = (size_t)(g.maxHalo + 1) * (sizeof(D4) + sizeof(int4) + 1) + 16;
  const int mod = pair_lj_only(s) ? s.P(0, 0, s.layer - 1).model.p.modifier : -1;
  // as many threads as the largest tile has atoms, in whole warps, up to PAIR64_THREADS
  const int th = std::min(PAIR64_THREADS, (g.tileAtoms + 31) / 32 * 32);
  if (compute) launch_fp64_mod<true>(s, A, smem, g.nTiles, th, mod);
  else launch_fp64_mod<false>(s, A, smem, g.nTiles, th, mod);
  CK(cudaGetLastError());
}

}  // namespace emdee
