// bodies.cu -- rigid bodies on the device: per-body force and torque, momentum
// and position updates, exact or NO_SQUISH rotation, kinetic energies, the
// rigid-body virial, and momentum assignment (src/EmDeeData.f90:157-189,
// 420-439, 823-953; src/ArBee.f90).  FP64, compiled with -fmad=false; four lanes
// per body in the boost and the exact rotation, one thread elsewhere.  Free atoms of a
// system with bodies go through index-list variants of the boost and move kernels.
#include <vector>

#include "chain.cuh"
#include "reduce.cuh"
#include "bodies.cuh"
#include "rigid.cuh"
#include "system.hpp"

namespace emdee {

// One warp per block: the per-body work is a long chain of FP64 operations, so bodies
// are spread over as many SMs as possible.  The grid reductions write their sums
// straight into pinned host memory.
static const int BODY_THREADS = 32;
// The boost and the exact rotation run on BODY_LANES lanes per body, one per quaternion
// component: the FP64 unit of an SM quarter takes 64 clocks per warp instruction however
// many of its lanes are active, so four times the warps with a quarter of the
// instructions each use all the units (4096 bodies on one lane each are 128 warps on
// 608 quarters).  4096 molecules: move 75 -> 31 us,
// boost 11 -> 8.2 us.
static const int BODY_LANES = 4, BODY_GROUP_THREADS = 128;

struct BodyLane {
  int i, c;        // body and lane (quaternion component)
  unsigned mask;   // the body's lanes
};
__device__ __forceinline__ BodyLane body_lane() {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, c = t % BODY_LANES;
  return BodyLane{t / BODY_LANES, c, 0xFu << ((threadIdx.x & 31) & ~(BODY_LANES - 1))};
}
// value x of lane k of the body
__device__ __forceinline__ double body_get(const BodyLane& g, double x, int k) {
  return __shfl_sync(g.mask, x, k, BODY_LANES);
}
// component c of B(q) v and of C(q) v (rb_B, rb_C): -q_k v in component 0, else q_0 v_c
// and the cross product with the sign that tells the two apart
__device__ __forceinline__ double body_BC(const double* q, const double* v, int c, bool isC) {
  if (c == 0) return -q[1] * v[0] - q[2] * v[1] - q[3] * v[2];
  const int a = c % 3, b = (c + 1) % 3;   // 0-based indices after c - 1, cyclic
  const double vc = c == 1 ? v[0] : c == 2 ? v[1] : v[2];
  const double qa = a == 0 ? q[1] : a == 1 ? q[2] : q[3], qb = b == 0 ? q[1] : b == 1 ? q[2] : q[3];
  const double va = a == 0 ? v[0] : a == 1 ? v[1] : v[2], vb = b == 0 ? v[0] : b == 1 ? v[1] : v[2];
  const double s = isC ? -1.0 : 1.0;
  return q[0] * vc + s * (qa * vb - qb * va);
}
// component k (0..2) of B(q)^T p (rb_Bt)
__device__ __forceinline__ double body_Bt(const double* q, const double* p, int k) {
  const int a = (k + 1) % 3, b = (k + 2) % 3;
  const double qk = k == 0 ? q[1] : k == 1 ? q[2] : q[3], pk = k == 0 ? p[1] : k == 1 ? p[2] : p[3];
  const double qa = a == 0 ? q[1] : a == 1 ? q[2] : q[3], pa = a == 0 ? p[1] : a == 1 ? p[2] : p[3];
  const double qb = b == 0 ? q[1] : b == 1 ? q[2] : q[3], pb = b == 0 ? p[1] : b == 1 ? p[2] : p[3];
  return -qk * p[0] + q[0] * pk + qb * pa - qa * pb;
}

// force_and_torque, then pcm and pi updates; KIN: 2KE translational (bodies) and
// rotational sums into result[0..5]; VIR: the sum over bodies and their atoms of F . delta
// (the body virial is its negative) into result[6], which saves k_body_virial's pass where a
// boost with sums follows the forces.  Lane c < 3 takes component c of the vectors.
template <bool KIN, bool VIR>
__global__ void __launch_bounds__(BODY_GROUP_THREADS) k_body_boost(BodyArgs A, const double* F, double CP,
                                                                   double CF, int translate, int rotate,
                                                                   double* partials, unsigned int* ticket,
                                                                   double* result, double* hostResult,
                                                                   const double* skip) {
  chain_wait();
  if (skip != nullptr && __double_as_longlong(*skip) != 0) return;   // a rebuild is due
  static_assert(KIN || !VIR, "the virial comes with the kinetic sums");
  constexpr int NQ = VIR ? 7 : KIN ? 6 : 1;
  double k6[NQ] = {};
  const BodyLane g = body_lane();
  if (g.i < A.nb) {
    BodyState& B = A.b[g.i];
    const int c = g.c, k = c < 3 ? c : 0, k1 = (k + 1) % 3, k2 = (k + 2) % 3;
    const int first = B.first, NP = B.NP;
    double f = 0.0, tau = 0.0;
    for (int j = 0; j < NP; j++) {
      const double* Fj = &F[3 * A.atom[first + j]];
      const double* dj = &A.delta[3 * (first + j)];
      f += Fj[k];
      if (VIR && c < 3) k6[NQ - 1] += Fj[k] * dj[k];
      tau += dj[k1] * Fj[k2] - dj[k2] * Fj[k1];
    }
    double pcm = B.pcm[k], omega = B.omega[k];
    const double MoI = B.MoI[k], invMoI = B.invMoI[k], invMass = B.invMass;
    if (translate) pcm = CP * pcm + CF * f;
    double pi = B.pi[c];
    if (rotate) {
      const double q[4] = {B.q[0], B.q[1], B.q[2], B.q[3]}, t = 2.0 * CF * tau;
      const double v[3] = {body_get(g, t, 0), body_get(g, t, 1), body_get(g, t, 2)};
      pi = CP * pi + body_BC(q, v, c, true);
      const double p[4] = {body_get(g, pi, 0), body_get(g, pi, 1), body_get(g, pi, 2), body_get(g, pi, 3)};
      omega = 0.5 * invMoI * body_Bt(q, p, k);
    }
    if (rotate) B.pi[c] = pi;
    if (c < 3) {
      B.F[c] = f;
      B.tau[c] = tau;
      B.pcm[c] = pcm;
      B.omega[c] = omega;
    }
    if constexpr (KIN) {
      const double kt = invMass * (pcm * pcm), kr = MoI * (omega * omega);
#pragma unroll
      for (int d = 0; d < 3; d++) {
        k6[d] = c == d ? kt : 0.0;
        k6[3 + d] = c == d ? kr : 0.0;
      }
    }
  }
  if (KIN) grid_reduce<NQ, BODY_GROUP_THREADS>(k6, partials, ticket, result, hostResult);
}

// rb_series_step (rigid.cuh) on the four lanes of a body: lane c sums the coefficients
// of quaternion component c and, for c < 3, of w_c; the others come by shuffles.
// Components of w are held in the lane's cyclic order x0 = w_{r+1}, x1 = w_{r+2},
// x2 = w_r (r = c, or 0 in lane 3), so that w_r' ~ x0 x1 in every lane.
//
// Order N: RB_SERIES_ORDER, or BODY_ORDER_WIDE in a warp with a body that turns by more
// than RB_SERIES_STEP: steps of BODY_STEP_WIDE, where the same bound on the first
// omitted term holds ((2 / pi 0.125)^11 = (2 / pi 0.184)^13 = 8e-13 of a first term that
// is itself small).  The few fast bodies set the kernel's time, a warp per quarter of an
// SM: one step of order 12 is 312 multiply-adds, two of order 10 are 440.  Signs are
// flipped on the integer pipe.
constexpr int BODY_ORDER_WIDE = 12;
constexpr double BODY_STEP_WIDE = 0.184;

__device__ __forceinline__ double flip(double x, long long mask) {
  return __longlong_as_double(__double_as_longlong(x) ^ mask);
}

template <int N>
__device__ __forceinline__ void body_series_step(const BodyLane& g, double kap, double (&w)[3], double (&q)[4]) {
  constexpr double inv[13] = {0.0,       1.0,       1.0 / 2.0, 1.0 / 3.0, 1.0 / 4.0,  1.0 / 5.0, 1.0 / 6.0,
                              1.0 / 7.0, 1.0 / 8.0, 1.0 / 9.0, 1.0 / 10.0, 1.0 / 11.0, 1.0 / 12.0};
  static_assert(N <= 12, "reciprocals up to 1 / 12");
  const int c = g.c, r = c < 3 ? c : 0, r1 = (r + 1) % 3, r2 = (r + 2) % 3;
  // component c of B(q) w = sum over k of sign * q_{c xor (k + 1)} w_k
  auto sgn = [&](int k) {   // rows of rb_B: (-,-,-), (+,-,+), (+,+,-), (-,+,+)
    const bool minus = c == 0 || (c == 1 && k == 1) || (c == 2 && k == 2) || (c == 3 && k == 0);
    return minus ? (long long)0x8000000000000000ull : 0ll;
  };
  const int p0 = c ^ (r1 + 1), p1 = c ^ (r2 + 1), p2 = c ^ (r + 1);
  const long long s0 = sgn(r1), s1 = sgn(r2), s2 = sgn(r);
  auto at3 = [](const double (&v)[3], int k) { return k == 0 ? v[0] : k == 1 ? v[1] : v[2]; };
  auto at4 = [](const double (&v)[4], int k) { return k == 0 ? v[0] : k == 1 ? v[1] : k == 2 ? v[2] : v[3]; };
  double X0[N + 1], X1[N + 1], X2[N + 1], B0[N + 1], B1[N + 1], B2[N + 1], Q[N + 1];
  X0[0] = at3(w, r1);
  X1[0] = at3(w, r2);
  X2[0] = at3(w, r);
  B0[0] = flip(at4(q, p0), s0);
  B1[0] = flip(at4(q, p1), s1);
  B2[0] = flip(at4(q, p2), s2);
  Q[0] = at4(q, c);
#pragma unroll
  for (int n = 0; n < N; n++) {
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int i = 0; i <= n; i++) {
      const int j = n - i;
      a = fma(X0[i], X1[j], a);
      b = fma(B0[j], X0[i], fma(B1[j], X1[i], fma(B2[j], X2[i], b)));
    }
    a *= kap * inv[n + 1];
    Q[n + 1] = 0.5 * inv[n + 1] * b;
    X0[n + 1] = body_get(g, a, r1);
    X1[n + 1] = body_get(g, a, r2);
    X2[n + 1] = body_get(g, a, r);
    B0[n + 1] = flip(body_get(g, Q[n + 1], p0), s0);
    B1[n + 1] = flip(body_get(g, Q[n + 1], p1), s1);
    B2[n + 1] = flip(body_get(g, Q[n + 1], p2), s2);
  }
  double x = X2[N], y = Q[N];   // small terms first
#pragma unroll
  for (int n = N - 1; n >= 0; n--) {
    x += X2[n];
    y += Q[n];
  }
  for (int k = 0; k < 3; k++) w[k] = body_get(g, x, k);
  for (int k = 0; k < 4; k++) q[k] = body_get(g, y, k);
}

// rcm update, rotation, atom positions rcm + delta (rotation branch only, as the reference),
// one lane per body: NO_SQUISH, and the bodies the series does not take
__device__ __forceinline__ void body_move_one(const BodyArgs& A, int i, double* __restrict__ R, double CR, double CP,
                                              double dt, int translate, int rotate, int mode) {
  BodyState b = A.b[i];
  if (translate)
    for (int k = 0; k < 3; k++) b.rcm[k] = CR * b.rcm[k] + CP * b.invMass * b.pcm[k];
  if (rotate) {
    const double* d = &A.d[3 * b.first];
    double* delta = &A.delta[3 * b.first];
    if (mode == 0) rb_rotate_elliptic(b, dt, d, delta);
    else rb_rotate_no_squish(b, dt, mode, d, delta);
    for (int j = 0; j < b.NP; j++)
      for (int k = 0; k < 3; k++) R[3 * A.atom[b.first + j] + k] = b.rcm[k] + delta[3 * j + k];
  }
  A.b[i] = b;
}

__global__ void __launch_bounds__(BODY_THREADS) k_body_move(BodyArgs A, double* __restrict__ R, double CR, double CP,
                                                            double dt, int translate, int rotate, int mode) {
  chain_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < A.nb) body_move_one(A, i, R, CR, CP, dt, translate, rotate, mode);
}

// The same with the exact rotation by the series (that of rb_rotate_series, summed in the order
// of the lanes) on BODY_LANES lanes per body.  Order and steps are those of the warp, so
// that its 8 bodies take them together: within the bound above (8e-13 of a small first term)
// a body's result depends on whether one of the others turns fast.
__global__ void __launch_bounds__(BODY_GROUP_THREADS) k_body_move_series(BodyArgs A, double* __restrict__ R, double CR,
                                                                         double CP, double dt, double invdt,
                                                                         int translate) {
  chain_wait();
  const BodyLane g = body_lane();
  // warps past the last body would read one that another warp writes
  if ((int)(blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / BODY_LANES >= A.nb) return;
  BodyState& B = A.b[min(g.i, A.nb - 1)];
  double MoI[3], omega[3], TwoKr = 0.0, Iw1 = 0.0, Iw2 = 0.0, invMoI[3];
  for (int k = 0; k < 3; k++) {
    MoI[k] = B.MoI[k];
    invMoI[k] = B.invMoI[k];
    omega[k] = B.omega[k];
    const double Iw = MoI[k] * omega[k];
    if (k == 1) Iw1 = Iw;
    if (k == 2) Iw2 = Iw;
    TwoKr += Iw * omega[k];
  }
  int steps;
  const double theta2 = TwoKr * invMoI[2] * (dt * dt);
  const bool series = rb_series_steps(theta2, MoI[2], Iw1 * Iw1 + Iw2 * Iw2, steps);
  const bool wide = __any_sync(0xffffffffu, series && steps > 1);
  if (g.i >= A.nb) return;
  if (!series) {
    if (g.c == 0) body_move_one(A, g.i, R, CR, CP, dt, translate, 1, 0);
    return;
  }
  if (wide) {
    steps = 0;
    while (theta2 > (BODY_STEP_WIDE * steps) * (BODY_STEP_WIDE * steps)) steps++;
  }
  const int c = g.c, k = c < 3 ? c : 0, first = B.first, NP = B.NP;
  double q[4] = {B.q[0], B.q[1], B.q[2], B.q[3]};
  double rcm = B.rcm[k];
  if (translate) rcm = CR * rcm + CP * B.invMass * B.pcm[k];
  const double h = steps == 0 ? 1.0 : steps == 1 ? dt : dt / steps,
               back = steps == 0 ? 1.0 : steps == 1 ? invdt : steps * invdt;
  const double kap = k == 0 ? (MoI[1] - MoI[2]) * invMoI[0]
                            : k == 1 ? (MoI[2] - MoI[0]) * invMoI[1] : (MoI[0] - MoI[1]) * invMoI[2];
  double w[3] = {h * omega[0], h * omega[1], h * omega[2]};
  if (wide)
    for (int n = 0; n < steps; n++) body_series_step<BODY_ORDER_WIDE>(g, kap, w, q);
  else if (steps > 0)
    body_series_step<RB_SERIES_ORDER>(g, kap, w, q);
  const double n2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3], f = 1.5 - 0.5 * n2;
  double v[3];
  for (int n = 0; n < 4; n++) q[n] *= f;
  for (int n = 0; n < 3; n++) {
    omega[n] = w[n] * back;
    v[n] = 2.0 * MoI[n] * omega[n];
  }
  const double r[3] = {body_get(g, rcm, 0), body_get(g, rcm, 1), body_get(g, rcm, 2)};
  for (int j = c; j < NP; j += BODY_LANES) {   // a lane per atom
    double t[4], delta[3];
    rb_B(q, &A.d[3 * (first + j)], t);
    rb_Ct(q, t, delta);
    const int a = A.atom[first + j];
    for (int n = 0; n < 3; n++) {
      A.delta[3 * (first + j) + n] = delta[n];
      R[3 * a + n] = r[n] + delta[n];
    }
  }
  __syncwarp(g.mask);   // every lane has read the state
  B.q[c] = c == 0 ? q[0] : c == 1 ? q[1] : c == 2 ? q[2] : q[3];
  B.pi[c] = body_BC(q, v, c, false);
  if (c < 3) {
    B.rcm[c] = rcm;
    B.omega[c] = c == 0 ? omega[0] : c == 1 ? omega[1] : omega[2];
  }
}

// W = sum over bodies and their atoms of F . delta (the body virial is -W)
__global__ void __launch_bounds__(BODY_THREADS) k_body_virial(BodyArgs A, const double* F,
                                                              double* partials, unsigned int* ticket, double* result,
                                                              double* hostResult, const double* skip) {
  chain_wait();
  if (skip != nullptr && __double_as_longlong(*skip) != 0) return;   // a rebuild is due
  double w[1] = {0.0};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < A.nb) {
    const BodyState& b = A.b[i];
    for (int j = 0; j < b.NP; j++)
      for (int k = 0; k < 3; k++) w[0] += F[3 * A.atom[b.first + j] + k] * A.delta[3 * (b.first + j) + k];
  }
  grid_reduce<1, BODY_THREADS>(w, partials, ticket, result, hostResult);
}

// momenta of body atoms -> pcm, pi, omega (src/EmDeeData.f90:172-186), with 2KE sums
__global__ void __launch_bounds__(BODY_THREADS) k_body_assign(BodyArgs A, const double* __restrict__ P,
                                                              double* partials, unsigned int* ticket, double* result,
                                                              double* hostResult) {
  double k6[6] = {0, 0, 0, 0, 0, 0};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < A.nb) {
    BodyState b = A.b[i];
    double Lm[3] = {0, 0, 0}, v[3], pi[4];
    for (int k = 0; k < 3; k++) b.pcm[k] = 0.0;
    for (int j = 0; j < b.NP; j++) {
      const double* Pj = &P[3 * A.atom[b.first + j]];
      double c[3];
      for (int k = 0; k < 3; k++) b.pcm[k] += Pj[k];
      rb_cross(&A.delta[3 * (b.first + j)], Pj, c);
      for (int k = 0; k < 3; k++) Lm[k] += c[k];
    }
    for (int k = 0; k < 3; k++) {
      k6[k] = b.invMass * (b.pcm[k] * b.pcm[k]);
      v[k] = 2.0 * Lm[k];
    }
    rb_C(b.q, v, pi);
    rb_assign_pi(b, pi);
    for (int k = 0; k < 3; k++) k6[3 + k] = b.MoI[k] * (b.omega[k] * b.omega[k]);
    A.b[i] = b;
  }
  grid_reduce<6, BODY_THREADS>(k6, partials, ticket, result, hostResult);
}

// particle momenta of body atoms (src/ArBee.f90:328-336) into P
__global__ void __launch_bounds__(BODY_THREADS) k_body_particle_momenta(BodyArgs A, double* P) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.nb) return;
  const BodyState& b = A.b[i];
  double t[4], omega[3];
  rb_B(b.q, b.omega, t);
  rb_Ct(b.q, t, omega);
  for (int j = 0; j < b.NP; j++) {
    double c[3];
    rb_cross(omega, &A.delta[3 * (b.first + j)], c);
    double m = A.M[b.first + j];
    for (int k = 0; k < 3; k++) P[3 * A.atom[b.first + j] + k] = m * (b.invMass * b.pcm[k] + c[k]);
  }
}

// free atoms only: boost and move through the free-atom list
template <bool KIN>
__global__ void __launch_bounds__(BODY_THREADS) k_boost_free(double* __restrict__ P, const double* F,
                                                             const double* __restrict__ invMass, const int* freeList,
                                                             int nfree, double CP, double CF, double* partials,
                                                             unsigned int* ticket, double* result, double* hostResult,
                                                             const double* skip) {
  chain_wait();
  if (skip != nullptr && __double_as_longlong(*skip) != 0) return;   // a rebuild is due
  double k2[3] = {0.0, 0.0, 0.0};
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nfree; q += gridDim.x * blockDim.x) {
    int i = freeList[q];
    for (int d = 0; d < 3; d++) {
      double p = CP * P[3 * i + d] + CF * F[3 * i + d];
      P[3 * i + d] = p;
      if (KIN) k2[d] += invMass[i] * (p * p);
    }
  }
  if (KIN) grid_reduce<3, BODY_THREADS>(k2, partials, ticket, result, hostResult);
}

__global__ void __launch_bounds__(BODY_THREADS) k_move_free(double* __restrict__ R, const double* P,
                                                            const double* __restrict__ invMass, const int* freeList,
                                                            int nfree, double CR, double CP) {
  chain_wait();
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nfree) return;
  int i = freeList[q];
  for (int d = 0; d < 3; d++) R[3 * i + d] = CR * R[3 * i + d] + CP * P[3 * i + d] * invMass[i];
}

// ---- host side -------------------------------------------------------------------


static int body_blocks(int n) { return n > 0 ? (n + BODY_THREADS - 1) / BODY_THREADS : 1; }
static int body_group_blocks(int n) {
  const int per = BODY_GROUP_THREADS / BODY_LANES;
  return n > 0 ? (n + per - 1) / per : 1;
}

static void ensure_scratch(System& s, int blocks, int nq) {
  int need = blocks * nq;
  if (s.bodyScratchCap < need) {
    CK(cudaFree(s.dBodyScratch));
    s.bodyScratchCap = need;
    CK(cudaMalloc(&s.dBodyScratch, sizeof(double) * need));
  }
}

// src/EmDeeData.f90:420-439: unwrap every body around its first atom, rebuild its
// frame on the host, and upload the unwrapped coordinates and the bodies
void bodies_update(System& s) {
  if (s.nbodies == 0) return;
  int N = s.natoms;
  std::vector<double> R((size_t)3 * N);
  CK(cudaMemcpyAsync(R.data(), s.dR, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, s.stream));
  CK(cudaStreamSynchronize(s.stream));
  double L = *s.Lbox, invL = 1.0 / L;
  for (int bi = 0; bi < s.nbodies; bi++) {
    BodyState& b = s.hBodies[bi];
    std::vector<double> c((size_t)3 * b.NP);
    for (int j = 0; j < b.NP; j++)
      for (int k = 0; k < 3; k++) c[3 * j + k] = R[3 * s.hBodyAtom[b.first + j] + k];
    for (int j = 1; j < b.NP; j++)
      for (int k = 0; k < 3; k++) c[3 * j + k] = c[3 * j + k] - L * std::round(invL * (c[3 * j + k] - c[k]));
    rb_update(b, &s.hBodyM[b.first], c.data(), &s.hBodyD[3 * b.first], &s.hBodyDelta[3 * b.first]);
    for (int j = 0; j < b.NP; j++)
      for (int k = 0; k < 3; k++) R[3 * s.hBodyAtom[b.first + j] + k] = c[3 * j + k];
  }
  // keep the dynamic state (pcm, pi, omega) the device holds
  std::vector<BodyState> dev(s.nbodies);
  CK(cudaMemcpy(dev.data(), s.dBodies, sizeof(BodyState) * s.nbodies, cudaMemcpyDeviceToHost));
  for (int bi = 0; bi < s.nbodies; bi++) {
    BodyState& b = s.hBodies[bi];
    for (int k = 0; k < 3; k++) {
      b.pcm[k] = dev[bi].pcm[k];
      b.omega[k] = dev[bi].omega[k];
      b.F[k] = dev[bi].F[k];
      b.tau[k] = dev[bi].tau[k];
    }
    for (int k = 0; k < 4; k++) b.pi[k] = dev[bi].pi[k];
  }
  size_t na = s.hBodyAtom.size();
  CK(cudaMemcpy(s.dBodies, s.hBodies.data(), sizeof(BodyState) * s.nbodies, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(s.dBodyD, s.hBodyD.data(), sizeof(double) * 3 * na, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(s.dBodyDelta, s.hBodyDelta.data(), sizeof(double) * 3 * na, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(s.dR, R.data(), sizeof(double) * 3 * N, cudaMemcpyHostToDevice));
}

// boost of free atoms (through the list) and bodies
void bodies_boost_launch(System& s, const System::BodyBoost& b, const double* skip, bool virial) {
  int freeBlocks = std::min(body_blocks(s.nfree), 1184);
  ensure_scratch(s, freeBlocks * 3 + body_group_blocks(s.nbodies) * 7, 1);
  if (b.translate && s.nfree > 0) {
    int blocks = freeBlocks;
    if (b.kinetic) {
      launch_chained(k_boost_free<true>, blocks, BODY_THREADS, 0, s.stream, s.dP, s.F(), s.dInvMass, s.dFree, s.nfree, b.CP, b.CF,
                                                                s.dBodyScratch, s.dTicket + 2, s.dResult + 10,
                                                                s.hResult + 10, skip);
    } else {
      launch_chained(k_boost_free<false>, blocks, BODY_THREADS, 0, s.stream, s.dP, s.F(), s.dInvMass, s.dFree, s.nfree, b.CP, b.CF,
                                                                 nullptr, nullptr, nullptr, nullptr, skip);
    }
    CK(cudaGetLastError());
    s.prof.total++;
  }
  auto kern = !b.kinetic ? k_body_boost<false, false> : virial ? k_body_boost<true, true> : k_body_boost<true, false>;
  launch_chained(kern, body_group_blocks(s.nbodies), BODY_GROUP_THREADS, 0, s.stream, body_args(s), s.F(), b.CP, b.CF,
                 b.translate, b.rotate, s.dBodyScratch + freeBlocks * 3, s.dTicket + 3, s.dResult + BODY_RESULT,
                 s.hResult + BODY_RESULT, skip);
  CK(cudaGetLastError());
  s.prof.total++;
}

void bodies_boost_sums(System& s, const System::BodyBoost& b) {
  const double* k6 = s.hResult + BODY_RESULT;
  for (int k = 0; k < 3; k++) {
    s.hResult[10 + k] = (b.translate && s.nfree > 0 ? s.hResult[10 + k] : 0.0) + k6[k];
    s.hResult[13 + k] = k6[3 + k];
  }
}

void bodies_move(System& s, double CR, double CP, double dt, bool translate, bool rotate, int mode) {
  if (translate && s.nfree > 0) {
    launch_chained(k_move_free, body_blocks(s.nfree), BODY_THREADS, 0, s.stream, s.dR, s.dP, s.dInvMass, s.dFree, s.nfree, CR,
                                                                      CP);
    CK(cudaGetLastError());
    s.prof.total++;
  }
  if (rotate && mode == 0)
    launch_chained(k_body_move_series, body_group_blocks(s.nbodies), BODY_GROUP_THREADS, 0, s.stream, body_args(s), s.dR, CR, CP,
                   dt, 1.0 / dt, translate);
  else
    launch_chained(k_body_move, body_blocks(s.nbodies), BODY_THREADS, 0, s.stream, body_args(s), s.dR, CR, CP, dt, translate,
                                                                       rotate, mode);
  CK(cudaGetLastError());
  s.prof.total++;
}

void bodies_virial_launch(System& s, const double* skip) {
  int blocks = body_blocks(s.nbodies);
  ensure_scratch(s, blocks, 1);
  launch_chained(k_body_virial, blocks, BODY_THREADS, 0, s.stream, body_args(s), s.F(), s.dBodyScratch, s.dTicket + 3,
                                                        s.dResult + BODY_RESULT + 6, s.hResult + BODY_RESULT + 6,
                 skip);
  CK(cudaGetLastError());
  s.prof.total++;
}

// bodies take their momenta from the particle momenta in dP; 2KE of bodies into k6
void bodies_assign(System& s, double* k6) {
  int blocks = body_blocks(s.nbodies);
  ensure_scratch(s, blocks, 6);
  k_body_assign<<<blocks, BODY_THREADS, 0, s.stream>>>(body_args(s), s.dP, s.dBodyScratch, s.dTicket + 3,
                                                       s.dResult + 16, s.hResult + 16);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(s.stream));
  for (int k = 0; k < 6; k++) k6[k] = s.hResult[16 + k];
}

void bodies_particle_momenta(System& s, double* dOut) {
  k_body_particle_momenta<<<body_blocks(s.nbodies), BODY_THREADS, 0, s.stream>>>(body_args(s), dOut);
  CK(cudaGetLastError());
}

void bodies_download(System& s) {
  CK(cudaStreamSynchronize(s.stream));
  CK(cudaMemcpy(s.hBodies.data(), s.dBodies, sizeof(BodyState) * s.nbodies, cudaMemcpyDeviceToHost));
}

void bodies_upload(System& s) {
  CK(cudaMemcpy(s.dBodies, s.hBodies.data(), sizeof(BodyState) * s.nbodies, cudaMemcpyHostToDevice));
}

}  // namespace emdee
