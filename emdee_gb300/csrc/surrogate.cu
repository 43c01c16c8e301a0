// surrogate.cu -- learned surrogate potential for hybrid Monte Carlo proposals
// (no counterpart in the reference; it serves the surrogate-proposal HMC
// workload: a binary Lennard-Jones mixture, many chains of the same size).
//
// Model (atom-centred, Behler-Parrinello style): for atom i of species s_i,
//   G_i[c, k] = sum_{j != i, s_j = c, r_ij < rc} exp(-(r_ij - mu_k)^2 / (2 w^2)) fc(r_ij),
//   fc(r) = (cos(pi r / rc) + 1) / 2,  mu_k = mu_0 + k (mu_15 - mu_0) / 15,  k = 0..15, c = 0..1,
//   E_i = w3 . silu(W2^T silu(W1^T G_i + b1) + b2) + b3 with one network per species
//   (32 -> 64 -> 64 -> 1), E = sum_i E_i,  F = -dE/dR.
// Kernels (one launch each, over all chains at once):
//   k_sg_pack      FP64 positions -> FP32, wrapped into the box
//   k_sg_list      Verlet lists within rc + skin from a cell list (per chain), a block
//                  per cell
//   k_sg_desc      descriptors, a warp per atom, Gaussians by the two-term product recurrence
//   k_sg_mlp_tc    per-species tiles of 128 atoms: forward and backward through the
//                  network on the tensor cores (tcgen05, BF16 operands, FP32
//                  accumulation): E_i and dE/dG_i; k_sg_mlp, tiles of 64 atoms by
//                  mma.sync m16n8k16, is kept for comparison
//   k_sg_force     the adjoint: F_i = -sum_j (dE/dG_i[s_j] + dE/dG_j[s_i]) . dh/dr r_hat
//   k_sg_udesc     training: u_i[c, k] = sum_j h'_k(r_ij) (v_i - v_j) . r_hat_ij, the
//                  force residual v pulled back to descriptor space
//   k_sg_train     training: per species, forward, tangent along u, and the
//                  backward pass of O_i = e_c E_i - (dE_i/dG_i . u_i), whose
//                  gradient is the gradient of the energy + force loss; weight
//                  gradients as tensor-core GEMMs over 64-atom tiles, per-block
//                  partials reduced in block order
//   k_sg_advance   trajectories: everything between two force evaluations
//   k_sg_adam      Adam update of the FP32 master parameters
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>

#include "chain.cuh"
#include "reduce.cuh"
#include "system.hpp"
#include "tile.cuh"

namespace emdee {

namespace sg {

constexpr int NG = 16, NS = 2, DIN = 32, H = 64;
// packed FP32 parameters per species: W1[32][64], b1[64], W2[64][64], b2[64], w3[64], b3
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + DIN * H, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H,
              OFF_W3 = OFF_B2 + H, OFF_B3 = OFF_W3 + H, PER_SPECIES = OFF_B3 + 1;
constexpr int NPARAM = NS * PER_SPECIES;
constexpr int TILE = 64;   // atoms per block tile (4 warps x 16)

struct Geometry {
  int chains, N, M;          // M cells per dimension (cell edge >= rc + skin)
  float L, invL, rc, rc2, rlist2, mu0, dmu, a;   // a = 1 / (2 w^2)
};

__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float dsilu(float x) {
  const float s = 1.f / (1.f + __expf(-x));
  return s * (1.f + x * (1.f - s));
}
__device__ __forceinline__ float d2silu(float x) {
  const float s = 1.f / (1.f + __expf(-x));
  return s * (1.f - s) * (2.f + x * (1.f - 2.f * s));
}

// ---- tensor-core tile GEMM -------------------------------------------------------
// D(16 x 8) += A(16 x 16, row-major) * B(16 x 8, "col": element (k, n) read from
// Bt[n][k]); fragment layouts of mma.sync.m16n8k16 (PTX ISA): lane = 4 g + t,
// A regs (g, 2t..2t+1), (g+8, ..), (g, 2t+8..), (g+8, 2t+8..); B regs (2t..2t+1, g),
// (2t+8.., g); C regs (g, 2t..2t+1), (g+8, 2t..2t+1).
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// four 8 x 8 BF16 matrices from shared memory: lane l supplies the address of row l % 8 of
// matrix l / 8; lane 4 g + t receives elements (g, 2t..2t+1) of each, or with TRANS
// (2t..2t+1, g)
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// acc[nt][4] += A(16 x K) * B(K x 8 NT), A row-major (lda), B given as Bt[n][k] (ldb)
template <int K, int NT>
__device__ __forceinline__ void warp_gemm(const __nv_bfloat16* A, int lda, const __nv_bfloat16* Bt, int ldb,
                                          float (&acc)[NT][4]) {
  const int lane = threadIdx.x & 31, row = lane & 7, mat = lane >> 3;
  const __nv_bfloat16* pa = A + (row + 8 * (mat & 1)) * lda + 8 * (mat >> 1);
  const __nv_bfloat16* pb = Bt + (row + 8 * (mat >> 1)) * ldb + 8 * (mat & 1);
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += 16) {
    uint32_t a[4];
    ldmatrix4<false>(a, pa + k0);
#pragma unroll
    for (int n = 0; n < NT; n += 2) {   // two column tiles per load
      uint32_t b[4];
      ldmatrix4<false>(b, pb + n * 8 * ldb + k0);
      const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
      mma16816(acc[n], a, b0);
      mma16816(acc[n + 1], a, b1);
    }
  }
}

// acc[nt][4] += A^T(16 x K) * B(K x 8 NT) with A and B stored by rows of k: A[k][m] (lda),
// B[k][n] (ldb), transposed as they are loaded
template <int K, int NT>
__device__ __forceinline__ void warp_gemm_t(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb,
                                            float (&acc)[NT][4]) {
  const int lane = threadIdx.x & 31, row = lane & 7, mat = lane >> 3;
  const __nv_bfloat16* pa = A + (row + 8 * (mat >> 1)) * lda + 8 * (mat & 1);
  const __nv_bfloat16* pb = B + (row + 8 * (mat & 1)) * ldb + 8 * (mat >> 1);
#pragma unroll
  for (int k0 = 0; k0 < K; k0 += 16) {
    uint32_t a[4];
    ldmatrix4<true>(a, pa + k0 * lda);
#pragma unroll
    for (int n = 0; n < NT; n += 2) {
      uint32_t b[4];
      ldmatrix4<true>(b, pb + k0 * ldb + n * 8);
      const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
      mma16816(acc[n], a, b0);
      mma16816(acc[n + 1], a, b1);
    }
  }
}

template <int NT>
__device__ __forceinline__ void zero(float (&acc)[NT][4]) {
#pragma unroll
  for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
}

// element (row, col) of fragment tile n, slot q (0..3)
__device__ __forceinline__ int frag_row(int q) { return ((threadIdx.x & 31) >> 2) + (q >= 2 ? 8 : 0); }
__device__ __forceinline__ int frag_col(int n, int q) { return n * 8 + 2 * (threadIdx.x & 3) + (q & 1); }

// shared-memory weights of one species, BF16, in both orientations
struct __align__(16) WeightsSmem {   // rows on 16-byte boundaries, for ldmatrix
  __nv_bfloat16 W1[DIN][H + 8];    // W1[k][n]        (B^T for dE/dG = dz1 W1^T)
  __nv_bfloat16 W1t[H][DIN + 8];   // W1^T[n][k]      (B^T for z1 = G W1)
  __nv_bfloat16 W2[H][H + 8];      // W2[k][n]        (B^T for da1 = dz2 W2^T)
  __nv_bfloat16 W2t[H][H + 8];     // W2^T[n][k]      (B^T for z2 = a1 W2)
  float b1[H], b2[H], w3[H], b3;
};

__device__ void load_weights(WeightsSmem& w, const float* p) {
  for (int q = threadIdx.x; q < DIN * H; q += blockDim.x) {
    const int k = q / H, n = q % H;
    const __nv_bfloat16 v = __float2bfloat16(p[OFF_W1 + q]);
    w.W1[k][n] = v;
    w.W1t[n][k] = v;
  }
  for (int q = threadIdx.x; q < H * H; q += blockDim.x) {
    const int k = q / H, n = q % H;
    const __nv_bfloat16 v = __float2bfloat16(p[OFF_W2 + q]);
    w.W2[k][n] = v;
    w.W2t[n][k] = v;
  }
  for (int q = threadIdx.x; q < H; q += blockDim.x) {
    w.b1[q] = p[OFF_B1 + q];
    w.b2[q] = p[OFF_B2 + q];
    w.w3[q] = p[OFF_W3 + q];
  }
  if (threadIdx.x == 0) w.b3 = p[OFF_B3];
}

// ---- geometry kernels ---------------------------------------------------------------

__device__ __forceinline__ float wrapped(double x, double L) { return (float)(x - L * floor(x / L)); }

// (the fourth component is not read)
__global__ void k_sg_pack(const double* __restrict__ R, int total, double L, float4* __restrict__ pos) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= total) return;
  float p[3];
  for (int d = 0; d < 3; d++) p[d] = wrapped(R[3 * q + d], L);
  pos[q] = make_float4(p[0], p[1], p[2], 0.f);
}

__device__ __forceinline__ int sg_cell(float x, const Geometry& G) {
  int c = (int)(x * G.invL * G.M);
  return c < 0 ? 0 : (c >= G.M ? G.M - 1 : c);
}

// cell counts per chain
__global__ void k_sg_count(const float4* __restrict__ pos, Geometry G, int* __restrict__ cellOf,
                           int* __restrict__ counts) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.chains * G.N) return;
  const int c = q / G.N;
  const float4 p = pos[q];
  const int cell = sg_cell(p.x, G) + G.M * (sg_cell(p.y, G) + G.M * sg_cell(p.z, G));
  cellOf[q] = cell;
  atomicAdd(&counts[c * G.M * G.M * G.M + cell], 1);
}

// one block: exclusive scan of all chains' cell counts (chains * M^3 entries)
__global__ void k_sg_scan(const int* counts, int n, int* starts) {
  __shared__ int ws[33];
  __shared__ int carry;
  __shared__ int buf[2048];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 2048) {
    for (int k = threadIdx.x; k < 2048; k += blockDim.x) buf[k] = base + k < n ? counts[base + k] : 0;
    __syncthreads();
    const int total = block_exclusive_scan<8>(buf, 2048, ws);
    for (int k = threadIdx.x; k < 2048; k += blockDim.x)
      if (base + k < n) starts[base + k] = buf[k] + carry;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) starts[n] = carry;
}

__global__ void k_sg_scatter(const int* __restrict__ cellOf, Geometry G, const int* __restrict__ starts,
                             int* __restrict__ cursor, int* __restrict__ sorted) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= G.chains * G.N) return;
  const int c = q / G.N, r = c * G.M * G.M * G.M + cellOf[q];
  sorted[starts[r] + atomicAdd(&cursor[r], 1)] = q;
}

// Deterministic order inside a cell (ascending atom index): a warp per cell, each atom's
// place is the number of atoms of the cell with a smaller index.  Cells of more than
// 32 * SORT_REGS atoms are sorted by lane 0.  (8 x 8000 atoms in cells of 64: one thread
// per cell took 343 us, 8 us so.)  SPARSE: a warp looks at 32 cells, of which most hold no or
// one atom, for those that hold more.
constexpr int SORT_REGS = 8;
__device__ __forceinline__ void sort_cell(int b, int m, int* __restrict__ sorted) {
  const int lane = threadIdx.x & 31;
  if (m > 32 * SORT_REGS) {
    if (lane == 0)
      for (int i = b + 1; i < b + m; i++) {
        const int v = sorted[i];
        int j = i - 1;
        while (j >= b && sorted[j] > v) {
          sorted[j + 1] = sorted[j];
          j--;
        }
        sorted[j + 1] = v;
      }
    return;
  }
  int v[SORT_REGS], place[SORT_REGS];
#pragma unroll
  for (int u = 0; u < SORT_REGS; u++) {
    v[u] = 32 * u + lane < m ? sorted[b + 32 * u + lane] : 0;
    place[u] = 0;
  }
#pragma unroll
  for (int w = 0; w < SORT_REGS; w++) {
    if (32 * w >= m) break;
    for (int k = 0; k < min(32, m - 32 * w); k++) {
      const int x = __shfl_sync(0xffffffffu, v[w], k);
#pragma unroll
      for (int u = 0; u < SORT_REGS; u++) place[u] += x < v[u] ? 1 : 0;
    }
  }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < SORT_REGS; u++)
    if (32 * u + lane < m) sorted[b + place[u]] = v[u];
}

template <bool SPARSE>
__global__ void k_sg_sort(const int* __restrict__ starts, int n, int* __restrict__ sorted) {
  const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (SPARSE) {
    const int r = 32 * warp + lane;
    unsigned todo = __ballot_sync(0xffffffffu, r < n && starts[r + 1] - starts[r] > 1);
    for (; todo != 0; todo &= todo - 1) {
      const int c = 32 * warp + __ffs(todo) - 1;
      sort_cell(starts[c], starts[c + 1] - starts[c], sorted);
    }
  } else if (warp < n) {
    const int b = starts[warp], m = starts[warp + 1] - b;
    if (m > 1) sort_cell(b, m, sorted);
  }
}

// rintf for |x| < 2^22 on the FP32 adders (the conversion unit runs at a quarter of
// their rate)
__device__ __forceinline__ float nearest(float x) { return __fadd_rn(__fadd_rn(x, 12582912.f), -12582912.f); }

// Verlet lists (global atom indices), entry e of atom q at list[q * cap + e], in the order
// of the neighbor cells and of their atoms.  A block per cell stages the candidates of
// its atoms (27 cells, or with M < 3 the whole chain) in shared memory; a warp goes
// through them side by side for LIST_ATOMS atoms at a time and places the accepted ones
// by ballots.  More than LIST_CAND candidates are taken in several stages.  Bound by
// instruction issue: 36 instructions per 32 candidates of one atom before the load and
// the loop were shared by LIST_ATOMS (8 x 8000 atoms: 142 -> 111 us; one thread per atom,
// gathering each candidate's index and position: 428 us).
// Where the chains have more cells than atoms the blocks are those of the atoms' cells
// instead: block b takes the cell of the b-th atom in cell order, if that is its first
// (BY_ATOM; forces with new lists of 2000 atoms in 54,872 cells: 206 -> 167 us).
constexpr int LIST_CAND = 2048, LIST_THREADS = 256, LIST_ATOMS = 2;
template <bool BY_ATOM>
__global__ void __launch_bounds__(LIST_THREADS) k_sg_list(const float4* __restrict__ pos, Geometry G,
                                                          const int* __restrict__ starts,
                                                          const int* __restrict__ sorted,
                                                          const int* __restrict__ cellOf, int cap,
                                                          int* __restrict__ list, int* __restrict__ count,
                                                          int* __restrict__ overflow) {
  __shared__ float4 cand[LIST_CAND];   // position (M >= 3: the image next to the cell) and index
  __shared__ int first[28], base[28];   // candidates of the neighbor cells: first slot, running count
  const int M = G.M, cells = M * M * M;
  int id = blockIdx.x;
  if (BY_ATOM) {
    const int q = sorted[blockIdx.x];
    id = q / G.N * cells + cellOf[q];
    if (starts[id] != (int)blockIdx.x) return;
  }
  const int chain = id / cells, cell = id % cells;
  const int x = cell % M, y = (cell / M) % M, z = cell / (M * M);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int own0 = starts[id], own1 = starts[id + 1];
  if (own0 == own1) return;
  const int ncell = M >= 3 ? 27 : 1;   // M < 3: every cell of the chain once
  if (threadIdx.x < ncell) {
    const int k = threadIdx.x, dx = k % 3 - 1, dy = k / 3 % 3 - 1, dz = k / 9 - 1;
    const int r = M >= 3 ? chain * cells + (x + dx + M) % M + M * ((y + dy + M) % M + M * ((z + dz + M) % M))
                         : chain * cells;
    first[k] = starts[r];
    base[k + 1] = M >= 3 ? starts[r + 1] - starts[r] : starts[(chain + 1) * cells] - starts[chain * cells];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    base[0] = 0;
    for (int k = 0; k < ncell; k++) base[k + 1] += base[k];
  }
  __syncthreads();
  const int total = base[ncell];
  int longest = 0;
  const unsigned below = (1u << lane) - 1u;
  // this warp's share of the cell's atoms
  const int o0 = own0 + (own1 - own0) * warp / (LIST_THREADS / 32),
            o1 = own0 + (own1 - own0) * (warp + 1) / (LIST_THREADS / 32);
  for (int c0 = 0; c0 < total; c0 += LIST_CAND) {
    const int nc = min(LIST_CAND, total - c0);
    if (c0 > 0) __syncthreads();
    // a warp per neighbor cell (the whole block where there is one)
    const int width = ncell == 1 ? LIST_THREADS : 32;
    for (int k = ncell == 1 ? 0 : warp; k < ncell; k += LIST_THREADS / 32) {
      float sx = 0.f, sy = 0.f, sz = 0.f;
      if (M >= 3) {   // cells across the box's faces: the image on this side
        const int nx = x + k % 3 - 1, ny = y + k / 3 % 3 - 1, nz = z + k / 9 - 1;
        sx = nx < 0 ? -G.L : nx >= M ? G.L : 0.f;
        sy = ny < 0 ? -G.L : ny >= M ? G.L : 0.f;
        sz = nz < 0 ? -G.L : nz >= M ? G.L : 0.f;
      }
      const int u0 = max(0, c0 - base[k]), u1 = min(base[k + 1] - base[k], c0 + nc - base[k]);
      for (int u = u0 + (ncell == 1 ? (int)threadIdx.x : lane); u < u1; u += width) {
        const int j = sorted[first[k] + u];
        float4 p = pos[j];
        p.x += sx;
        p.y += sy;
        p.z += sz;
        p.w = __int_as_float(j);
        cand[base[k] + u - c0] = p;
      }
    }
    __syncthreads();
    for (int o = o0; o < o1; o += LIST_ATOMS) {
      const int na = min(LIST_ATOMS, o1 - o);
      int q[LIST_ATOMS], n[LIST_ATOMS];
      float4 p[LIST_ATOMS];
      int* out[LIST_ATOMS];
#pragma unroll
      for (int a = 0; a < LIST_ATOMS; a++) {
        q[a] = sorted[min(o + a, o1 - 1)];
        p[a] = pos[q[a]];
        out[a] = list + (size_t)q[a] * cap;
        n[a] = c0 > 0 ? count[q[a]] : 0;
      }
      for (int c = lane; c - lane < nc; c += 32) {
        const bool have = c < nc;
        const float4 pj = cand[have ? c : 0];
        const int j = __float_as_int(pj.w);
#pragma unroll
        for (int a = 0; a < LIST_ATOMS; a++) {
          if (a >= na) break;
          float ex = p[a].x - pj.x, ey = p[a].y - pj.y, ez = p[a].z - pj.z;
          if (M < 4) {   // a neighbor cell may hold a nearer image
            ex -= G.L * nearest(ex * G.invL);
            ey -= G.L * nearest(ey * G.invL);
            ez -= G.L * nearest(ez * G.invL);
          }
          const bool in = have && j != q[a] && ex * ex + ey * ey + ez * ez < G.rlist2;
          const unsigned m = __ballot_sync(0xffffffffu, in);
          const int at = n[a] + __popc(m & below);
          if (in && at < cap) out[a][at] = j;
          n[a] += __popc(m);
        }
      }
#pragma unroll
      for (int a = 0; a < LIST_ATOMS; a++) {
        if (a >= na) break;
        if (lane == 0) count[q[a]] = n[a];
        longest = max(longest, n[a]);
      }
      __syncwarp();
    }
  }
  if (lane == 0 && longest > cap) atomicMax(overflow, longest);
}

struct PairGeom {
  float r, ux, uy, uz;   // distance and unit vector (i - j) / r
};

// h_k = g_k fc and dh_k/dr for the 16 Gaussians (two-term product recurrence:
// g_{k+1} = g_k q_k, q_{k+1} = q_k c, c = exp(-2 a dmu^2))
__device__ __forceinline__ void radial(float r, const Geometry& G, float cdecay, float (&h)[NG], float (&dh)[NG]) {
  float s, co;
  sincospif(r / G.rc, &s, &co);
  const float fc = 0.5f * (co + 1.f), dfc = -0.5f * 3.14159265f / G.rc * s;
  const float x0 = r - G.mu0;
  float gk = __expf(-G.a * x0 * x0);
  float qk = __expf(2.f * G.a * G.dmu * x0 - G.a * G.dmu * G.dmu);
#pragma unroll
  for (int k = 0; k < NG; k++) {
    const float xk = r - (G.mu0 + k * G.dmu);
    h[k] = gk * fc;
    dh[k] = gk * (dfc - 2.f * G.a * xk * fc);
    gk *= qk;
    qk *= cdecay;
  }
}

// The descriptor and adjoint kernels run a warp per atom.  The entries of the Verlet
// list (rc + skin) are tested 32 at a time and those within rc (43 % at rc 2.5, skin 0.8)
// gathered, in list order, in the warp's buffer; each full batch of 32 goes to
// batch(n, d, j): lane k < n holds neighbor k, d = (displacement, squared distance).  So
// the costly radial functions run on full warps; one thread per atom ran them for a
// warp whenever any lane's entry was within rc, on 3 warps per scheduler.  k_sg_desc
// leaves the neighbors within rc in `near`, from which the adjoint kernels at the same
// positions start (each_neighbor).
constexpr int WARP_ATOMS = 8;   // warps (atoms) per block
struct NeighborBuffer {
  float4 d[64];
  int j[64];
};

template <class F>
__device__ __forceinline__ void for_neighbors(const float4* pos, const Geometry& G, int q, const int* list,
                                              int n, NeighborBuffer& B, F&& batch) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const float4 pi = pos[q];
  int have = 0;
  for (int e = lane; e - lane < n; e += 32) {
    const int j = e < n ? list[e] : q;
    const float4 pj = pos[j];
    float ex = pi.x - pj.x, ey = pi.y - pj.y, ez = pi.z - pj.z;
    ex -= G.L * nearest(ex * G.invL);
    ey -= G.L * nearest(ey * G.invL);
    ez -= G.L * nearest(ez * G.invL);
    const float r2 = ex * ex + ey * ey + ez * ez;
    const bool in = e < n && r2 < G.rc2;
    const unsigned m = __ballot_sync(FULL, in);
    const int at = have + __popc(m & ((1u << lane) - 1u));
    if (in) {
      B.d[at] = make_float4(ex, ey, ez, r2);
      B.j[at] = j;
    }
    have += __popc(m);
    __syncwarp();
    if (have >= 32) {
      batch(32, B.d[lane], B.j[lane]);
      have -= 32;
      float4 d;
      int k = 0;
      if (lane < have) {
        d = B.d[32 + lane];
        k = B.j[32 + lane];
      }
      __syncwarp();
      if (lane < have) {
        B.d[lane] = d;
        B.j[lane] = k;
      }
      __syncwarp();
    }
  }
  if (have > 0) batch(have, lane < have ? B.d[lane] : make_float4(1.f, 1.f, 1.f, 3.f), lane < have ? B.j[lane] : q);
}

// batch(n, d, j) over the neighbors k_sg_desc left in `near`, 32 at a time
template <class F>
__device__ __forceinline__ void each_neighbor(const float4* pos, const Geometry& G, int q, const int* near,
                                              int n, F&& batch) {
  const int lane = threadIdx.x & 31;
  const float4 pi = pos[q];
  for (int e = 0; e < n; e += 32) {
    const int m = min(32, n - e), j = lane < m ? near[e + lane] : q;
    const float4 pj = pos[j];
    float ex = pi.x - pj.x, ey = pi.y - pj.y, ez = pi.z - pj.z;
    ex -= G.L * nearest(ex * G.invL);
    ey -= G.L * nearest(ey * G.invL);
    ez -= G.L * nearest(ez * G.invL);
    const float r2 = ex * ex + ey * ey + ez * ez;
    batch(m, lane < m ? make_float4(ex, ey, ez, r2) : make_float4(1.f, 1.f, 1.f, 3.f), j);
  }
}

__device__ __forceinline__ PairGeom unit_vector(const float4& d) {
  const float r = sqrtf(d.w), inv = 1.f / r;
  return PairGeom{r, d.x * inv, d.y * inv, d.z * inv};
}

// Sums of the batch's terms per (species, Gaussian): lane 16 c + k adds the terms of the
// neighbors of species c in list order.  H: row per neighbor, an odd stride.
constexpr int HROW = NG + 1;

// 8 x 8000 atoms: 195 us with one thread per atom, 92 us so.
__global__ void __launch_bounds__(32 * WARP_ATOMS) k_sg_desc(const float4* pos, Geometry G,
                                                             const uint8_t* __restrict__ species,
                                                             const int* list,
                                                             const int* count, int cap,
                                                             float* __restrict__ Gout, int* __restrict__ near,
                                                             int* __restrict__ nearCount) {
  chain_wait();
  __shared__ NeighborBuffer nbuf[WARP_ATOMS];
  __shared__ float hbuf[WARP_ATOMS][32 * HROW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * WARP_ATOMS + warp;
  if (q >= G.chains * G.N) return;
  const float cdecay = __expf(-2.f * G.a * G.dmu * G.dmu);
  float* H = hbuf[warp];
  const int k = lane & (NG - 1), chain0 = q - q % G.N;   // first atom of the chain
  const unsigned flip = lane < NG ? 0xffffffffu : 0u;   // species 0 in the lower lanes
  float acc = 0.f;
  int* out = near + (size_t)q * cap;
  int total = 0;
  for_neighbors(pos, G, q, list + (size_t)q * cap, min(count[q], cap), nbuf[warp], [&](int n, float4 d, int j) {
    if (lane < n) out[total + lane] = j;
    total += n;
    float h[NG], dh[NG];
    radial(sqrtf(d.w), G, cdecay, h, dh);
#pragma unroll
    for (int u = 0; u < NG; u++) H[lane * HROW + u] = h[u];
    const unsigned mine = (__ballot_sync(0xffffffffu, species[j - chain0] != 0) ^ flip) & (0xffffffffu >> (32 - n));
    __syncwarp();
    for (int b = 0; b < n; b += 8)
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const float x = H[(b + u) * HROW + k];
        acc += (mine >> (b + u)) & 1u ? x : 0.f;
      }
    __syncwarp();
  });
  Gout[(size_t)q * DIN + lane] = acc;
  if (lane == 0) nearCount[q] = total;
}

// F_i = -sum_j s_ij r_hat_ij, s_ij = sum_k (dEdG_i[s_j, k] + dEdG_j[s_i, k]) dh_k(r_ij).
// A lane per neighbor computes dh and r_hat; then four lanes per neighbor take four
// Gaussians each, so that a neighbor's 64 bytes of dE/dG are read side by side (eight
// lines per load instead of 32), and three of them add one force component each.
// 8 x 8000 atoms: 293 us with one thread per atom, 116 us so.
constexpr int DROW = NG + 4;   // rows of 16 + 4 floats: 16-byte aligned, in different banks
__global__ void __launch_bounds__(32 * WARP_ATOMS, 4) k_sg_force(const float4* pos, Geometry G,
                                                              const uint8_t* __restrict__ species,
                                                              const int* near,
                                                              const int* nearCount, int cap,
                                                              const float* dEdG,
                                                              double* __restrict__ F) {
  chain_wait();
  // per neighbor: dh[16], r_hat[3], index
  __shared__ __align__(16) float dbuf[WARP_ATOMS][32 * DROW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * WARP_ATOMS + warp;
  if (q >= G.chains * G.N) return;
  const float cdecay = __expf(-2.f * G.a * G.dmu * G.dmu);
  const int chain0 = q - q % G.N, si = species[q - chain0];   // first atom of the chain
  const int part = lane & 3, comp = part < 3 ? part : 0;
  float* D = dbuf[warp];
  const float4* own = reinterpret_cast<const float4*>(dEdG + (size_t)q * DIN) + part;
  const float4 own0 = own[0], own1 = own[NG / 4];   // this lane's Gaussians of both species
  float f = 0.f;
  each_neighbor(pos, G, q, near + (size_t)q * cap, nearCount[q], [&](int n, float4 d, int j) {
    {
      const PairGeom pg = unit_vector(d);
      float h[NG], dh[NG];
      radial(pg.r, G, cdecay, h, dh);
      float4* row = reinterpret_cast<float4*>(D + lane * DROW);
#pragma unroll
      for (int k = 0; k < NG; k += 4) row[k / 4] = make_float4(dh[k], dh[k + 1], dh[k + 2], dh[k + 3]);
      // the sign bit of the index carries the species
      row[NG / 4] = make_float4(pg.ux, pg.uy, pg.uz, __int_as_float(species[j - chain0] ? j | (int)0x80000000 : j));
    }
    __syncwarp();
    for (int b = 0; b < n; b += 8) {
      const int nb = b + (lane >> 2);
      const float* row = D + nb * DROW;
      const int code = __float_as_int(row[NG + 3]), jj = code & 0x7FFFFFFF;
      const float4 x = code < 0 ? own1 : own0, dh = *reinterpret_cast<const float4*>(row + 4 * part);
      const float4 y = reinterpret_cast<const float4*>(dEdG + (size_t)jj * DIN + si * NG)[part];
      float s = (x.x + y.x) * dh.x + (x.y + y.y) * dh.y + (x.z + y.z) * dh.z + (x.w + y.w) * dh.w;
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (nb < n) f -= s * row[NG + comp];
    }
    __syncwarp();
  });
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
  if (lane < 3) F[3 * (size_t)q + lane] = f;
}

// u_i[s_j, k] = sum_j dh_k(r_ij) (v_i - v_j) . r_hat_ij (force residual in descriptor space).
// 8 x 8000 atoms: 248 us with one thread per atom, 93 us so.
__global__ void __launch_bounds__(32 * WARP_ATOMS, 4) k_sg_udesc(const float4* pos, Geometry G,
                                                              const uint8_t* __restrict__ species,
                                                              const int* near,
                                                              const int* nearCount, int cap,
                                                              const float4* v, float* __restrict__ U) {
  chain_wait();
  __shared__ float hbuf[WARP_ATOMS][32 * HROW];
  __shared__ float wbuf[WARP_ATOMS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * WARP_ATOMS + warp;
  if (q >= G.chains * G.N) return;
  const float cdecay = __expf(-2.f * G.a * G.dmu * G.dmu);
  float* H = hbuf[warp];
  const int k = lane & (NG - 1), chain0 = q - q % G.N;   // first atom of the chain
  const unsigned flip = lane < NG ? 0xffffffffu : 0u;   // species 0 in the lower lanes
  const float4 vi = v[q];
  float acc = 0.f;
  each_neighbor(pos, G, q, near + (size_t)q * cap, nearCount[q], [&](int n, float4 d, int j) {
    const float4 vj = v[j];
    const PairGeom pg = unit_vector(d);
    float h[NG], dh[NG];
    radial(pg.r, G, cdecay, h, dh);
#pragma unroll
    for (int u = 0; u < NG; u++) H[lane * HROW + u] = dh[u];
    wbuf[warp][lane] = (vi.x - vj.x) * pg.ux + (vi.y - vj.y) * pg.uy + (vi.z - vj.z) * pg.uz;
    const unsigned mine = (__ballot_sync(0xffffffffu, species[j - chain0] != 0) ^ flip) & (0xffffffffu >> (32 - n));
    __syncwarp();
    for (int b = 0; b < n; b += 8)
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const float x = fmaf(H[(b + u) * HROW + k], wbuf[warp][b + u], acc);
        acc = (mine >> (b + u)) & 1u ? x : acc;
      }
    __syncwarp();
  });
  U[(size_t)q * DIN + lane] = acc;
}

// ---- network: inference -----------------------------------------------------------

// tiles: (first index into the atom list, count <= 64, species)
struct TileArgs {
  const int* atoms;    // atom indices (global), species by species within each chain
  const int3* tiles;   // (start, count, species)
  int ntiles;
};

struct MlpSmem {
  WeightsSmem w[NS];
  __nv_bfloat16 X[4][16][H + 8];   // per warp activations (BF16 GEMM operand)
  __nv_bfloat16 Y[4][16][H + 8];
};

// E_i and dE/dG_i for every atom; one block per tile of <= 64 atoms of one species
__global__ void __launch_bounds__(128) k_sg_mlp(TileArgs T, const float* __restrict__ params,
                                                const float* __restrict__ Gin, float* __restrict__ Eatom,
                                                float* __restrict__ dEdG) {
  extern __shared__ __align__(16) unsigned char raw[];
  MlpSmem& S = *reinterpret_cast<MlpSmem*>(raw);
  const int3 tile = T.tiles[blockIdx.x];
  const int sp = tile.z;
  load_weights(S.w[sp], params + sp * PER_SPECIES);
  __syncthreads();
  const WeightsSmem& W = S.w[sp];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int base = tile.x + warp * 16, nrow = min(16, tile.y - warp * 16);
  if (nrow <= 0) return;
  __nv_bfloat16(*X)[H + 8] = S.X[warp];
  __nv_bfloat16(*Y)[H + 8] = S.Y[warp];
  // G rows -> X (BF16)
  for (int q = lane; q < 16 * DIN; q += 32) {
    const int r = q / DIN, k = q % DIN;
    X[r][k] = __float2bfloat16(r < nrow ? Gin[(size_t)T.atoms[base + r] * DIN + k] : 0.f);
  }
  __syncwarp();
  float z1[8][4], z2[8][4];
  zero(z1);
  warp_gemm<DIN, 8>(&X[0][0], H + 8, &W.W1t[0][0], DIN + 8, z1);
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      z1[n][q] += W.b1[frag_col(n, q)];
      Y[frag_row(q)][frag_col(n, q)] = __float2bfloat16(silu(z1[n][q]));
    }
  __syncwarp();
  zero(z2);
  warp_gemm<H, 8>(&Y[0][0], H + 8, &W.W2t[0][0], H + 8, z2);
  float e[2] = {0.f, 0.f};   // rows g and g + 8
  __syncwarp();
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int col = frag_col(n, q);
      const float z = z2[n][q] + W.b2[col];
      e[q >> 1] += W.w3[col] * silu(z);
      X[frag_row(q)][col] = __float2bfloat16(W.w3[col] * dsilu(z));   // dE/dz2
    }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    e[h] += __shfl_xor_sync(0xffffffffu, e[h], 1);
    e[h] += __shfl_xor_sync(0xffffffffu, e[h], 2);
  }
  if ((lane & 3) == 0) {
    const int g = lane >> 2;
    if (g < nrow) Eatom[T.atoms[base + g]] = e[0] + W.b3;
    if (g + 8 < nrow) Eatom[T.atoms[base + g + 8]] = e[1] + W.b3;
  }
  __syncwarp();
  float d1[8][4];
  zero(d1);
  warp_gemm<H, 8>(&X[0][0], H + 8, &W.W2[0][0], H + 8, d1);   // dE/da1 = dE/dz2 W2^T
  __syncwarp();
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int q = 0; q < 4; q++) Y[frag_row(q)][frag_col(n, q)] = __float2bfloat16(d1[n][q] * dsilu(z1[n][q]));
  __syncwarp();
  float dg[4][4];
  zero(dg);
  warp_gemm<H, 4>(&Y[0][0], H + 8, &W.W1[0][0], H + 8, dg);   // dE/dG = dE/dz1 W1^T
#pragma unroll
  for (int n = 0; n < 4; n++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = frag_row(q);
      if (r < nrow) dEdG[(size_t)T.atoms[base + r] * DIN + frag_col(n, q)] = dg[n][q];
    }
}

// ---- network: inference on the 5th-generation tensor cores (tcgen05) --------------
//
// The same computation as k_sg_mlp (BF16 operands rounded at the same points, FP32
// accumulation) with tcgen05.mma: M = 128 atoms per tile (one species), operands in
// shared memory in the canonical K-major layout without swizzle, accumulators in
// tensor memory.  Persistent blocks of 256 threads take 128-atom tiles in turn and load
// the BF16 weights of a species at their first tile of it; threads r and r + 128 own row
// r of a tile, TMEM lane r (warp w reads lanes 32 (w mod 4).. + 31), and half of its
// columns each.  The kernel is bound by the latency of a tile's chain (loads, four GEMMs,
// 64 columns of silu and its derivative per row in between): with one thread per row and
// both species' weights loaded up front 8 x 8000 atoms took 67 us, so 37.  Thread 0
// issues each GEMM (one tcgen05.mma per K = 16) and commits it to an mbarrier that
// every thread waits on.  Per tile:
//   Z1 = G W1          TMEM columns   0..63   (K = 32)
//   A1 = silu(Z1 + b1) -> smem X,  Z2 = A1 W2               columns  64..127
//   E = w3 . silu(Z2 + b2) + b3,  dZ2 = w3 silu'(Z2 + b2) -> X
//   dA1 = dZ2 W2^T                                          columns 128..191
//   dZ1 = dA1 silu'(Z1 + b1) -> X,  dE/dG = dZ1 W1^T        columns 192..223 (N = 32)
// Waits are bounded: a wait that runs out sets *err, the block stops taking tiles,
// frees its tensor memory and returns (the host reports the error).

constexpr int TC_M = 128, TC_COLS = 256, TC_THREADS = 2 * TC_M;

// byte offset of element (r, k) of a K-major operand with K columns: 8 x 16-byte core
// matrices, consecutive along K (leading byte offset 128), row groups of 8 K/8 core
// matrices apart (stride byte offset 16 K)
__host__ __device__ constexpr int tc_off(int r, int k, int K) {
  return (r >> 3) * (K * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

struct TcWeights {   // one species, BF16 B operands (rows n, K contiguous) and FP32 vectors
  alignas(128) unsigned char B1[64 * 32 * 2];   // Z1:  B1[n][k] = W1[k][n]   (N 64, K 32)
  alignas(128) unsigned char B2[64 * 64 * 2];   // Z2:  B2[n][k] = W2[k][n]   (N 64, K 64)
  alignas(128) unsigned char B3[64 * 64 * 2];   // dA1: B3[n][k] = W2[n][k]   (N 64, K 64)
  alignas(128) unsigned char B4[32 * 64 * 2];   // dG:  B4[n][k] = W1[n][k]   (N 32, K 64)
  float b1[H], b2[H], w3[H], b3;
};

struct TcSmem {
  TcWeights w[NS];
  alignas(128) unsigned char G[TC_M * DIN * 2];   // A operand of Z1 (K 32)
  alignas(128) unsigned char X[TC_M * H * 2];     // A operand of the other GEMMs (K 64)
  float epart[TC_M];   // energies of the upper columns
  alignas(8) unsigned long long bar;
  unsigned int taddr;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start address, leading and stride byte offsets,
// descriptor version 1, no swizzle
__device__ __forceinline__ unsigned long long tc_sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N
__host__ __device__ constexpr uint32_t tc_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[128 x K] B[K x N], issued by one thread, K / 16 instructions
template <int K, int N>
__device__ __forceinline__ void tc_gemm(uint32_t dtmem, const unsigned char* A, const unsigned char* B) {
  const uint32_t a0 = smem_u32(A), b0 = smem_u32(B);
  constexpr uint32_t idesc = tc_idesc(TC_M, N);
#pragma unroll
  for (int s = 0; s < K / 16; s++) {
    const unsigned long long ad = tc_sdesc(a0 + 256u * s, 128u, 16u * K), bd = tc_sdesc(b0 + 256u * s, 128u, 16u * K);
    const uint32_t acc = s > 0 ? 1u : 0u;
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
  }
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

// bounded wait for the phase; false if it did not complete
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t phase) {
  for (int i = 0; i < (1 << 22); i++) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 or 32 consecutive FP32 columns of this thread's TMEM lane; tc_ld_wait before their use
__device__ __forceinline__ void tc_ld(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tc_ld(uint32_t taddr, float (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
        "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
        "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
      : "r"(taddr));
}
template <int N>
__device__ __forceinline__ void tc_ld_wait(float (&v)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < N; q++) asm volatile("" : "+f"(v[q]));   // the values are read after the wait
}

// 8 BF16 values (from 8 floats) into one 16-byte chunk of a K-major operand
__device__ __forceinline__ void tc_st8(unsigned char* base, int r, int k, int K, const float* v) {
  uint4 w;
  __nv_bfloat162 h[4];
#pragma unroll
  for (int q = 0; q < 4; q++) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
  memcpy(&w, h, 16);
  *reinterpret_cast<uint4*>(base + tc_off(r, k, K)) = w;
}

// Called by all TC_THREADS threads; four consecutive n at a time, every load in flight
__device__ void tc_load_weights(TcWeights& w, const float* p) {
  constexpr int L1 = DIN * H / 4 / TC_THREADS, L2 = H * H / 4 / TC_THREADS;
  static_assert(DIN * H == 4 * TC_THREADS * L1 && H * H == 4 * TC_THREADS * L2, "whole rounds of loads");
  float x[L1 + L2][4];
#pragma unroll
  for (int r = 0; r < L1 + L2; r++) {
    const float* src = p + (r < L1 ? OFF_W1 + 4 * (r * TC_THREADS + threadIdx.x)
                                   : OFF_W2 + 4 * ((r - L1) * TC_THREADS + threadIdx.x));
#pragma unroll
    for (int v = 0; v < 4; v++) x[r][v] = src[v];
  }
#pragma unroll
  for (int r = 0; r < L1 + L2; r++) {
    const bool first = r < L1;   // W1[k][n], else W2[k][n]
    const int q = 4 * ((first ? r : r - L1) * TC_THREADS + (int)threadIdx.x), k = q / H, n = q % H;
    const int K = first ? DIN : H;
    unsigned char* Bt = first ? w.B1 : w.B2;   // Bt[n][k]
    unsigned char* B = first ? w.B4 : w.B3;    // B[k][n] (rows: input or a1 index)
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const __nv_bfloat16 b = __float2bfloat16(x[r][v]);
      *reinterpret_cast<__nv_bfloat16*>(Bt + tc_off(n + v, k, K)) = b;
      *reinterpret_cast<__nv_bfloat16*>(B + tc_off(k, n + v, H)) = b;
    }
  }
  for (int q = threadIdx.x; q < H; q += TC_THREADS) {
    w.b1[q] = p[OFF_B1 + q];
    w.b2[q] = p[OFF_B2 + q];
    w.w3[q] = p[OFF_W3 + q];
  }
  if (threadIdx.x == 0) w.b3 = p[OFF_B3];
}

__global__ void __launch_bounds__(TC_THREADS, 2) k_sg_mlp_tc(TileArgs T, const float* params,
                                                             const float* Gin,
                                                             float* __restrict__ Eatom, float* __restrict__ dEdG,
                                                             int* __restrict__ err) {
  chain_wait();
  extern __shared__ __align__(1024) unsigned char raw[];
  TcSmem& S = *reinterpret_cast<TcSmem*>(raw);
  const int t = threadIdx.x, warp = t >> 5, row = t % TC_M, half = t / TC_M;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.taddr)),
                 "r"(TC_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  proxy_fence();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = S.taddr, bar = smem_u32(&S.bar);
  const uint32_t lane_base = (uint32_t)(32 * (warp & 3)) << 16;   // this warp's TMEM lanes
  constexpr int HC = H / 2, GC = DIN / 2;   // columns of a thread
  const int c0 = half * HC, g0 = half * GC;
  unsigned loaded = 0;   // species whose weights are in place
  uint32_t phase = 0;
  bool ok = true;
  // one GEMM: operands written by all threads before, accumulator read by all after;
  // ok stays block-uniform (every thread leaves the tile loop together)
  auto run = [&](auto&& issue) {
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    if (t == 0) {
      tc_fence_after();
      issue();
      tc_commit(bar);
    }
    ok = __syncthreads_and(tc_wait(bar, phase) ? 1 : 0) != 0;
    if (ok) phase ^= 1u;
    tc_fence_after();
  };
  for (int ti = blockIdx.x; ti < T.ntiles; ti += gridDim.x) {
    const int3 tile = T.tiles[ti];
    const TcWeights& W = S.w[tile.z];
    if (!(loaded >> tile.z & 1u)) {   // read by the GEMMs after the fence and barrier of run
      tc_load_weights(S.w[tile.z], params + tile.z * PER_SPECIES);
      loaded |= 1u << tile.z;
    }
    const bool have = row < tile.y;
    const int atom = have ? T.atoms[tile.x + row] : 0;
    {   // G row -> BF16 A operand
      float g[GC];
#pragma unroll
      for (int k = 0; k < GC; k += 4) {
        const float4 v =
            have ? *reinterpret_cast<const float4*>(Gin + (size_t)atom * DIN + g0 + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        g[k] = v.x;
        g[k + 1] = v.y;
        g[k + 2] = v.z;
        g[k + 3] = v.w;
      }
#pragma unroll
      for (int k = 0; k < GC; k += 8) tc_st8(S.G, row, g0 + k, DIN, g + k);
    }
    run([&] { tc_gemm<DIN, H>(tm + 0, S.G, W.B1); });
    if (!ok) break;
    float z[HC];
    tc_ld(tm + lane_base + c0, z);   // A1 = silu(Z1 + b1)
    tc_ld_wait(z);
#pragma unroll
    for (int q = 0; q < HC; q++) z[q] = silu(z[q] + W.b1[c0 + q]);
#pragma unroll
    for (int q = 0; q < HC; q += 8) tc_st8(S.X, row, c0 + q, H, z + q);
    run([&] { tc_gemm<H, H>(tm + 64, S.X, W.B2); });
    if (!ok) break;
    float e = 0.f;
    tc_ld(tm + lane_base + 64 + c0, z);   // E and dE/dZ2
    tc_ld_wait(z);
#pragma unroll
    for (int q = 0; q < HC; q++) {
      const float u = z[q] + W.b2[c0 + q];
      e += W.w3[c0 + q] * silu(u);
      z[q] = W.w3[c0 + q] * dsilu(u);
    }
#pragma unroll
    for (int q = 0; q < HC; q += 8) tc_st8(S.X, row, c0 + q, H, z + q);
    if (half == 1) S.epart[row] = e;
    run([&] { tc_gemm<H, H>(tm + 128, S.X, W.B3); });
    if (!ok) break;
    if (half == 0 && have) Eatom[atom] = (e + S.epart[row]) + W.b3;
    float d[HC];
    tc_ld(tm + lane_base + 128 + c0, d);   // dE/dZ1 = dE/dA1 silu'(Z1 + b1)
    tc_ld(tm + lane_base + c0, z);
    tc_ld_wait(d);
    tc_ld_wait(z);
#pragma unroll
    for (int q = 0; q < HC; q++) d[q] *= dsilu(z[q] + W.b1[c0 + q]);
#pragma unroll
    for (int q = 0; q < HC; q += 8) tc_st8(S.X, row, c0 + q, H, d + q);
    run([&] { tc_gemm<H, DIN>(tm + 192, S.X, W.B4); });
    if (!ok) break;
    float o[GC];
    tc_ld(tm + lane_base + 192 + g0, o);   // dE/dG
    tc_ld_wait(o);
    if (have)
#pragma unroll
      for (int q = 0; q < GC; q += 4)
        *reinterpret_cast<float4*>(dEdG + (size_t)atom * DIN + g0 + q) = make_float4(o[q], o[q + 1], o[q + 2], o[q + 3]);
  }
  if (!ok && t == 0) {
    atomicExch(err, 1);
    tc_wait(bar, phase);   // the GEMM in flight, if it completes after all (bounded)
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(TC_COLS) : "memory");
  }
}

// ---- network: training gradient -----------------------------------------------------
//
// Per atom: O_i = e_c(i) E_i - t_i,  t_i = dE_i/dG_i . u_i.  With z1 = G W1 + b1,
// a1 = silu(z1), z2 = a1 W2 + b2, a2 = silu(z2), E = a2 . w3 + b3 and the tangent
// dz1 = u W1, da1 = silu'(z1) dz1, dz2 = da1 W2, da2 = silu'(z2) dz2, t = da2 . w3:
//   dO/dw3 = e a2 - da2,                 dO/db3 = e
//   gz2  = e w3 silu'(z2) - w3 dz2 silu''(z2)        (dO/dz2)
//   gdz2 = -w3 silu'(z2)                               (dO/ddz2)
//   dO/dW2 = a1^T gz2 + da1^T gdz2,       dO/db2 = gz2
//   gz1  = (gz2 W2^T) silu'(z1) + (gdz2 W2^T) dz1 silu''(z1)
//   gdz1 = (gdz2 W2^T) silu'(z1)
//   dO/dW1 = G^T gz1 + u^T gdz1,          dO/db1 = gz1
// The weight gradients are GEMMs over the tile's atoms: [A1; dA1]^T [GZ2; GDZ2] and
// [G; U]^T [GZ1; GDZ1], K = 2 x 64 atoms, on the tensor cores.

struct TrainSmem {
  WeightsSmem w;
  __nv_bfloat16 in[2 * TILE][DIN + 8];       // rows: G (64), U (64)
  __nv_bfloat16 act[2 * TILE][H + 8];        // rows: a1 (64), da1 (64)
  __nv_bfloat16 gz2[2 * TILE][H + 8];        // rows: gz2 (64), gdz2 (64)
  __nv_bfloat16 gz1[2 * TILE][H + 8];        // rows: gz1 (64), gdz1 (64)
  float vb1[4][H], vb2[4][H], vw3[4][H], vb3[4];   // per warp
};

// Sums over the rows of a warp's fragments (rows g and g + 8 in slots q = 0, 1 and 2, 3):
// x[n][j] is this lane's sum for column 8 n + 2 t + j; lanes of equal t are added and
// the total goes to out[column].
__device__ __forceinline__ void column_sums(float (&x)[8][2], float* out) {
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int j = 0; j < 2; j++) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) x[n][j] += __shfl_xor_sync(0xffffffffu, x[n][j], o);
      if ((threadIdx.x & 31) < 4) out[frag_col(n, j)] += x[n][j];
    }
}

// Both species in one launch: blocks 0 .. nb0 - 1 process the tiles of species 0 (the
// first nt0 of T), the others those of species 1; each writes its gradient partial
// (PER_SPECIES floats) to part[b].  Bias and output-layer gradients are summed by
// shuffles per warp (shared-memory atomics, eight lanes to an address, were most of
// 2 x 419 us at 8 x 8000 atoms; 173 us so); the weight GEMMs take their operands
// transposed by ldmatrix, so that two blocks fit an SM (91 us).
__global__ void __launch_bounds__(128) k_sg_train(TileArgs T, int nt0, int nb0, const float* params,
                                                  const float* Gin, const float* Uin,
                                                  const float* eAtom, float* __restrict__ part) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(raw);
  const int species = (int)blockIdx.x < nb0 ? 0 : 1;
  const int t0 = species == 0 ? blockIdx.x : nt0 + blockIdx.x - nb0, t1 = species == 0 ? nt0 : T.ntiles,
            tstep = species == 0 ? nb0 : gridDim.x - nb0;
  load_weights(S.w, params + species * PER_SPECIES);
  for (int q = threadIdx.x; q < 4 * H; q += blockDim.x) (&S.vb1[0][0])[q] = (&S.vb2[0][0])[q] = (&S.vw3[0][0])[q] = 0.f;
  if (threadIdx.x < 4) S.vb3[threadIdx.x] = 0.f;
  __syncthreads();
  const WeightsSmem& W = S.w;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // weight-gradient accumulators: W2 (64 x 64): warp w owns rows 16w..16w+15 (8 n-tiles);
  // W1 (32 x 64): warp w owns rows 16 (w & 1).., columns 32 (w >> 1).. (4 n-tiles)
  float gW2[8][4], gW1[4][4];
  zero(gW2);
  zero(gW1);
  for (int ti = t0; ti < t1; ti += tstep) {
    const int3 tile = T.tiles[ti];
    const int r0 = warp * 16;   // this warp's rows in the tile
    const int nrow = max(0, min(16, tile.y - r0));
    // inputs: G and U rows (zero rows beyond the tile)
    for (int q = lane; q < 16 * DIN; q += 32) {
      const int r = q / DIN, k = q % DIN;
      const bool ok = r < nrow;
      const size_t a = ok ? (size_t)T.atoms[tile.x + r0 + r] : 0;
      S.in[r0 + r][k] = __float2bfloat16(ok ? Gin[a * DIN + k] : 0.f);
      S.in[TILE + r0 + r][k] = __float2bfloat16(ok ? Uin[a * DIN + k] : 0.f);
    }
    __syncwarp();
    float z1[8][4], dz1[8][4];
    zero(z1);
    zero(dz1);
    warp_gemm<DIN, 8>(&S.in[r0][0], DIN + 8, &W.W1t[0][0], DIN + 8, z1);
    warp_gemm<DIN, 8>(&S.in[TILE + r0][0], DIN + 8, &W.W1t[0][0], DIN + 8, dz1);
#pragma unroll
    for (int n = 0; n < 8; n++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = frag_row(q), c = frag_col(n, q);
        z1[n][q] += W.b1[c];
        const float a = r < nrow ? silu(z1[n][q]) : 0.f, da = r < nrow ? dsilu(z1[n][q]) * dz1[n][q] : 0.f;
        S.act[r0 + r][c] = __float2bfloat16(a);
        S.act[TILE + r0 + r][c] = __float2bfloat16(da);
      }
    __syncwarp();
    float z2[8][4], dz2[8][4];
    zero(z2);
    zero(dz2);
    warp_gemm<H, 8>(&S.act[r0][0], H + 8, &W.W2t[0][0], H + 8, z2);
    warp_gemm<H, 8>(&S.act[TILE + r0][0], H + 8, &W.W2t[0][0], H + 8, dz2);
    float e[2];
    {
      const int g = lane >> 2;
      e[0] = g < nrow ? eAtom[T.atoms[tile.x + r0 + g]] : 0.f;
      e[1] = g + 8 < nrow ? eAtom[T.atoms[tile.x + r0 + g + 8]] : 0.f;
    }
    float lb3 = 0.f, sb2[8][2], sw3[8][2];
#pragma unroll
    for (int n = 0; n < 8; n++) {
      sb2[n][0] = sb2[n][1] = sw3[n][0] = sw3[n][1] = 0.f;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = frag_row(q), c = frag_col(n, q);
        const float ec = e[q >> 1], z = z2[n][q] + W.b2[c], w3 = W.w3[c];
        const float s1 = dsilu(z), s2 = d2silu(z);
        const float g2 = ec * w3 * s1 - w3 * dz2[n][q] * s2, gd2 = -w3 * s1;
        const bool ok = r < nrow;
        S.gz2[r0 + r][c] = __float2bfloat16(ok ? g2 : 0.f);
        S.gz2[TILE + r0 + r][c] = __float2bfloat16(ok ? gd2 : 0.f);
        if (ok) {
          sb2[n][q & 1] += g2;
          sw3[n][q & 1] += ec * silu(z) - s1 * dz2[n][q];
        }
        if (ok && n == 0 && (q & 1) == 0 && (threadIdx.x & 3) == 0) lb3 += ec;
      }
    }
    column_sums(sb2, S.vb2[warp]);
    column_sums(sw3, S.vw3[warp]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lb3 += __shfl_xor_sync(0xffffffffu, lb3, o);
    if (lane == 0) S.vb3[warp] += lb3;
    __syncwarp();
    float p1[8][4], p2[8][4];
    zero(p1);
    zero(p2);
    warp_gemm<H, 8>(&S.gz2[r0][0], H + 8, &W.W2[0][0], H + 8, p1);          // gz2 W2^T
    warp_gemm<H, 8>(&S.gz2[TILE + r0][0], H + 8, &W.W2[0][0], H + 8, p2);   // gdz2 W2^T
    float sb1[8][2];
#pragma unroll
    for (int n = 0; n < 8; n++) {
      sb1[n][0] = sb1[n][1] = 0.f;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = frag_row(q), c = frag_col(n, q);
        const float s1 = dsilu(z1[n][q]), s2 = d2silu(z1[n][q]);
        const bool ok = r < nrow;
        const float g1 = p1[n][q] * s1 + p2[n][q] * dz1[n][q] * s2, gd1 = p2[n][q] * s1;
        S.gz1[r0 + r][c] = __float2bfloat16(ok ? g1 : 0.f);
        S.gz1[TILE + r0 + r][c] = __float2bfloat16(ok ? gd1 : 0.f);
        if (ok) sb1[n][q & 1] += g1;
      }
    }
    column_sums(sb1, S.vb1[warp]);
    __syncthreads();
    // dW2 += [a1; da1]^T [gz2; gdz2] (64 x 64 over 128 atoms), dW1 += [G; U]^T [gz1; gdz1]
    // (32 x 64)
    warp_gemm_t<2 * TILE, 8>(&S.act[0][16 * warp], H + 8, &S.gz2[0][0], H + 8, gW2);
    warp_gemm_t<2 * TILE, 4>(&S.in[0][16 * (warp & 1)], DIN + 8, &S.gz1[0][32 * (warp >> 1)], H + 8, gW1);
    __syncthreads();
  }
  // block partial, FP32: layout of the packed parameters of one species
  float* out = part + (size_t)blockIdx.x * PER_SPECIES;
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int q = 0; q < 4; q++) out[OFF_W2 + (16 * warp + frag_row(q)) * H + frag_col(n, q)] = gW2[n][q];
#pragma unroll
  for (int n = 0; n < 4; n++)
#pragma unroll
    for (int q = 0; q < 4; q++)
      out[OFF_W1 + (16 * (warp & 1) + frag_row(q)) * H + 32 * (warp >> 1) + frag_col(n, q)] = gW1[n][q];
  __syncthreads();
  for (int q = threadIdx.x; q < H; q += blockDim.x) {
    out[OFF_B1 + q] = S.vb1[0][q] + S.vb1[1][q] + S.vb1[2][q] + S.vb1[3][q];
    out[OFF_B2 + q] = S.vb2[0][q] + S.vb2[1][q] + S.vb2[2][q] + S.vb2[3][q];
    out[OFF_W3 + q] = S.vw3[0][q] + S.vw3[1][q] + S.vw3[2][q] + S.vw3[3][q];
  }
  if (threadIdx.x == 0) out[OFF_B3] = S.vb3[0] + S.vb3[1] + S.vb3[2] + S.vb3[3];
}

// grad[species][p] = sum over the species' blocks of part[b][p]: 8 slices of the blocks
// per parameter, each in order, then the slices in order
constexpr int REDUCE_PARAMS = 32, REDUCE_SLICES = 8;
__global__ void __launch_bounds__(REDUCE_PARAMS * REDUCE_SLICES) k_sg_reduce(const float* __restrict__ part, int nb0,
                                                                             int blocks, float* __restrict__ grad) {
  __shared__ float sum[REDUCE_SLICES][REDUCE_PARAMS];
  const int x = threadIdx.x % REDUCE_PARAMS, y = threadIdx.x / REDUCE_PARAMS;
  const int p = blockIdx.x * REDUCE_PARAMS + x, species = blockIdx.y;
  const int b0 = species == 0 ? 0 : nb0, b1 = species == 0 ? nb0 : blocks, per = (b1 - b0 + REDUCE_SLICES - 1) / REDUCE_SLICES;
  float s = 0.f;
  if (p < PER_SPECIES)
#pragma unroll 8
    for (int b = b0 + y * per; b < min(b1, b0 + (y + 1) * per); b++) s += part[(size_t)b * PER_SPECIES + p];
  sum[y][x] = s;
  __syncthreads();
  if (y != 0 || p >= PER_SPECIES) return;
  for (int k = 1; k < REDUCE_SLICES; k++) s += sum[k][x];
  grad[species * PER_SPECIES + p] = s;
}

// Residuals of the loss: per atom e = wE 2 (E_c - Etrue_c) / (N^2 C) of its chain and the
// vector v = wF 2 / (3 N C) (F - Ftrue); out[0] = sum (E - Etrue)^2, out[1] = sum |F - Ftrue|^2.
constexpr int RES_THREADS = 256;
__global__ void __launch_bounds__(RES_THREADS) k_sg_residual(const double* __restrict__ F,
                                                             const double* __restrict__ Ft,
                                                             const double* __restrict__ E,
                                                             const double* __restrict__ Et, int C, int N, double wE,
                                                             double fscale, float4* __restrict__ v,
                                                             float* __restrict__ eAtom, double* partials,
                                                             unsigned int* ticket, double* out, double* hostOut) {
  const int total = C * N;
  double s[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    float w[3];
    for (int k = 0; k < 3; k++) {
      const double d = __dsub_rn(F[3 * (size_t)i + k], Ft[3 * (size_t)i + k]);
      s[1] = __dadd_rn(s[1], __dmul_rn(d, d));
      w[k] = (float)__dmul_rn(fscale, d);
    }
    v[i] = make_float4(w[0], w[1], w[2], 0.f);
    const int c = i / N;
    const double x = __dsub_rn(E[c], Et[c]);
    eAtom[i] = (float)(wE * 2.0 * x / ((double)N * N * C));
    if (i == c * N) s[0] = __dadd_rn(s[0], __dmul_rn(x, x));
  }
  grid_reduce<2, RES_THREADS>(s, partials, ticket, out, hostOut);
}

__global__ void k_sg_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                          float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// per-chain sums of per-atom FP32 values in a fixed order (a block per chain)
__global__ void k_sg_chain_sum(const float* __restrict__ x, int N, double* __restrict__ out) {
  const int c = blockIdx.x;
  __shared__ double ws[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) s += (double)x[(size_t)c * N + i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += ws[w];
    out[c] = t;
  }
}

// velocity Verlet pieces for the chains (FP64, unit masses): END ends a step with a kick of
// half, BEGIN begins the next with a kick of half, the drift over dt and the FP32
// positions of k_sg_pack.  One pass per step instead of three.
template <bool END, bool BEGIN>
__global__ void k_sg_advance(double* __restrict__ R, double* __restrict__ P, const double* F, int n3,
                             double half, double dt, double L, float* __restrict__ pos) {
  chain_wait();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n3) return;
  const double f = half * F[q];
  double p = P[q];
  if (END) p = p + f;
  if (BEGIN) p = p + f;
  P[q] = p;
  if (BEGIN) {
    const double x = R[q] + dt * p;
    R[q] = x;
    pos[4 * (q / 3) + q % 3] = wrapped(x, L);
  }
}

}  // namespace sg

// ---- host ---------------------------------------------------------------------------

struct Surrogate {
  sg::Geometry G;
  int total = 0, cap = 0;
  double L = 0, skin = 0;
  uint8_t* dSpecies = nullptr;
  std::vector<int3> tiles, tiles128;   // tiles of <= 64 and of <= 128 atoms of one species
  int* dAtoms = nullptr;
  int3* dTiles = nullptr;
  int3* dTiles128 = nullptr;
  int* dTcError = nullptr;
  float4* dPos = nullptr;
  int *dCellOf = nullptr, *dCounts = nullptr, *dStarts = nullptr, *dCursor = nullptr, *dSorted = nullptr;
  int *dList = nullptr, *dCount = nullptr, *dOverflow = nullptr;
  int *dNear = nullptr, *dNearCount = nullptr;   // neighbors within rc at the positions of the last k_sg_desc
  float *dG = nullptr, *dEatom = nullptr, *dEdG = nullptr, *dU = nullptr, *dEres = nullptr;
  float4* dV = nullptr;
  float *dParams = nullptr, *dPart = nullptr, *dGrad = nullptr, *dM = nullptr, *dVar = nullptr;
  int trainBlocks = 0, trainBlocks0 = 0, tiles0 = 0;   // blocks of k_sg_train, those of species 0, tiles of species 0
  int3* dTrainTiles = nullptr;                          // the tiles of <= 64 atoms, species 0 first
  double *dF = nullptr, *dE = nullptr;                  // forces and energies of EmDee_surrogate_gradient
  double *dResPart = nullptr, *hLoss = nullptr;         // partials, then the sums; pinned sums
  unsigned int* dTicket = nullptr;
  double* dR0 = nullptr;   // positions of the last list build
};

static int sg_blocks(int n) { return (n + 255) / 256; }
static int sg_warp_blocks(int n) { return (n + sg::WARP_ATOMS - 1) / sg::WARP_ATOMS; }
static const int SG_RES_BLOCKS = 2 * 152;

static void sg_build_lists(Surrogate& S, const double* dR, cudaStream_t st) {
  using namespace sg;
  const int cells = S.G.chains * S.G.M * S.G.M * S.G.M;
  k_sg_pack<<<sg_blocks(S.total), 256, 0, st>>>(dR, S.total, S.L, S.dPos);
  CK(cudaMemsetAsync(S.dCounts, 0, sizeof(int) * cells, st));
  CK(cudaMemsetAsync(S.dCursor, 0, sizeof(int) * cells, st));
  k_sg_count<<<sg_blocks(S.total), 256, 0, st>>>(S.dPos, S.G, S.dCellOf, S.dCounts);
  k_sg_scan<<<1, 256, 0, st>>>(S.dCounts, cells, S.dStarts);
  k_sg_scatter<<<sg_blocks(S.total), 256, 0, st>>>(S.dCellOf, S.G, S.dStarts, S.dCursor, S.dSorted);
  const bool sparse = cells > S.total;
  const int per = sparse ? 256 : 8;   // cells per block
  (sparse ? k_sg_sort<true> : k_sg_sort<false>)<<<(cells + per - 1) / per, 256, 0, st>>>(S.dStarts, cells, S.dSorted);
  (sparse ? k_sg_list<true> : k_sg_list<false>)<<<std::min(cells, S.total), LIST_THREADS, 0, st>>>(
      S.dPos, S.G, S.dStarts, S.dSorted, S.dCellOf, S.cap, S.dList, S.dCount, S.dOverflow);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(S.dR0, dR, sizeof(double) * 3 * S.total, cudaMemcpyDeviceToDevice, st));
}

// Dynamic shared memory of k_sg_mlp_tc: at least 100 KB, so that at most two blocks
// (2 x 256 tensor-memory columns of the SM's 512) share an SM.
static size_t tc_smem_bytes() { return std::max(sizeof(sg::TcSmem) + 1024, (size_t)100 * 1024); }

// The network: tcgen05 kernel (default) or the mma.sync one (EMDEE_SG_MMA=sync).
static void sg_network(Surrogate& S, const float* dParams, cudaStream_t st) {
  using namespace sg;
  const char* e = getenv("EMDEE_SG_MMA");
  if (e && !strcmp(e, "sync")) {
    TileArgs T{S.dAtoms, S.dTiles, (int)S.tiles.size()};
    k_sg_mlp<<<T.ntiles, 128, sizeof(MlpSmem), st>>>(T, dParams, S.dG, S.dEatom, S.dEdG);
  } else {
    TileArgs T{S.dAtoms, S.dTiles128, (int)S.tiles128.size()};
    const int blocks = std::min(T.ntiles, 2 * 152);
    launch_chained(k_sg_mlp_tc, blocks, TC_THREADS, tc_smem_bytes(), st, T, dParams, S.dG, S.dEatom, S.dEdG, S.dTcError);
  }
  CK(cudaGetLastError());
}

}  // namespace emdee

using namespace emdee;

extern "C" {

int EmDee_surrogate_param_count(void) { return sg::NPARAM; }

// chains x N atoms (positions chain-major, FP64 [chains][N][3]); types[N] in {1, 2},
// shared by all chains; cubic box L; descriptor cut-off rc; Verlet-list skin; Gaussian
// centres mu0..mu15 (uniform), width w
void* EmDee_surrogate_create(int chains, int N, double L, const int* types, double rc, double skin, double mu0,
                             double mu15, double width) {
  using namespace sg;
  const char* task = "surrogate setup";
  if (chains < 1 || N < 2 || !(L > 0) || !(rc > 0)) fatal(task, "invalid arguments");
  Surrogate* S = new Surrogate;
  S->total = chains * N;
  S->L = L;
  S->skin = skin;
  Geometry& G = S->G;
  G.chains = chains;
  G.N = N;
  G.M = std::max(1, (int)std::floor(L / (rc + skin)));
  G.L = (float)L;
  G.invL = (float)(1.0 / L);
  G.rc = (float)rc;
  G.rc2 = (float)(rc * rc);
  G.rlist2 = (float)((rc + skin) * (rc + skin));
  G.mu0 = (float)mu0;
  G.dmu = (float)((mu15 - mu0) / 15.0);
  G.a = (float)(1.0 / (2.0 * width * width));
  std::vector<uint8_t> sp(N);
  for (int i = 0; i < N; i++) {
    if (types[i] != 1 && types[i] != 2) fatal(task, "species must be 1 or 2");
    sp[i] = (uint8_t)(types[i] - 1);
  }
  CK(cudaMalloc(&S->dSpecies, N));
  CK(cudaMemcpy(S->dSpecies, sp.data(), N, cudaMemcpyHostToDevice));
  // tiles of <= 64 atoms of one species, chain by chain, and over the same atom
  // list tiles of <= 128 (the tensor-memory kernel's M)
  std::vector<int> atoms;
  for (int c = 0; c < chains; c++)
    for (int s = 0; s < NS; s++) {
      std::vector<int> list;
      for (int i = 0; i < N; i++)
        if (sp[i] == s) list.push_back(c * N + i);
      const int first = (int)atoms.size();
      for (size_t b = 0; b < list.size(); b += TILE) {
        const int cnt = (int)std::min<size_t>(TILE, list.size() - b);
        S->tiles.push_back(make_int3((int)atoms.size(), cnt, s));
        atoms.insert(atoms.end(), list.begin() + b, list.begin() + b + cnt);
      }
      for (size_t b = 0; b < list.size(); b += TC_M)
        S->tiles128.push_back(make_int3(first + (int)b, (int)std::min<size_t>(TC_M, list.size() - b), s));
    }
  CK(cudaMalloc(&S->dAtoms, sizeof(int) * atoms.size()));
  CK(cudaMemcpy(S->dAtoms, atoms.data(), sizeof(int) * atoms.size(), cudaMemcpyHostToDevice));
  CK(cudaMalloc(&S->dTiles, sizeof(int3) * S->tiles.size()));
  CK(cudaMemcpy(S->dTiles, S->tiles.data(), sizeof(int3) * S->tiles.size(), cudaMemcpyHostToDevice));
  CK(cudaMalloc(&S->dTiles128, sizeof(int3) * S->tiles128.size()));
  CK(cudaMemcpy(S->dTiles128, S->tiles128.data(), sizeof(int3) * S->tiles128.size(), cudaMemcpyHostToDevice));
  CK(cudaMalloc(&S->dTcError, sizeof(int)));
  CK(cudaMemset(S->dTcError, 0, sizeof(int)));
  const int cells = chains * G.M * G.M * G.M;
  const double rho = N / (L * L * L);
  S->cap = std::max(64, ((int)(2.0 * 4.18879 * std::pow(rc + skin, 3) * rho) + 31) / 32 * 32);
  const size_t T = S->total;
  CK(cudaMalloc(&S->dPos, sizeof(float4) * T));
  CK(cudaMalloc(&S->dCellOf, sizeof(int) * T));
  CK(cudaMalloc(&S->dCounts, sizeof(int) * cells));
  CK(cudaMalloc(&S->dCursor, sizeof(int) * cells));
  CK(cudaMalloc(&S->dStarts, sizeof(int) * (cells + 1)));
  CK(cudaMalloc(&S->dSorted, sizeof(int) * T));
  CK(cudaMalloc(&S->dList, sizeof(int) * T * S->cap));
  CK(cudaMalloc(&S->dCount, sizeof(int) * T));
  CK(cudaMalloc(&S->dOverflow, sizeof(int)));
  CK(cudaMemset(S->dOverflow, 0, sizeof(int)));
  CK(cudaMalloc(&S->dG, sizeof(float) * T * DIN));
  CK(cudaMalloc(&S->dU, sizeof(float) * T * DIN));
  CK(cudaMalloc(&S->dEdG, sizeof(float) * T * DIN));
  CK(cudaMalloc(&S->dEatom, sizeof(float) * T));
  CK(cudaMalloc(&S->dEres, sizeof(float) * T));
  CK(cudaMalloc(&S->dV, sizeof(float4) * T));
  CK(cudaMalloc(&S->dNear, sizeof(int) * T * S->cap));
  CK(cudaMalloc(&S->dNearCount, sizeof(int) * T));
  CK(cudaMalloc(&S->dParams, sizeof(float) * NPARAM));
  CK(cudaMemset(S->dParams, 0, sizeof(float) * NPARAM));
  CK(cudaMalloc(&S->dGrad, sizeof(float) * NPARAM));
  CK(cudaMalloc(&S->dM, sizeof(float) * NPARAM));
  CK(cudaMalloc(&S->dVar, sizeof(float) * NPARAM));
  CK(cudaMemset(S->dM, 0, sizeof(float) * NPARAM));
  CK(cudaMemset(S->dVar, 0, sizeof(float) * NPARAM));
  {
    // two training blocks per SM, shared out by the species' tiles
    std::vector<int3> byType;
    for (int sp = 0; sp < NS; sp++)
      for (const int3& t : S->tiles)
        if (t.z == sp) byType.push_back(t);
    for (const int3& t : S->tiles) S->tiles0 += t.z == 0;
    const int nt = (int)byType.size(), nt1 = nt - S->tiles0, blocks = std::min(2 * 152, nt);
    int b0 = (int)std::lround((double)blocks * S->tiles0 / nt);
    if (S->tiles0 > 0 && b0 < 1) b0 = 1;
    if (nt1 > 0 && b0 > blocks - 1) b0 = std::max(S->tiles0 > 0 ? 1 : 0, blocks - 1);
    S->trainBlocks0 = b0;
    S->trainBlocks = nt1 > 0 ? std::max(blocks, b0 + 1) : b0;
    CK(cudaMalloc(&S->dTrainTiles, sizeof(int3) * nt));
    CK(cudaMemcpy(S->dTrainTiles, byType.data(), sizeof(int3) * nt, cudaMemcpyHostToDevice));
  }
  CK(cudaMalloc(&S->dPart, sizeof(float) * (size_t)S->trainBlocks * PER_SPECIES));
  CK(cudaMalloc(&S->dF, sizeof(double) * 3 * T));
  CK(cudaMalloc(&S->dE, sizeof(double) * chains));
  CK(cudaMalloc(&S->dResPart, sizeof(double) * (2 * SG_RES_BLOCKS + 2)));
  CK(cudaMallocHost(&S->hLoss, sizeof(double) * 2));
  CK(cudaMalloc(&S->dTicket, sizeof(unsigned int)));
  CK(cudaMemset(S->dTicket, 0, sizeof(unsigned int)));
  CK(cudaMalloc(&S->dR0, sizeof(double) * 3 * T));
  CK(cudaFuncSetAttribute(k_sg_mlp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlpSmem)));
  CK(cudaFuncSetAttribute(k_sg_mlp_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc_smem_bytes()));
  CK(cudaFuncSetAttribute(k_sg_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem)));
  return S;
}

void EmDee_surrogate_set_params(void* h, const float* params) {
  Surrogate& S = *(Surrogate*)h;
  CK(cudaMemcpy(S.dParams, params, sizeof(float) * sg::NPARAM, cudaMemcpyHostToDevice));
  CK(cudaMemset(S.dM, 0, sizeof(float) * sg::NPARAM));
  CK(cudaMemset(S.dVar, 0, sizeof(float) * sg::NPARAM));
}

void EmDee_surrogate_get_params(void* h, float* params) {
  Surrogate& S = *(Surrogate*)h;
  CK(cudaMemcpy(params, S.dParams, sizeof(float) * sg::NPARAM, cudaMemcpyDeviceToHost));
}

// lists (if wanted) or, unless they are in place, the FP32 positions; then the descriptors
static void sg_descriptors(Surrogate& S, const double* dR, bool rebuild, bool packed, cudaStream_t st) {
  using namespace sg;
  if (rebuild) sg_build_lists(S, dR, st);
  else if (!packed) k_sg_pack<<<sg_blocks(S.total), 256, 0, st>>>(dR, S.total, S.L, S.dPos);
  launch_chained(k_sg_desc, sg_warp_blocks(S.total), 32 * WARP_ATOMS, 0, st, S.dPos, S.G, S.dSpecies, S.dList, S.dCount,
                 S.cap, S.dG, S.dNear, S.dNearCount);
  CK(cudaGetLastError());
}

static void sg_forces(Surrogate& S, const double* dR, double* dF, double* dE, bool rebuild, bool packed,
                      cudaStream_t st) {
  using namespace sg;
  sg_descriptors(S, dR, rebuild, packed, st);
  sg_network(S, S.dParams, st);
  launch_chained(k_sg_force, sg_warp_blocks(S.total), 32 * WARP_ATOMS, 0, st, S.dPos, S.G, S.dSpecies, S.dNear,
                 S.dNearCount, S.cap, S.dEdG, dF);
  CK(cudaGetLastError());
  if (dE) k_sg_chain_sum<<<S.G.chains, 1024, 0, st>>>(S.dEatom, S.G.N, dE);
}

// Rebuilds the Verlet lists (rebuild != 0) and computes descriptors: dGout (optional, device,
// [chains * N][32] FP32)
void EmDee_surrogate_descriptors(void* h, const double* dR, float* dGout, int rebuild, void* stream) {
  Surrogate& S = *(Surrogate*)h;
  cudaStream_t st = (cudaStream_t)stream;
  sg_descriptors(S, dR, rebuild != 0, false, st);
  if (dGout) CK(cudaMemcpyAsync(dGout, S.dG, sizeof(float) * S.total * sg::DIN, cudaMemcpyDeviceToDevice, st));
}

// Surrogate forces (device FP64 [chains * N][3]) and energies per chain (device FP64 [chains]);
// lists rebuilt when rebuild != 0.  Returns the largest neighbor count seen (list capacity check).
int EmDee_surrogate_forces(void* h, const double* dR, double* dF, double* dE, int rebuild, void* stream) {
  Surrogate& S = *(Surrogate*)h;
  cudaStream_t st = (cudaStream_t)stream;
  sg_forces(S, dR, dF, dE, rebuild != 0, false, st);
  int ov = 0;
  if (rebuild) {
    int flags[2];
    CK(cudaMemcpyAsync(&flags[0], S.dOverflow, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&flags[1], S.dTcError, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    ov = flags[0];
    if (ov > S.cap) fatal("surrogate forces", "a Verlet list outgrew its capacity");
    if (flags[1]) fatal("surrogate forces", "a tensor-core GEMM of the network did not complete");
  }
  return ov;
}

// Per-atom energies, dE/dG (device, FP32) of the last surrogate_forces call
void EmDee_surrogate_atom_outputs(void* h, float* dEatom, float* dEdG, void* stream) {
  Surrogate& S = *(Surrogate*)h;
  cudaStream_t st = (cudaStream_t)stream;
  if (dEatom) CK(cudaMemcpyAsync(dEatom, S.dEatom, sizeof(float) * S.total, cudaMemcpyDeviceToDevice, st));
  if (dEdG) CK(cudaMemcpyAsync(dEdG, S.dEdG, sizeof(float) * S.total * sg::DIN, cudaMemcpyDeviceToDevice, st));
}

// Gradient of the loss  wE sum_c (E_c - Etrue_c)^2 / N^2 / chains + wF sum |F - Ftrue|^2 / (3 N chains)
// for configurations dR (device FP64, chains x N x 3) with reference energies dEtrue (device FP64,
// [chains]) and forces dFtrue (device FP64); lists are rebuilt.  dGrad (device FP32, NPARAM) receives
// the gradient; the loss terms are returned in loss[0] (energy) and loss[1] (force).
void EmDee_surrogate_gradient(void* h, const double* dR, const double* dEtrue, const double* dFtrue, double wE,
                              double wF, float* dGrad, double* loss, void* stream) {
  using namespace sg;
  Surrogate& S = *(Surrogate*)h;
  cudaStream_t st = (cudaStream_t)stream;
  const int C = S.G.chains, N = S.G.N;
  EmDee_surrogate_forces(h, dR, S.dF, S.dE, 1, stream);
  const double fscale = wF * 2.0 / (3.0 * N * C);
  k_sg_residual<<<std::min(SG_RES_BLOCKS, sg_blocks(S.total)), RES_THREADS, 0, st>>>(
      S.dF, dFtrue, S.dE, dEtrue, C, N, wE, fscale, S.dV, S.dEres, S.dResPart, S.dTicket,
      S.dResPart + 2 * SG_RES_BLOCKS, S.hLoss);
  launch_chained(k_sg_udesc, sg_warp_blocks(S.total), 32 * WARP_ATOMS, 0, st, S.dPos, S.G, S.dSpecies, S.dNear, S.dNearCount,
                                                                  S.cap, S.dV, S.dU);
  TileArgs T{S.dAtoms, S.dTrainTiles, (int)S.tiles.size()};
  launch_chained(k_sg_train, S.trainBlocks, 128, sizeof(TrainSmem), st, T, S.tiles0, S.trainBlocks0, S.dParams, S.dG, S.dU,
                                                            S.dEres, S.dPart);
  k_sg_reduce<<<dim3((PER_SPECIES + REDUCE_PARAMS - 1) / REDUCE_PARAMS, NS), REDUCE_PARAMS * REDUCE_SLICES, 0, st>>>(
      S.dPart, S.trainBlocks0, S.trainBlocks, dGrad);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(st));
  loss[0] = wE * S.hLoss[0] / ((double)N * N * C);
  loss[1] = wF * S.hLoss[1] / (3.0 * N * C);
}

// One Adam step on the device master parameters with gradient dGrad (device)
void EmDee_surrogate_adam(void* h, const float* dGrad, double lr, int step, void* stream) {
  Surrogate& S = *(Surrogate*)h;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  sg::k_sg_adam<<<(sg::NPARAM + 255) / 256, 256, 0, (cudaStream_t)stream>>>(S.dParams, dGrad, S.dM, S.dVar, sg::NPARAM,
                                                                            (float)lr, b1, b2, 1e-8f, c1, c2);
  CK(cudaGetLastError());
}

// n velocity-Verlet steps of the chains (device FP64 R, P [chains * N][3]) on the surrogate
// forces; F holds the forces of the current R on entry and on return.  The lists are those of
// the last call that rebuilt them (EmDee_surrogate_forces).  Returns the surrogate energies of the
// final positions in dE (device, [chains]).
void EmDee_surrogate_trajectory(void* h, double* dR, double* dP, double* dF, double* dE, int n, double dt,
                                void* stream) {
  Surrogate& S = *(Surrogate*)h;
  cudaStream_t st = (cudaStream_t)stream;
  const int n3 = 3 * S.total;
  auto advance = [&](void (*kernel)(double*, double*, const double*, int, double, double, double, float*)) {
    launch_chained(kernel, sg_blocks(n3), 256, 0, st, dR, dP, dF, n3, 0.5 * dt, dt, S.L, (float*)S.dPos);
  };
  for (int k = 0; k < n; k++) {
    advance(k == 0 ? sg::k_sg_advance<false, true> : sg::k_sg_advance<true, true>);
    sg_forces(S, dR, dF, k == n - 1 ? dE : nullptr, false, true, st);
  }
  if (n > 0) advance(sg::k_sg_advance<true, false>);
  CK(cudaGetLastError());
}

void EmDee_surrogate_destroy(void* h) {
  Surrogate* S = (Surrogate*)h;
  if (!S) return;
  void* ptrs[] = {S->dSpecies, S->dAtoms, S->dTiles, S->dTiles128, S->dTcError, S->dPos, S->dCellOf, S->dCounts, S->dStarts, S->dCursor,
                  S->dSorted, S->dList, S->dCount, S->dOverflow, S->dG, S->dU, S->dEdG, S->dEatom, S->dEres,
                  S->dV, S->dParams, S->dGrad, S->dM, S->dVar, S->dPart, S->dR0, S->dNear, S->dNearCount, S->dTrainTiles, S->dF, S->dE, S->dResPart,
                  S->dTicket};
  for (void* p : ptrs) cudaFree(p);
  cudaFreeHost(S->hLoss);
  delete S;
}

}  // extern "C"
