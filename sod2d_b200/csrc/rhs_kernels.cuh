// Element kernels of the compressible RHS for sm_100a.
//
// Layout (built once by sod_gpu_init):
//   conn[e][t]        0-based node id of tensor position t = i + n1*j + n1^2*k
//                     (natural 1-D GLL order, xi ascending)
//   geo[e][c][t]      c = 0..8: He(i,j) at c = i + 3j (= d xi_j / d x_i);
//                     c = 9: gpvol
//   slots             per element-node contributions: pass A's in element
//                     order (12 floats), all others at the node-sorted
//                     position slot_pos[e][t]
// A thread owns one Gauss point (= node) of one element, or a line of them
// along zeta (ColCfg: pass A, the Laplacian, the entropy pass); an element's
// nodal fields are staged in shared memory and differentiated with the 1-D
// GLL derivative matrix D[m][n] = l'_n(xi_m) (sum factorisation).  The
// 4x4 / 5x5 contractions are too small for tensor cores; they run on the
// FP32 pipes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef SOD_VEC_XI
#define SOD_VEC_XI 1
#endif
// Pass-B blocks resident per SM: 512 threads per SM, 128 registers each.
#ifndef SOD_RHS_THREADS_PER_SM
#define SOD_RHS_THREADS_PER_SM 512
#endif

namespace sod {

template <int P>
struct Cfg {
  static constexpr int N1 = P + 1;
  static constexpr int N = N1 * N1 * N1;
  static constexpr int NT = ((N + 31) / 32) * 32;  // threads per element
};

struct Phys {
  float gm1;      // gamma - 1
  float gogm1;    // gamma / (gamma - 1)
  float Rgas, Cp, Prt;
  float c_lps, c_rho, c_ener;
  float cp_pr;    // Cp / Pr
  float twoThirds;
};

// Programmatic dependent launch: a kernel started with launch_pdl (ctx.cuh)
// may begin while the kernel before it in the stream still runs.
// pdl_wait() returns when the kernels before are complete and visible (at
// once in an ordinary launch); pdl_trigger() lets a next kernel that was
// started so begin.  Every kernel waits before it triggers, so when one
// begins, all but its immediate predecessor are complete.  Before its wait
// it writes nothing and reads only what that predecessor does not write: the
// mesh, and in the loops of the solves arrays and parameters written before
// the loop (k_cg_update, k_cg_update32, k_cg_patch_z, k_patch_apply_tc).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// An iteration kernel of a solve that has ended (*stop not 0) leaves before
// its first load in every block after the first `wave` ones: those start when
// the kernels before have completed, so the wait costs nothing there, and the
// flag comes from L1.  (The first ones load the mesh before the wait.)  A
// launch after convergence is then mostly its blocks: an iteration of the
// FP32 pressure solve at 48^3 70 -> 17 us (126 while it runs, unchanged), the
// FP64 Jacobi solve at 32^3, whose last batch has a few, 16.2 -> 15.6 ms.
__device__ __forceinline__ bool ended_late(const int *stop, unsigned wave) {
  if (!stop || blockIdx.x < wave) return false;
  pdl_wait();
  return *stop != 0;
}

struct MeshDev {
  int nelem, npoin, npoin_w;
  const int *conn;      // [E][N]
  const float *geo;     // [E][10][N]
  const float *Dnat;    // [N1][N1]
  const float *Drot;    // [2][N1][8]: rows, then columns, of Dnat rotated to start at the
                        // diagonal: D[c][(c+s) % N1], D[(c+s) % N1][c], s = 0..P
  const double *D64;    // Drot in FP64
  const int *lpoin_w;   // 0-based
  const float *invMl;   // [npoin]
  const int *slot_ptr;  // [npoin+1]
  const int *slot_idx;  // [E*N], value e*N+t
  const int *slot_pos;  // [E*N]: node-sorted slot of element node (e, t); inverse of slot_idx
};

// 1-D summation order of the reference ([-1, +1, interior...] as natural
// indices): 0, P, 1, 2, ..., P-1.
template <int P>
__device__ __forceinline__ int ref_order(int s) {
  return s == 0 ? 0 : (s == 1 ? P : s - 1);
}

// Iso-parametric derivatives of a staged field at tensor position (i,j,k).
template <int P>
__device__ __forceinline__ void iso_grad(const float *__restrict__ f, int i, int j, int k,
                                         const float (&Di)[P + 1], const float (&Dj)[P + 1],
                                         const float (&Dk)[P + 1], float &g0, float &g1, float &g2) {
  constexpr int N1 = P + 1;
  g0 = 0.f; g1 = 0.f; g2 = 0.f;
  if constexpr (P == 3 && SOD_VEC_XI) {
    // the xi-line of a 4-node element row is one aligned 16-byte load
    const float4 v = *reinterpret_cast<const float4 *>(f + 4 * j + 16 * k);
    const float fx[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int s = 0; s < N1; ++s) {
      const int m = ref_order<P>(s);
      g0 = fmaf(Di[m], fx[m], g0);
      g1 = fmaf(Dj[m], f[i + N1 * m + N1 * N1 * k], g1);
      g2 = fmaf(Dk[m], f[i + N1 * j + N1 * N1 * m], g2);
    }
  } else {
#pragma unroll
    for (int s = 0; s < N1; ++s) {
      const int m = ref_order<P>(s);
      g0 = fmaf(Di[m], f[m + N1 * j + N1 * N1 * k], g0);
      g1 = fmaf(Dj[m], f[i + N1 * m + N1 * N1 * k], g1);
      g2 = fmaf(Dk[m], f[i + N1 * j + N1 * N1 * m], g2);
    }
  }
}

// Row c of a table of MeshDev::Drot.
template <int P>
__device__ __forceinline__ void load_drot(const float *__restrict__ tab, int c, float (&D)[P + 1]) {
  const float4 v = *reinterpret_cast<const float4 *>(tab + 8 * c);
  D[0] = v.x; D[1] = v.y; D[2] = v.z; D[3] = v.w;
  if (P == 4) D[4] = tab[8 * c + 4];
}

struct NodeQ {  // primitive quantities of one node
  float rho, u0, u1, u2, q0, q1, q2, p, h, T, mu;
};

// Equation of state at one node from the conserved variables, in the
// operation order of updateF (time_integ_ls.f90:574-587) and
// sutherland_viscosity (mod_fluid_viscosity.f90:21-41).
__device__ __forceinline__ void eos(const Phys &ph, float Rgas, float mu_factor, float rho,
                                    float q0, float q1, float q2, float E, NodeQ &s) {
  s.rho = rho; s.q0 = q0; s.q1 = q1; s.q2 = q2;
  s.u0 = q0 / rho; s.u1 = q1 / rho; s.u2 = q2 / rho;
  float umag = s.u0 * s.u0;
  umag = umag + s.u1 * s.u1;
  umag = umag + s.u2 * s.u2;
  const float eint = (E / rho) - 0.5f * umag;
  s.p = rho * ph.gm1 * eint;
  s.h = ph.gogm1 * s.p / rho;
  s.T = s.p / (rho * Rgas);
  s.mu = mu_factor * 1.458e-6f * powf(s.T, 1.5f) / (s.T + 110.4f);
}

// Equation of state of the element kernels: the operations of updateF
// (time_integ_ls.f90:574-587) and sutherland_viscosity
// (mod_fluid_viscosity.f90:21-41) with one reciprocal of rho in place of
// the divisions and T*sqrt(T) for T**1.5 (each within 2 ulp of the
// reference's FP32 value).
__device__ __forceinline__ void eos_fast(const Phys &ph, float invR, float mu_factor, float rho, float q0,
                                         float q1, float q2, float E, NodeQ &s) {
  const float ri = __frcp_rn(rho);
  s.rho = rho; s.q0 = q0; s.q1 = q1; s.q2 = q2;
  s.u0 = q0 * ri; s.u1 = q1 * ri; s.u2 = q2 * ri;
  float umag = s.u0 * s.u0;
  umag = umag + s.u1 * s.u1;
  umag = umag + s.u2 * s.u2;
  const float eint = E * ri - 0.5f * umag;
  s.p = rho * ph.gm1 * eint;
  s.h = ph.gogm1 * s.p * ri;
  s.T = s.p * ri * invR;
  s.mu = mu_factor * 1.458e-6f * (s.T * sqrtf(s.T)) * __frcp_rn(s.T + 110.4f);
}

// Asynchronous global -> shared copies (cp.async): the prefetch of the next
// element group holds no registers while it is in flight.
__device__ __forceinline__ void cp_async4(float *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float *dst, const void *src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Bulk (TMA) copies of contiguous per-element data into shared memory,
// completed on an mbarrier (transaction count).
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// dst (shared) and src (global) 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Shared -> global bulk copy: every writer of the source fences its stores
// (before the barrier that precedes the copy), one thread copies and waits
// until the source has been read.
__device__ __forceinline__ void bulk_s2g_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_s2g(void *dst, const void *src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\ncp.async.bulk.commit_group;\n" ::"l"(dst),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_s2g_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
}
// Bounded wait for the phase `parity` of bar (try_wait itself suspends the
// thread for a while): false after SOD_BULK_WAIT_LIMIT polls.
#ifndef SOD_BULK_WAIT_LIMIT
#define SOD_BULK_WAIT_LIMIT (1 << 24)
#endif
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity) {
  for (int it = 0; it < SOD_BULK_WAIT_LIMIT; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// The derivative matrix as a kernel argument: entries at fixed indices are
// operands from the constant bank.
template <int P, class V>
struct DMat {
  V d[P + 1][P + 1];
};

// Line-per-thread kernels: a thread owns the P + 1 points along zeta over its
// (i, j); 16 lanes (P = 3) or 25 of 32 (P = 4) take an element.
constexpr int COL_WARPS = 2;
template <int P>
struct ColCfg {
  static constexpr int LPE = P == 3 ? 16 : 32, EPW = 32 / LPE, EPB = COL_WARPS * EPW;  // lanes and elements
};
// The q-th node of a line is this many cyclic steps from the own node, own last.
template <int P>
__device__ __forceinline__ int col_step(int q) {
  return q == P ? 0 : (q == P - 1 ? 1 : q + 2);
}
// Matrix rows i and j for col_grad2: rotated at P = 3, natural at P = 4.
template <int P>
__device__ __forceinline__ void col_rows(const MeshDev &m, int i, int j, float (&Di)[P + 1], float (&Dj)[P + 1]) {
  if (P == 3) {
    load_drot<P>(m.Drot, i, Di);
    load_drot<P>(m.Drot, j, Dj);
  } else {
#pragma unroll
    for (int q = 0; q <= P; ++q) { Di[q] = m.Dnat[i * (P + 1) + q]; Dj[q] = m.Dnat[j * (P + 1) + q]; }
  }
}
// xi and eta derivatives at point (i, j, k) of a field staged in tensor
// order, its own value given; summed in the order in which pass B sums the
// gradients that the projections are compared with (their roundings cancel:
// rotated at P = 4, the mass residual's error grew by 5 %).
template <int P>
__device__ __forceinline__ void col_grad2(const float *__restrict__ f, int i, int j, int k, float own,
                                          const float (&Di)[P + 1], const float (&Dj)[P + 1], float &g0, float &g1) {
  constexpr int N1 = P + 1;
  const int r = N1 * N1 * k, c = i + N1 * j + r;
  g0 = g1 = 0.f;
#pragma unroll
  for (int q = 0; q < N1; ++q) {
    if (P == 3) {
      const int s = col_step<P>(q);
      const int ci = c + (i + s < N1 ? s : s - N1), cj = c + (j + s < N1 ? s : s - N1) * N1;
      g0 = fmaf(Di[s], q == P ? own : f[ci], g0);
      g1 = fmaf(Dj[s], q == P ? own : f[cj], g1);
    } else {
      const int mm = ref_order<P>(q);
      g0 = fmaf(Di[mm], f[mm + N1 * j + r], g0);
      g1 = fmaf(Dj[mm], f[i + N1 * mm + r], g1);
    }
  }
}

// ---------------------------------------------------------------------
// Pass A: LPS projections (full_proj_ijk, elem_stab.f90:474-562).  Writes
// gpvol * {tau00, tau01, tau02, tau11, tau12, tau22, grad rho (3), grad T
// (3)} per element node into element-ordered slots of width 12 (bulk copies;
// k_gather_proj reads them through the node->slot CSR).  tau = grad u + grad u^T
// - 2/3 div u I is symmetric (tau_ab and tau_ba are the same FP32 sum), so
// the reference's ProjMX/MY/MZ rows are read back from its 6 entries.
// Input: conserved state (SoA, reference layout) -> EOS in registers, or
// primitive rho/u/T (prim = true).
// ---------------------------------------------------------------------
// A thread owns a line along zeta (ColCfg): the shared and L1 pipe, not HBM,
// bound the one-point-per-thread form (75 % busy at 32^3: 60 staged words and
// 12 matrix words read per point; here 30 and 2).  RHS at 64^3 1.47 -> 1.43 ms.
// 8 to 10 blocks per SM are alike at order 3, 12 spill (1.53 ms).
template <int P, bool PRIM>
__global__ void __launch_bounds__(32 * COL_WARPS, P == 3 ? 10 : 8)
k_proj(MeshDev m, DMat<P, float> D, Phys ph, float Rgas, const float *__restrict__ a0, const float *__restrict__ a1,
       const float *__restrict__ a2, float *__restrict__ slots) {
  using L = ColCfg<P>;
  constexpr int N1 = P + 1, N2 = N1 * N1, N = N1 * N2, NF = 5;
  __shared__ __align__(16) float sm[L::EPB][NF][N];
  __shared__ __align__(16) float ost[L::EPB * N * 12];
  const int el = threadIdx.x / L::LPE, c = threadIdx.x % L::LPE;
  const long long e = (long long)blockIdx.x * L::EPB + el;
  const bool active = e < m.nelem && c < N2;
  const int i = c % N1, j = c / N1;
  const long long NP = m.npoin;
  int n[N1];
  float G[N1][10], Di[N1], Dj[N1];
  if (active) {  // mesh loads first: they depend on no earlier kernel
    const long long b = e * N + c;
#pragma unroll
    for (int k = 0; k < N1; ++k) n[k] = m.conn[b + N2 * k];
    const float *g = m.geo + e * 10 * N + c;
#pragma unroll
    for (int k = 0; k < N1; ++k)
#pragma unroll
      for (int q = 0; q < 10; ++q) G[k][q] = g[q * N + N2 * k];
    col_rows<P>(m, i, j, Di, Dj);
  }
  pdl_wait();
  pdl_trigger();
  float f[NF][N1];  // rho, T, u
  if (active) {
    float in[5][N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) {  // PRIM: a0 = rho, a1 = u(N,3), a2 = Tem; else rho, q(N,3), E
      in[0][k] = a0[n[k]];
      in[1][k] = a1[n[k]];
      in[2][k] = a1[n[k] + NP];
      in[3][k] = a1[n[k] + 2 * NP];
      in[4][k] = a2[n[k]];
    }
    const float invR = __frcp_rn(Rgas);
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      if (PRIM) {
        f[0][k] = in[0][k]; f[1][k] = in[4][k]; f[2][k] = in[1][k]; f[3][k] = in[2][k]; f[4][k] = in[3][k];
      } else {
        NodeQ s;
        eos_fast(ph, invR, 1.f, in[0][k], in[1][k], in[2][k], in[3][k], in[4][k], s);
        f[0][k] = s.rho; f[1][k] = s.T; f[2][k] = s.u0; f[3][k] = s.u1; f[4][k] = s.u2;
      }
#pragma unroll
      for (int q = 0; q < NF; ++q) sm[el][q][c + N2 * k] = f[q][k];
    }
  }
  __syncwarp();
  if (active) {
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      const float *He = G[k];
      const float gv = G[k][9];
      float gr[NF][3];  // physical gradients
#pragma unroll
      for (int q = 0; q < NF; ++q) {
        float g0, g1, g2 = 0.f;
        col_grad2<P>(sm[el][q], i, j, k, f[q][k], Di, Dj, g0, g1);
#pragma unroll
        for (int s = 0; s < N1; ++s) {
          const int mm = ref_order<P>(s);
          g2 = fmaf(D.d[k][mm], f[q][mm], g2);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) gr[q][a] = He[a] * g0 + He[a + 3] * g1 + He[a + 6] * g2;
      }
      const float divU = gr[2][0] + gr[3][1] + gr[4][2];
      float tau[3][3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int b = 0; b < 3; ++b) tau[a][b] = gr[2 + a][b] + gr[2 + b][a];
        tau[a][a] = tau[a][a] - ph.twoThirds * divU;
      }
      float4 *o = reinterpret_cast<float4 *>(ost + (el * N + c + N2 * k) * 12);
      o[0] = make_float4(gv * tau[0][0], gv * tau[0][1], gv * tau[0][2], gv * tau[1][1]);
      o[1] = make_float4(gv * tau[1][2], gv * tau[2][2], gv * gr[0][0], gv * gr[0][1]);
      o[2] = make_float4(gv * gr[0][2], gv * gr[1][0], gv * gr[1][1], gv * gr[1][2]);
    }
  }
  bulk_s2g_fence();
  __syncwarp();
  // the warp's elements leave by one bulk copy (48 N bytes each, a multiple of 16)
  if (threadIdx.x % 32 == 0) {
    const long long left = m.nelem - e;
    if (left > 0) {
      bulk_s2g(slots + e * N * 12, ost + el * N * 12, (unsigned)((left < L::EPW ? left : L::EPW) * N * 48));
      bulk_s2g_wait_read();
    }
  }
}

// ---------------------------------------------------------------------
// Pass B: convection (full_convec_ijk) and/or stabilised diffusion
// (full_diff_stab_ijk) of one element, summed per element node into
// node-sorted slots: a float4 array {mass, energy, mom x, mom y}, then a
// float array mom z.
//
// MODE_CONV: convective residual * fact_c.
// MODE_DIFF: LPS-stabilised diffusion * fact_d (full_diff_stab_ijk);
//   with MODE_NOLPS the plain diffusion of full_diffusion_ijk
//   (elem_diffu.f90:12-223).
// Input kinds:
//   IN_CONS : rho, q(N,3), E (conserved; EOS fused, h = E:=aux_h)
//   IN_PRIM : convection inputs u, q, rho, pr, E given directly
//   IN_DIFF : diffusion inputs rho, u, Tem, mu_fluid given directly
// ---------------------------------------------------------------------
enum { MODE_CONV = 1, MODE_DIFF = 2, MODE_NOLPS = 4 };
enum { IN_CONS = 0, IN_PRIM = 1, IN_DIFF = 2 };

struct RhsArgs {
  // conserved / primitive inputs (reference layout)
  const float *rho, *q, *E, *u, *pr, *Tem, *mu_fluid;
  float mu_factor;
  // diffusion inputs
  const float *mue_t;     // [nelem][N] tensor order (internal copy of mu_e)
  const float *musgs_t;   // [nelem][N] or null
  const float *tau_stab;  // (nelem)
  const float *rho_n;     // IN_DIFF: density of the nu_e and mu_sgs terms when it differs
                          // from rho (full_diffusion_ijk's rho_n); null: rho
  const float *proj12;    // [npoin][12] mass-inverted projections (internal):
                          // tau00 tau01 tau02 tau11 tau12 tau22 gradRho(3) gradT(3)
  float fact_c, fact_d;
  const int *stop;  // non-zero: return at once (an iteration that has ended); null: run
  int *err;  // mapped host flag: set when a bulk-copy wait of pass B gave up
};

// Staged fields of pass B, one entry per element node:
//   CONV+DIFF (conserved inputs): float4 (u0,u1,u2,H) and (rho,T,p,0)
//   CONV only : float2 pairs (u0,u1) (u2,rho) (q0,q1) (q2,p) (H,rho*H)
//   DIFF only : float2 pairs (u0,u1) (u2,rho), then T
// With the conserved inputs q = rho u, so every split-form term is a product
// of staged values and one product per line node serves momentum, mass and
// energy (FLUX2 below).  Instruction issue bounds this kernel: that form
// issues 829 instructions per Gauss point where 18 product fields, formed
// from each line node and differentiated one by one, took 1251 (k_rhs at
// 32^3 117.6 -> 102.1 us; RHS at 64^3 1.72 -> 1.55 ms), with the same error
// against FP64.
// With convection inputs u, q, rho, p, E given independently, the 18 product
// fields -- q_a u_b and u_a u_b (a <= b), rho*H*u_c and H*u_c -- are formed
// in registers from the staged values of each line node as it is read.
enum { PB_U01 = 0, PB_U2R = 1, PB_Q01 = 2, PB_Q2P = 3, PB_HRH = 4 };

// Shared-memory plan of k_rhs.  Two prefetch stages (the element group being
// computed and the next one), each holding, per thread of the block: the
// nodal inputs (NIN values gathered through the connectivity), J^-1 and
// gpvol (10), the node-sorted slot position, mu_e and mu_sgs, and the 12
// mass-inverted projections of the node; then the staging area of the
// element kernels (the paired fields, later the contravariant fluxes).
template <int P, int EPB, int MODE, int IN>
struct RhsPlan {
  static constexpr int N1 = P + 1, N = Cfg<P>::N, NT = Cfg<P>::NT, NTB = EPB * NT;
  static constexpr bool CONV = (MODE & MODE_CONV) != 0;
  static constexpr bool DIFF = (MODE & MODE_DIFF) != 0;
  static constexpr bool LPS = (MODE & MODE_NOLPS) == 0;
  static constexpr int NC = LPS ? 5 : 6;  // staged contravariant flux fields of the weak divergence
  // conserved inputs (q = rho u): two float4 per node, otherwise pairs
  static constexpr bool FLUX2 = CONV && IN == IN_CONS;
  static constexpr int NPAIR = FLUX2 ? 4 : (CONV ? 5 : 3);
  static constexpr int PB_T = 2;
  // IN_CONS: rho q0 q1 q2 E | IN_PRIM: rho u0 u1 u2 q0 q1 q2 p h | IN_DIFF: rho rho_n u0 u1 u2 T mu
  static constexpr int NIN = IN == IN_CONS ? 5 : (IN == IN_PRIM ? 9 : 7);
  static constexpr int O_IN = 0, O_GEO = NIN * NTB, O_POS = O_GEO + 10 * NTB, O_MUE = O_POS + NTB,
                       O_MUS = O_MUE + (DIFF ? NTB : 0), O_PROJ = O_MUS + (DIFF ? NTB : 0);
  static constexpr int STAGE = O_PROJ + (DIFF && LPS ? 12 * NTB : 0);  // floats (multiple of 4)
  static constexpr int SMF = (2 * NPAIR > 3 * NC) ? 2 * NPAIR : 3 * NC;  // staging floats per element node
  static constexpr int O_STG = 2 * STAGE;
  static constexpr size_t BYTES = (size_t)(2 * STAGE + EPB * SMF * N) * sizeof(float);
};


// Persistent element kernel of pass B: a block walks element groups
// blockIdx.x, blockIdx.x + gridDim.x, ... and, while it computes one group,
// its cp.async copies bring the next group's inputs into the other stage.
template <int P, int EPB, int MODE, int IN>
__global__ void __launch_bounds__(EPB *Cfg<P>::NT, SOD_RHS_THREADS_PER_SM / (EPB * Cfg<P>::NT))
k_rhs(MeshDev m, Phys ph, float Rgas, RhsArgs A, float *__restrict__ slots) {
  using L = RhsPlan<P, EPB, MODE, IN>;
  constexpr int N1 = L::N1, N = L::N, NT = L::NT, NTB = L::NTB, NC = L::NC, SMF = L::SMF, PB_T = L::PB_T;
  constexpr bool CONV = L::CONV, DIFF = L::DIFF, LPS = L::LPS, FLUX2 = L::FLUX2, ROT = P == 3 && (DIFF || FLUX2);
  static_assert(FLUX2 || !(CONV && DIFF), "convection with diffusion runs on the conserved state");
  extern __shared__ __align__(16) float dsm[];
  const int tid = threadIdx.x, el = tid / NT, t = tid % NT;
  const int i = t % N1, j = (t / N1) % N1, k = t / (N1 * N1);
  const long long NP = m.npoin;
  const long long ngroups = ((long long)m.nelem + EPB - 1) / EPB, G = gridDim.x;
  float *const sf = dsm + L::O_STG + el * SMF * N;
  float2 *const sp = reinterpret_cast<float2 *>(sf);
  float4 *const sq = reinterpret_cast<float4 *>(sf);
  const float invR = __frcp_rn(Rgas);
  // P = 3, one element per block: the element's J^-1 and gpvol (2560 B),
  // slot positions and mu_e (256 B each) are contiguous and 16-byte aligned
  // in global memory, and land with the stage's layout (stride N = NTB), so
  // one thread moves them with bulk copies; the gathered state and
  // projections stay per-thread cp.async.
  constexpr bool BULK = (P == 3 && EPB == 1);
  __shared__ __align__(8) unsigned long long mbar[2];
  unsigned phases = 0u;  // bit b: parity of the next completion of mbar[b]
  if (BULK && tid == 0) {
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (BULK) __syncthreads();

  // ROT (P = 3): a line is summed in cyclic steps 2, 3, 1 from the thread's
  // own node, which comes last, from registers: three shared loads per line
  // instead of four, in a kernel whose shared-memory pipe is 71 % busy
  // (wavefronts 17.1 -> 15.3 M at 32^3; k_rhs 102.1 -> 94.3 us, RHS at 64^3
  // 1.575 -> 1.515 ms).  Of the 24 orders this one rounds least on constant
  // and smooth fields (0.75 of the error of the order -1, +1, interior) and
  // the same on random ones.  At P = 4 the rotated rows of 5 conflict in
  // shared memory (136.4 against 133.5 us at 23x19x17): node ref_order(q).
  auto line_step = [](int q) -> int { return q == 0 ? 2 : (q == 1 ? 3 : (q == 2 ? 1 : 0)); };
  auto line_node = [&](int d, int q) -> int {
    const int cd = d == 0 ? i : (d == 1 ? j : k), stride = d == 0 ? 1 : (d == 1 ? N1 : N1 * N1);
    if (ROT) {
      const int s = line_step(q);
      return t + (cd + s < N1 ? s : s - N1) * stride;
    }
    return t + (ref_order<P>(q) - cd) * stride;
  };
  auto line_coef = [&](const float (&D)[N1], int q) -> float { return D[ROT ? line_step(q) : ref_order<P>(q)]; };
  auto load_row = [&](int c, bool col, float (&D)[N1]) {
    if (ROT) {
      load_drot<P>(m.Drot + (col ? 8 * N1 : 0), c, D);
    } else {
#pragma unroll
      for (int q = 0; q < N1; ++q) D[q] = col ? m.Dnat[q * N1 + c] : m.Dnat[c * N1 + q];
    }
  };
  auto node_of = [&](long long g) -> int {
    const long long e = g * EPB + el;
    return (g < ngroups && e < m.nelem && t < N) ? m.conn[e * N + t] : -1;
  };
  // this thread's copies for group g into stage stg (nd: its node, -1: none)
  auto issue = [&](float *stg, long long g, int nd) {
    if (BULK && tid == 0 && g < ngroups) {
      const long long e0 = g;  // one element per block
      unsigned long long *bar = &mbar[stg == dsm ? 0 : 1];
      const bool mus = DIFF && A.musgs_t;
      const unsigned bytes = (10u + 1u + (DIFF ? 1u : 0u) + (mus ? 1u : 0u)) * N * 4u;
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // earlier reads of this stage first
      mbar_expect_tx(bar, bytes);
      bulk_g2s(stg + L::O_GEO, m.geo + e0 * 10 * N, 10u * N * 4u, bar);
      bulk_g2s(stg + L::O_POS, m.slot_pos + e0 * N, N * 4u, bar);
      if (DIFF) bulk_g2s(stg + L::O_MUE, A.mue_t + e0 * N, N * 4u, bar);
      if (mus) bulk_g2s(stg + L::O_MUS, A.musgs_t + e0 * N, N * 4u, bar);
    }
    if (nd < 0) return;
    const long long e = g * EPB + el;
    if (IN == IN_CONS) {
      cp_async4(stg + L::O_IN + 0 * NTB + tid, A.rho + nd);
      cp_async4(stg + L::O_IN + 1 * NTB + tid, A.q + nd);
      cp_async4(stg + L::O_IN + 2 * NTB + tid, A.q + nd + NP);
      cp_async4(stg + L::O_IN + 3 * NTB + tid, A.q + nd + 2 * NP);
      cp_async4(stg + L::O_IN + 4 * NTB + tid, A.E + nd);
    } else if (IN == IN_PRIM) {
      cp_async4(stg + L::O_IN + 0 * NTB + tid, A.rho + nd);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        cp_async4(stg + L::O_IN + (1 + c) * NTB + tid, A.u + nd + c * NP);
        cp_async4(stg + L::O_IN + (4 + c) * NTB + tid, A.q + nd + c * NP);
      }
      cp_async4(stg + L::O_IN + 7 * NTB + tid, A.pr + nd);
      cp_async4(stg + L::O_IN + 8 * NTB + tid, A.E + nd);
    } else {
      cp_async4(stg + L::O_IN + 0 * NTB + tid, A.rho + nd);
      cp_async4(stg + L::O_IN + 1 * NTB + tid, (A.rho_n ? A.rho_n : A.rho) + nd);
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async4(stg + L::O_IN + (2 + c) * NTB + tid, A.u + nd + c * NP);
      cp_async4(stg + L::O_IN + 5 * NTB + tid, A.Tem + nd);
      cp_async4(stg + L::O_IN + 6 * NTB + tid, A.mu_fluid + nd);
    }
    if (!BULK) {
      const float *g0 = m.geo + e * 10 * N + t;
#pragma unroll
      for (int c = 0; c < 10; ++c) cp_async4(stg + L::O_GEO + c * NTB + tid, g0 + c * N);
      cp_async4(stg + L::O_POS + tid, m.slot_pos + e * N + t);
    }
    if (DIFF) {
      if (!BULK) {
        cp_async4(stg + L::O_MUE + tid, A.mue_t + e * N + t);
        if (A.musgs_t) cp_async4(stg + L::O_MUS + tid, A.musgs_t + e * N + t);
      }
      if (LPS) {
#pragma unroll
        for (int c = 0; c < 3; ++c) cp_async16(stg + L::O_PROJ + tid * 12 + 4 * c, A.proj12 + (long long)nd * 12 + 4 * c);
      }
    }
  };

  long long g = blockIdx.x;
  const int nd_first = node_of(g);
  int nd_next = node_of(g + G);
  pdl_wait();
  pdl_trigger();
  if (A.stop && *A.stop) return;
  issue(dsm, g, nd_first);
  cp_async_commit();
  for (int buf = 0; g < ngroups; g += G, buf ^= 1) {
    const float *cur = dsm + buf * L::STAGE;
    float *nxt = dsm + (buf ^ 1) * L::STAGE;
    cp_async_wait_all();  // this thread's copies of the current group have landed
    bool bulk_ok = true;
    if (BULK) {  // and the block's bulk copies of it
      bulk_ok = mbar_wait(&mbar[buf], (phases >> buf) & 1u);
      phases ^= 1u << buf;
    }
    const long long e = g * EPB + el;
    const bool active = (e < m.nelem) && (t < N);
    const float *gm = cur + L::O_GEO + tid;  // J^-1 (9 components) and gpvol, stride NTB
    NodeQ s;
    float mu = 0.f, rhon_in = 0.f, H = 0.f, rH = 0.f;
    if (active) {
      const float *in = cur + L::O_IN + tid;
      if (IN == IN_CONS && DIFF) {
        eos_fast(ph, invR, A.mu_factor, in[0], in[NTB], in[2 * NTB], in[3 * NTB], in[4 * NTB], s);
        mu = s.mu;
        const float ri = __frcp_rn(s.rho);
        // u = q / rho to half an ulp: rho u stands for q below
        s.u0 = fmaf(fmaf(-s.rho, s.u0, s.q0), ri, s.u0);
        s.u1 = fmaf(fmaf(-s.rho, s.u1, s.q1), ri, s.u1);
        s.u2 = fmaf(fmaf(-s.rho, s.u2, s.q2), ri, s.u2);
      } else if (IN == IN_CONS) {
        // convection alone (the IMEX stages): u, p and h by the divisions of
        // k_eos_end and k_aux_h.  eos_fast here raised the momentum's error
        // at Ma = 0.1, order 4, by 2 %; the step takes as long (2.23 ms at 32^3).
        eos(ph, Rgas, A.mu_factor, in[0], in[NTB], in[2 * NTB], in[3 * NTB], in[4 * NTB], s);
        s.T = 0.f;
      } else if (IN == IN_PRIM) {
        s.rho = in[0];
        s.u0 = in[NTB]; s.u1 = in[2 * NTB]; s.u2 = in[3 * NTB];
        s.q0 = in[4 * NTB]; s.q1 = in[5 * NTB]; s.q2 = in[6 * NTB];
        s.p = in[7 * NTB]; s.h = in[8 * NTB]; s.T = 0.f;
      } else {
        s.rho = in[0];
        rhon_in = in[NTB];
        s.u0 = in[2 * NTB]; s.u1 = in[3 * NTB]; s.u2 = in[4 * NTB];
        s.T = in[5 * NTB];
        mu = in[6 * NTB];
        s.q0 = s.q1 = s.q2 = 0.f; s.p = 0.f; s.h = 0.f;
      }
      if (CONV) {
        // H = h + k with k = |u|^2/2: the reference's split-form energy
        // terms for E:=h and for k enter with the same 1/4 weight, so their
        // flux fields are combined (rho*h*u + rho*k*u = rho*H*u, h*u + k*u = H*u).
        float kk = s.u0 * s.u0 * 0.5f;
        kk = kk + s.u1 * s.u1 * 0.5f;
        kk = kk + s.u2 * s.u2 * 0.5f;
        H = s.h + kk;
        rH = s.rho * H;
      }
      if (FLUX2) {
        sq[t] = make_float4(s.u0, s.u1, s.u2, H);
        sq[N + t] = make_float4(s.rho, s.T, s.p, 0.f);
      } else {
        sp[PB_U01 * N + t] = make_float2(s.u0, s.u1);
        sp[PB_U2R * N + t] = make_float2(s.u2, s.rho);
        if (CONV) {
          sp[PB_Q01 * N + t] = make_float2(s.q0, s.q1);
          sp[PB_Q2P * N + t] = make_float2(s.q2, s.p);
          sp[PB_HRH * N + t] = make_float2(H, rH);
        }
        if (DIFF) sf[2 * PB_T * N + t] = s.T;
      }
    }
    // staged pairs visible; every thread is done with the other stage
    if (!__syncthreads_and(bulk_ok)) {
      if (tid == 0) *(volatile int *)A.err = 1;  // a bulk copy never completed: stop, nothing else is in flight
      return;
    }
    if (g + G < ngroups) issue(nxt, g + G, nd_next);
    cp_async_commit();
    nd_next = node_of(g + 2 * G);  // consumed one group later

    float res[5] = {0.f, 0.f, 0.f, 0.f, 0.f};  // mass, energy, mom x,y,z
    float gradRho[3] = {0.f, 0.f, 0.f}, gradT[3] = {0.f, 0.f, 0.f};
    float gradU[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    if (FLUX2 && active) {
      // Split form with one product per line node.  With q = rho u and
      // U = u . He(:,d) (He of the output point), direction d contributes
      //   f S_d + sum_m D(m) w_m f_m + rho U sum_m D(m) f_m,
      //   w_m = rho_m U_m + rho_m U + rho U_m,  S_d = sum_m D(m) w_m
      // to 4 times the terms of f = u_a (momentum) and f = H (energy), and
      // S_d to twice the mass term; S = div q + rho div u + u . grad rho.
      const float2 z2 = make_float2(0.f, 0.f);
      float2 c01 = z2, c2H = z2;  // momentum x, y; momentum z, energy
      float divQ = 0.f, ugR = 0.f, gradP[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        float Dd[N1];
        load_row(d == 0 ? i : (d == 1 ? j : k), false, Dd);
        const float h[3] = {gm[(0 + 3 * d) * NTB], gm[(1 + 3 * d) * NTB], gm[(2 + 3 * d) * NTB]};
        const float Ud = h[0] * s.u0 + h[1] * s.u1 + h[2] * s.u2;
        float2 aU01 = z2, aU2H = z2, aRT = z2, d01 = z2, d2H = z2;
        float aP = 0.f, aQ = 0.f;
#pragma unroll
        for (int mm = 0; mm < N1; ++mm) {
          const bool own = ROT && mm == P;  // the node itself comes from its registers
          const float Dm = line_coef(Dd, mm);
          const float4 a = own ? make_float4(s.u0, s.u1, s.u2, H) : sq[line_node(d, mm)];
          const float4 b = own ? make_float4(s.rho, s.T, s.p, 0.f) : sq[N + line_node(d, mm)];
          const float2 a01 = make_float2(a.x, a.y), a2H = make_float2(a.z, a.w);
          const float2 D2 = make_float2(Dm, Dm);
          const float Um = fmaf(h[0], a.x, fmaf(h[1], a.y, h[2] * a.z)), q = b.x * Um;
          const float c = Dm * fmaf(s.rho, Um, fmaf(b.x, Ud, q));
          const float2 c2 = make_float2(c, c);
          aQ = fmaf(Dm, q, aQ);
          d01 = __ffma2_rn(c2, a01, d01);
          d2H = __ffma2_rn(c2, a2H, d2H);
          aU01 = __ffma2_rn(D2, a01, aU01);
          aU2H = __ffma2_rn(D2, a2H, aU2H);
          aRT = __ffma2_rn(D2, make_float2(b.x, b.y), aRT);
          aP = fmaf(Dm, b.z, aP);
        }
        const float2 Qd2 = make_float2(s.rho * Ud, s.rho * Ud);
        c01 = __fadd2_rn(c01, __ffma2_rn(Qd2, aU01, d01));
        c2H = __fadd2_rn(c2H, __ffma2_rn(Qd2, aU2H, d2H));
        divQ = divQ + aQ;
        ugR = ugR + Ud * aRT.x;
        const float dU[3] = {aU01.x, aU01.y, aU2H.x};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          gradRho[a] = gradRho[a] + h[a] * aRT.x;
          if (DIFF) gradT[a] = gradT[a] + h[a] * aRT.y;
          gradP[a] = gradP[a] + h[a] * aP;
#pragma unroll
          for (int b = 0; b < 3; ++b) gradU[a][b] = gradU[a][b] + h[b] * dU[a];
        }
      }
      const float gc = A.fact_c * gm[9 * NTB];
      const float S = divQ + s.rho * (gradU[0][0] + gradU[1][1] + gradU[2][2]) + ugR;
      res[0] = gc * (0.5f * S);
      res[1] = gc * (0.25f * (c2H.y + H * S));
      res[2] = gc * (0.25f * (c01.x + s.u0 * S) + gradP[0]);
      res[3] = gc * (0.25f * (c01.y + s.u1 * S) + gradP[1]);
      res[4] = gc * (0.25f * (c2H.x + s.u2 * S) + gradP[2]);
    }
    if (!FLUX2 && active) {
      // Physical-space sums, accumulated one reference direction d at a
      // time: d_a f = sum_d He(a,d) d_d f, and every convective term is
      // linear in the derivatives, so each direction's derivatives are
      // folded in as soon as they are formed.  Advective terms use the
      // contravariant velocities U_d = sum_b u_b He(b,d), Q_d = sum_b q_b He(b,d).
      float divQ = 0.f, QdH = 0.f, UdRH = 0.f, divRHu = 0.f, divHu = 0.f;
      float UdQ[3] = {0.f, 0.f, 0.f}, gradP[3] = {0.f, 0.f, 0.f}, divF[3] = {0.f, 0.f, 0.f},
            divG[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        float Dd[N1];
        load_row(d == 0 ? i : (d == 1 ? j : k), false, Dd);
        const float2 z2 = make_float2(0.f, 0.f);
        float2 aU01 = z2, aU2R = z2, aQ01 = z2, aQ2P = z2, aHRH = z2;
        float aT = 0.f;
        float2 aF0 = z2, aF1 = z2, aF2 = z2, aG0 = z2, aG1 = z2, aG2 = z2, aR0 = z2, aR1 = z2, aR2 = z2;
#pragma unroll
        for (int mm = 0; mm < N1; ++mm) {
          const bool own = ROT && mm == P;  // the node itself comes from its registers
          const float Dm = line_coef(Dd, mm);
          const float2 D2 = make_float2(Dm, Dm);
          const int tm = own ? t : line_node(d, mm);
          const float2 u01 = own ? make_float2(s.u0, s.u1) : sp[PB_U01 * N + tm];
          const float2 u2r = own ? make_float2(s.u2, s.rho) : sp[PB_U2R * N + tm];
          aU01 = __ffma2_rn(D2, u01, aU01);
          aU2R = __ffma2_rn(D2, u2r, aU2R);
          if (DIFF) aT = fmaf(Dm, own ? s.T : sf[2 * PB_T * N + tm], aT);
          if (CONV) {
            const float2 q01 = own ? make_float2(s.q0, s.q1) : sp[PB_Q01 * N + tm];
            const float2 q2p = own ? make_float2(s.q2, s.p) : sp[PB_Q2P * N + tm];
            const float2 hrh = own ? make_float2(H, rH) : sp[PB_HRH * N + tm];
            aQ01 = __ffma2_rn(D2, q01, aQ01);
            aQ2P = __ffma2_rn(D2, q2p, aQ2P);
            aHRH = __ffma2_rn(D2, hrh, aHRH);
            const float u0 = u01.x, u1 = u01.y, u2 = u2r.x, q0 = q01.x, q1 = q01.y, q2 = q2p.x;
            aF0 = __ffma2_rn(D2, make_float2(q0 * u0, q0 * u1), aF0);
            aF1 = __ffma2_rn(D2, make_float2(q0 * u2, q1 * u1), aF1);
            aF2 = __ffma2_rn(D2, make_float2(q1 * u2, q2 * u2), aF2);
            aG0 = __ffma2_rn(D2, make_float2(u0 * u0, u0 * u1), aG0);
            aG1 = __ffma2_rn(D2, make_float2(u0 * u2, u1 * u1), aG1);
            aG2 = __ffma2_rn(D2, make_float2(u1 * u2, u2 * u2), aG2);
            aR0 = __ffma2_rn(D2, make_float2(hrh.y * u0, hrh.y * u1), aR0);
            aR1 = __ffma2_rn(D2, make_float2(hrh.y * u2, hrh.x * u2), aR1);
            aR2 = __ffma2_rn(D2, make_float2(hrh.x * u0, hrh.x * u1), aR2);
          }
        }
        const float h[3] = {gm[(0 + 3 * d) * NTB], gm[(1 + 3 * d) * NTB], gm[(2 + 3 * d) * NTB]};
        const float dU[3] = {aU01.x, aU01.y, aU2R.x};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          gradRho[a] = gradRho[a] + h[a] * aU2R.y;
          if (DIFF) gradT[a] = gradT[a] + h[a] * aT;
#pragma unroll
          for (int b = 0; b < 3; ++b) gradU[a][b] = gradU[a][b] + h[b] * dU[a];
        }
        if (CONV) {
          const float dQ[3] = {aQ01.x, aQ01.y, aQ2P.x};
          // d_d of the symmetric F_ab = q_a u_b and G_ab = u_a u_b (a <= b)
          const float dF[3][3] = {{aF0.x, aF0.y, aF1.x}, {aF0.y, aF1.y, aF2.x}, {aF1.x, aF2.x, aF2.y}};
          const float dG[3][3] = {{aG0.x, aG0.y, aG1.x}, {aG0.y, aG1.y, aG2.x}, {aG1.x, aG2.x, aG2.y}};
          const float dRHu[3] = {aR0.x, aR0.y, aR1.x}, dHu[3] = {aR2.x, aR2.y, aR1.y};
          const float Ud = h[0] * s.u0 + h[1] * s.u1 + h[2] * s.u2;
          const float Qd = h[0] * s.q0 + h[1] * s.q1 + h[2] * s.q2;
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            divQ = divQ + h[a] * dQ[a];
            UdQ[a] = UdQ[a] + Ud * dQ[a];
            gradP[a] = gradP[a] + h[a] * aQ2P.y;
            divRHu = divRHu + h[a] * dRHu[a];
            divHu = divHu + h[a] * dHu[a];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
              divF[a] = divF[a] + h[b] * dF[a][b];
              divG[a] = divG[a] + h[b] * dG[a][b];
            }
          }
          QdH = QdH + Qd * aHRH.x;
          UdRH = UdRH + Ud * aHRH.y;
        }
      }
      if (CONV) {
        const float gv = gm[9 * NTB];
        const float u[3] = {s.u0, s.u1, s.u2}, q[3] = {s.q0, s.q1, s.q2};
        const float divU = gradU[0][0] + gradU[1][1] + gradU[2][2];
        float ugR = 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) ugR = ugR + u[a] * gradRho[a];
        const float Rmass = 0.5f * (divQ + s.rho * divU) + 0.5f * ugR;
        const float Rener =
            0.25f * (divRHu + H * divQ + rH * divU + s.rho * divHu) + 0.25f * (QdH + UdRH + H * ugR);
        res[0] = A.fact_c * (gv * Rmass);
        res[1] = A.fact_c * (gv * Rener);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          float QdU = 0.f;
#pragma unroll
          for (int b = 0; b < 3; ++b) QdU = QdU + q[b] * gradU[a][b];
          const float Rmom = 0.25f * (divF[a] + u[a] * divQ + q[a] * divU + s.rho * divG[a]) + gradP[a] +
                             0.25f * (u[a] * ugR + QdU + UdQ[a]);
          res[2 + a] = A.fact_c * (gv * Rmom);
        }
      }
    }

    if (DIFF) {
      // Fluxes at this Gauss point (first Gauss-point loop of
      // full_diff_stab_ijk, elem_stab.f90:296-385, or of full_diffusion_ijk,
      // elem_diffu.f90:99-164), then their contravariant components
      // gpvol * sum_i He(i,d) F_i, staged for the weak divergence.
      float C[NC][3];
      float nu_e = 0.f, kappa_e = 0.f;
      if (active) {
        const float mue = cur[L::O_MUE + tid];
        const float musgs = A.musgs_t ? cur[L::O_MUS + tid] : 0.f;
        const float rhon = IN == IN_DIFF ? rhon_in : s.rho;
        nu_e = ph.c_rho * mue * __frcp_rn(rhon);
        const float mu_fgp = mu + rhon * musgs;
        const float mu_egp = mue;
        kappa_e = mu * ph.cp_pr + ph.c_ener * mue * ph.cp_pr + ph.Cp * rhon * musgs * (1.f / 0.9f);
        const float divU = gradU[0][0] + gradU[1][1] + gradU[2][2];
        const float u[3] = {s.u0, s.u1, s.u2};
        float tau[3][3];
        float Fx[3], Fy[3], Fz[3], FT[3], FR[3];
        if (LPS) {
          const float ts = A.tau_stab[e];
#pragma unroll
          for (int a = 0; a < 3; ++a) {
#pragma unroll
            for (int b = 0; b < 3; ++b) tau[a][b] = gradU[a][b] + gradU[b][a];
            tau[a][a] = tau[a][a] - ph.twoThirds * divU;
          }
          const float4 *pj = reinterpret_cast<const float4 *>(cur + L::O_PROJ + tid * 12);
          const float4 p0 = pj[0], p1 = pj[1], p2 = pj[2];
          const float PX[3] = {p0.x, p0.y, p0.z}, PY[3] = {p0.y, p0.w, p1.x}, PZ[3] = {p0.z, p1.x, p1.y};
          const float PM[3] = {p1.z, p1.w, p2.x}, PE[3] = {p2.y, p2.z, p2.w};
          const float cl = -ph.c_lps * ts;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            Fx[d] = cl * (PX[d] - tau[0][d]) * rhon;
            Fy[d] = cl * (PY[d] - tau[1][d]) * rhon;
            Fz[d] = cl * (PZ[d] - tau[2][d]) * rhon;
            FT[d] = cl * (PE[d] - gradT[d]) * rhon * ph.cp_pr;
            FR[d] = cl * (PM[d] - gradRho[d]);
          }
        }
        float tauU[3] = {0.f, 0.f, 0.f};
        const float mt = mu_fgp + mu_egp;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            tauU[a] = tauU[a] + mt * (gradU[a][b] + gradU[b][a]) * u[b];
            tau[a][b] = mt * (gradU[a][b] + gradU[b][a]);
          }
          tauU[a] = tauU[a] - (mu_fgp)*ph.twoThirds * divU * u[a];
          tau[a][a] = tau[a][a] - (mu_fgp)*ph.twoThirds * divU;
        }
        if (LPS) {
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            Fx[d] = Fx[d] + tau[0][d];
            Fy[d] = Fy[d] + tau[1][d];
            Fz[d] = Fz[d] + tau[2][d];
            FT[d] = FT[d] + kappa_e * gradT[d] + tauU[d];
            FR[d] = FR[d] + nu_e * gradRho[d];
          }
        } else {
          // full_diffusion_ijk scales the neighbours' grad rho and grad T by
          // nu_e and kappa_e of the output Gauss point: stage them unscaled.
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            Fx[d] = tau[0][d];
            Fy[d] = tau[1][d];
            Fz[d] = tau[2][d];
            FT[d] = tauU[d];
            FR[d] = gradRho[d];
          }
        }
        const float gv = gm[9 * NTB];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float h0 = gm[(0 + 3 * d) * NTB], h1 = gm[(1 + 3 * d) * NTB], h2 = gm[(2 + 3 * d) * NTB];
          C[0][d] = gv * (h0 * FR[0] + h1 * FR[1] + h2 * FR[2]);
          C[1][d] = gv * (h0 * FT[0] + h1 * FT[1] + h2 * FT[2]);
          C[2][d] = gv * (h0 * Fx[0] + h1 * Fx[1] + h2 * Fx[2]);
          C[3][d] = gv * (h0 * Fy[0] + h1 * Fy[1] + h2 * Fy[2]);
          C[4][d] = gv * (h0 * Fz[0] + h1 * Fz[1] + h2 * Fz[2]);
          if (!LPS) C[NC - 1][d] = gv * (h0 * gradT[0] + h1 * gradT[1] + h2 * gradT[2]);
        }
      }
      __syncthreads();  // all reads of the staged pairs are done
      if (active) {
#pragma unroll
        for (int q = 0; q < NC; ++q)
#pragma unroll
          for (int d = 0; d < 3; ++d) sf[(q * 3 + d) * N + t] = C[q][d];
      }
      __syncthreads();
      if (active) {
        // Weak divergence: sum_d sum_m D[m][i_d] C_d(node with d-index m).
        float Dc[3][N1];
        load_row(i, true, Dc[0]);
        load_row(j, true, Dc[1]);
        load_row(k, true, Dc[2]);
        float wd[NC];
#pragma unroll
        for (int q = 0; q < NC; ++q) {
          float acc = 0.f;
#pragma unroll
          for (int mm = 0; mm < N1; ++mm)
#pragma unroll
            for (int d = 0; d < 3; ++d)
              acc = fmaf(line_coef(Dc[d], mm), ROT && mm == P ? C[q][d] : sf[(q * 3 + d) * N + line_node(d, mm)], acc);
          wd[q] = acc;
        }
        if (LPS) {
#pragma unroll
          for (int q = 0; q < 5; ++q) res[q] = res[q] + A.fact_d * wd[q];
        } else {
          res[0] = res[0] + A.fact_d * (nu_e * wd[0]);
          res[1] = res[1] + A.fact_d * (wd[1] + kappa_e * wd[NC - 1]);
#pragma unroll
          for (int q = 2; q < 5; ++q) res[q] = res[q] + A.fact_d * wd[q];
        }
      }
    }
    if (active) {
      // pass-B slots, node-sorted: [E*N] float4 (mass, energy, mom x, mom y),
      // then [E*N] mom z
      const long long sp5 = __float_as_int(cur[L::O_POS + tid]);
      reinterpret_cast<float4 *>(slots)[sp5] = make_float4(res[0], res[1], res[2], res[3]);
      slots[(long long)m.nelem * N * 4 + sp5] = res[4];
    }
    __syncthreads();  // the staging area is free for the next group
  }
  cp_async_wait_all();
}

// ---------------------------------------------------------------------
// Node-centric assembly of pass A: the 12 projections of a node are invMl
// times the Kahan-compensated sum of its slots in element order
// (deterministic).  Node-major [p][12] for pass B, or (REF) the reference's
// five (npoin,3) arrays, whose symmetric stress rows share entries.
// ---------------------------------------------------------------------
struct OutPtrs {
  float *p[5];
};
template <bool REF>
__global__ void k_gather_proj(MeshDev m, const float *__restrict__ slots, float *__restrict__ out, OutPtrs ref) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m.npoin) return;
  const int b = m.slot_ptr[p], en = m.slot_ptr[p + 1];
  const float sc = m.invMl[p];
  pdl_wait();
  pdl_trigger();
  float sum[12], cmp[12];
#pragma unroll
  for (int f = 0; f < 12; ++f) sum[f] = cmp[f] = 0.f;
  for (int s = b; s < en; ++s) {
    const float4 *v = reinterpret_cast<const float4 *>(slots + (long long)m.slot_idx[s] * 12);
    const float4 v0 = v[0], v1 = v[1], v2 = v[2];
    const float x[12] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w};
#pragma unroll
    for (int f = 0; f < 12; ++f) {  // Kahan summation
      const float y = x[f] - cmp[f];
      const float tt = sum[f] + y;
      cmp[f] = (tt - sum[f]) - y;
      sum[f] = tt;
    }
  }
#pragma unroll
  for (int f = 0; f < 12; ++f) sum[f] = sum[f] * sc;
  if (REF) {  // ref: ProjMX, ProjMY, ProjMZ, ProjMass, ProjEner
    constexpr int row[5][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}, {6, 7, 8}, {9, 10, 11}};
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int d = 0; d < 3; ++d) ref.p[a][p + m.npoin * d] = sum[row[a][d]];
  } else {
    float4 *o = reinterpret_cast<float4 *>(out + p * 12);
#pragma unroll
    for (int q = 0; q < 3; ++q) o[q] = make_float4(sum[4 * q], sum[4 * q + 1], sum[4 * q + 2], sum[4 * q + 3]);
  }
}

// ---------------------------------------------------------------------
// Assembly from node-sorted slots (written at slot_pos by k_rhs): node p's
// contributions are slots slot_ptr[p] .. slot_ptr[p+1]-1, in element
// order, so a warp streams one contiguous range with no index loads.
// ---------------------------------------------------------------------
// The 5 residuals from node-sorted pass-B slots into the reference's SoA
// outputs (optionally accumulated onto them), x invMl.
static __global__ void k_gather_sorted_res5(MeshDev m, const float *__restrict__ slots, long long zoff, OutPtrs out_soa,
                                     int accumulate, int use_invMl) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m.npoin) return;
  const float *sz = slots + 4 * zoff;
  const float4 *s4 = reinterpret_cast<const float4 *>(slots);
  const int b = m.slot_ptr[p], en = m.slot_ptr[p + 1];
  const float sc = use_invMl ? m.invMl[p] : 1.f;
  pdl_wait();
  pdl_trigger();
  float sum[5], cmp[5];
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    sum[f] = accumulate ? out_soa.p[f][p] : 0.f;
    cmp[f] = 0.f;
  }
  for (int s = b; s < en; ++s) {
    const float4 v = s4[s];
    const float x[5] = {v.x, v.y, v.z, v.w, sz[s]};
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const float y = x[f] - cmp[f];
      const float tt = sum[f] + y;
      cmp[f] = (tt - sum[f]) - y;
      sum[f] = tt;
    }
  }
#pragma unroll
  for (int f = 0; f < 5; ++f) out_soa.p[f][p] = sum[f] * sc;
}

}  // namespace sod
