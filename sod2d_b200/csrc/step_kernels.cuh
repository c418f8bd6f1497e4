// Kernels of the compressible time step around the RHS: SSP low-storage RK
// stage update (FP64 or FP32 state), equation of state, entropy-viscosity
// chain with the Ducros limiter, CFL time step and the analysis integrals.
#pragma once
#include "rhs_kernels.cuh"

namespace sod {

// Conserved state: 5 fields (rho, q0, q1, q2, E), each npoin long.
template <class T>
struct State5 {
  T *f[5];
};

// ---- RK stage update (time_integ_ls.f90:323-332 and :350-359) ---------
// first != 0: U2 += g*dt*R.  Otherwise U2 = l1*U1 + li*U2 + g*dt*R.
// The FP32 shadow (reference layout: rho, q(N,3), E) receives the result.
// The first stage also fills U1 with the level that U2 held, in place of a
// copy before the step; U1 is read only where l1 is not zero.  Bound by HBM
// (48^3, FP64, l1 = 0: 124 B a node in 62 us, 6.0 TB/s).
template <class T>
__global__ void k_stage(int npoin_w, long long npoin, const int *__restrict__ lpoin_w, State5<T> U1, State5<T> U2,
                        const float *__restrict__ Rmass, const float *__restrict__ Rmom,
                        const float *__restrict__ Rener, T l1, T li, T gdt, int first, float *__restrict__ rho32,
                        float *__restrict__ q32, float *__restrict__ E32) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  pdl_wait();
  pdl_trigger();
  const float R[5] = {Rmass[p], Rmom[p], Rmom[p + npoin], Rmom[p + 2 * npoin], Rener[p]};
  T u2[5], u1[5];
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    u2[f] = U2.f[f][p];
    u1[f] = (T)0;
    if (!first && l1 != (T)0) u1[f] = U1.f[f][p];
  }
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    if (first) U1.f[f][p] = u2[f];
    const T v = first ? u2[f] + gdt * (T)R[f] : l1 * u1[f] + li * u2[f] + gdt * (T)R[f];
    U2.f[f][p] = v;
    u2[f] = v;
  }
  rho32[p] = (float)u2[0];
  q32[p] = (float)u2[1];
  q32[p + npoin] = (float)u2[2];
  q32[p + 2 * npoin] = (float)u2[3];
  E32[p] = (float)u2[4];
}

// ---- end-of-step EOS (time_integ_ls.f90:391-407), with the Sutherland
// viscosity of the new temperature (as k_sutherland) when mu is given; u1,
// when given, receives the velocity that u held (level 1 <- level 2: here
// and not before the step, so that a step that fails in a callback leaves
// the velocity as it was, and by a store instead of an exchange of pointers,
// so that a captured step can be replayed; 24 B a node) ------------------
static __global__ void k_eos_end(int npoin_w, long long npoin, const int *__restrict__ lpoin_w, float gm1, float gamma,
                          float Rgas, const float *__restrict__ rho, const float *__restrict__ q,
                          const float *__restrict__ E, float *__restrict__ u, float *__restrict__ eint,
                          float *__restrict__ pr, float *__restrict__ csound, float *__restrict__ machno,
                          float *__restrict__ Tem, float mu_factor, float *__restrict__ mu,
                          float *__restrict__ u1) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  pdl_wait();
  pdl_trigger();
  const float r = rho[p];
  float umag = 0.f;
  float uu[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    uu[d] = q[p + npoin * d] / r;
    if (u1) u1[p + npoin * d] = u[p + npoin * d];
    u[p + npoin * d] = uu[d];
    umag = umag + uu[d] * uu[d];
  }
  const float ei = (E[p] / r) - 0.5f * umag;
  eint[p] = ei;
  const float pp = r * gm1 * ei;
  pr[p] = pp;
  const float c = sqrtf(gamma * pp / r);
  csound[p] = c;
  machno[p] = sqrtf(umag) / c;
  const float T = pp / (r * Rgas);
  Tem[p] = T;
  if (mu) mu[p] = mu_factor * 1.458e-6f * powf(T, 1.5f) / (T + 110.4f);
}

// ---- thermo_entropy, mod_entropy_viscosity.f90:411-433 ----------------
// eta1 <- eta2; eta2 <- rho/(g-1) log(max(p/p_inf, eps)/(rho/rho_inf)^g)
// (the flux u1 eta1 is formed by k_entropy_elem).
static __global__ void k_thermo_entropy(int npoin_w, const int *__restrict__ lpoin_w, float gamma,
                                 float p_inf, float rho_inf, const float *__restrict__ rho,
                                 const float *__restrict__ pr, float *__restrict__ eta1, float *__restrict__ eta2) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  pdl_wait();
  pdl_trigger();
  const float e1 = eta2[p];
  eta1[p] = e1;
  const float r = rho[p];
  eta2[p] = (r / (gamma - 1.0f)) * logf(fmaxf(pr[p] / p_inf, 1.1920929e-07f) / powf(r / rho_inf, gamma));
}

// ---- entropy flux residual + divergence + vorticity, one element pass --
// Node-sorted slots (as pass B's): a float4 and a float array with WANT_DC,
// else one float per element node.  Fields: 0 = generic_scalar_convec_ijk of (feta, eta1, u1)
// (elem_convec.f90:472-594), 1 = eval_divergence of u2
// (mod_operators.f90:485-570), 2..4 = compute_vorticity of u2 before the
// per-node averaging (mod_operators.f90:684-775).  WANT_DC = 0 skips 1..4.
// A thread owns a line along zeta (ColCfg), the fields taken one after the
// other: with a point per thread the shared and L1 pipe was 84 % busy with
// 120 staged words and 12 matrix words per point (here 70 and 2).
// The gathers of node values are the rest of its load: feta = u1 eta1, which
// thermo_entropy forms, is that product again here (feta null), not three
// more gathers.
template <int P, bool WANT_DC>
__global__ void __launch_bounds__(32 * COL_WARPS, P == 3 ? 6 : 4)
k_entropy_elem(MeshDev m, DMat<P, float> D, const float *__restrict__ feta, const float *__restrict__ eta1,
               const float *__restrict__ u1, const float *__restrict__ u2, float *__restrict__ slots,
               float fact) {
  using L = ColCfg<P>;
  constexpr int N1 = P + 1, N2 = N1 * N1, N = N1 * N2, NF = WANT_DC ? 10 : 7;  // eta, u1, feta, u2
  __shared__ float sm[L::EPB][NF][N];
  const int el = threadIdx.x / L::LPE, c = threadIdx.x % L::LPE;
  const long long e = (long long)blockIdx.x * L::EPB + el;
  const bool active = e < m.nelem && c < N2;
  const int i = c % N1, j = c / N1;
  const long long NP = m.npoin;
  int n[N1], pos[N1];
  float G[N1][10], Di[N1], Dj[N1];
  if (active) {  // mesh loads first (no other kernel writes them)
    const long long b = e * N + c;
#pragma unroll
    for (int k = 0; k < N1; ++k) { n[k] = m.conn[b + N2 * k]; pos[k] = m.slot_pos[b + N2 * k]; }
    const float *g = m.geo + e * 10 * N + c;
#pragma unroll
    for (int k = 0; k < N1; ++k)
#pragma unroll
      for (int q = 0; q < 10; ++q) G[k][q] = g[q * N + N2 * k];
    col_rows<P>(m, i, j, Di, Dj);
  }
  pdl_wait();
  pdl_trigger();
  if (active) {
    float in[NF][N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      in[0][k] = eta1[n[k]];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        in[1 + d][k] = u1[n[k] + NP * d];
        if (feta) in[4 + d][k] = feta[n[k] + NP * d];
        if (WANT_DC) in[(WANT_DC ? 7 : 0) + d][k] = u2[n[k] + NP * d];
      }
    }
#pragma unroll
    for (int k = 0; k < N1; ++k)
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (!feta) in[4 + d][k] = in[1 + d][k] * in[0][k];
#pragma unroll
    for (int q = 0; q < NF; ++q)
#pragma unroll
      for (int k = 0; k < N1; ++k) sm[el][q][c + N2 * k] = in[q][k];
  }
  __syncwarp();
  if (!active) return;
  // physical gradient of field q at this thread's points
  auto grad = [&](int q, float (&g)[N1][3]) {
    float col[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) col[k] = sm[el][q][c + N2 * k];
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      float g0, g1, g2 = 0.f;
      col_grad2<P>(sm[el][q], i, j, k, col[k], Di, Dj, g0, g1);
#pragma unroll
      for (int s = 0; s < N1; ++s) {
        const int mm = ref_order<P>(s);
        g2 = fmaf(D.d[k][mm], col[mm], g2);
      }
      const float *He = G[k];
#pragma unroll
      for (int a = 0; a < 3; ++a) g[k][a] = He[a] * g0 + He[a + 3] * g1 + He[a + 6] * g2;
    }
  };
  float g[N1][3], Re[N1], divU[N1], divFe[N1];
#pragma unroll
  for (int k = 0; k < N1; ++k) divU[k] = divFe[k] = 0.f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    grad(1 + d, g);
#pragma unroll
    for (int k = 0; k < N1; ++k) divU[k] += g[k][d];
    grad(4 + d, g);
#pragma unroll
    for (int k = 0; k < N1; ++k) divFe[k] += g[k][d];
  }
  grad(0, g);
#pragma unroll
  for (int k = 0; k < N1; ++k) {
    const int t = c + N2 * k;
    Re[k] = 0.5f * (divFe[k] + sm[el][0][t] * divU[k]);
#pragma unroll
    for (int a = 0; a < 3; ++a) Re[k] = Re[k] + 0.5f * (sm[el][1 + a][t] * g[k][a]);
    Re[k] = fact * (G[k][9] * Re[k]);
  }
  if (!WANT_DC) {
#pragma unroll
    for (int k = 0; k < N1; ++k) slots[pos[k]] = Re[k];
    return;
  }
  // divergence and the curl with the reference's Levi-Civita table
  // (CFDSolverBase.f90:1600-1606): curl_0 = g(1,2) - g(2,1), curl_1 =
  // g(2,0) - g(0,2), curl_2 = g(0,1) - g(1,0), g(j,k) = d u_j / d x_k
  float dv[N1], cu[N1][3];
  grad(NF - 3, g);
#pragma unroll
  for (int k = 0; k < N1; ++k) { dv[k] = g[k][0]; cu[k][1] = -g[k][2]; cu[k][2] = g[k][1]; }
  grad(NF - 2, g);
#pragma unroll
  for (int k = 0; k < N1; ++k) { dv[k] += g[k][1]; cu[k][0] = g[k][2]; cu[k][2] -= g[k][0]; }
  grad(NF - 1, g);
#pragma unroll
  for (int k = 0; k < N1; ++k) { dv[k] += g[k][2]; cu[k][0] -= g[k][1]; cu[k][1] += g[k][0]; }
#pragma unroll
  for (int k = 0; k < N1; ++k) {
    reinterpret_cast<float4 *>(slots)[pos[k]] = make_float4(Re[k], G[k][9] * dv[k], cu[k][0], cu[k][1]);
    slots[(long long)m.nelem * N * 4 + pos[k]] = cu[k][2];
  }
}

// Gather of the entropy pass: Reta (lumped: x invMl at working nodes),
// divU (raw), curl / lelpn (working nodes).  Kahan-compensated, element order.
template <bool WANT_DC>
__global__ void k_gather_entropy(MeshDev m, const float *__restrict__ slots, long long zoff,
                                 const int *__restrict__ lelpn, const int *__restrict__ is_work,
                                 float *__restrict__ Reta, float *__restrict__ divU, float *__restrict__ vort) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m.npoin) return;
  constexpr int NF = WANT_DC ? 5 : 1;
  const int b = m.slot_ptr[p], en = m.slot_ptr[p + 1];
  const float iml = m.invMl[p];
  const bool w = is_work[p] != 0;
  const float inv = WANT_DC && w ? (float)lelpn[p] : 1.f;
  pdl_wait();
  pdl_trigger();
  const float4 *s4 = reinterpret_cast<const float4 *>(slots);
  const float *sz = slots + 4 * zoff;
  float sum[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, cmp[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  for (int s = b; s < en; ++s) {
    float x[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (WANT_DC) {
      const float4 v = s4[s];
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; x[4] = sz[s];
    } else {
      x[0] = slots[s];
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const float y = x[f] - cmp[f];
      const float tt = sum[f] + y;
      cmp[f] = (tt - sum[f]) - y;
      sum[f] = tt;
    }
  }
  Reta[p] = sum[0] * iml;
  if (WANT_DC) {
    divU[p] = sum[1];
#pragma unroll
    for (int d = 0; d < 3; ++d) vort[p + m.npoin * d] = w ? sum[2 + d] / inv : sum[2 + d];
  }
}

// auxReta = (1.5 R2 - 0.5 R1) + (eta2 - eta1)/dt; R1 <- R2 (time_integ_ls.f90:437-443)
static __global__ void k_aux_reta(int npoin_w, const int *__restrict__ lpoin_w, float dt, float *__restrict__ Reta1,
                           const float *__restrict__ Reta2, const float *__restrict__ eta1,
                           const float *__restrict__ eta2, float *__restrict__ aux) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  aux[p] = (1.5f * Reta2[p] - 0.5f * Reta1[p]) + 1.0f * (eta2[p] - eta1[p]) / dt;
  Reta1[p] = Reta2[p];
}

// Minimum of rho over working nodes (order-independent, deterministic).
// out_bits starts as 0x7f7f7f7f (one memset); the reference's initial value
// 100000 enters in k_visc.
// grid of the node min / max reductions: 8 blocks of 256 per SM
constexpr int MINMAX_BLOCKS = 148 * 8;
static __global__ void k_min_rho(int npoin_w, const int *__restrict__ lpoin_w, const float *__restrict__ rho,
                          unsigned int *__restrict__ out_bits) {
  float v = 100000.0f;
  // four strides per trip with every load issued first (min is order-free)
  const int stride = gridDim.x * blockDim.x;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  for (; t + 3 * stride < npoin_w; t += 4 * stride) {
    int p[4];
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) p[u] = lpoin_w[t + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = rho[p[u]];
#pragma unroll
    for (int u = 0; u < 4; ++u) v = fminf(v, x[u]);
  }
  for (; t < npoin_w; t += stride) v = fminf(v, rho[lpoin_w[t]]);
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) atomicMin(out_bits, __float_as_uint(v));  // rho > 0: bit order = value order
}

// ---- smart_visc_spectral_imex (+ ducros_visc_limit) ---------------------
// mod_entropy_viscosity.f90:113-227 (high-Mach path) and :277-314.
// One warp per element.  mue_t is [e][t]; mue_ref (reference (nelem,ngaus)
// layout) is optional.  ducros = 0 skips the limiter (first step).
struct ViscArgs {
  const float *Reta, *rho, *u, *csound, *divU, *vort, *Ml, *helem, *helem_l_t;
  const unsigned int *min_rho_bits;
  float ce, cmax, cglob, ducros_min, inv_p;
  int ducros;
};

// A lane holds its nodes' loads (two at P = 3, four at P = 4), all issued
// before the element maximum is formed.
template <int P>
__global__ void k_visc(MeshDev m, ViscArgs A, const int *__restrict__ a_of_t, float *__restrict__ mue_t,
                       float *__restrict__ mue_ref) {
  constexpr int N = Cfg<P>::N, IT = (N + 31) / 32;
  const long long e = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x % 32;
  if (e >= m.nelem) return;
  const long long NP = m.npoin;
  int p[IT];
  float hl[IT];
  const float he = A.helem[e];
#pragma unroll
  for (int q = 0; q < IT; ++q) {
    const int t = lane + 32 * q;
    p[q] = t < N ? m.conn[e * N + t] : -1;
    hl[q] = A.ducros && t < N ? A.helem_l_t[e * N + t] : 1.f;
  }
  pdl_wait();
  pdl_trigger();
  const float norm = fminf(__uint_as_float(*A.min_rho_bits), 100000.0f);
  float um[IT], cs[IT], rh[IT], re[IT], dv[IT], vv[IT];
#pragma unroll
  for (int q = 0; q < IT; ++q) {
    if (p[q] < 0) continue;
    const long long n = p[q];
    const float u0 = A.u[n], u1 = A.u[n + NP], u2 = A.u[n + 2 * NP];
    cs[q] = A.csound[n];
    rh[q] = A.rho[n];
    re[q] = A.Reta[n];
    um[q] = sqrtf(u0 * u0 + u1 * u1 + u2 * u2);
    if (A.ducros) {
      dv[q] = A.divU[n] / A.Ml[n];
      const float v0 = A.vort[n], v1 = A.vort[n + NP], v2 = A.vort[n + 2 * NP];
      vv[q] = v0 * v0 + v1 * v1 + v2 * v2;
    }
  }
  float betae = 0.f;
#pragma unroll
  for (int q = 0; q < IT; ++q)
    if (p[q] >= 0) {
      const float aux1 = um[q] + 1.0f * cs[q];
      betae = fmaxf(betae, (rh[q] * he) * (A.cmax * A.inv_p) * aux1);
    }
  for (int o = 16; o > 0; o >>= 1) betae = fmaxf(betae, __shfl_xor_sync(0xffffffffu, betae, o));
  const float hp = he * A.inv_p;
#pragma unroll
  for (int q = 0; q < IT; ++q) {
    if (p[q] < 0) continue;
    const int t = lane + 32 * q;
    const float R1 = rh[q] * fabsf(re[q]) / norm;
    const float Ve = A.ce * R1 * (hp * hp);
    float mu = A.cglob * fminf(Ve, betae);
    if (A.ducros) {
      const float d2 = dv[q] * dv[q];
      const float eps = 1.1920929e-07f;
      const float phi = fminf((4.0f / 3.0f) * d2 / (d2 + vv[q] + eps), 1.0f);
      const float hq = 1.0f * um[q] / hl[q];
      const float phi2 = d2 / (d2 + hq * hq + eps);
      mu = mu * (fmaxf(phi - A.ducros_min, 0.f) * phi2 + A.ducros_min);
    }
    mue_t[e * N + t] = mu;
    if (mue_ref) mue_ref[e + m.nelem * a_of_t[t]] = mu;
  }
}

// ducros_visc_limit, mod_entropy_viscosity.f90:277-314, on a given mu_e in
// the reference's (nelem, ngaus) layout: mu_e *= max(phi - min, 0) phi2 +
// min with phi, phi2 from div u / Ml, the vorticity and |u| / helem_l (the
// reference's betae is computed there but unused).  Warp per element.
template <int P>
__global__ void k_ducros(MeshDev m, const float *__restrict__ u, const float *__restrict__ divU,
                         const float *__restrict__ vort, const float *__restrict__ Ml,
                         const float *__restrict__ helem_l_t, float ducros_min, const int *__restrict__ a_of_t,
                         float *__restrict__ mue_ref) {
  constexpr int N = Cfg<P>::N;
  const long long e = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x % 32;
  if (e >= m.nelem) return;
  const long long NP = m.npoin;
  for (int t = lane; t < N; t += 32) {
    const int p = m.conn[e * N + t];
    const float divUl = divU[p] / Ml[p];
    const float u0 = u[p], u1 = u[p + NP], u2 = u[p + 2 * NP];
    const float aux2 = sqrtf(u0 * u0 + u1 * u1 + u2 * u2);
    const float v0 = vort[p], v1 = vort[p + NP], v2 = vort[p + 2 * NP];
    const float vv = v0 * v0 + v1 * v1 + v2 * v2;
    const float d2 = divUl * divUl;
    const float eps = 1.1920929e-07f;  // epsilon(1.0) of real(4)
    const float phi = fminf((4.0f / 3.0f) * d2 / (d2 + vv + eps), 1.0f);
    const float hl = 1.0f * aux2 / helem_l_t[e * N + t];
    const float phi2 = d2 / (d2 + hl * hl + eps);
    float &mu = mue_ref[e + m.nelem * a_of_t[t]];
    mu = mu * (fmaxf(phi - ducros_min, 0.f) * phi2 + ducros_min);
  }
}

// Stage update of rk_4_ls_main on reference-layout FP32 arrays, working
// nodes, five fields (rho, E, q x/y/z): first stage U2 += (gam dt) R
// (time_integ_ls.f90:325-329), later stages U2 = l1 U1 + li U2 + (gam dt) R
// (:352-356), rounded as the reference (no contraction).
static __global__ void k_ls_stage_ref(int npoin_w, long long npoin, const int *__restrict__ lpoin_w, int first, float l1,
                               float li, float gam, float dt, const float *__restrict__ rho1,
                               const float *__restrict__ q1, const float *__restrict__ E1, float *__restrict__ rho2,
                               float *__restrict__ q2, float *__restrict__ E2, const float *__restrict__ Rmass,
                               const float *__restrict__ Rmom, const float *__restrict__ Rener) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  const float gdt = __fmul_rn(gam, dt);
  auto upd = [&](float u1, float u2, float r) {
    return first ? __fadd_rn(u2, __fmul_rn(gdt, r))
                 : __fadd_rn(__fadd_rn(__fmul_rn(l1, u1), __fmul_rn(li, u2)), __fmul_rn(gdt, r));
  };
  rho2[p] = upd(first ? 0.f : rho1[p], rho2[p], Rmass[p]);
  E2[p] = upd(first ? 0.f : E1[p], E2[p], Rener[p]);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const long long k = p + npoin * d;
    q2[k] = upd(first ? 0.f : q1[k], q2[k], Rmom[k]);
  }
}

// Sutherland viscosity at working nodes.
static __global__ void k_sutherland(int npoin_w, const int *__restrict__ lpoin_w, float mu_factor,
                             const float *__restrict__ Tem, float *__restrict__ mu) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  const float T = Tem[p];
  mu[p] = mu_factor * 1.458e-6f * powf(T, 1.5f) / (T + 110.4f);
}

// ---- adapt_dt_cfl, mod_time_ops.f90:11-62: per element, then min -------
// A warp takes two elements at P = 3 (one at P = 4), all loads of a lane's
// four nodes in flight, and a block issues one atomic: one atomic per element
// to the same word was half of this kernel's time (110,592 elements: 120 us).
// out_bits starts as 0x7f7f7f7f; the caller applies the reference's initial 1e14.
template <int P>
struct DtCfg {
  static constexpr int EPW = P == 3 ? 2 : 1, EPB = 8 * EPW;  // elements per warp, per block
};
template <int P>
__global__ void __launch_bounds__(256)
k_dt(MeshDev m, const float *__restrict__ helem, const float *__restrict__ u, const float *__restrict__ csound,
     const float *__restrict__ mu_fluid, const float *__restrict__ mue_t, const float *__restrict__ rho, float cfl_conv,
     float cfl_diff, unsigned int *__restrict__ out_bits) {
  constexpr int N = Cfg<P>::N, IT = (N + 31) / 32, EPW = DtCfg<P>::EPW;
  __shared__ unsigned sh[8];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const long long NP = m.npoin, e0 = (long long)blockIdx.x * DtCfg<P>::EPB + warp * EPW;
  int p[EPW][IT];
  float me[EPW][IT], um[EPW][IT], cs[EPW][IT], mu[EPW][IT], rh[EPW][IT];
#pragma unroll
  for (int w = 0; w < EPW; ++w)
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      const int t = lane + 32 * q;
      const bool in = e0 + w < m.nelem && t < N;
      p[w][q] = in ? m.conn[(e0 + w) * N + t] : -1;
      me[w][q] = in ? mue_t[(e0 + w) * N + t] : 0.f;
    }
#pragma unroll
  for (int w = 0; w < EPW; ++w)
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      if (p[w][q] < 0) continue;
      const long long n = p[w][q];
      um[w][q] = fmaxf(fmaxf(fabsf(u[n]), fabsf(u[n + NP])), fabsf(u[n + 2 * NP]));
      cs[w][q] = csound[n];
      mu[w][q] = mu_fluid[n];
      rh[w][q] = rho[n];
    }
  unsigned best = 0x7f7f7f7fu;
#pragma unroll
  for (int w = 0; w < EPW; ++w) {
    float L3 = 0.f, maxMU = 0.f;
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      if (p[w][q] < 0) continue;
      L3 = fmaxf(L3, um[w][q] + cs[w][q]);
      maxMU = fmaxf(maxMU, (0.0f + mu[w][q] + me[w][q]) / rh[w][q]);
    }
    for (int o = 16; o > 0; o >>= 1) {
      L3 = fmaxf(L3, __shfl_xor_sync(0xffffffffu, L3, o));
      maxMU = fmaxf(maxMU, __shfl_xor_sync(0xffffffffu, maxMU, o));
    }
    if (e0 + w < m.nelem) {
      const float hp = helem[e0 + w] / (float)(2 * P + 1);
      const float dconv = cfl_conv * hp / L3;
      const float ddiff = cfl_diff * (hp * hp) / maxMU;
      best = min(best, __float_as_uint(fminf(dconv, ddiff)));  // dt > 0: bit order = value order
    }
  }
  if (lane == 0) sh[warp] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) best = min(best, sh[w]);
    atomicMin(out_bits, best);
  }
}

// ---- analysis (mod_analysis.f90:10-168): per-element FP32 partials -----
// part[e*3 + 0] = sum_g gpvol*sum_a Ngp(g,a)*0.5*rho*|u|^2 (a)   (volAvg_EK)
// part[e*3 + 1] = sum_g gpvol*(mu+mu_e)*|curl u|^2                (eps_S)
// part[e*3 + 2] = sum_g gpvol*mu*(div u)^2                        (eps_D)
template <int P, int EPB>
__global__ void __launch_bounds__(EPB *Cfg<P>::NT)
k_analysis_elem(MeshDev m, const float *__restrict__ rho, const float *__restrict__ u,
                const float *__restrict__ mu_fluid, const float *__restrict__ mue_t,
                const float *__restrict__ Ngp_t /*[g][a] tensor order*/, float *__restrict__ part) {
  constexpr int N1 = Cfg<P>::N1, N = Cfg<P>::N, NT = Cfg<P>::NT;
  __shared__ __align__(16) float sm[EPB][4][N];
  __shared__ float red[EPB][3][NT / 32];
  const int el = threadIdx.x / NT, t = threadIdx.x % NT, lane = threadIdx.x % 32, w = t / 32;
  const long long e = (long long)blockIdx.x * EPB + el;
  const bool active = (e < m.nelem) && (t < N);
  const long long NP = m.npoin;
  int node = 0;
  if (active) {
    node = m.conn[e * N + t];
    const float u0 = u[node], u1 = u[node + NP], u2 = u[node + 2 * NP];
    sm[el][0][t] = u0; sm[el][1][t] = u1; sm[el][2][t] = u2;
    sm[el][3][t] = 0.5f * rho[node] * (u0 * u0 + u1 * u1 + u2 * u2);
  }
  __syncthreads();
  float r[3] = {0.f, 0.f, 0.f};
  if (active) {
    const int i = t % N1, j = (t / N1) % N1, k = t / (N1 * N1);
    float Di[N1], Dj[N1], Dk[N1];
#pragma unroll
    for (int s = 0; s < N1; ++s) { Di[s] = m.Dnat[i * N1 + s]; Dj[s] = m.Dnat[j * N1 + s]; Dk[s] = m.Dnat[k * N1 + s]; }
    const float *g = m.geo + e * 10 * N + t;
    float He[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) He[c] = g[c * N];
    const float gv = g[9 * N];
    float ek = 0.f;
    for (int a = 0; a < N; ++a) ek = fmaf(Ngp_t[t * N + a], sm[el][3][a], ek);
    float gu[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float a0, a1, a2;
      iso_grad<P>(sm[el][c], i, j, k, Di, Dj, Dk, a0, a1, a2);
#pragma unroll
      for (int b = 0; b < 3; ++b) gu[c][b] = He[b] * a0 + He[b + 3] * a1 + He[b + 6] * a2;
    }
    float div = gu[0][0] + gu[1][1] + gu[2][2];
    div = div * div;
    const float c0 = gu[1][2] - gu[2][1], c1 = gu[2][0] - gu[0][2], c2 = gu[0][1] - gu[1][0];
    const float curl2 = c0 * c0 + c1 * c1 + c2 * c2;
    const float mu = mu_fluid[node];
    r[0] = gv * ek;
    r[1] = gv * (mu + mue_t[e * N + t]) * curl2;
    r[2] = gv * mu * div;
  }
  // fixed-order block reduction per element
#pragma unroll
  for (int q = 0; q < 3; ++q)
    for (int o = 16; o > 0; o >>= 1) r[q] += __shfl_down_sync(0xffffffffu, r[q], o);
  if (lane == 0)
    for (int q = 0; q < 3; ++q) red[el][q][w] = r[q];
  __syncthreads();
  if (t == 0 && e < m.nelem) {
    for (int q = 0; q < 3; ++q) {
      float s = 0.f;
      for (int ww = 0; ww < NT / 32; ++ww) s += red[el][q][ww];
      part[e * 3 + q] = s;
    }
  }
}

// Deterministic FP64 sum of per-element partials: one block, fixed order.
static __global__ void k_sum_parts(long long nelem, const float *__restrict__ part, double *__restrict__ out3) {
  __shared__ double sh[3][1024];
  const int t = threadIdx.x;
  double s[3] = {0.0, 0.0, 0.0};
  for (long long e = t; e < nelem; e += blockDim.x)
    for (int q = 0; q < 3; ++q) s[q] += (double)part[e * 3 + q];
  for (int q = 0; q < 3; ++q) sh[q][t] = s[q];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (t < w)
      for (int q = 0; q < 3; ++q) sh[q][t] += sh[q][t + w];
    __syncthreads();
  }
  if (t == 0)
    for (int q = 0; q < 3; ++q) out3[q] = sh[q][0];
}

static __global__ void k_max_mach(int npoin_w, const int *__restrict__ lpoin_w, const float *__restrict__ machno,
                           unsigned int *__restrict__ out_bits) {
  float v = 0.f;
  const int stride = gridDim.x * blockDim.x;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  for (; t + 3 * stride < npoin_w; t += 4 * stride) {
    int p[4];
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) p[u] = lpoin_w[t + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = machno[p[u]];
#pragma unroll
    for (int u = 0; u < 4; ++u) v = fmaxf(v, x[u]);
  }
  for (; t < npoin_w; t += stride) v = fmaxf(v, machno[lpoin_w[t]]);
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out_bits, __float_as_uint(v));
}

}  // namespace sod
