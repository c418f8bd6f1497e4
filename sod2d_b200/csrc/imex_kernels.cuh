// Node kernels of the IMEX time integrator (imex_main,
// src/lib_sod2d/sources/time_integ_imex.f90:181-525) and of its implicit
// solve (conjGrad_imex, src/lib_sod2d/sources/mod_solver_imex.f90:25-342).
//
// Five-variable blocks are stored [mass N][energy N][momentum 3N], the
// order of the reference's x_vars(:,1..5).  Arithmetic is FP32 with the
// reference's operation order; the _rn intrinsics keep the compiler from
// contracting products into FMAs, so that the stage sums round as the
// reference's do.
#pragma once
#include "incomp_kernels.cuh"

namespace sod {

// Butcher tables, 1-based (ae explicit, ai implicit)
struct ImexCoef {
  float ae[5][5], ai[5][5];
};

// Stage right-hand side over all nodes, time_integ_imex.f90:342-391 (no
// source, wall model or buoyancy):
//   U2 = -dt R_stab - sum_{j<is} (dt ae(is,j) R_j + dt ai(is,j) D_j) + U1 Ml
// R, D: stage-major five-variable blocks; stab, lvl1: five-variable blocks.
static __global__ void k_imex_comb(long long npoin, int is, ImexCoef k, float dt, const float *__restrict__ Ml,
                            const float *__restrict__ R, const float *__restrict__ D, const float *__restrict__ stab,
                            const float *__restrict__ lvl1, float *__restrict__ rho2, float *__restrict__ E2,
                            float *__restrict__ q2) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npoin) return;
  const long long B = 5 * npoin;
  const float ml = Ml[p];
  float *out[5] = {rho2, E2, q2, q2 + npoin, q2 + 2 * npoin};
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const long long o = p + npoin * v;
    float a = __fmul_rn(-dt, stab[o]);
    for (int js = 1; js < is; ++js) {
      a = __fsub_rn(a, __fmul_rn(__fmul_rn(dt, k.ae[is][js]), R[(js - 1) * B + o]));
      a = __fsub_rn(a, __fmul_rn(__fmul_rn(dt, k.ai[is][js]), D[(js - 1) * B + o]));
    }
    out[v][p] = __fadd_rn(a, __fmul_rn(lvl1[o], ml));
  }
}

// h = gamma/(gamma-1) p / rho over the working nodes (time_integ_imex.f90:433)
static __global__ void k_aux_h(int npoin_w, const int *__restrict__ lpoin_w, float g_gm1, const float *__restrict__ rho,
                        const float *__restrict__ pr, float *__restrict__ h) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const int p = lpoin_w[t];
  h[p] = __fdiv_rn(__fmul_rn(g_gm1, pr[p]), rho[p]);
}

// Velocity and temperature of the CG argument v over the iterate's density
// (mod_solver_imex.f90:97-107, 160-167, 310-320): u = v_mom / x_mass,
// T = x_mass (gamma-1) (v_E / x_mass - |u|^2/2) / (x_mass Rgas).
__device__ __forceinline__ void imex_prim(float rhol, float El, const float (&q)[3], float gm1, float Rgas, long long p,
                                          long long npoin, float *__restrict__ au, float *__restrict__ aT) {
  float umag = 0.f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float ud = __fdiv_rn(q[d], rhol);
    au[p + npoin * d] = ud;
    umag = __fadd_rn(umag, __fmul_rn(ud, ud));
  }
  const float e = __fsub_rn(__fdiv_rn(El, rhol), __fmul_rn(0.5f, umag));
  aT[p] = __fdiv_rn(__fmul_rn(__fmul_rn(rhol, gm1), e), __fmul_rn(rhol, Rgas));
}

static __global__ void k_imex_prim(int npoin_w, long long npoin, const int *__restrict__ lpoin_w, float gm1, float Rgas,
                            const float *__restrict__ x, const float *__restrict__ v, float *__restrict__ au,
                            float *__restrict__ aT) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  const float q[3] = {v[p + npoin * 2], v[p + npoin * 3], v[p + npoin * 4]};
  imex_prim(x[p], v[p + npoin], q, gm1, Rgas, p, npoin, au, aT);
}

// qn = v Ml + qn fact dt over the working nodes, five variables
static __global__ void k_imex_op(int npoin_w, long long npoin, const int *__restrict__ lpoin_w, const float *__restrict__ Ml,
                          const float *__restrict__ v, float fact, float dt, float *__restrict__ qn) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  const float ml = Ml[p];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const long long o = p + npoin * k;
    qn[o] = __fadd_rn(__fmul_rn(v[o], ml), __fmul_rn(__fmul_rn(qn[o], fact), dt));
  }
}

// CG vector updates over the working nodes, five variables, M = Ml / dt:
//   mode 0: r = b - qn; z = r / M; p = z
//   mode 1: x += alpha p; r -= alpha qn; z1 = z; z = r / M
//   mode 2: p = z + beta p
static __global__ void k_imex_vec(int mode, int npoin_w, long long npoin, const int *__restrict__ lpoin_w,
                           const float *__restrict__ Ml, float dt, float alpha, float beta,
                           const float *__restrict__ b, float *__restrict__ x, float *__restrict__ r,
                           float *__restrict__ p, const float *__restrict__ qn, float *__restrict__ z,
                           float *__restrict__ z1) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long n = lpoin_w[t];
  const float M = __fdiv_rn(Ml[n], dt);
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const long long o = n + npoin * k;
    if (mode == 0) {
      const float rr = __fsub_rn(b[o], qn[o]);
      r[o] = rr;
      const float zz = __fdiv_rn(rr, M);
      z[o] = zz;
      p[o] = zz;
    } else if (mode == 1) {
      x[o] = __fadd_rn(x[o], __fmul_rn(alpha, p[o]));
      const float rr = __fsub_rn(r[o], __fmul_rn(alpha, qn[o]));
      r[o] = rr;
      z1[o] = z[o];
      z[o] = __fdiv_rn(rr, M);
    } else {
      p[o] = __fadd_rn(z[o], __fmul_rn(beta, p[o]));
    }
  }
}

// ---- the solve on the device (no global reductions) ---------------------------------
// The vector passes of conjGrad_imex, each fused with what follows it at the
// node, their sums taken by the last block (grid_sum): no host read inside an
// iteration.  One thread per node in reference order; `work` marks the
// working nodes.  z = r / M is formed again where it is used (M = Ml / dt),
// so no z is stored.  Node work bounds them: 5 to 15 arrays per pass.
constexpr int IMEX_THREADS = 256;

// Stage right-hand side (k_imex_comb), x = x0 = level 1, r = b - (x0 Ml +
// fact dt D(x0)), p = r / M with its velocity and temperature; ||r||^2 and
// r.z start the scalars.  One instantiation per stage: with the stage loop
// unrolled all its loads are in flight together (a runtime loop walked them
// two at a time: 0.2 ms more per step at 32^3).
template <int is>
__global__ void __launch_bounds__(IMEX_THREADS)
k_imex_start(long long npoin, const int *__restrict__ work, ImexCoef k, float dt, float fact, float gm1,
             float Rgas, double tol, const float *__restrict__ Ml, const float *__restrict__ R,
             const float *__restrict__ D, const float *__restrict__ stab, const float *__restrict__ lvl1,
             const float *__restrict__ Dx0, float *__restrict__ rho2, float *__restrict__ E2, float *__restrict__ q2,
             float *__restrict__ x, float *__restrict__ r, float *__restrict__ p, float *__restrict__ au,
             float *__restrict__ aT, CgScal *S, double *__restrict__ part, unsigned *ticket) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double v[2] = {0.0, 0.0};
  if (n < npoin) {
    const long long B = 5 * npoin;
    const float ml = Ml[n], M = __fdiv_rn(ml, dt);
    const bool w = work[n] != 0;
    float *out[5] = {rho2, E2, q2, q2 + npoin, q2 + 2 * npoin};
    float pv[5], x0 = 0.f, st[5], lv[5], dx[5], Rv[is - 1][5], Dv[is - 1][5];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const long long o = n + npoin * f;
      st[f] = stab[o]; lv[f] = lvl1[o]; dx[f] = Dx0[o];
#pragma unroll
      for (int js = 0; js < is - 1; ++js) { Rv[js][f] = R[js * B + o]; Dv[js][f] = D[js * B + o]; }
    }
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const long long o = n + npoin * f;
      float a = __fmul_rn(-dt, st[f]);
#pragma unroll
      for (int js = 1; js < is; ++js) {
        a = __fsub_rn(a, __fmul_rn(__fmul_rn(dt, k.ae[is][js]), Rv[js - 1][f]));
        a = __fsub_rn(a, __fmul_rn(__fmul_rn(dt, k.ai[is][js]), Dv[js - 1][f]));
      }
      const float l1 = lv[f], xm = __fmul_rn(l1, ml), bb = __fadd_rn(a, xm);
      if (!w) {
        out[f][n] = bb;
        continue;
      }
      if (f == 0) x0 = l1;
      const float rr = __fsub_rn(bb, __fadd_rn(xm, __fmul_rn(__fmul_rn(dx[f], fact), dt)));
      pv[f] = __fdiv_rn(rr, M);
      x[o] = l1;
      r[o] = rr;
      p[o] = pv[f];
      v[0] += (double)(rr * rr);
      v[1] += (double)(rr * pv[f]);
    }
    if (w) {
      const float q[3] = {pv[2], pv[3], pv[4]};
      imex_prim(x0, pv[1], q, gm1, Rgas, n, npoin, au, aT);
    }
  }
  double tot[2];
  if (grid_sum<2>(v, part, ticket, tot) && threadIdx.x == 0) {
    S->rz = tot[1];
    S->rr = tot[0];
    S->bnorm = sqrt(tot[0]);
    S->thr2 = tol * S->bnorm;
    S->iter = S->status = 0;
  }
}

// qn = p Ml + fact dt D(p) from the node-sorted slots of D(p) (summed as
// k_gather_sorted_res5), with p.qn and alpha.
static __global__ void __launch_bounds__(IMEX_THREADS)
k_imex_gather_op(MeshDev m, const int *__restrict__ work, const float *__restrict__ slots, long long zoff,
                 const float *__restrict__ Ml, float fact, float dt, const float *__restrict__ p,
                 float *__restrict__ qn, CgScal *S, double *__restrict__ part, unsigned *ticket) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x, N = m.npoin;
  int b = 0, en = 0;
  float ml = 0.f;
  const bool w = n < N && work[n] != 0;
  if (w) { b = m.slot_ptr[n]; en = m.slot_ptr[n + 1]; ml = Ml[n]; }
  pdl_wait();
  pdl_trigger();
  if (S->status) return;
  const float4 *s4 = reinterpret_cast<const float4 *>(slots);
  const float *sz = slots + 4 * zoff;
  float sum[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, cmp[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  for (int s = b; s < en; ++s) {
    const float4 y4 = s4[s];
    const float y5[5] = {y4.x, y4.y, y4.z, y4.w, sz[s]};
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const float y = y5[f] - cmp[f];
      const float tt = sum[f] + y;
      cmp[f] = (tt - sum[f]) - y;
      sum[f] = tt;
    }
  }
  double v[1] = {0.0};
  if (w) {
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const long long o = n + N * f;
      const float pv = p[o], qv = __fadd_rn(__fmul_rn(pv, ml), __fmul_rn(__fmul_rn(sum[f], fact), dt));
      qn[o] = qv;
      v[0] += (double)(pv * qv);
    }
  }
  double tot[1];
  if (grid_sum<1>(v, part, ticket, tot) && threadIdx.x == 0) S->alpha = (double)(float)(S->rz / tot[0]);
}

// x += alpha p ; r -= alpha qn ; ||r||^2, r.z, r.(z - z_old): beta and status
static __global__ void __launch_bounds__(IMEX_THREADS)
k_imex_update(long long npoin, const int *__restrict__ work, const float *__restrict__ Ml, float dt,
              const float *__restrict__ p, const float *__restrict__ qn, float *__restrict__ x, float *__restrict__ r,
              CgScal *S, double *__restrict__ part, unsigned *ticket) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool w = n < npoin && work[n] != 0;
  const float M = w ? __fdiv_rn(Ml[n], dt) : 1.f;
  pdl_wait();
  pdl_trigger();
  if (S->status) return;
  const float al = (float)S->alpha;
  double v[3] = {0.0, 0.0, 0.0};
  if (w) {
    float pv[5], qv[5], xv[5], rv[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const long long o = n + npoin * f;
      pv[f] = p[o]; qv[f] = qn[o]; xv[f] = x[o]; rv[f] = r[o];
    }
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      const long long o = n + npoin * f;
      x[o] = __fadd_rn(xv[f], __fmul_rn(al, pv[f]));
      const float rn = __fsub_rn(rv[f], __fmul_rn(al, qv[f])), zn = __fdiv_rn(rn, M), zo = __fdiv_rn(rv[f], M);
      r[o] = rn;
      v[0] += (double)(rn * rn);
      v[1] += (double)(rn * zn);
      v[2] += (double)(rn * (zn - zo));
    }
  }
  double tot[3];
  if (grid_sum<3>(v, part, ticket, tot) && threadIdx.x == 0) {
    S->iter += 1;
    S->rr = tot[0];
    const double nrm = sqrt(tot[0]);
    S->status = !isfinite(nrm) ? 3 : (nrm < S->thr2 ? 1 : 0);
    S->beta = (double)(float)(tot[2] / S->rz);
    S->rz = tot[1];
  }
}

// p = z + beta p with its velocity and temperature over the iterate's density
static __global__ void __launch_bounds__(IMEX_THREADS)
k_imex_dir(long long npoin, const int *__restrict__ work, const float *__restrict__ Ml, float dt, float gm1, float Rgas,
           const float *__restrict__ x, const float *__restrict__ r, float *__restrict__ p, float *__restrict__ au,
           float *__restrict__ aT, const CgScal *S) {
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool w = n < npoin && work[n] != 0;
  const float M = w ? __fdiv_rn(Ml[n], dt) : 1.f;
  pdl_wait();
  pdl_trigger();
  if (!w || S->status) return;
  const float be = (float)S->beta;
  float pv[5];
#pragma unroll
  for (int f = 0; f < 5; ++f) {
    const long long o = n + npoin * f;
    pv[f] = __fadd_rn(__fdiv_rn(r[o], M), __fmul_rn(be, p[o]));
    p[o] = pv[f];
  }
  const float q[3] = {pv[2], pv[3], pv[4]};
  imex_prim(x[n], pv[1], q, gm1, Rgas, n, npoin, au, aT);
}

// (rho, E, q) = x over the working nodes (mod_solver_imex.f90:331-338)
static __global__ void k_imex_out(int npoin_w, long long npoin, const int *__restrict__ lpoin_w, const float *__restrict__ x,
                           float *__restrict__ rho, float *__restrict__ E, float *__restrict__ q) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npoin_w) return;
  const long long p = lpoin_w[t];
  rho[p] = x[p];
  E[p] = x[p + npoin];
#pragma unroll
  for (int d = 0; d < 3; ++d) q[p + npoin * d] = x[p + npoin * (2 + d)];
}

}  // namespace sod
