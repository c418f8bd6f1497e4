// Kernels of the incompressible pressure path: matrix-free Laplacian
// (eval_laplacian_mult), its Jacobi diagonal, gradient, divergence,
// skew-symmetric convection, and the vector kernels of the (flexible)
// conjugate-gradient solvers with deterministic FP64 reductions.
#pragma once
#include "rhs_kernels.cuh"

namespace sod {

// Rows and columns of the 1-D derivative matrix in V, rotated to start at the
// diagonal (MeshDev::Drot, D64).
template <int P>
__device__ __forceinline__ void load_rot(const MeshDev &m, int c, bool col, double (&D)[P + 1]) {
  const double2 *r = reinterpret_cast<const double2 *>(m.D64 + 8 * (c + (col ? P + 1 : 0)));
  const double2 v0 = r[0], v1 = r[1];
  D[0] = v0.x; D[1] = v0.y; D[2] = v1.x; D[3] = v1.y;
  if (P == 4) D[4] = r[2].x;
}
template <int P>
__device__ __forceinline__ void load_rot(const MeshDev &m, int c, bool col, float (&D)[P + 1]) {
  load_drot<P>(m.Drot + (col ? 8 * (P + 1) : 0), c, D);
}

// ---- Laplacian: ResP = sum_e int grad N . grad p  (mod_operators.f90:16-112)
// V = float (reference arithmetic) or double.  Writes one V per element node
// into node-sorted slots (slot_pos), which the assembly sums contiguously.
// DIR (the CG iteration): the operand is the new search direction
// z + beta p, formed on the fly from z, the previous p and *beta (the
// update p = z + beta p itself is stored by k_cg_q).
//
// A thread owns the line of P + 1 points along zeta over its (i, j); 16
// lanes (P = 3) or 25 of 32 (P = 4) take an element, so nothing but warp
// barriers is needed.  The zeta derivatives and their transpose stay in
// registers with the matrix as constant operands; in xi and eta a point
// reads its line's other P nodes from shared memory, its own from registers
// (cyclic order 2, 3, .., 1, own: see k_rhs).  With one point per thread the
// shared and L1 pipe was 82 % busy -- 24 FP64 shared loads and 24 matrix
// loads per point -- and bound the kernel; this form has 12 and 4.  All of a
// thread's mesh loads (J^-1, weights, nodes, slot positions: 48 at P = 3)
// are in flight before the programmatic wait.
constexpr int LAP_WARPS = COL_WARPS;
template <int P>
struct LapCfg : ColCfg<P> {
  static constexpr int MINB = P == 3 ? 8 : 6;  // blocks per SM
};
template <int P, class V, bool DIR = false>
__global__ void __launch_bounds__(32 * LAP_WARPS, LapCfg<P>::MINB)
k_lap_elem(MeshDev m, DMat<P, V> D, const V *__restrict__ p, V *__restrict__ slots,
           const int *__restrict__ stop = nullptr, const V *__restrict__ z = nullptr,
           const double *__restrict__ beta = nullptr) {
  using L = LapCfg<P>;
  constexpr int N1 = P + 1, N2 = N1 * N1, N = N1 * N2;
  __shared__ V sm[L::EPB][2][N];
  const int el = threadIdx.x / L::LPE, c = threadIdx.x % L::LPE;
  const long long e = (long long)blockIdx.x * L::EPB + el;
  const bool active = e < m.nelem && c < N2;
  const int i = c % N1, j = c / N1;
  if (ended_late(stop, 148 * L::MINB)) return;
  int n[N1], pos[N1];
  float G[N1][10];
  V Di[N1], Dj[N1];
#pragma unroll
  for (int k = 0; k < N1; ++k) n[k] = pos[k] = 0;
  if (active) {
    const long long b = e * N + c;
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      n[k] = m.conn[b + N2 * k];
      pos[k] = m.slot_pos[b + N2 * k];
    }
    const float *g = m.geo + e * 10 * N + c;
#pragma unroll
    for (int k = 0; k < N1; ++k)
#pragma unroll
      for (int q = 0; q < 10; ++q) G[k][q] = g[q * N + N2 * k];
    load_rot<P>(m, i, false, Di);
    load_rot<P>(m, j, false, Dj);
  }
  // the q-th node of a line: cyclic step from the own node, own last
  auto step = [](int q) -> int { return q == P ? 0 : (q == P - 1 ? 1 : q + 2); };
  auto xi = [&](int q, int k) -> int { const int s = step(q); return c + (i + s < N1 ? s : s - N1) + N2 * k; };
  auto et = [&](int q, int k) -> int { const int s = step(q); return c + (j + s < N1 ? s : s - N1) * N1 + N2 * k; };
  V *A = sm[el][0], *B = sm[el][1];
  pdl_wait();
  pdl_trigger();
  if (stop && *stop) return;
  V f[N1];
  if (active) {
    const V bt = DIR ? (V)*beta : (V)0;
#pragma unroll
    for (int k = 0; k < N1; ++k) f[k] = DIR ? z[n[k]] + bt * p[n[k]] : p[n[k]];
#pragma unroll
    for (int k = 0; k < N1; ++k) A[c + N2 * k] = f[k];
  }
  __syncwarp();
  V C0[N1], C1[N1], C2[N1];
  if (active) {
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      V g0 = 0, g1 = 0, g2 = 0;
#pragma unroll
      for (int q = 0; q < N1; ++q) {
        g0 += Di[step(q)] * (q == P ? f[k] : A[xi(q, k)]);
        g1 += Dj[step(q)] * (q == P ? f[k] : A[et(q, k)]);
        const int mm = ref_order<P>(q);
        g2 += D.d[k][mm] * f[mm];
      }
      V He[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) He[q] = (V)G[k][q];
      const V gv = (V)G[k][9];
      V gP[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) gP[a] = He[a] * g0 + He[a + 3] * g1 + He[a + 6] * g2;
      C0[k] = gv * (He[0] * gP[0] + He[1] * gP[1] + He[2] * gP[2]);
      C1[k] = gv * (He[3] * gP[0] + He[4] * gP[1] + He[5] * gP[2]);
      C2[k] = gv * (He[6] * gP[0] + He[7] * gP[1] + He[8] * gP[2]);
    }
  }
  __syncwarp();  // the operand has been read
  if (active) {
#pragma unroll
    for (int k = 0; k < N1; ++k) { A[c + N2 * k] = C0[k]; B[c + N2 * k] = C1[k]; }
    load_rot<P>(m, i, true, Di);
    load_rot<P>(m, j, true, Dj);
  }
  __syncwarp();
  if (!active) return;
#pragma unroll
  for (int k = 0; k < N1; ++k) {
    V acc = 0;
#pragma unroll
    for (int q = 0; q < N1; ++q) {
      acc += Di[step(q)] * (q == P ? C0[k] : A[xi(q, k)]);
      acc += Dj[step(q)] * (q == P ? C1[k] : B[et(q, k)]);
      const int mm = ref_order<P>(q);
      acc += D.d[mm][k] * C2[mm];
    }
    slots[pos[k]] = acc;
  }
}

// Scalar node-sorted slots: out(p) = their Kahan sum in element order, onto
// out(p) when accumulate is set.
template <class V>
__global__ void k_gather_sorted1(MeshDev m, const V *__restrict__ slots, V *__restrict__ out, int accumulate) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m.npoin) return;
  const int b = m.slot_ptr[p], en = m.slot_ptr[p + 1];
  pdl_wait();
  pdl_trigger();
  V sum = accumulate ? out[p] : (V)0, cmp = 0;
  for (int s = b; s < en; ++s) {
    const V y = slots[s] - cmp;
    const V tt = sum + y;
    cmp = (tt - sum) - y;
    sum = tt;
  }
  out[p] = sum;
}

// Three values of a node from 4-wide node-sorted slots, the same sums.
__device__ __forceinline__ void node_sum3(const float4 *__restrict__ s4, int b, int en, float (&sum)[3]) {
  float cmp[3] = {0.f, 0.f, 0.f};
  sum[0] = sum[1] = sum[2] = 0.f;
  for (int s = b; s < en; ++s) {
    const float4 v = s4[s];
    const float x[3] = {v.x, v.y, v.z};
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const float y = x[f] - cmp[f];
      const float tt = sum[f] + y;
      cmp[f] = (tt - sum[f]) - y;
      sum[f] = tt;
    }
  }
}
static __global__ void k_gather_sorted3(MeshDev m, const float *__restrict__ slots, float *__restrict__ out,
                                        int use_invMl) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m.npoin) return;
  const int b = m.slot_ptr[p], en = m.slot_ptr[p + 1];
  const float sc = use_invMl ? m.invMl[p] : 1.f;
  pdl_wait();
  pdl_trigger();
  float sum[3];
  node_sum3(reinterpret_cast<const float4 *>(slots), b, en, sum);
#pragma unroll
  for (int f = 0; f < 3; ++f) out[p + m.npoin * f] = sum[f] * sc;
}

// ---- eval_laplacian_diag, mod_operators.f90:638-682 --------------------
// d(a) = sum_g gpvol(g) |grad N_a(g)|^2; with GLL collocation grad N_a(g)
// is non-zero only on the three lines through a.  One thread per node a
// of an element loops over the Gauss points of those lines.
template <int P>
__global__ void k_lap_diag_elem(MeshDev m, float *__restrict__ slots) {
  constexpr int N1 = Cfg<P>::N1, N = Cfg<P>::N;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)m.nelem * N) return;
  const long long e = idx / N;
  const int a = (int)(idx % N);
  const int ia = a % N1, ja = (a / N1) % N1, ka = a / (N1 * N1);
  const float *g = m.geo + e * 10 * N;
  float d = 0.f;
  auto add = [&](int i, int j, int k) {
    const int gp = i + N1 * (j + N1 * k);
    // iso-derivatives of N_a at gp: D[i][ia] d_{j,ja} d_{k,ka}, ...
    const float d0 = (j == ja && k == ka) ? m.Dnat[i * N1 + ia] : 0.f;
    const float d1 = (i == ia && k == ka) ? m.Dnat[j * N1 + ja] : 0.f;
    const float d2 = (i == ia && j == ja) ? m.Dnat[k * N1 + ka] : 0.f;
    if (d0 == 0.f && d1 == 0.f && d2 == 0.f) return;
    const float gv = g[9 * N + gp];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float gc = g[c * N + gp] * d0 + g[(c + 3) * N + gp] * d1 + g[(c + 6) * N + gp] * d2;
      d += gv * gc * gc;
    }
  };
  // the points of the three lines in ascending order; testing all N of an
  // element for each of its nodes took 390 us at 8,000 order-4 elements
  for (int k = 0; k < N1; ++k) {
    if (k != ka) { add(ia, ja, k); continue; }
    for (int j = 0; j < N1; ++j) {
      if (j != ja) { add(ia, j, k); continue; }
      for (int i = 0; i < N1; ++i) add(i, j, k);
    }
  }
  slots[m.slot_pos[idx]] = d;
}

// ---- gradient / divergence / incompressible convection ----------------
// Node-sorted slots.
// MODE 0: gradient of a scalar x: slots (width 4) = gpvol*grad x (3)
// MODE 1: divergence of u: slots (width 1) = gpvol * div u
// MODE 2: full_convec_ijk_incomp (elem_convec_incomp.f90:19-125): slots
//         (width 4) = gpvol * 0.5*(div(q u) + u div q + (u.grad) q)
// The mesh loads come before the programmatic wait and the staging barrier.
template <int P, int EPB, int MODE>
__global__ void __launch_bounds__(EPB *Cfg<P>::NT)
k_vec_elem(MeshDev m, const float *__restrict__ x, const float *__restrict__ u, const float *__restrict__ q,
           float *__restrict__ slots) {
  constexpr int N1 = Cfg<P>::N1, N = Cfg<P>::N, NT = Cfg<P>::NT;
  constexpr int NF = MODE == 0 ? 1 : (MODE == 1 ? 3 : 12);
  __shared__ __align__(16) float sm[EPB][NF][N];
  const int el = threadIdx.x / NT, t = threadIdx.x % NT;
  const long long e = (long long)blockIdx.x * EPB + el;
  const bool active = (e < m.nelem) && (t < N);
  const long long NP = m.npoin;
  float ul[3] = {0.f, 0.f, 0.f}, ql[3] = {0.f, 0.f, 0.f};
  int node = 0, pos = 0;
  float He[9], gv = 0.f;
  if (active) {
    node = m.conn[e * N + t];
    pos = m.slot_pos[e * N + t];
    const float *g = m.geo + e * 10 * N + t;
#pragma unroll
    for (int c = 0; c < 9; ++c) He[c] = g[c * N];
    gv = g[9 * N];
  }
  pdl_wait();
  pdl_trigger();
  if (active) {
    if (MODE == 0) sm[el][0][t] = x[node];
    if (MODE >= 1)
      for (int d = 0; d < 3; ++d) { ul[d] = u[node + NP * d]; sm[el][d][t] = (MODE == 1) ? ul[d] : 0.f; }
    if (MODE == 2) {
      for (int d = 0; d < 3; ++d) { ql[d] = q[node + NP * d]; sm[el][d][t] = ql[d]; }
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) sm[el][3 + a * 3 + b][t] = ql[a] * ul[b];
    }
  }
  __syncthreads();
  if (!active) return;
  const int i = t % N1, j = (t / N1) % N1, k = t / (N1 * N1);
  float Di[N1], Dj[N1], Dk[N1];
#pragma unroll
  for (int s = 0; s < N1; ++s) { Di[s] = m.Dnat[i * N1 + s]; Dj[s] = m.Dnat[j * N1 + s]; Dk[s] = m.Dnat[k * N1 + s]; }
  float out[3] = {0.f, 0.f, 0.f};
  float a0, a1, a2;
  if (MODE == 0) {
    iso_grad<P>(sm[el][0], i, j, k, Di, Dj, Dk, a0, a1, a2);
#pragma unroll
    for (int a = 0; a < 3; ++a) out[a] = gv * (He[a] * a0 + He[a + 3] * a1 + He[a + 6] * a2);
  } else if (MODE == 1) {
    float dv = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      iso_grad<P>(sm[el][c], i, j, k, Di, Dj, Dk, a0, a1, a2);
      dv += He[c] * a0 + He[c + 3] * a1 + He[c + 6] * a2;
    }
    out[0] = gv * dv;
  } else {
    float gradQ[3][3], divF[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      iso_grad<P>(sm[el][c], i, j, k, Di, Dj, Dk, a0, a1, a2);
#pragma unroll
      for (int b = 0; b < 3; ++b) gradQ[c][b] = He[b] * a0 + He[b + 3] * a1 + He[b + 6] * a2;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        iso_grad<P>(sm[el][3 + a * 3 + b], i, j, k, Di, Dj, Dk, a0, a1, a2);
        divF[a] += He[b] * a0 + He[b + 3] * a1 + He[b + 6] * a2;
      }
    const float divU = gradQ[0][0] + gradQ[1][1] + gradQ[2][2];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float r = 0.5f * (divF[a] + ul[a] * divU);
#pragma unroll
      for (int b = 0; b < 3; ++b) r = r + 0.5f * (ul[b] * gradQ[a][b]);
      out[a] = gv * r;
    }
  }
  if (MODE == 1)
    slots[pos] = out[0];
  else
    reinterpret_cast<float4 *>(slots)[pos] = make_float4(out[0], out[1], out[2], 0.f);
}

// ---- CG vector kernels (FP64 reductions, deterministic) ---------------
// Dot products over working nodes with FP64 accumulation, summed in a
// fixed order (deterministic).
constexpr int DOT_BLOCKS = 592;  // 4 blocks per SM on 148 SMs
constexpr int DOT_THREADS = 256;

// dot d = sum a[d]*(b[d] - c[d]) (c[d] may be null)
template <class V, int ND>
struct DotArgs {
  const V *a[ND];
  const V *b[ND];
  const V *c[ND];
};

// Single-block sum of DOT_BLOCKS partials per value, in a fixed order.
static __global__ void k_dot_final(int nd, const double *__restrict__ part, double *__restrict__ out) {
  __shared__ double sh[1024];
  for (int d = 0; d < nd; ++d) {
    double s = 0.0;
    for (int b = threadIdx.x; b < DOT_BLOCKS; b += blockDim.x) s += part[d * DOT_BLOCKS + b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
      if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[d] = sh[0];
    __syncthreads();
  }
}

// ND dot products in one launch: each block reduces its grid-stride share
// in a fixed order and stores a partial; the last block to take the ticket
// adds the partials in block order (deterministic) and resets the ticket.
template <class V, int ND>
__global__ void __launch_bounds__(DOT_THREADS) k_dot(int npoin_w, const int *__restrict__ lpoin_w,
                                                     DotArgs<V, ND> A, double *__restrict__ part,
                                                     unsigned *__restrict__ ticket, double *__restrict__ out) {
  __shared__ double sh[ND][DOT_THREADS];
  __shared__ bool last;
  double s[ND];
#pragma unroll
  for (int d = 0; d < ND; ++d) s[d] = 0.0;
  // grid-stride over the nodes; four strides per trip with every load issued
  // before the first product (same per-thread order as one stride per trip)
  const int stride = gridDim.x * blockDim.x;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  for (; t + 3 * stride < npoin_w; t += 4 * stride) {
    int p[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) p[u] = lpoin_w[t + u * stride];
    V av[4][ND], bv[4][ND];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        av[u][d] = A.a[d][p[u]];
        bv[u][d] = A.c[d] ? (V)(A.b[d][p[u]] - A.c[d][p[u]]) : A.b[d][p[u]];
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int d = 0; d < ND; ++d) s[d] += (double)(av[u][d] * bv[u][d]);
  }
  for (; t < npoin_w; t += stride) {
    const int p = lpoin_w[t];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const V bb = A.c[d] ? (V)(A.b[d][p] - A.c[d][p]) : A.b[d][p];
      s[d] += (double)(A.a[d][p] * bb);
    }
  }
#pragma unroll
  for (int d = 0; d < ND; ++d) sh[d][threadIdx.x] = s[d];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
#pragma unroll
      for (int d = 0; d < ND; ++d) sh[d][threadIdx.x] += sh[d][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int d = 0; d < ND; ++d) part[d * gridDim.x + blockIdx.x] = sh[d][0];
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v += __ldcg(part + d * gridDim.x + b);
    sh[d][threadIdx.x] = v;
  }
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
#pragma unroll
      for (int d = 0; d < ND; ++d) sh[d][threadIdx.x] += sh[d][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int d = 0; d < ND; ++d) out[d] = sh[d][0];
    *ticket = 0u;
  }
}

// ---- device-resident preconditioned CG -------------------------------------
// Scalars of the iteration kept in device memory between launches, so that
// the host only reads them once per batch of iterations.  The iteration
// kernels write nothing when status != 0 (what they still load: ended_late).
struct CgScal {
  double rz;     // r . z of the current residual
  double pq;     // p . A p
  double alpha, beta;
  double rr;     // ||r||^2 after the last update
  double thr2;   // (tol ||b||)^2; in the FP32 solve tol ||b||
  double bnorm;  // ||b|| of the FP32 solve
  int iter;      // iterations done in this solve
  int status;    // 0 running, 1 converged (recursive residual), 2 breakdown, 3 non-finite
};

// threads per block; nodes per thread of the update and assembly kernels
constexpr int CG_THREADS = 256, CG_U = 4, CG_QU = 2;
constexpr unsigned CG_WAVE = 148 * 4;  // see ended_late

// Node loops of the CG kernels handle several nodes per thread and issue all
// their loads before any store, so that each thread keeps several memory
// round trips in flight.
inline unsigned cg_blocks(long long n, int u) {
  const long long b = (n + (long long)CG_THREADS * u - 1) / ((long long)CG_THREADS * u);
  return (unsigned)(b < 1 ? 1 : b);
}

// Deterministic grid-wide sum of ND doubles: each block reduces its values
// in a fixed order and stores one partial; the last block to take a ticket
// adds the partials in block order.  Returns true (in every thread of that
// block only) with tot filled; the ticket is reset for the next launch.
template <int ND>
__device__ bool grid_sum(double (&v)[ND], double *__restrict__ part, unsigned *ticket, double (&tot)[ND]) {
  __shared__ double sh[ND][32];
  __shared__ bool last;
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, nw = blockDim.x / 32;
#pragma unroll
  for (int d = 0; d < ND; ++d)
    for (int o = 16; o > 0; o >>= 1) v[d] += __shfl_xor_sync(0xffffffffu, v[d], o);
  if (lane == 0)
#pragma unroll
    for (int d = 0; d < ND; ++d) sh[d][warp] = v[d];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      double s = 0.0;
      for (int w = 0; w < nw; ++w) s += sh[d][w];
      part[d * gridDim.x + blockIdx.x] = s;
    }
    // releases this block's partials, acquires the others'
    unsigned got;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;\n" : "=r"(got) : "l"(ticket) : "memory");
    last = got == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  // Eight partials of every value are requested before the first is added:
  // this block is alone on the GPU here, and one load at a time made the
  // tail of each sum grow by 0.6 us per load.
  constexpr int LD = 8;
  double s[ND];
#pragma unroll
  for (int d = 0; d < ND; ++d) s[d] = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += LD * blockDim.x) {
    double t[ND][LD];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int k = 0; k < LD; ++k) {
        const int bb = b + k * (int)blockDim.x;
        t[d][k] = bb < (int)gridDim.x ? __ldcg(part + d * gridDim.x + bb) : 0.0;
      }
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int k = 0; k < LD; ++k) s[d] += t[d][k];
  }
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    for (int o = 16; o > 0; o >>= 1) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
    if (lane == 0) sh[d][warp] = s[d];
  }
  __syncthreads();
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += sh[d][w];
    tot[d] = t;
  }
  if (threadIdx.x == 0) *ticket = 0u;
  return true;
}

// q = assembled Laplacian slots (Kahan, as k_gather_sorted1; written by
// k_lap_elem<DIR>) with the p.q partials; the last block sets alpha = rz / pq.
// The new search direction p = z + beta p is formed and stored here for every
// node with slots (the working nodes).  V = float: the reference's FP32
// solve, whose alpha is rounded to FP32 and taken as it comes.
template <class V>
__global__ void __launch_bounds__(CG_THREADS)
k_cg_q(MeshDev m, const V *__restrict__ slots, V *__restrict__ p, V *__restrict__ q, CgScal *S,
       double *__restrict__ part, unsigned *ticket, const V *__restrict__ z) {
  if (ended_late(&S->status, CG_WAVE)) return;
  constexpr int U = CG_QU, MS = 8;  // nodes per thread, slots loaded ahead per node
  const long long base = (long long)blockIdx.x * blockDim.x * U + threadIdx.x;
  int b[U], en[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long n = base + (long long)u * blockDim.x;
    b[u] = en[u] = 0;
    if (n < m.npoin) { b[u] = m.slot_ptr[n]; en[u] = m.slot_ptr[n + 1]; }
  }
  pdl_wait();
  pdl_trigger();
  // every load of the usual case (at most MS slots a node) in flight before
  // the status is looked at
  const int status = S->status;
  const V bt = (V)S->beta;
  double v[1] = {0.0};
  V pn[U], zn[U], y[U][MS];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long n = base + (long long)u * blockDim.x;
    pn[u] = zn[u] = 0;
    if (b[u] != en[u]) { pn[u] = p[n]; zn[u] = z[n]; }
#pragma unroll
    for (int k = 0; k < MS; ++k) y[u][k] = b[u] + k < en[u] ? slots[b[u] + k] : (V)0;
  }
  if (status) return;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long n = base + (long long)u * blockDim.x;
    V sum = 0, cmp = 0;
    for (int s0 = b[u]; s0 < en[u]; s0 += MS) {
      if (s0 != b[u])
#pragma unroll
        for (int k = 0; k < MS; ++k) y[u][k] = s0 + k < en[u] ? slots[s0 + k] : (V)0;
#pragma unroll
      for (int k = 0; k < MS; ++k) {
        if (s0 + k >= en[u]) break;
        const V yy = y[u][k] - cmp;
        const V tt = sum + yy;
        cmp = (tt - sum) - yy;
        sum = tt;
      }
    }
    if (b[u] != en[u]) {
      pn[u] = zn[u] + bt * pn[u];
      p[n] = pn[u];
      q[n] = sum;
      v[0] += (double)(pn[u] * sum);
    }
  }
  double tot[1];
  if (grid_sum<1>(v, part, ticket, tot) && threadIdx.x == 0) {
    S->pq = tot[0];
    if (sizeof(V) == 4) {
      S->alpha = (double)(float)(S->rz / tot[0]);
    } else if (!isfinite(tot[0])) {
      S->status = 3;
    } else if (!(tot[0] > 0.0)) {
      S->status = 2;
    } else {
      S->alpha = S->rz / tot[0];
    }
  }
}

// x += alpha p ; r -= alpha q ; with JAC also z = Minv r (the old z is Minv
// times the old r again), otherwise uf = (float)(Minv r) with Minv = D^-1/2;
// the last block records ||r||^2, detects convergence and, with JAC, sets
// the Polak-Ribiere beta = r.(z - z_old) / rz_old.  Runs over all nodes in
// order, with no index loads: Minv is 0 off the working nodes, which are
// left alone.  Minv (or D^-1/2) is read before the wait: k_cg_q, which comes
// before this kernel, does not write it.
template <bool JAC>
__global__ void __launch_bounds__(CG_THREADS)
k_cg_update(long long npoin, const double *__restrict__ p, const double *__restrict__ q,
            const double *__restrict__ Minv, double *__restrict__ x, double *__restrict__ r, double *__restrict__ z,
            CgScal *S, double *__restrict__ hist, int hist_cap, double *__restrict__ part, unsigned *ticket,
            float *__restrict__ uf) {
  if (ended_late(&S->status, CG_WAVE)) return;
  constexpr int U = CG_U;
  const long long base = (long long)blockIdx.x * blockDim.x * U + threadIdx.x;
  double mv[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    mv[u] = i < npoin ? Minv[i] : 0.0;
  }
  pdl_wait();
  pdl_trigger();
  const int status = S->status;
  const double a = S->alpha;
  double v[3] = {0.0, 0.0, 0.0};
  double pv[U], qv[U], xv[U], rv[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    if (i < npoin) { pv[u] = p[i]; qv[u] = q[i]; xv[u] = x[i]; rv[u] = r[i]; }
  }
  if (status) return;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    if (mv[u] == 0.0) continue;
    x[i] = xv[u] + a * pv[u];
    const double rn = rv[u] - a * qv[u];
    r[i] = rn;
    v[0] += rn * rn;
    if (JAC) {
      const double zn = rn * mv[u];
      z[i] = zn;
      v[1] += rn * zn;
      v[2] += rn * (rv[u] * mv[u]);
    } else {
      uf[i] = (float)(mv[u] * rn);  // D^-1/2 r for the learned preconditioner
    }
  }
  double tot[3];
  if (grid_sum<3>(v, part, ticket, tot) && threadIdx.x == 0) {
    const int it = S->iter + 1;
    S->iter = it;
    S->rr = tot[0];
    hist[(it - 1) % hist_cap] = tot[0];
    if (!isfinite(tot[0])) {
      S->status = 3;
    } else if (tot[0] < S->thr2) {
      S->status = 1;
    }
    if (JAC) {
      S->beta = (tot[1] - tot[2]) / S->rz;
      S->rz = tot[1];
    }
  }
}

// The same update of the reference's FP32 solve (mod_solver_incomp.f90:
// 395-440): z = r / M with M the Laplacian's diagonal (0 off the working
// nodes), FP64 sums of FP32 products, beta rounded to FP32, converged when
// ||r|| < thr2 (here tol ||b||).  M is read before the wait: k_cg_q does not
// write it.
static __global__ void __launch_bounds__(CG_THREADS)
k_cg_update32(long long npoin, const float *__restrict__ p, const float *__restrict__ q, const float *__restrict__ M,
              float *__restrict__ x, float *__restrict__ r, float *__restrict__ z, CgScal *S,
              double *__restrict__ part, unsigned *ticket) {
  if (ended_late(&S->status, CG_WAVE)) return;
  constexpr int U = CG_U;
  const long long base = (long long)blockIdx.x * blockDim.x * U + threadIdx.x;
  float mv[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    mv[u] = i < npoin ? M[i] : 0.f;
  }
  pdl_wait();
  pdl_trigger();
  const int status = S->status;
  const float a = (float)S->alpha;
  double v[3] = {0.0, 0.0, 0.0};
  float pv[U], qv[U], xv[U], rv[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    if (mv[u] != 0.f) { pv[u] = p[i]; qv[u] = q[i]; xv[u] = x[i]; rv[u] = r[i]; }
  }
  if (status) return;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    if (mv[u] == 0.f) continue;
    x[i] = xv[u] + a * pv[u];
    const float rn = rv[u] - a * qv[u], zn = rn / mv[u], zo = rv[u] / mv[u];
    r[i] = rn;
    z[i] = zn;
    v[0] += (double)(rn * rn);
    v[1] += (double)(rn * zn);
    v[2] += (double)(rn * (zn - zo));
  }
  double tot[3];
  if (grid_sum<3>(v, part, ticket, tot) && threadIdx.x == 0) {
    S->iter += 1;
    S->rr = tot[0];
    if (!isfinite(tot[0])) {
      S->status = 3;
    } else if (sqrt(tot[0]) < S->thr2) {
      S->status = 1;
    }
    S->beta = (double)(float)(tot[2] / S->rz);
    S->rz = tot[1];
  }
}

// Start of that solve: r = R - A x0 (Ax0 in q), z = r / M, x = p = 0 on
// every node; the last block sets the scalars.
static __global__ void __launch_bounds__(CG_THREADS)
k_cg_start32(long long npoin, const float *__restrict__ R, const float *__restrict__ q, const float *__restrict__ M,
             double tol, float *__restrict__ x, float *__restrict__ r, float *__restrict__ p, float *__restrict__ z,
             CgScal *S, double *__restrict__ part, unsigned *ticket) {
  constexpr int U = CG_U;
  const long long base = (long long)blockIdx.x * blockDim.x * U + threadIdx.x;
  double v[2] = {0.0, 0.0};
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + (long long)u * blockDim.x;
    if (i >= npoin) continue;
    const float mv = M[i];
    const float rn = mv != 0.f ? R[i] - q[i] : 0.f, zn = mv != 0.f ? rn / mv : 0.f;
    x[i] = 0.f;
    p[i] = 0.f;
    r[i] = rn;
    z[i] = zn;
    v[0] += (double)(rn * rn);
    v[1] += (double)(rn * zn);
  }
  double tot[2];
  if (grid_sum<2>(v, part, ticket, tot) && threadIdx.x == 0) {
    S->rz = tot[1];
    S->rr = tot[0];
    S->bnorm = sqrt(tot[0]);
    S->thr2 = tol * S->bnorm;
    S->alpha = S->beta = 0.0;
    S->iter = S->status = 0;
  }
}

// Learned preconditioner: z(n) = D^-1/2(n) (exp(alpha) D^-1/2(n) r(n) + sum of
// the node's contributions, stored contiguously from pptr[n]) (as
// k_patch_gather_perm), with the partials r.z and r.z_old; the last block
// sets beta and rz.  D^-1/2 and the parameter are read before the wait:
// k_patch_apply_tc, which comes before this kernel, does not write them.
static __global__ void __launch_bounds__(CG_THREADS)
k_cg_patch_z(long long npoin, const int *__restrict__ pptr, const float *__restrict__ ctr,
             const double *__restrict__ r, const double *__restrict__ Dh, const float *__restrict__ prm, int o_alpha,
             double *__restrict__ z, CgScal *S, double *__restrict__ part, unsigned *ticket) {
  constexpr int U = CG_U;
  const long long base = (long long)blockIdx.x * blockDim.x * U + threadIdx.x;
  int b[U], en[U];
  double dv[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long n = base + (long long)u * blockDim.x;
    b[u] = en[u] = 0;
    dv[u] = 0.0;
    if (n < npoin) { b[u] = pptr[n]; en[u] = pptr[n + 1]; dv[u] = Dh[n]; }
  }
  const double gam = exp((double)prm[o_alpha]);
  pdl_wait();
  pdl_trigger();
  if (S->status) return;
  double v[2] = {0.0, 0.0}, rv[U], zo[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long n = base + (long long)u * blockDim.x;
    if (b[u] != en[u]) { rv[u] = r[n]; zo[u] = z[n]; }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (b[u] == en[u]) continue;
    const long long n = base + (long long)u * blockDim.x;
    double acc = 0.0;
    for (int s0 = b[u]; s0 < en[u]; s0 += 8) {
      float y[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) y[k] = s0 + k < en[u] ? ctr[s0 + k] : 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) acc += (double)y[k];
    }
    const double zn = dv[u] * (gam * dv[u] * rv[u] + acc);
    z[n] = zn;
    v[0] += rv[u] * zn;
    v[1] += rv[u] * zo[u];
  }
  double tot[2];
  if (grid_sum<2>(v, part, ticket, tot) && threadIdx.x == 0) {
    S->beta = (tot[0] - tot[1]) / S->rz;
    S->rz = tot[0];
    if (!isfinite(S->beta)) S->status = 3;
  }
}

// harvest snapshot of the iterate and residual (skipped once stopped)
static __global__ void k_cg_snapshot(int npoin_w, const int *__restrict__ lpoin_w, const double *__restrict__ x,
                              const double *__restrict__ r, double *__restrict__ xs, float *__restrict__ rs,
                              const CgScal *S) {
  if (S->status) return;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < npoin_w; t += gridDim.x * blockDim.x) {
    const int i = lpoin_w[t];
    xs[i] = x[i];
    rs[i] = (float)r[i];
  }
}

}  // namespace sod

