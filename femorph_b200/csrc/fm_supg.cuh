// SUPG quasi-compressible element arithmetic, matrix-free (one thread = one
// element).
//
// Reference: src/femSUPGExplicitFluidSolver.cpp:1095-1498.  Per Gauss point
// the reference builds L, U, S, US, B, D, DB, H and accumulates five 24x24
// matrices (Mass, K1, K1+, K2, K3, K4), then forms k = -dt (K1+K2+K3+K4) u_e.
// Here each K_i u_e is evaluated directly from the Gauss-point quantities:
//   (K1 u)[a][c] += rho N_a (u.grad) u_c w                    (Bubnov convection)
//   (K2 u)[a][c] += sum_r B[r][a,c] (D(lambda, mu) B u)_r w   (viscous + penalty)
//   (K3 u)[a][c] += rho tau (u.grad N_a) (u.grad) u_c w       (SUPG)
//   (K4 u)[a][c] += rho nu_C dN_a/dx_c (div u) w              (grad-div)
// with w = detJ * weight, tau and nu_C from eval_stabilization (src lines
// 336-377) and lambda from eval_bulk_modulus (src lines 382-441).  The Mass
// and K1+ matrices do not reach the update (src lines 1325-1327, 806) and the
// Frobenius norms of K are diagnostics; none of them is formed.
#pragma once
#include "fm_device.cuh"

namespace fm {

// irSecondOrder rule (src/femIntegrationRule.cpp): tet4 4 points, weight
// (1/6)(1/4); hexa8 2x2x2 points at +-1/sqrt(3) in the reference's order,
// weight 1.
template <int NPE>
struct GaussRule;
template <>
struct GaussRule<4> {
  static constexpr int n = 4;
  __device__ static void point(int g, double q[3]) {
    const double a = 0.58541020, b = 0.13819660;
    q[0] = (g == 0) ? a : b;
    q[1] = (g == 1) ? a : b;
    q[2] = (g == 2) ? a : b;
  }
  __device__ static double weight() { return (1.0 / 6.0) * (1.0 / 4.0); }
};
template <>
struct GaussRule<8> {
  static constexpr int n = 8;
  __device__ static void point(int g, double q[3]) {
    const double s = 0.57735026918962573;  // 1/sqrt(3), correctly rounded
    const double sx[8] = {-s, s, s, -s, -s, s, s, -s};
    const double sy[8] = {-s, -s, s, s, -s, -s, s, s};
    const double sz[8] = {s, s, s, s, -s, -s, -s, -s};
    q[0] = sx[g];
    q[1] = sy[g];
    q[2] = sz[g];
  }
  __device__ static double weight() { return 8.0 * (1.0 / 8.0); }
};

// Shape functions and local derivatives (femTetra4.cpp:295-330,
// femHexa8.cpp:13-42).
template <int NPE>
__device__ __forceinline__ void shape(const double q[3], double N[NPE], double dN[NPE][3]) {
  if (NPE == 4) {
    N[0] = q[0]; N[1] = q[1]; N[2] = q[2]; N[3] = 1.0 - q[0] - q[1] - q[2];
    dN[0][0] = 1.0; dN[0][1] = 0.0; dN[0][2] = 0.0;
    dN[1][0] = 0.0; dN[1][1] = 1.0; dN[1][2] = 0.0;
    dN[2][0] = 0.0; dN[2][1] = 0.0; dN[2][2] = 1.0;
    dN[3][0] = -1.0; dN[3][1] = -1.0; dN[3][2] = -1.0;
  } else {
    const double c1[8] = {-1.0, 1.0, 1.0, -1.0, -1.0, 1.0, 1.0, -1.0};
    const double c2[8] = {-1.0, -1.0, 1.0, 1.0, -1.0, -1.0, 1.0, 1.0};
    const double c3[8] = {-1.0, -1.0, -1.0, -1.0, 1.0, 1.0, 1.0, 1.0};
#pragma unroll
    for (int a = 0; a < NPE; ++a) {
      const double fx = 1.0 + q[0] * c1[a], fy = 1.0 + q[1] * c2[a], fz = 1.0 + q[2] * c3[a];
      N[a] = 0.125 * fx * fy * fz;
      dN[a][0] = 0.125 * c1[a] * fy * fz;
      dN[a][1] = 0.125 * c2[a] * fx * fz;
      dN[a][2] = 0.125 * c3[a] * fx * fy;
    }
  }
}

// Shape values and local derivatives at the Gauss points, tabulated once per
// CTA in shared memory with the same expressions as shape<NPE> (identical
// values); the Gauss-point loops read them at warp-uniform addresses.
template <int NPE, typename T>
struct ShapeTable {
  T N[GaussRule<NPE>::n][NPE];
  T dN[GaussRule<NPE>::n][NPE][3];
};

template <int NPE, typename T>
__device__ __forceinline__ void fill_shape_table(ShapeTable<NPE, T>* t) {
  for (int g = threadIdx.x; g < GaussRule<NPE>::n; g += blockDim.x) {
    double q[3], Nf[NPE], dN[NPE][3];
    GaussRule<NPE>::point(g, q);
    shape<NPE>(q, Nf, dN);
#pragma unroll
    for (int a = 0; a < NPE; ++a) {
      t->N[g][a] = (T)Nf[a];
#pragma unroll
      for (int c = 0; c < 3; ++c) t->dN[g][a][c] = (T)dN[a][c];
    }
  }
}

// Jacobian J[a][b] = sum_n dN[n][a] x[n][b] (femElement.cpp:104-127), its
// cofactor inverse (femUtils.cpp:716-770), global derivatives
// gd[n][b] = sum_c inv[b][c] dN[n][c] (femElement.cpp:345-352) and the
// geometric matrix G[a][b] = sum_c inv[c][a] inv[c][b] (femElement.cpp:222-230).
// The local derivatives are read through dN(n, a): a register array, or a
// shared-memory table read where used.
template <int NPE, class DN>
__device__ __forceinline__ double jacobian_at(DN dN, const double* sx, const double* sy, const double* sz, const int ln[NPE],
                                              double inv[3][3]) {
  double J[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double j0 = 0.0, j1 = 0.0, j2 = 0.0;
#pragma unroll
    for (int n = 0; n < NPE; ++n) {
      const double d = dN(n, a);
      j0 += d * sx[ln[n]];
      j1 += d * sy[ln[n]];
      j2 += d * sz[ln[n]];
    }
    J[a][0] = j0; J[a][1] = j1; J[a][2] = j2;
  }
  const double m00 = J[0][0], m01 = J[0][1], m02 = J[0][2], m10 = J[1][0], m11 = J[1][1], m12 = J[1][2], m20 = J[2][0],
               m21 = J[2][1], m22 = J[2][2];
  const double det = m00 * (m11 * m22 - m21 * m12) - m01 * (m10 * m22 - m12 * m20) + m02 * (m10 * m21 - m11 * m20);
  const double id = 1.0 / det;
  inv[0][0] = (m11 * m22 - m21 * m12) * id;
  inv[0][1] = (m02 * m21 - m01 * m22) * id;
  inv[0][2] = (m01 * m12 - m02 * m11) * id;
  inv[1][0] = (m12 * m20 - m10 * m22) * id;
  inv[1][1] = (m00 * m22 - m02 * m20) * id;
  inv[1][2] = (m10 * m02 - m00 * m12) * id;
  inv[2][0] = (m10 * m21 - m20 * m11) * id;
  inv[2][1] = (m20 * m01 - m00 * m21) * id;
  inv[2][2] = (m00 * m11 - m10 * m01) * id;
  return det;
}

template <int NPE>
__device__ __forceinline__ double jacobian(const double dN[NPE][3], const double* sx, const double* sy, const double* sz,
                                           const int ln[NPE], double inv[3][3]) {
  return jacobian_at<NPE>([&](int n, int a) { return dN[n][a]; }, sx, sy, sz, ln, inv);
}

// Gauss-point geometry of one hexa8 element, formed once per placement and
// kept in HBM: per point g the inverse Jacobian (9 entries) and det J, entry
// q of point g at geo[(g * FM_GEO_PER_GP + q) * E + e] (coalesced over the
// tile's consecutive element slots).  The mesh does not move, so these are
// the values the element loop would form at every step from the same
// coordinates with the same expressions.
//
// The element loop streams it through shared memory: thread tid's rows of ten
// values sit in a column of NB rows (stride THREADS) that the thread fills
// for itself with asynchronous copies, NB - 1 points ahead, so neither a
// register nor a barrier is spent on the look-ahead.  (Asking L1 for the rows
// two points ahead and reading them there lost most of them again before
// their use: 12 warps x 3 points x 2.5 KB do not fit beside the tiles' shared
// memory; FP64 channel of 1 M hexa 0.438 -> 0.377 ms a step.)  PAIRED: the
// points once in hexa_point's order, else 0..7, `passes` times round (B-bar:
// n = 8..15 are points 0..7 again).
__device__ __forceinline__ int hexa_point(int n) { return (n & ~1) + ((n & 1) ^ ((n >> 1) & 1) ^ 1); }
__device__ __forceinline__ void copy_async(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
template <typename T, int THREADS, int NB, bool PAIRED>
struct GeoStream {
  T* column;
  const T* geo;  // the element's first value
  int64_t E;
  int passes;    // times round the points (PAIRED: once)
  // starts the copy of the n-th point; one group a call, also an empty one
  __device__ __forceinline__ void copy(int n) const {
    if (n < (PAIRED ? 8 : 8 * passes)) {
      const T* q = geo + (int64_t)(PAIRED ? hexa_point(n) : (n & 7)) * FM_GEO_PER_GP * E;
      T* d = column + (n & (NB - 1)) * FM_GEO_PER_GP * THREADS;
#pragma unroll
      for (int k = 0; k < FM_GEO_PER_GP; ++k) copy_async(d + k * THREADS, q + k * E);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // the copies an element's first row() expects to be on their way
  __device__ __forceinline__ void start() const {
#pragma unroll
    for (int n = 0; n < NB - 1; ++n) copy(n);
  }
  // the n-th point's inverse Jacobian; returns its determinant.  n = 0, 1, ...
  // in turn after start()
  __device__ __forceinline__ T row(int n, T inv[3][3]) const {
    copy(n + NB - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(NB - 1) : "memory");
    const T* d = column + (n & (NB - 1)) * FM_GEO_PER_GP * THREADS;
#pragma unroll
    for (int i = 0; i < 9; ++i) inv[i / 3][i % 3] = d[i * THREADS];
    return d[9 * THREADS];
  }
  // the same straight from memory (the FP64 form's B-bar passes: keeping the
  // stream going through them too cost the main loop 100 bytes of spill)
  __device__ __forceinline__ T load(int n, T inv[3][3]) const {
    const T* q = geo + (int64_t)(PAIRED ? hexa_point(n) : n) * FM_GEO_PER_GP * E;
#pragma unroll
    for (int i = 0; i < 9; ++i) inv[i / 3][i % 3] = __ldg(q + i * E);
    return __ldg(q + 9 * E);
  }
};
// Rows of the column: FP64 two (a third costs the third CTA an SM: 0.565
// instead of 0.377 ms), FP32 four (two 0.0729, four 0.0724 ms a step on the
// 93x37x29 AB2 + B-bar channel; read from L1 0.0767).
constexpr int FM_GEO_ROWS64 = 2, FM_GEO_ROWS32 = 4;
template <int THREADS>
using GeoStream64 = GeoStream<double, THREADS, FM_GEO_ROWS64, true>;
template <int THREADS>
using GeoStream32 = GeoStream<float, THREADS, FM_GEO_ROWS32, false>;

// Doubles of the tile kernels' per-thread region (hexa8): FP64 the 24 velocity
// coefficients and the geometry rows, mixed its geometry rows.
__host__ __device__ constexpr size_t supg_stage_doubles(int npe, bool mixed, int threads) {
  return npe == 4 ? 0
                  : (size_t)threads * (mixed ? FM_GEO_ROWS32 * FM_GEO_PER_GP / 2 : 24 + FM_GEO_ROWS64 * FM_GEO_PER_GP);
}
// Sets of accumulators (rings of warps).
__host__ __device__ constexpr int supg_acc_sets(int npe, bool mixed) { return npe == 4 && !mixed ? 2 : 1; }

// Inverse (cofactors, femUtils.cpp:716-770) and determinant of a 3x3 matrix.
__device__ __forceinline__ double inverse3(const double J[3][3], double inv[3][3]) {
  const double c0 = J[1][1] * J[2][2] - J[2][1] * J[1][2], c1 = J[1][2] * J[2][0] - J[1][0] * J[2][2],
               c2 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
  const double det = J[0][0] * c0 + J[0][1] * c1 + J[0][2] * c2;
  const double id = 1.0 / det;
  inv[0][0] = c0 * id;
  inv[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * id;
  inv[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * id;
  inv[1][0] = c1 * id;
  inv[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * id;
  inv[1][2] = (J[1][0] * J[0][2] - J[0][0] * J[1][2]) * id;
  inv[2][0] = c2 * id;
  inv[2][1] = (J[2][0] * J[0][1] - J[0][0] * J[2][1]) * id;
  inv[2][2] = (J[0][0] * J[1][1] - J[1][0] * J[0][1]) * id;
  return det;
}

// Signed sums of eight corner values (femHexa8.cpp:13-42 corner order) that
// give 8 x the coefficients of {1, x, y, z, xy, yz, xz, xyz}, and the
// transposed sums, node a taking sum_m sign_m(a) q[m]: 24 additions each.
__device__ __forceinline__ void hexa_to_modes(const double n[8], double m[8]) {
  const double a0 = n[1] + n[0], a1 = n[1] - n[0], b0 = n[2] + n[3], b1 = n[2] - n[3];
  const double e0 = n[5] + n[4], e1 = n[5] - n[4], f0 = n[6] + n[7], f1 = n[6] - n[7];
  const double p0 = b0 + a0, p2 = b0 - a0, p1 = b1 + a1, p4 = b1 - a1;
  const double q0 = f0 + e0, q2 = f0 - e0, q1 = f1 + e1, q4 = f1 - e1;
  m[0] = q0 + p0; m[3] = q0 - p0;
  m[2] = q2 + p2; m[5] = q2 - p2;
  m[1] = q1 + p1; m[6] = q1 - p1;
  m[4] = q4 + p4; m[7] = q4 - p4;
}
__device__ __forceinline__ void hexa_to_nodes(const double q[8], double n[8]) {
  const double zp0 = q[0] + q[3], zm0 = q[0] - q[3], zp2 = q[2] + q[5], zm2 = q[2] - q[5];
  const double zp1 = q[1] + q[6], zm1 = q[1] - q[6], zp4 = q[4] + q[7], zm4 = q[4] - q[7];
  const double a = zm0 - zm2, b = zm0 + zm2, c = zp0 - zp2, d = zp0 + zp2;      // even in x: y-z-, y+z-, y-z+, y+z+
  const double A = zm1 - zm4, Bx = zm1 + zm4, Cx = zp1 - zp4, D = zp1 + zp4;    // odd in x
  n[0] = a - A; n[1] = a + A;
  n[3] = b - Bx; n[2] = b + Bx;
  n[4] = c - Cx; n[5] = c + Cx;
  n[7] = d - D; n[6] = d + D;
}

// One tet4 element: k[a][c] = -dt (sum of the enabled K_i u_e)[a][c], its
// lambda (volume average) and regime (average of the Gauss-point regimes).
// The Jacobian, the velocity gradient, the metric G = J^-T J^-1, the shear
// part of the stress and the weight w are element constants, and with
// lN_a(g) = ALPHA (a = g) or BETA the velocity at the points is
// BETA sum_a u_a + (ALPHA - BETA) u_g; so only u_g, tau, nu_C, lambda and the
// convection (u_g . grad) u are formed per point, and the points enter the
// forces through sums,
//   k_a[c] = -dt w ( sum_d gd_a[d] T[c][d] + rho (BETA sum_g conv_g + (ALPHA - BETA) conv_a)[c] ),
//   T[c][d] = stress_cd (with sum_g lambda) + rho div sum_g nu_C delta_cd + rho sum_g tau_g u_g[d] conv_g[c],
// with gd_3 = -(gd_0 + gd_1 + gd_2).  u^T G^-1 u = |J^T u|^2 needs no inverse
// of G.  FP64 instructions are what bounds the tile kernel here (fixed
// latency chains at 12 warps an SM), so their number is what counts.
__device__ __forceinline__ void supg_element_tet(const DevProb& P, const double* sx, const double* sy, const double* sz,
                                                 const double* su, const double* sv, const double* sw, const int ln[4],
                                                 double k[4][3], double& lam_el, double& reg_el) {
  const double rho = P.rho, mu = P.mu, alpha = P.alpha;
  const double nu = mu / rho;
  const bool iK1 = (P.ex_mask & 4) != 0, iK2 = (P.ex_mask & 8) != 0, iK3 = (P.ex_mask & 16) != 0,
             iK4 = (P.ex_mask & 32) != 0;
  constexpr double A = 0.58541020, Bt = 0.13819660, AB = A - Bt;
  double J[3][3];  // J[a][c] = x_a[c] - x_3[c]
  {
    const double x3 = sx[ln[3]], y3 = sy[ln[3]], z3 = sz[ln[3]];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      J[a][0] = sx[ln[a]] - x3;
      J[a][1] = sy[ln[a]] - y3;
      J[a][2] = sz[ln[a]] - z3;
    }
  }
  double inv[3][3];
  const double det = inverse3(J, inv);
  // G's entries (symmetric), its trace and the G:G term of tau
  const double g00 = inv[0][0] * inv[0][0] + inv[1][0] * inv[1][0] + inv[2][0] * inv[2][0];
  const double g11 = inv[0][1] * inv[0][1] + inv[1][1] * inv[1][1] + inv[2][1] * inv[2][1];
  const double g22 = inv[0][2] * inv[0][2] + inv[1][2] * inv[1][2] + inv[2][2] * inv[2][2];
  const double h01 = 2.0 * (inv[0][0] * inv[0][1] + inv[1][0] * inv[1][1] + inv[2][0] * inv[2][1]);
  const double h02 = 2.0 * (inv[0][0] * inv[0][2] + inv[1][0] * inv[1][2] + inv[2][0] * inv[2][2]);
  const double h12 = 2.0 * (inv[0][1] * inv[0][2] + inv[1][1] * inv[1][2] + inv[2][1] * inv[2][2]);
  const double irG = 1.0 / (g00 + g11 + g22);
  const double t3 = (g00 * g00 + g11 * g11 + g22 * g22 + 0.5 * (h01 * h01 + h02 * h02 + h12 * h12)) * nu * nu * P.c_i;
  double U[4][3], gr[3][3], Us[3];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    U[a][0] = su[ln[a]];
    U[a][1] = sv[ln[a]];
    U[a][2] = sw[ln[a]];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double d0 = U[0][c] - U[3][c], d1 = U[1][c] - U[3][c], d2 = U[2][c] - U[3][c];
#pragma unroll
    for (int d = 0; d < 3; ++d) gr[c][d] = inv[d][0] * d0 + inv[d][1] * d1 + inv[d][2] * d2;
    Us[c] = Bt * ((U[0][c] + U[1][c]) + (U[2][c] + U[3][c]));
  }
  const double div = gr[0][0] + gr[1][1] + gr[2][2];
  double M[3][3], cs[3] = {0.0, 0.0, 0.0}, Ls = 0.0, Ns = 0.0, reg = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) M[d][0] = M[d][1] = M[d][2] = 0.0;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    double u[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) u[c] = Us[c] + AB * U[g][c];
    // eval_stabilization (dt term removed in the reference): tau = q^-1/2,
    // nu_C = 1 / (tr G tau) = q^1/2 / tr G
    const double q = t3 + u[0] * (g00 * u[0] + h01 * u[1] + h02 * u[2]) + u[1] * (g11 * u[1] + h12 * u[2]) +
                     u[2] * (g22 * u[2]);
    const double tau = rsqrt_nr(q);
    Ns += (q == 0.0) ? 0.0 : q * tau;
    // eval_bulk_modulus: lambda = alpha * max(mu/rho, sqrt(u^T G^-1 u))
    const double v0 = J[0][0] * u[0] + J[1][0] * u[1] + J[2][0] * u[2];
    const double v1 = J[0][1] * u[0] + J[1][1] * u[1] + J[2][1] * u[2];
    const double v2 = J[0][2] * u[0] + J[1][2] * u[1] + J[2][2] * u[2];
    const double l2 = sqrt_nr(v0 * v0 + v1 * v1 + v2 * v2);
    Ls += (nu < l2) ? l2 : nu;  // std::max(limit_1, limit_2)
    reg += (nu > l2) ? 1.0 : 2.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double cv = u[0] * gr[c][0] + u[1] * gr[c][1] + u[2] * gr[c][2];
      k[g][c] = cv;
      cs[c] += cv;
      const double tc = tau * cv;
#pragma unroll
      for (int d = 0; d < 3; ++d) M[d][c] += u[d] * tc;
    }
  }
  Ls *= alpha;
  lam_el = 0.25 * Ls;
  reg_el = 0.25 * reg;
  const double w = -P.dt * (det * GaussRule<4>::weight());
  const double rw = rho * w;
  double T[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < 3; ++d) T[c][d] = iK3 ? rw * M[d][c] : 0.0;
  if (iK2) {
    const double n = w * (div * Ls), m4 = 4.0 * (w * mu), m8 = 2.0 * m4;
    const double s01 = m4 * (gr[0][1] + gr[1][0]), s12 = m4 * (gr[1][2] + gr[2][1]), s02 = m4 * (gr[0][2] + gr[2][0]);
#pragma unroll
    for (int c = 0; c < 3; ++c) T[c][c] += n + m8 * gr[c][c];
    T[0][1] += s01; T[1][0] += s01;
    T[1][2] += s12; T[2][1] += s12;
    T[0][2] += s02; T[2][0] += s02;
  }
  if (iK4) {
    const double n = rw * div * (Ns * irG);
#pragma unroll
    for (int c = 0; c < 3; ++c) T[c][c] += n;
  }
  const double c1 = iK1 ? rw * AB : 0.0, c0 = iK1 ? rw * Bt : 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double b = c0 * cs[c];
    double f3 = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double f = T[c][0] * inv[0][a] + T[c][1] * inv[1][a] + T[c][2] * inv[2][a];
      k[a][c] = f + (b + c1 * k[a][c]);
      f3 += f;
    }
    k[3][c] = (b + c1 * k[3][c]) - f3;
  }
}

// One hexa8 element, same outputs.  The trilinear field is held by its eight
// coefficients in {1, x, y, z, xy, yz, xz, xyz} (local coordinates; C below,
// scaled by the powers of s = 1/sqrt(3) that the points +-s bring), a few
// additions of the nodal values, so a point's velocity and local gradient
// are sums of coefficients with signs instead of sums over eight nodes of
// tabulated shape values (16 additions a component for the two points of a
// pair with the same y and z, against 64 products), and the forces are
// gathered into the same eight coefficients (K; 25 additions a component
// and pair against 64 products) and taken back to the nodes once at the end.
// Nothing is read from shared memory inside the loop.  Per point every force
// is one matrix and one vector on the test function:
//   k_a[c] += sum_j W[c][j] dN_a/dxi_j + b[c] N_a,
//   W = (S + c4w I) J^-1 + c3w conv (J^-T u)^T,  b = c1w conv,
// S the stress terms of K2, c4w I those of K4.  u^T G^-1 u = |J^T u|^2 with
// J^T = det J x cof(J^-1) applied through two cross products.  The point
// geometry comes from the stored one (GeoStream).
//
// B-bar (eval_avg_shapeDeriv, src lines 660-707, and the B matrix rows 0-2,
// src lines 234-256).  With sd0[a][c] = sum_g w_g gd_g[a][c] / V the
// volume-averaged derivatives, B1 = (sd0[a][0] - gd[a][0]) / 3, B2 =
// gd[a][0] - B1 and likewise B3/B4, B5/B6 for y and z, the sums over the
// nodes are
//   strain:  eps_c = gr_cc - 2 d_c + (d_0 + d_1 + d_2),
//            d_c = (Dbar_c - gr_cc) / 3,  Dbar_c = sum_a sd0[a][c] u_c(a)
//   force:   r_c(a) w = gd[a][c] (w sig_c - q_c) + sd0[a][c] q_c,
//            q_c = w (sig_0 + sig_1 + sig_2 - 2 sig_c) / 3,
// so sd0 enters only through the element constants Dbar_c = sum_g w_g
// gr_g[c][c] / V (a pass before the Gauss loop) and sd0[a][c] Q_c,
// Q_c = sum_g q_c (a pass after it).
// BBAR is a template parameter so that the other elements do not hold its six
// element constants.
template <int THREADS, bool BBAR>
__device__ __forceinline__ void supg_element_hexa(const DevProb& P, const double* su, const double* sv, const double* sw,
                                                  const int ln[8], double* coef, double k[8][3], double& lam_el,
                                                  double& reg_el, const GeoStream64<THREADS>& geo) {
  const double rho = P.rho, mu = P.mu, alpha = P.alpha;
  const double nu = mu / rho;
  const bool iK1 = (P.ex_mask & 4) != 0, iK2 = (P.ex_mask & 8) != 0, iK3 = (P.ex_mask & 16) != 0,
             iK4 = (P.ex_mask & 32) != 0;
  constexpr double s = 0.57735026918962573;  // 1/sqrt(3), correctly rounded
  double K[8][3];
  // C in the thread's own shared-memory column (stride THREADS): 48 registers
  // less, which is what lets three CTAs an SM run without spilling (0.496 ->
  // 0.438 ms a step for 1 M hexa)
  auto Cv = [&](int m, int c) -> double& { return coef[(m * 3 + c) * THREADS]; };
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double* q = c == 0 ? su : (c == 1 ? sv : sw);
    double n[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) n[a] = q[ln[a]];
    double m[8];
    hexa_to_modes(n, m);
    Cv(0, c) = 0.125 * m[0]; Cv(1, c) = 0.125 * m[1]; Cv(2, c) = 0.125 * m[2]; Cv(3, c) = 0.125 * m[3];
    Cv(4, c) = (0.125 * s) * m[4]; Cv(5, c) = (0.125 * s) * m[5]; Cv(6, c) = (0.125 * s) * m[6];
    Cv(7, c) = (0.125 * s * s) * m[7];
#pragma unroll
    for (int a = 0; a < 8; ++a) K[a][c] = 0.0;
  }
  // pair p: the points x = +s and x = -s at y = sy s, z = sz s
  auto sign_y = [](int p) -> double { return (p & 1) ? 1.0 : -1.0; };
  auto sign_z = [](int p) -> double { return (p & 2) ? -1.0 : 1.0; };
  double vol = 0.0, lam_int = 0.0, reg = 0.0;
  double Dbar[3] = {0.0, 0.0, 0.0}, Qb[3] = {0.0, 0.0, 0.0};
  if constexpr (BBAR) {
    double bden = 0.0;
#pragma unroll 1
    for (int p = 0; p < 4; ++p) {
      const double sy = sign_y(p), sz = sign_z(p), yz = sy * sz;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const double sx = h ? -1.0 : 1.0;
        double inv[3][3];
        const double w = geo.load(2 * p + h, inv);
        bden += w;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double l0 = Cv(1, c) + sy * Cv(4, c) + sz * Cv(6, c) + yz * Cv(7, c);
          const double l1 = Cv(2, c) + sx * Cv(4, c) + sz * Cv(5, c) + (sx * sz) * Cv(7, c);
          const double l2 = Cv(3, c) + sx * Cv(6, c) + sy * Cv(5, c) + (sx * sy) * Cv(7, c);
          Dbar[c] += w * (inv[c][0] * l0 + inv[c][1] * l1 + inv[c][2] * l2);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) Dbar[c] /= bden;
  }
  // one point: velocity u, local gradient L[c][j] -> W, b (see above)
  auto point = [&](int n, const double u[3], const double L[3][3], double W[3][3], double b[3]) {
    double inv[3][3];
    const double det = geo.row(n, inv);
    double gr[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int d = 0; d < 3; ++d) gr[c][d] = inv[d][0] * L[c][0] + inv[d][1] * L[c][1] + inv[d][2] * L[c][2];
    const double div = gr[0][0] + gr[1][1] + gr[2][2];
    // eval_stabilization (dt term removed in the reference): tau = q^-1/2,
    // nu_C = 1 / (tr G tau) = q^1/2 / tr G, u^T G u = |J^-1 u|^2
    double trG, q;
    {
      const double g00 = inv[0][0] * inv[0][0] + inv[1][0] * inv[1][0] + inv[2][0] * inv[2][0];
      const double g11 = inv[0][1] * inv[0][1] + inv[1][1] * inv[1][1] + inv[2][1] * inv[2][1];
      const double g22 = inv[0][2] * inv[0][2] + inv[1][2] * inv[1][2] + inv[2][2] * inv[2][2];
      const double g01 = inv[0][0] * inv[0][1] + inv[1][0] * inv[1][1] + inv[2][0] * inv[2][1];
      const double g02 = inv[0][0] * inv[0][2] + inv[1][0] * inv[1][2] + inv[2][0] * inv[2][2];
      const double g12 = inv[0][1] * inv[0][2] + inv[1][1] * inv[1][2] + inv[2][1] * inv[2][2];
      trG = g00 + g11 + g22;
      q = (g00 * g00 + g11 * g11 + g22 * g22 + 2.0 * (g01 * g01 + g02 * g02 + g12 * g12)) * nu * nu * P.c_i;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double t = inv[c][0] * u[0] + inv[c][1] * u[1] + inv[c][2] * u[2];
        q += t * t;
      }
    }
    const double tau = rsqrt_nr(q);
    const double nuC = ((q == 0.0) ? 0.0 : q * tau) * rcp_nr(trG);
    // eval_bulk_modulus: lambda = alpha * max(mu/rho, sqrt(u^T G^-1 u));
    // J^T u / det J = (u . (r1 x r2), u . (r2 x r0), u . (r0 x r1)), r_i the
    // rows of J^-1
    double lam;
    {
      const double a0 = u[1] * inv[0][2] - u[2] * inv[0][1], a1 = u[2] * inv[0][0] - u[0] * inv[0][2],
                   a2 = u[0] * inv[0][1] - u[1] * inv[0][0];  // u x r0
      const double b0 = u[1] * inv[1][2] - u[2] * inv[1][1], b1 = u[2] * inv[1][0] - u[0] * inv[1][2],
                   b2 = u[0] * inv[1][1] - u[1] * inv[1][0];  // u x r1
      const double v0 = inv[2][0] * b0 + inv[2][1] * b1 + inv[2][2] * b2;
      const double v1 = inv[2][0] * a0 + inv[2][1] * a1 + inv[2][2] * a2;  // sign dropped (squared)
      const double v2 = inv[1][0] * a0 + inv[1][1] * a1 + inv[1][2] * a2;
      const double l2 = fabs(det) * sqrt_nr(v0 * v0 + v1 * v1 + v2 * v2);
      lam = alpha * ((nu < l2) ? l2 : nu);  // std::max(limit_1, limit_2)
      reg += (nu > l2) ? 1.0 : 2.0;
    }
    const double w = det;  // quadrature weight 1
    vol += w;
    lam_int += lam * w;
    double S[3][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
    if (iK2) {
      const double mw = mu * w, m2 = 2.0 * mw;
      double e[3] = {gr[0][0], gr[1][1], gr[2][2]}, tr = div;
      if constexpr (BBAR) {
        const double d0 = (1.0 / 3.0) * (Dbar[0] - e[0]), d1 = (1.0 / 3.0) * (Dbar[1] - e[1]),
                     d2 = (1.0 / 3.0) * (Dbar[2] - e[2]);
        const double t = d0 + d1 + d2;
        e[0] += t - 2.0 * d0;
        e[1] += t - 2.0 * d1;
        e[2] += t - 2.0 * d2;
        tr = e[0] + e[1] + e[2];
      }
      const double lt = lam * w * tr;
#pragma unroll
      for (int c = 0; c < 3; ++c) S[c][c] = lt + m2 * e[c];
      if constexpr (BBAR) {
        const double st = S[0][0] + S[1][1] + S[2][2];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double qc = (1.0 / 3.0) * (st - 2.0 * S[c][c]);
          Qb[c] += qc;
          S[c][c] -= qc;
        }
      }
      S[0][1] = S[1][0] = mw * (gr[0][1] + gr[1][0]);
      S[1][2] = S[2][1] = mw * (gr[1][2] + gr[2][1]);
      S[0][2] = S[2][0] = mw * (gr[0][2] + gr[2][0]);
    }
    if (iK4) {
      const double c4w = rho * nuC * div * w;
#pragma unroll
      for (int c = 0; c < 3; ++c) S[c][c] += c4w;
    }
    const double c1w = iK1 ? rho * w : 0.0, c3w = iK3 ? rho * tau * w : 0.0;
    double ut[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) ut[j] = u[0] * inv[0][j] + u[1] * inv[1][j] + u[2] * inv[2][j];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double cv = u[0] * gr[c][0] + u[1] * gr[c][1] + u[2] * gr[c][2];
      b[c] = c1w * cv;
      const double c3 = c3w * cv;
#pragma unroll
      for (int j = 0; j < 3; ++j)
        W[c][j] = c3 * ut[j] + (S[c][0] * inv[0][j] + S[c][1] * inv[1][j] + S[c][2] * inv[2][j]);
    }
  };
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    const double sy = sign_y(p), sz = sign_z(p), yz = sy * sz;
    double Wp[3][3], Wm[3][3], bp[3], bm[3];
    {
      double up[3], um[3], Lp[3][3], Lm[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double B0 = Cv(2, c) + sz * Cv(5, c), B1 = Cv(4, c) + sz * Cv(7, c);
        const double D0 = Cv(3, c) + sy * Cv(5, c), D1 = Cv(6, c) + sy * Cv(7, c);
        const double A1 = Cv(1, c) + sz * Cv(6, c) + sy * B1;
        const double Ev = sy * B0 + sz * Cv(3, c);
        up[c] = Cv(0, c) + s * (Ev + A1);
        um[c] = Cv(0, c) + s * (Ev - A1);
        Lp[c][0] = A1; Lp[c][1] = B0 + B1; Lp[c][2] = D0 + D1;
        Lm[c][0] = A1; Lm[c][1] = B0 - B1; Lm[c][2] = D0 - D1;
      }
      point(2 * p, up, Lp, Wp, bp);
      point(2 * p + 1, um, Lm, Wm, bm);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double bs = s * (bp[c] + bm[c]);
      const double Q = (Wp[c][0] + Wm[c][0]) + s * (bp[c] - bm[c]);
      const double es = Wp[c][1] + Wm[c][1], ed = Wp[c][1] - Wm[c][1];
      const double zs = Wp[c][2] + Wm[c][2], zd = Wp[c][2] - Wm[c][2];
      K[0][c] += bs;  // x 1/s at the end
      K[1][c] += Q;
      K[2][c] += es + sy * bs;
      K[3][c] += zs + sz * bs;
      K[4][c] += sy * Q + ed;                       // x s
      K[5][c] += sz * es + (sy * zs + yz * bs);     // x s
      K[6][c] += sz * Q + zd;                       // x s
      K[7][c] += yz * Q + (sz * ed + sy * zd);      // x s^2
    }
  }
  if (BBAR && iK2) {
    // k_a[c] += sd0[a][c] Q_c, sd0 formed again point by point
#pragma unroll
    for (int c = 0; c < 3; ++c) Qb[c] /= vol;
#pragma unroll 1
    for (int p = 0; p < 4; ++p) {
      const double sy = sign_y(p), sz = sign_z(p), yz = sy * sz;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const double sx = h ? -1.0 : 1.0;
        double inv[3][3];
        const double w = geo.load(2 * p + h, inv);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double f = w * Qb[c];
          const double w0 = f * inv[c][0], w1 = f * inv[c][1], w2 = f * inv[c][2];
          K[1][c] += w0;
          K[2][c] += w1;
          K[3][c] += w2;
          K[4][c] += sy * w0 + sx * w1;
          K[5][c] += sz * w1 + sy * w2;
          K[6][c] += sz * w0 + sx * w2;
          K[7][c] += yz * w0 + ((sx * sz) * w1 + (sx * sy) * w2);
        }
      }
    }
  }
  const double m = -0.125 * P.dt;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double q[8] = {(m / s) * K[0][c], m * K[1][c], m * K[2][c], m * K[3][c],
                         (m * s) * K[4][c], (m * s) * K[5][c], (m * s) * K[6][c], (m * s * s) * K[7][c]};
    double n[8];
    hexa_to_nodes(q, n);
#pragma unroll
    for (int a = 0; a < 8; ++a) k[a][c] = n[a];
  }
  lam_el = lam_int / vol;
  reg_el = reg / 8.0;
}

}  // namespace fm

namespace fm {

// ---------------------------------------------------------------------------
// Mixed precision SUPG element (FM_MIXED): the Gauss-point work in FP32,
// k = -dt K u_e converted to FP64 for the nodal accumulation, the AB2 history
// and the update, which stay FP64.  Coordinates and velocities enter FP32 as
// differences to the element's node 0, formed in FP64 (Xr, Ud; Xr[0] = Ud[0]
// = 0), so the Jacobian and the velocity gradient lose no digits to
// cancellation.  Elements flagged `precise` (aspect ratio above
// FM_MIXED_ASPECT_LIMIT) form the Jacobian and its inverse in FP64 from the
// staged FP64 coordinates.  The Jacobian, the global derivatives, the
// velocity and its gradient and the nodal terms run two components at a time
// in paired FP32 arithmetic (sm_100 FFMA2 / FMUL2; 5% off the mixed tile
// kernel for tet4 and hexa8).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float rcp_f(float x) {
  const float y = ptx_rcp_approx(x);
  return fmaf(y, fmaf(-x, y, 1.0f), y);  // one Newton step: full FP32 accuracy
}
__device__ __forceinline__ float rsqrt_f(float x) {
  const float y = ptx_rsqrt_approx(x);
  return y * fmaf(-0.5f * x, y * y, 1.5f);
}

// G = J^-T J^-1 (femElement.cpp:192-232), the G:G term of tau, (mu/rho)^2 cI G:G
// (eval_stabilization, src lines 336-377), and G's cofactor inverse
// (eval_bulk_modulus, src lines 382-441).
__device__ __forceinline__ void metric_f(const float inv[3][3], float nu, float cI, float G[3][3], float& t3,
                                         float iG[3][3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) G[a][b] = inv[0][a] * inv[0][b] + inv[1][a] * inv[1][b] + inv[2][a] * inv[2][b];
  t3 = 0.0f;
#pragma unroll
  for (int a = 0; a < 3; ++a) t3 += G[a][0] * G[a][0] + G[a][1] * G[a][1] + G[a][2] * G[a][2];
  t3 = t3 * nu * nu * cI;
  const float m00 = G[0][0], m01 = G[0][1], m02 = G[0][2], m10 = G[1][0], m11 = G[1][1], m12 = G[1][2],
              m20 = G[2][0], m21 = G[2][1], m22 = G[2][2];
  const float dG = m00 * (m11 * m22 - m21 * m12) - m01 * (m10 * m22 - m12 * m20) + m02 * (m10 * m21 - m11 * m20);
  const float idg = rcp_f(dG);
  iG[0][0] = (m11 * m22 - m21 * m12) * idg;
  iG[0][1] = (m02 * m21 - m01 * m22) * idg;
  iG[0][2] = (m01 * m12 - m02 * m11) * idg;
  iG[1][0] = (m12 * m20 - m10 * m22) * idg;
  iG[1][1] = (m00 * m22 - m02 * m20) * idg;
  iG[1][2] = (m10 * m02 - m00 * m12) * idg;
  iG[2][0] = (m10 * m21 - m20 * m11) * idg;
  iG[2][1] = (m20 * m01 - m00 * m21) * idg;
  iG[2][2] = (m00 * m11 - m10 * m01) * idg;
}

template <int NPE, class GEOS>
__device__ __forceinline__ void supg_element_mixed(const DevProb& P, const ShapeTable<NPE, float>& tab,
                                                   const ShapeTable<NPE, double>& tabd, const float Xr[NPE][3],
                                                   const float U0[3], const float Ud[NPE][3], bool precise,
                                                   const double* sx, const double* sy, const double* sz,
                                                   const int ln[NPE], double k[NPE][3], double& lam_el,
                                                   double& reg_el, const GEOS& geo) {
  constexpr bool GEO = NPE == 8;
  const float rho = (float)P.rho, mu = (float)P.mu, alpha = (float)P.alpha, cI = (float)P.c_i;
  const float nu = (float)(P.mu / P.rho);
  const bool bbar = (P.ex_mask & 2) != 0;
  const bool iK1 = (P.ex_mask & 4) != 0, iK2 = (P.ex_mask & 8) != 0, iK3 = (P.ex_mask & 16) != 0,
             iK4 = (P.ex_mask & 32) != 0;
  const float wq = (float)GaussRule<NPE>::weight();
  float kf[NPE][3];
#pragma unroll
  for (int a = 0; a < NPE; ++a) kf[a][0] = kf[a][1] = kf[a][2] = 0.0f;
  // shape values / local derivatives at Gauss point g: tet4 in closed form
  // (constant derivatives), hexa8 from the shared-memory table
  auto dNv = [&](int g, int a, int c) -> float {
    if (NPE == 4) return a == 3 ? -1.0f : (a == c ? 1.0f : 0.0f);
    return tab.dN[g][a][c];
  };
  auto Nv = [&](int g, int a) -> float {
    if (NPE == 4) {
      double q[3];
      GaussRule<NPE>::point(g, q);
      return a < 3 ? (float)q[a] : (float)(1.0 - q[0] - q[1] - q[2]);
    }
    return tab.N[g][a];
  };
  // per Gauss point: inverse Jacobian and det, FP32 or (precise) FP64; with
  // GEO read from the stored geometry (formed in FP64 for every element)
  auto geometry = [&](int g, float inv[3][3]) -> float {
    if constexpr (GEO) return geo.row(g, inv);
    if (precise) {
      double dN[NPE][3], invd[3][3];
#pragma unroll
      for (int a = 0; a < NPE; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) dN[a][c] = tabd.dN[g][a][c];
      const double det = jacobian<NPE>(dN, sx, sy, sz, ln, invd);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) inv[i][j] = (float)invd[i][j];
      return (float)det;
    }
    float J[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      // (J[a][0], J[a][1]) as one pair, J[a][2] alone
      float2 s01 = make_float2(0.0f, 0.0f);
      float s2 = 0.0f;
#pragma unroll
      for (int n = 1; n < NPE; ++n) {
        const float d = dNv(g, n, a);
        s01 = __ffma2_rn(make_float2(d, d), make_float2(Xr[n][0], Xr[n][1]), s01);
        s2 += d * Xr[n][2];
      }
      J[a][0] = s01.x; J[a][1] = s01.y; J[a][2] = s2;
    }
    const float c00 = J[1][1] * J[2][2] - J[2][1] * J[1][2], c01 = J[1][2] * J[2][0] - J[1][0] * J[2][2],
                c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
    const float det = J[0][0] * c00 + J[0][1] * c01 + J[0][2] * c02;
    const float id = rcp_f(det);
    inv[0][0] = c00 * id;
    inv[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * id;
    inv[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * id;
    inv[1][0] = c01 * id;
    inv[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * id;
    inv[1][2] = (J[1][0] * J[0][2] - J[0][0] * J[1][2]) * id;
    inv[2][0] = c02 * id;
    inv[2][1] = (J[2][0] * J[0][1] - J[0][0] * J[2][1]) * id;
    inv[2][2] = (J[0][0] * J[1][1] - J[1][0] * J[0][1]) * id;
    return det;
  };
  // volume-averaged derivatives for B-bar (eval_avg_shapeDeriv, src lines 660-707)
  float sd0[NPE][3];
  if (NPE == 8 && bbar) {
    float num[NPE][3], den = 0.0f;
#pragma unroll
    for (int a = 0; a < NPE; ++a) num[a][0] = num[a][1] = num[a][2] = 0.0f;
#pragma unroll 1
    for (int g = 0; g < GaussRule<NPE>::n; ++g) {
      float inv[3][3];
      const float w = geometry(g, inv) * wq;
      den += w;
#pragma unroll
      for (int a = 0; a < NPE; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
          num[a][b] += (inv[b][0] * dNv(g, a, 0) + inv[b][1] * dNv(g, a, 1) + inv[b][2] * dNv(g, a, 2)) * w;
    }
    const float iden = rcp_f(den);
#pragma unroll
    for (int a = 0; a < NPE; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) sd0[a][b] = num[a][b] * iden;
  }
  // tet4: inverse Jacobian, G, its G:G term and G's inverse are element
  // constants, formed once (the same values as at every Gauss point)
  float inv4[3][3], det4 = 0.0f, G4[3][3], t3_4 = 0.0f, iG4[3][3];
  if constexpr (NPE == 4) {
    det4 = geometry(0, inv4);
    metric_f(inv4, nu, cI, G4, t3_4, iG4);
  }
  float vol = 0.0f, lam_int = 0.0f, reg = 0.0f;
#pragma unroll 1
  for (int g = 0; g < GaussRule<NPE>::n; ++g) {
    float inv[3][3], G[3][3], t3, iG[3][3];
    float det;
    if constexpr (NPE == 4) {
      det = det4;
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          inv[a][b] = inv4[a][b];
          G[a][b] = G4[a][b];
          iG[a][b] = iG4[a][b];
        }
      t3 = t3_4;
    } else {
      det = geometry((NPE == 8 && bbar ? 8 : 0) + g, inv);
      metric_f(inv, nu, cI, G, t3, iG);
    }
    float gd[NPE][3];
    {
      const float2 i0 = make_float2(inv[0][0], inv[1][0]), i1 = make_float2(inv[0][1], inv[1][1]),
                   i2 = make_float2(inv[0][2], inv[1][2]);
#pragma unroll
      for (int a = 0; a < NPE; ++a) {
        const float d0 = dNv(g, a, 0), d1 = dNv(g, a, 1), d2 = dNv(g, a, 2);
        float2 q = __fmul2_rn(i0, make_float2(d0, d0));
        q = __ffma2_rn(i1, make_float2(d1, d1), q);
        q = __ffma2_rn(i2, make_float2(d2, d2), q);
        gd[a][0] = q.x; gd[a][1] = q.y;
        gd[a][2] = inv[2][0] * d0 + inv[2][1] * d1 + inv[2][2] * d2;
      }
    }
    float u[3], gr[3][3];
    {
      // (u0, u1) and (gr[c][0], gr[c][1]) as pairs
      float2 u01 = make_float2(U0[0], U0[1]);
      float u2 = U0[2];
      float2 g01[3] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
      float g2[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int a = 1; a < NPE; ++a) {
        const float Na = Nv(g, a);
        u01 = __ffma2_rn(make_float2(Na, Na), make_float2(Ud[a][0], Ud[a][1]), u01);
        u2 += Na * Ud[a][2];
        const float2 ga = make_float2(gd[a][0], gd[a][1]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          g01[c] = __ffma2_rn(ga, make_float2(Ud[a][c], Ud[a][c]), g01[c]);
          g2[c] += gd[a][2] * Ud[a][c];
        }
      }
      u[0] = u01.x; u[1] = u01.y; u[2] = u2;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        gr[c][0] = g01[c].x; gr[c][1] = g01[c].y; gr[c][2] = g2[c];
      }
    }
    const float div = gr[0][0] + gr[1][1] + gr[2][2];
    // eval_stabilization (dt term removed in the reference)
    const float trG = G[0][0] + G[1][1] + G[2][2];
    float t2 = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) t2 += u[a] * (G[a][0] * u[0] + G[a][1] * u[1] + G[a][2] * u[2]);
    const float tau = rsqrt_f(t2 + t3);
    const float nuC = rcp_f(trG * tau);
    // eval_bulk_modulus: lambda = alpha * max(mu/rho, sqrt(u^T G^-1 u))
    float lam, regime;
    {
      const float q2 = (iG[0][0] * u[0] + iG[0][1] * u[1] + iG[0][2] * u[2]) * u[0] +
                       (iG[1][0] * u[0] + iG[1][1] * u[1] + iG[1][2] * u[2]) * u[1] +
                       (iG[2][0] * u[0] + iG[2][1] * u[1] + iG[2][2] * u[2]) * u[2];
      const float l2 = q2 > 0.0f ? q2 * rsqrt_f(q2) : sqrtf(q2);  // sqrt; NaN for negative input as sqrt
      const float l1 = nu;
      lam = alpha * ((l1 < l2) ? l2 : l1);  // std::max(limit_1, limit_2)
      regime = (l1 > l2) ? 1.0f : 2.0f;
    }
    const float w = det * wq;
    vol += w;
    lam_int += lam * w;
    reg += regime;
    float conv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) conv[c] = u[0] * gr[c][0] + u[1] * gr[c][1] + u[2] * gr[c][2];
    float eps[6];
    if (NPE == 8 && bbar) {
      float e0 = 0.0f, e1 = 0.0f, e2 = 0.0f;
#pragma unroll
      for (int a = 1; a < NPE; ++a) {
        const float B1 = (1.0f / 3.0f) * (sd0[a][0] - gd[a][0]), B2 = gd[a][0] - B1;
        const float B3 = (1.0f / 3.0f) * (sd0[a][1] - gd[a][1]), B4 = gd[a][1] - B3;
        const float B5 = (1.0f / 3.0f) * (sd0[a][2] - gd[a][2]), B6 = gd[a][2] - B5;
        e0 += B2 * Ud[a][0] + B3 * Ud[a][1] + B5 * Ud[a][2];
        e1 += B1 * Ud[a][0] + B4 * Ud[a][1] + B5 * Ud[a][2];
        e2 += B1 * Ud[a][0] + B3 * Ud[a][1] + B6 * Ud[a][2];
      }
      // the node-0 term: B-bar rows sum to zero over the nodes, so the
      // differences to node 0 give the same strain
      eps[0] = e0; eps[1] = e1; eps[2] = e2;
    } else {
      eps[0] = gr[0][0]; eps[1] = gr[1][1]; eps[2] = gr[2][2];
    }
    eps[3] = gr[0][1] + gr[1][0];
    eps[4] = gr[1][2] + gr[2][1];
    eps[5] = gr[0][2] + gr[2][0];
    const float l2m = lam + 2.0f * mu;
    const float sig[6] = {l2m * eps[0] + lam * eps[1] + lam * eps[2], lam * eps[0] + l2m * eps[1] + lam * eps[2],
                          lam * eps[0] + lam * eps[1] + l2m * eps[2], mu * eps[3], mu * eps[4], mu * eps[5]};
    const float c1w = rho * w, c3w = rho * tau * w, c4w = rho * nuC * div * w;
    const float2 conv01 = make_float2(conv[0], conv[1]);
#pragma unroll
    for (int a = 0; a < NPE; ++a) {
      const float Aa = u[0] * gd[a][0] + u[1] * gd[a][1] + u[2] * gd[a][2];
      // (f0, f1) as a pair, f2 alone
      float2 f01 = make_float2(0.0f, 0.0f);
      float f2v = 0.0f;
      if (iK1) {
        const float t = c1w * Nv(g, a);
        f01 = __ffma2_rn(make_float2(t, t), conv01, f01);
        f2v += t * conv[2];
      }
      if (iK3) {
        const float t = c3w * Aa;
        f01 = __ffma2_rn(make_float2(t, t), conv01, f01);
        f2v += t * conv[2];
      }
      if (iK4) {
        f01 = __ffma2_rn(make_float2(c4w, c4w), make_float2(gd[a][0], gd[a][1]), f01);
        f2v += c4w * gd[a][2];
      }
      float f[3] = {f01.x, f01.y, f2v};
      if (iK2) {
        float r0, r1, r2;
        if (NPE == 8 && bbar) {
          const float B1 = (1.0f / 3.0f) * (sd0[a][0] - gd[a][0]), B2 = gd[a][0] - B1;
          const float B3 = (1.0f / 3.0f) * (sd0[a][1] - gd[a][1]), B4 = gd[a][1] - B3;
          const float B5 = (1.0f / 3.0f) * (sd0[a][2] - gd[a][2]), B6 = gd[a][2] - B5;
          r0 = B2 * sig[0] + B1 * sig[1] + B1 * sig[2];
          r1 = B3 * sig[0] + B4 * sig[1] + B3 * sig[2];
          r2 = B5 * sig[0] + B5 * sig[1] + B6 * sig[2];
        } else {
          r0 = gd[a][0] * sig[0];
          r1 = gd[a][1] * sig[1];
          r2 = gd[a][2] * sig[2];
        }
        // (f0, f1) as a pair
        float2 t01 = __ffma2_rn(make_float2(gd[a][1], gd[a][0]), make_float2(sig[3], sig[3]), make_float2(r0, r1));
        t01 = __ffma2_rn(make_float2(gd[a][2], gd[a][2]), make_float2(sig[5], sig[4]), t01);
        const float2 n01 = __ffma2_rn(t01, make_float2(w, w), make_float2(f[0], f[1]));
        f[0] = n01.x; f[1] = n01.y;
        f[2] += (r2 + gd[a][1] * sig[4] + gd[a][0] * sig[5]) * w;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) kf[a][c] += f[c];
    }
  }
  const double mdt = -P.dt;
#pragma unroll
  for (int a = 0; a < NPE; ++a)
#pragma unroll
    for (int c = 0; c < 3; ++c) k[a][c] = mdt * (double)kf[a][c];
  lam_el = (double)lam_int / (double)vol;
  reg_el = (double)reg / (double)GaussRule<NPE>::n;
}

}  // namespace fm
