// 2-D Q2/P1 residual + analytic Jacobian (Navier-Stokes, Newtonian or
// Carreau-Yasuda, optional energy): element matrices by sum factorisation,
// then every CSR row gathered from its elements.
//
// Same physics and results (to rounding) as the scalar kernel of
// gb_assemble.cu: the reference's assemble_momentum
// (src/mm_fill_momentum.c:100, fluid_stress :2834), assemble_continuity
// (src/mm_fill_continuity.c:119), assemble_energy (src/mm_fill_energy.c:109),
// carreau_viscosity (src/mm_viscosity.c:981), bouss_momentum_source
// (src/mm_std_models.c:125), the hard-set Dirichlet rows of
// put_dirichlet_in_matrix (src/bc_dirich.c:44) and the load_lec scatter
// (src/mm_fill.c:5175).
//
// What bounds it: the count of FP64 operations (GB300: a warp's FP64
// instruction every 16 clocks of an SM), and on small meshes launches and
// serial chains.  The dense loops over 9 points x 81 node pairs took ~33K
// FP64 lane operations an element, in one launch a colour with one element's
// points on 9 lanes.  Here:
//   - weighted mass matrices M_w(i,j) = sum_q phi_i phi_j w(q) (velocity and
//     temperature gradients, dA, the heat source) and the advection term as
//     two contractions of 1-D factors; the factors l_a l_b are symmetric, so a
//     mass matrix has 6 x 6 distinct values, the advection terms 9 x 6;
//   - H = sum_q dphi_i/dx_p w dphi_j/dx_r (w = dA, times the viscosity where
//     it varies) as one symmetric 18 x 18 product, upper triangle only: the
//     transpose stress term and through its trace the viscous one; with
//     Carreau viscosity a second one for d mu / d gammadot;
//   J_ab = M(-rho dA dv_a/dx_b) - mu H((b,i),(a,j)) + C((a,i),(b,j))
//          + delta_ab (S1 - mu tr H - mass)
// about 7K lane operations an element.  The element matrices go to a scratch
// array (node-pair blocks), every element at once, and assemble_rows_kernel
// builds each node's rows in shared memory from its elements in ascending
// order and writes them once: no zeroing of the matrix, no colours, and a
// result that does not depend on timing.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "gb_device.h"
#include "gb_launch.cuh"

namespace gb {

namespace s2 {

constexpr int NN = 9, NQ = 9, NP = 3, CENT = 8;
constexpr int NH = 18 * 19 / 2;  // upper triangle of an 18 x 18 product
constexpr int NT = 9 * 10 / 2;   // of a 9 x 9 one
// contractions: advection (two), velocity gradients (a, b), dA, temperature
// gradients, heat-source sensitivity
enum { C_S1 = 0, C_AB = 2, C_DA = 6, C_TV = 7, C_DH = 9 };
// their distinct values: 9 x 6 (advection along the first direction), 6 x 9
// (along the second), 6 x 6
__device__ __forceinline__ int mass_at(int c) { return c < 2 ? 54 * c : 108 + 36 * (c - 2); }

template <bool ENERGY, bool CARREAU>
struct Elem {
  static constexpr int NF = ENERGY ? 5 : 4;   // x y u v (T)
  static constexpr int NV = ENERGY ? 3 : 2;
  static constexpr int NC = ENERGY ? 10 : 7;
  double Xn[NF][NN];     // nodal values, lexicographic
  double Xd[NV][NN];     // time derivatives (transient)
  double Pn[NP];
  double rho;
  double A[NF][2][9];    // contracted over the first direction
  double F[NF][3][NQ];   // value, d/dxi_1, d/dxi_2 at the points
  double B[4][NQ];       // J^-1 [2 p + r]
  double w[NQ];          // weight of H
  double wT[NQ];         // dA (conduction, where w is not dA)
  double W[NC][NQ];
  double cR[NV][NQ];     // residual: phi part
  double tR[2][NV][NQ];  // residual: gradient part
  double psidA[NP][NQ];
  double cm[CARREAU ? NQ : 1];         // -dA (d mu / d gammadot) / gammadot
  double gam[CARREAU ? 3 : 1][NQ];     // shear rate tensor 00, 01, 11
  double G[2][NQ][NN];   // d phi_L / d x_p
  double cG[2][NQ][NN];  // w G
  double g[CARREAU ? 2 : 1][NQ][NN];   // grad phi . gamma_a
  double cg[CARREAU ? 2 : 1][NQ][NN];  // cm times it
  double T1[NC][3][9];   // contracted over the second direction
  double Mw[108 + 36 * (NC - 2)];  // over both
  double H[NH];
  double C[CARREAU ? NH : 1];
  double HT[ENERGY && CARREAU ? NT : 1];
  double div[NQ];        // div v at the points
  int bad;
};

__device__ __forceinline__ int tri(int n, int P, int R) {  // upper triangle of n x n
  const int a = P < R ? P : R, b = P < R ? R : P;
  return a * n - (a * (a - 1)) / 2 + b - a;
}

}  // namespace s2

template <bool ENERGY, bool CARREAU, bool JAC, int EPB, int NTH>
__global__ void __launch_bounds__(NTH)
    assemble_2d_kernel(AsmArgs A, const S2Tables *__restrict__ gtb, int nelem, S2Scratch out) {
  using namespace s2;
  using E2 = Elem<ENERGY, CARREAU>;
  constexpr int NF = E2::NF, NV = E2::NV, NC = E2::NC;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  E2 *S = reinterpret_cast<E2 *>(smem_raw);
  // the tables: a first read of each from L2 would cost every phase its trip
  __shared__ S2Tables stb;
  const S2Tables *tb = &stb;
  const int tid = threadIdx.x;
  static_assert(sizeof(S2Tables) % 8 == 0, "copied by doubles");
  for (int t = tid; t < (int)(sizeof(S2Tables) / 8); t += NTH)
    reinterpret_cast<double *>(&stb)[t] = reinterpret_cast<const double *>(gtb)[t];
  dependent_begin();
  const MaterialDev M = A.mat;
  const int e0 = blockIdx.x * EPB;
  const int live = min(EPB, nelem - e0);
  // every loop below runs over (element, item) pairs of the block's elements
#define GB_EACH(cnt)                                              \
  for (int t_ = tid; t_ < live * (cnt); t_ += NTH)                \
    if (const int el = t_ / (cnt), r = t_ - el * (cnt); true)

  GB_EACH(NN) {
    E2 &E = S[el];
    const int k = r, L = gtb->lex[k];
    const int n = A.conn[(int64_t)(e0 + el) * NN + k], f0 = A.fu[n];
    // coordinates from the centroid node's: only their differences count, and
    // a mesh far from the origin loses no digits to its offset
    const int nc = A.conn[(int64_t)(e0 + el) * NN + CENT];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      E.Xn[j][L] = A.coords[(int64_t)n * 2 + j] - A.coords[(int64_t)nc * 2 + j];
      E.Xn[2 + j][L] = A.x[f0 + j];
    }
    if (ENERGY) E.Xn[4][L] = A.x[f0 + 2];
    if (k == CENT) {
#pragma unroll
      for (int l = 0; l < NP; l++) E.Pn[l] = A.x[f0 + A.pofs + l];
      E.rho = A.elem_rho ? A.elem_rho[e0 + el] : M.density;
      E.bad = 0;
    }
    if (A.xdot) {
#pragma unroll
      for (int c = 0; c < NV; c++) E.Xd[c][L] = A.xdot[f0 + c];
    }
  }
  __syncthreads();
  // values and reference gradients at the points, one direction at a time
  GB_EACH(NF * 18) {
    E2 &E = S[el];
    const int f = r / 18, v = (r / 9) & 1, p = r % 9, a2 = p / 3, q1 = p % 3;
    const double *x = &E.Xn[f][3 * a2];
    const double(*l)[3] = tb->ell[v];
    E.A[f][v][p] = l[0][q1] * x[0] + l[1][q1] * x[1] + l[2][q1] * x[2];
  }
  __syncthreads();
  GB_EACH(NF * 27) {
    E2 &E = S[el];
    const int f = r / 27, d = (r / 9) % 3, q = r % 9, q2 = q / 3, q1 = q % 3;
    const double *a = &E.A[f][d == 1 ? 1 : 0][q1];
    const double(*l)[3] = tb->ell[d == 2 ? 1 : 0];
    E.F[f][d][q] = l[0][q2] * a[0] + l[1][q2] * a[3] + l[2][q2] * a[6];
  }
  __syncthreads();
  // per quadrature point
  GB_EACH(NQ) {
    E2 &E = S[el];
    const int q = r;
    const double rho = E.rho;
    double Jm[2][2], Gh[2][2], v[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      v[i] = E.F[2 + i][0][q];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        Jm[i][j] = E.F[j][1 + i][q];
        Gh[i][j] = E.F[2 + j][1 + i][q];
      }
    }
    const double det = Jm[0][0] * Jm[1][1] - Jm[0][1] * Jm[1][0];
    if (!(det > 0.0)) E.bad = 1;
    const double id = 1.0 / det;
    const double B[2][2] = {{Jm[1][1] * id, -Jm[0][1] * id}, {-Jm[1][0] * id, Jm[0][0] * id}};
    const double dA = tb->w[q] * det;
    double gv[2][2], gT[2] = {0.0, 0.0}, T = 0.0;  // gv[p][a] = d v_a / d x_p
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int a = 0; a < 2; a++) gv[p][a] = B[p][0] * Gh[0][a] + B[p][1] * Gh[1][a];
    if (ENERGY) {
      T = E.F[4][0][q];
#pragma unroll
      for (int p = 0; p < 2; p++) gT[p] = B[p][0] * E.F[4][1][q] + B[p][1] * E.F[4][2][q];
    }
    double mu = M.viscosity;
    const double g00 = 2.0 * gv[0][0], g01 = gv[0][1] + gv[1][0], g11 = 2.0 * gv[1][1];
    if (CARREAU) {
      const double s2v = g00 * g00 + 2.0 * g01 * g01 + g11 * g11;
      const double gd = sqrt(0.5 * fabs(s2v));
      const bool nz = gd > 1.0e-298;
      const double lg = M.lambda * gd;
      // (lg)^a and (1 + lg^a)^((n-1)/a); the other two powers of the model
      // follow by a division (unless lg^a underflows; where it overflows, a
      // finite number over lg meets the other quotient's zero)
      const double val2 = !nz ? 0.0 : (M.aexp == 2.0 ? lg * lg : pow(lg, M.aexp));
      const double base = 1.0 + val2;
      const double pw = pow(base, (M.nexp - 1.0) / M.aexp);
      mu = M.mu_inf + (M.mu0 - M.mu_inf) * pw;
      const double val = !nz ? 0.0
                             : (val2 > 1.0e-280 ? fmin(val2, 1.0e308) / lg
                                                : pow(lg, M.aexp - 1.0));
      const double dmu = (M.mu0 - M.mu_inf) * (M.nexp - 1.0) * M.lambda * val * (pw / base);
      E.cm[q] = nz ? -dA * (dmu / gd) : 0.0;
      E.gam[0][q] = g00;
      E.gam[CARREAU ? 1 : 0][q] = g01;
      E.gam[CARREAU ? 2 : 0][q] = g11;
    }
    E.w[q] = CARREAU ? mu * dA : dA;
    E.wT[q] = dA;
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int s = 0; s < 2; s++) E.B[2 * p + s][q] = B[p][s];
    const double psi[NP] = {1.0, tb->pt[q % 3], tb->pt[q / 3]};
    double P = 0.0;
#pragma unroll
    for (int l = 0; l < NP; l++) {
      P = fma(E.Pn[l], psi[l], P);
      E.psidA[l][q] = psi[l] * dA;
    }
    double vd[NV];
#pragma unroll
    for (int c = 0; c < NV; c++) vd[c] = 0.0;
    if (A.xdot)
      for (int L = 0; L < NN; L++)
#pragma unroll
        for (int c = 0; c < NV; c++) vd[c] = fma(tb->phi[q][L], E.Xd[c][L], vd[c]);
    E.div[q] = gv[0][0] + gv[1][1];
    const double rA = -rho * dA;
#pragma unroll
    for (int a = 0; a < 2; a++) {
#pragma unroll
      for (int b = 0; b < 2; b++) E.W[C_AB + 2 * a + b][q] = rA * gv[b][a];
      E.W[C_S1 + a][q] = rA * (v[0] * B[0][a] + v[1] * B[1][a]);
      double f = M.source[a];
      if (M.source_model == GB_SOURCE_BOUSSINESQ)
        f = ENERGY ? rho * M.source[a] * (-M.beta * (T - M.Tref)) : 0.0;
      // with the mass term -rho v_dot_a (src/mm_fill_momentum.c:471-500)
      E.cR[a][q] = dA * f + rA * (v[0] * gv[0][a] + v[1] * gv[1][a] + vd[a]);
    }
    E.tR[0][0][q] = -dA * (mu * g00 - P);
    E.tR[0][1][q] = E.tR[1][0][q] = -dA * (mu * g01);
    E.tR[1][1][q] = -dA * (mu * g11 - P);
    E.W[C_DA][q] = dA;
    if (ENERGY) {
      const double rc = rA * M.heat_capacity;
      double hs = 0.0, dhs = 0.0;
      if (M.hsm == GB_HEAT_SOURCE_CONSTANT) {
        hs = M.hs[0];
      } else if (M.hsm == GB_HEAT_SOURCE_EXPONENTIAL) {
        hs = M.hs[0] * exp(M.hs[1] * T);
        dhs = M.hs[1] * hs;
      }
      E.cR[NV - 1][q] = rc * (v[0] * gT[0] + v[1] * gT[1] + vd[NV - 1]) + dA * hs;
#pragma unroll
      for (int p = 0; p < 2; p++) {
        E.tR[p][NV - 1][q] = -M.conductivity * dA * gT[p];
        E.W[(ENERGY ? C_TV : 0) + p][q] = rc * gT[p];
      }
      E.W[ENERGY ? C_DH : 0][q] = dhs * dA;
    }
  }
  __syncthreads();
  // physical gradients; second direction of the contractions
  GB_EACH(NQ * NN) {
    E2 &E = S[el];
    const int q = r / NN, L = r % NN;
    const double d0 = tb->dref[q][L][0], d1 = tb->dref[q][L][1];
    const double x = E.B[0][q] * d0 + E.B[1][q] * d1, y = E.B[2][q] * d0 + E.B[3][q] * d1;
    E.G[0][q][L] = x;
    E.G[1][q][L] = y;
    if (JAC) {
      E.cG[0][q][L] = E.w[q] * x;
      E.cG[1][q][L] = E.w[q] * y;
    }
    if (CARREAU && JAC) {
      const double g01 = E.gam[CARREAU ? 1 : 0][q], cm = E.cm[q];
      const double g0 = x * E.gam[0][q] + y * g01;
      const double g1 = x * g01 + y * E.gam[CARREAU ? 2 : 0][q];
      E.g[0][q][L] = g0;
      E.g[CARREAU ? 1 : 0][q][L] = g1;
      E.cg[0][q][L] = cm * g0;
      E.cg[CARREAU ? 1 : 0][q][L] = cm * g1;
    }
  }
  // (dA only where the energy equation or the mass terms ask for it)
  const int skip = !ENERGY && A.mass_c == 0.0 ? C_DA : -1;
  if (JAC) {
    GB_EACH(NC * 18 + 9) {  // item: contraction, q1, pair of the second direction
      E2 &E = S[el];
      const bool d2 = r < 27;  // the advection along the second direction: 9 pairs
      const int c = d2 ? C_S1 + 1 : ((r - 27) / 18 == 0 ? C_S1 : (r - 27) / 18 + 1);
      const int p = d2 ? r : (r - 27) % 18, q1 = p % 3, u2 = p / 3;
      if (c == skip) continue;
      const double *pp = d2 ? tb->pp[1][u2] : tb->pu[u2], *w = &E.W[c][q1];
      E.T1[c][q1][u2] = pp[0] * w[0] + pp[1] * w[3] + pp[2] * w[6];
    }
  }
  __syncthreads();
  // residual rows; continuity rows; J_mP (and J_cv, its transpose)
  GB_EACH(NV * NN + NP) {
    const E2 &E = S[el];
    const int64_t e = e0 + el;
    double s = 0.0;
    if (r < NV * NN) {
      const int n = r / NN, L = r % NN;
      double s1 = 0.0, s2v = 0.0;
#pragma unroll 3
      for (int q = 0; q < NQ; q++) {
        s = fma(tb->phi[q][L], E.cR[n][q], s);
        s1 = fma(E.G[0][q][L], E.tR[0][n][q], s1);
        s2v = fma(E.G[1][q][L], E.tR[1][n][q], s2v);
      }
      out.R[e * (NV * NN) + tb->loc[L] * NV + n] = s + (s1 + s2v);
    } else {
      const int l = r - NV * NN;
      for (int q = 0; q < NQ; q++) s = fma(E.psidA[l][q], E.div[q], s);
      out.Rc[e * NP + l] = s;
      if (l == 0 && E.bad) {
        atomicAdd(A.status, 1);
        atomicMin(A.status + 1, (int)e);
      }
    }
  }
  if constexpr (JAC) {
  GB_EACH(2 * NN * NP) {
    const E2 &E = S[el];
    const int L = r / (2 * NP), a = (r / NP) % 2, l = r % NP;
    double s = 0.0;
#pragma unroll 3
    for (int q = 0; q < NQ; q++) s = fma(E.G[a][q][L], E.psidA[l][q], s);
    out.P[(int64_t)(e0 + el) * (2 * NN * NP) + (tb->loc[L] * 2 + a) * NP + l] = s;
  }
  GB_EACH(108 + 36 * (NC - 2)) {
    E2 &E = S[el];
    const int c = r < 108 ? r / 54 : 2 + (r - 108) / 36;
    if (c == skip) continue;
    const int m = r - mass_at(c), n2 = c == C_S1 + 1 ? 9 : 6, u1 = m / n2, u2 = m - u1 * n2;
    const double *pp = c == C_S1 ? tb->pp[1][u1] : tb->pu[u1];
    E.Mw[r] = pp[0] * E.T1[c][0][u2] + pp[1] * E.T1[c][1][u2] + pp[2] * E.T1[c][2][u2];
  }
  GB_EACH(NH) {
    E2 &E = S[el];
    const int pr = tb->hmap[r], P = pr >> 8, R = pr & 255;
    const int p = P / NN, i = P - p * NN, s = R / NN, j = R - s * NN;
    double h0 = 0.0, h1 = 0.0, h2 = 0.0;
#pragma unroll
    for (int q = 0; q < NQ; q += 3) {
      h0 = fma(E.G[p][q][i], E.cG[s][q][j], h0);
      h1 = fma(E.G[p][q + 1][i], E.cG[s][q + 1][j], h1);
      h2 = fma(E.G[p][q + 2][i], E.cG[s][q + 2][j], h2);
    }
    E.H[r] = (h0 + h1) + h2;
    if (CARREAU) {
      double c0 = 0.0;
#pragma unroll 3
      for (int q = 0; q < NQ; q++) c0 = fma(E.g[p][q][i], E.cg[s][q][j], c0);
      E.C[CARREAU ? r : 0] = c0;
    }
    if (ENERGY && CARREAU && P < NN && R < NN) {
      double c0 = 0.0;
#pragma unroll 3
      for (int q = 0; q < NQ; q++)
        c0 = fma(E.wT[q], E.G[0][q][i] * E.G[0][q][j] + E.G[1][q][i] * E.G[1][q][j], c0);
      E.HT[ENERGY && CARREAU ? tri(NN, i, j) : 0] = c0;
    }
  }
  __syncthreads();
  // node pairs
  GB_EACH(NN * NN) {
    const E2 &E = S[el];
    const int Li = tb->lex[r / NN], Lj = tb->lex[r % NN];
    const int ab1 = (Li % 3) * 3 + Lj % 3, ab2 = (Li / 3) * 3 + Lj / 3;
    const int u1 = tb->sym[ab1], u2 = tb->sym[ab2], u12 = 6 * u1 + u2;
    auto mass = [&](int c) { return E.Mw[mass_at(c) + u12]; };
    const double muf = CARREAU ? 1.0 : M.viscosity;
    const double S1 = E.Mw[6 * ab1 + u2] + E.Mw[54 + 9 * u1 + ab2];
    const double trH = E.H[tri(18, Li, Lj)] + E.H[tri(18, NN + Li, NN + Lj)];
    const bool tr = A.mass_c != 0.0;
    const double mdA = (ENERGY || tr) ? mass(C_DA) : 0.0;
    // the mass terms' sensitivity -(1 + 2 theta) / dt rho M(dA)
    // (src/mm_fill_momentum.c:1586-1590), times Cp on the energy row
    const double Mt = tr ? -A.mass_c * E.rho * mdA : 0.0;
    const double D = fma(-muf, trH, S1) + Mt;
    double *K = out.K + ((int64_t)(e0 + el) * (NN * NN) + r) * (NV * NV);
#pragma unroll
    for (int a = 0; a < 2; a++) {
#pragma unroll
      for (int b = 0; b < 2; b++) {
        double v = fma(-muf, E.H[tri(18, b * NN + Li, a * NN + Lj)], mass(C_AB + 2 * a + b));
        if (CARREAU) v += E.C[CARREAU ? tri(18, a * NN + Li, b * NN + Lj) : 0];
        if (a == b) v += D;
        K[a * NV + b] = v;
      }
      if (ENERGY)
        K[a * NV + NV - 1] =
            M.source_model == GB_SOURCE_BOUSSINESQ ? -E.rho * M.source[a] * M.beta * mdA : 0.0;
    }
    if (ENERGY) {
#pragma unroll
      for (int b = 0; b < 2; b++) K[(NV - 1) * NV + b] = mass((ENERGY ? C_TV : 0) + b);
      const double cond = CARREAU ? E.HT[ENERGY && CARREAU ? tri(NN, Li, Lj) : 0] : trH;
      K[(NV - 1) * NV + NV - 1] = fma(M.heat_capacity, S1 + Mt, -M.conductivity * cond) +
                                  mass(ENERGY ? C_DH : 0);
    }
  }
  }
#undef GB_EACH
}

// Every node's residual entries and CSR rows from its elements' blocks, one
// warp per node: the rows are built in shared memory, the elements added in
// ascending order (entries of one element go to different places), and
// written once, zeros included.  Bound by the memory traffic of the blocks
// and the rows.
template <bool ENERGY, bool JAC>
__global__ void __launch_bounds__(128)
    assemble_rows_kernel(AsmArgs A, S2Nodes nd, S2Scratch in) {
  dependent_begin();
  using namespace s2;
  constexpr int NV = ENERGY ? 3 : 2, Tr = ENERGY ? 2 : -1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double *blk = reinterpret_cast<double *>(smem_raw) + (size_t)w * nd.blkmax;
  const int n = blockIdx.x * 4 + w;
  if (n >= nd.num_nodes) return;
  const int f0 = A.fu[n], nr = A.fu[n + 1] - f0, nvn = A.pofs;
  const int p0 = nd.ne_ptr[n], p1 = nd.ne_ptr[n + 1];
  if (lane < nr) {
    double s = 0.0;
    if (!A.dbc[f0 + lane])
      for (int p = p0; p < p1; p++) {
        const int64_t e = nd.ne_list[p] / NN;
        const int k = nd.ne_list[p] % NN;
        if (lane < NV) s += in.R[e * (NV * NN) + k * NV + lane];
        // the pressures are the centroid's element's, whoever else has the node
        else if (lane >= nvn && k == CENT) s += in.Rc[e * NP + lane - nvn];
      }
    A.R[f0 + lane] = s;
  }
  if (!JAC) return;
  const int64_t r0 = A.rowptr[f0], r1 = A.rowptr[f0 + nr];
  const int size = (int)(r1 - r0);
  const int len = (int)(A.rowptr[f0 + 1] - r0);  // of every row but the energy row
  const int lenT = ENERGY ? (int)(A.rowptr[f0 + 3] - A.rowptr[f0 + 2]) : 0;
  auto row = [&](int r) { return r * len - (ENERGY && r > Tr ? len - lenT : 0); };
  const int base = A.nbr_ptr[n];
  // an element's share: up to three entries a lane of its 9 node blocks and
  // one of its pressure columns, loaded while the element before is added
  constexpr int KB = NN * NV * NV, KL = (KB + 31) / 32;
  struct Share {
    double v[KL], pv;
    int at[KL], pat;
  };
  auto load = [&](int p, Share &h) {
    const int ek = nd.ne_list[p];
    const int64_t e = ek / NN;
    const int k = ek % NN;
    const uint16_t *ns = A.elem_nslot + (int64_t)ek * NN;
    const double *K = in.K + (int64_t)ek * KB;
#pragma unroll
    for (int j = 0; j < KL; j++) {
      const int t = lane + 32 * j;
      if (t >= KB) {
        h.at[j] = -1;
        continue;
      }
      const int l = t / (NV * NV), a = (t / NV) % NV, b = t % NV, s = base + ns[l];
      h.v[j] = __ldcs(K + t);
      h.at[j] = row(a) + (a == Tr ? A.nbr_offT[s] : A.nbr_off[s]) + b;
    }
    h.pat = -1;
    if (lane < 2 * NP) {  // the element's pressures in the node's momentum rows
      const int a = lane / NP, l = lane % NP;
      h.pv = in.P[e * (2 * NN * NP) + (k * 2 + a) * NP + l];
      h.pat = row(a) + A.nbr_off[base + ns[CENT]] + nvn + l;
    }
  };
  Share cur, nxt;
  if (p0 < p1) load(p0, cur);
  for (int c = lane; c < size; c += 32) blk[c] = 0.0;
  __syncwarp();
  for (int p = p0; p < p1; p++) {
    if (p + 1 < p1) load(p + 1, nxt);
#pragma unroll
    for (int j = 0; j < KL; j++)
      if (cur.at[j] >= 0) blk[cur.at[j]] += cur.v[j];
    if (cur.pat >= 0) blk[cur.pat] += cur.pv;
    const int ek = nd.ne_list[p];
    if (ek % NN == CENT) {  // the continuity rows
      const uint16_t *ns = A.elem_nslot + (int64_t)ek * NN;
      const double *P = in.P + (int64_t)(ek / NN) * (2 * NN * NP);
      for (int t = lane; t < NP * NN * 2; t += 32) {
        const int l = t / (2 * NN), m = (t / 2) % NN, b = t & 1;
        blk[row(nvn + l) + A.nbr_off[base + ns[m]] + b] += P[(m * 2 + b) * NP + l];
      }
    }
    __syncwarp();
    cur = nxt;
  }
  // Dirichlet rows: 1 per element on the diagonal, once for a pressure (species
  // rows get theirs from the species kernel)
  int self = -1;
  if (p1 > p0) self = A.elem_nslot[(int64_t)nd.ne_list[p0] * NN + nd.ne_list[p0] % NN];
  for (int r = 0; r < nr; r++) {
    if (!A.dbc[f0 + r]) continue;
    const int rl = r == Tr ? lenT : len;
    for (int c = lane; c < rl; c += 32) blk[row(r) + c] = 0.0;
    __syncwarp();
    if (lane == 0 && self >= 0 && (r < NV || r >= nvn))
      blk[row(r) + (r == Tr ? A.nbr_offT[base + self] : A.nbr_off[base + self]) + r] =
          r < NV ? p1 - p0 : 1;
  }
  __syncwarp();
  double *out = A.vals + r0;
  for (int c = lane; c < size; c += 32) __stcs(out + c, blk[c]);
}

void build_s2_tables(const double *tab_phi, const double *tab_dphi, const double *tab_w,
                     const double *pt, const int (*loc9)[2], const double *ell,
                     const double *dell, S2Tables &T) {
  using namespace s2;
  for (int a = 0; a < 3; a++) {
    T.pt[a] = pt[a];
    for (int g = 0; g < 3; g++) {
      T.ell[0][a][g] = ell[a * 3 + g];
      T.ell[1][a][g] = dell[a * 3 + g];
      for (int b = 0; b < 3; b++) {
        T.pp[0][a * 3 + b][g] = ell[a * 3 + g] * ell[b * 3 + g];
        T.pp[1][a * 3 + b][g] = ell[a * 3 + g] * dell[b * 3 + g];
      }
    }
  }
  int nu = 0;
  for (int a = 0; a < 3; a++)
    for (int b = a; b < 3; b++, nu++) {
      T.sym[a * 3 + b] = T.sym[b * 3 + a] = nu;
      for (int g = 0; g < 3; g++) T.pu[nu][g] = T.pp[0][a * 3 + b][g];
    }
  for (int k = 0; k < NN; k++) {
    const int L = loc9[k][0] + 3 * loc9[k][1];
    T.lex[k] = L;
    T.loc[L] = k;
  }
  for (int q = 0; q < NQ; q++) {
    T.w[q] = tab_w[q];
    for (int L = 0; L < NN; L++) {
      const int k = T.loc[L];
      T.phi[q][L] = tab_phi[q * NN + k];
      for (int r = 0; r < 2; r++) T.dref[q][L][r] = tab_dphi[(q * NN + k) * 2 + r];
    }
  }
  int e = 0;
  for (int P = 0; P < 18; P++)
    for (int R = P; R < 18; R++) T.hmap[e++] = (uint16_t)((P << 8) | R);
}

size_t s2_scratch_values(bool energy, bool jac) {
  const size_t nv = energy ? 3 : 2;
  return s2::NN * nv + s2::NP + (jac ? 81 * nv * nv + 54 : 0);
}

template <bool ENERGY, bool CARREAU, bool JAC, int EPB, int NTH>
static cudaError_t launch_elems(const AsmArgs &a, const S2Tables *tb, int nelem,
                                const S2Scratch &s, cudaStream_t st) {
  const size_t sm = sizeof(s2::Elem<ENERGY, CARREAU>) * EPB;
  auto k = assemble_2d_kernel<ENERGY, CARREAU, JAC, EPB, NTH>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  launch_dependent(k, (nelem + EPB - 1) / EPB, NTH, sm, st, a, tb, nelem, s);
  return cudaGetLastError();
}

template <bool ENERGY, bool CARREAU, bool JAC>
static cudaError_t launch_2d(const AsmArgs &a, const S2Tables *tb, int nelem, const S2Nodes &nd,
                             const S2Scratch &s, int sms, cudaStream_t st) {
  // Four elements a CTA keep its lanes busy (us of the element kernel, one /
  // four / eight elements a CTA: 118K elements 2305 / 1891 / 1865, 96 x 32
  // Carreau 115 / 92 / 97, 1024 elements 25 / 25 / 24); a few elements are
  // spread over all SMs, one a CTA (54 elements 16 / 20 / 24).
  cudaError_t e = nelem < 4 * sms
                      ? launch_elems<ENERGY, CARREAU, JAC, 1, 64>(a, tb, nelem, s, st)
                      : launch_elems<ENERGY, CARREAU, JAC, 4, 128>(a, tb, nelem, s, st);
  if (e != cudaSuccess) return e;
  const size_t sm = JAC ? s2_rows_smem(nd.blkmax) : 0;
  auto k = assemble_rows_kernel<ENERGY, JAC>;
  if (JAC) {
    // the limit belongs to the process: the same for every mesh, so that a
    // thread with shorter rows does not lower it before this launch
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kS2RowsSmemMax);
    if (e != cudaSuccess) return e;
  }
  launch_dependent(k, (nd.num_nodes + 3) / 4, 128, sm, st, a, nd, s);
  return cudaGetLastError();
}

cudaError_t launch_assemble_2d(const AsmArgs &a, bool energy, bool carreau, bool jac,
                               const S2Tables *tb, int nelem, const S2Nodes &nd, double *scratch,
                               int sms, cudaStream_t st) {
  const size_t nv = energy ? 3 : 2, ne = nelem;
  S2Scratch s;
  s.K = scratch;  // first: 16-byte aligned blocks
  s.P = scratch + (jac ? ne * 81 * nv * nv : 0);
  s.R = s.P + (jac ? ne * 54 : 0);
  s.Rc = s.R + ne * 9 * nv;
#define GB_DISPATCH(EN, CA, JA) \
  if (energy == EN && carreau == CA && jac == JA) \
    return launch_2d<EN, CA, JA>(a, tb, nelem, nd, s, sms, st);
  GB_DISPATCH(false, false, true)
  GB_DISPATCH(false, true, true)
  GB_DISPATCH(true, false, true)
  GB_DISPATCH(true, true, true)
  GB_DISPATCH(false, false, false)
  GB_DISPATCH(false, true, false)
  GB_DISPATCH(true, false, false)
  GB_DISPATCH(true, true, false)
#undef GB_DISPATCH
  return cudaErrorInvalidValue;
}

}  // namespace gb
