// 3-D Q2/P1 element residual + analytic Jacobian (Newtonian Navier-Stokes,
// optional energy with a Boussinesq body force) with the fewest FP64
// operations: sum factorisation over the tensor-product HEX27 basis for
// every term whose test and trial functions are reference-element tensor
// products, and one symmetric product for the rest.
//
// Same physics and results (to rounding) as the scalar kernel of
// gb_assemble.cu: the reference's assemble_momentum
// (src/mm_fill_momentum.c:100, fluid_stress :2834), assemble_continuity
// (src/mm_fill_continuity.c:119), assemble_energy (src/mm_fill_energy.c:109),
// bouss_momentum_source (src/mm_std_models.c:125), the hard-set Dirichlet rows
// of put_dirichlet_in_matrix (src/bc_dirich.c:44) and the load_lec scatter
// (src/mm_fill.c:5175).
//
// Why: on GB300 FP64 runs at ~2 FMA per SM-cycle, on the scalar units and on
// the FP64 tensor path (mma.sync m8n8k4) alike, so the element kernel is
// bound by its count of FP64 operations, not by memory.  Per element:
//
//   field values and reference gradients at the 27 points: sum
//     factorisation, 3 passes over the 1-D factors (~5K FMA instead of 20K);
//   weighted mass matrices  M_w(i,j) = sum_q phi_i phi_j w(q)  for 13
//     weights (-rho dA dv_a/dx_b, -rho Cp dA dT/dx_b, dA) and the advection
//     term S1(i,j) = sum_q phi_i (-rho dA v . grad phi_j) written as three
//     such sums over reference derivatives: phi_i phi_j = prod_d
//     l_{i_d}(q_d) l_{j_d}(q_d), so each is three contractions, and since
//     l_a l_b has 6 distinct values a direction a mass matrix has 216, 162 +
//     324 + 648 FMA instead of 19,683 (an advection term 324, ~1,600 FMA);
//   residual rows: the same way, 729 FMA each instead of 2,916;
//   H((p,i),(r,j)) = sum_q dphi_i/dx_p dA dphi_j/dx_r: gives the transpose
//     stress term -mu H((b,i),(a,j)) of J_ab, and through its trace the
//     viscous term of J_aa and the conduction term of J_TT.  A thread keeps
//     the 3 x 3 block of a node pair i <= j in registers (9 FMA from 6 loads)
//     and forms J(i,j) and J(j,i) from it, 378 x 9 x 27 FMA.
//
//   J_ab   = M(-rho dA dv_a/dx_b) - mu H((b,i),(a,j)) + delta_ab (S1 - mu tr H)
//   J_TT   = Cp S1 - k tr H
//   J_Tb   = M(-rho Cp dA dT/dx_b),   J_aT = (df_a/dT) M(dA)
//   J_mP   = sum_q dphi_i/dx_a psi_l dA,   J_cv = J_mP^T
//
// That is ~160K FP64 operations per element against ~865K for the dense
// forms; at 2 FMA a clock 13,824 elements (24^3) cannot take less than
// ~3.8 ms.  Measured 4.27 ms, 5.45 ms for 324 products a mass matrix, a dense
// residual and H entry by entry through shared memory (two loads an FMA).
//
// The scatter adds into the CSR values with red.global.add.f64: the add runs
// in L2 instead of on the SM's FP64 pipe, and since the elements of one
// colour share no CSR row every entry receives one add per launch, so the
// result is deterministic.  One CTA of 192 threads per element (378 pairs in
// two rounds), persistent over the colour's element list.  Stages that
// follow one another share memory, 71 KB a CTA, so that three of them fill
// the gaps of each other's serial parts: H, the masses and the operands side
// by side left room for two (648 us instead of 575 us for 1,728 elements).
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "gb_device.h"
#include "gb_launch.cuh"

namespace gb {

namespace sf {

constexpr int NN = 27, NQ = 27, NP = 4, CENT = 20, NF = 7;
constexpr int NC = 16;  // sum-factorised contractions
enum { C_AB = 0, C_TV = 9, C_DA = 12, C_S1 = 13 };
// Their distinct values: phi_i phi_j = prod_d l_a l_b has 6 factors a
// direction (l_a l_b is symmetric), the advection term along direction d 9 in
// that one (l_a l'_b).
constexpr int SYM = 216, ADV = 324;
constexpr int NPAIR = 27 * 28 / 2;  // node pairs i <= j
constexpr int NT = 192;             // threads: two rounds of node pairs

struct Smem {
  double ell[2][3][3];   // [0] l_a(xi_g), [1] l'_a(xi_g)
  double pS[6][3];       // l_a l_b at xi_g, pair number sym[a*3+b]
  double pLD[9][3];      // l_a l'_b, index a*3+b
  double psidA[NP][NQ];
  double Bq[NQ][9];      // J^-1 [p][r]
  double dAq[NQ];
  double Mw[13][SYM];    // the contractions' values
  double S1[3][ADV];
  union {
    struct {             // fields at the nodes and, contracted, at the points
      double A[NF][2][NN];
      double B[NF][3][NN];
      double Xn[NF][NN];   // x y z u v w T at the nodes (lexicographic)
      double Xd[4][NN];    // u v w T time derivatives at the nodes (transient)
      double F[NF][4][NQ]; // value, d/dxi_1..3 at the points
    } iso;
    struct {
      double W[NC][NQ];      // weights of the sum-factorised contractions
      // residual of momentum a and energy 3: phi part, then the parts of the
      // reference gradients; contracted over the first and second direction
      double cR[4][4][NQ];
      double rP[4][3][NQ], rQ[4][2][NQ];
      double A[NC][81];   // contracted over the third direction [q12][pair]
      double B[13][3][36], BS[3][3][54];  // and the second [q1][pairs]
    } st;
    struct {
      double G[3][NQ][NN];   // d phi_L / d x_p at q
      double cG[3][NQ][NN];  // dA * G
    } g;
  } X;
  double Pn[NP];
  int sym[9];
  int lex[NN];    // lexicographic index of local node k
  int loc[NN];    // local node of lexicographic index L
  int nodes[NN];  // global node of local node k
};
// the points' set-up reads Xn, Xd and F while it writes W and cR
static_assert(offsetof(Smem, X.iso.Xn) >= offsetof(Smem, X.st.rP), "iso overlaps W, cR");

}  // namespace sf

template <bool ENERGY, bool JAC>
__global__ void __launch_bounds__(sf::NT, 3)
    assemble_sf_kernel(AsmArgs A, const SfTables *__restrict__ tb,
                       const int *__restrict__ elems, int nelem) {
  using namespace sf;
  constexpr int DIM = 3;
  constexpr int NV = DIM + (ENERGY ? 1 : 0);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &S = *reinterpret_cast<Smem *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x;
  const MaterialDev M = A.mat;

  // constant tables
  for (int t = tid; t < 18; t += nt) (&S.ell[0][0][0])[t] = (&tb->ell[0][0][0])[t];
  for (int t = tid; t < 27; t += nt) {
    const int a = t / 9, b = (t / 3) % 3, g = t % 3;
    const int lo = a < b ? a : b, u = lo * 3 - lo * (lo - 1) / 2 + (a < b ? b - a : a - b);
    S.pLD[a * 3 + b][g] = tb->pp[1][a * 3 + b][g];
    if (a <= b) S.pS[u][g] = tb->pp[0][a * 3 + b][g];
    S.sym[a * 3 + b] = u;
  }
  for (int t = tid; t < NN; t += nt) {
    S.lex[t] = tb->lex[t];
    S.loc[t] = tb->loc[t];
  }

  dependent_begin();
  for (int ei = blockIdx.x; ei < nelem; ei += gridDim.x) {
    const int e = elems[ei];
    const double rho_e = A.elem_rho ? A.elem_rho[e] : M.density;
    __syncthreads();  // the previous element is done with shared memory
    // ---- nodal data (lexicographic order)
    if (tid < NN) {
      const int k = tid, L = S.lex[k];
      const int n = A.conn[(int64_t)e * NN + k];
      S.nodes[k] = n;
      const int f0 = A.fu[n];
#pragma unroll
      for (int j = 0; j < DIM; j++) {
        S.X.iso.Xn[j][L] = A.coords[(int64_t)n * DIM + j];
        S.X.iso.Xn[3 + j][L] = A.x[f0 + j];
      }
      S.X.iso.Xn[6][L] = ENERGY ? A.x[f0 + DIM] : 0.0;
      if (k == CENT)
        for (int l = 0; l < NP; l++) S.Pn[l] = A.x[f0 + A.pofs + l];
      if (A.xdot) {
#pragma unroll
        for (int j = 0; j < DIM; j++) S.X.iso.Xd[j][L] = A.xdot[f0 + j];
        S.X.iso.Xd[3][L] = ENERGY ? A.xdot[f0 + DIM] : 0.0;
      }
    }
    __syncthreads();
    // ---- values and reference gradients at the points: three passes
    for (int t = tid; t < NF * 2 * 27; t += nt) {  // contract a1 -> q1 (l, l')
      const int f = t / 54, v = (t / 27) % 2, r = t % 27;
      const int a3 = r / 9, a2 = (r / 3) % 3, q1 = r % 3;
      const double *x = &S.X.iso.Xn[f][3 * a2 + 9 * a3];
      const double(*E)[3] = S.ell[v];
      S.X.iso.A[f][v][r] = E[0][q1] * x[0] + E[1][q1] * x[1] + E[2][q1] * x[2];
      (void)q1;
    }
    __syncthreads();
    for (int t = tid; t < NF * 3 * 27; t += nt) {  // contract a2 -> q2
      const int f = t / 81, w = (t / 27) % 3, r = t % 27;
      const int a3 = r / 9, q2 = (r / 3) % 3, q1 = r % 3;
      const int src = w == 2 ? 1 : 0;
      const double(*E)[3] = S.ell[w == 1 ? 1 : 0];
      const double *a = &S.X.iso.A[f][src][a3 * 9 + q1];
      S.X.iso.B[f][w][r] = E[0][q2] * a[0] + E[1][q2] * a[3] + E[2][q2] * a[6];
    }
    __syncthreads();
    for (int t = tid; t < NF * 4 * 27; t += nt) {  // contract a3 -> q3
      const int f = t / 108, d = (t / 27) % 4, q = t % 27;
      const int q3 = q / 9, q2 = (q / 3) % 3, q1 = q % 3;
      // d = 0 value, 1 d/dxi_1, 2 d/dxi_2, 3 d/dxi_3
      const int src = d == 1 ? 2 : (d == 2 ? 1 : 0);
      const double(*E)[3] = S.ell[d == 3 ? 1 : 0];
      const double *b = &S.X.iso.B[f][src][q2 * 3 + q1];
      S.X.iso.F[f][d][q] = E[0][q3] * b[0] + E[1][q3] * b[9] + E[2][q3] * b[18];
    }
    __syncthreads();
    // ---- per quadrature point (warp 0)
    if (warp == 0) {
      const int q = lane;
      double rc[NP] = {0.0, 0.0, 0.0, 0.0};
      bool bad = false;
      if (q < NQ) {
        double Jm[3][3], Gh[3][3], Th[3], v[3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
#pragma unroll
          for (int j = 0; j < 3; j++) {
            Jm[r][j] = S.X.iso.F[j][1 + r][q];
            Gh[r][j] = S.X.iso.F[3 + j][1 + r][q];
          }
          Th[r] = S.X.iso.F[6][1 + r][q];
          v[r] = S.X.iso.F[3 + r][0][q];
        }
        const double T = S.X.iso.F[6][0][q];
        const double c00 = Jm[1][1] * Jm[2][2] - Jm[1][2] * Jm[2][1];
        const double c01 = Jm[1][0] * Jm[2][2] - Jm[1][2] * Jm[2][0];
        const double c02 = Jm[1][0] * Jm[2][1] - Jm[1][1] * Jm[2][0];
        const double det = Jm[0][0] * c00 - Jm[0][1] * c01 + Jm[0][2] * c02;
        bad = !(det > 0.0);
        const double id = 1.0 / det;
        double B[3][3];
        B[0][0] = c00 * id;
        B[0][1] = -(Jm[0][1] * Jm[2][2] - Jm[2][1] * Jm[0][2]) * id;
        B[0][2] = (Jm[0][1] * Jm[1][2] - Jm[1][1] * Jm[0][2]) * id;
        B[1][0] = -c01 * id;
        B[1][1] = (Jm[0][0] * Jm[2][2] - Jm[2][0] * Jm[0][2]) * id;
        B[1][2] = -(Jm[0][0] * Jm[1][2] - Jm[1][0] * Jm[0][2]) * id;
        B[2][0] = c02 * id;
        B[2][1] = -(Jm[0][0] * Jm[2][1] - Jm[2][0] * Jm[0][1]) * id;
        B[2][2] = (Jm[0][0] * Jm[1][1] - Jm[1][0] * Jm[0][1]) * id;
        const double dA = A.tab_w[q] * det;
        double gv[3][3], gT[3];  // gv[p][a] = d v_a / d x_p
#pragma unroll
        for (int p = 0; p < 3; p++) {
#pragma unroll
          for (int a = 0; a < 3; a++)
            gv[p][a] = B[p][0] * Gh[0][a] + B[p][1] * Gh[1][a] + B[p][2] * Gh[2][a];
          gT[p] = B[p][0] * Th[0] + B[p][1] * Th[1] + B[p][2] * Th[2];
        }
        double psi[NP];
        psi[0] = 1.0;
        psi[1] = A.tab_pt[q % 3];
        psi[2] = A.tab_pt[(q % 9) / 3];
        psi[3] = A.tab_pt[q / 9];
        double P = 0.0;
#pragma unroll
        for (int l = 0; l < NP; l++) P = fma(S.Pn[l], psi[l], P);
        const double mu = M.viscosity, rho = rho_e;
        const double divv = gv[0][0] + gv[1][1] + gv[2][2];
        // time derivatives at the point (transient; load_fv's fv_dot)
        double vd[4] = {0.0, 0.0, 0.0, 0.0};
        if (A.xdot)
          for (int L = 0; L < NN; L++) {
            const double ph = __ldg(&tb->phi[q][L]);
#pragma unroll
            for (int c = 0; c < 4; c++) vd[c] = fma(ph, S.X.iso.Xd[c][L], vd[c]);
          }
#pragma unroll
        for (int l = 0; l < NP; l++) {
          S.psidA[l][q] = psi[l] * dA;
          rc[l] = psi[l] * dA * divv;
        }
#pragma unroll
        for (int a = 0; a < 3; a++) {
#pragma unroll
          for (int b = 0; b < 3; b++) S.X.st.W[C_AB + a * 3 + b][q] = -rho * dA * gv[b][a];
          S.X.st.W[C_TV + a][q] = ENERGY ? -rho * M.heat_capacity * dA * gT[a] : 0.0;
          S.X.st.W[C_S1 + a][q] = -rho * dA * (v[0] * B[0][a] + v[1] * B[1][a] + v[2] * B[2][a]);
          double f = M.source[a];
          if (M.source_model == GB_SOURCE_BOUSSINESQ)
            f = ENERGY ? rho * M.source[a] * (-M.beta * (T - M.Tref)) : 0.0;
          const double adv = v[0] * gv[0][a] + v[1] * gv[1][a] + v[2] * gv[2][a];
          // with the mass term -rho v_dot_a (src/mm_fill_momentum.c:471-500)
          S.X.st.cR[a][0][q] = dA * (f - rho * (adv + vd[a]));
          double t[3];
#pragma unroll
          for (int p = 0; p < 3; p++)
            t[p] = -dA * ((p == a ? -P : 0.0) + mu * (gv[a][p] + gv[p][a]));
#pragma unroll
          for (int r = 0; r < 3; r++)
            S.X.st.cR[a][1 + r][q] = B[0][r] * t[0] + B[1][r] * t[1] + B[2][r] * t[2];
        }
        S.X.st.W[C_DA][q] = dA;
        S.X.st.cR[3][0][q] = ENERGY ? -rho * M.heat_capacity * dA *
                                     (v[0] * gT[0] + v[1] * gT[1] + v[2] * gT[2] + vd[3])
                               : 0.0;
        const double kdA = ENERGY ? -M.conductivity * dA : 0.0;
#pragma unroll
        for (int r = 0; r < 3; r++)
          S.X.st.cR[3][1 + r][q] = kdA * (B[0][r] * gT[0] + B[1][r] * gT[1] + B[2][r] * gT[2]);
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
          for (int r = 0; r < 3; r++) S.Bq[q][p * 3 + r] = B[p][r];
        S.dAq[q] = dA;
      }
      // continuity residual rows and the det J status
#pragma unroll
      for (int l = 0; l < NP; l++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rc[l] += __shfl_xor_sync(0xffffffffu, rc[l], o);
      const unsigned anybad = __ballot_sync(0xffffffffu, bad);
      if (lane == 0) {
        if (anybad) {
          atomicAdd(A.status, 1);
          atomicMin(A.status + 1, e);
        }
        const int g0 = A.fu[S.nodes[CENT]] + A.pofs;
#pragma unroll
        for (int l = 0; l < NP; l++)
          if (!A.dbc[g0 + l]) atomicAdd(A.R + g0 + l, rc[l]);
      }
    }
    __syncthreads();
    // three contractions over the directions: masses and advection (A, B,
    // values), residual rows (rP, rQ, rows)
    constexpr int NRES = ENERGY ? 4 : 3;
    if (JAC) {
      for (int t = tid; t < NC * 81; t += nt) {
        const int c = t / 81, r = t % 81, q12 = r % 9, k3 = r / 9;
        if (k3 >= (c == C_S1 + 2 ? 9 : 6)) continue;
        const double *pp = c == C_S1 + 2 ? S.pLD[k3] : S.pS[k3];
        const double *w = &S.X.st.W[c][q12];
        S.X.st.A[c][k3 * 9 + q12] = pp[0] * w[0] + pp[1] * w[9] + pp[2] * w[18];
      }
    }
    for (int t = tid; t < NRES * 81; t += nt) {
      const int n = t / 81, p = (t / 27) % 3, r = t % 27, a1 = r % 3;
      const double *c = &S.X.st.cR[n][p == 0 ? 0 : 1 + p][r - a1];
      const double *l = S.ell[0][a1];
      double v = l[0] * c[0] + l[1] * c[1] + l[2] * c[2];
      if (p == 0) {
        const double *g = &S.X.st.cR[n][1][r - a1], *d = S.ell[1][a1];
        v += d[0] * g[0] + d[1] * g[1] + d[2] * g[2];
      }
      S.X.st.rP[n][p][r] = v;
    }
    __syncthreads();
    // ---- second direction; Dirichlet diagonals
    if (JAC) {
      for (int t = tid; t < 13 * 108; t += nt) {
        const int c = t / 108, r = t % 108, q1 = r / 36, k23 = r % 36;
        const double *pp = S.pS[k23 / 6], *A1 = &S.X.st.A[c][(k23 % 6) * 9 + q1];
        S.X.st.B[c][q1][k23] = pp[0] * A1[0] + pp[1] * A1[3] + pp[2] * A1[6];
      }
      for (int t = tid; t < 3 * 162; t += nt) {
        const int c = t / 162, r = t % 162, q1 = r / 54, k23 = r % 54;
        const int n3 = c == 2 ? 9 : 6, k2 = k23 / n3, k3 = k23 - k2 * n3;
        if (c == 0 && k2 >= 6) continue;
        const double *pp = c == 1 ? S.pLD[k2] : S.pS[k2];
        const double *A1 = &S.X.st.A[C_S1 + c][k3 * 9 + q1];
        S.X.st.BS[c][q1][k23] = pp[0] * A1[0] + pp[1] * A1[3] + pp[2] * A1[6];
      }
    }
    for (int t = tid; t < NRES * 54; t += nt) {
      const int n = t / 54, p = (t / 27) & 1, r = t % 27, a2 = (r / 3) % 3;
      const double *c = &S.X.st.rP[n][p ? 2 : 0][r - 3 * a2], *l = S.ell[0][a2];
      double v = l[0] * c[0] + l[1] * c[3] + l[2] * c[6];
      if (p == 0) {
        const double *g = &S.X.st.rP[n][1][r - 3 * a2], *d = S.ell[1][a2];
        v += d[0] * g[0] + d[1] * g[3] + d[2] * g[6];
      }
      S.X.st.rQ[n][p][r] = v;
    }
    if (JAC) {
      for (int t = tid; t < NN * NV + NP; t += nt) {
        int k, var;
        if (t < NN * NV) {
          k = t / NV;
          var = t - k * NV;
        } else {
          k = CENT;
          var = A.pofs + t - NN * NV;
        }
        const int nk = S.nodes[k];
        const int gr = A.fu[nk] + var;
        if (!A.dbc[gr]) continue;
        const int s = A.elem_nslot[(int64_t)e * NN * NN + k * NN + k];
        const int off = (ENERGY && var == DIM) ? A.nbr_offT[A.nbr_ptr[nk] + s]
                                               : A.nbr_off[A.nbr_ptr[nk] + s];
        atomicAdd(A.vals + A.rowptr[gr] + off + var, 1.0);
      }
    }
    __syncthreads();
    // ---- third direction
    for (int t = tid; t < NRES * NN; t += nt) {
      const int n = t / NN, L = t % NN, a3 = L / 9;
      const double *c = &S.X.st.rQ[n][0][L % 9], *g = &S.X.st.rQ[n][1][L % 9];
      const double *l = S.ell[0][a3], *d = S.ell[1][a3];
      const double v = l[0] * c[0] + l[1] * c[9] + l[2] * c[18] + d[0] * g[0] + d[1] * g[9] +
                       d[2] * g[18];
      const int gr = A.fu[S.nodes[S.loc[L]]] + n;
      if (!A.dbc[gr]) atomicAdd(A.R + gr, v);
    }
    if constexpr (JAC) {
    for (int t = tid; t < 13 * SYM; t += nt) {
      const int c = t / SYM, r = t % SYM, k23 = r % 36;
      const double *pp = S.pS[r / 36];
      S.Mw[c][r] = pp[0] * S.X.st.B[c][0][k23] + pp[1] * S.X.st.B[c][1][k23] +
                   pp[2] * S.X.st.B[c][2][k23];
    }
    for (int t = tid; t < 3 * ADV; t += nt) {
      const int c = t / ADV, r = t % ADV, n23 = c == 0 ? 36 : 54, k1 = r / n23, k23 = r - k1 * n23;
      const double *pp = c == 0 ? S.pLD[k1] : S.pS[k1];
      S.S1[c][r] = pp[0] * S.X.st.BS[c][0][k23] + pp[1] * S.X.st.BS[c][1][k23] +
                   pp[2] * S.X.st.BS[c][2][k23];
    }
    __syncthreads();
    // ---- physical gradients
    for (int t = tid; t < NQ * NN; t += nt) {
      const int q = t / NN, L = t - q * NN;
      const double *d = &tb->dref[q][L][0];
      const double d0 = __ldg(d), d1 = __ldg(d + 1), d2 = __ldg(d + 2);
      const double *B = S.Bq[q];
      const double dA = S.dAq[q];
#pragma unroll
      for (int p = 0; p < 3; p++) {
        const double g = B[3 * p] * d0 + B[3 * p + 1] * d1 + B[3 * p + 2] * d2;
        S.X.g.G[p][q][L] = g;
        S.X.g.cG[p][q][L] = dA * g;
      }
    }
    __syncthreads();
    // ---- node pairs (i, j), i <= j: the 3 x 3 block of H in registers, then
    // J(i, j) and J(j, i)
    {
      const double mu = M.viscosity, Cp = M.heat_capacity, kc = M.conductivity;
      double dfT[3];
#pragma unroll
      for (int a = 0; a < 3; a++)
        dfT[a] = (ENERGY && M.source_model == GB_SOURCE_BOUSSINESQ)
                     ? -rho_e * M.source[a] * M.beta
                     : 0.0;
      const uint16_t *ns = A.elem_nslot + (int64_t)e * NN * NN;
      const bool tr = A.mass_c != 0.0;
      for (int t = tid; t < NPAIR; t += nt) {
        const int pr = tb->pmap[t];
        const int Li = pr >> 5, Lj = pr & 31;
        double h[3][3];  // H((p, i), (r, j))
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
          for (int r = 0; r < 3; r++) h[p][r] = 0.0;
        const double *gi = &S.X.g.G[0][0][Li], *gj = &S.X.g.cG[0][0][Lj];
#pragma unroll 9
        for (int q = 0; q < NQ; q++) {
          double u[3], w[3];
#pragma unroll
          for (int p = 0; p < 3; p++) {
            u[p] = gi[(p * NQ + q) * NN];
            w[p] = gj[(p * NQ + q) * NN];
          }
#pragma unroll
          for (int p = 0; p < 3; p++)
#pragma unroll
            for (int r = 0; r < 3; r++) h[p][r] = fma(u[p], w[r], h[p][r]);
        }
        const int a1 = Li % 3, a2 = (Li / 3) % 3, a3 = Li / 9;
        const int b1 = Lj % 3, b2 = (Lj / 3) % 3, b3 = Lj / 9;
        const int s1 = S.sym[a1 * 3 + b1], s2 = S.sym[a2 * 3 + b2], s3 = S.sym[a3 * 3 + b3];
        const int m = (s1 * 6 + s2) * 6 + s3;
        const double trH = h[0][0] + h[1][1] + h[2][2];
        const double mdA = (ENERGY || tr) ? S.Mw[C_DA][m] : 0.0;
        // the mass terms' sensitivity -(1 + 2 theta) / dt rho M(dA)
        // (src/mm_fill_momentum.c:1586-1590), times Cp on the energy row
        const double Mt = tr ? -A.mass_c * rho_e * mdA : 0.0;
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
          for (int r = 0; r < 3; r++) h[p][r] *= -mu;
#pragma unroll 1
        for (int o = 0; o < (Li == Lj ? 1 : 2); o++) {  // rows of i, then of j
          const int ki = S.loc[o ? Lj : Li], kj = S.loc[o ? Li : Lj];
          const int f1 = o ? b1 * 3 + a1 : a1 * 3 + b1, f2 = o ? b2 * 3 + a2 : a2 * 3 + b2,
                    f3 = o ? b3 * 3 + a3 : a3 * 3 + b3;
          const double S1 = S.S1[0][(f1 * 6 + s2) * 6 + s3] + S.S1[1][(s1 * 9 + f2) * 6 + s3] +
                            S.S1[2][(s1 * 6 + s2) * 9 + f3];
          const double D = fma(-mu, trH, S1) + Mt;
          const int ni = S.nodes[ki];
          const int fi = A.fu[ni];
          const int nb = A.nbr_ptr[ni] + ns[ki * NN + kj];
          const int off = A.nbr_off[nb];
#pragma unroll
          for (int a = 0; a < 3; a++) {
            const int gr = fi + a;
            if (A.dbc[gr]) continue;
            double *row = A.vals + A.rowptr[gr] + off;
#pragma unroll
            for (int b = 0; b < 3; b++) {
              double v = (o ? h[a][b] : h[b][a]) + S.Mw[C_AB + a * 3 + b][m];
              if (a == b) v += D;
              atomicAdd(row + b, v);
            }
            if (ENERGY) atomicAdd(row + DIM, dfT[a] * mdA);
          }
          if (ENERGY) {
            const int gr = fi + DIM;
            if (!A.dbc[gr]) {
              double *row = A.vals + A.rowptr[gr] + A.nbr_offT[nb];
#pragma unroll
              for (int b = 0; b < 3; b++) atomicAdd(row + b, S.Mw[C_TV + b][m]);
              atomicAdd(row + DIM, fma(Cp, S1 + Mt, -kc * trH));
            }
          }
        }
      }
      // ---- J_mP / J_cv: two pressure modes of one (a, node)
      for (int t = tid; t < 3 * NN * 2; t += nt) {
        const int a = t / (NN * 2), L = (t >> 1) % NN, l0 = (t & 1) * 2;
        double s[2] = {0.0, 0.0};
#pragma unroll 9
        for (int q = 0; q < NQ; q++) {
          const double g = S.X.g.G[a][q][L];
          s[0] = fma(g, S.psidA[l0][q], s[0]);
          s[1] = fma(g, S.psidA[l0 + 1][q], s[1]);
        }
        const int k = S.loc[L], nk = S.nodes[k], nc = S.nodes[CENT];
        const int gr = A.fu[nk] + a, gc = A.fu[nc] + A.pofs + l0;
        double *row = A.vals + A.rowptr[gr] + A.nbr_off[A.nbr_ptr[nk] + ns[k * NN + CENT]] +
                      A.pofs + l0;
        const int oc = A.nbr_off[A.nbr_ptr[nc] + ns[CENT * NN + k]] + a;
#pragma unroll
        for (int l = 0; l < 2; l++) {
          if (!A.dbc[gr]) atomicAdd(row + l, s[l]);
          if (!A.dbc[gc + l]) atomicAdd(A.vals + A.rowptr[gc + l] + oc, s[l]);
        }
      }
    }
    }
  }
}

void build_sf_tables(const double *tab_phi, const double *tab_dphi, const int (*loc27)[3],
                     const double *ell, const double *dell, SfTables &T) {
  using namespace sf;
  for (int a = 0; a < 3; a++)
    for (int g = 0; g < 3; g++) {
      T.ell[0][a][g] = ell[a * 3 + g];
      T.ell[1][a][g] = dell[a * 3 + g];
    }
  for (int a = 0; a < 3; a++)
    for (int b = 0; b < 3; b++)
      for (int g = 0; g < 3; g++) {
        T.pp[0][a * 3 + b][g] = ell[a * 3 + g] * ell[b * 3 + g];
        T.pp[1][a * 3 + b][g] = ell[a * 3 + g] * dell[b * 3 + g];
      }
  for (int k = 0; k < NN; k++) {
    const int L = loc27[k][0] + 3 * loc27[k][1] + 9 * loc27[k][2];
    T.lex[k] = L;
    T.loc[L] = k;
  }
  for (int q = 0; q < NQ; q++)
    for (int L = 0; L < NN; L++) {
      const int k = T.loc[L];
      T.phi[q][L] = tab_phi[q * NN + k];
      for (int r = 0; r < 3; r++) T.dref[q][L][r] = tab_dphi[(q * NN + k) * 3 + r];
    }
  int e = 0;
  for (int i = 0; i < NN; i++)
    for (int j = i; j < NN; j++) T.pmap[e++] = (uint16_t)((i << 5) | j);
}

size_t assemble_sf_smem_bytes() { return sizeof(sf::Smem); }

template <bool ENERGY, bool JAC>
static cudaError_t launch_sf_t(const AsmArgs &a, const SfTables *tb, const int *elems,
                               int nelem, int grid_cap, cudaStream_t st) {
  const size_t sm = sizeof(sf::Smem);
  auto k = assemble_sf_kernel<ENERGY, JAC>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int grid = nelem < grid_cap ? nelem : grid_cap;
  if (grid <= 0) return cudaSuccess;
  launch_dependent(k, grid, sf::NT, sm, st, a, tb, elems, nelem);
  return cudaGetLastError();
}

cudaError_t launch_assemble_sf(const AsmArgs &a, bool energy, const SfTables *tb,
                               const int *elems, int nelem, int grid_cap, cudaStream_t st) {
  if (a.vals)
    return energy ? launch_sf_t<true, true>(a, tb, elems, nelem, grid_cap, st)
                  : launch_sf_t<false, true>(a, tb, elems, nelem, grid_cap, st);
  return energy ? launch_sf_t<true, false>(a, tb, elems, nelem, grid_cap, st)
                : launch_sf_t<false, false>(a, tb, elems, nelem, grid_cap, st);
}

}  // namespace gb
