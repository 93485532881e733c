// Species rows of the element residual and analytic Jacobian (dilute
// species, Galerkin; steady, or with the time-derivative terms of a
// transient step), in FP64 on sm_103a, with the coloured CSR scatter.
//
// Replaces, for these rows, assemble_mass_transport
// (src/mm_fill_species.c:194) with get_continuous_species_terms (:9739),
// fickian_flux (:12414) and the CONSTANT / USER species sources
// (:10117, :10146; the USER body is the Arrhenius rate of the problem
// description).  The species variable form is SPECIES_UNDEFINED_FORM (the
// reader's default, src/mm_as_alloc.c:140), so coeff_rho = 1:
//   R_w[i] = sum_q dA [ -phi_i (v . grad Y_w) + grad phi_i . (-D_w grad Y_w)
//                       + phi_i S_w ]
//   dR_w[i]/dY_w1[j] = dA [ (w == w1) (-phi_i v . grad phi_j
//                                     - D_w grad phi_i . grad phi_j)
//                           + phi_i phi_j dS_w/dY_w1 ]
//   dR_w[i]/dv_b[j]  = -dA phi_i phi_j dY_w/dx_b
//   dR_w[i]/dT[j]    =  dA phi_i phi_j dS_w/dT
// The momentum, continuity and energy rows do not depend on the species
// (constant density, no heat of reaction), so the flow kernels need not
// know about them; this kernel runs after the flow kernel of the same
// colour and writes only species rows.
//
// Work decomposition of the dense kernel (2-D elements, and path 1) mirrors the flow kernel: one CTA per element in 3-D,
// three in 2-D; phase 1 per quadrature point (geometry, fields, source),
// phase 2 per (quadrature point, node) (physical gradients), phase 3 per
// (i, j) node pairs, one species row block at a time to bound registers,
// then the scatter.  Elements of a colour share no node: no atomics.
#include <cuda_runtime.h>

#include <cstdint>

#include "gb_device.h"
#include "gb_launch.cuh"
#include "gb_element.cuh"

namespace gb {

namespace sp {

constexpr int MS = GB_MAX_SPECIES;

template <int DIM>
struct QPs {
  double dA;
  double B[DIM][DIM];
  double v[DIM];
  double gY[MS][DIM];
  double S[MS], dSdT[MS], dSdY[MS][MS];
  double Yd[MS];  // time derivatives (transient)
};

template <int DIM>
struct QNs {
  double phi;
  double g[DIM];
  double vg;  // v . grad phi
};

template <int DIM>
struct Elem {
  double X[Q2<DIM>::NN][DIM];
  double U[Q2<DIM>::NN][DIM];
  double Tn[Q2<DIM>::NN];
  double Yn[MS][Q2<DIM>::NN];
  double Ydn[MS][Q2<DIM>::NN];  // nodal time derivatives (transient)
  int nodes[Q2<DIM>::NN];
  int e;
  QPs<DIM> qp[Q2<DIM>::NQ];
  QNs<DIM> qn[Q2<DIM>::NQ][Q2<DIM>::NN];
};

}  // namespace sp

template <int DIM, bool ENERGY, bool JAC>
__global__ void __launch_bounds__(256)
    assemble_species_kernel(AsmArgs A, const int *__restrict__ elems, int nelem) {
  using C = Q2<DIM>;
  using sp::MS;
  constexpr int NN = C::NN, NQ = C::NQ, TPE = C::TPE, EPB = C::EPB, PPT = C::PPT;
  constexpr int OY = DIM + (ENERGY ? 1 : 0);  // offset of Y_0 among a node's unknowns
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Elem = sp::Elem<DIM>;
  Elem *S = reinterpret_cast<Elem *>(smem_raw);
  const int tid = threadIdx.x;
  const int slot = tid / TPE;
  const int lt = tid - slot * TPE;
  const int ebase = blockIdx.x * EPB;
  const bool thread_live = tid < TPE * EPB && ebase + slot < nelem;
  const double *__restrict__ tab_phi = A.tab_phi;
  const double *__restrict__ tab_dphi = A.tab_dphi;
  const MaterialDev &M = A.mat;
  const int ns = M.nspec;

  // ---- load element data
  for (int t = tid; t < EPB * NN; t += blockDim.x) {
    const int s = t / NN, k = t - s * NN;
    if (ebase + s >= nelem) continue;
    const int e = elems[ebase + s];
    const int n = A.conn[(int64_t)e * NN + k];
    Elem &E = S[s];
    E.nodes[k] = n;
    if (k == 0) E.e = e;
    const int f0 = A.fu[n];
#pragma unroll
    for (int j = 0; j < DIM; j++) {
      E.X[k][j] = A.coords[(int64_t)n * DIM + j];
      E.U[k][j] = A.x[f0 + j];
    }
    E.Tn[k] = ENERGY ? A.x[f0 + DIM] : 0.0;
    for (int w = 0; w < ns; w++) E.Yn[w][k] = A.x[f0 + OY + w];
    for (int w = 0; w < ns; w++) E.Ydn[w][k] = A.xdot ? A.xdot[f0 + OY + w] : 0.0;
  }
  __syncthreads();

  // ---- phase 1: one thread per quadrature point
  for (int t = tid; t < EPB * NQ; t += blockDim.x) {
    const int s = t / NQ, q = t - s * NQ;
    if (ebase + s >= nelem) continue;
    Elem &E = S[s];
    sp::QPs<DIM> &Q = E.qp[q];
    double Jm[DIM][DIM], v[DIM], T = 0.0, Y[MS], Yh[MS][DIM];
#pragma unroll
    for (int i = 0; i < DIM; i++) {
      v[i] = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; j++) Jm[i][j] = 0.0;
    }
#pragma unroll
    for (int w = 0; w < MS; w++) {
      Y[w] = 0.0;
#pragma unroll
      for (int i = 0; i < DIM; i++) Yh[w][i] = 0.0;
    }
    for (int k = 0; k < NN; k++) {
      const double ph = tab_phi[q * NN + k];
      double dph[DIM];
#pragma unroll
      for (int i = 0; i < DIM; i++) dph[i] = tab_dphi[(q * NN + k) * DIM + i];
#pragma unroll
      for (int i = 0; i < DIM; i++)
#pragma unroll
        for (int j = 0; j < DIM; j++) Jm[i][j] = fma(dph[i], E.X[k][j], Jm[i][j]);
#pragma unroll
      for (int a = 0; a < DIM; a++) v[a] = fma(ph, E.U[k][a], v[a]);
      if (ENERGY) T = fma(ph, E.Tn[k], T);
#pragma unroll
      for (int w = 0; w < MS; w++) {
        if (w >= ns) break;
        const double yk = E.Yn[w][k];
        Y[w] = fma(ph, yk, Y[w]);
#pragma unroll
        for (int i = 0; i < DIM; i++) Yh[w][i] = fma(dph[i], yk, Yh[w][i]);
      }
    }
    double det, B[DIM][DIM];
    if (DIM == 2) {
      det = Jm[0][0] * Jm[1][1] - Jm[0][1] * Jm[1][0];
      B[0][0] = Jm[1][1] / det;
      B[1][1] = Jm[0][0] / det;
      B[0][1] = -Jm[0][1] / det;
      B[1][0] = -Jm[1][0] / det;
    } else {
      const double c00 = Jm[1][1] * Jm[2][2] - Jm[1][2] * Jm[2][1];
      const double c01 = Jm[1][0] * Jm[2][2] - Jm[1][2] * Jm[2][0];
      const double c02 = Jm[1][0] * Jm[2][1] - Jm[1][1] * Jm[2][0];
      det = Jm[0][0] * c00 - Jm[0][1] * c01 + Jm[0][2] * c02;
      B[0][0] = c00 / det;
      B[0][1] = -(Jm[0][1] * Jm[2][2] - Jm[2][1] * Jm[0][2]) / det;
      B[0][2] = (Jm[0][1] * Jm[1][2] - Jm[1][1] * Jm[0][2]) / det;
      B[1][0] = -c01 / det;
      B[1][1] = (Jm[0][0] * Jm[2][2] - Jm[2][0] * Jm[0][2]) / det;
      B[1][2] = -(Jm[0][0] * Jm[1][2] - Jm[1][0] * Jm[0][2]) / det;
      B[2][0] = c02 / det;
      B[2][1] = -(Jm[0][0] * Jm[2][1] - Jm[2][0] * Jm[0][1]) / det;
      B[2][2] = (Jm[0][0] * Jm[1][1] - Jm[1][0] * Jm[0][1]) / det;
    }
    Q.dA = A.tab_w[q] * det;
#pragma unroll
    for (int p = 0; p < DIM; p++) {
      Q.v[p] = v[p];
#pragma unroll
      for (int i = 0; i < DIM; i++) Q.B[p][i] = B[p][i];
    }
#pragma unroll
    for (int w = 0; w < MS; w++) {
      if (w >= ns) break;
#pragma unroll
      for (int p = 0; p < DIM; p++) {
        double g = 0.0;
#pragma unroll
        for (int i = 0; i < DIM; i++) g = fma(B[p][i], Yh[w][i], g);
        Q.gY[w][p] = g;
      }
      // source and its sensitivities (CONSTANT: src/mm_fill_species.c:10117;
      // USER Arrhenius S = nu k0 exp(-E/T) Y_s: :10146-10190)
      double Sw = 0.0, dT = 0.0;
      for (int w1 = 0; w1 < MS; w1++) Q.dSdY[w][w1] = 0.0;
      if (M.ssm[w] == GB_SPECIES_SOURCE_CONSTANT) {
        Sw = M.ssp[w][0];
      } else if (M.ssm[w] == GB_SPECIES_SOURCE_ARRHENIUS) {
        const int src = (int)M.ssp[w][3];
        const double r = M.ssp[w][0] * exp(-M.ssp[w][1] / T);
        double ys = 0.0;
        for (int w1 = 0; w1 < MS; w1++)
          if (w1 == src) ys = Y[w1];
        Sw = M.ssp[w][2] * r * ys;
        dT = Sw * M.ssp[w][1] / (T * T);
        Q.dSdY[w][src] = M.ssp[w][2] * r;
      }
      Q.S[w] = Sw;
      Q.dSdT[w] = dT;
      double yd = 0.0;
      if (A.xdot)
        for (int k = 0; k < NN; k++) yd = fma(tab_phi[q * NN + k], E.Ydn[w][k], yd);
      Q.Yd[w] = yd;
    }
  }
  __syncthreads();

  // ---- phase 2: one thread per (quadrature point, node)
  for (int t = tid; t < EPB * NQ * NN; t += blockDim.x) {
    const int s = t / (NQ * NN), r = t - s * (NQ * NN), q = r / NN, k = r - q * NN;
    if (ebase + s >= nelem) continue;
    Elem &E = S[s];
    const sp::QPs<DIM> &Q = E.qp[q];
    sp::QNs<DIM> &W = E.qn[q][k];
    double dph[DIM], vg = 0.0;
#pragma unroll
    for (int i = 0; i < DIM; i++) dph[i] = tab_dphi[(q * NN + k) * DIM + i];
#pragma unroll
    for (int p = 0; p < DIM; p++) {
      double g = 0.0;
#pragma unroll
      for (int i = 0; i < DIM; i++) g = fma(Q.B[p][i], dph[i], g);
      W.g[p] = g;
      vg = fma(Q.v[p], g, vg);
    }
    W.phi = tab_phi[q * NN + k];
    W.vg = vg;
  }
  __syncthreads();
  if (!thread_live) return;

  Elem &E = S[slot];
  const int e = E.e;
  const int *nodes = E.nodes;
  const uint16_t *nslot = A.elem_nslot + (int64_t)e * NN * NN;

  // ---- residual rows (w, i): one thread each; Dirichlet rows get their
  // diagonal 1 instead (put_dirichlet_in_matrix, src/bc_dirich.c:44)
  if (lt < ns * NN) {
    const int w = lt / NN, i = lt - (lt / NN) * NN;
    const double nD = -M.diff[w];
    double Racc = 0.0;
    for (int q = 0; q < NQ; q++) {
      const sp::QPs<DIM> &Q = E.qp[q];
      const sp::QNs<DIM> &Wi = E.qn[q][i];
      double vgY = 0.0, dif = 0.0;
#pragma unroll
      for (int p = 0; p < DIM; p++) {
        vgY = fma(Q.v[p], Q.gY[w][p], vgY);
        dif = fma(Wi.g[p], nD * Q.gY[w][p], dif);
      }
      // with the mass term -Y_dot_w phi_i dA (coeff_rho = 1,
      // src/mm_fill_species.c:525-551)
      Racc += (-(vgY + Q.Yd[w]) * Wi.phi + dif + Q.S[w] * Wi.phi) * Q.dA;
    }
    const int node = nodes[i];
    const int gr = A.fu[node] + OY + w;
    if (A.dbc[gr]) {
      if (JAC) {
        const int s = nslot[i * NN + i];
        A.vals[A.rowptr[gr] + A.nbr_off[A.nbr_ptr[node] + s] + OY + w] += 1.0;
      }
    } else {
      A.R[gr] += Racc;
    }
  }
  if (!JAC) return;

  // ---- Jacobian node pairs, one species row block at a time
  const int pi = lt / (NN / PPT);
  const int pj0 = lt - pi * (NN / PPT);
  const int ni = nodes[pi];
  const int nb0 = A.nbr_ptr[ni];
  for (int w = 0; w < ns; w++) {
    const int gr = A.fu[ni] + OY + w;
    if (A.dbc[gr]) continue;  // uniform per thread: the row belongs to node pi
    const double nD = -M.diff[w];
    double JYY[PPT][MS], JYv[PPT][DIM], JYT[PPT];
#pragma unroll
    for (int m = 0; m < PPT; m++) {
      JYT[m] = 0.0;
#pragma unroll
      for (int b = 0; b < DIM; b++) JYv[m][b] = 0.0;
#pragma unroll
      for (int w1 = 0; w1 < MS; w1++) JYY[m][w1] = 0.0;
    }
    for (int q = 0; q < NQ; q++) {
      const sp::QPs<DIM> &Q = E.qp[q];
      const sp::QNs<DIM> &Wi = E.qn[q][pi];
      const double dA = Q.dA;
      double ngY[DIM], dSdY[MS];
#pragma unroll
      for (int b = 0; b < DIM; b++) ngY[b] = -Q.gY[w][b];
#pragma unroll
      for (int w1 = 0; w1 < MS; w1++) dSdY[w1] = Q.dSdY[w][w1];
      const double dSdT = Q.dSdT[w];
#pragma unroll
      for (int m = 0; m < PPT; m++) {
        const sp::QNs<DIM> &Wj = E.qn[q][pj0 + m * (NN / PPT)];
        double dot = 0.0;
#pragma unroll
        for (int p = 0; p < DIM; p++) dot = fma(Wi.g[p], Wj.g[p], dot);
        const double pij = Wi.phi * Wj.phi * dA;
        // with the mass term's sensitivity -(1 + 2 theta) / dt phi_i phi_j dA
        const double diag = fma(-Wi.phi, Wj.vg, nD * dot) * dA - A.mass_c * pij;
#pragma unroll
        for (int w1 = 0; w1 < MS; w1++)
          JYY[m][w1] = fma(dSdY[w1], pij, JYY[m][w1] + (w1 == w ? diag : 0.0));
#pragma unroll
        for (int b = 0; b < DIM; b++) JYv[m][b] = fma(ngY[b], pij, JYv[m][b]);
        JYT[m] = fma(dSdT, pij, JYT[m]);
      }
    }
    const int64_t rb = A.rowptr[gr];
#pragma unroll
    for (int m = 0; m < PPT; m++) {
      const int pj = pj0 + m * (NN / PPT);
      const int64_t base = rb + A.nbr_off[nb0 + nslot[pi * NN + pj]];
#pragma unroll
      for (int b = 0; b < DIM; b++) A.vals[base + b] += JYv[m][b];
      if (ENERGY) A.vals[base + DIM] += JYT[m];
#pragma unroll
      for (int w1 = 0; w1 < MS; w1++)
        if (w1 < ns) A.vals[base + OY + w1] += JYY[m][w1];
    }
  }
}

// ------------------------------------------------------------ 3-D
//
// The same rows for HEX27 elements with the fewest FP64 operations.  The dense
// kernel above needs 27 points x 729 node pairs x ~15 operations for every
// species row, 4.3 of the 5.3 ms of a 16 x 16 x 8 reacting channel's assembly,
// and GB300's FP64 rate bounds it.  Every term is a weighted sum of products of
// 1-D factors over the three directions, phi_i phi_j = prod_d l l, and a
// direction's factor has few distinct values: l_a l_b and l'_a l'_b are
// symmetric (6), l_a l'_b and l'_a l_b are not (9).  Contracting one direction
// at a time:
//   mass matrices (velocity, temperature and source sensitivities): 216
//     values, 1.1K FMA each;
//   advection S1 = sum phi_i (-dA v . grad phi_j): three of 324 values;
//   diffusion K = sum dA grad phi_i . grad phi_j through K_ab = dA B_a . B_b:
//     one of 216 values (a = b) and three of 486 (a < b, and their transposes).
// About 60K FMA an element with two species, against ~1M.  One CTA per element,
// persistent over the colour's list; the adds into the CSR rows run in L2
// (red.global.add), one per entry and launch.

namespace sp {

constexpr int Q = 27, SYM = 216, ADV = 324, MIX = 486;

struct Smem3 {
  // 1-D pair factors [pair][point]: l_a l_b, l'_a l'_b (6 each), l_a l'_b,
  // l'_a l_b (9 each)
  double pS[6][3], pD[6][3], pLD[9][3], pDL[9][3];
  double ell[2][3][3];
  double phi[Q][Q];
  double Xn[7 + MS][Q];      // x y z u v w T Y at the nodes, lexicographic
  double Yd[MS][Q];          // time derivatives
  union {
    struct {
      double A[7 + MS][2][Q], B[7 + MS][3][Q];
    } pass;
    struct {
      double A[10][9][9], B[10][3][81];
    } st;
  } u;
  double F[7 + MS][4][Q];    // value, d/dxi at the points
  double wS[3][Q], wK[6][Q], wM[Q];  // weights: S1, K_ab, dA
  double wY[MS][5][Q];       // per species: three velocities, T, its source species
  double cR[MS][4][Q];       // residual: phi part, reference-gradient parts
  double rP[MS][3][Q], rQ[MS][2][Q];
  double S1[3][ADV], KS[SYM], KM[3][MIX], Mm[SYM];
  double Mw[5][SYM];
  int sym[9];
  int lex[Q], loc[Q], nodes[Q];
};

}  // namespace sp

template <bool ENERGY, bool JAC>
__global__ void __launch_bounds__(256, 2)
    assemble_species_sf_kernel(AsmArgs A, const SfTables *__restrict__ tb,
                               const int *__restrict__ elems, int nelem) {
  using namespace sp;
  constexpr int NT = 256, OY = 3 + (ENERGY ? 1 : 0);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem3 &S = *reinterpret_cast<Smem3 *>(smem_raw);
  const int tid = threadIdx.x;
  const MaterialDev &M = A.mat;
  const int ns = M.nspec, nf = 7 + ns;
  // tables
  for (int t = tid; t < 18; t += NT) (&S.ell[0][0][0])[t] = (&tb->ell[0][0][0])[t];
  for (int t = tid; t < Q * Q; t += NT) (&S.phi[0][0])[t] = (&tb->phi[0][0])[t];
  for (int t = tid; t < Q; t += NT) {
    S.lex[t] = tb->lex[t];
    S.loc[t] = tb->loc[t];
  }
  if (tid < 27) {
    const int ab = tid / 3, g = tid % 3, a = ab / 3, b = ab % 3;
    const double la = tb->ell[0][a][g], lb = tb->ell[0][b][g];
    const double da = tb->ell[1][a][g], db = tb->ell[1][b][g];
    const int lo = min(a, b), u = lo * 3 - lo * (lo - 1) / 2 + max(a, b) - lo;
    S.pLD[ab][g] = la * db;
    S.pDL[ab][g] = da * lb;
    if (a <= b) {
      S.pS[u][g] = la * lb;
      S.pD[u][g] = da * db;
    }
    S.sym[ab] = u;
  }
  // contraction number c of a group: the factors of direction d (0..2)
  // shared group: 0-2 S1 along c, 3-5 K_cc, 6-8 K_ab (01, 02, 12), 9 dA
  auto factor = [&](int c, int d, int &n) -> const double(*)[3] {
    n = 6;
    if (c < 3 && d == c) {
      n = 9;
      return S.pLD;
    }
    if (c >= 3 && c < 6 && d == c - 3) return S.pD;
    if (c >= 6 && c < 9) {
      const int a = c == 8 ? 1 : 0, b = c == 6 ? 1 : 2;
      if (d == a || d == b) {
        n = 9;
        return d == a ? S.pDL : S.pLD;
      }
    }
    return S.pS;
  };

  dependent_begin();
  for (int ei = blockIdx.x; ei < nelem; ei += gridDim.x) {
    const int e = elems[ei];
    __syncthreads();  // the previous element is done with shared memory
    if (tid < Q) {
      const int k = tid, L = S.lex[k], n = A.conn[(int64_t)e * Q + k], f0 = A.fu[n];
      S.nodes[k] = n;
#pragma unroll
      for (int j = 0; j < 3; j++) {
        S.Xn[j][L] = A.coords[(int64_t)n * 3 + j];
        S.Xn[3 + j][L] = A.x[f0 + j];
      }
      S.Xn[6][L] = ENERGY ? A.x[f0 + 3] : 0.0;
      for (int w = 0; w < ns; w++) {
        S.Xn[7 + w][L] = A.x[f0 + OY + w];
        if (A.xdot) S.Yd[w][L] = A.xdot[f0 + OY + w];
      }
    }
    __syncthreads();
    // values and reference gradients at the points, one direction at a time
    for (int t = tid; t < nf * 54; t += NT) {
      const int f = t / 54, v = (t / 27) & 1, r = t % 27;
      const double *x = &S.Xn[f][3 * (r / 3)];
      const double(*l)[3] = S.ell[v];
      const int q1 = r % 3;
      S.u.pass.A[f][v][r] = l[0][q1] * x[0] + l[1][q1] * x[1] + l[2][q1] * x[2];
    }
    __syncthreads();
    for (int t = tid; t < nf * 81; t += NT) {
      const int f = t / 81, w = (t / 27) % 3, r = t % 27, q2 = (r / 3) % 3;
      const double *a = &S.u.pass.A[f][w == 2 ? 1 : 0][(r / 9) * 9 + r % 3];
      const double(*l)[3] = S.ell[w == 1 ? 1 : 0];
      S.u.pass.B[f][w][r] = l[0][q2] * a[0] + l[1][q2] * a[3] + l[2][q2] * a[6];
    }
    __syncthreads();
    for (int t = tid; t < nf * 108; t += NT) {
      const int f = t / 108, d = (t / 27) & 3, q = t % 27, q3 = q / 9;
      const double *b = &S.u.pass.B[f][d == 1 ? 2 : (d == 2 ? 1 : 0)][q % 9];
      const double(*l)[3] = S.ell[d == 3 ? 1 : 0];
      S.F[f][d][q] = l[0][q3] * b[0] + l[1][q3] * b[9] + l[2][q3] * b[18];
    }
    __syncthreads();
    // per quadrature point and species
    for (int t = tid; t < Q * ns; t += NT) {
      const int w = t / Q, q = t % Q;
      double J[3][3];
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int j = 0; j < 3; j++) J[r][j] = S.F[j][1 + r][q];
      const double c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
      const double c01 = J[1][0] * J[2][2] - J[1][2] * J[2][0];
      const double c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
      const double det = J[0][0] * c00 - J[0][1] * c01 + J[0][2] * c02, id = 1.0 / det;
      double B[3][3];
      B[0][0] = c00 * id;
      B[0][1] = -(J[0][1] * J[2][2] - J[2][1] * J[0][2]) * id;
      B[0][2] = (J[0][1] * J[1][2] - J[1][1] * J[0][2]) * id;
      B[1][0] = -c01 * id;
      B[1][1] = (J[0][0] * J[2][2] - J[2][0] * J[0][2]) * id;
      B[1][2] = -(J[0][0] * J[1][2] - J[1][0] * J[0][2]) * id;
      B[2][0] = c02 * id;
      B[2][1] = -(J[0][0] * J[2][1] - J[2][0] * J[0][1]) * id;
      B[2][2] = (J[0][0] * J[1][1] - J[1][0] * J[0][1]) * id;
      const double dA = A.tab_w[q] * det;
      const double v[3] = {S.F[3][0][q], S.F[4][0][q], S.F[5][0][q]}, T = S.F[6][0][q];
      double gY[3];
#pragma unroll
      for (int p = 0; p < 3; p++)
        gY[p] = B[p][0] * S.F[7 + w][1][q] + B[p][1] * S.F[7 + w][2][q] +
                B[p][2] * S.F[7 + w][3][q];
      if (JAC && w == 0) {
        S.wM[q] = dA;
#pragma unroll
        for (int r = 0; r < 3; r++)
          S.wS[r][q] = -dA * (v[0] * B[0][r] + v[1] * B[1][r] + v[2] * B[2][r]);
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
          for (int b = a; b < 3; b++)
            S.wK[a == b ? a : 2 + a + b][q] =
                dA * (B[0][a] * B[0][b] + B[1][a] * B[1][b] + B[2][a] * B[2][b]);
      }
      // source and its sensitivities (CONSTANT: src/mm_fill_species.c:10117;
      // USER Arrhenius S = nu k0 exp(-E/T) Y_s: :10146-10190)
      double Sw = 0.0, dT = 0.0, dY = 0.0;
      if (M.ssm[w] == GB_SPECIES_SOURCE_CONSTANT) {
        Sw = M.ssp[w][0];
      } else if (M.ssm[w] == GB_SPECIES_SOURCE_ARRHENIUS) {
        dY = M.ssp[w][2] * (M.ssp[w][0] * exp(-M.ssp[w][1] / T));
        Sw = dY * S.F[7 + (int)M.ssp[w][3]][0][q];
        dT = Sw * M.ssp[w][1] / (T * T);
      }
      double yd = 0.0;
      if (A.xdot)
        for (int L = 0; L < Q; L++) yd = fma(S.phi[q][L], S.Yd[w][L], yd);
      // with the mass term -Y_dot_w phi_i dA (coeff_rho = 1,
      // src/mm_fill_species.c:525-551)
      S.cR[w][0][q] = dA * (Sw - (v[0] * gY[0] + v[1] * gY[1] + v[2] * gY[2] + yd));
      const double nD = -M.diff[w] * dA;
#pragma unroll
      for (int r = 0; r < 3; r++)
        S.cR[w][1 + r][q] = nD * (B[0][r] * gY[0] + B[1][r] * gY[1] + B[2][r] * gY[2]);
      if (JAC) {
#pragma unroll
        for (int b = 0; b < 3; b++) S.wY[w][b][q] = -dA * gY[b];
        S.wY[w][3][q] = dA * dT;
        S.wY[w][4][q] = dA * dY;
      }
    }
    __syncthreads();
    // three passes over the directions: the residual rows, the contractions of
    // the shared group (A, B, then the values), then each species' masses
    const bool tr = A.mass_c != 0.0;
    const int nc = JAC ? (tr ? 10 : 9) : 0;
    for (int t = tid; t < ns * 81; t += NT) {
      const int w = t / 81, p = (t / 27) % 3, r = t % 27, q23 = r / 3, a1 = r % 3;
      const double *c = &S.cR[w][p == 0 ? 0 : 1 + p][3 * q23];
      double v = S.ell[0][a1][0] * c[0] + S.ell[0][a1][1] * c[1] + S.ell[0][a1][2] * c[2];
      if (p == 0) {
        const double *g = &S.cR[w][1][3 * q23];
        v += S.ell[1][a1][0] * g[0] + S.ell[1][a1][1] * g[1] + S.ell[1][a1][2] * g[2];
      }
      S.rP[w][p][3 * q23 + a1] = v;
    }
    for (int t = tid; t < nc * 81; t += NT) {
      const int c = t / 81, r = t % 81, q12 = r / 9, k3 = r % 9;
      int n3;
      const double(*f)[3] = factor(c, 2, n3);
      if (k3 >= n3) continue;
      const double *w = c < 3 ? &S.wS[c][q12] : (c < 9 ? &S.wK[c - 3][q12] : &S.wM[q12]);
      S.u.st.A[c][q12][k3] = f[k3][0] * w[0] + f[k3][1] * w[9] + f[k3][2] * w[18];
    }
    __syncthreads();
    for (int t = tid; t < ns * 54; t += NT) {
      const int w = t / 54, p = (t / 27) & 1, r = t % 27, q3 = r / 9, a2 = (r / 3) % 3;
      const double *c = &S.rP[w][p ? 2 : 0][9 * q3 + r % 3];
      double v = S.ell[0][a2][0] * c[0] + S.ell[0][a2][1] * c[3] + S.ell[0][a2][2] * c[6];
      if (p == 0) {
        const double *g = &S.rP[w][1][9 * q3 + r % 3];
        v += S.ell[1][a2][0] * g[0] + S.ell[1][a2][1] * g[3] + S.ell[1][a2][2] * g[6];
      }
      S.rQ[w][p][r] = v;
    }
    for (int t = tid; t < nc * 243; t += NT) {
      const int c = t / 243, r = t % 243, q1 = r / 81, k23 = r % 81;
      int n2, n3;
      const double(*f)[3] = factor(c, 1, n2);
      factor(c, 2, n3);
      if (k23 >= n2 * n3) continue;
      const int k2 = k23 / n3, k3 = k23 - k2 * n3;
      S.u.st.B[c][q1][k23] = f[k2][0] * S.u.st.A[c][q1][k3] + f[k2][1] * S.u.st.A[c][q1 + 3][k3] +
                             f[k2][2] * S.u.st.A[c][q1 + 6][k3];
    }
    __syncthreads();
    for (int t = tid; t < ns * Q; t += NT) {
      const int w = t / Q, L = t % Q, a3 = L / 9;
      const double *c = &S.rQ[w][0][L % 9], *g = &S.rQ[w][1][L % 9];
      const double v = S.ell[0][a3][0] * c[0] + S.ell[0][a3][1] * c[9] + S.ell[0][a3][2] * c[18] +
                       S.ell[1][a3][0] * g[0] + S.ell[1][a3][1] * g[9] + S.ell[1][a3][2] * g[18];
      const int k = S.loc[L], gr = A.fu[S.nodes[k]] + OY + w;
      // a Dirichlet row gets its diagonal 1 instead (put_dirichlet_in_matrix,
      // src/bc_dirich.c:44)
      if (!A.dbc[gr]) {
        atomicAdd(A.R + gr, v);
      } else if (JAC) {
        const int s = A.elem_nslot[(int64_t)e * Q * Q + k * Q + k];
        atomicAdd(A.vals + A.rowptr[gr] + A.nbr_off[A.nbr_ptr[S.nodes[k]] + s] + OY + w, 1.0);
      }
    }
    if constexpr (JAC) {
      auto last = [&](int c, int k1, int k23) {
        int n;
        const double(*f)[3] = factor(c, 0, n);
        return f[k1][0] * S.u.st.B[c][0][k23] + f[k1][1] * S.u.st.B[c][1][k23] +
               f[k1][2] * S.u.st.B[c][2][k23];
      };
      for (int t = tid; t < 3 * ADV; t += NT) {
        const int c = t / ADV, r = t % ADV, n23 = c == 0 ? 36 : 54;
        S.S1[c][r] = last(c, r / n23, r % n23);
      }
      for (int t = tid; t < SYM; t += NT) {
        const int k1 = t / 36, k23 = t % 36;
        S.KS[t] = last(3, k1, k23) + last(4, k1, k23) + last(5, k1, k23);
        if (tr) S.Mm[t] = last(9, k1, k23);
      }
      for (int t = tid; t < 3 * MIX; t += NT) {
        const int c = t / MIX, r = t % MIX, n23 = c == 2 ? 81 : 54;
        S.KM[c][r] = last(6 + c, r / n23, r % n23);
      }
      for (int w = 0; w < ns; w++) {
        __syncthreads();  // the groups before are done with the stages
        for (int t = tid; t < 5 * 54; t += NT) {
          const int c = t / 54, q12 = (t % 54) / 6, k3 = t % 6;
          const double *x = &S.wY[w][c][q12], *f = S.pS[k3];
          S.u.st.A[c][q12][k3] = f[0] * x[0] + f[1] * x[9] + f[2] * x[18];
        }
        __syncthreads();
        for (int t = tid; t < 5 * 108; t += NT) {
          const int c = t / 108, q1 = (t % 108) / 36, k23 = t % 36, k3 = k23 % 6;
          const double *f = S.pS[k23 / 6];
          S.u.st.B[c][q1][k23] = f[0] * S.u.st.A[c][q1][k3] + f[1] * S.u.st.A[c][q1 + 3][k3] +
                                 f[2] * S.u.st.A[c][q1 + 6][k3];
        }
        __syncthreads();
        for (int t = tid; t < 5 * SYM; t += NT) {
          const int c = t / SYM, r = t % SYM, k23 = r % 36;
          const double *f = S.pS[r / 36];
          S.Mw[c][r] = f[0] * S.u.st.B[c][0][k23] + f[1] * S.u.st.B[c][1][k23] +
                       f[2] * S.u.st.B[c][2][k23];
        }
        __syncthreads();
        // node pairs: combine and scatter
        const int src = M.ssm[w] == GB_SPECIES_SOURCE_ARRHENIUS ? (int)M.ssp[w][3] : -1;
        const uint16_t *nsl = A.elem_nslot + (int64_t)e * Q * Q;
        for (int t = tid; t < Q * Q; t += NT) {
          const int ki = t / Q, kj = t - ki * Q, ni = S.nodes[ki];
          const int gr = A.fu[ni] + OY + w;
          if (A.dbc[gr]) continue;
          const int Li = S.lex[ki], Lj = S.lex[kj];
          const int a1 = Li % 3, a2 = (Li / 3) % 3, a3 = Li / 9;
          const int b1 = Lj % 3, b2 = (Lj / 3) % 3, b3 = Lj / 9;
          const int f1 = a1 * 3 + b1, f2 = a2 * 3 + b2, f3 = a3 * 3 + b3;
          const int g1 = b1 * 3 + a1, g2 = b2 * 3 + a2, g3 = b3 * 3 + a3;
          const int s1 = S.sym[f1], s2 = S.sym[f2], s3 = S.sym[f3];
          const int m = (s1 * 6 + s2) * 6 + s3;
          const double adv = S.S1[0][(f1 * 6 + s2) * 6 + s3] + S.S1[1][(s1 * 9 + f2) * 6 + s3] +
                             S.S1[2][(s1 * 6 + s2) * 9 + f3];
          const double K = S.KS[m] +
                           (S.KM[0][(f1 * 9 + f2) * 6 + s3] + S.KM[0][(g1 * 9 + g2) * 6 + s3]) +
                           (S.KM[1][(f1 * 6 + s2) * 9 + f3] + S.KM[1][(g1 * 6 + s2) * 9 + g3]) +
                           (S.KM[2][(s1 * 9 + f2) * 9 + f3] + S.KM[2][(s1 * 9 + g2) * 9 + g3]);
          double d = fma(-M.diff[w], K, adv);
          // the mass term's sensitivity -(1 + 2 theta) / dt phi_i phi_j dA
          if (tr) d = fma(-A.mass_c, S.Mm[m], d);
          double *row = A.vals + A.rowptr[gr] + A.nbr_off[A.nbr_ptr[ni] + nsl[ki * Q + kj]];
#pragma unroll
          for (int b = 0; b < 3; b++) atomicAdd(row + b, S.Mw[b][m]);
          if (ENERGY) atomicAdd(row + 3, S.Mw[3][m]);
          atomicAdd(row + OY + w, src == w ? d + S.Mw[4][m] : d);
          if (src >= 0 && src != w) atomicAdd(row + OY + src, S.Mw[4][m]);
        }
      }
    }
  }
}

template <bool ENERGY, bool JAC>
static cudaError_t launch_species_sf(const AsmArgs &a, const SfTables *tb, const int *elems,
                                     int nelem, int sms, cudaStream_t st) {
  const size_t sm = sizeof(sp::Smem3);
  auto k = assemble_species_sf_kernel<ENERGY, JAC>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  const int grid = nelem < 2 * sms ? nelem : 2 * sms;
  if (grid <= 0) return cudaSuccess;
  launch_dependent(k, grid, 256, sm, st, a, tb, elems, nelem);
  return cudaGetLastError();
}

cudaError_t launch_assemble_species_sf(const AsmArgs &a, bool energy, bool jac,
                                       const SfTables *tb, const int *elems, int nelem, int sms,
                                       cudaStream_t st) {
  if (energy)
    return jac ? launch_species_sf<true, true>(a, tb, elems, nelem, sms, st)
               : launch_species_sf<true, false>(a, tb, elems, nelem, sms, st);
  return jac ? launch_species_sf<false, true>(a, tb, elems, nelem, sms, st)
             : launch_species_sf<false, false>(a, tb, elems, nelem, sms, st);
}

template <int DIM, bool ENERGY, bool JAC>
static cudaError_t launch_species_t(const AsmArgs &a, const int *elems, int nelem,
                                    cudaStream_t st) {
  using C = Q2<DIM>;
  const size_t sm = sizeof(sp::Elem<DIM>) * C::EPB;
  auto k = assemble_species_kernel<DIM, ENERGY, JAC>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  const int grid = (nelem + C::EPB - 1) / C::EPB;
  if (grid == 0) return cudaSuccess;
  k<<<grid, 256, sm, st>>>(a, elems, nelem);
  return cudaGetLastError();
}

cudaError_t launch_assemble_species(const AsmArgs &a, int dim, bool energy, bool jac,
                                    const int *elems, int nelem, cudaStream_t st) {
#define GB_DISPATCH(D, EN, JA) \
  if (dim == D && energy == EN && jac == JA) return launch_species_t<D, EN, JA>(a, elems, nelem, st);
  GB_DISPATCH(2, false, true)
  GB_DISPATCH(2, true, true)
  GB_DISPATCH(3, false, true)
  GB_DISPATCH(3, true, true)
  GB_DISPATCH(2, false, false)
  GB_DISPATCH(2, true, false)
  GB_DISPATCH(3, false, false)
  GB_DISPATCH(3, true, false)
#undef GB_DISPATCH
  return cudaErrorInvalidValue;
}

}  // namespace gb
