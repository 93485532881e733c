// ILU(0) of the scaled matrix, one node's block row per CTA, all nodes in one
// launch.
//
// The pattern is dense in node blocks (every unknown of a node couples with
// every unknown of every neighbour node; the energy row alone skips pressure
// columns), so the reference's scalar ILU(0) in node-major order is, block
// by block: for each lower neighbour node m (ascending)
//     L_nm   = A_nm U_mm^-1                 (triangular, <= 16 x 16)
//     A_nq  -= L_nm U_mq   for every q > m neighbouring both n and m
// then the dense elimination of the node's own diagonal block and the rest
// of its row.  Fill outside the pattern (energy row x pressure column) is
// dropped, as in ILU(0).  The node's block row lives in shared memory; the
// factored rows of lower nodes are read from global memory.  A pivot smaller
// than tau in magnitude (the row-scaled matrix has unit row sums) becomes
// +-tau: in the reference's node-major order an element without a pressure
// datum whose earlier velocity unknowns are all Dirichlet rows leaves an
// exactly singular pressure pivot.
//
// What bounds it: the chain of steps, not the arithmetic (the 16^3 cube needs
// 1.6 G FMA, 3 ms at the FP64 rate).  A node walks its up to 62 lower
// neighbours one after another, ~2.5 us each, and with a launch per dependency
// level every level paid the longest walk in full: 417 levels of 194 us.  But
// only a few of a node's lower neighbours belong to the levels just before it;
// the others are final long before.  So the nodes are drawn one by one from a
// list in level order, a CTA starts on its node at once and waits only where
// a neighbour is not final yet: per element of a 3-D box the chain is then
// 62 steps and 26 hand-overs instead of 26 whole walks.
//
// Per lower neighbour m (sm-th in the list):
//   - wait until m is final (warp 0 polls the flags of up to 32 neighbours
//     ahead, so most waits cost nothing);
//   - U_mm into shared memory, the columns of U_mq that step 2 needs into
//     registers (their list -- m's neighbours that are also n's -- was made
//     during the step before, from the node graph alone);
//   - step 1: L_nm, a warp per row, U_mm's columns in the lanes' registers;
//   - step 2: A_nq -= L_nm U_mq, a thread per column, several rows at once;
//     the next neighbour's U_mm is on its way meanwhile.
// Every pivot's reciprocal is kept with the factors, so that no step divides.
// (Rows one by one, U_mm between the steps and a division a step: 12.4 ms for
// the 16^3 cube instead of 11.2, 3.6 instead of 3.2 for 11^3 in FP32.)
// Each entry of the block row is updated at most once per m and in ascending
// m: the factors do not depend on timing.
//
// Progress: a node's lower neighbours come before it in the list, so the first
// unfinished node of the list is always held by a running CTA and has all it
// needs, however much of the grid is resident.  Waits are bounded: past
// spin_limit polls a CTA sets the error word and goes on.
#include <algorithm>

#include "gb_factor.h"

namespace gb {

static constexpr unsigned kAll = 0xffffffffu;

size_t ilu_smem_bytes(size_t tsize, const IluArgs &g) {
  const size_t mr = g.maxnr > 8 ? 16 : 8;
  return tsize * ((size_t)g.blkmax + 3 * mr * mr + 2 * mr) + sizeof(int64_t) * g.maxnb +
         sizeof(uint2) * 2 * g.lmax + sizeof(int) * (10 * (size_t)g.maxnb + 8) +
         sizeof(uint16_t) * ((size_t)g.lmax + 8);
}

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// NT threads a CTA, MR >= the most unknowns of a node
template <class T, int NT, int MR>
__global__ void __launch_bounds__(NT)
    ilu0_kernel(IluArgs g, const double *__restrict__ A, T *lu) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T *blk = reinterpret_cast<T *>(sm_raw);  // [nr][L] the node's block row
  T *lnm = blk + g.blkmax;                 // [MR][MR] L_nm
  T *umm2 = lnm + MR * MR;                 // [2][MR][MR] U_mm
  T *rdm2 = umm2 + 2 * MR * MR;            // [2][MR] its reciprocal pivots
  // per lower neighbour: start of its rows, length of its rows (energy row)
  int64_t *sr0 = reinterpret_cast<int64_t *>(rdm2 + 2 * MR);
  uint2 *list2 = reinterpret_cast<uint2 *>(sr0 + g.maxnb);  // [2][lmax] shared columns
  int *snb = reinterpret_cast<int *>(list2 + 2 * g.lmax);   // neighbours of n
  int *soff = snb + g.maxnb;               // their column offsets
  int *sndof = soff + g.maxnb;             // their unknown counts
  int *smb = sndof + g.maxnb, *smnb = smb + g.maxnb;      // m's neighbour list
  int *smoff = smnb + g.maxnb, *smoffT = smoff + g.maxnb; // m's own block in m's rows
  int *smL = smoffT + g.maxnb, *smLT = smL + g.maxnb;
  int *sfu = smLT + g.maxnb;               // m's first unknown
  int *s_np = sfu + g.maxnb;               // [2] entries of the lists
  int *s_misc = s_np + 2;                  // ticket, early
  uint16_t *cslot = reinterpret_cast<uint16_t *>(s_misc + 6);  // column -> neighbour slot
  T *rpiv = static_cast<T *>(g.rpiv);
  const int tid = threadIdx.x, lane = tid & 31;
  const int Tr = g.energy ? g.dim : -1;    // local index of the energy row

  for (;;) {
    if (tid == 0) s_misc[0] = atomicAdd(g.done + g.num_nodes, 1);
    __syncthreads();
    const int ticket = s_misc[0];
    if (ticket >= g.num_nodes) return;
    const int n = g.nodes[ticket];
    const int base = g.nbr_ptr[n], nb = g.nbr_ptr[n + 1] - base;
    const int f0 = g.fu[n], nr = g.fu[n + 1] - f0;
    const int self = g.nbr_self[n];
    const int64_t rp0 = g.rowptr[f0];
    if (tid < 2) s_np[tid] = 0;
    for (int s = tid; s < nb; s += NT) {
      const int q = g.nbr_node[base + s];
      const int fq = g.fu[q], nq = g.fu[q + 1] - fq;
      snb[s] = q;
      soff[s] = g.nbr_off[base + s];
      sndof[s] = nq;
      if (s < self) {
        const int mb = g.nbr_ptr[q], ms = mb + g.nbr_self[q];
        smb[s] = mb;
        smnb[s] = g.nbr_ptr[q + 1] - mb;
        smoff[s] = g.nbr_off[ms];
        smoffT[s] = g.nbr_offT[ms];
        sfu[s] = fq;
        const int64_t r0 = g.rowptr[fq];
        sr0[s] = r0;
        smL[s] = (int)(g.rowptr[fq + 1] - r0);
        smLT[s] = Tr >= 0 ? (int)(g.rowptr[fq + Tr + 1] - g.rowptr[fq + Tr]) : 0;
      }
    }
    __syncthreads();
    const int L = soff[nb - 1] + sndof[nb - 1];
    // start of row r among the node's rows: L entries each, the energy row LT
    const int LT = Tr >= 0 ? (int)(g.rowptr[f0 + Tr + 1] - g.rowptr[f0 + Tr]) : 0;
    auto row_of = [&](int64_t r0, int len, int lenT, int r) -> int64_t {
      return r0 + (int64_t)r * len - (Tr >= 0 && r > Tr ? len - lenT : 0);
    };
    // load the block row (full layout; energy-row pressure columns held at 0)
    for (int r = 0; r < nr; r++) {
      if (r == Tr) continue;
      const double *Ar = A + row_of(rp0, L, LT, r);
      for (int c = tid; c < L; c += NT) blk[r * L + c] = (T)__ldcs(Ar + c);
    }
    for (int s = tid; s < nb; s += NT)
      for (int d = 0; d < sndof[s]; d++) {
        const int c = soff[s] + d;
        cslot[c] = (uint16_t)s;
        if (Tr >= 0)
          blk[Tr * L + c] =
              d < g.nvn ? (T)A[row_of(rp0, L, LT, Tr) + g.nbr_offT[base + s] + d] : (T)0;
      }
    // the columns of U_mq for the neighbours q > m of m that are also n's
    auto make_list = [&](int sm, int h) {
      const int m = snb[sm], mb = smb[sm], mnb = smnb[sm];
      uint2 *list = list2 + h * g.lmax;
      for (int t = tid; t < mnb; t += NT) {
        const int q = g.nbr_node[mb + t];
        if (q <= m) continue;
        int lo = 0, hi = nb - 1;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (snb[mid] < q) lo = mid + 1; else hi = mid;
        }
        if (snb[lo] != q) continue;
        const int nq = sndof[lo], off = g.nbr_off[mb + t], offT = g.nbr_offT[mb + t];
        const int p = atomicAdd(s_np + h, nq);
        for (int d = 0; d < nq; d++)
          list[p + d] = make_uint2((unsigned)(off + d) | (unsigned)(offT + d) << 16,
                                   (unsigned)(soff[lo] + d) | (d >= g.nvn ? 0x80000000u : 0u));
      }
    };
    // U_mm and its reciprocal pivots: from memory by the last warps (the first
    // one waits for neighbours), then into shared memory
    constexpr int UPT = (MR * MR + MR + NT - 1) / NT;
    T uf[UPT];
    auto fetch_umm = [&](int sm) {
      const int nm = sndof[sm];
#pragma unroll
      for (int p = 0; p < UPT; p++) {
        const int w = NT - 1 - tid + p * NT, dk = w / MR, d = w % MR;
        uf[p] = (T)0;
        if (dk < nm) {
          if (d >= dk && d < nm && !(dk == Tr && d >= g.nvn))
            uf[p] = __ldcg(lu + row_of(sr0[sm], smL[sm], smLT[sm], dk) +
                           (dk == Tr ? smoffT[sm] : smoff[sm]) + d);
        } else if (dk == MR && d < nm) {
          uf[p] = __ldcg(rpiv + sfu[sm] + d);
        }
      }
    };
    auto store_umm = [&](int h) {
#pragma unroll
      for (int p = 0; p < UPT; p++) {
        const int w = NT - 1 - tid + p * NT;
        if (w < MR * MR) umm2[h * MR * MR + w] = uf[p];
        else if (w < MR * MR + MR) rdm2[h * MR + w - MR * MR] = uf[p];
      }
    };
    // warp 0: number of leading lower neighbours known to be final
    int ready = 0;
    auto wait_for = [&](int sm) {
      long long polls = 0;
      while (ready <= sm) {
        const int s = ready + lane;
        const unsigned ok = __ballot_sync(kAll, s < self && ld_acquire(g.done + snb[s]) != 0);
        ready += ok == kAll ? 32 : __ffs(~ok) - 1;
        if (ready <= sm && (++polls > g.spin_limit ||
                            ((polls & 1023) == 0 && *(volatile int *)g.error))) {
          if (lane == 0) atomicExch(g.error, 1);
          ready = self;
        }
      }
    };
    if (self > 0) {
      make_list(0, 0);
      if (tid < 32) wait_for(0);
      __syncthreads();
      fetch_umm(0);
      store_umm(0);
    }
    __syncthreads();
    for (int sm = 0; sm < self; sm++) {
      const int h = sm & 1, nm = sndof[sm], cm = soff[sm], np = s_np[h];
      const T *umm = umm2 + h * MR * MR, *rdm = rdm2 + h * MR;
      const uint2 *list = list2 + h * g.lmax;
      const int64_t r0 = sr0[sm];
      const int lenm = smL[sm], lenmT = smLT[sm];
      // a column of U_mq: nm values
      auto load_column = [&](uint2 e, T *u) {
        const T *p = lu + r0;
#pragma unroll
        for (int dk = 0; dk < MR; dk++) {
          u[dk] = (T)0;
          if (dk < nm) {
            if (dk != Tr) u[dk] = __ldcg(p + (e.x & 0xffff));
            else if (!(e.y >> 31)) u[dk] = __ldcg(p + (e.x >> 16));
          }
          p += dk == Tr ? lenmT : lenm;
        }
      };
      T u[MR];
      uint2 e = make_uint2(0, 0);
      if (tid < np) {
        e = list[tid];
        load_column(e, u);
      }
      if (tid == 0) s_misc[1] = sm + 1 < self && ready > sm + 1;
      // step 1: L_nm = A_nm U_mm^-1, a warp per row (lane d holds the row's
      // entry in m's column d): per pivot one shuffle, then every later column
      // updated at once
      if ((tid >> 5) < nr) {
        T ud[MR];  // lane's column of U_mm, zero up to its diagonal
#pragma unroll
        for (int dk = 0; dk < MR; dk++) ud[dk] = lane > dk && lane < nm ? umm[dk * MR + lane] : (T)0;
        const T rd = lane < nm ? rdm[lane] : (T)0;
        for (int r = tid >> 5; r < nr; r += NT >> 5) {
          T *br = blk + r * L + cm;
          // the energy row has no pressure columns
          const int last = r == Tr ? min(nm, g.nvn) : nm;
          T v = lane < nm ? br[lane] : (T)0, w = (T)0;
#pragma unroll
          for (int dk = 0; dk < MR; dk++) {
            if (dk >= last) break;
            const T l = __shfl_sync(kAll, v * rd, dk);
            if (lane == dk) w = l;
            if (lane < last) v -= l * ud[dk];  // zero where U_mm has no entry
          }
          if (lane < nm) {
            lnm[r * MR + lane] = w;
            br[lane] = lane < last ? w : v;
          }
        }
      }
      __syncthreads();
      // the next neighbour is final already: its U_mm now
      const bool early = s_misc[1] != 0;
      if (early) fetch_umm(sm + 1);  // on its way during step 2
      // step 2
      for (int f = tid; f < np; f += NT) {
        if (f != tid) {
          e = list[f];
          load_column(e, u);
        }
        // several rows at a time: their products are independent, one row's
        // wait for each other (2-D nodes have few rows)
        constexpr int RB = NT == 64 ? 2 : 4;
        T *col = blk + (e.y & 0x7fffffffu);
        for (int b0 = 0; b0 < nr; b0 += RB) {
          T v[RB];
#pragma unroll
          for (int i = 0; i < RB; i++) v[i] = b0 + i < nr ? col[(b0 + i) * L] : (T)0;
#pragma unroll
          for (int dk = 0; dk < MR; dk++) {
            if (dk >= nm) break;
#pragma unroll
            for (int i = 0; i < RB; i++) v[i] -= lnm[(b0 + i) * MR + dk] * u[dk];
          }
#pragma unroll
          for (int i = 0; i < RB; i++)
            if (b0 + i < nr && !(b0 + i == Tr && (e.y >> 31))) col[(b0 + i) * L] = v[i];
        }
      }
      if (early) store_umm(h ^ 1);
      if (sm + 1 < self) {
        make_list(sm + 1, h ^ 1);
        if (tid < 32) wait_for(sm + 1);
      }
      __syncthreads();
      if (tid == 0) s_np[h] = 0;
      if (sm + 1 < self && !early) {
        fetch_umm(sm + 1);
        store_umm(h ^ 1);
        __syncthreads();
      }
    }
    // own diagonal block: warp 0, lane d holds column d
    const int cs = soff[self];
    if (tid < 32) {
      for (int dk = 0; dk < nr; dk++) {
        T *rk = blk + dk * L + cs;
        T piv = rk[dk];
        if (fabs((double)piv) < g.tau) {
          piv = piv < (T)0 ? (T)-g.tau : (T)g.tau;
          if (lane == 0) atomicAdd(g.nfix, 1);
        }
        __syncwarp();
        if (lane == 0) rk[dk] = piv;
        // lane r divides row r's entry, then lane d updates column d
        if (lane > dk && lane < nr && !(lane == Tr && dk >= g.nvn))
          blk[lane * L + cs + dk] = blk[lane * L + cs + dk] / piv;
        __syncwarp();
        if (lane > dk && lane < nr) {
          const T ud = rk[lane];
          for (int r = dk + 1; r < nr; r++) {
            if (r == Tr && (dk >= g.nvn || lane >= g.nvn)) continue;
            blk[r * L + cs + lane] -= blk[r * L + cs + dk] * ud;
          }
        }
        __syncwarp();
      }
    }
    __syncthreads();
    if (tid < nr) rpiv[f0 + tid] = (T)1 / blk[tid * L + cs + tid];
    // the rest of the row: a thread per column, rows in order; then everything
    // goes back
    for (int c = tid; c < L; c += NT) {
      const int s = cslot[c], d = c - soff[s];
      if (s > self) {
        T x[MR];
#pragma unroll
        for (int r = 0; r < MR; r++) {
          if (r >= nr) break;
          T v = blk[r * L + c];
          if (!(r == Tr && d >= g.nvn)) {
#pragma unroll
            for (int k = 0; k < MR; k++) {
              if (k >= r) break;
              if (r == Tr && k >= g.nvn) continue;
              v -= blk[r * L + cs + k] * x[k];
            }
          }
          x[r] = v;
          blk[r * L + c] = v;
        }
      }
      for (int r = 0; r < nr; r++) {
        if (r != Tr) lu[row_of(rp0, L, LT, r) + c] = blk[r * L + c];
        else if (d < g.nvn) lu[row_of(rp0, L, LT, r) + g.nbr_offT[base + s] + d] = blk[r * L + c];
      }
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      st_release(g.done + n, 1);
    }
  }
}

template <class T, int NT, int MR>
static cudaError_t launch_ilu(const IluArgs &g, const double *A, T *lu, int sms,
                              cudaStream_t st) {
  const size_t sm = ilu_smem_bytes(sizeof(T), g);
  auto k = ilu0_kernel<T, NT, MR>;
  // the limit belongs to the process: the same for every problem, so that a
  // thread with shorter rows does not lower it before this launch
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kIluSmemMax);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, NT, sm);
  if (e != cudaSuccess) return e;
  const int grid = g.one_cta ? 1 : std::min(g.num_nodes, std::max(1, per_sm) * sms);
  k<<<grid, NT, sm, st>>>(g, A, lu);
  return cudaGetLastError();
}

template <class T>
cudaError_t ilu0_factor(const IluArgs &g, const double *A, T *lu, int sms, cudaStream_t st) {
  if (g.dim == 2)
    return g.maxnr > 8 ? launch_ilu<T, 64, 16>(g, A, lu, sms, st)
                       : launch_ilu<T, 64, 8>(g, A, lu, sms, st);
  // 16^3 cube: 11.2 ms with 128 threads, 12.3 with 192, 13.7 with 256
  return g.maxnr > 8 ? launch_ilu<T, 128, 16>(g, A, lu, sms, st)
                     : launch_ilu<T, 128, 8>(g, A, lu, sms, st);
}

template cudaError_t ilu0_factor<double>(const IluArgs &, const double *, double *, int,
                                         cudaStream_t);
template cudaError_t ilu0_factor<float>(const IluArgs &, const double *, float *, int,
                                        cudaStream_t);

}  // namespace gb
