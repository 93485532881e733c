// ILU(0) factorisation by nodes (gb_factor.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace gb {

// unknowns per node: nodal fields (<= 3 + 1 + GB_MAX_SPECIES) + P1 pressures
constexpr int kMaxNodeDofs = 16;

struct IluArgs {
  const int *fu;
  const int64_t *rowptr;
  const int *nbr_ptr, *nbr_node, *nbr_off, *nbr_offT;
  const int *nbr_self;  // every node's own position in its neighbour list
  const int *nodes;     // the nodes, every one after its lower neighbours
  int num_nodes;
  int dim, nvn, energy;
  int maxnb, lmax, blkmax, maxnr;  // neighbours, row length, block-row values, unknowns
  double tau;           // pivot floor
  int *nfix;            // floored pivots
  void *rpiv;           // reciprocal pivots, [unknowns] of the factors' type
  int *done;            // [num_nodes] set when a node's rows are final, then the ticket
  int *error;           // set when a wait gave up
  long long spin_limit; // polls before a wait gives up
  bool one_cta;         // on a grid of one CTA (an injected fault)
};

// Shared memory of one CTA for elements of size tsize, and the most there is.
constexpr int kIluSmemMax = 227 * 1024;
size_t ilu_smem_bytes(size_t tsize, const IluArgs &g);
// lu = ILU(0) factors of A in its pattern; g.done cleared beforehand
template <class T>
cudaError_t ilu0_factor(const IluArgs &g, const double *A, T *lu, int sms, cudaStream_t st);

}  // namespace gb
