// grad.cuh -- analytic RHF nuclear gradient kernels (defined in grad.cu).
#pragma once
#include <cuda_runtime.h>

#include "md_kernels.cuh"

constexpr int kGradMaxComp = 6;   // Cartesian components per shell slot (d)
constexpr int kGradCopies = 64;   // copies of the gradient, so that the atomics on 3 natom addresses spread
constexpr int kGradClasses = 21;  // angular classes (work counters)

struct GradArgs {
  // shells and the shell pairs (every unordered pair of shells of the molecule once)
  int npair;
  const int *pa, *pb;
  const int *L, *nprim, *poff, *func, *shell_atom;
  const double *center, *exps, *coefs;
  // kept primitive pairs: per shell pair the first one, how many, the offset of its tables and
  // the terms of one; per primitive pair its shell pair and its index ka * Kb + kb
  int nprimpair;
  const int *prb, *prc, *pair_nnz, *pp_pair, *pp_index;
  const long long* eoff;
  double4_32a* pP;  // (1/p, P)
  double* frac;     // a / p
  double* E64;      // E' tables
  double* ER;       // d E' / d(A-B), at 3 x the offset of E', x, y and z after one another
  const float* Qpair;  // Schwarz bound per shell pair (null: no screening)
  double qtol;         // quartets with Q_ab Q_cd below qtol are skipped
  double small[10];    // 0.0 .. 9.0
  // nuclei
  int natom;
  const double *xyz, *Z;
  // densities (N x N, device), the output dE/dR (kGradCopies x natom x 3, device; the sum
  // ends up in the first copy) and the work counters of the classes
  const double *P, *W;
  int N;
  double* grad;
  unsigned long long* work;
};

// pairs of one pair class that have a primitive pair left, by primitive count (groups of
// slots start[g] .. start[g + 1), at most prims[g] each), inside a group by Q descending
struct GradList {
  const int* list;
  int n, ngroup;
  int start[mmdg::kMaxGroups + 1], prims[mmdg::kMaxGroups];
};

cudaError_t mmdg_launch_rhf_gradient(const GradArgs& a, const mmdg::Geometry& g, const GradList* lists, int nstreams,
                                     const cudaStream_t* side, cudaEvent_t fork, const cudaEvent_t* join,
                                     cudaStream_t st);
