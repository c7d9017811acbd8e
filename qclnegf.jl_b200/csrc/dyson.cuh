// Arguments of the Dyson + Keldysh kernels, and the kernel of small bases.
#pragma once
#include "common.cuh"

namespace qcl {

template <typename RS> struct DysonArgs {
  int NE, Nk, N, m0;  // blocks of momenta m0 .. m0 + gridDim.y - 1
  const double* eps;
  double eta;
  const Cx<double>* h;  // (Nk, N, N), FP64 always
  const Cx<RS>* sigR;
  const Cx<RS>* sigL;
  const Cx<RS>* sigG;   // may be null
  Cx<RS>* GR;           // may be null
  Cx<RS>* GL;           // may be null
  Cx<RS>* GG;           // may be null
  double* scale;        // (NE, Nk), may be null
  Cx<double>* traceL;   // (NE, Nk) raw tr G<, may be null
  Cx<double>* traceG;   // (NE, Nk) raw tr G>, may be null
  int* status;
  int mcount;
};

// N_b <= 6 (dyson_small.cu: a translation unit of its own, loaded at its first
// launch; with the warp-per-block kernels the first small solve of a process
// took 7 ms more).
template <typename RS, typename RL, typename RM> int launch_dyson_small(const DysonArgs<RS>& a, cudaStream_t st);

}  // namespace qcl
