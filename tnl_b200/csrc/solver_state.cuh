// solver_state.cuh -- the solvers' device-resident scalars and the
// reference's stopping rule on them.
#pragma once

#include "internal.cuh"

namespace tnlb {

// Device-resident solver scalars.
struct DevState {
   double normb, s1, s2, alpha, beta, omega, rho, rho_old, r_ast_sqnorm, residue;
   double conv, div;
   int32_t it, done, maxit, minit;
   int32_t flag;
   uint32_t loops;  // bodies run by the current launch of a looping iteration graph
};

__device__ __forceinline__ bool check_next(const DevState& S)
{
   return !(isnan(S.residue) || S.it > S.maxit || (S.residue > S.div && S.it >= S.minit) ||
            (S.residue < S.conv && S.it >= S.minit));
}

// IterativeSolver::nextIteration (IterativeSolver.hpp:98-108).
__device__ __forceinline__ void next_iteration(DevState& S)
{
   const bool c = check_next(S);
   S.it++;
   if (!c) S.done = 1;
}

}  // namespace tnlb
