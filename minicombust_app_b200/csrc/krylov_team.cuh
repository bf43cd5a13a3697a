// Whole Krylov solves as one kernel, for systems small enough that the blocks
// of one launch hold them: a "team" of blocks -- a thread-block cluster, or a
// cooperative grid of one block per SM -- keeps the vectors in registers and
// the rows in shared memory, exchanges what neighbouring rows need through L2
// and takes its dot products through a team-wide sum that is also the barrier.
//
// At these sizes an iteration of the per-kernel solvers is bound by latency:
// each kernel's launch, its read of the solver state, and the tail of its
// reduction (block partials, a counter, the last block's second pass) -- 5 to
// 7 us a kernel however few the rows.  A team's sum costs 1.1 us (cluster of
// 16) or 2.5 us (148 blocks).  Measured, before and after: Jacobi PCG 14 -> 3.5
// us per iteration at 16,000 rows and 23 -> 8.5 us at 221,000; BiCGStab 20 ->
// 5.2 us at 3,000 rows and 29 -> 16 us at 262,000.
#pragma once

#include <cuda_runtime.h>

#include "krylov.cuh"

namespace mcb {

// Status of a finished team solve: the grid form's waits are bounded, and a block
// whose wait ran out has left without its rows' result whatever the others did.
template <typename State>
int team_status(const State &st, int status)
{
    return st.team[1] ? (int)KRYLOV_TIMEOUT : status;
}

// Jacobi-preconditioned CG (the method of k_pcg_init, k_pcg_iter1 and
// k_pcg_iter2, with the mean-zero projections): v.st->mean set when project
// (pcg_mean), v.x the initial guess when use_x0, else zero.  One launch leaves
// the solution (mean removed) in v.x and the state in v.st (team_status).  v.partials:
// [2][3][SMs] at least.  False (nothing launched) where no team holds N rows.
bool pcg_team(cudaStream_t s, const Ell &A, const PcgVectors &v, double rtol, double abs_floor, int max_iters,
              int use_x0);

// BiCGStab with one right-hand side (k_bicg_init, _1, _2, _3) from zero.
// rp: [N] pairs, vv: two vectors [N], partials as for pcg_team.
bool bicg_team(cudaStream_t s, const Ell &A, const double *b, double *x, double2 *rp, double *vv0, double *vv1,
               double *partials, BicgState<1> *st, double rtol, int max_iters);

} // namespace mcb
