// Jacobi sweeps on the momentum rows: the solver of u* where the diffusion
// numbers are small.
//
// A fluid row is (1 + sum k) x_P - sum k_nb x_nb with sum k the sum of its
// six Crank-Nicolson numbers, so a Jacobi sweep contracts the error by
// rho = max sum k / (1 + sum k): 0.01-0.1 on the grids and time steps of the
// workloads, where a sweep gains one or two digits.  A ghost row is solved
// from the sweep's new fluid values (its ghost partners' old ones), which
// contracts by (1 - w_self) / (1 + w_self) at worst, and not at all where a
// ghost's whole stencil is other ghosts; an outer row exactly (an extrapolated
// outlet cancels the row's second difference along its axis, so rho still
// bounds it).  No row's map exceeds 1 in the maximum norm: sweeps that do not
// converge stall, they do not grow.  A sweep reads c and x and writes x (12 bytes per cell and
// component in FP32) and reduces the residual of the x it reads, so the
// stopping test costs no pass of its own; a BiCGSTAB iteration moves 84
// bytes and gains about what two sweeps do.
//
// With rho above MS_RHO, or where the sweeps reach their limit, BiCGSTAB
// takes (over) the solve, with the caller's iteration cap for itself; the
// stopping test is the same one, on the true residual.  A BiCGSTAB iteration that passes it lands a digit or two below;
// the sweeps stop at the first pass, so their own test is MS_MARGIN of it
// (down to FP64's rounding), about one sweep more, and the solution is no
// further from the exact one (64^3 cavity, 200 steps from u^n at 1e-6:
// 3.8e-6 without the margin, the 1e-6 of the tests with it).
#pragma once

#include "krylov.h"

namespace ibm {

constexpr double MS_RHO = 0.5;   // largest contraction bound the sweeps are chosen for
constexpr double MS_MARGIN = 0.02;
constexpr int MS_LIMIT = 60;     // sweeps before BiCGSTAB takes over

// State of a solve.  MS_RUN = KS_RUN.  MS_A: done, x complete in the first
// buffer; MS_B: done with the sweep in progress, which writes the first
// buffer; MS_FALL: not converged within the limit.
enum { MS_RUN = 0, MS_A = 1, MS_B = 2, MS_FALL = 3, MS_FALL_B = 4 };

struct MScal {
    int state, sweeps;
    double bn2[3], rn2[3];
    int iters[3];   // sweeps after which the component met the test (-1: not yet)
};

struct MomSweep {
    bool use = false;
    double rho = 0.0;
    int ng = 0, nout1 = 0;
    bool split = false;        // outer rows read ghost cells: ghosts and outer rows in two launches
    bool full = false;         // ghost stencils read outer cells other than the faces' first layer
    const int *gcell = nullptr;
    int *outer1 = nullptr;
    uint8_t *gold = nullptr;   // [8 g + e]: the stencil entry is a ghost or outer cell (old value)
    MScal *scal = nullptr;
    ~MomSweep() { release(); }
    void release();
    // ks: km + kp per axis (interior); flag padded; gidx 8 per ghost.
    int setup(cudaStream_t s, const Grid &g, const double *const ks[3], const uint8_t *flag, const int *gcell_dev,
              const int *gcell, const int *gidx, int ng);
};

// A x = b for the three momentum components: b and x hold 3 n entries, w
// lends its second buffer, its reduction scratch and its scalars (filled as
// by bicgstab).  x_given: x holds the initial guess, else it starts from 0.
// ir (FP32 increment solve): ||b||^2 and ||c||^2 are already in it and the
// test is the increment solve's (krylov.h, solve_inc).
template <typename T>
int solve_sweeps(cudaStream_t st, const OpT<T> &A, MomSweep &ms, KrylovWork<T> &w, const T *b, T *x,
                 const SolveParams &prm, const IRScal *ir, SolveReport &rep);
// Recorded form; launch counts: *per_iter per sweep, *idle recorded but not
// run by a solve that the sweeps end.
template <typename T>
int record_sweeps(cudaStream_t st, const cudaStream_t *aux, const OpT<T> &A, MomSweep &ms, KrylovWork<T> &w,
                  const T *b, T *x, const SolveParams &prm, const IRScal *ir, int *per_iter, int *idle);

}  // namespace ibm
