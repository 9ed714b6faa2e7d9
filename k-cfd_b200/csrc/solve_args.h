// Arguments of one BiCGSTAB solve, shared by the persistent kernels (solver.cu) and the
// on-chip kernel (resident.cu).
#pragma once
#include "team.cuh"

namespace kcfd {

constexpr double kEps2 = 4.930380657631324e-32;  // float64 eps^2 (scipy rhotol/omegatol)

struct SolveArgs {
    int n;
    int lanes;
    // matrix of the Krylov iterations (the level-permuted copy when perm != null)
    const int* indptr;
    const int* indices;
    const double* vals64;
    const float* vals32;
    const int* perm;     // [n] permuted row -> caller row, or null
    double* px;          // [n*nrhs] permuted FP64 solution (perm only)
    double* pb;          // [n*nrhs] permuted FP64 rhs (perm only)
    // preconditioner
    void* dinv;          // Jacobi inverse diagonal, V
    const int* diag;     // [n] position of the diagonal (ILU)
    void* lu;            // [nnz] ILU factors, V
    void* ludinv;        // [n] 1 / u_ii, V
    const int* lev_ptr;  // [nlev+1] level row ranges
    int nlev;
    // vectors
    void* work;          // 9 V vectors of n*nrhs
    double* x;           // caller FP64 solution (x0 on entry)
    const double* b;     // caller FP64 rhs
    double* r64;         // MIXED outer residual
    // control
    int stop;
    int maxiter;
    int max_refine;
    int inner_maxiter;
    int max_restarts;    // KCFD_STOP_SCIPY: restarts on rho / omega breakdown (0: scipy's stop)
    double rtol, atol, inner_rtol;
    int* iters_out;
    double* relres_out;
    int* status_out;
    TeamCtl ctl;
};

// Verification passes of a batched FP64 solve (see solve_fp64).
constexpr int kVerifyPasses = 3;

}  // namespace kcfd
