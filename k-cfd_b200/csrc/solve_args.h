// Arguments of one BiCGSTAB solve and of a batch of them, shared by the persistent kernels
// (solver.cu) and the on-chip kernels (resident.cu).
#pragma once
#include <cstring>

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

struct BatchSys {
    int n, nnz;
    long long row_off;  // rows before this system in the packed vectors
    long long ptr_off;  // offset of its (n + 1) row pointers
    long long nnz_off;  // offset of its entries
};

struct BatchArgs {
    int nsys, lanes, mixed, precond, stop, maxiter, max_refine, inner_maxiter, max_restarts;
    int nq;  // systems in this launch's queue (order[0..nq))
    double rtol, atol, inner_rtol;
    const BatchSys* sys;
    const int* order;
    int* queue;
    const int* indptr;
    const int* indices;
    const double* vals64;
    float* vals32;
    void* dinv;
    int* lev;
    void* work;
    double* r64;
    double* x;
    const double* b;
    int* iters;
    double* relres;
    int* status;
};

// SolveArgs of system sid of a batch (everything but the team control).
template <typename V>
__device__ SolveArgs batch_args(const BatchArgs& B, int sid) {
    const BatchSys S = B.sys[sid];
    SolveArgs a;
    memset(&a, 0, sizeof(a));
    a.n = S.n;
    a.lanes = B.lanes;
    a.indptr = B.indptr + S.ptr_off;
    a.indices = B.indices + S.nnz_off;
    a.vals64 = B.vals64 + S.nnz_off;
    a.vals32 = B.vals32 ? B.vals32 + S.nnz_off : nullptr;
    a.dinv = (V*)B.dinv + S.row_off;
    a.lev_ptr = B.lev + 2 * sid;
    a.nlev = 1;
    a.work = (V*)B.work + 9 * S.row_off;
    a.x = B.x + S.row_off;
    a.b = B.b + S.row_off;
    a.r64 = B.r64 ? B.r64 + S.row_off : nullptr;
    a.stop = B.stop;
    a.maxiter = B.maxiter;
    a.max_refine = B.max_refine;
    a.inner_maxiter = B.inner_maxiter;
    a.max_restarts = B.max_restarts;
    a.rtol = B.rtol;
    a.atol = B.atol;
    a.inner_rtol = B.inner_rtol;
    a.iters_out = B.iters + sid;
    a.relres_out = B.relres + sid;
    a.status_out = B.status + sid;
    return a;
}

}  // namespace kcfd
