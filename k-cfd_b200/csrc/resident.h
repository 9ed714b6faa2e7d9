// Host interface of the on-chip BiCGSTAB (resident.cu).
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace kcfd {
struct SolveArgs;
struct BatchArgs;
namespace res {

constexpr int kMaxCtas = 16;

// Launch shape of an on-chip solve: one cluster of `ctas` CTAs (grid: a cooperative launch of
// one CTA per SM), each thread with `rows_per_thread` rows of at most `width` entries, `smem`
// bytes of shared memory per CTA, `scratch` doubles of device memory.
struct Plan {
    int ctas = 0;  // 0: the system does not fit on chip
    int rows_per_thread = 0, width = 0, smem = 0;
    bool grid = false;
    int comps = 1;  // > 1: the right-hand sides one after another
    size_t scratch = 0;
};

// Shape for a matrix of at most `width` entries a row whose levels start at rows lev[l]
// (lev.back() rows), on a cluster of up to max_ctas CTAs or, for max_ctas > 1, the grid.
Plan plan(int width, int nrhs, int precond, const std::vector<int>& lev, int max_ctas);

// Shape on the fewest CTAs that hold a system of n rows (Jacobi or no preconditioner, one
// right-hand side).
Plan plan_compact(int n, int width, int precond);

// One FP64 solve; a holds the caller's pointers (x, b, outputs) and the handle's pattern,
// values and preconditioner.
cudaError_t solve(const Plan& p, int nrhs, int precond, const SolveArgs& a, double* scratch, cudaStream_t st);

// Systems B.order[first .. first + count) of a batch, each by a cluster of its own.
cudaError_t batch(const Plan& p, const BatchArgs& B, int first, int count, cudaStream_t st);

}  // namespace res
}  // namespace kcfd
