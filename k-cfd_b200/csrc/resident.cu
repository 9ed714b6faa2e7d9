// On-chip BiCGSTAB of small systems: kernels and launches (design in resident.cuh).
#include "resident.cuh"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>

namespace kcfd {
namespace res {

template <int NRHS, int PREC, int R>
__global__ void __launch_bounds__(kBlock, 1) k_resident(SolveArgs a, int width) {
    extern __shared__ __align__(16) char store[];
    __shared__ Shared sh;
    ClusterTeam tm;
    int id;
    cluster_ids(tm.rank, tm.size, id);
    tm.sh = &sh;
    tm.budget = a.ctl.budget;
    tm.init();
    tm.finish(solve_on_chip<NRHS, PREC, R>(tm, a, width, store));
}

// One CTA per SM, for systems beyond a cluster. scratch: the gathered vector, then the
// partials of the reductions.
template <int NRHS, int PREC, int R>
__global__ void __launch_bounds__(kBlock, 1) k_resident_grid(SolveArgs a, int width, double* scratch, int comps) {
    extern __shared__ __align__(16) char store[];
    __shared__ Shared sh;
    GridTeam tm;
    tm.rank = blockIdx.x;
    tm.size = gridDim.x;
    tm.sh = &sh;
    tm.budget = a.ctl.budget;
    tm.count = a.ctl.bar;
    tm.err = a.ctl.err;
    tm.part = scratch + (size_t)(a.n + 1) * NRHS;
    tm.init();
    solve_on_chip<NRHS, PREC, R>(tm, a, width, store, scratch, NRHS == 1 ? comps : 1);
}

// Systems B.order[first + cluster index]: independent solves, one cluster each, scheduled by
// the hardware as SMs become free.
template <int PREC, int R>
__global__ void __launch_bounds__(kBlock, 1) k_resident_batch(BatchArgs B, int first, int width, long long budget) {
    extern __shared__ __align__(16) char store[];
    __shared__ Shared sh;
    ClusterTeam tm;
    int id;
    cluster_ids(tm.rank, tm.size, id);
    tm.sh = &sh;
    tm.budget = budget;
    tm.init();
    SolveArgs a = batch_args<double>(B, B.order[first + id]);
    a.dinv = nullptr;
    tm.finish(solve_on_chip<1, PREC, R>(tm, a, width, store));
}

// Rounds of a solve's steps on the teams above: a value into the gathered vector, a barrier, a
// gather from the next CTA, a reduction. CTA `late` comes `delay` cycles late to the second
// round's reduction. status[rank]: KCFD_OK when every sum was right, KCFD_BREAKDOWN when one
// was not, KCFD_TIMEOUT when the team gave up.
template <class Team>
__device__ bool selftest_rounds(Team& tm, double* vec, int late, long long delay, int* status) {
    bool right = true;
    auto rounds = [&]() {
        for (int round = 0; round < 4; ++round) {
            double* mine = vec + (Team::kGrid ? tm.rank : 0);
            if (threadIdx.x == 0) *mine = tm.rank + round;
            tm.sync();
            const int next = (tm.rank + 1) % tm.size;
            double v[1], tot[1];
            v[0] = threadIdx.x > 0 ? 0.0 : Team::kGrid ? __ldcg(vec + next) : ld_cluster(remote(smem_addr(vec), next));
            if (round == 1 && tm.rank == late)
                for (const long long t0 = clock64(); clock64() - t0 < delay;) __nanosleep(1000);
            tm.template reduce<1, 1>(v, tot);
            if (threadIdx.x == 0) right = right && tot[0] == tm.size * (0.5 * (tm.size - 1) + round);
            __syncthreads();
            if (tm.sh->fail) return false;
        }
        return true;
    };
    const bool ok = tm.settle(rounds());
    if (threadIdx.x == 0) status[tm.rank] = !ok ? 5 /*KCFD_TIMEOUT*/ : right ? KCFD_OK : KCFD_BREAKDOWN;
    return ok;
}

__global__ void __launch_bounds__(kBlock, 1) k_selftest_cluster(int* status, int late, long long delay, long long budget) {
    __shared__ Shared sh;
    __shared__ double vec;
    ClusterTeam tm;
    int id;
    cluster_ids(tm.rank, tm.size, id);
    tm.sh = &sh;
    tm.budget = budget;
    tm.init();
    tm.finish(selftest_rounds(tm, &vec, late, delay, status));
}

// scratch: a value per CTA, then the partials; ctl: the counter and the error flag.
__global__ void __launch_bounds__(kBlock, 1)
    k_selftest_grid(int* status, int late, long long delay, long long budget, double* scratch, int* ctl) {
    __shared__ Shared sh;
    GridTeam tm;
    tm.rank = blockIdx.x;
    tm.size = gridDim.x;
    tm.sh = &sh;
    tm.budget = budget;
    tm.count = (unsigned*)ctl;
    tm.err = ctl + 1;
    tm.part = scratch + tm.size;
    tm.init();
    tm.finish(selftest_rounds(tm, scratch, late, delay, status));
}

namespace {

// f(NRHS, PREC, R) as template arguments; false for a combination that is not compiled (more
// vectors than registers).
template <class F>
bool dispatch(int nrhs, int precond, int r, F f) {
#define KC_RES(N, P, RR)                                                                                   \
    if (nrhs == N && precond == P && r == RR) {                                                            \
        f(std::integral_constant<int, N>(), std::integral_constant<int, P>(), std::integral_constant<int, RR>()); \
        return true;                                                                                       \
    }
#define KC_RES_P(N, RR) KC_RES(N, 0, RR) KC_RES(N, 1, RR) KC_RES(N, 2, RR)
    KC_RES_P(1, 1) KC_RES_P(1, 2) KC_RES_P(1, 3) KC_RES_P(1, 4) KC_RES_P(1, 6) KC_RES_P(1, 8)
    KC_RES_P(2, 1) KC_RES_P(2, 2) KC_RES_P(2, 4)
    KC_RES_P(3, 1) KC_RES_P(3, 2) KC_RES_P(3, 3)
#undef KC_RES_P
#undef KC_RES
    return false;
}

void* kernel_of(int nrhs, int precond, int r) {  // nrhs 0: the batched kernel; nrhs + 4: the grid's
    void* k = nullptr;
    if (nrhs > 4) {
        dispatch(nrhs - 4, precond, r, [&](auto n, auto p, auto rr) { k = (void*)k_resident_grid<n(), p(), rr()>; });
        return k;
    }
    if (nrhs == 0) {
        dispatch(1, precond, r, [&](auto, auto p, auto rr) {
            if constexpr (p() != KCFD_PREC_ILU0) k = (void*)k_resident_batch<p(), rr()>;
        });
        return k;
    }
    dispatch(nrhs, precond, r, [&](auto n, auto p, auto rr) { k = (void*)k_resident<n(), p(), rr()>; });
    return k;
}

cudaLaunchConfig_t config(const Plan& p, cudaStream_t st, cudaLaunchAttribute* at, int clusters = 1) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(p.ctas * clusters);
    cfg.blockDim = dim3(kBlock);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// What the device grants a kernel: dynamic shared memory, and the largest cluster that can be
// resident at that much. Asked once per device and kernel, and only for one whose rows would
// hold the system: the questions load the kernel and take up to a millisecond each.
struct Limits {
    int smem = 0, ctas = 0;
};

// CTAs of a cooperative launch: one per SM.
int grid_ctas() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    return std::max(1, std::min(sms, kMaxGrid));
}

Limits limits(int nrhs, int precond, int r) {
    constexpr int kDevices = 64;
    static std::mutex mu;
    static Limits known[kDevices][8][3][9];
    int dev = 0;
    void* f = kernel_of(nrhs, precond, r);
    if (!f || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return Limits();
    std::lock_guard<std::mutex> lock(mu);
    Limits& L = known[dev][nrhs][precond][r];
    if (L.smem > 0) return L;
    int optin = 0;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, f) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes) != cudaSuccess ||
        cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return Limits();
    }
    Plan p;
    p.smem = optin - (int)fa.sharedSizeBytes;
    if (nrhs > 4) {
        // a cooperative launch needs all its CTAs resident together: one per SM at that much
        int coop = 0, per_sm = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kBlock, p.smem) != cudaSuccess || per_sm < 1) {
            cudaGetLastError();
            return Limits();
        }
        L.ctas = grid_ctas();
        L.smem = p.smem;
        return L;
    }
    for (p.ctas = kMaxCtas; p.ctas > 1; p.ctas /= 2) {
        int m = 0;
        cudaLaunchAttribute at[1];
        cudaLaunchConfig_t cfg = config(p, nullptr, at);
        if (cudaOccupancyMaxActiveClusters(&m, f, &cfg) == cudaSuccess && m >= 1) break;
        cudaGetLastError();
    }
    L.ctas = p.ctas;
    L.smem = p.smem;
    return L;
}

}  // namespace

Plan plan(int width, int nrhs, int precond, const std::vector<int>& lev, int max_ctas) {
    const int nlev = (int)lev.size() - 1;
    if (width < 1 || width > 64 || nlev > 4096) return Plan();
    auto rows_on = [&](int ctas) {
        int64_t rows = 0;
        for (int l = 0; l < nlev; ++l) rows += (lev[l + 1] - lev[l] + ctas - 1) / ctas;
        return rows;
    };
    // the fewest rows per thread first: a thread's rows are done one after another
    for (int r = 1; r <= 8; ++r) {
        int c = 1;
        while (c <= max_ctas && rows_on(c) > kBlock * r) ++c;
        if (c > max_ctas) continue;
        const Limits L = limits(nrhs, precond, r);
        size_t bytes = SIZE_MAX;
        dispatch(nrhs, precond, r, [&](auto n, auto p, auto rr) { bytes = Store<n(), p(), rr(), false>::bytes(width, nlev); });
        if (L.smem == 0 || bytes > (size_t)L.smem || c > L.ctas) continue;
        Plan p;
        p.ctas = c;
        p.rows_per_thread = r;
        p.width = width;
        p.smem = (int)bytes;
        return p;
    }
    // beyond a cluster: one CTA per SM. Right-hand sides that do not fit together are solved
    // one after another; with ILU(0) that is slower than the graph engine's joint solve
    // (216,000 hexes, three right-hand sides, us per iteration: Jacobi 3 x 13.8 against 76,
    // ILU(0) 3 x 34 against 88).
    const int sms = grid_ctas();
    for (int comps : {1, nrhs}) {
        if (max_ctas == 1 || (comps > 1 && precond == KCFD_PREC_ILU0)) break;
        const int joint = nrhs / comps;
        for (int r = 1; r <= 8; ++r) {
            if (rows_on(sms) > kBlock * r) continue;
            const Limits L = limits(joint + 4, precond, r);
            size_t bytes = SIZE_MAX;
            dispatch(joint, precond, r, [&](auto n, auto p, auto rr) { bytes = Store<n(), p(), rr(), true>::bytes(width, nlev); });
            if (L.smem == 0 || bytes > (size_t)L.smem) continue;
            Plan p;
            p.ctas = L.ctas;
            p.grid = true;
            p.comps = comps;
            p.rows_per_thread = r;
            p.width = width;
            p.smem = (int)bytes;
            p.scratch = (size_t)(lev[nlev] + 1) * joint + (size_t)2 * kMaxQ * L.ctas;
            return p;
        }
    }
    return Plan();
}

Plan plan_compact(int n, int width, int precond) {
    if (width < 1 || width > 64 || precond < 0 || precond > 1) return Plan();
    // two CTAs or more hold over 1,024 rows each; odd large counts are rounded up, which
    // leaves fewer shapes (launches) in a batch
    for (int c = 1; c <= kMaxCtas; c += c < 6 ? 1 : c < 12 ? 2 : 4)
        for (int r = c < 3 ? 1 : 8; r <= 8; ++r) {
            if ((int64_t)c * kBlock * r < n) continue;
            const Limits L = limits(0, precond, r);
            const size_t bytes = (size_t)kBlock * r * (8 + 12 * (size_t)width) + 16;
            if (L.ctas < c || bytes > (size_t)L.smem) continue;
            Plan p;
            p.ctas = c;
            p.rows_per_thread = r;
            p.width = width;
            p.smem = (int)bytes;
            return p;
        }
    return Plan();
}

cudaError_t batch(const Plan& p, const BatchArgs& B, int first, int count, cudaStream_t st) {
    BatchArgs args = B;
    int width = p.width;
    long long budget = 4000000000LL;  // ~2 s at 2 GHz per wait
    void* ptrs[] = {&args, &first, &width, &budget};
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config(p, st, at, count);
    return cudaLaunchKernelExC(&cfg, kernel_of(0, B.precond, p.rows_per_thread), ptrs);
}

cudaError_t solve(const Plan& p, int nrhs, int precond, const SolveArgs& a, double* scratch, cudaStream_t st) {
    SolveArgs args = a;
    int width = p.width;
    if (p.grid) {
        int comps = p.comps;
        void* ptrs[] = {&args, &width, &scratch, &comps};
        cudaError_t e = cudaMemsetAsync(a.ctl.bar, 0, sizeof(unsigned), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(a.ctl.err, 0, sizeof(int), st);
        if (e != cudaSuccess) return e;
        return cudaLaunchCooperativeKernel(kernel_of(nrhs / p.comps + 4, precond, p.rows_per_thread), dim3(p.ctas), dim3(kBlock), ptrs,
                                           p.smem, st);
    }
    void* ptrs[] = {&args, &width};
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config(p, st, at);
    return cudaLaunchKernelExC(&cfg, kernel_of(nrhs, precond, p.rows_per_thread), ptrs);
}

}  // namespace res
}  // namespace kcfd

extern "C" int kcfd_selftest_on_chip(int32_t grid, int32_t ctas, int64_t budget_cycles, int32_t late, int64_t late_cycles,
                                     double* scratch, int32_t* status, void* stream) {
    using namespace kcfd;
    KCFD_REQUIRE(scratch && status, "kcfd_selftest_on_chip: NULL argument");
    KCFD_REQUIRE(ctas >= 1 && ctas <= (grid ? 64 : 8) && late < ctas,
                 "kcfd_selftest_on_chip: 1 to 8 CTAs (grid: 64), late below that");
    KCFD_REQUIRE(budget_cycles > 0 && budget_cycles <= 4000000000LL && late_cycles >= 0 && late_cycles <= 100000000LL,
                 "kcfd_selftest_on_chip: budget or delay out of range");
    cudaStream_t st = (cudaStream_t)stream;
    long long budget = budget_cycles, delay = late_cycles;
    KCFD_CUDA(cudaMemsetAsync(status, 0, (ctas + 2) * sizeof(int32_t), st));
    if (grid) {
        int* ctl = status + ctas;
        void* ptrs[] = {&status, &late, &delay, &budget, &scratch, &ctl};
        KCFD_CUDA(cudaLaunchCooperativeKernel((void*)res::k_selftest_grid, dim3(ctas), dim3(res::kBlock), ptrs, 0, st));
        return KCFD_OK;
    }
    res::Plan p;
    p.ctas = ctas;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = res::config(p, st, at);
    void* ptrs[] = {&status, &late, &delay, &budget};
    KCFD_CUDA(cudaLaunchKernelExC(&cfg, (void*)res::k_selftest_cluster, ptrs));
    return KCFD_OK;
}
