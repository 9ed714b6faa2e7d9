// BiCGSTAB with the whole system on chip: one thread-block cluster per solve.
//
// A Krylov iteration of a system of some thousand rows is a chain of about ten dependent
// steps. On the persistent grid kernel each step is a round trip to L2 and each reduction a
// software barrier there (20 us per iteration on the 64^2 cavity's p' system, whose 0.5 MB
// take 0.1 us at HBM rate). Here everything stays in a cluster of 1 to 16 CTAs of 256
// threads for the whole solve:
//  * a thread owns R rows (1 to 8) and keeps their Krylov vectors in registers; R is
//    a template argument, so the vector phases have no loops and no address arithmetic. 256
//    threads leave 255 registers for it, and fewer warps make the block reductions cheaper;
//  * the matrix and the preconditioner lie in shared memory, entry-major ([entry][local
//    row], a compile-time stride: conflict-free, immediate offsets); a column is the
//    shared::cluster address of that row's element in the one gathered vector (phat, then
//    shat: every gather of one is over before the other is written), so a gather is a
//    single ld.shared::cluster (60 cycles in the own CTA, 240-280 in another one);
//  * each level's rows are split evenly over the CTAs; a CTA keeps its slices behind one
//    another (local rows), at the same local offsets in every CTA, unused ones zero;
//  * a reduction is a warp tree, a tree over the CTA's warps, one st.async of the CTA's
//    partial into every CTA (data and arrival in one message, so that no fence waits for
//    the stores before it) and a tree over the CTAs: every CTA adds the same numbers in the
//    same order and takes the same branches. Measured on 16 CTAs of 256 threads: 950
//    cycles, 1,640 with remote stores and a cluster barrier. The convergence test on ||s||
//    shares the reduction of t.s and t.t (t = A shat is wasted in the last iteration only),
//    so an iteration has three reductions and, for the gathers, two cluster barriers (440
//    cycles) plus two per further ILU level;
//  * the scalar state of right-hand side c lives in the registers of lane c of warp 0,
//    which broadcasts what the vector phases need.
// The hardware keeps the CTAs of a cluster resident together; the waits on an mbarrier are
// bounded all the same (status KCFD_TIMEOUT). A CTA that gives one up stays until no other can
// gather from it any more (ClusterTeam::settle).
//
// Larger systems take the same iteration on one cooperative launch with a CTA per SM
// (GridTeam): matrix and vectors on chip as above, the gathered vector in global memory (it
// stays in L2), a counter there for the barriers (2,450 cycles, whatever the CTA count) and
// the CTAs' partials beside it (3,400 to 4,100 cycles a reduction). As kernels of a graph
// loop the same steps cost 3.8 us each beyond their launch, most of it in the reductions'
// last-block hand-over: 45 us per ILU(0) iteration on 48^3 hexes, where this takes 22.5
// (Jacobi 30 and 11.5, three right-hand sides 58 and 19).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "kcfd_common.h"
#include "resident.h"
#include "solve_args.h"

namespace kcfd {
namespace res {

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
constexpr int kMaxQ = 9;   // values per reduction (three per right-hand side)
constexpr int kMaxGrid = 160;  // CTAs of the grid form

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The shared::cluster address of this CTA's shared address a in CTA `rank`.
__device__ __forceinline__ uint32_t remote(uint32_t a, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

__device__ __forceinline__ double ld_cluster(uint32_t a) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

template <int N>
__device__ __forceinline__ double tree_sum(const double* p) {
    double s[N];
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = p[i];
#pragma unroll
    for (int w = N / 2; w > 0; w >>= 1)
#pragma unroll
        for (int i = 0; i < w; ++i) s[i] += s[i + w];
    return s[0];
}

// What warp 0 tells the block about right-hand side c: flag bits.
enum { kDone = 1, kSconv = 2, kRestart = 4, kZero = 8 };

// Shared memory of the reductions and the scalar broadcast.
struct Shared {
    uint64_t bar[2];                     // arrivals of the CTAs' partials, alternating
    double warp[kMaxQ * kWarps];         // partials of this CTA's warps
    double part[2][kMaxQ * kMaxCtas];    // partials of a cluster's CTAs, 0 for absent ones
    double total[kMaxQ];                 // totals over the grid
    double al[3], om[3], be[3];          // alpha, omega, beta of each right-hand side
    int flags[3];
    int fail;                            // this CTA gave up a wait
    int any_fail;                        // cluster: one of its CTAs did
    int settled[kMaxCtas];               // cluster: CTAs that gather and send no more
    int status, iters;                   // of right-hand side 0, after a pass
};

// Sums over each warp of its threads' Q values, into sh->warp; a block barrier follows.
template <int Q>
__device__ __forceinline__ void warp_sums(double (&v)[Q], Shared* sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        double y[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) y[q] = __shfl_xor_sync(0xffffffffu, v[q], o);
#pragma unroll
        for (int q = 0; q < Q; ++q) v[q] += y[q];
    }
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < Q; ++q) sh->warp[q * kWarps + wid] = v[q];
    }
}

// The CTAs of one cluster; `uses` counts reductions (warp 0 keeps it).
//
// A wait that expires leaves its CTA without totals, so without the decisions of the others. It
// tells every CTA (any_fail), sends no more partials, and settles: it goes on meeting the
// others at their barriers, and stays for their gathers, until each of them has settled too.
// They do at the latest in their next reduction, which lacks its partials: that wait sees
// any_fail and gives up. Nothing of this is on the path of a solve whose waits do not expire
// but the look at any_fail between two polls.
struct ClusterTeam {
    static constexpr bool kGrid = false;
    int rank, size;
    Shared* sh;
    long long budget;  // clock64 cycles a wait may take
    unsigned uses;

    __device__ void init() {
        for (int i = threadIdx.x; i < kMaxQ * kMaxCtas; i += kBlock) sh->part[0][i] = sh->part[1][i] = 0.0;
        if (threadIdx.x == 0) {
            sh->fail = sh->any_fail = 0;
            for (int r = 0; r < kMaxCtas; ++r) sh->settled[r] = 0;
            for (int h = 0; h < 2; ++h)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh->bar[h])) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        uses = 0;
        sync();
    }

    // Orders every CTA's writes of the gathered vector before any CTA's following gathers.
    __device__ __forceinline__ void sync() const {
        if (size == 1) __syncthreads();
        else cluster_barrier();
    }

    __device__ void tell(int* flag) const {  // flag = 1 in every CTA
        const uint32_t at = smem_addr(flag);
        for (int r = 0; r < size; ++r)
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote(at, r)), "r"(1) : "memory");
    }

    // The end of a solve, ok: without an expired wait in this CTA. True, in every thread of every
    // CTA alike, when none expired. No CTA returns while another may gather from it.
    __device__ bool settle(bool ok) const {
        if (size == 1) return ok;
        if (threadIdx.x == 0) {
            if (!ok) tell(&sh->any_fail);
            tell(&sh->settled[rank]);
        }
        if (ok) {
            sync();  // the same barrier for all CTAs whose waits were met; the others meet it too
            return *(volatile int*)&sh->any_fail == 0;
        }
        for (int b = 0, n = 0; n < size && b < 1 << 20; ++b) {
            sync();
            n = 0;
            for (int r = 0; r < size; ++r) n += *(volatile int*)&sh->settled[r];
        }
        return false;
    }

    // Before the CTA ends. When every wait was met no partial is on its way to it. Otherwise some
    // may be, and nothing counts them any more: one takes below 1,000 cycles, this 1,000 times that.
    __device__ void finish(bool ok) const {
        if (ok) return;
        for (const long long t0 = clock64(); clock64() - t0 < 1000000;) __nanosleep(1000);
    }

    // Totals over the cluster of Q values per thread: tot[k] = total of value k NRHS + lane,
    // on lanes < NRHS of warp 0 (which then sets the scalar state; a block barrier follows).
    template <int Q, int NRHS>
    __device__ __forceinline__ void reduce(double (&v)[Q], double (&tot)[Q / NRHS]) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        warp_sums(v, sh);
        __syncthreads();
        if (wid != 0) return;
        // lane q sums value q over the warps, and the partials over the CTAs below
        const int q = lane < Q ? lane : Q - 1, c = lane < NRHS ? lane : 0;
        double s = tree_sum<kWarps>(sh->warp + q * kWarps);
        if (size > 1) {
            const unsigned h = uses & 1u, phase = (uses >> 1) & 1u;
            ++uses;
            const uint32_t bar = smem_addr(&sh->bar[h]), slot = smem_addr(&sh->part[h][rank]);
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(8 * Q * size)
                             : "memory");
            // (value, CTA) pairs over the lanes; a half of `part` is written again two
            // reductions on, which no CTA starts before every CTA has read these partials
            for (int e0 = 0; e0 < Q * size; e0 += 32) {
                const int e = e0 + lane, eq = e % Q, to = e / Q;
                const double y = __shfl_sync(0xffffffffu, s, eq);
                if (to < size)
                    asm volatile(
                        "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(
                            remote(slot + 8 * kMaxCtas * eq, to)),
                        "d"(y), "r"(remote(bar, to))
                        : "memory");
            }
            uint32_t ok = 0;
            const long long t0 = clock64();
            for (unsigned poll = 1;; ++poll) {
                asm volatile(
                    "{ .reg .pred p;\n"
                    "  mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                    "  selp.u32 %0, 1, 0, p; }"
                    : "=r"(ok)
                    : "r"(bar), "r"(phase)
                    : "memory");
                if (ok) break;
                if (poll % 16 == 0 && (*(volatile int*)&sh->any_fail != 0 || clock64() - t0 > budget)) break;
            }
            if (!ok) sh->fail = 1;
            __syncwarp();
            s = tree_sum<kMaxCtas>(sh->part[h] + q * kMaxCtas);
        }
#pragma unroll
        for (int k = 0; k < Q / NRHS; ++k) tot[k] = __shfl_sync(0xffffffffu, s, k * NRHS + c);
    }
};

// The CTAs of one cooperative launch, one per SM. The counter only grows: a barrier is
// complete when it reaches the number of arrivals so far.
struct GridTeam {
    static constexpr bool kGrid = true;
    int rank, size;
    Shared* sh;
    long long budget;
    unsigned* count;   // arrivals, zeroed before the launch
    int* err;          // set when a wait expired; every other wait then gives up
    double* part;      // [2][kMaxQ][size]
    unsigned target, uses;

    __device__ void init() {
        if (threadIdx.x == 0) sh->fail = 0;
        target = uses = 0;
        __syncthreads();
    }

    // One thread: arrive (releasing what the block wrote), and wait for every CTA.
    __device__ __forceinline__ void arrive_and_wait() {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned seen;
        const long long t0 = clock64();
        for (unsigned poll = 1;; ++poll) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
            if ((int)(seen - target) >= 0) return;
            if (poll % 64 == 0 && (*(volatile int*)err != 0 || clock64() - t0 > budget)) break;
        }
        atomicCAS(err, 0, 5 /*KCFD_TIMEOUT*/);
        sh->fail = 1;
    }

    __device__ __forceinline__ void sync() {
        __syncthreads();
        target += size;
        if (threadIdx.x == 0) arrive_and_wait();
        __syncthreads();
    }

    // As ClusterTeam::settle. No CTA reads another's shared memory, so one that gave up leaves by
    // itself; err then ends the others' waits.
    __device__ __forceinline__ bool settle(bool ok) {
        if (!ok) return false;
        sync();
        return !sh->fail;
    }

    __device__ __forceinline__ void finish(bool) const {}

    // As ClusterTeam::reduce, the partials through global memory.
    template <int Q, int NRHS>
    __device__ __forceinline__ void reduce(double (&v)[Q], double (&tot)[Q / NRHS]) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        warp_sums(v, sh);
        __syncthreads();
        target += size;
        // a half of `part` is written again two reductions on, which no CTA starts before
        // every CTA has read these partials
        double* slots = part + (size_t)(uses++ & 1u) * kMaxQ * size;
        if (wid == 0) {
            if (lane < Q) __stcg(slots + lane * size + rank, tree_sum<kWarps>(sh->warp + lane * kWarps));
            __syncwarp();
            if (lane == 0) arrive_and_wait();
        }
        __syncthreads();
        // warp w sums values w, w + kWarps, ... over the CTAs, all its loads in flight together
#pragma unroll
        for (int q0 = 0; q0 < Q; q0 += kWarps) {
            const int q = q0 + wid;
            if (q < Q) {
                double s[kMaxGrid / 32];
#pragma unroll
                for (int j = 0; j < kMaxGrid / 32; ++j) {
                    const int at = lane + 32 * j;
                    s[j] = at < size ? __ldcg(slots + q * size + at) : 0.0;
                }
                double total = 0.0;
#pragma unroll
                for (int j = 0; j < kMaxGrid / 32; ++j) total += s[j];
                total = warp_sum(total);
                if (lane == 0) sh->total[q] = total;
            }
        }
        __syncthreads();
        const int c = threadIdx.x < NRHS ? threadIdx.x : 0;
#pragma unroll
        for (int k = 0; k < Q / NRHS; ++k) tot[k] = sh->total[k * NRHS + c];
    }
};

// The system of one CTA, carved from its dynamic shared memory; kRows local rows.
template <int NRHS, int PREC, int R, bool GRID>
struct Store {
    static constexpr int kRows = kBlock * R;
    double* vec;     // [kRows * NRHS] the gathered vector (a cluster's; the grid's is global)
    double* val;     // [width][kRows]
    double* lu;      // [width][kRows] (ILU)
    uint32_t* col;   // [width][kRows] address (cluster) or first element (grid) in the gathered vector
    int* loc;        // [nlev + 1] first local row of each level
    int* lev;        // [nlev + 1] first row of each level

    static size_t bytes(int width, int nlev) {
        return (size_t)kRows * ((GRID ? 0 : 8 * NRHS) + width * (PREC == KCFD_PREC_ILU0 ? 20 : 12)) + 8 * (size_t)(nlev + 1);
    }
    __device__ Store(char* base, int width, int nlev) {
        vec = (double*)base;
        val = GRID ? vec : vec + kRows * NRHS;
        lu = val + kRows * width;
        col = (uint32_t*)(PREC == KCFD_PREC_ILU0 ? lu + kRows * width : lu);
        loc = (int*)(col + kRows * width);
        lev = loc + nlev + 1;
    }
};

// Last l with t[l] <= i (t ascending, t[0] <= i < t[n]).
__device__ __forceinline__ int level_of(const int* t, int n, int i) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (t[mid] <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// A thread's part of the system: rows threadIdx.x + kBlock u, u < R.
template <int NRHS, int PREC, int R, class Team>
struct System {
    static constexpr int kRows = kBlock * R;
    Store<NRHS, PREC, R, Team::kGrid> s;
    int width, nlev;
    double* vec;     // the gathered vector; an unused row's part of the grid's lies past the last row
    double di[R];    // 1 / diagonal of A (Jacobi) or of U (ILU), 0 on unused rows
    int lv[R];       // ILU level, -1 on unused rows
    int dk[R];       // position of the diagonal in the row (ILU)
    int gi[R];       // matrix row (grid only)

    // The matrix row of local row t, -1 for an unused one.
    __device__ __forceinline__ int row_of(const Team& tm, int t, int& l) const {
        if (t >= s.loc[nlev]) return -1;
        l = nlev == 1 ? 0 : level_of(s.loc, nlev, t);
        const int i = s.lev[l] + tm.rank * (s.loc[l + 1] - s.loc[l]) + (t - s.loc[l]);
        return i < s.lev[l + 1] ? i : -1;
    }

    // The caller's row of local row t, -1 for an unused one.
    __device__ __forceinline__ int caller_row(const Team& tm, const SolveArgs& a, int t) const {
        int l;
        const int i = row_of(tm, t, l);
        return i >= 0 && a.perm ? a.perm[i] : i;
    }

    // Component 0 of the thread's row u in the gathered vector.
    __device__ __forceinline__ double* own(int u) const {
        return vec + (Team::kGrid ? (size_t)gi[u] * NRHS : (size_t)(threadIdx.x + u * kBlock) * NRHS);
    }
    __device__ __forceinline__ double get(uint32_t a, int c) const {
        // grid: a plain load; L1 serves the rows' common neighbours (the barrier before a
        // gather acquires, which drops what L1 held before it)
        return Team::kGrid ? vec[a + c] : ld_cluster(a + 8 * c);
    }

    // acc[u] = (A g) of the thread's rows, entries summed in row order; the gathers of K
    // entries of all R rows are in flight together.
    __device__ __forceinline__ void spmv(double (&acc)[R][NRHS]) const {
        constexpr int V = R * NRHS, K = V <= (Team::kGrid ? 3 : 1) ? 8 : V <= (Team::kGrid ? 4 : 3) ? 4 : 2;
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int c = 0; c < NRHS; ++c) acc[u][c] = 0.0;
        const uint32_t* col = s.col + threadIdx.x;
        const double* val = s.val + threadIdx.x;
#pragma unroll 1
        for (int k = 0; k < width; k += K, col += K * kRows, val += K * kRows) {
            double y[K][R][NRHS];
#pragma unroll
            for (int j = 0; j < K; ++j)
                if (k + j < width) {
#pragma unroll
                    for (int u = 0; u < R; ++u) {
                        const uint32_t a = col[j * kRows + u * kBlock];
#pragma unroll
                        for (int c = 0; c < NRHS; ++c) y[j][u][c] = get(a, c);
                    }
                }
#pragma unroll
            for (int j = 0; j < K; ++j)
                if (k + j < width) {
#pragma unroll
                    for (int u = 0; u < R; ++u) {
                        const double v = val[j * kRows + u * kBlock];
#pragma unroll
                        for (int c = 0; c < NRHS; ++c) acc[u][c] += v * y[j][u][c];
                    }
                }
        }
    }

    // g = (LU)^-1 q in the gathered vector; the own rows' part also in z. Level 0 of the
    // forward and the last level of the backward sweep need no other rows; the caller syncs
    // before anything gathers g.
    __device__ __forceinline__ void sweeps(Team& tm, const double (&q)[R][NRHS], double (&z)[R][NRHS]) const {
        const int last = nlev - 1;
#pragma unroll 1
        for (int l = 0; l < 2 * nlev - 1; ++l) {
            const bool fwd = l < nlev;
            const int level = fwd ? l : 2 * last - l;
            if (l > 0) tm.sync();
            double acc[R][NRHS];
#pragma unroll
            for (int u = 0; u < R; ++u)
#pragma unroll
                for (int c = 0; c < NRHS; ++c) acc[u][c] = fwd ? q[u][c] : z[u][c];
            if constexpr (Team::kGrid) sweep_rows(level, fwd, acc);
#pragma unroll
            for (int u = 0; u < R; ++u) {
                if (lv[u] != level) continue;
                if constexpr (!Team::kGrid) sweep_row(u, fwd ? 0 : dk[u] + 1, fwd ? dk[u] : width, acc[u]);
                const double d = fwd && level != last ? 1.0 : di[u];
#pragma unroll
                for (int c = 0; c < NRHS; ++c) own(u)[c] = z[u][c] = acc[u][c] * d;
            }
        }
    }

    // acc -= sum over entries [k0, k1) of the thread's row u of lu[k] g[col k] (clusters: the
    // rows of a level one after another, 2,440 cycles for the sweeps of 7,200 triangles
    // against 2,700 with all in flight).
    __device__ __forceinline__ void sweep_row(int u, int k0, int k1, double (&acc)[NRHS]) const {
        constexpr int K = NRHS == 1 ? 4 : 2;
        const int at = threadIdx.x + u * kBlock;
#pragma unroll 1
        for (int k = k0; k < k1; k += K) {
            double y[K][NRHS];
#pragma unroll
            for (int j = 0; j < K; ++j)
                if (k + j < k1) {
                    const uint32_t a = s.col[(k + j) * kRows + at];
#pragma unroll
                    for (int c = 0; c < NRHS; ++c) y[j][c] = get(a, c);
                }
#pragma unroll
            for (int j = 0; j < K; ++j)
                if (k + j < k1) {
                    const double v = s.lu[(k + j) * kRows + at];
#pragma unroll
                    for (int c = 0; c < NRHS; ++c) acc[c] -= v * y[j][c];
                }
        }
    }

    // The same for all the thread's rows of a level, their gathers in flight together (the
    // grid, where a gather is an L2 read) and without branches: past its last entry a row
    // repeats it with value 0, and so does, throughout, a row of another level.
    __device__ __forceinline__ void sweep_rows(int level, bool fwd, double (&acc)[R][NRHS]) const {
        int at[R], len[R], most = 0;  // first entry's place, entries
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int k0 = fwd ? 0 : dk[u] + 1;
            len[u] = lv[u] == level ? (fwd ? dk[u] : width) - k0 : 0;
            at[u] = (len[u] > 0 ? k0 : 0) * kRows + threadIdx.x + u * kBlock;
            most = max(most, len[u]);
        }
        auto batch = [&](auto count, int k) {
            constexpr int K = count();
            double y[K][R][NRHS];
#pragma unroll
            for (int j = 0; j < K; ++j)
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    const uint32_t a = s.col[at[u] + max(min(k + j, len[u] - 1), 0) * kRows];
#pragma unroll
                    for (int c = 0; c < NRHS; ++c) y[j][u][c] = get(a, c);
                }
#pragma unroll
            for (int j = 0; j < K; ++j)
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    const double v = k + j < len[u] ? s.lu[at[u] + (k + j) * kRows] : 0.0;
#pragma unroll
                    for (int c = 0; c < NRHS; ++c) acc[u][c] -= v * y[j][u][c];
                }
        };
        constexpr int kStep = R * NRHS <= 4 ? 3 : 1;
        if (R * NRHS <= 3 && most > 3 && most <= 6) {  // a hex's neighbours at once
            batch(std::integral_constant<int, R * NRHS <= 3 ? 6 : 1>(), 0);
        } else {
#pragma unroll 1
            for (int k = 0; k < most; k += kStep) batch(std::integral_constant<int, kStep>(), k);
        }
    }

    // Level tables, matrix and preconditioner on chip.
    __device__ void load(const Team& tm, const SolveArgs& a) {
        for (int l = threadIdx.x; l <= nlev; l += kBlock) s.lev[l] = nlev == 1 ? (l ? a.n : 0) : a.lev_ptr[l];
        __syncthreads();
        if (threadIdx.x == 0) {
            int at = 0;
            for (int l = 0; l < nlev; ++l) {
                s.loc[l] = at;
                at += (s.lev[l + 1] - s.lev[l] + tm.size - 1) / tm.size;
            }
            s.loc[nlev] = at;
        }
        __syncthreads();
        const uint32_t v0 = smem_addr(s.vec);
        const double* lu = (const double*)a.lu;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int t = threadIdx.x + u * kBlock;
            int li = -1;
            const int i = row_of(tm, t, li);
            const int kb = i >= 0 ? __ldg(a.indptr + i) : 0, len = i >= 0 ? __ldg(a.indptr + i + 1) - kb : 0;
            double d = 0.0;
#pragma unroll 4
            for (int k = 0; k < width; ++k) {
                // padding: the own row (the grid's unused rows: the one past the last), value 0
                uint32_t adr = Team::kGrid ? (uint32_t)(i >= 0 ? i : a.n) * NRHS : remote(v0 + 8 * NRHS * t, tm.rank);
                double v = 0.0, f = 0.0;
                if (k < len) {
                    const int j = __ldg(a.indices + kb + k);
                    v = a.vals64[kb + k];
                    if (PREC == KCFD_PREC_ILU0) f = lu[kb + k];
                    if (PREC == KCFD_PREC_JACOBI && j == i) d += v;
                    if (Team::kGrid) {
                        adr = (uint32_t)j * NRHS;
                    } else {
                        const int l = nlev == 1 ? 0 : level_of(s.lev, nlev, j);
                        const int per = s.loc[l + 1] - s.loc[l];
                        const int at = j - s.lev[l], rk = at / per;
                        adr = remote(v0 + 8 * NRHS * (s.loc[l] + at - rk * per), rk);
                    }
                }
                s.val[k * kRows + t] = v;
                s.col[k * kRows + t] = adr;
                if (PREC == KCFD_PREC_ILU0) s.lu[k * kRows + t] = f;
            }
            di[u] = 0.0;
            lv[u] = -1;
            dk[u] = 0;
            gi[u] = i >= 0 ? i : a.n;
            if (i >= 0 && PREC == KCFD_PREC_JACOBI)  // batched systems are set up here
                di[u] = a.dinv ? ((const double*)a.dinv)[i] : (fabs(d) > 1e-30 ? 1.0 / d : 0.0);
            if (i >= 0 && PREC == KCFD_PREC_ILU0) {
                di[u] = ((const double*)a.ludinv)[i];
                lv[u] = li;
                dk[u] = __ldg(a.diag + i) - kb;
            }
        }
    }
};

// Scalar state of one right-hand side (lane c of warp 0).
struct Scalars {
    double rho = 0, rho_prev = 1, alpha = 1, omega = 1, beta = 0, thr = 0, bnorm = 0, rnorm = 0;
    int done = 1, status = KCFD_OK, iters = 0, restarts = 0, restart = 0;

    // Stopping and breakdown tests before iteration `it`, and its beta.
    __device__ void top(const SolveArgs& a, bool gpu, int it, int maxiter) {
        beta = 0.0;
        restart = 0;
        if (done) return;
        if (it >= maxiter) return stop(KCFD_MAXITER, maxiter);
        if (!gpu) {
            if (rnorm < thr) { done = 1; status = KCFD_OK; return; }
            if (fabs(rho) < kEps2 || (it > 0 && fabs(omega) < kEps2)) {
                if (restarts < a.max_restarts && rnorm > 0.0) {
                    // rhat = r, p = r (this iteration), rho = ||r||^2
                    restarts += 1;
                    restart = 1;
                    rho = rnorm * rnorm;
                    rho_prev = alpha = omega = 1.0;
                } else {
                    done = 1;
                    status = KCFD_BREAKDOWN;
                }
                return;
            }
            if (it > 0) beta = (rho / rho_prev) * (alpha / omega);
        } else {
            if (fabs(rho) < 1e-30) return stop(KCFD_BREAKDOWN, it + 1);
            beta = fabs(rho_prev * omega) > 1e-30 ? (rho / rho_prev) * (alpha / omega) : 0.0;
        }
        if (!isfinite(beta)) { done = 1; status = KCFD_BREAKDOWN; }
    }
    __device__ void stop(int st, int it) {
        done = 1;
        status = st;
        iters = it;
    }
};

// The iteration, from x and b (in t), with the scalar formulas and tests of bicgstab_body
// (solver.cu). Returns false when this CTA gave up a wait.
template <int NRHS, int PREC, int R, class Team>
__device__ __forceinline__ bool iterate(Team& tm, const System<NRHS, PREC, R, Team>& S, const SolveArgs& a, int maxiter,
                                        double (&x)[R][NRHS], double (&t)[R][NRHS], Scalars& sc) {
    constexpr bool kPrec = PREC != KCFD_PREC_NONE;
    Shared& sh = *tm.sh;
    const bool gpu = a.stop == KCFD_STOP_GPU;
    const int lane = threadIdx.x & 31;
    const bool mine = threadIdx.x < NRHS;
    double r[R][NRHS], rh[R][NRHS], p[R][NRHS], v[R][NRHS], ph[R][NRHS], shat[R][NRHS];
    double al[NRHS], om[NRHS], be[NRHS];
    int fl[NRHS];
    auto put = [&](const double (&y)[R][NRHS]) {  // y into the gathered vector
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int c = 0; c < NRHS; ++c) S.own(u)[c] = y[u][c];
    };
    auto publish = [&](int flags) {  // the lane's scalars, to the block
        sh.al[lane] = sc.alpha;
        sh.om[lane] = sc.omega;
        sh.be[lane] = sc.beta;
        sh.flags[lane] = (sc.done ? kDone : 0) | (sc.restart ? kRestart : 0) | flags;
    };
    // after the block barrier: every thread's copy; false when no right-hand side is left
    auto fetch = [&]() {
        int all = kDone;
#pragma unroll
        for (int c = 0; c < NRHS; ++c) {
            al[c] = sh.al[c];
            om[c] = sh.om[c];
            be[c] = sh.be[c];
            fl[c] = sh.flags[c];
            all &= fl[c];
        }
        return !(all & kDone);
    };
    bool active;
    {
        // r = b - A x, rhat = r, ||b||^2, ||r||^2
        double red[2 * NRHS], tot[2];
#pragma unroll
        for (int k = 0; k < 2 * NRHS; ++k) red[k] = 0.0;
        put(x);
        tm.sync();
        S.spmv(r);
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int c = 0; c < NRHS; ++c) {
                r[u][c] = rh[u][c] = t[u][c] - r[u][c];
                p[u][c] = v[u][c] = ph[u][c] = shat[u][c] = 0.0;
                red[c] += t[u][c] * t[u][c];
                red[NRHS + c] += r[u][c] * r[u][c];
            }
        tm.template reduce<2 * NRHS, NRHS>(red, tot);
        if (mine) {
            sc = Scalars();
            sc.done = 0;
            sc.bnorm = sqrt(tot[0]);
            sc.rnorm = sqrt(tot[1]);
            sc.rho = tot[1];
            sc.thr = gpu ? a.rtol : fmax(a.atol, a.rtol * sc.bnorm);
            sc.done = gpu ? sc.bnorm < 1e-30 : sc.bnorm == 0.0;
            const int zero = !gpu && sc.done ? kZero : 0;  // scipy returns b (== 0) as the solution
            if (!isfinite(tot[0]) || !isfinite(tot[1])) sc.stop(KCFD_BREAKDOWN, 0);
            sc.top(a, gpu, 0, maxiter);
            publish(zero);
        }
        __syncthreads();
        if (sh.fail) return false;
        active = fetch();
#pragma unroll
        for (int c = 0; c < NRHS; ++c)
            if (fl[c] & kZero) {
#pragma unroll
                for (int u = 0; u < R; ++u) x[u][c] = 0.0;
            }
    }
#pragma unroll 1
    for (int it = 0; active; ++it) {
        // ---- p, phat = M^-1 p ----
#pragma unroll
        for (int c = 0; c < NRHS; ++c) {
            if (fl[c] & kDone) continue;
#pragma unroll
            for (int u = 0; u < R; ++u) {
                double pn;
                if (gpu) pn = r[u][c] + be[c] * (p[u][c] - om[c] * v[u][c]);
                else if (it == 0 || (fl[c] & kRestart)) pn = r[u][c];
                else pn = (p[u][c] - om[c] * v[u][c]) * be[c] + r[u][c];
                if (fl[c] & kRestart) rh[u][c] = r[u][c];
                p[u][c] = pn;
                if (PREC == KCFD_PREC_JACOBI) ph[u][c] = S.di[u] * pn;
            }
        }
        if (PREC == KCFD_PREC_ILU0) S.sweeps(tm, p, ph);
        else put(kPrec ? ph : p);
        tm.sync();
        // ---- v = A phat, rhat.v ----
        double r1[NRHS], t1[1];
        S.spmv(v);
#pragma unroll
        for (int c = 0; c < NRHS; ++c) {
            r1[c] = 0.0;
#pragma unroll
            for (int u = 0; u < R; ++u) r1[c] += rh[u][c] * v[u][c];
        }
        tm.template reduce<NRHS, NRHS>(r1, t1);
        if (mine) {
            if (!sc.done) {
                if (gpu) sc.alpha = fabs(t1[0]) > 1e-30 ? sc.rho / t1[0] : 0.0;
                else if (t1[0] == 0.0) sc.stop(KCFD_BREAKDOWN, it + 1);
                else sc.alpha = sc.rho / t1[0];
                if (!sc.done && !isfinite(sc.alpha)) sc.stop(KCFD_BREAKDOWN, it + 1);
            }
            publish(0);
        }
        __syncthreads();
        if (sh.fail) return false;
        if (!fetch()) break;
        // ---- s = r - alpha v (in r), shat = M^-1 s, ||s||^2 ----
        double r3[3 * NRHS], t3[3];
#pragma unroll
        for (int k = 0; k < 3 * NRHS; ++k) r3[k] = 0.0;
#pragma unroll
        for (int c = 0; c < NRHS; ++c) {
            if (fl[c] & kDone) continue;
#pragma unroll
            for (int u = 0; u < R; ++u) {
                r[u][c] = r[u][c] - al[c] * v[u][c];
                if (PREC == KCFD_PREC_JACOBI) shat[u][c] = S.di[u] * r[u][c];
                r3[c] += r[u][c] * r[u][c];
            }
        }
        if (PREC == KCFD_PREC_ILU0) S.sweeps(tm, r, shat);
        else put(kPrec ? shat : r);
        tm.sync();
        // ---- t = A shat, t.s, t.t ----
        S.spmv(t);
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int c = 0; c < NRHS; ++c) {
                r3[NRHS + c] += t[u][c] * r[u][c];
                r3[2 * NRHS + c] += t[u][c] * t[u][c];
            }
        tm.template reduce<3 * NRHS, NRHS>(r3, t3);
        if (mine) {
            int sconv = 0;
            if (!sc.done) {
                const double sn = sqrt(t3[0]);
                if (!isfinite(sn)) {
                    sc.stop(KCFD_BREAKDOWN, it + 1);
                } else if (gpu ? sn / sc.bnorm < sc.thr : sn < sc.thr) {
                    sc.stop(KCFD_OK, it + 1);  // x += alpha phat below
                    sc.rnorm = sn;
                    sconv = kSconv;
                } else {
                    if (gpu) sc.omega = t3[2] > 1e-30 ? t3[1] / t3[2] : 0.0;
                    else sc.omega = t3[1] / t3[2];
                    if (!isfinite(sc.omega)) sc.stop(KCFD_BREAKDOWN, it + 1);
                }
            }
            publish(sconv);
        }
        __syncthreads();
        if (sh.fail) return false;
        active = fetch();
        // ---- x += alpha phat + omega shat, r = s - omega t, rhat.r, ||r||^2 ----
        double r4[2 * NRHS], t4[2];
#pragma unroll
        for (int k = 0; k < 2 * NRHS; ++k) r4[k] = 0.0;
#pragma unroll
        for (int c = 0; c < NRHS; ++c) {
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const double hp = kPrec ? ph[u][c] : p[u][c], hs = kPrec ? shat[u][c] : r[u][c];
                if (fl[c] & kSconv) x[u][c] += al[c] * hp;
                if (fl[c] & kDone) continue;
                if (gpu) x[u][c] += al[c] * hp + om[c] * hs;
                else x[u][c] = (x[u][c] + al[c] * hp) + om[c] * hs;
                r[u][c] = r[u][c] - om[c] * t[u][c];
                r4[c] += rh[u][c] * r[u][c];
                r4[NRHS + c] += r[u][c] * r[u][c];
            }
        }
        if (!active) break;
        tm.template reduce<2 * NRHS, NRHS>(r4, t4);
        if (mine) {
            if (!sc.done) {
                sc.rho_prev = sc.rho;
                sc.rho = t4[0];
                sc.rnorm = sqrt(t4[1]);
                sc.iters = it + 1;
                if (!isfinite(sc.rnorm) || !isfinite(sc.rho)) sc.stop(KCFD_BREAKDOWN, it + 1);
                else if (gpu && sc.rnorm / sc.bnorm < sc.thr) sc.stop(KCFD_OK, it + 1);
                sc.top(a, gpu, it + 1, maxiter);
            }
            publish(0);
        }
        __syncthreads();
        if (sh.fail) return false;
        active = fetch();
    }
    return true;
}

// FP64 solve on chip, with the true-residual passes of solve_fp64 (solver.cu). gvec: the
// grid's gathered vector, (n + 1) NRHS elements. comps > 1 (NRHS 1): that many interleaved
// right-hand sides, one after another on the same matrix. False when a wait expired.
template <int NRHS, int PREC, int R, class Team>
__device__ bool solve_on_chip(Team& tm, const SolveArgs& a, int width, char* store, double* gvec = nullptr,
                              int comps = 1) {
    System<NRHS, PREC, R, Team> S{Store<NRHS, PREC, R, Team::kGrid>(store, width, a.nlev), width, a.nlev};
    S.vec = Team::kGrid ? gvec : S.s.vec;
    S.load(tm, a);
    const int stride = NRHS * comps;
    const bool verify = NRHS == 1 && a.max_restarts > 0 && a.stop == KCFD_STOP_SCIPY;
    bool ok = true;
    for (int comp = 0; comp < comps && ok; ++comp) {
        double x[R][NRHS], t[R][NRHS];
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int o = S.caller_row(tm, a, threadIdx.x + u * kBlock);
#pragma unroll
            for (int c = 0; c < NRHS; ++c) x[u][c] = o >= 0 ? a.x[(size_t)o * stride + comp + c] : 0.0;
        }
        Scalars sc;
        int used = 0;
        for (int pass = 0;; ++pass) {
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int o = S.caller_row(tm, a, threadIdx.x + u * kBlock);
#pragma unroll
                for (int c = 0; c < NRHS; ++c) t[u][c] = o >= 0 ? a.b[(size_t)o * stride + comp + c] : 0.0;
            }
            ok = iterate<NRHS, PREC, R, Team>(tm, S, a, a.maxiter - used, x, t, sc);
            if (threadIdx.x == 0) {
                tm.sh->status = sc.status;
                tm.sh->iters = sc.iters;
            }
            __syncthreads();
            used += tm.sh->iters;
            if (!ok || !verify || pass >= kVerifyPasses || tm.sh->status != KCFD_OK || tm.sh->iters == 0 ||
                used >= a.maxiter)
                break;
            tm.sync();  // every gather of the last pass before the next one writes the vector
        }
        ok = tm.settle(ok);
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int o = S.caller_row(tm, a, threadIdx.x + u * kBlock);
#pragma unroll
            for (int c = 0; c < NRHS; ++c)
                if (o >= 0) a.x[(size_t)o * stride + comp + c] = x[u][c];
        }
        if (tm.rank == 0 && threadIdx.x < NRHS) {
            const int c = comp + threadIdx.x;
            if (a.iters_out) a.iters_out[c] = verify ? used : sc.iters;
            if (a.status_out) a.status_out[c] = ok ? sc.status : 5 /*KCFD_TIMEOUT*/;
            if (a.relres_out) a.relres_out[c] = sc.bnorm > 0 ? sc.rnorm / sc.bnorm : 0.0;
        }
        if (!Team::kGrid && a.ctl.err && tm.rank == 0 && threadIdx.x == 0) *a.ctl.err = ok ? 0 : 5 /*KCFD_TIMEOUT*/;
    }
    return ok;
}

}  // namespace res
}  // namespace kcfd
