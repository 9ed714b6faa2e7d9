// Face loops of the finite-volume operators, one thread per cell.
//
// A cell goes over its own faces (cf_ptr / cf_face, ascending reference face id: the
// reference's summation order), adds up its row's sums in registers and writes each of them
// once; a row's off-diagonal entries are written by its own thread only, so no face colours,
// atomics or zeroed accumulators are needed. Faces that lead to the same cell share one entry;
// a step that holds two of them adds them one after another. The colour-by-colour
// scatter that this replaces (one launch per colour, kept for meshes without cell lists)
// reads and rewrites the owner's and the neighbour's sums once per colour, with 8 bytes used
// of every 32-byte sector. A face's data is read twice, the second time mostly from L2.
// These loops are bound by the latency of the chain list -> face -> other cell and row entry:
// each step issues the loads of B faces before it uses any, and both slots of a face are
// loaded so that the row entry does not wait for the owner. (4 or 8 lanes per cell, a face
// per lane, coalesce better but keep fewer loads in flight: 97-183 us for the operators of
// operators.cu on 96^3 hexes against 54-67.)
#pragma once
#include <cuda_runtime.h>

#include "kcfd_common.h"

namespace kcfd {

// A face as one of its cells sees it; other == the cell itself on a boundary face.
struct CellFace {
    int f, other;
    bool own, in;  // the cell is its owner; it is an internal face
};

inline bool has_cell_lists(const kcfd_dmesh_t* m) { return m->cf_ptr && m->cf_face; }

// Op: Acc begin(m, i); Data load(m, i, face, acc) (loads only); double apply(face, data,
// acc), which adds to the sums and returns what the row's entry across the face gains (kOff;
// values in op.v); end(m, i, acc).
template <int B, class Op>
__global__ void __launch_bounds__(256) k_by_cell(kcfd_dmesh_t m, Op op) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n_cells) return;
    const int e1 = __ldg(m.cf_ptr + i + 1);
    typename Op::Acc acc = op.begin(m, i);
    for (int e = __ldg(m.cf_ptr + i); e < e1; e += B) {
        CellFace c[B];
        int on[B], no[B], nb[B];
        double old[B];
        typename Op::Data d[B];
#pragma unroll
        for (int u = 0; u < B; ++u) c[u].f = __ldg(m.cf_face + min(e + u, e1 - 1));
#pragma unroll
        for (int u = 0; u < B; ++u) {
            c[u].other = __ldg(m.owner + c[u].f);
            c[u].in = c[u].f < m.n_internal;
            nb[u] = c[u].in ? __ldg(m.neigh + c[u].f) : i;
            if constexpr (Op::kOff) {
                on[u] = c[u].in ? __ldg(m.slot_on + c[u].f) : 0;
                no[u] = c[u].in ? __ldg(m.slot_no + c[u].f) : 0;
            }
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
            c[u].own = c[u].other == i;
            if (c[u].own) c[u].other = nb[u];
            if constexpr (Op::kOff) {
                if (!c[u].own) on[u] = no[u];
                old[u] = c[u].in ? op.v[on[u]] : 0.0;
            }
            d[u] = op.load(m, i, c[u], acc);
        }
        if constexpr (Op::kOff) {
            bool shared = false;  // two faces to the same cell (not the padding of a last step)
#pragma unroll
            for (int u = 1; u < B; ++u)
#pragma unroll
                for (int w = 0; w < u; ++w) shared |= c[u].in && e + u < e1 && on[w] == on[u];
            if (shared) {
#pragma unroll
                for (int u = 0; u < B; ++u) {
                    if (e + u >= e1) break;
                    const double add = op.apply(c[u], d[u], acc);
                    if (c[u].in) op.v[on[u]] += add;
                }
                continue;
            }
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
            if (e + u >= e1) break;
            const double add = op.apply(c[u], d[u], acc);
            if constexpr (Op::kOff) {
                if (c[u].in) op.v[on[u]] = old[u] + add;
            }
        }
    }
    op.end(m, i, acc);
}

template <class Op>
void by_cell(const kcfd_dmesh_t* m, const Op& op, cudaStream_t st) {
    if (m->n_cells <= 0) return;
    // three faces a step: 32-62 registers. On 96^3 hexes (diffusion, convection, MUSCL): 67, 54
    // and 66 us. The sizes against one another, measured before a step looked for shared entries:
    // three 70, 57 and 66; two 70, 105 and 66; four 74, 57 and 76; six 84, 88 and 80
    k_by_cell<3, Op><<<(m->n_cells + 255) / 256, 256, 0, st>>>(*m, op);
}

// Boundary faces only: the thread of a cell's first boundary face does all of them.
// Op: Acc begin(m, i); face(m, i, f, acc); end(m, i, acc).
template <class Op>
__global__ void __launch_bounds__(256) k_by_boundary_cell(kcfd_dmesh_t m, Op op) {
    const int f0 = m.n_internal + blockIdx.x * blockDim.x + threadIdx.x;
    if (f0 >= m.n_faces) return;
    const int i = __ldg(m.owner + f0);
    const int e1 = __ldg(m.cf_ptr + i + 1);
    int e = __ldg(m.cf_ptr + i);
    while (e < e1 && __ldg(m.cf_face + e) < m.n_internal) ++e;
    if (e == e1 || __ldg(m.cf_face + e) != f0) return;
    typename Op::Acc acc = op.begin(m, i);
    for (; e < e1; ++e) {
        const int f = __ldg(m.cf_face + e);
        if (f >= m.n_internal) op.face(m, i, f, acc);
    }
    op.end(m, i, acc);
}

template <class Op>
void by_boundary_cell(const kcfd_dmesh_t* m, const Op& op, cudaStream_t st) {
    const int fb = m->n_faces - m->n_internal;
    if (fb > 0) k_by_boundary_cell<Op><<<(fb + 255) / 256, 256, 0, st>>>(*m, op);
}

// apply_boundary_conditions (core/fvm_operators.py:178-225) for nc right-hand sides
// sharing one matrix. bt: 0 zero_gradient, 1 dirichlet, 2 neumann per boundary face.
struct BoundaryOp {
    const int8_t* bt;
    const double *bv, *bg;
    int nc;
    const double *gamma, *mf;
    double *v, *diag, *rhs;
    struct Acc {
        double vd, dg, r[3];
    };
    __device__ Acc begin(const kcfd_dmesh_t& m, int i) const {
        Acc a{v[__ldg(m.diag_slot + i)], diag[i], {0.0, 0.0, 0.0}};
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (k < nc) a.r[k] = rhs[i * nc + k];
        return a;
    }
    __device__ void face(const kcfd_dmesh_t& m, int i, int f, Acc& a) const {
        const double d = __ldg(m.dlen + f);
        if (d < 1e-30) return;
        const int bi = f - m.n_internal, t = bt[bi];
        const double F = mf[f];
        if (t == 1) {
            const double c = gamma[i] * __ldg(m.area + f) / d;
            a.vd += c;
            a.dg += c;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (k >= nc) break;
                const double phib = bv[bi * nc + k];
                double add = c * phib;
                if (F < 0) add = add + (-F) * phib;
                a.r[k] += add;
            }
        } else if (t == 2) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (k < nc) a.r[k] += bg[bi] * __ldg(m.area + f);
        } else if (t == 0 && F < 0) {
            a.vd += -F;
            a.dg += -F;
        }
    }
    __device__ void end(const kcfd_dmesh_t& m, int i, const Acc& a) const {
        v[__ldg(m.diag_slot + i)] = a.vd;
        diag[i] = a.dg;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (k < nc) rhs[i * nc + k] = a.r[k];
    }
};

}  // namespace kcfd
