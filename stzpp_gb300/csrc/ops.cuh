// Row evaluation of the three operator kinds: acc -= sum_{blocks} A x over a
// node's 3x3x3 box, with or without the centre block, plus the centre solve.
// Reference: region::gauss_seidel (mg_3d_template/region.cc:1557-1762) and
// region::residual (region.cc:1008-1055); the constant stencil is the one of
// shear_sim_3d::set_up_stencil_base (src/shear_sim_3d.cpp:215-331).
#pragma once

#include "common.cuh"

namespace stzmg {

// Offsets (dx,dy,dz) of block b.
__host__ __device__ constexpr int bdx(int b) { return b % 3 - 1; }
__host__ __device__ constexpr int bdy(int b) { return (b / 3) % 3 - 1; }
__host__ __device__ constexpr int bdz(int b) { return b / 9 - 1; }
__host__ __device__ constexpr int nnz_axes(int b) {
    return (bdx(b) != 0) + (bdy(b) != 0) + (bdz(b) != 0);
}
// Whether entry e (row*3+col) of block b can be non-zero in the elasticity
// stencil: faces are diagonal, edges couple the two components of their
// plane symmetrically, corners are zero, the centre is full.
__host__ __device__ constexpr bool elastic_entry(int b, int e) {
    return b == 13 ? true
         : nnz_axes(b) == 1 ? (e == 0 || e == 4 || e == 8)
         : nnz_axes(b) == 2 ? (bdz(b) == 0 ? (e == 1 || e == 3)
                             : bdy(b) == 0 ? (e == 2 || e == 6)
                                           : (e == 5 || e == 7))
         : false;
}

// COH: the field is written by other blocks of the same launch (the
// persistent small-level kernel), so read it through L2 (ld.global.cg), not
// from a possibly stale L1 line.
template <typename T, bool COH = false>
__device__ inline void load3(const T *f, int npad, int s, T *v) {
    if (COH) {
        v[0] = load_l2(f + s);
        v[1] = load_l2(f + s + npad);
        v[2] = load_l2(f + s + 2 * npad);
    } else {
        v[0] = f[s];
        v[1] = f[s + npad];
        v[2] = f[s + 2 * npad];
    }
}

// ---------------------------------------------------------------- constant
// acc -= sum_{b (!= 13 unless WITH_CENTRE)} a[b] x_b   for an interior node.
template <typename T, bool ELASTIC, bool WITH_CENTRE>
__device__ inline void const_row(const ConstOp<T> &op, const Geom &g, const NbrOffsets &t,
                                 const T *__restrict__ x, T *acc) {
    // neighbour components first (only those the stencil uses), then arithmetic
    T v[27][3];
#pragma unroll
    for (int b = 0; b < 27; b++) {
        if (b == 13 && !WITH_CENTRE) continue;
        if (ELASTIC && nnz_axes(b) == 3) continue;
        int s = t.ox[bdx(b) + 1] + t.oy[bdy(b) + 1] + t.oz[bdz(b) + 1];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            bool used = !ELASTIC || b == 13;
#pragma unroll
            for (int r = 0; r < 3; r++) used = used || elastic_entry(b, 3 * r + c);
            v[b][c] = used ? x[s + c * g.npad] : T(0);
        }
    }
#pragma unroll
    for (int b = 0; b < 27; b++) {
        if (b == 13 && !WITH_CENTRE) continue;
        if (ELASTIC && nnz_axes(b) == 3) continue;
        if (ELASTIC && b != 13) {
#pragma unroll
            for (int e = 0; e < 9; e++)
                if (elastic_entry(b, e)) acc[e / 3] -= op.a[b][e] * v[b][e % 3];
        } else if (b == 13 && op.centre_diag) {
            // a diagonal centre block (the elasticity stencil): only its three
            // non-zero products are formed
            acc[0] -= op.a[13][0] * v[13][0];
            acc[1] -= op.a[13][4] * v[13][1];
            acc[2] -= op.a[13][8] * v[13][2];
        } else {
            matvec_sub(op.a[b], v[b], acc);
        }
    }
}

// ---------------------------------------------------------------- Lame
// Stencil of the variable-coefficient operator -dt*div(mu(grad u + grad u^T)
// + lam div(u) I): face blocks from midpoint-averaged coefficients, edge
// blocks from node values (block (+1,+1,0): a12 = (lam[i+1,j] + mu[i,j+1])/(4dxdy)).
// Reduces to the constant stencil for constant mu, lam.
template <typename T>
struct LameRow {
    T face[6][3];     // face diagonal, order x-, x+, y-, y+, z-, z+
    T centre[3];      // diagonal of the centre block
};

template <typename T>
__device__ inline void lame_faces(const LameOp<T> &op, const Geom &g, const NbrOffsets &t, int p,
                                  LameRow<T> &L, T mu_nb[6], T lam_nb[6]) {
    const T mu0 = op.mu[p], lam0 = op.lam[p];
    const int ctr_x = t.ox[1], ctr_y = t.oy[1], ctr_z = t.oz[1];
    const int sl[6] = {t.ox[0] + ctr_y + ctr_z, t.ox[2] + ctr_y + ctr_z, ctr_x + t.oy[0] + ctr_z,
                       ctr_x + t.oy[2] + ctr_z, ctr_x + ctr_y + t.oz[0], ctr_x + ctr_y + t.oz[2]};
    T cen[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int f = 0; f < 6; f++) {
        mu_nb[f] = op.mu[sl[f]];
        lam_nb[f] = op.lam[sl[f]];
        const int ax = f / 2;
        T mu_f = T(0.5) * (mu0 + mu_nb[f]);
        T lam_f = T(0.5) * (lam0 + lam_nb[f]);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            T v = (c == ax ? (lam_f + T(2) * mu_f) : mu_f) * op.ih2[ax];
            L.face[f][c] = -op.dt * v;
            cen[c] -= v;
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) L.centre[c] = -op.dt * cen[c];
}

// The same row in FP64, whose pipe bounds it: the factors dt/h^2 enter once
// per axis and pair instead of once per entry, 117 instructions for 187.
template <bool WITH_CENTRE>
__device__ inline void lame_row64(const LameOp<double> &op, const Geom &g, const NbrOffsets &t, int p,
                                  const double *__restrict__ x, double *acc, double *centre_out) {
    const int npad = g.npad;
    const int mid = t.ox[1] + t.oy[1] + t.oz[1];
    const double mu0 = op.mu[p], lam0 = op.lam[p];
    double mu[6], lam[6], cen[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
        double s[2], w[2], v[2][3];   // mu0 + mu, lam0 + lam + 2 (mu0 + mu) and x of the faces below and above
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int *o = ax == 0 ? t.ox : ax == 1 ? t.oy : t.oz;
            const int sl = mid - o[1] + o[2 * u];
            mu[2 * ax + u] = op.mu[sl];
            lam[2 * ax + u] = op.lam[sl];
            load3(x, npad, sl, v[u]);
            s[u] = mu0 + mu[2 * ax + u];
            w[u] = fma_rn(2.0, s[u], lam0 + lam[2 * ax + u]);
        }
        const double ss = s[0] + s[1], ws = w[0] + w[1];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double lo = c == ax ? w[0] : s[0], hi = c == ax ? w[1] : s[1];
            acc[c] = fma_rn(op.face[ax], fma_rn(hi, v[1][c], mul_rn(lo, v[0][c])), acc[c]);
            cen[c] = fma_rn(op.face[ax], c == ax ? ws : ss, cen[c]);
        }
    }
#pragma unroll
    for (int pr = 0; pr < 3; pr++) {
        const int r = pr == 2 ? 1 : 0, c = pr == 0 ? 1 : 2;
        double er = 0.0, ec = 0.0;
#pragma unroll
        for (int ir = 0; ir < 2; ir++)
#pragma unroll
            for (int ic = 0; ic < 2; ic++) {
                int d[3] = {1, 1, 1};
                d[r] = 2 * ir;
                d[c] = 2 * ic;
                const int sl = t.ox[d[0]] + t.oy[d[1]] + t.oz[d[2]];
                const double a = lam[2 * r + ir] + mu[2 * c + ic], b = lam[2 * c + ic] + mu[2 * r + ir];
                er = fma_rn(ir == ic ? a : -a, x[sl + c * npad], er);
                ec = fma_rn(ir == ic ? b : -b, x[sl + r * npad], ec);
            }
        acc[r] = fma_rn(op.edge[pr], er, acc[r]);
        acc[c] = fma_rn(op.edge[pr], ec, acc[c]);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        if (WITH_CENTRE) acc[c] = fma_rn(-cen[c], x[p + c * npad], acc[c]);
        if (centre_out) centre_out[c] = cen[c];
    }
}

// acc -= sum over the 18 non-zero off-centre blocks (and the centre if asked),
// the node's surroundings given by `at`: at.mu0, at.lam0 its coefficients,
// at.mu(f), at.lam(f) those of its face neighbours (x-, x+, y-, y+, z-, z+) and
// at.x(dx, dy, dz, c) the component c of a neighbour.
template <typename T, bool WITH_CENTRE, typename N>
__device__ __forceinline__ void lame_row_of(const LameOp<T> &op, const N &at, T *acc, T *centre_out) {
    T mu_nb[6], lam_nb[6], face[6][3], centre[3];
    T cen[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int f = 0; f < 6; f++) {
        mu_nb[f] = at.mu(f);
        lam_nb[f] = at.lam(f);
        const int ax = f / 2;
        T mu_f = T(0.5) * (at.mu0 + mu_nb[f]);
        T lam_f = T(0.5) * (at.lam0 + lam_nb[f]);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            T v = (c == ax ? (lam_f + T(2) * mu_f) : mu_f) * op.ih2[ax];
            face[f][c] = -op.dt * v;
            cen[c] -= v;
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) centre[c] = -op.dt * cen[c];
    // faces
#pragma unroll
    for (int f = 0; f < 6; f++) {
        const int ax = f / 2, d = f & 1 ? 1 : -1;
#pragma unroll
        for (int c = 0; c < 3; c++)
            acc[c] -= face[f][c] * at.x(ax == 0 ? d : 0, ax == 1 ? d : 0, ax == 2 ? d : 0, c);
    }
    // edges: component pair (r, c) in the plane of axes (r, c)
#pragma unroll
    for (int pr = 0; pr < 3; pr++) {
        const int r = pr == 2 ? 1 : 0, c = pr == 0 ? 1 : 2;
        const T ie = op.iedge[pr];
#pragma unroll
        for (int sr = -1; sr <= 1; sr += 2)
#pragma unroll
            for (int sc = -1; sc <= 1; sc += 2) {
                int d[3] = {0, 0, 0};
                d[r] = sr;
                d[c] = sc;
                const T sgn = T(sr * sc);
                // neighbour coefficient values: lam/mu at p + sr e_r and p + sc e_c
                const T lam_r = lam_nb[2 * r + (sr > 0)], mu_r = mu_nb[2 * r + (sr > 0)];
                const T lam_c = lam_nb[2 * c + (sc > 0)], mu_c = mu_nb[2 * c + (sc > 0)];
                const T a_rc = -op.dt * ((sgn * (lam_r + mu_c)) * ie);
                const T a_cr = -op.dt * ((sgn * (lam_c + mu_r)) * ie);
                acc[r] -= a_rc * at.x(d[0], d[1], d[2], c);
                acc[c] -= a_cr * at.x(d[0], d[1], d[2], r);
            }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        if (WITH_CENTRE) acc[c] -= centre[c] * at.x(0, 0, 0, c);
        if (centre_out) centre_out[c] = centre[c];
    }
}

// The surroundings in the level's fields.
template <typename T>
struct LameNode {
    const LameOp<T> &op;
    const NbrOffsets &t;
    const T *x_;
    int npad;
    T mu0, lam0;
    __device__ __forceinline__ LameNode(const LameOp<T> &op, const Geom &g, const NbrOffsets &t, int p, const T *x)
        : op(op), t(t), x_(x), npad(g.npad), mu0(op.mu[p]), lam0(op.lam[p]) {}
    __device__ __forceinline__ int face(int f) const {
        const int s = f & 1 ? 2 : 0;
        return t.ox[f / 2 == 0 ? s : 1] + t.oy[f / 2 == 1 ? s : 1] + t.oz[f / 2 == 2 ? s : 1];
    }
    __device__ __forceinline__ T mu(int f) const { return op.mu[face(f)]; }
    __device__ __forceinline__ T lam(int f) const { return op.lam[face(f)]; }
    __device__ __forceinline__ T x(int dx, int dy, int dz, int c) const {
        return x_[t.ox[dx + 1] + t.oy[dy + 1] + t.oz[dz + 1] + c * npad];
    }
};

template <typename T, bool WITH_CENTRE>
__device__ inline void lame_row(const LameOp<T> &op, const Geom &g, const NbrOffsets &t, int p,
                                const T *__restrict__ x, T *acc, T *centre_out) {
    if constexpr (sizeof(T) == 8) lame_row64<WITH_CENTRE>(op, g, t, p, x, acc, centre_out);
    else lame_row_of<T, WITH_CENTRE>(op, LameNode<T>(op, g, t, p, x), acc, centre_out);
}

template <typename T>
__device__ inline T lame_fix(const LameOp<T> &op, int p) {
    const T mu0 = op.mu[p], lam0 = op.lam[p];
    return (-op.dt * T(2)) * ((lam0 + T(2) * mu0) * op.ih2[0] + mu0 * op.ih2[1] + mu0 * op.ih2[2]);
}

// ---------------------------------------------------------------- dense
// FP32: acc -= the block's three products, block by block.  FP64, whose pipe
// issues one instruction per 64 cycles: the blocks' products accumulate with
// fused multiply-adds in four parts, blocks 7 d .. 7 d + 6, which dense.cu
// gives to the four schedulers of an SM; acc -= each part's sum in turn.
constexpr int kPartBlocks = 7;

template <typename T, bool WITH_CENTRE, bool COH = false>
__device__ inline void dense_row(const DenseOp<T> &op, const Geom &g, const NbrOffsets &t, int p,
                                 const T *__restrict__ x, T *acc) {
    const T *row = op.coef + coef_at(p);
    T part[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int b = 0; b < 27; b++) {
        int s = t.ox[bdx(b) + 1] + t.oy[bdy(b) + 1] + t.oz[bdz(b) + 1];
        // outside a non-periodic grid: coefficients are zero there
        if (!(b == 13 && !WITH_CENTRE) && s >= 0) {
            T v[3], a[9];
            load3<T, COH>(x, g.npad, s, v);
#pragma unroll
            for (int e = 0; e < 9; e++) a[e] = __ldg(row + (9 * b + e) * kCoefGroup);
            if (sizeof(T) == 4) {
                matvec_sub(a, v, acc);
            } else {
#pragma unroll
                for (int e = 0; e < 9; e++) part[e / 3] = fma_rn(a[e], v[e % 3], part[e / 3]);
            }
        }
        if (sizeof(T) == 8 && (b % kPartBlocks == kPartBlocks - 1 || b == 26)) {
#pragma unroll
            for (int r = 0; r < 3; r++) {
                acc[r] -= part[r];
                part[r] = T(0);
            }
        }
    }
}

// ---------------------------------------------------------------- plane
// Structural non-zeros of the coarse elasticity operators: entry (r,c) of the
// block at offset d can be non-zero only if r == c or d_r, d_c are both non-zero.
__host__ __device__ constexpr bool coarse_entry(int b, int e) {
    return (e / 3 == e % 3) ||
           ((e / 3 == 0 ? bdx(b) : e / 3 == 1 ? bdy(b) : bdz(b)) != 0 &&
            (e % 3 == 0 ? bdx(b) : e % 3 == 1 ? bdy(b) : bdz(b)) != 0);
}

// acc -= sum_b A_b x_b with entry e of block b read from cf[(9b + e) * stride]
// (shared memory with stride 1, or plane storage in global memory).
template <typename T, bool SPARSE, bool WITH_CENTRE, bool COH = false>
__device__ inline void plane_row_coef(const T *cf, int stride, const Geom &g, const NbrOffsets &t,
                                      const T *__restrict__ x, T *acc) {
    if constexpr (sizeof(T) == 8) {
        // FP64: arithmetic bound; load each neighbour right before its block
#pragma unroll
        for (int b = 0; b < 27; b++) {
            if (b == 13 && !WITH_CENTRE) continue;
            int s = t.ox[bdx(b) + 1] + t.oy[bdy(b) + 1] + t.oz[bdz(b) + 1];
            if (s < 0) continue;
            T v[3];
            load3<T, COH>(x, g.npad, s, v);
#pragma unroll
            for (int e = 0; e < 9; e++)
                if (!SPARSE || coarse_entry(b, e)) acc[e / 3] -= cf[(9 * b + e) * stride] * v[e % 3];
        }
    } else {
        // FP32: all neighbour loads are issued before the arithmetic so that
        // they are in flight together (one memory latency per node, not one per block)
        T v[27][3];
#pragma unroll
        for (int b = 0; b < 27; b++) {
            if (b == 13 && !WITH_CENTRE) continue;
            int s = t.ox[bdx(b) + 1] + t.oy[bdy(b) + 1] + t.oz[bdz(b) + 1];
            const int sc = s < 0 ? 0 : s;
            load3<T, COH>(x, g.npad, sc, v[b]);
            if (s < 0) v[b][0] = v[b][1] = v[b][2] = T(0);
        }
#pragma unroll
        for (int b = 0; b < 27; b++) {
            if (b == 13 && !WITH_CENTRE) continue;
#pragma unroll
            for (int e = 0; e < 9; e++)
                if (!SPARSE || coarse_entry(b, e)) acc[e / 3] -= cf[(9 * b + e) * stride] * v[b][e % 3];
        }
    }
}

}  // namespace stzmg
