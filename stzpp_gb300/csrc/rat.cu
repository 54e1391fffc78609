// Galerkin (RAT) coarse operators and their box bounds.
//
// Reference: region::fill_rat_bounds / compute_rats (mg_3d_template/
// region.cc:1848-1966) with rat_bound_*/rat_fill_* (2275-2466), A_red
// (2485-2538), A_add (2545-2578), grid_map/igrid_map (2587-2647) and the
// driver multigrid::compute_rats (multigrid.cc:330-344).
//
// The reference builds A_c = (1/8) P^T A P by scattering, for every fine row
// f, the row of A P (A_red) into the rows of f's coarse parents.  Here one
// thread owns coarse entries (coarse node I, offset J - I) and gathers
//     A_c[I,J] = sum_{f child of I} sum_{g child of J, g in box(f)}
//                (1/8 A[f,g]) w_P(g,J) w_P(f,I).
// All weights are powers of two, so every term is bit-identical to the
// reference's, and one fused multiply-add by the product of the weights adds
// it with the rounding of the addition alone; only the order of the additions
// differs.  (The FP64 pipe bounds the large levels: three products and a sum
// per term, and a whole Lame row per fine child, took 7.7 ms for the 32x32x33
// level below a 64x64x65 Lame level; now 1.3 ms.)  Entries are kept in
// the unwrapped offset convention of the reference's boxes (on a periodic
// dimension of size 2 or 1, offsets -1 and +1 are separate entries).
#include "launch.h"
#include "ops.cuh"

namespace stzmg {

constexpr int kRB = 128;

// Children of coarse index I along one dimension: fine range [lo, hi) and
// the fine index that coincides with I (igrid_map without the cropping);
// returns false when I is outside a non-periodic grid.
__device__ inline bool children(int I, int mf, int mc, int prd, int &lo, int &hi, int &c) {
    if (!prd && (I < 0 || I >= mc)) return false;
    int j = 2 * I;
    if (prd) { lo = j - 1; hi = j + 2; c = j; return true; }
    if (mf & 1) { lo = j == 0 ? 0 : j - 1; hi = j == mf - 1 ? mf : j + 2; c = j; }
    else if (j == mf) { lo = mf - 1; hi = mf; c = mf - 1; }
    else { lo = j == 0 ? 0 : j - 1; hi = j == mf - 2 ? mf - 1 : j + 2; c = j; }
    return true;
}

__device__ inline int wrapd(int a, int len) {
    a %= len;
    return a < 0 ? a + len : a;
}

// The same for a child of a coarse node: at most one period out.
__device__ inline int wrap_child(int a, int len) { return a < 0 ? a + len : a >= len ? a - len : a; }

// Block (d) of fine row f for the three operator kinds.
template <int KIND>
__device__ inline void fine_block(const LevelOp<double> &op, const Geom &g, int fs, bool interior,
                                  const double *mu_nb, const double *lam_nb, const LameRow<double> &L, int b,
                                  double *a) {
#pragma unroll
    for (int e = 0; e < 9; e++) a[e] = 0.0;
    if (KIND == OP_CONST) {
        const double *src = interior ? op.cop.a[b] : op.cop.fix;
        for (int e = 0; e < 9; e++) a[e] = src[e];
    } else if (KIND == OP_LAME) {
        if (!interior) {
            double f = lame_fix(op.lop, fs);
            a[0] = a[4] = a[8] = f;
            return;
        }
        int dx = bdx(b), dy = bdy(b), dz = bdz(b), nz = nnz_axes(b);
        if (nz == 0) {
            a[0] = L.centre[0]; a[4] = L.centre[1]; a[8] = L.centre[2];
        } else if (nz == 1) {
            int f = dx ? (dx > 0 ? 1 : 0) : dy ? (dy > 0 ? 3 : 2) : (dz > 0 ? 5 : 4);
            a[0] = L.face[f][0]; a[4] = L.face[f][1]; a[8] = L.face[f][2];
        } else if (nz == 2) {
            int d[3] = {dx, dy, dz};
            int r = dz == 0 ? 0 : (dy == 0 ? 0 : 1), c = dz == 0 ? 1 : 2;
            int sr = d[r], sc = d[c];
            const double ie = op.lop.iedge[r + c - 1], sgn = (double)(sr * sc);
            const double lam_r = lam_nb[2 * r + (sr > 0)], mu_r = mu_nb[2 * r + (sr > 0)];
            const double lam_c = lam_nb[2 * c + (sc > 0)], mu_c = mu_nb[2 * c + (sc > 0)];
            a[3 * r + c] = -op.lop.dt * ((sgn * (lam_r + mu_c)) * ie);
            a[3 * c + r] = -op.lop.dt * ((sgn * (lam_c + mu_r)) * ie);
        }
    } else if (KIND == OP_PLANE) {
        const int k = fs;   // callers pass the plane index for plane operators
        for (int e = 0; e < 9; e++) a[e] = op.pop.coef[(9 * b + e) * op.pop.O + k];
    } else {
        for (int e = 0; e < 9; e++) a[e] = op.dop.coef[coef_at(fs) + (9 * b + e) * kCoefGroup];
    }
}

// One dimension of a coarse entry: the children f of I, the children g of the
// target, which of f's neighbours f - 1, f, f + 1 are among them and with
// what weight (0 for those that are not).
struct RatDim {
    int slo, shi, sc, tlo, thi, tc;
    __device__ __forceinline__ bool set(int I, int off, int mf, int mc, int prd) {
        children(I, mf, mc, prd, slo, shi, sc);
        return children(I + off, mf, mc, prd, tlo, thi, tc);
    }
    // the weights' exponents: 2^-own, 2^-target, or kNone
    __device__ __forceinline__ int own(int f) const { return f != sc; }
    __device__ __forceinline__ int target(int g) const { return g < tlo || g >= thi ? kNone : g != tc; }
    static constexpr int kNone = 64;
};

// 2^-n, an integer shift: the FP64 pipe is for the sums.
__device__ __forceinline__ double weight(int n) { return __longlong_as_double((long long)(1023 - n) << 52); }

// Thread: coarse node p (OUT_PLANE: plane p), offset blockIdx.y, row
// blockIdx.z of the block.  The nine blocks of one z offset are loaded
// together: the small levels are bound by the latency of these loads.
template <int KIND, bool OUT_PLANE>
__global__ void __launch_bounds__(kRB) rat_kernel(Geom gf, Geom gc, const __grid_constant__ LevelOp<double> op,
                                                  double *__restrict__ coef_c) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, off = blockIdx.y, row = blockIdx.z;
    int I, J, K;
    if (OUT_PLANE) {
        // one coarse node per plane: the column i = j = 0
        if (p >= gc.o) return;
        I = 0; J = 0; K = p;
    } else if (p >= gc.npad || !slot_node(gc, p, I, J, K)) {
        return;
    }
    RatDim x, y, z;
    if (!(x.set(I, bdx(off), gf.m, gc.m, gf.xp) & y.set(J, bdy(off), gf.n, gc.n, gf.yp) &
          z.set(K, bdz(off), gf.o, gc.o, gf.zp)))
        return;   // entry stays zero
    double acc[3] = {0.0, 0.0, 0.0};
    for (int fz = z.slo; fz < z.shi; fz++) {
        const int fzw = wrap_child(fz, gf.o);
        for (int fy = y.slo; fy < y.shi; fy++) {
            const int fyw = wrap_child(fy, gf.n);
            for (int fx = x.slo; fx < x.shi; fx++) {
                const int wf = 3 + z.own(fz) + y.own(fy) + x.own(fx);   // the 1/8 too
                const int fxw = wrap_child(fx, gf.m);
                const double *src;
                int step = 1;
                bool interior = true;
                if (KIND == OP_CONST) {
                    interior = is_interior(gf, fxw, fyw, fzw);
                    src = &op.cop.a[0][0];
                } else if (KIND == OP_PLANE) {
                    src = op.pop.coef + fzw;
                    step = op.pop.O;
                } else {
                    src = op.dop.coef + coef_at(slot(gf, fxw, fyw, fzw));
                    step = kCoefGroup;
                }
                if (!interior) {   // a box of the centre alone
                    const int n = wf + z.target(fz) + y.target(fy) + x.target(fx);
                    if (n < RatDim::kNone)
#pragma unroll
                        for (int e = 0; e < 3; e++) acc[e] = fma_rn(op.cop.fix[3 * row + e], weight(n), acc[e]);
                    continue;
                }
                for (int dz = max(-1, z.tlo - fz); dz <= min(1, z.thi - 1 - fz); dz++) {
                    const int wz = wf + z.target(fz + dz);
                    double a[9][3];
                    int n[9];
#pragma unroll
                    for (int d = 0; d < 9; d++) {
                        n[d] = wz + y.target(fy + d / 3 - 1) + x.target(fx + d % 3 - 1);
                        const double *c = src + (size_t)(9 * (9 * (dz + 1) + d) + 3 * row) * step;
#pragma unroll
                        for (int e = 0; e < 3; e++) a[d][e] = n[d] < RatDim::kNone ? c[(size_t)e * step] : 0.0;
                    }
#pragma unroll
                    for (int d = 0; d < 9; d++)
                        if (n[d] < RatDim::kNone)
#pragma unroll
                            for (int e = 0; e < 3; e++) acc[e] = fma_rn(a[d][e], weight(n[d]), acc[e]);
                }
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const int entry = 9 * off + 3 * row + e;
        coef_c[OUT_PLANE ? (size_t)entry * gc.o + p : coef_at(p) + entry * kCoefGroup] = acc[e];
    }
}

// The same below a Lame level (thread: coarse node p, offset blockIdx.y): of
// each fine row only the blocks that reach the target, and only their non-zero
// entries, with lame_faces' and lame_row's arithmetic.
__global__ void __launch_bounds__(kRB) rat_lame_kernel(Geom gf, Geom gc, LameOp<double> op,
                                                       double *__restrict__ coef_c) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, off = blockIdx.y;
    int I, J, K;
    if (p >= gc.npad || !slot_node(gc, p, I, J, K)) return;
    RatDim x, y, z;
    if (!(x.set(I, bdx(off), gf.m, gc.m, gf.xp) & y.set(J, bdy(off), gf.n, gc.n, gf.yp) &
          z.set(K, bdz(off), gf.o, gc.o, gf.zp)))
        return;   // entry stays zero
    double acc[9];
#pragma unroll
    for (int e = 0; e < 9; e++) acc[e] = 0.0;
    for (int fz = z.slo; fz < z.shi; fz++) {
        const int fzw = wrap_child(fz, gf.o);
        for (int fy = y.slo; fy < y.shi; fy++) {
            const int fyw = wrap_child(fy, gf.n);
#pragma unroll 1
            for (int fx = x.slo; fx < x.shi; fx++) {
                const int wf = 3 + z.own(fz) + y.own(fy) + x.own(fx);   // the 1/8 too
                const int fxw = wrap_child(fx, gf.m), fs = slot(gf, fxw, fyw, fzw);
                if (!is_interior(gf, fxw, fyw, fzw)) {   // a box of the centre alone
                    const int n = wf + z.target(fz) + y.target(fy) + x.target(fx);
                    if (n < RatDim::kNone) {
                        const double f = lame_fix(op, fs);
#pragma unroll
                        for (int r = 0; r < 3; r++) acc[4 * r] = fma_rn(f, weight(n), acc[4 * r]);
                    }
                    continue;
                }
                const NbrOffsets t = nbr_offsets_sub(gf, fxw >> 1, fyw >> 1, fzw >> 1, fxw & 1, fyw & 1, fzw & 1);
                double mu[6], lam[6];
                const double mu0 = op.mu[fs], lam0 = op.lam[fs];
#pragma unroll
                for (int f = 0; f < 6; f++) {
                    const int s = f & 1 ? 2 : 0, ax = f / 2;
                    const int nb = t.ox[ax == 0 ? s : 1] + t.oy[ax == 1 ? s : 1] + t.oz[ax == 2 ? s : 1];
                    mu[f] = op.mu[nb];
                    lam[f] = op.lam[nb];
                }
                int wx[3], wy[3], wz[3];
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    wx[d] = wf + x.target(fx + d - 1);
                    wy[d] = y.target(fy + d - 1);
                    wz[d] = z.target(fz + d - 1);
                }
                // face f's diagonal entry of component c, without the factor -dt
                auto face = [&](int f, int c) {
                    const int ax = f / 2;
                    const double mu_f = 0.5 * (mu0 + mu[f]), lam_f = 0.5 * (lam0 + lam[f]);
                    return (c == ax ? (lam_f + 2.0 * mu_f) : mu_f) * op.ih2[ax];
                };
#pragma unroll
                for (int b = 0; b < 27; b++) {
                    const int dx = bdx(b), dy = bdy(b), dz = bdz(b), nz = nnz_axes(b);
                    if (nz == 3) continue;
                    const int n = wx[dx + 1] + wy[dy + 1] + wz[dz + 1];
                    if (n >= RatDim::kNone) continue;
                    const double w = weight(n);
                    if (nz == 0) {
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            double cen = 0.0;
#pragma unroll
                            for (int f = 0; f < 6; f++) cen -= face(f, c);
                            acc[4 * c] = fma_rn(-op.dt * cen, w, acc[4 * c]);
                        }
                    } else if (nz == 1) {
                        const int f = dx ? (dx > 0 ? 1 : 0) : dy ? (dy > 0 ? 3 : 2) : (dz > 0 ? 5 : 4);
#pragma unroll
                        for (int c = 0; c < 3; c++) acc[4 * c] = fma_rn(-op.dt * face(f, c), w, acc[4 * c]);
                    } else {
                        const int d[3] = {dx, dy, dz};
                        const int r = dz == 0 ? 0 : (dy == 0 ? 0 : 1), c = dz == 0 ? 1 : 2;
                        const double ie = op.iedge[r + c - 1], sgn = d[r] * d[c];
                        const int nr = 2 * r + (d[r] > 0), nc = 2 * c + (d[c] > 0);
                        acc[3 * r + c] = fma_rn(-op.dt * ((sgn * (lam[nr] + mu[nc])) * ie), w, acc[3 * r + c]);
                        acc[3 * c + r] = fma_rn(-op.dt * ((sgn * (lam[nc] + mu[nr])) * ie), w, acc[3 * c + r]);
                    }
                }
            }
        }
    }
    double *out = coef_c + coef_at(p) + 9 * off * kCoefGroup;
#pragma unroll
    for (int e = 0; e < 9; e++) out[e * kCoefGroup] = acc[e];
}

// How far a plane-invariant operator is from the structure of coarse_entry:
// out[0] the largest magnitude outside it, out[1] the largest ratio of that to
// a plane's largest entry (both zero before), and the planes with nothing
// outside it.  A block per 32 planes.
__global__ void __launch_bounds__(256) plane_structure_kernel(int O, const double *__restrict__ coef, double *out,
                                                              int *__restrict__ structured) {
    __shared__ unsigned long long all[8][32], far[8][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
    unsigned long long a = 0, f = 0;   // bits of magnitudes order as the values
    if (k < O)
#pragma unroll 8
        for (int v = wid; v < 243; v += 8) {
            const unsigned long long m = __double_as_longlong(coef[(size_t)v * O + k]) & 0x7fffffffffffffffull;
            a = max(a, m);
            if (!coarse_entry(v / 9, v % 9)) f = max(f, m);
        }
    all[wid][lane] = a;
    far[wid][lane] = f;
    __syncthreads();
    if (wid == 0 && k < O) {
        for (int w = 1; w < 8; w++) a = max(a, all[w][lane]), f = max(f, far[w][lane]);
        unsigned long long *o = reinterpret_cast<unsigned long long *>(out);
        structured[k] = f == 0;
        if (f) {
            atomicMax(o, f);
            atomicMax(o + 1, (unsigned long long)__double_as_longlong(__longlong_as_double(f) / __longlong_as_double(a)));
        }
    }
}

template <typename T>
__global__ void plane_dinv_kernel(int O, const T *__restrict__ coef, T *__restrict__ dinv, int *bad) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= O) return;
    T a[9], inv[9];
    for (int e = 0; e < 9; e++) a[e] = coef[(9 * 13 + e) * O + k];
    if (!inverse3(a, inv)) atomicExch(bad, 1);
    for (int e = 0; e < 9; e++) dinv[e * O + k] = inv[e];
}

template <typename T>
__global__ void dinv_kernel(Geom g, const T *__restrict__ coef, T *__restrict__ dinv, int *bad) {
    int p = blockIdx.x * blockDim.x + threadIdx.x, i, j, k;
    if (p >= g.npad) return;
    T a[9], inv[9], *out = dinv + dinv_at(p);
    if (!slot_node(g, p, i, j, k)) {
        for (int e = 0; e < 9; e++) out[e * kCoefGroup] = T(0);
        return;
    }
    for (int e = 0; e < 9; e++) a[e] = coef[coef_at(p) + (9 * 13 + e) * kCoefGroup];
    bool ok = inverse3(a, inv);
    if (!ok) atomicExch(bad, 1);
    for (int e = 0; e < 9; e++) out[e * kCoefGroup] = inv[e];
}

// grid_map (region.cc:2587-2604), with the reference's range checks
// reported through *bad.
__device__ inline void grid_map(int &lo, int &hi, int ma, int prd, int *bad) {
    if (prd) {
        if (lo < -ma || lo > ma - 1 || hi < 1 || hi > 2 * ma) atomicExch(bad, 2);
        lo = lo < 0 ? (lo - (ma & 1 ? 2 : 1)) / 2 : lo >> 1;
        hi = (hi + ((ma & 1) && hi > ma ? 1 : 2)) >> 1;
    } else {
        if (lo < 0 || lo > ma - 1 || hi < 1 || hi > ma) atomicExch(bad, 2);
        lo = (!(ma & 1) && lo == ma - 1 ? lo + 1 : lo) >> 1;
        hi = (hi + 2) >> 1;
    }
}

__global__ void top_bounds_kernel(Geom g, int *S) {
    int p = blockIdx.x * blockDim.x + threadIdx.x, i, j, k;
    if (p >= g.npad) return;
    bool used = slot_node(g, p, i, j, k);
    bool in = used && is_interior(g, i, j, k);
    for (int d = 0; d < 3; d++) {
        S[(size_t)(2 * d) * g.npad + p] = in ? -1 : 0;
        S[(size_t)(2 * d + 1) * g.npad + p] = in ? 2 : 1;
    }
}

// Coarse bounds: union over the children f of I of grid_map(box(f)) - I
// (fill_rat_bounds, region.cc:1848-1905).  Bounds are stored SoA, 6 x npad.
__global__ void rat_bounds_kernel(Geom gf, const int *__restrict__ Sf, Geom gc, int *__restrict__ Sc, int *bad) {
    int p = blockIdx.x * blockDim.x + threadIdx.x, I, J, K;
    if (p >= gc.npad) return;
    int box[6] = {0, 1, 0, 1, 0, 1};
    if (slot_node(gc, p, I, J, K)) {
        int lo[3], hi[3], c[3];
        children(I, gf.m, gc.m, gf.xp, lo[0], hi[0], c[0]);
        children(J, gf.n, gc.n, gf.yp, lo[1], hi[1], c[1]);
        children(K, gf.o, gc.o, gf.zp, lo[2], hi[2], c[2]);
        const int C[3] = {I, J, K};
        const int dims[3] = {gf.m, gf.n, gf.o}, prd[3] = {gf.xp, gf.yp, gf.zp};
        for (int fz = lo[2]; fz < hi[2]; fz++)
            for (int fy = lo[1]; fy < hi[1]; fy++)
                for (int fx = lo[0]; fx < hi[0]; fx++) {
                    const int f[3] = {fx, fy, fz};
                    const int fs = slot(gf, wrapd(fx, gf.m), wrapd(fy, gf.n), wrapd(fz, gf.o));
                    for (int d = 0; d < 3; d++) {
                        int l = f[d] + Sf[(size_t)(2 * d) * gf.npad + fs];
                        int h = f[d] + Sf[(size_t)(2 * d + 1) * gf.npad + fs];
                        // the reference maps boxes in the parent's global frame of the
                        // unwrapped fine index; wrapping f by whole periods shifts the
                        // coarse box by whole coarse periods, so map the wrapped box and
                        // shift back
                        int shift = 0;
                        if (prd[d]) {
                            int fw = wrapd(f[d], dims[d]);
                            shift = f[d] - fw;   // multiple of the fine period
                            l -= shift; h -= shift;
                        }
                        grid_map(l, h, dims[d], prd[d], bad);
                        if (prd[d] && shift) {
                            const int cper = d == 0 ? gc.m : d == 1 ? gc.n : gc.o;
                            l += (shift / dims[d]) * cper;
                            h += (shift / dims[d]) * cper;
                        }
                        if (l - C[d] < box[2 * d]) box[2 * d] = l - C[d];
                        if (h - C[d] > box[2 * d + 1]) box[2 * d + 1] = h - C[d];
                    }
                }
    }
    for (int e = 0; e < 6; e++) Sc[(size_t)e * gc.npad + p] = box[e];
}

__global__ void bounds_cb_to_nat_kernel(Geom g, const int *__restrict__ S, int *__restrict__ nat) {
    long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long npts = (long)g.m * g.n * g.o;
    if (t >= npts) return;
    int i = t % g.m, j = (t / g.m) % g.n, k = t / ((long)g.m * g.n);
    int s = slot(g, i, j, k);
    for (int e = 0; e < 6; e++) nat[6 * t + e] = S[(size_t)e * g.npad + s];
}

// Dense 27-block form of a top-level operator (for export and checks).
template <int KIND>
__global__ void expand_dense_kernel(Geom g, const __grid_constant__ LevelOp<double> op, double *__restrict__ coef) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
    int i, j, k;
    if (p >= g.npad || !slot_node(g, p, i, j, k)) return;
    const bool interior = (KIND == OP_DENSE || KIND == OP_PLANE) ? true : is_interior(g, i, j, k);
    double a[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (interior || b == 13) {
        LameRow<double> L;
        double mu_nb[6], lam_nb[6];
        if (KIND == OP_LAME && interior) {
            NbrOffsets nb = nbr_offsets(g, i, j, k);
            lame_faces(op.lop, g, nb, p, L, mu_nb, lam_nb);
        }
        fine_block<KIND>(op, g, KIND == OP_PLANE ? k : p, interior, mu_nb, lam_nb, L, b, a);
    }
    for (int e = 0; e < 9; e++) coef[coef_at(p) + (9 * b + e) * kCoefGroup] = a[e];
}

void launch_expand_dense(const LevelOp<double> &op, const Geom &g, double *coef, cudaStream_t st) {
    cudaMemsetAsync(coef, 0, sizeof(double) * coef_len(g.npad), st);
    dim3 grid((g.npad + kRB - 1) / kRB, 27);
    switch (op.kind) {
        case OP_CONST: expand_dense_kernel<OP_CONST><<<grid, kRB, 0, st>>>(g, op, coef); break;
        case OP_LAME: expand_dense_kernel<OP_LAME><<<grid, kRB, 0, st>>>(g, op, coef); break;
        case OP_PLANE: expand_dense_kernel<OP_PLANE><<<grid, kRB, 0, st>>>(g, op, coef); break;
        default: expand_dense_kernel<OP_DENSE><<<grid, kRB, 0, st>>>(g, op, coef); break;
    }
}

void launch_rat(const LevelOp<double> &fine, const Geom &gf, const Geom &gc, double *coef_c, bool plane,
                cudaStream_t st) {
    if (plane) {
        cudaMemsetAsync(coef_c, 0, sizeof(double) * 243 * (size_t)gc.o, st);
        dim3 grid((gc.o + 31) / 32, 27, 3);   // few planes: a warp a block
        if (fine.kind == OP_CONST) rat_kernel<OP_CONST, true><<<grid, 32, 0, st>>>(gf, gc, fine, coef_c);
        else rat_kernel<OP_PLANE, true><<<grid, 32, 0, st>>>(gf, gc, fine, coef_c);
        return;
    }
    cudaMemsetAsync(coef_c, 0, sizeof(double) * coef_len(gc.npad), st);
    dim3 grid((gc.npad + kRB - 1) / kRB, 27, 3);
    switch (fine.kind) {
        case OP_CONST: rat_kernel<OP_CONST, false><<<grid, kRB, 0, st>>>(gf, gc, fine, coef_c); break;
        case OP_LAME: grid.z = 1; rat_lame_kernel<<<grid, kRB, 0, st>>>(gf, gc, fine.lop, coef_c); break;
        case OP_PLANE: rat_kernel<OP_PLANE, false><<<grid, kRB, 0, st>>>(gf, gc, fine, coef_c); break;
        default: rat_kernel<OP_DENSE, false><<<grid, kRB, 0, st>>>(gf, gc, fine, coef_c); break;
    }
}

void launch_plane_structure(int O, const double *coef, double *out, int *structured, cudaStream_t st) {
    cudaMemsetAsync(out, 0, 2 * sizeof(double), st);
    plane_structure_kernel<<<(O + 31) / 32, 256, 0, st>>>(O, coef, out, structured);
}

template <typename T>
void launch_plane_dinv(int O, const T *coef, T *dinv, int *bad, cudaStream_t st) {
    plane_dinv_kernel<T><<<(O + 127) / 128, 128, 0, st>>>(O, coef, dinv, bad);
}
template void launch_plane_dinv<float>(int, const float *, float *, int *, cudaStream_t);
template void launch_plane_dinv<double>(int, const double *, double *, int *, cudaStream_t);

template <typename T>
void launch_dense_dinv(const Geom &g, const T *coef, T *dinv, int *bad, cudaStream_t st) {
    dinv_kernel<T><<<(g.npad + 255) / 256, 256, 0, st>>>(g, coef, dinv, bad);
}
template void launch_dense_dinv<float>(const Geom &, const float *, float *, int *, cudaStream_t);
template void launch_dense_dinv<double>(const Geom &, const double *, double *, int *, cudaStream_t);

void launch_top_bounds(const Geom &g, int *S, cudaStream_t st) {
    top_bounds_kernel<<<(g.npad + 255) / 256, 256, 0, st>>>(g, S);
}
void launch_rat_bounds(const Geom &gf, const int *fine_S, const Geom &gc, int *S_c, int *bad, cudaStream_t st) {
    rat_bounds_kernel<<<(gc.npad + 255) / 256, 256, 0, st>>>(gf, fine_S, gc, S_c, bad);
}
void launch_bounds_cb_to_nat(const Geom &g, const int *S, int *nat, cudaStream_t st) {
    bounds_cb_to_nat_kernel<<<(int)(((long)g.m * g.n * g.o + 255) / 256), 256, 0, st>>>(g, S, nat);
}

}  // namespace stzmg
