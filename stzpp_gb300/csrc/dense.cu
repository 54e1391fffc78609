// Gauss-Seidel sweep and residual of the levels whose rows are stored per node
// (OP_DENSE: Galerkin levels of variable coefficients, per-node stencils).
//
// A row is 26 neighbour blocks of 9 coefficients, 1 or 2 KB per node.  Large
// levels are bound by those bytes (FP32) or by the FP64 pipe, small ones, with
// few nodes per colour, by latency.  A thread per node does badly at all three:
// so the blocks of a row are spread over the warps of a CTA, lanes along the
// nodes (coalesced), and the parts are summed through shared memory in the
// order of dense_row (ops.cuh), which the colour launches use: the results are
// equal bit for bit.
//
//  * FP32: 32 nodes at a time, 13 warps with two blocks each; a 14th warp sums
//    the 26 products of a node and applies the inverse centre block.
//  * FP64: an SM scheduler issues an FP64 instruction every 64 cycles, whether
//    its warp has one active lane or 32 (measured), so the four schedulers
//    have to be loaded alike and the lanes filled: a team of four warps takes
//    10 nodes, a lane per node and row, a warp per part of dense_row (7, 6, 7
//    and 6 blocks), and the warps take turns at the sums.
//
// The sweep is two launches, the even planes and then the odd ones (colours
// 0-3 and 4-7; region::gauss_seidel, mg_3d_template/region.cc:1557-1762, in
// the 8-colour order).  A cluster of up to 8 CTAs runs the four colours of one
// plane, with a cluster barrier between two colours.  What does not depend on
// the colour before is loaded ahead of the barrier: the coefficients, and x of
// the planes above and below.
//
// On levels too small to fill the SMs a colour's chain is left: 21 FP64
// multiply-adds in a row, the sum, the store, the barrier and the loads, 3.4 us
// (all sweeps of 7x6x5 in one launch: 27.5 -> 26.9 us each, not kept).
//
// One sweep on GB300, before (one block a plane on planes of up to 64x64,
// else eight colour launches, a thread a node) and now:
//   64x64x65  FP32  310 -> 69 us     16x16x17  FP32   54 -> 14 us
//   49x41x33  FP64  328 -> 148 us    32x48x26  FP64  245 -> 66 us
//   7x6x5     FP64  118 -> 28 us
// and the residual of 49x41x33 in FP64 72 -> 59 us, of 16x16x17 in FP32 23 -> 3 us.
#include <algorithm>

#include "launch.h"
#include "ops.cuh"

namespace stzmg {

namespace {

// Entry d + 1 of a dimension's neighbour offsets, d known at run time.
__device__ __forceinline__ int pick(const int (&o)[3], int d) { return d == 0 ? o[1] : d < 0 ? o[0] : o[2]; }

// Offsets of the neighbours in the plane, of a node of colour q.
__device__ __forceinline__ void plane_offsets(const Geom &g, int I, int J, int q, NbrOffsets &t) {
    dim_offsets(I, q & 1, g.m, g.M2, g.xp, g.S, 1, t.ox);
    dim_offsets(J, (q >> 1) & 1, g.n, g.N2, g.yp, 2 * g.S, g.M2, t.oy);
}
__device__ __forceinline__ void z_offsets(const Geom &g, int K, int q, NbrOffsets &t) {
    dim_offsets(K, q >> 2, g.o, g.O2, g.zp, 4 * g.S, g.M2 * g.N2, t.oz);
}

// Sub-grid coordinates of a lane's node that moves on by a fixed number of
// slots per item (no division per item).
struct Walk {
    int t, I, J, K;
    int dt, dI, dJ, dK;
    __device__ __forceinline__ Walk(const Geom &g, int t0, int step) : t(t0), dt(step) {
        I = t0 % g.M2, J = t0 / g.M2 % g.N2, K = t0 / (g.M2 * g.N2);
        dI = step % g.M2, dJ = step / g.M2 % g.N2, dK = step / (g.M2 * g.N2);
    }
    __device__ __forceinline__ void next(const Geom &g) {
        t += dt;
        I += dI, J += dJ, K += dK;
        if (I >= g.M2) I -= g.M2, J++;
        if (J >= g.N2) J -= g.N2, K++;
    }
};

// The end of a colour.  A thread arrives when its own values are stored and
// loads what the next colour needs and does not depend on this one before it
// waits: a release waits for every load issued before it too.
__device__ __forceinline__ void colour_arrive(int cl) {
    if (cl > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void colour_wait(int cl) {
    if (cl > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
}

// ---------------------------------------------------------------- FP32
constexpr int kDotWarps = 13;                        // two blocks each: b and 26 - b
constexpr int kThreads32 = 32 * (kDotWarps + 1);     // the last warp sums

using DotTable = float[26][3][32];

// What a dot warp holds of its blocks w and 26 - w for one node per lane
// (coefficients of slot 0 for a lane without a node).
struct BlockPair {
    float a[2][9], v[2][3];
    int s[2];   // the neighbours' slots, negative outside the grid

    __device__ __forceinline__ void load(const DenseOp<float> &op, int w, int p, const NbrOffsets &t, bool valid) {
        const int dx = bdx(w), dy = bdy(w), dz = bdz(w);
        s[0] = valid ? pick(t.ox, dx) + pick(t.oy, dy) + pick(t.oz, dz) : -1;
        s[1] = valid ? pick(t.ox, -dx) + pick(t.oy, -dy) + pick(t.oz, -dz) : -1;
        const float *row = op.coef + coef_at(p) + 9 * w * kCoefGroup, *row2 = row + 9 * (26 - 2 * w) * kCoefGroup;
#pragma unroll
        for (int e = 0; e < 9; e++) {
            a[0][e] = __ldg(row + e * kCoefGroup);
            a[1][e] = __ldg(row2 + e * kCoefGroup);
        }
    }
    template <bool COH>
    __device__ __forceinline__ void load_x(const float *x, int npad) {
#pragma unroll
        for (int u = 0; u < 2; u++) load3<float, COH>(x, npad, max(s[u], 0), v[u]);
    }
    // the products, into the CTA's table (0 for a neighbour outside the grid)
    __device__ __forceinline__ void dots(int w, int lane, DotTable &out) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
            float(*o)[32] = out[u ? 25 - w : w];
            if (s[u] < 0) v[u][0] = v[u][1] = v[u][2] = 0.0f;
#pragma unroll
            for (int r = 0; r < 3; r++)
                o[r][lane] = dot3(a[u][3 * r], v[u][0], a[u][3 * r + 1], v[u][1], a[u][3 * r + 2], v[u][2]);
        }
    }
};

// Colours 4c .. 4c+3 of every plane of parity c, `cl` CTAs (one cluster) per
// plane; x is updated in place.
__global__ void __launch_bounds__(kThreads32, 2)
    gs_dense32_kernel(Geom g, int c, int cl, DenseOp<float> op, const float *r, float *x) {
    __shared__ DotTable dots[2];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int rank = blockIdx.x % cl, K = blockIdx.x / cl;
    const int plane = g.M2 * g.N2, per = ((plane + 31) / 32 + cl - 1) / cl;
    const bool sums = wid == kDotWarps;
    const bool inplane = wid >= 9;   // blocks 9 .. 12 and 14 .. 17; the other warps read the planes above and below
    const size_t np = (size_t)g.npad;
    const Walk start(g, 32 * rank + lane, 32 * cl);
    Walk at = start;
    BlockPair row;
    float acc[3], inv[9];
    int p = -1;   // the summing warp's node
    NbrOffsets nb;
    z_offsets(g, K, 4 * c, nb);
    // 32 nodes of colour q of the plane: all that may be read before the colour begins (first) or in it
    auto load = [&](int q, bool first, bool chained = false) {
        const bool valid = at.t < plane && 2 * at.I + (q & 1) < g.m && 2 * at.J + ((q >> 1) & 1) < g.n;
        const int s = valid ? q * g.S + K * plane + at.t : 0;
        if (!sums) {
            plane_offsets(g, at.I, at.J, q, nb);
            row.load(op, wid, s, nb, valid);
            if (chained) chain_wait();
            if (!inplane || !first) row.load_x<true>(x, g.npad);
        } else {
            p = valid ? s : -1;
#pragma unroll
            for (int e = 0; e < 9; e++) inv[e] = __ldg(op.dinv + dinv_at(s) + e * kCoefGroup);
            if (chained) chain_wait();
            load3(r, g.npad, s, acc);
        }
    };
    int buf = 0;
    load(4 * c, true, true);
#pragma unroll 1
    for (int q = 4 * c; q < 4 * c + 4; q++) {
#pragma unroll 1
        for (int n = 0; n < per; n++, buf ^= 1) {
            const bool last = n + 1 == per;
            if (last) at = start;
            else at.next(g);
            if (last && q == 4 * c + 3) chain_next();
            if (!sums) {
                if (inplane && n == 0) row.load_x<true>(x, g.npad);
                row.dots(wid, lane, dots[buf]);
                if (!last) load(q, false);
            }
            __syncthreads();   // the table is complete; the other one has been read
            if (sums) {
                if (p >= 0) {
#pragma unroll
                    for (int b = 0; b < 26; b++)
#pragma unroll
                        for (int e = 0; e < 3; e++) acc[e] -= dots[buf][b][e][lane];
                    x[p] = dot3(inv[0], acc[0], inv[1], acc[1], inv[2], acc[2]);
                    x[p + np] = dot3(inv[3], acc[0], inv[4], acc[1], inv[5], acc[2]);
                    x[p + 2 * np] = dot3(inv[6], acc[0], inv[7], acc[1], inv[8], acc[2]);
                }
                if (!last) load(q, false);
            }
        }
        if (q < 4 * c + 3) {   // the plane's next colour reads these values
            colour_arrive(cl);
            load(q + 1, true);
            colour_wait(cl);
        }
    }
}

// res = r - A x over every slot (unused slots get 0), 32 consecutive slots of
// a colour at a time, colour blockIdx.x % 8; NORM: the CTA's sum of
// |r - A x|^2 to partial.
template <bool NORM>
__global__ void __launch_bounds__(kThreads32)
    residual_dense32_kernel(Geom g, DenseOp<float> op, const float *r, const float *x, float *res,
                            double *partial) {
    __shared__ DotTable dots[2];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, q = blockIdx.x & 7;
    const bool sums = wid == kDotWarps;
    const size_t np = (size_t)g.npad;
    const int t0 = 32 * (blockIdx.x >> 3), step = 32 * (gridDim.x >> 3);
    Walk at(g, t0 + lane, step);
    BlockPair row;
    float acc[3], cen[9], v[3];
    int p = -1;
    bool valid = false;
    double sq = 0.0;
    auto load = [&](bool chained = false) {
        valid = at.t < g.S && 2 * at.I + (q & 1) < g.m && 2 * at.J + ((q >> 1) & 1) < g.n && 2 * at.K + (q >> 2) < g.o;
        const int s = valid ? q * g.S + at.t : 0;
        if (!sums) {
            NbrOffsets nb;
            plane_offsets(g, at.I, at.J, q, nb);
            z_offsets(g, at.K, q, nb);
            row.load(op, wid, s, nb, valid);
            if (chained) chain_wait();
            row.load_x<false>(x, g.npad);
        } else {
            p = at.t < g.S ? q * g.S + at.t : -1;
#pragma unroll
            for (int e = 0; e < 9; e++) cen[e] = __ldg(op.coef + coef_at(s) + (117 + e) * kCoefGroup);
            if (chained) chain_wait();
            load3(r, g.npad, s, acc);
            load3(x, g.npad, s, v);
        }
    };
    if (t0 < g.S) load(true);
    else chain_wait();
    int buf = 0;
    for (int t = t0; t < g.S; t += step, buf ^= 1) {
        const bool more = t + step < g.S;
        if (!more) chain_next();
        if (!sums) {
            row.dots(wid, lane, dots[buf]);
            at.next(g);
            if (more) load();
        }
        __syncthreads();
        if (sums) {
            if (valid) {
#pragma unroll
                for (int b = 0; b < 13; b++)
#pragma unroll
                    for (int e = 0; e < 3; e++) acc[e] -= dots[buf][b][e][lane];
                matvec_sub(cen, v, acc);
#pragma unroll
                for (int b = 13; b < 26; b++)
#pragma unroll
                    for (int e = 0; e < 3; e++) acc[e] -= dots[buf][b][e][lane];
                if (NORM)
                    sq += (double)acc[0] * (double)acc[0] + (double)acc[1] * (double)acc[1] +
                          (double)acc[2] * (double)acc[2];
            }
            if (res && p >= 0) {
#pragma unroll
                for (int e = 0; e < 3; e++) res[p + e * np] = valid ? acc[e] : 0.0f;
            }
            at.next(g);
            if (more) load();
        }
    }
    if (NORM && sums) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
        if (lane == 0) partial[blockIdx.x] = sq;
    }
}

// ---------------------------------------------------------------- FP64
constexpr int kNodes64 = 10;    // nodes of a team's item: lane 10 row + node
constexpr int kTeams = 4;
constexpr int kThreads64 = 128 * kTeams;

// The blocks of one part for one (node, row) per lane (coefficients of slot 0
// for a lane without a node).
struct RowPart {
    double a[kPartBlocks][3], v[kPartBlocks][3];
    int s[kPartBlocks];   // the neighbours' slots, negative outside the grid

    template <int PART, bool CENTRE>
    __device__ __forceinline__ void load_part(const DenseOp<double> &op, bool valid, int row, const NbrOffsets &t,
                                              int p) {
        const double *c = op.coef + coef_at(p) + 3 * row * kCoefGroup;
#pragma unroll
        for (int u = 0; u < kPartBlocks; u++) {
            const int b = PART * kPartBlocks + u;
            const bool here = b < 27 && (CENTRE || b != 13);
            s[u] = here && valid ? t.ox[bdx(b) + 1] + t.oy[bdy(b) + 1] + t.oz[bdz(b) + 1] : -1;
#pragma unroll
            for (int e = 0; e < 3; e++) a[u][e] = here ? __ldg(c + (9 * b + e) * kCoefGroup) : 0.0;
        }
    }
    // the block numbers have to be known when the kernel is compiled: the offsets then stay in registers
    template <bool CENTRE>
    __device__ __forceinline__ void load(const DenseOp<double> &op, bool valid, int part, int row, const NbrOffsets &t,
                                         int p) {
        if (part == 0) load_part<0, CENTRE>(op, valid, row, t, p);
        else if (part == 1) load_part<1, CENTRE>(op, valid, row, t, p);
        else if (part == 2) load_part<2, CENTRE>(op, valid, row, t, p);
        else load_part<3, CENTRE>(op, valid, row, t, p);
    }
    // x of the neighbours: of the node's own plane, of the other two, or all
    template <bool COH, bool OWN, bool OTHER>
    __device__ __forceinline__ void load_x(const double *x, int npad, int part) {
#pragma unroll
        for (int u = 0; u < kPartBlocks; u++) {
            const int b = part * kPartBlocks + u;
            const bool own = b >= 9 && b < 18;
            if (own ? !OWN : !OTHER) continue;
            load3<double, COH>(x, npad, max(s[u], 0), v[u]);
            if (s[u] < 0) v[u][0] = v[u][1] = v[u][2] = 0.0;
        }
    }
    __device__ __forceinline__ double sum() const {
        double t = 0.0;
#pragma unroll
        for (int u = 0; u < kPartBlocks; u++)
#pragma unroll
            for (int e = 0; e < 3; e++) t = fma_rn(a[u][e], v[u][e], t);
        return t;
    }
};

__device__ __forceinline__ void team_barrier(int team) {
    asm volatile("bar.sync %0, 128;" ::"r"(team + 1) : "memory");
}

// The lane's row of a 3x3 matrix times the three rows of its node.
__device__ __forceinline__ double row_times(const double (&m)[3], double acc, int node) {
    const double a0 = __shfl_sync(0xffffffffu, acc, node), a1 = __shfl_sync(0xffffffffu, acc, node + kNodes64),
                 a2 = __shfl_sync(0xffffffffu, acc, node + 2 * kNodes64);
    return dot3(m[0], a0, m[1], a1, m[2], a2);
}

__global__ void __launch_bounds__(kThreads64)
    gs_dense64_kernel(Geom g, int c, int cl, DenseOp<double> op, const double *r, double *x) {
    __shared__ double parts[kTeams][2][4][32];
    const int lane = threadIdx.x & 31, part = (threadIdx.x >> 5) & 3, team = threadIdx.x >> 7;
    const int row = lane / kNodes64, node = lane - kNodes64 * row;   // row 3: two idle lanes
    const int rank = blockIdx.x % cl, K = blockIdx.x / cl;
    const int plane = g.M2 * g.N2, groups = (plane + kNodes64 - 1) / kNodes64;
    const int per = (groups + cl * kTeams - 1) / (cl * kTeams);
    const size_t np = (size_t)g.npad;
    const Walk start(g, kNodes64 * (rank + cl * team) + node, kNodes64 * cl * kTeams);
    Walk at = start;
    RowPart rp;
    double acc = 0.0, inv[3] = {0.0, 0.0, 0.0};
    int p = -1;
    bool any = false;   // the item has a node: an empty one must not take the FP64 pipe from the others
    NbrOffsets nb;
    z_offsets(g, K, 4 * c, nb);
    // 10 nodes of colour q of the plane: all that may be read before the colour begins (first) or in it
    auto load = [&](int q, bool first, bool mine, bool chained = false) {
        const bool valid =
            row < 3 && at.t < plane && 2 * at.I + (q & 1) < g.m && 2 * at.J + ((q >> 1) & 1) < g.n;
        any = __any_sync(0xffffffffu, valid);
        if (!any) {
            if (chained) chain_wait();
            return;
        }
        const int s = valid ? q * g.S + K * plane + at.t : 0;
        plane_offsets(g, at.I, at.J, q, nb);
        rp.load<false>(op, valid, part, row < 3 ? row : 0, nb, s);
        if (chained) chain_wait();
        if (first) rp.load_x<true, false, true>(x, g.npad, part);
        else rp.load_x<true, true, true>(x, g.npad, part);
        p = valid ? s : -1;
        if (valid && mine) {
            acc = r[s + row * np];
#pragma unroll
            for (int e = 0; e < 3; e++) inv[e] = __ldg(op.dinv + dinv_at(s) + (3 * row + e) * kCoefGroup);
        }
    };
    int w = 0;   // items so far: the warps take turns at the sums
    load(4 * c, true, part == 0, true);
#pragma unroll 1
    for (int q = 4 * c; q < 4 * c + 4; q++) {
#pragma unroll 1
        for (int n = 0; n < per; n++, w++) {
            if (n + 1 == per && q == 4 * c + 3) chain_next();
            if (any) {   // the same for the whole team
                if (n == 0) rp.load_x<true, true, false>(x, g.npad, part);
                parts[team][w & 1][part][lane] = rp.sum();
                team_barrier(team);   // the item's parts are complete; the item before has been summed
                if ((w & 3) == part) {
#pragma unroll
                    for (int d = 0; d < 4; d++) acc -= parts[team][w & 1][d][lane];
                    const double xn = row_times(inv, acc, node);
                    if (p >= 0) x[p + row * np] = xn;
                }
            }
            if (n + 1 == per) {
                at = start;
            } else {
                at.next(g);
                load(q, false, ((w + 1) & 3) == part);
            }
        }
        if (q < 4 * c + 3) {   // the plane's next colour reads these values
            colour_arrive(cl);
            load(q + 1, true, (w & 3) == part);
            colour_wait(cl);
        }
    }
}

template <typename R, bool NORM>
__global__ void __launch_bounds__(kThreads64)
    residual_dense64_kernel(Geom g, DenseOp<double> op, const double *r, const double *x, R *res,
                            double *partial) {
    __shared__ double parts[kTeams][2][4][32];
    __shared__ double red[kThreads64 / 32];
    const int lane = threadIdx.x & 31, part = (threadIdx.x >> 5) & 3, team = threadIdx.x >> 7;
    const int row = lane / kNodes64, node = lane - kNodes64 * row;
    const size_t np = (size_t)g.npad;
    const int q = blockIdx.x & 7;
    const int t0 = kNodes64 * ((blockIdx.x >> 3) * kTeams + team), step = kNodes64 * (gridDim.x >> 3) * kTeams;
    Walk at(g, t0 + node, step);
    RowPart rp;
    double acc = 0.0, sq = 0.0;
    int p = -1;
    bool valid = false;
    auto load = [&](bool mine, bool chained = false) {
        valid = row < 3 && at.t < g.S && 2 * at.I + (q & 1) < g.m && 2 * at.J + ((q >> 1) & 1) < g.n &&
                2 * at.K + (q >> 2) < g.o;
        const int s = valid ? q * g.S + at.t : 0;
        NbrOffsets nb;
        plane_offsets(g, at.I, at.J, q, nb);
        z_offsets(g, at.K, q, nb);
        rp.load<true>(op, valid, part, row < 3 ? row : 0, nb, s);
        if (chained) chain_wait();
        rp.load_x<false, true, true>(x, g.npad, part);
        p = row < 3 && at.t < g.S ? q * g.S + at.t : -1;
        acc = valid && mine ? r[s + row * np] : 0.0;
    };
    if (t0 < g.S) load(part == 0, true);
    else chain_wait();
    for (int t = t0, n = 0; t < g.S; t += step, n++) {
        if (t + step >= g.S) chain_next();
        parts[team][n & 1][part][lane] = rp.sum();
        team_barrier(team);
        if ((n & 3) == part) {
            if (valid) {
#pragma unroll
                for (int d = 0; d < 4; d++) acc -= parts[team][n & 1][d][lane];
                if (NORM) sq = fma_rn(acc, acc, sq);
            }
            if (res && p >= 0) res[p + row * np] = (R)acc;
        }
        at.next(g);
        if (t + step < g.S) load(((n + 1) & 3) == part);
    }
    if (NORM) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
        if (lane == 0) red[threadIdx.x >> 5] = sq;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < kThreads64 / 32; w++) sq += red[w];
            partial[blockIdx.x] = sq;
        }
    }
}

}  // namespace

// One sweep of a level with per-node rows, two launches; the z extent is not
// odd and periodic (a colour would then meet itself across the wrap).  The
// cluster is as wide as a colour of the plane has groups of nodes, 8 CTAs at
// most.
template <typename T>
void launch_gs_sweep_dense(const LevelOp<T> &op, const Geom &g, const T *r, T *x, cudaStream_t st) {
    const int nodes = sizeof(T) == 4 ? 32 : kNodes64, groups = (g.M2 * g.N2 + nodes - 1) / nodes;
    const int cl = groups >= 8 ? 8 : groups >= 4 ? 4 : groups >= 2 ? 2 : 1;
    for (int c = 0; c < 2; c++) {
        const int planes = c == 0 ? (g.o + 1) / 2 : g.o / 2;
        if (planes == 0) continue;
        if constexpr (sizeof(T) == 4)
            launch_chained(gs_dense32_kernel, cl * planes, kThreads32, 0, st, cl, g, c, cl, op.dop, r, x);
        else
            launch_chained(gs_dense64_kernel, cl * planes, kThreads64, 0, st, cl, g, c, cl, op.dop, r, x);
    }
}

// res = r - A x of a level with per-node rows (res may be null); with partial
// non-null, per-CTA sums of |r - A x|^2.  Returns the number of CTAs: a
// multiple of 8 (a CTA walks the slots of one colour), two an SM in FP32 and
// one in FP64 at most.
template <typename T, typename R>
int launch_residual_dense(const LevelOp<T> &op, const Geom &g, const T *r, const T *x, R *res, double *partial,
                          cudaStream_t st) {
    static_assert(kDensePartials >= 8 * 38);
    if constexpr (sizeof(T) == 4) {
        const int grid = 8 * std::min((g.S + 31) / 32, 38);
        if (partial) launch_chained(residual_dense32_kernel<true>, grid, kThreads32, 0, st, 1, g, op.dop, r, x, res, partial);
        else launch_chained(residual_dense32_kernel<false>, grid, kThreads32, 0, st, 1, g, op.dop, r, x, res, nullptr);
        return grid;
    } else {
        const int items = (g.S + kNodes64 - 1) / kNodes64;
        const int grid = 8 * std::min((items + kTeams - 1) / kTeams, 19);
        if (partial)
            launch_chained(residual_dense64_kernel<R, true>, grid, kThreads64, 0, st, 1, g, op.dop, r, x, res, partial);
        else
            launch_chained(residual_dense64_kernel<R, false>, grid, kThreads64, 0, st, 1, g, op.dop, r, x, res, nullptr);
        return grid;
    }
}

template void launch_gs_sweep_dense<float>(const LevelOp<float> &, const Geom &, const float *, float *, cudaStream_t);
template void launch_gs_sweep_dense<double>(const LevelOp<double> &, const Geom &, const double *, double *,
                                            cudaStream_t);
template int launch_residual_dense<float, float>(const LevelOp<float> &, const Geom &, const float *, const float *,
                                                 float *, double *, cudaStream_t);
template int launch_residual_dense<double, double>(const LevelOp<double> &, const Geom &, const double *,
                                                   const double *, double *, double *, cudaStream_t);
template int launch_residual_dense<double, float>(const LevelOp<double> &, const Geom &, const double *,
                                                  const double *, float *, double *, cudaStream_t);

}  // namespace stzmg
