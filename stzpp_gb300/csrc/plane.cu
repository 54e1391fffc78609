// FP64 Gauss-Seidel sweep and residual of the plane-invariant coarse levels
// (OP_PLANE), where every node of a plane has the same row of 27 blocks, and
// the FP32 sweep of those that the bands (band.cu) do not take and that are
// small enough to be bound by latency.
//
// The FP64 pipe bounds the FP64 levels: an SM scheduler issues one instruction
// every 64 cycles, with one active lane or 32, so what counts is that lanes
// are full, that all four schedulers of every SM have warps, and the number of
// instructions.  A lane takes one row of one node (10 nodes a warp), the
// plane's row lies in shared memory, and a warp goes down the blocks in the
// order of plane_row_coef (ops.cuh), each entry a fused multiply-add, so that
// the results are those of the colour launches bit for bit.  On planes with
// the elasticity structure a lane skips what is zero in its row: 1, 2 or 3
// products for a face, edge or corner block instead of 3.  Those are the planes
// whose other entries are zero (PlaneOp::structured), and all planes where the
// other kernels of the level skip them too (PlaneOp::sparse: in FP32 up to 1e-9
// of the plane's largest entry).
//
// The sweep is two launches, the even planes and then the odd ones; a cluster
// of up to 8 CTAs runs the four colours of a plane (region::gauss_seidel,
// mg_3d_template/region.cc:1557-1762, in the 8-colour order), and the blocks
// below the plane, which come first and do not depend on the colour before,
// are done ahead of the cluster barrier.
//
// One sweep on GB300, before (eight colour launches, or one block a plane on
// planes of up to 32x32, a thread a node) and now:
//   80x48x65  260 -> 127 us   40x24x33  135 -> 45 us   20x12x17  100 -> 36 us
// and the residual of 80x48x65 168 -> 117 us.
#include <algorithm>

#include "launch.h"
#include "ops.cuh"

namespace stzmg {

namespace {

constexpr int kNodes = 10;   // of a warp: lane 10 row + node, two lanes idle

__device__ __forceinline__ void colour_arrive(int cl) {
    if (cl > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void colour_wait(int cl) {
    if (cl > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
}

// The row of the plane as lane `row` reads it: where its products of an edge
// block lie.  Pair n of axes (xy, xz, yz): components first < second of the
// block's two products in the order of the row, and whether the second is in
// the structure (a row across the pair has its diagonal alone).
struct LaneRow {
    int row, first[3], second[3];
    bool two[3];
    __device__ __forceinline__ explicit LaneRow(int r) : row(r) {
#pragma unroll
        for (int n = 0; n < 3; n++) {
            const int p = n == 2 ? 1 : 0, q = n == 0 ? 1 : 2;
            two[n] = r == p || r == q;
            first[n] = two[n] ? p : r;
            second[n] = two[n] ? q : r;
        }
    }
};

// acc -= blocks 9 d .. 9 d + 8 of the lane's row (d = 0, 1, 2: the planes
// below, at and above the node), x of the node's own plane through L2 when
// other CTAs write it (COH).
template <typename T, bool SPARSE, bool WITH_CENTRE, bool COH>
__device__ __forceinline__ T row_part(int d, const T *cf, const LaneRow &L, const NbrOffsets &t, const T *x, int npad,
                                      T acc) {
    const T *xr = x + t.oz[d];
    const bool zin = t.oz[d] >= 0;
    auto value = [&](const T *p, bool in) {
        T v = T(0);
        if (in) v = COH && d == 1 ? load_l2(p) : *p;
        return v;
    };
    T v[9][3];
#pragma unroll
    for (int n = 0; n < 9; n++) {
        const int dx = n % 3 - 1, dy = n / 3 - 1, s = t.ox[dx + 1] + t.oy[dy + 1];
        const bool in = zin && t.ox[dx + 1] >= 0 && t.oy[dy + 1] >= 0;
        const int axes = (dx != 0) + (dy != 0) + (d != 1);
        if (n == 4 && d == 1 && !WITH_CENTRE) continue;
        if (SPARSE && axes <= 1) {
            v[n][0] = value(xr + s + L.row * (size_t)npad, in);
        } else if (SPARSE && axes == 2) {
            const int pair = d == 1 ? 0 : dx != 0 ? 1 : 2;
            v[n][0] = value(xr + s + L.first[pair] * (size_t)npad, in);
            v[n][1] = value(xr + s + L.second[pair] * (size_t)npad, in);
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++) v[n][c] = value(xr + s + c * (size_t)npad, in);
        }
    }
    const T *c = cf + 81 * d + 3 * L.row;
#pragma unroll
    for (int n = 0; n < 9; n++) {
        const int dx = n % 3 - 1, dy = n / 3 - 1;
        const int axes = (dx != 0) + (dy != 0) + (d != 1);
        if (n == 4 && d == 1 && !WITH_CENTRE) continue;
        if (SPARSE && axes <= 1) {
            acc = fma_rn(-c[9 * n + L.row], v[n][0], acc);
        } else if (SPARSE && axes == 2) {
            const int pair = d == 1 ? 0 : dx != 0 ? 1 : 2;
            acc = fma_rn(-c[9 * n + L.first[pair]], v[n][0], acc);
            acc = fma_rn(L.two[pair] ? -c[9 * n + L.second[pair]] : T(-0.0), v[n][1], acc);
        } else {
#pragma unroll
            for (int e = 0; e < 3; e++) acc = fma_rn(-c[9 * n + e], v[n][e], acc);
        }
    }
    return acc;
}

template <typename T>
__device__ __forceinline__ void stage_row(const PlaneOp<T> &op, int k, T *cf) {
    for (int e = threadIdx.x; e < 252; e += blockDim.x)
        cf[e] = e < 243 ? op.coef[(size_t)e * op.O + k] : op.dinv[(size_t)(e - 243) * op.O + k];
    __syncthreads();
}

// One item of a lane's row, whichever structure its plane has.
template <bool WITH_CENTRE, bool COH, typename T>
__device__ __forceinline__ T any_row_part(bool sparse, int d, const T *cf, const LaneRow &L, const NbrOffsets &t,
                                          const T *x, int npad, T acc) {
    if (sparse) return row_part<T, true, WITH_CENTRE, COH>(d, cf, L, t, x, npad, acc);
    return row_part<T, false, WITH_CENTRE, COH>(d, cf, L, t, x, npad, acc);
}

constexpr int kMaxWarps = 12;   // two CTAs share an SM: their colours' barriers overlap

// Colours 4c .. 4c+3 of every plane of parity c, `cl` CTAs (one cluster) per
// plane; x is updated in place.
template <typename T>
__global__ void __launch_bounds__(32 * kMaxWarps, 2)
    gs_plane_rows_kernel(Geom g, int c, int cl, PlaneOp<T> op, const T *r, T *x) {
    __shared__ T cf[252];
    const int lane = threadIdx.x & 31, row = min(lane / kNodes, 2), node = lane % kNodes;
    const int rank = blockIdx.x % cl, K = blockIdx.x / cl, plane = g.M2 * g.N2;
    const int warps = cl * (blockDim.x >> 5), first = rank * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int groups = (plane + kNodes - 1) / kNodes, rounds = (groups + warps - 1) / warps;
    const size_t np = (size_t)g.npad;
    const LaneRow L(row);
    const bool sparse = op.sparse || op.structured[2 * K + c];
    stage_row(op, 2 * K + c, cf);
    chain_wait();
    NbrOffsets nb;
    dim_offsets(K, c, g.o, g.O2, g.zp, 4 * g.S, plane, nb.oz);
    int p = -1;
    bool any = false;   // an item without nodes must not take the FP64 pipe from the others
    T acc = T(0);
    // item n of this warp in colour q, and the blocks below its plane
    auto begin = [&](int q, int n) {
        const int t = kNodes * (first + n * warps) + node, J = t / g.M2, I = t - J * g.M2;
        const bool valid =
            lane < 3 * kNodes && t < plane && 2 * I + (q & 1) < g.m && 2 * J + ((q >> 1) & 1) < g.n;
        any = __any_sync(0xffffffffu, valid);
        if (!any) return;
        p = valid ? q * g.S + K * plane + t : -1;
        dim_offsets(valid ? I : 0, q & 1, g.m, g.M2, g.xp, g.S, 1, nb.ox);
        dim_offsets(valid ? J : 0, (q >> 1) & 1, g.n, g.N2, g.yp, 2 * g.S, g.M2, nb.oy);
        acc = valid ? r[p + row * np] : T(0);
        acc = any_row_part<false, true>(sparse, 0, cf, L, nb, x, g.npad, acc);
    };
    auto end = [&]() {
        if (!any) return;
        acc = any_row_part<false, true>(sparse, 1, cf, L, nb, x, g.npad, acc);
        acc = any_row_part<false, true>(sparse, 2, cf, L, nb, x, g.npad, acc);
        const T a0 = __shfl_sync(0xffffffffu, acc, node), a1 = __shfl_sync(0xffffffffu, acc, node + kNodes),
                a2 = __shfl_sync(0xffffffffu, acc, node + 2 * kNodes);
        const T *inv = cf + 243 + 3 * row;
        const T xn = dot3(inv[0], a0, inv[1], a1, inv[2], a2);
        if (p >= 0) x[p + row * np] = xn;
    };
    begin(4 * c, 0);
#pragma unroll 1
    for (int q = 4 * c; q < 4 * c + 4; q++) {
#pragma unroll 1
        for (int n = 0; n < rounds; n++) {
            if (n + 1 == rounds && q == 4 * c + 3) chain_next();
            end();
            if (n + 1 < rounds) begin(q, n + 1);
        }
        if (q < 4 * c + 3) {   // the plane's next colour reads these values
            colour_arrive(cl);
            begin(q + 1, 0);
            colour_wait(cl);
        }
    }
}

// res = r - A x of plane blockIdx.y (unused slots get 0): four colours, a warp per 10 slots.
__global__ void __launch_bounds__(256)
    residual_plane64_kernel(Geom g, PlaneOp<double> op, const double *r, const double *x, double *res) {
    __shared__ double cf[252];
    const int lane = threadIdx.x & 31, row = min(lane / kNodes, 2), node = lane % kNodes;
    const int k = blockIdx.y, c = k & 1, K = k >> 1, plane = g.M2 * g.N2, groups = (plane + kNodes - 1) / kNodes;
    const int item = blockIdx.x * 8 + (threadIdx.x >> 5);
    const size_t np = (size_t)g.npad;
    if (k < g.o) stage_row(op, k, cf);
    chain_wait();
    if (item >= 4 * groups) return;
    const int ab = item & 3, q = 4 * c + ab, t = kNodes * (item >> 2) + node, J = t / g.M2, I = t - J * g.M2;
    const bool slot = lane < 3 * kNodes && t < plane;
    const bool valid = slot && k < g.o && 2 * I + (ab & 1) < g.m && 2 * J + (ab >> 1) < g.n;
    const int p = q * g.S + K * plane + t;
    double acc = 0.0;
    if (__any_sync(0xffffffffu, valid)) {
        NbrOffsets nb;
        dim_offsets(K, c, g.o, g.O2, g.zp, 4 * g.S, plane, nb.oz);
        dim_offsets(valid ? I : 0, q & 1, g.m, g.M2, g.xp, g.S, 1, nb.ox);
        dim_offsets(valid ? J : 0, (q >> 1) & 1, g.n, g.N2, g.yp, 2 * g.S, g.M2, nb.oy);
        const LaneRow L(row);
        const bool sparse = op.structured[k];
        if (valid) acc = r[p + row * np];
#pragma unroll
        for (int d = 0; d < 3; d++) acc = any_row_part<true, false>(sparse, d, cf, L, nb, x, g.npad, acc);
    }
    chain_next();
    if (slot) res[p + row * np] = valid ? acc : 0.0;
}

}  // namespace

// One sweep, two launches; the z extent is not odd and periodic.  A warp per
// 10 nodes of a colour of the plane as far as 8 CTAs of 12 warps go, the
// warps spread over the CTAs before they are added to them: on a small plane a
// second warp on a scheduler only waits for the first.
template <typename T>
void launch_gs_sweep_plane(const PlaneOp<T> &op, const Geom &g, const T *r, T *x, cudaStream_t st) {
    const int groups = (g.M2 * g.N2 + kNodes - 1) / kNodes;
    const int cl = groups > 16 ? 8 : groups > 8 ? 4 : groups > 4 ? 2 : 1;
    const int warps = std::min(kMaxWarps, ((groups + cl - 1) / cl + 3) / 4 * 4);
    for (int c = 0; c < 2; c++) {
        const int planes = c == 0 ? (g.o + 1) / 2 : g.o / 2;
        if (planes == 0) continue;
        launch_chained(gs_plane_rows_kernel<T>, cl * planes, 32 * warps, 0, st, cl, g, c, cl, op, r, x);
    }
}

template void launch_gs_sweep_plane<float>(const PlaneOp<float> &, const Geom &, const float *, float *, cudaStream_t);
template void launch_gs_sweep_plane<double>(const PlaneOp<double> &, const Geom &, const double *, double *,
                                            cudaStream_t);

void launch_residual_plane64(const PlaneOp<double> &op, const Geom &g, const double *r, const double *x, double *res,
                             cudaStream_t st) {
    const int groups = (g.M2 * g.N2 + kNodes - 1) / kNodes;
    const dim3 grid((4 * groups + 7) / 8, 2 * g.O2);
    launch_chained(residual_plane64_kernel, grid, 256, 0, st, 1, g, op, r, x, res);
}

}  // namespace stzmg
