// Inverse of the dense bottom-level matrix in FP64: Gauss-Jordan elimination
// in place, partial pivoting, a panel of w columns at a time.  With the
// panel's pivot rows P (w x w) swapped into place and Q = P^-1, a panel step
// turns the n x n array into
//     panel columns: Q on the pivot rows, -A_i Q on the others,
//     other columns: Q A_P on the pivot rows, A_i - (A_i Q) A_P on the others,
// and after all of them the array is the inverse of the row-permuted matrix.
//
// Three launches a panel:
//  * gj_panel_kernel: one cluster of 16 CTAs (8 where 16 do not fit) holds the
//    panel in shared memory, rows spread over the CTAs, and eliminates its
//    columns one by one.  Per column every CTA sends its pivot candidate, with
//    the candidate's whole row, to the others, so one cluster barrier a column
//    is enough.
//  * gj_rows_kernel: the row swaps on the other columns; the pivot rows'
//    values go to a w x n scratch.
//  * gj_update_kernel: the rank-w update, 64 x 64 tiles.  A tile whose
//    multipliers are all zero is left alone: the bottom operator couples
//    neighbouring planes only, so most of the rows below a panel are.
// The panel needs few SMs for long (161 us at n = 1728), the update all of them
// (127 us): the next panel's columns are updated first, and its panel then runs
// on a second stream beside the update of the rest.
// The elimination of one column per launch that this replaces read and wrote
// the whole n x 2n array [M | I] for each of the n columns: n = 1728 (8x8x9
// nodes) took 55 ms, now 13 ms; the panels alone take 8.8 and the updates
// 6.8 (5.4 at the FP64 pipe's rate without the empty tiles).
#include <algorithm>

#include "launch.h"

namespace stzmg {

namespace {

constexpr int kMaxCtas = 16, kPanelThreads = 32 * kMaxCtas;
constexpr int kPanelSmem = 200 * 1024;   // a CTA's share of a panel

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Address of a shared-memory location in another CTA of the cluster.
__device__ __forceinline__ unsigned peer_address(const void *p, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void peer_store(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void peer_store(unsigned a, long long v) {
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void peer_store(unsigned a, int v) {
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Magnitudes are compared as the bits of |v|, which order as the values do (an
// FP64 comparison would take the FP64 pipe, 64 cycles a warp); a NaN is above
// every number.  Zero, infinity and NaN are no pivots.
__device__ __forceinline__ long long magnitude(double v) { return __double_as_longlong(v) & 0x7fffffffffffffffll; }
__device__ __forceinline__ bool no_pivot(long long m) { return m <= 0 || m >= 0x7ff0000000000000ll; }
__device__ __forceinline__ bool better(long long m, int i, long long than, int at) {
    return m > than || (m == than && (unsigned)i < (unsigned)at);
}

// 1/v, correctly rounded, by Newton steps from FP32's reciprocal: six
// FP64 instructions on the elimination's critical path, fewer than the division.
// Two steps leave less than an ulp of error, from where a third one rounds
// correctly unless v's significand is all ones (P. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34,
// 1990); without it reciprocals next to the middle between two doubles are off.
// That significand and values out of FP32's range take the division.
__device__ __forceinline__ double reciprocal(double v) {
    const long long b = __double_as_longlong(v), ones = (1ll << 52) - 1;
    const unsigned e = (unsigned)(b >> 52) & 0x7ff;
    if (e < 1023 - 100 || e > 1023 + 100 || (b & ones) == ones) return 1.0 / v;
    double y = (double)(1.0f / (float)v);
    y = fma_rn(fma_rn(-v, y, 1.0), y, y);
    y = fma_rn(fma_rn(-v, y, 1.0), y, y);
    return fma_rn(fma_rn(-v, y, 1.0), y, y);
}

// What a CTA sends for a column: its pivot candidate (the largest magnitude
// among its rows from the column's on; row -1 without one) and that row, and
// from the CTA that holds the column's own row, that row.
template <int W>
struct Offer {
    double row[W];
    long long mag;
    int index;
};

template <int W>
__global__ void __launch_bounds__(kPanelThreads)
    gj_panel_kernel(double *__restrict__ a, int n, int c0, int w, int ctas, int rows, int *__restrict__ pivots,
                    int *bad) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Offer<W> offers[2][kMaxCtas];
    __shared__ double own[2][W];   // the column's own row
    __shared__ double prow[W];     // the pivot row divided by the pivot
    __shared__ long long wmag[kPanelThreads / 32];
    __shared__ int widx[kPanelThreads / 32];
    double *s = reinterpret_cast<double *>(smem);   // column e of local row i: s[e * rows + i]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, rank = blockIdx.x;
    const int r0 = rank * rows, mine = max(0, min(rows, n - r0));
    for (int t = tid; t < mine * w; t += kPanelThreads) {
        const int i = t / w, e = t - i * w;
        s[e * rows + i] = a[(size_t)(r0 + i) * n + c0 + e];
    }
    __syncthreads();
    cluster_sync();   // every CTA runs before the first remote store
    for (int k = 0; k < w; k++) {
        const int c = c0 + k, b = k & 1;
        // this CTA's candidate: the largest |a(i, c)| of its rows i >= c, the lowest such row
        long long best = -1;
        int at = -1;
        for (int i = max(0, c - r0) + tid; i < mine; i += kPanelThreads) {
            const long long v = magnitude(s[k * rows + i]);
            if (v > best) best = v, at = r0 + i;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const long long v = __shfl_down_sync(0xffffffffu, best, o);
            const int j = __shfl_down_sync(0xffffffffu, at, o);
            if (better(v, j, best, at)) best = v, at = j;
        }
        if (lane == 0) wmag[wid] = best, widx[wid] = at;
        __syncthreads();
        best = wmag[0], at = widx[0];
        for (int v = 1; v < kPanelThreads / 32; v++)
            if (better(wmag[v], widx[v], best, at)) best = wmag[v], at = widx[v];
        // warp d sends to CTA d: the candidate and its row, and the column's own row
        if (wid < ctas) {
            Offer<W> *to = &offers[b][rank];
            if (lane == 0) {
                peer_store(peer_address(&to->mag, wid), best);
                peer_store(peer_address(&to->index, wid), at);
            }
            for (int e = lane; e < w; e += 32) {
                if (at >= 0) peer_store(peer_address(&to->row[e], wid), s[e * rows + at - r0]);
                if (c >= r0 && c < r0 + mine) peer_store(peer_address(&own[b][e], wid), s[e * rows + c - r0]);
            }
        }
        cluster_sync();
        int from = 0;
        best = offers[b][0].mag, at = offers[b][0].index;
        for (int d = 1; d < ctas; d++)
            if (better(offers[b][d].mag, offers[b][d].index, best, at))
                best = offers[b][d].mag, at = offers[b][d].index, from = d;
        if (tid < w) {
            const double inv = reciprocal(offers[b][from].row[k]);
            prow[tid] = tid == k ? inv : offers[b][from].row[tid] * inv;
            // rows c and the pivot's change places
            if (at >= r0 && at < r0 + mine) s[tid * rows + at - r0] = own[b][tid];
        }
        if (rank == 0 && tid == 0) {
            pivots[c] = max(at, c);
            if (no_pivot(best)) atomicExch(bad, 1);
        }
        __syncthreads();
        // eliminate column c from this CTA's rows; a row with a zero there stays
        for (int i = tid; i < mine; i += kPanelThreads) {
            if (r0 + i == c) {
                for (int e = 0; e < w; e++) s[e * rows + i] = prow[e];
                continue;
            }
            const double f = s[k * rows + i];
            if (magnitude(f) == 0) continue;
#pragma unroll
            for (int e = 0; e < W; e++)
                if (e < w && e != k) s[e * rows + i] -= f * prow[e];
            s[k * rows + i] = -f * prow[k];
        }
        __syncthreads();
    }
    for (int t = tid; t < mine * w; t += kPanelThreads) {
        const int i = t / w, e = t - i * w;
        a[(size_t)(r0 + i) * n + c0 + e] = s[e * rows + i];
    }
}

// The panel's row swaps on every other column; the pivot rows' values to
// `rows` (w x n) and zeros in their place.  A thread per column takes the
// w rows of the panel and the rows they change with into shared memory, so
// that all its loads are in flight together, and swaps them there.
template <int W>
__global__ void __launch_bounds__(64)
    gj_rows_kernel(double *__restrict__ a, int n, int c0, int w, const int *__restrict__ pivots,
                   double *__restrict__ rows) {
    __shared__ double val[2 * W][64];
    __shared__ int piv[W], with[W];   // row k changes with: row piv[k], held in val[with[k]]
    const int tid = threadIdx.x, q = blockIdx.x * 64 + tid;
    if (tid < w) piv[tid] = pivots[c0 + tid];
    __syncthreads();
    if (tid < w) {
        int j = 0;
        while (piv[j] != piv[tid]) j++;   // a row may be a pivot's place more than once
        with[tid] = piv[tid] < c0 + w ? piv[tid] - c0 : W + j;
    }
    __syncthreads();
    if (q >= n || (q >= c0 && q < c0 + w)) return;
#pragma unroll 8
    for (int k = 0; k < w; k++) {
        val[k][tid] = a[(size_t)(c0 + k) * n + q];
        if (with[k] == W + k) val[W + k][tid] = a[(size_t)piv[k] * n + q];
    }
    for (int k = 0; k < w; k++) {
        const double t = val[k][tid];
        val[k][tid] = val[with[k]][tid];
        val[with[k]][tid] = t;
    }
    for (int k = 0; k < w; k++) {
        rows[(size_t)k * n + q] = val[k][tid];
        a[(size_t)(c0 + k) * n + q] = 0.0;
        if (with[k] == W + k) a[(size_t)piv[k] * n + q] = val[W + k][tid];
    }
}

constexpr int kTile = 64;

// A(:, q) += panel(:, .) rows(., q) for the columns q of [q_lo, q_hi) that are
// not in [skip_lo, skip_hi).
template <int W>
__global__ void __launch_bounds__(256)
    gj_update_kernel(double *__restrict__ a, int n, int c0, int w, int q_lo, int q_hi, int skip_lo, int skip_hi,
                     const double *__restrict__ rows) {
    __shared__ double m[W][kTile + 1], v[W][kTile];
    const int tid = threadIdx.x, i0 = blockIdx.y * kTile, q0 = q_lo + blockIdx.x * kTile;
    int some = 0, filled = 0;
    for (int t = tid; t < kTile * W; t += 256) {
        const int i = t / W, e = t % W;
        const double f = i0 + i < n && e < w ? a[(size_t)(i0 + i) * n + c0 + e] : 0.0;
        m[e][i] = f;
        some |= magnitude(f) != 0;
        const int q = t % kTile, k = t / kTile;
        const bool in = q0 + q < q_hi && k < w && !(q0 + q >= skip_lo && q0 + q < skip_hi);
        const double g = in ? rows[(size_t)k * n + q0 + q] : 0.0;
        v[k][q] = g;
        filled |= magnitude(g) != 0;
    }
    const bool both = __syncthreads_or(some) != 0;
    if (__syncthreads_or(filled) == 0 || !both) return;
    // thread: rows ty + 16 u, columns tx + 16 v
    const int tx = tid & 15, ty = tid >> 4;
    double acc[4][4];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int z = 0; z < 4; z++) acc[u][z] = 0.0;
#pragma unroll 4
    for (int e = 0; e < W; e++) {
        double f[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; u++) f[u] = m[e][ty + 16 * u];
#pragma unroll
        for (int z = 0; z < 4; z++) g[z] = v[e][tx + 16 * z];
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int z = 0; z < 4; z++) acc[u][z] += f[u] * g[z];
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int z = 0; z < 4; z++) {
            const int i = i0 + ty + 16 * u, q = q0 + tx + 16 * z;
            if (i < n && q < q_hi && !(q >= skip_lo && q < skip_hi)) a[(size_t)i * n + q] += acc[u][z];
        }
}

// order[j]: the column of the array that belongs at column j of the inverse,
// the row swaps undone in reverse (one thread: n steps, once per set-up).
__global__ void gj_order_kernel(int n, const int *__restrict__ pivots, int *__restrict__ order) {
    extern __shared__ int ord[];
    for (int j = threadIdx.x; j < n; j += blockDim.x) ord[j] = j;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int c = n - 1; c >= 0; c--) {
            const int p = pivots[c], t = ord[c];
            ord[c] = ord[p];
            ord[p] = t;
        }
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += blockDim.x) order[j] = ord[j];
}

__global__ void gj_gather_kernel(const double *__restrict__ a, int n, const int *__restrict__ order,
                                 double *__restrict__ inv) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) inv[(size_t)blockIdx.y * n + q] = a[(size_t)blockIdx.y * n + order[q]];
}

// ------------------------------------------------------------ Fourier blocks
// The inverse of a plane-invariant bottom operator periodic in x and y.  The
// operator couples column (i, j) of nodes to column (i + dx, j + dy) through a
// block A(d) of order 3o that does not depend on (i, j), so a discrete Fourier
// transform in x and y leaves m n independent complex systems
//     D(t) = sum_d A(d) e^{i t.d},  t = 2 pi (kx / m, ky / n),
// and the inverse couples the columns through B(d) = 1/(m n) sum_t D(t)^-1
// e^{-i t.d}.  A CTA per t builds D(t) from the planes' rows and inverts it in
// shared memory by the same elimination as above; a column's magnitudes are
// compared by their squares unless those leave the exponent range.  On the host,
// one system after the other, 64 systems of order 27 took 11.6 ms; here 134 us.
constexpr int kFourierThreads = 256;
constexpr int kFourierOrder = 104;   // two arrays of order^2 doubles in shared memory

// Squares of magnitudes in here are far from the ends of the exponent range.
constexpr long long kSmallSquare = (1023ll - 900) << 52, kLargeSquare = (1023ll + 900) << 52;

// 2^-n for a value of about 2^n, within the range where both are normal numbers.
__device__ __forceinline__ double unit_of(double v) {
    const int n = (int)(magnitude(v) >> 52) - 1023;
    return __longlong_as_double((long long)(1023 - max(-1000, min(1000, n))) << 52);
}

// work: null, or 2 bs^2 doubles per CTA for systems beyond shared memory.
__global__ void __launch_bounds__(kFourierThreads)
    fourier_inverse_kernel(Geom g, PlaneOp<double> op, double2 *__restrict__ out, double *work, int *bad) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int bs = 3 * g.o, tid = threadIdx.x, kx = blockIdx.x % g.m, ky = blockIdx.x / g.m;
    double2 *prow = reinterpret_cast<double2 *>(smem), *col = prow + bs;
    int *order = reinterpret_cast<int *>(col + bs), *pivots = order + bs;
    double *re = work ? work + 2 * (size_t)blockIdx.x * bs * bs
                      : reinterpret_cast<double *>(smem + (size_t)bs * (2 * sizeof(double2) + 2 * sizeof(int)));
    double *im = re + bs * bs;
    __shared__ double2 wx[3], wy[3];
    __shared__ int piv, far;   // the pivot's row, and whether its square is out of range
    if (tid < 6) {   // e^{i t d}
        const int d = tid % 3 - 1;
        double sn, cs;
        if (tid < 3) sincospi(2.0 * ((kx * d) % g.m) / g.m, &sn, &cs);
        else sincospi(2.0 * ((ky * d) % g.n) / g.n, &sn, &cs);
        (tid < 3 ? wx : wy)[tid % 3] = make_double2(cs, sn);
    }
    for (int t = tid; t < 2 * bs * bs; t += kFourierThreads) re[t] = 0.0;
    __syncthreads();
    for (int t = tid; t < 9 * g.o; t += kFourierThreads) {   // row (k, a), columns (., c)
        const int k = t / 9, e = t % 9, a = e / 3, c = e % 3;
        for (int b = 0; b < 27; b++) {
            const int kk = wrap_or_out(k + b / 9 - 1, g.o, g.zp);
            if (kk < 0) continue;
            const double v = op.coef[(size_t)(9 * b + e) * op.O + k];
            const double2 x = wx[b % 3], y = wy[b / 3 % 3];
            const int at = (3 * k + a) * bs + 3 * kk + c;
            re[at] += v * (x.x * y.x - x.y * y.y);
            im[at] += v * (x.x * y.y + x.y * y.x);
        }
    }
    __syncthreads();
    for (int c = 0; c < bs; c++) {
        if (tid < 32) {
            long long best;
            int at;
            auto search = [&](auto size) {
                best = -1, at = c;
                for (int r = c + tid; r < bs; r += 32) {
                    const long long q = magnitude(size(re[r * bs + c], im[r * bs + c]));
                    if (q > best) best = q, at = r;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const long long v = __shfl_xor_sync(0xffffffffu, best, o);
                    const int j = __shfl_xor_sync(0xffffffffu, at, o);
                    if (better(v, j, best, at)) best = v, at = j;
                }
            };
            search([](double u, double v) { return u * u + v * v; });
            const bool extreme = best < kSmallSquare || best > kLargeSquare;
            if (extreme) search([](double u, double v) { return hypot(u, v); });
            if (tid == 0) {
                piv = pivots[c] = at;
                far = extreme;
                if (no_pivot(best)) atomicExch(bad, 1);
            }
        }
        __syncthreads();
        // swap rows c and piv; the pivot row over the pivot, and column c
        const int p = piv;
        const double unit = far ? unit_of(fmax(fabs(re[p * bs + c]), fabs(im[p * bs + c]))) : 1.0;
        double pr = re[p * bs + c], pi = im[p * bs + c];
        if (far) pr *= unit, pi *= unit;
        for (int e = tid; e < bs; e += kFourierThreads) {
            const double s2 = 1.0 / (pr * pr + pi * pi);
            double ir = pr * s2, ii = -pi * s2;
            if (far) ir *= unit, ii *= unit;
            const double ur = re[p * bs + e], ui = im[p * bs + e];
            prow[e] = e == c ? make_double2(ir, ii) : make_double2(ur * ir - ui * ii, ur * ii + ui * ir);
            const int r = e == p ? c : e;   // the row whose values are at e after the swap
            col[e] = make_double2(re[r * bs + c], im[r * bs + c]);
        }
        __syncthreads();
        for (int t = tid; t < bs * bs; t += kFourierThreads) {
            const int r = t / bs, e = t - r * bs;
            if (r == c) continue;
            const int from = (r == p ? c : r) * bs + e;
            const double2 f = col[r], q = prow[e];
            const double vr = e == c ? 0.0 : re[from], vi = e == c ? 0.0 : im[from];
            re[t] = vr - (f.x * q.x - f.y * q.y);
            im[t] = vi - (f.x * q.y + f.y * q.x);
        }
        __syncthreads();
        for (int e = tid; e < bs; e += kFourierThreads) re[c * bs + e] = prow[e].x, im[c * bs + e] = prow[e].y;
        __syncthreads();
    }
    if (tid == 0) {   // the row swaps, undone as column swaps
        for (int j = 0; j < bs; j++) order[j] = j;
        for (int c = bs - 1; c >= 0; c--) {
            const int t = order[c];
            order[c] = order[pivots[c]];
            order[pivots[c]] = t;
        }
    }
    __syncthreads();
    for (int t = tid; t < bs * bs; t += kFourierThreads) {
        const int r = t / bs, e = t - r * bs;
        out[(size_t)blockIdx.x * bs * bs + t] = make_double2(re[r * bs + order[e]], im[r * bs + order[e]]);
    }
}

// B(d), d = (blockIdx.y % m, blockIdx.y / m).
__global__ void fourier_blocks_kernel(int m, int n, int bs, const double2 *__restrict__ G, double *__restrict__ B) {
    extern __shared__ double2 w[];   // e^{-i t.d} of every t
    const int dx = blockIdx.y % m, dy = blockIdx.y / m, e = blockIdx.x * blockDim.x + threadIdx.x;
    for (int t = threadIdx.x; t < m * n; t += blockDim.x) {
        double xs, xc, ys, yc;
        sincospi(-2.0 * (t % m * dx % m) / m, &xs, &xc);
        sincospi(-2.0 * (t / m * dy % n) / n, &ys, &yc);
        w[t] = make_double2(xc * yc - xs * ys, xc * ys + xs * yc);
    }
    __syncthreads();
    if (e >= bs * bs) return;
    double s = 0.0;
    for (int t = 0; t < m * n; t++) {
        const double2 v = G[(size_t)t * bs * bs + e];
        s += v.x * w[t].x - v.y * w[t].y;
    }
    B[(size_t)blockIdx.y * bs * bs + e] = s / (m * n);
}

__global__ void fourier_expand_kernel(Geom g, const double *__restrict__ B, double *__restrict__ inv) {
    const int nr = 3 * g.m * g.n * g.o, bs = 3 * g.o;
    const int q = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
    if (q >= nr) return;
    const int p = r / 3, p2 = q / 3;
    int di = p2 % g.m - p % g.m, dj = p2 / g.m % g.n - p / g.m % g.n;
    if (di < 0) di += g.m;
    if (dj < 0) dj += g.n;
    const int k = p / (g.m * g.n), k2 = p2 / (g.m * g.n);
    inv[(size_t)r * nr + q] = B[((size_t)(di + g.m * dj) * bs + 3 * k + r % 3) * bs + 3 * k2 + q % 3];
}

__device__ __forceinline__ bool beyond_one_node(const Geom &g, const int *S, int s) {
    bool far = false;
#pragma unroll
    for (int e = 0; e < 6; e++) {
        const int v = S[(size_t)e * g.npad + s];
        far |= e & 1 ? v > 2 : v < -1;
    }
    return far;
}

// bad[1] is set when a node's box reaches beyond one node.
__global__ void box_check_kernel(Geom g, const int *__restrict__ S, int *bad) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= g.m * g.n * g.o) return;
    const int s = slot(g, p % g.m, p / g.m % g.n, p / (g.m * g.n));
    if (beyond_one_node(g, S, s)) atomicExch(bad + 1, 1);
}

// M (n x n, natural node order, 3 rows per node) from grouped rows and box
// bounds: the blocks of a node's box, added where wraps make two of them
// meet.  bad[1] is set when a box reaches beyond one node.
__global__ void bottom_matrix_kernel(Geom g, const double *__restrict__ coef, const int *__restrict__ S,
                                     double *__restrict__ M, int n, int *bad) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int p = t / 3, a = t - 3 * p;
    const int i = p % g.m, j = p / g.m % g.n, k = p / (g.m * g.n), s = slot(g, i, j, k);
    const double *row = coef + coef_at(s);
    int box[6];
    for (int e = 0; e < 6; e++) box[e] = S[(size_t)e * g.npad + s];
    if (box[0] < -1 || box[1] > 2 || box[2] < -1 || box[3] > 2 || box[4] < -1 || box[5] > 2) {
        atomicExch(bad + 1, 1);
        return;
    }
    for (int dk = box[4]; dk < box[5]; dk++)
        for (int dj = box[2]; dj < box[3]; dj++)
            for (int di = box[0]; di < box[1]; di++) {
                const int ii = wrap_or_out(i + di, g.m, g.xp), jj = wrap_or_out(j + dj, g.n, g.yp),
                          kk = wrap_or_out(k + dk, g.o, g.zp);
                if (ii < 0 || jj < 0 || kk < 0) continue;
                const int q = ii + g.m * (jj + g.n * kk), b = (di + 1) + 3 * (dj + 1) + 9 * (dk + 1);
                for (int c = 0; c < 3; c++) M[(size_t)t * n + 3 * q + c] += row[(9 * b + 3 * a + c) * kCoefGroup];
            }
}

// CTAs of the panel's cluster: 16 if the device runs such a cluster with this much shared memory, else 8.
template <int W>
int panel_ctas(int n) {
    cudaFuncSetAttribute(gj_panel_kernel<W>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    static SmemLimit limit;
    limit.allow(kPanelSmem, gj_panel_kernel<W>);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kPanelThreads);
    cfg.dynamicSmemBytes = kPanelSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, gj_panel_kernel<W>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        fit = 0;
    }
    return fit > 0 ? 16 : 8;
}

template <int W>
void launch_panel(double *a, int n, int c0, int ctas, int *pivots, int *bad, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kPanelThreads);
    // all of an SM's shared memory, so that no block of an update shares its FP64 pipe
    cfg.dynamicSmemBytes = kPanelSmem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, gj_panel_kernel<W>, a, n, c0, std::min(W, n - c0), ctas, (n + ctas - 1) / ctas, pivots, bad);
}

// A second stream, of the highest priority, and the events that order it.
struct SideStream {
    cudaStream_t st = nullptr;
    cudaEvent_t ready = nullptr, done = nullptr;
    SideStream() {
        int low = 0, high = 0;
        cudaDeviceGetStreamPriorityRange(&low, &high);
        if (cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, high) != cudaSuccess) st = nullptr;
        if (cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) != cudaSuccess) ready = nullptr;
        if (cudaEventCreateWithFlags(&done, cudaEventDisableTiming) != cudaSuccess) done = nullptr;
    }
    bool ok() const { return st && ready && done; }
    ~SideStream() {   // all three end when the work that uses them has
        if (ready) cudaEventDestroy(ready);
        if (done) cudaEventDestroy(done);
        if (st) cudaStreamDestroy(st);
    }
};

template <int W>
void eliminate(double *a, int n, double *rows, int *pivots, int *bad, cudaStream_t st) {
    const int ctas = panel_ctas<W>(n), tiles = (n + kTile - 1) / kTile;
    SideStream side;
    launch_panel<W>(a, n, 0, ctas, pivots, bad, st);
    for (int c0 = 0; c0 < n; c0 += W) {
        const int w = std::min(W, n - c0), c1 = c0 + w, c2 = std::min(n, c1 + W);
        gj_rows_kernel<W><<<(n + 63) / 64, 64, 0, st>>>(a, n, c0, w, pivots, rows);
        if (c1 < n) {
            gj_update_kernel<W><<<dim3(1, tiles), 256, 0, st>>>(a, n, c0, w, c1, c2, c0, c1, rows);
            if (side.ok()) {
                cudaEventRecord(side.ready, st);
                cudaStreamWaitEvent(side.st, side.ready, 0);
                launch_panel<W>(a, n, c1, ctas, pivots, bad, side.st);
                cudaEventRecord(side.done, side.st);
            }
        }
        gj_update_kernel<W><<<dim3(tiles, tiles), 256, 0, st>>>(a, n, c0, w, 0, n, c0, c2, rows);
        if (c1 < n) {
            if (side.ok()) cudaStreamWaitEvent(st, side.done, 0);
            else launch_panel<W>(a, n, c1, ctas, pivots, bad, st);
        }
    }
}

}  // namespace

// Shared memory of a system of order bs: two rows and the pivots; the system
// too, unless it works in the inverse's place, which is written last.  (With
// three columns or more an order is at most kMaxBottomNodes.)
static int fourier_smem(int bs) {
    return bs * (int)(2 * sizeof(double2) + 2 * sizeof(int)) +
           (bs <= kFourierOrder ? 2 * bs * bs * (int)sizeof(double) : 0);
}

// False where the blocks would not fit the scratch (n x n doubles): one or two
// columns, for which the plain inverse is as good.
bool launch_fourier_inverse(const PlaneOp<double> &op, const Geom &g, const int *S, double *inv, double *scratch,
                            int *bad, cudaStream_t st) {
    const int bs = 3 * g.o, cols = g.m * g.n, n = bs * cols;
    if (!g.xp || !g.yp || cols < 3) return false;
    const int smem = fourier_smem(bs), phases = cols * (int)sizeof(double2);
    static SmemLimit inverse_limit, blocks_limit;
    inverse_limit.allow(std::max(fourier_smem(kFourierOrder), fourier_smem(kMaxBottomNodes)), fourier_inverse_kernel);
    blocks_limit.allow(kMaxBottomNodes * (int)sizeof(double2), fourier_blocks_kernel);
    double2 *G = reinterpret_cast<double2 *>(scratch);
    double *B = scratch + 2 * (size_t)cols * bs * bs;
    box_check_kernel<<<(g.m * g.n * g.o + 127) / 128, 128, 0, st>>>(g, S, bad);
    fourier_inverse_kernel<<<cols, kFourierThreads, smem, st>>>(g, op, G,
                                                             bs <= kFourierOrder ? nullptr : inv, bad);
    fourier_blocks_kernel<<<dim3((bs * bs + 127) / 128, cols), 128, phases, st>>>(g.m, g.n, bs, G, B);
    fourier_expand_kernel<<<dim3((n + 255) / 256, n), 256, 0, st>>>(g, B, inv);
    return true;
}

void launch_bottom_matrix(const Geom &g, const double *coef, const int *S, double *M, int *bad, cudaStream_t st) {
    const int n = 3 * g.m * g.n * g.o;
    cudaMemsetAsync(M, 0, (size_t)n * n * sizeof(double), st);
    bottom_matrix_kernel<<<(n + 127) / 128, 128, 0, st>>>(g, coef, S, M, n, bad);
}

// Panels of 32 columns while an eighth of one fits a CTA's shared memory
// (n <= 6400), else of 16.
void launch_gauss_jordan(double *a, int n, double *inv, int *pivots, double *rows, int *bad, cudaStream_t st) {
    if ((n + 7) / 8 * 32 * (int)sizeof(double) <= kPanelSmem) eliminate<kInversePanel>(a, n, rows, pivots, bad, st);
    else eliminate<16>(a, n, rows, pivots, bad, st);
    gj_order_kernel<<<1, 1024, n * sizeof(int), st>>>(n, pivots, pivots + n);
    gj_gather_kernel<<<dim3((n + 255) / 256, n), 256, 0, st>>>(a, n, pivots + n, inv);
}

}  // namespace stzmg
