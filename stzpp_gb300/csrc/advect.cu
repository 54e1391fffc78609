// Quasi-static advection step of shear_sim_3d (src/shear_sim_3d.cpp:393-525)
// on the device: the part of step_forward_qs before the projection solve.
//
// Fields are device arrays of the reference's ghosted grid ((nx+4) x (ny+4)
// x (nz+4) points, 2 ghost layers, x fastest), one array per Field member
// (src/field.hh:11-22), the ghosts filled by the caller as the reference's
// set_up_ghost_regions / set_boundary_conditions do.  Three launches:
//
//  1. plastic_kernel: per interior cell, sbar (Field::dev) and, above the
//     yield stress, the adaptive sub-stepping of the STZ plastic rate
//     (adaptive_plastic_term, shear_sim_3d.cpp:108-147), which adds the
//     plastic change of chi to cchi; the new ad_Dpl into scratch;
//  2. update_kernel: the ENO2 advection of the stresses and chi, the
//     Truesdell terms and the chi diffusion (shear_sim_3d.cpp:413-525);
//  3. the new ad_Dpl copied over the old.
//
// The reference updates the points in place in z, y, x order, so a point's
// chi diffusion reads the new ad_Dpl of its interior -x, -y, -z neighbours
// and the previous step's value of the others; update_kernel reads the same.
// Every result is that of the reference's separately rounded operations in
// its order, so it equals the reference's except where it depends on exp (the
// plastic rate), which is CUDA's.
//
// The FP64 pipe bounds the step: one instruction takes it 64 cycles per warp
// and SM scheduler, a comparison or a lane without work as much as any other,
// against 2.8 GB (0.42 ms) of field traffic at 256^3 cells.  So the kernels
// spend as few FP64 instructions as give the same bits:
//  * a product by 2, 4 or 1/2 is exact, so it and the sum it enters are one
//    fused multiply-add;
//  * magnitudes and signs are compared as integers;
//  * the upwind side of eno2 selects operands, not code: the two sides are the
//    same operations up to a sign, and a warp never runs both;
//  * a quotient by a parameter takes five instructions (quotient_by);
//  * cells above the yield stress are collected per block and sub-stepped by
//    full warps, a lane taking the next cell when its own is done.
// 256^3 cells, 23 % above the yield stress: update 23.1 -> 13.3 ms, plastic
// 6.0 -> 2.0 ms; 48x40x24 cells: 107 -> 50 and 42 -> 25 us.
#include <cuda_runtime.h>

#include "stz_mg.h"

namespace {

constexpr int kG = 2;   // ghost layers
// Bound on the adaptive sub-steps of one cell (the reference loops until its
// remaining time is spent; an infinite or NaN-free but huge plastic rate
// would never end): a cell that reaches it stops and the step reports
// STZ_MG_ERR_NONFINITE.
constexpr int kMaxSubsteps = 1 << 22;

// Sums and products as fused multiply-adds by 1 and onto -0, with the same
// single rounding: an SM with all four schedulers busy issues one every 16
// cycles, but an FP64 addition or multiplication only every 19.  The constants
// are in memory, where the compiler cannot turn the operations back.
__constant__ double kOne = 1.0, kMinusZero = -0.0;
__device__ __forceinline__ double ad(double a, double b) { return __fma_rn(a, kOne, b); }
__device__ __forceinline__ double sb(double a, double b) { return __fma_rn(a, kOne, -b); }
__device__ __forceinline__ double ml(double a, double b) { return __fma_rn(a, b, kMinusZero); }
__device__ __forceinline__ double dv(double a, double b) { return __ddiv_rn(a, b); }

__device__ __forceinline__ unsigned long long bits(double a) { return (unsigned long long)__double_as_longlong(a); }
constexpr unsigned long long kInf = 0x7ff0000000000000ull, kSign = 0x8000000000000000ull;
// |a| > |b|, false with a NaN
__device__ __forceinline__ bool mag_above(double a, double b) {
    const unsigned long long u = bits(a) & ~kSign, v = bits(b) & ~kSign;
    return u > v && u <= kInf;
}
// a < 0, false with a NaN
__device__ __forceinline__ bool negative(double a) {
    const unsigned long long u = bits(a);
    return u > kSign && u <= (kSign | kInf);
}
// a with the sign bits of s turned over: a negation that is no FP64 instruction
// (256^3 cells: 16.4 ms with -o and -f3 in eno2, 15.4 ms so)
__device__ __forceinline__ double turned(double a, unsigned long long s) {
    return __longlong_as_double((long long)(bits(a) ^ s));
}
// b + 2^n a, one rounding, for c = 2^n: the product is exact
__device__ __forceinline__ double plus(double b, double c, double a) { return __fma_rn(c, a, b); }

// Correctly rounded quotients by a divisor that is the same everywhere.  With
// y the divisor's correctly rounded reciprocal, a y is within two ulps of the
// quotient, one step q + (a - b q) y leaves less than one, and the step from
// there is correctly rounded (P. Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990,
// theorem 7).  The remainders are exact while nothing nears the ends of the
// exponent range; beyond, the plain division.  The quotient of a zero is the
// first product, with its sign, which the steps would lose.
struct Divisor {
    double b, y;
    bool usual;   // 2^-100 < |b| < 2^100
};

__device__ __forceinline__ double quotient_by(double a, const Divisor &d) {
    const unsigned e = (unsigned)(bits(a) >> 52) & 0x7ff;
    const bool zero = (bits(a) << 1) == 0;
    if (!d.usual || !((e > 223 && e < 1823) || zero)) return dv(a, d.b);
    const double p = ml(a, d.y), q = __fma_rn(__fma_rn(-d.b, p, a), d.y, p);
    return zero ? p : __fma_rn(__fma_rn(-d.b, q, a), d.y, q);
}

struct AdvGrid {
    int nx, ny, nz;
    unsigned cells;
    long sx, sy, sz;   // strides of the ghosted grid: 1, nx + 4, (nx + 4)(ny + 4)
    long npts;
};

// The step's loop-invariant factors, each the reference's own rounded value
// (a correctly rounded division or product gives the same double wherever it
// is computed), worked out once on the host instead of per use: the FP64
// pipe bounds these kernels and a division costs it about ten operations.
struct AdvConst {
    double dxi, dyi, dzi;   // dx_inv = 1./dx (shear_sim_3d.cpp:46)
    double qx, qy, qz;      // .25*dx_inv (calculate_first_order_velocities)
    double hx, hy, hz;      // .5/h of eno2 with h = dx/dt (advection_grid_step)
    double gx, gy, gz;      // .5*dx_inv (chi_diffusion)
    double lx, ly, lz;      // dx_inv*dx_inv (chi_diffusion)
    double third;           // 1./3. (also Field::pressure's 1/3.)
    double dl2;             // diff_l*diff_l
    Divisor c0, sy, mu, bath, tau0, syc0;   // syc0: sy*c0 (calc_chi_F)
    double mu2;             // 2*mu
    double oe;              // omega*eps0
    double elastic;         // 0./2./mu: the new ad_Dpl of a cell below the yield stress over its sbar
};

// Cell t of the interior, x fastest.  Threads take consecutive cells across
// the ends of rows, so every lane has one whatever nx is (an idle lane costs
// the FP64 pipe as much); 2^32 cells would not fit the device's memory.
__device__ __forceinline__ long cell(const AdvGrid &g, unsigned t, int &i, int &j, int &k) {
    const unsigned r = t / (unsigned)g.nx;
    i = t - r * g.nx;
    k = r / (unsigned)g.ny;
    j = r - k * g.ny;
    return (i + kG) + g.sy * (j + kG) + g.sz * (k + kG);
}

// Field::dev (field.hh:147-184)
__device__ __forceinline__ double devstress(double s11, double s12, double s13, double s22, double s23, double s33,
                                            double third) {
    const double p = ml(-ad(ad(s11, s22), s33), third);
    const double t11 = ad(s11, p), t22 = ad(s22, p), t33 = ad(s33, p);
    double q = ml(0.5, ad(ad(ml(t11, t11), ml(t22, t22)), ml(t33, t33)));
    q = ad(ad(ad(q, ml(s12, s12)), ml(s13, s13)), ml(s23, s23));
    return __dsqrt_rn(q);
}

// calc_Dpl with calc_Lambda and calc_curly_c (shear_sim_3d.cpp:1170-1188)
__device__ __forceinline__ double plastic_rate(const stz_adv_params &P, const AdvConst &C, double sbar, double chi) {
    if (!(sbar >= P.sy)) return 0.0;
    const double lam = exp(dv(-P.ez, chi));
    const double oe = ml(C.oe, sbar);
    const double c1 = exp(quotient_by(sb(oe, P.delta), C.bath));
    const double c2 = exp(quotient_by(-ad(oe, P.delta), C.bath));
    const double cc = ml(0.5, ad(c1, c2));
    return quotient_by(ml(ml(lam, cc), sb(1.0, dv(P.sy, sbar))), C.tau0);
}

constexpr int kThreads = 256, kMaxRounds = 8;   // of a block, which takes up to 8 rounds of consecutive cells

__global__ void __launch_bounds__(kThreads)
    plastic_kernel(AdvGrid g, stz_adv_params P, AdvConst C, double dt, int rounds, const double *__restrict__ s11,
                   const double *__restrict__ s12, const double *__restrict__ s13, const double *__restrict__ s22,
                   const double *__restrict__ s23, const double *__restrict__ s33, const double *__restrict__ chi,
                   double *__restrict__ cchi, double *__restrict__ sbar_out, double *__restrict__ adapt_out,
                   double *__restrict__ adnew, double *__restrict__ flag) {
    __shared__ double yield_sbar[kThreads * kMaxRounds];
    __shared__ unsigned short yield_cell[kThreads * kMaxRounds];   // within the block's cells
    __shared__ int found, taken;
    const int lane = threadIdx.x & 31;
    const unsigned first = blockIdx.x * (unsigned)(kThreads * rounds);
    int i, j, k;
    if (threadIdx.x == 0) found = taken = 0;
    __syncthreads();
    for (int l = 0; l < rounds; l++) {
        const unsigned c = kThreads * l + threadIdx.x;
        bool above = false;
        double sbar0 = 0.0;
        if (first + c < g.cells) {
            const long p = cell(g, first + c, i, j, k);
            sbar0 = devstress(s11[p], s12[p], s13[p], s22[p], s23[p], s33[p], C.third);
            sbar_out[p] = sbar0;
            above = sbar0 > P.sy;
            if (!above) {
                adapt_out[p] = 0.0;
                adnew[p] = ml(C.elastic, sbar0);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, above);
        int base = 0;
        if (lane == 0 && m) base = atomicAdd(&found, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1));
        if (above) {
            yield_sbar[base] = sbar0;
            yield_cell[base] = (unsigned short)c;
        }
    }
    __syncthreads();
    // adaptive_plastic_term: sub-steps of at most eta in the scaled plastic strain
    const double eta = .0005;
    const int n = found;
    bool busy = false;
    long p = 0;
    double sbar0 = 0, chi0 = 0, sa = 0, ca = 0, tr = 0;
    int it = 0;
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !busy);
        if (idle) {   // the next cells, one per idle lane
            int base = 0;
            if (lane == 0) base = atomicAdd(&taken, __popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0) + __popc(idle & ((1u << lane) - 1));
            if (!busy && base < n) {
                busy = true;
                p = cell(g, first + yield_cell[base], i, j, k);
                sa = sbar0 = yield_sbar[base];
                ca = chi0 = chi[p];
                tr = dt;
                it = 0;
            }
            if (!__any_sync(0xffffffffu, busy)) break;
        }
        if (busy) {
            bool last = it++ == kMaxSubsteps;
            if (last) {
                flag[1] = 1.0;
            } else {
                const double d = plastic_rate(P, C, sa, ca);
                const double dp = quotient_by(ml(C.mu2, d), C.sy);
                // half of calc_chi_F (shear_sim_3d.cpp:1240-1244)
                const double F = quotient_by(ml(ml(d, sa), sb(P.chi_inf, ca)), C.syc0);
                double ts = tr;
                if (ml(dp, tr) > eta) {
                    ts = dv(eta, fabs(dp));
                    tr = sb(tr, ts);
                } else {
                    last = true;
                }
                sa = sb(sa, ml(ml(ts, dp), P.sy));
                ca = plus(ca, 2.0, ml(ts, F));
            }
            if (last) {
                cchi[p] = ad(cchi[p], sb(ca, chi0));
                const double adapt = sb(1.0, dv(sa, sbar0));
                if (adapt > 0) *flag = 1.0;
                adapt_out[p] = adapt;
                adnew[p] = ml(quotient_by(ml(adapt, 0.5), C.mu), sbar0);   // adapt/2. is exactly adapt*0.5
                busy = false;
            }
        }
    }
}

// eno2 (shear_sim_3d.cpp:1256-1266) along stride st from point p of field f,
// whose value there is f0, three times it f3; half_h = .5/h; neg: the
// velocity is negative.  Only the second difference on the upwind side enters
// the comparison.  With o the point two upwind and b the one between,
//   neg:  side (o - 2 b) + f0,   upwind  (-o + 4 b) - 3 f0
//   else: side (f0 - 2 b) + o,   upwind  (3 f0 - 4 b) + o.
__device__ __forceinline__ double eno2(double half_h, bool neg, const double *__restrict__ f, long p, long st, double f0,
                                       double f3) {
    const double fp = f[p + st], fm = f[p - st], o = f[neg ? p + 2 * st : p - 2 * st], b = neg ? fp : fm;
    const double c2 = ad(plus(fp, -2.0, f0), fm);
    const double side = ad(plus(neg ? o : f0, -2.0, b), neg ? f0 : o);
    const unsigned long long s = neg ? kSign : 0ull;
    const double up = ad(plus(turned(neg ? o : f3, s), neg ? 4.0 : -4.0, b), turned(neg ? f3 : o, s));
    return ml(half_h, mag_above(c2, side) ? up : sb(fp, fm));
}

// the alternating sum a - b + c - d + e - f + g - h of calculate_first_order_velocities
__device__ __forceinline__ double alt8(const double *__restrict__ f, long p, long a, long b, long c, long d, long e,
                                       long f_, long g, long h) {
    return sb(ad(sb(ad(sb(ad(sb(f[p + a], f[p + b]), f[p + c]), f[p + d]), f[p + e]), f[p + f_]), f[p + g]), f[p + h]);
}

// the cell's 8 nodes, in the order of the staggered velocities (shear_sim_3d.cpp:432-434)
__device__ __forceinline__ double node_mean(const double *__restrict__ f, long p, long X, long Y, long Z) {
    double t = ad(f[p], f[p + X]);
    t = ad(t, f[p + Z]);
    t = ad(t, f[p + X + Z]);
    t = ad(t, f[p + Y]);
    t = ad(t, f[p + X + Y]);
    t = ad(t, f[p + Y + Z]);
    t = ad(t, f[p + X + Y + Z]);
    return ml(0.125, t);
}

__device__ __forceinline__ double dot3r(double a, double x, double b, double y, double c, double z) {
    return ad(ad(ml(a, x), ml(b, y)), ml(c, z));
}

__global__ void __launch_bounds__(128) update_kernel(AdvGrid g, stz_adv_params P, AdvConst C, double dt, const double *__restrict__ u,
                              const double *__restrict__ v, const double *__restrict__ w,
                              const double *__restrict__ s11, const double *__restrict__ s12,
                              const double *__restrict__ s13, const double *__restrict__ s22,
                              const double *__restrict__ s23, const double *__restrict__ s33,
                              const double *__restrict__ chi, const double *__restrict__ adold,
                              const double *__restrict__ adapt_in, const double *__restrict__ adnew,
                              double *__restrict__ cs11, double *__restrict__ cs12, double *__restrict__ cs13,
                              double *__restrict__ cs22, double *__restrict__ cs23, double *__restrict__ cs33,
                              double *__restrict__ cchi) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.cells) return;
    int i, j, k;
    const long p = cell(g, t, i, j, k);
    const long X = g.sx, Y = g.sy, Z = g.sz;
    // calculate_first_order_velocities (shear_sim_3d.cpp:900-917)
    const double qx = C.qx, qy = C.qy, qz = C.qz;
    const double du_dx = ml(qx, alt8(u, p, X, 0, X + Y, Y, X + Z, Z, X + Y + Z, Y + Z));
    const double dv_dx = ml(qx, alt8(v, p, X, 0, X + Y, Y, X + Z, Z, X + Y + Z, Y + Z));
    const double dw_dx = ml(qx, alt8(w, p, X, 0, X + Y, Y, X + Z, Z, X + Y + Z, Y + Z));
    const double du_dy = ml(qy, alt8(u, p, Y, 0, X + Y, X, Y + Z, Z, X + Y + Z, X + Z));
    const double dv_dy = ml(qy, alt8(v, p, Y, 0, X + Y, X, Y + Z, Z, X + Y + Z, X + Z));
    const double dw_dy = ml(qy, alt8(w, p, Y, 0, X + Y, X, Y + Z, Z, X + Y + Z, X + Z));
    const double du_dz = ml(qz, alt8(u, p, Z, 0, X + Z, X, Y + Z, Y, X + Y + Z, X + Y));
    const double dv_dz = ml(qz, alt8(v, p, Z, 0, X + Z, X, Y + Z, Y, X + Y + Z, X + Y));
    const double dw_dz = ml(qz, alt8(w, p, Z, 0, X + Z, X, Y + Z, Y, X + Y + Z, X + Y));
    const double adapt = adapt_in[p];
    const double uc = node_mean(u, p, X, Y, Z), vc = node_mean(v, p, X, Y, Z), wc = node_mean(w, p, X, Y, Z);
    const bool un = negative(uc), vn = negative(vc), wn = negative(wc);
    // the velocity times the gradient of a field with value f0 at the cell
    auto advance = [&](const double *__restrict__ f, double f0) {
        const double f3 = ml(3.0, f0);
        return dot3r(uc, eno2(C.hx, un, f, p, X, f0, f3), vc, eno2(C.hy, vn, f, p, Y, f0, f3), wc,
                     eno2(C.hz, wn, f, p, Z, f0, f3));
    };
    const double a11 = s11[p], a12 = s12[p], a13 = s13[p], a22 = s22[p], a23 = s23[p], a33 = s33[p], c0 = chi[p];
    // the Truesdell terms (shear_sim_3d.cpp:476-481); t + 2 (a b) for t + (2 a) b
    const double t11 = plus(plus(ml(a11, sb(sb(du_dx, dv_dy), dw_dz)), 2.0, ml(a13, du_dz)), 2.0, ml(a12, du_dy));
    const double t12 = ad(ad(sb(ad(ml(a23, du_dz), ml(a13, dv_dz)), ml(a12, dw_dz)), ml(a22, du_dy)), ml(a11, dv_dx));
    const double t13 = sb(ad(ad(ad(ml(a33, du_dz), ml(a11, dw_dx)), ml(a23, du_dy)), ml(a12, dw_dy)), ml(a13, dv_dy));
    const double t22 = plus(plus(ml(a22, sb(sb(dv_dy, du_dx), dw_dz)), 2.0, ml(a23, dv_dz)), 2.0, ml(a12, dv_dx));
    const double t23 = ad(sb(ad(ad(ml(a33, dv_dz), ml(a22, dw_dy)), ml(a13, dv_dx)), ml(a23, du_dx)), ml(a12, dw_dx));
    const double t33 = plus(plus(ml(a33, sb(sb(dw_dz, dv_dy), du_dx)), 2.0, ml(a23, dw_dy)), 2.0, ml(a13, dw_dx));
    const double at = ml(adapt, C.third), na = -adapt;
    cs11[p] = ad(sb(ml(at, plus(ad(a33, a22), -2.0, a11)), advance(s11, a11)), ml(dt, t11));
    cs12[p] = ad(sb(ml(na, a12), advance(s12, a12)), ml(dt, t12));
    cs13[p] = ad(sb(ml(na, a13), advance(s13, a13)), ml(dt, t13));
    cs22[p] = ad(sb(ml(at, ad(plus(a11, -2.0, a22), a33)), advance(s22, a22)), ml(dt, t22));
    cs23[p] = ad(sb(ml(na, a23), advance(s23, a23)), ml(dt, t23));
    cs33[p] = ad(sb(ml(at, plus(ad(a11, a22), -2.0, a33)), advance(s33, a33)), ml(dt, t33));
    // chi: advection, then the diffusion (chi_diffusion, shear_sim_3d.cpp:1216-1236)
    double c = sb(cchi[p], advance(chi, c0));
    // ad_Dpl as the reference's in-place sweep sees it
    const double a0 = adnew[p];
    const double axm = i > 0 ? adnew[p - X] : adold[p - X], axp = adold[p + X];
    const double aym = j > 0 ? adnew[p - Y] : adold[p - Y], ayp = adold[p + Y];
    const double azm = k > 0 ? adnew[p - Z] : adold[p - Z], azp = adold[p + Z];
    const double cxm = chi[p - X], cxp = chi[p + X], cym = chi[p - Y], cyp = chi[p + Y], czm = chi[p - Z], czp = chi[p + Z];
    const double dD_dx = ml(C.gx, sb(axp, axm)), dD_dy = ml(C.gy, sb(ayp, aym));
    const double dD_dz = ml(C.gz, sb(azp, azm));
    const double gx = ml(C.gx, sb(cxp, cxm)), gy = ml(C.gy, sb(cyp, cym));
    const double gz = ml(C.gz, sb(czp, czm));
    const double lx = ml(C.lx, ad(plus(cxp, -2.0, c0), cxm));
    const double ly = ml(C.ly, ad(plus(cyp, -2.0, c0), cym));
    const double lz = ml(C.lz, ad(plus(czp, -2.0, c0), czm));
    const double ddx = ad(ml(dD_dx, gx), ml(a0, lx));
    const double ddy = ad(ml(dD_dy, gy), ml(a0, ly));
    const double ddz = ad(ml(dD_dz, gz), ml(a0, lz));
    const double diff = ml(C.dl2, ad(ad(ddx, ddy), ddz));
    cchi[p] = ad(c, quotient_by(diff, C.c0));
}

__global__ void copy_interior_kernel(AdvGrid g, const double *__restrict__ src, double *__restrict__ dst) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.cells) return;
    int i, j, k;
    const long p = cell(g, t, i, j, k);
    dst[p] = src[p];
}

}  // namespace

extern "C" int stz_mg_advection_step(const stz_adv_params *P, const stz_adv_fields *f, double dt, void *stream,
                            int *yielded) {
    if (!P || !f) return STZ_MG_ERR_ARG;
    if (P->nx < 1 || P->ny < 1 || P->nz < 1 || !(dt > 0)) return STZ_MG_ERR_ARG;
    const double *in[] = {f->u, f->v, f->w, f->s11, f->s12, f->s13, f->s22, f->s23, f->s33, f->chi};
    double *out[] = {f->ad_dpl, f->sbar, f->cs11, f->cs12, f->cs13, f->cs22, f->cs23, f->cs33, f->cchi, f->work};
    for (const double *q : in)
        if (!q) return STZ_MG_ERR_ARG;
    for (double *q : out)
        if (!q) return STZ_MG_ERR_ARG;
    AdvGrid g;
    g.nx = P->nx;
    g.ny = P->ny;
    g.nz = P->nz;
    g.cells = (unsigned)P->nx * P->ny * P->nz;
    g.sx = 1;
    g.sy = P->nx + 2 * kG;
    g.sz = g.sy * (P->ny + 2 * kG);
    g.npts = g.sz * (P->nz + 2 * kG);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    AdvConst C;
    C.dxi = 1. / P->dx;
    C.dyi = 1. / P->dy;
    C.dzi = 1. / P->dz;
    C.qx = .25 * C.dxi;
    C.qy = .25 * C.dyi;
    C.qz = .25 * C.dzi;
    C.hx = .5 / (P->dx / dt);
    C.hy = .5 / (P->dy / dt);
    C.hz = .5 / (P->dz / dt);
    C.gx = .5 * C.dxi;
    C.gy = .5 * C.dyi;
    C.gz = .5 * C.dzi;
    C.lx = C.dxi * C.dxi;
    C.ly = C.dyi * C.dyi;
    C.lz = C.dzi * C.dzi;
    C.third = 1. / 3.;
    C.dl2 = P->diff_l * P->diff_l;
    auto divisor = [](double b) {
        const double m = b < 0 ? -b : b;
        return Divisor{b, 1. / b, m > 0x1p-100 && m < 0x1p100};
    };
    C.c0 = divisor(P->c0);
    C.sy = divisor(P->sy);
    C.mu = divisor(P->mu);
    C.bath = divisor(P->bath_temp);
    C.tau0 = divisor(P->tau0);
    C.syc0 = divisor(P->sy * P->c0);
    C.mu2 = 2.0 * P->mu;
    C.oe = P->omega * P->eps0;
    C.elastic = 0.0 / P->mu;
    // work: adaptive terms, new ad_Dpl, then flags {a cell yielded, a cell hit kMaxSubsteps}
    double *adapt = f->work, *adnew = f->work + g.npts, *flag = f->work + 2 * g.npts;
    if (cudaMemsetAsync(flag, 0, 2 * sizeof(double), st) != cudaSuccess) return STZ_MG_ERR_CUDA;
    // cells per block: a long queue keeps the plastic warps full, but every SM wants blocks (four for each of 152)
    auto blocks = [&](unsigned per) { return g.cells / per + (g.cells % per != 0); };
    int rounds = kMaxRounds;
    while (rounds > 1 && blocks(kThreads * rounds) < 4 * 152) rounds /= 2;
    plastic_kernel<<<blocks(kThreads * rounds), kThreads, 0, st>>>(g, *P, C, dt, rounds, f->s11, f->s12, f->s13, f->s22,
                                                                  f->s23, f->s33, f->chi, f->cchi, f->sbar, adapt,
                                                                  adnew, flag);
    // a warp per SM scheduler and block: small grids spread evenly
    update_kernel<<<blocks(128), 128, 0, st>>>(g, *P, C, dt, f->u, f->v, f->w, f->s11, f->s12, f->s13, f->s22, f->s23,
                                               f->s33, f->chi, f->ad_dpl, adapt, adnew, f->cs11, f->cs12, f->cs13,
                                               f->cs22, f->cs23, f->cs33, f->cchi);
    copy_interior_kernel<<<blocks(256), 256, 0, st>>>(g, adnew, f->ad_dpl);
    if (cudaGetLastError() != cudaSuccess) return STZ_MG_ERR_CUDA;
    if (yielded) {
        double h[2] = {0, 0};
        if (cudaMemcpyAsync(h, flag, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return STZ_MG_ERR_CUDA;
        *yielded = h[0] != 0.0;
        if (h[1] != 0.0) return STZ_MG_ERR_NONFINITE;
    }
    return STZ_MG_OK;
}
