// File output in the reference's formats, with the values made on the device.
//
//  * z-slices of the solver's fields (region::output_x, output_r,
//    output_residual, mg_3d_template/region.cc:3062-3120), written in the
//    format of region::output_internal (region.cc:3135-3202): a float row
//    {m, x_0 .. x_{m-1}}, then per row j {y_j, m values}.  For vec3 fields the
//    reference converts each value through vec3::operator double (the squared
//    magnitude, src/vec3.hh:110-112): output_x and output_r write
//    float(|v|^2), output_residual float(|r|^2 * |r|^2).
//  * cubes of the simulation's Field members (shear_sim_3d::output_cube,
//    src/shear_sim_3d.cpp:1961-2158): for every x, the (y, z) plane with z
//    fastest, appended as floats to <dir>/<prefix>_grid.<frame>; the
//    node-based members (u, v, w, xi) include the top z node.
//
// Only the device-to-host copy of the finished float array crosses the bus
// (4 bytes per value instead of the Field's 224).
#include <sys/stat.h>
#include <sys/types.h>

#include <cstdio>
#include <string>
#include <vector>

#include "launch.h"
#include "stz_mg.h"

namespace stzmg {

namespace {

__constant__ double kOne = 1.0, kMinusZero = -0.0;
__device__ __forceinline__ double ad(double a, double b) { return __fma_rn(a, kOne, b); }
__device__ __forceinline__ double ml(double a, double b) { return __fma_rn(a, b, kMinusZero); }

// vec3::operator double: x*x + y*y + z*z
__device__ __forceinline__ double sq3(double x, double y, double z) { return ad(ad(ml(x, x), ml(y, y)), ml(z, z)); }

__global__ void slice_kernel(Geom g, const double *__restrict__ f, int k, int quartic, float *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (i >= g.m) return;
    const int s = slot(g, i, j, k);
    const size_t np = (size_t)g.npad;
    const double a = sq3(f[s], f[s + np], f[s + 2 * np]);
    out[i + (size_t)g.m * j] = __double2float_rn(quartic ? ml(a, a) : a);
}

constexpr int kG = 2;   // ghost layers of the simulation grid

// float(sqrt(q)) with the square root correctly rounded in FP64 first.  One
// Newton step from FP32's reciprocal root gives the root to 2^-42; the float
// it rounds to is the same unless it lies that near the middle between two
// floats, where the root is taken exactly, as it is out of FP32's range.  Four
// FP64 instructions for thirteen.
__device__ __forceinline__ float root(double q) {
    const unsigned e = (unsigned)(__double_as_longlong(q) >> 52);   // the sign too: negative is out of range
    if (e - (1023 - 100) > 200) return __double2float_rn(__dsqrt_rn(q));
    const float yf = rsqrtf((float)q);
    const double s0 = q * widen(yf), s = __fma_rn(__fma_rn(-s0, s0, q), widen(0.5f * yf), s0);
    const int past = (int)(__double_as_longlong(s) & 0x1fffffff) - 0x10000000;   // from the middle, in units of 2^-52
    if (abs(past) < 1 << 12) return __double2float_rn(__dsqrt_rn(q));
    return __double2float_rn(s);
}

// The fields run along x and the output along z, so a block turns a tile of 32
// x 32 values of one y over in shared memory: written straight from the
// threads that read it, every value of one of the two sides took a sector of
// its own (192^3 points: a velocity 68 us, the deviatoric stress 688 us, now
// 29 and 323 us).  The deviatoric stress is bound by the FP64 pipe: its
// sums and products are fused multiply-adds by 1 and onto -0 where that saves
// the pipe three cycles in nineteen, with constants the compiler cannot see.
constexpr int kTile = 32;

__global__ void __launch_bounds__(256) cube_kernel(stz_cube_fields f, int nx, int ny, int nz, int mode, int zsize,
                                                   float *__restrict__ out) {
    __shared__ float tile[kTile][kTile + 1];
    const long sy = nx + 2 * kG, sz = sy * (ny + 2 * kG);
    const int xtiles = (nx + kTile - 1) / kTile;
    const int x0 = (int)(blockIdx.x % xtiles) * kTile, z0 = (int)(blockIdx.x / xtiles) * kTile;
    for (int yy = blockIdx.y; yy < ny; yy += gridDim.y) {
        const int xx = x0 + threadIdx.x;
        for (int zt = threadIdx.y; zt < kTile; zt += 8) {
            const int zz = z0 + zt;
            if (xx >= nx || zz >= zsize) continue;
            const long p = (xx + kG) + sy * (yy + kG) + sz * (zz + kG);
            double v = 0;
            float root_of = 0.0f;   // mode 10
            switch (mode) {   // Field::fval (src/field.hh:157-177)
                case 0: v = f.u[p]; break;
                case 1: v = f.v[p]; break;
                case 2: v = f.w[p]; break;
                case 3: v = f.s11[p]; break;
                case 4: v = f.s12[p]; break;
                case 5: v = f.s13[p]; break;
                case 6: v = f.s22[p]; break;
                case 7: v = f.s23[p]; break;
                case 8: v = f.s33[p]; break;
                case 9:
                case 10: {
                    // pressure: -(s11+s22+s33)*(1/3.); dev: sqrt(0.5*(t11^2+t22^2+t33^2) + s12^2 + s13^2 + s23^2)
                    const double s11 = f.s11[p], s22 = f.s22[p], s33 = f.s33[p];
                    const double pr = ml(-ad(ad(s11, s22), s33), 1 / 3.);
                    if (mode == 9) {
                        v = pr;
                    } else {
                        const double t11 = ad(s11, pr), t22 = ad(s22, pr), t33 = ad(s33, pr);
                        const double s12 = f.s12[p], s13 = f.s13[p], s23 = f.s23[p];
                        // half of an exact sum's double: one rounding, of the addition
                        const double q = __fma_rn(0.5, sq3(t11, t22, t33), ml(s12, s12));
                        root_of = root(ad(ad(q, ml(s13, s13)), ml(s23, s23)));
                    }
                    break;
                }
                case 11: v = f.chi[p]; break;
                case 12: v = ml(f.chi[p], 21000.); break;
                case 13: v = f.xi_x[p]; break;
                case 14: v = f.xi_y[p]; break;
                default: v = f.xi_z[p]; break;
            }
            tile[zt][threadIdx.x] = mode == 10 ? root_of : __double2float_rn(v);
        }
        __syncthreads();
        const int zz = z0 + threadIdx.x;
        for (int xt = threadIdx.y; xt < kTile; xt += 8)
            if (x0 + xt < nx && zz < zsize) out[((long)(x0 + xt) * ny + yy) * zsize + zz] = tile[threadIdx.x][xt];
        __syncthreads();
    }
}

bool node_based(int mode) { return mode <= 2 || mode >= 13; }

}  // namespace

void launch_slice(const Geom &g, const double *f, int k, bool quartic, float *out, cudaStream_t st) {
    slice_kernel<<<dim3((g.m + 127) / 128, g.n), 128, 0, st>>>(g, f, k, quartic ? 1 : 0, out);
}

// The body of region::output_internal for one process (mp = np = 1).
bool write_slice_file(const float *vals, int m, int n, double ax, double bx, double ay, double by,
                      const char *filename) {
    FILE *fp = std::fopen(filename, "wb");
    if (!fp) return false;
    const double dx = (bx - ax) / (m - 1), dy = (by - ay) / (n - 1);
    std::vector<float> head(m + 1);
    head[0] = (float)m;
    for (int i = 0; i < m; i++) head[i + 1] = (float)(ax + dx * i);
    bool ok = std::fwrite(head.data(), sizeof(float), m + 1, fp) == (size_t)m + 1;
    for (int j = 0; ok && j < n; j++) {
        const float y = (float)(ay + dy * j);
        ok = std::fwrite(&y, sizeof(float), 1, fp) == 1 &&
             std::fwrite(vals + (size_t)m * j, sizeof(float), m, fp) == (size_t)m;
    }
    return std::fclose(fp) == 0 && ok;
}

}  // namespace stzmg

using namespace stzmg;

extern "C" int stz_mg_cube_values(const stz_cube_fields *f, int nx, int ny, int nz, int mode, float *out,
                                  void *stream) {
    if (!f || !out || nx < 1 || ny < 1 || nz < 1 || mode < 0 || mode > 15) return STZ_MG_ERR_ARG;
    const double *need = mode <= 2    ? (mode == 0 ? f->u : mode == 1 ? f->v : f->w)
                         : mode <= 10 ? f->s11
                         : mode <= 12 ? f->chi
                                      : (mode == 13 ? f->xi_x : mode == 14 ? f->xi_y : f->xi_z);
    if (!need) return STZ_MG_ERR_ARG;
    if (mode >= 3 && mode <= 10 && (!f->s12 || !f->s13 || !f->s22 || !f->s23 || !f->s33)) return STZ_MG_ERR_ARG;
    const int zsize = node_based(mode) ? nz + 1 : nz;
    const dim3 blocks((unsigned)((nx + kTile - 1) / kTile) * ((zsize + kTile - 1) / kTile), std::min(ny, 65535));
    cube_kernel<<<blocks, dim3(kTile, 8), 0, static_cast<cudaStream_t>(stream)>>>(*f, nx, ny, nz, mode, zsize, out);
    return cudaGetLastError() == cudaSuccess ? STZ_MG_OK : STZ_MG_ERR_CUDA;
}

extern "C" int stz_mg_output_cube(const stz_cube_fields *f, int nx, int ny, int nz, int mode, const char *dir,
                                  const char *prefix, int frame) {
    if (!dir || !prefix) return STZ_MG_ERR_ARG;
    const int zsize = (mode <= 2 || mode >= 13) ? nz + 1 : nz;
    const size_t n = (size_t)nx * ny * zsize;
    float *d = nullptr;
    if (cudaMalloc(&d, n * sizeof(float)) != cudaSuccess) return STZ_MG_ERR_OOM;
    std::vector<float> h(n);
    int rc = stz_mg_cube_values(f, nx, ny, nz, mode, d, nullptr);
    if (rc == STZ_MG_OK &&
        (cudaMemcpy(h.data(), d, n * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess))
        rc = STZ_MG_ERR_CUDA;
    cudaFree(d);
    if (rc != STZ_MG_OK) return rc;
    mkdir(dir, 0700);   // as the reference: create the folder if it does not exist
    const std::string path = std::string(dir) + "/" + prefix + "_grid." + std::to_string(frame);
    FILE *fp = std::fopen(path.c_str(), "a");
    if (!fp) return STZ_MG_ERR_ARG;
    const bool ok = std::fwrite(h.data(), sizeof(float), n, fp) == n;
    return (std::fclose(fp) == 0 && ok) ? STZ_MG_OK : STZ_MG_ERR_ARG;
}
