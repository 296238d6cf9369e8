// Pieces shared by the frequency-batched Delhommeau kernels (mh_batch.cu,
// mh_rings.cu): panel staging and the output of one (pair, frequency).
// Included after mh_device.cuh, once per translation unit.
#pragma once
#include "mh_device.cuh"
#include "mh_internal.h"

namespace mh {
namespace {

constexpr int kCols = 16;           // source columns per CTA, at most
constexpr int kAllwMaxFreqs = 128;  // frequencies per launch of the frequency-batched kernels
constexpr double kInv4Pi = 1.0 / (4.0 * kPi);

__device__ __forceinline__ void load_panel_field(Panel& p, int f, double v)
{
    if (f < 3) p.c[f] = v;
    else if (f < 6) p.n[f - 3] = v;
    else if (f == G_AREA) p.area = v;
    else if (f == G_RADIUS) p.radius = v;
    else p.v[f - G_V] = v;
}

__device__ __forceinline__ void stage_panels(Panel* sp, const double* __restrict__ geom, int64_t n,
                                             int64_t j0, int cols)
{
    for (int t = threadIdx.x; t < cols * G_NFIELDS; t += blockDim.x) {
        int f = t / cols, jj = t % cols;
        int64_t j = j0 + jj;
        load_panel_field(sp[jj], f, (j < n) ? geom[(int64_t)f * n + j] : 0.0);
    }
}

// One pair of the frequency-batched pass and its output: S, D (FP64 and the
// FP32 copy of D) and the tape of frequency z from the dimensionless
// (G, G_r, G_z) in o3.
struct AllwPair {
    double dx, dy, rho, inv_rho, area, sr, dr;
    double n0, n1, n2;  // the normal of D (source panel when direct), held in registers
    int64_t o;          // pair offset j * n + i
    bool wrt_first;
};

__device__ __forceinline__ void allw_emit(const AllwPair& q, int z, double k, const cplx o3[3], int64_t nn,
                                          double2* __restrict__ S64, double2* __restrict__ D64,
                                          float2* __restrict__ Dlo, double2* __restrict__ tape)
{
    const double r = k * q.rho;
    double d1 = 0.0, d2 = 0.0;
    if (fabs(r) > 1e-6) {
        const double f = k * q.inv_rho;  // k^2 / r
        d1 = q.wrt_first ? f * q.dx : -f * q.dx;
        d2 = q.wrt_first ? f * q.dy : -f * q.dy;
    }
    const double ka = k * q.area;
    const cplx s = ka * o3[0];
    const cplx g0 = (ka * d1) * o3[1], g1 = (ka * d2) * o3[1], g2 = (ka * k) * o3[2];
    const double Sr = q.sr - kInv4Pi * s.re, Si = -kInv4Pi * s.im;
    const double Dr = q.dr - kInv4Pi * (q.n0 * g0.re + q.n1 * g1.re + q.n2 * g2.re);
    const double Di = -kInv4Pi * (q.n0 * g0.im + q.n1 * g1.im + q.n2 * g2.im);
    const int64_t m = (int64_t)z * nn + q.o;
    S64[m] = make_double2(Sr, Si);
    D64[m] = make_double2(Dr, Di);
    Dlo[m] = make_float2((float)Dr, (float)Di);
    if (tape) {  // (G, G_r) for the adjoint of the same call
        tape[2 * m] = make_double2(o3[0].re, o3[0].im);
        tape[2 * m + 1] = make_double2(o3[1].re, o3[1].im);
    }
}

}  // namespace
}  // namespace mh
