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
// (G, G_r, G_z) in o3.  What does not depend on the frequency is multiplied out
// once per pair: S = sr + s0 k G, D = dr + k^2 (a G_r + c G_z).
struct AllwPair {
    double rho, sr, dr, s0, a, c;
    int64_t o;  // pair offset j * n + i
};

// nx, ny, nz: the normal of D, the source panel's when direct (whose derivative
// is by the second argument).
__device__ __forceinline__ AllwPair allw_pair(double dx, double dy, double rho, double area, double sr, double dr,
                                              double nx, double ny, double nz, bool direct, int64_t o)
{
    const double s0 = -kInv4Pi * area, h = rho > 0.0 ? s0 / rho * (nx * dx + ny * dy) : 0.0;
    return AllwPair{rho, sr, dr, s0, direct ? -h : h, s0 * nz, o};
}

__device__ __forceinline__ void allw_emit(const AllwPair& q, int z, double k, const cplx o3[3], int64_t nn,
                                          double2* __restrict__ S64, double2* __restrict__ D64,
                                          float2* __restrict__ Dlo, double2* __restrict__ tape)
{
    const double ks = k * q.s0, k2 = k * k, a = k * q.rho > 1e-6 ? q.a : 0.0;
    const double Sr = fma(ks, o3[0].re, q.sr), Si = ks * o3[0].im;
    const double Dr = fma(k2, fma(a, o3[1].re, q.c * o3[2].re), q.dr);
    const double Di = k2 * fma(a, o3[1].im, q.c * o3[2].im);
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
