// FP64 kernels: influence-matrix assembly, boundary conditions and the
// pressure -> force reduction.
//
// Assembly (src/matrix_assembly.jl:4-42): the frequency-independent Rankine
// terms by tiles with their near pairs listed, and the wave terms added where a
// tile is stored (mh_rankine.cuh).  For a fixed column the 128 threads of a CTA
// write 128 consecutive complex128 entries of the column-major matrix, so every
// store is a fully coalesced 2 KiB run.
#include <cuda_runtime.h>

#include "mh_device.cuh"
#include "mh_internal.h"
#include "mh_rankine.cuh"

namespace mh {

namespace {

constexpr double kInv4Pi = 1.0 / (4.0 * kPi);  // -1/(2 tau), tau = 2 pi (MarineHydro.jl:11)

// S and D with the -1/(4 pi) factor and the 1/2 diagonal of D: complex, with
// the wave terms kWave (bits) at wavenumber k added (either of S and D may be
// null), or the real Rankine parts.
template <uint32_t kWave>
struct AssembleOut {
    double2 *S, *D;
    const double* tab;
    double k;
    int direct;
    static __device__ __forceinline__ double take(double v) { return v; }
    __device__ __forceinline__ void store(int64_t o, bool diag, double s, double d, const double (*xs)[kRkRows],
                                          int row, const Panel& p) const
    {
        double si = 0.0, di = 0.0;
        if (kWave) {
            const double x[3] = {xs[0][row], xs[1][row], xs[2][row]};
            cplx w, g[3];
            pair_integrals(x, p, k, kWave, !direct, tab, w, g);
            const double n0 = direct ? p.n[0] : xs[3][row], n1 = direct ? p.n[1] : xs[4][row],
                         n2 = direct ? p.n[2] : xs[5][row];
            s += w.re;
            si = -kInv4Pi * w.im;
            d += n0 * g[0].re + n1 * g[1].re + n2 * g[2].re;
            di = -kInv4Pi * (n0 * g[0].im + n1 * g[1].im + n2 * g[2].im);
        }
        if (S) S[o] = make_double2(-kInv4Pi * s, si);
        if (D) D[o] = make_double2((diag ? 0.5 : 0.0) - kInv4Pi * d, di);
    }
};
struct RankineRealOut {
    double *S, *D;
    static __device__ __forceinline__ double take(double v) { return v; }
    __device__ __forceinline__ void store(int64_t o, bool diag, double s, double d, const double (*)[kRkRows], int,
                                          const Panel&) const
    {
        S[o] = -kInv4Pi * s;
        D[o] = (diag ? 0.5 : 0.0) - kInv4Pi * d;
    }
};

__device__ __forceinline__ void dof_at(const double* dof, int64_t dof_rows, int64_t n, int64_t i,
                                       double d[3])
{
    if (dof_rows == 1) {
        d[0] = dof[0];
        d[1] = dof[1];
        d[2] = dof[2];
    } else {
        d[0] = dof[i];
        d[1] = dof[n + i];
        d[2] = dof[2 * n + i];
    }
}

// src/waves.jl:4-18, :89-101
__global__ void k_radiation_bc(const double* __restrict__ geom, int64_t n,
                               const double* __restrict__ dof, int64_t dof_rows, double omega,
                               double2* __restrict__ bc)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d[3];
    dof_at(dof, dof_rows, n, i, d);
    double nd = geom[G_NX * n + i] * d[0] + geom[G_NY * n + i] * d[1] + geom[G_NZ * n + i] * d[2];
    bc[i] = make_double2(0.0, -omega * nd);  // -i omega (n . dof)
}

// src/waves.jl:121-142: v = (g k / omega) e^{i k wbar} (cos b e^{kz}, sin b e^{kz}, -i e^{kz})
__global__ void k_airy_bc(const double* __restrict__ geom, int64_t n, double omega, double beta,
                          double gacc, double2* __restrict__ bc)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double k = omega * omega / gacc;
    double cb, sb;
    sincos(beta, &sb, &cb);
    double x = geom[G_CX * n + i], y = geom[G_CY * n + i], z = geom[G_CZ * n + i];
    double wbar = x * cb + y * sb;
    double cih = exp(k * z);
    double sw, cw;
    sincos(k * wbar, &sw, &cw);
    double f = gacc * k / omega;
    cplx e = mk(f * cw, f * sw);
    cplx v0 = e * (cb * cih), v1 = e * (sb * cih), v2 = e * mk(0.0, -cih);
    double nx = geom[G_NX * n + i], ny = geom[G_NY * n + i], nz = geom[G_NZ * n + i];
    cplx vn = v0 * nx + v1 * ny + v2 * nz;
    bc[i] = make_double2(-vn.re, -vn.im);
}

// src/waves.jl:21-25 with p = i rho omega phi (src/waves.jl:34, :56).
// One CTA; a fixed-order tree reduction, so the result is deterministic.
__global__ void __launch_bounds__(1024)
k_force(const double* __restrict__ geom, int64_t n, const double2* __restrict__ phi,
        const double* __restrict__ dof, int64_t dof_rows, double rho, double omega,
        double2* __restrict__ F_out)
{
    __shared__ double sr[1024], si[1024];
    double ar = 0.0, ai = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double d[3];
        dof_at(dof, dof_rows, n, i, d);
        double amp = -(geom[G_NX * n + i] * d[0] + geom[G_NY * n + i] * d[1] +
                       geom[G_NZ * n + i] * d[2]);
        double w = amp * geom[G_AREA * n + i];
        double2 ph = phi[i];
        // i rho omega phi = rho omega (-phi.im, phi.re)
        ar += rho * omega * (-ph.y) * w;
        ai += rho * omega * (ph.x) * w;
    }
    sr[threadIdx.x] = ar;
    si[threadIdx.x] = ai;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            sr[threadIdx.x] += sr[threadIdx.x + s];
            si[threadIdx.x] += si[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) F_out[0] = make_double2(sr[0], si[0]);
}

}  // namespace

cudaError_t launch_assemble_f64(mh_ctx* ctx, const mh_mesh* m, double k, uint32_t mask, int direct,
                                const double* tab, double2* S, double2* D)
{
    const RankineGeom in{m->geom, m->n};
    const auto go = [&](auto out) { return launch_rankine_tile<double>(ctx, in, m->n, mask, direct, out); };
    switch (mask & (MH_GF_WU | MH_GF_DELHOMMEAU)) {
        case 0: return go(AssembleOut<0>{S, D, tab, k, direct});
        case MH_GF_WU: return go(AssembleOut<MH_GF_WU>{S, D, tab, k, direct});
        case MH_GF_DELHOMMEAU: return go(AssembleOut<MH_GF_DELHOMMEAU>{S, D, tab, k, direct});
        default: return go(AssembleOut<MH_GF_WU | MH_GF_DELHOMMEAU>{S, D, tab, k, direct});
    }
}

cudaError_t launch_rankine_real(mh_ctx* ctx, const mh_mesh* m, uint32_t mask, int direct, double* SR, double* DR)
{
    return launch_rankine_tile<double>(ctx, RankineGeom{m->geom, m->n}, m->n, mask, direct, RankineRealOut{SR, DR});
}

cudaError_t launch_radiation_bc(mh_ctx* ctx, const mh_mesh* m, const double* dof, int64_t dof_rows,
                                double omega, double2* bc)
{
    const int64_t n = m->n;
    k_radiation_bc<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(m->geom, n, dof, dof_rows,
                                                                         omega, bc);
    ctx->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_airy_bc(mh_ctx* ctx, const mh_mesh* m, double omega, double beta, double g,
                           double2* bc)
{
    const int64_t n = m->n;
    k_airy_bc<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(m->geom, n, omega, beta, g, bc);
    ctx->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_force(mh_ctx* ctx, const mh_mesh* m, const double2* phi, const double* dof,
                         int64_t dof_rows, double rho, double omega, double2* F_out)
{
    k_force<<<1, 1024, 0, ctx->stream>>>(m->geom, m->n, phi, dof, dof_rows, rho, omega, F_out);
    ctx->launches += 1;
    return cudaGetLastError();
}


}  // namespace mh
