// Construction of the tabulated Guevel-Delhommeau wave term (see mh_table.cuh)
// and the point-evaluation hook mh_wave_term.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "mh_internal.h"
#include "mh_device.cuh"
#include "mh_rings.cuh"

namespace mh {
namespace {

// B and C at the table nodes, from the FP64 adaptive quadrature.
__global__ void k_table_nodes(const double* __restrict__ rr, const double* __restrict__ zz, int n,
                              double* __restrict__ B, double* __restrict__ C,
                              double* __restrict__ E0, double* __restrict__ E1)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double r = rr[t], z = zz[t];
    cplx o[3];
    delh_dimless(r, z, o);
    double az = -z, R = hypot(r, z);
    double e = exp(z), J0 = j0(r), J1 = j1(r);
    double L = log(0.5 * (R + az));
    B[t] = o[0].re + 2.0 * e * J0 * L;
    C[t] = o[1].re - (2.0 * e * J1 * L - 2.0 * e * J0 * r / (R * (R + az)));
    E0[t] = e * J0;
    E1[t] = e * J1;
}

// Dimensionless (G, dG/dr, dG/dz) at arbitrary points.
__global__ void k_wave_term(const double* __restrict__ tab, uint32_t which, int64_t n,
                            const double* __restrict__ rr, const double* __restrict__ zz,
                            double* __restrict__ out)
{
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    cplx o[3];
    if (which == MH_GF_WU) wu_dimless(rr[t], zz[t], o);
    else if (tab) delh_dimless_table(tab, rr[t], zz[t], o);
    else delh_dimless(rr[t], zz[t], o);
    for (int q = 0; q < 3; ++q) {
        out[6 * t + 2 * q] = o[q].re;
        out[6 * t + 2 * q + 1] = o[q].im;
    }
}

void cheb_nodes(int n, double a, double b, std::vector<double>& x)
{
    x.resize(n);
    for (int k = 0; k < n; ++k)
        x[k] = 0.5 * (a + b) + 0.5 * (b - a) * std::cos(M_PI * (k + 0.5) / n);
}

// T[i * n + l]: weight of node l in the Chebyshev coefficient i.  Computed once per
// order (per cell it was 4 ms of cosines).
std::vector<double> cheb_weights(int n)
{
    std::vector<double> T((size_t)n * n);
    for (int i = 0; i < n; ++i)
        for (int l = 0; l < n; ++l) T[(size_t)i * n + l] = (i == 0 ? 1.0 : 2.0) / n * std::cos(M_PI * i * (l + 0.5) / n);
    return T;
}

// Chebyshev coefficients of an n x m block of node values (row = first coord), Tn and
// Tm the weights of the two orders.
void cheb_coeffs(int n, int m, const std::vector<double>& Tn, const std::vector<double>& Tm, const double* vals,
                 double* coef)
{
    std::vector<double> tmp((size_t)n * m);
    for (int i = 0; i < n; ++i)
        for (int l = 0; l < m; ++l) {
            double s = 0.0;
            for (int k = 0; k < n; ++k) s += Tn[(size_t)i * n + k] * vals[(size_t)k * m + l];
            tmp[(size_t)i * m + l] = s;
        }
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < m; ++j) {
            double s = 0.0;
            for (int l = 0; l < m; ++l) s += tmp[(size_t)i * m + l] * Tm[(size_t)j * m + l];
            coef[(size_t)i * m + j] = s;
        }
}

// P[i * n + m]: coefficient of u^m in T_i(u), i, m < n.
std::vector<double> cheb_to_powers(int n)
{
    std::vector<double> P((size_t)n * n, 0.0);
    P[0] = 1.0;
    if (n > 1) P[(size_t)n + 1] = 1.0;
    for (int i = 2; i < n; ++i)  // T_i = 2 u T_{i-1} - T_{i-2}
        for (int m = 0; m < n; ++m)
            P[(size_t)i * n + m] = (m > 0 ? 2.0 * P[(size_t)(i - 1) * n + m - 1] : 0.0) - P[(size_t)(i - 2) * n + m];
    return P;
}

// Where A[m][j] of the fragments that start at word `first` belongs (mh_contract.cuh).
size_t frag_at(int first, int cols, int m, int j)
{
    const int lane = 4 * (m % 8) + j % 4;
    return (size_t)first + 64 * ((m / 16) * frag_steps(cols) + j / 4) + 2 * lane + (m % 16) / 8;
}

}  // namespace

int ensure_delh_table(mh_ctx* ctx)
{
    if (ctx->delh_table) return MH_OK;
    // Node coordinates: rings, cells, polar patch.  The quadrature takes longest near the
    // surface, and a warp as long as its longest node, so nodes of one angle or depth stand
    // next to each other, the hardest first: k_table_nodes 18 ms; 28.6 with the rings last
    // and the nodes of a ring or cell by its rows, 22.1 with the rings first, 15.7 before
    // there were rings.
    std::vector<double> r, z;
    std::vector<double> xa, xb;
    size_t ring_at[kRings], nodes = (size_t)kTabNP * kTabNP + (size_t)kTabNCell * kTabNCell * kTabNC * kTabNC;
    for (int q = 0; q < kRings; ++q) nodes += (size_t)ring_fit_r(q) * ring_fit_a(q);
    r.reserve(nodes);
    z.reserve(nodes);
    for (int q = kRings - 1; q >= 0; --q) {
        ring_at[q] = r.size();
        cheb_nodes(ring_fit_r(q), 2.0 * (1 << q), 4.0 * (1 << q), xa);
        cheb_nodes(ring_fit_a(q), 0.0, 0.5 * M_PI, xb);
        for (const double al : xb) {
            const double sn = std::sin(al), cn = std::cos(al);
            for (const double R : xa) {
                r.push_back(R * sn);
                z.push_back(-R * cn);
            }
        }
    }
    const size_t cells_at = r.size();
    std::vector<double> xr((size_t)kTabNCell * kTabNC);
    for (int ir = 0; ir < kTabNCell; ++ir) {
        cheb_nodes(kTabNC, ir * kTabH, (ir + 1) * kTabH, xa);
        std::copy(xa.begin(), xa.end(), xr.begin() + (size_t)ir * kTabNC);
    }
    for (int iz = 0; iz < kTabNCell; ++iz) {
        cheb_nodes(kTabNC, iz * kTabH, (iz + 1) * kTabH, xb);
        for (int l = kTabNC - 1; l >= 0; --l) {  // from the surface
            r.insert(r.end(), xr.begin(), xr.end());
            z.insert(z.end(), xr.size(), -xb[l]);
        }
    }
    const size_t polar_at = r.size();
    cheb_nodes(kTabNP, 0.0, kTabRPolar, xa);
    cheb_nodes(kTabNP, 0.0, 0.5 * M_PI, xb);
    for (int k = 0; k < kTabNP; ++k)
        for (int l = 0; l < kTabNP; ++l) {
            r.push_back(xa[k] * std::sin(xb[l]));
            z.push_back(-xa[k] * std::cos(xb[l]));
        }
    const int n = (int)r.size();
    double *d_r = nullptr, *d_z = nullptr, *d_B = nullptr, *d_C = nullptr, *d_E0 = nullptr,
           *d_E1 = nullptr, *d_tab = nullptr;
    auto cleanup = [&]() {
        cudaFree(d_r);
        cudaFree(d_z);
        cudaFree(d_B);
        cudaFree(d_C);
        cudaFree(d_E0);
        cudaFree(d_E1);
    };
    size_t bytes = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d_r, bytes) != cudaSuccess || cudaMalloc(&d_z, bytes) != cudaSuccess ||
        cudaMalloc(&d_B, bytes) != cudaSuccess || cudaMalloc(&d_C, bytes) != cudaSuccess ||
        cudaMalloc(&d_E0, bytes) != cudaSuccess || cudaMalloc(&d_E1, bytes) != cudaSuccess ||
        cudaMalloc(&d_tab, sizeof(double) * kTabAllWords) != cudaSuccess) {
        cudaGetLastError();
        cleanup();
        cudaFree(d_tab);
        return set_err(ctx, MH_ERR_OOM, "allocation of the Delhommeau table failed");
    }
    std::vector<double> hB(n), hC(n), hE0(n), hE1(n), tab(kTabAllWords);
    cudaError_t e = cudaMemcpyAsync(d_r, r.data(), bytes, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_z, z.data(), bytes, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        k_table_nodes<<<(n + 127) / 128, 128, 0, ctx->stream>>>(d_r, d_z, n, d_B, d_C, d_E0, d_E1);
        ctx->launches += 1;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(hB.data(), d_B, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hC.data(), d_C, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hE0.data(), d_E0, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hE1.data(), d_E1, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        cleanup();
        cudaFree(d_tab);
        return set_err(ctx, MH_ERR_CUDA, "Delhommeau table nodes: %s", cudaGetErrorString(e));
    }
    // polar block: B, C, E0, E1, fitted on kTabNP x kTabNP nodes; the first
    // kTabNU rows (degrees in R) are kept, and again as fragments with the rows
    // in the monomial basis of u: T_i(u) = sum_m P[i][m] u^m
    std::vector<float> mono(4 * kTabPolarFn);
    {
        std::vector<double> full((size_t)kTabNP * kTabNP);
        const std::vector<double> P = cheb_to_powers(kTabNU);
        const std::vector<double> T = cheb_weights(kTabNP);
        const double* src[4] = {hB.data() + polar_at, hC.data() + polar_at, hE0.data() + polar_at, hE1.data() + polar_at};
        for (int q = 0; q < 4; ++q) {
            cheb_coeffs(kTabNP, kTabNP, T, T, src[q], full.data());
            for (int i = 0; i < kTabNU; ++i)
                for (int j = 0; j < kTabNV; ++j)
                    tab[(size_t)q * kTabPolarFn + i * kTabNV + j] = full[(size_t)i * kTabNP + j];
            for (int m = 0; m < kTabNU; ++m)
                for (int j = 0; j < kTabNV; ++j) {
                    double a = 0.0;
                    for (int i = m; i < kTabNU; ++i) a += P[(size_t)i * kTabNU + m] * full[(size_t)i * kTabNP + j];
                    tab[frag_at(kFragPolar, kTabNV, 4 * m + q, j)] = a;
                    mono[4 * (m * kTabNV + j) + q] = (float)a;
                }
        }
    }
    // cells
    {
        constexpr int nc = kTabNC * kTabNC;
        const std::vector<double> T = cheb_weights(kTabNC);
        std::vector<double> cell(nc);
        for (int iz = 0; iz < kTabNCell; ++iz)
            for (int ir = 0; ir < kTabNCell; ++ir)
                for (int f = 0; f < 2; ++f) {
                    const double* src = (f ? hC : hB).data() + cells_at;
                    for (int l = 0; l < kTabNC; ++l)
                        for (int k = 0; k < kTabNC; ++k)
                            cell[(size_t)k * kTabNC + l] =
                                src[((size_t)iz * kTabNC + kTabNC - 1 - l) * xr.size() + (size_t)ir * kTabNC + k];
                    cheb_coeffs(kTabNC, kTabNC, T, T, cell.data(),
                                tab.data() + kTabPolarWords + ((size_t)iz * kTabNCell + ir) * kTabCellWords + (size_t)f * nc);
                }
    }
    // rings: the same four functions, rows in powers of u
    for (int q = 0; q < kRings; ++q) {
        const int fr = ring_fit_r(q), fa = ring_fit_a(q), nu = ring_nu(q);
        const std::vector<double> P = cheb_to_powers(nu), Tr = cheb_weights(fr), Ta = cheb_weights(fa);
        std::vector<double> full((size_t)fr * fa), vals((size_t)fr * fa);
        const std::vector<double>* src[4] = {&hB, &hC, &hE0, &hE1};
        for (int f = 0; f < 4; ++f) {
            for (int k = 0; k < fr; ++k)
                for (int l = 0; l < fa; ++l) vals[(size_t)k * fa + l] = (*src[f])[ring_at[q] + (size_t)l * fr + k];
            cheb_coeffs(fr, fa, Tr, Ta, vals.data(), full.data());
            for (int m = 0; m < nu; ++m)
                for (int j = 0; j < ring_nv(q, m >= ring_head(q)); ++j) {
                    double a = 0.0;
                    for (int i = m; i < nu; ++i)
                        if (j < ring_nv(q, i >= ring_head(q))) a += P[(size_t)i * nu + m] * full[(size_t)i * fa + j];
                    const int head = 4 * ring_head_tiles(q), tail = m >= head;
                    tab[frag_at(ring_frags(q, tail), ring_nv(q, tail), 4 * (m - (tail ? head : 0)) + f, j)] = a;
                }
        }
    }
    e = upload_wave_constants(ctx, mono.data());
    if (e != cudaSuccess) {
        cleanup();
        cudaFree(d_tab);
        return set_err(ctx, MH_ERR_CUDA, "Delhommeau constants: %s", cudaGetErrorString(e));
    }
    e = cudaMemcpyAsync(d_tab, tab.data(), sizeof(double) * kTabAllWords, cudaMemcpyHostToDevice,
                        ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cleanup();
    if (e != cudaSuccess) {
        cudaFree(d_tab);
        return set_err(ctx, MH_ERR_CUDA, "Delhommeau table upload: %s", cudaGetErrorString(e));
    }
    ctx->delh_table = d_tab;
    return MH_OK;
}

const double* delh_table_for(mh_ctx* ctx, uint32_t mask, int* status)
{
    *status = MH_OK;
    if (!(mask & MH_GF_DELHOMMEAU) || ctx->delh_method == MH_DELHOMMEAU_EXACT) return nullptr;
    *status = ensure_delh_table(ctx);
    return ctx->delh_table;
}

cudaError_t launch_wave_term(mh_ctx* ctx, const double* tab, uint32_t which, int64_t n,
                             const double* r, const double* z, double* out)
{
    k_wave_term<<<(unsigned)((n + 127) / 128), 128, 0, ctx->stream>>>(tab, which, n, r, z, out);
    ctx->launches += 1;
    return cudaGetLastError();
}

}  // namespace mh
