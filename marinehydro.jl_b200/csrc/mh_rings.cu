// The frequency-batched tabulated Delhommeau pass past the polar patch.
#include <cuda_runtime.h>

#include "mh_rings.cuh"
#include "mh_wave.cuh"

namespace mh {
namespace {

// The frequencies at which a pair is in ring q, as k_wave_delh_allw: the alpha
// contraction once per pair that has a frequency in the ring, everything in
// FP64.  Exits at once when none was flagged (fall[q]).  A CTA
// lists the tile's pairs in the ring first and works through the list densely:
// rows next to each other differ in distance, so nearly every warp has some
// pair in the ring and a third to a half of its pairs.  A pair on an edge
// between rings may be written by two kernels and keeps the later one's value.
// One kernel per ring, so that each holds the shared memory its own rows need
// (29, 35 or 45 KB a CTA, with 8 KB for k, the rows and the list).
// Evaluating each point from the Cartesian cells instead (what this replaces)
// gathers 288 coefficients per thread from cells that differ between the
// threads of a warp, on top of exp, log, J0 and J1 per point.  Measured, us:
// cells -> this, N 2997, 24 frequencies, R below 3.4: 5806 -> 1786; two bodies,
// N 1456, 32 frequencies, R below 7: 2049 -> 747; N 870, 16 frequencies, R below
// 2.7: 258 -> 152, and its tangent (mh_jvp.cu) 424 -> 185.
constexpr int kRT = 64;  // threads (rows) per CTA
constexpr size_t ring_smem(int q) { return sizeof(double) * (3 * kAllwMaxFreqs + 4 * ring_nu(q) * kRT); }

template <int q>
__global__ void __launch_bounds__(kRT, q == 0 ? 6 : q == 1 ? 5 : 4)
k_wave_delh_ring(int* __restrict__ fall, const double* __restrict__ geom, int64_t n, int direct, int cols,
                 const double* __restrict__ tab, const double* __restrict__ kvec, int nb,
                 const double* __restrict__ SR, const double* __restrict__ DR, double2* __restrict__ S64, double2* __restrict__ D64,
                 float2* __restrict__ Dlo, double2* __restrict__ tape)
{
    if (fall[q] == 0) return;
    extern __shared__ double wsm[];
    double* logk = wsm;
    double* invk = logk + kAllwMaxFreqs;
    double* ksm = invk + kAllwMaxFreqs;
    double* w = ksm + kAllwMaxFreqs;  // [4 * NU][kRT]
    __shared__ Panel sp[kRingCols];
    __shared__ double xs[6][kRT];  // collocation points and their normals
    __shared__ unsigned short list[kRingCols * kRT];
    __shared__ int count;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        ksm[t] = kvec[t];
        logk[t] = log(kvec[t]);
        invk[t] = 1.0 / kvec[t];
    }
    __syncthreads();
    double kmax = 0.0;
    for (int z = 0; z < nb; ++z) kmax = fmax(kmax, ksm[z]);
    const int64_t nn = n * n;
    const int64_t j0 = (int64_t)blockIdx.y * cols, i0 = (int64_t)blockIdx.x * kRT;
    if (threadIdx.x == 0) count = 0;
    stage_panels(sp, geom, n, j0, cols);
    for (int c = 0; c < 6; ++c) xs[c][threadIdx.x] = geom[c * n + min(i0 + threadIdx.x, n - 1)];  // G_CX .. G_NZ
    __syncthreads();
    ring_list<kRT, q>(ksm, nb, kmax, cols, list, &count, fall, [&](int row, int c) {
        const Panel& p = sp[c];
        const double dx = xs[0][row] - p.c[0], dy = xs[1][row] - p.c[1], zeta = xs[2][row] + p.c[2];
        if (i0 + row >= n || j0 + c >= n) return -2.0;
        return -zeta >= 0.0 ? sqrt(dx * dx + dy * dy + zeta * zeta) : -1.0;
    });
    __syncthreads();
    const int total = count;
    constexpr int kZP = 4;  // frequencies per Horner pass
    for (int t0 = 0; t0 < total; t0 += kRT) {
        const bool mine = t0 + (int)threadIdx.x < total;
        const int item = list[min(t0 + (int)threadIdx.x, total - 1)], row = item % kRT, c = item / kRT;
        const Panel& p = sp[c];
        const int64_t o = (j0 + c) * n + i0 + row;
        const double dx = xs[0][row] - p.c[0], dy = xs[1][row] - p.c[1];
        // pair geometry (abstract_greens_function.jl:111-131 at k = 1)
        const double dis2 = dx * dx + dy * dy, purt = 1e-18;
        const double rho = (dis2 == 0.0) ? sqrt(dis2 + purt * purt) - purt : sqrt(dis2);
        const double zeta = xs[2][row] + p.c[2], az = -zeta;
        const double d = hypot(rho, zeta);
        ring_contract<kRT, q>(tab, 4.0 * atan2(rho, az) / kPi - 1.0, w);
        const double lp = log(0.5 * (d + az));
        const double gp = rho / (d * (d + az));
        const double inv_d2 = 2.0 / d;
        const AllwPair pair =
            allw_pair(dx, dy, rho, p.area, SR[o], DR[o], direct ? p.n[0] : xs[3][row], direct ? p.n[1] : xs[4][row],
                      direct ? p.n[2] : xs[5][row], direct, o);
        for (int z0 = 0; z0 < nb; z0 += kZP) {
            double R[kZP], val[kZP][4];
            bool in[kZP], any = false;
#pragma unroll
            for (int t = 0; t < kZP; ++t) {
                R[t] = ksm[min(z0 + t, nb - 1)] * d;
                in[t] = mine && z0 + t < nb && ring_in(q, R[t]);
                any |= in[t];
            }
            if (!__any_sync(0xffffffffu, any)) continue;
            ring_values<kRT, kZP, q>(w, R, val);
#pragma unroll
            for (int t = 0; t < kZP; ++t) {
                if (!in[t]) continue;
                const int z = z0 + t;
                const double ik = invk[z], L = logk[z] + lp;
                const double B = val[t][0], C = val[t][1], E0 = val[t][2], E1 = val[t][3];
                const double e0 = -2.0 * E0, e1 = 2.0 * E1;
                const double G_re = e0 * L + B, G_im = 2.0 * kPi * E0;
                cplx o3[3];
                o3[0] = mk(G_re, G_im);
                o3[1] = mk(fma(e1, L, fma(e0, gp * ik, C)), -2.0 * kPi * E1);
                o3[2] = mk(fma(inv_d2, ik, G_re), G_im);
                allw_emit(pair, z, ksm[z], o3, nn, S64, D64, Dlo, tape);
            }
        }
    }
}

template <int q>
cudaError_t launch_ring(const Batch& bt, const double* tab, const double* d_k, int m, const double* SR, const double* DR,
                        double2* S64, double2* D64, float2* Dlo, double2* tape, int* fall)
{
    const cudaError_t e = cudaFuncSetAttribute(k_wave_delh_ring<q>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)ring_smem(q));
    if (e != cudaSuccess) return e;
    const int cols = ring_cols(bt.n);
    k_wave_delh_ring<q><<<dim3((unsigned)((bt.n + kRT - 1) / kRT), (unsigned)((bt.n + cols - 1) / cols)), kRT, ring_smem(q), bt.ctx->stream>>>(
        fall, bt.m->geom, bt.n, bt.direct, cols, tab, d_k, m, SR, DR, S64, D64, Dlo, tape);
    bt.ctx->launches += 1;
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_wave_rings(const Batch& bt, const double* tab, const double* d_k, int m, const double* SR,
                              const double* DR, double2* S64, double2* D64, float2* Dlo, double2* tape, int* fall)
{
    cudaError_t e = launch_ring<0>(bt, tab, d_k, m, SR, DR, S64, D64, Dlo, tape, fall);
    if (e == cudaSuccess) e = launch_ring<1>(bt, tab, d_k, m, SR, DR, S64, D64, Dlo, tape, fall);
    if (e == cudaSuccess) e = launch_ring<2>(bt, tab, d_k, m, SR, DR, S64, D64, Dlo, tape, fall);
    return e;
}

}  // namespace mh
