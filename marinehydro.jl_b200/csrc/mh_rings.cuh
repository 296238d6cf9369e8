// Rings of the tabulated Guevel-Delhommeau wave term past the polar patch
// (mh_table.cuh): ring q covers R in [2^(q+1), 2^(q+2)) and all alpha, for the
// kernels that evaluate many frequencies of one panel pair.  Per function
// (B, C, E0, E1), row m holds the coefficient of u^m, u = (2 R - lo - hi) /
// (hi - lo), as a Chebyshev series in v(alpha); coefficients below 1e-14 in
// all four are dropped; the first ring_head rows keep ring_nv(q, 0) of them and
// the others ring_nv(q, 1) (row lengths fall from 25 to 3 in the first ring).
// Error against the quadrature ~5e-14.
// The coefficients sit in constant memory, which broadcasts the one that every
// thread of a warp reads; one copy per translation unit that includes this,
// written when a context builds its table (every context writes the same).
// 2997 panels x 24 frequencies, us: 7265 with the coefficients read from global
// memory (two 16-byte loads per column bound it), 4294 from constant memory
// with a loop of its own length for every row, 4004 with these fixed lengths, 2414
// with the pairs listed first (mh_rings.cu), 2232 with the Chebyshev values in
// registers instead of Clenshaw's recurrence.
#pragma once
#include "mh_internal.h"
#include "mh_device.cuh"

namespace mh {

constexpr int kRings = 3;
constexpr double kRingMax = 16.0;  // end of the last ring
constexpr int kRingCols = 8;         // source columns per CTA of the ring kernels, at most
constexpr __host__ __device__ int ring_fit_r(int q) { return q == 0 ? 24 : q == 1 ? 28 : 36; }  // fit nodes in R
constexpr __host__ __device__ int ring_fit_a(int q) { return q == 0 ? 36 : q == 1 ? 40 : 56; }  // and in alpha
constexpr __host__ __device__ int ring_nu(int q) { return q == 0 ? 14 : q == 1 ? 17 : 22; }     // rows
constexpr __host__ __device__ int ring_head(int q) { return q == 0 ? 8 : q == 1 ? 9 : 12; }     // rows of full length
constexpr __host__ __device__ int ring_nv(int q, int tail)                                      // columns
{
    return tail ? (q == 0 ? 19 : q == 1 ? 24 : 29) : (q == 0 ? 25 : q == 1 ? 30 : 36);
}
// column of row m's first coefficient in the packed table
constexpr __host__ __device__ int ring_at(int q, int m)
{
    const int h = ring_head(q), head = (m < h ? m : h) * ring_nv(q, 0), tail = (m > h ? m - h : 0) * ring_nv(q, 1);
    return (q ? ring_at(q - 1, ring_nu(q - 1)) : 0) + head + tail;
}

// The packed rings: coefficient (row m, column j, function f) of ring q at
// 4 (ring_at(q, m) + j) + f.
struct RingTable {
    double coef[4 * ring_at(kRings - 1, ring_nu(kRings - 1))];
};

static __constant__ RingTable c_rings;

// Whether R belongs to ring q, with margins of 1e-12 that let a pair on an edge
// be written by one kernel at least, whatever the rounding of R in each.
__device__ __forceinline__ bool ring_in(int q, double R)
{
    const double lo = q == 0 ? 2.0 : q == 1 ? 4.0 : 8.0;
    return R >= lo * (1.0 - 1e-12) && R < 2.0 * lo * (1.0 + 1e-12);
}

// Rows m0 .. m1 - 1 of ring q (of NV columns each) contracted with t[j] = T_j(v).
template <int T, int q, int NV, int m0, int m1, int N>
__device__ __forceinline__ void ring_contract_rows(const double (&t)[N], double* __restrict__ w)
{
#pragma unroll 1
    for (int row = m0; row < m1; ++row) {
        const int c = 4 * (ring_at(q, m0) + (row - m0) * NV);
        double b[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int col = 0; col < NV; ++col)
#pragma unroll
            for (int f = 0; f < 4; ++f) b[f] = fma(c_rings.coef[c + 4 * col + f], t[col], b[f]);
#pragma unroll
        for (int f = 0; f < 4; ++f) w[(4 * row + f) * T] = b[f];
    }
}

// The alpha direction of ring q contracted at v: w[(4 row + f) T], f = B, C,
// E0, E1, the coefficients of u^row (T threads' columns side by side).
template <int T, int q>
__device__ __forceinline__ void ring_contract(double v, double* __restrict__ w)
{
    double t[ring_nv(q, 0)];
    cheb_values(v, t);
    ring_contract_rows<T, q, ring_nv(q, 0), 0, ring_head(q)>(t, w);
    ring_contract_rows<T, q, ring_nv(q, 1), ring_head(q), ring_nu(q)>(t, w);
}

// The four functions at Z values of R in ring q, from its contraction.
template <int T, int Z, int q>
__device__ __forceinline__ void ring_values(const double* __restrict__ w, const double R[Z], double val[Z][4])
{
    constexpr double kInvLo = q == 0 ? 0.5 : q == 1 ? 0.25 : 0.125;
    double u[Z];
#pragma unroll
    for (int t = 0; t < Z; ++t) u[t] = 2.0 * kInvLo * R[t] - 3.0;  // hi = 2 lo
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const double c = w[(4 * (ring_nu(q) - 1) + f) * T];
#pragma unroll
        for (int t = 0; t < Z; ++t) val[t][f] = c;
    }
#pragma unroll 2
    for (int row = ring_nu(q) - 2; row >= 0; --row)
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const double c = w[(4 * row + f) * T];
#pragma unroll
            for (int t = 0; t < Z; ++t) val[t][f] = fma(val[t][f], u[t], c);
        }
}

// Lists the pairs of a tile (T rows by cols columns) that have a frequency in
// ring q: entry col * T + row, in no particular order.  ksm: the frequencies'
// k, kmax the largest.  Call it with all T threads, then synchronise.
// dist(row, col) gives d, -1 for a pair without a polar angle, -2 for one outside
// the matrix.  The first ring's pass, which sees every pair, flags what the later
// rings (fall[1], fall[2]) and the full table (fall[kRings]) have to do.
template <int T, int q, class Dist>
__device__ __forceinline__ void ring_list(const double* ksm, int nb, double kmax, int cols, unsigned short* list,
                                          int* count, int* fall, Dist dist)
{
    const int lane = threadIdx.x & 31;
    double top = 0.0;  // largest R
    for (int c = 0; c < cols; ++c) {
        const double d = dist((int)threadIdx.x, c), R = kmax * d;
        bool mine = false;
        if (__any_sync(0xffffffffu, R >= (q == 0 ? 2.0 : q == 1 ? 4.0 : 8.0) * (1.0 - 1e-12)))
            for (int z = 0; z < nb; ++z) mine = mine || ring_in(q, ksm[z] * d);
        if (q == 0) top = d >= 0.0 ? fmax(top, R) : d == -2.0 ? top : INFINITY;
        const unsigned vote = __ballot_sync(0xffffffffu, mine);
        if (!vote) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(count, __popc(vote));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (mine) list[at + __popc(vote & ((1u << lane) - 1u))] = (unsigned short)(c * T + threadIdx.x);
    }
    if (q == 0) {
        if (top >= 4.0 * (1.0 - 1e-12)) fall[1] = 1;
        if (top >= 8.0 * (1.0 - 1e-12)) fall[2] = 1;
        if (top >= kRingMax * (1.0 - 1e-12)) fall[kRings] = 1;
    }
}

// Source columns per CTA of 64 rows in the ring kernels: 8 at most, so that a
// list fills its warps, fewer where that leaves under 1500 CTAs.  (Fewer CTAs,
// each taking several tiles in turn, lost a third to imbalance: a tile's pairs
// are all in the ring or none of them.)
inline int ring_cols(int64_t n)
{
    int c = kRingCols;
    while (c > 1 && ((n + 63) / 64) * ((n + c - 1) / c) < 1500) c /= 2;
    return c;
}

}  // namespace mh
