// Rings of the tabulated Guevel-Delhommeau wave term past the polar patch
// (mh_table.cuh): ring q covers R in [2^(q+1), 2^(q+2)) and all alpha, for the
// kernels that evaluate many frequencies of one panel pair.  Per function
// (B, C, E0, E1), row m holds the coefficient of u^m, u = (2 R - lo - hi) /
// (hi - lo), as a Chebyshev series in v(alpha); coefficients below 1e-14 in
// all four are dropped; the first ring_head rows keep ring_nv(q, 0) of them and
// the others ring_nv(q, 1) (row lengths fall from 25 to 3 in the first ring).
// Error against the quadrature ~5e-14.
// 2997 panels x 24 frequencies, us: 7265 with the coefficients read from global
// memory a thread at a time (two 16-byte loads per column bound it), 4004 from
// constant memory, 2414 with the pairs listed first (mh_rings.cu), 2232 with the
// Chebyshev values in registers instead of Clenshaw's recurrence, 1786 with the
// matrix instruction (mh_contract.cuh).
// The polar patch has the same form for these kernels: its rows in powers of
// u = 2 R / kTabRPolar - 1.  After the alpha contraction each function is a
// degree-14 polynomial in u whose coefficients sum to less than 6 in absolute
// value (the Chebyshev coefficients decay faster than the basis change grows
// them), so Horner's rule in u is as accurate as Clenshaw's recurrence and takes
// one FMA per term instead of two operations.
#pragma once
#include "mh_internal.h"
#include "mh_device.cuh"
#include "mh_contract.cuh"

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
// The fragments (mh_contract.cuh) follow the table's cells: the polar patch, then
// each ring's tiles with a row of full length and its others.
constexpr int kFragPolar = kTabWords;
constexpr __host__ __device__ int ring_head_tiles(int q) { return frag_tiles(ring_head(q)); }
constexpr __host__ __device__ int ring_frags(int q, int tail)  // first word
{
    return tail ? ring_frags(q, 0) + frag_words(ring_head(q), ring_nv(q, 0))
         : q    ? ring_frags(q - 1, 1) + frag_words(ring_nu(q - 1) - 4 * ring_head_tiles(q - 1), ring_nv(q - 1, 1))
                : kFragPolar + frag_words(kTabNU, kTabNV);
}
constexpr int kTabAllWords = ring_frags(kRings, 0);

// Whether R belongs to ring q, with margins of 1e-12 that let a pair on an edge
// be written by one kernel at least, whatever the rounding of R in each.
__device__ __forceinline__ bool ring_in(int q, double R)
{
    const double lo = q == 0 ? 2.0 : q == 1 ? 4.0 : 8.0;
    return R >= lo * (1.0 - 1e-12) && R < 2.0 * lo * (1.0 + 1e-12);
}

// The alpha direction of ring q contracted at the warp's 32 v: w[w_at<T>(4 row +
// f, column)], f = B, C, E0, E1, the coefficients of u^row.  The whole warp takes
// part; it writes the columns of its own threads only.
template <int T, int q>
__device__ __forceinline__ void ring_contract(const double* __restrict__ tab, double v, double* __restrict__ w)
{
    constexpr int kHead = ring_head_tiles(q), kTail = frag_tiles(ring_nu(q) - 4 * kHead);
    const int base = threadIdx.x & ~31;
    const auto store = [&](int m, int p, double a, double b) {
        if (m < 4 * ring_nu(q)) *reinterpret_cast<double2*>(w + w_at<T>(m, base + p)) = make_double2(a, b);
    };
    __syncwarp();  // the last pairs' columns are read
#pragma unroll 1
    for (int g = 0; g < 4; g += 2) {
        double t[2][frag_steps(ring_nv(q, 0))];
        cheb_frags(v, g, t);
        contract_tiles<kHead, frag_steps(ring_nv(q, 0))>(tab + ring_frags(q, 0), g, t, store);
        contract_tiles<kTail, frag_steps(ring_nv(q, 1))>(
            tab + ring_frags(q, 1), g, t, [&](int m, int p, double a, double b) { store(16 * kHead + m, p, a, b); });
    }
    __syncwarp();
}

// The four functions at Z values of R in ring q, from the calling thread's column.
template <int T, int Z, int q>
__device__ __forceinline__ void ring_values(const double* __restrict__ w, const double R[Z], double val[Z][4])
{
    constexpr double kInvLo = q == 0 ? 0.5 : q == 1 ? 0.25 : 0.125;
    double u[Z];
#pragma unroll
    for (int t = 0; t < Z; ++t) u[t] = 2.0 * kInvLo * R[t] - 3.0;  // hi = 2 lo
    const int tid = threadIdx.x;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const double c = w[w_at<T>(4 * (ring_nu(q) - 1) + f, tid)];
#pragma unroll
        for (int t = 0; t < Z; ++t) val[t][f] = c;
    }
#pragma unroll 2
    for (int row = ring_nu(q) - 2; row >= 0; --row)
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const double c = w[w_at<T>(f, tid) + 4 * row * T];
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
