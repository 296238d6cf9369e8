// The alpha contraction of the frequency-batched Delhommeau kernels: for the 32
// pairs of a warp, w[m] = sum_j A[m][j] T_j(v), m = 4 row + function (B, C, E0,
// E1), j the Chebyshev degree in v(alpha), A the same for every pair.  A matrix
// product, done with the FP64 m16n8k4 matrix instruction: one instruction where
// the vector form takes 16 FMAs and 16 loads of their coefficients, which bound
// it (its issue slots, not the FP64 units, were full).  A sits in the table's
// buffer as the fragments the instruction takes, zero past its rows and columns,
// one coalesced 16-byte load a step.  Measured, us, one FMA per term with the
// coefficient in constant memory -> this: the first ring 2232 -> 1786 (2997 panels
// x 24 frequencies), 215 -> 152 (870 x 16) and its tangent 258 -> 185; the polar
// patch, whose output bounds it more, 1957 -> 1936 (2048 x 64), 206 -> 179 (870 x
// 16) and its tangent 413 -> 383, no change at 2997 x 24 (2215, 2208 to 2268).
#pragma once
#include <cuda_runtime.h>

namespace mh {

// Fragments of an A of 4 rows x 4 functions a tile and 4 columns a step: tile i,
// step s at 64 (i STEPS + s) doubles, lane l's pair there {A[m][j], A[m + 8][j]},
// m = 16 i + l / 4, j = 4 s + l % 4.
constexpr __host__ __device__ int frag_tiles(int rows) { return (rows + 3) / 4; }
constexpr __host__ __device__ int frag_steps(int cols) { return (cols + 3) / 4; }
constexpr __host__ __device__ int frag_words(int rows, int cols) { return 64 * frag_tiles(rows) * frag_steps(cols); }

__device__ __forceinline__ void mma_f64(double (&c)[4], double2 a, double b)
{
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a.x), "d"(a.y), "d"(b));
}

// A warp's pairs are contracted G groups of 8 at a time: 2 hide the instruction's
// latency better, 1 takes fewer registers (us for 1 and 2: the 2048 x 64 patch 1927
// and 2014, the first ring at 2997 x 24 1912 and 1787).
// The other operand for the groups g0 .. g0 + G - 1: t[g][s] = T_j(v of lane 8 (g0 +
// g) + l / 4), j = 4 s + l % 4, by T_{j+4} = 2 T_4 T_j - T_{|j-4|}.  The whole warp
// takes part.
template <int G, int STEPS>
__device__ __forceinline__ void cheb_frags(double v, int g0, double (&t)[G][STEPS])
{
    const int lane = threadIdx.x & 31, r = lane & 3;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const double x = __shfl_sync(0xffffffffu, v, 8 * (g0 + g) + (lane >> 2));
        const double t2 = fma(2.0 * x, x, -1.0), t3 = fma(2.0 * x, t2, -x), f = 2.0 * fma(2.0 * x, t3, -t2);
        double before = r == 0 ? 0.5 * f : r == 1 ? t3 : r == 2 ? t2 : x;
        t[g][0] = r == 0 ? 1.0 : r == 1 ? x : r == 2 ? t2 : t3;
#pragma unroll
        for (int s = 1; s < STEPS; ++s) {
            t[g][s] = fma(f, t[g][s - 1], -before);
            before = t[g][s - 1];
        }
    }
}

// store(m, pair, w[m] of lane pair, w[m] of lane pair + 1) for all m < 16 TILES and
// the pairs of t's groups, from the first STEPS steps of t.
template <int TILES, int STEPS, int G, int N, class Store>
__device__ __forceinline__ void contract_tiles(const double* __restrict__ frags, int g0,
                                               const double (&t)[G][N], Store store)
{
    const int lane = threadIdx.x & 31;
    const double2* a = reinterpret_cast<const double2*>(frags) + lane;
#pragma unroll 1
    for (int i = 0; i < TILES; ++i) {
        double c[G][4] = {};
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            const double2 f = __ldg(a + 32 * (i * STEPS + s));
#pragma unroll
            for (int g = 0; g < G; ++g) mma_f64(c[g], f, t[g][s]);
        }
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                store(16 * i + 8 * h + (lane >> 2), 8 * (g0 + g) + 2 * (lane & 3), c[g][2 * h], c[g][2 * h + 1]);
    }
}

// w[m * T + column], T columns (threads) of FP64 values, the columns of odd m
// exchanged in eights so that the 16-byte stores of contract_tiles' eight rows
// meet no bank twice.
template <int T>
__device__ __forceinline__ int w_at(int m, int column)
{
    return m * T + (column ^ (8 * (m & 1)));
}

}  // namespace mh
