// Shared device code of the batched complex FP32 LU (pivot-free, blocked):
// the diagonal-block factorisation with inverse diagonal blocks and the
// panel triangular solves, templated on the block size NB.
//
// Layout: matrices n x n column-major float2, `stride` elements apart;
// Dinv holds, per matrix and diagonal block, inv(L11) then inv(U11), each
// NB x NB column-major.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mh {
namespace {

__device__ __forceinline__ float2 cmulf(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 csubf(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a - b*c
__device__ __forceinline__ float2 cfms(float2 a, float2 b, float2 c)
{
    return make_float2(a.x - (b.x * c.x - b.y * c.y), a.y - (b.x * c.y + b.y * c.x));
}
// the same as a chain of four fused operations
__device__ __forceinline__ float2 cfms4(float2 a, float2 b, float2 c)
{
    return make_float2(fmaf(b.y, c.y, fmaf(-b.x, c.x, a.x)), fmaf(-b.y, c.x, fmaf(-b.x, c.y, a.y)));
}
__device__ __forceinline__ float2 cdivf(float2 a, float2 b)
{
    float d = b.x * b.x + b.y * b.y;
    return make_float2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}

// Factor the diagonal block [k0, k0+kb) of every matrix in place, and store
// inv(L11) (unit lower) and inv(U11) in Dinv (per matrix: n/NB blocks of
// 2 x NB x NB, column-major) for the triangular solves.
template <int NB, int THREADS = 256>
__global__ void __launch_bounds__(THREADS)
k_lu_diag(float2* __restrict__ A, int64_t n, int64_t stride, int64_t k0, float2* __restrict__ Dinv,
          int64_t dstride, int* __restrict__ bad)
{
    extern __shared__ float2 lu_diag_smem[];
    auto s = reinterpret_cast<float2 (*)[NB + 1]>(lu_diag_smem);            // s[row][col]
    auto w = reinterpret_cast<float2 (*)[NB + 1]>(lu_diag_smem + NB * (NB + 1));  // inverse
    const int64_t b = blockIdx.x;
    float2* M = A + b * stride;
    const int kb = (int)min((int64_t)NB, n - k0);
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        int r = t % NB, c = t / NB;
        s[r][c] = (r < kb && c < kb) ? M[(k0 + c) * n + k0 + r]
                                     : make_float2(r == c ? 1.f : 0.f, 0.f);
    }
    __syncthreads();
    for (int c = 0; c < kb; ++c) {
        float2 piv = s[c][c];
        float mag = piv.x * piv.x + piv.y * piv.y;
        if (threadIdx.x == 0 && !(mag > 1e-30f && mag < 3e38f)) atomicExch(bad + b, 1);
        for (int r = c + 1 + threadIdx.x; r < kb; r += blockDim.x) s[r][c] = cdivf(s[r][c], piv);
        __syncthreads();
        int m = kb - c - 1;
        for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
            int r = c + 1 + t % m, q = c + 1 + t / m;
            s[r][q] = cfms(s[r][q], s[r][c], s[c][q]);
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < kb * kb; t += blockDim.x) {
        int r = t % kb, c = t / kb;
        M[(k0 + c) * n + k0 + r] = s[r][c];
    }
    float2* out = Dinv + b * dstride + (k0 / NB) * 2 * NB * NB;
    // inv(L11), unit lower: W = I, then for t ascending the rows below t
    // subtract L[r][t] W[t][:] (row t is final at step t); all threads per sweep.
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int r = t % NB, c = t / NB;
        w[r][c] = make_float2(r == c ? 1.f : 0.f, 0.f);
    }
    __syncthreads();
    for (int t = 0; t + 1 < kb; ++t) {
        const int wdt = t + 1, cnt = (kb - 1 - t) * wdt;
        for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
            const int r = t + 1 + e / wdt, c = e % wdt;
            w[r][c] = cfms(w[r][c], s[r][t], w[t][c]);
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) out[t] = w[t % NB][t / NB];
    __syncthreads();
    // inv(U11): W = I, then for t descending the rows above t subtract
    // U[r][t] / U[t][t] W[t][:], and finally row r is scaled by 1 / U[r][r].
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int r = t % NB, c = t / NB;
        w[r][c] = make_float2(r == c ? 1.f : 0.f, 0.f);
    }
    __syncthreads();
    if (threadIdx.x < NB) {  // the padding column of w holds 1 / U[r][r]
        const int r = threadIdx.x;
        w[r][NB] = r < kb ? cdivf(make_float2(1.f, 0.f), s[r][r]) : make_float2(1.f, 0.f);
    }
    __syncthreads();
    for (int t = kb - 1; t >= 1; --t) {
        const int wdt = kb - t, cnt = t * wdt;
        const float2 f = w[t][NB];
        for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
            const int r = e / wdt, c = t + e % wdt;
            w[r][c] = cfms(w[r][c], cmulf(s[r][t], f), w[t][c]);
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int r = t % NB, c = t / NB;
        out[NB * NB + t] = (r < kb) ? cmulf(w[r][NB], w[r][c]) : w[r][c];
    }
}

// The B operands of the tensor-core panel TRSMs of a diagonal block, packed
// once here instead of by every TRSM CTA: 128 x 128 FP16 K-major no-swizzle
// images (8-row x 16-byte core matrices), rows R < 64 = [Re v | -Im v],
// rows 64 + R = [Im v | Re v] of the complex row v = column R of inv(U11)
// (image 0, for L21 = A21 inv(U11)) or row R of inv(L11) (image 1, for
// U12^T = A12^T inv(L11)^T).  x[c][r] (column-major) holds inv(L) strictly
// below the diagonal (unit diagonal implicit) and inv(U) on and above it.
// An item reads eight entries of v (as FP16 pairs Re, Im) and writes them to the
// four places of its two rows.
constexpr int kTrsmBImage = 128 * 128 * 2;  // bytes per image

template <int LD>
__device__ __forceinline__ void pack_trsm_b(const __half2 (*x)[LD], unsigned char* img)
{
    if (threadIdx.x >= 256) return;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int e = it * 256 + threadIdx.x;
        const int im = e >> 9, r = e & 63, cc = (e >> 6) & 7, t0 = cc * 8;
        __half2 v[8];
        const __half2 zero = __floats2half2_rn(0.f, 0.f), one = __floats2half2_rn(1.f, 0.f);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int t = t0 + q;
            if (im == 0) v[q] = t <= r ? x[r][t] : zero;                // inv(U)[t][r]
            else v[q] = t == r ? one : (r > t ? x[t][r] : zero);        // inv(L)[r][t]
        }
        uint4 re, pi;  // Re v, Im v
        auto bits = [](__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); };
        auto lo = [&](int q) { return bits(__lows2half2(v[q], v[q + 1])); };
        auto hi = [&](int q) { return bits(__highs2half2(v[q], v[q + 1])); };
        re = make_uint4(lo(0), lo(2), lo(4), lo(6));
        pi = make_uint4(hi(0), hi(2), hi(4), hi(6));
        const uint4 mi = make_uint4(pi.x ^ 0x80008000u, pi.y ^ 0x80008000u, pi.z ^ 0x80008000u, pi.w ^ 0x80008000u);
        unsigned char* o = img + (size_t)im * kTrsmBImage;
        auto at = [&](int row, int chunk) {
            return reinterpret_cast<uint4*>(o + ((chunk * 16 + row / 8) * 128 + (row % 8) * 16));
        };
        *at(r, cc) = re;
        *at(r, 8 + cc) = mi;
        *at(64 + r, cc) = pi;
        *at(64 + r, 8 + cc) = re;
    }
}

// k_lu_diag for NB = 64: factors and both triangular inverses in one blocked
// elimination, the whole block in registers.  A step takes the eight rows and
// columns K of a panel.  With the pivot block X_KK = L_K U_K,
//   c_iK = X_iK inv(U_K)  for every row i outside K: L below K, and above K
//                         the final columns K of inv(U);
//   R_Kj = inv(L_K) X_Kj  for every column j outside K: U right of K, and left
//                         of K the final rows K of inv(L).
// These four pieces leave for their places at once, and the step is one
// rank-8 update X_ij -= c_iK R_Kj of all entries, rows and columns in K
// starting from 0 with c = inv(U_K) and R = inv(L_K) there: below and right of
// K it makes the Schur complement, below and left what inv(L) needs, above and
// right what inv(U) needs; what it makes of the entries that have left is never
// read.  The pivot block is factored and inverted by the same elimination, one
// pivot at a time.
// Thread (ti, tj) of 16 x 16 holds the entries (ti + 16 a, tj + 16 b); a warp of
// its own, with a scheduler of its own, does the pivot blocks (two entries per lane,
// exchanged by shuffles), the next panel's while the others run this panel's
// update: they hand its eight rows and columns over first.  What bounds it: the 64 dependent pivot steps (a
// shuffle, a reciprocal and three products each), one CTA per matrix.
// The panel loop is not unrolled: with the panel as a compile-time index the
// code, run once, missed the instruction cache for a third of the time.
// The block is padded with the identity, so all panels run for any kb <= 64.
// Same outputs as k_lu_diag.  28 KB of shared memory, so that a CTA fits beside
// two CTAs of the trailing update on an SM.
// Measured on a B200: 44 us (panels of eight by one warp, then the inverses by
// recursive doubling: 36 barriers) -> 25 us a block (26 with the pivot warp on a
// scheduler that two others use); 64 matrices of 2048 beside their updates, 60 -> 37
// us.
constexpr int kDiag64Threads = 320;

__global__ void __launch_bounds__(kDiag64Threads)
k_lu_diag64(float2* __restrict__ A, int64_t n, int64_t stride, int64_t k0, float2* __restrict__ Dinv,
            int64_t dstride, int* __restrict__ bad, unsigned char* __restrict__ bimg, int64_t bstride)
{
    constexpr int NB = 64, kLd = 65, kPad = NB + 1;  // odd leading dimensions: no bank conflicts down a column
    __shared__ float2 c[8][kPad];  // c[m][i]: X_iK, then c_iK (row i in K: inv(U_K))
    __shared__ float2 r[8][kPad];  // r[m][j]: X_Kj, then R_Kj (column j in K: inv(L_K))
    __shared__ __align__(16) float2 iu[8][8];  // iu[t][m] = inv(U_K)[t][m], zero for t > m
    __shared__ __align__(16) float2 il[8][8];  // il[t][m] = inv(L_K)[m][t], 1 for t = m, zero for t > m
    __shared__ float2 pv[8][8];                // the next pivot block
    __shared__ float2 prow[8][8], pcol[8][8];  // its row k before step k, c of step k
    __shared__ __half2 hx[NB][kLd];            // hx[col][row]: the inverses as FP16 pairs
    const int64_t b0 = blockIdx.x;
    float2* M = A + b0 * stride + k0 * n + k0;
    float2* invL = Dinv + b0 * dstride + (k0 / NB) * 2 * NB * NB;
    float2* invU = invL + NB * NB;
    const int kb = (int)min((int64_t)NB, n - k0);
    // warps 0, 1, 2, 4, 5, 6, 8, 9 hold the block, warp 3 does the pivot blocks with
    // a scheduler of its own, warp 7 is not used
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tid = 32 * (warp - warp / 4) + lane, ti = tid & 15, tj = tid >> 4;
    const bool pivots = (warp & 3) == 3;
    const float2 z = make_float2(0.f, 0.f), one = make_float2(1.f, 0.f);
    float2 X[4][4];
    if (!pivots) {
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int i = ti + 16 * a, j = tj + 16 * b;
                X[a][b] = (i < kb && j < kb) ? M[(int64_t)j * n + i] : i == j ? one : z;
                if (i < j) invL[j * NB + i] = z;
                if (i > j) invU[j * NB + i] = z;
            }
        if (ti < 8 && tj < 8) pv[ti][tj] = X[0][0];
    }
    bool poor = false;
    __syncthreads();
#pragma unroll 1
    for (int K = -8; K < NB; K += 8) {
        if (pivots) {
            const int N = K + 8;  // the panel after K
            if (warp == 3 && N < NB) {
                // lane (i, g) holds the entries (i, g) and (i, g + 4) of the pivot block
                const int i = lane & 7, g = lane >> 3;
                float2 x[2] = {pv[i][g], pv[i][4 + g]};
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int ek = k >> 2, gk = k & 3;
                    auto from = [](float2 v, int src) {
                        return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
                    };
                    const float2 p = from(x[ek], 8 * gk + k), xk = from(x[ek], 8 * gk + i);
                    float2 pr[2] = {from(x[0], 8 * g + k), from(x[1], 8 * g + k)};
                    const float mag = fmaf(p.x, p.x, p.y * p.y);
                    const float im2 = 1.f / mag;
                    const float2 ip = make_float2(p.x * im2, -p.y * im2);
                    float2 ck = cmulf(xk, ip);
                    ck.x = i == k ? ip.x : ck.x;
                    ck.y = i == k ? ip.y : ck.y;
                    pcol[k][i] = ck;
                    if (i == k) {
                        prow[k][g] = x[0];
                        prow[k][g + 4] = x[1];
                    }
                    const bool own = g == gk;  // column k itself: 0 - c
                    pr[ek].x = own ? 1.f : pr[ek].x;
                    pr[ek].y = own ? 0.f : pr[ek].y;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const bool zero = i == k || (e == ek && own);
                        x[e].x = zero ? 0.f : x[e].x;
                        x[e].y = zero ? 0.f : x[e].y;
                        x[e] = cfms4(x[e], ck, pr[e]);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int j = g + 4 * e;
                    const float2 pc = pcol[j][i], pw = prow[i][j];  // i > j: L, inv(L); i <= j: inv(U), U
                    iu[i][j] = i <= j ? pc : z;
                    il[j][i] = i > j ? pw : i == j ? one : z;
                    if (N + i < kb && N + j < kb) M[(int64_t)(N + j) * n + N + i] = i > j ? pc : pw;
                    const float2 inv = i > j ? pw : pc;
                    (i > j ? invL : invU)[(N + j) * NB + N + i] = inv;
                    if (i == j) {
                        const float mag = fmaf(pw.x, pw.x, pw.y * pw.y);  // the pivot
                        poor = poor || (N + i < kb && !(mag > 1e-30f && mag < 3e38f));
                        invL[(N + j) * NB + N + i] = one;
                    }
                    hx[N + j][N + i] = __floats2half2_rn(inv.x, inv.y);
                }
            }
        } else if (K >= 0) {
#pragma unroll 2
            for (int m = 0; m < 8; ++m) {
                float2 cv[4], rv[4];
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    cv[a] = c[m][ti + 16 * a];
                    rv[a] = r[m][tj + 16 * a];
                }
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int a = 0; a < 4; ++a) X[a][b] = cfms4(X[a][b], cv[a], rv[b]);
            }
        }
        if (K + 8 >= NB) break;
        __syncthreads();  // c and r are read; the next pivot block's inverses are there
        const int N = K + 8;
        // a thread holds row N + (ti & 7) in a = nq, column N + (tj & 7) in b = nq
        const int nq = N >> 4, h = (N >> 3) & 1;
        const bool row_n = !pivots && (ti >> 3) == h, col_n = !pivots && (tj >> 3) == h;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q == nq) {
                if (row_n)
#pragma unroll
                    for (int b = 0; b < 4; ++b) r[ti & 7][tj + 16 * b] = X[q][b];
                if (col_n)
#pragma unroll
                    for (int a = 0; a < 4; ++a) c[tj & 7][ti + 16 * a] = X[a][q];
            }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if ((a == nq && row_n) || (b == nq && col_n)) X[a][b] = z;
        __syncthreads();
        // c (threads 0 .. 127) and R (128 .. 255): index eq, entries 4 mh .. 4 mh + 3, in place (a pair of lanes per index)
        const int eq = (tid >> 1) & 63, mh = tid & 1;
        const bool is_c = tid < 128;
        float2 acc[4] = {z, z, z, z};
        if (!pivots) {
            float2 (*v)[kPad] = is_c ? c : r;
            const float4* tab = reinterpret_cast<const float4*>(is_c ? &iu[0][0] : &il[0][0]) + 2 * mh;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const float2 x = make_float2(-v[t][eq].x, -v[t][eq].y);
                const float4 u0 = tab[4 * t], u1 = tab[4 * t + 1];
                acc[0] = cfms4(acc[0], x, make_float2(u0.x, u0.y));
                acc[1] = cfms4(acc[1], x, make_float2(u0.z, u0.w));
                acc[2] = cfms4(acc[2], x, make_float2(u1.x, u1.y));
                acc[3] = cfms4(acc[3], x, make_float2(u1.z, u1.w));
            }
            __syncwarp();
            if ((eq & ~7) == N) {  // in the panel: the operand itself
                const float4 u0 = tab[4 * (eq & 7)], u1 = tab[4 * (eq & 7) + 1];
                acc[0] = make_float2(u0.x, u0.y);
                acc[1] = make_float2(u0.z, u0.w);
                acc[2] = make_float2(u1.x, u1.y);
                acc[3] = make_float2(u1.z, u1.w);
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) v[4 * mh + s][eq] = acc[s];
        }
        __syncthreads();
        // the pivot block after this panel, updated ahead of the rest
        const int P = N + 8;
        if (!pivots && P < NB && (ti >> 3) == ((P >> 3) & 1) && (tj >> 3) == ((P >> 3) & 1)) {
            const int pq = P >> 4;
            float2 x = pq == 0 ? X[0][0] : pq == 1 ? X[1][1] : pq == 2 ? X[2][2] : X[3][3];
#pragma unroll
            for (int m = 0; m < 8; ++m) x = cfms4(x, c[m][ti + 16 * pq], r[m][tj + 16 * pq]);
            pv[ti & 7][tj & 7] = x;
        }
        __syncthreads();
        if (!pivots && (eq & ~7) != N) {
            // c and R to their places while the next pivot block is factored: past the panel the factors (L by
            // columns, U by rows), before it the inverses
            const bool past = eq >= N + 8;
            const int nin = N + 4 * mh;
            float2* out = past ? (is_c ? M + (int64_t)nin * n + eq : M + (int64_t)eq * n + nin)
                               : (is_c ? invU + nin * NB + eq : invL + eq * NB + nin);
            const int64_t step = is_c ? (past ? n : (int64_t)NB) : 1;
            const int live = !past ? 4 : eq < kb ? min(4, kb - nin) : 0;
#pragma unroll
            for (int s = 0; s < 4; ++s)
                if (s < live) out[s * step] = acc[s];
            if (!past)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    (is_c ? hx[nin + s][eq] : hx[eq][nin + s]) = __floats2half2_rn(acc[s].x, acc[s].y);
        }
    }
    if (poor) atomicExch(bad + b0, 1);
    __syncthreads();
    if (bimg) pack_trsm_b<kLd>(hx, bimg + b0 * bstride + (k0 / NB) * 2 * kTrsmBImage);
}

// blockIdx.y == 0: rows of L21 = A21 U11^-1; blockIdx.y == 1: columns of
// U12 = L11^-1 A12.  blockIdx.z = matrix.
template <int NB>
__global__ void __launch_bounds__(128)
k_lu_trsm(float2* __restrict__ A, int64_t n, int64_t stride, int64_t k0)
{
    __shared__ float2 s[NB][NB + 1];
    float2* M = A + (int64_t)blockIdx.z * stride;
    const int kb = (int)min((int64_t)NB, n - k0);
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        int r = t % NB, c = t / NB;
        s[r][c] = (r < kb && c < kb) ? M[(k0 + c) * n + k0 + r] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int64_t idx = k0 + kb + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    float2 v[NB];
    if (blockIdx.y == 0) {
        // row idx: x U11 = a  ->  x_c = (a_c - sum_{t<c} x_t u_tc) / u_cc
#pragma unroll
        for (int c = 0; c < NB; ++c) v[c] = (c < kb) ? M[(k0 + c) * n + idx] : make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < NB; ++c) {
            if (c < kb) {
                float2 acc = v[c];
#pragma unroll
                for (int t = 0; t < c; ++t) acc = cfms(acc, v[t], s[t][c]);
                v[c] = cdivf(acc, s[c][c]);
            }
        }
#pragma unroll
        for (int c = 0; c < NB; ++c)
            if (c < kb) M[(k0 + c) * n + idx] = v[c];
    } else {
        // column idx: L11 y = a (unit lower)  ->  y_r = a_r - sum_{t<r} l_rt y_t
        const float2* col = M + idx * n + k0;
#pragma unroll
        for (int r = 0; r < NB; ++r) v[r] = (r < kb) ? col[r] : make_float2(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < NB; ++r) {
            if (r < kb) {
                float2 acc = v[r];
#pragma unroll
                for (int t = 0; t < r; ++t) acc = cfms(acc, s[r][t], v[t]);
                v[r] = acc;
            }
        }
        float2* colw = M + idx * n + k0;
#pragma unroll
        for (int r = 0; r < NB; ++r)
            if (r < kb) colw[r] = v[r];
    }
}


// Dynamic shared memory of k_lu_diag<NB>.
template <int NB>
constexpr size_t lu_diag_smem_bytes() { return sizeof(float2) * 2 * NB * (NB + 1); }

}  // namespace
}  // namespace mh
