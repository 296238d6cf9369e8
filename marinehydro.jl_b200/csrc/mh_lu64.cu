// FP64 complex solve A X = B with partial pivoting for one matrix of moderate
// order: the calls for one frequency (forces, solve).  The FP64 batches and their
// adjoints keep cuSOLVER, whose factors the adjoint solves with again.  B rides
// along as further columns.  Small orders with few of them are all k_lu64_whole's, in
// one CTA (whole_most); else panels of kW columns, and per panel
//   k_lu64_panel   one CTA factors the panel in shared memory and records the row
//                  exchanges as a gather;
//   k_lu64_update  a CTA takes kC columns to the right (of A, then of B): gathers
//                  the exchanged rows, U12 = inv(L11) A12 by shuffles, A22 -= L21 U12;
// then k_lu64_back, a CTA per column of B, substitutes back.  The pivot is the
// entry of largest |re| + |im|, as in LAPACK's zgetrf; left of a panel nothing is
// exchanged, since L is not used again.  A zero pivot is refused, and so is a column
// without a number left where infinite entries (of A, or by overflow) brought that
// about; a NaN in A goes through to the solution.
// What bounds it: n dependent pivot searches (about 1 us each with the update of
// the panel's other columns in one CTA, 1.7 with 800 rows).  Measured, us, cuSOLVER's
// zgetrf and zgetrs -> this, one right-hand side: n 24 118 -> 29, 50 157 -> 69, 100 263
// -> 192, 200 505 -> 396, 400 1104 -> 859, 800 2673 -> 2124, 1000 3344 -> 2940, 1200 4533
// -> 3921.
#include <cuda_runtime.h>

#include <algorithm>

#include "mh_internal.h"

namespace mh {
namespace {

constexpr int kW = 16;              // panel columns
constexpr int kC = 8;               // columns per CTA of the update
constexpr int kSub = 4;             // panel columns eliminated before the others take their products
constexpr int kPanelThreads = 512;
constexpr int kUpdThreads = 256;
constexpr int kBackThreads = 512;
constexpr int kBlk = 32;            // rows per step of the back substitution
// Right-hand sides up to which one CTA does everything: its time grows with them (a
// CTA's threads walk all columns), the panels' hardly does.  us for the call's
// kernels, it and the panels: n 8, 32 right-hand sides 37 and 44; 32, 32 73 and 81, 48
// 84 and 82; 40, 24 101 and 104, 32 112 and 105; 50, 1 84 and 117, 16 102 and 118, 32
// 134 and 129, 64 180 and 126; 64, 12 128 and 135, 24 157 and 142; 72, 8 155 and 156;
// 80, 1 155 and 165, 6 173 and 166; 96, 1 200 and 197, 32 329 and 205.
constexpr int whole_most(int64_t n) { return n <= 32 ? 40 : n <= 86 ? (int)(88 - n) / 2 : n < 96; }

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// c - a b
__device__ __forceinline__ double2 cfms(double2 c, double2 a, double2 b)
{
    return make_double2(fma(-a.x, b.x, fma(a.y, b.y, c.x)), fma(-a.x, b.y, fma(-a.y, b.x, c.y)));
}
// 1 / a, scaled by a power of two near 1 / |a|: no overflow or underflow of |a|^2
__device__ __forceinline__ double2 cinv(double2 a)
{
    const int e = __double2hiint(fmax(fabs(a.x), fabs(a.y))) >> 20;  // biased exponent
    const double s = __hiloint2double((2046 - max(1, min(2045, e))) << 20, 0);
    const double x = a.x * s, y = a.y * s, d = s / fma(x, x, y * y);
    return make_double2(x * d, -y * d);
}

// Shared memory: the panel by columns, rows k0 .. n - 1, then which row of it
// stands in each; and the panel's width, fewer columns where the rows are many.
size_t panel_smem(int64_t rows, int w) { return (size_t)rows * (w * sizeof(double2) + sizeof(int)); }
constexpr size_t kPanelSmemMax = 226 * 1024;
int panel_width(int64_t rows)
{
    int w = (int)std::min<int64_t>(kW, rows);
    while (w > 4 && panel_smem(rows, w) > kPanelSmemMax) --w;
    return w;
}

// The largest of the warp's big >= 0 (its bits as an integer's, in two halves; -1
// where a lane has none) and a lane that has it.
__device__ __forceinline__ int warp_best(double& big)
{
    const unsigned hi = big < 0.0 ? 0u : (unsigned)__double2hiint(big) + 1u;
    const unsigned top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == top ? (unsigned)__double2loint(big) : 0u;
    const unsigned low = __reduce_max_sync(0xffffffffu, lo);
    big = top ? __hiloint2double((int)(top - 1u), (int)low) : -1.0;
    return __ffs(__ballot_sync(0xffffffffu, hi == top && lo == low)) - 1;
}

// gather: 2 kW pairs (to, from), rows of the matrix: where every row that moved,
// or is at the panel's top, comes from.  Steps of kSub columns, their products then
// applied to the panel's others in one pass: tall panels are bound by their traffic
// with shared memory (all columns updated at every step: 1630 us for 1347 at n 800,
// 142 for 120 at 100).  In a step two barriers per column: the pivot row is set
// aside, then every row is updated (old row j into the pivot's place) and looks for
// the next column's pivot on the way.
__global__ void __launch_bounds__(kPanelThreads)
k_lu64_panel(double2* __restrict__ A, int n, int k0, int w, int2* __restrict__ gather, int* __restrict__ info)
{
    extern __shared__ double2 p[];
    const int rows = n - k0, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    int* perm = reinterpret_cast<int*>(p + (size_t)rows * w);
    __shared__ double best[kPanelThreads / 32];
    __shared__ int where[kPanelThreads / 32];
    __shared__ int moved[kW];
    __shared__ double2 u[kSub];  // the pivot row in the step's columns
    double2* M = A + (int64_t)k0 * n + k0;
    double big = -1.0;
    int at = 0;
    for (int r = tid; r < rows; r += blockDim.x) {
        perm[r] = r;
#pragma unroll 4
        for (int c = 0; c < w; ++c) p[c * rows + r] = M[(int64_t)c * n + r];
        const double m = fabs(p[r].x) + fabs(p[r].y);
        if (m > big) {
            big = m;
            at = r;
        }
    }
    for (int j0 = 0; j0 < w; j0 += kSub) {
        const int e = min(j0 + kSub, w);
        for (int j = j0; j < e; ++j) {
            {
                const int from = warp_best(big);
                if (lane == from) {
                    best[warp] = big;
                    where[warp] = at;
                }
            }
            __syncthreads();  // also: the rows are updated
            big = lane < warps ? best[lane] : -1.0;
            at = lane < warps ? where[lane] : j;
            at = __shfl_sync(0xffffffffu, at, warp_best(big));
            if (!(big >= 0.0)) at = j;  // no number in the column
            const double2 piv = p[j * rows + at], ip = cinv(piv);
            if (tid < w) {
                const double2 t = p[tid * rows + at];
                if (tid >= j && tid < e) {
                    u[tid - j0] = t;
                } else {  // L and the columns past the step's are exchanged now
                    p[tid * rows + at] = p[tid * rows + j];
                    p[tid * rows + j] = t;
                }
            }
            if (tid == 0) {
                const int t = perm[j];
                perm[j] = perm[at];
                perm[at] = t;
                moved[j] = at;
                if (!(big > 0.0)) atomicCAS(info, 0, big == 0.0 ? k0 + j + 1 : -(k0 + j + 1));
            }
            __syncthreads();
            const int pr = at;
            big = -1.0;
            at = j + 1;
            for (int r = tid; r < rows; r += blockDim.x) {
                if (r < j || r == pr) continue;
                const int to = r == j ? pr : r;
                const double2 l = cmul(p[j * rows + r], ip);
                p[j * rows + to] = l;
                double2 a[kSub];
#pragma unroll
                for (int i = 1; i < kSub; ++i)
                    if (j + i < e) a[i] = p[(j + i) * rows + r];
#pragma unroll
                for (int i = 1; i < kSub; ++i)
                    if (j + i < e) {
                        a[i] = cfms(a[i], l, u[j + i - j0]);
                        p[(j + i) * rows + to] = a[i];
                    }
                if (j + 1 < e) {
                    const double m = fabs(a[1].x) + fabs(a[1].y);
                    if (m > big) {
                        big = m;
                        at = to;
                    }
                }
                if (r == j)
                    for (int c = j; c < e; ++c) p[c * rows + j] = u[c - j0];
            }
        }
        if (e == w) break;
        __syncthreads();  // the step's columns are final
        if (tid >= e && tid < w) {  // its rows of U, a thread per column
            double2* col = p + tid * rows + j0;
#pragma unroll
            for (int i = 1; i < kSub; ++i) {
                double2 t = col[i];
                for (int m = 0; m < i; ++m) t = cfms(t, p[(j0 + m) * rows + j0 + i], col[m]);
                col[i] = t;
            }
        }
        __syncthreads();
        big = -1.0;
        at = e;
        for (int r = tid; r < rows; r += blockDim.x) {
            if (r < e) continue;
            double2 l[kSub];
#pragma unroll
            for (int m = 0; m < kSub; ++m) l[m] = p[(j0 + m) * rows + r];
            for (int c = e; c < w; c += 2) {
                const bool two = c + 1 < w;
                double2* c0 = p + c * rows;
                double2* c1 = two ? c0 + rows : c0;
                double2 a0 = c0[r], a1 = c1[r], u0[kSub], u1[kSub];
#pragma unroll
                for (int m = 0; m < kSub; ++m) {
                    u0[m] = c0[j0 + m];
                    u1[m] = c1[j0 + m];
                }
#pragma unroll
                for (int m = 0; m < kSub; ++m) {
                    a0 = cfms(a0, l[m], u0[m]);
                    a1 = cfms(a1, l[m], u1[m]);
                }
                c0[r] = a0;
                if (two) c1[r] = a1;
                if (c == e) {
                    const double m = fabs(a0.x) + fabs(a0.y);
                    if (m > big) {
                        big = m;
                        at = r;
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int r = tid; r < rows; r += blockDim.x)
#pragma unroll 4
        for (int c = 0; c < w; ++c) M[(int64_t)c * n + r] = p[c * rows + r];
    if (tid < w) {
        gather[tid] = make_int2(k0 + tid, k0 + perm[tid]);
        gather[kW + tid] = make_int2(k0 + moved[tid], k0 + perm[moved[tid]]);
    }
}

// The whole solve in one CTA: the columns of A and B as one panel (ld n), the rows
// on `rows` threads (a multiple of 32, at least n) times blockDim / rows groups,
// each with every such group's fours of columns.  As k_lu64_panel otherwise, but
// neither L nor the exchanges are kept; then U x = y, a barrier a column.
__global__ void __launch_bounds__(kPanelThreads)
k_lu64_whole(const double2* __restrict__ A, double2* __restrict__ B, int n, int nrhs, int rows, int* __restrict__ info)
{
    extern __shared__ double2 p[];  // [n + nrhs][n]
    const int W = n + nrhs, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int r = tid % rows, group = tid / rows, groups = blockDim.x / rows;
    double2* u = p + (size_t)W * n;  // the pivot row, [W + 3]
    double2* dinv = u + W + 3;       // 1 / u_jj, [n]
    __shared__ double best[kPanelThreads / 32];
    __shared__ int where[kPanelThreads / 32];
    if (r < n)
        for (int c = group; c < W; c += groups)
            p[c * n + r] = c < n ? A[(int64_t)c * n + r] : B[(int64_t)(c - n) * n + r];
    __syncthreads();
    double big = r < n && group == 0 ? fabs(p[r].x) + fabs(p[r].y) : -1.0;
    if (!(big >= 0.0)) big = -1.0;
    int at = r;
    for (int j = 0; j < n; ++j) {
        {
            const int from = warp_best(big);
            if (lane == from) {
                best[warp] = big;
                where[warp] = at;
            }
        }
        __syncthreads();  // also: the rows are updated
        big = lane < warps ? best[lane] : -1.0;
        at = lane < warps ? where[lane] : j;
        at = __shfl_sync(0xffffffffu, at, warp_best(big));
        if (!(big >= 0.0)) at = j;  // no number in the column
        const double2 piv = p[j * n + at], ip = cinv(piv);
        for (int c = j + tid; c < W; c += blockDim.x) u[c] = p[c * n + at];
        if (tid == 0 && !(big > 0.0)) atomicCAS(info, 0, big == 0.0 ? j + 1 : -(j + 1));
        __syncthreads();
        const int pr = at;
        big = -1.0;
        at = j + 1;
        if (r >= j && r < n) {
            const int to = r == j ? pr : r;
            const double2 l = cmul(p[j * n + r], ip);
            for (int c = j + 1 + 4 * group; c < W; c += 4 * groups) {
                if (r != pr) {
                    double2 a[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (c + i < W) a[i] = p[(c + i) * n + r];
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[i] = cfms(a[i], l, u[c + i]);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (c + i < W) p[(c + i) * n + to] = a[i];
                    if (c == j + 1) {
                        const double m = fabs(a[0].x) + fabs(a[0].y);
                        if (m >= 0.0) {
                            big = m;
                            at = to;
                        }
                    }
                }
                if (r == j)
                    for (int i = 0; i < 4; ++i)
                        if (c + i < W) p[(c + i) * n + j] = u[c + i];
            }
        }
        if (tid == 0) dinv[j] = ip;
    }
    __syncthreads();
    for (int j = n - 1; j >= 0; --j) {
        const double2 inv = dinv[j];
        for (int q = group; q < nrhs; q += groups) {
            double2* y = p + (n + q) * n;
            const double2 x = cmul(y[j], inv);
            if (r < j) y[r] = cfms(y[r], p[j * n + r], x);
            if (r == j) B[(int64_t)q * n + j] = x;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kUpdThreads)
k_lu64_update(double2* __restrict__ A, double2* __restrict__ B, int n, int nrhs, int k0, int w,
              const int2* __restrict__ gather)
{
    __shared__ double2 top[kW][kC], l11[kW][kW + 1];
    const int right = n - k0 - w, tid = threadIdx.x;
    const auto column = [&](int c) {  // column c right of the panel, null past the last
        const int q = (int)blockIdx.x * kC + c;
        return q < right ? A + (int64_t)(k0 + w + q) * n : q < right + nrhs ? B + (int64_t)(q - right) * n : nullptr;
    };
    static_assert(kUpdThreads == 2 * kW * kC && kW * kW == kUpdThreads, "one gathered entry and one of L11 per thread");
    {
        const int e = tid % (2 * kW), c = tid / (2 * kW);
        double2* col = column(c);
        const bool live = col && e % kW < w;
        const int2 g = live ? gather[e] : make_int2(0, 0);
        const double2 v = live ? col[g.y] : make_double2(0.0, 0.0);
        const int i = tid % kW, m = tid / kW;
        l11[i][m] = m < i && i < w ? A[(int64_t)(k0 + m) * n + k0 + i] : make_double2(0.0, 0.0);
        __syncthreads();  // every gathered row is read
        if (e < kW) top[e][c] = v;
        else if (live && g.x >= k0 + w) col[g.x] = v;
    }
    __syncthreads();
    if (tid < kW * kC) {  // U12: a column per half warp, a row per lane
        const int i = tid % kW, c = tid / kW, base = tid & 16;
        double2 t = top[i][c];
#pragma unroll
        for (int m = 0; m < kW - 1; ++m) {
            const double2 u = make_double2(__shfl_sync(0xffffffffu, t.x, base + m), __shfl_sync(0xffffffffu, t.y, base + m));
            if (i > m) t = cfms(t, l11[i][m], u);  // not by its zeros: an infinite entry is to stay one
        }
        top[i][c] = t;
        double2* col = column(c);
        if (col && i < w) col[k0 + i] = t;
    }
    __syncthreads();
    for (int r = k0 + w + tid; r < n; r += kUpdThreads) {
        double2 l[kW];
#pragma unroll
        for (int m = 0; m < kW; ++m) l[m] = m < w ? A[(int64_t)(k0 + m) * n + r] : make_double2(0.0, 0.0);
        double2 a[kC];
#pragma unroll
        for (int c = 0; c < kC; ++c) {
            const double2* col = column(c);
            a[c] = col ? col[r] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int m = 0; m < kW; ++m)
#pragma unroll
            for (int c = 0; c < kC; ++c) a[c] = cfms(a[c], l[m], top[m][c]);
#pragma unroll
        for (int c = 0; c < kC; ++c) {
            double2* col = column(c);
            if (col) col[r] = a[c];
        }
    }
}

// U x = y in place, a CTA per column of B.  The next diagonal block is fetched
// while this one is solved.
__global__ void __launch_bounds__(kBackThreads)
k_lu64_back(const double2* __restrict__ A, double2* __restrict__ B, int n)
{
    extern __shared__ double2 x[];  // [n]
    __shared__ double2 u[kBlk][kBlk + 1];
    double2* col = B + (int64_t)blockIdx.x * n;
    const int tid = threadIdx.x;
    constexpr int kE = kBlk * kBlk / kBackThreads;
    double2 f[kE];
    const auto fetch = [&](int k) {
#pragma unroll
        for (int e = 0; e < kE; ++e) {
            const int i = (e * kBackThreads + tid) % kBlk, j = (e * kBackThreads + tid) / kBlk;
            f[e] = k >= 0 && k + j < n && i <= j ? A[(int64_t)(k + j) * n + k + i]
                                                 : make_double2(i == j ? 1.0 : 0.0, 0.0);
        }
    };
    int k = (n - 1) / kBlk * kBlk;
    fetch(k);
    for (int r = tid; r < n; r += kBackThreads) x[r] = col[r];
    for (; k >= 0; k -= kBlk) {
        const int w = min(kBlk, n - k);
#pragma unroll
        for (int e = 0; e < kE; ++e) u[(e * kBackThreads + tid) % kBlk][(e * kBackThreads + tid) / kBlk] = f[e];
        __syncthreads();  // also x
        fetch(k - kBlk);
        if (tid < kBlk) {
            double2 t = tid < w ? x[k + tid] : make_double2(0.0, 0.0);
            const double2 inv = cinv(u[tid][tid]);
#pragma unroll 4
            for (int j = kBlk - 1; j >= 0; --j) {
                double2 v = cmul(t, inv);
                v = make_double2(__shfl_sync(0xffffffffu, v.x, j), __shfl_sync(0xffffffffu, v.y, j));
                t = tid == j ? v : tid < j ? cfms(t, u[tid][j], v) : t;
            }
            if (tid < w) x[k + tid] = t;
        }
        __syncthreads();
        for (int r = tid; r < k; r += kBackThreads) {
            double2 t = x[r];
            for (int j0 = 0; j0 < w; j0 += 16) {
                double2 a[16];
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    a[j] = j0 + j < w ? A[(int64_t)(k + j0 + j) * n + r] : make_double2(0.0, 0.0);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (j0 + j < w) t = cfms(t, a[j], x[k + j0 + j]);
            }
            x[r] = t;
        }
        __syncthreads();
    }
    for (int r = tid; r < n; r += kBackThreads) col[r] = x[r];
}

// found: 1 a NaN, 2 an entry that is infinite and no NaN.
__global__ void k_lu64_scan(const double2* __restrict__ A, int64_t count, int* __restrict__ found)
{
    int f = 0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
        const double2 a = A[t];
        if (isnan(a.x) || isnan(a.y)) f |= 1;
        else if (isinf(a.x) || isinf(a.y)) f |= 2;
    }
    if (f) atomicOr(found, f);
}

}  // namespace

// What it takes: where it beats cuSOLVER.  By the order as above; by the right-hand
// sides since its products of A22 and B are not as fast as the library's.  us, cuSOLVER and
// it, 768 and 1500 of them: n 50 186 and 159, 188 and 220; 400 1592 and 1287, 1664 and
// 1817; 800 3804 and 3413, 4046 and 4565; 1200 6447 and 6428, 7032 and 8776.
bool lu64_takes(int64_t n, int64_t nrhs) { return n <= 1200 && nrhs <= 768; }

// info[0]: the first column (from 1) with a zero pivot, or minus the first without a
// number, 0 for none.  A holds the factors, or (whole) what came in: in the factors an
// infinite entry stays in its row of U, so a NaN that came in leaves none behind.
static int lu64_status(mh_ctx* ctx, int64_t n, const double2* A, bool whole, int* info)
{
    MH_CUDA_TRY(ctx, cudaGetLastError());
    int h = 0;
    MH_CUDA_TRY(ctx, cudaMemcpyAsync(&h, info, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    MH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    if (h < 0) {
        int found = 0;
        MH_CUDA_TRY(ctx, cudaMemsetAsync(info + 1, 0, sizeof(int), ctx->stream));
        k_lu64_scan<<<(unsigned)std::min<int64_t>((n * n + 255) / 256, 592), 256, 0, ctx->stream>>>(A, n * n, info + 1);
        ctx->launches += 1;
        MH_CUDA_TRY(ctx, cudaMemcpyAsync(&found, info + 1, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        MH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        const bool came_in = whole ? (found & 1) != 0 : (found & 2) == 0;
        h = came_in && n > 1 ? 0 : -h;
    }
    if (h > 0) return set_err(ctx, MH_ERR_SINGULAR, "zero pivot at column %d", h);
    return MH_OK;
}

// A X = B, A overwritten, X in place of B; MH_ERR_SINGULAR at a zero pivot.
int lu64_solve(mh_ctx* ctx, int64_t n, double2* A, double2* B, int nrhs)
{
    auto* gather = (int2*)ws_get(ctx, WS_PIV, sizeof(int2) * 2 * kW);
    auto* info = (int*)ws_get(ctx, WS_INFO, sizeof(int) * 2);
    if (!gather || !info) return MH_ERR_OOM;
    MH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu64_panel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kPanelSmemMax));
    MH_CUDA_TRY(ctx, cudaMemsetAsync(info, 0, sizeof(int), ctx->stream));
    if (nrhs <= whole_most(n)) {
        MH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_lu64_whole, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kPanelSmemMax));
        const size_t whole = sizeof(double2) * ((size_t)(n + nrhs) * (size_t)n + (size_t)(2 * n + nrhs + 3));
        const int rows = (int)(n + 31) / 32 * 32, groups = kPanelThreads / rows;
        k_lu64_whole<<<1, rows * groups, whole, ctx->stream>>>(A, B, (int)n, nrhs, rows, info);
        ctx->launches += 1;
        return lu64_status(ctx, n, A, true, info);
    }
    for (int64_t k0 = 0; k0 < n;) {
        const int w = panel_width(n - k0);
        const int threads = (int)std::min<int64_t>(kPanelThreads, (n - k0 + 31) / 32 * 32);
        k_lu64_panel<<<1, threads, panel_smem(n - k0, w), ctx->stream>>>(A, (int)n, (int)k0, w, gather, info);
        const int64_t cols = n - k0 - w + nrhs;
        k_lu64_update<<<(unsigned)((cols + kC - 1) / kC), kUpdThreads, 0, ctx->stream>>>(A, B, (int)n, nrhs, (int)k0, w,
                                                                                       gather);
        ctx->launches += 2;
        k0 += w;
    }
    k_lu64_back<<<nrhs, kBackThreads, sizeof(double2) * (size_t)n, ctx->stream>>>(A, B, (int)n);
    ctx->launches += 1;
    return lu64_status(ctx, n, A, false, info);
}

}  // namespace mh
