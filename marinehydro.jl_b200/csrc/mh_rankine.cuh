// The frequency-independent Rankine terms of all panel pairs (rankine.jl,
// rankine_reflected*.jl), by tiles of 128 collocation rows x C source columns.
//
// One term of a pair costs about 60 FP64 operations in the far field and
// some 1500 (four edges, each with a logarithm, an arc tangent and its
// gradient) within seven panel radii.  Near pairs are a few percent of a fine
// mesh but sit in one warp in five, so a thread that walks its pairs in
// order holds its warp for the near ones of its neighbours, and 16 pairs in
// series were 220 us of latency on any mesh.  Here the first pass writes the
// far field and lists the tile's near (pair, term) items in shared memory, the
// second takes the list densely, one item per thread, and the third adds the
// two terms (in term order, so the list's order does not matter) and stores;
// the FP64 assembly adds its wave term there, in the same launch.
// C = 4 columns where that makes eight CTAs per SM, one column below.
// Measured on a B200, us, 16 pairs in series per thread -> now:
//   Rankine parts: N 200 226 -> 12, 870 260 -> 58, 1456 302 -> 106, 2048 347
//   -> 164, 2997 529 -> 308; their tangent, N 870: 249 -> 77; FP64 assembly
//   with Wu's term: N 50 262 -> 14, 570 297 -> 81, 800 337 -> 97.
#pragma once
#include "mh_device.cuh"
#include "mh_internal.h"

namespace mh {

constexpr int kRkRows = 128;

// Fields f of panel j, and collocation point and normal of row i, as T.
struct RankineGeom {
    const double* geom;
    int64_t n;
    __device__ __forceinline__ void field(int f, int64_t j, double& v) const { v = geom[(int64_t)f * n + j]; }
};

template <class T, int C, class In, class Out>
__global__ void __launch_bounds__(kRkRows)
k_rankine_tile(In in, int64_t n, uint32_t mask, int direct, Out out)
{
    __shared__ PanelT<T> sp[C];
    __shared__ T xs[6][kRkRows];                    // collocation points, their normals
    __shared__ double part[2][2][C][kRkRows];       // [term][S or D]
    __shared__ unsigned short list[2 * C * kRkRows];
    __shared__ int count;
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t i = (int64_t)blockIdx.x * kRkRows + tid, j0 = (int64_t)blockIdx.y * C;
    if (tid == 0) count = 0;
    for (int t = tid; t < C * G_NFIELDS; t += kRkRows) {
        const int f = t / C, jj = t % C;
        T v;
        in.field(f, min(j0 + jj, n - 1), v);
        PanelT<T>& p = sp[jj];
        if (f < 3) p.c[f] = v;
        else if (f < 6) p.n[f - 3] = v;
        else if (f == G_AREA) p.area = v;
        else if (f == G_RADIUS) p.radius = v;
        else p.v[f - G_V] = v;
    }
    for (int c = 0; c < 6; ++c) in.field(c, min(i, n - 1), xs[c][tid]);  // G_CX .. G_NZ are fields 0 .. 5
    __syncthreads();
    const uint32_t refl = mask & (MH_GF_RANKINE_REFLECTED | MH_GF_RANKINE_REFLECTED_NEGATIVE);
    const bool has[2] = {(mask & MH_GF_RANKINE) != 0,
                         refl == MH_GF_RANKINE_REFLECTED || refl == MH_GF_RANKINE_REFLECTED_NEGATIVE};
    const double sgn = refl == MH_GF_RANKINE_REFLECTED_NEGATIVE ? -1.0 : 1.0;  // of the reflected term
    const double sg = direct ? 1.0 : -1.0;                                     // gradient with respect to the source, or the point
    // S and D parts of one term: its integral, and its gradient along the normal of D
    auto put = [&](int term, int jj, int row, const T& I, const T g[3]) {
        const PanelT<T>& p = sp[jj];
        const double a = term ? sgn : 1.0, az = term ? sg : 1.0;  // the reflected point's z derivative changes sign with x's
        T dn;
        if (direct) dn = p.n[0] * g[0] + p.n[1] * g[1] + az * (p.n[2] * g[2]);
        else dn = xs[3][row] * g[0] + xs[4][row] * g[1] + az * (xs[5][row] * g[2]);
        part[term][0][jj][row] = Out::take(a * I);
        part[term][1][jj][row] = Out::take((a * sg) * dn);
    };
    auto point = [&](int term, int row, T x[3]) {
        x[0] = xs[0][row];
        x[1] = xs[1][row];
        x[2] = term ? -xs[2][row] : xs[2][row];
    };
#pragma unroll 1
    for (int q = 0; q < 2 * C; ++q) {
        const int jj = q >> 1, term = q & 1;
        bool near = false;
        if (has[term]) {
            T x[3], I, g[3];
            point(term, tid, x);
            near = !rankine_far(x, sp[jj], I, g);
            if (!near) put(term, jj, tid, I, g);
        } else {
            part[term][0][jj][tid] = part[term][1][jj][tid] = 0.0;
        }
        near = near && i < n && j0 + jj < n;
        const unsigned vote = __ballot_sync(0xffffffffu, near);
        if (vote) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&count, __popc(vote));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (near) list[base + __popc(vote & ((1u << lane) - 1u))] = (unsigned short)(q * kRkRows + tid);
        }
    }
    __syncthreads();
    for (int t = tid; t < count; t += kRkRows) {
        const int q = list[t] / kRkRows, row = list[t] % kRkRows;
        T x[3], I, g[3];
        point(q & 1, row, x);
        rankine_near(x, sp[q >> 1], I, g);
        put(q & 1, q >> 1, row, I, g);
    }
    __syncthreads();
    if (i >= n) return;
#pragma unroll 1
    for (int jj = 0; jj < C && j0 + jj < n; ++jj)
        out.store((j0 + jj) * n + i, i == j0 + jj, part[0][0][jj][tid] + part[1][0][jj][tid],
                  part[0][1][jj][tid] + part[1][1][jj][tid], xs, tid, sp[jj]);
}

template <class T, class In, class Out>
cudaError_t launch_rankine_tile(mh_ctx* ctx, const In& in, int64_t n, uint32_t mask, int direct, const Out& out)
{
    const auto cd = [](int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); };
    const unsigned rows = cd(n, kRkRows);
    if ((int64_t)rows * cd(n, 4) >= 8 * 148)
        k_rankine_tile<T, 4, In, Out><<<dim3(rows, cd(n, 4)), kRkRows, 0, ctx->stream>>>(in, n, mask, direct, out);
    else
        k_rankine_tile<T, 1, In, Out><<<dim3(rows, (unsigned)n), kRkRows, 0, ctx->stream>>>(in, n, mask, direct, out);
    ctx->launches += 1;
    return cudaGetLastError();
}

// Source columns per CTA of 128 rows in the wave-term kernels (at most
// most), batch grids of them: the fewer columns, the more CTAs; 5000 (eleven
// waves of three per SM) keep the last wave small, and a CTA of one column still
// amortises the staging of its panel.  16 columns for every mesh left 26 CTAs
// for 200 panels: the frequency-batched Delhommeau pass, us, 16 columns ->
// this rule: N 200, 20 frequencies 199 -> 25; 870, 16 304 -> 231; 1456, 32
// 930 -> 811; 2048, 64 2457 -> 2376; 2997, 24 3162 -> 3073.
inline int wave_cols(int64_t n, int most, int64_t batch = 1)
{
    int c = most;
    while (c > 1 && ((n + kRkRows - 1) / kRkRows) * ((n + c - 1) / c) * batch < 5000) c /= 2;
    return c;
}

}  // namespace mh
