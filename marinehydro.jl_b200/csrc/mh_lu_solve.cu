// Triangular solves with the block-64 factors of launch_lu_tc: one thread-block
// cluster per matrix, every solved block handed to the cluster's CTAs through
// distributed shared memory.
//
// Row block i of both triangles belongs to CTA i mod cs of its matrix's cluster
// of cs CTAs.  Left-looking: x_i = b_i - sum_j T_ij y_j accumulates in registers
// over the blocks j before i in the triangle's order, then y_i = inv(T_ii) x_i.
// The owner's threads store y_i straight into the y table of every CTA of the
// cluster (st.async), and each store counts on that CTA's mbarrier of block i, so
// a CTA waits for a block on its own shared memory and reads it there: a step of
// the chain is one tile product, one inverse product and one hand-off, 2 us in
// all.  (Published through global memory, with a flag per block and a copy of y_j
// back into shared memory, a step took 5.3 us, and 8 to 13 us for odd n or more
// than four right-hand sides.)  With many matrices the shared-memory bandwidth of
// a tile bounds it (written, read and multiplied from there, 512 of some 700
// cycles).  us a solve, through global memory -> this: 2048 x 64 matrices with 3
// right-hand sides 498 -> 419, 2997 x 24 with 2 778 -> 375, 1456 x 32 with 3 214 -> 141,
// 2048 x 1 with 3 342 -> 138, 1224 x 16 with 8 513 -> 163.
// Where the right-hand sides' table of all blocks does not fit a CTA's shared memory
// in fewer passes, a CTA keeps the blocks it solved itself (kOwn): it publishes one
// by an arrival at every CTA of the cluster, and a warp of each fetches the y_j of
// every tile from its owner's shared memory into the tile's stage.  Any order then
// takes up to eight right-hand sides a pass: us a solve of 12,240 with 4 of them, the
// table of all blocks in four passes 13,160, this 3825, the streamed kernel through
// global memory 10,060; of 20,604 with 1 and 3, a right-looking kernel with flags in
// global memory 34,800 and 57,400, this 7240 and 8910, the streamed one 18,900 and 25,300.
// Every operand a CTA reads is known in advance (its blocks' tiles in order, each
// block followed by its inverse diagonal block), so four producer warps stream them
// through a ring of shared-memory stages with cp.async (16 bytes a copy where n is
// even, 8 otherwise; entries past the matrix are zero-filled) while eight consumer
// warps multiply, and the tile stream runs ahead of the chain.
// Cluster size: the most CTAs a matrix (up to 8, one per row block) that let all
// clusters run at once; a CTA's ring takes an SM's shared memory, and a second wave
// of clusters would double the chain.  A cluster lives in one GPC, so fewer fit than
// the SMs would hold: the runtime says how many (us a solve at 800 panels with 4
// right-hand sides, the SMs counted and this: 16 to 18 matrices 121 and 61, 23 and 24
// 119 and 63, 34 to 37 130 and 77, 38 to 45 98 and 78, the others as they were).
//
// Every wait is bounded: a stage wait that runs out marks the matrix in `bad` (2),
// a wait for a block marks it (3) and later blocks are not waited for; every block
// is still stored to every CTA, and the cluster leaves together once all stores
// have landed.  Failure injection (unset_flag): the first wait for another CTA's
// block polls a flag that nothing publishes.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "mh_internal.h"

namespace mh {
namespace {

constexpr int kScNB = 64;
constexpr int kScLd = 66;  // staged column stride in float2: 16-byte columns, the consumers' reads conflict-free
constexpr size_t kScTileBytes = sizeof(float2) * kScNB * kScLd;
constexpr int kScConsumers = 256;
constexpr int kScProducers = 4;                // producer warps (after eight consumer warps), columns dealt among them
constexpr int sc_threads(bool own) { return kScConsumers + 32 * (kScProducers + own); }
constexpr int kScMaxStages = 4;
constexpr size_t kScSmemMax = 226 * 1024;      // per CTA (227 KB less the barriers' alignment)
constexpr uint32_t kScWaitNs = 50000000;       // bounded waits: 50 ms of the global timer ...
constexpr uint32_t kScWaitHintNs = 1000;       // ... in polls that suspend at most ~1 us
constexpr int kScInjectPolls = 64;

// y table (own: of the CTA's blocks only), x_i of the block being solved (two of them,
// in turn), stages (own: with the y that a tile multiplies), barriers
size_t sc_smem(bool own, int cs, int64_t nblk, int nq, int stages)
{
    const int64_t blocks = own ? (nblk + cs - 1) / cs + stages : nblk;
    return sizeof(float2) * (size_t)(blocks + 2) * nq * kScNB + (size_t)stages * kScTileBytes +
           sizeof(uint64_t) * (size_t)(2 * kScMaxStages + 2 * nblk + 1);
}

__device__ __forceinline__ uint32_t sc_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void sc_init(uint64_t* bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(sc_smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ bool sc_try(uint32_t a, uint32_t phase)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(a), "r"(phase), "r"(kScWaitHintNs)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool sc_wait(uint64_t* bar, uint32_t phase)
{
    const uint32_t a = sc_smem_u32(bar);
    for (int it = 0; it < 8; ++it)  // the timer is read only where a wait is long
        if (sc_try(a, phase)) return true;
    uint32_t t0, t;  // the timer's low word: differences are exact across its 4.3 s wrap
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t0));
    do {
        if (sc_try(a, phase)) return true;
        asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    } while (t - t0 <= kScWaitNs);
    return false;
}

__device__ __forceinline__ bool sc_unset(const int* flag)  // failure injection: a wait on a flag that nothing publishes
{
    int v = 0, it = 0;
    do asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    while (v == 0 && ++it < kScInjectPolls);
    return v != 0;
}

__device__ __forceinline__ uint32_t sc_map(uint32_t addr, int rank)  // the same place in another CTA of the cluster
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void sc_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Block bi (in the triangle's order) of the CTA of this rank.
__device__ __forceinline__ int sc_own(int tri, int nown, int rank, int cs, int bi)
{
    return rank + cs * (tri == 0 ? bi : nown - 1 - bi);
}

// Partial sums of four rows r0 .. r0 + 3 of (tile) (y), over the lane's four
// columns: acc += T y.  16-byte reads of the tile (two rows of a column, or two
// columns of a row of the transposed one) touch every bank once; the y entries
// are shared by the two row groups of a warp.
template <bool kCT, int NQ>
__device__ __forceinline__ void sc_tile(const float2* __restrict__ st, const float2* __restrict__ y, int r0, int e,
                                        float2 (&acc)[4][NQ])
{
    auto add = [](float2& s, float tx, float ty, float2 v) {
        s.x = fmaf(tx, v.x, s.x);
        s.x = fmaf(-ty, v.y, s.x);
        s.y = fmaf(tx, v.y, s.y);
        s.y = fmaf(ty, v.x, s.y);
    };
    if (!kCT) {  // columns e, e + 16, ...
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int c = e + 16 * m;
            const float4 t01 = *reinterpret_cast<const float4*>(st + c * kScLd + r0);
            const float4 t23 = *reinterpret_cast<const float4*>(st + c * kScLd + r0 + 2);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float2 v = y[q * kScNB + c];
                add(acc[0][q], t01.x, t01.y, v);
                add(acc[1][q], t01.z, t01.w, v);
                add(acc[2][q], t23.x, t23.y, v);
                add(acc[3][q], t23.z, t23.w, v);
            }
        }
    } else {  // columns 2 e, 2 e + 1, 2 e + 32, 2 e + 33
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int c = 2 * e + 32 * m;
            float4 t[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) t[u] = *reinterpret_cast<const float4*>(st + (r0 + u) * kScLd + c);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(y + q * kScNB + c);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    add(acc[u][q], t[u].x, -t[u].y, make_float2(v.x, v.y));
                    add(acc[u][q], t[u].z, -t[u].w, make_float2(v.z, v.w));
                }
            }
        }
    }
}

// Sums over the 16 lanes of a row group: the first two steps halve the rows a
// lane holds (sum[q] ends as that of row 2 (e >> 3) + (e >> 2 & 1)), the others add
// up the four lanes of a row.
template <int NQ>
__device__ __forceinline__ void sc_reduce(const float2 (&acc)[4][NQ], int e, float2 (&sum)[NQ])
{
    float2 two[2][NQ];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float2 keep = e & 8 ? acc[u + 2][q] : acc[u][q], send = e & 8 ? acc[u][q] : acc[u + 2][q];
            two[u][q].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 8);
            two[u][q].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 8);
        }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const float2 keep = e & 4 ? two[1][q] : two[0][q], send = e & 4 ? two[0][q] : two[1][q];
        sum[q].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 4);
        sum[q].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 4);
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            sum[q].x += __shfl_xor_sync(0xffffffffu, sum[q].x, o);
            sum[q].y += __shfl_xor_sync(0xffffffffu, sum[q].y, o);
        }
}

// L U x = b (kCT = false) or U^H L^H x = b (true) for NQ right-hand sides, over
// X.  vec: the matrices and n allow 16-byte copies.
//
// kOwn: y_i of the second triangle replaces that of the first in its owner's table
// when nobody reads the first any more: it needs every later block's second y, whose
// owner had by then used all of the first triangle.
template <bool kCT, int NQ, bool kOwn>
__global__ void __launch_bounds__(sc_threads(kOwn), 1)
k_lu_solve_cluster(const float2* __restrict__ A, int64_t n, int64_t stride, const float2* __restrict__ Dinv,
                   int64_t dstride, float2* __restrict__ X, int64_t xstride, int stages, int vec, int* bad,
                   const int* done, const int* unset_flag)
{
    constexpr int NB = kScNB;
    extern __shared__ __align__(128) unsigned char sc_smem_raw[];
    uint32_t rank_u, cs_u;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank_u));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(cs_u));
    const int rank = (int)rank_u, cs = (int)cs_u;
    const int64_t b = blockIdx.x / cs_u;
    const int nblk = (int)((n + NB - 1) / NB);
    float2* tiles = reinterpret_cast<float2*>(sc_smem_raw);  // [stages][64][kScLd]
    float2* ytab = tiles + (size_t)stages * NB * kScLd;      // [nblk][NQ][64]; own: [ceil(nblk / cs)][NQ][64]
    float2* ystage = ytab + (size_t)(kOwn ? (nblk + cs - 1) / cs : nblk) * NQ * NB;  // own: [stages][NQ][64]
    float2* xs = ystage + (size_t)(kOwn ? stages : 0) * NQ * NB;                     // [2][NQ][64]
    uint64_t* full = reinterpret_cast<uint64_t*>(xs + 2 * NQ * NB);
    uint64_t* empty = full + kScMaxStages;
    uint64_t* ybar = empty + kScMaxStages;  // [2][nblk]
    uint64_t* turn = ybar + 2 * nblk;       // every CTA holds all blocks of the first triangle
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // read before the cluster's first barrier, and marked only after it, so the
    // CTAs of a cluster agree: a converged or marked matrix is left alone
    const bool skip = done && (done[b] || bad[b]);
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            sc_init(&full[s], 32 * (kScProducers + kOwn));  // every producer lane
            sc_init(&empty[s], kScConsumers / 32);     // every consumer warp
        }
        sc_init(turn, cs);
        for (int j = 0; j < 2 * nblk; ++j) {
            sc_init(&ybar[j], kOwn ? kScConsumers / 32 : 1);  // own: every consumer warp of the owner
            if (!kOwn)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                             :: "r"(sc_smem_u32(&ybar[j])), "r"((uint32_t)(NQ * NB * sizeof(float2))) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    sc_cluster_sync();
    if (skip) return;
    const float2* M = A + b * stride;
    const float2* Dv = Dinv + b * dstride;
    float2* x = X + b * xstride;
    const int nown = rank < nblk ? (nblk - 1 - rank) / cs + 1 : 0;
    if (kOwn && warp == kScConsumers / 32 + kScProducers) {  // the y of every tile, from its owner
        const uint32_t own0 = sc_smem_u32(ytab) + 16 * lane, to0 = sc_smem_u32(ystage) + 16 * lane;
        int s = 0;
        uint32_t phase = 1;
        bool gave_up = false;
        for (int tri = 0; tri < 2; ++tri) {
            int held = 0;  // blocks known to be solved, in the triangle's order
            for (int bi = 0; bi < nown; ++bi) {
                const int i = sc_own(tri, nown, rank, cs, bi);
                const int nt = tri == 0 ? i : nblk - 1 - i;
                for (int jj = 0; jj <= nt; ++jj) {
                    if (lane == 0 && !sc_wait(&empty[s], phase)) atomicExch(bad + b, 2);
                    __syncwarp();
                    if (jj < nt) {  // the inverse diagonal block takes none
                        const int j = tri == 0 ? jj : nblk - 1 - jj;
                        if (jj >= held) {
                            if (!gave_up) {
                                const bool there = unset_flag && j % cs != rank ? sc_unset(unset_flag)
                                                                                : sc_wait(&ybar[tri * nblk + j], 0);
                                gave_up = !__all_sync(0xffffffffu, there);
                                if (gave_up && lane == 0) atomicExch(bad + b, 3);
                            }
                            held = jj + 1;
                        }
                        const uint32_t from = sc_map(own0 + (uint32_t)((j / cs) * (NQ * NB * sizeof(float2))), j % cs);
                        const uint32_t to = to0 + (uint32_t)(s * (NQ * NB * sizeof(float2)));
                        float4 v[NQ];
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                                         : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q].z), "=f"(v[q].w)
                                         : "r"(from + (uint32_t)(q * NB * sizeof(float2))) : "memory");
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                                         :: "r"(to + (uint32_t)(q * NB * sizeof(float2))), "f"(v[q].x), "f"(v[q].y),
                                            "f"(v[q].z), "f"(v[q].w) : "memory");
                    }
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(sc_smem_u32(&full[s])) : "memory");
                    if (++s == stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        // every arrival of the cluster's CTAs has come in (also after a wait that ran out: every block is published)
        for (int j = 0; j < 2 * nblk; ++j)
            if (!sc_wait(&ybar[j], 0) && lane == 0) atomicExch(bad + b, 3);
    } else if (warp >= kScConsumers / 32) {  // producer warps: every kScProducers-th column each
        const int par = warp - kScConsumers / 32;
        const uint32_t tile0 = sc_smem_u32(tiles) + (uint32_t)((par * kScLd) * sizeof(float2));
        int s = 0;
        uint32_t phase = 1;  // of the stage's last release (the first round finds the stages free)
        for (int tri = 0; tri < 2; ++tri) {
            const int inv_off = ((tri == 0) != kCT) ? 0 : NB * NB;
            for (int bi = 0; bi < nown; ++bi) {
                const int i = sc_own(tri, nown, rank, cs, bi);
                const int nt = tri == 0 ? i : nblk - 1 - i;
                for (int jj = 0; jj <= nt; ++jj) {
                    if (lane == 0 && !sc_wait(&empty[s], phase)) atomicExch(bad + b, 2);
                    __syncwarp();
                    // tile (i, j): rows of block i and columns of block j (kCT: transposed), or the inverse diagonal
                    // block of i (whole, column-major); one column per warp instruction, the address stepped
                    const bool inv = jj == nt;
                    const int64_t i0 = (int64_t)i * NB, j0 = (int64_t)(tri == 0 ? jj : nblk - 1 - jj) * NB;
                    const int64_t r0 = kCT ? j0 : i0, c0 = kCT ? i0 : j0;
                    const int64_t ld = inv ? NB : n;
                    const char* g = reinterpret_cast<const char*>(
                        inv ? Dv + (int64_t)i * 2 * NB * NB + inv_off + par * NB : M + (c0 + par) * n + r0);
                    const int64_t step = ld * (int64_t)(kScProducers * sizeof(float2));
                    const bool whole = inv || (r0 + NB <= n && c0 + NB <= n);
                    const uint32_t dst = tile0 + (uint32_t)(s * (int)kScTileBytes);
                    constexpr uint32_t kDstStep = kScProducers * kScLd * sizeof(float2);
                    if (whole && (vec || inv)) {
                        g += 16 * lane;
                        const uint32_t d = dst + 16 * lane;
#pragma unroll
                        for (int c = 0; c < NB / kScProducers; ++c, g += step)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                         :: "r"(d + c * kDstStep), "l"(g) : "memory");
                    } else if (whole) {
                        g += 8 * lane;
                        const uint32_t d = dst + 8 * lane;
#pragma unroll
                        for (int c = 0; c < NB / kScProducers; ++c, g += step) {
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                                         :: "r"(d + c * kDstStep), "l"(g) : "memory");
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                                         :: "r"(d + c * kDstStep + 256), "l"(g + 256) : "memory");
                        }
                    } else {  // at the matrix's edge: entries past it are zeros (size 0, with an address inside)
                        const int rows = (int)min((int64_t)NB, n - r0), cols = (int)min((int64_t)NB, n - c0);
#pragma unroll 2
                        for (int c = 0; c < NB / kScProducers; ++c, g += step)
#pragma unroll
                            for (int hrow = 0; hrow < 2; ++hrow) {
                                const int rr = lane + 32 * hrow;
                                const bool ok = rr < rows && par + c * kScProducers < cols;
                                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;"
                                             :: "r"(dst + c * kDstStep + 8 * rr), "l"(ok ? g + 8 * rr : (const char*)M),
                                                "r"(ok ? 8 : 0) : "memory");
                            }
                    }
                    // this lane's arrival fires when its copies have landed
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];"
                                 :: "r"(sc_smem_u32(&full[s])) : "memory");
                    if (++s == stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // consumers: the 16 lanes of a row group share four rows; after a reduction a lane holds row `row`, as do the
        // three others of its four, which deal the right-hand sides and the cluster's CTAs among them (l4)
        const int e = lane & 15, l4 = lane & 3;
        const int r0 = 8 * warp + 4 * (lane >> 4), row = r0 + 2 * (e >> 3) + ((e >> 2) & 1);
        constexpr int kMine = (NQ + 3) / 4;  // right-hand sides l4, l4 + 4 of a lane
        int s = 0;
        uint32_t phase = 0;
        bool ok = true, gave_up = false;
        auto take = [&]() {
            if (!sc_wait(&full[s], phase) && ok) {
                ok = false;
                if (lane == 0) atomicExch(bad + b, 2);
            }
        };
        auto give = [&]() {
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(sc_smem_u32(&empty[s])) : "memory");
            if (++s == stages) {
                s = 0;
                phase ^= 1;
            }
        };
        auto hold = [&](int tri, int j) {
            if (gave_up) return;
            if (unset_flag && j % cs != rank) gave_up = !sc_unset(unset_flag);
            else gave_up = !sc_wait(&ybar[tri * nblk + j], 0);
            if (gave_up && lane == 0) atomicExch(bad + b, 3);
        };
        int parity = 0;
        for (int tri = 0; tri < 2; ++tri) {
            int held = 0;  // blocks of the triangle held so far, in its order (they arrive in it)
            for (int bi = 0; bi < nown; ++bi) {
                const int i = sc_own(tri, nown, rank, cs, bi);
                const int nt = tri == 0 ? i : nblk - 1 - i;
                const size_t yi = (size_t)(kOwn ? i / cs : i) * NQ;  // its place in the table
                const int64_t i0 = (int64_t)i * NB;
                const bool inside = i0 + row < n;
                // right-hand sides; the second triangle's are the first one's solution
                float2 rhs[kMine];
#pragma unroll
                for (int k = 0; k < kMine; ++k) {
                    const int q = l4 + 4 * k;
                    rhs[k] = make_float2(0.f, 0.f);
                    if (q < NQ && tri == 1) rhs[k] = ytab[(yi + q) * NB + row];
                    if (q < NQ && tri == 0 && inside) rhs[k] = x[(int64_t)q * n + i0 + row];
                }
                float2 acc[4][NQ], sum[NQ];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int q = 0; q < NQ; ++q) acc[u][q] = make_float2(0.f, 0.f);
                for (int jj = 0; jj < nt; ++jj) {
                    const int j = tri == 0 ? jj : nblk - 1 - jj;
                    take();
                    if (!kOwn && jj >= held) {
                        hold(tri, j);
                        held = jj + 1;
                    }
                    sc_tile<kCT, NQ>(tiles + (size_t)s * NB * kScLd,
                                     kOwn ? ystage + (size_t)s * NQ * NB : ytab + (size_t)j * NQ * NB, r0, e, acc);
                    give();
                }
                sc_reduce<NQ>(acc, e, sum);
                float2* xi = xs + parity * (NQ * NB);
                parity ^= 1;
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                    if ((q & 3) == l4)
                        xi[q * NB + row] = make_float2(rhs[q >> 2].x - sum[q].x, rhs[q >> 2].y - sum[q].y);
                asm volatile("bar.sync 1, %0;" :: "r"(kScConsumers) : "memory");
                take();
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int q = 0; q < NQ; ++q) acc[u][q] = make_float2(0.f, 0.f);
                sc_tile<kCT, NQ>(tiles + (size_t)s * NB * kScLd, xi, r0, e, acc);
                give();
                sc_reduce<NQ>(acc, e, sum);
                if constexpr (kOwn) {  // into the own table, then an arrival of every warp at every CTA of the cluster
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
                        if ((q & 3) == l4) ytab[(yi + q) * NB + row] = sum[q];
                    __syncwarp();
                    if (lane < cs)
                        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];"
                                     :: "r"(sc_map(sc_smem_u32(&ybar[tri * nblk + i]), lane)) : "memory");
                } else {
                    // the row's entries into every CTA of the cluster
                    for (int to = l4; to < cs; to += 4) {
                        const uint32_t at = sc_map(sc_smem_u32(ytab + yi * NB + row), to);
                        const uint32_t bar = sc_map(sc_smem_u32(&ybar[tri * nblk + i]), to);
#pragma unroll
                        for (int q = 0; q < NQ; ++q)
                            asm volatile(
                                "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];"
                                :: "r"(at + (uint32_t)(q * NB * sizeof(float2))), "f"(sum[q].x), "f"(sum[q].y), "r"(bar)
                                : "memory");
                    }
                }
                if (tri == 1 && inside) {
#pragma unroll
                    for (int q = 0; q < NQ; ++q)
                        if ((q & 3) == l4) x[(int64_t)q * n + i0 + row] = sum[q];
                }
            }
            if (kOwn) continue;
            // every block of this triangle has landed here: nothing is in flight to this CTA (also after a wait
            // that ran out: every block is stored in any case)
            for (int j = 0; j < nblk; ++j)
                if (!sc_wait(&ybar[tri * nblk + j], 0) && lane == 0) atomicExch(bad + b, 3);
            if (tri == 0) {
                // the second triangle overwrites the table once every CTA is here
                asm volatile("bar.sync 1, %0;" :: "r"(kScConsumers) : "memory");
                if (tid < cs)
                    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];"
                                 :: "r"(sc_map(sc_smem_u32(turn), tid)) : "memory");
                if (!sc_wait(turn, 0) && lane == 0) atomicExch(bad + b, 2);
            }
        }
    }
    __syncwarp();
    sc_cluster_sync();  // a CTA's shared memory is written by the others until here
}

using SolveKernel = void (*)(const float2*, int64_t, int64_t, const float2*, int64_t, float2*, int64_t, int, int, int*,
                             const int*, const int*);

template <bool kCT, bool kOwn>
SolveKernel solve_of(int nq)
{
    switch (nq) {
        case 1: return k_lu_solve_cluster<kCT, 1, kOwn>;
        case 2: return k_lu_solve_cluster<kCT, 2, kOwn>;
        case 3: return k_lu_solve_cluster<kCT, 3, kOwn>;
        case 4: return k_lu_solve_cluster<kCT, 4, kOwn>;
        case 5: return k_lu_solve_cluster<kCT, 5, kOwn>;
        case 6: return k_lu_solve_cluster<kCT, 6, kOwn>;
        case 7: return k_lu_solve_cluster<kCT, 7, kOwn>;
        default: return k_lu_solve_cluster<kCT, 8, kOwn>;
    }
}

// Right-hand sides of a pass: up to eight, as many as fit beside two stages (0: none).
int sc_most(bool own, int cs, int64_t nblk)
{
    int q = 8;
    while (q > 0 && sc_smem(own, cs, nblk, q, 2) > kScSmemMax) --q;
    return q;
}

cudaLaunchConfig_t solve_config(cudaLaunchAttribute (&at)[1], bool own, int nbatch, int cs, size_t smem,
                                cudaStream_t stream)
{
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)nbatch * (unsigned)cs);
    cfg.blockDim = dim3(sc_threads(own));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// CTAs per matrix: the most, up to eight and one per row block, that let the clusters
// of nbatch matrices run at once.  Every variant fills an SM's shared memory, so one
// of them stands for all.
cudaError_t cluster_size(mh_ctx* ctx, int nbatch, int64_t nblk, int* out)
{
    const SolveKernel k = k_lu_solve_cluster<false, 1, false>;
    const size_t smem = sc_smem(false, 1, 1, 1, kScMaxStages);
    cudaError_t e;
    int cs = (int)std::min<int64_t>(8, nblk);
    for (; cs > 1; --cs) {
        if ((int64_t)nbatch * cs > 148) continue;
        int& room = ctx->solve_clusters[cs];
        if (room == 0) {
            if ((e = raise_smem_cap((const void*)k, smem)) != cudaSuccess) return e;
            cudaLaunchAttribute at[1];
            const cudaLaunchConfig_t cfg = solve_config(at, false, 1, cs, smem, ctx->stream);
            if ((e = cudaOccupancyMaxActiveClusters(&room, (const void*)k, &cfg)) != cudaSuccess) {
                room = 0;
                return e;
            }
        }
        if (nbatch <= room) break;
    }
    *out = cs;
    return cudaSuccess;
}

}  // namespace

cudaError_t launch_lu_solve_cluster(mh_ctx* ctx, bool conj_trans, const float2* A, int64_t n, int64_t stride,
                                    int nbatch, const float2* Dinv, int64_t dstride, float2* X, int64_t xstride,
                                    int nrhs, int* bad, const int* done, const int* unset_flag, cudaStream_t stream)
{
    const int64_t nblk = (n + kScNB - 1) / kScNB;
    if (nrhs < 1 || !bad) return cudaErrorInvalidValue;
    int cs;
    cudaError_t e = cluster_size(ctx, nbatch, nblk, &cs);
    if (e != cudaSuccess) return e;
    // The table of all blocks in every CTA, or of its own in each (all orders that the device's memory holds fit
    // the latter): the former's step is shorter (us a solve, all and own: 870 panels x 16 matrices, 4 right-hand
    // sides 65 and 86, 2048 x 64, 3 419 and 443, 3552 x 8, 3 351 and 409), but its table costs passes (3552 x 8, 8 935
    // and 656; 8192, 4 4570 and 1780; 12,240, 8 26,470 and 6340) and, where the factors' stream bounds the solve,
    // stages (6144, 2 972 and 824; 12,240, 1 3310 and 2650) or, for odd n, the L1 that 8-byte copies go through (2997
    // x 24, 2 374 and 400, 3 528 and 431; 4095, 2 542 and 460).
    int most = sc_most(false, cs, nblk);
    while (most == 0 && sc_most(true, cs, nblk) == 0 && cs < 8) ++cs;
    const int most_own = sc_most(true, cs, nblk);
    const auto passes_of = [&](int m) { return m ? (nrhs + m - 1) / m : INT_MAX; };
    const int vec = n % 2 == 0 && stride % 2 == 0 && ((uintptr_t)A & 15) == 0;
    bool own = passes_of(most_own) < passes_of(most);
    if (!own && most && nblk >= 46 && most_own)
        own = sc_smem(false, cs, nblk, (nrhs + passes_of(most) - 1) / passes_of(most), kScMaxStages) >
              (vec ? kScSmemMax : kScSmemMax - 30 * 1024);
    if (own) most = most_own;
    if (most == 0) return cudaErrorInvalidValue;
    const int passes = passes_of(most);
    for (int p = 0, q0 = 0; p < passes; ++p) {  // even shares
        const int nq = (nrhs - q0 + passes - p - 1) / (passes - p);
        int stages = 2;
        while (stages < kScMaxStages && sc_smem(own, cs, nblk, nq, stages + 1) <= kScSmemMax) ++stages;
        const SolveKernel k = conj_trans ? (own ? solve_of<true, true>(nq) : solve_of<true, false>(nq))
                                         : (own ? solve_of<false, true>(nq) : solve_of<false, false>(nq));
        const size_t smem = sc_smem(own, cs, nblk, nq, stages);
        if ((e = raise_smem_cap((const void*)k, smem)) != cudaSuccess) return e;
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = solve_config(at, own, nbatch, cs, smem, stream);
        if ((e = cudaLaunchKernelEx(&cfg, k, A, n, stride, Dinv, dstride, X + (int64_t)q0 * n, xstride, stages, vec, bad,
                                    done, unset_flag)) != cudaSuccess)
            return e;
        ctx->launches += 1;
        q0 += nq;
    }
    return cudaGetLastError();
}

}  // namespace mh
