// dev_chol.cu -- blocked right-looking Cholesky factorization and solve in
// FP64 (reference src/ParallelAlgorithms.c:361-447, which ends in LAPACK
// dpotrf/dpotrs).
//
// M is column-major with leading dimension ld >= n + 1. The right-hand side b
// is carried as row n: the factorization then produces, in that row, the
// forward-substitution result z = L^-1 b, and one backward sweep gives x.
//
// Failed pivots keep LAPACK's behaviour: a pivot that is not positive is
// stored without its square root and reported (first failure, 1-based) in
// device flag 0. In full IRWLS the system matrix is bordered by the labels
// with a zero corner, so its last pivot fails by construction; the reference
// ignores that failure and solves with the stored negative Schur complement,
// and so does this code.
//
// Two factorizations with the same arithmetic per element (so the same
// bits): one cooperative launch scheduled by data flow (the default, below
// chol_df_kernel), and a multi-launch sequence per panel of 32 columns (a
// launch that solves the rows below the diagonal block against it, and a
// launch that applies the rank-32 update to the lower trailing matrix and
// factors the next diagonal block).
#include <math.h>

#include <atomic>

#include <cooperative_groups.h>

#include "dev_common.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int NB = 32;

// Factors the nb x nb diagonal block at (k0, k0) held in D (shared, NB x NB,
// lower part valid), with LAPACK dpotrf's failed-pivot behaviour, leaving
// the reciprocal of each stored pivot in rp. Uses the whole CTA; ends synced.
// FP64 runs at a fraction of the FP32 rate on this part, so every dependent
// FP64 operation on this serial path costs tens of cycles: the pivot's
// reciprocal square root is formed once and the column is scaled by it (as
// dpotf2 scales by 1 / ajj).
__device__ void factor_block(double (*D)[NB + 1], double *rp, int nb, int k0, int *flags, int *failed_at) {
    const int tid = threadIdx.x;
    if (tid == 0) *failed_at = -1;
    __syncthreads();
    for (int c = 0; c < nb; ++c) {
        if (tid == 0) {
            const double s = D[c][c];
            if (s > 0.0) {
                const double r = rsqrt(s);
                D[c][c] = s * r;
                rp[c] = r;
            } else {
                if (*failed_at < 0) *failed_at = c;  // stored without its root, as dpotrf leaves it
                rp[c] = 1.0 / s;
            }
        }
        __syncthreads();
        const double r = rp[c];
        for (int rr = c + 1 + tid; rr < nb; rr += blockDim.x) D[rr][c] = D[rr][c] * r;
        __syncthreads();
        const int m = nb - c - 1;
        for (int t = tid; t < m * m; t += blockDim.x) {
            const int rr = c + 1 + t / m, j = c + 1 + t % m;
            if (j <= rr) D[rr][j] = fma(-D[rr][c], D[j][c], D[rr][j]);
        }
        __syncthreads();
    }
    if (tid == 0 && *failed_at >= 0) atomicCAS(flags, 0, k0 + *failed_at + 1);
}

// Inverse of the factored block (its reciprocal pivots in rp): each entry a
// dot product split over 8 lanes of a warp, four columns to a warp,
// Di[c][j] = -(sum_{j <= t < c} D[c][t] Di[t][j]) rp[c], entry (c, j)'s lane q
// summing t = j + q, j + q + 8, ... Warps w and w + 4, which share an SM
// quarter's FP64 unit, take column groups w and 7 - w: 34 rows to form
// between them everywhere (46 and 22 at the ends with groups in warp order,
// where a 32-column inverse took 28000 cycles).
// Di zeroed by the caller; blockDim.x >= 256, the first eight warps call.
__device__ void invert_columns(double (*D)[NB + 1], double (*Di)[NB + 1], const double *rp, int nb) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // (every lane of a warp runs the same iterations so that the shuffles
    // always see the whole warp; the first row below a warp's four columns
    // is the first it has to form)
    const int j0 = 4 * (warp < 4 ? warp : 11 - warp), j = j0 + (lane >> 3), q = lane & 7;
    if (q == 0 && j < nb) Di[j][j] = rp[j];
    __syncwarp();
    for (int c = j0 + 1; c < nb; ++c) {
        const bool live = j < nb && c > j;
        double acc = 0.0, d[4], e[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // (all of the row's loads before its FMAs)
            const int t = min(j + q + 8 * k, NB - 1);
            d[k] = D[c][t];
            e[k] = Di[t][j];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (live && j + q + 8 * k < c) acc = fma(d[k], e[k], acc);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4, 8);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2, 8);
        acc += __shfl_xor_sync(0xffffffffu, acc, 1, 8);
        if (live && q == 0) Di[c][j] = -acc * rp[c];
        __syncwarp();
    }
}

__device__ void invert_block(double (*D)[NB + 1], double (*Di)[NB + 1], const double *rp, int nb) {
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) Di[t / NB][t % NB] = 0.0;
    __syncthreads();
    invert_columns(D, Di, rp, nb);
    __syncthreads();
}

__device__ void factor_invert_block(double (*D)[NB + 1], double (*Di)[NB + 1], double *rp, int nb, int k0,
                                    int *flags, int *failed_at) {
    factor_block(D, rp, nb, k0, flags, failed_at);
    invert_block(D, Di, rp, nb);
}

// Panel solve of the rows r < nr of T (columns c < nb) against the factored
// diagonal block D with reciprocal pivots rp, in place, by forward
// substitution: x_c = (a_c - sum_{t < c} x_t D[c][t]) rp[c], the sum taken
// by FMAs in increasing t. Used by both factorizations, so they agree bit
// for bit. blockDim.x == 256; ends synced.
__device__ void subst_block(double (*T)[NB + 1], int nr, double (*D)[NB + 1], const double *rp, int nb) {
    const int tid = threadIdx.x;
    for (int t = 0; t < nb; ++t) {
        for (int r = tid; r < nr; r += blockDim.x) T[r][t] = T[r][t] * rp[t];
        __syncthreads();
        const int m = nb - t - 1;
        for (int e = tid; e < nr * m; e += blockDim.x) {
            const int r = e / m, c = t + 1 + e % m;
            T[r][c] = fma(-T[r][t], D[c][t], T[r][c]);
        }
        __syncthreads();
    }
}

__device__ void store_block(double *M, int ld, int k0, int nb, double (*D)[NB + 1], double (*Di)[NB + 1],
                            double *Dinv) {
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int r = t / NB, c = t % NB;
        if (r < nb && c <= r) M[(size_t)(k0 + c) * ld + k0 + r] = D[r][c];
        Dinv[t] = Di[r][c];
    }
}

// First diagonal block (the others are factored by the trailing update of
// the previous panel).
__global__ void __launch_bounds__(256) chol_factor0_kernel(double *__restrict__ M, int n, int ld,
                                                           int *__restrict__ flags, double *__restrict__ Dinv) {
    __shared__ double D[NB][NB + 1], Di[NB][NB + 1];
    __shared__ double rp[NB];
    __shared__ int failed_at;
    const int nb = min(NB, n);
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int r = t / NB, c = t % NB;
        D[r][c] = (r < nb && c <= r) ? M[(size_t)c * ld + r] : 0.0;
    }
    __syncthreads();
    factor_invert_block(D, Di, rp, nb, 0, flags, &failed_at);
    store_block(M, ld, 0, nb, D, Di, Dinv);
}

// Panel solve: rows i >= k0 + nb (and the right-hand-side row n when present)
// get L[i, k0:k0+nb] = A[i, k0:k0+nb] D^-T by forward substitution against
// the factored diagonal block (from M, its reciprocal pivots from the
// diagonal of the stored inverse). 8 rows per CTA.
__global__ void __launch_bounds__(256) chol_trsm_kernel(double *__restrict__ M, int ld, int k0, int nb, int nrows,
                                                        const double *__restrict__ Dinv) {
    __shared__ double D[NB][NB + 1];
    __shared__ double A[8][NB + 1];
    __shared__ double rp[NB];
    const int tid = threadIdx.x;
    const int i0 = k0 + nb + blockIdx.x * 8;
    for (int t = tid; t < NB * NB; t += 256) {
        const int r = t / NB, c = t % NB;
        D[r][c] = (r < nb && c <= r) ? M[(size_t)(k0 + c) * ld + k0 + r] : 0.0;
    }
    if (tid < NB) rp[tid] = Dinv[tid * (NB + 1)];
    {
        const int c = tid / 8, r = tid % 8;  // 256 = 32 columns x 8 rows
        const int i = i0 + r;
        A[r][c] = (c < nb && i < nrows) ? M[(size_t)(k0 + c) * ld + i] : 0.0;
    }
    __syncthreads();
    const int nr = min(8, nrows - i0);
    subst_block(A, nr, D, rp, nb);
    const int c = tid / 8, r = tid % 8;
    const int i = i0 + r;
    if (c < nb && i < nrows) M[(size_t)(k0 + c) * ld + i] = A[r][c];
}

// Trailing update of the lower part: M[i][j] -= sum_t L[i][t] L[j][t] over the
// panel columns t, for k1 <= j <= i < nrows, j < n. One 32x32 tile per CTA.
// The CTA of tile (0, 0) then factors and inverts that tile, which is the
// next panel's diagonal block.
__global__ void __launch_bounds__(256) chol_update_kernel(double *__restrict__ M, int n, int ld, int k0, int nb,
                                                          int nrows, int *__restrict__ flags,
                                                          double *__restrict__ Dinv_next) {
    const int bj = blockIdx.x, bi = blockIdx.y;
    if (bi < bj) return;
    const int k1 = k0 + nb;
    const int r0 = k1 + bi * 32, c0 = k1 + bj * 32;
    __shared__ double Li[32][NB + 1];
    __shared__ double Lj[32][NB + 1];
    __shared__ int failed_at;
    const int tid = threadIdx.x;
    for (int t = tid; t < 32 * NB; t += 256) {
        const int r = t % 32, k = t / 32;
        const int gi = r0 + r, gj = c0 + r;
        Li[r][k] = (k < nb && gi < nrows) ? M[(size_t)(k0 + k) * ld + gi] : 0.0;
        Lj[r][k] = (k < nb && gj < n) ? M[(size_t)(k0 + k) * ld + gj] : 0.0;
    }
    __syncthreads();
    const int r = tid % 32;
    for (int cc = tid / 32; cc < 32; cc += 8) {
        const int gi = r0 + r, gj = c0 + cc;
        if (gi >= nrows || gj >= n || gj > gi) continue;
        double acc = 0.0;
#pragma unroll 8
        for (int k = 0; k < NB; ++k) acc = fma(Li[r][k], Lj[cc][k], acc);
        double *p = M + (size_t)gj * ld + gi;
        *p = *p - acc;
    }
    if (bi != 0 || bj != 0) return;
    // next diagonal block: reuse Li / Lj as D / Di
    __syncthreads();
    const int nb2 = min(NB, n - k1);
    for (int t = tid; t < NB * NB; t += 256) {
        const int rr = t / NB, c = t % NB;
        Li[rr][c] = (rr < nb2 && c <= rr) ? M[(size_t)(k1 + c) * ld + k1 + rr] : 0.0;
    }
    __syncthreads();
    __shared__ double rp[NB];
    factor_invert_block(Li, Lj, rp, nb2, k1, flags, &failed_at);
    store_block(M, ld, k1, nb2, Li, Lj, Dinv_next);
}

// The two dot products of a backward-sweep block, shared by both sweeps so
// that they give the same bits: each as four interleaved partial FMA chains
// (the dependent chain of one FP64 FMA per term is four times shorter) added
// as (s0 + s1) + (s2 + s3).
// x_t = sum_{t <= c < nb} Di[c][t] yb[c]
__device__ __forceinline__ double sweep_dot(const double (*Di)[NB + 1], const double *yb, int t, int nb) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    int c = t;
    for (; c + 3 < nb; c += 4) {
        a0 = fma(Di[c][t], yb[c], a0);
        a1 = fma(Di[c + 1][t], yb[c + 1], a1);
        a2 = fma(Di[c + 2][t], yb[c + 2], a2);
        a3 = fma(Di[c + 3][t], yb[c + 3], a3);
    }
    for (; c < nb; ++c) a0 = fma(Di[c][t], yb[c], a0);
    return (a0 + a1) + (a2 + a3);
}

// sum_{c < nb} col[c] xb[c]
__device__ __forceinline__ double sweep_row(const double *col, const double *xb, int nb) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    int c = 0;
    for (; c + 3 < nb; c += 4) {
        a0 = fma(col[c], xb[c], a0);
        a1 = fma(col[c + 1], xb[c + 1], a1);
        a2 = fma(col[c + 2], xb[c + 2], a2);
        a3 = fma(col[c + 3], xb[c + 3], a3);
    }
    for (; c < nb; ++c) a0 = fma(col[c], xb[c], a0);
    return (a0 + a1) + (a2 + a3);
}

// Backward sweep L^T x = z, z in row n of M; one CTA, z in shared memory,
// 32-row blocks from the bottom: x_b = D_b^-T y_b (parallel dots with the
// stored inverse), then the rows above are updated.
__global__ void __launch_bounds__(256) chol_backsolve_kernel(const double *__restrict__ M, int n, int ld,
                                                             const double *__restrict__ Dinv,
                                                             double *__restrict__ x) {
    extern __shared__ double z[];
    __shared__ double Di[NB][NB + 1];
    __shared__ double yb[NB];
    const int tid = threadIdx.x;
    for (int c = tid; c < n; c += blockDim.x) z[c] = M[(size_t)c * ld + n];
    const int nblk = (n + NB - 1) / NB;
    for (int b = nblk - 1; b >= 0; --b) {
        const int r0 = b * NB, r1 = min(n, r0 + NB);
        for (int t = tid; t < NB * NB; t += blockDim.x) Di[t / NB][t % NB] = Dinv[(size_t)b * NB * NB + t];
        __syncthreads();
        if (tid < NB) yb[tid] = (r0 + tid < r1) ? z[r0 + tid] : 0.0;
        __syncthreads();
        if (tid < r1 - r0) z[r0 + tid] = sweep_dot(Di, yb, tid, r1 - r0);
        __syncthreads();
        for (int r = tid; r < r0; r += blockDim.x) z[r] = z[r] - sweep_row(M + (size_t)r * ld + r0, z + r0, r1 - r0);
        __syncthreads();
    }
    for (int c = tid; c < n; c += blockDim.x) x[c] = z[c];
}

__global__ void zero_upper_kernel(double *__restrict__ M, int n, int ld) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)n * n;
         t += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(t / n), r = (int)(t % n);
        if (r < c) M[(size_t)c * ld + r] = 0.0;
    }
}

// ---------------------------------------------------------------------------
// The same factorization in one cooperative launch, scheduled by data flow.
//
// The lower blocked matrix (32 x 32 tiles (i, j), i >= j, the right-hand-side
// row n included as a row) is a list of tasks in column-major order; task t
// belongs to CTA t mod G, and each CTA runs its tasks in order, keeping its
// tile in shared memory. A tile takes the updates of panels k = 0 ... j - 1,
// then either factors itself (i == j) or solves against diagonal block j.
// Every tile is published four columns at a time (a release store of its
// column count after the data; readers poll it with acquire loads and read the
// data from L2), and its readers take the columns as they come: the panel
// solves run four columns behind the pivots, and the next diagonal tile's
// last update four columns behind the panel solves, so that a panel costs its
// pivot chain plus one trailing step of each instead of the sum of whole
// tiles. In each CTA one warp polls and loads ahead into a ring of steps, one
// stores and publishes, and eight compute: a poll and its loads take about
// 1300 cycles and a publication 1400, which would otherwise add to each step. Every dependency of a task has a smaller index, and all CTAs are
// resident (cooperative launch), so the smallest unfinished task can always
// run: no wait is circular.
//
// What bounds it: an FP64 instruction of one warp takes 65 cycles on this part
// and holds its SM quarter's FP64 unit for that long (76 with all four busy),
// so a panel of 32 pivots is a chain of 32 (reciprocal square root 370 cycles,
// scale, diagonal update). One warp runs that chain on a quarter of its own
// (factor_stream); six warps on the other three scale the columns and apply the
// rank-1 updates.
// Whole tiles at a time, with three CTA barriers per pivot, a panel took 40 to
// 48 us.
//
// Every element gets the multi-launch path's operations in the same order:
// per panel, acc = sum over the panel's 32 columns by FMA from zero, then
// M - acc; the diagonal blocks as factor_block; the panel solves by forward
// substitution (subst_block's operations). The results are the same bits. A
// diagonal block is published before its inverse is formed: only the backward
// sweep, after this launch, reads the inverse.
//
// The waits are bounded: one that runs out (which needs a fault in this
// schedule) sets the pivot status to -1 and the tensor-core status word to
// CHOL_WAIT_CODE, and the CTA stops; the others then run out too.
// ---------------------------------------------------------------------------
constexpr long long DF_WAIT_LIMIT = 1LL << 22;
constexpr int CHOL_WAIT_CODE = 0x40000000;
// polls of the computing warps for the loader, which gives up after DF_WAIT_LIMIT polls of
// L2 (1300 cycles each) or TC_WAIT_LIMIT of its own barrier: 16 times those
constexpr long long COMPUTE_WAIT_LIMIT = 16 * TC_WAIT_LIMIT;
static_assert(COMPUTE_WAIT_LIMIT >= 256 * DF_WAIT_LIMIT, "the loader's verdict comes first");
constexpr int DFC = 4;               // columns per published step
constexpr int DFQ = NB / DFC;        // steps of a tile
constexpr int DFR = 6;               // ring slots of steps
constexpr int DF_THREADS = 320;      // warps 0-7 compute, 8 loads, 9 publishes
// named barriers: the pivots' three (factor_stream), finished columns of a
// diagonal block, the compute warps' own two
constexpr int BAR_ROOT = 1, BAR_COL = 2, BAR_NEXT = 3, BAR_PUB = 4;
constexpr int BAR_ALL = BAR_PUB + DFQ, BAR_STEP = BAR_ALL + 1, BAR_ROOT2 = BAR_STEP + 1;
static_assert(BAR_ROOT2 < 16, "named barriers");

__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}
template <int ID, int COUNT>
__device__ __forceinline__ void bar_sync() {
    asm volatile("bar.sync %0, %1;\n" ::"n"(ID), "n"(COUNT) : "memory");
}
template <int ID, int COUNT>
__device__ __forceinline__ void bar_arrive() {
    asm volatile("bar.arrive %0, %1;\n" ::"n"(ID), "n"(COUNT) : "memory");
}
// (barrier numbers known at run time only)
__device__ __forceinline__ void bar_sync_at(int id, int count) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive_at(int id, int count) {
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(count) : "memory");
}

// One step of columns in shared memory: rows of the tile's own block row (or
// of the diagonal block), rows of the other block row, the reciprocal pivots.
struct DfSlot {
    double a[NB][DFC + 1], b[NB][DFC + 1], rp[DFC];
};
struct DfShared {
    double T[NB][NB + 1], Di[NB][NB + 1];
    double rp[NB], rhs[NB];
    // factor_stream, by step parity: the scaled column, the next unscaled one,
    // the diagonal, the pivot and its reciprocal root
    double col[2][NB], next[2][NB], diag[2][NB], piv[2], root[2];
    DfSlot slot[DFR];
    // pub: one per step of a tile, so that the computing warps may run ahead
    // of the publisher; used again after done, the publisher's end of a tile
    uint64_t full[DFR], empty[DFR], pub[DFQ], done;
    volatile int bad[DFR], stop;  // the loader gave up in a slot; the computing warps did
};

// Factors the nb x nb diagonal block in T (lower part valid) with
// factor_block's operations, handing its columns to the publishing warp as
// they are finished. The pivots are one dependent chain -- reciprocal root of
// s_t, the scaled element below it, s_(t+1) = D - l l -- which warp 0 alone
// runs, on scalars, an SM quarter to itself: about 650 cycles a pivot (501 the
// chain alone, 806 when that warp also scaled the column and held the
// diagonal). Warp 1 (lane =
// row) scales column t, keeps the diagonal and signals the publisher; warps 2,
// 3, 5, 6 and 7 hold the 496 elements below the diagonal, in column order, 32
// to a register: group g on warp number g mod 5, the first of a step's live
// groups holding the next column. Barriers: BAR_ROOT and BAR_ROOT2 pass r_t for
// even and odd t (warps 0, 1), BAR_COL the scaled column t (1, updates),
// BAR_NEXT the unscaled column t + 1 and the diagonal (updates, 1, 0); one
// barrier from BAR_PUB on per DFC finished columns. A warp that only arrives
// must not arrive at a barrier again before those that wait at it have: warp 0
// passes BAR_NEXT of step t, which warp 1 joins after BAR_ROOT of step t, between
// its arrivals of steps t and t + 2 but not of t and t + 1, hence the two. What a step hands out lies in one of two buffers by its
// parity: each is written again only after its readers have passed a later
// barrier. Signs are tested on the bits: an FP64 compare would take the unit
// for 65 cycles.
struct FactorPart {
    int er[4], ec[4];  // an update thread's elements (row, column; column -1: none)
    int c0[4], c1[4];  // first and last column of the warp's groups (the warp's)
};
__device__ void factor_part(FactorPart &f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = warp < 4 ? warp - 2 : warp - 3;  // 0 ... 4 on the update warps
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        // element e of the strictly lower part in column order
        int e = (u + 5 * x) * 32 + lane, c = 0;
        while (c < NB - 1 && e >= NB - 1 - c) {
            e -= NB - 1 - c;
            ++c;
        }
        f.ec[x] = c < NB - 1 ? c : -1;  // past the last element: never live
        f.er[x] = c < NB - 1 ? c + 1 + e : 0;
        f.c0[x] = __shfl_sync(0xffffffffu, f.ec[x], 0);
        f.c1[x] = __reduce_max_sync(0xffffffffu, f.ec[x]);
    }
}
__device__ void factor_stream(DfShared &sh, const FactorPart &f, int nb, int k0, int *flags) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int NEXT = 32 * 7, COL = 32 * 6;
    double(*D)[NB + 1] = sh.T;
    if (warp == 0) {
        double s = D[0][0], a = D[1][0], g = D[1][1];  // (read before warp 1 may scale column 0)
        int failed = -1;
        for (int t = 0; t < nb; ++t) {
            const long long bits = __double_as_longlong(s);
            const bool ok = bits > 0 && bits <= 0x7ff0000000000000LL;  // s > 0.0
            const double r = ok ? rsqrt(s) : 1.0 / s;
            if (!ok && failed < 0) failed = t;  // stored without its root, as dpotrf leaves it
            sh.root[t & 1] = r;  // (every lane: the same value)
            sh.piv[t & 1] = s;
            if (t & 1) bar_arrive<BAR_ROOT2, 64>();
            else bar_arrive<BAR_ROOT, 64>();
            if (t + 1 < nb) {
                if (t > 0) {
                    bar_sync<BAR_NEXT, NEXT>();  // of step t - 1: column t and the diagonal
                    a = sh.next[t & 1][t + 1];
                    g = sh.diag[(t - 1) & 1][t + 1];
                }
                const double l = a * r;
                s = fma(-l, l, g);
            } else if (t > 0) {
                bar_arrive<BAR_NEXT, NEXT>();
            }
        }
        if (lane == 0 && failed >= 0) atomicCAS(flags, 0, k0 + failed + 1);
    } else if (warp == 1) {
        double dg = lane < nb ? D[lane][lane] : 0.0;
        for (int t = 0; t < nb; ++t) {
            const double c0 = t == 0 ? D[lane][0] : 0.0;
            if (t > 0) bar_sync<BAR_NEXT, NEXT>();
            const double c = t == 0 ? c0 : sh.next[t & 1][lane];
            if (t & 1) bar_sync<BAR_ROOT2, 64>();
            else bar_sync<BAR_ROOT, 64>();
            const double r = sh.root[t & 1], s = sh.piv[t & 1];
            const long long bits = __double_as_longlong(s);
            const bool ok = bits > 0 && bits <= 0x7ff0000000000000LL;
            const double a = lane == t ? s : lane > t && lane < nb ? c : 0.0;
            const double l = a * r;
            sh.col[t & 1][lane] = l;
            __syncwarp();
            if (t + 1 < nb) bar_arrive<BAR_COL, COL>();
            if (lane >= t) D[lane][t] = lane == t && !ok ? s : l;
            if (lane == t) sh.rp[t] = r;
            dg = fma(-l, l, dg);  // (of use for lanes > t)
            sh.diag[t & 1][lane] = dg;
            __syncwarp();
            if ((t & (DFC - 1)) == DFC - 1 || t == nb - 1) bar_arrive_at(BAR_PUB + t / DFC, 64);
        }
    } else if (warp != 4) {
        double v[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) v[x] = f.ec[x] > 0 ? D[f.er[x]][f.ec[x]] : 0.0;
        for (int t = 0; t + 1 < nb; ++t) {
            bar_sync<BAR_COL, COL>();
            const double *l = sh.col[t & 1];
            double lr[4], lc[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                lr[x] = l[f.er[x]];
                lc[x] = l[max(f.ec[x], 0)];
            }
            bool told = false;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (f.c1[x] <= t) continue;  // no live element
                // the next column lies in the first live groups
                const bool now = f.c0[x] <= t + 1;
                if (!told && !now) {
                    bar_arrive<BAR_NEXT, NEXT>();
                    told = true;
                }
                if (f.ec[x] > t) v[x] = fma(-lr[x], lc[x], v[x]);
                if (now) {
                    if (f.ec[x] == t + 1) sh.next[(t + 1) & 1][f.er[x]] = v[x];
                    __syncwarp();
                }
            }
            if (!told) bar_arrive<BAR_NEXT, NEXT>();
        }
    }
    bar_sync<BAR_ALL, 256>();
}

// ready: columns published of diag[j] at ready[j] (j < nbc), of tile L(i, j)
// at ready[nbc + j * nbr + i]. b: the right-hand side (row n), or NULL when
// it is in row n of M already. ninv: the leading diagonal blocks whose inverse the
// sweep reads; of the others it gets the reciprocal pivots (the diagonal). The
// last block's inverse, which nothing else hides, goes when the sweep substitutes
// that block: 50 us a solve of order 64, with the inverse 59.
__global__ void __launch_bounds__(DF_THREADS, 1) chol_df_kernel(double *__restrict__ M, int n, int ld, int nrows,
                                                                const double *__restrict__ b, int *__restrict__ flags,
                                                                double *__restrict__ Dinv,
                                                                unsigned *__restrict__ ready, int *__restrict__ abort,
                                                                int ninv) {
    chain_open();  // (the sweep may be made resident; it waits for the whole of this)
    extern __shared__ __align__(16) unsigned char df_smem[];
    DfShared &sh = *(DfShared *)df_smem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nbc = (n + NB - 1) / NB, nbr = (nrows + NB - 1) / NB;
    if (tid == 0) {
        for (int q = 0; q < DFR; ++q) {
            mbar_init(&sh.full[q], 32);
            mbar_init(&sh.empty[q], 8);
        }
        for (int q = 0; q < DFQ; ++q) mbar_init(&sh.pub[q], 8);
        mbar_init(&sh.done, 1);
        sh.stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        // the pivot status; every block that can fail comes after tile 0 (CTA
        // 0's) by the chain of published tiles
        if (blockIdx.x == 0) *flags = 0;
    }
    __syncthreads();
    int step = 0;  // ring steps so far, the same in the loading and computing warps

    if (warp == 8) {
        // the loader: per step, polls the two column counts (lanes 0 and 1),
        // then brings the columns into a ring slot
        int t = 0;
        for (int j = 0; j < nbc; ++j) {
            for (int i = j; i < nbr; ++i, ++t) {
                if (t % (int)gridDim.x != (int)blockIdx.x) continue;
                const int r0 = NB * i, c0 = NB * j;
                const int nr = min(NB, nrows - r0), nc = min(NB, n - c0);
                for (int k = 0; k <= j; ++k) {
                    if (k == j && i == j) break;
                    const int kc = NB * k;
                    const unsigned *p = k == j ? ready + j : ready + nbc + (size_t)k * nbr + (lane == 1 ? j : i);
                    int have = 0;
                    for (int q = 0; q < DFQ; ++q, ++step) {
                        const int s = step % DFR, done = DFC * q;
                        bool ok = step < DFR || mbar_wait(smem_u32(&sh.empty[s]), (unsigned)(step / DFR - 1) & 1u);
                        if (have <= done) {
                            for (long long it = 0; ok; ++it) {
                                const int v = lane < 2 ? (int)ld_acquire_u32(p) : NB;
                                have = __reduce_min_sync(0xffffffffu, v);
                                if (have > done) break;
                                if (it >= DF_WAIT_LIMIT) ok = false;
                                if ((it & 63) == 63) {
                                    if (ld_relaxed_u32((const unsigned *)abort)) ok = false;
                                    __nanosleep(32);
                                }
                                ok = __all_sync(0xffffffffu, ok);
                            }
                            __syncwarp();
                        }
                        DfSlot &sl = sh.slot[s];
                        if (lane == 0) sh.bad[s] = !ok;
                        if (ok) {
                            double va[DFC], vb[DFC], vr = 0.0;
#pragma unroll
                            for (int h = 0; h < DFC; ++h) {
                                const double *col = M + (size_t)(kc + done + h) * ld;
                                if (k == j) {
                                    va[h] = __ldcg(col + c0 + lane);
                                } else {
                                    va[h] = lane < nr ? __ldcg(col + r0 + lane) : 0.0;
                                    vb[h] = i != j && lane < nc ? __ldcg(col + c0 + lane) : 0.0;
                                }
                            }
                            if (k == j && lane < DFC)
                                vr = __ldcg(Dinv + (size_t)j * NB * NB + (done + lane) * (NB + 1));
#pragma unroll
                            for (int h = 0; h < DFC; ++h) {
                                sl.a[lane][h] = va[h];
                                if (k < j && i != j) sl.b[lane][h] = vb[h];
                            }
                            if (k == j && lane < DFC) sl.rp[lane] = vr;
                        }
                        mbar_arrive(&sh.full[s]);
                        if (!ok) {
                            if (lane == 0) {
                                *(volatile int *)abort = 1;
                                atomicExch(flags, -1);
                                atomicExch(flags + 1, CHOL_WAIT_CODE | (int)blockIdx.x);
                            }
                            return;
                        }
                    }
                }
            }
        }
        return;
    }

    if (warp == 9) {
        // the publisher: stores finished columns and releases their count
        int t = 0, tasks = 0, below = 0;  // tiles so far, and those below the diagonal
        for (int j = 0; j < nbc; ++j) {
            for (int i = j; i < nbr; ++i, ++t) {
                if (t % (int)gridDim.x != (int)blockIdx.x) continue;
                const int r0 = NB * i, c0 = NB * j;
                const int nr = min(NB, nrows - r0), nc = min(NB, n - c0);
                for (int q = 0; DFC * q < nc; ++q) {
                    const int q1 = min(nc, DFC * q + DFC);
                    bool ok = true;
                    if (i == j) {
                        // (a diagonal tile gives up before it is factored)
                        if (q == 0) ok = mbar_wait(smem_u32(&sh.pub[0]), (unsigned)tasks & 1u) && !sh.stop;
                        if (ok) bar_sync_at(BAR_PUB + q, 64);
                    } else {
                        ok = mbar_wait(smem_u32(&sh.pub[q]), (unsigned)(q == 0 ? tasks : below) & 1u) && !sh.stop;
                    }
                    if (!__all_sync(0xffffffffu, ok)) return;
                    for (int c = DFC * q; c < q1; ++c)
                        if (lane < nr && (i != j || (lane >= c && lane < nc)))
                            M[(size_t)(c0 + c) * ld + r0 + lane] = sh.T[lane][c];
                    if (i == j && lane >= DFC * q && lane < q1)
                        Dinv[(size_t)j * NB * NB + lane * (NB + 1)] = sh.rp[lane];
                    __syncwarp();
                    if (lane == 0)
                        st_release_u32(i == j ? ready + j : ready + nbc + (size_t)j * nbr + i, q1 == nc ? NB : q1);
                }
                if (lane == 0) mbar_arrive(&sh.done);
                ++tasks;
                below += i != j;
            }
        }
        return;
    }

    int t = 0, tasks = 0, told = 0;  // told: publication steps of the current tile
    // this thread's elements of a diagonal tile's lower triangle
    int dr[3], dc[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const int e = tid + 256 * x;
        int r = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
        while (r * (r + 1) / 2 > e) --r;
        while ((r + 1) * (r + 2) / 2 <= e) ++r;
        dr[x] = r;
        dc[x] = e - r * (r + 1) / 2;
    }
    FactorPart part;
    factor_part(part);
    const bool third = tid < NB * (NB + 1) / 2 - 512;
    const int r = tid % NB, u = tid / NB;
    bool good = true;
    // the slot of the next step, or false when the loader gave up. The loader's bounds
    // end first and it always says which: a thread that gave up by itself would leave
    // the others at the next barrier.
    auto take = [&](int s) {
        return mbar_wait(smem_u32(&sh.full[s]), (unsigned)(step / DFR) & 1u, COMPUTE_WAIT_LIMIT) && !sh.bad[s];
    };
    auto give = [&](int s) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[s]);
        ++step;
    };
    for (int j = 0; j < nbc && good; ++j) {
        for (int i = j; i < nbr && good; ++i, ++t) {
            if (t % (int)gridDim.x != (int)blockIdx.x) continue;
            const int r0 = NB * i, c0 = NB * j;
            const int nr = min(NB, nrows - r0), nc = min(NB, n - c0);
            // T is free when the publisher has stored the previous tile
            if (tasks > 0) good = mbar_wait(smem_u32(&sh.done), (unsigned)(tasks - 1) & 1u);
            ++tasks;
            told = 0;
            for (int e = tid; e < NB * NB; e += 256) {
                const int rr = e % NB, c = e / NB;
                double v = 0.0;
                if (rr < nr && c < nc && (i != j || c <= rr))
                    v = b && r0 + rr == n ? b[c0 + c] : __ldcg(M + (size_t)(c0 + c) * ld + r0 + rr);
                sh.T[rr][c] = v;
            }
            bar_sync<BAR_ALL, 256>();
            for (int k = 0; k < j && good; ++k) {
                double acc[4] = {0.0, 0.0, 0.0, 0.0};
                for (int q = 0; q < DFQ; ++q) {
                    const int s = step % DFR;
                    good = take(s);
                    if (!good) break;
                    const DfSlot &sl = sh.slot[s];
                    if (i != j) {
#pragma unroll
                        for (int h = 0; h < DFC; ++h)
#pragma unroll
                            for (int x = 0; x < 4; ++x) acc[x] = fma(sl.a[r][h], sl.b[u + 8 * x][h], acc[x]);
                    } else {
#pragma unroll
                        for (int h = 0; h < DFC; ++h)
#pragma unroll
                            for (int x = 0; x < 3; ++x)
                                if (x < 2 || third) acc[x] = fma(sl.a[dr[x]][h], sl.a[dc[x]][h], acc[x]);
                    }
                    give(s);
                }
                if (!good) break;
                // (each element is its thread's own until the barrier below)
                if (i != j) {
#pragma unroll
                    for (int x = 0; x < 4; ++x)
                        if (r < nr && u + 8 * x < nc) sh.T[r][u + 8 * x] = sh.T[r][u + 8 * x] - acc[x];
                } else {
#pragma unroll
                    for (int x = 0; x < 3; ++x)
                        if ((x < 2 || third) && dr[x] < nr && dc[x] < nc)
                            sh.T[dr[x]][dc[x]] = sh.T[dr[x]][dc[x]] - acc[x];
                }
            }
            // every thread has seen the same slots, so `good` is the CTA's
            if (!good) break;
            bar_sync<BAR_ALL, 256>();
            if (i == j) {
                if (lane == 0) mbar_arrive(&sh.pub[0]);  // the publisher may join the factor
                // row nc of this tile is the right-hand side
                for (int e = tid; e < NB * NB; e += 256) {
                    const int rr = e % NB, c = e / NB;
                    if (rr == nc && rr < nr && c < nc) sh.rhs[c] = sh.T[rr][c];
                    if (rr >= nc || c > rr) sh.T[rr][c] = 0.0;
                    sh.Di[rr][c] = 0.0;
                }
                bar_sync<BAR_ALL, 256>();
                factor_stream(sh, part, nc, c0, flags);
                // the right-hand-side row, by the panel solves' substitution:
                // warp 4 (whose columns of the inverse are the shortest) with
                // lane = column
                if (nr > nc && warp == 4) {
                    double v = lane < nc ? sh.rhs[lane] : 0.0;
                    for (int q = 0; q < nc; ++q) {
                        if (lane == q) v = v * sh.rp[q];
                        const double x = __shfl_sync(0xffffffffu, v, q);
                        if (lane > q && lane < nc) v = fma(-x, sh.T[lane][q], v);
                    }
                    if (lane < nc) M[(size_t)(c0 + lane) * ld + r0 + nc] = v;
                }
                // the inverse (for the backward sweep after this launch)
                if (j < ninv) invert_columns(sh.T, sh.Di, sh.rp, nc);
                else if (tid < nc) sh.Di[tid][tid] = sh.rp[tid];
                bar_sync<BAR_ALL, 256>();
                for (int e = tid; e < NB * NB; e += 256) Dinv[(size_t)j * NB * NB + e] = sh.Di[e / NB][e % NB];
            } else {
                // the panel solve, DFC columns at a time: within them by
                // warps 0 to DFC - 1 (one column each, lane = row), then the
                // later columns (a tile below a diagonal block has whole
                // columns, nc == NB). Column c is updated by warps c mod 8 and
                // (c + 4) mod 8 in turn; BAR_ALL is between them.
                for (int q = 0; q < DFQ; ++q) {
                    const int s = step % DFR, done = DFC * q;
                    good = take(s);
                    if (!good) break;
                    const DfSlot &sl = sh.slot[s];
                    if (u < DFC) {
                        double v = sh.T[r][done + u];
#pragma unroll
                        for (int h = 0; h < DFC; ++h) {
                            if (u == h) {
                                v = v * sl.rp[h];
                                sh.T[r][done + h] = v;
                            }
                            if (h < DFC - 1) {
                                bar_sync<BAR_STEP, 32 * DFC>();
                                if (u > h) v = fma(-sh.T[r][done + h], sl.a[done + u][h], v);
                            }
                        }
                    }
                    bar_sync<BAR_ALL, 256>();
                    if (lane == 0) mbar_arrive(&sh.pub[q]);
                    told = q + 1;
                    for (int c = done + DFC + u; c < NB; c += 8) {
                        double z = sh.T[r][c];
#pragma unroll
                        for (int h = 0; h < DFC; ++h) z = fma(-sh.T[r][done + h], sl.a[c][h], z);
                        sh.T[r][c] = z;
                    }
                    give(s);
                }
            }
        }
    }
    if (!good) {
        // tell the publisher to stop
        sh.stop = 1;
        __syncwarp();
        if (lane == 0)
            for (int q = told; q < DFQ; ++q) mbar_arrive(&sh.pub[q]);
    }
}

// CTAs of the data-flow factorization on the current device (one per SM at
// most, all resident), or 0 when a cooperative launch is not possible.
// Computed per device and published once, as for the backward sweep.
int df_capacity() {
    constexpr int kDevices = 64;
    static std::atomic<int> cap_plus1[kDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (dev < 0 || dev >= kDevices) return 0;
    int c = cap_plus1[dev].load(std::memory_order_acquire);
    if (c == 0) {
        int coop = 0, per_sm = 0, sms = 0, cap = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaFuncSetAttribute(chol_df_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(DfShared)) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chol_df_kernel, DF_THREADS, sizeof(DfShared)) !=
                cudaSuccess)
            cudaGetLastError();
        else if (coop && per_sm > 0)
            cap = sms;
        c = cap + 1;
        cap_plus1[dev].store(c, std::memory_order_release);
    }
    return c - 1;
}

int g_chol_path = 0;  // 0: data flow when possible, 1: multi-launch, 2: data flow only

// Words of the ready list for order n (with the right-hand-side row): one per
// diagonal block, one per tile, one abort word.
size_t df_ready_words(int n, int has_b) {
    const size_t nbc = (size_t)(n + NB - 1) / NB, nbr = (size_t)(n + has_b + NB - 1) / NB;
    return nbc + nbc * nbr + 1;
}

// The backward sweep of chol_backsolve_kernel on several CTAs (a cooperative launch): thread t
// of CTA k owns row 256 k + t of z, which is row n of M updated in place.
// Per 32-row block from the bottom, every CTA forms x_b = D_b^-T y_b in
// shared memory from the block's rows of z (final since the previous block),
// CTA 0 stores it, and the owners of the rows above subtract L_b^T x_b; every
// value takes the single-CTA sweep's FMAs in the same order, so the results
// are the same bits. A grid barrier closes each block; the next block's
// inverse is loaded into the other shared buffer before it.
__global__ void __launch_bounds__(256) chol_backsolve_coop_kernel(double *__restrict__ M, int n, int ld,
                                                                  const double *__restrict__ Dinv,
                                                                  double *__restrict__ x) {
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    __shared__ double Di[2][NB][NB + 1];  // this block's inverse and the next one's, loaded ahead
    __shared__ double yb[NB];
    __shared__ double xb[NB];
    const int tid = threadIdx.x;
    const int r = blockIdx.x * blockDim.x + tid;
    double *z = M + n;  // z[c] at z[c * ld]
    const int nblk = (n + NB - 1) / NB;
    for (int t = tid; t < NB * NB; t += blockDim.x)
        Di[(nblk - 1) & 1][t / NB][t % NB] = Dinv[(size_t)(nblk - 1) * NB * NB + t];
    for (int b = nblk - 1; b >= 0; --b) {
        const int r0 = b * NB, r1 = min(n, r0 + NB), u = b & 1;
        if (tid < NB) yb[tid] = (r0 + tid < r1) ? z[(size_t)(r0 + tid) * ld] : 0.0;
        __syncthreads();
        if (tid < r1 - r0) {
            const double v = sweep_dot(Di[u], yb, tid, r1 - r0);
            xb[tid] = v;
            if (blockIdx.x == 0) x[r0 + tid] = v;
        }
        __syncthreads();
        if (r < r0) z[(size_t)r * ld] = z[(size_t)r * ld] - sweep_row(M + (size_t)r * ld + r0, xb, r1 - r0);
        if (b > 0)
            for (int t = tid; t < NB * NB; t += blockDim.x)
                Di[u ^ 1][t / NB][t % NB] = Dinv[(size_t)(b - 1) * NB * NB + t];
        grid.sync();
    }
}

// The same sweep in one thread-block cluster of g <= 8 CTAs (orders up to
// 2048), block b of 32 rows on CTA b mod g with its z in shared memory. Per
// block from the bottom its owner forms x_b and sends it into every CTA's
// shared memory (st.async, one mbarrier and one place per block, so nothing is
// reused and no CTA waits for a slower one). Warps 0 to 3 of the owner of
// block b - 1 apply x_b to it as it arrives and go on to x_(b-1): that is the
// chain, one block's update and dot product per block. Warps 4 to 7 apply x_b
// to the CTA's blocks further up (in a CTA whose chain warps are at work, once
// they have sent x_(b-1): they share the FP64 units) and hand block q to the
// chain warps when x_(q+2) is in it. A dot product's four partial chains
// (sweep_dot, sweep_row) run on four lanes, eight FMAs each, instead of one
// after another on one: 65 cycles per FP64 instruction whatever the lanes.
// subst: the last block by substitution with its L and reciprocal pivots, 5000
// cycles once, instead of an inverse formed at the factorization's end.
//
// The waits are bounded, by `limit` polls. A thread whose wait runs out goes on
// without waiting, on whatever it has: every barrier is reached by all its threads
// and every x_b is sent, so nobody else is left standing, and the pivot status -1
// and the status word CHOL_WAIT_CODE tell the caller that x is not a solution. A CTA
// leaves when all that was sent to it has arrived: a store still under way would
// land in the shared memory of whatever runs there next.
__device__ __forceinline__ double chains_sum(double a) {
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    return a + __shfl_xor_sync(0xffffffffu, a, 2);  // (a0 + a1) + (a2 + a3)
}

constexpr int SWB = 8;                // blocks of a CTA
constexpr int SWN = 8 * SWB;          // blocks of the largest order
struct SweepShared {
    double z[SWB][NB], xb[SWN][NB], Di[2][NB][NB + 1];
    double rp[NB];                  // reciprocal pivots of the last block (with subst)
    uint64_t got[SWN], ready[SWB];  // x_b has arrived; a block has all but its last update
};
__global__ void __launch_bounds__(256, 1) chol_sweep_cluster_kernel(const double *__restrict__ M, int n, int ld,
                                                                    const double *__restrict__ Dinv,
                                                                    double *__restrict__ x,
                                                                    int *__restrict__ flags,
                                                                    int *__restrict__ info,
                                                                    unsigned *__restrict__ clear, int words,
                                                                    int subst, long long limit) {
    chain_wait();
    chain_open();
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    __shared__ SweepShared sh;
    const int g = (int)cl.num_blocks(), me = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31;
    const int row = 8 * ((tid >> 5) & 3) + (lane >> 2), ch = tid & 3;  // row of a block, partial chain
    const int nblk = (n + NB - 1) / NB;
    // the factorization's ready list, done with: zeros for the next one
    for (int t = 256 * me + tid; t < words; t += 256 * g) clear[t] = 0;
    for (int e = tid; e < SWB * NB; e += 256) {
        const int c = ((e / NB) * g + me) * NB + e % NB;
        sh.z[e / NB][e % NB] = c < n ? M[(size_t)c * ld + n] : 0.0;
    }
    if (tid < SWB) mbar_init(&sh.ready[tid], 4);
    if (tid < nblk) {
        mbar_init(&sh.got[tid], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(&sh.got[tid])),
                     "r"(8 * min(NB, n - NB * tid)));
    }
    auto load_inv = [&](int b, int t0, int nt) {
        for (int t = t0; t < NB * NB; t += nt) sh.Di[b & 1][t / NB][t % NB] = Dinv[(size_t)b * NB * NB + t];
    };
    if ((nblk - 1) % g == me) {
        const int b = nblk - 1, nb = n - NB * b;
        if (subst) {
            for (int t = tid; t < NB * NB; t += 256) {
                const int r = t % NB, c = t / NB;
                if (c <= r && r < nb) sh.Di[b & 1][r][c] = M[(size_t)(NB * b + c) * ld + NB * b + r];
            }
            if (tid < nb) sh.rp[tid] = Dinv[(size_t)b * NB * NB + tid * NB + tid];
        } else {
            load_inv(b, tid, 256);
        }
    }
    cl.sync();
    // this thread's values of rows of L_b^T for block q (4 k + ch)
    auto load_row = [&](int q, int b, double *v) {
        const double *col = M + (size_t)(NB * q + row) * ld + NB * b;
        if (NB * b + NB <= n)
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = col[4 * k + ch];
    };
    // z of block q minus those rows times x_b
    auto update = [&](int q, int b, const double *v) {
        const int nb = min(NB, n - NB * b);
        const double *xs = sh.xb[b];
        double a = 0.0;
        if (nb == NB) {
#pragma unroll
            for (int k = 0; k < 8; ++k) a = fma(v[k], xs[4 * k + ch], a);
        } else {
            const double *col = M + (size_t)(NB * q + row) * ld + NB * b;
            for (int k = 0; k < nb / 4; ++k) a = fma(col[4 * k + ch], xs[4 * k + ch], a);
            if (ch == 0)
                for (int c = nb / 4 * 4; c < nb; ++c) a = fma(col[c], xs[c], a);
        }
        a = chains_sum(a);
        if (ch == 0) sh.z[q / g][row] = sh.z[q / g][row] - a;
    };
    bool ok = true;
    if (tid < 128) {
        double pre[8];
        for (int b = nblk - 1; b >= 0; --b) {
            if (b % g == me) {
                const int nb = min(NB, n - NB * b), t = row, K = t < nb ? (nb - t) / 4 : 0;
                const double(*D)[NB + 1] = sh.Di[b & 1];
                const double *yb = sh.z[b / g];
                double a = 0.0;
                if (subst && b == nblk - 1) {
                    if (tid < 32) {
                        double v = lane < nb ? sh.z[b / g][lane] : 0.0;
                        for (int q = nb - 1; q >= 0; --q) {
                            const double l = D[q][min(lane, q)];
                            if (lane == q) v = v * sh.rp[q];
                            const double xq = __shfl_sync(0xffffffffu, v, q);
                            if (lane < q) v = fma(-l, xq, v);
                        }
                        if (lane < nb) sh.z[b / g][lane] = v;
                    }
                    asm volatile("bar.sync 1, 128;\n" ::: "memory");
                    if (t < nb) a = yb[t];
                } else {
                    for (int k = 0; k < K; ++k) a = fma(D[t + 4 * k + ch][t], yb[t + 4 * k + ch], a);
                    if (ch == 0)
                        for (int c = t + 4 * K; c < nb; ++c) a = fma(D[c][t], yb[c], a);
                    a = chains_sum(a);
                }
                if (t < nb) {
                    // lane ch of the row sends to CTAs ch, ch + 4
                    if (b > 0)
                        for (int r = ch; r < g; r += 4) {
                            uint32_t dst, bar;
                            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                                         : "=r"(dst)
                                         : "r"(smem_u32(&sh.xb[b][t])), "r"(r));
                            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                                         : "=r"(bar)
                                         : "r"(smem_u32(&sh.got[b])), "r"(r));
                            asm volatile(
                                "st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n" ::"r"(dst),
                                "l"(__double_as_longlong(a)), "r"(bar)
                                : "memory");
                        }
                    if (ch == 0) x[NB * b + t] = a;
                }
                asm volatile("bar.sync 1, 128;\n" ::: "memory");  // all have read the inverse: its buffer is free
            }
            if (b > 0 && (b - 1) % g == me) {
                load_inv(b - 1, tid, 128);
                load_row(b - 1, b, pre);
                // x_(b+1) and all before it are in the block (none when b is the last)
                if (b + 1 < nblk) ok = ok && mbar_wait(smem_u32(&sh.ready[(b - 1) / g]), 0u, limit);
                ok = ok && mbar_wait(smem_u32(&sh.got[b]), 0u, limit);
                update(b - 1, b, pre);
                asm volatile("bar.sync 1, 128;\n" ::: "memory");
            }
        }
    } else {
        for (int b = nblk - 1; b >= 2; --b) {
            // this CTA's blocks q <= b - 2, the next to be handed over first
            int q = b - 2 - ((b - 2 - me) % g + g) % g;
            if (q < 0) continue;
            double v[8];
            load_row(q, b, v);
            ok = ok && mbar_wait(smem_u32(&sh.got[b]), 0u, limit);
            if ((b - 1) % g == me) ok = ok && mbar_wait(smem_u32(&sh.got[b - 1]), 0u, limit);
            for (; q >= 0; q -= g) {
                update(q, b, v);
                if (q == b - 2) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.ready[q / g]);
                }
                if (q >= g) load_row(q - g, b, v);
            }
        }
    }
    // every x_b but x_0 goes to every CTA
    if (tid > 0 && tid < nblk && !mbar_wait(smem_u32(&sh.got[tid]), 0u)) ok = false;
    if (!ok) {
        atomicExch(flags, -1);
        atomicExch(flags + 1, CHOL_WAIT_CODE | 0x10000 | me);
    }
    cl.sync();  // (all have reported)
    if (info && me == 0 && tid == 0) *info = atomicAdd(flags, 0);
}

// Polls of a sweep's waits (irwls_debug_sweep_wait).
std::atomic<long long> g_sweep_wait{TC_WAIT_LIMIT};

// CTAs of the cooperative sweep for order n on the current device, or 0 when
// they cannot all be resident at once (the single-CTA sweep is used then).
// The capacity is computed per device from the device's own attributes (the
// library context need not exist: the allocation-free solve runs without it)
// and published only once computed; concurrent first calls compute the same
// value. Only errors of these queries are cleared, never one the caller left.
int coop_backsolve_ctas(int n) {
    constexpr int kDevices = 64;
    static std::atomic<int> cap_plus1[kDevices];  // 0: not computed yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (dev < 0 || dev >= kDevices) return 0;
    int c = cap_plus1[dev].load(std::memory_order_acquire);
    if (c == 0) {
        int coop = 0, per_sm = 0, sms = 0, cap = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chol_backsolve_coop_kernel, 256, 0) != cudaSuccess)
            cudaGetLastError();
        else if (coop)
            cap = per_sm * sms;
        c = cap + 1;
        cap_plus1[dev].store(c, std::memory_order_release);
    }
    const int g = (n + 255) / 256;
    return g <= c - 1 ? g : 0;
}

// Whether a cluster of g <= 8 CTAs of the sweep can run on the current device.
bool sweep_cluster_ok() {
    constexpr int kDevices = 64;
    static std::atomic<int> state[kDevices];  // 0: not known, 1: no, 2: yes
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (dev < 0 || dev >= kDevices) return false;
    int v = state[dev].load(std::memory_order_acquire);
    if (v == 0) {
        int has = 0;
        if (cudaDeviceGetAttribute(&has, cudaDevAttrClusterLaunch, dev) != cudaSuccess) {
            cudaGetLastError();
            has = 0;
        }
        v = has ? 2 : 1;
        state[dev].store(v, std::memory_order_release);
    }
    return v == 2;
}

int chol_enqueue_panels(double *d_M, int n, int ld, int nrows, int *flags, double *Dinv, cudaStream_t st);
int chol_enqueue_backsolve(double *d_M, int n, int ld, double *d_x, double *Dinv, int *flags, int *d_info,
                           cudaStream_t st, unsigned *clear, size_t words, bool chained, bool subst);

// Whether the cluster sweep takes order n.
bool cluster_sweep_for(int n) { return n <= 8 * SWB * NB && sweep_cluster_ok(); }

// Enqueues the whole factorization (and the solve with d_x) on `st`, with Dinv
// holding ceil(n/32) blocks of 32x32 doubles. Row n of M (the right-hand side) is
// scratch on return: which backward sweep runs decides what it holds.
// ready: the data-flow path's list (df_ready_words words, all zero; it is left all
// zero, by the cluster sweep or a memset: clearing it before the factorization
// instead cost each solve 4 us), or NULL for the multi-launch path. chained: the
// sweep may be a chained launch (a stream of this library). order: every block of the
// sweep through its inverse (irwls_dev_chol_solve_order).
// d_b: the right-hand side, or NULL when row n of M holds
// it. The pivot status starts at zero here; it goes to d_info (or NULL) too.
int chol_enqueue(double *d_M, int n, int ld, const double *d_b, double *d_x, int *flags, double *Dinv, int *d_info,
                 cudaStream_t st, unsigned *ready = nullptr, bool chained = false, bool order = false) {
    const int has_b = d_x != nullptr;
    const int nrows = n + has_b;
    const int G = ready && g_chol_path != 1 ? df_capacity() : 0;
    const bool subst = !order && cluster_sweep_for(n);
    cudaError_t e = cudaSuccess;
    if (G > 0) {
        // one cooperative launch of the data-flow factorization
        const size_t words = df_ready_words(n, has_b);
        const int nbc = (n + NB - 1) / NB, nbr = (nrows + NB - 1) / NB;
        const int tasks = nbc * (2 * nbr - nbc + 1) / 2;
        int grid = std::min(G, tasks);
        int *abort = (int *)(ready + words - 1);
        const double *b = has_b ? d_b : nullptr;
        int ninv = has_b ? nbc - subst : 0;
        void *args[] = {&d_M, &n, &ld, (void *)&nrows, &b, &flags, &Dinv, &ready, &abort, &ninv};
        e = cudaLaunchCooperativeKernel((const void *)chol_df_kernel, dim3(grid), dim3(DF_THREADS), args,
                                            sizeof(DfShared), st);
        if (e != cudaSuccess) {
            irwls_set_error(-2, "CUDA error in chol_df (cooperative): %s", cudaGetErrorString(e));
            return -2;
        }
        irwls_count_launch(1);
        if (has_b && cluster_sweep_for(n)) {
            const int rc = chol_enqueue_backsolve(d_M, n, ld, d_x, Dinv, flags, d_info, st, ready, words, chained, subst);
            if (rc) cudaMemsetAsync(ready, 0, words * sizeof(unsigned), st);
            return rc;
        }
        e = cudaMemsetAsync(ready, 0, words * sizeof(unsigned), st);
        if (e != cudaSuccess) {
            irwls_set_error(-2, "CUDA error clearing the ready list: %s", cudaGetErrorString(e));
            return -2;
        }
    } else if (g_chol_path == 2) {
        irwls_set_error(-2, "the data-flow Cholesky needs a cooperative launch");
        return -2;
    } else {
        e = cudaMemsetAsync(flags, 0, sizeof(int), st);
        if (e == cudaSuccess && d_b && has_b)  // b becomes row n: M[c*ld + n] = b[c]
            e = cudaMemcpy2DAsync(d_M + n, (size_t)ld * sizeof(double), d_b, sizeof(double), sizeof(double), n,
                                  cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) {
            irwls_set_error(-2, "rhs copy: %s", cudaGetErrorString(e));
            return -2;
        }
        const int rc = chol_enqueue_panels(d_M, n, ld, nrows, flags, Dinv, st);
        if (rc) return rc;
    }
    if (has_b) return chol_enqueue_backsolve(d_M, n, ld, d_x, Dinv, flags, d_info, st, nullptr, 0, false, subst);
    if (d_info && (e = cudaMemcpyAsync(d_info, flags, sizeof(int), cudaMemcpyDeviceToDevice, st)) != cudaSuccess) {
        irwls_set_error(-2, "pivot status: %s", cudaGetErrorString(e));
        return -2;
    }
    return 0;
}

// The multi-launch factorization: per panel a solve launch and an update
// launch (whose tile (0, 0) factors the next diagonal block).
int chol_enqueue_panels(double *d_M, int n, int ld, int nrows, int *flags, double *Dinv, cudaStream_t st) {
    chol_factor0_kernel<<<1, 256, 0, st>>>(d_M, n, ld, flags, Dinv);
    IRWLS_LAUNCH_CHECK("chol_factor0");
    for (int k0 = 0; k0 < n; k0 += NB) {
        const int nb = min(NB, n - k0);
        const int below = nrows - (k0 + nb);
        if (below <= 0) break;
        chol_trsm_kernel<<<ceil_div(below, 8), 256, 0, st>>>(d_M, ld, k0, nb, nrows,
                                                             Dinv + (size_t)(k0 / NB) * NB * NB);
        IRWLS_LAUNCH_CHECK("chol_trsm");
        if (k0 + nb < n) {
            dim3 g(ceil_div(n - (k0 + nb), 32), ceil_div(below, 32));
            chol_update_kernel<<<g, 256, 0, st>>>(d_M, n, ld, k0, nb, nrows, flags,
                                                  Dinv + (size_t)(k0 / NB + 1) * NB * NB);
            IRWLS_LAUNCH_CHECK("chol_update");
        }
    }
    return 0;
}

// The backward sweep L^T x = z (z in row n of M): the cluster form up to order
// 2048, the cooperative one above, one CTA where neither can run. They give
// the same bits.
int chol_enqueue_backsolve(double *d_M, int n, int ld, double *d_x, double *Dinv, int *flags, int *d_info,
                           cudaStream_t st, unsigned *clear, size_t words, bool chained, bool subst) {
    {
        if (cluster_sweep_for(n)) {
            // two blocks a CTA, up to eight CTAs: one block's update holds the
            // FP64 units for 0.45 us, the chain of a block takes about 1.3
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(std::min(8, (n + 2 * NB - 1) / (2 * NB)));
            cfg.blockDim = dim3(256);
            cfg.stream = st;
            cudaLaunchAttribute at[2];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = cfg.gridDim.x;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = at;
            cfg.numAttrs = chained ? 2 : 1;
            const cudaError_t e = cudaLaunchKernelEx(&cfg, chol_sweep_cluster_kernel, (const double *)d_M, n, ld,
                                                     (const double *)Dinv, d_x, flags, d_info, clear, (int)words, (int)subst,
                                                     g_sweep_wait.load());
            if (e != cudaSuccess) {
                irwls_set_error(-2, "CUDA error in chol_sweep (cluster): %s", cudaGetErrorString(e));
                return -2;
            }
            irwls_count_launch(1);
            return 0;
        }
        cudaError_t ei = cudaSuccess;
        if (d_info) ei = cudaMemcpyAsync(d_info, flags, sizeof(int), cudaMemcpyDeviceToDevice, st);
        if (ei != cudaSuccess) {
            irwls_set_error(-2, "pivot status: %s", cudaGetErrorString(ei));
            return -2;
        }
        const int g = coop_backsolve_ctas(n);
        if (g > 0) {
            void *args[] = {&d_M, &n, &ld, &Dinv, &d_x};
            const cudaError_t e = cudaLaunchCooperativeKernel((const void *)chol_backsolve_coop_kernel, dim3(g),
                                                              dim3(256), args, 0, st);
            if (e != cudaSuccess) {
                irwls_set_error(-2, "CUDA error in chol_backsolve (cooperative): %s", cudaGetErrorString(e));
                return -2;
            }
            irwls_count_launch(1);
            return 0;
        }
        const size_t smem = (size_t)n * sizeof(double);
        if (smem > 48 * 1024) {
            if (smem > 160 * 1024) {
                irwls_set_error(-6, "system of order %d exceeds the backward-solve tile", n);
                return -6;
            }
            allow_smem(chol_backsolve_kernel);
        }
        chol_backsolve_kernel<<<1, 256, smem, st>>>(d_M, n, ld, Dinv, d_x);
        IRWLS_LAUNCH_CHECK("chol_backsolve");
    }
    return 0;
}


}  // namespace

extern "C" int irwls_dev_zero_upper(double *d_M, int n, int ld) {
    if (n <= 1) return 0;
    zero_upper_kernel<<<ceil_div((long long)n * n, 256) < 4096 ? ceil_div((long long)n * n, 256) : 4096, 256, 0,
                        irwls_stream()>>>(d_M, n, ld);
    IRWLS_LAUNCH_CHECK("zero_upper");
    return 0;
}

static int chol_solve(double *d_M, int n, int ld, const double *d_b, double *d_x, bool order) {
    if (n <= 0) return 0;
    if (ld < n + 1) {
        irwls_set_error(-6, "Cholesky leading dimension %d < n + 1 = %d", ld, n + 1);
        return -6;
    }
    int *flags = irwls_dev_flags();
    const int npanel = ceil_div(n, NB);
    // factored diagonal blocks: the context's grow-only scratch slot 0
    double *diag = (double *)irwls_ctx_scratch(0, (size_t)npanel * NB * NB * sizeof(double));
    if (!diag) return -3;
    // ready list of the data-flow path: the context's grow-only slot 3
    unsigned *ready = (unsigned *)irwls_ctx_scratch_zeroed(3, df_ready_words(n, d_x != nullptr) * sizeof(unsigned));
    if (!ready) return -3;
    if (irwls_prof_on()) irwls_prof_begin(IRWLS_PROF_CHOL);
    int rc = chol_enqueue(d_M, n, ld, d_b, d_x, flags, diag, nullptr, irwls_stream(), ready, true, order);
    if (rc) return rc;
    if (irwls_prof_on()) irwls_prof_end(IRWLS_PROF_CHOL);
    return 0;
}

extern "C" int irwls_dev_chol_solve(double *d_M, int n, int ld, const double *d_b, double *d_x) {
    return chol_solve(d_M, n, ld, d_b, d_x, false);
}

// The same with the backward sweep's last block through its inverse as the others,
// for callers whose results move far beyond its rounding (IRWLSpar on SGMA
// centroids can multiply that by 10^8).
extern "C" int irwls_dev_chol_solve_order(double *d_M, int n, int ld, const double *d_b, double *d_x) {
    return chol_solve(d_M, n, ld, d_b, d_x, true);
}

extern "C" int irwls_chol_sweep_ctas(int n) { return coop_backsolve_ctas(n); }

// Test hook: 0 = the data-flow factorization where a cooperative launch is
// possible (default), 1 = the multi-launch factorization, 2 = data flow only.
extern "C" void irwls_debug_chol_path(int mode) { g_chol_path = mode >= 0 && mode <= 2 ? mode : 0; }

// Test hook: polls of the cluster sweep's waits (0: each runs out at once; below: the
// default).
extern "C" void irwls_debug_sweep_wait(long long polls) { g_sweep_wait.store(polls >= 0 ? polls : TC_WAIT_LIMIT); }

// -1 in *info: a bounded wait of the solve ran out.
extern "C" int irwls_dev_pivot_status(int *info) {
    *info = 0;
    cudaError_t e = cudaMemcpyAsync(info, irwls_dev_flags(), sizeof(int), cudaMemcpyDeviceToHost, irwls_stream());
    if (e == cudaSuccess) e = cudaStreamSynchronize(irwls_stream());
    if (e != cudaSuccess) {
        irwls_set_error(-2, "CUDA error reading the pivot status: %s", cudaGetErrorString(e));
        return -2;
    }
    return 0;
}

namespace {
// out = A v (trans = 0) or out = A^T v (trans = 1) for a column-major size x
// size matrix; one warp per output entry.
__global__ void gemv_kernel(const double *__restrict__ A, const double *__restrict__ v, double *__restrict__ out,
                            int size, int trans) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= size) return;
    double acc = 0.0;
    if (trans)
        for (int i = lane; i < size; i += 32) acc = fma(A[(size_t)w * size + i], v[i], acc);
    else
        for (int j = lane; j < size; j += 32) acc = fma(A[(size_t)j * size + w], v[j], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[w] = acc;
}
}  // namespace

extern "C" int irwls_dev_gemv(const double *d_A, const double *d_v, double *d_out, int size, int trans) {
    if (size <= 0) return 0;
    gemv_kernel<<<ceil_div((long long)size * 32, 256), 256, 0, irwls_stream()>>>(d_A, d_v, d_out, size, trans);
    IRWLS_LAUNCH_CHECK("gemv");
    return 0;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the Cholesky solve.
//
// Some callers cannot let a library allocate device memory while they run: a
// serving process that reserved the device's memory for its own pool
// allocator at start-up (a cudaMalloc in the middle of a request can fail, or
// force the pool to give memory back), or a latency-sensitive caller for whom
// cudaMalloc/cudaFree must not run because they can synchronize the whole
// device. irwls_chol_solve_noalloc serves them: the caller passes the matrix,
// the right-hand side and the output (all device memory the caller owns) and a
// stream, and the call itself allocates nothing. Its only scratch is the
// file-scope array below, which every GPU that loads this library holds until
// the process exits.
//
// The scratch keeps the inverted 32x32 diagonal blocks (one per panel), the
// status words and the ready list of the data-flow factorization, which
// sizes it for matrices of order up to IRWLS_NOALLOC_MAX_ORDER (4096: 1 MiB
// of blocks and 65 KiB of ready words, about 1.06 MiB in all).
// ---------------------------------------------------------------------------
#define IRWLS_NOALLOC_MAX_ORDER 4096
#define IRWLS_NOALLOC_PANELS (IRWLS_NOALLOC_MAX_ORDER / NB)
// ready words of the data-flow factorization at the largest order (with the
// right-hand-side row), rounded up to whole doubles
#define IRWLS_NOALLOC_READY (IRWLS_NOALLOC_PANELS + IRWLS_NOALLOC_PANELS * (IRWLS_NOALLOC_PANELS + 1) + 1)

static __device__ __align__(256) double
    g_noalloc_scratch[IRWLS_NOALLOC_PANELS * NB * NB + 32 + (IRWLS_NOALLOC_READY + 1) / 2];

#define IRWLS_NOALLOC_DEVICES 64
static double *g_noalloc_addr[IRWLS_NOALLOC_DEVICES];  // device address of the array, per device

extern "C" int irwls_chol_solve_noalloc(double *d_M, int n, int ld, const double *d_b, double *d_x, int *d_info,
                                        void *stream) {
    irwls_clear_error();
    // A CUDA error the caller left pending would be taken for one of this
    // call's launches (each launch is checked with cudaGetLastError, which
    // clears it): refuse instead, and leave the caller's error in place.
    cudaError_t pending = cudaPeekAtLastError();
    if (pending != cudaSuccess) {
        irwls_set_error(-14, "irwls_chol_solve_noalloc: a CUDA error is already pending (%s); not cleared",
                        cudaGetErrorString(pending));
        return -14;
    }
    if (n <= 0) return 0;
    if (n > IRWLS_NOALLOC_MAX_ORDER) {
        irwls_set_error(-11, "irwls_chol_solve_noalloc: order %d exceeds its limit of %d", n, IRWLS_NOALLOC_MAX_ORDER);
        return -11;
    }
    if (ld < n + 1) {
        irwls_set_error(-6, "irwls_chol_solve_noalloc: leading dimension %d < n + 1 = %d", ld, n + 1);
        return -6;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= IRWLS_NOALLOC_DEVICES) {
        irwls_set_error(-2, "irwls_chol_solve_noalloc: no usable current device (%s)", cudaGetErrorString(e));
        return -2;
    }
    // Set-up, once per device, with that device current: the host-side name
    // of the array is not a device address, so ask the runtime for it.
    if (!g_noalloc_addr[dev]) {
        double *p = nullptr;
        e = cudaGetSymbolAddress((void **)&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            irwls_set_error(-2, "irwls_chol_solve_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return -2;
        }
        g_noalloc_addr[dev] = p;
    }
    double *diag = g_noalloc_addr[dev];
    int *flags = (int *)(diag + IRWLS_NOALLOC_PANELS * NB * NB);
    unsigned *ready = (unsigned *)(diag + IRWLS_NOALLOC_PANELS * NB * NB + 32);
    cudaStream_t st = (cudaStream_t)stream;
    // order <= 4096: the backward sweep's vector fits the default 48 KiB
    return chol_enqueue(d_M, n, ld, d_b, d_x, flags, diag, d_info, st, ready);
}
