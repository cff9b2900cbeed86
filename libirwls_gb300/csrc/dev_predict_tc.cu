// dev_predict_tc.cu -- RBF row sums f_i = b + sum_j w_j k(t_i, s_j) with
// FP64-accurate kernel values from the tensor cores and the integer pipe: the
// plain form's prediction (reference src/LIBIRWLS-predict.c:56-131) and the error
// updates of its full training (src/full-train.c:436-510).
//
// On the FP64 pipe a kernel value costs two instructions per stored feature and
// 16 for its exponential, 5.5 ms for 20000 rows against 3000 vectors of 12
// stored features, all of it at that pipe's peak. Here:
//
// 1. Each row (of either set) gets a power of two sigma >= its norm |x| and
//    every value becomes the integer N = round(x / sigma 2^55), in 7 balanced
//    base-256 digits, exact in bf16 (as the operands of the plain Gram,
//    dev_gram_tc.cu; values of at least sigma / 4 exactly, the others within
//    2^-56 sigma).
// 2. A CTA takes a 128-row tile against 64-vector tiles: per 16 features the 33
//    digit pairs of the levels u >= 5 go to 8 accumulators of 128 x 64 FP32 in
//    tensor memory, every partial sum an integer below 2^24 over 96 features;
//    the levels combine to the integer T = sum N N' 2^-48 (the dropped levels
//    weigh below 2^-61 sigma sigma' per feature).
// 3. y = log2(e) gamma (q_i + q_j) - 2 log2(e) gamma sigma_i sigma_j 2^-62 T
//    in 64-bit fixed point (its unit 2^-56, or below 2^-56 of the largest term, but
//    no coarser than FP64 sums of the nearest rows: fixed_point_of), then
//    2^-y by exp2_fixed. The value times w_j is added in FP64, in vector order
//    per strip of 16 of every 64 vectors; the strips' sums in a fixed order.
//
// Against a 64-bit evaluation the decision values are within 2.5e-16 of their
// size, the ordered FP64 sums within 1.5e-15 (20000 one-hot rows of 54 features,
// 3000 vectors). Those take 5475 us of kernel time, this 456 us and 50 us of
// preparation. Bound: the epilogue's integer instructions (about 120 per value,
// 41 % of the issue slots, latency between them the rest); the MMAs (33 x 32
// cycles per 16 features of a tile pair) run while the epilogue forms the kernel
// values of the tile before (480 us when it held the accumulators for them).
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "dev_common.cuh"
#include "exp2_fixed.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int PS = 7;                          // digits per value
constexpr int PM = 128, PN = 64, PK = 16;      // rows x vectors of a tile pair, features per stage
constexpr int PPIECE = PM * PK;                // elements of one digit piece (4 KB)
constexpr int PNS = 5;                         // ring stages
constexpr int PLEV = 8;                        // kept levels (u = 5 ... 12)
constexpr int PDRAIN = 6;                      // stages between drains (96 features)
constexpr uint32_t PA_STAGE = PS * PPIECE * 2;     // 28 KB
constexpr uint32_t PB_PIECE = PN * PK * 2;         // 2 KB
constexpr uint32_t P_STAGE = PA_STAGE + PS * PB_PIECE;
static_assert(7LL * PDRAIN * PK * 128 * 128 < (1LL << 24), "level sums must stay exact");
static_assert((5LL * 256 + 6) * PDRAIN * PK * 128 * 128 < (1LL << 31), "levels 3 and 2 combine in 32 bits");

// Element offset of (row r of the 128-row tile, k of the 16-feature block) in a piece.
__device__ __forceinline__ int ppiece_off(int r, int k) { return (r >> 3) * 128 + (k >> 3) * 64 + (r & 7) * 8 + (k & 7); }

constexpr int TOPS = 4;  // words of a set's maxima (row_scales_kernel)

// Per row: e with 2^e >= |x| (-2000: a zero row), and over the set the largest
// |q| (with q) and the largest |x|^2 (floats rounded up a little, as bits), with w
// the high half of the largest |w|, and with q the complement of the smallest |q|
// (rounded down); with rp that of infinity where a row's
// indices do not increase (a vector that names a feature twice: its products add
// both). One warp per row.
__global__ void __launch_bounds__(256) row_scales_kernel(const double *__restrict__ X, int ld, int width,
                                                         const double *__restrict__ q,
                                                         const double *__restrict__ w, const int *__restrict__ rp,
                                                         const int *__restrict__ ci, int n, int *__restrict__ ex,
                                                         unsigned *__restrict__ top) {
    __shared__ unsigned big[TOPS];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < TOPS) big[threadIdx.x] = 0;
    __syncthreads();
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const double *row = X + (size_t)i * ld;
        unsigned long long mx = 0;
        for (int t = lane; t < width; t += 32) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(row[t]) & 0x7fffffffffffffffULL;
            mx = b > mx ? b : mx;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long b = __shfl_xor_sync(0xffffffffu, mx, o);
            mx = b > mx ? b : mx;
        }
        const int E = (int)(mx >> 52);  // (subnormal rows count as zero)
        const int e = E == 0 ? -2000 : E - 1023 + ((mx & ((1ULL << 52) - 1)) != 0 ? 1 : 0);
        // |x|^2 / 4^e in FP32: values scaled by their exponent difference
        float rho = 0.f;
        if (E != 0) {
            for (int t = lane; t < width; t += 32) {
                const unsigned long long b = (unsigned long long)__double_as_longlong(row[t]) & 0x7fffffffffffffffULL;
                const int d = (int)(b >> 52) - 1023 - e;
                if ((b >> 52) != 0 && d > -60) {
                    const float m = __uint_as_float(0x3f800000u | (uint32_t)((b >> 29) & 0x7fffffu));
                    const float x = ldexpf(m, d);
                    rho = fmaf(x, x, rho);
                }
            }
            for (int o = 16; o > 0; o >>= 1) rho += __shfl_xor_sync(0xffffffffu, rho, o);
        }
        bool bad = false;
        if (rp)
            for (int t = rp[i] + 1 + lane; t < rp[i + 1]; t += 32) bad |= ci[t] <= ci[t - 1];
        bad = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            const float up = 1.001f;  // (the row's sum was rounded: at most 12288 terms over 32 lanes)
            // |x|^2 / 4^e <= rho: e grows by half of log2(rho), up
            const int grow = E == 0 ? 0 : (ilogbf(rho * up) >> 1) + 1;
            ex[i] = E == 0 ? -2000 : e + max(grow, 0);
            // (the order of non-negative floats is that of their bits; an
            // overflow to infinity makes the caller take the other path)
            if (q) {
                atomicMax(big, __float_as_uint(fabsf((float)q[i]) * up));
                atomicMax(big + 3, ~__float_as_uint(fabsf((float)q[i]) * 0.999f));
            }
            atomicMax(big + 1, __float_as_uint(E == 0 ? 0.f : ldexpf(rho * up, 2 * e)));
            if (w || bad) atomicMax(big + 2, bad ? 0x7ff00000u : (unsigned)__double2hiint(w[i]) & 0x7fffffffu);
        }
    }
    __syncthreads();
    if (threadIdx.x < TOPS && big[threadIdx.x]) atomicMax(top + threadIdx.x, big[threadIdx.x]);
}

// round(x 2^(55 - e)) for |x| <= 2^e, ties away from zero.
__device__ __forceinline__ long long fixed55(double x, int e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((b >> 52) & 0x7ff);
    if (E == 0) return 0;
    // x = M 2^(E - 1075)
    const unsigned long long M = (b & ((1ULL << 52) - 1)) | (1ULL << 52);
    const int sh = 1075 + e - 55 - E;  // >= -3 since |x| <= 2^e
    long long N = 0;
    if (sh <= 0) N = (long long)(M << min(-sh, 3));
    else if (sh < 64) N = (long long)((M + (1ULL << (sh - 1))) >> sh);
    return (b >> 63) ? -N : N;
}

// The digits of 8 features of a row in one 16-byte store per piece. Rows >= n
// and features >= width are zeros.
__global__ void __launch_bounds__(256) row_slice_kernel(const double *__restrict__ X, int ld, int width, int n,
                                                        const int *__restrict__ ex, int rows, int npb,
                                                        __nv_bfloat16 *__restrict__ S) {
    __shared__ uint16_t bf[257];  // bf16 bits of -128 ... 128
    for (int t = threadIdx.x; t < 257; t += 256) {
        const __nv_bfloat16 h = __float2bfloat16_rn((float)(t - 128));
        bf[t] = *(const uint16_t *)&h;
    }
    __syncthreads();
    const long long items = (long long)rows * npb * 2;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < items;
         t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t % rows);
        const long long g = t / rows;  // 8-feature group
        const int e = i < n ? ex[i] : -2000;
        uint32_t w[PS][4];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = (int)g * 8 + k;
            long long N = 0;
            if (e > -2000 && c < width) N = fixed55(X[(size_t)i * ld + c], e);
#pragma unroll
            for (int s = 0; s < PS; ++s) {
                int d;
                if (s < PS - 1) {
                    d = (int)(N & 255);
                    if (d >= 128) d -= 256;
                    N = (N - d) >> 8;
                } else {
                    d = (int)N;  // |d| <= 128
                }
                const uint32_t hb = bf[d + 128];
                if (k & 1) w[s][k >> 1] |= hb << 16;
                else w[s][k >> 1] = hb;
            }
        }
        const int pb = (int)(g >> 1), half = (int)(g & 1);
        const size_t base = (((size_t)(i >> 7) * npb + pb) * PS) * PPIECE + ppiece_off(i & 127, half * 8);
#pragma unroll
        for (int s = 0; s < PS; ++s)
            *(uint4 *)(S + base + (size_t)s * PPIECE) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    }
}

__global__ void row_norms_kernel(const double *__restrict__ q, int n, unsigned long long cg, int ec, int fb,
                                 long long *__restrict__ a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = fixed_scaled(q[i], cg, ec, fb);
}

// The same of the row's own fixed point, for raw rows (their kernel is that of the
// differences: FP64 norms would leave c |x|^2 2^-53 of them, the integers leave
// units of y): T_ii = sum N N 2^-48, in the products' unit, summed to 2^-32 of it
// before it is rounded (a product's floor per feature put all of a set's values
// 3.2e-15 off at 784 features). A warp per row.
__global__ void __launch_bounds__(256) row_norms_raw_kernel(const double *__restrict__ X, int ld, int width, int n,
                                                            const int *__restrict__ ex, unsigned long long cg, int ec,
                                                            int fb, long long *__restrict__ a) {
    const int lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const int e = ex[i];
        long long T = 0, low = 0;
        if (e > -2000)
            for (int t = lane; t < width; t += 32) {
                const long long N = fixed55(X[(size_t)i * ld + t], e) << 8;
                T += __mul64hi(N, N);
                low += (unsigned long long)(N * N) >> 32;
            }
        for (int o = 16; o > 0; o >>= 1) {
            T += __shfl_xor_sync(0xffffffffu, T, o);
            low += __shfl_xor_sync(0xffffffffu, low, o);
        }
        T += (low + (1LL << 31)) >> 32;
        // c |x|^2 2^fb = T cg 2^(2 e - 62 - ec + fb)
        const int sh = -(2 * e + 2 - ec + fb);
        const long long m = (long long)__umul64hi((unsigned long long)T, cg);
        if (lane == 0) a[i] = e <= -2000 ? 0 : sh <= 0 ? m << min(-sh, 3) : sh < 64 ? (m >> (sh - 1)) + 1 >> 1 : 0;
    }
}

struct PredictArgs {
    const __nv_bfloat16 *T, *S;  // digit slices of the rows and of the vectors
    int npb;                     // 16-feature blocks
    int n, nsv, per, P;          // rows, vectors, vector tiles per chunk, chunks
    const int *nsvp;             // the number of vectors on the device (at most nsv), or NULL
    const int *et, *es;          // row and vector scales
    const long long *at, *as;    // norm terms
    const double *w;
    int fb, emax, shr;           // unit of y; the largest e_j; y's product part is
    unsigned long long g;        //   (T g_j 2^-64) 2^(e_i - shr) with g_j = g 2^(e_j - emax)
    double *part;                // [strip][row]: strips of P chunks x column groups
};

// EW = 16 epilogue warps: 128 rows x 4 groups of 16 vectors. MULTI: more than
// 96 features, several drains per tile pair. FB: as exp2_fixed.
template <bool MULTI, int FB>
__global__ void __launch_bounds__(128 + 32 * 16, 1) predict_tc_kernel(PredictArgs p, int *flags) {
    constexpr int EW = 16, CW = PN / (EW / 4);  // columns of a group
    extern __shared__ __align__(1024) unsigned char p_smem[];
    __shared__ __align__(8) uint64_t full[PNS], empty[PNS], accf, acce, done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ unsigned long long table[256];
    __shared__ double sw[2][PN];
    __shared__ __align__(16) ulonglong2 sag[2][PN];  // norm term, multiplier of T
    unsigned char *smem = p_smem + ((1024 - (smem_u32(p_smem) & 1023)) & 1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = blockIdx.x, z = blockIdx.y;
    const int nsv = p.nsvp ? p.nsvp[0] : p.nsv;
    const int nt = (nsv + PN - 1) / PN;
    const int j0 = z * p.per, jn = max(0, min(nt, j0 + p.per) - j0);
    const int nd = (p.npb + PDRAIN - 1) / PDRAIN;  // drains per tile pair
    const int nst = jn * p.npb;
    for (int t = threadIdx.x; t < 256; t += blockDim.x) table[t] = exp2_table_entry(t);
    if (threadIdx.x == 0) {
        for (int b = 0; b < PNS; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], 1);
        }
        mbar_init(&accf, 1);
        mbar_init(&acce, EW);
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::);
        abort_flag = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        // producer: a stage's A pieces in one copy, the B half-pieces one by one
        if (lane == 0) {
            const uint32_t base = smem_u32(smem);
            int issued = 0;
            for (int u = 0; u < nst && !abort_flag; ++u) {
                const int jt = j0 + u / p.npb, kb = u % p.npb, slot = u % PNS;
                if (u >= PNS && !mbar_wait(smem_u32(&empty[slot]), (uint32_t)(u / PNS - 1) & 1u)) abort_flag = 1;
                if (abort_flag) break;
                const __nv_bfloat16 *A = p.T + ((size_t)I * p.npb + kb) * PS * PPIECE;
                const __nv_bfloat16 *B = p.S + ((size_t)(jt >> 1) * p.npb + kb) * PS * PPIECE + (jt & 1) * (PN / 8) * 128;
                const uint32_t sb = base + slot * P_STAGE, fbar = smem_u32(&full[slot]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fbar), "r"(P_STAGE));
                bulk_g2s(sb, A, PA_STAGE, fbar);
#pragma unroll
                for (int s = 0; s < PS; ++s)
                    bulk_g2s(sb + PA_STAGE + s * PB_PIECE, B + (size_t)s * PPIECE, PB_PIECE, fbar);
                issued = u + 1;
            }
            for (int u = issued > PNS ? issued - PNS : 0; u < issued; ++u)
                if (!mbar_wait(smem_u32(&full[u % PNS]), (uint32_t)(u / PNS) & 1u)) abort_flag = 1;
        }
        __syncwarp();
    } else if (warp == 1) {
        // MMA issue: level u - 5 += sum_{s+t=u} A_s B_t (as the plain Gram)
        if (lane == 0) {
            const uint32_t base = smem_u32(smem);
            int blk = 0;  // drain blocks so far
            for (int u = 0; u < nst && !abort_flag; ++u) {
                const int kb = u % p.npb, kin = kb % PDRAIN;
                if (kin == 0 && blk >= 1 && !mbar_wait(smem_u32(&acce), (uint32_t)(blk - 1) & 1u)) {
                    abort_flag = 1;
                    break;
                }
                const int slot = u % PNS;
                if (!mbar_wait(smem_u32(&full[slot]), (uint32_t)(u / PNS) & 1u)) {
                    abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
                const uint32_t sa = base + slot * P_STAGE, sbb = sa + PA_STAGE;
#pragma unroll
                for (int s = PS - 1; s >= 0; --s) {
                    const uint64_t da = tc_desc_lbo_sbo(sa + s * (PPIECE * 2), 128, 256);
                    const bool lone = s == PS - 2;  // (PS - 2, 0) alone starts the lowest level
#pragma unroll
                    for (int t0 = s < 5 ? 5 - s : 0; t0 < PS; t0 += (lone && t0 == 0) ? 1 : 4) {
                        const int np = lone && t0 == 0 ? 1 : PS - t0 < 4 ? PS - t0 : 4;
                        const uint64_t db = tc_desc_lbo_sbo(sbb + t0 * PB_PIECE, 128, 256);
                        const bool acc = kin > 0 || !(s == PS - 1 || (lone && t0 == 0));
                        mma_bf16(tmem + (uint32_t)(s + t0 - 5) * PN, da, db, tc_idesc(PM, PN * np), acc ? 1u : 0u);
                    }
                }
                tc_commit(&empty[slot]);
                if (kin == PDRAIN - 1 || kb == p.npb - 1) {
                    tc_commit(&accf);
                    ++blk;
                }
            }
            tc_commit(&done);
            if (!mbar_wait(smem_u32(&done), 0u)) abort_flag = 1;
        }
        __syncwarp();
    } else if (warp >= 4) {
        const int qr = warp & 3, gr = (warp - 4) >> 2, et = threadIdx.x - 128;
        const int row = PM * I + 32 * qr + lane;
        const bool live = row < p.n;
        const int shift = live ? min(p.shr - p.et[row], 63) : 63;
        const long long ai = live ? p.at[row] : 0;
        double sum = 0.0, nw = 0.0;
        ulonglong2 ng = {0, 0};
        long long T[CW];
        // vector et of tile t into registers (past the end: weight 0, 2^-y <= 1)
        auto fetch = [&](int t) {
            const int j = PN * t + et;
            nw = j < nsv ? p.w[j] : 0.0;
            ng.x = j < nsv ? (unsigned long long)p.as[j] : 1ULL << 62;
            ng.y = j < nsv ? p.g >> min(p.emax - p.es[j], 63) : 0;
        };
        if (et < PN && jn > 0) {
            fetch(j0);
            sw[0][et] = nw;
            sag[0][et] = ng;
        }
        bool stop = false;
        int blk = 0;
        for (int jj = 0; jj < jn && !stop; ++jj) {
            const double *w = sw[jj & 1];
            const ulonglong2 *ag = sag[jj & 1];
            if (et < PN && jj + 1 < jn) fetch(j0 + jj + 1);
            if (MULTI)
#pragma unroll
                for (int c = 0; c < CW; ++c) T[c] = nd >> 1;  // (l[0] >> 8 takes half a unit off per drain)
            for (int d = 0; d < nd; ++d, ++blk) {
                // (this barrier also publishes the tile's vectors, and after it
                // nobody reads the other buffer)
                const bool got = mbar_wait(smem_u32(&accf), (uint32_t)blk & 1u);
                const int bad = (!got || abort_flag) ? 1 : 0;
                int any;
                asm volatile(
                    "{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\nselp.s32 %0, 1, 0, q;\n}\n"
                    : "=r"(any)
                    : "r"(bad), "n"(32 * EW)
                    : "memory");
                if (any) {
                    stop = true;  // (the same in every epilogue thread)
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
                const uint32_t lanes = tmem + ((uint32_t)(32 * qr) << 16) + CW * gr;
                if (et < PN && d == 0) {
                    sw[(jj & 1) ^ 1][et] = nw;
                    sag[(jj & 1) ^ 1][et] = ng;
                }
#pragma unroll
                for (int c4 = 0; c4 < CW; c4 += 4) {
                    uint32_t L[PLEV][4];
#pragma unroll
                    for (int v = 0; v < PLEV; ++v)
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                                     : "=r"(L[v][0]), "=r"(L[v][1]), "=r"(L[v][2]), "=r"(L[v][3])
                                     : "r"(lanes + v * PN + c4));
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::);
                    if (c4 + 4 == CW) {
                        // the last read of this block: the next may start
                        asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
                        if (lane == 0) mbar_arrive(&acce);
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        int l[PLEV];
#pragma unroll
                        for (int v = 0; v < PLEV; ++v) l[v] = __float2int_rn(__uint_as_float(L[v][c]));
                        // units of 2^(8 v - 8) for level v: pairs of levels in 32 bits
                        // (1, 2 and 3 x 2^21, 4 x 2^21 at most; see above for 3 and 2)
                        const long long th = (long long)(l[7] * 256 + l[6]) * 65536 + (l[5] * 256 + l[4]);
                        const long long t = (th << 24) + (long long)(l[3] * 256 + l[2]) * 256 + (l[1] + (l[0] >> 8));
                        T[c4 + c] = MULTI ? T[c4 + c] + t : t;
                    }
                }
            }
            if (stop) break;
            // the kernel values, while the next tile's products run
#pragma unroll
            for (int c = 0; c < CW; ++c) {
                const ulonglong2 a = ag[CW * gr + c];
                const long long m = __mul64hi(T[c], (long long)a.y);
                const long long y = ai + (long long)a.x - (m >> shift);
                sum = fma(w[CW * gr + c], exp2_fixed<FB>(y, p.fb, table), sum);
            }
        }
        if (stop) abort_flag = 1;
        if (live && !stop) p.part[(size_t)(z * (EW / 4) + gr) * p.n + row] = sum;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
    if (threadIdx.x == 0 && abort_flag) atomicExch(flags + 1, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
}

// f_i = bias + the strips in order; the sign when hard.
__global__ void predict_finish_kernel(const double *__restrict__ part, int strips, int n, double bias, int hard,
                                      double *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double f = bias;
    for (int s = 0; s < strips; ++s) f = __dadd_rn(f, part[(size_t)s * n + i]);
    out[i] = hard ? (f >= 0.0 ? 1.0 : -1.0) : f;
}

// out_i = init_i +- (the strips in order) sa_i - tail, as kernel_rowsum_kernel.
__global__ void rowsum_finish_kernel(const double *__restrict__ part, int strips, int n, const int *__restrict__ ia,
                                     const double *__restrict__ sa, int op, const double *init,  // may alias out
                                     const double *__restrict__ tail, double *out) {
    chain_wait();
    chain_open();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double f = 0.0;
#pragma unroll 8
    for (int s = 0; s < strips; ++s) f = __dadd_rn(f, part[(size_t)s * n + i]);
    if (sa) f = __dmul_rn(f, sa[ia ? ia[i] : i]);
    const double f0 = init ? init[i] : 0.0;
    f = op > 0 ? __dadd_rn(f0, f) : __dsub_rn(f0, f);
    out[i] = tail ? __dsub_rn(f, tail[0]) : f;
}

// The digits, scales and norm terms of the rows idx[0 ... n - 1] of a sliced set as
// a sliced set of their own (zero digits up to whole 128-row tiles).
__global__ void __launch_bounds__(256) gather_slices_kernel(const uint4 *__restrict__ S, const int *__restrict__ ex,
                                                            const long long *__restrict__ a, int npb,
                                                            const int *__restrict__ idx, int n,
                                                            const int *__restrict__ np, uint4 *__restrict__ oS,
                                                            int *__restrict__ oex, long long *__restrict__ oa) {
    chain_wait();
    chain_open();
    if (np) n = np[0];
    constexpr int TILE = PS * PPIECE / 8;  // 16-byte units of a 16-feature block of a tile
    const int units = npb * PS * 2;        // of a row
    const long long items = (long long)((n + PM - 1) / PM * PM) * units;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < items;
         t += (long long)gridDim.x * blockDim.x) {
        // (neighbouring threads: the rows of a core matrix, 128 contiguous bytes)
        const int i = (int)(t / (8 * units)) * 8 + (int)(t & 7), u = (int)(t / 8 % units);
        const int pb = u / (2 * PS), s = u % (2 * PS) >> 1, h = u & 1;
        const int r = i < n ? idx[i] : 0;
        const uint4 v = i < n ? S[((size_t)(r >> 7) * npb + pb) * TILE + s * (PPIECE / 8) + ppiece_off(r & 127, 8 * h) / 8]
                              : make_uint4(0, 0, 0, 0);
        oS[((size_t)(i >> 7) * npb + pb) * TILE + s * (PPIECE / 8) + ppiece_off(i & 127, 8 * h) / 8] = v;
        if (u == 0 && i < n) {
            oex[i] = ex[r];
            oa[i] = a[r];
        }
    }
}

size_t slice_bytes(long long rows, int npb) { return (size_t)((rows + PM - 1) / PM) * npb * PS * PPIECE * 2; }

// The fixed point of y from the maxima of the two sets (row_scales_kernel: |q|,
// |x|^2, for the vectors |w|, and the smallest |q|), and cg 2^-ec = gamma log2(e);
// false: not for it. One unit serves all pairs, and the largest norms set it: a unit
// above 2^-53 is taken only where it is below half an ulp of c (q_i + q_j), which FP64
// sums round to, for the smallest norms too. (One row of |x|^2 = 10^7 among rows of 10,
// gamma 0.1: unit 2^-40, the other rows' values 3.5e-14 off, in FP64 3.4e-17. Rows of
// 400 to 450 apart by 1, gamma 0.25: unit 2^-51, 3.7e-17 off, in FP64 1.8e-15.)
// Raw rows (no q) take it in units of 2^-56, from 16 features on 2^-55: there it is as
// close as the differences' squares summed in FP64 (rms of a value at a common offset
// of the rows: 3.4e-17 and 3.4e-17 in FP64 at 20 features and 2^-55, 3.8e-17 and
// 3.3e-17 at 4), in larger units it is not (2^-53: 7.5e-17). And the products' dropped levels
// weigh 0.083 units of T per feature in a row's product with itself or a row near it (the
// digits agree), where the norms have them whole: y is off by
// 0.17 width c sigma^2 2^-62 there, where differences give 0 (784 features and an
// exponent of 62: all values 3.2e-15 off; FP64 sums 6e-17). Raw rows are taken while
// that stays below 2^-54: width times the exponent up to 1536 (3.5e-17 and 3.5e-17 in
// FP64 at 1320, 4.2e-17 and 3.7e-17 at 1960).
bool fixed_point_of(double gamma, bool raw, int width, const float *ht, const float *hs, PredictArgs *a,
                    unsigned long long *cg, int *ec) {
    unsigned wtop;
    memcpy(&wtop, hs + 2, sizeof wtop);
    if (!(ht[1] < 1e30f && hs[1] < 1e30f) || wtop >= 0x7ff00000u) return false;
    // |y| <= c (|q_i| + |q_j|) + 2 c |x_i| |x_j| < 2^(62 - fb), c = gamma log2(e)
    const double ym = gamma * 1.4426950408889634 *
                      ((double)ht[raw] + (double)hs[raw] + 2.0 * sqrt((double)ht[1] * (double)hs[1]));
    if (!(ym < 1e8)) return false;
    a->fb = ym < 32.0 ? 56 : 60 - ilogb(ym);
    scaled_gamma(gamma, cg, ec);
    // sigma < 2 |x| (1.001): the largest exponents (of zero rows: never less than -74)
    const int ei = ht[1] > 0.f ? (ilogb((double)ht[1]) >> 1) + 1 : -74;
    a->emax = hs[1] > 0.f ? (ilogb((double)hs[1]) >> 1) + 1 : -74;
    // y's product part = 2 c 2^(e_i + e_j) 2^-62 T 2^fb; no left shift in it
    a->fb = std::min(a->fb, *ec - 3 - ei - a->emax);
    if (!raw && a->fb < 53) {
        unsigned low[2];
        float qmin[2];
        memcpy(low, ht + 3, sizeof low[0]);
        memcpy(low + 1, hs + 3, sizeof low[0]);
        for (unsigned &v : low) v = ~v;
        memcpy(qmin, low, sizeof qmin);
        if (a->fb < 32 ||
            !(ldexp(1.0, 54 - a->fb) <= gamma * 1.4426950408889634 * ((double)qmin[0] + (double)qmin[1])))
            return false;
    }
    // (sigma^2 is at most 4 |x|^2, so c sigma^2 at most ym)
    if (raw && (a->fb < (width < 16 ? 56 : 55) || ym * width > 1536.0)) return false;
    a->g = *cg;
    a->shr = *ec - 3 - a->fb - a->emax;
    return true;
}

// Chunks of nt vector tiles for `it` row tiles: the fewest rounds of items over the
// SMs, an item's start taken as a quarter of a tile.
int best_chunks(int it, int nt, int sms, long long most = 1 << 30) {
    int best = 1;
    double cost = 1e300;
    for (int P = 1; P <= nt && P <= most && P <= std::max(64, 16 * sms / it); ++P) {
        const int per = ceil_div(nt, P);
        const double c = ceil_div((long long)it * ceil_div(nt, per), sms) * (per + 0.25);
        if (c < cost * 0.999) {
            cost = c;
            best = P;
        }
    }
    return best;
}

constexpr int GR = 4;  // strips of a chunk (column groups of predict_tc_kernel)

void launch_predict(const PredictArgs &a, int tiles) {
    auto kern = a.npb > PDRAIN ? (a.fb == 56 ? predict_tc_kernel<true, 56> : predict_tc_kernel<true, 0>)
                               : (a.fb == 56 ? predict_tc_kernel<false, 56> : predict_tc_kernel<false, 0>);
    allow_smem(kern);
    kern<<<dim3(tiles, a.P), 128 + 32 * 16, (size_t)PNS * P_STAGE + 1024, irwls_stream()>>>(a, irwls_dev_flags());
    irwls_count_launch(1);
}

void launch_norms(const irwls_dev_set *X, bool raw, int n, const int *ex, unsigned long long cg, int ec, int fb,
                  long long *a) {
    if (raw)
        row_norms_raw_kernel<<<std::min(ceil_div(n, 8), 2048), 256, 0, irwls_stream()>>>(X->X, X->ld, X->width, n, ex,
                                                                                       cg, ec, fb, a);
    else row_norms_kernel<<<ceil_div(n, 256), 256, 0, irwls_stream()>>>(X->q, n, cg, ec, fb, a);
    irwls_count_launch(1);
}

int slice_grid(long long rows, int npb, int sms) {
    return (int)std::max<long long>(1, std::min<long long>(ceil_div(rows * npb * 2, 256), 16LL * sms));
}

}  // namespace

// The plain form's prediction on the tensor cores; 1 when the sizes or values
// are not for it (the caller then sums on the FP64 pipe): not the RBF kernel, more than 12288 features (what the FP64 path takes) or 4 GB of vector
// slices, a vector that names a feature twice, a gamma outside (1e-30, 1e6),
// features or weights that are not finite, values whose squares leave FP32's
// range or whose y does not fit a fixed point as fine as FP64, no room for the workspace, or
// fewer than 500000 kernel values: the preparation and the host's wait for the
// maxima cost about 60 us. A call with 500000 values (1000 vectors) took 190 us there
// and 200 here with 20 features a row, 192 and 178 with 12 of 54, 1558 and 919 with
// 300; with 250 vectors 202 and 208, 202 and 186, 1364 and 745.
extern "C" int irwls_predict_exact(const irwls_dev_set *T, int n, const irwls_dev_set *S, int nSV, const double *d_w,
                                   double bias, int hard, double *d_out) {
    constexpr double MIN_VALUES = 5.0e5;
    if (n < 1 || nSV < 1 || (double)n * nSV < MIN_VALUES || T->mode != S->mode ||
        S->mode == IRWLS_K_LINEAR || !T->X || !S->X)
        return 1;
    const bool raw = S->mode == IRWLS_K_RAW_RBF;
    if (raw ? T->width != S->width : !S->rp || !S->ci) return 1;
    const int width = std::max(T->width, S->width);
    const int npb = ceil_div(width, PK);
    const double gamma = -S->neg_gamma;
    if (std::max(width, T->ld) > 12288 || slice_bytes(nSV, npb) > ((size_t)4 << 30)) return 1;
    if (!(gamma > 1e-30 && gamma < 1e6)) return 1;
    const int sms = irwls_num_sms() > 0 ? irwls_num_sms() : 148;
    // rows per slab: 2 GB of slices
    const long long tiles_fit = std::max<long long>(1, (long long)(irwls_slab_bytes((size_t)2 << 30) / slice_bytes(PM, npb)));
    const int slab = (int)std::min<long long>((long long)PM * tiles_fit, (long long)ceil_div(n, PM) * PM);
    const int nt = ceil_div(nSV, PN), it = ceil_div(std::min(n, slab), PM);
    const int per = ceil_div(nt, best_chunks(it, nt, sms)), P = ceil_div(nt, per);
    const size_t rn = (size_t)std::min(n, slab);
    const size_t off_s = (slice_bytes(slab, npb) + 255) & ~(size_t)255;
    const size_t off_et = off_s + ((slice_bytes(nSV, npb) + 255) & ~(size_t)255);
    const size_t off_es = off_et + ((size_t)n * 4 + 255 & ~(size_t)255), off_at = off_es + ((size_t)nSV * 4 + 255 & ~(size_t)255);
    const size_t off_as = off_at + (size_t)n * 8 + 256, off_top = off_as + (size_t)nSV * 8 + 256;
    const size_t off_part = (off_top + 1024) & ~(size_t)255;
    unsigned char *ws = nullptr;
    if (irwls_dev_malloc_try((void **)&ws, off_part + (size_t)P * GR * rn * sizeof(double)))
        return 1;  // (no room for it: the FP64 rows need none)
    __nv_bfloat16 *dT = (__nv_bfloat16 *)ws, *dS = (__nv_bfloat16 *)(ws + off_s);
    int *et = (int *)(ws + off_et), *es = (int *)(ws + off_es);
    long long *at = (long long *)(ws + ((off_at + 255) & ~(size_t)255)), *as = (long long *)(ws + ((off_as + 255) & ~(size_t)255));
    unsigned *top = (unsigned *)(ws + ((off_top + 255) & ~(size_t)255));
    int rc = irwls_dev_memset(top, 0, 2 * TOPS * sizeof(unsigned));
    auto fail = [&](int code) {
        irwls_dev_free(ws);
        return code;
    };
    if (rc) return fail(rc);
    const int gt = std::min(ceil_div(n, 8), 4 * sms), gs = std::min(ceil_div(nSV, 8), 4 * sms);
    row_scales_kernel<<<gt, 256, 0, irwls_stream()>>>(T->X, T->ld, T->width, raw ? nullptr : T->q, nullptr, nullptr, nullptr, n,
                                                     et, top);
    irwls_count_launch(1);
    row_scales_kernel<<<gs, 256, 0, irwls_stream()>>>(S->X, S->ld, S->width, raw ? nullptr : S->q, d_w, raw ? nullptr : S->rp, S->ci,
                                                     nSV, es, top + TOPS);
    irwls_count_launch(1);
    row_slice_kernel<<<slice_grid((long long)ceil_div(nSV, PM) * PM, npb, sms), 256, 0, irwls_stream()>>>(S->X, S->ld, S->width, nSV, es, ceil_div(nSV, PM) * PM, npb, dS);
    irwls_count_launch(1);
    if ((rc = irwls_check_launch("predict_prepare"))) return fail(rc);
    float h[2 * TOPS];
    if (irwls_dev_d2h(h, top, sizeof h) || irwls_dev_sync()) return fail(-2);
    PredictArgs a = {};
    unsigned long long cg;
    int ec;
    if (!fixed_point_of(gamma, raw, width, h, h + TOPS, &a, &cg, &ec)) return fail(1);
    launch_norms(T, raw, n, et, cg, ec, a.fb, at);
    launch_norms(S, raw, nSV, es, cg, ec, a.fb, as);
    a.T = dT;
    a.S = dS;
    a.npb = npb;
    a.nsv = nSV;
    a.per = per;
    a.P = P;
    a.es = es;
    a.as = as;
    a.w = d_w;
    a.part = (double *)(ws + off_part);
    for (int r0 = 0; r0 < n && !rc; r0 += slab) {
        const int rows = std::min(slab, n - r0), tiles = ceil_div(rows, PM);
        a.n = rows;
        a.et = et + r0;
        a.at = at + r0;
        row_slice_kernel<<<slice_grid((long long)tiles * PM, npb, sms), 256, 0, irwls_stream()>>>(T->X + (size_t)r0 * T->ld, T->ld, T->width, rows, et + r0, tiles * PM, npb, dT);
        irwls_count_launch(1);
        launch_predict(a, tiles);
        predict_finish_kernel<<<ceil_div(rows, 256), 256, 0, irwls_stream()>>>(a.part, P * GR, rows, bias, hard, d_out + r0);
        irwls_count_launch(1);
        rc = irwls_check_launch("predict_tc");
    }
    irwls_dev_free(ws);
    if (rc) return rc;
    const int tc = irwls_tc_status();
    if (tc) {
        irwls_set_error(-13, "a tensor-core pipeline wait of the prediction ran out (code %d)", tc);
        return -13;
    }
    return 0;
}

// ---- row sums within one set ------------------------------------------------

// A set's digits, kept over a training, and room for lists of its rows.
struct ExactRows {
    unsigned char *ws;
    __nv_bfloat16 *S, *bS, *aS;  // all rows; a list of vectors; a list of rows
    int *ex, *bex, *aex;
    long long *q, *bq, *aq;
    double *part;
    int n, npb, na, sms;
    size_t nparts;
    PredictArgs p;
};

extern "C" void irwls_exact_rows_free(void *h) {
    ExactRows *E = (ExactRows *)h;
    if (!E) return;
    irwls_dev_free(E->ws);
    free(E);
}

// Rows 0 ... n - 1 of X for row sums of all or up to na listed rows against lists
// of rows; NULL where irwls_predict_exact would return 1, or above 4 GB, and where a
// launch or a copy failed: an error is recorded then, and only then.
extern "C" void *irwls_exact_rows_create(const irwls_dev_set *X, int n, int na) {
    const double gamma = -X->neg_gamma;
    const bool raw = X->mode == IRWLS_K_RAW_RBF;
    if (n < 1 || X->mode == IRWLS_K_LINEAR || !X->X || (!raw && (!X->rp || !X->ci)) || X->ld > 12288 ||
        !(gamma > 1e-30 && gamma < 1e6))
        return nullptr;
    const int npb = ceil_div(X->width, PK), sms = irwls_num_sms() > 0 ? irwls_num_sms() : 148;
    na = std::min(na, n);
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t sb = up(slice_bytes(n, npb)), ab = up(slice_bytes(na, npb)), n4 = up((size_t)n * 4), n8 = up((size_t)n * 8);
    // partial sums: all rows in up to 16 chunks, lists of up to 2048 rows in any number
    const size_t nparts = (size_t)GR * std::max<size_t>((size_t)n * 16, (size_t)std::min(na, 2048) * ceil_div(n, PN));
    const size_t total = 2 * sb + ab + 3 * (n4 + n8) + 256 + up(nparts * sizeof(double));
    if (total > ((size_t)4 << 30)) return nullptr;
    ExactRows *E = (ExactRows *)calloc(1, sizeof(ExactRows));
    if (!E) return nullptr;  // (as without room on the device)
    if (irwls_dev_malloc_try((void **)&E->ws, total)) {
        free(E);
        return nullptr;
    }
    unsigned char *w = E->ws;
    auto take = [&](size_t b) {
        unsigned char *r = w;
        w += b;
        return r;
    };
    E->S = (__nv_bfloat16 *)take(sb);
    E->bS = (__nv_bfloat16 *)take(sb);
    E->aS = (__nv_bfloat16 *)take(ab);
    E->ex = (int *)take(n4), E->bex = (int *)take(n4), E->aex = (int *)take(n4);
    E->q = (long long *)take(n8), E->bq = (long long *)take(n8), E->aq = (long long *)take(n8);
    unsigned *top = (unsigned *)take(256);
    E->part = (double *)w;
    E->nparts = nparts;
    E->n = n, E->npb = npb, E->na = na, E->sms = sms;
    float h[TOPS];
    int rc = irwls_dev_memset(top, 0, TOPS * sizeof(unsigned));
    row_scales_kernel<<<std::min(ceil_div(n, 8), 4 * sms), 256, 0, irwls_stream()>>>(X->X, X->ld, X->width,
                                                                                  raw ? nullptr : X->q, nullptr,
                                                                                  raw ? nullptr : X->rp, X->ci, n,
                                                                                  E->ex, top);
    irwls_count_launch(1);
    row_slice_kernel<<<slice_grid((long long)ceil_div(n, PM) * PM, npb, sms), 256, 0, irwls_stream()>>>(
        X->X, X->ld, X->width, n, E->ex, ceil_div(n, PM) * PM, npb, E->S);
    irwls_count_launch(1);
    rc = rc || irwls_check_launch("exact_rows") || irwls_dev_d2h(h, top, sizeof h) || irwls_dev_sync();
    unsigned long long cg;
    int ec;
    if (rc || !fixed_point_of(gamma, raw, X->width, h, h, &E->p, &cg, &ec)) {
        irwls_exact_rows_free(E);
        return nullptr;
    }
    launch_norms(X, raw, n, E->ex, cg, ec, E->p.fb, E->q);
    E->p.npb = npb;
    return E;
}

// The arguments of irwls_dev_kernel_rowsum_n with the vectors' signs in cb; the list
// has at most nBmax rows. 1: fewer than 500000 kernel values (the caller then takes
// the FP64 kernel; the line is the predictions'). 4000 raw rows of 20 values, 500
// in the working set: 30 us a call with its gathers and sums, there 286.
extern "C" int irwls_exact_rowsum(void *h, const int *d_ia, int nA, const int *d_ib, const int *d_nB, int nBmax,
                                  const double *d_cb, const double *d_sa, int op, const double *d_init,
                                  const double *d_tail, double *d_out) {
    ExactRows *E = (ExactRows *)h;
    if (!E || nA < 1 || nBmax < 1 || (double)nA * nBmax < 5.0e5 || (d_ia ? nA > E->na : nA > E->n) || nBmax > E->n)
        return 1;
    PredictArgs a = E->p;
    const int it = ceil_div(nA, PM), nt = ceil_div(nBmax, PN);
    a.per = ceil_div(nt, best_chunks(it, nt, E->sms, (long long)(E->nparts / GR / nA)));
    a.P = ceil_div(nt, a.per);
    if (d_ia) {
        launch_chained(gather_slices_kernel, dim3(slice_grid((long long)nA * PS, E->npb, E->sms)), dim3(256), 0,
                       (const uint4 *)E->S, E->ex, E->q, E->npb, d_ia, nA, nullptr, (uint4 *)E->aS, E->aex, E->aq);
        irwls_count_launch(1);
    }
    launch_chained(gather_slices_kernel, dim3(slice_grid((long long)nBmax * PS, E->npb, E->sms)), dim3(256), 0,
                   (const uint4 *)E->S, E->ex, E->q, E->npb, d_ib, nBmax, d_nB, (uint4 *)E->bS, E->bex, E->bq);
    irwls_count_launch(1);
    a.T = d_ia ? E->aS : E->S;
    a.et = d_ia ? E->aex : E->ex;
    a.at = d_ia ? E->aq : E->q;
    a.S = E->bS;
    a.es = E->bex;
    a.as = E->bq;
    a.n = nA;
    a.nsv = nBmax;
    a.nsvp = d_nB;
    a.w = d_cb;
    a.part = E->part;
    if (irwls_prof_on()) irwls_prof_begin(IRWLS_PROF_ROWSUM);
    launch_predict(a, it);
    if (irwls_prof_on()) irwls_prof_end(IRWLS_PROF_ROWSUM);
    launch_chained(rowsum_finish_kernel, dim3(ceil_div(nA, 256)), dim3(256), 0, E->part, a.P * GR, nA, d_ia, d_sa, op,
                   d_init, d_tail, d_out);
    irwls_count_launch(1);
    return irwls_check_launch("exact_rowsum");
}
