// dev_gram_tc.cu -- IRWLSpar's Gram on the tensor cores, through exact integer
// slices, in two digit forms: base 256 (the plain form, FP64 accuracy) and
// base 128 (the precision form).
//
//   G = A'^T A',   A' = [sd * KSC[act, :], day]   (nact x (m + 1)),
//
// the K1/K2 system of IRWLSpar (reference src/budgeted-train.c:379-430).
// FP64 on this part runs at about 1/64 of the FP32 rate, so the product is
// formed on the bf16 tensor cores with every partial sum exact:
//
// 1. Each column c of A' gets a power of two sigma_c >= max_p |A'_pc| (a
//    column-max pass), and each entry becomes the integer
//    N_pc = round(A'_pc / sigma_c * 2^F), |N| <= 2^F, F = 48 (base 128) or 55,
//    by integer operations on its bits. N is written in 7 balanced digits
//    d_0 .. d_6 of base B (d_0 lowest), |d_s| <= B/2: small integers, exact in
//    bf16.
// 2. sum_p N_pi N_pj = sum_u B^u L_u(i, j), L_u = sum_{s+t=u} sum_p
//    d_s(p,i) d_t(p,j). The top 7 (base 128) or 8 levels are kept (28 or 33
//    digit pairs); the dropped ones weigh at most about 2^-46 or 2^-61 of
//    sigma_i sigma_j per row, with random signs.
// 3. A CTA owns a 128 x 64 tile of G and one split-K chunk of the rows. Per
//    16-row stage the digit-pair products go to one accumulator of 128 x 64
//    FP32 per level in tensor memory (448 or all of its 512 columns). A level
//    sums at most 7 pairs of products of magnitude <= (B/2)^2, so over 512
//    (base 128) or 128 rows every partial sum is an integer below 2^24: exact
//    in FP32, whatever the order of accumulation. After that many rows the
//    epilogue drains the levels into a 96-bit integer per entry, so the whole
//    sum stays exact.
// 4. G_ij = sigma_i sigma_j 2^-GSCALE T_ij, written as the FP64 partials that
//    gram_reduce_kernel adds to KC.
//
// Operands reach shared memory by bulk copies: the slices are stored in the
// shared-memory image of a stage (per 128-column tile and 16-row block, the
// digit pieces of 128 x 16 in canonical K-major core-matrix order). Warp 0
// copies, lane 0 of warp 1 issues the MMAs, warps 4-11 drain. Every wait is
// bounded; a timeout sets device flag word 1.
#include <cuda_bf16.h>
#include <stdint.h>

#include <algorithm>

#include "dev_common.cuh"
#include "tc_ptx.cuh"

namespace {

// The two digit forms, 7 balanced digits each of base 2^BITS.
//   GramDigits<7>: the precision form. GFRAC 48, levels u >= 6 (28 digit
//   pairs, 7 accumulators), drained every 512 rows.
//   GramDigits<8>: the plain form. GFRAC 55, levels u >= 5 (33 pairs, 8
//   accumulators, all of tensor memory), drained every 128 rows. Entries of at
//   least 2^-2 of their column's scale are represented exactly, the others
//   within 2^-56 of it, and the dropped levels weigh below 2^-61 of
//   sigma_i sigma_j per row: together below the rounding of an FP64
//   accumulation (up to 2^-54 of the partial sum per addition). One level less
//   (2^-53 per row) moved the weights of 2000 to 48000-row trainings two to
//   fifteen times further from a 64-bit reference than the FP64 product did.
// A level sums at most 7 pairs of products of magnitude <= 2^(2 BITS - 2), so
// over the rows between two drains every FP32 partial sum is an integer below
// 2^24. The 33 products run on the tensor cores at about 40 TFLOP/s
// FP64-equivalent, where the FP64 pipe of this part gives 1.06 at most.
constexpr int GS = 7;                  // digits per entry
constexpr int GM = 128, GN = 64;       // tile of G: rows (A' columns) x columns
constexpr int GBK = 16;                // rows of A' per stage
constexpr int GPIECE = GM * GBK;       // elements of one digit piece (4 KB)
constexpr int GNS = 5;                 // ring stages
constexpr int G_THREADS = 384;
constexpr uint32_t A_STAGE = GS * GPIECE * 2;      // 28 KB: 7 pieces of 128 rows
constexpr uint32_t B_PIECE = GN * GBK * 2;         // 2 KB: 64 rows of one piece
constexpr uint32_t G_STAGE = A_STAGE + GS * B_PIECE;  // 42 KB

template <int BITS>
struct GramDigits {
    static constexpr int HALF = 1 << (BITS - 1);        // digits in [-HALF, HALF], exact in bf16
    static constexpr int GFRAC = BITS * GS - 1;         // N = round(v * 2^GFRAC), |v| <= 1
    static constexpr int LOW = BITS == 7 ? GS - 1 : GS - 2;  // lowest kept level
    static constexpr int LEVELS = 2 * (GS - 1) - LOW + 1;
    static constexpr int GPAIRS = BITS == 7 ? 28 : 33;  // digit pairs of the kept levels
    static constexpr int GSCALE = 2 * GFRAC - BITS * LOW;    // G = sigma_i sigma_j 2^-GSCALE T
    static constexpr int GDRAIN = BITS == 7 ? 32 : 8;   // stages between drains
    static_assert(LEVELS * GN <= 512, "level accumulators exceed tensor memory");
    static_assert((long long)GS * GDRAIN * GBK * HALF * HALF < (1LL << 24), "level sums must stay exact");
};

// Element offset of (row r of the 128-row tile, k of the 16-row block) in a
// digit piece: 8 x 8 core matrices, 128 bytes apart along k, 256 along r.
__device__ __forceinline__ int piece_off(int r, int k) { return (r >> 3) * 128 + (k >> 3) * 64 + (r & 7) * 8 + (k & 7); }

// ceil(log2 |v|) from the bits of a normal double v: its exponent, plus one
// unless v is a power of two.
__device__ __forceinline__ int ceil_log2_bits(unsigned long long b) {
    return (int)((b >> 52) & 0x7ff) - 1023 + ((b & ((1ULL << 52) - 1)) != 0 ? 1 : 0);
}

constexpr int NO_EXP = -2000;  // zero or subnormal: no scale

// ceil(log2 |v|) of v = RN(a * b), the FP64 product, or NO_EXP when v is zero
// or subnormal. Away from the products whose rounding can land on a power
// of two (mantissa products within 2^-18 of 2 or 4) and from the exponent
// range's ends, it follows from the operands' exponents and an FP32 product
// of their leading mantissa bits (relative error below 2^-21), with no FP64
// operation; the rest take the FP64 product.
__device__ __forceinline__ int prod_ceil_log2(double a, double b) {
    const unsigned long long ua = (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffULL;
    const unsigned long long ub = (unsigned long long)__double_as_longlong(b) & 0x7fffffffffffffffULL;
    const int Ea = (int)(ua >> 52), Eb = (int)(ub >> 52);
    if (Ea > 0 && Eb > 0 && Ea + Eb >= 1030 && Ea + Eb <= 3060) {
        const unsigned long long ma = ua & ((1ULL << 52) - 1), mb = ub & ((1ULL << 52) - 1);
        const int e = Ea + Eb - 2046;  // exponent of the product of the leading ones
        if (ma == 0 && mb == 0) return e;  // two powers of two: the exact product
        const float pr = __uint_as_float(0x3f800000u | (uint32_t)(ma >> 29)) *
                         __uint_as_float(0x3f800000u | (uint32_t)(mb >> 29));
        if (pr <= 2.0f - 0x1p-18f) return e + 1;                       // in (1, 2): not a power of two
        if (pr >= 2.0f + 0x1p-17f && pr <= 4.0f - 0x1p-17f) return e + 2;  // in (2, 4)
    }
    const unsigned long long v = (unsigned long long)__double_as_longlong(__dmul_rn(a, b)) & 0x7fffffffffffffffULL;
    return (v >> 52) == 0 ? NO_EXP : ceil_log2_bits(v);
}

// Column scales of A': per column the largest ceil(log2 |v|) over the active
// rows, stored as the bits of 2^that (so that col_exp reads it back; a
// column with no normal entry stays 0). A CTA takes GCM rows and 256 columns, a
// thread one column with the loads of GCR rows in flight. An entry whose
// exponents alone bound it by the maximum so far (|a b| < 2^(Ea + Eb - 2044)) is
// done with three integer instructions, which is nearly every one: 50000 x 300
// takes 26 us, with every entry's product formed and two rows in flight 58.
// The maximum does not depend on the order the entries are visited in.
constexpr int GCM = 64, GCR = 8;
__global__ void __launch_bounds__(256) gram_colmax_kernel(const double *__restrict__ KSC, int m,
                                                          const int *__restrict__ act, int nact,
                                                          const double *__restrict__ sd,
                                                          const double *__restrict__ day,
                                                          unsigned long long *__restrict__ cmax) {
    chain_wait();
    chain_open();
    const int p0 = blockIdx.x * GCM, p1 = min(nact, p0 + GCM);
    const int c = 256 * blockIdx.y + threadIdx.x;
    if (c > m) return;
    int mx = NO_EXP;
    if (c == m) {
        for (int p = p0; p < p1; ++p) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(day[p]) & 0x7fffffffffffffffULL;
            if ((b >> 52) != 0) mx = max(mx, ceil_log2_bits(b));
        }
    } else {
        for (int p = p0; p < p1; p += GCR) {
            double x[GCR];
#pragma unroll
            for (int k = 0; k < GCR; ++k) x[k] = KSC[(size_t)act[min(p + k, p1 - 1)] * m + c];
#pragma unroll
            for (int k = 0; k < GCR; ++k) {
                const double w = sd[min(p + k, p1 - 1)];
                const int bound = ((__double2hiint(w) >> 20) & 0x7ff) + ((__double2hiint(x[k]) >> 20) & 0x7ff) - 2044;
                if (bound > mx) mx = max(mx, prod_ceil_log2(w, x[k]));
            }
        }
    }
    if (mx > NO_EXP) atomicMax(cmax + c, (unsigned long long)(mx + 1023) << 52);
}

// sigma_c = 2^e_c, the smallest power of two >= the column maximum (e = -1100:
// the column is zero).
__device__ __forceinline__ int col_exp(unsigned long long mxbits) {
    const int E = (int)((mxbits >> 52) & 0x7ff);
    if (E == 0) return -1100;
    const bool pow2 = (mxbits & ((1ULL << 52) - 1)) == 0;
    return E - 1023 + (pow2 ? 0 : 1);
}

// round(v * 2^(FRAC - e)) for |v| <= 2^e, ties away from zero, from the bits
// of v (no FP64 pipe).
template <int FRAC>
__device__ __forceinline__ long long fixed_point(double v, int e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int E = (int)((b >> 52) & 0x7ff);
    if (E == 0) return 0;  // zero (subnormals, below 2^-1022, are dropped)
    const unsigned long long M = (b & ((1ULL << 52) - 1)) | (1ULL << 52);
    // v = M 2^(E - 1075); N = M 2^(E - 1075 + FRAC - e) = M >> sh
    const int sh = 1075 + e - FRAC - E;  // >= 52 - FRAC since |v| <= 2^e
    long long N = 0;
    if (FRAC > 52 && sh <= 0) N = (long long)(M << min(-sh, FRAC - 52));
    else if (sh < 64) N = (long long)((M + (1ULL << (sh - 1))) >> sh);
    return (b >> 63) ? -N : N;
}

// The slices of A'. Thread = (column c, group of 8 rows): the digits of the
// group's entries, one 16-byte store per digit piece. Rows >= nact and
// columns > m are written as zeros.
template <int BITS>
__global__ void __launch_bounds__(256) gram_slice_kernel(const double *__restrict__ KSC, int m,
                                                         const int *__restrict__ act, int nact,
                                                         const double *__restrict__ sd,
                                                         const double *__restrict__ day,
                                                         const unsigned long long *__restrict__ cmax, int ncols,
                                                         int npb, __nv_bfloat16 *__restrict__ S) {
    chain_wait();
    chain_open();
    constexpr int HALF = GramDigits<BITS>::HALF;
    __shared__ uint16_t bf[2 * HALF + 1];  // bf16 bits of -HALF ... HALF
    for (int t = threadIdx.x; t <= 2 * HALF; t += 256) {
        const __nv_bfloat16 h = __float2bfloat16_rn((float)(t - HALF));
        bf[t] = *(const uint16_t *)&h;
    }
    __syncthreads();
    const long long items = (long long)ncols * npb * 2;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < items;
         t += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(t % ncols);
        const long long g = t / ncols;  // 8-row group
        const int pb = (int)(g >> 1), half = (int)(g & 1);
        const int e = c <= m ? col_exp(cmax[c]) : -1100;
        uint32_t w[GS][4];  // digit s of the 8 rows, packed bf16 pairs
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int p = pb * GBK + half * 8 + k;
            long long N = 0;
            if (p < nact && c <= m && e > -1100) {
                const double v = c < m ? __dmul_rn(sd[p], KSC[(size_t)act[p] * m + c]) : day[p];
                N = fixed_point<GramDigits<BITS>::GFRAC>(v, e);
            }
#pragma unroll
            for (int s = 0; s < GS; ++s) {
                int d;
                if (s < GS - 1) {
                    d = (int)(N & (2 * HALF - 1));
                    if (d >= HALF) d -= 2 * HALF;
                    N = (N - d) >> BITS;
                } else {
                    d = (int)N;  // |d| <= HALF
                }
                const uint32_t hb = bf[d + HALF];
                if (k & 1) w[s][k >> 1] |= hb << 16;
                else w[s][k >> 1] = hb;
            }
        }
        const int ct = c >> 7, r = c & 127;
        const size_t base = ((size_t)ct * npb + pb) * GS * GPIECE + piece_off(r, half * 8);
#pragma unroll
        for (int s = 0; s < GS; ++s)
            *(uint4 *)(S + base + (size_t)s * GPIECE) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    }
}

// tcgen05.ld of 4 consecutive columns of this warp's 32 lanes.
__device__ __forceinline__ void tc_ld4(uint32_t addr, float *v) {
    uint32_t r0, r1, r2, r3;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::);
    v[0] = __uint_as_float(r0);
    v[1] = __uint_as_float(r1);
    v[2] = __uint_as_float(r2);
    v[3] = __uint_as_float(r3);
}

// Records the first wait that ran out in device flag word 1 as
// role * 10^8 + cta * 1000 + stage (role 1: producer empty, 2: producer
// drain, 3: MMA acc-empty, 4: MMA full, 5: MMA done, 6: drain acc-full).
__device__ __forceinline__ void gram_timeout(int *flags, int role, int cta, int k) {
    atomicCAS(flags + 1, 0, role * 100000000 + min(cta, 99999) * 1000 + min(max(k, 0), 999));
}

// 96-bit accumulator hi * 2^32 + lo (hi signed).
struct Acc96 {
    long long hi;
    uint32_t lo;
};

__device__ __forceinline__ void acc_add(Acc96 &a, long long xh, uint32_t xl) {
    const uint32_t lo = a.lo + xl;
    a.hi += xh + (lo < xl ? 1 : 0);
    a.lo = lo;
}

// Tile (I, J) of G for split-K chunk z: rows 128 I ... of G (columns of A'),
// columns 64 J ...; stages [z * spc, min(npb, (z + 1) * spc)) of 16 rows.
template <int BITS>
__global__ void __launch_bounds__(G_THREADS, 1) gram_tc_kernel(const __nv_bfloat16 *__restrict__ S, int npb, int spc,
                                                               int m, const unsigned long long *__restrict__ cmax,
                                                               double *__restrict__ part, int *flags) {
    chain_wait();
    chain_open();
    using Cfg = GramDigits<BITS>;
    constexpr int LOW = Cfg::LOW, LEVELS = Cfg::LEVELS, GSCALE = Cfg::GSCALE, GDRAIN = Cfg::GDRAIN;
    const int J = blockIdx.x, I = blockIdx.y, z = blockIdx.z;
    if (GN * J > GM * I + GM - 1 || GN * J >= m) return;  // above the diagonal or past the last column
    extern __shared__ __align__(1024) unsigned char g_smem[];
    __shared__ __align__(8) uint64_t full[GNS], empty[GNS], accf, acce, done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    unsigned char *smem = g_smem + ((1024 - (smem_u32(g_smem) & 1023)) & 1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k0 = z * spc, nst = max(0, min(npb, k0 + spc) - k0);
    const int cta = (int)(blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z));
    const int nblk = (nst + GDRAIN - 1) / GDRAIN;
    if (threadIdx.x == 0) {
        for (int b = 0; b < GNS; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], 1);
        }
        mbar_init(&accf, 1);
        mbar_init(&acce, 8);
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
        // producer: the A tile's pieces in one copy, the B half-pieces one by one
        if (lane == 0) {
            const uint32_t base = smem_u32(smem);
            const __nv_bfloat16 *Ab = S + ((size_t)I * npb + k0) * GS * GPIECE;
            const __nv_bfloat16 *Bb = S + ((size_t)(J >> 1) * npb + k0) * GS * GPIECE + (J & 1) * (GN / 8) * 128;
            int issued = 0;
            for (int k = 0; k < nst; ++k) {
                const int slot = k % GNS;
                if (k >= GNS && !mbar_wait(smem_u32(&empty[slot]), (uint32_t)(k / GNS - 1) & 1u)) {
                    gram_timeout(flags, 1, cta, k);
                    abort_flag = 1;
                }
                if (abort_flag) break;
                const uint32_t sb = base + slot * G_STAGE, fb = smem_u32(&full[slot]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fb), "r"(G_STAGE));
                bulk_g2s(sb, Ab + (size_t)k * GS * GPIECE, A_STAGE, fb);
#pragma unroll
                for (int s = 0; s < GS; ++s)
                    bulk_g2s(sb + A_STAGE + s * B_PIECE, Bb + ((size_t)k * GS + s) * GPIECE, B_PIECE, fb);
                issued = k + 1;
            }
            for (int k = issued > GNS ? issued - GNS : 0; k < issued; ++k)
                if (!mbar_wait(smem_u32(&full[k % GNS]), (uint32_t)(k / GNS) & 1u)) {
                    gram_timeout(flags, 2, cta, k);
                    abort_flag = 1;
                }
        }
        __syncwarp();
    } else if (warp == 1) {
        // MMA issue: level u - LOW += sum_{s+t=u} A_s B_t, u = LOW ... 2 GS - 2
        if (lane == 0) {
            const uint32_t base = smem_u32(smem);
            for (int k = 0; k < nst && !abort_flag; ++k) {
                const int blk = k / GDRAIN, kin = k % GDRAIN;
                if (kin == 0 && blk >= 1) {
                    if (!mbar_wait(smem_u32(&acce), (uint32_t)(blk - 1) & 1u)) {
                        gram_timeout(flags, 3, cta, k);
                        abort_flag = 1;
                        break;
                    }
                }
                const int slot = k % GNS;
                if (!mbar_wait(smem_u32(&full[slot]), (uint32_t)(k / GNS) & 1u)) {
                    gram_timeout(flags, 4, cta, k);
                    abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
                const uint32_t sa = base + slot * G_STAGE, sbb = sa + A_STAGE;
                // A piece s against the B pieces t = LOW-s ... GS-1, which lie
                // consecutively in shared memory and so form one operand of
                // up to 64 GS rows whose products land on consecutive levels:
                // ten MMAs of N <= 256 for the 28 pairs (thirteen for 33), each
                // A piece read once per MMA instead of once per pair. The
                // first product of a drain block on each level starts it:
                // piece GS-1 covers all levels with LOW = GS - 1, all but the
                // lowest with LOW = GS - 2, whose first is (GS-2, 0). The sums
                // are exact integers, so the grouping does not change them.
#pragma unroll
                for (int s = GS - 1; s >= 0; --s) {
                    const uint64_t da = tc_desc_lbo_sbo(sa + s * (GPIECE * 2), 128, 256);
                    const bool lone = LOW == GS - 2 && s == GS - 2;  // piece 0 by itself
#pragma unroll
                    for (int t0 = LOW > s ? LOW - s : 0; t0 < GS; t0 += (lone && t0 == 0) ? 1 : 4) {
                        const int np = lone && t0 == 0 ? 1 : GS - t0 < 4 ? GS - t0 : 4;  // B pieces of this MMA
                        const uint64_t db = tc_desc_lbo_sbo(sbb + t0 * B_PIECE, 128, 256);
                        const bool acc = kin > 0 || !(s == GS - 1 || (lone && t0 == 0));
                        mma_bf16(tmem + (uint32_t)(s + t0 - LOW) * GN, da, db, tc_idesc(GM, GN * np), acc ? 1u : 0u);
                    }
                }
                tc_commit(&empty[slot]);
                if (kin == GDRAIN - 1 || k == nst - 1) tc_commit(&accf);
            }
            tc_commit(&done);
            if (!mbar_wait(smem_u32(&done), 0u)) {
                gram_timeout(flags, 5, cta, nst);
                abort_flag = 1;
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        // drain: lanes 32 (warp % 4) ..., columns 32 h ... 32 h + 31
        const int q = warp & 3, h = (warp - 4) >> 2;
        Acc96 T[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) T[j] = Acc96{0, 0u};
        for (int blk = 0; blk < nblk; ++blk) {
            const bool got = mbar_wait(smem_u32(&accf), (uint32_t)blk & 1u);
            if (!got) gram_timeout(flags, 6, cta, blk * GDRAIN);
            const int bad = (!got || abort_flag) ? 1 : 0;
            int any;
            asm volatile(
                "{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.or.pred q, 1, 256, p;\nselp.s32 %0, 1, 0, q;\n}\n"
                : "=r"(any)
                : "r"(bad));
            if (any) {
                abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
            const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16) + 32 * h;
#pragma unroll
            for (int c4 = 0; c4 < 32; c4 += 4) {
                float L[LEVELS][4];
#pragma unroll
                for (int v = 0; v < LEVELS; ++v) tc_ld4(lanes + v * GN + c4, L[v]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    // the upper four levels and the lower three or four by
                    // Horner in 64-bit integers (at most 2^48 and a little),
                    // then T += t_hi 2^UP + t_lo
                    constexpr int UP = BITS * (LEVELS - 4);  // 21 or 32
                    constexpr int B = 1 << BITS;
                    long long th = __float2int_rn(L[LEVELS - 1][j]);
#pragma unroll
                    for (int v = LEVELS - 2; v >= LEVELS - 4; --v) th = th * B + __float2int_rn(L[v][j]);
                    long long tl = __float2int_rn(L[LEVELS - 5][j]);
#pragma unroll
                    for (int v = LEVELS - 6; v >= 0; --v) tl = tl * B + __float2int_rn(L[v][j]);
                    if constexpr (UP == 32) T[c4 + j].hi += th;
                    else acc_add(T[c4 + j], th >> (32 - UP), (uint32_t)th << UP);
                    acc_add(T[c4 + j], tl >> 32, (uint32_t)tl);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
            if (lane == 0) mbar_arrive(&acce);
        }
        if (!abort_flag) {
            const int r = GM * I + 32 * q + lane;
            if (r <= m) {
                const int er = col_exp(cmax[r]);
                double *out = part + (size_t)z * (m + 1) * m + (size_t)r * m;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const int c = GN * J + 32 * h + j;
                    if (c < m && c <= r) {
                        const int ec = col_exp(cmax[c]);
                        double g = 0.0;
                        if (er > -1100 && ec > -1100) {
                            const double t = fma((double)T[j].hi, 4294967296.0, (double)T[j].lo);
                            g = ldexp(t, er + ec - GSCALE);
                        }
                        out[c] = g;
                    }
                }
            }
        }
    }
    if (threadIdx.x == 0 && abort_flag) gram_timeout(flags, 9, cta, 0);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
}

size_t slices_bytes(int rows, int m) {
    const size_t ct = (size_t)ceil_div(m + 1, GM), npb = (size_t)ceil_div(std::max(rows, 1), GBK);
    return ct * npb * GS * GPIECE * sizeof(__nv_bfloat16);
}

// bf16 tensor-core flops issued by gram_tc_kernel since the last read (28 or
// 33 digit-pair products per 128 x 64 x 16 step of every tile).
double g_tc_flops = 0.0;

// The Gram in digit form BITS, the active rows taken in slabs of at most
// `slab` rows (the slices of one slab are the workspace; the column scales
// are those of all rows). P >= the number of slabs bounds the partials.
template <int BITS>
int gram_run(const double *d_KSC, int m, const int *d_act, int nact, const double *d_sd, const double *d_day,
             const double *d_KC, double *d_K1, int ldK1, double *d_part, int P, void *d_ws, int slab) {
    using Cfg = GramDigits<BITS>;
    const int sms = irwls_num_sms() > 0 ? irwls_num_sms() : 148;
    const int ct = ceil_div(m + 1, GM), nt = ceil_div(m, GN);
    const int nslab = std::max(1, ceil_div(nact, slab));
    __nv_bfloat16 *S = (__nv_bfloat16 *)d_ws;
    unsigned long long *cmax = (unsigned long long *)((char *)d_ws + slices_bytes(std::min(nact, slab), m));
    // tiles of the lower part, and enough chunks to give every SM one CTA
    int tiles = 0;
    for (int I = 0; I < ct; ++I)
        for (int J = 0; J < nt; ++J)
            if (GN * J <= GM * I + GM - 1) ++tiles;
    if (irwls_prof_on()) irwls_prof_begin(IRWLS_PROF_GRAM_SLICE);
    if (irwls_dev_memset(cmax, 0, (size_t)(m + 1) * sizeof(unsigned long long))) return -1;
    if (nact > 0) {
        launch_chained(gram_colmax_kernel, dim3(ceil_div(nact, GCM), ceil_div(m + 1, 256)), dim3(256), 0, d_KSC, m,
                       d_act, nact, d_sd, d_day, cmax);
        IRWLS_LAUNCH_CHECK("gram_colmax");
    }
    const size_t smem = (size_t)GNS * G_STAGE + 1024;
    allow_smem(gram_tc_kernel<BITS>);
    int parts = 0;
    for (int a = 0, n = 0; n < nslab; a += slab, ++n) {
        const int rows = std::min(slab, nact - a);
        const int npb = ceil_div(std::max(rows, 1), GBK);
        int pz = std::max(1, std::min(P / nslab, sms / std::max(tiles, 1)));
        pz = std::min(pz, npb);
        const int spc = ceil_div(npb, pz);
        pz = ceil_div(npb, spc);
        if (irwls_prof_on() && n > 0) irwls_prof_begin(IRWLS_PROF_GRAM_SLICE);
        const long long items = (long long)ct * GM * npb * 2;
        launch_chained(gram_slice_kernel<BITS>, dim3((int)std::min<long long>(ceil_div(items, 256), 16LL * sms)),
                       dim3(256), 0, d_KSC, m, d_act + a, rows, d_sd + a, d_day + a, cmax, ct * GM, npb, S);
        if (irwls_prof_on()) irwls_prof_end(IRWLS_PROF_GRAM_SLICE);
        IRWLS_LAUNCH_CHECK("gram_slice");
        if (irwls_prof_on()) irwls_prof_begin(IRWLS_PROF_GRAM);
        launch_chained(gram_tc_kernel<BITS>, dim3(nt, ct, pz), dim3(G_THREADS), smem, S, npb, spc, m, cmax,
                       d_part + (size_t)parts * (m + 1) * m, irwls_dev_flags());
        g_tc_flops += (double)tiles * npb * GBK * GM * GN * 2.0 * Cfg::GPAIRS;
        if (irwls_prof_on()) irwls_prof_end(IRWLS_PROF_GRAM);
        IRWLS_LAUNCH_CHECK("gram_tc");
        parts += pz;
    }
    return irwls_par_gram_reduce(d_part, parts, m, d_KC, d_K1, ldK1);
}

// Rows per slab of the plain form: 4 GB of slices at most, so that the
// workspace stays small beside K_nm itself (14 bytes of digits per 8-byte
// entry) whatever the number of rows.
constexpr size_t SLAB_BYTES = 4ULL << 30;
int slab_rows(int m) {
    const size_t per = slices_bytes(GBK, m);  // one 16-row block of every column tile
    return (int)std::min<size_t>(std::max<size_t>(irwls_slab_bytes(SLAB_BYTES) / per, 1) * GBK, 1u << 30);
}

}  // namespace

extern "C" double irwls_gram_tc_flops(int reset) {
    const double f = g_tc_flops;
    if (reset) g_tc_flops = 0.0;
    return f;
}

// Workspace of irwls_par_gram_tc for up to l active rows: the slices, then the
// m + 1 column maxima.
extern "C" size_t irwls_par_gram_tc_bytes(int l, int m) {
    return slices_bytes(l, m) + (size_t)(m + 1) * sizeof(unsigned long long) + 256;
}

// K1 (column-major, leading dimension ldK1, lower part) = KC + the Gram of
// the active rows, row m = K2; P bounds the split-K chunks (part holds at
// least P partials).
extern "C" int irwls_par_gram_tc(const double *d_KSC, int m, const int *d_act, int nact, const double *d_sd,
                                 const double *d_day, const double *d_KC, double *d_K1, int ldK1, double *d_part,
                                 int P, void *d_ws) {
    return gram_run<7>(d_KSC, m, d_act, nact, d_sd, d_day, d_KC, d_K1, ldK1, d_part, P, d_ws, std::max(nact, 1));
}

// The plain form's Gram, its workspace and the fewest partials
// that P may allow for l rows (one per slab).
extern "C" size_t irwls_par_gram_bytes(int l, int m) {
    return slices_bytes(std::min(l, slab_rows(m)), m) + (size_t)(m + 1) * sizeof(unsigned long long) + 256;
}
extern "C" int irwls_par_gram_min_parts(int l, int m) { return std::max(1, ceil_div(l, slab_rows(m))); }
extern "C" int irwls_par_gram(const double *d_KSC, int m, const int *d_act, int nact, const double *d_sd,
                              const double *d_day, const double *d_KC, double *d_K1, int ldK1, double *d_part, int P,
                              void *d_ws) {
    return gram_run<8>(d_KSC, m, d_act, nact, d_sd, d_day, d_KC, d_K1, ldK1, d_part, P, d_ws, slab_rows(m));
}
