// dev_sgma_ahead.cu -- the candidates' whitened kernel rows ahead of their step.
//
// SGMA scores candidate c of a step through w_c = L^-1 k_C(c) (mixed.c). The
// candidates of every step are drawn before the first one, so w does not have
// to wait for its step: when centroid s is chosen, element s of w follows for
// all later candidates by one step of forward substitution,
//   w_s = (k(c_s, c) - sum_{t < s} L_st w_t) / L_ss,
// where L_st is w_t of the chosen candidate and L_ss^2 = k(c_s, c_s) + jitter -
// |w|^2, with |w|^2 carried along (src/budgeted-train.c:247-279). One kernel per
// step does that, together with the chosen column of Q, between one selection and
// the next scores. Extending an explicit L^-1 and multiplying the 64 new kernel
// rows by it at the step itself takes six more dependent kernels: at 60000 rows
// and 200 of 400 centroids a step took 92 us with them and takes 58.
// Both cost m^3 / 6 x 64 FP64 multiply-adds over a training; this one reads the
// later candidates' w (64 s (m - s) doubles per step) where that read L^-1.
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "blocked_bf16.cuh"
#include "dev_common.cuh"

namespace {

constexpr int NCAND = 64;
constexpr int SG = 8;  // warps of a CTA: they split the sums over t and over the features
constexpr int WP = 128;  // rows of W copied to shared memory before the choice is known

struct AheadArgs {
    KView X;
    const int *cand, *cent;
    const int *best;       // the chosen slot of step s; NULL for the class means (s < 2)
    int s, m, l, kbn;      // kbn: 32-column blocks of Q and of a step's W image
    double *W;             // [t][64 m]: w_t of every candidate
    double *ss, *kcc;      // |w|^2 so far and k(c, c) of every candidate
    float *dd;             // |Q_c - w|^2 so far (with eps)
    double *L;             // rows of the factor
    double *eta;           // of the next step's candidates
    __nv_bfloat16 *Wb;     // the steps' W images (blocked_bf16.cuh)
    __nv_bfloat16 *Qb;
    float *qn;
    const float *resid;    // [candidate of step s][row]: Q w - k
    unsigned *eps;
    int ncta;              // candidate CTAs; the others write Q's column
};

// This warp's share of sum_k a_k b_k, or of sum_k (a_k - b_k)^2 for raw rows:
// a: the lane's dense row, b: the centroid (shared by all lanes).
__device__ __forceinline__ double part_kernel(const KView &X, const double *a, int gc, int g) {
    double acc = 0.0;
    if (X.mode == IRWLS_K_RAW_RBF) {
        const int per = (X.width + SG - 1) / SG, k1 = min(X.width, (g + 1) * per);
        const double *b = X.X + (size_t)gc * X.ld;
#pragma unroll 4
        for (int k = g * per; k < k1; ++k) {
            const double d = a[k] - b[k];
            acc = fma(d, d, acc);
        }
        return acc;
    }
    const int p0 = X.rp[gc], p1 = X.rp[gc + 1], per = (p1 - p0 + SG - 1) / SG;
    const int e = min(p1, p0 + (g + 1) * per);
#pragma unroll 4
    for (int p = p0 + g * per; p < e; ++p) acc = fma(X.cv[p], a[X.ci[p]], acc);
    return acc;
}
__device__ __forceinline__ double kernel_value(const KView &X, double v, double qa, double qb) {
    if (X.mode == IRWLS_K_LINEAR) return v;
    return exp(X.ng * (X.mode == IRWLS_K_RAW_RBF ? v : qa + qb - 2.0 * v));
}

// k(c, c) of every candidate from j0 on, and zeros in its sums. A warp each.
__global__ void __launch_bounds__(256) ahead_init_kernel(KView X, const int *__restrict__ cand, int j0, int n,
                                                         double *__restrict__ ss, double *__restrict__ kcc,
                                                         float *__restrict__ dd) {
    const int lane = threadIdx.x & 31;
    const int j = j0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (j >= n) return;
    const int gc = cand[j];
    double v = 0.0;
    if (X.mode != IRWLS_K_RAW_RBF)
        for (int p = X.rp[gc] + lane; p < X.rp[gc + 1]; p += 32)
            v = fma(X.cv[p], X.X[(size_t)gc * X.ld + X.ci[p]], v);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) {
        ss[j] = 0.0;
        kcc[j] = kernel_value(X, v, X.q[gc], X.q[gc]);
        if (dd) dd[j] = 0.f;
    }
}

// Row s of L in FP32 (s values, then 1 / L_ss) for the direct Q column.
__global__ void ahead_lrow_kernel(const double *__restrict__ L, int ldL, int s, float *__restrict__ lrow) {
    for (int t = threadIdx.x; t < s; t += blockDim.x) lrow[t] = __double2float_rn(L[(size_t)s * ldL + t]);
    if (threadIdx.x == 0) lrow[s] = __double2float_rn(1.0 / L[(size_t)s * ldL + s]);
}

// CTA b < ncta: 32 candidates of the later steps, a lane each; warp g adds every
// SG-th term of the sum over t and its share of the kernel value's features. The
// others: Q's column s, q_i = -r_i / L_ss from the residuals of the chosen candidate.
// Latency bounds it (the chosen candidate's row, the sums, one exponential), so what
// does not depend on the choice -- W up to row s - 1, written by the kernel of step
// s - 1, three launches back -- is fetched while the selection runs.
__global__ void __launch_bounds__(32 * SG) sgma_ahead_kernel(AheadArgs p) {
    extern __shared__ __align__(16) double wbuf[];  // WP rows of W at most, then row s of L
    __shared__ double piv[2];                       // L_ss, its reciprocal
    __shared__ double red[2][SG][33];
    const int s = p.s, lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const size_t nc = (size_t)NCAND * p.m;
    const int sp = min(s, WP);
    double *l2 = wbuf + 32 * sp;
    const size_t j0 = (size_t)NCAND * max(2, s + 1) + 32 * blockIdx.x;
    if ((int)blockIdx.x < p.ncta) {
        for (int t = threadIdx.x; t < 16 * sp; t += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(wbuf + 2 * t)),
                         "l"(p.W + (t >> 4) * nc + j0 + 2 * (t & 15)));
        for (int t = WP + g; t < s; t += SG)
            if (lane < 2) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p.W + t * nc + j0 + 16 * lane));
        if (p.X.ld <= 128)
            for (int k = 16 * g; k < p.X.ld; k += 16 * SG)
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p.X.X + (size_t)p.cand[j0 + lane] * p.X.ld + k));
    }
    chain_wait();
    chain_open();
    const bool chosen = p.best != nullptr;
    const int bb = chosen ? p.best[0] : 0, gc = p.cent[s];
    const size_t jb = (size_t)NCAND * s + bb;
    if (g == 0) {
        const double l3 = chosen ? sqrt((p.kcc[jb] + 0.00001) - p.ss[jb]) : p.L[(size_t)s * p.m + s];
        if (lane == 0) {
            piv[0] = l3;
            piv[1] = 1.0 / l3;
        }
    }
    const bool row = chosen && blockIdx.x == 0;  // writes row s of L
    if (row)
        for (int t = threadIdx.x; t < s; t += blockDim.x) p.L[(size_t)s * p.m + t] = p.W[t * nc + jb];
    if ((int)blockIdx.x >= p.ncta) {
        __syncthreads();
        if (row && threadIdx.x == 0) p.L[(size_t)s * p.m + s] = piv[0];
        const float inv = __double2float_rn(piv[1]);
        const float *r = p.resid + (size_t)bb * p.l;
        const int n = (gridDim.x - p.ncta) * blockDim.x;
        for (int i = (blockIdx.x - p.ncta) * blockDim.x + threadIdx.x; i < p.l; i += n)
            put_q(i, s, -r[i] * inv, p.Qb, p.kbn, p.qn);
        return;
    }
    for (int t = threadIdx.x; t < s; t += blockDim.x)
        l2[t] = chosen ? p.W[t * nc + jb] : p.L[(size_t)s * p.m + t];
    const size_t j = j0 + lane;  // < nc: ncta covers 64 each
    const int gj = p.cand[j];
    const double kp = part_kernel(p.X, p.X.X + (size_t)gj * p.X.ld, gc, g);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    double a0 = 0.0, a1 = 0.0;
    int t = g;
    for (; t + SG < sp; t += 2 * SG) {
        a0 = fma(l2[t], wbuf[32 * t + lane], a0);
        a1 = fma(l2[t + SG], wbuf[32 * (t + SG) + lane], a1);
    }
    for (; t < sp; t += SG) a0 = fma(l2[t], wbuf[32 * t + lane], a0);
    for (; t + 7 * SG < s; t += 8 * SG) {
        double w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) w[u] = p.W[(size_t)(t + u * SG) * nc + j];
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
            a0 = fma(l2[t + u * SG], w[u], a0);
            a1 = fma(l2[t + (u + 1) * SG], w[u + 1], a1);
        }
    }
    for (; t < s; t += SG) a0 = fma(l2[t], p.W[(size_t)t * nc + j], a0);
    red[0][g][lane] = a0 + a1;
    red[1][g][lane] = kp;
    __syncthreads();
    if (g != 0) return;
    double dot = 0.0, kv = 0.0;
#pragma unroll
    for (int k = 0; k < SG; ++k) {
        dot += red[0][k][lane];
        kv += red[1][k][lane];
    }
    const double w = (kernel_value(p.X, kv, p.X.q[gj], p.X.q[gc]) - dot) * piv[1];
    const double sum = fma(w, w, p.ss[j]);
    p.W[(size_t)s * nc + j] = w;
    p.ss[j] = sum;
    const int step = (int)(j / NCAND), c = (int)(j % NCAND);
    const float xf = __double2float_rn(w);
    __nv_bfloat16 pc[3];
    bf16_pieces3(xf, pc);
    __nv_bfloat16 *Wb = p.Wb + (size_t)step * p.kbn * QB_NP * WB_PIECE;
#pragma unroll
    for (int k = 0; k < QB_NP; ++k) Wb[wb_index(c, s, k)] = pc[k];
    float dd = 0.f;
    if (p.eps) {
        // the candidate's own row of Q (its training row) is w itself
        const float q = chosen ? -p.resid[(size_t)bb * p.l + gj] * __double2float_rn(piv[1])
                               : bf16_join3(p.Qb[qb_index(gj, s, p.kbn, 0)], p.Qb[qb_index(gj, s, p.kbn, 1)],
                                            p.Qb[qb_index(gj, s, p.kbn, 2)]);
        const float d = xf - q;
        dd = fmaf(d, d, p.dd[j]);
        p.dd[j] = dd;
    }
    if (step == max(2, s + 1)) {
        p.eta[c] = 1.0 - sum;
        // a NaN keeps its (large) bits in the maximum
        if (p.eps) atomicMax(p.eps, __float_as_uint(fabsf(sqrtf(dd))));
    }
    if (row && lane == 0) p.L[(size_t)s * p.m + s] = piv[0];
}

}  // namespace

// Bytes of the workspace for a budget of m and Q's leading dimension ldq: the
// whitened rows, their W images, three values per candidate.
extern "C" size_t irwls_sgma_ahead_bytes(int m, int ldq) {
    return (size_t)NCAND * m * ((size_t)m * sizeof(double) + (size_t)ldq * 2 * QB_NP + 2 * sizeof(double) + sizeof(float)) +
           1024;
}

// The W image of step s in the workspace.
extern "C" const void *irwls_sgma_ahead_image(const void *ws, int m, int ldq, int s) {
    return (const char *)ws + (size_t)NCAND * m * (m + 2) * sizeof(double) + (size_t)s * NCAND * ldq * 2 * QB_NP;
}

extern "C" int irwls_sgma_ahead_init(const irwls_dev_set *X, const int *d_cand, int m, int ldq, void *ws) {
    const size_t nc = (size_t)NCAND * m;
    double *ss = (double *)ws + nc * m, *kcc = ss + nc;
    char *img = (char *)irwls_sgma_ahead_image(ws, m, ldq, 0);
    float *dd = (float *)(img + nc * ldq * 2 * QB_NP);
    if (irwls_dev_memset(img, 0, nc * ldq * 2 * QB_NP)) return -1;
    const long long n = (long long)nc - 2 * NCAND;
    if (n <= 0) return 0;
    ahead_init_kernel<<<ceil_div(n, 8), 256, 0, irwls_stream()>>>(kview(X), d_cand, 2 * NCAND, (int)nc, ss, kcc, dd);
    IRWLS_LAUNCH_CHECK("ahead_init");
    return 0;
}

extern "C" int irwls_sgma_ahead_lrow(const double *d_L, int ldL, int s, float *d_lrow) {
    ahead_lrow_kernel<<<1, 32, 0, irwls_stream()>>>(d_L, ldL, s, d_lrow);
    IRWLS_LAUNCH_CHECK("ahead_lrow");
    return 0;
}

// After centroid s is known (d_best: its slot among the step's candidates, NULL
// for the class means, whose row of L and column of Q are there): element s of the
// later candidates, eta and the W image of the next step's, Q's column s.
extern "C" int irwls_sgma_ahead_step(const irwls_dev_set *X, int l, const int *d_cand, const int *d_cent,
                                     const int *d_best, int s, int m, int ldq, double *d_L, void *ws, void *Qb,
                                     float *d_qn, const float *d_rq, double *d_eta, unsigned *d_eps) {
    const size_t nc = (size_t)NCAND * m;
    AheadArgs a = {};
    a.X = kview(X);
    a.cand = d_cand;
    a.cent = d_cent;
    a.best = d_best;
    a.s = s;
    a.m = m;
    a.l = l;
    a.kbn = ldq / 32;
    a.W = (double *)ws;
    a.ss = a.W + nc * m;
    a.kcc = a.ss + nc;
    a.Wb = (__nv_bfloat16 *)irwls_sgma_ahead_image(ws, m, ldq, 0);
    a.dd = (float *)((char *)a.Wb + nc * ldq * 2 * QB_NP);
    a.L = d_L;
    a.eta = d_eta;
    a.Qb = (__nv_bfloat16 *)Qb;
    a.qn = d_qn;
    a.resid = d_rq;
    a.eps = d_eps;
    a.ncta = 2 * std::max(0, m - std::max(2, s + 1));
    const int sms = irwls_num_sms() > 0 ? irwls_num_sms() : 148;
    const int nq = d_best ? std::max(1, std::min(ceil_div(l, 256), 4 * sms)) : 0;
    if (a.ncta + nq == 0) return 0;
    const size_t smem = ((size_t)32 * std::min(s, WP) + std::max(1, s)) * sizeof(double);
    if (smem > 40 * 1024) allow_smem(sgma_ahead_kernel);
    launch_chained(sgma_ahead_kernel, dim3(a.ncta + nq), dim3(32 * SG), smem, a);
    IRWLS_LAUNCH_CHECK("sgma_ahead");
    return 0;
}
