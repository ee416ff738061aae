// dpmm_niw.cuh -- FP64 block-level helpers shared by the Hastings kernels (dpmm_hastings.cu), the parameter
// draws (dpmm_params.cu) and the split/merge screen (dpmm_screen.cu): the posterior + log marginal
// likelihood of NIW statistics with a block factorisation, the Dirichlet-multinomial marginal likelihood,
// a triangular inverse.
//
// Reference arithmetic restated (DPMMSubClusters/):
//   posterior            priors/niw.cpp:23-49, priors/multinomial_prior.cpp:12-22
//   log marginal lik.    priors/niw.cpp:122-138 (+ logdet.h:4-26 Cholesky branch,
//                        utils.cpp:94-102), priors/multinomial_prior.cpp:56-67
// lgamma is CUDA's lgamma(double).
#pragma once

#include <math.h>

#include "dpmm_internal.h"

namespace dpmm {

// ------------------------------------------------------------------------------ block-level helpers
// One block per statistics slot or pair: kHThreads threads for the Dirichlet terms and reductions; the
// NIW kernels run BlockChol<DP>::T threads (below).

constexpr int kHThreads = 128;

static __device__ __forceinline__ double warp_sum_d(double v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sum over the block (red: 33 doubles of shared memory); every thread gets the total
static __device__ double block_sum(double v, double* red)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = warp_sum_d(v);
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[q];
        red[32] = s;
    }
    __syncthreads();
    return red[32];
}

// Optional by-products of niw_lml_block for the screen: sum of log diag(psi') (the Hadamard bound of log
// det psi'), trace(psi') and log det psi' itself.
struct NiwExtras {
    double hd, tr, ld;
};

// Dirichlet-multinomial log marginal likelihood of statistics (n, sum [+ sum2]) by the block
static __device__ double mult_lml_block(int D, double n, const double* sum, const double* sum2, const double* alpha0,
                                        double* red)
{
    if (n == 0) return 0.0;
    double s0 = 0, sp = 0, acc = 0;
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        const double a0 = alpha0[d], ap = a0 + (sum2 ? sum[d] + sum2[d] : sum[d]);
        s0 += a0;
        sp += ap;
        acc += lgamma(ap) - lgamma(a0);
    }
    s0 = block_sum(s0, red);
    sp = block_sum(sp, red);
    acc = block_sum(acc, red);
    return lgamma(s0) - lgamma(sp) + acc;
}

// ------------------------------------------------------------------------------ block factorisation
// One block factors the posterior scale matrix psi' of one statistics slot (or pair) as L' diag(p) L'^T
// (unit lower L', pivots p) in shared memory.  Element A(i, k), k <= i, starts at M[i LD + k] and ends
// there as R(i, k) = L'(i, k) p_k; L'(i, k), k < i, is kept at M[k LD + i], so that both factors of the
// update A(i, k) -= L'(i, j) R(k, j) are read without bank conflicts (LD odd).
//
// Bound: the chain to the last pivot.  Each column needs a reciprocal (68 clocks), the quotient's six
// dependent operations (8 each), one broadcast (27) and one multiply-add after the column before it, about
// 11e3 clocks at D = 64.  A block barrier per column and an update of the whole trailing matrix between two
// columns (the right-looking form with the matrix in registers that this replaces) cost about 2400 clocks
// a column.  Here one warp factors and a lane owns rows lane, lane + 32, ..: a panel of 8 columns first takes
// the updates of all columns before it (8 independent chains per row, no barrier: 11.5e3 clocks in all at
// D = 64) and is then factored with shuffles only (14.4e3).  Every element sees the same operations in the
// same order as in the right-looking form: the results are equal bit for bit.  The other warps compute the
// terms that need no factor meanwhile.
// Measured, D = 64: a list of 16 pairs 85 -> 27 us, 300 slots 98 -> 29 us; 2016 pairs at D = 50 261 -> 95 us.
template <int DP>
struct BlockChol {
    static constexpr int T = DP > 64 ? 256 : 128;                   // threads per block
    static constexpr int C = (T / DP) < DP ? (T / DP) : DP;         // thread classes of the diagonal sums
    static constexpr int LD = DP + 1;
    // shared memory in doubles: the matrix, posterior mean, reduction scratch, pivots, lgamma terms, scalars
    static constexpr int MP = DP * LD, RED = MP + DP, PIV = RED + 33, GT = PIV + DP, SC = GT + DP, SMEM = SC + 16;
    static constexpr size_t bytes = sizeof(double) * SMEM;
};

// Correctly rounded quotients by one divisor b: with y = RN(1 / b), a quotient q within an ulp of a / b and the
// exact remainder a - b q, RN(q + (a - b q) y) is RN(a / b) (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990, theorem on the final step of a
// division); the first correction brings a y (two roundings) within the ulp.  No branch, so that several
// quotients by one b run side by side (6 dependent operations each after the reciprocal), where the compiler
// keeps two divisions one after the other (a panel of 8 columns: 400 -> 190 clocks a column).  Both sides are
// scaled by the power of two that brings b to 1/4 .. 1/2: no product leaves the range where the quotient does not.
// Equal bit for bit to a / b for quotients of 2^-960 and above in magnitude (below, the remainder is not exact
// and the last two places may differ) and for zero, infinite and NaN operands and results: there the
// corrections would make NaN of an infinity, and a y already is the quotient.
struct Divisor {
    double b, y, scale;
    __device__ __forceinline__ explicit Divisor(double d)
    {
        const int e = (__double2hiint(d) >> 20) & 0x7ff;
        scale = __hiloint2double((2044 - min(e, 2043)) << 20, 0);
        b = d * scale;
        y = 1.0 / b;
    }
    __device__ __forceinline__ double operator()(double a) const
    {
        a *= scale;
        const double q0 = a * y;
        const bool normal = (unsigned)(__double2hiint(q0) & 0x7ff00000) - 0x00100000u < 0x7fe00000u;
        const double q1 = fma(fma(-b, q0, a), y, q0);
        const double q2 = fma(fma(-b, q1, a), y, q1);
        return normal ? q2 : q0;
    }
};

// element e of the D (D - 1) / 2 below the diagonal: columns q and D - 2 - q together hold D of them
static __device__ __forceinline__ void strict_lower(int D, int e, int& i, int& j)
{
    const int q = e / D, o = e - q * D;
    const bool first = o < D - 1 - q;
    j = first ? q : D - 2 - q;
    i = first ? q + 1 + o : D - 1 - (o - (D - 1 - q));
}

// Updates of the panel's columns b0 .. b0 + PB - 1 (a[r][c] = A(lane + 32 r, b0 + c)) by the columns before
// it, rows from 32 R0 on (the rows above are finished).
template <int DP, int R0, int RP, int PB>
static __device__ __forceinline__ void ldl_update(const double* M, double (&a)[RP][PB], int b0, int lane)
{
    constexpr int LD = BlockChol<DP>::LD;
#pragma unroll 4
    for (int j = 0; j < b0; ++j) {
        double l[RP], u[PB];
#pragma unroll
        for (int c = 0; c < PB; ++c) u[c] = M[(b0 + c) * LD + j];
#pragma unroll
        for (int r = R0; r < RP; ++r) l[r] = M[j * LD + lane + 32 * r];
#pragma unroll
        for (int r = R0; r < RP; ++r)
#pragma unroll
            for (int c = 0; c < PB; ++c) a[r][c] -= l[r] * u[c];
    }
}

// The factorisation by one whole warp; piv[j] receives the pivots (a pivot that is not positive divides
// as 1).
template <int DP>
static __device__ __forceinline__ void warp_ldl(double* M, int D, double* piv)
{
    constexpr int LD = BlockChol<DP>::LD, RP = (DP + 31) / 32, PB = DP < 8 ? DP : 8;
    const int lane = threadIdx.x & 31;
    for (int b0 = 0; b0 < D; b0 += PB) {
        double a[RP][PB];
#pragma unroll
        for (int r = 0; r < RP; ++r)
#pragma unroll
            for (int c = 0; c < PB; ++c) a[r][c] = lane + 32 * r < DP ? M[(lane + 32 * r) * LD + b0 + c] : 0.0;
        const int ro = b0 >> 5;   // the panel's own rows are rows 32 ro + ..
        if constexpr (RP == 1) {
            if (DP >= 32 || lane < DP) ldl_update<DP, 0>(M, a, b0, lane);
        } else {
            switch (ro) {
            case 0: ldl_update<DP, 0>(M, a, b0, lane); break;
            case 1: ldl_update<DP, 1>(M, a, b0, lane); break;
            case 2: ldl_update<DP, (RP > 2 ? 2 : 1)>(M, a, b0, lane); break;
            default: ldl_update<DP, (RP > 3 ? 3 : 1)>(M, a, b0, lane); break;
            }
        }
        __syncwarp();
#pragma unroll
        for (int jj = 0; jj < PB; ++jj) {
            const int j = b0 + jj;
            if (j >= D) break;
            double own[PB];   // this lane's values of the panel's own rows, column jj
            double oj = a[0][jj];
#pragma unroll
            for (int r = 1; r < RP; ++r) oj = r == ro ? a[r][jj] : oj;
#pragma unroll
            for (int c = 0; c < PB; ++c) own[c] = c >= jj ? __shfl_sync(0xffffffffu, oj, (b0 + c) & 31) : 0.0;
            const double p = own[jj];
            const double pj = p > 0 ? p : 1.0;
            const Divisor by_pj(pj);
            if (lane == 0) piv[j] = p;
#pragma unroll
            for (int r = 0; r < RP; ++r) {
                const int i = lane + 32 * r;
                const bool act = i > j && i < D;
                const double ci = by_pj(act ? a[r][jj] : pj);
                if (i >= j && i < D) M[i * LD + j] = a[r][jj];
                if (act) M[j * LD + i] = ci;
#pragma unroll
                for (int c = jj + 1; c < PB; ++c) a[r][c] -= ci * own[c];
            }
        }
        __syncwarp();
    }
}

// After warp_ldl: the lower Cholesky factor L(i, j) = R(i, j) / sqrt(p_j) in place of L' (M[j LD + i], i >= j), and
// xd[j] = 1 / L(j, j), by the block (ends with a barrier).
template <int DP>
static __device__ __forceinline__ void block_ldl_to_cholesky(double* M, int D, double* piv, double* xd)
{
    constexpr int LD = BlockChol<DP>::LD;
    for (int j = threadIdx.x; j < D; j += blockDim.x) {
        const double p = piv[j], sq = sqrt(p > 0 ? p : 1.0);
        piv[j] = sq;
        const double d = p / sq;
        M[j * LD + j] = d;
        xd[j] = 1.0 / d;
    }
    // zeros past D in the columns of L, for the unrolled inverse
    for (int e = threadIdx.x; e < D * (DP - D); e += blockDim.x) M[(e / (DP - D)) * LD + D + e % (DP - D)] = 0.0;
    __syncthreads();
    const int total = D / 2 * (D - 1) + (D & 1) * (D / 2);   // D (D - 1) / 2 below the diagonal
#pragma unroll 4
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        int i, j;
        strict_lower(D, e, i, j);
        M[j * LD + i] = Divisor(piv[j])(M[i * LD + j]);
    }
    __syncthreads();
}

// X = L^-1 (lower) from L at M[j LD + i], i >= j: X(i, k) replaces R at M[i LD + k], k < i; the diagonal
// X(j, j) = 1 / L(j, j) is in xd.  Row i of X depends on L and on itself only, so thread i < DP walks its row
// from the diagonal to the left, X(i, j) = -X(j, j) sum_{k > j} X(i, k) L(k, j) (the order of LAPACK's unblocked
// triangular inverse), without a barrier.  The sum is one chain of multiply-adds (its order is kept): the
// row stays in registers and the loops are unrolled, so that nothing but the chain (8 clocks a term) is
// left; its terms past i are zeros.  M must hold finite values up to row and column DP - 1 (zeros past D).
template <int DP>
static __device__ __forceinline__ void rows_tri_inverse(double* M, int D, const double* xd, int i)
{
    constexpr int LD = BlockChol<DP>::LD;
    double x[DP];
#pragma unroll
    for (int k = 0; k < DP; ++k) x[k] = k == i ? xd[k] : 0.0;
    const int last = i | 31;   // the warp's longest row
#pragma unroll
    for (int j = DP - 2; j >= 0; --j) {
        if (j >= last || j >= D - 1) continue;
        double y = 0.0;
#pragma unroll
        for (int k = j + 1; k < DP; ++k) y += x[k] * M[j * LD + k];
        if (j < i) {
            x[j] = -xd[j] * y;
            M[i * LD + j] = x[j];
        }
    }
}

// log det of the matrix that warp_ldl factored: sum of log pivots in every thread, or NaN if a pivot is not
// positive.
template <int DP>
static __device__ double block_log_pivots(int D, const double* piv, double* red)
{
    const int t = threadIdx.x;
    double lp = 0, bad = 0;
    for (int j = t; j < D; j += blockDim.x) {
        const double p = piv[j];
        bad += !(p > 0);
        lp += log(p > 0 ? p : 1.0);
    }
    const double ldp = block_sum(lp, red);
    return block_sum(bad, red) > 0 ? NAN : ldp;
}

// the warp of the block that factors: consecutive blocks of an SM (148 apart) take another scheduler each
static __device__ __forceinline__ int chol_warp()
{
    return (int)((blockIdx.x + blockIdx.x / 148u) % (blockDim.x >> 5));
}

struct NoSideWork {
    __device__ __forceinline__ void operator()(int, int) const {}
};

// NIW posterior and log marginal likelihood (niw.cpp:23-49, 122-138; statistics (n, sum, S) plus the
// optional (sum2, S2) aggregated into them, niw.cpp:140-148) by one block of BlockChol<DP>::T threads,
// D <= DP.  sh: BlockChol<DP>::SMEM doubles of shared memory (posterior mean at MP).  The posterior scale
// psi' (upper triangle mirrored, as selfadjointView<Upper>) is built in shared memory and factored by one
// warp; the others compute the terms that need no factor, then side(index, count).  Valid in every thread;
// sh keeps the factors (see above).
// With allow_empty, an empty slot (n = 0) is factored too (its posterior is the prior; the
// parameter draw needs the factor) and its statistics are read as zero; otherwise it returns 0.
template <int DP, typename Side = NoSideWork>
__device__ double niw_lml_block(int D, double n, const double* sum, const double* S, const double* sum2,
                                const double* S2, double k0, double v0, const double* m0, const double* psi0,
                                double ld0, double* sh, NiwExtras* ex = nullptr, bool allow_empty = false,
                                const Side& side = Side())
{
    using BC = BlockChol<DP>;
    if (n == 0 && !allow_empty) return 0.0;   // posterior == prior (niw.cpp:27-30): every term cancels
    const bool has = n > 0;
    double* mp = sh + BC::MP;
    double* red = sh + BC::RED;
    double* gt = sh + BC::GT;
    double* sc = sh + BC::SC;
    const int t = threadIdx.x;
    const double kp = k0 + n, vp = v0 + n;
    for (int d = t; d < D; d += blockDim.x)
        mp[d] = (m0[d] * k0 + (has ? (sum2 ? sum[d] + sum2[d] : sum[d]) : 0.0)) / kp;
    __syncthreads();
    // rows q and D - 1 - q together hold D + 1 elements: the lower triangle in equal strips, batches of loads
    // in flight
    const int total = (D + 1) / 2 * (D + 1);
    const Divisor by_vp(vp);
    constexpr int BATCH = 6;
    for (int e0 = t; e0 < total; e0 += BATCH * blockDim.x) {
        double sv[BATCH], ps[BATCH];
        int ri[BATCH], ci[BATCH];
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
            const int e = e0 + q * (int)blockDim.x;
            const int pr = e / (D + 1), o = e - pr * (D + 1);
            int i = pr, k = o;
            if (o > pr) {
                i = D - 1 - pr;
                k = o - pr - 1;
            }
            const bool ok = e < total && !(o > pr && 2 * pr == D - 1);   // the middle row of an odd D has no partner
            ri[q] = ok ? i : -1;
            ci[q] = k;
            const size_t ki = (size_t)i * D + k;   // upper-triangle source: row k <= column i
            ps[q] = ok ? psi0[ki] : 0.0;
            sv[q] = ok && has ? S[ki] : 0.0;
            if (S2 && ok && has) sv[q] += S2[ki];
        }
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
            if (ri[q] < 0) continue;
            const int i = ri[q], k = ci[q];
            const double tm = v0 * ps[q] + k0 * m0[k] * m0[i];
            sh[i * BC::LD + k] = by_vp(tm - kp * mp[k] * mp[i] + sv[q]);
        }
    }
    __syncthreads();
    if (ex) {
        const int i = t % DP, c = t / DP;
        double h = 0, tr = 0;
        if (c < BC::C && i < D && i % BC::C == c) {
            h = log(sh[i * BC::LD + i]);
            tr = sh[i * BC::LD + i];
        }
        ex->hd = block_sum(h, red);
        ex->tr = block_sum(tr, red);
    }
    const int warp = t >> 5, cw = chol_warp();
    if (warp == cw) {
        warp_ldl<DP>(sh, D, sh + BC::PIV);
    } else {
        const int tt = t - (warp > cw ? 32 : 0), nt = (int)blockDim.x - 32;
        if (tt < 3) sc[tt] = log(tt == 0 ? v0 : tt == 1 ? vp : k0 / kp);
        for (int q = nt - 1 - tt; q < D; q += nt) {
            const int d = 1 + q;
            gt[q] = lgamma(vp / 2.0 + (1 - d) / 2.0) - lgamma(v0 / 2.0 + (1 - d) / 2.0);
        }
        side(tt, nt);
    }
    __syncthreads();
    const double ld = block_log_pivots<DP>(D, sh + BC::PIV, red);
    if (ex) ex->ld = ld;
    double g = 0.0;
    for (int q = t; q < D; q += blockDim.x) g += gt[q];
    g = block_sum(g, red);
    return -n * D * 0.5 * log(M_PI) + g + (v0 / 2.0) * (D * sc[0] + ld0) - (vp / 2.0) * (D * sc[1] + ld) +
           (D / 2.0) * sc[2];
}

// merge log Hastings ratio of clusters i < j (shared_actions.cpp:88-99) by one block
template <int DP>
__device__ double merge_log_hr_block(const double* __restrict__ stats, int stat_len, int D, int gauss, double k0,
                                     double v0, double ld0, const double* __restrict__ prior,
                                     const double* __restrict__ lml, int i, int j, double alpha, double* sh)
{
    const double* si = stats + (size_t)(3 * i) * stat_len;
    const double* sj = stats + (size_t)(3 * j) * stat_len;
    const double ni = si[0], nj = sj[0];
    if (ni == 0 || nj == 0) return NAN;
    const double n = ni + nj;
    double* lg = sh + BlockChol<DP>::SC + 4;   // the ratio's gamma terms, one thread each
    auto terms = [&](int q, int) {
        if (q < 8) {
            const double at = q == 0 ? alpha : q == 1 ? 0.5 * alpha : q == 2 ? n : q == 3 ? n + alpha
                            : q == 4 ? ni + 0.5 * alpha : q == 5 ? ni : q == 6 ? nj : nj + 0.5 * alpha;
            lg[q] = lgamma(at);
        }
    };
    double lij;
    if (gauss) {
        lij = niw_lml_block<DP>(D, n, si + 1, si + 1 + D, sj + 1, sj + 1 + D, k0, v0, prior, prior + D, ld0, sh, nullptr,
                                false, terms);
    } else {
        terms((int)threadIdx.x, 0);
        lij = mult_lml_block(D, n, si + 1, sj + 1, prior, sh + BlockChol<DP>::RED);   // (its barriers order lg)
    }
    return -log(alpha) + lg[0] - 2 * lg[1] + lg[2] - lg[3] + lg[4] - lg[5] - lg[6] + lg[7] + lij - lml[3 * i] -
           lml[3 * j];
}

// Kernels templated on DP are launched through this: DPV is the padded dimension (4 ... 128), and
// `body` a statement using the constexpr DP.
#define DPMM_WITH_DP(DPV, body)                                   \
    switch (DPV) {                                                \
    case 4: { constexpr int DP = 4; body; } break;                \
    case 8: { constexpr int DP = 8; body; } break;                \
    case 16: { constexpr int DP = 16; body; } break;              \
    case 32: { constexpr int DP = 32; body; } break;              \
    case 64: { constexpr int DP = 64; body; } break;              \
    default: { constexpr int DP = 128; body; } break;             \
    }

// split log Hastings ratio of cluster k (local_clusters_actions.cpp:222-233) from the slot counts
// and the log marginal likelihoods of slots 3k, 3k+1, 3k+2; NaN when a sub-cluster is empty
static __device__ double split_log_hr_slot(const double* __restrict__ stats, int stat_len,
                                           const double* __restrict__ lml, int k, double alpha)
{
    const double n = stats[(size_t)(3 * k) * stat_len], nl = stats[(size_t)(3 * k + 1) * stat_len],
                 nr = stats[(size_t)(3 * k + 2) * stat_len];
    if (nl == 0 || nr == 0) return NAN;
    return log(alpha) + lgamma(nl) + lml[3 * k + 1] + lgamma(nr) + lml[3 * k + 2] - (lgamma(n) + lml[3 * k]);
}

}  // namespace dpmm
