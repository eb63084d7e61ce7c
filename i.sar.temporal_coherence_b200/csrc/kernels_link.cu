/* The exact tier of phase linking (any number of dates up to 64; see
 * tc_link_exact_kernel below) and the choice between the link kernels. Stages
 * (tcoh.cl:603-744):
 *
 *   coherence matrix T_ij = C_ij / sqrt(C_ii C_jj), optional magnitude bias
 *   correction (tcoh.cl:610-636);
 *   pair coherences |T_ij| (tcoh.cl:515-527, 639);
 *   connectivity of the non-zero T_ij under the bias correction (tcoh.cl:494-513,
 *   644-647);
 *   the eigenvector of T's largest eigenvalue (EVD) or of the smallest of |T|^-1 o
 *   T (EMI) (tcoh.cl:649-694, by the method of tcoh.cl:201-444);
 *   unit phasors relative to the median date (or the strongest component when it
 *   is negligible) and the Pepe-Lanari goodness of fit (tcoh.cl:696-744).
 *
 * Stacks of up to 32 dates go to kernels_link_half.cu (two pixels per warp), EVD
 * of 33 to 64 dates to kernels_link_wide.cu (two warps per pixel), both in float
 * from a Gram kernel's sums, handing the pixels that need it to the exact tier;
 * EMI of 33 to 64 dates is all exact tier.
 */
#include "link_float.cuh"

#include <math.h>

#define FULL 0xffffffffu

namespace {

template <typename R>
__device__ __forceinline__ R wsum(R v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1)
        v += __shfl_xor_sync(FULL, v, o);
    return v;
}

__device__ __forceinline__ double wmaxd(double v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1)
        v = fmax(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

/* Number of eigenvalues of the double tridiagonal (d, e) below x, from the
   three-term recurrence of the leading principal minors, p_i = (d_i - x)
   p_{i-1} - e2_{i-1} p_{i-2}, whose ratios q_i = p_i / p_{i-1} are the pivots of
   the LDL^T factorization (a negative pivot is a sign change between consecutive
   minors): one FMA on the dependency chain per step, no division. The minors
   are rescaled by powers of two to stay in range; a pivot of magnitude below
   pivmin becomes -pivmin. */
__device__ __forceinline__ int sturmd_minors(const double *d, const double *e2, int n, double x,
                                             double pivmin)
{
    double pm = 1.0, p = d[0] - x;

    if (fabs(p) < pivmin)
        p = -pivmin;
    int c = p < 0.0;

    for (int i = 1; i < n; i++) {
        double pn = fma(d[i] - x, p, -e2[i - 1] * pm);

        if (fabs(pn) < pivmin * fabs(p))
            pn = -pivmin * p;
        c += (pn < 0.0) != (p < 0.0);
        pm = p;
        p = pn;
        const double a = fabs(p);

        if (a > 0x1p400 || a < 0x1p-400) {
            const double sc = a > 1.0 ? 0x1p-400 : 0x1p400;

            p *= sc;
            pm *= sc;
        }
    }
    return c;
}

__device__ __forceinline__ int sturmf(const float *d, const float *e2, int n, float x,
                                      float pivmin)
{
    float q = d[0] - x;
    int c = q < 0.f;

    for (int i = 1; i < n; i++) {
        if (fabsf(q) < pivmin)
            q = -pivmin;
        q = d[i] - x - __fdividef(e2[i - 1], q);
        c += q < 0.f;
    }
    return c;
}

/* Pseudo-inverse of the symmetric W (double, full storage) in place, from
   its cyclic Jacobi eigendecomposition; eigenvalues |l| < 1e-9 are dropped
   (tests/reference.py:151-156). V is workspace (n x ld). Returns status
   bits. */
__device__ unsigned jacobi_pinv(int n, int ld, double *W, double *V, double *lam, int lane)
{
    unsigned status = TC_STATUS_ITER_CAP;

    for (int r = lane; r < n; r += 32)
        for (int j = 0; j < n; j++)
            V[r * ld + j] = r == j ? 1.0 : 0.0;
    __syncwarp();
    for (int sweep = 0; sweep < 60; sweep++) {
        double off = 0.0, dg = 0.0;

        for (int r = lane; r < n; r += 32)
            for (int j = 0; j < n; j++) {
                const double w = W[r * ld + j];

                if (j == r)
                    dg += w * w;
                else
                    off += w * w;
            }
        off = wsum<double>(off);
        dg = wsum<double>(dg);
        if (off <= 1.0e-30 * dg) {
            status = 0;
            break;
        }
        for (int p = 0; p < n - 1; p++)
            for (int q = p + 1; q < n; q++) {
                const double apq = W[p * ld + q];

                if (apq == 0.0)
                    continue;
                const double app = W[p * ld + p], aqq = W[q * ld + q];
                const double theta = (aqq - app) / (2.0 * apq);
                const double t = (theta >= 0.0 ? 1.0 : -1.0) /
                                 (fabs(theta) + sqrt(theta * theta + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;

                __syncwarp();
                for (int r = lane; r < n; r += 32) {
                    if (r != p && r != q) {
                        const double akp = W[r * ld + p], akq = W[r * ld + q];

                        W[r * ld + p] = c * akp - s * akq;
                        W[r * ld + q] = s * akp + c * akq;
                    }
                    const double vkp = V[r * ld + p], vkq = V[r * ld + q];

                    V[r * ld + p] = c * vkp - s * vkq;
                    V[r * ld + q] = s * vkp + c * vkq;
                }
                __syncwarp();
                for (int r = lane; r < n; r += 32)
                    if (r != p && r != q) {
                        W[p * ld + r] = W[r * ld + p];
                        W[q * ld + r] = W[r * ld + q];
                    }
                if (lane == 0) {
                    W[p * ld + p] = app - t * apq;
                    W[q * ld + q] = aqq + t * apq;
                    W[p * ld + q] = 0.0;
                    W[q * ld + p] = 0.0;
                }
                __syncwarp();
            }
    }
    for (int r = lane; r < n; r += 32)
        lam[r] = W[r * ld + r];
    __syncwarp();
    for (int i = lane; i < n; i += 32)
        for (int j = 0; j < n; j++) {
            double s = 0.0;

            for (int k = 0; k < n; k++) {
                const double l = lam[k];

                if (fabs(l) >= 1.0e-9)
                    s += V[i * ld + k] * V[j * ld + k] / l;
            }
            W[i * ld + j] = s;
        }
    __syncwarp();
    return status;
}

/* ------------------------------------------------------------------ */
/* The exact tier: a pixel from double-precision coherence sums.       */
/* ------------------------------------------------------------------ */

/* EMI divides by |T|, whose condition number reaches 1e5 - 1e6 on noisy or
   highly coherent stacks: the float rounding of the coherence sums and of
   their normalisation (a few 1e-7 relative) then moves gamma by up to 1e-3,
   however exactly the rest is computed. And the bias correction zeroes an
   entry at L m2 <= 1, a jump of gamma by up to 2 / (n (n - 1)) that float
   sums may place on the other side of the threshold. This tier recomputes
   a pixel from its samples with everything in double: the masked sums
   C = sum over SHPs q of s_q s_q^H (tcoh.cl:567-602, as tests/reference.py
   sums them), T and its bias correction (tcoh.cl:610-636); for EMI |T|^-1
   (ex_inverse: the symmetric sweep, Gauss-Jordan with partial pivoting,
   or the Jacobi pseudo-inverse with the absolute floor 1e-9 of
   tests/reference.py:151-156) and M = |T|^-1 o T, for EVD T itself; the
   Householder reduction to a real tridiagonal, the wanted eigenvalue by
   multisection on Sturm counts, inverse iteration and the
   back-transformation; then the phasors and gamma (tcoh.cl:696-744). It
   runs every pixel of the 33-64-date EMI path, and the pixels that the
   float kernels flag: ill-conditioned EMI pixels up to 32 dates, and with
   the bias correction any pixel with an entry at its threshold.

   One CTA of four warps per pixel, every matrix in packed upper-triangle
   storage (index tc_pidx) in shared memory, so that three pixels fit an
   SM at 60 dates: the sums and T (then M, in place) in complex double,
   |T| and its inverse in double (then a float copy of T for gamma in the
   same place). The sums accumulate in registers, each thread one to three
   2 x BC blocks of the triangle, over the SHP samples staged 16 candidates
   at a time, converted to double once at staging (a conversion costs four
   double FMAs' issue). */

constexpr int EX_THREADS = 128;
/* CTAs per SM: register blocks of the sums per thread NB = 1 (up to 32
   dates, 71 blocks of 2 x 4 entries at most) leave room for 6, NB = 3 (up
   to 64 dates) for 3 */
__host__ __device__ constexpr int ex_ctas(int nb) { return nb == 1 ? 6 : 3; }
constexpr int EX_KC = 16;         /* candidates per staging block */
/* the multisection's spacing: EX_THREADS points split an interval into
   EX_THREADS + 1 parts */
constexpr double EX_INV_POINTS = 1.0 / (EX_THREADS + 1);
constexpr int EX_NB = 3;          /* register blocks per thread, n <= 64 */
__host__ __device__ constexpr int ex_nb_for(int n) { return n <= 32 ? 1 : EX_NB; }
/* Columns per register block (2 rows x BC): 2 while the triangle's blocks
   fit one per thread (up to 30 dates), else 4. */
__host__ __device__ inline int ex_blocks(int n, int bc)
{
    const int rp = (n + 1) / 2, cg = (n + bc - 1) / bc;
    int nb = 0;

    for (int ip = 0; ip < rp; ip++)
        nb += cg - (2 * ip) / bc;
    return nb;
}
__host__ __device__ inline int ex_bc_for(int n) { return ex_blocks(n, 2) <= EX_THREADS ? 2 : 4; }
/* Row stride of the staged samples: n rounded up to 4, zero-padded. */
__host__ __device__ inline int ex_sld(int n) { return (n + 3) & ~3; }

struct ExLayout {
    int n, npu, nblk, ld;
    int off_T, off_G, off_tab, off_blk, off_stage, off_cand, off_vec, off_adj;
    int bytes;
};

struct ExWs {
    double2 *T;       /* [npu] sums, then T, then M */
    double *G;        /* [npu] |T|, then its inverse */
    float2 *Tf;       /* [npu] T in float, over G once M is formed */
    unsigned short *tab, *blk, *cand;
    double2 *stage;   /* [EX_KC][ex_sld(n)] */
    double *d, *e, *e2, *y, *lu, *rrow, *nrm, *red;
    double2 *v, *w, *tau, *z;
    float2 *zs;
    unsigned long long *adj;
    int *ints;        /* [0] candidates, [1] flags, [2..5] per warp, [6] next queue entry */
};

__host__ __device__ inline ExLayout ex_layout(int n, int area)
{
    ExLayout L;
    int off = 0;
    auto take = [&](int bytes) {
        const int o = off;

        off += (bytes + 15) & ~15;
        return o;
    };
    L.n = n;
    L.npu = tc_npu(n);
    L.ld = n | 1;
    L.nblk = ex_blocks(n, ex_bc_for(n));
    L.off_T = take(16 * L.npu);
    L.off_G = take(8 * L.npu);
    L.off_tab = take(2 * L.npu);
    L.off_blk = take(2 * L.nblk);
    /* the staged samples; once the sums are formed, up to 32 dates, the
       full |T| of the Gauss-Jordan inverse tier */
    L.off_stage = take(n <= 32 && 8 * n * n > 16 * EX_KC * ex_sld(n) ? 8 * n * n
                                                                      : 16 * EX_KC * ex_sld(n));
    L.off_cand = take(2 * area);
    L.off_vec = take(8 * (8 * 64 + 16 + 4 * 64) + 16 * 5 * 64 + 8 * 64 + 16);
    L.off_adj = take(8 * 64);
    L.bytes = off;
    return L;
}

__device__ __forceinline__ ExWs ex_ws(unsigned char *base, const ExLayout &L)
{
    ExWs w;
    double *v = (double *)(base + L.off_vec);

    w.T = (double2 *)(base + L.off_T);
    w.G = (double *)(base + L.off_G);
    w.Tf = (float2 *)(base + L.off_G);
    w.tab = (unsigned short *)(base + L.off_tab);
    w.blk = (unsigned short *)(base + L.off_blk);
    w.stage = (double2 *)(base + L.off_stage);
    w.cand = (unsigned short *)(base + L.off_cand);
    w.d = v;
    w.e = v + 64;
    w.e2 = v + 128;
    w.y = v + 192;
    w.rrow = v + 256;
    w.nrm = v + 320;
    w.red = v + 384;        /* 2 x 8 */
    w.lu = v + 400;         /* 4 x 64 */
    double2 *c = (double2 *)(v + 400 + 256);

    w.v = c;
    w.w = c + 64;
    w.tau = c + 128;
    w.z = c + 192;
    w.zs = (float2 *)(c + 320);
    w.ints = (int *)(w.zs + 64);
    w.adj = (unsigned long long *)(base + L.off_adj);
    return w;
}

/* 1 / x in double: a float reciprocal refined by two Newton steps
   r <- r (2 - x r), each doubling the correct bits (24 -> 48 -> 96, so
   within an ulp or two of 1 / x). For |x| in the float range: the LU
   pivots here, clamped to at least 1e-13 of the tridiagonal's norm, which
   is of order 1 or more (T has a unit diagonal, |T|^-1 o T one of 1 or
   more, a pseudo-inverse's at least about 1 / n^2). */
__device__ __forceinline__ double ex_rcp(double x)
{
    double r = (double)__frcp_rn((float)x);

    r = r * fma(-x, r, 2.0);
    return r * fma(-x, r, 2.0);
}

/* 1 / x for any x: ex_rcp inside [1e-30, 1e30] in magnitude, else the
   division. */
__device__ __forceinline__ double ex_rcp_any(double x)
{
    const double a = fabs(x);

    return a > 1.0e-30 && a < 1.0e30 ? ex_rcp(x) : 1.0 / x;
}

/* Block sums over the CTA (every thread gets them); red holds 8 doubles. */
__device__ __forceinline__ double2 ex_sum2(double a, double b, double *red)
{
    a = wsum<double>(a);
    b = wsum<double>(b);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = a;
        red[4 + (threadIdx.x >> 5)] = b;
    }
    __syncthreads();
    return make_double2(red[0] + red[1] + red[2] + red[3], red[4] + red[5] + red[6] + red[7]);
}

/* The same without the leading barrier, for callers that alternate
   between two halves of red (red + 8 * parity) with a barrier between two
   uses of one half. */
__device__ __forceinline__ double2 ex_sum2p(double a, double b, double *red)
{
    a = wsum<double>(a);
    b = wsum<double>(b);
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = a;
        red[4 + (threadIdx.x >> 5)] = b;
    }
    __syncthreads();
    return make_double2(red[0] + red[1] + red[2] + red[3], red[4] + red[5] + red[6] + red[7]);
}

/* Packed (i, j) of the upper triangle for any order of i, j. */
__device__ __forceinline__ int ex_sym(int n, int i, int j)
{
    return i <= j ? tc_pidx(n, i, j) : tc_pidx(n, j, i);
}

/* M_ij (Hermitian) from packed upper storage. */
__device__ __forceinline__ double2 ex_m(const double2 *P, int n, int i, int j)
{
    if (i <= j)
        return P[tc_pidx(n, i, j)];
    const double2 m = P[tc_pidx(n, j, i)];

    return make_double2(m.x, -m.y);
}

/* The pixel's SHP candidates (window indices) into w.cand; their number.
   Mask word i of the pixel is words[i * stride]. */
__device__ int ex_candidates(const TcStrip &s, const uint32_t *words, long long stride,
                             const ExWs &w)
{
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        uint32_t bits = lane < s.mask_words ? words[lane * stride] : 0u;

        if (lane == s.mask_words - 1 && (s.area & 31))
            bits &= (1u << (s.area & 31)) - 1u; /* candidates only */
        const int cnt = __popc(bits);
        int off = cnt;

#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, off, o);

            if (lane >= o)
                off += v;
        }
        if (lane == 31)
            w.ints[0] = off;
        off -= cnt;
        while (bits) {
            const int b = __ffs(bits) - 1;

            bits &= bits - 1;
            w.cand[off++] = (unsigned short)(lane * 32 + b);
        }
    }
    __syncthreads();
    return w.ints[0];
}

/* C = sum of s_q s_q^H over the candidates, in double, into w.T (packed);
   NB register blocks per thread (L.nblk <= NB * EX_THREADS). */
template <int NB, int BC>
__device__ void ex_gram(const TcStrip &s, const float2 *slc, int py0, int px0, int ncand,
                        const ExWs &w, const ExLayout &L)
{
    const int n = s.n, t = threadIdx.x;
    const int sld = ex_sld(n);
    double2 acc[NB][2][BC];
    int bi[NB], bj[NB];

#pragma unroll
    for (int b = 0; b < NB; b++) {
        const int id = t + b * EX_THREADS;

        bi[b] = bj[b] = -1;
        if (id < L.nblk) {
            bi[b] = 2 * (w.blk[id] >> 8);
            bj[b] = BC * (w.blk[id] & 255);
        }
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int q = 0; q < BC; q++)
                acc[b][r][q] = make_double2(0.0, 0.0);
    }
    for (int c0 = 0; c0 < ncand; c0 += EX_KC) {
        const int kc = min(EX_KC, ncand - c0);

        for (int q = t >> 5; q < kc; q += EX_THREADS / 32) {
            const int u = w.cand[c0 + q], dy = u / s.wr, dx = u - dy * s.wr;
            const float2 *src = slc + ((long long)(py0 + dy) * s.W + px0 + dx) * n;

            for (int d = t & 31; d < sld; d += 32) {
                float2 v = d < n ? src[d] : make_float2(0.f, 0.f);

                if (!isfinite(v.x) || !isfinite(v.y))
                    v = make_float2(0.f, 0.f);
                w.stage[q * sld + d] = make_double2(v.x, v.y);
            }
        }
        __syncthreads();
#pragma unroll
        for (int b = 0; b < NB; b++) {
            if (bi[b] < 0)
                continue;
            for (int q = 0; q < kc; q++) {
                const double2 *row = w.stage + q * sld;
                double2 a[2], cj[BC];

#pragma unroll
                for (int r = 0; r < 2; r++)
                    a[r] = row[bi[b] + r];
#pragma unroll
                for (int jj = 0; jj < BC; jj++)
                    cj[jj] = row[bj[b] + jj];
#pragma unroll
                for (int r = 0; r < 2; r++)
#pragma unroll
                    for (int jj = 0; jj < BC; jj++) {
                        /* a conj(b) */
                        acc[b][r][jj].x = fma(a[r].x, cj[jj].x, fma(a[r].y, cj[jj].y, acc[b][r][jj].x));
                        acc[b][r][jj].y = fma(a[r].y, cj[jj].x, fma(-a[r].x, cj[jj].y, acc[b][r][jj].y));
                    }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int b = 0; b < NB; b++) {
        if (bi[b] < 0)
            continue;
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int jj = 0; jj < BC; jj++) {
                const int i = bi[b] + r, j = bj[b] + jj;

                if (i < n && j < n && i <= j)
                    w.T[tc_pidx(n, i, j)] = acc[b][r][jj];
            }
    }
    __syncthreads();
}

/* T from the sums (tcoh.cl:611-636 in double, as tests/reference.py:124-142)
   and |T|. */
__device__ void ex_coherence(int n, int npu, const TcLinkConst &k, int looks, const ExWs &w)
{
    const int t = threadIdx.x;

    for (int i = t; i < n; i += EX_THREADS)
        w.nrm[i] = sqrt(w.T[tc_pidx(n, i, i)].x);
    __syncthreads();
    const double fl = (double)looks, ifl1 = looks > 1 ? 1.0 / (fl - 1.0) : 0.0;

    for (int q = t; q < npu; q += EX_THREADS) {
        const int i = w.tab[q] >> 8, j = w.tab[q] & 255;
        double2 v = make_double2(1.0, 0.0);

        if (i != j) {
            const double dd = w.nrm[i] * w.nrm[j];
            const double2 cs = w.T[q];

            v = make_double2(0.0, 0.0);
            if (dd > 0.0) {
                const double rdd = ex_rcp_any(dd);

                v = make_double2(cs.x * rdd, cs.y * rdd);
                if (k.bias && looks > 1) {
                    const double m2 = v.x * v.x + v.y * v.y;
                    const double m2c = (fl * m2 - 1.0) * ifl1;
                    const double f = (m2 > 0.0 && m2c > 0.0) ? sqrt(m2c * ex_rcp_any(m2)) : 0.0;

                    v.x *= f;
                    v.y *= f;
                }
            }
        }
        w.T[q] = v;
        w.G[q] = hypot(v.x, v.y);
    }
    __syncthreads();
}

/* Whether the non-zero coherences link all dates (tcoh.cl:494-513). */
__device__ bool ex_linked(int n, const ExWs &w)
{
    const int t = threadIdx.x;

    for (int i = t; i < n; i += EX_THREADS) {
        unsigned long long a = 0ull;

        for (int j = 0; j < n; j++)
            if (j != i && w.G[ex_sym(n, i, j)] != 0.0)
                a |= 1ull << j;
        w.adj[i] = a;
    }
    __syncthreads();
    if (t < 32) {
        const unsigned long long all = n == 64 ? ~0ull : (1ull << n) - 1ull;
        unsigned long long reached = 1ull, frontier = 1ull;

        for (int it = 0; it < n; it++) {
            unsigned long long mine = 0ull;

            if ((frontier >> t) & 1ull)
                mine |= w.adj[t];
            if (t + 32 < n && ((frontier >> (t + 32)) & 1ull))
                mine |= w.adj[t + 32];
            const unsigned lo = __reduce_or_sync(FULL, (unsigned)mine);
            const unsigned hi = __reduce_or_sync(FULL, (unsigned)(mine >> 32));
            const unsigned long long nw = (((unsigned long long)hi << 32) | lo) & ~reached;

            if (!nw)
                break;
            reached |= nw;
            frontier = nw;
        }
        if (t == 0)
            w.ints[1] = reached == all;
    }
    __syncthreads();
    return w.ints[1] != 0;
}

/* A^-1 in place of the packed symmetric A by the symmetric sweep
   (Gauss-Jordan elimination without pivoting in the form that keeps the
   matrix symmetric; Goodnight, The American Statistician 33, 1979):
   sweeping pivot k maps a_ij -> a_ij - a_ik a_kj / a_kk,
   a_ik, a_kj -> a_ik / a_kk, a_kk -> -1 / a_kk, and all pivots leave
   -A^-1, negated back at the end. It takes indefinite matrices. False when
   a pivot's magnitude is not above floor_ (A is then as it was).

   The matrix is in registers, TPR threads per row: thread h of a row has the
   columns c = h mod TPR, in the order of the pivots to come (register q: column
   TPR (shift + q) + h), so that pivot k is register 0 of the threads h = k mod
   TPR, with static indices, and TPR pivots make one shift of the registers.
   Those threads publish the pivot column, which is the pivot row (the matrix
   stays symmetric), in the order in which each thread reads its part; the next
   column goes out as soon as it is updated, into the other of two buffers, so
   that one barrier a pivot suffices. With the packed triangle in shared memory
   every update came with four shared accesses and its index arithmetic: 297
   thousand cycles a pixel at 60 dates, 50 thousand now (63 and 24 at 30); the
   link stage of 40 x 1024 pixels at 60 dates, EMI, 37.4 -> 27.8 ms. */
template <int TPR>
__device__ bool ex_sweep(int n, const ExWs &w, double *A, double floor_)
{
    constexpr int NR = EX_THREADS / TPR, CP = NR / TPR; /* rows; columns per thread */
    constexpr int PS = CP + 2; /* parts 16 bytes apart modulo the banks */
    const int t = threadIdx.x, i = t / TPR, h = t % TPR;
    double g[CP];
    int shift = 0;
    /* place of row i's entry in a buffer */
    auto place = [&](int sh) { return (i % TPR) * PS + ((i / TPR - sh) & (CP - 1)); };

#pragma unroll
    for (int q = 0; q < CP; q++) {
        const int c = TPR * q + h;

        g[q] = i < n && c < n ? A[ex_sym(n, i, c)] : 0.0;
    }
    if (h == 0)
        w.lu[place(0)] = g[0];
    __syncthreads();
#pragma unroll 1
    for (int base = 0; base < n; base += TPR) {
#pragma unroll
        for (int s = 0; s < TPR; s++) {
            const int k = base + s;

            if (k >= n)
                break;
            const double *r = w.lu + TPR * PS * (k & 1);
            double *rn = w.lu + TPR * PS * ((k + 1) & 1);
            const double d = r[s * PS];

            if (!(fabs(d) > floor_)) {
                __syncthreads();
                return false;
            }
            const double id = ex_rcp_any(d);
            /* the pivot row scales by 1 / a_kk: a_kj - (1 - 1 / a_kk) a_kj */
            const double f = i == k ? 1.0 - id : r[place(shift)] * id;
            auto update = [&](int q) { g[q] = fma(-f, r[h * PS + q], g[q]); };

            update(0);
            update(1);
            if (h == (s + 1) % TPR)
                rn[place(shift + (s + 1 == TPR))] = s + 1 == TPR ? g[1] : g[0];
#pragma unroll
            for (int q = 2; q < CP; q++)
                update(q);
            if (h == s)
                g[0] = i == k ? -id : f;
            if (s + 1 == TPR) {
                const double g0 = g[0];

#pragma unroll
                for (int q = 0; q < CP - 1; q++)
                    g[q] = g[q + 1];
                g[CP - 1] = g0;
                shift++;
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int q = 0; q < CP; q++) {
        const int c = TPR * ((shift + q) & (CP - 1)) + h;

        if (i <= c && c < n)
            A[tc_pidx(n, i, c)] = -g[q];
    }
    __syncthreads();
    return true;
}

/* Whether the packed inverse is finite and moderate: n max|inv_ij| < 1e8,
   which keeps every eigenvalue of |T| above the pseudo-inverse floor 1e-9
   of tests/reference.py:151-156, where the pseudo-inverse is the inverse. */
__device__ bool ex_moderate(int n, int npu, const ExWs &w, const double *A)
{
    const int t = threadIdx.x;
    double mx = 0.0;

    for (int q = t; q < npu; q += EX_THREADS) {
        const double v = A[q];

        mx = v == v ? fmax(mx, fabs(v)) : INFINITY;
    }
    mx = wmaxd(mx);
    __syncthreads();
    if ((t & 31) == 0)
        w.red[t >> 5] = mx;
    __syncthreads();
    mx = fmax(fmax(w.red[0], w.red[1]), fmax(w.red[2], w.red[3]));
    __syncthreads();
    return mx <= 1.0e300 && n * mx < 1.0e8;
}

/* A^-1 in place of the full n x n A (row-major) by Gauss-Jordan
   elimination with partial pivoting (the row of the largest magnitude in
   the pivot column; the column permutation is undone at the end). It takes
   indefinite and ill-conditioned matrices; false when a pivot falls below
   1e-14 of the largest entry (numerically singular). */
__device__ bool ex_gauss_jordan(int n, const ExWs &w, double *A)
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int *perm = (int *)w.adj;
    double amax = 0.0;

    for (int e = t; e < n * n; e += EX_THREADS)
        amax = fmax(amax, fabs(A[e]));
    amax = wmaxd(amax);
    if (lane == 0)
        w.red[warp] = amax;
    __syncthreads();
    amax = fmax(fmax(w.red[0], w.red[1]), fmax(w.red[2], w.red[3]));
    __syncthreads();
    for (int k = 0; k < n; k++) {
        /* pivot row: the largest |A[i][k]|, i >= k */
        double v = t >= k && t < n ? fabs(A[t * n + k]) : -1.0;
        int idx = t;

#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const double ov = __shfl_xor_sync(FULL, v, o);
            const int oi = __shfl_xor_sync(FULL, idx, o);

            if (ov > v || (ov == v && oi < idx)) {
                v = ov;
                idx = oi;
            }
        }
        if (lane == 0) {
            w.red[warp] = v;
            w.ints[2 + warp] = idx;
        }
        __syncthreads();
        int p = w.ints[2];
        double best = w.red[0];

        for (int q = 1; q < EX_THREADS / 32; q++)
            if (w.red[q] > best) {
                best = w.red[q];
                p = w.ints[2 + q];
            }
        __syncthreads();
        if (!(best > 1.0e-14 * amax))
            return false;
        if (t == 0)
            perm[k] = p;
        /* swap rows p and k, then scale row k (its pivot becomes 1 / piv) */
        const double piv = A[p * n + k];

        __syncthreads();
        for (int j = t; j < n; j += EX_THREADS) {
            const double rk = A[k * n + j], rp = A[p * n + j];

            A[p * n + j] = rk;
            A[k * n + j] = (j == k ? 1.0 : rp) / piv;
        }
        __syncthreads();
        for (int i = t; i < n; i += EX_THREADS)
            w.rrow[i] = i == k ? 0.0 : A[i * n + k];
        __syncthreads();
        for (int i = warp; i < n; i += EX_THREADS / 32)
            if (i != k)
                for (int j = lane; j < n; j += 32)
                    A[i * n + j] = (j == k ? 0.0 : A[i * n + j]) - A[k * n + j] * w.rrow[i];
        __syncthreads();
    }
    /* undo the row swaps on the columns of the inverse, last swap first */
    for (int k = n - 1; k >= 0; k--) {
        const int p = perm[k];

        if (p != k)
            for (int i = t; i < n; i += EX_THREADS) {
                const double x = A[i * n + k];

                A[i * n + k] = A[i * n + p];
                A[i * n + p] = x;
            }
        __syncthreads();
    }
    return true;
}

/* |T|^-1 into w.G (which holds |T|), in tiers: the symmetric sweep with
   pivots above 1e-5; else Gauss-Jordan elimination with partial pivoting
   on the full |T| (in shared memory, the staged samples' region, up to 32
   dates; in the CTA's global scratch W above); else, or when the inverse is
   not moderate, the Jacobi eigen-pseudo-inverse with the absolute floor
   1e-9 (tests/reference.py:151-156) on warp 0. Returns status bits. */
template <int TPR>
__device__ unsigned ex_inverse(int n, int npu, int ld, const ExWs &w, double *W)
{
    const int t = threadIdx.x;

    if (ex_sweep<TPR>(n, w, w.G, 1.0e-5) && ex_moderate(n, npu, w, w.G))
        return 0;
    double *A = n <= 32 ? (double *)w.stage : W;

    for (int i = t >> 5; i < n; i += EX_THREADS / 32)
        for (int j = t & 31; j < n; j += 32) {
            const double2 v = ex_m(w.T, n, i, j);

            A[i * n + j] = i == j ? 1.0 : hypot(v.x, v.y);
        }
    __syncthreads();
    if (ex_gauss_jordan(n, w, A)) {
        for (int q = t; q < npu; q += EX_THREADS) {
            const int i = w.tab[q] >> 8, j = w.tab[q] & 255;

            w.G[q] = 0.5 * (A[i * n + j] + A[j * n + i]);
        }
        __syncthreads();
        if (ex_moderate(n, npu, w, w.G))
            return TC_STATUS_EMI_PIVOTED;
    }
    __syncthreads();
    unsigned st = TC_STATUS_EMI_PINV;

    if (t < 32) {
        double *V = W + n * ld, *lam = W + 2 * n * ld;

        for (int r = t; r < n; r += 32)
            for (int j = 0; j < n; j++) {
                const double2 v = ex_m(w.T, n, r, j);

                W[r * ld + j] = r == j ? 1.0 : hypot(v.x, v.y);
            }
        __syncwarp();
        st |= jacobi_pinv(n, ld, W, V, lam, t);
        for (int r = t; r < n; r += 32)
            for (int j = r; j < n; j++)
                w.G[tc_pidx(n, r, j)] = W[r * ld + j];
    }
    if (t == 0)
        w.ints[1] = (int)st;
    __syncthreads();
    return (unsigned)w.ints[1];
}

/* Row i = k + 1 + t / R of M22 v (the trailing block at step k, v in w.v),
   R threads per row, thread h = t % R taking the columns j = h mod R: M_ij
   = conj(P(j, i)) for j < i, at rb(j) + i - j with rb(j) = j (2n - j + 1) /
   2, then P(i, j) for j >= i, contiguous. Separate accumulators for the two
   products of each part keep the FMA chains one deep; the R threads' sums
   are combined by shuffles (every thread gets its row's). */
template <int R>
__device__ __forceinline__ void ex_matvec_rows(int n, int k, const ExWs &w, int t, int &i, int &h,
                                               double &sx, double &sy)
{
    i = k + 1 + t / R;
    h = t % R;
    sx = sy = 0.0;
    if (i < n) {
        int j = k + 1 + h;
        int idx = j * (2 * n - j + 1) / 2 + (i - j);
        double ax = 0.0, bx = 0.0, ay = 0.0, by = 0.0;

        for (; j < i; j += R) {
            const double2 m = w.T[idx], v = w.v[j];

            ax = fma(m.x, v.x, ax);
            bx = fma(m.y, v.y, bx);
            ay = fma(m.x, v.y, ay);
            by = fma(m.y, v.x, by);
            idx += R * (n - j) - R * (R + 1) / 2;
        }
        sx = ax + bx;
        sy = ay - by;
        ax = bx = ay = by = 0.0;
        for (idx = i * (2 * n - i + 1) / 2 + (j - i); j < n; j += R, idx += R) {
            const double2 m = w.T[idx], v = w.v[j];

            ax = fma(m.x, v.x, ax);
            bx = fma(m.y, v.y, bx);
            ay = fma(m.x, v.y, ay);
            by = fma(m.y, v.x, by);
        }
        sx += ax - bx;
        sy += ay + by;
    }
#pragma unroll
    for (int o = 1; o < R; o <<= 1) {
        sx += __shfl_xor_sync(FULL, sx, o);
        sy += __shfl_xor_sync(FULL, sy, o);
    }
}

/* Householder reduction of the packed Hermitian M (w.T) to the real
   tridiagonal (w.d, w.e), zhetd2 form; reflector k's vector is left in
   packed row k (entries k + 2 ..; its entry k + 1 is 1) and its scalar in
   w.tau[k]. Two forms: up to 32 dates five CTA barriers a step
   (ex_householder_cta); above, three (ex_householder_lean: every warp
   reduces the pivot column itself, and w = p + h v is formed where the
   rank-2 update reads it), which pays where the steps are many. */
__device__ void ex_householder_cta(int n, int npu, const ExWs &w)
{
    const int t = threadIdx.x;

    for (int k = 0; k < n - 1; k++) {
        /* column k below the diagonal: x_r = conj(M_k,r) */
        double xn2 = 0.0;

        if (t < n - k - 2) {
            const double2 a = w.T[tc_pidx(n, k, k + 2 + t)];

            xn2 = a.x * a.x + a.y * a.y;
        }
        /* two barriers separate this half of red from its last use */
        xn2 = ex_sum2p(xn2, 0.0, w.red).x;
        const double2 am = w.T[tc_pidx(n, k, k + 1)];
        const double ax = am.x, ay = -am.y; /* alpha = x_k+1 */
        double beta, tr = 0.0, ti = 0.0, sr = 0.0, si = 0.0;

        if (xn2 == 0.0 && ay == 0.0)
            beta = ax;
        else {
            beta = -copysign(sqrt(ax * ax + ay * ay + xn2), ax);
            const double rb = ex_rcp_any(beta);

            tr = (beta - ax) * rb;
            ti = -ay * rb;
            const double dr = ax - beta, di = ay, rden = ex_rcp_any(dr * dr + di * di);

            sr = dr * rden;
            si = -di * rden;
        }
        const bool reflect = tr != 0.0 || ti != 0.0;

        if (t < n) {
            double2 v = make_double2(0.0, 0.0);

            if (t == k + 1)
                v = make_double2(1.0, 0.0);
            else if (t > k + 1 && reflect) {
                const double2 a = w.T[tc_pidx(n, k, t)];
                const double xr = a.x, xi = -a.y;

                v = make_double2(xr * sr - xi * si, xr * si + xi * sr);
                w.T[tc_pidx(n, k, t)] = v;
            }
            w.v[t] = v;
        }
        if (t == 0) {
            w.d[k] = w.T[tc_pidx(n, k, k)].x;
            w.e[k] = beta;
            w.tau[k] = make_double2(tr, ti);
        }
        __syncthreads();
        if (!reflect)
            continue;
        /* p = M22 v over rows k+1 .. n-1, four threads per row */
        double sx, sy;
        int i, h;

        ex_matvec_rows<4>(n, k, w, t, i, h, sx, sy);
        const double2 wl = make_double2(tr * sx - ti * sy, tr * sy + ti * sx);
        double pr = 0.0, pi = 0.0;

        if (i < n && h == 0) {
            const double2 v = w.v[i];

            pr = wl.x * v.x + wl.y * v.y;
            pi = wl.x * v.y - wl.y * v.x;
        }
        const double2 pp = ex_sum2p(pr, pi, w.red + 8);
        const double hr = -0.5 * (tr * pp.x - ti * pp.y), hi = -0.5 * (tr * pp.y + ti * pp.x);

        if (i < n && h == 0) {
            const double2 v = w.v[i];

            w.w[i] = make_double2(wl.x + hr * v.x - hi * v.y, wl.y + hr * v.y + hi * v.x);
        }
        __syncthreads();
        /* M22 -= v w^H + w v^H over the trailing triangle (contiguous) */
        for (int q = tc_pidx(n, k + 1, k + 1) + t; q < npu; q += EX_THREADS) {
            const int r = w.tab[q] >> 8, j = w.tab[q] & 255;
            const double2 vr = w.v[r], wr = w.w[r], vj = w.v[j], wj = w.w[j];
            double2 a = w.T[q];

            a.x -= vr.x * wj.x + vr.y * wj.y + wr.x * vj.x + wr.y * vj.y;
            a.y -= vr.y * wj.x - vr.x * wj.y + wr.y * vj.x - wr.x * vj.y;
            w.T[q] = a;
        }
        __syncthreads();
    }
    if (t == 0)
        w.d[n - 1] = w.T[tc_pidx(n, n - 1, n - 1)].x;
    __syncthreads();
}

__device__ void ex_householder_lean(int n, int npu, const ExWs &w)
{
    const int t = threadIdx.x;

    for (int k = 0; k < n - 1; k++) {
        /* column k below the diagonal: x_r = conj(M_k,r); every warp
           reduces it itself (no CTA barrier) */
        const int lane = t & 31;
        double xn2 = 0.0;

        for (int r = lane; r < n - k - 2; r += 32) {
            const double2 a = w.T[tc_pidx(n, k, k + 2 + r)];

            xn2 = fma(a.x, a.x, fma(a.y, a.y, xn2));
        }
        xn2 = wsum<double>(xn2);
        const double2 am = w.T[tc_pidx(n, k, k + 1)];
        const double ax = am.x, ay = -am.y; /* alpha = x_k+1 */
        double beta, tr = 0.0, ti = 0.0, sr = 0.0, si = 0.0;

        if (xn2 == 0.0 && ay == 0.0)
            beta = ax;
        else {
            beta = -copysign(sqrt(ax * ax + ay * ay + xn2), ax);
            const double rb = ex_rcp_any(beta);

            tr = (beta - ax) * rb;
            ti = -ay * rb;
            const double dr = ax - beta, di = ay, rden = ex_rcp_any(dr * dr + di * di);

            sr = dr * rden;
            si = -di * rden;
        }
        const bool reflect = tr != 0.0 || ti != 0.0;
        /* v, into w.v now and into column k of T (which keeps the
           reflectors) after the barrier: other warps may still be reading
           the column */
        double2 vk = make_double2(0.0, 0.0);

        if (t < n) {
            if (t == k + 1)
                vk = make_double2(1.0, 0.0);
            else if (t > k + 1 && reflect) {
                const double2 a = w.T[tc_pidx(n, k, t)];
                const double xr = a.x, xi = -a.y;

                vk = make_double2(xr * sr - xi * si, xr * si + xi * sr);
            }
            w.v[t] = vk;
        }
        if (t == 0) {
            w.d[k] = w.T[tc_pidx(n, k, k)].x;
            w.e[k] = beta;
            w.tau[k] = make_double2(tr, ti);
        }
        __syncthreads();
        if (!reflect)
            continue;
        if (t > k + 1 && t < n)
            w.T[tc_pidx(n, k, t)] = vk;
        /* p = M22 v over rows k+1 .. n-1, two threads per row */
        double sx, sy;
        int i, h;

        ex_matvec_rows<2>(n, k, w, t, i, h, sx, sy);
        const double2 wl = make_double2(tr * sx - ti * sy, tr * sy + ti * sx);
        double pr = 0.0, pi = 0.0;

        if (i < n && h == 0) {
            const double2 v = w.v[i];

            pr = wl.x * v.x + wl.y * v.y;
            pi = wl.x * v.y - wl.y * v.x;
            /* w = wl + h v, the correction h known after the barrier */
            w.w[i] = wl;
        }
        pr = wsum<double>(pr);
        pi = wsum<double>(pi);
        if (lane == 0) {
            w.red[t >> 5] = pr;
            w.red[4 + (t >> 5)] = pi;
        }
        __syncthreads();
        const double ppx = w.red[0] + w.red[1] + w.red[2] + w.red[3];
        const double ppy = w.red[4] + w.red[5] + w.red[6] + w.red[7];
        const double hr = -0.5 * (tr * ppx - ti * ppy), hi = -0.5 * (tr * ppy + ti * ppx);

        /* M22 -= v w^H + w v^H over the trailing triangle (contiguous) */
        for (int q = tc_pidx(n, k + 1, k + 1) + t; q < npu; q += EX_THREADS) {
            const int r = w.tab[q] >> 8, j = w.tab[q] & 255;
            const double2 vr = w.v[r], vj = w.v[j], lr = w.w[r], lj = w.w[j];
            const double2 wr = make_double2(lr.x + hr * vr.x - hi * vr.y, lr.y + hr * vr.y + hi * vr.x);
            const double2 wj = make_double2(lj.x + hr * vj.x - hi * vj.y, lj.y + hr * vj.y + hi * vj.x);
            double2 a = w.T[q];

            a.x -= vr.x * wj.x + vr.y * wj.y + wr.x * vj.x + wr.y * vj.y;
            a.y -= vr.y * wj.x - vr.x * wj.y + wr.y * vj.x - wr.x * vj.y;
            w.T[q] = a;
        }
        __syncthreads();
    }
    if (t == 0)
        w.d[n - 1] = w.T[tc_pidx(n, n - 1, n - 1)].x;
    __syncthreads();
}

/* LEAN (above 32 dates) or not, chosen at compile time so that each kernel
   holds only the code it runs: the chains here are latency-bound and
   sensitive to instruction-cache misses. */
template <bool LEAN>
__device__ void ex_householder(int n, int npu, const ExWs &w)
{
    if constexpr (LEAN)
        ex_householder_lean(n, npu, w);
    else
        ex_householder_cta(n, npu, w);
}

/* Eigenvalue of rank `index` of (w.d, w.e) (0: the smallest, for EMI;
   n - 1: the largest, for EVD) by 128-way multisection on double Sturm
   counts, then its eigenvector by inverse iteration (thread 0), then
   z = Q y by the reflectors (warp 0): into w.z. Returns status bits. */
__device__ unsigned ex_eigvec(int n, int index, const ExWs &w)
{
    const int t = threadIdx.x;
    unsigned status = 0;
    double lo = INFINITY, hi = -INFINITY;

    if (t < n) {
        const double rad = (t > 0 ? fabs(w.e[t - 1]) : 0.0) + (t < n - 1 ? fabs(w.e[t]) : 0.0);

        lo = w.d[t] - rad;
        hi = w.d[t] + rad;
        if (t < n - 1)
            w.e2[t] = w.e[t] * w.e[t];
    }
    {
        double a = lo, b = hi;

#pragma unroll
        for (int o = 16; o; o >>= 1) {
            a = fmin(a, __shfl_xor_sync(FULL, a, o));
            b = fmax(b, __shfl_xor_sync(FULL, b, o));
        }
        __syncthreads();
        if ((t & 31) == 0) {
            w.red[t >> 5] = a;
            w.red[4 + (t >> 5)] = b;
        }
        __syncthreads();
        lo = fmin(fmin(w.red[0], w.red[1]), fmin(w.red[2], w.red[3]));
        hi = fmax(fmax(w.red[4], w.red[5]), fmax(w.red[6], w.red[7]));
        __syncthreads();
    }
    const double norm = fmax(fabs(lo), fabs(hi));

    lo -= 1.0e-12 * norm + 1e-300;
    hi += 1.0e-12 * norm + 1e-300;
    /* float Sturm counts first (on float copies in the LU's region), down to
       a few float ulps of the spectrum's scale; then, the interval widened
       by the float counts' possible error, double counts */
    float *df = (float *)w.lu, *e2f = df + 64;

    for (int r = t; r < n; r += EX_THREADS) {
        df[r] = (float)w.d[r];
        if (r < n - 1)
            e2f[r] = (float)w.e2[r];
    }
    __syncthreads();
    for (int fr = 0; fr < 4 && hi - lo > 1.0e-6 * norm; fr++) {
        const double xq = lo + (hi - lo) * ((double)(t + 1) * EX_INV_POINTS);
        const bool gt = sturmf(df, e2f, n, (float)xq, 1.0e-30f + 1.0e-14f * (float)norm) > index;
        const unsigned bal = __ballot_sync(FULL, gt);

        if ((t & 31) == 0)
            w.ints[2 + (t >> 5)] = bal ? (t & ~31) + __ffs(bal) - 1 : EX_THREADS;
        __syncthreads();
        const int f = min(min(w.ints[2], w.ints[3]), min(w.ints[4], w.ints[5]));
        const double nlo = f == 0 ? lo : lo + (hi - lo) * ((double)f * EX_INV_POINTS);
        const double nhi =
            f == EX_THREADS ? hi : lo + (hi - lo) * ((double)(f + 1) * EX_INV_POINTS);

        __syncthreads();
        lo = nlo;
        hi = nhi;
    }
    lo -= 4.0e-7 * norm;
    hi += 4.0e-7 * norm;
    const double pivmin = 1e-290 + 1e-28 * norm;
    int round = 0;

    for (; round < 12; round++) {
        if (hi - lo <= 2.0e-15 * norm)
            break;
        const double xq = lo + (hi - lo) * ((double)(t + 1) * EX_INV_POINTS);
        const bool gt = sturmd_minors(w.d, w.e2, n, xq, pivmin) > index;
        const unsigned bal = __ballot_sync(FULL, gt);

        if ((t & 31) == 0)
            w.ints[2 + (t >> 5)] = bal ? (t & ~31) + __ffs(bal) - 1 : EX_THREADS;
        __syncthreads();
        const int f = min(min(w.ints[2], w.ints[3]), min(w.ints[4], w.ints[5]));
        double nlo, nhi;

        if (f == EX_THREADS) {
            nlo = lo + (hi - lo) * ((double)EX_THREADS * EX_INV_POINTS);
            nhi = hi;
        }
        else {
            nhi = lo + (hi - lo) * ((double)(f + 1) * EX_INV_POINTS);
            nlo = f == 0 ? lo : lo + (hi - lo) * ((double)f * EX_INV_POINTS);
        }
        __syncthreads();
        if (!(nlo > lo || nhi < hi))
            break;
        lo = fmax(nlo, lo);
        hi = fmin(nhi, hi);
    }
    if (round == 12)
        status |= TC_STATUS_ITER_CAP;
    const double lambda = 0.5 * (lo + hi);

    /* Inverse iteration: LU of T - lambda I with partial pivoting, three
       solves from a vector of ones (the method of tcoh.cl:342-410). The
       recurrences carry their running values in registers; the shared
       arrays only hold what a later pass reads. */
    if (t == 0) {
        const double tiny = 1.0e-13 * (norm > 1e-300 ? norm : 1e-300);
        double *__restrict__ lu = w.lu;
        double *__restrict__ y = w.y;
        const double *__restrict__ dg = w.d;
        const double *__restrict__ eg = w.e;
        unsigned long long piv = 0ull;
        double dd = dg[0] - lambda, s1 = n > 1 ? eg[0] : 0.0;

        for (int kk = 0; kk < n - 1; kk++) {
            const double sub = eg[kk], nd = dg[kk + 1] - lambda;
            const double ns = kk + 1 < n - 1 ? eg[kk + 1] : 0.0;

            if (fabs(dd) >= fabs(sub)) {
                if (fabs(dd) < tiny)
                    dd = dd < 0.0 ? -tiny : tiny;
                const double rd = ex_rcp(dd), l = sub * rd;

                lu[4 * kk] = rd;
                lu[4 * kk + 1] = s1;
                lu[4 * kk + 2] = 0.0;
                lu[4 * kk + 3] = l;
                dd = nd - l * s1;
                s1 = ns;
            }
            else {
                const double rs = ex_rcp(sub), l = dd * rs;

                piv |= 1ull << kk;
                lu[4 * kk] = rs;
                lu[4 * kk + 1] = nd;
                lu[4 * kk + 2] = ns;
                lu[4 * kk + 3] = l;
                dd = s1 - l * nd;
                s1 = -l * ns;
            }
        }
        if (fabs(dd) < tiny)
            dd = dd < 0.0 ? -tiny : tiny;
        lu[4 * (n - 1)] = ex_rcp(dd);
        lu[4 * (n - 1) + 1] = 0.0;
        lu[4 * (n - 1) + 2] = 0.0;
        for (int kk = 0; kk < n; kk++)
            y[kk] = 1.0;
        for (int it = 0; it < 3; it++) {
            /* forward: the row interchanges and L, y[kk] final once the
               step leaves it */
            double cur = y[0];

            for (int kk = 0; kk < n - 1; kk++) {
                double a = cur, b = y[kk + 1];

                if ((piv >> kk) & 1ull) {
                    const double tmp = a;

                    a = b;
                    b = tmp;
                }
                y[kk] = a;
                cur = b - lu[4 * kk + 3] * a;
            }
            y[n - 1] = cur;
            /* backward: U, the next two solution entries in registers */
            double y1 = 0.0, y2 = 0.0, nrm = 0.0;

            for (int kk = n - 1; kk >= 0; kk--) {
                const double v = (y[kk] - lu[4 * kk + 1] * y1 - lu[4 * kk + 2] * y2) * lu[4 * kk];

                y[kk] = v;
                y2 = y1;
                y1 = v;
                nrm = fmax(nrm, fabs(v));
            }
            const double inv = 1.0 / nrm; /* may exceed the float range */

            for (int kk = 0; kk < n; kk++)
                y[kk] *= inv;
        }
    }
    __syncthreads();
    /* z = H_0 ... H_n-2 y (warp 0, rows lane and lane + 32), two
       reflectors at a time in application order (H_n-2 first): with
       a = v_0^H z, b = v_1^H z and g = v_1^H v_0 reduced over the warp at
       once, h_0 = tau_0 a, h_1 = tau_1 (b - g h_0), z -= v_0 h_0 + v_1 h_1,
       which is the one-by-one application rearranged. */
    if (t < 32) {
        double2 z[2];

#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int r = t + 32 * q;

            z[q] = make_double2(r < n ? w.y[r] : 0.0, 0.0);
        }
        for (int b0 = n - 2; b0 >= 0; b0 -= 2) {
            double2 vq[2][2], ta[2];

#pragma unroll
            for (int m = 0; m < 2; m++) {
                const int kk = b0 - m;

                ta[m] = kk >= 0 ? w.tau[kk] : make_double2(0.0, 0.0);
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int r = t + 32 * q;

                    vq[m][q] = make_double2(0.0, 0.0);
                    if (kk >= 0 && r == kk + 1)
                        vq[m][q] = make_double2(1.0, 0.0);
                    else if (kk >= 0 && r > kk + 1 && r < n)
                        vq[m][q] = w.T[tc_pidx(n, kk, r)];
                }
            }
            double rd[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};

#pragma unroll
            for (int q = 0; q < 2; q++) {
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    rd[2 * m] += vq[m][q].x * z[q].x + vq[m][q].y * z[q].y;
                    rd[2 * m + 1] += vq[m][q].x * z[q].y - vq[m][q].y * z[q].x;
                }
                rd[4] += vq[1][q].x * vq[0][q].x + vq[1][q].y * vq[0][q].y;
                rd[5] += vq[1][q].x * vq[0][q].y - vq[1][q].y * vq[0][q].x;
            }
#pragma unroll
            for (int e = 0; e < 6; e++)
                rd[e] = wsum<double>(rd[e]);
            double2 h[2];

            h[0] = make_double2(ta[0].x * rd[0] - ta[0].y * rd[1], ta[0].x * rd[1] + ta[0].y * rd[0]);
            {
                const double sx = rd[2] - (rd[4] * h[0].x - rd[5] * h[0].y);
                const double sy = rd[3] - (rd[4] * h[0].y + rd[5] * h[0].x);

                h[1] = make_double2(ta[1].x * sx - ta[1].y * sy, ta[1].x * sy + ta[1].y * sx);
            }
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    z[q].x -= vq[m][q].x * h[m].x - vq[m][q].y * h[m].y;
                    z[q].y -= vq[m][q].x * h[m].y + vq[m][q].y * h[m].x;
                }
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int r = t + 32 * q;

            if (r < n)
                w.z[r] = z[q];
        }
    }
    __syncthreads();
    return status;
}

/* Unit phasors relative to the median date (tcoh.cl:700-724) into w.zs
   (warp 0), then gamma over the pairs (tcoh.cl:728-744), every thread. */
__device__ float ex_gamma(int n, int npu, const ExWs &w)
{
    const int t = threadIdx.x;

    if (t < 32) {
        double m[2];

#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int r = t + 32 * q;

            m[q] = r < n ? hypot(w.z[r].x, w.z[r].y) : 0.0;
        }
        double mx = fmax(m[0], m[1]);

        mx = wmaxd(mx);
        int ref = n / 2;

        if (hypot(w.z[ref].x, w.z[ref].y) <= 1.0e-3 * mx) {
            int last = -1;

#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int r = t + 32 * q;

                if (r < n && m[q] == mx)
                    last = max(last, r);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1)
                last = max(last, __shfl_xor_sync(FULL, last, o));
            ref = last;
        }
        const double2 zr = w.z[ref];
        const double refm = hypot(zr.x, zr.y);
        const double refr = zr.x / refm, refi = -zr.y / refm, floor_ = 1.0e-3 * mx;

#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int r = t + 32 * q;

            if (r < n) {
                const double2 z = w.z[r];
                const double re = z.x * refr - z.y * refi, im = z.x * refi + z.y * refr;
                const double mm = hypot(re, im);

                w.zs[r] = mm > floor_ ? make_float2((float)(re / mm), (float)(im / mm))
                                      : make_float2(1.f, 0.f);
            }
        }
    }
    __syncthreads();
    float sr = 0.f, si = 0.f;

    for (int q = t; q < npu; q += EX_THREADS) {
        const int i = w.tab[q] >> 8, j = w.tab[q] & 255;

        if (i == j)
            continue;
        const float2 u = unit_phasor(w.Tf[q]);
        const float2 zi = w.zs[i], zj = w.zs[j];
        const float wr = zi.x * zj.x + zi.y * zj.y, wi = zi.x * zj.y - zi.y * zj.x;

        sr += u.x * wr - u.y * wi;
        si += u.x * wi + u.y * wr;
    }
    const double2 ssum = ex_sum2(sr, si, w.red);

    return (float)(hypot(ssum.x, ssum.y) / (0.5 * n * (n - 1)));
}

/* queue: null for every pixel of the chunk c (with its mask), else the
   queue's entries (TcExactQueue, any pixels of the strip; c unused). */
template <int NB, int BC>
__global__ void __launch_bounds__(EX_THREADS, ex_ctas(NB))
tc_link_exact_kernel(TcStrip s, TcChunk c, TcLinkConst k, ExLayout L,
                     const float2 *__restrict__ slc, const uint32_t *__restrict__ mask,
                     const int *__restrict__ count, int *queue, int qstride,
                     const unsigned short *__restrict__ upper_tab,
                     const unsigned short *__restrict__ pair_tab, double *__restrict__ scratch,
                     float *__restrict__ coh, float *__restrict__ pairs,
                     float *__restrict__ phases, unsigned char *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const ExWs w = ex_ws(smem, L);
    const int n = s.n, npu = L.npu, t = threadIdx.x, ld = L.ld;
    const long long plane = (long long)s.rows * s.cols;
    double *W = scratch + (size_t)blockIdx.x * (2 * n * ld + 64);

    for (int q = t; q < npu; q += EX_THREADS)
        w.tab[q] = upper_tab[q];
    if (t == 0) {
        const int rp = (n + 1) / 2, cg = (n + BC - 1) / BC;
        int b = 0;

        for (int ip = 0; ip < rp; ip++)
            for (int jg = (2 * ip) / BC; jg < cg; jg++)
                w.blk[b++] = (unsigned short)(ip << 8 | jg);
    }
    __syncthreads();
    const int total = queue ? queue[0] : c.npix;
    /* A chunk's pixels go to the CTAs in turn. Queued pixels vary more in
       cost (pivoted inverses, unlinked dates, several chunks' worth of
       flagged pixels of every kind): after its first, each CTA takes the
       next untaken entry from the queue's counter buf[1]. The barriers
       order thread 0's write of the index after every thread's read of the
       previous one. */
    auto next_item = [&](int it) -> int {
        if (!queue)
            return it + gridDim.x;
        __syncthreads();
        if (t == 0)
            w.ints[6] = gridDim.x + atomicAdd(queue + 1, 1);
        __syncthreads();
        return w.ints[6];
    };

    for (int it = blockIdx.x; it < total; it = next_item(it)) {
        const int *entry = queue ? queue + TC_QUEUE_HEAD + (long long)it * qstride : nullptr;
        int y, x;

        if (entry) {
            y = entry[0] / s.cols;
            x = entry[0] - y * s.cols;
        }
        else {
            tc_pixel_yx(c, it, y, x);
            if (y >= c.row0 + c.nrows || y >= s.rows || x >= s.cols)
                continue;
        }
        const long long out = (long long)y * s.cols + x;
        const int looks = count[out];

        if (looks < k.min_looks) {
            if (t == 0)
                coh[out] = NAN;
            for (int q = t; q < k.npairs; q += EX_THREADS)
                pairs[q * plane + out] = NAN;
            if (phases)
                for (int r = t; r < n; r += EX_THREADS)
                    phases[out * n + r] = NAN;
            if (status && t == 0)
                status[out] = 0;
            continue;
        }
        const int ncand =
            entry ? ex_candidates(s, (const uint32_t *)entry + 1, 1, w)
                  : ex_candidates(s, mask + it, c.npix, w);

        ex_gram<NB, BC>(s, slc, y, x, ncand, w, L);
        ex_coherence(n, npu, k, looks, w);
        for (int q = t; q < k.npairs; q += EX_THREADS) {
            const int i = pair_tab[q] >> 8, j = pair_tab[q] & 255;

            pairs[q * plane + out] = (float)w.G[tc_pidx(n, i, j)];
        }
        if (k.bias && !ex_linked(n, w)) {
            if (t == 0)
                coh[out] = NAN;
            if (phases)
                for (int r = t; r < n; r += EX_THREADS)
                    phases[out * n + r] = NAN;
            if (status && t == 0)
                status[out] = TC_STATUS_UNLINKED;
            __syncthreads();
            continue;
        }
        unsigned st = TC_STATUS_FP64;

        if (k.emi) {
            st |= ex_inverse<(NB > 1 ? 2 : 4)>(n, npu, ld, w, W);
            /* M = |T|^-1 o T in place of T; T in float in place of |T|^-1 */
            for (int q = t; q < npu; q += EX_THREADS) {
                const double g = w.G[q];
                const double2 v = w.T[q];

                w.T[q] = make_double2(g * v.x, g * v.y);
                w.Tf[q] = make_float2((float)v.x, (float)v.y);
            }
        }
        else
            /* EVD: T itself; T in float in place of |T| */
            for (int q = t; q < npu; q += EX_THREADS) {
                const double2 v = w.T[q];

                w.Tf[q] = make_float2((float)v.x, (float)v.y);
            }
        __syncthreads();
        ex_householder<(NB > 1)>(n, npu, w);
        st |= ex_eigvec(n, k.emi ? 0 : n - 1, w);
        const float gamma = ex_gamma(n, npu, w);

        if (t == 0)
            coh[out] = gamma;
        if (phases)
            for (int r = t; r < n; r += EX_THREADS) {
                const float2 u = w.zs[r];

                phases[out * n + r] = atan2f(u.y, u.x);
            }
        if (status && t == 0)
            status[out] = (unsigned char)st;
        __syncthreads();
    }
}

} // namespace

static size_t exact_scratch_bytes(int n, int sms)
{
    /* per CTA: |T| and the Jacobi eigenvectors in full storage, and the
       eigenvalues, for the pseudo-inverse tier */
    return (size_t)sms * ex_ctas(ex_nb_for(n)) * (2 * n * (n | 1) + 64) * sizeof(double);
}

template <int NB, int BC>
static cudaError_t launch_exact_nb(const TcStrip &s, const TcChunk &c, const TcLinkConst &k,
                                   const float *slc, const uint32_t *mask, const int *count,
                                   const TcExactQueue *q, const unsigned short *upper_tab,
                                   const unsigned short *pair_tab, double *scratch, float *coh,
                                   float *pairs, float *phases, unsigned char *status, int sms,
                                   cudaStream_t st)
{
    const ExLayout L = ex_layout(s.n, s.area);
    const int ctas = sms * ex_ctas(NB);
    int blocks = ctas;

    if (!q && c.npix < ctas)
        blocks = c.npix;
    if (q && q->pending < ctas)
        blocks = (int)q->pending;
    const cudaError_t e = tc_allow_smem(tc_link_exact_kernel<NB, BC>);

    if (e != cudaSuccess)
        return e;
    tc_link_exact_kernel<NB, BC><<<blocks, EX_THREADS, L.bytes, st>>>(
        s, c, k, L, (const float2 *)slc, mask, count, q ? q->buf : nullptr, q ? q->stride : 0,
        upper_tab, pair_tab, scratch, coh, pairs, phases, status);
    return cudaGetLastError();
}

static cudaError_t launch_exact(const TcStrip &s, const TcChunk &c, const TcLinkConst &k,
                                const float *slc, const uint32_t *mask, const int *count,
                                const TcExactQueue *q, const unsigned short *upper_tab,
                                const unsigned short *pair_tab, double *scratch, float *coh,
                                float *pairs, float *phases, unsigned char *status, int sms,
                                cudaStream_t st)
{
    if (ex_nb_for(s.n) == 1 && ex_bc_for(s.n) == 2)
        return launch_exact_nb<1, 2>(s, c, k, slc, mask, count, q, upper_tab, pair_tab, scratch,
                                     coh, pairs, phases, status, sms, st);
    if (ex_nb_for(s.n) == 1)
        return launch_exact_nb<1, 4>(s, c, k, slc, mask, count, q, upper_tab, pair_tab, scratch,
                                     coh, pairs, phases, status, sms, st);
    return launch_exact_nb<EX_NB, 4>(s, c, k, slc, mask, count, q, upper_tab, pair_tab, scratch,
                                     coh, pairs, phases, status, sms, st);
}

bool tc_link_needs_gram(int n, int emi)
{
    return n <= 32 || !emi;
}

size_t tc_link_scratch_bytes(int n, int sms)
{
    /* the 32-date kernel and the exact tier run one after the other */
    const size_t a = tc_link_half_scratch_bytes(n, sms), b = exact_scratch_bytes(n, sms);

    return a > b ? a : b;
}

bool tc_link_queues(int n, const TcLinkConst &k)
{
    /* the float kernels hand pixels to the exact tier with EMI and with
       the bias correction; EMI above 32 dates is all exact */
    return (k.emi || k.bias) && !(n > 32 && k.emi);
}

size_t tc_exact_queue_bytes(int mask_words, long long capacity)
{
    return sizeof(int) * (TC_QUEUE_HEAD + (size_t)capacity * (1 + mask_words));
}

cudaError_t tc_flush_exact(const TcStrip &s, const TcLinkConst &k, TcExactQueue *q,
                           const float *slc, const int *count, const unsigned short *upper_tab,
                           const unsigned short *pair_tab, double *scratch, float *coh,
                           float *pairs, float *phases, unsigned char *status, int sms,
                           cudaStream_t st)
{
    cudaError_t e = cudaSuccess;

    if (q->pending > 0) {
        TcChunk none = {};

        if ((e = launch_exact(s, none, k, slc, nullptr, count, q, upper_tab, pair_tab, scratch,
                              coh, pairs, phases, status, sms, st)) == cudaSuccess)
            e = cudaMemsetAsync(q->buf, 0, sizeof(int) * TC_QUEUE_HEAD, st);
    }
    q->pending = 0;
    return e;
}

cudaError_t tc_launch_link(const TcStrip &s, const TcChunk &c, const TcLinkConst &k,
                           const float2 *gram, const float *slc, const uint32_t *mask,
                           const int *count, TcExactQueue *q,
                           const unsigned short *upper_tab, const unsigned short *pair_tab,
                           double *scratch, float *coh, float *pairs, float *phases,
                           unsigned char *status, int sms, cudaStream_t st)
{
    cudaError_t e;
    const bool queued = tc_link_queues(s.n, k);

    if (queued && (!q || !q->buf || q->stride != 1 + s.mask_words ||
                   q->pending + c.npix > q->capacity))
        return cudaErrorInvalidValue;
    int *qb = queued ? q->buf : nullptr;
    const int qs = queued ? q->stride : 0;

    if (s.n > 32 && k.emi)
        return launch_exact(s, c, k, slc, mask, count, nullptr, upper_tab, pair_tab, scratch, coh,
                            pairs, phases, status, sms, st);
    if (s.n <= 32)
        e = tc_launch_link_half(s, c, k, gram, mask, count, upper_tab, pair_tab, scratch, coh,
                                pairs, phases, status, qb, qs, sms, st);
    else
        e = tc_launch_link_wide(s, c, k, gram, mask, count, upper_tab, pair_tab, coh, pairs,
                                phases, status, qb, qs, sms, st);
    if (e == cudaSuccess && queued)
        q->pending += c.npix;
    return e;
}
