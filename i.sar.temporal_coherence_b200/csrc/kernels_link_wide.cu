/* Phase linking (EVD) and temporal coherence for stacks of 33 to 64 dates: two
 * warps per pixel, one matrix row per lane in registers.
 *
 * The stages and their numerics are those of kernels_link_half.cu (see there
 * and kernels_link.cu for the reference lines). T stays in shared memory in
 * full, its upper triangle for the pair coherences and the goodness of fit, its
 * lower one for the Householder vectors; the matrix under reduction is in
 * registers (64 columns of a row: 128 of them), where a step's matrix-vector
 * product and rank-2 update cost twelve fused multiply-adds and three shared
 * loads per column. Both warps of a pixel meet at a named barrier twice a step.
 * Six pixels per SM (twelve warps of 168 registers; five above 62 dates, by
 * shared memory): against four with 255 registers, 34.4 and 36.3 ms on 96 x 2048
 * pixels at 60 dates, a Householder step 0.55k cycles per pixel instead of 0.78k.
 *
 * Bound by latency: a step's reductions, barriers and shared-memory round trips
 * (short scoreboard) with three warps per scheduler, half of the issue slots in
 * use. With the matrix itself in shared memory (a warp per pixel, twelve
 * pixels per SM) each multiply-add came with its own loads and stores of the
 * matrix and a step's serial work was done by one lane: 55.8 ms on the same
 * pixels, 6.29 against 4.25 ms on 61 x 517 at 45 dates.
 */
#include "link_float.cuh"

#include <math.h>

#define FULL 0xffffffffu

namespace {

constexpr int WD_PIXELS = 6;  /* pixels per CTA and SM, at most */
constexpr int WD_PAD = 80;    /* v and w beyond the last row: whole blocks of 8 columns */
constexpr int WD_BATCH = 6;   /* entries of T per lane and turn of load_T */

struct WideLayout {
    int n, ld;
    int off_vw, off_lu, off_tau, off_d, off_e, off_e2, off_nrm, off_z, off_red;
    int per_pixel;
};

/* A pixel's two warps. */
struct Duo {
    int lane, warp, row, bar;
};

__device__ __forceinline__ void meet(const Duo &g)
{
    asm volatile("bar.sync %0, 64;" ::"r"(g.bar) : "memory");
}

struct Ws {
    float2 *T;                     /* n x ld */
    float2 *vw;                    /* Householder v and w of even steps, of odd steps */
    float2 *c;                     /* the pivot column */
    float4 *lu;                    /* 64 */
    float2 *tau, *z;               /* z: the eigenvector, then the phasors */
    float *d, *e, *e2, *nrm, *red; /* red: 2 x 48 floats */
};

__device__ __forceinline__ Ws workspace(unsigned char *base, const WideLayout &L)
{
    Ws w;

    w.T = (float2 *)base;
    w.vw = (float2 *)(base + L.off_vw);
    w.c = w.vw + 4 * WD_PAD;
    w.lu = (float4 *)(base + L.off_lu);
    w.tau = (float2 *)(base + L.off_tau);
    w.d = (float *)(base + L.off_d);
    w.e = (float *)(base + L.off_e);
    w.e2 = (float *)(base + L.off_e2);
    w.nrm = (float *)(base + L.off_nrm);
    w.z = (float2 *)(base + L.off_z);
    w.red = (float *)(base + L.off_red);
    return w;
}

WideLayout wide_layout(int n)
{
    WideLayout L;
    int off = 0;
    auto take = [&](int bytes) {
        const int o = off;

        off += (bytes + 15) & ~15;
        return o;
    };

    L.n = n;
    L.ld = n | 1;
    take(8 * n * L.ld);
    L.off_vw = take(8 * 5 * WD_PAD);
    L.off_lu = take(16 * 64);
    L.off_tau = take(8 * 64);
    L.off_d = take(4 * 64);
    L.off_e = take(4 * 64);
    L.off_e2 = take(4 * 64);
    L.off_nrm = take(4 * 64);
    L.off_z = take(8 * 64);
    L.off_red = take(4 * 96);
    L.per_pixel = off;
    return L;
}

__device__ __forceinline__ float wsum(float v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1)
        v += __shfl_xor_sync(FULL, v, o);
    return v;
}

/* ------------------------------------------------------------------ */
/* Coherence matrix.                                                   */
/* ------------------------------------------------------------------ */

/* T of pixel p from its packed Gram sums (tcoh.cl:611-636), both triangles; the
   lanes take the packed entries in turn, six at a time with the next twelve in
   flight. Returns whether a bias decision lies within TC_BIAS_BAND of its
   threshold. */
__device__ bool load_T(int n, int ld, const TcLinkConst &k, int looks,
                       const float2 *__restrict__ sums, const unsigned short *upper_tab,
                       const Ws &w, const Duo &g)
{
    const int npu = tc_npu(n), i0 = g.row;
    const float fl = (float)looks;
    const bool debias = k.bias && looks > 1;
    const float ilm1 = debias ? __frcp_rn(__fsub_rn(fl, 1.0f)) : 0.f;
    float2 a[WD_BATCH], b[WD_BATCH], c[WD_BATCH];
    bool near = false;
    auto fetch = [&](float2 (&v)[WD_BATCH], int t0) {
#pragma unroll
        for (int u = 0; u < WD_BATCH; u++) {
            const int q = i0 + 64 * (t0 + u);

            v[u] = q < npu ? sums[q] : make_float2(0.f, 0.f);
        }
    };

    const float dii = i0 < n ? sums[tc_pidx(n, i0, i0)].x : 0.f;

    fetch(a, 0);
    fetch(b, WD_BATCH);
    w.nrm[i0] = __fsqrt_rn(dii);
    /* norms whose products leave the middle of the float range take the
       general form */
    const bool odd = i0 < n && !(dii > 1.0e-20f && dii < 1.0e20f);
    const bool plain = !__any_sync(FULL, odd);

    if (g.lane == 0)
        w.red[g.warp] = plain ? 1.f : 0.f;
    meet(g);
    const bool all_plain = w.red[0] + w.red[1] == 2.f;

#pragma unroll 1
    for (int t0 = 0; 64 * t0 < npu; t0 += WD_BATCH) {
        int ij[WD_BATCH];
        float2 t[WD_BATCH];

        fetch(c, t0 + 2 * WD_BATCH);
#pragma unroll
        for (int u = 0; u < WD_BATCH; u++)
            ij[u] = upper_tab[min(i0 + 64 * (t0 + u), npu - 1)];
        if (all_plain) {
            float ni[WD_BATCH], nj[WD_BATCH];

#pragma unroll
            for (int u = 0; u < WD_BATCH; u++) {
                ni[u] = w.nrm[ij[u] >> 8];
                nj[u] = w.nrm[ij[u] & 255];
            }
#pragma unroll
            for (int u = 0; u < WD_BATCH; u++) {
                bool edge = false;

                t[u] = t_entry(a[u], ni[u], nj[u], fl, ilm1, debias, edge);
                near |= edge & ((ij[u] >> 8) != (ij[u] & 255)) & (i0 + 64 * (t0 + u) < npu);
            }
        }
        else {
#pragma unroll 1
            for (int u = 0; u < WD_BATCH; u++) {
                bool edge = false;
                float2 au = a[0];
                int iju = ij[0];

#pragma unroll
                for (int x = 1; x < WD_BATCH; x++)
                    if (x == u) {
                        au = a[x];
                        iju = ij[x];
                    }
                const float2 tu = t_entry_any(au, w.nrm[iju >> 8], w.nrm[iju & 255], fl, debias,
                                              edge);

                near |= edge & ((iju >> 8) != (iju & 255)) & (i0 + 64 * (t0 + u) < npu);
#pragma unroll
                for (int x = 0; x < WD_BATCH; x++)
                    if (x == u)
                        t[x] = tu;
            }
        }
#pragma unroll
        for (int u = 0; u < WD_BATCH; u++) {
            const int i = ij[u] >> 8, j = ij[u] & 255;

            if (i0 + 64 * (t0 + u) < npu) {
                w.T[i * ld + j] = i == j ? make_float2(1.f, 0.f) : t[u];
                if (i != j)
                    w.T[j * ld + i] = make_float2(t[u].x, -t[u].y);
            }
        }
#pragma unroll
        for (int u = 0; u < WD_BATCH; u++) {
            a[u] = b[u];
            b[u] = c[u];
        }
    }
    near = __any_sync(FULL, near);
    if (g.lane == 0)
        w.red[48 + g.warp] = near ? 1.f : 0.f;
    meet(g);
    return w.red[48] + w.red[49] > 0.f;
}

/* Whether the non-zero coherences link all dates: the dates reached from date
   0, expanded one at a time (votes over the entries of its row; each warp does
   it for itself). */
__device__ bool linked(int n, int ld, const float2 *T, const Duo &g)
{
    const unsigned long long all = n == 64 ? ~0ull : (1ull << n) - 1ull;
    unsigned long long reached = 1ull, todo = 1ull;

    while (todo && reached != all) {
        const int f = __ffsll((long long)todo) - 1;
        const int j = g.lane + 32;
        const float2 a = T[f * ld + g.lane];
        const float2 b = j < n ? T[f * ld + j] : make_float2(0.f, 0.f);
        const unsigned lo = __ballot_sync(FULL, a.x != 0.f || a.y != 0.f);
        const unsigned hi = __ballot_sync(FULL, b.x != 0.f || b.y != 0.f);
        const unsigned long long nw = (((unsigned long long)hi << 32) | lo) & ~reached;

        reached |= nw;
        todo = (todo & (todo - 1ull)) | nw;
    }
    return reached == all;
}

/* ------------------------------------------------------------------ */
/* Householder reduction.                                              */
/* ------------------------------------------------------------------ */

struct Head {
    float beta, dk;
    float2 tau, scale;
};

/* As kernels_link_half.cu's reflector. */
__device__ __forceinline__ void reflector(Head &h, float2 alpha, float xn2)
{
    const bool zero = xn2 == 0.f && alpha.y == 0.f;
    const float s2 = __fadd_rn(fmaf(alpha.x, alpha.x, __fmul_rn(alpha.y, alpha.y)), xn2);
    float beta = -copysignf(sqrt_rn(s2), alpha.x), ib = rcp_rn(beta);
    float dr = alpha.x - beta, di = alpha.y;
    float iden = rcp_rn(fmaf(di, di, __fmul_rn(dr, dr)));

    if (!zero && !(s2 > 1.0e-24f && s2 < 1.0e24f)) {
        /* columns near the ends of the float range: rarely, if ever */
        beta = -copysignf(sqrtf(s2), alpha.x);
        ib = __frcp_rn(beta);
        dr = alpha.x - beta;
        iden = __frcp_rn(fmaf(di, di, __fmul_rn(dr, dr)));
    }
    h.beta = zero ? alpha.x : beta;
    h.tau = zero ? make_float2(0.f, 0.f)
                 : make_float2(__fmul_rn(beta - alpha.x, ib), __fmul_rn(-alpha.y, ib));
    h.scale = make_float2(__fmul_rn(dr, iden), __fmul_rn(-di, iden));
    if (h.tau.x == 0.f && h.tau.y == 0.f)
        h.scale = make_float2(1.f, 0.f);
}

/* Reduction of the pixel's matrix to real tridiagonal form, row g.row in r; at
   step k the pivot column is r[0]. The two warps meet twice a step. The column
   c goes to the other lanes as it is, with the sums that its reflector comes
   from, and A v = scale * (A c) + column k + 1 (v = scale * c below row k + 1, 1
   in it), so that the square root and the reciprocals run beside the
   matrix-vector product. With w = tau A v (without the multiple of v that makes
   the update Hermitian) and s = -Re(tau (w^H v)) the update is
       A -= v w^H + (w + s v) v^H,
   so that v and w go out together with the partial sums of w^H v. They stay
   readable through the next step (two buffers): the update of the far columns
   runs across the next column's meeting. A warp whose rows are all reduced
   skips the arithmetic. */
__device__ void householder(float2 (&r)[64], int n, int ld, const Ws &w, const Duo &g)
{
    const int i = g.row;
    float4 mine = make_float4(0.f, 0.f, 0.f, 0.f);
    float dk = 0.f;

    for (int q = 64 + g.lane; q < WD_PAD; q += 32) {
        w.vw[2 * g.warp * WD_PAD + q] = make_float2(0.f, 0.f);
        w.vw[(2 * g.warp + 1) * WD_PAD + q] = make_float2(0.f, 0.f);
        w.c[q] = make_float2(0.f, 0.f);
    }
    /* red: [0, 1] sub-diagonal, [2] diagonal, [4 + warp] norm below; [8 + 2
       warp, 9 + 2 warp] w^H v */
    auto publish = [&](int k) {
        w.c[i] = r[0];
        if (i == k + 1)
            *(float2 *)w.red = r[0];
        if (i == k)
            w.red[2] = r[0].x;
    };
    auto below = [&](int k) {
        return i >= k + 2 && i < n ? fmaf(r[0].x, r[0].x, __fmul_rn(r[0].y, r[0].y)) : 0.f;
    };

    publish(0);
    {
        const float x = wsum(below(0));

        if (g.lane == 0)
            w.red[4 + g.warp] = x;
    }
    meet(g);

#pragma unroll 1
    for (int k = 0; k < n - 1; k++) {
        const int len = n - 1 - k;
        const bool live = 32 * g.warp + 31 > k;
        const float2 *ck = w.c + k;
        float2 *vk = w.vw + 2 * WD_PAD * (k & 1) + k, *wk = vk + WD_PAD;
        Head h;

        {
            const float4 a = *(const float4 *)w.red;
            const float2 x = *(const float2 *)(w.red + 4);

            h.dk = a.z;
            reflector(h, make_float2(a.x, a.y), x.x + x.y);
        }
        if (i == k)
            mine = make_float4(h.dk, h.beta, h.tau.x, h.tau.y);
        float2 pa = make_float2(0.f, 0.f), pb = pa, pc = pa, pd = pa;

        if (live) {
#pragma unroll
            for (int jb = 2; jb < 64; jb += 8) {
                if (jb > len)
                    break;
                float2 x[8];

#pragma unroll
                for (int u = 0; u < 8; u++)
                    x[u] = ck[jb + u];
#pragma unroll
                for (int u = 0; u < 8 && jb + u < 64; u += 2) {
                    const int jj = jb + u;

                    pa.x = fmaf(r[jj].x, x[u].x, pa.x);
                    pa.y = fmaf(r[jj].x, x[u].y, pa.y);
                    pb.x = fmaf(-r[jj].y, x[u].y, pb.x);
                    pb.y = fmaf(r[jj].y, x[u].x, pb.y);
                    if (jj + 1 < 64) {
                        pc.x = fmaf(r[jj + 1].x, x[u + 1].x, pc.x);
                        pc.y = fmaf(r[jj + 1].x, x[u + 1].y, pc.y);
                        pd.x = fmaf(-r[jj + 1].y, x[u + 1].y, pd.x);
                        pd.y = fmaf(r[jj + 1].y, x[u + 1].x, pd.y);
                    }
                }
            }
        }
        float2 v = cscale(r[0], h.scale);

        v.x = i > k + 1 && i < n ? v.x : i == k + 1 ? 1.f : 0.f;
        v.y = i > k + 1 && i < n ? v.y : 0.f;
        float2 p = cscale(make_float2((pa.x + pb.x) + (pc.x + pd.x), (pa.y + pb.y) + (pc.y + pd.y)),
                          h.scale);

        p.x += r[1].x;
        p.y += r[1].y;
        float2 wi = i > k ? cscale(p, h.tau) : make_float2(0.f, 0.f);

        vk[i - k] = v;
        wk[i - k] = wi;
        {
            float2 s = make_float2(fmaf(wi.x, v.x, wi.y * v.y), fmaf(wi.x, v.y, -wi.y * v.x));

#pragma unroll
            for (int o = 16; o; o >>= 1) {
                const float x = __shfl_xor_sync(FULL, s.x, o), y = __shfl_xor_sync(FULL, s.y, o);

                s.x += x;
                s.y += y;
            }
            if (g.lane == 0)
                *(float2 *)(w.red + 8 + 2 * g.warp) = s;
        }
        meet(g);
        {
            const float4 s = *(const float4 *)(w.red + 8);
            const float sc = -fmaf(h.tau.x, s.x + s.z, -h.tau.y * (s.y + s.w));

            wi.x = fmaf(sc, v.x, wi.x);
            wi.y = fmaf(sc, v.y, wi.y);
        }
        const float2 nv = make_float2(-v.x, -v.y), nw = make_float2(-wi.x, -wi.y);

        /* Column k + 1 first, the next pivot column. */
        {
            const float2 x = vk[1], y = wk[1];

            r[0] = r2(r[1], nv, nw, make_float4(x.x, x.y, y.x, y.y));
        }
        publish(k + 1);
        float x = below(k + 1);

        dk = r[0].x;
        if (i > k && i < n)
            w.T[i * ld + k] = v;
#pragma unroll
        for (int jb = 2; jb < 64; jb += 8) {
            if (live && jb <= len) {
                float2 x[8], y[8];

                /* the loads of a block, then its updates term by term */
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    x[u] = vk[jb + u];
                    y[u] = wk[jb + u];
                }
#pragma unroll
                for (int u = 0; u < 8 && jb + u < 64; u++) {
                    r[jb + u - 1].x = fmaf(nv.x, y[u].x, r[jb + u].x);
                    r[jb + u - 1].y = fmaf(nv.y, y[u].x, r[jb + u].y);
                }
#pragma unroll
                for (int u = 0; u < 8 && jb + u < 64; u++) {
                    r[jb + u - 1].x = fmaf(nv.y, y[u].y, r[jb + u - 1].x);
                    r[jb + u - 1].y = fmaf(-nv.x, y[u].y, r[jb + u - 1].y);
                }
#pragma unroll
                for (int u = 0; u < 8 && jb + u < 64; u++) {
                    r[jb + u - 1].x = fmaf(nw.x, x[u].x, r[jb + u - 1].x);
                    r[jb + u - 1].y = fmaf(nw.y, x[u].x, r[jb + u - 1].y);
                }
#pragma unroll
                for (int u = 0; u < 8 && jb + u < 64; u++) {
                    r[jb + u - 1].x = fmaf(nw.y, x[u].y, r[jb + u - 1].x);
                    r[jb + u - 1].y = fmaf(-nw.x, x[u].y, r[jb + u - 1].y);
                }
            }
            if (jb == 2)
                x += __shfl_xor_sync(FULL, x, 16);
            else if (jb == 10)
                x += __shfl_xor_sync(FULL, x, 8);
            else if (jb == 18) {
                x += __shfl_xor_sync(FULL, x, 4);
                x += __shfl_xor_sync(FULL, x, 2);
            }
            else if (jb == 26) {
                x += __shfl_xor_sync(FULL, x, 1);
                if (g.lane == 0)
                    w.red[4 + g.warp] = x;
                meet(g);
            }
        }
    }
    if (i < n - 1) {
        w.d[i] = mine.x;
        w.e[i] = mine.y;
        w.tau[i] = make_float2(mine.z, mine.w);
    }
    if (i == n - 1)
        w.d[i] = dk;
    meet(g);
}

/* ------------------------------------------------------------------ */
/* Eigenvector.                                                        */
/* ------------------------------------------------------------------ */

/* Eigenvalues of the tridiagonal below x (kernels_link_half.cu's sturm16). */
__device__ __forceinline__ int sturm(const float *d, const float *e2, int n, float x, float pivmin)
{
    const float rsmall = rcp_approx(-pivmin);
    float q = d[0] - x;
    int c = q < 0.f;

#pragma unroll 4
    for (int i = 1; i < n; i++) {
        const float r = rcp_approx(q);

        q = fmaf(-e2[i - 1], fabsf(q) < pivmin ? rsmall : r, d[i] - x);
        c += q < 0.f;
    }
    return c;
}

/* Largest eigenvalue of the tridiagonal (w.d, w.e), by 65-way multisection of
   its Gershgorin interval down to 1e-7 of the spectrum's scale. */
__device__ float largest_eigenvalue(int n, const Ws &w, const Duo &g, float &norm,
                                    unsigned &status)
{
    const int i = g.row;
    float lo = INFINITY, hi = -INFINITY;

    if (i < n) {
        const float rad = (i > 0 ? fabsf(w.e[i - 1]) : 0.f) + (i < n - 1 ? fabsf(w.e[i]) : 0.f);

        lo = w.d[i] - rad;
        hi = w.d[i] + rad;
        if (i < n - 1)
            w.e2[i] = w.e[i] * w.e[i];
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(FULL, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, o));
    }
    if (g.lane == 0)
        *(float2 *)(w.red + 2 * g.warp) = make_float2(lo, hi);
    meet(g);
    {
        const float4 b = *(const float4 *)w.red;

        lo = fminf(b.x, b.z);
        hi = fmaxf(b.y, b.w);
    }
    norm = fmaxf(fabsf(lo), fabsf(hi));
    lo -= 1.0e-6f * norm + 1.0e-30f;
    hi += 1.0e-6f * norm + 1.0e-30f;
    const float pivmin = 1.0e-30f + 1.0e-14f * norm;
    int round = 0;

    for (; round < 20 && hi - lo > 1.0e-7f * norm; round++) {
        const float step = (hi - lo) * (1.0f / 65.0f);
        const float xq = fmaf(step, (float)(i + 1), lo);
        const unsigned gt = __ballot_sync(FULL, sturm(w.d, w.e2, n, xq, pivmin) > n - 1);
        unsigned *box = (unsigned *)w.red + 8 + 2 * (round & 1);

        if (g.lane == 0)
            box[g.warp] = gt;
        meet(g);
        const unsigned long long above = ((unsigned long long)box[1] << 32) | box[0];
        const int f = above ? __ffsll((long long)above) - 1 : 64;
        const float nlo = f > 0 ? fmaxf(fmaf(step, (float)f, lo), lo) : lo;
        const float nhi = f < 64 ? fminf(fmaf(step, (float)(f + 1), lo), hi) : hi;

        if (!(nlo > lo || nhi < hi))
            break;
        lo = nlo;
        hi = nhi;
    }
    if (round == 20)
        status |= TC_STATUS_ITER_CAP;
    return 0.5f * (lo + hi);
}

/* Partially pivoted LU of tri - lambda I into w.lu (one warp, all lanes alike);
   rows from n on are those of the identity. Returns the pivot bits. */
__device__ unsigned long long tri_lu(int n, float lambda, float tiny, const Ws &w, const Duo &g)
{
    unsigned long long piv = 0ull;
    float dd = w.d[0] - lambda, s1 = w.e[0];
    float nd = w.d[1] - lambda, ns = n > 2 ? w.e[1] : 0.f, sub = w.e[0];

#pragma unroll 1
    for (int k = 0; k < n - 1; k++) {
        /* the next row's entries and reciprocal while this one's chain runs */
        const int k2 = min(k + 2, n - 1);
        const float nd2 = w.d[k2] - lambda, ns2 = k + 2 < n - 1 ? w.e[k2] : 0.f;
        const float rs = rcp_approx(sub);
        const bool swap = !(fabsf(dd) >= fabsf(sub));
        const float dc = fabsf(dd) < tiny ? (dd < 0.f ? -tiny : tiny) : dd;
        const float rd = swap ? rs : rcp_approx(dc);
        const float l = (swap ? dd : sub) * rd;
        const float m = swap ? nd : s1, o = swap ? s1 : nd;

        if (g.lane == 0)
            w.lu[k] = make_float4(rd, m, swap ? ns : 0.f, l);
        if (swap)
            piv |= 1ull << k;
        dd = fmaf(-l, m, o);
        s1 = swap ? -l * ns : ns;
        sub = ns;
        nd = nd2;
        ns = ns2;
    }
    const float dc = fabsf(dd) < tiny ? (dd < 0.f ? -tiny : tiny) : dd;

    if (g.lane == 0)
        w.lu[n - 1] = make_float4(rcp_approx(dc), 0.f, 0.f, 0.f);
    for (int q = n + g.lane; q < 64; q += 32)
        w.lu[q] = make_float4(1.f, 0.f, 0.f, 0.f);
    __syncwarp();
    return piv;
}

/* The tridiagonal eigenvector of lambda by three solves from a vector of ones
   (tcoh.cl:342-410), into w.z (real parts); by one warp, all lanes alike, the
   iterate in registers. */
__device__ __noinline__ void inverse_iteration(int n, float lambda, float norm, Ws w, Duo g)
{
    const float tiny = 1.0e-6f * fmaxf(norm, 1.0e-30f);
    const unsigned long long piv = tri_lu(n, lambda, tiny, w, g);
    float y[64];
    int at = 0; /* stays 0: the factors of a chunk of eight rows are not loaded
                   before the chunk ahead of it has begun (all 64 rows' factors
                   do not fit the registers beside y) */

#pragma unroll
    for (int k = 0; k < 64; k++)
        y[k] = 1.f;
#pragma unroll 1
    for (int it = 0; it < 3; it++) {
#pragma unroll
        for (int k = 0; k < 63; k++) {
            if (k % 8 == 0 && k >= 8)
                asm volatile("" : "+r"(at), "+f"(y[k - 8]));
            const bool swap = ((piv >> k) & 1ull) != 0ull;
            const float a = swap ? y[k + 1] : y[k], b = swap ? y[k] : y[k + 1];

            y[k] = a;
            y[k + 1] = fmaf(-w.lu[at + k].w, a, b);
        }
        float nrm = 0.f, odd = 0.f;

#pragma unroll
        for (int k = 63; k >= 0; k--) {
            if (k % 8 == 7 && k < 56)
                asm volatile("" : "+r"(at), "+f"(y[k + 8]));
            const float4 u = w.lu[at + k];
            float v = y[k];

            if (k < 63)
                v = fmaf(-u.y, y[k + 1], v);
            if (k < 62)
                v = fmaf(-u.z, y[k + 2], v);
            y[k] = v * u.x;
            if (k & 1)
                odd = fmaxf(odd, k < n ? fabsf(y[k]) : 0.f);
            else
                nrm = fmaxf(nrm, k < n ? fabsf(y[k]) : 0.f);
        }
        const float inv = __frcp_rn(fmaxf(nrm, odd));

#pragma unroll
        for (int k = 0; k < 64; k++)
            y[k] *= inv;
    }
    if (g.lane == 0)
#pragma unroll
        for (int k = 0; k < 64; k++)
            w.z[k] = make_float2(k < n ? y[k] : 0.f, 0.f);
}

/* x <- Q x, Q = H_0 H_1 .. H_{n-2}, on the lanes' rows: four reflectors at a
   time with their products with x and with one another summed at once
   (kernels_link_half.cu's apply_q). */
__device__ void apply_q(int n, int ld, const Ws &w, const Duo &g, float2 &x)
{
    const int i = g.row, gl = g.lane & 15;

#pragma unroll 1
    for (int b = 0; b < n - 1; b += 4) {
        float2 v[4], ta[4];
        float r[20];
        int p = 0;

#pragma unroll
        for (int m = 0; m < 4; m++) {
            const int k = n - 2 - (b + m), kc = max(k, 0);
            const bool in = k >= 0 && i > k && i < n;
            const float2 vi = w.T[min(i, n - 1) * ld + kc], t = w.tau[kc];

            v[m] = make_float2(in ? vi.x : 0.f, in ? vi.y : 0.f);
            ta[m] = make_float2(k >= 0 ? t.x : 0.f, k >= 0 ? t.y : 0.f);
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
            r[2 * m] = v[m].x * x.x + v[m].y * x.y;
            r[2 * m + 1] = v[m].x * x.y - v[m].y * x.x;
#pragma unroll
            for (int j = 0; j < m; j++, p++) {
                r[8 + 2 * p] = v[m].x * v[j].x + v[m].y * v[j].y;
                r[9 + 2 * p] = v[m].x * v[j].y - v[m].y * v[j].x;
            }
        }
#pragma unroll
        for (int o = 8; o; o >>= 1) {
            const bool up = (gl & o) != 0;

#pragma unroll
            for (int e = 0; e < o; e++) {
                const float give = up ? r[e] : r[e + o], keep = up ? r[e + o] : r[e];

                r[e] = keep + __shfl_xor_sync(FULL, give, o);
            }
            if (o >= 4)
#pragma unroll
                for (int e = 16; e < 16 + o / 4; e++) {
                    const float give = up ? r[e] : r[e + o / 4], keep = up ? r[e + o / 4] : r[e];

                    r[e] = keep + __shfl_xor_sync(FULL, give, o);
                }
            else
                r[16] += __shfl_xor_sync(FULL, r[16], o);
        }
        r[0] += __shfl_xor_sync(FULL, r[0], 16);
        r[16] += __shfl_xor_sync(FULL, r[16], 16);
        /* per warp 20 sums; alternate blocks alternate halves of red */
        float *red = w.red + 48 * ((b >> 2) & 1);

        if (g.lane < 16)
            red[20 * g.warp + gl] = r[0];
        if (g.lane < 16 && (gl & 3) == 0)
            red[20 * g.warp + 16 + (gl >> 2)] = r[16];
        meet(g);
#pragma unroll
        for (int e = 0; e < 20; e += 4) {
            const float4 s = *(const float4 *)(red + e), t = *(const float4 *)(red + 20 + e);

            r[e] = s.x + t.x;
            r[e + 1] = s.y + t.y;
            r[e + 2] = s.z + t.z;
            r[e + 3] = s.w + t.w;
        }
        float2 h[4];

        p = 0;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            float sx = r[2 * m], sy = r[2 * m + 1];

#pragma unroll
            for (int j = 0; j < m; j++, p++) {
                const float gx = r[8 + 2 * p], gy = r[9 + 2 * p];

                sx -= gx * h[j].x - gy * h[j].y;
                sy -= gx * h[j].y + gy * h[j].x;
            }
            h[m] = make_float2(ta[m].x * sx - ta[m].y * sy, ta[m].x * sy + ta[m].y * sx);
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
            x.x -= v[m].x * h[m].x - v[m].y * h[m].y;
            x.y -= v[m].x * h[m].y + v[m].y * h[m].x;
        }
    }
}

/* Unit phasors relative to the median date (tcoh.cl:700-724) into w.z, then the
   goodness of fit (tcoh.cl:728-744), on every lane. */
__device__ float goodness(int n, int ld, const Ws &w, const Duo &g, float2 z,
                          const unsigned short *upper_tab)
{
    const int i = g.row;
    const float m = i < n ? hypotf(z.x, z.y) : 0.f;
    float mx = m;

#pragma unroll
    for (int o = 16; o; o >>= 1)
        mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, o));
    w.vw[i] = z;
    if (g.lane == 0)
        w.red[40 + g.warp] = mx; /* the other warp may still read apply_q's sums */
    meet(g);
    mx = fmaxf(w.red[40], w.red[41]);
    int ref = n / 2;
    float2 zr = w.vw[ref];

    if (hypotf(zr.x, zr.y) <= 1.0e-3f * mx) {
        for (int q = 0; q < n; q++) {
            const float2 zq = w.vw[q];

            if (hypotf(zq.x, zq.y) == mx)
                ref = q;
        }
        zr = w.vw[ref];
    }
    const float refm = hypotf(zr.x, zr.y);
    const float refr = zr.x / refm, refi = -zr.y / refm;
    const float re = z.x * refr - z.y * refi, im = z.x * refi + z.y * refr;
    const float mm = hypotf(re, im);

    w.z[i] = i < n && mm > mx * 1.0e-3f ? make_float2(re / mm, im / mm) : make_float2(1.f, 0.f);
    meet(g);
    const int npu = tc_npu(n);
    float sr = 0.f, si = 0.f;

#pragma unroll 4
    for (int q = i; q < npu; q += 64) {
        const int a = upper_tab[q] >> 8, b = upper_tab[q] & 255;
        const float2 u = unit_phasor(w.T[a * ld + b]), za = w.z[a], zb = w.z[b];
        const float wr = za.x * zb.x + za.y * zb.y, wi = za.x * zb.y - za.y * zb.x;

        sr += a == b ? 0.f : u.x * wr - u.y * wi;
        si += a == b ? 0.f : u.x * wi + u.y * wr;
    }
    sr = wsum(sr);
    si = wsum(si);
    if (g.lane == 0)
        *(float2 *)(w.red + 48 + 2 * g.warp) = make_float2(sr, si);
    meet(g);
    const float4 s = *(const float4 *)(w.red + 48);

    return hypotf(s.x + s.z, s.y + s.w) / (0.5f * n * (n - 1));
}

__global__ void __launch_bounds__(64 * WD_PIXELS)
tc_link_wide_kernel(TcStrip s, TcChunk c, TcLinkConst k, WideLayout L,
                    const float2 *__restrict__ gram, const int *__restrict__ count,
                    const unsigned short *__restrict__ upper_tab,
                    const unsigned short *__restrict__ pair_tab, float *__restrict__ coh,
                    float *__restrict__ pairs, float *__restrict__ phases,
                    unsigned char *__restrict__ status, const uint32_t *__restrict__ mask,
                    int *__restrict__ queue, int qstride)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int slot = threadIdx.x >> 6, slots = blockDim.x >> 6;
    const int n = s.n, ld = L.ld, npu = tc_npu(n);
    const long long plane = (long long)s.rows * s.cols;
    const Ws w = workspace(smem + (size_t)slot * L.per_pixel, L);
    unsigned short *s_upper = (unsigned short *)(smem + (size_t)slots * L.per_pixel);
    Duo g;

    g.lane = threadIdx.x & 31;
    g.warp = (threadIdx.x >> 5) & 1;
    g.row = threadIdx.x & 63;
    g.bar = 1 + slot;
    for (int e = threadIdx.x; e < npu; e += blockDim.x)
        s_upper[e] = upper_tab[e];
    __syncthreads();

    /* The pixels of a CTA go their own way: one pixel's serial stages (a third
       of its time) overlap the others' reduction. With CTA barriers between the
       stages, as the kernel for up to 32 dates has them, the link stage took 41.4
       ms instead of 34.4 (96 x 2048 at 60 dates). */
    for (int p = blockIdx.x * slots + slot; p < c.npix; p += gridDim.x * slots) {
        int y, x;

        tc_pixel_yx(c, p, y, x);
        if (y >= c.row0 + c.nrows || y >= s.rows || x >= s.cols)
            continue;
        const long long out = (long long)y * s.cols + x;
        const int looks = count[out];
        unsigned st = 0;
        bool estimate = looks >= k.min_looks;

        if (!estimate)
            for (int t = g.row; t < k.npairs; t += 64)
                pairs[t * plane + out] = NAN;
        else {
            const bool edge = load_T(n, ld, k, looks, gram + tc_gram_at(npu, p, 0), s_upper, w, g);

            if (queue && edge && g.row == 0)
                tc_exact_push(queue, qstride, out, mask, c.npix, p);
            for (int t = g.row; t < k.npairs; t += 64) {
                const float2 v = w.T[(pair_tab[t] >> 8) * ld + (pair_tab[t] & 255)];

                pairs[t * plane + out] = hypotf(v.x, v.y);
            }
            if (k.bias && !linked(n, ld, w.T, g)) {
                estimate = false;
                st = TC_STATUS_UNLINKED;
                meet(g); /* T is read until here */
            }
        }
        if (!estimate) {
            if (g.row == 0) {
                coh[out] = NAN;
                if (status)
                    status[out] = (unsigned char)st;
            }
            if (phases && g.row < n)
                phases[out * n + g.row] = NAN;
            continue;
        }
        {
            /* columns from n on read what follows the row, inside the workspace */
            const float2 *row = w.T + opaque(min(g.row, n - 1) * ld);
            float2 r[64];

#pragma unroll
            for (int j = 0; j < 64; j++) {
                const float2 t = row[j];

                r[j] = make_float2(g.row < n && j < n ? t.x : 0.f,
                                   g.row < n && j < n ? t.y : 0.f);
            }
            meet(g);
            householder(r, n, ld, w, g);
        }
        float norm;
        const float lambda = largest_eigenvalue(n, w, g, norm, st);

        if (g.warp == 0)
            inverse_iteration(n, lambda, norm, w, g);
        meet(g);
        float2 z = w.z[g.row];

        apply_q(n, ld, w, g, z);
        const float gamma = goodness(n, ld, w, g, z, s_upper);

        if (g.row == 0) {
            coh[out] = gamma;
            if (status)
                status[out] = (unsigned char)st;
        }
        if (phases && g.row < n) {
            const float2 u = w.z[g.row];

            phases[out * n + g.row] = atan2f(u.y, u.x);
        }
        meet(g);
    }
}

} // namespace

cudaError_t tc_launch_link_wide(const TcStrip &s, const TcChunk &c, const TcLinkConst &k,
                                const float2 *gram, const uint32_t *mask, const int *count,
                                const unsigned short *upper_tab, const unsigned short *pair_tab,
                                float *coh, float *pairs, float *phases, unsigned char *status,
                                int *queue, int qstride, int sms, cudaStream_t st)
{
    const WideLayout L = wide_layout(s.n);
    const size_t tab = ((size_t)tc_npu(s.n) * 2 + 15) & ~(size_t)15;
    int pixels = (int)((TC_SMEM_MAX - tab) / L.per_pixel);

    if (pixels > WD_PIXELS)
        pixels = WD_PIXELS;
    /* few pixels: over all SMs rather than in full CTAs on some */
    if (pixels > (c.npix + sms - 1) / sms)
        pixels = (c.npix + sms - 1) / sms;
    const size_t smem = (size_t)pixels * L.per_pixel + tab;
    const int want = (c.npix + pixels - 1) / pixels;
    const int blocks = want < sms ? want : sms;
    const cudaError_t e = tc_allow_smem(tc_link_wide_kernel);

    if (e != cudaSuccess)
        return e;
    tc_link_wide_kernel<<<blocks, 64 * pixels, smem, st>>>(
        s, c, k, L, gram, count, upper_tab, pair_tab, coh, pairs, phases, status, mask, queue,
        qstride);
    return cudaGetLastError();
}
