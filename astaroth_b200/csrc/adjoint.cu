/*
 * Discrete adjoint of one RK3 substep (acDeviceIntegrateSubstepAdjoint).
 *
 * The forward substep in 2N form (acc-runtime/stdlib/integrators.h:11-29,
 * host model src/utils/modelsolver.cc:1078-1175) is
 *     w_s     = alpha_s w_{s-1} + dt R(f_s)
 *     f_{s+1} = f_s + beta_s w_s
 * with R the 6th-order MHD right-hand side on the periodic mesh.  Its adjoint
 * maps the adjoints (lf, lw) of (f_{s+1}, w_s) to those of (f_s, w_{s-1}):
 *     lw <- lw + beta_s lf
 *     lf <- lf + dt J_R(f_s)^T lw
 *     lw <- alpha_s lw
 * and accumulates d/d(nu, eta) of dt lw . R.  J_R^T is applied in two
 * passes: adj_local_kernel evaluates, per cell, the reverse of the RHS into the
 * adjoints mu of the 46 derivative slots (mhd_rhs_adjoint.cuh), adds the 8
 * value slots to lf directly and stores the 38 others; adj_gather_kernel then
 * applies the transposed stencils at wrapped (periodic) interior indices, so
 * mu needs no halo fill: first derivatives are antisymmetric (D^T = -D),
 * second, Laplacian and the diagonal mixed stencils are symmetric, so the
 * gather for a vector field is - div-like first-derivative terms + lap + grad
 * div of the slot fields.  The gather runs one output field per block.
 *
 * The slot arrays have one of two layouts (ac_adjoint_pairs).  Packed, they hold
 * the interior cells only (x fastest, rows of nx): with nx even every pair of x
 * neighbours is then one aligned 16-byte value, and adj_gather2_kernel forms two
 * cells per thread from such loads.  Otherwise they are laid out as the fields,
 * and the cells of a thread have one index in both.
 */
#include "internal.h"
#include "mhd_rhs_adjoint.cuh"
#include "stencil_plain.cuh"

namespace {

/* z planes per thread of the gather.  Consecutive planes of one column share
 * most stencil taps through L1, but the kernel is latency-bound, and one plane
 * per thread (8x the blocks) measured 10% faster per adjoint substep at 64^3
 * than 2, 4 or 8 planes.  (The local kernel also keeps one plane per thread:
 * a loop there spills its 254 registers.) */
constexpr int KZ = 1;

/* index of interior cell (i, j, k) in a packed slot array */
__device__ __forceinline__ long long
mu_idx(const Geom& g, const int i, const int j, const int k)
{
    return i + (long long)g.nx * (j + (long long)g.ny * k);
}

template <bool PACKED>
__global__ void __launch_bounds__(128)
adj_local_kernel(const Geom g, const AdjointFields a, const StencilCoef sc, const PhysConst pc,
                 const double beta, const double dt, double* __restrict__ pgrad)
{
    __shared__ double red[2 * 4];
    const int i = threadIdx.x + blockIdx.x * blockDim.x;
    const int j = threadIdx.y + blockIdx.y * blockDim.y;
    const int k = blockIdx.z;
    double gnu = 0, geta = 0;
    if (i < g.nx && j < g.ny && k < g.nz) {
        const long long idx   = geom_idx(g, i + NGHOST, j + NGHOST, k + NGHOST);
        const long long st[3] = {1, (long long)g.px, g.pxy};
        const long long midx  = PACKED ? mu_idx(g, i, j, k) : idx;
        double lam[AC_NF];
#pragma unroll
        for (int q = 0; q < AC_NF; ++q) {
            const double w = a.lw[q][idx] + beta * a.lf[q][idx];
            a.lw[q][idx]   = w;
            lam[q]         = dt * w;
        }
        ScalD<double> L, S;
        VecD<double> U, A;
        scal_derivs(a.f[VTXBUF_LNRHO] + idx, st, sc, L);
        scal_derivs(a.f[VTXBUF_ENTROPY] + idx, st, sc, S);
        {
            const double* uc[3] = {a.f[VTXBUF_UUX] + idx, a.f[VTXBUF_UUY] + idx,
                                   a.f[VTXBUF_UUZ] + idx};
            vec_derivs(uc, st, sc, U);
            const double* ac[3] = {a.f[VTXBUF_AX] + idx, a.f[VTXBUF_AY] + idx,
                                   a.f[VTXBUF_AZ] + idx};
            vec_derivs(ac, st, sc, A);
        }
        /* the rate order of mhd_rates: lnrho, ux, uy, uz, ax, ay, az, entropy */
        double mu[MU_COUNT];
        mhd_rates_adjoint(L, S, U, A, phys_cast<double>(pc), lam, mu, gnu, geta);
        /* value slots need no stencil: their transpose is the identity */
        const int vslot[AC_NF] = {MU_L + MU_SV,     MU_U + MU_VV,     MU_U + MU_VV + 1,
                                  MU_U + MU_VV + 2, MU_A + MU_VV,     MU_A + MU_VV + 1,
                                  MU_A + MU_VV + 2, MU_S + MU_SV};
#pragma unroll
        for (int q = 0; q < AC_NF; ++q)
            a.lf[q][idx] += mu[vslot[q]];
#pragma unroll
        for (int m = 0; m < MU_COUNT; ++m) {
            const bool value_slot = m == MU_L + MU_SV || m == MU_S + MU_SV ||
                                    (m >= MU_U + MU_VV && m < MU_U + MU_VV + 3) ||
                                    (m >= MU_A + MU_VV && m < MU_A + MU_VV + 3);
            if (!value_slot)
                a.mu[m][midx] = mu[m];
        }
    }
    /* block sums of the parameter adjoints, one atomic per block and value */
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gnu += __shfl_xor_sync(0xffffffffu, gnu, o);
        geta += __shfl_xor_sync(0xffffffffu, geta, o);
    }
    if (lane == 0) {
        red[2 * warp]     = gnu;
        red[2 * warp + 1] = geta;
    }
    __syncthreads();
    if (tid == 0) {
        double s0 = 0, s1 = 0;
        for (int w = 0; w < 4; ++w) {
            s0 += red[2 * w];
            s1 += red[2 * w + 1];
        }
        atomicAdd(pgrad, s0);
        atomicAdd(pgrad + 1, s1);
    }
}

/* Periodic neighbour offsets of one interior cell: o[a][d + 3] is the index
 * offset of the interior cell d steps away along axis a, wrapped.  The slot
 * arrays mu are read only at interior cells, so they need no halo fill. */
struct Wrap {
    long long o[3][7];
};

__device__ __forceinline__ int
wrap(const int v, const int n)
{
    const int r = v % n;
    return r < 0 ? r + n : r;
}

__device__ __forceinline__ void
make_wrap(const Geom& g, const int i, const int j, const int k, Wrap& w)
{
#pragma unroll
    for (int d = -3; d <= 3; ++d) {
        w.o[0][d + 3] = (long long)(wrap(i + d, g.nx) - i);
        w.o[1][d + 3] = (long long)(wrap(j + d, g.ny) - j) * g.px;
        w.o[2][d + 3] = (long long)(wrap(k + d, g.nz) - k) * g.pxy;
    }
}

/* sum_k c_k (f[+k] - f[-k]) along axis A */
template <int A>
__device__ __forceinline__ double
wd1(const double* f, const Wrap& w, const double* c)
{
    double r = c[0] * (__ldg(f + w.o[A][4]) - __ldg(f + w.o[A][2]));
    r        = fma(c[1], __ldg(f + w.o[A][5]) - __ldg(f + w.o[A][1]), r);
    r        = fma(c[2], __ldg(f + w.o[A][6]) - __ldg(f + w.o[A][0]), r);
    return r;
}

/* sum_k d_k (f[+k] + f[-k]) along axis A (centre excluded) */
template <int A>
__device__ __forceinline__ double
wd2s(const double* f, const Wrap& w, const double* d)
{
    double r = d[1] * (__ldg(f + w.o[A][4]) + __ldg(f + w.o[A][2]));
    r        = fma(d[2], __ldg(f + w.o[A][5]) + __ldg(f + w.o[A][1]), r);
    r        = fma(d[3], __ldg(f + w.o[A][6]) + __ldg(f + w.o[A][0]), r);
    return r;
}

/* sum_k e_k (f(+k,+k) + f(-k,-k) - f(+k,-k) - f(-k,+k)) along axes A, B */
template <int A, int B>
__device__ __forceinline__ double
wmix(const double* f, const Wrap& w, const double* e)
{
    double r = 0;
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        const double t = (__ldg(f + w.o[A][3 + k] + w.o[B][3 + k]) +
                          __ldg(f + w.o[A][3 - k] + w.o[B][3 - k])) -
                         (__ldg(f + w.o[A][3 + k] + w.o[B][3 - k]) +
                          __ldg(f + w.o[A][3 - k] + w.o[B][3 + k]));
        r = k == 1 ? e[0] * t : fma(e[k - 1], t, r);
    }
    return r;
}

__device__ __forceinline__ double
wlap(const double* f, const Wrap& w, const StencilCoef& sc)
{
    return (sc.d2[0][0] + sc.d2[1][0] + sc.d2[2][0]) * __ldg(f) + wd2s<0>(f, w, sc.d2[0]) +
           wd2s<1>(f, w, sc.d2[1]) + wd2s<2>(f, w, sc.d2[2]);
}

/* - sum_a D_a g_a + lap(l): the transposed first-derivative and Laplacian
 * terms of one output field (D1^T = -D1, the Laplacian is symmetric) */
__device__ __forceinline__ double
gather_gl(const AdjointFields& a, const int g0, const int l, const long long idx, const Wrap& w,
          const StencilCoef& sc)
{
    double acc = -wd1<0>(a.mu[g0] + idx, w, sc.d1[0]);
    acc -= wd1<1>(a.mu[g0 + 1] + idx, w, sc.d1[1]);
    acc -= wd1<2>(a.mu[g0 + 2] + idx, w, sc.d1[2]);
    return acc + wlap(a.mu[l] + idx, w, sc);
}

/* (grad div)^T = grad div of the three gd slots, component C */
template <int C>
__device__ __forceinline__ double
gather_gd(const AdjointFields& a, const int gd0, const long long idx, const Wrap& w,
          const StencilCoef& sc)
{
    const double* g0 = a.mu[gd0] + idx;
    const double* g1 = a.mu[gd0 + 1] + idx;
    const double* g2 = a.mu[gd0 + 2] + idx;
    if (C == 0)
        return (sc.d2[0][0] * __ldg(g0) + wd2s<0>(g0, w, sc.d2[0])) +
               wmix<0, 1>(g1, w, sc.mix[0]) + wmix<0, 2>(g2, w, sc.mix[1]);
    if (C == 1)
        return wmix<0, 1>(g0, w, sc.mix[0]) + (sc.d2[1][0] * __ldg(g1) + wd2s<1>(g1, w, sc.d2[1])) +
               wmix<1, 2>(g2, w, sc.mix[2]);
    return wmix<0, 2>(g0, w, sc.mix[1]) + wmix<1, 2>(g1, w, sc.mix[2]) +
           (sc.d2[2][0] * __ldg(g2) + wd2s<2>(g2, w, sc.d2[2]));
}

/* Slot arrays laid out as the fields.  One output field per block
 * (blockIdx.z = zblock * AC_NF + q), so a block reads only the slot arrays of
 * that field; KZ planes per thread. */
__global__ void __launch_bounds__(128)
adj_gather_kernel(const Geom g, const AdjointFields a, const StencilCoef sc, const double alpha)
{
    const int i = threadIdx.x + blockIdx.x * blockDim.x;
    const int j = threadIdx.y + blockIdx.y * blockDim.y;
    const int q = blockIdx.z % AC_NF;
    if (i >= g.nx || j >= g.ny)
        return;
    const int k1 = min((int)(blockIdx.z / AC_NF + 1) * KZ, g.nz);
    for (int k = blockIdx.z / AC_NF * KZ; k < k1; ++k) {
        const long long idx = geom_idx(g, i + NGHOST, j + NGHOST, k + NGHOST);
        Wrap w;
        make_wrap(g, i, j, k, w);
        double add;
        if (q == VTXBUF_LNRHO || q == VTXBUF_ENTROPY) {
            const int m = q == VTXBUF_LNRHO ? MU_L : MU_S;
            add         = gather_gl(a, m + MU_SG, m + MU_SLAP, idx, w, sc);
        }
        else {
            const int m = q <= VTXBUF_UUZ ? MU_U : MU_A;
            const int c = q <= VTXBUF_UUZ ? q - VTXBUF_UUX : q - VTXBUF_AX;
            add         = gather_gl(a, m + MU_VG + 3 * c, m + MU_VLAP + c, idx, w, sc);
            add += c == 0 ? gather_gd<0>(a, m + MU_VGD, idx, w, sc)
                          : c == 1 ? gather_gd<1>(a, m + MU_VGD, idx, w, sc)
                                   : gather_gd<2>(a, m + MU_VGD, idx, w, sc);
        }
        a.lf[q][idx] += add;
        a.lw[q][idx] *= alpha;
    }
}

/* ---- two x neighbours per thread (packed slot arrays, nx even) ----
 * The gather is bound by its loads through L1 (about 490 taps a cell).  As pairs a
 * row's seven x taps of both cells are 5 loads instead of 14, a y or z tap one
 * instead of two.  The sums are those of the functions above, term by term.
 * Measured per adjoint substep (both kernels): 64^3 195 -> 152 us, 96^3 632 -> 484,
 * 32^3 27.5 -> 23.6.  Eight blocks per SM at 64 registers, with a little spilled, beat
 * four at 110 (168 us at 64^3): the kernel waits for L1 and L2. */
struct WrapPair {
    int x[5];       /* offsets of the pairs -2 .. 2 from the cell's */
    int y[7], z[7]; /* offsets of the rows, planes -3 .. 3 */
};

struct D2 {
    double v[2];
};

__device__ __forceinline__ D2
ldp(const double* p)
{
    const double2 t = __ldg(reinterpret_cast<const double2*>(p));
    return D2{{t.x, t.y}};
}

template <int A>
__device__ __forceinline__ int
off2(const WrapPair& w, const int d)
{
    return A == 1 ? w.y[d + 3] : w.z[d + 3];
}

/* x - 4 .. x + 5 of one row (x: the pair's first cell) */
struct Row {
    double v[10];
};
template <unsigned PAIRS> /* bit d: pair d - 2 is loaded */
__device__ __forceinline__ void
load_row(const double* f, const WrapPair& w, Row& r)
{
#pragma unroll
    for (int d = 0; d < 5; ++d)
        if (PAIRS >> d & 1u) {
            const D2 t   = ldp(f + w.x[d]);
            r.v[2 * d]     = t.v[0];
            r.v[2 * d + 1] = t.v[1];
        }
}

__device__ __forceinline__ void
pd1x(const Row& r, const double* c, D2& o)
{
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double* m = r.v + 4 + s;
        double t        = c[0] * (m[1] - m[-1]);
        t               = fma(c[1], m[2] - m[-2], t);
        o.v[s]          = fma(c[2], m[3] - m[-3], t);
    }
}
__device__ __forceinline__ void
pd2x(const Row& r, const double* d, D2& o)
{
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double* m = r.v + 4 + s;
        double t        = d[1] * (m[1] + m[-1]);
        t               = fma(d[2], m[2] + m[-2], t);
        o.v[s]          = fma(d[3], m[3] + m[-3], t);
    }
}
template <int A>
__device__ __forceinline__ D2
pd1(const double* f, const WrapPair& w, const double* c)
{
    D2 r;
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        const D2 p = ldp(f + off2<A>(w, k)), m = ldp(f + off2<A>(w, -k));
#pragma unroll
        for (int s = 0; s < 2; ++s)
            r.v[s] = k == 1 ? c[0] * (p.v[s] - m.v[s]) : fma(c[k - 1], p.v[s] - m.v[s], r.v[s]);
    }
    return r;
}
template <int A>
__device__ __forceinline__ D2
pd2s(const double* f, const WrapPair& w, const double* d)
{
    D2 r;
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        const D2 p = ldp(f + off2<A>(w, k)), m = ldp(f + off2<A>(w, -k));
#pragma unroll
        for (int s = 0; s < 2; ++s)
            r.v[s] = k == 1 ? d[1] * (p.v[s] + m.v[s]) : fma(d[k], p.v[s] + m.v[s], r.v[s]);
    }
    return r;
}
/* wmix<0, B> */
template <int B, int K>
__device__ __forceinline__ void
pmixx_k(const double* f, const WrapPair& w, const double* e, D2& r)
{
    /* the pairs that hold x - K, x + K of both cells */
    constexpr unsigned P = K == 1 ? 0x0eu : K == 2 ? 0x0au : 0x1bu;
    Row p, m;
    load_row<P>(f + off2<B>(w, K), w, p);
    load_row<P>(f + off2<B>(w, -K), w, m);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double t = (p.v[4 + s + K] + m.v[4 + s - K]) - (m.v[4 + s + K] + p.v[4 + s - K]);
        r.v[s]         = K == 1 ? e[0] * t : fma(e[K - 1], t, r.v[s]);
    }
}
template <int B>
__device__ __forceinline__ D2
pmixx(const double* f, const WrapPair& w, const double* e)
{
    D2 r;
    pmixx_k<B, 1>(f, w, e, r);
    pmixx_k<B, 2>(f, w, e, r);
    pmixx_k<B, 3>(f, w, e, r);
    return r;
}
/* wmix<1, 2> */
__device__ __forceinline__ D2
pmixyz(const double* f, const WrapPair& w, const double* e)
{
    D2 r;
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        const D2 pp = ldp(f + w.y[3 + k] + w.z[3 + k]), mm = ldp(f + w.y[3 - k] + w.z[3 - k]);
        const D2 pm = ldp(f + w.y[3 + k] + w.z[3 - k]), mp = ldp(f + w.y[3 - k] + w.z[3 + k]);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double t = (pp.v[s] + mm.v[s]) - (pm.v[s] + mp.v[s]);
            r.v[s]         = k == 1 ? e[0] * t : fma(e[k - 1], t, r.v[s]);
        }
    }
    return r;
}

/* One output field per block (blockIdx.y = z * AC_NF + q), a pair of cells per
 * thread, the pairs of a plane counted through its rows. */
__global__ void __launch_bounds__(128, 8)
adj_gather2_kernel(const Geom g, const AdjointFields a, const StencilCoef sc, const double alpha)
{
    const int M = g.nx / 2;
    const int t = blockIdx.x * 128 + threadIdx.x;
    const int q = blockIdx.y % AC_NF, k = blockIdx.y / AC_NF;
    if (t >= M * g.ny)
        return;
    const int j = t / M, m = t - j * M, i = 2 * m;
    WrapPair w;
#pragma unroll
    for (int d = -2; d <= 2; ++d)
        w.x[d + 2] = 2 * (wrap(m + d, M) - m);
#pragma unroll
    for (int d = -3; d <= 3; ++d) {
        w.y[d + 3] = (wrap(j + d, g.ny) - j) * g.nx;
        w.z[d + 3] = (wrap(k + d, g.nz) - k) * g.nx * g.ny;
    }
    const long long midx = mu_idx(g, i, j, k);
    const bool scal      = q == VTXBUF_LNRHO || q == VTXBUF_ENTROPY;
    const int b          = q == VTXBUF_LNRHO ? MU_L : q == VTXBUF_ENTROPY ? MU_S
                           : q <= VTXBUF_UUZ ? MU_U : MU_A;
    const int c  = q <= VTXBUF_UUZ ? q - VTXBUF_UUX : q - VTXBUF_AX; /* vectors only */
    const int g0 = scal ? b + MU_SG : b + MU_VG + 3 * c;
    const int l  = scal ? b + MU_SLAP : b + MU_VLAP + c;
    D2 add;
    { /* gather_gl */
        Row r;
        D2 u;
        load_row<0x1fu>(a.mu[g0] + midx, w, r);
        pd1x(r, sc.d1[0], u);
        const D2 v = pd1<1>(a.mu[g0 + 1] + midx, w, sc.d1[1]);
        const D2 z = pd1<2>(a.mu[g0 + 2] + midx, w, sc.d1[2]);
        Row lr;
        D2 lx;
        load_row<0x1fu>(a.mu[l] + midx, w, lr);
        pd2x(lr, sc.d2[0], lx);
        const D2 ly = pd2s<1>(a.mu[l] + midx, w, sc.d2[1]);
        const D2 lz = pd2s<2>(a.mu[l] + midx, w, sc.d2[2]);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            double acc = -u.v[s];
            acc -= v.v[s];
            acc -= z.v[s];
            add.v[s] = acc + ((sc.d2[0][0] + sc.d2[1][0] + sc.d2[2][0]) * lr.v[4 + s] + lx.v[s] +
                              ly.v[s] + lz.v[s]);
        }
    }
    if (!scal) { /* gather_gd */
        const double* f0 = a.mu[b + MU_VGD] + midx;
        const double* f1 = a.mu[b + MU_VGD + 1] + midx;
        const double* f2 = a.mu[b + MU_VGD + 2] + midx;
        D2 x, y, z;
        if (c == 0) {
            Row r;
            load_row<0x1fu>(f0, w, r);
            pd2x(r, sc.d2[0], x);
#pragma unroll
            for (int s = 0; s < 2; ++s)
                x.v[s] = sc.d2[0][0] * r.v[4 + s] + x.v[s];
            y = pmixx<1>(f1, w, sc.mix[0]);
            z = pmixx<2>(f2, w, sc.mix[1]);
        }
        else if (c == 1) {
            x            = pmixx<1>(f0, w, sc.mix[0]);
            const D2 ctr = ldp(f1);
            y            = pd2s<1>(f1, w, sc.d2[1]);
#pragma unroll
            for (int s = 0; s < 2; ++s)
                y.v[s] = sc.d2[1][0] * ctr.v[s] + y.v[s];
            z = pmixyz(f2, w, sc.mix[2]);
        }
        else {
            x            = pmixx<2>(f0, w, sc.mix[1]);
            y            = pmixyz(f1, w, sc.mix[2]);
            const D2 ctr = ldp(f2);
            z            = pd2s<2>(f2, w, sc.d2[2]);
#pragma unroll
            for (int s = 0; s < 2; ++s)
                z.v[s] = sc.d2[2][0] * ctr.v[s] + z.v[s];
        }
#pragma unroll
        for (int s = 0; s < 2; ++s)
            add.v[s] += x.v[s] + y.v[s] + z.v[s];
    }
    const long long idx = geom_idx(g, i + NGHOST, j + NGHOST, k + NGHOST);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        a.lf[q][idx + s] += add.v[s];
        a.lw[q][idx + s] *= alpha;
    }
}

/* the blocks of adj_gather_kernel: 32 x 4 cells of a plane and a field */
const dim3 kTile(32, 4, 1);
dim3
tiles_of(const Geom& g)
{
    return dim3((unsigned)((g.nx + kTile.x - 1) / kTile.x), (unsigned)((g.ny + kTile.y - 1) / kTile.y),
                (unsigned)g.nz);
}

} // namespace

/* Pairs need an even nx and 32-bit offsets.  They halve the threads, which pays from about
 * 1.75 waves of the other gather's blocks (seven per SM) on: us per adjoint substep, cells /
 * pairs: 16^3 16.9 / 18.1, 26 x 20 x 30 (1.2 waves) 21.1 / 23.3, 28^3 (1.5) 23.0 / 24.3,
 * 32^3 (2.0) 26.5 / 24.7, 16 x 16 x 80 (2.5) 31.6 / 27.2, 64^3 169 / 152.  With nx odd, cells of
 * packed arrays were slower than cells of arrays like the fields' (a second set of
 * indices, 90 registers against 72): 65 x 64 x 64 252 against 227, 95 x 79 x 80 412 / 374. */
bool
ac_adjoint_pairs(const Geom& g)
{
    const dim3 b           = tiles_of(g);
    const long long blocks = (long long)b.x * b.y * b.z * AC_NF;
    return g.nx % 2 == 0 && 4 * blocks >= 7 * (7LL * AC_SMS) &&
           (long long)g.nx * g.ny * g.nz < (1LL << 31);
}

cudaError_t
ac_launch_adjoint_substep(const Geom& g, const AdjointFields& a, const StencilCoef& sc,
                          const PhysConst& pc, const double alpha, const double beta,
                          const double dt, double* pgrad, cudaStream_t stream,
                          unsigned long long* launches)
{
    const dim3 bpg   = tiles_of(g);
    const bool pairs = ac_adjoint_pairs(g);
    if (pairs)
        adj_local_kernel<true><<<bpg, kTile, 0, stream>>>(g, a, sc, pc, beta, dt, pgrad);
    else
        adj_local_kernel<false><<<bpg, kTile, 0, stream>>>(g, a, sc, pc, beta, dt, pgrad);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    const unsigned zb = (unsigned)((g.nz + KZ - 1) / KZ);
    if ((long long)zb * AC_NF > 65535)
        return cudaErrorInvalidConfiguration;
    if (pairs) {
        const dim3 ppg((unsigned)((g.nx / 2 * g.ny + 127) / 128), (unsigned)g.nz * AC_NF);
        adj_gather2_kernel<<<ppg, 128, 0, stream>>>(g, a, sc, alpha);
    }
    else {
        const dim3 gpg(bpg.x, bpg.y, zb * AC_NF);
        adj_gather_kernel<<<gpg, kTile, 0, stream>>>(g, a, sc, alpha);
    }
    if (launches)
        *launches += 2;
    return cudaGetLastError();
}
