/*
 * The substep kernel: 2.5-D blocking with the work of every cell split over
 * four warp groups, for FP64 and FP32-compensated meshes.
 *
 * A block owns an (x, y) tile of 32 x 4 cells (FP64) or 32 x 8 cells (FP32,
 * two cells per thread: rows y and y + 4 of the tile as one packed value) and
 * marches along z over a chunk of planes.  TMA (cp.async.bulk.tensor.4d,
 * CTA-local) brings one plane of all 8 fields, halo included, into a ring of
 * shared-memory slots.  The 16 warps are four roles of four warps; the warps
 * with the same number mod 4 hold the same 32 cells (values), so they share 32
 * lanes of tensor memory, through which all intermediate values pass:
 *
 *   in-plane, hydro / magnetic   reads plane L = i of its four fields (lnrho and
 *       uu; aa and entropy) from shared memory in interval i, each tap once:
 *       the x and y differences D^k f = f(+k) - f(-k) and sums S^k give the
 *       in-plane first and second derivatives and the diagonal xy mixed
 *       derivatives (the plane's record).
 *       The xz and yz mixed derivatives use the separable form of the diagonal
 *       stencil (acc-runtime/stdlib/derivs.h:591-690),
 *       D_az f(z) = sum_k e_k [D_a^k f(z+k) - D_a^k f(z-k)], as six running sums
 *       per term in registers, each moved on by one plane as it is added to.
 *   solve, hydro / magnetic      of plane p = i - 4 in interval i: the z
 *       derivatives from a queue of eight planes, the record, the finished
 *       mixed sums; the two groups exchange 7 + 10 values through tensor memory
 *       (the RHS's two exponentials among them, one formed by each), and in
 *       interval i + 1 form their four rates and the RK update.  The previous state
 *       comes by TMA too, a tile of the plane ahead of time: loaded by the threads,
 *       its latency was in every interval (FP64 256^3 substep 1.07 against 0.90 ms
 *       for substep 0, which reads none; now 0.95).
 *
 * One block barrier per interval orders everything: what an interval stores is
 * read in a later one, and every tensor-memory area has one slot more than the
 * planes that are alive (record: 5, mixed sums: 2, queue: 8, exchange: 2), so
 * no slot is written while it is read.
 *
 * What bounds it (B200, 256^3): FP64 issues on 68% of cycles with the FP64 pipe
 * 55% busy and shared memory 65%; FP32 issues on 63-66%.  One warp of every role
 * per scheduler keeps all of these in use at once; two groups of one kind
 * (one barrier per plane, 8 warps) issued on 59%.  Measured against that kernel,
 * per RK3 step: 256^3 FP64 3.60 -> 3.01 ms, FP32 3.09 -> 2.5 ms; 128^3 0.60 ->
 * 0.46 and 0.50 -> 0.36 ms.  A barrier per quarter instead of the block's lets
 * the roles drift apart, and the instruction cache then misses (FP32 0.98 -> 1.18
 * ms a substep); a fifth role for uz, Az and the scalars takes the registers
 * that the solve roles need (FP64 1.10, FP32 1.05 ms); barriers that let the
 * in-plane roles run a plane ahead cost more instructions than the wait.
 *
 * Folded coefficients: only nu lap u + (nu/3 + zeta) grad div u and
 * (grad div A - lap A) / mu0 enter the equations, so the in-plane groups form
 * these combinations from coefficients that the host has multiplied out
 * (SplitCoef), and derivatives that no equation uses (the diagonal of grad A)
 * are not formed.
 *
 * Reference: singlepass_solve / twopass_solve_intermediate,
 * acc-runtime/samples/mhd_modular/mhdsolver.ac:279-426,524-612 (every tap is a
 * separate load there, acc-runtime/acc/stencilgen.c:2205).
 *
 * Waits on mbarriers are bounded: a wait that gives up sets *err and the kernel
 * still runs to completion (no barrier is skipped); the host turns *err into
 * AC_FAILURE.
 */
#include <cuda.h>
#include <atomic>
#include <initializer_list>
#include <type_traits>
#include <vector>

#include "internal.h"
#include "mhd_rhs.cuh"
#include "pack.cuh"
#include "tma_ring.cuh"
#include "tmem.cuh"

namespace {

using namespace tma_ring;

constexpr int TX      = 32;
constexpr int WARPS_Y = 4;                     /* warps per role */
constexpr int ROLES   = 4;
constexpr int STH     = WARPS_Y * TX; /* threads of a role */
constexpr int THREADS = ROLES * STH;
/* registers per thread: the block is launched with 128 each, and the in-plane
 * roles pass 8 to the solve roles (setmaxnreg; checked in init_split).  Measured
 * at 256^3, per step: FP64 3.01 ms against 3.26 with 128 each and 3.27 with 112
 * and 144; FP32 2.47 against 2.54 and 2.33. */
constexpr int REGS_INPLANE = 120, REGS_SOLVE = 136;

template <typename V>
struct SplitTile {
    typedef typename Pack<V>::T T;
    static constexpr int TY    = WARPS_Y * Pack<V>::N; /* cells along y */
    static constexpr int HY    = TY + 2 * NGHOST;
    static constexpr int HXP   = sizeof(T) == 8 ? TX + 2 * NGHOST : 40; /* rows of 16-byte multiples */
    static constexpr int PLANE = HXP * HY;
    static constexpr int SLOT  = AC_NF * PLANE;
    static constexpr unsigned SLOT_BYTES = SLOT * sizeof(T);
    static constexpr int RING  = 4;
    /* the tile of one plane of one previous-state array (no halo; x from the
     * 16-byte boundary at or before the tile) */
    static constexpr int PX0   = sizeof(T) == 8 ? 2 : 0; /* first x of the tile's box */
    static constexpr int PXW   = sizeof(T) == 8 ? 34 : 36;
    static constexpr int PFLD  = PXW * TY;
    static constexpr unsigned PARR_BYTES = AC_NF * PFLD * sizeof(T);
    static constexpr int PARR  = sizeof(T) == 8 ? 1 : 3; /* arrays: previous value; FP32 also the
                                                          * compensation words, old and new */
    static constexpr unsigned PSLOT_BYTES = PARR * PARR_BYTES;
    static constexpr int PRING = sizeof(T) == 8 ? 4 : 3;
    static constexpr size_t P_OFF      = (size_t)RING * SLOT_BYTES;
    static constexpr size_t RED_OFF    = P_OFF + (size_t)PRING * PSLOT_BYTES; /* CFL commit */
    static constexpr size_t BAR_OFF    = RED_OFF + 512;
    static constexpr int NBARS         = RING + PRING; /* mbarriers: planes, previous state */
    static constexpr size_t SMEM_BYTES = BAR_OFF + NBARS * sizeof(uint64_t) + 16;
};

/* tensor maps of a launch */
struct SplitMaps {
    CUtensorMap plane;   /* in-buffer values, a tile with its halo */
    CUtensorMap prev;    /* out-buffer values, a tile */
    CUtensorMap prev_lo; /* FP32: their compensation words */
    CUtensorMap lo;      /* FP32: the in-buffer's compensation words */
};

/* Coefficients with everything known on the host multiplied out. */
template <typename V>
struct SplitCoef {
    V d1[3][3];  /* first derivative, [axis][k-1] */
    /* Laplacians of lnrho, s and A in a unit (lap_unit; FP64: 1) that the factors gicp_l,
     * gm1_l, eta and nim take back: sides, [axis][k-1]; what d2c[a] adds to the centre of
     * the other two axes; centres of all axes and of two */
    V d2[3][3];
    V d2c[3];
    V c_all, c_xy, c_yz, c_xz;
    /* hydro: nu lap u_c + vg d/dx_c div u, vg = nu/3 + zeta */
    V vd[3][3]; /* (nu + vg) d2 sides: axis c of component c */
    V vn[3][3]; /* nu d2 sides: the other axes */
    V vc[3];    /* the centre of component c, all axes */
    V vcl[3];   /* FP32: what vc lacks to cancel the sides exactly.  Rounded to FP32 alone it
                 * changes a constant u by up to 6e-8 of itself per nu/ds^2 of time, in one
                 * direction (512^3, 100 steps: 1.6e-6 of max|u|; with this 1.1e-7) */
    V vm[3][3]; /* vg mix, [xy, xz, yz][k-1] */
    V vmn[2][3]; /* -vg mix, [xz, yz] */
    /* magnetic: j = (grad div A - lap A) / mu0 */
    V mm[3][3]; /* mix / mu0 */
    V mmn[2][3];
    V nim;      /* -1/mu0 (times lap_unit) */
    V up[3][4]; /* upwinding, [axis][k]: centre and sides */
    /* equations */
    V m23, two, one_half, nu, inv_cp, ncs2, gicp, gm1, gicp_l, gm1_l, gm1_lnrho0, inv_exp_lnT0, eta,
        eta_mu0, zeta, K;
};

/* v over what FP32 holds of it */
inline double
made_up(const double v)
{
    const double r = v / (double)(float)v;
    return r > 0.5 && r < 2 ? r : 1; /* (1 for zero and for what FP32 does not hold) */
}

/* FP32: a unit for Laplacians that are only used times the factors f.  The sides of an
 * isotropic mesh are 270, -27 and 2 in units of 1/(180 ds^2) and the centre is -1470, so
 * that in 1/m of it (ds: the smallest spacing), m a whole number, all of them are FP32
 * numbers and a constant has no Laplacian: only the factors times the unit are rounded, and
 * m is the one of 64 for which these are rounded least (to about 1.5e-8 of themselves).
 * Rounded at 1/ds^2 every coefficient was off by up to 6e-8, by chance of the spacing, and a
 * constant had a Laplacian of 5e-7 / ds^2 of its value at 512^3 (entropy 3.0e-7 off FP64
 * after 100 steps). */
inline long double
lap_unit(const StencilCoef& s, const std::initializer_list<double> f)
{
    const double base = fmax(s.d2[0][1], fmax(s.d2[1][1], s.d2[2][1])) / 270;
    double least      = 1;
    int best          = 1;
    for (int m = 1; m <= 64; ++m) {
        double off = 0;
        for (const double v : f)
            off = fmax(off, fabs(made_up(v * base / m) - 1));
        if (off < least) {
            least = off;
            best  = m;
        }
    }
    return (long double)base / best;
}

template <typename V>
SplitCoef<V>
make_coef(const StencilCoef& s, const PhysConst& p)
{
    SplitCoef<V> c;
    auto D          = [](const long double v) { return Pack<V>::dup((double)v); };
    constexpr bool FP32 = Pack<V>::N == 2;
    const long double nu = p.nu, vg = (long double)p.nu / 3 + p.zeta, im = p.inv_mu0;
    /* K multiplies the Laplacians of lnrho and s too: their factors make up for its rounding */
    const double kr      = FP32 ? made_up(p.K) : 1;
    const long double unit =
        FP32 ? lap_unit(s, {p.gamma_inv_cp * kr, p.gamma_m1 * kr, p.eta, p.inv_mu0}) : 1;
    /* The heating eta mu0 j^2 / rho + 2 nu S:S + zeta (div u)^2 is used times exp(-lnT0) only:
     * that factor makes up for the rounding of nu, the others for what it then is off */
    const double by_T = FP32 ? p.inv_exp_lnT0 * made_up(p.nu) : p.inv_exp_lnT0;
    const double rest = FP32 ? made_up(by_T) / made_up(p.nu) : 1;
    for (int a = 0; a < 3; ++a) {
        for (int k = 0; k < 3; ++k) {
            c.d1[a][k] = D(s.d1[a][k]);
            c.d2[a][k] = D(s.d2[a][k + 1] / unit);
            c.vd[a][k] = D((nu + vg) * s.d2[a][k + 1]);
            c.vn[a][k] = D(nu * s.d2[a][k + 1]);
            c.vm[a][k] = D(vg * s.mix[a][k]);
            c.mm[a][k] = D(im * s.mix[a][k]);
            if (a > 0) {
                c.vmn[a - 1][k] = D(-vg * s.mix[a][k]);
                c.mmn[a - 1][k] = D(-im * s.mix[a][k]);
            }
        }
        for (int k = 0; k < 4; ++k)
            c.up[a][k] = D(s.up[a][k]);
        c.vc[a]  = D(nu * ((long double)s.d2[0][0] + s.d2[1][0] + s.d2[2][0]) + vg * s.d2[a][0]);
    }
    if (FP32)
        for (int q = 0; q < 3; ++q) {
            long double sides = 0; /* of the FP32 coefficients */
            for (int a = 0; a < 3; ++a)
                for (int k = 0; k < 3; ++k)
                    sides += 2 * (long double)(float)(a == q ? (double)((nu + vg) * s.d2[a][k + 1])
                                                             : (double)(nu * s.d2[a][k + 1]));
            const double centre = (double)(nu * ((long double)s.d2[0][0] + s.d2[1][0] + s.d2[2][0]) +
                                           vg * s.d2[q][0]);
            c.vcl[q] = D(-sides - (long double)(float)centre);
        }
    /* centres: FP64 the sums of the three axes'; FP32 minus the sums of the rounded sides,
     * rounded once (they differ where the spacings do) */
    auto in_T    = [](const long double v) { return (long double)(typename Pack<V>::T)(double)v; };
    long double ctr[3];
    for (int a = 0; a < 3; ++a) {
        ctr[a] = s.d2[a][0];
        if (FP32) {
            ctr[a] = 0;
            for (int k = 1; k <= 3; ++k)
                ctr[a] -= 2 * in_T(s.d2[a][k] / unit);
        }
    }
    const long double all = ctr[0] + ctr[1] + ctr[2];
    c.c_all = D(all);
    c.c_xy  = D(ctr[0] + ctr[1]);
    c.c_yz  = D(ctr[1] + ctr[2]);
    c.c_xz  = D(ctr[0] + ctr[2]);
    c.d2c[0] = D(FP32 ? all - in_T(ctr[1] + ctr[2]) : ctr[0]);
    c.d2c[1] = D(FP32 ? all - in_T(ctr[0] + ctr[2]) : ctr[1]);
    c.d2c[2] = D(FP32 ? all - in_T(ctr[0] + ctr[1]) : ctr[2]);
    c.nim          = D(-im * unit);
    c.m23          = D(-2.0L / 3);
    c.two          = D(2);
    c.one_half     = D(0.5);
    c.nu           = D(nu);
    c.inv_cp       = D(p.inv_cp);
    c.ncs2         = D(-p.cs2_sound);
    c.gicp         = D(p.gamma_inv_cp);
    c.gm1          = D(p.gamma_m1);
    c.gicp_l       = D(p.gamma_inv_cp * kr * unit);
    c.gm1_l        = D(p.gamma_m1 * kr * unit);
    c.gm1_lnrho0   = D(-(long double)p.gamma_m1 * p.lnrho0);
    c.inv_exp_lnT0 = D(by_T);
    c.eta          = D(p.eta * unit);
    c.eta_mu0      = D(p.eta_mu0 * rest);
    c.zeta         = D(p.zeta * rest);
    c.K            = D(p.K);
    return c;
}

/* ---- tensor memory: columns (32-bit words, two per value) of a thread's lane ---- */
template <int N>
struct TWords { /* N values */
    uint32_t w[2 * N];
    template <typename V>
    __device__ __forceinline__ void set(const int i, const V v)
    {
        to_words(v, w + 2 * i);
    }
    template <typename V>
    __device__ __forceinline__ V get(const int i) const
    {
        V v;
        from_words(w + 2 * i, v);
        return v;
    }
    __device__ __forceinline__ void store(const uint32_t a) const { tmem::st_n<2 * N>(a, w); }
    __device__ __forceinline__ void load(const uint32_t a) { tmem::ld_n<2 * N>(a, w); }
    __device__ __forceinline__ void tie()
    {
#pragma unroll
        for (int i = 0; i < 2 * N; ++i)
            asm volatile("" : "+r"(w[i]));
    }
};

/* the record of a plane: hydro values, magnetic values */
enum {
    H_C   = 0,            /* component c at H_C + 3c: d/dx, d/dy, viscous force in the plane */
    H_SX  = H_C + 9,      /* lnrho: d/dx, d/dy, Laplacian without its z sides */
    H_SY,
    H_SL,
    M_SX,                 /* entropy, as lnrho */
    M_SY,
    M_SL,
    M_L0,                 /* lap A_c in the plane (centres: x, y and for c < 2 also z), and for */
    M_Q0,                 /* c < 2 j_c without its z sides and mixed sums */
    M_L1,
    M_Q1,
    M_BZ,
    M_L2,
    M_DXAZ,
    M_DYAZ,
    REC_N
};
constexpr int REC_MN = REC_N - M_SX; /* the magnetic group's part */
constexpr int HX_N = 7;               /* exchange: grad lnrho, lap lnrho, 2 S:S, div u, exp(-lnrho) */
constexpr int MX_N = 10; /* grad s, j, B, exp(gamma s/cp + (gamma-1)(lnrho - lnrho0)) */

constexpr uint32_t REC_SLOTS = 5, Q_SLOTS = 8;
constexpr uint32_t ACC_W   = 2 * 6;            /* mixed sums of a plane: three per group */
constexpr uint32_t ZQ_W    = 2 * 4;            /* one plane's four values */
constexpr uint32_t ZQ_G    = Q_SLOTS * ZQ_W;   /* one group's queue */
constexpr uint32_t XCH_W   = 2 * (HX_N + MX_N);
constexpr uint32_t TM_COLS = 512;
/* UPWD: the hydro record also has the in-plane upwinding terms |ux| d_x + |uy| d_y
 * of lnrho, ux, uy, uz behind the values above */
template <bool UPWD>
struct Tm {
    static constexpr int HN         = M_SX + (UPWD ? 4 : 0); /* the hydro group's part */
    static constexpr uint32_t REC_W = 2 * (HN + REC_MN);
    static constexpr uint32_t ACC0  = REC_SLOTS * REC_W;
    static constexpr uint32_t ZQ0   = ACC0 + 2 * ACC_W;
    static constexpr uint32_t XCH0  = ZQ0 + 2 * ZQ_G;
    static_assert(XCH0 + 2 * XCH_W <= TM_COLS, "tensor-memory columns");
};

/* ---- shared memory ---- */

/* the value at offset (dx, dy) of this thread's cell(s); p points at the field's
 * value at the (first) cell */
template <typename V>
struct Tap {
    typedef typename Pack<V>::T T;
    const T* p;
    __device__ __forceinline__ V operator()(const int dx, const int dy) const
    {
        const T* a = p + dy * SplitTile<V>::HXP + dx;
        if constexpr (Pack<V>::N == 2)
            return f2(a[0], a[WARPS_Y * SplitTile<V>::HXP]);
        else
            return a[0];
    }
};

template <typename V>
__device__ __forceinline__ void
diffs_x(const Tap<V>& t, V d[3])
{
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        d[k - 1] = t(k, 0) - t(-k, 0);
}
template <typename V>
__device__ __forceinline__ void
diffs_y(const Tap<V>& t, V d[3])
{
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        d[k - 1] = t(0, k) - t(0, -k);
}
/* differences and sums along x and y */
template <typename V>
__device__ __forceinline__ void
taps_xy(const Tap<V>& t, V dx[3], V sx[3], V dy[3], V sy[3])
{
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        const V a = t(k, 0), b = t(-k, 0), c = t(0, k), d = t(0, -k);
        dx[k - 1] = a - b;
        sx[k - 1] = a + b;
        dy[k - 1] = c - d;
        sy[k - 1] = c + d;
    }
}
template <typename V>
__device__ __forceinline__ V
dot3(const V a[3], const V c[3])
{
    return vfma(c[2], a[2], vfma(c[1], a[1], c[0] * a[0]));
}
/* r + sum_k c_k a_k */
template <typename V>
__device__ __forceinline__ V
dot3p(const V a[3], const V c[3], const V r)
{
    return vfma(c[2], a[2], vfma(c[1], a[1], vfma(c[0], a[0], r)));
}
/* r + sum_k e_k (f(+k,+k) + f(-k,-k) - f(+k,-k) - f(-k,+k)) in the plane */
template <typename V>
__device__ __forceinline__ V
dxy(const Tap<V>& t, const V e[3], V r)
{
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        r = vfma(e[k - 1], (t(k, k) + t(-k, -k)) - (t(k, -k) + t(-k, k)), r);
    return r;
}

/* One plane's contribution to the running sums of a mixed term: plane L adds
 * +e_k d_k to plane L - k and -e_k d_k to plane L + k.  acc[j] holds plane
 * L - 3 + j; the finished sum of plane L - 3 is returned and the others move on
 * by one plane as they are added to (no register copies but one).  FIRST: the
 * term's first contribution of the plane (moves on); else it adds in place. */
template <typename V>
__device__ __forceinline__ V
mixed_first(V acc[6], const V d[3], const V e[3], const V ne[3])
{
    const V done = vfma(e[2], d[2], acc[0]);
    acc[0]       = vfma(e[1], d[1], acc[1]);
    acc[1]       = vfma(e[0], d[0], acc[2]);
    acc[2]       = acc[3];
    acc[3]       = vfma(ne[0], d[0], acc[4]);
    acc[4]       = vfma(ne[1], d[1], acc[5]);
    acc[5]       = ne[2] * d[2];
    return done;
}
template <typename V>
__device__ __forceinline__ V
mixed_second(V acc[6], const V done, const V d[3], const V e[3], const V ne[3])
{
    acc[0] = vfma(e[1], d[1], acc[0]);
    acc[1] = vfma(e[0], d[0], acc[1]);
    acc[3] = vfma(ne[0], d[0], acc[3]);
    acc[4] = vfma(ne[1], d[1], acc[4]);
    acc[5] = vfma(ne[2], d[2], acc[5]);
    return vfma(e[2], d[2], done);
}

template <typename V>
__device__ __forceinline__ V
viscous_centre(const SplitCoef<V>& c, const int q, const V v)
{
    if constexpr (Pack<V>::N == 2)
        return vfma(c.vc[q], v, c.vcl[q] * v);
    else
        return c.vc[q] * v;
}

/* everything a role needs that does not change with the plane */
struct Chunk {
    int z0, z1, pfirst, plast;
    uint32_t tl; /* tensor-memory lane address */
    uint64_t *rfull, *pfull; /* ring slots loaded: planes, previous state */
};

/* The end of an interval: this thread's tensor-memory accesses are ordered
 * before those that any thread makes after it, and the shared-memory slots read
 * in it are free (the memory clobbers of the barrier and of the fences beside it
 * keep the reads of a slot before its refill).  Called by a whole converged warp:
 * the tensor-memory wait is warp-collective (.sync.aligned), as are the loads and
 * stores, so a __syncwarp() stands between each of them and any code before it
 * that single threads branch around. */
__device__ __forceinline__ void
interval_end()
{
    tmem::wait_st();
    tmem::fence_before_sync();
    asm volatile("bar.sync 0;" ::: "memory");
    tmem::fence_after_sync();
}

/* The previous state of plane p of the tile, into slot (p - z0) mod PRING (by
 * one thread): FP64 the value that the out-buffer holds; FP32 the compensation
 * words of the in-buffer and, after substep 0, both words of the out-buffer. */
template <typename V>
__device__ __forceinline__ void
load_prev(const SplitMaps* maps, const Chunk& ch, typename Pack<V>::T* smem, const int p,
          const bool use_prev, const int x0, const int y0)
{
    typedef SplitTile<V> S;
    if (p < ch.z0 || p >= ch.z1 || !(use_prev || Pack<V>::N == 2))
        return;
    const int sl       = (p - ch.z0) % S::PRING;
    unsigned char* dst = reinterpret_cast<unsigned char*>(smem) + S::P_OFF + sl * S::PSLOT_BYTES;
    uint64_t* bar      = &ch.pfull[sl];
    const int x = x0 + S::PX0, y = y0 + NGHOST, z = p + NGHOST;
    if (Pack<V>::N == 1) {
        mbar_arrive_expect_tx(bar, S::PARR_BYTES);
        tma_load_plane(dst, &maps->prev, bar, x, y, z);
    }
    else {
        mbar_arrive_expect_tx(bar, use_prev ? 3 * S::PARR_BYTES : S::PARR_BYTES);
        tma_load_plane(dst, &maps->lo, bar, x, y, z);
        if (use_prev) {
            tma_load_plane(dst + S::PARR_BYTES, &maps->prev, bar, x, y, z);
            tma_load_plane(dst + 2 * S::PARR_BYTES, &maps->prev_lo, bar, x, y, z);
        }
    }
}

/* ---------------------------------------------------------------------------
 * The in-plane roles.
 * ------------------------------------------------------------------------- */
template <typename V, int GROUP, bool UPWD>
__device__ __forceinline__ bool
inplane_role(const SplitMaps* maps, const SplitCoef<V>& c, const Chunk& ch,
             typename Pack<V>::T* smem, const int cell_off, const bool loader, const bool use_prev,
             const int x0, const int y0, const bool skip_last)
{
    typedef SplitTile<V> S;
    constexpr int QS = GROUP == 0 ? VTXBUF_LNRHO : VTXBUF_ENTROPY;
    constexpr int Q0 = GROUP == 0 ? VTXBUF_UUX : VTXBUF_AX;
    const long long wlim = skip_last ? kDebugWaitLimit : kWaitLimit;
    bool ok = true;
    V acc[3][6];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int j = 0; j < 6; ++j)
            acc[a][j] = Pack<V>::dup(0.0);
    int slot = 0;
    unsigned phase = 0;
    typedef Tm<UPWD> TM;
    uint32_t rec = ch.tl + (GROUP == 0 ? 0u : 2u * TM::HN); /* record slot, stepped with the plane */
    uint32_t r5  = 0;
    /* (the first plane takes record slot 0: the solve roles count alike) */
#pragma unroll 1
    for (int L = ch.pfirst; L <= ch.plast; ++L) {
        if (ok)
            ok = mbar_wait_bounded(&ch.rfull[slot], phase, wlim);
        __syncwarp();
        const typename Pack<V>::T* pl = smem + slot * S::SLOT + cell_off;
        const Tap<V> ts{pl + QS * S::PLANE};
        const Tap<V> t0{pl + Q0 * S::PLANE}, t1{pl + (Q0 + 1) * S::PLANE},
            t2{pl + (Q0 + 2) * S::PLANE};
        const V vs = ts(0, 0), v0 = t0(0, 0), v1 = t1(0, 0), v2 = t2(0, 0);
        const V* e1 = GROUP == 0 ? c.vm[1] : c.mm[1];
        const V* e2 = GROUP == 0 ? c.vm[2] : c.mm[2];
        const V* n1 = GROUP == 0 ? c.vmn[0] : c.mmn[0];
        const V* n2 = GROUP == 0 ? c.vmn[1] : c.mmn[1];
        TWords<3> fin; /* the finished mixed sums of plane L - 3 */
        if (L >= ch.z0 && L < ch.z1) {
            V dx[3], sx[3], dy[3], sy[3];
            if constexpr (GROUP == 0) {
                TWords<TM::HN> r;
                [[maybe_unused]] const V au = vabs(v0), av = vabs(v1);
                auto upwind = [&](const int q, const V v) {
                    if constexpr (UPWD)
                        r.set(M_SX + q, vfma(au, dot3p(sx, &c.up[0][1], c.up[0][0] * v),
                                             av * dot3p(sy, &c.up[1][1], c.up[1][0] * v)));
                };
                taps_xy(ts, dx, sx, dy, sy);
                upwind(0, vs);
                r.set(H_SX, dot3(dx, c.d1[0]));
                r.set(H_SY, dot3(dy, c.d1[1]));
                r.set(H_SL, dot3p(sy, c.d2[1], dot3p(sx, c.d2[0], c.c_all * vs)));
                taps_xy(t0, dx, sx, dy, sy);
                upwind(1, v0);
                const V done = mixed_first(acc[2], dx, e1, n1);
                r.set(H_C + 0, dot3(dx, c.d1[0]));
                r.set(H_C + 1, dot3(dy, c.d1[1]));
                r.set(H_C + 2, dxy(t1, c.vm[0], dot3p(sy, c.vn[1], dot3p(sx, c.vd[0], viscous_centre(c, 0, v0)))));
                taps_xy(t1, dx, sx, dy, sy);
                upwind(2, v1);
                fin.set(2, mixed_second(acc[2], done, dy, e2, n2));
                r.set(H_C + 3, dot3(dx, c.d1[0]));
                r.set(H_C + 4, dot3(dy, c.d1[1]));
                r.set(H_C + 5, dxy(t0, c.vm[0], dot3p(sy, c.vd[1], dot3p(sx, c.vn[0], viscous_centre(c, 1, v1)))));
                taps_xy(t2, dx, sx, dy, sy);
                upwind(3, v2);
                fin.set(0, mixed_first(acc[0], dx, e1, n1));
                fin.set(1, mixed_first(acc[1], dy, e2, n2));
                r.set(H_C + 6, dot3(dx, c.d1[0]));
                r.set(H_C + 7, dot3(dy, c.d1[1]));
                r.set(H_C + 8, dot3p(sy, c.vn[1], dot3p(sx, c.vn[0], viscous_centre(c, 2, v2))));
                __syncwarp();
                r.store(rec);
            }
            else {
                TWords<REC_MN> r;
                auto set = [&](const int i, const V v) { r.set(i - M_SX, v); };
                taps_xy(ts, dx, sx, dy, sy);
                set(M_SX, dot3(dx, c.d1[0]));
                set(M_SY, dot3(dy, c.d1[1]));
                set(M_SL, dot3p(sy, c.d2[1], dot3p(sx, c.d2[0], c.c_all * vs)));
                taps_xy(t0, dx, sx, dy, sy);
                const V done = mixed_first(acc[2], dx, e1, n1);
                const V dyAx = dot3(dy, c.d1[1]);
                {
                    const V Y = dot3p(sy, c.d2[1], c.c_yz * v0);
                    set(M_L0, dot3p(sx, c.d2[0], vfma(c.d2c[0], v0, Y)));
                    set(M_Q0, dxy(t1, c.mm[0], c.nim * Y));
                }
                taps_xy(t1, dx, sx, dy, sy);
                fin.set(2, mixed_second(acc[2], done, dy, e2, n2));
                {
                    const V X = dot3p(sx, c.d2[0], c.c_xz * v1);
                    set(M_L1, dot3p(sy, c.d2[1], vfma(c.d2c[1], v1, X)));
                    set(M_Q1, dxy(t0, c.mm[0], c.nim * X));
                }
                set(M_BZ, dot3(dx, c.d1[0]) - dyAx);
                taps_xy(t2, dx, sx, dy, sy);
                fin.set(0, mixed_first(acc[0], dx, e1, n1));
                fin.set(1, mixed_first(acc[1], dy, e2, n2));
                set(M_L2, dot3p(sy, c.d2[1], dot3p(sx, c.d2[0], c.c_xy * v2)));
                set(M_DXAZ, dot3(dx, c.d1[0]));
                set(M_DYAZ, dot3(dy, c.d1[1]));
                __syncwarp();
                r.store(rec);
            }
        }
        else {
            /* a halo plane only feeds the mixed sums and the z queue */
            V d[3], e[3];
            diffs_x(t0, d);
            const V done = mixed_first(acc[2], d, e1, n1);
            diffs_y(t1, e);
            fin.set(2, mixed_second(acc[2], done, e, e2, n2));
            diffs_x(t2, d);
            fin.set(0, mixed_first(acc[0], d, e1, n1));
            diffs_y(t2, e);
            fin.set(1, mixed_first(acc[1], e, e2, n2));
            __syncwarp();
        }
        fin.store(ch.tl + TM::ACC0 + (uint32_t)((L - NGHOST) & 1) * ACC_W + GROUP * 6u);
        {
            TWords<4> q;
            q.set(0, vs);
            q.set(1, v0);
            q.set(2, v1);
            q.set(3, v2);
            q.store(ch.tl + TM::ZQ0 + GROUP * ZQ_G + (uint32_t)(L & 7) * ZQ_W);
        }
        interval_end();
        if (loader) {
            /* plane L is read: its slot takes plane L + RING; the solve of plane
             * L - 5 is done: its previous-state slot takes that of plane L - 5 + PRING */
            const int next = L + S::RING;
            if (next <= ch.plast && !(skip_last && next == ch.plast)) {
                mbar_arrive_expect_tx(&ch.rfull[slot], S::SLOT_BYTES);
                tma_load_plane(smem + slot * S::SLOT, &maps->plane, &ch.rfull[slot], x0, y0,
                               next + NGHOST);
            }
            if (L - 5 >= ch.z0)
                load_prev<V>(maps, ch, smem, L - 5 + S::PRING, use_prev, x0, y0);
        }
        if (++slot == S::RING) {
            slot = 0;
            phase ^= 1;
        }
        rec = ++r5 == REC_SLOTS ? (r5 = 0, rec - (REC_SLOTS - 1) * TM::REC_W) : rec + TM::REC_W;
    }
    __syncwarp();
    interval_end(); /* the last solve interval's exchange */
    return ok;
}

/* ---------------------------------------------------------------------------
 * The solve roles.
 * ------------------------------------------------------------------------- */

/* window of one field: d/dz and the second-derivative sides from planes p-3 .. p+3 */
template <typename V>
__device__ __forceinline__ void
z_derivs(const TWords<4> w[7], const int i, const V d1[3], const V d2[3], V& g, V& s)
{
    const V m3 = w[0].template get<V>(i), m2 = w[1].template get<V>(i), m1 = w[2].template get<V>(i);
    const V p1 = w[4].template get<V>(i), p2 = w[5].template get<V>(i), p3 = w[6].template get<V>(i);
    g = vfma(d1[2], p3 - m3, vfma(d1[1], p2 - m2, d1[0] * (p1 - m1)));
    s = vfma(d2[2], p3 + m3, vfma(d2[1], p2 + m2, d2[0] * (p1 + m1)));
}

/* the upwinding derivative along z */
template <typename V>
__device__ __forceinline__ V
z_upwind(const TWords<4> w[7], const int i, const V u[4])
{
    V r = u[0] * w[3].template get<V>(i);
#pragma unroll
    for (int k = 1; k <= 3; ++k)
        r = vfma(u[k], w[3 + k].template get<V>(i) + w[3 - k].template get<V>(i), r);
    return r;
}

template <typename V>
struct RkV {
    V dt, beta, ab;
};

/* output arrays of a role's four fields */
template <typename T>
struct RoleFields {
    T* out[4];
    T* outl[4];
};

/* The single-pass 2N update (rk_update, rk_update_comp) of field k and its
 * store.  p: this thread's cell in the first field of the role in the
 * previous-state slot. */
template <bool PREV>
__device__ __forceinline__ void
update_store(const RoleFields<double>& f, const int k, const long long i0, const bool a0,
             const double val, const double prev, const double rate, const RkV<double>& rk)
{
    double upd = rk.dt * rate;
    if (PREV)
        upd = fma(rk.ab, val - prev, upd);
    const double o = fma(rk.beta, upd, val);
    if (a0)
        f.out[k][i0] = o;
}
template <bool PREV>
__device__ __forceinline__ void
update_store(const RoleFields<double>& f, const int k, const long long i0, const long long,
             const bool a0, const bool, const double val, const double* p, const double rate,
             const RkV<double>& rk)
{
    update_store<PREV>(f, k, i0, a0, val, PREV ? p[k * SplitTile<double>::PFLD] : 0.0, rate, rk);
}
template <bool PREV>
__device__ __forceinline__ void
update_store(const RoleFields<float>& f, const int k, const long long i0, const long long i1,
             const bool a0, const bool a1, const F2 h, const float* p, const F2 rate,
             const RkV<F2>& rk)
{
    typedef SplitTile<F2> S;
    constexpr int ARR = AC_NF * S::PFLD;
    auto at = [&](const int arr) {
        const float* q = p + arr * ARR + k * S::PFLD;
        return f2(q[0], q[WARPS_Y * S::PXW]);
    };
    const F2 lo = at(0);
    F2 upd      = rk.dt * rate;
    if (PREV)
        upd = vfma(rk.ab, (h - at(1)) + (lo - at(2)), upd);
    /* (scalar products: a packed product may be fused with the sums below, and the
     * increment would then not be the FP32 value that rk_update_comp adds) */
    const F2 inc = f2(__fmul_rn(lo_of(rk.beta), lo_of(upd)), __fmul_rn(hi_of(rk.beta), hi_of(upd)));
    const F2 s   = h + inc;
    const F2 bb  = s - h;
    const F2 e   = (h - (s - bb)) + (inc - bb);
    const F2 l2  = lo + e;
    const F2 oh  = s + l2;
    const F2 ol  = l2 - (oh - s);
    if (a0) {
        f.out[k][i0]  = lo_of(oh);
        f.outl[k][i0] = lo_of(ol);
    }
    if (a1) {
        f.out[k][i1]  = hi_of(oh);
        f.outl[k][i1] = hi_of(ol);
    }
}

__device__ __forceinline__ void
cfl_cells(const double u2, const double b2, const double irho, const double cs2, double m[3],
          const bool a0, const bool, const bool with_sum)
{
    if (a0)
        cfl_accumulate(u2, b2, irho, cs2, m, with_sum);
}
__device__ __forceinline__ void
cfl_cells(const F2 u2, const F2 b2, const F2 irho, const float cs2, float m[3], const bool a0,
          const bool a1, const bool with_sum)
{
    if (a0)
        cfl_accumulate(lo_of(u2), lo_of(b2), lo_of(irho), cs2, m, with_sum);
    if (a1)
        cfl_accumulate(hi_of(u2), hi_of(b2), hi_of(irho), cs2, m, with_sum);
}

/* Planes loaded by the threads of the solve roles, for FP64 meshes whose rows are
 * no multiple of 16 bytes (nx odd), which TMA does not take: 8-byte asynchronous
 * copies, whose completion arrives on the slot's mbarrier as TMA's does. */
struct PlaneCopier {
    static constexpr int N = 2; /* elements of a field's plane per thread */
    typedef SplitTile<double> S;
    static_assert(S::PLANE <= N * 2 * STH, "a field's plane");
    int src[N]; /* offset in the plane, -1: none */
    int t;
    __device__ __forceinline__ void init(const Geom& g, const int t0, const int x0, const int y0)
    {
        t = t0;
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int e = t + n * 2 * STH;
            const int y = y0 + e / S::HXP, x = x0 + e % S::HXP;
            src[n] = e < S::PLANE && x < g.mx && y < g.my ? x + y * g.px : -1;
        }
    }
    /* plane L (interior z index) of all fields into slot sl; every thread of the
     * two roles calls it */
    __device__ __forceinline__ void copy(const Geom& g, const FieldsT<double>& f, const int L,
                                         double* smem, const int sl, uint64_t* bar) const
    {
        const long long off = (long long)(L + NGHOST) * g.pxy;
#pragma unroll
        for (int q = 0; q < AC_NF; ++q)
#pragma unroll
            for (int n = 0; n < N; ++n)
                if (src[n] >= 0)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                     smem_addr(smem + sl * S::SLOT + q * S::PLANE + t + n * 2 * STH)),
                                 "l"(f.in[q] + off + src[n])
                                 : "memory");
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar))
                     : "memory");
    }
};

template <typename V, int GROUP, bool PREV, bool UPWD, bool LDG>
__device__ __forceinline__ bool
solve_role(const Geom& g, const RoleFields<typename Pack<V>::T>& f, const SplitCoef<V>& c,
           const RkV<V>& rk, const Chunk& ch, const typename Pack<V>::T* prev, const int lx,
           const int ly, const int x, const int y, const bool do_cfl,
           const bool cfl_sum, const typename Pack<V>::T cs2, typename Pack<V>::T cm[3],
           const FieldsT<typename Pack<V>::T>& fields, typename Pack<V>::T* smem,
           const bool skip_last)
{
    typedef SplitTile<V> S;
    bool ok = true;
    [[maybe_unused]] PlaneCopier pc;
    /* plane L into its slot, if the chunk has it */
    auto copy_plane = [&](const int L) {
        if constexpr (LDG)
            if (L <= ch.plast && !(skip_last && L == ch.plast)) {
                const int sl = (L - ch.pfirst) % S::RING;
                pc.copy(g, fields, L, smem, sl, &ch.rfull[sl]);
            }
    };
    if constexpr (LDG) {
        pc.init(g, (GROUP * WARPS_Y + ly) * TX + lx, x - lx, y - ly);
        for (int i = 0; i < S::RING; ++i)
            copy_plane(ch.pfirst + i);
    }
    /* the stores of cells outside the mesh are skipped */
    const int y1  = y + WARPS_Y;
    const bool a0 = x < g.nx && y < g.ny, a1 = x < g.nx && y1 < g.ny;
    long long i0 = geom_idx(g, x + NGHOST, y + NGHOST, ch.z0 + NGHOST);
    long long i1 = geom_idx(g, x + NGHOST, y1 + NGHOST, ch.z0 + NGHOST);
    constexpr bool WAITS = !LDG && (PREV || Pack<V>::N == 2); /* previous-state slots are used */
    const typename Pack<V>::T* pcell =
        prev + 4 * GROUP * S::PFLD + ly * S::PXW + lx + (NGHOST - S::PX0);
    int pslot       = 0;
    unsigned pphase = 0;
    typedef Tm<UPWD> TM;
    const uint32_t zq = ch.tl + TM::ZQ0 + GROUP * ZQ_G;
    uint32_t r5 = 3 % REC_SLOTS; /* record slot of plane z0 = pfirst + 3 */
    uint32_t rec = ch.tl + r5 * TM::REC_W;
#pragma unroll 1
    for (int i = 0; i < 7; ++i) {
        __syncwarp(); /* after the copies, whose threads differ */
        interval_end();
        copy_plane(ch.pfirst + i + S::RING);
    }
#pragma unroll 1
    for (int p = ch.z0; p < ch.z1; ++p) {
        [[maybe_unused]] typename Pack<V>::T own[4] = {0, 0, 0, 0};
        if constexpr (LDG && PREV)
            if (a0) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    own[k] = f.out[k][i0];
            }
        __syncwarp(); /* after the loads above and the last plane's stores: cells in the mesh only */
        TWords<4> w[7];
#pragma unroll
        for (int k = 0; k < 7; ++k)
            w[k].load(zq + (uint32_t)((p - 3 + k) & 7) * ZQ_W);
        tmem::wait_ld();
#pragma unroll
        for (int k = 0; k < 7; ++k)
            w[k].tie();
        const uint32_t xslot = ch.tl + TM::XCH0 + (uint32_t)(p & 1) * XCH_W;
        const uint32_t aslot = ch.tl + TM::ACC0 + (uint32_t)(p & 1) * ACC_W + GROUP * 6u;
        V val[4], rr[4];
        if constexpr (GROUP == 0) {
            TWords<TM::HN> r;
            TWords<3> a;
            r.load(rec);
            a.load(aslot);
            const V lnrho = w[3].template get<V>(0), ux = w[3].template get<V>(1), uy = w[3].template get<V>(2),
                    uz = w[3].template get<V>(3);
            V gl[3], gz[3], s2[4];
            z_derivs(w, 0, c.d1[2], c.d2[2], gl[2], s2[0]);
            z_derivs(w, 1, c.d1[2], c.vn[2], gz[0], s2[1]);
            z_derivs(w, 2, c.d1[2], c.vn[2], gz[1], s2[2]);
            z_derivs(w, 3, c.d1[2], c.vd[2], gz[2], s2[3]);
            [[maybe_unused]] V upz[4];
            if constexpr (UPWD) {
                const V aw = vabs(uz);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    upz[q] = aw * z_upwind(w, q, c.up[2]);
            }
            tmem::wait_ld();
            r.tie();
            a.tie();
            if constexpr (UPWD) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    upz[q] = upz[q] + r.template get<V>(M_SX + q);
            }
            gl[0] = r.template get<V>(H_SX);
            gl[1] = r.template get<V>(H_SY);
            V gr[3][3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                gr[q][0] = r.template get<V>(H_C + 3 * q);
                gr[q][1] = r.template get<V>(H_C + 3 * q + 1);
                gr[q][2] = gz[q];
            }
            V visc[3];
#pragma unroll
            for (int q = 0; q < 3; ++q)
                visc[q] = (r.template get<V>(H_C + 3 * q + 2) + a.template get<V>(q)) + s2[1 + q];
            const V irho = ac_exp(-lnrho);
            /* strain: D_c = 2 S_cc, o = 2 S_ab */
            const V divu = gr[0][0] + gr[1][1] + gr[2][2];
            const V m    = c.m23 * divu;
            const V D0 = vfma(c.two, gr[0][0], m), D1 = vfma(c.two, gr[1][1], m),
                    D2 = vfma(c.two, gr[2][2], m);
            const V o01 = gr[0][1] + gr[1][0], o02 = gr[0][2] + gr[2][0], o12 = gr[1][2] + gr[2][1];
            {
                TWords<HX_N> xw;
                xw.set(0, gl[0]);
                xw.set(1, gl[1]);
                xw.set(2, gl[2]);
                xw.set(3, r.template get<V>(H_SL) + s2[0]);
                /* 2 S:S */
                xw.set(4, vfma(c.one_half, vfma(D2, D2, vfma(D1, D1, D0 * D0)),
                               vfma(o12, o12, vfma(o02, o02, o01 * o01))));
                xw.set(5, divu);
                xw.set(6, irho);
                __syncwarp();
                xw.store(xslot);
            }
            interval_end();
            copy_plane(p + 4 + S::RING);
            if (WAITS && ok)
                ok = mbar_wait_bounded(&ch.pfull[pslot], pphase);
            __syncwarp();
            TWords<MX_N> mx;
            mx.load(xslot + 2 * HX_N);
            const V nux = -ux, nuy = -uy, nuz = -uz;
            const V r0 = vfma(nux, gl[0], vfma(nuy, gl[1], vfma(nuz, gl[2], -divu)));
            V t[3];
            {
                /* 2 nu S grad lnrho */
                const V n0 = c.nu * gl[0], n1 = c.nu * gl[1], n2 = c.nu * gl[2];
                t[0] = vfma(D0, n0, vfma(o01, n1, vfma(o02, n2, visc[0])));
                t[1] = vfma(o01, n0, vfma(D1, n1, vfma(o12, n2, visc[1])));
                t[2] = vfma(o02, n0, vfma(o12, n1, vfma(D2, n2, visc[2])));
            }
#pragma unroll
            for (int q = 0; q < 3; ++q)
                t[q] = vfma(gr[q][0], nux, vfma(gr[q][1], nuy, vfma(gr[q][2], nuz, t[q])));
            tmem::wait_ld();
            mx.tie();
            const V ncs2 = c.ncs2 * mx.template get<V>(9);
            const V B0 = mx.template get<V>(6), B1 = mx.template get<V>(7), B2 = mx.template get<V>(8);
            const V j0 = mx.template get<V>(3), j1 = mx.template get<V>(4), j2 = mx.template get<V>(5);
            const V nB0 = -B0, nB1 = -B1, nB2 = -B2;
            const V jxB[3] = {vfma(j1, B2, j2 * nB1), vfma(j2, B0, j0 * nB2), vfma(j0, B1, j1 * nB0)};
            if constexpr (UPWD)
                rr[0] = r0 + upz[0];
            else
                rr[0] = r0;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const V pg = vfma(c.inv_cp, mx.template get<V>(q), gl[q]);
                rr[1 + q]  = vfma(irho, jxB[q], vfma(ncs2, pg, t[q]));
                if constexpr (UPWD)
                    rr[1 + q] = rr[1 + q] + upz[1 + q];
            }
            val[0] = lnrho;
            val[1] = ux;
            val[2] = uy;
            val[3] = uz;
        }
        else {
            TWords<REC_MN> r;
            TWords<3> a;
            TWords<4> uw; /* lnrho, ux, uy, uz */
            r.load(rec + 2 * TM::HN);
            a.load(aslot);
            uw.load(ch.tl + TM::ZQ0 + (uint32_t)(p & 7) * ZQ_W);
            const V ent = w[3].template get<V>(0);
            V gs[3], s2[4], dzAx, dzAy, unused;
            z_derivs(w, 0, c.d1[2], c.d2[2], gs[2], s2[0]);
            z_derivs(w, 1, c.d1[2], c.d2[2], dzAx, s2[1]);
            z_derivs(w, 2, c.d1[2], c.d2[2], dzAy, s2[2]);
            z_derivs(w, 3, c.d1[2], c.d2[2], unused, s2[3]);
            val[0] = w[3].template get<V>(1);
            val[1] = w[3].template get<V>(2);
            val[2] = w[3].template get<V>(3);
            val[3] = ent;
            tmem::wait_ld();
            r.tie();
            a.tie();
            uw.tie();
            auto R = [&](const int i) { return r.template get<V>(i - M_SX); };
            const V E = ac_exp(vfma(c.gicp, ent, vfma(c.gm1, uw.template get<V>(0), c.gm1_lnrho0)));
            gs[0] = R(M_SX);
            gs[1] = R(M_SY);
            const V laps = R(M_SL) + s2[0];
            const V B0 = R(M_DYAZ) - dzAy, B1 = dzAx - R(M_DXAZ), B2 = R(M_BZ);
            const V l2 = R(M_L2);
            const V j0 = vfma(c.nim, s2[1], R(M_Q0) + a.template get<V>(0));
            const V j1 = vfma(c.nim, s2[2], R(M_Q1) + a.template get<V>(1));
            const V j2 = vfma(c.nim, l2, a.template get<V>(2));
            const V lap0 = R(M_L0) + s2[1], lap1 = R(M_L1) + s2[2];
            const V lap2 = l2 + vfma(c.d2c[2], val[2], s2[3]);
            {
                TWords<MX_N> xw;
                xw.set(0, gs[0]);
                xw.set(1, gs[1]);
                xw.set(2, gs[2]);
                xw.set(3, j0);
                xw.set(4, j1);
                xw.set(5, j2);
                xw.set(6, B0);
                xw.set(7, B1);
                xw.set(8, B2);
                xw.set(9, E);
                __syncwarp();
                xw.store(xslot + 2 * HX_N);
            }
            interval_end();
            copy_plane(p + 4 + S::RING);
            if (WAITS && ok)
                ok = mbar_wait_bounded(&ch.pfull[pslot], pphase);
            __syncwarp();
            TWords<HX_N> hx;
            hx.load(xslot);
            const V ux = uw.template get<V>(1), uy = uw.template get<V>(2), uz = uw.template get<V>(3);
            const V nux = -ux, nuy = -uy, nuz = -uz;
            /* u x B + eta lap A */
            rr[0] = vfma(uy, B2, vfma(nuz, B1, c.eta * lap0));
            rr[1] = vfma(uz, B0, vfma(nux, B2, c.eta * lap1));
            rr[2] = vfma(ux, B1, vfma(nuy, B0, c.eta * lap2));
            const V inv_T = c.inv_exp_lnT0 * ac_rcp(E);
            const V jj    = vfma(j2, j2, vfma(j1, j1, j0 * j0));
            const V adv   = vfma(nux, gs[0], vfma(nuy, gs[1], nuz * gs[2]));
            tmem::wait_ld();
            hx.tie();
            const V irho = hx.template get<V>(6);
            if (do_cfl)
                cfl_cells(vfma(uz, uz, vfma(uy, uy, ux * ux)), vfma(B2, B2, vfma(B1, B1, B0 * B0)),
                          irho, cs2, cm, a0, a1, cfl_sum);
            const V divu = hx.template get<V>(5);
            const V H    = vfma(irho * c.eta_mu0, jj,
                                vfma(c.nu, hx.template get<V>(4), c.zeta * divu * divu));
            V heat = vfma(c.gicp_l, laps, c.gm1_l * hx.template get<V>(3));
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const V s = vfma(c.gicp, gs[q], c.gm1 * hx.template get<V>(q));
                heat      = vfma(s, s, heat);
            }
            rr[3] = vfma(inv_T, H, vfma(c.K * irho, heat, adv));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if constexpr (LDG)
                update_store<PREV>(f, k, i0, a0, val[k], own[k], rr[k], rk);
            else
                update_store<PREV>(f, k, i0, i1, a0, a1, val[k],
                                   pcell + pslot * (S::PSLOT_BYTES / sizeof(typename Pack<V>::T)),
                                   rr[k], rk);
        }
        if (WAITS && ++pslot == S::PRING) {
            pslot = 0;
            pphase ^= 1;
        }
        i0 += g.pxy;
        i1 += g.pxy;
        rec = ++r5 == REC_SLOTS ? (r5 = 0, rec - (REC_SLOTS - 1) * TM::REC_W) : rec + TM::REC_W;
    }
    if constexpr (LDG) /* no copy into this block's shared memory is left in flight */
        asm volatile("cp.async.wait_all;" ::: "memory");
    return ok;
}

/* Number of plane loads issued into ring slot sl for the planes pfirst .. plast
 * (plane p goes to slot (p - pfirst) mod RING), without plast when skipped. */
__device__ __forceinline__ int
loads_into(const int ring, const int sl, const int pfirst, const int plast, const bool skip_last)
{
    const int np = plast - pfirst + 1;
    int n        = sl < np ? (np - 1 - sl) / ring + 1 : 0;
    if (skip_last && (plast - pfirst) % ring == sl)
        --n;
    return n;
}

/* LDG: the planes by PlaneCopier instead of TMA */
template <typename V, bool PREV, bool UPWD, bool LDG>
__global__ void __launch_bounds__(THREADS, 1)
solve_split_kernel(const __grid_constant__ SplitMaps maps, const Geom g,
                   const FieldsT<typename Pack<V>::T> f, const __grid_constant__ SplitCoef<V> c,
                   const RkV<V> rk, const int zlo, const int zhi, const int zchunk, int* err,
                   unsigned long long* cfl, const bool cfl_sum, const typename Pack<V>::T cs2,
                   const bool skip_last)
{
    typedef SplitTile<V> S;
    typedef typename Pack<V>::T T;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* smem         = reinterpret_cast<T*>(smem_raw);
    T* red          = reinterpret_cast<T*>(smem_raw + S::RED_OFF);
    uint64_t* bars  = reinterpret_cast<uint64_t*>(smem_raw + S::BAR_OFF);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + S::NBARS);
    const int lx   = threadIdx.x;
    /* blockDim.x == 32: one warp per y; the shuffle tells the compiler that it is
     * uniform, so that tensor-memory addresses stay in uniform registers */
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.y, 0);
    const int ly   = warp & (WARPS_Y - 1);
    const int role = warp / WARPS_Y;
    const int tid  = warp * TX + lx;
    const int x0   = blockIdx.x * TX;
    const int y0   = blockIdx.y * S::TY;
    Chunk ch;
    ch.z0     = zlo + (int)blockIdx.z * zchunk;
    ch.z1     = min(ch.z0 + zchunk, zhi);
    ch.pfirst = ch.z0 - NGHOST;
    ch.plast  = ch.z1 - 1 + NGHOST;

    if (tid == 0) {
        for (int s = 0; s < S::NBARS; ++s)
            mbar_init(&bars[s], LDG && s < S::RING ? 2 * STH : 1);
        fence_barrier_init();
    }
    __syncwarp();
    if (warp == 1)
        tmem::alloc(tslot, TM_COLS);
    tmem::fence_before_sync();
    __syncthreads();
    tmem::fence_after_sync();
    /* the set-up above overlaps the end of the halo fill (ac_launch_overlapped) */
    ac_let_successor_start();
    ac_wait_predecessor();
    const uint32_t tbase = *tslot;
    ch.tl                = tmem::lane_base(tbase, warp);
    ch.rfull             = bars;
    ch.pfull             = bars + S::RING;
    if (!LDG && tid == 0) {
        const int pend = min(ch.plast, ch.pfirst + S::RING - 1);
        for (int q = ch.pfirst; q <= pend; ++q) {
            /* the fault-path test switch skips the load of the last plane */
            if (skip_last && q == ch.plast)
                continue;
            const int s = q - ch.pfirst;
            mbar_arrive_expect_tx(&bars[s], S::SLOT_BYTES);
            tma_load_plane(smem + (size_t)s * S::SLOT, &maps.plane, &bars[s], x0, y0, q + NGHOST);
        }
        /* (later planes' slots are refilled from the interval of plane z0 + 5 on) */
        for (int p = ch.z0; p < ch.z0 + S::PRING; ++p)
            load_prev<V>(&maps, ch, smem, p, PREV, x0, y0);
    }
    __syncwarp(); /* setmaxnreg is warp-collective */

    const int cell_off = (ly + NGHOST) * S::HXP + (lx + NGHOST);
    const int x = x0 + lx, y = y0 + ly;
    T cm[3] = {0, 0, 0};
    bool ok = true;
    T* prev = reinterpret_cast<T*>(smem_raw + S::P_OFF);
    if (role == 0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_INPLANE));
        ok = inplane_role<V, 0, UPWD>(&maps, c, ch, smem, cell_off, !LDG && ly == 0 && lx == 0, PREV, x0, y0,
                                skip_last);
    }
    else if (role == 1) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_INPLANE));
        ok = inplane_role<V, 1, UPWD>(&maps, c, ch, smem, cell_off, false, PREV, x0, y0, skip_last);
    }
    else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_SOLVE));
        RoleFields<T> rf;
        if (role == 2) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                rf.out[k]  = f.out[k];
                rf.outl[k] = f.out_lo[k];
            }
            ok = solve_role<V, 0, PREV, UPWD, LDG>(g, rf, c, rk, ch, prev, lx, ly, x, y, false, cfl_sum, cs2,
                                        cm, f, smem, skip_last);
        }
        else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                rf.out[k]  = f.out[4 + k];
                rf.outl[k] = f.out_lo[4 + k];
            }
            ok = solve_role<V, 1, PREV, UPWD, LDG>(g, rf, c, rk, ch, prev, lx, ly, x, y, cfl != nullptr, cfl_sum,
                                        cs2, cm, f, smem, skip_last);
        }
    }
    __syncthreads();
    if (cfl)
        cfl_commit(cm, red, cfl);
    if (!ok)
        *(volatile int*)err = 1; /* (may be host memory) */
    /* no copy into this block's shared memory is left in flight */
    if (!LDG && tid == 0) {
        drain_ring(bars, S::RING, [&](const int sl) {
            return loads_into(S::RING, sl, ch.pfirst, ch.plast, skip_last);
        });
        if (PREV || Pack<V>::N == 2)
            drain_ring(ch.pfull, S::PRING, [&](const int sl) {
                return loads_into(S::PRING, sl, ch.z0, ch.z1 - 1, false);
            });
    }
    /* every thread's tensor-memory accesses are complete before the columns are freed */
    __syncwarp();
    tmem::fence_before_sync();
    __syncthreads();
    tmem::fence_after_sync();
    if (warp == 1)
        tmem::dealloc(tbase, TM_COLS);
}

/* Planes per block: nz in c equal chunks, c with the least (waves of one block
 * per SM) x (intervals of a block: its planes, 6 halo planes and two of the
 * solve roles' lag); the longest chunks on a tie.  Small meshes so come out as
 * one wave of short chunks, large ones as few long ones. */
int
split_zchunk(const int tiles, const int nz, const int sms, long long* intervals = nullptr)
{
    int best       = nz;
    long long cost = 0;
    for (int c = 1; c <= nz; ++c) {
        const int zc           = (nz + c - 1) / c;
        const long long blocks = (long long)tiles * ((nz + zc - 1) / zc);
        const long long t      = (blocks + sms - 1) / sms * (zc + 2 * NGHOST + 2);
        if (cost == 0 || t < cost) {
            cost = t;
            best = zc;
        }
    }
    if (intervals)
        *intervals = cost;
    return best;
}

/* Whether the automatic choice takes this kernel with planes loaded by the threads (FP64,
 * nx odd) and not the plain kernel.  Both have the same tiles.  A block here takes about
 * 1.25 us an interval; the plain kernel, one plane a block and two blocks per SM, about
 * 4.3 us (6.2 with upwinding) for as many as fit the GPU: at its best where the mesh is
 * small or a few planes thin.  Per substep, plain / this: 33^3 12.5 / 15.6 us,
 * 125 x 13 x 9 6.3 / 10.5, 255 x 255 x 3 26 / 43, 65^3 47 / 52; 73^3 58 / 58,
 * 35 x 40 x 100 31 / 29, 103^3 183 / 123; this over plain with upwinding: 33^3 1.16,
 * 39^3 0.96, 49^3 0.85. */
bool
split_beats_plain(const Geom& g, const bool upwind)
{
    const int tiles = (g.nx + TX - 1) / TX * ((g.ny + WARPS_Y - 1) / WARPS_Y);
    long long intervals;
    split_zchunk(tiles, g.nz, AC_SMS, &intervals);
    return intervals <= (upwind ? 5.0 : 3.5) * tiles * g.nz / (2.0 * AC_SMS);
}

template <typename V, typename T>
cudaError_t
launch_split(const Geom& g, const SplitMaps& tm, const FieldsT<T>& f, const StencilCoef& sc,
             const PhysConst& pc, const RkCoef& rk, int* err, unsigned long long* cfl,
             cudaStream_t stream, unsigned long long* launches, const int sms,
             [[maybe_unused]] const bool threads_load, const bool overlap)
{
    typedef SplitTile<V> S;
    const int nzr = pc.zhi - pc.zlo;
    if (nzr <= 0)
        return cudaSuccess;
    const int bx = (g.nx + TX - 1) / TX, by = (g.ny + S::TY - 1) / S::TY;
    const int zc = split_zchunk(bx * by, nzr, sms);
    const dim3 bpg(bx, by, (nzr + zc - 1) / zc);
    const dim3 tpb(TX, ROLES * WARPS_Y, 1);
    const SplitCoef<V> c = make_coef<V>(sc, pc);
    RkV<V> r;
    r.dt   = Pack<V>::dup(rk.dt);
    r.beta = Pack<V>::dup(rk.beta);
    r.ab   = Pack<V>::dup(rk.ab);
    const bool sum = pc.cfl_sum != 0, skip = pc.debug_skip_load != 0;
    cudaError_t e = cudaSuccess;
    auto launch = [&](auto kernel) {
        e = ac_launch_overlapped(kernel, bpg, tpb, S::SMEM_BYTES, stream, overlap, tm, g, f, c, r,
                                 pc.zlo, pc.zhi, zc, err, cfl, sum, (T)pc.cs2_sound, skip);
    };
    auto pick = [&](auto ldg) {
        constexpr bool LDG = decltype(ldg)::value;
        if (pc.upwind)
            rk.step > 0 ? launch(solve_split_kernel<V, true, true, LDG>)
                        : launch(solve_split_kernel<V, false, true, LDG>);
        else
            rk.step > 0 ? launch(solve_split_kernel<V, true, false, LDG>)
                        : launch(solve_split_kernel<V, false, false, LDG>);
    };
    if constexpr (sizeof(T) == 8) {
        if (threads_load)
            pick(std::true_type{});
        else
            pick(std::false_type{});
    }
    else
        pick(std::false_type{});
    if (launches)
        ++*launches;
    return e;
}

template <typename V>
cudaError_t
init_split()
{
    std::vector<const void*> forms = {(const void*)solve_split_kernel<V, false, false, false>,
                                      (const void*)solve_split_kernel<V, true, false, false>,
                                      (const void*)solve_split_kernel<V, false, true, false>,
                                      (const void*)solve_split_kernel<V, true, true, false>};
    if constexpr (Pack<V>::N == 1)
        forms.insert(forms.end(), {(const void*)solve_split_kernel<V, false, false, true>,
                                   (const void*)solve_split_kernel<V, true, false, true>,
                                   (const void*)solve_split_kernel<V, false, true, true>,
                                   (const void*)solve_split_kernel<V, true, true, true>});
    for (const void* fn : forms) {
        cudaFuncAttributes a;
        cudaError_t e = cudaFuncGetAttributes(&a, fn);
        if (e != cudaSuccess)
            return e;
        /* setmaxnreg only moves registers that the block was launched with */
        if (a.numRegs * ROLES < 2 * (REGS_INPLANE + REGS_SOLVE))
            return cudaErrorInvalidConfiguration;
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SplitTile<V>::SMEM_BYTES);
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

} // namespace

bool
ac_make_split_maps(SplitBufferMaps* m, void* hi, float* lo, const Geom& g, const int precision)
{
    typedef SplitTile<double> D;
    typedef SplitTile<F2> F;
    /* FP64 rows of an odd number of values are no multiple of 16 bytes: no tensor
     * map, the threads load the planes.  125^3: 0.56 ms per step, the plain kernel
     * 0.90 (128^3 by TMA 0.46); which of the two is faster depends on the size. */
    m->threads_load = precision == 0 && (g.nx & 1) && g.nx >= TX && g.ny >= WARPS_Y;
    for (int upwind = 0; upwind < 2; ++upwind)
        m->automatic[upwind] = !m->threads_load || split_beats_plain(g, upwind != 0);
    if (m->threads_load)
        return true;
    if (!ac_tiled_supported(g, precision) || g.my < (precision == 0 ? D::HY : F::HY))
        return false;
    if (precision == 0)
        return ac_encode_field_map(&m->plane, hi, g, 0, D::HXP, D::HY) &&
               ac_encode_field_map(&m->tile, hi, g, 0, D::PXW, D::TY);
    return ac_encode_field_map(&m->plane, hi, g, 1, F::HXP, F::HY) &&
           ac_encode_field_map(&m->tile, hi, g, 1, F::PXW, F::TY) &&
           ac_encode_field_map(&m->tile_lo, lo, g, 1, F::PXW, F::TY);
}

/* Once per GPU and precision (function attributes are the GPU's). */
cudaError_t
ac_solve_split_init(const int precision)
{
    static std::atomic<unsigned long long> done[2]; /* bit: device id */
    int id        = 0;
    cudaError_t e = cudaGetDevice(&id);
    if (e != cudaSuccess)
        return e;
    const unsigned long long bit = id < 64 ? 1ull << id : 0;
    if (done[precision] & bit)
        return cudaSuccess;
    e = precision == 0 ? init_split<double>() : init_split<F2>();
    if (e == cudaSuccess)
        done[precision] |= bit;
    return e;
}

cudaError_t
ac_launch_solve_split64(const Geom& g, const SplitBufferMaps& in, const SplitBufferMaps& out, const Fields64& f,
                        const StencilCoef& sc, const PhysConst& pc, const RkCoef& rk, int* err,
                        unsigned long long* cfl, cudaStream_t stream, unsigned long long* launches,
                        const int sms, const bool overlap)
{
    return launch_split<double>(g, SplitMaps{in.plane, out.tile, out.tile_lo, in.tile_lo}, f, sc, pc,
                                rk, err, cfl, stream, launches, sms, in.threads_load, overlap);
}

cudaError_t
ac_launch_solve_split32(const Geom& g, const SplitBufferMaps& in, const SplitBufferMaps& out, const Fields32& f,
                        const StencilCoef& sc, const PhysConst& pc, const RkCoef& rk, int* err,
                        unsigned long long* cfl, cudaStream_t stream, unsigned long long* launches,
                        const int sms, const bool overlap)
{
    return launch_split<F2>(g, SplitMaps{in.plane, out.tile, out.tile_lo, in.tile_lo}, f, sc, pc,
                                rk, err, cfl, stream, launches, sms, in.threads_load, overlap);
}
