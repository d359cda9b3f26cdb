// The 2D node of the fast build: streaming interpolation order, macroscopic
// fields and collision, with the rounding of every operation written out.
//
// Included by lbm_kernels.cu inside namespace lbm::LBM_NS (fast build only).
// The direct-load, resident, march and batch kernels all run these functions,
// in kernels that advance one time level or several; with explicit rounding
// (no contraction left to the compiler) a node's new state is the same bits in
// every one of them, so a run does not depend on how its iterations were
// grouped into launches.

__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// The stencil of a node along an axis of n nodes is the window of three nodes
// win_lo .. win_lo + 2: centred inside, one-sided at both ends (2B:246-296).
__device__ __forceinline__ int win_lo(int i, int n) { return i == 0 ? 0 : (i == n - 1 ? n - 3 : i - 1); }

// The six weights of node i (both shift signs) in window order, from the table
// order (a, m, b): (1, 0, 2) at the first node, (n-2, n-1, n-3) at the last.
template <class C, class W>
__device__ __forceinline__ void window_weights(const W *t, int i, int n, C wp[3], C wm[3])
{
    const C a0 = C(t[0]), a1 = C(t[1]), a2 = C(t[2]), b0 = C(t[3]), b1 = C(t[4]), b2 = C(t[5]);
    if (i == 0) {
        wp[0] = a1; wp[1] = a0; wp[2] = a2;
        wm[0] = b1; wm[1] = b0; wm[2] = b2;
    } else if (i == n - 1) {
        wp[0] = a2; wp[1] = a0; wp[2] = a1;
        wm[0] = b2; wm[1] = b0; wm[2] = b1;
    } else {
        wp[0] = a0; wp[1] = a1; wp[2] = a2;
        wm[0] = b0; wm[1] = b1; wm[2] = b2;
    }
}

// three-point interpolation in window order; lin2 + fma_(w2, ., .) is the same
// sum split at its last term (march kernels form the first two terms early)
template <class C>
__device__ __forceinline__ C lin2(C w0, C w1, C a, C m) { return fma_(w1, m, mul_(w0, a)); }
template <class C>
__device__ __forceinline__ C lin3(const C w[3], C a, C m, C b) { return fma_(w[2], b, lin2(w[0], w[1], a, m)); }

// the same with the operands in table order (a, m, b)
template <class C>
__device__ __forceinline__ C ip3(const C w[3], C a, C m, C b) { return fma_(w[2], b, fma_(w[1], m, mul_(w[0], a))); }

// and in an order that is the same from either end of the window
template <class C>
__device__ __forceinline__ C sym3(const C w[3], C a, C m, C b)
{
    return fma_(w[1], m, add_(mul_(w[0], a), mul_(w[2], b)));
}

// the collision's constants (relax_setup, lbm_internal.h) in the compute type
template <class C>
struct Relax {
    C Snu, Sq, sig, gbeta, dt, hdt, c6, c7;
};
template <class C>
__device__ __forceinline__ Relax<C> relax_of(const Geo &G)
{
    const double *r = G.relax;
    return {C(r[0]), C(r[1]), C(r[2]), C(r[3]), C(r[4]), C(r[5]), C(r[6]), C(r[7])};
}

// 1 / a for a density a (near 1): the hardware's approximation, then one step
// of the third-order Newton (Halley) iteration r (1 + e + e^2), e = 1 - a r,
// in FP64, one Newton step in FP32; within an ulp of the exact quotient.  No
// range checks: 3 dependent operations where a checked division branches.
__device__ __forceinline__ double rcp_(double a)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
    const double e = fma_(-a, r, 1.0);
    return fma_(r, fma_(e, e, e), r);
}
__device__ __forceinline__ float rcp_(float a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return fma_(r, fma_(-a, r, 1.0f), r);
}

// macro_u, macro_t (2M:726-753), collision_U (2M:431-520) and collision_T
// (2M:522-569) at one node: moments from sums and differences of opposite
// populations, momentum reused as rho u, the inverse transform grouped by
// opposite pairs (113 operations).  f, g: the streamed populations, F0: the
// force of the collision that produced them, Tc: the conduction profile (DEVT);
// DEV / DEVT: deviation form (FP32 storage), where m0 = rho - 1 and Tn = T - Tc.
// (A form with a shorter dependent chain, every population one multiply-add
// behind 1/rho, takes 125 operations and was 3 % slower in every kernel: the
// instructions a warp has to issue bound it, not the chain.)
template <class C, bool DEV, bool DEVT>
__device__ __forceinline__ void node2d(const C (&f)[9], const C (&g)[5], C F0, const Relax<C> &K, C Tc, C (&fp)[9],
                                       C (&gp)[5], C &Fy, C &rho, C &u, C &v, C &T)
{
    const C s13 = add_(f[1], f[3]), d13 = sub_(f[1], f[3]);
    const C s24 = add_(f[2], f[4]), d24 = sub_(f[2], f[4]);
    const C s57 = add_(f[5], f[7]), d57 = sub_(f[5], f[7]);
    const C s68 = add_(f[6], f[8]), d68 = sub_(f[6], f[8]);
    const C A = add_(s13, s24), D = add_(s57, s68);
    const C ex = sub_(d57, d68), ey = add_(d57, d68);
    const C m0 = add_(f[0], add_(A, D));
    const C m1 = fma_(C(-4.0), f[0], fma_(C(2.0), D, -A));
    const C m2 = fma_(C(4.0), f[0], fma_(C(-2.0), A, D));
    const C jx = add_(d13, ex), m4 = fma_(C(-2.0), d13, ex);
    const C jy = add_(d24, ey), m6 = fma_(C(-2.0), d24, ey);
    const C m7 = sub_(s13, s24), m8 = sub_(s57, s68);
    rho = DEV ? add_(C(1.0), m0) : m0;
    const C rinv = rcp_(rho);
    const C jyF = fma_(K.hdt, F0, jy);
    u = mul_(jx, rinv);
    v = mul_(jyF, rinv);
    const C g13 = add_(g[1], g[3]), g24 = add_(g[2], g[4]);
    const C n3 = add_(g13, g24);
    const C Tn = add_(g[0], n3);
    T = DEVT ? add_(Tc, Tn) : Tn;
    Fy = mul_(mul_(K.gbeta, T), rho);
    const C a = mul_(K.c7, Fy);
    const C va = mul_(v, a), ua = mul_(u, a);
    const C e1 = mul_(jx, u);
    const C es = fma_(jyF, v, e1), ed = fma_(-jyF, v, e1), uv = mul_(jx, v);
    const C es3 = mul_(C(3.0), es);
    const C p1 = fma_(C(3.0), va, fma_(-K.Snu, sub_(m1, fma_(C(-2.0), m0, es3)), m1));
    const C p2 = fma_(C(-3.0), va, fma_(-K.Snu, sub_(m2, sub_(m0, es3)), m2));
    const C p4 = fma_(-K.Sq, add_(m4, jx), m4);
    const C p5 = fma_(K.dt, Fy, jy);
    const C p6 = fma_(-K.c6, Fy, fma_(-K.Sq, add_(m6, jyF), m6));
    const C p7 = sub_(fma_(-K.Snu, sub_(m7, ed), m7), va);
    const C p8 = fma_(C(0.5), ua, fma_(-K.Snu, sub_(m8, uv), m8));
    const C t9 = mul_(m0, C(1.0 / 9.0));
    fp[0] = fma_(C(1.0 / 9.0), sub_(p2, p1), t9);
    const C ca = fma_(C(-1.0 / 18.0), p2, fma_(C(-1.0 / 36.0), p1, t9));
    const C cd = fma_(C(1.0 / 36.0), p2, fma_(C(1.0 / 18.0), p1, t9));
    const C cx = fma_(C(0.25), p7, ca), cy = fma_(C(-0.25), p7, ca);
    const C ox = sub_(jx, p4), oy = sub_(p5, p6);
    fp[1] = fma_(C(1.0 / 6.0), ox, cx);
    fp[3] = fma_(C(-1.0 / 6.0), ox, cx);
    fp[2] = fma_(C(1.0 / 6.0), oy, cy);
    fp[4] = fma_(C(-1.0 / 6.0), oy, cy);
    const C X = fma_(C(1.0 / 12.0), p4, mul_(C(1.0 / 6.0), jx));
    const C Y = fma_(C(1.0 / 12.0), p6, mul_(C(1.0 / 6.0), p5));
    const C dp = fma_(C(0.25), p8, cd), dm = fma_(C(-0.25), p8, cd);
    const C xy = add_(X, Y), xm = sub_(X, Y);
    fp[5] = add_(dp, xy);
    fp[7] = sub_(dp, xy);
    fp[8] = add_(dm, xm);
    fp[6] = sub_(dm, xm);
    const C n1 = sub_(g[1], g[3]), n2 = sub_(g[2], g[4]), n4 = sub_(g13, g24);
    const C q1 = fma_(-K.sig, fma_(-T, u, n1), n1);
    const C q2 = fma_(-K.sig, fma_(-T, v, n2), n2);
    const C q3 = fma_(C(-1.9), fma_(C(-0.5), Tn, n3), n3);
    const C q4 = fma_(C(-1.9), n4, n4);
    gp[0] = sub_(Tn, q3);
    const C b = mul_(C(0.25), q3);
    const C bx = fma_(C(0.25), q4, b), by = fma_(C(-0.25), q4, b);
    gp[1] = fma_(C(0.5), q1, bx);
    gp[3] = fma_(C(-0.5), q1, bx);
    gp[2] = fma_(C(0.5), q2, by);
    gp[4] = fma_(C(-0.5), q2, by);
}

// streaming's wall rules (bounceback_u 2B:731-768, bounceback_T 2B:770-801) at
// node (i, j): cen(q) is the post-collision population q of the node itself,
// planes 0..8 f, 9..13 g
template <class C, bool DEVT, class Cen>
__device__ __forceinline__ void walls2d(int i, int j, int nx, int ny, C Thot, C Tcold, C Tc, Cen cen, C (&f)[9],
                                        C (&g)[5])
{
    if (i == 0) {
        f[1] = cen(3); f[5] = cen(7); f[8] = cen(6);
        g[1] = fma_(C(0.25), DEVT ? sub_(Thot, Tc) : Thot, -cen(12));
    }
    if (i == nx - 1) {
        f[3] = cen(1); f[6] = cen(8); f[7] = cen(5);
        g[3] = fma_(C(0.25), DEVT ? sub_(Tcold, Tc) : Tcold, -cen(10));
    }
    if (j == ny - 1) {
        f[4] = cen(2); f[7] = cen(5); f[8] = cen(6);
        g[4] = cen(11);
    }
    if (j == 0) {
        f[2] = cen(4); f[5] = cen(7); f[6] = cen(8);
        g[2] = cen(13);
    }
}
