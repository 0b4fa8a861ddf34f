// Per-cell ideal-GRMHD physics for the sm_100a kernels: metric algebra, fluid
// state, fluxes and fast speeds, PPM reconstruction, geometric source and the
// primitive-variable inversion chain. Templated on the arithmetic type so the
// mixed-precision step can run reconstruction/flux/EMF in float.
//
// Expression shapes follow the reference device code so that a build without
// FMA contraction reproduces it to the last bit (apart from pow(), whose CUDA
// and C-library roundings may differ by one ulp):
//   lower/raise                    GPU_metric.h:3-34
//   gamma/ucon/bcon/get_state      GPU_phys_mhd.h:672-761
//   primtoflux (+ fast speeds)     GPU_phys_mhd.h:432-628
//   calc_entropy                   GPU_phys_mhd.h:631-670
//   para (PPM, MC-2 slopes)        GPU_interp.h:60-111
//   source                         GPU_phys_mhd.h:34-175
//   Utoprim_2d + Noble Newton      GPU_utoprim_2d.h
//   Utoprim_1dvsq2fix1             GPU_utoprim_1dvsq2fix1.h
//   Utoprim_1dfix1                 GPU_utoprim_1dfix1.h
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include <type_traits>

#include "hamr_pow.cuh"

namespace hamr {

enum { RHO = 0, UU = 1, U1 = 2, U2 = 3, U3 = 4, B1 = 5, B2 = 6, B3 = 7, KTOT = 8, NPR = 9 };
enum { FACE1 = 0, FACE2 = 1, CORN = 2, CENT = 3, FACE3 = 4 };

constexpr double SMALL_D = 1.e-20;
constexpr double NEWT_TOL = 1.0e-10;
constexpr double MIN_NEWT_TOL = 1.0e-10;
constexpr int MAX_NEWT_ITER = 30;
constexpr int EXTRA_NEWT_ITER = 2;
constexpr double W_TOO_BIG = 1.e20;
constexpr double UTSQ_TOO_BIG = 1.e20;
constexpr double FAIL_VAL = 1.e30;

// The strict build (HAMR_STRICT, compiled without contraction) keeps the
// reference's operation order and roundings, which pins the arithmetic to the
// reference bit for bit; the production build may use any form of the same
// formulas that is as accurate. Code that differs says so with this flag.
#ifdef HAMR_STRICT
constexpr bool STRICT = true;
#else
constexpr bool STRICT = false;
#endif

// a b + c as one fused operation, and a b on its own, in the production build:
// whatever the compiler would contract where it inlines a formula, kernels that
// share it agree to the last bit (a block alone and in an ensemble). The strict
// build, compiled without contraction, has no choice to pin.
__device__ __forceinline__ double mad(double a, double b, double c) { return STRICT ? a * b + c : fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return STRICT ? a * b + c : fmaf(a, b, c); }
__device__ __forceinline__ double mul(double a, double b) { return STRICT ? a * b : __dmul_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return STRICT ? a * b : __fmul_rn(a, b); }

// Which of two forms a formula takes. The plain one, the reference's text with
// whatever the compiler contracts in it: the strict build (which contracts
// nothing), and the float step of the face-frame solvers (FT: HLLC, HLLD), whose
// contact speed is the cancelling root of a quadratic: there a changed last bit
// of an edge value or of an EMF moves u^2 by up to 1e-3 of its norm in a step, so
// their float arithmetic stays as it is, bit for bit (tests/test_gpu_mixed_face_frame.py).
// Everything else takes the shorter form, its fused operations spelled out.
template <typename T, bool FT>
constexpr bool plain_forms = STRICT || (FT && sizeof(T) == sizeof(float));

template <typename T>
struct Geo {
    T gcov[10], gcon[10], g;
    T lapse, rlapse;   // 1/sqrt(-g^tt) and its reciprocal, each rounded once
    T al;              // float only: the double lapse rounded once (lapse is the approximate
                       // root of the converted g^tt, which the face-frame solvers keep)
};

// the lapse of a filled Geo, computed in place (ucon_calc's operations)
template <typename T>
__device__ __forceinline__ void geo_lapse(Geo<T> &o);

template <typename T>
struct State {
    T ucon[4], ucov[4], bcon[4], bcov[4];
};

template <typename T> __device__ __forceinline__ T d_sqrt(T x);
template <> __device__ __forceinline__ double d_sqrt<double>(double x);   // below, with the reciprocal
template <> __device__ __forceinline__ float d_sqrt<float>(float x) { return sqrtf(x); }
template <typename T> __device__ __forceinline__ T d_pow(T x, T y);
template <> __device__ __forceinline__ double d_pow<double>(double x, double y) { return STRICT ? pow(x, y) : pow_tab(x, y); }
// float (the mixed step's entropy K = P rho^-gam of the face states, which
// only the entropy flux carries): the fast exp2(y log2 x) intrinsic, relative
// error a few 1e-6 at the atmosphere's densities against powf's ulp; measured
// on the 384 x 192 x 192 torus: the three float flux kernels 6.05 -> 5.59 ms
// per step, L1 of every field against FP64 after 1000 steps unchanged
template <> __device__ __forceinline__ float d_pow<float>(float x, float y) { return __powf(x, y); }

// Reciprocal and square root of the production build, by Newton's iteration
// (Goldschmidt's form for the root) from the hardware's approximations, which
// are good to about 2^-20: the reciprocal's one third-order step,
// r (1 + e + e^2) with e = 1 - b r, leaves e^3; the root's second-order step and
// final residual leave 2^-80; each then rounds within 0.6 ulp
// (tests/test_gpu_reciprocal.py). A zero, infinite or NaN operand, where the
// residuals are NaN, keeps the approximation's own exact answer. Three and
// seven FP64 operations without a branch: the step takes eleven of them per
// face and four per Newton iteration of the inversion, in dependent chains.
__device__ __forceinline__ bool not_finite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ double rcp_nr(double b) {
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(b));
    const double e = fma(-b, r0, 1.0);
    const double r = fma(r0, fma(e, e, e), r0);
    return not_finite(r) ? r0 : r;
}
// the same where a zero or infinite operand needs no answer (its NaN is caught
// by the caller)
__device__ __forceinline__ double rcp_nr_finite(double b) {
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(b));
    const double e = fma(-b, r0, 1.0);
    return fma(r0, fma(e, e, e), r0);
}
// sqrt(x) and 1/sqrt(x) of a positive normal x
__device__ __forceinline__ double sqrt_nr_pos(double x, double &rs) {
    double r0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(x));
    const double g = x * r0, h = 0.5 * r0;
    const double e = fma(-g, h, 0.5);
    const double g1 = fma(g, e, g), h1 = fma(h, e, h);
    const double s = fma(fma(-g1, g1, x), h1, g1);
    const double r1 = 2.0 * h1;
    rs = fma(r1, fma(-s, r1, 1.0), r1);   // not evaluated where it is not used
    return s;
}
__device__ __noinline__ double sqrt_rest(double x) { return sqrt(x); }
__device__ __forceinline__ bool pos_normal(double x) { return (unsigned)__double2hiint(x) - 0x00100000u < 0x7fe00000u; }
__device__ __forceinline__ double sqrt_nr(double x) {
    double rs;
    return pos_normal(x) ? sqrt_nr_pos(x, rs) : sqrt_rest(x);
}
template <> __device__ __forceinline__ double d_sqrt<double>(double x) { return STRICT ? sqrt(x) : sqrt_nr(x); }
// 1 / x in the arithmetic of the build
template <typename T> __device__ __forceinline__ T d_rcp(T x) {
    if constexpr (std::is_same<T, double>::value && !STRICT) return rcp_nr(x);
    else return T(1.0) / x;
}

template <typename T> __device__ __forceinline__ T d_fabs(T x) { return x < T(0) ? -x : x; }
__device__ __forceinline__ double d_fabs(double x) { return fabs(x); }   // an operand modifier, not a comparison
__device__ __forceinline__ float d_fabs(float x) { return fabsf(x); }
// x^(-1/2), correctly rounded in all but vanishingly rare near-midpoint cases,
// so that it agrees with a correctly rounded host pow(x, -0.5): the IEEE
// quotient 1/sqrt(x) (within about one ulp) takes one Newton step
// y + y (1 - x y^2) / 2 whose residual is formed exactly with fused
// multiply-adds (y^2 = h + l split by an fma, then 1 - x h - x l), leaving
// an error near 2^-104 relative before the final rounding (Newton-Raphson
// refinement of the reciprocal square root with an fma residual, as in
// Markstein's IA-64 division and square-root algorithms).
template <typename T> __device__ __forceinline__ T d_rsqrt(T x);
template <> __device__ __forceinline__ double d_rsqrt<double>(double x) {
    if (!(x > 1.0e-300) || x > 1.0e300) return pow(x, -0.5);   // y*y would leave the normal range: the plain pow
    const double y = 1. / sqrt(x);
    const double h = y * y;
    const double l = fma(y, y, -h);
    const double r = fma(-x, l, fma(-x, h, 1.));
    return fma(0.5 * y, r, y);
}
template <> __device__ __forceinline__ float d_rsqrt<float>(float x) { return powf(x, -0.5f); }
// a / b correctly rounded, given rb = RN(1/b) (b a per-launch constant whose
// reciprocal the host rounds once): q0 = RN(a rb), the residual r = a - b q0
// exactly by one fused multiply-add, then RN(q0 + r rb). This is the final
// correction step of Newton-Raphson division (P. Markstein, IBM J. Res. Dev.
// 34 (1990) 111-119): with rb within half an ulp of 1/b and q0 within an ulp
// of a/b it yields the correctly rounded quotient, barring overflow and
// underflow of the residual: for b a zone width (2^-100 < b < 2^100) the
// quotient is the IEEE one bit for bit whenever 2^-900 <= |a| <= 2^900, and
// for a = +-0 (a zero residual leaves q0, which keeps the sign of a). The
// step's dividends -- a step size times a difference of fluxes -- are zero
// or far inside that range (below it, where the residual turns subnormal,
// the quotient can be one ulp off). Three operations per use instead of a
// full division with its special-case branch.
__device__ __forceinline__ double div_rcp(double a, double b, double rb) {
    const double q0 = a * rb;
    const double r = fma(-q0, b, a);
    if constexpr (!STRICT) return fma(r, rb, q0);   // but for the sign of a zero the same
    return r == 0.0 ? q0 : fma(r, rb, q0);
}

// div_rcp that also returns the IEEE quotient where an operand is infinite
// or the divisor zero: there the residual is not finite (0 * inf or
// inf - inf) and q0 is already the IEEE result (+-inf, +-0 or NaN)
__device__ __forceinline__ double div_rcp_inf(double a, double b, double rb) {
    const double q0 = a * rb;
    const double r = fma(-q0, b, a);
    if constexpr (!STRICT) return not_finite(r) ? q0 : fma(r, rb, q0);
    return (r == 0.0 || !(fabs(r) <= 1.7976931348623157e308)) ? q0 : fma(r, rb, q0);
}

// the same where an infinite operand need not give the IEEE quotient (the
// conserved variables of a zone: an infinite one fails the inversion either way)
__device__ __forceinline__ double div_rcp_fin(double a, double b, double rb) {
    return STRICT ? div_rcp_inf(a, b, rb) : div_rcp(a, b, rb);
}

template <typename T>
__device__ __forceinline__ void geo_lapse(Geo<T> &o) {
    o.lapse = T(1.) / d_sqrt(-o.gcon[0]);
    o.rlapse = T(1.) / o.lapse;   // not read by the float quotients
    o.al = o.lapse;
}

// Quotients a_k / b that share one divisor. In double precision: one reciprocal
// of b, then per quotient a product (within 1.5 ulp, as accurate as the sums
// these quotients enter), or in the strict build the exact form (div_rcp_inf:
// the IEEE quotient bit for bit for 2^-900 <= |a| <= 2^900, zeros and
// infinities). Other types (float, whose division is the approximate one, and
// the adjoint's dual numbers) divide as written.
template <typename T>
struct Divisor {
    T b, rb;
    __device__ __forceinline__ explicit Divisor(T b_) : b(b_), rb(b_) {
        if constexpr (std::is_same<T, double>::value) rb = d_rcp(b_);
    }
    // with the divisor's reciprocal already at hand (rounded once, 1/b)
    __device__ __forceinline__ Divisor(T b_, T rb_) : b(b_), rb(rb_) {}
    __device__ __forceinline__ T div(T a) const {
        if constexpr (std::is_same<T, double>::value) return STRICT ? div_rcp_inf(a, b, rb) : a * rb;
        else return a / b;
    }
};

// the same with IEEE quotients in both builds: the conserved variables' u^t
// (ucon_calc), and HLLD's pressure solve, which differences a residual over a
// relative step of 1e-10, so that the last bits of its quotients are what its
// root is good to
template <typename T>
struct ExactDivisor {
    T b, rb;
    __device__ __forceinline__ explicit ExactDivisor(T b_) : b(b_), rb(T(1.0) / b_) {}
    __device__ __forceinline__ ExactDivisor(T b_, T rb_) : b(b_), rb(rb_) {}
    __device__ __forceinline__ T div(T a) const {
        if constexpr (std::is_same<T, double>::value) return div_rcp_inf(a, b, rb);
        else return a / b;
    }
};

template <typename T> __device__ __forceinline__ T d_max(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T d_min(T a, T b) { return a < b ? a : b; }

// G, the metric's type, may differ from the state's T: the adjoint runs these
// routines on dual numbers over a plain-double (constant) metric
template <typename T, typename G>
__device__ __forceinline__ void lower4(const T *u, const G *g, T *o) {
    o[0] = g[0] * u[0] + g[1] * u[1] + g[2] * u[2] + g[3] * u[3];
    o[1] = g[1] * u[0] + g[4] * u[1] + g[5] * u[2] + g[6] * u[3];
    o[2] = g[2] * u[0] + g[5] * u[1] + g[7] * u[2] + g[8] * u[3];
    o[3] = g[3] * u[0] + g[6] * u[1] + g[8] * u[2] + g[9] * u[3];
}
template <typename T, typename G>
__device__ __forceinline__ void raise4(const T *u, const G *g, T *o) { lower4(u, g, o); }

template <typename T>
__device__ __forceinline__ T dot4(const T *a, const T *b) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3];
}

template <typename T, typename G>
__device__ __forceinline__ void gamma_calc(const T *pr, const Geo<G> &gm, T *gamma) {
    const G *g = gm.gcov;
    T qsq = g[4] * pr[U1] * pr[U1] + g[7] * pr[U2] * pr[U2] + g[9] * pr[U3] * pr[U3]
          + T(2.) * (g[5] * pr[U1] * pr[U2] + g[6] * pr[U1] * pr[U3] + g[8] * pr[U2] * pr[U3]);
    if (qsq < T(0.)) {
        if (d_fabs(qsq) > T(1.E-10)) { *gamma = T(1.); return; }
        qsq = T(1.E-10);
    }
    *gamma = d_sqrt(T(1.) + qsq);
}

// u_mu, dot product, u^mu and b^mu of the HLL sides and the centre EMFs in both
// precisions: fused sums, u~^i u~_i nested, one reciprocal and no division
// (beta^j / alpha = alpha g^tj). Where plain_forms holds, the forms below.
template <typename T>
__device__ __forceinline__ void lower_hll(const T *u, const T *g, T *o) {
    o[0] = mad(g[3], u[3], mad(g[2], u[2], mad(g[1], u[1], mul(g[0], u[0]))));
    o[1] = mad(g[6], u[3], mad(g[5], u[2], mad(g[4], u[1], mul(g[1], u[0]))));
    o[2] = mad(g[8], u[3], mad(g[7], u[2], mad(g[5], u[1], mul(g[2], u[0]))));
    o[3] = mad(g[9], u[3], mad(g[8], u[2], mad(g[6], u[1], mul(g[3], u[0]))));
}
template <typename T>
__device__ __forceinline__ T dot_hll(const T *a, const T *b) {
    return mad(a[3], b[3], mad(a[2], b[2], mad(a[1], b[1], mul(a[0], b[0]))));
}
template <typename T>
__device__ __forceinline__ void ucon_hll(const T *pr, const Geo<T> &gm, T *ucon) {
    const T *g = gm.gcov;
    const T u1 = pr[U1], u2 = pr[U2], u3 = pr[U3];
    const T q1 = mad(g[4], u1, mul(T(2.), mad(g[5], u2, mul(g[6], u3))));
    const T q2 = mad(g[7], u2, mul(T(2.), mul(g[8], u3)));
    const T qsq = mad(u1, q1, mad(u2, q2, mul(mul(g[9], u3), u3)));
    // clamped as gamma_calc: 1 where it is negative beyond rounding
    const T gamma = qsq < T(-1.E-10) ? T(1.) : d_sqrt(T(1.) + (qsq < T(0.) ? T(1.E-10) : qsq));
    const T alpha = sizeof(T) == sizeof(double) ? gm.lapse : gm.al;
    ucon[0] = mul(gamma, gm.rlapse);
#pragma unroll
    for (int j = 1; j < 4; j++) ucon[j] = mad(-gamma, mul(gm.gcon[j], alpha), pr[U1 + j - 1]);
}
template <typename T>
__device__ __forceinline__ void bcon_hll(const T *pr, const T *ucon, const T *ucov, T *bcon) {
    bcon[0] = mad(pr[B3], ucov[3], mad(pr[B2], ucov[2], mul(pr[B1], ucov[1])));
    const T ru = d_rcp(ucon[0]);
#pragma unroll
    for (int j = 1; j < 4; j++) bcon[j] = mul(mad(bcon[0], ucon[j], pr[B1 - 1 + j]), ru);
}

// u^mu of a state. The production build's double form is ucon_hll, but for exact
// quotients by alpha where the caller asks for them: the conserved variables
// that the update starts from, since the inversion multiplies u^t by alpha again
// and a product with the rounded 1/alpha would scale a column's mass by the same
// last bit every step (tests/test_gpu_column_mass.py).
template <typename T, typename G>
__device__ __forceinline__ void ucon_calc(const T *pr, const Geo<G> &gm, T *ucon, bool exact = false) {
    const G alpha = gm.lapse;   // 1/sqrt(-g^tt), from the Geo (tabulated or geo_lapse)
    bool shorter = false;
    if constexpr (std::is_same<T, double>::value && std::is_same<T, G>::value && !STRICT) {
        shorter = !exact;
        if (shorter) ucon_hll(pr, gm, ucon);
    }
    if (!shorter) {
        G beta[4];
        T gamma;
        gamma_calc(pr, gm, &gamma);
#pragma unroll
        for (int j = 1; j < 4; j++) beta[j] = gm.gcon[j] * alpha * alpha;
        if constexpr (std::is_same<T, G>::value) {
            const ExactDivisor<T> da(alpha, gm.rlapse);   // four quotients by the lapse
            ucon[0] = da.div(gamma);
#pragma unroll
            for (int j = 1; j < 4; j++) ucon[j] = pr[U1 + j - 1] - da.div(gamma * beta[j]);
        } else {
            ucon[0] = gamma / alpha;
#pragma unroll
            for (int j = 1; j < 4; j++) ucon[j] = pr[U1 + j - 1] - gamma * beta[j] / alpha;
        }
    }
}

template <typename T>
__device__ __forceinline__ void bcon_calc(const T *pr, const T *ucon, const T *ucov, T *bcon) {
    bcon[0] = pr[B1] * ucov[1] + pr[B2] * ucov[2] + pr[B3] * ucov[3];
    const Divisor<T> du(ucon[0]);
#pragma unroll
    for (int j = 1; j < 4; j++) bcon[j] = du.div(pr[B1 - 1 + j] + bcon[0] * ucon[j]);
}

template <typename T, typename G>
__device__ __forceinline__ void get_state(const T *pr, const Geo<G> &gm, State<T> &q, bool exact = false) {
    ucon_calc(pr, gm, q.ucon, exact);
    lower4(q.ucon, gm.gcov, q.ucov);
    bcon_calc(pr, q.ucon, q.ucov, q.bcon);
    lower4(q.bcon, gm.gcov, q.bcov);
}

template <typename T>
__device__ __forceinline__ T entropy(T gam, const T *pr) {
    T P = (gam - T(1.0)) * pr[UU];
    return P * d_pow(pr[RHO], -gam);
}

// Fluxes in direction dir (dir == 0: conserved variables); with dir != 0 the
// fast magnetosonic speeds along dir as well. `ent` is the entropy K of pr,
// computed once per state by the caller.
template <typename T, typename G>
__device__ __forceinline__ void primtoflux(T gam, const T *pr, const State<T> &q, int dir, const Geo<G> &gm,
                                           T ent, T *flux, T *vmax, T *vmin) {
    T mhd[4];
    T u = pr[UU];
    T P = (gam - T(1.)) * u;
    T w = pr[RHO] + P + u;
    T bsq = dot4(q.bcon, q.bcov);
    T eta = w + bsq;
    T ptot = P + T(0.5) * bsq;
    flux[RHO] = pr[RHO] * q.ucon[dir];
#pragma unroll
    for (int j = 0; j < 4; j++)
        mhd[j] = eta * q.ucon[dir] * q.ucov[j] + ptot * (dir == j ? T(1.) : T(0.)) - q.bcon[dir] * q.bcov[j];
    flux[UU] = mhd[0] + flux[RHO];
    flux[U1] = mhd[1];
    flux[U2] = mhd[2];
    flux[U3] = mhd[3];
    flux[B1] = q.bcon[1] * q.ucon[dir] - q.bcon[dir] * q.ucon[1];
    flux[B2] = q.bcon[2] * q.ucon[dir] - q.bcon[dir] * q.ucon[2];
    flux[B3] = q.bcon[3] * q.ucon[dir] - q.bcon[dir] * q.ucon[3];
    flux[KTOT] = flux[RHO] * ent;
#pragma unroll
    for (int k = 0; k < NPR; k++) flux[k] *= gm.g;
    if (dir != 0) {
        G Acon_0, Acon_js;
        if (dir == 1) { Acon_0 = gm.gcon[1]; Acon_js = gm.gcon[4]; }
        else if (dir == 2) { Acon_0 = gm.gcon[2]; Acon_js = gm.gcon[7]; }
        else { Acon_0 = gm.gcon[3]; Acon_js = gm.gcon[9]; }
        T cs2 = gam * (gam - T(1.)) * pr[UU] / w;
        T va2 = bsq / eta;
        T cms2 = cs2 + va2 - cs2 * va2;
        if (cms2 < T(0.)) cms2 = T(SMALL_D);
        if (cms2 > T(1.)) cms2 = T(1.);
        const G Asq = Acon_js, Bsq = gm.gcon[0], AB = Acon_0;
        T Au = q.ucon[dir], Bu = q.ucon[0];
        T Au2 = Au * Au, Bu2 = Bu * Bu, AuBu = Au * Bu;
        T A = Bu2 - (Bsq + Bu2) * cms2;
        T B = T(2.) * (AuBu - (AB + AuBu) * cms2);
        T C = Au2 - (Asq + Au2) * cms2;
        T discr = B * B - T(4.) * A * C;
        if ((discr < T(0.0)) && (discr > T(-1.e-10))) discr = T(0.0);
        else if (discr < T(-1.e-10)) discr = T(0.);
        discr = d_sqrt(discr);
        const Divisor<T> d2a(T(2.) * A);
        T vp = d2a.div(-(-B + discr));
        T vm = d2a.div(-(-B - discr));
        *vmax = d_max(vp, vm);
        *vmin = d_min(vp, vm);
    }
}

// One side of an HLL face in the production build: fluxes along DIR and
// conserved variables, both without sqrt(-g) (the caller's HLL weights carry
// it), and the fast speeds along DIR. get_state and primtoflux in both
// directions in one, sharing what they share, and with
//   b^i u^t - b^t u^i = B^i                 (the conserved field)
//   c_s^2 + v_A^2 - c_s^2 v_A^2 = (gamma P + b^2) / (w + b^2)
//   (w + b^2) u_t + rho = rho (1 + u_t) + (gamma u + b^2) u_t
// the last because the energy row carries the rest-mass flux, which cancels
// most of it: 1 + u_t is formed first, without the rounding of either, and the
// halved quadratic for the speeds. The normal field's flux is zero and left
// out.
template <int DIR, typename T>
__device__ __forceinline__ void hll_side(T gam, const T *pr, const Geo<T> &gm, T *F, T *U, T &vmax, T &vmin) {
    T u[4], ul[4], b[4], bl[4];
    ucon_hll(pr, gm, u);
    lower_hll(u, gm.gcov, ul);
    bcon_hll(pr, u, ul, b);
    lower_hll(b, gm.gcov, bl);
    const T rho = pr[RHO];
    const T P = mul(gam - T(1.), pr[UU]);
    const T bsq = dot_hll(b, bl);
    const T gub = mad(gam, pr[UU], bsq), eta = rho + gub;
    const T ptot = mad(T(0.5), bsq, P);
    const T ent = mul(P, d_pow(rho, -gam));
    F[RHO] = mul(rho, u[DIR]);
    U[RHO] = mul(rho, u[0]);
    F[KTOT] = mul(F[RHO], ent);
    U[KTOT] = mul(U[RHO], ent);
    const T et = mad(rho, T(1.) + ul[0], mul(gub, ul[0]));
    F[UU] = mad(et, u[DIR], mul(-b[DIR], bl[0]));
    U[UU] = mad(et, u[0], mul(-b[0], bl[0])) + ptot;
    const T ed = mul(eta, u[DIR]), e0 = mul(eta, u[0]);
#pragma unroll
    for (int j = 1; j < 4; j++) {
        F[UU + j] = mad(ed, ul[j], mul(-b[DIR], bl[j]));
        U[UU + j] = mad(e0, ul[j], mul(-b[0], bl[j]));
    }
    F[UU + DIR] += ptot;
#pragma unroll
    for (int j = 1; j < 4; j++)
        if (j != DIR) {
            F[B1 + j - 1] = mad(b[j], u[DIR], mul(-b[DIR], u[j]));
            U[B1 + j - 1] = pr[B1 + j - 1];
        }
    T c2 = mul(mad(gam, P, bsq), d_rcp(eta));
    if (c2 < T(0.)) c2 = T(SMALL_D);
    if (c2 > T(1.)) c2 = T(1.);
    constexpr int sdd = DIR == 1 ? 4 : (DIR == 2 ? 7 : 9);
    const T u02 = mul(u[0], u[0]), u0d = mul(u[0], u[DIR]), ud2 = mul(u[DIR], u[DIR]);
    const T A = mad(-c2, gm.gcon[0] + u02, u02);
    const T B = mad(-c2, gm.gcon[DIR] + u0d, u0d);
    const T C = mad(-c2, gm.gcon[sdd] + ud2, ud2);
    T disc = mad(B, B, mul(-A, C));
    if (disc < T(0.)) disc = T(0.);
    disc = d_sqrt(disc);
    const T rA = d_rcp(A);
    const T vp = mul(B - disc, rA), vm = mul(B + disc, rA);
    vmax = d_max(vp, vm);
    vmin = d_min(vp, vm);
}

// monotonized-central slope with the GPU's steepening factor 2 (slope_lim,
// GPU_interp.h:2-38); a zone's face values are y -+ slope/2
template <typename T>
__device__ __forceinline__ T slope_lim(T y1, T y2, T y3) {
    const T Dqm = T(2.0) * (y2 - y1);
    const T Dqp = T(2.0) * (y3 - y2);
    const T Dqc = T(0.5) * (y3 - y1);
    const T s = Dqm * Dqp;
    if (s <= T(0.)) return T(0.);
    if (d_fabs(Dqm) < d_fabs(Dqp) && d_fabs(Dqm) < d_fabs(Dqc)) return Dqm;
    if (d_fabs(Dqp) < d_fabs(Dqc)) return Dqp;
    return Dqc;
}

// a / 6 for PPM's edge correction: in the strict build's double precision by
// the exact reciprocal form (div_rcp; the IEEE quotient bit for bit for
// 2^-900 <= |a| <= 2^900 and zeros, the range of differences of limited
// slopes of the state), in the production build's a product, else the type's
// own division
template <typename T>
__device__ __forceinline__ T div6(T a) {
    if constexpr (std::is_same<T, double>::value) return STRICT ? div_rcp(a, 6.0, 1.0 / 6.0) : mul(a, 1.0 / 6.0);
    else return a / T(6.0);
}

// x < 0 and x > 0 of a double from the bits of its upper word, so that the
// test runs on the integer pipe and not on the FP64 one, where PPM's dozen
// comparisons per value would queue with its arithmetic. Same answers as the
// comparison, infinities, zeros of either sign and NaNs (false) included,
// save that a magnitude below 2^-1042 counts as zero.
__device__ __forceinline__ bool is_neg(double x) { return (unsigned)__double2hiint(x) - 0x80000001u < 0x7ff00000u; }
__device__ __forceinline__ bool is_pos(double x) { return (unsigned)__double2hiint(x) - 1u < 0x7ff00000u; }
__device__ __forceinline__ bool is_neg(float x) { return x < 0.f; }
__device__ __forceinline__ bool is_pos(float x) { return x > 0.f; }

// PPM in three parts, each a value that neighbouring zones share, so that a
// kernel that walks or shares a row evaluates it once:
//   ppm_slope   the limited slope of a zone (its five-zone stencils overlap
//               three times), min(2|a|, 2|b|, |a + b|/2) with the sign of the
//               centred difference, zero at an extremum. The doublings of the
//               reference's form are folded into one exact scaling at the end
//               (powers of two), which gives the same value bit for bit, NaNs
//               included (tests/test_gpu_nan_reconstruction.py; in double a
//               product of the differences below 2^-1042 counts as zero);
//   ppm_face    the interpolated value between two zones, the upper edge of
//               one and the lower edge of the next;
//   ppm_limit   the monotonised edges of a zone from its value and the two.
template <typename T>
__device__ __forceinline__ T ppm_slope(T y0, T y1, T y2) {
    const T a = y1 - y0, b = y2 - y1, c = y2 - y0;
    const T m = d_min(d_fabs(c), T(4.) * d_min(d_fabs(a), d_fabs(b)));
    // the product's sign; in float scaled as the reference's, so that it
    // underflows no earlier
    const T s = sizeof(T) == 4 ? (T(4.) * a) * b : a * b;
    // a product at an extremum too, whose factor is zero there: a NaN stays one
    return (is_pos(c) ? m : -m) * (is_pos(s) ? T(0.5) : T(0.));
}
template <bool FT, typename T>
__device__ __forceinline__ T ppm_face(T y1, T y2, T dq1, T dq2) {
    if constexpr (plain_forms<T, FT>) return T(0.5) * (y2 + y1) - div6(dq2 - dq1);
    else return mad(T(0.5), y2 + y1, -div6(dq2 - dq1));
}
template <bool FT, typename T>
__device__ __forceinline__ void ppm_limit(T y, T l, T r, T &lout, T &rout) {
    const T qa = (r - y) * (y - l);
    const T qd = (r - l);
    if constexpr (plain_forms<T, FT>) {
        const T qe = T(6.0) * (y - T(0.5) * (l + r));
        if (qa <= T(0.)) { l = y; r = y; }
        if (qd * (qd - qe) < T(0.0)) l = T(3.0) * y - T(2.0) * r;
        else if (qd * (qd + qe) < T(0.0)) r = T(3.0) * y - T(2.0) * l;
    } else {
        const T qe = mul(T(6.0), mad(T(-0.5), l + r, y));
        if (qa <= T(0.)) { l = y; r = y; }
        if (is_neg(qd * (qd - qe))) l = mad(T(3.0), y, T(-2.0) * r);
        else if (is_neg(qd * (qd + qe))) r = mad(T(3.0), y, T(-2.0) * l);
    }
    lout = l;
    rout = r;
}

// the plain form of a whole zone: the same values as the three parts, but
// sharing no part with another zone. How the compiler contracts the solver that
// follows depends on the code before it, and this is the text that goes with
// the bits above.
template <typename T>
__device__ __forceinline__ void para_plain(const T *y, T &lout, T &rout) {
    T dq[5];
#pragma unroll
    for (int i = 1; i < 4; i++) {
        T Dqm = T(2.) * (y[i] - y[i - 1]);
        T Dqp = T(2.) * (y[i + 1] - y[i]);
        T Dqc = T(0.5) * (y[i + 1] - y[i - 1]);
        T aDqm = d_fabs(Dqm), aDqp = d_fabs(Dqp), aDqc = d_fabs(Dqc);
        T s = Dqm * Dqp;
        Dqm = d_min(aDqm, aDqp);
        if (aDqc < Dqm) {
            if (Dqc > T(0.)) dq[i] = (aDqc) * (T)(s > T(0.));
            else dq[i] = (-aDqc) * (T)(s > T(0.));
        } else {
            if (Dqc > T(0.)) dq[i] = (Dqm) * (T)(s > T(0.));
            else dq[i] = (-Dqm) * (T)(s > T(0.));
        }
    }
    const T l = T(0.5) * (y[2] + y[1]) - div6(dq[2] - dq[1]);
    const T r = T(0.5) * (y[3] + y[2]) - div6(dq[3] - dq[2]);
    ppm_limit<true>(y[2], l, r, lout, rout);
}

// PPM face values of the middle of five zones: l = lower edge, r = upper edge
template <bool FT = false, typename T>
__device__ __forceinline__ void para(const T *y, T &lout, T &rout) {
    if constexpr (plain_forms<T, FT>) {
        para_plain(y, lout, rout);
    } else {
        const T d1 = ppm_slope(y[0], y[1], y[2]), d2 = ppm_slope(y[1], y[2], y[3]), d3 = ppm_slope(y[2], y[3], y[4]);
        ppm_limit<FT>(y[2], ppm_face<FT>(y[1], y[2], d1, d2), ppm_face<FT>(y[2], y[3], d2, d3), lout, rout);
    }
}

// the two states at the face between the third and fourth of six zones: the
// upper edge of the third (hi2) and the lower edge of the fourth (lo3)
template <bool FT, typename T>
__device__ __forceinline__ void para_face(const T *y, T &hi2, T &lo3) {
    T drop;
    if constexpr (plain_forms<T, FT>) {
        para_plain(y, drop, hi2);
        para_plain(y + 1, lo3, drop);
    } else {
        T dq[4];
#pragma unroll
        for (int k = 0; k < 4; k++) dq[k] = ppm_slope(y[k], y[k + 1], y[k + 2]);
        const T f1 = ppm_face<FT>(y[1], y[2], dq[0], dq[1]), f2 = ppm_face<FT>(y[2], y[3], dq[1], dq[2]),
                f3 = ppm_face<FT>(y[3], y[4], dq[2], dq[3]);
        ppm_limit<FT>(y[2], f1, f2, drop, hi2);
        ppm_limit<FT>(y[3], f2, f3, lo3, drop);
    }
}

// ---------------------------------------------------------------- inversion
struct InvQ {
    double Bcon[4], Qcon[4], ncon[4], Bsq, QdotB, QdotBsq, Qtsq, Qdotn, D;
};

// per-zone constants of the inversion: gamma and the metric values it
// divides by, with their reciprocals rounded once (exact divisions, div_rcp),
// and the lapse and the normal observer's n_t. Either tabulated per (i, j)
// column or computed in place (inv_consts), with the same operations.
struct InvK {
    double gam, rgam, gdet, rgdet, alpha, ncov;
};

__device__ __forceinline__ InvK inv_consts(double gam, double rgam, double gdet, const double *gcon) {
    return InvK{gam, rgam, gdet, 1.0 / gdet, 1.0 / sqrt(-gcon[0]), -sqrt(-1. / gcon[0])};
}

__device__ __forceinline__ void inv_scalars_n(const double *U, const double *gcov, const double *gcon, double ncov,
                                              InvQ &s) {
    double Bcov[4], Qcov[4], Qsq;
    s.Bcon[0] = 0.;
    for (int i = 1; i < 4; i++) s.Bcon[i] = U[B1 + i - 1];
    lower4(s.Bcon, gcov, Bcov);
    for (int i = 0; i < 4; i++) Qcov[i] = U[UU + i];
    raise4(Qcov, gcon, s.Qcon);
    s.Bsq = 0.;
    for (int i = 1; i < 4; i++) s.Bsq += s.Bcon[i] * Bcov[i];
    s.QdotB = 0.;
    for (int i = 0; i < 4; i++) s.QdotB += Qcov[i] * s.Bcon[i];
    s.QdotBsq = s.QdotB * s.QdotB;
    s.ncon[0] = gcon[0] * ncov;
    s.ncon[1] = gcon[1] * ncov;
    s.ncon[2] = gcon[2] * ncov;
    s.ncon[3] = gcon[3] * ncov;
    s.Qdotn = s.Qcon[0] * ncov;
    Qsq = 0.;
    for (int i = 0; i < 4; i++) Qsq += Qcov[i] * s.Qcon[i];
    s.Qtsq = Qsq + s.Qdotn * s.Qdotn;
    s.D = U[RHO];
}

__device__ __forceinline__ void inv_scalars(const double *U, const double *gcov, const double *gcon, InvQ &s) {
    inv_scalars_n(U, gcov, gcon, -sqrt(-1. / gcon[0]), s);
}

__device__ __forceinline__ int guess_utsq(const double *gcov, const double *prim, double *out) {
    double utsq = gcov[4] * prim[U1] * prim[U1];
    utsq += 2. * gcov[5] * prim[U2] * prim[U1];
    utsq += 2. * gcov[6] * prim[U3] * prim[U1];
    utsq += gcov[7] * prim[U2] * prim[U2];
    utsq += 2 * gcov[8] * prim[U3] * prim[U2];
    utsq += gcov[9] * prim[U3] * prim[U3];
    if ((utsq < 0.) && (fabs(utsq) < 1.0e-13)) utsq = fabs(utsq);
    if (utsq < 0. || utsq > UTSQ_TOO_BIG) return 2;
    *out = utsq;
    return 0;
}

__device__ __forceinline__ void set_velocity(const InvQ &s, double gamma, double W, double *prim) {
    const Divisor<double> dw(W);   // the three quotients by W
    const double gw = STRICT ? gamma / (W + s.Bsq) : gamma * d_rcp(W + s.Bsq);
    for (int i = 1; i < 4; i++) {
        double Qtcon = s.Qcon[i] + s.ncon[i] * s.Qdotn;
        prim[U1 + i - 1] = gw * (Qtcon + dw.div(s.QdotB * s.Bcon[i]));
    }
}

// the same with the divisions by gdet in the exact reciprocal form
__device__ __forceinline__ int inv_prologue_k(const double *U, const InvK &k, double *prim, double *Ut) {
    if (U[0] <= 0.) return -100;
    for (int i = B1; i <= B3; i++) prim[i] = div_rcp_fin(U[i], k.gdet, k.rgdet);
    Ut[RHO] = div_rcp_fin(k.alpha * U[RHO], k.gdet, k.rgdet);
    Ut[UU] = div_rcp_fin(k.alpha * (U[UU] - U[RHO]), k.gdet, k.rgdet);
    for (int i = U1; i <= U3; i++) Ut[i] = div_rcp_fin(k.alpha * U[i], k.gdet, k.rgdet);
    for (int i = B1; i <= B3; i++) Ut[i] = div_rcp_fin(k.alpha * U[i], k.gdet, k.rgdet);
    return 0;
}

__device__ __forceinline__ int inv_prologue(const double *U, double gdet, const double *gcon, double *prim, double *Ut) {
    if (U[0] <= 0.) return -100;
    for (int i = B1; i <= B3; i++) prim[i] = U[i] / gdet;
    double alpha = 1.0 / sqrt(-gcon[0]);
    Ut[RHO] = alpha * U[RHO] / gdet;
    Ut[UU] = alpha * (U[UU] - U[RHO]) / gdet;
    for (int i = U1; i <= U3; i++) Ut[i] = alpha * U[i] / gdet;
    for (int i = B1; i <= B3; i++) Ut[i] = alpha * U[i] / gdet;
    return 0;
}

__device__ __forceinline__ double vsq_of_W(double W, double Bsq, double Qtsq, double QdotBsq) {
    double Wsq = W * W;
    double Xsq = (Bsq + W) * (Bsq + W);
    const double num = Wsq * Qtsq + QdotBsq * (Bsq + 2. * W);
    return STRICT ? num / (Wsq * Xsq) : num * d_rcp(Wsq * Xsq);
}

// Noble et al. 2006, 2D Newton-Raphson on (W, v^2). The divisions by gamma
// and gdet use their reciprocals in the exact form (div_rcp_inf): the same
// quotients, bit for bit, for the dividends this solver meets (an energy
// density or a conserved variable, between 2^-900 and 2^900, zero, or
// non-finite).
__device__ __forceinline__ int utoprim_2d_k(const InvK &k, const double *U, const double *gcov, const double *gcon,
                                            double *prim) {
    const double gam = k.gam, rgam = k.rgam;
    double Ut[NPR], pt[5];
    int ret = inv_prologue_k(U, k, prim, Ut);
    if (ret) return ret;
    for (int i = 0; i < B1; i++) pt[i] = prim[i];
    InvQ s;
    inv_scalars_n(Ut, gcov, gcon, k.ncov, s);
    double utsq;
    if (guess_utsq(gcov, pt, &utsq)) return 2;
    double gammasq = 1. + utsq;
    double gamma = d_sqrt(gammasq);
    double rho0 = STRICT ? s.D / gamma : s.D * d_rcp(gamma);
    double u = pt[UU];
    double p = (gam - 1.) * u;
    double w = rho0 + u + p;
    double W_last = w * gammasq;
    int i_increase = 0;
    while (((W_last * W_last * W_last * (W_last + 2. * s.Bsq) - s.QdotBsq * (2. * W_last + s.Bsq)) <= W_last * W_last * (s.Qtsq - s.Bsq * s.Bsq)) && (i_increase < 10)) {
        W_last *= 10.;
        i_increase++;
    }
    double x0 = fabs(W_last);
    double vs = fabs(vsq_of_W(W_last, s.Bsq, s.Qtsq, s.QdotBsq));
    double x1 = (vs > 1.) ? (1.0 - 1.e-15) : vs;
    // Newton iterations (general_newton_raphson, func_vsq)
    double f = 1., df = 1., errx = 1.;
    bool converged = false;
    int n_iter = 0, i_extra = 0, doing_extra = 0, keep = 1;
    const double Bsq = s.Bsq, Qtsq = s.Qtsq, QdotBsq = s.QdotBsq, Qdotn = s.Qdotn, D = s.D;
    // 1/x0 of the current iterate: t23 of this iteration, and the divisor of
    // the previous iteration's errx (the same x0), one reciprocal for both
    double rx0 = d_rcp(x0);
    while (keep) {
        double t11, t18, dx0, dx1;
        if constexpr (STRICT) {
            double Wsq = x0 * x0;
            double gtmp = 1. - x1;
            double p_tmp = div_rcp_inf((gam - 1.) * (fma(x0, gtmp, -D * sqrt(gtmp))), gam, rgam);
            double dPdW = div_rcp_inf((gam - 1.) * (1. - x1), gam, rgam);
            double dPdvsq = div_rcp_inf((gam - 1.) * (fma(0.5, D / sqrt(1. - x1), -x0)), gam, rgam);
            double t2 = -0.5 * Bsq + dPdvsq;
            double t3 = Bsq + x0;
            double t4 = t3 * t3;
            double t9 = 1. / Wsq;
            t11 = Qtsq - x1 * t4 + QdotBsq * (Bsq + 2.0 * x0) * t9;
            double t16 = QdotBsq * t9;
            t18 = -Qdotn - 0.5 * Bsq * (1.0 + x1) + 0.5 * t16 - x0 + p_tmp;
            double t21 = 1. / t3;
            double t23 = rx0;
            double t24 = t16 * t23;
            double t25 = -1.0 + dPdW - t24;
            double t35 = t25 * t3 + (Bsq - 2.0 * dPdvsq) * (QdotBsq + x1 * Wsq * x0) * t9 * t23;
            double t36 = 1. / t35;
            dx0 = -(t2 * t11 + t4 * t18) * t21 * t36;
            double t40 = (x1 + t24) * t3;
            dx1 = -(-t25 * t11 - 2.0 * t40 * t18) * t21 * t36;
        } else {
            // the same residuals and Jacobian with x0^-2 = (1/x0)^2,
            // (QdotBsq + x1 x0^3) / x0^3 = t24 + x1, the two divisions of each
            // increment as one, and the root of 1 - x1 with its reciprocal
            const double gtmp = 1. - x1;
            double rs;
            const double sg = sqrt_nr_pos(gtmp, rs);   // 1e-15 <= gtmp <= 1
            const double kg = (gam - 1.) * rgam;
            const double p_tmp = kg * fma(x0, gtmp, -D * sg);
            const double dPdvsq = kg * fma(0.5 * D, rs, -x0);
            const double t2 = fma(-0.5, Bsq, dPdvsq);
            const double t3 = Bsq + x0;
            const double t4 = t3 * t3;
            const double t16 = QdotBsq * (rx0 * rx0);
            const double t24 = t16 * rx0;
            const double t40 = x1 + t24;
            t11 = fma(t16, fma(2.0, x0, Bsq), fma(-x1, t4, Qtsq));
            t18 = -Qdotn - 0.5 * Bsq * (1.0 + x1) + 0.5 * t16 - x0 + p_tmp;
            const double t25 = fma(kg, gtmp, -1.0) - t24;
            const double t35 = fma(t25, t3, fma(-2.0, dPdvsq, Bsq) * t40);
            const double r = rcp_nr_finite(t3 * t35);
            dx0 = -fma(t2, t11, t4 * t18) * r;
            dx1 = fma(t25, t11, 2.0 * (t40 * t3) * t18) * r;
        }
        df = -t11 * t11 - t18 * t18;
        f = -0.5 * df;
        double xo0 = x0;
        x0 += dx0;
        x1 += dx1;
        x0 = fabs(x0);
        x0 = (x0 > W_TOO_BIG) ? xo0 : x0;
        x1 = (x1 < 0.) ? 0. : x1;
        x1 = (x1 > 1.) ? (1. - 1.e-15) : x1;
        if constexpr (STRICT) {
            rx0 = 1. / x0;
            errx = (x0 == 0.) ? fabs(x0 - xo0) : fabs(div_rcp_inf(x0 - xo0, x0, rx0));
            converged = fabs(errx) <= NEWT_TOL;
        } else {
            // the same test without the quotient; an iterate of zero, which no
            // root is, does not converge
            rx0 = rcp_nr_finite(x0);
            converged = fabs(x0 - xo0) <= NEWT_TOL * x0;
        }
        if (converged && (doing_extra == 0) && (EXTRA_NEWT_ITER > 0)) doing_extra = 1;
        if (doing_extra == 1) i_extra++;
        if ((converged && (doing_extra == 0)) || (i_extra > EXTRA_NEWT_ITER) || (n_iter >= (MAX_NEWT_ITER - 1)))
            keep = 0;
        n_iter++;
    }
    static_assert(MIN_NEWT_TOL >= NEWT_TOL, "one tolerance decides convergence");
    int retval = 0;
    if ((isfinite(f) == 0) || (isfinite(df) == 0)) retval = 2;
    else if (!converged) retval = 1;
    double W = x0, vsq = x1;
    if ((retval != 0) || (W == FAIL_VAL)) return retval * 100 + 1;
    if (W <= 0. || W > W_TOO_BIG) return 3;
    if (vsq >= 1.) return 4;
    double gtmp = d_sqrt(1. - vsq);
    gamma = d_rcp(gtmp);
    rho0 = s.D * gtmp;
    w = W * (1. - vsq);
    p = div_rcp_inf((gam - 1.) * (w - rho0), gam, rgam);
    u = w - (rho0 + p);
    if (rho0 <= 0.) return 5;
    if (u <= 0.) return 6;
    pt[RHO] = rho0;
    pt[UU] = u;
    set_velocity(s, gamma, W, pt);
    for (int i = 0; i < B1; i++) prim[i] = pt[i];
    return 0;
}

__device__ __forceinline__ int utoprim_2d(double gam, const double *U, const double *gcov, const double *gcon,
                                          double gdet, double *prim) {
    return utoprim_2d_k(inv_consts(gam, 1.0 / gam, gdet, gcon), U, gcov, gcon, prim);
}

// a / b in the arithmetic of the build: the fallback's iterations are one zone's
// dependent chain, a dozen of them with eight quotients and a power each
__device__ __forceinline__ double quot(double a, double b) { return STRICT ? a / b : a * rcp_nr(b); }

__device__ __forceinline__ double W_of_vsq2(double gam, double vsq, double *p, double *rho, double *u, double D, double K) {
    double gtmp = (1. - vsq);
    *rho = D * d_sqrt(gtmp);
    *p = K * d_pow(*rho, gam);
    *u = quot(*p, gam - 1.);
    return quot(*rho + *u + *p, gtmp);
}

// entropy-based 1D solve in v^2
__device__ __noinline__ int utoprim_1dvsq2fix1(double gam, const double *U, const double *gcov, const double *gcon, double gdet, double *prim) {
    double Ut[NPR], pt[5];
    int ret = inv_prologue(U, gdet, gcon, prim, Ut);
    if (ret) return ret;
    for (int i = 0; i < B1; i++) pt[i] = prim[i];
    double K = U[KTOT] / U[RHO];
    InvQ s;
    inv_scalars(Ut, gcov, gcon, s);
    double utsq, p, rho, u;
    if (guess_utsq(gcov, pt, &utsq)) return 2;
    double gammasq = 1. + utsq;
    double x = 1. - 1. / gammasq;
    double f = 1., df = 1., errx = 1., W = 0., W_old;
    int n_iter = 0, i_extra = 0, doing_extra = 0, keep = 1;
    // W(x) of the current iterate: the one formed for the convergence test of
    // the iteration before
    double Wc = W_of_vsq2(gam, x, &p, &rho, &u, s.D, K);
    while (keep) {
        double Wsq = Wc * Wc;
        double dWdvsq = quot(gam * (2. - gam) * p + (gam - 1.) * rho, 2. * (gam - 1.) * (1. - x) * (1. - x));
        double fact_tmp = (s.Bsq + Wc);
        double resid = s.Qtsq - x * fact_tmp * fact_tmp + quot(s.QdotBsq * (s.Bsq + 2. * Wc), Wsq);
        double jac = -fact_tmp * (fact_tmp + 2. * dWdvsq * (x + quot(s.QdotBsq, Wc * Wsq)));
        double dx = quot(-resid, jac);
        f = 0.5 * resid * resid;
        df = -2. * f;
        double xo = x;
        x += dx;
        x = (x >= 1.0) ? (0.5 * (xo + 1.)) : x;
        x = (x < -1.e-10) ? (0.5 * xo) : x;
        x = fabs(x);
        W_old = W;
        W = Wc = W_of_vsq2(gam, x, &p, &rho, &u, s.D, K);
        errx = (W == 0.) ? fabs(W - W_old) : fabs(quot(W - W_old, W));
        errx += (x == 0.) ? fabs(x - xo) : fabs(quot(x - xo, x));
        if ((fabs(errx) <= NEWT_TOL) && (doing_extra == 0) && (EXTRA_NEWT_ITER > 0)) doing_extra = 1;
        if (doing_extra == 1) i_extra++;
        if (((fabs(errx) <= NEWT_TOL) && (doing_extra == 0)) || (i_extra > EXTRA_NEWT_ITER) || (n_iter >= (MAX_NEWT_ITER - 1)))
            keep = 0;
        n_iter++;
    }
    int retval = 0;
    if ((isfinite(f) == 0) || (isfinite(df) == 0)) retval = 2;
    else if (fabs(errx) > d_min(NEWT_TOL, MIN_NEWT_TOL)) retval = 1;
    if (retval != 0) return retval * 100 + 1;
    double vsq = x;
    if ((vsq >= 1.) || (vsq < 0.)) return 4;
    double rho0;
    W = W_of_vsq2(gam, vsq, &p, &rho0, &u, s.D, K);
    double gtmp = sqrt(1. - vsq);
    double gamma = 1. / gtmp;
    if (rho0 <= 0.) return 5;
    if (u <= 0.) return 6;
    pt[RHO] = rho0;
    pt[UU] = u;
    set_velocity(s, gamma, W, pt);
    for (int i = 0; i < B1; i++) prim[i] = pt[i];
    return 0;
}

// inner density solve of the W-based entropy fallback (gnr2 / func_gnr2_rho)
__device__ __forceinline__ int rho_solve(double gam, double *xr, double D, double K, double W_for) {
    double f = 1., df = 1., errx = 1.;
    int n_iter = 0, keep = 1;
    double x = *xr;
    while (keep) {
        double A = D * D;
        double B0 = A * gam * K;
        double B = B0 / (gam - 1.);
        double C = pow(x, gam - 1.);
        double resid = x * W_for - A - B * C;
        double jac = W_for - B0 * C / x;
        double dx = -resid / jac;
        f = 0.5 * resid * resid;
        df = -2. * f;
        double xo = x;
        x += dx;
        x = fabs(x);
        errx = (x == 0.) ? fabs(x - xo) : fabs((x - xo) / x);
        if ((fabs(errx) <= 1.0e-15) || (n_iter >= (MAX_NEWT_ITER - 1))) keep = 0;
        n_iter++;
    }
    *xr = x;
    if ((isfinite(f) == 0) || (isfinite(df) == 0) || (isfinite(x) == 0)) return 2;
    if (fabs(errx) > 1.0e-10) return 1;
    return 0;
}

// entropy-based 1D solve in W
__device__ __noinline__ int utoprim_1dfix1(double gam, const double *U, const double *gcov, const double *gcon, double gdet, double *prim) {
    double Ut[NPR], pt[5];
    int ret = inv_prologue(U, gdet, gcon, prim, Ut);
    if (ret) return ret;
    for (int i = 0; i < B1; i++) pt[i] = prim[i];
    double K = U[KTOT] / U[RHO];
    InvQ s;
    inv_scalars(Ut, gcov, gcon, s);
    double utsq;
    if (guess_utsq(gcov, pt, &utsq)) return 2;
    const double Bsq = s.Bsq, Qtsq = s.Qtsq, QdotBsq = s.QdotBsq, D = s.D;
    double gammasq = 1. + utsq;
    double gamma = sqrt(gammasq);
    double rho0 = D / gamma;
    double p = K * pow(rho0, gam);
    double u = p / (gam - 1.);
    double w = rho0 + u + p;
    double W_last = w * gammasq;
    int i_increase = 0;
    while (((W_last * W_last * W_last * (W_last + 2. * Bsq) - QdotBsq * (2. * W_last + Bsq)) <= W_last * W_last * (Qtsq - Bsq * Bsq)) && (i_increase < 10)) {
        W_last *= 10.;
        i_increase++;
    }
    const double rho_for = rho0;
    double x = W_last;
    double f = 1., df = 1., errx = 1.;
    int n_iter = 0, i_extra = 0, doing_extra = 0, keep = 1;
    while (keep) {
        // func_1d_orig1
        double xr = rho_for, rho_g = rho_for;
        int ntries = 0;
        while ((rho_solve(gam, &xr, D, K, x)) && (ntries++ < 10)) {
            rho_g *= 10.;
            xr = rho_g;
        }
        double rho = xr;
        double t1 = D * D;
        double t2 = QdotBsq * t1;
        double t3 = t2 * Bsq;
        double t5 = Bsq * Bsq;
        double t8 = t1 * Bsq;
        double t10 = t1 * x;
        double t21 = x * x;
        double t23 = rho * rho;
        double t26 = 1. / t1;
        double resid = (t3 + (2.0 * t2 + ((Qtsq - t5) * t1 + (-2.0 * t8 - t10) * x) * x) * x + (t5 + (2.0 * Bsq + x) * x) * t21 * t23) * t26 / t21;
        double t29 = t1 * t1;
        double t30 = QdotBsq * t29;
        double t32 = gam * K;
        double t33 = pow(rho, 1.0 * gam);
        double t34 = t32 * t33;
        double t38 = t23 * t33;
        double t51 = gam * t1 * K * t33;
        double t67 = t21 * x;
        double jac = -2.0 * (t30 * Bsq * t34 + (t30 * t34 + ((-t38 * Bsq * t32 + Bsq * gam * t1 * K * t33) * t1 + (-t38 * gam * K + t51) * t1 * x) * t21) * x + ((-t3 + (-t2 + (-t8 - t10) * t21) * x) * x + (-t5 - Bsq * x) * t67 * t23) * t23) * t26 / (t51 - x * t23) / t67;
        double dx = -resid / jac;
        f = 0.5 * resid * resid;
        df = -2. * f;
        double xo = x;
        x += dx;
        int ii = 0;
        while (((x * x * x * (x + 2. * Bsq) - QdotBsq * (2. * x + Bsq)) <= x * x * (Qtsq - Bsq * Bsq)) && (ii < 10)) {
            x -= (1. * ii) * dx / 10.;
            ii++;
        }
        x = fabs(x);
        errx = (x == 0.) ? fabs(x - xo) : fabs((x - xo) / x);
        if ((fabs(errx) <= NEWT_TOL) && (doing_extra == 0) && (EXTRA_NEWT_ITER > 0)) doing_extra = 1;
        if (doing_extra == 1) i_extra++;
        if (((fabs(errx) <= NEWT_TOL) && (doing_extra == 0)) || (i_extra > EXTRA_NEWT_ITER) || (n_iter >= (MAX_NEWT_ITER - 1)))
            keep = 0;
        n_iter++;
    }
    int retval = 0;
    if ((isfinite(f) == 0) || (isfinite(df) == 0) || (isfinite(x) == 0)) retval = 2;
    else if (fabs(errx) > d_min(NEWT_TOL, MIN_NEWT_TOL)) retval = 1;
    double W = x;
    if ((retval != 0) || (W == FAIL_VAL)) return retval * 100 + 1;
    if (W <= 0. || W > W_TOO_BIG) return 3;
    double vsq = vsq_of_W(W, Bsq, Qtsq, QdotBsq);
    if (vsq >= 1.) return 4;
    double gtmp = sqrt(1. - vsq);
    gamma = 1. / gtmp;
    rho0 = D * gtmp;
    p = K * pow(rho0, gam);
    u = p / (gam - 1.);
    if (rho0 <= 0.) return 5;
    if (u <= 0.) return 6;
    pt[RHO] = rho0;
    pt[UU] = u;
    set_velocity(s, gamma, W, pt);
    for (int i = 0; i < B1; i++) prim[i] = pt[i];
    return 0;
}

// Newman & Hamlin 2014: fixed point on the pressure, W from the closed-form
// root of a cubic, Aitken extrapolation when three successive pressures
// contract (Utoprim_NM, GPU_utoprim_nm.h). The pressure history is a window
// of the last three values: the reference's array holds three entries but is
// indexed up to the iteration count, and only the last three are ever read.
__device__ __forceinline__ int utoprim_nm(double gam, const double *U, const double *gcov, const double *gcon,
                                          double gdet, double *prim) {
    double Ut[NPR], pt[5];
    int ret = inv_prologue(U, gdet, gcon, prim, Ut);
    if (ret) return ret;
    for (int i = 0; i < B1; i++) pt[i] = prim[i];
    InvQ s;
    inv_scalars(Ut, gcov, gcon, s);
    const double Bsq = s.Bsq, QdotBsq = s.QdotBsq, Qtsq = s.Qtsq, Qdotn = s.Qdotn;
    constexpr double PI_D = 3.14159265358979323846;
    double a, phi, epsilon, z = 0., vsq, w, gamma = 1., rho0 = 0., u = 0., errx, p_old, p_new;
    double pm2 = 0., pm1;   // pressures of iterations iter-2 and iter-1
    int iter = 0, iter_tot = 0, set_variables = 0;
    pm1 = (gam - 1.) * pt[UU];
    p_new = pm1;
    const double d = 0.5 * (Qtsq * Bsq - QdotBsq);
    if (d < 0.0) return 1;
    do {
        set_variables = 0;
        a = -Qdotn + p_new + 0.5 * Bsq;
        phi = acos(1. / a * sqrt((27. * d) / (4. * a)));
        epsilon = a / 3. - 2. / 3. * a * cos(2. / 3. * phi + 2. / 3. * PI_D);
        z = epsilon - Bsq;
        vsq = (Qtsq * z * z + QdotBsq * (Bsq + 2. * z)) / (z * z * pow(Bsq + z, 2.));
        if (fabs(vsq) < 1e-15) vsq = 0.0;
        if (fabs(vsq) >= 1.0) return 1;
        w = z * (1. - vsq);
        gamma = 1. / sqrt(1. - vsq);
        rho0 = Ut[RHO] / gamma;
        u = (w - rho0) / gam;
        iter++;
        iter_tot++;
        const double pc = (gam - 1.) * u;
        p_old = pm1;
        p_new = pc;
        bool restart = false;
        if (iter >= 2) {
            const double R = (pc - pm1) / (pm1 - pm2);
            if (R < 1. && R > 0.) {
                set_variables = 1;
                p_new = pm1 + (pc - pm1) / (1. - R);
                p_old = pc;
                iter = 0;
                restart = true;
            }
        }
        if (restart) {
            pm1 = p_new;   // the history restarts from the extrapolated pressure
        } else {
            pm2 = pm1;
            pm1 = pc;
        }
        errx = fabs(p_new - p_old) / fabs(p_new + p_old);
    } while (errx > NEWT_TOL && iter_tot < 30);
    if (fabs(errx) > d_min(NEWT_TOL, MIN_NEWT_TOL)) return 1;
    if (set_variables == 1) {
        a = -Qdotn + p_new + 0.5 * Bsq;
        phi = acos(1. / a * sqrt((27. * d) / (4. * a)));
        epsilon = a / 3. - 2. / 3. * a * cos(2. / 3. * phi + 2. / 3. * PI_D);
        z = epsilon - Bsq;
        vsq = (Qtsq * z * z + QdotBsq * (Bsq + 2. * z)) / (z * z * pow(Bsq + z, 2.));
        const double Wsq = 1. / (1. - vsq);
        w = z / Wsq;
        if (vsq >= 1.0 || vsq < 0. || z <= 0. || z > 1.e20 || !isfinite(vsq) || !isfinite(z)) return 4;
        gamma = sqrt(Wsq);
        rho0 = Ut[RHO] / gamma;
        u = (w - rho0) / gam;
        p_new = (gam - 1.) * u;
    }
    if (rho0 < 0.0) return 5;
    if (p_new < 0.0) return 6;
    pt[RHO] = rho0;
    pt[UU] = u;
    for (int i = 1; i < 4; i++) {
        const double Qtcon = s.Qcon[i] + s.ncon[i] * s.Qdotn;
        pt[U1 + i - 1] = gamma / (z + Bsq) * (Qtcon + s.QdotB * s.Bcon[i] / z);
    }
    for (int i = 0; i < B1; i++) prim[i] = pt[i];
    return 0;
}

// ---------------------------------------------------------------- HLLC
// (fluxcalc2D_FT, calc_HLLC, calc_HLLC_hydro, primtoflux_FT, vchar_FT:
// GPU_hllc.h:3-396, 903-1111; set_Mud: hllc.c:20-164)
__host__ __device__ __forceinline__ int sym4(int a, int b) {
    return a == b ? (a == 0 ? 0 : (a == 1 ? 4 : (a == 2 ? 7 : 9)))
                  : (a + b == 1 ? 1 : (a + b == 2 ? 2 : (a == 0 || b == 0 ? 3 : (a + b == 3 ? 5 : (a + b == 4 ? 6 : 8)))));
}

// orthonormal frame of a face of direction dir, from the face metric; (d, e, f)
// is the cyclic order starting at dir
template <typename T>
__device__ __forceinline__ void set_mud(const Geo<T> &gm, int dir, T Mud[4][4], T Mi[4][4]) {
    const int d = dir, e = dir % 3 + 1, f = (dir + 1) % 3 + 1;
#define GU(a, b) gm.gcon[sym4(a, b)]
#define GD(a, b) gm.gcov[sym4(a, b)]
    const T A = -d_rsqrt(-GU(0, 0));
    const T B = d_rsqrt((GU(0, 0)) * (GU(0, 0) * GU(d, d) - GU(0, d) * GU(0, d)));
    const T C = d_rsqrt(GD(f, f));
    const T D = d_rsqrt((GD(f, f)) * (GD(e, e) * GD(f, f) - GD(e, f) * GD(e, f)));
    for (int a = 0; a < 4; a++)
        for (int b = 0; b < 4; b++) Mud[a][b] = Mi[a][b] = T(0.);
    Mud[0][0] = A * GU(0, 0);
    Mud[d][0] = A * GU(0, d);
    Mud[d][d] = B * (GU(0, d) * GU(0, d) - GU(0, 0) * GU(d, d));
    Mud[e][0] = A * GU(0, e);
    Mud[e][d] = B * (GU(0, d) * GU(0, e) - GU(0, 0) * GU(d, e));
    Mud[e][e] = D * GD(f, f);
    Mud[f][0] = A * GU(0, f);
    Mud[f][d] = B * (GU(0, d) * GU(0, f) - GU(0, 0) * GU(d, f));
    Mud[f][e] = -D * GD(e, f);
    Mud[f][f] = C;
    const T E = GU(0, d) * GU(d, e) - GU(d, d) * GU(0, e);
    const T F = GU(0, d) * GU(0, e) - GU(0, 0) * GU(d, e);
    const T G = GU(0, d) * GU(d, f) - GU(d, d) * GU(0, f);
    const T H = GU(0, d) * GU(0, f) - GU(0, 0) * GU(d, f);
    Mi[0][0] = -A;
    Mi[d][0] = B * GU(0, d);
    Mi[d][d] = -B * GU(0, 0);
    Mi[e][0] = B * B * E * GU(0, 0) / (D * GD(f, f));
    Mi[e][d] = B * B * F * GU(0, 0) / (D * GD(f, f));
    Mi[e][e] = T(1.) / (D * GD(f, f));
    Mi[f][0] = (B * B / C) * GU(0, 0) * (G + E * GD(e, f) / GD(f, f));
    Mi[f][d] = (B * B / C) * GU(0, 0) * (H + F * GD(e, f) / GD(f, f));
    Mi[f][e] = (T(1.) / C) * GD(e, f) / GD(f, f);
    Mi[f][f] = T(1.) / C;
#undef GU
#undef GD
}

template <typename T>
__device__ __forceinline__ void primtoflux_ft(T gam, const T *pr, const T *ucon, const T *bcon, int dir, T *flux) {
    flux[RHO] = pr[RHO] * ucon[dir];
    const T P = (gam - T(1.)) * pr[UU];
    const T w = P + pr[RHO] + pr[UU];
    const T bsq = -bcon[0] * bcon[0] + bcon[1] * bcon[1] + bcon[2] * bcon[2] + bcon[3] * bcon[3];
    const T eta = w + bsq;
    const T ptot = P + T(0.5) * bsq;
    flux[UU] = -eta * ucon[dir] * ucon[0] + ptot * T(dir == 0 ? 1. : 0.) + bcon[dir] * bcon[0];
    for (int j = 1; j < 4; j++) flux[UU + j] = eta * ucon[dir] * ucon[j] + ptot * T(dir == j ? 1. : 0.) - bcon[dir] * bcon[j];
    for (int k = B1; k <= B3; k++) flux[k] = bcon[k - 4] * ucon[dir] - bcon[dir] * ucon[k - 4];
    flux[KTOT] = flux[RHO] * P * d_pow(pr[RHO], -gam);
}

template <typename T>
__device__ __forceinline__ void vchar_ft(T gam, const T *pr, const T *ucon, const T *bcon, int dir, T *vmax, T *vmin) {
    const T bsq = -bcon[0] * bcon[0] + bcon[1] * bcon[1] + bcon[2] * bcon[2] + bcon[3] * bcon[3];
    const T EF = pr[RHO] + gam * pr[UU];
    const T cs2 = gam * (gam - T(1.)) * pr[UU] / EF;
    const T EE = bsq + EF;
    const T va2 = bsq / EE;
    T cms2 = cs2 + va2 - cs2 * va2;
    if (cms2 < T(0.)) cms2 = T(SMALL_D);
    if (cms2 > T(1.)) cms2 = T(1.);
    const T Asq = T(1.), Bsq = T(-1.);
    const T Au = ucon[dir], Bu = ucon[0];
    const T Au2 = Au * Au, Bu2 = Bu * Bu, AuBu = Au * Bu;
    const T A = Bu2 - (Bsq + Bu2) * cms2;
    const T B = T(2.) * (AuBu - (AuBu) * cms2);
    const T C = Au2 - (Asq + Au2) * cms2;
    T discr = B * B - T(4.) * A * C;
    if ((discr < T(0.0)) && (discr > T(-1.e-10))) discr = T(0.0);
    else if (discr < T(-1.e-10)) discr = T(0.);
    discr = d_sqrt(discr);
    const Divisor<T> d2a(T(2.) * A);
    const T vp = d2a.div(-(-B + discr));
    const T vm = d2a.div(-(-B - discr));
    if (vp > vm) { *vmax = vp; *vmin = vm; }
    else { *vmax = vm; *vmin = vp; }
}

template <typename T>
__device__ __forceinline__ void hllc_hydro(int dir, const T *lu, const T *ru, T iv, T cmin, T cmax, T FT[2][NPR],
                                           const T FH[2][NPR], const T *Fl, const T *Fr, const T *Ul, const T *Ur) {
    const int U_1 = UU + dir, U_2 = UU + dir % 3 + 1, U_3 = UU + (dir + 1) % 3 + 1;
    const int B_1 = B1 + dir - 1, B_2 = B1 + dir % 3, B_3 = B1 + (dir + 1) % 3;
    bool fail = false;
    const T A = -FH[1][UU];
    const T B = -FH[1][U_1] + FH[0][UU];
    const T C = FH[0][U_1];
    const T D = B * B - T(4.) * A * C;
    const T vcon = (-B - d_sqrt(D)) / (T(2.) * A);
    const T ptot = -(-FH[1][UU]) * vcon + FH[1][U_1];
    if (!(d_fabs(ptot) > T(0.)) || (vcon < cmin) || (vcon > cmax) || !(d_fabs(vcon) > T(0.))) fail = true;
    if (cmax > iv && vcon <= iv && !fail) {
        const Divisor<T> dc(cmax - vcon + T(SMALL_D));
        const T s = dc.div(cmax - ru[dir] / ru[0]);
        FT[0][RHO] = s * Ur[RHO];
        FT[0][UU] = dc.div(cmax * Ur[UU] + Ur[U_1] - ptot * vcon);
        FT[0][U_1] = (-FT[0][UU] + ptot) * vcon;
        FT[0][U_2] = s * Ur[U_2];
        FT[0][U_3] = s * Ur[U_3];
        FT[0][B_1] = FH[0][B_1];
        FT[0][B_2] = s * Ur[B_2];
        FT[0][B_3] = s * Ur[B_3];
        FT[0][KTOT] = s * Ur[KTOT];
        for (int k = 0; k < NPR; k++) FT[1][k] = (Fr[k] + cmax * (FT[0][k] - Ur[k]));
    } else if (cmin < iv && vcon >= iv && !fail) {
        const Divisor<T> dc(cmin - vcon + T(SMALL_D));
        const T s = dc.div(cmin - lu[dir] / lu[0]);
        FT[0][RHO] = s * Ul[RHO];
        FT[0][UU] = dc.div(cmin * Ul[UU] + Ul[U_1] - ptot * vcon);
        FT[0][U_1] = (-FT[0][UU] + ptot) * vcon;
        FT[0][U_2] = s * Ul[U_2];
        FT[0][U_3] = s * Ul[U_3];
        FT[0][B_1] = FH[0][B_1];
        FT[0][B_2] = s * Ul[B_2];
        FT[0][B_3] = s * Ul[B_3];
        FT[0][KTOT] = s * Ul[KTOT];
        for (int k = 0; k < NPR; k++) FT[1][k] = (Fl[k] + cmin * (FT[0][k] - Ul[k]));
    } else {
        for (int k = 0; k < NPR; k++) { FT[0][k] = FH[0][k]; FT[1][k] = FH[1][k]; }
    }
}

template <typename T>
__device__ __forceinline__ void hllc_mhd(int dir, const T *lu, const T *ru, T iv, T cmin, T cmax, T FT[2][NPR],
                                         const T FH[2][NPR], const T *Fl, const T *Fr, const T *Ul, const T *Ur) {
    const int G_1 = dir, G_2 = dir % 3 + 1, G_3 = (dir + 1) % 3 + 1;
    const int U_1 = UU + G_1, U_2 = UU + G_2, U_3 = UU + G_3;
    const int B_1 = B1 + G_1 - 1, B_2 = B1 + G_2 - 1, B_3 = B1 + G_3 - 1;
    T vcon[4];
    vcon[0] = T(0.);
    bool fail = false;
    const T A = -FH[1][UU] - (FH[0][B_2] * FH[1][B_2] + FH[0][B_3] * FH[1][B_3]);
    const T B = -FH[1][U_1] + FH[0][UU] + (FH[0][B_2] * FH[0][B_2] + FH[0][B_3] * FH[0][B_3]) +
                (FH[1][B_2] * FH[1][B_2] + FH[1][B_3] * FH[1][B_3]);
    const T C = FH[0][U_1] - (FH[0][B_2] * FH[1][B_2] + FH[0][B_3] * FH[1][B_3]);
    const T D = B * B - T(4.) * A * C;
    vcon[G_1] = (-B - d_sqrt(D)) / (T(2.) * A);
    const Divisor<T> db(FH[0][B_1]);
    vcon[G_2] = db.div(FH[0][B_2] * vcon[G_1] - FH[1][B_2]);
    vcon[G_3] = db.div(FH[0][B_3] * vcon[G_1] - FH[1][B_3]);
    const T gammasq = T(1.) / (T(1.) - (vcon[1] * vcon[1] + vcon[2] * vcon[2] + vcon[3] * vcon[3]));
    const Divisor<T> dg(gammasq);
    const T vB = (vcon[1] * FH[0][B1] + vcon[2] * FH[0][B2] + vcon[3] * FH[0][B3]);
    const T ptot = -(-FH[1][UU] - FH[0][B_1] * (vB)) * vcon[dir] + FH[1][U_1] + dg.div(FH[0][B_1] * FH[0][B_1]);   // pow(x, 2): x*x is its correctly rounded value
    if (!(d_fabs(ptot) > T(0.)) || (vcon[G_1] < cmin) || (vcon[G_1] > cmax) || !(d_fabs(vcon[G_1]) > T(0.))) fail = true;
    if (cmax > iv && vcon[dir] <= iv && !fail) {
        const Divisor<T> dc(cmax - vcon[dir] + T(SMALL_D));
        FT[0][RHO] = dc.div(cmax - ru[dir] / ru[0]) * Ur[RHO];
        FT[0][UU] = dc.div(cmax * Ur[UU] + Ur[U_1] - ptot * vcon[dir] + vB * FH[0][B_1]);
        FT[0][U_1] = (-FT[0][UU] + ptot) * vcon[dir] - vB * FH[0][B_1];
        FT[0][U_2] = dc.div(-FH[0][B_1] * (dg.div(FH[0][B_2]) + vB * vcon[G_2]) + cmax * Ur[U_2] - Fr[U_2]);
        FT[0][U_3] = dc.div(-FH[0][B_1] * (dg.div(FH[0][B_3]) + vB * vcon[G_3]) + cmax * Ur[U_3] - Fr[U_3]);
        FT[0][B_1] = FH[0][B_1];
        FT[0][B_2] = FH[0][B_2];
        FT[0][B_3] = FH[0][B_3];
        FT[0][KTOT] = dc.div(cmax - ru[dir] / ru[0]) * Ur[KTOT];
        for (int k = 0; k < NPR; k++) FT[1][k] = (Fr[k] + cmax * (FT[0][k] - Ur[k]));
    } else if (cmin < iv && vcon[dir] >= iv && !fail) {
        const Divisor<T> dc(cmin - vcon[dir] + T(SMALL_D));
        FT[0][RHO] = dc.div(cmin - lu[dir] / lu[0]) * Ul[RHO];
        FT[0][UU] = dc.div(cmin * Ul[UU] + Ul[U_1] - ptot * vcon[dir] + vB * FH[0][B_1]);
        FT[0][U_1] = (-FT[0][UU] + ptot) * vcon[dir] - vB * FH[0][B_1];
        FT[0][U_2] = dc.div(-FH[0][B_1] * (dg.div(FH[0][B_2]) + vB * vcon[G_2]) + cmin * Ul[U_2] - Fl[U_2]);
        FT[0][U_3] = dc.div(-FH[0][B_1] * (dg.div(FH[0][B_3]) + vB * vcon[G_3]) + cmin * Ul[U_3] - Fl[U_3]);
        FT[0][B_1] = FH[0][B_1];
        FT[0][B_2] = FH[0][B_2];
        FT[0][B_3] = FH[0][B_3];
        FT[0][KTOT] = dc.div(cmin - lu[dir] / lu[0]) * Ul[KTOT];
        for (int k = 0; k < NPR; k++) FT[1][k] = (Fl[k] + cmin * (FT[0][k] - Ul[k]));
    } else {
        for (int k = 0; k < NPR; k++) { FT[0][k] = FH[0][k]; FT[1][k] = FH[1][k]; }
    }
}

// HLLD (calc_HLLD and helpers, GPU_hllc.h:398-876; HLLD builds, marked "Does
// not work yet" in the reference's config.h:482), in the operation order of
// the reference, including its two slips that shape the result: G adds the
// second transverse residual instead of its square (GPU_hllc.h:808,822), and
// the right intermediate speed check takes vcon_ar[3] * vcon_al[3]
// (GPU_hllc.h:673).
template <typename T>
struct HlldFan {
    T K_al[4], B_al[4], K_ar[4], B_ar[4], v_al[4], v_ar[4], v_cl[4], v_cr[4], B_c[4];
    T eta_l, eta_r, w_al, w_ar;
};

// one side's outer intermediate state and Alfven K vector for a total
// pressure guess (the first half of calc_error_HLLD for side S = cmin or cmax)
template <typename T>
__device__ __forceinline__ void hlld_side(int dir, T ptot, T S, T sgn, T BX, const T *R, T *v, T *Bs, T *K, T &w,
                                          T &eta) {
    const int G_1 = dir, G_2 = dir % 3 + 1, G_3 = (dir + 1) % 3 + 1;
    const int U_1 = UU + G_1, U_2 = UU + G_2, U_3 = UU + G_3;
    const int B_1 = B1 + G_1 - 1, B_2 = B1 + G_2 - 1, B_3 = B1 + G_3 - 1;
    const T A = R[U_1] + S * R[UU] + ptot * (T(1.) - S * S);
    const T G = R[B_2] * R[B_2] + R[B_3] + R[B_3];
    const T C = R[U_2] * R[B_2] + R[U_3] * R[B_3];
    const T Q = -A - G + (BX * BX) * (T(1.) - S * S);
    const T X = BX * (A * S * BX + C) - (A + G) * (S * ptot - R[UU]);
    const ExactDivisor<T> dX(X);   // quotients sharing a divisor (exact form in FP64)
    v[G_1] = dX.div(BX * (A * BX + S * C) - (A + G) * (ptot + R[U_1]));
    v[G_2] = dX.div(Q * R[U_2] + R[B_2] * (C + BX * (S * R[U_1] + R[UU])));
    v[G_3] = dX.div(Q * R[U_3] + R[B_3] * (C + BX * (S * R[U_1] + R[UU])));
    w = ptot + (-R[UU] - (v[G_1] * R[U_1] + v[G_2] * R[U_2] + v[G_3] * R[U_3])) / (S - v[G_1] + T(SMALL_D));
    Bs[G_1] = BX;
    const ExactDivisor<T> dS(S - v[G_1]);
    Bs[G_2] = dS.div(R[B_2] - Bs[G_1] * v[G_2]);
    Bs[G_3] = dS.div(R[B_3] - Bs[G_1] * v[G_3]);
    eta = sgn * ((T)(BX > T(0.0)) - (T)(BX <= T(0.0))) * d_sqrt(d_fabs(w));
    const ExactDivisor<T> dden(S * ptot - R[UU] + BX * eta);
    K[G_1] = dden.div(R[U_1] + ptot + R[B_1] * eta);
    K[G_2] = dden.div(R[U_2] + R[B_2] * eta);
    K[G_3] = dden.div(R[U_3] + R[B_3] * eta);
}

// calc_error_HLLD (GPU_hllc.h:685-876, its live second half)
template <typename T>
__device__ __forceinline__ T hlld_error(int dir, T ptot, T cmin, T cmax, T BX, const T *R_l, const T *R_r,
                                        HlldFan<T> &f) {
    const int G_1 = dir, G_2 = dir % 3 + 1, G_3 = (dir + 1) % 3 + 1;
    hlld_side(dir, ptot, cmin, T(-1.), BX, R_l, f.v_al, f.B_al, f.K_al, f.w_al, f.eta_l);
    hlld_side(dir, ptot, cmax, T(1.), BX, R_r, f.v_ar, f.B_ar, f.K_ar, f.w_ar, f.eta_r);
    f.B_c[G_1] = BX;
    const ExactDivisor<T> dK(f.K_ar[dir] - f.K_al[dir] + T(1e-12));
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int Gt = t ? G_3 : G_2;
        f.B_c[Gt] = dK.div((f.B_ar[Gt] * (f.K_ar[G_1] - f.v_ar[dir]) + f.B_ar[dir] * f.v_ar[Gt]) -
                           (f.B_al[Gt] * (f.K_al[G_1] - f.v_al[dir]) + f.B_al[dir] * f.v_al[Gt]));
    }
    const T delta_Kx = (f.K_ar[dir] - f.K_al[dir]);
    T B_hat[4];
    B_hat[1] = delta_Kx * f.B_c[1];
    B_hat[2] = delta_Kx * f.B_c[2];
    B_hat[3] = delta_Kx * f.B_c[3];
    const T kl2 = f.K_al[1] * f.K_al[1] + f.K_al[2] * f.K_al[2] + f.K_al[3] * f.K_al[3];
    const T kr2 = f.K_ar[1] * f.K_ar[1] + f.K_ar[2] * f.K_ar[2] + f.K_ar[3] * f.K_ar[3];
    const T Y_l = (T(1.) - kl2) / (f.eta_l * delta_Kx - (f.K_al[1] * B_hat[1] + f.K_al[2] * B_hat[2] + f.K_al[3] * B_hat[3]));
    const T Y_r = (T(1.) - kr2) / (f.eta_r * delta_Kx - (f.K_ar[1] * B_hat[1] + f.K_ar[2] * B_hat[2] + f.K_ar[3] * B_hat[3]));
    const T error = delta_Kx * (T(1.) - f.B_ar[dir] * (Y_r - Y_l));
    const T kbl = f.eta_l - (f.K_al[1] * f.B_c[1] + f.K_al[2] * f.B_c[2] + f.K_al[3] * f.B_c[3]);
    const T kbr = f.eta_r - (f.K_ar[1] * f.B_c[1] + f.K_ar[2] * f.B_c[2] + f.K_ar[3] * f.B_c[3]);
    const ExactDivisor<T> dkl(kbl), dkr(kbr);
#pragma unroll
    for (int q = 1; q < 4; q++) {
        f.v_cl[q] = (f.K_al[q] - dkl.div(f.B_c[q] * (T(1.) - kl2)));
        f.v_cr[q] = (f.K_ar[q] - dkr.div(f.B_c[q] * (T(1.) - kr2)));
    }
    f.v_cl[dir] = (f.v_cl[dir] + f.v_cr[dir]) * T(0.5);
    f.v_cr[dir] = f.v_cl[dir];
    return error;
}

// calc_HLLD_pres (GPU_hllc.h:425-531): HLLC estimate of the total pressure,
// then at most 12 secant-Newton steps on hlld_error
template <typename T>
__device__ __noinline__ T hlld_pres(int dir, int &fail_c, int &fail_d, T cmin, T cmax, const T FH[2][NPR], const T *R_l,
                                    const T *R_r, HlldFan<T> &f) {
    const int G_1 = dir, G_2 = dir % 3 + 1, G_3 = (dir + 1) % 3 + 1;
    const int U_1 = UU + G_1;
    const int B_1 = B1 + G_1 - 1, B_2 = B1 + G_2 - 1, B_3 = B1 + G_3 - 1;
    T vcon[4];
    vcon[0] = T(0.);
    T A = -FH[1][UU] - (FH[0][B_2] * FH[1][B_2] + FH[0][B_3] * FH[1][B_3]);
    T B = -FH[1][U_1] + FH[0][UU] + (FH[0][B_2] * FH[0][B_2] + FH[0][B_3] * FH[0][B_3]) +
          (FH[1][B_2] * FH[1][B_2] + FH[1][B_3] * FH[1][B_3]);
    T C = FH[0][U_1] - (FH[0][B_2] * FH[1][B_2] + FH[0][B_3] * FH[1][B_3]);
    T D = B * B - T(4.) * A * C;
    vcon[G_1] = (-B - d_sqrt(d_max(T(0.), D))) / (T(2.) * A);
    vcon[G_2] = (FH[0][B_2] * vcon[G_1] - FH[1][B_2]) / FH[0][B_1];
    vcon[G_3] = (FH[0][B_3] * vcon[G_1] - FH[1][B_3]) / FH[0][B_1];
    const T gammasq = T(1.) / (T(1.) - (vcon[1] * vcon[1] + vcon[2] * vcon[2] + vcon[3] * vcon[3]));
    if ((vcon[dir] < cmin) || (vcon[dir] > cmax) || !(d_fabs(vcon[dir]) > T(0.))) fail_c = 1;
    const T v_dot_B = (vcon[1] * FH[0][B1] + vcon[2] * FH[0][B2] + vcon[3] * FH[0][B3]);
    const T ptot_HLLC =
        -(-FH[1][UU] - FH[0][B_1] * (v_dot_B)) * vcon[dir] + FH[1][U_1] + FH[0][B_1] * FH[0][B_1] / gammasq;
    T ptot = ptot_HLLC;
    if (!(d_fabs(ptot) > T(0.))) {
        // hydrodynamic estimate
        fail_c = 1;
        A = T(1.);
        B = (-FH[0][UU] - FH[1][U_1]);
        C = -FH[0][U_1] * FH[1][UU] + FH[1][U_1] * FH[0][UU];
        D = B * B - T(4.) * A * C;
        ptot = (-B + d_sqrt(d_max(T(0.), D))) / (T(2.) * A);
        if (!(d_fabs(ptot) > T(0.))) {
            fail_d = 1;
            return T(-10.);
        }
    }
    T ptot_old = ptot, d_ptot = T(0.);
    T error_1 = hlld_error(dir, ptot, cmin, cmax, FH[0][B_1], R_l, R_r, f);
    for (int n_iter = 0;; n_iter++) {
        const T error_2 = hlld_error(dir, ptot + T(1e-10) * d_fabs(ptot), cmin, cmax, FH[0][B_1], R_l, R_r, f);
        ptot_old = ptot;
        const T de_dptot = (error_2 - error_1) / (T(1e-10) * d_fabs(ptot));
        d_ptot = error_1 / de_dptot;
        ptot = ptot - d_ptot;
        if (ptot < T(0.)) ptot = T(0.5) * d_fabs(ptot);
        error_1 = hlld_error(dir, ptot, cmin, cmax, FH[0][B_1], R_l, R_r, f);
        if ((d_fabs(ptot - ptot_old) <= T(1e-8) * d_fabs(ptot + ptot_old)) || n_iter > 10) break;
    }
    if (!(d_fabs(ptot) > T(0.)) || ((d_fabs(d_ptot) > T(1e-8) * d_fabs(ptot + ptot_old)))) {
        ptot = ptot_HLLC;
        fail_d = 1;
    }
    return ptot;
}

// check_HLLD_par (GPU_hllc.h:635-683); true to reject the fan
template <typename T>
__device__ __forceinline__ bool hlld_check(int dir, T cmin, T cmax, T ptot, HlldFan<T> &f) {
    const int G_1 = dir;
    bool fail = false;
#pragma unroll
    for (int t = 0; t < 3; t++) {
        const int Gt = t == 0 ? G_1 : (t == 1 ? dir % 3 + 1 : (dir + 1) % 3 + 1);
        f.v_cl[Gt] = (f.v_cl[Gt] + f.v_cr[Gt]) * T(0.5);
        f.v_cr[Gt] = f.v_cl[Gt];
    }
    if (f.v_cl[G_1] < f.K_al[G_1] || f.v_cl[G_1] < cmin) fail = true;
    if (f.v_cl[G_1] > f.K_ar[G_1] || f.v_cl[G_1] > cmax) fail = true;
    T vsq = (f.v_cl[1] * f.v_cl[1] + f.v_cl[2] * f.v_cl[2] + f.v_cl[3] * f.v_cl[3]);
    if (!(vsq < T(0.999))) fail = true;
    if (d_fabs(f.w_al) <= d_fabs(ptot) || f.v_al[G_1] <= cmin || f.K_al[G_1] <= cmin || f.w_al <= T(0.)) fail = true;
    if (d_fabs(f.w_ar) <= d_fabs(ptot) || f.v_ar[G_1] >= cmax || f.K_ar[G_1] >= cmax || f.w_ar <= T(0.)) fail = true;
    vsq = (f.v_al[1] * f.v_al[1] + f.v_al[2] * f.v_al[2] + f.v_al[3] * f.v_al[3]);
    if (!(vsq < T(0.999))) fail = true;
    vsq = (f.v_ar[1] * f.v_ar[1] + f.v_ar[2] * f.v_ar[2] + f.v_ar[3] * f.v_al[3]);
    if (!(vsq < T(0.999))) fail = true;
    vsq = (f.K_al[1] * f.K_al[1] + f.K_al[2] * f.K_al[2] + f.K_al[3] * f.K_al[3]);
    if (!(vsq < T(0.999))) fail = true;
    vsq = (f.K_ar[1] * f.K_ar[1] + f.K_ar[2] * f.K_ar[2] + f.K_ar[3] * f.K_ar[3]);
    if (!(vsq < T(0.999))) fail = true;
    return fail;
}

// outer intermediate state (between the fast and Alfven waves) of side S
template <typename T>
__device__ __forceinline__ void hlld_outer(int dir, T S, const T *R, T ptot, const T *v, const T *Bs, T BX, T *X) {
    const int G_1 = dir, G_2 = dir % 3 + 1, G_3 = (dir + 1) % 3 + 1;
    const T v_dot_B = v[1] * Bs[1] + v[2] * Bs[2] + v[3] * Bs[3];
    const ExactDivisor<T> dS(S - v[G_1]);
    X[RHO] = dS.div(R[RHO]);
    X[UU] = (R[UU] - ptot * v[G_1] + v_dot_B * Bs[G_1]) / (S - v[G_1] + T(SMALL_D));
    X[UU + G_1] = (-X[UU] + ptot) * v[G_1] - v_dot_B * Bs[G_1];
    X[UU + G_2] = (-X[UU] + ptot) * v[G_2] - v_dot_B * Bs[G_2];
    X[UU + G_3] = (-X[UU] + ptot) * v[G_3] - v_dot_B * Bs[G_3];
    X[B1 + G_1 - 1] = BX;
    X[B1 + G_2 - 1] = Bs[G_2];
    X[B1 + G_3 - 1] = Bs[G_3];
    X[KTOT] = dS.div(R[KTOT]);
}

// inner intermediate state (between the Alfven wave and the contact)
template <typename T>
__device__ __forceinline__ void hlld_inner(int dir, const T *Xa, T Ka, const T *va, T ptot, const T *vc, const T *Bc,
                                           T BX, T *X) {
    const int G_1 = dir, G_2 = dir % 3 + 1, G_3 = (dir + 1) % 3 + 1;
    const T v_dot_B = vc[1] * Bc[1] + vc[2] * Bc[2] + vc[3] * Bc[3];
    const ExactDivisor<T> dK(Ka - vc[G_1]);
    X[RHO] = dK.div(Xa[RHO] * (Ka - va[G_1]));
    X[UU] = dK.div(-(-Ka * Xa[UU] - Xa[UU + G_1] + ptot * vc[G_1] - v_dot_B * Xa[B1 + G_1 - 1]));
    X[UU + G_1] = (-Xa[UU] + ptot) * vc[G_1] - v_dot_B * Bc[G_1];
    X[UU + G_2] = (-Xa[UU] + ptot) * vc[G_2] - v_dot_B * Bc[G_2];
    X[UU + G_3] = (-Xa[UU] + ptot) * vc[G_3] - v_dot_B * Bc[G_3];
    X[B1 + G_1 - 1] = BX;
    X[B1 + G_2 - 1] = Bc[G_2];
    X[B1 + G_3 - 1] = Bc[G_3];
    X[KTOT] = dK.div(Xa[KTOT] * (Ka - va[G_1]));
}

// calc_HLLD (GPU_hllc.h:398-423): HLLD star fluxes where the fan passes every
// check, else HLLC where its estimate held, else HLL. The face at exactly
// the right Alfven speed (iv == K_ar), where the reference leaves the flux
// unset, takes HLL.
template <typename T>
__device__ __noinline__ void hlld_mhd(int dir, const T *lu, const T *ru, T iv, T cmin, T cmax, T FT[2][NPR],
                                      const T FH[2][NPR], const T *Fl, const T *Fr, const T *Ul, const T *Ur) {
    T R_l[NPR], R_r[NPR];
    HlldFan<T> f;
    int fail_c = 0, fail_d = 0;
    for (int k = 0; k < NPR; k++) R_l[k] = (cmin * Ul[k] - Fl[k]);
    for (int k = 0; k < NPR; k++) R_r[k] = (cmax * Ur[k] - Fr[k]);
    const T ptot = hlld_pres(dir, fail_c, fail_d, cmin, cmax, FH, R_l, R_r, f);
    if (fail_d == 0 && hlld_check(dir, cmin, cmax, ptot, f)) fail_d = 1;
    if (fail_d == 0) {
        const T BX = FH[0][B1 + dir - 1];
        T X_a[NPR], X_c[NPR];
        if ((cmin < iv) && (iv <= f.K_al[dir])) {
            hlld_outer(dir, cmin, R_l, ptot, f.v_al, f.B_al, BX, X_a);
            for (int k = 0; k < NPR; k++) { FT[0][k] = X_a[k]; FT[1][k] = Fl[k] + cmin * (X_a[k] - Ul[k]); }
        } else if ((f.K_al[dir] < iv) && (iv <= f.v_cl[dir])) {
            hlld_outer(dir, cmin, R_l, ptot, f.v_al, f.B_al, BX, X_a);
            hlld_inner(dir, X_a, f.K_al[dir], f.v_al, ptot, f.v_cl, f.B_c, BX, X_c);
            for (int k = 0; k < NPR; k++) {
                FT[0][k] = X_c[k];
                FT[1][k] = Fl[k] + cmin * (X_a[k] - Ul[k]) + f.K_al[dir] * (X_c[k] - X_a[k]);
            }
        } else if ((f.v_cr[dir] <= iv) && (iv < f.K_ar[dir])) {
            hlld_outer(dir, cmax, R_r, ptot, f.v_ar, f.B_ar, BX, X_a);
            hlld_inner(dir, X_a, f.K_ar[dir], f.v_ar, ptot, f.v_cr, f.B_c, BX, X_c);
            for (int k = 0; k < NPR; k++) {
                FT[0][k] = X_c[k];
                FT[1][k] = Fr[k] + cmax * (X_a[k] - Ur[k]) + f.K_ar[dir] * (X_c[k] - X_a[k]);
            }
        } else if ((cmax > iv) && (iv > f.K_ar[dir])) {
            hlld_outer(dir, cmax, R_r, ptot, f.v_ar, f.B_ar, BX, X_a);
            for (int k = 0; k < NPR; k++) { FT[0][k] = X_a[k]; FT[1][k] = Fr[k] + cmax * (X_a[k] - Ur[k]); }
        } else {
            for (int k = 0; k < NPR; k++) { FT[0][k] = FH[0][k]; FT[1][k] = FH[1][k]; }
        }
    } else if (fail_c == 0) {
        hllc_mhd(dir, lu, ru, iv, cmin, cmax, FT, FH, Fl, Fr, Ul, Ur);
    } else {
        for (int k = 0; k < NPR; k++) { FT[0][k] = FH[0][k]; FT[1][k] = FH[1][k]; }
    }
}

// HLLC flux of one face (states carry the normal field already); returns ctop
// from the coordinate-frame fast speeds, as the HLL path
template <int DIR, typename T, bool HLLD = false>
__device__ __forceinline__ T hllc_face(T gam, const T *pl, const T *pr, const Geo<T> &gm, T *Fout) {
    State<T> ql, qr;
    T cmax_l, cmin_l, cmax_r, cmin_r, vd[NPR];
    get_state(pl, gm, ql);
    get_state(pr, gm, qr);
    primtoflux(gam, pl, ql, DIR, gm, T(0.), vd, &cmax_l, &cmin_l);
    primtoflux(gam, pr, qr, DIR, gm, T(0.), vd, &cmax_r, &cmin_r);
    const T cmax1 = d_fabs(d_max(d_max(T(0.), cmax_l), cmax_r));
    const T cmin1 = d_fabs(d_max(d_max(T(0.), -cmin_l), -cmin_r));
    const T ctop = d_max(cmax1, cmin1);
    T Mud[4][4], Mi[4][4];
    set_mud(gm, DIR, Mud, Mi);
    T lu[4], lb[4], ru[4], rb[4];
    for (int a = 0; a < 4; a++) {
        lu[a] = T(0.0); lb[a] = T(0.0); ru[a] = T(0.0); rb[a] = T(0.0);
        for (int b = 0; b < 4; b++) {
            lu[a] += ql.ucon[b] * Mi[a][b];
            lb[a] += ql.bcon[b] * Mi[a][b];
            ru[a] += qr.ucon[b] * Mi[a][b];
            rb[a] += qr.bcon[b] * Mi[a][b];
        }
    }
    T Fl[NPR], Fr[NPR], Ul[NPR], Ur[NPR], FT[2][NPR], FH[2][NPR];
    primtoflux_ft(gam, pl, lu, lb, DIR, Fl);
    primtoflux_ft(gam, pr, ru, rb, DIR, Fr);
    primtoflux_ft(gam, pl, lu, lb, 0, Ul);
    primtoflux_ft(gam, pr, ru, rb, 0, Ur);
    vchar_ft(gam, pl, lu, lb, DIR, &cmax_l, &cmin_l);
    vchar_ft(gam, pr, ru, rb, DIR, &cmax_r, &cmin_r);
    const T cmax = d_max(cmax_r, cmax_l);
    const T cmin = d_min(cmin_r, cmin_l);
    constexpr int sdd = DIR == 1 ? 4 : (DIR == 2 ? 7 : 9);
    const T iv = gm.gcon[DIR] / (d_sqrt(gm.gcon[DIR] * gm.gcon[DIR] - gm.gcon[0] * gm.gcon[sdd]));
    if (cmax <= iv) {
        for (int k = 0; k < NPR; k++) { FT[0][k] = Ur[k]; FT[1][k] = Fr[k]; }
    } else if (cmin >= iv) {
        for (int k = 0; k < NPR; k++) { FT[0][k] = Ul[k]; FT[1][k] = Fl[k]; }
    } else {
        const Divisor<T> dh(cmax - cmin + T(SMALL_D));   // the 18 HLL-state quotients share it
        for (int k = 0; k < NPR; k++) FH[0][k] = dh.div(Fl[k] - Fr[k] + cmax * Ur[k] - cmin * Ul[k]);
        for (int k = 0; k < NPR; k++)
            FH[1][k] = dh.div(cmax * Fl[k] - cmin * Fr[k] + cmax * cmin * (Ur[k] - Ul[k]));
        const bool do_hydro = d_fabs(FH[0][DIR + B1 - 1] * FH[0][DIR + B1 - 1] * lu[0] * ru[0]) < T(1.e-10) * d_fabs(FH[0][UU]);
        if (do_hydro) hllc_hydro(DIR, lu, ru, iv, cmin, cmax, FT, FH, Fl, Fr, Ul, Ur);
        else if constexpr (HLLD) hlld_mhd(DIR, lu, ru, iv, cmin, cmax, FT, FH, Fl, Fr, Ul, Ur);
        else hllc_mhd(DIR, lu, ru, iv, cmin, cmax, FT, FH, Fl, Fr, Ul, Ur);
    }
    T F1[NPR];
    for (int j1 = 0; j1 < 4; j1++) {
        F1[j1 + UU] = T(0.);
        for (int j2 = 0; j2 < 4; j2++) {
            F1[j1 + UU] += FT[0][j2 + UU] * Mud[DIR][0] * Mi[j2][j1];
            F1[j1 + UU] += FT[1][j2 + UU] * Mud[DIR][DIR] * Mi[j2][j1];
        }
    }
    FT[0][U3] = T(0.);
    FT[1][U3] = -FT[0][B1 - 1 + DIR];
    for (int j1 = 1; j1 < 4; j1++) {
        F1[j1 + U3] = T(0.);
        for (int j2 = 0; j2 < 4; j2++) {
            F1[j1 + U3] += FT[0][j2 + U3] * Mud[DIR][0] * Mud[j1][j2];
            F1[j1 + U3] += FT[1][j2 + U3] * Mud[DIR][DIR] * Mud[j1][j2];
        }
    }
    F1[RHO] = FT[0][RHO] * Mud[DIR][0];
    F1[RHO] += FT[1][RHO] * Mud[DIR][DIR];
    F1[KTOT] = FT[0][KTOT] * Mud[DIR][0];
    F1[KTOT] += FT[1][KTOT] * Mud[DIR][DIR];
    F1[UU] += F1[RHO];
    for (int k = 0; k < NPR; k++) Fout[k] = gm.g * F1[k];
    return ctop;
}

// ---------------------------------------------------------------- floors
// Opt-in floors: the drift-frame floor of fixup_cell for an ideal gas
// without radiation or a neutron star (GPU_fixup.h:1025-1800; the same
// algorithm as fixup1zone, fixup.c:57-664). Both bodies are compiled out
// (#if 0) in the reference, whose shipped step applies no floor. Constants
// of the torus build (config.h:274-287, 533).
constexpr double RHOMINLIMIT = 1.e-20;
constexpr double UUMINLIMIT = 1.e-20;
constexpr double BSQORHOMAX = 25.;
constexpr double BSQOUMAX = 750.;
constexpr double UORHOMAX = 150.;
constexpr double GAMMAMAX = 80.;

// Lorentz factor w.r.t. the normal observer with its failure flag
// (gamma_calc, GPU_phys_mhd.h:740-761)
__device__ __forceinline__ int gamma_calc_flag(const double *pr, const Geo<double> &gm, double *gamma) {
    const double *g = gm.gcov;
    double qsq = g[4] * pr[U1] * pr[U1] + g[7] * pr[U2] * pr[U2] + g[9] * pr[U3] * pr[U3]
               + 2. * (g[5] * pr[U1] * pr[U2] + g[6] * pr[U1] * pr[U3] + g[8] * pr[U2] * pr[U3]);
    if (qsq < 0.) {
        if (fabs(qsq) > 1.E-10) { *gamma = 1.; return 1; }
        qsq = 1.E-10;
    }
    *gamma = sqrt(1. + qsq);
    return 0;
}

// u^t from the coordinate 3-velocity v^i (ut_calc_3vel, GPU_phys_mhd.h:18-31)
__device__ __forceinline__ double ut_of_3vel(const double *vcon, const Geo<double> &gm) {
    const double *g = gm.gcov;
    const double AA = g[0];
    const double BB = 2. * (g[1] * vcon[1] + g[2] * vcon[2] + g[3] * vcon[3]);
    const double CC = g[4] * vcon[1] * vcon[1] + g[7] * vcon[2] * vcon[2] + g[9] * vcon[3] * vcon[3]
                    + 2. * (g[5] * vcon[1] * vcon[2] + g[6] * vcon[1] * vcon[3] + g[8] * vcon[2] * vcon[3]);
    double DD = -1. / (AA + BB + CC);
    const double one_over_alpha_sq = -gm.gcon[0];
    if (DD < one_over_alpha_sq) DD = one_over_alpha_sq;
    return sqrt(DD);
}

// True when the floors may change the zone: false only for a zone clearly
// above every floor and below the Lorentz cap, where floor_zone changes
// nothing and returns 0. b^2 = (B^i B_i + (B^i u_i)^2) / (u^t)^2 with
// u_i = g_ij u~^j and (u^t)^2 = (1 + u~^i u~_i) (-g^tt), all without a
// division or a square root; every test keeps a relative margin of 1e-6 (far
// above the rounding of either form of b^2), so a zone near a threshold goes
// to floor_zone, which decides exactly as the reference does.
__device__ __forceinline__ bool floor_may_apply(const double *pf, const Geo<double> &gm) {
    const double *g = gm.gcov;
    const double v1 = pf[U1], v2 = pf[U2], v3 = pf[U3];
    const double w1 = g[4] * v1 + g[5] * v2 + g[6] * v3;
    const double w2 = g[5] * v1 + g[7] * v2 + g[8] * v3;
    const double w3 = g[6] * v1 + g[8] * v2 + g[9] * v3;
    const double qsq = v1 * w1 + v2 * w2 + v3 * w3;
    const double b1 = pf[B1], b2 = pf[B2], b3 = pf[B3];
    const double BB = b1 * (g[4] * b1 + g[5] * b2 + g[6] * b3) + b2 * (g[5] * b1 + g[7] * b2 + g[8] * b3)
                    + b3 * (g[6] * b1 + g[8] * b2 + g[9] * b3);
    const double Bu = b1 * w1 + b2 * w2 + b3 * w3;
    const double num = (BB + Bu * Bu) * (1. + 1e-6);
    const double den = (1. + qsq) * -gm.gcon[0];
    const double rho = pf[RHO], u = pf[UU];
    if (qsq > -1e-11 && 1. + qsq < 6399. && rho > RHOMINLIMIT * (1. + 1e-6) && u > UUMINLIMIT * (1. + 1e-6) &&
        BSQORHOMAX * rho * den > num && BSQOUMAX * u * den > num && UORHOMAX * rho > u * (1. + 1e-6))
        return false;
    return true;
}

// Apply the floors to the primitives pf of one zone (centre metric gm).
// Returns 4 when the final Lorentz factor cannot be formed (the flag the
// fixup kernel turns into pflag = -333), else 0.
__device__ __noinline__ int floor_zone(double gam, double *pf, const Geo<double> &gm) {
    State<double> q;
    get_state(pf, gm, q);   // state before the floors
    const double bsq = dot4(q.bcon, q.bcov);
    double u = pf[UU];
    double pre[5];
#pragma unroll
    for (int k = 0; k < 5; k++) pre[k] = pf[k];
    double rhoflr = RHOMINLIMIT, uuflr = UUMINLIMIT;
    // tie the floors to the local field and internal energy
    if (rhoflr < bsq / BSQORHOMAX) rhoflr = bsq / (BSQORHOMAX);
    if (uuflr < bsq / BSQOUMAX) uuflr = bsq / (BSQOUMAX);
    if (rhoflr < u / UORHOMAX) rhoflr = u / (UORHOMAX);
    if (rhoflr < RHOMINLIMIT) rhoflr = RHOMINLIMIT;
    if (uuflr < UUMINLIMIT) uuflr = UUMINLIMIT;
    int dofloor = 0;
    if (pf[RHO] < rhoflr) { pf[RHO] = rhoflr; dofloor = 1; }
    if (u < uuflr) { pf[UU] = uuflr; u = uuflr; dofloor = 1; }
    // drift frame: keep the velocity perpendicular to B, set the parallel
    // part from B.Q of the state before the floors (Noble et al. 2006, eq. 26)
    double trans = 10. * bsq / (pf[RHO] < u ? pf[RHO] : u) - 1.;
    if (dofloor && trans > 0.) {
        if (trans > 1.) trans = 1.;
        const double betapar = -q.bcon[0] / ((bsq + SMALL_D) * q.ucon[0]);
        double betasq = betapar * betapar * bsq;
        const double betasqmax = 1. - 1. / (GAMMAMAX * GAMMAMAX);
        if (betasq > betasqmax) betasq = betasqmax;
        const double gamma = 1. / sqrt(1 - betasq);
        double ucondr[4], Bcon[4], Bcov[4], vcon[4];
#pragma unroll
        for (int m = 0; m < 4; m++) ucondr[m] = gamma * (q.ucon[m] + betapar * q.bcon[m]);
        Bcon[0] = 0.;
#pragma unroll
        for (int m = 1; m < 4; m++) Bcon[m] = pf[B1 - 1 + m];
        lower4(Bcon, gm.gcov, Bcov);
        const double udotB = dot4(q.ucon, Bcov);
        const double Bsq = dot4(Bcon, Bcov);
        const double B = sqrt(Bsq);
        const double wold = pre[RHO] + pre[UU] * gam;
        const double QdotB = udotB * wold * q.ucon[0];
        const double wnew = pf[RHO] + pf[UU] * gam;
        const double x = 2. * QdotB / (B * wnew * ucondr[0] + SMALL_D);
        const double vpar = x / (ucondr[0] * (1. + sqrt(1. + x * x)));
        const double one_over_ucondr_t = 1. / ucondr[0];
        vcon[0] = 1.;
#pragma unroll
        for (int m = 1; m < 4; m++) vcon[m] = vpar * Bcon[m] / (B + SMALL_D) + ucondr[m] * one_over_ucondr_t;
        const double ut = ut_of_3vel(vcon, gm);
        // u^mu = u^t v^mu, then the relative 4-velocity u~^i = u^i + gamma beta^i / alpha
        // (ucon_to_utcon, GPU_phys_mhd.h:3-15)
        const double alpha = 1. / sqrt(-gm.gcon[0]);
        const double gam_n = alpha * (ut * vcon[0]);
#pragma unroll
        for (int m = 1; m < 4; m++) {
            const double utcon = ut * vcon[m] + gam_n * (gm.gcon[m] * alpha * alpha) / alpha;
            pf[m + UU] = utcon * trans + pre[m + UU] * (1. - trans);
        }
    }
    // limit the Lorentz factor w.r.t. the normal observer
    double gamma;
    if (gamma_calc_flag(pf, gm, &gamma)) return 4;
    if (gamma > GAMMAMAX) {
        const double f = sqrt((GAMMAMAX * GAMMAMAX - 1.) / (gamma * gamma - 1.));
        pf[U1] *= f;
        pf[U2] *= f;
        pf[U3] *= f;
    }
    return 0;
}

}  // namespace hamr
