// bia_pair.cuh -- per-pair BIA solvers in FP64 for sm_100a.
//
// One unordered pair (i, j) with relative state r = x_i - x_j, g = v_i - v_j is
// reduced to a planar two-body problem (bia/bia.f90:284-314), classified by its
// energy (bia/bia.f90:156-166) and advanced over dt by the hyperbola, parabola or
// ellipse solver (bia/find_hyperbola.f90, find_parabola.f90, find_ellipse.f90) or by
// the per-pair RKF4(5) (bia/find_dXYUV_RKF.f90).  The result is the pair's
// half-displacement h (bia/bia.f90:173-185): i receives +h, j receives -h.
//
// The formulas follow the reference's CPU path; CUDA's double-precision math
// functions replace glibc's, and nvcc's FMA contraction is left on, so results agree
// with the CPU oracle to rounding, not bit for bit.  The same deviations as the
// oracle are taken where the reference is undefined or fails in FP64: uninitialised
// theta_stock, bracket exit without a result, iterations that end unconverged
// (bracketed re-solve), and pairs with zero |g| or |L| or with |e^2 - 1| < 0.1 (the
// classical parametrisations lose up to every digit there), which are advanced by a
// universal-variable (Stumpff function) solver.
#pragma once
#include <cstdint>

namespace bia {

constexpr double kPi = 3.14159265358979323846264338327950288419716939937510582097494;

enum PairClass { kHyperbola = 0, kParabola = 1, kEllipse = 2, kDegenerate = 3, kRkf = 4, kUniversal = 5 };

// |e^2 - 1| below which ALG pairs use the universal-variable solver
constexpr double kNearUnitEcc = 0.1;

struct PairParams {
    double dt;
    double err;      // ERR, residual threshold for the not-converged count
    double relerr;   // RKF tolerances
    double abserr;
    int itr;         // Newton cap ITR
    int method;      // 0 RKF, 1 ALG, 2 universal variables for every pair
};

// Per-thread counters, reduced per warp before one atomic per counter.
struct PairCounters {
    int cls[6];
    int it_hyp, it_ell, it_par, it_uv;
    int rkf_steps;
    int nonconverged;
    int bracket_exits;
    int fallbacks;
    int nonfinite;
    int learned, learned_fallbacks, learned_coarse;  // BIA_METHOD_LEARNED
    int timeouts;
    int learned_fp32;  // FP32 Newton steps of the learned pairs' first correction
};

__device__ __forceinline__ void counters_zero(PairCounters &c)
{
#pragma unroll
    for (int k = 0; k < 6; k++) c.cls[k] = 0;
    c.it_hyp = c.it_ell = c.it_par = c.it_uv = 0;
    c.rkf_steps = c.nonconverged = c.bracket_exits = c.fallbacks = c.nonfinite = 0;
    c.learned = c.learned_fallbacks = c.learned_coarse = c.timeouts = c.learned_fp32 = 0;
}

// 1/sqrt(x) of a normal x: the hardware approximation and one step
// of Householder's third-order iteration y (1 + e/2 + 3/8 e^2), e = 1 - x y^2 (measured
// at most 2^-19.04 over 1e9 values; the next term, 5/16 e^3, is below 3e-18).  Zero, subnormal
// and infinite x give NaN or infinity: its callers test for them.
__device__ __forceinline__ double rsqrt_normal(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-__dmul_rn(x, y), y, 1.0);
    return fma(fma(e, 0.375, 0.5), __dmul_rn(y, e), y);
}

// The same of any x.
static __device__ __noinline__ double rsqrt_small(double x) { return rsqrt(x); }
__device__ __forceinline__ double rsqrt_any(double x) { return x > 1e-290 ? rsqrt_normal(x) : rsqrt_small(x); }

// c x^(-3/2) of a normal x from the same approximation y, whose square is exact (its low half is zero), and one step
// of Householder's third-order iteration: c y^3 (1 + 3/2 e + 15/8 e^2), e = 1 - x y^2; the next term, 35/16 e^3,
// is below 3e-17.
__device__ __forceinline__ double scaled_rsqrt3_normal(double c, double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double y2 = y * y;
    const double e = fma(-x, y2, 1.0);
    const double c3 = (c * y) * y2;
    return fma(c3 * e, fma(e, 1.875, 1.5), c3);
}

// 1/x of a normal x with a normal reciprocal: the hardware approximation y and one step of Householder's
// third-order iteration, y (1 + e + e^2), e = 1 - x y (the next term, e^3, is below 1e-17).  Zero gives NaN; 2^1022
// and beyond, whose reciprocals are subnormal, give 0, which a Newton step must not take for a root (uv_iterate).
__device__ __forceinline__ double rcp_normal(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// Uncontracted IEEE operations: the frame is formed as the CPU path forms it.
__device__ __forceinline__ double m_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double a_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double s_(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double d_(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double dot3_(const double a[3], const double b[3])
{
    return a_(a_(m_(a[0], b[0]), m_(a[1], b[1])), m_(a[2], b[2]));
}

// bia/bia.f90:284-314.  Returns true for a degenerate pair (|g| == 0 or |L| == 0):
// then the frame is the line of motion and Y has a single nonzero position axis.
__device__ __forceinline__ bool frame_xi_eta(const double r[3], const double g[3], double e_xi[3],
                                             double e_eta[3], double Y[4])
{
    const double gsq = dot3_(g, g);
    const double gm = __dsqrt_rn(gsq);
    double L[3];
    L[0] = s_(m_(r[1], g[2]), m_(r[2], g[1]));
    L[1] = s_(m_(r[2], g[0]), m_(r[0], g[2]));
    L[2] = s_(m_(r[0], g[1]), m_(r[1], g[0]));
    const double Lsq = dot3_(L, L);
    if (gm == 0.0 || Lsq == 0.0) {
        if (gm == 0.0) {
            const double rm = __dsqrt_rn(dot3_(r, r));
#pragma unroll
            for (int k = 0; k < 3; k++) { e_xi[k] = d_(r[k], rm); e_eta[k] = 0.0; }
            Y[0] = rm; Y[1] = 0.0; Y[2] = 0.0; Y[3] = 0.0;
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++) { e_eta[k] = d_(g[k], gm); e_xi[k] = 0.0; }
            Y[0] = 0.0;
            Y[1] = dot3_(r, e_eta);
            Y[2] = 0.0;
            Y[3] = gm;
        }
        return true;
    }
    double ez[3];
    const double iL = rsqrt_any(Lsq);
    const double ig = rsqrt_any(gsq);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        e_eta[k] = g[k] * ig;
        ez[k] = L[k] * iL;
    }
    e_xi[0] = s_(m_(e_eta[1], ez[2]), m_(e_eta[2], ez[1]));
    e_xi[1] = s_(m_(e_eta[2], ez[0]), m_(e_eta[0], ez[2]));
    e_xi[2] = s_(m_(e_eta[0], ez[1]), m_(e_eta[1], ez[0]));
    Y[0] = dot3_(r, e_xi);
    Y[2] = 0.0;
    Y[1] = dot3_(r, e_eta);
    Y[3] = gm;
    return false;
}

// ---------------------------------------------------------------------------
// bia/find_hyperbola.f90:1-166.  Returns the main-loop iteration count.
//
// The reference's time equation and Newton iteration in theta, evaluated through the
// half angle: with (sh, ch) = sincos(theta/2) and (s0h, c0h) = sincos(theta_0/2),
//   sin((theta_0 +- theta)/2) = s0h ch +- c0h sh,  sin theta = 2 sh ch,
//   cos theta = 1 - 2 sh^2,  cos theta - cos theta_0 = 2 sin((theta_0+theta)/2) sin((theta_0-theta)/2),
// so one sincos replaces the reference's sin, sin and sincos per evaluation, and the
// denominator cos theta - cos theta_0 is a product instead of a difference.
// ---------------------------------------------------------------------------
constexpr double kFewUlps = 8.9e-16;  // four ulps of 1

struct HypConsts {
    double tn_0, cs_0, sn_0, s0h, c0h, time_end_;
};

// (sh, ch) of half an angle in (-pi, pi] from its sine and cosine, without cancellation
__device__ __forceinline__ void half_angle(double sn, double cs, double &sh, double &ch)
{
    const double t = fma(0.5, fabs(cs), 0.5);
    const double it = rsqrt_normal(t);
    const double big = t * it, small = 0.5 * sn * it;  // cos or sin of the half angle, and the other
    ch = cs >= 0.0 ? big : fabs(small);
    sh = cs >= 0.0 ? small : copysign(big, sn);
}

// find_theta (bia/find_hyperbola.f90:149-165): residual e and derivative d at theta;
// sp, sm = sin((theta_0 +- theta)/2) for the bracket test.  kFast: one reciprocal for
// 1/(2 sp sm) and sp/sm (sp sm inside the bracket, so not zero); else divisions, whose infinities
// at the bracket's ends hyp_safe needs.
template <bool kFast = true>
__device__ __forceinline__ void hyp_eval(const HypConsts &c, double theta, double &e, double &d,
                                         double &sp, double &sm)
{
    double sh, ch;
    sincos(0.5 * theta, &sh, &ch);
    sp = c.s0h * ch + c.c0h * sh;
    sm = c.s0h * ch - c.c0h * sh;
    double Dinv, ratio;
    if (kFast) {
        const double i = rcp_normal(sp * sm);
        Dinv = 0.5 * i;
        ratio = sp * sp * i;
    } else {
        Dinv = 1.0 / (2.0 * sp * sm);
        ratio = sp / sm;
    }
    const double sn = 2.0 * sh * ch;
    const double cs = 1.0 - 2.0 * sh * sh;
    e = c.tn_0 * sn * Dinv - c.time_end_ + log(ratio);
    d = c.tn_0 * (1.0 - c.cs_0 * cs) * (Dinv * Dinv) + c.sn_0 * Dinv;
}

// Bracketed Newton-bisection on the same time equation, used only when the reference's
// loop ends without a small residual.  The equation is monotonic on (-theta_0, theta_0):
// increasing for repulsive pairs (tn_0 > 0), decreasing for attractive ones.
static __device__ __noinline__ double hyp_safe(const HypConsts c, double x)
{
    const double theta_0 = atan2(c.sn_0, c.cs_0);
    double lo = -theta_0, hi = theta_0;
    const double dir = (c.tn_0 > 0.0) ? 1.0 : -1.0;
    if (!(x > lo && x < hi)) x = 0.0;
    for (int it = 0; it < 400; it++) {
        double f, d, sp, sm;
        hyp_eval<false>(c, x, f, d, sp, sm);
        if (f == 0.0) break;
        if (f * dir < 0.0) lo = x; else hi = x;
        double xn = x - f / d;
        if (!(xn > lo && xn < hi)) xn = 0.5 * (lo + hi);
        if (xn == x) break;
        x = xn;
    }
    return x;
}

// The reference's second candidate start, from the atan guess (bia/find_hyperbola.f90:71-89): its
// residual there and the start one Newton step on.
static __device__ __noinline__ double hyp_guess(const HypConsts c, double *error)
{
    const double theta_0 = atan2(c.sn_0, c.cs_0);
    const double theta = 2.0 / kPi * theta_0 * atan(c.time_end_ / c.tn_0);
    double d, sp, sm;
    hyp_eval<false>(c, theta, *error, d, sp, sm);
    return (*error == 0.0) ? theta : theta - *error / d;
}

// Divisions and roots are reciprocals and reciprocal roots shared between the quantities that need
// them.  The start's sine and cosine are formed from the state, cos theta = cos theta_0 + b sin theta_0/r
// and sin theta = +-(r.g/r) sin theta_0/g_0, and its angle from both by atan2, where the reference takes
// acos of the cosine (an ulp of it near pericentre is up to 1e-10 of displacement) and sines and
// cosines of the angle back; 2 sp sm = cos theta - cos theta_0 = b sin theta_0/r is known without
// cancellation.  The reference's second start guess is tried only where the Newton step from the start is
// not small against the distance to the asymptotes (below 1e-3 of it the step's error is 1e-6, and the
// guess, an angle from scratch, never the better one).
//
// The squares of distance, velocity and angular momentum have to be normal numbers (rsqrt_normal): below about
// 1e-154 of each a pair comes out non-finite and is counted so.  Nothing else leaves the type's range before they do.
//
// What bounds the ALG kernels: FP64 operations in dependent chains (atan2, log, and a sine, cosine and log an
// evaluation), 46 % of the FP64 pipe and 68 % of the issue slots at 22 of 32 lanes on mixed classes.  So the
// work per pair is what counts.  Step at n = 32768, Plummer / Coulomb: 71.0 / 83.0 ms with divisions, roots and
// angles throughout; 43.5 / 54.7 with shared reciprocals and the start's sines from the state (the
// ellipse's too); 39.1 / 57.0 from the Taylor start, but with the rounding floor still walked by a few
// lanes; 29.7 / 43.6 when a step of a few ulps ends the iteration (3.1 -> 1.0 evaluations a pair).  The
// interaction part's error against the exact step went from 8.8e-5 to 6.0e-5 of its norm on Plummer, from 4.0e-8
// to 3.5e-8 on Coulomb.
__device__ __forceinline__ int hyperbola(double eps_th, double dt, int ITR, const double YZ[4],
                                         double YN[4], double *error_end, int *bracket_exit,
                                         int *fallback)
{
    const double X_ini = YZ[0], Y_ini = YZ[1], U_ini = YZ[2], V_ini = YZ[3];
    const double r_g = X_ini * U_ini + Y_ini * V_ini;
    const double Lz = X_ini * V_ini - Y_ini * U_ini;
    const double aL = fabs(Lz);
    const double r2 = X_ini * X_ini + Y_ini * Y_ini;
    const double ir = rsqrt_normal(r2);
    const double g2 = U_ini * U_ini + V_ini * V_ini;
    const double W = g2 + 2.0 * eps_th * ir;
    const double ig_0 = rsqrt_normal(W);
    const double g_0 = W * ig_0;
    const double bg = eps_th * ig_0;           // b_0 g_0
    const double b_g = (bg * ig_0) * ig_0;     // b_0 / g_0, without the cube of a velocity
    const double b = aL * ig_0;
    HypConsts c;
    const double iden0 = rsqrt_normal(bg * bg + Lz * Lz);
    c.cs_0 = bg * iden0;
    c.sn_0 = aL * iden0;
    const double ieps = rcp_normal(eps_th);
    c.tn_0 = aL * (g_0 * ieps);
    half_angle(c.sn_0, c.cs_0, c.s0h, c.c0h);
    // the start: sine, cosine and angle
    const double bs = b * c.sn_0;
    const double D_i = bs * ir;  // cos theta - cos theta_0 = 2 sp sm
    const double sgn = Lz > 0.0 ? 1.0 : -1.0;
    double sn = sgn * (r_g * ir) * (c.sn_0 * ig_0), cs = c.cs_0 + D_i;
    const double theta_ini = atan2(sn, cs);
    const double inrm = rsqrt_normal(sn * sn + cs * cs);
    sn *= inrm;
    cs *= inrm;
    double sh, ch;
    half_angle(sn, cs, sh, ch);
    // sp sm = D_i / 2; the larger of the two is a sum without cancellation.  Away from the asymptotes the
    // smaller one is taken from the angle too, as the iteration takes it: there rounding alone counts, and
    // what start and end share cancels
    const double big = c.s0h * ch + c.c0h * fabs(sh);
    const double prod = D_i > 0.1 ? big * (c.s0h * ch - c.c0h * fabs(sh)) : 0.5 * D_i;
    const double q_i = prod * rcp_normal(big * big);  // the smaller over the larger: sm/sp, or sp/sm for theta < 0
    const double Dinv_i = 0.5 * rcp_normal(prod);
    // state and dimensionless time there (bia/find_hyperbola.f90:46-64)
    const double g0_cs0_sn0 = sgn * g_0 * c.cs_0 * rcp_normal(c.sn_0);
    const double cs_a = (cs * X_ini + sn * Y_ini) * ir;
    const double sn_a = (cs * Y_ini - sn * X_ini) * ir;
    const double lq = log(q_i);
    const double tau_ini = c.tn_0 * sn * Dinv_i + (sn >= 0.0 ? -lq : lq);
    const double time_ini = tau_ini * b_g;
    const double time_end = time_ini + sgn * dt;
    c.time_end_ = (time_end * g_0) * (W * ieps);  // time_end g_0 / b_0

    // the start of the iteration: one Newton step on (its residual is known already), or the guess
    const double error_ini_ = tau_ini - c.time_end_;
    const double d_ini = c.tn_0 * (1.0 - c.cs_0 * cs) * (Dinv_i * Dinv_i) + c.sn_0 * Dinv_i;
    const double step_ini = error_ini_ * rcp_normal(d_ini);
    double theta_end = (error_ini_ == 0.0) ? theta_ini : theta_ini - step_ini;
    double error_ = error_ini_;
    if (fabs(step_ini) <= 1e-3 * (big * q_i)) {  // big q_i: the sine of half the smaller distance
        // on from the Newton step by theta(t)'s Taylor series to third order (theta' = L/r^2,
        // r'' = L^2/r^3 + eps/r^2): the first evaluation then meets the rounding floor
        const double tr = ir * dt;
        const double rho = (r_g * ir) * tr;
        const double kap = ((Lz * Lz * ir + eps_th) * ir) * (tr * tr);
        theta_end = theta_ini - step_ini * (1.0 + (rho * rho - rho - kap * (1.0 / 3.0)));
    } else {
        double error_gss_;
        const double th_gss_end = hyp_guess(c, &error_gss_);
        if (!(fabs(error_gss_) > 10.0 * fabs(error_ini_))) {
            theta_end = th_gss_end;
            error_ = error_gss_;
        }
    }
    // minimum-residual Newton loop with cycle detection (bia/find_hyperbola.f90:93-120).
    // The reference compares each residual with every earlier one (error_restore_); here
    // the last four are kept in registers (h0 newest): an indexed history array lives in
    // local memory, whose write-back was most of the ALG kernel's DRAM traffic.  A cycle
    // only arises once the iteration sits at the rounding floor, where the iterates that
    // repeat are a few ulps apart; cycles of period 1-4 stop at the same iteration as in
    // the reference, a longer one runs on to the ITR cap with the same stock update rule.
    double err_stock = error_;
    double theta_stock = theta_end;
    double best_res = fabs(error_);
    const double kNoResidual = __longlong_as_double(0x7ff8000000000000LL);  // compares unequal
    double h0 = kNoResidual, h1 = kNoResidual, h2 = kNoResidual, h3 = kNoResidual;
    // A Newton step of at most four ulps of the angle ends it too: what follows would be the residuals'
    // rounding, on a few of the warp's lanes.
    int IR = 0;
    *bracket_exit = 0;
    while (IR < ITR) {
        const double theta_now = theta_end;
        double e, d, sp, sm;
        hyp_eval(c, theta_now, e, d, sp, sm);
        if (sp * sm < 0.0) {
            *bracket_exit = 1;
            break;
        }
        error_ = e;
        theta_end = (e == 0.0) ? theta_now : theta_now - e * rcp_normal(d);
        IR++;
        if (error_ == h0 || error_ == h1 || error_ == h2 || error_ == h3) break;
        h3 = h2;
        h2 = h1;
        h1 = h0;
        h0 = error_;
        best_res = fmin(best_res, fabs(error_));
        if (fabs(error_) < fabs(err_stock)) {
            err_stock = error_ * b_g;
            theta_stock = theta_end;
            if (fabs(err_stock) < 2e-16) break;
        }
        if (fabs(theta_end - theta_now) <= kFewUlps * fabs(theta_now)) break;
    }
    *error_end = error_ * b_g;
    *fallback = 0;
    if (!(best_res <= 1e-8 * (1.0 + fabs(c.time_end_)))) {  // the reference loop did not converge
        theta_stock = hyp_safe(c, theta_stock);
        *fallback = 1;
    }
    // end state (bia/find_hyperbola.f90:126-142): sine and cosine of the full angle, as the reference
    // takes them
    double sn_end, cs_end;
    sincos(theta_stock, &sn_end, &cs_end);
    const double r_end = bs * rcp_normal(cs_end - c.cs_0);
    // velocity (g_0/sin theta_0) (cos theta_0 sin theta, 1 - cos theta_0 cos theta): its change
    const double du_end = g0_cs0_sn0 * (sn_end - sn);
    const double dv_end = g0_cs0_sn0 * (cs - cs_end);
    YN[0] = r_end * (cs_end * cs_a - sn_end * sn_a);
    YN[1] = r_end * (cs_end * sn_a + sn_end * cs_a);
    YN[2] = YZ[2] + (du_end * cs_a - dv_end * sn_a);
    YN[3] = YZ[3] + (du_end * sn_a + dv_end * cs_a);
    return IR;
}

// ---------------------------------------------------------------------------
// bia/find_ellipse.f90:1-157 (with its contained Newton).  Returns ir.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double f_sign(double a, double b) { return (b >= 0.0) ? fabs(a) : -fabs(a); }

// Bracketed Newton-bisection for Kepler's equation xi - e sin(xi) = M (root in
// [M - |e|, M + |e|]), used only when the reference's iteration ends unconverged.
static __device__ __noinline__ double kepler_safe(double M, double e, double x)
{
    const double ae = fabs(e);
    double lo = M - ae, hi = M + ae;
    if (!(x >= lo && x <= hi)) x = M;
    for (int it = 0; it < 400; it++) {
        double sx, cx;
        sincos(x, &sx, &cx);
        const double f = x - e * sx - M;
        if (f == 0.0) break;
        if (f < 0.0) lo = x; else hi = x;
        double xn = x - f / (1.0 - e * cx);
        if (!(xn > lo && xn < hi)) xn = 0.5 * (lo + hi);
        if (xn == x) break;
        x = xn;
    }
    return x;
}

static __device__ __noinline__ int ellipse(double eps_th, double dt, int ITR, const double YZ[4], double YN[4],
                                double *error, int *fallback)
{
    const double X_ini = YZ[0], Y_ini = YZ[1], U_ini = YZ[2], V_ini = YZ[3];
    const double g2_ini = U_ini * U_ini + V_ini * V_ini;
    const double r2 = X_ini * X_ini + Y_ini * Y_ini;
    const double ir = rsqrt_normal(r2);
    const double r_ini = r2 * ir;
    const double W = g2_ini + 2.0 * eps_th * ir;
    const double L = X_ini * V_ini - Y_ini * U_ini;
    const double r_g_ini = X_ini * U_ini + Y_ini * V_ini;
    const double iga = f_sign(rsqrt_normal(-W), L);  // 1 / g_a
    const double g_a = -W * iga;
    const double a = -eps_th * (iga * iga);
    const double b = L * iga;
    const double ia = W * rcp_normal(eps_th);
    const double omega_a = g_a * ia;
    // the start's eccentric anomaly E, its sine and cosine and the eccentricity from the state itself:
    // a e (sin E, cos E) = (r.g / g_a, a - r).  (The reference's sqrt((a g_a)^2 - L^2) / (a g_a) is off by
    // 1e-8 on a circular orbit, and not of one piece with the angle.)
    double ecc = fabs(a - r_ini) * ia;
    double xi_ini, s_ini, c_ini;
    bool from_angle = false;
    if (r_g_ini == 0.0) {
        if (r_ini < a) {
            xi_ini = 0.0;
        } else if (r_ini == a) {
            xi_ini = atan2(Y_ini, X_ini);
            ecc = 0.0;
        } else {
            xi_ini = f_sign(kPi, L);
        }
        from_angle = true;
    } else {
        s_ini = r_g_ini * iga;
        c_ini = a - r_ini;
        xi_ini = atan2(s_ini, c_ini);
        const double n2 = s_ini * s_ini + c_ini * c_ini;
        const double in = rsqrt_normal(n2);
        s_ini *= in;
        c_ini *= in;
        ecc = n2 * in * ia;
        from_angle = !(n2 > 1e-290);
        if (from_angle) ecc = sqrt(n2) * ia;
    }
    if (from_angle) sincos(xi_ini, &s_ini, &c_ini);
    const double px = a * (c_ini - ecc), py = b * s_ini;  // the start in the orbit's frame
    const double tau_ini = xi_ini - ecc * s_ini;
    const double tau_end = fma(omega_a, dt, tau_ini);
    *error = 0.0;
    if (dt == 0.0) {
#pragma unroll
        for (int k = 0; k < 4; k++) YN[k] = YZ[k];
        return 0;
    }
    // Kepler's equation tau_end = xi - e sin(xi) by the reference's Newton loop
    // (bia/find_ellipse.f90:106-157).  Start: one Newton step from the initial anomaly
    // xi_ini, whose residual is omega dt, instead of the reference's start from the mean
    // anomaly (xi_2 + delta_ini, bia/find_ellipse.f90:116-129), which needs ~8 steps on
    // average and fails outright for e near 1; the root is the same.  A small step goes on by the
    // reversion of q x + (e s/2) x^2 + (e c/6) x^3 - ... = omega dt, q = 1 - e c, to fourth order, and the
    // first evaluation meets the rounding floor.  A Newton step of at most four ulps ends the loop, and
    // the end state turns the last iterate's sine and cosine by the last step.
    int ir_ = 0;
    const double error_ini = tau_end - xi_ini + ecc * s_ini;
    double xi_2 = xi_ini;
    double error_tm2 = error_ini;
    double s2 = s_ini, c2 = c_ini;
    const double iq = rcp_normal(1.0 - ecc * c_ini);
    double xi = error_ini * iq;
    if (fabs(xi) <= 1e-2) {
        const double A = 0.5 * ecc * s_ini * iq, B = (1.0 / 6.0) * ecc * c_ini * iq;
        const double A2 = A * A;
        xi *= 1.0 + xi * (xi * (2.0 * A2 - B + xi * A * (5.0 * (B - A2) + 1.0 / 12.0)) - A);
    }
    xi = xi_ini + xi;
    double xi_1 = __longlong_as_double(0x7ff8000000000000LL);  // unset: compares unequal
    double error_tm1 = error_tm2;
    double last = 1.0;  // the step from the iterate whose sine and cosine are s2, c2
    bool conv = false;
    while (xi_1 != xi_2 && ir_ <= ITR) {
        ir_++;
        xi_1 = xi;
        sincos(xi_1, &s2, &c2);
        error_tm1 = tau_end - xi_1 + ecc * s2;
        last = error_tm1 * rcp_normal(1.0 - ecc * c2);
        xi = xi_1 + last;
        if (error_tm1 == 0.0 || error_tm1 == error_tm2 || error_tm1 + error_tm2 == 0.0 ||
            fabs(last) <= kFewUlps * fabs(xi_1)) {
            *error = error_tm1;
            conv = true;
            break;
        }
        ir_++;
        xi_2 = xi;
        sincos(xi_2, &s2, &c2);
        error_tm2 = tau_end - xi_2 + ecc * s2;
        last = error_tm2 * rcp_normal(1.0 - ecc * c2);
        xi = xi_2 + last;
        if (error_tm2 == 0.0 || error_tm1 == error_tm2 || error_tm1 + error_tm2 == 0.0 ||
            fabs(last) <= kFewUlps * fabs(xi_2)) {
            *error = error_tm2;
            conv = true;
            break;
        }
    }
    if (xi_1 == xi_2) conv = true;
    *fallback = 0;
    if (!conv && !(fmin(fabs(error_tm1), fabs(error_tm2)) <= 1e-8 * (1.0 + fabs(tau_end)))) {
        xi = kepler_safe(tau_end, ecc, xi);
        *fallback = 1;
        last = 1.0;
    }
    double sn_end, cs_end;
    if (fabs(last) <= 1e-8) {  // xi = last iterate + last, to the second order (the next is 1e-24)
        const double h2 = 1.0 - 0.5 * last * last;
        sn_end = fma(s2, h2, c2 * last);
        cs_end = fma(c2, h2, -s2 * last);
    } else {
        sincos(xi, &sn_end, &cs_end);
    }
    const double xx_end = a * (cs_end - ecc);
    const double yy_end = b * sn_end;
    const double gr = g_a * rcp_normal(1.0 - ecc * cs_end);  // a g_a / r
    const double uu_end = -gr * sn_end;
    const double vv_end = b * ia * gr * cs_end;
    // the rotation from the orbit's frame: the start's position in both (the reference takes the
    // difference of the two angles by atan2, and its sine and cosine back); no fourth power of a distance
    const double in = rsqrt_normal(px * px + py * py) * ir;
    const double cs_alp = (px * X_ini + py * Y_ini) * in, sn_alp = (px * Y_ini - py * X_ini) * in;
    YN[0] = xx_end * cs_alp - yy_end * sn_alp;
    YN[1] = xx_end * sn_alp + yy_end * cs_alp;
    YN[2] = uu_end * cs_alp - vv_end * sn_alp;
    YN[3] = uu_end * sn_alp + vv_end * cs_alp;
    return ir_;
}

// ---------------------------------------------------------------------------
// bia/find_parabola.f90:1-143 (diagnostic prints dropped).  Returns iterations.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double par_time(double r_min, double g_max, double theta)
{
    double sn, cs;
    sincos(theta, &sn, &cs);
    return (2.0 + cs) * sn / ((1.0 + cs) * (1.0 + cs)) * 4.0 * r_min / (3.0 * g_max);
}

static __device__ __noinline__ int parabola(double eps_th, double DT, const double YZ[4], double YN[4],
                                     double *error_time)
{
    constexpr int NI = 99;
    double theta_Newton[NI + 1], error_Newton[NI + 1];
    const double r_ini = sqrt(YZ[0] * YZ[0] + YZ[1] * YZ[1]);
    const double r_dot_g = YZ[0] * YZ[2] + YZ[1] * YZ[3];
    const double r_crs_g = YZ[0] * YZ[3] - YZ[1] * YZ[2];
    const double g_max = -2.0 * eps_th / r_crs_g;
    const double r_min = r_crs_g / g_max;
    const double x_ini = 2.0 * r_min - r_ini;
    const double y_ini = f_sign(2.0 * r_min * sqrt(r_ini / r_min - 1.0), r_dot_g);
    const double theta_ini = atan2(y_ini, x_ini);
    const double time_ini = par_time(r_min, g_max, theta_ini);
    const double time_end = time_ini + DT;
    const double t_ = 3.0 * g_max / (4.0 * r_min) * time_end;
    const double sq = sqrt(1.0 + t_ * t_);
    const double theta_gss = 2.0 * atan(pow(sq + t_, 1.0 / 3) - pow(sq - t_, 1.0 / 3));
    double theta = theta_gss, err_tm_min = 1e99, thetamin = theta;
    int i_min = 1, i;
    for (i = 1; i <= NI; i++) {
        const double err_tm = par_time(r_min, g_max, theta) - time_end;
        error_Newton[i] = err_tm;
        const double ch = cos(theta * 0.5);
        const double ch2 = ch * ch;
        const double dtheta = -err_tm / (r_min / (g_max * (ch2 * ch2)));
        if (fabs(err_tm) < err_tm_min) {
            err_tm_min = fabs(err_tm);
            thetamin = theta;
            i_min = i;
        }
        theta = theta + dtheta;
        theta_Newton[i] = theta;
        if (dtheta == 0.0) break;
        if (theta - dtheta == theta) break;
        bool cyc = false;
        for (int j = 1; j <= i - 1; j++)
            if (error_Newton[i] == error_Newton[j]) { cyc = true; break; }
        if (cyc) { theta = theta_Newton[i_min]; break; }
    }
    if (i == NI + 1) theta = thetamin;
    const double theta_end = theta;
    double sn_b, cs_b;
    sincos(theta_end * 0.5, &sn_b, &cs_b);
    const double r_end = r_min / (cs_b * cs_b);
    const double g_end = g_max * cs_b;
    double st, ct;
    sincos(theta_end, &st, &ct);
    const double x_end = r_end * ct, y_end = r_end * st;
    const double u_end = -g_end * sn_b, v_end = g_end * cs_b;
    const double s1 = x_ini * YZ[1] - y_ini * YZ[0];
    const double c1 = x_ini * YZ[0] + y_ini * YZ[1];
    const double tmp = 1.0 / sqrt(s1 * s1 + c1 * c1);
    const double sn_g = s1 * tmp, cs_g = c1 * tmp;
    YN[0] = x_end * cs_g - y_end * sn_g;
    YN[1] = x_end * sn_g + y_end * cs_g;
    YN[2] = u_end * cs_g - v_end * sn_g;
    YN[3] = u_end * sn_g + v_end * cs_g;
    *error_time = time_end - par_time(r_min, g_max, theta_end);
    return (i > NI) ? NI : i;
}

// ---------------------------------------------------------------------------
// bia/find_dXYUV_RKF.f90:1-170: per-pair RKF4(5) with step doubling on the planar
// relative equation r'' = eps r/|r|^3 (moon_2D).  Returns ier; YN = step-doubled
// solution, *error = max of (yln - yhn)/31.
// ---------------------------------------------------------------------------
struct Fehlberg {
    static constexpr double AL2 = 1.0 / 4, AL3 = 3.0 / 8, AL4 = 12.0 / 13, AL5 = 1.0, AL6 = 1.0 / 2;
    static constexpr double B21 = 1.0 / 4;
    static constexpr double B31 = 3.0 / 32, B32 = 9.0 / 32;
    static constexpr double B41 = 1932.0 / 2197, B42 = -7200.0 / 2197, B43 = 7296.0 / 2197;
    static constexpr double B51 = 439.0 / 216, B52 = -8.0, B53 = 3680.0 / 513, B54 = -845.0 / 4104;
    static constexpr double B61 = -8.0 / 27, B62 = 2.0, B63 = -3544.0 / 2565, B64 = 1859.0 / 4104,
                            B65 = -11.0 / 40;
    static constexpr double GA1 = 16.0 / 135, GA3 = 6656.0 / 12825, GA4 = 28561.0 / 56430,
                            GA5 = -9.0 / 50, GA6 = 2.0 / 55;
    static constexpr double DA1 = 1.0 / 360, DA3 = -128.0 / 4275, DA4 = -2197.0 / 75240,
                            DA5 = 1.0 / 50, DA6 = 2.0 / 55;
};

// Acceleration (ax, ay) = eps (x, y) / r^3 of moon_2D.  kNormal: eps r^-3 from one reciprocal square
// root (x^2 + y^2 a normal number), at about half the FP64 instructions of the reference's
// eps / (rsq sqrt(rsq)) (bia/find_dXYUV_RKF.f90:15-23), which the other form keeps.
template <bool kNormal>
__device__ __forceinline__ void moon_acc(double eps_th, double x, double y, double &ax, double &ay)
{
    const double rsq = x * x + y * y;
    double aaa;
    if (kNormal) {
        aaa = scaled_rsqrt3_normal(eps_th, rsq);
    } else {
        aaa = eps_th / (rsq * sqrt(rsq));
    }
    ax = x * aaa;
    ay = y * aaa;
}

// bia/find_dXYUV_RKF.f90:150-157 fehl on the planar state (x, y, u, v) from y0 with its acceleration
// a1 = (ax, ay); er written when kWantEr.  A position's derivative is the stage's velocity
// u0 + h sum_m B_sm a_m, so the position of stage s is x0 + c_s h u0 + h^2 sum_m N_sm a_m with
// N = B B (and GA B, DA B for the new position and its error): the accelerations are all that is
// kept, no stage velocity is formed, and a step takes 62 operations for its sums instead of 100.  (h^2 has to be a
// normal number: below |h| of 1e-154 the accelerations do not reach the positions.)
struct FehlbergNested {
    using F = Fehlberg;
    static constexpr double N31 = F::B32 * F::B21;
    static constexpr double N41 = F::B42 * F::B21 + F::B43 * F::B31, N42 = F::B43 * F::B32;
    static constexpr double N51 = F::B52 * F::B21 + F::B53 * F::B31 + F::B54 * F::B41,
                            N52 = F::B53 * F::B32 + F::B54 * F::B42, N53 = F::B54 * F::B43;
    static constexpr double N61 = F::B62 * F::B21 + F::B63 * F::B31 + F::B64 * F::B41 + F::B65 * F::B51,
                            N62 = F::B63 * F::B32 + F::B64 * F::B42 + F::B65 * F::B52,
                            N63 = F::B64 * F::B43 + F::B65 * F::B53, N64 = F::B65 * F::B54;
    static constexpr double G1 = F::GA3 * F::B31 + F::GA4 * F::B41 + F::GA5 * F::B51 + F::GA6 * F::B61,
                            G2 = F::GA3 * F::B32 + F::GA4 * F::B42 + F::GA5 * F::B52 + F::GA6 * F::B62,
                            G3 = F::GA4 * F::B43 + F::GA5 * F::B53 + F::GA6 * F::B63,
                            G4 = F::GA5 * F::B54 + F::GA6 * F::B64, G5 = F::GA6 * F::B65;
    static constexpr double D1 = F::DA3 * F::B31 + F::DA4 * F::B41 + F::DA5 * F::B51 + F::DA6 * F::B61,
                            D2 = F::DA3 * F::B32 + F::DA4 * F::B42 + F::DA5 * F::B52 + F::DA6 * F::B62,
                            D3 = F::DA4 * F::B43 + F::DA5 * F::B53 + F::DA6 * F::B63,
                            D4 = F::DA5 * F::B54 + F::DA6 * F::B64, D5 = F::DA6 * F::B65;
};

template <bool kNormal, bool kWantEr>
__device__ __forceinline__ void fehl4(double eps_th, double h, const double y0[4], const double a1[2], double yn[4],
                                      double er[4])
{
    using F = Fehlberg;
    using N = FehlbergNested;
    const double h2 = h * h;
    const double hu[2] = {h * y0[2], h * y0[3]};
    double a2[2], a3[2], a4[2], a5[2], a6[2], p[2];
#pragma unroll
    for (int i = 0; i < 2; i++) p[i] = fma(F::AL2, hu[i], y0[i]);
    moon_acc<kNormal>(eps_th, p[0], p[1], a2[0], a2[1]);
#pragma unroll
    for (int i = 0; i < 2; i++) p[i] = fma(h2, N::N31 * a1[i], fma(F::AL3, hu[i], y0[i]));
    moon_acc<kNormal>(eps_th, p[0], p[1], a3[0], a3[1]);
#pragma unroll
    for (int i = 0; i < 2; i++) p[i] = fma(h2, N::N41 * a1[i] + N::N42 * a2[i], fma(F::AL4, hu[i], y0[i]));
    moon_acc<kNormal>(eps_th, p[0], p[1], a4[0], a4[1]);
#pragma unroll
    for (int i = 0; i < 2; i++)
        p[i] = fma(h2, N::N51 * a1[i] + N::N52 * a2[i] + N::N53 * a3[i], y0[i] + hu[i]);
    moon_acc<kNormal>(eps_th, p[0], p[1], a5[0], a5[1]);
#pragma unroll
    for (int i = 0; i < 2; i++)
        p[i] = fma(h2, N::N61 * a1[i] + N::N62 * a2[i] + N::N63 * a3[i] + N::N64 * a4[i],
                   fma(F::AL6, hu[i], y0[i]));
    moon_acc<kNormal>(eps_th, p[0], p[1], a6[0], a6[1]);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        yn[i] = y0[i] + fma(h2, N::G1 * a1[i] + N::G2 * a2[i] + N::G3 * a3[i] + N::G4 * a4[i] + N::G5 * a5[i], hu[i]);
        yn[2 + i] = fma(h, F::GA1 * a1[i] + F::GA3 * a3[i] + F::GA4 * a4[i] + F::GA5 * a5[i] + F::GA6 * a6[i],
                        y0[2 + i]);
    }
    if (kWantEr) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            er[i] = h2 * (N::D1 * a1[i] + N::D2 * a2[i] + N::D3 * a3[i] + N::D4 * a4[i] + N::D5 * a5[i]);
            er[2 + i] = h * (F::DA1 * a1[i] + F::DA3 * a3[i] + F::DA4 * a4[i] + F::DA5 * a5[i] + F::DA6 * a6[i]);
        }
    }
}

// x^(1/5) of the step control: an FP32 power and two Newton steps on y^-5 = 1/x in FP64 (quadratic: 1e-6,
// 3e-12, 3e-23 before rounding), where x is well inside FP32's range; else pow.
__device__ __forceinline__ double fifth_root(double x)
{
    if (!(x > 1e-30 && x < 1e30)) return pow(x, 0.2);
    double y = (double)powf((float)x, -0.2f);  // x^(-1/5): y (6 - x y^5) / 5
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double y2 = y * y;
        y = y * fma(-0.2 * x, y2 * y2 * y, 1.2);
    }
    const double y2 = y * y;
    return x * (y2 * y2);  // x x^(-4/5)
}

// The step with its control, two copies of the Fehlberg step in all (the low step, tried and, to the
// end, repeated; the half step): four inlined copies fetched more instructions than the SM's caches
// hold.  What bounds it: the FP64 pipe (67 % busy, 2225 instructions a pair of four steps) and the
// latency of a stage's dependent chain at 16 warps per SM; 24 warps spill and are no faster (5.98 against 5.79
// ms).  Coulomb step at n = 8191: 12.8 ms with divisions and roots, 6.9 with reciprocal square
// roots, fifth roots and one division for the error norm, 6.0 without stage velocities, 5.8 with
// two copies.  kNormal: r^2 stays a normal number over the step (rkf_pair decides by the pair's
// initial state).
template <bool kNormal>
static __device__ __noinline__ int rkf_pair_form(double eps_th, double xe, double relerr, double abserr,
                                                 const double YZ[4], double YN[4], double *error, int *nacc)
{
    const int itemax = 100000;
    const double epsmin = 1e-15;
    double yh0[4], yl0[4], yln[4], yhn[4], er[4];
#pragma unroll
    for (int i = 0; i < 4; i++) { yh0[i] = YZ[i]; yl0[i] = YZ[i]; yhn[i] = YZ[i]; }
    double al[2];  // the acceleration of yl0
    moon_acc<kNormal>(eps_th, yl0[0], yl0[1], al[0], al[1]);
    const double f0[4] = {yl0[2], yl0[3], al[0], al[1]};
    double toldy = 1.7976931348623157e308;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (f0[i] != 0.0) {
            const double tol = relerr * fabs(yl0[i]) + abserr;
            toldy = fmin(toldy, fabs(tol / f0[i]));
        }
    }
    double h = (toldy == 1.7976931348623157e308) ? epsmin * xe : fmin(xe / 100.0, fifth_root(toldy));
    double x = 0.0;
    int ier = 10000, n = 0;
    *error = 0.0;
    bool last = false;  // the step to the end, its size set, is under way
    for (int iter = 0;;) {
        if (!last && ++iter > itemax) break;
        fehl4<kNormal, true>(eps_th, h, yl0, al, yln, er);
        double erret = 0.0;
        if (!last) {
            bool bad = false;
            if (relerr == 0.0) {  // one tolerance: the largest |er| over it, one division for four
                const double m = fmax(fmax(fabs(er[0]), fabs(er[1])), fmax(fabs(er[2]), fabs(er[3])));
                bad = abserr == 0.0;
                erret = fmax(0.0, m / abserr);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const double et = relerr / 2.0 * (fabs(yl0[i]) + fabs(yln[i])) + abserr;
                    if (et == 0.0) bad = true;
                    erret = fmax(erret, fabs(er[i]) / et);
                }
            }
            if (bad) { ier = 20000; break; }
            if (erret > 1.0) {
                h = (erret >= 59049.0) ? 0.1 * h : 0.9 * h / fifth_root(erret);
                if (h <= epsmin) { ier = 30000; break; }
                continue;
            }
            if (!(x + h < xe)) {  // the same low step once more, to xe exactly
                last = true;
                h = xe - x;
                continue;
            }
        }
        double ymid[4];
#pragma unroll
        for (int i = 0; i < 4; i++) ymid[i] = yh0[i];
#pragma unroll 1
        for (int half = 0; half < 2; half++) {
            double am[2];
            moon_acc<kNormal>(eps_th, ymid[0], ymid[1], am[0], am[1]);
            fehl4<kNormal, false>(eps_th, h * 0.5, ymid, am, yhn, er);
#pragma unroll
            for (int i = 0; i < 4; i++) ymid[i] = yhn[i];
        }
        n++;
        if (last) {
            double m = (yln[0] - yhn[0]) / 31.0;
#pragma unroll
            for (int i = 1; i < 4; i++) m = fmax(m, (yln[i] - yhn[i]) / 31.0);
            *error = m;
            ier = 0;
            break;
        }
        x = x + h;
#pragma unroll
        for (int i = 0; i < 4; i++) { yl0[i] = yln[i]; yh0[i] = yhn[i]; }
        moon_acc<kNormal>(eps_th, yl0[0], yl0[1], al[0], al[1]);
        h = (erret <= 1.889568e-4) ? 5.0 * h : 0.9 * h / fifth_root(erret);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) YN[i] = yhn[i];
    *nacc = n;
    return ier;
}

// The reciprocal-square-root form where the initial separation and its change over the step are far from the
// ends of the type's range (nothing physical is not), else the reference's divisions.
__device__ __forceinline__ int rkf_pair(double eps_th, double xe, double relerr, double abserr, const double YZ[4],
                                        double YN[4], double *error, int *nacc)
{
    const double r2 = YZ[0] * YZ[0] + YZ[1] * YZ[1];
    const double d2 = (YZ[2] * YZ[2] + YZ[3] * YZ[3]) * (xe * xe);
    if (r2 > 1e-200 && r2 < 1e200 && d2 < 1e200)
        return rkf_pair_form<true>(eps_th, xe, relerr, abserr, YZ, YN, error, nacc);
    return rkf_pair_form<false>(eps_th, xe, relerr, abserr, YZ, YN, error, nacc);
}

// ---------------------------------------------------------------------------
// Universal-variable propagation of r'' = eps r/|r|^3 (mu = -eps) with Stumpff
// functions (Danby, Fundamentals of Celestial Mechanics, 2nd ed., 6.7-6.9).  Uniformly
// well conditioned for every conic and for radial or zero-velocity pairs; the
// displacement from free motion is formed without cancellation:
//   r(t) - r0 - v0 dt = -(mu/r0) s^2 c2 r0vec - mu s^3 c3 v0vec
//   v(t) - v0         = -(mu/(r r0)) s c1 r0vec - (mu/r) s^2 c2 v0vec
// with s the root of r0 s c1 + sigma0 s^2 c2 + mu s^3 c3 = dt (bracketed Newton).
// No transcendental function is called: the Stumpff functions come from a series at
// |x| <= 0.1 and the duplication formulas c0(4x) = 2c0^2 - 1, c1(4x) = c0 c1,
// c2(4x) = c1^2/2, c3(4x) = (c2 + c0 c3)/4.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void stumpff(double x, double c[4])
{
    if (fabs(x) <= 1e-6) {
        // three terms: the next ones, x^3/8! and x^3/9!, are below 3e-23
        const double c2 = 0.5 - x * (1.0 / 24 - x * (1.0 / 720));
        const double c3 = 1.0 / 6 - x * (1.0 / 120 - x * (1.0 / 5040));
        c[0] = 1.0 - x * c2;
        c[1] = 1.0 - x * c3;
        c[2] = c2;
        c[3] = c3;
        return;
    }
    if (fabs(x) <= 1e-2) {
        // the first five terms: the next ones, x^5/12! and x^5/13!, are below 2e-19
        const double c2 = 0.5 - x * (1.0 / 24 - x * (1.0 / 720 - x * (1.0 / 40320 - x * (1.0 / 3628800))));
        const double c3 = 1.0 / 6 - x * (1.0 / 120 - x * (1.0 / 5040 - x * (1.0 / 362880 - x * (1.0 / 39916800))));
        c[0] = 1.0 - x * c2;
        c[1] = 1.0 - x * c3;
        c[2] = c2;
        c[3] = c3;
        return;
    }
    int n = 0;
    while (fabs(x) > 0.1 && n < 200) { x *= 0.25; n++; }
    // c2 = sum (-x)^j / (2+2j)!, c3 = sum (-x)^j / (3+2j)!, j = 0..10 (|x| <= 0.1)
    double c2 = 1.0 / 620448401733239439360000.0;    // 1/24!
    double c3 = 1.0 / 15511210043330985984000000.0;  // 1/25!
    c2 = 1.0 / 20922789888000.0 - x * (1.0 / 6402373705728000.0 - x * (1.0 / 2432902008176640000.0 - x * (1.0 / 1124000727777607680000.0 - x * c2)));
    c3 = 1.0 / 355687428096000.0 - x * (1.0 / 121645100408832000.0 - x * (1.0 / 51090942171709440000.0 - x * (1.0 / 25852016738884976640000.0 - x * c3)));
    c2 = 0.5 - x * (1.0 / 24 - x * (1.0 / 720 - x * (1.0 / 40320 - x * (1.0 / 3628800 - x * (1.0 / 479001600 - x * (1.0 / 87178291200.0 - x * c2))))));
    c3 = 1.0 / 6 - x * (1.0 / 120 - x * (1.0 / 5040 - x * (1.0 / 362880 - x * (1.0 / 39916800 - x * (1.0 / 6227020800.0 - x * (1.0 / 1307674368000.0 - x * c3))))));
    double c1 = 1.0 - x * c3;
    double c0 = 1.0 - x * c2;
    for (; n > 0; n--) {
        const double c3n = (c2 + c0 * c3) * 0.25;
        const double c2n = c1 * c1 * 0.5;
        const double c1n = c0 * c1;
        const double c0n = 2.0 * c0 * c0 - 1.0;
        c0 = c0n; c1 = c1n; c2 = c2n; c3 = c3n;
    }
    c[0] = c0; c[1] = c1; c[2] = c2; c[3] = c3;
}

// iteration cap of the universal-variable solver; a pair that reaches it is counted as
// not converged
constexpr int kUvItMax = 200;

// The universal-variable pair in pieces (prepare, start, iterate, compose) so that other
// solvers can supply their own start; uv_halfdisp chains them.
struct UvPair {
    double mu, r0, sig, beta;
    double ir0;  // 1 / r0, so that start and composition need one division fewer each
};

__device__ __forceinline__ UvPair uv_prepare(double eps_th, const double r[3], const double g[3])
{
    UvPair p;
    p.mu = -eps_th;
    // one reciprocal square root for both r0 and 1/r0 (rsqrt: within 1 ulp)
    const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    p.ir0 = rsqrt(r2);
    p.r0 = (r2 > 0.0) ? r2 * p.ir0 : 0.0;
    p.sig = r[0] * g[0] + r[1] * g[1] + r[2] * g[2];
    const double v2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
    p.beta = 2.0 * p.mu * p.ir0 - v2;
    return p;
}

// Third-order start: the reversion of t = r0 s + (sig/2) s^2 + ((mu - beta r0)/6) s^3 + O(s^4),
//   s = x - (sig / (2 r0)) x^2 + (sig^2/2 - r0 (mu - beta r0)/6) x^3 / r0^2,  x = dt / r0,
// leaves a relative error O((dt/T)^3), so at small steps the first Newton correction is
// already below the 1e-10 acceptance of uv_iterate (the second-order start needed two).
__device__ __forceinline__ double uv_start(const UvPair &p, double dt)
{
    const double x = dt * p.ir0;
    const double a2 = -0.5 * p.sig * p.ir0;
    const double a3 = (0.5 * p.sig * p.sig - p.r0 * (p.mu - p.beta * p.r0) * (1.0 / 6.0)) * (p.ir0 * p.ir0);
    const double s = x + x * x * (a2 + x * a3);
    return (s > 0.0) ? s : x;
}

// Fifth-order start of the universal-variable method and the split learned step's plain
// pairs, in dimensionless form.  The universal Kepler equation
//   t = b1 s + b2 s^2 + b3 s^3 + b4 s^4 + b5 s^5 + O(s^6),
//   b1 = r0, b2 = sig/2, b3 = (mu - beta r0)/6, b4 = -sig beta/24, b5 = beta (beta r0 - mu)/120
// (the Stumpff series of r0 s c1 + sig s^2 c2 + mu s^3 c3) is inverted with the Lagrange
// reversion coefficients (Abramowitz and Stegun 3.6.25):
//   a1 = 1/b1, a2 = -b2/b1^3, a3 = (2 b2^2 - b1 b3)/b1^5, a4 = (5 b1 b2 b3 - b1^2 b4 - 5 b2^3)/b1^7,
//   a5 = (6 b1^2 b2 b4 + 3 b1^2 b3^2 + 14 b2^4 - b1^3 b5 - 21 b1 b2^2 b3)/b1^9,
//   s = a1 t + a2 t^2 + a3 t^3 + a4 t^4 + a5 t^5 + O(t^6).
// With x = dt/r0, y = sig dt/(2 r0^2), m = mu/r0, z = (m - beta) x^2/6 and w = beta x^2 the
// relative terms c_k = a_(k+1) dt^k / a1 are
//   c1 = -y, c2 = 2y^2 - z, c3 = y (5z + w/12 - 5y^2),
//   c4 = y^2 (14y^2 - 21z - w/2) + z (3z + w/20),
// and s = x S with S = 1 + c1 + c2 + c3 + c4 (about 25 FP64 operations instead of 65 for the
// same sum from the a_k).  When every |c_k| <= Q^k with Q = 3e-4 (the step is that small
// against the pair's time scales) the sum is exact: its truncation is below 1.1e-17
// relative, a tenth of an FP64 ulp (checked in extended precision against the solved equation
// on 12000 attractive and repulsive pairs drawn around that boundary), so no Newton
// correction runs and uv_compose_series composes the half-displacement from S.  Otherwise
// uv_series_start gives the start of uv_iterate.  The ALG kernels keep uv_start:
// changing the code they inline changes how the compiler contracts their own FP64
// expressions.  Every product and sum is written out (fma, __dmul_rn) so that each kernel
// that inlines this computes the same bits and takes the same branch: the ensemble's systems
// equal their own steps bit for bit.
struct UvSeries {
    double x, y, x2, w, c2;
    double mh;  // -m/2
    double S;   // s = x S where exact
    double tail;  // c3 + c4
    bool exact;
};

__device__ __forceinline__ UvSeries uv_series(const UvPair &p, double dt)
{
    UvSeries q;
    q.x = __dmul_rn(dt, p.ir0);
    const double m = __dmul_rn(p.mu, p.ir0);
    q.mh = -0.5 * m;
    q.y = __dmul_rn(__dmul_rn(0.5 * p.sig, p.ir0), q.x);
    q.x2 = __dmul_rn(q.x, q.x);
    q.w = __dmul_rn(p.beta, q.x2);
    const double y = q.y, w = q.w;
    const double z = __dmul_rn(__dsub_rn(m, p.beta), __dmul_rn(q.x2, 1.0 / 6.0));
    const double y2 = __dmul_rn(y, y);
    q.c2 = fma(2.0 * y, y, -z);
    const double c3 = __dmul_rn(y, fma(-5.0, y2, fma(w, 1.0 / 12.0, 5.0 * z)));
    const double c4 = fma(z, fma(3.0, z, __dmul_rn(w, 0.05)), __dmul_rn(y2, fma(14.0, y2, fma(-21.0, z, -0.5 * w))));
    constexpr double Q = 3e-4;
    const bool small = fabs(y) <= Q && fabs(q.c2) <= Q * Q && fabs(c3) <= Q * Q * Q && fabs(c4) <= Q * Q * Q * Q;
    q.tail = c3 + c4;
    q.S = 1.0 + (q.c2 - y + q.tail);
    q.exact = small && q.S > 0.0 && dt > 0.0;  // s = x S > 0
    return q;
}

// The start for a pair whose series is not exact (uv_iterate corrects it): the fifth-order sum where its last
// terms are small (at steps a few times the exactness bound its error is ~1e-13 and the first Newton
// correction is below uv_iterate's acceptance; with the third-order sum it took two: 16384-body Coulomb cube at
// dt = 1e-3, universal-variable step 3.37 -> 2.95 ms), else the third-order one.
__device__ __forceinline__ double uv_series_start(const UvSeries &q)
{
    const double s = __dmul_rn(q.x, fabs(q.tail) <= 0.02 ? q.S : 1.0 + (q.c2 - q.y));
    return (s > 0.0) ? s : q.x;
}

// Half-displacement of an exact series pair: the coefficients of uv_compose in the series'
// variables.  With K = -m x^2/2 (= -mu dt^2/(2 r0^3)), A = S^2 c2(w S^2), B = S^3 c3(w S^2)
// and rho = r0/r(s):
//   (f - 1)/2 = K A,  (g - dt)/2 = K dt B,  (g' - 1)/2 = K A rho,  f'/2 = -(m/2)(x/r0) S c1 rho,
// and r(s)/r0 = 1 + d with d = -w S^2 c2 + 2 y S c1 - 2 K A (r(s) = r0 c0 + sig s c1 +
// mu s^2 c2 and c0 = 1 - beta s^2 c2), formed without cancellation.  rho is the alternating
// series of 1/(1 + d) to d^5 where |d| <= 1e-3 (truncation below 1e-18), else a division.
// f'/2 is formed as (K/dt) S c1 rho (K/dt = -(m/2) x/r0; 1/dt is the same for every pair).
// The factor 1/2 of the half-displacement is inside K (a power of two: the same bits).
__device__ __forceinline__ void uv_compose_series(const UvPair &p, const UvSeries &q, double dt, const double r[3],
                                                  const double g[3], double h[6])
{
    const double S = q.S;
    const double S2 = __dmul_rn(S, S);
    const double arg = __dmul_rn(q.w, S2);
    double c[4];
    stumpff(arg, c);
    const double A = __dmul_rn(S2, c[2]);
    const double B = __dmul_rn(__dmul_rn(S2, S), c[3]);
    const double K = __dmul_rn(q.mh, q.x2);
    const double fm1 = __dmul_rn(K, A);
    const double gmdt = __dmul_rn(__dmul_rn(K, dt), B);
    const double d = fma(-arg, c[2], fma(__dmul_rn(2.0 * q.y, S), c[1], -2.0 * fm1));
    double rho;
    if (fabs(d) <= 1e-3) {
        const double nd = -d;
        rho = fma(nd, fma(nd, fma(nd, fma(nd, fma(nd, 1.0, 1.0), 1.0), 1.0), 1.0), 1.0);
    } else {
        rho = 1.0 / (1.0 + d);
    }
    const double gdm1 = __dmul_rn(fm1, rho);
    const double fdot = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(K, 1.0 / dt), S), c[1]), rho);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        h[k] = fma(fm1, r[k], __dmul_rn(gmdt, g[k]));
        h[3 + k] = fma(fdot, r[k], __dmul_rn(gdm1, g[k]));
    }
}

// Safeguarded Newton on F(s) = t(s) - dt, F' = r(s) > 0, with the bracket [lo, hi]
// (F(0) = -dt < 0; hi < 0 until an upper bound is seen).  A Newton step that leaves the
// bracket, or is not below half the step before last, is replaced by bisection, so the
// bracket at least halves every two iterations: on hyperbolic branches Newton from far
// above the root moves only ~1/sqrt(-beta) per step.  So is a step where 1/F' is not a normal
// number (rcp_normal: 0, which would look converged).  Returns the iterations
// (kUvItMax + 1 when the cap was reached).
// ifp (optional): 1 / F' at the last evaluation, for uv_compose (F' = r(s)).
__device__ __forceinline__ int uv_iterate(const UvPair &p, double dt, double &s_io, double *ifp = nullptr)
{
    double c[4];
    double s = s_io;
    double lo = 0.0, hi = -1.0, dx = 1e300, dxold = 1e300;
    double ifp_last = 0.0;
    int it;
    for (it = 1; it <= kUvItMax; it++) {
        stumpff(p.beta * s * s, c);
        const double F = p.r0 * s * c[1] + p.sig * s * s * c[2] + p.mu * s * s * s * c[3] - dt;
        const double Fp = p.r0 * c[0] + p.sig * s * c[1] + p.mu * s * s * c[2];
        if (F == 0.0) break;
        ifp_last = rcp_normal(Fp);
        const double step = F * ifp_last;
        const bool slope = Fp > 0x1p-1021 && Fp < 0x1p1021;
        if (slope && fabs(step) <= 4.0 * 2.220446049250313e-16 * fabs(s)) {
            s = s - step;  // converged: the remaining correction is a few ulps
            break;
        }
        if (F < 0.0) lo = s; else hi = s;  // a NaN F (overflow far above the root) lowers hi
        double sn = s - step;
        const bool newton = slope && (sn > lo) && (hi < 0.0 || sn < hi) &&
                            (hi < 0.0 || fabs(step) <= 0.5 * dxold);
        if (!newton) sn = (hi > 0.0) ? 0.5 * (lo + hi) : 2.0 * s;
        dxold = dx;
        dx = fabs(sn - s);
        s = sn;
        if (dx <= 4.0 * 2.220446049250313e-16 * fabs(s)) break;  // bracket collapsed
        // Newton converges quadratically: after a step of relative size 1e-10 the next
        // one would be below rounding, so s is final without another evaluation
        if (newton && dx <= 1e-10 * fabs(s)) break;
    }
    s_io = s;
    if (ifp) *ifp = ifp_last;
    return it;
}

// One Halley step on the same equation from s: returns the step ds (s_new = s - ds).
// F'' = dr/ds = sig c0 + (mu - beta r0) s c1.  NaN where the reciprocal is not a normal number (rcp_normal: 0,
// which would look converged): learned_finish leaves the pair to uv_iterate.
__device__ __forceinline__ double uv_halley_step(const UvPair &p, double dt, double s)
{
    double c[4];
    stumpff(p.beta * s * s, c);
    const double F = p.r0 * s * c[1] + p.sig * s * s * c[2] + p.mu * s * s * s * c[3] - dt;
    const double Fp = p.r0 * c[0] + p.sig * s * c[1] + p.mu * s * s * c[2];
    const double Fpp = p.sig * c[0] + (p.mu - p.beta * p.r0) * s * c[1];
    const double den = Fp * Fp - 0.5 * F * Fpp;
    return den < 0x1p1021 ? F * (Fp * rcp_normal(den)) : __longlong_as_double(0x7ff8000000000000LL);
}

// Half-displacement from the solved s: f - 1, g - dt, f', g' - 1 from the Stumpff
// functions (no cancellation at small s).  irr_hint (optional, 0: none): an approximation
// of 1/r(s), such as uv_iterate's last 1/F'; within 1e-8 of it one Newton-Raphson step for
// the reciprocal (x + x (1 - r x)) gives 1/r(s) to ~1e-16, else 1/r(s) is divided out.
// kTwoSteps (the universal-variable method and the split step's plain pairs after Newton
// iterations, the learned finish): two Newton-Raphson steps from a hint within 1e-4
// (error e^4 <= 1e-16); the ALG kernels keep the one-step form.
template <bool kTwoSteps = false>
__device__ __forceinline__ void uv_compose(const UvPair &p, double s, const double r[3], const double g[3],
                                           double h[6], double irr_hint = 0.0)
{
    double c[4];
    stumpff(p.beta * s * s, c);
    const double s2c2 = s * s * c[2], s3c3 = s * s * s * c[3];
    const double rr = p.r0 * c[0] + p.sig * s * c[1] + p.mu * s2c2;
    const double e = fma(-rr, irr_hint, 1.0);
    double irr;
    if (kTwoSteps) {
        if (irr_hint != 0.0 && fabs(e) <= 1e-4) {
            const double x1 = fma(irr_hint, e, irr_hint);
            irr = fma(x1, fma(-rr, x1, 1.0), x1);
        } else {
            irr = rcp_normal(rr);
        }
    } else {
        irr = (irr_hint != 0.0 && fabs(e) <= 1e-8) ? fma(irr_hint, e, irr_hint) : rcp_normal(rr);
    }
    // the half-displacement's factor 1/2 is taken into the coefficients: scaling by a power of
    // two is exact, so h is the same as (f - 1) r + (g - dt) v halved afterwards, at four
    // multiplications instead of six
    const double fm1 = -0.5 * p.mu * s2c2 * p.ir0;
    const double gmdt = -0.5 * p.mu * s3c3;
    const double fdot = -0.5 * p.mu * s * c[1] * (irr * p.ir0);
    const double gdm1 = -0.5 * p.mu * s2c2 * irr;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        h[k] = fm1 * r[k] + gmdt * g[k];
        h[3 + k] = fdot * r[k] + gdm1 * g[k];
    }
}

__device__ __forceinline__ int uv_halfdisp(double eps_th, double dt, const double r[3], const double g[3],
                                           double h[6])
{
#pragma unroll
    for (int k = 0; k < 6; k++) h[k] = 0.0;
    if (dt == 0.0) return 0;
    const UvPair p = uv_prepare(eps_th, r, g);
    double s = uv_start(p, dt);
    double ifp;
    const int it = uv_iterate(p, dt, s, &ifp);
    uv_compose(p, s, r, g, h, ifp);
    return it;
}

// uv_halfdisp from the fifth-order start: no Newton correction where the series alone is
// exact (returns 0 iterations for those pairs).  The ALG kernels keep uv_halfdisp.
__device__ __forceinline__ int uv_halfdisp_fast(double eps_th, double dt, const double r[3], const double g[3],
                                                double h[6])
{
#pragma unroll
    for (int k = 0; k < 6; k++) h[k] = 0.0;
    if (dt == 0.0) return 0;
    const UvPair p = uv_prepare(eps_th, r, g);
    const UvSeries q = uv_series(p, dt);
    if (q.exact) {
        uv_compose_series(p, q, dt, r, g, h);
        return 0;
    }
    double s = uv_series_start(q);
    double ifp = 0.0;
    const int it = uv_iterate(p, dt, s, &ifp);
    uv_compose<true>(p, s, r, g, h, ifp);
    return it;
}

// ---------------------------------------------------------------------------
// The short-step pair: f and g by their own power series in dt, without branches.
//
// With w = g dt, a = r.w/r0^2, b = |w|^2/r0^2, U = mu dt^2/r0^3 and q = b - U, the Taylor series
// of f, g, f' and g' (from f'' = -U f/rho^3, rho^2 = |f r + g v|^2 in units of r0 and dt) are
//   f - 1   = -(U/2) (1 + p1 + p2 + p3 + p4 + p5),      f' dt  = -U (1 + 3/2 p1 + 2 p2 + 5/2 p3 + 3 p4 + 7/2 p5),
//   g - dt  = -(U dt/6) (1 + g1 + g2 + g3 + g4),        g' - 1 = -(U/2) (1 + 4/3 g1 + 5/3 g2 + 2 g3 + 7/3 g4),
//   p1 = -a,  p2 = 5/4 a^2 - q/4 - U/12,  p3 = -(a/4) (7a^2 - 3q - U),
//   p4 = a^2 (21/8 a^2 - 7/4 q - 7/12 U) + q (q/8 + U/15) + U^2/360,  p5 ~ -a p4,  and
//   g1 = 3/2 p1,  g2 = 9/5 p2 + U/10,  g3 = 2 p3 - a U/4,  g4 ~ 15/7 p4.
//
// A pair is a short-step one where b + |U| <= 1.9e-7.  As a^2 <= b, the terms c_k of uv_series are
// then inside its exactness bounds (3e-4)^k (c2 = a^2/2 - q/6, c3 = (a/2) (-9/2 c2 + a^2 + U/12),
// c4 = a^2 (7/8 a^2 - 3/4 q - U/8) + q (3/40 q + U/120); checked on 2e7 points of the region), so
// these pairs take no Newton iteration there either, and |a| <= 4.4e-4, p3 <= 9e-11, p4 <= 4e-14.  The
// terms from p3 on (and the U terms of g2, which multiply a contribution of at most 2e-4 of h) are
// formed in FP32: their rounding stays below 2e-17 of the result.  What is left out (p5 beyond -a p4,
// g4 in g - dt, the sixth order) is below that too.  Everything from p2 down is FP64.
//
// It works on w (relative velocities times dt, so that neither dt/r0 nor its square is formed; the difference is taken
// before the product, walk_diff) and leaves the
// constant factors of the half-displacement to the sums: h = 1/4 (H[0..2]) and (1/2)/dt (H[3..5]).
// Returns false, H undefined, for any other pair: the caller takes the general solver.  Every
// operation is written out, so that each kernel that inlines it computes the same bits; H
// changes sign exactly with r and w.
// ---------------------------------------------------------------------------
struct UvFastStep {
    double dt, dt2;
    bool on;  // steps whose square and reciprocal are far from the limits of the type
};

__device__ __forceinline__ UvFastStep uv_fast_step(double dt)
{
    return {dt, dt * dt, dt > 1e-100 && dt < 1e100};
}

// cdt2: eps_ij dt^2
__device__ __forceinline__ bool uv_fast_pair(double cdt2, const double r[3], const double w[3], double H[6])
{
    const double r2 = fma(r[2], r[2], fma(r[1], r[1], __dmul_rn(r[0], r[0])));
    const double rw = fma(r[2], w[2], fma(r[1], w[1], __dmul_rn(r[0], w[0])));
    const double w2 = fma(w[2], w[2], fma(w[1], w[1], __dmul_rn(w[0], w[0])));
    const double ir = rsqrt_normal(r2);
    const double ir2 = __dmul_rn(ir, ir);
    const double nU = __dmul_rn(__dmul_rn(cdt2, ir), ir2);  // -U
    const double a = __dmul_rn(rw, ir2);
    const double q = fma(w2, ir2, nU);

    // the short-step test and the terms from the third order on, in FP32
    const float af = __double2float_rn(a), qf = __double2float_rn(q), Uf = -__double2float_rn(nU);
    const bool ok = __fadd_rn(__fadd_rn(qf, Uf), fabsf(Uf)) <= 1.9e-7f;
    const float A = __fmul_rn(af, af);
    const float p3 = __fmul_rn(__fmul_rn(-0.25f, af), __fmaf_rn(7.0f, A, __fmaf_rn(-3.0f, qf, -Uf)));
    const float p4 = __fmaf_rn(A, __fmaf_rn(2.625f, A, __fmaf_rn(-1.75f, qf, __fmul_rn(-7.0f / 12.0f, Uf))),
                               __fmaf_rn(qf, __fmaf_rn(0.125f, qf, __fmul_rn(1.0f / 15.0f, Uf)),
                                         __fmul_rn(Uf, __fmul_rn(1.0f / 360.0f, Uf))));
    const float p45 = __fmaf_rn(-af, p4, p4);
    const float cf = __fadd_rn(p3, p45);
    const float cfd = __fmaf_rn(2.5f, p3, __fmul_rn(3.0f, p45));
    const float aU = __fmul_rn(af, Uf);
    const float cg = __fmaf_rn(2.0f / 3.0f, p3, __fmaf_rn(-0.25f / 3.0f, aU, __fmul_rn(0.1f / 3.0f, Uf)));
    const float cgd = __fmaf_rn(2.0f, p3, __fmaf_rn(2.5f, p4, __fmaf_rn(-0.25f, aU, __fmul_rn(1.0f / 12.0f, Uf))));

    // the leading terms in FP64, the small ones first (a multiply-add with one constant operand each, so
    // that no constant waits in a register): the four series, that of g - dt over 3, of g' - 1 over 2
    const double p2 = fma(1.25, __dmul_rn(a, a), fma(-0.25, q, __dmul_rn(1.0 / 12.0, nU)));
    const double sf = __dadd_rn(__dsub_rn(__dadd_rn(p2, (double)cf), a), 1.0);
    const double sfd = __dadd_rn(fma(2.0, fma(-0.75, a, p2), (double)cfd), 1.0);
    const double sg = __dadd_rn(fma(0.6, p2, fma(-0.5, a, (double)cg)), 1.0 / 3.0);
    const double sgd = __dadd_rn(__dsub_rn(fma(1.5, p2, (double)cgd), a), 0.5);
    const double F = __dmul_rn(nU, sf), G = __dmul_rn(nU, sg);
    const double Fd = __dmul_rn(nU, sfd), Gd = __dmul_rn(nU, sgd);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        H[k] = fma(F, r[k], __dmul_rn(G, w[k]));
        H[3 + k] = fma(Fd, r[k], __dmul_rn(Gd, w[k]));
    }
    return ok;
}


// ---------------------------------------------------------------------------
// One pair: frame, classification, solve, half-displacement (bia/bia.f90:141-191).
// Returns the half-displacement in h[6] = (dX, dY, dZ, dU, dV, dW)/2 terms.
// ---------------------------------------------------------------------------
// ALG pair classes (bia/bia.f90:156-166 plus the guards): the branch each pair takes.
enum AlgClass { kClsHyp = 0, kClsEll = 1, kClsUv = 2, kClsPar = 3, kClsDeg = 4 };

// Branch of an ALG pair: E == 0 exactly keeps the reference's parabola branch; zero |g| or
// |L| (degenerate) and |e^2 - 1| = |E| L^2 / eps^2 < 0.1 go to the universal-variable
// solver; otherwise hyperbola (E > 0) or ellipse (E < 0).
__device__ __forceinline__ int alg_classify(double eps_ij, const double r[3], const double g[3], double &E_out,
                                            double &Lsq_out)
{
    const double gsq = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
    const double L0 = r[1] * g[2] - r[2] * g[1];
    const double L1 = r[2] * g[0] - r[0] * g[2];
    const double L2 = r[0] * g[1] - r[1] * g[0];
    const double Lsq = L0 * L0 + L1 * L1 + L2 * L2;
    const double rsq = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    double E_ij = gsq + 2.0 * eps_ij * rsqrt_normal(rsq);
    // near zero (a parabola is E == 0 exactly) and beyond the approximation's range, the root and division
    if (!(fabs(E_ij) > 1e-12 * gsq && rsq > 1e-290)) E_ij = gsq + 2.0 * eps_ij / sqrt(rsq);
    E_out = E_ij;
    Lsq_out = Lsq;
    if (E_ij == 0.0) return kClsPar;
    if (gsq == 0.0 || Lsq == 0.0) return kClsDeg;
    if (fabs(E_ij) * Lsq < kNearUnitEcc * (eps_ij * eps_ij)) return kClsUv;
    return (E_ij > 0.0) ? kClsHyp : kClsEll;
}

__device__ __forceinline__ int alg_classify(double eps_ij, const double r[3], const double g[3])
{
    double E, Lsq;
    return alg_classify(eps_ij, r, g, E, Lsq);
}

// |g| == 0 or |L| == 0: the pair's frame is degenerate (counted apart from the other
// universal-variable pairs)
__device__ __forceinline__ bool pair_degenerate(const double r[3], const double g[3])
{
    const double gsq = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
    const double L0 = r[1] * g[2] - r[2] * g[1];
    const double L1 = r[2] * g[0] - r[0] * g[2];
    const double L2 = r[0] * g[1] - r[1] * g[0];
    return gsq == 0.0 || (L0 * L0 + L1 * L1 + L2 * L2) == 0.0;
}

// M: the compiled method (kMethodRkf or kMethodAlg); each kernel is
// instantiated per method so it carries only that method's code and registers.
constexpr int kMethodRkf = 0, kMethodAlg = 1, kMethodUniversal = 2, kMethodLearned = 3;

__device__ __forceinline__ void count_nonfinite(const double h[6], PairCounters &cnt)
{
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 6; k++) finite = finite && isfinite(h[k]);
    if (!finite) cnt.nonfinite++;
}

// Half-displacement from the in-plane solution: h = ((dr . e - g dt) / 2, (dg . e) / 2)
// (bia/bia.f90:170-191).
__device__ __forceinline__ void compose_halfdisp(const PairParams &P, const double g[3], const double e_xi[3],
                                                 const double e_eta[3], const double YZ[4],
                                                 const double YN[4], double h[6])
{
    const double dr_xi = YN[0] - YZ[0], dr_eta = YN[1] - YZ[1];
    const double dg_xi = YN[2] - YZ[2], dg_eta = YN[3] - YZ[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        h[k] = (dr_xi * e_xi[k] + dr_eta * e_eta[k] - g[k] * P.dt) * 0.5;
        h[3 + k] = (dg_xi * e_xi[k] + dg_eta * e_eta[k]) * 0.5;
    }
}

// ALG pair whose class C is known (kClsHyp, kClsEll or kClsPar): frame, conic solver,
// half-displacement (bia/bia.f90:141-191).
template <int C>
__device__ __forceinline__ void alg_conic_pair(const PairParams &P, double eps_ij, const double r[3],
                                               const double g[3], double h[6], PairCounters &cnt)
{
    double e_xi[3], e_eta[3], YZ[4], YN[4];
    double error = 0.0;
    frame_xi_eta(r, g, e_xi, e_eta, YZ);
    if (C == kClsHyp) {
        int bx = 0, fb = 0;
        cnt.it_hyp += hyperbola(eps_ij, P.dt, P.itr, YZ, YN, &error, &bx, &fb);
        cnt.bracket_exits += bx;
        cnt.fallbacks += fb;
        cnt.cls[kHyperbola]++;
    } else if (C == kClsEll) {
        int fb = 0;
        cnt.it_ell += ellipse(eps_ij, P.dt, P.itr, YZ, YN, &error, &fb);
        cnt.fallbacks += fb;
        cnt.cls[kEllipse]++;
    } else {
        cnt.it_par += parabola(eps_ij, P.dt, YZ, YN, &error);
        cnt.cls[kParabola]++;
    }
    if (fabs(error) > P.err) cnt.nonconverged++;
    compose_halfdisp(P, g, e_xi, e_eta, YZ, YN, h);
    count_nonfinite(h, cnt);
}

// ALG pair of the rare classes (parabola, degenerate, near-unit eccentricity): c is
// alg_classify's answer for it.
__device__ __forceinline__ void alg_rare_pair(const PairParams &P, double eps_ij, const double r[3],
                                              const double g[3], double h[6], PairCounters &cnt, int c)
{
    if (c == kClsPar) {
        alg_conic_pair<kClsPar>(P, eps_ij, r, g, h, cnt);
    } else {
        const int it = uv_halfdisp(eps_ij, P.dt, r, g, h);
        cnt.it_uv += it;
        if (it > kUvItMax) cnt.nonconverged++;
        cnt.cls[c == kClsDeg ? kDegenerate : kUniversal]++;
        count_nonfinite(h, cnt);
    }
}

template <int M>
__device__ __forceinline__ void pair_halfdisp(const PairParams &P, double eps_ij, const double r[3],
                                              const double g[3], double h[6], PairCounters &cnt)
{
    if (M == kMethodAlg) {
        const int c = alg_classify(eps_ij, r, g);
        if (c == kClsUv || c == kClsDeg) {
            alg_rare_pair(P, eps_ij, r, g, h, cnt, c);
        } else {
            // one copy of the frame and composition for the three conic branches
            double e_xi[3], e_eta[3], YZ[4], YN[4];
            double error = 0.0;
            frame_xi_eta(r, g, e_xi, e_eta, YZ);
            if (c == kClsHyp) {
                int bx = 0, fb = 0;
                cnt.it_hyp += hyperbola(eps_ij, P.dt, P.itr, YZ, YN, &error, &bx, &fb);
                cnt.bracket_exits += bx;
                cnt.fallbacks += fb;
                cnt.cls[kHyperbola]++;
            } else if (c == kClsEll) {
                int fb = 0;
                cnt.it_ell += ellipse(eps_ij, P.dt, P.itr, YZ, YN, &error, &fb);
                cnt.fallbacks += fb;
                cnt.cls[kEllipse]++;
            } else {
                cnt.it_par += parabola(eps_ij, P.dt, YZ, YN, &error);
                cnt.cls[kParabola]++;
            }
            if (fabs(error) > P.err) cnt.nonconverged++;
            compose_halfdisp(P, g, e_xi, e_eta, YZ, YN, h);
            count_nonfinite(h, cnt);
        }
    } else {
        double e_xi[3], e_eta[3], YZ[4], YN[4];
        double error = 0.0;
        const bool degenerate = frame_xi_eta(r, g, e_xi, e_eta, YZ);
        int nacc = 0;
        rkf_pair(eps_ij, P.dt, P.relerr, P.abserr, YZ, YN, &error, &nacc);
        cnt.cls[degenerate ? kDegenerate : kRkf]++;
        cnt.rkf_steps += nacc;
        if (fabs(error) > P.err) cnt.nonconverged++;
        compose_halfdisp(P, g, e_xi, e_eta, YZ, YN, h);
        count_nonfinite(h, cnt);
    }
}

}  // namespace bia
