// rf_device.cuh - device-side building blocks shared by the assembly and
// velocity kernels: quadrature tables, the analytic inner integral of
// Int_analytical.f90 and the Stokeslet/doublet tensor.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace rf {

constexpr int kMaxN = 8;
constexpr int kMaxLQ = 48;  // NoQI <= 16

// Per-run tables in device memory, staged to shared memory by each CTA.
struct Tables {
    int N, LQ;
    double pv[kMaxLQ];               // Gauss points on [-1,1]   (quadrature.f90:78-84)
    double wv[kMaxLQ];               // weights (sum 2)
    double P[kMaxN + 1][kMaxLQ];     // P_m(pv[q]), m = 0..N      (matrix_assembly.f90:36-56)
    double eps2;                     // slenderness squared
    double D1;                       // 0.75/(d-2)                 (matrix_assembly.f90:462)
    double Ek[kMaxN + 1];            // E_k                        (:484)
    double gamma[kMaxN + 1];         // gamma_k                    (:582)
    double d;                        // -log(eps^2 e)
    double e;                        // 2
    double half_force[3];            // 0.5 * ExtForce
    double force[3];                 // ExtForce
};

// Legendre P_m = scale_m * sum_p a_mp s^p with the integer coefficients of the
// Fortran combinations (Int_analytical.f90:213-288), highest power first.
__host__ __device__ constexpr double leg_scale(int m) {
    return m <= 1 ? 1.0 : (m <= 3 ? 0.5 : (m <= 5 ? 0.125 : (m <= 7 ? 0.0625 : 1.0 / 128.0)));
}
__host__ __device__ constexpr double leg_coef(int m, int p) {
    // row m, power p
    return m == 0 ? (p == 0 ? 1 : 0)
         : m == 1 ? (p == 1 ? 1 : 0)
         : m == 2 ? (p == 2 ? 3 : p == 0 ? -1 : 0)
         : m == 3 ? (p == 3 ? 5 : p == 1 ? -3 : 0)
         : m == 4 ? (p == 4 ? 35 : p == 2 ? -30 : p == 0 ? 3 : 0)
         : m == 5 ? (p == 5 ? 63 : p == 3 ? -70 : p == 1 ? 15 : 0)
         : m == 6 ? (p == 6 ? 231 : p == 4 ? -315 : p == 2 ? 105 : p == 0 ? -5 : 0)
         : m == 7 ? (p == 7 ? 429 : p == 5 ? -693 : p == 3 ? 315 : p == 1 ? -35 : 0)
         : (p == 8 ? 6435 : p == 6 ? -12012 : p == 4 ? 6930 : p == 2 ? -1260 : p == 0 ? 35 : 0);
}

// Moments I_n = int s^n/R, J_n = int s^n/R^3, S_n = int s^n/R^5 over s in
// [-1,1], R = |R0 - s pb|, n = 0..N+2 (Int_analytical.f90:72-207).
// Forward recursion when c < 10, backward recursion from n = 27 otherwise,
// closed forms for n = 0, 1 with the d < 1e-14 special branch.
// The FP64 instance follows the reference formulas; divisions by loop
// constants are folded into compile-time reciprocals.
// Non-contracted FP64 arithmetic: the reference evaluates the closed forms
// and the forward recursion without fused multiply-adds, and the forward
// recursion amplifies every rounding difference, so these parts follow the
// Fortran operation order exactly.
__device__ __forceinline__ double fmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double fsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double fdiv(double a, double b) { return __ddiv_rn(a, b); }

// x / OM for a small integer OM, correctly rounded: q = RN(x r), r = RN(1/OM),
// then one step with the exact remainder, RN(q + (x - q OM) r) (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990).  q is within two units of the quotient, so the remainder is a
// multiple of q's unit below 2^6 units and the fused multiply-add forms it
// exactly; the corrected sum is off by less than 2^-50 units before its
// rounding, and x / OM (OM = 2^k times an odd m) is either representable or at
// least 1/(2m) units away from a rounding boundary.  Three instructions for
// the general division's dozen.
template <int OM>
__device__ __forceinline__ double div_const(double x) {
    constexpr int m = OM < 0 ? -OM : OM;
    constexpr double r = 1.0 / OM;
    const double q = __dmul_rn(x, r);
    if constexpr ((m & (m - 1)) == 0) return q;  // a power of two: exact
    else return __fma_rn(__fma_rn(-q, (double)OM, x), r, q);
}

// 1/x and 1/sqrt(x) of a positive normal x, within two units: the hardware's
// approximation y (relative error below 2^-19), then the series in e = 1 - x y
// (1/x = y / (1 - e)) or e = 1 - x y^2 (1/sqrt(x) = y (1 - e)^(-1/2)) up to
// e^2; the first neglected terms are e^3 and 5/16 e^3.  Three and five FP64
// operations and no branch.
__device__ __forceinline__ double rcp_pos(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsqrt_pos(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
// a / b from y = 1/b within u units (2^-53, relative; u is 2 for rcp_pos(b) and
// below 13 for the products of reciprocals that the closed forms pass), and
// sqrt(x): one correction with the remainder (Markstein 1990, as div_const).
// The quotient to be corrected is within u + 1 units, the remainder formed to a
// rounding of itself, so that the corrected sum is off by less than (u + 1)
// (u + 2) 2^-53 units before its rounding, 2^-45 at the most: the correctly
// rounded value except where the quotient or root lies that close to a rounding
// boundary.  The compiler's division and square root branch to a path for
// subnormal and special operands, so that the ten divisions of the closed forms
// run one after the other; these interleave, and quotients of one denominator
// share its reciprocal.  A zero or infinite operand gives NaN (the reference's
// formulas are singular there).
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}
__device__ __forceinline__ double sqrt_pos(double x) {
    const double y = rsqrt_pos(x);
    const double g = __dmul_rn(x, y);
    return __fma_rn(__fma_rn(-g, g, x), 0.5 * y, g);
}

// Steps n .. K-1 of the reference's forward recursion (Int_analytical.f90:
// 123-136, 172-176, 197-200) in its operation order; Fortran nn = n + 1.
template <int n, int K>
struct ForwardStep {
    __device__ __forceinline__ static void run(double b, double c, double ue, double ub, double *I, double *J,
                                               double *S) {
        if constexpr (n < K) {
            const double t1 = div_const<-n>(ue);
            const double t2 = div_const<-n>(n % 2 == 1 ? ub : -ub);  // sb**(ii-2) ub
            const double t3 = fmul(div_const<-n>(fmul(0.5 - n, b)), I[n - 1]);
            const double t4 = fmul(div_const<-n>(fmul(n - 1.0, c)), I[n - 2]);
            I[n] = fadd(fsub(fsub(t2, t1), t3), t4);
            J[n] = fsub(fsub(I[n - 2], fmul(b, J[n - 1])), fmul(c, J[n - 2]));
            S[n] = fsub(fsub(J[n - 2], fmul(b, S[n - 1])), fmul(c, S[n - 2]));
            ForwardStep<n + 1, K>::run(b, c, ue, ub, I, J, S);
        }
    }
};

constexpr double kFormsMaxC = 1e100;  // largest |R0|^2 at which moments_fp64 uses reciprocals

template <int N>
__device__ __forceinline__ void moments_fp64(double b, double c, double *I, double *J, double *S) {
    constexpr int K = N + 3;
    // Int_analytical.f90:96-102
    const double ue = sqrt_pos(fadd(fadd(1.0, b), c));
    const double ub = sqrt_pos(fadd(fsub(1.0, b), c));
    const double te = fadd(1.0, fmul(0.5, b));
    const double tb = fadd(-1.0, fmul(0.5, b));
    const double d = fsub(c, fmul(fmul(0.25, b), b));
    const double rue = rcp_pos(ue), rub = rcp_pos(ub);
    const double j1c = fadd(div_by(-1.0, ue, rue), div_by(1.0, ub, rub));
    // :113-114
    I[0] = fsub(log(fabs(fadd(fadd(2.0, b), fmul(2.0, ue)))), log(fabs(fadd(fadd(-2.0, b), fmul(2.0, ub)))));
    I[1] = fsub(fsub(ue, ub), fmul(fmul(0.5, b), I[0]));
    // :162-170, 189-196
    if (d < 1e-14) {
        const double e1 = fadd(1.0, fmul(b, 0.5)), e2 = fadd(-1.0, fmul(b, 0.5));  // b/2 is exact
        J[0] = fadd(fdiv(-1.0, fmul(2.0, fmul(e1, e1))), fdiv(1.0, fmul(2.0, fmul(e2, e2))));
        J[1] = fsub(j1c, fmul(fmul(b, 0.5), J[0]));
        const double p = fadd(2.0, b), m = fadd(-2.0, b);
        const double p2 = fmul(p, p), m2 = fmul(m, m);
        S[0] = fadd(fdiv(-4.0, fmul(p2, p2)), fdiv(4.0, fmul(m2, m2)));
        S[1] = fsub(fadd(fdiv(-8.0, fmul(3.0, fmul(p2, p))), fdiv(8.0, fmul(3.0, fmul(m2, m)))),
                    fmul(fmul(b, 0.5), S[0]));
    } else if (c > kFormsMaxC) {
        // the products of d, ue and ub overflow from c = 10^122 on, and a quotient
        // by infinity is zero, which the reciprocals below do not give
        const double ue3 = fmul(fmul(ue, ue), ue), ub3 = fmul(fmul(ub, ub), ub), d3 = fmul(3.0, d), d6 = fmul(6.0, d);
        J[0] = fsub(fdiv(te, fmul(d, ue)), fdiv(tb, fmul(d, ub)));
        J[1] = fsub(j1c, fmul(fmul(b, 0.5), J[0]));
        S[0] = fadd(fsub(fdiv(fadd(2.0, b), fmul(d6, ue3)), fdiv(fadd(-2.0, b), fmul(d6, ub3))),
                    fmul(fdiv(2.0, d3), J[0]));
        S[1] = fsub(fadd(fdiv(-fadd(b, fmul(2.0, c)), fmul(d6, ue3)), fdiv(fadd(-b, fmul(2.0, c)), fmul(d6, ub3))),
                    fmul(fdiv(b, d3), J[0]));
    } else {
        const double due = fmul(d, ue), dub = fmul(d, ub), d3 = fmul(3.0, d), d6 = fmul(6.0, d);
        const double de = fmul(d6, fmul(fmul(ue, ue), ue)), db = fmul(d6, fmul(fmul(ub, ub), ub));
        // the reciprocals of the five products of d, ue and ub from theirs
        const double rd = rcp_pos(d), r6 = rd * (1.0 / 6.0);
        const double rde = r6 * rue * rue * rue, rdb = r6 * rub * rub * rub, rd3 = rd * (1.0 / 3.0);
        J[0] = fsub(div_by(te, due, rd * rue), div_by(tb, dub, rd * rub));
        J[1] = fsub(j1c, fmul(fmul(b, 0.5), J[0]));
        S[0] = fadd(fsub(div_by(fadd(2.0, b), de, rde), div_by(fadd(-2.0, b), db, rdb)),
                    fmul(div_by(2.0, d3, rd3), J[0]));
        S[1] = fsub(fadd(div_by(-fadd(b, fmul(2.0, c)), de, rde), div_by(fadd(-b, fmul(2.0, c)), db, rdb)),
                    fmul(div_by(b, d3, rd3), J[0]));
    }
    if (c < 10.0) {
        // forward recursion, :123-136, 172-176, 197-200
        ForwardStep<2, K>::run(b, c, ue, ub, I, J, S);
    } else {
        // backward recursion from n = 27 (:137-157, 177-183, 201-206); stable, so
        // folded constants and fused arithmetic are used here
        const double ic = 1.0 / c;
        double i1 = 0.0, i2 = 0.0, j1 = 0.0, j2 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll
        for (int n = 27; n >= 2; --n) {
            const double nn = n;                                       // Fortran nn = ii - 1
            const double a0 = (nn + 2.0) / (nn + 1.0);
            const double r2 = 1.0 / (nn + 2.0);
            const double cb = (1.0 - 2.0 * (nn + 2.0)) / (2.0 * (nn + 2.0));
            const double sbp = ((n + 1) % 2 == 0) ? 1.0 : -1.0;        // (-1)^(nn+1)
            const double in = a0 * ic * (ue * r2 - sbp * ub * r2 + cb * b * i1 - i2);
            const double jn = ic * (in - b * j1 - j2);
            const double sn = ic * (jn - b * s1 - s2);
            if (n < K) { I[n] = in; J[n] = jn; S[n] = sn; }
            i2 = i1; i1 = in; j2 = j1; j1 = jn; s2 = s1; s1 = sn;
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 far points.  The kernels that need the moments only as
// u_p = I_p + 2 eps^2 J_p (p = 0..N) and v_p = J_p - 6 eps^2 S_p (p = 0..N+2)
// take a far point (10 <= c < 4096, outside a cone about the source axis) through the
// backward recursion alone, run down to n = 0: the three-term relations that
// the reference uses for n >= 2 hold at n = 0, 1 too.  That leaves out the two
// logarithms and ten divisions of the closed forms: about 260 FP64
// instructions for the reference's 450.  Where the lines lie: below c = 10 the
// reference recurs forward and amplifies every rounding, so those points
// follow its operation order (moments_fp64); in the cone (d = c - b^2/4 below
// kAxisRatio c: 1 point in 2000 of an isotropic suspension; kAxisRatioNear c
// while c < 16) its closed forms lose digits to the divisions by d and its
// start at n = 27 leaves up to 2e-9 |J_0|, and parity with it is kept; from 64
// half-lengths on its closed forms' cancellation (a relative error that grows
// like c, 4e-9 at c = 10^6) would show against the recursion likewise.
// The start (far_top): zero starting values reach n <= 7 damped by c^(-n/2)
// times a polynomial in n, and an even start is closer than an odd one, so it
// falls with c.  The lines lie where the Legendre combinations (m <= 5) of I_n,
// J_n, S_n, relative to I_0, J_0, S_0 and against 40 digits, have a mean, median
// and largest error over isotropic directions that are no larger than those of
// the reference's formulas in FP64 (its start at 27, the closed forms'
// cancellation): mean of J just above the lines 16, 45, 65, 105, 190, 420 9.6e-13,
// 7e-16, 1e-15, 2e-15, 5e-15, 9e-15 (reference 2.2e-12, 8e-15, 2e-14, 2e-14,
// 6e-14, 1e-13), and at 10 and 13 1.2e-12 and 6e-13 (2e-10, 1e-11).  N = 8 with
// its four steps more likewise.  Lines at 16, 20, 30, 48, 80, 150 left up to 100
// times the reference's error; the higher starts cost 0.5 ms of an assembly and
// 0.6 ms of the velocities at M = 4000 (21.8 and 14.4 ms).
constexpr double kFarC = 10.0;
constexpr double kFarMaxC = 4096.0;
constexpr double kAxisRatio = 1e-3, kAxisRatioNear = 1e-2;
__device__ __forceinline__ bool far_point(double b, double c) {
    return c >= kFarC && c < kFarMaxC && fma(-0.25 * b, b, c) >= (c < 16.0 ? kAxisRatioNear : kAxisRatio) * c;
}
__device__ __forceinline__ int far_top(float c) {
    return 16 + 2 * ((c < 420.f) + (c < 190.f) + (c < 105.f) + (c < 65.f) + (c < 45.f) + (c < 16.f) + (c < 13.f));
}

// Step n: I_n = -(1 + r/2) (b/c) I_{n+1} - (1 + r) (1/c) I_{n+2} + r w, r =
// 1/(n+1), w = (ue -+ ub)/c.  r comes from a table in shared memory for the
// steps above Far<N>::kTail, which run as a loop (a fully unrolled recursion
// exceeds the instruction cache that a scheduler's warps share).  N > 5 needs
// n up to 10 and starts four steps higher.
template <int N>
struct Far {
    static constexpr int kShift = N <= 5 ? 0 : 4;
    static constexpr int kTail = N <= 5 ? 8 : 10;
    static constexpr int kCoef = 30 + kShift - kTail;  // entries of the table
    // entry t of the table: r of step kTail + 1 + t
    __device__ __forceinline__ static double coef(int t) { return 1.0 / (kTail + 2.0 + t); }
};

struct FarState {
    double nicb, hicb, nic, wp, wm, ic;      // -b/c, -b/(2c), -1/c, (ue - ub)/c, (ue + ub)/c, 1/c
    double i1, i2, j1, j2, s1, s2;           // I, c J, c^2 S at n + 1, n + 2
    __device__ __forceinline__ void step(double r, double w) {
        const double in = fma(fma(r, hicb, nicb), i1, fma(fma(r, nic, nic), i2, r * w));
        const double jn = fma(nicb, j1, fma(nic, j2, in));
        const double sn = fma(nicb, s1, fma(nic, s2, jn));
        i2 = i1; i1 = in; j2 = j1; j1 = jn; s2 = s1; s1 = sn;
    }
};

// the last steps, n .. 0; u_n and v_n to out as soon as they are formed
template <int N, int n, typename OUT>
__device__ __forceinline__ void far_tail(FarState &f, double e2, double e6, OUT &&out) {
    if constexpr (n >= 0) {
        f.step(1.0 / (n + 1.0), n % 2 == 1 ? f.wp : f.wm);
        if constexpr (n <= N) out.u(n, fma(e2, f.j1, f.i1));
        if constexpr (n <= N + 2) out.v(n, fma(f.ic, f.j1, e6 * f.s1));
        far_tail<N, n - 1>(f, e2, e6, out);
    }
}

// u_p and v_p of a far point, from the start its own c asks for: a point's
// moments do not depend on the points beside it.  coef: the table above.
// ue ub = sqrt((1 + c)^2 - b^2) and (ue + ub)^2 = 2 (1 + c + ue ub); ue - ub =
// 2b / (ue + ub).
template <int N, typename OUT>
__device__ __forceinline__ void moments_far_fp64(double b, double c, double eps2, const double *coef, OUT &&out) {
    const double t = 1.0 + c, pp = fma(t, t, -b * b);
    const double us2 = 2.0 * fma(pp, rsqrt_pos(pp), t);
    const double ius = rsqrt_pos(us2);
    FarState f;
    f.ic = rcp_pos(c);
    f.nic = -f.ic;
    f.nicb = f.nic * b;
    f.hicb = 0.5 * f.nicb;
    f.wp = -2.0 * f.nicb * ius;
    f.wm = us2 * ius * f.ic;
    f.i1 = f.i2 = f.j1 = f.j2 = f.s1 = f.s2 = 0.0;
    const double *k = coef + (far_top((float)c) + Far<N>::kShift - Far<N>::kTail - 2);  // of the odd step below the start
#pragma unroll 1
    for (; k >= coef; k -= 2) {
        f.step(k[1], f.wm);  // even n
        f.step(k[0], f.wp);  // odd n
    }
    const double e2 = 2.0 * eps2 * f.ic;
    far_tail<N, Far<N>::kTail>(f, e2, -3.0 * e2 * f.ic, out);
}

// The same families of any point from the reference's moments.
template <int N, typename OUT>
__device__ __forceinline__ void moments_near_uv(double b, double c, double eps2, OUT &&out) {
    double I[N + 3], J[N + 3], S[N + 3];
    moments_fp64<N>(b, c, I, J, S);
#pragma unroll
    for (int p = 0; p <= N; ++p) out.u(p, fma(2.0 * eps2, J[p], I[p]));
#pragma unroll
    for (int p = 0; p <= N + 2; ++p) out.v(p, fma(-6.0 * eps2, S[p], J[p]));
}

// First index of the FP32 backward recursion.  Its starting values
// I = J = S = 0 at n + 1, n + 2 are wrong by the true moments there; the error
// reaches n = 0 damped by c^(-n/2) (the recursion's homogeneous solutions grow
// like |lambda|^n, lambda^2 + b lambda + c = 0, |lambda| = sqrt(c) since
// d >= 0) times a polynomial in n that is largest for the S moments of a point
// on the source axis.  From n = 32 that error is below FP32 rounding for every
// c >= 6 and every direction: with sampled b, the Legendre combinations of the
// moments stay within 8e-7 of |X_0| (X = I, J, S) at c = 6, 6.5, 7, 8 on and
// off the axis; from the reference's n = 27 the on-axis S error is 1e-5 at c = 6.
constexpr int kBackTop = 32;

// FP32 moments by the backward recursion alone, run down to n = 0.  The
// three-term relations that the reference uses for n >= 2
// (Int_analytical.f90:137-157, 177-183, 201-206) hold at n = 0 and 1 as well:
// d/ds[s^(n+1) R] = ((n+2) s^(n+2) + (n+3/2) b s^(n+1) + (n+1) c s^n) / R and
// s^n / R = s^n (s^2 + b s + c) / R^3.  The reference's n = 0, 1 closed forms
// (a logarithm of a ratio close to 1, ue - ub - b I_0 / 2, 1/ub - 1/ue and the
// S_0, S_1 differences over d) cancel by a factor that grows like c: a pair
// 100 fiber half-lengths apart loses every FP32 digit in them, and at a point
// near the source axis the 1/d forms cancel too.  The recursion has neither
// cancellation: ue - ub enters only as 2b / (ue + ub), and d not at all.
// Accurate for c >= 6 in every direction (see kBackTop).
template <int N>
__device__ __forceinline__ void moments_backward_fp32(float b, float c, float *I, float *J, float *S) {
    constexpr int K = N + 3;
    const float xe = 1.0f + b + c, xb = 1.0f - b + c;
    const float ue = xe * rsqrtf(xe), ub = xb * rsqrtf(xb);
    const float ic = __fdividef(1.0f, c);
    const float icb = ic * b;
    const float icwp = __fdividef(2.0f * b, ue + ub) * ic;  // (ue - ub) / c
    const float icwm = (ue + ub) * ic;
    const float nic = -ic, nicb = -icb, ic2 = ic * ic;
    // J and S are carried as c J_n and c^2 S_n: their steps become two fused
    // multiply-adds each, c J_n = I_n - (b/c) c J_{n+1} - (1/c) c J_{n+2} and
    // c^2 S_n = c J_n - (b/c) c^2 S_{n+1} - (1/c) c^2 S_{n+2}
    float i1 = 0.f, i2 = 0.f, j1 = 0.f, j2 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int n = kBackTop; n >= 0; --n) {
        // I_n = (ue - (-1)^(n+1) ub - (n+3/2) b I_{n+1} - (n+2) I_{n+2}) / ((n+1) c)
        const float a0 = (n + 2.0f) / (n + 1.0f);
        const float r2 = 1.0f / (n + 2.0f);
        const float cb = (1.0f - 2.0f * (n + 2.0f)) / (2.0f * (n + 2.0f));
        const float icw = ((n + 1) % 2 == 0) ? icwp : icwm;
        const float in = fmaf((a0 * cb) * icb, i1, fmaf(-a0 * ic, i2, (a0 * r2) * icw));
        const float jn = fmaf(nicb, j1, fmaf(nic, j2, in));
        const float sn = fmaf(nicb, s1, fmaf(nic, s2, jn));
        if (n < K) { I[n] = in; J[n] = jn * ic; S[n] = sn * ic2; }
        i2 = i1; i1 = in; j2 = j1; j1 = jn; s2 = s1; s1 = sn;
    }
}

// The same recursion for two points at once on Blackwell's packed FP32 units
// (__ffma2_rn / __fmul2_rn: one instruction, two FMAs, each rounded exactly as
// fmaf): component .x is one point, .y the other, every operation and its
// order as in moments_backward_fp32, so the moments are bit-identical.
template <int N>
__device__ __forceinline__ void moments_backward_fp32x2(float2 b, float2 c, float2 *I, float2 *J, float2 *S) {
    constexpr int K = N + 3;
    const float xe0 = 1.0f + b.x + c.x, xb0 = 1.0f - b.x + c.x;
    const float xe1 = 1.0f + b.y + c.y, xb1 = 1.0f - b.y + c.y;
    const float ue0 = xe0 * rsqrtf(xe0), ub0 = xb0 * rsqrtf(xb0);
    const float ue1 = xe1 * rsqrtf(xe1), ub1 = xb1 * rsqrtf(xb1);
    const float ic0 = __fdividef(1.0f, c.x), ic1 = __fdividef(1.0f, c.y);
    const float2 ic = make_float2(ic0, ic1);
    const float2 icb = make_float2(ic0 * b.x, ic1 * b.y);
    const float2 icwp = make_float2(__fdividef(2.0f * b.x, ue0 + ub0) * ic0, __fdividef(2.0f * b.y, ue1 + ub1) * ic1);
    const float2 icwm = make_float2((ue0 + ub0) * ic0, (ue1 + ub1) * ic1);
    const float2 nic = make_float2(-ic0, -ic1), nicb = make_float2(-icb.x, -icb.y);
    const float2 ic2 = make_float2(ic0 * ic0, ic1 * ic1);
    const float2 z = make_float2(0.f, 0.f);
    float2 i1 = z, i2 = z, j1 = z, j2 = z, s1 = z, s2 = z;
#pragma unroll
    for (int n = kBackTop; n >= 0; --n) {
        const float a0 = (n + 2.0f) / (n + 1.0f);
        const float r2 = 1.0f / (n + 2.0f);
        const float cb = (1.0f - 2.0f * (n + 2.0f)) / (2.0f * (n + 2.0f));
        const float2 icw = ((n + 1) % 2 == 0) ? icwp : icwm;
        const float2 ca = __fmul2_rn(make_float2(a0 * cb, a0 * cb), icb);
        const float2 cn = __fmul2_rn(make_float2(-a0, -a0), ic);
        const float2 cw = __fmul2_rn(make_float2(a0 * r2, a0 * r2), icw);
        const float2 in = __ffma2_rn(ca, i1, __ffma2_rn(cn, i2, cw));
        const float2 jn = __ffma2_rn(nicb, j1, __ffma2_rn(nic, j2, in));
        const float2 sn = __ffma2_rn(nicb, s1, __ffma2_rn(nic, s2, jn));
        if (n < K) {
            I[n] = in;
            J[n] = __fmul2_rn(jn, ic);
            S[n] = __fmul2_rn(sn, ic2);
        }
        i2 = i1; i1 = in; j2 = j1; j1 = jn; s2 = s1; s1 = sn;
    }
}

// Geometry of one (target point, source fiber) item in FP32 for the moments:
// b = -2 p.R0, c = |R0|^2, and the three quantities that the closed forms
// need near the source and that c and b determine only through cancellation:
// ue^2 = 1 + b + c = |R0 - p|^2, ub^2 = 1 - b + c = |R0 + p|^2 and
// d = c - b^2/4 = |R0 x p|^2 (|p| = 1).  Formed from the vectors they keep
// their relative accuracy when a target point comes within 1e-4 of the
// source fiber (fibers that touch or cross); from b and c they round to zero
// or below, and the closed forms then take the root or logarithm of a
// negative number.
struct Geom32 {
    float b, c, ue2, ub2, d;
    __device__ __forceinline__ Geom32(float r0x, float r0y, float r0z, float px, float py, float pz) {
        b = -2.0f * (px * r0x + py * r0y + pz * r0z);
        c = r0x * r0x + r0y * r0y + r0z * r0z;
        const float ex = r0x - px, ey = r0y - py, ez = r0z - pz;
        const float fx = r0x + px, fy = r0y + py, fz = r0z + pz;
        ue2 = ex * ex + ey * ey + ez * ez;
        ub2 = fx * fx + fy * fy + fz * fz;
        const float cx = fmaf(r0y, pz, -r0z * py), cy = fmaf(r0z, px, -r0x * pz), cz = fmaf(r0x, py, -r0y * px);
        d = cx * cx + cy * cy + cz * cz;
    }
};

// FP32 moments for every point of the plain FP32 method and for the far field
// (c >= near_c >= 10) of the tile mixed-precision kernel.  For c >= 6 the
// backward recursion alone (moments_backward_fp32; it needs only b and c): the
// reference switches at 10 in FP64, but its forward recursion amplifies
// rounding by orders of magnitude as c approaches 10, which FP32 cannot
// absorb, while from 6 on the backward recursion is accurate to FP32 rounding.
// Below 6 (plain FP32 method only) the reference's closed forms and forward
// recursion on ue^2, ub^2 and d formed from the vectors (Geom32), the closed
// forms rewritten without the cancellation te/ue - tb/ub (which loses all FP32
// digits when the target point lies near the source axis):
// te/ue - tb/ub = 2b d / ((te ub + tb ue) ue ub) when te and tb share a sign.
// FAR = true: the caller guarantees c >= 6 (far pairs of the split assembly).
template <int N, bool FAR = false>
__device__ __forceinline__ void moments_fp32(const Geom32 &g, float *I, float *J, float *S) {
    const float b = g.b, c = g.c;
    if (FAR || c >= 6.0f) {
        moments_backward_fp32<N>(b, c, I, J, S);
        return;
    }
    constexpr int K = N + 3;
    const float ue = sqrtf(g.ue2);
    const float ub = sqrtf(g.ub2);
    const float te = 1.0f + 0.5f * b;
    const float tb = -1.0f + 0.5f * b;
    const float d = g.d;
    const float iue = __frcp_rn(ue), iub = __frcp_rn(ub), id = __frcp_rn(d);
    // log((2te + 2ue)/(2tb + 2ub)) with the smaller operand formed stably
    const float ae = (te >= 0.f) ? (te + ue) : d * __frcp_rn(ue - te);
    const float ab = (tb >= 0.f) ? (tb + ub) : d * __frcp_rn(ub - tb);
    I[0] = logf(ae * __frcp_rn(ab));
    I[1] = ue - ub - 0.5f * b * I[0];
    if (d < 1e-6f * c && te * tb > 0.f) {
        // point on the source axis beyond its ends: the d -> 0 limits
        // (Int_analytical.f90:162-164, 189-191).  Within the span (te tb < 0:
        // fibers that touch or cross) the general forms below hold with the
        // accurate d and have no cancellation.
        J[0] = 0.5f * (__frcp_rn(tb * tb) - __frcp_rn(te * te));
        J[1] = -iue + iub - 0.5f * b * J[0];
        const float p = 2.0f + b, m = -2.0f + b;
        const float ip = __frcp_rn(p), im = __frcp_rn(m);
        const float ip2 = ip * ip, im2 = im * im;
        S[0] = 4.0f * (im2 * im2 - ip2 * ip2);
        S[1] = (8.0f / 3.0f) * (im2 * im - ip2 * ip) - 0.5f * b * S[0];
    } else {
        // (te/ue - tb/ub)/d; with te, tb of one sign te/ue - tb/ub = 2b d / ((te ub + tb ue) ue ub)
        if (te * tb > 0.f) J[0] = 2.0f * b * __frcp_rn((te * ub + tb * ue) * ue * ub);
        else J[0] = (te * iue - tb * iub) * id;
        J[1] = -iue + iub - 0.5f * b * J[0];
        const float iue3 = iue * iue * iue, iub3 = iub * iub * iub;
        S[0] = ((2.0f + b) * iue3 - (-2.0f + b) * iub3) * (id * (1.0f / 6.0f)) + (2.0f / 3.0f) * id * J[0];
        S[1] = (-(b + 2.0f * c) * iue3 + (-b + 2.0f * c) * iub3) * (id * (1.0f / 6.0f)) -
               b * (1.0f / 3.0f) * id * J[0];
    }
#pragma unroll
    for (int n = 2; n < K; ++n) {
        const float nn = n + 1.0f;
        const float r = 1.0f / (1.0f - nn);
        const float sbp = (n % 2 == 1) ? 1.0f : -1.0f;
        I[n] = -ue * r + sbp * ub * r - (0.5f - (nn - 1.0f)) * b * r * I[n - 1] + (nn - 2.0f) * c * r * I[n - 2];
        J[n] = I[n - 2] - b * J[n - 1] - c * J[n - 2];
        S[n] = J[n - 2] - b * S[n - 1] - c * S[n - 2];
    }
}

// Outer products of R0 and the source direction pb shared by every Legendre
// weight, packed 11,22,33,12,13,23.
template <typename T>
struct Outer {
    T rr[6], pr[6], pp[6];
    __device__ __forceinline__ Outer(T r0x, T r0y, T r0z, T px, T py, T pz) {
        rr[0] = r0x * r0x; rr[1] = r0y * r0y; rr[2] = r0z * r0z;
        rr[3] = r0x * r0y; rr[4] = r0x * r0z; rr[5] = r0y * r0z;
        pr[0] = (T)2 * px * r0x; pr[1] = (T)2 * py * r0y; pr[2] = (T)2 * pz * r0z;
        pr[3] = px * r0y + r0x * py; pr[4] = px * r0z + r0x * pz; pr[5] = py * r0z + r0y * pz;
        pp[0] = px * px; pp[1] = py * py; pp[2] = pz * pz;
        pp[3] = px * py; pp[4] = px * pz; pp[5] = py * pz;
    }
};

// Legendre-weighted moments for weight m and the tensor G_m (6 packed
// components 11,22,33,12,13,23), Int_analytical.f90:213-288 and 735-746:
// G = L11 I + L12 R0R0 - L13 (pb R0 + R0 pb) + L14 pb pb
//   + 2 eps^2 (L12 I - 3 L22 R0R0 + 3 L23 (pb R0 + R0 pb) - 3 L24 pb pb)
// Each L is scale_m * (sum of integer-weighted moments), highest power first.
template <typename T, int m>
__device__ __forceinline__ void g_coeffs(const T *I, const T *J, const T *S, T eps2, T &cI, T &cRR, T &cPR,
                                         T &cPP) {
    T l11 = 0, l12 = 0, l13 = 0, l14 = 0, l22 = 0, l23 = 0, l24 = 0;
#pragma unroll
    for (int p = m; p >= 0; --p) {
        if (leg_coef(m, p) != 0) {
            const T a = (T)leg_coef(m, p);
            l11 += a * I[p];
            l12 += a * J[p];
            l13 += a * J[p + 1];
            l14 += a * J[p + 2];
            l22 += a * S[p];
            l23 += a * S[p + 1];
            l24 += a * S[p + 2];
        }
    }
    const T sc = (T)leg_scale(m);
    l11 *= sc; l12 *= sc; l13 *= sc; l14 *= sc; l22 *= sc; l23 *= sc; l24 *= sc;
    const T e2 = (T)2 * eps2;
    cI = l11 + e2 * l12;                // identity
    cRR = l12 - (T)3 * e2 * l22;        // R0 R0
    cPR = -l13 + (T)3 * e2 * l23;       // pb R0 + R0 pb
    cPP = l14 - (T)3 * e2 * l24;        // pb pb
}

template <typename T, int m>
__device__ __forceinline__ void g_tensor(const T *I, const T *J, const T *S, const Outer<T> &o, T eps2, T *G) {
    T cI, cRR, cPR, cPP;
    g_coeffs<T, m>(I, J, S, eps2, cI, cRR, cPR, cPP);
#pragma unroll
    for (int c = 0; c < 6; ++c) G[c] = cRR * o.rr[c] + cPR * o.pr[c] + cPP * o.pp[c] + (c < 3 ? cI : (T)0);
}

// Store G_m for m = 0..N straight to shared memory as it is formed:
// dst[(m*6 + c) * ld], converting to double.
template <typename T, int N, int m = 0>
struct GStore {
    __device__ __forceinline__ static void run(const T *I, const T *J, const T *S, const Outer<T> &o, T eps2,
                                               double *dst, int ld) {
        T G[6];
        g_tensor<T, m>(I, J, S, o, eps2, G);
#pragma unroll
        for (int c = 0; c < 6; ++c) dst[(m * 6 + c) * ld] = (double)G[c];
        GStore<T, N, m + 1>::run(I, J, S, o, eps2, dst, ld);
    }
};
template <typename T, int N>
struct GStore<T, N, N + 1> {
    __device__ __forceinline__ static void run(const T *, const T *, const T *, const Outer<T> &, T, double *, int) {}
};

// The analytic inner integral for all weights, stored to shared memory.
template <int N>
__device__ __forceinline__ void inner_analytic_store_fp64(double r0x, double r0y, double r0z, double px, double py,
                                                          double pz, double eps2, double *dst, int ld) {
    double I[N + 3], J[N + 3], S[N + 3];
    const double b = fmul(-2.0, fadd(fadd(fmul(px, r0x), fmul(py, r0y)), fmul(pz, r0z)));
    const double c = fadd(fadd(fmul(r0x, r0x), fmul(r0y, r0y)), fmul(r0z, r0z));
    moments_fp64<N>(b, c, I, J, S);
    const Outer<double> o(r0x, r0y, r0z, px, py, pz);
    GStore<double, N>::run(I, J, S, o, eps2, dst, ld);
}

template <int N>
__device__ __forceinline__ void inner_analytic_store_fp32(float r0x, float r0y, float r0z, float px, float py,
                                                          float pz, float eps2, double *dst, int ld) {
    float I[N + 3], J[N + 3], S[N + 3];
    moments_fp32<N>(Geom32(r0x, r0y, r0z, px, py, pz), I, J, S);
    const Outer<float> o(r0x, r0y, r0z, px, py, pz);
    GStore<float, N>::run(I, J, S, o, eps2, dst, ld);
}

// Numeric inner integral (quadrature.f90:100-164): 3-point Gauss on each
// panel of the source fiber, kernel
// K = I/R + RR/R^3 + 2 eps^2 (I/R^3 - 3 RR/R^5), weighted by P_m.  The FP64
// instance takes every power of R from one reciprocal square root and fuses:
// the reference's formulas spell out seventeen divisions and a square root per
// point pair, which were nine tenths of the numeric assembly (M = 300: 1.47 ->
// 0.44 ms).  Against extended precision the blocks of pairs 0.3 to 0.01 apart
// are off by at most 5e-15 .. 1.2e-14 of their largest entry either way.
template <int N>
__device__ __forceinline__ void inner_numeric_fp64(double xbx, double xby, double xbz, const double *xs,
                                                   const double *ts, const double *pv, const double *wP,
                                                   int LQ, double eps2, double (*G)[6]) {
#pragma unroll
    for (int m = 0; m <= N; ++m)
#pragma unroll
        for (int c = 0; c < 6; ++c) G[m][c] = 0.0;
    const double e2 = 2.0 * eps2, e6 = 6.0 * eps2;
#pragma unroll 1
    for (int s = 0; s < LQ; ++s) {
        const double sp = pv[s];
        const double Rx = xbx - fma(ts[0], sp, xs[0]);
        const double Ry = xby - fma(ts[1], sp, xs[1]);
        const double Rz = xbz - fma(ts[2], sp, xs[2]);
        const double ir = rsqrt_pos(fma(Rx, Rx, fma(Ry, Ry, Rz * Rz)));
        const double ir2 = ir * ir, ir3 = ir2 * ir;
        const double diag = fma(e2, ir3, ir), off = ir3 * fma(-e6, ir2, 1.0);
        const double ox = off * Rx, oy = off * Ry, oz = off * Rz;
        const double K[6] = {fma(ox, Rx, diag), fma(oy, Ry, diag), fma(oz, Rz, diag), ox * Ry, ox * Rz, oy * Rz};
#pragma unroll
        for (int m = 0; m <= N; ++m) {
            const double w = wP[m * kMaxLQ + s];
#pragma unroll
            for (int c = 0; c < 6; ++c) G[m][c] = fma(w, K[c], G[m][c]);
        }
    }
}

template <int N>
__device__ __forceinline__ void inner_numeric_fp32(float xbx, float xby, float xbz, const float *xs,
                                                   const float *ts, const float *pv, const float *wP, int LQ,
                                                   float eps2, float (*G)[6]) {
#pragma unroll
    for (int m = 0; m <= N; ++m)
#pragma unroll
        for (int c = 0; c < 6; ++c) G[m][c] = 0.0f;
    for (int s = 0; s < LQ; ++s) {
        const float sp = pv[s];
        const float Rx = xbx - (xs[0] + ts[0] * sp);
        const float Ry = xby - (xs[1] + ts[1] * sp);
        const float Rz = xbz - (xs[2] + ts[2] * sp);
        const float R2 = Rx * Rx + Ry * Ry + Rz * Rz;
        const float ir = rsqrtf(R2);
        const float ir3 = ir * ir * ir;
        const float ir5 = ir3 * ir * ir;
        const float e2 = 2.0f * eps2;
        const float diag = ir + e2 * ir3;
        const float off = ir3 - 3.0f * e2 * ir5;
        float K[6];
        K[0] = diag + Rx * Rx * off;
        K[1] = diag + Ry * Ry * off;
        K[2] = diag + Rz * Rz * off;
        K[3] = Rx * Ry * off;
        K[4] = Rx * Rz * off;
        K[5] = Ry * Rz * off;
#pragma unroll
        for (int m = 0; m <= N; ++m) {
            const float w = wP[m * kMaxLQ + s];
#pragma unroll
            for (int c = 0; c < 6; ++c) G[m][c] += w * K[c];
        }
    }
}

// D = A B + C for one 8x8x4 FP64 tile (warp-wide; every lane of the warp
// takes part).  Lane l holds A[l/4][l%4], B[l%4][l/4], C/D[l/4][2(l%4)+{0,1}].
__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b, double c0, double c1) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%5};\n"
                 : "=d"(d0), "=d"(d1)
                 : "d"(a), "d"(b), "d"(c0), "d"(c1));
}

__device__ __forceinline__ int sym_index(int a, int b) {
    // packed index of the symmetric 3x3 component (a,b)
    return a == b ? a : (a + b == 1 ? 3 : (a + b == 2 ? 4 : 5));
}

}  // namespace rf
