// gk_physics.cuh -- pointwise device physics of the finite-volume update.
//
// Included inside the mode namespace (gk_parity / gk_fast).  Every
// expression keeps the reference's association order.  The parity unit is
// compiled with -fmad=false and uses correctly rounded division and square
// root (div_rn, sqrt_rn below where their operands are in range, else CUDA's
// IEEE operations), as on the host: results are bit-identical
// to the reference built without -ffast-math.  The fast unit (GK_FASTMATH) lets the
// compiler contract to FMA and replaces division, reciprocal and square root
// by the branch-free refinements below.
#pragma once

// libstdc++ std::max / std::min: max(a,b) = (a<b)?b:a, min(a,b) = (b<a)?b:a.
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }

#if GK_FASTMATH
// Reciprocal, quotient and square root for finite, positive, normal
// arguments (densities, pressures, sound speeds, wave-speed differences).
// Each starts from the hardware approximation (PTX rcp.approx.ftz.f64 /
// rsqrt.approx.ftz.f64, about 2^-22 relative error) and applies one
// third-order step of the binomial series, which cubes the relative error:
//   reciprocal  e = 1 - b*y,    y' = y*(1 + e + e^2)
//   rsqrt       d = 1 - x*y^2,  y' = y*(1 + d/2 + 3d^2/8)
// (the series of (1 - e)^-1 and (1 - d)^-1/2 to second order; one step does
// the work of two Newton steps in fewer operations).  The square root is
// x*rsqrt(x) with one Newton correction of the residual x - s*s (Markstein,
// IBM J. Res. Dev. 34(1), 1990).  The result is within a few ulp of the IEEE
// value; there is no slow path and no branch.
__device__ __forceinline__ double rcp_nr(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsqrt_nr(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double d = fma(-x * y, y, 1.0);
    return fma(y, d * fma(0.375, d, 0.5), y);
}
__device__ __forceinline__ double sqrt_nr(double x) {
    const double y = rsqrt_nr(x);
    const double s = x * y;
    const double r = fma(-s, s, x);
    return fma(r, 0.5 * y, s);
}
__device__ __forceinline__ double rcp_ranged(double b, bool& bad) {
    bad = false;
    return rcp_nr(b);
}
// The step taken on the product instead of its factor: the same operations in a
// chain one shorter (a/b, and g/sqrt(x) with x/sqrt(x) where both are used).  KH
// 4096^2 944 -> 930 us per step, 2001x1503 199.2 -> 197.1, RT 1024x3072 326.8 -> 324.6.
// Dividing for c beside s* (from the numerator and denominator) shortens the chain
// again but needs registers: KH 1024^2 71.6 -> 72.5, 4096^2 930 -> 950.
__device__ __forceinline__ double div_nr(double a, double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0), q = a * y;
    return fma(q, fma(e, e, e), q);
}
__device__ __forceinline__ void rsqrt_products(double g, double x, double& gr, double& xr) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double q = x * y, d = fma(-q, y, 1.0), h = g * y;
    const double t = d * fma(0.375, d, 0.5);
    gr = fma(h, t, h);
    xr = fma(q, t, q);
}
#define GK_DIV(a, b) div_nr((a), (b))
#define GK_RCP(b) rcp_nr(b)
#define GK_SQRT(x) sqrt_nr(x)

// Fast mode's sign and order decisions on the integer pipes, from the bit
// patterns: the FP64 pipe bounds the stage kernel, and a compare there costs
// as much as an add.  They differ from the IEEE compares only on -0 and on
// NaNs (fast mode's contract is a tolerance; a non-finite state is still
// caught by the CFL reduction).
__device__ __forceinline__ double pos_part(double x) {  // max(x, 0)
    return __double2hiint(x) < 0 ? 0.0 : x;
}
__device__ __forceinline__ double neg_part(double x) {  // min(0, x)
    return __double2hiint(x) < 0 ? x : 0.0;
}
__device__ __forceinline__ bool ge0(double x) { return __double2hiint(x) >= 0; }        // x >= 0
__device__ __forceinline__ bool le0(double x) { return __double_as_longlong(x) <= 0; }  // x <= 0
// max(x, f) for a positive floor f (signed 64-bit order of the patterns is
// the order of the values when f > 0)
__device__ __forceinline__ double floor_at(double x, double f) {
    return __double_as_longlong(x) < __double_as_longlong(f) ? f : x;
}
#define GK_MAX0(x) pos_part(x)
#define GK_MIN0(x) neg_part(x)
#define GK_GE0(x) ge0(x)
#define GK_LE0(x) le0(x)
#define GK_FLOOR(x, f) floor_at((x), (f))
#define GK_BELOW(x, f) (__double_as_longlong(x) < __double_as_longlong(f))
// max of two non-negative values (speeds): their bit patterns order alike
#define GK_MAXNN(a, b) (__double_as_longlong(a) < __double_as_longlong(b) ? (b) : (a))
#else
// Parity mode: IEEE division and square root (correctly rounded on the GPU
// as on the host), for operands of any size.
#define GK_DIV(a, b) ((a) / (b))
#define GK_RCP(b) rcp_any(b)
#define GK_SQRT(x) sqrt_any(x)
// the reference's compares and std::max/min
#define GK_FLOOR(x, f) smax((x), (f))
#define GK_BELOW(x, f) ((x) < (f))
#define GK_MAXNN(a, b) smax((a), (b))

// Correctly rounded quotient, reciprocal and square root without a branch,
// for operands in range (hi words checked by the callers through the `bad`
// flags below).  CUDA's IEEE operations test their operands and branch to a
// slow path each; with about 30 of them per row those branches cut the fused
// stage's code into pieces between which no two Riemann problems can
// interleave (branch_resolving and wait stalls, the FP64 pipe 52 % busy).
// Here the checks are integer tests folded into one flag per phase, and the
// whole phase is redone with the IEEE operations where it is set.
//
// Division (Markstein, IBM J. Res. Dev. 34(1), 1990; Muller et al., Handbook
// of Floating-Point Arithmetic, ch. 4): with y the correctly rounded 1/b and q
// a faithful quotient, r = a - b q is exact and fma(r, y, q) is the correctly
// rounded a/b.  The seed's relative error is below 2^-19.9 (measured over
// every upper word), so y1 is within 0.51 ulp; one Newton step from it rounds
// 1/b correctly unless b's significand is all ones (the only 53-bit divisor B
// of 2^106 - 1 = B M, where 1/b lies 2^-106 above a midpoint), which rounds
// up (ones_up).  q comes from the seed's quotient corrected with y1 (error
// 0.5 + 2^-20 ulp).  Square root: Goldschmidt's iteration to within an ulp,
// then the exact residual; before its last rounding it is within 2^-51 ulp of
// the root, and of the arguments whose roots lie that near a midpoint every
// one rounds correctly (tests/test_gpu_parity_math.py runs them all).
// Against CUDA's operations: 1.7e10 random pairs and 1.1e10 quotients next to
// midpoints without a difference.
__device__ __forceinline__ double rcp_seed(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
}
__device__ __forceinline__ double ones_up(double y, double b) {
    const bool ones = ((__double2hiint(b) | (int)0xfff00000) & __double2loint(b)) == -1;
    return __hiloint2double(__double2hiint(y), __double2loint(y) | (ones ? 1 : 0));
}
// div_rn_plain: for a significand of b that is not all ones.
template <bool ONES>
__device__ __forceinline__ double div_rn_t(double a, double b) {
    const double y0 = rcp_seed(b);
    const double e = fma(-b, y0, 1.0);
    const double y1 = fma(y0, fma(e, e, e), y0);
    const double q0 = a * y0;
    const double q1 = fma(fma(-b, q0, a), y1, q0);
    double y = fma(y1, fma(-b, y1, 1.0), y1);
    if (ONES) y = ones_up(y, b);
    return fma(fma(-b, q1, a), y, q1);
}
__device__ __forceinline__ double div_rn(double a, double b) { return div_rn_t<true>(a, b); }
__device__ __forceinline__ double div_rn_plain(double a, double b) { return div_rn_t<false>(a, b); }
__device__ __forceinline__ double rcp_rn(double b) {
    const double y0 = rcp_seed(b);
    const double e = fma(-b, y0, 1.0);
    const double y1 = fma(y0, fma(e, e, e), y0);
    return ones_up(fma(y1, fma(-b, y1, 1.0), y1), b);
}
__device__ __forceinline__ double sqrt_rn(double x) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
    const double g0 = x * y0, h0 = 0.5 * y0;
    const double e = fma(-g0, h0, 0.5);
    const double t = fma(1.5 * e, e, e);  // (1 - 2e)^-1/2 = 1 + e + 3/2 e^2 + ...
    const double g = fma(g0, t, g0), h = fma(h0, t, h0);
    return fma(fma(-g, g, x), h, g);
}

// Range tests.  The upper words of doubles, read as floats, keep the order of
// the values, and a double that is not finite (or above 2^1016) reads as a
// float infinity or NaN; so the tests of a phase run as NaN-propagating float
// minima and maxima, whose absolute values and signs cost nothing, and one
// compare at the end.
__device__ __forceinline__ int hi(double x) { return __double2hiint(x); }
__device__ __forceinline__ float top(double x) { return __int_as_float(__double2hiint(x)); }
__device__ __forceinline__ float pow2_top(int k) { return __int_as_float((1023 + k) << 20); }
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ bool is_zero(double x) {
    return ((hi(x) & 0x7fffffff) | __double2loint(x)) == 0;
}
// 0 < |x| < 2^-400: too small for the exact residuals
__device__ __forceinline__ bool tiny(double x) {
    return fabsf(top(x)) < pow2_top(-400) && !is_zero(x);
}
// 2^lo <= x < 2^up
__device__ __forceinline__ bool in_pos(double x, int lo, int up) {
    return top(x) >= pow2_top(lo) && top(x) < pow2_top(up);
}
// all ones in x's significand: 0xffffffff, else less
__device__ __forceinline__ unsigned ones_of(double x) {
    return (unsigned)((hi(x) | (int)0xfff00000) & __double2loint(x));
}
// Densities and pressures in [2^-60, 2^100) and speeds below 2^100 keep every
// product, quotient and residual of the Riemann problem (hllc_ranged) normal
// and finite; the floors (2^-53) are inside.
constexpr int kLo = -60, kUp = 100;

// 1/x in range, with the range test left to the caller's flag.
__device__ __forceinline__ double rcp_ranged(double x, bool& bad) {
    bad = !in_pos(x, kLo, kUp);
    return rcp_rn(x);
}
// 1/x, and sqrt(x), each with its own range test.
__device__ __forceinline__ double rcp_any(double x) {
    if (in_pos(x, kLo, kUp)) return rcp_rn(x);
    return 1.0 / x;
}
__device__ __forceinline__ double sqrt_any(double x) {
    if (in_pos(x, -500, 500)) return sqrt_rn(x);
    return sqrt(x);
}
#endif

// Half the van Leer slope: what the PLM face states u +- 0.5*sigma add.  Fast
// mode: (a*b)/(a+b) for ab > 0 else 0, without the two scalings by 2 and 1/2.
// Parity mode: the same quotient, which is exactly 0.5*((2ab)/(a+b)) unless a
// scaling underflows; the record tells where it might not be the reference's
// value (a product below 2^-400, a sum above 2^400 or with all ones).
#if GK_FASTMATH
struct SlopeRange {};
__device__ __forceinline__ void clear(SlopeRange&) {}
__device__ __forceinline__ double vanleer_half(double a, double b, SlopeRange&) {
    const double multi = a * b;
    const double h = GK_DIV(multi, a + b);
    return GK_LE0(multi) ? 0.0 : h;
}
__device__ __forceinline__ double vanleer_half_any(double a, double b) {
    SlopeRange none;
    return vanleer_half(a, b, none);
}
#else
// Range record of a phase's slopes: the smallest product and the largest sum
// (as floats), and whether a sum's significand is all ones.
struct SlopeRange {
    float lo, up;
    unsigned ones;
};
__device__ __forceinline__ void clear(SlopeRange& r) {
    r.lo = pow2_top(0);
    r.up = 0.f;
    r.ones = 0u;
}
__device__ __forceinline__ bool out_of_range(const SlopeRange& r) {
    return !(r.lo >= pow2_top(-400) && r.up < pow2_top(400)) || r.ones == 0xffffffffu;
}
__device__ __forceinline__ double vanleer_half(double a, double b, SlopeRange& r) {
    const double multi = a * b, sum = a + b;
    const bool none = multi <= 0.0;
    r.lo = min_nan(r.lo, none ? pow2_top(0) : top(multi));
    r.up = max_nan(r.up, fabsf(top(sum)));
    r.ones = max(r.ones, ones_of(sum));
    const double h = div_rn_plain(multi, sum);
    return none ? 0.0 : h;
}
// Half of Reconstruction::VanLeer (reconstruction.hpp:36-42).
__device__ __noinline__ double vanleer_half_any(double a, double b) {
    const double multi = a * b;
    return 0.5 * ((multi <= 0.0) ? 0.0 : GK_DIV(2.0 * multi, a + b));
}
#endif

struct Flux5 {
    double d, n, t1, t2, e;  // density, normal momentum, tangential 1/2, energy
};

// Flux::RiemannSolver for one face (hllc.cpp:22-101), HLLC after Toro
// ch. 10 with the PVRS pressure estimate.  Velocities come as (normal,
// tangential 1, tangential 2) in the reference's rotation
// (IVLX, IVLY, IVLZ = hllc.cpp:25-27).  T2 = false drops the second
// tangential component, which callers use only when it is exactly zero (2D
// runs with vz = 0): every term it contributes is then an exact zero.
//
// The reference combines its star sides as f = selectl*fl + selectr*fr with
// selectl = (ss >= 0) ? 1 : 0 (hllc.cpp:75-94), and so does parity mode here; fast
// mode evaluates the selected side only, which differs where the unused side is
// not finite, or in the sign of a zero.
#if GK_FASTMATH
template <bool T2>
__device__ __forceinline__ void hllc_any(double denl, double vxl, double vyl, double vzl, double prel,
                                         double denr, double vxr, double vyr, double vzr, double prer,
                                         const gk::Phys& ph, Flux5& f) {
    const double gamma = ph.gamma;
    // sqrt(gamma*p/rho) = (gamma*p) * rsqrt(gamma*p*rho): one root, no quotient
    const double gpl = gamma * prel, gpr = gamma * prer;
    double al, ar, unused;
    rsqrt_products(gpl, gpl * denl, al, unused);
    rsqrt_products(gpr, gpr * denr, ar, unused);
    // 2p* of the PVRS estimate; max(p*, 0) is not taken, as only max(p* - p, 0)
    // of positive pressures p is used
    const double pvrs2 = fma(-0.25 * ((vxr - vxl) * (denl + denr)), al + ar, prel + prer);
    // a*q = sqrt(gamma p/rho) * sqrt(1 + cq max(p*/p - 1, 0)) = sqrt(gamma X/rho)
    // with X = p + cq max(p* - p, 0): one root per side, no quotient.
    // Branch-free on purpose: a skip when p* <= p (as in parity mode) was
    // measured slower, because it splits the straight-line code in which the
    // x- and y-face solves of a row interleave.
    const double gxl = fma(ph.hgcq, GK_MAX0(fma(-2.0, prel, pvrs2)), gpl);
    const double gxr = fma(ph.hgcq, GK_MAX0(fma(-2.0, prer, pvrs2)), gpr);
    // S - v = -+ gX rsqrt(gX rho), and rho (S - v) = -+ (gX rho) rsqrt(gX rho)
    double dvl, dvr, ml, mr;
    rsqrt_products(gxl, gxl * denl, dvl, ml);
    rsqrt_products(gxr, gxr * denr, dvr, mr);
    ml = -ml;
    double sl = vxl - dvl;
    double sr = vxr + dvr;
    // the contact speed's numerator and (negative) denominator, with rho (S - v)
    // of each side formed once
    const double num = prer - prel + ml * vxl - mr * vxr, den = ml - mr;
    double ss = GK_DIV(num, den);
    // The selected side: its kinetic energy from the selected velocities, and
    // E + p as p/(gamma-1) + p + rho k/2 in one product with gamma/(gamma-1).
    // m = rho (S - v) of the side, formed for the contact speed, carries the
    // star-state terms:
    //   rho (vn^2 + c S) = f1 vn + c m,   rho c ss (S - vn) = c ss m.
    const bool left = GK_LE0(num);
    double d = left ? denl : denr, vn = left ? vxl : vxr, v1 = left ? vyl : vyr;
    double v2 = left ? vzl : vzr, p = left ? prel : prer, s = left ? sl : sr;
    const double m = left ? ml : mr;
    double k = T2 ? (vn * vn + v1 * v1 + v2 * v2) : (vn * vn + v1 * v1);
    double ep = p * ph.gm1Rec1 + 0.5 * d * k;  // E + p
    double sc = left ? GK_MIN0(s) : GK_MAX0(s);
    double c = GK_DIV(sc * (ss - vn), s - ss);
    double vc = vn + c;
    double f1 = d * vc;
    f.d = f1;
    f.n = f1 * vn + (c * m + p);
    f.t1 = f1 * v1;
    f.t2 = T2 ? f1 * v2 : 0.0;
    f.e = ep * vc + c * ss * m;
}
#else
template <bool T2>
__device__ __forceinline__ void hllc_any(double denl, double vxl, double vyl, double vzl, double prel,
                                         double denr, double vxr, double vyr, double vzr, double prer,
                                         const gk::Phys& ph, Flux5& f) {
    const double gamma = ph.gamma;
    // EquationOfState::SoundSpeed (eos.hpp:27-29)
    double al = sqrt(GK_DIV(gamma * prel, denl));
    double ar = sqrt(GK_DIV(gamma * prer, denr));
    double prePVRS = 0.5 * (prel + prer) - 0.125 * (vxr - vxl) * (denl + denr) * (al + ar);
    prePVRS = smax(prePVRS, 0.0);
    double ql, qr;
    // q = sqrt(1 + 0.5*(1+1/gamma)*max(p*/p - 1, 0)) is exactly 1 whenever
    // p* <= p with p > 0, so the division and root are skipped there.
    ql = 1.0;
    qr = 1.0;
    if (!(prePVRS <= prel && prel > 0.0)) {
        double temp = smax(GK_DIV(prePVRS, prel) - 1, 0.0);
        ql = sqrt(1 + ph.cq * temp);
    }
    if (!(prePVRS <= prer && prer > 0.0)) {
        double temp = smax(GK_DIV(prePVRS, prer) - 1, 0.0);
        qr = sqrt(1 + ph.cq * temp);
    }
    double sl = vxl - al * ql;
    double sr = vxr + ar * qr;
    double ss = GK_DIV(prer - prel + denl * vxl * (sl - vxl) - denr * vxr * (sr - vxr),
                       denl * (sl - vxl) - denr * (sr - vxr));
    // EquationOfState::EGas (eos.hpp:30-32) + kinetic energy
    double kl = T2 ? (vxl * vxl + vyl * vyl + vzl * vzl) : (vxl * vxl + vyl * vyl);
    double kr = T2 ? (vxr * vxr + vyr * vyr + vzr * vzr) : (vxr * vxr + vyr * vyr);
    double el = prel * ph.gm1Rec + 0.5 * denl * kl;
    double er = prer * ph.gm1Rec + 0.5 * denr * kr;
    double cl = GK_DIV(smin(0.0, sl) * (ss - vxl), sl - ss);
    double cr = GK_DIV(smax(0.0, sr) * (ss - vxr), sr - ss);
    double selectl = (ss >= 0) ? 1.0 : 0.0;
    double selectr = 1.0 - selectl;
    double fl1 = denl * (vxl + cl);
    double fl2 = denl * (vxl * vxl + cl * sl) + prel;
    double fl3 = fl1 * vyl;
    double fl5 = (el + prel) * (vxl + cl) + denl * cl * ss * (sl - vxl);
    double fr1 = denr * (vxr + cr);
    double fr2 = denr * (vxr * vxr + cr * sr) + prer;
    double fr3 = fr1 * vyr;
    double fr5 = (er + prer) * (vxr + cr) + denr * cr * ss * (sr - vxr);
    f.d = selectl * fl1 + selectr * fr1;
    f.n = selectl * fl2 + selectr * fr2;
    f.t1 = selectl * fl3 + selectr * fr3;
    if (T2) {
        double fl4 = fl1 * vzl;
        double fr4 = fr1 * vzr;
        f.t2 = selectl * fl4 + selectr * fr4;
    } else {
        f.t2 = 0.0;
    }
    f.e = selectl * fl5 + selectr * fr5;
}
#endif

#if GK_FASTMATH
// Fast mode has one form: no lane is ever out of its range.
struct HllcAux {};
template <bool T2>
__device__ __forceinline__ void hllc_ranged(double denl, double vxl, double vyl, double vzl,
                                            double prel, double denr, double vxr, double vyr,
                                            double vzr, double prer, const gk::Phys& ph, Flux5& f,
                                            bool&, HllcAux&) {
    hllc_any<T2>(denl, vxl, vyl, vzl, prel, denr, vxr, vyr, vzr, prer, ph, f);
}
template <bool T2>
__device__ __forceinline__ void hllc_redo(double, double, double, double, double, double, double,
                                          double, double, double, const gk::Phys&, Flux5&, bool,
                                          const HllcAux&) {}
#else
// The Riemann problem for states in range, straight-line, and only its
// selected side: with both sides finite the reference's
// selectl*fl + selectr*fr is the selected side's flux, except that a -0 of it
// becomes +0 where the other side's component is positive.  `bad` is set
// where an operand is out of range (the flux must come from hllc_any); aux
// keeps what hllc_redo needs to give a -0 the reference's sign.
struct HllcAux {
    double ss, so;  // contact speed, the other side's wave speed
    bool zero;      // a component of the selected side is -0
};
template <bool T2>
__device__ __forceinline__ void hllc_ranged(double denl, double vxl, double vyl, double vzl,
                                            double prel, double denr, double vxr, double vyr,
                                            double vzr, double prer, const gk::Phys& ph, Flux5& f,
                                            bool& bad, HllcAux& aux) {
    const double gamma = ph.gamma;
    // range record: lo of what must be at least 2^-60, up of what must stay
    // below 2^100 in size
    float lo = min3(top(denl), top(prel), min_nan(top(denr), top(prer)));
    float up = max3(top(denl), top(prel), max_nan(top(denr), top(prer)));
    up = max3(up, fabsf(top(vxl)), fabsf(top(vxr)));
    up = max3(up, fabsf(top(vyl)), fabsf(top(vyr)));
    if (T2) up = max3(up, fabsf(top(vzl)), fabsf(top(vzr)));
    const double al = sqrt_rn(div_rn(gamma * prel, denl));
    const double ar = sqrt_rn(div_rn(gamma * prer, denr));
    double prePVRS = 0.5 * (prel + prer) - 0.125 * (vxr - vxl) * (denl + denr) * (al + ar);
    prePVRS = hi(prePVRS) < 0 ? 0.0 : prePVRS;  // zero, or at least 2^-114 by its terms
    // q = sqrt(1 + cq max(p*/p - 1, 0))
    double tl = div_rn(prePVRS, prel) - 1, tr = div_rn(prePVRS, prer) - 1;
    tl = hi(tl) < 0 ? 0.0 : tl;
    tr = hi(tr) < 0 ? 0.0 : tr;
    const double ql = sqrt_rn(1 + ph.cq * tl), qr = sqrt_rn(1 + ph.cq * tr);
    const double sl = vxl - al * ql, sr = vxr + ar * qr;
    const double dl = sl - vxl, dr = sr - vxr;
    const double num = prer - prel + denl * vxl * dl - denr * vxr * dr;
    const double den = denl * dl - denr * dr;  // negative
    const double ss = div_rn_plain(num, den);
    const double bl = sl - ss, br = sr - ss;  // negative, positive
    lo = min3(lo, -top(den), min_nan(-top(bl), top(br)));
    const bool left = top(ss) >= 0.f;  // ss >= 0, -0 included (ss is 0 or at least 2^-600)
    const double d = left ? denl : denr, vn = left ? vxl : vxr, v1 = left ? vyl : vyr;
    const double v2 = T2 ? (left ? vzl : vzr) : 0.0, p = left ? prel : prer, s = left ? sl : sr;
    const double sv = left ? dl : dr;
    // a/b with b = S - S* made negative (a/b = (-a)/(-b)): a zero quotient of
    // div_rn has the IEEE sign for b < 0 only
    const double sc = left ? (hi(s) < 0 ? s : 0.0) : (hi(s) < 0 ? 0.0 : s);
    const double a = sc * (ss - vn);
    const double b = left ? bl : -br;
    up = max3(up, top(prePVRS), max3(fabsf(top(num)), fabsf(top(ss)), fabsf(top(a))));
    bad |= !(lo >= pow2_top(kLo) && up < pow2_top(kUp)) || tiny(num) || tiny(a) ||
           max(ones_of(den), ones_of(b)) == 0xffffffffu;
    const double c = div_rn_plain(left ? a : -a, b);
    const double k = T2 ? (vn * vn + v1 * v1 + v2 * v2) : (vn * vn + v1 * v1);
    const double e = p * ph.gm1Rec + 0.5 * d * k;
    const double vc = vn + c;
    const double f1 = d * vc;
    f.d = f1;
    f.n = d * (vn * vn + c * s) + p;
    f.t1 = f1 * v1;
    f.t2 = T2 ? f1 * v2 : 0.0;
    f.e = (e + p) * vc + d * c * ss * sv;
    constexpr int kNeg = (int)0x80000000;
    aux.zero = hi(f.d) == kNeg || hi(f.t1) == kNeg || (T2 && hi(f.t2) == kNeg) || hi(f.e) == kNeg;
    aux.ss = ss;
    aux.so = left ? sr : sl;
}

// hllc_any kept out of line: it runs for few lanes, and inlined it would
// stretch the row loop over more instruction lines.
struct HllcStates {
    double denl, vxl, vyl, vzl, prel, denr, vxr, vyr, vzr, prer;
};
template <bool T2>
__device__ __noinline__ Flux5 hllc_far(HllcStates w, double gamma, double gm1Rec, double cq) {
    gk::Phys ph;
    ph.gamma = gamma;
    ph.gm1Rec = gm1Rec;
    ph.cq = cq;
    Flux5 f;
    hllc_any<T2>(w.denl, w.vxl, w.vyl, w.vzl, w.prel, w.denr, w.vxr, w.vyr, w.vzr, w.prer, ph, f);
    return f;
}

// Completes hllc_ranged where it set `bad` or aux.zero.  The sign of the
// other side's mass flux is that of v + c, and c's sign and size come from
// the seed reciprocal (relative error 2^-19): unless v and c cancel to 2^-16,
// that sign is certain.  The momenta's signs follow from it; a -0 energy flux
// and a cancellation take the full evaluation.
template <bool T2>
__device__ __forceinline__ void hllc_redo(double denl, double vxl, double vyl, double vzl,
                                          double prel, double denr, double vxr, double vyr,
                                          double vzr, double prer, const gk::Phys& ph, Flux5& f,
                                          bool bad, const HllcAux& aux) {
    if (!bad && aux.zero) {
        const bool left = aux.ss >= 0;
        const double vo = left ? vxr : vxl, v1 = left ? vyr : vyl, v2 = left ? vzr : vzl;
        const double sc = left ? smax(0.0, aux.so) : smin(0.0, aux.so);
        const double a = sc * (aux.ss - vo);
        const double c = a * rcp_seed(aux.so - aux.ss);
        const double vc = vo + c;
        const bool sure = is_zero(a) || (hi(vc) & 0x7fffffff) + (16 << 20) >= (hi(c) & 0x7fffffff);
        constexpr int kNeg = (int)0x80000000;
        bad = !sure || hi(f.e) == kNeg;
        const int neg = hi(vc);  // sign bit of the other side's mass flux
        auto zero = [&](double& x, int other) {  // -0 + 0*y: -0 for y < 0 or -0, else +0
            if (hi(x) == kNeg) {
                bad = bad || __double2loint(x) != 0;
                x = other < 0 ? x : 0.0;
            }
        };
        zero(f.d, neg);
        zero(f.t1, neg ^ hi(v1));
        if (T2) zero(f.t2, neg ^ hi(v2));
    }
    if (bad)
        f = hllc_far<T2>(HllcStates{denl, vxl, vyl, vzl, prel, denr, vxr, vyr, vzr, prer},
                              ph.gamma, ph.gm1Rec, ph.cq);
}
#endif

// Flux::RiemannSolver for one face of any state.
template <bool T2>
__device__ __forceinline__ void hllc(double denl, double vxl, double vyl, double vzl, double prel,
                                     double denr, double vxr, double vyr, double vzr, double prer,
                                     const gk::Phys& ph, Flux5& f) {
    bool bad = !ph.ranged;
    HllcAux aux;
    hllc_ranged<T2>(denl, vxl, vyl, vzl, prel, denr, vxr, vyr, vzr, prer, ph, f, bad, aux);
#if !GK_FASTMATH
    if (bad || aux.zero)
        hllc_redo<T2>(denl, vxl, vyl, vzl, prel, denr, vxr, vyr, vzr, prer, ph, f, bad, aux);
#endif
}
