// hxg_math64.cuh -- FP64 elementary functions of the sample loops.
//
// The loops are bound by the FP64 pipe (one warp instruction per two clocks
// and SM quarter), so each function is cut to the arguments the loops have:
// no branches for denormals, signs or huge arguments on the common path, and
// a call of the CUDA function outside the stated range.  The bounds below come from
// the rounding of each step; u = 2^-53, an ulp is that of the exact result.
#pragma once

#include "hxg_common.cuh"

namespace hxg {

// 2^(j/64) for j = 0..63, correctly rounded to FP64.
__device__ const double kExp2Tab64[64] = {
    1.0, 1.0108892860517005, 1.0218971486541166, 1.0330248790212284,
    1.0442737824274138, 1.0556451783605572, 1.0671404006768237, 1.0787607977571199,
    1.0905077326652577, 1.102382583307841, 1.1143867425958924, 1.1265216186082418,
    1.1387886347566916, 1.1511892299529827, 1.1637248587775775, 1.1763969916502812,
    1.189207115002721, 1.202156731452703, 1.215247359980469, 1.22848053610687,
    1.241857812073484, 1.255380757024691, 1.2690509571917332, 1.2828700160787783,
    1.2968395546510096, 1.3109612115247644, 1.3252366431597413, 1.339667524053303,
    1.3542555469368927, 1.3690024229745905, 1.383909881963832, 1.3989796725383112,
    1.4142135623730951, 1.42961333839197, 1.4451808069770467, 1.460917794180647,
    1.4768261459394993, 1.4929077282912648, 1.5091644275934228, 1.5255981507445384,
    1.5422108254079407, 1.559004400237837, 1.5759808451078865, 1.593142151342267,
    1.6104903319492543, 1.6280274218573478, 1.645755478153965, 1.6636765803267364,
    1.681792830507429, 1.7001063537185235, 1.718619298122478, 1.7373338352737062,
    1.7562521603732995, 1.7753764925265212, 1.7947090750031072, 1.8142521755003989,
    1.8340080864093424, 1.8539791250833855, 1.8741676341103, 1.8945759815869656,
    1.9152065613971474, 1.9360617934922943, 1.9571441241754002, 1.978456026387951,
};

// The CUDA functions for arguments outside the loops' range, out of line so
// that they cost the loops no registers.
static __device__ __noinline__ double exp_cold(double a) { return exp(a); }
static __device__ __noinline__ double2 sincospi_cold(double x) {
  double2 r;
  sincospi(x, &r.x, &r.y);
  return r;
}

// Coefficients of the functions below.  In constant memory an FP64 instruction
// takes them as an operand; as literals each would take two moves.
struct Coef64 {
  double magic, k64_ln2, ln2_64_hi, ln2_64_lo, e5, e4, e3;
  double s[7], c[7], floor52, r3;
};
static __constant__ Coef64 kC64 = {
    6755399441055744.0,  // 1.5 * 2^52
    92.33248261689366, 0.010830424696249145, 3.623510646634843e-19,  // 64/ln2, ln2/64
    1. / 120., 1. / 24., 1. / 6.,
    {1.5707963267948966, -0.6459640975062443, 0.07969262624603957, -0.0046817541322824235,
     0.00016044115029168176, -3.5986417545158488e-06, 5.633721016175482e-08},
    {-1.2337005501361697, 0.2536695079010469, -0.020863480763315442, 0.000919260274225031,
     -2.5202036991529147e-05, 4.710615657669183e-07, -6.321892462224222e-09},
    4503599627370496.0, 0.375};

// e^a for |a| < 682 (kRange: other arguments go to exp).  Table-driven reduction
// (Tang, ACM TOMS 15, 1989): k = nearest integer of 64 a / ln2, r = a - k ln2/64
// with ln2/64 in two parts and |r| <= ln2/128; e^a = 2^(k >> 6) 2^((k & 63)/64) e^r,
// e^r from its Taylor series to degree 5.  Within 1.4 ulp: half for the table, half
// for the last step, 0.3 for the series (3.4e-17).  10 FP64 instructions.
template <bool kRange>
__device__ __forceinline__ double exp64(double a) {
  if (kRange && ((unsigned)__double2hiint(a) & 0x7fffffffu) >= 0x40855000u) return exp_cold(a);
  const double t = fma(a, kC64.k64_ln2, kC64.magic);
  const int k = __double2loint(t);
  const double kd = t - kC64.magic;
  double r = fma(-kd, kC64.ln2_64_hi, a);
  r = fma(-kd, kC64.ln2_64_lo, r);
  double p = fma(r, kC64.e5, kC64.e4);
  p = fma(p, r, kC64.e3);
  p = fma(p, r, 0.5);
  p = fma(p, r * r, r);
  const double w = __ldg(&kExp2Tab64[k & 63]);
  const double e = fma(w, p, w);
  return __hiloint2double(__double2hiint(e) + ((k >> 6) << 20), __double2loint(e));
}

// 1/sqrt(t) for normal t > 0: the hardware estimate y, e = 1 - t y^2 below 2^-19, and
// y (1 - e)^-1/2 by its binomial series to e^2 (Householder's iteration of third
// order; 5/16 e^3 is left).  Within 1.05 ulp: the rounding of t y is half of e's.
__device__ __forceinline__ double rsqrt64(double t) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(t));
  const double e = fma(-t * y, y, 1.0);
  return fma(y * e, fma(e, kC64.r3, 0.5), y);
}

// sqrt(t) and ir = 1/sqrt(t) for normal t > 0; one Newton step on the root, whose
// residual is exact: within 0.51 ulp.
__device__ __forceinline__ double sqrt64(double t, double &ir) {
  ir = rsqrt64(t);
  const double r = t * ir;
  return fma(fma(-r, r, t), 0.5 * ir, r);
}

// 1/d for normal d whose reciprocal is normal: the hardware estimate y, e = 1 - d y
// below 2^-19, and y (1 - e)^-1 by its geometric series to e^2 (Householder's
// iteration of third order).  Within 0.55 ulp.  Not for a zero, subnormal or
// infinite d: those give NaN.
__device__ __forceinline__ double rcp64(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// sin and cos of h quarter turns (pi h / 2).  h is reduced to f in
// [-1/2, 1/2] exactly; minimax polynomials in f^2 (Remez fits made for this file; as
// FP64 coefficients they give sin(pi f/2)/f to 5e-17 relative, cos(pi f/2) to
// 2.3e-17) and the quadrant from integer operations.  Within 2 u of the exact values,
// the sine polynomial within 2.4 u relative, also near its zeros.
__device__ __forceinline__ void sincos_quarter(double h, double &s, double &c) {
  if (((unsigned)__double2hiint(h) & 0x7fffffffu) >= 0x43000000u) {  // |h| >= 2^49
    const double2 r = sincospi_cold(0.5 * h);
    s = r.x;
    c = r.y;
    return;
  }
  const double t = h + kC64.magic;
  const int n = __double2loint(t);
  const double f = h - (t - kC64.magic);
  const double u = f * f;
  double ps = fma(u, kC64.s[6], kC64.s[5]), pc = fma(u, kC64.c[6], kC64.c[5]);
#pragma unroll
  for (int k = 4; k >= 0; --k) {
    ps = fma(ps, u, kC64.s[k]);
    pc = fma(pc, u, kC64.c[k]);
  }
  ps *= f;
  pc = fma(pc, u, 1.0);
  const bool odd = n & 1;
  const double a = odd ? pc : ps, b = odd ? ps : pc;
  s = __hiloint2double(__double2hiint(a) ^ ((n & 2) << 30), __double2loint(a));
  c = __hiloint2double(__double2hiint(b) ^ (((n + 1) & 2) << 30), __double2loint(b));
}

// a b + c d in two parts, to 4 u^2 (|a b| + |c d|): the products' and the sum's rounding
// errors are exact (FMA; Knuth's two-sum).
__device__ __forceinline__ void dot2_64(double a, double b, double c, double d, double &hi,
                                        double &lo) {
  const double p = a * b, q = c * d;
  hi = p + q;
  const double t = hi - p;
  lo = ((p - (hi - t)) + (q - t)) + (fma(a, b, -p) + fma(c, d, -q));
}

// x^a for normal x > 0: x = 2^E m with m in [0.7, 1.42), and a E split into an integer
// and a rest, so that the argument of the one exponential stays below about |a| / 2 and
// its rounding with it.  Within (1.5 |a| + 4) u relative: 1.1 |a| u of a log m, 0.4 |a| u
// of the sum, 2.7 u of the exponential.  pow for other x and for |a E| of 900 and more.
__device__ inline double pow_k(double x, double a) {
  int hi = __double2hiint(x);
  const int e = ((hi - 0x3fe6a09e) >> 20);
  const double m = __hiloint2double(hi - (e << 20), __double2loint(x));
  const double E = (double)e, p = a * E;
  if (!(fabs(p) < 900.) || hi < 0x00100000 || hi >= 0x7ff00000) return pow(x, a);
  const double n = rint(p);
  const double r = fma((p - n) + fma(a, E, -p), 0.6931471805599453, a * log(m));
  return ldexp(exp64<true>(r), (int)n);
}

// sqrt of v >= 0
__device__ inline double sqrt_pos(double v) {
  double ir;
  return v > 1e-290 ? sqrt64(v, ir) : sqrt(v);
}

}  // namespace hxg
