// FP64 kernels of the undulator step.
//
// The values are the reference's to a few roundings, not bit for bit: products are fused
// into sums where the code says fma (the unit is compiled with --fmad=false, so nowhere
// else), quotients by gamma and gammaz are products with reciprocals, phases are turned
// instead of passed through sin and cos, the focusing maps and the undulator's factor are
// short series in their usual range, and the ADI's lines are solved in segments
// (adi_plain.cuh). Where a last bit is amplified, it is the reference's: 1 / btpar0 is the
// rounded quotient of the rounded root (recip_sqrt_1m). Operation order otherwise follows
// the cited reference lines.
//
// Layout: particles are structure-of-arrays, slice-major (index is*np + ip);
// fields are [nslice][ngrid*ngrid] double2, storage order with the ring start
// `first`; the deposited source is [nslice][ngrid*ngrid] double2 indexed by
// beam slice.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "g4gpu_internal.h"
#include "launch_chain.cuh"
#include "philox.cuh"

namespace g4 {
namespace {

struct C2 {
  double x, y;
};
__device__ __forceinline__ C2 ld(const double2 *p) {
  double2 v = *p;
  return {v.x, v.y};
}
__device__ __forceinline__ void st(double2 *p, C2 v) { *p = make_double2(v.x, v.y); }
__device__ __forceinline__ C2 cadd(C2 a, C2 b) { return {a.x + b.x, a.y + b.y}; }
// The std::complex<double> product (ac - bd, ad + bc), with each component's first
// product fused into its sum: one rounding fewer per component than GCC's evaluation
// (a last-bit difference), and two FP64 instructions instead of three
__device__ __forceinline__ C2 cmul_fma(C2 a, C2 b) { return {fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x)}; }
// a + i b l for real b. The ADI's cstep and off-diagonal coefficients c[k] are purely
// imaginary (FieldSolverADI.cpp:139, 161-165: real part exactly 0), so the reference's
// complex product i b l is exactly (-b l.y, b l.x); here it is fused into the sum (a
// last-bit difference, two FP64 instructions instead of four).
__device__ __forceinline__ C2 add_imul(C2 a, double b, C2 l) { return {fma(-b, l.y, a.x), fma(b, l.x, a.y)}; }
// d - w n for complex w, both products fused into the difference (four FP64
// instructions instead of six)
__device__ __forceinline__ C2 sub_cmul(C2 d, C2 w, C2 n) {
  return {fma(-w.x, n.x, fma(w.y, n.y, d.x)), fma(-w.x, n.y, fma(-w.y, n.x, d.y))};
}
// real * complex
__device__ __forceinline__ C2 rmul(double s, C2 a) { return {s * a.x, s * a.y}; }
// complex * real
__device__ __forceinline__ C2 mulr(C2 a, double s) { return {a.x * s, a.y * s}; }

// |v| < 2^-k for the exponent field ek = 1023 - k: a comparison of the high word's
// magnitude bits (integer pipe; NaN and infinities fail)
__device__ __forceinline__ bool below_pow2(double v, int ek) {
  return (__double2hiint(v) & 0x7fffffff) < (ek << 20);
}

// TrackBeam::applyDrift / applyFQuad / applyDQuad (TrackBeam.cpp:84-116). The
// divisions by gammaz are multiplications by igz = 1 / gammaz (the products differ
// from the quotients in the last bit).
// With foc^2 = |q| / gammaz and omg = foc delz, the maps' elements are even series in
// omg: of z = q delz^2 / gammaz (positive focusing, negative defocusing),
//   cos or cosh(omg) = 1 - z/2 + z^2/24 - z^3/720,   sin or sinh(omg) / foc =
//   delz (1 - z/6 + z^2/120 - z^3/5040),
// the omitted terms below 2^-63 for |z| < 2^-12. An undulator's natural focusing has z of
// 1e-7 to 1e-6 over half a period, so the square root, the two trigonometric calls and the
// division (about 65 FP64 instructions a plane and half step) become 15. Larger z, a
// quadrupole, takes the calls. Planar undulator, 320 x 8192 particles: push 2150 -> 1660 us;
// helical (both planes focus), 64 x 4096: 295 -> 196 us.
__device__ __forceinline__ void plane_step(int kind, double q, double qd2, double off, double delz,
                                           double &x, double &p, double igz) {
  if (kind == 0) {
    x = fma(p * delz, igz, x);
    return;
  }
  const double z = qd2 * igz;  // qd2 = q delz^2
  double a1, a2;
  if (below_pow2(z, 1023 - 12)) {
    a1 = fma(z, fma(z, fma(z, -1. / 720., 1. / 24.), -0.5), 1.);
    a2 = delz * fma(z, fma(z, fma(z, -1. / 5040., 1. / 120.), -1. / 6.), 1.);
  } else if (kind == 1) {
    const double foc = sqrt(q * igz), omg = foc * delz;
    a1 = cos(omg);
    a2 = sin(omg) / foc;
  } else {
    const double foc = sqrt(-q * igz), omg = foc * delz;
    a1 = cosh(omg);
    a2 = sinh(omg) / foc;
  }
  const double xtmp = x - off;
  x = fma(a1, xtmp, fma(a2 * p, igz, off));
  p = fma(-a2 * q, xtmp, a1 * p);  // a3 gammaz = -a2 foc^2 gammaz = -a2 q
}

// 1 / gammaz of TrackBeam::track (gammaz^2 = gamma^2 - 1 - aw^2 - px^2 - py^2) given itg =
// 1 / gamma: with h = (1 + aw^2 + px^2 + py^2) / gamma^2, itg (1 - h)^(-1/2) by its series,
// 1 + h/2 + 3h^2/8, for h below 2^-18 (the next term is below 2^-55; h is 3e-8 at 5.8 GeV);
// else one reciprocal square root. Both are within an ulp or two of the reference's sqrt
// and quotients.
__device__ __forceinline__ double inv_gammaz(const StepConst &sc, double g, double itg, double px, double py) {
  const double h = fma(py, py, fma(px, px, sc.one_aw_t2)) * (itg * itg);
  if (below_pow2(h, 1023 - 18)) return itg * fma(h, fma(h, 0.375, 0.5), 1.);
  return rsqrt(fma(-py, py, fma(-px, px, fma(g, g, -1.) - sc.aw_t2)));
}

// TrackBeam::track over half a step (TrackBeam.cpp:66-76); `last` applies the
// corrector kick first (TrackBeam.cpp:37-38, 118-128). itg: 1 / g.
__device__ __forceinline__ void transverse(const StepConst &sc, bool last, double g, double itg, double &x,
                                           double &y, double &px, double &py) {
  if (last && sc.corr) {
    px += sc.cxk;
    py += sc.cyk;
  } else if (!last && sc.chic) {
    // TrackBeam::applyChicane (TrackBeam.cpp:224-240): the chicane's transfer minus the
    // drift over its length, which the two half steps then add back
    const double gz = sqrt(g * g - 1 - px * px - py * py);
    double tmp = x;
    x = sc.cm[0] * tmp + sc.cm[1] * px / gz;
    px = sc.cm[2] * tmp * gz + sc.cm[3] * px;
    tmp = y;
    y = sc.cm[4] * tmp + sc.cm[5] * py / gz;
    py = sc.cm[6] * tmp * gz + sc.cm[7] * py;
  }
  const double delz = sc.half_delz;
  const double igz = inv_gammaz(sc, g, itg, px, py);
  plane_step(sc.kindx, sc.qx, sc.qdx2, sc.xoff, delz, x, px, igz);
  plane_step(sc.kindy, sc.qy, sc.qdy2, sc.yoff, delz, y, py, igz);
}

// Field::getLLGridpoint (Field.cpp:160-174). Returns the lower-left cell and the
// weights. A particle within rounding of the upper edge can land on index
// ngrid-1, where the reference's right/upper neighbour carries weight exactly 0;
// the neighbour index is then clamped so that no access leaves the grid.
struct Cell {
  int i00, i10, i01, i11;
  double wx, wy;  // the lower-left weights, 1 - ux and 1 - uy
  double ux, uy;  // the cell coordinates' fractions: the upper/right neighbours' weights
};
// The reference divides x + gridmax by the spacing; the push forms the cell coordinate
// as fma(x, 1 / dgrid, gridmax / dgrid) with host-computed factors (the weights then
// differ in the last bit, and a particle within rounding of a cell boundary may take the
// neighbouring cell, where the bilinear weights give the same value).
// |v| < gm for gm > 0 as an integer comparison of the magnitudes' bit patterns: the
// same verdict as -gm < v < gm for every v (NaN fails both), without the FP64 pipe.
__device__ __forceinline__ bool inside(double v, double gm) {
  return (unsigned long long)(__double_as_longlong(v) & 0x7fffffffffffffffLL) <
         (unsigned long long)__double_as_longlong(gm);
}
// floor(t) and the fraction t - floor(t), both exact, for 0 <= t < 2^31, from the bit
// pattern on the integer pipe (no FP64 rounding, conversion or subtraction): the
// significand's bits below the binary point, shifted up to a normalised significand,
// are the fraction.
__device__ __forceinline__ int floor_frac(double t, double &frac) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(t);
  const int e = (int)(b >> 52) - 1023;
  if (e < 0) {  // t < 1
    frac = t;
    return 0;
  }
  const int sh = 52 - e;  // bits below the binary point
  const unsigned long long m = (b & ((1ULL << 52) - 1)) | (1ULL << 52);
  const unsigned long long fb = m & ((1ULL << sh) - 1);
  const int ip = (int)(m >> sh);
  if (fb == 0) {
    frac = 0.;
    return ip;
  }
  const int lz = __clzll((long long)fb);  // fb < 2^52: lz >= 12; its leading one at bit 63 - lz
  const unsigned long long mant = (fb << (lz - 11)) & ((1ULL << 52) - 1);
  frac = __longlong_as_double((long long)(((unsigned long long)(1023 + 63 - lz - sh) << 52) | mant));
  return ip;
}
__device__ __forceinline__ bool ll_gridpoint(double gm, double idg, double gmi, int ng, double x, double y,
                                             Cell &c) {
  if (inside(x, gm) && inside(y, gm)) {
    // x > -gm, so the coordinate is positive
    const int ix = floor_frac(fma(x, idg, gmi), c.ux), iy = floor_frac(fma(y, idg, gmi), c.uy);
    c.wx = 1. - c.ux;
    c.wy = 1. - c.uy;
    int ix1 = ix + 1 < ng ? ix + 1 : ix;
    int iy1 = iy + 1 < ng ? iy + 1 : iy;
    c.i00 = ix + iy * ng;
    c.i10 = ix1 + iy * ng;
    c.i01 = ix + iy1 * ng;
    c.i11 = ix1 + iy1 * ng;
    return true;
  }
  return false;
}

// 1 / x given r, the reciprocal of a nearby value: for e = 1 - x r below 2^-18, r (1 + e +
// e^2) (the omitted e^3 is below 2^-54), else the division. The RK4 stages of a step change
// gamma by far less than that, so each stage's 1 / gamma follows from the previous one.
__device__ __forceinline__ double recip_near(double x, double r) {
  const double e = fma(-x, r, 1.);
  if (!below_pow2(e, 1023 - 18)) return 1. / x;
  return fma(r, fma(e, e, e), r);
}

// 1 / sqrt(a) as the correctly rounded quotient of 1 by the correctly rounded square
// root (BeamSolver::ODE's btpar0 = sqrt(...), 1 / btpar0), without the square root and
// the division when a = 1 - d, |d| < 2^-14 (btpar0 is 1 - O(1 / gamma^2)):
//  - s0 = 1 - d/2 - d^2/8 - d^3/16 (Taylor series of sqrt(1 - d); the omitted terms
//    are below 2^-60) is within an ulp of sqrt(a). Tuckerman's rounding test picks
//    RN(sqrt(a)) among s0 and its neighbours: with u = next(s0) - s0, sqrt(a) lies above
//    s0 + u/2 iff a > s0 next(s0), the sign of fma(s0, next(s0), -a) (exact: a and
//    s0 next(s0) are multiples of a spacing above u^2 / 4), and the same below.
//  - q0 = 1 + e + e^2 + e^3 for e = 1 - s (exact) is within an ulp of 1 / s. The residual
//    1 - s q0 is exact, and q0 is RN(1 / s) iff it is smaller in magnitude than s g / 2,
//    g the spacing of the doubles on its side of q0 (2^-52 in [1, 2), 2^-53 below 1);
//    1 / s is never a midpoint, as s is a double.
// Both tests run on the integer pipe but the three residuals. Bit-identical to
// 1. / sqrt(a) (checked against IEEE sqrt and division on 1.5e8 arguments either side
// of 1); outside the range, sqrt and the division.
__device__ __forceinline__ double recip_sqrt_near1(double a) {
  const double d = 1. - a;
  if (!below_pow2(d, 1023 - 14)) return 1. / sqrt(a);
  double s = fma(d, fma(d, fma(d, -1. / 16., -1. / 8.), -0.5), 1.);
  const long long sb = __double_as_longlong(s);
  const double su = __longlong_as_double(sb + 1), sd = __longlong_as_double(sb - 1);
  if (__double2hiint(fma(s, su, -a)) < 0) s = su;
  else if (__double2hiint(fma(s, sd, -a)) >= 0) s = sd;
  const double e = 1. - s;
  double q = 1. + fma(fma(e, e, e), e, e);
  const long long qb = __double_as_longlong(q), rb = __double_as_longlong(fma(-s, q, 1.));
  const bool up = rb > 0;  // 1 / s > q
  const bool wide = up ? qb >= 0x3FF0000000000000LL : qb > 0x3FF0000000000000LL;
  const long long hb = __double_as_longlong(s) - ((wide ? 53LL : 54LL) << 52);  // s g / 2
  if ((rb & 0x7fffffffffffffffLL) > hb) q = __longlong_as_double(qb + (up ? 1 : -1));
  return q;
}

// The same on the integer pipe, which the push leaves idle while a warp's FP64 instruction
// holds its scheduler for 64 cycles: ib = 1 / btpar0 and om = 1 - ib (exact), for a = 1 - M
// 2^-53 with 0 < M < 2^31 (a 5.8 GeV beam has M of 3e8; others take recip_sqrt_near1).
//   sqrt(a) = 1 - S 2^-53:  S = M/2 + M^2 2^-56 + M^3 2^-110, to the nearest integer;
//   1 / sqrt = 1 + Q 2^-52: Q = S/2 + S^2 2^-54 + S^3 2^-107, to the nearest integer;
// the terms left out are below 2^-44 of a unit, and neither value is ever halfway between
// two doubles. Equal to 1. / sqrt(a) for every M of the range. About 45 integer
// instructions for 12 FP64 ones, four times a particle.
__device__ __forceinline__ void recip_sqrt_1m(double a, double &ib, double &om) {
  constexpr long long kOne = 0x3FF0000000000000LL;
  const long long m = kOne - __double_as_longlong(a);
  if ((unsigned long long)(m - 1) >= 0x7fffffffULL) {
    ib = recip_sqrt_near1(a);
    om = 1. - ib;
    return;
  }
  const unsigned M = (unsigned)m;
  const unsigned long long M2 = (unsigned long long)M * M;
  const unsigned long long M3 = ((unsigned long long)(unsigned)(M2 >> 31) * M) >> 23;  // M^3 2^-54
  const unsigned long long t = ((unsigned long long)(M & 1u) << 55) + M2 + M3 + (1ULL << 55);
  const unsigned S = (M >> 1) + (unsigned)(t >> 56);
  const unsigned long long S2 = (unsigned long long)S * S;
  const unsigned long long S3 = ((unsigned long long)(unsigned)(S2 >> 30) * S) >> 23;  // S^3 2^-53
  const unsigned long long t2 = ((unsigned long long)(S & 1u) << 53) + S2 + S3 + (1ULL << 53);
  const unsigned Q = (S >> 1) + (unsigned)(t2 >> 54);
  ib = __longlong_as_double(kOne + Q);
  // -Q 2^-52, Q in [1, 2^30): its leading one at bit 31 - lz
  const int lz = __clz((int)Q);
  const unsigned long long mant = ((unsigned long long)Q << (21 + lz)) & 0xfffffffffffffULL;
  om = __longlong_as_double((long long)(0x8000000000000000ULL | ((unsigned long long)(1023 - 52 + 31 - lz) << 52) | mant));
}

// BeamSolver::ODE (BeamSolver.cpp:144-163), given ctmp = sum over the fields of rpart
// e^{-i rharm tthet} and itg = 1 / tgam. Two of the reference's four divisions become
// products with the reciprocals 1 / tgam and 1 / btpar0 (the latter rounded as the
// reference's sqrt and quotient round it, so that xks (1 - 1/btpar0), which xks ~ 1e11
// amplifies, is the reference's value; a last-bit change of 1 / tgam changes btper0 /
// tgam^2 ~ 1e-8 far below the last bit of btpar0); ztemp1 = -2 / xks comes with the step
// constants.
// ACC: how the stage's derivative f enters the RK4 accumulators k2: 0 k2 = f (the first
// two stages, where the reference adds f to zero), 1 k2 = -k2 / 2 + f and 2 k2 = 2 k2 + f
// (the third and fourth, where the reference scales k2 by -0.5 or 2 first): each one
// fma, exact as the reference's product (a scaling by a power of two) and rounded sum.
template <int ACC>
__device__ __forceinline__ void ode(const StepConst &sc, C2 ctmp, double btpar, double ez, double itg, double &k2gg,
                                    double &k2pp) {
  const double btper0 = fma(sc.ztemp1, ctmp.x, btpar);
  double ib, om;
  recip_sqrt_1m(fma(-btper0, itg * itg, 1.), ib, om);
  const double fpp = fma(sc.xks, om, sc.xku), fgg = fma(ctmp.y * ib, itg, -ez);
  if (ACC == 0) {
    k2pp = fpp;
    k2gg = fgg;
  } else {
    const double scale = ACC == 1 ? -0.5 : 2.0;
    k2pp = fma(scale, k2pp, fpp);
    k2gg = fma(scale, k2gg, fgg);
  }
}

// e^{i eps} by its Taylor series, for |eps| < 1/4: the first omitted terms are
// eps^14 / 14! (cosine) and eps^13 / 13! (sine), below 1e-19 at 1/4.
// the RK4 weights' divisions by 6 as products with 1 / 6 (a last-bit difference)
constexpr double kSixth = 1. / 6.;
__device__ __forceinline__ C2 expi_small(double e) {
  const double z = e * e;
  double c = fma(z, 1. / 479001600., -1. / 3628800.);
  c = fma(z, c, 1. / 40320.);
  c = fma(z, c, -1. / 720.);
  c = fma(z, c, 1. / 24.);
  c = fma(z, c, -0.5);
  c = fma(z, c, 1.);
  double sn = fma(z, -1. / 39916800., 1. / 362880.);
  sn = fma(z, sn, -1. / 5040.);
  sn = fma(z, sn, 1. / 120.);
  sn = fma(z, sn, -1. / 6.);
  sn = fma(z, sn, 1.);
  return {c, sn * e};
}
// The same for |eps| < 1/16, the usual case (the remainder is the phase slip of the
// particle's energy and angle offsets over a stage, ~1e-2 rad at 3 sigma of the
// benchmark beam), on the integer pipe: z = eps^2 and the series
//   1 - cos = z/2 - z^2/24 + z^3/720 - z^4/40320,   1 - sin/eps = z/6 - z^2/120 + z^3/5040
//   - z^4/362880
// in fixed point (2^-64 units, the two highest terms in 32 bits), each within 2^-58, the
// first omitted terms below 2^-61; both are then subtracted from 1 in the bit pattern,
// rounded to its 2^-53 spacing. One FP64 instruction (the product with eps) instead of ten.
__device__ __forceinline__ C2 expi_tiny(double e) {
  constexpr long long kOne = 0x3FF0000000000000LL;
  constexpr unsigned long long kMant = (1ULL << 52) - 1;
  const unsigned long long b = (unsigned long long)(__double_as_longlong(e) & 0x7fffffffffffffffLL);
  const int sh = (int)(b >> 52) - 1011;  // |e| 2^64 = significand 2^sh; sh <= 7
  const unsigned long long m = (b & kMant) | (1ULL << 52);
  const unsigned long long ef = sh >= 0 ? m << sh : (sh > -64 ? m >> -sh : 0ULL);
  const unsigned long long z = __umul64hi(ef, ef);  // z 2^64 < 2^56
  const unsigned zh = (unsigned)(z >> 24);          // z 2^40
  // 2^41 (1/720 - z/40320), 2^44 (1/5040 - z/362880)
  const unsigned c3 = 3054198966u - __umulhi(zh, 213044u), s3 = 3490513104u - __umulhi(zh, 189372u);
  const unsigned long long c2 = 768614336404564650ULL - (((unsigned long long)zh * c3) >> 17);  // 2^64 / 24 - ..
  const unsigned long long s2 = 153722867280912930ULL - (((unsigned long long)zh * s3) >> 20);  // 2^64 / 120 - ..
  const unsigned long long oc = (z >> 1) - __umul64hi(z, __umul64hi(z, c2));
  const unsigned long long os = __umul64hi(z, 3074457345618258602ULL - __umul64hi(z, s2));     // 2^64 / 6
  const double c = __longlong_as_double(kOne - (long long)((oc + 1024) >> 11));
  const double f = __longlong_as_double(kOne - (long long)((os + 1024) >> 11));
  return {c, f * e};
}

// e^{i e} for the remainder e of a rotation
__device__ __forceinline__ C2 expi(double e) {
  if (below_pow2(e, 1023 - 4)) return expi_tiny(e);
  if (below_pow2(e, 1023 - 2)) return expi_small(e);
  double sn, c;
  sincos(e, &sn, &c);
  return {c, sn};
}
// a conj(b)
__device__ __forceinline__ C2 cmul_conj(C2 a, C2 b) {
  return {fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y)};
}

// sqrt(1 + d): for |d| < 2^-10 its Taylor series to d^5 (the next term, 21/1024 d^6, is
// below 2^-65), five FP64 instructions instead of eight. The undulator factor's d is
// (ku y)^2, 1e-4 at 25 um.
__device__ __forceinline__ double sqrt_1p(double d) {
  if (!below_pow2(d, 1023 - 10)) return sqrt(1. + d);
  return fma(d, fma(d, fma(d, fma(d, fma(d, 7. / 256., -5. / 128.), 1. / 16.), -1. / 8.), 0.5), 1.);
}

// Deposition of one particle into the source of every field
// (FieldSolverADI.cpp:19-51; FieldSolverFFT.cpp:19-51 is identical).
// cs: (cos, sin) of rharm_k * theta of every field, or null (computed here).
// The source scale of field k for a slice of current cur and npd particles
// (FieldSolverADI.cpp:21-22), in the reference's operation order.
__device__ __forceinline__ double deposit_scale(const StepConst &sc, const FieldStep &fs, double cur, double npd) {
  double scl = fs.fc * kVacimp * cur * fs.xks * sc.delz;
  scl /= 4 * kEev * npd * fs.dgrid * fs.dgrid;
  return scl;
}

// scls: every field's deposit_scale for this slice, or null (computed here). ig: 1 / g,
// or 0 (divided here).
template <int NF>
__device__ __forceinline__ void deposit_particle(const StepConst &sc, double2 *const *src,
                                                 size_t slice_off, int ng, double cur,
                                                 double npd, double g, double th, double x,
                                                 double y, const C2 *cs = nullptr, const double *scls = nullptr,
                                                 double ig = 0.) {
#pragma unroll
  for (int k = 0; k < NF; k++) {
    if (k >= sc.nfld) break;
    const FieldStep &fs = sc.f[k];
    if (!fs.dep_on) continue;
    Cell c;
    if (!ll_gridpoint(fs.gridmax, fs.idgrid, fs.gm_idg, ng, x, y, c)) continue;
    const double scl = scls ? scls[k] : deposit_scale(sc, fs, cur, npd);
    double dfaw2;
    if (sc.centred) {
      dfaw2 = fma(sc.ky * y, y, sc.kx * x * x);
    } else {
      const double dx = x - sc.ax, dy = y - sc.ay;
      dfaw2 = fma(2., fma(sc.grady, dy, sc.gradx * dx), fma(sc.ky * dy, dy, sc.kx * dx * dx));
    }
    const double faw = sqrt_1p(dfaw2);
    double part = ig != 0. ? faw * scl * ig : faw * scl / g;
    double s, co;
    if (cs) {
      co = cs[k].x;
      s = cs[k].y;
    } else {
      sincos(fs.rharm * th, &s, &co);
    }
    C2 cpart = mulr(C2{s, co}, part);
    double2 *d = src[k] + slice_off;
    double w = c.wx * c.wy;
    atomicAdd(&d[c.i00].x, w * cpart.x);
    atomicAdd(&d[c.i00].y, w * cpart.y);
    w = c.ux * c.wy;
    atomicAdd(&d[c.i10].x, w * cpart.x);
    atomicAdd(&d[c.i10].y, w * cpart.y);
    w = c.wx * c.uy;
    atomicAdd(&d[c.i01].x, w * cpart.x);
    atomicAdd(&d[c.i01].y, w * cpart.y);
    w = c.ux * c.uy;
    atomicAdd(&d[c.i11].x, w * cpart.x);
    atomicAdd(&d[c.i11].y, w * cpart.y);
  }
}

struct Ptrs {
  double *gamma, *theta, *x, *y, *px, *py;
  const double *current;
  const double2 *field[G4GPU_MAX_FIELDS];
  double2 *src[G4GPU_MAX_FIELDS];
  // space charge: the short-range field per particle and the long-range loss per
  // slice (null: zero), and which part of the step a launch runs (0 all, 1 the first
  // transverse half step, 2 the rest)
  const double *ez, *eloss;
  int mode;
  // wakes: the loss of every slice (eV/m, Collective::apply), null without them
  const double *wake;
  // particles per slice (one4one windows), null: np in every slice
  const int *count;
  // incoherent radiation: the stream of the step (ctr null: off)
  IsrStream isr;
  // the cached e^{i rharm theta} of every field ([nfield][pstride]) and its validity flag
  // (DeviceBeam::phasor), null: none
  double2 *phasor;
  const int *phasor_ok;
  size_t pstride;
};

// particles of slice is: np, or the slice's own count
__device__ __forceinline__ int slice_np(const Ptrs &p, int is, int np) {
  return p.count ? min(p.count[is], np) : np;
}

// Beam::track (Beam.cpp:296-311): half transverse step, BeamSolver::advance with
// the bilinear field gather and RK4 (BeamSolver.cpp:48-141), half transverse step
// with the corrector; then, with `deposit`, the source deposition of the
// following Field::track. One thread per particle; blockIdx.y is the slice.
template <int NF>
__global__ void __launch_bounds__(512) k_push(StepConst sc, Ptrs p, int ns, int np, int ng,
                                              int deposit) {
  chain_wait();
  int is = blockIdx.y;
  int ip = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = slice_np(p, is, np);
  // the slice's source scales, one thread per field (the block is one slice)
  __shared__ double scls[NF];
  if (deposit && threadIdx.x < NF && (int)threadIdx.x < sc.nfld)
    scls[threadIdx.x] = deposit_scale(sc, sc.f[threadIdx.x], p.current[is], (double)n);
  __syncthreads();
  if (ip >= n) return;
  size_t o = (size_t)is * np + ip;
  double g = p.gamma[o], th = p.theta[o], x = p.x[o], y = p.y[o], px = p.px[o], py = p.py[o];
  size_t ncell = (size_t)ng * ng;

  double itg = 1. / g;  // 1 / gamma, of each RK4 stage from the previous one's
  if (p.mode != 2) transverse(sc, false, g, itg, x, y, px, py);
  if (p.mode == 1) {
    p.x[o] = x;
    p.y[o] = y;
    p.px[o] = px;
    p.py[o] = py;
    return;
  }
  // BeamSolver.cpp:50, 61: ez = the particle's short-range field + the slice's loss
  const double ez = (p.ez ? p.ez[o] : 0.) + (p.eloss ? p.eloss[is] : 0.);

  // BeamSolver::advance, BeamSolver.cpp:53-80
  double gamma = g;
  const double theta0 = sc.autophase != 0. ? th + sc.autophase : th;
  double awloc;
  if (sc.centred) {
    awloc = fma(0.5, fma(sc.ky * y, y, sc.kx * x * x), 1.);
  } else {
    const double dx = x - sc.ax, dy = y - sc.ay;
    awloc = fma(sc.grady, dy, fma(sc.gradx, dx, fma(0.5, fma(sc.ky * dy, dy, sc.kx * dx * dx), 1.)));
  }
  const double btpar = fma(sc.aw2 * awloc, awloc, fma(py, py, fma(px, px, 1.)));
  // Each field's drive rpart e^{-i h theta} at the start of the step (cs: e^{i h theta}, the
  // phasor the last push left, turned by the step's phase offset, or a sincos), and turned
  // by the step's nominal phase advance over half a step and over the step: a stage then
  // multiplies by e^{-i e}, e = h (its phase advance - the nominal one), one complex product
  // instead of a rotated phasor's and the drive's.
  const bool cached = p.phasor && *p.phasor_ok;
  C2 c0 = {0, 0}, chalf[NF], cfull[NF], bfull[NF];
#pragma unroll
  for (int k = 0; k < NF; k++) {
    if (k >= sc.nfld) break;
    const FieldStep &fs = sc.f[k];
    int islice = (is + fs.first) % ns;
    const double2 *f = p.field[k] + (size_t)islice * ncell;
    Cell c;
    C2 drive = {0, 0};
    if (ll_gridpoint(fs.gridmax, fs.idgrid, fs.gm_idg, ng, x, y, c)) {
      // bilinear: along x on both rows, then along y
      const C2 f00 = ld(f + c.i00), f10 = ld(f + c.i10), f01 = ld(f + c.i01), f11 = ld(f + c.i11);
      const C2 lo = {fma(c.ux, f10.x - f00.x, f00.x), fma(c.ux, f10.y - f00.y, f00.y)};
      const C2 hi = {fma(c.ux, f11.x - f01.x, f01.x), fma(c.ux, f11.y - f01.y, f01.y)};
      drive = rmul(fs.rtmp * awloc, C2{fma(c.uy, hi.x - lo.x, lo.x), -fma(c.uy, hi.y - lo.y, lo.y)});
    }
    C2 cs;
    if (cached) {
      cs = ld(p.phasor + k * p.pstride + o);
      if (sc.autophase != 0.) {  // and by the rounding of theta0
        cs = cmul_fma(cs, C2{fs.rot_auto[0], fs.rot_auto[1]});
        cs = add_imul(cs, fs.rharm * ((theta0 - th) - sc.autophase), cs);
      }
    } else {
      double sn, co;
      sincos(fs.rharm * theta0, &sn, &co);
      cs = C2{co, sn};
    }
    drive = cmul_conj(drive, cs);
    c0 = k == 0 ? drive : cadd(c0, drive);
    chalf[k] = cmul_conj(drive, C2{fs.rot_half[0], fs.rot_half[1]});
    cfull[k] = cmul_conj(drive, C2{fs.rot_full[0], fs.rot_full[1]});
    bfull[k] = cmul_fma(cs, C2{fs.rot_full[0], fs.rot_full[1]});
  }
  // sum over the fields of their nominal drives turned by the remainder of the advance dth
  auto drive_at = [&](const C2 *cn, double dth, double dnom) {
    const double d = dth - dnom;
    C2 sum = {0, 0};
#pragma unroll
    for (int k = 0; k < NF; k++) {
      if (k >= sc.nfld) break;
      const C2 v = cmul_conj(cn[k], expi(sc.f[k].rharm == 1. ? d : sc.f[k].rharm * d));
      sum = k == 0 ? v : cadd(sum, v);
    }
    return sum;
  };

  // BeamSolver::RungeKutta, BeamSolver.cpp:89-141, the phase as its advance dth from theta0
  double k2gg, k2pp, k3gg, k3pp;
  ode<0>(sc, c0, btpar, ez, itg, k2gg, k2pp);
  double stpz = sc.half_delz;
  gamma = fma(stpz, k2gg, gamma);
  double dth = stpz * k2pp;
  k3gg = k2gg;
  k3pp = k2pp;
  itg = recip_near(gamma, itg);
  ode<0>(sc, drive_at(chalf, dth, sc.dnom_half), btpar, ez, itg, k2gg, k2pp);
  gamma = fma(stpz, k2gg - k3gg, gamma);
  dth = fma(stpz, k2pp - k3pp, dth);
  k3gg *= kSixth;
  k3pp *= kSixth;
  itg = recip_near(gamma, itg);
  ode<1>(sc, drive_at(chalf, dth, sc.dnom_half), btpar, ez, itg, k2gg, k2pp);  // k2 = -k2 / 2 + f
  stpz = sc.delz;
  gamma = fma(stpz, k2gg, gamma);
  dth = fma(stpz, k2pp, dth);
  k3gg -= k2gg;
  k3pp -= k2pp;
  itg = recip_near(gamma, itg);
  ode<2>(sc, drive_at(cfull, dth, sc.dnom_full), btpar, ez, itg, k2gg, k2pp);  // k2 = 2 k2 + f
  gamma = fma(stpz, fma(k2gg, kSixth, k3gg), gamma);
  dth = fma(stpz, fma(k2pp, kSixth, k3pp), dth);
  double theta = theta0 + dth;
  // the deposition's phasors, kept for the next push and the records: turned by the advance of
  // the phase as it is stored (the rounding of a phase of thousands of radians, step after step,
  // would part them from it: 1e-11 after 600 steps of 8 rad)
  C2 cs[NF];
  if (deposit || p.phasor) {
    const double d = (theta - theta0) - sc.dnom_full;
#pragma unroll
    for (int k = 0; k < NF; k++) {
      if (k >= sc.nfld) break;
      cs[k] = cmul_fma(bfull[k], expi(sc.f[k].rharm == 1. ? d : sc.f[k].rharm * d));
    }
  }

  // Incoherent::apply (Incoherent.cpp:66-77): one draw per beamlet of nbins particles
  if (p.isr.ctr) {
    const double u = isr_uniform(p.isr.seed, *p.isr.ctr, is, ip / p.isr.nbins);
    gamma += -sc.isr_avg + sc.isr_sig * (2 * u - 1);
  }
  // Collective::apply (Collective.cpp:119-128), before the second half step
  if (p.wake) gamma += p.wake[is] * sc.delz / kEev;
  // TrackBeam::applyR56 (TrackBeam.cpp:260-277)
  if (sc.chic) {
    const double th0 = theta;
    theta += sc.r56 * (gamma - sc.gammaref);
    const double r = theta - th0;
    if (deposit || p.phasor) {
#pragma unroll
      for (int k = 0; k < NF; k++) {
        if (k >= sc.nfld) break;
        double sn, co;
        sincos(sc.f[k].rharm * r, &sn, &co);
        cs[k] = cmul_fma(cs[k], C2{co, sn});
      }
    }
  }

  itg = recip_near(gamma, itg);
  transverse(sc, true, gamma, itg, x, y, px, py);

  p.gamma[o] = gamma;
  p.theta[o] = theta;
  p.x[o] = x;
  p.y[o] = y;
  p.px[o] = px;
  p.py[o] = py;
  if (p.phasor) {
#pragma unroll
    for (int k = 0; k < NF; k++) {
      if (k >= sc.nfld) break;
      st(p.phasor + k * p.pstride + o, cs[k]);
    }
  }
  if (deposit) {
    deposit_particle<NF>(sc, p.src, (size_t)is * ncell, ng, p.current[is], (double)n, gamma,
                         theta, x, y, cs, scls, itg);
  }
}

// Deposition alone, for a Field::track without a preceding push.
template <int NF>
__global__ void __launch_bounds__(256) k_deposit(StepConst sc, Ptrs p, int ns, int np, int ng) {
  int is = blockIdx.y;
  int ip = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = slice_np(p, is, np);
  if (ip >= n) return;
  size_t o = (size_t)is * np + ip;
  size_t ncell = (size_t)ng * ng;
  deposit_particle<NF>(sc, p.src, (size_t)is * ncell, ng, p.current[is], (double)n, p.gamma[o],
                       p.theta[o], p.x[o], p.y[o]);
}

// ADI coefficient set: c[ng], cbet[ng], cwet[ng] (FieldSolverADI.cpp:125-182), and the
// segmented solves' powers [2][kSegPow]: kappa^{j+1}, kappa^{j+1} / (1 - kappa^2), followed
// by cbet of the column and of the row solve (solve_cbets, g4gpu_api.cpp)
struct Coef {
  const double2 *c, *cbet, *cwet, *pw;
};

// Right-hand side term cstep * (second difference) with the reference's operand
// order (FieldSolverADI.cpp:64-86): (next - 2 u) + prev, one-sided at the edges.
// next - 2 u as one fma: 2 u is exact, so the single rounding of the fma is the
// reference's rounding of the difference (bit-identical, one FP64 instruction fewer)
__device__ __forceinline__ C2 sub2(C2 next, C2 u) { return {fma(-2.0, u.x, next.x), fma(-2.0, u.y, next.y)}; }
__device__ __forceinline__ C2 lap(bool has_prev, bool has_next, C2 prev, C2 u, C2 next) {
  if (!has_prev) return sub2(next, u);
  if (!has_next) return sub2(prev, u);
  return cadd(sub2(next, u), prev);
}

// First ADI half step: implicit along x (tridagx, FieldSolverADI.cpp:63-75, 94-104).
// One thread per (slice, row); writes the intermediate field to tmp.
__global__ void __launch_bounds__(128) k_adi_x(const double2 *__restrict__ field,
                                               const double2 *__restrict__ src,
                                               double2 *__restrict__ tmp, Coef cf, double cstep,
                                               int ns, int ng, int first) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)ns * ng) return;
  int ii = (int)(t / ng), iy = (int)(t % ng);
  size_t ncell = (size_t)ng * ng;
  int i = (ii + first) % ns;
  const double2 *u = field + (size_t)i * ncell + (size_t)iy * ng;
  // a null source means no deposition this step (outside the undulator or an even
  // harmonic): the reference then solves with a zero source (FieldSolverADI.cpp:14-16)
  const double2 *s = src ? src + (size_t)ii * ncell + (size_t)iy * ng : nullptr;
  double2 *w = tmp + (size_t)i * ncell + (size_t)iy * ng;
  bool hp = iy > 0, hn = iy < ng - 1;
  C2 prev = {0, 0};
  for (int k = 0; k < ng; k++) {
    C2 uc = ld(u + k);
    C2 un = hn ? ld(u + k + ng) : C2{0, 0};
    C2 us = hp ? ld(u + k - ng) : C2{0, 0};
    C2 sv = s ? ld(s + k) : C2{0, 0};
    C2 r = add_imul(cadd(sv, uc), cstep, lap(hp, hn, us, uc, un));
    // r - c[k] u_{k-1} with c[k] = (0, -mlow[k]); c[0] = 0
    C2 v = (k == 0) ? cmul_fma(r, ld(cf.cbet)) : cmul_fma(add_imul(r, -cf.c[k].y, prev), ld(cf.cbet + k));
    st(w + k, v);
    prev = v;
  }
  C2 next = prev;
  for (int k = ng - 2; k >= 0; k--) {
    C2 v = sub_cmul(ld(w + k), ld(cf.cwet + k + 1), next);
    st(w + k, v);
    next = v;
  }
}

// Second ADI half step: implicit along y (tridagy, FieldSolverADI.cpp:77-89, 106-122).
// One thread per (slice, column); reads tmp, writes the field.
__global__ void __launch_bounds__(128) k_adi_y(double2 *__restrict__ field,
                                               const double2 *__restrict__ src,
                                               const double2 *__restrict__ tmp, Coef cf,
                                               double cstep, int ns, int ng, int first) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)ns * ng) return;
  int ii = (int)(t / ng), ix = (int)(t % ng);
  size_t ncell = (size_t)ng * ng;
  int i = (ii + first) % ns;
  double2 *u = field + (size_t)i * ncell + ix;
  const double2 *s = src ? src + (size_t)ii * ncell + ix : nullptr;
  const double2 *w = tmp + (size_t)i * ncell + ix;
  bool hp = ix > 0, hn = ix < ng - 1;
  C2 prev = {0, 0};
  for (int k = 0; k < ng; k++) {
    size_t o = (size_t)k * ng;
    C2 wc = ld(w + o);
    C2 wn = hn ? ld(w + o + 1) : C2{0, 0};
    C2 wp = hp ? ld(w + o - 1) : C2{0, 0};
    C2 sv = s ? ld(s + o) : C2{0, 0};
    C2 r = add_imul(cadd(sv, wc), cstep, lap(hp, hn, wp, wc, wn));
    C2 v = (k == 0) ? cmul_fma(r, ld(cf.cbet)) : cmul_fma(add_imul(r, -cf.c[k].y, prev), ld(cf.cbet + k));
    st(u + o, v);
    prev = v;
  }
  C2 next = prev;
  for (int k = ng - 2; k >= 0; k--) {
    size_t o = (size_t)k * ng;
    C2 v = sub_cmul(ld(u + o), ld(cf.cwet + k + 1), next);
    st(u + o, v);
    next = v;
  }
}

#include "adi_plain.cuh"

#include "diag_plain.cuh"

Ptrs make_ptrs(const DeviceBeam &b, void *const *field, void *const *src, int nfld) {
  Ptrs p{};
  p.gamma = (double *)b.gamma;
  p.theta = (double *)b.theta;
  p.x = (double *)b.x;
  p.y = (double *)b.y;
  p.px = (double *)b.px;
  p.py = (double *)b.py;
  p.current = b.current;
  p.count = b.count;
  p.phasor = (double2 *)b.phasor;
  p.phasor_ok = b.phasor_ok;
  for (int k = 0; k < nfld && k < G4GPU_MAX_FIELDS; k++) {
    p.field[k] = field ? (const double2 *)field[k] : nullptr;
    p.src[k] = src ? (double2 *)src[k] : nullptr;
  }
  return p;
}

// FP64 space charge in the reference's arithmetic
struct PlainSC {
  using R = double;
  using R2 = double2;
  using Th = double;
  using Step = StepConst;
  static constexpr bool kPlain = true;
  static __device__ __forceinline__ double gamma(const StepConst &, double g) { return g; }
  static __device__ __forceinline__ void half(const StepConst &s, double g, double &x, double &y, double &px,
                                              double &py) {
    transverse(s, false, g, 1. / g, x, y, px, py);
  }
  static __device__ __forceinline__ double2 eil(double th, int l) {
    double s, c;
    sincos((double)l * th, &s, &c);
    return make_double2(c, -s);
  }
};

}  // namespace
}  // namespace g4

#include "sc_kernels.cuh"

namespace g4 {

namespace {

// Collective::update for one rank (Collective.cpp:144-161): the window's current
// interpolated to the fine grid, in electrons per fine slice, and its derivative
__global__ void k_wake_profile(const double *cur, int ncur, int ns_hr, double ds, double dscur, double *curh,
                               double *dcur) {
  const int is = blockIdx.x * blockDim.x + threadIdx.x;
  if (is >= ns_hr) return;
  const double s = ds * (double)is;
  unsigned idx = (unsigned)(int)floor(s / dscur);
  if (idx > (unsigned)ncur) idx = (unsigned)ncur;  // s < ncur dscur: never taken
  const double c0 = idx < (unsigned)ncur ? cur[idx] : 0., c1 = idx + 1 < (unsigned)ncur ? cur[idx + 1] : 0.;
  const double wei = 1 - (s - idx * dscur) / dscur;
  double v = wei * c0 + (1 - wei) * c1;
  v *= ds / kCe;
  curh[is] = v;
  dcur[is] = -(c1 - c0) * ds / kCe / dscur;
}

// Collective.cpp:167-179: the wake of slice ic from the fine points ahead of each of
// its `sample` fine points, averaged; loss = external + wake (eV/m), lossf = loss / eev
// in FP32 for the mixed push. One CTA per slice.
__global__ void __launch_bounds__(256) k_wake_slices(const double *curh, const double *dcur, const double *res,
                                                     const double *geo, const double *rou, const double *ext,
                                                     int ns_hr, int sample, double *loss, float *lossf) {
  __shared__ double red[256 / 32];
  const int ic = blockIdx.x, tid = threadIdx.x;
  double w = 0;
  for (int j = 0; j < sample; j++) {
    const int is = ic * sample + j;
    for (int i = tid; i < ns_hr - is; i += blockDim.x) {
      w += curh[is + i] * (res[i] + rou[i]);
      w += dcur[is + i] * geo[i];
    }
  }
  for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  if ((tid & 31) == 0) red[tid >> 5] = w;
  __syncthreads();
  if (tid == 0) {
    double t = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += red[i];
    const double l = ext[ic] + t / (double)sample;
    loss[ic] = l;
    lossf[ic] = (float)(l / kEev);
  }
}

}  // namespace

void launch_wake_update(const Launch &L, const double *cur, int nslice, int ns_hr, double ds, const double *ext,
                        const double *res, const double *geo, const double *rou, double *scratch, double *loss,
                        float *lossf) {
  cudaStream_t s = (cudaStream_t)L.stream;
  const double dscur = ds * (unsigned)ns_hr / nslice;
  int sample = (int)(dscur / ds);
  if (sample < 1) sample = 1;
  k_wake_profile<<<(ns_hr + 255) / 256, 256, 0, s>>>(cur, nslice, ns_hr, ds, dscur, scratch, scratch + ns_hr);
  k_wake_slices<<<nslice, 256, 0, s>>>(scratch, scratch + ns_hr, res, geo, rou, ext, ns_hr, sample, loss, lossf);
}

size_t sc_bytes_per_mode(int ng, int mixed) {
  return (size_t)ng * (mixed ? sizeof(float2) + sizeof(float) : sizeof(double2) + sizeof(double));
}
size_t sc_max_smem() { return 220 * 1024; }

void launch_sc_plain(const Launch &L, const ScConst &c, const StepConst &step, const DeviceBeam &b,
                     const ScBuffers &buf, int part) {
  ScBeam<PlainSC> sb{(double *)b.gamma, (double *)b.x,           (double *)b.y, (double *)b.px,
                     (double *)b.py,    (const double *)b.theta, b.current,    b.count};
  sc_launch<PlainSC>(L, c, step, sb, buf, part);
}

void launch_push_plain(const Launch &L, const StepConst &sc, const DeviceBeam &b,
                       void *const *field, void *const *src, int ns, int np, int ngrid,
                       int deposit, int block) {
  launch_push_plain_sc(L, sc, b, field, src, ns, np, ngrid, deposit, block, 0, nullptr, nullptr, nullptr,
                       IsrStream{});
}

namespace {
__global__ void k_isr_advance(unsigned long long *ctr) { *ctr += 1; }
}  // namespace

void launch_isr_advance(void *stream, unsigned long long *ctr) {
  k_isr_advance<<<1, 1, 0, (cudaStream_t)stream>>>(ctr);
}

void launch_push_plain_sc(const Launch &L, const StepConst &sc, const DeviceBeam &b, void *const *field,
                          void *const *src, int ns, int np, int ngrid, int deposit, int block, int mode,
                          const void *ez, const double *eloss, const void *wake, const IsrStream &isr) {
  Ptrs p = make_ptrs(b, field, src, sc.nfld);
  if (isr.ctr && (sc.isr_avg != 0 || sc.isr_sig != 0) && mode != 1) p.isr = isr;
  p.mode = mode;
  p.ez = (const double *)ez;
  p.eloss = eloss;
  p.wake = (const double *)wake;
  if (mode == 1) deposit = 0;
  p.pstride = (size_t)ns * np;
  // a launch that only moves the particles transversely leaves theta and the cache as
  // they are
  if (mode == 1) p.phasor = nullptr;
  dim3 grid((np + block - 1) / block, ns);
  cudaStream_t s = (cudaStream_t)L.stream;
  switch (sc.nfld) {
    case 1: chain_launch(k_push<1>, grid, block, 0, s, 0, sc, p, ns, np, ngrid, deposit); break;
    case 2: chain_launch(k_push<2>, grid, block, 0, s, 0, sc, p, ns, np, ngrid, deposit); break;
    case 3: chain_launch(k_push<3>, grid, block, 0, s, 0, sc, p, ns, np, ngrid, deposit); break;
    default: chain_launch(k_push<G4GPU_MAX_FIELDS>, grid, block, 0, s, 0, sc, p, ns, np, ngrid, deposit); break;
  }
  // every particle's phasor now matches its phase (bytes of 1: a nonzero flag)
  if (p.phasor) cudaMemsetAsync((void *)p.phasor_ok, 1, sizeof(int), s);
}

void launch_deposit_plain(const Launch &L, const StepConst &sc, const DeviceBeam &b,
                          void *const *src, int ns, int np, int ngrid) {
  Ptrs p = make_ptrs(b, nullptr, src, sc.nfld);
  dim3 grid((np + 255) / 256, ns);
  cudaStream_t s = (cudaStream_t)L.stream;
  switch (sc.nfld) {
    case 1: k_deposit<1><<<grid, 256, 0, s>>>(sc, p, ns, np, ngrid); break;
    case 2: k_deposit<2><<<grid, 256, 0, s>>>(sc, p, ns, np, ngrid); break;
    case 3: k_deposit<3><<<grid, 256, 0, s>>>(sc, p, ns, np, ngrid); break;
    default: k_deposit<G4GPU_MAX_FIELDS><<<grid, 256, 0, s>>>(sc, p, ns, np, ngrid); break;
  }
}

namespace {
// How launch_adi_plain cuts the lines of a window: L lines a CTA, nseg segments a line
// (0: one thread per line, k_adi_x / k_adi_y), threads a CTA.
struct AdiShape {
  int L, nseg, threads;
};
// Why these: a warp's FP64 instruction holds its scheduler for 64 cycles whatever lanes
// are active, so the solve wants full warps, enough of them on every SM, and no more
// segments than that takes (each adds 8 W instructions a line). Measured (both half
// steps, step factor 0.034, W 13; in brackets one thread per line):
//   1 slice x 255^2     L 2, nseg 19   33 us (688)      22 x 101^2   L 4, nseg 6   40 us (292)
//   4 x 151^2           L 2, nseg 8    33 us (428)      60 x 151^2   L 8, nseg 4  111 us (446)
//   320 x 151^2         L 8, nseg 4   510 us (870)      2000 x 101^2 L 8, nseg 4 1480 us (1925)
// so: at four CTAs an SM of 8 lines and segments of about 36 elements, that; below, the
// most segments and fewer lines, down to 2. Two segments of 16 lines fill a warp where
// the warm-up leaves no more (2000 x 101^2: 1567 us). One segment is slower than one thread
// per line (320 x 151^2: 967 us), as are lines of which two do not fit shared memory.
AdiShape adi_shape(int ns, int ng, int W) {
  const int most = W > 0 ? ng / W : 1;
  if (most < 2) return {0, 0, 128};
  AdiShape s{8, 4 * std::max(1, (ng + 70) / 144), 64};
  const long long bands = (long long)ns * ((ng + 7) / 8);
  if (bands < 4 * device_sms()) {
    s.L = bands < device_sms() ? 2 : 4;
    s.threads = 128;
    s.nseg = s.threads / s.L;
  } else if (most < 4) {
    s.L = 16;
  }
  s.nseg = std::min(s.nseg, most);
  while (s.L > 2 && (size_t)s.L * (ng | 1) * sizeof(double2) > 100 * 1024) s.L /= 2;
  if ((size_t)s.L * (ng | 1) * sizeof(double2) > 100 * 1024) return {0, 0, 128};
  s.threads = std::max(s.threads, (s.L * s.nseg + 31) / 32 * 32);
  if (s.threads > 512) {
    s.threads = 512;
    s.nseg = 512 / s.L;
  }
  return s;
}

template <int L>
void launch_adi_lines(cudaStream_t st, int phase, const AdiShape &a, double2 *field, double2 *src, double2 *tmp,
                      const Coef &cf, double c, int ns, int ng, int first, int W, int has_src) {
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !(configured.load() & (1ull << dev))) {
    cudaFuncSetAttribute(adi64::k_adi_rows<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    cudaFuncSetAttribute(adi64::k_adi_cols<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    if (dev < 64) configured.fetch_or(1ull << dev);
  }
  const int nband = (ng + L - 1) / L, nco = std::min(W, ng);
  const size_t smem = adi64::lines_bytes(L, L * (phase == 0 ? ng | 1 : ng), a.nseg, nco, W);
  const unsigned blocks = (unsigned)ns * (unsigned)nband;
  if (phase == 0)
    chain_launch(adi64::k_adi_rows<L>, blocks, a.threads, smem, st, 0, field, src, tmp, cf, c, ns, ng, first, nband, a.nseg,
                 nco, W, has_src);
  else
    chain_launch(adi64::k_adi_cols<L>, blocks, a.threads, smem, st, 0, field, src, tmp, cf, c, ns, ng, first, nband, a.nseg,
                 nco, W);
}
}  // namespace

void launch_adi_plain(const Launch &L, const StepConst &sc, int k, int phase, void *field, void *src, void *tmp,
                      const void *coef, const void *pow, int ns, int ngrid, int has_src) {
  const double2 *cb = (const double2 *)coef;
  cudaStream_t s = (cudaStream_t)L.stream;
  const FieldStep &f = sc.f[k];
  const double2 *pw = (const double2 *)pow;
  const AdiShape a = adi_shape(ns, ngrid, f.tw);
  const Coef cf{cb, a.L ? pw + (phase == 1 ? 2 : 3) * kSegPow : cb + ngrid, cb + 2 * ngrid, pw};
  double2 *u = (double2 *)field, *sv = (double2 *)src, *w = (double2 *)tmp;
  switch (a.L) {
    case 2: return launch_adi_lines<2>(s, phase, a, u, sv, w, cf, f.cstep, ns, ngrid, f.first, f.tw, has_src);
    case 4: return launch_adi_lines<4>(s, phase, a, u, sv, w, cf, f.cstep, ns, ngrid, f.first, f.tw, has_src);
    case 8: return launch_adi_lines<8>(s, phase, a, u, sv, w, cf, f.cstep, ns, ngrid, f.first, f.tw, has_src);
    case 16: return launch_adi_lines<16>(s, phase, a, u, sv, w, cf, f.cstep, ns, ngrid, f.first, f.tw, has_src);
    default: break;
  }
  // one thread per line, each line's sweep the reference's single sequential pass
  const double2 *sr = has_src ? sv : nullptr;
  const long long n = (long long)ns * ngrid;
  const unsigned blocks = (unsigned)((n + 127) / 128);
  if (phase == 0)
    k_adi_x<<<blocks, 128, 0, s>>>(u, sr, w, cf, f.cstep, ns, ngrid, f.first);
  else
    k_adi_y<<<blocks, 128, 0, s>>>(u, sr, w, cf, f.cstep, ns, ngrid, f.first);
}

namespace {
// One CTA of threads per column width of the grid (two or more columns a thread above
// 256), so that the FP64 pipe, which a warp's instruction holds whatever lanes are active,
// runs full warps.
int diag_threads(int ng) {
  const int per = (ng + 255) / 256, cols = (ng + per - 1) / per;
  return std::max(128, (cols + 31) / 32 * 32);
}
// Particles a thread: the reduction over a CTA costs its threads about 35 FP64
// instructions each, a particle 14, so 8 of them where that still leaves two CTAs an SM,
// fewer in a window of few slices (1 slice x 8192: 32 CTAs of 256).
int diag_chunk(int ns, int np, int nt) {
  int m = 8;
  while (m > 1 && (long long)ns * ((np + m * nt - 1) / (m * nt)) < 2 * device_sms()) m /= 2;
  return m * nt;
}
// Rows a CTA: 32, or fewer down to 2 for about four CTAs an SM.
int diag_rows(int nslice, int ng) {
  return (int)std::max(2LL, std::min(32LL, (long long)nslice * ng / (4 * device_sms())));
}
template <int NH>
void launch_diag_nh(cudaStream_t s, const diag64::Args &a, unsigned blocks, int nt) {
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !(configured.load() & (1ull << dev))) {
    cudaFuncSetAttribute(diag64::k_diag<NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    if (dev < 64) configured.fetch_or(1ull << dev);
  }
  const size_t smem = (size_t)diag64::kSlots<NH> * (nt + 1) * sizeof(double);
  diag64::k_diag<NH><<<blocks, nt, smem, s>>>(a);
}
}  // namespace

size_t diag_plain_scratch(int ns, int np, int nharm, int ng, int nfield, size_t *counters) {
  const int nt = diag_threads(ng), chunk = diag_chunk(ns, np, nt), rows = diag_rows(ns * nfield, ng);
  *counters = (size_t)ns * (1 + nfield);
  return (size_t)ns * ((np + chunk - 1) / chunk) * beam_diag_width(nharm <= 1 ? 1 : nharm <= 3 ? 3 : G4GPU_MAX_HARM) +
         (size_t)nfield * ns * ((ng + rows - 1) / rows) * kFieldSums;
}

void launch_diag_plain(const Launch &L, const DeviceBeam &b, void *const *field, int nfield, int h1, int ns, int np,
                       int ngrid, int nharm, double gref, bool beam, bool fields, double *rec, double *scratch,
                       unsigned *count) {
  diag64::Args a{};
  a.p = make_ptrs(b, field, nullptr, nfield);
  const int nt = diag_threads(ngrid);
  a.ns = ns;
  a.np = np;
  a.nharm = nharm;
  a.ng = ngrid;
  a.gref = gref;
  a.chunk = diag_chunk(ns, np, nt);
  a.nbc = beam ? (np + a.chunk - 1) / a.chunk : 0;
  a.rows = diag_rows(ns * nfield, ngrid);
  a.nfc = (ngrid + a.rows - 1) / a.rows;
  a.ph1 = h1 >= 0 && b.phasor ? (const double2 *)b.phasor + (size_t)h1 * ns * np : nullptr;
  a.rec = rec;
  a.part = scratch;
  a.count = count;
  const unsigned blocks = (unsigned)ns * a.nbc + (fields ? (unsigned)nfield * ns * a.nfc : 0u);
  if (!blocks) return;
  cudaStream_t s = (cudaStream_t)L.stream;
  if (nharm <= 1)
    launch_diag_nh<1>(s, a, blocks, nt);
  else if (nharm <= 3)
    launch_diag_nh<3>(s, a, blocks, nt);
  else
    launch_diag_nh<G4GPU_MAX_HARM>(s, a, blocks, nt);
}

}  // namespace g4
