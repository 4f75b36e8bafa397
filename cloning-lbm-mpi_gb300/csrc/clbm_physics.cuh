// clbm_physics.cuh -- per-node D2Q9 BGK physics used by every kernel.
//
// Two arithmetic policies:
//  * ref64: FP64 in the reference's exact operation order with explicit
//    round-to-nearest intrinsics, so nothing is contracted into an FMA; the
//    results are bit-identical to the reference's g++ build
//    (src/lbm_src/streamCollCompute.cpp:19-41, src/lbm_src/force.cpp:26-48).
//    Terms that the reference multiplies by a lattice velocity of 0 are
//    dropped and the +-1 products are written as additions/subtractions: both
//    are exact, and only the sign of an exactly-zero intermediate could differ.
//  * f32: FP32 populations stored as g = f - w[k] ("shifted"), collision and
//    drag terms evaluated on the shifted values so that the O(1) rest parts
//    cancel analytically instead of in rounding.
#pragma once
#include <type_traits>

#include "clbm_common.cuh"

namespace clbm {

// ---------------------------------------------------------------- ref64 ----
#define DADD __dadd_rn
#define DSUB __dsub_rn
#define DMUL __dmul_rn
#define DDIV __ddiv_rn

struct Moments64 {
  double rho, jx, jy;
};

// rho, jx, jy summed in the reference's k order (streamCollCompute.cpp:21-27)
__device__ __forceinline__ Moments64 moments_ref64(const double f[9]) {
  Moments64 m;
  double r = f[0];
#pragma unroll
  for (int k = 1; k < 9; k++) r = DADD(r, f[k]);
  m.rho = r;
  m.jx = DADD(DSUB(DSUB(DADD(DSUB(f[1], f[3]), f[5]), f[6]), f[7]), f[8]);
  m.jy = DSUB(DSUB(DADD(DADD(DSUB(f[2], f[4]), f[5]), f[6]), f[7]), f[8]);
  return m;
}

// Quotients by one divisor, each the correctly rounded a / b.  The FP64 pipe
// (about two operations per clock and SM) bounds every FP64 kernel, and three
// divisions by the same density are a sixth of a collision.  Markstein's
// method (IBM J. Res. Dev. 34, 1990): with y the correctly rounded 1/b and q
// next to a / b, r = a - b q is exact and q + r y rounds to a / b.  Here y
// comes from the hardware approximation by a cubic step (3 operations, within
// a unit) and a correcting step (2), yl = (1 - b y) y is what it still lacks
// (2), and a quotient costs 4: q = a y + a yl is within half a unit (1 + 2^-50)
// of Q = a / b.  The rounded value then differs from Q by at most
// |Q - q| |b y - 1|, 2^-54 b units for 0.5 <= b < 1 and 2^-55 b for 1 <= b < 2,
// while no midpoint of two doubles lies within 2^-54 / b (2^-53 / b) of a
// quotient: it rounds as Q does.  A significand of b that is all ones (where
// the correcting step may fail), a density outside [0.5, 2) or numerators at
// the ends of the exponent range take the division.
struct Divisor64 {
  double b, y, yl;
  bool ok;
};
__device__ __forceinline__ Divisor64 divisor64(double b) {
  Divisor64 d;
  d.b = b;
  const int hi = __double2hiint(b);
  d.ok = (unsigned)(hi - 0x3fe00000) < 0x00200000u && !((hi & 0xfffff) == 0xfffff && __double2loint(b) == -1);
  double y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
  const double e = __fma_rn(-b, y0, 1.0);
  const double y1 = __fma_rn(__fma_rn(e, e, e), y0, y0);
  d.y = __fma_rn(__fma_rn(-b, y1, 1.0), y1, y1);
  d.yl = DMUL(__fma_rn(-b, d.y, 1.0), d.y);
  return d;
}
// whether a is far from the ends of the exponent range (or zero)
__device__ __forceinline__ bool mid_range64(double a) {
  const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
  return h - 0x10000000u < 0x60000000u || (h | (unsigned)__double2loint(a)) == 0u;
}
__device__ __forceinline__ double div64(double a, const Divisor64 &d) {
  const double q = __fma_rn(a, d.y, DMUL(a, d.yl));
  const double v = __fma_rn(__fma_rn(-d.b, q, a), d.y, q);
  // a zero keeps its sign
  return __hiloint2double(__double2hiint(v) | (__double2hiint(a) & 0x80000000), __double2loint(v));
}

// The velocity of the collision, shifted by the force (streamCollCompute.cpp:28-29)
__device__ __forceinline__ void velocity_ref64(const Moments64 &m, double half_beta, double &ux, double &uy) {
  const Divisor64 d = divisor64(m.rho);
  if (d.ok && mid_range64(m.jx) && mid_range64(m.jy) && mid_range64(half_beta)) {
    ux = DADD(div64(m.jx, d), div64(half_beta, d));
    uy = div64(m.jy, d);
  } else {
    ux = DADD(DDIV(m.jx, m.rho), DDIV(half_beta, m.rho));
    uy = DDIV(m.jy, m.rho);
  }
}

// Sums of doubles on the integer pipe.  An FP64 operation occupies an SM's FP64
// pipe for 16 cycles per warp, while the integer pipes take eight warp
// instructions in that time and are otherwise nearly idle here, so correctly
// rounded additions of values of known size are quicker in 64-bit fixed point:
// a double x, |x| < 1, as x 2^61 rounded to odd (fx: bit 0 also says that
// lower bits were cut off, which happens below 2^-8), and fx_round rounds a sum
// to nearest even where a double of its size would be rounded.  Round-to-odd
// keeps the side and the ties of what was cut off through a sum with an even
// value (1, a rounded value of 2^-8 or more, a double of 2^-7 or more) that is
// itself 2^-7 or more, so that two bits or more are rounded away.
typedef long long fx_t;
constexpr fx_t FX_ONE = 1ll << 61;
__device__ __forceinline__ fx_t fx_abs(double x) {  // of |x|
  const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
  const int e = (int)(hi >> 20);
  const unsigned long long m =
      (((unsigned long long)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | (unsigned)__double2loint(x)) << 9;
  const unsigned s = min((unsigned)(1023 - e), 63u);
  const unsigned long long y = m >> s;
  return (fx_t)(y | (unsigned long long)((y << s) != m));
}
__device__ __forceinline__ fx_t fx(double x) {
  const fx_t y = fx_abs(x);
  return __double2hiint(x) < 0 ? -y : y;
}
// of a positive x in [2^-9, 1): exact
__device__ __forceinline__ fx_t fx_exact(double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  const unsigned long long m =
      (((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x)) << 9;
  return (fx_t)(m >> (1023 - (int)(hi >> 20)));
}
// bits below the last place of a double of this value (0: none to round)
__device__ __forceinline__ int fx_drop(fx_t v) {
  int p;
  asm("bfind.s32 %0, %1;" : "=r"(p) : "r"((int)(v >> 32)));
  return max(p - 20, 0);
}
__device__ __forceinline__ fx_t fx_round(fx_t v) {
  const int k = fx_drop(v);
  const unsigned mask = (1u << k) - 1u;
  v += (fx_t)((mask >> 1) + (((unsigned)v >> k) & mask & 1u));
  return v & ~(fx_t)mask;
}
__device__ __forceinline__ double fx_double(fx_t r) {  // of a positive rounded value of 2^-8 or more
  const int k = fx_drop(r);
  return __longlong_as_double((r >> k) + ((fx_t)(1013 + k) << 52));
}
__device__ __forceinline__ double fx_signed_double(fx_t r) {  // of any rounded value
  const double d = __ll2double_rn(r);  // exact
  return r == 0 ? 0.0 : __hiloint2double(__double2hiint(d) - (61 << 20), __double2loint(d));
}

// 1 + 3 eu + 4.5 eu^2 + u2 for eu = e and eu = -e, u2 = -1.5 |u|^2
// (streamCollCompute.cpp:32-34): the products of -e are those of e with the
// sign changed, exactly, so an opposite pair of directions shares them.  t3 = 3 e,
// h = 4.5 e.
__device__ __forceinline__ void feq_pair_ref64(double e, double t3, double h, double u2, double &plus, double &minus) {
  const double ee = DMUL(h, e);
  plus = DADD(DADD(DADD(1.0, t3), ee), u2);
  minus = DADD(DADD(DSUB(1.0, t3), ee), u2);
}
// The same; where |e| < 0.3 (slow), in fixed point: every sum then lies in
// [0.1, 2.4).  u = fx_abs(u2).
__device__ __forceinline__ void feq_pair_ref64(bool slow, double e, double t3, double h, double u2, fx_t u,
                                               double &plus, double &minus) {
  if (slow) {
    const fx_t t = fx(t3), q = fx_abs(DMUL(h, e));
    plus = fx_double(fx_round(fx_round(fx_round(FX_ONE + t) + q) - u));
    minus = fx_double(fx_round(fx_round(fx_round(FX_ONE - t) + q) - u));
  } else {
    feq_pair_ref64(e, t3, h, u2, plus, minus);
  }
}
// |ux|, |uy| < 0x3fc30000: 0.1484, so that |ux +- uy| < 0.297 -- for every
// thread of the warp that is here, as all such choices (a divided warp would
// go both ways)
__device__ __forceinline__ bool warp_all(bool v) { return __all_sync(__activemask(), v); }
__device__ __forceinline__ bool slow_ref64(double ux, double uy) {
  return warp_all(((unsigned)__double2hiint(ux) & 0x7fffffffu) < 0x3fc30000u &&
                  ((unsigned)__double2hiint(uy) & 0x7fffffffu) < 0x3fc30000u);
}

// moments_ref64 in fixed point, for populations in [2^-9, 1), those of the
// moving directions below 1/4 (every partial sum is then below 3).
__device__ __forceinline__ bool mid_ref64(const double f[9]) {
  unsigned lo = (unsigned)__double2hiint(f[0]), hi = 0;
#pragma unroll
  for (int k = 1; k < 9; k++) {
    lo = min(lo, (unsigned)__double2hiint(f[k]));
    hi = max(hi, (unsigned)__double2hiint(f[k]));
  }
  return warp_all(lo >= 0x3f600000u && hi < 0x3fd00000u && (unsigned)__double2hiint(f[0]) < 0x3ff00000u);
}
__device__ __forceinline__ Moments64 moments_fx(const double f[9]) {
  fx_t v[9];
#pragma unroll
  for (int k = 0; k < 9; k++) v[k] = fx_exact(f[k]);
  fx_t r = v[0];
#pragma unroll
  for (int k = 1; k < 9; k++) r = fx_round(r + v[k]);
  fx_t x = fx_round(v[1] - v[3]), y = fx_round(v[2] - v[4]);
  x = fx_round(fx_round(fx_round(fx_round(x + v[5]) - v[6]) - v[7]) + v[8]);
  y = fx_round(fx_round(fx_round(fx_round(y + v[5]) + v[6]) - v[7]) - v[8]);
  Moments64 m;
  m.rho = fx_double(r);
  m.jx = fx_signed_double(x);
  m.jy = fx_signed_double(y);
  return m;
}
// rho, jx, jy as moments_ref64 sums them, one for all uses of a node
__device__ __forceinline__ Moments64 moments64(const double f[9]) {
  return mid_ref64(f) ? moments_fx(f) : moments_ref64(f);
}

// out = (a + b) + c, the last two steps of the post-collision populations: in
// fixed point where b is in [2^-7, 1) and both sums are at least 2^-7
__device__ __forceinline__ void sum3_ref64(const double a[9], const double b[9], const double c[9], double out[9]) {
  unsigned lo = 0xffffffffu, hi = 0, top = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    lo = min(lo, (unsigned)__double2hiint(b[k]));
    hi = max(hi, (unsigned)__double2hiint(b[k]));
    top = max(top, max((unsigned)__double2hiint(a[k]) & 0x7fffffffu, ((unsigned)__double2hiint(c[k]) & 0x7fffffffu) + 0x100000u));
  }
  if (warp_all(lo >= 0x3f800000u && hi < 0x3ff00000u && top < 0x3ff00000u)) {
    fx_t least = FX_ONE;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const fx_t s = fx_round(fx(a[k]) + fx_exact(b[k])), v = fx_round(s + fx(c[k]));
      least = min(least, min(s, v));
      out[k] = fx_double(v);
    }
    if (warp_all(least >= (1ll << 54))) return;
  }
#pragma unroll
  for (int k = 0; k < 9; k++) out[k] = DADD(DADD(a[k], b[k]), c[k]);
}

// BGK collision with the Guo forcing term, velocity shifted by beta/(2 rho)
// (streamCollCompute.cpp:28-37), every value the reference's, bit for bit.
// wcb[k] = (w[k]*(1 - omega/2))*beta.  The reference evaluates c_k.u, the
// equilibrium and the drive 3 (cx - ux) + 9 cx eu direction by direction;
// here what differs between directions in sign only is formed once: c_k.u of
// opposite directions, 3 ux (the drive's of cx = 0), 3 (1 + ux) (minus the
// drive's of cx = -1), the products w rho: 147 FP64 operations a node (about
// 205 direction by direction, with three divisions), about 60 of which, the
// sums, go to the integer pipe where the values are of ordinary size (moments64,
// feq_pair_ref64, sum3_ref64).  256 clones of 256x64: 2.72 G updates per second
// direction by direction, 3.52 by pairs (1192 us a step), 5.46 with the sums
// in fixed point (768 us).  One node per thread: at one clone of 129x129 (four
// warps an SM) the chain of dependent operations bounds it, 10.5 -> 10.1 us.
// m = moments64(f).
__device__ __forceinline__ void collide_ref64(const double f[9], const Moments64 &m, double out[9], double beta,
                                              const double wcb[9], double omega,
                                              double om1, double *ux_o = nullptr, double *uy_o = nullptr) {
  double ux, uy;
  velocity_ref64(m, DMUL(0.5, beta), ux, uy);
  const double u2 = DMUL(-1.5, DADD(DMUL(ux, ux), DMUL(uy, uy)));
  const double es = DADD(ux, uy), ed = DSUB(ux, uy);  // c_5.u = -c_7.u, c_8.u = -c_6.u
  const double t3x = DMUL(3.0, ux);
  const bool slow = slow_ref64(ux, uy);
  const fx_t u = fx_abs(u2);
  double q[9];
  q[0] = DADD(1.0, u2);
  const double hx = DMUL(4.5, ux), hs = DMUL(4.5, es), hd = DMUL(4.5, ed);
  feq_pair_ref64(slow, ux, t3x, hx, u2, u, q[1], q[3]);
  feq_pair_ref64(slow, uy, DMUL(3.0, uy), DMUL(4.5, uy), u2, u, q[2], q[4]);
  feq_pair_ref64(slow, es, DMUL(3.0, es), hs, u2, u, q[5], q[7]);
  feq_pair_ref64(slow, ed, DMUL(3.0, ed), hd, u2, u, q[8], q[6]);
  // 9 eu = 2 (4.5 eu), rounding included, so its sum with the rest of the
  // drive is one fused operation on an exact product
  const double right = DMUL(3.0, DSUB(1.0, ux)), left = DMUL(3.0, DADD(1.0, ux));
  double drive[9];
  drive[0] = DMUL(wcb[0], -t3x);
  drive[2] = drive[4] = DMUL(wcb[1], -t3x);
  drive[1] = DMUL(wcb[1], __fma_rn(2.0, hx, right));
  drive[5] = DMUL(wcb[5], __fma_rn(2.0, hs, right));
  drive[8] = DMUL(wcb[5], __fma_rn(2.0, hd, right));
  drive[3] = DMUL(wcb[1], __fma_rn(2.0, hx, -left));
  drive[7] = DMUL(wcb[5], __fma_rn(2.0, hs, -left));
  drive[6] = DMUL(wcb[5], __fma_rn(2.0, hd, -left));
  const double r0 = DMUL(w_of(0), m.rho), r1 = DMUL(w_of(1), m.rho), r5 = DMUL(w_of(5), m.rho);
  double old[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    old[k] = DMUL(f[k], om1);
    q[k] = DMUL(DMUL(k == 0 ? r0 : (k <= 4 ? r1 : r5), q[k]), omega);
  }
  sum3_ref64(old, q, drive, out);
  if (ux_o) *ux_o = ux;
  if (uy_o) *uy_o = uy;
}

// Non-equilibrium second moments with the UNshifted velocity, m = moments64(f)
// (FP64 sums: few lanes of a warp are at the square's side, and the fixed-point
// chain is the longer one, 10.65 -> 10.2 us a step of one 129x129 clone)
// (force.cpp:26-46): pi_xx = sum fneq cx cx, pi_xy = sum fneq cx cy.
__device__ __forceinline__ void pi_ref64(const double f[9], const Moments64 &m, double &pxx,
                                         double &pxy) {
  const Divisor64 d = divisor64(m.rho);
  const bool fast = d.ok && mid_range64(m.jx) && mid_range64(m.jy);
  const double uy = fast ? div64(m.jy, d) : DDIV(m.jy, m.rho);
  const double ux = fast ? div64(m.jx, d) : DDIV(m.jx, m.rho);
  const double u2 = DMUL(-1.5, DADD(DMUL(ux, ux), DMUL(uy, uy)));
  const double es = DADD(ux, uy), ed = DSUB(ux, uy);
  double q[9];
  feq_pair_ref64(ux, DMUL(3.0, ux), DMUL(4.5, ux), u2, q[1], q[3]);
  feq_pair_ref64(es, DMUL(3.0, es), DMUL(4.5, es), u2, q[5], q[7]);
  feq_pair_ref64(ed, DMUL(3.0, ed), DMUL(4.5, ed), u2, q[8], q[6]);
  const double r1 = DMUL(w_of(1), m.rho), r5 = DMUL(w_of(5), m.rho);
  double fneq[9];
#pragma unroll
  for (int k = 1; k < 9; k++)
    if (cx_of(k) != 0) fneq[k] = DSUB(f[k], DMUL(k <= 4 ? r1 : r5, q[k]));
  pxx = DADD(DADD(DADD(DADD(DADD(fneq[1], fneq[3]), fneq[5]), fneq[6]), fneq[7]), fneq[8]);
  pxy = DSUB(DADD(DSUB(fneq[5], fneq[6]), fneq[7]), fneq[8]);
}

// ------------------------------------------------------------------ f32 ----
// Shifted populations g = f - w.  With drho = rho - 1:
//   geq_k = feq_k - w_k = w_k (drho + rho (3 eu + 4.5 eu^2 - 1.5 u^2))
//   g*_k  = (1 - omega) g_k + omega geq_k + F_k

// FP32 body force of a node under a random field: beta (1 + eps m), with
// explicit rounding steps so that no kernel contracts or reorders it
// differently (the streaming and cluster-resident kernels must agree bit for
// bit); eps = 0 gives beta exactly.
__device__ __forceinline__ float field_beta_f32(float beta, float eps, float m) {
  return __fmul_rn(beta, __fmaf_rn(eps, m, 1.0f));
}

namespace f32op {
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
}  // namespace f32op

// Packed FP32 arithmetic (Blackwell f32x2): each lane is the IEEE
// round-to-nearest operation of its scalar counterpart, so a packed
// expression gives the same bits as the two scalar ones it replaces.
namespace f32x2op {
__device__ __forceinline__ float lo(f2_t v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi(f2_t v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2_t add(f2_t a, f2_t b) {
  f2_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t sub(f2_t a, f2_t b) {
  f2_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t mul(f2_t a, f2_t b) {
  f2_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t fma(f2_t a, f2_t b, f2_t c) {
  f2_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
}  // namespace f32x2op

// 1/x by the hardware reciprocal approximation (the value x / y takes in
// fast approximate division for x = 1, without its range fix-ups: x here is
// a density near 1)
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The collision organised by opposite pairs (k, opp k): they share |c.u|, so
// with e = c_k.u the equilibria split into an even part
// w (drho + rho (4.5 e^2 - 1.5 u^2)) and an odd part +-3 w rho e, and the
// Guo terms into w fb (9 cx e - 3 ux) and +-3 w fb cx.  Returns drho.
//
// Free of systematic rounding bias in the momentum.  The equilibrium
// momentum rho u (~0.05) is ~10^4 times the body force added per step
// (~1e-6), so a rounding that errs the same way at every node and step,
// even by a fraction of an ulp, acts as a spurious body force of a sizeable
// fraction of the real one and the flow drifts over an interval series.
// Three such roundings are avoided:
//  * the velocity shift: jx + beta/2 rounds a fixed offset onto the grid of
//    jx, the same error at every node; ux = jx/rho + (beta/2)/rho is formed
//    by one fused multiply-add of the exact product jx * (1/rho) instead;
//  * the weights: the odd parts carry the momentum through the coefficients
//    3 w omega, and float(1/9) is 7.5e-9 too large, which puts 7.5e-9 rho u
//    of momentum into every node and step; the coefficients here are
//    c13 ~ omega/3 and c2 ~ omega/12 with omega' = 2 c13 + 4 c2 and
//    om1 = 1 - omega' exact, so the odd parts relax the momentum by exactly
//    the factor the (1 - omega') g_k terms leave;
//  * rho near 1: omega * (3 rho) rounds a near-constant product the same way
//    at many nodes; the odd parts use rho u = ux + drho ux instead, a fused
//    multiply-add of an exact product.
// The remaining roundings act on operands with effectively random low bits.
// Every operation is an explicitly rounded intrinsic (the fused
// multiply-adds chosen here, none left to the compiler), so the result is the
// same bit for bit in every kernel that inlines it.
//
// The four direction pairs are evaluated two at a time in packed f32x2
// arithmetic: the axis pairs (1,3) and (2,4) in lanes 0 and 1 with e = (ux,
// uy), the diagonal pairs (5,7) and (6,8) with e = (ux + uy, uy - ux).  Lane
// 1 of the axis Guo term is fma(0, uy, fx) = fx and its odd part
// fma(c13, ty, -0) = c13 ty, so every lane is the scalar expression of its
// pair; the k -> (k, opp k) sums and differences of the moments are packed
// the same way.  k holds the run's constants in lane pairs (F32Pairs).
__device__ __forceinline__ float collide_f32_pairs(const float g[9], float out[9], float omega,
                                                   const F32Force &f, const F32Pairs &k) {
  using namespace f32op;
  namespace X = f32x2op;
  const f2_t g12 = f2_bits(g[1], g[2]), g34 = f2_bits(g[3], g[4]);
  const f2_t g56 = f2_bits(g[5], g[6]), g78 = f2_bits(g[7], g[8]);
  const f2_t a1324 = X::add(g12, g34), d1324 = X::sub(g12, g34);  // (g1 +- g3, g2 +- g4)
  const f2_t a5768 = X::add(g56, g78);                            // (g5 + g7, g6 + g8)
  const float s57 = sub(g[5], g[7]), t86 = sub(g[8], g[6]);
  const float drho = add(add(add(g[0], X::lo(a1324)), X::hi(a1324)), add(X::lo(a5768), X::hi(a5768)));
  // jy's s57 + (g6 - g8) is s57 - t86: the rounded g6 - g8 is exactly -t86
  const float jx = add(X::lo(d1324), add(s57, t86));
  const float jy = add(X::hi(d1324), sub(s57, t86));
  const float rho = add(1.0f, drho);
  // 1/(1 + drho): the hardware approximation r0 of 1/rho refined by one
  // Newton-Raphson step on the unrounded density, r0 + r0 ((1 - r0) - drho r0)
  // (1 - r0 is exact: r0 is near 1)
  const float r0 = rcp_approx(rho);
  const float inv = fma(r0, fma(-drho, r0, sub(1.0f, r0)), r0);
  const float ux = fma(jx, inv, mul(f.hb, inv));
  const float uy = mul(jy, inv);
  const float tx = fma(drho, ux, ux), ty = fma(drho, uy, uy);  // rho u
  const float u2 = mul(1.5f, fma(ux, ux, mul(uy, uy)));
  const float base = fma(-rho, u2, drho);  // even part before the e^2 term (per unit weight)
  const float fx = mul(f.fbm3, ux);         // Guo even part for cx = 0 (per unit weight)
  // k = 0
  out[0] = fma(X::lo(k.om1), g[0], mul(4.0f / 9.0f, fma(omega, base, fx)));
  const float r45 = mul(4.5f, rho);
  const f2_t R45 = f2_bits(r45, r45), BASE = f2_bits(base, base), FX = f2_bits(fx, fx);
  // axis pairs: lane 0 (1,3) e = ux, cx = 1; lane 1 (2,4) e = uy, cx = 0
  {
    const f2_t e = f2_bits(ux, uy), t = f2_bits(tx, ty);
    const f2_t ev = X::mul(k.w9, X::fma(k.omega, X::fma(X::mul(R45, e), e, BASE), X::fma(k.fb9_0, e, FX)));
    const f2_t od = X::fma(k.c13, t, k.f13_0);
    const f2_t o12 = X::fma(k.om1, g12, X::add(ev, od)), o34 = X::fma(k.om1, g34, X::sub(ev, od));
    out[1] = X::lo(o12);
    out[2] = X::hi(o12);
    out[3] = X::lo(o34);
    out[4] = X::hi(o34);
  }
  // diagonal pairs: lane 0 (5,7) e = ux + uy, cx = 1; lane 1 (6,8) e = uy - ux, cx = -1
  {
    const f2_t e = f2_bits(add(ux, uy), sub(uy, ux)), t = f2_bits(add(tx, ty), sub(ty, tx));
    const f2_t ev = X::mul(k.w36, X::fma(k.omega, X::fma(X::mul(R45, e), e, BASE), X::fma(k.fb9_m, e, FX)));
    const f2_t od = X::fma(k.c2, t, k.f2_m);
    const f2_t o56 = X::fma(k.om1, g56, X::add(ev, od)), o78 = X::fma(k.om1, g78, X::sub(ev, od));
    out[5] = X::lo(o56);
    out[6] = X::hi(o56);
    out[7] = X::lo(o78);
    out[8] = X::hi(o78);
  }
  return drho;
}

// collide_f32_pairs of two nodes at once, node h in lane h of every operand:
// 77 packed operations and two reciprocals for two nodes, where one node at a
// time spends 34 scalar and 21 packed ones.  Every lane takes the operations
// of collide_f32_pairs in the same order with the same roundings.  Packed
// arithmetic has no operand negation, so the chain from the reciprocal on
// runs on negated values (nr = -1/rho, nux = -ux, ...): a rounded product or
// fused multiply-add of negated operands is the negated result, exactly, and
// the signs are taken back by an add for a sub and by negated constants
// (F32Force2).  Left out are the two identities of collide_f32_pairs' lane 1,
// fma(0, uy, fx) = fx and c13 ty - 0 = c13 ty (the sign of a zero aside).
// Returns drho of both nodes.
__device__ __forceinline__ f2_t collide_f32_nodes(const f2_t g[9], f2_t out[9], const F32Pairs &k,
                                                  const F32Force2 &f) {
  namespace X = f32x2op;
  const f2_t a13 = X::add(g[1], g[3]), a24 = X::add(g[2], g[4]);
  const f2_t d13 = X::sub(g[1], g[3]), d24 = X::sub(g[2], g[4]);
  const f2_t s57 = X::sub(g[5], g[7]), t86 = X::sub(g[8], g[6]);
  const f2_t drho = X::add(X::add(X::add(g[0], a13), a24), X::add(X::add(g[5], g[7]), X::add(g[6], g[8])));
  const f2_t jx = X::add(d13, X::add(s57, t86));
  const f2_t jy = X::add(d24, X::sub(s57, t86));
  const f2_t nrho = X::sub(k.mone, drho);
  const f2_t nr0 = f2_bits(rcp_approx(X::lo(nrho)), rcp_approx(X::hi(nrho)));
  const f2_t ninv = X::fma(nr0, X::fma(drho, nr0, X::add(k.one, nr0)), nr0);
  const f2_t nux = X::fma(jx, ninv, X::mul(f.hb, ninv));
  const f2_t nuy = X::mul(jy, ninv);
  const f2_t ntx = X::fma(drho, nux, nux), nty = X::fma(drho, nuy, nuy);
  const f2_t u2 = X::mul(k.c15, X::fma(nux, nux, X::mul(nuy, nuy)));
  const f2_t base = X::fma(nrho, u2, drho);
  const f2_t fx = X::mul(f.nfbm3, nux);
  const f2_t r45 = X::mul(k.mc45, nrho);
  out[0] = X::fma(k.om1, g[0], X::mul(k.w49, X::fma(k.omega, base, fx)));
  {  // (1, 3): e = ux, cx = 1
    const f2_t ev = X::mul(k.w9, X::fma(k.omega, X::fma(X::mul(r45, nux), nux, base), X::fma(f.nfb9, nux, fx)));
    const f2_t nod = X::fma(k.c13, ntx, f.nf13);
    out[1] = X::fma(k.om1, g[1], X::sub(ev, nod));
    out[3] = X::fma(k.om1, g[3], X::add(ev, nod));
  }
  {  // (2, 4): e = uy, cx = 0
    const f2_t ev = X::mul(k.w9, X::fma(k.omega, X::fma(X::mul(r45, nuy), nuy, base), fx));
    const f2_t nod = X::mul(k.c13, nty);
    out[2] = X::fma(k.om1, g[2], X::sub(ev, nod));
    out[4] = X::fma(k.om1, g[4], X::add(ev, nod));
  }
  {  // (5, 7): e = ux + uy, cx = 1
    const f2_t ne = X::add(nux, nuy);
    const f2_t ev = X::mul(k.w36, X::fma(k.omega, X::fma(X::mul(r45, ne), ne, base), X::fma(f.nfb9, ne, fx)));
    const f2_t nod = X::fma(k.c2, X::add(ntx, nty), f.nf2);
    out[5] = X::fma(k.om1, g[5], X::sub(ev, nod));
    out[7] = X::fma(k.om1, g[7], X::add(ev, nod));
  }
  {  // (6, 8): e = uy - ux, cx = -1
    const f2_t ne = X::sub(nuy, nux);
    const f2_t ev = X::mul(k.w36, X::fma(k.omega, X::fma(X::mul(r45, ne), ne, base), X::fma(f.fb9, ne, fx)));
    const f2_t nod = X::fma(k.c2, X::sub(nty, ntx), f.f2);
    out[6] = X::fma(k.om1, g[6], X::sub(ev, nod));
    out[8] = X::fma(k.om1, g[8], X::add(ev, nod));
  }
  return drho;
}

// The FP32 collision of one node of run R; field: the node's random-field
// value, or nullptr under the uniform body force.
__device__ __forceinline__ float collide_f32_run(const RunDev &R, const float S[9], float P[9],
                                                 const float *field = nullptr, float feps = 0.f) {
  if (field) {
    const F32Force f = f32_force(field_beta_f32(R.f_beta, feps, *field), R.f_cforce);
    F32Pairs k = R.f_pairs;
    f32_pairs_force(k, f);
    return collide_f32_pairs(S, P, R.f_omega, f, k);
  }
  return collide_f32_pairs(S, P, R.f_omega, R.f_force, R.f_pairs);
}

// Drag terms from shifted populations, rest parts removed analytically:
//   pi_xx = sum_{cx!=0} g - drho/3 - rho ux^2,  pi_xy = g5 - g6 + g7 - g8 - rho ux uy
// and the West/East rho/3 becomes drho/3 (the +-1/3 cancel between sides).
// (explicitly rounded like collide_f32_pairs)
__device__ __forceinline__ void pi_f32(const float g[9], float &drho_o, float &pxx, float &pxy) {
  using namespace f32op;
  const float a57 = add(g[5], g[7]), a68 = add(g[6], g[8]);
  const float s57 = sub(g[5], g[7]);
  const float drho = add(add(add(g[0], add(g[1], g[3])), add(g[2], g[4])), add(a57, a68));
  const float jx = add(sub(g[1], g[3]), add(s57, sub(g[8], g[6])));
  const float jy = add(sub(g[2], g[4]), add(s57, sub(g[6], g[8])));
  const float rho = add(1.0f, drho);
  const float ux = __fdiv_rn(jx, rho), uy = __fdiv_rn(jy, rho);
  const float sxx = add(add(g[1], g[3]), add(a57, a68));
  const float rux = mul(rho, ux);
  drho_o = drho;
  pxx = fma(-rux, ux, fma(-drho, 1.0f / 3.0f, sxx));
  pxy = fma(-rux, uy, sub(a57, a68));
}

// Momentum-exchange drag of one perimeter node.  A slot k that the square
// bounces back holds S(n,k) = P(n, opp k): the population that left n towards
// the solid along c_{opp k} and came back along c_k, handing the body
// c_{opp k} P - c_k S = -2 c_k S of momentum.  The x parts are summed in k
// order (c_kx = 0 slots carry none).  FP64 on f; FP32 on the shifted g, whose
// missing rest parts -2 c_kx w_k cancel over the perimeter (West against East
// row by row, corner against corner, +-c_x pairs on North and South).
template <bool F64>
__device__ __forceinline__ typename std::conditional<F64, double, float>::type me_node_term(
    const typename std::conditional<F64, double, float>::type S[9], int mask) {
  typename std::conditional<F64, double, float>::type v = 0;
#pragma unroll
  for (int k = 1; k < 9; k++) {
    if (cx_of(k) == 0 || !((mask >> k) & 1)) continue;
    if constexpr (F64) {
      const double s2 = DADD(S[k], S[k]);
      v = cx_of(k) < 0 ? DADD(v, s2) : DSUB(v, s2);
    } else {
      const float s2 = __fadd_rn(S[k], S[k]);
      v = cx_of(k) < 0 ? __fadd_rn(v, s2) : __fsub_rn(v, s2);
    }
  }
  return v;
}

// Drag terms of one perimeter node, stored at [term][clone] so that the
// reduction reads them coalesced: West (x = xmin, index y - ymin), East,
// North (y = ymax, index x - xmin), South.  Stress integration (drag_mode 0):
// FP64 the reference's per-node expressions (force.cpp:48, :78, :108, :138),
// FP32 a shifted variant without the +-1/3 that cancel between West and East.
// Momentum exchange (drag_mode 1): the node's me_node_term in its West or
// East slot (corners included) or its North or South slot, 0 in the North and
// South slots of the corners, so every node counts once.
template <bool F64>
__device__ __forceinline__ void store_drag_terms(
    const RunDev &R, const typename std::conditional<F64, double, float>::type S[9], int x, int y,
    int clone, typename std::conditional<F64, double, float>::type *T, const Moments64 *m64 = nullptr) {
  const int sy = R.ymax - R.ymin, sx = R.xmax - R.xmin;
  // (32-bit offsets: a step's terms of one run are under 2^32, since W >= 3
  // and its populations, 18 W H values a clone, fit the device)
  const unsigned nc = R.nclones;
  if (R.drag_mode == 1) {
    const auto v = me_node_term<F64>(S, bounce_mask(R, x, y));
    const bool corner_x = x == R.xmin || x == R.xmax;
    if (x == R.xmin) T[(unsigned)(y - R.ymin) * nc + clone] = v;
    if (x == R.xmax) T[(unsigned)(sy + 1 + y - R.ymin) * nc + clone] = v;
    if (y == R.ymax) T[(unsigned)(2 * (sy + 1) + x - R.xmin) * nc + clone] = corner_x ? 0 : v;
    if (y == R.ymin) T[(unsigned)(2 * (sy + 1) + sx + 1 + x - R.xmin) * nc + clone] = corner_x ? 0 : v;
    return;
  }
  typename std::conditional<F64, double, float>::type west, east, north, south;
  if constexpr (F64) {
    double pxx, pxy;
    pi_ref64(S, *m64, pxx, pxy);
    const double rho = m64->rho;
    const double third = 1. / 3.;
    const double c = R.cforce;
    west = DADD(DMUL(rho, third), DMUL(c, pxx));
    east = DSUB(DMUL(-rho, third), DMUL(c, pxx));
    north = DMUL(-c, pxy);
    south = DMUL(c, pxy);
  } else {
    float drho, pxx, pxy;
    pi_f32(S, drho, pxx, pxy);
    const float c = R.f_cforce;
    west = __fmaf_rn(drho, 1.0f / 3.0f, __fmul_rn(c, pxx));
    east = -west;
    north = __fmul_rn(-c, pxy);
    south = __fmul_rn(c, pxy);
  }
  if (x == R.xmin) T[(unsigned)(y - R.ymin) * nc + clone] = west;
  if (x == R.xmax) T[(unsigned)(sy + 1 + y - R.ymin) * nc + clone] = east;
  if (y == R.ymax) T[(unsigned)(2 * (sy + 1) + x - R.xmin) * nc + clone] = north;
  if (y == R.ymin) T[(unsigned)(2 * (sy + 1) + sx + 1 + x - R.xmin) * nc + clone] = south;
}

}  // namespace clbm
