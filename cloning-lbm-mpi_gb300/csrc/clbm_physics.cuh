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
  bool mid;  // warp-uniform: every population of ordinary size (mid_ref64)
};

// rho, jx, jy summed in the reference's k order (streamCollCompute.cpp:21-27)
__device__ __forceinline__ Moments64 moments_ref64(const double f[9]) {
  Moments64 m;
  m.mid = false;
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

// Doubles on the integer pipes.  An FP64 operation occupies an SM's FP64 pipe
// for 16 cycles per warp, while the other pipes take a warp instruction in a
// quarter of a cycle to two and are otherwise nearly idle here, so correctly
// rounded sums and products of values of known size are quicker in 64-bit
// fixed point: a double x as x 2^61 (fx_t), with what lies below that rounded
// to odd (bit 0 also says that lower bits were cut off), and fx_round rounds a
// sum or product to nearest even where a double of its size would be rounded.
// Round-to-odd keeps the side and the ties of what was cut off through a sum
// with an even value, and the rounding is right where it takes two bits or more
// away: results of 2^-7 or more (2^54 before rounding).
typedef long long fx_t;
typedef unsigned long long fxu_t;
constexpr fx_t FX_ONE = 1ll << 61;
// significand of |x| with its leading one (none for a subnormal), as an integer
__device__ __forceinline__ fxu_t fx_significand(double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  return ((fxu_t)((hi & 0xfffffu) | (hi & 0x7ff00000u ? 0x100000u : 0u)) << 32) | (unsigned)__double2loint(x);
}
__device__ __forceinline__ fx_t fx_abs(double x) {  // of |x| < 1
  const fxu_t m = fx_significand(x) << 9;
  const unsigned s = min(1023u - (((unsigned)__double2hiint(x) & 0x7fffffffu) >> 20), 63u);
  const fxu_t y = m >> s;
  return (fx_t)(y | (fxu_t)((y << s) != m));
}
// of a positive x in [2^-9, 1): exact
__device__ __forceinline__ fx_t fx_exact(double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  const fxu_t m = (((fxu_t)((hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x)) << 9;
  return (fx_t)(m >> (1023 - (int)(hi >> 20)));
}
// Round to the 53 bits of a double (none to round below 2^-8).  A leading bit
// at 63 - z takes 11 - z bits away: mask has them, half half a unit less one.
struct FxPlace {
  unsigned mask, half, shift;
};
__device__ __forceinline__ FxPlace fx_place(fx_t v) {
  FxPlace p;
  asm("{\n\t.reg .u32 z;\n\t"
      "bfind.shiftamt.s32 z, %3;\n\t"
      "shr.u32 %0, 2047, z;\n\t"
      "shr.u32 %1, 1023, z;\n\t"
      "sub.u32 %2, 11, z;\n\t}"
      : "=r"(p.mask), "=r"(p.half), "=r"(p.shift)
      : "r"((int)(v >> 32)));
  return p;
}
__device__ __forceinline__ fx_t fx_round(fx_t v) {
  const FxPlace p = fx_place(v);
  v += (fx_t)(p.half + (((unsigned)v >> (p.shift & 31)) & p.mask & 1u));
  return v & ~(fx_t)p.mask;
}
// a b 2^-64, rounded to odd
__device__ __forceinline__ fx_t fx_mul(fxu_t a, fxu_t b) {
  const unsigned al = (unsigned)a, ah = (unsigned)(a >> 32), bl = (unsigned)b, bh = (unsigned)(b >> 32);
  const fxu_t p = (fxu_t)al * bl;
  const fxu_t q = (fxu_t)ah * bl + (p >> 32);
  const fxu_t r = (fxu_t)al * bh + (unsigned)q;
  const fxu_t h = (fxu_t)ah * bh + (q >> 32) + (r >> 32);
  return (fx_t)(h | (fxu_t)(((unsigned)p | (unsigned)r) != 0u));
}
// a positive value of 2^-8 or more, rounded, as a double (a carry out of the
// significand goes to the exponent)
__device__ __forceinline__ double fx_double(fx_t v) {
  const FxPlace p = fx_place(v);
  v += (fx_t)(p.half + (((unsigned)v >> (p.shift & 31)) & p.mask & 1u));
  v >>= p.shift & 31;
  return __hiloint2double((int)(v >> 32) + (int)((1013 + p.shift) << 20), (int)v);
}
// any rounded value as a double (a conversion would take the FP64 pipe)
__device__ __forceinline__ double fx_signed_double(fx_t r) {
  const fxu_t m = (fxu_t)(r < 0 ? -r : r);
  const int z = __clzll((fx_t)m);  // 64 for zero
  const fxu_t v = m << (z & 63) >> 11;  // leading one at 52
  const int hi = (int)(v >> 32) + ((1023 + 1 - z) << 20);
  return m == 0 ? 0.0 : __hiloint2double(hi | ((int)(r >> 32) & (int)0x80000000u), (int)v);
}
// 3 |x|, rounded as a double, for |x| < 0.32
__device__ __forceinline__ fx_t fx_abs3(double x) {
  fxu_t m = 3u * (fx_significand(x) << 9);  // leading one at 62 or 63
  const unsigned k = 10u + (unsigned)(m >> 63), mask = (1u << k) - 1u;
  m += (fxu_t)((mask >> 1) + (((unsigned)m >> k) & 1u));
  m &= ~(fxu_t)mask;
  const unsigned s = min(1023u - (((unsigned)__double2hiint(x) & 0x7fffffffu) >> 20), 63u);
  const fxu_t y = m >> s;
  return (fx_t)(y | (fxu_t)((y << s) != m));
}
// A choice between fixed point and FP64 is made for every thread of the warp
// that is here: a divided warp would go both ways.
__device__ __forceinline__ bool warp_all(bool v) { return __all_sync(__activemask(), v); }

// moments_ref64 in fixed point, for populations in [2^-8, 1), those of the
// moving directions below 1/4 (every partial sum is then below 3).
__device__ __forceinline__ bool mid_ref64(const double f[9]) {
  unsigned lo = (unsigned)__double2hiint(f[0]), hi = 0;
#pragma unroll
  for (int k = 1; k < 9; k++) {
    lo = min(lo, (unsigned)__double2hiint(f[k]));
    hi = max(hi, (unsigned)__double2hiint(f[k]));
  }
  return warp_all(lo >= 0x3f700000u && hi < 0x3fd00000u && (unsigned)__double2hiint(f[0]) < 0x3ff00000u);
}
__device__ __forceinline__ Moments64 moments_fx(const fx_t v[9]) {
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
  m.mid = true;
  return m;
}
// A thread's node on its way through the collision, in shared memory: in
// registers it takes 90 and more (ten blocks of 64 threads an SM), and rows
// allow loops over the directions, whose straight-line code, 50 KB, was
// waiting for instructions.  f: fixed point where the moments are (mid), else
// the bits of the double.
template <int BLOCK>
struct Node64 {
  fx_t f[9][BLOCK], q[9][BLOCK];
  double drive[9][BLOCK];
};
__device__ __forceinline__ void column_fence() { asm volatile("" ::: "memory"); }  // no value kept in a register
template <int BLOCK>
__device__ __forceinline__ double node_f(const Node64<BLOCK> &s, bool mid, int k) {
  const fx_t v = s.f[k][threadIdx.x];
  return mid ? fx_double(v) : __longlong_as_double(v);
}
// rho, jx, jy as moments_ref64 sums them, one for all uses of a node
template <int BLOCK>
__device__ __forceinline__ Moments64 moments64(Node64<BLOCK> &s, const double f[9]) {
  Moments64 m;
  if (mid_ref64(f)) {
    fx_t v[9];
#pragma unroll
    for (int k = 0; k < 9; k++) s.f[k][threadIdx.x] = v[k] = fx_exact(f[k]);
    m = moments_fx(v);
  } else {
    m = moments_ref64(f);
#pragma unroll
    for (int k = 0; k < 9; k++) s.f[k][threadIdx.x] = __double_as_longlong(f[k]);
  }
  column_fence();
  return m;
}

// 1 + 3 eu + 4.5 eu^2 + u2 for eu = e and eu = -e, u2 = -1.5 |u|^2
// (streamCollCompute.cpp:32-34): the products of -e are those of e with the
// sign changed, exactly, so an opposite pair of directions shares them.  t3 = 3 e,
// ee = 4.5 e e.
__device__ __forceinline__ void feq_pair_ref64(double t3, double ee, double u2, double &plus, double &minus) {
  plus = DADD(DADD(DADD(1.0, t3), ee), u2);
  minus = DADD(DADD(DSUB(1.0, t3), ee), u2);
}
// In fixed point where |e| < 0.3 (every sum then lies in [0.1, 2.4)); u = -u2.
__device__ __forceinline__ void feq_pair_fx(double e, double ee, fx_t u, fx_t &plus, fx_t &minus) {
  const fx_t t3 = fx_abs3(e), q = fx_abs(ee), t = __double2hiint(e) < 0 ? -t3 : t3;
  plus = fx_round(fx_round(fx_round(FX_ONE + t) + q) - u);
  minus = fx_round(fx_round(fx_round(FX_ONE - t) + q) - u);
}

// The post-collision populations (f om1 + (w rho) q omega) + drive of a node in
// fixed point, q = 1 + 3 eu + 4.5 eu^2 + u2 by directions; false where a value
// is not of the size that needs.  r0 = w[0] rho in [1/4, 1/2): the other
// products w rho are a quarter and a sixteenth of it, so all have its
// significand, and all quotients of scale go to the place of omega's.
template <int BLOCK>
__device__ __forceinline__ bool relax_fx(Node64<BLOCK> &s64, double r0, double omega, double om1) {
  const int t = threadIdx.x;
  const int e1 = (int)(((unsigned)__double2hiint(om1) & 0x7fffffffu) >> 20);  // om1 = 2^(e1 - 1023) M1 2^-63
  const fxu_t M1 = fx_significand(om1) << 11, R = fx_significand(r0) << 11;
  const unsigned s1 = om1 == 0.0 ? 2 : 1024 - e1, low1 = (1u << s1) - 1u;
  const fx_t sign1 = __double2hiint(om1) < 0 ? -1 : 0;
  const fxu_t Om = fx_significand(omega) << ((__double2hiint(omega) >> 20) - 1016);  // omega 2^59
  int least = 0x7fffffff;
#pragma unroll 3
  for (int k = 0; k < 9; k++) {
    // q r0 2^62, rounded; its product with omega at 2^61
    const fx_t b = fx_mul((fxu_t)fx_round(fx_mul((fxu_t)s64.q[k][t], R)), k == 0 ? Om << 4 : (k <= 4 ? Om << 2 : Om));
    // |f om1| at 2^(1085 - e1), rounded, then at 2^61
    const fx_t a = fx_round(fx_mul((fxu_t)s64.f[k][t] << 2, M1));
    const fx_t a1 = (fx_t)((fxu_t)a >> s1) | (fx_t)(((unsigned)a & low1) != 0u);
    const fx_t s = fx_round(b) + (a1 ^ sign1) + (sign1 & 1);
    const double d = s64.drive[k][t];
    const fx_t sign = __double2hiint(d) >> 31;
    const fx_t v = fx_round(s) + (fx_abs(d) ^ sign) + (sign & 1);
    least = min(least, min((int)(b >> 32), min((int)(s >> 32), (int)(v >> 32))));
    s64.q[k][t] = __double_as_longlong(fx_double(v));
  }
  return least >= 1 << 22;
}

// BGK collision with the Guo forcing term, velocity shifted by beta/(2 rho)
// (streamCollCompute.cpp:28-37), every value the reference's, bit for bit.
// wcb[k] = (w[k]*(1 - omega/2))*beta.  The reference evaluates c_k.u, the
// equilibrium and the drive 3 (cx - ux) + 9 cx eu direction by direction;
// here what differs between directions in sign only is formed once: c_k.u of
// opposite directions, 3 ux (the drive's of cx = 0), 3 (1 + ux) (minus the
// drive's of cx = -1), the products w rho: 147 FP64 operations a node (about
// 205 direction by direction, with three divisions).  Where the values are of
// ordinary size the sums and the products of the relaxation, 81 of them, go to
// the integer pipes (moments64, feq_pair_fx, relax_fx), elsewhere, a warp at a
// time, they stay FP64.  256 clones of 256x64, us a step: 1540 direction by
// direction, 1192 by pairs, 768 with the sums in fixed point, 731 with the
// products too, 545 with the node in shared memory and loops over directions
// (3 unrolled; 615 unrolled in full, which waits for instructions), 534 with
// fx_place; 498 with the drag's terms in other blocks, 479 with 3 e, 4 wcb[1] and
// the signed sums' conversion off the FP64 pipe too: 55 operations are left to
// it, it is busy 75% of the time (back-to-back products reach 86%) and the integer
// ALU 71%, so that what is moved from one to the other gains no more.
// At one clone of 129x129 (four warps an SM) the chain of dependent operations
// bounds a step whatever the pipe: 10.05 us with the sums in fixed point, 10.3 in
// this form.
// s and m: the node and moments64 of it.
template <int BLOCK>
__device__ __forceinline__ void collide_ref64(Node64<BLOCK> &s, const Moments64 &m, double out[9], double half_beta,
                                              const double wcb[9], double omega,
                                              double om1, double *ux_o = nullptr, double *uy_o = nullptr) {
  double ux, uy;
  velocity_ref64(m, half_beta, ux, uy);
  const double u2 = DMUL(-1.5, DADD(DMUL(ux, ux), DMUL(uy, uy)));
  const double es = DADD(ux, uy), ed = DSUB(ux, uy);  // c_5.u = -c_7.u, c_8.u = -c_6.u
  const double t3x = DMUL(3.0, ux);
  const double hx = DMUL(4.5, ux), hs = DMUL(4.5, es), hd = DMUL(4.5, ed);
  const double eex = DMUL(hx, ux), eey = DMUL(DMUL(4.5, uy), uy), ees = DMUL(hs, es), eed = DMUL(hd, ed);
  // 9 eu = 2 (4.5 eu), rounding included, so its sum with the rest of the
  // drive is one fused operation on an exact product
  const double right = DMUL(3.0, DSUB(1.0, ux)), left = DMUL(3.0, DADD(1.0, ux));
  double (*drive)[BLOCK] = s.drive;
  const int t = threadIdx.x;
  const double up = DMUL(wcb[1], -t3x);
  drive[2][t] = drive[4][t] = up;
  // wcb[0] is four times wcb[1], and so are the products where neither they nor
  // wcb are at the ends of the exponent range
  drive[0][t] = mid_range64(up) && up != 0.0 && mid_range64(wcb[1])
                    ? __hiloint2double(__double2hiint(up) + 0x200000, __double2loint(up))
                    : DMUL(wcb[0], -t3x);
  drive[1][t] = DMUL(wcb[1], __fma_rn(2.0, hx, right));
  drive[5][t] = DMUL(wcb[5], __fma_rn(2.0, hs, right));
  drive[8][t] = DMUL(wcb[5], __fma_rn(2.0, hd, right));
  drive[3][t] = DMUL(wcb[1], __fma_rn(2.0, hx, -left));
  drive[7][t] = DMUL(wcb[5], __fma_rn(2.0, hs, -left));
  drive[6][t] = DMUL(wcb[5], __fma_rn(2.0, hd, -left));
  const double r0 = DMUL(w_of(0), m.rho);
  if (ux_o) *ux_o = ux;
  if (uy_o) *uy_o = uy;
  if (m.mid) {
    // |u| below 0.1484, r0 in [1/4, 1/2), drives below 1/2, omega in [1/16, 2),
    // |om1| in [2^-29, 1) or zero
    unsigned top = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) top = max(top, (unsigned)__double2hiint(drive[k][t]) & 0x7fffffffu);
    const unsigned o1 = (unsigned)__double2hiint(om1) & 0x7fffffffu;
    if (warp_all(max((unsigned)__double2hiint(ux) & 0x7fffffffu, (unsigned)__double2hiint(uy) & 0x7fffffffu) < 0x3fc30000u &&
                 (unsigned)__double2hiint(r0) - 0x3fd00000u < 0x100000u && top < 0x3fe00000u &&
                 (unsigned)__double2hiint(omega) - 0x3fb00000u < 0x500000u &&
                 (o1 - 0x3e200000u < 0x1d00000u || om1 == 0.0))) {
      fx_t (*q)[BLOCK] = s.q;
      const fx_t u = fx_abs(u2);
      q[0][t] = fx_round(FX_ONE - u);
      q[1][t] = __double_as_longlong(ux), q[3][t] = __double_as_longlong(eex);
      q[2][t] = __double_as_longlong(uy), q[4][t] = __double_as_longlong(eey);
      q[5][t] = __double_as_longlong(es), q[7][t] = __double_as_longlong(ees);
      q[8][t] = __double_as_longlong(ed), q[6][t] = __double_as_longlong(eed);
      column_fence();
#pragma unroll 1
      for (int j = 0; j < 4; j++) {
        const int kp = j < 2 ? j + 1 : 3 * j - 1, km = j < 2 ? j + 3 : 9 - j;
        fx_t plus, minus;
        feq_pair_fx(__longlong_as_double(q[kp][t]), __longlong_as_double(q[km][t]), u, plus, minus);
        q[kp][t] = plus;
        q[km][t] = minus;
      }
      if (warp_all(relax_fx(s, r0, omega, om1))) {
#pragma unroll
        for (int k = 0; k < 9; k++) out[k] = __longlong_as_double(q[k][t]);
        return;
      }
    }
  }
  double q[9];
  q[0] = DADD(1.0, u2);
  feq_pair_ref64(t3x, eex, u2, q[1], q[3]);
  feq_pair_ref64(DMUL(3.0, uy), eey, u2, q[2], q[4]);
  feq_pair_ref64(DMUL(3.0, es), ees, u2, q[5], q[7]);
  feq_pair_ref64(DMUL(3.0, ed), eed, u2, q[8], q[6]);
  const double r1 = DMUL(w_of(1), m.rho), r5 = DMUL(w_of(5), m.rho);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double feq = DMUL(k == 0 ? r0 : (k <= 4 ? r1 : r5), q[k]);
    out[k] = DADD(DADD(DMUL(node_f(s, m.mid, k), om1), DMUL(feq, omega)), drive[k][t]);
  }
}

// Non-equilibrium second moments with the UNshifted velocity
// (force.cpp:26-46): pi_xx = sum fneq cx cx, pi_xy = sum fneq cx cy, m the
// moments of f.  (FP64 sums: the perimeter's few warps leave the FP64 pipe
// free, and the fixed-point chain is the longer one.)
__device__ __forceinline__ void pi_ref64(const double f[9], const Moments64 &m, double &pxx,
                                         double &pxy) {
  const Divisor64 d = divisor64(m.rho);
  const bool fast = d.ok && mid_range64(m.jx) && mid_range64(m.jy);
  const double uy = fast ? div64(m.jy, d) : DDIV(m.jy, m.rho);
  const double ux = fast ? div64(m.jx, d) : DDIV(m.jx, m.rho);
  const double u2 = DMUL(-1.5, DADD(DMUL(ux, ux), DMUL(uy, uy)));
  const double es = DADD(ux, uy), ed = DSUB(ux, uy);
  double q[9];
  feq_pair_ref64(DMUL(3.0, ux), DMUL(DMUL(4.5, ux), ux), u2, q[1], q[3]);
  feq_pair_ref64(DMUL(3.0, es), DMUL(DMUL(4.5, es), es), u2, q[5], q[7]);
  feq_pair_ref64(DMUL(3.0, ed), DMUL(DMUL(4.5, ed), ed), u2, q[8], q[6]);
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
