// FP64 face evaluation of the fused stage kernels: the same values, bit for
// bit, as the plain expressions of fv_numerics.cuh, with the divisions
// arranged for the FP64 pipe.
//
// A face takes 28 divisions (two per limited variable and side, the
// primitives, the Mach numbers).  Written as `/` each is a reciprocal
// sequence of its own behind a test and a call for operands outside the
// normal range, and a zero numerator (a difference of equal cells: every
// uniform region, every direction a flow does not vary in) takes the call.
// The tests also keep the compiler from overlapping the divisions' dependent
// chains.  Here
//   - a quotient is a few dependent multiply-adds without a branch: zero
//     numerators need nothing special, and the twenty limiter divisions of a
//     face overlap;
//   - quotients with one denominator (u, v, w and H by the density; both
//     Mach numbers by the face's speed of sound) share its reciprocal, and
//     the constant 1/cv is a literal;
//   - operands for which the sequence is not proven exact are noted in a
//     Guard, and a face with any of them is evaluated again by the plain
//     expressions (out of line; a face in some 2e4 for the reciprocal's
//     excluded denominators, no other for flows in any usual range).
//
// Exactness (after Markstein's theorems: P. Markstein, IBM J. Res. Dev. 34,
// 1990; J.-M. Muller et al., Handbook of Floating-Point Arithmetic, ch. 4).
// A quotient q within one ulp of a/b with its exact residual r = a - b q
// gives fl(q + r y) = the correctly rounded a/b unless the error of r y
// reaches the distance of a/b from a midpoint of two doubles.  That distance
// is at least 2^-53/m ulp, m in [1, 2) the significand of b; next to a
// midpoint |a/b - q| is half an ulp, so |b y - 1| < 2^-52/m is enough.
// Recip's y is y0 (1 + e + e^2 + e^3), e = 1 - b y0, rounded: |b y - 1| <=
// m 2^-54 + |e| 2^-53 + e^4 (half an ulp of y, the rounding of the polynomial,
// its truncation).  With m = 2 (1 - n) both hold where n > |e|/2 + 2^52 e^4.
// y0 is PTX's rcp.approx.ftz.f64.  Its |e|, a function of the upper significand
// field but for the exact product, is at most 2^-19.94 over all fields on the
// B200 and 2^-20.95 where the upper 12 bits are ones.  Guard takes out the
// denominators whose upper 20 significand bits are ones, n <= 2^-21, and the
// bound asks for n > 2^-21.95 next to them and n > 2^-20.93 anywhere
// (tests/f64_seed.cu goes through every field).  18 bits would cover |e| up to
// 2^-19 at any denominator, but a waiting CTA pays for the fallback: 64^3 59.5
// -> 61.7 us a stage, 128^3 389.0 -> 391.5.  The first quotient a y is within
// 1.5 ulp, one residual step makes it faithful, the second correctly rounds it.
//
// G cell-updates/s a stage of a periodic 192^3 AUSM+ patch on the B200: 2.57
// with `/`, 4.02 with these quotients, 5.66 with one copy of the face code too
// (fv_stage_tile).
#pragma once

#include "fv_numerics.cuh"

namespace dn {

#ifdef __CUDACC__   // (a host test of this arithmetic restates the two instructions)
// largest of three floats, NaN if any is
__device__ __forceinline__ float max_nan(float a, float b, float c)
{
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(a) : "f"(a), "f"(b), "f"(c));
  return a;
}
// approximate reciprocal from the upper 32 bits
__device__ __forceinline__ double rcp_seed(double b)
{
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
}
#endif

// What a thread's fast evaluation must not be trusted for.  The extrema of
// high words (exponent and upper significand) are accumulated and judged
// once per face.
struct Guard {
  static constexpr int exp_hi(int e) { return (1023 + e) << 20; }   // high word of 2^e
  unsigned mant = 0;           // largest upper-significand field of a denominator
  float dmax = 0.0f;           // largest |difference|: its high word read as a float (same order; NaN stays)
  unsigned zmin = 0xffffffffu; // smallest nonzero numerator (high word - 1: zero wraps to the top)
  int lo = 0x7fffffff, hi = 0; // extrema of what must be positive
  bool minus_zero = false;     // a difference of -0 (or a denormal next to it)
  __device__ __forceinline__ void den(double b) { mant = max(mant, (unsigned)__double2hiint(b) & 0xfffffu); }
  __device__ __forceinline__ void diff(double x, double y)
  {
    dmax = max_nan(dmax, fabsf(__int_as_float(__double2hiint(x))), fabsf(__int_as_float(__double2hiint(y))));
  }
  __device__ __forceinline__ void num(double x) { zmin = min(zmin, ((unsigned)__double2hiint(x) & 0x7fffffffu) - 1u); }
  __device__ __forceinline__ void positive(double x)
  {
    lo = min(lo, __double2hiint(x));
    hi = max(hi, __double2hiint(x));
  }
  // trusted: denominators whose upper 20 significand bits are not all ones, numerators
  // above 2^-500, differences below 2^400 over denominators of at least 1e-10,
  // positive quantities in [2^-300, 2^300] (NaN is outside)
  __device__ __forceinline__ bool any() const
  {
    return mant == 0xfffffu || !(dmax < __int_as_float(exp_hi(400))) || zmin < (unsigned)exp_hi(-500) ||
           lo < exp_hi(-300) || hi >= exp_hi(300) || minus_zero;
  }
};

// x * 2^n by its exponent field (x normal, result normal)
__device__ __forceinline__ double scale2(double x, int n)
{
  return __hiloint2double(__double2hiint(x) + n * 0x100000, __double2loint(x));
}

// A denominator with its reciprocal y.
struct Recip {
  double b, y;
  __device__ __forceinline__ Recip(double d, Guard& g) : b(d)
  {
    g.den(d);
    const double y0 = rcp_seed(d);
    const double e = __fma_rn(-d, y0, 1.0);
    const double t = __fma_rn(__fma_rn(e, e, e), e, e);
    y = __fma_rn(y0, t, y0);
  }
  __device__ __forceinline__ constexpr Recip(double d, double inv) : b(d), y(inv) {}
  // a / b (a zero or in the guarded range; a zero quotient may come out as +0)
  __device__ __forceinline__ double quot(double a) const
  {
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
  }
  // 1 / b
  __device__ __forceinline__ double inverse() const { return __fma_rn(__fma_rn(-b, y, 1.0), y, y); }
};

// Half the van Albada limiter values (van_albada) of N pairs of differences,
// exact halving included: 0.5 * (r*r + r) / (r*r + 1), r = d2 / non_zero(d1,
// 1e-10).  The pairs advance step by step together, so that N dependent
// chains overlap.
template <int N>
__device__ __forceinline__ void half_van_albada(const double (&d1)[N], const double (&d2)[N], double (&out)[N], Guard& g)
{
  // non_zero: |d1| < eps becomes eps with the sign of d1 (-0, which counts as
  // positive, is left to the guard)
  constexpr unsigned long long eps = 0x3ddb7cdfd9d7bdbbull;     // 1e-10
  double b[N], y[N], e[N], q[N], num[N];
  #pragma unroll
  for (int c = 0; c < N; ++c) {
    const int h = __double2hiint(d1[c]);
    g.minus_zero |= h == (int)0x80000000;
    if (c & 1) g.diff(d1[c], d1[c - 1]);
    const bool small = fabs(d1[c]) < 1e-10;
    b[c] = __hiloint2double(small ? ((int)(eps >> 32) | (h & (int)0x80000000)) : h,
                            small ? (int)(unsigned)eps : __double2loint(d1[c]));
    g.den(b[c]);
    y[c] = rcp_seed(b[c]);
  }
  // r = d2 / b (Recip)
  #pragma unroll
  for (int c = 0; c < N; ++c) e[c] = __fma_rn(-b[c], y[c], 1.0);
  #pragma unroll
  for (int c = 0; c < N; ++c) q[c] = __fma_rn(e[c], e[c], e[c]);
  #pragma unroll
  for (int c = 0; c < N; ++c) e[c] = __fma_rn(q[c], e[c], e[c]);
  #pragma unroll
  for (int c = 0; c < N; ++c) y[c] = __fma_rn(y[c], e[c], y[c]);
  #pragma unroll
  for (int c = 0; c < N; ++c) q[c] = __dmul_rn(d2[c], y[c]);
  #pragma unroll
  for (int n = 0; n < 2; ++n) {
    #pragma unroll
    for (int c = 0; c < N; ++c) e[c] = __fma_rn(-b[c], q[c], d2[c]);
    #pragma unroll
    for (int c = 0; c < N; ++c) q[c] = __fma_rn(e[c], y[c], q[c]);
  }
  // num / den with everything scaled so that the quotient comes out halved:
  // the residual of half the quotient against 2 den is that of the quotient,
  // and times y/2 it corrects the half
  #pragma unroll
  for (int c = 0; c < N; ++c) {
    const double rr = __dmul_rn(q[c], q[c]);
    num[c] = __dadd_rn(rr, q[c]);
    b[c] = __dadd_rn(rr, 1.0);
    g.den(b[c]);
    y[c] = rcp_seed(b[c]);
  }
  #pragma unroll
  for (int c = 0; c < N; ++c) e[c] = __fma_rn(-b[c], y[c], 1.0);
  #pragma unroll
  for (int c = 0; c < N; ++c) q[c] = __fma_rn(e[c], e[c], e[c]);
  #pragma unroll
  for (int c = 0; c < N; ++c) e[c] = __fma_rn(q[c], e[c], e[c]);
  #pragma unroll
  for (int c = 0; c < N; ++c) {
    y[c] = scale2(y[c], -1);
    b[c] = scale2(b[c], 1);
  }
  #pragma unroll
  for (int c = 0; c < N; ++c) y[c] = __fma_rn(y[c], e[c], y[c]);
  #pragma unroll
  for (int c = 0; c < N; ++c) q[c] = __dmul_rn(num[c], y[c]);
  #pragma unroll
  for (int n = 0; n < 2; ++n) {
    #pragma unroll
    for (int c = 0; c < N; ++c) e[c] = __fma_rn(-b[c], q[c], num[c]);
    #pragma unroll
    for (int c = 0; c < N; ++c) q[c] = __fma_rn(e[c], y[c], q[c]);
  }
  #pragma unroll
  for (int c = 0; c < N; ++c) out[c] = q[c];
}

// Where a face reads its cells: cells c-2, c-1 | c, c+1 of variable v at
// m2[v*s2], m1[v*S], p0[v*S], p1[v*S] for the plane variable stride S.  sl,
// sr: cells c-2 and c+1 exist; where one does not, m2 or p1 points to the
// cell next to it again, which makes that side's slope zero (the reference's
// first-order state).
struct FaceCells {
  const double *m2, *m1, *p0, *p1;
  int s2;
  bool sl, sr;
};

// Limited states of both sides of a face.
template <int S>
__device__ __forceinline__ void limited_states(const FaceCells& f, double vl[5], double vr[5], Guard& g)
{
  double d1[10], d2[10], h[10];
  #pragma unroll
  for (int v = 0; v < 5; ++v) {
    vl[v] = f.m1[v * S];
    vr[v] = f.p0[v * S];
    const double d = __dsub_rn(vr[v], vl[v]);
    d1[2 * v] = __dsub_rn(vl[v], f.m2[v * f.s2]);
    d1[2 * v + 1] = __dsub_rn(vr[v], f.p1[v * S]);
    d2[2 * v] = d;
    d2[2 * v + 1] = -d;
    g.num(d);
  }
  g.diff(d2[0], d2[2]);
  g.diff(d2[4], d2[6]);
  g.diff(d2[8], d2[8]);
  half_van_albada(d1, d2, h, g);
  #pragma unroll
  for (int v = 0; v < 5; ++v) {
    vl[v] = __dadd_rn(vl[v], __dmul_rn(h[2 * v], d1[2 * v]));
    vr[v] = __dadd_rn(vr[v], __dmul_rn(h[2 * v + 1], d1[2 * v + 1]));
  }
}

// Primitive face-side state (face_side); d is the reciprocal of its density.
__device__ __forceinline__ FaceSide<double> face_side_fast(const double var[5], const Recip& d, Guard& g)
{
  FaceSide<double> s;
  const double r = var[0], rE = var[4];
  g.positive(r);
  const double ir = d.inverse();
  const double u = __dmul_rn(var[1], ir), v = __dmul_rn(var[2], ir), w = __dmul_rn(var[3], ir);
  const double ke = __dadd_rn(__dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)), __dmul_rn(w, w));
  const double t = __fma_rn(-0.5, ke, __dmul_rn(rE, ir));       // the product 0.5 * ke is exact
  g.positive(t);
  constexpr double icv = 1.0 / Gas::cv;
  const double Tt = Recip(Gas::cv, icv).quot(t);
  const double p = __dmul_rn(__dmul_rn(r, Gas::R), Tt);
  constexpr double gR = Gas::gamma * Gas::R;
  const double a = sqrt(__dmul_rn(gR, Tt));
  const double h = __dadd_rn(rE, p);
  g.positive(h);
  s.r = r; s.u = u; s.v = v; s.w = w; s.p = p; s.a = a;
  s.H = d.quot(h);
  return s;
}

// AUSM split Mach number and pressure polynomials of one side (ausm_m4,
// ausm_p5), S = +1 or -1, both branches selected: for |M| >= 1 the
// reference's M1/M is exactly 1 or 0.
template <int S>
__device__ __forceinline__ void ausm_split_fast(double M, double& m4, double& p5)
{
  const int h = __double2hiint(M);
  const bool outer = (h & 0x7fffffff) >= 0x3ff00000;
  const bool toward = S > 0 ? h >= 0 : h < 0;            // S M > 0 (M = 0 is not outer)
  const double q = __dadd_rn(M, (double)S), qo = __dadd_rn(M, (double)-S);
  const double m2 = __dmul_rn(0.25 * S, __dmul_rn(q, q));
  const double m2o = __dmul_rn(-0.25 * S, __dmul_rn(qo, qo));
  // 2 s m2o is exact, so 1 - 2 s m2o rounds once
  const double in4 = __dmul_rn(m2, __fma_rn(-2.0 * S, m2o, 1.0));
  const double in5 = __dmul_rn(m2, __dsub_rn(__dsub_rn(2.0 * S, M), __dmul_rn(__dmul_rn(3.0 * S, M), m2o)));
  m4 = outer ? (toward ? M : 0.0) : in4;
  p5 = outer ? (toward ? 1.0 : 0.0) : in5;
}

// AUSM+ face flux (ausm_plus) with normal along axis dir.
__device__ __forceinline__ void ausm_plus_fast(int dir, const FaceSide<double>& L, const FaceSide<double>& Rs, double A,
                                               double flux[5], Guard& g)
{
  const double un_l = dir == 0 ? L.u : (dir == 1 ? L.v : L.w);
  const double un_r = dir == 0 ? Rs.u : (dir == 1 ? Rs.v : Rs.w);
  const double a = __dmul_rn(0.5, __dadd_rn(L.a, Rs.a));
  g.positive(a);
  g.num(un_l);
  g.num(un_r);
  const Recip d(a, g);
  double m4l, p5l, m4r, p5r;
  ausm_split_fast<1>(d.quot(un_l), m4l, p5l);
  ausm_split_fast<-1>(d.quot(un_r), m4r, p5r);
  const double M = __dadd_rn(m4l, m4r);
  const double p = __dadd_rn(__dmul_rn(p5l, L.p), __dmul_rn(p5r, Rs.p));
  // one of the split mass fluxes' Mach numbers (M + |M|)/2, (M - |M|)/2 is M, the other 0
  const double rM = __dmul_rn(M > 0.0 ? L.r : Rs.r, M == 0.0 ? 0.0 : M);
  const double f0 = __dmul_rn(__dmul_rn(a, A), rM);
  const double h0 = __dmul_rn(0.5, f0);
  const double g0 = fabs(h0);
  const double Ap = __dmul_rn(A, p);
  const double pu = __dmul_rn(h0, __dadd_rn(L.u, Rs.u)), du = __dmul_rn(g0, __dsub_rn(Rs.u, L.u));
  const double pv = __dmul_rn(h0, __dadd_rn(L.v, Rs.v)), dv = __dmul_rn(g0, __dsub_rn(Rs.v, L.v));
  const double pw = __dmul_rn(h0, __dadd_rn(L.w, Rs.w)), dw = __dmul_rn(g0, __dsub_rn(Rs.w, L.w));
  const double ph = __dmul_rn(h0, __dadd_rn(L.H, Rs.H)), dh = __dmul_rn(g0, __dsub_rn(Rs.H, L.H));
  flux[0] = f0;
  flux[1] = __dsub_rn(dir == 0 ? __dadd_rn(pu, Ap) : pu, du);
  flux[2] = __dsub_rn(dir == 1 ? __dadd_rn(pv, Ap) : pv, dv);
  flux[3] = __dsub_rn(dir == 2 ? __dadd_rn(pw, Ap) : pw, dw);
  flux[4] = __dsub_rn(ph, dh);
}

// The AUSM+ scheme as the stage kernel takes it: the flux of a face with
// normal along axis dir from its limited states, fast with a guard, and
// plain.
struct AusmPlusFace {
  static __device__ __forceinline__ void fast(int dir, const double vl[5], const double vr[5], double A, double F[5],
                                              Guard& g)
  {
    ausm_plus_fast(dir, face_side_fast(vl, Recip(vl[0], g), g), face_side_fast(vr, Recip(vr[0], g), g), A, F, g);
  }
  template <int DIR>
  static __device__ __forceinline__ void plain(const double vl[5], const double vr[5], double A, double F[5])
  {
    ausm_plus<DIR>(face_side(vl), face_side(vr), A, F);
  }
};

// A face by the plain expressions, out of line.
template <class Scheme, int S>
__device__ __noinline__ void face_flux_plain(int dir, const FaceCells& c, double A, double* F)
{
  double vl[5], vr[5];
  for (int v = 0; v < 5; ++v) {
    const double a = c.m1[v * S], b = c.p0[v * S];
    vl[v] = upwind2_left(c.m2[v * c.s2], a, b, c.sl);
    vr[v] = upwind2_right(a, b, c.p1[v * S], c.sr);
  }
  if (dir == 0) Scheme::template plain<0>(vl, vr, A, F);
  else if (dir == 1) Scheme::template plain<1>(vl, vr, A, F);
  else Scheme::template plain<2>(vl, vr, A, F);
}

// Flux through a face with normal along axis dir.
template <class Scheme, int S>
__device__ __forceinline__ void face_flux(int dir, const FaceCells& c, double A, double F[5])
{
  Guard g;
  double vl[5], vr[5];
  limited_states<S>(c, vl, vr, g);
  Scheme::fast(dir, vl, vr, A, F, g);
  if (g.any()) {
    double f[5];
    const FaceCells d = c;
    face_flux_plain<Scheme, S>(dir, d, A, f);
    for (int v = 0; v < 5; ++v) F[v] = f[v];
  }
}

} // namespace dn
