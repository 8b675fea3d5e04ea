// Device-side pointwise physics of the second-order (PLM) MHD path, FP64.
//
// Each function restates one piece of the reference for sm_100a: scalar
// registers instead of 8x8 arrays, structural zeros of the Roe eigenvectors
// skipped (adding an exact zero term does not change an IEEE sum of finite
// values), matrix entries kept as the reference writes them.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <math_constants.h>

#include "hc_common.h"

#define HC_DEV __device__ __forceinline__

namespace hc {

// Level kernels loop over flat indices below 2^31 (hc_ctx_create bounds
// the level size), so their loops and index splits run in 32-bit unsigned
// arithmetic.  takeMod returns t mod n and leaves t / n in t.
HC_DEV unsigned takeMod(unsigned& t, unsigned n) {
  const unsigned q = t / n, r = t - q * n;
  t = q;
  return r;
}
#define HC_LEVEL_LOOP(t, n) for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < (n); t += gridDim.x * blockDim.x)

HC_DEV double dmin(double a, double b) { return b < a ? b : a; }  // std::min
HC_DEV double dmax(double a, double b) { return a < b ? b : a; }  // std::max

// A double whose sums and products round exactly as written: the compiler
// may contract a plain a * b + c into one fused operation or not, and does
// so differently from kernel to kernel and with the register cap, while
// results must not depend on the tile or the batch a face is computed in.
// Fused operations are asked for with mad.
struct Rn {
  double v;
  HC_DEV Rn(double x) : v(x) {}
  HC_DEV Rn() {}
  HC_DEV operator double() const { return v; }
};
HC_DEV Rn operator+(Rn a, Rn b) { return __dadd_rn(a.v, b.v); }
HC_DEV Rn operator-(Rn a, Rn b) { return __dsub_rn(a.v, b.v); }
HC_DEV Rn operator*(Rn a, Rn b) { return __dmul_rn(a.v, b.v); }
HC_DEV Rn operator-(Rn a) { return -a.v; }
HC_DEV Rn operator+(Rn a, double b) { return a + Rn(b); }
HC_DEV Rn operator+(double a, Rn b) { return Rn(a) + b; }
HC_DEV Rn operator-(Rn a, double b) { return a - Rn(b); }
HC_DEV Rn operator-(double a, Rn b) { return Rn(a) - b; }
HC_DEV Rn operator*(Rn a, double b) { return a * Rn(b); }
HC_DEV Rn operator*(double a, Rn b) { return Rn(a) * b; }
HC_DEV Rn mad(Rn a, Rn b, Rn c) { return fma(a.v, b.v, c.v); }
HC_DEV Rn dot3(Rn a0, Rn b0, Rn a1, Rn b1, Rn a2, Rn b2) { return mad(a2, b2, mad(a1, b1, a0 * b0)); }

// Reciprocal and reciprocal square root by one third-order (Halley) step of
// the residual from the hardware's approximate seed: with e = 1 - x y,
// 1 / x = y (1 + e + e^2 + O(e^3)); with e = 1 - x y^2,
// 1 / sqrt(x) = y (1 + e/2 + 3 e^2/8 + O(e^3)).  The seed is good to 20
// bits, so the errors stay below 1.01 and 1.53 units of 2^-53, in four and six
// FP64 operations where a correctly rounded division or square root takes
// ten and more behind a range branch.  x must be normal (the callers'
// operands are physical magnitudes kept away from 0); a zero, subnormal or
// non-finite x gives a non-finite result.
HC_DEV double rcpN(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// 1 / rho of a density: 0 for infinity, as the division gives.
HC_DEV double rcpDensity(double rho) { return rho == CUDART_INF ? 0.0 : rcpN(rho); }
HC_DEV double rsqrtN(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(__dmul_rn(-x, y), y, 1.0);
  return fma(__dmul_rn(y, e), fma(0.375, e, 0.5), y);
}
// sqrt(x) with one Newton correction of x rsqrt(x) (good to the last bit).
// 0 for x below 1e-290 (far below any squared speed), negative ones
// included; infinity and NaN are returned as they are, so an infinite speed
// stays infinite.
HC_DEV double sqrtN(double x) {
  const double y = rsqrtN(x), s = __dmul_rn(x, y);
  const double root = fma(0.5 * y, fma(-s, s, x), s);
  return x <= 1e-290 ? 0.0 : (x < CUDART_INF ? root : x);
}

// Half the limited slope of a cell with differences a, b to its neighbours
// (src/BoxOp_SecondOrder.H:7-37).  LIM: 0 unlimited, 1 minmod (limiter 1 or
// 2), 3 monotonized central: the smaller of |a + b| / 4 and min(|a|, |b|)
// with the differences' sign, 0 where they differ in sign.  The candidates
// keep their signs through the selection, so no sign is taken off and put
// back.  Where the product of the differences is NaN the reference takes
// std::min / std::max of the two: NaN for a NaN a, a for a NaN b (a NaN cell
// does not reach past the faces next to it), and of 0 and an infinity 0, but
// infinity for 0 and +inf.  That value (odd) is formed for every face with one
// product and an integer selection, ahead of the choice: from comparisons, in
// a branch, or inside the choice it made the second-order steps 4 to 37 %
// slower.
template <int LIM>
HC_DEV Rn halfSlope(Rn a, Rn b) {
  const Rn q = 0.25 * (a + b);
  if (LIM == 0) return q;
  const double small = fabs(b.v) < fabs(a.v) ? b.v : a.v;
  const double t = LIM == 1 ? 0.5 * small : (fabs(small) < fabs(q.v) ? small : q.v);
  const double sign = a * b;
  const double h = 0.5 * small;
  const double odd =
      __hiloint2double(__double2hiint(b.v) == 0x7ff00000 ? 0x7ff00000 : __double2hiint(h), __double2loint(h));
  return sign > 0.0 ? t : (sign <= 0.0 ? 0.0 : odd);
}

// Left and right states of a face from its four cells, one component.
template <int LIM>
HC_DEV void plmComponent(double mm, double m, double c, double p, double& lo, double& hi) {
  const Rn a = Rn(m) - mm, b = Rn(c) - m, d = Rn(p) - c;
  lo = m + halfSlope<LIM>(a, b);
  hi = c - halfSlope<LIM>(b, d);
}

// Left state of a face from cells (i-2, i-1, i) only (the "lo" half of the
// reference's pair), with its complete-state fallback.
template <int LIM>
HC_DEV void plmLeft(const double* mm, const double* m, const double* c, double lo[8]) {
#pragma unroll
  for (int k = 0; k < NC; ++k) lo[k] = m[k] + halfSlope<LIM>(Rn(m[k]) - mm[k], Rn(c[k]) - m[k]);
  if (!(lo[0] >= kRHO00 && lo[4] >= 0)) {
#pragma unroll
    for (int k = 0; k < NC; ++k) lo[k] = m[k];
  }
}

// Right state of a face from cells (i-1, i, i+1) only.
template <int LIM>
HC_DEV void plmRight(const double* m, const double* c, const double* p, double hi[8]) {
#pragma unroll
  for (int k = 0; k < NC; ++k) hi[k] = c[k] - halfSlope<LIM>(Rn(c[k]) - m[k], Rn(p[k]) - c[k]);
  if (!(hi[0] >= kRHO00 && hi[4] >= 0)) {
#pragma unroll
    for (int k = 0; k < NC; ++k) hi[k] = c[k];
  }
}

// src/MHD_Roe8Wave.H:604-629.  invGm1 = 1/(gamma-1) replaces the division
// by (gamma-1) (one rounding of difference, inside the parity tolerance);
// sqrt(x / rho) is x / sqrt(x rho), one reciprocal root.
HC_DEV void rusanovDissipation(double out[8], const double* wl, const double* wr, double gamma, double invGm1) {
  constexpr double inv4Pi = 0.079577471545947667884441881686257181;
  Rn energy[2];
  double speed = 0.0;
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const double* w = side == 0 ? wl : wr;
    const Rn v2 = dot3(w[1], w[1], w[2], w[2], w[3], w[3]), b2 = dot3(w[5], w[5], w[6], w[6], w[7], w[7]);
    energy[side] = mad(0.5 * inv4Pi, b2, mad(0.5 * Rn(w[0]), v2, Rn(w[4]) * invGm1));
    const Rn x = mad(inv4Pi, b2, gamma * Rn(w[4])), xr = x * w[0];
    const double fast = xr > 1e-290 && xr < CUDART_INF ? __dmul_rn(x, rsqrtN(xr)) : sqrt(x.v / w[0]);
    speed = fmax(speed, Rn(fabs(w[1])) + fast);
  }
  const Rn s = speed;
  out[0] = s * (Rn(wr[0]) - wl[0]);
  out[4] = s * (energy[1] - energy[0]);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    out[1 + d] = s * mad(wr[0], wr[1 + d], -(Rn(wl[0]) * wl[1 + d]));
    out[5 + d] = s * (Rn(wr[5 + d]) - wl[5 + d]);
  }
}

// src/MHD_Roe8Wave.H:16-600: D = |A|(U_R - U_L) with arithmetic averages,
// eight-wave entropy fix and (CHECK) the intermediate-state fan walk.
// Returns false where the reference requests the Rusanov fallback.
//
// The kernels that call it are bound by the FP64 pipe and by registers, so
// the solver is written to need few of both:
//  * With arithmetic averages the jumps of the primitive variables are exact
//    in closed form: the velocity jumps are the plain differences, and the
//    pressure jump is dp + (gamma - 1)/8 |dv|^2 drho (the sound speed's
//    pressure likewise mean p + |dB|^2 / 32 pi); the differences of large
//    energies of the conserved form, and their cancellation, drop out.
//  * The waves come in pairs +-: each pair shares an even and an odd part of
//    its strength and of its eigenvector.
//  * Transverse vectors are taken along t = (hyy, hzz) and n = (-hzz, hyy):
//    fast and slow waves have only t components, Alfven waves only n.
//  * The fan walk runs in the frame of the mean velocity and mean field,
//    where a wave changes five numbers (density, two momenta, one field
//    component, thermal energy): thermal energy is the same in every frame.
//    thermal >= 0 is tested as rho (e - b^2/8 pi) >= m^2 / 2, no division.
//  * Square roots and reciprocals by rsqrtN / rcpN.
// Measured on a B200 when it replaced the eigenvector matrices: second-order
// Roe step at 96 x 64^2 x 6 12.65 -> 7.34 ms (3.84 now, with the stage kernel's
// own changes); fourth-order Roe step at 64 x 64^2 x 6 13.96 -> 12.26 ms (9.9).
template <bool CHECK>
__device__ __forceinline__ bool roe8Body(double out[8], const double* wl, const double* wr, double gamma, double del2,
                                         double invHg) {
  const Rn RhoL = wl[0], PL = wl[4], RhoR = wr[0], PR = wr[4];
  if (!(RhoL > 0.0 && RhoR > 0.0 && PL > 0.0 && PR > 0.0)) return false;
  constexpr double k4 = 0.079577471545947667884441881686257181, k8 = 0.5 * k4, s2 = 0.707106781186547524400844362104849039;
  constexpr double sqPi = 1.772453850905516027298167483341145183, sq2Pi = 2.506628274631000502415765284811045253;
  constexpr double smallB2 = 1.0e-18;
  const Rn Rho = 0.5 * (RhoL + RhoR);
  const Rn U = 0.5 * (Rn(wl[1]) + wr[1]), V = 0.5 * (Rn(wl[2]) + wr[2]), W = 0.5 * (Rn(wl[3]) + wr[3]);
  const Rn BX = 0.5 * (Rn(wl[5]) + wr[5]), BY = 0.5 * (Rn(wl[6]) + wr[6]), BZ = 0.5 * (Rn(wl[7]) + wr[7]);
  const Rn dR = RhoL - RhoR, dU = Rn(wl[1]) - wr[1], dV = Rn(wl[2]) - wr[2], dW = Rn(wl[3]) - wr[3];
  const Rn dBX = Rn(wl[5]) - wr[5], dBY = Rn(wl[6]) - wr[6], dBZ = Rn(wl[7]) - wr[7];
  const Rn dv2 = dot3(dU, dU, dV, dV, dW, dW), db2 = dot3(dBX, dBX, dBY, dBY, dBZ, dBZ);
  const Rn dP = mad(0.125 * (gamma - 1.0) * dR, dv2, PL - PR);
  const Rn rs = rsqrtN(Rho), iRho = rs * rs, sqRho = Rho * rs;
  const Rn iLR = rcpN(RhoL * RhoR) * gamma, AL2 = PL * RhoR * iLR, AR2 = PR * RhoL * iLR;
  Rn cc = gamma * iRho * mad(0.25 * k8, db2, 0.5 * (PL + PR));
  {
    const Rn lo = AL2 > AR2 ? AR2 : AL2, hi = AL2 > AR2 ? AL2 : AR2;
    if (cc < lo) cc = lo;
    if (cc > hi) cc = hi;
  }
  if (!(cc > 0.0) || !isfinite(cc.v)) return false;
  const Rn rc = rsqrtN(cc), c = cc * rc, icc = rc * rc;
  const Rn b = fabs(BX.v) * (0.5 / sqPi) * rs, bb = b * b;
  const Rn BYZ2 = mad(BZ, BZ, BY * BY);
  Rn hyy = s2, hzz = s2, aaf = bb > cc ? bb : cc, aas = bb > cc ? cc : bb;
  if (!(BYZ2 < smallB2)) {
    const Rn rb = rsqrtN(BYZ2);
    hyy = BY * rb;
    hzz = BZ * rb;
    // The slow speed is a difference of nearly equal numbers where bb is
    // small; rounded as the reference rounds it (no fused product), so that
    // h = szb and the slow speed is 0 where bb vanishes.  A NaN of overflowed
    // squares counts as 0, as in the reference's maximum.
    const Rn szb = cc + (bb + k4 * BYZ2 * iRho);
    const Rn h = sqrtN(dmax(0.0, szb * szb - 4.0 * cc * bb));
    aas = 0.5 * (szb - h);
    aaf = 0.5 * (szb + h);
    if (aas <= 0.0) aas = 0.0;
    else if (aas >= cc) aas = cc;
    if (aaf <= cc) aaf = cc;
  }
  const Rn as = sqrtN(aas), af = sqrtN(aaf);
  const Rn dfs = aaf - aas;
  Rn alf = 1.0, als = 0.0;
  if (!(dfs < 1.0e-8)) {
    const Rn nf = cc - aas, ns = aaf - cc, idfs = rcpN(dfs);
    alf = nf <= 0.0 ? 0.0 : ns <= 0.0 ? 1.0 : sqrtN(nf * idfs);
    als = nf <= 0.0 ? 1.0 : ns <= 0.0 ? 0.0 : sqrtN(ns * idfs);
  }
  const double sih = BX >= 0.0 ? 1.0 : -1.0;
  // jumps along t and n
  const Rn tv = mad(hzz, dW, hyy * dV), nv = mad(hyy, dW, -(hzz * dV));
  const Rn tb = mad(hzz, dBZ, hyy * dBY), nb = mad(hyy, dBZ, -(hzz * dBY));
  // eigenvector entries: fast F*, slow S* (momentum entries times Rho, the
  // pressure entry over gamma - 1), Alfven GM (momentum) and GB (field)
  const Rn fa = alf * af, sa = als * as;
  const Rn F0 = Rho * alf, S0 = Rho * als, F1 = Rho * fa, S1 = Rho * sa, Ft = -(sih * S1), St = sih * F1;
  const Rn pe = cc * invHg, be = 2.0 * sqPi * sqRho * c, F4 = F0 * pe, S4 = S0 * pe, Fb = be * als, Sb = -(be * alf);
  const Rn GM = s2 * Rho, GB = -(sih * sq2Pi) * sqRho;
  // strengths (src/MHD_Roe8Wave.H:428-498)
  const Rn al0 = mad(-icc, dP, dR);
  const Rn oa = (-0.5 * sih / sq2Pi) * rs * nb, al2 = mad(s2, nv, oa), al3 = mad(s2, nv, -oa);
  const Rn w1 = 0.5 * icc, e1 = w1 * iRho * dP, m1 = (0.25 / sqPi) * (rc * rs) * tb, stv = sih * tv;
  const Rn ef = mad(als, m1, alf * e1), es = mad(-alf, m1, als * e1);
  const Rn of = w1 * mad(-sa, stv, fa * dU), os = w1 * mad(fa, stv, sa * dU);
  const Rn al4 = ef + of, al5 = ef - of, al6 = es + os, al7 = es - os;
  const Rn e2 = U + b, e3 = U - b, e4 = U + af, e5 = U - af, e6 = U + as, e7 = U - as;
  if (CHECK) {
    // Walk the wave fan in speed order 5, 3, 7, 0, 1, 6, 2, 4 from the left
    // state (src/MHD_Roe8Wave.H:500-548), amplitudes -alpha; a state between
    // two waves of one speed is not tested.
    const Rn hR = 0.5 * RhoL, bx2 = 0.25 * (dBX * dBX);
    Rn r = RhoL, mx = hR * dU, mt = hR * tv, mn = hR * nv, bt = 0.5 * tb, bn = 0.5 * nb;
    Rn th = mad(0.25 * k8, db2, mad(0.25 * hR, dv2, PL * invHg));
    bool ok = true;
    auto test = [&](bool distinct) {
      const Rn lhs = r * mad(-k8, mad(bn, bn, mad(bt, bt, bx2)), th);
      ok = ok && (!distinct || (r > 0.0 && lhs >= 0.5 * dot3(mx, mx, mt, mt, mn, mn)));
    };
    r = mad(-al5, F0, r); mx = mad(al5, F1, mx); mt = mad(al5, Ft, mt); th = mad(-al5, F4, th); bt = mad(-al5, Fb, bt);
    test(e3 > e5);
    mn = mad(-al3, GM, mn); bn = mad(al3, GB, bn);
    test(e7 > e3);
    r = mad(-al7, S0, r); mx = mad(al7, S1, mx); mt = mad(al7, St, mt); th = mad(-al7, S4, th); bt = mad(-al7, Sb, bt);
    test(U > e7);
    r = r - al0;  // the entropy and the divergence wave share the speed U; the latter takes dBX / 2 to -dBX / 2
    test(e6 > U);
    r = mad(-al6, S0, r); mx = mad(-al6, S1, mx); mt = mad(-al6, St, mt); th = mad(-al6, S4, th); bt = mad(-al6, Sb, bt);
    test(e2 > e6);
    mn = mad(-al2, GM, mn); bn = mad(-al2, GB, bn);
    test(e4 > e2);
    if (!ok) return false;
  }
  // Entropy-fixed |lambda| (src/MHD_Roe8Wave.H:243-311) times alpha.
  const Rn del = del2 * (Rn(fabs(U.v)) + fabs(V.v) + fabs(W.v) + af), del22 = del * del, idel = 0.5 * rcpN(del);
  auto lam = [&](Rn e) -> Rn {
    const double z = fabs(e.v);
    return z >= del ? Rn(z) : Rn(mad(z, z, del22) * idel);
  };
  const Rn l0 = lam(U), lu0 = l0 * al0, lu1 = l0 * dBX;
  const Rn p2 = lam(e2) * al2, p3 = lam(e3) * al3, p4 = lam(e4) * al4, p5 = lam(e5) * al5, p6 = lam(e6) * al6,
           p7 = lam(e7) * al7;
  const Rn Ap = p2 + p3, Am = p2 - p3, Fp = p4 + p5, Fm = p4 - p5, Sp = p6 + p7, Sm = p6 - p7;
  const Rn ra0 = mad(S0, Sp, mad(F0, Fp, lu0));
  const Rn R1 = mad(S1, Sm, F1 * Fm), Rt = mad(St, Sm, Ft * Fm), Rn_ = GM * Ap;
  const Rn Bt = mad(Sb, Sp, Fb * Fp), Bn = GB * Am;
  const Rn R2 = mad(-hzz, Rn_, hyy * Rt), R3 = mad(hyy, Rn_, hzz * Rt);
  const Rn r6 = mad(-hzz, Bn, hyy * Bt), r7 = mad(hyy, Bn, hzz * Bt);
  const Rn kk = 0.5 * dot3(U, U, V, V, W, W);
  out[0] = -ra0;
  out[1] = -mad(U, ra0, R1);
  out[2] = -mad(V, ra0, R2);
  out[3] = -mad(W, ra0, R3);
  out[4] = -(mad(kk, ra0, dot3(U, R1, V, R2, W, R3)) + mad(S4, Sp, F4 * Fp) + k4 * dot3(BX, lu1, BY, r6, BZ, r7));
  out[5] = -lu1;
  out[6] = -r6;
  out[7] = -r7;
  bool ok = true;
#pragma unroll
  for (int q = 0; q < 8; ++q) ok = ok && isfinite(out[q]);
  return ok;
}

// src/MHD_SecondOrderFlux.H:34-74: local-frame MHD flux of both states,
// Roe (with Rusanov fallback) or Rusanov dissipation, rotated back and
// multiplied by radialArea*|adjA|.
template <bool ROE>
HC_DEV void secondOrderFaceFlux(double out[8], const double* l, const double* r, const FaceGeom& g, double radialArea,
                                double gamma, double invGm1, double entropy) {
  constexpr double inv4pi = 1.0 / (4.0 * kPi);
  double loc[2][8];
  Rn flux[8];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const double* s = side == 0 ? l : r;
    double* q = loc[side];
    q[0] = s[0];
    q[4] = s[4];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      q[1 + i] = dot3(g.f[3 * i], s[1], g.f[3 * i + 1], s[2], g.f[3 * i + 2], s[3]);
      q[5 + i] = dot3(g.f[3 * i], s[5], g.f[3 * i + 1], s[6], g.f[3 * i + 2], s[7]);
    }
    const Rn v2 = dot3(q[1], q[1], q[2], q[2], q[3], q[3]), b2 = dot3(q[5], q[5], q[6], q[6], q[7], q[7]);
    const Rn vb = dot3(q[1], q[5], q[2], q[6], q[3], q[7]);
    const Rn magnetic = 0.5 * inv4pi * b2, pressure = magnetic + q[4];
    const Rn energy = mad(0.5 * Rn(q[0]), v2, mad(q[4], invGm1, magnetic));
    const Rn mass = Rn(q[0]) * q[1], bn = -inv4pi * Rn(q[5]);
    Rn f[8];
    f[0] = mass;
    f[4] = mad(bn, vb, (energy + pressure) * q[1]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      f[1 + i] = mad(bn, q[5 + i], i == 0 ? mad(mass, q[1], pressure) : mass * q[1 + i]);
      f[5 + i] = mad(q[1], q[5 + i], -(Rn(q[1 + i]) * q[5]));
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) flux[c] = side == 0 ? f[c] : flux[c] + f[c];
  }
  double diss[8];
  bool done = false;
  if (ROE) done = roe8Body<true>(diss, loc[0], loc[1], gamma, entropy, invGm1);
  if (!done) rusanovDissipation(diss, loc[0], loc[1], gamma, invGm1);
  const Rn area = 0.5 * (Rn(radialArea) * g.norm);
  Rn num[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) num[c] = area * (flux[c] - diss[c]);
  out[0] = num[0];
  out[4] = num[4];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    out[1 + i] = dot3(g.f[i], num[1], g.f[3 + i], num[2], g.f[6 + i], num[3]);
    out[5 + i] = dot3(g.f[i], num[5], g.f[3 + i], num[6], g.f[6 + i], num[7]);
  }
}

// src/MHD_StateConversion.H:11-32 (no constant-background magnetic test).
HC_DEV void cartesianPrimitiveFromConserved(double out[8], const double in[8], double inverseJ, double gamma) {
  Rn u[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) u[c] = Rn(in[c]) * inverseJ;
  const Rn rho = u[0] < kMP / 100 ? kMP / 100 : u[0].v;
  const Rn inv = rcpDensity(rho);
  out[0] = rho;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    out[1 + d] = u[1 + d] * inv;
    out[5 + d] = u[5 + d];
  }
  // rho |v|^2 as m . v, but inf * 0 (no kinetic energy at all) of an infinite density
  const Rn m2 = inv.v == 0.0 ? CUDART_NAN : dot3(u[1], out[1], u[2], out[2], u[3], out[3]).v;
  const Rn b2 = dot3(u[5], u[5], u[6], u[6], u[7], u[7]);
  const Rn pressure = (gamma - 1.0) * (mad(-0.5, m2, u[4]) - (0.125 / kPi) * b2);
  out[4] = pressure < 0.0 ? 0.0 : pressure.v;
}

// Inner analytic wind, native conserved variables at Cartesian point X and
// time t (src/BoxOp_PreStage.H:7-47, f_radialoutflowIBCs).
HC_DEV void windConserved(double gam, double r_BC, double strength, const double X[3], double t, double u[8]) {
  const double r = sqrt(X[0] * X[0] + X[1] * X[1] + X[2] * X[2]);
  const double theta = atan2(sqrt(X[0] * X[0] + X[1] * X[1]), X[2]);
  const double phi = atan2(X[1], X[0]);
  const double p0 = 1.0e-7, rho0 = 700 * kMP, u0 = 500.0 * 1e5;
  const double rho = rho0 * pow(r_BC / r, 2.0);
  const double p = p0 * pow(r_BC / r, 2.0 * gam);
  const double carr_rot_time = 25.38 * 24 * 60 * 60;
  const double omega = 2.0 * kPi / carr_rot_time;
  const double phit = phi - omega * t;
  const double perturbationScale = strength / 100.0;
  const double sinTheta = sin(theta);
  const double angularPattern = pow(sinTheta, 5) * sin(5 * phit) + pow(sinTheta, 10) * sin(10 * phit);
  const double ur = u0 - perturbationScale * u0 / 3 * angularPattern;
  u[0] = rho;
  u[1] = ur * rho;
  u[2] = u[3] = u[5] = u[6] = u[7] = 0.0;
  const double umag = sqrt(u[1] * u[1]) / u[0];
  u[4] = p / (gam - 1.0) + 0.5 * u[0] * umag * umag + 0.0 / 8.0 / kPi;
}

// Native averages of one cell from fourth-order Cartesian averages
// (src/MHD_CachedCartesianConversion.H:65-124): c0 points at the cell's
// component 0 (neighbours j +- 1 at +-sj, k +- 1 at +-sk, components sc
// apart); cf at the cell's 27 conversion coefficients (<A>^-1, D1 <A>,
// D2 <A>), the neighbours' at +-cj, +-ck.
HC_DEV void o4NativeCore(const double* c0, long sj, long sk, long sc, const double* cf,
                         long cj, long ck, double out[8]) {
  out[0] = c0[0];
  out[4] = c0[4 * sc];
  const long nOff[4] = {sj, -sj, sk, -sk};
  const long cOff[4] = {cj, -cj, ck, -ck};
#pragma unroll
  for (int grp = 0; grp < 2; ++grp) {
    const int st = grp == 0 ? 1 : 5;
    const double* cs = c0 + st * sc;
    double q[4][3];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double* I = cf + cOff[e];
      const double* x = cs + nOff[e];
      const double x0 = x[0];
      const double x1 = x[sc];
      const double x2 = x[2 * sc];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        double v = 0.0;
        v += I[3 * r] * x0 * 1.0;
        v += I[3 * r + 1] * x1 * 1.0;
        v += I[3 * r + 2] * x2 * 1.0;
        q[e][r] = v;
      }
    }
    double d1[3], d2[3], corrected[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      d1[r] = 0.5 * (q[0][r] - q[1][r]);
      d2[r] = 0.5 * (q[2][r] - q[3][r]);
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double first = 0.0, second = 0.0;
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        first += cf[9 + 3 * r + s] * d1[s] * (-1.0 / 12.0);
        second += cf[18 + 3 * r + s] * d2[s] * (-1.0 / 12.0);
      }
      double correction = 0.0;
      correction += first;
      correction += second;
      corrected[r] = cs[r * sc] + correction;
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double v = 0.0;
#pragma unroll
      for (int s = 0; s < 3; ++s) v += cf[3 * r + s] * corrected[s] * 1.0;
      out[st + r] = v;
    }
  }
}

// Classical RK4 after a stage (the tableau of src/MHD_AMRRungeKutta.H:10-12)
// of the eight components at offset `at`, n apart.
template <class U>
HC_DEV void rkUpdate(const U& u, double dt, long at, long n, const Rn kv[8]) {
  const Rn fb = dt * (u.stage == 0 || u.stage == 3 ? 1.0 / 6 : 1.0 / 3), fa = dt * (u.stage == 2 ? 1.0 : 0.5);
  double v[8], w[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    v[q] = u.stage == 3 ? 0.0 : u.ju[at + q * n];
    w[q] = u.stage == 0 ? v[q] : u.acc[at + q * n];
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const double sum = mad(fb, kv[q], w[q]);
    if (u.stage == 3) {
      u.ju[at + q * n] = sum;
    } else {
      u.acc[at + q * n] = sum;
      u.next[at + q * n] = mad(fa, kv[q], v[q]);
    }
  }
}

}  // namespace hc
